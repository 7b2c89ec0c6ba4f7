"""Workloads of the FK / seismogram library as a user's program runs them.

Each case is one call of a public entry point on sizes of the repository's own configurations
(gemini_unified_b200/configs.py) or on generic ones: FK spectra of a frequency slab, the ASKI set
run, seismograms of many stations, SPECFEM-coupling time series, and the batched inverse transform.
``listed`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes what a program
holds before the call, ``run`` is the call, ``work`` its unavoidable bytes and flops, and ``exact``
the same outputs in plain 64-bit arithmetic where they have a closed formula (the degree sums,
wavenumber integrals, filters and transforms; the FK spectra come from an adaptive ODE integration
and have none).
"""
from __future__ import annotations

import ctypes
import dataclasses
import math

import numpy as np
import torch

from gemini_unified_b200 import configs, fk as F, model as M

PI_F = 3.1415927410125732          # the reference's single-precision pi, widened
TWO_PI_F = 2.0 * PI_F

# radial nodes below the surface: the configurations' own blocks
BLOCKS = {
    "one": ([1], [10000.0]),                         # one source at 10 km
    "four": ([4], [10000.0]),
    "depths": ([1, 19], [5000.0, 695000.0 / 19.0]),  # 20 depths, 5..700 km
    "crust24": ([24], [1000.0]),                     # regional: 24 depths, 1..24 km
    "crust7": ([7], [1000.0]),
}


# ---------------------------------------------------------------------------
#  The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one frequency of the small global band: the per-frequency call of the reference's loop
        dict(name="fk_one_frequency", kind="fk", earth="prem", backend=2, tlen=1024.0, fmax=0.05, p=3.5e-4,
             jf1=8, jf2=8, blocks="one", source="MOMENT", stress=False, host=True, f64=True),
        # the whole small global band (18,169 solves), spectra for one event depth
        dict(name="fk_global_small", kind="fk", earth="prem", backend=2, tlen=1024.0, fmax=0.05, p=3.5e-4,
             jf1=2, jf2=52, blocks="one", source="MOMENT", stress=False, host=False, f64=False),
        # the same band in the reference's operation order (parity backend)
        dict(name="fk_global_small_fp64", kind="fk", earth="prem", backend=1, tlen=1024.0, fmax=0.05, p=3.5e-4,
             jf1=2, jf2=52, blocks="one", source="MOMENT", stress=False, host=False, f64=True),
        # force sources with stresses, transversely isotropic model, a slab as one rank of a job gets it
        dict(name="fk_force_stress_slab", kind="fk", earth="prem_ti", backend=2, tlen=2048.0, fmax=0.2, p=4.0e-4,
             jf1=120, jf2=181, blocks="four", source="FORCE", stress=True, host=False, f64=True),
        # the library's benchmark band: 658,944 solves, 37 nodes
        dict(name="fk_batched_band", kind="fk", earth="prem", backend=2, tlen=2048.0, fmax=0.2, p=4.0e-4,
             jf1=2, jf2=411, blocks="depths", source="MOMENT", stress=False, host=False, f64=False),
        # regional mode: a crustal model to 1 Hz, 24 source depths (82,000 solves)
        dict(name="fk_regional", kind="fk", earth="crust", backend=2, tlen=102.4, fmax=1.0, p=1.0 / 1600.0,
             jf1=2, jf2=103, blocks="crust24", source="MOMENT", stress=False, host=False, f64=False),
        # waveform-inversion kernels: DSV spectra with derivatives of a set of source nodes
        dict(name="aski_set", kind="aski", earth="prem", backend=2, tlen=2048.0, fmax=0.2, p=4.0e-4, jf1=200, jf2=207,
             blocks="depths", source="MOMENT", nsrc=9),
        # one event, a station list, a source wavelet and reduction times: the everyday seismogram job
        dict(name="synth_one_event", kind="synth", mode="global", backend=2, tlen=1024.0, fmax=0.05, p=3.5e-4,
             nsta=50, nmt=1, source="MOMENT", nsamp=2048, opts=True, host=True),
        # Green's functions of a large network: 4000 stations x 6 unit moment tensors x 8192 samples
        dict(name="synth_network", kind="synth", mode="global", backend=2, tlen=2048.0, fmax=0.2, p=4.0e-4,
             nsta=4000, nmt=6, source="MOMENT", nsamp=8192, opts=False, host=False),
        # regional seismograms (wavenumber integrals), single forces, an odd number of stations
        dict(name="synth_regional_force", kind="synth", mode="regional", backend=2, tlen=102.4, fmax=5.0, p=1.0 / 1600.0,
             nsta=1001, nmt=3, source="FORCE", nsamp=2048, opts=False, host=False),
        # SPECFEM coupling: velocity and traction at the boundary points of one node
        dict(name="coupling_box", kind="coupling", backend=2, tlen=2048.0, fmax=0.2, p=4.0e-4, npts=1000,
             source="MOMENT", nsamp=1024),
        # the batched frequency-to-time transform alone, an odd number of series
        dict(name="ifft_batch", kind="ifft", backend=2, tlen=2048.0, fmax=0.2, ntr=12001, nsamp=8192),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# flops of one (omega, l) solve, from the solver's own step counters: a + b f
FLOPS = {"prem": (1.4e6, 4.05e7), "prem_ti": (1.4e6, 4.05e7), "crust": (0.9e6, 0.9e6)}


def _fk_flops(c, g):
    a, b = FLOPS[c["earth"]]
    jf = np.arange(c["jf1"], c["jf2"] + 1)
    return float(np.sum(g.nwn[jf - 1] * (a + b * (jf - 1) * g.df)))


def draw(rng):
    kind = rng.choice(["fk", "fk", "fk", "aski", "synth", "synth", "synth", "coupling", "ifft"])
    backend = 2 if rng.random() < 0.8 else 1
    if kind in ("fk", "aski"):
        while True:
            if kind == "fk" and rng.random() < 0.3:
                c = dict(kind="fk", earth="crust", backend=backend, tlen=102.4, fmax=round(rng.uniform(0.4, 2.0), 2),
                         p=1.0 / 1600.0, blocks=rng.choice(["crust24", "crust7"]))
            else:
                c = dict(kind=kind, earth=rng.choice(["prem", "prem", "prem_ti"]), backend=backend,
                         tlen=rng.choice([1024.0, 2048.0]), fmax=round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4),
                         p=rng.choice([3.5e-4, 4.0e-4]), blocks=rng.choice(["one", "four", "depths"]))
            c["source"] = rng.choice(["MOMENT", "MOMENT", "FORCE"])
            g = _grid(c)
            n = min(g.nf2 - g.nf1 + 1, _logint(rng, 1, 400))
            if kind == "aski":
                n = min(n, 12)
                c["blocks"] = rng.choice(["four", "depths"])
                c["nsrc"] = rng.randint(1, 4 if c["blocks"] == "four" else 9)
            c["jf1"] = rng.randint(g.nf1, g.nf2 - n + 1)
            c["jf2"] = c["jf1"] + n - 1
            cost = _fk_flops(c, g) * (4.0 if backend == 1 else 1.0) * (0.4 * c["nsrc"] if kind == "aski" else 1.0)
            if cost > 2.5e12:
                continue
            if kind == "fk":
                c["stress"] = rng.random() < 0.3
                c["host"] = rng.random() < 0.3
                c["f64"] = rng.random() < 0.3
            return c
    if kind == "synth":
        regional = rng.random() < 0.4
        nmt = rng.choice([1, 2, 3, 6])
        nsta = _logint(rng, 1, 4000 if not regional else 1500)
        c = dict(kind="synth", mode="regional" if regional else "global", backend=backend,
                 nsta=nsta, nmt=nmt, source=rng.choice(["MOMENT", "FORCE"]), opts=rng.random() < 0.25,
                 host=nsta * nmt < 1000 and rng.random() < 0.3)
        if regional:
            c.update(tlen=102.4, fmax=round(rng.uniform(0.5, 5.0), 2), p=1.0 / 1600.0, nsamp=rng.choice([1024, 2048, 4096]))
        else:
            c.update(tlen=rng.choice([1024.0, 2048.0]), fmax=round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4),
                     p=rng.choice([3.5e-4, 4.0e-4]), nsamp=rng.choice([1024, 2048, 4096, 8192]))
        return c
    if kind == "coupling":
        return dict(kind="coupling", backend=backend, tlen=rng.choice([1024.0, 2048.0]),
                    fmax=round(math.exp(rng.uniform(math.log(0.02), math.log(0.2))), 4), p=rng.choice([3.5e-4, 4.0e-4]),
                    npts=_logint(rng, 10, 1000), source=rng.choice(["MOMENT", "FORCE"]), nsamp=rng.choice([1024, 2048]))
    return dict(kind="ifft", backend=backend, tlen=2048.0, fmax=round(math.exp(rng.uniform(math.log(0.01), math.log(0.24))), 4),
                ntr=_logint(rng, 1, 20000), nsamp=rng.choice([1024, 2048, 4096, 8192]))


# ---------------------------------------------------------------------------
#  Inputs
# ---------------------------------------------------------------------------
def _params(c):
    glob = 0 if c.get("earth") == "crust" or c.get("mode") == "regional" else 1
    kw = dict(tlen=c["tlen"], fmax=c["fmax"], p1lim=c["p"], p2lim=c["p"], frac=0.0, eps=1.0e-5, global_=glob,
              source_type=c.get("source", "MOMENT"), stressflag=bool(c.get("stress", False)))
    if not glob:
        kw["xlen"] = 2.56e6
    return M.FKParams(**kw)


def _grid(c):
    return M.frequency_grid(_params(c), 6371000.0)


def _earth(c, rng):
    """The case's earth model with its velocities and density changed by up to 1 % (smoothly in depth)."""
    m = configs.regional_crust() if c["earth"] == "crust" else configs.prem(isotropic=c["earth"] == "prem")
    x = m.depth / m.rearth

    def wiggle():
        a, ph = rng.uniform(-0.005, 0.005, 2), rng.uniform(0.0, 2.0 * np.pi, 2)
        return 1.0 + a[0] * np.sin(7.0 * x + ph[0]) + a[1] * np.sin(23.0 * x + ph[1])

    p, s, r = wiggle(), wiggle(), wiggle()
    return dataclasses.replace(m, vpv=m.vpv * p, vph=m.vph * p, vsv=m.vsv * s, vsh=m.vsh * s, ro=m.ro * r)


def _spectra(rng, nsp, nkf):
    """float32 FK coefficients: log-normal amplitudes, uniform phases."""
    amp = 10.0 ** np.clip(rng.normal(-3.0, 1.0, size=(nsp, nkf)), -6.0, 0.0)
    ph = rng.uniform(0.0, 2.0 * np.pi, size=(nsp, nkf))
    return (amp * np.cos(ph)).astype(np.float32), (amp * np.sin(ph)).astype(np.float32)


def _filter(c):
    return (2.0, 0.05, 4.0, 0.6 * c["fmax"]) if c.get("mode") == "regional" else (2.0, 0.002, 4.0, 0.8 * c["fmax"])


def _fft_length(nf2, nsamp):
    n = 2
    while n < 2 * nf2:
        n *= 2
    return max(n, nsamp)


def _synth_inputs(c, seed):
    rng = np.random.default_rng(seed)
    g = _grid(c)
    nsp = 10 if c["source"] == "MOMENT" else 5
    gr, gi = _spectra(rng, nsp, int(g.nkfmax))
    n = c["nsta"]
    if c["mode"] == "regional":
        theta = rng.uniform(1.0, 200.0, n) * 1000.0 / 6371000.0
    else:
        theta = np.radians(rng.uniform(0.5, 179.5, n))
    phi, prop = rng.uniform(-np.pi, np.pi, n), rng.uniform(-np.pi, np.pi, n)
    k = 6 if c["source"] == "MOMENT" else 3
    mt = np.eye(k) if c["nmt"] == k else rng.normal(size=(c["nmt"], k))
    nsamp = _fft_length(g.nf2, c["nsamp"])
    dt = 1.0 / (nsamp * g.df)
    o = {}
    if c["opts"]:
        t = np.arange(41) * dt
        o = dict(tred=rng.uniform(0.0, 60.0 * dt, n), stf=np.exp(-((t - 12.0 * dt) / (5.0 * dt)) ** 2).astype(np.float32),
                 tanf_stf=-8.0 * dt)
    return dict(g=g, nsp=nsp, gr=gr, gi=gi, theta=theta, phi=phi, prop=prop, mt=np.ascontiguousarray(mt), nsamp=nsamp, dt=dt,
                nwn=np.ascontiguousarray(g.nwn, np.int32), o=o)


ELCON = np.array([1.1e11 + 1e8j, 1.2e11 + 1e8j, 4e10, 4.5e10 + 5e7j, 4.4e10, 0, 0])   # a crustal solid
ANGLES = (0.3, 1.0, 0.5, 1.2)    # colatitude and longitude of the source and of the box centre
RE_NODE = 6361000.0


def _coupling_inputs(c, seed):
    rng = np.random.default_rng(seed)
    g = _grid(c)
    moment = c["source"] == "MOMENT"
    nsp = 20 if moment else 10
    gr, gi = _spectra(rng, nsp, int(g.nkfmax))
    for b in ([8, 16], [18, 20]) if moment else ([4, 8], [9, 10]):   # the radial derivatives' columns
        gr[b[0]:b[1]] *= np.float32(5.0e-5)
        gi[b[0]:b[1]] *= np.float32(5.0e-5)
    n = c["npts"]
    nrm = rng.normal(size=(n, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    mt = np.array([1.0, -0.4, 0.7, 0.3, -0.5, 0.2]) if moment else np.array([0.8, -0.3, 0.6])
    zel = ELCON[None, :] * (1.0 + 0.01 * np.arange(g.nf2)[:, None] * g.df)
    nsamp = _fft_length(g.nf2, c["nsamp"])
    return dict(g=g, nsp=nsp, gr=gr, gi=gi, delta=np.radians(rng.uniform(5.0, 90.0, n)),
                xi=np.radians(rng.uniform(-180.0, 180.0, n)), nrm=np.ascontiguousarray(nrm), mt=mt,
                zel=np.ascontiguousarray(zel), nsamp=nsamp, dt=1.0 / (nsamp * g.df),
                nwn=np.ascontiguousarray(g.nwn, np.int32))


def _ifft_inputs(c, seed):
    df = 1.0 / c["tlen"]
    nf2 = int(math.floor(c["fmax"] / df + 0.5)) + 1
    rng = np.random.default_rng(seed)
    sp = rng.normal(size=(c["ntr"], nf2)) + 1j * rng.normal(size=(c["ntr"], nf2))
    sp *= np.exp(-3.0 * np.arange(nf2) / nf2)[None, :]
    nsamp = _fft_length(nf2, c["nsamp"])
    return dict(df=df, sigma=5.0 * df, nf1=2, nf2=nf2, sp=sp, nsamp=nsamp, dt=1.0 / (nsamp * df))


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _check(ctx, rc):
    if rc >= 2:
        raise RuntimeError(F.lib().gem_last_error(ctx._h).decode())


def prepare(case, seed):
    c = dict(case)
    k = c["kind"]
    s = dict(c=c)
    if k in ("fk", "aski"):
        rng = np.random.default_rng(seed)
        m = _earth(c, rng)
        blocks, dr = BLOCKS[c["blocks"]]
        ex = M.ExternalRadialNodes.from_blocks(m, blocks, dr, 0.0, m.rearth)
        p, g = _params(c), _grid(c)
        jre = ex.node_index(m.rearth)
        s.update(fk=F.GeminiFK(m, ex, backend=c["backend"]), p=p, jre=jre)
        nkf = int(g.nwn[c["jf1"] - 1: c["jf2"]].sum())
        if k == "fk":
            if not c["host"]:
                n = ex.nnod * M.nsp_for(p) * nkf
                if c["f64"]:
                    s["g64"] = torch.empty(2 * n, dtype=torch.float64, device="cuda")
                else:
                    s["re"] = torch.empty(n, dtype=torch.float32, device="cuda")
                    s["im"] = torch.empty(n, dtype=torch.float32, device="cuda")
        else:
            js = sorted(set(np.linspace(1, jre, c["nsrc"]).astype(int).tolist() + [jre]))
            s["js"] = np.ascontiguousarray(js, np.int32)
            n = ex.nnod * nkf * (len(js) * M.nsp_dsv(c["source"]) + M.nsp_dsv("FORCE"))
            s["re"] = torch.empty(n, dtype=torch.float32, device="cuda")
            s["im"] = torch.empty(n, dtype=torch.float32, device="cuda")
            s["pc"] = F.fk_params_c(p, jre)
        s["status"] = torch.empty(nkf, dtype=torch.int32, device="cuda")
        return s
    if k == "ifft":
        i = _ifft_inputs(c, seed)
        s.update(i, ctx=F.FrequencyTime(backend=c["backend"]), sp=torch.from_numpy(i["sp"]).cuda())
        s["out"] = torch.empty((c["ntr"], i["nsamp"]), dtype=torch.float32, device="cuda")
        return s
    if k == "synth":
        i = _synth_inputs(c, seed)
        g = i["g"]
        par = F.synth_params(g, i["nsp"], i["nsamp"], i["dt"], _filter(c), velocity=c["opts"],
                             global_=0 if c["mode"] == "regional" else 1, source_type=c["source"])
        s.update(i, par=par)
        if c["host"]:
            m = configs.prem()
            s["fk"] = F.GeminiFK(m, M.ExternalRadialNodes.from_blocks(m, [1], [10000.0], 0.0, m.rearth), backend=c["backend"])
            return s
        s["ctx"] = F.FrequencyTime(backend=c["backend"])
        s["dgr"], s["dgi"] = torch.from_numpy(i["gr"]).cuda(), torch.from_numpy(i["gi"]).cuda()
        s["out"] = torch.empty((c["nsta"], len(i["mt"]), 3, i["nsamp"]), dtype=torch.float32, device="cuda")
        if i["o"]:
            o = i["o"]
            s["opt"] = F.StationOpts(_p(o["tred"]), None, None, len(o["stf"]), float(o["tanf_stf"]), _p(o["stf"]))
        return s
    i = _coupling_inputs(c, seed)
    g = i["g"]
    f = _filter(c)
    s.update(i, ctx=F.FrequencyTime(backend=c["backend"]))
    s["cp"] = F.CouplingParams(nf1=g.nf1, nf2=g.nf2, nwnmax=g.nwnmax, nkfmax=int(g.nkfmax), nsp=i["nsp"], df=g.df,
                               sigma=g.sigma, re=RE_NODE, nsamp=i["nsamp"], dt=i["dt"], tred=0.0, order_highpass=int(f[0]),
                               fc_highpass=f[1], order_lowpass=int(f[2]), fc_lowpass=f[3], thetas=ANGLES[0],
                               phis=ANGLES[1], thetac=ANGLES[2], phic=ANGLES[3], spectra=0,
                               istyp=1 if c["source"] == "MOMENT" else 0)
    s["dgr"], s["dgi"] = torch.from_numpy(i["gr"]).cuda(), torch.from_numpy(i["gi"]).cuda()
    s["out"] = torch.empty((c["npts"], 6, i["nsamp"]), dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------
#  One pass
# ---------------------------------------------------------------------------
def run(s):
    c, L = s["c"], F.lib()
    k = c["kind"]
    if k == "fk":
        if c["host"]:
            re, im, g64, st = s["fk"].run(s["p"], s["jre"], c["jf1"], c["jf2"], f64=c["f64"], raise_on_failure=False)
            return {"re": re, "im": im, "status": st, **({"g64": g64} if c["f64"] else {})}
        if c["f64"]:
            s["fk"].run_device(s["p"], s["jre"], c["jf1"], c["jf2"], gf64=s["g64"].data_ptr(), status=s["status"].data_ptr())
            return {"g64": s["g64"], "status": s["status"]}
        s["fk"].run_device(s["p"], s["jre"], c["jf1"], c["jf2"], gfre=s["re"].data_ptr(), gfim=s["im"].data_ptr(),
                           status=s["status"].data_ptr())
        return {"re": s["re"], "im": s["im"], "status": s["status"]}
    if k == "aski":
        _check(s["fk"], L.gem_fk_run_aski_device(s["fk"]._h, ctypes.byref(s["pc"]), len(s["js"]), _p(s["js"]), c["jf1"],
                                                 c["jf2"], s["re"].data_ptr(), s["im"].data_ptr(), None,
                                                 s["status"].data_ptr(), None))
        return {"re": s["re"], "im": s["im"], "status": s["status"]}
    if k == "ifft":
        s["ctx"].run_device(s["nf1"], s["nf2"], s["df"], s["sigma"], c["ntr"], s["sp"].data_ptr(), s["nf2"], s["nsamp"],
                            s["dt"], s["out"].data_ptr())
        return s["out"]
    if k == "synth":
        if c["host"]:
            return s["fk"].synthetics(s["par"], s["nwn"], s["gr"], s["gi"], s["theta"], s["phi"], s["prop"], s["mt"], **s["o"])
        a = (s["ctx"]._h, ctypes.byref(s["par"]), _p(s["nwn"]), s["dgr"].data_ptr(), s["dgi"].data_ptr(), c["nsta"],
             _p(s["theta"]), _p(s["phi"]), _p(s["prop"]), len(s["mt"]), _p(s["mt"]))
        if s["o"]:
            _check(s["ctx"], L.gem_synth_run_device_opts(*a, ctypes.byref(s["opt"]), s["out"].data_ptr(), None))
        else:
            _check(s["ctx"], L.gem_synth_run_device(*a, s["out"].data_ptr(), None))
        return s["out"]
    _check(s["ctx"], L.gem_coupling_run_device(s["ctx"]._h, ctypes.byref(s["cp"]), _p(s["nwn"]), s["dgr"].data_ptr(),
                                               s["dgi"].data_ptr(), _p(s["zel"]), _p(s["mt"]), c["npts"], _p(s["delta"]),
                                               _p(s["xi"]), _p(s["nrm"]), None, s["out"].data_ptr(), None))
    return {"velocity": s["out"][:, :3], "traction": s["out"][:, 3:]}


# ---------------------------------------------------------------------------
#  What a pass cannot do without
# ---------------------------------------------------------------------------
def _fft_flops(n):
    return 2.5 * n * math.log2(n)      # real output


def work(case):
    c = dict(case)
    k = c["kind"]
    if k == "ifft":
        nf2 = int(math.floor(c["fmax"] * c["tlen"] + 0.5)) + 1
        n = _fft_length(nf2, c["nsamp"])
        return {"bytes": c["ntr"] * (16.0 * (nf2 - 1) + 4.0 * n), "flops": c["ntr"] * _fft_flops(n)}
    g = _grid(c)
    if k in ("fk", "aski"):
        blocks = BLOCKS[c["blocks"]][0]
        nnod = sum(blocks) + 1
        nkf = int(g.nwn[c["jf1"] - 1: c["jf2"]].sum())
        if k == "fk":
            per = M.nsp_for(_params(c)) * (16.0 if c["f64"] else 8.0) + (8.0 * M.nsp_for(_params(c)) if c["f64"] and c["host"] else 0.0)
            return {"bytes": nkf * (nnod * per + 4.0), "flops": _fk_flops(c, g)}
        ns = c["nsrc"] * M.nsp_dsv(c["source"]) + M.nsp_dsv("FORCE")
        return {"bytes": nkf * (nnod * ns * 8.0 + 4.0), "flops": _fk_flops(c, g) * (1.0 + 0.3 * c["nsrc"])}
    nwn = g.nwn[g.nf1 - 1:].astype(np.float64)
    nf = len(nwn)
    n = _fft_length(g.nf2, c["nsamp"])
    if k == "synth":
        nsum, nsp, nel = (14, 10, 6) if c["source"] == "MOMENT" else (7, 5, 3)
        ntr = 3.0 * c["nsta"] * c["nmt"]
        return {"bytes": 8.0 * nsp * nwn.sum() + 4.0 * ntr * n + 24.0 * c["nsta"],
                "flops": 4.0 * nsum * nwn.sum() * c["nsta"] + 8.0 * nel * ntr * nf + ntr * _fft_flops(n)}
    nsum, nsp = (42, 20) if c["source"] == "MOMENT" else (21, 10)
    return {"bytes": 8.0 * nsp * nwn.sum() + 24.0 * c["npts"] * n + 40.0 * c["npts"],
            "flops": 4.0 * nsum * nwn.sum() * c["npts"] + 6.0 * c["npts"] * _fft_flops(n)}


# ---------------------------------------------------------------------------
#  The same outputs in plain 64-bit arithmetic
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _time_series(X, nf1, df, sigma, nsamp, dt):
    """x(t_i) = df e^{sigma t_i} Re(inverse DFT of the Hermitian spectrum X [.., nf], first bin nf1-1)."""
    full = torch.zeros(X.shape[:-1] + (nsamp // 2 + 1,), dtype=torch.complex128, device=X.device)
    full[..., nf1 - 1: nf1 - 1 + X.shape[-1]] = X
    x = torch.fft.irfft(full, n=nsamp, norm="forward")
    x *= df * torch.exp(sigma * dt * torch.arange(nsamp, dtype=torch.float64, device=X.device))
    return x


def _butterworth(f, df, sigma, spec):
    """Band-pass at the complex frequencies f - i sigma / 2 pi (orders and corner frequencies in spec)."""
    fc = f - 1j * sigma / TWO_PI_F
    h = np.ones_like(fc)
    for j in range(1, int(spec[0]) + 1):
        z = fc / spec[1]
        h = h * z / (z - np.exp(1j * PI_F * (j - 0.5) / int(spec[0])))
    for j in range(1, int(spec[2]) + 1):
        z = fc / spec[3]
        h = h * (-1j) / (z - np.exp(1j * PI_F * (j - 0.5) / int(spec[2])))
    return h


def _legendre(theta, lmax, second):
    """P_l^m (m <= 2), dP/dtheta, P/sin and (second) d2P/dtheta2, d/dtheta(P/sin): {name m: [lmax+1, n]}."""
    ct, st = torch.cos(theta), torch.sin(theta)
    T = {}
    for m in range(3):
        P = torch.zeros((lmax + 1, len(theta)), dtype=torch.float64, device=theta.device)
        P[m] = {0: torch.ones_like(st), 1: st, 2: 3.0 * st * st}[m]
        if lmax > m:
            P[m + 1] = ct * (2 * m + 1) * P[m]
        for l in range(m + 2, lmax + 1):
            P[l] = (ct * (2 * l - 1) * P[l - 1] - (l + m - 1) * P[l - 2]) / (l - m)
        l = torch.arange(lmax + 1, dtype=torch.float64, device=theta.device)[:, None]
        prev = torch.cat([torch.zeros_like(P[:1]), P[:-1]])
        D = (l * ct * P - (l + m) * prev) / st
        D[:m] = 0.0
        T["p", m], T["d", m] = P, D
        if m:
            T["s", m] = P / st
        if second:
            T["dd", m] = -(ct / st) * D + (m * m / (st * st) - l * (l + 1.0)) * P
            T["dd", m][:m] = 0.0
            if m:
                T["ds", m] = (D - (ct / st) * P) / st
    return T


# the sums of displacement: table, first degree, factor over l(l+1), column; moment tensors and single forces
MOMENT_SUMS = [("p0", 0, 0, 0), ("p0", 0, 0, 1), ("p1", 1, 2, 2), ("p2", 2, 2, 3), ("d0", 1, 0, 4), ("d0", 1, 0, 5),
               ("d1", 1, 2, 6), ("d2", 2, 2, 7), ("s1", 1, 2, 8), ("s2", 2, 4, 9), ("d1", 1, 2, 8), ("d2", 2, -2, 9),
               ("s1", 1, 2, 6), ("s2", 2, -4, 7)]
FORCE_SUMS = [("p0", 0, 0, 0), ("p1", 1, -2, 1), ("d0", 1, 0, 2), ("d1", 1, -2, 3), ("s1", 1, -2, 4), ("d1", 1, 2, 4),
              ("s1", 1, 2, 3)]


def _taper(lmax, nl):
    """cos^2 taper over the last fifth of the degrees 0..lmax."""
    jt = max(1, min(lmax, int(math.floor(lmax * 0.8 + 0.5))))
    l = np.arange(nl, dtype=np.float64)
    c = np.cos(l / (lmax * 0.2 * 2.0 / PI_F) - 0.8 / 0.2 * 0.5 * PI_F) ** 2
    return np.where(l < jt, 1.0, c)


def _degree_sums(g, gr, gi, tables, sums):
    """W[k] [nf, n] complex: sum over degrees of (2l+1)/4pi factor taper G(l) table(l), per sum and frequency."""
    dev = next(iter(tables.values())).device
    nf, nl = g.nf2 - g.nf1 + 1, int(g.nwnmax)
    l = np.arange(nl, dtype=np.float64)
    ll1 = np.float32(l * (l + 1)).astype(np.float64)
    tap = np.zeros((nf, nl))
    idx = np.zeros((nf, nl), np.int64)
    off = 0
    for i in range(nf):
        n = int(g.nwn[g.nf1 - 1 + i])
        tap[i, :n] = _taper(n - 1, n)
        idx[i] = off + np.minimum(np.arange(nl), n - 1)
        off += n
    base = torch.from_numpy(tap * (2.0 * l + 1.0) / (4.0 * PI_F)).to(dev)
    idx = torch.from_numpy(idx).to(dev)
    gr, gi = torch.from_numpy(gr).to(dev).double(), torch.from_numpy(gi).to(dev).double()
    out = []
    for name, l0, fac, col in sums:
        w = np.where(l >= l0, fac / np.maximum(ll1, 1.0) if fac else 1.0, 0.0)
        a = base * torch.from_numpy(w).to(dev)
        out.append(torch.complex((a * gr[col][idx]) @ tables[name], (a * gi[col][idx]) @ tables[name]))
    return out


def _wn_kernel(kind, wn, b0, b1, b2, re, x):
    if kind == 0:
        return wn * b0
    if kind == 1:
        return 2.0 / re * b1
    if kind == 2:
        return wn * 2.0 * b2
    if kind == 3:
        return wn * (-wn * re) * b1
    if kind == 4:
        return wn * 2.0 * (b0 - b1 / (wn * x))
    if kind == 5:
        return wn * 2.0 * wn * re * (b1 - 2.0 * b2 / (wn * x))
    if kind == 6:
        return wn * 2.0 * b1 / (wn * x)
    return wn * 4.0 * wn * re * b2 / (wn * x)


WN_KIND = {"FORCE": [0, 1, 3, 4, 6, 4, 6], "MOMENT": [0, 0, 1, 2, 3, 3, 4, 5, 6, 7, 4, 5, 6, 7]}
WN_SIGN = {"FORCE": [1, -1, 1, -1, -1, 1, 1], "MOMENT": [1] * 11 + [-1, 1, -1]}


def _wavenumber_integrals(c, g, par, gr, gi, theta):
    """W[k] [nf, n]: trapezoid / Filon integrals of the regional mode with their end terms."""
    dev = theta.device
    j0, j1 = torch.special.bessel_j0, torch.special.bessel_j1
    y0, y1 = torch.special.bessel_y0, torch.special.bessel_y1
    re, dwn = par.rearth, par.dwn
    x = torch.clamp(theta * re, min=3.0 / (dwn * 1.0e9))
    j3 = (3.0 / x / dwn).long() + 2
    xdk = x * dwn
    Fw = (1.0 - torch.cos(xdk)) / xdk / x
    nl, nf = int(g.nwnmax), g.nf2 - g.nf1 + 1
    j = torch.arange(1, nl + 1, device=dev)[:, None]
    w = torch.where(j < j3, torch.full_like(x, dwn)[None], torch.where(j == j3, 0.5 * dwn + Fw, 2.0 * Fw)) * (j >= 2)
    wn = (j - 1).double() * dwn
    a = torch.where(j >= 2, wn * x, torch.ones_like(x))
    b0, b1 = j0(a), j1(a)
    b2 = -b0 + 2.0 / a * b1
    wns = torch.where(j >= 2, wn, torch.ones_like(wn))
    scale = re * re / (2.0 * PI_F)
    kinds, signs, cols = WN_KIND[c["source"]], WN_SIGN[c["source"]], [s[3] for s in (MOMENT_SUMS if c["source"] == "MOMENT" else FORCE_SUMS)]
    tab = {k: _wn_kernel(k, wns, b0, b1, b2, re, x) * w * scale for k in set(kinds)}
    n_f = np.array([int(g.nwn[g.nf1 - 1 + i]) for i in range(nf)])
    tap, idx, off = np.zeros((nf, nl)), np.zeros((nf, nl), np.int64), 0
    for i, n in enumerate(n_f):
        jt = max(1, min(int(n), int(math.floor(n * 0.8 + 0.5))))
        jj = np.arange(1, n + 1)
        cc = np.cos((jj - 1) * dwn / ((n - 1) * dwn * 0.2 * 2.0 / PI_F) - 0.8 / 0.2 * 0.5 * PI_F) ** 2
        tap[i, :n] = np.where(jj < jt, 1.0, cc)
        idx[i] = off + np.minimum(np.arange(nl), n - 1)
        off += int(n)
    tap, idx = torch.from_numpy(tap).to(dev), torch.from_numpy(idx).to(dev)
    gr, gi = torch.from_numpy(gr).to(dev).double(), torch.from_numpy(gi).to(dev).double()
    nn = torch.from_numpy(n_f).to(dev)[:, None]
    rows = torch.arange(nf, device=dev)[:, None]
    tn = tap[rows, nn - 1]
    i3 = torch.clamp(j3[None, :], max=nl).expand(nf, -1)
    t3 = tap[rows, i3 - 1]

    def at(kind, jj, neumann):
        wv = (jj - 1).double() * dwn
        q = wv * x[None, :]
        c0, c1 = (y0(q), y1(q)) if neumann else (j0(q), j1(q))
        return _wn_kernel(kind, wv, c0, c1, -c0 + 2.0 / q * c1, re, x[None, :])

    out = []
    ends = {}
    for k in set(kinds):
        ends[k] = (at(k, nn, False), at(k, nn, True), at(k, i3, True))
    for kind, sg, col in zip(kinds, signs, cols):
        G = torch.complex(gr[col], gi[col])[idx] * tap
        W = torch.complex(G.real @ tab[kind], G.imag @ tab[kind])
        Gn, G3 = torch.complex(gr[col], gi[col])[idx][rows, nn - 1], torch.complex(gr[col], gi[col])[idx][rows, i3 - 1]
        jn, yn, y3 = ends[kind]
        filon = -(Gn * jn) * (tn * Fw) + (Gn * yn * tn - G3 * y3 * t3) / x * (1.0 - torch.sin(xdk) / xdk)
        at3 = -(Gn * jn) * (tn * Fw)
        trap = -(Gn * jn) * (tn * 0.5 * dwn)
        corr = torch.where(nn > j3, filon, torch.where(nn == j3, at3, trap)) * scale
        out.append(sg * (W + corr))
    return out


def _combine_moment(w, m, cphi, sphi, c2, s2):
    t1, t2 = m[3] * cphi + m[4] * sphi, (m[2] - m[1]) * c2 - 2.0 * m[5] * s2
    t3, t4 = m[4] * cphi - m[3] * sphi, (m[2] - m[1]) * s2 + 2.0 * m[5] * c2
    return [w[0] * m[0] + w[1] * (m[1] + m[2]) + w[2] * t1 + w[3] * t2,
            w[4] * m[0] + w[5] * (m[1] + m[2]) + (w[6] + w[8]) * t1 + (w[7] + w[9]) * t2,
            (w[10] + w[12]) * t3 + (w[11] + w[13]) * t4]


def _combine_force(w, f, cphi, sphi):
    fh = f[1] * cphi + f[2] * sphi
    return [w[0] * f[0] + w[1] * fh, w[2] * f[0] + (w[3] + w[4]) * fh, (w[5] + w[6]) * (f[1] * sphi - f[2] * cphi)]


def _exact_synth(c, seed):
    i = _synth_inputs(c, seed)
    g, dev = i["g"], _dev()
    par = F.synth_params(g, i["nsp"], i["nsamp"], i["dt"], _filter(c), velocity=c["opts"],
                         global_=0 if c["mode"] == "regional" else 1, source_type=c["source"])
    theta = torch.from_numpy(i["theta"]).to(dev)
    if c["mode"] == "regional":
        w = _wavenumber_integrals(c, g, par, i["gr"], i["gi"], theta)
    else:
        T = {k[0] + str(k[1]): v for k, v in _legendre(theta, int(g.nwnmax) - 1, False).items()}
        w = _degree_sums(g, i["gr"], i["gi"], T, MOMENT_SUMS if c["source"] == "MOMENT" else FORCE_SUMS)
        del T
    f = np.arange(g.nf1 - 1, g.nf2) * par.df
    h = torch.from_numpy(_butterworth(f, par.df, par.sigma, _filter(c))).to(dev)[:, None]
    om = torch.from_numpy(TWO_PI_F * f).to(dev)[:, None]
    if c["opts"]:
        tr = torch.from_numpy(i["o"]["tred"]).to(dev)[None, :]
        h = h * torch.exp(torch.complex(par.sigma * tr.expand(len(f), -1), om * tr)) * 1j * torch.complex(om, torch.full_like(om, -par.sigma))
    phi, prop = torch.from_numpy(i["phi"]).to(dev), torch.from_numpy(i["prop"]).to(dev)
    ca, sa = torch.cos(prop), torch.sin(prop)
    out = torch.empty((c["nsta"], len(i["mt"]), 3, i["nsamp"]), dtype=torch.float64, device=dev)
    for q, m in enumerate(i["mt"]):
        if c["source"] == "MOMENT":
            z = _combine_moment(w, m, torch.cos(phi), torch.sin(phi), torch.cos(2.0 * phi), torch.sin(2.0 * phi))
        else:
            z = _combine_force(w, m, torch.cos(phi), torch.sin(phi))
        for k, v in enumerate((z[0], -ca * z[1] + sa * z[2], sa * z[1] + ca * z[2])):
            out[:, q, k] = _time_series((v * h).T.contiguous(), g.nf1, par.df, par.sigma, i["nsamp"], i["dt"])
    if c["opts"]:      # source wavelet: y_k = dt sum_n x_{k - n + nhm} s_n
        stf = torch.from_numpy(i["o"]["stf"].astype(np.float64)).to(dev)
        n, nhm = i["nsamp"], int(math.floor(abs(i["o"]["tanf_stf"]) / i["dt"] + 0.5))
        x, y = out, torch.zeros_like(out)
        for q in range(len(stf)):
            d = q - nhm                                  # sample k takes x[k - d]
            a, b = max(0, d), min(n, n + d)
            y[..., a:b] += i["dt"] * stf[q] * x[..., a - d:b - d]
        out = y
    return out


def _exact_coupling(c, seed):
    i = _coupling_inputs(c, seed)
    g, dev = i["g"], _dev()
    delta, xi = torch.from_numpy(i["delta"]).to(dev), torch.from_numpy(i["xi"]).to(dev)
    T = {k[0] + str(k[1]): v for k, v in _legendre(delta, int(g.nwnmax) - 1, True).items()}
    moment = c["source"] == "MOMENT"
    disp = MOMENT_SUMS if moment else FORCE_SUMS
    # columns: U, V per spheroidal jump, their derivatives, W, dW/dr per toroidal jump
    col_t = {8: 16, 9: 17} if moment else {4: 8}
    col_r = {**{k: k + 8 for k in range(8)}, 8: 18, 9: 19} if moment else {**{k: k + 4 for k in range(4)}, 4: 9}
    up = {"p0": "d0", "p1": "d1", "p2": "d2", "d0": "dd0", "d1": "dd1", "d2": "dd2", "s1": "ds1", "s2": "ds2"}
    # the theta derivative of a table of order 0 starts at degree 1 (its value at degree 0 is zero)
    sets = [[(t, l0, fac, col_t.get(k, k)) for t, l0, fac, k in disp], [(t, l0, fac, col_r[k]) for t, l0, fac, k in disp],
            [(up[t], max(l0, 1), fac, col_t.get(k, k)) for t, l0, fac, k in disp]]
    W = [_degree_sums(g, i["gr"], i["gi"], T, s) for s in sets]
    del T
    cphi, sphi, c2, s2 = torch.cos(xi), torch.sin(xi), torch.cos(2.0 * xi), torch.sin(2.0 * xi)
    m, re = i["mt"], RE_NODE
    if moment:
        u, ur, ut = (_combine_moment(w, m, cphi, sphi, c2, s2) for w in W)
        # d/dphi of the azimuthal factors: cos -> -sin, sin -> cos, and twice that for the double angle
        t1, t2 = -m[3] * sphi + m[4] * cphi, -2.0 * (m[2] - m[1]) * s2 - 4.0 * m[5] * c2
        t3, t4 = -m[4] * sphi - m[3] * cphi, 2.0 * (m[2] - m[1]) * c2 - 4.0 * m[5] * s2
        w = W[0]
        uf = [w[2] * t1 + w[3] * t2, (w[6] + w[8]) * t1 + (w[7] + w[9]) * t2, (w[10] + w[12]) * t3 + (w[11] + w[13]) * t4]
    else:
        u, ur, ut = (_combine_force(w, m, cphi, sphi) for w in W)
        w, fp, fq = W[0], -m[1] * sphi + m[2] * cphi, m[1] * cphi + m[2] * sphi
        uf = [w[1] * fp, (w[3] + w[4]) * fp, (w[5] + w[6]) * fq]
    ut = [v / re for v in ut]
    uf = [v / (re * torch.sin(delta)) for v in uf]
    rtd = re * torch.tan(delta)
    err, ett, eff = ur[0], ut[1] + u[0] / re, uf[2] + u[0] / re + u[1] / rtd
    ert, erf, etf = 0.5 * (ut[0] + ur[1] - u[1] / re), 0.5 * (uf[0] + ur[2] - u[2] / re), 0.5 * (uf[1] + ut[2] - u[2] / rtd)
    A, C, Fc, Lc, N = (torch.from_numpy(np.ascontiguousarray(i["zel"][g.nf1 - 1:, q])).to(dev)[:, None] for q in range(5))
    S = torch.stack([torch.stack([C * err + Fc * (ett + eff), 2.0 * Lc * ert, 2.0 * Lc * erf]),
                     torch.stack([2.0 * Lc * ert, Fc * err + A * (ett + eff) - 2.0 * N * eff, 2.0 * N * etf]),
                     torch.stack([2.0 * Lc * erf, 2.0 * N * etf, Fc * err + A * (ett + eff) - 2.0 * N * ett])])
    # rotation: local spherical (r, theta, phi) -> local Cartesian at the source -> global -> box
    cd, sd = torch.cos(delta), torch.sin(delta)
    z = torch.zeros_like(cd)
    R = torch.stack([torch.stack([sd * cphi, cd * cphi, -sphi]), torch.stack([sd * sphi, cd * sphi, cphi]),
                     torch.stack([cd, -sd, z])])

    def gc_from_lc(t, p):
        return np.array([[math.cos(t) * math.cos(p), -math.sin(p), math.sin(t) * math.cos(p)],
                         [math.cos(t) * math.sin(p), math.cos(p), math.sin(t) * math.sin(p)],
                         [-math.sin(t), 0.0, math.cos(t)]])

    Q = gc_from_lc(0.0, 0.5 * PI_F).T @ gc_from_lc(ANGLES[2], ANGLES[3]).T @ gc_from_lc(ANGLES[0], ANGLES[1])
    R = torch.einsum("ij,jkn->ikn", torch.from_numpy(Q).to(dev), R).to(torch.complex128)
    v = torch.einsum("ikn,kfn->ifn", R, torch.stack(u))
    nrm = torch.from_numpy(i["nrm"]).to(dev).to(torch.complex128)
    back = torch.einsum("jln,nj->ln", R, nrm)
    tr = torch.einsum("ikn,klfn,ln->ifn", R, S, back)
    f = np.arange(g.nf1 - 1, g.nf2) * g.df
    h = torch.from_numpy(_butterworth(f, g.df, g.sigma, _filter(c))).to(dev)[None, :, None]
    om = torch.from_numpy(1j * (TWO_PI_F * f - 1j * g.sigma)).to(dev)[None, :, None]
    ts = lambda q: _time_series(q.permute(2, 0, 1).contiguous(), g.nf1, g.df, g.sigma, i["nsamp"], i["dt"])
    return {"velocity": ts(v * h * om), "traction": ts(tr * h)}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "ifft":
        i = _ifft_inputs(c, seed)
        sp = torch.from_numpy(i["sp"]).to(_dev())[:, i["nf1"] - 1:]
        return _time_series(sp, i["nf1"], i["df"], i["sigma"], i["nsamp"], i["dt"])
    if c["kind"] == "synth":
        return _exact_synth(c, seed)
    if c["kind"] == "coupling":
        return _exact_coupling(c, seed)
    return None    # FK spectra: an adaptive integration to a given accuracy, no closed 64-bit value
