"""The fast build's Bulirsch-Stoer step over the forms of an earth model it
distinguishes: isotropic (density, C and L evaluated) or not, knots on a regular
grid or searched, and steps that stay in one or two knot intervals or cross
several (fine knots at low frequency).  Reference: the FP64 form, which repeats
the reference's arithmetic and evaluates all constants; the spectra must agree
to 1e-8 of each spectrum's largest value, the FP64 spectral bar."""
import dataclasses

import numpy as np
import pytest

from gemini_unified_b200 import configs, model as M

pytestmark = pytest.mark.gpu


def _refined(m, n):
    """The model with n - 1 knots added in every knot interval of its layers (linear in between)."""
    cols = ("depth", "ro", "vpv", "vph", "vsv", "vsh", "eta", "qk", "qm")
    new = {c: [] for c in cols}
    top = []
    bot = m.ikbot
    for nl in range(m.nlay):
        a, b = (m.iktop[0] - 1, m.iktop[0] - 1) if nl == 0 else (bot[nl] - 1, m.iktop[nl] - 1)
        k = 1 if nl == 0 or (b - a) * n + 1 > 60 else n
        x = np.arange((b - a) * k + 1) / k + a
        for c in cols:
            new[c].append(np.interp(x, np.arange(m.nk), getattr(m, c)))
        top.append(sum(len(v) for v in new["ro"]))
    new = {c: np.concatenate(v) for c, v in new.items()}
    return dataclasses.replace(m, nk=len(new["ro"]), iktop=np.asarray(top, np.int32), **new)


MODELS = {
    "isotropic": lambda: configs.prem(),
    "transversely_isotropic": lambda: configs.prem(isotropic=False),
    "searched_knots": lambda: dataclasses.replace(configs.prem(), equidis=0),
    "fine_knots": lambda: _refined(configs.prem(), 2),
    "fine_searched_knots_ti": lambda: dataclasses.replace(_refined(configs.prem(isotropic=False), 2), equidis=0),
}


@pytest.mark.parametrize("name", sorted(MODELS))
@pytest.mark.parametrize("source,stress", [("MOMENT", False), ("FORCE", True)])
def test_fast_step_matches_the_fp64_form(gpu, name, source, stress):
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, GEM_BACKEND_GPU_FP64, GeminiFK
    w = configs.WORKLOADS["global_small"]
    m = MODELS[name]()
    ex = w.nodes(m)
    jre = ex.node_index(w.rec_radius)
    p = dataclasses.replace(w.params, source_type=source, stressflag=stress)
    for jf in (2, 9, 52):       # the lowest frequencies take the longest steps
        ref = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FP64).run(p, jre, jf, jf, f32=False)
        got = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST).run(p, jre, jf, jf, f32=False)
        np.testing.assert_array_equal(got[3], ref[3])
        np.testing.assert_array_equal(np.isnan(got[2]), np.isnan(ref[2]))
        scale = np.nanmax(np.abs(ref[2]), axis=2, keepdims=True)
        err = np.abs(got[2] - ref[2]) / np.where(scale > 0, scale, 1.0)
        assert np.nanmax(err) <= 1e-8


def _ocean(m):
    """The model with its top layer made an ocean."""
    sel = slice(int(m.ikbot[-1]) - 1, int(m.iktop[-1]))
    new = {}
    for c, v in (("ro", 1020.0), ("vpv", 1450.0), ("vph", 1450.0), ("vsv", 0.0), ("vsh", 0.0)):
        new[c] = getattr(m, c).copy()
        new[c][sel] = v
    iflso = m.iflso.copy()
    iflso[-1] = 1
    return dataclasses.replace(m, iflso=iflso, **new)


# The start radii (a warp per solve and motion type) with and without a fluid core, with an
# ocean (toroidal motion ends at its bottom) and in a full space; the first and last degree
# of the lowest, a middle and the highest frequency.  The FP64 form repeats the reference's
# arithmetic: 1e-10 of each frequency's largest value, as for the other models.
START_MODELS = {"core": lambda: configs.prem(), "ocean": lambda: _ocean(configs.prem()), "crust": configs.regional_crust,
                "full_space": lambda: dataclasses.replace(configs.prem(), fsflag=1)}


@pytest.mark.parametrize("name", sorted(START_MODELS))
def test_start_radii_of_other_models_match_oracle(gpu, name):
    import oracle
    from gemini_unified_b200.fk import GeminiFK
    w = configs.WORKLOADS["global_small"]
    m = START_MODELS[name]()
    ex = w.nodes(m)
    jre = next(j for j in range(ex.nnod, 0, -1) if ex.state[j - 1] == 0)
    g = M.frequency_grid(w.params, m.rearth)
    fk, o = GeminiFK(m, ex), oracle.Oracle(m, ex)
    pc = M.fk_params_c(w.params, jre)
    for jf in (g.nf1, 20, g.nf2):
        n = int(g.nwn[jf - 1])
        _, _, got, st = fk.run(w.params, jre, jf, jf, f32=False, raise_on_failure=False)
        for iwn in (1, 2, n // 2, n):
            ref, sto, _ = o.fk_frequency(pc, jf, n, 10, iwn, iwn)
            a, b = got[:, :, iwn - 1], ref[:, :, iwn - 1]
            assert st[iwn - 1] == sto[iwn - 1]
            assert np.array_equal(np.isnan(a), np.isnan(b))
            ok = ~np.isnan(b)
            assert np.abs(a[ok] - b[ok]).max(initial=0.0) <= 1e-10 * max(np.abs(b[ok]).max(initial=0.0), 1e-300)


RINV = r"""
#include <cuda_runtime.h>
#define GEM_NS probe
#define GEM_FAST 1
#include "fk_kernel.h"
#include "fk_solver.cuh"
__global__ void rinv_kernel(const double* x, double* r, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = probe::rinv(x[i]);
}
extern "C" int rinv_of(const double* x, double* r, int n) {
  rinv_kernel<<<(n + 255) / 256, 256>>>(x, r, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_reciprocal(gpu, tmp_path):
    """rinv, an approximation to 20 bits with one third-order step: its cube, 2^-60, is 0.008 of
    half a unit in the last place beside the rounding of the last operation; 0.52 ulp over the exponents
    at which neither x nor 1/x leaves the normal numbers."""
    import ctypes
    import os
    import subprocess
    import torch
    from gemini_unified_b200 import build
    src, so = tmp_path / "rinv.cu", str(tmp_path / "rinv.so")
    src.write_text(RINV)
    subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "--fmad=true", "-Xcompiler", "-fPIC", "-shared", "-I", build.CSRC,
                    str(src), "-o", so], check=True, capture_output=True)
    rng = np.random.default_rng(7)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1000, 1000, n)) * rng.choice([-1.0, 1.0], n)
    x[:4] = 1.0, -2.0, np.nextafter(2.0, 0.0), np.nextafter(1.0, 2.0)
    d_x = torch.from_numpy(x).cuda()
    d_r = torch.empty_like(d_x)
    torch.cuda.synchronize()
    assert ctypes.CDLL(so).rinv_of(ctypes.c_void_p(d_x.data_ptr()), ctypes.c_void_p(d_r.data_ptr()), n) == 0
    r = d_r.cpu().numpy()
    err = np.abs((x.astype(np.longdouble) * r - 1) / x / np.spacing(np.abs(r)))
    assert r[0] == 1.0 and r[1] == -0.5 and float(err.max()) <= 0.52
