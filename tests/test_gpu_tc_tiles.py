"""Tile edges of the tensor-core sums: column counts around the narrow tile (one
launch), one and two wide tiles (two launches that pass partial sums), for the
synthetics (6 slices) and the coupling (7 slices).  Reference: the FP64 form;
bars as in the other tests of the mixed form, 1e-5 per trace and 1e-8 of each
coupling spectrum's largest value."""
import dataclasses

import numpy as np
import pytest

from gemini_unified_b200 import configs, model as M

pytestmark = pytest.mark.gpu
W = dataclasses.replace(configs.GLOBAL_SMALL, params=dataclasses.replace(configs.GLOBAL_SMALL.params, fmax=0.03))


@pytest.fixture(scope="module")
def ctx(gpu):
    from gemini_unified_b200.fk import GeminiFK
    from gemini_unified_b200.synth_run import fk_coefficients
    m = W.model()
    ex = W.nodes(m)
    g = M.frequency_grid(W.params, m.rearth)
    gr, gi = fk_coefficients(20, int(g.nkfmax))
    return g, gr, gi, {b: GeminiFK(m, ex, backend=b) for b in (1, 2)}


def _synthetics(ctx, backend, n):
    from gemini_unified_b200.fk import synth_params
    g, gr, gi, fk = ctx
    rng = np.random.default_rng(n)
    theta = np.radians(rng.uniform(1.0, 170.0, n))
    phi, prop = rng.uniform(-3.0, 3.0, (2, n))
    sp = synth_params(g, 10, 1024, 1.0, W.filspecs)
    return fk[backend].synthetics(sp, g.nwn, gr[:10], gi[:10], theta, phi, prop, np.eye(6)[[0, 4]])


@pytest.mark.parametrize("n", [1, 79, 80, 81, 159, 160, 161, 321])
def test_synthetics_at_tile_edges(ctx, n):
    got, ref = _synthetics(ctx, 2, n).astype(np.float64), _synthetics(ctx, 1, n).astype(np.float64)
    err = np.linalg.norm(got - ref, axis=-1) / np.linalg.norm(ref, axis=-1)
    assert np.all(np.isfinite(got)) and err.max() <= 1e-5


@pytest.mark.parametrize("n", [1, 64, 65, 127, 128, 129, 257])
def test_coupling_at_tile_edges(ctx, n):
    from gemini_unified_b200.fk import CouplingParams
    g, gr, gi, fk = ctx
    rng = np.random.default_rng(n)
    cp = CouplingParams(nf1=g.nf1, nf2=g.nf2, nwnmax=g.nwnmax, nkfmax=int(g.nkfmax), nsp=20, df=g.df, sigma=g.sigma,
                        re=6361000.0, nsamp=1024, dt=1.0, tred=0.0, order_highpass=2, fc_highpass=0.002,
                        order_lowpass=4, fc_lowpass=0.02, thetas=0.3, phis=1.0, thetac=0.5, phic=1.2, spectra=1)
    zel = np.tile(np.array([1.1e11 + 1e8j, 1.2e11 + 1e8j, 4e10, 4.5e10 + 5e7j, 4.4e10, 0, 0]), (g.nf2, 1))
    nrm = rng.normal(size=(n, 3))
    a = (g.nwn, gr, gi, zel, np.array([1.0, -0.4, 0.7, 0.3, -0.5, 0.2]), np.radians(rng.uniform(5.0, 90.0, n)),
         rng.uniform(-3.0, 3.0, n), nrm / np.linalg.norm(nrm, axis=1, keepdims=True))
    got, ref = fk[2].coupling(cp, *a), fk[1].coupling(cp, *a)
    assert np.all(np.isfinite(got))
    assert np.max(np.abs(got - ref) / np.abs(ref).max(axis=2, keepdims=True)) <= 1e-8


def test_wait_limit_in_the_two_launch_form(ctx):
    from gemini_unified_b200.model import GeminiError
    fk = ctx[3][2]
    fk.tc_wait_limit(1)
    with pytest.raises(GeminiError, match="timed out"):
        _synthetics(ctx, 2, 200)
    fk.tc_wait_limit(0)
    test_synthetics_at_tile_edges(ctx, 200)


def test_device_memory_of_a_call(ctx):
    """A call holds the FP64 tables and sums, the slices of both operands, the spectra and small
    inputs, and no more than the coefficient rows besides (20000 stations: 1.15 GB; the tables'
    exponents and the partial sums of the two launches would add 0.44 GB)."""
    import ctypes
    import torch
    from gemini_unified_b200.fk import FrequencyTime, lib, synth_params
    g, gr, gi, _ = ctx
    rng = np.random.default_rng(3)
    sp = synth_params(g, 10, 512, 1.0 / (512 * g.df), W.filspecs)
    ft = FrequencyTime(backend=2)
    d = [torch.from_numpy(np.ascontiguousarray(a[:10])).cuda() for a in (gr, gi)]
    nwn, mt = np.ascontiguousarray(g.nwn, np.int32), np.ascontiguousarray(np.eye(6)[[1]])
    vp = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    free = []
    for n in (200, 20000):
        out = torch.empty((n, 1, 3, 512), dtype=torch.float32, device="cuda")
        theta = np.radians(rng.uniform(1.0, 170.0, n))
        phi, prop = rng.uniform(-3.0, 3.0, n), rng.uniform(-3.0, 3.0, n)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
        assert lib().gem_synth_run_device(ft._h, ctypes.byref(sp), vp(nwn), d[0].data_ptr(), d[1].data_ptr(), n, vp(theta), vp(phi),
                                          vp(prop), 1, vp(mt), out.data_ptr(), None) < 2
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    nf, lcap = g.nf2 - g.nf1 + 1, int(g.nwnmax)
    kp, rows = -(-lcap // 64) * 64, 2 * nf * 14
    most = n * (8 * lcap * 8 + rows * 8 + 3 * g.nf2 * 16 + 6 * 8 * kp) + rows * (6 * kp + 8 * lcap)
    assert free[2] - free[3] <= most + (8 << 20)   # allocations come in steps of 2 MB
