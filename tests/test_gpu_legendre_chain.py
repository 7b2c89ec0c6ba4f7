"""Legendre tables and their scales at the edges of the 32-degree chunks and
32-column blocks, poles and zero rows included.  Reference: the FP64 form, whose
tables come from the plain recurrence; bars as in the other tests of the mixed
form, 1e-5 of a station's three traces and 1e-8 of each coupling spectrum's
largest value."""
import dataclasses

import numpy as np
import pytest

from gemini_unified_b200 import configs, model as M

pytestmark = pytest.mark.gpu
W = configs.GLOBAL_SMALL


@pytest.fixture(scope="module")
def fk(gpu):
    from gemini_unified_b200.fk import GeminiFK
    m = W.model()
    ex = W.nodes(m)
    return M.frequency_grid(W.params, m.rearth), {b: GeminiFK(m, ex, backend=b) for b in (1, 2)}


def _grid(g, n):
    """40 frequencies whose counts rise to n degrees and stay there."""
    nwn = np.zeros(g.nf1 + 39, np.int32)
    nwn[g.nf1 - 1:] = np.minimum(n, 3 + np.arange(40))
    return dataclasses.replace(g, nf2=len(nwn), nwn=nwn, nwnmax=n)


def _angles(nsta, rng):
    a = np.radians(rng.uniform(5.0, 90.0, nsta))
    a[nsta // 2] = 0.0   # sin = 0: the special values
    return a


@pytest.mark.parametrize("n,nsta", [(3, 1), (31, 33), (32, 31), (33, 32), (34, 5), (35, 65)])
def test_synthetics(fk, n, nsta):
    from gemini_unified_b200.fk import synth_params
    from gemini_unified_b200.synth_run import fk_coefficients
    g = _grid(fk[0], n)
    gr, gi = fk_coefficients(10, int(g.nkfmax))
    rng = np.random.default_rng(n)
    sp = synth_params(g, 10, 512, 1.0 / (512 * g.df), W.filspecs)
    a = (g.nwn, gr, gi, _angles(nsta, rng), rng.uniform(-3, 3, nsta), rng.uniform(-3, 3, nsta), np.eye(6)[[1, 4]])
    got, ref = (fk[1][b].synthetics(sp, *a).astype(np.float64) for b in (2, 1))
    norm = np.linalg.norm(ref, axis=(2, 3))
    assert np.all(np.isfinite(got)) and norm.min() > 0.0
    assert np.max(np.linalg.norm(got - ref, axis=(2, 3)) / norm) <= 1e-5


@pytest.mark.parametrize("n,npts", [(3, 1), (31, 33), (32, 31), (33, 32), (35, 65)])
def test_coupling(fk, n, npts):
    from gemini_unified_b200.fk import CouplingParams
    from gemini_unified_b200.synth_run import fk_coefficients
    g = _grid(fk[0], n)
    gr, gi = fk_coefficients(20, int(g.nkfmax))
    rng = np.random.default_rng(n)
    cp = CouplingParams(nf1=g.nf1, nf2=g.nf2, nwnmax=g.nwnmax, nkfmax=int(g.nkfmax), nsp=20, df=g.df, sigma=g.sigma,
                        re=6361000.0, nsamp=512, dt=1.0, tred=0.0, order_highpass=2, fc_highpass=0.002,
                        order_lowpass=4, fc_lowpass=0.02, thetas=0.3, phis=1.0, thetac=0.5, phic=1.2, spectra=1)
    zel = np.tile(np.array([1.1e11 + 1e8j, 1.2e11 + 1e8j, 4e10, 4.5e10 + 5e7j, 4.4e10, 0, 0]), (g.nf2, 1))
    nrm = rng.normal(size=(npts, 3))
    a = (g.nwn, gr, gi, zel, np.array([1.0, -0.4, 0.7, 0.3, -0.5, 0.2]), _angles(npts, rng),
         rng.uniform(-3.0, 3.0, npts), nrm / np.linalg.norm(nrm, axis=1, keepdims=True))
    got, ref = fk[1][2].coupling(cp, *a), fk[1][1].coupling(cp, *a)
    ok = np.isfinite(ref)   # the strain of a point on the axis is not defined
    assert np.array_equal(np.isfinite(got), ok)
    top = np.where(ok, np.abs(ref), 0.0).max(axis=2, keepdims=True)
    assert np.all(np.abs(got - ref)[ok] <= np.broadcast_to(1e-8 * top, ok.shape)[ok])


@pytest.mark.parametrize("nsta", [81, 200])
def test_partial_sums_beside_the_tables(fk, nsta):
    """Many frequencies of few degrees: the partial sums of the two launches do not fit the tables."""
    test_synthetics(fk, 35, nsta)
    test_coupling(fk, 35, nsta)
