"""Coefficient rows of the tensor-core sums around the degrees that a block keeps
(2048 with 256 threads, 4096 with 512) and beyond, where rows are formed twice.
Reference: the FP64 form; bar as in the other tests of the mixed form, 1e-5 of a
station's three traces."""
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


def _grid(g, counts):
    nwn = np.zeros(g.nf1 + 2, np.int32)
    nwn[g.nf1 - 1:] = counts
    return dataclasses.replace(g, nf2=len(nwn), nwn=nwn, nwnmax=max(counts))


def _run(fk, g, seed, gr, gi):
    from gemini_unified_b200.fk import synth_params
    rng = np.random.default_rng(seed)
    sp = synth_params(g, 10, 512, 1.0 / (512 * g.df), W.filspecs)
    a = (g.nwn, gr, gi, np.radians(rng.uniform(5.0, 150.0, 7)), rng.uniform(-3, 3, 7), rng.uniform(-3, 3, 7),
         np.eye(6)[[1, 4]])
    return (fk[1][b].synthetics(sp, *a).astype(np.float64) for b in (2, 1))


def _check(got, ref):
    norm = np.linalg.norm(ref, axis=(2, 3))
    assert np.all(np.isfinite(got)) and norm.min() > 0.0
    assert np.max(np.linalg.norm(got - ref, axis=(2, 3)) / norm) <= 1e-5


def test_undefined_below_the_first_degree(fk):
    """Horizontal spectra at degree 0, which no sum reads, and small values."""
    from gemini_unified_b200.synth_run import fk_coefficients
    g = _grid(fk[0], [300, 5, 299])
    gr, gi = (1e-28 * np.asarray(c, np.float32) for c in fk_coefficients(10, int(g.nkfmax)))
    for start in np.cumsum([0, 300, 5]):
        gr[4:, start], gi[4:, start] = np.nan, np.inf
    a, b = _run(fk, g, 300, gr, gi)
    _check(a, b)


@pytest.mark.parametrize("n", [1023, 2047, 2048, 2049, 4095, 4096, 4097, 9000])
def test_rows(fk, n):
    from gemini_unified_b200.synth_run import fk_coefficients
    g = _grid(fk[0], [n, 5, n - 1])   # rows of very different length share a tile
    _check(*_run(fk, g, n, *fk_coefficients(10, int(g.nkfmax))))


@pytest.mark.parametrize("counts", [(300, 0, 299), (3000, 0, 2999), (9000, 0, 2, 0), (300, 1, 299)])
def test_frequency_without_degrees(fk, counts):
    """A frequency without degrees (or with degree 0 alone) adds nothing: the other
    rows of its tile are as long as ever.  The spectra vanish there in the FP64 form."""
    from gemini_unified_b200.synth_run import fk_coefficients
    nwn = np.zeros(fk[0].nf1 - 1 + len(counts), np.int32)
    nwn[fk[0].nf1 - 1:] = counts
    g = dataclasses.replace(fk[0], nf2=len(nwn), nwn=nwn, nwnmax=max(counts))
    _check(*_run(fk, g, counts[0], *fk_coefficients(10, int(g.nkfmax))))
