"""The adjoint phase of a set of ASKI sources as one queue: source counts from
one up, a repeated source, sources out of order, every queue granularity (runs
of positions that cross from one source to the next) and failing solves."""
import dataclasses

import numpy as np
import pytest

from gemini_unified_b200 import configs, model as M

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(gpu):
    from gemini_unified_b200.fk import GeminiFK
    w = dataclasses.replace(configs.GLOBAL_SMALL, nnod_blocks=[4], dr_blocks=[10000.0])
    m = w.model()
    ex = w.nodes(m)
    return w, m, ex, ex.node_index(w.rec_radius), {b: GeminiFK(m, ex, backend=b) for b in (1, 2)}


def _rel(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    assert np.array_equal(na, nb)
    return np.abs(a[~na] - b[~na]).max() / np.abs(b[~na]).max()


@pytest.mark.parametrize("backend", [1, 2])
@pytest.mark.parametrize("srcs", [(-1,), (-1, 1), (2, -1, 2), (5, 3, -1, 1)])
def test_set_run_equals_single_source_runs(setup, srcs, backend):
    """Round-off apart (the minors' final normalisation differs between the node ranges): 1e-12."""
    w, m, ex, jre, fks = setup
    fk = fks[backend]
    js = [jre if j < 0 else j for j in srcs]
    force = dataclasses.replace(w.params, source_type="FORCE")
    first = None
    for gran in range(4):
        fk.queue_set([0, 0, gran])
        res = fk.aski_spectra(w.params, js, jre, 3, 6, f32=False)
        if first is None:
            first = res
        for (_, _, a, sa), (_, _, b, sb) in zip(res, first):
            assert np.all(sa == 0)
            np.testing.assert_array_equal(a, b)
    fk.queue_set([0, 0, 0])
    for (_, _, a, _), (s, q) in zip(first, [(s, w.params) for s in js] + [(jre, force)]):
        assert _rel(a, fk.run_dsv(q, s, 3, 6, f32=False)[2]) <= 1e-12


def test_failing_solves_keep_their_status(setup):
    """With an unreachable accuracy every solve of degree > 0 fails as a single-source run's does."""
    w, m, ex, jre, fks = setup
    p = dataclasses.replace(w.params, eps=1.0e-30)
    one = fks[1].run_dsv(p, jre, 4, 4, f32=False, raise_on_failure=False)
    many = fks[1].aski_spectra(p, [1, jre], jre, 4, 4, f32=False, raise_on_failure=False)
    assert np.all(one[3][1:] != 0)
    for _, _, a, st in many:
        np.testing.assert_array_equal(st[1:], one[3][1:])
        assert np.all(a[:, :, 1:] == 0)
