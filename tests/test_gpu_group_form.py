"""The group form of the fast solver's phases (small slabs) against the thread
form, which a run takes when its instruments are on: both make the same
arithmetic in the same order, so the spectra, statuses and step counts must be
equal bit for bit.  Slabs from a few solves to more than the groups in flight,
every system (toroidal, minors, fluid, degree 0, adjoint), isotropic or not,
sources, stresses, DSV output, accuracies that need the seventh attempt and
rejected steps, and one that fails every solve."""
import dataclasses

import numpy as np
import pytest

from gemini_unified_b200 import configs, model as M

pytestmark = pytest.mark.gpu
G = configs.GLOBAL_SMALL
R = configs.REGIONAL_SMALL
COUNTS = ("steps_ok", "steps_rej", "attempts", "sysmats", "matvecs", "flops")

CASES = {
    "lowest_frequency": (G, True, dict(), 2, 2),
    "one_frequency": (G, True, dict(), 30, 30),
    "several": (G, True, dict(), 40, 46),
    "anisotropic_stress": (G, False, dict(source_type="FORCE", stressflag=True), 20, 21),
    "tight_accuracy": (G, True, dict(eps=1.0e-8), 12, 12),
    "loose_accuracy": (G, True, dict(eps=1.0e-2), 25, 26),
    "failing": (G, True, dict(eps=1.0e-30), 4, 4),
    "regional": (R, True, dict(), 20, 24),
    "regional_stress": (R, True, dict(stressflag=True), 60, 60),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_group_form_equals_thread_form(gpu, name):
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, GeminiFK
    w, iso, kw, lo, hi = CASES[name]
    m = w.model() if iso else configs.prem(isotropic=False)
    ex = w.nodes(m)
    jre = ex.node_index(w.rec_radius)
    p = dataclasses.replace(w.params, **kw)
    fk = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST)
    got = fk.run(p, jre, lo, hi, raise_on_failure=False)
    cg = fk.stats()
    fk.instrument(True)
    ref = fk.run(p, jre, lo, hi, raise_on_failure=False)
    cr = fk.stats()
    fk.instrument(False)
    for a, b in zip(got, ref):
        np.testing.assert_array_equal(a, b)
    assert [cg[k] for k in COUNTS] == [cr[k] for k in COUNTS]
    assert (name == "failing") == bool(np.any(got[3] != 0))


@pytest.mark.parametrize("source", ["MOMENT", "FORCE"])
def test_group_form_of_dsv_and_set_runs(gpu, source):
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, GeminiFK
    w = dataclasses.replace(G, nnod_blocks=[4], dr_blocks=[10000.0])
    m = w.model()
    ex = w.nodes(m)
    jre = ex.node_index(w.rec_radius)
    p = dataclasses.replace(w.params, source_type=source)
    fk = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST)
    one = fk.run_dsv(p, 2, 15, 16)
    many = fk.aski_spectra(p, [1, 3, jre], jre, 15, 16)
    fk.instrument(True)
    for a, b in zip(one, fk.run_dsv(p, 2, 15, 16)):
        np.testing.assert_array_equal(a, b)
    for x, y in zip(many, fk.aski_spectra(p, [1, 3, jre], jre, 15, 16)):
        for a, b in zip(x, y):
            np.testing.assert_array_equal(a, b)
    fk.instrument(False)


def test_autotuner_times_the_thread_form(gpu):
    """The settings that the autotuner chooses are the thread form's: on a slab that runs in the
    group form (96 solves, about three times faster) it times the thread form all the same."""
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, NSCHED, GeminiFK
    m = G.model()
    ex = G.nodes(m)
    jre = ex.node_index(G.rec_radius)
    fk = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST)
    ms = fk.autotune(G.params, jre, 8, 8, repeats=3)["ms"]
    group = []
    for _ in range(5):
        fk.run(G.params, jre, 8, 8)
        group.append(fk.stats()["phase_ms"][1])
    assert ms[:NSCHED, 1].min() > 1.5 * min(group)


def test_settings_of_the_thread_form_give_identical_spectra(gpu):
    """Every schedule, deferral and granularity of the form of one lane per solve, which a run
    with instruments takes at every size, against the group form: bit for bit."""
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, NDEFER, NGRAN, NSCHED, GeminiFK
    m = G.model()
    ex = G.nodes(m)
    jre = ex.node_index(G.rec_radius)
    fk = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST)
    ref = fk.run(G.params, jre, 40, 52, f32=False)[2]
    fk.instrument(True)
    for put, n in ((fk.schedule_set, NSCHED), (fk.defer_set, NDEFER), (fk.queue_set, NGRAN)):
        for i in range(n):
            put([i, i, i])
            got = fk.run(G.params, jre, 40, 52, f32=False)[2]
            assert int(fk.instrument_read()[0][3]) > 0   # lane attempts, which the thread form counts
            np.testing.assert_array_equal(got, ref)
    fk.instrument(False)


@pytest.mark.parametrize("srcs", [(-1, 1), (5, 3, -1, 1)])
def test_granularities_of_a_set_run_in_the_thread_form(gpu, srcs):
    """Runs of queue positions that cross from one source to the next, with one lane per solve."""
    from gemini_unified_b200.fk import GEM_BACKEND_GPU_FAST, NGRAN, GeminiFK
    w = dataclasses.replace(G, nnod_blocks=[4], dr_blocks=[10000.0])
    m = w.model()
    ex = w.nodes(m)
    jre = ex.node_index(w.rec_radius)
    fk = GeminiFK(m, ex, backend=GEM_BACKEND_GPU_FAST)
    js = [jre if j < 0 else j for j in srcs]
    ref = fk.aski_spectra(w.params, js, jre, 3, 6, f32=False)
    fk.instrument(True)
    for q in range(NGRAN):
        fk.queue_set([q, q, q])
        for a, b in zip(fk.aski_spectra(w.params, js, jre, 3, 6, f32=False), ref):
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x, y)
    fk.instrument(False)
