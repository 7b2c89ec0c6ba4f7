"""Fast inverse FFT at the edges of its two first passes (bands below and above
1/16 of the transform), of one trace per CTA and many, and of its output paths
(8-byte stores, odd sample counts, unaligned series).  Reference: numpy's
transform and the exponential in FP64; bar: two roundings to float32, 2^-23 of
the largest sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ft(gpu):
    from gemini_unified_b200.fk import FrequencyTime, GEM_BACKEND_GPU_FAST
    return FrequencyTime(backend=GEM_BACKEND_GPU_FAST)


def _case(ns, nf2, ntr, sigma=0.001):
    rng = np.random.default_rng(nf2)
    nf1 = 2 + nf2 // 100
    x = rng.normal(size=(ntr, nf2)) + 1j * rng.normal(size=(ntr, nf2))
    x[:, :nf1 - 1] = 0
    full = np.zeros((ntr, ns // 2 + 1), complex)
    full[:, :nf2] = x
    return nf1, x, np.fft.irfft(full, n=ns, axis=1) * np.exp(sigma * np.arange(ns))


def _check(got, ref):
    assert np.all(np.abs(got.astype(np.float64) - ref).max(axis=1) <= 2.0 ** -23 * np.abs(ref).max(axis=1))


@pytest.mark.parametrize("ns", [512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("band", ["low", "edge", "above", "wide"])
def test_bands(ft, ns, band):
    nf2 = {"low": 7, "edge": ns // 16, "above": ns // 16 + 1, "wide": ns // 4 + 3}[band]
    nf1, x, ref = _case(ns, nf2, 37)
    _check(ft.run(nf1, nf2, 1.0 / ns, 0.001, x, ns, 1.0), ref)


@pytest.mark.parametrize("ns,nsamp", [(512, 511), (8192, 8191), (8192, 6000), (8192, 513), (8192, 400)])
def test_decimated_length(ft, ns, nsamp):
    """ndec = 1 with fewer samples than the transform gives."""
    nf2 = ns // 4 + 3   # ns follows from the band
    nf1, x, ref = _case(ns, nf2, 5)
    _check(ft.run(nf1, nf2, 1.0 / ns, 0.001, x, nsamp, 1.0), ref[:, :nsamp])


@pytest.mark.parametrize("ns", [512, 8192])
def test_many_traces_and_unaligned_series(ft, ns):
    import torch
    ntr, nf2 = 1201, ns // 16
    nf1, x, ref = _case(ns, nf2, ntr)
    d_x = torch.from_numpy(x).cuda()
    d_t = torch.zeros(ntr * ns + 1, dtype=torch.float32, device="cuda")
    ft.run_device(nf1, nf2, 1.0 / ns, 0.001, ntr, d_x.data_ptr(), nf2, ns, 1.0, d_t[1:].data_ptr())
    _check(d_t[1:].reshape(ntr, ns).cpu().numpy(), ref)
