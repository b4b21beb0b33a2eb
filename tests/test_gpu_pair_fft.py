"""GPU checks of the packed power-of-two kernels (fft_pair.cuh).

They run the plans of the scalar kernels with two butterflies per thread, so
every output is compared bit for bit with the scalar kernels, which a context
tuned to 32 points per thread still runs (spx_set_fft_tuning): lengths that
fill the transform, fall one short (odd: 8-byte loads), end inside it, and
samples that start off a 16-byte boundary.
"""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1024, 2048, 4096, 8192, 16384, 32768, 49152, 98304, 131072, 147456, 196608, 262144]
MODES = ("complex", "mag", "mag2", "magphase")


def _samples(beams, n, offset, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f = torch.randn(beams * n + offset, 2, generator=g, device="cuda")
    return torch.view_as_complex(f)[offset:].reshape(beams, n)


@pytest.fixture(scope="module")
def scalar(spx):
    """A context whose power-of-two transforms run the scalar kernels."""
    from spectrum_gb300._capi import lib
    c = spx.Context(0)
    for nfft in SIZES:
        c.check(lib.spx_set_fft_tuning(c.h, nfft, 32, 0))
    return c


def _same(a, b):
    import torch
    return torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("nfft", SIZES)
def test_outputs_equal_the_scalar_kernels(spx, scalar, nfft):
    for n, offset, window in ((nfft, 0, spx.WINDOW_HANN), (nfft - 1, 0, spx.WINDOW_BLACKMAN),
                              (nfft // 2 + 2, 0, spx.WINDOW_NONE), (nfft - 2, 1, spx.WINDOW_HAMMING), (1, 1, 0)):
        x = _samples(5, n, offset, nfft + n)
        for out in MODES:
            a, b = (spx.fft(x, nfft, window, out, 0.25, ctx=c) for c in (None, scalar))
            assert _same(a, b), (nfft, n, offset, out)


@pytest.mark.parametrize("nfft", SIZES)
def test_inverse_and_unaligned_output_equal_the_scalar_kernels(spx, scalar, nfft):
    import torch
    x = _samples(3, nfft, 0, nfft)
    ref = spx.ifft(x, ctx=scalar)
    assert _same(spx.ifft(x), ref)
    y = torch.empty(3 * nfft + 1, dtype=torch.complex64, device="cuda")[1:].reshape(3, nfft)
    assert _same(spx.ifft(x, out=y), ref)
    z = x.clone()
    spx.ifft(z, out=z)
    assert _same(z, ref)
    half, full = (spx.fft_r2c(x.real.contiguous(), nfft, spx.WINDOW_HANN, f) for f in (False, True))
    assert _same(half, spx.fft_r2c(x.real.contiguous(), nfft, spx.WINDOW_HANN, False, ctx=scalar))
    assert _same(full, spx.fft_r2c(x.real.contiguous(), nfft, spx.WINDOW_HANN, True, ctx=scalar))


@pytest.mark.parametrize("nfft", [1 << 19, 1 << 20, 1 << 21])
def test_big_transform_modes_agree(spx, nfft):
    """The output modes of the 2^19 .. 2^21-point transforms (different ways out
    of the row kernel) hold the same spectrum bit for bit, and it is the
    library FFT's within FP32 rounding; odd lengths take 8-byte loads."""
    import torch
    for n, offset in ((nfft, 0), (nfft // 2 + 1, 1)):
        x = _samples(2, n, offset, nfft + n)
        z = spx.fft(x, nfft, spx.WINDOW_HANN)
        w = torch.sin(torch.pi * torch.arange(n, device="cuda", dtype=torch.float64) / (n - 1)) ** 2
        ref = torch.fft.fft(x.to(torch.complex128) * w, n=nfft)
        assert ((z - ref).abs().max() / ref.abs().max()).item() < 1e-6  # ~ log2(N) roundings of 6e-8
        m2 = spx.magnitude(z, 1.0, squared=True)
        assert _same(spx.fft(x, nfft, spx.WINDOW_HANN, "mag2"), m2)
        assert _same(spx.fft(x, nfft, spx.WINDOW_HANN, "mag"), spx.magnitude(z))
        assert _same(spx.fft(x, nfft, spx.WINDOW_HANN, "magphase"), spx.mag_phase(z))


@pytest.mark.parametrize("nfft", [32768, 49152, 65536, 131072, 262144])
def test_maxima_of_row_spectra_equal_the_composed_search(spx, nfft):
    """All maxima from the row layout of the two-launch transforms against the
    transform in bin order and the search on it: windows that start and end
    inside a column, cover one column, the whole spectrum or nothing."""
    import torch
    cb = nfft // 1024  # bins per column
    x = _samples(3, nfft // 2 + 3, 0, nfft)
    spec = spx.fft(x, nfft, spx.WINDOW_HANN)
    for start, end in ((0, 0), (1, nfft), (cb - 1, cb + 1), (cb, 2 * cb), (5 * cb + 3, nfft // 2 + cb // 2 + 1),
                       (nfft - 3, nfft), (cb + 1, cb + 2), (7, 7)):
        for sigma in (0.0, 3.0):
            kw = dict(search_start=start, search_end=end, max_per_beam=2000, refine=spx.REFINE_PARABOLIC,
                      thresh_sigma=sigma, sample_rate=1e6)
            out, counts = spx.fft_peaks(x, nfft, spx.WINDOW_HANN, spx.PEAK_ALL, **kw)
            ref, rc = spx.all_maxima(spec, **kw)
            assert torch.equal(counts, rc), (start, end, sigma)
            for b in range(3):
                n = min(int(rc[b]), ref.shape[1])
                assert torch.equal(out[b, :n], ref[b, :n]), (start, end, sigma, b)


@pytest.mark.parametrize("nfft", [5, 500, 1000, 2000, 3001, 5000, 10007, 20011, 50021, 100003])
def test_chirp_z_in_one_launch_equals_the_launches(spx, nfft):
    """Lengths with other prime factors: the one-launch chirp-z transform (m up
    to 16384) and the one with its products inside the m-point transforms (m up
    to 262144) against the five launches over the scalar kernels, which a
    context tuned for the m-point transform still runs."""
    import torch
    from spectrum_gb300._capi import lib
    general = spx.Context(0)
    m = spx.next_pow2(2 * nfft - 1)
    if m >= 1024:
        general.check(lib.spx_set_fft_tuning(general.h, m, 32, 0))
    for n, offset, window in ((nfft, 0, spx.WINDOW_NONE), (nfft - 1, 1, spx.WINDOW_HANN),
                              (nfft // 2 + 1, 0, spx.WINDOW_BLACKMAN), (1, 0, spx.WINDOW_NONE)):
        x = _samples(3, n, offset, nfft + n)
        for out in MODES:
            assert _same(spx.fft(x, nfft, window, out, 0.5), spx.fft(x, nfft, window, out, 0.5, ctx=general)), (n, out)
    x = _samples(3, nfft, 1, nfft)
    ref = spx.ifft(x, ctx=general)
    y = x.clone()
    spx.ifft(y, out=y)
    assert _same(y, ref)
    r = x.real.contiguous()
    for full in (False, True):
        assert _same(spx.fft_r2c(r, nfft, spx.WINDOW_HANN, full),
                     spx.fft_r2c(r, nfft, spx.WINDOW_HANN, full, ctx=general))


def _hard_beams(x):
    """Beams without a maximum, with ties, NaN, infinities and magnitudes whose squares leave FP32."""
    x[0] = 0
    x[1] = 1
    x[2, 0] = complex(float("nan"), 1.0)
    x[3, -1] = complex(float("inf"), 0.0)
    x[4] *= 1e25
    x[5] *= 1e-25
    x[6, x.shape[1] // 2:] = x[6, :x.shape[1] - x.shape[1] // 2].clone()
    return x


@pytest.mark.parametrize("nfft", [1024, 2048, 4096, 8192, 16384])
def test_topk_equals_the_scalar_kernels(spx, scalar, nfft):
    import torch
    for n, offset, k, lo, hi in ((nfft, 0, 1, 0, 0), (nfft - 1, 0, 8, 1, nfft), (nfft, 1, 32, 2, nfft - 1),
                                 (nfft // 2, 0, 7, nfft // 2 - 33, nfft // 2 + 33), (nfft, 0, 9, 5, 6), (3, 0, 32, 0, 0),
                                 (nfft, 0, 4, nfft - 2, nfft - 1), (nfft, 0, 4, 9, 9)):
        x = _hard_beams(_samples(9, n, offset, nfft + n + k))
        a, b = (spx.fft_peaks(x, nfft, spx.WINDOW_HANN, spx.PEAK_TOPK, 1e6, lo, hi, max_per_beam=k, refine=1, ctx=c)
                for c in (None, scalar))
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]), (nfft, n, k, lo, hi)


@pytest.mark.parametrize("nfft", [1024, 2048, 4096, 8192, 16384])
def test_one_and_two_peaks_equal_the_scalar_kernels(spx, scalar, nfft):
    import torch
    for n, offset, rng in ((nfft, 0, 0), (nfft - 1, 0, nfft), (nfft // 2, 1, 2), (5, 0, 77), (nfft, 0, nfft - 1)):
        x = _hard_beams(_samples(9, n, offset, nfft + n + rng))
        for mode in (spx.PEAK_ONE, spx.PEAK_TWO):
            a, b = (spx.fft_peaks(x, nfft, spx.WINDOW_BLACKMAN, mode, 1e6, search_range=rng, ctx=c)[0]
                    for c in (None, scalar))
            assert torch.equal(a, b), (nfft, n, rng, mode)
    for rng in (1, nfft + 1):
        for c in (None, scalar):
            with pytest.raises(Exception, match="search_range must be in"):
                spx.fft_peaks(x, nfft, 0, spx.PEAK_TWO, 1e6, search_range=rng, ctx=c)


@pytest.mark.parametrize("nfft,beams,k", [(1024, 2050, 3), (2048, 1030, 32), (4096, 520, 1), (8192, 300, 8), (16384, 130, 2)])
def test_learned_topk_equals_its_three_steps(spx, nfft, beams, k):
    import torch
    from spectrum_gb300.learned import MLPRefiner
    net = MLPRefiner(seed=5)
    x = _hard_beams(_samples(beams, nfft, 0, nfft))
    out, counts, amp, used = net.fft_peaks(x, nfft, spx.WINDOW_HANN, k, 1e6, search_start=1, search_end=nfft)
    spec = spx.fft(x, nfft, spx.WINDOW_HANN)
    ref, n = spx.topk(spec, k, sample_rate=1e6, search_start=1, search_end=nfft, refine=1)
    ramp, rused = net.refine(spec, ref, n, nfft, 1e6)
    for a, b in ((out, ref), (counts, n), (amp.view(torch.int32), ramp.view(torch.int32)), (used, rused)):
        assert torch.equal(a, b)


TWIN_SIZES = [n for n in (2 ** a * 3 ** b for a in range(13) for b in range(1, 9)) if 1024 < n < 16384]


@pytest.mark.parametrize("nfft", sorted(TWIN_SIZES))
def test_two_beams_per_cta_equal_the_scalar_kernels(spx, nfft):
    import torch
    from spectrum_gb300._capi import lib
    other = spx.Context(0)
    other.check(lib.spx_set_fft_tuning(other.h, nfft, 32, 0))
    for beams, n, offset, window in ((1, nfft, 0, spx.WINDOW_HANN), (2, nfft - 1, 1, spx.WINDOW_BLACKMAN),
                                     (5, nfft // 2 + 1, 0, spx.WINDOW_NONE), (4, 1, 1, 0)):
        x = _samples(beams, n, offset, nfft + n)
        x[beams - 1, 0] = complex(float("inf"), 0.0)  # (stays in its beam)
        for out in MODES:
            a, b = (spx.fft(x, nfft, window, out, 0.25, ctx=c) for c in (None, other))
            assert _same(a, b), (nfft, beams, n, out)
    x = _samples(3, nfft, 0, nfft)
    ref = spx.ifft(x, ctx=other)
    assert _same(spx.ifft(x), ref)
    y = torch.empty(3 * nfft + 1, dtype=torch.complex64, device="cuda")[1:].reshape(3, nfft)
    assert _same(spx.ifft(x, out=y), ref)
    z = x.clone()
    spx.ifft(z, out=z)
    assert _same(z, ref)
    r = x.real.contiguous()
    for full in (False, True):
        assert _same(spx.fft_r2c(r, nfft, 1, full), spx.fft_r2c(r, nfft, 1, full, ctx=other))
