"""GPU check of all maxima of C x 16384 points with C = 3, 6, 9, 12 where device memory
is short: these sizes use two buffers of a spectrum each; with room for little more
than one, the call still gives the lists that it gives with room for both."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft,beams", [(49152, 2001), (196608, 500)])
def test_room_for_one_spectrum_is_enough(spx, cuda, nfft, beams):
    import torch
    n = 1001
    g = torch.Generator(device="cuda")
    g.manual_seed(nfft + beams)
    x = torch.view_as_complex(torch.randn(beams, n, 2, generator=g, device="cuda"))

    def search(ctx):
        return spx.fft_peaks(x, nfft, spx.WINDOW_HANN, spx.PEAK_ALL, sample_rate=1e6, max_per_beam=40, thresh_sigma=1.0,
                             refine=spx.REFINE_PARABOLIC, ctx=ctx)

    roomy, tight = spx.Context(0), spx.Context(0)
    out, counts = search(roomy)
    assert int(counts.min()) > 0
    roomy.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spectrum = beams * nfft * 8
    # buffers are a quarter larger than asked for: one of 1.25 spectra fits, a second one does not
    rest = torch.empty(torch.cuda.mem_get_info()[0] - spectrum * 7 // 4, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            o, c = search(tight)
            torch.cuda.synchronize()
            assert torch.equal(c, counts) and torch.equal(o, out)
    finally:
        del rest
        torch.cuda.empty_cache()
    o, c = search(tight)
    assert torch.equal(c, counts) and torch.equal(o, out)
