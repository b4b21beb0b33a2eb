"""GPU check of 2^19- and 2^20-point transforms at the two ways of reading the scratch
between their launches (up to 64 MB of it, and beyond): the bits of each beam alone."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft,beams", [(1 << 19, 16), (1 << 19, 17), (1 << 20, 8), (1 << 20, 9)])
@pytest.mark.parametrize("mode", ["complex", "mag", "magphase"])
def test_every_beam_equals_the_beam_alone(spx, cuda, nfft, beams, mode):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(nfft + beams)
    x = torch.view_as_complex(torch.randn(beams, nfft, 2, generator=g, device="cuda"))
    all_ = spx.fft(x, nfft, spx.WINDOW_HANN, mode)
    for b in range(beams):
        assert torch.equal(all_[b].view(torch.int32), spx.fft(x[b:b + 1], nfft, spx.WINDOW_HANN, mode)[0].view(torch.int32))


@pytest.mark.parametrize("nfft,beams", [(1 << 19, 1), (1 << 19, 3), (1 << 20, 2)])
def test_inverse_and_real_input_equal_the_complex_spectrum(spx, cuda, nfft, beams):
    """Their outputs come from the bits of spx_fft: reversed and scaled by a power of
    two, and the half of a real beam's spectrum (with its mirror)."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(nfft + beams)
    x = torch.view_as_complex(torch.randn(beams, nfft, 2, generator=g, device="cuda"))
    y = torch.view_as_real(spx.ifft(x))
    f = torch.view_as_real(spx.fft(x, nfft)).roll(-1, 1).flip(1) * (1.0 / nfft)
    assert torch.equal(y, f)
    r = x.real.contiguous()
    half, full = (torch.view_as_real(spx.fft_r2c(r, nfft, spx.WINDOW_HANN, m)) for m in (False, True))
    c = torch.view_as_real(spx.fft(torch.complex(r, torch.zeros_like(r)), nfft, spx.WINDOW_HANN))
    n = nfft // 2 + 1
    assert torch.equal(half, c[:, :n]) and torch.equal(full[:, :n], c[:, :n])
    mirror = c[:, 1:nfft // 2].flip(1)
    assert torch.equal(full[:, n:, 0], mirror[..., 0]) and torch.equal(full[:, n:, 1], -mirror[..., 1])
