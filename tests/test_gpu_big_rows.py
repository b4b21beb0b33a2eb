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
