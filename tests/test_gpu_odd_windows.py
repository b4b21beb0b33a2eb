"""GPU check of windowed beams of odd length and off a 16-byte boundary in the packed
kernels: the pair of samples that straddles the end of a beam takes nothing from
what follows it, neither in the samples (infinities behind the beam) nor in the
window's table, and every start gives the bits of a beam alone on a boundary."""
import pytest

pytestmark = pytest.mark.gpu

# one launch, two launches (powers of two and C = 3), 2^19 .. 2^21, chirp-z in one launch and in four
SIZES = [1024, 4096, 8192, 16384, 32768, 49152, 262144, 1 << 19, 1 << 20, 1 << 21, 1000, 5000, 100003]


@pytest.mark.parametrize("nfft", SIZES)
@pytest.mark.parametrize("window", [1, 4])
def test_the_pair_at_the_end_stays_inside_the_beam(spx, cuda, nfft, window):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(nfft + window)
    for n in {1, 3, nfft // 2 | 1, nfft - 1 - nfft % 2}:
        one = torch.view_as_complex(torch.randn(n, 2, generator=g, device="cuda"))
        buf = torch.full((4 * n + 2,), complex(float("inf"), float("nan")), dtype=torch.complex64, device="cuda")
        ref = torch.view_as_real(spx.fft(one.reshape(1, n), nfft, window))
        assert bool(torch.isfinite(ref).all())
        for start in (0, 1):  # beams 0 and 2 of three: 16-byte boundaries or 8 bytes off, the others infinite
            x = buf[start:start + 3 * n].view(3, n)
            x[0], x[2] = one, one
            got = torch.view_as_real(spx.fft(x, nfft, window))
            for b in (0, 2):
                assert torch.equal(got[b].view(torch.int32), ref[0].view(torch.int32)), (n, start, b)
            x[0], x[2] = buf[-1], buf[-1]
