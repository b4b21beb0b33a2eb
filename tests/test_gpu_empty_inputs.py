"""GPU check that searches of beams without samples stay refused, whatever the count of
beams (an empty shape with no beams either has nothing to search in)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(0, 0), (3, 0), (0,), (2, 3, 0)])
def test_no_samples_are_refused(spx, cuda, shape):
    import torch
    x = torch.empty(shape, dtype=torch.complex64, device=cuda)
    for mode in (spx.PEAK_ONE, spx.PEAK_TWO, spx.PEAK_ALL, spx.PEAK_TOPK):
        with pytest.raises(RuntimeError):
            spx.fft_peaks(x, 1024, spx.WINDOW_HANN, mode, max_per_beam=3)


def test_no_beams_give_no_peaks(spx, cuda):
    import torch
    x = torch.empty((0, 1024), dtype=torch.complex64, device=cuda)
    out, counts = spx.fft_peaks(x, 1024, spx.WINDOW_HANN, spx.PEAK_TOPK, max_per_beam=3)
    assert out.shape == (0, 3, 8) and counts.shape == (0,)
