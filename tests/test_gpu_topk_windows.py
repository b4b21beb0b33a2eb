"""GPU check of spx_topk where only some warps of a beam have bins to look at: search
windows around the 256 bins of a warp's step, empty ones among them, against the
oracle (indices, order and counts)."""
import numpy as np
import pytest

from oracle import spectrum_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 4, 5, 32])
@pytest.mark.parametrize("bins", [0, 1, 2, 31, 255, 256, 257, 511, 513, 1023, 1025, 1793, 2047, 3000])
def test_short_windows(spx, cuda, k, bins):
    import torch
    rng = np.random.default_rng(100 * bins + k)
    nfft, start = 4096, 7
    s = (rng.standard_normal((6, nfft)) + 1j * rng.standard_normal((6, nfft))).astype(np.complex64)
    s[4] = 1.0  # no maxima
    s[5, 1::2] *= 0.0  # one at every other bin
    out, counts = spx.topk(torch.from_numpy(s).to(cuda), k, sample_rate=1e6, search_start=start, search_end=start + bins)
    ref, rc = orc.topk(None, s, nfft, 1e6, k, start, start + bins)
    assert np.array_equal(counts.cpu().numpy(), rc)
    got = spx.maxvalues_to_numpy(out)
    for b in range(len(s)):
        assert np.array_equal(got[b, :rc[b]]["index"], ref[b, :rc[b]]["index"]), b
        assert np.array_equal(got[b, :rc[b]]["magnitude"], ref[b, :rc[b]]["magnitude"]), b
