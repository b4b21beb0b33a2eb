"""GPU check of the batch launches of batch_rows.cuh: every C x M they take
(C in {2, 3, 4, 6, 8, 9}, the seven local sizes), full, odd and short sample
counts, every window and search windows with odd edges, against spx_fft_peaks
on each beam alone, bit for bit.  The batch is large enough to take them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOCAL = (16384, 15552, 13824, 13122, 12288, 11664, 6561)


def _beams():
    n_points, nffts = [], []
    for m in LOCAL:
        for c in (2, 3, 4, 6, 8, 9):
            nfft = c * m
            if not 16384 < nfft <= 147456:
                continue
            for n in (nfft, nfft - nfft // 7 - (nfft // 7) % 2 - 1):
                n_points.append(n)
                nffts.append(nfft)
    n_points += [1000, 5001, 16384, 30000]  # beams of the cluster kernel among them
    nffts += [1024, 5184, 16384, 2 * 17496]
    return np.array(n_points), np.array(nffts)


@pytest.mark.parametrize("window,k,start,end", [(0, 3, 0, 0), (1, 8, 0, 0), (2, 32, 77, 0), (3, 1, 5000, 5301),
                                                (4, 5, 1, 1 << 30)])
def test_every_size_equals_the_beam_alone(spx, cuda, window, k, start, end):
    import torch
    from spectrum_gb300.batch import Batch
    n_points, nffts = _beams()
    assert nffts[nffts > 16384].sum() >= 1 << 22
    g = torch.Generator(device="cuda")
    g.manual_seed(window + 1)
    x = torch.view_as_complex(torch.randn(int(n_points.sum()), 2, generator=g, device="cuda"))
    b = Batch(n_points, nffts, window=window, k=k, sample_rate=1e6, search_start=start, search_end=end)
    out, counts = (t.clone() for t in b.run(x))
    pos = 0
    for i, (n, nfft) in enumerate(zip(n_points, nffts)):
        e = min(end, int(nfft) - 1) if end else 0
        o, c = spx.fft_peaks(x[pos:pos + n].reshape(1, -1).contiguous(), int(nfft), window, spx.PEAK_TOPK,
                             sample_rate=1e6, max_per_beam=k, refine=spx.REFINE_PARABOLIC, search_start=start,
                             search_end=e)
        pos += n
        m = int(c[0])
        assert int(counts[i]) == m, (i, n, nfft)
        assert torch.equal(out[i, :m], o[0, :m]), (i, n, nfft)
