"""GPU check of batches whose local sizes change after creation, large enough for
the launches of batch_rows.cuh: a batch created at a local size of the cluster
kernel moves to each local size with rows of 6561 and 13122 points (first radix 9)
and back, through every call that rebuilds its tables, and runs as one launch set,
per size and as a captured graph.  Every list equals spx_fft_peaks on that beam at
the plan in force, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nfft,start,sizes", [(26244, 8748, (13122,)), (39366, 4374, (13122, 6561)),
                                              (52488, 8748, (6561, 13122))])
def test_local_sizes_changed_after_creation(spx, cuda, tmp_path, nfft, start, sizes):
    import torch
    from spectrum_gb300.batch import Batch
    beams = (1 << 22) // nfft + 3
    n = nfft - 1 - nfft % 2  # odd
    ctx = spx.Context(cuda.index or 0)
    g = torch.Generator(device="cuda")
    g.manual_seed(nfft)
    x = torch.view_as_complex(torch.randn(beams * n, 2, generator=g, device="cuda"))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        first = Batch([n], [nfft], window=1, k=5, sample_rate=1e6, ctx=ctx)
        first.set_local_size(nfft, start)  # plans belong to the context
        b = Batch([n] * beams, [nfft] * beams, window=1, k=5, sample_rate=1e6, ctx=ctx)
        assert b.local_size(nfft) == start
        b.run(x)

        def check(local):
            assert b.local_size(nfft) == local
            o, c = spx.fft_peaks(x.view(beams, n), nfft, 1, spx.PEAK_TOPK, sample_rate=1e6, max_per_beam=5,
                                 refine=spx.REFINE_PARABOLIC, ctx=ctx)
            assert int(c.min()) == 5

            def same(result):
                assert torch.equal(result[1], c) and torch.equal(result[0], o)
                b.out.zero_()
                b.counts.zero_()
            b.out.zero_()
            same(b.run(x))
            same(b.run_per_size(x))
            b.capture(x, stream=s)
            same(b.replay(stream=s))

        check(start)
        for i, local in enumerate(sizes):
            b.set_local_size(nfft, local)
            check(local)
            path = tmp_path / f"plans{i}"
            b.save_plans(path)
            b.set_local_size(nfft, start)
            check(start)
            assert b.load_plans(path) == 1
            check(local)
            b.set_cluster(9)
            check(local)
            b.set_cluster(0)
        b.autotune(x)
        check(b.local_size(nfft))
