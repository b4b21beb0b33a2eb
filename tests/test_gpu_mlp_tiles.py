"""GPU checks of the tiled training kernels (mlp_tile_kernel, mlp_reduce_kernel):
row counts around a tile (32) and around the most CTAs a pass uses (304 tiles),
where a CTA takes several tiles, against the FP64 oracle; the same bits twice."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 304 * 32 - 1, 304 * 32 + 1, 20000])
def test_loss_and_gradients_match_the_oracle(spx, cuda, rows):
    import torch
    from spectrum_gb300.learned import MLPRefiner
    r = MLPRefiner(seed=5)
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, 10)).astype(np.float32)
    t = (0.3 * rng.standard_normal((rows, 2))).astype(np.float32)
    m = (rng.uniform(size=rows) > 0.2).astype(np.int32)
    xd, td, md = (torch.from_numpy(v).to(cuda) for v in (x, t, m))
    g, loss = r.gradients(xd, td, md)
    lref, gref = mo.loss_and_grad(r.params, x, t, m)
    # sums of `rows` FP32 products: rounding grows with sqrt(rows), at most
    # ~150 * 6e-8 of the gradient's norm
    assert np.linalg.norm(g.cpu().numpy() - gref) <= 1e-5 * np.linalg.norm(gref) + 1e-12
    assert abs(float(loss) - lref) <= 1e-5 * abs(lref) + 1e-12
    g2, loss2 = r.gradients(xd, td, md)
    assert torch.equal(g, g2) and torch.equal(loss, loss2)
    y, _ = mo.forward(r.params, x)
    assert np.abs(r.forward(xd).cpu().numpy() - y).max() <= 2e-5 * np.abs(y).max()
