"""GPU check that the gradients' FP32 additions run in chains of at most 512 rows at
every minibatch: one row carries 2^25 times the gradient of each other, so that a
chain loses the rows behind it, and what is lost shows how long it was."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [512, 304 * 512, 304 * 512 + 33, 1 << 20])
def test_what_one_large_row_hides(spx, cuda, rows):
    import torch
    from spectrum_gb300.learned import LAYOUT, MLPRefiner
    r = MLPRefiner(seed=0)
    p = np.concatenate([np.full(int(np.prod(shape)), {"W1": 0.125, "W2": 0.03125, "W3": 0.0625}.get(name, 0.25), np.float32)
                        for name, shape, _ in LAYOUT])  # all positive: no cancellation
    r.set_params(p)
    x = np.full((1, 10), 0.5, np.float32)
    y0 = r.forward(torch.from_numpy(x).to(cuda)).cpu().numpy()[0]
    t = np.tile(y0 - np.float32(2.0 ** -7), (2, 1)).astype(np.float32)
    t[0] = y0 - np.float32(2.0 ** 18)
    xd = torch.from_numpy(x).to(cuda).expand(rows, 10).contiguous()
    td = torch.from_numpy(t[1:]).to(cuda).expand(rows, 2).contiguous()
    td[0] = torch.from_numpy(t[0]).to(cuda)
    g, _ = r.gradients(xd, td, None)
    # rows 0 and 1 alone by the oracle, in its own normalisation (2 rows)
    (_, g0), (_, g1) = (mo.loss_and_grad(p, np.repeat(x, 2, 0), np.stack([t[i], t[i]]), np.ones(2, np.int32))
                        for i in (0, 1))
    ref = (g0 + (rows - 1) * g1) / rows  # each pair of equal rows is one row's gradient
    # a chain of 512 rows rounds 512 times and a row's gradient takes three inner
    # products of up to 64 terms: (512 + 200) x 2^-24 of the sum; 3449 rows behind
    # the large one would lose 3449 x 2^-25 of it, more than twice as much
    assert np.all(np.abs(g.cpu().numpy() - ref) <= 712 * 2.0 ** -24 * np.abs(ref))
