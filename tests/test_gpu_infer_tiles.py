"""Surrogate queries at the edges of the tile order: rounds of the grid's groups, what is left of a round, one row.
Every row is a computation of its own, so a batch's answers are those of the same rows asked 100 at a time, bit for
bit; against the oracle the forward is held by the surrogate's own tests."""
import numpy as np
import pytest

from photonprop_b200 import surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rounds,more", [(0, 1), (0, 127), (0, 129), (0, 3001), (1, -128), (1, -1), (1, 0), (1, 1),
                                         (1, 148 * 128 + 5), (3, 130)])
def test_rows_do_not_depend_on_the_batch(rounds, more):
    import torch
    n = rounds * torch.cuda.get_device_properties(0).multi_processor_count * 4 * 128 + more
    net = surrogate.MLP(0, 3)
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(size=(n, 4)).astype(np.float32)).cuda()
    out = torch.full((5, n), float("nan"), device="cuda")
    net.forward(x, out, n, physical=False)
    torch.cuda.synchronize()
    assert bool(torch.isfinite(out).all())
    for at in sorted({0, max(0, n - 100), *rng.integers(0, n, 6).tolist()}):
        k = min(100, n - at)
        part = torch.empty((5, k), device="cuda")
        net.forward(x[at:at + k].contiguous(), part, k, physical=False)
        torch.cuda.synchronize()
        assert torch.equal(part, out[:, at:at + k])
