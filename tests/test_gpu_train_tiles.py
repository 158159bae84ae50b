"""The training kernel at the edges of its 128-row tiles: loss, every parameter block's gradient and the Adam step
against the FP64 oracle that rounds to BF16 where the kernel does (the 2e-2 relative bound of test_gpu_surrogate.py),
and rows that the mask leaves out."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,keep", [(1, 1.0), (127, 0.8), (128, 1.0), (129, 0.5), (4097, 0.7)])
def test_step_at_tile_edges(n, keep):
    import torch
    from photonprop_b200 import surrogate as sg
    net = sg.MLP(0, 5)
    p = net.get_params().astype(np.float64)
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 4)).astype(np.float32)
    yt = rng.normal(size=(n, 5)).astype(np.float32)
    mask = (rng.uniform(0.1, 1.0, size=(n, 5)) * (rng.uniform(size=(n, 5)) < keep)).astype(np.float32)
    mask[0, 0] = 1.0
    d = [torch.from_numpy(a).cuda() for a in (x, yt, mask)]
    loss, g = net.train_step(*d, n, 0.0, want_grads=True)
    ref_loss, ref_g = omlp.loss_and_grads(p, x.astype(np.float64), yt.astype(np.float64), mask.astype(np.float64))
    assert loss == pytest.approx(ref_loss, rel=1e-2)
    off = 0
    for name, shape in omlp.SIZES:
        k = int(np.prod(shape))
        err = np.linalg.norm(g[off:off + k] - ref_g[off:off + k]) / max(np.linalg.norm(ref_g[off:off + k]), 1e-12)
        assert err < 2e-2, (name, err)
        off += k
    np.testing.assert_array_equal(net.get_params(), p.astype(np.float32))  # lr = 0 moves nothing
    loss2, _ = net.train_step(*d, n, 1e-3)  # the gradients do not carry over from the step before
    assert loss2 == pytest.approx(loss, rel=1e-6)
    step = net.get_params().astype(np.float64) - p
    big = np.abs(g) > 1e-4 * np.abs(g).max()
    np.testing.assert_allclose(step[big], -1e-3 * np.sign(g[big]), rtol=2e-2)  # Adam's first step is lr sign(g)
    # the tensor-core copies follow the masters: inference answers like a network made from them
    other = sg.MLP(0, 6)
    other.set_params(net.get_params())
    q = torch.from_numpy(rng.normal(size=(200, 4)).astype(np.float32)).cuda()
    a, b = torch.zeros((5, 200), device="cuda"), torch.zeros((5, 200), device="cuda")
    net.forward(q, a, 200)
    other.forward(q, b, 200)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    net.close()
    other.close()


def test_empty_mask_moves_nothing():
    import torch
    from photonprop_b200 import surrogate as sg
    net = sg.MLP(0, 5)
    z = torch.zeros((200, 5), device="cuda")
    loss, g = net.train_step(torch.ones((200, 4), device="cuda"), z + 1.0, z, 200, 0.0, want_grads=True)
    assert loss == 0.0 and not np.any(g)
    net.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 3001, 148 * 128, 148 * 128 + 1, 80_000])
def test_a_query_is_answered_alike_in_any_batch(n):
    """Tiles over blocks and groups: the rows of a batch of n are those of a batch of 100,001, bit for bit."""
    import torch
    from photonprop_b200 import surrogate as sg
    net = sg.MLP(0, 8)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((100_001, 4), generator=g, device="cuda")
    a, b = torch.zeros((5, 100_001), device="cuda"), torch.full((5, n), 7.0, device="cuda")
    net.forward(x, a, 100_001)
    net.forward(x[:n].contiguous(), b, n)
    torch.cuda.synchronize()
    assert torch.equal(a[:, :n], b)
    want, _ = omlp.forward(net.get_params().astype(np.float64), x[-5:].cpu().numpy().astype(np.float64))
    np.testing.assert_allclose(a[:, -5:].cpu().numpy().T, want, rtol=2e-2, atol=2e-2)
    net.close()
