"""The mixture fit with several rounds of pairs per warp: more pairs than warps on the chip, rows of a few hundred to
more than a warp's 896 entries, full, sparse and empty, so that pairs open the next round, wait behind an over-long
one, or are gathered and dropped for lack of room.  Every row is written (the output starts as a sentinel), each as
the FP64 restatement gives it, and as the same row gives alone; tolerances as in test_gpu_mixture_fit.py."""
import numpy as np
import pytest

import photonprop_b200 as pp
from test_gpu_mixture_fit import _em

pytestmark = pytest.mark.gpu
SENTINEL = -12345.0


def _fit(hist, shift, t0, bw, iters):
    import torch
    d = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (hist, shift)]
    o = torch.full((len(hist), 5), SENTINEL, dtype=torch.float32, device="cuda")
    pp._lib.check(pp._lib.load().pp_gamma_mixture_fit(d[0].data_ptr(), len(hist), hist.shape[1], t0, bw,
                                                      d[1].data_ptr(), o.data_ptr(), iters, None))
    return o.cpu().numpy()


def _unlabelled(rows):
    """Where the two shapes have met (rows of one filled bin), either may be called the first: the larger weight."""
    r = np.array(rows, dtype=np.float64)
    met = np.abs(r[..., 1] - r[..., 2]) <= 1e-5 * r[..., 2]
    r[..., 0] = np.where(met, np.maximum(r[..., 0], 1 - r[..., 0]), r[..., 0])
    return r


@pytest.mark.parametrize("n,bins,iters", [(5000, 400, 4), (7500, 1200, 3), (40_000, 90, 2)])
@pytest.mark.parametrize("order", ["mixed", "long-first"])
def test_many_rounds(n, bins, iters, order):
    rng = np.random.default_rng(n + bins)
    t0, bw = 0.0, 1.0
    centre = t0 + (np.arange(bins) + 0.5) * bw
    shift = rng.uniform(-5.0, 0.1 * bins, n).astype(np.float32)
    filled = rng.choice([0.0, 0.004, 0.1, 0.3, 0.7, 1.0], n, p=[0.1, 0.1, 0.2, 0.2, 0.2, 0.2])
    if order == "long-first":
        filled = np.sort(filled)[::-1]
    hist = np.where(rng.random((n, bins)) < filled[:, None], rng.uniform(0.2, 3.0, (n, bins)), 0.0)
    hist *= np.exp(-centre / (0.3 * bins))
    got = _fit(hist, shift, t0, bw, iters)
    assert not (got == SENTINEL).any()
    light = (hist * (centre[None, :] > shift[:, None].astype(np.float64))).sum(1) > 0
    np.testing.assert_array_equal(np.isnan(got).any(1), ~light)
    for i in rng.integers(0, n, 150):
        want = _em(hist[i], centre - np.float64(shift[i]), iters)
        np.testing.assert_allclose(_unlabelled(got[i]), _unlabelled(want), rtol=2e-5, atol=1e-6, err_msg=str(i))
    few = rng.integers(0, n, 60)  # the same rows in other company: one or two to a block, and in another order
    np.testing.assert_allclose(_unlabelled(_fit(hist[few], shift[few], t0, bw, iters)), _unlabelled(got[few]), rtol=2e-5,
                               atol=1e-6)
