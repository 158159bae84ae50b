"""The Gamma-mixture fit against an FP64 restatement of its EM (scipy's digamma), over histograms that are empty,
sparse, full and longer than a warp's part of shared memory, many pairs to a warp and one.  The results are FP32:
2e-5 relative (two dozen roundings of 6e-8, and the EM path's own 1e-9), 1e-6 for the log-likelihood's zero."""
import numpy as np
import pytest
from scipy import special

import photonprop_b200 as pp

pytestmark = pytest.mark.gpu


def _inv_digamma(y):
    a = np.exp(y) + 0.5 if y >= -2.22 else -1.0 / (y + 0.5772156649015329)
    for _ in range(8):
        a = max(a - (special.digamma(a) - y) / special.polygamma(1, a), 1e-3)
    return float(a)


def _em(h, t, iters):
    ok = (h > 0) & (t > 0)
    h, t = h[ok], t[ok]
    if not len(h):
        return np.full(5, np.nan)
    lt, s0 = np.log(t), h.sum()
    m = (h * t).sum() / s0
    v = max((h * t * t).sum() / s0 - m * m, 1e-6 * m * m + 1e-12)
    a0 = max(m * m / v, 0.05)
    w, a, th = 0.5, [max(0.5 * a0, 0.02), 2.0 * a0], v / m
    for _ in range(iters):
        p = [np.log(f) - x * np.log(th) - special.gammaln(x) + (x - 1) * lt - t / th for f, x in zip((w, 1 - w), a)]
        mx = np.maximum(*p)
        e = [np.exp(q - mx) for q in p]
        r = e[0] / (e[0] + e[1])
        ll = (h * (mx + np.log(e[0] + e[1]))).sum() / s0
        S = [[(h * q).sum(), (h * q * t).sum(), (h * q * lt).sum()] for q in (r, 1 - r)]
        w = min(max(S[0][0] / (S[0][0] + S[1][0]), 1e-4), 1 - 1e-4)
        for _ in range(3):
            th = (S[0][1] + S[1][1]) / (a[0] * S[0][0] + a[1] * S[1][0])
            a = [_inv_digamma(q[2] / q[0] - np.log(th)) if q[0] > 0 else x for q, x in zip(S, a)]
    if a[0] > a[1]:
        a, w = a[::-1], 1 - w
    return np.array([w, a[0], a[1], th, ll])


@pytest.mark.parametrize("n,bins,iters", [(1, 1000, 60), (3, 1, 5), (40, 33, 7), (700, 31, 3), (300, 200, 30),
                                          (5000, 50, 2), (2, 3000, 20)])
def test_matches_restatement(n, bins, iters):
    import torch
    rng = np.random.default_rng(bins + n)
    t0, bw = -3.0, 0.5
    centre = t0 + (np.arange(bins) + 0.5) * bw
    shift = rng.uniform(t0 - 5.0, t0 + 0.3 * bins * bw, n).astype(np.float32)
    shift[0] = -10.0
    hist = np.zeros((n, bins))
    for i in range(n):
        y = centre - np.float64(shift[i])
        f = np.where(y > 0, np.maximum(y, 0.1) ** rng.uniform(-0.5, 2.0) * np.exp(-np.maximum(y, 0) / (0.1 * bins)), 0)
        if i % 7 != 3 and f.sum() > 0:  # every seventh stays empty
            lam = f / f.sum() * 10.0 ** rng.uniform(0.5, 5.0)
            hist[i] = rng.poisson(lam) * rng.uniform(0.05, 0.2, bins)
    hist[0] = rng.uniform(0.5, 2.0, bins)  # every bin filled
    d = [torch.from_numpy(x).cuda() for x in (hist, shift)]
    o = torch.zeros((n, 5), dtype=torch.float32, device="cuda")
    pp._lib.check(pp._lib.load().pp_gamma_mixture_fit(d[0].data_ptr(), n, bins, t0, bw, d[1].data_ptr(), o.data_ptr(),
                                                      iters, None))
    got = o.cpu().numpy().astype(np.float64)
    for i in range(n) if n <= 700 else rng.integers(0, n, 200):
        want = _em(hist[i], centre - np.float64(shift[i]), iters)
        np.testing.assert_allclose(got[i], want, rtol=2e-5, atol=1e-6, err_msg=str((i, got[i], want)))
