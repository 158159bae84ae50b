"""The event likelihood over hit counts around a warp, a pass of 128 hits and a chunk, sources around a tile of 512,
and hits whose density leaves the range that is summed directly (far tails, hits before every source, a hit at time 0,
terms that are not finite), against the FP64 oracle: rtol 1e-10 as in test_gpu_event.py.  Where the density is below
the FP64 range, which the oracle sums as it is, the reference is the log-sum-exp of scipy's log-densities."""
import numpy as np
import pytest
from scipy import special, stats

from photonprop_b200 import event as ev
from oracle import event as OE

pytestmark = pytest.mark.gpu


def _params(rng, H, M, S):
    p = np.empty((H, M, S, 6))
    p[..., 0] = rng.uniform(0.01, 3.0, (H, M, S))
    p[..., 1] = rng.uniform(0.0, 1.0, (H, M, S))
    p[..., 2] = rng.uniform(0.2, 6.0, (H, M, S))
    p[..., 3] = rng.uniform(1.0, 30.0, (H, M, S))
    p[..., 4] = rng.uniform(0.5, 8.0, (H, M, S))
    p[..., 5] = rng.uniform(0.0, 150.0, (H, M, S))
    p[..., 0, 5] = 0.0
    return p


def _log_space(p, x):
    A, w, a1, a2, th, sh = p.T
    y = np.asarray(x)[:, None] - sh
    with np.errstate(divide="ignore", invalid="ignore"):
        g = [np.log(f * A / A.sum()) + stats.gamma.logpdf(y, a, scale=th) for f, a in ((w, a1), (1 - w, a2))]
    return stats.poisson.logpmf(len(x), A.sum()) + special.logsumexp(np.concatenate(g, 1), axis=1).sum()


def _check(prop, p, hits, mode="shifted", ref=None):
    got = ev.event_llh(prop, p, hits, mode=mode)
    for h in range(p.shape[0]):
        for m in range(p.shape[1]):
            with np.errstate(divide="ignore", invalid="ignore"):
                want = ref(p[h, m], hits[m]) if ref else OE.module_llh(p[h, m], hits[m], None, mode)
            if np.isfinite(want):
                assert got[h, m] == pytest.approx(want, rel=1e-10, abs=1e-9), (h, m)
            else:
                assert got[h, m] == want, (h, m)


@pytest.mark.parametrize("S", [1, 3, 4, 5, 511, 512, 513])
@pytest.mark.parametrize("mode", ["reference", "shifted"])
def test_hit_counts_and_source_tiles(propagator, S, mode):
    rng = np.random.default_rng(S)
    counts = [0, 1, 31, 32, 33, 96, 127, 128, 129, 300]
    p = _params(rng, 2, len(counts), S)
    _check(propagator, p, [rng.uniform(0.5, 200.0, n) for n in counts], mode)


def test_more_hits_than_a_chunk(propagator):
    rng = np.random.default_rng(5)
    p = _params(rng, 64, 2, 7)
    _check(propagator, p, [np.sort(rng.uniform(0.5, 200.0, n)) for n in (20_000, 1025)])


def test_densities_beyond_the_direct_sum(propagator):
    rng = np.random.default_rng(6)
    p = _params(rng, 1, 5, 40)
    p[0, :, :, 4] = np.minimum(p[0, :, :, 4], 2.0)  # theta: exp(-x / theta) below 1e-300 at 2000 ns
    p[0, 2, :, 5] = -1.0  # hits at time 0 and tiny times
    p[0, 3, :, 0] = 0.0   # no light at all
    p[0, 3, 0, 0] = 1e-3
    p[0, 4, :, 2] = 3.0
    p[0, 4, 5, 2] = 400.0  # a shape whose first factor is far below the range near its shift
    hits = [np.array([2000.0, 1500.0, 50.0, 1400.0]), np.array([-5.0, 10.0]), np.array([0.0, 1e-295, 3.0]),
            np.array([40.0, 900.0]), np.array([1e-3, 2e-3, 60.0])]
    _check(propagator, p, hits, ref=_log_space)


def test_terms_that_are_not_finite(propagator):
    """A source with a NaN leaves no density to the hits it reaches: -inf, as the log-sum-exp of its terms gives."""
    rng = np.random.default_rng(7)
    p = _params(rng, 1, 3, 10)
    p[0, 1, 3, 2] = np.inf
    p[0, 2, 3, 4] = np.nan
    got = ev.event_llh(propagator, p, [np.array([300.0]), np.array([300.0]), np.array([300.0])])
    assert np.isfinite(got[0, 0]) and got[0, 2] == -np.inf
