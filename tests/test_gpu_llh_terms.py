"""A source whose first shape is infinite: its log-density (-inf + inf at any time) is not a number, which leaves the
hits that it reaches without a density, -inf, as the log-sum-exp of the terms has always given; the module beside it
is not touched (rtol 1e-10 as in test_gpu_event.py)."""
import numpy as np
import pytest
from scipy import stats

from photonprop_b200 import event as ev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,at", [(10, 3), (1, 0), (600, 555)])
def test_infinite_shape(propagator, S, at):
    rng = np.random.default_rng(S)
    p = np.empty((1, 2, S, 6))
    p[..., 0] = rng.uniform(0.01, 3.0, (1, 2, S))
    p[..., 1] = rng.uniform(0.1, 0.9, (1, 2, S))
    p[..., 2] = rng.uniform(0.2, 6.0, (1, 2, S))
    p[..., 3] = rng.uniform(1.0, 30.0, (1, 2, S))
    p[..., 4] = rng.uniform(0.5, 8.0, (1, 2, S))
    p[..., 5] = rng.uniform(0.0, 150.0, (1, 2, S))
    p[0, 1, at, 2] = np.inf
    hits = [np.array([300.0, 170.0]), np.array([300.0, 170.0, 220.0])]
    got = ev.event_llh(propagator, p, hits)
    A, w, a1, a2, th, sh = p[0, 0].T
    y = hits[0][:, None] - sh
    f = sum(v * A / A.sum() * stats.gamma.pdf(y, a, scale=th) for v, a in ((w, a1), (1 - w, a2))).sum(1)
    assert got[0, 0] == pytest.approx(stats.poisson.logpmf(len(y), A.sum()) + np.log(f).sum(), rel=1e-10, abs=1e-9)
    assert got[0, 1] == -np.inf
