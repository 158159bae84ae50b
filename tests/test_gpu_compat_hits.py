"""Compat mode where most photons hit and many steps are left to the others, so that the batched kernel refills its
idle lanes: the same hits, sums and step counts as one launch per pair, for pairs that end within a granule, runs that
change pair while lanes are refilled, and step limits on either side of the rule."""
import numpy as np
import pytest

import photonprop_b200 as pp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_steps", [10, 24, 25, 26, 150])
@pytest.mark.parametrize("n,photons", [(1, 20_000), (40, 1501), (300, 33)])
def test_as_one_launch_per_pair(propagator, n, photons, max_steps):
    import torch
    pairs = pp.batches.mixed_batch(n, seed=n, cone_fraction=0.0)
    # emission within 1 rad of +z: a sphere at 0.21 / sin(f) is met by a share f of the photons, here 0 to 1 by pair
    f = (0.5 + np.arange(n)) / n if n > 1 else np.array([0.7])
    pairs["target"] = pairs["pos"]
    pairs["target"][:, 2] += (0.21 / np.sin(f)).astype(np.float32)
    pairs["radius"], pairs["n_photons"] = 0.21, photons + np.arange(n) % 5
    ro = pp.RunOptions(mode="compat", max_steps=max_steps, hist_bins=20)
    cap = 1 << 17
    want = propagator.propagate_plain(pairs, ro, hit_capacity=cap)
    got = propagator.propagate(pairs, ro, hit_capacity=cap)
    assert got.n_hits == want.n_hits > 0.4 * int(pairs["n_photons"].sum())
    assert got.sorted_hits().tobytes() == want.sorted_hits().tobytes()
    np.testing.assert_allclose(got.stats, want.stats, rtol=1e-12)
    np.testing.assert_allclose(got.hist, want.hist, rtol=1e-12, atol=1e-300)
    d = torch.from_numpy(pairs.view(np.uint8).copy()).cuda()
    cnt = torch.zeros(4, dtype=torch.int64, device="cuda")
    st = torch.zeros((n, 8), dtype=torch.float64, device="cuda")
    hist = torch.zeros((n, 20), dtype=torch.float64, device="cuda")
    propagator.propagate_device(d, n, ro, None, 0, cnt, st, hist)
    assert int(cnt[1]) == propagator.made_steps(d, n, ro)
