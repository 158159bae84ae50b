"""pp_propagate's copies around its pinned staging: pairs, result blocks and hits of sizes on either side of what is
staged (1000 pairs, 512 KiB of results, 256 hits), and hit capacities of 0, below and above the hits, against one
launch per pair."""
import numpy as np
import pytest

import photonprop_b200 as pp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pairs,bins,photons", [(1, 0, 300_000), (1, 500, 20_000), (60, 1000, 20_000),
                                                  (64, 1000, 20_000), (65, 1000, 20_000), (1024, 10, 500),
                                                  (1025, 10, 500), (7, 10_000, 4000)])
@pytest.mark.parametrize("compact_cap", [0, 3, 256, 1 << 18])
def test_copies(propagator, n_pairs, bins, photons, compact_cap):
    pairs = pp.batches.mixed_batch(n_pairs, seed=n_pairs, cone_fraction=0.0)
    pairs["target"] *= 1.2 / np.linalg.norm(pairs["target"], axis=1, keepdims=True)
    pairs["n_photons"] = photons
    ro = pp.RunOptions(mode="physical", t_max=60.0, hist_bins=bins)
    want = propagator.propagate_plain(pairs, ro, hit_capacity=1 << 18)
    assert want.n_hits > 3  # 155 to thousands: fewer and more than are staged
    got = propagator.propagate(pairs, ro, hit_capacity=compact_cap)
    assert got.n_hits == want.n_hits and got.overflow == (want.n_hits > compact_cap)
    assert len(got.hits) == min(compact_cap, want.n_hits)
    np.testing.assert_allclose(got.stats, want.stats, rtol=1e-12)
    np.testing.assert_allclose(got.hist, want.hist, rtol=1e-12, atol=1e-300)
    key = {(int(h["pair"]), int(h["photon"])): h.tobytes() for h in want.hits}
    assert all(key[(int(h["pair"]), int(h["photon"]))] == h.tobytes() for h in got.hits)
    if not got.overflow:
        assert got.sorted_hits().tobytes() == want.sorted_hits().tobytes()
