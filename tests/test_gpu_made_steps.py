"""Steps that are made against steps that are counted: the same where no photon ends out of reach (compat mode, an
unbounded time), none where every photon starts out of reach, and in between the counted ones less one for each photon
that ends out of reach, which are the photons that neither hit nor run out of time or steps."""
import numpy as np
import pytest

import photonprop_b200 as pp

pytestmark = pytest.mark.gpu


def _both(prop, pairs, ro):
    import torch
    d = torch.from_numpy(pairs.view(np.uint8).copy()).cuda()
    cnt = torch.zeros(4, dtype=torch.int64, device="cuda")
    stats = torch.zeros((len(pairs), 8), dtype=torch.float64, device="cuda")
    prop.propagate_device(d, len(pairs), ro, None, 0, cnt, stats, None)
    return prop.made_steps(d, len(pairs), ro), int(cnt[1])


def _pairs(n, distance):
    p = pp.batches.mixed_batch(n, seed=4, cone_fraction=0.5)
    p["target"] = p["pos"] + distance * np.array([0.6, 0.0, 0.8], dtype=np.float32)
    p["n_photons"] = 1000 + 37 * np.arange(n)
    p["n_photons"][0] = 0
    return p


@pytest.mark.parametrize("n", [1, 5, 40])
def test_made_and_counted(propagator, n):
    ro = dict(mode="physical", hist_bins=0, write_hits=False)
    pairs = _pairs(n + 1, 30.0)
    photons = int(pairs["n_photons"].sum())
    assert _both(propagator, pairs, pp.RunOptions(t_max=1.0, **ro)) == (0, photons)  # 0.2 m of 30
    made, counted = _both(propagator, pairs, pp.RunOptions(t_max=1e8, max_steps=7, **ro))
    assert made == counted > photons
    made, counted = _both(propagator, pairs, pp.RunOptions(t_max=300.0, **ro))
    assert counted - photons <= made < counted
    iso = pairs.copy()
    iso["emitter"], iso["track_len"] = 0, 0.0
    made, counted = _both(propagator, iso, pp.RunOptions(mode="compat", hist_bins=0, write_hits=False))
    assert made == counted > 0
    assert propagator.made_steps(None, 0, pp.RunOptions(**ro)) == 0
