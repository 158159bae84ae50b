"""The batched kernel at the edges of its warp passes: photon counts around a
pass of 32, pairs whose photons all start out of reach among pairs in reach,
step limits of 1 and 2, isotropic scattering and a single wavelength, photon
by photon against the FP64 oracle (the tolerances of tests/_parity.py)."""
import numpy as np
import pytest

import photonprop_b200 as pp
from oracle import oracle as O
from _parity import check_matched, match_hits, to_oracle_opts, to_oracle_pairs

pytestmark = pytest.mark.gpu


def _pairs(counts, distances, cone, seed):
    p = pp.batches.mixed_batch(len(counts), seed=seed, cone_fraction=1.0 if cone else 0.0)
    d = p["target"] / np.linalg.norm(p["target"], axis=1, keepdims=True)
    p["target"] = d * np.asarray(distances)[:, None]
    p["n_photons"] = counts
    return p


def _check(prop, tables, pairs, ro, label, min_hits):
    res = prop.propagate(pairs, ro, hit_capacity=1 << 20)
    h, s, hist, steps, total = O.propagate(tables, to_oracle_pairs(pairs), to_oracle_opts(ro))
    assert total >= min_hits, (label, total)
    g, o, ng, no = match_hits(res.hits, h)
    check_matched(g, o, ng, no, label)
    np.testing.assert_array_equal(res.stats[:, 6], pairs["n_photons"])
    plain = prop.propagate_plain(pairs, ro, hit_capacity=1 << 20)
    assert plain.n_hits == res.n_hits
    np.testing.assert_array_equal(plain.sorted_hits().view(np.uint8), res.sorted_hits().view(np.uint8))


@pytest.mark.parametrize("cone", [False, True])
@pytest.mark.parametrize("max_steps,g", [(1, 0.95), (2, 0.95), (1000, 0.0), (1000, 0.95)])
def test_physical_ragged_counts_and_out_of_reach_pairs(propagator, oracle_tables, cone, max_steps, g):
    near = [1, 31, 32, 33, 0, 63, 64, 65, 4095, 4097, 150_000, 200_001]
    pairs = np.concatenate([_pairs(near, [1.5] * len(near), cone, 3),
                            _pairs([100, 40_000], [400.0, 60.0], cone, 4),  # beyond t_max: never staged
                            _pairs([100_001], [2.0], cone, 5)])
    ro = pp.RunOptions(mode="physical", g=g, max_steps=max_steps, t_max=40.0, hist_bins=40)
    _check(propagator, oracle_tables, pairs, ro, f"edges cone={cone} {max_steps} {g}", 100)


@pytest.mark.parametrize("max_steps", [1, 2, 10])
def test_compat_ragged_counts(propagator, oracle_tables, max_steps):
    counts = [1, 31, 32, 33, 0, 4097, 20_001]
    pairs = _pairs(counts, [1.5] * len(counts), False, 6)
    pairs["target"] = (0.0, 0.0, 1.5)
    pairs["target"][3] = (0.0, 0.0, 20.0)
    ro = pp.RunOptions(mode="compat", max_steps=max_steps, hist_bins=0, pmt_weight=False)
    _check(propagator, oracle_tables, pairs, ro, f"compat edges {max_steps}", 100)


def test_single_wavelength(medium, oracle_medium):
    pmt = pp.p_one_pmt_acc
    with pp.Propagator(medium, pp.Monochromatic(430.0), pmt, device=0) as prop:
        knots = prop.knots().astype(np.float64)
        assert knots.tolist() == [430.0]
        tables = O.make_tables(oracle_medium, knots, pmt=(pmt.wavelengths, pmt.acceptance))
        pairs = _pairs([50_000, 33], [2.0, 1.5], False, 7)
        _check(prop, tables, pairs, pp.RunOptions(mode="physical", t_max=60.0, hist_bins=60), "430 nm", 20)


def test_step_count_of_photons_out_of_reach(propagator):
    """A photon that starts out of reach counts one step: the one that would end it."""
    import torch
    dev = torch.device("cuda:0")
    pairs = _pairs([1000, 33, 77_777], [400.0, 500.0, 600.0], False, 8)
    d_pairs = torch.from_numpy(pairs.view(np.uint8).copy()).to(dev)
    cnt = torch.zeros(4, dtype=torch.int64, device=dev)
    st = torch.zeros((3, 8), dtype=torch.float64, device=dev)
    hits = torch.zeros(64, dtype=torch.uint8, device=dev)
    ro = pp.RunOptions(mode="physical", t_max=500.0, hist_bins=0)
    propagator.propagate_device(d_pairs, 3, ro, hits, 0, cnt, st, None)
    torch.cuda.synchronize()
    assert cnt.tolist() == [0, int(pairs["n_photons"].sum()), 0, 0]
