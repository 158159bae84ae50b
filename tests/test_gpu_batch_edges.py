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


@pytest.mark.parametrize("n_pairs,chunk", [(1, 0), (3, 1), (4095, 33), (4096, 0), (4097, 100_000), (9001, 0)])
def test_work_queue_covers_every_photon(propagator, n_pairs, chunk):
    """Tiles of the set-up scan (4096 pairs), empty pairs and run lengths: every photon is propagated exactly once
    (the same hits and step count as one launch per pair, histograms that start 8 bytes off a 16-byte boundary)."""
    import torch
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(n_pairs)
    counts = rng.integers(0, 200, n_pairs) * (rng.uniform(size=n_pairs) < 0.7)
    counts[rng.integers(0, n_pairs)] = 100_000
    pairs = _pairs(counts, np.full(n_pairs, 1.2), False, n_pairs)
    bins, cap = 31, 1 << 16
    ro = pp.RunOptions(mode="physical", t_max=31.0, hist_bins=bins, chunk_photons=chunk)
    d_pairs = torch.from_numpy(pairs.view(np.uint8).copy()).to(dev)
    hits = torch.zeros(cap * 64, dtype=torch.uint8, device=dev)
    cnt = torch.full((4,), 7, dtype=torch.int64, device=dev)
    st = torch.full((n_pairs, 8), 3.0, dtype=torch.float64, device=dev)
    flat = torch.full((n_pairs * bins + 2,), 5.0, dtype=torch.float64, device=dev)
    propagator.propagate_device(d_pairs, n_pairs, ro, hits, cap, cnt, st, flat[1:-1])
    torch.cuda.synchronize()
    n = int(cnt[0])
    h = hits[:n * 64].cpu().numpy().view(pp.HIT_DTYPE)
    h = h[np.lexsort((h["photon"], h["pair"]))]
    want = propagator.propagate_plain(pairs[counts > 0], ro, hit_capacity=cap)
    w = want.sorted_hits()
    w["pair"] = np.flatnonzero(counts > 0)[w["pair"]]
    np.testing.assert_array_equal(h.view(np.uint8), w.view(np.uint8))
    steps = 0  # photons are a function of (seed, index): a pair alone makes the same steps
    one_cnt = torch.zeros(4, dtype=torch.int64, device=dev)
    for i in rng.permutation(np.flatnonzero(counts > 0))[:20] if n_pairs > 20 else np.flatnonzero(counts > 0):
        propagator.propagate_plain_device(d_pairs[80 * i:], pairs[i:i + 1], 0, ro, hits, 0, one_cnt, st[i:i + 1],
                                          torch.zeros(bins, dtype=torch.float64, device=dev))
        steps += int(one_cnt[1])
    if n_pairs <= 20:
        assert steps == int(cnt[1])
    assert int(cnt[1]) >= int(counts.sum()) and cnt[2:].tolist() == [1 if n > cap else 0, 0]
    s = st.cpu().numpy()
    np.testing.assert_array_equal(s[:, 6], counts)
    np.testing.assert_array_equal(np.bincount(h["pair"], minlength=n_pairs), s[:, 0])
    assert float(flat[0]) == 5.0 and float(flat[-1]) == 5.0
    hist = flat[1:-1].reshape(n_pairs, bins).cpu().numpy()
    np.testing.assert_allclose(hist.sum(1), s[:, 1], rtol=1e-12, atol=1e-300)
