"""Light sources over interval counts around a block's seven, every emitter, and the cross product over ragged source
and module counts, against the FP64 oracle and the records they are made of (whole records, byte for byte)."""
import numpy as np
import pytest

import photonprop_b200 as pp
from photonprop_b200 import lightyield as ly
from oracle import lightyield as OL
from oracle import tables as tb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("intervals,particles", [(1, 1), (6, 2), (7, 3), (8, 1), (15, 5), (301, 2)])
def test_interval_groups(propagator, intervals, particles):  # energies that the FP32 particle record holds exactly
    rng = np.random.default_rng(intervals)
    d = rng.normal(size=(particles, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    types = list(ly.ParticleType)
    parts = [ly.Particle(tuple(rng.uniform(-5, 5, 3)), tuple(d[i]), float(i), float(np.float32(10 ** rng.uniform(0, 4))),
                         types[i % 3]) for i in range(particles)]
    src, ng = ly.particles_to_sources(propagator, parts, (0.0, 0.05 * intervals), 0.05, mode="metres", emitter="cascade")
    assert ng == intervals + 1 and len(src) == particles * intervals
    g = 0.05 * np.arange(ng)
    om = tb.cascadia(35.0, 2.0)
    for i, p in enumerate(parts):
        ref = OL.elongated_sources(p.position, p.direction, p.time, p.energy, p.type, g, om, (300.0, 800.0), "metres")
        s = src[i * intervals:(i + 1) * intervals]
        assert np.all(np.abs(s["n_photons"] - np.array([r[2] for r in ref])) <= (np.abs(s["n_photons"]) > 0))
        assert np.count_nonzero(s["n_photons"] != np.array([r[2] for r in ref])) <= 1
        np.testing.assert_allclose(s["pos"], np.array([r[0] for r in ref]), rtol=1e-6, atol=1e-5)
        np.testing.assert_allclose(s["dir"], np.tile(p.direction, (intervals, 1)), rtol=1e-6)
        assert np.all(s["emitter"] == pp._lib.EMITTER_CASCADE) and not np.any(s["reserved"])


@pytest.mark.parametrize("n_s,n_t", [(1, 1), (1, 513), (51, 1), (7, 3), (52, 64), (1000, 13)])
def test_cross_product_records(propagator, n_s, n_t):
    rng = np.random.default_rng(n_s)
    src = rng.integers(0, 256, n_s * 80, dtype=np.uint8).view(pp.PAIR_DTYPE)
    tg = rng.uniform(-50, 50, (n_t, 4)).astype(np.float32)
    seed = 2**63 + 12345
    got = ly.cross_pairs(propagator, src, tg, seed=seed)
    want = np.repeat(src, n_t)
    want["target"] = np.tile(tg[:, :3], (n_s, 1))
    want["radius"] = np.tile(tg[:, 3], n_s)
    want["seed"] = [pp.pair_seed(seed, i) for i in range(n_s * n_t)]
    assert got.tobytes() == want.tobytes()
