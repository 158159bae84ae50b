"""Performance cases: the calls a user of photonprop_b200 makes, over the sizes the library is used at.

propagate_host    Propagator.propagate on host arrays: single sources and requests of a few pairs (latency)
propagate_device  Propagator.propagate_device on device buffers: whole batches and event-driven batches
fits              modelling.propagate_fit: reference-compatible propagation, reweighting and Gamma fits
forward, train    the surrogate network: queries, and one training step with its gradients
mixture           the Gamma-mixture fit of arrival-time histograms (the surrogate's training targets)
llh               the event likelihood of many hypotheses
lightyield        particles -> light sources -> source x module pairs
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

PKG_ROOT = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "photonprop.jl_b200")
if PKG_ROOT not in sys.path:
    sys.path.insert(0, PKG_ROOT)

import photonprop_b200 as pp  # noqa: E402
from photonprop_b200 import _lib, lightyield, modelling, surrogate  # noqa: E402

N_800 = 1.3713        # group index at 800 nm of the likelihood's time shifts
C_VAC = 0.299792458   # m/ns
HIT_ROWS = 2048       # rows of hit records that come back, in (pair, photon) order
HIT_COLUMNS = ("pos", "time", "dir0", "weight", "dir", "wavelength", "dist", "pair", "photon")


def listed():
    return [
        # the isotropic point source that also runs on a CPU: one small call, all latency
        {"name": "point-1e5", "kind": "propagate_host", "pairs": 1, "n_min": 1e5, "n_max": 1e5,
         "d_min": 10.0, "d_max": 10.0, "cone": 0.0, "bins": 500, "mode": "physical"},
        # one request of the serving stream: tens of uneven pairs, isotropic and cone emitters
        {"name": "request-33-pairs", "kind": "propagate_host", "pairs": 33, "n_min": 1e4, "n_max": 1e6,
         "d_min": 2.0, "d_max": 150.0, "cone": 0.5, "bins": 1000, "mode": "physical"},
        # the headline batch
        {"name": "mixed-4096-pairs", "kind": "propagate_device", "pairs": 4096, "n_min": 1e4, "n_max": 1e7,
         "d_min": 2.0, "d_max": 150.0, "cone": 0.5, "bins": 1000, "gev": 0.0},
        # a 10 GeV shower: 200 cascade-profile sources x 500 modules, about 1e4 photons per pair
        {"name": "event-1e5-cascade-pairs", "kind": "propagate_device", "pairs": 0, "n_min": 0.0, "n_max": 0.0,
         "d_min": 0.0, "d_max": 0.0, "cone": 0.0, "bins": 1000, "gev": 10.0},
        # a quick fit table, and a large one whose hits take a share of the time
        {"name": "fits-20x25", "kind": "fits", "photons": 1000000, "distances": 20, "angles": 25},
        {"name": "fits-100x250", "kind": "fits", "photons": 20000000, "distances": 100, "angles": 250},
        # surrogate queries: a full batch, and the few thousand of a small detector (ragged)
        {"name": "queries-1e6", "kind": "forward", "n": 1000000},
        {"name": "queries-3001", "kind": "forward", "n": 3001},
        # one Adam step at the batch the surrogate is trained with
        {"name": "train-4096", "kind": "train", "n": 4096},
        # training targets of one chunk of pairs
        {"name": "mixture-20000", "kind": "mixture", "n": 20000, "bins": 1000, "iters": 60},
        # 64 energy hypotheses of a 100 GeV shower
        {"name": "likelihood-64", "kind": "llh", "hypotheses": 64, "modules": 500, "sources": 200,
         "hits": 46000, "mode": "shifted"},
        # the same shower's sources, and a pair with every module
        {"name": "sources-and-pairs", "kind": "lightyield", "particles": 1, "intervals": 200,
         "modules": 500},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["propagate_host", "propagate_host", "propagate_device", "propagate_device", "fits", "forward",
                       "train", "mixture", "llh", "lightyield"])
    if kind == "propagate_host":  # 1 to 64 pairs, at most a few 1e7 photons
        n_min = _log(rng, 1e3, 1e5)
        d_min = rng.uniform(2.0, 40.0)
        return {"kind": kind, "pairs": int(round(_log(rng, 1, 64))), "n_min": n_min, "n_max": n_min * _log(rng, 1, 30),
                "d_min": d_min, "d_max": d_min + rng.uniform(0.0, 110.0), "cone": rng.choice([0.0, 0.5, 1.0]),
                "bins": rng.choice([0, 137, 500, 1000]), "mode": rng.choice(["physical", "physical", "compat"])}
    if kind == "propagate_device":
        if rng.random() < 0.5:  # a shower of 1 to 30 GeV
            return {"kind": kind, "pairs": 0, "n_min": 0.0, "n_max": 0.0, "d_min": 0.0, "d_max": 0.0, "cone": 0.0,
                    "bins": rng.choice([250, 1000]), "gev": _log(rng, 1.0, 30.0)}
        pairs = int(round(_log(rng, 60, 4096)))
        n_min = _log(rng, 1e3, 1e5)
        d_min = rng.uniform(2.0, 40.0)
        n_max = min(1e7, n_min * _log(rng, 1, 1000), max(n_min, 5e9 / pairs))
        return {"kind": kind, "pairs": pairs, "n_min": n_min, "n_max": n_max,
                "d_min": d_min, "d_max": d_min + rng.uniform(0.0, 110.0), "cone": rng.choice([0.0, 0.5, 1.0]),
                "bins": rng.choice([0, 333, 1000]), "gev": 0.0}
    if kind == "fits":  # up to 1e9 photons in all
        distances = int(round(_log(rng, 5, 100)))
        return {"kind": kind, "photons": int(_log(rng, 1e5, 1e9 / distances)), "distances": distances,
                "angles": int(round(_log(rng, 7, 250)))}
    if kind == "forward":
        return {"kind": kind, "n": int(_log(rng, 100, 1e6))}
    if kind == "train":
        return {"kind": kind, "n": int(_log(rng, 200, 16384))}
    if kind == "mixture":
        return {"kind": kind, "n": int(_log(rng, 200, 20000)), "bins": rng.choice([200, 500, 1000]),
                "iters": rng.choice([30, 60])}
    if kind == "llh":
        modules = int(_log(rng, 20, 500))
        return {"kind": kind, "hypotheses": int(round(_log(rng, 1, 64))), "modules": modules,
                "sources": int(_log(rng, 5, 700 if modules < 100 else 200)), "hits": int(modules * _log(rng, 3, 90)),
                "mode": rng.choice(["shifted", "shifted", "reference"])}
    return {"kind": kind, "particles": int(round(_log(rng, 1, 60))), "intervals": int(_log(rng, 20, 300)),
            "modules": int(_log(rng, 3, 500))}


# ---- what a program has in hand before the call ---------------------------------------------------------------

_propagators = {}


def _propagator(name="seawater"):
    """A program's one context for its medium: 35 permille sea water, or the Cascadia site of the fit tables."""
    if name not in _propagators:
        m = pp.make_seawater(35.0, 2.0) if name == "seawater" else pp.make_cascadia_medium_properties()
        _propagators[name] = pp.Propagator(m, pp.CherenkovSpectrum((300.0, 800.0), 20, m), pp.p_one_pmt_acc, device=0)
    return _propagators[name]


def _detector(n):
    """n modules on strings 20 m apart, 20 per string, 5 m between modules."""
    strings = -(-n // 20)
    side = int(math.ceil(math.sqrt(strings)))
    xyz = [((i // 20 % side - 0.5 * (side - 1)) * 20.0, (i // 20 // side - 0.5 * (side - 1)) * 20.0,
            -40.0 + 5.0 * (i % 20), 0.21) for i in range(n)]
    return np.array(xyz, dtype=np.float32)


def _particles(n, rng, gev=None):
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return [lightyield.Particle(tuple(rng.uniform(-10, 10, 3)), tuple(d[i]), float(rng.uniform(0, 50)),
                                gev if gev else float(10 ** rng.uniform(0, 3)),
                                rng.choice(list(lightyield.ParticleType))) for i in range(n)]


def _mixed_pairs(case, seed):
    pairs = pp.batches.mixed_batch(case["pairs"], seed=seed, n_min=case["n_min"], n_max=case["n_max"],
                                   d_min=case["d_min"], d_max=case["d_max"], cone_fraction=case["cone"])
    if case.get("mode") == "compat":  # the reference's kernel emits isotropic photons only
        pairs["emitter"] = _lib.EMITTER_ISOTROPIC
        pairs["track_len"] = 0.0
    return pairs


def prepare(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    dev = torch.device("cuda", 0)
    kind = case["kind"]
    if kind == "propagate_host":
        opts = pp.RunOptions(mode=case["mode"], t_max=1000.0, hist_bins=case["bins"], pmt_weight=True)
        return {"kind": kind, "prop": _propagator(), "pairs": _mixed_pairs(case, seed), "opts": opts}
    if kind == "propagate_device":
        prop = _propagator()
        if case["gev"]:
            part = [lightyield.Particle(tuple(rng.uniform(-5, 5, 3)), (0.0, 0.0, 1.0), 0.0, case["gev"],
                                        lightyield.ParticleType.EMinus)]
            src, _ = lightyield.particles_to_sources(prop, part, (0.0, 20.0), 0.1, mode="metres", emitter="cascade")
            pairs = lightyield.cross_pairs(prop, src, _detector(500), seed=seed)
        else:
            pairs = _mixed_pairs(case, seed)
        n, bins, cap = len(pairs), case["bins"], 1 << 22
        opts = pp.RunOptions(mode="physical", t_max=1000.0, hist_bins=bins, cascade=bool(case["gev"]))
        return {"kind": kind, "prop": prop, "n": n, "opts": opts, "cap": cap,
                "pairs": torch.from_numpy(pairs.view(np.uint8).copy()).to(dev),
                "hits": torch.zeros(cap * 64, dtype=torch.uint8, device=dev),
                "counters": torch.zeros(4, dtype=torch.int64, device=dev),
                "stats": torch.zeros((n, 8), dtype=torch.float64, device=dev),
                "hist": torch.zeros((n, bins), dtype=torch.float64, device=dev) if bins else None}
    if kind == "fits":
        pairs, _, angles = modelling.fit_pairs(case["photons"], case["distances"], case["angles"], 300.0, seed)
        return {"kind": kind, "prop": _propagator("cascadia"), "pairs": pairs, "angles": angles,
                "opts": pp.RunOptions(mode="compat", pmt_weight=True, hist_bins=0)}
    if kind in ("forward", "train"):
        n = case["n"]
        net = surrogate.MLP(0, seed)
        s = {"kind": kind, "net": net, "n": n}
        if kind == "forward":
            net.set_normalization([1.2, 0.0, 5.5, 0.5], [0.5, 0.6, 0.9, 0.5], [-14.0, 0.0, 0.0, 1.0, 2.0],
                                  [2.0, 1.0, 0.5, 0.5, 0.7])
            s["x"] = torch.from_numpy(_features(rng, n)).to(dev)
            s["out"] = torch.zeros((5, n), dtype=torch.float32, device=dev)
            return s
        x = (_features(rng, n) - np.float32([1.2, 0.0, 5.5, 0.5])) / np.float32([0.5, 0.6, 0.9, 0.5])
        y = np.stack([np.tanh(x @ rng.normal(size=4)) + 0.3 * rng.normal(size=n) for _ in range(5)], axis=1)
        m = np.ones((n, 5))
        m[:, 0] = rng.uniform(0.0, 1.0, n)
        m[:, 1:] = (rng.uniform(size=(n, 1)) < 0.6) & (rng.uniform(size=(n, 4)) < 0.95)
        for k, v in (("x", x), ("y", y), ("mask", m)):
            s[k] = torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).to(dev)
        return s
    if kind == "mixture":
        hist, shift = _histograms(case["n"], case["bins"], seed, dev)
        return {"kind": kind, "hist": hist, "shift": shift, "n": case["n"], "bins": case["bins"],
                "iters": case["iters"], "out": torch.zeros((case["n"], 5), dtype=torch.float32, device=dev)}
    if kind == "llh":
        p, off, times = _event(case, rng)
        return {"kind": kind, "prop": _propagator(), "mode": _lib.LLH_REFERENCE if case["mode"] == "reference"
                else _lib.LLH_SHIFTED, "params": torch.from_numpy(p).to(dev), "offsets": torch.from_numpy(off).to(dev),
                "times": torch.from_numpy(times).to(dev),
                "out": torch.zeros(p.shape[:2], dtype=torch.float64, device=dev)}
    parts = lightyield.particles_array(_particles(case["particles"], rng))
    n_src = case["particles"] * case["intervals"]
    return {"kind": kind, "prop": _propagator(), "case": dict(case), "seed": seed, "n_src": n_src,
            "parts": torch.from_numpy(parts.view(np.uint8).copy()).to(dev),
            "modules": torch.from_numpy(_detector(case["modules"])).to(dev),
            "sources": torch.zeros((n_src, 80), dtype=torch.uint8, device=dev),
            "pairs": torch.zeros((n_src * case["modules"], 80), dtype=torch.uint8, device=dev)}


def _features(rng, n):
    return np.stack([rng.uniform(np.log10(2), np.log10(150), n), rng.uniform(-1, 1, n), rng.uniform(4, 7, n),
                     rng.integers(0, 2, n)], axis=1).astype(np.float32)


def _histograms(n, bins, seed, dev):
    """Arrival-time histograms (1 ns bins) as the propagation leaves them: 3 to 1e5 weighted hits per pair, most of
    them in the first nanoseconds after the geometric time, the others in a tail of tens of nanoseconds."""
    g = torch.Generator(device=dev).manual_seed(seed)
    u = torch.rand((n, 5), generator=g, device=dev, dtype=torch.float64)
    hits = 10.0 ** (0.5 + 4.5 * u[:, 0])
    shift = 0.5 * bins * u[:, 1]
    w, theta, a2 = 0.3 + 0.6 * u[:, 2], 5.0 + 40.0 * u[:, 3], 1.0 + 2.0 * u[:, 4]
    t = (torch.arange(bins, device=dev, dtype=torch.float64) + 0.5)[None, :] - shift[:, None]
    y = t.clamp_min(0.05)

    def pdf(a):
        return torch.exp((a - 1.0) * torch.log(y / theta[:, None]) - y / theta[:, None] - torch.lgamma(a)) \
            / theta[:, None]

    f = (w[:, None] * pdf(torch.full((n, 1), 0.6, device=dev, dtype=torch.float64))
         + (1.0 - w[:, None]) * pdf(a2[:, None])) * (t > 0)
    counts = torch.poisson(hits[:, None] * f / f.sum(1, keepdim=True).clamp_min(1e-30), generator=g)
    return counts * 0.07, shift.float()


def _event(case, rng):
    """A shower along +z seen by a detector: (hypotheses' parameters, hit offsets, hit times), CSR by module."""
    H, M, S = case["hypotheses"], case["modules"], case["sources"]
    mods = _detector(M)[:, :3].astype(np.float64)
    src = np.stack([np.full(S, 1.7), np.full(S, -2.3), 20.0 * (np.arange(S) + 0.5) / S], axis=1)
    d = np.linalg.norm(mods[:, None, :] - src[None, :, :], axis=2)
    z = (np.arange(S) + 0.5) / S
    share = z ** 3 * np.exp(-9.0 * z)
    a = share[None, :] * np.exp(-d / 30.0) / np.maximum(d, 1.0) ** 2
    a *= case["hits"] / a.sum()
    prm = np.empty((M, S, 6))
    prm[..., 0] = a
    prm[..., 1] = rng.uniform(0.2, 0.95, (M, S))
    prm[..., 2] = rng.uniform(0.2, 1.2, (M, S))
    prm[..., 3] = rng.uniform(1.2, 6.0, (M, S))
    prm[..., 4] = rng.uniform(3.0, 25.0, (M, S))
    prm[..., 5] = src[None, :, 2] / C_VAC + (d - 0.21) * N_800 / C_VAC
    counts = rng.poisson(a.sum(1))
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    times = np.zeros(max(int(off[-1]), 1))
    for k in range(M):
        n = int(counts[k])
        if not n:
            continue
        j = rng.choice(S, size=n, p=a[k] / a[k].sum())
        q = prm[k, j]
        shape = np.where(rng.uniform(size=n) < q[:, 1], q[:, 2], q[:, 3])
        first = prm[k, :, 5].min()  # every hit has a source that can have made it
        times[off[k]:off[k + 1]] = np.sort(np.maximum(first + 0.01, q[:, 5] + rng.gamma(shape, q[:, 4])))
    hyp = np.repeat(prm[None], H, axis=0)
    hyp[..., 0] *= np.geomspace(0.5, 2.0, H)[:, None, None] if H > 1 else 1.0
    hyp[..., 4] *= rng.uniform(0.95, 1.05, (H, 1, 1))
    return hyp, off, times


# ---- one pass -------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "propagate_host":
        r = s["prop"].propagate(s["pairs"], s["opts"])
        h = np.zeros(HIT_ROWS, dtype=_lib.HIT_DTYPE)  # as many rows for every seed; stats and hist hold all hits
        k = min(len(r.hits), HIT_ROWS)
        h[:k] = r.sorted_hits()[:k]
        out = {c: h[c] for c in HIT_COLUMNS}
        out.update(n_hits=r.n_hits, stats=r.stats, hist=r.hist)
        return out
    if kind == "propagate_device":
        s["prop"].propagate_device(s["pairs"], s["n"], s["opts"], s["hits"], s["cap"], s["counters"], s["stats"],
                                   s["hist"], stream=torch.cuda.current_stream())
        return {"counters": s["counters"], "stats": s["stats"], "hist": s["hist"]}
    if kind == "fits":
        r = modelling.propagate_fit(s["prop"], s["pairs"], s["angles"], s["opts"])
        return {"fits": r.fits, "moments": r.moments, "stats": r.stats, "n_hits": r.n_hits}
    if kind == "forward":
        s["net"].forward(s["x"], s["out"], s["n"], physical=True, stream=torch.cuda.current_stream())
        return s["out"]
    if kind == "train":
        loss, grads = s["net"].train_step(s["x"], s["y"], s["mask"], s["n"], 1e-3, want_grads=True)
        return {"loss": loss, "grads": grads}
    if kind == "mixture":
        _lib.check(_lib.load().pp_gamma_mixture_fit(s["hist"].data_ptr(), s["n"], s["bins"], 0.0, 1.0,
                                                    s["shift"].data_ptr(), s["out"].data_ptr(), s["iters"],
                                                    torch.cuda.current_stream().cuda_stream))
        return s["out"]
    if kind == "llh":
        H, M, S, _ = s["params"].shape
        _lib.check(_lib.load().pp_event_llh_device(
            s["prop"].handle, s["mode"], H, S, M, s["params"].data_ptr(), None, s["offsets"].data_ptr(),
            s["times"].data_ptr(), s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream), s["prop"].handle)
        return s["out"]
    c, n_grid, st = s["case"], ctypes.c_int64(0), torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.load().pp_particles_to_sources_device(
        s["prop"].handle, s["parts"].data_ptr(), c["particles"], 0.0, 0.1 * c["intervals"], 0.1, _lib.LY_METRES, 300.0,
        800.0, _lib.EMITTER_CASCADE, s["sources"].data_ptr(), s["n_src"], ctypes.byref(n_grid), st), s["prop"].handle)
    _lib.check(_lib.load().pp_cross_pairs_device(
        s["prop"].handle, s["sources"].data_ptr(), s["n_src"], s["modules"].data_ptr(), c["modules"], s["seed"],
        s["pairs"].data_ptr(), st), s["prop"].handle)
    # pp_pair: pos, t0, dir, track, target, radius (12 floats), photons, seed (2 words of 64 bits), emitter
    return {"sources": s["sources"].view(torch.float32)[:, :12], "photons": s["sources"].view(torch.int64)[:, 6],
            "pairs": s["pairs"]}


# ---- what the path cannot do without ---------------------------------------------------------------------------

STEPS = 4.3            # mean steps of a photon in the 1000 ns window of the mixed batch
FLOPS_STEP, FLOPS_START = 70.0, 60.0  # FP32 operations (a fused multiply-add is two) of a step and of an emission
MLP_FLOPS = 2.0 * (4 * 128 + 2 * 128 * 128 + 128 * 5)


def _photons(case):
    if case.get("gev"):
        return 500 * 2.3e5 * case["gev"]  # about 2.3e5 photons per GeV of a shower
    lo, hi = case["n_min"], case["n_max"]
    return case["pairs"] * (lo if hi <= lo * 1.0001 else (hi - lo) / math.log(hi / lo))


def work(case):
    kind = case["kind"]
    if kind.startswith("propagate"):
        pairs = 100000 if case.get("gev") else case["pairs"]
        steps = 10.0 if case.get("mode") == "compat" else STEPS
        return {"bytes": pairs * (80 + 64 + 8 * case["bins"]),
                "flops": _photons(case) * (steps * FLOPS_STEP + FLOPS_START)}
    if kind == "fits":
        photons = case["photons"] * case["distances"]
        return {"bytes": 0.036 * photons * 64 + case["distances"] * case["angles"] * 56,
                "flops": photons * (10 * FLOPS_STEP + FLOPS_START) + 0.036 * photons * case["angles"] * 18}
    if kind == "forward":
        return {"bytes": case["n"] * 36, "flops": case["n"] * MLP_FLOPS}
    if kind == "train":
        return {"bytes": case["n"] * 56 + 6 * 34437 * 4, "flops": 3 * case["n"] * MLP_FLOPS}
    if kind == "mixture":  # about a third of the bins hold hits; two densities each, in 64 bits
        return {"bytes": case["n"] * (8 * case["bins"] + 24),
                "flops": case["n"] * case["bins"] * case["iters"] / 3 * 100.0}
    if kind == "llh":  # two densities for every (hit, source, hypothesis), in 64 bits
        return {"bytes": 48 * case["hypotheses"] * case["modules"] * case["sources"] + 8 * case["hits"],
                "flops": 100.0 * case["hypotheses"] * case["sources"] * case["hits"]}
    n_src = case["particles"] * case["intervals"]
    return {"bytes": n_src * 80 * (1 + case["modules"]), "flops": 50 * 150.0 * (n_src + case["particles"])}


# ---- the values in 64 bits ---------------------------------------------------------------------------------------

def exact(case, seed):
    """The propagation has none here: its outputs are sums over photons that follow the library's own random numbers
    through tens of scatterings, and a photon at the rim of a sphere hits or misses by the last bit."""
    kind = case["kind"]
    if kind.startswith("propagate") or kind == "fits":
        return None
    s = prepare(case, seed)
    return {"forward": _exact_forward, "train": _exact_train, "mixture": _exact_mixture, "llh": _exact_llh,
            "lightyield": _exact_lightyield}[kind](s)


def _weights(net):
    p = torch.from_numpy(net.get_params().astype(np.float64)).cuda()
    out, at = [], 0
    for shape in ((128, 4), (128,), (128, 128), (128,), (128, 128), (128,), (5, 128), (5,)):
        n = math.prod(shape)
        out.append(p[at:at + n].reshape(shape).clone().requires_grad_())
        at += n
    return out


def _net(w, x):
    h = x
    for i in range(0, 6, 2):
        h = torch.nn.functional.gelu(h @ w[i].T + w[i + 1], approximate="tanh")
    return h @ w[6].T + w[7]


def _exact_forward(s):
    xm, xs, ym, ys = (torch.from_numpy(a.astype(np.float64)).cuda() for a in s["net"].get_normalization())
    with torch.no_grad():
        x = s["x"].double()
        y = _net(_weights(s["net"]), (x - xm) / xs) * ys + ym
        mu = torch.exp(y[:, 0] + x[:, 2] * math.log(10.0))
        return torch.stack([mu, torch.sigmoid(y[:, 1]), *torch.exp(y[:, 2:]).T])


def _exact_train(s):
    w = _weights(s["net"])
    m = s["mask"].double()
    loss = (m * (_net(w, s["x"].double()) - s["y"].double()) ** 2).sum() / m.sum()
    loss.backward()
    return {"loss": float(loss), "grads": torch.cat([p.grad.reshape(-1) for p in w])}


def _exact_mixture(s):
    h, n = s["hist"], s["n"]
    t = (torch.arange(s["bins"], device=h.device, dtype=torch.float64) + 0.5)[None, :] - s["shift"].double()[:, None]
    h = torch.where((t > 0) & (h > 0), h, torch.zeros_like(h))
    t = torch.where(h > 0, t, torch.ones_like(t))
    lt = torch.log(t)
    s0 = h.sum(1)
    m = (h * t).sum(1) / s0
    v = torch.maximum((h * t * t).sum(1) / s0 - m * m, 1e-6 * m * m + 1e-12)
    a0 = (m * m / v).clamp_min(0.05)
    w, a1, a2, th = torch.full_like(m, 0.5), (0.5 * a0).clamp_min(0.02), 2.0 * a0, v / m
    ll = None

    def inv_digamma(y):
        a = torch.where(y >= -2.22, torch.exp(y) + 0.5, -1.0 / (y + 0.5772156649015329))
        for _ in range(8):
            a = (a - (torch.digamma(a) - y) / torch.polygamma(1, a)).clamp_min(1e-3)
        return a

    for _ in range(s["iters"]):
        c1 = torch.log(w) - a1 * torch.log(th) - torch.lgamma(a1)
        c2 = torch.log1p(-w) - a2 * torch.log(th) - torch.lgamma(a2)
        p1 = c1[:, None] + (a1[:, None] - 1) * lt - t / th[:, None]
        p2 = c2[:, None] + (a2[:, None] - 1) * lt - t / th[:, None]
        r = torch.sigmoid(p1 - p2)
        ll = (h * torch.logaddexp(p1, p2)).sum(1) / s0
        ha, hb = h * r, h * (1 - r)
        sa = [ha.sum(1), (ha * t).sum(1), (ha * lt).sum(1)]
        sb = [hb.sum(1), (hb * t).sum(1), (hb * lt).sum(1)]
        w = (sa[0] / (sa[0] + sb[0])).clamp(1e-4, 1 - 1e-4)
        for _ in range(3):
            th = (sa[1] + sb[1]) / (a1 * sa[0] + a2 * sb[0])
            a1 = torch.where(sa[0] > 0, inv_digamma(sa[2] / sa[0] - torch.log(th)), a1)
            a2 = torch.where(sb[0] > 0, inv_digamma(sb[2] / sb[0] - torch.log(th)), a2)
    swap = a1 > a2
    out = torch.stack([torch.where(swap, 1 - w, w), torch.where(swap, a2, a1), torch.where(swap, a1, a2), th, ll], 1)
    return torch.where((s0 > 0)[:, None], out, torch.full_like(out, math.nan))


def _exact_llh(s):
    p, off, x = s["params"], s["offsets"], s["times"]
    H, M, S, _ = p.shape
    n = off[1:] - off[:-1]
    module = torch.repeat_interleave(torch.arange(M, device=p.device), n)
    mu = p[..., 0].sum(2)
    out = torch.where(n > 0, n * torch.log(mu) - mu - torch.lgamma(n.double() + 1.0), -mu)
    for h in range(H):
        for at in range(0, len(module), 4096):
            k = module[at:at + 4096]
            a, w, a1, a2, th, shift = p[h, k].unbind(2)
            y = x[at:at + 4096, None] - shift
            ok = y > 0
            y = torch.where(ok, y, torch.ones_like(y))
            lq = torch.log(a / mu[h, k][:, None]) - y / th

            def term(f, al):
                v = lq + torch.log(f) - torch.lgamma(al) - al * torch.log(th) + (al - 1) * torch.log(y)
                return torch.where(ok & (f > 0) & (al > 0), v, torch.full_like(v, -math.inf))

            lf = torch.logsumexp(torch.cat([term(w, a1), term(1 - w, a2)], 1), 1)
            out[h].index_add_(0, k, lf)
    return out


def _exact_lightyield(s):
    c = s["case"]
    q = s["parts"].cpu().numpy().view(_lib.PARTICLE_DTYPE)
    mid = 0.1 * (np.arange(c["intervals"]) + 0.5)
    src = np.zeros((len(q), c["intervals"], 12))
    src[..., 0:3] = q["pos"].astype(np.float64)[:, None, :] + mid[None, :, None] * q["dir"].astype(np.float64)[:, None]
    src[..., 3] = q["time"].astype(np.float64)[:, None] + mid[None, :] / C_VAC
    src[..., 4:7] = q["dir"].astype(np.float64)[:, None, :]
    return {"sources": src.reshape(-1, 12), "photons": None, "pairs": None}
