"""The fit stage's moments over angle counts around a warp's 32, 64 and 128 and record counts around a run's 32, with
residuals of either sign, zero weights, refractive indices outside the table and angles that are not numbers, against
the FP64 restatement (the tolerances of test_gpu_fit.py: moments 2e-4, fits from the same moments 1e-9)."""
import numpy as np
import pandas as pd
import pytest

from photonprop_b200 import modelling as md
from oracle import fits as OF

pytestmark = pytest.mark.gpu


def _table(rng, n):
    return pd.DataFrame({"tres": rng.gamma(1.5, 20.0, n) * np.where(rng.uniform(size=n) < 0.9, 1.0, -1.0),
                         "initial_theta": rng.uniform(0.0, np.pi, n), "ref_ix": rng.uniform(1.33, 1.39, n),
                         "abs_weight": rng.uniform(0.0, 1.0, n) * (rng.uniform(size=n) < 0.95),
                         "wavelength": rng.uniform(300.0, 600.0, n)})


def _pmt(propagator, wl):
    return propagator.device_eval(10, np.asarray(wl))[:, 0]


@pytest.mark.parametrize("n_angles", [1, 31, 32, 33, 64, 65, 129, 600])
@pytest.mark.parametrize("n", [1, 33, 40_000])
def test_moments_at_edges(propagator, n_angles, n):
    rng = np.random.default_rng(n + n_angles)
    df = _table(rng, n)
    df.loc[0, ["tres", "abs_weight"]] = 12.5, 0.5
    angles = np.linspace(0.0, np.pi, n_angles)
    got = md.fit_photon_dist(angles, df, 10_000, propagator=propagator)
    some = rng.permutation(n_angles)[:7]
    want, mom = OF.fit_photon_dist(angles[some], df["tres"].to_numpy(), df["initial_theta"].to_numpy(),
                                   df["ref_ix"].to_numpy(), df["abs_weight"].to_numpy(),
                                   _pmt(propagator, df["wavelength"]), 10_000)
    np.testing.assert_allclose(got["det_fraction"].to_numpy()[some], want[:, 3], rtol=2e-4)
    if n > 1000:
        np.testing.assert_allclose(got["fit_alpha"].to_numpy()[some], want[:, 1], rtol=2e-3)
        np.testing.assert_allclose(got["fit_theta"].to_numpy()[some], want[:, 2], rtol=2e-3)


def test_rows_that_are_not_numbers(propagator):
    """An index outside 1.1-1.5 has no normalisation (NaN, as the reference's BoundsError), an angle that is not a
    number no weight: the row makes the sums NaN.  A table without light has no fit."""
    rng = np.random.default_rng(1)
    for col, value in (("ref_ix", 1.7), ("initial_theta", np.nan), ("abs_weight", np.nan)):
        df = _table(rng, 100)
        df.loc[50, col] = value
        assert np.all(np.isnan(md.fit_photon_dist([0.3, 1.0], df, 1000, propagator=propagator)["det_fraction"]))
    df = _table(rng, 100)
    df["abs_weight"] = 0.0
    out = md.fit_photon_dist([0.3, 1.0], df, 1000, propagator=propagator)
    assert np.all(out["det_fraction"] == 0.0) and np.all(np.isnan(out["fit_alpha"]))


def test_negative_and_tiny_weights_keep_their_sign_and_size(propagator):
    rng = np.random.default_rng(2)
    df = _table(rng, 500)
    a = md.fit_photon_dist([0.7], df, 1, propagator=propagator)["det_fraction"][0]
    for f in (-1.0, 1e-36):
        d2 = df.copy()
        d2["abs_weight"] *= f
        b = md.fit_photon_dist([0.7], d2, 1, propagator=propagator)["det_fraction"][0]
        assert b == pytest.approx(f * a, rel=1e-5)
