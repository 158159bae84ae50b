"""The FP64 special functions of the mixture fit and the event likelihood against extended precision, to the bounds
that their comments state.  exp: the table's exp2 (1 ulp by CUDA's accuracy table), the last rounding (0.5), the
reduced argument, series and its rounding (below 0.06): 1.6 ulp.  ln: the table's entry and the remainder, 2e-16, and
ln 2's own rounding times the exponent with two roundings, 1.5 ulp.  psi and psi': the first terms that the series
leave out at x = 6 (9.7e-12, 2.1e-10) and a dozen roundings.  Reciprocal: the cube of 2^-20 and one rounding."""
import numpy as np
import pytest
from scipy import special

pytestmark = pytest.mark.gpu
LD = np.longdouble


def _eval(prop, op, x):
    return prop.device_eval(op, x)


def test_exp(propagator):
    rng = np.random.default_rng(1)
    step = np.log(2.0) / 32
    edge = (rng.integers(-32000, 32000, 4001) + 0.5) * step  # between two entries of the table
    x = np.concatenate([rng.uniform(-708, 708, 40_000), rng.normal(0, 1, 20_000), edge, np.nextafter(edge, 0),
                        [0.0, -0.0, 5e-324, -1e-300, 1e-17, -708.0, 708.0]])
    x = np.clip(x, -708, 708)
    got, want = _eval(propagator, 13, x)[:, 0], np.exp(x.astype(LD))
    err = np.abs(got.astype(LD) - want) / np.spacing(want.astype(np.float64))
    assert err.max() <= 1.6, (x[err.argmax()], float(err.max()))
    ends = _eval(propagator, 13, np.array([-1e4, -np.inf, -709.0, 709.0, 1e300, np.inf]))[:, 0]
    np.testing.assert_allclose(ends, np.exp([-708.0] * 3 + [708.0] * 3), rtol=1e-3)
    print("exp_tab: max error", float(err.max()), "ulp")


@pytest.mark.parametrize("n", [1, 31, 33, 200])
def test_exp_of_a_part_of_a_warp(propagator, n):
    x = np.linspace(-3.0, 3.0, n)
    np.testing.assert_allclose(_eval(propagator, 13, x)[:, 0], np.exp(x), rtol=5e-16)


def test_log(propagator):
    rng = np.random.default_rng(2)
    edge = (1 + np.arange(32) / 32.0)[:, None] * 2.0 ** rng.integers(-1000, 1000, (32, 50))
    edge = np.concatenate([edge.ravel(), (1 + np.arange(32) / 32.0)])
    x = np.concatenate([10.0 ** rng.uniform(-307, 308, 40_000), rng.uniform(0.5, 2.0, 20_000), edge,
                        np.nextafter(edge, 0), np.nextafter(edge, 1e309), 1 + rng.normal(0, 1e-9, 1000),
                        [2.2250738585072014e-308, 1.7976931348623157e308]])
    x = np.maximum(x, 2.2250738585072014e-308)
    got, want = _eval(propagator, 14, x)[:, 0], np.log(x.astype(LD))
    err = np.abs(got.astype(LD) - want)
    over = err - LD(2e-16) - 1.5 * np.spacing(np.abs(want).astype(np.float64))
    assert over.max() <= 0, (x[over.argmax()], float(err[over.argmax()]))
    print("log_tab: max error in [0.5, 2]", float(err[(x >= 0.5) & (x <= 2)].max()), "beyond, in ulp",
          float((err / np.spacing(np.abs(want).astype(np.float64)))[(x < 0.5) | (x > 2)].max()))


def test_psi(propagator):
    rng = np.random.default_rng(3)
    x = np.concatenate([10.0 ** rng.uniform(-3, 6, 20_000), rng.uniform(0.02, 12.0, 20_000),
                        [1e-3, 1.0, 1.4616321449683622, 2.0, np.nextafter(6.0, 0), 6.0, np.nextafter(6.0, 9)]])
    got, psi, psi1 = _eval(propagator, 15, x), special.digamma(x), special.polygamma(1, x)
    e0, e1 = np.abs(got[:, 0] - psi), np.abs(got[:, 1] - psi1)
    assert (e0 <= 1e-11 + 4e-15 * np.abs(psi)).all(), (x[e0.argmax()], e0.max())
    assert (e1 <= 3e-10 + 8e-15 * psi1).all(), (x[e1.argmax()], e1.max())
    print("psi_both: max error for x >= 0.1", e0[x >= 0.1].max(), e1[x >= 0.1].max())


def test_reciprocal(propagator):
    rng = np.random.default_rng(4)
    x = np.concatenate([rng.uniform(1, 2, 40_000), 1 + 2.0 ** -rng.uniform(1, 52, 4000), [1.0, 2.0],
                        np.nextafter([1.0, 2.0], [2.0, 1.0])])
    got, want = _eval(propagator, 16, x)[:, 0], 1 / x.astype(LD)
    err = np.abs(got.astype(LD) - want) / np.spacing(np.minimum(want, np.nextafter(1.0, 0)).astype(np.float64))
    assert err.max() <= 1.0, (x[err.argmax()], float(err.max()))
    print("reciprocal_1_2: max error", float(err.max()), "ulp")
