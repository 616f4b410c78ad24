"""GPU test of the FP64 form's pair terms: the field of a single source is one
term, and has to be the double that the same expression gives on the CPU, bit
for bit (IEEE products, root and quotient).  Squared distances next to a square's
midpoint (1 + k units in the last place), over the exponent range, and masses
whose quotients are small, subnormal or large."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(how):
    r = np.random.default_rng(7)
    n = 1 << 16
    if how == "midpoints":
        # dx = 1, dy^2 ~ k 2^-52: r^2 = 1 + k ulp, whose root lies next to a midpoint for odd k
        k = np.arange(1, n + 1, dtype=np.float64)
        return np.stack([np.ones(n), np.sqrt(k) * 2.0 ** -26, np.zeros(n)], 1)
    if how == "ordinary":
        return r.normal(0.0, 1.0, (n, 3))
    return r.normal(0.0, 1.0, (n, 3)) * 2.0 ** r.integers(-150, 150, (n, 1)).astype(np.float64)


def _terms(q, m, h, law):
    """The reference's expressions for a source at the origin, in their order."""
    d = 0.0 - q
    r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
    if law == "plummer":
        x = r2 + h * h
        fac, pot = m / (x * np.sqrt(x)), -m / np.sqrt(x)
    else:
        r, hi = np.sqrt(r2), 1.0 / h
        h3, u = hi * hi * hi, np.sqrt(r2) * hi
        near = m * h3 * (10.666666666667 + u * u * (32.0 * u - 38.4))
        mid = m * h3 * (21.333333333333 - 48.0 * u + 38.4 * (u * u) - 10.666666666667 * (u * u * u)
                        - 0.066666666667 / (u * u * u))
        fac = np.where(r >= h, m / (r2 * r), np.where(u < 0.5, near, mid))
        pn = m * hi * (-2.8 + u * u * (5.333333333333 + u * u * (6.4 * u - 9.6)))
        pm = m * hi * (-3.2 + 0.066666666667 / u
                       + u * u * (10.666666666667 + u * (-16.0 + u * (9.6 - 2.133333333333 * u))))
        pot = np.where(r >= h, -m / r, np.where(u < 0.5, pn, pm))
    return d * fac[:, None], pot


@pytest.mark.parametrize("law", ["spline", "plummer"])
@pytest.mark.parametrize("m", [1.0, 1.0 / 3.0, 3e-294, 7e-300, 2.0 ** -1060, 1.7e300])
@pytest.mark.parametrize("how", ["midpoints", "ordinary", "exponents"])
def test_terms_are_the_cpu_ones(nb, how, m, law):
    q, h = _points(how), 0.5 if how == "ordinary" else 1e-60
    d = {"pos": np.zeros((1, 3)), "vel": np.zeros((1, 3)), "mass": np.array([m])}
    sim = nb.Simulation(d, ForceSofteningTable=[h] * 6, TimeStep=1e-3, precision="fp64", law=law)
    acc, pot = nb.force_and_potential_at_points(sim, q, h)
    with np.errstate(all="ignore"):
        want, wpot = _terms(q, m, h, law)
    # a compensated sum turns an overflowed term into NaN
    want[~np.isfinite(want)] = np.nan
    wpot[~np.isfinite(wpot)] = np.nan
    np.testing.assert_array_equal(acc, want)
    np.testing.assert_array_equal(pot, wpot)
