"""GPU test of pairs inside the softening length whose separation has a square
that FP32 cannot hold, or holds as a subnormal number: the spline's inner terms,
m d (32/3) / h^3 and -2.8 m / h, not the bound that the near loop starts from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FAC = 10.666666666667


def _pair(d):
    u = np.array([0.36, -0.48, 0.8])
    return {"pos": np.array([0.0 * u, d * u]), "vel": np.zeros((2, 3)), "mass": np.array([0.25, 0.75])}, u


@pytest.mark.parametrize("pot", [False, True])
@pytest.mark.parametrize("d", [1e-30, 1e-25, 1.6e-23, 4e-23, 1e-19, 1e-10])
@pytest.mark.parametrize("h", [1e-3, 1.0])
def test_two_particles(nb, h, d, pot):
    """FP32 terms: relative 1e-5."""
    data, u = _pair(d)
    sim = nb.Simulation(data, ForceSofteningTable=[h] * 6, TimeStep=1e-3)
    nb.compute_force(sim, want_potential=pot)
    g = nb.get_all_data(sim)
    want = np.stack([0.75 * d * u, -0.25 * d * u]) * FAC / h ** 3
    np.testing.assert_allclose(g["acc"], want, rtol=1e-5, atol=0)
    if pot:
        np.testing.assert_allclose(g["pot"], [-2.8 * 0.75 / h, -2.8 * 0.25 / h], rtol=1e-5, atol=0)


def test_engine(nb):
    """One engine step from rest: v = a dt / 2 after the half kicks."""
    h, d, dt = 1e-3, 1e-24, 1e-3
    data, u = _pair(d)
    eng = nb.Engine(max_particles=64, max_systems=1)
    i = eng.submit(data, h, dt, 1)
    eng.run_until_idle()
    got = eng.fetch(i, 2)
    a0 = np.stack([0.75 * d * u, -0.25 * d * u]) * FAC / h ** 3
    v, x = 0.5 * dt * a0, data["pos"].copy()
    x = x + v * dt
    s = x[1] - x[0]
    a1 = np.stack([0.75 * s, -0.25 * s]) * FAC / h ** 3
    np.testing.assert_allclose(got["pos"], x, rtol=1e-5, atol=1e-5 * d)
    np.testing.assert_allclose(got["vel"], v + a1 * dt - 0.5 * dt * a1, rtol=2e-4, atol=0)
