"""GPU test of the Morton order: the permutation that a step leaves (read from its
checkpoint image) against numpy's stable sort of the same keys, at the sizes
where the cluster sort changes its shape and where the chain of kernels takes
over, with coincident particles (ties) and with a plane (a flat box)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spread(v):
    v = v.astype(np.uint64)
    out = np.zeros_like(v)
    for b in range(21):
        out |= ((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return out


def _order(pos):
    key = np.zeros(len(pos), dtype=np.uint64)
    for k in range(3):
        p = pos[:, k]
        lo, hi = p.min(), p.max()
        f = np.clip((p - lo) / (hi - lo), 0.0, 1.0) if hi > lo else np.zeros_like(p)
        key |= _spread((f * 2097151.0).astype(np.uint64)) << np.uint64(k)
    return np.argsort(key, kind="stable")


@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1025, 8192, 8193, 16385, 32769, 65537, 131072, 131073])
@pytest.mark.parametrize("kind", ["sphere", "ties", "plane"])
def test_order_is_the_stable_sort(nb, n, kind):
    rng = np.random.default_rng(n)
    pos = rng.normal(0.0, 1.0, (n, 3))
    if kind == "ties":
        pos = np.round(pos, 1)
    if kind == "plane":
        pos[:, 1] = 0.25
    d = {"pos": pos, "vel": np.zeros((n, 3)), "mass": np.full(n, 1.0 / n)}
    sim = nb.Simulation(d, ForceSofteningTable=[0.05] * 6, TimeStep=1e-6, TimeEnd=1.0, resort_every=1)
    nb.step(sim, 1)
    pos = nb.get_all_data(sim)["pos"]
    image = sim.checkpoint()
    perm = np.frombuffer(image, dtype=np.int32, offset=len(image) - (4 * n + 7) // 8 * 8)[:n]
    np.testing.assert_array_equal(perm, _order(pos))
