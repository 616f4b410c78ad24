"""GPU test of a checkpoint image whose clock holds another word in the place that
the adaptive step counts its blocks in (unused in images): the restored run
takes the same steps."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TICKET_FROM_END = 12  # of the clock, before the int64 count of outputs


@pytest.mark.parametrize("word", [1, -1, 7])
def test_word_does_not_matter(nb, word):
    L = nb._lib
    lib = L.load()
    sim = nb.Simulation(nb.plummer(1000, seed=3), ForceSofteningTable=[0.01] * 6, TimeEnd=1.0, MaxStep=1e-2)
    nb.compute_force(sim)
    nb.init_timesteps(sim)
    nb.leapfrog_half_kick(sim, +1)
    nb.step(sim, 3)
    size = ctypes.c_int64()
    L.check(sim.handle, lib.nb_checkpoint_size(sim.handle, ctypes.byref(size)))
    img = ctypes.create_string_buffer(size.value)
    L.check(sim.handle, lib.nb_checkpoint_save(sim.handle, img, size))
    nb.step(sim, 6)
    want, t = nb.get_all_data(sim), sim.time()
    # magic[8], version, n, bytes, params_size, clock_size, params, between, order_steps, clock
    clock_size = ctypes.c_int64.from_buffer(img, 40).value
    at = 48 + ctypes.sizeof(L.nb_params) + 16 + clock_size - TICKET_FROM_END
    assert ctypes.c_int32.from_buffer(img, at).value == 0
    ctypes.c_int32.from_buffer(img, at).value = word
    L.check(sim.handle, lib.nb_checkpoint_load(sim.handle, img, size))
    nb.step(sim, 6)
    got = nb.get_all_data(sim)
    assert sim.time() == t
    for k in ("pos", "vel", "acc", "ti_begstep", "ti_endstep"):
        np.testing.assert_array_equal(got[k], want[k])
