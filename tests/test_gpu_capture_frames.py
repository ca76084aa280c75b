"""Captured frames that go to the host in groups equal, bit for bit, those read
back one by one, where a run fills the buffer exactly, partly, several times,
or not at all (frames too large to be grouped)."""

from __future__ import annotations

import numpy as np
import pytest
from gpu_cases import random_state

from lattice_boltzmann_d3q19_b200 import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("shape,steps,every", [((5, 4, 3), 7, 1), ((9, 6, 8), 11, 4), ((61, 40, 20), 70, 1),
                                               ((64, 64, 24), 16, 1), ((64, 64, 24), 15, 1), ((96, 96, 90), 2, 1)])
def test_frames_match_single_readbacks(storage, shape, steps, every):
    f0 = random_state(shape, 8, amp=0.01)
    with Lattice(shape, 0.7, storage=storage, periodic=(True, False, True), wall_velocity={"y+": (0.05, 0.0, 0.0)}) as lat:
        for _ in range(2):  # the second capture finds the buffer there
            lat.set_populations(f0)
            at, rho, u = lat.run_capture(steps, every)
            f_end = lat.get_populations()
        lat.set_populations(f0)
        done = 0
        for k, s in enumerate(at):
            for _ in range(int(s) - done):
                lat.run_capture(1, 1)  # the kernels a capture steps with
            done = int(s)
            r, v = lat.rho_u()
            assert r.tobytes() == rho[k].tobytes() and v.tobytes() == u[k].tobytes(), (k, s)
        assert np.array_equal(lat.get_populations(), f_end)
