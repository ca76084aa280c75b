"""The f64 readback kernel of the reduced storages: rho and u equal, bit for
bit, to those of the state's populations summed in the engine's order by the
step kernel's own readback (run_capture), for one, two and four cells per
thread, and for output arrays that only one cell per thread can write."""

from __future__ import annotations

import numpy as np
import pytest
import torch
from gpu_cases import random_state

from lattice_boltzmann_d3q19_b200 import Lattice

pytestmark = pytest.mark.gpu


def _flags(shape, seed):
    rng = np.random.default_rng(seed)
    flags = (rng.random(shape) < 0.05).astype(np.uint8)
    flags[0], flags[-1] = 2, 3
    return flags


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("shape", [(7, 5, 4), (6, 4, 8), (5, 3, 6), (9, 6, 130), (4, 7, 9), (3, 1, 1), (5, 4, 132)])
@pytest.mark.parametrize("kind", ["flags", "walls", "drag"])
def test_readback_matches_the_step_kernels(storage, shape, kind):
    kw = {"flags": dict(inflow_u=(0.04, 0.0, 0.0)),
          "walls": dict(periodic=(False, False, False), wall_velocity={"y+": (0.05, 0.0, 0.0), "z-": (0.0, 0.01, 0.0)}),
          "drag": dict(force_mode="drag", drag_k=0.05, body_force=(1e-5, 0.0, 0.0))}[kind]
    with Lattice(shape, 0.7, storage=storage, **kw) as lat:
        if kind == "flags":
            lat.set_flags(_flags(shape, 4))
        if kind == "drag":
            lat.set_porosity(np.random.default_rng(2).random(shape).astype(np.float32))
        lat.set_populations(random_state(shape, 3, amp=0.02))
        n = lat.n
        for pre in (True, False):
            if not pre:
                lat.step(4)
            got = lat.rho_u()
            for shift in (0, 1):  # 16-byte aligned device arrays, and arrays 8 bytes off
                rho = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
                u = torch.zeros(3 * n + 2, dtype=torch.float64, device="cuda")
                torch.cuda.synchronize()
                lat.rho_u_device(rho[shift:].data_ptr(), u[shift:].data_ptr())
                lat.synchronize()
                assert rho[shift:shift + n].cpu().numpy().tobytes() == got[0].tobytes()
                assert u[shift:shift + 3 * n].cpu().numpy().tobytes() == got[1].tobytes()
                assert float(rho[n + 1 if shift == 0 else 0]) == 0.0 and float(u[3 * n + 1 if shift == 0 else 0]) == 0.0
            only = torch.zeros(n, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            lat.rho_u_device(only.data_ptr(), None)
            lat.synchronize()
            assert only.cpu().numpy().tobytes() == got[0].tobytes()
            if not pre:  # the step kernel reads back the state it advances from
                _, rho_f, u_f = lat.run_capture(1, 1)
                assert rho_f[0].tobytes() == got[0].tobytes() and u_f[0].tobytes() == got[1].tobytes()
