"""Gradients of the reduced storages under every force model (the plain-cell
kernel has two orders of its loads, chosen by storage and force model) against
the f64 tape of the same lattice."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_cases import random_state
from lattice_boltzmann_d3q19_b200 import Lattice

pytestmark = pytest.mark.gpu

SHAPE, STEPS = (24, 10, 12), 12
# Every step rounds a population of size w to 2^-24 (f32) of it, 2^-11 (f16) or 2^-8
# (bf16) of its deviation (a few per cent of it here), and the adjoint is linear in
# the state's velocities: STEPS such errors of one sign, ten times over for the
# maximum against the norm.
TOL = {"f32": 10 * STEPS * 2.0**-24, "f16": 10 * STEPS * 0.05 * 2.0**-11, "bf16": 10 * STEPS * 0.05 * 2.0**-8}


def _gradient(storage, force, periodic):
    rng = np.random.default_rng(3)
    flags = np.zeros(SHAPE, np.uint8)
    flags[6:8, 3:5, 4:7] = 1
    flags[0], flags[-1] = 2, 3
    kw = {"drag_k": 0.05} if force == "drag" else {"body_force": (1e-5, 0.0, 2e-6)} if force == "uniform" else {}
    with Lattice(SHAPE, 0.7, storage=storage, periodic=periodic, force_mode=force, inflow_u=(0.04, 0.0, 0.0),
                 wall_velocity={"y+": (0.05, 0.0, 0.0)} if not periodic[1] else None, **kw) as lat:
        lat.set_flags(flags)
        if force == "field":
            lat.set_force_field(1e-5 * rng.standard_normal((3, *SHAPE)))
        if force == "drag":
            lat.set_porosity(rng.random(SHAPE).astype(np.float32))
        lat.set_populations(random_state(SHAPE, 4, amp=0.02))
        gr = torch.from_numpy(np.random.default_rng(5).standard_normal(SHAPE)).cuda()
        gu = torch.from_numpy(np.random.default_rng(6).standard_normal((3, *SHAPE))).cuda()
        gf = torch.empty((19, *SHAPE), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        with lat.tape(STEPS, 5) as tape:
            tape.backward(gr.data_ptr(), gu.data_ptr(), None, gf.data_ptr())
            lat.synchronize()
        return gf.cpu().numpy()


@pytest.mark.parametrize("force", ["none", "uniform", "field", "drag"])
@pytest.mark.parametrize("periodic", [(True, True, True), (True, False, True)])
def test_reduced_storage_gradients(force, periodic):
    want = _gradient("f64", force, periodic)
    for storage, tol in TOL.items():
        err = np.abs(_gradient(storage, force, periodic) - want).max() / np.abs(want).max()
        assert err < tol, (storage, err, tol)
