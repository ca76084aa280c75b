"""Where f16 / bf16 lattices with an odd nz step in flat quads, and, with the
quads switched on, their bits against the one-cell kernel's for every force
model, boundary kind, row length and remainder of n by 4."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
from gpu_cases import random_state

from lattice_boltzmann_d3q19_b200 import Lattice
from lattice_boltzmann_d3q19_b200 import _native as N

pytestmark = pytest.mark.gpu

WALLS = {"y+": (0.05, 0.0, 0.0), "x-": (0.0, 0.01, 0.0), "z-": (0.0, 0.02, 0.0)}
OPEN, Y, SIX = (True, True, True), (True, False, True), (False, False, False)


def _flat(lat, mode=-1) -> bool:
    used = C.c_int32()
    N.check(N.lib().lbm_test_flat_quads(lat.handle, mode, C.byref(used)))
    return bool(used.value)


@pytest.mark.parametrize("shape,periodic,spheres,flat", [
    # slower in flat quads: 1.11x, 1.08x, 1.06x, 1.33x, 1.03x
    ((71, 71, 71), SIX, False, False), ((177, 16, 177), Y, False, False), ((209, 16, 209), SIX, False, False),
    ((333, 333, 9), SIX, False, False), ((471, 471, 9), SIX, False, False),
    # faster: 1.06x, 1.16x, 1.09x, 1.10x, 1.21x
    ((89, 89, 89), SIX, False, True), ((101, 101, 101), Y, False, True), ((250, 16, 251), Y, False, True),
    ((213, 40, 41), OPEN, True, True), ((127, 127, 127), OPEN, False, True)])
def test_used_where_faster(shape, periodic, spheres, flat):
    with Lattice(shape, 0.6, storage="f16", periodic=periodic, wall_velocity=WALLS) as lat:
        if spheres:
            flags = np.zeros(shape, np.uint8)
            flags[80:90, 10:20, 10:20] = 1
            flags[0], flags[-1] = 2, 3
            lat.set_flags(flags)
        assert _flat(lat) == flat


def test_refused_where_the_lattice_cannot():
    for kw in (dict(shape=(8, 8, 8), storage="f16"), dict(shape=(8, 8, 3), storage="f16"),
               dict(shape=(8, 8, 7), storage="f32"), dict(shape=(8, 8, 7), storage="bf16", cells_per_thread=1)):
        with Lattice(kw.pop("shape"), 0.6, **kw) as lat:
            assert not _flat(lat)
            assert N.lib().lbm_test_flat_quads(lat.handle, 1, None) == N.LBM_ERR_UNSUPPORTED


def _cases():
    rng = np.random.default_rng(8)
    shapes = [(9, 7, 5), (6, 11, 7), (5, 3, 9), (7, 5, 13), (1, 9, 7), (9, 1, 5), (2, 2, 11), (12, 10, 31)]
    assert {int(np.prod(s)) % 4 for s in shapes} == {0, 1, 2, 3}
    for shape in shapes:
        flags = (rng.random(shape) < 0.05).astype(np.uint8)
        if shape[0] > 4:
            flags[0], flags[-1] = 2, 3
        for force in ("none", "uniform", "field", "drag"):
            for periodic in (OPEN, Y, (True, True, False), SIX):
                for fl in (None, flags):
                    yield shape, force, periodic, fl


@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_bits_of_the_one_cell_kernel(storage):
    rng = np.random.default_rng(9)
    for shape, force, periodic, flags in _cases():
        f0 = random_state(shape, 11, amp=0.02)
        field = 1e-4 * rng.standard_normal((3, *shape))
        alpha = rng.random(shape).astype(np.float32)
        kw = {"drag_k": 0.05, "body_force": (1e-6, 0.0, 0.0)} if force == "drag" else \
            {"body_force": (1e-5, 0.0, 2e-6)} if force == "uniform" else {}
        got = []
        for mode in (0, 1):
            with Lattice(shape, 0.65, storage=storage, periodic=periodic, wall_velocity=WALLS, force_mode=force,
                         inflow_u=(0.04, 0.0, 0.0), **kw) as lat:
                if flags is not None:
                    lat.set_flags(flags)
                if force == "field":
                    lat.set_force_field(field)
                if force == "drag":
                    lat.set_porosity(alpha)
                assert _flat(lat, mode) == bool(mode)
                lat.set_populations(f0)
                lat.step(1)
                lat.step(4)
                got.append((lat.get_populations(), *lat.rho_u()))
        for a, b in zip(*got, strict=True):
            assert a.tobytes() == b.tobytes(), (shape, force, periodic, flags is not None)


def test_windows_of_planes():
    """Windows of any width (wide ones in flat quads, thin ones one cell per thread), in any
    order, give the bits of whole steps."""
    shape = (24, 11, 7)
    flags = (np.random.default_rng(2).random(shape) < 0.05).astype(np.uint8)
    f0 = random_state(shape, 12, amp=0.02)
    for windows in ([(0, 24)], [(0, 12), (12, 24)], [(1, 23), (0, 1), (23, 24)], [(0, 13), (13, 24)],
                    [(x, x + 1) for x in range(24)]):
        got = []
        for mode in (0, 1):
            with Lattice(shape, 0.65, storage="f16", periodic=Y, wall_velocity=WALLS) as lat:
                lat.set_flags(flags)
                _flat(lat, mode)
                lat.set_populations(f0)
                lat.step(1)
                for _ in range(4):
                    if mode == 0:
                        lat.step(1)
                        continue
                    for w in windows:
                        lat.step_planes(*w)
                    lat.step_commit()
                got.append(lat.get_populations())
        assert got[0].tobytes() == got[1].tobytes(), windows
