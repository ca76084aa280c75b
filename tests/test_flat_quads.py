"""Quads of the flat cell array (16-bit storage, rows of odd length): the index
arithmetic of the four-cell step on the CPU, and the step itself on a GPU
against the one-cell kernel and the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from lattice_boltzmann_d3q19_b200 import VELOCITIES

FAST_TOL = {"f16": 2e-4, "bf16": 2e-3}


@pytest.mark.parametrize("shape", [(3, 7, 5), (1, 6, 5), (2, 5, 7), (4, 9, 6), (3, 8, 9), (2, 3, 13), (1, 1, 5),
                                   (1, 2, 9), (6, 1, 5), (3, 5, 75), (2, 7, 10), (2, 11, 31)])
def test_quad_sources(shape):
    """k_step4_flat's loads restated: the aligned groups hold each cell's pull
    source, edge values replace the wrapped ones, and nothing lies outside
    the buffer."""
    nx, ny, nz = shape
    n, nynz = nx * ny * nz, ny * nz
    stride = (n + 3) // 4 * 4
    elements = 19 * stride + 32
    for i0 in range(0, n - 3, 4):
        x, y, z0 = i0 // nynz, i0 // nz % ny, i0 % nz
        if z0 + 3 >= nz and (y < 1 or y > ny - 3):
            continue  # a rule quad
        X = [(x - 1) % nx * nynz, x * nynz, (x + 1) % nx * nynz]
        Y = [(y - 1) % ny * nz, y * nz, (y + 1) % ny * nz]
        je = nz - 1 - z0
        jz = 0 if z0 == 0 else (je + 1 if je < 3 else 4)
        for d, (cx, cy, cz) in enumerate(VELOCITIES):
            p = X[1 - cx] + Y[1 - cy] + z0 - cz
            hi, a = p & 2, p & ~3
            ra, rb = list(range(a + 2 * hi, a + 2 * hi + 4)), [a + 4 - hi, a + 5 - hi]
            assert all(0 <= d * stride + e < elements for e in ra + rb)
            v = (rb + ra if hi else ra + rb)[p & 1:][:4]
            if cz == 1 and jz < 4:
                v[jz] = p + jz + nz
            if cz == -1 and je < 4:
                v[je] = p + je - nz
            for k in range(4):
                i = i0 + k
                xs, ys, zs = (i // nynz - cx) % nx, (i // nz % ny - cy) % ny, (i % nz - cz) % nz
                assert v[k] == (xs * ny + ys) * nz + zs


def _lattices():
    """(name, Lattice arguments, flags, setup arguments) with odd nz,
    large enough (and with few enough rule cells) to step in flat quads:
    rows of 5 cells up, one row or one plane per axis, n % 4 = 0 .. 3, quads
    that straddle planes."""
    rng = np.random.default_rng(5)
    out = []
    for shape in [(301, 141, 5), (260, 111, 7), (131, 11, 145), (1, 1501, 151), (1500, 1, 151), (5, 2, 21001),
                  (40, 53, 101)]:
        flags = (rng.random(shape) < 0.001).astype(np.uint8)
        if shape[0] > 4:
            flags[0], flags[-1] = 2, 3
        out.append((f"spheres {shape}", dict(shape=shape, tau=0.6, inflow_u=(0.04, 0.0, 0.0)), flags, {}))
        walls = {"y+": (0.05, 0.0, 0.0), "x-": (0.0, 0.01, 0.0), "z-": (0.0, 0.02, 0.0)}
        for periodic in [(True, True, True), (False, False, False), (True, False, True), (True, True, False)]:
            out.append((f"walls {shape} {periodic}",
                        dict(shape=shape, tau=0.7, periodic=periodic, wall_velocity=walls), None, {}))
    for shape in [(40, 53, 101), (39, 53, 103)]:
        few = (rng.random(shape) < 0.001).astype(np.uint8)
        out.append((f"field {shape}", dict(shape=shape, tau=0.8, force_mode="field"), few,
                    dict(force=1e-4 * rng.standard_normal((3, *shape)))))
        out.append((f"drag {shape}", dict(shape=shape, tau=0.7, force_mode="drag", drag_k=0.05,
                                          body_force=(1e-6, 0.0, 0.0)), few,
                    dict(porosity=rng.random(shape).astype(np.float32))))
        out.append((f"uniform {shape}", dict(shape=shape, tau=0.7, force_mode="uniform",
                                             body_force=(1e-5, 0.0, 2e-6)), None, {}))
    return out


def _make(kw, flags, setup, storage, **more):
    from lattice_boltzmann_d3q19_b200 import Lattice

    kw = dict(kw)
    lat = Lattice(kw.pop("shape"), kw.pop("tau"), storage=storage, **kw, **more)
    if flags is not None:
        lat.set_flags(flags)
    if "force" in setup:
        lat.set_force_field(setup["force"])
    if "porosity" in setup:
        lat.set_porosity(setup["porosity"])
    return lat


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_flat_quads_match_the_one_cell_kernel(storage):
    """The bits of the one-cell kernel, whole and split into plane windows."""
    from gpu_cases import random_state

    for k, (name, kw, flags, setup) in enumerate(_lattices()):
        f0 = random_state(kw["shape"], 30 + k, amp=0.02)
        got = []
        for more in ({}, {"cells_per_thread": 1}):
            with _make(kw, flags, setup, storage, **more) as lat:
                lat.set_populations(f0)
                for n in (1, 2, 3):
                    lat.step(n)
                got.append(lat.get_populations())
        assert got[0].tobytes() == got[1].tobytes(), name
        nx = kw["shape"][0]
        if nx < 3:
            continue
        with _make(kw, flags, setup, storage) as lat:
            lat.set_populations(f0)
            lat.step(1)
            for _ in range(5):
                for x0, x1 in ((1, nx - 1), (0, 1), (nx - 1, nx)):
                    lat.step_planes(x0, x1)
                lat.step_commit()
            assert lat.get_populations().tobytes() == got[0].tobytes(), name


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["f16", "bf16"])
def test_flat_quads_against_oracle(storage):
    from gpu_cases import pair, random_state
    from lattice_boltzmann_d3q19_b200 import geometry

    shape = (80, 57, 63)
    flags, _ = geometry.sphere_channel(shape, n_spheres=6, radius=(2.0, 5.0), seed=3)
    for kw in (dict(flags=flags, inflow_u=(0.04, 0.0, 0.0)),
               dict(periodic=(False, False, False), wall_velocity={"y+": (0.05, 0.0, 0.0)})):
        gpu, cpu = pair(shape, 0.6, storage, **kw)
        f0 = random_state(shape, 8, amp=0.01)
        with gpu:
            gpu.set_populations(f0)
            cpu.set_populations(f0)
            gpu.step(15)
            cpu.step(15)
            assert float(np.max(np.abs(gpu.get_populations() - cpu.get_populations()))) <= FAST_TOL[storage]
