"""Walled lattices large enough to be stepped out of their natural order (face
items first, whole or plane by plane): the bits of the plane windows, which
are stepped in order, and of the oracle."""

from __future__ import annotations

import numpy as np
import pytest
from gpu_cases import pair, random_state
from helpers import same_bytes

from lattice_boltzmann_d3q19_b200 import Lattice

pytestmark = pytest.mark.gpu

WALLS = {"x-": (0.01, 0.0, 0.02), "y+": (0.05, 0.0, 0.0), "z-": (0.0, 0.03, 0.0), "z+": (-0.02, 0.0, 0.0)}
PERIODIC = [(False, False, False), (True, False, True), (True, True, False), (False, True, True), (False, True, False),
            (False, False, True)]


@pytest.mark.parametrize("storage,shape", [
    ("f64", (70, 50, 40)), ("f64", (2, 231, 301)), ("f64", (300, 1, 400)), ("f32", (41, 73, 80)),
    ("f32", (3, 2, 40000)), ("f16", (31, 55, 61)), ("bf16", (41, 73, 82)), ("f16", (60, 200, 122))])
def test_order_leaves_the_bits(storage, shape):
    f0 = random_state(shape, 5, amp=0.01)
    for periodic in PERIODIC:
        with Lattice(shape, 0.7, storage=storage, periodic=periodic, wall_velocity=WALLS) as lat:
            lat.set_populations(f0)
            lat.step(6)
            f = lat.get_populations()
            lat.set_populations(f0)
            lat.step(1)
            for _ in range(5):
                lat.step_planes(0, shape[0])
                lat.step_commit()
            assert same_bytes(lat.get_populations(), f), periodic


@pytest.mark.parametrize("periodic", PERIODIC[:3])
def test_f64_against_the_oracle(periodic):
    shape = (52, 47, 44)
    gpu, cpu = pair(shape, 0.63, periodic=periodic, wall_velocity=WALLS)
    f0 = random_state(shape, 6)
    with gpu:
        gpu.set_populations(f0)
        cpu.set_populations(f0)
        gpu.step(5)
        cpu.step(5)
        assert same_bytes(gpu.get_populations(), cpu.get_populations())
