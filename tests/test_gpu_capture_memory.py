"""The frame buffer of captures: one for the GPU and not one for each lattice
that has captured, given back on request, and safe with several threads."""

from __future__ import annotations

import gc
import threading

import numpy as np
import pytest
import torch
from gpu_cases import random_state

from lattice_boltzmann_d3q19_b200 import Lattice
from lattice_boltzmann_d3q19_b200 import _native as N

pytestmark = pytest.mark.gpu

SHAPE, STEPS, MB = (64, 32, 12), 64, 1 << 20  # f64: 51 MB of frames


def _free() -> int:
    gc.collect()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _capture(storage="f64", seed=1):
    lat = Lattice(SHAPE, 0.7, storage=storage, periodic=(True, False, True), wall_velocity={"y+": (0.05, 0.0, 0.0)})
    lat.set_populations(random_state(SHAPE, seed, amp=0.01))
    return lat, lat.run_capture(STEPS, 1)[1:]


def test_lattices_share_one_buffer():
    _capture("f32")[0].close()
    free = _free()
    lats = [_capture("f32" if k % 2 else "f64", k)[0] for k in range(10)]
    assert free - _free() < 200 * MB  # the lattices themselves: under 10 MB each
    for lat in lats:
        lat.close()
    N.check(N.lib().lbm_release_workspace())
    assert _free() > free + 40 * MB


def test_threads():
    want = [_capture("f64" if k % 2 else "f16", k)[1] for k in range(4)]
    got = [None] * 4

    def run(k):
        for _ in range(5):
            got[k] = _capture("f64" if k % 2 else "f16", k)[1]

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (r0, u0), (r1, u1) in zip(want, got, strict=True):
        assert np.array_equal(r0, r1) and np.array_equal(u0, u1)
