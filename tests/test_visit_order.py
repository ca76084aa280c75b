"""The computed visit order of walled lattices (FaceFirst): every item once,
items on walled faces apart from the others, checked on the CPU by the header's
own code; on a GPU, lattices beyond the size from which it is used give the
bits of plane windows, which are stepped in order."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from helpers import same_bytes

CSRC = Path(__file__).resolve().parents[1] / "bit-physics_b200" / "csrc"

# Exit status 0, or a message: for every size up to 7 and every set of walled
# axes, item() is a permutation, x-face items come first, then y-face items,
# and within each plane z-face items before the others.
PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "lbm_device.cuh"
int main()
{
    for (int nx = 1; nx <= 7; ++nx)
        for (int ny = 1; ny <= 7; ++ny)
            for (int nz = 1; nz <= 7; ++nz)
                for (unsigned w = 0; w < 8; ++w) {
                    const unsigned walled[3] = {w & 1u, (w >> 1) & 1u, (w >> 2) & 1u};
                    lbm::FaceFirst F;
                    F.init(nx, ny, nz, walled);
                    const int n = nx * ny * nz;
                    std::vector<int> seen(n, 0);
                    int last = -1;
                    for (int t = 0; t < n; ++t) {
                        const int i = F.item(t);
                        if (i < 0 || i >= n || seen[i]++) return printf("item %d of %dx%dx%d, walls %u: %d\n", t, nx, ny, nz, w, i);
                        const int x = i / (ny * nz), y = i / nz % ny, z = i % nz;
                        const bool fx = walled[0] && (x == 0 || x == nx - 1), fy = walled[1] && (y == 0 || y == ny - 1),
                                   fz = walled[2] && (z == 0 || z == nz - 1);
                        const int at = fx ? 0 : fy ? 1 : 2 + 2 * x + (fz ? 0 : 1);
                        if (at < last) return printf("order of item %d of %dx%dx%d, walls %u\n", t, nx, ny, nz, w);
                        last = at;
                    }
                }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_every_item_once(tmp_path):
    src, exe = tmp_path / "order.cu", tmp_path / "order"
    src.write_text(PROGRAM)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", f"-I{CSRC}",
                    f"-I{CSRC.parents[1] / 'include'}", "-o", str(exe), str(src)], check=True, capture_output=True)
    got = subprocess.run([str(exe)], capture_output=True, text=True)
    assert got.returncode == 0, got.stdout


WALLS = {"x-": (0.01, 0.0, 0.02), "y+": (0.05, 0.0, 0.0), "z-": (0.0, 0.03, 0.0), "z+": (-0.02, 0.0, 0.0)}
X, Y, XY, Z = (False, True, True), (True, False, True), (False, False, True), (True, True, False)
SIX = (False, False, False)


@pytest.mark.gpu
@pytest.mark.parametrize("storage,shape,walls", [
    ("f64", (70, 72, 70), [X, Y, XY]), ("f64", (2, 300, 600), [X, Y, XY]), ("f64", (1, 601, 600), [X, XY]),
    ("f64", (500, 1, 702), [Y, XY]), ("f64", (400, 2, 450), [Y, XY]),
    ("f32", (90, 91, 90), [X, Y, XY]), ("f32", (2, 300, 1200), [X, XY]), ("f32", (1, 900, 802), [X, XY]),
    ("f32", (300, 2, 1202), [Y, XY]), ("f32", (901, 1, 802), [Y, XY]), ("f32", (600, 600, 2), [X, Y, XY]),
    ("f16", (118, 113, 110), [X, Y, Z, XY, SIX]), ("f16", (30, 24001, 2), [Z, SIX]), ("bf16", (1, 1400, 1002), [Z, SIX]),
    ("bf16", (1400, 1, 1002), [Z, SIX]), ("f16", (2, 702, 1002), [X, SIX]), ("f16", (1002, 2, 702), [Y, SIX])])
def test_beyond_l2_leaves_the_bits(storage, shape, walls):
    from gpu_cases import random_state
    from lattice_boltzmann_d3q19_b200 import Lattice

    n = shape[0] * shape[1] * shape[2]
    # the sizes from which the order is computed instead of listed
    assert 2 * 19 * {"f64": 8, "f32": 4}.get(storage, 2) * n > 100 << 20
    f0 = random_state(shape, 5, amp=0.01)
    for periodic in walls:
        with Lattice(shape, 0.7, storage=storage, periodic=periodic, wall_velocity=WALLS) as lat:
            lat.set_populations(f0)
            lat.step(4)
            f = lat.get_populations()
            lat.set_populations(f0)
            lat.step(1)
            for _ in range(3):
                lat.step_planes(0, shape[0])
                lat.step_commit()
            assert same_bytes(lat.get_populations(), f), periodic
