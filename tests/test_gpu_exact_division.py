"""The f64 collision's multiplication form of its divisions: bit-identical to
the oracle's divisions for ordinary populations at many tau, and for cells and
forces outside the range it is used in (negative, zero, tiny, huge, infinite
and NaN populations), which take the dividing path."""

from __future__ import annotations

import numpy as np
import pytest

from lattice_boltzmann_d3q19_b200 import reference as R

pytestmark = pytest.mark.gpu


def _same(a, b):
    """Equal values, zeros of equal sign, NaN where the other has NaN."""
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and a[~nan].tobytes() == b[~nan].tobytes()


@pytest.mark.parametrize("tau", [0.5000000001, 0.51, 0.56, 2.0 / 3.0, 0.7, 0.75, 1.0, 1.7, 1.9999999999999998, 97.3,
                                 1048576.0, 3e6, 1e300])
@pytest.mark.parametrize("forced", [False, True])
def test_ordinary_populations_bit_exact(oracle_mod, tau, forced):
    O = oracle_mod
    shape = (24, 17, 29)
    rng = np.random.default_rng(int(tau * 1e6) % 2**31)
    f = O.feq_field(1.0 + 0.1 * rng.standard_normal(shape), 0.1 * rng.standard_normal((3, *shape)))
    f *= 1.0 + 0.05 * rng.standard_normal(f.shape)
    F = 1e-4 * rng.standard_normal((3, *shape)) if forced else None
    if forced:
        F[:, :, ::3] = 0.0
        F[1, :, ::5] = -0.0
    assert _same(R.bgk_step(f, tau, F), O.bgk_step(f, tau, F))


@pytest.mark.parametrize("forced", [False, True])
def test_cells_outside_the_range_bit_exact(oracle_mod, forced):
    O = oracle_mod
    shape = (16, 12, 20)
    rng = np.random.default_rng(9)
    f = O.feq_field(1.0 + 0.01 * rng.standard_normal(shape), 0.02 * rng.standard_normal((3, *shape)))
    odd = [0.0, -0.0, -1e-3, 5e-324, 1e-320, -1e-310, 2.0**-301, 2.0**-300, 1e-91, 2.0**99, 2.0**100, 1e31, -1e200,
           1e308, np.inf, -np.inf, np.nan]
    flat = f.reshape(19, -1)
    for k, v in enumerate(odd):  # one odd direction; a few; every direction of a cell
        flat[(3 * k) % 19, 10 * k] = v
        flat[rng.integers(0, 19, 5), 10 * k + 400] = v
        flat[:, 10 * k + 1000] = v
    F = None
    if forced:
        F = 1e-5 * rng.standard_normal((3, *shape))
        Ff = F.reshape(3, -1)
        for k, v in enumerate(odd):
            Ff[k % 3, 10 * k + 2000] = v
    with np.errstate(all="ignore"):
        for tau in (0.56, 0.7):
            assert _same(R.bgk_step(f, tau, F), O.bgk_step(f, tau, F))
            wall = ((0.05, 0.0, -0.01), (0.0, 0.0, 0.0))
            assert _same(R.apply_bounce_back_y_walls(f, *wall), O.apply_bounce_back_y_walls(f, *wall))
