"""Tapes that take over the device memory of earlier ones on their lattice
give the bits of a fresh lattice's tape, and the special-cell list is whole
where its scan spans several chunks."""

from __future__ import annotations

import numpy as np
import pytest
import torch
from adjoint_cases import case, gpu_lattice
from test_gpu_adjoint import rel_err, tape_grads, torch_grads

from lattice_boltzmann_d3q19_b200 import _native as N

pytestmark = pytest.mark.gpu


def _backward(lat, tape):
    shape = lat.shape
    gr = torch.full(shape, 0.25, dtype=torch.float64, device="cuda")
    gu = torch.linspace(-1.0, 1.0, 3 * lat.n, dtype=torch.float64, device="cuda")
    ga = torch.empty(shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tape.backward(gr.data_ptr(), gu.data_ptr(), ga.data_ptr())
    lat.synchronize()
    return ga.cpu().numpy()


def test_tapes_in_succession_match_fresh_ones():
    c = case("drag_channel")
    # the same size (reused), a larger tape, a much smaller one, a larger again
    runs = [(20, 5), (20, 5), (40, 4), (3, 1), (20, 5)]

    def fresh(steps, every):
        with gpu_lattice(c, "f32") as lat:
            lat.set_populations(c["f0"])
            with lat.tape(steps, every) as t:
                return _backward(lat, t)

    want = [fresh(*r) for r in runs]
    lat = gpu_lattice(c, "f32")
    for run, w in zip(runs, want, strict=True):
        lat.set_populations(c["f0"])
        with lat.tape(*run) as t:
            assert _backward(lat, t).tobytes() == w.tobytes()
    # two tapes alive at once, destroyed in either order, one after its lattice
    lat.set_populations(c["f0"])
    a = lat.tape(20, 5)
    lat.set_populations(c["f0"])
    b = lat.tape(40, 4)
    assert _backward(lat, a).tobytes() == want[0].tobytes()
    assert _backward(lat, b).tobytes() == want[2].tobytes()
    a.close()
    N.check(N.lib().lbm_release_workspace())
    lat.close()
    b.close()


def test_gradient_where_the_list_spans_scan_chunks():
    # 1,089,792 cells: 1065 counting blocks, two chunks of the scan
    c = case("drag_channel", shape=(1032, 33, 32))
    _, ga, gf = tape_grads(c, 2, 2)
    _, gat, gft = torch_grads(c, 2)
    assert np.abs(gat).max() > 0
    assert rel_err(ga, gat) < 1e-9 and rel_err(gf, gft) < 1e-9
