"""Whose memory a tape works in: a tape's own allocation is given back when it
is destroyed, autograd.run's comes from PyTorch's allocator and stays usable by
it, and the engine's own allocations reach what PyTorch merely caches."""

from __future__ import annotations

import gc

import numpy as np
import pytest
import torch
from adjoint_cases import case, gpu_lattice

from lattice_boltzmann_d3q19_b200 import Lattice, LbmError, autograd
from lattice_boltzmann_d3q19_b200 import _native as N

pytestmark = pytest.mark.gpu

SHAPE, STEPS, EVERY = (128, 128, 64), 60, 30  # f32: a tape of 2.7 GB
MB = 1 << 20


def _free() -> int:
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def _drag(shape=SHAPE):
    return Lattice(shape, 0.6, storage="f32", force_mode="drag", drag_k=0.05, inflow_u=(0.04, 0.0, 0.0))


def _gradient(lat, alpha):
    rho, u = autograd.run(lat, alpha, STEPS, checkpoint_every=EVERY)
    (g,) = torch.autograd.grad(autograd.box_kinetic_energy(rho, u, (1, 40)), alpha)
    return g


def test_a_destroyed_tape_leaves_nothing():
    with _drag() as lat:
        lat.set_porosity(np.full(SHAPE, 0.5, np.float32))
        lat.set_equilibrium()
        before = _free()
        for _ in range(2):
            lat.set_equilibrium()
            tape = lat.tape(STEPS, EVERY)
            assert tape.nbytes == lat.tape_bytes(STEPS, EVERY) > 2000 * MB
            assert _free() < before - 2000 * MB
            tape.close()
            assert _free() > before - 64 * MB


@pytest.mark.parametrize("own_stream", [False, True])
def test_pytorch_can_use_a_finished_tapes_memory(own_stream):
    with _drag() as lat:
        alpha = torch.full(SHAPE, 0.5, device="cuda", requires_grad=True)
        with torch.cuda.stream(torch.cuda.Stream() if own_stream else torch.cuda.default_stream()):
            _gradient(lat, alpha)  # whatever the lattice allocates once
            free = _free()
            for _ in range(3):
                _gradient(lat, alpha)
            # all but 1 GB of what is free without a tape, which is less than the tape took
            block = torch.empty(free - 1024 * MB, dtype=torch.uint8, device="cuda")
            del block
            torch.cuda.empty_cache()


def test_the_engine_can_use_what_pytorch_caches():
    free = _free()
    block = torch.empty(free - 2048 * MB, dtype=torch.uint8, device="cuda")
    del block  # cached
    with Lattice((256, 256, 128), 0.6) as lat:  # 2.8 GB
        lat.set_populations(np.broadcast_to(1.0 / 19.0, (19, 256, 256, 128)))
        lat.step(1)
        lat.synchronize()
    torch.cuda.empty_cache()


def test_reused_and_foreign_memory_leave_the_bits():
    c = case("drag_channel")
    shape = c["shape"]
    gr = torch.full(shape, 0.25, dtype=torch.float64, device="cuda")
    gu = torch.linspace(-1.0, 1.0, 3 * int(np.prod(shape)), dtype=torch.float64, device="cuda")

    def backward(lat, memory=None):
        lat.set_populations(c["f0"])
        ga = torch.full(shape, 7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        with lat.tape(20, 6, memory) as t:
            t.backward(gr.data_ptr(), gu.data_ptr(), ga.data_ptr())
            lat.synchronize()
        return ga.cpu().numpy().tobytes()

    with gpu_lattice(c, "f32") as lat:
        want = backward(lat)
        need = lat.tape_bytes(20, 6)
        memory = torch.full((need + 256,), 255, dtype=torch.uint8, device="cuda")
        assert backward(lat, memory) == want
        assert backward(lat, memory) == want  # what the last tape left in it does not matter
        lat.set_populations(c["f0"])
        for bad in (memory[:need - 1], memory[8:8 + need], torch.empty(need, dtype=torch.uint8)):
            with pytest.raises(LbmError) as e:
                lat.tape(20, 6, bad)
            assert e.value.code == N.LBM_ERR_INVALID
        for args in ((0, 5), (5, 0)):
            with pytest.raises(LbmError) as e:
                lat.tape_bytes(*args)
            assert e.value.code == N.LBM_ERR_INVALID


def test_forward_and_backward_on_different_streams():
    shape = (64, 48, 40)
    alpha0 = torch.rand(shape, generator=torch.Generator().manual_seed(1)).cuda()
    seed = torch.linspace(-1.0, 1.0, 3 * alpha0.numel(), dtype=torch.float64, device="cuda").view(3, *shape)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()

    def run(forward, backward, junk):
        got = []
        with _drag(shape) as lat:
            for _ in range(4):
                alpha = alpha0.clone().requires_grad_(True)
                torch.cuda.synchronize()
                with torch.cuda.stream(forward):
                    rho, u = autograd.run(lat, alpha, 30, checkpoint_every=10)
                    node = u.grad_fn
                torch.cuda.synchronize()
                with torch.cuda.stream(backward):
                    ga, *_ = autograd._LatticeRun.backward(node, None, seed)  # on a stream of its own
                nbytes = lat.tape_bytes(30, 10)
                del rho, u, node  # the memory is free again, the backward pass maybe still running
                if junk:
                    with torch.cuda.stream(forward):
                        torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
                got.append(ga.cpu().numpy().tobytes())
        return got

    want = run(one, one, False)
    assert len(set(want)) == 1
    assert run(one, one, True) == want
    assert run(one, two, True) == want
