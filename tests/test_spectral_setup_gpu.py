"""A direct start whose set-up fails half way: the call goes on with multigrid,
and a later call sets the factors up again.

The set-up is made to fail on the host: while another stream of the thread is
being captured (relaxed mode, so allocations are allowed) the runtime answers a
device-wide wait, which the set-up makes after its allocations, with an error.
The box is cubic and wall-bounded, where the handle's own solves are multigrid
and the first ApplyProjection forms the factors.
"""
import ctypes

import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
N = (32, 16, 16)
RELAXED, NON_BLOCKING = 2, 1


def project(sim, u):
    sim.set_field("velocity", u)
    for f in ("p", "gp"):  # the state a projection reads and leaves
        sim.set_field(f, np.zeros(sim.layout(f)))
    sim.ApplyProjection(0.0, 0.7, False)
    return sim.get_field("velocity")


def test_setup_that_fails_half_way(cuda_dev):
    import torch
    u = np.random.default_rng(5).uniform(-1, 1, (3,) + N[::-1])
    want = project(cuda_dev.Incflo(decks.abl(*N, steps=2)), u)
    sim = cuda_dev.Incflo(decks.abl(*N, steps=2))
    torch.cuda.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cu.cuStreamCreate(ctypes.byref(stream), NON_BLOCKING) == 0
    assert cu.cuStreamBeginCapture_v2(stream, RELAXED) == 0
    try:
        during = project(sim, u)
    finally:
        cu.cuStreamEndCapture(stream, ctypes.byref(graph))
        cu.cuStreamDestroy_v2(stream)
    assert sim.scalar("nodal_iters") > 0 and sim.scalar("nodal_direct") == 0
    after = project(sim, u)
    assert sim.scalar("nodal_iters") == 0 and sim.scalar("nodal_direct") == 1
    # the same operations on the same input: the same bits; the multigrid stops at 2.2e-11 of the right-hand side
    assert np.array_equal(after, want)
    assert np.abs(during - want).max() <= 1e-8 * np.abs(want).max()


def test_scalars_tell_the_start(cuda_dev):
    cubic, flat = cuda_dev.Incflo(decks.abl(*N, steps=2)), cuda_dev.Incflo(decks.abl(*N, steps=2, dz=10.0))
    for sim in (cubic, flat):
        sim.InitData()
        assert sim.step()
        for s in ("mac_direct", "nodal_direct"):
            assert sim.scalar(s) == float(sim is flat)
    cubic.ApplyProjection(0.0, 0.7, False)
    assert cubic.scalar("mac_direct") == 0 and cubic.scalar("nodal_direct") == 1
    flat.set_precision(1)
    assert flat.step()
    assert flat.scalar("mac_direct") == 0 and flat.scalar("nodal_direct") == 0
