"""Multigrid steps whose coarsest level is swept by one CTA: levels of more than
512 points in shared memory (two levels of 1000 and 1680 cells, a single level
of 5720), and a level beyond its size, in global memory (14872 cells under
52 x 52 x 44).  FP64 against the oracle, mixed precision against FP64.

FP64 tolerance: the parity tolerance of the other step tests.  Mixed: the
stated error of the form over a step, 1e-6 relative L2 of the velocity.  A
single level as large as 42 x 42 x 10 is not compared: its nodal solve stops 3.1e-9
of the pressure from the oracle's after the same 16 V-cycles, in the 256-thread
form of the sweeps as in this one (which agree to 7e-15).
"""
import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
TOL = 1e-9


def rel(a, b, name=""):
    if name == "p":
        a, b = a - a.mean(), b - b.mean()
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("n", [(40, 40, 40), (28, 20, 24), (26, 22, 10), (52, 52, 44)])
@pytest.mark.parametrize("walls", [True, False])
def test_swept_bottom(cuda_dev, oracle_mod, n, walls):
    d = decks.abl(*n, steps=4) + "ks.mg_warm_start = 0\n"
    if not walls:
        d = d.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")
    g, m, o = cuda_dev.Incflo(d), cuda_dev.Incflo(d + "ks.precision = mixed\n"), oracle_mod.Oracle(d)
    for side in (g, m, o):
        side.InitData()
        assert side.step()
    assert o.scalar("mac_iters") < 200 and o.scalar("nodal_iters") < 200
    for f in ("velocity", "p", "gp", "u_mac", "v_mac", "w_mac"):
        assert rel(g.get_field(f), o.get_field(f), f) <= TOL, f
    for s in ("mac", "nodal"):
        assert m.scalar(s + "_res") <= m.scalar(s + "_target")
    u, v = m.get_field("velocity"), g.get_field("velocity")
    assert np.linalg.norm(u - v) <= 1e-6 * np.linalg.norm(v)
