"""Godunov steps on boxes whose sizes cut the advection kernels' marches and
x rows unevenly (rows of 36 and 40 cells, several rows a block, a row longer
than a block; marches of 1, 2 and 4 faces with remainders), against the oracle.
Tolerance: the parity tolerance of the other step tests.
"""
import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
TOL = 1e-9


@pytest.mark.parametrize("n", [(36, 12, 8), (40, 36, 44), (264, 8, 12), (96, 64, 44), (516, 8, 8)])
@pytest.mark.parametrize("walls", [True, False])
def test_step_matches_oracle(cuda_dev, oracle_mod, n, walls):
    d = decks.abl(*n, steps=4, dz=10.0)
    if not walls:
        d = d.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")
    g, o = cuda_dev.Incflo(d), oracle_mod.Oracle(d)
    g.InitData()
    o.InitData()
    assert g.step() and o.step()
    for f in ("velocity", "conv_term", "u_mac", "v_mac", "w_mac"):
        a, b = g.get_field(f), o.get_field(f)
        assert np.abs(a - b).max() <= TOL * max(np.abs(b).max(), 1e-300), f
