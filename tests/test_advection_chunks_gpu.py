"""Godunov steps on boxes whose sizes cut the advection kernels' marches and
x rows unevenly (rows of 36 and 40 cells, several rows a block, rows longer
than a block; marches of 1, 2 and 4 faces with remainders), against the oracle.

The long rows (264 and 516 cells) repeat a short box, which the oracle
advances: its multigrid does not converge on boxes that long and thin (200
V-cycles leave 1e-3 of the target), and the flow repeats with its initial field.
Tolerance: the parity tolerance of the other step tests.
"""
import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
TOL = 1e-9


@pytest.mark.parametrize("n,times", [((36, 12, 8), 1), ((40, 36, 44), 1), ((24, 8, 12), 11), ((96, 64, 44), 1), ((12, 8, 8), 43)])
@pytest.mark.parametrize("walls", [True, False])
def test_step_matches_oracle(cuda_dev, oracle_mod, n, times, walls):
    def deck(nx):
        d = decks.abl(nx, n[1], n[2], steps=4, dz=10.0)
        return d if walls else d.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")

    g, o = cuda_dev.Incflo(deck(n[0] * times)), oracle_mod.Oracle(deck(n[0]))
    g.set_field("velocity", np.ascontiguousarray(np.tile(o.get_field("velocity"), (1, 1, 1, times))))
    g.InitData()
    o.InitData()
    assert g.step() and o.step()
    assert o.scalar("mac_iters") < 200 and o.scalar("nodal_iters") < 200
    for f in ("velocity", "conv_term", "u_mac", "v_mac", "w_mac"):
        a, b = g.get_field(f), o.get_field(f)
        a, b = a[..., :n[0] * times], np.tile(b[..., :n[0]], (1, 1, 1, times))
        assert np.abs(a - b).max() <= TOL * np.abs(b).max(), f
