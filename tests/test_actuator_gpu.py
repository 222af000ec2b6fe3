"""Disk spreading through tabulated 1D Gaussian factors, disks grouped into
launches by their boxes: disjoint and overlapping disks, boxes cut by the
domain, an oblique axis, against the oracle's point-by-point sum on the same
initial velocity.

Tolerance: a factor exp(-r^2), r^2 <= 16, carries at most 16 x 3 + 2 roundings
of 1.1e-16, a product of three 1.7e-14 of its value, the sampled velocity (the
same trilinear sum) a few more; 1e-12 of the maximum leaves a decade and a half.
"""
import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu

CASES = {
    "disjoint": dict(nx=96, ny=32, nz=32, dcells=6, cts=(0.7, 0.8, 0.6), eps_cells=1.0),
    "overlapping": dict(nx=64, ny=32, nz=32, dcells=10, cts=(0.7, 0.8, 0.6, 0.75), eps_cells=2.0),
    "cut by the domain": dict(nx=48, ny=16, nz=16, dcells=14, cts=(0.7, 0.8), eps_cells=2.5, nr=3, nt=7),
    "one point": dict(nx=32, ny=16, nz=16, dcells=4, cts=(0.9,), eps_cells=1.0, nr=1, nt=1),
}


@pytest.mark.parametrize("oblique", [False, True])
@pytest.mark.parametrize("case", sorted(CASES))
def test_spreading_matches_oracle(cuda_dev, oracle_mod, case, oblique):
    d = decks.disks(steps=2, **CASES[case])
    if oblique:
        d = d.replace("disk_normal = -1.0 0.0 0.0", "disk_normal = -0.9 0.3 0.0")
    g, o = cuda_dev.Incflo(d), oracle_mod.Oracle(d)
    for side in (g, o):
        side.compute_dt()
        side.pre_advance()
    a, b = g.get_field("actuator_src_term"), o.get_field("actuator_src_term")
    assert np.abs(b).max() > 0
    assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
