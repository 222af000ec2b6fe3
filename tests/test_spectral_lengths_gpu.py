"""Direct start of the Poisson solves on long lines (one x row a block above 512
points, 8 to 1 y columns a block, shared memory above 48 and 98 KB, up to five
passes of one transform) and where its residual misses the stopping test.

Long lines: boxes of equal extents, so a mode's column in z has a condition number
of at most (nz / pi)^2, below 4.  What is left is the transforms' rounding, log2(n)
times 1.1e-16 of the right-hand side's rms in every mode, which the lowest modes
divide by their eigenvalue: n log2(n) / 2 pi roundings, 9e-13 of the pressure at
4096 points.  1e-11 leaves a decade, for both sides of the comparison.

Missed test: decks with a target of 1e-30 of the right-hand side run all 200
V-cycles from the direct solution.  The boxes are those of the other direct-start
tests, and so are the tolerances.
"""
import numpy as np
import pytest

import test_spectral_gpu as base
from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
LENGTHS = [(600, 8, 4), (3072, 4, 4), (4096, 4, 4), (10, 400, 6), (6, 800, 4), (4, 1600, 4), (4, 4096, 4)]
STRICT = "%s_proj.mg_rtol = 1e-30\n%s_proj.mg_atol = 0\n"


def project_and_compare(cuda_dev, n, walls, extra=""):
    sim = cuda_dev.Incflo(base.deck(n, walls, extra))
    u = np.random.default_rng(n[0] + 3 * n[1]).uniform(-1, 1, (3,) + n[::-1])
    sim.set_field("velocity", u)
    sim.ApplyProjection(0.0, 0.7, False)
    want = base.nodal_reference(u, walls, 0.7 / 1.225)
    p = sim.get_field("p")[0]
    for a, b in zip((sim.get_field("velocity"), sim.get_field("gp"), p - p.mean()), (want[0], want[1], want[2] - want[2].mean())):
        assert np.abs(a - b).max() <= base.TOL * np.abs(b).max()
    assert sim.scalar("nodal_direct") == 1
    return sim


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", LENGTHS)
def test_nodal_projection_on_long_lines(cuda_dev, monkeypatch, n, walls):
    monkeypatch.setattr(base, "H", tuple(2000.0 / m for m in n))
    sim = project_and_compare(cuda_dev, n, walls)
    assert sim.scalar("nodal_iters") == 0 and sim.scalar("nodal_res") <= sim.scalar("nodal_target")


@pytest.mark.parametrize("n", [(600, 8, 4), (10, 400, 6)])
def test_mac_projection_on_long_lines(cuda_dev, monkeypatch, n):
    monkeypatch.setattr(base, "H", tuple(2000.0 / m for m in n))
    sim = cuda_dev.Incflo(base.deck(n, True))
    sim.InitData()
    assert sim.step()
    assert sim.scalar("mac_direct") == 1 and sim.scalar("mac_iters") == 0
    assert sim.scalar("mac_divu_rel") <= 1e-12


@pytest.mark.parametrize("walls", [True, False])
def test_nodal_cycles_after_a_missed_test(cuda_dev, walls):
    sim = project_and_compare(cuda_dev, (32, 16, 8), walls, STRICT % ("nodal", "nodal"))
    assert sim.scalar("nodal_iters") == 200 and sim.scalar("nodal_res") > sim.scalar("nodal_target")


@pytest.mark.parametrize("walls", [True, False])
def test_mac_cycles_after_a_missed_test(cuda_dev, walls):
    out = []
    for extra in (STRICT % ("mac", "mac"), ""):
        sim = cuda_dev.Incflo(base.deck((32, 16, 8), walls, extra))
        sim.InitData()
        assert sim.step()
        assert sim.scalar("mac_direct") == 1 and sim.scalar("mac_iters") == (200 if extra else 0)
        assert sim.scalar("mac_divu_rel") <= 1e-12
        out.append(sim.get_field("velocity"))
    assert np.abs(out[0] - out[1]).max() <= 1e-9 * np.abs(out[1]).max()


def test_mixed_reverse_cycles_after_a_missed_test(cuda_dev):
    """The reverse solves of a mixed-precision handle: FP32 cycles from the direct solution."""
    out = []
    for extra in (STRICT % ("mac", "mac") + STRICT % ("nodal", "nodal"), ""):
        d, lo, hi, _ = decks.adjoint_c3(32, 32, 16, dcells=4, n_disks=2)
        sim = cuda_dev.Incflo(d + "ks.precision = mixed\n" + extra)
        sim.InitData()
        sim.set_objective_box(lo, hi)
        sim.objective(seed=True)
        sim.adjoint_step()
        for s in ("mac", "nodal"):
            assert sim.scalar(s + "_direct") == 1 and sim.scalar(s + "_iters") == (200 if extra else 0)
        out.append([sim.get_field("velocity_adjoint"), sim.get_field("gp_adjoint"), sim.ct_gradient()])
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()
