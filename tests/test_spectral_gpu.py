"""Direct start of the Poisson solves (ks_spectral.cu): transforms of every
radix (2 to 13, alone and in products), periodic and wall-bounded columns,
unequal spacings.

The nodal projection is compared with a numpy solve of the same operator
(transforms in x and y, a dense solve per mode in z).  Both are FP64 with a
condition number of at most (n / pi)^2 times the squared aspect ratio, below
1e4 on these boxes: 1e-11 relative leaves two decades over that times epsilon.
The MAC projection is checked by its own residual: after a step the divergence
of the face velocities is below 1e-12 of max|u| / h (the solve's rounding, the
multigrid tolerance being 2e-11), and no V-cycle ran.
"""
import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
TOL = 1e-11
H = (20.0, 15.0, 10.0)


def deck(n, walls, extra=""):
    nx, ny, nz = n
    d = decks.abl(nx, ny, nz, steps=10)
    d = d.replace("geometry.prob_hi = %s %s %s" % (nx * 20.0, ny * 20.0, nz * 20.0),
                  "geometry.prob_hi = %r %r %r" % (nx * H[0], ny * H[1], nz * H[2]))
    assert repr(ny * H[1]) in d
    if not walls:
        d = d.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")
    return d + extra


def nodal_reference(u, walls, sigma):
    """(u - sigma G phi, G phi, phi) with sigma A phi = D u."""
    nz, ny, nx = u.shape[1:]
    if walls:
        g = np.stack([np.concatenate([s * u[n, :1], u[n], s * u[n, -1:]]) for n, s in ((0, 1), (1, 1), (2, -1))])
    else:
        g = np.concatenate([u[:, -1:], u], 1)

    def dif(a, ax):
        return a - np.roll(a, 1, ax)

    def avg(a, ax):
        return 0.5 * (a + np.roll(a, 1, ax))

    rhs = 0.5 * (avg(dif(g[0], 2), 1)[1:] + avg(dif(g[0], 2), 1)[:-1]) / H[0]
    rhs += 0.5 * (avg(dif(g[1], 1), 2)[1:] + avg(dif(g[1], 1), 2)[:-1]) / H[1]
    rhs += avg(avg(g[2, 1:] - g[2, :-1], 2), 1) / H[2]
    nn = rhs.shape[0]
    w = np.ones(nn)
    if walls:
        w[0] = w[-1] = 0.5
    K, Mz = np.zeros((nn, nn)), np.zeros((nn, nn))
    for k in range(nn):
        for q in (k - 1, k + 1):
            q = (-q if q < 0 else (2 * (nn - 1) - q if q >= nn else q)) if walls else q % nn
            K[k, q] -= 1.0 / H[2] ** 2
            Mz[k, q] += 1.0 / 6.0
        K[k, k] += 2.0 / H[2] ** 2
        Mz[k, k] += 2.0 / 3.0
    R = np.fft.rfft2(rhs) / sigma
    P = np.zeros_like(R)
    for j in range(ny):
        for i in range(nx // 2 + 1):
            a, b = 2 * np.pi * i / nx, 2 * np.pi * j / ny
            kx, ky = (2 - 2 * np.cos(a)) / H[0] ** 2, (2 - 2 * np.cos(b)) / H[1] ** 2
            mx, my = (2 + np.cos(a)) / 3, (2 + np.cos(b)) / 3
            A = -((kx * my + mx * ky) * Mz + mx * my * K)
            r = R[:, j, i]
            P[:, j, i] = np.linalg.lstsq(A, r - (w @ r) / w.sum(), rcond=None)[0] if i == 0 and j == 0 else np.linalg.solve(A, r)
    p = np.fft.irfft2(P, s=(ny, nx))
    n = p if walls else np.concatenate([p, p[:1]])

    def up(a, ax):
        return np.roll(a, -1, ax)

    def mean4(a, x, y):
        return 0.25 * (a + up(a, x) + up(a, y) + up(up(a, x), y))

    gx = 0.5 * (up(n, 2) - n + up(up(n, 2) - n, 1)) / H[0]
    gy = 0.5 * (up(n, 1) - n + up(up(n, 1) - n, 2)) / H[1]
    gp = np.stack([0.5 * (gx[1:] + gx[:-1]), 0.5 * (gy[1:] + gy[:-1]), mean4(n[1:] - n[:-1], 1, 2) / H[2]])
    return u - sigma * gp, gp, p


SIZES = [(4, 6, 4), (8, 10, 6), (14, 4, 8), (22, 16, 4), (26, 18, 6), (32, 42, 8), (64, 12, 10), (30, 128, 4), (256, 8, 6)]


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", SIZES)
def test_nodal_projection_matches_numpy(cuda_dev, n, walls):
    sim = cuda_dev.Incflo(deck(n, walls))
    rng = np.random.default_rng(n[0] * 1000 + n[1])
    u = rng.uniform(-1, 1, (3, n[2], n[1], n[0]))
    sim.set_field("velocity", u)
    sim.ApplyProjection(0.0, 0.7, False)
    assert sim.scalar("nodal_iters") == 0
    assert sim.scalar("nodal_res") <= sim.scalar("nodal_target")
    want = nodal_reference(u, walls, 0.7 / 1.225)
    p = sim.get_field("p")[0]
    got = (sim.get_field("velocity"), sim.get_field("gp"), p - p.mean())
    for a, b in zip(got, (want[0], want[1], want[2] - want[2].mean())):
        assert np.abs(a - b).max() <= TOL * np.abs(b).max()


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", SIZES[1:])
def test_mac_projection_is_exact(cuda_dev, n, walls):
    sim = cuda_dev.Incflo(deck(n, walls))
    sim.InitData()
    assert sim.step()
    assert sim.scalar("mac_iters") == 0 and sim.scalar("mac_res") <= sim.scalar("mac_target")
    assert sim.scalar("mac_divu_rel") <= 1e-12


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-7), ("mixed", 1e-4)])
@pytest.mark.parametrize("n", [(32, 32, 16), (48, 20, 24)])
def test_reverse_step_with_direct_solves(cuda_dev, n, precision, tol):
    """A reverse step whose forward solves (FP64) or reverse solves (mixed) start
    directly, against the same step on multigrid iterates from zero.  The
    multigrid's tolerance of 2e-11 on the residual leaves up to 1e-8 of an
    adjoint field (condition number below 1e3), FP32 roundings 1e-5.
    """
    out = []
    for warm in (1, 0):
        d, lo, hi, _ = decks.adjoint_c3(*n, dcells=4, n_disks=2)
        sim = cuda_dev.Incflo(d + "ks.precision = %s\nks.mg_warm_start = %d\n" % (precision, warm))
        sim.InitData()
        sim.set_objective_box(lo, hi)
        sim.objective(seed=True)
        sim.adjoint_step()
        assert (sim.scalar("mac_iters") == 0) == (warm == 1 and precision == "mixed")  # the last MAC solve is the reverse one
        out.append([sim.get_field("velocity_adjoint"), sim.get_field("gp_adjoint"), sim.ct_gradient()])
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()


def test_multigrid_where_it_is_asked_for(cuda_dev):
    """ks.mg_warm_start = 0, a limit on the V-cycles, mixed precision or a count
    with a large prime keep the multigrid solve, to the same fields."""
    n = (32, 32, 16)
    cubic = cuda_dev.Incflo(decks.abl(*n, steps=4))
    cubic.InitData()
    assert cubic.step() and cubic.scalar("nodal_iters") > 0 and cubic.scalar("mac_iters") > 0
    cubic.ApplyProjection(0.0, 0.7, False)
    assert cubic.scalar("nodal_iters") == 0
    out = {}
    for key, extra in (("direct", ""), ("zero", "ks.mg_warm_start = 0\n"), ("limit", "nodal_proj.maxiter = 60\nmac_proj.maxiter = 60\n")):
        sim = cuda_dev.Incflo(deck(n, True, extra))
        sim.InitData()
        assert sim.step()
        assert (sim.scalar("nodal_iters") == 0) == (key == "direct")
        out[key] = sim.get_field("velocity")
    mix = cuda_dev.Incflo(deck(n, True))
    mix.set_precision(1)  # a handle may change form between calls
    mix.InitData()
    assert mix.step() and mix.scalar("nodal_iters") > 0 and mix.scalar("mac_iters") > 0
    mix.set_precision(0)
    assert mix.step() and mix.scalar("nodal_iters") == 0 and mix.scalar("mac_iters") == 0
    mix.set_precision(1)  # the warm start reads the potential the direct solve left
    assert mix.step() and mix.scalar("mac_iters") > 0 and mix.scalar("mac_res") <= mix.scalar("mac_target")
    for key in ("zero", "limit"):
        assert np.abs(out[key] - out["direct"]).max() <= 1e-9 * np.abs(out["direct"]).max()
    sim = cuda_dev.Incflo(deck((68, 32, 16), True))
    sim.set_field("velocity", np.random.default_rng(1).uniform(-1, 1, (3, 16, 32, 68)))
    sim.ApplyProjection(0.0, 0.7, False)
    assert sim.scalar("nodal_iters") > 0
