"""FP32 Smagorinsky and viscous marches of the mixed-precision form at the edges
of their blocks (32 columns, 8 rows, chunks of layers), against FP64.

Tolerances (e = 2^-24, U = max|u|, h the smallest spacing): a staged velocity is
off by e U.  mu_t: a central gradient is off by e U / h, a one-sided one by 8/3 of
that, and |S| moves by at most 2 sqrt(9) of the largest: 16 e U / h times
rho (Cs Delta)^2.  Viscous term: a flux combines at most 5 gradients, each off by
2 e U / h and at most 2 U / h, rounded at most 8 times, (10 + 80) e mu U / h; six
faces over h: 540 e mu U / h^2.
"""
import ctypes

import numpy as np
import pytest

from kynema_sgf_gb300 import decks

pytestmark = pytest.mark.gpu
E32 = 2.0 ** -24


@pytest.mark.parametrize("walls", [True, False])
@pytest.mark.parametrize("n", [(8, 8, 4), (20, 12, 8), (36, 28, 6), (32, 8, 20), (68, 20, 36)])
def test_marches(cuda_dev, n, walls):
    import torch
    d = decks.abl(*n, steps=2, dz=10.0)
    if not walls:
        d = d.replace("geometry.is_periodic = 1 1 0", "geometry.is_periodic = 1 1 1")
    m, g = cuda_dev.Incflo(d + "ks.precision = mixed\n"), cuda_dev.Incflo(d)
    for side in (m, g):
        side.InitData()
        assert side.step()
    u, v = m.get_field("velocity_old"), g.get_field("velocity_old")
    U, h = np.abs(u).max(), np.array([20.0, 20.0, 10.0])
    assert np.abs(u - v).max() <= 1e-8 * U  # the projected initial velocity, FP64 in both
    mu = m.get_field("velocity_mueff")
    cs2 = 1.225 * 0.135 ** 2 * np.prod(h) ** (2.0 / 3.0)
    assert np.abs(mu - g.get_field("velocity_mueff")).max() <= 16 * E32 * U / h.min() * cs2
    # the FP64 term of the same velocity, viscosity and wall gradient
    dev = [torch.from_numpy(a.ravel().copy()).cuda() for a in (u, mu)]
    wg = torch.from_numpy(m.get_field("wall_grad").ravel().copy()).cuda() if walls else None
    out = torch.empty_like(dev[0])
    ptr = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    assert cuda_dev.load_library().ks_divtau_noalloc(ptr(dev[0]), ptr(dev[1]), ptr(wg), ptr(out), *n, *h, int(not walls), int(walls), None) == 0
    torch.cuda.synchronize()
    got = m.get_field("diff_term").ravel()
    assert np.abs(got - out.cpu().numpy()).max() <= 540 * E32 * mu.max() * U / h.min() ** 2
