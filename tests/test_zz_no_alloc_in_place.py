"""ks_divtau_noalloc: the one-launch form against the in-place form (output over
the velocity, fluxes formed first), over block edges and remainders.  The two
round differently: 1e-13 of the maximum is a few hundred roundings of a term
that sums 18 fluxes of cancelling differences on O(1) fields.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(4, 4, 4), (32, 32, 16), (34, 6, 10), (66, 10, 4), (128, 64, 32), (6, 64, 34)])
@pytest.mark.parametrize("form", ["periodic", "slip", "wall"])
def test_in_place_equals_out_of_place(cuda_dev, n, form):
    import torch
    nx, ny, nz = n
    gen = torch.Generator(device="cuda").manual_seed(nx + ny + nz)
    vel = torch.rand((3, nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    mu = 0.5 + torch.rand((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    wg = torch.rand((2, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    lib = cuda_dev.load_library()

    def call(v, out):
        torch.cuda.synchronize()
        rc = lib.ks_divtau_noalloc(ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(mu.data_ptr()),
                                   ctypes.c_void_p(wg.data_ptr()) if form == "wall" else None, ctypes.c_void_p(out.data_ptr()), nx, ny, nz,
                                   1.0, 0.7, 1.3, int(form == "periodic"), int(form == "wall"), None)
        torch.cuda.synchronize()
        assert rc == 0
        return out

    a = call(vel, torch.full_like(vel, float("nan")))
    v = vel.clone()
    b = call(v, v)
    assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())
