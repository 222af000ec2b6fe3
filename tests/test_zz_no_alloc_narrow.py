"""ks_divtau_noalloc on boxes of few columns in x, where a warp of the one-launch
form holds several rows: against the form that forms all fluxes first (a call in
place) at the edges of its blocks (4, 8 and 16 columns, 8 to 2 rows, marches
cut to the box), and no slower than it on long boxes.  The tolerance is that of the
other in-place tests; on 32 lanes a row the long boxes took 1.2 to 3.4 times as
long as in place, a warp of several rows about a half.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def caller(ks, n, form, in_place):
    import torch
    nx, ny, nz = n
    gen = torch.Generator(device="cuda").manual_seed(nx + ny + nz)
    vel = torch.rand((3, nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    mu = 0.5 + torch.rand((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    wg = torch.rand((2, ny, nx), generator=gen, device="cuda", dtype=torch.float64)
    out = vel if in_place else torch.full_like(vel, float("nan"))
    stream = torch.cuda.current_stream()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (vel, mu, wg, out)]

    def call():
        rc = ks.load_library().ks_divtau_noalloc(p[0], p[1], p[2] if form == "wall" else None, p[3], nx, ny, nz, 1.0, 0.7, 1.3,
                                                 int(form == "periodic"), int(form == "wall"), ctypes.c_void_p(stream.cuda_stream))
        assert rc == 0
        return out

    call.keep = (vel, mu, wg)
    return call


@pytest.mark.parametrize("n", [(4, 4, 4), (4, 10, 34), (6, 6, 6), (8, 8, 8), (8, 10, 34), (10, 4, 18), (14, 6, 4), (16, 16, 16), (16, 2050, 6), (18, 4, 4)])
@pytest.mark.parametrize("form", ["periodic", "slip", "wall"])
def test_narrow_boxes(cuda_dev, n, form):
    a, b = caller(cuda_dev, n, form, False)(), caller(cuda_dev, n, form, True)()
    assert float((a - b).abs().max()) <= 1e-13 * float(b.abs().max())


@pytest.mark.parametrize("n", [(4, 256, 256), (4, 4, 16384), (4, 6, 10922), (4, 10, 6552), (8, 8, 4096), (12, 10, 2184)])
def test_no_slower_than_face_by_face(cuda_dev, n):
    import torch

    def best(in_place):
        call, ms = caller(cuda_dev, n, "periodic", in_place), []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                call()
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms)

    assert best(False) <= best(True)
