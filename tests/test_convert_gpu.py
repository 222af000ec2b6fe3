"""FP64 <-> FP32 conversions on the integer pipe (d2f, f2d) and scalings by two on
the exponent field (twice, half_fin, half_of), bit for bit against IEEE
conversion and arithmetic in numpy: ties, the ends of both ranges, subnormals,
zeros, infinities and both kinds of NaN (which become quiet ones).

The functions are device inlines; the test compiles a kernel around each.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = """
#include "ks_decide.cuh"
using namespace ks;
enum { D2F, F2D, TWICE, HALF_FIN, HALF_OF };
template <int OP, typename In, typename Out>
__global__ void k(const In* x, Out* y, long long n) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= n) return;
    if constexpr (OP == D2F) y[t] = d2f(x[t]);
    else if constexpr (OP == F2D) y[t] = f2d(x[t]);
    else if constexpr (OP == TWICE) y[t] = twice(x[t]);
    else if constexpr (OP == HALF_FIN) y[t] = half_fin(x[t]);
    else y[t] = half_of(x[t]);
}
template <int OP, typename In, typename Out>
int run(const void* x, void* y, long long n) {
    In* a = nullptr;
    Out* b = nullptr;
    if (cudaMalloc(&a, n * sizeof(In)) || cudaMalloc(&b, n * sizeof(Out))) return 1;
    if (cudaMemcpy(a, x, n * sizeof(In), cudaMemcpyHostToDevice)) return 1;
    k<OP, In, Out><<<(unsigned)((n + 255) / 256), 256>>>(a, b, n);
    const int rc = cudaMemcpy(y, b, n * sizeof(Out), cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    return rc;
}
extern "C" int op(int which, const void* x, void* y, long long n) {
    switch (which) {
        case D2F: return run<D2F, double, float>(x, y, n);
        case F2D: return run<F2D, float, double>(x, y, n);
        case TWICE: return run<TWICE, double, double>(x, y, n);
        case HALF_FIN: return run<HALF_FIN, double, double>(x, y, n);
        default: return run<HALF_OF, double, double>(x, y, n);
    }
}
"""
D2F, F2D, TWICE, HALF_FIN, HALF_OF = range(5)


@pytest.fixture(scope="module")
def op(cuda_dev, tmp_path_factory):
    from kynema_sgf_gb300 import build
    d = tmp_path_factory.mktemp("convert")
    (d / "convert.cu").write_text(SOURCE)
    cmd = [build.nvcc()] + build.ARCH + build.FLAGS + ["-I", ROOT + "/kynema_sgf_gb300/csrc", "-shared", "-o", str(d / "convert.so"), str(d / "convert.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(d / "convert.so"))

    def call(which, x, out):
        x = np.ascontiguousarray(x)
        y = np.empty(x.shape, out)
        assert lib.op(which, x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(x.size)) == 0
        return y

    return call


def floats():
    """Random patterns, and every exponent with the first, last and some middle mantissas."""
    rng = np.random.default_rng(7)
    e = np.arange(256, dtype=np.uint32)[:, None] << 23
    m = np.array([0, 1, 2, 3, 0x3fffff, 0x400000, 0x400001, 0x7ffffe, 0x7fffff], np.uint32)[None]
    b = np.concatenate([(e | m).ravel(), rng.integers(0, 1 << 31, 1 << 20, dtype=np.uint32)])
    return np.concatenate([b, b | np.uint32(1 << 31)]).view(np.float32)


def doubles():
    """Random patterns; the floats, the ties between neighbours and both sides of each; the ends of the FP64 range."""
    rng = np.random.default_rng(8)
    f = floats()
    f = f[np.isfinite(f)]
    b = f.view(np.uint32) & np.uint32(0x7fffffff)
    lo = b.view(np.float32).astype(np.float64)
    up = (b + np.uint32(1)).view(np.float32).astype(np.float64)
    up = np.where(np.isinf(up), 2.0 ** 128, up)
    tie = 0.5 * (lo + up)  # exact
    v = np.concatenate([lo, tie, np.nextafter(tie, 0.0), np.nextafter(tie, np.inf), np.nextafter(lo, np.inf), np.nextafter(lo, 0.0)])
    e = np.arange(2048, dtype=np.uint64)[:, None] << np.uint64(52)
    m = np.array([0, 1, 0x8000000000000, 0xfffffffffffff], np.uint64)[None]
    bits = np.concatenate([v.view(np.uint64), (e | m).ravel(), rng.integers(0, 1 << 63, 1 << 20, dtype=np.uint64)])
    return np.concatenate([bits, bits | np.uint64(1 << 63)]).view(np.float64)


def check(got, want, quiet):
    nan = np.isnan(want)
    u = {4: np.uint32, 8: np.uint64}[got.dtype.itemsize]
    assert np.array_equal(got.view(u)[~nan], want.view(u)[~nan])
    assert np.isnan(got[nan]).all() and ((got.view(u)[nan] & u(quiet)) != 0).all()


def test_double_to_float(op):
    x = doubles()
    with np.errstate(all="ignore"):
        check(op(D2F, x, np.float32), x.astype(np.float32), 1 << 22)


def test_float_to_double(op):
    x = floats()
    with np.errstate(all="ignore"):
        check(op(F2D, x, np.float64), x.astype(np.float64), 1 << 51)


def test_scalings_by_two(op):
    x = doubles()
    a = np.abs(x)
    fin, normal = np.isfinite(x), a >= 2.0 ** -1022
    s = x[fin & normal & (a < 2.0 ** 1023)]  # beyond: the exponent field overflows
    assert np.array_equal(op(TWICE, s, np.float64), 2.0 * s)
    s = x[fin]
    want = np.where(np.abs(s) >= 2.0 ** -1021, 0.5 * s, 0.0)  # a half below the normal range is zero
    assert np.array_equal(op(HALF_FIN, s, np.float64), want)
    with np.errstate(invalid="ignore"):
        want = np.where(fin & (a < 2.0 ** -1021), 0.0, 0.5 * x)
    got = op(HALF_OF, x, np.float64)
    assert np.array_equal(got[~np.isnan(x)], want[~np.isnan(x)]) and np.isnan(got[np.isnan(x)]).all()
