// Shared device definitions: grid descriptor, index maps with periodic wrap,
// boundary-condition accessors and kernel declarations.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>

namespace ks {

enum ZBC { ZPER = 0, ZSLIP = 1, ZWALLMODEL = 2 };

constexpr double kSmallVel = 1.0e-8;  // AMReX-Hydro small_vel

// Uniform single-box grid.  x and y are periodic; z is periodic (zper = 1) or
// bounded by a slip wall / wall-model wall at each end.
struct Grid {
    int nx, ny, nz;
    int zper;
    int zlo, zhi;
    double dx, dy, dz;
    double idx, idy, idz;  // 1/dx, 1/dy, 1/dz (FP64 division is expensive on this GPU)
    long long N;    // cells
    long long NFz;  // z faces stored: nx*ny*(nz+1)
};

__host__ __device__ inline long long cidx(const Grid& g, int i, int j, int k) {
    return ((long long)k * g.ny + j) * g.nx + i;
}
__host__ __device__ inline int wrapn(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
// any i: a tile or a warp's segment may be wider than the grid, but one period is the
// rule, and the two remainders take some 40 instructions (a loop in their place is
// slower still)
__device__ inline int wrap_tile(int i, int n) {
    i = wrapn(i, n);
    if ((unsigned)i >= (unsigned)n) i = (i % n + n) % n;
    return i;
}
// Marches of a thread per column, up to 128 columns of a row a block: the column,
// the launch, and 16 layers a march or fewer where that leaves less than `warps`.
#ifdef __CUDACC__
__device__ inline bool column_of(const Grid& g, int& i, int& j) {
    const unsigned nb = ((unsigned)g.nx + blockDim.x - 1) / blockDim.x, b = blockIdx.x / nb;
    i = (int)((blockIdx.x - b * nb) * blockDim.x + threadIdx.x);
    j = (int)b;
    return i < g.nx;
}
#endif
inline int column_threads(const Grid& g) { return g.nx > 96 ? 128 : 32 * ((g.nx + 31) / 32); }
inline dim3 column_grid(const Grid& g, int kc) {
    const int t = column_threads(g);
    return dim3((unsigned)((g.nx + t - 1) / t) * (unsigned)g.ny, (unsigned)((g.nz + kc - 1) / kc));
}
inline int march_layers(const Grid& g, int warps) {
    const long long kc = g.N / (32LL * warps);
    return kc < 1 ? 1 : (kc > 16 ? 16 : (int)kc);
}
__host__ __device__ inline double hd(const Grid& g, int d) { return d == 0 ? g.dx : (d == 1 ? g.dy : g.dz); }
__host__ __device__ inline double ihd(const Grid& g, int d) { return d == 0 ? g.idx : (d == 1 ? g.idy : g.idz); }
__host__ __device__ inline int nd(const Grid& g, int d) { return d == 0 ? g.nx : (d == 1 ? g.ny : g.nz); }
__host__ __device__ inline int nzfaces(const Grid& g) { return g.zper ? g.nz : g.nz + 1; }

// Face arrays: x and y faces use the cell index of the cell on their high
// side (N entries, periodic); z faces use nx*ny*(nz+1) storage with layer k
// at k-1/2 (walls) or wrap into [0,nz) (periodic).
__host__ __device__ inline long long fidx(const Grid& g, int d, int i, int j, int k) {
    i = wrapn(i, g.nx);
    j = wrapn(j, g.ny);
    if (d != 2 || g.zper) k = wrapn(k, g.nz);
    return cidx(g, i, j, k);
}

#ifdef __CUDACC__
// Cell-centred velocity (or rho*velocity) with fill-patch ghost values:
// periodic wrap in x, y (and z); at walls the tangential components take the
// high-order extrapolation to the face, (15 q0 - 10 q1 + 3 q2)/8, in every
// ghost layer and the normal component is 0.  The field is stored as S
// (FP64, or its FP32 copy in the mixed-precision advection); the value is
// returned in the arithmetic type T of the caller.
template <typename T = double, typename S = double>
struct VelFPT {
    const S* v;
    Grid g;
    T scale;
    __device__ inline T operator()(int n, int i, int j, int k) const {
        i = wrapn(i, g.nx);
        j = wrapn(j, g.ny);
        const long long N = g.N;
        const S* c = v + n * N;
        if (g.zper) return scale * (T)(c[cidx(g, i, j, wrapn(k, g.nz))]);
        if (k < 0) {
            if (n == 2) return T(0);
            const T q0 = (T)(c[cidx(g, i, j, 0)]), q1 = (T)(c[cidx(g, i, j, 1)]), q2 = (T)(c[cidx(g, i, j, 2)]);
            return scale * (T(0.125) * (T(15) * q0 - T(10) * q1 + T(3) * q2));
        }
        if (k >= g.nz) {
            if (n == 2) return T(0);
            const int t = g.nz - 1;
            const T q0 = (T)(c[cidx(g, i, j, t)]), q1 = (T)(c[cidx(g, i, j, t - 1)]), q2 = (T)(c[cidx(g, i, j, t - 2)]);
            return scale * (T(0.125) * (T(15) * q0 - T(10) * q1 + T(3) * q2));
        }
        return scale * (T)(c[cidx(g, i, j, k)]);
    }
};
using VelFP = VelFPT<double>;

#endif

inline unsigned nblocks(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// ---- FP64 decisions on the integer pipe.
// On this GPU every FP64 instruction -- DFMA, DADD, DMUL, and also the
// compares (DSETP) and min/max (DMNMX) -- issues at one sixty-fourth of the
// FP32 rate, while 64-bit integer compares and selects cost no FP64 issue
// slot.  Doubles that are not NaN order like their bit patterns read as
// sign-magnitude integers, so signs, comparisons, minima and maxima are taken
// on the bits.  Results equal the FP64 forms for every non-NaN operand, except
// that -0 orders below +0 (min/max may return the other zero).  NaN operands
// are not ordered like IEEE does; a NaN field still reaches the host through
// the arithmetic it enters and the residual / CFL maxima (imax_abs keeps it).
#ifdef __CUDACC__
// The casts are opaque moves: given __double_as_longlong the compiler recognises
// masks and comparisons of the pattern and turns them back into FP64 compares.
__device__ __forceinline__ long long dbits(double x) {
    long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}
__device__ __forceinline__ double bitsd(long long b) {
    double x;
    asm("mov.b64 %0, %1;" : "=d"(x) : "l"(b));
    return x;
}
constexpr long long kMag = 0x7fffffffffffffffLL;
// signed integer with the order of the doubles
__device__ __forceinline__ long long okey(double x) {
    const long long b = dbits(x);
    return b ^ ((b >> 63) & kMag);
}
__device__ __forceinline__ bool igt0(double x) { return dbits(x) > 0; }   // x > 0
__device__ __forceinline__ bool ile0(double x) { return dbits(x) <= 0; }  // x <= 0
__device__ __forceinline__ bool ilt0(double x) { return okey(x) < -1; }   // x < 0 (-0 is not)
__device__ __forceinline__ bool ige0(double x) { return okey(x) >= -1; }  // x >= 0 (-0 is)
// ilt / imin / imax order -0 below +0 (okey(-0) = -1, okey(+0) = 0), where IEEE
// compares them equal: a +-0 tie goes to the signed zero's order, not to the
// first operand as fmin / fmax may
__device__ __forceinline__ bool ilt(double a, double b) { return okey(a) < okey(b); }
__device__ __forceinline__ double imin(double a, double b) { return okey(a) < okey(b) ? a : b; }
__device__ __forceinline__ double imax(double a, double b) { return okey(a) > okey(b) ? a : b; }
// Magnitudes and signs are taken on the high word: the compiler turns the same
// masks on the 64-bit pattern back into fabs, copysign and negation, which
// issue as FP64 instructions.
__device__ __forceinline__ double hiword(double x, int hi) { return __hiloint2double(hi, __double2loint(x)); }
__device__ __forceinline__ double iabs(double x) { return hiword(x, __double2hiint(x) & 0x7fffffff); }
__device__ __forceinline__ double ineg(double x) { return hiword(x, __double2hiint(x) ^ (int)0x80000000); }
// |x| < c for c > 0
__device__ __forceinline__ bool iabs_lt(double x, double c) { return (dbits(x) & kMag) < dbits(c); }
// |a| < |b|
__device__ __forceinline__ bool iabs_lt2(double a, double b) { return (dbits(a) & kMag) < (dbits(b) & kMag); }
// a and b non-zero with the same sign (a * b > 0 unless the product underflows)
__device__ __forceinline__ bool isame_sign(double a, double b) {
    return (dbits(a) ^ dbits(b)) >= 0 && (dbits(a) & kMag) != 0 && (dbits(b) & kMag) != 0;
}
// copysign(m, s)
__device__ __forceinline__ double isign(double m, double s) {
    return hiword(m, (__double2hiint(m) & 0x7fffffff) | (__double2hiint(s) & (int)0x80000000));
}
// ---- FP32 <-> FP64 on the integer pipe.  A conversion instruction takes an
// FP64 issue slot (74 cycles of a warp), these about ten integer instructions,
// and give the same bits: round to nearest even, FP32 subnormals included; a
// NaN becomes a quiet NaN.  What is not zero or normal in FP32 takes the call.
// They pay in kernels bound by FP64 issue (viscous tile on 256x256x128: 520 us
// with conversions, 450 with these); kernels that wait on memory keep the
// conversion (k_adj_edges_gather 573 us, 769 with these).
static __device__ __noinline__ float d2f_rare(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29), r = lo & 0x1fffffffu;
    const int e = (int)((hi >> 20) & 0x7ffu) - 896;  // biased FP32 exponent
    unsigned b = 0u;
    if (e <= 0) {  // FP32 subnormal or zero
        const int s = 1 - e;
        const unsigned f = m | 0x800000u;
        if (s <= 24) {
            const unsigned q = f >> s, rem = f & ((1u << s) - 1u), half = 1u << (s - 1);
            b = q + (rem > half || (rem == half && (r || (q & 1u))));
        }
    } else {
        b = e == 1151 && (m | r) ? 0x7fffffffu : 0x7f800000u;
    }
    return __uint_as_float((hi & 0x80000000u) | b);
}
__device__ __forceinline__ float d2f(double x) {
    const int h = __double2hiint(x);
    if ((unsigned)((h & 0x7ff00000) - 0x38100000) >= 0x0fe00000u && ((h & 0x7fffffff) | __double2loint(x)) != 0) return d2f_rare(x);
    // round at bit 29, then the exponent's bias: its top bit inverted
    const long long v = dbits(x), q = v + 0x0fffffff + ((v >> 29) & 1);
    const unsigned t = ((unsigned)(q >> 29) & 0x7fffffffu) ^ 0x40000000u;
    return __uint_as_float(((h & 0x7fffffff) == 0 ? 0u : t) | ((unsigned)h & 0x80000000u));
}
static __device__ __noinline__ double f2d_rare(float x) {
    const unsigned b = __float_as_uint(x), sign = b & 0x80000000u;
    unsigned m = b & 0x7fffffu, e = 1151u;
    if ((b & 0x7f800000u) == 0u) {
        const int s = __clz((int)m) - 8;  // normalise
        m = (m << s) & 0x7fffffu;
        e = 1u - (unsigned)s;
    } else if (m) {
        m |= 0x400000u;
    }
    return __hiloint2double((int)(sign | ((e + 896u) << 20) | (m >> 3)), (int)(m << 29));
}
__device__ __forceinline__ double f2d(float x) {
    const unsigned b = __float_as_uint(x), a = b & 0x7fffffffu;
    if (a - 0x00800000u >= 0x7f000000u && a != 0u) return f2d_rare(x);
    const unsigned h = ((unsigned)((int)b >> 3) & 0x8fffffffu) + (a == 0u ? 0u : 0x38000000u);
    return __hiloint2double((int)h, (int)(b << 29));
}
template <typename To>
__device__ __forceinline__ To to(double x) {
    if constexpr (sizeof(To) == 8) return x;
    else return d2f(x);
}
template <typename To>
__device__ __forceinline__ To to(float x) {
    if constexpr (sizeof(To) == 4) return x;
    else return f2d(x);
}

// max that keeps a NaN operand (fmax drops it): a non-finite residual or CFL
// maximum must reach the host's finiteness checks
__device__ __forceinline__ double nmax(double a, double b) {
    if ((dbits(a) & kMag) > 0x7ff0000000000000LL) return a;
    if ((dbits(b) & kMag) > 0x7ff0000000000000LL) return b;
    return imax(a, b);
}
// running max of |x| kept as bits: NaN patterns order above infinity, so a
// NaN operand survives to the host
__device__ __forceinline__ long long imax_abs(long long m, double x) {
    const long long b = dbits(x) & kMag;
    return b > m ? b : m;
}
#endif

}  // namespace ks
