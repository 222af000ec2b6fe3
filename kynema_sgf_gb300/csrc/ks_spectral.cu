// Direct solution of the two Poisson problems of the step on uniform grids
// that are periodic in x and y: Fourier transforms in x and y turn either
// operator (the 7-point MAC Laplacian, the 27-point Q1 nodal one, both tensor
// products of symmetric 1D stencils) into one tridiagonal system in z per
// horizontal mode.
//
// Five kernels, all in FP64:
//   k_fft_x (forward): planes 2m and 2m + 1 of the real right-hand side are the
//     real and imaginary part of one complex plane, so no work goes to
//     redundant conjugate modes;
//   k_fft_y (forward), in place;
//   k_modes_z: a thread owns the mode pair (kx, ky), (-kx, -ky), separates the
//     two real planes' coefficients, runs the elimination up and the
//     substitution down in place and merges them again;
//   k_fft_y, k_fft_x (inverse).
//
// What bounds them is FP64 issue (an FP64 warp instruction holds its pipe for
// about 80 cycles on this GPU): the transforms spend about 25 FP64
// instructions per complex point and direction, the z pass 5.5 per real
// point, 57 per point in all, where one V-cycle of the same problem spends 43
// (MAC) or 89 (nodal) and 8 to 70 of them are needed.  The transforms
// therefore take the radix order with the fewest twiddle products (largest
// radix first, no twiddles in the first pass) and leave re-ordering to the
// Stockham index map; the first pass reads and the last pass writes global
// memory directly, the passes between exchange through shared memory.
#include <algorithm>

#include "ks_decide.cuh"
#include "ks_launch.hpp"

namespace ks {

namespace {

struct Line {  // one transform length
    int n, np;
    int r[12];  // radices, first pass first
    const double2* tw;  // exp(-2 pi i q / n), q < n
};

__device__ inline double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ inline double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ inline double2 cmul(double2 a, double2 w) { return make_double2(fma(-a.y, w.y, a.x * w.x), fma(a.y, w.x, a.x * w.y)); }

__device__ inline void dft4(double2& a, double2& b, double2& c, double2& d) {
    const double2 t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = csub(b, d);
    a = cadd(t0, t2);
    c = csub(t0, t2);
    b = make_double2(t1.x + t3.y, t1.y - t3.x);
    d = make_double2(t1.x - t3.y, t1.y + t3.x);
}

// v <- its DFT of length R (exp(-2 pi i j k / R)), in place.  Odd R: sums and
// differences of the entries j and R - j, the roots from the line's table.
template <int R>
__device__ inline void dft(double2 (&v)[R], const Line& P) {
    if constexpr (R == 2) {
        const double2 t = v[0];
        v[0] = cadd(t, v[1]);
        v[1] = csub(t, v[1]);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        constexpr double h = 0.70710678118654752440;
        dft4(v[0], v[2], v[4], v[6]);  // even entries: X0..X3 in v0, v2, v4, v6
        dft4(v[1], v[3], v[5], v[7]);
        const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
        const double s1 = o1.x + o1.y, d1 = o1.y - o1.x, s3 = o3.x + o3.y, d3 = o3.y - o3.x;
        v[0] = cadd(e0, o0);
        v[4] = csub(e0, o0);
        v[1] = make_double2(fma(h, s1, e1.x), fma(h, d1, e1.y));
        v[5] = make_double2(fma(-h, s1, e1.x), fma(-h, d1, e1.y));
        v[2] = make_double2(e2.x + o2.y, e2.y - o2.x);
        v[6] = make_double2(e2.x - o2.y, e2.y + o2.x);
        v[3] = make_double2(fma(h, d3, e3.x), fma(-h, s3, e3.y));
        v[7] = make_double2(fma(-h, d3, e3.x), fma(h, s3, e3.y));
    } else {
        constexpr int H = (R - 1) / 2;
        double2 a[H], b[H];
        double co[H], si[H];
        const double2 x0 = v[0];
        double2 s = x0;
        const int q = P.n / R;
#pragma unroll
        for (int j = 0; j < H; ++j) {
            a[j] = cadd(v[j + 1], v[R - 1 - j]);
            b[j] = csub(v[j + 1], v[R - 1 - j]);
            s = cadd(s, a[j]);
            const double2 w = P.tw[(j + 1) * q];
            co[j] = w.x;
            si[j] = -w.y;
        }
        v[0] = s;
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            double2 p = x0, g = make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 1; j <= H; ++j) {
                const int m = (j * k) % R;  // root index; m > H is the mirrored root
                const double c = co[(m > H ? R - m : m) - 1], sn = m > H ? -si[R - m - 1] : si[m - 1];
                p = make_double2(fma(a[j - 1].x, c, p.x), fma(a[j - 1].y, c, p.y));
                g = make_double2(fma(b[j - 1].x, sn, g.x), fma(b[j - 1].y, sn, g.y));
            }
            v[k] = make_double2(p.x + g.y, p.y - g.x);
            v[R - k] = make_double2(p.x - g.y, p.y + g.x);
        }
    }
}

// One Stockham pass over L lines: butterfly b of a line takes the entries
// b + r n / R, turns entry r by the root of index (b mod ns) r n / (ns R) and
// writes its DFT to (b / ns) ns R + b mod ns + r ns.  COL: the lines are the
// fastest index of a thread (columns of a plane), else the butterflies are
// (rows).
template <int R, bool COL, typename Ld, typename St>
__device__ inline void pass(const Line& P, int L, int ns, const Ld& ld, const St& st) {
    const int nb = P.n / R, step = P.n / (ns * R);
    for (int t = threadIdx.x; t < nb * L; t += blockDim.x) {
        const int b = COL ? t / L : t % nb, l = COL ? t % L : t / nb;
        const int g = b / ns, k = b - g * ns;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ld(l, b + r * nb);
        if (ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], P.tw[k * r * step]);
        }
        dft<R>(v, P);
#pragma unroll
        for (int r = 0; r < R; ++r) st(l, g * ns * R + k + r * ns, v[r]);
    }
}

// L lines: loads by ld(line, index), stores by st(line, index, value), the
// passes between through the two halves of shared memory sh (index map at).
template <bool COL, typename Ld, typename St, typename At>
__device__ inline void transform(const Line& P, int L, double2* sh, int half, const Ld& ld, const St& st, const At& at) {
    int ns = 1;
    for (int q = 0; q < P.np; ++q) {
        const bool first = q == 0, last = q + 1 == P.np;
        const double2* in = sh + ((q & 1) ? 0 : half);
        double2* out = sh + ((q & 1) ? half : 0);
        auto l2 = [&](int l, int i) { return first ? ld(l, i) : in[at(l, i)]; };
        auto s2 = [&](int l, int i, double2 v) {
            if (last) st(l, i, v);
            else out[at(l, i)] = v;
        };
        switch (P.r[q]) {
            case 2: pass<2, COL>(P, L, ns, l2, s2); break;
            case 3: pass<3, COL>(P, L, ns, l2, s2); break;
            case 4: pass<4, COL>(P, L, ns, l2, s2); break;
            case 5: pass<5, COL>(P, L, ns, l2, s2); break;
            case 7: pass<7, COL>(P, L, ns, l2, s2); break;
            case 8: pass<8, COL>(P, L, ns, l2, s2); break;
            case 11: pass<11, COL>(P, L, ns, l2, s2); break;
            default: pass<13, COL>(P, L, ns, l2, s2); break;
        }
        ns *= P.r[q];
        __syncthreads();
    }
}

__device__ inline double2 swapri(double2 v) { return make_double2(v.y, v.x); }

// x transforms of `rows` complex rows (plane pairs m, rows j): forward from the
// real planes 2m, 2m + 1 of f (a plane past nz counts as zero), inverse (the
// forward transform with real and imaginary parts exchanged on both sides)
// back to them, times scale.
template <bool INV>
__global__ void __launch_bounds__(128) k_fft_x(Line P, int ny, int nz, int rows, int L, const double* f, double2* C, double* out, double scale) {
    extern __shared__ double2 sh[];
    const int n = P.n, r0 = blockIdx.x * L, live = min(L, rows - r0);
    const int pitch = n + (n >> 3) + 1;
    auto at = [&](int l, int i) { return l * pitch + i + (i >> 3); };
    const long long plane = (long long)n * ny;
    auto ld = [&](int l, int i) {
        const int row = r0 + l;
        if (INV) return swapri(C[(long long)row * n + i]);
        const int m = row / ny, j = row - m * ny;
        const long long a = 2 * m * plane + (long long)j * n + i;
        return make_double2(f[a], 2 * m + 1 < nz ? f[a + plane] : 0.0);
    };
    auto st = [&](int l, int i, double2 v) {
        const int row = r0 + l;
        if (!INV) {
            C[(long long)row * n + i] = v;
            return;
        }
        const int m = row / ny, j = row - m * ny;
        const long long a = 2 * m * plane + (long long)j * n + i;
        out[a] = scale * v.y;  // real part
        if (2 * m + 1 < nz) out[a + plane] = scale * v.x;
    };
    transform<false>(P, live, sh, L * pitch, ld, st, at);
}

// y transforms in place: a block takes L neighbouring columns of one complex plane
__global__ void __launch_bounds__(128) k_fft_y(Line P, int nx, int tiles, int L, double2* C, int inv) {
    extern __shared__ double2 sh[];
    const int n = P.n, m = blockIdx.x / tiles, x0 = (blockIdx.x - m * tiles) * L, live = min(L, nx - x0);
    double2* c = C + (long long)m * n * nx + x0;
    auto at = [&](int l, int i) { return i * L + l; };
    auto ld = [&](int l, int i) {
        const double2 v = c[(long long)i * nx + l];
        return inv ? swapri(v) : v;
    };
    auto st = [&](int l, int i, double2 v) { c[(long long)i * nx + l] = inv ? swapri(v) : v; };
    transform<true>(P, live, sh, n * L, ld, st, at);
}

// Tridiagonal systems in z, one per mode (ax, ky), ax = min(kx, nx - kx):
// (e, d, e) with the end rows of a wall-bounded column replaced (d_k = d + e at
// a Neumann wall of cells, d / 2 at a mirrored node row whose equation is
// halved), or cyclic.
__device__ inline void mode_coef(const SpectralZ& Z, int ax, int ky, double& d, double& e) {
    const double lx = Z.lx[ax], ly = Z.ly[ky];
    if (Z.nodal) {
        const double mx = Z.mx[ax], my = Z.my[ky], s = lx * my + mx * ly, t = mx * my;
        e = t * Z.iz2 - (1.0 / 6.0) * s;
        d = -2.0 * t * Z.iz2 - (2.0 / 3.0) * s;
    } else {
        e = Z.iz2;
        d = -(lx + ly) - 2.0 * Z.iz2;
    }
}
__device__ inline double mode_diag(const SpectralZ& Z, int k, double d, double e) {
    if (Z.zper || (k > 0 && k < Z.nz - 1)) return d;
    return Z.nodal ? 0.5 * d : d + e;
}

// The factors of every mode, formed once per handle: the inverse pivots, and
// for cyclic columns (their last unknown eliminated: nu = nz - 1) the column
// w = T^-1 (-e, 0, ..., 0, -e) and the inverse Schur complement.  The mode
// (0, 0) is singular: its last pivot is dropped, which pins the last plane's
// mean to zero.
__global__ void k_modes_setup(SpectralZ Z) {
    const int na = Z.nx / 2 + 1, nk = Z.ny / 2 + 1, M = na * nk;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M) return;
    const int ky = t / na, ax = t - ky * na;
    double d, e;
    mode_coef(Z, ax, ky, d, e);
    const int nu = Z.zper ? Z.nz - 1 : Z.nz;
    double piv = 0.0;
    for (int k = 0; k < nu; ++k) {
        const double dk = mode_diag(Z, k, d, e);
        piv = 1.0 / (k == 0 ? dk : dk - e * e * piv);
        if (t == 0 && !Z.zper && k == nu - 1) piv = 0.0;
        Z.dinv[(long long)k * M + t] = piv;
    }
    if (!Z.zper) return;
    double y = -e;
    Z.w[t] = y;
    for (int k = 1; k < nu; ++k) {
        y = -e * Z.dinv[(long long)(k - 1) * M + t] * y;
        if (k == nu - 1) y -= e;
        Z.w[(long long)k * M + t] = y;
    }
    double x = 0.0;
    for (int k = nu - 1; k >= 0; --k) {
        const double di = Z.dinv[(long long)k * M + t];
        x = Z.w[(long long)k * M + t] * di - e * di * x;
        Z.w[(long long)k * M + t] = x;
    }
    Z.schur[t] = t == 0 ? 0.0 : 1.0 / (d + e * (Z.w[t] + Z.w[(long long)(nu - 1) * M + t]));
}

// The z systems of all modes, in place on the transformed plane pairs C: the
// elimination marches a column up, the substitution down.  The coefficients of
// the real planes 2m and 2m + 1 are
//   A = (C + conj C~) / 2,   B = (C - conj C~) / 2i,
// C~ the entry of the opposite mode (the factor 1/2 is left to the output's
// scale); on the way up the pair's two slots hold the eliminated A and B.
//
// A box has few modes (2080 on 64^3), each a serial chain whose length is its
// FP64 instructions, so two neighbouring lanes share a mode: the systems of the
// real and the imaginary parts are independent.  Lane part 0 holds (Re A, Re B),
// part 1 (Im A, Im B), and they exchange B where C is merged again.  kAhead
// pairs are loaded a group before they are used, and the column's kind is a
// template argument (a branch not taken costs its FP64 issue slots):
// a solve on 64^3 66 -> 40 us, 32^3 30 -> 20, 128x128x64 52 -> 30, 256x256x128
// 131 -> 108.
constexpr int kAhead = 4;
template <int NODAL, int ZPER>
__global__ void __launch_bounds__(64) k_modes_z(SpectralZ Z, double2* C) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, kx = t >> 1, part = t & 1, ky = blockIdx.y;
    const int ox = kx == 0 ? 0 : Z.nx - kx, oy = ky == 0 ? 0 : Z.ny - ky;
    // the pairs of a warp stay together to its end (the exchange below): lanes
    // past the row, and on the other half of a self-conjugate row, idle
    const bool live = kx < Z.nx && !(oy == ky && kx > ox);
    if (!__any_sync(0xffffffffu, live)) return;
    const bool self = oy == ky && ox == kx;
    const int ax = live ? min(kx, Z.nx - kx) : 0, na = Z.nx / 2 + 1, M = na * (Z.ny / 2 + 1), md = ky * na + ax;
    const long long plane = (long long)Z.nx * Z.ny;
    const int nz = Z.nz, np = (nz + 1) / 2, nu = ZPER ? nz - 1 : nz;
    double2* c = C + (long long)ky * Z.nx + (live ? kx : 0);
    double2* o = C + (long long)oy * Z.nx + (live ? ox : 0);
    double d, e;
    mode_coef(Z, ax, ky, d, e);
    const double* dinv = Z.dinv + md;
    // the lane's part of A and B from the entries p of the mode and q of its opposite
    auto sep = [&](double2 p, double2 q, double& a, double& b) {
        a = (part ? p.y : p.x) + (part ? ineg(q.y) : q.x);
        b = (part ? q.x : p.y) + (part ? ineg(p.x) : q.y);
    };
    double last = 0.0;  // cyclic: the eliminated unknown x(nz - 1)
    if (ZPER && live) {
        const double* w = Z.w + md;
        double s = 0.0;
#pragma unroll 4
        for (int m = 0; m < np; ++m) {
            double a, b;
            sep(c[m * plane], o[m * plane], a, b);
            const double w0 = 2 * m < nu ? w[(long long)(2 * m) * M] : 1.0, w1 = 2 * m + 1 < nu ? w[(long long)(2 * m + 1) * M] : 1.0;
            s = fma(w0, a, s);
            s = fma(w1, b, s);
        }
        last = Z.schur[md] * s;
    }
    struct Pair {
        double2 p, q;
        double da, db;
    };
    auto load = [&](int m) {
        Pair r{};
        if (!live || m < 0 || m >= np) return r;
        r.p = c[m * plane];
        r.q = o[m * plane];
        r.da = dinv[(long long)(2 * m) * M];
        r.db = 2 * m + 1 < nu ? dinv[(long long)(2 * m + 1) * M] : 0.0;
        return r;
    };
    // up: z_k = b_k - e dinv_{k-1} z_{k-1}
    double z = 0.0, di = 0.0;
    Pair cur[kAhead], nxt[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) cur[u] = load(u);
    for (int m0 = 0; m0 < np; m0 += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) nxt[u] = load(m0 + kAhead + u);
        __syncwarp();  // both lanes of a mode have read what one of them overwrites
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int m = m0 + u, k = 2 * m;
            if (m >= np) break;
            double a, b;
            sep(cur[u].p, cur[u].q, a, b);
            if (NODAL && !ZPER) {  // the mirrored end rows are halved
                a = k == 0 || k == nz - 1 ? half_of(a) : a;
                b = k + 1 == nz - 1 ? half_of(b) : b;
            }
            if (ZPER && (m == 0 || m >= np - 2)) {  // first and last row
                if (k == 0) a = fma(-e, last, a);
                if (k == nu - 1) a = fma(-e, last, a);
                if (k + 1 == nu - 1) b = fma(-e, last, b);
            }
            a = fma(-e * di, z, a);
            b = fma(-e * cur[u].da, a, b);
            if (live) {
                double* cc = reinterpret_cast<double*>(c + m * plane);
                double* oo = reinterpret_cast<double*>(o + m * plane);
                if (self) {  // both planes' coefficients are real: part 0 keeps them in one slot
                    if (part == 0) {
                        cc[0] = a;
                        cc[1] = b;
                    }
                } else {
                    cc[part] = a;
                    oo[part] = b;
                }
            }
            z = b;
            di = cur[u].db;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) cur[u] = nxt[u];
    }
    // down: x_k = dinv_k z_k - e dinv_k x_{k+1}, and C = A + i B, C~ = conj A + i conj B
    double x = 0.0;
    struct Row {
        double a, b, da, db;
    };
    auto down = [&](int m) {
        Row r{};
        if (!live || m < 0) return r;
        const double* cc = reinterpret_cast<const double*>(c + m * plane);
        const double* oo = reinterpret_cast<const double*>(o + m * plane);
        if (self) {
            r.a = part == 0 ? cc[0] : 0.0;
            r.b = part == 0 ? cc[1] : 0.0;
        } else {
            r.a = cc[part];
            r.b = oo[part];
        }
        r.da = dinv[(long long)(2 * m) * M];
        r.db = 2 * m + 1 < nu ? dinv[(long long)(2 * m + 1) * M] : 0.0;
        return r;
    };
    Row rc[kAhead], rn[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) rc[u] = down(np - 1 - u);
    for (int m0 = np - 1; m0 >= 0; m0 -= kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) rn[u] = down(m0 - kAhead - u);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int m = m0 - u, k = 2 * m;
            if (m < 0) break;
            double a = rc[u].a, b = rc[u].b;
            if (k + 1 < nu) {
                b = rc[u].db * fma(-e, x, b);
                x = b;
            } else {
                b = ZPER && k + 1 < nz ? last : 0.0;  // folded into rows 0 and nz - 2; past the last node plane
            }
            if (!ZPER || k < nu) {
                a = rc[u].da * fma(-e, x, a);
                x = a;
            } else {
                a = last;
            }
            const double y = __shfl_xor_sync(0xffffffffu, b, 1);
            if (live) {
                double* cc = reinterpret_cast<double*>(c + m * plane);
                double* oo = reinterpret_cast<double*>(o + m * plane);
                cc[part] = a + (part ? y : ineg(y));
                if (!self) oo[part] = y + (part ? ineg(a) : a);
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) rc[u] = rn[u];
    }
}

}  // namespace

// radices of a transform length: 8s and 4s first (fewest twiddle products),
// then the odd primes up to 13; false when another prime remains
bool spectral_radices(int n, int& np, int r[12]) {
    np = 0;
    if (n < 2 || n > kSpectralMax) return false;
    int p2 = 0;
    while (n % 2 == 0) {
        n /= 2;
        ++p2;
    }
    while (p2 > 4 || p2 == 3) {
        r[np++] = 8;
        p2 -= 3;
    }
    while (p2 >= 2) {
        r[np++] = 4;
        p2 -= 2;
    }
    if (p2) r[np++] = 2;
    for (int p : {13, 11, 7, 5, 3})
        while (n % p == 0) {
            r[np++] = p;
            n /= p;
        }
    return n == 1;
}

void launch_spectral_setup(Ctx& c, const SpectralZ& Z) {
    const int M = (Z.nx / 2 + 1) * (Z.ny / 2 + 1);
    KS_LAUNCH(c, k_modes_setup, nblocks(M, 128), 128, 8.0 * M * Z.nz, Z);
}

// phi = (unscaled operator)^-1 rhs times scale
void launch_spectral_solve(Ctx& c, const SpectralZ& Z, const double2* tw_x, const double2* tw_y, const double* rhs, double* phi, double* work,
                           double scale) {
    Line X{}, Y{};
    X.n = Z.nx;
    Y.n = Z.ny;
    X.tw = tw_x;
    Y.tw = tw_y;
    spectral_radices(X.n, X.np, X.r);
    spectral_radices(Y.n, Y.np, Y.r);
    double2* C = reinterpret_cast<double2*>(work);
    const int np = (Z.nz + 1) / 2, rows = np * Z.ny;
    const double pts = (double)Z.nx * Z.ny * Z.nz, cb = 16.0 * np * Z.nx * Z.ny;
    // rows a block: about one radix-8 butterfly per thread of 128; columns a
    // block: 8 neighbouring complex values are one 128-byte segment.  Shared
    // memory up to 3072 points a line, two blocks an SM: 98 KB (y), 111 KB (x,
    // whose rows are padded); at 4096 points 131 and 147 KB.
    const int lx = std::max(1, std::min(16, 1024 / X.n)), ly = Y.n <= 384 ? 8 : (Y.n <= 768 ? 4 : (Y.n <= 1536 ? 2 : 1));
    const size_t sx = 2 * sizeof(double2) * (size_t)lx * (X.n + X.n / 8 + 1), sy = 2 * sizeof(double2) * (size_t)ly * Y.n;
    const int tiles = (Z.nx + ly - 1) / ly, gx = (rows + lx - 1) / lx;
    KS_LAUNCH_SMEM(c, k_fft_x<false>, gx, 128, sx, 8.0 * pts + cb, X, Z.ny, Z.nz, rows, lx, rhs, C, (double*)nullptr, 1.0);
    KS_LAUNCH_SMEM(c, k_fft_y, np * tiles, 128, sy, 2.0 * cb, Y, Z.nx, tiles, ly, C, 0);
    const dim3 gz((unsigned)((2 * Z.nx + 63) / 64), (unsigned)(Z.ny / 2 + 1));
    const auto modes = Z.nodal ? (Z.zper ? k_modes_z<1, 1> : k_modes_z<1, 0>) : (Z.zper ? k_modes_z<0, 1> : k_modes_z<0, 0>);
    KS_LAUNCH_NAMED(c, "k_modes_z", modes, gz, 64, 4.0 * cb + 8.0 * 2.0 * (Z.nx / 2 + 1) * (Z.ny / 2 + 1) * Z.nz, Z, C);
    KS_LAUNCH_SMEM(c, k_fft_y, np * tiles, 128, sy, 2.0 * cb, Y, Z.nx, tiles, ly, C, 1);
    KS_LAUNCH_SMEM(c, k_fft_x<true>, gx, 128, sx, 8.0 * pts + cb, X, Z.ny, Z.nz, rows, lx, (const double*)nullptr, C, phi, scale);
}

// the transforms' shared memory above 48 KB has to be allowed once per device
bool spectral_prepare_device() {
    const int most = (int)(2 * sizeof(double2) * (kSpectralMax + kSpectralMax / 8 + 1));
    return cudaFuncSetAttribute(k_fft_x<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess &&
           cudaFuncSetAttribute(k_fft_x<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess &&
           cudaFuncSetAttribute(k_fft_y, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
}

}  // namespace ks
