// Pointwise and stencil passes of the advance: initial fields, Smagorinsky,
// momentum sources, wall model, tensor diffusion (+ RK2 correction), RHS
// assembly, projection updates, CFL / norm reductions and the actuator-disk
// sampling and Gaussian spreading.  One thread per output point; periodic
// wrap and wall boundary conditions are applied inside the kernels (no ghost
// cells are stored).
#include <algorithm>
#include <cmath>

#include "ks_launch.hpp"

namespace ks {

namespace {

constexpr int BS = 256;
constexpr int MAXPARTS = 1216;  // 152 SMs x 8

// cell index -> (i, j, k) in 32-bit arithmetic (grids hold fewer than 2^31
// cells; a 64-bit division costs as much issue as tens of FP64 operations)
__device__ inline void cell_of(const Grid& g, long long t, int& i, int& j, int& k) {
    const unsigned u = (unsigned)t, r = u / (unsigned)g.nx;
    i = (int)(u - r * (unsigned)g.nx);
    k = (int)(r / (unsigned)g.ny);
    j = (int)(r - (unsigned)k * (unsigned)g.ny);
}

template <int OPMAX>
__device__ inline double block_reduce(double v) {
    __shared__ double sh[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_down_sync(0xffffffffu, v, o);
        v = OPMAX ? nmax(v, x) : v + x;
    }
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    v = (threadIdx.x < nw) ? sh[threadIdx.x] : (OPMAX ? -1.0e300 : 0.0);
    if (w == 0)
        for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_down_sync(0xffffffffu, v, o);
            v = OPMAX ? nmax(v, x) : v + x;
        }
    return v;
}

inline int parts_for(long long n) {
    long long b = (n + BS - 1) / BS;
    return (int)(b < MAXPARTS ? (b < 1 ? 1 : b) : MAXPARTS);
}

__device__ inline uint64_t splitmix64(uint64_t x) {
    uint64_t z = x + 0x9e3779b97f4a7c15ULL;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

// ---------------------------------------------------------------- init
// TaylorGreenVortex::initialize_fields (src/physics/TaylorGreenVortex.cpp:22-54)
__global__ void k_init_tgv(Grid g, double* vel, double x0, double y0, double z0, double Lx, double Ly, double Lz) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    const double tp = 6.283185307179586476925;
    const double x = x0 + (i + 0.5) * g.dx, y = y0 + (j + 0.5) * g.dy, z = z0 + (k + 0.5) * g.dz;
    vel[t] = sin(tp * x / Lx) * cos(tp * y / Ly) * cos(tp * z / Lz);
    vel[g.N + t] = -cos(tp * x / Lx) * sin(tp * y / Ly) * cos(tp * z / Lz);
    vel[2 * g.N + t] = 0.0;
}

// Synthetic ABL / free-stream start: log-law or uniform mean plus uniform
// noise of amplitude amp below zmax, SplitMix64 keyed on (seed, comp, k, j, i).
__global__ void k_init_abl(Grid g, double* vel, int loglaw, double U0, double U1, double U2, double ut_k, double z0, double amp,
                           double zmax_rel, unsigned long long seed) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    const double z = (k + 0.5) * g.dz;
    const double U[3] = {U0, U1, U2};
    for (int n = 0; n < 3; ++n) {
        double val = U[n];
        if (loglaw) val = (n == 0) ? ut_k * log(z / z0) : 0.0;
        if (amp > 0.0 && z < zmax_rel) {
            const uint64_t idx = (uint64_t)n * (uint64_t)g.N + (uint64_t)t;
            const uint64_t r = splitmix64(seed * 0x100000001b3ULL ^ idx);
            const double u01 = (double)(r >> 11) * (1.0 / 9007199254740992.0);
            val += amp * (2.0 * u01 - 1.0);
        }
        vel[n * g.N + t] = val;
    }
}

__global__ void k_fill(double* p, double v, long long n) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < n) p[t] = v;
}
__global__ void k_copy(double* d, const double* s, long long n) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t < n) d[t] = s[t];
}

// ---------------------------------------------------------------- Smagorinsky
// mu_eff = mu + rho Cs^2 Delta^2 |S| (src/turbulence/LES/Smagorinsky.cpp:22-62,
// strain rate src/fvm/strainrate.H:24-86, one-sided z stencils at walls
// src/fvm/stencils.H:166-330).
// alpha_eff = mu / Pr + mu_t / Pr_t (TurbModelBase.H:28-35) when alpha is set.
// Where the model is off both are the molecular values.
__global__ void k_mu_molecular(long long N, double* mueff, double mu, double* alpha, double mu_pr) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= N) return;
    mueff[t] = mu;
    if (alpha) alpha[t] = mu_pr;
}

// FP64 form: columns marched in z, the column's own values carried and the
// neighbour offsets formed once, as the FP64 issue of about 27 instructions and
// a square root (7.5 more) should bound it, not the index maps of the 18 reads
// of the thread-per-cell form (256x256x128: 1400 us, 575 now).
__global__ void __launch_bounds__(128) k_smag_col(Grid g, const double* vel, double* mueff, double mu, double rhofac, double* alpha, double mu_pr,
                                                  double iprt, int kc) {
    int i, j;
    if (!column_of(g, i, j)) return;
    const int k0 = blockIdx.y * kc, k1 = min(k0 + kc, g.nz);
    const long long N = g.N;
    const int sz = g.nx * g.ny;
    const int xp = i + 1 == g.nx ? 1 - g.nx : 1, xm = i == 0 ? g.nx - 1 : -1;
    const int yp = (j + 1 == g.ny ? 1 - g.ny : 1) * g.nx, ym = (j == 0 ? g.ny - 1 : -1) * g.nx;
    const VelFPT<double, double> V{vel, g, 1.0};
    const double hx = 0.5 * g.idx, hy = 0.5 * g.idy, hz = 0.5 * g.idz;
    const double* p = vel + (long long)k0 * sz + j * g.nx + i;
    double dn[3], at[3];
    for (int n = 0; n < 3; ++n) {
        dn[n] = V(n, i, j, k0 - 1);
        at[n] = p[n * N];
    }
    for (int k = k0; k < k1; ++k, p += sz) {
        double up[3], gz[3], sxy, syz, szx;
        for (int n = 0; n < 3; ++n) up[n] = k + 1 < g.nz ? p[n * N + sz] : V(n, i, j, k + 1);
        const double ux = hx * (p[xp] - p[xm]), vy = hy * (p[N + yp] - p[N + ym]);
        sxy = hy * (p[yp] - p[ym]) + hx * (p[N + xp] - p[N + xm]);
        const double wx = p[2 * N + xp] - p[2 * N + xm], wy = p[2 * N + yp] - p[2 * N + ym];
        if (!g.zper && (k == 0 || k == g.nz - 1)) {  // one-sided through the wall (ghost) value
            double a = 1.0 / 3.0, b = 1.0, c = -4.0 / 3.0;
            if (k == g.nz - 1) { a = 4.0 / 3.0; b = -1.0; c = -1.0 / 3.0; }
            for (int n = 0; n < 3; ++n) gz[n] = (a * up[n] + b * at[n] + c * dn[n]) * g.idz;
            syz = gz[1] + hy * wy;
            szx = hx * wx + gz[0];
        } else {
            syz = hz * (up[1] - dn[1]) + hy * wy;
            szx = hx * wx + hz * (up[0] - dn[0]);
            gz[2] = hz * (up[2] - dn[2]);
        }
        const double s = sqrt(2.0 * (ux * ux + vy * vy + gz[2] * gz[2]) + (sxy * sxy + syz * syz + szx * szx));
        const double mut = rhofac * s;
        const long long t = ((long long)k * g.ny + j) * g.nx + i;
        mueff[t] = mu + mut;
        if (alpha) alpha[t] = mu_pr + iprt * mut;
        for (int n = 0; n < 3; ++n) {
            dn[n] = at[n];
            at[n] = up[n];
        }
    }
}

// Mixed-precision form: the same march over the FP32 copy of the velocity.  Its
// values come from L1 (15 loads a cell), the strain rate is FP32 throughout, and
// mu_eff is formed in FP64.  The sums are written out operation by operation: the
// FP32 advection's branches follow every bit of the step, so the bits are kept
// whatever the compiler would contract.  256x256x128: 230 us as tiles of 32 x 4 x 4
// cells, whose staging spent four integer remainders on each of 2.4 values a
// cell, 72 now; 512x512x256 1798 and 473.
__global__ void __launch_bounds__(128) k_smag_march(Grid g, const float* vel, double* mueff, double mu, double rhofac, double* alpha,
                                                    double mu_pr, double iprt, int kc) {
    int i, j;
    if (!column_of(g, i, j)) return;
    const int k0 = blockIdx.y * kc, k1 = min(k0 + kc, g.nz);
    const long long N = g.N;
    const int sz = g.nx * g.ny;
    const int xp = i + 1 == g.nx ? 1 - g.nx : 1, xm = i == 0 ? g.nx - 1 : -1;
    const int yp = (j + 1 == g.ny ? 1 - g.ny : 1) * g.nx, ym = (j == 0 ? g.ny - 1 : -1) * g.nx;
    const VelFPT<float, float> V{vel, g, 1.0f};
    const float hx = 0.5f * d2f(g.idx), hy = 0.5f * d2f(g.idy), hz = 0.5f * d2f(g.idz), iz = d2f(g.idz);
    const float* p = vel + (long long)k0 * sz + j * g.nx + i;
    long long t = (long long)k0 * sz + j * g.nx + i;
    float dn[3], at[3];
    for (int n = 0; n < 3; ++n) {
        dn[n] = V(n, i, j, k0 - 1);
        at[n] = p[n * N];
    }
    for (int k = k0; k < k1; ++k, p += sz, t += sz) {
        float up[3], gx[3], gy[3], gz[3];
        for (int n = 0; n < 3; ++n) up[n] = k + 1 < g.nz ? p[n * N + sz] : V(n, i, j, k + 1);
        for (int n = 0; n < 3; ++n) {
            const float* v = p + n * N;
            gx[n] = hx * (v[xp] - v[xm]);
            gy[n] = hy * (v[yp] - v[ym]);
        }
        if (!g.zper && (k == 0 || k == g.nz - 1)) {  // one-sided through the wall (ghost) value
            float a = 1.0f / 3.0f, b = 1.0f, c = -4.0f / 3.0f;
            if (k == g.nz - 1) { a = 4.0f / 3.0f; b = -1.0f; c = -1.0f / 3.0f; }
            for (int n = 0; n < 3; ++n) gz[n] = fmaf(c, dn[n], fmaf(a, up[n], b * at[n])) * iz;
        } else {
            for (int n = 0; n < 3; ++n) gz[n] = hz * (up[n] - dn[n]);
        }
        const float sxy = __fadd_rn(gy[0], gx[1]), syz = __fadd_rn(gz[1], gy[2]), szx = __fadd_rn(gx[2], gz[0]);
        const float s2 = fmaf(gz[2], gz[2], fmaf(gx[0], gx[0], gy[1] * gy[1])), t2 = fmaf(szx, szx, fmaf(sxy, sxy, syz * syz));
        const float s = sqrtf(fmaf(2.0f, s2, t2));
        const double mut = rhofac * f2d(s);
        mueff[t] = __dadd_rn(mu, mut);
        if (alpha) alpha[t] = fma(iprt, mut, mu_pr);
        for (int n = 0; n < 3; ++n) {
            dn[n] = at[n];
            at[n] = up[n];
        }
    }
}

// ---------------------------------------------------------------- sources
// src = rho (-gp/rho + geostrophic + Coriolis(u_old) + body + actuator)
// (icns_ops.H:78-124, PDEOps.H:94-145, GeostrophicForcing.cpp:103-,
// CoriolisForcing.cpp:60-108, BodyForce.cpp:117-169, ActuatorForcing.cpp:19-29)
// The sources are affine in the Old velocity, so the launcher folds them on
// the host: src_n = (c_n - gp_n) + sum_m M_nm u_m + rho act_n + rho g_n beta (T0 - theta),
// with c = rho (geostrophic + body + ABLForcing) and M = rho x the Coriolis
// map.  About 12 FP64 instructions per cell where the term-by-term form took 45.
struct SrcCoef {
    double c[3];
    double M[3][3];
    double rho, bous_g[3], T_ref;
};
// Which terms run is a template argument: as a run-time flag each absent term
// still took its FP64 issue slots, predicated off (22 for 12 a cell: 351 us on
// 256x256x128, 200 now).
template <int COR, int ACT, int BOUS, int PLAIN>
__global__ void k_sources(Grid g, const double* vel, const double* gp, const double* act, double* src, SrcCoef s, const double* theta) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    const long long N = g.N;
    double f[3];
    for (int n = 0; n < 3; ++n) f[n] = s.c[n] - gp[n * N + t];
    if (COR) {
        const double u0 = vel[t], u1 = vel[N + t], u2 = vel[2 * N + t];
        for (int n = 0; n < 3; ++n) {
            if constexpr (PLAIN) f[n] += s.M[n][0] * u0 + s.M[n][1] * u1 + s.M[n][2] * u2;
            else f[n] = fma(s.M[n][2], u2, fma(s.M[n][1], u1, fma(s.M[n][0], u0, f[n])));
        }
    }
    if (ACT)
        for (int n = 0; n < 3; ++n) f[n] += s.rho * act[n * N + t];
    if (BOUS) {  // BoussinesqBuoyancy.cpp:22-50: rho g beta (T0 - theta)
        const double dT = s.T_ref - theta[t];
        for (int n = 0; n < 3; ++n) f[n] += s.bous_g[n] * dT;
    }
    for (int n = 0; n < 3; ++n) src[n * N + t] = f[n];
}

// ---------------------------------------------------------------- ABL wall
// plane sums over the first cell layer: u, v, |u_h|
__global__ void k_plane_sums(Grid g, const double* vel, double* parts, int np) {
    double su = 0, sv = 0, sm = 0;
    const long long M = (long long)g.nx * g.ny;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < M; t += (long long)gridDim.x * blockDim.x) {
        const double u = vel[t], v = vel[g.N + t];
        su += u; sv += v; sm += sqrt(u * u + v * v);
    }
    su = block_reduce<0>(su);
    sv = block_reduce<0>(sv);
    sm = block_reduce<0>(sm);
    if (threadIdx.x == 0) { parts[blockIdx.x] = su; parts[np + blockIdx.x] = sv; parts[2 * np + blockIdx.x] = sm; }
}

// wall-normal gradient of the tangential velocity at z-lo: tau rho / mu_eff
// (ABLWallFunction.cpp:236-347, ShearStress.H:22-167), Old velocity.
__global__ void k_wall_grad(Grid g, const double* vel, const double* mueff, double* wg, int type, double ut2, double um0, double um1,
                            double vm, double rho) {
    const long long M = (long long)g.nx * g.ny;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= M) return;
    const double u = vel[t], v = vel[g.N + t];
    const double ws = sqrt(u * u + v * v);
    double tx, ty;
    if (type == 0) {  // moeng
        tx = ((u - um0) * vm + ws * um0) / (vm * vm) * ut2;
        ty = ((v - um1) * vm + ws * um1) / (vm * vm) * ut2;
    } else if (type == 1) {  // constant
        tx = um0 / vm * ut2;
        ty = um1 / vm * ut2;
    } else if (type == 2) {  // local
        tx = u / fmax(ws, 1.0e-6) * ut2;
        ty = v / fmax(ws, 1.0e-6) * ut2;
    } else {  // schumann
        tx = u / vm * ut2;
        ty = v / vm * ut2;
    }
    const double m = mueff[t];
    wg[t] = tx * rho / m;
    wg[M + t] = ty * rho / m;
}

// ---------------------------------------------------------------- diffusion
// Velocity seen by the tensor operator: periodic wrap; across a z wall the
// normal component is odd-reflected (Dirichlet 0), the tangential ones are
// even-reflected (Neumann) or shifted so that the face gradient equals the
// wall-model gradient (inhomogeneous Neumann).
struct VelDiff {
    const double* v;
    const double* wg;
    Grid g;
    __device__ inline double operator()(int n, int i, int j, int k) const {
        i = wrapn(i, g.nx);
        j = wrapn(j, g.ny);
        const double* c = v + n * g.N;
        if (g.zper) return c[cidx(g, i, j, wrapn(k, g.nz))];
        if (k < 0) {
            const double q0 = c[cidx(g, i, j, 0)];
            if (n == 2) return -q0;
            if (g.zlo == ZWALLMODEL) return q0 - wg[(long long)n * g.nx * g.ny + (long long)j * g.nx + i] * g.dz;
            return q0;
        }
        if (k >= g.nz) {
            const double q0 = c[cidx(g, i, j, g.nz - 1)];
            return n == 2 ? -q0 : q0;
        }
        return c[cidx(g, i, j, k)];
    }
};

// Flux of mu (grad u + grad u^T) - 2/3 mu div(u) I through the d-face at the
// low side of cell (i,j,k).
__device__ inline void tensor_flux(const Grid& g, const VelDiff& V, const double* mu, int d, int i, int j, int k, double F[3]) {
    int e[3] = {0, 0, 0};
    e[d] = 1;
    const int im = i - e[0], jm = j - e[1], km = k - e[2];
    // face viscosity
    double mf;
    const long long cc = cidx(g, wrapn(i, g.nx), wrapn(j, g.ny), g.zper ? wrapn(k, g.nz) : (k < g.nz ? k : g.nz - 1));
    if (d == 2 && !g.zper && k == 0) mf = mu[cidx(g, wrapn(i, g.nx), wrapn(j, g.ny), 0)];
    else if (d == 2 && !g.zper && k == g.nz) mf = mu[cidx(g, wrapn(i, g.nx), wrapn(j, g.ny), g.nz - 1)];
    else {
        const long long cm = cidx(g, wrapn(im, g.nx), wrapn(jm, g.ny), g.zper ? wrapn(km, g.nz) : km);
        mf = 0.5 * (mu[cm] + mu[cc]);
    }
    const double ih[3] = {g.idx, g.idy, g.idz};
    double gr[3][3];  // gr[m][n] = d u_n / d x_m on the face
    for (int n = 0; n < 3; ++n) {
        for (int m = 0; m < 3; ++m) {
            if (m == d) {
                gr[m][n] = (V(n, i, j, k) - V(n, im, jm, km)) * ih[m];
            } else {
                int f[3] = {0, 0, 0};
                f[m] = 1;
                gr[m][n] = 0.25 *
                           (V(n, i + f[0], j + f[1], k + f[2]) + V(n, im + f[0], jm + f[1], km + f[2]) - V(n, i - f[0], j - f[1], k - f[2]) -
                            V(n, im - f[0], jm - f[1], km - f[2])) *
                           ih[m];
            }
        }
    }
    const double dv = gr[0][0] + gr[1][1] + gr[2][2];
    for (int n = 0; n < 3; ++n) {
        if (n == d) F[n] = mf * (2.0 * gr[d][d] - (2.0 / 3.0) * dv);
        else F[n] = mf * (gr[d][n] + gr[n][d]);
    }
}

// Tensor fluxes on the d-faces, all three components, computed once per face.
__global__ void k_tau_flux(Grid g, int d, const double* vel, const double* mueff, const double* wg, double* F0, double* F1, double* F2) {
    const int nzl = (d == 2) ? nzfaces(g) : g.nz;
    const long long M = (long long)g.nx * g.ny * nzl;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= M) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    VelDiff V{vel, wg, g};
    double F[3];
    tensor_flux(g, V, mueff, d, i, j, k, F);
    const long long f = fidx(g, d, i, j, k);
    F0[f] = F[0];
    F1[f] = F[1];
    F2[f] = F[2];
}

struct Flux9 {
    const double* p[9];
};

// divtau = sum_d (F_d(c + e_d) - F_d(c)) / h_d ; mode 0: store; mode 1: also
// forces = (src + divtau)/rho; mode 2: out = base + 0.5 dt (divtau - dold)/rho
__global__ void k_tau_div(Grid g, Flux9 F, double* out, int mode, const double* src, double* forces, const double* base,
                          const double* dold, double dt, double rho) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    const double ih[3] = {g.idx, g.idy, g.idz};
    const double irho = 1.0 / rho;  // once per thread
    double acc[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) {
        const long long lo = fidx(g, d, i, j, k), hi = fidx(g, d, i + (d == 0), j + (d == 1), k + (d == 2));
        for (int n = 0; n < 3; ++n) acc[n] += (F.p[3 * d + n][hi] - F.p[3 * d + n][lo]) * ih[d];
    }
    const long long N = g.N;
    if (mode == 0) {
        for (int n = 0; n < 3; ++n) out[n * N + t] = acc[n];
    } else if (mode == 1) {
        for (int n = 0; n < 3; ++n) {
            out[n * N + t] = acc[n];
            forces[n * N + t] = (src[n * N + t] + acc[n]) * irho;
        }
    } else {
        for (int n = 0; n < 3; ++n) out[n * N + t] = base[n * N + t] + 0.5 * dt * (acc[n] - dold[n * N + t]) * irho;
    }
}

// ---- fused tiled form of k_tau_flux + k_tau_div.  A block owns a
// TX x TY x TZ tile of cells; it stages the velocity seen by the flux stencil
// (VelDiff, ghosts included) and mu_eff for the tile plus a one-cell halo in
// shared memory, computes every face flux the tile needs once (the same
// arithmetic as tensor_flux) into shared memory, then forms the divergence
// and the mode epilogue of k_tau_div for its cells.  No face arrays touch HBM.
// Bound by instruction issue and shared memory: with wrap_tile in place of four
// remainders for each of 2.4 staged values a cell 395 -> 328 us on 256x256x128,
// 3.20 -> 2.62 ms on 512x512x256 (a z march over 32 x 8 columns took 468 us and
// 3.68 ms: its larger blocks leave too few warps to hide a layer's latency).
constexpr int TTX = 32, TTY = 4, TTZ = 4;
constexpr int THX = TTX + 2, THY = TTY + 2, THZ = TTZ + 2;
constexpr int TNH = THX * THY * THZ;
constexpr int TNFX = (TTX + 1) * TTY * TTZ, TNFY = TTX * (TTY + 1) * TTZ, TNFZ = TTX * TTY * (TTZ + 1);
constexpr size_t tau_smem() { return sizeof(float) * (4 * (size_t)TNH + 3 * ((size_t)TNFX + TNFY + TNFZ)); }

// Epilogue of the tensor-diffusion kernels (acc = divtau(vel) of a cell):
//   0: out = acc
//   1: out = acc, forces = (src + acc) / rho
//   2: out = base + 0.5 dt (acc - dold) / rho                        (explicit RK2 correction)
//   3: out = (rho base + dt (0.5 (conv_o + conv_n) + 0.5 (dold + acc) + src)) / rho  (MOL corrector_rhs)
//   7: out = x + omega dinv (base - rho x + dt acc), x = vel           (Jacobi sweep of rho x - dt divtau x = base)
//   8: out = base - rho x + dt acc                                    (its residual)
// Modes 7 and 8 write block maxima of the residual's magnitude to parts when it is set.
struct TauEpi {
    int mode;
    const double *src, *base, *dold, *conv_o, *conv_n, *dinv;
    double* forces;
    double* parts;
    double dt, rho, omega;
    double irho;  // 1 / rho, formed on the host
    double hdr;   // dt / (2 rho)
    double hdt;   // dt / 2
};

// FP32 form (mixed precision, modes 0-2): staged values, face fluxes and their
// arithmetic are FP32, the FP64 inputs rounded once when staged; the epilogue
// runs in FP64.
template <int MODE, int V32>
__global__ void __launch_bounds__(TTX* TTY* TTZ) k_divtau_tile(Grid g, const double* vel, const float* vel32, const double* mueff, const double* wg, double* out,
                                                               TauEpi E) {
    using T = float;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* sm = reinterpret_cast<T*>(sm_raw);
    T* sV = sm;                // [3][THZ][THY][THX]
    T* sM = sm + 3 * TNH;      // [THZ][THY][THX]
    T* sFx = sm + 4 * TNH;     // [3][TTZ][TTY][TTX + 1]
    T* sFy = sFx + 3 * TNFX;   // [3][TTZ][TTY + 1][TTX]
    T* sFz = sFy + 3 * TNFY;   // [3][TTZ + 1][TTY][TTX]
    const int i0 = blockIdx.x * TTX, j0 = blockIdx.y * TTY, k0 = blockIdx.z * TTZ;
    const int tid = threadIdx.x;
    const int nthr = TTX * TTY * TTZ;
    const VelDiff V{vel, wg, g};
    auto hidx = [](int hx, int hy, int hz) { return (hz * THY + hy) * THX + hx; };
    for (int h = tid; h < TNH; h += nthr) {
        const int hx = h % THX, hy = (h / THX) % THY, hz = h / (THX * THY);
        // a tile may be wider than the grid (nx < TTX): wrap x, y (and periodic z) fully
        const int gi = wrap_tile(i0 + hx - 1, g.nx), gj = wrap_tile(j0 + hy - 1, g.ny);
        int gk = k0 + hz - 1;
        if (g.zper) gk = wrap_tile(gk, g.nz);
        if (V32 && gk >= 0 && gk < g.nz) {
            const long long c = cidx(g, gi, gj, gk);
            for (int n = 0; n < 3; ++n) sV[n * TNH + h] = vel32[n * g.N + c];
        } else {  // no FP32 copy, or a ghost across a wall (formed in FP64)
            for (int n = 0; n < 3; ++n) sV[n * TNH + h] = d2f(V(n, gi, gj, gk));
        }
        const int kk = g.zper ? gk : (gk < 0 ? 0 : (gk >= g.nz ? g.nz - 1 : gk));
        sM[h] = d2f(mueff[cidx(g, gi, gj, kk)]);
    }
    __syncthreads();
    const T ih[3] = {d2f(g.idx), d2f(g.idy), d2f(g.idz)};
    const T qh[3] = {T(0.25) * ih[0], T(0.25) * ih[1], T(0.25) * ih[2]};
    // flux through the d-face at the low side of halo cell (hx, hy, hz)
    auto flux = [&](int d, int hx, int hy, int hz, int gk, T F[3]) {
        const int e0 = (d == 0), e1 = (d == 1), e2 = (d == 2);
        const int mx = hx - e0, my = hy - e1, mz = hz - e2;
        T mf;
        if (d == 2 && !g.zper && gk == 0) mf = sM[hidx(hx, hy, hz)];
        else if (d == 2 && !g.zper && gk == g.nz) mf = sM[hidx(mx, my, mz)];
        else mf = T(0.5) * (sM[hidx(mx, my, mz)] + sM[hidx(hx, hy, hz)]);
        T gr[3][3];
        const int hc = hidx(hx, hy, hz), hm = hidx(mx, my, mz);
        for (int n = 0; n < 3; ++n) {
            const T* v = sV + n * TNH;
            for (int m = 0; m < 3; ++m) {
                if (m == d) {
                    gr[m][n] = (v[hc] - v[hm]) * ih[m];
                } else {  // mean of the two cells' central differences along m
                    const int f = m == 0 ? 1 : (m == 1 ? THX : THX * THY);
                    gr[m][n] = qh[m] * ((v[hc + f] + v[hm + f]) - (v[hc - f] + v[hm - f]));
                }
            }
        }
        const T dv = gr[0][0] + gr[1][1] + gr[2][2];
        for (int n = 0; n < 3; ++n) {
            if (n == d) F[n] = mf * (T(2) * gr[d][d] - T(2.0 / 3.0) * dv);
            else F[n] = mf * (gr[d][n] + gr[n][d]);
        }
    };
    for (int f = tid; f < TNFX + TNFY + TNFZ; f += nthr) {
        T F[3];
        if (f < TNFX) {
            const int fx = f % (TTX + 1), fy = (f / (TTX + 1)) % TTY, fz = f / ((TTX + 1) * TTY);
            flux(0, fx + 1, fy + 1, fz + 1, k0 + fz, F);
            for (int n = 0; n < 3; ++n) sFx[n * TNFX + f] = F[n];
        } else if (f < TNFX + TNFY) {
            const int q = f - TNFX;
            const int fx = q % TTX, fy = (q / TTX) % (TTY + 1), fz = q / (TTX * (TTY + 1));
            flux(1, fx + 1, fy + 1, fz + 1, k0 + fz, F);
            for (int n = 0; n < 3; ++n) sFy[n * TNFY + q] = F[n];
        } else {
            const int q = f - TNFX - TNFY;
            const int fx = q % TTX, fy = (q / TTX) % TTY, fz = q / (TTX * TTY);
            flux(2, fx + 1, fy + 1, fz + 1, k0 + fz, F);
            for (int n = 0; n < 3; ++n) sFz[n * TNFZ + q] = F[n];
        }
    }
    __syncthreads();
    const int tx = tid % TTX, ty = (tid / TTX) % TTY, tz = tid / (TTX * TTY);
    const int i = i0 + tx, j = j0 + ty, k = k0 + tz;
    const bool live = i < g.nx && j < g.ny && k < g.nz;
    const double irho = E.irho, hdt = E.hdt;
    const long long N = g.N, t = live ? cidx(g, i, j, k) : 0;
    for (int n = 0; n < 3 && live; ++n) {
        const int ax = (tz * TTY + ty) * (TTX + 1) + tx;
        const int ay = (tz * (TTY + 1) + ty) * TTX + tx;
        const int az = (tz * TTY + ty) * TTX + tx;
        T acc_t = (sFx[n * TNFX + ax + 1] - sFx[n * TNFX + ax]) * ih[0];
        acc_t += (sFy[n * TNFY + ay + TTX] - sFy[n * TNFY + ay]) * ih[1];
        acc_t += (sFz[n * TNFZ + az + TTX * TTY] - sFz[n * TNFZ + az]) * ih[2];
        const double acc = f2d(acc_t);
        const long long m = n * N + t;
        if constexpr (MODE == 0) {
            out[m] = acc;
        } else if constexpr (MODE == 1) {
            out[m] = acc;
            E.forces[m] = (E.src[m] + acc) * irho;
        } else {
            out[m] = E.base[m] + hdt * (acc - E.dold[m]) * irho;
        }
    }
}

// ---- FP64 form: columns marched in z.  The kernel is bound by FP64 issue, so
// it spends as few FP64 instructions a cell as the term allows:
// - a face's transverse derivatives are means of its two cells' central
//   differences, so each cell's differences are formed once (nine subtractions,
//   three of them merged in pairs into the part of the divergence that a
//   direction's face needs) and both faces of the cell in a direction add them;
// - grid spacings are ratios folded into one FMA per component, and the face
//   viscosity carries 1 / h^2 of the flux's own direction, so a flux enters the
//   divergence by a subtraction alone;
// - a march keeps the z faces and the in-plane differences of the next layer.
// 79 FP64 instructions a cell with an epilogue, 5.6 for the halo and 26 a column
// at the start of a march (counters, 256x256x64: 90.2 a cell), where the tile
// kernel's per-face differences, repeated on the tile's halo, took about 130.
// A block owns 32 x TY columns and keeps three layers of the velocity (with a
// one-cell halo) and two of the viscosity in shared memory; the layer after
// next is loaded while the current one is computed.  Its warps: one per row of
// columns; one each for the row below and above (the cell differences the y
// faces need, and the upper row's faces); one for the columns left (lanes 0 ..)
// and right (lanes 16 ..) of the block.
// On 256x256x128: 2.25 ms as tiles (96 % of the FP64 issue rate), 1.50 ms now.
//
// WX < 32 (boxes of at most 16 columns in x, MODE 0): a warp holds 32 / WX rows
// of WX columns, a block one such warp and the three of the halo.  On 32 lanes
// a row of 4 leaves 28 idle: 4x256x256 351 us and 4x4x16384 621, where fluxes
// formed face by face take 158 and 146 (193 and 183 under walls); 72 and 129 now.
template <int TY, int WX>
struct TauPlanes {
    static constexpr int NR = TY * (32 / WX);  // rows of a block
    double V[3][3][NR + 2][WX + 2];  // [layer mod 3][component]: row and column 0 are the halo
    double M[2][NR + 2][WX + 2];     // [layer mod 2]
    double QX[3][NR][WX + 2];        // cell differences for x faces: divergence part, du/dy, du/dz
    double QY[3][NR + 2][WX];        // for y faces: divergence part, dv/dx, dv/dz
    double FX[3][NR][WX + 1], FY[3][NR + 1][WX];
};
struct TauCoef {                  // spacing ratios (see k_divtau_col)
    double gx, gy, gz;            // 1 / (2 h^2)
    double xy, xz, yx, yz, zx, zy;  // transverse weights: hx / (4 hy) on x faces, ...
    double lx, ly, lz;            // -hx / (8 hy), -hy / (8 hx), -hz / (8 hx)
    double ryz, rxz, rxy;         // hy / hz, hx / hz, hx / hy
};
inline TauCoef tau_coef(const Grid& g) {
    const double x = g.dx, y = g.dy, z = g.dz;
    return TauCoef{0.5 * g.idx * g.idx, 0.5 * g.idy * g.idy, 0.5 * g.idz * g.idz, 0.25 * x / y, 0.25 * x / z, 0.25 * y / x, 0.25 * y / z,
                   0.25 * z / x,        0.25 * z / y,        -0.125 * x / y,      -0.125 * y / x, -0.125 * z / x, y / z, x / z, x / y};
}

constexpr int kNarrowBlocks = 6;  // blocks of the narrow forms on an SM

// MODE (TauEpi) is a template argument: the other modes' instructions, predicated
// off, took 7 of 92 FP64 issue slots a cell.
template <int TY, int MODE, int WX>
__global__ void __launch_bounds__(32 * (TY + 3), WX == 32 ? 2 : kNarrowBlocks) k_divtau_col(Grid g, TauCoef K, const double* vel, const double* mueff,
                                                                                           const double* wg, double* out, TauEpi E, int kc) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    TauPlanes<TY, WX>& S = *reinterpret_cast<TauPlanes<TY, WX>*>(sm_raw);
    constexpr int NR = TauPlanes<TY, WX>::NR;
    static_assert((NR + 2) * (WX + 2) <= 32 * (TY + 3), "a thread stages one column");
    const int tid = threadIdx.x, w = tid >> 5, l = tid & 31;
    const int i0 = blockIdx.x * WX, j0 = blockIdx.y * NR, k0 = blockIdx.z * kc, k1 = min(k0 + kc, g.nz);
    const long long N = g.N;
    const int sz = g.nx * g.ny;
    // ---- staging: thread tid loads one column of the (NR + 2) x (WX + 2) footprint
    // (a block may be wider than the grid: x and y wrap fully)
    const bool loads = tid < (NR + 2) * (WX + 2);
    const int lx = tid % (WX + 2), ly = tid / (WX + 2);
    const int col = loads ? (((j0 + ly - 1) % g.ny + g.ny) % g.ny) * g.nx + ((i0 + lx - 1) % g.nx + g.nx) % g.nx : 0;
    struct Cell {
        double v[3], m;
    };
    auto fetch = [&](int k) {  // layer -1 and nz are the ghosts VelDiff gives
        Cell c;
        const int kk = g.zper ? (k < 0 ? k + g.nz : (k >= g.nz ? k - g.nz : k)) : (k < 0 ? 0 : (k >= g.nz ? g.nz - 1 : k));
        const double* p = vel + (long long)kk * sz + col;
        for (int n = 0; n < 3; ++n) c.v[n] = p[n * N];
        c.m = mueff[(long long)kk * sz + col];
        if (!g.zper && (k < 0 || k >= g.nz)) {
            c.v[2] = ineg(c.v[2]);
            if (k < 0 && g.zlo == ZWALLMODEL)
                for (int n = 0; n < 2; ++n) c.v[n] -= wg[(long long)n * sz + col] * g.dz;
        }
        return c;
    };
    auto stage = [&](const Cell& c, int s, int k) {
        for (int n = 0; n < 3; ++n) S.V[s][n][ly][lx] = c.v[n];
        S.M[k & 1][ly][lx] = c.m;
    };
    int sm = 0, sc = 1, sp = 2;  // slots of layers k - 1, k, k + 1
    double mu = 0.0;             // viscosity of layer k - 1, then k, of the thread's column
    if (loads) {
        const Cell c = fetch(k0 - 1);
        stage(c, sm, k0 - 1);
    }
    __syncthreads();
    const bool mainw = w < TY;
    const int y = w * (32 / WX) + l / WX + 1, x = l % WX + 1;
    // the halo's warps: lanes of the rows below and above, then of the columns
    // left and right of the block
    constexpr int kSide = 2 * WX < 32 ? 32 : 2 * WX, kHalf = NR < 16 ? 16 : NR;
    static_assert(kSide + 2 * kHalf <= 96, "three warps hold the halo");
    const int h = tid - 32 * TY, hq = h - kSide;
    const int yh = h < WX ? 0 : NR + 1, xh = h % WX + 1;
    const int sr = hq % kHalf, sx = hq < kHalf ? 0 : WX + 1;
    const bool side = hq >= 0 && hq < 2 * kHalf && sr < NR;
    if (mainw) mu = S.M[(k0 - 1) & 1][y][x];
    __syncthreads();
    if (loads) {
        const Cell a = fetch(k0), b = fetch(k0 + 1);
        stage(a, sc, k0);
        stage(b, sp, k0 + 1);
    }
    __syncthreads();
    // in-plane differences of a layer: du/dx, dv/dy, their part of the
    // divergence in units of du/dx, dw/dx, dw/dy
    struct Plane {
        double dx, dy, c, wx, wy, v[3];
    };
    auto plane = [&](int s) {
        Plane q;
        for (int n = 0; n < 3; ++n) q.v[n] = S.V[s][n][y][x];
        q.dx = S.V[s][0][y][x + 1] - S.V[s][0][y][x - 1];
        q.dy = S.V[s][1][y + 1][x] - S.V[s][1][y - 1][x];
        q.c = q.dx + K.rxy * q.dy;
        q.wx = S.V[s][2][y][x + 1] - S.V[s][2][y][x - 1];
        q.wy = S.V[s][2][y + 1][x] - S.V[s][2][y - 1][x];
        return q;
    };
    auto zflux = [&](const Plane& a, const Plane& b, double msum, double F[3]) {
        const double G = msum * K.gz, G43 = msum * (K.gz * (4.0 / 3.0));
        F[0] = G * ((b.v[0] - a.v[0]) + K.zx * (a.wx + b.wx));
        F[1] = G * ((b.v[1] - a.v[1]) + K.zy * (a.wy + b.wy));
        F[2] = G43 * ((b.v[2] - a.v[2]) + K.lz * (a.c + b.c));
    };
    // differences across z and in the plane that the x faces (and y faces) of cell (yy, xx) need
    auto xcell = [&](int yy, int xx, double dy, double q[3]) {
        q[0] = dy + K.ryz * (S.V[sp][2][yy][xx] - S.V[sm][2][yy][xx]);
        q[1] = S.V[sc][0][yy + 1][xx] - S.V[sc][0][yy - 1][xx];
        q[2] = S.V[sp][0][yy][xx] - S.V[sm][0][yy][xx];
    };
    auto ycell = [&](int yy, int xx, double dx, double q[3]) {
        q[0] = dx + K.rxz * (S.V[sp][2][yy][xx] - S.V[sm][2][yy][xx]);
        q[1] = S.V[sc][1][yy][xx + 1] - S.V[sc][1][yy][xx - 1];
        q[2] = S.V[sp][1][yy][xx] - S.V[sm][1][yy][xx];
    };
    auto xflux = [&](int yy, int xx, int m, double F[3]) {  // low x face of footprint cell (yy, xx)
        const double ms = S.M[m][yy][xx] + S.M[m][yy][xx - 1], G = ms * K.gx, G43 = ms * (K.gx * (4.0 / 3.0));
        F[0] = G43 * ((S.V[sc][0][yy][xx] - S.V[sc][0][yy][xx - 1]) + K.lx * (S.QX[0][yy - 1][xx] + S.QX[0][yy - 1][xx - 1]));
        F[1] = G * ((S.V[sc][1][yy][xx] - S.V[sc][1][yy][xx - 1]) + K.xy * (S.QX[1][yy - 1][xx] + S.QX[1][yy - 1][xx - 1]));
        F[2] = G * ((S.V[sc][2][yy][xx] - S.V[sc][2][yy][xx - 1]) + K.xz * (S.QX[2][yy - 1][xx] + S.QX[2][yy - 1][xx - 1]));
    };
    auto yflux = [&](int yy, int xx, int m, double F[3]) {  // low y face
        const double ms = S.M[m][yy][xx] + S.M[m][yy - 1][xx], G = ms * K.gy, G43 = ms * (K.gy * (4.0 / 3.0));
        F[0] = G * ((S.V[sc][0][yy][xx] - S.V[sc][0][yy - 1][xx]) + K.yx * (S.QY[1][yy][xx - 1] + S.QY[1][yy - 1][xx - 1]));
        F[1] = G43 * ((S.V[sc][1][yy][xx] - S.V[sc][1][yy - 1][xx]) + K.ly * (S.QY[0][yy][xx - 1] + S.QY[0][yy - 1][xx - 1]));
        F[2] = G * ((S.V[sc][2][yy][xx] - S.V[sc][2][yy - 1][xx]) + K.yz * (S.QY[2][yy][xx - 1] + S.QY[2][yy - 1][xx - 1]));
    };
    Plane pc{};
    double fz[3] = {0.0, 0.0, 0.0};
    if (mainw) {
        const Plane pm = plane(sm);
        pc = plane(sc);
        const double m0 = S.M[k0 & 1][y][x];
        zflux(pm, pc, mu + m0, fz);
        mu = m0;
    }
    const int i = i0 + x - 1, j = j0 + y - 1;
    const bool live = mainw && i < g.nx && j < g.ny;
    long long rmax = 0;
    for (int k = k0; k < k1; ++k) {
        const int m = k & 1;
        Cell nxt{};
        const bool more = loads && k + 1 < k1;
        if (more) nxt = fetch(k + 2);
        // ---- cell differences of layer k, z fluxes on its upper faces
        Plane pn{};
        double fzn[3] = {0.0, 0.0, 0.0}, q[3];
        if (mainw) {
            pn = plane(sp);
            const double mn = S.M[m ^ 1][y][x];
            zflux(pc, pn, mu + mn, fzn);
            mu = mn;
            xcell(y, x, pc.dy, q);
            for (int n = 0; n < 3; ++n) S.QX[n][y - 1][x] = q[n];
            ycell(y, x, pc.dx, q);
            for (int n = 0; n < 3; ++n) S.QY[n][y][x - 1] = q[n];
        } else if (h < 2 * WX) {
            ycell(yh, xh, S.V[sc][0][yh][xh + 1] - S.V[sc][0][yh][xh - 1], q);
            for (int n = 0; n < 3; ++n) S.QY[n][yh][xh - 1] = q[n];
        } else if (side) {
            xcell(sr + 1, sx, S.V[sc][1][sr + 2][sx] - S.V[sc][1][sr][sx], q);
            for (int n = 0; n < 3; ++n) S.QX[n][sr][sx] = q[n];
        }
        __syncthreads();
        // ---- fluxes on the low x and y faces
        double fx[3], fy[3];
        if (mainw) {
            xflux(y, x, m, fx);
            yflux(y, x, m, fy);
            for (int n = 0; n < 3; ++n) {
                S.FX[n][y - 1][x - 1] = fx[n];
                S.FY[n][y - 1][x - 1] = fy[n];
            }
        } else if (h >= WX && h < 2 * WX) {
            yflux(NR + 1, xh, m, fy);
            for (int n = 0; n < 3; ++n) S.FY[n][NR][xh - 1] = fy[n];
        } else if (side && sx) {
            xflux(sr + 1, WX + 1, m, fx);
            for (int n = 0; n < 3; ++n) S.FX[n][sr][WX] = fx[n];
        }
        __syncthreads();
        // ---- divergence and the mode's epilogue
        if (live) {
            const long long t = ((long long)k * g.ny + j) * g.nx + i;
#pragma unroll
            for (int n = 0; n < 3; ++n) {
                const double acc = ((S.FX[n][y - 1][x] - fx[n]) + (S.FY[n][y][x - 1] - fy[n])) + (fzn[n] - fz[n]);
                const long long o = n * N + t;
                if constexpr (MODE == 0) {
                    out[o] = acc;
                } else if constexpr (MODE == 1) {
                    out[o] = acc;
                    E.forces[o] = (E.src[o] + acc) * E.irho;
                } else if constexpr (MODE == 2) {
                    out[o] = E.base[o] + E.hdr * (acc - E.dold[o]);
                } else if constexpr (MODE == 3) {
                    out[o] = (E.rho * E.base[o] + E.dt * (0.5 * (E.conv_o[o] + E.conv_n[o]) + 0.5 * E.dold[o] + 0.5 * acc + E.src[o])) * E.irho;
                } else {
                    const double r = E.base[o] - E.rho * pc.v[n] + E.dt * acc;
                    rmax = imax_abs(rmax, r);
                    out[o] = MODE == 7 ? pc.v[n] + E.omega * E.dinv[o] * r : r;
                }
            }
        }
        pc = pn;
        for (int n = 0; n < 3; ++n) fz[n] = fzn[n];
        // layer k + 2 replaces layer k - 1 (read before the first barrier) and
        // the viscosity of layer k (before the second)
        if (more) stage(nxt, sm, k + 2);
        const int s = sm;
        sm = sc;
        sc = sp;
        sp = s;
        __syncthreads();
    }
    if constexpr (MODE >= 7) {
        if (!E.parts) return;  // uniform over the block
        for (int o = 16; o > 0; o >>= 1) {
            const long long b = __shfl_xor_sync(0xffffffffu, rmax, o);
            rmax = b > rmax ? b : rmax;
        }
        __shared__ long long wmax[TY];
        if (mainw && l == 0) wmax[w] = rmax;
        __syncthreads();
        if (tid == 0) {
            for (int r = 0; r < TY; ++r) rmax = wmax[r] > rmax ? wmax[r] : rmax;
            E.parts[(blockIdx.z * (long long)gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = bitsd(rmax);
        }
    }
}

// Launch shape: rows a block and layers a march.  A march does about 0.6
// layers' work more than its layers (the low z face and two staged layers), and
// an SM runs two blocks at a time, so the march is the one whose blocks, dealt
// to 304 places, finish first: 96^3 takes 12 layers (169 us; 203 at 1, 222 at
// 16), 64^3 4 (64; 68 at 1, 92 at 12, 229 at 32), 192x160x96 10 (548; 657 at 1,
// 576 at 12), 256x256x128 16 (1498; 1471 at 10, 1847 at 1).  It is within 2 % of
// the best of them but on 128x128x64, where it takes 16 layers (223 us) and 4
// take 206.  Blocks of 4 rows only where those of 8 leave places empty: 32x32x16
// 12 us against 15.  `narrow`: the forms of at most 16 columns, six blocks an SM.
struct TauShape {
    int ty, wx, kc;
    dim3 grid;
};
inline TauShape tau_shape(const Grid& g, bool narrow = false) {
    TauShape s{8, 32, 1, dim3(1, 1, 1)};
    if (narrow && g.nx <= 16) {
        s.ty = 1;
        s.wx = g.nx <= 4 ? 4 : (g.nx <= 8 ? 8 : 16);
    }
    const int bx = (g.nx + s.wx - 1) / s.wx;
    if (s.wx == 32 && (long long)bx * ((g.ny + 7) / 8) * g.nz < 304) s.ty = 4;  // small grids: more blocks
    const int rows = s.ty * (32 / s.wx), by = (g.ny + rows - 1) / rows, places = 152 * (s.wx == 32 ? 2 : kNarrowBlocks);
    double best = 0.0;
    for (int kc = 1; kc <= 16 && kc <= g.nz; ++kc) {
        const long long blocks = (long long)bx * by * ((g.nz + kc - 1) / kc);
        const double cost = (double)((blocks + places - 1) / places) * (kc + 0.6);
        if (kc == 1 || cost < best) {
            best = cost;
            s.kc = kc;
        }
    }
    s.grid = dim3((unsigned)bx, (unsigned)by, (unsigned)((g.nz + s.kc - 1) / s.kc));
    return s;
}

// predictor_rhs (src/equation_systems/CompRHSOps.H:32-141); fac = 1 explicit,
// 1/2 Crank-Nicolson, 0 implicit
// PLAIN (here, in k_sources and in k_mac_correct): the products as they stand,
// for the mixed-precision form, whose FP32 advection turns a change of the last
// bit into another trajectory; the FP64 form folds them (dtr = dt / rho).
template <int PLAIN>
__global__ void k_pred_rhs(long long N3, const double* vo, const double* conv, const double* src, const double* dt_, double* vel, double dt,
                           double rho, double irho, double fac, double dtr) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= N3) return;
    if constexpr (PLAIN) vel[t] = (rho * vo[t] + dt * (conv[t] + src[t] + fac * dt_[t])) * irho;
    else vel[t] = vo[t] + dtr * ((conv[t] + src[t]) + fac * dt_[t]);
}

// ---------------------------------------------------------------- projection
__global__ void k_proj_pre(long long N3, double* vel, const double* vo, const double* gp, double sr, int add_gp, int sub_old) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= N3) return;
    double v = vel[t];
    if (add_gp) v += gp[t] * sr;  // sr = scaling / rho, formed on the host
    if (sub_old) v -= vo[t];
    vel[t] = v;
}

// Nodal divergence of the cell velocity at node t (the MLNodeLaplacian
// right-hand side).  The cell velocity is seen with periodic wrap and mirror
// images across z walls (normal component odd, tangential even; the sign flip
// is taken on the bits).  Each direction's four edge differences are summed
// before its one scale q = dx^-1 / 4.
__device__ inline double nodal_div_at(const Grid& g, const double* vel, unsigned t, int& k, double qx, double qy, double qz) {
    const unsigned r = t / (unsigned)g.nx;
    const int i = (int)(t - r * (unsigned)g.nx);
    k = (int)(r / (unsigned)g.ny);
    const int j = (int)(r - (unsigned)k * (unsigned)g.ny);
    const int im = i == 0 ? g.nx - 1 : i - 1, jm = j == 0 ? g.ny - 1 : j - 1;
    // cell layers k - 1 and k as seen from the node (mirrored at walls)
    int kk[2];
    bool flip[2];
    for (int c = 0; c < 2; ++c) {
        int q = k - c;
        flip[c] = false;
        if (g.zper) q = q < 0 ? q + g.nz : (q >= g.nz ? q - g.nz : q);
        else if (q < 0) { q = -1 - q; flip[c] = true; }
        else if (q >= g.nz) { q = 2 * g.nz - 1 - q; flip[c] = true; }
        kk[c] = q;
    }
    const long long N = g.N;
    // the 8 cells around the node: layers k-1 (c = 1) and k (c = 0), columns (i, j), (i-1, j), (i, j-1), (i-1, j-1)
    double u[2][4], v[2][4], w[2][4];
    for (int c = 0; c < 2; ++c) {
        const long long r0 = (long long)kk[c] * g.ny;
        const long long o[4] = {(r0 + j) * g.nx + i, (r0 + j) * g.nx + im, (r0 + jm) * g.nx + i, (r0 + jm) * g.nx + im};
        for (int q = 0; q < 4; ++q) {
            u[c][q] = vel[o[q]];
            v[c][q] = vel[N + o[q]];
            const double z = vel[2 * N + o[q]];
            w[c][q] = flip[c] ? bitsd(dbits(z) ^ ~kMag) : z;
        }
    }
    double dx = 0, dy = 0, dz = 0;
    for (int c = 0; c < 2; ++c) {
        dx += (u[c][0] - u[c][1]) + (u[c][2] - u[c][3]);
        dy += (v[c][0] - v[c][2]) + (v[c][1] - v[c][3]);
    }
    // z: differences of w between the layers k and k - 1 over the four cells
    dz = ((w[0][0] - w[1][0]) + (w[0][1] - w[1][1])) + ((w[0][2] - w[1][2]) + (w[0][3] - w[1][3]));
    return qx * dx + (qy * dy + qz * dz);
}

// Nodal divergence into the right-hand side, with weighted partial sums
// (boundary nodes carry half weight) for the solvability shift.  A thread
// walks a chunk of the node column (i, j); the four cells around the column
// in cell layer c (mirrored at walls as in nodal_div_at) give
//   X(c) = (u(i,j) - u(i-1,j)) + (u(i,j-1) - u(i-1,j-1)),
//   Y(c) = (v(i,j) - v(i,j-1)) + (v(i-1,j) - v(i-1,j-1))
// and their four w values, and node k combines layers k and k - 1 in
// nodal_div_at's order (the same result): each cell layer is loaded and
// differenced once for the two nodes it borders, 20 FP64 operations per node
// where nodal_div_at spends 28.
__global__ void k_nodal_rhs(Grid g, const double* vel, double* rhs, double* parts, int np, double qx, double qy, double qz, int kc) {
    const int nzn = g.zper ? g.nz : g.nz + 1;
    const int nch = (nzn + kc - 1) / kc;
    const unsigned M = (unsigned)(g.nx * g.ny * nch);
    const long long N = g.N;
    double ws = 0, wt = 0;
    struct Lay {
        double X, Y, w[4];
    };
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
        const unsigned r = t / (unsigned)g.nx;
        const int i = (int)(t - r * (unsigned)g.nx);
        const int ch = (int)(r / (unsigned)g.ny);
        const int j = (int)(r - (unsigned)ch * (unsigned)g.ny);
        const int im = i == 0 ? g.nx - 1 : i - 1, jm = j == 0 ? g.ny - 1 : j - 1;
        auto layer = [&](int q, Lay& L) {
            bool flip = false;
            if (g.zper) q = q < 0 ? q + g.nz : (q >= g.nz ? q - g.nz : q);
            else if (q < 0) { q = -1 - q; flip = true; }
            else if (q >= g.nz) { q = 2 * g.nz - 1 - q; flip = true; }
            const long long r0 = (long long)q * g.ny;
            const long long o[4] = {(r0 + j) * g.nx + i, (r0 + j) * g.nx + im, (r0 + jm) * g.nx + i, (r0 + jm) * g.nx + im};
            double u[4], v[4];
            for (int m = 0; m < 4; ++m) {
                u[m] = vel[o[m]];
                v[m] = vel[N + o[m]];
                const double z = vel[2 * N + o[m]];
                L.w[m] = flip ? bitsd(dbits(z) ^ ~kMag) : z;
            }
            L.X = (u[0] - u[1]) + (u[2] - u[3]);
            L.Y = (v[0] - v[2]) + (v[1] - v[3]);
        };
        const int k0 = ch * kc, k1 = min(k0 + kc, nzn);
        Lay lo, hi;  // cell layers k - 1 and k
        layer(k0 - 1, lo);
        for (int k = k0; k < k1; ++k) {
            layer(k, hi);
            const double dx = hi.X + lo.X, dy = hi.Y + lo.Y;
            const double dz = ((hi.w[0] - lo.w[0]) + (hi.w[1] - lo.w[1])) + ((hi.w[2] - lo.w[2]) + (hi.w[3] - lo.w[3]));
            const double dv = qx * dx + (qy * dy + qz * dz);
            rhs[((long long)k * g.ny + j) * g.nx + i] = dv;
            const double wgt = (!g.zper && (k == 0 || k == nzn - 1)) ? 0.5 : 1.0;
            ws += wgt * dv;
            wt += wgt;
            lo = hi;
        }
    }
    ws = block_reduce<0>(ws);
    wt = block_reduce<0>(wt);
    if (threadIdx.x == 0) { parts[blockIdx.x] = ws; parts[np + blockIdx.x] = wt; }
}

// Post-projection diagnostic: per-block max-norm of the nodal divergence of
// the velocity (the operator the projection drives to zero) and of |u|.
// Both maxima are kept as bits, so a NaN survives to the host.
__global__ void k_nodal_divmax(Grid g, const double* vel, double* parts, int np, double qx, double qy, double qz) {
    const int nzn = g.zper ? g.nz : g.nz + 1;
    const unsigned M = (unsigned)(g.nx * g.ny * nzn);
    const unsigned stride = gridDim.x * blockDim.x;
    long long md = 0, mu = 0;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += stride) {
        int k;
        md = imax_abs(md, nodal_div_at(g, vel, t, k, qx, qy, qz));
    }
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < (unsigned)(3 * g.N); t += stride) mu = imax_abs(mu, vel[t]);
    const double a = block_reduce<1>(bitsd(md)), b = block_reduce<1>(bitsd(mu));
    if (threadIdx.x == 0) { parts[blockIdx.x] = a; parts[np + blockIdx.x] = b; }
}

// u -= sigma G phi ; gp = (or +=) G phi ; optional add-back of u_old.  G is the
// cell gradient of the nodal phi (the mean of the four edge differences in
// each direction), formed from the cell's 8 corner nodes with shared pair sums;
// q = dx^-1 / 4 and sigma q are folded on the host.
__global__ void k_nodal_post_cells(Grid g, const double* phi, double* vel, const double* vo, double* gp, double qx, double qy, double qz,
                                   double sqx, double sqy, double sqz, int add_old, int incr) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    const int ip = i + 1 == g.nx ? 0 : i + 1, jp = j + 1 == g.ny ? 0 : j + 1;
    const int kp = (g.zper && k + 1 == g.nz) ? 0 : k + 1;  // nodes 0..nz at walls
    const long long sy = g.nx, sz = (long long)g.nx * g.ny;
    const long long r0 = k * sz, r1 = kp * sz, c0 = j * sy, c1 = jp * sy;
    const double n000 = phi[r0 + c0 + i], n100 = phi[r0 + c0 + ip], n010 = phi[r0 + c1 + i], n110 = phi[r0 + c1 + ip];
    const double n001 = phi[r1 + c0 + i], n101 = phi[r1 + c0 + ip], n011 = phi[r1 + c1 + i], n111 = phi[r1 + c1 + ip];
    const double za = n000 + n001, zb = n100 + n101, zc = n010 + n011, zd = n110 + n111;
    const double gx = (zb + zd) - (za + zc), gy = (zc + zd) - (za + zb);
    const double gz = ((n001 + n101) + (n011 + n111)) - ((n000 + n100) + (n010 + n110));
    const double Gv[3] = {gx, gy, gz}, q[3] = {qx, qy, qz}, sq[3] = {sqx, sqy, sqz};
    const long long N = g.N;
    for (int n = 0; n < 3; ++n) {
        double v = vel[n * N + t] - sq[n] * Gv[n];
        if (add_old) v += vo[n * N + t];
        vel[n * N + t] = v;
        const double G = q[n] * Gv[n];
        if (incr) gp[n * N + t] += G;
        else gp[n * N + t] = G;
    }
}

__global__ void k_nodal_post_nodes(long long M, const double* phi, double* p, int incr) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= M) return;
    if (incr) p[t] += phi[t];
    else p[t] = phi[t];
}

// MAC divergence + partial sums
__global__ void k_mac_rhs(Grid g, const double* um, const double* vm, const double* wm, double* rhs, double* parts, int np) {
    double s = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.N; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        cell_of(g, t, i, j, k);
        const double r = (um[fidx(g, 0, i + 1, j, k)] - um[t]) * g.idx + (vm[fidx(g, 1, i, j + 1, k)] - vm[t]) * g.idy +
                         (wm[fidx(g, 2, i, j, k + 1)] - wm[fidx(g, 2, i, j, k)]) * g.idz;
        rhs[t] = r;
        s += r;
    }
    s = block_reduce<0>(s);
    if (threadIdx.x == 0) parts[blockIdx.x] = s;
}

// Post-projection diagnostic: per-block maxima of |div u_mac| (the MAC
// projection's exact discrete divergence) and of the face speeds, as bits.
__global__ void k_mac_divmax(Grid g, const double* um, const double* vm, const double* wm, double* parts, int np) {
    long long md = 0, mu = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.N; t += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        cell_of(g, t, i, j, k);
        const double r = (um[fidx(g, 0, i + 1, j, k)] - um[t]) * g.idx + (vm[fidx(g, 1, i, j + 1, k)] - vm[t]) * g.idy +
                         (wm[fidx(g, 2, i, j, k + 1)] - wm[fidx(g, 2, i, j, k)]) * g.idz;
        md = imax_abs(md, r);
        mu = imax_abs(imax_abs(imax_abs(mu, um[t]), vm[t]), wm[fidx(g, 2, i, j, k)]);
    }
    const double a = block_reduce<1>(bitsd(md)), b = block_reduce<1>(bitsd(mu));
    if (threadIdx.x == 0) { parts[blockIdx.x] = a; parts[np + blockIdx.x] = b; }
}

// bx = beta / dx, ...
template <int PLAIN>
__global__ void k_mac_correct(Grid g, const double* phi, double* um, double* vm, double* wm, double beta, double bx, double by, double bz) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= g.N) return;
    int i, j, k;
    cell_of(g, t, i, j, k);
    const double p0 = phi[t];
    const double px = phi[cidx(g, wrapn(i - 1, g.nx), j, k)], py = phi[cidx(g, i, wrapn(j - 1, g.ny), k)];
    if constexpr (PLAIN) {
        um[t] -= beta * (p0 - px) * g.idx;
        vm[t] -= beta * (p0 - py) * g.idy;
        if (g.zper || k > 0) wm[t] -= beta * (p0 - phi[cidx(g, i, j, k == 0 ? g.nz - 1 : k - 1)]) * g.idz;
    } else {
        um[t] -= bx * (p0 - px);
        vm[t] -= by * (p0 - py);
        if (g.zper || k > 0) wm[t] -= bz * (p0 - phi[cidx(g, i, j, k == 0 ? g.nz - 1 : k - 1)]);
    }
}

// ---------------------------------------------------------------- reductions
__global__ void k_cfl(Grid g, const double* vel, const double* src, const double* mu, double rho, double* parts, int np) {
    // The maxima of |u_n|, |src_n| and mu are taken on the integer pipe and
    // scaled once per thread: rounding is monotone, so max(|u|) / dx equals
    // max(|u| / dx) exactly, and no FP64 instruction runs per cell.
    const double dxi[3] = {g.idx, g.idy, g.idz};
    const double irho = 1.0 / rho;
    const double dxinv2 = 2.0 * (dxi[0] * dxi[0] + dxi[1] * dxi[1] + dxi[2] * dxi[2]);
    long long um[3] = {0, 0, 0}, sm[3] = {0, 0, 0}, mm = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.N; t += (long long)gridDim.x * blockDim.x) {
        for (int n = 0; n < 3; ++n) {
            um[n] = imax_abs(um[n], vel[n * g.N + t]);
            sm[n] = imax_abs(sm[n], src[n * g.N + t]);
        }
        mm = imax_abs(mm, mu[t]);  // mu_eff >= 0
    }
    double c = 0, d = 0, f = 0;
    for (int n = 0; n < 3; ++n) {
        c = nmax(c, bitsd(um[n]) * dxi[n]);
        f = nmax(f, bitsd(sm[n]) * dxi[n] * irho);
    }
    d = bitsd(mm) * dxinv2 * irho;
    c = block_reduce<1>(c);
    d = block_reduce<1>(d);
    f = block_reduce<1>(f);
    if (threadIdx.x == 0) { parts[blockIdx.x] = c; parts[np + blockIdx.x] = d; parts[2 * np + blockIdx.x] = f; }
}

__global__ void k_ke(Grid g, const double* vel, double rho, double* parts) {
    double s = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.N; t += (long long)gridDim.x * blockDim.x)
        for (int n = 0; n < 3; ++n) {
            const double v = vel[n * g.N + t];
            s += 0.5 * rho * v * v;
        }
    s = block_reduce<0>(s);
    if (threadIdx.x == 0) parts[blockIdx.x] = s;
}

__global__ void k_reduce(const double* parts, int np, int op_max, double* out) {
    const int comp = blockIdx.x;
    double v = op_max ? -1.0e300 : 0.0;
    for (int m = threadIdx.x; m < np; m += blockDim.x) {
        const double x = parts[comp * np + m];
        v = op_max ? nmax(v, x) : v + x;
    }
    v = op_max ? block_reduce<1>(v) : block_reduce<0>(v);
    if (threadIdx.x == 0) out[comp] = v;
}

// a -= s[0] / den (den > 0) or a -= s[0] / s[1]; with parts, block maxima of
// |a| after the shift.  Grid-stride, so the FP64 division is formed once per
// thread rather than once per element.
__global__ void k_sub_ratio(double* a, long long n, const double* s, double den, double* parts) {
    const double r = s[0] / (den > 0.0 ? den : s[1]);
    long long mb = 0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double v = a[t] - r;
        a[t] = v;
        mb = imax_abs(mb, v);
    }
    if (!parts) return;
    const double m = block_reduce<1>(bitsd(mb));
    if (threadIdx.x == 0) parts[blockIdx.x] = m;
}

// ---------------------------------------------------------------- actuator
// Trilinear sampling of the velocity at disk points
// (ActuatorContainer.cpp:284-360); ghosts follow the fill-patch rules.
__global__ void k_act_sample(Grid g, const double* vel, const double* pts, int npts, double x0, double y0, double z0, double* out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npts) return;
    VelFP V{vel, g, 1.0};
    const double fx = (pts[3 * p] - x0 - 0.5 * g.dx) / g.dx;
    const double fy = (pts[3 * p + 1] - y0 - 0.5 * g.dy) / g.dy;
    const double fz = (pts[3 * p + 2] - z0 - 0.5 * g.dz) / g.dz;
    const int i = (int)floor(fx), j = (int)floor(fy), k = (int)floor(fz);
    const double wx = fx - i, wy = fy - j, wz = fz - k;
    for (int n = 0; n < 3; ++n) {
        double s = 0;
        for (int c = 0; c < 2; ++c)
            for (int b = 0; b < 2; ++b)
                for (int a = 0; a < 2; ++a) {
                    const double w = (a ? wx : 1 - wx) * (b ? wy : 1 - wy) * (c ? wz : 1 - wz);
                    s += w * V(n, i + a, j + b, k + c);
                }
        out[3 * p + n] = s;
    }
}

// Gaussian spreading of ring-point forces (disk_spreading.H:45-105,
// actuator_utils.H:45-60) over the cells of the cut-off box of a disk.
// The kernel exp(-|x - p|^2 / eps^2) is a product of three 1D factors, and
// disks do not move: k_act_tables forms the factors of every (point, cell
// column of one direction) once per handle, and the spread multiplies them.
// Evaluated per (point, cell) it took three FP64 divisions and an exp, about
// 45 FP64 issue slots for each of the 100 points of a cell, and one launch and
// two host waits a disk: 340 us a disk of 18 cells' diameter, 5.4 ms a step of
// a 16-disk farm.
__global__ void k_act_tables(Grid g, const ActDisk* D, const double* pts, double x0, double y0, double z0, double* E, float* R) {
    const ActDisk d = D[blockIdx.y];
    const int S = d.n[0] + d.n[1] + d.n[2];
    const double gfac = 0.17958712212516656 / (d.eps * d.eps * d.eps);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < d.npts * S; t += gridDim.x * blockDim.x) {
        const int m = t / S;
        int q = t - m * S, dir = 0;
        while (q >= d.n[dir]) q -= d.n[dir++];
        const double o = dir == 0 ? x0 : (dir == 1 ? y0 : z0), h = hd(g, dir);
        const double r = (pts[3 * (d.p0 + m) + dir] - (o + (d.lo[dir] + q + 0.5) * h)) / d.eps;
        E[d.tab + t] = (dir == 0 ? gfac : 1.0) * exp(-r * r);
        R[d.tab + t] = (float)(r * r);
    }
}

// Sum over a disk's points of w_m g3(x - p_m) at cell (a, b, c) of its box.
// The cut-off |x - p|^2 < 16 eps^2 is decided on the FP32 squares, whose sum is
// off by less than 1e-5, and within 0.01 of it on the FP64 distance itself.
__device__ inline double act_sum(const Grid& g, const ActDisk& d, const double* pts, const double* w, const double* E, const float* R, double x0,
                                 double y0, double z0, int a, int b, int c) {
    const int S = d.n[0] + d.n[1] + d.n[2];
    const int ob = d.n[0] + b, oc = d.n[0] + d.n[1] + c;
    double s = 0;
    for (int m = 0; m < d.npts; ++m) {
        const long long q = d.tab + (long long)m * S;
        const float r2 = R[q + a] + R[q + ob] + R[q + oc];
        if (r2 > 16.01f) continue;
        if (r2 > 15.99f) {
            const double* p = pts + 3 * (d.p0 + m);
            const double rx = (p[0] - (x0 + (d.lo[0] + a + 0.5) * g.dx)) / d.eps, ry = (p[1] - (y0 + (d.lo[1] + b + 0.5) * g.dy)) / d.eps,
                         rz = (p[2] - (z0 + (d.lo[2] + c + 0.5) * g.dz)) / d.eps;
            if (!(rx * rx + ry * ry + rz * rz < 16.0)) continue;
        }
        s += E[q + a] * E[q + ob] * (E[q + oc] * w[d.p0 + m]);
    }
    return s;
}

// One launch spreads the disks d0 .. d0 + gridDim.y - 1, whose boxes are
// disjoint; overlapping disks go in launches of their own, in disk order.
__global__ void k_act_spread(Grid g, double* act, const ActDisk* D, int d0, const double* pts, const double* w, const double* E, const float* R,
                             double x0, double y0, double z0) {
    const ActDisk d = D[d0 + blockIdx.y];
    const int M = d.n[0] * d.n[1] * d.n[2];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= M) return;
    const int a = t % d.n[0], r = t / d.n[0], b = r % d.n[1], c = r / d.n[1];
    const double s = act_sum(g, d, pts, w, E, R, x0, y0, z0, a, b, c);
    if (s == 0.0) return;
    const long long cc = cidx(g, d.lo[0] + a, d.lo[1] + b, d.lo[2] + c);
    act[cc] += s * d.ax[0];
    act[g.N + cc] += s * d.ax[1];
    act[2 * g.N + cc] += s * d.ax[2];
}

// disk adjoint: per disk (blockIdx.y) block sums over its box of
// sum_x (actb(x) . n) B(x), B(x) = sum_m w_m g3(x - p_m)
__global__ void k_act_adj_dot(Grid g, const double* actb, const ActDisk* D, const double* pts, const double* w, const double* E, const float* R,
                              double x0, double y0, double z0, double* parts) {
    const ActDisk d = D[blockIdx.y];
    const int M = d.n[0] * d.n[1] * d.n[2];
    double acc = 0.0;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M; t += gridDim.x * blockDim.x) {
        const int a = t % d.n[0], r = t / d.n[0], b = r % d.n[1], c = r / d.n[1];
        const double s = act_sum(g, d, pts, w, E, R, x0, y0, z0, a, b, c);
        const long long cc = cidx(g, d.lo[0] + a, d.lo[1] + b, d.lo[2] + c);
        acc += s * (actb[cc] * d.ax[0] + actb[g.N + cc] * d.ax[1] + actb[2 * g.N + cc] * d.ax[2]);
    }
    acc = block_reduce<0>(acc);
    if (threadIdx.x == 0) parts[blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

}  // namespace

// ---------------------------------------------------------------- launchers

constexpr double B8 = 8.0;  // bytes per FP64 value

void launch_init_tgv(Ctx& c, const Grid& g, double* vel, const double plo[3], const double L[3]) {
    KS_LAUNCH(c, k_init_tgv, nblocks(g.N, BS), BS, B8 * 3 * g.N, g, vel, plo[0], plo[1], plo[2], L[0], L[1], L[2]);
}
void launch_init_abl(Ctx& c, const Grid& g, double* vel, int loglaw, const double U[3], double ut_k, double z0, double amp,
                     double zmax_rel, unsigned long long seed) {
    KS_LAUNCH(c, k_init_abl, nblocks(g.N, BS), BS, B8 * 3 * g.N, g, vel, loglaw, U[0], U[1], U[2], ut_k, z0, amp, zmax_rel, seed);
}
void launch_fill(Ctx& c, double* p, double v, long long n) { KS_LAUNCH(c, k_fill, nblocks(n, BS), BS, B8 * n, p, v, n); }
void launch_copy(Ctx& c, double* d, const double* s, long long n) { KS_LAUNCH(c, k_copy, nblocks(n, BS), BS, B8 * 2 * n, d, s, n); }
void launch_smagorinsky(Ctx& c, const Grid& g, const double* vel, double* mueff, const Scalars& s, double* alpha, int fp32,
                        const float* vel32) {
    if (!s.temp) alpha = nullptr;
    const double bytes = B8 * ((s.smag ? 4 : 1) + (alpha ? 1 : 0)) * g.N;
    if (!s.smag) {
        KS_LAUNCH(c, k_mu_molecular, nblocks(g.N, BS), BS, bytes, g.N, mueff, s.mu, alpha, s.mu_pr);
    } else if (fp32) {
        // layers a march: 16, fewer where that leaves less than 4096 warps
        const int kc = march_layers(g, 4096);
        KS_LAUNCH(c, k_smag_march, column_grid(g, kc), column_threads(g), bytes - 12.0 * g.N, g, vel32, mueff, s.mu, s.rho * s.smag_fac,
                  alpha, s.mu_pr, s.iprt, kc);
    } else {
        // layers a march: 16, fewer where that leaves less than 2048 warps
        const int kc = march_layers(g, 2048);
        KS_LAUNCH(c, k_smag_col, column_grid(g, kc), column_threads(g), bytes, g, vel, mueff, s.mu, s.rho * s.smag_fac, alpha, s.mu_pr, s.iprt, kc);
    }
}
// src = rho (-gp/rho + geostrophic + Coriolis(u_old) + body + actuator + Boussinesq + ABLForcing)
// (icns_ops.H:78-124, PDEOps.H:94-145, GeostrophicForcing.cpp:103-, CoriolisForcing.cpp:60-108,
// BodyForce.cpp:117-169, ActuatorForcing.cpp:19-29): the Coriolis acceleration
//   ae e + an n + au u,  ae = f (un sin - h uu cos), an = -f ue sin, au = h f ue cos
// (e, n, u the east / north / up unit vectors, ue = e.u etc., f = corfac, h = hfac) is the linear map
//   M = f sin (e n^T - n e^T) + f h cos (u e^T - e u^T).
void launch_sources(Ctx& c, const Grid& g, const double* vel_old, const double* gp, const double* act, double* src, const Scalars& s,
                    const double* theta, int plain) {
    SrcCoef k{};
    k.rho = s.rho;
    k.T_ref = s.T_ref;
    for (int n = 0; n < 3; ++n) {
        double a = 0.0;
        if (s.geo) a += (n == 2 ? s.hfac : 1.0) * s.gf[n];
        if (s.body) a += (s.body_osc ? std::cos(s.body_omega * s.t_nph) : 1.0) * s.body_force[n];
        if (s.ablf && n < 2) a += s.ablf_force[n];
        k.c[n] = s.rho * a;
        k.bous_g[n] = s.rho * s.grav[n] * s.beta_T;
        for (int m = 0; m < 3; ++m)
            k.M[n][m] = coriolis_map(s, n, m);
    }
    using Kern = void (*)(Grid, const double*, const double*, const double*, double*, SrcCoef, const double*);
    static const Kern kern[2][8] = {{k_sources<0, 0, 0, 0>, k_sources<1, 0, 0, 0>, k_sources<0, 1, 0, 0>, k_sources<1, 1, 0, 0>,
                                     k_sources<0, 0, 1, 0>, k_sources<1, 0, 1, 0>, k_sources<0, 1, 1, 0>, k_sources<1, 1, 1, 0>},
                                    {k_sources<0, 0, 0, 1>, k_sources<1, 0, 0, 1>, k_sources<0, 1, 0, 1>, k_sources<1, 1, 0, 1>,
                                     k_sources<0, 0, 1, 1>, k_sources<1, 0, 1, 1>, k_sources<0, 1, 1, 1>, k_sources<1, 1, 1, 1>}};
    const Kern run = kern[plain ? 1 : 0][(s.cor ? 1 : 0) + (s.act ? 2 : 0) + (s.bous ? 4 : 0)];
    KS_LAUNCH_NAMED(c, "k_sources", run, nblocks(g.N, BS), BS, B8 * (6 + 3 * s.cor + 3 * s.act + s.bous) * g.N, g, vel_old, gp, act, src, k, theta);
}
void launch_plane_sums(Ctx& c, const Grid& g, const double* vel, double* parts, int* np) {
    *np = parts_for((long long)g.nx * g.ny);
    KS_LAUNCH(c, k_plane_sums, *np, BS, B8 * 2 * g.nx * g.ny, g, vel, parts, *np);
}
void launch_wall_grad(Ctx& c, const Grid& g, const double* vel_old, const double* mueff, double* wg, int type, double ut2, double um0,
                      double um1, double vm, double rho) {
    KS_LAUNCH(c, k_wall_grad, nblocks((long long)g.nx * g.ny, BS), BS, B8 * 5 * g.nx * g.ny, g, vel_old, mueff, wg, type, ut2, um0,
              um1, vm, rho);
}
void launch_divtau_faces(Ctx& c, const Grid& g, const double* vel, const double* mueff, const double* wg, double* out, int mode,
                         const double* src, double* forces, const double* base, const double* dold, double dt, double rho,
                         double* const fl[9]) {
    for (int d = 0; d < 3; ++d) {
        const long long M = (long long)g.nx * g.ny * (d == 2 ? nzfaces(g) : g.nz);
        KS_LAUNCH(c, k_tau_flux, nblocks(M, BS), BS, B8 * (4.0 * g.N + 3.0 * M), g, d, vel, mueff, wg, fl[3 * d], fl[3 * d + 1],
                  fl[3 * d + 2]);
    }
    Flux9 F;
    for (int m = 0; m < 9; ++m) F.p[m] = fl[m];
    const double per_cell = 9 + 3 + (mode == 1 ? 6 : 0) + (mode == 2 ? 6 : 0);
    KS_LAUNCH(c, k_tau_div, nblocks(g.N, BS), BS, B8 * per_cell * g.N, g, F, out, mode, src, forces, base, dold, dt, rho);
}

template <int MODE>
static void launch_divtau_mode(Ctx& c, const Grid& g, const double* vel, const double* mueff, const double* wg, double* out, const TauEpi& E,
                               double bytes) {
    const TauShape s = tau_shape(g, MODE == 0);
    const TauCoef K = tau_coef(g);
    if constexpr (MODE == 0) {
        if (s.wx < 32) {
            const auto run = s.wx == 4 ? k_divtau_col<1, 0, 4> : (s.wx == 8 ? k_divtau_col<1, 0, 8> : k_divtau_col<1, 0, 16>);
            const size_t smem = s.wx == 4 ? sizeof(TauPlanes<1, 4>) : (s.wx == 8 ? sizeof(TauPlanes<1, 8>) : sizeof(TauPlanes<1, 16>));
            KS_LAUNCH_SMEM_NAMED(c, "k_divtau_col", run, s.grid, 32 * 4, smem, bytes, g, K, vel, mueff, wg, out, E, s.kc);
            return;
        }
    }
    const auto k4 = k_divtau_col<4, MODE, 32>;
    const auto k8 = k_divtau_col<8, MODE, 32>;
    if (s.ty == 4) {
        KS_LAUNCH_SMEM_NAMED(c, "k_divtau_col", k4, s.grid, 32 * 7, sizeof(TauPlanes<4, 32>), bytes, g, K, vel, mueff, wg, out, E, s.kc);
    } else {
        cudaFuncSetAttribute(k8, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TauPlanes<8, 32>));
        KS_LAUNCH_SMEM_NAMED(c, "k_divtau_col", k8, s.grid, 32 * 11, sizeof(TauPlanes<8, 32>), bytes, g, K, vel, mueff, wg, out, E, s.kc);
    }
}
static void launch_divtau_col(Ctx& c, const Grid& g, const double* vel, const double* mueff, const double* wg, double* out, const TauEpi& E,
                              double bytes) {
    switch (E.mode) {
        case 0: launch_divtau_mode<0>(c, g, vel, mueff, wg, out, E, bytes); break;
        case 1: launch_divtau_mode<1>(c, g, vel, mueff, wg, out, E, bytes); break;
        case 2: launch_divtau_mode<2>(c, g, vel, mueff, wg, out, E, bytes); break;
        case 3: launch_divtau_mode<3>(c, g, vel, mueff, wg, out, E, bytes); break;
        case 7: launch_divtau_mode<7>(c, g, vel, mueff, wg, out, E, bytes); break;
        default: launch_divtau_mode<8>(c, g, vel, mueff, wg, out, E, bytes); break;
    }
}
static_assert(sizeof(TauPlanes<4, 32>) <= 48 * 1024, "needs no shared memory attribute");
void launch_divtau(Ctx& c, const Grid& g, const double* vel, const double* mueff, const double* wg, double* out, int mode,
                   const double* src, double* forces, const double* base, const double* dold, double dt, double rho, int fp32,
                   const float* vel32) {
    const double per_cell = 4 + 3 + (mode == 1 ? 6 : 0) + (mode == 2 ? 6 : 0);
    TauEpi E{mode, src, base, dold, nullptr, nullptr, nullptr, forces, nullptr, dt, rho, 0.0, 1.0 / rho, 0.5 * dt / rho, 0.5 * dt};
    if (fp32) {
        const dim3 grid((g.nx + TTX - 1) / TTX, (g.ny + TTY - 1) / TTY, (g.nz + TTZ - 1) / TTZ);
        const auto run = vel32 ? (mode == 0 ? k_divtau_tile<0, 1> : (mode == 1 ? k_divtau_tile<1, 1> : k_divtau_tile<2, 1>))
                               : (mode == 0 ? k_divtau_tile<0, 0> : (mode == 1 ? k_divtau_tile<1, 0> : k_divtau_tile<2, 0>));
        KS_LAUNCH_SMEM_NAMED(c, "k_divtau_tile", run, grid, TTX * TTY * TTZ, tau_smem(), B8 * per_cell * g.N, g, vel, vel32, mueff, wg, out, E);
    } else {
        launch_divtau_col(c, g, vel, mueff, wg, out, E, B8 * per_cell * g.N);
    }
}
void launch_divtau_corrector(Ctx& c, const Grid& g, const double* vel, const double* mueff, const double* wg, double* out, const double* vel_old,
                             const double* conv_old, const double* conv_new, const double* dold, const double* src, double dt, double rho) {
    TauEpi E{3, src, vel_old, dold, conv_old, conv_new, nullptr, nullptr, nullptr, dt, rho, 0.0, 1.0 / rho, 0.5 * dt / rho, 0.5 * dt};
    launch_divtau_col(c, g, vel, mueff, wg, out, E, B8 * 22.0 * g.N);
}
int divtau_blocks(const Grid& g) {
    const TauShape s = tau_shape(g);
    return (int)(s.grid.x * s.grid.y * s.grid.z);
}
void launch_divtau_jacobi(Ctx& c, const Grid& g, const double* x, const double* mueff, const double* wg, const double* b, const double* dinv,
                          double* out, double rho, double dtd, double omega, double* parts) {
    TauEpi E{omega > 0.0 ? 7 : 8, nullptr, b, nullptr, nullptr, nullptr, dinv, nullptr, parts, dtd, rho, omega, 1.0 / rho, 0.5 * dtd / rho, 0.5 * dtd};
    launch_divtau_col(c, g, x, mueff, wg, out, E, B8 * ((omega > 0.0 ? 13.0 : 10.0) * g.N));
}
void launch_predictor_rhs(Ctx& c, const Grid& g, const double* vo, const double* conv, const double* src, const double* dtau, double* vel,
                          double dt, double rho, double fac, int plain) {
    const auto run = plain ? k_pred_rhs<1> : k_pred_rhs<0>;
    KS_LAUNCH_NAMED(c, "k_pred_rhs", run, nblocks(3 * g.N, BS), BS, B8 * 15 * g.N, 3 * g.N, vo, conv, src, dtau, vel, dt, rho, 1.0 / rho, fac, dt / rho);
}
void launch_proj_pre(Ctx& c, const Grid& g, double* vel, const double* vo, const double* gp, double scaling, double rho, int add_gp,
                     int sub_old) {
    KS_LAUNCH(c, k_proj_pre, nblocks(3 * g.N, BS), BS, B8 * 3 * (2 + add_gp + sub_old) * g.N, 3 * g.N, vel, vo, gp, scaling / rho, add_gp, sub_old);
}
void launch_nodal_rhs(Ctx& c, const Grid& g, const double* vel, double* rhs, double* parts, int* np) {
    const int nzn = g.zper ? g.nz : g.nz + 1;
    const long long M = (long long)g.nx * g.ny * nzn;
    const long long work = M / 300000;  // node layers per thread: long columns on large grids
    const int kc = (int)(work < 2 ? 2 : (work > 16 ? 16 : work));
    *np = parts_for((long long)g.nx * g.ny * ((nzn + kc - 1) / kc));
    KS_LAUNCH(c, k_nodal_rhs, *np, BS, B8 * (3 * g.N + M), g, vel, rhs, parts, *np, 0.25 * g.idx, 0.25 * g.idy, 0.25 * g.idz, kc);
}
void launch_nodal_divmax(Ctx& c, const Grid& g, const double* vel, double* parts, int* np) {
    const long long M = (long long)g.nx * g.ny * (g.zper ? g.nz : g.nz + 1);
    *np = parts_for(M);
    KS_LAUNCH(c, k_nodal_divmax, *np, BS, B8 * 3 * g.N, g, vel, parts, *np, 0.25 * g.idx, 0.25 * g.idy, 0.25 * g.idz);
}
void launch_nodal_post(Ctx& c, const Grid& g, const double* phi, double* vel, const double* vo, double* gp, double* p, double sigma,
                       int add_old, int incr) {
    const long long M = (long long)g.nx * g.ny * (g.zper ? g.nz : g.nz + 1);
    const double qx = 0.25 * g.idx, qy = 0.25 * g.idy, qz = 0.25 * g.idz;
    KS_LAUNCH(c, k_nodal_post_cells, nblocks(g.N, BS), BS, B8 * (M + (9 + 3 * add_old + 3 * incr) * g.N), g, phi, vel, vo, gp, qx, qy, qz,
              sigma * qx, sigma * qy, sigma * qz, add_old, incr);
    KS_LAUNCH(c, k_nodal_post_nodes, nblocks(M, BS), BS, B8 * (2 + incr) * M, M, phi, p, incr);
}
void launch_mac_rhs(Ctx& c, const Grid& g, const double* um, const double* vm, const double* wm, double* rhs, double* parts, int* np) {
    *np = parts_for(g.N);
    KS_LAUNCH(c, k_mac_rhs, *np, BS, B8 * (3 * g.N + g.NFz), g, um, vm, wm, rhs, parts, *np);
}
void launch_mac_divmax(Ctx& c, const Grid& g, const double* um, const double* vm, const double* wm, double* parts, int* np) {
    *np = parts_for(g.N);
    KS_LAUNCH(c, k_mac_divmax, *np, BS, B8 * (2 * g.N + g.NFz), g, um, vm, wm, parts, *np);
}
void launch_mac_correct(Ctx& c, const Grid& g, const double* phi, double* um, double* vm, double* wm, double beta, int plain) {
    const auto run = plain ? k_mac_correct<1> : k_mac_correct<0>;
    KS_LAUNCH_NAMED(c, "k_mac_correct", run, nblocks(g.N, BS), BS, B8 * 7 * g.N, g, phi, um, vm, wm, beta, beta * g.idx, beta * g.idy, beta * g.idz);
}
void launch_cfl(Ctx& c, const Grid& g, const double* vel, const double* src, const double* mu, double rho, double* parts, int* np) {
    *np = parts_for(g.N);
    KS_LAUNCH(c, k_cfl, *np, BS, B8 * 7 * g.N, g, vel, src, mu, rho, parts, *np);
}
void launch_ke(Ctx& c, const Grid& g, const double* vel, double rho, double* parts, int* np) {
    *np = parts_for(g.N);
    KS_LAUNCH(c, k_ke, *np, BS, B8 * 3 * g.N, g, vel, rho, parts);
}
void launch_reduce(Ctx& c, const double* parts, int np, int ncomp, int op_max, double* out) {
    KS_LAUNCH(c, k_reduce, ncomp, 256, B8 * (np + 1) * ncomp, parts, np, op_max, out);
}
void launch_sub_ratio(Ctx& c, double* a, long long n, const double* s, double den, double* parts, int* np) {
    const int nb = parts_for(n);
    if (np) *np = nb;
    KS_LAUNCH(c, k_sub_ratio, nb, BS, B8 * 2 * n, a, n, s, den, parts);
}
void launch_act_sample(Ctx& c, const Grid& g, const double* vel, const double* pts, int npts, const double plo[3], double* out) {
    KS_LAUNCH(c, k_act_sample, nblocks(npts, 64), 64, B8 * 6 * npts, g, vel, pts, npts, plo[0], plo[1], plo[2], out);
}
void launch_act_tables(Ctx& c, const Grid& g, const ActDisk* D, int nd, long long entries, const double* pts, const double plo[3], double* E,
                       float* R) {
    const long long b = (entries / std::max(1, nd) + BS - 1) / BS;
    const dim3 grid((unsigned)std::max(1LL, std::min(1024LL, b)), (unsigned)nd);
    KS_LAUNCH(c, k_act_tables, grid, BS, 12.0 * entries, g, D, pts, plo[0], plo[1], plo[2], E, R);
}
void launch_act_spread(Ctx& c, const Grid& g, double* act, const ActDisk* D, int d0, int nd, long long cells, const double* pts, const double* w,
                       const double* E, const float* R, const double plo[3]) {
    const dim3 grid(nblocks(cells, 128), (unsigned)nd);
    KS_LAUNCH(c, k_act_spread, grid, 128, B8 * 6 * cells * nd, g, act, D, d0, pts, w, E, R, plo[0], plo[1], plo[2]);
}
void launch_act_adj_dot(Ctx& c, const Grid& g, const double* actb, const ActDisk* D, int nd, long long cells, const double* pts, const double* w,
                        const double* E, const float* R, const double plo[3], double* parts) {
    const dim3 grid(kActParts, (unsigned)nd);
    KS_LAUNCH(c, k_act_adj_dot, grid, 128, B8 * 3 * cells * nd, g, actb, D, pts, w, E, R, plo[0], plo[1], plo[2], parts);
}

}  // namespace ks
