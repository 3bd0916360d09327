// Effective potential on sm_100a: the rest of an SCF iteration's potential update
// (src/physics/EffectivePotential.cpp:44-177, non-spin-polarised):
//   * FD first derivatives of a scalar field (src/operators/Gradient.cpp:17-60), periodic or
//     zero (Dirichlet) ghosts per direction;
//   * GGA-PBE exchange-correlation per grid point and the divergence of the GGA flux
//     (src/xc/XCFunctional.cpp:193-273; the reference evaluates the functional with libxc's
//     XC_GGA_X_PBE + XC_GGA_C_PBE, here it is this file's own restatement of the published
//     functional, below);
//   * the vector kernels of the AAR Poisson iteration (src/solvers/PoissonSolver.cpp:43-159):
//     fused preconditioner / history / save, Richardson and Anderson updates, residual, and
//     deterministic dot products (fixed block partition, fixed-order sums).
// FP64 throughout; one field of nd = nx ny nz points, x fastest.
#include <cmath>
#include <type_traits>

#include "kernels.h"
#include "lynx_common.cuh"

namespace lynxb {

namespace {

constexpr int kVThreads = 256;
constexpr int kDotBlocks = 296;  // 2 x 148 SMs: the dot-product partition (fixed, so sums are reproducible)

// d/d(direction) of x at a point: sum_{p=1..R} D1[p] (x[+p] - x[-p]), accumulated from zero in
// increasing p (the reference's order); ghosts wrap (periodic) or read zero (Dirichlet).  o: the point,
// c: its position of n along the direction, s: the element stride.
template <int R>
__device__ __forceinline__ double fd_deriv(const double* __restrict__ x, const double* __restrict__ d1, int o, int c,
                                           int n, int s, bool per) {
    double u[R], d[R];
#pragma unroll
    for (int p = 1; p <= R; ++p) {
        const bool wu = c + p >= n, wd = c - p < 0;
        u[p - 1] = x[o + (wu ? p - n : p) * s];
        d[p - 1] = x[o + (wd ? n - p : -p) * s];
        if (wu && !per) u[p - 1] = 0.0;
        if (wd && !per) d[p - 1] = 0.0;
    }
    double val = 0.0;
#pragma unroll
    for (int p = 1; p <= R; ++p) val += d1[p] * (u[p - 1] - d[p - 1]);
    return val;
}

// ------------------------------------------------------------------------------------------
// GGA-PBE, spin-unpolarised, as published: J. P. Perdew, K. Burke, M. Ernzerhof, Phys. Rev.
// Lett. 77, 3865 (1996), with the uniform-gas correlation of J. P. Perdew, Y. Wang, Phys. Rev.
// B 45, 13244 (1992).  Energy per particle
//   eps = eps_x^unif(rho) F_x(s) + eps_c^unif(r_s) + H(r_s, t),
//   eps_x^unif = -(3/4)(3/pi)^(1/3) rho^(1/3),  k_F = (3 pi^2 rho)^(1/3),  s^2 = sigma / (2 k_F rho)^2,
//   F_x = 1 + kappa - kappa / (1 + mu s^2 / kappa),
//   eps_c^unif = -2 A (1 + a1 r_s) ln(1 + 1 / (2 A (b1 r_s^(1/2) + b2 r_s + b3 r_s^(3/2) + b4 r_s^2))),
//   t^2 = sigma / (2 k_s rho)^2 with k_s^2 = 4 k_F / pi,
//   H = gamma ln(1 + (beta/gamma) t^2 (1 + A' t^2) / (1 + A' t^2 + A'^2 t^4)),
//   A' = (beta/gamma) / (exp(-eps_c^unif / gamma) - 1),  gamma = (1 - ln 2) / pi^2.
// Constants: kappa = 0.804, beta = 0.06672455060314922, mu = beta pi^2 / 3; PW92 parameters for
// zeta = 0 with A at the 7-digit value 0.0310907 (the "modified" PW92 that PBE correlation is
// usually paired with).  vrho = d(rho eps)/d rho and vsigma = d(rho eps)/d sigma are carried
// alongside the value as forward-mode dual numbers, exact to rounding.
// ------------------------------------------------------------------------------------------
struct Dual {
    double v, r, s;  // value, d/d rho, d/d sigma
};
__device__ __forceinline__ Dual dconst(double c) { return {c, 0.0, 0.0}; }
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.r + b.r, a.s + b.s}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.r - b.r, a.s - b.s}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) {
    return {a.v * b.v, a.r * b.v + a.v * b.r, a.s * b.v + a.v * b.s};
}
__device__ __forceinline__ Dual operator*(double c, Dual a) { return {c * a.v, c * a.r, c * a.s}; }
__device__ __forceinline__ Dual operator+(double c, Dual a) { return {c + a.v, a.r, a.s}; }
__device__ __forceinline__ Dual operator*(Dual a, double c) { return {c * a.v, c * a.r, c * a.s}; }
__device__ __forceinline__ Dual operator-(double c, Dual a) { return {c - a.v, -a.r, -a.s}; }
// one division for the value and one reciprocal for both derivatives (FP64 divisions are most of the
// functional's time)
__device__ __forceinline__ Dual operator/(double c, Dual a) {
    const double i = 1.0 / a.v, q = c / a.v, m = -q * i;
    return {q, m * a.r, m * a.s};
}
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    const double i = 1.0 / b.v, q = a.v / b.v;
    return {q, (a.r - q * b.r) * i, (a.s - q * b.s) * i};
}
__device__ __forceinline__ Dual dlog(Dual a) {
    const double i = 1.0 / a.v;
    return {log(a.v), a.r * i, a.s * i};
}
__device__ __forceinline__ Dual dexp(Dual a) {
    const double e = exp(a.v);
    return {e, e * a.r, e * a.s};
}
__device__ __forceinline__ Dual dsqrt(Dual a) {
    const double q = sqrt(a.v);
    const double h = 0.5 / q;
    return {q, h * a.r, h * a.s};
}
__device__ __forceinline__ Dual dcbrt(Dual a) {
    const double q = cbrt(a.v);
    const double h = 1.0 / (3.0 * q * q);
    return {q, h * a.r, h * a.s};
}

constexpr double kPi = 3.14159265358979323846;
constexpr double kPbeKappa = 0.804;
constexpr double kPbeBeta = 0.06672455060314922;

__device__ void pbe_point(double rho, double sigma, double* exc, double* vrho, double* vsigma) {
    const double mu = kPbeBeta * kPi * kPi / 3.0;
    const double gam = (1.0 - log(2.0)) / (kPi * kPi);
    const double cx = 0.75 * cbrt(3.0 / kPi);       // -eps_x^unif / rho^(1/3)
    const double ckf = cbrt(3.0 * kPi * kPi);       // k_F / rho^(1/3)
    const double c31 = cbrt(3.0 / (4.0 * kPi));     // r_s rho^(1/3)
    const double pwA = 0.0310907, pwa1 = 0.21370, pwb1 = 7.5957, pwb2 = 3.5876, pwb3 = 1.6382, pwb4 = 0.49294;
    const Dual r{rho, 1.0, 0.0}, s{sigma, 0.0, 1.0};
    const Dual r13 = dcbrt(r);
    const Dual kf = ckf * r13;
    const Dual rr = r * r;
    // exchange
    const Dual exu = (-cx) * r13;
    const Dual s2 = s / (4.0 * (kf * kf * rr));
    const Dual fx = (1.0 + kPbeKappa) - kPbeKappa / (1.0 + (mu / kPbeKappa) * s2);
    // correlation
    const Dual rs = c31 / r13;
    const Dual srs = dsqrt(rs);
    const Dual den = (2.0 * pwA) * (pwb1 * srs + pwb2 * rs + pwb3 * (rs * srs) + pwb4 * (rs * rs));
    const Dual ecu = (-2.0 * pwA) * ((1.0 + pwa1 * rs) * dlog(1.0 + dconst(1.0) / den));
    const Dual t2 = s * (kPi / 16.0) / (kf * rr);
    const Dual Ap = (kPbeBeta / gam) / (dexp((-1.0 / gam) * ecu) - dconst(1.0));
    const Dual At2 = Ap * t2;
    const Dual H = gam * dlog(1.0 + (kPbeBeta / gam) * (t2 * (1.0 + At2) / (1.0 + At2 + At2 * At2)));
    const Dual eps = exu * fx + ecu + H;
    const Dual F = r * eps;
    *exc = eps.v;
    *vrho = F.r;
    *vsigma = F.s;
}

// rho_xc = max(rho + rho_core, 1e-14): the density the functional sees when a core density is
// given (src/physics/EffectivePotential.cpp:127-134).
__global__ void rho_xc_kernel(const double* __restrict__ rho, const double* __restrict__ core,
                              double* __restrict__ out, long long nd) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nd; t += (long long)gridDim.x * blockDim.x) {
        const double v = rho[t] + core[t];
        out[t] = (v > 1e-14) ? v : 1e-14;
    }
}

// Per point: the gradient of rho, sigma (lapc_T metric for non-orthogonal cells), the functional, and the
// GGA flux f = v2xc lapc_T grad(rho).  Points with rho <= 1e-14 contribute nothing (exc = vrho = v2xc
// = 0).  With rhs: also the Poisson right-hand side 4 pi (rho0 + rho_b) (rho0: without the core density).
// 36 neighbours through L1, three fields less written and read than with the gradient apart; with the
// divisions of the derivatives shared, and no host step before the last kernel, the whole potential of
// 90^3 points takes 0.157 ms (0.299 with 19 launches and two mean values read back in between).
template <int R>
__global__ void __launch_bounds__(128)
    grad_pbe_kernel(const double* __restrict__ rho, const GradGeom g, const XcMetric m, double* __restrict__ fx,
                    double* __restrict__ fy, double* __restrict__ fz, double* __restrict__ vxc,
                    double* __restrict__ exc, double* __restrict__ v2xc, const double* __restrict__ rho0,
                    const double* __restrict__ rho_b, double* __restrict__ rhs) {
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= g.nx * g.ny * g.nz) return;
    const int row = t / g.nx, i = t - row * g.nx, k = row / g.ny, j = row - k * g.ny;
    const double dx = fd_deriv<R>(rho, g.D1[0], t, i, g.nx, 1, g.periodic[0] != 0);
    const double dy = fd_deriv<R>(rho, g.D1[1], t, j, g.ny, g.nx, g.periodic[1] != 0);
    const double dz = fd_deriv<R>(rho, g.D1[2], t, k, g.nz, g.nx * g.ny, g.periodic[2] != 0);
    const double rx = rho[t];
    double sig;
    if (m.orth) {
        sig = dx * dx + dy * dy + dz * dz;
    } else {
        sig = m.L[0] * dx * dx + m.L[4] * dy * dy + m.L[8] * dz * dz + 2.0 * m.L[1] * dx * dy +
              2.0 * m.L[2] * dx * dz + 2.0 * m.L[5] * dy * dz;
    }
    double e = 0.0, vr = 0.0, vs = 0.0;
    if (rx > 1e-14) pbe_point(rx, sig, &e, &vr, &vs);
    const double w = 2.0 * vs;
    exc[t] = e;
    vxc[t] = vr;
    if (v2xc) v2xc[t] = w;
    if (m.orth) {
        fx[t] = dx * w;
        fy[t] = dy * w;
        fz[t] = dz * w;
    } else {
        fx[t] = (m.L[0] * dx + m.L[1] * dy + m.L[2] * dz) * w;
        fy[t] = (m.L[3] * dx + m.L[4] * dy + m.L[5] * dz) * w;
        fz[t] = (m.L[6] * dx + m.L[7] * dy + m.L[8] * dz) * w;
    }
    if (rhs) {
        const double fpi = 4.0 * kPi;
        double q = fpi * rho0[t];
        if (rho_b) q += fpi * rho_b[t];
        rhs[t] = q;
    }
}

// v -= d_x fx, then -= d_y fy, then -= d_z fz (the reference's three separate updates, in order); with
// phi: also veff = v + phi.
template <int R>
__global__ void __launch_bounds__(128)
    div_sub_kernel(double* __restrict__ v, const GradGeom g, const double* __restrict__ fx,
                   const double* __restrict__ fy, const double* __restrict__ fz, const double* __restrict__ phi,
                   double* __restrict__ veff) {
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= g.nx * g.ny * g.nz) return;
    const int row = t / g.nx, i = t - row * g.nx, k = row / g.ny, j = row - k * g.ny;
    double a = v[t];
    a -= fd_deriv<R>(fx, g.D1[0], t, i, g.nx, 1, g.periodic[0] != 0);
    a -= fd_deriv<R>(fy, g.D1[1], t, j, g.ny, g.nx, g.periodic[1] != 0);
    a -= fd_deriv<R>(fz, g.D1[2], t, k, g.nz, g.nx * g.ny, g.periodic[2] != 0);
    v[t] = a;
    if (phi) veff[t] = a + phi[t];
}

// ------------------------------------------------------------------------------------------
// AAR vector kernels.
// ------------------------------------------------------------------------------------------
// f = w r; with col >= 0 the history column col: X = x - x_old, F = f - f_old; then x_old = x,
// f_old = f (src/solvers/PoissonSolver.cpp:103-115 in one pass).
__global__ void aar_pre_kernel(const double* __restrict__ r, const double* __restrict__ x, double* __restrict__ x_old,
                               double* __restrict__ f, double* __restrict__ f_old, double* __restrict__ X,
                               double* __restrict__ F, double w, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double fi = w * r[t];
        const double xi = x[t];
        if (X) {
            X[t] = xi - x_old[t];
            F[t] = fi - f_old[t];
        }
        x_old[t] = xi;
        f_old[t] = fi;
        f[t] = fi;
    }
}

// x = x_old + c f - sum_j g[j] (X_j + c F_j)   (Richardson: cols = 0, c = omega)
__global__ void aar_update_kernel(double* __restrict__ x, const double* __restrict__ x_old, const double* __restrict__ f,
                                  const double* __restrict__ X, const double* __restrict__ F, AarGamma g, double c,
                                  long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        double v = x_old[t] + c * f[t];
        for (int j = 0; j < g.cols; ++j) v -= g.g[j] * (X[(long long)j * n + t] + c * F[(long long)j * n + t]);
        x[t] = v;
    }
}

__global__ void sub_kernel(const double* __restrict__ b, const double* __restrict__ a, double* __restrict__ r,
                           long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        r[t] = b[t] - a[t];
}

// Partial sums of up to kMaxDots dot products u_k . v_k over a fixed partition of [0, n):
// part[k * gridDim.x + block].  Block sums in a fixed shared-memory tree.
__global__ void dots_partial_kernel(DotList L, long long n, double* __restrict__ part) {
    __shared__ double sh[kVThreads];
    const long long per = (n + gridDim.x - 1) / gridDim.x;
    const long long lo = blockIdx.x * per;
    const long long hi = min(n, lo + per);
    for (int k = 0; k < L.count; ++k) {
        double a = 0.0;
        for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) a += L.u[k][t] * L.v[k][t];
        sh[threadIdx.x] = a;
        __syncthreads();
        for (int h = blockDim.x / 2; h > 0; h >>= 1) {
            if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
            __syncthreads();
        }
        if (threadIdx.x == 0) part[(long long)k * gridDim.x + blockIdx.x] = sh[0];
        __syncthreads();
    }
}

// out[k] = sum over blocks of part[k][*], in a fixed tree (one CTA per dot).
__global__ void dots_final_kernel(const double* __restrict__ part, int nblk, double* __restrict__ out) {
    __shared__ double sh[kVThreads];
    double a = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) a += part[(long long)blockIdx.x * nblk + b];
    sh[threadIdx.x] = a;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

// out = sa a (+ sa b) - s   (b may be null)
__global__ void add_shift_kernel(const double* __restrict__ a, const double* __restrict__ b, double s, double sa,
                                 double* __restrict__ out, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        double v = sa * a[t];
        if (b) v += sa * b[t];
        out[t] = v - s;
    }
}

// z[i] *= s[i] * scale over the half-spectrum of a real 3-D FFT (the periodic Poisson solve).
__global__ void spec_scale_kernel(double2* __restrict__ z, const double* __restrict__ s, double scale, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double f = s[t] * scale;
        z[t] = make_double2(z[t].x * f, z[t].y * f);
    }
}

// s[i] = 1 / Re(g_hat[i]) (0 for the mean mode i = 0 and for modes whose symbol vanishes).
__global__ void inv_symbol_kernel(const double2* __restrict__ g, double* __restrict__ s, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double v = g[t].x;
        s[t] = (t == 0 || fabs(v) < 1e-300) ? 0.0 : 1.0 / v;
    }
}

int grid_for(long long n) {
    long long b = (n + kVThreads - 1) / kVThreads;
    if (b > 148 * 16) b = 148 * 16;
    return (int)(b < 1 ? 1 : b);
}

int launch_ok(const char* what) {
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s launch failed: %s", what, cudaGetErrorString(e));
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

}  // namespace

namespace {
template <typename F>
int with_radius(int R, F f) {
    switch (R) {
        case 1: f(std::integral_constant<int, 1>{}); return LYNX_OK;
        case 2: f(std::integral_constant<int, 2>{}); return LYNX_OK;
        case 3: f(std::integral_constant<int, 3>{}); return LYNX_OK;
        case 4: f(std::integral_constant<int, 4>{}); return LYNX_OK;
        case 5: f(std::integral_constant<int, 5>{}); return LYNX_OK;
        case 6: f(std::integral_constant<int, 6>{}); return LYNX_OK;
        case 7: f(std::integral_constant<int, 7>{}); return LYNX_OK;
        case 8: f(std::integral_constant<int, 8>{}); return LYNX_OK;
        default: set_error("FD half-width %d outside the supported range 1..8", R); return LYNX_ERR_UNSUPPORTED;
    }
}
}  // namespace

int launch_div_sub(double* v, const GradGeom& g, const double* fx, const double* fy, const double* fz,
                   const double* phi, double* veff, cudaStream_t st) {
    const int blocks = (int)(((long long)g.nx * g.ny * g.nz + 127) / 128);
    LYNX_TRY(with_radius(g.R, [&](auto r) {
        div_sub_kernel<decltype(r)::value><<<blocks, 128, 0, st>>>(v, g, fx, fy, fz, phi, veff);
    }));
    return launch_ok("GGA divergence");
}

int launch_rho_xc(const double* rho, const double* core, double* out, long long nd, cudaStream_t st) {
    rho_xc_kernel<<<grid_for(nd), kVThreads, 0, st>>>(rho, core, out, nd);
    return launch_ok("core density");
}

int launch_grad_pbe(const double* rho, const GradGeom& g, const XcMetric& m, double* fx, double* fy, double* fz,
                    double* vxc, double* exc, double* v2xc, const double* rho0, const double* rho_b, double* rhs,
                    cudaStream_t st) {
    const int blocks = (int)(((long long)g.nx * g.ny * g.nz + 127) / 128);
    LYNX_TRY(with_radius(g.R, [&](auto r) {
        grad_pbe_kernel<decltype(r)::value><<<blocks, 128, 0, st>>>(rho, g, m, fx, fy, fz, vxc, exc, v2xc, rho0, rho_b,
                                                                    rhs);
    }));
    return launch_ok("GGA-PBE");
}

int launch_aar_pre(const double* r, const double* x, double* x_old, double* f, double* f_old, double* X, double* F,
                   double w, long long n, cudaStream_t st) {
    aar_pre_kernel<<<grid_for(n), kVThreads, 0, st>>>(r, x, x_old, f, f_old, X, F, w, n);
    return launch_ok("AAR preconditioner");
}

int launch_aar_update(double* x, const double* x_old, const double* f, const double* X, const double* F,
                      const AarGamma& g, double c, long long n, cudaStream_t st) {
    aar_update_kernel<<<grid_for(n), kVThreads, 0, st>>>(x, x_old, f, X, F, g, c, n);
    return launch_ok("AAR update");
}

int launch_sub(const double* b, const double* a, double* r, long long n, cudaStream_t st) {
    sub_kernel<<<grid_for(n), kVThreads, 0, st>>>(b, a, r, n);
    return launch_ok("residual");
}

int launch_add_shift(const double* a, const double* b, double s, double sa, double* out, long long n,
                     cudaStream_t st) {
    add_shift_kernel<<<grid_for(n), kVThreads, 0, st>>>(a, b, s, sa, out, n);
    return launch_ok("shift");
}

int launch_spec_scale(double2* z, const double* s, double scale, long long n, cudaStream_t st) {
    spec_scale_kernel<<<grid_for(n), kVThreads, 0, st>>>(z, s, scale, n);
    return launch_ok("spectral scale");
}

int launch_inv_symbol(const double2* g, double* s, long long n, cudaStream_t st) {
    inv_symbol_kernel<<<grid_for(n), kVThreads, 0, st>>>(g, s, n);
    return launch_ok("Poisson symbol");
}

size_t dots_work_bytes() { return sizeof(double) * ((size_t)kMaxDots * kDotBlocks + kMaxDots); }

int launch_dots(const DotList& L, long long n, void* work, double* host_out, cudaStream_t st) {
    if (L.count <= 0 || L.count > kMaxDots) {
        set_error("internal error: %d dot products (at most %d)", L.count, kMaxDots);
        return LYNX_ERR_BAD_ARG;
    }
    double* part = static_cast<double*>(work);
    double* out = part + (size_t)kMaxDots * kDotBlocks;
    dots_partial_kernel<<<kDotBlocks, kVThreads, 0, st>>>(L, n, part);
    LYNX_TRY(launch_ok("dot products"));
    dots_final_kernel<<<L.count, kVThreads, 0, st>>>(part, kDotBlocks, out);
    LYNX_TRY(launch_ok("dot products"));
    LYNX_CUDA_TRY(cudaMemcpyAsync(host_out, out, sizeof(double) * L.count, cudaMemcpyDeviceToHost, st));
    LYNX_CUDA_TRY(cudaStreamSynchronize(st));
    return LYNX_OK;
}

}  // namespace lynxb
