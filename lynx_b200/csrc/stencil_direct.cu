// Chebyshev step, one thread per grid point, neighbours straight from global memory (L1 / L2):
//
//   out = a * (-0.5 * Lap x + V .* x) + b * x + d * xold
//
// Used for complex blocks of any size and for small real ones.
//   * A step of a small cell (Si8 at 10 states: 1.2 MB a block, all of it in L2) is bound by latency:
//     the pipelined kernel's prologue (barriers, first bulk copies, 13 planes of the z-window) and
//     its long unrolled code take longer than the work.  Here the 6 R loads of a point are
//     independent, so a launch is about one memory latency: 7.2 us against 9.6 (24^3, 10 states,
//     FP32), 5.0 against 9.3 for one state.  The loads bind above 1.25 MB a block (6 R words a point
//     through L1 against about 8 in the pipelined kernel): 28^3, 24 states, FP32 15.6 us against
//     11.4.  The rule direct_step_pays draws the line there.
//   * Complex blocks: a window of 2R + 1 complex planes leaves the pipelined kernel one or two points a
//     thread, too few warps and a long chain of phase products; here the many resident threads hide
//     the loads and a wrapped neighbour costs one product.  Si8 at a k-point, 32^3, 24 states: 27.9
//     us against 60 (FP32), 68.7 against 88.9 (FP64); 44^3, 40 states: 102 against 232, 309 against
//     735.  A whole degree of Si64 at a k-point, 60^3, 160 states: 1.36 ms against 2.76 (FP32), 3.69
//     against 6.23 (FP64).
//
// Sums in the pipelined kernel's order (z pairs, y rows from below, x pairs, centre, V, xold).
// Non-orthogonal cells: the first derivatives along y and z, which the mixed terms are made of, come
// from the same loads.
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "lynx_common.cuh"
#include "stencil.cuh"

namespace lynxb {
namespace {

template <typename T>
struct DirectArgs {
    using S = typename ScalarOf<T>::type;
    int nx, ny, nz, nxp;
    long long ld_x, ld_old, ld_out, ld_g;
    S cx[kMaxR1], cy[kMaxR1], cz[kMaxR1], d1y[kMaxR1], d1z[kMaxR1];
    S diag, diag_lo, a, d;
    T phl[3], phr[3];
};

template <typename T, int R, bool XOLD, bool GRAD>
__global__ void __launch_bounds__(128)
    direct_step_kernel(const T* x, const T* xold, T* __restrict__ out, const typename ScalarOf<T>::type* V,
                       T* __restrict__ gy, T* __restrict__ gz, const DirectArgs<T> A) {
    using S = typename ScalarOf<T>::type;
    pdl_wait();
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= A.nx * A.ny * A.nz) return;
    const int row = t / A.nx, i = t - row * A.nx;
    const int k = row / A.ny, j = row - k * A.ny;
    const int plane = A.nxp * A.ny;
    const int o = row * A.nxp + i;
    const T* xb = x + (long long)blockIdx.y * A.ld_x;
    // neighbour at distance p along one direction (position c of n, element stride s), times the
    // ghost multiplier where it wraps
    auto up = [&](int c, int n, int s, int p, const T& ph) {
        const bool w = c + p >= n;
        const T v = xb[o + (w ? p - n : p) * s];
        return w ? pmul(v, ph) : v;
    };
    auto dn = [&](int c, int n, int s, int p, const T& ph) {
        const bool w = c - p < 0;
        const T v = xb[o + (w ? n - p : -p) * s];
        return w ? pmul(v, ph) : v;
    };
    T zu[R], zd[R], yu[R], yd[R], xu[R], xd[R];
#pragma unroll
    for (int p = 1; p <= R; ++p) {
        zu[p - 1] = up(k, A.nz, plane, p, A.phr[2]);
        zd[p - 1] = dn(k, A.nz, plane, p, A.phl[2]);
        yu[p - 1] = up(j, A.ny, A.nxp, p, A.phr[1]);
        yd[p - 1] = dn(j, A.ny, A.nxp, p, A.phl[1]);
        xu[p - 1] = up(i, A.nx, 1, p, A.phr[0]);
        xd[p - 1] = dn(i, A.nx, 1, p, A.phl[0]);
    }
    const T xc = xb[o];
    T xo;
    if constexpr (XOLD) xo = xold[(long long)blockIdx.y * A.ld_old + o];
    const S v = V[o];
    T acc = vscale(A.cz[1], vadd(zu[0], zd[0]));
#pragma unroll
    for (int p = 2; p <= R; ++p) acc = fmac(acc, A.cz[p], vadd(zu[p - 1], zd[p - 1]));
#pragma unroll
    for (int p = R; p >= 1; --p) acc = fmac(acc, A.cy[p], yd[p - 1]);
#pragma unroll
    for (int p = 1; p <= R; ++p) acc = fmac(acc, A.cy[p], yu[p - 1]);
#pragma unroll
    for (int p = 1; p <= R; ++p) acc = fmac(acc, A.cx[p], vadd(xu[p - 1], xd[p - 1]));
    acc = fmac(acc, A.diag, xc);
    if (sizeof(S) == sizeof(float)) acc = fmac(acc, A.diag_lo, xc);
    acc = fmac(acc, A.a * v, xc);
    if constexpr (XOLD) acc = fmac(acc, A.d, xo);
    out[(long long)blockIdx.y * A.ld_out + o] = acc;
    if constexpr (GRAD) {
        T sy = vzero(T()), sz = vzero(T());
#pragma unroll
        for (int p = 1; p <= R; ++p) {
            sy = fmac(sy, A.d1y[p], vadd(yu[p - 1], vscale(S(-1), yd[p - 1])));
            sz = fmac(sz, A.d1z[p], vadd(zu[p - 1], vscale(S(-1), zd[p - 1])));
        }
        gy[(long long)blockIdx.y * A.ld_g + o] = sy;
        gz[(long long)blockIdx.y * A.ld_g + o] = sz;
    }
}

}  // namespace

template <typename T, typename S>
int launch_direct_step(const StencilGeom& g, int nxp, const T* x, long long ldx, const T* xold, long long ldo, T* out,
                       long long ldout, const S* V, int ncol, double a, double b, double d, const T* phl,
                       const T* phr, const NonOrthGeom* ng, T* gy, T* gz, long long ldg, cudaStream_t st) {
    if (g.R < 1 || g.R > 8) {
        set_error("FD half-width %d outside the supported range 1..8", g.R);
        return LYNX_ERR_UNSUPPORTED;
    }
    if (g.nx < g.R || g.ny < g.R || g.nz < g.R) {
        set_error("grid %dx%dx%d smaller than the FD half-width %d", g.nx, g.ny, g.nz, g.R);
        return LYNX_ERR_UNSUPPORTED;
    }
    if (g.nx > kDirectMaxNx) {
        set_error("nx = %d above the supported maximum %d", g.nx, kDirectMaxNx);
        return LYNX_ERR_UNSUPPORTED;
    }
    if (ncol <= 0) return LYNX_OK;
    if (ncol > 65535) {
        set_error("too many columns (%d) for one launch", ncol);
        return LYNX_ERR_UNSUPPORTED;
    }
    DirectArgs<T> A;
    A.nx = g.nx;
    A.ny = g.ny;
    A.nz = g.nz;
    A.nxp = nxp;
    A.ld_x = ldx;
    A.ld_old = ldo;
    A.ld_out = ldout;
    A.ld_g = ldg;
    for (int p = 0; p < kMaxR1; ++p) {
        const bool in = p >= 1 && p <= g.R;
        A.cx[p] = in ? (S)(-0.5 * a * g.D2x[p]) : S(0);
        A.cy[p] = in ? (S)(-0.5 * a * g.D2y[p]) : S(0);
        A.cz[p] = in ? (S)(-0.5 * a * g.D2z[p]) : S(0);
        A.d1y[p] = in && ng ? (S)ng->D1y[p] : S(0);
        A.d1z[p] = in && ng ? (S)ng->D1z[p] : S(0);
    }
    centre_coef<S>(g, a, b, A.cx, A.cy, A.cz, &A.diag, &A.diag_lo);
    A.a = (S)a;
    A.d = (S)d;
    for (int k = 0; k < 3; ++k) {
        A.phl[k] = phl[k];
        A.phr[k] = phr[k];
    }
    const int np = g.nx * g.ny * g.nz;
    dim3 grid((np + 127) / 128, ncol);
    const bool xo = xold != nullptr && d != 0.0;
    auto go = [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        auto kern = ng ? (xo ? direct_step_kernel<T, R, true, true> : direct_step_kernel<T, R, false, true>)
                       : (xo ? direct_step_kernel<T, R, true, false> : direct_step_kernel<T, R, false, false>);
        launch_pdl(kern, grid, 128, 0, st, x, xold, out, V, gy, gz, A);
    };
    switch (g.R) {
        case 1: go(std::integral_constant<int, 1>{}); break;
        case 2: go(std::integral_constant<int, 2>{}); break;
        case 3: go(std::integral_constant<int, 3>{}); break;
        case 4: go(std::integral_constant<int, 4>{}); break;
        case 5: go(std::integral_constant<int, 5>{}); break;
        case 6: go(std::integral_constant<int, 6>{}); break;
        case 7: go(std::integral_constant<int, 7>{}); break;
        case 8: go(std::integral_constant<int, 8>{}); break;
    }
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("direct stencil launch failed: %s", cudaGetErrorString(e));
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

#define LYNX_DIRECT_INST(T, S)                                                                                      \
    template int launch_direct_step<T, S>(const StencilGeom&, int, const T*, long long, const T*, long long, T*,    \
                                          long long, const S*, int, double, double, double, const T*, const T*,     \
                                          const NonOrthGeom*, T*, T*, long long, cudaStream_t);
LYNX_DIRECT_INST(double, double)
LYNX_DIRECT_INST(float, float)
LYNX_DIRECT_INST(double2, double)
LYNX_DIRECT_INST(float2, float)

}  // namespace lynxb
