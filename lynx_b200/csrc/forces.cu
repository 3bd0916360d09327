// Nonlocal forces, nonlocal and kinetic stress (src/physics/Forces.cpp:509-797,
// src/physics/Stress.cpp:1041-1784), FP64.
//
// Both need projections of the orbitals' FD gradients, and only at the sphere points (a quarter of
// the grid).  The gradient blocks are never written: sphere_kernel takes the 36 neighbours of each
// sphere point straight from the orbitals (an atom's neighbourhood of one column fits in L1), and
// kinetic_kernel sums the six products of the gradients of all points as it marches through z.
// One read of the orbitals each.  Forces and stress of Si64 (60^3, 160 states) together: 12.3 ms with a
// gradient block written per direction (1.0 ms each), a gather of every block and three weighted copies
// of the projectors made on the host on each call (about 4 ms); 2.0 ms here.
#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "lynx_common.cuh"
#include "nonlocal.cuh"
#include "stencil.cuh"

namespace lynxb {
namespace {

__device__ __forceinline__ double re_cmul(double a, double b) { return a * b; }  // Re(conj(a) b)
__device__ __forceinline__ double re_cmul(double2 a, double2 b) { return a.x * b.x + a.y * b.y; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 vsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double phase_mul(double v, double, double) { return v; }
__device__ __forceinline__ double2 phase_mul(double2 v, double re, double im) { return acc_phase(v, re, im); }

template <typename T>
struct GradCoef {
    int nx, ny, nz, R, orth;
    double d1[3][kMaxR1];
    T phl[3], phr[3];
    double ui[9];  // Cartesian gradient = ui * lattice-direction gradients (non-orthogonal cells)
    double h[3], uvec[9];
};

// FD derivative of column x along one direction: position c of n, element stride s.
template <typename T>
__device__ __forceinline__ T fd_dir(const T* __restrict__ x, long long o, int c, int n, long long s, int R,
                                    const double* __restrict__ d1, const T& phl, const T& phr) {
    T g = vzero(T());
#pragma unroll 6
    for (int p = 1; p <= R; ++p) {
        const bool wu = c + p >= n, wd = c - p < 0;
        T u = x[o + (long long)(wu ? p - n : p) * s];
        T d = x[o + (long long)(wd ? n - p : -p) * s];
        if (wu) u = pmul(u, phr);
        if (wd) d = pmul(d, phl);
        g = fmac(g, d1[p], vsub(u, d));
    }
    return g;
}

// One CTA = one atom and one column.  Tiles of 256 sphere points: every thread evaluates one point
// (psi, and the gradient components - for the stress times the position relative to the image - all
// times the image's Bloch phase) into shared memory; then warp w accumulates the projections on
// projectors w, w + 8, ... with the lanes along the points.  The products of the projections, summed
// over the projectors with Gamma and weighted with the occupation, go to part[atom][column][NV + 1]:
// NV components and |alpha|^2.  FORCE: NV = 3, beta_d; STRESS: NV = 6, beta_ab for xx xy xz yy yz zz.
template <typename T, bool STRESS, int MJ>
__global__ void __launch_bounds__(256)
    sphere_kernel(const T* __restrict__ psi, long long ld, int ncol, NLView tab, const GradCoef<T> G,
                  const double* __restrict__ img_pos, const double* __restrict__ occ, double dV,
                  double* __restrict__ part) {
    constexpr int NV = STRESS ? 6 : 3;
    __shared__ T val[NV + 1][256];
    __shared__ long long cbase[256];
    __shared__ int cstride[256];
    __shared__ double red[8][NV + 1];
    const int a = blockIdx.x, n = blockIdx.y, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int np = tab.atom_nproj[a], poff = tab.atom_poff[a];
    const int i0 = tab.atom_img_ptr[a], i1 = tab.atom_img_ptr[a + 1];
    const double* chi = reinterpret_cast<const double*>(tab.chi);
    const T* x = psi + (long long)n * ld;
    int total = 0;
    if (np > 0)
        for (int ii = i0; ii < i1; ++ii) total += tab.img_ndc[tab.atom_img_list[ii]];
    T acc[MJ][NV + 1];
#pragma unroll
    for (int m = 0; m < MJ; ++m)
#pragma unroll
        for (int v = 0; v <= NV; ++v) acc[m][v] = vzero(T());
    for (int p0 = 0; p0 < total; p0 += 256) {
        __syncthreads();
        const int p = p0 + tid;
        if (p < total) {
            int l = p, im = 0, ndc = 0;
            for (int ii = i0; ii < i1; ++ii) {  // the point's image
                im = tab.atom_img_list[ii];
                ndc = tab.img_ndc[im];
                if (l < ndc) break;
                l -= ndc;
            }
            cbase[tid] = tab.img_chi_off[im] + l;
            cstride[tid] = ndc;
            const int o = tab.gpos[tab.img_goff[im] + l];
            const int row = o / G.nx, i = o - row * G.nx, k = row / G.ny, j = row - k * G.ny;
            T g[3] = {fd_dir(x, o, i, G.nx, 1, G.R, G.d1[0], G.phl[0], G.phr[0]),
                      fd_dir(x, o, j, G.ny, G.nx, G.R, G.d1[1], G.phl[1], G.phr[1]),
                      fd_dir(x, o, k, G.nz, (long long)G.nx * G.ny, G.R, G.d1[2], G.phl[2], G.phr[2])};
            const double pr = tab.img_phase[2 * im], pi = tab.img_phase[2 * im + 1];
            val[NV][tid] = phase_mul(x[o], pr, pi);
            if constexpr (STRESS) {
                if (!G.orth) {
                    T c[3];
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        c[q] = vadd(vadd(vscale(G.ui[3 * q], g[0]), vscale(G.ui[3 * q + 1], g[1])),
                                    vscale(G.ui[3 * q + 2], g[2]));
#pragma unroll
                    for (int q = 0; q < 3; ++q) g[q] = c[q];
                }
                double r[3] = {i * G.h[0] - img_pos[3 * im], j * G.h[1] - img_pos[3 * im + 1],
                               k * G.h[2] - img_pos[3 * im + 2]};
                if (!G.orth) {
                    const double r0 = r[0], r1 = r[1], r2 = r[2];
#pragma unroll
                    for (int q = 0; q < 3; ++q) r[q] = r0 * G.uvec[q] + r1 * G.uvec[3 + q] + r2 * G.uvec[6 + q];
                }
#pragma unroll
                for (int q = 0; q < 3; ++q) g[q] = phase_mul(g[q], pr, pi);
                val[0][tid] = vscale(r[0], g[0]);
                val[1][tid] = vscale(r[1], g[0]);
                val[2][tid] = vscale(r[2], g[0]);
                val[3][tid] = vscale(r[1], g[1]);
                val[4][tid] = vscale(r[2], g[1]);
                val[5][tid] = vscale(r[2], g[2]);
            } else {
#pragma unroll
                for (int q = 0; q < 3; ++q) val[q][tid] = phase_mul(g[q], pr, pi);
            }
        }
        __syncthreads();
        const int np0 = min(256, total - p0);
        // the projector values of all eight steps of the tile first: their latency is paid once
        double c[8][MJ];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int q = min(lane + 32 * u, np0 - 1);
            const double* cp = chi + cbase[q];
            const long long st = cstride[q];
#pragma unroll
            for (int m = 0; m < MJ; ++m) c[u][m] = lane + 32 * u < np0 ? cp[min(w + 8 * m, np - 1) * st] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int q = min(lane + 32 * u, np0 - 1);
#pragma unroll
            for (int v = 0; v <= NV; ++v) {
                const T xv = val[v][q];
#pragma unroll
                for (int m = 0; m < MJ; ++m) acc[m][v] = fmac(acc[m][v], c[u][m], xv);
            }
        }
    }
    double s[NV + 1];
#pragma unroll
    for (int v = 0; v <= NV; ++v) s[v] = 0.0;
#pragma unroll
    for (int m = 0; m < MJ; ++m) {
        const int jp = w + 8 * m;
#pragma unroll
        for (int v = 0; v <= NV; ++v)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[m][v] = vadd(acc[m][v], shfl_x(acc[m][v], o));
        if (jp < np) {
            const double gm = tab.gamma[poff + jp] * dV * dV;
#pragma unroll
            for (int v = 0; v <= NV; ++v) s[v] = fma(gm, re_cmul(acc[m][NV], acc[m][v]), s[v]);
        }
    }
    if (lane == 0)
#pragma unroll
        for (int v = 0; v <= NV; ++v) red[w][v] = s[v];
    __syncthreads();
    if (tid <= NV) {
        double t = 0.0;
        for (int u = 0; u < 8; ++u) t += red[u][tid];
        part[((long long)a * ncol + n) * (NV + 1) + tid] = occ[n] * t;
    }
}

// out[a * nv + v] = scale * sum over the columns of part[a][n][v] (v < nv), ea[a] = escale * the last.
__global__ void __launch_bounds__(256)
    sphere_reduce_kernel(const double* __restrict__ part, int ncol, int nv, double scale, double escale,
                         double* __restrict__ out, double* __restrict__ ea) {
    __shared__ double red[8];
    const int a = blockIdx.x, v = blockIdx.y;
    double s = 0.0;
    for (int n = threadIdx.x; n < ncol; n += 256) s += part[((long long)a * ncol + n) * (nv + 1) + v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int u = 0; u < 8; ++u) t += red[u];
        if (v < nv) out[a * nv + v] = scale * t;
        else ea[a] = escale * t;
    }
}

// Six products of the Cartesian gradients, part[column][CTA of the column][6] = sum over the CTA's
// points of Re(conj(g_a) g_b).  CTA = a band of rows of one column and a chunk of planes; a thread
// owns two rows' points at one x and marches through z with the 2 R + 1 planes of its points in
// registers (complex: one row's); the plane's rows with R halo rows on either side are staged in shared memory for the x
// and y neighbours (three buffers: the copies of the next two planes overlap this plane's sums, and one
// barrier a plane suffices).
constexpr int kKinThreads = 512;
template <typename T> constexpr int kin_ry() { return ScalarOf<T>::cplx ? 1 : 2; }  // window registers
template <typename T, int R, bool PH>
__global__ void __launch_bounds__(kKinThreads, 1)
    kinetic_kernel(const T* __restrict__ psi, long long ld, const GradCoef<T> G, int tyt, int zchunk, int ncta,
                   double* __restrict__ part) {
    constexpr int RY = kin_ry<T>(), W = 2 * R + 1;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* tile = reinterpret_cast<T*>(sm_raw);  // [3][TY + 2R][nx]
    __shared__ double red[kKinThreads / 32][6];
    const int nx = G.nx, ny = G.ny, nz = G.nz, tid = threadIdx.x;
    const int TY = tyt * RY, rows = TY + 2 * R;
    const int y0 = blockIdx.x * TY, z0 = blockIdx.z * zchunk, z1 = min(nz, z0 + zchunk);
    const T* x = psi + (long long)blockIdx.y * ld;
    const int px = tid % nx, ty = tid / nx;
    const long long plane = (long long)nx * ny;
    bool own[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) own[r] = ty < tyt && y0 + ty * RY + r < ny;
    auto stage = [&](int z, int b) {
        const T* src = x + z * plane;
        T* dst = tile + (size_t)b * rows * nx;
        for (int e = tid; e < rows * nx; e += kKinThreads) {
            int gy = y0 - R + e / nx;
            gy += gy < 0 ? ny : 0;
            gy -= gy >= ny ? ny : 0;  // a band's last rows may lie past the cell: any valid row does
            gy = min(gy, ny - 1);
            const T* s = src + (long long)gy * nx + e % nx;
            if constexpr (sizeof(T) == 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(dst + e)), "l"(s) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(dst + e)), "l"(s) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto load = [&](int z, int r) {
        const bool wu = z >= nz, wd = z < 0;
        const int zz = wu ? z - nz : wd ? z + nz : z;
        T v = vzero(T());
        if (own[r]) v = x[zz * plane + (long long)(y0 + ty * RY + r) * nx + px];
        if (PH && wu) v = pmul(v, G.phr[2]);
        if (PH && wd) v = pmul(v, G.phl[2]);
        return v;
    };
    T win[W][RY];
#pragma unroll
    for (int k = 0; k < W; ++k)
#pragma unroll
        for (int r = 0; r < RY; ++r) win[k][r] = load(z0 - R + k, r);
    double s[6] = {0, 0, 0, 0, 0, 0};
    stage(z0, 0);
    if (z0 + 1 < z1) stage(z0 + 1, 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    int b = 0;
    for (int z = z0; z < z1; ++z) {
        T nxt[RY];
#pragma unroll
        for (int r = 0; r < RY; ++r) nxt[r] = z + 1 < z1 ? load(z + R + 1, r) : vzero(T());
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // the plane has landed, and every thread is done with the one before
        if (z + 2 < z1) stage(z + 2, b == 0 ? 2 : b - 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        const T* tl = tile + (size_t)b * rows * nx;
#pragma unroll
        for (int r = 0; r < RY; ++r) {
            if (!own[r]) continue;
            const int yl = ty * RY + r;
            const T* row = tl + (yl + R) * nx;
            T g[3] = {vzero(T()), vzero(T()), vzero(T())};
#pragma unroll
            for (int p = 1; p <= R; ++p) {
                const bool wu = px + p >= nx, wd = px - p < 0;
                T u = row[px + (wu ? p - nx : p)], d = row[px + (wd ? nx - p : -p)];
                if (PH && wu) u = pmul(u, G.phr[0]);
                if (PH && wd) d = pmul(d, G.phl[0]);
                g[0] = fmac(g[0], G.d1[0][p], vsub(u, d));
                u = row[px + p * nx];
                d = row[px - p * nx];
                if (PH && y0 + yl + p >= ny) u = pmul(u, G.phr[1]);
                if (PH && y0 + yl - p < 0) d = pmul(d, G.phl[1]);
                g[1] = fmac(g[1], G.d1[1][p], vsub(u, d));
                g[2] = fmac(g[2], G.d1[2][p], vsub(win[R + p][r], win[R - p][r]));
            }
            if (!G.orth) {
                T c[3];
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    c[q] = vadd(vadd(vscale(G.ui[3 * q], g[0]), vscale(G.ui[3 * q + 1], g[1])),
                                vscale(G.ui[3 * q + 2], g[2]));
#pragma unroll
                for (int q = 0; q < 3; ++q) g[q] = c[q];
            }
            s[0] += re_cmul(g[0], g[0]);
            s[1] += re_cmul(g[0], g[1]);
            s[2] += re_cmul(g[0], g[2]);
            s[3] += re_cmul(g[1], g[1]);
            s[4] += re_cmul(g[1], g[2]);
            s[5] += re_cmul(g[2], g[2]);
        }
#pragma unroll
        for (int k = 0; k + 1 < W; ++k)
#pragma unroll
            for (int r = 0; r < RY; ++r) win[k][r] = win[k + 1][r];
#pragma unroll
        for (int r = 0; r < RY; ++r) win[W - 1][r] = nxt[r];
        b = b == 2 ? 0 : b + 1;
    }
#pragma unroll
    for (int v = 0; v < 6; ++v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[v] += __shfl_xor_sync(0xffffffffu, s[v], o);
        if ((tid & 31) == 0) red[tid >> 5][v] = s[v];
    }
    __syncthreads();
    if (tid < 6) {
        double t = 0.0;
        for (int u = 0; u < kKinThreads / 32; ++u) t += red[u][tid];
        part[((long long)blockIdx.y * ncta + blockIdx.z * gridDim.x + blockIdx.x) * 6 + tid] = t;
    }
}

// The same sums with every neighbour read from global memory: rows longer than a CTA, or planes too
// large for shared memory.
constexpr int kPointCtas = 64;
template <typename T>
__global__ void __launch_bounds__(256)
    kinetic_point_kernel(const T* __restrict__ psi, long long ld, const GradCoef<T> G, double* __restrict__ part) {
    __shared__ double red[8][6];
    const T* x = psi + (long long)blockIdx.y * ld;
    const long long nd = (long long)G.nx * G.ny * G.nz;
    double s[6] = {0, 0, 0, 0, 0, 0};
    for (long long o = blockIdx.x * 256LL + threadIdx.x; o < nd; o += kPointCtas * 256LL) {
        const long long row = o / G.nx;
        const int i = (int)(o - row * G.nx), k = (int)(row / G.ny), j = (int)(row - (long long)k * G.ny);
        T g[3] = {fd_dir(x, o, i, G.nx, 1, G.R, G.d1[0], G.phl[0], G.phr[0]),
                  fd_dir(x, o, j, G.ny, G.nx, G.R, G.d1[1], G.phl[1], G.phr[1]),
                  fd_dir(x, o, k, G.nz, (long long)G.nx * G.ny, G.R, G.d1[2], G.phl[2], G.phr[2])};
        if (!G.orth) {
            T c[3];
#pragma unroll
            for (int q = 0; q < 3; ++q)
                c[q] = vadd(vadd(vscale(G.ui[3 * q], g[0]), vscale(G.ui[3 * q + 1], g[1])), vscale(G.ui[3 * q + 2], g[2]));
#pragma unroll
            for (int q = 0; q < 3; ++q) g[q] = c[q];
        }
        s[0] += re_cmul(g[0], g[0]);
        s[1] += re_cmul(g[0], g[1]);
        s[2] += re_cmul(g[0], g[2]);
        s[3] += re_cmul(g[1], g[1]);
        s[4] += re_cmul(g[1], g[2]);
        s[5] += re_cmul(g[2], g[2]);
    }
#pragma unroll
    for (int v = 0; v < 6; ++v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[v] += __shfl_xor_sync(0xffffffffu, s[v], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][v] = s[v];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double t = 0.0;
        for (int u = 0; u < 8; ++u) t += red[u][threadIdx.x];
        part[((long long)blockIdx.y * kPointCtas + blockIdx.x) * 6 + threadIdx.x] = t;
    }
}

// out[v] = scale * sum_n occ[n] sum over the column's CTAs of part[n][cta][v], in a fixed order.
__global__ void __launch_bounds__(256)
    kinetic_reduce_kernel(const double* __restrict__ part, const double* __restrict__ occ, int ncol, int ncta,
                          double scale, double* __restrict__ out) {
    __shared__ double red[8];
    const int v = blockIdx.x;
    double s = 0.0;
    for (int e = threadIdx.x; e < ncol * ncta; e += 256) s += occ[e / ncta] * part[(long long)e * 6 + v];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int u = 0; u < 8; ++u) t += red[u];
        out[v] = scale * t;
    }
}

template <typename T>
GradCoef<T> grad_coef(const ForceGeom& g, const T* phl, const T* phr) {
    GradCoef<T> G;
    G.nx = g.nx;
    G.ny = g.ny;
    G.nz = g.nz;
    G.R = g.R;
    G.orth = g.orth ? 1 : 0;
    for (int d = 0; d < 3; ++d) {
        for (int p = 0; p < kMaxR1; ++p) G.d1[d][p] = (p >= 1 && p <= g.R) ? g.D1[d][p] : 0.0;
        G.phl[d] = phl[d];
        G.phr[d] = phr[d];
        G.h[d] = g.h[d];
    }
    for (int i = 0; i < 9; ++i) {
        G.ui[i] = g.ui[i];
        G.uvec[i] = g.uvec[i];
    }
    return G;
}

struct KinPlan {
    int tyt, nbands, zchunk, nzch;
};
KinPlan kin_plan(const ForceGeom& g, int ncol, int ry) {
    KinPlan k;
    k.tyt = std::max(1, std::min(kKinThreads / g.nx, (g.ny + ry - 1) / ry));
    k.nbands = (g.ny + k.tyt * ry - 1) / (k.tyt * ry);
    k.tyt = ((g.ny + k.nbands - 1) / k.nbands + ry - 1) / ry;  // bands of equal height
    // two waves of CTAs: chunks of at least 6 planes
    const long long base = (long long)k.nbands * ncol;
    int nz = (int)std::max<long long>(1, std::min<long long>((2 * 148 + base - 1) / base, g.nz / 6));
    k.zchunk = (g.nz + nz - 1) / nz;
    k.nzch = (g.nz + k.zchunk - 1) / k.zchunk;
    return k;
}

int status(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s launch failed: %s", what, cudaGetErrorString(e));
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

NLView view64(const NLDev& nl) {
    NLView v{};
    v.n_atom = nl.n_atom;
    v.n_img = nl.n_img;
    v.n_pts = nl.n_pts;
    v.atom_img_ptr = nl.atom_img_ptr;
    v.atom_img_list = nl.atom_img_list;
    v.atom_nproj = nl.atom_nproj;
    v.atom_poff = nl.atom_poff;
    v.gamma = nl.gamma;
    v.img_atom = nl.img_atom;
    v.img_ndc = nl.img_ndc;
    v.img_goff = nl.img_goff;
    v.img_chi_off = nl.img_chi_off;
    v.img_phase = nl.img_phase;
    v.gpos = nl.gpos;
    v.chi = nl.chi64;
    return v;
}

}  // namespace

static int check_geom(const ForceGeom& g, int ncol) {
    if (g.R < 1 || g.R > 8) {
        set_error("gradient: bad half-width %d", g.R);
        return LYNX_ERR_BAD_ARG;
    }
    if (g.nx < g.R || g.ny < g.R || g.nz < g.R) {
        set_error("grid %dx%dx%d smaller than the FD half-width %d", g.nx, g.ny, g.nz, g.R);
        return LYNX_ERR_UNSUPPORTED;
    }
    if (ncol > 65535) {
        set_error("too many columns (%d) for one launch", ncol);
        return LYNX_ERR_UNSUPPORTED;
    }
    return LYNX_OK;
}

size_t sphere_work_bytes(int n_atom, int ncol, bool stress) {
    return sizeof(double) * (size_t)n_atom * ncol * (stress ? 7 : 4);
}

template <typename T>
int launch_sphere_terms(const NLDev& nl, const ForceGeom& g, const T* psi, long long ld, int ncol, const T* phl,
                        const T* phr, const double* img_pos, const double* occ, double scale, double escale,
                        double dV, bool stress, double* work, double* out, double* ea, cudaStream_t st) {
    if (nl.n_atom == 0 || ncol <= 0) return LYNX_OK;
    if (nl.max_np > 32) {
        set_error("%d projectors per atom exceed the kernel's limit of 32", nl.max_np);
        return LYNX_ERR_UNSUPPORTED;
    }
    LYNX_TRY(check_geom(g, ncol));
    const GradCoef<T> G = grad_coef<T>(g, phl, phr);
    const NLView v = view64(nl);
    dim3 grid(nl.n_atom, ncol);
    auto go = [&](auto mj) {
        constexpr int MJ = decltype(mj)::value;
        if (stress) sphere_kernel<T, true, MJ><<<grid, 256, 0, st>>>(psi, ld, ncol, v, G, img_pos, occ, dV, work);
        else sphere_kernel<T, false, MJ><<<grid, 256, 0, st>>>(psi, ld, ncol, v, G, img_pos, occ, dV, work);
    };
    if (nl.max_np <= 8) go(std::integral_constant<int, 1>{});
    else if (nl.max_np <= 16) go(std::integral_constant<int, 2>{});
    else if (nl.max_np <= 24) go(std::integral_constant<int, 3>{});
    else go(std::integral_constant<int, 4>{});
    const int nv = stress ? 6 : 3;
    sphere_reduce_kernel<<<dim3(nl.n_atom, nv + 1), 256, 0, st>>>(work, ncol, nv, scale, escale, out, ea);
    count_launch(2);
    return status("nonlocal force / stress");
}

size_t kinetic_work_bytes(const ForceGeom& g, int ncol, bool cplx) {
    const KinPlan k = kin_plan(g, ncol, cplx ? kin_ry<double2>() : kin_ry<double>());
    return sizeof(double) * 6 * (size_t)std::max(k.nbands * k.nzch, kPointCtas) * ncol;
}

template <typename T>
int launch_kinetic(const ForceGeom& g, const T* psi, long long ld, int ncol, const T* phl, const T* phr, bool phased,
                   const double* occ, double scale, double* work, double* out, cudaStream_t st) {
    LYNX_TRY(check_geom(g, ncol));
    const GradCoef<T> G = grad_coef<T>(g, phl, phr);
    constexpr int ry = kin_ry<T>();
    const KinPlan k = kin_plan(g, ncol, ry);
    const size_t smem = sizeof(T) * 3 * (size_t)(k.tyt * ry + 2 * g.R) * g.nx;
    if (g.nx > kKinThreads || smem > 200 * 1024) {
        kinetic_point_kernel<T><<<dim3(kPointCtas, ncol), 256, 0, st>>>(psi, ld, G, work);
        kinetic_reduce_kernel<<<6, 256, 0, st>>>(work, occ, ncol, kPointCtas, scale, out);
        count_launch(2);
        return status("kinetic stress");
    }
    dim3 grid(k.nbands, ncol, k.nzch);
    const int ncta = k.nbands * k.nzch;
    auto go = [&](auto rc) -> int {
        constexpr int R = decltype(rc)::value;
        auto kern = phased ? kinetic_kernel<T, R, true> : kinetic_kernel<T, R, false>;
        LYNX_CUDA_TRY(smem_cap(kern, smem));
        kern<<<grid, kKinThreads, smem, st>>>(psi, ld, G, k.tyt, k.zchunk, ncta, work);
        return LYNX_OK;
    };
    switch (g.R) {
        case 1: LYNX_TRY(go(std::integral_constant<int, 1>{})); break;
        case 2: LYNX_TRY(go(std::integral_constant<int, 2>{})); break;
        case 3: LYNX_TRY(go(std::integral_constant<int, 3>{})); break;
        case 4: LYNX_TRY(go(std::integral_constant<int, 4>{})); break;
        case 5: LYNX_TRY(go(std::integral_constant<int, 5>{})); break;
        case 6: LYNX_TRY(go(std::integral_constant<int, 6>{})); break;
        case 7: LYNX_TRY(go(std::integral_constant<int, 7>{})); break;
        case 8: LYNX_TRY(go(std::integral_constant<int, 8>{})); break;
    }
    kinetic_reduce_kernel<<<6, 256, 0, st>>>(work, occ, ncol, ncta, scale, out);
    count_launch(2);
    return status("kinetic stress");
}

#define LYNX_FORCE_INST(T)                                                                                           \
    template int launch_sphere_terms<T>(const NLDev&, const ForceGeom&, const T*, long long, int, const T*, const T*, \
                                        const double*, const double*, double, double, double, bool, double*,         \
                                        double*, double*, cudaStream_t);                                             \
    template int launch_kinetic<T>(const ForceGeom&, const T*, long long, int, const T*, const T*, bool,             \
                                   const double*, double, double*, double*, cudaStream_t);
LYNX_FORCE_INST(double)
LYNX_FORCE_INST(double2)

}  // namespace lynxb
