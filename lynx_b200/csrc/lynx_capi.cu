// C ABI of lynx_b200: context set-up, operator entry points and the CheFSI driver.
//
// The driver mirrors EigenSolver::solve_impl (src/solvers/EigenSolver.cpp:739-818):
//   filter (degree m)  ->  Cholesky-QR  ->  project  ->  subspace eigensolve  ->  rotate,
// with two B200-specific changes that keep the arithmetic identical:
//   * the three filter buffers rotate by pointer (the reference GPU path copies
//     two full blocks per degree step, src/solvers/EigenSolver.cu:190-191);
//   * the Cholesky factor R of the overlap is folded into the subspace matrix and
//     the rotation, Hs' = R^-T Hs R^-1 and psi = Y (R^-1 Q), which equals the
//     reference's Y <- Y R^-1; Hs = dV Y^T H Y; psi = Y Q, but needs no pass of
//     trsm over the Nd x N block and lets H*Y run on the unorthogonalised Y.
#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>
#include <cufft.h>
#include <curand.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <map>
#include <mutex>
#include <type_traits>
#include <string>
#include <thread>
#include <vector>

#include "kernels.h"
#include "lynx_common.cuh"
#include "stencil.cuh"
#include "stencil_pipe.cuh"

namespace lynxb {

static thread_local std::string g_last_error;
static std::atomic<long long> g_launches{0};

void set_error(const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_last_error = buf;
}

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

cudaError_t raise_smem_cap(const void* func, size_t bytes) {
    // The default cap of 48 KB counts a kernel's static shared memory too (below 16 KB wherever both are used).
    if (bytes <= 32 * 1024) return cudaSuccess;
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> caps;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cap = caps[{dev, func}];
    if (bytes <= cap) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cap = bytes;
    return e;
}

// Growable device buffer.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    int tag = 0;  // layout the contents were written in (0 = none)
    int ensure(size_t b) {
        if (b <= bytes) return LYNX_OK;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, b);
        if (e != cudaSuccess) {
            cudaGetLastError();
            set_error("cudaMalloc(%zu) failed: %s", b, cudaGetErrorString(e));
            return LYNX_ERR_OOM;
        }
        bytes = b;
        return LYNX_OK;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <typename T> T* as() const { return static_cast<T*>(p); }
};

// ---------------------------------------------------------------------------
// Elementwise helper kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cvt_val(double& d, float s) { d = (double)s; }
__device__ __forceinline__ void cvt_val(float& d, double s) { d = (float)s; }
__device__ __forceinline__ void cvt_val(double& d, double s) { d = s; }
__device__ __forceinline__ void cvt_val(float& d, float s) { d = s; }
__device__ __forceinline__ void cvt_val(double2& d, float2 s) { d = make_double2(s.x, s.y); }
__device__ __forceinline__ void cvt_val(float2& d, double2 s) { d = make_float2((float)s.x, (float)s.y); }
__device__ __forceinline__ void cvt_val(double2& d, double2 s) { d = s; }

template <typename Dst, typename Src>
__global__ void convert_cols_kernel(Dst* __restrict__ dst, long long ldd, const Src* __restrict__ src,
                                    long long lds, long long nrow, int ncol) {
    const long long total = nrow * ncol;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long c = i / nrow, r = i - c * nrow;
        cvt_val(dst[c * ldd + r], src[c * lds + r]);
    }
}

template <typename Dst, typename Src>
int convert_cols(Dst* dst, long long ldd, const Src* src, long long lds, long long nrow, int ncol,
                 cudaStream_t st) {
    const long long total = nrow * ncol;
    if (total == 0) return LYNX_OK;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148LL * 16);
    convert_cols_kernel<Dst, Src><<<blocks, 256, 0, st>>>(dst, ldd, src, lds, nrow, ncol);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return LYNX_OK;
}

// Symmetrise (real) / Hermitise (complex) an N x N column-major matrix in place.
__global__ void symmetrize_kernel(double* A, int N) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i < j && j < N) {
        const double v = 0.5 * (A[i + (long long)j * N] + A[j + (long long)i * N]);
        A[i + (long long)j * N] = v;
        A[j + (long long)i * N] = v;
    }
}
__global__ void hermitize_kernel(double2* A, int N) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i < N && j < N) {
        if (i < j) {
            const double2 a = A[i + (long long)j * N], b = A[j + (long long)i * N];
            const double2 v = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
            A[i + (long long)j * N] = v;
            A[j + (long long)i * N] = make_double2(v.x, -v.y);
        } else if (i == j) {
            A[i + (long long)i * N].y = 0.0;
        }
    }
}

// Complex blocks on the real tensor-core kernels (mixed precision, k-point).  A complex block
// Y = Yr + i Yi (columns of ld complex elements) is split into the planar real block
// [Yr | Yi] (2N columns of ld floats); then
//   [Yr | Yi]^T [Yr | Yi] = [[Yr^T Yr, Yr^T Yi], [Yi^T Yr, Yi^T Yi]]  gives  Y^H Y, and
//   [Yr | Yi] [[Wr, Wi], [-Wi, Wr]] = [Re(Y W) | Im(Y W)].
__global__ void planar_kernel(const float2* __restrict__ Y, long long ld, int N, float* __restrict__ P) {
    const long long total = ld * N;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long j = t / ld, p = t - j * ld;
        const float2 v = Y[t];
        P[j * ld + p] = v.x;
        P[(j + N) * ld + p] = v.y;
    }
}

// Complex N x N products from the real 2N x 2N ones (column-major): M (Hermitian, upper triangle
// from the upper triangle of Mp) and H (all entries from the full Hp):
//   X(a, b) = Xp(a, b) + Xp(N+a, N+b) + i (Xp(a, N+b) - Xp(N+a, b)).
__global__ void combine_gram_kernel(const double* __restrict__ Mp, const double* __restrict__ Hp, int N,
                                    double2* __restrict__ M, double2* __restrict__ H) {
    const int a = blockIdx.y * blockDim.y + threadIdx.y;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= N || b >= N) return;
    const long long n2 = 2LL * N;
    auto at = [n2](const double* X, long long r, long long c) { return X[r + c * n2]; };
    H[a + (long long)b * N] =
        make_double2(at(Hp, a, b) + at(Hp, N + a, N + b), at(Hp, a, N + b) - at(Hp, N + a, b));
    if (a <= b) {
        // Mp holds its upper triangle only: Mp(N+a, b) = Mp(b, N+a)
        M[a + (long long)b * N] =
            make_double2(at(Mp, a, b) + at(Mp, N + a, N + b), at(Mp, a, N + b) - at(Mp, b, N + a));
    }
}

// Wt = [[Wr, Wi], [-Wi, Wr]] (2N x 2N, column-major) from the complex N x N W.
__global__ void wtilde_kernel(const double2* __restrict__ W, int N, double* __restrict__ Wt) {
    const int n = blockIdx.y * blockDim.y + threadIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N || j >= N) return;
    const long long n2 = 2LL * N;
    const double2 w = W[n + (long long)j * N];
    Wt[n + j * n2] = w.x;
    Wt[n + (j + N) * n2] = w.y;
    Wt[(n + N) + j * n2] = -w.y;
    Wt[(n + N) + (j + N) * n2] = w.x;
}

// psi[j][p] = (R[j][p], R[N + j][p]) for the Nd points of N columns (R: FP64, column stride Nd).
__global__ void interleave_kernel(const double* __restrict__ R, long long Nd, int N, double2* __restrict__ psi,
                                  long long ldp) {
    const long long total = Nd * N;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long j = t / Nd, p = t - j * Nd;
        psi[j * ldp + p] = make_double2(R[j * Nd + p], R[(j + N) * Nd + p]);
    }
}

// Electron density of one (spin, k-point) block: rho[i] (+)= sum_n w[n] |psi_n(i)|^2, the states in
// order (src/electronic/ElectronDensity.cpp:85-121, with w[n] = spin factor * k weight * f_n and
// w[n] = 0 where the reference skips f_n < 1e-16).  One thread per grid point: the reads of every
// column are coalesced, and the sum has a fixed order.
__device__ __forceinline__ double abs2(double v) { return v * v; }
__device__ __forceinline__ double abs2(double2 v) { return v.x * v.x + v.y * v.y; }
template <typename T>
__global__ void density_kernel(const T* __restrict__ psi, long long ld, long long nd, int ncol,
                               const double* __restrict__ w, double* __restrict__ rho, int accumulate) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nd;
         i += (long long)gridDim.x * blockDim.x) {
        double s = accumulate ? rho[i] : 0.0;
        for (int n = 0; n < ncol; ++n) {
            const double wn = w[n];
            if (wn != 0.0) s = fma(wn, abs2(psi[(long long)n * ld + i]), s);
        }
        rho[i] = s;
    }
}

template <typename T>
int launch_density(const T* psi, long long ld, long long nd, int ncol, const double* w, double* rho, bool accumulate,
                   cudaStream_t st) {
    if (nd <= 0) return LYNX_OK;
    const int blocks = (int)std::min<long long>((nd + 255) / 256, 148LL * 16);
    density_kernel<T><<<blocks, 256, 0, st>>>(psi, ld, nd, ncol, w, rho, accumulate ? 1 : 0);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return LYNX_OK;
}
template int launch_density<double>(const double*, long long, long long, int, const double*, double*, bool,
                                    cudaStream_t);
template int launch_density<double2>(const double2*, long long, long long, int, const double*, double*, bool,
                                     cudaStream_t);

// out[i] = sum_n u_n(i) v_n(i), the columns in order: one read of both blocks (the gradient of <g, H psi>
// in the potential; as a product block and a sum of it, 161 us at Si64 with 160 states, 94 us here).
// V: points per thread, loaded as one vector.
template <int V>
__global__ void __launch_bounds__(128)
    pair_density_kernel(const double* __restrict__ u, const double* __restrict__ v, long long ld, long long nd,
                        int ncol, double* __restrict__ out) {
    using T = typename std::conditional<V == 2, double2, double>::type;
    const long long i = (blockIdx.x * 128LL + threadIdx.x) * V;
    if (i >= nd) return;
    double s[V] = {};
#pragma unroll 8
    for (int n = 0; n < ncol; ++n) {
        const T a = __ldcs(reinterpret_cast<const T*>(u + n * ld + i)), b = __ldcs(reinterpret_cast<const T*>(v + n * ld + i));
        const double* ap = reinterpret_cast<const double*>(&a);
        const double* bp = reinterpret_cast<const double*>(&b);
#pragma unroll
        for (int q = 0; q < V; ++q) s[q] = fma(ap[q], bp[q], s[q]);
    }
#pragma unroll
    for (int q = 0; q < V; ++q) out[i + q] = s[q];
}

// Sets *flag when an entry of the N x N column-major matrix A is NaN or Inf (comps doubles per
// entry: 1 real, 2 complex; upper: only entries on or above the diagonal are valid).
__global__ void nonfinite_kernel(const double* __restrict__ A, int N, int comps, int upper, int* __restrict__ flag) {
    const long long n2 = (long long)N * N;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n2; t += (long long)gridDim.x * blockDim.x) {
        const long long j = t / N, i = t - j * N;
        if (upper && i > j) continue;
        for (int q = 0; q < comps; ++q)
            if (!isfinite(A[t * comps + q])) *flag = 1;
    }
}

// One CTA waits, with at most `spins` tries, for a phase of an mbarrier that nothing completes:
// the bounded wait of the pipelined kernels, made to run out.  It gives up, flags the error and
// returns, which leaves the context usable.
__global__ void wait_selftest_kernel(int spins, int* __restrict__ err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, spins)) atomicExch(err, 1);
}

}  // namespace lynxb

using namespace lynxb;

// ---------------------------------------------------------------------------
// Context
// ---------------------------------------------------------------------------
struct lynx_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    int nx = 0, ny = 0, nz = 0, Nd = 0, fd_order = 0, R = 0;
    bool orth = true;
    int bc[3] = {0, 0, 0};
    double latvec[9] = {0}, uvec[9] = {0}, lapcT[9] = {0}, L[3] = {0, 0, 0};
    double jac = 0, dx = 0, dy = 0, dz = 0, dV = 0, maxeig = 0;
    std::vector<double> w1, w2, D2x, D2y, D2z, D1x, D1y, D1z, D2xy, D2xz, D2yz;
    double kpt[3] = {0, 0, 0};
    // nonlocal
    bool has_nl = false;
    NLDev nl;
    std::vector<DevBuf> nl_bufs;
    std::vector<double> img_shift;  // host copy for phase updates
    // handles
    cublasHandle_t cublas = nullptr;
    cusolverDnHandle_t cusolver = nullptr;
    // work buffers
    DevBuf wbuf[4];       // filter / RR blocks (any precision)
    DevBuf cvt[2];        // FP64 copies of FP32 blocks for the Rayleigh-Ritz products
    DevBuf alpha;         // nonlocal projections
    DevBuf v32;           // FP32 copy of Veff
    DevBuf Ms, Hs, eigd, solver_work, info;
    DevBuf lz[4];         // Lanczos vectors
    DevBuf io_psi, io_v;  // staging for the host-pointer solve
    DevBuf vpad64, vpad32;  // Veff in the padded row layouts of the pipelined stencil
    // Set by a kernel whose bounded wait gave up: an int in mapped host memory, so that looking at it after
    // a synchronisation is a host read (a copy of 4 bytes to pageable memory cost as much as a small call's
    // kernel).  Pinned host memory for the results of a pass likewise.
    int* err_h = nullptr;
    int* err_d = nullptr;
    double* res_h = nullptr;
    size_t res_n = 0;
    // Marks the work on `alpha` that a call left in flight (leave_in_flight): lynx_set_stream makes
    // another stream wait for it.
    cudaEvent_t in_flight = nullptr;
    bool pending = false;
    DevBuf gwork;           // slices, exponents and split partials of the tensor-core Gram
    DevBuf rwork;           // slices and exponents of the tensor-core rotation
    DevBuf cplx_work;       // planar split and real 2N x 2N products of the mixed k-point Rayleigh-Ritz
    bool no_tc_gram = false;  // diagnostic switch: FP64 library products for the mixed path
    bool autotune = true;     // time the compiled stencil launch shapes on first use per grid
    int force_shape = -1;     // diagnostic: compiled stencil launch shape used for every launch
    int host_block = 128;     // columns per block of the pipelined host-to-device copy
    std::map<std::array<long long, 8>, int> pipe_shape;  // chosen launch shape per (type, grid, columns, fused, xold)
    bool fuse_nl = true;      // add the nonlocal term inside the stencil when the spheres are disjoint
    // with fuse_nl: the stencil also writes compact sphere-point copies of its output and the
    // next step gathers from them (measured slower than the direct gather on B200: off)
    bool fuse_compact_gather = false;
    struct NLMap {
        DevBuf ptmap, rowstart;
        std::vector<int> rowstart_h;
        int mp = 0;
    };
    std::map<int, NLMap> nl_maps;  // per padded row length: compact point map of the sphere points
    DevBuf nlW;                    // compact (chi alpha) values, columns of ldw
    DevBuf xsbuf[2];               // compact sphere-point copies of consecutive filter blocks
    DevBuf gradbuf[2];             // first derivatives along y and z (non-orthogonal cells)
    DevBuf fpart, fwork;           // forces, stress: partial sums; occupations, positions, results
    // Host-input pipelining: a copy stream, and for the duration of one host-pointer solve the
    // first column of every column block with the event that marks its arrival on the device.
    cudaStream_t copy_stream = nullptr;
    std::vector<std::pair<int, cudaEvent_t>> col_blocks;
    int col_total = 0;  // columns of all blocks together
    // nonlocal tables re-indexed for padded row layouts: nxp -> tables
    std::map<int, NLDev> nl_layouts;
    std::vector<DevBuf> nl_layout_bufs;
    std::vector<int> h_gpos, h_pt_grid;  // host copies of the unpadded grid indices
    // lynx_eigensolver_solve_density: the density request of the current pass
    struct DensityReq {
        bool on = false, done = false;
        double nelectron = 0, beta = 0, weight = 0, ef = 0;
        int smearing = 0;
        double* rho = nullptr;
    } dens;
    DevBuf dens_w, dens_part;
    // effective potential: AAR / XC work fields, a zero potential and a ones field, dot-product scratch
    DevBuf vwork, vzero, vones, dotw, xcwork;
    // periodic Poisson by FFT: plans and the inverse symbol of -Lap (made on first use)
    bool poisson_direct = true;
    bool fft_ready = false;
    cufftHandle fft_fwd = 0, fft_inv = 0;
    DevBuf fft_sym, fft_z;
    // lynx_time_filter_step with with_nonlocal = 2: events around the stencil kernel alone
    bool time_stencil = false;
    cudaEvent_t kt[2] = {nullptr, nullptr};
    double kt_ms = 0.0;
    int kt_n = 0;
};

namespace {

// Makes the context's device current and creates the cuBLAS / cuSOLVER handles on first
// use, so that lynx_create itself needs no GPU (set-up queries work on a CPU-only host).
int activate(lynx_ctx* c) {
    LYNX_CUDA_TRY(cudaSetDevice(c->device));
    if (!c->cublas) {
        if (cublasCreate(&c->cublas) != CUBLAS_STATUS_SUCCESS) {
            c->cublas = nullptr;
            set_error("cuBLAS initialisation failed");
            return LYNX_ERR_CUDA;
        }
    }
    if (!c->cusolver) {
        if (cusolverDnCreate(&c->cusolver) != CUSOLVER_STATUS_SUCCESS) {
            c->cusolver = nullptr;
            set_error("cuSOLVER initialisation failed");
            return LYNX_ERR_CUDA;
        }
    }
    return LYNX_OK;
}

double fract(int n, int k) {
    // n! / ((n-k)! (n+k)!)
    double num = 1.0, den = 1.0;
    for (int i = n - k + 1; i <= n; ++i) num *= i;
    for (int i = n + 1; i <= n + k; ++i) den *= i;
    return num / den;
}

void mat3_inverse(const double* a, double* inv) {
    const double det = a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
                       a[2] * (a[3] * a[7] - a[4] * a[6]);
    inv[0] = (a[4] * a[8] - a[5] * a[7]) / det;
    inv[1] = (a[2] * a[7] - a[1] * a[8]) / det;
    inv[2] = (a[1] * a[5] - a[2] * a[4]) / det;
    inv[3] = (a[5] * a[6] - a[3] * a[8]) / det;
    inv[4] = (a[0] * a[8] - a[2] * a[6]) / det;
    inv[5] = (a[2] * a[3] - a[0] * a[5]) / det;
    inv[6] = (a[3] * a[7] - a[4] * a[6]) / det;
    inv[7] = (a[1] * a[6] - a[0] * a[7]) / det;
    inv[8] = (a[0] * a[4] - a[1] * a[3]) / det;
}

// Central-difference weights of order 2*FDn (Fornberg), scaled to the grid and,
// for non-orthogonal cells, to the Laplacian metric lapc_T = (U^-1)^T U^-1 of the
// unit lattice vectors U (the conventions of src/operators/FDStencil.cpp:73-152
// and src/core/Lattice.cpp:13-51).
void build_stencil(lynx_ctx* c) {
    const int n = c->R + 1;
    c->w1.assign(n, 0.0);
    c->w2.assign(n, 0.0);
    for (int p = 1; p < n; ++p) {
        const double sgn = (p % 2 == 1) ? 1.0 : -1.0;
        c->w1[p] = sgn * fract(c->R, p) / p;
        c->w2[0] -= 2.0 / ((double)p * p);
        c->w2[p] = sgn * 2.0 * fract(c->R, p) / ((double)p * p);
    }
    // lattice
    for (int i = 0; i < 3; ++i) {
        double len = 0;
        for (int j = 0; j < 3; ++j) len += c->latvec[3 * i + j] * c->latvec[3 * i + j];
        len = std::sqrt(len);
        c->L[i] = len;
        for (int j = 0; j < 3; ++j) c->uvec[3 * i + j] = c->latvec[3 * i + j] / len;
    }
    const double* a = c->latvec;
    c->jac = std::fabs(a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
                       a[2] * (a[3] * a[7] - a[4] * a[6]));
    double uinv[9];
    mat3_inverse(c->uvec, uinv);
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            double s = 0;
            for (int k = 0; k < 3; ++k) s += uinv[3 * k + i] * uinv[3 * k + j];
            c->lapcT[3 * i + j] = s;
        }
    const int ni[3] = {c->bc[0] == LYNX_BC_PERIODIC ? c->nx : c->nx - 1,
                       c->bc[1] == LYNX_BC_PERIODIC ? c->ny : c->ny - 1,
                       c->bc[2] == LYNX_BC_PERIODIC ? c->nz : c->nz - 1};
    c->dx = c->L[0] / ni[0];
    c->dy = c->L[1] / ni[1];
    c->dz = c->L[2] / ni[2];
    c->dV = c->jac / ((double)ni[0] * ni[1] * ni[2]);
    const double ix = 1.0 / c->dx, iy = 1.0 / c->dy, iz = 1.0 / c->dz;
    c->D1x.resize(n);
    c->D1y.resize(n);
    c->D1z.resize(n);
    c->D2x.resize(n);
    c->D2y.resize(n);
    c->D2z.resize(n);
    c->D2xy.assign(n, 0.0);
    c->D2xz.assign(n, 0.0);
    c->D2yz.assign(n, 0.0);
    const double gx = c->orth ? 1.0 : c->lapcT[0], gy = c->orth ? 1.0 : c->lapcT[4],
                 gz = c->orth ? 1.0 : c->lapcT[8];
    for (int p = 0; p < n; ++p) {
        c->D1x[p] = c->w1[p] * ix;
        c->D1y[p] = c->w1[p] * iy;
        c->D1z[p] = c->w1[p] * iz;
        c->D2x[p] = gx * c->w2[p] * ix * ix;
        c->D2y[p] = gy * c->w2[p] * iy * iy;
        c->D2z[p] = gz * c->w2[p] * iz * iz;
        if (!c->orth) {
            c->D2xy[p] = 2.0 * c->lapcT[1] * c->w1[p] * ix;
            c->D2xz[p] = 2.0 * c->lapcT[2] * c->w1[p] * ix;
            c->D2yz[p] = 2.0 * c->lapcT[5] * c->w1[p] * iy;
        }
    }
    if (c->orth) {
        const double PI = 3.14159265358979323846;
        const double sx = (c->nx - c->nx % 2) / (double)c->nx, sy = (c->ny - c->ny % 2) / (double)c->ny,
                     sz = (c->nz - c->nz % 2) / (double)c->nz;
        double m = c->D2x[0] + c->D2y[0] + c->D2z[0];
        for (int p = 1; p <= c->R; ++p)
            m += 2.0 * (c->D2x[p] * std::cos(PI * p * sx) + c->D2y[p] * std::cos(PI * p * sy) +
                        c->D2z[p] * std::cos(PI * p * sz));
        c->maxeig = -0.5 * m;
    } else {
        double m = std::fabs(c->D2x[0]) + std::fabs(c->D2y[0]) + std::fabs(c->D2z[0]);
        for (int p = 1; p <= c->R; ++p) {
            m += 2.0 * (std::fabs(c->D2x[p]) + std::fabs(c->D2y[p]) + std::fabs(c->D2z[p]));
            m += 2.0 * (std::fabs(c->D2xy[p]) + std::fabs(c->D2xz[p]) + std::fabs(c->D2yz[p]));
        }
        c->maxeig = 0.5 * m;
    }
}

StencilGeom geom(const lynx_ctx* c) {
    StencilGeom g;
    g.nx = c->nx;
    g.ny = c->ny;
    g.nz = c->nz;
    g.R = c->R;
    g.D2x = c->D2x.data();
    g.D2y = c->D2y.data();
    g.D2z = c->D2z.data();
    return g;
}

// Ghost multipliers: 1 for periodic, 0 for Dirichlet; Bloch phases for complex data.
template <typename T> void ghost_phases(const lynx_ctx* c, bool use_k, T* phl, T* phr);
template <> void ghost_phases<double>(const lynx_ctx* c, bool, double* phl, double* phr) {
    for (int d = 0; d < 3; ++d) phl[d] = phr[d] = (c->bc[d] == LYNX_BC_PERIODIC) ? 1.0 : 0.0;
}
template <> void ghost_phases<float>(const lynx_ctx* c, bool, float* phl, float* phr) {
    for (int d = 0; d < 3; ++d) phl[d] = phr[d] = (c->bc[d] == LYNX_BC_PERIODIC) ? 1.0f : 0.0f;
}
template <> void ghost_phases<double2>(const lynx_ctx* c, bool use_k, double2* phl, double2* phr) {
    for (int d = 0; d < 3; ++d) {
        if (c->bc[d] != LYNX_BC_PERIODIC) {
            phl[d] = phr[d] = make_double2(0, 0);
            continue;
        }
        const double th = use_k ? c->kpt[d] * c->L[d] : 0.0;
        phl[d] = make_double2(std::cos(th), -std::sin(th));
        phr[d] = make_double2(std::cos(th), std::sin(th));
    }
}
template <> void ghost_phases<float2>(const lynx_ctx* c, bool use_k, float2* phl, float2* phr) {
    double2 l[3], r[3];
    ghost_phases<double2>(c, use_k, l, r);
    for (int d = 0; d < 3; ++d) {
        phl[d] = make_float2((float)l[d].x, (float)l[d].y);
        phr[d] = make_float2((float)r[d].x, (float)r[d].y);
    }
}

int update_nl_phases(lynx_ctx* c) {
    if (!c->has_nl || c->nl.n_img == 0) return LYNX_OK;
    std::vector<double> ph(2 * c->nl.n_img);
    for (int i = 0; i < c->nl.n_img; ++i) {
        const double th = -(c->kpt[0] * c->img_shift[3 * i] + c->kpt[1] * c->img_shift[3 * i + 1] +
                            c->kpt[2] * c->img_shift[3 * i + 2]);
        ph[2 * i] = std::cos(th);
        ph[2 * i + 1] = std::sin(th);
    }
    LYNX_CUDA_TRY(cudaMemcpyAsync(c->nl.img_phase, ph.data(), ph.size() * sizeof(double), cudaMemcpyHostToDevice,
                                  c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return LYNX_OK;
}

template <typename T> struct Real;
template <> struct Real<double> { using type = double; };
template <> struct Real<float> { using type = float; };
template <> struct Real<double2> { using type = double; };
template <> struct Real<float2> { using type = float; };

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Grids whose blocks are kept in padded rows for the pipelined stencil: it pairs adjacent x points, and
// takes an odd nx in periodic cells at FD order 12 (rows longer than kOddMaxNx may not fit its stages).
// Other grids keep unpadded rows.  Complex blocks run the direct kernel, which takes any rows.
constexpr int kOddMaxNx = 255;
template <typename T> bool pipe_capable(const lynx_ctx* c) {
    if (ScalarOf<T>::cplx || c->nx % 2 == 0) return true;
    return c->R == 6 && c->nx <= kOddMaxNx && c->bc[0] == LYNX_BC_PERIODIC && c->bc[1] == LYNX_BC_PERIODIC &&
           c->bc[2] == LYNX_BC_PERIODIC;
}

// Grows a work buffer; new storage is zeroed so that the padding elements of padded
// row layouts read as zero.
int ensure_zeroed(lynx_ctx* c, DevBuf& b, size_t bytes) {
    if (bytes <= b.bytes) return LYNX_OK;
    LYNX_TRY(b.ensure(bytes));
    LYNX_CUDA_TRY(cudaMemsetAsync(b.p, 0, b.bytes, c->stream));
    return LYNX_OK;
}

// Work buffer in a given row layout (tag): grown and/or re-zeroed when the layout changes,
// so padding elements never hold bytes of another layout.
int ensure_layout(lynx_ctx* c, DevBuf& b, size_t bytes, int tag) {
    if (bytes > b.bytes) {
        LYNX_TRY(b.ensure(bytes));
        b.tag = -1;
    }
    if (b.tag != tag) {
        LYNX_CUDA_TRY(cudaMemsetAsync(b.p, 0, b.bytes, c->stream));
        b.tag = tag;
    }
    return LYNX_OK;
}

// Copy/convert the valid points of ncol columns between row layouts (row length nxp, column stride ld).
template <typename Dst, typename Src>
__global__ void __launch_bounds__(256) repack_kernel(Dst* __restrict__ dst, int dnxp, long long dld,
                                                     const Src* __restrict__ src, int snxp, long long sld, int nx,
                                                     long long nrows) {
    // one warp per grid row (lanes along x), eight rows per CTA and grid-stride over the rows
    // (a few hundred CTAs per column rather than one per eight rows), blockIdx.y = column
    for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < nrows; r += (long long)gridDim.x * 8) {
        const Src* s = src + (long long)blockIdx.y * sld + r * snxp;
        Dst* d = dst + (long long)blockIdx.y * dld + r * dnxp;
        for (int xi = threadIdx.x & 31; xi < nx; xi += 32) cvt_val(d[xi], s[xi]);
    }
}

template <typename Dst, typename Src>
int repack(lynx_ctx* c, Dst* dst, int dnxp, long long dld, const Src* src, int snxp, long long sld, int ncol) {
    const long long nrows = (long long)c->ny * c->nz;
    if (nrows == 0 || ncol <= 0) return LYNX_OK;
    for (int c0 = 0; c0 < ncol; c0 += 65535) {  // grid.y limit
        const int nc = std::min(65535, ncol - c0);
        dim3 grid((unsigned)std::min<long long>((nrows + 7) / 8, 128), (unsigned)nc);
        repack_kernel<Dst, Src><<<grid, 256, 0, c->stream>>>(dst + (long long)c0 * dld, dnxp, dld,
                                                             src + (long long)c0 * sld, snxp, sld, c->nx, nrows);
        count_launch();
    }
    LYNX_CUDA_TRY(cudaGetLastError());
    return LYNX_OK;
}

// Uploads a host table into a buffer of its own, on the context's stream: a plain cudaMemcpy from
// pageable memory may return while its copy is still under way on the legacy stream, which kernels on a
// non-blocking stream do not wait for.  (The source may go: pageable memory is staged before the call
// returns.)
int upload_table(lynx_ctx* c, DevBuf& b, const void* src, size_t bytes) {
    LYNX_TRY(b.ensure(std::max<size_t>(bytes, 16)));
    if (!bytes) return LYNX_OK;
    LYNX_CUDA_TRY(cudaMemcpyAsync(b.p, src, bytes, cudaMemcpyHostToDevice, c->stream));
    return LYNX_OK;
}

// Nonlocal tables whose grid indices address rows of length nxp.
int nl_for(lynx_ctx* c, int nxp, const NLDev** out) {
    if (nxp == c->nx) {
        *out = &c->nl;
        return LYNX_OK;
    }
    auto it = c->nl_layouts.find(nxp);
    if (it != c->nl_layouts.end()) {
        *out = &it->second;
        return LYNX_OK;
    }
    auto remap = [&](const std::vector<int>& g) {
        std::vector<int> r(g.size());
        for (size_t i = 0; i < g.size(); ++i) {
            const int xi = g[i] % c->nx;
            const int rest = g[i] / c->nx;
            r[i] = xi + nxp * rest;
        }
        return r;
    };
    NLDev d = c->nl;
    const std::vector<int> gp = remap(c->h_gpos), pg = remap(c->h_pt_grid);
    c->nl_layout_bufs.emplace_back();
    DevBuf& b1 = c->nl_layout_bufs.back();
    LYNX_TRY(upload_table(c, b1, gp.data(), gp.size() * 4));
    d.gpos = b1.as<int>();
    c->nl_layout_bufs.emplace_back();
    DevBuf& b2 = c->nl_layout_bufs.back();
    LYNX_TRY(upload_table(c, b2, pg.data(), pg.size() * 4));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));  // the context may change streams
    d.pt_grid = b2.as<int>();
    c->nl_layouts[nxp] = d;
    *out = &c->nl_layouts[nxp];
    return LYNX_OK;
}

// Compact point map of the sphere points for rows of length nxp (row pitch mp = nxp rounded up
// to 4): ptmap[(z * ny + y) * mp + x] = compact number of grid point (x, y, z) or -1, and
// rowstart[z * ny + y] = compact number of the first sphere point at or after that row.
int nl_map_for(lynx_ctx* c, int nxp, const lynx_ctx::NLMap** out) {
    auto it = c->nl_maps.find(nxp);
    if (it != c->nl_maps.end()) {
        *out = &it->second;
        return LYNX_OK;
    }
    lynx_ctx::NLMap& m = c->nl_maps[nxp];
    m.mp = (nxp + 3) & ~3;
    const long long rows = (long long)c->ny * c->nz;
    std::vector<int> pm((size_t)rows * m.mp, -1);
    m.rowstart_h.assign(rows + 1, 0);
    const std::vector<int>& pg = c->h_pt_grid;  // grid order, rows of nx
    for (size_t p = 0; p < pg.size(); ++p) {
        const int x = pg[p] % c->nx;
        const long long row = pg[p] / c->nx;
        pm[(size_t)row * m.mp + x] = (int)p;
        m.rowstart_h[row + 1]++;
    }
    for (long long r = 0; r < rows; ++r) m.rowstart_h[r + 1] += m.rowstart_h[r];
    LYNX_TRY(upload_table(c, m.ptmap, pm.data(), pm.size() * sizeof(int)));
    LYNX_TRY(upload_table(c, m.rowstart, m.rowstart_h.data(), m.rowstart_h.size() * sizeof(int)));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    *out = &m;
    return LYNX_OK;
}

// Veff (FP64, Nd, device) in scalar type S with rows of length nxp.
template <typename S>
int veff_layout(lynx_ctx* c, const double* v, int nxp, const S** out) {
    if (std::is_same<S, double>::value && nxp == c->nx && aligned16(v)) {
        *out = reinterpret_cast<const S*>(v);
        return LYNX_OK;
    }
    DevBuf& b = std::is_same<S, double>::value ? c->vpad64 : c->vpad32;
    LYNX_TRY(ensure_zeroed(c, b, sizeof(S) * (size_t)nxp * c->ny * c->nz));
    LYNX_TRY(repack<S, double>(c, b.as<S>(), nxp, 0, v, c->nx, 0, 1));
    *out = b.as<S>();
    return LYNX_OK;
}

int ensure_errflag(lynx_ctx* c) {
    if (c->err_h) return LYNX_OK;
    LYNX_CUDA_TRY(cudaHostAlloc(&c->err_h, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
    *c->err_h = 0;
    LYNX_CUDA_TRY(cudaHostGetDevicePointer(&c->err_d, c->err_h, 0));
    return LYNX_OK;
}

// The end of a call: waits for its work and reports a bounded wait that gave up.  It waits whichever
// kernels ran, not only where there is a flag to look at: the blocks, row layouts and projections that
// the work uses are the context's, and the next call may come on another stream.  Recorded work (stream
// capture) has nothing to wait for; kernels with bounded waits are not recorded, as their flag could not
// be looked at.
int check_errflag(lynx_ctx* c) {
    if (!c->err_h) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        LYNX_CUDA_TRY(cudaStreamIsCapturing(c->stream, &cap));
        if (cap != cudaStreamCaptureStatusNone) return LYNX_OK;
    }
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    c->pending = false;
    if (!c->err_h) return LYNX_OK;
    volatile int* flag = c->err_h;
    if (*flag) {
        *flag = 0;
        set_error("a bounded device-side wait gave up (shared-memory pipeline did not complete)");
        return LYNX_ERR_TIMEOUT;
    }
    return LYNX_OK;
}

// The end of a call that returns with work in flight on the context's projections.
int leave_in_flight(lynx_ctx* c) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    LYNX_CUDA_TRY(cudaStreamIsCapturing(c->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) return LYNX_OK;
    if (!c->in_flight) LYNX_CUDA_TRY(cudaEventCreateWithFlags(&c->in_flight, cudaEventDisableTiming));
    LYNX_CUDA_TRY(cudaEventRecord(c->in_flight, c->stream));
    c->pending = true;
    return LYNX_OK;
}

// One fused step: out = a*(H_loc x) + b*x + d*xold, plus the nonlocal part a*Vnl x.
// Blocks use rows of length nxp (nxp == nx: the caller's unpadded layout); V uses the same rows.
// 16-byte aligned layouts run the pipelined kernel, others the direct one.
// Launch-shape autotuner of the pipelined stencil.  The first launch for a given (type, grid,
// columns) times every compiled shape on the actual arguments (one untimed launch each, to load
// the module, then one timed launch) and keeps the fastest for the context; every shape writes
// bitwise the same output, and the last timed launch leaves it in place.  The filter never
// lets `out` alias `x` or `xold`, so repeating the launch is harmless.
template <typename T, typename S>
int pipe_launch_tuned(lynx_ctx* c, int nxp, const T* x, long long ldx, const T* xold, long long ldo, T* out,
                      long long ldout, const S* V, int ncol, double a, double b, double d, const T* phl,
                      const T* phr, const PipeNLHost* nlh) {
    const StencilGeom g = geom(c);
    const int nsh = pipe_shape_count<T>(g.R, g.nx);
    const std::array<long long, 8> key = {(long long)sizeof(T), (long long)ScalarOf<T>::cplx, nxp, c->ny, c->nz,
                                          ncol, nlh != nullptr, xold != nullptr && d != 0.0};
    if (c->force_shape >= 0)
        return launch_cheb_pipe<T, S>(g, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                      c->err_d, c->stream, c->force_shape < nsh ? c->force_shape : 0, nlh);
    auto it = c->pipe_shape.find(key);
    if (it != c->pipe_shape.end() || nsh <= 1 || !c->autotune) {
        const int si = (it != c->pipe_shape.end()) ? it->second : 0;
        return launch_cheb_pipe<T, S>(g, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                      c->err_d, c->stream, si, nlh);
    }
    cudaEvent_t e0, e1;
    LYNX_CUDA_TRY(cudaEventCreate(&e0));
    LYNX_CUDA_TRY(cudaEventCreate(&e1));
    int best = -1;
    float best_ms = 1e30f;
    int rc = LYNX_OK;
    for (int si = 0; si < nsh && rc == LYNX_OK; ++si) {
        rc = launch_cheb_pipe<T, S>(g, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                    c->err_d, c->stream, si, nlh);
        if (rc == LYNX_ERR_UNSUPPORTED) {  // this shape's stages do not fit: try the others
            rc = LYNX_OK;
            continue;
        }
        if (rc != LYNX_OK) break;
        cudaEventRecord(e0, c->stream);
        rc = launch_cheb_pipe<T, S>(g, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                    c->err_d, c->stream, si, nlh);
        cudaEventRecord(e1, c->stream);
        if (rc != LYNX_OK) break;
        if (cudaEventSynchronize(e1) != cudaSuccess) {
            set_error("stencil autotuning failed: %s", cudaGetErrorString(cudaGetLastError()));
            rc = LYNX_ERR_CUDA;
            break;
        }
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best_ms) {
            best_ms = ms;
            best = si;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc != LYNX_OK) return rc;
    if (best < 0) {
        set_error("no compiled launch shape of the pipelined stencil fits this grid");
        return LYNX_ERR_UNSUPPORTED;
    }
    c->pipe_shape[key] = best;
    // leave the chosen shape's (identical) output as the result of record
    return launch_cheb_pipe<T, S>(g, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                  c->err_d, c->stream, best, nlh);
}

// Adds the duration of the stencil launch bracketed by c->kt[0] (recorded before it) and an event
// recorded now; waits for it.
int stencil_time_add(lynx_ctx* c) {
    LYNX_CUDA_TRY(cudaEventRecord(c->kt[1], c->stream));
    LYNX_CUDA_TRY(cudaEventSynchronize(c->kt[1]));
    float ms = 0.0f;
    LYNX_CUDA_TRY(cudaEventElapsedTime(&ms, c->kt[0], c->kt[1]));
    c->kt_ms += ms;
    c->kt_n += 1;
    return LYNX_OK;
}

// The one-thread-per-point kernel (stencil_direct.cu) takes complex blocks, and real ones that are
// small enough to be bound by latency (both sides measured: see that file).
constexpr long long kDirectRealBytes = 1250000;
template <typename T> bool direct_step_pays(const lynx_ctx* c, int ncol) {
    return c->nx <= kDirectMaxNx && c->Nd * (long long)ncol * (long long)sizeof(T) <= kDirectRealBytes;
}

// Columns of the block that a step's ncol columns belong to.
int whole_cols(const lynx_ctx* c, int ncol) { return c->col_total > 0 ? c->col_total : ncol; }

// One Chebyshev step out = a H x + b x + d xold (H with the nonlocal term when tables are set).
// With the fused nonlocal path, xs_in (optional) is the compact sphere-point copy of x written
// by the previous step, and xs_out (optional) receives the compact copy of out; *xs_written
// tells the caller whether it was written (the fused path was taken).
template <typename T>
int cheb_step(lynx_ctx* c, int nxp, const T* x, long long ldx, const T* xold, long long ldo, T* out, long long ldout,
              const typename Real<T>::type* V, int ncol, double a, double b, double d, bool use_k,
              const T* xs_in = nullptr, T* xs_out = nullptr, bool* xs_written = nullptr) {
    if (xs_written) *xs_written = false;
    using S = typename Real<T>::type;
    T phl[3], phr[3];
    ghost_phases<T>(c, use_k, phl, phr);
    const bool pipe_ok = pipe_capable<T>(c) && (nxp * sizeof(S)) % 16 == 0 && (ldx * sizeof(T)) % 16 == 0 &&
                         (ldout * sizeof(T)) % 16 == 0 && (!xold || (ldo * sizeof(T)) % 16 == 0) && aligned16(x) &&
                         aligned16(out) && (!xold || aligned16(xold)) && aligned16(V);
    if (!pipe_ok && nxp != c->nx) {
        set_error("internal error: padded layout that is not 16-byte aligned");
        return LYNX_ERR_BAD_ARG;
    }
    const int ncolp = ((ncol + kNLColBlock - 1) / kNLColBlock) * kNLColBlock;
    // Fused nonlocal term: real data, periodic cell, pipelined kernel, disjoint spheres.  The
    // values (chi alpha) are expanded to the compact point numbering and added by the stencil
    // kernel itself (out += a * W), in the order the separate scatter would add them.
    // Few atoms: one kernel after the stencil does the gather and the term together.
    const bool few_pairs = nl_few_atoms<T>(c->nl, whole_cols(c, ncol));
    const bool few = c->has_nl && c->nl.compact && c->nl.max_np <= 32 && few_pairs;
    const bool fuse = c->has_nl && !few && c->fuse_nl && c->orth && pipe_ok && !ScalarOf<T>::cplx && !use_k && c->nl.compact &&
                      c->nl.n_colors == 1 && geom(c).R == 6 && c->bc[0] == LYNX_BC_PERIODIC &&
                      c->bc[1] == LYNX_BC_PERIODIC && c->bc[2] == LYNX_BC_PERIODIC;
    const long long ldw = ((long long)c->nl.n_pts + 3) & ~3LL;  // compact column stride
    const bool direct =
        ScalarOf<T>::cplx || !pipe_ok || (!fuse && c->force_shape < 0 && direct_step_pays<T>(c, ncol));
    const NLDev* nl = nullptr;
    if (c->has_nl) LYNX_TRY(nl_for(c, nxp, &nl));
    if (c->has_nl && !few) {
        LYNX_TRY(c->alpha.ensure(sizeof(T) * (size_t)c->nl.total_proj * ncolp));
        if (fuse && xs_in) {
            // gather from the dense compact copy: entries index it through ent_pt
            NLDev cv = *nl;
            cv.gpos = c->nl.ent_pt;
            LYNX_TRY(launch_nl_gather<T>(cv, xs_in, ldw, ncol, c->alpha.as<T>(), ncolp, c->dV, c->stream, few_pairs));
        } else {
            LYNX_TRY(launch_nl_gather<T>(*nl, x, ldx, ncol, c->alpha.as<T>(), ncolp, c->dV, c->stream, few_pairs));
        }
    }
    const long long ldg = (long long)nxp * c->ny * c->nz;
    NonOrthGeom ng{};
    T *gy = nullptr, *gz = nullptr;
    if (!c->orth) {
        // mixed-derivative terms of a non-orthogonal cell, from two first-derivative blocks
        for (int i = 0; i < 2; ++i) LYNX_TRY(c->gradbuf[i].ensure(sizeof(T) * (size_t)ldg * ncol));
        gy = c->gradbuf[0].as<T>();
        gz = c->gradbuf[1].as<T>();
        ng = NonOrthGeom{c->nx, c->ny, c->nz, geom(c).R, c->D1y.data(), c->D1z.data(), c->D2xy.data(), c->D2xz.data(),
                         c->D2yz.data()};
    }
    if (direct) {
        if (c->time_stencil) LYNX_CUDA_TRY(cudaEventRecord(c->kt[0], c->stream));
        LYNX_TRY(launch_direct_step<T, S>(geom(c), nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                          c->orth ? nullptr : &ng, gy, gz, ldg, c->stream));
        if (c->time_stencil) LYNX_TRY(stencil_time_add(c));
    }
    if constexpr (!ScalarOf<T>::cplx) {
        if (!direct) {
            LYNX_TRY(ensure_errflag(c));
            if (fuse) {
                const lynx_ctx::NLMap* nm = nullptr;
                LYNX_TRY(nl_map_for(c, nxp, &nm));
                LYNX_TRY(c->nlW.ensure(sizeof(T) * (size_t)ldw * ncol));
                LYNX_TRY(launch_nl_expand<T>(*nl, c->nlW.as<T>(), ldw, ncol, c->alpha.as<T>(), ncolp, c->stream));
                PipeNLHost nh{c->nlW.p, ldw, nm->ptmap.as<int>(), nm->mp, nm->rowstart.as<int>(), &nm->rowstart_h,
                              xs_out};
                if (c->time_stencil) LYNX_CUDA_TRY(cudaEventRecord(c->kt[0], c->stream));
                LYNX_TRY(pipe_launch_tuned<T, S>(c, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                                 &nh));
                if (c->time_stencil) LYNX_TRY(stencil_time_add(c));
                if (xs_written) *xs_written = (xs_out != nullptr);
                return LYNX_OK;
            }
            if (c->time_stencil) LYNX_CUDA_TRY(cudaEventRecord(c->kt[0], c->stream));
            LYNX_TRY(pipe_launch_tuned<T, S>(c, nxp, x, ldx, xold, ldo, out, ldout, V, ncol, a, b, d, phl, phr,
                                             nullptr));
            if (c->time_stencil) LYNX_TRY(stencil_time_add(c));
        }
    }
    if (!c->orth)
        LYNX_TRY(launch_nonorth_terms<T>(ng, nxp, x, ldx, gy, gz, ldg, out, ldout, ncol, a, phl, phr, c->stream,
                                         direct));
    if (few) LYNX_TRY(launch_nl_apply<T>(*nl, x, ldx, out, ldout, ncol, c->dV, (S)a, c->stream));
    else if (c->has_nl)
        LYNX_TRY(launch_nl_scatter<T, S>(*nl, out, ldout, ncol, c->alpha.as<T>(), ncolp, (S)a, c->stream));
    return LYNX_OK;
}

// Chebyshev filter (src/solvers/EigenSolver.cpp:559-619) on blocks of type T with rows of
// length nxp.  X (column stride ldX) is read at the first two steps only; bufs[0..2]
// (column stride ldb) rotate.  Returns the block holding the filtered Y in *yout.
// Compact sphere-point buffers (two, used alternately) for the fused nonlocal path; null when
// the path does not apply.
template <typename T>
int compact_bufs(lynx_ctx* c, int ncol, T* xs[2]) {
    xs[0] = xs[1] = nullptr;
    if (ScalarOf<T>::cplx || !c->has_nl || !c->fuse_nl || !c->fuse_compact_gather || !c->nl.compact ||
        c->nl.n_colors != 1 || nl_few_atoms<T>(c->nl, whole_cols(c, ncol)))
        return LYNX_OK;
    const long long ldw = ((long long)c->nl.n_pts + 3) & ~3LL;
    for (int i = 0; i < 2; ++i) {
        LYNX_TRY(c->xsbuf[i].ensure(sizeof(T) * (size_t)ldw * ncol));
        xs[i] = c->xsbuf[i].as<T>();
    }
    return LYNX_OK;
}

template <typename T>
int filter_blocks(lynx_ctx* c, int nxp, const T* X, long long ldX, T* bufs[3], long long ldb,
                  const typename Real<T>::type* V, int ncol, double lc, double emin, double emax, int degree,
                  bool use_k, T** yout, const T** ys_out = nullptr) {
    const double e = (emax - lc) / 2.0;
    const double cc = (emax + lc) / 2.0;
    const double sigma1 = e / (emin - cc);
    double sigma = sigma1;
    T* xs[2];
    LYNX_TRY(compact_bufs<T>(c, ncol, xs));
    const T* xin = nullptr;  // compact copy of the current x, when the previous step wrote one
    bool wr = false;
    // Y = (sigma1/e) (H X - c X)
    const double s0 = sigma1 / e;
    LYNX_TRY(cheb_step<T>(c, nxp, X, ldX, nullptr, 0, bufs[0], ldb, V, ncol, s0, -cc * s0, 0.0, use_k, nullptr, xs[0],
                          &wr));
    xin = wr ? xs[0] : nullptr;
    const T* xold = X;
    long long ldold = ldX;
    int iy = 0;
    for (int k = 2; k <= degree; ++k) {
        const double sigma_new = 1.0 / (2.0 / sigma1 - sigma);
        const double gamma = 2.0 * sigma_new / e;
        const int inew = (iy + 1) % 3;
        T* xo = xs[(k - 1) & 1];
        LYNX_TRY(cheb_step<T>(c, nxp, bufs[iy], ldb, xold, ldold, bufs[inew], ldb, V, ncol, gamma, -gamma * cc,
                              -sigma * sigma_new, use_k, xin, xo, &wr));
        xin = wr ? xo : nullptr;
        xold = bufs[iy];
        ldold = ldb;
        iy = inew;
        sigma = sigma_new;
    }
    *yout = bufs[iy];
    if (ys_out) *ys_out = xin;
    return LYNX_OK;
}


// Filter of the caller's FP64 block X (unpadded rows, column stride ldX) in FP64, on internal
// blocks with rows of length nxp (16-byte multiples).  *Y (and *HY = H*Y when requested) are
// left in internal storage with column stride *ldb.
template <typename T64>
int run_filter64(lynx_ctx* c, const T64* X, long long ldX, const double* veff, int N, double lc, double emin,
                 double emax, int degree, bool use_k, bool want_hy, T64** Y, T64** HY, long long* ldb, int* nxp) {
    using S = typename Real<T64>::type;
    *nxp = pipe_capable<T64>(c) ? pipe_row_elems(c->nx, sizeof(S)) : c->nx;
    *ldb = (long long)(*nxp) * c->ny * c->nz;
    const size_t blk = sizeof(T64) * (size_t)(*ldb) * N;
    const bool direct = (*nxp == c->nx) && (ldX * sizeof(T64)) % 16 == 0 && aligned16(X);
    const int tag = (int)(sizeof(T64) * 1000 + *nxp);
    for (int i = 0; i < (direct ? 3 : 4); ++i) LYNX_TRY(ensure_layout(c, c->wbuf[i], blk, tag));
    const S* Vp = nullptr;
    LYNX_TRY(veff_layout<S>(c, veff, *nxp, &Vp));
    const T64* Xin = X;
    long long ldin = ldX;
    if (!direct) {
        LYNX_TRY(repack<T64, T64>(c, c->wbuf[3].as<T64>(), *nxp, *ldb, X, c->nx, ldX, N));
        Xin = c->wbuf[3].as<T64>();
        ldin = *ldb;
    }
    T64* bufs[3] = {c->wbuf[0].as<T64>(), c->wbuf[1].as<T64>(), c->wbuf[2].as<T64>()};
    const T64* ys = nullptr;
    LYNX_TRY(filter_blocks<T64>(c, *nxp, Xin, ldin, bufs, *ldb, Vp, N, lc, emin, emax, degree, use_k, Y, &ys));
    if (want_hy) {
        *HY = (*Y == bufs[0]) ? bufs[1] : bufs[0];
        LYNX_TRY(cheb_step<T64>(c, *nxp, *Y, *ldb, nullptr, 0, *HY, *ldb, Vp, N, 1.0, 0.0, 0.0, use_k, ys));
    }
    return LYNX_OK;
}

// Same in FP32 (T32 = float / float2) from the caller's FP64 block.
template <typename T32, typename T64>
int run_filter32(lynx_ctx* c, const T64* X, long long ldX, const double* veff, int N, double lc, double emin,
                 double emax, int degree, bool use_k, bool want_hy, T32** Y, T32** HY, long long* ldb, int* nxp) {
    using S = typename Real<T32>::type;
    *nxp = pipe_capable<T32>(c) ? pipe_row_elems(c->nx, sizeof(S)) : c->nx;
    *ldb = (long long)(*nxp) * c->ny * c->nz;
    const size_t blk = sizeof(T32) * (size_t)(*ldb) * N;
    const int tag = (int)(sizeof(T32) * 1000 + *nxp);
    for (int i = 0; i < 4; ++i) LYNX_TRY(ensure_layout(c, c->wbuf[i], blk, tag));
    const S* Vp = nullptr;
    LYNX_TRY(veff_layout<S>(c, veff, *nxp, &Vp));
    T32* X32 = c->wbuf[3].as<T32>();
    T32* bufs[3] = {c->wbuf[0].as<T32>(), c->wbuf[1].as<T32>(), c->wbuf[2].as<T32>()};
    // Column blocks: every column is filtered independently, so blocks give bitwise the same
    // result; a block waits for the event that marks its arrival (host-pointer solve), and the
    // copies of later blocks overlap the filtering of earlier ones.
    std::vector<std::pair<int, cudaEvent_t>> blocks = c->col_blocks;
    if (blocks.empty()) blocks.push_back({0, nullptr});
    for (size_t bi = 0; bi < blocks.size(); ++bi) {
        const int b0 = blocks[bi].first;
        const int nb = (bi + 1 < blocks.size() ? blocks[bi + 1].first : N) - b0;
        if (blocks[bi].second) LYNX_CUDA_TRY(cudaStreamWaitEvent(c->stream, blocks[bi].second, 0));
        const long long o = (long long)b0 * (*ldb);
        LYNX_TRY(repack<T32, T64>(c, X32 + o, *nxp, *ldb, X + (long long)b0 * ldX, c->nx, ldX, nb));
        T32* bb[3] = {bufs[0] + o, bufs[1] + o, bufs[2] + o};
        T32* yb = nullptr;
        const T32* ys = nullptr;
        LYNX_TRY(filter_blocks<T32>(c, *nxp, X32 + o, *ldb, bb, *ldb, Vp, nb, lc, emin, emax, degree, use_k, &yb, &ys));
        const int iy = (yb == bb[0]) ? 0 : (yb == bb[1] ? 1 : 2);  // the same buffer for every block
        *Y = bufs[iy];
        if (want_hy) {
            *HY = (iy == 0) ? bufs[1] : bufs[0];
            LYNX_TRY(cheb_step<T32>(c, *nxp, yb, *ldb, nullptr, 0, *HY + o, *ldb, Vp, nb, 1.0, 0.0, 0.0, use_k, ys));
        }
    }
    return LYNX_OK;
}

}  // namespace

namespace {
// ---------------------------------------------------------------------------
// Rayleigh-Ritz in FP64 (cuBLAS / cuSOLVER), real and complex.
// ---------------------------------------------------------------------------
#define CUBLAS_TRY(expr)                                                  \
    do {                                                                  \
        cublasStatus_t _s = (expr);                                       \
        if (_s != CUBLAS_STATUS_SUCCESS) {                                \
            set_error("%s failed: cublas status %d", #expr, (int)_s);    \
            return LYNX_ERR_CUDA;                                         \
        }                                                                 \
    } while (0)
#define CUSOLVER_TRY(expr)                                                \
    do {                                                                  \
        cusolverStatus_t _s = (expr);                                     \
        if (_s != CUSOLVER_STATUS_SUCCESS) {                              \
            set_error("%s failed: cusolver status %d", #expr, (int)_s);  \
            return LYNX_ERR_CUDA;                                         \
        }                                                                 \
    } while (0)

// Flags (device int) a NaN or Inf among the entries of the N x N matrix A (asynchronous).
int check_finite(lynx_ctx* c, const double* A, int N, int comps, bool upper, int* flag) {
    const long long n2 = (long long)N * N;
    const int blocks = (int)std::min<long long>((n2 + 255) / 256, 148LL * 8);
    nonfinite_kernel<<<blocks, 256, 0, c->stream>>>(A, N, comps, upper ? 1 : 0, flag);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return LYNX_OK;
}

int finish_rr(lynx_ctx* c, int N, double* eig_host) {
    const size_t need = (size_t)N + 2;  // Ritz values, then info
    if (c->res_n < need) {
        if (c->res_h) cudaFreeHost(c->res_h);
        c->res_h = nullptr;
        c->res_n = 0;
        LYNX_CUDA_TRY(cudaHostAlloc(&c->res_h, need * sizeof(double), cudaHostAllocPortable));
        c->res_n = need;
    }
    int info[3] = {0, 0, 0};
    LYNX_CUDA_TRY(cudaMemcpyAsync(c->res_h, c->eigd.p, N * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    LYNX_CUDA_TRY(cudaMemcpyAsync(c->res_h + N, c->info.p, 3 * sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    std::memcpy(eig_host, c->res_h, N * sizeof(double));
    std::memcpy(info, c->res_h + N, 3 * sizeof(int));
    if (info[2] != 0) {
        set_error("non-finite entries in the overlap or projected Hamiltonian (NaN/Inf in the orbitals or Veff)");
        return LYNX_ERR_NONFINITE;
    }
    if (info[0] != 0) {
        set_error("Cholesky factorization of the overlap failed (info=%d)", info[0]);
        return info[0] > 0 ? LYNX_ERR_CHOL_FAIL : LYNX_ERR_BAD_ARG;
    }
    if (info[1] != 0) {
        set_error("subspace eigensolver failed (info=%d, N=%d)", info[1], N);
        return info[1] > 0 ? LYNX_ERR_EIG_FAIL : LYNX_ERR_BAD_ARG;
    }
    for (int i = 0; i < N; ++i)
        if (!std::isfinite(eig_host[i])) {
            set_error("non-finite Ritz value at index %d", i);
            return LYNX_ERR_NONFINITE;
        }
    return LYNX_OK;
}

// Subspace part of the Rayleigh-Ritz step, given Ms = dV Y^T Y and Hs = dV Y^T HY in c->Ms /
// c->Hs (Ms: at least the upper triangle): Hs' = R^-T sym(Hs) R^-1 with R^T R = Ms,
// eigenpairs of Hs' (values into c->eigd), W = R^-1 Q left in c->Hs.  Asynchronous.
int rr_small_real(lynx_ctx* c, int N) {
    double* Ms = c->Ms.as<double>();
    double* Hs = c->Hs.as<double>();
    const double one = 1.0;
    {
        dim3 b(16, 16), g((N + 15) / 16, (N + 15) / 16);
        symmetrize_kernel<<<g, b, 0, c->stream>>>(Hs, N);
        count_launch();
    }
    int lw1 = 0, lw2 = 0;
    CUSOLVER_TRY(cusolverDnDpotrf_bufferSize(c->cusolver, CUBLAS_FILL_MODE_UPPER, N, Ms, N, &lw1));
    CUSOLVER_TRY(cusolverDnDsyevd_bufferSize(c->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, N, Hs,
                                             N, c->eigd.as<double>(), &lw2));
    const int lw = std::max(lw1, lw2);
    LYNX_TRY(c->solver_work.ensure((size_t)lw * sizeof(double)));
    int* info = c->info.as<int>();  // zeroed by rr_alloc_small
    LYNX_TRY(check_finite(c, Ms, N, 1, true, info + 2));
    LYNX_TRY(check_finite(c, Hs, N, 1, false, info + 2));
    CUSOLVER_TRY(cusolverDnDpotrf(c->cusolver, CUBLAS_FILL_MODE_UPPER, N, Ms, N, c->solver_work.as<double>(), lw,
                                  info));
    CUBLAS_TRY(cublasDtrsm(c->cublas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_T, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    CUBLAS_TRY(cublasDtrsm(c->cublas, CUBLAS_SIDE_RIGHT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    CUSOLVER_TRY(cusolverDnDsyevd(c->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, N, Hs, N,
                                  c->eigd.as<double>(), c->solver_work.as<double>(), lw, info + 1));
    CUBLAS_TRY(cublasDtrsm(c->cublas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    return LYNX_OK;
}

// rr_small_real, then psi = Yrot W by cuBLAS DGEMM (Yrot: FP64 block with Nd rows).
int rr_subspace_real(lynx_ctx* c, const double* Yrot, long long ldY, double* psi, long long ldp, int N,
                     double* eig_host) {
    LYNX_TRY(rr_small_real(c, N));
    const double one = 1.0, zero = 0.0;
    CUBLAS_TRY(cublasDgemm(c->cublas, CUBLAS_OP_N, CUBLAS_OP_N, c->Nd, N, N, &one, Yrot, ldY, c->Hs.as<double>(), N,
                           &zero, psi, ldp));
    return finish_rr(c, N, eig_host);
}

int rr_alloc_small(lynx_ctx* c, int N, size_t elem) {
    const size_t nn = (size_t)N * N;
    LYNX_TRY(c->Ms.ensure(nn * elem));
    LYNX_TRY(c->Hs.ensure(nn * elem));
    LYNX_TRY(c->eigd.ensure(N * sizeof(double)));
    LYNX_TRY(c->info.ensure(3 * sizeof(int)));
    CUBLAS_TRY(cublasSetStream(c->cublas, c->stream));
    CUSOLVER_TRY(cusolverDnSetStream(c->cusolver, c->stream));
    // info[0]: potrf, info[1]: syevd, info[2]: a NaN / Inf seen in the products or their inputs
    LYNX_CUDA_TRY(cudaMemsetAsync(c->info.p, 0, 3 * sizeof(int), c->stream));
    return LYNX_OK;
}

// psi_out = Y R^-1 Q, eig = eig(R^-T (dV Y^T HY) R^-1), R^T R = dV Y^T Y; products by cuBLAS (FP64).
int rayleigh_ritz_real(lynx_ctx* c, const double* Y, long long ldY, const double* HY, long long ldH,
                       double* psi, long long ldp, int N, double* eig_host) {
    LYNX_TRY(rr_alloc_small(c, N, sizeof(double)));
    const double dV = c->dV, zero = 0.0;
    // The overlap as a full product: the library splits the long K of a GEMM over the SMs, but not that of
    // a rank-k update (Si64, 160 states: 0.43 ms against 2.8).
    CUBLAS_TRY(cublasDgemm(c->cublas, CUBLAS_OP_T, CUBLAS_OP_N, N, N, c->Nd, &dV, Y, ldY, Y, ldY, &zero,
                           c->Ms.as<double>(), N));
    CUBLAS_TRY(cublasDgemm(c->cublas, CUBLAS_OP_T, CUBLAS_OP_N, N, N, c->Nd, &dV, Y, ldY, HY, ldH, &zero,
                           c->Hs.as<double>(), N));
    return rr_subspace_real(c, Y, ldY, psi, ldp, N, eig_host);
}

// Fermi level of this pass's Ritz values (Occupation::find_fermi_level for one spin and one
// k-point, every state weighted by the request's weight) and the density weights
// w[n] = weight * f_n on the device (0 where f_n < 1e-16, which the reference skips).
int density_weights(lynx_ctx* c, const double* eig, int N) {
    std::vector<double> wt(N, c->dens.weight), occ(N);
    LYNX_TRY(lynx_fermi_level(eig, wt.data(), N, c->dens.nelectron, c->dens.beta, c->dens.smearing, &c->dens.ef));
    LYNX_TRY(lynx_occupations(eig, N, c->dens.ef, c->dens.beta, c->dens.smearing, occ.data()));
    for (int n = 0; n < N; ++n) wt[n] = (occ[n] < 1e-16) ? 0.0 : c->dens.weight * occ[n];
    LYNX_TRY(c->dens_w.ensure(sizeof(double) * N));
    LYNX_CUDA_TRY(cudaMemcpyAsync(c->dens_w.p, wt.data(), sizeof(double) * N, cudaMemcpyHostToDevice, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));  // wt is a host temporary
    return LYNX_OK;
}

// Mixed precision, real: Gram products and rotation of the FP32 blocks on the tensor cores
// (exact int8 slice products, FP64 combination), subspace algebra in FP64.  More states than
// the rotation kernel stages take the rotation by DGEMM on an FP64 copy of Y.
int rayleigh_ritz_mixed_real(lynx_ctx* c, const float* Y32, const float* HY32, long long ldb, int nxp, double* psi,
                             long long ldp, int N, double* eig_host) {
    LYNX_TRY(rr_alloc_small(c, N, sizeof(double)));
    const GramPlan plan = gram_plan(ldb, N);  // all ldb rows: pad elements are zero
    LYNX_TRY(c->gwork.ensure(plan.work_bytes));
    LYNX_TRY(ensure_errflag(c));
    LYNX_TRY(launch_gram_i8(Y32, HY32, ldb, ldb, N, c->dV, plan, c->gwork.p, c->gwork.bytes, c->Ms.as<double>(),
                            c->Hs.as<double>(), c->err_d, c->info.as<int>() + 2, c->stream));
    if (rot_supported(N)) {
        // rotation on the tensor cores, straight from the FP32 block into the caller's psi
        const RotPlan rp = rot_plan(ldb, N);
        LYNX_TRY(c->rwork.ensure(rp.work_bytes));
        LYNX_TRY(launch_colexp(c->Ms.as<double>(), N, c->rwork.p, rp, ldb, c->stream));
        LYNX_TRY(rr_small_real(c, N));
        if (c->dens.on) {
            // The Ritz values first (checked as after any pass): their occupations weight the
            // density, which the rotation accumulates from the FP64 orbitals it writes.
            LYNX_TRY(finish_rr(c, N, eig_host));
            LYNX_TRY(density_weights(c, eig_host, N));
            const int ntn = (N + 127) / 128;
            LYNX_TRY(c->dens_part.ensure(sizeof(double) * (size_t)ntn * c->Nd));
            RotDensity rd{c->dens_w.as<double>(), c->dens_part.as<double>(), c->dens.rho, c->Nd, false};
            LYNX_TRY(launch_rot_i8(Y32, ldb, ldb, c->nx, nxp, c->Hs.as<double>(), N, rp, c->rwork.p, c->rwork.bytes,
                                   psi, ldp, c->err_d, c->stream, &rd));
            c->dens.done = true;
            LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
            return LYNX_OK;
        }
        LYNX_TRY(launch_rot_i8(Y32, ldb, ldb, c->nx, nxp, c->Hs.as<double>(), N, rp, c->rwork.p, c->rwork.bytes, psi,
                               ldp, c->err_d, c->stream));
        return finish_rr(c, N, eig_host);
    }
    const long long Nd = c->Nd;
    LYNX_TRY(c->cvt[0].ensure(sizeof(double) * (size_t)Nd * N));
    LYNX_TRY(repack<double, float>(c, c->cvt[0].as<double>(), c->nx, Nd, Y32, nxp, ldb, N));
    return rr_subspace_real(c, c->cvt[0].as<double>(), Nd, psi, ldp, N, eig_host);
}

int rr_alloc_small_cplx(lynx_ctx* c, int N) {
    const size_t nn = (size_t)N * N;
    LYNX_TRY(c->Ms.ensure(nn * sizeof(double2)));
    LYNX_TRY(c->Hs.ensure(nn * sizeof(double2)));
    LYNX_TRY(c->eigd.ensure(N * sizeof(double)));
    LYNX_TRY(c->info.ensure(3 * sizeof(int)));
    CUBLAS_TRY(cublasSetStream(c->cublas, c->stream));
    CUSOLVER_TRY(cusolverDnSetStream(c->cusolver, c->stream));
    LYNX_CUDA_TRY(cudaMemsetAsync(c->info.p, 0, 3 * sizeof(int), c->stream));
    return LYNX_OK;
}

// Subspace part of the complex Rayleigh-Ritz step, given Ms = dV Y^H Y (upper triangle) and
// Hs = dV Y^H HY in c->Ms / c->Hs: Hs' = R^-H herm(Hs) R^-1 with R^H R = Ms, eigenpairs of Hs'
// (values into c->eigd), W = R^-1 Q left in c->Hs.  Asynchronous.
int rr_small_cplx(lynx_ctx* c, int N) {
    cuDoubleComplex* Ms = c->Ms.as<cuDoubleComplex>();
    cuDoubleComplex* Hs = c->Hs.as<cuDoubleComplex>();
    const cuDoubleComplex one = make_cuDoubleComplex(1, 0);
    {
        dim3 b(16, 16), g((N + 15) / 16, (N + 15) / 16);
        hermitize_kernel<<<g, b, 0, c->stream>>>(reinterpret_cast<double2*>(Hs), N);
        count_launch();
    }
    int lw1 = 0, lw2 = 0;
    CUSOLVER_TRY(cusolverDnZpotrf_bufferSize(c->cusolver, CUBLAS_FILL_MODE_UPPER, N, Ms, N, &lw1));
    CUSOLVER_TRY(cusolverDnZheevd_bufferSize(c->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, N, Hs,
                                             N, c->eigd.as<double>(), &lw2));
    const int lw = std::max(lw1, lw2);
    LYNX_TRY(c->solver_work.ensure((size_t)lw * sizeof(cuDoubleComplex)));
    int* info = c->info.as<int>();
    cuDoubleComplex* work = c->solver_work.as<cuDoubleComplex>();
    LYNX_TRY(check_finite(c, reinterpret_cast<const double*>(Ms), N, 2, true, info + 2));
    LYNX_TRY(check_finite(c, reinterpret_cast<const double*>(Hs), N, 2, false, info + 2));
    CUSOLVER_TRY(cusolverDnZpotrf(c->cusolver, CUBLAS_FILL_MODE_UPPER, N, Ms, N, work, lw, info));
    CUBLAS_TRY(cublasZtrsm(c->cublas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_C, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    CUBLAS_TRY(cublasZtrsm(c->cublas, CUBLAS_SIDE_RIGHT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    CUSOLVER_TRY(cusolverDnZheevd(c->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, N, Hs, N,
                                  c->eigd.as<double>(), work, lw, info + 1));
    CUBLAS_TRY(cublasZtrsm(c->cublas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT,
                           N, N, &one, Ms, N, Hs, N));
    return LYNX_OK;
}

int rayleigh_ritz_cplx(lynx_ctx* c, const double2* Y, long long ldY, const double2* HY, long long ldH,
                       double2* psi, long long ldp, int N, double* eig_host) {
    LYNX_TRY(rr_alloc_small_cplx(c, N));
    cuDoubleComplex* Ms = c->Ms.as<cuDoubleComplex>();
    cuDoubleComplex* Hs = c->Hs.as<cuDoubleComplex>();
    const cuDoubleComplex* Yz = reinterpret_cast<const cuDoubleComplex*>(Y);
    const cuDoubleComplex* HYz = reinterpret_cast<const cuDoubleComplex*>(HY);
    const double dV = c->dV, zero_r = 0.0;
    const cuDoubleComplex one = make_cuDoubleComplex(1, 0), zero = make_cuDoubleComplex(0, 0),
                          dVz = make_cuDoubleComplex(dV, 0);
    CUBLAS_TRY(cublasZherk(c->cublas, CUBLAS_FILL_MODE_UPPER, CUBLAS_OP_C, N, c->Nd, &dV, Yz, ldY, &zero_r, Ms, N));
    CUBLAS_TRY(cublasZgemm(c->cublas, CUBLAS_OP_C, CUBLAS_OP_N, N, N, c->Nd, &dVz, Yz, ldY, HYz, ldH, &zero, Hs, N));
    LYNX_TRY(rr_small_cplx(c, N));
    CUBLAS_TRY(cublasZgemm(c->cublas, CUBLAS_OP_N, CUBLAS_OP_N, c->Nd, N, N, &one, Yz, ldY, Hs, N, &zero,
                           reinterpret_cast<cuDoubleComplex*>(psi), ldp));
    return finish_rr(c, N, eig_host);
}

// Mixed precision, k-point: the Gram products and the rotation of the FP32 complex blocks on the
// real tensor-core kernels, through the planar split [Yr | Yi] (2N real states); subspace algebra
// in complex FP64.
int rayleigh_ritz_mixed_cplx(lynx_ctx* c, const float2* Y32, const float2* HY32, long long ldb, int nxp,
                             double2* psi, long long ldp, int N, double* eig_host) {
    const int N2 = 2 * N;
    const long long Nd = c->Nd;
    LYNX_TRY(rr_alloc_small_cplx(c, N));
    // planar copies of Y and HY, the real 2N x 2N products, Wt, and the planar FP64 rotation output
    const size_t pl_bytes = sizeof(float) * (size_t)ldb * N2;
    const size_t sq_bytes = sizeof(double) * (size_t)N2 * N2;
    LYNX_TRY(c->cplx_work.ensure(2 * pl_bytes + 3 * sq_bytes));
    float* Yp = reinterpret_cast<float*>(c->cplx_work.p);
    float* Hp = Yp + (size_t)ldb * N2;
    double* Mpl = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(c->cplx_work.p) + 2 * pl_bytes);
    double* Hpl = Mpl + (size_t)N2 * N2;
    double* Wt = Hpl + (size_t)N2 * N2;
    LYNX_TRY(c->cvt[0].ensure(sizeof(double) * (size_t)Nd * N2));
    double* R = c->cvt[0].as<double>();
    const int blocks = (int)std::min<long long>((ldb * N + 255) / 256, 148LL * 16);
    planar_kernel<<<blocks, 256, 0, c->stream>>>(Y32, ldb, N, Yp);
    planar_kernel<<<blocks, 256, 0, c->stream>>>(HY32, ldb, N, Hp);
    count_launch(2);
    const GramPlan plan = gram_plan(ldb, N2);  // all ldb rows: pad elements are zero
    LYNX_TRY(c->gwork.ensure(plan.work_bytes));
    LYNX_TRY(ensure_errflag(c));
    LYNX_TRY(launch_gram_i8(Yp, Hp, ldb, ldb, N2, c->dV, plan, c->gwork.p, c->gwork.bytes, Mpl, Hpl,
                            c->err_d, c->info.as<int>() + 2, c->stream));
    const RotPlan rp = rot_plan(ldb, N2);
    LYNX_TRY(c->rwork.ensure(rp.work_bytes));
    LYNX_TRY(launch_colexp(Mpl, N2, c->rwork.p, rp, ldb, c->stream));  // scaling of the 2N planar states
    {
        dim3 b(16, 16), g((N + 15) / 16, (N + 15) / 16);
        combine_gram_kernel<<<g, b, 0, c->stream>>>(Mpl, Hpl, N, c->Ms.as<double2>(), c->Hs.as<double2>());
        count_launch();
    }
    LYNX_TRY(rr_small_cplx(c, N));
    {
        dim3 b(16, 16), g((N + 15) / 16, (N + 15) / 16);
        wtilde_kernel<<<g, b, 0, c->stream>>>(c->Hs.as<double2>(), N, Wt);
        count_launch();
    }
    LYNX_TRY(launch_rot_i8(Yp, ldb, ldb, c->nx, nxp, Wt, N2, rp, c->rwork.p, c->rwork.bytes, R, Nd,
                           c->err_d, c->stream));
    const int ib = (int)std::min<long long>((Nd * N + 255) / 256, 148LL * 16);
    interleave_kernel<<<ib, 256, 0, c->stream>>>(R, Nd, N, psi, ldp);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return finish_rr(c, N, eig_host);
}

int rayleigh_ritz(lynx_ctx* c, const double* Y, long long ldY, const double* HY, long long ldH, double* psi,
                  long long ldp, int N, double* eig) {
    return rayleigh_ritz_real(c, Y, ldY, HY, ldH, psi, ldp, N, eig);
}
int rayleigh_ritz(lynx_ctx* c, const double2* Y, long long ldY, const double2* HY, long long ldH, double2* psi,
                  long long ldp, int N, double* eig) {
    return rayleigh_ritz_cplx(c, Y, ldY, HY, ldH, psi, ldp, N, eig);
}

// Few states: products, subspace algebra and rotation in four launches (small_rr.cu).
template <typename T>
int rayleigh_ritz_small(lynx_ctx* c, const T* Y, const T* HY, long long ldb, int nxp, void* psi, long long ldp, int N,
                        double* eig_host) {
    const size_t wide = ScalarOf<T>::cplx ? sizeof(double2) : sizeof(double);
    const long long rows = (long long)nxp * c->ny * c->nz;  // pad elements are zero
    LYNX_TRY(rr_alloc_small(c, N, wide));
    LYNX_TRY(c->gwork.ensure(small_rr_work_bytes(rows, N, wide)));
    LYNX_TRY(launch_small_rr<T>(Y, HY, ldb, rows, c->nx, nxp, c->Nd, N, c->dV, c->gwork.p, c->Ms.p, c->Hs.p,
                                c->eigd.as<double>(), c->info.as<int>(), psi, ldp, c->stream));
    return finish_rr(c, N, eig_host);
}

// Mixed precision above kSmallRRMax states: products of 23-bit digits on the tensor cores, or FP64 products of
// the FP32 blocks where the caller wants them and for odd nx.  Those blocks had FP64 products before their
// rows were padded for the pipelined stencil, and the digits would take bits from the result: over 49^3 to
// 61^3 points and 145 to 179 states the density lies 8.4e-8 from its 64-bit value with digits, 3.9e-8 with
// FP64 products (relative 2-norm; the Ritz values 4e-8 either way).
bool use_tc_products(const lynx_ctx* c) { return c->nx % 2 == 0 && !c->no_tc_gram; }

// ---------------------------------------------------------------------------
// CheFSI pass.  T64 = FP64 storage type (double / double2), T32 = FP32 (float / float2).
// ---------------------------------------------------------------------------
template <typename T64, typename T32>
int solve_impl(lynx_ctx* c, T64* psi, double* eig, const double* veff, int N, int ld, double lc, double emin,
               double emax, int degree, int precision, double* lc_out, bool use_k) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    LYNX_CHECK_ARG(psi != nullptr && eig != nullptr && veff != nullptr, "null pointer");
    LYNX_CHECK_ARG(N > 0, "nband must be positive");
    LYNX_CHECK_ARG(degree >= 1, "cheb_degree must be >= 1");
    LYNX_CHECK_ARG(precision == LYNX_PREC_FP64 || precision == LYNX_PREC_MIXED, "unknown precision");
    LYNX_CHECK_ARG(emax > lc && emin < lc, "spectral bounds must satisfy eigmin < lambda_cutoff < eigmax");
    LYNX_TRY(activate(c));
    const long long Nd = c->Nd;
    const long long ldp = ld > 0 ? ld : Nd;
    LYNX_CHECK_ARG(ldp >= Nd, "ld < Nd");
    const size_t blk64 = sizeof(T64) * (size_t)Nd * N;
    long long ldb = 0;
    int nxp = 0;
    if (precision == LYNX_PREC_FP64) {
        T64 *Y = nullptr, *HY = nullptr;
        LYNX_TRY(run_filter64<T64>(c, psi, ldp, veff, N, lc, emin, emax, degree, use_k, true, &Y, &HY, &ldb, &nxp));
        if (small_rr_supported(N)) {
            LYNX_TRY(rayleigh_ritz_small<T64>(c, Y, HY, ldb, nxp, psi, ldp, N, eig));
        } else if (nxp == c->nx) {
            LYNX_TRY(rayleigh_ritz(c, Y, ldb, HY, ldb, psi, ldp, N, eig));
        } else {
            LYNX_TRY(c->cvt[0].ensure(blk64));
            LYNX_TRY(c->cvt[1].ensure(blk64));
            LYNX_TRY(repack<T64, T64>(c, c->cvt[0].as<T64>(), c->nx, Nd, Y, nxp, ldb, N));
            LYNX_TRY(repack<T64, T64>(c, c->cvt[1].as<T64>(), c->nx, Nd, HY, nxp, ldb, N));
            LYNX_TRY(rayleigh_ritz(c, c->cvt[0].as<T64>(), Nd, c->cvt[1].as<T64>(), Nd, psi, ldp, N, eig));
        }
    } else {
        T32 *Y = nullptr, *HY = nullptr;
        LYNX_TRY(run_filter32<T32, T64>(c, psi, ldp, veff, N, lc, emin, emax, degree, use_k, true, &Y, &HY, &ldb,
                                        &nxp));
        if (small_rr_supported(N) && !c->no_tc_gram) {
            LYNX_TRY(rayleigh_ritz_small<T32>(c, Y, HY, ldb, nxp, psi, ldp, N, eig));
            LYNX_TRY(check_errflag(c));
            if (lc_out) *lc_out = eig[N - 1] + 0.1;
            return LYNX_OK;
        }
        if constexpr (std::is_same<T32, float>::value) {
            if (use_tc_products(c)) {
                LYNX_TRY(rayleigh_ritz_mixed_real(c, Y, HY, ldb, nxp, reinterpret_cast<double*>(psi), ldp, N, eig));
                LYNX_TRY(check_errflag(c));
                if (lc_out) *lc_out = eig[N - 1] + 0.1;
                return LYNX_OK;
            }
        } else {
            if (use_tc_products(c) && rot_supported(2 * N)) {
                LYNX_TRY(rayleigh_ritz_mixed_cplx(c, Y, HY, ldb, nxp, reinterpret_cast<double2*>(psi), ldp, N, eig));
                LYNX_TRY(check_errflag(c));
                if (lc_out) *lc_out = eig[N - 1] + 0.1;
                return LYNX_OK;
            }
        }
        // Rayleigh-Ritz products on FP64 copies of the FP32 blocks.
        LYNX_TRY(c->cvt[0].ensure(blk64));
        LYNX_TRY(c->cvt[1].ensure(blk64));
        LYNX_TRY(repack<T64, T32>(c, c->cvt[0].as<T64>(), c->nx, Nd, Y, nxp, ldb, N));
        LYNX_TRY(repack<T64, T32>(c, c->cvt[1].as<T64>(), c->nx, Nd, HY, nxp, ldb, N));
        LYNX_TRY(rayleigh_ritz(c, c->cvt[0].as<T64>(), Nd, c->cvt[1].as<T64>(), Nd, psi, ldp, N, eig));
    }
    LYNX_TRY(check_errflag(c));
    if (lc_out) *lc_out = eig[N - 1] + 0.1;
    return LYNX_OK;
}

// Bisection count of eigenvalues of the symmetric tridiagonal (d, e) below x (Sturm sequence).
int sturm_count(const std::vector<double>& d, const std::vector<double>& e, int n, double x) {
    int cnt = 0;
    double q = 1.0;
    for (int i = 0; i < n; ++i) {
        const double off = (i > 0) ? e[i - 1] * e[i - 1] : 0.0;
        q = d[i] - x - (i > 0 ? off / q : 0.0);
        if (q == 0.0) q = -1e-300;
        if (q < 0) ++cnt;
    }
    return cnt;
}

// Smallest and largest eigenvalue of an n x n symmetric tridiagonal matrix by bisection.
void tridiag_extremes(const std::vector<double>& d, const std::vector<double>& e, int n, double* lo,
                      double* hi) {
    double gl = d[0], gu = d[0];
    for (int i = 0; i < n; ++i) {
        const double r = (i > 0 ? std::fabs(e[i - 1]) : 0.0) + (i < n - 1 ? std::fabs(e[i]) : 0.0);
        gl = std::min(gl, d[i] - r);
        gu = std::max(gu, d[i] + r);
    }
    const double span = std::max(std::fabs(gl), std::fabs(gu));
    auto bisect = [&](int k) {  // k-th smallest (0-based)
        double a = gl - 1e-12 * span - 1e-300, b = gu + 1e-12 * span + 1e-300;
        for (int it = 0; it < 200; ++it) {
            const double m = 0.5 * (a + b);
            if (m == a || m == b) break;
            if (sturm_count(d, e, n, m) > k) b = m;
            else a = m;
        }
        return 0.5 * (a + b);
    };
    *lo = bisect(0);
    *hi = bisect(n - 1);
}

template <typename T>
__global__ void lanczos_update_kernel(T* __restrict__ vp1, T* __restrict__ vj, T* __restrict__ vjm1, double a,
                                      double b, long long n) {
    // vp1 -= a*vj + b*vjm1; vjm1 = vj
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        vp1[i] = vp1[i] - a * vj[i] - b * vjm1[i];
        vjm1[i] = vj[i];
    }
}

// Lanczos extreme-eigenvalue estimate (src/solvers/Lanczos.hpp:92-200), vectors on the device.
// Real data: Nv = Nd doubles; complex: Nv = 2*Nd doubles viewed as interleaved complex.
template <typename T>
int lanczos_impl(lynx_ctx* c, const double* veff, double tol, int max_iter, double* eigmin, double* eigmax,
                 bool use_k) {
    LYNX_CHECK_ARG(c && veff && eigmin && eigmax, "null pointer");
    LYNX_CHECK_ARG(max_iter >= 1, "max_iter must be >= 1");
    LYNX_TRY(activate(c));
    const bool cplx = sizeof(T) == sizeof(double2);
    const long long Nv = cplx ? 2LL * c->Nd : c->Nd;  // doubles per vector
    for (int i = 0; i < 3; ++i) LYNX_TRY(c->lz[i].ensure(Nv * sizeof(double)));
    double* vjm1 = c->lz[0].as<double>();
    double* vj = c->lz[1].as<double>();
    double* vp1 = c->lz[2].as<double>();
    // Start vector: srand(1); entries rand()/RAND_MAX.  For complex entries the reference
    // writes Complex(rand()/RAND_MAX, rand()/RAND_MAX), whose GCC build draws the imaginary
    // part first; the same order is kept so both start from the same vector.
    std::vector<double> h(Nv);
    std::srand(1);
    if (cplx) {
        for (long long i = 0; i < Nv; i += 2) {
            h[i + 1] = (double)std::rand() / RAND_MAX;
            h[i] = (double)std::rand() / RAND_MAX;
        }
    } else {
        for (long long i = 0; i < Nv; ++i) h[i] = (double)std::rand() / RAND_MAX;
    }
    double nrm = 0;
    for (double v : h) nrm += v * v;
    const double sc = 1.0 / std::sqrt(nrm);
    for (double& v : h) v *= sc;
    LYNX_CUDA_TRY(cudaMemcpyAsync(vjm1, h.data(), Nv * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    CUBLAS_TRY(cublasSetStream(c->cublas, c->stream));
    const double* Vl = nullptr;
    LYNX_TRY(veff_layout<double>(c, veff, c->nx, &Vl));
    auto Happly = [&](const double* x, double* y) -> int {
        return cheb_step<T>(c, c->nx, reinterpret_cast<const T*>(x), c->Nd, nullptr, 0, reinterpret_cast<T*>(y),
                            c->Nd, Vl, 1, 1.0, 0.0, 0.0, use_k);
    };
    auto dot = [&](const double* x, const double* y, double* r) -> int {
        CUBLAS_TRY(cublasDdot(c->cublas, (int)Nv, x, 1, y, 1, r));  // Re<x,y> for interleaved complex too
        return LYNX_OK;
    };
    auto norm = [&](const double* x, double* r) -> int {
        CUBLAS_TRY(cublasDnrm2(c->cublas, (int)Nv, x, 1, r));
        return LYNX_OK;
    };
    std::vector<double> a(max_iter + 1, 0.0), b(max_iter + 1, 0.0);
    LYNX_TRY(Happly(vjm1, vj));
    LYNX_TRY(dot(vjm1, vj, &a[0]));
    {
        const double m = -a[0];
        CUBLAS_TRY(cublasDaxpy(c->cublas, (int)Nv, &m, vjm1, 1, vj, 1));
    }
    LYNX_TRY(norm(vj, &b[0]));
    if (b[0] == 0.0) {
        set_error("Lanczos start vector spans an invariant subspace");
        return LYNX_ERR_NONFINITE;
    }
    {
        const double s = 1.0 / b[0];
        CUBLAS_TRY(cublasDscal(c->cublas, (int)Nv, &s, vj, 1));
    }
    double emin = 0, emax = 0, pmin = 0, pmax = 0, errmin = tol + 1, errmax = tol + 1;
    int j = 0;
    std::vector<double> d, e;
    const int blocks = (int)std::min<long long>((Nv + 255) / 256, 148 * 8);
    while ((errmin > tol || errmax > tol) && j < max_iter) {
        LYNX_TRY(Happly(vj, vp1));
        LYNX_TRY(dot(vj, vp1, &a[j + 1]));
        lanczos_update_kernel<double><<<blocks, 256, 0, c->stream>>>(vp1, vj, vjm1, a[j + 1], b[j], Nv);
        count_launch();
        LYNX_TRY(norm(vp1, &b[j + 1]));
        if (b[j + 1] == 0.0) break;
        const double s = 1.0 / b[j + 1];
        LYNX_CUDA_TRY(cudaMemcpyAsync(vj, vp1, Nv * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
        CUBLAS_TRY(cublasDscal(c->cublas, (int)Nv, &s, vj, 1));
        const int n = j + 2;
        d.assign(a.begin(), a.begin() + n);
        e.assign(b.begin(), b.begin() + n);
        tridiag_extremes(d, e, n, &emin, &emax);
        errmin = std::fabs(emin - pmin);
        errmax = std::fabs(emax - pmax);
        pmin = emin;
        pmax = emax;
        ++j;
    }
    LYNX_TRY(check_errflag(c));
    *eigmax = emax * 1.01;
    *eigmin = emin - 0.1;
    return LYNX_OK;
}

// Brent's root finder (R. P. Brent, Algorithms for Minimization Without Derivatives, 1973, ch. 4)
// for f(a) f(b) <= 0, absolute tolerance tol.
template <typename F>
double brent_zero(F f, double a, double b, double tol, int max_iter) {
    double fa = f(a), fb = f(b);
    double c = a, fc = fa, d = b - a, e = d;
    for (int it = 0; it < max_iter; ++it) {
        if ((fb > 0 && fc > 0) || (fb < 0 && fc < 0)) {
            c = a;
            fc = fa;
            d = e = b - a;
        }
        if (std::fabs(fc) < std::fabs(fb)) {
            a = b;
            b = c;
            c = a;
            fa = fb;
            fb = fc;
            fc = fa;
        }
        const double tol1 = 2.0 * std::numeric_limits<double>::epsilon() * std::fabs(b) + 0.5 * tol;
        const double m = 0.5 * (c - b);
        if (std::fabs(m) <= tol1 || fb == 0.0) return b;
        if (std::fabs(e) >= tol1 && std::fabs(fa) > std::fabs(fb)) {
            // inverse quadratic interpolation, or secant when only two points differ
            const double s = fb / fa;
            double p, q;
            if (a == c) {
                p = 2.0 * m * s;
                q = 1.0 - s;
            } else {
                const double qa = fa / fc, r = fb / fc;
                p = s * (2.0 * m * qa * (qa - r) - (b - a) * (r - 1.0));
                q = (qa - 1.0) * (r - 1.0) * (s - 1.0);
            }
            if (p > 0) q = -q;
            else p = -p;
            if (2.0 * p < std::min(3.0 * m * q - std::fabs(tol1 * q), std::fabs(e * q))) {
                e = d;
                d = p / q;
            } else {
                d = m;
                e = d;
            }
        } else {
            d = m;
            e = d;
        }
        a = b;
        fa = fb;
        b += (std::fabs(d) > tol1) ? d : (m > 0 ? tol1 : -tol1);
        fb = f(b);
    }
    return b;
}

double smear(double x, double beta, int type) {
    if (type == LYNX_SMEAR_FERMI_DIRAC) {
        const double t = x * beta;
        if (t > 50.0) return 0.0;
        if (t < -50.0) return 1.0;
        return 1.0 / (1.0 + std::exp(t));
    }
    return 0.5 * std::erfc(beta * x);
}

}  // namespace

// ---------------------------------------------------------------------------
// Exported C entry points
// ---------------------------------------------------------------------------
extern "C" {

const char* lynx_status_string(int s) {
    switch (s) {
        case LYNX_OK: return "ok";
        case LYNX_ERR_BAD_ARG: return "bad argument";
        case LYNX_ERR_CUDA: return "CUDA error";
        case LYNX_ERR_OOM: return "out of device memory";
        case LYNX_ERR_CHOL_FAIL: return "Cholesky factorization failed";
        case LYNX_ERR_EIG_FAIL: return "subspace eigensolver failed";
        case LYNX_ERR_NONFINITE: return "non-finite values";
        case LYNX_ERR_TIMEOUT: return "device wait timed out";
        case LYNX_ERR_NOT_SETUP: return "not set up";
        case LYNX_ERR_UNSUPPORTED: return "unsupported configuration";
        case LYNX_ERR_BRACKET: return "Fermi level cannot be bracketed";
        default: return "unknown status";
    }
}

const char* lynx_last_error(void) { return g_last_error.c_str(); }
int lynx_version(void) { return 1; }
long long lynx_launch_count(int reset) {
    return reset ? g_launches.exchange(0) : g_launches.load();
}

int lynx_create(lynx_ctx** out, int device, int nx, int ny, int nz, int fd_order, const double* latvec,
                int orthogonal, const int* bc) {
    LYNX_CHECK_ARG(out != nullptr && latvec != nullptr, "null pointer");
    *out = nullptr;
    LYNX_CHECK_ARG(nx > 0 && ny > 0 && nz > 0, "grid dimensions must be positive");
    // Grid points are counted in 32 bits: by the thread of a block of up to 128 past the last point, and in
    // rows rounded up to four elements.
    LYNX_CHECK_ARG((nx + 3LL) / 4 * 4 * ny <= INT_MAX / nz && (nx + 3LL) / 4 * 4 * ny * nz <= INT_MAX - 128,
                   "more grid points than 32-bit indices hold");
    LYNX_CHECK_ARG(fd_order >= 2 && fd_order % 2 == 0, "FD order must be even and >= 2");
    lynx_ctx* c = new lynx_ctx();
    c->device = device;
    c->nx = nx;
    c->ny = ny;
    c->nz = nz;
    c->Nd = nx * ny * nz;
    c->fd_order = fd_order;
    c->R = fd_order / 2;
    c->orth = orthogonal != 0;
    for (int d = 0; d < 3; ++d) c->bc[d] = bc ? bc[d] : LYNX_BC_PERIODIC;
    std::memcpy(c->latvec, latvec, 9 * sizeof(double));
    build_stencil(c);
    if (!(c->jac > 1e-14)) {
        delete c;
        set_error("lattice vectors are coplanar");
        return LYNX_ERR_BAD_ARG;
    }
    *out = c;
    return LYNX_OK;
}

int lynx_destroy(lynx_ctx* c) {
    if (!c) return LYNX_OK;
    const bool used = c->cublas != nullptr;  // the device was touched by this context
    if (used) {
        cudaSetDevice(c->device);
        if (c->stream) cudaStreamSynchronize(c->stream);
        else cudaDeviceSynchronize();
    }
    for (auto& b : c->wbuf) b.release();
    for (auto& b : c->cvt) b.release();
    for (auto& b : c->lz) b.release();
    for (auto& b : c->nl_bufs) b.release();
    c->alpha.release();
    c->v32.release();
    c->Ms.release();
    c->Hs.release();
    c->eigd.release();
    c->solver_work.release();
    c->info.release();
    c->io_psi.release();
    c->io_v.release();
    c->vpad64.release();
    c->vpad32.release();
    if (c->err_h) cudaFreeHost(c->err_h);
    if (c->res_h) cudaFreeHost(c->res_h);
    if (c->in_flight) cudaEventDestroy(c->in_flight);
    c->gwork.release();
    c->rwork.release();
    c->nlW.release();
    c->xsbuf[0].release();
    c->xsbuf[1].release();
    c->gradbuf[0].release();
    c->gradbuf[1].release();
    c->fpart.release();
    c->fwork.release();
    if (c->copy_stream) cudaStreamDestroy(c->copy_stream);
    for (cudaEvent_t e : c->kt)
        if (e) cudaEventDestroy(e);
    for (auto& b : c->nl_layout_bufs) b.release();
    for (auto& kv : c->nl_maps) {
        kv.second.ptmap.release();
        kv.second.rowstart.release();
    }
    for (DevBuf* b : {&c->cplx_work, &c->dens_w, &c->dens_part, &c->vwork, &c->vzero, &c->vones, &c->dotw, &c->xcwork, &c->fft_sym,
                      &c->fft_z})
        b->release();
    if (c->fft_ready) {
        cufftDestroy(c->fft_fwd);
        cufftDestroy(c->fft_inv);
    }
    if (c->cublas) cublasDestroy(c->cublas);
    if (c->cusolver) cusolverDnDestroy(c->cusolver);
    delete c;
    return LYNX_OK;
}

int lynx_set_stream(lynx_ctx* c, void* stream) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (c->pending && s != c->stream) {
        LYNX_CUDA_TRY(cudaSetDevice(c->device));
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        LYNX_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
        // (recorded work is ordered by whoever replays it)
        if (cap == cudaStreamCaptureStatusNone) LYNX_CUDA_TRY(cudaStreamWaitEvent(s, c->in_flight, 0));
    }
    c->stream = s;
    return LYNX_OK;
}

int lynx_grid_info(const lynx_ctx* c, int* nd, double* dV, double* maxeig) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    if (nd) *nd = c->Nd;
    if (dV) *dV = c->dV;
    if (maxeig) *maxeig = c->maxeig;
    return LYNX_OK;
}

int lynx_stencil_coeffs(const lynx_ctx* c, double* d2x, double* d2y, double* d2z, double* d2xy, double* d2xz,
                        double* d2yz, double* d1x, double* d1y, double* d1z) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    auto cp = [&](double* dst, const std::vector<double>& v) {
        if (dst) std::memcpy(dst, v.data(), v.size() * sizeof(double));
    };
    cp(d2x, c->D2x);
    cp(d2y, c->D2y);
    cp(d2z, c->D2z);
    cp(d2xy, c->D2xy);
    cp(d2xz, c->D2xz);
    cp(d2yz, c->D2yz);
    cp(d1x, c->D1x);
    cp(d1y, c->D1y);
    cp(d1z, c->D1z);
    return LYNX_OK;
}

int lynx_set_nonlocal(lynx_ctx* c, int n_img, const int* img_atom, const int* img_ndc, const double* img_shift,
                      const int* gpos, const double* chi, int n_atom, const int* atom_nproj, const double* gamma) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    LYNX_TRY(activate(c));
    for (auto& b : c->nl_bufs) b.release();
    c->nl_bufs.clear();
    for (auto& b : c->nl_layout_bufs) b.release();
    c->nl_layout_bufs.clear();
    c->nl_layouts.clear();
    for (auto& kv : c->nl_maps) {
        kv.second.ptmap.release();
        kv.second.rowstart.release();
    }
    c->nl_maps.clear();
    c->h_gpos.clear();
    c->h_pt_grid.clear();
    c->nl = NLDev();
    c->has_nl = false;
    c->img_shift.clear();
    if (n_img == 0) return LYNX_OK;
    LYNX_CHECK_ARG(n_img > 0 && n_atom > 0, "counts must be positive");
    LYNX_CHECK_ARG(img_atom && img_ndc && img_shift && gpos && chi && atom_nproj && gamma, "null table");
    // per-atom projector offsets and image lists
    std::vector<int> poff(n_atom + 1, 0), nproj(atom_nproj, atom_nproj + n_atom);
    int max_np = 0;
    for (int a = 0; a < n_atom; ++a) {
        LYNX_CHECK_ARG(nproj[a] >= 0, "negative projector count");
        poff[a + 1] = poff[a] + nproj[a];
        max_np = std::max(max_np, nproj[a]);
    }
    std::vector<int> img_ptr(n_atom + 1, 0), img_list(n_img);
    std::vector<long long> goff(n_img), choff(n_img);
    long long tot = 0, totchi = 0;
    for (int i = 0; i < n_img; ++i) {
        LYNX_CHECK_ARG(img_atom[i] >= 0 && img_atom[i] < n_atom, "image atom index out of range");
        LYNX_CHECK_ARG(img_ndc[i] >= 0, "negative image point count");
        goff[i] = tot;
        choff[i] = totchi;
        tot += img_ndc[i];
        totchi += (long long)img_ndc[i] * nproj[img_atom[i]];
        img_ptr[img_atom[i] + 1]++;
    }
    for (int a = 0; a < n_atom; ++a) img_ptr[a + 1] += img_ptr[a];
    {
        std::vector<int> fill(img_ptr.begin(), img_ptr.end() - 1);
        for (int i = 0; i < n_img; ++i) img_list[fill[img_atom[i]]++] = i;  // image order preserved per atom
    }
    for (long long k = 0; k < tot; ++k)
        LYNX_CHECK_ARG(gpos[k] >= 0 && gpos[k] < c->Nd, "grid position out of range");
    // CSR over distinct grid points, entries in (image, local index) order.
    std::vector<long long> keys(tot);
    {
        long long k = 0;
        for (int i = 0; i < n_img; ++i)
            for (int l = 0; l < img_ndc[i]; ++l, ++k) keys[k] = ((long long)gpos[k] << 32) | (unsigned)k;
    }
    std::sort(keys.begin(), keys.end());
    std::vector<int> pt_grid, pt_ptr, ent_img(tot), ent_loc(tot);
    std::vector<int> owner_img(tot), owner_loc(tot);
    {
        long long k = 0;
        for (int i = 0; i < n_img; ++i)
            for (int l = 0; l < img_ndc[i]; ++l, ++k) {
                owner_img[k] = i;
                owner_loc[k] = l;
            }
    }
    for (long long s = 0; s < tot; ++s) {
        const int g = (int)(keys[s] >> 32);
        const long long k = keys[s] & 0xFFFFFFFFLL;
        if (pt_grid.empty() || pt_grid.back() != g) {
            pt_grid.push_back(g);
            pt_ptr.push_back((int)s);
        }
        ent_img[s] = owner_img[k];
        ent_loc[s] = owner_loc[k];
    }
    pt_ptr.push_back((int)tot);
    // Greedy colouring of the images: two images that share a grid point get different
    // colours, so the register-tiled scatter can run one colour class per launch with a single
    // writer per output element.  Images are coloured in index order (deterministic).
    std::vector<int> color(n_img, -1), color_img;
    int n_colors = 0;
    {
        std::vector<std::vector<int>> adj(n_img);
        for (size_t p = 0; p + 1 < pt_ptr.size(); ++p)
            for (int u = pt_ptr[p]; u < pt_ptr[p + 1]; ++u)
                for (int v = u + 1; v < pt_ptr[p + 1]; ++v)
                    if (ent_img[u] != ent_img[v]) {
                        adj[ent_img[u]].push_back(ent_img[v]);
                        adj[ent_img[v]].push_back(ent_img[u]);
                    }
        for (int i = 0; i < n_img; ++i) {
            unsigned long long used = 0;
            for (int j : adj[i])
                if (color[j] >= 0 && color[j] < 64) used |= 1ull << color[j];
            const int cl = (~used) ? __builtin_ctzll(~used) : 64;
            color[i] = cl;
            n_colors = std::max(n_colors, cl + 1);
        }
        if (n_colors <= kNLMaxColors) {
            for (int k = 0; k < n_colors; ++k)
                for (int i = 0; i < n_img; ++i)
                    if (color[i] == k) color_img.push_back(i);
        } else {
            n_colors = 0;
        }
    }
    std::vector<float> chi32(totchi);
    for (long long k = 0; k < totchi; ++k) chi32[k] = (float)chi[k];
    // upload
    auto up = [&](const void* src, size_t bytes, void** dst) -> int {
        c->nl_bufs.emplace_back();
        DevBuf& b = c->nl_bufs.back();
        LYNX_TRY(upload_table(c, b, src, bytes));
        *dst = b.p;
        return LYNX_OK;
    };
    c->nl_bufs.reserve(36);
    NLDev& d = c->nl;
    d.n_atom = n_atom;
    d.n_img = n_img;
    d.n_pts = (int)pt_grid.size();
    d.max_np = max_np;
    d.total_proj = poff[n_atom];
    LYNX_TRY(up(img_ptr.data(), img_ptr.size() * 4, (void**)&d.atom_img_ptr));
    LYNX_TRY(up(img_list.data(), img_list.size() * 4, (void**)&d.atom_img_list));
    LYNX_TRY(up(nproj.data(), nproj.size() * 4, (void**)&d.atom_nproj));
    LYNX_TRY(up(poff.data(), poff.size() * 4, (void**)&d.atom_poff));
    LYNX_TRY(up(gamma, (size_t)poff[n_atom] * 8, (void**)&d.gamma));
    LYNX_TRY(up(img_atom, (size_t)n_img * 4, (void**)&d.img_atom));
    LYNX_TRY(up(img_ndc, (size_t)n_img * 4, (void**)&d.img_ndc));
    LYNX_TRY(up(goff.data(), goff.size() * 8, (void**)&d.img_goff));
    LYNX_TRY(up(choff.data(), choff.size() * 8, (void**)&d.img_chi_off));
    std::vector<double> ph(2 * n_img, 0.0);
    for (int i = 0; i < n_img; ++i) ph[2 * i] = 1.0;
    LYNX_TRY(up(ph.data(), ph.size() * 8, (void**)&d.img_phase));
    LYNX_TRY(up(gpos, (size_t)tot * 4, (void**)&d.gpos));
    LYNX_TRY(up(chi, (size_t)totchi * 8, (void**)&d.chi64));
    LYNX_TRY(up(chi32.data(), (size_t)totchi * 4, (void**)&d.chi32));
    LYNX_TRY(up(pt_grid.data(), pt_grid.size() * 4, (void**)&d.pt_grid));
    LYNX_TRY(up(pt_ptr.data(), pt_ptr.size() * 4, (void**)&d.pt_ptr));
    LYNX_TRY(up(ent_img.data(), ent_img.size() * 4, (void**)&d.ent_img));
    LYNX_TRY(up(ent_loc.data(), ent_loc.size() * 4, (void**)&d.ent_loc));
    d.n_colors = n_colors;
    {
        // compact numbering: distinct points in grid order; every entry its own point
        d.compact = ((long long)pt_grid.size() == tot);
        if (d.compact) {
            std::vector<int> ent_pt(tot), pt_meta(2 * tot);
            std::vector<double> cp64((size_t)max_np * tot, 0.0);
            std::vector<float> cp32((size_t)max_np * tot, 0.0f);
            for (long long s2 = 0; s2 < tot; ++s2) {
                const long long k = keys[s2] & 0xFFFFFFFFLL;  // entry (image-major) of point s2
                ent_pt[k] = (int)s2;
                const int im = owner_img[k], l = owner_loc[k], a = img_atom[im];
                pt_meta[2 * s2] = poff[a];
                pt_meta[2 * s2 + 1] = nproj[a];
                for (int j = 0; j < nproj[a]; ++j) {
                    const double v = chi[choff[im] + (long long)j * img_ndc[im] + l];
                    cp64[(size_t)j * tot + s2] = v;
                    cp32[(size_t)j * tot + s2] = (float)v;
                }
            }
            LYNX_TRY(up(ent_pt.data(), ent_pt.size() * 4, (void**)&d.ent_pt));
            LYNX_TRY(up(pt_meta.data(), pt_meta.size() * 4, (void**)&d.pt_meta));
            {
                // expansion tiles: distinct atoms of every kExpTilePts consecutive points
                const long long ntile = (tot + kExpTilePts - 1) / kExpTilePts;
                std::vector<std::vector<int>> tatoms(ntile);
                std::vector<unsigned char> slot(tot);
                int amax = 0;
                for (long long t = 0; t < ntile; ++t) {
                    auto& at = tatoms[t];
                    for (long long s2 = t * kExpTilePts; s2 < std::min<long long>(tot, (t + 1) * kExpTilePts); ++s2) {
                        const long long k = keys[s2] & 0xFFFFFFFFLL;
                        const int a = img_atom[owner_img[k]];
                        auto f = std::find(at.begin(), at.end(), a);
                        if (f == at.end()) {
                            at.push_back(a);
                            f = at.end() - 1;
                        }
                        slot[s2] = (unsigned char)(f - at.begin());
                    }
                    amax = std::max(amax, (int)at.size());
                }
                std::vector<int> flat((size_t)ntile * amax, -1);
                for (long long t = 0; t < ntile; ++t)
                    std::copy(tatoms[t].begin(), tatoms[t].end(), flat.begin() + t * amax);
                d.exp_amax = amax;
                LYNX_TRY(up(flat.data(), flat.size() * 4, (void**)&d.exp_tile_atoms));
                LYNX_TRY(up(slot.data(), slot.size(), (void**)&d.pt_slot));
            }
            LYNX_TRY(up(cp64.data(), cp64.size() * 8, (void**)&d.chi_pt64));
            LYNX_TRY(up(cp32.data(), cp32.size() * 4, (void**)&d.chi_pt32));
        }
    }
    if (n_colors > 0) {
        for (int k = 0, o = 0; k < n_colors; ++k) {
            d.color_off[k] = o;
            for (int i = 0; i < n_img; ++i) o += (color[i] == k);
            d.color_off[k + 1] = o;
        }
        LYNX_TRY(up(color_img.data(), color_img.size() * 4, (void**)&d.color_img));
        std::vector<int> tiles;  // (image, first point) pairs, colour by colour
        for (int k = 0; k < n_colors; ++k) {
            d.color_toff[k] = (int)(tiles.size() / 2);
            for (int q = d.color_off[k]; q < d.color_off[k + 1]; ++q)
                for (int g0 = 0; g0 < img_ndc[color_img[q]]; g0 += kNLTilePts) {
                    tiles.push_back(color_img[q]);
                    tiles.push_back(g0);
                }
            d.color_toff[k + 1] = (int)(tiles.size() / 2);
        }
        LYNX_TRY(up(tiles.data(), tiles.size() * 4, (void**)&d.color_tiles));
    }
    c->img_shift.assign(img_shift, img_shift + 3 * n_img);
    c->h_gpos.assign(gpos, gpos + tot);
    c->h_pt_grid = pt_grid;
    c->has_nl = true;
    return update_nl_phases(c);
}

int lynx_set_kpoint(lynx_ctx* c, const double* k) {
    LYNX_CHECK_ARG(c != nullptr && k != nullptr, "null pointer");
    LYNX_TRY(activate(c));
    for (int d = 0; d < 3; ++d) c->kpt[d] = k[d];
    return update_nl_phases(c);
}

int lynx_hamiltonian_apply(lynx_ctx* c, const double* psi, const double* veff, double* y, int ncol, int ld,
                           double cs) {
    LYNX_CHECK_ARG(c && psi && veff && y, "null pointer");
    LYNX_CHECK_ARG(ncol >= 0, "negative ncol");
    LYNX_TRY(activate(c));
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    const double* Vl = nullptr;
    LYNX_TRY(veff_layout<double>(c, veff, c->nx, &Vl));
    LYNX_TRY(cheb_step<double>(c, c->nx, psi, l, nullptr, 0, y, l, Vl, ncol, 1.0, cs, 0.0, false));
    return check_errflag(c);
}

int lynx_hamiltonian_apply_kpt(lynx_ctx* c, const double* psi, const double* veff, double* y, int ncol, int ld,
                               double cs) {
    LYNX_CHECK_ARG(c && psi && veff && y, "null pointer");
    LYNX_CHECK_ARG(ncol >= 0, "negative ncol");
    LYNX_TRY(activate(c));
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    const double* Vl = nullptr;
    LYNX_TRY(veff_layout<double>(c, veff, c->nx, &Vl));
    LYNX_TRY(cheb_step<double2>(c, c->nx, reinterpret_cast<const double2*>(psi), l, nullptr, 0,
                                reinterpret_cast<double2*>(y), l, Vl, ncol, 1.0, cs, 0.0, true));
    return check_errflag(c);
}

int lynx_nonlocal_apply(lynx_ctx* c, const double* psi, double* hpsi, int ncol, int ld) {
    LYNX_CHECK_ARG(c && psi && hpsi, "null pointer");
    LYNX_CHECK_ARG(ncol > 0, "ncol must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    if (!c->has_nl) return LYNX_OK;
    LYNX_TRY(activate(c));
    const int ncolp = ((ncol + kNLColBlock - 1) / kNLColBlock) * kNLColBlock;
    LYNX_TRY(c->alpha.ensure(sizeof(double) * (size_t)c->nl.total_proj * ncolp));
    LYNX_TRY(launch_nl_gather<double>(c->nl, psi, l, ncol, c->alpha.as<double>(), ncolp, c->dV, c->stream,
                                      nl_few_atoms<double>(c->nl, ncol)));
    LYNX_TRY(launch_nl_scatter<double, double>(c->nl, hpsi, l, ncol, c->alpha.as<double>(), ncolp, 1.0, c->stream));
    return leave_in_flight(c);
}

int lynx_nonlocal_apply_kpt(lynx_ctx* c, const double* psi, double* hpsi, int ncol, int ld) {
    LYNX_CHECK_ARG(c && psi && hpsi, "null pointer");
    LYNX_CHECK_ARG(ncol > 0, "ncol must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    if (!c->has_nl) return LYNX_OK;
    LYNX_TRY(activate(c));
    const int ncolp = ((ncol + kNLColBlock - 1) / kNLColBlock) * kNLColBlock;
    LYNX_TRY(c->alpha.ensure(sizeof(double2) * (size_t)c->nl.total_proj * ncolp));
    LYNX_TRY(launch_nl_gather<double2>(c->nl, reinterpret_cast<const double2*>(psi), l, ncol,
                                       c->alpha.as<double2>(), ncolp, c->dV, c->stream,
                                       nl_few_atoms<double2>(c->nl, ncol)));
    LYNX_TRY(launch_nl_scatter<double2, double>(c->nl, reinterpret_cast<double2*>(hpsi), l, ncol,
                                                c->alpha.as<double2>(), ncolp, 1.0, c->stream));
    return leave_in_flight(c);
}

static int filter_entry(lynx_ctx* c, const double* X, double* Y, const double* veff, int ncol, int ld, double lc,
                        double emin, double emax, int degree, int precision, bool cplx) {
    LYNX_CHECK_ARG(c && X && Y && veff, "null pointer");
    LYNX_CHECK_ARG(ncol > 0 && degree >= 1, "ncol and degree must be positive");
    LYNX_CHECK_ARG(precision == LYNX_PREC_FP64 || precision == LYNX_PREC_MIXED, "unknown precision");
    LYNX_CHECK_ARG(emax > lc && emin < lc, "spectral bounds must satisfy eigmin < lambda_cutoff < eigmax");
    LYNX_TRY(activate(c));
    const long long Nd = c->Nd, l = ld > 0 ? ld : Nd;
    LYNX_CHECK_ARG(l >= Nd, "ld < Nd");
    long long ldb = 0;
    int nxp = 0;
    if (precision == LYNX_PREC_FP64) {
        if (cplx) {
            double2 *out = nullptr, *unused = nullptr;
            LYNX_TRY(run_filter64<double2>(c, reinterpret_cast<const double2*>(X), l, veff, ncol, lc, emin, emax,
                                           degree, true, false, &out, &unused, &ldb, &nxp));
            LYNX_TRY(repack<double2, double2>(c, reinterpret_cast<double2*>(Y), c->nx, l, out, nxp, ldb, ncol));
        } else {
            double *out = nullptr, *unused = nullptr;
            LYNX_TRY(run_filter64<double>(c, X, l, veff, ncol, lc, emin, emax, degree, false, false, &out, &unused,
                                          &ldb, &nxp));
            LYNX_TRY(repack<double, double>(c, Y, c->nx, l, out, nxp, ldb, ncol));
        }
    } else {
        if (cplx) {
            float2 *out = nullptr, *unused = nullptr;
            LYNX_TRY(run_filter32<float2, double2>(c, reinterpret_cast<const double2*>(X), l, veff, ncol, lc, emin,
                                                   emax, degree, true, false, &out, &unused, &ldb, &nxp));
            LYNX_TRY(repack<double2, float2>(c, reinterpret_cast<double2*>(Y), c->nx, l, out, nxp, ldb, ncol));
        } else {
            float *out = nullptr, *unused = nullptr;
            LYNX_TRY(run_filter32<float, double>(c, X, l, veff, ncol, lc, emin, emax, degree, false, false, &out,
                                                 &unused, &ldb, &nxp));
            LYNX_TRY(repack<double, float>(c, Y, c->nx, l, out, nxp, ldb, ncol));
        }
    }
    LYNX_TRY(check_errflag(c));
    return LYNX_OK;
}

int lynx_chebyshev_filter(lynx_ctx* c, const double* X, double* Y, const double* veff, int ncol, int ld, double lc,
                          double emin, double emax, int degree, int precision) {
    return filter_entry(c, X, Y, veff, ncol, ld, lc, emin, emax, degree, precision, false);
}

int lynx_chebyshev_filter_kpt(lynx_ctx* c, const double* X, double* Y, const double* veff, int ncol, int ld,
                              double lc, double emin, double emax, int degree, int precision) {
    return filter_entry(c, X, Y, veff, ncol, ld, lc, emin, emax, degree, precision, true);
}

int lynx_eigensolver_solve(lynx_ctx* c, double* psi, double* eig, const double* veff, int nband, int ld, double lc,
                           double emin, double emax, int degree, int precision, double* lc_out) {
    return solve_impl<double, float>(c, psi, eig, veff, nband, ld, lc, emin, emax, degree, precision, lc_out, false);
}

int lynx_eigensolver_solve_kpt(lynx_ctx* c, double* psi, double* eig, const double* veff, int nband, int ld,
                               double lc, double emin, double emax, int degree, int precision, double* lc_out) {
    return solve_impl<double2, float2>(c, reinterpret_cast<double2*>(psi), eig, veff, nband, ld, lc, emin, emax,
                                       degree, precision, lc_out, true);
}

int lynx_eigensolver_solve_host(lynx_ctx* c, double* psi, double* eig, const double* veff, int nband, int ld,
                                double lc, double emin, double emax, int degree, int precision, double* lc_out) {
    LYNX_CHECK_ARG(c && psi && eig && veff, "null pointer");
    LYNX_CHECK_ARG(nband > 0, "nband must be positive");
    LYNX_TRY(activate(c));
    const long long Nd = c->Nd, l = ld > 0 ? ld : Nd;
    LYNX_CHECK_ARG(l >= Nd, "ld < Nd");
    DevBuf& dpsi = c->io_psi;
    DevBuf& dv = c->io_v;
    LYNX_TRY(dpsi.ensure(sizeof(double) * (size_t)Nd * nband));
    LYNX_TRY(dv.ensure(sizeof(double) * (size_t)Nd));
    LYNX_CUDA_TRY(cudaMemcpyAsync(dv.p, veff, Nd * 8, cudaMemcpyHostToDevice, c->stream));
    // Mixed precision, real, pipelined layout: copy psi in column blocks (host_block columns, the
    // remainder last) on a second stream; the filter starts on a block as soon as it has landed
    // (see run_filter32).
    const bool pipelined = precision == LYNX_PREC_MIXED && pipe_capable<float>(c) && nband >= 256;
    std::vector<cudaEvent_t> evs;
    if (pipelined) {
        if (!c->copy_stream) LYNX_CUDA_TRY(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
        cudaEvent_t start;
        LYNX_CUDA_TRY(cudaEventCreateWithFlags(&start, cudaEventDisableTiming));
        evs.push_back(start);
        LYNX_CUDA_TRY(cudaEventRecord(start, c->stream));  // earlier work on the stream is done with dpsi
        LYNX_CUDA_TRY(cudaStreamWaitEvent(c->copy_stream, start, 0));
        c->col_blocks.clear();
        for (int b0 = 0; b0 < nband;) {
            const int nb = std::min(c->host_block, nband - b0);
            cudaEvent_t ev;
            LYNX_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
            evs.push_back(ev);
            LYNX_CUDA_TRY(cudaMemcpy2DAsync(dpsi.as<double>() + (size_t)b0 * Nd, Nd * 8, psi + (size_t)b0 * l, l * 8,
                                            Nd * 8, nb, cudaMemcpyHostToDevice, c->copy_stream));
            LYNX_CUDA_TRY(cudaEventRecord(ev, c->copy_stream));
            c->col_blocks.push_back({b0, ev});
            b0 += nb;
        }
    } else {
        LYNX_CUDA_TRY(cudaMemcpy2DAsync(dpsi.p, Nd * 8, psi, l * 8, Nd * 8, nband, cudaMemcpyHostToDevice, c->stream));
    }
    c->col_total = pipelined ? nband : 0;
    int st = lynx_eigensolver_solve(c, dpsi.as<double>(), eig, dv.as<double>(), nband, (int)Nd, lc, emin, emax,
                                    degree, precision, lc_out);
    c->col_blocks.clear();
    c->col_total = 0;
    if (pipelined) {
        cudaStreamSynchronize(c->copy_stream);
        for (cudaEvent_t e : evs) cudaEventDestroy(e);
    }
    if (st == LYNX_OK) {
        cudaError_t e = cudaMemcpy2DAsync(psi, l * 8, dpsi.p, Nd * 8, Nd * 8, nband, cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
        if (e != cudaSuccess) {
            set_error("copy-out failed: %s", cudaGetErrorString(e));
            st = LYNX_ERR_CUDA;
        }
    }
    cudaStreamSynchronize(c->stream);
    return st;
}

int lynx_time_filter_step(lynx_ctx* c, const double* veff, int ncol, int precision, int with_nonlocal, int reps,
                          double* ms_per_step) {
    LYNX_CHECK_ARG(c && veff && ms_per_step, "null pointer");
    LYNX_CHECK_ARG(ncol > 0 && reps > 0, "ncol and reps must be positive");
    LYNX_CHECK_ARG(precision == LYNX_PREC_FP64 || precision == LYNX_PREC_MIXED, "unknown precision");
    LYNX_TRY(activate(c));
    const size_t esz = precision == LYNX_PREC_FP64 ? sizeof(double) : sizeof(float);
    const int nxp = pipe_capable<float>(c) ? pipe_row_elems(c->nx, esz) : c->nx;
    const long long ldb = (long long)nxp * c->ny * c->nz;
    for (int i = 0; i < 3; ++i) LYNX_TRY(ensure_layout(c, c->wbuf[i], esz * (size_t)ldb * ncol, (int)(esz * 1000 + nxp)));
    const bool nl = c->has_nl;
    if (!with_nonlocal) c->has_nl = false;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int st = LYNX_OK;
    if (with_nonlocal == 2) {  // time the stencil kernel alone (its nonlocal term fused when it applies)
        for (int i = 0; i < 2; ++i)
            if (!c->kt[i]) LYNX_CUDA_TRY(cudaEventCreate(&c->kt[i]));
        c->kt_ms = 0.0;
        c->kt_n = 0;
    }
    const float* v32 = nullptr;
    const double* v64 = nullptr;
    if (precision == LYNX_PREC_MIXED) st = veff_layout<float>(c, veff, nxp, &v32);
    else st = veff_layout<double>(c, veff, nxp, &v64);
    for (int r = -1; r < reps && st == LYNX_OK; ++r) {  // r = -1: untimed warm-up launch
        if (r == 0) cudaEventRecord(e0, c->stream);
        c->time_stencil = (with_nonlocal == 2 && r >= 0);
        const int a = (r + 3) % 3, b = (r + 4) % 3, o = (r + 5) % 3;
        if (precision == LYNX_PREC_FP64)
            st = cheb_step<double>(c, nxp, c->wbuf[a].as<double>(), ldb, c->wbuf[b].as<double>(), ldb,
                                   c->wbuf[o].as<double>(), ldb, v64, ncol, 0.5, -0.1, -0.25, false);
        else
            st = cheb_step<float>(c, nxp, c->wbuf[a].as<float>(), ldb, c->wbuf[b].as<float>(), ldb,
                                  c->wbuf[o].as<float>(), ldb, v32, ncol, 0.5, -0.1, -0.25, false);
    }
    c->time_stencil = false;
    cudaEventRecord(e1, c->stream);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    c->has_nl = nl;
    if (st != LYNX_OK) return st;
    LYNX_CUDA_TRY(cudaGetLastError());
    LYNX_TRY(check_errflag(c));
    *ms_per_step = (with_nonlocal == 2) ? (c->kt_n ? c->kt_ms / c->kt_n : 0.0) : ms / reps;
    return LYNX_OK;
}

int lynx_lanczos_bounds(lynx_ctx* c, const double* veff, double tol, int max_iter, double* emin, double* emax) {
    return lanczos_impl<double>(c, veff, tol, max_iter, emin, emax, false);
}

int lynx_lanczos_bounds_kpt(lynx_ctx* c, const double* veff, double tol, int max_iter, double* emin, double* emax) {
    return lanczos_impl<double2>(c, veff, tol, max_iter, emin, emax, true);
}

int lynx_fermi_level(const double* eigs, const double* w, int n, double ne, double beta, int smearing, double* ef) {
    LYNX_CHECK_ARG(eigs && w && ef, "null pointer");
    LYNX_CHECK_ARG(n > 0, "no eigenvalues for the Fermi level search");
    LYNX_CHECK_ARG(beta > 0, "beta must be positive");
    double emin = eigs[0], emax = eigs[0];
    for (int i = 1; i < n; ++i) {
        emin = std::min(emin, eigs[i]);
        emax = std::max(emax, eigs[i]);
    }
    auto resid = [&](double x) {
        double s = 0;
        for (int i = 0; i < n; ++i) s += w[i] * smear(eigs[i] - x, beta, smearing);
        return s - ne;
    };
    double a = emin - 10.0 / beta, b = emax + 10.0 / beta;
    if (resid(a) * resid(b) > 0) {
        a = emin - 100.0 / beta;
        b = emax + 100.0 / beta;
        if (resid(a) * resid(b) > 0) {
            set_error("cannot bracket the Fermi level");
            return LYNX_ERR_BRACKET;
        }
    }
    *ef = brent_zero(resid, a, b, 1e-14, 200);
    return LYNX_OK;
}

int lynx_occupations(const double* eigs, int n, double ef, double beta, int smearing, double* occ) {
    LYNX_CHECK_ARG(eigs && occ, "null pointer");
    for (int i = 0; i < n; ++i) occ[i] = smear(eigs[i] - ef, beta, smearing);
    return LYNX_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Nonlocal apply without device allocation.
//
// lynx_nonlocal_apply keeps its projector coefficients alpha in a context buffer that grows
// with cudaMalloc on first use.  Some callers must not allocate at that point: a host program
// that reserves its whole device-memory budget up front (cudaMalloc then fails or evicts its
// own pool), and code that interleaves the apply with latency-critical work on other streams
// (cudaFree synchronises the whole device, and cudaMalloc may).  This entry point keeps alpha
// in a fixed file-scope device array instead, so a call issues only kernel launches.
//
// Limits: alpha needs total_proj x ncolp doubles (ncolp = ncol rounded up to 32); requests
// larger than kNoAllocScratchBytes are rejected with LYNX_ERR_BAD_ARG (split the columns).
// The scratch array is shared by every context on a device: calls that overlap in time (two
// streams or two host threads on one device) race on it and must be serialised by the caller.
// The first call on a device resolves the array's address (cudaGetSymbolAddress, which also
// loads the module) and should be made once before any stream capture is begun.  The address is
// kept for the life of the process: after cudaDeviceReset (which frees every allocation and
// context of the process, so no lynx context survives it either) the library must be reloaded
// before this entry point is used again.  Nothing in the scratch needs to start at zero: the
// gather writes every alpha element the scatter reads.
// ---------------------------------------------------------------------------------------------
namespace {
constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;  // 8 MiB = 1 Mi doubles
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
constexpr int kNoAllocMaxDevices = 64;
std::atomic<void*> g_noalloc_addr[kNoAllocMaxDevices];

int noalloc_scratch(int device, void** out) {
    if (device < 0 || device >= kNoAllocMaxDevices) {
        set_error("device index %d out of range for the no-allocation scratch", device);
        return LYNX_ERR_BAD_ARG;
    }
    void* p = g_noalloc_addr[device].load(std::memory_order_acquire);
    if (!p) {
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) {
            cudaGetLastError();
            set_error("cudaGetSymbolAddress(no-allocation scratch) failed: %s", cudaGetErrorString(e));
            return LYNX_ERR_CUDA;
        }
        g_noalloc_addr[device].store(p, std::memory_order_release);
    }
    *out = p;
    return LYNX_OK;
}
}  // namespace

static ForceGeom force_geom(const lynx_ctx* c) {
    ForceGeom g{c->nx, c->ny, c->nz, c->R, c->orth, {c->D1x.data(), c->D1y.data(), c->D1z.data()},
                {c->dx, c->dy, c->dz}, {}, {}};
    std::copy(c->uvec, c->uvec + 9, g.uvec);
    if (!c->orth) mat3_inverse(c->uvec, g.ui);  // Cartesian gradients: D_cart = uvec^-1 D_lattice
    return g;
}

// Nonlocal forces (src/physics/Forces.cpp:509-797): projections of psi and of its FD derivative along
// each lattice direction, reduced per atom with the occupations (forces.cu).
template <typename T>
int nonlocal_force_impl(lynx_ctx* c, const T* psi, int nband, int ld, const double* occ, double spn, double efac,
                        double* force, double* energy, bool use_k) {
    LYNX_CHECK_ARG(c && psi && occ && force, "null pointer");
    LYNX_CHECK_ARG(nband > 0, "nband must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    if (!c->has_nl) {
        if (energy) *energy = 0.0;
        return LYNX_OK;
    }
    LYNX_TRY(activate(c));
    const int na = c->nl.n_atom;
    LYNX_TRY(c->fpart.ensure(sphere_work_bytes(na, nband, false)));
    LYNX_TRY(c->fwork.ensure(sizeof(double) * ((size_t)nband + 4 * (size_t)na)));
    double* docc = c->fwork.as<double>();
    double* dforce = docc + nband;  // [na][3], then the energies [na]
    LYNX_CUDA_TRY(cudaMemcpyAsync(docc, occ, sizeof(double) * nband, cudaMemcpyHostToDevice, c->stream));
    T phl[3], phr[3];
    ghost_phases<T>(c, use_k, phl, phr);
    LYNX_TRY(launch_sphere_terms<T>(c->nl, force_geom(c), psi, l, nband, phl, phr, nullptr, docc, -spn, efac, c->dV,
                                    false, c->fpart.as<double>(), dforce, dforce + 3 * na, c->stream));
    std::vector<double> res(4 * (size_t)na);
    LYNX_CUDA_TRY(cudaMemcpyAsync(res.data(), dforce, sizeof(double) * res.size(), cudaMemcpyDeviceToHost, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    std::copy(res.begin(), res.begin() + 3 * na, force);
    if (energy) {
        double e = 0.0;
        for (int a = 0; a < na; ++a) e += res[3 * (size_t)na + a];
        *energy = e;
    }
    return LYNX_OK;
}

extern "C" int lynx_nonlocal_force(lynx_ctx* c, const double* psi, int nband, int ld, const double* occ, double occfac,
                                   double* force, double* energy_nl) {
    return nonlocal_force_impl<double>(c, psi, nband, ld, occ, 2.0 * occfac, occfac, force, energy_nl, false);
}

extern "C" int lynx_nonlocal_force_kpt(lynx_ctx* c, const double* psi_z, int nband, int ld, const double* occ,
                                       double spn_fac_wk, double* force, double* energy_nl) {
    return nonlocal_force_impl<double2>(c, reinterpret_cast<const double2*>(psi_z), nband, ld, occ, spn_fac_wk,
                                        0.5 * spn_fac_wk, force, energy_nl, true);
}

// Kinetic and nonlocal stress of one (spin, k-point) block, un-normalised (Voigt xx, xy, xz, yy,
// yz, zz), with of = occfac (Gamma) or spn_fac_wk / 2 (k-point):
//   stress_k[ab]  = -of dV sum_n g_n Re <D_a psi_n, D_b psi_n>       (Cartesian FD gradients)
//   stress_nl[ab] = -2 of sum_n g_n sum_j Gamma_j Re(conj(alpha_nj) beta^ab_nj) - delta_ab E_nl
//   beta^ab = dV sum_img e^{-ik.R} chi (r - R_img)_b D_a psi,  E_nl = of sum g Gamma |alpha|^2
// (src/physics/Stress.cpp:1041-1784; the GPU path's assembly src/physics/GPUForce.cu:471-680).
// The gradients are formed where they are used (forces.cu); the sums over bands run on the device, the
// sum over atoms on the host, each in a fixed order.
template <typename T>
int stress_impl(lynx_ctx* c, const T* psi, int nband, int ld, const double* occ, double of, const double* img_pos,
                double* stress_k, double* stress_nl, bool use_k) {
    LYNX_CHECK_ARG(c && psi && occ && stress_k && stress_nl, "null pointer");
    LYNX_CHECK_ARG(nband > 0, "nband must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    LYNX_CHECK_ARG(!c->has_nl || img_pos, "image positions are required when projectors are set");
    if (!c->orth) {
        const double* u = c->uvec;
        const double det = u[0] * (u[4] * u[8] - u[5] * u[7]) - u[1] * (u[3] * u[8] - u[5] * u[6]) +
                           u[2] * (u[3] * u[7] - u[4] * u[6]);
        LYNX_CHECK_ARG(std::fabs(det) > 1e-14, "singular lattice");
    }
    LYNX_TRY(activate(c));
    const int na = c->has_nl ? c->nl.n_atom : 0;
    const ForceGeom g = force_geom(c);
    LYNX_TRY(c->fpart.ensure(std::max(kinetic_work_bytes(g, nband, ScalarOf<T>::cplx), sphere_work_bytes(na, nband, true))));
    const size_t npos = c->has_nl ? 3 * (size_t)c->nl.n_img : 0;
    LYNX_TRY(c->fwork.ensure(sizeof(double) * ((size_t)nband + npos + 7 * (size_t)na + 6)));
    double* docc = c->fwork.as<double>();
    double* dpos = docc + nband;
    double* dres = dpos + npos;  // kinetic [6], then [na][6], then the energies [na]
    LYNX_CUDA_TRY(cudaMemcpyAsync(docc, occ, sizeof(double) * nband, cudaMemcpyHostToDevice, c->stream));
    if (npos)
        LYNX_CUDA_TRY(cudaMemcpyAsync(dpos, img_pos, sizeof(double) * npos, cudaMemcpyHostToDevice, c->stream));
    T phl[3], phr[3];
    ghost_phases<T>(c, use_k, phl, phr);
    bool phased = ScalarOf<T>::cplx;
    for (int d = 0; d < 3; ++d) phased |= c->bc[d] != LYNX_BC_PERIODIC;
    LYNX_TRY(launch_kinetic<T>(g, psi, l, nband, phl, phr, phased, docc, -of * c->dV, c->fpart.as<double>(), dres,
                               c->stream));
    if (na)
        LYNX_TRY(launch_sphere_terms<T>(c->nl, g, psi, l, nband, phl, phr, dpos, docc, -2.0 * of, of, c->dV, true,
                                        c->fpart.as<double>(), dres + 6, dres + 6 + 6 * na, c->stream));
    std::vector<double> res(6 + 7 * (size_t)na);
    LYNX_CUDA_TRY(cudaMemcpyAsync(res.data(), dres, sizeof(double) * res.size(), cudaMemcpyDeviceToHost, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    double enl = 0.0;
    for (int a = 0; a < na; ++a) enl += res[6 + 6 * (size_t)na + a];
    for (int v = 0; v < 6; ++v) {
        stress_k[v] = res[v];
        double sum = 0.0;
        for (int a = 0; a < na; ++a) sum += res[6 + (size_t)a * 6 + v];
        stress_nl[v] = c->has_nl ? sum - ((v == 0 || v == 3 || v == 5) ? enl : 0.0) : 0.0;
    }
    return LYNX_OK;
}

extern "C" int lynx_kinetic_nonlocal_stress(lynx_ctx* c, const double* psi, int nband, int ld, const double* occ,
                                            double occfac, const double* img_pos, double* stress_k,
                                            double* stress_nl) {
    return stress_impl<double>(c, psi, nband, ld, occ, occfac, img_pos, stress_k, stress_nl, false);
}

extern "C" int lynx_kinetic_nonlocal_stress_kpt(lynx_ctx* c, const double* psi_z, int nband, int ld,
                                                const double* occ, double spn_fac_wk, const double* img_pos,
                                                double* stress_k, double* stress_nl) {
    return stress_impl<double2>(c, reinterpret_cast<const double2*>(psi_z), nband, ld, occ, 0.5 * spn_fac_wk, img_pos,
                                stress_k, stress_nl, true);
}

extern "C" int lynx_randomize_orbitals(lynx_ctx* c, double* psi, int nband, int ld, unsigned long long seed,
                                       int is_complex) {
    LYNX_CHECK_ARG(c && psi, "null pointer");
    LYNX_CHECK_ARG(nband > 0, "nband must be positive");
    LYNX_CHECK_ARG(ld == 0 || ld == c->Nd, "the start orbitals fill contiguous columns: ld must be Nd (or 0)");
    LYNX_TRY(activate(c));
    curandGenerator_t g = nullptr;
    if (curandCreateGenerator(&g, CURAND_RNG_PSEUDO_DEFAULT) != CURAND_STATUS_SUCCESS) {
        set_error("curandCreateGenerator failed");
        return LYNX_ERR_CUDA;
    }
    const size_t n = (size_t)c->Nd * nband * (is_complex ? 2 : 1);
    curandStatus_t r = curandSetStream(g, c->stream);
    if (r == CURAND_STATUS_SUCCESS) r = curandSetPseudoRandomGeneratorSeed(g, seed);
    if (r == CURAND_STATUS_SUCCESS) r = curandGenerateUniformDouble(g, psi, n);
    curandDestroyGenerator(g);
    if (r != CURAND_STATUS_SUCCESS) {
        set_error("cuRAND uniform generation failed (status %d)", (int)r);
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

extern "C" int lynx_randomize_orbitals_all(lynx_ctx* c, double** psi, int nspin_local, int spin_start, int nkpts,
                                           int nband, int is_complex) {
    LYNX_CHECK_ARG(c && psi, "null pointer");
    LYNX_CHECK_ARG(nband > 0 && nspin_local > 0 && nkpts > 0, "block counts must be positive");
    const int nsk = nspin_local * nkpts;
    for (int i = 0; i < nsk; ++i) LYNX_CHECK_ARG(psi[i] != nullptr, "null block pointer");
    LYNX_TRY(activate(c));
    curandGenerator_t g = nullptr;
    if (curandCreateGenerator(&g, CURAND_RNG_PSEUDO_DEFAULT) != CURAND_STATUS_SUCCESS) {
        set_error("curandCreateGenerator failed");
        return LYNX_ERR_CUDA;
    }
    const size_t n = (size_t)c->Nd * nband * (is_complex ? 2 : 1);
    curandStatus_t r = curandSetStream(g, c->stream);
    for (int i = 0; i < nsk && r == CURAND_STATUS_SUCCESS; ++i) {
        const int s = i / nkpts;
        const unsigned long long seed = (unsigned long long)(spin_start + s) * 1000ULL + (unsigned long long)i * 13ULL + 1ULL;
        r = curandSetPseudoRandomGeneratorSeed(g, seed);
        if (r == CURAND_STATUS_SUCCESS) r = curandGenerateUniformDouble(g, psi[i], n);
    }
    curandDestroyGenerator(g);
    if (r != CURAND_STATUS_SUCCESS) {
        set_error("cuRAND uniform generation failed (status %d)", (int)r);
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

extern "C" int lynx_eigensolver_solve_batch(lynx_ctx** ctxs, int nb, double** psi, double** eig,
                                            const double** veff, const int* nband, const int* ld,
                                            const double* lambda_cutoff, const double* eigmin, const double* eigmax,
                                            const int* is_kpt, int degree, int precision,
                                            double* lambda_cutoff_out) {
    LYNX_CHECK_ARG(nb >= 0, "negative batch size");
    if (nb == 0) return LYNX_OK;
    LYNX_CHECK_ARG(ctxs && psi && eig && veff && nband && ld && lambda_cutoff && eigmin && eigmax && is_kpt,
                   "null pointer");
    for (int i = 0; i < nb; ++i) LYNX_CHECK_ARG(ctxs[i] != nullptr, "null context in the batch");
    std::vector<int> st(nb, LYNX_OK);
    std::vector<std::string> msg(nb);
    // problems that share a context run one after another on the same thread
    std::map<lynx_ctx*, std::vector<int>> groups;
    for (int i = 0; i < nb; ++i) groups[ctxs[i]].push_back(i);
    auto run = [&](const std::vector<int>& idx) {
        for (int i : idx) {
            double* lco = lambda_cutoff_out ? lambda_cutoff_out + i : nullptr;
            st[i] = is_kpt[i] ? lynx_eigensolver_solve_kpt(ctxs[i], psi[i], eig[i], veff[i], nband[i], ld[i],
                                                           lambda_cutoff[i], eigmin[i], eigmax[i], degree, precision,
                                                           lco)
                              : lynx_eigensolver_solve(ctxs[i], psi[i], eig[i], veff[i], nband[i], ld[i],
                                                       lambda_cutoff[i], eigmin[i], eigmax[i], degree, precision, lco);
            if (st[i] != LYNX_OK) msg[i] = lynx_last_error();
        }
    };
    std::vector<std::thread> th;
    th.reserve(groups.size());
    for (auto& g : groups) th.emplace_back(run, std::cref(g.second));
    for (auto& t : th) t.join();
    for (int i = 0; i < nb; ++i)
        if (st[i] != LYNX_OK) {
            set_error("batch problem %d: %s", i, msg[i].c_str());
            return st[i];
        }
    return LYNX_OK;
}

extern "C" int lynx_set_option(lynx_ctx* c, int option, int value) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    switch (option) {
        case LYNX_OPT_AUTOTUNE: c->autotune = value != 0; return LYNX_OK;
        case LYNX_OPT_FUSE_NONLOCAL: c->fuse_nl = value != 0; return LYNX_OK;
        case LYNX_OPT_TC_RAYLEIGH_RITZ: c->no_tc_gram = value == 0; return LYNX_OK;
        case LYNX_OPT_COMPACT_GATHER: c->fuse_compact_gather = value != 0; return LYNX_OK;
        case LYNX_OPT_POISSON_DIRECT: c->poisson_direct = value != 0; return LYNX_OK;
        case LYNX_OPT_STENCIL_SHAPE: c->force_shape = value > 0 ? value - 1 : -1; return LYNX_OK;
        case LYNX_OPT_HOST_COPY_BLOCK: c->host_block = value > 0 ? value : 128; return LYNX_OK;
        default: set_error("unknown option %d", option); return LYNX_ERR_BAD_ARG;
    }
}

extern "C" int lynx_gram_mixed(lynx_ctx* c, const float* Y, const float* HY, long long ld, long long rows, int n,
                               double scale, double* Ms, double* Hs) {
    LYNX_CHECK_ARG(c && Y && HY && Ms && Hs, "null pointer");
    LYNX_CHECK_ARG(n > 0 && rows > 0 && ld >= rows, "need n > 0, rows > 0 and ld >= rows");
    LYNX_TRY(activate(c));
    const GramPlan plan = gram_plan(rows, n);
    LYNX_TRY(c->gwork.ensure(plan.work_bytes));
    LYNX_TRY(c->info.ensure(3 * sizeof(int)));
    LYNX_TRY(ensure_errflag(c));
    int* bad = c->info.as<int>() + 2;
    LYNX_CUDA_TRY(cudaMemsetAsync(bad, 0, sizeof(int), c->stream));
    LYNX_TRY(launch_gram_i8(Y, HY, ld, rows, n, scale, plan, c->gwork.p, c->gwork.bytes, Ms, Hs, c->err_d,
                            bad, c->stream));
    int h = 0;
    LYNX_CUDA_TRY(cudaMemcpyAsync(&h, bad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    LYNX_TRY(check_errflag(c));  // synchronises the stream
    if (h) {
        set_error("NaN or Inf in the FP32 blocks of the Gram products");
        return LYNX_ERR_NONFINITE;
    }
    return LYNX_OK;
}

extern "C" int lynx_rotate_mixed(lynx_ctx* c, const float* Y, long long ld, long long rows, const double* Ms,
                                 const double* W, int n, double* psi, long long ldp) {
    LYNX_CHECK_ARG(c && Y && Ms && W && psi, "null pointer");
    LYNX_CHECK_ARG(n > 0 && rows > 0 && ld >= rows && ldp >= rows, "need n > 0, rows > 0, ld >= rows, ldp >= rows");
    if (!rot_supported(n)) {
        set_error("the tensor-core rotation takes at most %d states", (int)(200 * 1024 / (33 * sizeof(float))));
        return LYNX_ERR_UNSUPPORTED;
    }
    LYNX_TRY(activate(c));
    const RotPlan rp = rot_plan(rows, n);
    LYNX_TRY(c->rwork.ensure(rp.work_bytes));
    LYNX_TRY(ensure_errflag(c));
    LYNX_TRY(launch_colexp(Ms, n, c->rwork.p, rp, rows, c->stream));
    LYNX_TRY(launch_rot_i8(Y, ld, rows, 1, 1, W, n, rp, c->rwork.p, c->rwork.bytes, psi, ldp, c->err_d,
                           c->stream));
    return check_errflag(c);
}

extern "C" int lynx_selftest_wait_timeout(lynx_ctx* c, int spins) {
    LYNX_CHECK_ARG(c != nullptr, "null context");
    LYNX_CHECK_ARG(spins >= 1 && spins <= (1 << 20), "spins must lie in [1, 2^20]");
    LYNX_TRY(activate(c));
    LYNX_TRY(ensure_errflag(c));
    wait_selftest_kernel<<<1, 32, 0, c->stream>>>(spins, c->err_d);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return check_errflag(c);
}

extern "C" int lynx_electron_density(lynx_ctx* c, const double* psi, int nband, int ld, const double* occ,
                                     double weight, double* rho, int is_complex, int accumulate) {
    LYNX_CHECK_ARG(c && psi && occ && rho, "null pointer");
    LYNX_CHECK_ARG(nband > 0, "nband must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    LYNX_TRY(activate(c));
    std::vector<double> w(nband);
    for (int n = 0; n < nband; ++n) w[n] = (occ[n] < 1e-16) ? 0.0 : weight * occ[n];
    LYNX_TRY(c->dens_w.ensure(sizeof(double) * nband));
    LYNX_CUDA_TRY(cudaMemcpyAsync(c->dens_w.p, w.data(), sizeof(double) * nband, cudaMemcpyHostToDevice, c->stream));
    if (is_complex)
        LYNX_TRY(launch_density<double2>(reinterpret_cast<const double2*>(psi), l, c->Nd, nband,
                                         c->dens_w.as<double>(), rho, accumulate != 0, c->stream));
    else
        LYNX_TRY(launch_density<double>(psi, l, c->Nd, nband, c->dens_w.as<double>(), rho, accumulate != 0,
                                        c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));  // w is a host temporary
    return LYNX_OK;
}

extern "C" int lynx_pair_density(lynx_ctx* c, const double* u, const double* v, int ncol, int ld, double* out) {
    LYNX_CHECK_ARG(c && u && v && out, "null pointer");
    LYNX_CHECK_ARG(ncol > 0, "ncol must be positive");
    const long long l = ld > 0 ? ld : c->Nd, nd = c->Nd;
    LYNX_CHECK_ARG(l >= nd, "ld < Nd");
    LYNX_TRY(activate(c));
    const bool pairs = nd % 2 == 0 && l % 2 == 0 && aligned16(u) && aligned16(v);
    if (pairs)
        pair_density_kernel<2><<<(unsigned)((nd / 2 + 127) / 128), 128, 0, c->stream>>>(u, v, l, nd, ncol, out);
    else
        pair_density_kernel<1><<<(unsigned)((nd + 127) / 128), 128, 0, c->stream>>>(u, v, l, nd, ncol, out);
    count_launch();
    LYNX_CUDA_TRY(cudaGetLastError());
    return LYNX_OK;
}

extern "C" int lynx_eigensolver_solve_density(lynx_ctx* c, double* psi, double* eig, const double* veff, int nband,
                                              int ld, double lc, double emin, double emax, int degree, int precision,
                                              double* lc_out, double nelectron, double beta, int smearing,
                                              double weight, double* rho, double* ef_out) {
    LYNX_CHECK_ARG(c && rho, "null pointer");
    LYNX_CHECK_ARG(beta > 0 && weight > 0 && nelectron > 0, "nelectron, beta and weight must be positive");
    c->dens = lynx_ctx::DensityReq();
    c->dens.on = true;
    c->dens.nelectron = nelectron;
    c->dens.beta = beta;
    c->dens.smearing = smearing;
    c->dens.weight = weight;
    c->dens.rho = rho;
    int st = solve_impl<double, float>(c, psi, eig, veff, nband, ld, lc, emin, emax, degree, precision, lc_out, false);
    const bool fused = c->dens.done;
    c->dens.on = false;
    if (st != LYNX_OK) return st;
    if (!fused) {  // FP64 pass (or more states than the tensor-core rotation takes): separate kernel
        std::vector<double> wt(nband, weight), occ(nband);
        double ef = 0.0;
        LYNX_TRY(lynx_fermi_level(eig, wt.data(), nband, nelectron, beta, smearing, &ef));
        LYNX_TRY(lynx_occupations(eig, nband, ef, beta, smearing, occ.data()));
        c->dens.ef = ef;
        LYNX_TRY(lynx_electron_density(c, psi, nband, ld, occ.data(), weight, rho, 0, 0));
    }
    if (ef_out) *ef_out = c->dens.ef;
    return LYNX_OK;
}

// ---------------------------------------------------------------------------
// Effective potential (src/physics/EffectivePotential.cpp:44-177): GGA-PBE exchange-correlation,
// the AAR Poisson solve and V_eff = V_xc + phi, FP64 on one field of Nd points.
// ---------------------------------------------------------------------------
namespace {

GradGeom grad_geom(const lynx_ctx* c) {
    GradGeom g{};
    g.nx = c->nx;
    g.ny = c->ny;
    g.nz = c->nz;
    g.R = c->R;
    for (int d = 0; d < 3; ++d) g.periodic[d] = c->bc[d] == LYNX_BC_PERIODIC ? 1 : 0;
    for (int p = 0; p <= c->R; ++p) {
        g.D1[0][p] = c->D1x[p];
        g.D1[1][p] = c->D1y[p];
        g.D1[2][p] = c->D1z[p];
    }
    return g;
}

// -Lap x on one field, the Poisson operator (src/solvers/PoissonSolver.cpp:248-253, a = -1): the
// Chebyshev step kernel with V = 0, a = 2 (a * (-1/2) Lap), b = d = 0 and the nonlocal term off.
int neg_laplacian(lynx_ctx* c, const double* x, double* out) {
    LYNX_TRY(ensure_zeroed(c, c->vzero, sizeof(double) * (size_t)c->Nd));
    const bool nl = c->has_nl;
    c->has_nl = false;
    const int st = cheb_step<double>(c, c->nx, x, c->Nd, nullptr, 0, out, c->Nd, c->vzero.as<double>(), 1, 2.0, 0.0,
                                     0.0, false);
    c->has_nl = nl;
    return st;
}

// Gaussian elimination with partial pivoting on a small dense system, rows whose pivot is below
// 1e-14 in magnitude skipped in both sweeps: the rule of src/core/NumericalMethods.cpp:84-113,
// which the AAR step relies on when its history columns are nearly dependent.  A: n x n row-major
// (overwritten), b: right-hand side, overwritten by the solution.
void solve_small(std::vector<double>& A, std::vector<double>& b, int n) {
    for (int k = 0; k < n; ++k) {
        int piv = k;
        for (int i = k + 1; i < n; ++i)
            if (std::fabs(A[i * n + k]) > std::fabs(A[piv * n + k])) piv = i;
        if (piv != k) {
            for (int j = 0; j < n; ++j) std::swap(A[k * n + j], A[piv * n + j]);
            std::swap(b[k], b[piv]);
        }
        const double d = A[k * n + k];
        if (std::fabs(d) < 1e-14) continue;
        for (int i = k + 1; i < n; ++i) {
            const double f = A[i * n + k] / d;
            for (int j = k + 1; j < n; ++j) A[i * n + j] -= f * A[k * n + j];
            b[i] -= f * b[k];
        }
    }
    for (int k = n - 1; k >= 0; --k) {
        if (std::fabs(A[k * n + k]) < 1e-14) continue;
        for (int j = k + 1; j < n; ++j) b[k] -= A[k * n + j] * b[j];
        b[k] /= A[k * n + k];
    }
}

int dots(lynx_ctx* c, const DotList& L, double* out) {
    LYNX_TRY(c->dotw.ensure(dots_work_bytes()));
    return launch_dots(L, c->Nd, c->dotw.p, out, c->stream);
}

// AAR iteration for -Lap phi = b (src/solvers/PoissonSolver.cpp:43-159, CPU semantics: b is
// used as given, phi is the start and the result).  m history columns, Anderson every p-th
// step, Richardson weight omega, Anderson weight beta, Jacobi weight -1 / (D2x[0] + D2y[0] +
// D2z[0]) (:17-37); stops when ||b - A phi|| <= tol ||b||, checked after Anderson steps only.
int poisson_aar(lynx_ctx* c, const double* b, double* phi, double tol, int max_iter, int* iters) {
    const int m = 7, p = 6;
    const double omega = 0.6, beta = 0.6;
    const long long N = c->Nd;
    const double diag = c->D2x[0] + c->D2y[0] + c->D2z[0];
    const double w = std::fabs(diag) < 1e-14 ? 1.0 : -1.0 / diag;
    LYNX_TRY(c->vwork.ensure(sizeof(double) * (size_t)N * (5 + 2 * m)));
    double* base = c->vwork.as<double>();
    double* r = base;
    double* f = base + N;
    double* f_old = base + 2 * N;
    double* x_old = base + 3 * N;
    double* Ax = base + 4 * N;
    double* X = base + 5 * N;
    double* F = X + (size_t)m * N;
    LYNX_CUDA_TRY(cudaMemsetAsync(f_old, 0, sizeof(double) * N, c->stream));
    LYNX_CUDA_TRY(cudaMemcpyAsync(x_old, phi, sizeof(double) * N, cudaMemcpyDeviceToDevice, c->stream));
    DotList L{};
    L.count = 1;
    L.u[0] = b;
    L.v[0] = b;
    double bn2 = 0.0;
    LYNX_TRY(dots(c, L, &bn2));
    const double abs_tol = tol * std::sqrt(bn2);
    LYNX_TRY(neg_laplacian(c, phi, Ax));
    LYNX_TRY(launch_sub(b, Ax, r, N, c->stream));
    double rn = abs_tol + 1.0;
    int it = 0;
    while (rn > abs_tol && it < max_iter) {
        const int col = it > 0 ? (it - 1) % m : -1;
        LYNX_TRY(launch_aar_pre(r, phi, x_old, f, f_old, col >= 0 ? X + (size_t)col * N : nullptr,
                                col >= 0 ? F + (size_t)col * N : nullptr, w, N, c->stream));
        AarGamma g{};
        if ((it + 1) % p == 0 && it > 0) {
            const int cols = std::min(it, m);
            DotList D{};
            int k = 0;
            for (int i = 0; i < cols; ++i) {
                D.u[k] = F + (size_t)i * N;
                D.v[k++] = f;
            }
            for (int i = 0; i < cols; ++i)
                for (int j = 0; j <= i; ++j) {
                    D.u[k] = F + (size_t)i * N;
                    D.v[k++] = F + (size_t)j * N;
                }
            D.count = k;
            double vals[kMaxDots];
            LYNX_TRY(dots(c, D, vals));
            std::vector<double> A((size_t)cols * cols), gam(vals, vals + cols);
            for (int i = 0, q = cols; i < cols; ++i)
                for (int j = 0; j <= i; ++j, ++q) A[i * cols + j] = A[j * cols + i] = vals[q];
            solve_small(A, gam, cols);
            g.cols = cols;
            for (int i = 0; i < cols; ++i) g.g[i] = gam[i];
            LYNX_TRY(launch_aar_update(phi, x_old, f, X, F, g, beta, N, c->stream));
            LYNX_TRY(neg_laplacian(c, phi, Ax));
            LYNX_TRY(launch_sub(b, Ax, r, N, c->stream));
            DotList R{};
            R.count = 1;
            R.u[0] = r;
            R.v[0] = r;
            double rr = 0.0;
            LYNX_TRY(dots(c, R, &rr));
            rn = std::sqrt(rr);
        } else {
            g.cols = 0;
            LYNX_TRY(launch_aar_update(phi, x_old, f, X, F, g, omega, N, c->stream));
            LYNX_TRY(neg_laplacian(c, phi, Ax));
            LYNX_TRY(launch_sub(b, Ax, r, N, c->stream));
        }
        ++it;
    }
    if (iters) *iters = it;
    LYNX_TRY(check_errflag(c));
    return LYNX_OK;
}

// Periodic cells: -Lap phi = b solved exactly in Fourier space.  The FD operator (with the
// mixed-derivative terms of a non-orthogonal cell) is a circular convolution with its own impulse
// response g = A delta_0, so phi_hat = b_hat / g_hat, the mean mode set to zero.  g comes from the
// same stencil kernel the AAR iteration applies, so phi solves the same discrete equation, to
// rounding, instead of to the iteration's tolerance; b must have zero mean.
int poisson_direct(lynx_ctx* c, const double* b, double* phi) {
    const long long N = c->Nd;
    const long long nh = (long long)c->nz * c->ny * (c->nx / 2 + 1);
    auto fft_check = [](cufftResult r, const char* what) -> int {
        if (r == CUFFT_SUCCESS) return LYNX_OK;
        set_error("%s failed (cuFFT status %d)", what, (int)r);
        return r == CUFFT_ALLOC_FAILED ? LYNX_ERR_OOM : LYNX_ERR_CUDA;
    };
    LYNX_TRY(c->fft_z.ensure(sizeof(double2) * (size_t)nh));
    double2* z = c->fft_z.as<double2>();
    if (!c->fft_ready) {
        LYNX_TRY(fft_check(cufftPlan3d(&c->fft_fwd, c->nz, c->ny, c->nx, CUFFT_D2Z), "cufftPlan3d"));
        if (cufftPlan3d(&c->fft_inv, c->nz, c->ny, c->nx, CUFFT_Z2D) != CUFFT_SUCCESS) {
            cufftDestroy(c->fft_fwd);
            set_error("cufftPlan3d (inverse) failed");
            return LYNX_ERR_CUDA;
        }
        c->fft_ready = true;
        LYNX_TRY(c->fft_sym.ensure(sizeof(double) * (size_t)nh));
        LYNX_TRY(c->vwork.ensure(sizeof(double) * (size_t)N * 2));
        double* d = c->vwork.as<double>();
        double* g = d + N;
        const double one = 1.0;
        LYNX_CUDA_TRY(cudaMemsetAsync(d, 0, sizeof(double) * N, c->stream));
        LYNX_CUDA_TRY(cudaMemcpyAsync(d, &one, sizeof(double), cudaMemcpyHostToDevice, c->stream));
        LYNX_TRY(neg_laplacian(c, d, g));
        LYNX_TRY(fft_check(cufftSetStream(c->fft_fwd, c->stream), "cufftSetStream"));
        LYNX_TRY(fft_check(cufftExecD2Z(c->fft_fwd, g, z), "cufftExecD2Z"));
        LYNX_TRY(launch_inv_symbol(z, c->fft_sym.as<double>(), nh, c->stream));
        LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));  // `one` is a host temporary
    }
    LYNX_TRY(fft_check(cufftSetStream(c->fft_fwd, c->stream), "cufftSetStream"));
    LYNX_TRY(fft_check(cufftSetStream(c->fft_inv, c->stream), "cufftSetStream"));
    LYNX_TRY(fft_check(cufftExecD2Z(c->fft_fwd, const_cast<double*>(b), z), "cufftExecD2Z"));
    LYNX_TRY(launch_spec_scale(z, c->fft_sym.as<double>(), 1.0 / (double)N, nh, c->stream));
    LYNX_TRY(fft_check(cufftExecZ2D(c->fft_inv, z, phi), "cufftExecZ2D"));
    count_launch(3);
    return LYNX_OK;
}

// Sum of a field (the global mean over Nd points is sum / Nd).
int field_sum(lynx_ctx* c, const double* x, double* sum) {
    if (c->vones.bytes < sizeof(double) * (size_t)c->Nd) {
        LYNX_TRY(ensure_zeroed(c, c->vzero, sizeof(double) * (size_t)c->Nd));
        LYNX_TRY(c->vones.ensure(sizeof(double) * (size_t)c->Nd));
        LYNX_TRY(launch_add_shift(c->vzero.as<double>(), nullptr, -1.0, 1.0, c->vones.as<double>(), c->Nd, c->stream));
    }
    DotList L{};
    L.count = 1;
    L.u[0] = x;
    L.v[0] = c->vones.as<double>();
    return dots(c, L, sum);
}

}  // namespace

// Gradient, functional and flux of the exchange-correlation part (asynchronous); *f: the three flux
// fields that launch_div_sub takes.  With rhs also the Poisson right-hand side.
static int xc_terms(lynx_ctx* c, const double* rho, const double* rho_core, double* vxc, double* exc,
                    double* dxcdgrho, const double* rho_b, double* rhs, double** f) {
    const long long N = c->Nd;
    // scratch: 3 flux fields, the core-corrected density, the Poisson right-hand side
    LYNX_TRY(c->xcwork.ensure(sizeof(double) * (size_t)N * 5));
    *f = c->xcwork.as<double>();
    const double* rx = rho;
    if (rho_core) {
        double* t = *f + 3 * N;
        LYNX_TRY(launch_rho_xc(rho, rho_core, t, N, c->stream));
        rx = t;
    }
    XcMetric mt{};
    mt.orth = c->orth ? 1 : 0;
    for (int i = 0; i < 9; ++i) mt.L[i] = c->lapcT[i];
    return launch_grad_pbe(rx, grad_geom(c), mt, *f, *f + N, *f + 2 * N, vxc, exc, dxcdgrho, rho, rho_b, rhs,
                           c->stream);
}

extern "C" int lynx_xc_gga_pbe(lynx_ctx* c, const double* rho, const double* rho_core, double* vxc, double* exc,
                               double* dxcdgrho) {
    LYNX_CHECK_ARG(c && rho && vxc && exc, "null pointer");
    LYNX_CHECK_ARG(c->nx > c->R && c->ny > c->R && c->nz > c->R, "grid smaller than the FD half-width");
    LYNX_TRY(activate(c));
    const long long N = c->Nd;
    double* f = nullptr;
    LYNX_TRY(xc_terms(c, rho, rho_core, vxc, exc, dxcdgrho, nullptr, nullptr, &f));
    LYNX_TRY(launch_div_sub(vxc, grad_geom(c), f, f + N, f + 2 * N, nullptr, nullptr, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return LYNX_OK;
}

extern "C" int lynx_poisson_solve(lynx_ctx* c, const double* rhs, double* phi, double tol, int max_iter, int* iters) {
    LYNX_CHECK_ARG(c && rhs && phi, "null pointer");
    LYNX_CHECK_ARG(tol > 0.0, "tol must be positive");
    LYNX_CHECK_ARG(c->nx > c->R && c->ny > c->R && c->nz > c->R, "grid smaller than the FD half-width");
    LYNX_TRY(activate(c));
    LYNX_TRY(poisson_aar(c, rhs, phi, tol, max_iter > 0 ? max_iter : 3000, iters));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return LYNX_OK;
}

extern "C" int lynx_effective_potential(lynx_ctx* c, const double* rho, const double* rho_b, const double* rho_core,
                                        double poisson_tol, double* veff, double* vxc, double* exc, double* phi,
                                        int* poisson_iters) {
    LYNX_CHECK_ARG(c && rho && veff && vxc && exc && phi, "null pointer");
    LYNX_CHECK_ARG(poisson_tol > 0.0, "poisson_tol must be positive");
    LYNX_TRY(activate(c));
    const long long N = c->Nd;
    const bool periodic = c->bc[0] == LYNX_BC_PERIODIC && c->bc[1] == LYNX_BC_PERIODIC && c->bc[2] == LYNX_BC_PERIODIC;
    if (c->poisson_direct && periodic) {
        // No host step in between: the mean of the right-hand side and of phi is the Fourier mode that the
        // inverse symbol sets to zero, and V_eff is added up where the divergence is.
        LYNX_CHECK_ARG(c->nx > c->R && c->ny > c->R && c->nz > c->R, "grid smaller than the FD half-width");
        LYNX_TRY(c->xcwork.ensure(sizeof(double) * (size_t)N * 5));
        double* rhs = c->xcwork.as<double>() + 4 * N;
        double* f = nullptr;
        LYNX_TRY(xc_terms(c, rho, rho_core, vxc, exc, nullptr, rho_b, rhs, &f));
        LYNX_TRY(poisson_direct(c, rhs, phi));
        LYNX_TRY(launch_div_sub(vxc, grad_geom(c), f, f + N, f + 2 * N, phi, veff, c->stream));
        LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
        if (poisson_iters) *poisson_iters = 0;
        return LYNX_OK;
    }
    // 1. exchange-correlation
    LYNX_TRY(lynx_xc_gga_pbe(c, rho, rho_core, vxc, exc, nullptr));
    // 2. Poisson: rhs = 4 pi rho + 4 pi rho_b with its mean removed;
    //    the right-hand side is built in veff, which is written last (EffectivePotential.cpp:44-60)
    const double fpi = 4.0 * 3.14159265358979323846;
    LYNX_TRY(launch_add_shift(rho, rho_b, 0.0, fpi, veff, N, c->stream));
    double sum = 0.0;
    LYNX_TRY(field_sum(c, veff, &sum));
    LYNX_TRY(launch_add_shift(veff, nullptr, sum / (double)N, 1.0, veff, N, c->stream));
    LYNX_TRY(poisson_aar(c, veff, phi, poisson_tol, 3000, poisson_iters));
    // phi shifted to zero mean (EffectivePotential.cpp:64-70)
    LYNX_TRY(field_sum(c, phi, &sum));
    LYNX_TRY(launch_add_shift(phi, nullptr, sum / (double)N, 1.0, phi, N, c->stream));
    // 3. V_eff = V_xc + phi
    LYNX_TRY(launch_add_shift(vxc, phi, 0.0, 1.0, veff, N, c->stream));
    LYNX_CUDA_TRY(cudaStreamSynchronize(c->stream));
    return LYNX_OK;
}

extern "C" int lynx_nonlocal_apply_noalloc(lynx_ctx* c, const double* psi, double* hpsi, int ncol, int ld) {
    LYNX_CHECK_ARG(c && psi && hpsi, "null pointer");
    LYNX_CHECK_ARG(ncol > 0, "ncol must be positive");
    const long long l = ld > 0 ? ld : c->Nd;
    LYNX_CHECK_ARG(l >= c->Nd, "ld < Nd");
    if (!c->has_nl) return LYNX_OK;
    const int ncolp = ((ncol + kNLColBlock - 1) / kNLColBlock) * kNLColBlock;
    const size_t need = sizeof(double) * (size_t)c->nl.total_proj * (size_t)ncolp;
    if (need > kNoAllocScratchBytes) {
        set_error("no-allocation nonlocal apply needs %zu bytes of scratch for %d projectors x %d columns; "
                  "the limit is %zu bytes: apply fewer columns per call",
                  need, c->nl.total_proj, ncol, kNoAllocScratchBytes);
        return LYNX_ERR_BAD_ARG;
    }
    LYNX_CUDA_TRY(cudaSetDevice(c->device));
    void* scratch = nullptr;
    LYNX_TRY(noalloc_scratch(c->device, &scratch));
    double* alpha = static_cast<double*>(scratch);
    LYNX_TRY(launch_nl_gather<double>(c->nl, psi, l, ncol, alpha, ncolp, c->dV, c->stream,
                                      nl_few_atoms<double>(c->nl, ncol)));
    return launch_nl_scatter<double, double>(c->nl, hpsi, l, ncol, alpha, ncolp, 1.0, c->stream);
}
