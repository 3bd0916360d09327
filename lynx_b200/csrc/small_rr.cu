// Rayleigh-Ritz step of few states (N <= kSmallRRMax), FP64 arithmetic on blocks of any type:
//   Ms = dV Y^H Y, Hs = dV Y^H HY;  Ms = L L^H;  L^-1 Hs L^-H = Q e Q^H;  W = L^-H Q;  psi = Y W
// (src/solvers/EigenSolver.cpp:622-681).
//
// For 16 to 24 states the arithmetic is a few microseconds; as library calls the step is about 50
// launches (the products on one or two CTAs, the eigensolver a chain of tiny kernels): 0.75 ms of a
// 1.25 ms pass of Si8.  Here it is four launches: partial products over chunks of the points on
// every SM, their sum, one CTA that does all the subspace algebra in shared memory, and the rotation
// straight from the (padded) block into the caller's layout.  FP32 blocks are multiplied in FP64, so
// the products are those of the library path.
//
// The line at 40 states is what the register and task layout below holds.  Us a pass beyond its filter, 40
// states here against 41 by library (mixed: tensor-core) products, FP64 / mixed: 30^3 517 / 513 against
// 867 / 1022, 60^3 902 / 824 against 1136 / 1339, 90^3 1897 / 1784 against 1768 / 1878; at a k-point 20^3 605 / 593
// against 1241 / 1035, 60^3 2151 / 1429 against 9681 / 1853.
//
// Subspace eigenproblem: cyclic Jacobi rotations (Golub and Van Loan, Matrix Computations, sec. 8.5),
// N/2 disjoint pairs at a time (round-robin order); all 2 x 2 blocks of a round are updated at once,
// so a round is two barriers.  Converged when no off-diagonal entry exceeds 2^-54 of the norm.
#include <algorithm>

#include "kernels.h"
#include "lynx_common.cuh"
#include "stencil.cuh"

namespace lynxb {
namespace {

constexpr int kTilePts = 32;  // points per staged tile of the products
constexpr int kEigThreads = 512;
constexpr int kMaxSweeps = 40;

template <typename T> struct Wide;
template <> struct Wide<float> { using type = double; };
template <> struct Wide<double> { using type = double; };
template <> struct Wide<float2> { using type = double2; };
template <> struct Wide<double2> { using type = double2; };

__device__ __forceinline__ double widen(float v) { return v; }
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double2 widen(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 widen(double2 v) { return v; }
// acc + conj(a) b, a b, conj(a)
__device__ __forceinline__ double cmac(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ double2 cmac(double2 acc, double2 a, double2 b) {
    return make_double2(fma(a.y, b.y, fma(a.x, b.x, acc.x)), fma(-a.y, b.x, fma(a.x, b.y, acc.y)));
}
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double cj(double a) { return a; }
__device__ __forceinline__ double2 cj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double re(double a) { return a; }
__device__ __forceinline__ double re(double2 a) { return a.x; }
__device__ __forceinline__ double mod(double a) { return fabs(a); }
__device__ __forceinline__ double mod(double2 a) { return sqrt(fma(a.x, a.x, a.y * a.y)); }
// |a|, and e = a / |a| (1 for a = 0)
__device__ __forceinline__ double mod_phase(double a, double& e) {
    e = a < 0.0 ? -1.0 : 1.0;
    return fabs(a);
}
__device__ __forceinline__ double mod_phase(double2 a, double2& e) {
    const double s = fma(a.x, a.x, a.y * a.y);
    if (!(s > 0x1p-900)) return 0.0;
    const double r = rsqrt(s);
    e = make_double2(a.x * r, a.y * r);
    return s * r;
}
__device__ __forceinline__ bool fin(double a) { return isfinite(a); }
__device__ __forceinline__ bool fin(double2 a) { return isfinite(a.x) && isfinite(a.y); }
__device__ __forceinline__ double amax(double a) { return fabs(a); }
__device__ __forceinline__ double amax(double2 a) { return fmax(fabs(a.x), fabs(a.y)); }
__device__ __forceinline__ void set_re(double& a, double v) { a = v; }
__device__ __forceinline__ void set_re(double2& a, double v) { a = make_double2(v, 0.0); }
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// Partial products of one chunk of the points: part[chunk][0: Ms, 1: Hs][i + j N] (Ms: i <= j only
// read).  A thread owns 2 x 2 entries, so a point costs it four shared loads.
template <typename T>
__global__ void __launch_bounds__(256)
    small_gram_kernel(const T* __restrict__ Y, const T* __restrict__ H, long long ld, long long rows, int N,
                      long long chunk, typename Wide<T>::type* __restrict__ part) {
    using W = typename Wide<T>::type;
    constexpr int LD = kTilePts + 1;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int N2 = (N + 1) / 2;
    W* ys = reinterpret_cast<W*>(sm_raw);  // [2 N2][LD]
    W* hs = ys + (size_t)2 * N2 * LD;
    const long long r0 = (long long)blockIdx.x * chunk, r1 = min(rows, r0 + chunk);
    const int nt = N2 * N2 + N2 * (N2 + 1) / 2;  // Hs blocks, then the blocks of Ms on and above the diagonal
    constexpr int NQ = 3;                        // N <= 40: at most 610 blocks for 256 threads
    W acc[NQ][4];
    int bi[NQ], bj[NQ];
    const W* rhs[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int e = threadIdx.x + 256 * q;
        bi[q] = bj[q] = 0;
        rhs[q] = hs;
        if (e < N2 * N2) {
            bi[q] = e % N2;
            bj[q] = e / N2;
        } else if (e < nt) {
            int r = e - N2 * N2, j = 0;
            while (r > j) r -= ++j;
            bi[q] = r;
            bj[q] = j;
            rhs[q] = ys;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[q][u] = vzero(W());
    }
    for (long long p0 = r0; p0 < r1; p0 += kTilePts) {
        __syncthreads();
        for (int e = threadIdx.x; e < 2 * N2 * kTilePts; e += 256) {
            const int n = e / kTilePts, p = e % kTilePts;
            const bool ok = n < N && p0 + p < r1;
            ys[n * LD + p] = ok ? widen(Y[(long long)n * ld + p0 + p]) : vzero(W());
            hs[n * LD + p] = ok ? widen(H[(long long)n * ld + p0 + p]) : vzero(W());
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (threadIdx.x + 256 * q >= nt) break;
            const W* a = ys + 2 * bi[q] * LD;
            const W* b = rhs[q] + 2 * bj[q] * LD;
#pragma unroll 8
            for (int p = 0; p < kTilePts; ++p) {
                const W a0 = a[p], a1 = a[LD + p], b0 = b[p], b1 = b[LD + p];
                acc[q][0] = cmac(acc[q][0], a0, b0);
                acc[q][1] = cmac(acc[q][1], a1, b0);
                acc[q][2] = cmac(acc[q][2], a0, b1);
                acc[q][3] = cmac(acc[q][3], a1, b1);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int e = threadIdx.x + 256 * q;
        if (e >= nt) break;
        W* o = part + ((long long)blockIdx.x * 2 + (e < N2 * N2 ? 1 : 0)) * N * N;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = 2 * bi[q] + (u & 1), j = 2 * bj[q] + (u >> 1);
            if (i < N && j < N) o[i + j * N] = acc[q][u];
        }
    }
}

// Ms, Hs = dV * sum over the chunks, in order: eight lanes take every eighth chunk of one entry.
template <typename W>
__global__ void __launch_bounds__(256)
    small_reduce_kernel(const W* __restrict__ part, int nch, int N, double dV, W* __restrict__ Ms,
                        W* __restrict__ Hs) {
    const int e = (blockIdx.x * 256 + threadIdx.x) >> 3, l = threadIdx.x & 7;
    const int n2 = N * N;
    W s = vzero(W());
    const bool ok = e < 2 * n2 && (e >= n2 || e % N <= e / N);
    if (ok)
        for (int c = l; c < nch; c += 8) s = vadd(s, part[(long long)c * 2 * n2 + e]);
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) {
        if constexpr (ScalarOf<W>::cplx) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
        } else {
            s += __shfl_xor_sync(0xffffffffu, s, o);
        }
    }
    if (ok && l == 0) (e < n2 ? Ms : Hs)[e < n2 ? e : e - n2] = vscale(dV, s);
}

// All of the subspace algebra in one CTA.  info[0]: Cholesky, info[1]: eigensolver (> 0: failed),
// info[2]: a non-finite entry in Ms (upper) or Hs.  On success eig holds the ascending eigenvalues
// and Hs is overwritten by W (column-major).
template <typename W>
__global__ void __launch_bounds__(kEigThreads)
    small_eig_kernel(const W* __restrict__ Ms, W* __restrict__ Hs, int N, double* __restrict__ eig,
                     int* __restrict__ info) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int n2 = N * N, tid = threadIdx.x;
    const int NP = (N + 1) & ~1;  // players of the round robin (one idle when N is odd)
    W* L = reinterpret_cast<W*>(sm_raw);  // [i + j N], lower triangle of the factor
    W* A = L + n2;
    W* V = A + n2;
    W* ph = V + n2;                                   // [NP/2] phase of the pair's entry
    double* cs = reinterpret_cast<double*>(ph + NP / 2);  // [NP/2][2] cosine, sine
    double* dg = cs + NP;                             // [NP/2][3] new diagonal and off-diagonal entries
    double* red = dg + NP + NP / 2;                            // [kEigThreads / 32]
    int* pq = reinterpret_cast<int*>(red + kEigThreads / 32);  // [NP/2][2] rows of the pair (p < 0: idle)
    int* rank = pq + NP;                              // [N]
    __shared__ double big[kEigThreads / 32];
    __shared__ int bad, chol, moved;
    if (tid == 0) bad = chol = 0;
    __syncthreads();
    for (int e = tid; e < n2; e += kEigThreads) {
        const int i = e % N, j = e / N;
        const W m = i <= j ? Ms[e] : cj(Ms[j + i * N]);
        const W a = Hs[e], b = cj(Hs[j + i * N]);
        if (!fin(m) || !fin(a)) bad = 1;
        L[e] = m;
        A[e] = vscale(0.5, vadd(a, b));
        W one = vzero(W());
        if (i == j) {
            set_re(L[e], re(m));
            set_re(A[e], re(a));
            set_re(one, 1.0);
        }
        V[e] = one;
    }
    __syncthreads();
    if (bad) {
        if (tid == 0) info[2] = 1;
        return;
    }
    // Ms = L L^H, column by column (right-looking)
    for (int k = 0; k < N; ++k) {
        const double piv = re(L[k + k * N]);
        __syncthreads();
        if (!(piv > 0.0)) {  // the same value in every thread
            if (tid == 0) info[0] = k + 1;
            return;
        }
        const double r = sqrt(piv), ri = 1.0 / r;
        for (int i = k + tid; i < N; i += kEigThreads) {
            if (i == k) set_re(L[k + k * N], r);
            else L[i + k * N] = vscale(ri, L[i + k * N]);
        }
        __syncthreads();
        const int m = N - k - 1;
        for (int e = tid; e < m * m; e += kEigThreads) {
            const int i = k + 1 + e % m, j = k + 1 + e / m;
            if (i >= j) L[i + j * N] = sub(L[i + j * N], mul(L[i + k * N], cj(L[j + k * N])));
        }
        __syncthreads();
    }
    // A <- L^-1 A, then A <- A L^-H
    for (int k = 0; k < N; ++k) {
        const double ri = 1.0 / re(L[k + k * N]);
        for (int j = tid; j < N; j += kEigThreads) A[k + j * N] = vscale(ri, A[k + j * N]);
        __syncthreads();
        for (int e = tid; e < (N - k - 1) * N; e += kEigThreads) {
            const int i = k + 1 + e % (N - k - 1), j = e / (N - k - 1);
            A[i + j * N] = sub(A[i + j * N], mul(L[i + k * N], A[k + j * N]));
        }
        __syncthreads();
    }
    for (int k = 0; k < N; ++k) {
        const double ri = 1.0 / re(L[k + k * N]);
        for (int i = tid; i < N; i += kEigThreads) A[i + k * N] = vscale(ri, A[i + k * N]);
        __syncthreads();
        for (int e = tid; e < (N - k - 1) * N; e += kEigThreads) {
            const int j = k + 1 + e / N, i = e % N;
            A[i + j * N] = sub(A[i + j * N], mul(A[i + k * N], cj(L[j + k * N])));
        }
        __syncthreads();
    }
    // symmetric part, its norm and its largest entry
    double nrm = 0.0, top = 0.0;
    for (int e = tid; e < n2; e += kEigThreads) {
        const int i = e % N, j = e / N;
        if (i > j) continue;
        const W h = vscale(0.5, vadd(A[e], cj(A[j + i * N])));
        if (!fin(h)) bad = 1;
        A[e] = h;
        A[j + i * N] = cj(h);
        if (i == j) set_re(A[e], re(h));
        const double v = mod(h);
        nrm = fma(v, i == j ? v : 2.0 * v, nrm);
        top = fmax(top, amax(h));
    }
    auto sum_all = [&](double v) {  // over the CTA, in a fixed order
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((tid & 31) == 0) red[tid >> 5] = v;
        __syncthreads();
        v = 0.0;
        for (int w = 0; w < kEigThreads / 32; ++w) v += red[w];
        return v;
    };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    if ((tid & 31) == 0) big[tid >> 5] = top;
    nrm = sum_all(nrm);
    top = 0.0;
    for (int w = 0; w < kEigThreads / 32; ++w) top = fmax(top, big[w]);
    if (bad) {
        if (tid == 0) info[2] = 1;
        return;
    }
    // Entries whose squares leave the range of FP64 are scaled by a power of two, and the eigenvalues back.
    double up = 1.0;
    if (top > 0.0 && (top > 0x1p+400 || top < 0x1p-400)) {
        const int k = max(-1000, min(1000, ilogb(top)));
        up = ldexp(1.0, k);
        const double dn = ldexp(1.0, -k);
        double s = 0.0;
        __syncthreads();  // red is summed up again
        for (int e = tid; e < n2; e += kEigThreads) {
            A[e] = vscale(dn, A[e]);
            const double v = mod(A[e]);
            s = fma(v, v, s);
        }
        nrm = sum_all(s);
    }
    const double thr = 0x1p-54 * sqrt(nrm), inv = nrm > 0.0 ? rsqrt(nrm) : 0.0;
    // Jacobi sweeps.  A thread's tasks are the same in every round (2 x 2 blocks (P, Q) of A, then rows i of
    // V and pairs Q): their indices are worked out once.
    const int np2 = NP / 2;
    constexpr int NT = 3;  // N <= 40: 400 + 800 tasks
    int ta[NT], tb[NT];    // (P, Q), or (-1 - i, Q), or (0, -1): nothing
#pragma unroll
    for (int k = 0; k < NT; ++k) {
        const int w = tid + k * kEigThreads;
        ta[k] = 0;
        tb[k] = -1;
        if (w < np2 * np2) {
            ta[k] = w % np2;
            tb[k] = w / np2;
        } else if (w < np2 * np2 + np2 * N) {
            const int f = w - np2 * np2;
            ta[k] = -1 - f % N;
            tb[k] = f / N;
        }
    }
    bool done = false;
    for (int sweep = 0; sweep < kMaxSweeps && !done; ++sweep) {
        // done when nothing is left to rotate
        if (tid == 0) moved = 0;
        __syncthreads();
        for (int e = tid; e < n2; e += kEigThreads)
            if (e % N < e / N && mod(A[e]) > thr) moved = 1;
        __syncthreads();
        done = moved == 0;
        if (done) break;
        for (int rnd = 0; rnd < NP - 1; ++rnd) {
            __syncthreads();
            if (tid < np2) {
                int p = rnd + tid, q = rnd + NP - 1 - tid;  // round robin, modulo NP - 1
                if (p >= NP - 1) p -= NP - 1;
                if (q >= NP - 1) q -= NP - 1;
                if (tid == 0) p = NP - 1;
                if (p > q) {
                    const int s = p;
                    p = q;
                    q = s;
                }
                double c = 1.0, s = 0.0;
                W e = vzero(W());
                set_re(e, 1.0);
                const bool idle = q >= N;
                if (!idle) {
                    // t = tan of the angle that zeroes the entry, 2 m / (d + sign(d) sqrt(d^2 + 4 m^2)), d = aqq -
                    // app.  An FP32 angle does: the rotation is orthogonal to FP64 for any t, and what
                    // is left of the entry, 1e-7 of it, goes in the next sweep (FP64 divisions and square
                    // roots one after another were most of a round's time).
                    const W apq = A[p + q * N];
                    const double app = re(A[p + p * N]), aqq = re(A[q + q * N]);
                    const double m = mod_phase(apq, e), d = aqq - app;
                    dg[3 * tid] = app;
                    dg[3 * tid + 1] = aqq;
                    if (m > thr) {
                        const float ms = (float)(m * inv), ds = (float)(d * inv);
                        const double t = 2.0f * ms / (ds + copysignf(sqrtf(fmaf(ds, ds, 4.0f * ms * ms)), ds));
                        c = rsqrt(fma(t, t, 1.0));
                        s = t * c;
                        const double c2 = c * c;
                        dg[3 * tid] = fma(c2 * t, fma(t, d, -2.0 * m), app);
                        dg[3 * tid + 1] = fma(-c2 * t, fma(t, d, -2.0 * m), aqq);
                        dg[3 * tid + 2] = c2 * (m - t * fma(m, t, d));
                    } else {
                        set_re(e, 1.0);  // not rotated: no phase either
                    }
                }
                cs[2 * tid] = c;
                cs[2 * tid + 1] = idle ? 2.0 : s;  // 2: nothing to do for this pair
                ph[tid] = e;
                pq[2 * tid] = p;
                pq[2 * tid + 1] = q;
            }
            __syncthreads();
            // columns p' = c p - s e* q, q' = s p + c e* q, rows by the conjugate
#pragma unroll
            for (int k = 0; k < NT; ++k) {
                if (tb[k] < 0) break;
                if (ta[k] >= 0) {
                    const int P = ta[k], Q = tb[k];
                    const int p1 = pq[2 * P], q1 = pq[2 * P + 1], p2 = pq[2 * Q], q2 = pq[2 * Q + 1];
                    const bool v1 = q1 < N, v2 = q2 < N;
                    const double c1 = cs[2 * P], s1 = v1 ? cs[2 * P + 1] : 0.0;
                    const double c2 = cs[2 * Q], s2 = v2 ? cs[2 * Q + 1] : 0.0;
                    if (s1 == 0.0 && s2 == 0.0) continue;
                    if (P == Q) {
                        set_re(A[p1 + p1 * N], dg[3 * P]);
                        set_re(A[q1 + q1 * N], dg[3 * P + 1]);
                        set_re(A[p1 + q1 * N], dg[3 * P + 2]);
                        A[q1 + p1 * N] = A[p1 + q1 * N];
                        continue;
                    }
                    const W z = vzero(W());
                    const W app = A[p1 + p2 * N];
                    const W apq = v2 ? A[p1 + q2 * N] : z;
                    const W aqp = v1 ? A[q1 + p2 * N] : z;
                    const W aqq = v1 && v2 ? A[q1 + q2 * N] : z;
                    // columns
                    const W e2 = cj(ph[Q]);
                    const W xq = mul(apq, e2), yq = mul(aqq, e2);
                    const W b00 = sub(vscale(c2, app), vscale(s2, xq)), b01 = vadd(vscale(s2, app), vscale(c2, xq));
                    const W b10 = sub(vscale(c2, aqp), vscale(s2, yq)), b11 = vadd(vscale(s2, aqp), vscale(c2, yq));
                    // rows
                    const W e1 = ph[P];
                    const W r10 = mul(b10, e1), r11 = mul(b11, e1);
                    A[p1 + p2 * N] = sub(vscale(c1, b00), vscale(s1, r10));
                    if (v2) A[p1 + q2 * N] = sub(vscale(c1, b01), vscale(s1, r11));
                    if (v1) A[q1 + p2 * N] = vadd(vscale(s1, b00), vscale(c1, r10));
                    if (v1 && v2) A[q1 + q2 * N] = vadd(vscale(s1, b01), vscale(c1, r11));
                } else {
                    const int Q = tb[k], i = -1 - ta[k];
                    const int p2 = pq[2 * Q], q2 = pq[2 * Q + 1];
                    const double c2 = cs[2 * Q], s2 = cs[2 * Q + 1];
                    if (q2 >= N || s2 == 0.0) continue;
                    const W a = V[i + p2 * N], b = mul(V[i + q2 * N], cj(ph[Q]));
                    V[i + p2 * N] = sub(vscale(c2, a), vscale(s2, b));
                    V[i + q2 * N] = vadd(vscale(s2, a), vscale(c2, b));
                }
            }
        }
        __syncthreads();
    }
    if (!done) {
        if (tid == 0) info[1] = 1;
        return;
    }
    // ascending order (ties by index)
    for (int i = tid; i < N; i += kEigThreads) {
        const double v = re(A[i + i * N]);
        int r = 0;
        for (int j = 0; j < N; ++j) {
            const double u = re(A[j + j * N]);
            r += (u < v || (u == v && j < i)) ? 1 : 0;
        }
        rank[i] = r;
        eig[r] = up * v;
    }
    // V <- L^-H V
    for (int k = N - 1; k >= 0; --k) {
        const double ri = 1.0 / re(L[k + k * N]);
        __syncthreads();
        for (int j = tid; j < N; j += kEigThreads) V[k + j * N] = vscale(ri, V[k + j * N]);
        __syncthreads();
        for (int e = tid; e < k * N; e += kEigThreads) {
            const int i = e % k, j = e / k;
            V[i + j * N] = sub(V[i + j * N], mul(cj(L[k + i * N]), V[k + j * N]));
        }
    }
    __syncthreads();
    for (int e = tid; e < n2; e += kEigThreads) Hs[e % N + rank[e / N] * N] = V[e];
}

// psi(:, j) = sum_i Y(:, i) W(i, j), FP64 sums in the order of i; thread = one grid point x
// kRotCols columns.  psi stays as it is where the subspace algebra failed (info): W is not there then.
constexpr int kRotCols = 8;
template <typename T>
__global__ void __launch_bounds__(128)
    small_rotate_kernel(const T* __restrict__ Y, long long ld, int nx, int nxp, long long nd, int N,
                        const typename Wide<T>::type* __restrict__ W, const int* __restrict__ info,
                        typename Wide<T>::type* __restrict__ psi, long long ldp) {
    using D = typename Wide<T>::type;
    __shared__ D ws[kSmallRRMax * kRotCols];
    if (info[0] | info[1] | info[2]) return;
    const int j0 = blockIdx.y * kRotCols;
    for (int e = threadIdx.x; e < N * kRotCols; e += 128) {
        const int i = e / kRotCols, j = j0 + e % kRotCols;
        ws[e] = j < N ? W[i + j * N] : vzero(D());
    }
    __syncthreads();
    const long long r = (long long)blockIdx.x * 128 + threadIdx.x;
    if (r >= nd) return;
    const T* y = Y + r + (r / nx) * (nxp - nx);
    D acc[kRotCols];
#pragma unroll
    for (int c = 0; c < kRotCols; ++c) acc[c] = vzero(D());
#pragma unroll 4
    for (int i = 0; i < N; ++i) {
        const D v = cj(widen(y[(long long)i * ld]));
#pragma unroll
        for (int c = 0; c < kRotCols; ++c) acc[c] = cmac(acc[c], v, ws[i * kRotCols + c]);
    }
#pragma unroll
    for (int c = 0; c < kRotCols; ++c)
        if (j0 + c < N) psi[(long long)(j0 + c) * ldp + r] = acc[c];
}

int small_chunks(long long rows) { return (int)std::max<long long>(1, std::min<long long>(148, (rows + 63) / 64)); }

}  // namespace

bool small_rr_supported(int n) { return n <= kSmallRRMax; }

size_t small_rr_work_bytes(long long rows, int n, size_t wide) { return (size_t)small_chunks(rows) * 2 * n * n * wide; }

template <typename T>
int launch_small_rr(const T* Y, const T* HY, long long ld, long long rows, int nx, int nxp, long long nd, int n,
                    double dV, void* work, void* Ms, void* Hs, double* eig, int* info, void* psi, long long ldp,
                    cudaStream_t st) {
    using W = typename Wide<T>::type;
    const int nch = small_chunks(rows);
    const long long chunk = (rows + nch - 1) / nch;
    W* part = static_cast<W*>(work);
    W* ms = static_cast<W*>(Ms);
    W* hs = static_cast<W*>(Hs);
    const int np = (n + 1) & ~1;
    const size_t sg = sizeof(W) * (size_t)2 * np * (kTilePts + 1);
    LYNX_CUDA_TRY(smem_cap(small_gram_kernel<T>, sg));
    small_gram_kernel<T><<<nch, 256, sg, st>>>(Y, HY, ld, rows, n, chunk, part);
    small_reduce_kernel<W><<<(2 * n * n * 8 + 255) / 256, 256, 0, st>>>(part, nch, n, dV, ms, hs);
    const size_t se = sizeof(W) * ((size_t)3 * n * n + np / 2) + sizeof(double) * (2 * np + np / 2 + kEigThreads / 32) +
                      sizeof(int) * (np + n);
    LYNX_CUDA_TRY(smem_cap(small_eig_kernel<W>, se));
    small_eig_kernel<W><<<1, kEigThreads, se, st>>>(ms, hs, n, eig, info);
    dim3 grid((unsigned)((nd + 127) / 128), (n + kRotCols - 1) / kRotCols);
    small_rotate_kernel<T><<<grid, 128, 0, st>>>(Y, ld, nx, nxp, nd, n, hs, info, static_cast<W*>(psi), ldp);
    count_launch(4);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("small Rayleigh-Ritz launch failed: %s", cudaGetErrorString(e));
        return LYNX_ERR_CUDA;
    }
    return LYNX_OK;
}

#define LYNX_SMALL_INST(T)                                                                                        \
    template int launch_small_rr<T>(const T*, const T*, long long, long long, int, int, long long, int, double,   \
                                    void*, void*, void*, double*, int*, void*, long long, cudaStream_t);
LYNX_SMALL_INST(float)
LYNX_SMALL_INST(double)
LYNX_SMALL_INST(float2)
LYNX_SMALL_INST(double2)

}  // namespace lynxb
