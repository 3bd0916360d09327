// Host-side launch interfaces of the lynx_b200 kernels (implemented in the .cu files).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

namespace lynxb {

template <typename T> struct ScalarOf;

constexpr int kMaxR1 = 9;  // FD half-width bound + 1 (coefficient arrays 0..R)

// Geometry + FD coefficients of one cell for the fused stencil kernel.
struct StencilGeom {
    int nx, ny, nz;
    int R;               // FD half-width
    const double* D2x;   // FDn+1 scaled second-derivative coefficients (host)
    const double* D2y;
    const double* D2z;
};

// Mixed-derivative coefficients of a non-orthogonal cell (host arrays of R+1 values).
struct NonOrthGeom {
    int nx, ny, nz, R;
    const double* D1y;
    const double* D1z;
    const double* D2xy;
    const double* D2xz;
    const double* D2yz;
};
// out += a * (-1/2) * (mixed-derivative part of Lap x); gy, gz: scratch blocks like x (column
// stride ldg).  nonorth.cu.
// have_grads: gy and gz already hold the first derivatives of x (launch_direct_step).
template <typename T>
int launch_nonorth_terms(const NonOrthGeom& g, int nxp, const T* x, long long ldx, T* gy, T* gz, long long ldg, T* out,
                         long long ldout, int ncol, double a, const T* phl, const T* phr, cudaStream_t st,
                         bool have_grads = false);
// The Chebyshev step of complex blocks and small real ones, one thread per point (stencil_direct.cu,
// any half-width, row pitch and alignment).  ng (may be null): also write the first derivatives of x along y and z
// to gy and gz (column stride ldg).
constexpr int kDirectMaxNx = 512;  // longest rows of the direct step
template <typename T, typename S>
int launch_direct_step(const StencilGeom& g, int nxp, const T* x, long long ldx, const T* xold, long long ldo, T* out,
                       long long ldout, const S* V, int ncol, double a, double b, double d, const T* phl,
                       const T* phr, const NonOrthGeom* ng, T* gy, T* gz, long long ldg, cudaStream_t st);

// Centre coefficient of a Chebyshev step, -0.5 a (D2x[0] + D2y[0] + D2z[0]) + b, for neighbour
// coefficients c[p] = -0.5 a D2[p] stored in precision S, returned as a (hi, lo) pair in S.
// FP32 (S = float): the centre is moved by the neighbours' rounding, -2 sum (c32 - c64), so the
// FP32 operator keeps the FP64 row sum (a constant keeps its exact kinetic energy), and it is
// carried as two floats.  A single float of ~40 Ha is off by up to 1.3e-6 Ha, and so would be
// every Ritz value of the mixed pass, shifted uniformly.  FP64: hi = the centre, lo = 0.
template <typename S>
void centre_coef(const StencilGeom& g, double a, double b, const S* cx, const S* cy, const S* cz, S* hi, S* lo) {
    double c = -0.5 * a * (g.D2x[0] + g.D2y[0] + g.D2z[0]) + b;
    if (sizeof(S) == sizeof(float)) {
        for (int p = 1; p <= g.R; ++p)
            c -= 2.0 * (((double)cx[p] + 0.5 * a * g.D2x[p]) + ((double)cy[p] + 0.5 * a * g.D2y[p]) +
                        ((double)cz[p] + 0.5 * a * g.D2z[p]));
    }
    *hi = (S)c;
    *lo = (S)(c - (double)*hi);
}

// Padded row length used by the pipelined stencil: rows and Veff rows must be 16-byte multiples.
inline int pipe_row_elems(int nx, size_t scalar_size) {
    const int q = (int)(16 / scalar_size);
    return ((nx + q - 1) / q) * q;
}

// Fused nonlocal term for the pipelined stencil: out += a * W[ptmap[point]] at sphere points
// (W: compact (chi alpha) values, column stride ldw; ptmap row pitch mp; rowstart and its host
// copy: first compact point number of every grid row (z * ny + y), nz * ny + 1 entries).
struct PipeNLHost {
    const void* W;
    long long ldw;
    const int* ptmap;
    int mp;
    const int* rowstart;
    const std::vector<int>* rowstart_host;
    void* xs_out;  // optional compact copy of out at the sphere points (column stride ldw)
};

// Pipelined stencil on 16-byte aligned, row-padded (nxp) blocks; V padded the same way.
// err: device int set to 1 if a bounded shared-memory wait gives up.
template <typename T, typename S>
int launch_cheb_pipe(const StencilGeom& g, int nxp, const T* x, long long ldx, const T* xold, long long ldo, T* out,
                     long long ldout, const S* V, int ncol, double a, double b, double d, const T* phl, const T* phr,
                     int* err, cudaStream_t st, int shape = 0, const struct PipeNLHost* nlh = nullptr);
// Number of launch shapes for FD half-width R: compiled shapes x two y-band splits (shape
// indices 0 .. count-1; any shape gives bitwise the same result, they differ in speed only).
// (odd nx: one).
template <typename T>
int pipe_shape_count(int R, int nx);

// Rayleigh-Ritz Gram products Ms = dV Y^T Y (upper triangle), Hs = dV Y^T HY of FP32 blocks
// (rows x n, column stride ld) on the tensor cores: exact int8-slice products, FP64 result,
// Ms/Hs n x n column-major.  work: gram_plan(rows, n).work_bytes, 256-byte aligned.
// nonfinite (device int, may be null) is set to 1 when Y or HY holds a NaN or Inf.
struct GramPlan {
    long long ldk;      // padded K (rows) of the slice arrays
    int npad;           // N rounded up to the 128-state tile
    int nsplit, kper;   // K chunks and 128-row K steps per chunk
    size_t slice_bytes, exp_bytes, ws_bytes, work_bytes;
};
GramPlan gram_plan(long long rows, int n);
int launch_gram_i8(const float* Y, const float* HY, long long ld, long long rows, int n, double dV,
                   const GramPlan& p, void* work, size_t work_bytes, double* Ms, double* Hs, int* err,
                   int* nonfinite, cudaStream_t st);

// Subspace rotation psi = Y W on the tensor cores (exact int8 slices, FP64 output written into
// an unpadded layout with column stride ldp); gram_tc.cu.  launch_colexp must run on the
// overlap Ms (before its Cholesky factorisation) to fix the per-state scaling.
struct RotPlan {
    long long ldk;  // row stride (bytes) of the slice arrays, >= N
    size_t a_bytes, b_bytes, erow_bytes, col_bytes, work_bytes, smem_rows;
};
RotPlan rot_plan(long long rows, int n);
bool rot_supported(int n);
int launch_colexp(const double* Ms, int n, void* work, const RotPlan& p, long long rows, cudaStream_t st);
// Electron density from the rotation's epilogue: rho[r] (+)= sum_j w[j] psi[r][j]^2 over the
// npts unpadded grid points, with the per-column-tile partials in part (ceil(n / 128) * npts
// doubles) reduced in tile order.
struct RotDensity {
    const double* w;  // [n] weights (device)
    double* part;
    double* rho;      // [npts] (device)
    long long npts;
    bool accumulate;
};
int launch_rot_i8(const float* Y, long long ldy, long long rows, int nx, int nxp, const double* W, int n,
                  const RotPlan& p, void* work, size_t work_bytes, double* psi, long long ldp, int* err,
                  cudaStream_t st, const RotDensity* dens = nullptr);
// rho[i] (+)= sum_n w[n] |psi[n * ld + i]|^2 over nd points (T = double or double2; w device).
template <typename T>
int launch_density(const T* psi, long long ld, long long nd, int ncol, const double* w, double* rho, bool accumulate,
                   cudaStream_t st);

// Rayleigh-Ritz step of few states (small_rr.cu): products in FP64, one CTA for the subspace algebra.
// Y, HY: blocks of n columns, ld >= rows elements apart, rows of nxp with nx valid points (pads
// zero); Ms, Hs: n x n scratch of the wide type (double / double2), psi: nd points per column, stride
// ldp.  info as in rr_alloc_small.  work: small_rr_work_bytes.
constexpr int kSmallRRMax = 40;
bool small_rr_supported(int n);
size_t small_rr_work_bytes(long long rows, int n, size_t wide);
template <typename T>
int launch_small_rr(const T* Y, const T* HY, long long ld, long long rows, int nx, int nxp, long long nd, int n,
                    double dV, void* work, void* Ms, void* Hs, double* eig, int* info, void* psi, long long ldp,
                    cudaStream_t st);

// Effective potential (veff.cu), FP64 fields of nx ny nz points, x fastest.
struct GradGeom {
    int nx, ny, nz, R;
    int periodic[3];          // per direction: 1 periodic ghosts, 0 zero (Dirichlet) ghosts
    double D1[3][kMaxR1];     // first-derivative weights / spacing, index 1..R
};
struct XcMetric {
    int orth;
    double L[9];  // lapc_T, row-major (non-orthogonal cells)
};
constexpr int kAarMaxHist = 16;
struct AarGamma {
    int cols;
    double g[kAarMaxHist];
};
constexpr int kMaxDots = 48;
struct DotList {
    int count;
    const double* u[kMaxDots];
    const double* v[kMaxDots];
};
int launch_rho_xc(const double* rho, const double* core, double* out, long long nd, cudaStream_t st);
// Gradient of rho, GGA-PBE per point and the GGA flux v2xc lapc_T grad(rho) in fx, fy, fz; with rhs also
// 4 pi (rho0 + rho_b) (rho_b may be null).
int launch_grad_pbe(const double* rho, const GradGeom& g, const XcMetric& m, double* fx, double* fy, double* fz,
                    double* vxc, double* exc, double* v2xc, const double* rho0, const double* rho_b, double* rhs,
                    cudaStream_t st);
// v -= div f; with phi also veff = v + phi.
int launch_div_sub(double* v, const GradGeom& g, const double* fx, const double* fy, const double* fz,
                   const double* phi, double* veff, cudaStream_t st);
int launch_aar_pre(const double* r, const double* x, double* x_old, double* f, double* f_old, double* X, double* F,
                   double w, long long n, cudaStream_t st);
int launch_aar_update(double* x, const double* x_old, const double* f, const double* X, const double* F,
                      const AarGamma& g, double c, long long n, cudaStream_t st);
int launch_sub(const double* b, const double* a, double* r, long long n, cudaStream_t st);
// out = sa a (+ sa b) - s  (b may be null)
int launch_add_shift(const double* a, const double* b, double s, double sa, double* out, long long n,
                     cudaStream_t st);
// Periodic Poisson by FFT: z *= s * scale (half-spectrum), s = 1 / Re(FFT of the operator's
// impulse response) with the mean mode set to zero.
int launch_spec_scale(double2* z, const double* s, double scale, long long n, cudaStream_t st);
int launch_inv_symbol(const double2* g, double* s, long long n, cudaStream_t st);
size_t dots_work_bytes();
// Dot products u_k . v_k (deterministic order), copied to host_out; synchronises the stream.
int launch_dots(const DotList& L, long long n, void* work, double* host_out, cudaStream_t st);

// Launches issued by the library (diagnostic counter, incremented by every launcher).
void count_launch(int n = 1);

}  // namespace lynxb

namespace lynxb {

// Device copy of the nonlocal projector tables (see nonlocal.cuh for the layout).
constexpr int kNLMaxColors = 16;  // colour classes the register-tiled scatter accepts
constexpr int kNLTilePts = 64;    // points per tile of the register-tiled nonlocal kernels

struct NLDev {
    int n_atom = 0, n_img = 0, n_pts = 0, max_np = 0, total_proj = 0;
    // Images in colour classes with pairwise disjoint grid points (n_colors = 0: not coloured,
    // the pull-style scatter is used); class k is color_img[color_off[k] .. color_off[k+1]).
    int n_colors = 0;
    int color_off[kNLMaxColors + 1] = {};
    int* color_img = nullptr;
    // (image, first point) of every 64-point tile, colour class k at color_toff[k] .. [k+1]
    int color_toff[kNLMaxColors + 1] = {};
    int2* color_tiles = nullptr;
    // Compact per-point form (only when no grid point lies in two spheres): the distinct
    // points numbered in grid order, ent_pt[entry] = point number of every (image, point) entry.
    bool compact = false;
    int* ent_pt = nullptr;
    int2* pt_meta = nullptr;     // [n_pts] (first projector row, projector count) of the point's atom
    double* chi_pt64 = nullptr;  // [max_np][n_pts] projector values in point order
    float* chi_pt32 = nullptr;
    // Tiles of kExpTilePts consecutive points for the expansion kernel: the distinct atoms of
    // tile t in order of first appearance, exp_tile_atoms[t * exp_amax + slot] (-1 past the
    // tile's count), and every point's slot in its tile.
    int exp_amax = 0;
    int* exp_tile_atoms = nullptr;
    unsigned char* pt_slot = nullptr;
    int* atom_img_ptr = nullptr;
    int* atom_img_list = nullptr;
    int* atom_nproj = nullptr;
    int* atom_poff = nullptr;
    double* gamma = nullptr;
    int* img_atom = nullptr;
    int* img_ndc = nullptr;
    long long* img_goff = nullptr;
    long long* img_chi_off = nullptr;
    double* img_phase = nullptr;
    int* gpos = nullptr;
    double* chi64 = nullptr;
    float* chi32 = nullptr;
    int* pt_grid = nullptr;
    int* pt_ptr = nullptr;
    int* ent_img = nullptr;
    int* ent_loc = nullptr;
};

// Column block widths of the nonlocal kernels; alpha rows are padded to a multiple of kNLColBlock.
constexpr int kNLColBlock = 32;
// Points per tile of the compact expansion kernel (128 threads x 4 consecutive points).
constexpr int kExpTilePts = 512;

template <typename T>
int launch_nl_gather(const NLDev& nl, const T* x, long long ld, int ncol, T* alpha, int ncolp, double dV,
                     cudaStream_t st, bool few);
// Few atoms and columns: a gather by (atom, 64 columns) leaves most SMs idle, and one kernel can take an
// atom's gather and its term together, one CTA per 2 or 4 columns.  Every CTA reads the atom's projector
// values again, so with many (atom, column) pairs the staged gather and the term fused into the stencil
// are the better ones.  Us a degree, FP32 / FP64, this kernel against those: 8 atoms (30^3), 256 columns
// 84 / 128 against 105 / 144, 520 columns 163 / 238 against 146 / 223; 16 atoms, 128 columns 88 / 130
// against 111 / 139, 256 columns 161 / 244 against 144 / 215; 24 atoms, 64 columns 62 / 106 against 91 / 130, 256
// columns 246 / 337 against 191 / 282.  Complex data have the atom kernel's gather in any case, and here
// save the scatter.  cols: the columns of the caller's whole block, also where it is filtered in column
// blocks (the two gathers add in different orders).
constexpr int kNLFewAtoms = 32;
constexpr long long kNLFewPairs = 2048;  // real data: atoms x columns
template <typename T>
bool nl_few_atoms(const NLDev& nl, int cols) {
    return nl.n_atom < kNLFewAtoms && (ScalarOf<T>::cplx || (long long)nl.n_atom * cols <= kNLFewPairs);
}
// out += scale * chi Gamma dV chi^T x in one kernel (disjoint spheres: nl.compact, at most 32
// projectors per atom); bitwise launch_nl_gather + launch_nl_scatter for few atoms and complex data.
template <typename T>
int launch_nl_apply(const NLDev& nl, const T* x, long long ld, T* out, long long ldo, int ncol, double dV,
                    typename ScalarOf<T>::type scale, cudaStream_t st);
template <typename T, typename S>
int launch_nl_scatter(const NLDev& nl, T* out, long long ld, int ncol, const T* alpha, int ncolp, S scale,
                      cudaStream_t st);
// Forces and stress (forces.cu): grid, host FD first-derivative coefficients (R + 1 per direction),
// spacings, and for non-orthogonal cells ui = uvec^-1 and uvec (row-major).
struct ForceGeom {
    int nx, ny, nz, R;
    bool orth;
    const double* D1[3];
    double h[3], ui[9], uvec[9];
};
// Per atom a: out[a][v] = scale * sum_n occ[n] sum_j Gamma_j Re(conj(alpha_j) beta_jv) and ea[a] = escale
// * sum_n occ[n] sum_j Gamma_j |alpha_j|^2, with alpha = dV chi^T psi, beta_v the projections of the FD
// derivatives along the three lattice directions (v < 3), or (stress) of the Cartesian derivatives
// times the position relative to the image (img_pos, device), v = xx xy xz yy yz zz.  All device.
size_t sphere_work_bytes(int n_atom, int ncol, bool stress);
template <typename T>
int launch_sphere_terms(const NLDev& nl, const ForceGeom& g, const T* psi, long long ld, int ncol, const T* phl,
                        const T* phr, const double* img_pos, const double* occ, double scale, double escale,
                        double dV, bool stress, double* work, double* out, double* ea, cudaStream_t st);
// out[v] = scale * sum_n occ[n] sum_r Re(conj(D_a psi_n) D_b psi_n), v = xx xy xz yy yz zz (Cartesian FD
// gradients); phased: some ghost multiplier is not 1.
size_t kinetic_work_bytes(const ForceGeom& g, int ncol, bool cplx);
template <typename T>
int launch_kinetic(const ForceGeom& g, const T* psi, long long ld, int ncol, const T* phl, const T* phr, bool phased,
                   const double* occ, double scale, double* work, double* out, cudaStream_t st);
// W[col * ldw + point] = (chi alpha)(point, col) on the compact point numbering (nl.compact).
template <typename T>
int launch_nl_expand(const NLDev& nl, T* W, long long ldw, int ncol, const T* alpha, int ncolp, cudaStream_t st);

}  // namespace lynxb
