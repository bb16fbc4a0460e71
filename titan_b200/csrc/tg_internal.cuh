// Internal declarations shared by the CUDA translation units of libtitan_gpu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>
#include <vector>

namespace tg {

// Lets `kernel` be launched with `bytes` of dynamic shared memory.  The limit belongs to the function,
// for all threads of the process, not to a launch: every call sets the largest that the device allows,
// so that no thread lowers it between another one's call and launch.
template <class K>
inline cudaError_t allow_smem(K kernel, size_t bytes) {
  int dev = 0, optin = 0;
  cudaFuncAttributes at{};
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, kernel);
  if (e != cudaSuccess) return e;
  const int most = optin - (int)at.sharedSizeBytes;
  if (bytes > (size_t)std::max(most, 0)) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

// ---------------------------------------------------------------------------
// complex FP64 helpers (double2 = re, im)
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ double2 cmk(double r, double i) { return make_double2(r, i); }
__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__host__ __device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
// acc + a*b
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 acc) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
  return acc;
}
// acc - a*b
__device__ __forceinline__ double2 cfms(double2 a, double2 b, double2 acc) {
  acc.x = fma(-a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(-a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
  return acc;
}
// 1/a with scaling against overflow
__device__ __forceinline__ double2 crecip(double2 a) {
  double s = fmax(fabs(a.x), fabs(a.y));
  if (s == 0.0) return make_double2(0.0, 0.0);
  double xr = a.x / s, yr = a.y / s;
  double den = s * (xr * xr + yr * yr);
  return make_double2(xr / den, -yr / den);
}

// Reciprocal of a positive double by Newton-Raphson: start from the
// hardware approximation (rcp.approx.ftz.f64, about 20 correct bits) and
// apply r <- r + r (1 - s r) three times (quadratic convergence, so well past
// 53 bits); the result is within a few ulp of 1/s.
__device__ __forceinline__ double rcp_newton(double s) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(s));
  double e = fma(-s, r, 1.0);
  r = fma(r, e, r);
  e = fma(-s, r, 1.0);
  r = fma(r, e, r);
  e = fma(-s, r, 1.0);
  r = fma(r, e, r);
  return r;
}

// 1/a = conj(a) / |a|^2 for pivots of moderate magnitude (|a|^2 well inside
// the double range, true for z - H(k) entries); returns 0 for a == 0.
__device__ __forceinline__ double2 crecip_fast(double2 a) {
  const double s = fma(a.x, a.x, a.y * a.y);
  if (s == 0.0) return make_double2(0.0, 0.0);
  const double r = rcp_newton(s);
  return make_double2(a.x * r, -a.y * r);
}

// ---------------------------------------------------------------------------
// Output transforms of the Green-function kernel
// ---------------------------------------------------------------------------
enum GreenMode : int {
  MODE_RAW = 0,       // G column-major per point (test hook)
  MODE_A_IMAG = 1,    // w * G, pair-block layout
  MODE_B_IMAG = 2,    // G^T, pair-block layout
  MODE_A_REAL = 3,    // w * (G - G^dagger), pair-block layout
  MODE_B_REAL = 4,    // conj(G), pair-block layout
  MODE_EXPECT = 5,    // accumulate diagonal site blocks (occupations / moments)
  MODE_HK = 6,        // H(k) only (no inversion), column-major per point
};

// A set of (k, z) points.  kind 0: flattened imaginary-axis list (y, kp, w per
// point).  kind 1: real axis, point p = nep * nk + ik with energy x2[nep],
// weight p2[nep] * w[ik], k = kp[ik].  kind 2: explicit (z, k) list (test hook).
struct PointSet {
  int kind = 0;
  const double* y = nullptr;
  const double* kp = nullptr;
  const double* w = nullptr;
  const double* x2 = nullptr;
  const double* p2 = nullptr;
  const double2* z = nullptr;
  int64_t nk = 0;
};

struct GreenArgs {
  PointSet pts;
  int64_t p0 = 0, np = 0;     // point range
  double zr = 0.0, zi = 0.0;  // z = (zr + x2) + i (zi + y)
  double q[3] = {0, 0, 0};
  int mode = MODE_RAW;
  // system
  int n = 0;                  // dimH
  int n_neigh = 0;
  const double* R = nullptr;  // [n_neigh][3]
  const int* pair_start = nullptr;   // [nat*nat+1]
  const int* pair_neigh = nullptr;   // [nblk]
  const double2* pair_t = nullptr;   // [nblk][nmax*nmax], t(or, oc) at oc*nmax + or
  int nmax = 0;
  int n_atoms = 0;
  const int* row_atom = nullptr;     // [n]
  const int* row_orb = nullptr;      // [n]
  const int* row_spin = nullptr;     // [n]
  const double2* h0 = nullptr;       // column-major n x n
  // outputs
  double2* out = nullptr;            // per-point operand / matrix
  double2* out2 = nullptr;           // optional second operand from the same inverse
  int mode2 = MODE_RAW;
  const int* outmap = nullptr;       // [n*n] row*n + col of pair-block slot o
  double2* acc = nullptr;            // MODE_EXPECT: per-CTA sums, 2 n complex each
  const int* exp_rows = nullptr;     // MODE_EXPECT: up / down row of every orbital
  int* status = nullptr;             // first singular point (1-based), atomicMin
  // optional precomputed H(k) table (row-major n x n per k) with a k-major
  // traversal: work item wi -> k index wi / n_e, energy index wi % n_e
  const double2* htab = nullptr;
  int64_t n_e = 0;
  int64_t nk_tab = 0;
  const double* ylist = nullptr;     // imaginary parts of the energies (structured imaginary axis)
  // optional eigendecomposition of every k of the k-major traversal (spectral Green
  // functions; with or without htab): eigU[k][r][a] row-major, eigL[k][a];
  // outinv[r*n + c] = pair-block slot of (r, c)
  const double2* eigU = nullptr;
  const double* eigL = nullptr;
  // optional Householder tridiagonalisation of every k of the k-major traversal (dimensions
  // where G from eigenvectors is not used): T's diagonal triD[k][n] and off-diagonal triE[k][n], the rows
  // trirows[tri_ns] of Q as triQ[k][s][c]; the output is G over those rows and columns
  const double* triD = nullptr;
  const double* triE = nullptr;
  const double2* triQ = nullptr;
  const int* trirows = nullptr;
  int tri_ns = 0;
  double2* triws = nullptr;          // factors of the pass's points (tri_ws_entries)
  const int* outinv = nullptr;
  // optional exponent sidecars of out / out2 (spectral G only): per stored value the
  // frexp exponent of max(|Re|, |Im|), -32768 for zero or subnormal
  int16_t* eout = nullptr;
  int16_t* eout2 = nullptr;
  // energy split of a tabulated imaginary-axis pass: y_side = +1 keeps the points with
  // Im z >= y_split (spectral kernel), -1 those below (blocked Gauss-Jordan kernel); other
  // kernels ignore it and evaluate every point
  double y_split = 0.0;
  int y_side = 0;
  // device workspace of the kernels that exchange data through global memory (the
  // thread-block-cluster Gauss-Jordan kernel: green_cluster_ws_bytes)
  void* ws = nullptr;
  size_t ws_bytes = 0;
};

// true when launch_green evaluates these arguments with the spectral kernel (the only
// one that writes exponent sidecars)
bool green_is_spectral(const GreenArgs& a);

// Launch the fused H(k) + Gauss-Jordan kernel for any supported n.
// Returns cudaErrorInvalidValue for an unsupported dimension.
cudaError_t launch_green(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used);
int green_supported(int n);
int green_warp_supported(int n, int mode);
cudaError_t launch_green_warp(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used);
// blocked Gauss-Jordan on the FP64 tensor cores (dimensions 18, 36, 40, 54, 72, 90): one CTA per
// matrix, at most green_max_ctas(n) CTAs per SM (per-CTA partial sums of MODE_EXPECT)
constexpr int green_max_ctas(int n) { return n <= 18 ? 24 : 15; }
int green_mma_supported(int n, int mode);
cudaError_t launch_green_mma(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used);
// any dimension up to 288, MODE_RAW only: one thread-block cluster per matrix
int green_cluster_supported(int n, int mode);
int green_cluster_size(int n);
size_t green_cluster_ws_bytes(int n, int num_sms);
cudaError_t launch_green_cluster(const GreenArgs& a, int num_sms, cudaStream_t s);

// weight of point pl of a pass: k-major (an H(k) table or its decompositions) or mesh order
__device__ __forceinline__ double point_weight(const GreenArgs& g, int64_t pl) {
  const int64_t wi = g.p0 + pl;
  if (g.htab || g.eigU || g.triQ) {
    const int64_t ik = wi / g.n_e, ie = wi % g.n_e;
    return g.pts.kind == 0 ? g.pts.w[ie * g.nk_tab + ik] : g.pts.p2[ie] * g.pts.w[ik];
  }
  if (g.pts.kind == 0) return g.pts.w[wi];
  if (g.pts.kind == 1) return g.pts.p2[wi / g.pts.nk] * g.pts.w[wi % g.pts.nk];
  return 1.0;
}

// Weighted sums over the column-major Green functions of a pass, added into per-CTA slices of
// acc: products of the spin blocks of orbital pairs (16 sums each, rows (a up, a down, b up,
// b down) per pair; pair_partials slices; with two matrices also the sums with the two
// exchanged, after the others), and single entries (row, column) (entry_partials)
size_t pair_partials(int n, int nlist, bool two, int num_sms, int64_t np);
cudaError_t launch_pairs(const GreenArgs& g, const double2* Ga, const double2* Gb, const int4* pairs, int nlist,
                         int num_sms, double2* acc, cudaStream_t s);
int entry_partials(int64_t np, int num_sms);
cudaError_t launch_entries(const GreenArgs& g, const double2* G, const int2* entries, int ne, int num_sms,
                           double2* acc, cudaStream_t s);

// FP64 pair-block contraction: Cpart[split][cpair_off + u*M + v] += sum_p A[p][off+u] B[p][off+v]
struct PairTile { int pair; int u0; int v0; };
cudaError_t launch_gemm64(const double2* A, const double2* B, int64_t ld, int64_t np, int nsplit,
                          const PairTile* tiles, int ntiles, const int* pair_M, const int* pair_aoff,
                          const int64_t* pair_coff, double2* Cpart, int64_t cstride, cudaStream_t s);

// chi assembly: chi(R, C) column-major from C/D partial sums.
cudaError_t launch_chi_epilogue(const double2* Cpart, const double2* Dpart, int nsplit, int64_t cstride,
                                int dimens, const int* decode, const int* norb, const int64_t* pair_coff,
                                int n_atoms, double scale, double2* chi, cudaStream_t s);

int gemm64_tile();
// H(k) table for a k list (plus q): H[k][r][c] = h0 + H_nl(k + q)
cudaError_t launch_hk_table(const GreenArgs& a, const double* kp, int64_t nk, const double* d_q, double2* phase_ws,
                            double2* H, cudaStream_t s);
cudaError_t launch_reduce_blocks(const double2* part, int nblocks, int len, double2* out, cudaStream_t s);

// Spectral Green functions: eigendecomposition of an H(k) table (ws: eig_ws_bytes of device
// memory for the rotations of `chunk` matrices at a time, eig_chunk where there is room) and G from
// (U, lambda)
int eig_supported(int n);
int eig_fast(int n);
int64_t eig_chunk(int n, int64_t nk);
size_t eig_ws_bytes(int n, int64_t nk, int64_t chunk);
int64_t eig_launches(int64_t nk, int64_t chunk);   // kernels of launch_eig
cudaError_t launch_eig(const double2* H, int64_t nk, int n, double2* U, double* lam, void* ws, int64_t chunk,
                       int* status, int num_sms, cudaStream_t s);
// Reflector I - tau v v^H of LAPACK's zlarfg that takes the vector (alpha, x) to (beta, 0), from
// rest = |x|^2: beta = -sign(Re alpha) |(alpha, x)|, tau = (beta - alpha) / beta, v = (1, sc x); none
// (tau = 0) when x = 0 and alpha is real.  A vector whose squares may underflow, |(alpha, x)|^2 below
// kReflectorTiny, is passed times kReflectorUp (tau and v are the same for it): the reflector of one
// with denormal squares would not be unitary.
constexpr double kReflectorTiny = 1e-270, kReflectorUp = 0x1p600, kReflectorDown = 0x1p-600;
struct Reflector {
  bool any;
  double beta;
  double2 tau, sc;
};
__device__ __forceinline__ double reflector_norm2(double2 alpha, double rest) {
  return fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, rest));
}
__device__ __forceinline__ Reflector reflector(double2 alpha, double rest) {
  Reflector h{!(rest == 0.0 && alpha.y == 0.0), alpha.x, make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  if (h.any) {
    h.beta = -copysign(sqrt(reflector_norm2(alpha, rest)), alpha.x);
    const double ib = 1.0 / h.beta;
    h.tau = make_double2((h.beta - alpha.x) * ib, -alpha.y * ib);
    const double dr = alpha.x - h.beta, di = alpha.y;
    const double inv = 1.0 / fma(dr, dr, di * di);
    h.sc = make_double2(dr * inv, -di * inv);
  }
  return h;
}

// Householder tridiagonalisation of an H(k) table in shared memory, dimensions up to 96 (H is
// kept; rows null: every row of Q)
int hh_small_supported(int n);
cudaError_t launch_hh_small(const double2* H, int64_t nk, int n, const int* rows, int ns, double* D, double* E,
                            double2* Q, int num_sms, cudaStream_t s);
int spectral_supported(int mode, int mode2, bool has_out2);
// Resolvents from a Householder tridiagonalisation per k: H (an H(k) table, overwritten) ->
// T (D, E) and the rows `rows` of Q; G over those rows per point of a k-major pass (MODE_RAW)
int tri_supported(int n);
cudaError_t launch_tridiag(double2* H, int64_t nk, int n, const int* rows, int ns, double* D, double* E,
                           double2* Q, int num_sms, cudaStream_t s);
size_t tri_ws_entries(int n, int64_t np);
cudaError_t launch_green_tri(const GreenArgs& g, int num_sms, cudaStream_t s);
// per-CTA slices [grid][2 n] of the energy-summed diagonal spin blocks (uu, dd, ud, du per orbital)
cudaError_t launch_spec_expect(const double2* U, const double* lam, int64_t nk, int n, const double* ylist, int64_t n_e,
                               const double* w, double zr, double zi, const int* rows, double2* partial, int grid,
                               cudaStream_t s);
// out[ie][r] = -Im G_rr(e_ie + i eta) / pi summed over the tabulated k with weights w
cudaError_t launch_spec_ldos(const double2* U, const double* lam, const double* w, int64_t nk, int n,
                             const double* e, int n_e, double eta, double* out, int num_sms, cudaStream_t s);
cudaError_t launch_green_spectral(const GreenArgs& g, const double2* U, const double* lam, const int* outinv,
                                  int num_sms, cudaStream_t s);

// Linear SOC: X_p = G_p V G_p, and a column-major G_p into a pair-block operand layout
size_t gvg_smem_bytes(int n);
cudaError_t launch_gvg(const double2* G, const double2* V, int n, int64_t np, double2* X, int num_sms,
                       cudaStream_t s);
cudaError_t launch_operand(const double2* G, int n, int64_t np, int64_t p0, const PointSet& pts, int mode,
                           const int* outmap, double2* out, int num_sms, cudaStream_t s);
// operand of a Green-function launch g from its column-major G (MODE_RAW output of g):
// ld slots per point, outmap[o] = r * n + c (an orbital subset in pair-block order)
// eout (null: none): the operand's exponent sidecar (exponent_code16 of every value written)
cudaError_t launch_gather(const GreenArgs& g, const double2* G, int mode, const int* outmap, int64_t ld, double2* out,
                          int16_t* eout, int num_sms, cudaStream_t s);

// frexp exponent of max(|Re|, |Im|) from the bits (the exponent field - 1022 for a normal
// number), -32768 for zero or a subnormal: the exponent sidecar the split quantiser's row
// maxima read instead of the FP64 values
__device__ __forceinline__ int16_t exponent_code16(double2 v) {
  const double m = fmax(fabs(v.x), fabs(v.y));
  const int f = (int)((__double_as_longlong(m) >> 52) & 0x7ff);
  return f == 0 ? (int16_t)-32768 : (int16_t)(f - 1022);
}

// Disturbance-response vertex (eintshe): one launch per pass over RAW G1 / G2
struct SheLaunch {
  const GreenArgs* g = nullptr;   // system tables (n, neighbours, hopping blocks)
  const double2* G1 = nullptr;
  const double2* G2 = nullptr;
  int64_t p0 = 0, np = 0;
  PointSet pts;
  int real_axis = 0;
  int dimens = 0;
  const int* tab = nullptr;       // [4][n / 2]
  const int* ia = nullptr;
  const int* norb = nullptr;
  // register-tiled second stage: 3 x 3 tiles of the (sigma, s', site) output blocks, code
  // sigma | s' << 2 | site << 4 | x0 << 14 | y0 << 20, and the first df row of each site
  const int* ztiles = nullptr;
  int n_ztiles = 0;
  int n_frags = 0;                // sum_i ceil(n_i / 2)^2: 8 x 8 fragments of the sites' entries
  const int* rowoff = nullptr;
  double ue[3] = {0, 0, 0};
  unsigned char spins[3][16] = {};
  double2* partial = nullptr;     // [grid][4 dimens]
  int grid = 0;
  // k-major point order of a tabulated pass (n_e > 0): point p0 + pl -> k = klist[p / n_e],
  // energy p % n_e, as the inversion kernels walk an H(k) table
  int64_t n_e = 0, nk_tab = 0;
  const double* klist = nullptr;
};
// CTAs of one vertex launch (SMs x resident CTAs); 0 when the shared memory does not fit
int she_grid(int n, int dimens, int n_neigh, int n_frags, int num_sms);
cudaError_t launch_she(const SheLaunch& l, cudaStream_t s);
cudaError_t launch_she_prefactor(const double2* P, const double2* df, int dimens, double scale, double2* out,
                                 cudaStream_t s);

}  // namespace tg
