// Disturbance-response integrand of eintshe (source/eintshe.F90:2-309).
//
// Per (k, E) point, with V = dtdk(k) = sum_n i (u.R_n) t_n exp(i k.R_n) in the
// spinless orbital space (source/dtdksub.F90:2-28; rows: the neighbour's basis
// site, columns: site i), the integrand on the diagonal site blocks is
//   imaginary axis (eintshe.F90:104-179):
//     df[(s, i, mu, nu), s'] += w [ G1^{ab}(i nu, j g) V(j g, l x) G2^{cd}(l x, i mu)
//                                 + conj(G2^{a'b'}(i mu, l x)) V(j g, l x) conj(G1^{c'd'}(j g, i nu)) ]
//   real axis (eintshe.F90:226-249):
//     df[(s, i, mu, nu), s'] += -i w (G1 - G1^+)^{ab}(i nu, j g) V(j g, l x) (G2^+)^{cd}(l x, i mu)
// where the four spins (a, b, c, d) of each term are fixed by (s, s') through
// the reference's tables.  G1 = G(k + q, E + e), G2 = G(k, E).
//
// Work split: one CTA per point at a time (grid-stride), V built in shared
// memory from per-neighbour phases, then two small products per term:
// Y^b = L[:, spin b] V (n x no) and Z = Y^b R[spin c, :] restricted to the
// output entries, which form n_i x n_i blocks per (sigma, s', site).  Each CTA
// owns a slice (4 dimens complex) of a per-CTA global array, so successive
// launches (passes) accumulate without atomics; the slices are summed once at the
// end.  Three variants: when the fragments of all sites' entries fit in the
// registers of eight warps and the Green functions in shared memory, both products
// run on the FP64 tensor cores (she_mma_kernel); else, when they fit (dimH up to
// about 48 for small dimens), both Green functions are staged row-major in shared
// memory and the slice is held there; larger cells read the column-major inversion
// output through L1 / L2 and add into the slice in place.  The last two are
// register-tiled (2 x 3 and 3 x 3 outputs per thread), bound by shared memory.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

struct SheArgs {
  const double2* G1 = nullptr;    // [np][n][n] column-major, G(k + q, E + e)
  const double2* G2 = nullptr;    // [np][n][n] column-major, G(k, E)
  int64_t p0 = 0, np = 0;
  PointSet pts;                   // kind 0 (imaginary list) or 1 (real axis)
  int n = 0, no = 0, dimens = 0, n_neigh = 0, nmax = 0, n_atoms = 0;
  const double* R = nullptr;
  const int* pair_start = nullptr;
  const int* pair_neigh = nullptr;
  const double2* pair_t = nullptr;
  const int* tab = nullptr;       // [4][no]: full row (spin up), full row (spin down), site, orbital in site
  const int* ia = nullptr;        // first row of each site
  const int* norb = nullptr;
  const int* ztiles = nullptr;    // second-stage tiles: sigma | s' << 2 | i << 4 | x0 << 14 | y0 << 20
  int n_ztiles = 0;
  const int* rowoff = nullptr;    // first df row of each site
  int real_axis = 0;
  double ue[3] = {0, 0, 0};
  unsigned char spins[3][16] = {};   // term t, (s * 4 + s') -> a << 3 | b << 2 | c << 1 | d (0 = up)
  double2* partial = nullptr;        // [gridDim][4 dimens], df(row, s') at s' dimens + row
  int64_t n_e = 0, nk_tab = 0;       // k-major order of a tabulated pass (n_e > 0)
  const double* klist = nullptr;
};

// threads of the register-tiled variants
constexpr int kSheThreads = 288;

struct SheSmem {
  int s1, s2, m, y, acc, ph, tab;   // offsets in double2 units (tab: in bytes)
  size_t bytes;
};

// Row strides of the staged Green functions and of Y: odd, so the 16-byte reads of a
// quarter warp on rows a few apart fall into distinct bank groups.
__host__ __device__ inline int she_sst(int n) { return n | 1; }
__host__ __device__ inline int she_yst(int no) { return no | 1; }

// Shared-memory layout.  STAGED: both Green functions (row-major, stride she_sst) and
// the df partial live in shared memory; otherwise they are read from / accumulated in
// global memory (L1 / L2) and only V, Y and the tables are staged.  V^T is read from
// V with swapped indices.
__host__ __device__ inline SheSmem she_layout(int n, int dimens, int n_neigh, bool staged) {
  const int no = n / 2;
  SheSmem L;
  int o = 0;
  L.s1 = o; o += staged ? n * she_sst(n) : 0;
  L.s2 = o; o += staged ? n * she_sst(n) : 0;
  L.m = o; o += no * no;
  L.y = o; o += 2 * n * she_yst(no);
  L.acc = o; o += staged ? 4 * dimens : 0;
  L.ph = o; o += n_neigh > 0 ? n_neigh : 1;
  L.tab = o * (int)sizeof(double2);
  L.bytes = (size_t)L.tab + sizeof(int) * 4 * (size_t)no;
  return L;
}

// n x n operand of a term, element (r, c).  Shared-memory operands are row-major
// and already transformed; global operands are the column-major inversion output
// with the transform applied on read.
struct RowMajor {
  const double2* p;
  int n;
  __device__ __forceinline__ double2 operator()(int r, int c) const { return p[r * n + c]; }
};
enum GlobKind : int { GK_G = 0, GK_CONJ = 1, GK_ANTI = 2, GK_DAGGER = 3 };
struct ColMajor {
  const double2* g;
  int n, kind;   // G, conj(G), G - G^+, G^+
  __device__ __forceinline__ double2 operator()(int r, int c) const {
    const double2 x = g[(size_t)c * n + r];
    if (kind == GK_G) return x;
    if (kind == GK_CONJ) return make_double2(x.x, -x.y);
    const double2 xt = g[(size_t)r * n + c];
    if (kind == GK_ANTI) return make_double2(x.x - xt.x, x.y + xt.y);
    return make_double2(xt.x, -xt.y);
  }
};

// One sandwich term.  M: no x no row-major (the middle factor as used: V or V^T).
// Z(r, col) = sum_{o1, o2} L(r, row_b(o2)) M(o2, o1) R(row_c(o1), col) for the
// output rows (r, col) of each df entry; acc[s' dimens + row] += f Z, in two stages:
// Y^b = L[:, spin b] M for both spins b (2 n x no), then Z from Y and R.
// First stage, register-tiled: each thread computes a 2 x 3 tile (rows r, columns o1) of
// Y^b, so five L and M values loaded per o2 feed six complex FMAs (2 x 18 x 6 = 216 tiles
// at n = 36: one round of the CTA).
template <class LM>
__device__ void she_y_tiled(const SheArgs& a, LM L, const double2* M, bool mt, double2* Y, const int* tab) {
  const int n = a.n, no = a.no, yst = she_yst(no);
  const int tr = (n + 1) / 2, to = (no + 2) / 3;
  for (int t = threadIdx.x; t < 2 * tr * to; t += blockDim.x) {
    const int b = t / (tr * to), r0 = 2 * ((t / to) % tr), q0 = 3 * (t % to);
    const int* rowb = tab + b * no;
    double2 z[2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) z[k][l] = make_double2(0.0, 0.0);
    for (int o2 = 0; o2 < no; ++o2) {
      const int cb = rowb[o2];
      double2 lv[2], mv[3];
#pragma unroll
      for (int k = 0; k < 2; ++k) lv[k] = r0 + k < n ? L(r0 + k, cb) : make_double2(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < 3; ++l)
        mv[l] = q0 + l < no ? (mt ? M[(q0 + l) * no + o2] : M[o2 * no + q0 + l]) : make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) z[k][l] = cfma(lv[k], mv[l], z[k][l]);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l)
        if (r0 + k < n && q0 + l < no) Y[(b * n + r0 + k) * yst + q0 + l] = z[k][l];
  }
  __syncthreads();
}

// Second stage, register-tiled: the df entries of one (sigma, s', site i) form an n_i x n_i
// block Z(x, y) = sum_o1 Y^b(ia + sa n_i + x, o1) R(row_c(o1), ia + sd n_i + y) with
// (mu, nu) = (y, x) when rows_are_nu else (x, y); each thread takes 3 x 3 tiles of blocks.
template <class RM>
__device__ void she_z_tiled(const SheArgs& a, const double2* Y, RM R, double2* acc, const int* tab,
                            const unsigned char* spins, double2 f, bool rows_are_nu) {
  const int n = a.n, no = a.no, D = a.dimens, yst = she_yst(no);
  for (int t = threadIdx.x; t < a.n_ztiles; t += blockDim.x) {
    const int code = a.ztiles[t];
    const int sigma = code & 3, sp = (code >> 2) & 3, i = (code >> 4) & 1023;
    const int x0 = (code >> 14) & 63, y0 = (code >> 20) & 63;
    const int sc = spins[sigma * 4 + sp];
    const int sa = (sc >> 3) & 1, b = (sc >> 2) & 1, c = (sc >> 1) & 1, sd = sc & 1;
    const int ni = a.norb[i], ia = a.ia[i];
    const double2* Yb = Y + (b * n + ia + sa * ni) * yst;
    const int* rowc = tab + c * no;
    const int col0 = ia + sd * ni + y0;
    double2 z[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) z[k][l] = make_double2(0.0, 0.0);
    for (int o1 = 0; o1 < no; ++o1) {
      const int rc = rowc[o1];
      double2 yv[3], rv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) yv[k] = x0 + k < ni ? Yb[(x0 + k) * yst + o1] : make_double2(0.0, 0.0);
#pragma unroll
      for (int l = 0; l < 3; ++l) rv[l] = y0 + l < ni ? R(rc, col0 + l) : make_double2(0.0, 0.0);
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) z[k][l] = cfma(yv[k], rv[l], z[k][l]);
    }
    const int base = sp * D + a.rowoff[i] + sigma;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) {
        if (x0 + k >= ni || y0 + l >= ni) continue;
        const int mu = rows_are_nu ? y0 + l : x0 + k, nu = rows_are_nu ? x0 + k : y0 + l;
        const int o = base + 4 * (mu * ni + nu);
        acc[o] = cfma(f, z[k][l], acc[o]);
      }
  }
}

template <class LM, class RM>
__device__ void she_term(const SheArgs& a, LM L, const double2* M, bool mt, RM R, double2* Y, double2* acc,
                         const int* tab, const unsigned char* spins, double2 f, bool rows_are_nu) {
  she_y_tiled(a, L, M, mt, Y, tab);
  she_z_tiled(a, Y, R, acc, tab, spins, f, rows_are_nu);
  __syncthreads();
}

// k and weight of point p
__device__ __forceinline__ void she_point(const SheArgs& a, int64_t p, double& kx, double& ky, double& kz, double& w) {
  if (a.n_e > 0) {
    const int64_t ik = p / a.n_e, ie = p % a.n_e;
    kx = a.klist[3 * ik];
    ky = a.klist[3 * ik + 1];
    kz = a.klist[3 * ik + 2];
    w = a.pts.kind == 0 ? a.pts.w[ie * a.nk_tab + ik] : a.pts.p2[ie] * a.pts.w[ik];
  } else if (a.pts.kind == 0) {
    kx = a.pts.kp[3 * p];
    ky = a.pts.kp[3 * p + 1];
    kz = a.pts.kp[3 * p + 2];
    w = a.pts.w[p];
  } else {
    const int64_t nep = p / a.pts.nk, ik = p % a.pts.nk;
    kx = a.pts.kp[3 * ik];
    ky = a.pts.kp[3 * ik + 1];
    kz = a.pts.kp[3 * ik + 2];
    w = a.pts.p2[nep] * a.pts.w[ik];
  }
}

// i (u.R) exp(i k.R) per neighbour cell
__device__ __forceinline__ void she_phases(const SheArgs& a, double kx, double ky, double kz, double2* ph) {
  for (int nb = threadIdx.x; nb < a.n_neigh; nb += blockDim.x) {
    const double* Rn = a.R + 3 * nb;
    const double th = kx * Rn[0] + ky * Rn[1] + kz * Rn[2];
    const double ur = a.ue[0] * Rn[0] + a.ue[1] * Rn[1] + a.ue[2] * Rn[2];
    double sn, cs;
    sincos(th, &sn, &cs);
    ph[nb] = make_double2(-ur * sn, ur * cs);
  }
}

// V(orr of site sj, occ of site si): the row on the neighbour's basis site, the column on site si
__device__ __forceinline__ double2 she_vertex(const SheArgs& a, const double2* ph, int sj, int si, int orr, int occ) {
  const int pb = sj * a.n_atoms + si;
  double2 v = make_double2(0, 0);
  for (int b = a.pair_start[pb]; b < a.pair_start[pb + 1]; ++b)
    v = cfma(ph[a.pair_neigh[b]], a.pair_t[(size_t)b * a.nmax * a.nmax + occ * a.nmax + orr], v);
  return v;
}

// STAGED: Green functions and the df slice in shared memory.
template <bool STAGED>
__global__ void __launch_bounds__(kSheThreads) she_kernel(SheArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = a.n, no = a.no, D = a.dimens;
  const SheSmem L = she_layout(n, D, a.n_neigh, STAGED);
  double2* base = reinterpret_cast<double2*>(smem);
  double2* S1 = base + L.s1;
  double2* S2 = base + L.s2;
  double2* M = base + L.m;
  double2* Y = base + L.y;
  const int sst = she_sst(n);
  double2* ph = base + L.ph;
  int* tab = reinterpret_cast<int*>(smem + L.tab);
  double2* mine = a.partial + (size_t)blockIdx.x * 4 * D;
  double2* acc = STAGED ? base + L.acc : mine;
  if (STAGED) {
    for (int e = threadIdx.x; e < 4 * D; e += blockDim.x) acc[e] = mine[e];
  }
  for (int e = threadIdx.x; e < 4 * no; e += blockDim.x) tab[e] = a.tab[e];
  __syncthreads();
  for (int64_t pl = blockIdx.x; pl < a.np; pl += gridDim.x) {
    double kx, ky, kz, w;
    she_point(a, a.p0 + pl, kx, ky, kz, w);
    she_phases(a, kx, ky, kz, ph);
    const double2* g1 = a.G1 + pl * (int64_t)n * n;
    const double2* g2 = a.G2 + pl * (int64_t)n * n;
    if (STAGED) {
      // Green functions of the point, row-major; real axis: S1 = G1 - G1^+, S2 = G2^+
      if (!a.real_axis) {
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
          const int c = e / n, r = e % n;
          S1[r * sst + c] = g1[e];
          S2[r * sst + c] = g2[e];
        }
      } else {
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
          const int r = e / n, c = e % n;
          const double2 x = g1[(size_t)c * n + r], xt = g1[(size_t)r * n + c];
          S1[r * sst + c] = make_double2(x.x - xt.x, x.y + xt.y);
          const double2 y = g2[(size_t)r * n + c];
          S2[r * sst + c] = make_double2(y.x, -y.y);
        }
      }
    }
    __syncthreads();
    // V(rr, cc): rr on the neighbour's basis site, cc on site i
    for (int e = threadIdx.x; e < no * no; e += blockDim.x) {
      const int rr = e / no, cc = e % no;
      M[rr * no + cc] = she_vertex(a, ph, tab[2 * no + rr], tab[2 * no + cc], tab[3 * no + rr], tab[3 * no + cc]);
    }
    __syncthreads();
    if (STAGED) {
      if (!a.real_axis) {
        she_term(a, RowMajor{S1, sst}, M, false, RowMajor{S2, sst}, Y, acc, tab, a.spins[0], make_double2(w, 0.0),
                 true);
        for (int e = threadIdx.x; e < n * sst; e += blockDim.x) {
          S1[e].y = -S1[e].y;
          S2[e].y = -S2[e].y;
        }
        __syncthreads();
        she_term(a, RowMajor{S2, sst}, M, true, RowMajor{S1, sst}, Y, acc, tab, a.spins[1], make_double2(w, 0.0),
                 false);
      } else {
        she_term(a, RowMajor{S1, sst}, M, false, RowMajor{S2, sst}, Y, acc, tab, a.spins[2], make_double2(0.0, -w),
                 true);
      }
    } else {
      if (!a.real_axis) {
        she_term(a, ColMajor{g1, n, GK_G}, M, false, ColMajor{g2, n, GK_G}, Y, acc, tab, a.spins[0], make_double2(w, 0.0),
                 true);
        she_term(a, ColMajor{g2, n, GK_CONJ}, M, true, ColMajor{g1, n, GK_CONJ}, Y, acc, tab, a.spins[1],
                 make_double2(w, 0.0), false);
      } else {
        she_term(a, ColMajor{g1, n, GK_ANTI}, M, false, ColMajor{g2, n, GK_DAGGER}, Y, acc, tab, a.spins[2],
                 make_double2(0.0, -w), true);
      }
    }
  }
  if (STAGED)
    for (int e = threadIdx.x; e < 4 * D; e += blockDim.x) mine[e] = acc[e];
}

// --------------------------------------------------------------------------- on the FP64 tensor cores
// Per site i the entries of a term are one matrix product: with rows u = (b, a, x) and columns
// v = (c, d, y) (a, d the outer spins, b, c the inner ones)
//   Z_i(u, v) = sum_o1 Y^b(a x, o1) R(c o1, d y),   4 n_i x 4 n_i with K = no,
// and (a, b, c, d) takes each of its 16 values for exactly one (sigma, s').  The second
// imaginary-axis term exchanges the roles of the outer orbitals (rows on mu) and its spins are
// (d, c, b, a) of the first, so its transpose adds to the same entries:
//   df_i(u, v) += Y0_i R0_i + R1_i^T Y1_i^T.
// Green functions are staged with the spin as the slow index of rows and columns, so all
// operands are plain strided matrices.  8 x 8 fragments, four real DMMAs (m8n8k4) each and four
// o1: a warp keeps up to kSheFrags of the entries' fragments in registers for the launch.
// Strides: G 2 or 6 mod 8 (its use as a k x columns operand), Y 4 mod 8 (rows x k), so that the
// 16-byte reads of a quarter warp fall apart.  Bound by the FP64 tensor pipe: 2 (2 n no^2 + 16 sum_i n_i^2 no) complex products per
// imaginary point, and 25 % more in padded fragments for sites of nine orbitals.  Two such
// sites: 28.4 ms for 0.36 M points of both axes with register-tiled products on the scalar units,
// 22.1 ms here (61 % of the pipe at the imaginary points).
constexpr int kSheMmaThreads = 256;
constexpr int kSheFrags = 7;   // fragments of a warp

struct SheMma {
  int sg, sm, sy;             // strides of G, V, Y
  int g2, m, y, ph, ints;     // offsets in double2 units
  size_t bytes;
};

__host__ __device__ inline SheMma she_mma_layout(int n, int n_neigh) {
  const int no = n / 2;
  auto stride = [](int least, int res) { return (least - res + 7) / 8 * 8 + res; };   // >= least, res mod 8
  SheMma L;
  const int s2 = stride(n, 2), s6 = stride(n, 6), m2 = stride(no, 2), m6 = stride(no, 6);
  L.sg = s2 < s6 ? s2 : s6;
  L.sm = m2 < m6 ? m2 : m6;
  L.sy = stride(no, 4);
  int o = n * L.sg;
  L.g2 = o; o += n * L.sg;
  L.m = o;  o += no * L.sm;
  L.y = o;  o += 2 * 2 * n * L.sy;
  L.ph = o; o += n_neigh > 0 ? n_neigh : 1;
  L.ints = o;
  L.bytes = sizeof(double2) * (size_t)o + sizeof(int) * ((size_t)5 * no + 8 * kSheFrags + 16);
  return L;
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// c[0..1] + i c[2..3] += a b (CONJ: conj(a) b)
template <bool CONJ>
__device__ __forceinline__ void she_mma(double (&c)[4], double2 a, double2 b) {
  const double na = -a.y;
  dmma(c[0], c[1], a.x, b.x);
  dmma(c[2], c[3], a.x, b.y);
  dmma(c[0], c[1], CONJ ? a.y : na, b.y);
  dmma(c[2], c[3], CONJ ? na : a.y, b.x);
}

// first stage of a term: Y(b n + r, o1) = f sum_o2 L(r, b no + o2) M(o2, o1), fragments dealt to
// the warps from `warp0` on; M transposed and L conjugated for the second term (T)
template <bool T>
__device__ __forceinline__ void she_mma_y(const SheMma& L, int n, int no, const double2* G, const double2* M,
                                          double2* Y, double2 f, int warp0) {
  const int lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int nrf = (2 * n + 7) / 8, ncf = (no + 7) / 8;
  for (int t = warp0; t < nrf * ncf; t += kSheMmaThreads / 32) {
    const int row0 = 8 * (t / ncf) + g8, col0 = 8 * (t % ncf) + g8;
    const int row = min(row0, 2 * n - 1), col = min(col0, no - 1);
    const int b = row >= n;
    const double2* pa = G + (row - b * n) * L.sg + b * no;
    const double2* pb = T ? M + col * L.sm : M + col;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int k = t4; k < no + t4; k += 4) {
      const bool in = k < no;
      const double2 av = in ? pa[k] : make_double2(0.0, 0.0);
      const double2 bv = in ? (T ? pb[k] : pb[k * L.sm]) : make_double2(0.0, 0.0);
      she_mma<T>(c, av, bv);
    }
    if (row0 < 2 * n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o1 = 8 * (t % ncf) + 2 * t4 + h;
        if (o1 < no) Y[row * L.sy + o1] = cmul(f, make_double2(c[h], c[2 + h]));
      }
  }
}

__global__ void __launch_bounds__(kSheMmaThreads, 2) she_mma_kernel(SheArgs a, SheMma L, int nfrag) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = a.n, no = a.no, D = a.dimens;
  double2* S1 = reinterpret_cast<double2*>(smem);
  double2* S2 = S1 + L.g2;
  double2* M = S1 + L.m;
  double2* Y = S1 + L.y;
  double2* ph = S1 + L.ph;
  int* perm = reinterpret_cast<int*>(S1 + L.ints);   // [n] row of H -> spin * no + orbital
  int* site = perm + n;                              // [no] site of an orbital
  int* orb = site + no;                              // [no] orbital in its site
  int* frag = orb + no;                              // [8 kSheFrags] site | fr << 10 | fc << 20
  int* inv = frag + 8 * kSheFrags;                   // [16] (a, b, c, d) -> sigma | s' << 2
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  for (int e = threadIdx.x; e < n; e += blockDim.x) perm[a.tab[e]] = e;
  for (int e = threadIdx.x; e < no; e += blockDim.x) {
    site[e] = a.tab[2 * no + e];
    orb[e] = a.tab[3 * no + e];
  }
  if (threadIdx.x < 16) inv[a.spins[a.real_axis ? 2 : 0][threadIdx.x]] = (int)(threadIdx.x >> 2) | (int)(threadIdx.x & 3) << 2;
  if (threadIdx.x == 0) {
    int f = 0;
    for (int i = 0; i < a.n_atoms; ++i) {
      const int nf = (a.norb[i] + 1) / 2;
      for (int fr = 0; fr < nf; ++fr)
        for (int fc = 0; fc < nf; ++fc) frag[f++] = i | fr << 10 | fc << 20;
    }
  }
  __syncthreads();
  double2* mine = a.partial + (size_t)blockIdx.x * 4 * D;
  // df entry of the lane's element h of fragment j, or -1
  auto entry = [&](int j, int h) {
    const int f = warp + 8 * j;
    if (f >= nfrag) return -1;
    const int i = frag[f] & 1023, u = 8 * ((frag[f] >> 10) & 1023) + g8, v = 8 * (frag[f] >> 20) + 2 * t4 + h;
    const int ni = a.norb[i];
    if (u >= 4 * ni || v >= 4 * ni) return -1;
    const int b = u / (2 * ni), sa = u / ni & 1, nu = u % ni, c = v / (2 * ni), d = v / ni & 1, mu = v % ni;
    const int sp = inv[sa << 3 | b << 2 | c << 1 | d];
    return (sp >> 2) * D + a.rowoff[i] + (sp & 3) + 4 * (mu * ni + nu);
  };
  double acc[kSheFrags][4];
#pragma unroll
  for (int j = 0; j < kSheFrags; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int o = entry(j, h);
      const double2 v = o >= 0 ? mine[o] : make_double2(0.0, 0.0);
      acc[j][h] = v.x;
      acc[j][2 + h] = v.y;
    }
  // a run of points per CTA: in k-major order most have the k of the one before, and its V
  double vx = 0.0, vy = 0.0, vz = 0.0;
  bool have = false;
  const int64_t end = a.np * (blockIdx.x + 1) / gridDim.x;
  for (int64_t pl = a.np * blockIdx.x / gridDim.x; pl < end; ++pl) {
    double kx, ky, kz, w;
    she_point(a, a.p0 + pl, kx, ky, kz, w);
    const bool fresh = !have || kx != vx || ky != vy || kz != vz;
    const double2* g1 = a.G1 + pl * (int64_t)n * n;
    const double2* g2 = a.G2 + pl * (int64_t)n * n;
    // Green functions of the point, spin-major; real axis: S1 = G1 - G1^+, S2 = G2^+
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const int c = e / n, r = e - c * n;
      if (!a.real_axis) {
        const int o = perm[r] * L.sg + perm[c];
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(S1 + o)),
                     "l"(g1 + e)
                     : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(S2 + o)),
                     "l"(g2 + e)
                     : "memory");
      } else {
        const double2 x = g1[e], xt = g1[(size_t)r * n + c], y = g2[e];
        S1[perm[r] * L.sg + perm[c]] = make_double2(x.x - xt.x, x.y + xt.y);
        S2[perm[c] * L.sg + perm[r]] = make_double2(y.x, -y.y);
      }
    }
    if (fresh) {
      she_phases(a, kx, ky, kz, ph);
      __syncthreads();
      for (int e = threadIdx.x; e < no * no; e += blockDim.x) {
        const int rr = e / no, cc = e - rr * no;
        M[rr * L.sm + cc] = she_vertex(a, ph, site[rr], site[cc], orb[rr], orb[cc]);
      }
      have = true;
      vx = kx;
      vy = ky;
      vz = kz;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const double2 f = a.real_axis ? make_double2(0.0, -w) : make_double2(w, 0.0);
    double2* Y1 = Y + 2 * n * L.sy;
    she_mma_y<false>(L, n, no, S1, M, Y, f, warp);
    if (!a.real_axis) she_mma_y<true>(L, n, no, S2, M, Y1, f, 7 - warp);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSheFrags; ++j) {
      const int fi = warp + 8 * j;
      if (fi >= nfrag) continue;
      const int code = frag[fi], i = code & 1023, ni = a.norb[i], off = a.ia[i] >> 1;
      // (past the site's rows or columns: any valid one, the entries are not stored)
      const int u = min(8 * ((code >> 10) & 1023) + g8, 4 * ni - 1), v = min(8 * (code >> 20) + g8, 4 * ni - 1);
      const int ub = u >= 2 * ni, vb = v >= 2 * ni;
      const int ur = u - ub * 2 * ni, vr = v - vb * 2 * ni;
      // row / column of a spin-major matrix: outer spin * no + orbital
      const int uo = (ur >= ni ? no - ni : 0) + off + ur, vo = (vr >= ni ? no - ni : 0) + off + vr;
      {
        const double2* pa = Y + (ub * n + uo) * L.sy;
        const double2* pb = S2 + vb * no * L.sg + vo;
#pragma unroll 2
        for (int k = t4; k < no + t4; k += 4) {
          const bool in = k < no;
          she_mma<false>(acc[j], in ? pa[k] : make_double2(0.0, 0.0), in ? pb[k * L.sg] : make_double2(0.0, 0.0));
        }
      }
      if (!a.real_axis) {
        const double2* pa = S1 + ub * no * L.sg + uo;
        const double2* pb = Y1 + (vb * n + vo) * L.sy;
#pragma unroll 2
        for (int k = t4; k < no + t4; k += 4) {
          const bool in = k < no;
          she_mma<true>(acc[j], in ? pa[k * L.sg] : make_double2(0.0, 0.0), in ? pb[k] : make_double2(0.0, 0.0));
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < kSheFrags; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int o = entry(j, h);
      if (o >= 0) mine[o] = make_double2(acc[j][h], acc[j][2 + h]);
    }
}

// tchi(r, s') = scale sum_c P(r, c) df(c, s'), P column-major (dimens x dimens); P == nullptr: identity
__global__ void she_prefactor_kernel(const double2* __restrict__ P, const double2* __restrict__ df, int D, double scale,
                                     double2* __restrict__ out) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= 4 * D) return;
  const int sp = o / D, r = o % D;
  double2 s = make_double2(0, 0);
  if (P) {
    for (int c = 0; c < D; ++c) s = cfma(P[(size_t)c * D + r], df[(size_t)sp * D + c], s);
  } else {
    s = df[o];
  }
  out[o] = cscale(s, scale);
}

}  // namespace

// Variant choice: the tensor-core kernel when eight warps hold the fragments of all entries and
// its shared memory fits, else the staged kernel when its shared memory fits, else the
// global-operand kernel; 0 bytes when none fits.
enum SheVariant { SHE_GLOBAL = 0, SHE_STAGED = 1, SHE_MMA = 2 };

struct ShePlan {
  SheVariant v = SHE_GLOBAL;
  SheMma mma;
  size_t bytes = 0;
  int threads = kSheThreads;
  const void* fn = nullptr;
};

int she_optin() {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  return optin;
}

ShePlan she_plan(int n, int dimens, int n_neigh, int n_frags) {
  const size_t optin = (size_t)she_optin();
  ShePlan p;
  if (n_frags <= 8 * kSheFrags) {
    const SheMma m = she_mma_layout(n, n_neigh);
    if (m.bytes <= optin) {
      p.v = SHE_MMA;
      p.mma = m;
      p.bytes = m.bytes;
      p.threads = kSheMmaThreads;
      p.fn = (const void*)she_mma_kernel;
      return p;
    }
  }
  p.bytes = she_layout(n, dimens, n_neigh, true).bytes;
  p.v = p.bytes <= optin ? SHE_STAGED : SHE_GLOBAL;
  p.fn = p.v == SHE_STAGED ? (const void*)she_kernel<true> : (const void*)she_kernel<false>;
  if (p.v == SHE_GLOBAL) p.bytes = she_layout(n, dimens, n_neigh, false).bytes;
  if (p.bytes > optin) p.bytes = 0;
  return p;
}

int she_grid(int n, int dimens, int n_neigh, int n_frags, int num_sms) {
  const ShePlan p = she_plan(n, dimens, n_neigh, n_frags);
  if (p.bytes == 0) return 0;
  if (allow_smem(p.fn, p.bytes) != cudaSuccess) return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.fn, p.threads, p.bytes) != cudaSuccess) return 0;
  return num_sms * std::max(per_sm, 1);
}

cudaError_t launch_she(const SheLaunch& l, cudaStream_t s) {
  if (l.grid <= 0) return cudaErrorInvalidValue;
  SheArgs a;
  a.G1 = l.G1;
  a.G2 = l.G2;
  a.p0 = l.p0;
  a.np = l.np;
  a.pts = l.pts;
  a.n = l.g->n;
  a.no = l.g->n / 2;
  a.dimens = l.dimens;
  a.n_neigh = l.g->n_neigh;
  a.nmax = l.g->nmax;
  a.n_atoms = l.g->n_atoms;
  a.R = l.g->R;
  a.pair_start = l.g->pair_start;
  a.pair_neigh = l.g->pair_neigh;
  a.pair_t = l.g->pair_t;
  a.tab = l.tab;
  a.ia = l.ia;
  a.norb = l.norb;
  a.ztiles = l.ztiles;
  a.n_ztiles = l.n_ztiles;
  a.rowoff = l.rowoff;
  a.real_axis = l.real_axis;
  for (int i = 0; i < 3; ++i) a.ue[i] = l.ue[i];
  for (int t = 0; t < 3; ++t)
    for (int i = 0; i < 16; ++i) a.spins[t][i] = l.spins[t][i];
  a.partial = l.partial;
  a.n_e = l.n_e;
  a.nk_tab = l.nk_tab;
  a.klist = l.klist;
  const ShePlan p = she_plan(a.n, a.dimens, a.n_neigh, l.n_frags);
  if (p.bytes == 0) return cudaErrorInvalidValue;
  cudaError_t e = allow_smem(p.fn, p.bytes);
  if (e != cudaSuccess) return e;
  if (p.v == SHE_MMA)
    she_mma_kernel<<<l.grid, p.threads, p.bytes, s>>>(a, p.mma, l.n_frags);
  else if (p.v == SHE_STAGED)
    she_kernel<true><<<l.grid, p.threads, p.bytes, s>>>(a);
  else
    she_kernel<false><<<l.grid, p.threads, p.bytes, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_she_prefactor(const double2* P, const double2* df, int dimens, double scale, double2* out,
                                 cudaStream_t s) {
  const int total = 4 * dimens;
  she_prefactor_kernel<<<(total + 127) / 128, 128, 0, s>>>(P, df, dimens, scale, out);
  return cudaGetLastError();
}

}  // namespace tg
