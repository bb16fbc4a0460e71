// Blocked complex Gauss-Jordan inversion with FP64 tensor-core updates, fused with H(k).
//
// One CTA of W warps owns one (k, z) matrix in shared memory (row-major, odd stride, so that
// the 16-byte accesses of a quarter warp to neighbouring rows or columns fall into distinct
// banks).  Columns are eliminated in panels of four, the K of one DMMA (mma.sync m8n8k4 .f64;
// tcgen05 has no FP64 kind):
//   * warp 0 factors the n x 4 panel in registers, a lane per row (two or three rows per
//     lane beyond 32): per column the largest |Re| + |Im| of the rows not yet used, first
//     row on ties (zgetrf's izamax choice; three integer warp reductions on the bits of the
//     value), then the in-place Gauss-Jordan step on the four columns.  Its result X holds
//     the inverse of the 4 x 4 pivot block P in the pivot rows, -A_r P^-1 in the others.
//   * every other column is updated as A <- A' + X A_P (A' = A with the pivot rows zeroed, A_P
//     the four pivot rows before the update): 8 x 8 fragments, four real DMMAs each.  A warp
//     owns whole blocks of 8 columns, so A_P is read by the warp that overwrites it.
//   * look-ahead: warp 0 applies the update to the next panel's four columns itself, in
//     registers, and factors it while the other warps update the rest; one CTA barrier per
//     panel.
// Rows are never swapped: G[r][s] = X[piv[r]][pinv[s]], applied by the output stage, which
// writes the operand layouts (w G, G^T, w (G - G^+), conj G), raw G, H(k) or the
// expectation sums.
//
// What bounds it: shared memory (the A fragments of the updates; L1 at 59 to 69 % of its rate, the
// FP64 tensor pipe at 44 to 49 %) and, at the small dimensions, warp 0's chain of four pivots per
// panel (about 3500 cycles).  Cycles per matrix and SM on one B200, before (Gauss-Jordan steps of
// rank one, matrix in registers) and now: dimension 18: 4400 and 2240, 36: 17500 and 10400, 54:
// 73600 and 29000, 72: 180000 and 62000, 90: 357000 and 118000.  Panels of 8 were slower (36:
// 19800, 72: 81500, 90: 212000): the factorisation grows faster than the updates shrink.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

constexpr int kPanel = 4;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

template <int N>
struct MmaDim {
  static constexpr int NB = (N + 7) / 8;        // row and column blocks of 8
  static constexpr int S = N + 1;               // row stride, odd (N is even)
  static constexpr int NP = (N + kPanel - 1) / kPanel;
  static constexpr int X_SIZE = N * kPanel;
};

struct MmaSmem {
  size_t a, x, prow, phase, piv, pinv, acc, total;
};

template <int N>
__host__ __device__ inline MmaSmem mma_smem(int n_neigh, bool expect) {
  using D = MmaDim<N>;
  MmaSmem L;
  size_t o = 0;
  L.a = o;     o += sizeof(double2) * (size_t)N * D::S;
  L.x = o;     o += sizeof(double2) * 2 * (size_t)D::X_SIZE;
  L.prow = o;  o += sizeof(double2) * 2 * kPanel;
  L.phase = o; o += sizeof(double2) * (size_t)(n_neigh > 0 ? n_neigh : 1);
  L.acc = o;   o += expect ? sizeof(double2) * 2 * (size_t)N : 0;   // MODE_EXPECT sums (4 per orbital)
  L.piv = o;   o += sizeof(int) * (size_t)(kPanel * D::NP);
  L.pinv = o;  o += sizeof(int) * (size_t)N;
  L.total = (o + 15) & ~size_t(15);
  return L;
}

template <int W>
__device__ __forceinline__ void cta_sync() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}

// Factors panel t (columns 4 t ..): reads the columns from A, writes X to Xb and back into
// A's columns, the pivot rows to piv.  One warp; `used` holds a bit per row slot of the lane.
// PEND: the update of panel t - 1 (its X in Xp) has not reached these columns yet; it is applied
// here to the rows in registers.  Returns false when a column has no usable pivot.
template <int N, bool PEND>
__device__ __forceinline__ bool factor_panel(double2* A, const double2* Xp, double2* Xb, double2* prow, int* piv, int t,
                                             unsigned& used) {
  using D = MmaDim<N>;
  constexpr int RS = (N + 31) / 32;
  const int lane = threadIdx.x & 31;
  const int k0 = kPanel * t;
  bool ok = true;
  double2 v[RS][kPanel];
#pragma unroll
  for (int s = 0; s < RS; ++s) {
    const int r = lane + 32 * s;
#pragma unroll
    for (int c = 0; c < kPanel; ++c)
      v[s][c] = r < N && (N % kPanel == 0 || k0 + c < N) ? A[r * D::S + k0 + c] : make_double2(0.0, 0.0);
  }
  if (PEND) {
    int q[kPanel];
#pragma unroll
    for (int k = 0; k < kPanel; ++k) q[k] = piv[k0 - kPanel + k];   // (panel t - 1 is a full one)
#pragma unroll
    for (int s = 0; s < RS; ++s) {
      const int r = lane + 32 * s;
      if (r == q[0] || r == q[1] || r == q[2] || r == q[3]) {
#pragma unroll
        for (int c = 0; c < kPanel; ++c) v[s][c] = make_double2(0.0, 0.0);
      }
    }
#pragma unroll
    for (int k = 0; k < kPanel; ++k) {
      double2 b[kPanel], x[RS];
#pragma unroll
      for (int c = 0; c < kPanel; ++c)
        b[c] = N % kPanel == 0 || k0 + c < N ? A[q[k] * D::S + k0 + c] : make_double2(0.0, 0.0);
#pragma unroll
      for (int s = 0; s < RS; ++s) x[s] = lane + 32 * s < N ? Xp[(lane + 32 * s) * kPanel + k] : make_double2(0.0, 0.0);
#pragma unroll
      for (int s = 0; s < RS; ++s)
#pragma unroll
        for (int c = 0; c < kPanel; ++c) v[s][c] = cfma(x[s], b[c], v[s][c]);
    }
    __syncwarp();   // every lane has read the pivot rows' columns before they are overwritten
  }
  // pivot of column c: its row, or -1 past the last column
  auto search = [&](int c, unsigned long long& key, int& row) {
    key = 0ull;
    row = 0x7fffffff;
#pragma unroll
    for (int s = 0; s < RS; ++s) {
      const int r = lane + 32 * s;
      const double m = fabs(v[s][c].x) + fabs(v[s][c].y);
      const bool cand = r < N && !((used >> s) & 1u) && m > 0.0;
      const unsigned long long b = cand ? (unsigned long long)__double_as_longlong(m) : 0ull;
      if (cand && b > key) {   // bits of |Re| + |Im| (0: none, zero or NaN), first row on ties
        key = b;
        row = r;
      }
    }
  };
  unsigned long long key;
  int row;
  search(0, key, row);
  unsigned mhi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
#pragma unroll
  for (int c = 0; c < kPanel; ++c) {
    if (N % kPanel != 0 && k0 + c >= N) {   // past the last column: an inert step
      if (lane == 0) piv[k0 + c] = -1;
#pragma unroll
      for (int s = 0; s < RS; ++s) v[s][c] = make_double2(0.0, 0.0);
      continue;
    }
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const bool any = (mhi | mlo) != 0u;
    int p = (int)__reduce_min_sync(0xffffffffu, any && hi == mhi && lo == mlo ? (unsigned)row : 0x7fffffffu);
    if (!any) {
      // no pivot: flag the point and go on with any unused row (its result is not used)
      ok = false;
      int fr = 0x7fffffff;
#pragma unroll
      for (int s = RS - 1; s >= 0; --s)
        if (lane + 32 * s < N && !((used >> s) & 1u)) fr = lane + 32 * s;
      p = (int)__reduce_min_sync(0xffffffffu, (unsigned)fr);
    }
    double2* pr = prow + kPanel * (c & 1);
    const bool owner = lane == (p & 31);
    const int slot = p >> 5;   // the same in every lane
#pragma unroll
    for (int s = 0; s < RS; ++s)
      if (slot == s && owner) {
#pragma unroll
        for (int cc = 0; cc < kPanel; ++cc) pr[cc] = v[s][cc];
        used |= 1u << s;
        piv[k0 + c] = p;
      }
    __syncwarp();
    double2 pv[kPanel];
#pragma unroll
    for (int cc = 0; cc < kPanel; ++cc) pv[cc] = pr[cc];
    const double2 d = crecip_fast(pv[c]);
#pragma unroll
    for (int cc = 0; cc < kPanel; ++cc) pv[cc] = cc == c ? d : cmul(pv[cc], d);
    double2 f[RS];
#pragma unroll
    for (int s = 0; s < RS; ++s) f[s] = v[s][c];
    // the next column first: its pivot search runs while the others are updated
    const bool next = c + 1 < kPanel && (N % kPanel == 0 || k0 + c + 1 < N);
    if (next) {
      const int nc = c + 1 < kPanel ? c + 1 : c;
#pragma unroll
      for (int s = 0; s < RS; ++s) v[s][nc] = cfms(f[s], pv[nc], v[s][nc]);
      search(nc, key, row);   // (the pivot row is marked used, so its stale value does not count)
      mhi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    }
#pragma unroll
    for (int cc = 0; cc < kPanel; ++cc) {
      if (next && cc == c + 1) continue;
#pragma unroll
      for (int s = 0; s < RS; ++s) v[s][cc] = cfms(f[s], pv[cc], cc == c ? make_double2(0.0, 0.0) : v[s][cc]);
    }
#pragma unroll
    for (int s = 0; s < RS; ++s)
      if (slot == s && owner) {
#pragma unroll
        for (int cc = 0; cc < kPanel; ++cc) v[s][cc] = pv[cc];
      }
  }
#pragma unroll
  for (int s = 0; s < RS; ++s) {
    const int r = lane + 32 * s;
    if (r < N) {
#pragma unroll
      for (int c = 0; c < kPanel; ++c) {
        Xb[r * kPanel + c] = v[s][c];
        if (N % kPanel == 0 || k0 + c < N) A[r * D::S + k0 + c] = v[s][c];
      }
    }
  }
  return ok;
}

// A <- A' + X A_P on the J column blocks jf, jf + step, ..; the four columns of panel t (they
// hold X) and those of panel t + 1 (left to warp 0) are not stored.  Fragment rows and columns
// past N read whatever lies there (clamped rows, the next row's first columns) and are not
// stored either.
template <int N, int J>
__device__ __forceinline__ void update_blocks(double2* A, const double2* Xb, const int* piv, int t, int ahead, int jf,
                                              int step) {
  using D = MmaDim<N>;
  const int lane = threadIdx.x & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int* pp = piv + kPanel * t;
  const int p0 = pp[0], p1 = pp[1], p2 = pp[2], p3 = pp[3];
  const int pr = t4 == 0 ? p0 : t4 == 1 ? p1 : t4 == 2 ? p2 : p3;
  double2 b[J];
  bool keep[J];
#pragma unroll
  for (int i = 0; i < J; ++i) {
    const int j = jf + i * step;
    const int panel = 2 * j + (t4 >> 1);   // panel of this lane's two columns of block j
    const int bp = 2 * j + (g8 >> 2);      // panel of the column of A_P that this lane holds
    const bool col = bp != t && !(ahead && bp == t + 1) && (N % 8 == 0 || 8 * j + g8 < N);
    b[i] = col && (N % kPanel == 0 || pr >= 0) ? A[pr * D::S + 8 * j + g8] : make_double2(0.0, 0.0);
    keep[i] = panel == t || (ahead && panel == t + 1) || (N % 8 != 0 && 8 * j + 2 * t4 >= N);
  }
  __syncwarp();   // A_P is read before any lane overwrites it
#pragma unroll 2
  for (int bi = 0; bi < D::NB; ++bi) {
    const int r = 8 * bi + g8;
    const int rc = N % 8 == 0 ? r : min(r, N - 1);
    const double2 x = Xb[rc * kPanel + t4];
    const bool zero = r == p0 || r == p1 || r == p2 || r == p3;
#pragma unroll
    for (int i = 0; i < J; ++i) {
      double2* c = A + rc * D::S + 8 * (jf + i * step) + 2 * t4;
      double2 c0 = make_double2(0.0, 0.0), c1 = c0;
      if (!zero && !keep[i]) {
        c0 = c[0];
        c1 = c[1];
      }
      dmma(c0.x, c1.x, x.x, b[i].x);
      dmma(c0.y, c1.y, x.x, b[i].y);
      dmma(c0.x, c1.x, -x.y, b[i].y);
      dmma(c0.y, c1.y, x.y, b[i].x);
      if (!keep[i] && (N % 8 == 0 || r < N)) {
        c[0] = c0;
        c[1] = c1;
      }
    }
  }
}

// every column block first, first + step, .. in pairs
template <int N>
__device__ __forceinline__ void update_list(double2* A, const double2* Xb, const int* piv, int t, int ahead, int first,
                                            int step) {
  using D = MmaDim<N>;
  int j = first;
  for (; j + step < D::NB; j += 2 * step) update_blocks<N, 2>(A, Xb, piv, t, ahead, j, step);
  if (j < D::NB) update_blocks<N, 1>(A, Xb, piv, t, ahead, j, step);
}

// OUT: 0 = operand / raw outputs, 1 = MODE_EXPECT, 2 = MODE_HK
template <int N, int W, int MINB, int OUT>
__global__ void __launch_bounds__(32 * W, MINB) green_mma_kernel(GreenArgs a) {
  using D = MmaDim<N>;
  constexpr int T = 32 * W, NN = N * N;
  extern __shared__ __align__(16) unsigned char smem[];
  const MmaSmem L = mma_smem<N>(a.n_neigh, OUT == 1);
  double2* A = reinterpret_cast<double2*>(smem + L.a);
  double2* X = reinterpret_cast<double2*>(smem + L.x);
  double2* prow = reinterpret_cast<double2*>(smem + L.prow);
  double2* phase = reinterpret_cast<double2*>(smem + L.phase);
  double2* eacc = reinterpret_cast<double2*>(smem + L.acc);
  int* piv = reinterpret_cast<int*>(smem + L.piv);
  int* pinv = reinterpret_cast<int*>(smem + L.pinv);
  const int tid = threadIdx.x;
  // Warp 0 factors; the others update.  The scalar FP64 of the panel and the DMMAs share a
  // sub-partition's pipe (warp id mod 4), so with W = 8 the fourth warp, its neighbour, takes no
  // column blocks; with W = 2 every second pair of CTAs exchanges the two roles, or all the
  // updates of an SM would sit on two of its four pipes.
  int role = tid >> 5;
  if (W == 2) {
    if (tid == 0) {
      unsigned wid;
      asm volatile("mov.u32 %0, %%warpid;" : "=r"(wid));
      piv[0] = (int)(wid >> 2) & 1;
    }
    __syncthreads();
    role ^= piv[0];   // one choice for the CTA
    __syncthreads();
  }
  constexpr int NU = W == 1 ? 1 : W == 8 ? 6 : W - 1;   // updating warps
  const int mine = W == 8 ? (role == 4 ? -1 : role > 4 ? role - 2 : role - 1) : role - 1;

  for (int e = tid; e < N * D::S; e += T) A[e] = make_double2(0.0, 0.0);
  if (OUT == 1)
    for (int e = tid; e < 2 * N; e += T) eacc[e] = make_double2(0.0, 0.0);
  cta_sync<W>();

  for (int64_t pl = blockIdx.x; pl < a.np; pl += gridDim.x) {
    // ---- point data ------------------------------------------------------------
    double zr, zi, w;
    int64_t ktab = -1;
    if (a.htab) {
      const int64_t wi = a.p0 + pl;
      const int64_t ik = wi / a.n_e, ie = wi % a.n_e;
      ktab = ik;
      if (a.pts.kind == 0) {
        zr = a.zr;
        zi = a.zi + a.ylist[ie];
        // energy split: the spectral kernel writes the points with Im z >= y_split
        if (a.y_side < 0 && zi >= a.y_split) continue;
        w = a.pts.w[ie * a.nk_tab + ik];
      } else {
        zr = a.zr + a.pts.x2[ie];
        zi = a.zi;
        w = a.pts.p2[ie] * a.pts.w[ik];
      }
    } else {
      const int64_t p = a.p0 + pl;
      int64_t ik = p;
      if (a.pts.kind == 0) {
        zr = a.zr;
        zi = a.zi + a.pts.y[p];
        w = a.pts.w[p];
      } else if (a.pts.kind == 1) {
        const int64_t nep = p / a.pts.nk;
        ik = p % a.pts.nk;
        zr = a.zr + a.pts.x2[nep];
        zi = a.zi;
        w = a.pts.p2[nep] * a.pts.w[ik];
      } else {
        zr = a.pts.z[p].x;
        zi = a.pts.z[p].y;
        w = 1.0;
      }
      const double kx = a.pts.kp[3 * ik] + a.q[0], ky = a.pts.kp[3 * ik + 1] + a.q[1],
                   kz = a.pts.kp[3 * ik + 2] + a.q[2];
      for (int nb = tid; nb < a.n_neigh; nb += T) {
        const double th = kx * a.R[3 * nb] + ky * a.R[3 * nb + 1] + kz * a.R[3 * nb + 2];
        double s, c;
        sincos(th, &s, &c);
        phase[nb] = make_double2(c, s);
      }
      cta_sync<W>();
    }

    // ---- A = z 1 - H(k) ---------------------------------------------------------
    if (ktab >= 0) {
      const double2* Hk = a.htab + ktab * NN;
#pragma unroll 4
      for (int e = tid; e < NN; e += T) {
        const int r = e / N, c = e % N;
        const double2 h = Hk[e];
        A[r * D::S + c] = r == c ? make_double2(zr - h.x, zi - h.y) : make_double2(-h.x, -h.y);
      }
    } else {
#pragma unroll 2
      for (int e = tid; e < NN; e += T) {
        const int c = e / N, r = e % N;   // column-major walk: h0 and the hopping blocks are stored by columns
        double2 h = a.h0[e];
        if (a.row_spin[r] == a.row_spin[c]) {
          const int pb = a.row_atom[r] * a.n_atoms + a.row_atom[c];
          const double2* tb = a.pair_t + (size_t)a.row_orb[c] * a.nmax + a.row_orb[r];
          const int b1 = a.pair_start[pb + 1];
          for (int b = a.pair_start[pb]; b < b1; ++b)
            h = cfma(phase[a.pair_neigh[b]], tb[(size_t)b * a.nmax * a.nmax], h);
        }
        if (OUT == 2) a.out[pl * NN + e] = h;
        else A[r * D::S + c] = r == c ? make_double2(zr - h.x, zi - h.y) : make_double2(-h.x, -h.y);
      }
    }
    cta_sync<W>();
    if (OUT == 2) continue;

    // ---- blocked Gauss-Jordan ------------------------------------------------------
    unsigned used = 0u;
    bool ok = true;
    if (role == 0) ok = factor_panel<N, false>(A, nullptr, X, prow, piv, 0, used);
    cta_sync<W>();
#pragma unroll 1
    for (int t = 0; t < D::NP; ++t) {
      const double2* Xt = X + (t & 1) * D::X_SIZE;
      double2* Xn = X + ((t + 1) & 1) * D::X_SIZE;
      const bool more = t + 1 < D::NP;
      if (W == 1) {
        update_list<N>(A, Xt, piv, t, 0, 0, 1);
        __syncwarp();
        if (more) ok &= factor_panel<N, false>(A, nullptr, Xn, prow, piv, t + 1, used);
      } else if (role == 0) {
        if (more) ok &= factor_panel<N, true>(A, Xt, Xn, prow, piv, t + 1, used);
      } else if (mine >= 0) {
        update_list<N>(A, Xt, piv, t, more ? 1 : 0, mine, NU);
      }
      cta_sync<W>();
    }
    if (role == 0 && (tid & 31) == 0 && !ok && a.status) {
      const int64_t pidx = a.p0 + pl + 1;
      atomicMin(a.status, (int)(pidx < 0x7fffffff ? pidx : 0x7fffffff));
    }
    for (int k = tid; k < N; k += T) pinv[piv[k]] = k;
    cta_sync<W>();

    // ---- output stage -----------------------------------------------------------
    if (OUT == 0) {
      const int nout = a.out2 ? 2 : 1;
      for (int slot = 0; slot < nout; ++slot) {
        const int mode = slot == 0 ? a.mode : a.mode2;
        double2* dst = (slot == 0 ? a.out : a.out2) + pl * (int64_t)NN;
#pragma unroll 2
        for (int o = tid; o < NN; o += T) {
          double2 v;
          if (mode == MODE_RAW) {
            const int r = o % N, c = o / N;
            v = A[piv[r] * D::S + pinv[c]];
          } else {
            const int rc = a.outmap[o];
            const int r = rc / N, c = rc % N;
            if (mode == MODE_A_IMAG) {
              v = cscale(A[piv[r] * D::S + pinv[c]], w);
            } else if (mode == MODE_B_IMAG) {
              v = A[piv[c] * D::S + pinv[r]];
            } else if (mode == MODE_A_REAL) {
              v = cscale(csub(A[piv[r] * D::S + pinv[c]], cconj(A[piv[c] * D::S + pinv[r]])), w);
            } else {
              v = cconj(A[piv[r] * D::S + pinv[c]]);
            }
          }
          dst[o] = v;
        }
      }
    } else {
      for (int o = tid; o < N / 2; o += T) {
        const int ru = a.exp_rows[2 * o], rd = a.exp_rows[2 * o + 1];
        const double2* Au = A + piv[ru] * D::S;
        const double2* Ad = A + piv[rd] * D::S;
        const int cu = pinv[ru], cd = pinv[rd];
        eacc[4 * o + 0] = cadd(eacc[4 * o + 0], cscale(Au[cu], w));
        eacc[4 * o + 1] = cadd(eacc[4 * o + 1], cscale(Ad[cd], w));
        eacc[4 * o + 2] = cadd(eacc[4 * o + 2], cscale(Au[cd], w));
        eacc[4 * o + 3] = cadd(eacc[4 * o + 3], cscale(Ad[cu], w));
      }
    }
    cta_sync<W>();
  }

  if (OUT == 1) {
    double2* dst = a.acc + (size_t)blockIdx.x * (2 * N);
    for (int e = tid; e < 2 * N; e += T) dst[e] = eacc[e];
  }
}

template <int N, int W, int MINB, int OUT>
cudaError_t launch_o(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  const size_t smem = mma_smem<N>(a.n_neigh, OUT == 1).total;
  int dev = 0, max_smem = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem > (size_t)max_smem) return cudaErrorInvalidValue;
  auto kern = green_mma_kernel<N, W, MINB, OUT>;
  cudaError_t err = allow_smem(kern, smem);
  if (err != cudaSuccess) return err;
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * W, smem);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  per_sm = std::min(per_sm, green_max_ctas(N));   // per-CTA partial sums of MODE_EXPECT are sized for these
  int64_t grid = std::min<int64_t>((int64_t)num_sms * per_sm, a.np);
  if (grid_used) *grid_used = (int)grid;
  kern<<<(unsigned)grid, 32 * W, smem, s>>>(a);
  return cudaGetLastError();
}

template <int N, int W, int MINB>
cudaError_t launch_n(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  if (a.mode == MODE_EXPECT) return launch_o<N, W, MINB, 1>(a, num_sms, s, grid_used);
  if (a.mode == MODE_HK) return launch_o<N, W, MINB, 2>(a, num_sms, s, grid_used);
  return launch_o<N, W, MINB, 0>(a, num_sms, s, grid_used);
}

}  // namespace

int green_mma_supported(int n, int mode) {
  const bool nok = n == 18 || n == 36 || n == 40 || n == 54 || n == 72 || n == 90;
  const bool mok = mode == MODE_RAW || mode == MODE_A_IMAG || mode == MODE_B_IMAG || mode == MODE_A_REAL ||
                   mode == MODE_B_REAL || mode == MODE_EXPECT || mode == MODE_HK;
  return nok && mok;
}

cudaError_t launch_green_mma(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  if (a.np <= 0) {
    if (grid_used) *grid_used = 0;
    return cudaSuccess;
  }
  // warps per matrix, resident CTAs: enough matrices per SM to hide the factoring warp where the
  // matrix is small, enough warps to update beside it where few matrices fit.  Neighbouring
  // choices measured slower (36: 1, 3 and 4 warps; 54: 3, 5 and 7; 72: 5 to 9; 90: 7 to 13).
  // At 18 the 24 matrices of an SM take 80 registers a lane (one Newton step of a bulk cell 16.6 ms;
  // 20 matrices 16.8, 16 matrices 17.5).
  switch (a.n) {
    case 18: return launch_n<18, 1, 24>(a, num_sms, s, grid_used);
    case 36: return launch_n<36, 2, 8>(a, num_sms, s, grid_used);
    case 40: return launch_n<40, 2, 6>(a, num_sms, s, grid_used);
    case 54: return launch_n<54, 4, 3>(a, num_sms, s, grid_used);
    case 72: return launch_n<72, 4, 2>(a, num_sms, s, grid_used);
    case 90: return launch_n<90, 8, 1>(a, num_sms, s, grid_used);
  }
  return cudaErrorInvalidValue;
}

}  // namespace tg
