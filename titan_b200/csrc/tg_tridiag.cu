// Resolvents of large Hermitian H(k) on meshes whose energies share a k list, without an
// eigendecomposition.
//
// Per k, H = Q T Q^H with T real symmetric tridiagonal: the Householder reduction of
// LAPACK's zhetd2 (lower form) with zlarfg's reflectors H_j = I - tau_j v_j v_j^H, which
// make every off-diagonal beta_j real, so Q = H_0 H_1 ... H_{n-2}.  Then for every z
//   G_SS(k, z) = Q_S (z - T)^-1 Q_S^H,
// Q_S being the rows S of Q the caller needs (the d orbitals of a d-only chi, or all rows).
// The reduction runs once per k for all energies; per (k, z) the tridiagonal solve
// (z - T) X = Q_S^H costs O(n |S|) and G_SS = Q_S X is a complex GEMM on the FP64 tensor
// cores (mma.sync m8n8k4 .f64).  z - T is factored without pivoting: its pivots obey
// Im d_{i+1} = Im z + e_i^2 Im d_i / |d_i|^2 >= Im z > 0, so none vanishes for Im z > 0.
// Like Gauss-Jordan, the result is the resolvent of H + dH with |dH| ~ eps |H| (both steps
// are backward stable reductions), without the eigenvector mixing that makes spectral G
// less accurate near the real axis.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

constexpr int kTriThreads = 256;

__device__ __forceinline__ double2 warp_sum2(double2 v) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// not volatile: the scheduler may interleave the MMAs of independent accumulators (a chain on
// one accumulator keeps its order through the data dependence, so results do not change)
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Reduction of one H(k) per CTA for dimensions whose matrix does not fit in shared memory.
//
// A: [nk][n][n] row-major H(k) table rows, overwritten; rows[ns]: the rows S of Q to form.
// Out: D[k][i] = T(i, i), E[k][i] = T(i + 1, i) (E[k][n - 1] = 0), Q[k][s][c] = Q(rows[s], c).
// Panels of 8 reflectors, as in LAPACK's zlatrd: inside a panel the trailing matrix is only
// read (once per reflector, A v), with the panel's own changes V W^H + W V^H applied to the
// vectors; it is rewritten once per panel, by FP64 tensor-core products of depth 8, and the
// rows of Q pass through registers once per panel.  Bound by the reads of A v from L2 / HBM
// (16 n^3 / 3 bytes per matrix, two rows and all their loads in flight per warp) and by shared
// memory (71 % of its rate).  196 matrices of dimension 288: 55 ms with a row pass per
// reflector, 13.5 ms now.
constexpr int kPanThreads = 512;
constexpr int kPanNb = 8;              // reflectors per panel
constexpr int kPanS = kPanNb + 4;      // row stride of V and W: 4 mod 8, fragment reads apart
constexpr int kPanSeg = 9;             // 32-column segments of a row: n <= 288

__host__ __device__ inline size_t hh_panel_smem(int n) {
  return sizeof(double2) * ((size_t)n * kPanS * 2 + (size_t)n * kPanNb + 2 * (size_t)n + 4 * kPanNb);
}

__global__ void __launch_bounds__(kPanThreads, 1) hh_panel_kernel(double2* __restrict__ A, int64_t nk, int n,
                                                                const int* __restrict__ rows, int ns,
                                                                double* __restrict__ D, double* __restrict__ E,
                                                                double2* __restrict__ Q) {
  extern __shared__ __align__(16) double2 psm[];
  double2* V = psm;                          // [n][kPanS] reflectors of the panel
  double2* W = V + (size_t)n * kPanS;        // [n][kPanS]
  double2* Vt = W + (size_t)n * kPanS;       // [kPanNb][n] V again, contiguous along a reflector
  double2* x = Vt + (size_t)n * kPanNb;      // [n] current column
  double2* p = x + n;                        // [n] A v, then tau (A v - ..)
  double2* cw = p + n;                       // [kPanNb] W^H v
  double2* cv = cw + kPanNb;                 // [kPanNb] V^H v
  double2* taus = cv + kPanNb;               // [kPanNb]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = kPanThreads / 32;
  const double2 zero = make_double2(0.0, 0.0);
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    double2* Ak = A + k * (int64_t)n * n;
    double2* Qk = Q + k * (int64_t)ns * n;
    for (int e = tid; e < ns * n; e += kPanThreads)
      Qk[e] = make_double2(e % n == rows[e / n] ? 1.0 : 0.0, 0.0);
    for (int j0 = 0; j0 + 1 < n; j0 += kPanNb) {
      const int nb = min(kPanNb, n - 1 - j0);
      for (int jj = 0; jj < nb; ++jj) {
        const int j = j0 + jj;
        // column j with the panel's changes (A is Hermitian: its row j, conjugated)
        for (int i = j + tid; i < n; i += kPanThreads) {
          double2 a = cconj(Ak[(int64_t)j * n + i]);
          for (int t = 0; t < jj; ++t)
            a = cfms(V[i * kPanS + t], cconj(W[j * kPanS + t]), cfms(W[i * kPanS + t], cconj(V[j * kPanS + t]), a));
          x[i] = a;
        }
        __syncthreads();
        double part = 0.0;
        for (int i = j + 2 + lane; i < n; i += 32) part = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, part));
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        double2 alpha = x[j + 1];
        double up = 1.0, down = 1.0;
        if (reflector_norm2(alpha, part) < kReflectorTiny) {   // (the same in every thread)
          up = kReflectorUp;
          down = kReflectorDown;
          alpha = cscale(alpha, up);
          part = 0.0;
          for (int i = j + 2 + lane; i < n; i += 32) {
            const double2 xi = cscale(x[i], up);
            part = fma(xi.x, xi.x, fma(xi.y, xi.y, part));
          }
          for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        }
        const Reflector h = reflector(alpha, part);
        const bool refl = h.any;
        const double2 tau = h.tau;
        if (tid == 0) {
          D[k * n + j] = x[j].x;
          E[k * n + j] = h.beta * down;
          taus[jj] = tau;
        }
        // v (zero up to row j; all zero without a reflector)
        for (int i = tid; i < n; i += kPanThreads) {
          const double2 vi = !refl || i <= j ? zero : i == j + 1 ? make_double2(1.0, 0.0) : cmul(cscale(x[i], up), h.sc);
          V[i * kPanS + jj] = vi;
          Vt[jj * n + i] = vi;
        }
        __syncthreads();
        const double2* v = Vt + (size_t)jj * n;
        if (refl) {
          // A v, two rows per warp
          for (int r = j + 1 + 2 * warp; r < n; r += 2 * nw) {
            const double2* A0 = Ak + (int64_t)r * n;
            const bool two = r + 1 < n;
            double2 a0[kPanSeg], a1[kPanSeg];
#pragma unroll
            for (int u = 0; u < kPanSeg; ++u) {
              const int c = lane + 32 * u;
              const bool in = c > j && c < n;
              a0[u] = in ? A0[c] : zero;
              a1[u] = in && two ? A0[n + c] : zero;
            }
            double2 s0 = zero, s1 = zero;
#pragma unroll
            for (int u = 0; u < kPanSeg; ++u) {
              const int c = lane + 32 * u;
              if (c > j && c < n) {
                const double2 vc = v[c];
                s0 = cfma(a0[u], vc, s0);
                s1 = cfma(a1[u], vc, s1);
              }
            }
            s0 = warp_sum2(s0);
            s1 = warp_sum2(s1);
            if (lane == 0) {
              p[r] = s0;
              if (two) p[r + 1] = s1;
            }
          }
          for (int t = warp; t < 2 * jj; t += nw) {
            const double2* M = t < jj ? W + t : V + (t - jj);
            double2 s = zero;
            for (int c = j + 1 + lane; c < n; c += 32) s = cfma(cconj(M[c * kPanS]), v[c], s);
            s = warp_sum2(s);
            if (lane == 0) (t < jj ? cw[t] : cv[t - jj]) = s;
          }
        }
        __syncthreads();
        for (int r = j + 1 + tid; r < n && refl; r += kPanThreads) {
          double2 a = p[r];
          for (int t = 0; t < jj; ++t)
            a = cfms(V[r * kPanS + t], cw[t], cfms(W[r * kPanS + t], cv[t], a));
          p[r] = cmul(tau, a);
        }
        __syncthreads();
        // w = p - (tau / 2) (p^H v) v
        double2 dot = zero;
        if (refl)
          for (int r = j + 1 + lane; r < n; r += 32) dot = cfma(cconj(p[r]), v[r], dot);
        dot = warp_sum2(dot);
        const double2 a2 = cscale(cmul(tau, dot), -0.5);
        for (int r = tid; r < n; r += kPanThreads)
          W[r * kPanS + jj] = refl && r > j ? cfma(a2, v[r], p[r]) : zero;
        __syncthreads();
      }
      // columns of V and W past the panel's reflectors count as zero below
      for (int e = tid; e < n * (kPanNb - nb); e += kPanThreads) {
        const int i = e / (kPanNb - nb), t = nb + e % (kPanNb - nb);
        V[i * kPanS + t] = W[i * kPanS + t] = zero;
      }
      __syncthreads();
      // A22 -= V W^H + W V^H in 8 x 8 fragments (rows and columns from the first 8-block boundary
      // at or below the panel's end: what lies before it is not read again)
      const int b0 = (j0 + nb) / 8, nbk = (n + 7) / 8, side = nbk - b0;
      const int g8 = lane >> 2, t4 = lane & 3;
      for (int f = warp; f < side * side; f += nw) {
        const int r = 8 * (b0 + f / side) + g8, c = 8 * (b0 + f % side) + 2 * t4;
        const int cb = 8 * (b0 + f % side) + g8;
        double2* Ap = Ak + (int64_t)r * n + c;
        const bool in0 = r < n && c < n, in1 = r < n && c + 1 < n;
        double2 c0 = in0 ? Ap[0] : zero, c1 = in1 ? Ap[1] : zero;
#pragma unroll
        for (int h = 0; h < kPanNb; h += 4) {
          const double2 av = r < n ? V[r * kPanS + h + t4] : zero, aw = r < n ? W[r * kPanS + h + t4] : zero;
          const double2 bw = cb < n ? W[cb * kPanS + h + t4] : zero, bv = cb < n ? V[cb * kPanS + h + t4] : zero;
          // -(a conj(b)): real part -ar br - ai bi, imaginary part -ai br + ar bi
          dmma(c0.x, c1.x, -av.x, bw.x);
          dmma(c0.y, c1.y, -av.y, bw.x);
          dmma(c0.x, c1.x, -av.y, bw.y);
          dmma(c0.y, c1.y, av.x, bw.y);
          dmma(c0.x, c1.x, -aw.x, bv.x);
          dmma(c0.y, c1.y, -aw.y, bv.x);
          dmma(c0.x, c1.x, -aw.y, bv.y);
          dmma(c0.y, c1.y, aw.x, bv.y);
        }
        if (in0) Ap[0] = c0;
        if (in1) Ap[1] = c1;
      }
      // Q_S <- Q_S H_j0 H_j0+1 ..: a row per warp in registers, y = q v, q -= tau y v^H
      for (int s = warp; s < ns; s += nw) {
        double2* Qs = Qk + (int64_t)s * n;
        double2 q[kPanSeg];
#pragma unroll
        for (int u = 0; u < kPanSeg; ++u) {
          const int c = lane + 32 * u;
          q[u] = c < n ? Qs[c] : zero;
        }
        for (int t = 0; t < nb; ++t) {
          const double2* v = Vt + (size_t)t * n;
          double2 y = zero;
#pragma unroll
          for (int u = 0; u < kPanSeg; ++u) {
            const int c = lane + 32 * u;
            if (c < n) y = cfma(q[u], v[c], y);
          }
          const double2 ty = cmul(taus[t], warp_sum2(y));
#pragma unroll
          for (int u = 0; u < kPanSeg; ++u) {
            const int c = lane + 32 * u;
            if (c < n) q[u] = cfms(ty, cconj(v[c]), q[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < kPanSeg; ++u) {
          const int c = lane + 32 * u;
          if (c < n) Qs[c] = q[u];
        }
      }
      __syncthreads();   // (orders this CTA's writes of A before the next panel's reads)
    }
    if (tid == 0) {
      D[k * n + n - 1] = Ak[(int64_t)(n - 1) * n + n - 1].x;
      E[k * n + n - 1] = 0.0;
    }
    __syncthreads();
  }
}

// G of S x S per point (k, z) of a k-major pass.  z - T = L D L^T (complex symmetric, no pivoting),
// so with Q_S(s, :) the rows of Q
//   G(s, c) = sum_i w_i(s) d_i^-1 v_i(c),   w = L^-1 Q_S(s, :)^T,   v = L^-1 Q_S(c, :)^H:
// both factors are forward sweeps y_i = b_i + l_{i-1} y_{i-1}, one thread per row and per column
// with its state in registers, so the sum streams over i in chunks of 8 (two DMMA steps) and no
// solved block is ever stored.  Neither factor is solved backwards, and its rounding errors are
// those of the LU solve (the same pivots; measured on the slabs down to Im z = 1e-3).
//
// tri_lu_kernel: the serial recurrence of the pivots, one thread per point, to global memory
// (l_{i-1} and 1 / d_i, 32 bytes per i).
__global__ void __launch_bounds__(64) tri_lu_kernel(GreenArgs a, double2* __restrict__ ld) {
  const int n = a.n;
  for (int64_t pl = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; pl < a.np; pl += (int64_t)gridDim.x * blockDim.x) {
    const int64_t wi = a.p0 + pl;
    const int64_t ik = wi / a.n_e, ie = wi % a.n_e;
    double zx, zy;
    if (a.pts.kind == 0) {
      zx = a.zr;
      zy = a.zi + a.ylist[ie];
    } else {
      zx = a.zr + a.pts.x2[ie];
      zy = a.zi;
    }
    const double* Dk = a.triD + ik * n;
    const double* Ek = a.triE + ik * n;
    double2* out = ld + pl * 2 * (int64_t)n;
    // d_0 = z - D_0, l_i = E_i / d_i, d_{i+1} = z - D_{i+1} - E_i l_i
    double2 d = make_double2(zx - Dk[0], zy), l = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
      const double s2 = d.x * d.x + d.y * d.y;
      if (s2 == 0.0 && a.status) {
        const int64_t pidx = wi + 1;
        atomicMin(a.status, (int)(pidx < 0x7fffffff ? pidx : 0x7fffffff));
      }
      // |d|^2 >= (Im z)^2 keeps the Newton reciprocal in its range; the division covers the rest
      const double inv = s2 > 1e-300 ? rcp_newton(s2) : (s2 > 0.0 ? 1.0 / s2 : 0.0);
      const double2 id = make_double2(d.x * inv, -d.y * inv);
      out[2 * i] = l;
      out[2 * i + 1] = id;
      if (i + 1 < n) {
        const double e = Ek[i];
        l = cscale(id, e);
        d = make_double2(zx - Dk[i + 1] - e * l.x, zy - e * l.y);
      }
    }
  }
}

// One CTA per point and tile of G: eight warps in a 4 x 2 grid, FM x FN fragments of 8 x 8 each
// (tile 32 FM x 16 FN).  Per chunk of 8 steps i every sweeping thread fetches its 8 entries of
// Q_S two chunks ahead (cp.async, its own 128 bytes, so no barrier), advances its state and
// leaves w_i / d_i or v_i in the double-buffered operand tiles; one barrier per chunk.  The
// DMMAs bound it: 4 FM FN per warp and 4 steps against FM + FN shared-memory reads.  At 288 with
// 160 rows: 74 ms when a thread swept a whole column before the products, 59 ms now (69 % of the
// FP64 tensor pipe); 62 ms with all warps sweeping at the same time.
constexpr int kTriK = 8, kTriStages = 3;

template <int FM, int FN>
struct TriTile {
  static constexpr int TM = 32 * FM, TN = 16 * FN;
  static constexpr int SA = TM + 2, SB = TN + 2;   // 2 mod 8: four steps i and two rows apart
  static constexpr int SQ = kTriK + 1;
  static constexpr size_t smem =
      sizeof(double2) * (kTriStages * ((size_t)(TM + TN) * SQ + 2 * kTriK) + 2 * kTriK * (size_t)(SA + SB));
};

template <int FM, int FN>
__global__ void __launch_bounds__(kTriThreads, 1) tri_green_kernel(GreenArgs a, const double2* __restrict__ ld,
                                                                  int tiles_m, int tiles_n) {
  using TT = TriTile<FM, FN>;
  constexpr int TM = TT::TM, TN = TT::TN, SA = TT::SA, SB = TT::SB, SQ = TT::SQ;
  static_assert(TM + TN <= kTriThreads, "a thread per row and per column of the tile");
  extern __shared__ __align__(16) double2 tsm[];
  double2* qst = tsm;                                              // [stage][TM + TN][SQ]
  double2* lst = qst + kTriStages * (size_t)(TM + TN) * SQ;        // [stage][2 kTriK]
  double2* As = lst + kTriStages * 2 * kTriK;                      // [2][kTriK][SA]
  double2* Bs = As + 2 * kTriK * SA;                               // [2][kTriK][SB]
  const int n = a.n, ns = a.tri_ns;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int wm = (warp >> 1) * 8 * FM, wn = (warp & 1) * 8 * FN;
  const int64_t nn = (int64_t)n * n;
  const int nch = (n + kTriK - 1) / kTriK;
  const int tiles = tiles_m * tiles_n;
  const int64_t items = a.np * tiles;
  const bool sweeps = tid < TM + TN, isrow = tid < TM;
  double2 state = make_double2(0.0, 0.0);

  // this thread's row or column of the item's tile (null past the end), and its chunk loads
  auto source = [&](int64_t item) -> const double2* {
    const int64_t pl = item / tiles;
    const int t = (int)(item - pl * tiles);
    const int64_t ik = (a.p0 + pl) / a.n_e;
    const int s = isrow ? (t % tiles_m) * TM + tid : (t / tiles_m) * TN + tid - TM;
    return sweeps && s < ns ? a.triQ + (ik * ns + s) * (int64_t)n : nullptr;
  };
  auto fetch = [&](int64_t item, const double2* q, int ck) {
    const int st = ck % kTriStages, i0 = ck * kTriK;
    if (q) {
      double2* dst = qst + ((size_t)st * (TM + TN) + tid) * SQ;
#pragma unroll
      for (int u = 0; u < kTriK; ++u) {
        const bool in = i0 + u < n;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                         (unsigned)__cvta_generic_to_shared(dst + u)),
                     "l"(in ? q + i0 + u : q), "r"(in ? 16 : 0));
      }
    }
    if (tid < 2 * kTriK) {
      const bool in = i0 + (tid >> 1) < n;
      const double2* src = ld + (item / tiles) * 2 * (int64_t)n + (in ? 2 * i0 + tid : 0);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(lst + st * 2 * kTriK + tid)),
                   "l"(src), "r"(in ? 16 : 0));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  auto advance = [&](bool live, int ck) {   // chunk ck of the sweep into operand buffer ck & 1
    if (!sweeps) return;
    const int st = ck % kTriStages;
    const double2* q = qst + ((size_t)st * (TM + TN) + tid) * SQ;
    const double2* l = lst + st * 2 * kTriK;
    double2* dst = isrow ? As + (ck & 1) * kTriK * SA + tid : Bs + (ck & 1) * kTriK * SB + tid - TM;
    const int step = isrow ? SA : SB;
    double2 b[kTriK];
#pragma unroll
    for (int u = 0; u < kTriK; ++u) b[u] = live ? q[u] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < kTriK; ++u) {   // (past n: l, 1 / d and q are zero)
      if (!isrow) b[u].y = -b[u].y;
      state = cfma(l[2 * u], state, b[u]);
      b[u] = isrow ? cmul(state, l[2 * u + 1]) : state;
    }
#pragma unroll
    for (int u = 0; u < kTriK; ++u) dst[u * step] = b[u];
  };

  int64_t item = blockIdx.x;
  const double2* q = item < items ? source(item) : nullptr;
  if (item < items) {
    fetch(item, q, 0);
    if (nch > 1) fetch(item, q, 1);
    else asm volatile("cp.async.commit_group;\n" ::);
  }
  for (; item < items; item += gridDim.x) {
    double cr[FM][FN][2], ci[FM][FN][2];
#pragma unroll
    for (int u = 0; u < FM; ++u)
#pragma unroll
      for (int v = 0; v < FN; ++v) cr[u][v][0] = cr[u][v][1] = ci[u][v][0] = ci[u][v][1] = 0.0;
    state = make_double2(0.0, 0.0);
    // before chunk ck is multiplied, chunk ck + 1 is swept into the other operand buffer
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    advance(q != nullptr, 0);
    if (2 < nch) fetch(item, q, 2);
    else asm volatile("cp.async.commit_group;\n" ::);
    const int64_t nitem = item + gridDim.x;
    const double2* nq = nitem < items ? source(nitem) : nullptr;
    for (int ck = 0; ck < nch; ++ck) {
      asm volatile("cp.async.wait_group 1;\n" ::);
      __syncthreads();   // operands of chunk ck and the factors of chunk ck + 1 are in place
      // the two warps of a sub-partition (w and w + 4) sweep one before and one after their
      // products, so that its FP64 pipe always has one of them multiplying
      if (warp < 4 && ck + 1 < nch) advance(q != nullptr, ck + 1);
      if (ck + 3 < nch) fetch(item, q, ck + 3);
      else asm volatile("cp.async.commit_group;\n" ::);
      const double2* A = As + (ck & 1) * kTriK * SA;
      const double2* B = Bs + (ck & 1) * kTriK * SB;
#pragma unroll 1
      for (int kk = 0; kk < kTriK; kk += 4) {
        double2 bv[FN];
#pragma unroll
        for (int v = 0; v < FN; ++v) bv[v] = B[(kk + t4) * SB + wn + 8 * v + g8];
#pragma unroll
        for (int u = 0; u < FM; ++u) {
          const double2 av = A[(kk + t4) * SA + wm + 8 * u + g8];
#pragma unroll
          for (int v = 0; v < FN; ++v) {
            dmma(cr[u][v][0], cr[u][v][1], av.x, bv[v].x);
            dmma(ci[u][v][0], ci[u][v][1], av.x, bv[v].y);
            dmma(cr[u][v][0], cr[u][v][1], -av.y, bv[v].y);
            dmma(ci[u][v][0], ci[u][v][1], av.y, bv[v].x);
          }
        }
      }
      if (warp >= 4 && ck + 1 < nch) advance(q != nullptr, ck + 1);
    }
    // the next item's first chunks travel while this one's results leave
    __syncthreads();
    if (nitem < items) {
      fetch(nitem, nq, 0);
      if (nch > 1) fetch(nitem, nq, 1);
      else asm volatile("cp.async.commit_group;\n" ::);
    }
    const int64_t pl = item / tiles;
    const int t = (int)(item - pl * tiles);
    const int rb = (t % tiles_m) * TM + wm, cb = (t / tiles_m) * TN + wn;
    double2* Gp = a.out + pl * nn;
#pragma unroll
    for (int u = 0; u < FM; ++u) {
      const int row = rb + 8 * u + g8;
      if (row >= ns) continue;
      const int r = a.trirows[row];
#pragma unroll
      for (int v = 0; v < FN; ++v)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = cb + 8 * v + 2 * t4 + h;
          if (c < ns) Gp[(int64_t)a.trirows[c] * n + r] = make_double2(cr[u][v][h], ci[u][v][h]);
        }
    }
    q = nq;
  }
}

}  // namespace

int tri_supported(int n) { return n >= 2 && n <= 288; }

cudaError_t launch_tridiag(double2* H, int64_t nk, int n, const int* rows, int ns, double* D, double* E,
                           double2* Q, int num_sms, cudaStream_t s) {
  if (nk <= 0) return cudaSuccess;
  if (n < 2 || ns <= 0 || ns > n) return cudaErrorInvalidValue;
  // the matrix in shared memory where it fits (no pass over it goes to L2)
  if (hh_small_supported(n)) return launch_hh_small(H, nk, n, rows, ns, D, E, Q, num_sms, s);
  if (n > 32 * kPanSeg) return cudaErrorInvalidValue;
  const size_t smem = hh_panel_smem(n);
  cudaError_t e = allow_smem(hh_panel_kernel, smem);
  if (e != cudaSuccess) return e;
  const int64_t grid = std::min<int64_t>(nk, (int64_t)num_sms);
  hh_panel_kernel<<<(unsigned)grid, kPanThreads, smem, s>>>(H, nk, n, rows, ns, D, E, Q);
  return cudaGetLastError();
}

namespace {

template <int FM, int FN>
cudaError_t launch_tri_tile(const GreenArgs& g, int num_sms, cudaStream_t s) {
  using TT = TriTile<FM, FN>;
  auto kernel = tri_green_kernel<FM, FN>;
  cudaError_t e = allow_smem(kernel, TT::smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTriThreads, TT::smem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  const int tm = (g.tri_ns + TT::TM - 1) / TT::TM, tn = (g.tri_ns + TT::TN - 1) / TT::TN;
  const int64_t grid = std::min<int64_t>(g.np * tm * tn, (int64_t)num_sms * per_sm);
  kernel<<<(unsigned)grid, kTriThreads, TT::smem, s>>>(g, g.triws, tm, tn);
  return cudaGetLastError();
}

}  // namespace

size_t tri_ws_entries(int n, int64_t np) { return (size_t)np * 2 * n; }

cudaError_t launch_green_tri(const GreenArgs& g, int num_sms, cudaStream_t s) {
  if (g.np <= 0) return cudaSuccess;
  if (g.mode != MODE_RAW || g.out2 || !g.triD || !g.triE || !g.triQ || !g.trirows || !g.triws || g.tri_ns <= 0 ||
      g.tri_ns > g.n || g.n_e <= 0)
    return cudaErrorInvalidValue;
  if (!tri_supported(g.n)) return cudaErrorInvalidValue;
  const int64_t blocks = std::min<int64_t>((g.np + 63) / 64, (int64_t)num_sms * 16);
  tri_lu_kernel<<<(unsigned)blocks, 64, 0, s>>>(g, g.triws);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  // the tile shape whose tiles cover the fewest entries of G beyond ns x ns (the DMMAs of the
  // padding cost as much as the others); larger ones first, for their operand reuse and because
  // every tile of a point sweeps its own rows and columns again (160 rows: 160 x 80 twice, 90 rows:
  // 96 x 96 once)
  struct Shape {
    int m, n;
  };
  const Shape shapes[] = {{160, 80}, {96, 96}, {128, 64}, {64, 64}};
  int best = 0;
  int64_t least = 0;
  for (int i = 0; i < 4; ++i) {
    const int64_t area = (int64_t)((g.tri_ns + shapes[i].m - 1) / shapes[i].m * shapes[i].m) *
                         ((g.tri_ns + shapes[i].n - 1) / shapes[i].n * shapes[i].n);
    if (i == 0 || area < least) {
      best = i;
      least = area;
    }
  }
  switch (best) {
    case 0: return launch_tri_tile<5, 5>(g, num_sms, s);
    case 1: return launch_tri_tile<3, 6>(g, num_sms, s);
    case 2: return launch_tri_tile<4, 4>(g, num_sms, s);
    default: return launch_tri_tile<2, 4>(g, num_sms, s);
  }
}

}  // namespace tg
