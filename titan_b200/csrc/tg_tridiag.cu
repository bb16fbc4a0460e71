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

// sum over the block, returned to every thread (red: 2 doubles per warp)
__device__ double2 block_sum2(double2 v, double* red) {
  v = warp_sum2(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) {
    red[2 * warp] = v.x;
    red[2 * warp + 1] = v.y;
  }
  __syncthreads();
  double2 t = make_double2(0.0, 0.0);
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    t.x += red[2 * w];
    t.y += red[2 * w + 1];
  }
  return t;
}

// A: [nk][n][n] row-major H(k) table rows, overwritten; rows[ns]: the rows S of Q to form.
// Out: D[k][i] = T(i, i), E[k][i] = T(i + 1, i) (E[k][n - 1] = 0), Q[k][s][c] = Q(rows[s], c).
// One CTA per k; a warp per row for the matrix-vector products and rank-2 updates.
__global__ void __launch_bounds__(kTriThreads) hh_tridiag_kernel(double2* __restrict__ A, int64_t nk, int n,
                                                                 const int* __restrict__ rows, int ns,
                                                                 double* __restrict__ D, double* __restrict__ E,
                                                                 double2* __restrict__ Q) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* v = reinterpret_cast<double2*>(smem);      // [n] reflector
  double2* w = v + n;                                 // [n] p, then w
  double* red = reinterpret_cast<double*>(w + n);     // [2 * warps]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    double2* Ak = A + k * (int64_t)n * n;
    double2* Qk = Q + k * (int64_t)ns * n;
    for (int64_t e = threadIdx.x; e < (int64_t)ns * n; e += blockDim.x) {
      const int s = (int)(e / n), col = (int)(e % n);
      Qk[e] = make_double2(col == rows[s] ? 1.0 : 0.0, 0.0);
    }
    for (int j = 0; j + 1 < n; ++j) {
      const int m = n - j - 1;
      // x = A(j+1:, j) into v; |x(1:)|^2
      double part = 0.0;
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const double2 x = Ak[(int64_t)(j + 1 + i) * n + j];
        v[i] = x;
        if (i > 0) part += x.x * x.x + x.y * x.y;
      }
      const double xn2 = block_sum2(make_double2(part, 0.0), red).x;   // its barriers publish v
      const double2 alpha = v[0];
      const bool refl = !(xn2 == 0.0 && alpha.y == 0.0);
      // zlarfg: beta = -sign(Re alpha) |(alpha, x)|, tau = (beta - alpha) / beta, v = x / (alpha - beta)
      const double beta = refl ? -copysign(sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xn2), alpha.x) : alpha.x;
      if (threadIdx.x == 0) {
        D[k * n + j] = Ak[(int64_t)j * n + j].x;
        E[k * n + j] = beta;
      }
      __syncthreads();   // alpha read by every thread before v changes
      if (!refl) continue;
      const double2 tau = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
      {
        const double dr = alpha.x - beta, di = alpha.y;
        const double inv = 1.0 / (dr * dr + di * di);
        const double2 sc = make_double2(dr * inv, -di * inv);
        for (int i = threadIdx.x; i < m; i += blockDim.x) v[i] = i == 0 ? make_double2(1.0, 0.0) : cmul(v[i], sc);
      }
      __syncthreads();
      // p = tau A22 v into w: a warp per row, lanes along the row
      for (int r = warp; r < m; r += nw) {
        const double2* Ar = Ak + (int64_t)(j + 1 + r) * n + (j + 1);
        double2 acc = make_double2(0.0, 0.0);
        for (int col = lane; col < m; col += 32) acc = cfma(Ar[col], v[col], acc);
        acc = warp_sum2(acc);
        if (lane == 0) w[r] = cmul(tau, acc);
      }
      __syncthreads();
      // w = p - (tau / 2) (p^H v) v
      double2 dp = make_double2(0.0, 0.0);
      for (int i = threadIdx.x; i < m; i += blockDim.x) dp = cfma(cconj(w[i]), v[i], dp);
      dp = block_sum2(dp, red);
      const double2 a2 = cscale(cmul(tau, dp), -0.5);
      for (int i = threadIdx.x; i < m; i += blockDim.x) w[i] = cfma(a2, v[i], w[i]);
      __syncthreads();
      // A22 -= v w^H + w v^H
      for (int r = warp; r < m; r += nw) {
        double2* Ar = Ak + (int64_t)(j + 1 + r) * n + (j + 1);
        const double2 vr = v[r], wr = w[r];
        for (int col = lane; col < m; col += 32)
          Ar[col] = csub(Ar[col], cadd(cmul(vr, cconj(w[col])), cmul(wr, cconj(v[col]))));
      }
      // Q_S <- Q_S H_j on columns j+1..: y = Q_S(:, j+1:) v, Q_S(:, j+1:) -= tau y v^H
      for (int s = warp; s < ns; s += nw) {
        double2* Qs = Qk + (int64_t)s * n + (j + 1);
        double2 acc = make_double2(0.0, 0.0);
        for (int col = lane; col < m; col += 32) acc = cfma(Qs[col], v[col], acc);
        const double2 ty = cmul(tau, warp_sum2(acc));
        for (int col = lane; col < m; col += 32) Qs[col] = csub(Qs[col], cmul(ty, cconj(v[col])));
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      D[k * n + n - 1] = Ak[(int64_t)(n - 1) * n + n - 1].x;
      E[k * n + n - 1] = 0.0;
    }
    __syncthreads();
  }
}

// not volatile: the scheduler may interleave the MMAs of independent accumulators (a chain on
// one accumulator keeps its order through the data dependence, so results do not change)
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
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
// DMMAs bound it: 4 FM FN per warp and 4 steps against FM + FN shared-memory reads.
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
      if (ck + 1 < nch) advance(q != nullptr, ck + 1);
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
  const size_t smem = sizeof(double2) * 2 * (size_t)n + sizeof(double) * 2 * (kTriThreads / 32);
  const int64_t grid = std::min<int64_t>(nk, (int64_t)num_sms * 4);
  hh_tridiag_kernel<<<(unsigned)grid, kTriThreads, smem, s>>>(H, nk, n, rows, ns, D, E, Q);
  return cudaGetLastError();
}

namespace {

template <int FM, int FN>
cudaError_t launch_tri_tile(const GreenArgs& g, int num_sms, cudaStream_t s) {
  using TT = TriTile<FM, FN>;
  auto kernel = tri_green_kernel<FM, FN>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TT::smem);
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
  // padding cost as much as the others); larger ones first, for their operand reuse
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
