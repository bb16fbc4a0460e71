// FP64 dense kernels for the RPA Dyson solve chi = (1 + chi_hf U)^-1 chi_hf
// (calculate_chi.F90:85-89): [1 + chi_hf U | chi_hf] is factored by a blocked right-looking
// LU with partial pivoting (zgetrf's izamax choice) that carries the right-hand sides along,
// then solved backwards.  All matrices are column-major.
//
// Blocks of 64 columns, factored in panels of 8: a panel is one CTA (its rows stay in shared
// memory while eight pivots are eliminated), the rest of the 64-column block one CTA per four
// columns, the trailing matrix and the right-hand sides one triangular solve of the block's
// 64 rows and one GEMM of depth 64 on the FP64 tensor cores (zgemm_kernel).  The multipliers
// are applied to the right-hand sides at once and not needed again, so rows are swapped in
// the columns of the block and to its right only.
//
// What bounds it: at dimension 1600 the GEMMs (8 n^3 for chi_hf U, 8/3 n^3 for the LU, 8 n^3
// for the solve) take most of the time, the panels (one SM at a time, about a microsecond a
// column) the rest; small matrices are bound by the panels.  Dimension 1600, one call with its
// host copies: 54 ms with panels of 8 and these GEMMs, 18.6 ms with row-major operands transposed
// on the device and staged copies as well (157 ms with column by column elimination), 17.2 ms
// with panel rows in registers.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/titan_gpu.h"
#include "tg_internal.cuh"

namespace tg {
namespace {

constexpr int kBlock = 64;    // columns of an outer block, depth of the trailing GEMM
constexpr int kPan = 8;       // columns of a panel
constexpr int kPanThreads = 1024;
constexpr int kUpdCols = 4;   // columns per CTA inside a block
constexpr int kSolveCols = 16;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// C (m x n) = A (m x k) B (k x n) (+ 1 on the diagonal when ADD1), or C -= A B
// ---------------------------------------------------------------------------
// CTA tile 64 x 64, eight warps of 32 x 16, K in stages of 8 through a three-stage cp.async
// ring; rows of the stages 66 complex apart, so the fragment reads of a quarter warp (four k,
// two rows) fall into distinct banks.
constexpr int kGT = 64, kGK = 8, kGS = kGT + 2, kGStages = 3;
constexpr size_t kGemmSmem = sizeof(double2) * kGStages * 2 * kGK * kGS;

template <bool SUB>
__global__ void __launch_bounds__(256, 2) zgemm_kernel(int m, int n, int k, const double2* __restrict__ A, int64_t lda,
                                                       const double2* __restrict__ B, int64_t ldb, double2* C,
                                                       int64_t ldc, int add1) {
  extern __shared__ __align__(16) double2 gsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int wm = 32 * (warp & 1), wn = 16 * (warp >> 1);
  const int r0 = blockIdx.x * kGT, c0 = blockIdx.y * kGT;
  auto As = [&](int st) { return gsm + (size_t)st * 2 * kGK * kGS; };
  auto load = [&](int st, int k0) {
    double2* a = As(st);
    double2* b = a + kGK * kGS;
    for (int e = tid; e < kGK * kGT; e += 256) {
      const int kk = e / kGT, r = e % kGT;
      const bool ok = k0 + kk < k && r0 + r < m;
      const double2* src = ok ? A + (int64_t)(k0 + kk) * lda + r0 + r : A;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(a + kk * kGS + r)),
                   "l"(src), "r"(ok ? 16 : 0));
      const int kb = e % kGK, cc = e / kGK;
      const bool okb = k0 + kb < k && c0 + cc < n;
      const double2* sb = okb ? B + (int64_t)(c0 + cc) * ldb + k0 + kb : B;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(b + kb * kGS + cc)),
                   "l"(sb), "r"(okb ? 16 : 0));
    }
  };
  double cr[4][2][2], ci[4][2][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;
  const int ns = (k + kGK - 1) / kGK;
#pragma unroll
  for (int s = 0; s < kGStages - 1; ++s) {
    if (s < ns) load(s, s * kGK);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int s = 0; s < ns; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kGStages - 2));
    __syncthreads();   // stage s has landed, and everyone is done with the one loaded next
    if (s + kGStages - 1 < ns) load((s + kGStages - 1) % kGStages, (s + kGStages - 1) * kGK);
    asm volatile("cp.async.commit_group;\n" ::);
    const double2* a = As(s % kGStages);
    const double2* b = a + kGK * kGS;
#pragma unroll
    for (int kk = 0; kk < kGK; kk += 4) {
      double2 av[4], bv[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = a[(kk + t4) * kGS + wm + 8 * i + g8];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = b[(kk + t4) * kGS + wn + 8 * j + g8];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dmma(cr[i][j][0], cr[i][j][1], av[i].x, bv[j].x);
          dmma(ci[i][j][0], ci[i][j][1], av[i].x, bv[j].y);
          dmma(cr[i][j][0], cr[i][j][1], -av[i].y, bv[j].y);
          dmma(ci[i][j][0], ci[i][j][1], av[i].y, bv[j].x);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + wm + 8 * i + g8;
    if (r >= m) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + wn + 8 * j + 2 * t4 + h;
        if (c >= n) continue;
        double2* p = C + (int64_t)c * ldc + r;
        double2 v = make_double2(cr[i][j][h], ci[i][j][h]);
        if (SUB) v = csub(*p, v);
        else if (add1 && r == c) v.x += 1.0;
        *p = v;
      }
  }
}

template <bool SUB>
cudaError_t zgemm(int m, int n, int k, const double2* A, int64_t lda, const double2* B, int64_t ldb, double2* C,
                  int64_t ldc, int add1, cudaStream_t s) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  cudaError_t e =
      cudaFuncSetAttribute(zgemm_kernel<SUB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
  if (e != cudaSuccess) return e;
  const dim3 g((m + kGT - 1) / kGT, (n + kGT - 1) / kGT);
  zgemm_kernel<SUB><<<g, 256, kGemmSmem, s>>>(m, n, k, A, lda, B, ldb, C, ldc, add1);
  return cudaGetLastError();
}

// largest key of the warp and the first row that has it, by integer reductions on the key's two
// words
__device__ __forceinline__ void warp_best(unsigned long long& key, int& row) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  row = (int)__reduce_min_sync(0xffffffffu, hi == mhi && lo == mlo ? (unsigned)row : 0x7fffffffu);
  key = (unsigned long long)mhi << 32 | mlo;
}

// ---------------------------------------------------------------------------
// panel: columns j0 .. j0 + nb - 1 of M, rows j0 .. n - 1
// ---------------------------------------------------------------------------
// Rows are dealt to the threads; a thread keeps reducing its own rows, so a column costs one
// block-wide pivot search and one barrier for the swapped rows.  STAGED: the panel is copied to
// shared memory (row-major, padded) for the eight steps; larger n works on global memory.
// piv[j] = row swapped with row j (absolute), status = first column without a pivot (1-based).
template <bool STAGED>
__global__ void __launch_bounds__(kPanThreads, 1) panel_kernel(int n, int j0, int nb, double2* __restrict__ M,
                                                               int* __restrict__ piv, int* status) {
  extern __shared__ __align__(16) double2 psm[];
  __shared__ unsigned long long skey[32];
  __shared__ int srow[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, T = blockDim.x, nw = T >> 5;
  const int rows = n - j0;
  double2* P = psm;
  auto at = [&](int r, int c) -> double2& {   // r relative to j0
    return STAGED ? P[r * (kPan + 1) + c] : M[(int64_t)(j0 + c) * n + j0 + r];
  };
  if (STAGED) {
    for (int c = 0; c < nb; ++c)
      for (int r = tid; r < rows; r += T) P[r * (kPan + 1) + c] = M[(int64_t)(j0 + c) * n + j0 + r];
    __syncthreads();
  }
  for (int c = 0; c < nb; ++c) {
    // largest |Re| + |Im| of column c among rows >= c, first row on ties
    unsigned long long key = 0ull;
    int row = 0x7fffffff;
    for (int r = tid; r < rows; r += T) {
      if (r < c) continue;
      const double2 v = at(r, c);
      const double m = fabs(v.x) + fabs(v.y);
      const unsigned long long b = m > 0.0 ? (unsigned long long)__double_as_longlong(m) : 0ull;
      if (b > key) {
        key = b;
        row = r;
      }
    }
    warp_best(key, row);
    if (lane == 0) {
      skey[warp] = key;
      srow[warp] = row;
    }
    __syncthreads();
    key = lane < nw ? skey[lane] : 0ull;
    row = lane < nw ? srow[lane] : 0x7fffffff;
    warp_best(key, row);
    const int p = key == 0ull ? c : row;
    if (tid == 0) {
      piv[j0 + c] = j0 + p;
      if (key == 0ull) atomicMin(status, j0 + c + 1);
    }
    if (tid < nb && p != c) {
      const double2 t = at(c, tid);
      at(c, tid) = at(p, tid);
      at(p, tid) = t;
    }
    __syncthreads();
    double2 u[kPan];
#pragma unroll
    for (int cc = 0; cc < kPan; ++cc) u[cc] = cc >= c && cc < nb ? at(c, cc) : make_double2(0.0, 0.0);
    double2 diag = u[0];
#pragma unroll
    for (int cc = 1; cc < kPan; ++cc)
      if (cc == c) diag = u[cc];
    const double2 d = crecip(diag);
    for (int r = tid; r < rows; r += T) {
      if (r <= c) continue;
      const double2 f = cmul(at(r, c), d);
      at(r, c) = f;
#pragma unroll
      for (int cc = 1; cc < kPan; ++cc)
        if (cc > c && cc < nb) at(r, cc) = cfms(f, u[cc], at(r, cc));
    }
    __syncthreads();   // the next search and swap read other threads' rows
  }
  if (STAGED)
    for (int c = 0; c < nb; ++c)
      for (int r = tid; r < rows; r += T) M[(int64_t)(j0 + c) * n + j0 + r] = P[r * (kPan + 1) + c];
}

// The same for at most kPanThreads rows, a thread per row with the row's panel columns in
// registers: rows are exchanged by exchanging their positions, and only the pivot row passes
// through shared memory, so a column costs two barriers.  Bound by its chain of reductions,
// barriers and the reciprocal: 11.7 us for a panel of 320 rows (21.9 us with the panel in shared
// memory), 17 us for 1024 (40 us for the 1600 that stay there; two rows per thread would not fit
// the registers of 1024 threads).
__global__ void __launch_bounds__(kPanThreads, 1) panel_rows_kernel(int n, int j0, int nb, double2* __restrict__ M,
                                                                    int* __restrict__ piv, int* status) {
  __shared__ unsigned long long skey[32];
  __shared__ int spos[32];
  __shared__ double2 u[kPan];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int rows = n - j0;
  int pos = tid < rows ? tid : -1;   // position of this thread's row
  double2 v[kPan];
#pragma unroll
  for (int c = 0; c < kPan; ++c)
    v[c] = tid < rows && c < nb ? M[(int64_t)(j0 + c) * n + j0 + tid] : make_double2(0.0, 0.0);
#pragma unroll
  for (int c = 0; c < kPan; ++c) {
    if (c >= nb) break;
    // largest |Re| + |Im| of column c among positions >= c, first position on ties
    const double m = fabs(v[c].x) + fabs(v[c].y);
    unsigned long long key = pos >= c && m > 0.0 ? (unsigned long long)__double_as_longlong(m) : 0ull;
    int at = key != 0ull ? pos : 0x7fffffff;
    warp_best(key, at);
    if (lane == 0) {
      skey[warp] = key;
      spos[warp] = at;
    }
    __syncthreads();
    key = lane < nw ? skey[lane] : 0ull;
    at = lane < nw ? spos[lane] : 0x7fffffff;
    warp_best(key, at);
    const int p = key == 0ull ? c : at;
    if (tid == 0) {
      piv[j0 + c] = j0 + p;
      if (key == 0ull) atomicMin(status, j0 + c + 1);
    }
    const bool pivot = pos == p;
    if (pivot) {
#pragma unroll
      for (int cc = c; cc < kPan; ++cc) u[cc] = v[cc];
    }
    pos = pivot ? c : pos == c ? p : pos;
    __syncthreads();
    if (pos > c) {
      const double2 f = cmul(v[c], crecip(u[c]));
      v[c] = f;
#pragma unroll
      for (int cc = c + 1; cc < kPan; ++cc) v[cc] = cfms(f, u[cc], v[cc]);
    }
  }
  if (pos >= 0)
#pragma unroll
    for (int c = 0; c < kPan; ++c)
      if (c < nb) M[(int64_t)(j0 + c) * n + j0 + pos] = v[c];
}

// Net effect of the row swaps piv[j0 .. j0 + nb) (rows relative to j0, nb <= kBlock): row j < nb
// receives the old row top[j], row row[j] = piv[j0 + j] - j0, when >= nb, the old row
// ext[first[j]] (first[j]: the first of the swaps with that row).  Every thread calls it.
struct NetSwaps {
  int row[kBlock], top[kBlock], ext[kBlock], first[kBlock];
};
__device__ __forceinline__ void net_swaps(NetSwaps& w, const int* __restrict__ piv, int j0, int nb) {
  const int t = threadIdx.x;
  if (t < nb) {
    w.row[t] = w.ext[t] = piv[j0 + t] - j0;
    w.top[t] = t;
  }
  __syncthreads();
  if (t < nb) {
    int f = t;
    for (int i = t - 1; i >= 0; --i)
      if (w.row[i] == w.row[t]) f = i;
    w.first[t] = f;
  }
  __syncthreads();
  if (t == 0)
    for (int j = 0; j < nb; ++j) {
      int& o = w.row[j] < nb ? w.top[w.row[j]] : w.ext[w.first[j]];
      const int x = w.top[j];
      w.top[j] = o;
      o = x;
    }
  __syncthreads();
}

// the panel (j0, nb) applied inside its block's columns [k0, k1): row swaps, and right of the
// panel the rank-nb update.  One CTA per kUpdCols columns.
__global__ void __launch_bounds__(512) block_update_kernel(int n, int j0, int nb, int k0, int k1,
                                                           double2* __restrict__ M, const int* __restrict__ piv) {
  __shared__ NetSwaps sw;
  __shared__ double2 T[kPan][kUpdCols], V[kPan][kUpdCols], Lt[kPan][kPan];
  const int tid = threadIdx.x, rows = n - j0;
  // the block's columns without the panel's
  auto col = [&](int i) {
    const int c = k0 + blockIdx.x * kUpdCols + i;
    return c < j0 ? c : c + nb;
  };
  net_swaps(sw, piv, j0, nb);
  if (tid < kPan * kUpdCols) {
    const int j = tid / kUpdCols, i = tid % kUpdCols, c = col(i);
    if (j < nb && c < k1) {
      T[j][i] = M[(int64_t)c * n + j0 + sw.top[j]];
      V[j][i] = M[(int64_t)c * n + j0 + sw.ext[sw.first[j]]];
    }
  } else if (tid >= 64 && tid < 64 + kPan * kPan) {
    const int j = (tid - 64) / kPan, r = (tid - 64) % kPan;
    if (j < nb && r < nb) Lt[r][j] = M[(int64_t)(j0 + j) * n + j0 + r];
  }
  __syncthreads();
  if (tid < kUpdCols) {
    const int c = col(tid);
    if (c < k1) {
      for (int j = 0; j < nb; ++j)
        if (sw.row[j] >= nb) M[(int64_t)c * n + j0 + sw.row[j]] = V[j][tid];
      if (c >= j0)   // unit lower solve of the top rows
        for (int j = 1; j < nb; ++j)
          for (int l = 0; l < j; ++l) T[j][tid] = cfms(Lt[j][l], T[l][tid], T[j][tid]);
      for (int j = 0; j < nb; ++j) M[(int64_t)c * n + j0 + j] = T[j][tid];
    }
  }
  __syncthreads();   // (also orders this CTA's swapped rows before the update below)
  for (int r = nb + tid; r < rows; r += blockDim.x) {
    double2 l[kPan];
#pragma unroll
    for (int j = 0; j < kPan; ++j) l[j] = j < nb ? M[(int64_t)(j0 + j) * n + j0 + r] : make_double2(0.0, 0.0);
#pragma unroll 2
    for (int i = 0; i < kUpdCols; ++i) {
      const int c = col(i);
      if (c < j0 || c >= k1) continue;
      double2* x = M + (int64_t)c * n + j0 + r;
      double2 v = *x;
#pragma unroll
      for (int j = 0; j < kPan; ++j)
        if (j < nb) v = cfms(l[j], T[j][i], v);
      *x = v;
    }
  }
}

// right of a factored block (k0, nb): row swaps and the unit lower solve of its nb rows, on
// the columns c0 .. n - 1 of M and all columns of R.  One CTA per kSolveCols columns.
__global__ void __launch_bounds__(256) block_solve_kernel(int n, int k0, int nb, int c0, double2* __restrict__ M,
                                                          double2* __restrict__ R, const int* __restrict__ piv) {
  extern __shared__ __align__(16) double2 ssm[];
  double2* T = ssm;                                  // [kBlock][kSolveCols]
  double2* V = T + kBlock * kSolveCols;              // [kBlock][kSolveCols]
  double2* Ls = V + kBlock * kSolveCols;             // [kBlock][kBlock] L(r, c) at c * kBlock + r
  __shared__ NetSwaps sw;
  const int tid = threadIdx.x, nm = n - c0;
  auto colp = [&](int i) -> double2* {
    const int c = blockIdx.x * kSolveCols + i;
    return c < nm ? M + (int64_t)(c0 + c) * n : c - nm < n ? R + (int64_t)(c - nm) * n : nullptr;
  };
  net_swaps(sw, piv, k0, nb);
  for (int e = tid; e < nb * kBlock; e += 256) {
    const int c = e / kBlock, r = e % kBlock;
    if (r < nb) Ls[e] = M[(int64_t)(k0 + c) * n + k0 + r];
  }
  for (int e = tid; e < nb * kSolveCols; e += 256) {
    const int j = e % nb, i = e / nb;
    const double2* x = colp(i);
    if (x) {
      T[j * kSolveCols + i] = x[k0 + sw.top[j]];
      V[j * kSolveCols + i] = x[k0 + sw.ext[sw.first[j]]];
    }
  }
  __syncthreads();
  for (int e = tid; e < nb * kSolveCols; e += 256) {
    const int j = e % nb, i = e / nb;
    double2* x = colp(i);
    if (x && sw.row[j] >= nb) x[k0 + sw.row[j]] = V[j * kSolveCols + i];
  }
  const int i = tid % kSolveCols, rg = tid / kSolveCols;
  for (int j = 0; j + 1 < nb; ++j) {
    const double2 t = T[j * kSolveCols + i];
    for (int r = j + 1 + rg; r < nb; r += 256 / kSolveCols)
      T[r * kSolveCols + i] = cfms(Ls[j * kBlock + r], t, T[r * kSolveCols + i]);
    __syncthreads();
  }
  for (int e = tid; e < nb * kSolveCols; e += 256) {
    const int j = e % nb, ii = e / nb;
    double2* x = colp(ii);
    if (x) x[k0 + j] = T[j * kSolveCols + ii];
  }
}

// rows k0 .. k0 + nb - 1 of R <- U(k0.., k0..)^-1 R (upper, non-unit)
__global__ void __launch_bounds__(256) back_solve_kernel(int n, int k0, int nb, const double2* __restrict__ M,
                                                         double2* __restrict__ R) {
  extern __shared__ __align__(16) double2 ssm[];
  double2* T = ssm;                        // [kBlock][kSolveCols]
  double2* Us = T + kBlock * kSolveCols;   // [kBlock][kBlock] U(r, c) at c * kBlock + r
  double2* dinv = Us + kBlock * kBlock;    // [kBlock]
  const int tid = threadIdx.x;
  const int cb = blockIdx.x * kSolveCols;
  for (int e = tid; e < nb * kBlock; e += 256) {
    const int c = e / kBlock, r = e % kBlock;
    if (r < nb) {
      const double2 u = M[(int64_t)(k0 + c) * n + k0 + r];
      Us[e] = u;
      if (r == c) dinv[c] = crecip(u);
    }
  }
  for (int e = tid; e < nb * kSolveCols; e += 256) {
    const int j = e % nb, i = e / nb;
    if (cb + i < n) T[j * kSolveCols + i] = R[(int64_t)(cb + i) * n + k0 + j];
  }
  __syncthreads();
  const int i = tid % kSolveCols, rg = tid / kSolveCols;
  for (int j = nb - 1; j >= 0; --j) {
    const double2 t = cmul(T[j * kSolveCols + i], dinv[j]);
    for (int r = rg; r < j; r += 256 / kSolveCols)
      T[r * kSolveCols + i] = cfms(Us[j * kBlock + r], t, T[r * kSolveCols + i]);
    __syncthreads();
  }
  for (int e = tid; e < nb * kSolveCols; e += 256) {
    const int j = e % nb, ii = e / nb;
    if (cb + ii < n) R[(int64_t)(cb + ii) * n + k0 + j] = cmul(T[j * kSolveCols + ii], dinv[j]);
  }
}

// out = in^T, n x n
__global__ void __launch_bounds__(256) transpose_kernel(int n, const double2* __restrict__ in,
                                                        double2* __restrict__ out) {
  __shared__ double2 t[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = y; i < 32; i += 8)
    if (r0 + i < n && c0 + x < n) t[i][x] = in[(size_t)(r0 + i) * n + c0 + x];
  __syncthreads();
  for (int i = y; i < 32; i += 8)
    if (c0 + i < n && r0 + x < n) out[(size_t)(c0 + i) * n + r0 + x] = t[x][i];
}

}  // namespace

cudaError_t launch_transpose(int n, const double2* in, double2* out, cudaStream_t s) {
  const dim3 g((n + 31) / 32, (n + 31) / 32);
  transpose_kernel<<<g, 256, 0, s>>>(n, in, out);
  return cudaGetLastError();
}

// work (n x n) and chi (n x n) are overwritten; piv[n]
cudaError_t dyson_device(int n, const double2* chi_hf, const double2* U, double2* work, double2* chi, int* piv,
                         int* status, cudaStream_t s) {
  cudaError_t e;
  auto run = [&](cudaError_t x) { return e = x, x == cudaSuccess; };
  int dev = 0, optin = 0;
  if (!run(cudaGetDevice(&dev))) return e;
  if (!run(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev))) return e;
  const size_t solve_smem = sizeof(double2) * (2 * kBlock * kSolveCols + kBlock * kBlock);
  const size_t back_smem = sizeof(double2) * (kBlock * kSolveCols + kBlock * kBlock + kBlock);
  const size_t pan_bytes = sizeof(double2) * (kPan + 1);
  const size_t pan_static = 1024;   // the kernel's own static shared memory, rounded up
  if (!run(cudaFuncSetAttribute(panel_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(optin - pan_static))))
    return e;
  if (!run(cudaFuncSetAttribute(block_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve_smem)))
    return e;
  if (!run(cudaFuncSetAttribute(back_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)back_smem)))
    return e;
  if (!run(zgemm<false>(n, n, n, chi_hf, n, U, n, work, n, 1, s))) return e;   // work = 1 + chi_hf U
  if (!run(cudaMemcpyAsync(chi, chi_hf, sizeof(double2) * (size_t)n * n, cudaMemcpyDeviceToDevice, s))) return e;
  for (int k0 = 0; k0 < n; k0 += kBlock) {
    const int k1 = std::min(n, k0 + kBlock);
    for (int j0 = k0; j0 < k1; j0 += kPan) {
      const int nb = std::min(kPan, k1 - j0);
      const size_t pb = pan_bytes * (size_t)(n - j0);
      if (n - j0 <= kPanThreads)
        panel_rows_kernel<<<1, std::max(64, (n - j0 + 31) / 32 * 32), 0, s>>>(n, j0, nb, work, piv, status);
      else if (pb + pan_static <= (size_t)optin)
        panel_kernel<true><<<1, kPanThreads, pb, s>>>(n, j0, nb, work, piv, status);
      else panel_kernel<false><<<1, kPanThreads, 0, s>>>(n, j0, nb, work, piv, status);
      const int others = k1 - k0 - nb;
      if (others > 0)
        block_update_kernel<<<(others + kUpdCols - 1) / kUpdCols, 512, 0, s>>>(n, j0, nb, k0, k1, work, piv);
    }
    const int nb = k1 - k0;
    const int cols = (n - k1) + n;
    block_solve_kernel<<<(cols + kSolveCols - 1) / kSolveCols, 256, solve_smem, s>>>(n, k0, nb, k1, work, chi, piv);
    const double2* L21 = work + (int64_t)k0 * n + k1;
    if (!run(zgemm<true>(n - k1, n - k1, nb, L21, n, work + (int64_t)k1 * n + k0, n, work + (int64_t)k1 * n + k1, n, 0, s)))
      return e;
    if (!run(zgemm<true>(n - k1, n, nb, L21, n, chi + k0, n, chi + k1, n, 0, s))) return e;
  }
  for (int k0 = (n - 1) / kBlock * kBlock; k0 >= 0; k0 -= kBlock) {
    const int nb = std::min(kBlock, n - k0);
    back_solve_kernel<<<(n + kSolveCols - 1) / kSolveCols, 256, back_smem, s>>>(n, k0, nb, work, chi);
    if (!run(zgemm<true>(k0, n, nb, work + (int64_t)k0 * n, n, chi + k0, n, chi, n, 0, s))) return e;
  }
  return cudaGetLastError();
}

}  // namespace tg
