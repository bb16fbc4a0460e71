// Weighted sums over the Green functions of a pass (column-major, MODE_RAW): products of
// entries for the Jacobian, its adjoint and the exchange coupling, single entries for the
// on-site blocks, and the sum of per-CTA partial results.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

constexpr int kPairThreads = 256;

// stride of a matrix staged in shared memory: 1 mod 8 complex, so that neighbouring rows and
// neighbouring columns fall into distinct banks
__host__ __device__ inline int pair_stride(int n) { return (n + 6) / 8 * 8 + 1; }

// A pair is an orbital a of one site and an orbital b of another (or the same), as the rows
// (a up, a down, b up, b down); per pair and point p
//   acc[s' + 2 t + 4 t' + 8 s] += w_p Ga(a s', b t) Gb(b t', a s)
// and, where Ga and Gb differ, the same with the two exchanged in the second half of the npairs =
// 2 nlist sums (both from one reading of the matrices),
// into the CTA's slice of acc (zeroed before the first pass of a call).
// A thread owns one pair for the whole launch, its 16 sums in registers; tpm threads share a
// point (blockDim / tpm points at a time), blockIdx.y takes tpm pairs each.  STAGED: the
// point's matrices are copied to shared memory first, where the 8 entries of a pair-point (64
// FMAs) cost as many cycles as its arithmetic; otherwise (two matrices beyond the shared
// memory) they are read through L1.  Bound by the reading of G (16 n^2 bytes per matrix): the
// GG tensor of 29160 matrices of dimension 72 takes 1.5 ms beside 6.6 ms for their inversion (46 ms
// together when the inversion kernel formed the products itself, from one CTA's registers).
template <bool STAGED>
__global__ void __launch_bounds__(kPairThreads, 2) pair_kernel(GreenArgs g, const double2* __restrict__ Ga,
                                                            const double2* __restrict__ Gb,
                                                            const int4* __restrict__ pairs, int nlist, int npairs,
                                                            int tpm,
                                                            double2* __restrict__ acc) {
  extern __shared__ __align__(16) double2 psm[];
  const int n = g.n, S = STAGED ? pair_stride(n) : n;
  const int64_t nn = (int64_t)n * n;
  const int slots = blockDim.x / tpm;
  const int m = threadIdx.x / tpm, lt = threadIdx.x % tpm;
  const int pi = blockIdx.y * tpm + lt;
  const bool two = Ga != Gb;
  const int64_t mat = (int64_t)n * S;
  const bool mine = m < slots && pi < npairs;
  const int4 pr = mine ? pairs[pi % nlist] : make_int4(0, 0, 0, 0);
  const bool swapped = pi >= nlist;   // second half of a two-matrix call: Gb in the first factor
  double2 s16[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) s16[q] = make_double2(0.0, 0.0);
  for (int64_t base = (int64_t)blockIdx.x * slots; base < g.np; base += (int64_t)gridDim.x * slots) {
    const int64_t pl = base + m;
    const double2 *xa, *xb;
    if (STAGED) {
      const int here = (int)min((int64_t)slots, g.np - base);
      for (int k = 0; k < (two ? 2 : 1); ++k) {
        const double2* src = (k ? Gb : Ga) + base * nn;
        double2* dst = psm + k * slots * mat;
        for (int e = threadIdx.x; e < here * (int)nn; e += blockDim.x) {
          const int mm = e / (int)nn, rc = e - mm * (int)nn, c = rc / n, r = rc - c * n;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                           (unsigned)__cvta_generic_to_shared(dst + mm * mat + c * S + r)),
                       "l"(src + e));
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
      asm volatile("cp.async.wait_group 0;\n" ::);
      __syncthreads();
      xa = psm + (m < slots ? m : 0) * mat;
      xb = two ? xa + slots * mat : xa;
    } else {
      xa = Ga + pl * nn;
      xb = Gb + pl * nn;
    }
    if (mine && pl < g.np) {
      const double w = point_weight(g, pl);
      if (swapped) {
        const double2* t = xa;
        xa = xb;
        xb = t;
      }
      const int ra[2] = {pr.x, pr.y}, rb[2] = {pr.z, pr.w};
      double2 u[2][2], v[2][2];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          u[s][t] = cscale(xa[(int64_t)rb[t] * S + ra[s]], w);   // Ga(a s, b t)
          v[t][s] = xb[(int64_t)ra[s] * S + rb[t]];              // Gb(b t, a s)
        }
#pragma unroll
      for (int q = 0; q < 16; ++q) s16[q] = cfma(u[q & 1][(q >> 1) & 1], v[(q >> 2) & 1][(q >> 3) & 1], s16[q]);
    }
    if (STAGED) __syncthreads();
  }
  if (mine) {
    double2* dst = acc + (((int64_t)blockIdx.x * slots + m) * npairs + pi) * 16;
#pragma unroll
    for (int q = 0; q < 16; ++q) dst[q] = cadd(dst[q], s16[q]);
  }
}

// acc[blockIdx.x][e] += sum_p w_p G_p(entries[e].x, entries[e].y); one thread per entry
__global__ void __launch_bounds__(256) entries_kernel(GreenArgs g, const double2* __restrict__ G,
                                                      const int2* __restrict__ entries, int ne,
                                                      double2* __restrict__ acc) {
  const int e = blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  const int2 rc = entries[e];
  const int64_t nn = (int64_t)g.n * g.n;
  const double2* x = G + (int64_t)rc.y * g.n + rc.x;
  double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int64_t pl = blockIdx.x; pl < g.np; pl += gridDim.x) {
    const double w = point_weight(g, pl);
    const double2 v = x[pl * nn];
    s.x = fma(w, v.x, s.x);
    s.y = fma(w, v.y, s.y);
  }
  double2* dst = acc + (int64_t)blockIdx.x * ne + e;
  *dst = cadd(*dst, s);
}

// out[e] = sum_b part[b][e]: 32 entries per CTA, the partials dealt to 8 thread rows
__global__ void __launch_bounds__(256) reduce_blocks_kernel(const double2* __restrict__ part, int nblocks, int len,
                                                            double2* __restrict__ out) {
  __shared__ double2 sum[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + x;
  double2 s = make_double2(0.0, 0.0);
  if (e < len) {
#pragma unroll 4
    for (int b = y; b < nblocks; b += 8) s = cadd(s, part[(int64_t)b * len + e]);
  }
  sum[y][x] = s;
  __syncthreads();
  if (y == 0 && e < len) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s = cadd(s, sum[k][x]);
    out[e] = s;
  }
}

struct PairPlan {
  int tpm, slots, tiles, grid;
  bool staged;
  size_t smem;
};

// threads per point: the pairs in equal tiles of at most kPairThreads; several points per CTA
// where they are few.  A CTA needs one matrix (two when Ga and Gb differ) per point.
cudaError_t pair_plan(int n, int npairs, bool two, int num_sms, int64_t np, PairPlan& p) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  p.tiles = (npairs + kPairThreads - 1) / kPairThreads;
  p.tpm = ((npairs + p.tiles - 1) / p.tiles + 31) / 32 * 32;
  const size_t mat = sizeof(double2) * (size_t)n * pair_stride(n) * (two ? 2 : 1);
  p.slots = std::max(1, kPairThreads / p.tpm);
  while (p.slots > 1 && mat * p.slots > (size_t)optin / 2) --p.slots;
  p.staged = mat * p.slots <= (size_t)optin;
  p.smem = p.staged ? mat * p.slots : 0;
  const int per_sm = p.smem * 2 + 4096 <= (size_t)optin ? 2 : 1;
  p.grid = (int)std::max<int64_t>(1, std::min<int64_t>((np + p.slots - 1) / p.slots,
                                                       std::max(1, num_sms * per_sm / p.tiles)));
  return cudaSuccess;
}

}  // namespace

size_t pair_partials(int n, int nlist, bool two, int num_sms, int64_t np) {
  PairPlan p;
  const int npairs = two ? 2 * nlist : nlist;
  if (npairs <= 0 || pair_plan(n, npairs, two, num_sms, np, p) != cudaSuccess) return 1;
  return (size_t)p.grid * p.slots;
}

cudaError_t launch_pairs(const GreenArgs& g, const double2* Ga, const double2* Gb, const int4* pairs, int nlist,
                         int num_sms, double2* acc, cudaStream_t s) {
  if (nlist <= 0 || g.np <= 0) return cudaSuccess;
  const int npairs = Ga != Gb ? 2 * nlist : nlist;
  PairPlan p;
  cudaError_t e = pair_plan(g.n, npairs, Ga != Gb, num_sms, g.np, p);
  if (e != cudaSuccess) return e;
  const dim3 grid(p.grid, p.tiles);
  if (p.staged) {
    e = allow_smem(pair_kernel<true>, p.smem);
    if (e != cudaSuccess) return e;
    pair_kernel<true><<<grid, p.tpm * p.slots, p.smem, s>>>(g, Ga, Gb, pairs, nlist, npairs, p.tpm, acc);
  } else {
    pair_kernel<false><<<grid, p.tpm * p.slots, 0, s>>>(g, Ga, Gb, pairs, nlist, npairs, p.tpm, acc);
  }
  return cudaGetLastError();
}

int entry_partials(int64_t np, int num_sms) { return (int)std::max<int64_t>(1, std::min<int64_t>(np, num_sms * 2)); }

cudaError_t launch_entries(const GreenArgs& g, const double2* G, const int2* entries, int ne, int num_sms,
                           double2* acc, cudaStream_t s) {
  if (ne <= 0 || g.np <= 0) return cudaSuccess;
  const dim3 grid(entry_partials(g.np, num_sms), (ne + 255) / 256);
  entries_kernel<<<grid, 256, 0, s>>>(g, G, entries, ne, acc);
  return cudaGetLastError();
}

cudaError_t launch_reduce_blocks(const double2* part, int nblocks, int len, double2* out, cudaStream_t s) {
  if (len <= 0) return cudaSuccess;
  reduce_blocks_kernel<<<(len + 31) / 32, 256, 0, s>>>(part, nblocks, len, out);
  return cudaGetLastError();
}

}  // namespace tg
