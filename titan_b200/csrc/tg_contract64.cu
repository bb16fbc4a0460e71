// FP64 chi0 contraction and epilogues.
//
// The 16 spin-block products of eintshechi.F90:86-104 are, for every site
// pair (i, j), one complex GEMM over the (k, E) points:
//
//   C_ij[u][v] = sum_p A_p[u] B_p[v],   u = (a1 nu, a2 gama), v = (b1 mu, b2 xi)
//
// with A_p = w_p G1_ij and B_p = (G2^T)_ij on the imaginary axis and
// A_p = w_p (G1 - G1^dagger)_ij, B_p = conj(G2)_ij on the real axis
// (eintshechi.F90:146-164).  The chi element is then picked out of C in the
// epilogue (chi = C_ij + conj(C_ji) with permuted indices, Fint = -i D_ij).
// This file holds the FP64 tensor-core GEMM (the plain-precision GPU path) and the
// chi assembly epilogue.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

// One CTA per output tile of 112 x 112 and K-range; points in stages of KC through a cp.async
// ring.  A stage's row of one point is 2 mod 8 complex long, so the fragment reads of a quarter
// warp (four points, two rows) fall into distinct banks.
//
// 112 = 14 fragments: three tiles cover the 324 = 4 9^2 rows of two spd sites to 93 %.  Each of
// the four sub-partitions of the SM (warp id mod 4) takes one 56 x 56 quadrant, 7 x 7 fragments
// of 8 x 8 complex (four real DMMAs m8n8k4 per fragment and four points) dealt to its four
// warps in columns of 2, 2, 2 and 1, so that the four FP64 pipes, which bound the kernel, have
// equal work.  Fragments past the site pair's rows or columns are skipped.  The FP64 tensor pipe
// is 76 % busy; chi at finite q of two spd sites (dimension 648) spent 147 ms here on the scalar
// FP64 units and 115 ms now.
constexpr int KC = 16;            // points per shared-memory stage
constexpr int kStages = 3;
constexpr int kTile = 112;
constexpr int kQuad = kTile / 2;
constexpr int kFM = 7, kFN = 2;   // fragments of a warp
constexpr int kThreads = 512;
constexpr int kLoaders = 4 * kTile;   // threads that copy KC / 4 elements of either operand per stage
constexpr int kS = kTile + 2;
constexpr size_t kSmem = sizeof(double2) * kStages * 2 * KC * kS;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(kThreads, 1)
gemm64_kernel(const double2* __restrict__ A, const double2* __restrict__ B, int64_t ld, int64_t np, int nsplit,
              const PairTile* __restrict__ tiles, const int* __restrict__ pair_M, const int* __restrict__ pair_aoff,
              const int64_t* __restrict__ pair_coff, double2* __restrict__ Cpart, int64_t cstride) {
  extern __shared__ __align__(16) double2 smem64[];   // [stage][A, B][KC][kS]
  const int tile_id = blockIdx.x / nsplit;
  const int split = blockIdx.x % nsplit;
  const PairTile t = tiles[tile_id];
  const int M = pair_M[t.pair];
  const int aoff = pair_aoff[t.pair];
  const int64_t p_begin = np * split / nsplit;
  const int64_t p_end = np * (split + 1) / nsplit;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int wm = (warp & 1) * kQuad, wn = ((warp >> 1) & 1) * kQuad + (warp >> 2) * 8 * kFN;
  // this warp's fragments inside the site pair
  const int fm = max(0, min(kFM, (M - t.u0 - wm + 7) / 8));
  const int fn = max(0, min((warp >> 2) == 3 ? 1 : kFN, (M - t.v0 - wn + 7) / 8));

  double cr[kFM][kFN][2], ci[kFM][kFN][2];
#pragma unroll
  for (int i = 0; i < kFM; ++i)
#pragma unroll
    for (int j = 0; j < kFN; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

  // a loader copies column `col` of the points kk0, kk0 + 4, .. of every stage
  const int kk0 = tid / kTile, col = tid % kTile;
  const bool loads = tid < kLoaders;
  const bool ina = t.u0 + col < M, inb = t.v0 + col < M;
  const double2* ga = A + (p_begin + kk0) * ld + aoff + (ina ? t.u0 + col : 0);
  const double2* gb = B + (p_begin + kk0) * ld + aoff + (inb ? t.v0 + col : 0);
  const unsigned sdst = (unsigned)__cvta_generic_to_shared(smem64 + kk0 * kS + col);
  int left = (int)(p_end - p_begin) - kk0;   // points from this thread's next one to the end
  auto load_stage = [&](int buf) {
    if (loads) {
      const unsigned d = sdst + (unsigned)(buf * 2 * KC * kS * sizeof(double2));
#pragma unroll
      for (int h = 0; h < KC / 4; ++h) {
        const bool in = left > 4 * h;
        const unsigned o = (unsigned)(4 * h * kS * sizeof(double2));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d + o), "l"(in ? ga + 4 * h * ld : A),
                     "r"(in && ina ? 16 : 0));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                         d + o + (unsigned)(KC * kS * sizeof(double2))),
                     "l"(in ? gb + 4 * h * ld : B), "r"(in && inb ? 16 : 0));
      }
      ga += KC * ld;
      gb += KC * ld;
      left -= KC;
    }
  };

  const int64_t nstages = (p_end - p_begin + KC - 1) / KC;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nstages) load_stage(s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  int buf = 0, fill = kStages - 1;   // stage to multiply, stage to load
  for (int64_t s = 0; s < nstages; ++s) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 2));
    __syncthreads();   // stage s has landed, and every warp is done with the one loaded next
    if (s + kStages - 1 < nstages) load_stage(fill);
    fill = fill + 1 == kStages ? 0 : fill + 1;
    asm volatile("cp.async.commit_group;\n" ::);
    const double2* as = smem64 + (size_t)buf * 2 * KC * kS + t4 * kS + wm + g8;
    const double2* bs = smem64 + (size_t)buf * 2 * KC * kS + (KC + t4) * kS + wn + g8;
    buf = buf + 1 == kStages ? 0 : buf + 1;
    if (fn == 0) continue;
#pragma unroll 1
    for (int kk = 0; kk < KC; kk += 4) {
      const double2 b0 = bs[kk * kS];
      if (fn == kFN) {
        const double2 b1 = bs[kk * kS + 8];
#pragma unroll
        for (int i = 0; i < kFM; ++i) {
          if (i >= fm) break;
          const double2 av = as[kk * kS + 8 * i];
          dmma(cr[i][0][0], cr[i][0][1], av.x, b0.x);
          dmma(ci[i][0][0], ci[i][0][1], av.x, b0.y);
          dmma(cr[i][1][0], cr[i][1][1], av.x, b1.x);
          dmma(ci[i][1][0], ci[i][1][1], av.x, b1.y);
          dmma(cr[i][0][0], cr[i][0][1], -av.y, b0.y);
          dmma(ci[i][0][0], ci[i][0][1], av.y, b0.x);
          dmma(cr[i][1][0], cr[i][1][1], -av.y, b1.y);
          dmma(ci[i][1][0], ci[i][1][1], av.y, b1.x);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kFM; ++i) {
          if (i >= fm) break;
          const double2 av = as[kk * kS + 8 * i];
          dmma(cr[i][0][0], cr[i][0][1], av.x, b0.x);
          dmma(ci[i][0][0], ci[i][0][1], av.x, b0.y);
          dmma(cr[i][0][0], cr[i][0][1], -av.y, b0.y);
          dmma(ci[i][0][0], ci[i][0][1], av.y, b0.x);
        }
      }
    }
  }
  double2* C = Cpart + (int64_t)split * cstride + pair_coff[t.pair];
#pragma unroll
  for (int i = 0; i < kFM; ++i) {
    const int u = t.u0 + wm + 8 * i + g8;
    if (i >= fm || u >= M) continue;
#pragma unroll
    for (int j = 0; j < kFN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int v = t.v0 + wn + 8 * j + 2 * t4 + h;
        if (j >= fn || v >= M) continue;
        double2* c = C + (int64_t)u * M + v;
        *c = cadd(*c, make_double2(cr[i][j][h], ci[i][j][h]));
      }
  }
}

// a(s): spin of the G1 side, b(s): spin of the G2 side for chi index s = 1..4
// (0 = up, 1 = down), read off the table of eintshechi.F90:86-104.
__device__ __forceinline__ int spin_a(int s) { return (s == 0 || s == 2) ? 1 : 0; }
__device__ __forceinline__ int spin_b(int s) { return (s >= 2) ? 1 : 0; }

__global__ void chi_epilogue_kernel(const double2* __restrict__ Cpart, const double2* __restrict__ Dpart, int nsplit,
                                    int64_t cstride, int dimens, const int* __restrict__ decode,
                                    const int* __restrict__ norb, const int64_t* __restrict__ pair_coff, int n_atoms,
                                    double scale, double2* __restrict__ chi) {
  const int64_t total = (int64_t)dimens * dimens;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int R = (int)(idx % dimens), Cc = (int)(idx / dimens);   // column-major (Fortran)
    const int dr = decode[R], dc = decode[Cc];
    const int s1 = dr & 3, i = (dr >> 2) & 1023, mu = (dr >> 12) & 63, nu = (dr >> 18) & 63;
    const int s2 = dc & 3, j = (dc >> 2) & 1023, ga = (dc >> 12) & 63, xi = (dc >> 18) & 63;
    const int ni = norb[i], nj = norb[j];
    const int a1 = spin_a(s1), b1 = spin_b(s1), a2 = spin_a(s2), b2 = spin_b(s2);
    // C_ij[(a1 nu, a2 gama), (b1 mu, b2 xi)]
    const int Mij = 4 * ni * nj;
    const int64_t u = (int64_t)(a1 * ni + nu) * (2 * nj) + (a2 * nj + ga);
    const int64_t v = (int64_t)(b1 * ni + mu) * (2 * nj) + (b2 * nj + xi);
    const int64_t off_ij = pair_coff[i * n_atoms + j] + u * Mij + v;
    // C_ji[(a2 gama, a1 nu), (b2 xi, b1 mu)]
    const int64_t u2 = (int64_t)(a2 * nj + ga) * (2 * ni) + (a1 * ni + nu);
    const int64_t v2 = (int64_t)(b2 * nj + xi) * (2 * ni) + (b1 * ni + mu);
    const int64_t off_ji = pair_coff[j * n_atoms + i] + u2 * Mij + v2;
    double2 c1 = make_double2(0, 0), c2 = c1, d = c1;
    for (int sp = 0; sp < nsplit; ++sp) {
      c1 = cadd(c1, Cpart[sp * cstride + off_ij]);
      c2 = cadd(c2, Cpart[sp * cstride + off_ji]);
      if (Dpart) d = cadd(d, Dpart[sp * cstride + off_ij]);
    }
    // chi_imag + Fint, Fint = -i D
    double2 val = cadd(c1, cconj(c2));
    val = cadd(val, make_double2(d.y, -d.x));
    chi[idx] = cscale(val, scale);
  }
}

}  // namespace

cudaError_t launch_gemm64(const double2* A, const double2* B, int64_t ld, int64_t np, int nsplit,
                          const PairTile* tiles, int ntiles, const int* pair_M, const int* pair_aoff,
                          const int64_t* pair_coff, double2* Cpart, int64_t cstride, cudaStream_t s) {
  if (np <= 0 || ntiles <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(gemm64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return e;
  gemm64_kernel<<<ntiles * nsplit, kThreads, kSmem, s>>>(A, B, ld, np, nsplit, tiles, pair_M, pair_aoff, pair_coff,
                                                         Cpart, cstride);
  return cudaGetLastError();
}

cudaError_t launch_chi_epilogue(const double2* Cpart, const double2* Dpart, int nsplit, int64_t cstride,
                                int dimens, const int* decode, const int* norb, const int64_t* pair_coff,
                                int n_atoms, double scale, double2* chi, cudaStream_t s) {
  const int64_t total = (int64_t)dimens * dimens;
  int blocks = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
  chi_epilogue_kernel<<<blocks, 256, 0, s>>>(Cpart, Dpart, nsplit, cstride, dimens, decode, norb, pair_coff,
                                             n_atoms, scale, chi);
  return cudaGetLastError();
}

int gemm64_tile() { return kTile; }

}  // namespace tg
