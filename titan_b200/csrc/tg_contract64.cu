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

// One CTA per output tile and K-range: WM x WN warps of FM x FN fragments (8 x 8 complex, four
// real DMMAs m8n8k4 per fragment and four points), points in stages of KC through a cp.async
// ring.  A stage's row of one point is 2 mod 8 complex longer than the tile, so the fragment
// reads of a quarter warp (four points, two rows) fall into distinct banks.
//   112 x 112 (7 x 2 warps of 2 x 7): three tiles cover the 324 = 4 9^2 rows of two spd sites
//     (93 % of the tile area used)
//   104 x 104 (13 x 1 warps of 1 x 13): the 100 = 4 5^2 rows of the d orbitals (92 %)
// Bound by the FP64 tensor pipe: 56 (52) DMMAs per warp, four points and 9 (14) shared-memory
// reads.
constexpr int KC = 8;             // points per shared-memory stage
constexpr int kStages = 3;

template <int WM, int WN, int FM, int FN>
struct Gemm64 {
  static constexpr int TILE = 8 * WM * FM;
  static_assert(TILE == 8 * WN * FN, "square tiles");
  static constexpr int THREADS = 32 * WM * WN;
  static constexpr int S = TILE + (TILE % 8 == 0 ? 2 : 0);
  static constexpr size_t smem = sizeof(double2) * kStages * 2 * KC * S;
};
using GemmWide = Gemm64<7, 2, 2, 7>;
using GemmD = Gemm64<13, 1, 1, 13>;

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

template <int WM, int WN, int FM, int FN>
__global__ void __launch_bounds__(32 * WM * WN, 1)
gemm64_kernel(const double2* __restrict__ A, const double2* __restrict__ B, int64_t ld, int64_t np, int nsplit,
              const PairTile* __restrict__ tiles, const int* __restrict__ pair_M, const int* __restrict__ pair_aoff,
              const int64_t* __restrict__ pair_coff, double2* __restrict__ Cpart, int64_t cstride) {
  using G = Gemm64<WM, WN, FM, FN>;
  constexpr int TILE = G::TILE, S = G::S, T = G::THREADS;
  extern __shared__ __align__(16) double2 smem64[];   // [stage][A, B][KC][S]
  const int tile_id = blockIdx.x / nsplit;
  const int split = blockIdx.x % nsplit;
  const PairTile t = tiles[tile_id];
  const int M = pair_M[t.pair];
  const int aoff = pair_aoff[t.pair];
  const int64_t p_begin = np * split / nsplit;
  const int64_t p_end = np * (split + 1) / nsplit;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g8 = lane >> 2, t4 = lane & 3;
  const int wm = (warp % WM) * 8 * FM, wn = (warp / WM) * 8 * FN;

  double cr[FM][FN][2], ci[FM][FN][2];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j) cr[i][j][0] = cr[i][j][1] = ci[i][j][0] = ci[i][j][1] = 0.0;

  // a thread copies column `col` of the points kk and kk + 4 of every stage
  static_assert(2 * T == KC * TILE, "two elements of either operand per thread and stage");
  const int kk0 = tid / TILE, col = tid % TILE;
  const bool ina = t.u0 + col < M, inb = t.v0 + col < M;
  const double2* ga = A + (p_begin + kk0) * ld + aoff + (ina ? t.u0 + col : 0);
  const double2* gb = B + (p_begin + kk0) * ld + aoff + (inb ? t.v0 + col : 0);
  const unsigned sdst = (unsigned)__cvta_generic_to_shared(smem64 + kk0 * S + col);
  int left = (int)(p_end - p_begin) - kk0;   // points from this thread's next one to the end
  auto load_stage = [&](int buf) {
    const unsigned d = sdst + (unsigned)(buf * 2 * KC * S * sizeof(double2));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool in = left > 4 * h;
      const unsigned o = (unsigned)(4 * h * S * sizeof(double2));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d + o), "l"(in ? ga + 4 * h * ld : A),
                   "r"(in && ina ? 16 : 0));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       d + o + (unsigned)(KC * S * sizeof(double2))),
                   "l"(in ? gb + 4 * h * ld : B), "r"(in && inb ? 16 : 0));
    }
    ga += KC * ld;
    gb += KC * ld;
    left -= KC;
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
    const double2* as = smem64 + (size_t)buf * 2 * KC * S + t4 * S + wm + g8;
    const double2* bs = smem64 + (size_t)buf * 2 * KC * S + (KC + t4) * S + wn + g8;
    buf = buf + 1 == kStages ? 0 : buf + 1;
#pragma unroll 1
    for (int kk = 0; kk < KC; kk += 4) {
      double2 av[FM];
#pragma unroll
      for (int i = 0; i < FM; ++i) av[i] = as[kk * S + 8 * i];
#pragma unroll
      for (int j = 0; j < FN; ++j) {
        const double2 bv = bs[kk * S + 8 * j];
#pragma unroll
        for (int i = 0; i < FM; ++i) {
          dmma(cr[i][j][0], cr[i][j][1], av[i].x, bv.x);
          dmma(ci[i][j][0], ci[i][j][1], av[i].x, bv.y);
        }
#pragma unroll
        for (int i = 0; i < FM; ++i) {
          dmma(cr[i][j][0], cr[i][j][1], -av[i].y, bv.y);
          dmma(ci[i][j][0], ci[i][j][1], av[i].y, bv.x);
        }
      }
    }
  }
  double2* C = Cpart + (int64_t)split * cstride + pair_coff[t.pair];
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    const int u = t.u0 + wm + 8 * i + g8;
    if (u >= M) continue;
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int v = t.v0 + wn + 8 * j + 2 * t4 + h;
        if (v >= M) continue;
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

namespace {

template <int WM, int WN, int FM, int FN>
cudaError_t launch_gemm64_t(const double2* A, const double2* B, int64_t ld, int64_t np, int nsplit,
                            const PairTile* tiles, int ntiles, const int* pair_M, const int* pair_aoff,
                            const int64_t* pair_coff, double2* Cpart, int64_t cstride, cudaStream_t s) {
  using G = Gemm64<WM, WN, FM, FN>;
  auto kernel = gemm64_kernel<WM, WN, FM, FN>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem);
  if (e != cudaSuccess) return e;
  kernel<<<ntiles * nsplit, G::THREADS, G::smem, s>>>(A, B, ld, np, nsplit, tiles, pair_M, pair_aoff, pair_coff, Cpart,
                                                     cstride);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_gemm64(const double2* A, const double2* B, int64_t ld, int64_t np, int nsplit, int tile,
                          const PairTile* tiles, int ntiles, const int* pair_M, const int* pair_aoff,
                          const int64_t* pair_coff, double2* Cpart, int64_t cstride, cudaStream_t s) {
  if (np <= 0 || ntiles <= 0) return cudaSuccess;
  if (tile == GemmD::TILE)
    return launch_gemm64_t<13, 1, 1, 13>(A, B, ld, np, nsplit, tiles, ntiles, pair_M, pair_aoff, pair_coff, Cpart,
                                         cstride, s);
  return launch_gemm64_t<7, 2, 2, 7>(A, B, ld, np, nsplit, tiles, ntiles, pair_M, pair_aoff, pair_coff, Cpart, cstride,
                                     s);
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

// tile side for the site pairs of a layout (pair_M[n_pairs] rows each): the one whose tiles
// cover the smaller area (DMMAs of the padding cost as much as the others), 112 on ties
int gemm64_tile(int n_pairs, const int* pair_M) {
  double wide = 0.0, d = 0.0;
  for (int i = 0; i < n_pairs; ++i) {
    const double a = (pair_M[i] + GemmWide::TILE - 1) / GemmWide::TILE * GemmWide::TILE;
    const double b = (pair_M[i] + GemmD::TILE - 1) / GemmD::TILE * GemmD::TILE;
    wide += a * a;
    d += b * b;
  }
  return d < wide ? GemmD::TILE : GemmWide::TILE;
}

}  // namespace tg
