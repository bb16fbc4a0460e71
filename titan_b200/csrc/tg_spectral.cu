// Spectral Green functions on tabulated k meshes.
//
// When every energy of a pass uses the same k list (uniform imaginary-axis
// meshes, the real-axis BZ), one H(k) serves every (E, k) point of that k.
// H(k) is Hermitian, H = U diag(lambda) U^+, so for every z at once
//   G(k, z) = (z - H(k))^-1 = U diag(1 / (z - lambda)) U^+,
// which for a block of energies is one GEMM with K = dimH:
//   G[z][(r, c)] = sum_a D[z][a] P[a][(r, c)],   D[z][a] = 1 / (z - lambda_a),
//   P[a][(r, c)] = U[r][a] conj(U[c][a]).
// The GEMM runs on the FP64 tensor cores (mma.sync m8n8k4 .f64; tcgen05 has no
// FP64 kind); P is formed on the fly from U in shared memory.  The same form
// gives G - G^+ with D = 2 i Im(1 / (z - lambda)).
//
// The eigendecompositions come from tg_eig.cu (H + dH = U Lambda U^+ with |dH| ~ eps |H|, U
// unitary to eps, eigenvalues as Rayleigh quotients), one per k for all energies and
// frequencies, so G agrees with the inverse to roundoff times |H| / dist(z, spectrum).
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

constexpr int kSpecZ = 16;          // energies of a tile (two m8 fragments)
constexpr int kSpecGroups = 4;      // largest number of 16-energy groups of a task
constexpr int kSpecThreads = 256;

// --------------------------------------------------------------------------- G from (U, lambda)
// not volatile: the scheduler may interleave the MMAs of independent accumulators (a chain on
// one accumulator keeps its order through the data dependence, so results do not change)
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

struct SpecArgs {
  GreenArgs g;
  const double2* U = nullptr;   // [nk][n][n]
  const double* lam = nullptr;  // [nk][n]
  const int* outinv = nullptr;  // [n*n] pair-block slot of (r, c) = r * n + c
  int kp = 0;                   // K padded to a multiple of 4
  int nz = kSpecZ;              // energies per task, a multiple of 16
};

// row stride of U and D in shared memory: 4 mod 8 complex, so that the fragment reads of a
// quarter warp (two rows, four columns) fall into distinct banks
__host__ __device__ inline int spec_stride(int kp) { return kp % 8 == 4 ? kp : kp + 4; }

__host__ __device__ inline size_t spec_smem(int n, int kp, int nz) {
  const int S = spec_stride(kp);
  const int nb = (n + 3) / 4, tiles = nb * (nb + 1) / 2;
  return sizeof(double2) * ((size_t)n * S + (size_t)nz * S) + sizeof(double) * nz + sizeof(int) * nz +
         sizeof(int) * (size_t)tiles;
}

// frexp exponent of max(|Re|, |Im|) read from the bits (exponent field - 1022 for a
// normal number); zero and subnormal values give -32768
__device__ __forceinline__ uint32_t exponent_pair(double2 a, double2 b) {
  return (uint32_t)(uint16_t)exponent_code16(a) | (uint32_t)(uint16_t)exponent_code16(b) << 16;
}

// two adjacent complex numbers, 32-byte aligned, in one store (a whole sector)
__device__ __forceinline__ void store_pair(double2* p, double2 a, double2 b) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y) : "memory");
}

// G = X + i Y with X = sum_a Re(D_a) P_a and Y = sum_a Im(D_a) P_a, both Hermitian because every
// P_a = u_a u_a^H is: only the entries r <= c are formed, G(r, c) = X + i Y and
// G(c, r) = conj(X) + i conj(Y).  One task is a k and up to 64 energies; a warp takes tiles of
// 16 energies and 4 x 4 pairs of the upper triangle (90 % of the tiles' pairs are needed at n = 36,
// 83 % in tiles of 2 x 8), four real DMMAs per 8 pairs, 8 energies and 4 eigenvalues, and a lane
// writes a 2 x 2 block and its mirror image, four runs of 32 bytes.
// Im(D) alone (ANTI: w (G - G^+) = w 2 i Y) takes half of them.  Bound by the FP64 tensor pipe
// (65 %) and, up to n = 36 or so, by the G output as well (16 n^2 bytes per point and operand).
// The spectrum of two spd sites, 0.6 M imaginary and 1.3 M real points: 79 ms with every entry
// formed, 51 ms from one triangle in tiles of 2 x 8 pairs and 16 energies per task, 47 ms now.
template <bool ANTI>
__global__ void __launch_bounds__(kSpecThreads, 2) spec_green_kernel(SpecArgs sa) {
  extern __shared__ __align__(16) unsigned char smem[];
  const GreenArgs& a = sa.g;
  const int n = a.n, kp = sa.kp, nn = n * n, S = spec_stride(kp), nz = sa.nz;
  double2* Us = reinterpret_cast<double2*>(smem);          // [n][S]
  double2* Ds = Us + (size_t)n * S;                         // [nz][S]
  double* ws = reinterpret_cast<double*>(Ds + (size_t)nz * S);
  int* item = reinterpret_cast<int*>(ws + nz);              // pass-local point of each row, -1 = none
  int* tiles = item + nz;                                   // r | c0 << 16
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarp = blockDim.x >> 5;
  const int g8 = lane >> 2, t4 = lane & 3;
  int ntile = 0;
  for (int r0 = 0; r0 < n; r0 += 4)
    for (int c0 = r0; c0 < n; c0 += 4, ++ntile)
      if (ntile % (int)blockDim.x == (int)threadIdx.x) tiles[ntile] = r0 | c0 << 16;
  const int64_t ne = a.n_e;
  const int64_t per_k = (ne + nz - 1) / nz;
  const int64_t ik0 = a.p0 / ne, ik1 = (a.p0 + a.np - 1) / ne;
  const int64_t ntask = (ik1 - ik0 + 1) * per_k;
  // position (p, q) of the output holds G(p, q), or G(q, p) (G^T, and column-major raw G)
  const bool swap = a.mode == MODE_B_IMAG || a.mode == MODE_RAW;
  const bool swap2 = a.mode2 == MODE_B_IMAG;
  const bool scaled = a.mode == MODE_A_IMAG || a.mode == MODE_A_REAL;
  const bool conj = a.mode == MODE_B_REAL;
  for (int64_t t = blockIdx.x; t < ntask; t += gridDim.x) {
    const int64_t ik = ik0 + t / per_k;
    const int64_t ie0 = (t % per_k) * nz;
    const int groups = (int)((min((int64_t)nz, ne - ie0) + kSpecZ - 1) / kSpecZ);
    // rows of this task
    if (threadIdx.x < nz) {
      const int64_t ie = ie0 + threadIdx.x;
      const int64_t wi = ik * ne + ie;
      const bool kept = a.y_side <= 0 || a.pts.kind != 0 || (ie < ne && a.zi + a.ylist[ie] >= a.y_split);
      item[threadIdx.x] = (ie < ne && wi >= a.p0 && wi < a.p0 + a.np && kept) ? (int)(wi - a.p0) : -1;
    }
    const double2* Uk = sa.U + ik * (int64_t)nn;
    for (int e = threadIdx.x; e < n * kp; e += blockDim.x) {
      const int r = e / kp, aa = e % kp;
      if (aa < n) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(Us + r * S + aa)),
                     "l"(Uk + r * n + aa)
                     : "memory");
      } else {
        Us[r * S + aa] = make_double2(0.0, 0.0);
      }
    }
    __syncthreads();
    // D[z][a] and the weights
    const double* lk = sa.lam + ik * n;
    for (int e = threadIdx.x; e < groups * kSpecZ * kp; e += blockDim.x) {
      const int zr = e / kp, aa = e % kp;
      double2 dv = make_double2(0.0, 0.0);
      if (item[zr] >= 0 && aa < n) {
        const int64_t ie = ie0 + zr;
        double x, y;
        if (a.pts.kind == 0) {
          x = a.zr;
          y = a.zi + a.ylist[ie];
        } else {
          x = a.zr + a.pts.x2[ie];
          y = a.zi;
        }
        x -= lk[aa];
        const double s = x * x + y * y;
        if (s == 0.0) {
          if (a.status) {
            const int64_t pidx = a.p0 + item[zr] + 1;
            atomicMin(a.status, (int)(pidx < 0x7fffffff ? pidx : 0x7fffffff));
          }
        } else {
          const double inv = 1.0 / s;
          dv = ANTI ? make_double2(0.0, -2.0 * y * inv) : make_double2(x * inv, -y * inv);
        }
      }
      Ds[zr * S + aa] = dv;
    }
    if (threadIdx.x < nz) {
      double w = 0.0;
      if (item[threadIdx.x] >= 0) {
        const int64_t ie = ie0 + threadIdx.x;
        w = a.pts.kind == 0 ? a.pts.w[ie * a.nk_tab + ik] : a.pts.p2[ie] * a.pts.w[ik];
      }
      ws[threadIdx.x] = w;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // U, under way while D was formed
    __syncthreads();
    for (int tl = warp, z0 = 0;; tl += nwarp) {
      while (tl >= ntile) {
        tl -= ntile;
        z0 += kSpecZ;
      }
      if (z0 >= groups * kSpecZ) break;
      const int r0 = tiles[tl] & 0xffff, c0 = tiles[tl] >> 16;
      // the lane's block of the output: rows r, r + 1 and columns c, c + 1 (n is even, so they
      // exist together); the positions of (r + i, c) and (c + i, r), each starting a pair of
      // adjacent ones, are looked up before the products, which hide the latency
      const int r = r0 + 2 * (t4 & 1), c = c0 + 2 * (t4 >> 1);
      const bool mine = r <= c && c < n;   // (below the diagonal of a diagonal tile: a lane above it has the pair)
      int pu[2] = {0, 0}, pl_[2] = {0, 0};
      if (mine)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          pu[i] = a.mode == MODE_RAW ? (r + i) * n + c : sa.outinv[(r + i) * n + c];
          pl_[i] = a.mode == MODE_RAW ? (c + i) * n + r : sa.outinv[(c + i) * n + r];
        }
      // column j of a product's B fragment: row r0 + j % 4 and column c0 + 2 (j / 4) + f
      const double2* ur = Us + (size_t)min(r0 + (g8 & 3), n - 1) * S + t4;
      const double2* uc = Us + (size_t)min(c0 + 2 * (g8 >> 2), n - 2) * S + t4;
      const double2* dp = Ds + (size_t)(z0 + g8) * S + t4;
      double xr[2][2][2], xi[2][2][2], yr[2][2][2], yi[2][2][2];   // [column f][energy block][row h]
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) xr[i][m][h] = xi[i][m][h] = yr[i][m][h] = yi[i][m][h] = 0.0;
      for (int k0 = 0; k0 < kp; k0 += 4) {
        const double2 uv = ur[k0];
        const double2 pv[2] = {cmul(uv, cconj(uc[k0])), cmul(uv, cconj(uc[S + k0]))};
        const double2 dv[2] = {dp[k0], dp[8 * S + k0]};
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (!ANTI) dmma(xr[i][m][0], xr[i][m][1], dv[m].x, pv[i].x);
            if (!ANTI) dmma(xi[i][m][0], xi[i][m][1], dv[m].x, pv[i].y);
            dmma(yr[i][m][0], yr[i][m][1], dv[m].y, pv[i].x);
            dmma(yi[i][m][0], yi[i][m][1], dv[m].y, pv[i].y);
          }
      }
      if (!mine) continue;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int zr = z0 + m * 8 + g8;
        const int pt = item[zr];
        if (pt < 0) continue;
        const double w = ws[zr];
        double2 up[2][2], lo[2][2];   // G(r + i, c + h), G(c + i, r + h)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            up[h][i] = make_double2(xr[i][m][h] - yi[i][m][h], xi[i][m][h] + yr[i][m][h]);
            lo[i][h] = make_double2(xr[i][m][h] + yi[i][m][h], yr[i][m][h] - xi[i][m][h]);
          }
        auto put = [&](double2* out, int16_t* eout, int pos, double2 v0, double2 v1, bool sc) {
          if (sc) {
            v0 = cscale(v0, w);
            v1 = cscale(v1, w);
          } else if (conj) {
            v0 = cconj(v0);
            v1 = cconj(v1);
          }
          const int64_t o = (int64_t)pt * nn + pos;
          store_pair(out + o, v0, v1);
          if (eout) *reinterpret_cast<uint32_t*>(eout + o) = exponent_pair(v0, v1);
        };
        if (c == r) {
          // positions (r + i, r + h) hold G(r + i, r + h) = up, or its transpose
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            put(a.out, a.eout, pu[i], swap ? up[0][i] : up[i][0], swap ? up[1][i] : up[i][1], scaled);
            if (a.out2)
              put(a.out2, a.eout2, pu[i], swap2 ? up[0][i] : up[i][0], swap2 ? up[1][i] : up[i][1], !swap2);
          }
        } else {
          // G(q, p) at position (p, q): rows r + i take G(c + h, r + i), rows c + i take G(r + h, c + i)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            put(a.out, a.eout, pu[i], swap ? lo[0][i] : up[i][0], swap ? lo[1][i] : up[i][1], scaled);
            put(a.out, a.eout, pl_[i], swap ? up[0][i] : lo[i][0], swap ? up[1][i] : lo[i][1], scaled);
            if (a.out2) {
              put(a.out2, a.eout2, pu[i], swap2 ? lo[0][i] : up[i][0], swap2 ? lo[1][i] : up[i][1], !swap2);
              put(a.out2, a.eout2, pl_[i], swap2 ? up[0][i] : lo[i][0], swap2 ? up[1][i] : lo[i][1], !swap2);
            }
          }
        }
      }
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------- LDOS from (U, lambda)
constexpr int kLdosE = 64;   // energies per CTA: eight per warp

// out[ie][r] += (eta / pi) sum_{k in this CTA's chunk} w_k sum_a |U[k][r][a]|^2 / ((e_ie - lambda_ka)^2 + eta^2),
// i.e. -Im G_rr(k, e + i eta) / pi summed over the chunk (atomicAdd into out): per k a real GEMM
// [energies x n] x [n x n] on the FP64 tensor cores, the weighted |U|^2 and the Lorentzians
// formed in shared memory.  Strides of 4 mod 16 doubles keep the 8-byte fragment reads (eight
// rows, four columns) apart.  NF: column fragments of a warp (all n columns).  Dimension 72, 501
// energies: 7 ms with a thread per energy and row, 0.67 ms now.
__host__ __device__ inline int ldos_stride(int n) { return (n + 11) / 16 * 16 + 4; }

template <int NF>
__global__ void __launch_bounds__(256) spec_ldos_kernel(const double2* __restrict__ U, const double* __restrict__ lam,
                                                        const double* __restrict__ w, int64_t nk, int n,
                                                        const double* __restrict__ e, int n_e, double eta,
                                                        int64_t k_per_cta, double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int S = ldos_stride(n);
  double* P = reinterpret_cast<double*>(smem);   // [8 NF][S] w |U[r][a]|^2 (zero rows and columns past n)
  double* L = P + 8 * NF * S;                     // [kLdosE][S]
  const int e0 = blockIdx.x * kLdosE;
  const int ne = min(kLdosE, n_e - e0);
  const int64_t k0 = (int64_t)blockIdx.y * k_per_cta, k1 = min(nk, k0 + k_per_cta);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int kp = (n + 3) / 4 * 4;
  for (int o = threadIdx.x; o < (8 * NF + kLdosE) * S; o += blockDim.x) P[o] = 0.0;
  double c[NF][2];
#pragma unroll
  for (int f = 0; f < NF; ++f) c[f][0] = c[f][1] = 0.0;
  for (int64_t k = k0; k < k1; ++k) {
    __syncthreads();
    const double2* Uk = U + k * (int64_t)n * n;
    const double wk = w[k];
#pragma unroll 4
    for (int o = threadIdx.x; o < n * n; o += blockDim.x) {
      const double2 u = Uk[o];
      P[(o / n) * S + o % n] = wk * fma(u.x, u.x, u.y * u.y);
    }
#pragma unroll 2
    for (int o = threadIdx.x; o < ne * n; o += blockDim.x) {
      const int ie = o / n, a = o % n;
      const double x = e[e0 + ie] - lam[k * n + a];
      L[ie * S + a] = 1.0 / fma(x, x, eta * eta);
    }
    __syncthreads();
    const double* La = L + (8 * warp + g8) * S + t4;
    const double* Pb = P + g8 * S + t4;
    for (int a = 0; a < kp; a += 4) {
      const double av = La[a];
#pragma unroll
      for (int f = 0; f < NF; ++f) dmma(c[f][0], c[f][1], av, Pb[8 * f * S + a]);
    }
  }
  const double f0 = eta / 3.141592653589793238462643383279502884;
  const int ie = 8 * warp + g8;
  if (ie < ne) {
#pragma unroll
    for (int f = 0; f < NF; ++f)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = 8 * f + 2 * t4 + h;
        if (r < n) atomicAdd(out + (int64_t)(e0 + ie) * n + r, f0 * c[f][h]);
      }
  }
}

// --------------------------------------------------------------------------- expectation sums from (U, lambda)
// For the occupations and moments only the orbital-diagonal spin blocks of G summed over
// the energies of each k are needed:
//   S(r, c) = sum_ie w(ie, k) G_rc(k, z_ie) = sum_a U[r][a] f_a conj(U[c][a]),
//   f_a = sum_ie w(ie, k) / (z_ie - lambda_a),  z_ie = zr + i (zi + y_ie),
// so each k costs n x n_e divisions and 4 n entries of n terms.  out: per-CTA slices of
// [n / 2 orbitals][uu, dd, ud, du] (rows[2 o], rows[2 o + 1] = up / down row of orbital o).
__global__ void __launch_bounds__(256) spec_expect_kernel(const double2* __restrict__ U, const double* __restrict__ lam,
                                                          int64_t nk, int n, const double* __restrict__ ylist,
                                                          int64_t n_e, const double* __restrict__ w, double zr,
                                                          double zi, const int* __restrict__ rows,
                                                          double2* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* f = reinterpret_cast<double2*>(smem);   // [n]
  double2* acc = f + n;                            // [2 n]
  for (int e = threadIdx.x; e < 2 * n; e += blockDim.x) acc[e] = make_double2(0.0, 0.0);
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    __syncthreads();
    for (int a = threadIdx.x; a < n; a += blockDim.x) {
      const double l = lam[k * n + a];
      double fr = 0.0, fi = 0.0;
      const double x = zr - l;
      for (int64_t ie = 0; ie < n_e; ++ie) {
        const double y = zi + ylist[ie];
        const double inv = w[ie * nk + k] / (x * x + y * y);
        fr = fma(x, inv, fr);
        fi = fma(-y, inv, fi);
      }
      f[a] = make_double2(fr, fi);
    }
    __syncthreads();
    const double2* Uk = U + k * (int64_t)n * n;
    for (int e = threadIdx.x; e < 2 * n; e += blockDim.x) {
      const int o = e >> 2, q = e & 3;
      const int ru = rows[2 * o], rd = rows[2 * o + 1];
      const int r = (q == 0 || q == 2) ? ru : rd, c = (q == 0 || q == 3) ? ru : rd;
      double2 s = make_double2(0.0, 0.0);
      for (int a = 0; a < n; ++a) s = cfma(cmul(Uk[(int64_t)r * n + a], f[a]), cconj(Uk[(int64_t)c * n + a]), s);
      acc[e] = cadd(acc[e], s);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * n; e += blockDim.x) partial[(size_t)blockIdx.x * 2 * n + e] = acc[e];
}

}  // namespace

// --------------------------------------------------------------------------- host side
cudaError_t launch_spec_expect(const double2* U, const double* lam, int64_t nk, int n, const double* ylist, int64_t n_e,
                               const double* w, double zr, double zi, const int* rows, double2* partial, int grid,
                               cudaStream_t s) {
  if (nk <= 0) return cudaSuccess;
  const size_t smem = sizeof(double2) * 3 * (size_t)n;
  spec_expect_kernel<<<grid, 256, smem, s>>>(U, lam, nk, n, ylist, n_e, w, zr, zi, rows, partial);
  return cudaGetLastError();
}

cudaError_t launch_spec_ldos(const double2* U, const double* lam, const double* w, int64_t nk, int n,
                             const double* e, int n_e, double eta, double* out, int num_sms, cudaStream_t s) {
  if (nk <= 0 || n_e <= 0) return cudaSuccess;
  if (n > 96) return cudaErrorInvalidValue;
  const int nf = (n + 7) / 8;
  const size_t smem = sizeof(double) * (size_t)ldos_stride(n) * (8 * (nf <= 3 ? 3 : nf <= 6 ? 6 : nf <= 9 ? 9 : 12) + kLdosE);
  auto kernel = nf <= 3   ? spec_ldos_kernel<3>
                : nf <= 6 ? spec_ldos_kernel<6>
                : nf <= 9 ? spec_ldos_kernel<9>
                          : spec_ldos_kernel<12>;
  cudaError_t err = allow_smem(kernel, smem);
  if (err != cudaSuccess) return err;
  err = cudaMemsetAsync(out, 0, sizeof(double) * (size_t)n_e * n, s);
  if (err != cudaSuccess) return err;
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem);
  if (err != cudaSuccess) return err;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  const int eb = (n_e + kLdosE - 1) / kLdosE;
  const int64_t kchunks = std::max<int64_t>(1, std::min<int64_t>(nk, (int64_t)per_sm * num_sms / eb));
  const int64_t kper = (nk + kchunks - 1) / kchunks;
  const dim3 grid((unsigned)eb, (unsigned)((nk + kper - 1) / kper));
  kernel<<<grid, 256, smem, s>>>(U, lam, w, nk, n, e, n_e, eta, kper, out);
  return cudaGetLastError();
}

int spectral_supported(int mode, int mode2, bool has_out2) {
  const bool m = mode == MODE_RAW || mode == MODE_A_IMAG || mode == MODE_B_IMAG || mode == MODE_A_REAL ||
                 mode == MODE_B_REAL;
  if (!m) return 0;
  if (has_out2)
    return (mode == MODE_A_IMAG && mode2 == MODE_B_IMAG) || (mode == MODE_B_IMAG && mode2 == MODE_A_IMAG);
  return 1;
}

cudaError_t launch_green_spectral(const GreenArgs& g, const double2* U, const double* lam, const int* outinv,
                                  int num_sms, cudaStream_t s) {
  if (g.np <= 0) return cudaSuccess;
  if (g.n_e <= 0 || !U || !lam) return cudaErrorInvalidValue;
  if (!spectral_supported(g.mode, g.mode2, g.out2 != nullptr)) return cudaErrorInvalidValue;
  if (g.n % 2 || (g.mode != MODE_RAW && !outinv)) return cudaErrorInvalidValue;   // entries leave in pairs
  SpecArgs sa;
  sa.g = g;
  sa.U = U;
  sa.lam = lam;
  sa.outinv = outinv;
  sa.kp = (g.n + 3) / 4 * 4;
  auto kernel = g.mode == MODE_A_REAL ? spec_green_kernel<true> : spec_green_kernel<false>;
  int dev = 0, optin = 0, smax = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  if (e != cudaSuccess) return e;
  // energies of a task: the more, the fewer loads of U and barriers, as long as two blocks share
  // an SM (one where two could not do with 16 either) and every block has a few tasks
  const int64_t ne = g.n_e;
  const int64_t nks = (g.p0 + g.np - 1) / ne - g.p0 / ne + 1;
  auto tasks = [&](int nz) { return nks * ((ne + nz - 1) / nz); };
  auto blocks = [&](int nz) { return std::min<int64_t>(2, smax / ((int64_t)spec_smem(g.n, sa.kp, nz) + 1024)); };
  for (int nz = kSpecZ * kSpecGroups; nz > kSpecZ; nz /= 2)
    if (spec_smem(g.n, sa.kp, nz) <= (size_t)optin && blocks(nz) == blocks(kSpecZ) &&
        nz - kSpecZ < ne && tasks(nz) >= 4 * blocks(nz) * num_sms) {
      sa.nz = nz;
      break;
    }
  const size_t smem = spec_smem(g.n, sa.kp, sa.nz);
  e = allow_smem(kernel, smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSpecThreads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  const int64_t ntask = tasks(sa.nz);
  const int64_t grid = std::min<int64_t>(ntask, (int64_t)num_sms * per_sm);
  kernel<<<(unsigned)grid, kSpecThreads, smem, s>>>(sa);
  return cudaGetLastError();
}

}  // namespace tg
