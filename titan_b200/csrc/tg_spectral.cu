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

constexpr int kSpecZ = 16;          // energies per task (two m8 fragments)
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
};

__host__ __device__ inline size_t spec_smem(int n, int kp) {
  return sizeof(double2) * ((size_t)n * kp + (size_t)kSpecZ * kp) + sizeof(double) * kSpecZ + sizeof(int) * kSpecZ;
}

// (row, col) of G that lands in output slot o for a mode
__device__ __forceinline__ void slot_rc(const SpecArgs& sa, int mode, int o, int& r, int& c) {
  const int n = sa.g.n;
  if (mode == MODE_RAW) {
    r = o % n;
    c = o / n;
    return;
  }
  const int rc = sa.g.outmap[o];
  if (mode == MODE_B_IMAG) {   // G^T
    c = rc / n;
    r = rc % n;
  } else {
    r = rc / n;
    c = rc % n;
  }
}

// frexp exponent of max(|Re|, |Im|) read from the bits (exponent field - 1022 for a
// normal number); zero and subnormal values give -32768
__device__ __forceinline__ int16_t exponent_code(double2 v) {
  const double m = fmax(fabs(v.x), fabs(v.y));
  const int f = (int)((__double_as_longlong(m) >> 52) & 0x7ff);
  return f == 0 ? (int16_t)-32768 : (int16_t)(f - 1022);
}

// five CTAs per SM (the occupancy its ~30 KB of shared memory allows at n = 36): 48
// registers with a 4-byte spill, measured faster than 64 registers at four CTAs
// ANTI (MODE_A_REAL, w (G - G^+)): the diagonal -2i y / |z - lambda|^2 is purely
// imaginary, so two of the four DMMAs per step would multiply by zero and are skipped
// THREADS = 1024 (one CTA per SM) where the shared memory of U leaves room for one CTA only
// (n > 72): 32 warps instead of 8 hide the DMMA and shared-memory latencies
template <bool ANTI, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == kSpecThreads ? 5 : 1) spec_green_kernel(SpecArgs sa) {
  extern __shared__ __align__(16) unsigned char smem[];
  const GreenArgs& a = sa.g;
  const int n = a.n, kp = sa.kp, nn = n * n;
  double2* Us = reinterpret_cast<double2*>(smem);          // [n][kp]
  double2* Ds = Us + (size_t)n * kp;                        // [kSpecZ][kp]
  double* ws = reinterpret_cast<double*>(Ds + (size_t)kSpecZ * kp);
  int* item = reinterpret_cast<int*>(ws + kSpecZ);          // pass-local point of each row, -1 = none
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarp = blockDim.x >> 5;
  const int64_t ne = a.n_e;
  const int64_t per_k = (ne + kSpecZ - 1) / kSpecZ;
  const int64_t ik0 = a.p0 / ne, ik1 = (a.p0 + a.np - 1) / ne;
  const int64_t ntask = (ik1 - ik0 + 1) * per_k;
  const bool anti = ANTI;
  for (int64_t t = blockIdx.x; t < ntask; t += gridDim.x) {
    const int64_t ik = ik0 + t / per_k;
    const int64_t ie0 = (t % per_k) * kSpecZ;
    // rows of this task
    if (threadIdx.x < kSpecZ) {
      const int64_t ie = ie0 + threadIdx.x;
      const int64_t wi = ik * ne + ie;
      const bool kept = a.y_side <= 0 || a.pts.kind != 0 || (ie < ne && a.zi + a.ylist[ie] >= a.y_split);
      item[threadIdx.x] = (ie < ne && wi >= a.p0 && wi < a.p0 + a.np && kept) ? (int)(wi - a.p0) : -1;
    }
    const double2* Uk = sa.U + ik * (int64_t)nn;
    for (int e = threadIdx.x; e < n * kp; e += blockDim.x) {
      const int r = e / kp, aa = e % kp;
      Us[e] = aa < n ? Uk[r * n + aa] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    // D[z][a] and the weights
    const double* lk = sa.lam + ik * n;
    for (int e = threadIdx.x; e < kSpecZ * kp; e += blockDim.x) {
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
          dv = anti ? make_double2(0.0, -2.0 * y * inv) : make_double2(x * inv, -y * inv);
        }
      }
      Ds[e] = dv;
    }
    if (threadIdx.x < kSpecZ) {
      double w = 0.0;
      if (item[threadIdx.x] >= 0) {
        const int64_t ie = ie0 + threadIdx.x;
        w = a.pts.kind == 0 ? a.pts.w[ie * a.nk_tab + ik] : a.pts.p2[ie] * a.pts.w[ik];
      }
      ws[threadIdx.x] = w;
    }
    __syncthreads();
    // G tiles: 16 energies x 8 output slots per warp step
    const int g8 = lane >> 2, t4 = lane & 3;
    const int nfrag = (nn + 7) / 8;
    for (int nf = warp; nf < nfrag; nf += nwarp) {
      int rb = 0, cb = 0;
      const int ob = nf * 8 + g8;
      if (ob < nn) slot_rc(sa, a.mode, ob, rb, cb);
      const double2* ur = Us + (size_t)rb * kp;
      const double2* uc = Us + (size_t)cb * kp;
      double cr[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, ci[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
      for (int k0 = 0; k0 < kp; k0 += 4) {
        const int ka = k0 + t4;
        const double2 pv = cmul(ur[ka], cconj(uc[ka]));
#pragma unroll
        for (int mf = 0; mf < 2; ++mf) {
          const double2 dv = Ds[(mf * 8 + g8) * kp + ka];
          if (!ANTI) dmma(cr[mf][0], cr[mf][1], dv.x, pv.x);
          dmma(cr[mf][0], cr[mf][1], -dv.y, pv.y);
          if (!ANTI) dmma(ci[mf][0], ci[mf][1], dv.x, pv.y);
          dmma(ci[mf][0], ci[mf][1], dv.y, pv.x);
        }
      }
#pragma unroll
      for (int mf = 0; mf < 2; ++mf) {
        const int zr = mf * 8 + g8;
        const int pl = item[zr];
        if (pl < 0) continue;
        const double w = ws[zr];
        // the lane's two slots are adjacent (nn is even): one 4-byte store of both exponents
        const int o0 = nf * 8 + 2 * t4;
        uint32_t codes = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int o = o0 + j;
          if (o >= nn) continue;
          const double2 v = make_double2(cr[mf][j], ci[mf][j]);
          double2 v1 = v;
          if (a.mode == MODE_A_IMAG || a.mode == MODE_A_REAL) v1 = cscale(v, w);
          else if (a.mode == MODE_B_REAL) v1 = cconj(v);
          a.out[(int64_t)pl * nn + o] = v1;
          codes |= (uint32_t)(uint16_t)exponent_code(v1) << (16 * j);
          if (a.out2) {
            // the other imaginary-axis operand of the same G: v = G[r][c] goes to slot
            // (c, r) of the G^T layout (mode2 B) or, times w, to slot (r, c) of the G layout (mode2 A)
            int r, c;
            slot_rc(sa, a.mode, o, r, c);
            const bool tr = a.mode2 == MODE_B_IMAG;
            const int64_t i2 = (int64_t)pl * nn + sa.outinv[tr ? c * n + r : r * n + c];
            const double2 v2 = tr ? v : cscale(v, w);
            a.out2[i2] = v2;
            if (a.eout2) a.eout2[i2] = exponent_code(v2);
          }
        }
        if (a.eout && o0 < nn) *reinterpret_cast<uint32_t*>(a.eout + (int64_t)pl * nn + o0) = codes;
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
// rows, four columns) apart.  NF: column fragments of a warp (all n columns).
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
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
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
  if (g.out2 && !outinv) return cudaErrorInvalidValue;
  if ((g.eout || g.eout2) && g.n % 2) return cudaErrorInvalidValue;   // paired 4-byte exponent stores
  SpecArgs sa;
  sa.g = g;
  sa.U = U;
  sa.lam = lam;
  sa.outinv = outinv;
  sa.kp = (g.n + 3) / 4 * 4;
  const size_t smem = spec_smem(g.n, sa.kp);
  const bool anti = g.mode == MODE_A_REAL;
  auto kernel = anti ? spec_green_kernel<true, kSpecThreads> : spec_green_kernel<false, kSpecThreads>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSpecThreads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  int threads = kSpecThreads;
  if (per_sm == 1) {
    kernel = anti ? spec_green_kernel<true, 1024> : spec_green_kernel<false, 1024>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 1024, smem);
    if (e != cudaSuccess) return e;
    if (per_sm <= 0) return cudaErrorInvalidValue;
    threads = 1024;
  }
  const int64_t ne = g.n_e;
  const int64_t ntask = ((g.p0 + g.np - 1) / ne - g.p0 / ne + 1) * ((ne + kSpecZ - 1) / kSpecZ);
  const int64_t grid = std::min<int64_t>(ntask, (int64_t)num_sms * per_sm);
  kernel<<<(unsigned)grid, threads, smem, s>>>(sa);
  return cudaGetLastError();
}

}  // namespace tg
