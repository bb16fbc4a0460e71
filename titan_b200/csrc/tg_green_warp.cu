// Warp-per-matrix fused H(k) + complex Gauss-Jordan inversion, FP64, for dimensions 4, 8, 16, 20.
//
// A warp owns one (k, z) matrix at a time.  Its lanes form a 4 x 8 grid; lane (tr, tc) keeps rows
// r = tr + 4 rr and columns c = tc + 8 cc in registers (cyclic distribution, padded slots are an
// inert identity).  Per elimination step k = tck + 8 kk (slot kk compile-time, lane column tck
// runtime):
//   * the lanes owning column k pick the largest |Re|+|Im| among the rows not yet used (the
//     zgetrf/izamax choice) by shuffles;
//   * the owners of row p publish the scaled pivot row a_p/a_pk, the owners of column k the
//     multipliers (a_pk - 1 for row p itself, so the update below needs no branch), both in the
//     warp's shared memory, double-buffered by step parity: one __syncwarp per step;
//   * every lane applies  a <- a - f * pvd  to its register block.
// Rows are never swapped; G[r][s] = X[piv[r]][pinv[s]] is applied when the result leaves through
// the output stage.  The warps are persistent and independent; H(k) comes either from a
// precomputed table (k-major walk, so each table row is reused from L2 across energies) or is
// summed here.
#include "tg_internal.cuh"

namespace tg {

namespace {

constexpr int kWarps = 8;        // largest number of matrices of a CTA
constexpr int TR = 4, TC = 8;    // lane grid

template <int N>
struct WarpDim {
  static constexpr int RB = (N + TR - 1) / TR;
  static constexpr int CB = (N + TC - 1) / TC;
  static constexpr int NR = TR * RB;
  static constexpr int NC = TC * CB;
};

struct WarpSmem {
  size_t stage, bufs, phase, piv, pinv, zw, acc, per_warp;
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~size_t(15); }

__host__ __device__ inline WarpSmem warp_smem(int n, int nr, int nc, int n_neigh) {
  WarpSmem L;
  size_t o = 0;
  L.stage = o; o = al16(o + sizeof(double2) * (size_t)n * n);
  L.bufs = o;  o = al16(o + sizeof(double2) * 2 * (size_t)(nr + nc));
  L.phase = o; o = al16(o + sizeof(double2) * (size_t)(n_neigh > 0 ? n_neigh : 1));
  L.piv = o;   o = al16(o + sizeof(int) * (size_t)n);
  L.pinv = o;  o = al16(o + sizeof(int) * (size_t)n);
  L.zw = o;    o = al16(o + sizeof(double) * 8);
  L.acc = o;   o = al16(o + sizeof(double2) * 2 * (size_t)n);           // MODE_EXPECT sums (4 per orbital)
  L.per_warp = o;
  return L;
}

__device__ __forceinline__ double2 shfl_d2(double2 v, int src) {
  v.x = __shfl_sync(0xffffffffu, v.x, src);
  v.y = __shfl_sync(0xffffffffu, v.y, src);
  return v;
}

// OUT: 0 = operand / raw outputs, 1 = MODE_EXPECT, 2 = MODE_HK
template <int N, int OUT>
__global__ void __launch_bounds__(32 * kWarps, 1) green_warp_kernel(GreenArgs a) {
  using D = WarpDim<N>;
  constexpr int RB = D::RB, CB = D::CB, NR = D::NR, NC = D::NC;
  extern __shared__ __align__(16) unsigned char smem[];
  const WarpSmem L = warp_smem(N, NR, NC, a.n_neigh);
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* base = smem + (size_t)warp * L.per_warp;
  double2* X = reinterpret_cast<double2*>(base + L.stage);
  double2* bufs = reinterpret_cast<double2*>(base + L.bufs);
  double2* phase = reinterpret_cast<double2*>(base + L.phase);
  int* piv = reinterpret_cast<int*>(base + L.piv);
  int* pinv = reinterpret_cast<int*>(base + L.pinv);
  double* zw = reinterpret_cast<double*>(base + L.zw);
  double2* eacc = reinterpret_cast<double2*>(base + L.acc);
  const int tr = lane / TC, tc = lane % TC;

  if (OUT == 1) {
    for (int e = lane; e < 2 * N; e += 32) eacc[e] = make_double2(0, 0);
  }
  __syncwarp();

  const int64_t nwarps = (int64_t)gridDim.x * warps;
  for (int64_t pl = (int64_t)blockIdx.x * warps + warp; pl < a.np; pl += nwarps) {
    // ---- point data ------------------------------------------------------------
    int64_t ktab = -1;
    if (a.htab) ktab = (a.p0 + pl) / a.n_e;
    if (lane == 0) {
      double zr, zi, kx = 0, ky = 0, kz = 0, w;
      if (a.htab) {
        const int64_t wi = a.p0 + pl;
        const int64_t ik = wi / a.n_e, ie = wi % a.n_e;
        if (a.pts.kind == 0) {
          zr = a.zr;
          zi = a.zi + a.ylist[ie];
          w = a.pts.w[ie * a.nk_tab + ik];
        } else {
          zr = a.zr + a.pts.x2[ie];
          zi = a.zi;
          w = a.pts.p2[ie] * a.pts.w[ik];
        }
      } else {
        const int64_t p = a.p0 + pl;
        if (a.pts.kind == 0) {
          zr = a.zr;
          zi = a.zi + a.pts.y[p];
          kx = a.pts.kp[3 * p]; ky = a.pts.kp[3 * p + 1]; kz = a.pts.kp[3 * p + 2];
          w = a.pts.w[p];
        } else if (a.pts.kind == 1) {
          const int64_t nep = p / a.pts.nk, ik = p % a.pts.nk;
          zr = a.zr + a.pts.x2[nep];
          zi = a.zi;
          kx = a.pts.kp[3 * ik]; ky = a.pts.kp[3 * ik + 1]; kz = a.pts.kp[3 * ik + 2];
          w = a.pts.p2[nep] * a.pts.w[ik];
        } else {
          zr = a.pts.z[p].x;
          zi = a.pts.z[p].y;
          kx = a.pts.kp[3 * p]; ky = a.pts.kp[3 * p + 1]; kz = a.pts.kp[3 * p + 2];
          w = 1.0;
        }
      }
      zw[0] = zr; zw[1] = zi; zw[2] = kx + a.q[0]; zw[3] = ky + a.q[1]; zw[4] = kz + a.q[2]; zw[5] = w;
    }
    __syncwarp();
    if (ktab < 0) {
      const double kx = zw[2], ky = zw[3], kz = zw[4];
      for (int nb = lane; nb < a.n_neigh; nb += 32) {
        const double th = kx * a.R[3 * nb] + ky * a.R[3 * nb + 1] + kz * a.R[3 * nb + 2];
        double s, c;
        sincos(th, &s, &c);
        phase[nb] = make_double2(c, s);
      }
      __syncwarp();
    }

    // ---- A = z 1 - H(k) into registers ------------------------------------------
    double2 A[RB][CB];
    {
      const double2 zc = make_double2(zw[0], zw[1]);
#pragma unroll
      for (int rr = 0; rr < RB; ++rr) {
        const int r = tr + TR * rr;
#pragma unroll
        for (int cc = 0; cc < CB; ++cc) {
          const int c = tc + TC * cc;
          double2 v = make_double2(r == c ? 1.0 : 0.0, 0.0);   // inert padding
          if (r < N && c < N) {
            double2 h;
            if (ktab >= 0) {
              h = a.htab[ktab * (N * N) + r * N + c];
            } else {
              h = a.h0[(size_t)c * N + r];
              if (a.row_spin[r] == a.row_spin[c]) {
                const int orr = a.row_orb[r], oc = a.row_orb[c];
                const int pb = a.row_atom[r] * a.n_atoms + a.row_atom[c];
                for (int b = a.pair_start[pb]; b < a.pair_start[pb + 1]; ++b)
                  h = cfma(phase[a.pair_neigh[b]], a.pair_t[(size_t)b * a.nmax * a.nmax + oc * a.nmax + orr], h);
              }
            }
            v = make_double2(-h.x, -h.y);
            if (r == c) v = cadd(v, zc);
          }
          A[rr][cc] = v;
        }
      }
    }

    if (OUT == 2) {
      const double2 zc = make_double2(zw[0], zw[1]);
#pragma unroll
      for (int rr = 0; rr < RB; ++rr)
#pragma unroll
        for (int cc = 0; cc < CB; ++cc) {
          const int r = tr + TR * rr, c = tc + TC * cc;
          if (r < N && c < N) {
            double2 v = A[rr][cc];
            if (r == c) v = csub(v, zc);
            a.out[pl * N * N + (size_t)c * N + r] = make_double2(-v.x, -v.y);
          }
        }
      __syncwarp();
      continue;
    }

    // ---- Gauss-Jordan with implicit partial pivoting -----------------------------
    unsigned used = 0u;     // bit rr: row tr + TR*rr already used as a pivot row
    for (int k = lane; k < N; k += 32) pinv[k] = k;   // (stays valid where rows are used twice, see below)
    bool singular = false;
#pragma unroll
    for (int kk = 0; kk < CB; ++kk) {
#pragma unroll 1
      for (int tck = 0; tck < TC; ++tck) {
        const int k = tck + TC * kk;
        if (k >= N) break;
        const int buf = k & 1;
        const bool own_col = (tc == tck);
        double best = -1.0;
        int brow = 0x7fffffff;
        double2 bval = make_double2(0, 0);
        if (own_col) {
#pragma unroll
          for (int rr = 0; rr < RB; ++rr) {
            const int r = tr + TR * rr;
            const double v = fabs(A[rr][kk].x) + fabs(A[rr][kk].y);
            if (r < N && !((used >> rr) & 1u) && (v > best || (v == best && r < brow))) {
              best = v;
              brow = r;
              bval = A[rr][kk];
            }
          }
        }
        // reduce over the lanes of lane column tck
#pragma unroll
        for (int m = TC; m < 32; m <<= 1) {
          const double ob = __shfl_xor_sync(0xffffffffu, best, m);
          const int orow = __shfl_xor_sync(0xffffffffu, brow, m);
          const double2 oval = shfl_d2(bval, lane ^ m);
          if (ob > best || (ob == best && orow < brow)) {
            best = ob;
            brow = orow;
            bval = oval;
          }
        }
        best = __shfl_sync(0xffffffffu, best, tck);
        // (a column of nothing but NaN: any row will do, the point is flagged and its result not used)
        const int p = min(__shfl_sync(0xffffffffu, brow, tck), N - 1);
        const double2 apk = shfl_d2(bval, tck);
        if (!(best > 0.0)) singular = true;
        const double2 d = crecip_fast(apk);
        const int ptr = p % TR, prr = p / TR;
        double2* pvd = bufs + buf * (NR + NC);
        double2* fcol = pvd + NC;
        if (tr == ptr) {
#pragma unroll
          for (int cc = 0; cc < CB; ++cc) {
            double2 v = A[0][cc];
#pragma unroll
            for (int rr = 1; rr < RB; ++rr)
              if (rr == prr) v = A[rr][cc];
            pvd[tc + TC * cc] = (cc == kk && own_col) ? d : cmul(v, d);
          }
          used |= 1u << prr;
        }
        if (own_col) {
#pragma unroll
          for (int rr = 0; rr < RB; ++rr) {
            const int r = tr + TR * rr;
            double2 f = A[rr][kk];
            if (r == p) f.x -= 1.0;
            fcol[r] = f;
          }
        }
        if (lane == 0) piv[k] = p;
        __syncwarp();
        double2 pv[CB];
#pragma unroll
        for (int cc = 0; cc < CB; ++cc) pv[cc] = pvd[tc + TC * cc];
#pragma unroll
        for (int rr = 0; rr < RB; ++rr) {
          const int r = tr + TR * rr;
          const double2 f = fcol[r];
          if (own_col) A[rr][kk] = make_double2(r == p ? 1.0 : 0.0, 0.0);
#pragma unroll
          for (int cc = 0; cc < CB; ++cc) A[rr][cc] = cfms(f, pv[cc], A[rr][cc]);
        }
      }
    }
    if (lane == 0 && singular && a.status) {
      const int64_t pidx = a.p0 + pl + 1;
      atomicMin(a.status, (int)(pidx < 0x7fffffff ? pidx : 0x7fffffff));
    }
    // ---- stage X and the permutation in shared memory --------------------------
#pragma unroll
    for (int rr = 0; rr < RB; ++rr)
#pragma unroll
      for (int cc = 0; cc < CB; ++cc) {
        const int r = tr + TR * rr, c = tc + TC * cc;
        if (r < N && c < N) X[r * N + c] = A[rr][cc];
      }
    __syncwarp();
    for (int k = lane; k < N; k += 32) pinv[piv[k]] = k;
    __syncwarp();

    // ---- output stage -----------------------------------------------------------
    const int NN = N * N;
    const double w = zw[5];
    if (OUT == 0) {
      const int nout = a.out2 ? 2 : 1;
      for (int slot = 0; slot < nout; ++slot) {
        const int mode = slot == 0 ? a.mode : a.mode2;
        double2* dst = (slot == 0 ? a.out : a.out2) + pl * (int64_t)NN;
        for (int o = lane; o < NN; o += 32) {
          double2 v;
          if (mode == MODE_RAW) {
            const int r = o % N, c = o / N;
            v = X[piv[r] * N + pinv[c]];
          } else {
            const int rc = a.outmap[o];
            const int r = rc / N, c = rc % N;
            if (mode == MODE_A_IMAG) {
              v = cscale(X[piv[r] * N + pinv[c]], w);
            } else if (mode == MODE_B_IMAG) {
              v = X[piv[c] * N + pinv[r]];
            } else if (mode == MODE_A_REAL) {
              v = cscale(csub(X[piv[r] * N + pinv[c]], cconj(X[piv[c] * N + pinv[r]])), w);
            } else {
              v = cconj(X[piv[r] * N + pinv[c]]);
            }
          }
          dst[o] = v;
        }
      }
    } else if (OUT == 1) {
      for (int o = lane; o < N / 2; o += 32) {
        const int ru = a.exp_rows[2 * o], rd = a.exp_rows[2 * o + 1];
        eacc[4 * o + 0] = cadd(eacc[4 * o + 0], cscale(X[piv[ru] * N + pinv[ru]], w));
        eacc[4 * o + 1] = cadd(eacc[4 * o + 1], cscale(X[piv[rd] * N + pinv[rd]], w));
        eacc[4 * o + 2] = cadd(eacc[4 * o + 2], cscale(X[piv[ru] * N + pinv[rd]], w));
        eacc[4 * o + 3] = cadd(eacc[4 * o + 3], cscale(X[piv[rd] * N + pinv[ru]], w));
      }
    }
    __syncwarp();
  }

  if (OUT == 1) {
    __syncwarp();
    double2* dst = a.acc + ((size_t)blockIdx.x * warps + warp) * (2 * N);
    for (int e = lane; e < 2 * N; e += 32) dst[e] = eacc[e];
  }
}

template <int N, int OUT>
cudaError_t launch_o(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  using D = WarpDim<N>;
  const WarpSmem L = warp_smem(N, D::NR, D::NC, a.n_neigh);
  int dev = 0;
  cudaGetDevice(&dev);
  int max_smem = 0;
  cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  int warps = kWarps;
  while (warps > 1 && L.per_warp * warps > (size_t)max_smem) --warps;
  const size_t smem = L.per_warp * warps;
  if (smem > (size_t)max_smem) return cudaErrorInvalidValue;
  auto kern = green_warp_kernel<N, OUT>;
  cudaError_t err = allow_smem(kern, smem);
  if (err != cudaSuccess) return err;
  const int threads = 32 * warps;
  int per_sm = 0;
  err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
  if (err != cudaSuccess) return err;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  // partial sums of MODE_EXPECT: at most 8 + warps - 1 matrices per SM at a time
  if (per_sm * warps > kWarps) per_sm = (kWarps + warps - 1) / warps;
  int64_t grid = (int64_t)num_sms * per_sm;
  const int64_t need = (a.np + warps - 1) / warps;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  if (grid_used) *grid_used = (int)grid * warps;   // partial slots (one per warp)
  kern<<<(unsigned)grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_n(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  if (a.mode == MODE_EXPECT) return launch_o<N, 1>(a, num_sms, s, grid_used);
  if (a.mode == MODE_HK) return launch_o<N, 2>(a, num_sms, s, grid_used);
  return launch_o<N, 0>(a, num_sms, s, grid_used);
}

}  // namespace

// Warp-per-matrix path: raw / operand / expectation / H(k) modes.
int green_warp_supported(int n, int mode) {
  const bool nok = n == 4 || n == 8 || n == 16 || n == 20;
  const bool mok = mode == MODE_RAW || mode == MODE_A_IMAG || mode == MODE_B_IMAG || mode == MODE_A_REAL ||
                   mode == MODE_B_REAL || mode == MODE_EXPECT || mode == MODE_HK;
  return nok && mok;
}

cudaError_t launch_green_warp(const GreenArgs& a, int num_sms, cudaStream_t s, int* grid_used) {
  if (a.np <= 0) {
    if (grid_used) *grid_used = 0;
    return cudaSuccess;
  }
  switch (a.n) {
    case 4: return launch_n<4>(a, num_sms, s, grid_used);
    case 8: return launch_n<8>(a, num_sms, s, grid_used);
    case 16: return launch_n<16>(a, num_sms, s, grid_used);
    case 20: return launch_n<20>(a, num_sms, s, grid_used);
  }
  return cudaErrorInvalidValue;
}

}  // namespace tg
