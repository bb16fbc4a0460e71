// Eigendecompositions and tridiagonalisations of an H(k) table, one Hermitian matrix per k.
//
// Four kernels, each parallel over the k in its own way:
//   1. hh_small_kernel: H = Q T Q^H, T real symmetric tridiagonal (the Householder reduction of
//      LAPACK's zhetd2, lower form, with zlarfg's reflectors), one CTA per k with the matrix in
//      shared memory; Q is accumulated backwards in place.  Also used for the resolvents of
//      tg_tridiag.cu at dimensions up to 96.
//   2. ql_kernel: T = Z diag(lambda) Z^T by the implicitly shifted QL iteration (Martin and
//      Wilkinson, 1968; Dubrulle, 1970), one thread per k with d and e in shared memory.
//      The iteration is a serial chain of n^2 plane rotations, so only the number of k hides
//      it; its rotations go to global memory.
//   3. eig_apply_kernel: U = Q Z, one CTA per k with Q in shared memory and a thread per real
//      row (rotations of columns act on every row alone, without any barrier).
//   4. eig_finish_kernel: one Newton-Schulz step U <- U (1 - (U^H U - 1) / 2) and Rayleigh
//      quotients of H for the eigenvalues, its products on the FP64 tensor cores.
// About 46 n^3 flops per matrix (reduction and Q 16/3 n^3 each, 1.3 n^2 rotations of 2 n real rows
// 16 n^3, post-pass 20 n^3) against the 10 sweeps of 24 n^3 of a cyclic Jacobi iteration, whose
// rotations also need a CTA barrier per round.  Measured: 9801 matrices of dimension 36 in
// 24 ms with Jacobi rotations, 3.7 ms now (1.5, 0.5, 1.1 and 0.6 ms for the four kernels); 1331 of
// dimension 72 in 45 ms and 5.5 ms, of which the serial chains of ql_kernel take 1.7 ms.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

constexpr int kHhMax = 96;          // largest dimension of hh_small_kernel (three rows per lane)
constexpr int kHhThreads = 480;
constexpr int kQlIterations = 60;   // per eigenvalue

__host__ __device__ inline int odd_stride(int n) { return n | 1; }

__device__ __forceinline__ double2 warp_sum2(double2 v) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  return v;
}

// --------------------------------------------------------------------------- 1. tridiagonalisation
// B holds A column by column with an odd stride (A(r, c) at c S + r), both triangles.  The warps
// share the trailing block by 32 rows (a lane per row, so the vector entry of a column is one
// broadcast) and by columns; for Q by 32 columns and by rows.  Per reflector: norm and vector
// (warp 0), product A v with the column parts added up through shared memory, update
//   A <- A - v p^H - q v^H,  p = tau A v, q = p - Re(tau p^H v) v,
// four barriers; per reflector of Q two.  The loops read four entries before they write the
// first (the compiler cannot tell the stores from the next loads apart).  Bound by shared
// memory: 15 wavefronts per 32 entries and reflector for the reduction, 14 for Q (29 and 23
// with neighbouring lanes on the columns of a row), n^3 / 3 entries each.
constexpr int kHhBatch = 4;

__global__ void __launch_bounds__(kHhThreads) hh_small_kernel(const double2* __restrict__ H, int64_t nk, int n,
                                                            const int* __restrict__ rows, int ns,
                                                            double* __restrict__ D, double* __restrict__ E,
                                                            double2* __restrict__ Q) {
  extern __shared__ __align__(16) double2 hsm[];
  const int S = odd_stride(n);
  double2* B = hsm;
  double2* v = B + n * S;
  double2* p = v + n;
  double2* taus = p + n;
  double2* dots = taus + n;     // [3] per 32 rows, then tau of the step
  double2* parts = dots + 4;    // [warps][32]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const double2 zero = make_double2(0.0, 0.0);
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    const double2* Hk = H + k * (int64_t)n * n;
#pragma unroll 4
    for (int e = tid; e < n * n; e += blockDim.x) B[(e % n) * S + e / n] = Hk[e];
    __syncthreads();
    for (int j = 0; j + 1 < n; ++j) {
      const int m = n - j - 1;
      double2* col = B + j * S + j + 1;
      if (warp == 0) {
        double2 x[3];
        double part = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int r = lane + 32 * i;
          x[i] = r < m ? col[r] : zero;
          if (r > 0) part = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, part));
        }
        double2 alpha = col[0];
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        double down = 1.0;
        if (reflector_norm2(alpha, part) < kReflectorTiny) {   // (the same in every lane)
          part = 0.0;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            x[i] = cscale(x[i], kReflectorUp);
            if (lane + 32 * i > 0) part = fma(x[i].x, x[i].x, fma(x[i].y, x[i].y, part));
          }
          for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
          alpha = cscale(alpha, kReflectorUp);
          down = kReflectorDown;
        }
        const Reflector h = reflector(alpha, part);
        if (h.any) {
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int r = lane + 32 * i;
            if (r < m) {
              const double2 vr = r == 0 ? make_double2(1.0, 0.0) : cmul(x[i], h.sc);
              v[r] = vr;
              col[r] = vr;   // kept for Q; the column is done with
            }
          }
        }
        if (lane == 0) {
          D[k * n + j] = B[j * S + j].x;
          E[k * n + j] = h.beta * down;
          taus[j] = h.tau;
        }
      }
      __syncthreads();
      const double2 tau = taus[j];
      if (tau.x == 0.0 && tau.y == 0.0) continue;   // no reflector (the same in every thread)
      // row block and column part of this warp
      const int nrb = (m + 31) >> 5, np = nw / nrb;
      const int rb = warp % nrb, cp = warp / nrb, r = 32 * rb + lane;
      double2* Ar = B + (j + 1) * S + j + 1 + r;
      const bool mine = cp < np && r < m;
      double2 acc = zero, acc1 = zero;
      if (mine) {
        int c = cp;
        for (; c + 3 * np < m; c += 4 * np) {
          acc = cfma(Ar[c * S], v[c], acc);
          acc1 = cfma(Ar[(c + np) * S], v[c + np], acc1);
          acc = cfma(Ar[(c + 2 * np) * S], v[c + 2 * np], acc);
          acc1 = cfma(Ar[(c + 3 * np) * S], v[c + 3 * np], acc1);
        }
        for (; c < m; c += np) acc = cfma(Ar[c * S], v[c], acc);
      }
      parts[32 * warp + lane] = cadd(acc, acc1);
      __syncthreads();
      if (cp == 0) {
        double2 a = zero;
        for (int q = 0; q < np; ++q) a = cadd(a, parts[32 * (q * nrb + rb) + lane]);
        const double2 pr = cmul(tau, a);
        if (r < m) p[r] = pr;
        const double2 d = warp_sum2(r < m ? cmul(cconj(pr), v[r]) : zero);
        if (lane == 0) dots[rb] = d;
      }
      __syncthreads();
      if (mine) {
        double2 dot = dots[0];
        for (int q = 1; q < nrb; ++q) dot = cadd(dot, dots[q]);
        const double t2 = -cmul(tau, dot).x;   // 2 Re(-tau (p^H v) / 2)
        const double2 vr = v[r], pr = p[r];
        const double2 qr = make_double2(fma(t2, vr.x, pr.x), fma(t2, vr.y, pr.y));
        for (int c0 = cp; c0 < m; c0 += kHhBatch * np) {
          double2 a[kHhBatch];
#pragma unroll
          for (int u = 0; u < kHhBatch; ++u) {
            const int c = c0 + u * np;
            a[u] = c < m ? cfms(qr, cconj(v[c]), cfms(vr, cconj(p[c]), Ar[c * S])) : zero;
          }
#pragma unroll
          for (int u = 0; u < kHhBatch; ++u)
            if (c0 + u * np < m) Ar[(c0 + u * np) * S] = a[u];
        }
      }
      __syncthreads();
    }
    if (tid == 0) {
      D[k * n + n - 1] = B[(n - 1) * S + n - 1].x;
      E[k * n + n - 1] = 0.0;
    }
    // Q = H_0 H_1 .. H_{n-2} backwards: step j fills the block of rows and columns > j
    for (int j = n - 2; j >= 0; --j) {
      const int m = n - j - 1;
      const double2 tau = taus[j];
      const bool refl = tau.x != 0.0 || tau.y != 0.0;
      const double2* vj = B + j * S + j + 1;
      const int nrb = (m + 31) >> 5, np = nw / nrb;
      const int rb = warp % nrb, rp = warp / nrb, ct = 32 * rb + lane;   // this thread's column, row part
      const bool mine = rp < np && ct < m;
      double2* col = B + (j + 1 + ct) * S + j + 1;
      if (refl) {
        double2 y = zero, y1 = zero;
        if (mine && ct > 0) {
          int r = 1 + rp;
          for (; r + 3 * np < m; r += 4 * np) {
            y = cfma(cconj(vj[r]), col[r], y);
            y1 = cfma(cconj(vj[r + np]), col[r + np], y1);
            y = cfma(cconj(vj[r + 2 * np]), col[r + 2 * np], y);
            y1 = cfma(cconj(vj[r + 3 * np]), col[r + 3 * np], y1);
          }
          for (; r < m; r += np) y = cfma(cconj(vj[r]), col[r], y);
        }
        parts[32 * warp + lane] = cadd(y, y1);
      }
      __syncthreads();
      if (mine) {
        double2 y = zero;
        if (ct == 0) y = make_double2(1.0, 0.0);   // column j + 1 enters as a unit vector
        else if (refl)
          for (int q = 0; q < np; ++q) y = cadd(y, parts[32 * (q * nrb + rb) + lane]);
        const double2 ty = cmul(tau, y);
        if (refl || ct == 0)
          for (int r0 = 1 + rp; r0 < m; r0 += kHhBatch * np) {
            double2 a[kHhBatch];
#pragma unroll
            for (int u = 0; u < kHhBatch; ++u) {
              const int r = r0 + u * np;
              const double2 vr = refl && r < m ? vj[r] : zero;   // (no reflector: the unit vector stays)
              a[u] = cfms(ty, vr, ct > 0 && r < m ? col[r] : zero);
            }
#pragma unroll
            for (int u = 0; u < kHhBatch; ++u)
              if (r0 + u * np < m) col[r0 + u * np] = a[u];
          }
        if (rp == 0) col[0] = make_double2((ct == 0 ? 1.0 : 0.0) - ty.x, -ty.y);
      }
      __syncthreads();
    }
    double2* Qk = Q + k * (int64_t)ns * n;
#pragma unroll 2
    for (int e = tid; e < ns * n; e += blockDim.x) {
      const int s = e / n, c = e - s * n;
      const int r = rows ? rows[s] : s;
      Qk[e] = r == 0 || c == 0 ? make_double2(r == c ? 1.0 : 0.0, 0.0) : B[c * S + r];
    }
    __syncthreads();
  }
}

// --------------------------------------------------------------------------- 2. QL iteration
// d, e: [nk][n]; rot: [nk][cap] (c, s) in the order they act, sweep: [nk][scap] lowest column
// l | top column m << 16 of each sweep (its rotations act on columns (i, i + 1), i = m - 1 .. l),
// nsweep: [nk].  A lane whose lists would overflow, or an eigenvalue that does not settle, sets
// status.  `lanes` matrices per warp: the warp runs as long as the longest sweep of its lanes, so
// few matrices are spread over more warps.
__global__ void __launch_bounds__(32) ql_kernel(const double* __restrict__ D, const double* __restrict__ E,
                                                int64_t k0, int64_t nk, int n, double* __restrict__ lam,
                                                double2* __restrict__ rot, int cap, int* __restrict__ sweep, int scap,
                                                int* __restrict__ nsweep, int lanes, int* __restrict__ status) {
  extern __shared__ __align__(16) double qsm[];
  const int lane = threadIdx.x;
  const int64_t kl = (int64_t)blockIdx.x * lanes + lane;
  if (lane >= lanes || kl >= nk) return;   // (no barrier below)
  const int64_t k = k0 + kl;
  double* d = qsm + lane;            // d[32 i]
  double* e = qsm + 32 * n + lane;   // e[32 i]
  double an = 0.0;
  for (int i = 0; i < n; ++i) {
    const double di = D[k * n + i], ei = i + 1 < n ? E[k * n + i] : 0.0;
    d[32 * i] = di;
    e[32 * i] = ei;
    an = fmax(an, fabs(di) + fabs(ei));
  }
  double2* rk = rot + kl * cap;
  int* sk = sweep + kl * scap;
  int nr = 0, nsw = 0;
  bool ok = true;
  const double tiny = 1e-17 * an;
  for (int l = 0; l < n && ok; ++l) {
    for (int it = 0;; ++it) {
      int m = l;
      for (; m + 1 < n; ++m)
        if (fabs(e[32 * m]) <= 0x1p-53 * (fabs(d[32 * m]) + fabs(d[32 * (m + 1)])) + tiny) break;
      if (m == l) break;
      if (it == kQlIterations || nr + (m - l) > cap || nsw == scap) {
        ok = false;
        break;
      }
      // shift: the eigenvalue of the leading 2 x 2 block nearer d_l
      const double dl = d[32 * l], el = e[32 * l];
      double g = (d[32 * (l + 1)] - dl) / (2.0 * el);
      g = d[32 * m] - dl + el / (g + copysign(sqrt(fma(g, g, 1.0)), g));
      double s = 1.0, c = 1.0, pp = 0.0, dn = d[32 * m];
      sk[nsw++] = l | m << 16;
      for (int i = m - 1; i >= l; --i) {
        const double ei = e[32 * i], di = d[32 * i];
        const double f = s * ei, b = c * ei;
        const double q = fma(f, f, g * g);
        double ir, r;
        if (q > 1e-280) {
          ir = rsqrt(q);
          r = q * ir;
        } else {   // both below 1e-140: scaled
          const double big = fmax(fabs(f), fabs(g));
          const double fs = big > 0.0 ? f / big : 0.0, gs = big > 0.0 ? g / big : 1.0;
          const double rs = sqrt(fma(fs, fs, gs * gs));
          r = big * rs;
          ir = 0.0;
          s = fs / rs;
          c = gs / rs;
        }
        e[32 * (i + 1)] = r;
        if (ir != 0.0) {
          s = f * ir;
          c = g * ir;
        }
        // the pair (c, s) is a rotation to the last digit: s^2 + c^2 within rounding of 1
        g = dn - pp;
        const double t = fma(di - g, s, 2.0 * c * b);
        pp = s * t;
        d[32 * (i + 1)] = g + pp;
        g = fma(c, t, -b);
        dn = di;
        rk[nr++] = make_double2(c, s);
      }
      d[32 * l] = dn - pp;
      e[32 * l] = g;
      e[32 * m] = 0.0;
    }
  }
  nsweep[kl] = nsw;
  for (int i = 0; i < n; ++i) lam[k * n + i] = d[32 * i];
  if (!ok) atomicMin(status, (int)(k < 0x7ffffffe ? k + 1 : 0x7fffffff));
}

// --------------------------------------------------------------------------- 3. vectors
// The Hermitian n x n scratch of the post-pass: the full array (odd stride), or (PACKED, where
// it does not fit beside U) the upper triangle column by column.
template <bool PACKED>
struct HermA {
  double2* a;
  int n, S;
  __device__ __forceinline__ double2 get(int i, int j) const {   // (PACKED)
    return i <= j ? a[j * (j + 1) / 2 + i] : cconj(a[i * (i + 1) / 2 + j]);
  }
  __host__ __device__ static int entries(int n) { return PACKED ? n * (n + 1) / 2 : n * n; }
  __host__ __device__ static size_t storage(int n) {
    return PACKED ? (size_t)n * (n + 1) / 2 : (size_t)n * odd_stride(n);
  }
  __device__ __forceinline__ int at(int i, int j) const { return PACKED ? j * (j + 1) / 2 + i : i * S + j; }
  // (i, j) of entry e (i <= j when PACKED)
  __device__ __forceinline__ void ij(int e, int& i, int& j) const {
    if (!PACKED) {
      i = e / n;
      j = e - i * n;
      return;
    }
    j = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
    while (j * (j + 1) / 2 > e) --j;
    while ((j + 1) * (j + 2) / 2 <= e) ++j;
    i = e - j * (j + 1) / 2;
  }
};

constexpr int kEigCols = 3;   // columns per lane of the post-pass row products: n <= 96
constexpr int kFinThreads = 256;

constexpr int kEigFrags = 9;   // largest NF of the post-pass: n <= 72 without packing

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}

// c += X Y (or X^H Y) for the 8 x 8 fragment at (i0, j0) of two n x n matrices in shared memory
// (stride S), on the FP64 tensor cores: the lane's columns j0 + 2 t4, j0 + 2 t4 + 1 of row i0 + g8
template <bool HERM>
__device__ __forceinline__ void frag_product(const double2* X, const double2* Y, int n, int S, int i0, int j0,
                                             double2& c0, double2& c1) {
  const int lane = threadIdx.x & 31, g8 = lane >> 2, t4 = lane & 3;
  const int i = min(i0 + g8, n - 1), j = min(j0 + g8, n - 1);   // clamped: those results are not used
#pragma unroll 2
  for (int k0 = 0; k0 < n; k0 += 4) {
    const int k = k0 + t4;
    const bool in = k < n;
    double2 a = in ? (HERM ? X[k * S + i] : X[i * S + k]) : make_double2(0.0, 0.0);
    const double2 b = in ? Y[k * S + j] : make_double2(0.0, 0.0);
    if (HERM) a.y = -a.y;
    dmma(c0.x, c1.x, a.x, b.x);
    dmma(c0.y, c1.y, a.x, b.y);
    dmma(c0.x, c1.x, -a.y, b.y);
    dmma(c0.y, c1.y, a.y, b.x);
  }
}

// U <- Q Z for every k: U holds Q on entry (row-major).  A thread per real row (Re or Im part of a
// row of Q), which the rotations of columns combine with nothing else; they are staged through
// shared memory as many whole sweeps at a time as kRotRoom holds.  Bound by shared memory: one
// 8-byte load and store per row and rotation.
constexpr int kRotRoom = 512;

__global__ void __launch_bounds__(192) eig_apply_kernel(int64_t nk, int n, const double2* __restrict__ rot, int cap,
                                                        const int* __restrict__ sweep, int scap,
                                                        const int* __restrict__ nsweep, double2* __restrict__ Uio) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int S = odd_stride(n);
  double2* U = reinterpret_cast<double2*>(smem);   // [n][S]
  double2* stage = U + n * S;                      // [kRotRoom]
  const int tid = threadIdx.x;
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    double2* Uk = Uio + k * (int64_t)n * n;
#pragma unroll 4
    for (int e = tid; e < n * n; e += blockDim.x) U[(e / n) * S + e % n] = Uk[e];
    double* row = reinterpret_cast<double*>(U + (tid >> 1) * S) + (tid & 1);
    const double2* rk = rot + k * cap;
    const int* sk = sweep + k * scap;
    const int nsw = nsweep[k];
    __syncthreads();
    for (int w0 = 0; w0 < nsw;) {
      int w1 = w0, cnt = 0;
      while (w1 < nsw) {
        const int lm = sk[w1], len = (lm >> 16) - (lm & 0xffff);
        if (w1 > w0 && cnt + len > kRotRoom) break;   // (one sweep, n - 1 rotations, always fits)
        cnt += len;
        ++w1;
      }
      for (int e = tid; e < cnt; e += blockDim.x) stage[e] = rk[e];
      __syncthreads();
      if (tid < 2 * n) {
        const double2* t = stage;
        for (int w = w0; w < w1; ++w) {
          const int lm = sk[w], l = lm & 0xffff, m = lm >> 16;
          double x = row[2 * m];
          int i = m - 1;
          for (; i >= l + 3; i -= 4, t += 4) {
            const double f0 = row[2 * i], f1 = row[2 * i - 2], f2 = row[2 * i - 4], f3 = row[2 * i - 6];
            const double2 r0 = t[0], r1 = t[1], r2 = t[2], r3 = t[3];
            row[2 * i + 2] = fma(r0.y, f0, r0.x * x);
            x = fma(r0.x, f0, -(r0.y * x));
            row[2 * i] = fma(r1.y, f1, r1.x * x);
            x = fma(r1.x, f1, -(r1.y * x));
            row[2 * i - 2] = fma(r2.y, f2, r2.x * x);
            x = fma(r2.x, f2, -(r2.y * x));
            row[2 * i - 4] = fma(r3.y, f3, r3.x * x);
            x = fma(r3.x, f3, -(r3.y * x));
          }
          for (; i >= l; --i, ++t) {
            const double f = row[2 * i];
            row[2 * i + 2] = fma(t->y, f, t->x * x);
            x = fma(t->x, f, -(t->y * x));
          }
          row[2 * l] = x;
        }
      }
      __syncthreads();
      rk += cnt;
      w0 = w1;
    }
#pragma unroll 4
    for (int e = tid; e < n * n; e += blockDim.x) Uk[e] = U[(e / n) * S + e % n];
    __syncthreads();
  }
}

// Post-pass: H: [nk][n][n] row-major; U: in Q Z, out the eigenvectors U[r][a]; lam: [nk][n].
// NF: 8-column fragments of a row block in registers (n <= 8 NF)
template <bool PACKED, int NF>
__global__ void __launch_bounds__(kFinThreads) eig_finish_kernel(const double2* __restrict__ H, int64_t nk, int n,
                                                                 double2* __restrict__ Uio, double* __restrict__ lam) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int S = odd_stride(n);
  double2* U = reinterpret_cast<double2*>(smem);   // [n][S]
  const HermA<PACKED> A{U + n * S, n, S};
  const int na = HermA<PACKED>::entries(n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
  const int g8 = lane >> 2, t4 = lane & 3;
  for (int64_t k = blockIdx.x; k < nk; k += gridDim.x) {
    const double2* Hk = H + k * (int64_t)n * n;
    double2* Uk = Uio + k * (int64_t)n * n;
#pragma unroll 4
    for (int e = tid; e < n * n; e += blockDim.x) U[(e / n) * S + e % n] = Uk[e];
    __syncthreads();
    // Post-pass: re-orthonormalised vectors and Rayleigh-quotient eigenvalues.
    //  (1) E = U^H U - 1 (Hermitian)
    if (!PACKED) {
      const int nf = (n + 7) / 8;
      for (int f = warp; f < nf * nf; f += nwarps) {
        const int fi = f / nf, fj = f % nf;
        if (fj < fi) continue;   // its transpose is written with the upper fragment
        double2 c0 = make_double2(0.0, 0.0), c1 = c0;
        frag_product<true>(U, U, n, S, 8 * fi, 8 * fj, c0, c1);
        const int i = 8 * fi + g8, j = 8 * fj + 2 * t4;
        if (i < n && j < n) {   // (n is even: j + 1 < n too)
          if (i == j) c0.x -= 1.0;
          if (i == j + 1) c1.x -= 1.0;
          A.a[i * S + j] = c0;
          A.a[i * S + j + 1] = c1;
          if (fj > fi) {
            A.a[j * S + i] = cconj(c0);
            A.a[(j + 1) * S + i] = cconj(c1);
          }
        }
      }
    } else {
      for (int e = tid; e < na; e += blockDim.x) {
        int i, j;
        A.ij(e, i, j);
        double2 acc = make_double2(i == j ? -1.0 : 0.0, 0.0);
        for (int r = 0; r < n; ++r) acc = cfma(cconj(U[r * S + i]), U[r * S + j], acc);
        A.a[A.at(i, j)] = acc;
      }
    }
    __syncthreads();
    //  (2) one Newton-Schulz step U <- U (1 - E / 2): a warp per 8 rows (or per row), the rows
    //  read before they are written
    if (!PACKED) {
      const int nf = (n + 7) / 8;
      for (int fi = warp; fi < nf; fi += nwarps) {
        double2 c[2 * NF];
#pragma unroll
        for (int fj = 0; fj < NF; ++fj) {
          c[2 * fj] = c[2 * fj + 1] = make_double2(0.0, 0.0);
          if (fj < nf) frag_product<false>(U, A.a, n, S, 8 * fi, 8 * fj, c[2 * fj], c[2 * fj + 1]);
        }
        __syncwarp();
        const int i = 8 * fi + g8;
#pragma unroll
        for (int fj = 0; fj < NF; ++fj) {
          const int j = 8 * fj + 2 * t4;
          if (fj < nf && i < n && j < n) {
            U[i * S + j] = csub(U[i * S + j], cscale(c[2 * fj], 0.5));
            U[i * S + j + 1] = csub(U[i * S + j + 1], cscale(c[2 * fj + 1], 0.5));
          }
        }
        __syncwarp();
      }
    } else {
      for (int r = warp; r < n; r += nwarps) {
        double2 x[kEigCols];
#pragma unroll
        for (int m = 0; m < kEigCols; ++m) {
          x[m] = make_double2(0.0, 0.0);
          const int j = lane + 32 * m;
          if (j < n)
            for (int i = 0; i < n; ++i) x[m] = cfma(U[r * S + i], A.get(i, j), x[m]);
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < kEigCols; ++m) {
          const int j = lane + 32 * m;
          if (j < n) U[r * S + j] = csub(U[r * S + j], cscale(x[m], 0.5));
        }
        __syncwarp();
      }
    }
    __syncthreads();
    //  (3) lambda_a = Re u_a^H Hs u_a with Hs = (H + H^H) / 2 from the table
    for (int e = tid; e < na; e += blockDim.x) {
      int r, c;
      A.ij(e, r, c);
      const double2 x = Hk[r * n + c], y = Hk[c * n + r];
      A.a[A.at(r, c)] = r == c ? make_double2(x.x, 0.0) : make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
    }
    __syncthreads();
    for (int e = tid; e < n * n; e += blockDim.x) Uk[e] = U[(e / n) * S + e % n];
    if (!PACKED) {
      // W = Hs U in place (a warp per 8 rows), then one thread per eigenvalue
      const int nf = (n + 7) / 8;
      for (int fi = warp; fi < nf; fi += nwarps) {
        double2 c[2 * NF];
#pragma unroll
        for (int fj = 0; fj < NF; ++fj) {
          c[2 * fj] = c[2 * fj + 1] = make_double2(0.0, 0.0);
          if (fj < nf) frag_product<false>(A.a, U, n, S, 8 * fi, 8 * fj, c[2 * fj], c[2 * fj + 1]);
        }
        __syncwarp();
        const int i = 8 * fi + g8;
#pragma unroll
        for (int fj = 0; fj < NF; ++fj) {
          const int j = 8 * fj + 2 * t4;
          if (fj < nf && i < n && j < n) {
            A.a[i * S + j] = c[2 * fj];
            A.a[i * S + j + 1] = c[2 * fj + 1];
          }
        }
        __syncwarp();
      }
      __syncthreads();
      for (int a = tid; a < n; a += blockDim.x) {
        double l = 0.0;
        for (int r = 0; r < n; ++r) {
          const double2 u = U[r * S + a], w = A.a[r * S + a];
          l = fma(u.x, w.x, fma(u.y, w.y, l));   // Re(conj(u) w)
        }
        lam[k * n + a] = l;
      }
    } else {
      // no room for W: a warp per eigenvalue, lanes over the rows r of sum_r conj(u_r) (Hs u)_r
      for (int a = warp; a < n; a += nwarps) {
        double l = 0.0;
        for (int r = lane; r < n; r += 32) {
          double2 w = make_double2(0.0, 0.0);
          for (int c = 0; c < n; ++c) w = cfma(A.get(r, c), U[c * S + a], w);
          const double2 u = U[r * S + a];
          l = fma(u.x, w.x, fma(u.y, w.y, l));
        }
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) lam[k * n + a] = l;
      }
    }
    __syncthreads();
  }
}

int optin_smem() {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  return optin;
}

size_t fin_smem(int n, bool packed) {
  return sizeof(double2) *
         ((size_t)n * odd_stride(n) + (packed ? HermA<true>::storage(n) : HermA<false>::storage(n)));
}

// the post-pass with the packed scratch: beyond the fragments of a row block, or the memory
bool fin_packed(int n, int optin) { return n > 8 * kEigFrags || fin_smem(n, false) > (size_t)optin; }

// warps per matrix: 32 rows each, times the parts of the columns (few where several matrices
// share an SM, as many as there are registers for where one fills it)
int hh_warps(int n) { return n <= 32 ? 2 : n <= 40 ? 4 : n <= 64 ? 6 : n <= 76 ? 9 : 15; }

size_t hh_smem(int n) {
  return sizeof(double2) * ((size_t)n * odd_stride(n) + 3 * (size_t)n + 4 + 32 * (size_t)hh_warps(n));
}

// rotations and sweeps kept per k: the iteration takes about 1.3 n^2 rotations in 2.3 n sweeps
int ql_cap(int n) { return 3 * n * n + 32; }
int ql_sweeps(int n) { return 8 * n + 16; }

}  // namespace

// U and a scratch matrix both whole in shared memory (dimensions up to 72 or so): there G from
// (U, lambda) costs 8 n^3 flops per point like the tridiagonal resolvents, without their sweeps;
// beyond, the packed post-pass runs one matrix per SM and the tridiagonalisation alone is
// cheaper per k
int eig_fast(int n) {
  if (n % 2 != 0 || n < 2 || n > 32 * kEigCols) return 0;
  return fin_smem(n, false) <= (size_t)optin_smem();
}

int eig_supported(int n) {
  if (n % 2 != 0 || n < 2 || n > 32 * kEigCols) return 0;
  const int optin = optin_smem();
  return fin_smem(n, fin_packed(n, optin)) <= (size_t)optin;
}

int hh_small_supported(int n) { return n >= 2 && n <= kHhMax && hh_smem(n) <= (size_t)optin_smem(); }

cudaError_t launch_hh_small(const double2* H, int64_t nk, int n, const int* rows, int ns, double* D, double* E,
                            double2* Q, int num_sms, cudaStream_t s) {
  if (nk <= 0) return cudaSuccess;
  if (!hh_small_supported(n) || ns <= 0 || ns > n) return cudaErrorInvalidValue;
  const size_t smem = hh_smem(n);
  const int threads = 32 * hh_warps(n);
  cudaError_t e = allow_smem(hh_small_kernel, smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hh_small_kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  const int64_t grid = std::min<int64_t>(nk, (int64_t)num_sms * per_sm);
  hh_small_kernel<<<(unsigned)grid, threads, smem, s>>>(H, nk, n, rows, ns, D, E, Q);
  return cudaGetLastError();
}

// at most 1 GiB of rotations
int64_t eig_chunk(int n, int64_t nk) {
  return std::max<int64_t>(1, std::min<int64_t>(nk, ((int64_t)1 << 30) / ((int64_t)ql_cap(n) * 16)));
}

size_t eig_ws_bytes(int n, int64_t nk, int64_t chunk) {
  return (size_t)chunk * ((size_t)ql_cap(n) * sizeof(double2) + (size_t)ql_sweeps(n) * sizeof(int) + sizeof(int)) +
         (size_t)nk * n * 2 * sizeof(double) + 256;
}

int64_t eig_launches(int64_t nk, int64_t chunk) { return nk > 0 ? 1 + 3 * ((nk + chunk - 1) / chunk) : 0; }

cudaError_t launch_eig(const double2* H, int64_t nk, int n, double2* U, double* lam, void* ws, int64_t chunk,
                       int* status, int num_sms, cudaStream_t s) {
  if (nk <= 0) return cudaSuccess;
  if (!eig_supported(n) || chunk <= 0) return cudaErrorInvalidValue;
  const int cap = ql_cap(n), scap = ql_sweeps(n);
  double2* rot = static_cast<double2*>(ws);
  double* D = reinterpret_cast<double*>(rot + chunk * cap);
  double* E = D + nk * n;
  int* sweep = reinterpret_cast<int*>(E + nk * n);
  int* nsweep = sweep + chunk * scap;
  cudaError_t e = launch_hh_small(H, nk, n, nullptr, n, D, E, U, num_sms, s);
  if (e != cudaSuccess) return e;
  const size_t qsmem = sizeof(double) * 64 * (size_t)n;
  e = allow_smem(ql_kernel, qsmem);
  if (e != cudaSuccess) return e;
  const bool packed = fin_packed(n, optin_smem());
  const size_t fsmem = fin_smem(n, packed);
  auto fin = packed            ? eig_finish_kernel<true, 1>
             : n <= 24         ? eig_finish_kernel<false, 3>
             : n <= 40         ? eig_finish_kernel<false, 5>
             : n <= 56         ? eig_finish_kernel<false, 7>
                               : eig_finish_kernel<false, kEigFrags>;
  e = allow_smem(fin, fsmem);
  if (e != cudaSuccess) return e;
  const size_t asmem = sizeof(double2) * ((size_t)n * odd_stride(n) + kRotRoom);
  const int athreads = (2 * n + 31) / 32 * 32;
  e = allow_smem(eig_apply_kernel, asmem);
  if (e != cudaSuccess) return e;
  int per_sm = 0, aper_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fin, kFinThreads, fsmem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&aper_sm, eig_apply_kernel, athreads, asmem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0 || aper_sm <= 0) return cudaErrorInvalidValue;
  for (int64_t k0 = 0; k0 < nk; k0 += chunk) {
    const int64_t m = std::min(chunk, nk - k0);
    int lanes = 32;
    while (lanes > 2 && (m + lanes - 1) / lanes < 4 * num_sms) lanes /= 2;
    ql_kernel<<<(unsigned)((m + lanes - 1) / lanes), 32, qsmem, s>>>(D, E, k0, m, n, lam, rot, cap, sweep, scap,
                                                                    nsweep, lanes, status);
    double2* Uk = U + k0 * (int64_t)n * n;
    eig_apply_kernel<<<(unsigned)std::min<int64_t>(m, (int64_t)num_sms * aper_sm), athreads, asmem, s>>>(
        m, n, rot, cap, sweep, scap, nsweep, Uk);
    fin<<<(unsigned)std::min<int64_t>(m, (int64_t)num_sms * per_sm), kFinThreads, fsmem, s>>>(
        H + k0 * (int64_t)n * n, m, n, Uk, lam + k0 * n);
  }
  return cudaGetLastError();
}

}  // namespace tg
