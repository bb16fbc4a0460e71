// Linear-SOC susceptibility (eintshechilinearsoc, source/eintshechi.F90:182-414).
//
// With G0 = (z - H0)^-1 for the Hamiltonian without the local spin-orbit blocks and
// V the SOC blocks (hamiltklinearsoc, mod_hamiltonian.F90:304-396), the reference's
// greenlinearsoc (mod_greenfunction.F90:141-202) forms G0 V G0 per point and
//   chi_lsoc = chi(G0 V G0 (k+q, E+e), G0(k, E)) + chi(G0(k+q, E+e), G0 V G0 (k, E)),
// chi(., .) being the same bilinear integrand as chi0.  Here the per-point pieces are
// two kernels around the existing inversion and contraction kernels:
//   gvg_kernel      X_p = G_p V G_p from the column-major inversion output (one CTA
//                   per point, G, V and V G staged in shared memory, FP64);
//   operand_kernel  a column-major G_p (or X_p) into the pair-block operand layouts of
//                   the contraction (w G, G^T, w (G - G^+), conj G) with the point weights.
#include "tg_internal.cuh"

#include <algorithm>

namespace tg {

namespace {

// X[p] = G[p] V G[p], all column-major n x n; Gs, T row-major in shared memory
__global__ void __launch_bounds__(256) gvg_kernel(const double2* __restrict__ G, const double2* __restrict__ V, int n,
                                                  int64_t np, double2* __restrict__ X) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int nn = n * n;
  double2* Vs = reinterpret_cast<double2*>(smem);
  double2* Gs = Vs + nn;
  double2* T = Gs + nn;
  for (int e = threadIdx.x; e < nn; e += blockDim.x) {
    const int c = e / n, r = e % n;
    Vs[r * n + c] = V[e];
  }
  for (int64_t p = blockIdx.x; p < np; p += gridDim.x) {
    __syncthreads();
    const double2* g = G + p * (int64_t)nn;
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
      const int c = e / n, r = e % n;
      Gs[r * n + c] = g[e];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
      const int r = e / n, c = e % n;
      double2 s = make_double2(0.0, 0.0);
      for (int m = 0; m < n; ++m) s = cfma(Vs[r * n + m], Gs[m * n + c], s);
      T[e] = s;
    }
    __syncthreads();
    double2* x = X + p * (int64_t)nn;
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
      const int c = e / n, r = e % n;   // column-major write, consecutive threads down a column
      double2 s = make_double2(0.0, 0.0);
      for (int m = 0; m < n; ++m) s = cfma(Gs[r * n + m], T[m * n + c], s);
      x[e] = s;
    }
  }
}

// out[p][o] = transform of G_p at the pair-block slot o (outmap[o] = r * n + c), p in the pass
__global__ void operand_kernel(const double2* __restrict__ G, int n, int64_t np, int64_t p0, PointSet pts, int mode,
                               const int* __restrict__ outmap, double2* __restrict__ out) {
  const int64_t nn = (int64_t)n * n;
  const int64_t total = np * nn;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pl = idx / nn;
    const int o = (int)(idx % nn);
    const int rc = outmap[o];
    const int r = rc / n, c = rc % n;
    const double2* g = G + pl * nn;
    const int64_t p = p0 + pl;
    double w;
    if (pts.kind == 0) {
      w = pts.w[p];
    } else {
      w = pts.p2[p / pts.nk] * pts.w[p % pts.nk];
    }
    const double2 grc = g[(int64_t)c * n + r];
    double2 v;
    if (mode == MODE_A_IMAG) {
      v = cscale(grc, w);
    } else if (mode == MODE_B_IMAG) {
      v = g[(int64_t)r * n + c];   // G^T
    } else if (mode == MODE_A_REAL) {
      const double2 gcr = g[(int64_t)r * n + c];
      v = cscale(make_double2(grc.x - gcr.x, grc.y + gcr.y), w);
    } else {
      v = cconj(grc);
    }
    out[idx] = v;
  }
}

// out[p][o] = transform of the column-major G_p (n x n) at slot o of an operand layout with
// ld slots per point (outmap[o] = r * n + c, a subset of G's entries in pair-block order);
// the weights follow the point traversal of the Green-function launch g (tabulated k-major
// or the flattened list), as the fused output stages do
// A thread keeps its slot for all points of its block's share, so that the slot's row and column
// and the points' weights (a 64-bit division each) are worked out once; neighbouring slots read
// whole sectors of G.  Bound by HBM (32 bytes per slot and point, 48 with both halves of
// G - G^+).  The 160 d rows of 16 layers: 5.7 ms a call with the divisions per entry, 4.8 ms.
constexpr int kGatherPoints = 32;

template <int MODE>
__global__ void __launch_bounds__(256) gather_kernel(GreenArgs g, const double2* __restrict__ G,
                                                     const int* __restrict__ outmap, int64_t ld,
                                                     double2* __restrict__ out, int16_t* __restrict__ eout) {
  __shared__ double ws[kGatherPoints];
  const int n = g.n;
  const int64_t nn = (int64_t)n * n;
  const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int rc = o < ld ? outmap[o] : 0;
  const int r = rc / n, c = rc - r * n;
  const int64_t at = (int64_t)c * n + r, att = (int64_t)r * n + c;   // G(r, c) and G(c, r)
  for (int64_t p0 = blockIdx.y * (int64_t)kGatherPoints; p0 < g.np; p0 += gridDim.y * (int64_t)kGatherPoints) {
    const int here = (int)min((int64_t)kGatherPoints, g.np - p0);
    __syncthreads();
    if (threadIdx.x < here) ws[threadIdx.x] = point_weight(g, p0 + threadIdx.x);
    __syncthreads();
    if (o >= ld) continue;
#pragma unroll 4
    for (int i = 0; i < here; ++i) {
      const double2* gp = G + (p0 + i) * nn;
      double2 v;
      if (MODE == MODE_A_IMAG) {
        v = cscale(gp[at], ws[i]);
      } else if (MODE == MODE_B_IMAG) {
        v = gp[att];   // G^T
      } else if (MODE == MODE_A_REAL) {
        const double2 x = gp[at], xt = gp[att];
        v = cscale(make_double2(x.x - xt.x, x.y + xt.y), ws[i]);
      } else {
        v = cconj(gp[at]);
      }
      out[(p0 + i) * ld + o] = v;
      if (eout) eout[(p0 + i) * ld + o] = exponent_code16(v);
    }
  }
}

}  // namespace

cudaError_t launch_gather(const GreenArgs& g, const double2* G, int mode, const int* outmap, int64_t ld, double2* out,
                          int16_t* eout, int num_sms, cudaStream_t s) {
  if (g.np <= 0) return cudaSuccess;
  if (mode != MODE_A_IMAG && mode != MODE_B_IMAG && mode != MODE_A_REAL && mode != MODE_B_REAL)
    return cudaErrorInvalidValue;
  const int64_t bx = (ld + 255) / 256, chunks = (g.np + kGatherPoints - 1) / kGatherPoints;
  if (bx > 0x7fffffff) return cudaErrorInvalidValue;
  // a few waves of eight blocks per SM
  const int64_t by = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(chunks, 65535), num_sms * 32 / bx));
  const dim3 grid((unsigned)bx, (unsigned)by);
  switch (mode) {
    case MODE_A_IMAG: gather_kernel<MODE_A_IMAG><<<grid, 256, 0, s>>>(g, G, outmap, ld, out, eout); break;
    case MODE_B_IMAG: gather_kernel<MODE_B_IMAG><<<grid, 256, 0, s>>>(g, G, outmap, ld, out, eout); break;
    case MODE_A_REAL: gather_kernel<MODE_A_REAL><<<grid, 256, 0, s>>>(g, G, outmap, ld, out, eout); break;
    default: gather_kernel<MODE_B_REAL><<<grid, 256, 0, s>>>(g, G, outmap, ld, out, eout); break;
  }
  return cudaGetLastError();
}

size_t gvg_smem_bytes(int n) { return sizeof(double2) * 3 * (size_t)n * n; }

cudaError_t launch_gvg(const double2* G, const double2* V, int n, int64_t np, double2* X, int num_sms,
                       cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  const size_t smem = gvg_smem_bytes(n);
  cudaError_t e = allow_smem(gvg_kernel, smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gvg_kernel, 256, smem);
  if (e != cudaSuccess) return e;
  if (per_sm <= 0) return cudaErrorInvalidValue;
  const int64_t grid = std::min<int64_t>(np, (int64_t)num_sms * per_sm);
  gvg_kernel<<<(unsigned)grid, 256, smem, s>>>(G, V, n, np, X);
  return cudaGetLastError();
}

cudaError_t launch_operand(const double2* G, int n, int64_t np, int64_t p0, const PointSet& pts, int mode,
                           const int* outmap, double2* out, int num_sms, cudaStream_t s) {
  if (np <= 0) return cudaSuccess;
  const int64_t total = np * (int64_t)n * n;
  const int64_t grid = std::min<int64_t>((total + 255) / 256, (int64_t)num_sms * 16);
  operand_kernel<<<(unsigned)grid, 256, 0, s>>>(G, n, np, p0, pts, mode, outmap, out);
  return cudaGetLastError();
}

}  // namespace tg
