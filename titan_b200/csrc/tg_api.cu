// C ABI of libtitan_gpu (declared in include/titan_gpu.h).
//
// The context owns every device buffer; host arrays stay caller-owned.  The
// orchestration per chi0(q, omega) call mirrors eintshechi.F90:2-178:
//   imaginary axis, in passes of P points:  G2 = G(k, Ef + i(y + eta'))  -> B operand
//                                           G1 = G(k+q, Ef + e + i(y + eta)) -> A operand
//                                           C += A^T B per site pair (contraction)
//   real axis (|e| >= 1e-15), same with z on [Ef - e, Ef]             -> D
//   epilogue: chiorb_hf = (C + conj(C_swapped) - i D) / 2 pi
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <string>
#include <vector>

#include "../../include/titan_gpu.h"
#include "tg_internal.cuh"
#include "tg_split.cuh"
#include "tg_stage.cuh"

using namespace tg;

namespace tg {
cudaError_t dyson_device(int n, const double2* chi_hf, const double2* U, double2* work, double2* chi, int* piv,
                         int* status, cudaStream_t s);
cudaError_t launch_transpose(int n, const double2* in, double2* out, cudaStream_t s);
}

namespace {

constexpr double kPi = 3.141592653589793238462643383279502884;
constexpr int kTriQSlots = 8;   // tridiagonalisations of H(k + q) kept at once by tg_chi0_qbatch

template <class T>
struct DevArray {
  T* p = nullptr;
  size_t n = 0;
  DevArray() = default;
  DevArray(const DevArray&) = delete;
  DevArray& operator=(const DevArray&) = delete;
  ~DevArray() { free_(); }
  void free_() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  cudaError_t ensure(size_t count) {
    if (count <= n && p) return cudaSuccess;
    free_();
    cudaError_t e = cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
  cudaError_t upload(const T* h, size_t count, cudaStream_t s) {
    cudaError_t e = ensure(count);
    if (e != cudaSuccess) return e;
    if (count == 0) return cudaSuccess;
    return cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s);
  }
};

// Layout of the chi0 contraction over a subset of each site's orbitals (tg_set_chi_orbitals):
// the pair-block operand layout of those orbitals (slot o -> entry outmap[o] = r * dimH + c
// of the full G), its contraction tiles and split groups, and the epilogue's row decode.
struct ChiLayout {
  int dimens = 0;
  int nsel = 0;                       // rows of G that enter chi (2 sum nc)
  std::vector<int> nc;                // chi orbitals per site
  std::vector<int> pair_M, pair_aoff;
  std::vector<int64_t> pair_coff;
  std::vector<PairTile> tiles;
  SplitLayout split;
  DevArray<int> d_rows;               // the nsel rows of G that enter chi, site by site
  DevArray<int> d_outmap, d_decode, d_norb, d_pair_M, d_pair_aoff;
  DevArray<int64_t> d_pair_coff;
  DevArray<PairTile> d_tiles;
  DevArray<SplitGroup> d_sgA, d_sgB;
  DevArray<SplitTile> d_stiles;
};

// what the chi0 helpers read: the full layout of tg_set_system or a ChiLayout; gather: the
// Green-function kernels write G column-major and launch_gather forms the operands
struct ChiView {
  int dimens = 0;
  int64_t ld = 0;                     // operand slots per point
  bool gather = false;
  const int *outmap = nullptr, *decode = nullptr, *norb = nullptr, *pair_M = nullptr, *pair_aoff = nullptr;
  const int64_t* pair_coff = nullptr;
  const PairTile* tiles = nullptr;
  int ntiles = 0;
  const SplitLayout* split = nullptr;
  const SplitGroup *sgA = nullptr, *sgB = nullptr;
  const SplitTile* stiles = nullptr;
  const int* rows = nullptr;          // the rows of G that enter chi
  int nrows = 0;
};

}  // namespace

struct tg_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 148;
  std::string err;
  bool sys_set = false, h0_set = false, imag_set = false, real_set = false;
  // system
  int n_atoms = 0, nmax = 0, dimH = 0, dimens = 0, n_neigh = 0;
  std::vector<int> norb, ia;            // ia[i] = first row of site i
  std::vector<int> pair_M, pair_aoff;   // per pair (i*nat + j)
  std::vector<int64_t> pair_coff;
  std::vector<PairTile> tiles;
  DevArray<double> d_R;
  DevArray<int> d_pair_start, d_pair_neigh, d_row_atom, d_row_orb, d_row_spin, d_outmap, d_decode, d_norb,
      d_pair_M, d_pair_aoff, d_exp_rows, d_gg_desc;
  DevArray<int64_t> d_pair_coff;
  DevArray<double2> d_pair_t, d_h0;
  DevArray<PairTile> d_tiles;
  // meshes
  int64_t n_imag = 0, n_realk = 0;
  DevArray<double> d_y, d_kp, d_w, d_rkp, d_rw, d_x2, d_p2;
  // uniform imaginary-axis mesh: n_e energies x the same nk_u k points (energy-major)
  bool imag_uniform = false;
  int64_t n_e_u = 0, nk_u = 0;
  DevArray<double> d_ylist, d_klist_u, d_qvec;
  DevArray<double2> d_htab[4], d_hphase;   // H(k), H(k+q) for the imaginary and real k lists
  // workspace
  DevArray<double2> d_A, d_B, d_C, d_D, d_chi, d_acc, d_acc_red;
  DevArray<double2> d_zlist, d_gout;
  DevArray<double> d_klist;
  DevArray<int> d_status;
  // split-precision contraction
  SplitLayout split;
  DevArray<SplitGroup> d_sgA, d_sgB;
  DevArray<SplitTile> d_stiles;
  DevArray<int8_t> d_digA, d_digB;
  DevArray<unsigned long long> d_m64A, d_m64B;
  DevArray<int16_t> d_e16A, d_e16B;   // exponent sidecars of the FP64 operands (spectral G)
  DevArray<int> d_EA, d_EB, d_chunks, d_split_err;
  std::vector<double> h_y;   // imaginary-axis energies per point (chunk boundaries)
  std::vector<double> h_klist_u, h_rkp;   // host copies of the uniform k list and the real-axis BZ
  DevArray<double2> d_dy;
  DevArray<int> d_piv;
  cudaEvent_t ev[8] = {};
  double last_ms[4] = {0, 0, 0, 0};
  // optional per-launch timing: (kind, start, stop) event pairs of the last call
  bool profile = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> ev_used;
  double kind_ms[4] = {0, 0, 0, 0};   // 0 inversion, 1 contraction, 2 epilogue, 3 split quantisation
  int kind_n[4] = {0, 0, 0, 0};
  int64_t launches = 0;   // kernels launched by the last chi0 call
  int64_t pass_points = 0;     // points per pass (bounded workspace)
  // spectral Green functions: eigendecomposition of each H(k) table, inverse output map
  int green_method = 0;   // TG_GREEN_AUTO / TG_GREEN_GAUSS_JORDAN / TG_GREEN_SPECTRAL
  DevArray<double2> d_eigU[4];
  DevArray<double> d_eigL[4];
  DevArray<unsigned char> d_eigws;   // rotations and tridiagonal matrices of launch_eig
  DevArray<double2> d_hchunk;   // bounded H(k) scratch of eigendecompositions built chunk by chunk
  DevArray<int> d_outinv, d_eig_status;
  DevArray<double> d_ldos_e, d_ldos;
  // linear SOC: V, G V G of both Green functions, four operands, chi_lsoc partials
  DevArray<double2> d_vsoc, d_lsb[6], d_Cl, d_Dl;
  // disturbance response (eintshe)
  DevArray<int> d_she_tab, d_ia, d_she_ztiles, d_she_rowoff;
  DevArray<double2> d_she_part, d_she_sum, d_she_pref, d_she_out;
  // autotuned K-range split counts per contraction layout (precision, tiles, pass K-steps)
  bool autotune = true;
  std::vector<std::pair<std::vector<int64_t>, int>> tuned;
  int last_nsplit[2] = {0, 0};   // FP64, split
  DevArray<double2> d_tune;
  // split-format error bound of the last chi0 call: per result [imaginary, real] x site pair
  // sums, and the relative normwise bounds (0 for FP64 results)
  DevArray<double> d_bound;
  std::vector<double> err_bound;
  // split precision: points per chunk (one scale per operand element and chunk); 1024
  // keeps every 4 x 4 spin block holding >= 1e-8 of the largest within 1e-9 on the sq2
  // workload (6e-10 measured)
  int split_chunk = 1024;
  // chi0 over a subset of orbitals (tg_set_chi_orbitals)
  bool chi_sel_on = false;
  ChiLayout chi_sel;
  DevArray<double2> d_graw;   // column-major G of a pass (gathered chi0 operands)
  DevArray<int> d_allrows;    // 0 .. dimH - 1
  // Householder tridiagonalisations per k list (same slots as the H tables)
  // (slots 4 .. 4 + kTriQSlots - 1: one per wave vector of a q-batched real axis)
  DevArray<double> d_triD[4 + kTriQSlots], d_triE[4 + kTriQSlots];
  DevArray<double2> d_triQ[4 + kTriQSlots];
  DevArray<double2> d_triws;   // factors of z - T of a pass's points
  DevArray<unsigned char> d_clws;   // workspace of the thread-block-cluster Gauss-Jordan kernel
  HostStage stage;   // large transfers between pageable host arrays and the device
  // tg_expectation_noalloc: device address of the library's fixed scratch array on this
  // context's device (looked up by the context's first no-alloc call)
  double2* noalloc_ptr = nullptr;
};

namespace {

// launch-kind timing (kind 0 = green/inversion, 1 = contraction, 2 = epilogue)
cudaEvent_t pool_event(tg_ctx* c) {
  if (!c->ev_pool.empty()) {
    cudaEvent_t e = c->ev_pool.back();
    c->ev_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

struct KindTimer {
  tg_ctx* c;
  int kind;
  cudaEvent_t a = nullptr, b = nullptr;
  KindTimer(tg_ctx* ctx, int k) : c(ctx), kind(k) {
    if (!c->profile) return;
    a = pool_event(c);
    b = pool_event(c);
    cudaEventRecord(a, c->stream);
  }
  ~KindTimer() {
    if (kind == 0 || kind == 2) c->launches += 1;   // contraction / quantize launches are counted where issued
    if (!c->profile) return;
    cudaEventRecord(b, c->stream);
    c->ev_used.push_back({kind, {a, b}});
  }
};

void profile_begin(tg_ctx* c) {
  c->launches = 0;
  for (int k = 0; k < 4; ++k) {
    c->kind_ms[k] = 0;
    c->kind_n[k] = 0;
  }
}

void profile_end(tg_ctx* c) {
  if (!c->profile) return;
  cudaStreamSynchronize(c->stream);
  for (auto& u : c->ev_used) {
    float ms = 0;
    cudaEventElapsedTime(&ms, u.second.first, u.second.second);
    c->kind_ms[u.first] += ms;
    c->kind_n[u.first] += 1;
    c->ev_pool.push_back(u.second.first);
    c->ev_pool.push_back(u.second.second);
  }
  c->ev_used.clear();
}

int set_err(tg_ctx* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  return code;
}

int cuda_err(tg_ctx* c, cudaError_t e, const char* where) {
  if (e == cudaSuccess) return TG_OK;
  cudaGetLastError();   // reported here; else the next call's first launch would report it again
  std::string m = std::string(where) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return set_err(c, TG_ERR_NOMEM, m);
  return set_err(c, TG_ERR_CUDA, m);
}

#define TG_CHECK(c, call, where)                      \
  do {                                                \
    cudaError_t _e = (call);                          \
    if (_e != cudaSuccess) return cuda_err(c, _e, where); \
  } while (0)

// a transfer between a host array and the device, complete on return
cudaError_t copy_host(tg_ctx* c, void* dst, const void* src, size_t bytes, bool to_device) {
  return c->stage.copy(c->device, c->stream, dst, src, bytes, to_device);
}

GreenArgs base_args(tg_ctx* c) {
  GreenArgs a;
  a.n = c->dimH;
  a.n_neigh = c->n_neigh;
  a.R = c->d_R.p;
  a.pair_start = c->d_pair_start.p;
  a.pair_neigh = c->d_pair_neigh.p;
  a.pair_t = c->d_pair_t.p;
  a.nmax = c->nmax;
  a.n_atoms = c->n_atoms;
  a.row_atom = c->d_row_atom.p;
  a.row_orb = c->d_row_orb.p;
  a.row_spin = c->d_row_spin.p;
  a.h0 = c->d_h0.p;
  a.outmap = c->d_outmap.p;
  a.status = c->d_status.p;
  a.ws = c->d_clws.p;
  a.ws_bytes = c->d_clws.n;
  return a;
}

// entry points whose Green functions are reduced inside the single-SM kernels' output
// stages: the dimension must have one of those kernels
int require_native(tg_ctx* c, const char* who) {
  if (green_supported(c->dimH)) return TG_OK;
  char b[256];
  snprintf(b, sizeof b,
           "%s: dimH = %d has no single-SM Gauss-Jordan kernel (dimensions 4, 8, 16, 18, 20, 36, 40, 54, 72, 90); "
           "larger systems are served by tg_chi0, tg_chi0_batch, tg_green_batch, tg_hamiltk_batch and tg_dyson",
           who, c->dimH);
  return set_err(c, TG_ERR_ARG, b);
}

int check_ready(tg_ctx* c, bool need_imag, bool need_real) {
  if (!c) return TG_ERR_ARG;
  if (!c->sys_set) return set_err(c, TG_ERR_STATE, "tg_set_system has not been called");
  if (!c->h0_set) return set_err(c, TG_ERR_STATE, "tg_set_h0 has not been called");
  if (need_imag && !c->imag_set) return set_err(c, TG_ERR_STATE, "tg_set_imag_mesh has not been called");
  if (need_real && !c->real_set) return set_err(c, TG_ERR_STATE, "tg_set_real_mesh has not been called");
  return TG_OK;
}

int reset_status(tg_ctx* c) {
  const int big = 0x7fffffff;
  TG_CHECK(c, cudaMemcpyAsync(c->d_status.p, &big, sizeof(int), cudaMemcpyHostToDevice, c->stream), "status");
  return TG_OK;
}

int read_status(tg_ctx* c) {
  int st = 0;
  TG_CHECK(c, cudaMemcpyAsync(&st, c->d_status.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream), "status");
  TG_CHECK(c, cudaStreamSynchronize(c->stream), "sync");
  if (st != 0x7fffffff) {
    char buf[128];
    snprintf(buf, sizeof buf, "singular (z - H(k)) at point %d", st);
    c->err = buf;
    return st;
  }
  return TG_OK;
}

int64_t pass_size(tg_ctx* c, int64_t np, int64_t operand_bytes = (int64_t)3 << 30) {
  // two operand buffers of P * dimH^2 complex each, operand_bytes apiece
  const int64_t per = (int64_t)c->dimH * c->dimH * sizeof(double2);
  int64_t P = operand_bytes;
  P /= per;
  P = std::max<int64_t>(P, 1024);
  P = (P / 64) * 64;
  return std::min<int64_t>(P, std::max<int64_t>(np, 1));
}

int nsplit_for(tg_ctx* c) {
  const int nt = (int)c->tiles.size();
  int s = std::max(1, c->num_sms / std::max(nt, 1));
  return std::min(s, 64);
}

// H(k + q) table for a k list into d_htab[slot]
int build_htab(tg_ctx* c, int slot, const double* d_k, int64_t nk, const double* q) {
  const size_t nn = (size_t)c->dimH * c->dimH;
  TG_CHECK(c, c->d_htab[slot].ensure((size_t)nk * nn), "alloc H table");
  TG_CHECK(c, c->d_hphase.ensure((size_t)nk * std::max(c->n_neigh, 1)), "alloc phases");
  TG_CHECK(c, c->d_qvec.upload(q, 3, c->stream), "upload q");
  GreenArgs a = base_args(c);
  TG_CHECK(c, launch_hk_table(a, d_k, nk, c->d_qvec.p, c->d_hphase.p, c->d_htab[slot].p, c->stream), "H table");
  c->launches += 2;
  return TG_OK;
}

// chi0 and the LDOS use spectral Green functions unless Gauss-Jordan is forced; the
// disturbance integral and the occupations only when TG_GREEN_SPECTRAL asks for them (see
// tg_set_green_method)
bool spectral_on(tg_ctx* c) { return c->green_method != TG_GREEN_GAUSS_JORDAN && eig_supported(c->dimH); }
bool spectral_forced(tg_ctx* c) { return c->green_method == TG_GREEN_SPECTRAL && eig_supported(c->dimH); }
// chi0 on meshes whose energies share a k list: spectral G where the eigensolver's post-pass
// holds two matrices in shared memory (or when asked for), else under TG_GREEN_AUTO G from a
// Householder tridiagonalisation per k (cheaper per k than the whole eigendecomposition, and as
// accurate as Gauss-Jordan near the real axis)
bool chi_spectral(tg_ctx* c) {
  return spectral_on(c) && (eig_fast(c->dimH) || c->green_method == TG_GREEN_SPECTRAL);
}
bool chi_tridiag(tg_ctx* c) {
  return !chi_spectral(c) && c->green_method == TG_GREEN_AUTO && tri_supported(c->dimH);
}

// workspace of launch_eig for tables of nk matrices, `chunk` of them at a time: fewer where the
// device memory does not hold the rotations of all that 1 GiB would
int ensure_eig_ws(tg_ctx* c, int64_t nk, int64_t& chunk) {
  for (chunk = eig_chunk(c->dimH, nk);; chunk = (chunk + 1) / 2) {
    const cudaError_t e = c->d_eigws.ensure(eig_ws_bytes(c->dimH, nk, chunk));
    if (e != cudaErrorMemoryAllocation || chunk <= 64) return cuda_err(c, e, "alloc rotations");
    cudaGetLastError();
  }
}

// eigendecomposition of every row of H table `slot` (spectral Green functions)
int build_eig(tg_ctx* c, int slot, int64_t nk) {
  const size_t nn = (size_t)c->dimH * c->dimH;
  TG_CHECK(c, c->d_eigU[slot].ensure((size_t)nk * nn), "alloc eigenvectors");
  TG_CHECK(c, c->d_eigL[slot].ensure((size_t)nk * c->dimH), "alloc eigenvalues");
  int64_t chunk = 0;
  int rc = ensure_eig_ws(c, nk, chunk);
  if (rc) return rc;
  KindTimer kt(c, 0);   // (counts one launch)
  c->launches += eig_launches(nk, chunk) - 1;
  TG_CHECK(c, launch_eig(c->d_htab[slot].p, nk, c->dimH, c->d_eigU[slot].p, c->d_eigL[slot].p, c->d_eigws.p, chunk,
                         c->d_eig_status.p, c->num_sms, c->stream),
           "eigendecomposition");
  return TG_OK;
}

// U and lambda of H(k + q) for a k list whose H table is not kept (too long to be resident):
// the table is built and diagonalised in chunks of at most 2 GiB in a scratch buffer, and only
// the eigendecompositions stay, in eigenvector slot `slot`
int build_eig_chunked(tg_ctx* c, int slot, const double* d_k, int64_t nk, const double* q) {
  const int64_t n = c->dimH, nn = n * n;
  const int64_t kc = std::max<int64_t>(1, std::min<int64_t>(nk, ((int64_t)2 << 30) / (nn * 16)));
  TG_CHECK(c, c->d_eigU[slot].ensure((size_t)nk * nn), "alloc eigenvectors");
  TG_CHECK(c, c->d_eigL[slot].ensure((size_t)nk * n), "alloc eigenvalues");
  TG_CHECK(c, c->d_hchunk.ensure((size_t)kc * nn), "alloc H chunk");
  TG_CHECK(c, c->d_hphase.ensure((size_t)kc * std::max(c->n_neigh, 1)), "alloc phases");
  int64_t chunk = 0;
  int rc = ensure_eig_ws(c, kc, chunk);
  if (rc) return rc;
  TG_CHECK(c, c->d_qvec.upload(q, 3, c->stream), "upload q");
  const GreenArgs a = base_args(c);
  KindTimer kt(c, 0);
  for (int64_t k0 = 0; k0 < nk; k0 += kc) {
    const int64_t m = std::min(kc, nk - k0);
    TG_CHECK(c, launch_hk_table(a, d_k + 3 * k0, m, c->d_qvec.p, c->d_hphase.p, c->d_hchunk.p, c->stream),
             "H table");
    TG_CHECK(c, launch_eig(c->d_hchunk.p, m, (int)n, c->d_eigU[slot].p + k0 * nn, c->d_eigL[slot].p + k0 * n,
                           c->d_eigws.p, std::min(chunk, m), c->d_eig_status.p, c->num_sms, c->stream),
             "eigendecomposition");
    c->launches += 2 + eig_launches(m, chunk);
  }
  c->launches -= 1;   // (the timer counts one)
  return TG_OK;
}

// whether eigendecompositions of nk points in the eigenvector slots s0 and s1 (-1: none)
// leave room: what they add to the current allocations within half the free device memory
bool eig_room(tg_ctx* c, int64_t nk, int s0, int s1) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return false;
  const size_t nn = (size_t)c->dimH * c->dimH;
  double need = 0.0;
  for (int sl : {s0, s1}) {
    if (sl < 0) continue;
    const size_t want = (size_t)nk * nn;
    if (c->d_eigU[sl].n < want) need += (double)(want - c->d_eigU[sl].n) * sizeof(double2);
    need += (double)nk * c->dimH * sizeof(double);
  }
  const size_t kc = std::min<size_t>((size_t)nk, std::max<size_t>(1, ((size_t)2 << 30) / (nn * 16)));
  if (c->d_hchunk.n < kc * nn) need += (double)(kc * nn - c->d_hchunk.n) * sizeof(double2);
  const size_t ws = eig_ws_bytes(c->dimH, kc, eig_chunk(c->dimH, kc));
  if (c->d_eigws.n < ws) need += (double)(ws - c->d_eigws.n);
  return need <= 0.5 * (double)fr;
}

// Householder tridiagonalisation of H(k + q) for a k list into slot `slot`: T and the rows
// v.rows of Q, built chunk by chunk in the bounded H scratch (only T and Q_S are kept)
int build_tri_chunked(tg_ctx* c, int slot, const double* d_k, int64_t nk, const double* q, const ChiView& v) {
  const int64_t n = c->dimH, nn = n * n, ns = v.nrows;
  const int64_t kc = std::max<int64_t>(1, std::min<int64_t>(nk, ((int64_t)2 << 30) / (nn * 16)));
  TG_CHECK(c, c->d_triD[slot].ensure((size_t)nk * n), "alloc T");
  TG_CHECK(c, c->d_triE[slot].ensure((size_t)nk * n), "alloc T");
  TG_CHECK(c, c->d_triQ[slot].ensure((size_t)nk * ns * n), "alloc Q rows");
  TG_CHECK(c, c->d_hchunk.ensure((size_t)kc * nn), "alloc H chunk");
  TG_CHECK(c, c->d_hphase.ensure((size_t)kc * std::max(c->n_neigh, 1)), "alloc phases");
  TG_CHECK(c, c->d_qvec.upload(q, 3, c->stream), "upload q");
  const GreenArgs a = base_args(c);
  KindTimer kt(c, 0);
  for (int64_t k0 = 0; k0 < nk; k0 += kc) {
    const int64_t m = std::min(kc, nk - k0);
    TG_CHECK(c, launch_hk_table(a, d_k + 3 * k0, m, c->d_qvec.p, c->d_hphase.p, c->d_hchunk.p, c->stream),
             "H table");
    TG_CHECK(c, launch_tridiag(c->d_hchunk.p, m, (int)n, v.rows, (int)ns, c->d_triD[slot].p + k0 * n,
                               c->d_triE[slot].p + k0 * n, c->d_triQ[slot].p + k0 * ns * n, c->num_sms, c->stream),
             "tridiagonalisation");
    c->launches += 3;
  }
  c->launches -= 1;   // (the timer counts one)
  return TG_OK;
}

// whether tridiagonalisations of nk points in slots s0 and s1 (-1: none) fit: what they add to
// the current allocations (and the H chunk) within half the free device memory
bool tri_room_slots(tg_ctx* c, int64_t nk, int64_t ns, const std::vector<int>& slots) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) return false;
  const size_t n = c->dimH, nn = n * n;
  double need = 0.0;
  for (int sl : slots) {
    if (sl < 0) continue;
    const size_t want = (size_t)nk * ns * n;
    if (c->d_triQ[sl].n < want) need += (double)(want - c->d_triQ[sl].n) * sizeof(double2);
    need += 2.0 * nk * n * sizeof(double);
  }
  const size_t kc = std::min<size_t>((size_t)nk, std::max<size_t>(1, ((size_t)2 << 30) / (nn * 16)));
  if (c->d_hchunk.n < kc * nn) need += (double)(kc * nn - c->d_hchunk.n) * sizeof(double2);
  return need <= 0.5 * (double)fr;
}

bool tri_room(tg_ctx* c, int64_t nk, int64_t ns, int s0, int s1) { return tri_room_slots(c, nk, ns, {s0, s1}); }

int reset_eig_status(tg_ctx* c) {
  const int big = 0x7fffffff;
  TG_CHECK(c, c->d_eig_status.ensure(1), "alloc");
  TG_CHECK(c, cudaMemcpyAsync(c->d_eig_status.p, &big, sizeof(int), cudaMemcpyHostToDevice, c->stream), "status");
  return TG_OK;
}

int read_eig_status(tg_ctx* c) {
  int v = 0x7fffffff;
  TG_CHECK(c, cudaMemcpyAsync(&v, c->d_eig_status.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream), "status");
  TG_CHECK(c, cudaStreamSynchronize(c->stream), "sync");
  if (v != 0x7fffffff) {
    char b[128];
    snprintf(b, sizeof b, "eigensolver did not converge for table row %d", v - 1);
    return set_err(c, TG_ERR_NUMERIC, b);
  }
  return TG_OK;
}

// the real-axis BZ is the uniform imaginary-axis k list (same points, same order): its
// H(k) tables and eigendecompositions are those of the imaginary axis
bool real_k_is_imag_k(tg_ctx* c) { return c->imag_uniform && c->real_set && c->h_rkp == c->h_klist_u; }

// the chi0 layout in use: the selected orbitals, or every orbital (gathered when the fused
// Green-function kernels have no operand output stage for this dimension)
ChiView full_view(tg_ctx* c);

ChiView chi_view(tg_ctx* c) {
  if (!c->chi_sel_on) return full_view(c);
  ChiLayout& L = c->chi_sel;
  ChiView v;
  v.dimens = L.dimens;
  v.ld = (int64_t)L.nsel * L.nsel;
  v.gather = true;
  v.outmap = L.d_outmap.p; v.decode = L.d_decode.p; v.norb = L.d_norb.p;
  v.pair_M = L.d_pair_M.p; v.pair_aoff = L.d_pair_aoff.p; v.pair_coff = L.d_pair_coff.p;
  v.tiles = L.d_tiles.p; v.ntiles = (int)L.tiles.size(); v.split = &L.split;
  v.sgA = L.d_sgA.p; v.sgB = L.d_sgB.p; v.stiles = L.d_stiles.p;
  v.rows = L.d_rows.p; v.nrows = L.nsel;
  return v;
}

// ChiLayout of the orbitals orbs[i] (ascending local indices) of every site i
int build_chi_layout(tg_ctx* c, const std::vector<std::vector<int>>& orbs, ChiLayout& L) {
  const int nat = c->n_atoms, n = c->dimH, np2 = nat * nat;
  L.nc.assign(nat, 0);
  int dens = 0, nsel = 0;
  for (int i = 0; i < nat; ++i) {
    L.nc[i] = (int)orbs[i].size();
    dens += L.nc[i] * L.nc[i];
    nsel += 2 * L.nc[i];
  }
  L.dimens = 4 * dens;
  L.nsel = nsel;
  L.pair_M.assign(np2, 0);
  L.pair_aoff.assign(np2, 0);
  L.pair_coff.assign(np2, 0);
  L.tiles.clear();
  std::vector<int> outmap((size_t)nsel * nsel);
  // full-G row of the x-th selected row of site i: spin block x / nc, orbital orbs[i][x % nc]
  auto row_of = [&](int i, int x) { return c->ia[i] + (x / L.nc[i]) * c->norb[i] + orbs[i][x % L.nc[i]]; };
  int aoff = 0;
  int64_t coff = 0;
  const int T = gemm64_tile();
  for (int i = 0; i < nat; ++i)
    for (int j = 0; j < nat; ++j) {
      const int p = i * nat + j;
      const int M = 4 * L.nc[i] * L.nc[j];
      L.pair_M[p] = M;
      L.pair_aoff[p] = aoff;
      L.pair_coff[p] = coff;
      const int ni2 = 2 * L.nc[i], nj2 = 2 * L.nc[j];
      for (int x = 0; x < ni2; ++x)
        for (int y = 0; y < nj2; ++y) outmap[aoff + x * nj2 + y] = row_of(i, x) * n + row_of(j, y);
      for (int u0 = 0; u0 < M; u0 += T)
        for (int v0 = 0; v0 < M; v0 += T) L.tiles.push_back(PairTile{p, u0, v0});
      aoff += M;
      coff += (int64_t)M * M;
    }
  // chi row decode over the selected orbitals (sigmaimunu2i order restricted to them)
  std::vector<int> decode(L.dimens);
  int kount = 0;
  for (int i = 0; i < nat; ++i)
    for (int mu = 0; mu < L.nc[i]; ++mu)
      for (int nu = 0; nu < L.nc[i]; ++nu)
        for (int sg = 0; sg < 4; ++sg) decode[kount++] = sg | (i << 2) | (mu << 12) | (nu << 18);
  split_build_layout(np2, L.pair_M.data(), L.pair_aoff.data(), L.split);
  cudaStream_t s = c->stream;
  std::vector<int> rows;
  for (int i = 0; i < nat; ++i)
    for (int x = 0; x < 2 * L.nc[i]; ++x) rows.push_back(row_of(i, x));
  TG_CHECK(c, L.d_rows.upload(rows.data(), rows.size(), s), "upload");
  TG_CHECK(c, L.d_outmap.upload(outmap.data(), outmap.size(), s), "upload");
  TG_CHECK(c, L.d_decode.upload(decode.data(), decode.size(), s), "upload");
  TG_CHECK(c, L.d_norb.upload(L.nc.data(), nat, s), "upload");
  TG_CHECK(c, L.d_pair_M.upload(L.pair_M.data(), np2, s), "upload");
  TG_CHECK(c, L.d_pair_aoff.upload(L.pair_aoff.data(), np2, s), "upload");
  TG_CHECK(c, L.d_pair_coff.upload(L.pair_coff.data(), np2, s), "upload");
  TG_CHECK(c, L.d_tiles.upload(L.tiles.data(), L.tiles.size(), s), "upload");
  TG_CHECK(c, L.d_sgA.upload(L.split.groupsA.data(), L.split.groupsA.size(), s), "upload");
  TG_CHECK(c, L.d_sgB.upload(L.split.groupsB.data(), L.split.groupsB.size(), s), "upload");
  TG_CHECK(c, L.d_stiles.upload(L.split.tiles.data(), L.split.tiles.size(), s), "upload");
  TG_CHECK(c, cudaStreamSynchronize(s), "sync");
  return TG_OK;
}

// every orbital, in the layout of tg_set_system
ChiView full_view(tg_ctx* c) {
  ChiView v;
  v.dimens = c->dimens;
  v.ld = (int64_t)c->dimH * c->dimH;
  v.gather = !green_supported(c->dimH);
  v.outmap = c->d_outmap.p; v.decode = c->d_decode.p; v.norb = c->d_norb.p;
  v.pair_M = c->d_pair_M.p; v.pair_aoff = c->d_pair_aoff.p; v.pair_coff = c->d_pair_coff.p;
  v.tiles = c->d_tiles.p; v.ntiles = (int)c->tiles.size(); v.split = &c->split;
  v.sgA = c->d_sgA.p; v.sgB = c->d_sgB.p; v.stiles = c->d_stiles.p;
  v.rows = c->d_allrows.p; v.nrows = c->dimH;
  return v;
}

int nsplit_view(tg_ctx* c, const ChiView& v) {
  int s = std::max(1, c->num_sms / std::max(v.ntiles, 1));
  return std::min(s, 64);
}

// contraction of one pass into Cpart on the FP64 path
int contract(tg_ctx* c, const ChiView& v, const double2* A, const double2* B, int64_t np, double2* Cpart, int nsplit,
             int64_t cstride) {
  c->launches += 1;
  TG_CHECK(c, launch_gemm64(A, B, v.ld, np, nsplit, v.tiles, v.ntiles, v.pair_M, v.pair_aoff, v.pair_coff, Cpart,
                            cstride, c->stream),
           "contraction (fp64)");
  return TG_OK;
}

// chunks of a pass: runs of equal key (energy), at most maxc points each
template <class Key>
SplitChunks make_chunks(int64_t np, int maxc, Key key) {
  SplitChunks ch;
  int64_t i = 0;
  ch.kstart.push_back(0);
  while (i < np) {
    const auto k0 = key(i);
    int64_t j = i + 1;
    while (j < np && j - i < maxc && key(j) == k0) ++j;
    const int cnt = (int)(j - i);
    const int nk = (cnt + kSplitK - 1) / kSplitK;
    const int ci = (int)ch.count.size();
    ch.slot0.push_back((int)i);
    ch.count.push_back(cnt);
    ch.kstart.push_back(ch.kstart.back() + nk);
    for (int t = 0; t < nk; ++t) ch.kchunk.push_back(ci);
    i = j;
  }
  return ch;
}

// chunks of a k-major pass over a tabulated mesh of ne energies (work item p0 + i = k * ne
// + energy): the slots of one energy are ne apart, so every energy of the pass is cut into
// chunks of at most maxc points with stride ne
SplitChunks make_chunks_kmajor(int64_t p0, int64_t np, int64_t ne, int maxc) {
  SplitChunks ch;
  ch.stride = (int)ne;
  ch.kstart.push_back(0);
  const int64_t e0 = p0 % ne;
  for (int64_t ie = 0; ie < ne; ++ie) {
    const int64_t first = (ie - e0 + ne) % ne;   // first slot of energy ie
    if (first >= np) continue;
    const int64_t total = (np - 1 - first) / ne + 1;
    for (int64_t done = 0; done < total; done += maxc) {
      const int cnt = (int)std::min<int64_t>(maxc, total - done);
      const int nk = (cnt + kSplitK - 1) / kSplitK;
      const int ci = (int)ch.count.size();
      ch.slot0.push_back((int)(first + done * ne));
      ch.count.push_back(cnt);
      ch.kstart.push_back(ch.kstart.back() + nk);
      for (int t = 0; t < nk; ++t) ch.kchunk.push_back(ci);
    }
  }
  return ch;
}

// uploads the chunk tables and sizes the digit / exponent buffers of a pass
int split_prepare(tg_ctx* c, const ChiView& v, const SplitChunks& ch, SplitPassDev& pd) {
  const int nc = ch.n_chunks(), nks = ch.n_ksteps();
  std::vector<int> buf;
  buf.reserve(3 * nc + 1 + nks);
  buf.insert(buf.end(), ch.slot0.begin(), ch.slot0.end());
  buf.insert(buf.end(), ch.count.begin(), ch.count.end());
  buf.insert(buf.end(), ch.kstart.begin(), ch.kstart.end());
  buf.insert(buf.end(), ch.kchunk.begin(), ch.kchunk.end());
  TG_CHECK(c, c->d_chunks.upload(buf.data(), buf.size(), c->stream), "upload chunks");
  pd.n_chunks = nc;
  pd.n_ksteps = nks;
  pd.stride = ch.stride;
  pd.max_count = nc > 0 ? *std::max_element(ch.count.begin(), ch.count.end()) : 0;
  pd.slot0 = c->d_chunks.p;
  pd.count = c->d_chunks.p + nc;
  pd.kstart = c->d_chunks.p + 2 * nc;
  pd.kchunk = c->d_chunks.p + 3 * nc + 1;
  const size_t ld = (size_t)v.ld;
  TG_CHECK(c, c->d_digA.ensure((size_t)nks * v.split->groupsA.size() * kSplitABlock), "alloc digits A");
  TG_CHECK(c, c->d_digB.ensure((size_t)nks * v.split->groupsB.size() * kSplitBBlock), "alloc digits B");
  TG_CHECK(c, c->d_m64A.ensure((size_t)nc * ld), "alloc");
  TG_CHECK(c, c->d_m64B.ensure((size_t)nc * ld), "alloc");
  TG_CHECK(c, c->d_EA.ensure((size_t)nc * ld), "alloc");
  TG_CHECK(c, c->d_EB.ensure((size_t)nc * ld), "alloc");
  return TG_OK;
}

// FP64 operand of a pass -> digits (which = 0: A, 1: B)
// (e16: the operand's exponent sidecar when its Green functions wrote one, else null)
int split_quantize_operand(tg_ctx* c, const ChiView& v, int which, const double2* X, const SplitPassDev& pd,
                           const int16_t* e16) {
  const int64_t ld = v.ld;
  unsigned long long* m64 = which ? c->d_m64B.p : c->d_m64A.p;
  TG_CHECK(c, cudaMemsetAsync(m64, 0, sizeof(unsigned long long) * pd.n_chunks * ld, c->stream), "memset");
  if (e16)
    TG_CHECK(c, split_rowmax_e16(e16, ld, pd, m64, c->stream), "split rowmax (sidecar)");
  else
    TG_CHECK(c, split_rowmax(X, ld, pd, m64, c->stream), "split rowmax");
  if (which == 0)
    TG_CHECK(c, split_quantize(X, ld, pd, v.sgA, (int)v.split->groupsA.size(), kSplitRowsA, false, m64, c->d_EA.p,
                               c->d_digA.p, c->stream),
             "split quantize A");
  else
    TG_CHECK(c, split_quantize(X, ld, pd, v.sgB, (int)v.split->groupsB.size(), kSplitColsB, true, m64, c->d_EB.p,
                               c->d_digB.p, c->stream),
             "split quantize B");
  c->launches += 2;
  return TG_OK;
}

// bnd (null: none): the pass's quantisation bound per site pair, added into bnd[n_pairs]
int split_contract_pass(tg_ctx* c, const ChiView& v, const SplitPassDev& pd, double2* Cpart, int nsplit,
                        int64_t cstride, double* bnd = nullptr) {
  if (bnd) {
    TG_CHECK(c, split_bound(c->d_m64A.p, c->d_m64B.p, v.ld, pd, v.pair_M, v.pair_aoff, c->n_atoms * c->n_atoms, bnd,
                            c->stream),
             "split bound");
    c->launches += 1;
  }
  SplitContractArgs sa;
  sa.A = c->d_digA.p;
  sa.B = c->d_digB.p;
  sa.GA = (int)v.split->groupsA.size();
  sa.GB = (int)v.split->groupsB.size();
  sa.tiles = v.stiles;
  sa.ntiles = (int)v.split->tiles.size();
  sa.nsplit = nsplit;
  sa.pass = pd;
  sa.EA = c->d_EA.p;
  sa.EB = c->d_EB.p;
  sa.ld = v.ld;
  sa.pair_M = v.pair_M;
  sa.pair_aoff = v.pair_aoff;
  sa.pair_coff = v.pair_coff;
  sa.C = Cpart;
  sa.cstride = cstride;
  sa.err = c->d_split_err.p;
  sa.num_ctas = c->num_sms;
  c->launches += 1;
  TG_CHECK(c, split_contract(sa, c->stream), "contraction (split)");
  return TG_OK;
}

// per-result accumulators of the split bound (results x [imaginary, real] x site pairs)
int bound_begin(tg_ctx* c, bool split, int n_res) {
  c->err_bound.assign((size_t)n_res, std::nan(""));   // until the call completes
  if (!split) return TG_OK;
  const size_t len = (size_t)n_res * 2 * c->n_atoms * c->n_atoms;
  TG_CHECK(c, c->d_bound.ensure(len), "alloc bound");
  TG_CHECK(c, cudaMemsetAsync(c->d_bound.p, 0, sizeof(double) * len, c->stream), "memset");
  return TG_OK;
}

double* bound_at(tg_ctx* c, bool split, int res, int axis) {
  return split ? c->d_bound.p + ((size_t)res * 2 + axis) * c->n_atoms * c->n_atoms : nullptr;
}

// after the results are on the host (stream synchronised): chi = (C_ij + conj C_ji - i D_ij) / 2 pi
// entry by entry, so ||E_chi||_F <= (2 ||E_C||_F + ||E_D||_F) / 2 pi, and per site pair
// ||E_C,t||_F <= 2 sqrt(2) 6.02 2^-46 sum_c count_c ||2^E_A|| ||2^E_B|| (a complex product is four
// real products, each within 6.02 2^(E_A + E_B - 46) per point); relative to ||chi||_F of the
// result as returned (FP64 accumulation rounding, which the FP64 path shares, not included)
int bound_finish(tg_ctx* c, bool split, int n_res, int64_t cstride, const double* chiorb) {
  if (!split) {
    c->err_bound.assign((size_t)n_res, 0.0);
    return TG_OK;
  }
  const int np2 = c->n_atoms * c->n_atoms;
  std::vector<double> h((size_t)n_res * 2 * np2);
  TG_CHECK(c, cudaMemcpy(h.data(), c->d_bound.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost), "copy bound");
  const double kappa = 2.0 * std::sqrt(2.0) * 6.02 * std::ldexp(1.0, -46) / (2.0 * kPi);
  for (int r = 0; r < n_res; ++r) {
    double sc = 0.0, sd = 0.0;
    for (int t = 0; t < np2; ++t) {
      const double bc = h[((size_t)r * 2) * np2 + t], bd = h[((size_t)r * 2 + 1) * np2 + t];
      sc += bc * bc;
      sd += bd * bd;
    }
    const double err = kappa * (2.0 * std::sqrt(sc) + std::sqrt(sd));
    double part[8] = {};   // independent sums: one chain of additions would bound the loop
    const double* x = chiorb + 2 * (size_t)r * cstride;
    for (int64_t i = 0; i < 2 * cstride; i += 8)   // (cstride is a square of a multiple of 4)
      for (int j = 0; j < 8; ++j) part[j] += x[i + j] * x[i + j];
    double nrm = 0.0;
    for (double y : part) nrm += y;
    nrm = std::sqrt(nrm);
    c->err_bound[r] = err == 0.0 ? 0.0 : (nrm > 0.0 ? err / nrm : HUGE_VAL);
  }
  return TG_OK;
}

// K-range split count of the contraction of a pass of P points: the cost-model choice, or
// with autotuning on, the fastest of 1, 2, 4, ..., 64 and the count that fills every SM
// equally, measured once per layout (precision,
// tiles, K-steps of a pass) on zero operands (the kernels' time does not depend on the
// values) with CUDA events, into scratch accumulators, and cached in the context
int choose_nsplit(tg_ctx* c, const ChiView& v, bool split, int64_t P, int* out) {
  const int model = split ? split_nsplit((int)v.split->tiles.size(), c->num_sms, P / kSplitK) : nsplit_view(c, v);
  *out = model;
  if (!c->autotune || P <= 0) {
    c->last_nsplit[split ? 1 : 0] = model;
    return TG_OK;
  }
  const std::vector<int64_t> key = {split ? 1 : 0, v.ntiles, (int64_t)(split ? v.split->tiles.size() : 0), P,
                                    (int64_t)v.dimens, (int64_t)c->split_chunk};
  for (auto& kv : c->tuned)
    if (kv.first == key) {
      *out = kv.second;
      c->last_nsplit[split ? 1 : 0] = kv.second;
      return TG_OK;
    }
  cudaStream_t s = c->stream;
  const int64_t cstride = (int64_t)v.dimens * v.dimens;
  SplitPassDev pd;
  if (split) {
    const int64_t chunk = c->split_chunk;
    const SplitChunks ch = make_chunks(P, c->split_chunk, [&](int64_t i) { return i / chunk; });
    int rc = split_prepare(c, v, ch, pd);
    if (rc) return rc;
    TG_CHECK(c, cudaMemsetAsync(c->d_digA.p, 0, c->d_digA.n, s), "memset");
    TG_CHECK(c, cudaMemsetAsync(c->d_digB.p, 0, c->d_digB.n, s), "memset");
    TG_CHECK(c, cudaMemsetAsync(c->d_EA.p, 0, sizeof(int) * c->d_EA.n, s), "memset");
    TG_CHECK(c, cudaMemsetAsync(c->d_EB.p, 0, sizeof(int) * c->d_EB.n, s), "memset");
    TG_CHECK(c, c->d_split_err.ensure(1), "alloc");
    TG_CHECK(c, cudaMemsetAsync(c->d_split_err.p, 0, sizeof(int), s), "memset");
  } else {
    TG_CHECK(c, c->d_A.ensure((size_t)P * v.ld), "alloc A");
    TG_CHECK(c, c->d_B.ensure((size_t)P * v.ld), "alloc B");
    TG_CHECK(c, cudaMemsetAsync(c->d_A.p, 0, sizeof(double2) * P * v.ld, s), "memset");
    TG_CHECK(c, cudaMemsetAsync(c->d_B.p, 0, sizeof(double2) * P * v.ld, s), "memset");
  }
  float best_ms = 0.f;
  int best = model;
  // 1, 2, 4, .. 64 and the smallest count whose tiles fill every SM equally (37 for the 36 and
  // 216 tiles of two spd sites on 148 SMs)
  const int tiles = split ? (int)v.split->tiles.size() : v.ntiles;
  std::vector<int> counts = {1, 2, 4, 8, 16, 32, 64};
  for (int ns = 1; ns <= 64; ++ns)
    if ((int64_t)tiles * ns % c->num_sms == 0) {
      if (std::find(counts.begin(), counts.end(), ns) == counts.end()) counts.push_back(ns);
      break;
    }
  for (int ns : counts) {
    if ((int64_t)ns * v.ntiles > (int64_t)64 * c->num_sms * 64) continue;
    TG_CHECK(c, c->d_tune.ensure((size_t)ns * cstride), "alloc tuning accumulators");
    float ms = 0.f;
    for (int rep = 0; rep < 2; ++rep) {   // the first launch warms up
      TG_CHECK(c, cudaMemsetAsync(c->d_tune.p, 0, sizeof(double2) * ns * cstride, s), "memset");
      TG_CHECK(c, cudaEventRecord(c->ev[6], s), "event");
      int rc = split ? split_contract_pass(c, v, pd, c->d_tune.p, ns, cstride)
                     : contract(c, v, c->d_A.p, c->d_B.p, P, c->d_tune.p, ns, cstride);
      if (rc) return rc;
      TG_CHECK(c, cudaEventRecord(c->ev[7], s), "event");
      TG_CHECK(c, cudaEventSynchronize(c->ev[7]), "sync");
      TG_CHECK(c, cudaEventElapsedTime(&ms, c->ev[6], c->ev[7]), "timing");
    }
    if (ns == 1 || ms < best_ms) {
      best_ms = ms;
      best = ns;
    }
  }
  c->tuned.push_back({key, best});
  c->last_nsplit[split ? 1 : 0] = best;
  *out = best;
  return TG_OK;
}

// Green functions of a chi0 pass into the operand buffers: fused (the kernel writes the
// operand layouts), or gathered (column-major G into d_graw, then the view's slots)
// whether the launch of g (through chi_green) writes an exponent sidecar beside its operand:
// the spectral kernel does, and so does the gather kernel for every gathered operand
bool writes_sidecar(const ChiView& v, const GreenArgs& g) { return v.gather || g.triQ || green_is_spectral(g); }

int chi_green(tg_ctx* c, const ChiView& v, const GreenArgs& g, const char* what) {
  // the tridiagonalised path writes G column-major only: its operands are always gathered
  if (!v.gather && !g.triQ) {
    TG_CHECK(c, launch_green(g, c->num_sms, c->stream, nullptr), what);
    return TG_OK;
  }
  GreenArgs r = g;
  r.mode = MODE_RAW;
  r.out = c->d_graw.p;
  r.out2 = nullptr;
  r.eout = r.eout2 = nullptr;
  if (g.triQ) {
    TG_CHECK(c, c->d_triws.ensure(tri_ws_entries(c->dimH, g.np)), "alloc factors");
    r.triws = c->d_triws.p;
    c->launches += 1;
  }
  TG_CHECK(c, launch_green(r, c->num_sms, c->stream, nullptr), what);
  TG_CHECK(c, launch_gather(g, c->d_graw.p, g.mode, v.outmap, v.ld, g.out, g.eout, c->num_sms, c->stream), what);
  if (g.out2)
    TG_CHECK(c, launch_gather(g, c->d_graw.p, g.mode2, v.outmap, v.ld, g.out2, g.eout2, c->num_sms, c->stream),
             what);
  c->launches += g.out2 ? 2 : 1;
  return TG_OK;
}

}  // namespace

extern "C" {

int tg_create(int device, tg_ctx** out) {
  if (!out) return TG_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0) return TG_ERR_CUDA;
  if (device < 0 || device >= ndev) return TG_ERR_ARG;
  tg_ctx* c = new tg_ctx();
  c->device = device;
  e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
  for (int i = 0; i < 8 && e == cudaSuccess; ++i) e = cudaEventCreate(&c->ev[i]);
  if (e == cudaSuccess) e = c->d_status.ensure(1);
  if (e != cudaSuccess) {
    tg_destroy(c);
    return TG_ERR_CUDA;
  }
  *out = c;
  return TG_OK;
}

int tg_destroy(tg_ctx* c) {
  if (!c) return TG_OK;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  c->d_R.free_(); c->d_pair_start.free_(); c->d_pair_neigh.free_(); c->d_row_atom.free_();
  c->d_row_orb.free_(); c->d_row_spin.free_(); c->d_outmap.free_(); c->d_decode.free_(); c->d_norb.free_();
  c->d_pair_M.free_(); c->d_pair_aoff.free_(); c->d_exp_rows.free_(); c->d_gg_desc.free_(); c->d_pair_coff.free_();
  c->d_pair_t.free_(); c->d_h0.free_(); c->d_tiles.free_(); c->d_y.free_(); c->d_kp.free_(); c->d_w.free_();
  c->d_rkp.free_(); c->d_rw.free_(); c->d_x2.free_(); c->d_p2.free_(); c->d_A.free_(); c->d_B.free_();
  c->d_C.free_(); c->d_D.free_(); c->d_chi.free_(); c->d_acc.free_(); c->d_acc_red.free_(); c->d_zlist.free_();
  c->d_gout.free_(); c->d_klist.free_(); c->d_status.free_();
  c->d_sgA.free_(); c->d_sgB.free_(); c->d_stiles.free_(); c->d_digA.free_(); c->d_digB.free_();
  c->d_m64A.free_(); c->d_m64B.free_(); c->d_EA.free_(); c->d_EB.free_(); c->d_chunks.free_(); c->d_split_err.free_();
  c->d_dy.free_(); c->d_piv.free_();
  c->d_ylist.free_(); c->d_klist_u.free_(); c->d_qvec.free_(); c->d_hphase.free_();
  for (int t = 0; t < 4; ++t) c->d_htab[t].free_();
  c->d_hchunk.free_();
  for (int i = 0; i < 8; ++i)
    if (c->ev[i]) cudaEventDestroy(c->ev[i]);
  for (cudaEvent_t e : c->ev_pool) cudaEventDestroy(e);
  for (auto& u : c->ev_used) {
    cudaEventDestroy(u.second.first);
    cudaEventDestroy(u.second.second);
  }
  c->stage.release();
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;   // every DevArray member frees what the calls above did not
  return TG_OK;
}

const char* tg_last_error(const tg_ctx* c) { return c ? c->err.c_str() : "null context"; }

int tg_system_shape(const tg_ctx* c, int* n_atoms, int* norb_max, int* norb) {
  if (!c || !n_atoms || !norb_max) return TG_ERR_ARG;
  if (!c->sys_set) return TG_ERR_STATE;
  *n_atoms = c->n_atoms;
  *norb_max = c->nmax;
  if (norb)
    for (int i = 0; i < c->n_atoms; ++i) norb[i] = c->norb[i];
  return TG_OK;
}

int tg_set_system(tg_ctx* c, int n_atoms, const int* norb, int norb_max, int n_neigh, const double* cell_vec,
                  const int* basis_idx, const int* is_hopping, const double* t0i) {
  if (!c) return TG_ERR_ARG;
  if (n_atoms <= 0 || n_atoms > 1023 || !norb || norb_max <= 0 || norb_max > 63 || n_neigh < 0)
    return set_err(c, TG_ERR_ARG, "tg_set_system: bad sizes");
  if (n_neigh > 0 && (!cell_vec || !basis_idx || !is_hopping || !t0i))
    return set_err(c, TG_ERR_ARG, "tg_set_system: null neighbour arrays");
  cudaSetDevice(c->device);
  c->n_atoms = n_atoms;
  c->nmax = norb_max;
  c->n_neigh = n_neigh;
  c->norb.assign(norb, norb + n_atoms);
  for (int i = 0; i < n_atoms; ++i)
    if (c->norb[i] <= 0 || c->norb[i] > norb_max) return set_err(c, TG_ERR_ARG, "tg_set_system: norb out of range");
  c->ia.resize(n_atoms);
  int pos = 0, dens = 0;
  for (int i = 0; i < n_atoms; ++i) {
    c->ia[i] = pos;
    pos += 2 * c->norb[i];
    dens += c->norb[i] * c->norb[i];
  }
  c->dimH = pos;
  c->dimens = 4 * dens;
  if (!green_supported(c->dimH) && !green_cluster_supported(c->dimH, MODE_RAW)) {
    char b[128];
    snprintf(b, sizeof b, "dimH = %d is beyond the largest supported dimension (288)", c->dimH);
    return set_err(c, TG_ERR_ARG, b);
  }
  c->chi_sel_on = false;
  if (!green_supported(c->dimH))
    TG_CHECK(c, c->d_clws.ensure(green_cluster_ws_bytes(c->dimH, c->num_sms)), "alloc cluster workspace");
  const int n = c->dimH;
  // row tables
  std::vector<int> ratom(n), rorb(n), rspin(n);
  for (int i = 0; i < n_atoms; ++i)
    for (int s = 0; s < 2; ++s)
      for (int o = 0; o < c->norb[i]; ++o) {
        const int r = c->ia[i] + s * c->norb[i] + o;
        ratom[r] = i;
        rorb[r] = o;
        rspin[r] = s;
      }
  // hopping blocks grouped by (row atom = neighbour basis index j, col atom = i)
  const int np2 = n_atoms * n_atoms;
  std::vector<std::vector<std::pair<int, int>>> lists(np2);   // (neighbour, site i)
  for (int k = 0; k < n_neigh; ++k) {
    const int j = basis_idx[k] - 1;
    if (j < 0 || j >= n_atoms) return set_err(c, TG_ERR_ARG, "tg_set_system: basis_idx out of range");
    for (int i = 0; i < n_atoms; ++i)
      if (is_hopping[(size_t)k * n_atoms + i]) lists[j * n_atoms + i].push_back({k, i});
  }
  std::vector<int> pstart(np2 + 1, 0), pneigh;
  std::vector<double2> pt;
  const size_t blk = (size_t)norb_max * norb_max;
  for (int pidx = 0; pidx < np2; ++pidx) {
    pstart[pidx] = (int)pneigh.size();
    for (auto& kv : lists[pidx]) {
      const int k = kv.first, i = kv.second;
      pneigh.push_back(k);
      const double* src = t0i + 2 * (((size_t)k * n_atoms + i) * blk);
      for (size_t e = 0; e < blk; ++e) pt.push_back(make_double2(src[2 * e], src[2 * e + 1]));
    }
  }
  pstart[np2] = (int)pneigh.size();
  // pair-block operand layout, C offsets, output map, gemm tiles
  c->pair_M.assign(np2, 0);
  c->pair_aoff.assign(np2, 0);
  c->pair_coff.assign(np2, 0);
  std::vector<int> outmap((size_t)n * n);
  int aoff = 0;
  int64_t coff = 0;
  c->tiles.clear();
  const int T = gemm64_tile();
  for (int i = 0; i < n_atoms; ++i)
    for (int j = 0; j < n_atoms; ++j) {
      const int p = i * n_atoms + j;
      const int M = 4 * c->norb[i] * c->norb[j];
      c->pair_M[p] = M;
      c->pair_aoff[p] = aoff;
      c->pair_coff[p] = coff;
      const int ni2 = 2 * c->norb[i], nj2 = 2 * c->norb[j];
      for (int x = 0; x < ni2; ++x)
        for (int y = 0; y < nj2; ++y) outmap[aoff + x * nj2 + y] = (c->ia[i] + x) * n + (c->ia[j] + y);
      for (int u0 = 0; u0 < M; u0 += T)
        for (int v0 = 0; v0 < M; v0 += T) c->tiles.push_back(PairTile{p, u0, v0});
      aoff += M;
      coff += (int64_t)M * M;
    }
  // chi row decode: sigmaimunu2i order (sigma fastest, then nu, mu, site)
  std::vector<int> decode(c->dimens);
  int kount = 0;
  for (int i = 0; i < n_atoms; ++i)
    for (int mu = 0; mu < c->norb[i]; ++mu)
      for (int nu = 0; nu < c->norb[i]; ++nu)
        for (int s = 0; s < 4; ++s) decode[kount++] = s | (i << 2) | (mu << 12) | (nu << 18);
  // expectation rows (up, down) per orbital
  std::vector<int> exprows(n);
  {
    int o = 0;
    for (int i = 0; i < n_atoms; ++i)
      for (int mu = 0; mu < c->norb[i]; ++mu) {
        exprows[2 * o] = c->ia[i] + mu;
        exprows[2 * o + 1] = c->ia[i] + c->norb[i] + mu;
        ++o;
      }
  }
  cudaStream_t s = c->stream;
  std::vector<double> R(cell_vec, cell_vec + 3 * (size_t)n_neigh);
  TG_CHECK(c, c->d_R.upload(R.data(), R.size(), s), "upload R");
  TG_CHECK(c, c->d_pair_start.upload(pstart.data(), pstart.size(), s), "upload");
  TG_CHECK(c, c->d_pair_neigh.upload(pneigh.data(), pneigh.size(), s), "upload");
  TG_CHECK(c, c->d_pair_t.upload(pt.data(), pt.size(), s), "upload");
  TG_CHECK(c, c->d_row_atom.upload(ratom.data(), n, s), "upload");
  TG_CHECK(c, c->d_row_orb.upload(rorb.data(), n, s), "upload");
  TG_CHECK(c, c->d_row_spin.upload(rspin.data(), n, s), "upload");
  TG_CHECK(c, c->d_outmap.upload(outmap.data(), outmap.size(), s), "upload");
  {
    std::vector<int> all(n);
    for (int r = 0; r < n; ++r) all[r] = r;
    TG_CHECK(c, c->d_allrows.upload(all.data(), all.size(), s), "upload");
  }
  {
    std::vector<int> outinv((size_t)n * n);
    for (size_t o = 0; o < outmap.size(); ++o) outinv[outmap[o]] = (int)o;
    TG_CHECK(c, c->d_outinv.upload(outinv.data(), outinv.size(), s), "upload");
  }
  TG_CHECK(c, c->d_decode.upload(decode.data(), decode.size(), s), "upload");
  TG_CHECK(c, c->d_norb.upload(c->norb.data(), n_atoms, s), "upload");
  TG_CHECK(c, c->d_pair_M.upload(c->pair_M.data(), np2, s), "upload");
  TG_CHECK(c, c->d_pair_aoff.upload(c->pair_aoff.data(), np2, s), "upload");
  TG_CHECK(c, c->d_pair_coff.upload(c->pair_coff.data(), np2, s), "upload");
  TG_CHECK(c, c->d_tiles.upload(c->tiles.data(), c->tiles.size(), s), "upload");
  TG_CHECK(c, c->d_exp_rows.upload(exprows.data(), exprows.size(), s), "upload");
  split_build_layout(np2, c->pair_M.data(), c->pair_aoff.data(), c->split);
  TG_CHECK(c, c->d_sgA.upload(c->split.groupsA.data(), c->split.groupsA.size(), s), "upload");
  TG_CHECK(c, c->d_sgB.upload(c->split.groupsB.data(), c->split.groupsB.size(), s), "upload");
  TG_CHECK(c, c->d_stiles.upload(c->split.tiles.data(), c->split.tiles.size(), s), "upload");
  TG_CHECK(c, cudaStreamSynchronize(s), "sync");
  c->sys_set = true;
  c->h0_set = false;
  return TG_OK;
}

int tg_set_h0(tg_ctx* c, int dimH, const double* h0) {
  if (!c) return TG_ERR_ARG;
  if (!c->sys_set) return set_err(c, TG_ERR_STATE, "tg_set_system has not been called");
  if (dimH != c->dimH || !h0) return set_err(c, TG_ERR_ARG, "tg_set_h0: dimH mismatch");
  cudaSetDevice(c->device);
  TG_CHECK(c, c->d_h0.upload(reinterpret_cast<const double2*>(h0), (size_t)dimH * dimH, c->stream), "upload h0");
  TG_CHECK(c, cudaStreamSynchronize(c->stream), "sync");
  c->h0_set = true;
  return TG_OK;
}

int tg_set_imag_mesh(tg_ctx* c, int64_t n_points, const double* y, const double* kp, const double* w) {
  if (!c) return TG_ERR_ARG;
  if (n_points < 0 || (n_points > 0 && (!y || !kp || !w))) return set_err(c, TG_ERR_ARG, "tg_set_imag_mesh: bad args");
  cudaSetDevice(c->device);
  TG_CHECK(c, c->d_y.upload(y, n_points, c->stream), "upload y");
  TG_CHECK(c, c->d_kp.upload(kp, 3 * n_points, c->stream), "upload kp");
  TG_CHECK(c, c->d_w.upload(w, n_points, c->stream), "upload w");
  c->h_y.assign(y, y + n_points);
  // uniform structure: consecutive blocks of constant y, all with the first block's k list
  c->imag_uniform = false;
  if (n_points > 0) {
    int64_t nk = 1;
    while (nk < n_points && y[nk] == y[0]) ++nk;
    bool ok = (n_points % nk) == 0;
    const int64_t ne = ok ? n_points / nk : 0;
    std::vector<double> ylist;
    for (int64_t e = 0; ok && e < ne; ++e) {
      const double ye = y[e * nk];
      ylist.push_back(ye);
      for (int64_t i = 0; i < nk && ok; ++i) {
        const int64_t p = e * nk + i;
        ok = y[p] == ye && kp[3 * p] == kp[3 * i] && kp[3 * p + 1] == kp[3 * i + 1] && kp[3 * p + 2] == kp[3 * i + 2];
      }
    }
    if (ok && ne > 1) {
      TG_CHECK(c, c->d_ylist.upload(ylist.data(), ne, c->stream), "upload ylist");
      TG_CHECK(c, c->d_klist_u.upload(kp, 3 * nk, c->stream), "upload klist");
      c->h_klist_u.assign(kp, kp + 3 * nk);
      c->imag_uniform = true;
      c->n_e_u = ne;
      c->nk_u = nk;
    }
  }
  TG_CHECK(c, cudaStreamSynchronize(c->stream), "sync");
  c->n_imag = n_points;
  c->imag_set = true;
  return TG_OK;
}

int tg_set_real_mesh(tg_ctx* c, int64_t n_k, const double* kp, const double* w) {
  if (!c) return TG_ERR_ARG;
  if (n_k < 0 || (n_k > 0 && (!kp || !w))) return set_err(c, TG_ERR_ARG, "tg_set_real_mesh: bad args");
  cudaSetDevice(c->device);
  TG_CHECK(c, c->d_rkp.upload(kp, 3 * n_k, c->stream), "upload kp");
  TG_CHECK(c, c->d_rw.upload(w, n_k, c->stream), "upload w");
  TG_CHECK(c, cudaStreamSynchronize(c->stream), "sync");
  c->h_rkp.assign(kp, kp + 3 * n_k);
  c->n_realk = n_k;
  c->real_set = true;
  return TG_OK;
}

int tg_set_autotune(tg_ctx* c, int enable) {
  if (!c) return TG_ERR_ARG;
  c->autotune = enable != 0;
  if (!c->autotune) c->tuned.clear();
  return TG_OK;
}

int tg_tuning(const tg_ctx* c, int* nsplit_fp64, int* nsplit_split) {
  if (!c || !nsplit_fp64 || !nsplit_split) return TG_ERR_ARG;
  *nsplit_fp64 = c->last_nsplit[0];
  *nsplit_split = c->last_nsplit[1];
  return TG_OK;
}

int tg_chi0_error_bound(tg_ctx* c, int n, double* bound) {
  if (!c) return TG_ERR_ARG;
  if (!bound || n != (int)c->err_bound.size())
    return set_err(c, TG_ERR_ARG, "tg_chi0_error_bound: n must be the number of results of the last chi0 call");
  for (int i = 0; i < n; ++i) bound[i] = c->err_bound[i];
  return TG_OK;
}

int tg_set_split_chunk(tg_ctx* c, int points) {
  if (!c) return TG_ERR_ARG;
  if (points < 0 || points > kSplitMaxChunk)
    return set_err(c, TG_ERR_ARG, "tg_set_split_chunk: points must lie in [0, 16384]");
  c->split_chunk = points == 0 ? 1024 : points;
  return TG_OK;
}

int tg_set_chi_orbitals(tg_ctx* c, const int* mask) {
  if (!c) return TG_ERR_ARG;
  if (!c->sys_set) return set_err(c, TG_ERR_STATE, "tg_set_system has not been called");
  cudaSetDevice(c->device);
  if (!mask) {
    c->chi_sel_on = false;
    return TG_OK;
  }
  std::vector<std::vector<int>> orbs(c->n_atoms);
  int total = 0;
  for (int i = 0; i < c->n_atoms; ++i)
    for (int mu = 0; mu < c->norb[i]; ++mu)
      if (mask[(size_t)i * c->nmax + mu]) {
        orbs[i].push_back(mu);
        ++total;
      }
  if (total == 0) return set_err(c, TG_ERR_ARG, "tg_set_chi_orbitals: no orbital selected");
  c->chi_sel_on = false;
  int rc = build_chi_layout(c, orbs, c->chi_sel);
  if (rc) return rc;
  c->chi_sel_on = true;
  return TG_OK;
}

int tg_chi0_batch(tg_ctx* c, const double* q, int n_omega, const double* e, double Ef, double eta, double etap,
                  int n_real, const double* x2, const double* p2, int precision, int dimens, double* chiorb_hf) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if (!q || !e || n_omega <= 0 || !chiorb_hf) return set_err(c, TG_ERR_ARG, "tg_chi0: null argument");
  const ChiView v = chi_view(c);
  if (dimens != v.dimens) return set_err(c, TG_ERR_ARG, "tg_chi0: dimens mismatch (see tg_set_chi_orbitals)");
  if (precision != TG_PREC_FP64 && precision != TG_PREC_SPLIT) return set_err(c, TG_ERR_ARG, "tg_chi0: precision");
  bool any_real = false;
  for (int w = 0; w < n_omega; ++w) any_real |= std::fabs(e[w]) >= 1e-15;
  if (any_real && (n_real <= 0 || !x2 || !p2)) return set_err(c, TG_ERR_ARG, "tg_chi0: real-axis points missing");
  if (any_real && !c->real_set) return set_err(c, TG_ERR_STATE, "tg_set_real_mesh has not been called");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int n = c->dimH;
  const int64_t nn = (int64_t)n * n;
  const bool split = precision == TG_PREC_SPLIT;
  const int64_t cstride = (int64_t)v.dimens * v.dimens;
  // workspace
  // 6 GiB operands (about 25 GB with the digit planes and tables at dimH = 36): a k-major
  // pass over a tabulated mesh then holds ~2400 points per energy, so the split
  // contraction's chunk ends (one per energy and pass) cost little
  const int64_t P = pass_size(c, std::max<int64_t>(c->n_imag, (int64_t)n_real * c->n_realk), (int64_t)6 << 30);
  int nsplit = 1;
  if ((rc = choose_nsplit(c, v, split, P, &nsplit))) return rc;
  if (split) {
    TG_CHECK(c, c->d_split_err.ensure(1), "alloc");
    TG_CHECK(c, c->d_e16A.ensure((size_t)P * nn), "alloc exponents A");
    TG_CHECK(c, c->d_e16B.ensure((size_t)P * nn), "alloc exponents B");
    TG_CHECK(c, cudaMemsetAsync(c->d_split_err.p, 0, sizeof(int), s), "memset");
  }
  if ((rc = bound_begin(c, split, n_omega))) return rc;
  TG_CHECK(c, c->d_A.ensure((size_t)P * v.ld), "alloc A");
  TG_CHECK(c, c->d_B.ensure((size_t)P * v.ld), "alloc B");
  if (v.gather || chi_tridiag(c)) TG_CHECK(c, c->d_graw.ensure((size_t)P * nn), "alloc G");
  TG_CHECK(c, c->d_C.ensure((size_t)n_omega * nsplit * cstride), "alloc C");
  TG_CHECK(c, c->d_D.ensure((size_t)n_omega * nsplit * cstride), "alloc D");
  TG_CHECK(c, c->d_chi.ensure((size_t)cstride), "alloc chi");
  TG_CHECK(c, cudaMemsetAsync(c->d_C.p, 0, sizeof(double2) * n_omega * nsplit * cstride, s), "memset");
  TG_CHECK(c, cudaMemsetAsync(c->d_D.p, 0, sizeof(double2) * n_omega * nsplit * cstride, s), "memset");
  if (any_real) {
    TG_CHECK(c, c->d_x2.upload(x2, (size_t)n_omega * n_real, s), "upload x2");
    TG_CHECK(c, c->d_p2.upload(p2, (size_t)n_omega * n_real, s), "upload p2");
  }
  rc = reset_status(c);
  if (rc) return rc;
  profile_begin(c);
  float t_green = 0, t_con = 0, t_epi = 0;
  cudaEvent_t *ev = c->ev;
  TG_CHECK(c, cudaEventRecord(ev[0], s), "event");
  // ---------------- H(k) tables (k-major traversal) ----------------
  const bool q_zero = q[0] == 0.0 && q[1] == 0.0 && q[2] == 0.0;
  const double zero3[3] = {0.0, 0.0, 0.0};
  const bool spec = chi_spectral(c);
  // otherwise, on meshes whose energies share a k list: G over the rows chi needs from a
  // Householder tridiagonalisation per k, kept as T and those rows of Q (built from bounded H
  // chunks); its operands are gathered
  const bool tri_ok = chi_tridiag(c);
  const bool tri_imag = tri_ok && c->imag_uniform && c->nk_u > 0 &&
                        tri_room(c, c->nk_u, v.nrows, 0, q_zero ? -1 : 1);
  if (tri_imag) {
    if ((rc = build_tri_chunked(c, 0, c->d_klist_u.p, c->nk_u, zero3, v))) return rc;
    if (!q_zero && (rc = build_tri_chunked(c, 1, c->d_klist_u.p, c->nk_u, q, v))) return rc;
  }
  const bool alias_tri = tri_imag && any_real && real_k_is_imag_k(c);
  const bool tri_real = tri_ok && any_real && !alias_tri && c->n_realk > 0 &&
                        tri_room(c, c->n_realk, v.nrows, 2, q_zero ? -1 : 3);
  if (tri_real) {
    if ((rc = build_tri_chunked(c, 2, c->d_rkp.p, c->n_realk, zero3, v))) return rc;
    if (!q_zero && (rc = build_tri_chunked(c, 3, c->d_rkp.p, c->n_realk, q, v))) return rc;
  }
  const bool tab_imag = !tri_imag && c->imag_uniform &&
                        (int64_t)c->nk_u * c->dimH * c->dimH * 16 <= ((int64_t)8 << 30);
  const bool tab_real = !tri_real && !alias_tri && any_real &&
                        (int64_t)c->n_realk * c->dimH * c->dimH * 16 <= ((int64_t)8 << 30);
  if (spec && (rc = reset_eig_status(c))) return rc;
  if (tab_imag) {
    if ((rc = build_htab(c, 0, c->d_klist_u.p, c->nk_u, zero3))) return rc;
    if (spec && (rc = build_eig(c, 0, c->nk_u))) return rc;
    if (!q_zero && (rc = build_htab(c, 1, c->d_klist_u.p, c->nk_u, q))) return rc;
    if (!q_zero && spec && (rc = build_eig(c, 1, c->nk_u))) return rc;
  }
  // real-axis slots 2 / 3 alias the imaginary-axis slots 0 / 1 when the k lists coincide
  const bool alias_real = (tab_imag && tab_real && real_k_is_imag_k(c)) || alias_tri;
  const int rslot0 = alias_real ? 0 : 2, rslot1 = alias_real ? 1 : 3;
  // a real-axis BZ of its own: spectral Green functions from eigendecompositions built out of
  // bounded H chunks (only U and lambda are kept, so long BZs qualify too) when they fit in
  // memory, else Gauss-Jordan on resident H tables when those fit
  const bool eig_real = any_real && !alias_real && spec && eig_room(c, c->n_realk, 2, q_zero ? -1 : 3);
  const bool tab_real_gj = tab_real && !alias_real && !eig_real;
  const bool kmajor_real = alias_real || tab_real_gj || eig_real || tri_real;
  if (tab_real_gj) {
    if ((rc = build_htab(c, 2, c->d_rkp.p, c->n_realk, zero3))) return rc;
    if (!q_zero && (rc = build_htab(c, 3, c->d_rkp.p, c->n_realk, q))) return rc;
  }
  if (eig_real) {
    if ((rc = build_eig_chunked(c, 2, c->d_rkp.p, c->n_realk, zero3))) return rc;
    if (!q_zero && (rc = build_eig_chunked(c, 3, c->d_rkp.p, c->n_realk, q))) return rc;
  }
  auto use_table = [&](GreenArgs& g, int slot, int64_t n_e, int64_t nk, const double* ylist) {
    g.n_e = n_e;
    g.nk_tab = nk;
    g.ylist = ylist;
    if (slot < 2 ? tri_imag : tri_real) {
      g.htab = nullptr;
      g.triD = c->d_triD[slot].p;
      g.triE = c->d_triE[slot].p;
      g.triQ = c->d_triQ[slot].p;
      g.trirows = v.rows;
      g.tri_ns = v.nrows;
      return;
    }
    g.htab = eig_real && slot >= 2 ? nullptr : c->d_htab[slot].p;
    if (spec && (slot < 2 || eig_real)) {
      g.eigU = c->d_eigU[slot].p;
      g.eigL = c->d_eigL[slot].p;
      g.outinv = c->d_outinv.p;
    }
  };
  // ---------------- imaginary axis ----------------
  for (int64_t p0 = 0; p0 < c->n_imag; p0 += P) {
    const int64_t np = std::min<int64_t>(P, c->n_imag - p0);
    GreenArgs g2 = base_args(c);
    g2.pts.kind = 0;
    g2.pts.y = c->d_y.p;
    g2.pts.kp = c->d_kp.p;
    g2.pts.w = c->d_w.p;
    g2.p0 = p0;
    g2.np = np;
    g2.zr = Ef;
    g2.zi = etap;
    g2.mode = MODE_B_IMAG;
    g2.out = c->d_B.p;
    if (tab_imag || tri_imag) use_table(g2, 0, c->n_e_u, c->nk_u, c->d_ylist.p);
    // G1 = G2 when e = 0, q = 0 and eta = eta': one inversion feeds both operands
    int w_start = 0;
    if (e[0] == 0.0 && q_zero && eta == etap) {
      g2.out2 = c->d_A.p;
      g2.mode2 = MODE_A_IMAG;
      w_start = 1;
    }
    // the split row maxima read exponent sidecars when the spectral kernel or the gather
    // kernel writes the operand
    const bool e16_g2 = split && writes_sidecar(v, g2);
    if (e16_g2) {
      g2.eout = c->d_e16B.p;
      if (g2.out2) g2.eout2 = c->d_e16A.p;
    }
    cudaEventRecord(ev[1], s);
    {
      KindTimer kt(c, 0);
      if ((rc = chi_green(c, v, g2, "green (imag, G2)"))) return rc;
    }
    cudaEventRecord(ev[2], s);
    float ms = 0;
    SplitPassDev pd;
    if (split) {
      KindTimer kt(c, 3);
      const double* yv = c->h_y.data() + p0;
      const SplitChunks ch = tab_imag || tri_imag ? make_chunks_kmajor(p0, np, c->n_e_u, c->split_chunk)
                                      : make_chunks(np, c->split_chunk, [&](int64_t i) { return yv[i]; });
      if ((rc = split_prepare(c, v, ch, pd))) return rc;
      if ((rc = split_quantize_operand(c, v, 1, c->d_B.p, pd, e16_g2 ? c->d_e16B.p : nullptr))) return rc;
    }
    if (w_start == 1) {
      if (split) {
        {
          KindTimer kq(c, 3);
          if ((rc = split_quantize_operand(c, v, 0, c->d_A.p, pd, e16_g2 ? c->d_e16A.p : nullptr))) return rc;
        }
        KindTimer kt(c, 1);
        rc = split_contract_pass(c, v, pd, c->d_C.p, nsplit, cstride, bound_at(c, split, 0, 0));
      } else {
        KindTimer kt(c, 1);
        rc = contract(c, v, c->d_A.p, c->d_B.p, np, c->d_C.p, nsplit, cstride);
      }
      if (rc) return rc;
    }
    for (int w = w_start; w < n_omega; ++w) {
      GreenArgs g1 = g2;
      g1.out2 = nullptr;
      g1.eout = g1.eout2 = nullptr;
      g1.zr = Ef + e[w];
      g1.zi = eta;
      g1.q[0] = q[0]; g1.q[1] = q[1]; g1.q[2] = q[2];
      g1.mode = MODE_A_IMAG;
      g1.out = c->d_A.p;
      if (tab_imag || tri_imag) {
        use_table(g1, q_zero ? 0 : 1, c->n_e_u, c->nk_u, c->d_ylist.p);
        g1.q[0] = g1.q[1] = g1.q[2] = 0.0;   // q is inside the table
      }
      const bool e16_g1 = split && writes_sidecar(v, g1);
      if (e16_g1) g1.eout = c->d_e16A.p;
      {
        KindTimer kt(c, 0);
        if ((rc = chi_green(c, v, g1, "green (imag, G1)"))) return rc;
      }
      {
        double2* Cw = c->d_C.p + (size_t)w * nsplit * cstride;
        if (split) {
          {
            KindTimer kq(c, 3);
            rc = split_quantize_operand(c, v, 0, c->d_A.p, pd, e16_g1 ? c->d_e16A.p : nullptr);
          }
          KindTimer kt(c, 1);
          if (!rc) rc = split_contract_pass(c, v, pd, Cw, nsplit, cstride, bound_at(c, split, w, 0));
        } else {
          KindTimer kt(c, 1);
          rc = contract(c, v, c->d_A.p, c->d_B.p, np, Cw, nsplit, cstride);
        }
      }
      if (rc) return rc;
    }
    cudaEventRecord(ev[4], s);
    TG_CHECK(c, cudaEventSynchronize(ev[4]), "sync");
    cudaEventElapsedTime(&ms, ev[1], ev[2]);
    t_green += ms;
    cudaEventElapsedTime(&ms, ev[2], ev[4]);
    t_con += ms;   // includes the G1 inversions of w >= 1 (split below is approximate)
  }
  // the real-axis time is measured from here (also when the imaginary-axis list is empty:
  // an event that was never recorded would make cudaEventElapsedTime fail below)
  TG_CHECK(c, cudaEventRecord(ev[4], s), "event");
  // ---------------- real axis ----------------
  for (int w = 0; w < n_omega; ++w) {
    if (std::fabs(e[w]) < 1e-15) continue;
    const int64_t ntot = (int64_t)n_real * c->n_realk;
    for (int64_t p0 = 0; p0 < ntot; p0 += P) {
      const int64_t np = std::min<int64_t>(P, ntot - p0);
      GreenArgs gr = base_args(c);
      gr.pts.kind = 1;
      gr.pts.kp = c->d_rkp.p;
      gr.pts.w = c->d_rw.p;
      gr.pts.x2 = c->d_x2.p + (size_t)w * n_real;
      gr.pts.p2 = c->d_p2.p + (size_t)w * n_real;
      gr.pts.nk = c->n_realk;
      gr.p0 = p0;
      gr.np = np;
      // G2 = G(k, x2 + i eta') -> conj(G2)
      gr.zr = 0.0;
      gr.zi = etap;
      gr.mode = MODE_B_REAL;
      gr.out = c->d_B.p;
      if (kmajor_real) use_table(gr, rslot0, n_real, c->n_realk, nullptr);
      const bool e16_rb = split && writes_sidecar(v, gr);
      gr.eout = e16_rb ? c->d_e16B.p : nullptr;
      {
        KindTimer kt(c, 0);
        if ((rc = chi_green(c, v, gr, "green (real, G2)"))) return rc;
      }
      // G1 = G(k + q, x2 + e + i eta) -> w (G1 - G1^dagger)
      gr.zr = e[w];
      gr.zi = eta;
      gr.q[0] = q[0]; gr.q[1] = q[1]; gr.q[2] = q[2];
      gr.mode = MODE_A_REAL;
      gr.out = c->d_A.p;
      if (kmajor_real) {
        use_table(gr, q_zero ? rslot0 : rslot1, n_real, c->n_realk, nullptr);
        gr.q[0] = gr.q[1] = gr.q[2] = 0.0;
      }
      const bool e16_ra = split && writes_sidecar(v, gr);
      gr.eout = e16_ra ? c->d_e16A.p : nullptr;
      {
        KindTimer kt(c, 0);
        if ((rc = chi_green(c, v, gr, "green (real, G1)"))) return rc;
      }
      {
        double2* Dw = c->d_D.p + (size_t)w * nsplit * cstride;
        if (split) {
          SplitPassDev pr;
          const int64_t nrk = c->n_realk, pbase = p0;
          {
            KindTimer kq(c, 3);
            const SplitChunks ch = kmajor_real ? make_chunks_kmajor(pbase, np, n_real, c->split_chunk)
                                            : make_chunks(np, c->split_chunk,
                                                          [&](int64_t i) { return (pbase + i) / nrk; });
            rc = split_prepare(c, v, ch, pr);
            if (!rc) rc = split_quantize_operand(c, v, 1, c->d_B.p, pr, e16_rb ? c->d_e16B.p : nullptr);
            if (!rc) rc = split_quantize_operand(c, v, 0, c->d_A.p, pr, e16_ra ? c->d_e16A.p : nullptr);
          }
          KindTimer kt(c, 1);
          if (!rc) rc = split_contract_pass(c, v, pr, Dw, nsplit, cstride, bound_at(c, split, w, 1));
        } else {
          KindTimer kt(c, 1);
          rc = contract(c, v, c->d_A.p, c->d_B.p, np, Dw, nsplit, cstride);
        }
      }
      if (rc) return rc;
    }
  }
  cudaEventRecord(ev[5], s);
  // ---------------- epilogue per frequency ----------------
  for (int w = 0; w < n_omega; ++w) {
    KindTimer kt(c, 2);
    TG_CHECK(c, launch_chi_epilogue(c->d_C.p + (size_t)w * nsplit * cstride, c->d_D.p + (size_t)w * nsplit * cstride,
                                    nsplit, cstride, v.dimens, v.decode, v.norb, v.pair_coff,
                                    c->n_atoms, 1.0 / (2.0 * kPi), c->d_chi.p, s),
             "epilogue");
    TG_CHECK(c, copy_host(c, chiorb_hf + 2 * (size_t)w * cstride, c->d_chi.p, sizeof(double2) * cstride, false),
             "copy chi");
  }
  cudaEventRecord(ev[6], s);
  TG_CHECK(c, cudaEventSynchronize(ev[6]), "sync");
  float ms_real = 0, ms_epi = 0, ms_tot = 0;
  cudaEventElapsedTime(&ms_real, ev[4], ev[5]);
  cudaEventElapsedTime(&ms_epi, ev[5], ev[6]);
  cudaEventElapsedTime(&ms_tot, ev[0], ev[6]);
  t_epi = ms_epi;
  c->last_ms[0] = t_green;
  c->last_ms[1] = t_con + ms_real;
  c->last_ms[2] = t_epi;
  c->last_ms[3] = ms_tot;
  profile_end(c);
  rc = read_status(c);
  if (rc) return rc;
  if (spec && (rc = read_eig_status(c))) return rc;
  if (split) {
    int err = 0;
    TG_CHECK(c, cudaMemcpy(&err, c->d_split_err.p, sizeof(int), cudaMemcpyDeviceToHost), "split status");
    if (err) {
      char b[128];
      snprintf(b, sizeof b, "split contraction: a bounded wait expired (site %d)", err);
      return set_err(c, TG_ERR_TIMEOUT, b);
    }
  }
  return bound_finish(c, split, n_omega, cstride, chiorb_hf);
}

int tg_chi0(tg_ctx* c, const double* q, double e, double Ef, double eta, double etap, int n_real, const double* x2,
            const double* p2, int precision, int dimens, double* chiorb_hf) {
  return tg_chi0_batch(c, q, 1, &e, Ef, eta, etap, n_real, x2, p2, precision, dimens, chiorb_hf);
}

}  // extern "C"

namespace {

// chi0 for n_q wave vectors and n_omega frequencies with G2 shared by all of them: on meshes
// without H(k) tables (adaptive imaginary axes, large real-axis BZs) G2 = G(k, z) does not
// depend on q, so every pass inverts and quantises it once and contracts it with G1(k + q, z + e)
// of every (q, e); on the real axis G2(k, x2 + i eta') depends on e (through x2) but not on q:
// with spectral Green functions every (q, e) forms it again from U(k) instead, with
// tridiagonalised ones (every H(k + q) decomposed up front) it serves every q.
// Accumulators: n_q x n_omega x nsplit chi-sized partials for each axis.
int chi0_qshared(tg_ctx* c, int n_q, const double* qs, int n_omega, const double* e, double Ef, double eta,
                 double etap, int n_real, bool split, double* chiorb_hf) {
  cudaStream_t s = c->stream;
  const ChiView v = chi_view(c);
  const int n = c->dimH;
  const int64_t nn = (int64_t)n * n;
  const int64_t cstride = (int64_t)v.dimens * v.dimens;
  const int64_t P = pass_size(c, std::max<int64_t>(c->n_imag, (int64_t)n_real * c->n_realk), (int64_t)6 << 30);
  int nsplit = 1;
  int rc = choose_nsplit(c, v, split, P, &nsplit);
  if (rc) return rc;
  const int64_t nacc = (int64_t)n_q * n_omega * nsplit * cstride;
  if (split) {
    TG_CHECK(c, c->d_split_err.ensure(1), "alloc");
    TG_CHECK(c, cudaMemsetAsync(c->d_split_err.p, 0, sizeof(int), s), "memset");
  }
  TG_CHECK(c, c->d_A.ensure((size_t)P * v.ld), "alloc A");
  TG_CHECK(c, c->d_B.ensure((size_t)P * v.ld), "alloc B");
  if (v.gather || chi_tridiag(c)) TG_CHECK(c, c->d_graw.ensure((size_t)P * nn), "alloc G");
  TG_CHECK(c, c->d_C.ensure((size_t)nacc), "alloc C");
  TG_CHECK(c, c->d_D.ensure((size_t)nacc), "alloc D");
  TG_CHECK(c, c->d_chi.ensure((size_t)cstride), "alloc chi");
  TG_CHECK(c, cudaMemsetAsync(c->d_C.p, 0, sizeof(double2) * nacc, s), "memset");
  TG_CHECK(c, cudaMemsetAsync(c->d_D.p, 0, sizeof(double2) * nacc, s), "memset");
  if ((rc = bound_begin(c, split, n_q * n_omega))) return rc;
  auto acc_at = [&](double2* base, int iq, int w) { return base + ((size_t)iq * n_omega + w) * nsplit * cstride; };
  if ((rc = reset_status(c))) return rc;
  profile_begin(c);
  cudaEvent_t* ev = c->ev;
  TG_CHECK(c, cudaEventRecord(ev[0], s), "event");
  auto contract_into = [&](const SplitPassDev& pd, int64_t np, double2* Cw, double* bnd) -> int {
    if (split) {
      KindTimer kt(c, 1);
      return split_contract_pass(c, v, pd, Cw, nsplit, cstride, bnd);
    }
    KindTimer kt(c, 1);
    return contract(c, v, c->d_A.p, c->d_B.p, np, Cw, nsplit, cstride);
  };
  // ---------------- imaginary axis: G2 once per pass ----------------
  for (int64_t p0 = 0; p0 < c->n_imag; p0 += P) {
    const int64_t np = std::min<int64_t>(P, c->n_imag - p0);
    GreenArgs g2 = base_args(c);
    g2.pts.kind = 0;
    g2.pts.y = c->d_y.p;
    g2.pts.kp = c->d_kp.p;
    g2.pts.w = c->d_w.p;
    g2.p0 = p0;
    g2.np = np;
    g2.zr = Ef;
    g2.zi = etap;
    g2.mode = MODE_B_IMAG;
    g2.out = c->d_B.p;
    {
      KindTimer kt(c, 0);
      if ((rc = chi_green(c, v, g2, "green (imag, G2)"))) return rc;
    }
    SplitPassDev pd;
    if (split) {
      KindTimer kq(c, 3);
      const double* yv = c->h_y.data() + p0;
      const SplitChunks ch = make_chunks(np, c->split_chunk, [&](int64_t i) { return yv[i]; });
      if ((rc = split_prepare(c, v, ch, pd))) return rc;
      if ((rc = split_quantize_operand(c, v, 1, c->d_B.p, pd, nullptr))) return rc;
    }
    for (int iq = 0; iq < n_q; ++iq)
      for (int w = 0; w < n_omega; ++w) {
        GreenArgs g1 = g2;
        g1.zr = Ef + e[w];
        g1.zi = eta;
        g1.q[0] = qs[3 * iq]; g1.q[1] = qs[3 * iq + 1]; g1.q[2] = qs[3 * iq + 2];
        g1.mode = MODE_A_IMAG;
        g1.out = c->d_A.p;
        {
          KindTimer kt(c, 0);
          if ((rc = chi_green(c, v, g1, "green (imag, G1)"))) return rc;
        }
        if (split) {
          KindTimer kq(c, 3);
          if ((rc = split_quantize_operand(c, v, 0, c->d_A.p, pd, nullptr))) return rc;
        }
        if ((rc = contract_into(pd, np, acc_at(c->d_C.p, iq, w), bound_at(c, split, iq * n_omega + w, 0)))) return rc;
      }
  }
  // ---------------- real axis, spectral or tridiagonalised ----------------
  // the real-axis BZ is one k list for every energy: with its eigendecompositions, or its
  // Householder tridiagonalisations (H(k) once, H(k + q) once per q, from bounded H chunks), G2
  // and G1 of every frequency cost a GEMM per point (or block of energies); G2 is formed again
  // for each q, which costs far less than sharing an inversion per point
  bool any_real = false;
  for (int w = 0; w < n_omega; ++w) any_real |= std::fabs(e[w]) >= 1e-15;
  const bool eig_real = any_real && chi_spectral(c) && eig_room(c, c->n_realk, 2, 3);
  const bool tri_real = any_real && !eig_real && chi_tridiag(c) && tri_room(c, c->n_realk, v.nrows, 2, 3);
  if (eig_real || tri_real) {
    const double zero3[3] = {0.0, 0.0, 0.0};
    const bool e16 = split;   // the spectral kernel or the gather kernel writes every operand here
    if (e16) {
      TG_CHECK(c, c->d_e16A.ensure((size_t)P * nn), "alloc exponents A");
      TG_CHECK(c, c->d_e16B.ensure((size_t)P * nn), "alloc exponents B");
    }
    if (eig_real) {
      if ((rc = reset_eig_status(c))) return rc;
      if ((rc = build_eig_chunked(c, 2, c->d_rkp.p, c->n_realk, zero3))) return rc;
    } else if ((rc = build_tri_chunked(c, 2, c->d_rkp.p, c->n_realk, zero3, v))) {
      return rc;
    }
    auto use_eig = [&](GreenArgs& g, int slot) {
      g.htab = nullptr;
      g.n_e = n_real;
      g.nk_tab = c->n_realk;
      g.ylist = nullptr;
      if (eig_real) {
        g.eigU = c->d_eigU[slot].p;
        g.eigL = c->d_eigL[slot].p;
        g.outinv = c->d_outinv.p;
      } else {
        g.triD = c->d_triD[slot].p;
        g.triE = c->d_triE[slot].p;
        g.triQ = c->d_triQ[slot].p;
        g.trirows = v.rows;
        g.tri_ns = v.nrows;
      }
    };
    const int64_t ntot = (int64_t)n_real * c->n_realk;
    // slot of each wave vector's H(k + q) decomposition (2: that of H(k), for q = 0)
    std::vector<int> qslot(n_q, 2), nzq;
    for (int iq = 0; iq < n_q; ++iq) {
      const double* qi = qs + 3 * iq;
      if (!(qi[0] == 0.0 && qi[1] == 0.0 && qi[2] == 0.0)) nzq.push_back(iq);
    }
    // every pass and frequency: G2 once (and quantised once), then G1 of each wave vector in iqs
    auto real_passes = [&](const std::vector<int>& iqs) -> int {
      for (int w = 0; w < n_omega; ++w) {
        if (std::fabs(e[w]) < 1e-15) continue;
        for (int64_t p0 = 0; p0 < ntot; p0 += P) {
          const int64_t np = std::min<int64_t>(P, ntot - p0);
          GreenArgs gr = base_args(c);
          gr.pts.kind = 1;
          gr.pts.kp = c->d_rkp.p;
          gr.pts.w = c->d_rw.p;
          gr.pts.x2 = c->d_x2.p + (size_t)w * n_real;
          gr.pts.p2 = c->d_p2.p + (size_t)w * n_real;
          gr.pts.nk = c->n_realk;
          gr.p0 = p0;
          gr.np = np;
          gr.zr = 0.0;
          gr.zi = etap;
          gr.mode = MODE_B_REAL;
          gr.out = c->d_B.p;
          gr.eout = e16 ? c->d_e16B.p : nullptr;
          use_eig(gr, 2);
          int rc2 = 0;
          {
            KindTimer kt(c, 0);
            if ((rc2 = chi_green(c, v, gr, "green (real, G2)"))) return rc2;
          }
          SplitPassDev pr;
          if (split) {
            KindTimer kq(c, 3);
            const SplitChunks ch = make_chunks_kmajor(p0, np, n_real, c->split_chunk);
            if ((rc2 = split_prepare(c, v, ch, pr))) return rc2;
            if ((rc2 = split_quantize_operand(c, v, 1, c->d_B.p, pr, e16 ? c->d_e16B.p : nullptr))) return rc2;
          }
          for (int iq : iqs) {
            GreenArgs g1 = gr;
            g1.zr = e[w];
            g1.zi = eta;
            g1.mode = MODE_A_REAL;
            g1.out = c->d_A.p;
            g1.eout = e16 ? c->d_e16A.p : nullptr;
            use_eig(g1, qslot[iq]);
            {
              KindTimer kt(c, 0);
              if ((rc2 = chi_green(c, v, g1, "green (real, G1)"))) return rc2;
            }
            if (split) {
              KindTimer kq(c, 3);
              if ((rc2 = split_quantize_operand(c, v, 0, c->d_A.p, pr, e16 ? c->d_e16A.p : nullptr))) return rc2;
            }
            if ((rc2 = contract_into(pr, np, acc_at(c->d_D.p, iq, w), bound_at(c, split, iq * n_omega + w, 1))))
              return rc2;
          }
        }
      }
      return TG_OK;
    };
    // tridiagonalisations of every H(k + q) at once, where they fit, let G2 serve every q
    std::vector<int> qslots;
    for (size_t j = 0; j < nzq.size(); ++j) qslots.push_back(4 + (int)j);
    const bool share = tri_real && n_q > 1 && (int)nzq.size() <= kTriQSlots &&
                       tri_room_slots(c, c->n_realk, v.nrows, qslots);
    if (share) {
      for (size_t j = 0; j < nzq.size(); ++j) {
        const int iq = nzq[j];
        qslot[iq] = qslots[j];
        if ((rc = build_tri_chunked(c, qslot[iq], c->d_rkp.p, c->n_realk, qs + 3 * iq, v))) return rc;
      }
      std::vector<int> all(n_q);
      for (int iq = 0; iq < n_q; ++iq) all[iq] = iq;
      if ((rc = real_passes(all))) return rc;
    } else {
      for (int iq = 0; iq < n_q; ++iq) {
        const double* qi = qs + 3 * iq;
        const bool qz = qi[0] == 0.0 && qi[1] == 0.0 && qi[2] == 0.0;
        if (!qz) {
          qslot[iq] = 3;
          if (eig_real && (rc = build_eig_chunked(c, 3, c->d_rkp.p, c->n_realk, qi))) return rc;
          if (tri_real && (rc = build_tri_chunked(c, 3, c->d_rkp.p, c->n_realk, qi, v))) return rc;
        }
        if ((rc = real_passes({iq}))) return rc;
      }
    }
  }
  // ---------------- real axis: G2 once per pass and frequency ----------------
  for (int w = 0; w < n_omega && !eig_real && !tri_real; ++w) {
    if (std::fabs(e[w]) < 1e-15) continue;
    const int64_t ntot = (int64_t)n_real * c->n_realk;
    for (int64_t p0 = 0; p0 < ntot; p0 += P) {
      const int64_t np = std::min<int64_t>(P, ntot - p0);
      GreenArgs gr = base_args(c);
      gr.pts.kind = 1;
      gr.pts.kp = c->d_rkp.p;
      gr.pts.w = c->d_rw.p;
      gr.pts.x2 = c->d_x2.p + (size_t)w * n_real;
      gr.pts.p2 = c->d_p2.p + (size_t)w * n_real;
      gr.pts.nk = c->n_realk;
      gr.p0 = p0;
      gr.np = np;
      gr.zr = 0.0;
      gr.zi = etap;
      gr.mode = MODE_B_REAL;
      gr.out = c->d_B.p;
      {
        KindTimer kt(c, 0);
        if ((rc = chi_green(c, v, gr, "green (real, G2)"))) return rc;
      }
      SplitPassDev pr;
      const int64_t nrk = c->n_realk, pbase = p0;
      if (split) {
        KindTimer kq(c, 3);
        const SplitChunks ch = make_chunks(np, c->split_chunk, [&](int64_t i) { return (pbase + i) / nrk; });
        if ((rc = split_prepare(c, v, ch, pr))) return rc;
        if ((rc = split_quantize_operand(c, v, 1, c->d_B.p, pr, nullptr))) return rc;
      }
      for (int iq = 0; iq < n_q; ++iq) {
        GreenArgs g1 = gr;
        g1.zr = e[w];
        g1.zi = eta;
        g1.q[0] = qs[3 * iq]; g1.q[1] = qs[3 * iq + 1]; g1.q[2] = qs[3 * iq + 2];
        g1.mode = MODE_A_REAL;
        g1.out = c->d_A.p;
        {
          KindTimer kt(c, 0);
          if ((rc = chi_green(c, v, g1, "green (real, G1)"))) return rc;
        }
        if (split) {
          KindTimer kq(c, 3);
          if ((rc = split_quantize_operand(c, v, 0, c->d_A.p, pr, nullptr))) return rc;
        }
        if ((rc = contract_into(pr, np, acc_at(c->d_D.p, iq, w), bound_at(c, split, iq * n_omega + w, 1))))
          return rc;
      }
    }
  }
  TG_CHECK(c, cudaEventRecord(ev[5], s), "event");
  // ---------------- epilogue per (q, frequency) ----------------
  for (int iq = 0; iq < n_q; ++iq)
    for (int w = 0; w < n_omega; ++w) {
      KindTimer kt(c, 2);
      TG_CHECK(c, launch_chi_epilogue(acc_at(c->d_C.p, iq, w), acc_at(c->d_D.p, iq, w), nsplit, cstride, v.dimens,
                                      v.decode, v.norb, v.pair_coff, c->n_atoms, 1.0 / (2.0 * kPi), c->d_chi.p, s),
               "epilogue");
      TG_CHECK(c, copy_host(c, chiorb_hf + 2 * ((size_t)iq * n_omega + w) * cstride, c->d_chi.p,
                            sizeof(double2) * cstride, false),
               "copy chi");
    }
  TG_CHECK(c, cudaEventRecord(ev[6], s), "event");
  TG_CHECK(c, cudaEventSynchronize(ev[6]), "sync");
  float ms_tot = 0, ms_epi = 0;
  cudaEventElapsedTime(&ms_tot, ev[0], ev[6]);
  cudaEventElapsedTime(&ms_epi, ev[5], ev[6]);
  c->last_ms[0] = 0.0;
  c->last_ms[1] = ms_tot - ms_epi;
  c->last_ms[2] = ms_epi;
  c->last_ms[3] = ms_tot;
  profile_end(c);
  if ((rc = read_status(c))) return rc;
  if (eig_real && (rc = read_eig_status(c))) return rc;
  if (split) {
    int err = 0;
    TG_CHECK(c, cudaMemcpy(&err, c->d_split_err.p, sizeof(int), cudaMemcpyDeviceToHost), "split status");
    if (err) {
      char b[128];
      snprintf(b, sizeof b, "split contraction: a bounded wait expired (site %d)", err);
      return set_err(c, TG_ERR_TIMEOUT, b);
    }
  }
  return bound_finish(c, split, n_q * n_omega, cstride, chiorb_hf);
}

}  // namespace

extern "C" {

int tg_chi0_qbatch(tg_ctx* c, int n_q, const double* q, int n_omega, const double* e, double Ef, double eta,
                   double etap, int n_real, const double* x2, const double* p2, int precision, int dimens,
                   double* chiorb_hf) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if (n_q <= 0 || !q || !e || n_omega <= 0 || !chiorb_hf) return set_err(c, TG_ERR_ARG, "tg_chi0_qbatch: bad args");
  const ChiView v = chi_view(c);
  if (dimens != v.dimens) return set_err(c, TG_ERR_ARG, "tg_chi0_qbatch: dimens mismatch (see tg_set_chi_orbitals)");
  if (precision != TG_PREC_FP64 && precision != TG_PREC_SPLIT)
    return set_err(c, TG_ERR_ARG, "tg_chi0_qbatch: precision");
  bool any_real = false;
  for (int w = 0; w < n_omega; ++w) any_real |= std::fabs(e[w]) >= 1e-15;
  if (any_real && (n_real <= 0 || !x2 || !p2)) return set_err(c, TG_ERR_ARG, "tg_chi0_qbatch: real-axis points missing");
  if (any_real && !c->real_set) return set_err(c, TG_ERR_STATE, "tg_set_real_mesh has not been called");
  const int64_t cstride = (int64_t)dimens * dimens;
  // tabulated imaginary axes: H(k + q) tables and their eigendecompositions are per q, so
  // the frequencies of one q share G2 and the q run one after another; otherwise one G2 per
  // pass serves every q (both axes then sum H(k) inside the inversion kernels)
  const bool tab_imag = c->imag_uniform && (int64_t)c->nk_u * c->dimH * c->dimH * 16 <= ((int64_t)8 << 30);
  // (likewise on uniform meshes whose dimension takes the tridiagonalised path of tg_chi0_batch)
  const bool tri_imag = c->imag_uniform && chi_tridiag(c);
  if (n_q == 1 || tab_imag || tri_imag) {
    double tot[4] = {0, 0, 0, 0};
    std::vector<double> bounds;
    for (int iq = 0; iq < n_q; ++iq) {
      rc = tg_chi0_batch(c, q + 3 * iq, n_omega, e, Ef, eta, etap, n_real, x2, p2, precision, dimens,
                         chiorb_hf + 2 * (size_t)iq * n_omega * cstride);
      if (rc) return rc;
      for (int k = 0; k < 4; ++k) tot[k] += c->last_ms[k];
      bounds.insert(bounds.end(), c->err_bound.begin(), c->err_bound.end());
    }
    for (int k = 0; k < 4; ++k) c->last_ms[k] = tot[k];
    c->err_bound = bounds;
    return TG_OK;
  }
  cudaSetDevice(c->device);
  if (any_real) {
    TG_CHECK(c, c->d_x2.upload(x2, (size_t)n_omega * n_real, c->stream), "upload x2");
    TG_CHECK(c, c->d_p2.upload(p2, (size_t)n_omega * n_real, c->stream), "upload p2");
  }
  return chi0_qshared(c, n_q, q, n_omega, e, Ef, eta, etap, n_real, precision == TG_PREC_SPLIT, chiorb_hf);
}

int tg_last_timing(const tg_ctx* c, double* ms) {
  if (!c || !ms) return TG_ERR_ARG;
  for (int i = 0; i < 4; ++i) ms[i] = c->last_ms[i];
  for (int i = 0; i < 3; ++i) {
    ms[4 + 2 * i] = c->kind_ms[i];
    ms[5 + 2 * i] = c->kind_n[i];
  }
  ms[10] = (double)c->launches;
  ms[11] = c->kind_ms[3];
  ms[12] = c->kind_n[3];
  return TG_OK;
}

int tg_profile(tg_ctx* c, int enable) {
  if (!c) return TG_ERR_ARG;
  c->profile = enable != 0;
  return TG_OK;
}

}  // extern "C"

namespace {

// room for the H(k) tables of nk points in slots 0 .. slots - 1; without it both are given back and
// the inversion kernels form H(k) themselves
bool htab_room(tg_ctx* c, int slots, int64_t nk) {
  const size_t nn = (size_t)c->dimH * c->dimH;
  if (nk * (int64_t)nn * 16 > ((int64_t)8 << 30)) return false;
  bool ok = c->d_hphase.ensure((size_t)nk * std::max(c->n_neigh, 1)) == cudaSuccess;
  for (int i = 0; i < slots && ok; ++i) ok = c->d_htab[i].ensure((size_t)nk * nn) == cudaSuccess;
  if (ok) return true;
  cudaGetLastError();
  c->d_hphase.free_();
  for (int i = 0; i < slots; ++i) c->d_htab[i].free_();
  return false;
}

// the imaginary-axis points at Ef + i (y + eta) in a, and with q those of G(k - q) in b; on a
// uniform mesh with H(k) tables of its k list in the slots 0 and 1, or neither of them
int imag_points(tg_ctx* c, double Ef, double eta, const double* q, GreenArgs& a, GreenArgs* b) {
  a = base_args(c);
  a.pts.kind = 0;
  a.pts.y = c->d_y.p;
  a.pts.kp = c->d_kp.p;
  a.pts.w = c->d_w.p;
  a.zr = Ef;
  a.zi = eta;
  const double zero3[3] = {0.0, 0.0, 0.0};
  const bool table = c->imag_uniform && htab_room(c, q ? 2 : 1, c->nk_u);
  int rc;
  if (table) {
    if ((rc = build_htab(c, 0, c->d_klist_u.p, c->nk_u, zero3))) return rc;
    a.htab = c->d_htab[0].p;
    a.n_e = c->n_e_u;
    a.nk_tab = c->nk_u;
    a.ylist = c->d_ylist.p;
  }
  if (!q) return TG_OK;
  *b = a;
  const double mq[3] = {-q[0], -q[1], -q[2]};
  if (table) {
    if ((rc = build_htab(c, 1, c->d_klist_u.p, c->nk_u, mq))) return rc;
    b->htab = c->d_htab[1].p;
  } else {
    for (int i = 0; i < 3; ++i) b->q[i] = mq[i];
  }
  return TG_OK;
}

// raw Green functions of P points in each of the buffers; P is halved while the device memory does
// not hold them
int ensure_pass(tg_ctx* c, std::initializer_list<DevArray<double2>*> bufs, int64_t& P) {
  for (;;) {
    cudaError_t e = cudaSuccess;
    for (auto* b : bufs)
      if (e == cudaSuccess) e = b->ensure((size_t)P * c->dimH * c->dimH);
    if (e != cudaErrorMemoryAllocation || P <= 64) return cuda_err(c, e, "alloc G");
    cudaGetLastError();
    for (auto* b : bufs) b->free_();
    P = std::max<int64_t>(64, P / 2);
  }
}

// out[e] = sum over the np points that points(a) sets of w G(ent[e].x, ent[e].y): raw Green functions
// of at most 1 GiB per pass, summed by the entry kernel (their buffer is taken before the tables of
// points(a), which can be done without)
template <class Points>
int entry_sums(tg_ctx* c, int64_t np, const std::vector<int2>& ent, std::vector<double2>& out, const char* what,
               Points points) {
  cudaStream_t s = c->stream;
  const int ne = (int)ent.size();
  out.assign(ent.size(), make_double2(0.0, 0.0));
  int64_t P = pass_size(c, np, (int64_t)1 << 30);
  const int parts = entry_partials(P, c->num_sms);
  TG_CHECK(c, c->d_gg_desc.upload(reinterpret_cast<const int*>(ent.data()), 2 * ent.size(), s), "upload");
  TG_CHECK(c, c->d_acc.ensure((size_t)parts * ne), "alloc acc");
  TG_CHECK(c, c->d_acc_red.ensure(ne), "alloc acc");
  int rc = ensure_pass(c, {&c->d_graw}, P);
  if (rc) return rc;
  GreenArgs a;
  if ((rc = points(a))) return rc;
  TG_CHECK(c, cudaMemsetAsync(c->d_acc.p, 0, sizeof(double2) * (size_t)parts * ne, s), "memset");
  if ((rc = reset_status(c))) return rc;
  a.mode = MODE_RAW;
  a.out = c->d_graw.p;
  for (int64_t p0 = 0; p0 < np; p0 += P) {
    a.p0 = p0;
    a.np = std::min<int64_t>(P, np - p0);
    TG_CHECK(c, launch_green(a, c->num_sms, s, nullptr), what);
    TG_CHECK(c, launch_entries(a, c->d_graw.p, reinterpret_cast<const int2*>(c->d_gg_desc.p), ne, c->num_sms,
                               c->d_acc.p, s),
             "entry sums");
  }
  TG_CHECK(c, launch_reduce_blocks(c->d_acc.p, parts, ne, c->d_acc_red.p, s), "reduce");
  TG_CHECK(c, cudaMemcpyAsync(out.data(), c->d_acc_red.p, sizeof(double2) * ne, cudaMemcpyDeviceToHost, s), "copy");
  return read_status(c);
}

// h[16 b + q]: the 16 spin products of orbital pair b summed over the imaginary axis, with
// G(k) in both factors, or (q not null) with G(k) in the first and G(k - q) in the second one,
// and then hs[..] with the two exchanged
int imag_pairs(tg_ctx* c, double Ef, double eta, const double* q, const std::vector<int4>& pairs,
               std::vector<double2>& h, std::vector<double2>* hs) {
  cudaStream_t s = c->stream;
  const int npairs = (int)pairs.size(), len = 16 * npairs, sets = q ? 2 : 1;
  h.assign(len, make_double2(0.0, 0.0));
  if (hs) hs->assign(len, make_double2(0.0, 0.0));
  if (npairs == 0) return TG_OK;
  int64_t P = pass_size(c, c->n_imag, (int64_t)1 << 30);
  const size_t parts = pair_partials(c->dimH, npairs, q != nullptr, c->num_sms, P);
  TG_CHECK(c, c->d_gg_desc.upload(reinterpret_cast<const int*>(pairs.data()), 4 * pairs.size(), s), "upload pairs");
  const int4* dp = reinterpret_cast<const int4*>(c->d_gg_desc.p);
  TG_CHECK(c, c->d_acc.ensure(sets * parts * len), "alloc acc");
  TG_CHECK(c, c->d_acc_red.ensure((size_t)sets * len), "alloc acc");
  int rc = q ? ensure_pass(c, {&c->d_A, &c->d_B}, P) : ensure_pass(c, {&c->d_A}, P);
  if (rc) return rc;
  profile_begin(c);
  GreenArgs a, b;
  if ((rc = imag_points(c, Ef, eta, q, a, &b))) return rc;
  if (!q) b = a;
  TG_CHECK(c, cudaMemsetAsync(c->d_acc.p, 0, sizeof(double2) * sets * parts * len, s), "memset");
  if ((rc = reset_status(c))) return rc;
  a.mode = b.mode = MODE_RAW;
  a.out = c->d_A.p;
  b.out = q ? c->d_B.p : c->d_A.p;
  for (int64_t p0 = 0; p0 < c->n_imag; p0 += P) {
    a.p0 = b.p0 = p0;
    a.np = b.np = std::min<int64_t>(P, c->n_imag - p0);
    {
      KindTimer kt(c, 0);
      TG_CHECK(c, launch_green(a, c->num_sms, s, nullptr), "green (k)");
    }
    if (q) {
      KindTimer kt(c, 0);
      TG_CHECK(c, launch_green(b, c->num_sms, s, nullptr), "green (k - q)");
    }
    KindTimer kt(c, 1);
    c->launches += 1;
    TG_CHECK(c, launch_pairs(a, a.out, b.out, dp, npairs, c->num_sms, c->d_acc.p, s), "pair sums");
  }
  {
    KindTimer kt(c, 2);
    TG_CHECK(c, launch_reduce_blocks(c->d_acc.p, (int)parts, sets * len, c->d_acc_red.p, s), "reduce");
  }
  TG_CHECK(c, cudaMemcpyAsync(h.data(), c->d_acc_red.p, sizeof(double2) * len, cudaMemcpyDeviceToHost, s), "copy");
  if (hs && q)
    TG_CHECK(c, cudaMemcpyAsync(hs->data(), c->d_acc_red.p + len, sizeof(double2) * len, cudaMemcpyDeviceToHost, s),
             "copy");
  profile_end(c);
  return read_status(c);
}

}  // namespace

extern "C" {

int tg_expectation(tg_ctx* c, double Ef, double eta, double* rho, double* mx, double* my, double* mz, double* mp) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_expectation"))) return rc;
  if (!rho || !mx || !my || !mz || !mp) return set_err(c, TG_ERR_ARG, "tg_expectation: null output");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int n = c->dimH;
  const int len = 2 * n;   // 4 complex per orbital, n/2 orbitals
  const int maxgrid = c->num_sms * (green_max_ctas(n) + 1);
  TG_CHECK(c, c->d_acc.ensure((size_t)maxgrid * len), "alloc acc");
  TG_CHECK(c, c->d_acc_red.ensure(len), "alloc acc");
  GreenArgs a;
  if ((rc = imag_points(c, Ef, eta, nullptr, a, nullptr))) return rc;
  a.p0 = 0;
  a.np = c->n_imag;
  a.mode = MODE_EXPECT;
  a.exp_rows = c->d_exp_rows.p;
  a.acc = c->d_acc.p;
  rc = reset_status(c);
  if (rc) return rc;
  int grid = 0;
  if (a.htab && spectral_forced(c)) {
    // uniform mesh: one eigendecomposition per k, the energy sum folded into f_a per k
    if ((rc = reset_eig_status(c))) return rc;
    if ((rc = build_eig(c, 0, c->nk_u))) return rc;
    grid = (int)std::min<int64_t>(c->nk_u, maxgrid);
    c->launches += 1;
    TG_CHECK(c, launch_spec_expect(c->d_eigU[0].p, c->d_eigL[0].p, c->nk_u, n, c->d_ylist.p, c->n_e_u, c->d_w.p, Ef,
                                   eta, c->d_exp_rows.p, c->d_acc.p, grid, s),
             "expectation (spectral)");
    if ((rc = read_eig_status(c))) return rc;
  } else {
    TG_CHECK(c, launch_green(a, c->num_sms, s, &grid), "green (expectation)");
  }
  TG_CHECK(c, launch_reduce_blocks(c->d_acc.p, grid, len, c->d_acc_red.p, s), "reduce");
  std::vector<double2> h(len);
  TG_CHECK(c, cudaMemcpyAsync(h.data(), c->d_acc_red.p, sizeof(double2) * len, cudaMemcpyDeviceToHost, s), "copy");
  rc = read_status(c);
  if (rc) return rc;
  // mod_expectation.F90:121-147
  int o = 0;
  const double pi = kPi;
  for (int i = 0; i < c->n_atoms; ++i) {
    for (int mu = 0; mu < c->nmax; ++mu) {
      const size_t idx = (size_t)i * c->nmax + mu;
      if (mu >= c->norb[i]) {
        rho[idx] = mx[idx] = my[idx] = mz[idx] = 0.0;
        mp[2 * idx] = mp[2 * idx + 1] = 0.0;
        continue;
      }
      const double2 uu = h[4 * o], dd = h[4 * o + 1], ud = h[4 * o + 2], du = h[4 * o + 3];
      const double nu_ = 0.5 + uu.x / pi, nd_ = 0.5 + dd.x / pi;
      rho[idx] = nu_ + nd_;
      mz[idx] = nu_ - nd_;
      const double mpr = (du.x + ud.x) / pi, mpi = (du.y - ud.y) / pi;
      mx[idx] = mpr;
      my[idx] = mpi;
      mp[2 * idx] = mpr;
      mp[2 * idx + 1] = mpi;
      ++o;
    }
  }
  return TG_OK;
}

int tg_gg_tensor(tg_ctx* c, double Ef, double eta, int orbital_resolved, const int* dmask, double* T) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_gg_tensor"))) return rc;
  if (!T || (orbital_resolved && !dmask)) return set_err(c, TG_ERR_ARG, "tg_gg_tensor: null argument");
  cudaSetDevice(c->device);
  const int nat = c->n_atoms;
  // groups per site
  std::vector<std::vector<std::vector<int>>> rowg(nat), colg(nat);
  int nrow = 0, ncol = 0;
  for (int i = 0; i < nat; ++i) {
    // d orbitals of the site from dmask(norb_max, n_atoms) (Types%dOrbs)
    const int no = c->norb[i];
    if (orbital_resolved) {
      std::vector<int> rest;
      for (int o = 0; o < no; ++o) {
        if (dmask[(size_t)i * c->nmax + o]) {
          rowg[i].push_back({o});
          colg[i].push_back({o});
        } else {
          rest.push_back(o);
        }
      }
      rowg[i].push_back(rest);
    } else {
      std::vector<int> all;
      for (int o = 0; o < no; ++o) all.push_back(o);
      rowg[i].push_back(all);
      colg[i].push_back(all);
    }
    nrow = std::max<int>(nrow, (int)rowg[i].size());
    ncol = std::max<int>(ncol, (int)colg[i].size());
  }
  // every orbital pair (row orbital of any site, column orbital of any site) is summed on the
  // device; the groups of several orbitals are added up here
  std::vector<int4> pairs;
  std::vector<int> block;   // output block of a pair
  for (int i = 0; i < nat; ++i)
    for (int j = 0; j < nat; ++j)
      for (int h = 0; h < (int)colg[j].size(); ++h)
        for (int nu : colg[j][h])
          for (int g = 0; g < (int)rowg[i].size(); ++g)
            for (int mu : rowg[i][g]) {
              pairs.push_back(make_int4(c->ia[i] + mu, c->ia[i] + c->norb[i] + mu, c->ia[j] + nu,
                                        c->ia[j] + c->norb[j] + nu));
              block.push_back(((i * nat + j) * nrow + g) * ncol + h);
            }
  std::vector<double2> h;
  if ((rc = imag_pairs(c, Ef, eta, nullptr, pairs, h, nullptr))) return rc;
  const size_t total = (size_t)nat * nat * nrow * ncol * 16;
  std::memset(T, 0, sizeof(double) * 2 * total);
  for (size_t b = 0; b < block.size(); ++b)
    for (int q = 0; q < 16; ++q) {
      const size_t dst = (size_t)block[b] * 16 + q;
      T[2 * dst] += h[16 * b + q].x;
      T[2 * dst + 1] += h[16 * b + q].y;
    }
  return TG_OK;
}

int tg_fermi_column(tg_ctx* c, double Ef, double eta, double* D) {
  int rc = check_ready(c, false, true);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_fermi_column"))) return rc;
  if (!D) return set_err(c, TG_ERR_ARG, "tg_fermi_column: null output");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  double one = 1.0, ef = Ef;
  TG_CHECK(c, c->d_x2.upload(&ef, 1, s), "upload");
  TG_CHECK(c, c->d_p2.upload(&one, 1, s), "upload");
  // the spin blocks uu, dd, ud, du of every orbital's diagonal
  std::vector<int2> ent;
  for (int i = 0; i < c->n_atoms; ++i)
    for (int mu = 0; mu < c->norb[i]; ++mu) {
      const int u = c->ia[i] + mu, d = u + c->norb[i];
      ent.push_back(make_int2(u, u));
      ent.push_back(make_int2(d, d));
      ent.push_back(make_int2(u, d));
      ent.push_back(make_int2(d, u));
    }
  auto points = [&](GreenArgs& a) {
    a = base_args(c);
    a.pts.kind = 1;
    a.pts.kp = c->d_rkp.p;
    a.pts.w = c->d_rw.p;
    a.pts.x2 = c->d_x2.p;
    a.pts.p2 = c->d_p2.p;
    a.pts.nk = c->n_realk;
    a.zr = 0.0;
    a.zi = eta;
    return TG_OK;
  };
  std::vector<double2> g, h(ent.size());
  if ((rc = entry_sums(c, c->n_realk, ent, g, "green (fermi column)", points))) return rc;
  for (size_t o = 0; o + 3 < g.size(); o += 4) {   // traces with 1, sigma_x, sigma_y, sigma_z
    const double2 uu = g[o], dd = g[o + 1], ud = g[o + 2], du = g[o + 3];
    h[o] = cadd(uu, dd);
    h[o + 1] = cadd(du, ud);
    h[o + 2] = cmul(make_double2(0.0, 1.0), csub(ud, du));
    h[o + 3] = csub(uu, dd);
  }
  // D(4, norb_max, n_atoms); orbital counter o runs over the sites' orbitals
  int o = 0;
  for (int i = 0; i < c->n_atoms; ++i) {
    for (int mu = 0; mu < c->nmax; ++mu)
      for (int q = 0; q < 4; ++q) {
        const size_t dst = ((size_t)i * c->nmax + mu) * 4 + q;
        if (mu < c->norb[i]) {
          D[2 * dst] = h[4 * (o + mu) + q].x;
          D[2 * dst + 1] = h[4 * (o + mu) + q].y;
        } else {
          D[2 * dst] = D[2 * dst + 1] = 0.0;
        }
      }
    o += c->norb[i];
  }
  return TG_OK;
}

int tg_green_batch(tg_ctx* c, int64_t nz, const double* z, const double* kp, double* G) {
  int rc = check_ready(c, false, false);
  if (rc) return rc;
  if (nz < 0 || (nz > 0 && (!z || !kp || !G))) return set_err(c, TG_ERR_ARG, "tg_green_batch: bad args");
  if (nz == 0) return TG_OK;
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int64_t nn = (int64_t)c->dimH * c->dimH;
  TG_CHECK(c, c->d_zlist.upload(reinterpret_cast<const double2*>(z), nz, s), "upload z");
  TG_CHECK(c, c->d_klist.upload(kp, 3 * nz, s), "upload k");
  TG_CHECK(c, c->d_gout.ensure((size_t)nz * nn), "alloc G");
  GreenArgs a = base_args(c);
  a.pts.kind = 2;
  a.pts.z = c->d_zlist.p;
  a.pts.kp = c->d_klist.p;
  a.np = nz;
  a.mode = MODE_RAW;
  a.out = c->d_gout.p;
  rc = reset_status(c);
  if (rc) return rc;
  TG_CHECK(c, launch_green(a, c->num_sms, s, nullptr), "green (batch)");
  TG_CHECK(c, cudaMemcpyAsync(G, c->d_gout.p, sizeof(double2) * nz * nn, cudaMemcpyDeviceToHost, s), "copy G");
  return read_status(c);
}

int tg_hamiltk_batch(tg_ctx* c, int64_t nk, const double* kp, double* H) {
  int rc = check_ready(c, false, false);
  if (rc) return rc;
  if (nk < 0 || (nk > 0 && (!kp || !H))) return set_err(c, TG_ERR_ARG, "tg_hamiltk_batch: bad args");
  if (nk == 0) return TG_OK;
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int64_t nn = (int64_t)c->dimH * c->dimH;
  std::vector<double2> zeros(nk, make_double2(0.0, 0.0));
  TG_CHECK(c, c->d_zlist.upload(zeros.data(), nk, s), "upload z");
  TG_CHECK(c, c->d_klist.upload(kp, 3 * nk, s), "upload k");
  TG_CHECK(c, c->d_gout.ensure((size_t)nk * nn), "alloc H");
  GreenArgs a = base_args(c);
  a.pts.kind = 2;
  a.pts.z = c->d_zlist.p;
  a.pts.kp = c->d_klist.p;
  a.np = nk;
  a.mode = MODE_HK;
  a.out = c->d_gout.p;
  if (green_supported(c->dimH)) {
    TG_CHECK(c, launch_green(a, c->num_sms, s, nullptr), "hamiltk");
    TG_CHECK(c, cudaMemcpyAsync(H, c->d_gout.p, sizeof(double2) * nk * nn, cudaMemcpyDeviceToHost, s), "copy H");
    TG_CHECK(c, cudaStreamSynchronize(s), "sync");
    return TG_OK;
  }
  // other dimensions: the row-major H(k) table, transposed to Fortran order on the host
  const double zero3[3] = {0.0, 0.0, 0.0};
  TG_CHECK(c, c->d_hphase.ensure((size_t)nk * std::max(c->n_neigh, 1)), "alloc phases");
  TG_CHECK(c, c->d_qvec.upload(zero3, 3, s), "upload q");
  TG_CHECK(c, launch_hk_table(a, c->d_klist.p, nk, c->d_qvec.p, c->d_hphase.p, c->d_gout.p, s), "H table");
  std::vector<double2> tab((size_t)nk * nn);
  TG_CHECK(c, cudaMemcpyAsync(tab.data(), c->d_gout.p, sizeof(double2) * nk * nn, cudaMemcpyDeviceToHost, s),
           "copy H");
  TG_CHECK(c, cudaStreamSynchronize(s), "sync");
  const int n = c->dimH;
  for (int64_t k = 0; k < nk; ++k)
    for (int r = 0; r < n; ++r)
      for (int cc = 0; cc < n; ++cc) {
        const double2 v = tab[(size_t)k * nn + (size_t)r * n + cc];
        H[2 * ((size_t)k * nn + (size_t)cc * n + r)] = v.x;
        H[2 * ((size_t)k * nn + (size_t)cc * n + r) + 1] = v.y;
      }
  return TG_OK;
}

int tg_set_green_method(tg_ctx* c, int method) {
  if (!c) return TG_ERR_ARG;
  if (method != TG_GREEN_AUTO && method != TG_GREEN_GAUSS_JORDAN && method != TG_GREEN_SPECTRAL)
    return set_err(c, TG_ERR_ARG, "tg_set_green_method: unknown method");
  c->green_method = method;
  return TG_OK;
}

int tg_eig_batch(tg_ctx* c, int64_t nk, const double* kp, double* lam, double* U) {
  int rc = check_ready(c, false, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_eig_batch"))) return rc;
  if (nk < 0 || (nk > 0 && (!kp || !lam || !U))) return set_err(c, TG_ERR_ARG, "tg_eig_batch: bad args");
  if (nk == 0) return TG_OK;
  if (!eig_supported(c->dimH)) return set_err(c, TG_ERR_ARG, "tg_eig_batch: dimH too large for the eigensolver");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const double zero3[3] = {0.0, 0.0, 0.0};
  TG_CHECK(c, c->d_klist.upload(kp, 3 * nk, s), "upload k");
  if ((rc = build_htab(c, 0, c->d_klist.p, nk, zero3))) return rc;
  if ((rc = reset_eig_status(c))) return rc;
  if ((rc = build_eig(c, 0, nk))) return rc;
  const size_t nn = (size_t)c->dimH * c->dimH;
  TG_CHECK(c, cudaMemcpyAsync(lam, c->d_eigL[0].p, sizeof(double) * nk * c->dimH, cudaMemcpyDeviceToHost, s), "copy");
  TG_CHECK(c, cudaMemcpyAsync(U, c->d_eigU[0].p, sizeof(double2) * nk * nn, cudaMemcpyDeviceToHost, s), "copy");
  return read_eig_status(c);
}

int tg_chi0_linear_soc(tg_ctx* c, const double* q, double e, double Ef, double eta, double etap, int n_real,
                       const double* x2, const double* p2, const double* vsoc, int dimens, double* chiorb_hf,
                       double* chiorb_lsoc) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_chi0_linear_soc"))) return rc;
  if (!q || !vsoc || !chiorb_hf || !chiorb_lsoc) return set_err(c, TG_ERR_ARG, "tg_chi0_linear_soc: null argument");
  if (dimens != c->dimens) return set_err(c, TG_ERR_ARG, "tg_chi0_linear_soc: dimens mismatch");
  const bool real = std::fabs(e) >= 1e-15;
  if (real && (n_real <= 0 || !x2 || !p2)) return set_err(c, TG_ERR_ARG, "tg_chi0_linear_soc: real-axis points missing");
  if (real && !c->real_set) return set_err(c, TG_ERR_STATE, "tg_set_real_mesh has not been called");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int n = c->dimH;
  const int64_t nn = (int64_t)n * n;
  {
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
    if (gvg_smem_bytes(n) > (size_t)optin)
      return set_err(c, TG_ERR_ARG, "tg_chi0_linear_soc: dimH too large for the G V G kernel (3 dimH^2 complex in shared memory)");
  }
  const int64_t cstride = (int64_t)c->dimens * c->dimens;
  const int nsplit = nsplit_for(c);
  const ChiView fv = full_view(c);
  // eight P x dimH^2 buffers per pass: P a quarter of the chi0 pass
  int64_t P = pass_size(c, std::max<int64_t>(c->n_imag, real ? (int64_t)n_real * c->n_realk : 0)) / 4;
  P = std::max<int64_t>(64, (P / 64) * 64);
  TG_CHECK(c, c->d_A.ensure((size_t)P * nn), "alloc");
  TG_CHECK(c, c->d_B.ensure((size_t)P * nn), "alloc");
  for (int k = 0; k < 6; ++k) TG_CHECK(c, c->d_lsb[k].ensure((size_t)P * nn), "alloc");
  TG_CHECK(c, c->d_vsoc.upload(reinterpret_cast<const double2*>(vsoc), (size_t)nn, s), "upload V");
  DevArray<double2>* parts[4] = {&c->d_C, &c->d_D, &c->d_Cl, &c->d_Dl};
  for (auto* d : parts) {
    TG_CHECK(c, d->ensure((size_t)nsplit * cstride), "alloc partials");
    TG_CHECK(c, cudaMemsetAsync(d->p, 0, sizeof(double2) * nsplit * cstride, s), "memset");
  }
  TG_CHECK(c, c->d_chi.ensure((size_t)cstride), "alloc chi");
  if (real) {
    TG_CHECK(c, c->d_x2.upload(x2, n_real, s), "upload x2");
    TG_CHECK(c, c->d_p2.upload(p2, n_real, s), "upload p2");
  }
  if ((rc = reset_status(c))) return rc;
  profile_begin(c);
  double2 *X1 = c->d_lsb[0].p, *X2 = c->d_lsb[1].p, *oA = c->d_lsb[2].p, *oB = c->d_lsb[3].p, *oAx = c->d_lsb[4].p,
          *oBx = c->d_lsb[5].p;
  auto pass = [&](GreenArgs g, bool real_axis, double2* C, double2* Cl) -> int {
    // G2 = G0(k, E), G1 = G0(k + q, E + e) column-major; X = G V G of both
    g.mode = MODE_RAW;
    g.out = c->d_B.p;
    {
      KindTimer kt(c, 0);
      TG_CHECK(c, launch_green(g, c->num_sms, s, nullptr), "green (G2)");
    }
    g.zr += e;
    g.zi = eta;
    g.q[0] = q[0];
    g.q[1] = q[1];
    g.q[2] = q[2];
    g.out = c->d_A.p;
    {
      KindTimer kt(c, 0);
      TG_CHECK(c, launch_green(g, c->num_sms, s, nullptr), "green (G1)");
    }
    c->launches += 6;
    TG_CHECK(c, launch_gvg(c->d_A.p, c->d_vsoc.p, n, g.np, X1, c->num_sms, s), "G V G (1)");
    TG_CHECK(c, launch_gvg(c->d_B.p, c->d_vsoc.p, n, g.np, X2, c->num_sms, s), "G V G (2)");
    const int ma = real_axis ? MODE_A_REAL : MODE_A_IMAG, mb = real_axis ? MODE_B_REAL : MODE_B_IMAG;
    TG_CHECK(c, launch_operand(c->d_A.p, n, g.np, g.p0, g.pts, ma, c->d_outmap.p, oA, c->num_sms, s), "operand");
    TG_CHECK(c, launch_operand(c->d_B.p, n, g.np, g.p0, g.pts, mb, c->d_outmap.p, oB, c->num_sms, s), "operand");
    TG_CHECK(c, launch_operand(X1, n, g.np, g.p0, g.pts, ma, c->d_outmap.p, oAx, c->num_sms, s), "operand");
    TG_CHECK(c, launch_operand(X2, n, g.np, g.p0, g.pts, mb, c->d_outmap.p, oBx, c->num_sms, s), "operand");
    KindTimer kt(c, 1);
    if ((rc = contract(c, fv, oA, oB, g.np, C, nsplit, cstride))) return rc;
    if ((rc = contract(c, fv, oAx, oB, g.np, Cl, nsplit, cstride))) return rc;
    return contract(c, fv, oA, oBx, g.np, Cl, nsplit, cstride);
  };
  const GreenArgs base = base_args(c);
  for (int64_t p0 = 0; p0 < c->n_imag; p0 += P) {
    GreenArgs g = base;
    g.pts.kind = 0;
    g.pts.y = c->d_y.p;
    g.pts.kp = c->d_kp.p;
    g.pts.w = c->d_w.p;
    g.p0 = p0;
    g.np = std::min<int64_t>(P, c->n_imag - p0);
    g.zr = Ef;
    g.zi = etap;
    if ((rc = pass(g, false, c->d_C.p, c->d_Cl.p))) return rc;
  }
  if (real) {
    const int64_t ntot = (int64_t)n_real * c->n_realk;
    for (int64_t p0 = 0; p0 < ntot; p0 += P) {
      GreenArgs g = base;
      g.pts.kind = 1;
      g.pts.kp = c->d_rkp.p;
      g.pts.w = c->d_rw.p;
      g.pts.x2 = c->d_x2.p;
      g.pts.p2 = c->d_p2.p;
      g.pts.nk = c->n_realk;
      g.p0 = p0;
      g.np = std::min<int64_t>(P, ntot - p0);
      g.zr = 0.0;
      g.zi = etap;
      if ((rc = pass(g, true, c->d_D.p, c->d_Dl.p))) return rc;
    }
  }
  double* outs[2] = {chiorb_hf, chiorb_lsoc};
  DevArray<double2>* cs[2][2] = {{&c->d_C, &c->d_D}, {&c->d_Cl, &c->d_Dl}};
  for (int k = 0; k < 2; ++k) {
    {
      KindTimer kt(c, 2);
      TG_CHECK(c, launch_chi_epilogue(cs[k][0]->p, cs[k][1]->p, nsplit, cstride, c->dimens, c->d_decode.p, c->d_norb.p,
                                      c->d_pair_coff.p, c->n_atoms, 1.0 / (2.0 * kPi), c->d_chi.p, s),
               "epilogue");
    }
    TG_CHECK(c, copy_host(c, outs[k], c->d_chi.p, sizeof(double2) * cstride, false), "copy");
  }
  profile_end(c);
  return read_status(c);
}

int tg_jij(tg_ctx* c, const double* q, double Ef, double eta, const double* evec, const double* Um, const int* dmask,
           double* J) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_jij"))) return rc;
  if (!q || !evec || !Um || !dmask || !J) return set_err(c, TG_ERR_ARG, "tg_jij: null argument");
  cudaSetDevice(c->device);
  const int nat = c->n_atoms, nmax = c->nmax;
  // pairs of d orbitals of every two sites
  std::vector<int4> pairs;
  std::vector<int> site;
  for (int i = 0; i < nat; ++i)
    for (int j = 0; j < nat; ++j)
      for (int be = 0; be < c->norb[j]; ++be)
        for (int al = 0; al < c->norb[i]; ++al) {
          if (!dmask[(size_t)i * nmax + al] || !dmask[(size_t)j * nmax + be]) continue;
          pairs.push_back(make_int4(c->ia[i] + al, c->ia[i] + c->norb[i] + al, c->ia[j] + be,
                                    c->ia[j] + c->norb[j] + be));
          site.push_back(i * nat + j);
        }
  std::vector<double2> hp, hq, h((size_t)nat * nat * 32, make_double2(0.0, 0.0));
  if ((rc = imag_pairs(c, Ef, eta, q, pairs, hp, &hq))) return rc;
  for (size_t b = 0; b < site.size(); ++b)
    for (int x = 0; x < 16; ++x) {
      double2* t = h.data() + (size_t)site[b] * 32;
      t[x] = cadd(t[x], hp[16 * b + x]);
      t[16 + x] = cadd(t[16 + x], hq[16 * b + x]);
    }
  // sigma_a[s][s'] (0 = up), a = x, y, z
  const double2 sig[3][2][2] = {{{{0, 0}, {1, 0}}, {{1, 0}, {0, 0}}},
                                {{{0, 0}, {0, -1}}, {{0, 1}, {0, 0}}},
                                {{{1, 0}, {0, 0}}, {{0, 0}, {-1, 0}}}};
  // V(T16, a, b) = sum sigma_a[s][s'] sigma_b[t][t'] T[s' + 2t + 4t' + 8s]
  auto vertex = [&](const double2* T16, int a, int b) {
    double2 v = make_double2(0.0, 0.0);
    for (int ss = 0; ss < 2; ++ss)
      for (int sp = 0; sp < 2; ++sp)
        for (int t = 0; t < 2; ++t)
          for (int tp = 0; tp < 2; ++tp)
            v = cadd(v, cmul(cmul(sig[a][ss][sp], sig[b][t][tp]), T16[sp + 2 * t + 4 * tp + 8 * ss]));
    return v;
  };
  const double f = -1.0 / (2.0 * kPi);
  for (int i = 0; i < nat; ++i)
    for (int j = 0; j < nat; ++j) {
      const double2* T = h.data() + (size_t)(i * nat + j) * 32;
      double2 V[3][3], Vs[3][3];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          V[a][b] = vertex(T, a, b);
          Vs[a][b] = cconj(vertex(T + 16, a, b));
        }
      for (int mu = 0; mu < 3; ++mu)
        for (int nu = 0; nu < 3; ++nu) {
          double2 acc = make_double2(0.0, 0.0);
          for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) {
              // c^i_{mu a} = -Um_i / 2 (delta_{mu a} - e_{i mu} e_{i a})
              const double ci = -0.5 * Um[i] * ((mu == a ? 1.0 : 0.0) - evec[3 * i + mu] * evec[3 * i + a]);
              const double cj = -0.5 * Um[j] * ((nu == b ? 1.0 : 0.0) - evec[3 * j + nu] * evec[3 * j + b]);
              acc = cadd(acc, cscale(cadd(V[a][b], Vs[a][b]), ci * cj));
            }
          const size_t o = (size_t)i + (size_t)nat * (j + (size_t)nat * (mu + 3 * (size_t)nu));
          J[2 * o] = f * acc.x;
          J[2 * o + 1] = f * acc.y;
        }
    }
  return TG_OK;
}

int tg_smunu(tg_ctx* c, double Ef, double eta, double* S) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_smunu"))) return rc;
  if (!S) return set_err(c, TG_ERR_ARG, "tg_smunu: null output");
  cudaSetDevice(c->device);
  const int nat = c->n_atoms, nmax = c->nmax;
  // entries (r, c) of every on-site block, site by site, row-major inside the 2n x 2n block
  std::vector<int> desc, site_off(nat + 1, 0);
  for (int i = 0; i < nat; ++i) {
    const int n2 = 2 * c->norb[i];
    for (int x = 0; x < n2; ++x)
      for (int y = 0; y < n2; ++y) {
        desc.push_back(c->ia[i] + x);
        desc.push_back(c->ia[i] + y);
      }
    site_off[i + 1] = site_off[i] + n2 * n2;
  }
  std::vector<int2> ent;
  for (size_t e = 0; e + 1 < desc.size(); e += 2) ent.push_back(make_int2(desc[e], desc[e + 1]));
  std::vector<double2> h;
  auto points = [&](GreenArgs& a) { return imag_points(c, Ef, eta, nullptr, a, nullptr); };
  if ((rc = entry_sums(c, c->n_imag, ent, h, "green (on-site blocks)", points))) return rc;
  // calcSmunu: imgXY(mu, nu) = (A(nu X, mu Y) + conj(A(mu Y, nu X))) / 2 pi, 1/2 on the uu / dd diagonals
  const double tpi = 2.0 * kPi;
  std::fill(S, S + (size_t)2 * nmax * nmax * 3 * nat, 0.0);
  for (int i = 0; i < nat; ++i) {
    const int n = c->norb[i], n2 = 2 * n;
    auto A = [&](int x, int y) { return h[site_off[i] + x * n2 + y]; };
    auto img = [&](int sx, int sy, int mu, int nu) {   // spins sx (row of nu), sy (column of mu)
      const double2 p = A(sx * n + nu, sy * n + mu), q = A(sy * n + mu, sx * n + nu);
      return make_double2((p.x + q.x) / tpi, (p.y - q.y) / tpi);
    };
    for (int mu = 0; mu < n; ++mu)
      for (int nu = 0; nu < n; ++nu) {
        double2 uu = img(0, 0, mu, nu), dd = img(1, 1, mu, nu);
        const double2 ud = img(0, 1, mu, nu), du = img(1, 0, mu, nu);
        if (mu == nu) {
          uu.x += 0.5;
          dd.x += 0.5;
        }
        const double2 k1 = cadd(ud, du), k2 = cmul(make_double2(0.0, 1.0), csub(ud, du)), k3 = csub(uu, dd);
        const double2 ks[3] = {k1, k2, k3};
        for (int k = 0; k < 3; ++k) {
          const size_t o = (size_t)mu + (size_t)nmax * (nu + (size_t)nmax * (k + 3 * (size_t)i));
          S[2 * o] = ks[k].x;
          S[2 * o + 1] = ks[k].y;
        }
      }
  }
  return TG_OK;
}

int tg_gs_orbital(tg_ctx* c, double Ef, double eta, double* gupgd) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_gs_orbital"))) return rc;
  if (!gupgd) return set_err(c, TG_ERR_ARG, "tg_gs_orbital: null output");
  cudaSetDevice(c->device);
  const int nat = c->n_atoms, nmax = c->nmax;
  // entries (i mu s, i nu s) of the two spin-diagonal blocks of every site: s = up, then down
  std::vector<int> desc, site_off(nat + 1, 0);
  for (int i = 0; i < nat; ++i) {
    const int n = c->norb[i];
    for (int sp = 0; sp < 2; ++sp)
      for (int mu = 0; mu < n; ++mu)
        for (int nu = 0; nu < n; ++nu) {
          desc.push_back(c->ia[i] + sp * n + mu);
          desc.push_back(c->ia[i] + sp * n + nu);
        }
    site_off[i + 1] = site_off[i] + 2 * n * n;
  }
  std::vector<int2> ent;
  for (size_t e = 0; e + 1 < desc.size(); e += 2) ent.push_back(make_int2(desc[e], desc[e + 1]));
  std::vector<double2> h;
  auto points = [&](GreenArgs& a) { return imag_points(c, Ef, eta, nullptr, a, nullptr); };
  if ((rc = entry_sums(c, c->n_imag, ent, h, "green (on-site spin blocks)", points))) return rc;
  // gupgd(nu, mu, i) = (1/pi) sum w (G(i mu up, i nu up) + G(i mu dn, i nu dn))  (mod_expectation.F90:957-975)
  std::fill(gupgd, gupgd + (size_t)2 * nmax * nmax * nat, 0.0);
  for (int i = 0; i < nat; ++i) {
    const int n = c->norb[i];
    for (int mu = 0; mu < n; ++mu)
      for (int nu = 0; nu < n; ++nu) {
        const double2 up = h[site_off[i] + mu * n + nu], dn = h[site_off[i] + n * n + mu * n + nu];
        const size_t o = (size_t)nu + (size_t)nmax * (mu + (size_t)nmax * i);
        gupgd[2 * o] = (up.x + dn.x) / kPi;
        gupgd[2 * o + 1] = (up.y + dn.y) / kPi;
      }
  }
  return TG_OK;
}

int tg_ldos(tg_ctx* c, int n_e, const double* e, double eta, double* ldosu, double* ldosd) {
  int rc = check_ready(c, false, true);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_ldos"))) return rc;
  if (n_e < 0 || (n_e > 0 && (!e || !ldosu || !ldosd))) return set_err(c, TG_ERR_ARG, "tg_ldos: bad args");
  if (n_e == 0) return TG_OK;
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int n = c->dimH, nat = c->n_atoms, nmax = c->nmax;
  auto put = [&](int ie, int i, int mu, double up, double dn) {
    const size_t o = ((size_t)ie * nat + i) * nmax + mu;
    ldosu[o] = up;
    ldosd[o] = dn;
  };
  std::fill(ldosu, ldosu + (size_t)n_e * nat * nmax, 0.0);
  std::fill(ldosd, ldosd + (size_t)n_e * nat * nmax, 0.0);
  if (!spectral_on(c)) {
    // Gauss-Jordan per (k, e): the sigma_0 / sigma_z traces of G_ii of the Fermi-column kernel
    std::vector<double> D((size_t)2 * 4 * nmax * nat);
    const double pi = kPi;
    for (int ie = 0; ie < n_e; ++ie) {
      if ((rc = tg_fermi_column(c, e[ie], eta, D.data()))) return rc;
      for (int i = 0; i < nat; ++i)
        for (int mu = 0; mu < c->norb[i]; ++mu) {
          const double* d = D.data() + 2 * 4 * ((size_t)i * nmax + mu);
          put(ie, i, mu, -(d[1] + d[7]) / (2.0 * pi), -(d[1] - d[7]) / (2.0 * pi));
        }
    }
    return TG_OK;
  }
  // spectral: one eigendecomposition per k of the real-axis BZ, every energy from it
  const double zero3[3] = {0.0, 0.0, 0.0};
  if ((rc = reset_eig_status(c))) return rc;
  if ((rc = build_htab(c, 2, c->d_rkp.p, c->n_realk, zero3))) return rc;
  if ((rc = build_eig(c, 2, c->n_realk))) return rc;
  TG_CHECK(c, c->d_ldos_e.upload(e, n_e, s), "upload energies");
  TG_CHECK(c, c->d_ldos.ensure((size_t)n_e * n), "alloc ldos");
  c->launches += 1;
  TG_CHECK(c, launch_spec_ldos(c->d_eigU[2].p, c->d_eigL[2].p, c->d_rw.p, c->n_realk, n, c->d_ldos_e.p, n_e, eta,
                               c->d_ldos.p, c->num_sms, s),
           "ldos");
  std::vector<double> h((size_t)n_e * n);
  TG_CHECK(c, cudaMemcpyAsync(h.data(), c->d_ldos.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s), "copy");
  if ((rc = read_eig_status(c))) return rc;   // synchronises the stream
  for (int ie = 0; ie < n_e; ++ie)
    for (int i = 0; i < nat; ++i)
      for (int mu = 0; mu < c->norb[i]; ++mu)
        put(ie, i, mu, h[(size_t)ie * n + c->ia[i] + mu], h[(size_t)ie * n + c->ia[i] + c->norb[i] + mu]);
  return TG_OK;
}

int tg_dyson(tg_ctx* c, int dimens, const double* chi_hf, const double* umat, double* chi) {
  return tg_dyson_order(c, dimens, chi_hf, 0, umat, 0, chi);
}

int tg_dyson_order(tg_ctx* c, int dimens, const double* chi_hf, int chi_rows, const double* umat, int umat_rows,
                   double* chi) {
  if (!c) return TG_ERR_ARG;
  if (dimens <= 0 || !chi_hf || !umat || !chi) return set_err(c, TG_ERR_ARG, "tg_dyson: bad args");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const size_t nn = (size_t)dimens * dimens;
  TG_CHECK(c, c->d_dy.ensure(4 * nn), "alloc dyson");
  TG_CHECK(c, c->d_piv.ensure(dimens), "alloc piv");
  double2* X = c->d_dy.p;
  double2* U = X + nn;
  double2* W = U + nn;
  double2* R = W + nn;
  int rc = reset_status(c);
  if (rc) return rc;
  // a row-major matrix arrives in a free buffer and is transposed into its place
  TG_CHECK(c, copy_host(c, chi_rows ? W : X, chi_hf, sizeof(double2) * nn, true), "upload");
  if (chi_rows) TG_CHECK(c, launch_transpose(dimens, W, X, s), "transpose");
  TG_CHECK(c, copy_host(c, umat_rows ? R : U, umat, sizeof(double2) * nn, true), "upload");
  if (umat_rows) TG_CHECK(c, launch_transpose(dimens, R, U, s), "transpose");
  TG_CHECK(c, dyson_device(dimens, X, U, W, R, c->d_piv.p, c->d_status.p, s), "dyson");
  TG_CHECK(c, copy_host(c, chi, R, sizeof(double2) * nn, false), "copy");
  return read_status(c);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// tg_she: disturbance response to an electric field (eintshe.F90:2-309)
// ---------------------------------------------------------------------------
namespace {

// (sigma, sigma') -> spin blocks (X, Y, Z, W) of the imaginary-axis integrand
//   G1^X V G2^Y + conj(G2^Z) V^T conj(G1^W)          (eintshe.F90:104-179)
// 'u' = up, 'd' = down; the first letter is the row spin.  sigma-major order.
const char* const kSheImag[16][4] = {
    {"dd", "uu", "uu", "dd"}, {"du", "uu", "uu", "ud"}, {"dd", "du", "ud", "dd"}, {"du", "du", "ud", "ud"},
    {"ud", "uu", "uu", "du"}, {"uu", "uu", "uu", "uu"}, {"ud", "du", "ud", "du"}, {"uu", "du", "ud", "uu"},
    {"dd", "ud", "du", "dd"}, {"du", "ud", "du", "ud"}, {"dd", "dd", "dd", "dd"}, {"du", "dd", "dd", "ud"},
    {"ud", "ud", "du", "du"}, {"uu", "ud", "du", "uu"}, {"ud", "dd", "dd", "du"}, {"uu", "dd", "dd", "uu"}};
// (sigma, sigma') -> (X, X', Y) of the real-axis integrand
//   -i (G1^X - (G1^{X'})^+) V (G2^Y)^+               (eintshe.F90:226-249)
// X' is always X with its two spins exchanged, so the first factor is the
// X block of G1 - G1^+.
const char* const kSheReal[16][3] = {
    {"dd", "dd", "uu"}, {"du", "ud", "uu"}, {"dd", "dd", "ud"}, {"du", "ud", "ud"},
    {"ud", "du", "uu"}, {"uu", "uu", "uu"}, {"ud", "du", "ud"}, {"uu", "uu", "ud"},
    {"dd", "dd", "du"}, {"du", "ud", "du"}, {"dd", "dd", "dd"}, {"du", "ud", "dd"},
    {"ud", "du", "du"}, {"uu", "uu", "du"}, {"ud", "du", "dd"}, {"uu", "uu", "dd"}};

int spin_bit(char x) { return x == 'd' ? 1 : 0; }
unsigned char spin_code(char a, char b, char c, char d) {
  return (unsigned char)(spin_bit(a) << 3 | spin_bit(b) << 2 | spin_bit(c) << 1 | spin_bit(d));
}

// kernel spin codes (outer row spin, inner spin of L, inner spin of R, outer column spin)
void she_spin_codes(unsigned char spins[3][16]) {
  for (int t = 0; t < 16; ++t) {
    const char *X = kSheImag[t][0], *Y = kSheImag[t][1], *Z = kSheImag[t][2], *W = kSheImag[t][3];
    spins[0][t] = spin_code(X[0], X[1], Y[0], Y[1]);
    spins[1][t] = spin_code(Z[0], Z[1], W[0], W[1]);
    const char *XR = kSheReal[t][0], *YR = kSheReal[t][2];
    spins[2][t] = spin_code(XR[0], XR[1], YR[1], YR[0]);
  }
}

}  // namespace

extern "C" int tg_she(tg_ctx* c, const double* q, double e, double Ef, double eta, double etap, int n_real,
                      const double* x2, const double* p2, const double* efield, const double* prefactor, int dimens,
                      double* tchi) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if ((rc = require_native(c, "tg_she"))) return rc;
  if (!q || !efield || !tchi) return set_err(c, TG_ERR_ARG, "tg_she: null argument");
  if (dimens != c->dimens) return set_err(c, TG_ERR_ARG, "tg_she: dimens mismatch");
  const bool real = std::fabs(e) >= 1e-15;
  if (real && (n_real <= 0 || !x2 || !p2)) return set_err(c, TG_ERR_ARG, "tg_she: real-axis points missing");
  if (real && !c->real_set) return set_err(c, TG_ERR_STATE, "tg_set_real_mesh has not been called");
  cudaSetDevice(c->device);
  cudaStream_t s = c->stream;
  const int n = c->dimH, no = n / 2, D = c->dimens;
  const int64_t nn = (int64_t)n * n;
  int n_frags = 0;
  for (int i = 0; i < c->n_atoms; ++i) n_frags += ((c->norb[i] + 1) / 2) * ((c->norb[i] + 1) / 2);
  const int grid = she_grid(n, D, c->n_neigh, n_frags, c->num_sms);
  if (grid <= 0) return set_err(c, TG_ERR_ARG, "tg_she: dimH / dimens too large for the shared-memory vertex kernel");
  // orbital tables of the kernel
  std::vector<int> tab((size_t)4 * no);
  {
    int o = 0;
    for (int i = 0; i < c->n_atoms; ++i)
      for (int m = 0; m < c->norb[i]; ++m, ++o) {
        tab[o] = c->ia[i] + m;
        tab[no + o] = c->ia[i] + c->norb[i] + m;
        tab[2 * no + o] = i;
        tab[3 * no + o] = m;
      }
  }
  TG_CHECK(c, c->d_she_tab.upload(tab.data(), tab.size(), s), "upload tables");
  TG_CHECK(c, c->d_ia.upload(c->ia.data(), c->ia.size(), s), "upload ia");
  // vertex second stage: 3 x 3 tiles of every (sigma, s', site) block of n_i x n_i df
  // entries, and the first df row of each site (rows in sigmaimunu2i order: sigma fastest,
  // then nu, mu, site)
  const int nat = c->n_atoms;
  std::vector<int> ztiles, rowoff(nat);
  for (int i = 0, off = 0; i < nat; ++i) {
    rowoff[i] = off;
    off += 4 * c->norb[i] * c->norb[i];
  }
  for (int sg = 0; sg < 4; ++sg)
    for (int sp = 0; sp < 4; ++sp)
      for (int i = 0; i < nat; ++i)
        for (int x0 = 0; x0 < c->norb[i]; x0 += 3)
          for (int y0 = 0; y0 < c->norb[i]; y0 += 3) ztiles.push_back(sg | sp << 2 | i << 4 | x0 << 14 | y0 << 20);
  TG_CHECK(c, c->d_she_ztiles.upload(ztiles.data(), ztiles.size(), s), "upload tiles");
  TG_CHECK(c, c->d_she_rowoff.upload(rowoff.data(), rowoff.size(), s), "upload");
  const int n_ztiles = (int)ztiles.size();
  TG_CHECK(c, c->d_she_part.ensure((size_t)grid * 4 * D), "alloc partials");
  TG_CHECK(c, c->d_she_sum.ensure((size_t)4 * D), "alloc");
  TG_CHECK(c, c->d_she_out.ensure((size_t)4 * D), "alloc");
  TG_CHECK(c, cudaMemsetAsync(c->d_she_part.p, 0, sizeof(double2) * grid * 4 * D, s), "memset");
  if (prefactor) TG_CHECK(c, c->d_she_pref.upload(reinterpret_cast<const double2*>(prefactor), (size_t)D * D, s), "upload");
  const int64_t P = pass_size(c, std::max<int64_t>(c->n_imag, real ? (int64_t)n_real * c->n_realk : 0));
  TG_CHECK(c, c->d_A.ensure((size_t)P * nn), "alloc G1");
  TG_CHECK(c, c->d_B.ensure((size_t)P * nn), "alloc G2");
  if (real) {
    TG_CHECK(c, c->d_x2.upload(x2, n_real, s), "upload x2");
    TG_CHECK(c, c->d_p2.upload(p2, n_real, s), "upload p2");
  }
  rc = reset_status(c);
  if (rc) return rc;
  profile_begin(c);
  TG_CHECK(c, cudaEventRecord(c->ev[0], s), "event");
  // H(k) tables (k-major traversal) and, for spectral Green functions, their eigendecompositions
  const bool q_zero = q[0] == 0.0 && q[1] == 0.0 && q[2] == 0.0;
  const double zero3[3] = {0.0, 0.0, 0.0};
  const bool tab_imag = c->imag_uniform && (int64_t)c->nk_u * nn * 16 <= ((int64_t)8 << 30);
  const bool tab_real = real && (int64_t)c->n_realk * nn * 16 <= ((int64_t)8 << 30);
  const bool spec = spectral_forced(c);
  // AUTO at n = 36 on a tabulated imaginary axis: spectral G for the energies with
  // Im z >= 10 eta (its eps |H| / Im z error is negligible there; the nanoribbon goldens
  // hold with the split at 10 eta), the blocked Gauss-Jordan kernel below and on the real axis.
  // Measured against Gauss-Jordan alone (ms, 64 and 20 imaginary energies, 8 real ones): 36, 61 x 61 k:
  // 34.3 / 37.8 and 15.8 / 14.5, 13 x 13 k: 3.0 / 2.0 and 2.2 / 0.9; the split on at the other
  // dimensions: 18, 14^3 k: 8.2 / 8.6 and 3.9 / 3.4; 54, 30 x 30 k: 32.2 / 36.4 and 16.5 / 13.8; 72,
  // 8^3 k: 59.7 / 64.9 and 29.1 / 24.2.  It pays by the energies per k and the number of k rather
  // than by the dimension; it is kept to the dimension it was brought in for.
  const bool hybrid = !spec && c->green_method == TG_GREEN_AUTO && tab_imag && eig_supported(n) &&
                      n == 36 && green_mma_supported(n, MODE_RAW);
  const double y_split = 10.0 * eta;
  if ((spec || hybrid) && (tab_imag || tab_real) && (rc = reset_eig_status(c))) return rc;
  auto tables = [&](int slot, const double* d_k, int64_t nk, bool shift) -> int {
    if ((rc = build_htab(c, slot, d_k, nk, shift ? q : zero3))) return rc;
    if ((spec || (hybrid && slot < 2)) && (rc = build_eig(c, slot, nk))) return rc;
    return TG_OK;
  };
  if (tab_imag) {
    if ((rc = tables(0, c->d_klist_u.p, c->nk_u, false))) return rc;
    if (!q_zero && (rc = tables(1, c->d_klist_u.p, c->nk_u, true))) return rc;
  }
  const bool alias_real = tab_imag && tab_real && real_k_is_imag_k(c);
  const int rslot0 = alias_real ? 0 : 2, rslot1 = alias_real ? 1 : 3;
  if (tab_real && !alias_real) {
    if ((rc = tables(2, c->d_rkp.p, c->n_realk, false))) return rc;
    if (!q_zero && (rc = tables(3, c->d_rkp.p, c->n_realk, true))) return rc;
  }
  auto use_table = [&](GreenArgs& g, int slot, int64_t n_e, int64_t nk, const double* ylist) {
    g.htab = c->d_htab[slot].p;
    g.n_e = n_e;
    g.nk_tab = nk;
    g.ylist = ylist;
    g.q[0] = g.q[1] = g.q[2] = 0.0;   // q is inside the table
    if (spec) {
      g.eigU = c->d_eigU[slot].p;
      g.eigL = c->d_eigL[slot].p;
      g.outinv = c->d_outinv.p;
    } else {
      g.eigU = nullptr;
      g.eigL = nullptr;
    }
  };
  GreenArgs base = base_args(c);
  SheLaunch l;
  l.g = &base;
  l.dimens = D;
  l.tab = c->d_she_tab.p;
  l.ia = c->d_ia.p;
  l.norb = c->d_norb.p;
  l.ztiles = c->d_she_ztiles.p;
  l.n_ztiles = n_ztiles;
  l.n_frags = n_frags;
  l.rowoff = c->d_she_rowoff.p;
  for (int i = 0; i < 3; ++i) l.ue[i] = efield[i];
  she_spin_codes(l.spins);
  l.partial = c->d_she_part.p;
  l.grid = grid;
  // one pass: G2 = G(k, E), G1 = G(k + q, E + e), both column-major per point, then the
  // vertex; slot2 / slot1 >= 0: H(k) tables of G2 / G1 with n_e energies per k (k-major order)
  // one G launch, or for the hybrid the spectral part (eigendecomposition of the slot) and
  // the Gauss-Jordan part of the same points
  auto green = [&](GreenArgs g, int slot, bool split, const char* what) -> int {
    if (!split) {
      KindTimer kt(c, 0);
      TG_CHECK(c, launch_green(g, c->num_sms, s, nullptr), what);
      return TG_OK;
    }
    GreenArgs gs = g;
    gs.eigU = c->d_eigU[slot].p;
    gs.eigL = c->d_eigL[slot].p;
    gs.outinv = c->d_outinv.p;
    gs.y_split = y_split;
    gs.y_side = 1;
    GreenArgs gj = g;
    gj.eigU = nullptr;
    gj.eigL = nullptr;
    gj.y_split = y_split;
    gj.y_side = -1;
    KindTimer kt(c, 0);
    TG_CHECK(c, launch_green(gs, c->num_sms, s, nullptr), what);
    TG_CHECK(c, launch_green(gj, c->num_sms, s, nullptr), what);
    c->launches += 1;
    return TG_OK;
  };
  auto pass = [&](GreenArgs g, int real_axis, int slot2, int slot1, int64_t n_e, int64_t nk,
                  const double* ylist, const double* klist) -> int {
    const bool split = hybrid && !real_axis && slot2 >= 0;
    g.mode = MODE_RAW;
    g.out = c->d_B.p;
    if (slot2 >= 0) use_table(g, slot2, n_e, nk, ylist);
    if ((rc = green(g, slot2, split, "green (G2)"))) return rc;
    g.zr += e;
    g.zi = eta;
    g.q[0] = q[0];
    g.q[1] = q[1];
    g.q[2] = q[2];
    g.out = c->d_A.p;
    if (slot1 >= 0) use_table(g, slot1, n_e, nk, ylist);
    if ((rc = green(g, slot1, split, "green (G1)"))) return rc;
    l.n_e = slot2 >= 0 ? n_e : 0;
    l.nk_tab = nk;
    l.klist = klist;
    l.G1 = c->d_A.p;
    l.G2 = c->d_B.p;
    l.p0 = g.p0;
    l.np = g.np;
    l.pts = g.pts;
    l.real_axis = real_axis;
    {
      KindTimer kt(c, 1);
      c->launches += 1;
      TG_CHECK(c, launch_she(l, s), "disturbance vertex");
    }
    return TG_OK;
  };
  for (int64_t p0 = 0; p0 < c->n_imag; p0 += P) {
    GreenArgs g = base;
    g.pts.kind = 0;
    g.pts.y = c->d_y.p;
    g.pts.kp = c->d_kp.p;
    g.pts.w = c->d_w.p;
    g.p0 = p0;
    g.np = std::min<int64_t>(P, c->n_imag - p0);
    g.zr = Ef;
    g.zi = etap;
    if (tab_imag) rc = pass(g, 0, 0, q_zero ? 0 : 1, c->n_e_u, c->nk_u, c->d_ylist.p, c->d_klist_u.p);
    else rc = pass(g, 0, -1, -1, 0, 0, nullptr, nullptr);
    if (rc) return rc;
  }
  if (real) {
    const int64_t ntot = (int64_t)n_real * c->n_realk;
    for (int64_t p0 = 0; p0 < ntot; p0 += P) {
      GreenArgs g = base;
      g.pts.kind = 1;
      g.pts.kp = c->d_rkp.p;
      g.pts.w = c->d_rw.p;
      g.pts.x2 = c->d_x2.p;
      g.pts.p2 = c->d_p2.p;
      g.pts.nk = c->n_realk;
      g.p0 = p0;
      g.np = std::min<int64_t>(P, ntot - p0);
      g.zr = 0.0;
      g.zi = etap;
      if (tab_real) rc = pass(g, 1, rslot0, q_zero ? rslot0 : rslot1, n_real, c->n_realk, nullptr, c->d_rkp.p);
      else rc = pass(g, 1, -1, -1, 0, 0, nullptr, nullptr);
      if (rc) return rc;
    }
  }
  {
    KindTimer kt(c, 2);
    TG_CHECK(c, launch_reduce_blocks(c->d_she_part.p, grid, 4 * D, c->d_she_sum.p, s), "reduce");
  }
  {
    KindTimer kt(c, 2);
    TG_CHECK(c, launch_she_prefactor(prefactor ? c->d_she_pref.p : nullptr, c->d_she_sum.p, D, 1.0 / (2.0 * kPi),
                                     c->d_she_out.p, s),
             "prefactor");
  }
  TG_CHECK(c, cudaMemcpyAsync(tchi, c->d_she_out.p, sizeof(double2) * 4 * D, cudaMemcpyDeviceToHost, s), "copy");
  TG_CHECK(c, cudaEventRecord(c->ev[6], s), "event");
  TG_CHECK(c, cudaEventSynchronize(c->ev[6]), "sync");
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev[0], c->ev[6]);
  c->last_ms[3] = ms;
  profile_end(c);
  rc = read_status(c);
  if (rc) return rc;
  if ((spec || hybrid) && (tab_imag || tab_real)) return read_eig_status(c);
  return TG_OK;
}

// ---------------------------------------------------------------------------
// tg_expectation_noalloc: occupations and moments without device allocation.
//
// For callers that cannot let a library call allocate device memory: a host
// that hands the GPU's memory to its own pool or to another solver up front and
// budgets every byte of HBM itself, so that a cudaMalloc inside a library call
// would fail or break that budget.  tg_expectation allocates its
// partial sums (and an H(k) table) on first use; this variant keeps the partial
// sums in a fixed 8 MiB device array compiled into the library and sums H(k)
// inside the inversion kernel instead of tabulating it.
//
// * Size limit: (16 x SMs + 1) x 2 dimH complex doubles (25 x SMs up to dimH 18) must fit in 8 MiB
//   (dimH <= 90 on a 148-SM B200 needs 6.8 MB); larger requests, and dimensions
//   that only the general-dimension kernel handles, return TG_ERR_ARG before
//   any work.
// * Method: always Gauss-Jordan per (k, z) point, whatever tg_set_green_method
//   chose (the default choice of tg_expectation; its TG_GREEN_SPECTRAL form would
//   need eigenvector tables in allocated memory).
// * Setup: the first call on a context looks up the array's device address on
//   the context's device (cudaGetSymbolAddress with that device current, which
//   also loads this module there if it is not loaded yet) and keeps it in the
//   context; make that first call before any stream capture.  After a
//   cudaDeviceReset the context's stream and buffers are gone as well: destroy
//   the context and create a new one, which looks the address up again.
// * Nothing in the scratch has to start at zero: every partial slot the
//   reduction reads is written by the kernel of the same call.
// * One array serves every context and stream of a device: calls that overlap
//   in time on the same device race on it.  A call returns only after its
//   results are on the host, so calls made one after another are safe.
// ---------------------------------------------------------------------------
namespace {
constexpr size_t kNoAllocScratchBytes = (size_t)8 << 20;
constexpr int kNoAllocMaxLen = 512;   // 2 dimH complex sums per partial slot
}  // namespace

static __device__ __align__(256) double2 g_noalloc_scratch[kNoAllocScratchBytes / sizeof(double2)];

namespace {
// device address of the scratch on the context's device (looked up on the context's
// first call, with that device current)
int noalloc_scratch(tg_ctx* c, double2** out) {
  if (!c->noalloc_ptr) {
    void* q = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&q, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_err(c, e, "tg_expectation_noalloc: scratch address");
    c->noalloc_ptr = static_cast<double2*>(q);
  }
  *out = c->noalloc_ptr;
  return TG_OK;
}
}  // namespace

extern "C" int tg_expectation_noalloc(tg_ctx* c, double Ef, double eta, double* rho, double* mx, double* my,
                                      double* mz, double* mp) {
  int rc = check_ready(c, true, false);
  if (rc) return rc;
  if (!rho || !mx || !my || !mz || !mp) return set_err(c, TG_ERR_ARG, "tg_expectation_noalloc: null output");
  const int n = c->dimH;
  const int len = 2 * n;
  // partial slots: the one-warp kernel runs at most 15 matrices per SM, the blocked one green_max_ctas
  const size_t slots = (size_t)c->num_sms * (green_max_ctas(n) + 1);
  const size_t need = (slots + 1) * (size_t)len * sizeof(double2);
  if (!green_supported(n))
    return set_err(c, TG_ERR_ARG, "tg_expectation_noalloc: this dimension needs the general-dimension kernel, "
                                  "which keeps its Green functions in allocated memory");
  if (len > kNoAllocMaxLen || need > kNoAllocScratchBytes) {
    char b[160];
    snprintf(b, sizeof b, "tg_expectation_noalloc: needs %zu bytes of scratch, the fixed scratch holds %zu",
             need, kNoAllocScratchBytes);
    return set_err(c, TG_ERR_ARG, b);
  }
  cudaSetDevice(c->device);
  double2* scratch = nullptr;
  if ((rc = noalloc_scratch(c, &scratch))) return rc;
  double2* partial = scratch;
  double2* reduced = scratch + slots * len;
  cudaStream_t s = c->stream;
  GreenArgs a = base_args(c);
  a.pts.kind = 0;
  a.pts.y = c->d_y.p;
  a.pts.kp = c->d_kp.p;
  a.pts.w = c->d_w.p;
  a.p0 = 0;
  a.np = c->n_imag;
  a.zr = Ef;
  a.zi = eta;
  a.mode = MODE_EXPECT;
  a.exp_rows = c->d_exp_rows.p;
  a.acc = partial;
  rc = reset_status(c);
  if (rc) return rc;
  int grid = 0;
  TG_CHECK(c, launch_green(a, c->num_sms, s, &grid), "green (expectation, no-alloc)");
  TG_CHECK(c, launch_reduce_blocks(partial, grid, len, reduced, s), "reduce");
  double2 h[kNoAllocMaxLen];
  TG_CHECK(c, cudaMemcpyAsync(h, reduced, sizeof(double2) * len, cudaMemcpyDeviceToHost, s), "copy");
  rc = read_status(c);
  if (rc) return rc;
  // mod_expectation.F90:121-147
  int o = 0;
  for (int i = 0; i < c->n_atoms; ++i) {
    for (int mu = 0; mu < c->nmax; ++mu) {
      const size_t idx = (size_t)i * c->nmax + mu;
      if (mu >= c->norb[i]) {
        rho[idx] = mx[idx] = my[idx] = mz[idx] = 0.0;
        mp[2 * idx] = mp[2 * idx + 1] = 0.0;
        continue;
      }
      const double2 uu = h[4 * o], dd = h[4 * o + 1], ud = h[4 * o + 2], du = h[4 * o + 3];
      const double nu_ = 0.5 + uu.x / kPi, nd_ = 0.5 + dd.x / kPi;
      rho[idx] = nu_ + nd_;
      mz[idx] = nu_ - nd_;
      const double mpr = (du.x + ud.x) / kPi, mpi = (du.y - ud.y) / kPi;
      mx[idx] = mpr;
      my[idx] = mpi;
      mp[2 * idx] = mpr;
      mp[2 * idx + 1] = mpi;
      ++o;
    }
  }
  return TG_OK;
}
