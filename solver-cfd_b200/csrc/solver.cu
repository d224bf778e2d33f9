// solver.cu -- host orchestration and the C ABI (include/acs.h).
//
// A batch owns one device allocation holding, per case, the metric arrays, the porous fields and
// the rotating field buffers (see acs_dev.cuh), plus the case table, the control words and a
// tile table covering every case.  One pseudo-iteration is a fixed sequence of launches over the
// tile table (U stages, V stages, P, T stages, C stages, control).  acs_batch_run captures that
// sequence once as the body of a CUDA graph WHILE node whose condition kernel keeps looping
// while any case is active, so a whole multi-step run is one graph launch with no host round
// trip.  A single case (acs_handle) is a batch of one.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/acs.h"
#include "acs_dev.cuh"
#include "fast.h"
#include "chip_plan.h"
#include "engine_api.h"
#include "kernels.h"
#include "tile_engine.h"
#include "transfer.h"
#include "warmstart.h"

namespace acs {

thread_local std::string g_err;

int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

#define CU(call)                                                                                 \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess) return fail(ACS_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

namespace {

constexpr int kMinN = 6;
constexpr int kMaxN = 1 << 15;

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct FieldLoc { int family; int role; };  // family: 0 U, 1 V, 2 P, 3 T, 4 C
FieldLoc field_loc(int f) {
  switch (f) {
    case ACS_UM: return {0, R_PHYS};
    case ACS_UM_TAU: return {0, R_TAU};
    case ACS_UM_N_TAU: return {0, R_NTAU};
    case ACS_VM: return {1, R_PHYS};
    case ACS_VM_TAU: return {1, R_TAU};
    case ACS_VM_N_TAU: return {1, R_NTAU};
    case ACS_P: return {2, 0};
    case ACS_PN: return {2, 1};
    case ACS_T: return {3, R_PHYS};
    case ACS_T_TAU: return {3, R_TAU};
    case ACS_T_N_TAU: return {3, R_NTAU};
    case ACS_C: return {4, R_PHYS};
    case ACS_C_TAU: return {4, R_TAU};
    case ACS_C_N_TAU: return {4, R_NTAU};
  }
  return {-1, -1};
}

}  // namespace

struct Batch {
  int n = 0;
  std::vector<acs_params> prm;
  std::vector<CaseDev> hc;    // host copy of the case table
  std::vector<CaseCtl> hk;    // host copy of the control words
  std::vector<char> t_unity;  // T known to be identically 1 (the buoyancy term vanishes)
  char* pool = nullptr;
  size_t pool_bytes = 0;
  CaseDev* dc = nullptr;
  CaseCtl* dk = nullptr;
  Tile* dtiles = nullptr;
  int ntiles = 0;
  int* d_nactive = nullptr;
  long long* d_iter = nullptr;
  int* d_iters = nullptr;
  double* d_err = nullptr;
  long long stats_cap = 0;
  bool ctl_stale = false;     // hk holds changes that the device's control words do not have yet
  double* d_stage = nullptr;  // staging of field transfers: device, and pinned host for per-routine calls
  double* h_stage = nullptr;
  size_t d_stage_cap = 0, h_stage_cap = 0;  // doubles
  bool stage_moved = false;   // the stream has changed since d_stage was last used
  int* h_flag = nullptr;  // mapped host word for the host-polled loop
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  bool graph_conditional = true;
  bool overlap = true;  // tile engine: programmatic dependent launches inside the loop body
  bool use_fast = false;
  FastPlan* fast = nullptr;
  long long launches = 0;
  long long body_kernels = 0;
  int graph_steps = -1;  // n_steps the graph's loop bound was built for
  int engine = 0;        // 0 = persistent cluster engine, 1 = graph of per-stage kernels,
                         // 2 = graph of TMA-tiled kernels (tile_engine.cu)
  // tile engine: tile table, tensor maps, TMA timeout word (set up on first use)
  Tile* d_tetiles = nullptr;
  int n_tetiles = 0;
  TeMaps* d_temaps = nullptr;
  int* d_te_err = nullptr;
  int nodes_per_cta = 1536;
  int l1_loads = 1;      // FAST engine: load cluster-written arrays through L1
  int threads = 512;     // FAST engine: threads per CTA (256 or 512)
  int ctas_per_sm = 1;   // FAST engine with 256 threads: 1 or 2 resident CTAs per SM
  int staged = 1;        // FAST engine: stage stencil arrays in shared memory where they fit
  bool on_chip = true;   // ACS_OPT_ON_CHIP
  int used = 0;          // enum acs_used of the last run
  std::vector<int> cluster_override;  // per case: CTAs of its cluster (0 = from nodes_per_cta)
  std::vector<char> chip_ok;          // per case: it has one porosity, no partly porous cells, no artificial
                                      // divergence damping (b_art) and constants in range (chip_divisors)
  bool user_nodes = false;            // nodes_per_cta was set by the caller
  std::vector<int> chip_k;            // per case: CTAs of its on-chip cluster (0 = cluster engine); built on
                                      // first use, emptied when a launch option changes
  double chip_us = 0.0;               // ChipPlan::us
  int* d_cases = nullptr;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> ev;
  // learned warm start (warmstart.cu): canvas size, per-case previous fields and increments
  int ws_H = 0, ws_W = 0;
  int ws_has_prev = 0;
  int ws_calls = 0;   // feature calls since acs_batch_ws_enable (3 give two increments)
  int ws_order = 1;   // ACS_OPT_EXTRAP_ORDER
  char* ws_pool = nullptr;
  WsCase* d_ws = nullptr;
  unsigned long long* d_ws_res = nullptr;
  int* d_ws_choice = nullptr;
  double* d_ws_ss = nullptr;  // per case and field: sum of inc^2, then the RMS of inc
  double* d_ws_sc = nullptr;

  ~Batch() {
    if (ws_pool) cudaFree(ws_pool);
    if (d_ws) cudaFree(d_ws);
    if (d_ws_res) cudaFree(d_ws_res);
    if (d_ws_choice) cudaFree(d_ws_choice);
    if (d_ws_ss) cudaFree(d_ws_ss);
    if (d_ws_sc) cudaFree(d_ws_sc);
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    if (fast) fast_destroy(fast);
    if (pool) cudaFree(pool);
    if (d_iters) cudaFree(d_iters);
    if (d_err) cudaFree(d_err);
    if (d_stage) cudaFree(d_stage);
    if (h_stage) cudaFreeHost(h_stage);
    if (h_flag) cudaFreeHost(h_flag);
    if (d_cases) cudaFree(d_cases);
    if (d_tetiles) cudaFree(d_tetiles);
    if (d_temaps) cudaFree(d_temaps);
    if (d_te_err) cudaFree(d_te_err);
    for (auto s : side) cudaStreamDestroy(s);
    for (auto e : ev) cudaEventDestroy(e);
    if (own_stream && stream) cudaStreamDestroy(stream);
  }

  double* buf(int c, int family, int idx) const {
    const CaseDev& d = hc[c];
    switch (family) {
      case 0: return d.U[idx];
      case 1: return d.V[idx];
      case 2: return d.P[idx];
      case 3: return d.T[idx];
      case 4: return d.C[idx];
    }
    return nullptr;
  }
  int role_index(int c, FieldLoc L) const {
    const CaseCtl& k = hk[c];
    if (L.role == R_NTAU && k.ntau_alias && (L.family <= 1 || hc[c].solve_scalars))
      L.role = k.ntau_alias == 1 ? R_PHYS : R_TAU;
    switch (L.family) {
      case 0: return k.ru[L.role];
      case 1: return k.rv[L.role];
      case 2: return L.role == 1 ? k.rp_read : k.rp[0];
      case 3: return k.rt[L.role];
      case 4: return k.rc[L.role];
    }
    return 0;
  }
};

// Checks of the parameter block that every entry point taking an acs_params shares (sizes are
// checked by the caller, whose limits differ).
int validate_params(const acs_params& p) {
  if (p.scheme != 0 && p.scheme != 1) return fail(ACS_E_ARG, "scheme must be 0 or 1");
  if (p.bc != 0 && p.bc != 1) return fail(ACS_E_ARG, "bc must be 0 or 1");
  if (p.arith != ACS_ARITH_EXACT && p.arith != ACS_ARITH_FAST) return fail(ACS_E_ARG, "arith must be 0 or 1");
  if (p.itc_max < 2) return fail(ACS_E_ARG, "itc_max must be at least 2");
  if (p.continuity != 0 && p.continuity != 1) return fail(ACS_E_ARG, "continuity must be 0 or 1");
  if (!(p.Re > 0) || !(p.Pe > 0) || !(p.Sc > 0) || !(p.Da > 0)) return fail(ACS_E_ARG, "Re, Pe, Sc, Da must be positive");
  return ACS_OK;
}

namespace {

int validate(const acs_grid& g, const acs_params& p) {
  if (!g.x || !g.y || !g.xm || !g.ym || !g.epsilon1 || !g.liga_poros) return fail(ACS_E_ARG, "null grid array");
  if (g.imax != p.imax || g.jmax != p.jmax) return fail(ACS_E_ARG, "grid and params disagree on imax/jmax");
  if (p.imax < kMinN || p.jmax < kMinN || p.imax > kMaxN || p.jmax > kMaxN)
    return fail(ACS_E_SIZE, "imax and jmax must lie in [6, 32768]");
  return validate_params(p);
}

// Binary porous structure (eps, liga) in {(1,0), (phi,1)} for one phi.
bool binary_porosity(const acs_grid& g, double* phi) {
  const size_t nc = (size_t)g.imax * g.jmax;
  double ph = -1.0;
  for (size_t q = 0; q < nc; ++q) {
    const double e = g.epsilon1[q], l = g.liga_poros[q];
    if (l == 0.0) {
      if (e != 1.0) return false;
    } else if (l == 1.0) {
      if (ph < 0.0) ph = e;
      if (e != ph || !(e > 0.0)) return false;
    } else {
      return false;
    }
  }
  *phi = ph < 0.0 ? 1.0 : ph;
  return true;
}

// Divisors of the EXACT on-chip arithmetic (chip_exact.cu): metric differences, porosity and drag
// constants must be positive and far from the exponent limits.
bool chip_divisors(const acs_grid& g, const acs_params& p, double phi) {
  auto ok = [](double v) { return v >= 0x1p-60 && v <= 0x1p60; };
  bool r = ok(phi) && ok(1.0 * (phi - 1.0) + 1.0) && ok(p.Re * p.Da) && ok(p.Re) && ok(p.Pe) && ok(p.Re * p.Sc) &&
           std::fabs(p.Cf) <= 0x1p200;
  for (int i = 1; i < g.imax; ++i) r = r && ok(g.x[i] - g.x[i - 1]);
  for (int j = 1; j < g.jmax; ++j) r = r && ok(g.y[j] - g.y[j - 1]);
  for (int i = 2; i < g.imax; ++i) r = r && ok(g.xm[i] - g.xm[i - 1]);  // interior cells only
  for (int j = 2; j < g.jmax; ++j) r = r && ok(g.ym[j] - g.ym[j - 1]);
  return r;
}

int push_ctl(Batch& b);
int flush_ctl(Batch& b);

// Whether a caller is capturing the batch's stream.
bool capturing(const Batch& b) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(b.stream, &st) != cudaSuccess) {  // (the legacy stream, while another one is captured)
    cudaGetLastError();
    return false;
  }
  return st != cudaStreamCaptureStatusNone;
}

int field_dims(const CaseDev& d, int family, int* w, int* h) {
  *w = family == 0 ? d.nx + 1 : d.nx;
  *h = family == 1 ? d.ny + 1 : d.ny;
  return 0;
}

// Staging buffers of at least n doubles, kept with the batch, which therefore stay below STAGE_MAX:
// transfers of more than that go in parts, and a field larger than that by a 2-D copy of its own.  Without
// the bound the state of a case would need device memory twice.  64 MiB is all 14 fields of 770 x 770 nodes.
constexpr long long STAGE_MAX = 8ll << 20;
int stage_dev(Batch& b, size_t n) {
  if (b.stage_moved) {  // transfers on the former stream may still use it; freeing it waits for them
    if (b.d_stage) cudaFree(b.d_stage);
    b.d_stage = nullptr;
    b.d_stage_cap = 0;
    b.stage_moved = false;
  }
  if (n <= b.d_stage_cap) return ACS_OK;
  CU(cudaStreamSynchronize(b.stream));
  if (b.d_stage) cudaFree(b.d_stage);
  b.d_stage = nullptr;
  b.d_stage_cap = 0;
  CU(cudaMalloc(&b.d_stage, n * sizeof(double)));
  b.d_stage_cap = n;
  return ACS_OK;
}
int stage_host(Batch& b, size_t n) {
  if (n <= b.h_stage_cap) return ACS_OK;
  if (b.h_stage) cudaFreeHost(b.h_stage);
  b.h_stage = nullptr;
  b.h_stage_cap = 0;
  CU(cudaMallocHost(&b.h_stage, n * sizeof(double)));
  b.h_stage_cap = n;
  return ACS_OK;
}

long long field_size(const Batch& b, int c, int family) {
  int w, h;
  field_dims(b.hc[c], family, &w, &h);
  return (long long)w * h;
}

// Adds a field of case c to a list of transfers.
void add_move(const Batch& b, MoveList& m, int c, int family, int idx) {
  const CaseDev& d = b.hc[c];
  int w, h;
  field_dims(d, family, &w, &h);
  m.f[m.n++] = FieldMove{b.buf(c, family, idx), m.total, w, h};
  m.pitch = d.pitch;
  m.total += (long long)w * h;
}

bool all_ones(const double* a, size_t n) {
  for (size_t q = 0; q < n; ++q)
    if (a[q] != 1.0) return false;
  return true;
}

// Before field `field` of case c is overwritten: control changes and copies that its role needs.
// Returns the field's place in *L.
int prepare_upload(Batch& b, int c, int field, const double* host, FieldLoc* out) {
  FieldLoc L = field_loc(field);
  if (L.family < 0) return fail(ACS_E_ARG, "unknown field id");
  if (field == ACS_UM_TAU || field == ACS_VM_TAU) {
    b.hk[c].tau_dirty = 1;
    b.ctl_stale = true;
  }
  if (L.role == R_NTAU && L.family != 2 && b.hk[c].ntau_alias) {
    // give every n_tau array its own values again before one of them is overwritten
    CaseCtl& k = b.hk[c];
    const CaseDev& d = b.hc[c];
    const int nfam = d.solve_scalars ? 4 : 2;
    const int fams[4] = {0, 1, 3, 4};
    for (int q = 0; q < nfam; ++q) {
      const int f = fams[q];
      const int src = b.role_index(c, FieldLoc{f, R_NTAU});
      const int* roles = f == 0 ? k.ru : f == 1 ? k.rv : f == 3 ? k.rt : k.rc;
      CU(cudaMemcpyAsync(b.buf(c, f, roles[R_NTAU]), b.buf(c, f, src), sizeof(double) * d.n_elems,
                         cudaMemcpyDeviceToDevice, b.stream));
    }
    k.ntau_alias = 0;
    b.ctl_stale = true;
  }
  if (L.family == 2) {
    // p and pn share one buffer after a non-exit iteration; give pn its own buffer first
    CaseCtl& k = b.hk[c];
    if (k.rp_read == k.rp[0]) {
      const CaseDev& d = b.hc[c];
      CU(cudaMemcpyAsync(d.P[k.rp[1]], d.P[k.rp[0]], sizeof(double) * d.n_elems, cudaMemcpyDeviceToDevice, b.stream));
      k.rp_read = k.rp[1];
      b.ctl_stale = true;
    }
  }
  if (field == ACS_T) b.t_unity[c] = all_ones(host, (size_t)b.hc[c].nx * b.hc[c].ny);
  *out = L;
  return ACS_OK;
}

// A field straight from or to a contiguous host array, without the staging buffer.
int put(Batch& b, int c, int family, int idx, const double* host) {
  const CaseDev& d = b.hc[c];
  int w, h;
  field_dims(d, family, &w, &h);
  if (w == d.pitch)
    CU(cudaMemcpyAsync(b.buf(c, family, idx), host, (size_t)w * h * 8, cudaMemcpyHostToDevice, b.stream));
  else
    CU(cudaMemcpy2DAsync(b.buf(c, family, idx), (size_t)d.pitch * 8, host, (size_t)w * 8, (size_t)w * 8, h,
                         cudaMemcpyHostToDevice, b.stream));
  return ACS_OK;
}

int get(Batch& b, int c, int family, int idx, double* host) {
  const CaseDev& d = b.hc[c];
  int w, h;
  field_dims(d, family, &w, &h);
  if (w == d.pitch)
    CU(cudaMemcpyAsync(host, b.buf(c, family, idx), (size_t)w * h * 8, cudaMemcpyDeviceToHost, b.stream));
  else
    CU(cudaMemcpy2DAsync(host, (size_t)w * 8, b.buf(c, family, idx), (size_t)d.pitch * 8, (size_t)w * 8, h,
                         cudaMemcpyDeviceToHost, b.stream));
  return ACS_OK;
}

// Whether a field goes straight to or from its array instead of through the staging buffer: one larger
// than the buffer, and one whose rows follow one another in the case's buffer too, which needs one plain
// copy (1024 x 512, pinned: up 87 us, down 85; staged 94 and 94).
bool direct(const Batch& b, int c, int family) {
  int w, h;
  field_dims(b.hc[c], family, &w, &h);
  return (long long)w * h > STAGE_MAX || w == b.hc[c].pitch;
}

bool pinned(const void* host) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, host) != cudaSuccess) cudaGetLastError();
  return a.type == cudaMemoryTypeHost;
}

// Uploads while a caller captures the batch's stream into a graph: a replay may come when the staging
// buffer has been replaced, and a capture must not allocate, so every field goes by a copy of its own.
int capture_uploads(Batch& b, int c, int n, const int* fields, const double* const* host) {
  int r = flush_ctl(b);
  for (int q = 0; q < n && !r; ++q) {
    FieldLoc L;
    r = prepare_upload(b, c, fields[q], host[q], &L);
    if (!r && b.ctl_stale) r = push_ctl(b);
    if (!r) r = put(b, c, L.family, b.role_index(c, L), host[q]);
  }
  return r;
}

// The transfers listed in m, through the staging buffer; host[q]: the array of m.f[q].
int move_in(Batch& b, MoveList& m, const double* const* host) {
  if (!m.n) return ACS_OK;
  int r = stage_dev(b, (size_t)m.total);
  if (r) return r;
  for (int q = 0; q < m.n; ++q)
    CU(cudaMemcpyAsync(b.d_stage + m.f[q].off, host[q], sizeof(double) * m.f[q].w * m.f[q].h, cudaMemcpyHostToDevice, b.stream));
  move_to_case(m, b.d_stage, nullptr, CaseCtl{}, b.stream);
  CU(cudaGetLastError());
  m = MoveList{};
  return ACS_OK;
}
int move_out(Batch& b, MoveList& m, double* const* host) {
  if (!m.n) return ACS_OK;
  int r = stage_dev(b, (size_t)m.total);
  if (r) return r;
  move_from_case(m, b.d_stage, nullptr, b.stream);
  CU(cudaGetLastError());
  for (int q = 0; q < m.n; ++q)
    CU(cudaMemcpyAsync(host[q], b.d_stage + m.f[q].off, sizeof(double) * m.f[q].w * m.f[q].h, cudaMemcpyDeviceToHost, b.stream));
  m = MoveList{};
  return ACS_OK;
}

// n distinct fields of case c from contiguous host arrays, each applied in the order given.
int upload_fields(Batch& b, int c, int n, const int* fields, const double* const* host) {
  if (capturing(b)) return capture_uploads(b, c, n, fields, host);
  MoveList m{};
  const double* src[MOVE_MAX];
  for (int q = 0; q < n; ++q) {
    const FieldLoc l = field_loc(fields[q]);
    if (l.role == R_NTAU && l.family >= 0 && l.family != 2 && b.hk[c].ntau_alias) {
      // n_tau arrays get their own copies now, of what the fields before this one have become
      if (int r = move_in(b, m, src)) return r;
    }
    FieldLoc L;
    int r = prepare_upload(b, c, fields[q], host[q], &L);
    if (r) return r;
    if (direct(b, c, L.family)) {
      if ((r = put(b, c, L.family, b.role_index(c, L), host[q]))) return r;
      continue;
    }
    if (m.total + field_size(b, c, L.family) > STAGE_MAX && (r = move_in(b, m, src))) return r;
    src[m.n] = host[q];
    add_move(b, m, c, L.family, b.role_index(c, L));
  }
  return move_in(b, m, src);
}

int download_fields(Batch& b, int c, int n, const int* fields, double* const* host) {
  MoveList m{};
  double* dst[MOVE_MAX];
  for (int q = 0; q < n; ++q) {
    FieldLoc L = field_loc(fields[q]);
    if (L.family < 0) return fail(ACS_E_ARG, "unknown field id");
    int r = 0;
    // a single field into pinned memory: the copy by rows (51 x 51: 12 us, 153 x 153: 15) beats kernel and
    // copy (17, 20); pageable memory takes rows slower (153 x 153: 50 to 56 against 40)
    if (direct(b, c, L.family) || (n == 1 && pinned(host[q]))) {
      if ((r = get(b, c, L.family, b.role_index(c, L), host[q]))) return r;
      continue;
    }
    if (m.total + field_size(b, c, L.family) > STAGE_MAX && (r = move_out(b, m, dst))) return r;
    dst[m.n] = host[q];
    add_move(b, m, c, L.family, b.role_index(c, L));
  }
  if (int r = move_out(b, m, dst)) return r;
  CU(cudaStreamSynchronize(b.stream));
  return ACS_OK;
}

int refresh_flags(Batch& b) {
  for (int c = 0; c < b.n; ++c) {
    CaseDev& d = b.hc[c];
    const acs_params& p = b.prm[c];
    int f = d.flags & ~F_BUOY;
    if (p.InvFr2 != 0.0 && (p.solve_scalars || !b.t_unity[c])) f |= F_BUOY;
    if (f != d.flags) {
      d.flags = f;
      CU(cudaMemcpyAsync(b.dc + c, &d, sizeof(CaseDev), cudaMemcpyHostToDevice, b.stream));
    }
  }
  return ACS_OK;
}

int push_ctl(Batch& b) {
  b.ctl_stale = false;
  CU(cudaMemcpyAsync(b.dk, b.hk.data(), sizeof(CaseCtl) * b.n, cudaMemcpyHostToDevice, b.stream));
  return ACS_OK;
}
// Before kernels that read the control words outside a run.  While a caller captures the stream, the words
// that earlier uploads changed are copied at once, on a stream of their own: work outside the graph needs
// them too.
int flush_ctl(Batch& b) {
  if (!b.ctl_stale) return ACS_OK;
  if (!capturing(b)) return push_ctl(b);
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  CU(cudaThreadExchangeStreamCaptureMode(&mode));
  cudaStream_t s = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMemcpyAsync(b.dk, b.hk.data(), sizeof(CaseCtl) * b.n, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (s) cudaStreamDestroy(s);
  CU(cudaThreadExchangeStreamCaptureMode(&mode));
  CU(e);
  b.ctl_stale = false;
  return ACS_OK;
}
int pull_ctl(Batch& b) {
  CU(cudaMemcpyAsync(b.hk.data(), b.dk, sizeof(CaseCtl) * b.n, cudaMemcpyDeviceToHost, b.stream));
  CU(cudaStreamSynchronize(b.stream));
  return ACS_OK;
}

void reset_roles(CaseCtl& k) {
  for (int r = 0; r < 3; ++r) k.ru[r] = k.rv[r] = k.rt[r] = k.rc[r] = r;
  k.rp[0] = 0;
  k.rp[1] = 1;
  k.rp_read = 1;
  k.ntau_alias = 0;
  k.tau_dirty = 1;
}

// Grid arrays may be host or device pointers (acs_mesh_channel_device writes device arrays): a
// grid with any array in device memory is copied to host storage before the pool is built.
int host_grids(const acs_grid* grids, int n, std::vector<acs_grid>& hg, std::vector<std::vector<double>>& store) {
  hg.assign(grids, grids + n);
  for (int c = 0; c < n; ++c) {
    acs_grid& g = hg[c];
    const double** arr[6] = {&g.x, &g.y, &g.xm, &g.ym, &g.epsilon1, &g.liga_poros};
    const size_t len[6] = {(size_t)g.imax, (size_t)g.jmax, (size_t)g.imax + 1, (size_t)g.jmax + 1,
                           (size_t)g.imax * g.jmax, (size_t)g.imax * g.jmax};
    for (int k = 0; k < 6; ++k) {
      cudaPointerAttributes a{};
      if (cudaPointerGetAttributes(&a, *arr[k]) != cudaSuccess) {
        cudaGetLastError();
        continue;  // not known to CUDA: host memory
      }
      if (a.type != cudaMemoryTypeDevice) continue;
      store.emplace_back(len[k]);
      if (cudaMemcpy(store.back().data(), *arr[k], sizeof(double) * len[k], cudaMemcpyDeviceToHost) != cudaSuccess)
        return fail(ACS_E_CUDA, "copying a device grid array");
      *arr[k] = store.back().data();
    }
  }
  return ACS_OK;
}

int create_batch(const acs_grid* grids_in, const acs_params* params, int n, Batch** out) {
  if (!grids_in || !params || n <= 0 || !out) return fail(ACS_E_ARG, "null argument or n <= 0");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return fail(ACS_E_CUDA, "no CUDA device");
  for (int c = 0; c < n; ++c) {
    int r = validate(grids_in[c], params[c]);
    if (r) return r;
  }
  std::vector<acs_grid> hg;
  std::vector<std::vector<double>> grid_store;
  if (int r = host_grids(grids_in, n, hg, grid_store)) return r;
  const acs_grid* grids = hg.data();
  const bool fast = params[0].arith == ACS_ARITH_FAST;
  for (int c = 1; c < n; ++c)
    if ((params[c].arith == ACS_ARITH_FAST) != fast) return fail(ACS_E_ARG, "all cases of a batch must use one arith mode");

  // Layout of the pool: [case table][control][tiles][counters] then per case
  // [metrics][eps][liga][mask][U x3][V x3][P x2][T x3][C x3][S x4].
  std::vector<size_t> off(n);
  std::vector<size_t> sizes(n);
  size_t total = 0;
  for (int c = 0; c < n; ++c) {
    const int nx = params[c].imax, ny = params[c].jmax;
    const size_t ne = align_up(nx + 1, 4) * (size_t)(ny + 1);
    size_t sz = align_up(sizeof(double) * (2 * nx + 2 * ny + 6), 256) + 2 * align_up(8 * ne, 256) +
                align_up(ne, 256) + 22 * align_up(8 * ne, 256);
    off[c] = total;
    sizes[c] = sz;
    total += align_up(sz, 256);
  }
  std::vector<Tile> tiles;
  for (int c = 0; c < n; ++c)
    for (int j0 = 1; j0 <= params[c].jmax + 1; j0 += TILE_Y)
      for (int i0 = 1; i0 <= params[c].imax + 1; i0 += TILE_X) tiles.push_back({c, i0, j0, 0});
  const size_t a_case = align_up(sizeof(CaseDev) * n, 256);
  const size_t a_ctl = align_up(sizeof(CaseCtl) * n, 256);
  const size_t a_tile = align_up(sizeof(Tile) * tiles.size(), 256);
  const size_t head = a_case + a_ctl + a_tile + 256;

  Batch* b = new Batch();
  b->n = n;
  b->prm.assign(params, params + n);
  b->hc.resize(n);
  b->hk.assign(n, CaseCtl{});
  b->t_unity.assign(n, 0);
  b->chip_ok.assign(n, 0);
  b->use_fast = fast;
  b->pool_bytes = head + total;
  cudaError_t e = cudaMalloc(&b->pool, b->pool_bytes);
  if (e != cudaSuccess) {
    delete b;
    return fail(ACS_E_NOMEM, std::string("cudaMalloc of the case pool: ") + cudaGetErrorString(e));
  }
  e = cudaMemset(b->pool, 0, b->pool_bytes);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete b;
    return fail(ACS_E_CUDA, std::string("batch set-up: ") + cudaGetErrorString(e));
  }
  b->own_stream = true;
  char* p = b->pool;
  b->dc = (CaseDev*)p;
  b->dk = (CaseCtl*)(p + a_case);
  b->dtiles = (Tile*)(p + a_case + a_ctl);
  b->d_nactive = (int*)(p + a_case + a_ctl + a_tile);
  b->d_iter = (long long*)(p + a_case + a_ctl + a_tile + 64);
  b->ntiles = (int)tiles.size();
  char* base = p + head;
  std::vector<double> stage;
  for (int c = 0; c < n; ++c) {
    const acs_grid& g = grids[c];
    const acs_params& pr = params[c];
    const int nx = pr.imax, ny = pr.jmax;
    const int pitch = (int)align_up(nx + 1, 4);
    const size_t ne = (size_t)pitch * (ny + 1);
    char* q = base + off[c];
    CaseDev& d = b->hc[c];
    std::memset(&d, 0, sizeof(d));
    d.nx = nx; d.ny = ny; d.pitch = pitch;
    d.scheme = pr.scheme; d.bc = pr.bc; d.solve_scalars = pr.solve_scalars; d.itc_max = pr.itc_max;
    d.continuity = pr.continuity;
    d.Re = pr.Re; d.Pe = pr.Pe; d.Sc = pr.Sc; d.Da = pr.Da; d.Cf = pr.Cf; d.g = pr.g;
    d.InvFr2 = pr.InvFr2; d.v_in = pr.v_in; d.T_in = pr.T_in; d.C_in = pr.C_in; d.b_art = pr.b_art;
    d.beta = pr.beta; d.dt = pr.dt; d.dtau = pr.dtau; d.eps = pr.eps;
    d.n_elems = (long long)ne;
    stage.assign(2 * nx + 2 * ny + 6, 0.0);
    double* X = stage.data();
    double* Y = X + (nx + 1);
    double* XM = Y + (ny + 1);
    double* YM = XM + (nx + 2);
    for (int i = 1; i <= nx; ++i) X[i] = g.x[i - 1];
    for (int j = 1; j <= ny; ++j) Y[j] = g.y[j - 1];
    for (int i = 1; i <= nx + 1; ++i) XM[i] = g.xm[i - 1];
    for (int j = 1; j <= ny + 1; ++j) YM[j] = g.ym[j - 1];
    double* dm = (double*)q;
    d.x = dm; d.y = dm + (nx + 1); d.xm = d.y + (ny + 1); d.ym = d.xm + (nx + 2);
    CU(cudaMemcpy(dm, stage.data(), sizeof(double) * stage.size(), cudaMemcpyHostToDevice));
    q += align_up(sizeof(double) * (2 * nx + 2 * ny + 6), 256);
    double* deps = (double*)q; q += align_up(8 * ne, 256);
    double* dliga = (double*)q; q += align_up(8 * ne, 256);
    uint8_t* dmask = (uint8_t*)q; q += align_up(ne, 256);
    std::vector<double> pe(ne, 1.0), pl(ne, 0.0);
    std::vector<uint8_t> pm(ne, 0);
    bool porous = false;
    for (int j = 1; j <= ny; ++j)
      for (int i = 1; i <= nx; ++i) {
        const size_t s = (size_t)(i - 1) + (size_t)(j - 1) * nx;
        const size_t t = (size_t)lin(i, j, pitch);
        pe[t] = g.epsilon1[s];
        pl[t] = g.liga_poros[s];
        pm[t] = g.liga_poros[s] != 0.0;
        porous |= g.liga_poros[s] != 0.0;
      }
    CU(cudaMemcpy(deps, pe.data(), 8 * ne, cudaMemcpyHostToDevice));
    CU(cudaMemcpy(dliga, pl.data(), 8 * ne, cudaMemcpyHostToDevice));
    CU(cudaMemcpy(dmask, pm.data(), ne, cudaMemcpyHostToDevice));
    d.epsf = deps; d.liga = dliga; d.mask = dmask;
    double phi = 1.0;
    if (binary_porosity(g, &phi)) d.flags |= F_BINARY;
    d.phi = phi;
    b->chip_ok[c] = (d.flags & F_BINARY) && pr.b_art == 0.0 && (fast || chip_divisors(g, pr, phi));
    if (pr.b_art != 0.0) d.flags |= F_BART;
    if (porous) d.flags |= F_POROUS;
    if (pr.InvFr2 != 0.0 && pr.solve_scalars) d.flags |= F_BUOY;
    double** bufs[5] = {d.U, d.V, d.P, d.T, d.C};
    const int counts[5] = {3, 3, 2, 3, 3};
    for (int f = 0; f < 5; ++f)
      for (int r = 0; r < counts[f]; ++r) {
        bufs[f][r] = (double*)q;
        q += align_up(8 * ne, 256);
      }
    for (int r = 0; r < 4; ++r) { d.S[r] = (double*)q; q += align_up(8 * ne, 256); }
    for (int r = 0; r < 4; ++r) { d.S2[r] = (double*)q; q += align_up(8 * ne, 256); }
    reset_roles(b->hk[c]);
  }
  if (fast) {
    int r = fast_create(b->hc, grids, params, &b->fast);
    if (r) {
      delete b;
      return r;
    }
  }
  e = cudaMemcpy(b->dc, b->hc.data(), sizeof(CaseDev) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->dk, b->hk.data(), sizeof(CaseCtl) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(b->dtiles, tiles.data(), sizeof(Tile) * tiles.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    delete b;
    return fail(ACS_E_CUDA, std::string("batch upload: ") + cudaGetErrorString(e));
  }
  *out = b;
  return ACS_OK;
}

// ---- launch sequences --------------------------------------------------------------------------
// solve_U: three stages, each followed by bcUV(stage array, vm_tau) (equations.f90:259-296)
void seq_u(Batch& b) {
  for (int s = 1; s <= 3; ++s) {
    (b.use_fast ? launch_u_stage_fast : launch_u_stage_exact)(s, b.dc, b.dk, b.dtiles, b.ntiles, b.stream);
    launch_bc_uv(b.dc, b.dk, b.n, s - 1, b.stream);
  }
  b.launches += 6;
}

// solve_V: three stages, each followed by bcUV(um_tau, stage array) (equations.f90:561-598)
void seq_v(Batch& b) {
  for (int s = 1; s <= 3; ++s) {
    (b.use_fast ? launch_v_stage_fast : launch_v_stage_exact)(s, b.dc, b.dk, b.dtiles, b.ntiles, b.stream);
    launch_bc_uv(b.dc, b.dk, b.n, 3 + s - 1, b.stream);
  }
  b.launches += 6;
}

// solve_P: the stages fuse pointwise; the intermediate bcP(pi) never reaches the interior
void seq_p(Batch& b) {
  (b.use_fast ? launch_p_fast : launch_p_exact)(b.dc, b.dk, b.dtiles, b.ntiles, b.stream);
  launch_bc_cell(b.dc, b.dk, b.n, 0, b.stream);
  b.launches += 2;
}

// solve_Z / solve_C: three stages, each followed by bcZ / bcC
void seq_s(Batch& b, bool is_c) {
  const int w0 = is_c ? 4 : 1;
  for (int s = 1; s <= 3; ++s) {
    (b.use_fast ? launch_s_stage_fast : launch_s_stage_exact)(is_c, s, b.dc, b.dk, b.dtiles, b.ntiles, b.stream);
    launch_bc_cell(b.dc, b.dk, b.n, w0 + s - 1, b.stream);
  }
  b.launches += 6;
}

// one launch of the timed kernel (acs_batch_time_kernel)
void launch_timed_kernel(Batch& b, int kernel) {
  switch (kernel) {
    case 0: (b.use_fast ? launch_u_stage_fast : launch_u_stage_exact)(1, b.dc, b.dk, b.dtiles, b.ntiles, b.stream); break;
    case 1: (b.use_fast ? launch_v_stage_fast : launch_v_stage_exact)(1, b.dc, b.dk, b.dtiles, b.ntiles, b.stream); break;
    case 2: (b.use_fast ? launch_p_fast : launch_p_exact)(b.dc, b.dk, b.dtiles, b.ntiles, b.stream); break;
    case 3: (b.use_fast ? launch_s_stage_fast : launch_s_stage_exact)(false, 1, b.dc, b.dk, b.dtiles, b.ntiles, b.stream); break;
    case 4: (b.use_fast ? launch_s_stage_fast : launch_s_stage_exact)(true, 1, b.dc, b.dk, b.dtiles, b.ntiles, b.stream); break;
    case 5: te_launch_uv(2, b.dc, b.dk, b.d_tetiles, b.n_tetiles, b.d_temaps, b.d_te_err, false, b.stream); break;
    case 6: te_launch_ptc(b.dc, b.dk, b.d_tetiles, b.n_tetiles, b.d_temaps, b.d_te_err, false, b.stream); break;
  }
}

bool any_scalars(const Batch& b) {
  for (auto& p : b.prm)
    if (p.solve_scalars) return true;
  return false;
}

// Tile engine set-up: tile table over every case, a tensor map per case buffer and box size.
int te_setup(Batch& b) {
  if (b.d_temaps) return ACS_OK;
  if (!b.use_fast) return fail(ACS_E_UNSUPPORTED, "the tile engine computes in the FAST arithmetic only");
  std::vector<Tile> tiles;
  for (int c = 0; c < b.n; ++c) te_case_tiles(c, b.hc[c].pitch, b.hc[c].ny, tiles);
  std::vector<TeMaps> maps(b.n);
  const int er = te_encode_maps(b.hc, maps.data());
  if (er) return fail(ACS_E_CUDA, er == 1 ? "cuTensorMapEncodeTiled is not available from the driver"
                                           : "cuTensorMapEncodeTiled rejected a case buffer");
  CU(te_prepare());
  CU(cudaMalloc(&b.d_tetiles, sizeof(Tile) * tiles.size()));
  CU(cudaMalloc(&b.d_temaps, sizeof(TeMaps) * b.n));
  CU(cudaMalloc(&b.d_te_err, sizeof(int)));
  CU(cudaMemcpy(b.d_tetiles, tiles.data(), sizeof(Tile) * tiles.size(), cudaMemcpyHostToDevice));
  CU(cudaMemcpy(b.d_temaps, maps.data(), sizeof(TeMaps) * b.n, cudaMemcpyHostToDevice));
  CU(cudaMemset(b.d_te_err, 0, sizeof(int)));
  b.n_tetiles = (int)tiles.size();
  return ACS_OK;
}

// What k_control's last block does at the end of an iteration (mode, handle, max_iters, host flag set by
// build_graph).
LoopEnd loop_end(Batch& b, int mode) {
  LoopEnd e{};
  e.mode = mode;
  e.tau_bc = b.engine == 2;
  e.iter_count = b.d_iter;
  e.ticket = b.d_nactive + 32;
  return e;
}

cudaError_t launch_control(Batch& b, const LoopEnd& end) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(b.n);
  cfg.blockDim = dim3(256);
  cfg.stream = b.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = b.engine == 2 && b.overlap ? 1 : 0;
  b.launches += 1;
  return cudaLaunchKernelEx(&cfg, k_control, (const CaseDev*)b.dc, b.dk, b.d_iters, b.d_err, b.d_nactive, end);
}

// One pseudo-iteration of the tile engine: U/V stages 1-3, P + T/C, control.  Returns the first launch error,
// as loop_body does: a loop body without one of its kernels must not run (k_control ends the loop).
cudaError_t te_iteration(Batch& b, const LoopEnd& end) {
  cudaError_t e = cudaSuccess;
  for (int s = 1; s <= 3 && e == cudaSuccess; ++s)
    e = te_launch_uv(s, b.dc, b.dk, b.d_tetiles, b.n_tetiles, b.d_temaps, b.d_te_err, b.overlap && s > 1, b.stream);
  if (e == cudaSuccess) e = te_launch_ptc(b.dc, b.dk, b.d_tetiles, b.n_tetiles, b.d_temaps, b.d_te_err, b.overlap, b.stream);
  b.launches += 4;
  return e == cudaSuccess ? launch_control(b, end) : e;
}

// one pseudo-iteration (main.f90:122-150) for every active case
cudaError_t seq_iteration(Batch& b, const LoopEnd& end) {
  seq_u(b);
  seq_v(b);
  seq_p(b);
  if (any_scalars(b)) {
    seq_s(b, false);
    seq_s(b, true);
  }
  return launch_control(b, end);
}

// The body of the pseudo-time loop, captured on the batch's stream.
cudaError_t loop_body(Batch& b, const LoopEnd& end) {
  cudaGetLastError();
  const cudaError_t e = b.engine == 2 ? te_iteration(b, end) : seq_iteration(b, end);
  const cudaError_t any = cudaGetLastError();  // of the launches whose status is not returned
  return e != cudaSuccess ? e : any;
}

long long max_total_iterations(const Batch& b, int n_steps) {
  long long m = 0;
  for (auto& p : b.prm) m = std::max(m, (long long)p.itc_max * (long long)n_steps);
  return m + 2;
}

int build_graph(Batch& b, int n_steps) {
  if (b.gexec) { cudaGraphExecDestroy(b.gexec); b.gexec = nullptr; }
  if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
  const long long saved = b.launches;
  // ACS_NO_CONDITIONAL_GRAPH=1 selects the host-polled loop below (profilers cannot look inside
  // a graph that holds conditional nodes)
  if (getenv("ACS_NO_CONDITIONAL_GRAPH")) b.graph_conditional = false;
  if (b.graph_conditional) {
    cudaGraph_t g;
    CU(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle h;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault);
    cudaGraphNode_t node;
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    if (e == cudaSuccess) e = cudaGraphAddNode(&node, g, nullptr, 0, &np);
    if (e == cudaSuccess) {
      cudaGraph_t body = np.conditional.phGraph_out[0];
      e = cudaStreamBeginCaptureToGraph(b.stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
      if (e == cudaSuccess) {
        const long long l0 = b.launches;
        LoopEnd end = loop_end(b, LOOP_COND);
        end.handle = h;
        end.max_iters = max_total_iterations(b, n_steps);
        const cudaError_t launched = loop_body(b, end);
        b.body_kernels = b.launches - l0;
        e = cudaStreamEndCapture(b.stream, &body);
        if (launched != cudaSuccess) e = launched;
      }
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&b.gexec, g, 0);
    if (e == cudaSuccess) {
      b.graph = g;
      b.launches = saved;
      return ACS_OK;
    }
    cudaGetLastError();
    cudaGraphDestroy(g);
    b.launches = saved;
    if (b.engine == 2 && b.overlap) {  // once more without overlapped launches
      b.overlap = false;
      return build_graph(b, n_steps);
    }
    b.graph_conditional = false;  // fall back to the host-polled loop below
  }
  // host-polled: the graph holds one iteration plus a flag publish
  if (!b.h_flag) CU(cudaHostAlloc(&b.h_flag, sizeof(int), cudaHostAllocMapped));
  int* d_flag = nullptr;
  CU(cudaHostGetDevicePointer(&d_flag, b.h_flag, 0));
  cudaGraph_t g;
  CU(cudaStreamBeginCapture(b.stream, cudaStreamCaptureModeThreadLocal));
  const long long l0 = b.launches;
  LoopEnd end = loop_end(b, LOOP_FLAG);
  end.host_flag = d_flag;
  const cudaError_t launched = loop_body(b, end);
  b.body_kernels = b.launches - l0;
  CU(cudaStreamEndCapture(b.stream, &g));
  if (launched != cudaSuccess) {
    cudaGraphDestroy(g);
    return fail(ACS_E_CUDA, std::string("loop body: ") + cudaGetErrorString(launched));
  }
  CU(cudaGraphInstantiate(&b.gexec, g, 0));
  b.graph = g;
  b.launches = saved;
  return ACS_OK;
}

int run_engine(Batch& b);
int run_graph(Batch& b, int n_steps);
bool chip_beats_tiles(Batch& b);

int run_batch(Batch& b, int n_steps, int* itc, int* iters, double* err, int* status) {
  if (n_steps <= 0) return fail(ACS_E_ARG, "n_steps must be positive");
  int r = refresh_flags(b);
  if (r) return r;
  const long long need = (long long)b.n * n_steps;
  if (need > b.stats_cap) {
    if (b.d_iters) cudaFree(b.d_iters);
    if (b.d_err) cudaFree(b.d_err);
    b.d_iters = nullptr;
    b.d_err = nullptr;
    CU(cudaMalloc(&b.d_iters, sizeof(int) * need));
    CU(cudaMalloc(&b.d_err, sizeof(double) * need));
    b.stats_cap = need;
    if (b.gexec) { cudaGraphExecDestroy(b.gexec); b.gexec = nullptr; }
    if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
  }
  for (int c = 0; c < b.n; ++c) {
    CaseCtl& k = b.hk[c];
    k.itc = itc ? itc[c] : 1;
    k.step = 0;
    k.n_steps = n_steps;
    k.k = 0;
    k.active = 1;
    k.status = 0;
    k.copy_phys = 0;
    k.res_u = k.res_v = k.res_p = 0;
    k.total_iters = 0;
    k.scalars = b.prm[c].solve_scalars ? 1 : 0;
  }
  r = push_ctl(b);
  if (r) return r;
  CU(cudaMemsetAsync(b.d_nactive, 0, 256, b.stream));
  b.used = 0;
  if (b.engine == 0 || (b.engine == 2 && chip_beats_tiles(b))) {
    r = run_engine(b);
    if (r) return r;
  } else {
    b.used = b.engine == 2 ? ACS_USED_TILE : ACS_USED_GRAPH;
    r = run_graph(b, n_steps);
    if (r) return r;
  }
  r = pull_ctl(b);
  if (r) return r;
  if (iters) CU(cudaMemcpy(iters, b.d_iters, sizeof(int) * need, cudaMemcpyDeviceToHost));
  if (err) CU(cudaMemcpy(err, b.d_err, sizeof(double) * need, cudaMemcpyDeviceToHost));
  bool failed = false;
  for (int c = 0; c < b.n; ++c) {
    if (itc) itc[c] = b.hk[c].itc;
    if (status) status[c] = b.hk[c].status;
    failed |= b.hk[c].status == ACS_CASE_FAILED;
    b.hk[c].active = 0;
  }
  CU(cudaMemsetAsync(b.d_iter, 0, sizeof(long long), b.stream));
  r = push_ctl(b);
  if (r) return r;
  CU(cudaStreamSynchronize(b.stream));
  if (failed) return fail(ACS_E_STATE, "a case failed: NaN or infinite residual");
  return ACS_OK;
}

int run_graph(Batch& b, int n_steps) {
  int r;
  if (b.engine == 2) {
    r = te_setup(b);
    if (r) return r;
  }
  // the graph bakes in the loop bound; rebuild when n_steps changes the bound
  if (!b.gexec || b.graph_steps != n_steps) {
    r = build_graph(b, n_steps);
    if (r) return r;
    b.graph_steps = n_steps;
  }
  if (b.graph_conditional) {
    CU(cudaGraphLaunch(b.gexec, b.stream));
    CU(cudaStreamSynchronize(b.stream));
  } else {
    const long long cap = max_total_iterations(b, n_steps);
    for (long long it = 0; it < cap; ++it) {
      CU(cudaGraphLaunch(b.gexec, b.stream));
      if ((it & 15) == 15) {
        CU(cudaStreamSynchronize(b.stream));
        if (*(volatile int*)b.h_flag == 0) break;
      }
    }
    CU(cudaStreamSynchronize(b.stream));
  }
  long long iters_done = 0;
  CU(cudaMemcpy(&iters_done, b.d_iter, sizeof(long long), cudaMemcpyDeviceToHost));
  b.launches = iters_done * b.body_kernels;
  if (b.engine == 2) {
    int te_err = 0;
    CU(cudaMemcpy(&te_err, b.d_te_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (te_err) return fail(ACS_E_CUDA, "tile engine: a TMA wait timed out (the results of this run are not valid)");
  }
  return ACS_OK;
}

// Cluster size for a case: about nodes_per_cta nodes per CTA, at most 16 CTAs, strips of at
// least 4 node rows.
int cluster_size(const Batch& b, int c) {
  const CaseDev& d = b.hc[c];
  const long long nodes = (long long)(d.nx + 1) * (d.ny + 1);
  int K = (int)((nodes + b.nodes_per_cta - 1) / b.nodes_per_cta);
  if (c < (int)b.cluster_override.size() && b.cluster_override[c] > 0) K = b.cluster_override[c];
  K = std::max(1, std::min(K, 16));
  K = std::min(K, std::max(1, (d.ny + 1) / 4));
  return K;
}

PlanCase plan_case(const Batch& b, int c) {
  const CaseDev& d = b.hc[c];
  const bool user = b.user_nodes || (c < (int)b.cluster_override.size() && b.cluster_override[c] > 0);
  return {d.nx, d.ny, d.pitch, d.solve_scalars != 0, b.on_chip && b.chip_ok[c], user ? cluster_size(b, c) : 0};
}

void chip_plan(Batch& b) {
  if ((int)b.chip_k.size() == b.n) return;
  std::vector<PlanCase> cases;
  for (int c = 0; c < b.n; ++c) cases.push_back(plan_case(b, c));
  ChipPlan p = plan_chip(cases, b.use_fast, b.use_fast ? chip_resident_fast : chip_resident_exact);
  b.chip_k = std::move(p.k);
  b.chip_us = p.us;
}

// Whether a batch on the tile engine is faster on chip.  The model of the tile engine's time is 50 us, or 30 and
// 0.165 per 1000 nodes once its tiles fill the device; a few cases in clusters iterate side by side in 6 to 28 us.
// Measured with the loop's five overlapped launches, tiles and on chip, us per pseudo-iteration: one case of
// 51 x 51 45 and 7.6, of 153 x 153 44 and 28; three of 101 x 147 46 and 19; of 153 x 153 7 55 and 28, 8 55 and 55,
// 15 92 and 83 (left on the tiles), 28 140 and 111, 56 248 and 222, 64 280 and 277, 128 505 and 526; 512 of
// 51 x 51 358 and 153 (32 x 32 tiles pad small cases); without scalars 64 of 153 x 153 188 and 132, 8 of 200 x 180
// 59 and 49.  Only a clear advantage of the modelled times counts.
bool chip_beats_tiles(Batch& b) {
  chip_plan(b);
  double nodes = 0.0;
  for (int c = 0; c < b.n; ++c) nodes += (double)b.hc[c].nx * b.hc[c].ny;
  return b.chip_us > 0.0 && b.chip_us < 0.8 * std::max(50.0, 30.0 + 1.65e-4 * nodes);
}

// One launch per cluster size and engine, each on its own stream so the classes run side by side.
int run_engine(Batch& b) {
  chip_plan(b);
  // classes 0..16: cluster engine by cluster size; from 17 on the on-chip engine by cluster size,
  // with bit 0 of class / 17 - 1: the physical-step arrays on chip too, bit 1: QUICK
  constexpr int kClasses = 5 * 17;
  std::vector<std::vector<int>> groups(kClasses);
  for (int c = 0; c < b.n; ++c) {
    const int K = b.chip_k[c];
    const int kind = 1 + (K && chip_bytes(plan_case(b, c), K, true) ? 1 : 0) + (b.hc[c].scheme == 0 ? 2 : 0);
    groups[!K ? cluster_size(b, c) : 17 * kind + K].push_back(c);
  }
  if (!b.d_cases) CU(cudaMalloc(&b.d_cases, sizeof(int) * b.n));
  std::vector<int> order;
  std::vector<std::pair<int, int>> launches;  // (class, offset)
  for (int k = kClasses - 1; k >= 0; --k) {
    if (groups[k].empty()) continue;
    launches.push_back({k, (int)order.size()});
    order.insert(order.end(), groups[k].begin(), groups[k].end());
  }
  CU(cudaMemcpyAsync(b.d_cases, order.data(), sizeof(int) * order.size(), cudaMemcpyHostToDevice, b.stream));
  for (int c = 0; c < b.n; ++c) {
    std::memset(b.hk[c].slot, 0, sizeof(b.hk[c].slot));
  }
  int r = push_ctl(b);
  if (r) return r;
  while (b.side.size() < launches.size()) {
    cudaStream_t s;
    CU(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    b.side.push_back(s);
    cudaEvent_t e;
    CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    b.ev.push_back(e);
  }
  cudaEvent_t fork;
  CU(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
  CU(cudaEventRecord(fork, b.stream));
  b.launches = 0;
  for (size_t g = 0; g < launches.size(); ++g) {
    const int cls = launches[g].first, K = cls % 17;
    const int off = launches[g].second;
    const int cnt = (int)groups[cls].size();
    cudaStream_t s = g == 0 ? b.stream : b.side[g];
    if (g) CU(cudaStreamWaitEvent(s, fork, 0));
    cudaError_t e;
    if (cls >= 17) {
      const bool phys = (cls / 17 - 1) & 1, quick = (cls / 17 - 1) & 2;
      size_t smem = 0;
      for (int q = 0; q < cnt; ++q) smem = std::max(smem, chip_bytes(plan_case(b, order[off + q]), K, phys));
      ChipArgs a{b.dc, b.dk, b.d_cases + off, b.d_iters, b.d_err, b.engine == 2 ? R_PHYS : R_NTAU, b.engine == 2};
      e = (b.use_fast ? launch_chip_fast : launch_chip_exact)(a, K, cnt, phys, quick, smem, s);
    } else {
    // staging slot: the largest strip of the size class plus two halo rows on each side
    long long slot = 0;
    for (int q = 0; q < cnt; ++q) {
      const CaseDev& d = b.hc[order[off + q]];
      const long long rows = (d.ny + 1 + K - 1) / K + 4;
      slot = std::max(slot, (rows * d.pitch + 1) / 2 * 2);
    }
    const bool stg = b.use_fast && b.staged && b.ctas_per_sm == 1 &&
                     (long long)STAGE_SLOTS * slot * 8 <= STAGE_MAX_BYTES;
    EngineArgs a{b.dc, b.dk, b.d_cases + off, b.d_iters, b.d_err, stg ? (int)slot : 0};
    e = b.use_fast ? launch_engine_fast(a, K, cnt, s, b.l1_loads, b.threads, b.ctas_per_sm, stg ? 1 : 0)
                   : launch_engine_exact(a, K, cnt, s);
    }
    if (e != cudaSuccess) {
      cudaEventDestroy(fork);
      return fail(ACS_E_CUDA, std::string("engine launch (cluster ") + std::to_string(K) + "): " + cudaGetErrorString(e));
    }
    b.launches += 1;
    b.used |= cls >= 17 ? ACS_USED_CHIP : ACS_USED_CLUSTER;
    if (g) {
      CU(cudaEventRecord(b.ev[g], s));
      CU(cudaStreamWaitEvent(b.stream, b.ev[g], 0));
    }
  }
  cudaEventDestroy(fork);
  CU(cudaStreamSynchronize(b.stream));
  CU(cudaGetLastError());
  return ACS_OK;
}

// Per-routine calls run one routine's launches on case 0 with identity roles.  The driver's arrays
// cross PCIe in one copy each way through pinned staging, the control word travels with them, and the host
// waits once.
struct RoutineIO { int family, role; const double* in; double* out; };

long long routine_total(const Batch& b, const RoutineIO* io, int n) {
  long long t = 4;
  for (int q = 0; q < n; ++q) t += field_size(b, 0, io[q].family);
  return t;
}

int begin_routine(Batch& b, const RoutineIO* io, int n) {
  CaseCtl& k = b.hk[0];
  reset_roles(k);
  k.active = 1;
  k.scalars = 1;
  k.res_u = k.res_v = k.res_p = 0;
  if (routine_total(b, io, n) > STAGE_MAX) {
    int r = push_ctl(b);
    for (int q = 0; q < n && !r; ++q) r = put(b, 0, io[q].family, io[q].role, io[q].in);
    return r;
  }
  MoveList m{};
  for (int q = 0; q < n; ++q) add_move(b, m, 0, io[q].family, io[q].role);
  int r = stage_dev(b, (size_t)m.total + 4);
  if (!r) r = stage_host(b, (size_t)m.total + 4);
  if (r) return r;
  for (int q = 0; q < n; ++q) std::memcpy(b.h_stage + m.f[q].off, io[q].in, sizeof(double) * m.f[q].w * m.f[q].h);
  CU(cudaMemcpyAsync(b.d_stage, b.h_stage, sizeof(double) * m.total, cudaMemcpyHostToDevice, b.stream));
  move_to_case(m, b.d_stage, b.dk, k, b.stream);
  CU(cudaGetLastError());
  b.ctl_stale = false;
  return ACS_OK;
}

int end_routine(Batch& b, const RoutineIO* io, int n) {
  CaseCtl& k = b.hk[0];
  if (routine_total(b, io, n) > STAGE_MAX) {
    CU(cudaGetLastError());
    int r = 0;
    for (int q = 0; q < n && !r; ++q) r = get(b, 0, io[q].family, io[q].role, io[q].out);
    if (!r) r = pull_ctl(b);
    k.active = 0;
    if (!r) r = push_ctl(b);
    if (!r) CU(cudaStreamSynchronize(b.stream));
    return r;
  }
  MoveList m{};
  for (int q = 0; q < n; ++q) add_move(b, m, 0, io[q].family, io[q].role);
  int r = stage_dev(b, (size_t)m.total + 4);
  if (!r) r = stage_host(b, (size_t)m.total + 4);
  if (r) return r;
  move_from_case(m, b.d_stage, b.dk, b.stream);
  CU(cudaGetLastError());
  CU(cudaMemcpyAsync(b.h_stage, b.d_stage, sizeof(double) * (m.total + 3), cudaMemcpyDeviceToHost, b.stream));
  CU(cudaStreamSynchronize(b.stream));
  for (int q = 0; q < n; ++q) std::memcpy(io[q].out, b.h_stage + m.f[q].off, sizeof(double) * m.f[q].w * m.f[q].h);
  std::memcpy(&k.res_u, b.h_stage + m.total, 8);
  std::memcpy(&k.res_v, b.h_stage + m.total + 1, 8);
  std::memcpy(&k.res_p, b.h_stage + m.total + 2, 8);
  k.active = 0;
  return ACS_OK;
}

double bits_to_double(unsigned long long v) {
  double d;
  std::memcpy(&d, &v, 8);
  return d;
}

}  // namespace
}  // namespace acs

using acs::Batch;
using acs::fail;

struct acs_batch { Batch* b; };
struct acs_handle { Batch* b; };

extern "C" {

const char* acs_last_error(void) { return acs::g_err.c_str(); }
const char* acs_version(void) { return "acs-b200 1.0 (sm_100a, FP64)"; }

int acs_device_count(int* n) {
  if (!n) return acs::fail(ACS_E_ARG, "null");
  if (cudaGetDeviceCount(n) != cudaSuccess) {
    *n = 0;
    cudaGetLastError();
  }
  return ACS_OK;
}

int acs_batch_create(const acs_grid* grids, const acs_params* params, int n_cases, acs_batch** out) {
  if (!out) return acs::fail(ACS_E_ARG, "null out");
  Batch* b = nullptr;
  int r = acs::create_batch(grids, params, n_cases, &b);
  if (r) return r;
  *out = new acs_batch{b};
  return ACS_OK;
}

int acs_batch_destroy(acs_batch* h) {
  if (!h) return ACS_OK;
  delete h->b;
  delete h;
  return ACS_OK;
}

int acs_batch_set_stream(acs_batch* h, void* s) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  if (b.gexec) { cudaGraphExecDestroy(b.gexec); b.gexec = nullptr; }
  if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
  b.stage_moved = true;
  if (s) {
    if (b.own_stream) cudaStreamDestroy(b.stream);
    b.stream = (cudaStream_t)s;
    b.own_stream = false;
  }
  return ACS_OK;
}

int acs_batch_set_field(acs_batch* h, int c, int field, const double* host) {
  if (!h || !host) return acs::fail(ACS_E_ARG, "null argument");
  if (c < 0 || c >= h->b->n) return acs::fail(ACS_E_ARG, "case id out of range");
  return acs::upload_fields(*h->b, c, 1, &field, &host);
}

int acs_batch_set_fields(acs_batch* h, int c, int n, const int* fields, const double* const* host) {
  if (!h || !fields || !host || n < 1 || n > acs::MOVE_MAX) return acs::fail(ACS_E_ARG, "bad argument");
  if (c < 0 || c >= h->b->n) return acs::fail(ACS_E_ARG, "case id out of range");
  for (int q = 0; q < n; ++q)
    if (!host[q]) return acs::fail(ACS_E_ARG, "null argument");
  return acs::upload_fields(*h->b, c, n, fields, host);
}

int acs_batch_get_field(acs_batch* h, int c, int field, double* host) {
  if (!h || !host) return acs::fail(ACS_E_ARG, "null argument");
  if (c < 0 || c >= h->b->n) return acs::fail(ACS_E_ARG, "case id out of range");
  return acs::download_fields(*h->b, c, 1, &field, &host);
}

int acs_batch_get_fields(acs_batch* h, int c, int n, const int* fields, double* const* host) {
  if (!h || !fields || !host || n < 1 || n > acs::MOVE_MAX) return acs::fail(ACS_E_ARG, "bad argument");
  if (c < 0 || c >= h->b->n) return acs::fail(ACS_E_ARG, "case id out of range");
  for (int q = 0; q < n; ++q)
    if (!host[q]) return acs::fail(ACS_E_ARG, "null argument");
  return acs::download_fields(*h->b, c, n, fields, host);
}

int acs_batch_cell_fields(acs_batch* h, int c, double* u, double* v, double* vel_mag) {
  if (!h || !u || !v || !vel_mag) return acs::fail(ACS_E_ARG, "null argument");
  Batch& b = *h->b;
  if (c < 0 || c >= b.n) return acs::fail(ACS_E_ARG, "case id out of range");
  const acs::CaseDev& d = b.hc[c];
  // the results go through the T/C stage scratch of the cluster engine, which no step keeps
  double* out[3] = {d.S2[0], d.S2[1], d.S2[2]};
  CU(acs::launch_cell_fields(b.buf(c, 0, b.role_index(c, acs::FieldLoc{0, acs::R_PHYS})),
                             b.buf(c, 1, b.role_index(c, acs::FieldLoc{1, acs::R_PHYS})), d.nx, d.ny, d.pitch,
                             out[0], out[1], out[2], b.stream));
  double* host[3] = {u, v, vel_mag};
  for (int f = 0; f < 3; ++f)
    CU(cudaMemcpy2DAsync(host[f], (size_t)d.nx * 8, out[f], (size_t)d.pitch * 8, (size_t)d.nx * 8, d.ny,
                         cudaMemcpyDeviceToHost, b.stream));
  CU(cudaStreamSynchronize(b.stream));
  return ACS_OK;
}

int acs_batch_run(acs_batch* h, int n_steps, int* itc, int* iters, double* err, int* status) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  return acs::run_batch(*h->b, n_steps, itc, iters, err, status);
}

int acs_batch_ws_enable(acs_batch* h, int H, int W) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  for (int c = 0; c < b.n; ++c)
    if (b.hc[c].nx + 1 > W || b.hc[c].ny + 1 > H) return acs::fail(ACS_E_SIZE, "canvas smaller than (nx+1) x (ny+1)");
  if (H <= 0 || W <= 0 || (long long)H * W > (1LL << 30)) return acs::fail(ACS_E_ARG, "bad canvas size");
  if (!b.ws_pool) {
    size_t bytes = 0;
    for (int c = 0; c < b.n; ++c) bytes += 3 * acs::WS_FIELDS * acs::align_up(8 * b.hc[c].n_elems, 256);
    CU(cudaMalloc(&b.ws_pool, bytes));
    CU(cudaMemsetAsync(b.ws_pool, 0, bytes, b.stream));
    std::vector<acs::WsCase> hw(b.n);
    char* q = b.ws_pool;
    for (int c = 0; c < b.n; ++c)
      for (int f = 0; f < acs::WS_FIELDS; ++f) {
        hw[c].prev[f] = (double*)q; q += acs::align_up(8 * b.hc[c].n_elems, 256);
        hw[c].inc[f] = (double*)q; q += acs::align_up(8 * b.hc[c].n_elems, 256);
        hw[c].incp[f] = (double*)q; q += acs::align_up(8 * b.hc[c].n_elems, 256);
      }
    CU(cudaMalloc(&b.d_ws, sizeof(acs::WsCase) * b.n));
    CU(cudaMemcpyAsync(b.d_ws, hw.data(), sizeof(acs::WsCase) * b.n, cudaMemcpyHostToDevice, b.stream));
    CU(cudaMalloc(&b.d_ws_res, sizeof(unsigned long long) * 3 * b.n));
    CU(cudaMalloc(&b.d_ws_choice, sizeof(int) * b.n));
    CU(cudaMalloc(&b.d_ws_ss, sizeof(double) * acs::WS_OUT * b.n));
    CU(cudaMalloc(&b.d_ws_sc, sizeof(double) * acs::WS_OUT * b.n));
    CU(cudaMemsetAsync(b.d_ws_sc, 0, sizeof(double) * acs::WS_OUT * b.n, b.stream));
    CU(cudaStreamSynchronize(b.stream));
  }
  b.ws_H = H;
  b.ws_W = W;
  b.ws_has_prev = 0;
  b.ws_calls = 0;
  return ACS_OK;
}

int acs_batch_ws_features(acs_batch* h, float* X, float* inc_scale) {
  if (!h || !X) return acs::fail(ACS_E_ARG, "null argument");
  Batch& b = *h->b;
  if (!b.ws_pool) return acs::fail(ACS_E_STATE, "warm start not enabled");
  if (int r = acs::flush_ctl(b)) return r;
  acs::launch_ws_features(b.dc, b.dk, b.d_ws, b.n, b.ws_H, b.ws_W, b.ws_has_prev, b.d_ws_ss, b.d_ws_sc, X, inc_scale,
                          b.stream);
  CU(cudaGetLastError());
  b.ws_has_prev = 1;
  ++b.ws_calls;
  return ACS_OK;
}

int acs_batch_ws_target(acs_batch* h, float* T, float* Wt) {
  if (!h || !T || !Wt) return acs::fail(ACS_E_ARG, "null argument");
  Batch& b = *h->b;
  if (!b.ws_pool) return acs::fail(ACS_E_STATE, "warm start not enabled");
  if (int r = acs::flush_ctl(b)) return r;
  acs::launch_ws_target(b.dc, b.dk, b.d_ws, b.n, b.ws_H, b.ws_W, b.d_ws_sc, T, Wt, b.stream);
  CU(cudaGetLastError());
  return ACS_OK;
}

int acs_batch_set_start(acs_batch* h, const float* Y, int ldy, const float* scale, int policy, int* chosen,
                        double* res0) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  if (!b.ws_pool) return acs::fail(ACS_E_STATE, "warm start not enabled");
  if (policy < 0 || policy > 2) return acs::fail(ACS_E_ARG, "policy must be 0, 1 or 2");
  if (Y && (!scale || ldy < acs::WS_FIELDS)) return acs::fail(ACS_E_ARG, "Y needs scale and ldy >= 5");
  // the quadratic candidate needs two increments, i.e. three feature calls; before that, linear
  if (int r = acs::flush_ctl(b)) return r;
  const int order = (b.ws_order == 2 && b.ws_calls >= 3) ? 2 : 1;
  acs::launch_ws_start(b.dc, b.dk, b.d_ws, b.n, b.ws_H, b.ws_W, b.d_ws_sc, Y, ldy, scale, policy, order,
                       b.d_ws_res, b.d_ws_choice, b.stream);
  CU(cudaGetLastError());
  int r = acs::pull_ctl(b);  // the commit kernel set tau_dirty where the prediction was kept
  if (r) return r;
  if (chosen) CU(cudaMemcpy(chosen, b.d_ws_choice, sizeof(int) * b.n, cudaMemcpyDeviceToHost));
  if (res0) {
    std::vector<unsigned long long> bits(3 * b.n);
    CU(cudaMemcpy(bits.data(), b.d_ws_res, sizeof(unsigned long long) * 3 * b.n, cudaMemcpyDeviceToHost));
    for (int q = 0; q < 3 * b.n; ++q) res0[q] = acs::bits_to_double(bits[q]);
    if (!Y)
      for (int c = 0; c < b.n; ++c) res0[3 * c + 2] = std::nan("");
  }
  return ACS_OK;
}

int acs_batch_time_kernel(acs_batch* h, int kernel, int reps, double* ms_mean, long long* cells) {
  if (!h || !ms_mean || reps <= 0 || kernel < 0 || kernel > 6) return acs::fail(ACS_E_ARG, "bad argument");
  Batch& b = *h->b;
  if (kernel >= 5) {
    int r = acs::te_setup(b);
    if (r) return r;
  }
  std::vector<acs::CaseCtl> saved = b.hk;
  long long nc = 0;
  for (int c = 0; c < b.n; ++c) {
    b.hk[c].active = 1;
    b.hk[c].scalars = 1;
    const int nx = b.hc[c].nx, ny = b.hc[c].ny;
    nc += kernel == 0 ? (long long)(nx - 3) * (ny - 2) : kernel == 1 ? (long long)(nx - 2) * (ny - 3)
          : kernel >= 5 ? (long long)nx * ny : (long long)(nx - 2) * (ny - 2);
  }
  int r = acs::push_ctl(b);
  if (r) return r;
  cudaEvent_t e0, e1;
  CU(cudaEventCreate(&e0));
  CU(cudaEventCreate(&e1));
  auto one = [&]() { acs::launch_timed_kernel(b, kernel); };
  // the pressure kernels write pn (and the tile engine's P/T/C kernel T and C of role n_tau): keep
  // copies in stage scratch
  auto save = [&](bool back) -> int {
    for (int c = 0; c < b.n; ++c) {
      const acs::CaseDev& d = b.hc[c];
      const acs::CaseCtl& k = b.hk[c];
      double* live[3] = {d.P[k.rp[1]], d.T[k.rt[acs::R_NTAU]], d.C[k.rc[acs::R_NTAU]]};
      const int nf = kernel == 6 ? 3 : 1;
      for (int f = 0; f < nf; ++f) {
        double* a = back ? live[f] : d.S[1 + f];
        double* z = back ? d.S[1 + f] : live[f];
        CU(cudaMemcpyAsync(a, z, 8 * d.n_elems, cudaMemcpyDeviceToDevice, b.stream));
      }
    }
    return ACS_OK;
  };
  if (kernel == 2 || kernel == 6) {
    r = save(false);
    if (r) return r;
  }
  one();  // warm
  CU(cudaEventRecord(e0, b.stream));
  for (int i = 0; i < reps; ++i) one();
  CU(cudaEventRecord(e1, b.stream));
  CU(cudaEventSynchronize(e1));
  float ms = 0.f;
  CU(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  CU(cudaGetLastError());
  if (kernel == 2 || kernel == 6) {
    r = save(true);
    if (r) return r;
  }
  *ms_mean = ms / reps;
  if (cells) *cells = nc;
  for (int c = 0; c < b.n; ++c) {  // the residual slots were touched; restore the control words
    saved[c].res_u = saved[c].res_v = saved[c].res_p = 0;
  }
  b.hk = saved;
  r = acs::push_ctl(b);
  if (!r) CU(cudaStreamSynchronize(b.stream));
  return r;
}

int acs_batch_set_cluster_size(acs_batch* h, int c, int ctas) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  if (c < 0 || c >= b.n) return acs::fail(ACS_E_ARG, "case id out of range");
  if (ctas < 0 || ctas > 16) return acs::fail(ACS_E_ARG, "cluster size must be 0..16");
  if ((int)b.cluster_override.size() < b.n) b.cluster_override.assign(b.n, 0);
  b.cluster_override[c] = ctas;
  b.chip_k.clear();
  return ACS_OK;
}

int acs_batch_set_tolerance(acs_batch* h, int c, double eps) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  if (c < 0 || c >= b.n) return acs::fail(ACS_E_ARG, "case id out of range");
  if (!(eps > 0.0) || !std::isfinite(eps)) return acs::fail(ACS_E_ARG, "tolerance must be positive and finite");
  b.prm[c].eps = eps;
  b.hc[c].eps = eps;
  // stream-ordered: launches already queued keep the old value, the next ones see the new one
  CU(cudaMemcpyAsync(&b.dc[c].eps, &b.hc[c].eps, sizeof(double), cudaMemcpyHostToDevice, b.stream));
  CU(cudaStreamSynchronize(b.stream));
  return ACS_OK;
}

int acs_batch_set_option(acs_batch* h, int option, long long value) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  Batch& b = *h->b;
  switch (option) {
    case ACS_OPT_ENGINE: {
      if (value < 0 || value > 2) return acs::fail(ACS_E_ARG, "engine must be 0, 1 or 2");
      if (value == 2) {
        int r = acs::te_setup(b);
        if (r) return r;
      }
      if (b.engine != (int)value) {  // the captured loop body belongs to the previous engine
        if (b.gexec) { cudaGraphExecDestroy(b.gexec); b.gexec = nullptr; }
        if (b.graph) { cudaGraphDestroy(b.graph); b.graph = nullptr; }
        b.graph_steps = -1;
      }
      b.engine = (int)value;
      return ACS_OK;
    }
    case ACS_OPT_NODES_PER_CTA:
      if (value < 64 || value > (1 << 22)) return acs::fail(ACS_E_ARG, "nodes per CTA out of range");
      b.nodes_per_cta = (int)value;
      b.user_nodes = true;
      b.chip_k.clear();
      return ACS_OK;
    case ACS_OPT_L1_LOADS:
      b.l1_loads = value ? 1 : 0;
      return ACS_OK;
    case ACS_OPT_THREADS:
      if (value != 256 && value != 512) return acs::fail(ACS_E_ARG, "threads must be 256 or 512");
      b.threads = (int)value;
      return ACS_OK;
    case ACS_OPT_CTAS_PER_SM:
      if (value != 1 && value != 2) return acs::fail(ACS_E_ARG, "CTAs per SM must be 1 or 2");
      b.ctas_per_sm = (int)value;
      return ACS_OK;
    case ACS_OPT_STAGED:
      b.staged = value ? 1 : 0;
      return ACS_OK;
    case ACS_OPT_ON_CHIP:
      if (value != 0 && value != 1) return acs::fail(ACS_E_ARG, "on-chip option must be 0 or 1");
      b.on_chip = value == 0;
      b.chip_k.clear();
      return ACS_OK;
    case ACS_OPT_EXTRAP_ORDER:
      if (value != 1 && value != 2) return acs::fail(ACS_E_ARG, "extrapolation order must be 1 or 2");
      b.ws_order = (int)value;
      return ACS_OK;
  }
  return acs::fail(ACS_E_ARG, "unknown option");
}

int acs_set_option(acs_handle* h, int option, long long value) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  acs_batch tmp{h->b};
  return acs_batch_set_option(&tmp, option, value);
}

int acs_batch_launch_count(acs_batch* h, long long* n) {
  if (!h || !n) return acs::fail(ACS_E_ARG, "null");
  *n = h->b->launches;
  return ACS_OK;
}

int acs_batch_engines_used(acs_batch* h, int* used) {
  if (!h || !used) return acs::fail(ACS_E_ARG, "null");
  *used = h->b->used;
  return ACS_OK;
}

int acs_create(const acs_grid* g, const acs_params* p, acs_handle** out) {
  if (!out) return acs::fail(ACS_E_ARG, "null out");
  Batch* b = nullptr;
  int r = acs::create_batch(g, p, 1, &b);
  if (r) return r;
  *out = new acs_handle{b};
  return ACS_OK;
}

int acs_destroy(acs_handle* h) {
  if (!h) return ACS_OK;
  delete h->b;
  delete h;
  return ACS_OK;
}

int acs_set_stream(acs_handle* h, void* s) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  acs_batch tmp{h->b};
  return acs_batch_set_stream(&tmp, s);
}

int acs_set_field(acs_handle* h, int field, const double* host) {
  if (!h || !host) return acs::fail(ACS_E_ARG, "null argument");
  return acs::upload_fields(*h->b, 0, 1, &field, &host);
}

int acs_get_field(acs_handle* h, int field, double* host) {
  if (!h || !host) return acs::fail(ACS_E_ARG, "null argument");
  return acs::download_fields(*h->b, 0, 1, &field, &host);
}

int acs_cell_fields(acs_handle* h, double* u, double* v, double* vel_mag) {
  if (!h) return acs::fail(ACS_E_ARG, "null handle");
  acs_batch tmp{h->b};
  return acs_batch_cell_fields(&tmp, 0, u, v, vel_mag);
}

int acs_physical_steps(acs_handle* h, int n_steps, int* itc, int* iters, double* err, int* status) {
  if (!h || !itc) return acs::fail(ACS_E_ARG, "null argument");
  int st = 0;
  int r = acs::run_batch(*h->b, n_steps, itc, iters, err, &st);
  if (status) *status = st;
  return r;
}

int acs_launch_count(acs_handle* h, long long* n) {
  if (!h || !n) return acs::fail(ACS_E_ARG, "null");
  *n = h->b->launches;
  return ACS_OK;
}

int acs_engines_used(acs_handle* h, int* used) {
  if (!h || !used) return acs::fail(ACS_E_ARG, "null");
  *used = h->b->used;
  return ACS_OK;
}

#define NEED(x) if (!(x)) return acs::fail(ACS_E_ARG, "null argument: " #x)

int acs_solve_u(acs_handle* h, const double* um, const double* um_tau, double* vm_tau, const double* p,
                double* um_n_tau, double* residual_u) {
  NEED(h); NEED(um); NEED(um_tau); NEED(vm_tau); NEED(p); NEED(um_n_tau); NEED(residual_u);
  Batch& b = *h->b;
  const acs::RoutineIO in[4] = {{0, acs::R_PHYS, um, nullptr}, {0, acs::R_TAU, um_tau, nullptr},
                                {1, acs::R_TAU, vm_tau, nullptr}, {2, 1, p, nullptr}};
  const acs::RoutineIO out[2] = {{0, acs::R_NTAU, nullptr, um_n_tau}, {1, acs::R_TAU, nullptr, vm_tau}};
  int r = acs::refresh_flags(b);
  if (!r) r = acs::begin_routine(b, in, 4);
  if (r) return r;
  acs::seq_u(b);
  r = acs::end_routine(b, out, 2);
  if (!r) *residual_u = acs::bits_to_double(b.hk[0].res_u);
  return r;
}

int acs_solve_v(acs_handle* h, const double* vm, double* um_tau, const double* vm_tau, const double* p,
                const double* T, double* vm_n_tau, double* residual_v) {
  NEED(h); NEED(vm); NEED(um_tau); NEED(vm_tau); NEED(p); NEED(T); NEED(vm_n_tau); NEED(residual_v);
  Batch& b = *h->b;
  const acs::RoutineIO in[5] = {{1, acs::R_PHYS, vm, nullptr}, {0, acs::R_TAU, um_tau, nullptr},
                                {1, acs::R_TAU, vm_tau, nullptr}, {2, 1, p, nullptr}, {3, acs::R_PHYS, T, nullptr}};
  const acs::RoutineIO out[2] = {{1, acs::R_NTAU, nullptr, vm_n_tau}, {0, acs::R_TAU, nullptr, um_tau}};
  b.t_unity[0] = acs::all_ones(T, (size_t)b.hc[0].nx * b.hc[0].ny);
  int r = acs::refresh_flags(b);
  if (!r) r = acs::begin_routine(b, in, 5);
  if (r) return r;
  acs::seq_v(b);
  r = acs::end_routine(b, out, 2);
  if (!r) *residual_v = acs::bits_to_double(b.hk[0].res_v);
  return r;
}

int acs_solve_p(acs_handle* h, const double* p, const double* um_n_tau, const double* vm_n_tau, double* pn,
                double* residual_p) {
  NEED(h); NEED(p); NEED(um_n_tau); NEED(vm_n_tau); NEED(pn); NEED(residual_p);
  Batch& b = *h->b;
  const acs::RoutineIO in[3] = {{2, 0, p, nullptr}, {0, acs::R_NTAU, um_n_tau, nullptr}, {1, acs::R_NTAU, vm_n_tau, nullptr}};
  const acs::RoutineIO out[1] = {{2, 1, nullptr, pn}};
  int r = acs::begin_routine(b, in, 3);
  if (r) return r;
  acs::seq_p(b);
  r = acs::end_routine(b, out, 1);
  if (!r) *residual_p = acs::bits_to_double(b.hk[0].res_p);
  return r;
}

static int solve_scalar(acs_handle* h, bool is_c, const double* um_n_tau, const double* vm_n_tau, const double* Z,
                        double* Z_n_tau, const double* Z_tau) {
  NEED(h); NEED(um_n_tau); NEED(vm_n_tau); NEED(Z); NEED(Z_n_tau); NEED(Z_tau);
  Batch& b = *h->b;
  const int fam = is_c ? 4 : 3;
  const acs::RoutineIO in[4] = {{0, acs::R_NTAU, um_n_tau, nullptr}, {1, acs::R_NTAU, vm_n_tau, nullptr},
                                {fam, acs::R_PHYS, Z, nullptr}, {fam, acs::R_TAU, Z_tau, nullptr}};
  const acs::RoutineIO out[1] = {{fam, acs::R_NTAU, nullptr, Z_n_tau}};
  int r = acs::begin_routine(b, in, 4);
  if (r) return r;
  acs::seq_s(b, is_c);
  return acs::end_routine(b, out, 1);
}

int acs_solve_z(acs_handle* h, const double* um_n_tau, const double* vm_n_tau, const double* T, double* T_n_tau,
                const double* T_tau) {
  return solve_scalar(h, false, um_n_tau, vm_n_tau, T, T_n_tau, T_tau);
}

int acs_solve_c(acs_handle* h, const double* um_n_tau, const double* vm_n_tau, const double* Cc, double* C_n_tau,
                const double* C_tau) {
  return solve_scalar(h, true, um_n_tau, vm_n_tau, Cc, C_n_tau, C_tau);
}

}  // extern "C"
