// C-ABI of nemoh_b200 (include/nemoh_b200.h): context, device memory, and the
// per-frequency pipeline  assembly -> LU -> triangular solves -> S*sigma ->
// pressure/force integration, batched over frequencies and symmetry classes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdint>
#include <functional>
#include <initializer_list>
#include <utility>
#include <memory>
#include <mutex>
#include <numeric>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/nemoh_b200.h"
#include "assembly.cuh"
#include "fd_setup.h"
#include "kochin.cuh"
#include "preproc.cuh"
#include "freesurface.cuh"
#include "postproc.cuh"
#include "linalg.cuh"
#include "mixed.cuh"
#include "oz_gemm.cuh"

using namespace nb200;

namespace {

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~DevBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = 0;
  }
  // small buffers (descriptors, scratch) always grow with headroom
  cudaError_t ensure(size_t n, bool headroom = false) {
    return grow_alloc(&p, &bytes, n, headroom || n < (size_t(64) << 20));
  }
  template <class T>
  T* as() const { return reinterpret_cast<T*>(p); }
};

// pinned host staging (parameters and slot lists uploaded per assembly group)
struct HostBuf {
  void* p = nullptr;
  size_t bytes = 0;
  ~HostBuf() { release(); }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
  }
  // grows to twice the request: freeing pinned memory synchronizes the device,
  // so staging buffers of growing batches should grow rarely
  cudaError_t ensure(size_t n) {
    if (n <= bytes) return cudaSuccess;
    release();
    const size_t want = std::max<size_t>(2 * n, 4096);
    cudaError_t e = cudaMallocHost(&p, want);
    if (e == cudaSuccess) {
      bytes = want;
    } else {
      p = nullptr;
      cudaGetLastError();   // returned; not left for a later launch check
    }
    return e;
  }
  template <class T>
  T* as() const { return reinterpret_cast<T*>(p); }
};

struct Fail {
  int code;
  std::string msg;
};

// event that orders the context's stream against a caller's stream; released
// on every path out of the call, errors included
struct ScopedEvent {
  cudaEvent_t e = nullptr;
  ~ScopedEvent() {
    if (e) cudaEventDestroy(e);
  }
};

// A body kept resident on the device (nemoh_b200_add_body): its panel
// geometry, environment, generalised normals and its own NQ state (the
// reference's NQ, left by the body's last finite-depth solve).
struct BodyState {
  int np = 0, nfa = 0, nsymy = 0, nint = 0;
  double rho = 0, g = 0, depth = 0, zer = 0, gm = 0;
  int nq_state = 0;
  int ndof = 0;   // radiation DOFs of serving requests (nemoh_b200_set_body_dofs)
  DevBuf d_xyz, d_m, d_rec, d_rows, d_nds, d_dofs;
  std::vector<char> wide;   // oz_wide of the mesh
  // frequency-independent Rankine part per depth regime (0 deep water, 1
  // finite depth), kept with the resident body once evaluated
  DevBuf rk[2];
  bool rk_valid[2] = {false, false};
};

// a launch sequence seen before (key of its shapes and buffers) and, from its
// second sighting on, its captured graph
struct GraphEntry {
  unsigned long long key;
  cudaGraphExec_t exec;
};

}  // namespace

struct nemoh_ctx {
  int device = 0;
  int mode = NEMOH_B200_FP64;
  std::string err;
  cudaStream_t stream = nullptr;
  long long launches = 0;
  // tables
  double h_xr[TAB_IR + 2], h_xz[TAB_JZ + 2];
  DevBuf d_xr, d_xz, d_apd, d_lag, d_thr, d_status, d_gm;
  // mesh
  int np = 0, nfa = 0, nsymy = 0;
  double rho = 0, g = 0, depth = 0, zer = 0, gm = 0;
  double ro_eps2 = 0;   // largest x with sqrt(x) <= 1e-4
  DevBuf d_xyz, d_m, d_rec, d_rows;
  std::vector<char> wide;   // oz_wide of the mesh
  // per-call workspace
  DevBuf d_D, d_S, d_X, d_Y, d_diag, d_inv, d_oms, d_slots, d_nvel, d_nds, d_force, d_kochin, d_pre, d_fs, d_irf;
  HostBuf h_oms, h_slots;
  int cap_slots = 0, cap_nrhs = 0, cap_nfa = 0, cap_cls = 0;   // what ensure_batch last provided
  MixedWork mixed;
  Lanes lanes;               // side streams for groups of systems in the LU and triangular solves
  // pipelined batches: the first frequencies' FP32 LU on stream2 (with its own
  // lanes) while the main stream assembles the rest
  cudaStream_t stream2 = nullptr;
  Lanes lanes2;
  cudaEvent_t ev_pipe[2] = {nullptr, nullptr};
  int nq_state = 0;          // the reference's NQ, left by the last finite-depth solve
  double w_previous = -1.;   // factor cache key of solve_problem
  int cached_fd = 0, cached_nexp = 0;
  // Rankine part of the current mesh per depth regime; valid until the mesh
  // changes, re-evaluated at the start of every multi-frequency call
  DevBuf d_rk[2];
  bool rk_valid[2] = {false, false};
  size_t rk_body_bytes = 0;   // Rankine caches held by resident bodies
  bool lu64 = false;         // d_D holds FP64 LU factors (FP64 mode, or a mixed-mode fallback)
  float t_asm = 0, t_fac = 0, t_sol = 0, t_lu = 0;   // t_lu: the factorization alone, within t_fac
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  cudaEvent_t ev_lu[2] = {nullptr, nullptr};
  bool lu_timed = false;
  // resident bodies and the descriptions of the current ragged batch
  std::vector<std::unique_ptr<BodyState>> bodies;
  DevBuf d_roff, d_rord, d_smesh, d_items, d_bnvel, d_bforce, d_reqs;
  DevBuf d_froff, d_frord, d_fx, d_fy;   // partial FP64 fallback of a ragged batch
  DevBuf d_flow;                         // workspace of the FP64 dataflow sweep
  OzWork oz;                             // operand images of the FP64 LU's trailing updates
  long long tensor_updates = 0;          // FP64 trailing updates issued on the tensor cores so far
  long long fallback_systems = 0;         // systems re-solved with FP64 factors so far
  HostBuf h_rag, h_reqs;
  // CUDA graphs of cross-body batches (nemoh_b200_set_graphs)
  bool graph_mode = false;
  std::vector<GraphEntry> graphs;
  long long graph_captures = 0, graph_replays = 0;
};

#define CK(call)                                                                                 \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess)                                                                       \
      throw Fail{e_ == cudaErrorMemoryAllocation ? NEMOH_B200_ENOMEM : NEMOH_B200_ECUDA,         \
                 std::string(#call) + ": " + cudaGetErrorString(e_)};                            \
  } while (0)

#define LAUNCHED(ctx)                        \
  do {                                       \
    ++(ctx)->launches;                       \
    CK(cudaGetLastError());                  \
  } while (0)

static int guarded(nemoh_ctx* ctx, const std::function<void()>& f);

// Empty when every non-null pointer is device (or managed) memory that
// `device` can address; otherwise the reason. Run before any launch, so that a
// host buffer or another GPU's buffer handed to a *_device entry point is a
// status code instead of an illegal-address fault.
static std::string device_pointer_problem(int device, std::initializer_list<std::pair<const void*, const char*>> ptrs) {
  for (const auto& pn : ptrs) {
    if (!pn.first) continue;
    cudaPointerAttributes at{};
    const cudaError_t e = cudaPointerGetAttributes(&at, pn.first);
    if (e != cudaSuccess) {
      cudaGetLastError();   // clear the sticky-free error of the query
      return std::string(pn.second) + ": not a CUDA pointer (" + cudaGetErrorString(e) + ")";
    }
    if (at.type == cudaMemoryTypeManaged) continue;
    if (at.type != cudaMemoryTypeDevice)
      return std::string(pn.second) + (at.type == cudaMemoryTypeHost ? ": pinned host memory, device memory expected"
                                                                      : ": host memory, device memory expected");
    if (at.device != device)
      return std::string(pn.second) + ": memory of device " + std::to_string(at.device) + ", not of device " +
             std::to_string(device);
  }
  return std::string();
}

namespace {

const double kPI = 4. * std::atan(1.);

int ncls(const nemoh_ctx* c) { return c->nsymy ? 2 : 1; }

void check_status(nemoh_ctx* c) {
  int st = 0;
  CK(cudaMemcpyAsync(&st, c->d_status.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if (st) {
    CK(cudaMemsetAsync(c->d_status.p, 0, sizeof(int), c->stream));
    const char* m = st == ST_TC_TIMEOUT ? "tensor-core update timed out waiting on its operands"
                    : st == ST_SWEEP_TIMEOUT ? "triangular sweep timed out waiting on a solved block"
                    : st == ST_PIVOT ? "PIVOT INFERIEUR A 1.E-20 (GAUSSZ)"
                    : st == ST_PANEL_AREA ? "area of a panel is too small (GOMG)"
                    : st == ST_AKZ_UNDEFINED ? "AKZ > -1.5E-6: wave term undefined in the reference"
                                              : "device error";
    throw Fail{st, m};
  }
}

// Host-side setup of one frequency (SOLVE_BEM.f90:62-84 and the preambles of
// SOLVE_POTENTIAL_*_DIRECT). W is the reference's 2*PI/T.
// The mesh-dependent inputs of the per-frequency setup: gravity, depth, GM
// and the NQ state that the finite-depth solves leave (the context's current
// mesh, or a resident body).
struct Env {
  double g, depth, gm;
  int* nq_state;
};

void omega_params_env(const Env& e, double W, OmegaParams& om, bool advance_nq);

// depth regime of a frequency: finite depth unless the depth is infinite (0)
// or K h >= 20 (Solver/Core/SOLVE_BEM.f90:66, the deep-water branch)
bool finite_depth(const Env& e, double W) {
  const double kwave = W * W / e.g;
  return !((e.depth == 0.) || (kwave * e.depth >= 20));
}

void omega_params(nemoh_ctx* c, double W, OmegaParams& om, bool advance_nq) {
  omega_params_env(Env{c->g, c->depth, c->gm, &c->nq_state}, W, om, advance_nq);
}

void omega_params_env(const Env& env, double W, OmegaParams& om, bool advance_nq) {
  std::memset(&om, 0, sizeof om);
  om.w = W;
  om.h = env.depth;
  const bool fd = finite_depth(env, W);
  if (std::fabs(W) < 1.E-4) throw Fail{NEMOH_B200_EOMEGA, "ABS(WR) < 1.E-4"};
  double qq[MAX_NQ + 2], cq[MAX_NQ + 2];
  if (!fd) {
    om.fd = 0;
    om.k0 = W * W / env.g;
    const int n = theta_quadrature(om.k0 * env.gm, qq, cq);
    // NQ is not set on this path (SOLVE_BEM_INFD_DIRECT.f90:79): the
    // free-surface-panel theta sum runs NQ (left by the last finite-depth
    // solve) times over this path's weights, which are zero past n.
    om.nq = std::min(*env.nq_state, n);
    for (int i = 1; i <= om.nq; ++i) {
      om.cq[i] = cq[i];
      om.ct[i] = std::cos(qq[i]);
      om.st[i] = std::sin(qq[i]);
    }
  } else {
    om.fd = 1;
    const double AKH0 = W * W * env.depth / env.g;
    double AMH;
    int st = finite_depth_root(AKH0, &AMH);
    if (st) throw Fail{st, "ERREUR DANS LA RECHERCHE DE LA RACINE (X0)"};
    const double AKH = AMH * std::tanh(AMH);
    const double AM0 = AMH / env.depth;
    om.k0 = AM0;
    om.amh = AMH;
    const int n = theta_quadrature(AM0 * env.gm, qq, cq);
    if (advance_nq) *env.nq_state = n;   // NQ=N (SOLVE_BEM_FD_DIRECT.f90:99)
    om.nq = 0;                         // CQ is zero on this path (COMPUTE_GREEN_FD.f90:874)
    int nexp = 0;
    st = exponential_fit(AKH, AMH, &nexp, om.ambda, om.ar);
    if (st) throw Fail{st, st == ST_LISC ? "LISC: positive exponent" : "exponential fit failed"};
    om.nexp = nexp;
    om.ambda[nexp + 1] = 0.;
    om.ar[nexp + 1] = 2.;
    const double A = (AMH + AKH) * (AMH + AKH) / (env.depth * (AMH * AMH - AKH * AKH + AKH));
    const double ADPI2 = -A / (8. * kPI * kPI), ADPI = -A / (8 * kPI);
    om.coe1 = ADPI2 / AM0;
    om.coe2 = ADPI / AM0;
    om.coe3 = ADPI2;
    om.coe4 = ADPI;
  }
}

// Mesh upload and panel geometry (INITIALIZE + PRE_PROC_MESH: GOMG, ZER and
// GM): nodes and connectivity to the device, GOMG there, ZER on the host
// (PREPARE_MESH.f90:58-69: the largest pairwise |dx| is max - min), GM by a
// device reduction. Synchronises the context's stream.
void upload_geometry(nemoh_ctx* c, int np, int nfa, int nsymy, const double* xyz, const int* m1234, DevBuf& d_xyz,
                     DevBuf& d_m, DevBuf& d_rec, DevBuf& d_rows, double& zer, double& gm, std::vector<char>& wide) {
  for (int i = 0; i < 4 * nfa; ++i)
    if (m1234[i] < 1 || m1234[i] > np) throw Fail{NEMOH_B200_EINVAL, "panel node index out of range"};
  double xmin = xyz[0], xmax = xyz[0], ymin = xyz[1], ymax = xyz[1], yabs = 0;
  for (int i = 0; i < np; ++i) {
    xmin = std::min(xmin, xyz[3 * i]);
    xmax = std::max(xmax, xyz[3 * i]);
    ymin = std::min(ymin, xyz[3 * i + 1]);
    ymax = std::max(ymax, xyz[3 * i + 1]);
    yabs = std::max(yabs, std::fabs(xyz[3 * i + 1]));
  }
  const double GL0 = xmax - xmin;
  const double BL = nsymy ? 2. * yabs : ymax - ymin;
  zer = -1.E-5 * std::max(GL0, BL);
  wide = oz_wide(nfa, xyz, m1234);
  CK(d_xyz.ensure(sizeof(double) * 3 * np));
  CK(d_m.ensure(sizeof(int) * 4 * nfa));
  CK(d_rec.ensure(sizeof(PanelRec) * nfa));
  CK(d_rows.ensure(sizeof(double) * 6 * nfa));
  CK(cudaMemcpyAsync(d_xyz.p, xyz, sizeof(double) * 3 * np, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(d_m.p, m1234, sizeof(int) * 4 * nfa, cudaMemcpyHostToDevice, c->stream));
  gomg_kernel<<<(nfa + 127) / 128, 128, 0, c->stream>>>(nfa, d_xyz.as<double>(), d_m.as<int>(), d_rec.as<PanelRec>(),
                                                       d_rows.as<double>(), c->d_status.as<int>());
  LAUNCHED(c);
  CK(cudaMemsetAsync(c->d_gm.p, 0, sizeof(unsigned long long), c->stream));
  gm_kernel<<<592, 256, 0, c->stream>>>(np, nsymy, d_xyz.as<double>(), c->d_gm.as<unsigned long long>());
  LAUNCHED(c);
  unsigned long long bits = 0;
  CK(cudaMemcpyAsync(&bits, c->d_gm.p, sizeof bits, cudaMemcpyDeviceToHost, c->stream));
  check_status(c);
  std::memcpy(&gm, &bits, sizeof bits);
}

// capacity: frequencies per device batch
int batch_capacity(nemoh_ctx* c, int nrhs, int want) {
  if (want <= c->cap_slots && nrhs <= c->cap_nrhs && c->nfa == c->cap_nfa && ncls(c) == c->cap_cls)
    return want;   // buffers already fit (same mesh size as the last batch)
  // a mixed batch grows into the room of an earlier FP64 fallback's images
  if (c->mode == NEMOH_B200_MIXED) c->oz.release();
  size_t fr = 0, tot = 0;
  CK(cudaMemGetInfo(&fr, &tot));
  const size_t N = c->nfa, cls = ncls(c);
  size_t per = (2 * cls * N * N + 2 * cls * N * (size_t)std::max(nrhs, 1)) * sizeof(double2) + sizeof(OmegaParams) +
               cls * DIAG_SCRATCH * sizeof(double2) + cls * ((N + TB - 1) / TB) * 2 * TB * TB * sizeof(double2);
  if (c->mode == NEMOH_B200_MIXED) per += mixed_bytes_per_system(N) * cls;
  else if (N > LU_OUTER) per += oz_bytes_per_system(N) * cls;
  // existing buffers count as available
  size_t have = c->d_D.bytes + c->d_S.bytes + c->d_X.bytes + c->d_Y.bytes + c->d_inv.bytes + c->mixed.bytes() +
                c->oz.bytes();
  size_t budget = (size_t)((fr + have) * 0.8);
  // room for the Rankine caches of both depth regimes that are not allocated yet
  for (int r = 0; r < 2; ++r) {
    const size_t need = cls * N * N * sizeof(double2);
    if (c->d_rk[r].bytes < need) budget -= std::min(budget, need);
  }
  int cap = (int)std::max<size_t>(1, budget / per);
  return std::min(cap, want);
}

void ensure_batch(nemoh_ctx* c, int slots, int nrhs) {
  const size_t N = c->nfa, cls = ncls(c);
  const size_t mats = (size_t)slots * cls * N * N * sizeof(double2);
  CK(c->d_D.ensure(mats));
  CK(c->d_S.ensure(mats));
  const size_t rhs = (size_t)slots * cls * N * std::max(nrhs, 1) * sizeof(double2);
  CK(c->d_X.ensure(rhs));
  CK(c->d_Y.ensure(rhs));
  CK(c->d_diag.ensure((size_t)slots * cls * DIAG_SCRATCH * sizeof(double2)));
  if (c->mode == NEMOH_B200_FP64)
    CK(c->d_inv.ensure((size_t)slots * cls * ((N + TB - 1) / TB) * 2 * TB * TB * sizeof(double2)));
  CK(c->d_oms.ensure((size_t)slots * sizeof(OmegaParams)));
  CK(c->d_slots.ensure((size_t)slots * sizeof(int)));
  CK(c->h_oms.ensure((size_t)slots * sizeof(OmegaParams)));
  CK(c->h_slots.ensure((size_t)slots * sizeof(int)));
  if (c->mode == NEMOH_B200_MIXED) CK(c->mixed.ensure(slots * (int)cls, (int)N, std::max(nrhs, 1)));
  if ((int)N != c->cap_nfa || (int)cls != c->cap_cls) {   // capacities count slots of this mesh size
    c->cap_slots = c->cap_nrhs = 0;
    c->cap_nfa = (int)N;
    c->cap_cls = (int)cls;
  }
  c->cap_slots = std::max(c->cap_slots, slots);
  c->cap_nrhs = std::max(c->cap_nrhs, std::max(nrhs, 1));
}

GreenCtx green_ctx(nemoh_ctx* c) {
  GreenCtx g;
  g.xr = c->d_xr.as<double>();
  g.xz = c->d_xz.as<double>();
  g.apd = c->d_apd.as<double4>();
  g.xlag = c->d_lag.as<double4>();
  g.zlag = c->d_lag.as<double4>() + 2 * (TAB_IR + 2);
  g.thr = c->d_thr.as<StencilThresholds>();
  g.zer = c->zer;
  g.nsymy = c->nsymy;
  g.status = c->d_status.as<int>();
  g.ro_eps2 = c->ro_eps2;
  return g;
}

// Upload the parameters of slots [s0, s1) (already in c->h_oms) and assemble
// those frequencies: deep-water slots first, then finite-depth ones. Ragged
// batches pass each slot's mesh on the device (dmesh) and its order on the
// host (host_n); each launch's grid is then sized by its largest slot.
// One assembly group: its slots [s0, s1) ordered deep water first, and the
// launch shape of each depth regime.
struct AsmGroup {
  int s0, s1, ninfd, nfd, n_infd, n_fd;
  bool slot_rk_infd = false, slot_rk_fd = false;   // ragged: a slot of the regime has no Rankine cache
};

// uploads the parameters and slot order of slots [s0, s1) (already in c->h_oms);
// host_rk (ragged) flags the slots whose body has a Rankine cache
AsmGroup assemble_upload(nemoh_ctx* c, int s0, int s1, const int* host_n, const char* host_rk = nullptr) {
  const int N = c->nfa;
  const OmegaParams* hom = c->h_oms.as<OmegaParams>();
  int* hs = c->h_slots.as<int>() + s0;
  AsmGroup ag{s0, s1, 0, 0, 0, 0};
  for (int s = s0; s < s1; ++s)
    if (!hom[s].fd) {
      hs[ag.ninfd++] = s;
      ag.n_infd = std::max(ag.n_infd, host_n ? host_n[s] : N);
      ag.slot_rk_infd |= !(host_rk && host_rk[s]);
    }
  for (int s = s0; s < s1; ++s)
    if (hom[s].fd) {
      hs[ag.ninfd + ag.nfd++] = s;
      ag.n_fd = std::max(ag.n_fd, host_n ? host_n[s] : N);
      ag.slot_rk_fd |= !(host_rk && host_rk[s]);
    }
  CK(cudaMemcpyAsync(c->d_oms.as<OmegaParams>() + s0, hom + s0, (size_t)(s1 - s0) * sizeof(OmegaParams),
                     cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->d_slots.as<int>() + s0, hs, (size_t)(s1 - s0) * sizeof(int), cudaMemcpyHostToDevice,
                     c->stream));
  return ag;
}

void assemble_launch(nemoh_ctx* c, const AsmGroup& ag, const SlotMesh* dmesh);

void assemble_range(nemoh_ctx* c, int s0, int s1, const SlotMesh* dmesh = nullptr, const int* host_n = nullptr,
                    const char* host_rk = nullptr) {
  assemble_launch(c, assemble_upload(c, s0, s1, host_n, host_rk), dmesh);
}

// The Rankine part of one mesh in one depth regime into buf (evaluated once,
// then kept while `valid` holds); returns the cache.
const double2* rankine_cache(nemoh_ctx* c, GreenCtx g, const PanelRec* rec, const double* rows, int n, int nsymy,
                             double depth, bool fd, DevBuf& buf, bool& valid) {
  if (valid) return buf.as<double2>();
  const size_t nn = (size_t)n * n;
  CK(buf.ensure((nsymy + 1) * nn * sizeof(double2)));
  g.nsymy = nsymy;
  const dim3 grid((n + ASM_ROWS - 1) / ASM_ROWS, (n + ASM_TJ - 1) / ASM_TJ);
  if (fd)
    rankine_cache_kernel<true><<<grid, ASM_ROWS, 0, c->stream>>>(g, 2. * depth, rec, rows, n, buf.as<double2>());
  else
    rankine_cache_kernel<false><<<grid, ASM_ROWS, 0, c->stream>>>(g, 0., rec, rows, n, buf.as<double2>());
  LAUNCHED(c);
  valid = true;
  return buf.as<double2>();
}

// the current mesh's cache of one regime
const double2* mesh_rankine(nemoh_ctx* c, bool fd) {
  return rankine_cache(c, green_ctx(c), c->d_rec.as<PanelRec>(), c->d_rows.as<double>(), c->nfa, c->nsymy, c->depth,
                       fd, c->d_rk[fd], c->rk_valid[fd]);
}

// The Rankine and wave passes of one group (reads only device buffers). The
// current mesh reads its Rankine caches; a ragged group (dmesh) reads each
// body's cache through its slot description, and runs the per-slot Rankine
// pass only when a slot of the regime has none (ag.slot_rk_*).
void assemble_launch(nemoh_ctx* c, const AsmGroup& ag, const SlotMesh* dmesh) {
  const int N = c->nfa, cls = ncls(c);
  const int s0 = ag.s0, ninfd = ag.ninfd, nfd = ag.nfd, n_infd = ag.n_infd, n_fd = ag.n_fd;
  GreenCtx g = green_ctx(c);
  const long long NN = (long long)N * N;
  AsmOut o{c->d_D.as<double2>(), c->d_S.as<double2>(), cls * NN};
  // the mixed LU factors an FP32 copy of D: the wave pass writes it with the final D
  if (c->mode == NEMOH_B200_MIXED) o.d32 = c->mixed.lu;
  dim3 blk(ASM_ROWS);
  const OmegaParams* dom = c->d_oms.as<OmegaParams>();
  const PanelRec* rec = c->d_rec.as<PanelRec>();
  const double* rows = c->d_rows.as<double>();
  const int* ds = c->d_slots.as<int>() + s0;
  if (ninfd) {
    const int n = n_infd;
    if (!dmesh) {
      o.rk = mesh_rankine(c, false);
    } else if (ag.slot_rk_infd) {
      dim3 grid((n + ASM_ROWS - 1) / ASM_ROWS, (n + ASM_TJ - 1) / ASM_TJ, (unsigned)ninfd);
      rankine_kernel<false><<<grid, blk, 0, c->stream>>>(g, dom, ds, rec, rows, n, o, dmesh);
      LAUNCHED(c);
    }
    const unsigned wt = (n + WS_T - 1) / WS_T;
    wave_sym_kernel<false><<<dim3(wt * (wt + 1) / 2, 1, (unsigned)ninfd), WS_THREADS, 0, c->stream>>>(g, dom, ds, rec,
                                                                                                      n, o, dmesh);
    LAUNCHED(c);
  }
  if (nfd) {
    const int n = n_fd;
    if (!dmesh) {
      o.rk = mesh_rankine(c, true);
    } else if (ag.slot_rk_fd) {
      dim3 grid((n + ASM_ROWS - 1) / ASM_ROWS, (n + ASM_TJ - 1) / ASM_TJ, (unsigned)nfd);
      rankine_kernel<true><<<grid, blk, 0, c->stream>>>(g, dom, ds + ninfd, rec, rows, n, o, dmesh);
      LAUNCHED(c);
    }
    const unsigned wt = (n + WS_T - 1) / WS_T;
    wave_sym_kernel<true><<<dim3(wt * (wt + 1) / 2, 1, (unsigned)nfd), WS_THREADS, 0, c->stream>>>(
        g, dom, ds + ninfd, rec, n, o, dmesh);
    LAUNCHED(c);
  }
}

// The systems of a batch: nsys systems of order n (uniform, the current mesh),
// or of orders up to n described by rg (ragged, several bodies). images: the
// context holds the operand images of their FP64 updates (fp64_images, once per
// batch and before a launch sequence that may be captured). wide: the panels whose
// updates stay on the FP64 pipe (oz_wide, for any of the systems).
struct Shape {
  int n;
  Ragged rg;
  std::vector<char> wide;
  bool images = false;
  bool wide_panel(int k0) const { return k0 / LU_OUTER < (int)wide.size() && wide[k0 / LU_OUTER]; }
};
Shape uniform_shape(const nemoh_ctx* c) { return Shape{c->nfa, Ragged(), c->wide}; }

// sum of f(order - k) over the batch's systems that reach beyond column k (a
// ragged batch's orders decrease)
template <class F>
double trailing_sum(const Shape& sh, int nsys, int k, F f) {
  if (!sh.rg.host_ord) return k < sh.n ? nsys * (double)f(sh.n - k) : 0.;
  double t = 0.;
  for (int s = 0; s < nsys && sh.rg.host_ord[s] > k; ++s) t += f(sh.rg.host_ord[s] - k);
  return t;
}

Batch dbatch(nemoh_ctx* c, const Shape& sh) {
  // FP64 keeps the per-step row-strip updates (FP64 GEMM tiles beat the fused strip solve there)
  return make_batch<double2>(c->d_D.as<double2>(), sh.n, c->d_diag.as<double2>(), nullptr, sh.rg);
}

// Operand images of the FP64 LU's tensor-core updates (oz_gemm.cuh) for nsys
// systems of order up to sh.n; false where there is no trailing update or no
// room for them (the FP64 fallback of a mixed batch that fills the device): the
// update then runs on the FP64 pipe.
bool fp64_images(nemoh_ctx* c, int nsys, const Shape& sh, bool headroom = false) {
  if (!tc_enabled() || trailing_sum(sh, nsys, LU_OUTER, [](double rest) { return rest * rest; }) < OZ_MIN_ENTRIES)
    return false;
  bool any = false;
  for (int k0 = 0; k0 + LU_OUTER < sh.n; k0 += LU_OUTER) any |= !sh.wide_panel(k0);
  if (!any) return false;
  if (c->oz.grows(nsys, sh.n)) {   // images that can't grow stay for the batches that they are large enough for
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    const size_t need = nsys * oz_bytes_per_system(sh.n), room = fr + c->oz.bytes();
    if (need > room) return false;
    headroom = headroom && need + need / 4 <= room;
  }
  return c->oz.ensure(nsys, sh.n, headroom) == cudaSuccess;
}

void factor_fp64(nemoh_ctx* c, int nsys, const Shape& sh) {
  Batch b = dbatch(c, sh);
  const int N = sh.n;
  const bool images = sh.images;
  // Panel pairs are merged where the update fills the device: after the first
  // panel only the next panel's columns and rows are updated, the rest of the
  // trailing matrix takes both panels' products in the next panel's update, so
  // its bulk is read and written once per pair. deferred: the groups (by their
  // first system) whose last panel's bulk is still to come.
  std::map<int, bool> deferred;
  static std::atomic<unsigned long long> attr{0};
  once_per_device(attr, [] {
    CK(cudaFuncSetAttribute(zgemm_update_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            zgemm_smem<double2>()));
  });
  lu_two_level<double2>(
      b, nsys, c->d_status.as<int>(), c->stream, c->launches,
      [&](Batch bg, int ns, cudaStream_t sg, int s0, int k0, int kend) {
        bool& late = deferred[s0];
        const bool tensor =
            late || (images && !sh.wide_panel(k0) &&
                     trailing_sum(sh, nsys, kend, [](double rest) { return rest * rest; }) >= OZ_MIN_ENTRIES);
        if (!tensor) {
          zgemm_update<double2>(bg, k0, kend - k0, Rect{kend, bg.n, kend, bg.n}, ns, sg);
          ++c->launches;
          return;
        }
        const int set = (k0 / LU_OUTER) & 1;
        const OzStride st = oz_stride(c->oz);
        const OzSet cur = oz_set(c->oz, set, s0);
        int* status = c->d_status.as<int>();
        ++c->tensor_updates;
        oz_prep(cur, st, bg, k0, ns, sg, c->launches);
        if (late) {
          oz_apply(cur, oz_set(c->oz, set ^ 1, s0), st, bg, k0, ns, sg, c->launches, status, false);
          late = false;
        } else {
          late = kend + LU_OUTER < bg.n && !sh.wide_panel(kend) &&
                 trailing_sum(sh, nsys, kend, oz_tiles) >= OZ_MERGE_TILES;
          oz_apply(cur, OzSet(), st, bg, k0, ns, sg, c->launches, status, late);
        }
      },
      &c->lanes, sh.rg.host_ord);
  CK(cudaGetLastError());
  static std::atomic<unsigned long long> attr2{0};
  once_per_device(attr2, [] {
    CK(cudaFuncSetAttribute(inv_diag_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            inv_diag_smem<double2>()));
  });
  const int nblk = (N + TB - 1) / TB;
  inv_diag_kernel<double2><<<dim3(nblk, 1, nsys), INV_THREADS, inv_diag_smem<double2>(), c->stream>>>(
      b, c->d_inv.as<double2>(), nblk);
  LAUNCHED(c);
}

// workspace of an FP64 dataflow sweep over nsys systems of order up to n
SweepSync fp64_sync(nemoh_ctx* c, int nsys, int n) {
  CK(c->d_flow.ensure(2 * flow_ws_ints(nsys, (n + TB - 1) / TB) * sizeof(int), true));
  return SweepSync{c->d_flow.as<int>(), c->d_status.as<int>()};
}

// solve the factored systems for the right-hand sides in X (result in X)
void trsm_fp64(nemoh_ctx* c, int nsys, int nrhs, const Shape& sh) {
  const SweepSync sync = fp64_sync(c, nsys, sh.n);
  CK(trsm_sweep_tuned<double2>(dbatch(c, sh), c->d_inv.as<double2>(), c->d_X.as<double2>(), c->d_Y.as<double2>(), nsys,
                               nrhs, c->stream, c->launches, nullptr, sync));
  CK(cudaGetLastError());
}

// Mixed precision: refine the FP32-LU solution; when refinement does not
// reach the tolerance (the FP32 factors are too inaccurate, as near an
// irregular frequency where the system is close to singular) the batch is
// factored again in FP64 on the device and solved from the original
// right-hand sides, which the refinement kept in mixed.b. d_D then holds the
// FP64 factors (lu64) instead of the matrix.
void mixed_fallback(nemoh_ctx* c, int nsys, int nrhs, Shape sh) {
  MixedWork& w = c->mixed;
  const size_t N = sh.n;
  CK(c->d_inv.ensure((size_t)nsys * ((N + TB - 1) / TB) * 2 * TB * TB * sizeof(double2)));
  CK(cudaMemcpyAsync(c->d_X.p, w.b, (size_t)nsys * N * nrhs * sizeof(double2), cudaMemcpyDeviceToDevice, c->stream));
  sh.images = fp64_images(c, nsys, sh);
  factor_fp64(c, nsys, sh);
  trsm_fp64(c, nsys, nrhs, sh);
  c->lu64 = true;
  w.last_iterations = -1;
  ++w.fallbacks;
}

// Ragged batches (many bodies): only the systems whose refinement missed the
// tolerance are factored again in FP64 (their matrices are still in d_D; the
// FP32 LU worked on its copy) and solved from their kept right-hand sides;
// the others keep their refined solutions.
void mixed_fallback_ragged(nemoh_ctx* c, int nsys, int nrhs, const Shape& sh) {
  MixedWork& w = c->mixed;
  const int nv = nsys * nrhs;
  std::vector<unsigned long long> h(2 * (size_t)nv);
  CK(cudaMemcpyAsync(h.data(), w.norms, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  std::vector<int> bad;
  for (int s = 0; s < nsys; ++s) {
    bool fail = false;
    for (int p = 0; p < nrhs; ++p) {
      double rn, bn;
      std::memcpy(&rn, &h[(size_t)s * nrhs + p], 8);
      std::memcpy(&bn, &h[(size_t)nv + (size_t)s * nrhs + p], 8);
      const double r = bn > 0 ? rn / bn : rn;
      fail = fail || !(r <= REFINE_TOL);
    }
    if (fail) bad.push_back(s);
  }
  if (bad.empty() || (int)bad.size() == nsys) {
    mixed_fallback(c, nsys, nrhs, sh);
    return;
  }
  const int nf = (int)bad.size();
  std::vector<long long> off_f(nf);
  std::vector<int> ord_f(nf);
  for (int j = 0; j < nf; ++j) {
    off_f[j] = sh.rg.host_off[bad[j]];
    ord_f[j] = sh.rg.host_ord[bad[j]];
  }
  const size_t N = sh.n, xs = N * nrhs, xf = (size_t)ord_f[0] * nrhs;
  CK(c->d_froff.ensure(nf * sizeof(long long)));
  CK(c->d_frord.ensure(nf * sizeof(int)));
  CK(c->d_fx.ensure((size_t)nf * xf * sizeof(double2), true));
  CK(c->d_fy.ensure((size_t)nf * xf * sizeof(double2), true));
  CK(c->d_inv.ensure((size_t)nf * ((ord_f[0] + TB - 1) / TB) * 2 * TB * TB * sizeof(double2)));
  CK(cudaMemcpyAsync(c->d_froff.p, off_f.data(), nf * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->d_frord.p, ord_f.data(), nf * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  double2* fx = c->d_fx.as<double2>();
  double2* X = c->d_X.as<double2>();
  for (int j = 0; j < nf; ++j)   // a system's right-hand sides: ord x nrhs, contiguous
    CK(cudaMemcpyAsync(fx + j * xf, w.b + bad[j] * xs, (size_t)ord_f[j] * nrhs * sizeof(double2),
                       cudaMemcpyDeviceToDevice, c->stream));
  Shape shf{ord_f[0], Ragged{c->d_froff.as<long long>(), c->d_frord.as<int>(), ord_f.data(), off_f.data()}, sh.wide};
  shf.images = fp64_images(c, nf, shf);
  factor_fp64(c, nf, shf);
  const SweepSync sync = fp64_sync(c, nf, shf.n);
  CK(trsm_sweep_tuned<double2>(dbatch(c, shf), c->d_inv.as<double2>(), fx, c->d_fy.as<double2>(), nf, nrhs,
                               c->stream, c->launches, nullptr, sync));
  for (int j = 0; j < nf; ++j)
    CK(cudaMemcpyAsync(X + bad[j] * xs, fx + j * xf, (size_t)ord_f[j] * nrhs * sizeof(double2),
                       cudaMemcpyDeviceToDevice, c->stream));
  w.last_iterations = -1;
  w.fallbacks += 1;
  c->fallback_systems += nf;
}

void mixed_solve(nemoh_ctx* c, int nsys, int nrhs, const Shape& sh) {
  MixedWork& w = c->mixed;
  mixed_solve_refine(w, c->d_D.as<double2>(), sh.n, nsys, c->d_X.as<double2>(), c->d_Y.as<double2>(), nrhs,
                     c->stream, c->launches, sh.rg);
  CK(cudaGetLastError());
  if (w.last_residual <= REFINE_TOL) return;
  if (sh.rg.host_off) mixed_fallback_ragged(c, nsys, nrhs, sh);
  else mixed_fallback(c, nsys, nrhs, sh);
}

// pre (mixed precision, uniform batches): systems [0, pre) were factored on
// stream2, whose event ev_pipe[1] the refinement waits for
void factor_and_solve(nemoh_ctx* c, int nsys, int nrhs, bool have_rhs, Shape sh, int pre = 0) {
  c->lu64 = c->mode == NEMOH_B200_FP64;
  CK(cudaEventRecord(c->ev_lu[0], c->stream));
  if (c->mode == NEMOH_B200_MIXED) {
    mixed_factor(c->mixed, c->d_D.as<double2>(), sh.n, nsys - pre, c->d_status.as<int>(), c->stream, c->launches,
                 &c->lanes, /*have_f32=*/true, sh.rg, -1, pre);
    if (pre) CK(cudaStreamWaitEvent(c->stream, c->ev_pipe[1], 0));
    CK(cudaGetLastError());
    CK(cudaEventRecord(c->ev_lu[1], c->stream));
    if (have_rhs) mixed_solve(c, nsys, nrhs, sh);
  } else {
    if (!sh.rg.host_off) sh.images = fp64_images(c, nsys, sh);   // a ragged batch has them with its buffers
    factor_fp64(c, nsys, sh);
    CK(cudaEventRecord(c->ev_lu[1], c->stream));
    if (have_rhs) trsm_fp64(c, nsys, nrhs, sh);
  }
  c->lu_timed = true;
}

// adds the factorization's share of the last factor_and_solve (after a sync)
void add_lu_time(nemoh_ctx* c) {
  if (!c->lu_timed) return;
  float ms = 0;
  CK(cudaEventElapsedTime(&ms, c->ev_lu[0], c->ev_lu[1]));
  c->t_lu += ms;
  c->lu_timed = false;
}

void potential(nemoh_ctx* c, int nsys, int nrhs, const Shape& sh) {
  const int N = sh.n;
  const long long xs = (long long)N * nrhs;
  const Batch s = make_batch<double2>(c->d_S.as<double2>(), N, nullptr, nullptr, sh.rg);
  CK(cudaMemsetAsync(c->d_Y.p, 0, (size_t)nsys * xs * sizeof(double2), c->stream));
  matvec_acc(s, c->d_X.as<double2>(), xs, c->d_Y.as<double2>(), xs, nrhs, nsys, 1.0, c->stream);
  LAUNCHED(c);
}

// frequencies whose host setup is done before their assembly is launched
constexpr int ASM_GROUP = 8;

// Pipelined batch (mixed precision, off unless NEMOH_B200_PIPELINE gives the
// percentage of the batch): the FP32 LU of the first frequencies runs on
// stream2 (highest priority) while the main stream assembles the rest.
// Returns the number of frequencies factored early (0: no pipeline).
// Measured on the barge workload it is slower (76.3 against 74.0 ms per
// 40-frequency step at 50%; the two-sphere step 389 against 386 ms): the
// assembly keeps every SM's FP64 pipe busy, so the LU's CTAs only take time
// from it, and the LU of each half alone is as latency-bound as the whole.
int pipeline_split(const nemoh_ctx* c, int nw) {
  static const int pct = [] {
    const char* e = std::getenv("NEMOH_B200_PIPELINE");
    const int v = e ? std::atoi(e) : 0;
    return std::max(0, std::min(90, v));
  }();
  if (c->mode != NEMOH_B200_MIXED || nw < 2 || pct == 0) return 0;
  return std::max(1, std::min(nw - 1, nw * pct / 100));
}

// shared by the host and device-pointer batched entry points
void solve_frequencies_impl(nemoh_ctx* c, int nomega, const double* omegas, int nrhs, const double2* nvel_d, int nint,
                            const double* nds_d, double2* force_d) {
  if (!c->nfa) throw Fail{NEMOH_B200_EINVAL, "no mesh"};
  if (nrhs < 1 || nrhs > MAX_RHS) throw Fail{NEMOH_B200_ECAPACITY, "nrhs must be in 1..16"};
  const int N = c->nfa, cls = ncls(c);
  const int cap = batch_capacity(c, nrhs, nomega);
  ensure_batch(c, cap, nrhs);
  c->t_asm = c->t_fac = c->t_sol = c->t_lu = 0;
  // a multi-frequency call evaluates the Rankine part once per depth regime it meets
  c->rk_valid[0] = c->rk_valid[1] = false;
  for (int w0 = 0; w0 < nomega; w0 += cap) {
    const int nw = std::min(cap, nomega - w0);
    // host setup of each frequency (in the caller's order, which the NQ state
    // follows) overlapped with the assembly of the groups set up before it
    OmegaParams* hom = c->h_oms.as<OmegaParams>();
    const int split = pipeline_split(c, nw);
    CK(cudaEventRecord(c->ev[0], c->stream));
    int done = 0;
    for (int i = 0; i < nw; ++i) {
      const double T = 2. * kPI / omegas[w0 + i];
      omega_params(c, 2. * kPI / T, hom[i], true);
      if (i + 1 == nw || i + 1 - done >= ASM_GROUP || i + 1 == split) {
        assemble_range(c, done, i + 1);
        done = i + 1;
        if (done == split) {   // the first frequencies are assembled: factor them beside the rest
          CK(cudaEventRecord(c->ev_pipe[0], c->stream));
          CK(cudaStreamWaitEvent(c->stream2, c->ev_pipe[0], 0));
          mixed_factor(c->mixed, c->d_D.as<double2>(), N, split * cls, c->d_status.as<int>(), c->stream2,
                       c->launches, &c->lanes2, /*have_f32=*/true);
          CK(cudaGetLastError());
          CK(cudaEventRecord(c->ev_pipe[1], c->stream2));
        }
      }
    }
    CK(cudaEventRecord(c->ev[1], c->stream));
    fold_rhs_kernel<<<dim3((N + 127) / 128, nrhs, nw), 128, 0, c->stream>>>(
        nvel_d + (long long)w0 * nrhs * cls * N, N, c->nsymy, nrhs, c->d_X.as<double2>());
    LAUNCHED(c);
    factor_and_solve(c, nw * cls, nrhs, true, uniform_shape(c), split * cls);
    CK(cudaEventRecord(c->ev[2], c->stream));
    potential(c, nw * cls, nrhs, uniform_shape(c));
    if (nint > 0) {
      force_kernel<<<dim3(nint, nrhs, nw), 256, 0, c->stream>>>(c->d_Y.as<double2>(), c->d_oms.as<OmegaParams>(), N,
                                                                c->nsymy, nrhs, nint, nds_d, c->rho,
                                                                force_d + (long long)w0 * nrhs * nint);
      LAUNCHED(c);
    }
    CK(cudaEventRecord(c->ev[3], c->stream));
    check_status(c);
    float a, f, s;
    CK(cudaEventElapsedTime(&a, c->ev[0], c->ev[1]));
    CK(cudaEventElapsedTime(&f, c->ev[1], c->ev[2]));
    CK(cudaEventElapsedTime(&s, c->ev[2], c->ev[3]));
    c->t_asm += a;
    c->t_fac += f;
    c->t_sol += s;
    add_lu_time(c);
  }
  c->w_previous = -1.;  // the batch reused the cached-factor slot
}

// ---------------------------------------------------------------------------
// Cross-body batches. The reference solves one body at a time, frequency by
// frequency (NEMOH.f90:129-143); here (resident body, frequency) items of
// different bodies share one launch sequence: their systems are sorted by
// decreasing order and every kernel of the pipeline takes each system's own
// order and place (ragged batch), so one launch covers the same step of every
// system of the batch.
// ---------------------------------------------------------------------------

// device bytes of the operand images of one item's FP64 updates, in a ragged batch
// whose largest order is nmax
size_t item_image_bytes(const nemoh_ctx* c, const BodyState& b, int nmax) {
  const bool tensor = c->mode == NEMOH_B200_FP64 && tc_enabled() && nmax > LU_OUTER;
  return tensor ? (b.nsymy + 1) * oz_bytes_per_system(nmax) : 0;
}

// device bytes one item adds to a ragged batch whose largest order is nmax
size_t item_bytes(const nemoh_ctx* c, const BodyState& b, int nmax, int nrhs) {
  const size_t n = b.nfa, cls = b.nsymy + 1, nm = nmax, nblk = (nm + TB - 1) / TB;
  size_t per_sys = 2 * nm * nrhs * sizeof(double2) + DIAG_SCRATCH * sizeof(double2) +
                   nblk * 2 * TB * TB * sizeof(double2) + 64;
  size_t mats = 2 * n * n * sizeof(double2);
  if (c->mode == NEMOH_B200_MIXED) {
    mats += n * n * sizeof(float2);
    per_sys += nm * nrhs * (2 * sizeof(double2) + 2 * sizeof(float2)) + (DIAG_SCRATCH + PINV_SCRATCH) * sizeof(float2) +
               nblk * 2 * TB * TB * sizeof(float2) + tc_bytes_per_system(nm);
  }
  return cls * (mats + per_sys) + item_image_bytes(c, b, nmax) + sizeof(OmegaParams) + sizeof(SlotMesh) +
         sizeof(ItemDesc);
}

// one ragged batch: items[0..k) index the caller's arrays, already in
// decreasing order of their body's panel count
void ragged_batch(nemoh_ctx* c, const int* items, int k, const int* body, const double* omegas, int nrhs,
                  const std::vector<long long>& nvel_off, const std::vector<long long>& force_off,
                  const double2* nvel_d, double2* force_d, bool headroom) {
  std::vector<long long> off;
  std::vector<int> ord, host_n(k);
  std::vector<char> has_rk(k);
  std::vector<SlotMesh> sm(k);
  std::vector<ItemDesc> it(k);
  std::vector<char> wide(c->bodies[body[items[0]]]->wide.size());
  long long mat = 0;
  int nint_max = 0;
  for (int j = 0; j < k; ++j) {
    const int i = items[j];
    const BodyState& b = *c->bodies[body[i]];
    for (size_t q = 0; q < b.wide.size(); ++q) wide[q] |= b.wide[q];
    const bool fd = finite_depth(Env{b.g, b.depth, b.gm, nullptr}, 2. * kPI / (2. * kPI / omegas[i]));
    has_rk[j] = b.rk_valid[fd];
    sm[j] = SlotMesh{b.d_rec.as<PanelRec>(), b.d_rows.as<double>(), mat, b.nfa, b.nsymy, b.zer,
                     has_rk[j] ? b.rk[fd].as<double2>() : nullptr};
    it[j] = ItemDesc{nvel_off[i], force_off[i], b.d_nds.as<double>(), b.rho, b.nfa, b.nsymy, (int)ord.size(), b.nint};
    host_n[j] = b.nfa;
    nint_max = std::max(nint_max, b.nint);
    for (int cc = 0; cc <= b.nsymy; ++cc) {
      off.push_back(mat);
      ord.push_back(b.nfa);
      mat += (long long)b.nfa * b.nfa;
    }
  }
  const int nsys = (int)ord.size(), nmax = ord[0];
  const size_t N = nmax, V = (size_t)nsys * N * nrhs;
  // batches of different bodies keep setting new footprints: grow with
  // headroom, when the batch leaves room for it
  CK(c->d_D.ensure((size_t)mat * sizeof(double2), headroom));
  CK(c->d_S.ensure((size_t)mat * sizeof(double2), headroom));
  CK(c->d_X.ensure(V * sizeof(double2), headroom));
  CK(c->d_Y.ensure(V * sizeof(double2), headroom));
  CK(c->d_diag.ensure((size_t)nsys * DIAG_SCRATCH * sizeof(double2), headroom));
  if (c->mode == NEMOH_B200_FP64)
    CK(c->d_inv.ensure((size_t)nsys * ((N + TB - 1) / TB) * 2 * TB * TB * sizeof(double2), headroom));
  else
    CK(c->mixed.ensure(nsys, nmax, nrhs, (size_t)mat, headroom));
  CK(c->d_oms.ensure((size_t)k * sizeof(OmegaParams)));
  CK(c->d_slots.ensure((size_t)k * sizeof(int)));
  CK(c->h_oms.ensure((size_t)k * sizeof(OmegaParams)));
  CK(c->h_slots.ensure((size_t)k * sizeof(int)));
  // descriptions through one pinned staging buffer (the batch ends with a
  // synchronisation, so the next batch may rewrite it)
  const size_t b_off = 0, b_ord = b_off + ((nsys * sizeof(long long) + 255) & ~size_t(255));
  const size_t b_sm = b_ord + ((nsys * sizeof(int) + 255) & ~size_t(255));
  const size_t b_it = b_sm + ((k * sizeof(SlotMesh) + 255) & ~size_t(255));
  const size_t b_end = b_it + k * sizeof(ItemDesc);
  CK(c->h_rag.ensure(b_end));
  CK(c->d_roff.ensure(nsys * sizeof(long long)));
  CK(c->d_rord.ensure(nsys * sizeof(int)));
  CK(c->d_smesh.ensure(k * sizeof(SlotMesh)));
  CK(c->d_items.ensure(k * sizeof(ItemDesc)));
  char* hr = c->h_rag.as<char>();
  std::memcpy(hr + b_off, off.data(), nsys * sizeof(long long));
  std::memcpy(hr + b_ord, ord.data(), nsys * sizeof(int));
  std::memcpy(hr + b_sm, sm.data(), k * sizeof(SlotMesh));
  std::memcpy(hr + b_it, it.data(), k * sizeof(ItemDesc));
  CK(cudaMemcpyAsync(c->d_roff.p, hr + b_off, nsys * sizeof(long long), cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->d_rord.p, hr + b_ord, nsys * sizeof(int), cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->d_smesh.p, hr + b_sm, k * sizeof(SlotMesh), cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(c->d_items.p, hr + b_it, k * sizeof(ItemDesc), cudaMemcpyHostToDevice, c->stream));
  // the uniform path's buffers and cached factors no longer hold what they did
  c->cap_nfa = -1;
  c->w_previous = -1.;
  const long long xs = (long long)N * nrhs;
  Shape sh{nmax, Ragged{c->d_roff.as<long long>(), c->d_rord.as<int>(), ord.data(), off.data()}, wide};
  if (c->mode == NEMOH_B200_FP64) sh.images = fp64_images(c, nsys, sh, headroom);
  OmegaParams* hom = c->h_oms.as<OmegaParams>();
  auto host_setup = [&](int j) {
    BodyState& b = *c->bodies[body[items[j]]];
    const double T = 2. * kPI / omegas[items[j]];
    omega_params_env(Env{b.g, b.depth, b.gm, &b.nq_state}, 2. * kPI / T, hom[j], true);
  };
  auto fold = [&] {
    fold_rhs_ragged_kernel<<<dim3((nmax + 127) / 128, nrhs, k), 128, 0, c->stream>>>(
        nvel_d, c->d_items.as<ItemDesc>(), nrhs, xs, c->d_X.as<double2>());
    LAUNCHED(c);
  };
  auto potential_forces = [&] {
    potential(c, nsys, nrhs, sh);
    if (nint_max > 0) {
      force_ragged_kernel<<<dim3(nint_max, nrhs, k), 256, 0, c->stream>>>(
          c->d_Y.as<double2>(), c->d_items.as<ItemDesc>(), c->d_oms.as<OmegaParams>(), nrhs, xs, force_d);
      LAUNCHED(c);
    }
  };
  if (!c->graph_mode) {
    // host setup of each item overlapped with the assembly of the groups set up before it
    CK(cudaEventRecord(c->ev[0], c->stream));
    int done = 0;
    for (int j = 0; j < k; ++j) {
      host_setup(j);
      if (j + 1 == k || j + 1 - done >= ASM_GROUP) {
        assemble_range(c, done, j + 1, c->d_smesh.as<SlotMesh>(), host_n.data(), has_rk.data());
        done = j + 1;
      }
    }
    CK(cudaEventRecord(c->ev[1], c->stream));
    fold();
    factor_and_solve(c, nsys, nrhs, true, sh);
    CK(cudaEventRecord(c->ev[2], c->stream));
    potential_forces();
    CK(cudaEventRecord(c->ev[3], c->stream));
    check_status(c);
    float a, f, s;
    CK(cudaEventElapsedTime(&a, c->ev[0], c->ev[1]));
    CK(cudaEventElapsedTime(&f, c->ev[1], c->ev[2]));
    CK(cudaEventElapsedTime(&s, c->ev[2], c->ev[3]));
    c->t_asm += a;
    c->t_fac += f;
    c->t_sol += s;
    add_lu_time(c);
    return;
  }
  // Graph mode: every host setup and upload first, then one launch sequence
  // that reads device buffers only. The second batch with the same launch
  // sequence (same shapes, buffers and pointers) is captured, later ones
  // replay the captured graph.
  std::vector<AsmGroup> groups;
  for (int j0 = 0; j0 < k; j0 += ASM_GROUP) {
    const int j1 = std::min(k, j0 + ASM_GROUP);
    for (int j = j0; j < j1; ++j) host_setup(j);
    groups.push_back(assemble_upload(c, j0, j1, host_n.data(), has_rk.data()));
  }
  const bool mixed = c->mode == NEMOH_B200_MIXED;
  const int max_it = refine_max_it(), passes = mixed ? std::min(REFINE_CHUNK, max_it) : 0;
  // the FP64 sweeps' workspace grows here, never inside a captured sequence
  if (!mixed) fp64_sync(c, nsys, nmax);
  // a captured sequence holds every buffer address it was captured with: the
  // key covers them all, so a buffer that moved since is captured again
  std::vector<long long> sig = {c->mode, nrhs, k, nsys, nmax, nint_max, passes, (long long)nvel_d,
                                (long long)force_d, (long long)c->d_D.p, (long long)c->d_S.p, (long long)c->d_X.p,
                                (long long)c->d_Y.p, (long long)c->d_diag.p, (long long)c->d_inv.p,
                                (long long)c->d_oms.p, (long long)c->d_slots.p, (long long)c->d_smesh.p,
                                (long long)c->d_items.p, (long long)c->d_roff.p, (long long)c->d_rord.p,
                                (long long)c->mixed.lu, (long long)c->mixed.diag, (long long)c->mixed.b,
                                (long long)c->mixed.r, (long long)c->mixed.rf, (long long)c->mixed.yf,
                                (long long)c->mixed.inv, (long long)c->mixed.pinv, (long long)c->mixed.norms,
                                (long long)c->mixed.state, (long long)c->mixed.tc.a, (long long)c->mixed.tc.b,
                                (long long)c->mixed.tc.wv, (long long)c->mixed.flow, (long long)c->mixed.act,
                                (long long)c->d_flow.p, (long long)sh.images,
                                // the images only where the sequence holds them: a mixed batch's
                                // FP64 fallback runs outside it, with images of its own size
                                sh.images ? (long long)c->oz.a : 0, sh.images ? (long long)c->oz.b : 0,
                                sh.images ? (long long)c->oz.sc : 0};
  for (const AsmGroup& g : groups)
    sig.insert(sig.end(), {g.ninfd, g.nfd, g.n_infd, g.n_fd, (long long)g.slot_rk_infd, (long long)g.slot_rk_fd});
  sig.insert(sig.end(), ord.begin(), ord.end());
  sig.insert(sig.end(), sh.wide.begin(), sh.wide.end());
  unsigned long long key = 1469598103934665603ull;   // FNV-1a over the signature
  for (long long v : sig)
    for (int b = 0; b < 8; ++b) key = (key ^ (unsigned long long)((v >> (8 * b)) & 0xff)) * 1099511628211ull;
  GraphEntry* ge = nullptr;
  for (GraphEntry& e : c->graphs)
    if (e.key == key) ge = &e;
  CK(cudaEventRecord(c->ev[0], c->stream));
  auto issue = [&] {
    for (const AsmGroup& g : groups) assemble_launch(c, g, c->d_smesh.as<SlotMesh>());
    fold();
    c->lu64 = !mixed;
    if (mixed) {
      mixed_factor(c->mixed, c->d_D.as<double2>(), nmax, nsys, c->d_status.as<int>(), c->stream, c->launches,
                   &c->lanes, /*have_f32=*/true, sh.rg);
      const RefineArgs a{c->d_D.as<double2>(), nmax, nsys, nrhs, c->d_X.as<double2>(), sh.rg};
      mixed_refine_begin(c->mixed, a, max_it, c->stream, c->launches);
      mixed_refine_passes(c->mixed, a, passes, c->stream, c->launches);
    } else {
      factor_fp64(c, nsys, sh);
      trsm_fp64(c, nsys, nrhs, sh);
    }
    potential_forces();
  };
  if (ge && ge->exec) {
    CK(cudaGraphLaunch(ge->exec, c->stream));
    ++c->graph_replays;
  } else if (ge) {   // second sighting: capture, then launch the graph
    cudaGraph_t gr = nullptr;
    CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
    try {
      issue();
    } catch (...) {
      cudaStreamEndCapture(c->stream, &gr);
      if (gr) cudaGraphDestroy(gr);
      throw;
    }
    CK(cudaStreamEndCapture(c->stream, &gr));
    const cudaError_t e = cudaGraphInstantiate(&ge->exec, gr, 0);
    cudaGraphDestroy(gr);
    CK(e);
    CK(cudaGraphLaunch(ge->exec, c->stream));
    ++c->graph_captures;
  } else {   // first sighting: run as is and remember the sequence
    issue();
    if (c->graphs.size() >= 16) {
      if (c->graphs.front().exec) cudaGraphExecDestroy(c->graphs.front().exec);
      c->graphs.erase(c->graphs.begin());
    }
    c->graphs.push_back(GraphEntry{key, nullptr});
  }
  CK(cudaEventRecord(c->ev[3], c->stream));
  check_status(c);
  float s = 0;
  CK(cudaEventElapsedTime(&s, c->ev[0], c->ev[3]));
  c->t_sol += s;   // graph mode times the batch as a whole
  if (mixed) {
    // refinement passes beyond those in the sequence, and the FP64 fallback,
    // run as ordinary launches; the potential and forces are then redone
    const RefineArgs a{c->d_D.as<double2>(), nmax, nsys, nrhs, c->d_X.as<double2>(), sh.rg};
    bool more = mixed_refine_read(c->mixed, c->stream), redo = false;
    for (int it = passes; more && it < max_it; it += REFINE_CHUNK) {
      mixed_refine_passes(c->mixed, a, std::min(REFINE_CHUNK, max_it - it), c->stream, c->launches);
      more = mixed_refine_read(c->mixed, c->stream);
      redo = true;
    }
    if (c->mixed.last_residual > REFINE_TOL) {
      mixed_fallback_ragged(c, nsys, nrhs, sh);
      redo = true;
    }
    if (redo) {
      potential_forces();
      check_status(c);
    }
  }
}

// Rankine caches of the bodies and depth regimes a call needs, evaluated once
// and kept with the resident body, while the bodies' caches stay within
// NEMOH_B200_RANKINE_CACHE_BYTES (default: a quarter of the device memory);
// a body beyond it gets the per-slot Rankine pass in every batch.
size_t body_rankine_cap() {
  size_t fr = 0, tot = 0;
  CK(cudaMemGetInfo(&fr, &tot));
  size_t cap = tot / 4;
  if (const char* e = std::getenv("NEMOH_B200_RANKINE_CACHE_BYTES")) cap = (size_t)std::max(0LL, std::atoll(e));
  return cap;
}

// one body's cache of one depth regime, if it fits the budget
void body_rankine(nemoh_ctx* c, BodyState& b, bool fd, size_t cap) {
  if (b.rk_valid[fd]) return;
  const size_t bytes = (size_t)(b.nsymy + 1) * b.nfa * b.nfa * sizeof(double2);
  if (c->rk_body_bytes + bytes > cap) return;
  GreenCtx g = green_ctx(c);
  g.zer = b.zer;
  rankine_cache(c, g, b.d_rec.as<PanelRec>(), b.d_rows.as<double>(), b.nfa, b.nsymy, b.depth, fd, b.rk[fd],
                b.rk_valid[fd]);
  c->rk_body_bytes += bytes;
}

void ensure_body_rankine(nemoh_ctx* c, int nitem, const int* body, const double* omegas) {
  const size_t cap = body_rankine_cap();
  for (int i = 0; i < nitem; ++i) {
    BodyState& b = *c->bodies[body[i]];
    body_rankine(c, b, finite_depth(Env{b.g, b.depth, b.gm, nullptr}, 2. * kPI / (2. * kPI / omegas[i])), cap);
  }
}

void solve_bodies_impl(nemoh_ctx* c, int nitem, const int* body, const double* omegas, int nrhs,
                       const double2* nvel_d, double2* force_d) {
  if (nrhs < 1 || nrhs > MAX_RHS) throw Fail{NEMOH_B200_ECAPACITY, "nrhs must be in 1..16"};
  std::vector<long long> nvel_off(nitem), force_off(nitem);
  long long ov = 0, of = 0;
  for (int i = 0; i < nitem; ++i) {
    const BodyState& b = *c->bodies[body[i]];
    nvel_off[i] = ov;
    force_off[i] = of;
    ov += (long long)(b.nsymy + 1) * b.nfa * nrhs;
    of += (long long)b.nint * nrhs;
  }
  // decreasing panel count; stable, so each body's frequencies keep the
  // caller's order, which the body's NQ state follows
  std::vector<int> idx(nitem);
  std::iota(idx.begin(), idx.end(), 0);
  std::stable_sort(idx.begin(), idx.end(),
                   [&](int a, int b) { return c->bodies[body[a]]->nfa > c->bodies[body[b]]->nfa; });
  c->t_asm = c->t_fac = c->t_sol = c->t_lu = 0;
  // the resident bodies' Rankine caches first, so that the budget below sees them
  ScopedEvent rk0, rk1;
  CK(cudaEventCreate(&rk0.e));
  CK(cudaEventCreate(&rk1.e));
  CK(cudaEventRecord(rk0.e, c->stream));
  ensure_body_rankine(c, nitem, body, omegas);
  CK(cudaEventRecord(rk1.e, c->stream));
  // admission by HBM footprint: 80% of the free memory, the batch's own
  // buffers counted as free
  auto held_bytes = [&] {   // but for the images
    return c->d_D.bytes + c->d_S.bytes + c->d_X.bytes + c->d_Y.bytes + c->d_inv.bytes + c->d_diag.bytes +
           c->mixed.bytes();
  };
  auto free_bytes = [&] {
    size_t fr = 0, tot = 0;
    CK(cudaMemGetInfo(&fr, &tot));
    // the FP64 updates' images are a mixed batch's only while it falls back
    const size_t images = c->mode == NEMOH_B200_FP64 ? c->oz.bytes() : 0;
    return (size_t)((fr + held_bytes() + images) * 0.8);
  };
  size_t budget = free_bytes();
  // an earlier fallback's images are given back where the call needs the room and they
  // are more than a trifle of it (those of one or two systems stay)
  if (c->mode == NEMOH_B200_MIXED && c->oz.bytes() > budget / 64) {
    size_t need = 0;
    for (int i : idx) need += item_bytes(c, *c->bodies[body[i]], c->bodies[body[idx[0]]]->nfa, nrhs);
    if (need > budget) {
      c->oz.release();
      budget = free_bytes();
    }
  }
  // NEMOH_B200_BATCH_BYTES lowers the budget (tests use it to split a call
  // into several batches)
  if (const char* e = std::getenv("NEMOH_B200_BATCH_BYTES")) {
    const long long v = std::atoll(e);
    if (v > 0) budget = std::min(budget, (size_t)v);
  }
  int pos = 0;
  while (pos < nitem) {
    const int nmax = c->bodies[body[idx[pos]]]->nfa;
    size_t used = 0, images = 0;
    int end = pos;
    while (end < nitem) {
      const BodyState& b = *c->bodies[body[idx[end]]];
      const size_t need = item_bytes(c, b, nmax, nrhs);
      if (end > pos && used + need > budget) break;
      used += need;
      images += item_image_bytes(c, b, nmax);
      ++end;
    }
    // The matrices of smaller hulls are a smaller part of their batch and its images
    // a larger one, while the buffers keep the size that the batches of larger hulls
    // gave them: the images may fill the budget and an eighth (0.9 of the free
    // memory) beside what is held, and the batch is cut to that. Where less than a
    // quarter of them fits, its updates run on the FP64 pipe instead.
    const size_t others = std::max(held_bytes(), used - images), most = budget + budget / 8;
    const size_t room = std::max(c->oz.bytes(), most > others ? most - others : 0);
    if (images > room && images / 4 <= room)
      for (; end > pos + 1 && images > room; --end) {
        const BodyState& b = *c->bodies[body[idx[end - 1]]];
        used -= item_bytes(c, b, nmax, nrhs);
        images -= item_image_bytes(c, b, nmax);
      }
    // the buffers' growth headroom (a quarter) only where the batch leaves room
    ragged_batch(c, idx.data() + pos, end - pos, body, omegas, nrhs, nvel_off, force_off, nvel_d, force_d,
                 used + used / 4 <= budget);
    pos = end;
  }
  float ms = 0;   // the batches ended with a synchronisation
  CK(cudaEventElapsedTime(&ms, rk0.e, rk1.e));
  c->t_asm += ms;
}

}  // namespace

static int guarded(nemoh_ctx* ctx, const std::function<void()>& f) {
  try {
    if (ctx) CK(cudaSetDevice(ctx->device));
    f();
    return NEMOH_B200_OK;
  } catch (const Fail& e) {
    if (ctx) ctx->err = e.msg;
    // a failed runtime call leaves its error as the thread's last error; it is
    // reported here, so the next entry point's launch checks must not see it
    // again (an error that the context keeps comes back on its next call)
    cudaGetLastError();
    return e.code;
  } catch (const std::exception& e) {
    if (ctx) ctx->err = e.what();
    return NEMOH_B200_EINVAL;
  }
}

extern "C" {

int nemoh_b200_create(nemoh_ctx** out, int device, int precision_mode) {
  if (!out) return NEMOH_B200_EINVAL;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return NEMOH_B200_ENODEV;
  if (device < 0 || device >= ndev) return NEMOH_B200_EINVAL;
  if (precision_mode != NEMOH_B200_FP64 && precision_mode != NEMOH_B200_MIXED) return NEMOH_B200_EINVAL;
  nemoh_ctx* c = new nemoh_ctx();
  c->device = device;
  c->mode = precision_mode;
  int st = guarded(c, [&] {
    CK(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    for (auto& e : c->ev) CK(cudaEventCreate(&e));
    for (auto& e : c->ev_lu) CK(cudaEventCreate(&e));
    for (int g = 0; g < LANES; ++g) {
      CK(cudaStreamCreateWithFlags(&c->lanes.s[g], cudaStreamNonBlocking));
      CK(cudaEventCreateWithFlags(&c->lanes.join[g], cudaEventDisableTiming));
    }
    CK(cudaEventCreateWithFlags(&c->lanes.fork, cudaEventDisableTiming));
    // the early LU of a pipelined batch runs at the highest stream priority:
    // its latency-bound launches take SMs as the assembly's CTAs retire
    int prio_lo = 0, prio_hi = 0;
    CK(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
    CK(cudaStreamCreateWithPriority(&c->stream2, cudaStreamNonBlocking, prio_hi));
    for (int g = 0; g < LANES; ++g) {
      CK(cudaStreamCreateWithPriority(&c->lanes2.s[g], cudaStreamNonBlocking, prio_hi));
      CK(cudaEventCreateWithFlags(&c->lanes2.join[g], cudaEventDisableTiming));
    }
    CK(cudaEventCreateWithFlags(&c->lanes2.fork, cudaEventDisableTiming));
    for (auto& e : c->ev_pipe) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    CK(c->d_status.ensure(sizeof(int)));
    CK(cudaMemsetAsync(c->d_status.p, 0, sizeof(int), c->stream));
    c->mixed.status = c->d_status.as<int>();
    CK(c->d_gm.ensure(sizeof(unsigned long long)));
    // Green tables (CREK): nodes on the host, 251-point theta integrals on the device
    table_nodes(c->h_xr, c->h_xz);
    double cqt[NPINTE + 2], qqt[NPINTE + 2], ctt[NPINTE + 2];
    simpson_251(cqt, qqt);
    for (int i = 1; i <= NPINTE; ++i) ctt[i] = std::cos(qqt[i]);
    DevBuf dq, dc;
    CK(dq.ensure(sizeof cqt));
    CK(dc.ensure(sizeof ctt));
    CK(c->d_xr.ensure(sizeof c->h_xr));
    CK(c->d_xz.ensure(sizeof c->h_xz));
    CK(c->d_apd.ensure(sizeof(double4) * TAB_IR * TAB_JZ));
    CK(cudaMemcpyAsync(c->d_xr.p, c->h_xr, sizeof c->h_xr, cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemcpyAsync(c->d_xz.p, c->h_xz, sizeof c->h_xz, cudaMemcpyHostToDevice, c->stream));
    // 3-node Lagrange stencils of both axes: nodes and reciprocal denominators
    std::vector<double> lag(8 * (size_t)(TAB_IR + 2 + TAB_JZ + 2), 0.);
    auto stencils = [&](const double* x, int n, double* out) {
      for (int k = 2; k < n; ++k) {
        const double a = x[k - 1], b = x[k], cc = x[k + 1];
        double* q = out + 8 * k;
        q[0] = a; q[1] = b; q[2] = cc;
        q[3] = 1. / ((a - b) * (a - cc));
        q[4] = 1. / ((b - cc) * (b - a));
        q[5] = 1. / ((cc - a) * (cc - b));
      }
    };
    stencils(c->h_xr, TAB_IR, lag.data());
    stencils(c->h_xz, TAB_JZ, lag.data() + 8 * (TAB_IR + 2));
    CK(c->d_lag.ensure(lag.size() * sizeof(double)));
    CK(cudaMemcpyAsync(c->d_lag.p, lag.data(), lag.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemcpyAsync(dq.p, cqt, sizeof cqt, cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemcpyAsync(dc.p, ctt, sizeof ctt, cudaMemcpyHostToDevice, c->stream));
    crek_kernel<<<(TAB_IR * TAB_JZ + 127) / 128, 128, 0, c->stream>>>(c->d_xr.as<double>(), c->d_xz.as<double>(),
                                                                     dq.as<double>(), dc.as<double>(),
                                                                     c->d_apd.as<double4>());
    LAUNCHED(c);
    // RO > 1e-4 (VNSFD exponential images) decided on RO^2: the largest
    // double whose correctly rounded square root is still <= 1e-4
    double t = 1.E-8;
    while (std::sqrt(std::nextafter(t, 1.)) <= 1.E-4) t = std::nextafter(t, 1.);
    while (std::sqrt(t) > 1.E-4) t = std::nextafter(t, 0.);
    c->ro_eps2 = t;
    StencilThresholds thr;
    stencil_thresholds(&thr);
    CK(c->d_thr.ensure(sizeof thr));
    CK(cudaMemcpyAsync(c->d_thr.p, &thr, sizeof thr, cudaMemcpyHostToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  });
  if (st) {
    nemoh_b200_destroy(c);
    return st;
  }
  *out = c;
  return NEMOH_B200_OK;
}

int nemoh_b200_destroy(nemoh_ctx* c) {
  if (!c) return NEMOH_B200_OK;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  for (int g = 0; g < LANES; ++g) {
    if (c->lanes.s[g]) cudaStreamSynchronize(c->lanes.s[g]);
    if (c->lanes2.s[g]) cudaStreamSynchronize(c->lanes2.s[g]);
  }
  if (c->stream2) cudaStreamSynchronize(c->stream2);
  for (GraphEntry& g : c->graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  for (auto& e : c->ev)
    if (e) cudaEventDestroy(e);
  for (auto& e : c->ev_lu)
    if (e) cudaEventDestroy(e);
  for (int g = 0; g < LANES; ++g) {
    if (c->lanes.join[g]) cudaEventDestroy(c->lanes.join[g]);
    if (c->lanes.s[g]) cudaStreamDestroy(c->lanes.s[g]);
  }
  if (c->lanes.fork) cudaEventDestroy(c->lanes.fork);
  for (int g = 0; g < LANES; ++g) {
    if (c->lanes2.join[g]) cudaEventDestroy(c->lanes2.join[g]);
    if (c->lanes2.s[g]) cudaStreamDestroy(c->lanes2.s[g]);
  }
  if (c->lanes2.fork) cudaEventDestroy(c->lanes2.fork);
  for (auto& e : c->ev_pipe)
    if (e) cudaEventDestroy(e);
  if (c->stream2) cudaStreamDestroy(c->stream2);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return NEMOH_B200_OK;
}

const char* nemoh_b200_last_error(const nemoh_ctx* c) { return c ? c->err.c_str() : "null context"; }

long long nemoh_b200_launch_count(const nemoh_ctx* c) { return c ? c->launches : 0; }

int nemoh_b200_set_mesh(nemoh_ctx* c, int np, int nfa, int nsymy, const double* xyz, const int* m1234, double rho,
                        double g, double depth) {
  if (!c || np < 2 || nfa < 1 || !xyz || !m1234 || !(g > 0)) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    for (int i = 0; i < 4 * nfa; ++i)   // before the context changes
      if (m1234[i] < 1 || m1234[i] > np) throw Fail{NEMOH_B200_EINVAL, "panel node index out of range"};
    c->np = np;
    c->nfa = nfa;
    c->nsymy = (nsymy == 1) ? 1 : 0;
    c->rho = rho;
    c->g = g;
    c->depth = depth;
    c->w_previous = -1.;
    c->nq_state = 0;
    c->rk_valid[0] = c->rk_valid[1] = false;
    upload_geometry(c, np, nfa, c->nsymy, xyz, m1234, c->d_xyz, c->d_m, c->d_rec, c->d_rows, c->zer, c->gm,
                    c->wide);
  });
}

int nemoh_b200_add_body(nemoh_ctx* c, int np, int nfa, int nsymy, const double* xyz, const int* m1234, double rho,
                        double g, double depth, int nint, const double* nds, int* body_id) {
  if (!c || np < 2 || nfa < 1 || !xyz || !m1234 || !(g > 0) || nint < 0 || (nint > 0 && !nds) || !body_id)
    return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    auto b = std::make_unique<BodyState>();
    b->np = np;
    b->nfa = nfa;
    b->nsymy = (nsymy == 1) ? 1 : 0;
    b->rho = rho;
    b->g = g;
    b->depth = depth;
    b->nint = nint;
    upload_geometry(c, np, nfa, b->nsymy, xyz, m1234, b->d_xyz, b->d_m, b->d_rec, b->d_rows, b->zer, b->gm,
                    b->wide);
    const size_t nds_elems = (size_t)nint * nfa * (b->nsymy + 1);
    CK(b->d_nds.ensure(std::max<size_t>(1, nds_elems) * sizeof(double)));
    if (nint) CK(cudaMemcpyAsync(b->d_nds.p, nds, nds_elems * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    c->bodies.push_back(std::move(b));
    *body_id = (int)c->bodies.size() - 1;
  });
}

int nemoh_b200_body_count(const nemoh_ctx* c) { return c ? (int)c->bodies.size() : 0; }

int nemoh_b200_prepare_bodies(nemoh_ctx* c) {
  if (!c) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const size_t cap = body_rankine_cap();
    for (auto& bp : c->bodies) {
      body_rankine(c, *bp, false, cap);   // deep water: any body at high enough frequencies
      if (bp->depth != 0.) body_rankine(c, *bp, true, cap);
    }
    CK(cudaStreamSynchronize(c->stream));
  });
}

int nemoh_b200_set_autotune(int on) {
  set_sweep_autotune(on != 0);
  return NEMOH_B200_OK;
}

int nemoh_b200_set_graphs(nemoh_ctx* c, int on) {
  if (!c) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    CK(cudaStreamSynchronize(c->stream));
    for (GraphEntry& g : c->graphs)
      if (g.exec) cudaGraphExecDestroy(g.exec);
    c->graphs.clear();
    c->graph_mode = on != 0;
  });
}

int nemoh_b200_graph_stats(const nemoh_ctx* c, long long* captures, long long* replays) {
  if (!c) return NEMOH_B200_EINVAL;
  if (captures) *captures = c->graph_captures;
  if (replays) *replays = c->graph_replays;
  return NEMOH_B200_OK;
}

static int bodies_args_ok(const nemoh_ctx* c, int nitem, const int* body, const double* omegas) {
  if (!c || nitem < 1 || !body || !omegas) return 0;
  for (int i = 0; i < nitem; ++i)
    if (body[i] < 0 || body[i] >= (int)c->bodies.size()) return 0;
  return 1;
}

static void bodies_sizes(const nemoh_ctx* c, int nitem, const int* body, int nrhs, size_t* nvel, size_t* force) {
  *nvel = *force = 0;
  for (int i = 0; i < nitem; ++i) {
    const BodyState& b = *c->bodies[body[i]];
    *nvel += (size_t)(b.nsymy + 1) * b.nfa * nrhs;
    *force += (size_t)b.nint * nrhs;
  }
}

int nemoh_b200_solve_bodies(nemoh_ctx* c, int nitem, const int* body, const double* omegas, int nrhs,
                            const double* nvel, double* force) {
  if (!bodies_args_ok(c, nitem, body, omegas) || nrhs < 1 || !nvel || !force) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    if (nrhs > MAX_RHS) throw Fail{NEMOH_B200_ECAPACITY, "nrhs must be in 1..16"};
    size_t nv = 0, nf = 0;
    bodies_sizes(c, nitem, body, nrhs, &nv, &nf);
    CK(c->d_bnvel.ensure(nv * sizeof(double2), true));
    CK(c->d_bforce.ensure(std::max<size_t>(1, nf) * sizeof(double2), true));
    CK(cudaMemcpyAsync(c->d_bnvel.p, nvel, nv * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    solve_bodies_impl(c, nitem, body, omegas, nrhs, c->d_bnvel.as<double2>(), c->d_bforce.as<double2>());
    if (nf) CK(cudaMemcpyAsync(force, c->d_bforce.p, nf * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  });
}

int nemoh_b200_set_body_dofs(nemoh_ctx* c, int body, int ndof, const int* dof_kind, const double* dof_dir,
                             const double* dof_axis) {
  if (!c || body < 0 || body >= (int)c->bodies.size() || ndof < 0 || ndof + 1 > MAX_RHS ||
      (ndof > 0 && (!dof_kind || !dof_dir || !dof_axis)))
    return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    std::vector<PreDof> v(ndof);
    for (int q = 0; q < ndof; ++q) {
      if (dof_kind[q] != 1 && dof_kind[q] != 2) throw Fail{NEMOH_B200_EINVAL, "DOF kind must be 1 or 2"};
      v[q].kind = dof_kind[q];
      v[q].body = 1;
      for (int d = 0; d < 3; ++d) {
        v[q].dir[d] = dof_dir[3 * q + d];
        v[q].axis[d] = dof_axis[3 * q + d];
      }
    }
    BodyState& b = *c->bodies[body];
    CK(b.d_dofs.ensure(std::max<size_t>(1, v.size()) * sizeof(PreDof)));
    if (ndof) CK(cudaMemcpyAsync(b.d_dofs.p, v.data(), v.size() * sizeof(PreDof), cudaMemcpyHostToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    b.ndof = ndof;
  });
}

int nemoh_b200_solve_requests(nemoh_ctx* c, int nreq, const int* body, const double* omegas, const double* betas,
                              double* force) {
  if (!bodies_args_ok(c, nreq, body, omegas) || !betas || !force) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const int ndof = c->bodies[body[0]]->ndof, nrhs = 1 + ndof;
    for (int i = 0; i < nreq; ++i)
      if (c->bodies[body[i]]->ndof != ndof)
        throw Fail{NEMOH_B200_EINVAL, "the bodies of one call must have the same number of DOFs"};
    size_t nv = 0, nf = 0;
    bodies_sizes(c, nreq, body, nrhs, &nv, &nf);
    CK(c->d_bnvel.ensure(nv * sizeof(double2), true));
    CK(c->d_bforce.ensure(std::max<size_t>(1, nf) * sizeof(double2), true));
    CK(c->h_reqs.ensure((size_t)nreq * sizeof(ReqDesc)));
    CK(c->d_reqs.ensure((size_t)nreq * sizeof(ReqDesc)));
    ReqDesc* rq = c->h_reqs.as<ReqDesc>();
    long long off = 0;
    int nmax = 0;
    for (int i = 0; i < nreq; ++i) {
      const BodyState& b = *c->bodies[body[i]];
      const double k = preproc_wavenumber(omegas[i], b.g, b.depth);
      rq[i] = ReqDesc{b.d_xyz.as<double>(), b.d_m.as<int>(), b.d_dofs.as<PreDof>(),
                      PreWave{omegas[i], k, std::cos(betas[i]), std::sin(betas[i])}, b.g, b.depth, off, b.nfa,
                      b.nsymy, ndof};
      off += (long long)(b.nsymy + 1) * b.nfa * nrhs;
      nmax = std::max(nmax, b.nfa);
    }
    CK(cudaMemcpyAsync(c->d_reqs.p, rq, (size_t)nreq * sizeof(ReqDesc), cudaMemcpyHostToDevice, c->stream));
    request_rhs_kernel<<<dim3((nmax + 127) / 128, 2, nreq), 128, 0, c->stream>>>(c->d_reqs.as<ReqDesc>(),
                                                                                c->d_bnvel.as<double2>());
    LAUNCHED(c);
    solve_bodies_impl(c, nreq, body, omegas, nrhs, c->d_bnvel.as<double2>(), c->d_bforce.as<double2>());
    if (nf) CK(cudaMemcpyAsync(force, c->d_bforce.p, nf * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  });
}

int nemoh_b200_solve_bodies_device(nemoh_ctx* c, int nitem, const int* body, const double* omegas, int nrhs,
                                   const double* nvel_device, double* force_device, void* stream) {
  if (!bodies_args_ok(c, nitem, body, omegas) || nrhs < 1 || !nvel_device || !force_device) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const std::string bad =
        device_pointer_problem(c->device, {{nvel_device, "nvel_device"}, {force_device, "force_device"}});
    if (!bad.empty()) throw Fail{NEMOH_B200_EINVAL, bad};
    cudaStream_t user = reinterpret_cast<cudaStream_t>(stream);
    ScopedEvent ev;
    CK(cudaEventCreateWithFlags(&ev.e, cudaEventDisableTiming));
    CK(cudaEventRecord(ev.e, user));
    CK(cudaStreamWaitEvent(c->stream, ev.e, 0));
    solve_bodies_impl(c, nitem, body, omegas, nrhs, reinterpret_cast<const double2*>(nvel_device),
                      reinterpret_cast<double2*>(force_device));
    CK(cudaEventRecord(ev.e, c->stream));
    CK(cudaStreamWaitEvent(user, ev.e, 0));
  });
}

int nemoh_b200_get_geometry(nemoh_ctx* c, double* out, double* zer) {
  if (!c || !out || !c->nfa) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    std::vector<PanelRec> r(c->nfa);
    CK(cudaMemcpyAsync(r.data(), c->d_rec.p, sizeof(PanelRec) * c->nfa, cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    const int n = c->nfa;
    for (int i = 0; i < n; ++i) {
      out[i] = r[i].xn; out[n + i] = r[i].yn; out[2 * n + i] = r[i].zn;
      out[3 * n + i] = r[i].xg; out[4 * n + i] = r[i].yg; out[5 * n + i] = r[i].zg;
      out[6 * n + i] = r[i].aire; out[7 * n + i] = r[i].tdis;
    }
    if (zer) *zer = c->zer;
  });
}

int nemoh_b200_get_tables(nemoh_ctx* c, double* xr, double* xz, double* apd) {
  if (!c) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    std::vector<double4> t(TAB_IR * TAB_JZ);
    CK(cudaMemcpyAsync(t.data(), c->d_apd.p, sizeof(double4) * t.size(), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    if (xr) for (int i = 1; i <= TAB_IR; ++i) xr[i - 1] = c->h_xr[i];
    if (xz) for (int j = 1; j <= TAB_JZ; ++j) xz[j - 1] = c->h_xz[j];
    if (apd)
      for (size_t q = 0; q < t.size(); ++q) {
        apd[q] = t[q].x;
        apd[TAB_IR * TAB_JZ + q] = t[q].y;
        apd[2 * TAB_IR * TAB_JZ + q] = t[q].z;
        apd[3 * TAB_IR * TAB_JZ + q] = t[q].w;
      }
  });
}

int nemoh_b200_assemble(nemoh_ctx* c, double omega, double* dp, double* dm, double* sp, double* sm,
                        int* depth_mode) {
  if (!c || !c->nfa || !(omega > 0)) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    ensure_batch(c, 1, 1);
    OmegaParams& om = c->h_oms.as<OmegaParams>()[0];
    const double T = 2. * kPI / omega;
    omega_params(c, 2. * kPI / T, om, true);
    assemble_range(c, 0, 1);
    check_status(c);
    const size_t NN = (size_t)c->nfa * c->nfa, b = NN * sizeof(double2);
    const bool two = c->nsymy == 1;
    if (dp) CK(cudaMemcpyAsync(dp, c->d_D.p, b, cudaMemcpyDeviceToHost, c->stream));
    if (dm) CK(cudaMemcpyAsync(dm, c->d_D.as<double2>() + (two ? NN : 0), b, cudaMemcpyDeviceToHost, c->stream));
    if (sp) CK(cudaMemcpyAsync(sp, c->d_S.p, b, cudaMemcpyDeviceToHost, c->stream));
    if (sm) CK(cudaMemcpyAsync(sm, c->d_S.as<double2>() + (two ? NN : 0), b, cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    if (depth_mode) *depth_mode = om.fd;
    c->w_previous = -1.;
  });
}

int nemoh_b200_solve_problem(nemoh_ctx* c, double period, const double* nvel, double* zigb, double* zigs,
                             double* zpb, double* zps, int* nexp) {
  if (!c || !c->nfa || !nvel || !(period > 0)) return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const int N = c->nfa, cls = ncls(c);
    const double W = 2. * kPI / period;
    ensure_batch(c, 1, 1);
    if (W != c->w_previous) {
      OmegaParams& om = c->h_oms.as<OmegaParams>()[0];
      omega_params(c, W, om, true);
      assemble_range(c, 0, 1);
      factor_and_solve(c, cls, 1, false, uniform_shape(c));
      check_status(c);
      c->w_previous = W;
      c->cached_fd = om.fd;
      c->cached_nexp = om.nexp;
    } else if (c->cached_fd) {
      OmegaParams tmp;
      omega_params(c, W, tmp, true);  // NQ/LISC side state of a repeated call
    }
    // right-hand sides B = (NVEL(I) +- NVEL(I+NFA))/2 (SOLVE_BEM_INFD_DIRECT.f90:123-131)
    const std::complex<double>* v = reinterpret_cast<const std::complex<double>*>(nvel);
    std::vector<std::complex<double>> B((size_t)cls * N);
    for (int s = 0; s < cls; ++s) {
      const double BX = s == 0 ? 1. : -1.;
      for (int i = 0; i < N; ++i) B[(size_t)s * N + i] = c->nsymy ? (v[i] + BX * v[i + N]) * 0.5 : v[i];
    }
    CK(cudaMemcpyAsync(c->d_X.p, B.data(), B.size() * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    if (c->lu64) trsm_fp64(c, cls, 1, uniform_shape(c));
    else mixed_solve(c, cls, 1, uniform_shape(c));
    std::vector<std::complex<double>> zol((size_t)cls * N), phi((size_t)cls * N);
    CK(cudaMemcpyAsync(zol.data(), c->d_X.p, zol.size() * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    potential(c, cls, 1, uniform_shape(c));
    CK(cudaMemcpyAsync(phi.data(), c->d_Y.p, phi.size() * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    check_status(c);
    auto put = [](double* o, int i, std::complex<double> z) {
      if (o) { o[2 * i] = z.real(); o[2 * i + 1] = z.imag(); }
    };
    for (int i = 0; i < N; ++i) {
      if (c->nsymy) {
        put(zigb, i, zol[i] + zol[N + i]);
        put(zigs, i, zol[i] - zol[N + i]);
        put(zpb, i, phi[i] + phi[N + i]);
        put(zps, i, phi[i] - phi[N + i]);
      } else {
        put(zigb, i, zol[i]);
        put(zigs, i, 0.);
        put(zpb, i, phi[i]);
        put(zps, i, 0.);
      }
    }
    if (nexp) *nexp = c->cached_fd ? c->cached_nexp : 0;
  });
}

int nemoh_b200_solve_frequencies(nemoh_ctx* c, int nomega, const double* omegas, int nrhs, const double* nvel,
                                 int nint, const double* nds, double* force) {
  if (!c || nomega < 1 || !omegas || !nvel || nrhs < 1 || nint < 0 || (nint > 0 && (!nds || !force)))
    return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    // sizes are checked before any copy reads the caller's buffers
    if (!c->nfa) throw Fail{NEMOH_B200_EINVAL, "no mesh"};
    if (nrhs > MAX_RHS) throw Fail{NEMOH_B200_ECAPACITY, "nrhs must be in 1..16"};
    const int N = c->nfa, cls = ncls(c);
    const size_t nv = (size_t)cls * N * nrhs * nomega;
    CK(c->d_nvel.ensure(nv * sizeof(double2)));
    CK(c->d_nds.ensure(std::max<size_t>(1, (size_t)nint * cls * N) * sizeof(double)));
    CK(c->d_force.ensure(std::max<size_t>(1, (size_t)nint * nrhs * nomega) * sizeof(double2)));
    CK(cudaMemcpyAsync(c->d_nvel.p, nvel, nv * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    if (nint)
      CK(cudaMemcpyAsync(c->d_nds.p, nds, (size_t)nint * cls * N * sizeof(double), cudaMemcpyHostToDevice,
                         c->stream));
    solve_frequencies_impl(c, nomega, omegas, nrhs, c->d_nvel.as<double2>(), nint, c->d_nds.as<double>(),
                           c->d_force.as<double2>());
    if (nint)
      CK(cudaMemcpyAsync(force, c->d_force.p, (size_t)nint * nrhs * nomega * sizeof(double2),
                         cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  });
}

int nemoh_b200_solve_frequencies_device(nemoh_ctx* c, int nomega, const double* omegas, int nrhs,
                                        const double* nvel_device, int nint, const double* nds_device,
                                        double* force_device, void* stream) {
  if (!c || nomega < 1 || !omegas || !nvel_device || nrhs < 1 || nint < 0 ||
      (nint > 0 && (!nds_device || !force_device)))
    return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const std::string bad = device_pointer_problem(
        c->device, {{nvel_device, "nvel_device"}, {nds_device, "nds_device"}, {force_device, "force_device"}});
    if (!bad.empty()) throw Fail{NEMOH_B200_EINVAL, bad};
    cudaStream_t user = reinterpret_cast<cudaStream_t>(stream);
    ScopedEvent ev;
    CK(cudaEventCreateWithFlags(&ev.e, cudaEventDisableTiming));
    CK(cudaEventRecord(ev.e, user));
    CK(cudaStreamWaitEvent(c->stream, ev.e, 0));
    solve_frequencies_impl(c, nomega, omegas, nrhs, reinterpret_cast<const double2*>(nvel_device), nint, nds_device,
                           reinterpret_cast<double2*>(force_device));
    CK(cudaEventRecord(ev.e, c->stream));
    CK(cudaStreamWaitEvent(user, ev.e, 0));
  });
}

int nemoh_b200_kochin(nemoh_ctx* c, double period, double xeff, double yeff, int ntheta, const double* theta,
                      int nprob, const double* zigb, const double* zigs, double* hkochin) {
  if (!c || !c->nfa || !(period > 0) || ntheta < 0 || nprob < 0 || (ntheta > 0 && (!theta || !hkochin)) ||
      (nprob > 0 && !zigb) || (nprob > 0 && c->nsymy && !zigs))
    return NEMOH_B200_EINVAL;
  if (ntheta == 0 || nprob == 0) return NEMOH_B200_OK;
  return guarded(c, [&] {
    // wave number of SOLVE_BVP (SOLVE_BEM.f90:62-84): W^2/G, or AMH/Depth from X0
    const double W = 2. * kPI / period;
    double kwave = W * W / c->g;
    if (!((c->depth == 0.) || (kwave * c->depth >= 20))) {
      double AMH;
      const int st = finite_depth_root(W * W * c->depth / c->g, &AMH);
      if (st) throw Fail{st, "ERREUR DANS LA RECHERCHE DE LA RACINE (X0)"};
      kwave = AMH / c->depth;
    }
    const double ye = c->nsymy ? 0. : yeff;   // INITIALIZATION.f90:60
    const int N = c->nfa;
    const size_t ns = (size_t)N * nprob, nh = (size_t)ntheta * nprob;
    std::vector<double2> cs(ntheta);
    for (int t = 0; t < ntheta; ++t) cs[t] = make_double2(std::cos(theta[t]), std::sin(theta[t]));
    const size_t bytes = (2 * ns + nh + ntheta) * sizeof(double2);
    CK(c->d_kochin.ensure(bytes));
    double2* db = c->d_kochin.as<double2>();
    double2* ds = db + ns;
    double2* dh = ds + ns;
    double2* dc = dh + nh;
    CK(cudaMemcpyAsync(db, zigb, ns * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    if (c->nsymy) CK(cudaMemcpyAsync(ds, zigs, ns * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemcpyAsync(dc, cs.data(), ntheta * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    CK(cudaMemsetAsync(dh, 0, nh * sizeof(double2), c->stream));
    kochin_kernel<<<dim3((N + KOCHIN_THREADS - 1) / KOCHIN_THREADS, ntheta), KOCHIN_THREADS, 0, c->stream>>>(
        c->d_xyz.as<double>(), c->d_m.as<int>(), c->d_rows.as<double>(), N, c->nsymy, kwave, c->depth, xeff, ye, dc,
        nprob, db, ds, ntheta, dh);
    LAUNCHED(c);
    CK(cudaMemcpyAsync(hkochin, dh, nh * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  });
}

int nemoh_b200_free_surface(nemoh_ctx* c, double period, int npts, const double* xy, int nprob, const double* zigb,
                            const double* zigs, double* eta) {
  if (!c || !c->nfa || !(period > 0) || npts < 0 || nprob < 0 || (npts > 0 && (!xy || !eta)) ||
      (nprob > 0 && !zigb) || (nprob > 0 && c->nsymy && !zigs))
    return NEMOH_B200_EINVAL;
  if (npts == 0 || nprob == 0) return NEMOH_B200_OK;
  return guarded(c, [&] {
    const int N = c->nfa;
    const double W = 2. * kPI / period;
    OmegaParams om;
    omega_params(c, W, om, false);
    const bool fd = field_forms(om, W, c->g, c->depth);
    const size_t ns = (size_t)N * FS_MAXP, nphi = (size_t)npts * FS_MAXP;
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
    const size_t o_om = take(sizeof(OmegaParams)), o_xy = take(npts * sizeof(double2)),
                 o_b = take(ns * sizeof(double2)), o_s = take(ns * sizeof(double2)), o_p = take(nphi * sizeof(double2));
    CK(c->d_fs.ensure(off));
    char* base = c->d_fs.as<char>();
    cudaStream_t st = c->stream;
    CK(cudaMemcpyAsync(base + o_om, &om, sizeof om, cudaMemcpyHostToDevice, st));
    std::vector<double2> pts(npts);
    for (int q = 0; q < npts; ++q) pts[q] = make_double2(xy[2 * q], xy[2 * q + 1]);
    CK(cudaMemcpyAsync(base + o_xy, pts.data(), npts * sizeof(double2), cudaMemcpyHostToDevice, st));
    GreenCtx g = green_ctx(c);
    std::vector<std::complex<double>> phi(nphi);
    const std::complex<double> scale(0., W / c->g);   // ETA = i W / G PHI
    for (int p0 = 0; p0 < nprob; p0 += FS_MAXP) {
      const int np = std::min(FS_MAXP, nprob - p0);
      CK(cudaMemcpyAsync(base + o_b, zigb + 2 * (size_t)N * p0, (size_t)N * np * sizeof(double2),
                         cudaMemcpyHostToDevice, st));
      if (c->nsymy)
        CK(cudaMemcpyAsync(base + o_s, zigs + 2 * (size_t)N * p0, (size_t)N * np * sizeof(double2),
                           cudaMemcpyHostToDevice, st));
      CK(cudaMemsetAsync(base + o_p, 0, (size_t)npts * np * sizeof(double2), st));
      const dim3 grid((npts + FS_POINTS - 1) / FS_POINTS, (N + FS_PANELS - 1) / FS_PANELS);
      auto args = [&](auto kernel) {
        kernel<<<grid, FS_POINTS, fs_smem(np), st>>>(
            g, reinterpret_cast<const OmegaParams*>(base + o_om), c->d_rec.as<PanelRec>(), N,
            reinterpret_cast<const double2*>(base + o_xy), npts, np, reinterpret_cast<const double2*>(base + o_b),
            reinterpret_cast<const double2*>(base + o_s), reinterpret_cast<double2*>(base + o_p));
      };
      if (fd) args(freesurface_kernel<true>);
      else args(freesurface_kernel<false>);
      LAUNCHED(c);
      CK(cudaMemcpyAsync(phi.data(), base + o_p, (size_t)npts * np * sizeof(double2), cudaMemcpyDeviceToHost, st));
      check_status(c);
      for (size_t q = 0; q < (size_t)npts * np; ++q) {
        const std::complex<double> e = scale * phi[q];
        eta[2 * ((size_t)npts * p0 + q)] = e.real();
        eta[2 * ((size_t)npts * p0 + q) + 1] = e.imag();
      }
    }
  });
}

int nemoh_b200_irf(nemoh_ctx* c, int nw, const double* w, int nrad, int nint, const double* damping,
                   const double* added_mass, int ntime, double dt, double* K, double* ainf) {
  if (!c || nw < 1 || nrad < 0 || nint < 0 || ntime < 0 || !(dt > 0) || !w || !K || !ainf ||
      (nrad * nint > 0 && (!damping || !added_mass)))
    return NEMOH_B200_EINVAL;
  const int npair = nrad * nint;
  if (npair == 0) return NEMOH_B200_OK;
  for (int l = 0; l < nw; ++l)
    if (!(w[l] != 0.)) return NEMOH_B200_EINVAL;   // CM(l)/w(l)
  return guarded(c, [&] {
    const size_t nc = (size_t)nw * npair, nk = (size_t)std::max(ntime, 1) * npair;
    CK(c->d_irf.ensure((nw + 3 * nc + nk + npair) * sizeof(double)));
    double* dw = c->d_irf.as<double>();
    double* dB = dw + nw;
    double* dA = dB + nc;
    double* dcm = dA + nc;
    double* dK = dcm + nc;
    double* dai = dK + nk;
    cudaStream_t st = c->stream;
    CK(cudaMemcpyAsync(dw, w, nw * sizeof(double), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dB, damping, nc * sizeof(double), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dA, added_mass, nc * sizeof(double), cudaMemcpyHostToDevice, st));
    const unsigned chunks = (npair + IRF_CH - 1) / IRF_CH;
    if (ntime > 0) {
      irf_kernel<<<(ntime + IRF_THREADS - 1) / IRF_THREADS * chunks, IRF_THREADS, 0, st>>>(nw, dw, npair, dB, ntime,
                                                                                           dt, dK);
      LAUNCHED(c);
    }
    irf_added_mass_kernel<<<nw * chunks, IRF_THREADS, 0, st>>>(
        nw, dw, npair, dA, ntime, dt, dK, dcm);
    LAUNCHED(c);
    irf_average_kernel<<<(npair + 127) / 128, 128, 0, st>>>(nw, npair, dcm, dai);
    LAUNCHED(c);
    if (ntime > 0) CK(cudaMemcpyAsync(K, dK, (size_t)ntime * npair * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(ainf, dai, npair * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
  });
}

static int body_conditions_impl(nemoh_ctx* c, const int* panel_body, double xeff, double yeff, int nomega,
                                const double* omegas, int nbeta, const double* betas, int ndof, const int* dof_kind,
                                const int* dof_body, const double* dof_dir, const double* dof_axis, int nforce,
                                const int* force_kind, const int* force_body, const double* force_dir,
                                const double* force_axis, double* nvel_d, double* nds_d, double* fk_d,
                                cudaStream_t user, bool host_out, double* nvel_h, double* nds_h, double* fk_h) {
  if (!c || !c->nfa || nomega < 0 || nbeta < 0 || ndof < 0 || nforce < 0 || (nomega > 0 && !omegas) ||
      (nbeta > 0 && !betas) || (ndof > 0 && (!dof_kind || !dof_dir || !dof_axis)) ||
      (nforce > 0 && (!force_kind || !force_dir || !force_axis)))
    return NEMOH_B200_EINVAL;
  return guarded(c, [&] {
    const int N = c->nfa, nc = N * (c->nsymy + 1), npb = nbeta + ndof;
    std::vector<PreWave> waves((size_t)nomega * nbeta);
    for (int w = 0; w < nomega; ++w) {
      const double k = preproc_wavenumber(omegas[w], c->g, c->depth);
      for (int b = 0; b < nbeta; ++b) waves[(size_t)w * nbeta + b] = PreWave{omegas[w], k, std::cos(betas[b]), std::sin(betas[b])};
    }
    auto spec = [](int n, const int* kind, const int* body, const double* dir, const double* axis) {
      std::vector<PreDof> v(n);
      for (int q = 0; q < n; ++q) {
        if (kind[q] != 1 && kind[q] != 2) throw Fail{NEMOH_B200_EINVAL, "DOF kind must be 1 or 2"};
        v[q].kind = kind[q];
        v[q].body = body ? body[q] : 1;
        for (int d = 0; d < 3; ++d) {
          v[q].dir[d] = dir[3 * q + d];
          v[q].axis[d] = axis[3 * q + d];
        }
      }
      return v;
    };
    const std::vector<PreDof> dofs = spec(ndof, dof_kind, dof_body, dof_dir, dof_axis);
    const std::vector<PreDof> frc = spec(nforce, force_kind, force_body, force_dir, force_axis);
    const size_t n_nvel = (size_t)nc * npb * nomega, n_nds = (size_t)nforce * nc, n_fk = (size_t)nforce * nbeta * nomega;
    // device staging: specs, waves, panel bodies, and (host outputs) the results
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
    const size_t o_w = take(waves.size() * sizeof(PreWave)), o_d = take(dofs.size() * sizeof(PreDof)),
                 o_f = take(frc.size() * sizeof(PreDof)), o_b = take(panel_body ? N * sizeof(int) : 0),
                 o_nv = take(host_out ? n_nvel * sizeof(double2) : 0), o_nd = take(host_out ? n_nds * sizeof(double) : 0),
                 o_fk = take(host_out ? n_fk * sizeof(double2) : 0);
    CK(c->d_pre.ensure(std::max<size_t>(off, 256)));
    char* base = c->d_pre.as<char>();
    cudaStream_t st = c->stream;
    ScopedEvent ev;
    if (!host_out) {
      const std::string bad = device_pointer_problem(
          c->device, {{nvel_d, "nvel_device"}, {nds_d, "nds_device"}, {fk_d, "fk_device"}});
      if (!bad.empty()) throw Fail{NEMOH_B200_EINVAL, bad};
      CK(cudaEventCreateWithFlags(&ev.e, cudaEventDisableTiming));
      CK(cudaEventRecord(ev.e, user));
      CK(cudaStreamWaitEvent(st, ev.e, 0));
    }
    if (!waves.empty()) CK(cudaMemcpyAsync(base + o_w, waves.data(), waves.size() * sizeof(PreWave), cudaMemcpyHostToDevice, st));
    if (!dofs.empty()) CK(cudaMemcpyAsync(base + o_d, dofs.data(), dofs.size() * sizeof(PreDof), cudaMemcpyHostToDevice, st));
    if (!frc.empty()) CK(cudaMemcpyAsync(base + o_f, frc.data(), frc.size() * sizeof(PreDof), cudaMemcpyHostToDevice, st));
    if (panel_body) CK(cudaMemcpyAsync(base + o_b, panel_body, N * sizeof(int), cudaMemcpyHostToDevice, st));
    double2* nv = host_out ? reinterpret_cast<double2*>(base + o_nv) : reinterpret_cast<double2*>(nvel_d);
    double* nd = host_out ? (nds_h ? reinterpret_cast<double*>(base + o_nd) : nullptr) : nds_d;
    double2* fk = host_out ? (fk_h ? reinterpret_cast<double2*>(base + o_fk) : nullptr) : reinterpret_cast<double2*>(fk_d);
    if (fk && n_fk) CK(cudaMemsetAsync(fk, 0, n_fk * sizeof(double2), st));
    if (nv || nd || fk) {
      preproc_kernel<<<dim3((N + 127) / 128, c->nsymy + 1), 128, 0, st>>>(
          c->d_xyz.as<double>(), c->d_m.as<int>(), panel_body ? reinterpret_cast<const int*>(base + o_b) : nullptr, N,
          c->nsymy, c->rho, c->g, c->depth, xeff, yeff, reinterpret_cast<const PreWave*>(base + o_w), nomega, nbeta,
          reinterpret_cast<const PreDof*>(base + o_d), ndof, reinterpret_cast<const PreDof*>(base + o_f), nforce, nv, nd,
          fk);
      LAUNCHED(c);
    }
    if (host_out) {
      if (nvel_h && n_nvel) CK(cudaMemcpyAsync(nvel_h, nv, n_nvel * sizeof(double2), cudaMemcpyDeviceToHost, st));
      if (nds_h && n_nds) CK(cudaMemcpyAsync(nds_h, nd, n_nds * sizeof(double), cudaMemcpyDeviceToHost, st));
      if (fk_h && n_fk) CK(cudaMemcpyAsync(fk_h, fk, n_fk * sizeof(double2), cudaMemcpyDeviceToHost, st));
      CK(cudaStreamSynchronize(st));
    } else {
      CK(cudaEventRecord(ev.e, st));
      CK(cudaStreamWaitEvent(user, ev.e, 0));
      // the staged specs must outlive the kernel: wait before the next call may overwrite them
      CK(cudaStreamSynchronize(st));
    }
  });
}

int nemoh_b200_body_conditions(nemoh_ctx* c, const int* panel_body, double xeff, double yeff, int nomega,
                               const double* omegas, int nbeta, const double* betas, int ndof, const int* dof_kind,
                               const int* dof_body, const double* dof_dir, const double* dof_axis, int nforce,
                               const int* force_kind, const int* force_body, const double* force_dir,
                               const double* force_axis, double* nvel, double* nds, double* fk) {
  if (!nvel && (nomega * (nbeta + ndof)) > 0) return NEMOH_B200_EINVAL;
  return body_conditions_impl(c, panel_body, xeff, yeff, nomega, omegas, nbeta, betas, ndof, dof_kind, dof_body,
                              dof_dir, dof_axis, nforce, force_kind, force_body, force_dir, force_axis, nullptr,
                              nullptr, nullptr, nullptr, true, nvel, nds, fk);
}

int nemoh_b200_body_conditions_device(nemoh_ctx* c, const int* panel_body, double xeff, double yeff, int nomega,
                                      const double* omegas, int nbeta, const double* betas, int ndof,
                                      const int* dof_kind, const int* dof_body, const double* dof_dir,
                                      const double* dof_axis, int nforce, const int* force_kind, const int* force_body,
                                      const double* force_dir, const double* force_axis, double* nvel_device,
                                      double* nds_device, double* fk_device, void* stream) {
  if (!nvel_device && (nomega * (nbeta + ndof)) > 0) return NEMOH_B200_EINVAL;
  return body_conditions_impl(c, panel_body, xeff, yeff, nomega, omegas, nbeta, betas, ndof, dof_kind, dof_body,
                              dof_dir, dof_axis, nforce, force_kind, force_body, force_dir, force_axis, nvel_device,
                              nds_device, fk_device, reinterpret_cast<cudaStream_t>(stream), false, nullptr, nullptr,
                              nullptr);
}

int nemoh_b200_last_refinement(nemoh_ctx* c, int* iterations, double* residual) {
  if (!c) return NEMOH_B200_EINVAL;
  if (iterations) *iterations = c->mixed.last_iterations;
  if (residual) *residual = c->mixed.last_residual;
  return NEMOH_B200_OK;
}

int nemoh_b200_last_timings(nemoh_ctx* c, double* a, double* f, double* s) {
  if (!c) return NEMOH_B200_EINVAL;
  if (a) *a = c->t_asm;
  if (f) *f = c->t_fac;
  if (s) *s = c->t_sol;
  return NEMOH_B200_OK;
}

int nemoh_b200_fallback_count(const nemoh_ctx* c, long long* batches, long long* systems) {
  if (!c) return NEMOH_B200_EINVAL;
  if (batches) *batches = c->mixed.fallbacks;
  if (systems) *systems = c->fallback_systems;
  return NEMOH_B200_OK;
}

int nemoh_b200_last_factor_ms(nemoh_ctx* c, double* lu_ms) {
  if (!c || !lu_ms) return NEMOH_B200_EINVAL;
  *lu_ms = c->t_lu;
  return NEMOH_B200_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// diagnostics (include/nemoh_b200_diag.h): host setup only, no device needed
// ---------------------------------------------------------------------------
#include "../../include/nemoh_b200_diag.h"

// the short reciprocals in place: rsqrt3 of x, crecip of p and q
static __global__ void reciprocals_kernel(int n, double* x, double2* p, float2* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] = rsqrt3(x[i]);
  p[i] = crecip(p[i]);
  q[i] = crecip(q[i]);
}

extern "C" {

int nemoh_b200_diag_dispersion_root(double ak, double* root) { return finite_depth_root(ak, root); }

int nemoh_b200_diag_exponential_fit(double akh, double amh, int* nexp, double* ambda, double* ar) {
  double a[MAX_NEXP + 1] = {0}, r[MAX_NEXP + 1] = {0};
  int st = exponential_fit(akh, amh, nexp, a, r);
  for (int i = 1; i <= MAX_NEXP; ++i) {
    ambda[i - 1] = a[i];
    ar[i - 1] = r[i];
  }
  return st;
}

int nemoh_b200_diag_theta_quadrature(double akk, double* qq, double* cq) {
  double q[MAX_NQ + 2], c[MAX_NQ + 2];
  const int n = theta_quadrature(akk, q, c);
  for (int i = 1; i <= n; ++i) {
    qq[i - 1] = q[i];
    cq[i - 1] = c[i];
  }
  return n;
}

int nemoh_b200_diag_stencil_thresholds(double* kj8, double* kj5, double* ki5) {
  StencilThresholds t;
  stencil_thresholds(&t);
  for (int k = 0; k < 48; ++k) {
    kj8[k] = t.kj8[k];
    kj5[k] = t.kj5[k];
    ki5[k] = t.ki5[k];
  }
  return 0;
}

}  // extern "C"

// FP64 FMA throughput of the device: every thread runs eight independent FMA
// chains (enough to cover the pipe's latency with eight CTAs of 256 threads
// per SM), iters steps each; 2 FLOP per FMA.
__global__ void __launch_bounds__(256) dfma_peak_kernel(double* out, int iters, double b, double c) {
  double a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = (threadIdx.x + j) * 1e-9;
#pragma unroll 1
  for (int i = 0; i < iters; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = fma(a[j], b, c);
  double s = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += a[j];
  if (s == 12345.678) out[0] = s;   // keeps the chains live; never true for these inputs
}

extern "C" {

int nemoh_b200_diag_fp64_peak(int device, double* tflops) {
  if (!tflops) return NEMOH_B200_EINVAL;
  *tflops = 0;
  int prev = -1;
  cudaGetDevice(&prev);
  int sms = 0;
  if (cudaSetDevice(device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return NEMOH_B200_ECUDA;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  double* out = nullptr;
  int rc = NEMOH_B200_OK;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess || cudaEventCreate(&e0) != cudaSuccess ||
      cudaEventCreate(&e1) != cudaSuccess || cudaMalloc(&out, sizeof(double)) != cudaSuccess) {
    rc = NEMOH_B200_ECUDA;
  } else {
    const int blocks = sms * 8, threads = 256, iters = 4096;
    double best = 0;
    for (int rep = 0; rep < 4; ++rep) {
      cudaEventRecord(e0, st);
      dfma_peak_kernel<<<blocks, threads, 0, st>>>(out, iters, 1.0000001, 1e-7);
      cudaEventRecord(e1, st);
      float ms = 0;
      if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess || ms <= 0) {
        rc = NEMOH_B200_ECUDA;
        break;
      }
      const double flop = 2.0 * 8.0 * iters * (double)blocks * threads;
      best = std::max(best, flop / (ms * 1e-3) / 1e12);
    }
    *tflops = best;
  }
  if (out) cudaFree(out);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (st) cudaStreamDestroy(st);
  if (prev >= 0) cudaSetDevice(prev);
  return rc;
}

// A dataflow sweep whose wait cannot end: one system of order 128 (two row
// blocks) with the item counter started past level 0, so the level-1 item
// waits on a ready flag that no item raises. The wait runs out, records
// ST_SWEEP_TIMEOUT and the launch returns; the device stays usable.
long long nemoh_b200_diag_tensor_updates(const nemoh_ctx* c) { return c ? c->tensor_updates : 0; }

int nemoh_b200_diag_sweep_timeout(int device, int* status, double* ms) {
  if (!status || !ms) return NEMOH_B200_EINVAL;
  return guarded(nullptr, [&] {
    CK(cudaSetDevice(device));
    const int n = 128, nblk = 2;
    DevBuf A, inv, X, Y, ws, st;
    CK(A.ensure((size_t)n * n * sizeof(double2)));
    CK(inv.ensure((size_t)nblk * 2 * TB * TB * sizeof(double2)));
    CK(X.ensure((size_t)n * sizeof(double2)));
    CK(Y.ensure((size_t)n * sizeof(double2)));
    CK(ws.ensure(flow_ws_ints(1, nblk) * sizeof(int)));
    CK(st.ensure(sizeof(int)));
    CK(cudaMemset(A.p, 0, A.bytes));
    CK(cudaMemset(inv.p, 0, inv.bytes));
    CK(cudaMemset(X.p, 0, X.bytes));
    CK(cudaMemset(Y.p, 0, Y.bytes));
    CK(cudaMemset(ws.p, 0, ws.bytes));
    CK(cudaMemset(st.p, 0, sizeof(int)));
    const int first = 1;   // the item counter skips the level-0 item
    CK(cudaMemcpy(ws.p, &first, sizeof(int), cudaMemcpyHostToDevice));
    const BatchT<double2> b = make_batch<double2>(A.as<double2>(), n, nullptr, nullptr, Ragged());
    const int smem = flow_smem<double2, 1>() + (nblk + 1) * (int)sizeof(int);
    ScopedEvent e0, e1;
    CK(cudaEventCreate(&e0.e));
    CK(cudaEventCreate(&e1.e));
    CK(cudaEventRecord(e0.e, 0));
    trsm_flow_kernel<double2, 1, true><<<1, FL_THREADS, smem>>>(b, inv.as<double2>(), nblk, 1, X.as<double2>(),
                                                                Y.as<double2>(), n, ws.as<int>(), st.as<int>(),
                                                                nullptr);
    CK(cudaGetLastError());
    CK(cudaEventRecord(e1.e, 0));
    CK(cudaEventSynchronize(e1.e));
    float t = 0;
    CK(cudaEventElapsedTime(&t, e0.e, e1.e));
    *ms = t;
    CK(cudaMemcpy(status, st.p, sizeof(int), cudaMemcpyDeviceToHost));
  });
}

int nemoh_b200_diag_reciprocals(int device, int n, const double* x, double* rs, const double* p, double* rp,
                                const float* q, float* rq) {
  if (n < 1 || !x || !rs || !p || !rp || !q || !rq) return NEMOH_B200_EINVAL;
  return guarded(nullptr, [&] {
    CK(cudaSetDevice(device));
    DevBuf dx, dp, dq;
    CK(dx.ensure((size_t)n * sizeof(double)));
    CK(dp.ensure((size_t)n * sizeof(double2)));
    CK(dq.ensure((size_t)n * sizeof(float2)));
    CK(cudaMemcpy(dx.p, x, (size_t)n * sizeof(double), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(dp.p, p, (size_t)n * sizeof(double2), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(dq.p, q, (size_t)n * sizeof(float2), cudaMemcpyHostToDevice));
    reciprocals_kernel<<<(n + 255) / 256, 256>>>(n, dx.as<double>(), dp.as<double2>(), dq.as<float2>());
    CK(cudaGetLastError());
    CK(cudaMemcpy(rs, dx.p, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(rp, dp.p, (size_t)n * sizeof(double2), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(rq, dq.p, (size_t)n * sizeof(float2), cudaMemcpyDeviceToHost));
  });
}

int nemoh_b200_diag_fp64_update(int device, int n, int nsys, const int* orders, int panels, double* a) {
  if (!a || nsys < 1 || panels < 1 || panels > 2 || n <= panels * LU_OUTER) return NEMOH_B200_EINVAL;
  for (int s = 0; orders && s < nsys; ++s)
    if (orders[s] < 1 || orders[s] > (s ? orders[s - 1] : n)) return NEMOH_B200_EINVAL;
  if (orders && orders[0] != n) return NEMOH_B200_EINVAL;
  return guarded(nullptr, [&] {
    CK(cudaSetDevice(device));
    DevBuf A, off, ord, st;
    OzWork w;
    const size_t nn = (size_t)n * n, bytes = nsys * nn * sizeof(double2);
    CK(A.ensure(bytes));
    CK(st.ensure(sizeof(int)));
    CK(w.ensure(nsys, n));
    CK(cudaMemset(st.p, 0, sizeof(int)));
    CK(cudaMemcpy(A.p, a, bytes, cudaMemcpyHostToDevice));
    Ragged rg;
    if (orders) {
      std::vector<long long> o(nsys);
      for (int s = 0; s < nsys; ++s) o[s] = (long long)(s * nn);
      CK(off.ensure(nsys * sizeof(long long)));
      CK(ord.ensure(nsys * sizeof(int)));
      CK(cudaMemcpy(off.p, o.data(), nsys * sizeof(long long), cudaMemcpyHostToDevice));
      CK(cudaMemcpy(ord.p, orders, nsys * sizeof(int), cudaMemcpyHostToDevice));
      rg.off = off.as<long long>();
      rg.ord = ord.as<int>();
    }
    const Batch b = make_batch<double2>(A.as<double2>(), n, nullptr, nullptr, rg);
    long long launches = 0;
    for (int p = 0; p < panels; ++p) {
      const OzSet cur = oz_set(w, p, 0);
      oz_prep(cur, oz_stride(w), b, p * LU_OUTER, nsys, 0, launches);
      oz_apply(cur, p ? oz_set(w, 0, 0) : OzSet(), oz_stride(w), b, p * LU_OUTER, nsys, 0, launches, st.as<int>(),
               p + 1 < panels);
    }
    CK(cudaGetLastError());
    int status = 0;
    CK(cudaMemcpy(&status, st.p, sizeof(int), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(a, A.p, bytes, cudaMemcpyDeviceToHost));
    if (status) throw Fail{status, "tensor-core update timed out waiting on its operands"};
  });
}

int nemoh_b200_diag_sweep_tuning(long long* keys_tuned, int n, int nsys, int nrhs, int single, int* cluster_size) {
  SweepTuner& t = sweep_tuner();
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(t.mu);
  if (keys_tuned) *keys_tuned = t.tuned;
  if (cluster_size) {
    auto it = t.best.find(sweep_key(dev, single != 0, n, nsys, nrhs));
    *cluster_size = it == t.best.end() ? 0 : it->second;
  }
  return 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Factor-and-solve of device-resident systems that allocates nothing.
//
// Callers that cannot allocate: hosts that keep the device's memory under
// their own allocator -- a PyTorch process whose caching allocator holds the
// free HBM, or a batching server that sized its batches to the memory left
// (nemoh_b200.serving admits frequencies by HBM footprint) -- where a
// cudaMalloc inside the call could fail after admission, or force the host's
// pool to give memory back; and hosts running several solves side by side on
// one device, where the device-wide synchronisation of cudaFree would stall
// the other streams. This entry point therefore takes every buffer from the
// caller and keeps its scratch in one static device array of fixed size.
//
// Scratch layout (offsets rounded to 256 bytes):
//   status word (int)                    must be 0 when the factorization starts:
//                                        the call clears it on its stream first
//   nsys x 3 x 32x32 complex             factored diagonal block of the current
//                                        LU step and the inverses of its two
//                                        triangles (written before they are read)
//   nsys x nblk x 2 x 64x64 complex      inverses of the 64x64 diagonal blocks
//                                        of L and U (written before read)
//   nsys x n x nrhs complex              intermediate vector of the triangular
//                                        solves (written before read)
// Only the status word has to start at zero. Every call on a device shares
// the one array: calls whose work overlaps on the GPU (other streams, other
// host threads) race on it and give wrong results; serialise them.
// ---------------------------------------------------------------------------
namespace {

static __device__ __align__(256) unsigned char g_noalloc_scratch[NEMOH_B200_NOALLOC_SCRATCH_BYTES];

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[kNoallocMaxDevices] = {};

size_t noalloc_align(size_t x) { return (x + 255) & ~size_t(255); }

// scratch bytes needed for nsys systems of order n with nrhs right-hand sides
size_t noalloc_bytes(long long n, long long nsys, long long nrhs) {
  const long long nblk = (n + TB - 1) / TB;
  return noalloc_align(sizeof(int)) + noalloc_align((size_t)nsys * DIAG_SCRATCH * sizeof(double2)) +
         noalloc_align((size_t)(nsys * nblk * 2) * TB * TB * sizeof(double2)) +
         noalloc_align((size_t)(nsys * n * nrhs) * sizeof(double2));
}

void noalloc_message(char* msg, int len, const std::string& s) {
  if (msg && len > 0) {
    std::snprintf(msg, (size_t)len, "%s", s.c_str());
  }
}

}  // namespace

extern "C" int nemoh_b200_factor_solve_device_noalloc(int device, int n, int nsys, double* a_device, int nrhs,
                                                      double* x_device, void* stream, char* msg, int msg_len) {
  noalloc_message(msg, msg_len, "");
  if (device < 0 || device >= kNoallocMaxDevices || n < 1 || nsys < 1 || nrhs < 1 || nrhs > MAX_RHS || !a_device ||
      !x_device || (reinterpret_cast<uintptr_t>(a_device) & 15) || (reinterpret_cast<uintptr_t>(x_device) & 15)) {
    noalloc_message(msg, msg_len, "invalid argument (device, n >= 1, nsys >= 1, 1 <= nrhs <= 16, 16-byte aligned "
                                  "device pointers)");
    return NEMOH_B200_EINVAL;
  }
  const size_t need = noalloc_bytes(n, nsys, nrhs);
  if (need > (size_t)NEMOH_B200_NOALLOC_SCRATCH_BYTES) {
    noalloc_message(msg, msg_len,
                    "scratch of " + std::to_string(need) + " bytes needed for n=" + std::to_string(n) +
                        ", nsys=" + std::to_string(nsys) + ", nrhs=" + std::to_string(nrhs) + " exceeds the fixed " +
                        std::to_string((size_t)NEMOH_B200_NOALLOC_SCRATCH_BYTES) + "-byte scratch");
    return NEMOH_B200_ECAPACITY;
  }
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
  auto fail = [&](cudaError_t e, const char* what) {
    noalloc_message(msg, msg_len, std::string(what) + ": " + cudaGetErrorString(e));
    if (prev >= 0) cudaSetDevice(prev);
    return NEMOH_B200_ECUDA;
  };
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(e, "cudaSetDevice");
  {
    const std::string bad = device_pointer_problem(device, {{a_device, "a_device"}, {x_device, "x_device"}});
    if (!bad.empty()) {
      noalloc_message(msg, msg_len, bad);
      if (prev >= 0) cudaSetDevice(prev);
      return NEMOH_B200_EINVAL;
    }
  }
  unsigned char* base = nullptr;
  {
    // set-up, once per device (the first call on the device): look up the
    // scratch array's address and raise the dynamic shared-memory limits
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess) return fail(e, "cudaGetSymbolAddress");
      const int trsm_smem = (2 * TB * MAX_RHS + TB * TB) * (int)sizeof(double2);
      const cudaError_t a[4] = {
          cudaFuncSetAttribute(zgemm_update_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               zgemm_smem<double2>()),
          cudaFuncSetAttribute(inv_diag_kernel<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               inv_diag_smem<double2>()),
          cudaFuncSetAttribute(trsm_fused_kernel<double2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               trsm_smem),
          cudaFuncSetAttribute(trsm_fused_kernel<double2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               trsm_smem)};
      for (cudaError_t x : a)
        if (x != cudaSuccess) return fail(x, "cudaFuncSetAttribute");
      g_noalloc_ptr[device] = static_cast<unsigned char*>(p);
    }
    base = g_noalloc_ptr[device];
  }
  const long long nblk = (n + TB - 1) / TB;
  int* status = reinterpret_cast<int*>(base);
  size_t off = noalloc_align(sizeof(int));
  double2* diag = reinterpret_cast<double2*>(base + off);
  off += noalloc_align((size_t)nsys * DIAG_SCRATCH * sizeof(double2));
  double2* inv = reinterpret_cast<double2*>(base + off);
  off += noalloc_align((size_t)(nsys * nblk * 2) * TB * TB * sizeof(double2));
  double2* y = reinterpret_cast<double2*>(base + off);

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BatchT<double2> b{reinterpret_cast<double2*>(a_device), (long long)n * n, n, diag};
  e = cudaMemsetAsync(status, 0, sizeof(int), st);
  if (e != cudaSuccess) return fail(e, "cudaMemsetAsync");
  // the FP64 no-pivot blocked LU of the context path, step by step
  for (int k = 0; k < n; k += LU_NB) {
    const int nb = std::min(LU_NB, n - k), rest = n - k - nb;
    const int nrb = (rest + LU_RB - 1) / LU_RB, ncb = (rest + LU_CB - 1) / LU_CB;
    lu_diag_kernel<double2><<<dim3(1, 1, nsys), LU_DIAG_THREADS, 0, st>>>(b, k, status);
    lu_panel_kernel<double2><<<dim3(std::max(1, nrb + ncb), 1, nsys), LU_PT, 0, st>>>(b, k, n);
    if (rest > 0) zgemm_update<double2>(b, k, nb, Rect{k + nb, n, k + nb, n}, nsys, st);
  }
  inv_diag_kernel<double2><<<dim3((unsigned)nblk, 1, nsys), INV_THREADS, inv_diag_smem<double2>(), st>>>(b, inv,
                                                                                                      (int)nblk);
  long long launches = 0;
  trsm_launch<double2>(b, inv, reinterpret_cast<double2*>(x_device), y, nsys, nrhs, st, launches);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(e, "kernel launch");
  int h_status = 0;
  e = cudaMemcpyAsync(&h_status, status, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return fail(e, "cudaMemcpyAsync");
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(e, "cudaStreamSynchronize");
  if (prev >= 0) cudaSetDevice(prev);
  if (h_status == ST_PIVOT) {
    noalloc_message(msg, msg_len, "PIVOT INFERIEUR A 1.E-20 (GAUSSZ)");
    return NEMOH_B200_EPIVOT;
  }
  if (h_status) {
    noalloc_message(msg, msg_len, "device error " + std::to_string(h_status));
    return NEMOH_B200_ECUDA;
  }
  return NEMOH_B200_OK;
}
