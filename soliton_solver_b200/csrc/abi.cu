// abi.cu -- C ABI of libsoliton_b200 (declared in include/soliton_b200.h).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <initializer_list>
#include <limits>
#include <mutex>
#include <type_traits>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda.h>
#include <cudaTypedefs.h>

#include "../../include/soliton_b200.h"
#include "common.cuh"
#include "flow.cuh"
#include "rk.cuh"
#include "coop.cuh"
#include "plain.cuh"
#include "batch.cuh"
#include "render.cuh"
#include "init.cuh"
#include "observe.cuh"
#include "adjoint.cuh"
#include "text.cuh"
#include "theories.cuh"
#define SSB_INSTANCE extern
#include "instances.cuh"

namespace ssb {
SSB_COOP_INSTANCES
SSB_BATCH_INSTANCES
SSB_PLAIN_INSTANCES
}

using namespace ssb;

namespace {

constexpr int TX = 16, TY = 64, NT = 256;  // fused tile: 16 x 64 sites, 256 threads
constexpr int COOP_MAX_TILES = 4096;        // energy partials kept for the cooperative step
constexpr int TRAJ_CAP = 1024;              // device trajectory slots used by ss_step
constexpr size_t STAGE_TAIL = 64 + 192;      // bytes of HostStage::host behind the trajectories: status, state
constexpr size_t ALIGN = 256;
// Tensor maps of a bound handle (halo boxes): phi and V of the caller's buffers and of the
// workspace's pair in the tile shapes of phases A and B, l1 and l2 in phase B's
enum { TM_A = 0, TM_B = 4, TM_L = 8, TM_COUNT = 10 };  // TM_A + 2 * pair + (0 phi, 1 V); TM_L + (0 l1, 1 l2)

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

#define CK(call)                                                                        \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) return fail(SS_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

size_t align_up(size_t v) { return (v + ALIGN - 1) / ALIGN * ALIGN; }

// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

// 3-D map over component planes (dims y, x, component) whose box is one staged
// tile: (TY + 8) x (TX + 4) x NF.  Fails (-> plain loads) when the buffer or its
// row pitch is not 16-byte aligned.
bool encode_tile_map(CUtensorMap* m, const void* ptr, size_t es, int X, int Y, int NF, int tx = TX, int ty = TY) {
  if (!ptr || ((uintptr_t)ptr) % 16 || ((size_t)Y * es) % 16) return false;
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)Y, (cuuint64_t)X, (cuuint64_t)NF};
  cuuint64_t strides[2] = {(cuuint64_t)Y * es, (cuuint64_t)X * Y * es};
  cuuint32_t box[3] = {(cuuint32_t)(ty + 8), (cuuint32_t)(tx + 4), (cuuint32_t)NF};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, es == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3,
                  const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

}  // namespace

// Mapped page-locked staging of a handle: the energy and err trajectories of one ss_step chunk and
// the status of the call, written by the kernels themselves, and behind them the step state as read
// back by read_state.  Page-locking a block costs about 60 us and releasing one waits for the device,
// so a destroyed handle's block is kept for the next handle: at most STAGE_KEEP blocks (17 KB each)
// in the process, the others are released.
struct HostStage {
  double* host = nullptr;
  double* dev = nullptr;  // its device address
  bool busy = false;      // a launch or copy that writes it has not been waited for
};

namespace {
constexpr size_t STAGE_KEEP = 4;
std::mutex g_stage_mutex;
HostStage g_stage_free[STAGE_KEEP];
size_t g_stage_count = 0;

cudaError_t stage_take(HostStage& s) {
  {
    std::lock_guard<std::mutex> lock(g_stage_mutex);
    while (g_stage_count) {
      const HostStage t = g_stage_free[--g_stage_count];
      cudaPointerAttributes a;  // a device reset in between takes the blocks with it
      if (cudaPointerGetAttributes(&a, t.host) == cudaSuccess && a.type == cudaMemoryTypeHost) {
        s = t;
        return cudaSuccess;
      }
      cudaGetLastError();
    }
  }
  HostStage t;
  cudaError_t e = cudaHostAlloc((void**)&t.host, 2 * TRAJ_CAP * sizeof(double) + STAGE_TAIL,
                                cudaHostAllocMapped | cudaHostAllocPortable);
  if (e == cudaSuccess && (e = cudaHostGetDevicePointer((void**)&t.dev, t.host, 0)) != cudaSuccess) cudaFreeHost(t.host);
  if (e == cudaSuccess) s = t;
  return e;
}
void stage_give(HostStage& s) {
  if (!s.host) return;
  if (!s.busy) {
    std::lock_guard<std::mutex> lock(g_stage_mutex);
    if (g_stage_count < STAGE_KEEP) {
      g_stage_free[g_stage_count++] = s;
      s = HostStage{};
      return;
    }
  }
  cudaFreeHost(s.host);  // waits for the device
  s = HostStage{};
}
}  // namespace

struct ss_handle {
  int theory = 0, precision = 0, nf = 0;
  double pf_raw[32] = {};  // the packed p_f as given (initial-condition kernels read it)
  Grid G{};
  Phys P{};
  size_t elem = 8;
  int nblocks = 0;        // 16 x 64 tiles (gradient, energy, densities)
  int plain_sum_blocks = 0, plain_max_blocks = 0;
  // bound buffers
  void* field = nullptr;
  void* vel = nullptr;
  char* ws = nullptr;
  size_t ws_bytes = 0;
  cudaStream_t stream = nullptr;
  // workspace carve (fused)
  StepState* st = nullptr;
  double* partial = nullptr;
  double* traj_E = nullptr;
  double* traj_err = nullptr;
  // fused flow buffers: l1, l2 and the second phi, V that steps alternate with
  void* l[4] = {nullptr, nullptr, nullptr, nullptr};
  void* phi2 = nullptr;
  void* vel2 = nullptr;
  // plain extras
  void* k[4] = {nullptr, nullptr, nullptr, nullptr};
  void* temp = nullptr;
  void* eg = nullptr;
  double* d1 = nullptr;
  double* d2 = nullptr;
  double* en = nullptr;
  double* entmp = nullptr;
  double E_last_host = NAN;
  std::vector<double> host_partial;
  bool pinned = false;  // a stage's variant was pinned (ss_set_variant): the two-launch step runs it
  int coop = 0;  // small lattices: 1 + tile shape of the cooperative step (0: two launches per step)
  // TMA maps of the bound buffers (index constants TM_*)
  CUtensorMap tm[TM_COUNT];
  bool tma = false;
  int num_sms = 148;
  // per flow mode: 1 = persistent pipelined kernel, 0 = one tile per CTA (autotuned).  The
  // gradient's (0) and phase B's (3, 4) are read; 1, 2, 5 and fuse23 are kept as pinned.  The
  // gradient starts with one tile per CTA: us FP32 2048^2, pipelined -> one tile, chiral magnet 43 ->
  // 33, baby Skyrme 48 -> 33, Abelian Higgs 47 -> 33, s+id 77 -> 62; 1024^2 13.5 -> 10.5, 14.5 -> 12.4,
  // 14.5 -> 10.5, 22.7 -> 18.6.
  int use_pipe[N_FLOW_MODES] = {0, 1, 1, 1, 1, 1, 0};
  float tune_ms[N_FLOW_MODES][2] = {};
  int fuse23 = 1;  // stages 2 and 3 in one kernel (TMA staging only)
  long long wait_cycles = WAIT_CYCLES;
  mutable int inject_timeout = 0;  // test hook, consumed by the next launch that waits
  cudaGraphExec_t graph = nullptr;  // captured n-step relaxation (ss_graph_create)
  const double* force = nullptr;    // FP64 flows: field added to the gradient rows (ss_set_forcing)
  HostStage stage;  // taken on first use
  ~ss_handle() {
    if (graph) cudaGraphExecDestroy(graph);
    stage_give(stage);
  }
};

namespace {

// ---------------------------------------------------------------------------
// workspace layout
// ---------------------------------------------------------------------------
size_t layout(ss_handle* h, char* base) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = base ? base + off : nullptr;
    off = align_up(off + bytes);
    return p;
  };
  const size_t field_bytes = h->elem * (size_t)h->nf * (size_t)h->G.N;
  h->st = (StepState*)take(sizeof(StepState));
  // partials: per tile of 16 rows one for each quantity of an observables pass, or one per
  // tile of 8 rows in the step's phases
  const size_t np = (size_t)std::max(std::max(OBS_MAX * h->nblocks, COOP_MAX_TILES), std::max(h->plain_sum_blocks, h->plain_max_blocks));
  h->partial = (double*)take(np * sizeof(double));
  h->traj_E = (double*)take(TRAJ_CAP * sizeof(double));
  h->traj_err = (double*)take(TRAJ_CAP * sizeof(double));
  if (h->precision == SS_PLAIN_FP64) {
    for (int i = 0; i < 4; ++i) h->k[i] = take(field_bytes);
    for (int i = 0; i < 4; ++i) h->l[i] = take(field_bytes);
    h->temp = take(field_bytes);
    h->eg = take(field_bytes);
    h->d1 = (double*)take(2 * field_bytes);
    h->d2 = (double*)take(4 * field_bytes);
    h->en = (double*)take((size_t)h->G.N * sizeof(double));
    h->entmp = (double*)take((size_t)h->G.N * sizeof(double));
  } else {
    for (int i = 0; i < 2; ++i) h->l[i] = take(field_bytes);
    h->l[2] = h->l[3] = nullptr;
    h->phi2 = take(field_bytes);
    h->vel2 = take(field_bytes);
    take(field_bytes);  // unused: callers know the workspace as five field-sized buffers at least
  }
  return off;
}

// Interior tiles load and store y-adjacent site pairs of global buffers as one vector: rows of
// even length in buffers (null: none) aligned to two elements of `es` bytes.
int site_pairs(const Grid& G, size_t es, std::initializer_list<const void*> bufs) {
  bool ok = G.Y % 2 == 0;
  for (const void* p : bufs) ok = ok && (uintptr_t)p % (2 * es) == 0;
  return ok ? 1 : 0;
}

// ---------------------------------------------------------------------------
// parameter decoding (packed arrays of each theory's pack_device_params)
// ---------------------------------------------------------------------------
int decode(ss_handle* h, int theory, const int32_t* p_i, int n_i, const double* p_f, int n_f) {
  static const int need_i[4] = {16, 20, 12, 14};
  static const int need_f[4] = {15, 14, 11, 25};
  static const int theory_nf[4] = {4, 3, 4, 6};
  if (theory < 0 || theory > 3) return fail(SS_ERR_ARG, "unknown theory id %d", theory);
  if (!p_i || !p_f) return fail(SS_ERR_ARG, "p_i/p_f must not be NULL");
  if (n_i < need_i[theory] || n_f < need_f[theory])
    return fail(SS_ERR_ARG, "packed params too short for theory %d: n_i=%d (need %d), n_f=%d (need %d)", theory, n_i,
                need_i[theory], n_f, need_f[theory]);
  for (int i = 0; i < n_f && i < 32; ++i) h->pf_raw[i] = p_f[i];
  Grid& G = h->G;
  G.X = p_i[0];
  G.Y = p_i[1];
  G.halo = p_i[2];
  const int nc = p_i[3], nf = p_i[4];
  if (G.X < 1 || G.Y < 1) return fail(SS_ERR_ARG, "xlen/ylen must be positive (got %d, %d)", G.X, G.Y);
  if (nc != 2) return fail(SS_ERR_ARG, "number_coordinates must be 2 (got %d)", nc);
  if (nf != theory_nf[theory])
    return fail(SS_ERR_ARG, "number_total_fields=%d but theory %d has %d components", nf, theory, theory_nf[theory]);
  if (G.halo < 2) return fail(SS_ERR_ARG, "halo must be >= 2 for the 5-point stencils (got %d)", G.halo);
  G.N = (long long)G.X * G.Y;
  if ((long long)p_i[5] != G.N || (long long)p_i[6] != G.N * nf)
    return fail(SS_ERR_ARG, "p_i[5]/p_i[6] (dim_grid/dim_fields) inconsistent with xlen*ylen*nf");
  G.killkinen = p_i[7] ? 1 : 0;
  G.unit_mag = p_i[9] ? 1 : 0;
  G.pairs = site_pairs(G, 1, {});
  G.lsx = p_f[2];
  G.lsy = p_f[3];
  G.dA = p_f[4];
  G.dt = p_f[5];
  G.ihx = 1.0 / G.lsx;
  G.ihy = 1.0 / G.lsy;
  G.ihx2 = 1.0 / (G.lsx * G.lsx);
  G.ihy2 = 1.0 / (G.lsy * G.lsy);
  G.ih2dA = 1.0 / (2.0 * G.dA);
  if (!(G.lsx > 0) || !(G.lsy > 0) || !std::isfinite(G.lsx) || !std::isfinite(G.lsy) || !std::isfinite(G.dA) ||
      !std::isfinite(G.dt))
    return fail(SS_ERR_ARG, "lattice spacings / time step must be finite and positive");
  h->nf = nf;
  {
    const double c12 = 1.0 / 12.0, c23 = 2.0 / 3.0, c43 = 4.0 / 3.0;
    double* k = G.kd;
    k[GK_C23HX] = c23 * G.ihx;   k[GK_MC12HX] = -c12 * G.ihx;
    k[GK_C43HX2] = c43 * G.ihx2; k[GK_MC12HX2] = -c12 * G.ihx2;
    k[GK_C23HY] = c23 * G.ihy;   k[GK_MC12HY] = -c12 * G.ihy;
    k[GK_C43HY2] = c43 * G.ihy2; k[GK_MC12HY2] = -c12 * G.ihy2;
    k[GK_C43HD] = c43 * G.ih2dA; k[GK_MC12HD] = -c12 * G.ih2dA;
    k[GK_DT] = G.dt; k[GK_MDT] = -G.dt; k[GK_HDT] = 0.5 * G.dt; k[GK_DT6] = G.dt / 6.0; k[GK_SIXTH] = 1.0 / 6.0;
    for (int i = 0; i < 16; ++i) G.kf[i] = (float)G.kd[i];
  }
  Phys& P = h->P;
  memset(&P, 0, sizeof(P));
  switch (theory) {
    case SS_THEORY_CHIRAL_MAGNET: {
      if (p_i[10] != 3) return fail(SS_ERR_ARG, "chiral magnet needs number_magnetization_fields=3");
      P.c[0] = p_f[6];
      P.c[1] = p_f[7];
      P.c[2] = p_f[8];
      double D00 = 0, D01 = 0, D10 = 0, D11 = 0;  // chiral_magnet/kernels.py:151-160
      if (p_i[11]) {
        D00 = -1.0; D11 = -1.0;
      } else if (p_i[12]) {
        D01 = -1.0; D10 = 1.0;
      } else if (p_i[13]) {
        D00 = 1.0; D11 = -1.0;
      } else if (p_i[14]) {
        const double s = 0.7071067811865476;
        D00 = -s; D01 = -s; D10 = s; D11 = -s;
      }
      P.c[3] = D00; P.c[4] = D01; P.c[5] = D10; P.c[6] = D11;
      P.k[0] = p_i[15] ? 1 : 0;
      if (P.k[0] && !(P.c[2] != 0.0)) return fail(SS_ERR_ARG, "demag needs coup_mu != 0");
      break;
    }
    case SS_THEORY_BABY_SKYRME: {
      if (p_i[10] != 3) return fail(SS_ERR_ARG, "baby Skyrme needs number_magnetization_fields=3");
      P.c[0] = p_f[6];
      P.c[1] = p_f[7];
      for (int i = 0; i < 8; ++i) P.k[i] = p_i[11 + i] ? 1 : 0;
      P.k[8] = p_i[19];
      if (P.k[6] && P.k[8] < 1) return fail(SS_ERR_ARG, "broken potential needs N >= 1");
      break;
    }
    case SS_THEORY_GINZBURG_LANDAU: {
      P.c[0] = p_f[6];
      P.c[1] = p_f[7];
      P.c[2] = p_f[8];
      P.c[3] = p_f[9];
      if (!(P.c[0] != 0.0)) return fail(SS_ERR_ARG, "q must be nonzero");
      break;
    }
    case SS_THEORY_ANISOTROPIC: {
      for (int i = 0; i < 11; ++i) P.c[i] = p_f[6 + i];
      const double a1 = p_f[8], a2 = p_f[9], b1 = p_f[10], b2 = p_f[11], b3 = p_f[12], b4 = p_f[13];
      const double u1 = p_f[17], u2 = p_f[18], th = p_f[19];
      // vacuum energy density subtracted per site (anisotropic_superconductor/kernels.py:169)
      P.c[11] = a1 * u1 * u1 + a2 * u2 * u2 + b1 * u1 * u1 * u1 * u1 + b2 * u2 * u2 * u2 * u2 + b3 * u1 * u1 * u2 * u2 +
                2.0 * b4 * u1 * u1 * u2 * u2 * std::cos(2.0 * th);
      if (!(P.c[1] != 0.0)) return fail(SS_ERR_ARG, "Q must be nonzero");
      break;
    }
  }
  switch (theory) {
    case SS_THEORY_CHIRAL_MAGNET: ChiralMagnet::derive(P); break;
    case SS_THEORY_BABY_SKYRME: BabySkyrme::derive(P); break;
    case SS_THEORY_GINZBURG_LANDAU: GinzburgLandau::derive(P); break;
    case SS_THEORY_ANISOTROPIC: Anisotropic::derive(P); break;
  }
  for (int i = 0; i < 24; ++i) P.cf[i] = (float)P.c[i];
  return SS_OK;
}

int check_bound(const ss_handle* h) {
  if (!h) return fail(SS_ERR_ARG, "NULL handle");
  if (!h->ws) return fail(SS_ERR_STATE, "no workspace bound: call ss_bind first");
  return SS_OK;
}

// Tile shapes of the cooperative step (rows, columns, threads; SPLIT: two threads per site
// pair, one per stencil field, which takes FP64 baby Skyrme 128^2 from 11.4 to 9.1 us per
// step).  8 x 32 tiles hold FP32 lattices of up to ~110 000 sites (three CTAs per SM), 16 x 32
// up to ~220 000, 16 x 64 up to ~300 000; about half that in FP64.
constexpr int N_COOP_SHAPES = 3;
constexpr int COOP_TX[N_COOP_SHAPES] = {8, 16, 16};
constexpr int COOP_TY[N_COOP_SHAPES] = {32, 32, 64};
constexpr int COOP_NT[N_COOP_SHAPES] = {256, 128, 256};
constexpr bool COOP_SPLIT[N_COOP_SHAPES] = {true, false, false};
int coop_tiles(const Grid& G, int shape) {
  const long long t = (long long)((G.X + COOP_TX[shape] - 1) / COOP_TX[shape]) * ((G.Y + COOP_TY[shape] - 1) / COOP_TY[shape]);
  return (int)std::min(t, 0x7fffffffLL);
}

// Opt a kernel into more than 48 KB of dynamic shared memory, once per device.
// `done` is owned by the caller's template instantiation.
template <class K>
void set_smem(K kernel, size_t bytes, unsigned long long& done) {
  if (bytes <= 32 * 1024) return;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (done >> dev) & 1ULL) return;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (dev < 64) done |= 1ULL << dev;
}

dim3 grid_1d(long long n) {
  long long b = (n + 255) / 256;
  if (b > 148 * 16) b = 148 * 16;
  if (b < 1) b = 1;
  return dim3((unsigned)b);
}

// ---------------------------------------------------------------------------
// per-(theory, precision) implementation
// ---------------------------------------------------------------------------
template <class TH, typename R>
struct Fused {
  static constexpr size_t BUF = tile_buf_bytes<R, TH::NF, TX, TY>();

  // the gradient hook: one tile per CTA, or (FP32) persistent and TMA-pipelined
  static constexpr int PIPE_STAGES = 212 * 1024 / BUF > 4 ? 4 : (int)(212 * 1024 / BUF);
  template <bool TMA_>
  static int launch_grad_tile(const ss_handle* h, const FlowArgs<R>& A) {
    auto k = flow_kernel<TH, R, TX, TY, NT, TMA_>;
    static unsigned long long done = 0;
    set_smem(k, BUF, done);
    k<<<h->nblocks, NT, BUF, h->stream>>>(A);
    CK(cudaGetLastError());
    return SS_OK;
  }
  // whether a mode has a pipelined variant: the gradient's for FP32, phase B's (M_S3, M_S4) for both
  // precisions; phase A's (M_S1 and M_S2) is accepted for FP32 and ignored
  static bool uses_pipe(int mode) { return sizeof(R) == 4 || mode == M_S3 || mode == M_S4; }

  // tma: use the TMA-staged instantiations (A.tm_phi must describe A.phi)
  static int launch(const ss_handle* h, const FlowArgs<R>& A0, bool tma) {
    FlowArgs<R> A = A0;
    A.tx_extra = take_injection(h, tma);
    if (!tma) return launch_grad_tile<false>(h, A);
    if constexpr (sizeof(R) == 4) {
      if (h->use_pipe[M_GRAD]) {
        auto k = flow_kernel_pipe<TH, R, TX, TY, 2 * NT, PIPE_STAGES>;
        static unsigned long long done = 0;
        set_smem(k, PIPE_STAGES * BUF, done);
        k<<<std::min(h->nblocks, h->num_sms), 2 * NT, PIPE_STAGES * BUF, h->stream>>>(A);
        CK(cudaGetLastError());
        return SS_OK;
      }
    }
    return launch_grad_tile<true>(h, A);
  }
  // bytes the next TMA barrier expects beyond its loads (the injected timeout, consumed)
  static unsigned take_injection(const ss_handle* h, bool tma) {
    if (!tma || !h->inject_timeout) return 0u;
    h->inject_timeout = 0;
    return 16u;
  }

  static FlowArgs<R> base_args(const ss_handle* h) {
    FlowArgs<R> A;
    memset(&A, 0, sizeof(A));
    A.wait_cycles = h->wait_cycles;
    A.G = h->G;
    A.P = h->P;
    A.st = h->st;
    return A;
  }

  // ---- the RK4 step (rk.cuh) ------------------------------------------------
  static constexpr int TXA = StepShape<TH, R, PH_A>::TX;

  // tensor maps of a phase's inputs (phi and V of the pair that A.phi belongs to)
  static StepMaps phase_maps(const ss_handle* h, const StepArgs<R>& A, int maps) {
    const int pair = (const void*)A.phi == h->phi2 ? 1 : 0;
    return StepMaps{h->tm[maps + 2 * pair], h->tm[maps + 2 * pair + 1], h->tm[TM_L], h->tm[TM_L + 1]};
  }
  template <bool TMA_, int PH>
  static int launch_phase(const ss_handle* h, StepArgs<R>& A) {
    using SH = StepShape<TH, R, PH, TMA_>;
    constexpr size_t smem = step_smem<TH, R, PH, TMA_>();
    auto k = step_kernel<TH, R, TMA_, PH>;
    static unsigned long long done = 0;  // one per instantiation
    set_smem(k, smem, done);
    A.tx_extra = take_injection(h, TMA_);
    const int tiles = ((h->G.X + SH::TX - 1) / SH::TX) * ((h->G.Y + TY - 1) / TY);
    k<<<tiles, SH::NT, smem, h->stream>>>(phase_maps(h, A, PH == PH_B ? TM_B : TM_A), A);
    CK(cudaGetLastError());
    return SS_OK;
  }
  static int launch_phase_pipe(const ss_handle* h, StepArgs<R>& A) {
    using SH = PipeShape<TH, R>;
    auto k = step_kernel_pipe<TH, R>;
    static unsigned long long done = 0;  // one per instantiation
    set_smem(k, SH::SMEM, done);
    A.tx_extra = take_injection(h, true);
    const int tiles = ((h->G.X + SH::TX - 1) / SH::TX) * ((h->G.Y + SH::TY - 1) / SH::TY);
    k<<<std::min(tiles, SH::CTAS * h->num_sms), SH::NT, SH::SMEM, h->stream>>>(phase_maps(h, A, TM_B), A);
    CK(cudaGetLastError());
    return SS_OK;
  }
  static int launch_energy(const ss_handle* h, StepArgs<R>& A, const CUtensorMap& map) {
    using SH = EnergyPipe<TH, R>;
    auto k = step_energy_pipe<TH, R>;
    static unsigned long long done = 0;  // one per instantiation
    set_smem(k, SH::SLOTS * SH::SLOT, done);
    A.tx_extra = take_injection(h, true);
    const int tiles = ((h->G.X + SH::TX - 1) / SH::TX) * ((h->G.Y + SH::TY - 1) / SH::TY);
    k<<<std::min(tiles, SH::CTAS * h->num_sms), SH::NT, SH::SLOTS * SH::SLOT, h->stream>>>(map, A);
    CK(cudaGetLastError());
    return SS_OK;
  }
  template <int PH>
  static int launch_phase(const ss_handle* h, StepArgs<R>& A) {
    if (!h->tma) return launch_phase<false, PH>(h, A);
    if constexpr (PH == PH_E) {
      return launch_energy(h, A, phase_maps(h, A, TM_A).phi);
    } else {
      if (PH == PH_B && h->use_pipe[M_S4]) return launch_phase_pipe(h, A);
      return launch_phase<true, PH>(h, A);
    }
  }

  static StepArgs<R> step_args(const ss_handle* h) {
    StepArgs<R> A;
    memset(&A, 0, sizeof(A));
    A.wait_cycles = h->wait_cycles;
    A.G = h->G;
    A.P = h->P;
    A.st = h->st;
    A.partial = h->partial;
    A.force = h->force;
    A.l1 = A.out_l1 = (R*)h->l[0];
    A.l2 = A.out_l2 = (R*)h->l[1];
    A.E_idx = -1;
    A.err_idx = -1;
    A.prev_energy = NAN;
    return A;
  }
  // phi and V of buffer pair `pair` (0: the caller's, 1: the workspace's) as a phase's inputs
  static void set_input(const ss_handle* h, StepArgs<R>& A, int pair) {
    A.phi = (const R*)(pair ? h->phi2 : h->field);
    A.vel = (const R*)(pair ? h->vel2 : h->vel);
  }

  // ---- small lattices: all steps of a call in one cooperative launch (coop.cuh) ----
  template <int S, int VW>
  static int launch_coop(const ss_handle* h, const StepArgs<R>& A, const CoopArgs<R>& C, int* capacity) {
    constexpr int CX = COOP_TX[S], CY = COOP_TY[S], CN = COOP_NT[S];
    using CT = CoopTile<TH, R, CX, CY, CN, COOP_SPLIT[S]>;
    if constexpr (CT::SMEM > 220 * 1024) {
      if (capacity) *capacity = 0;
      return capacity ? SS_OK : fail(SS_ERR_ARG, "bad cooperative shape");
    } else {
      // too many tiles by the kernel's bounds alone: the kernel is not loaded to ask for its occupancy
      // (20 to 200 us for the first bind of a process whose lattice can never use it)
      if (capacity && coop_tiles(h->G, S) > coop_ctas<TH, R, CX, CY, CN, COOP_SPLIT[S]>() * h->num_sms) {
        *capacity = 0;
        return SS_OK;
      }
      auto k = coop_step_kernel<TH, R, CX, CY, CN, COOP_SPLIT[S], VW>;
      static unsigned long long done = 0;
      set_smem(k, CT::SMEM, done);
      if (capacity) {  // co-resident CTAs
        int occ = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, CN, CT::SMEM) != cudaSuccess) occ = 0;
        *capacity = occ * h->num_sms;
        return SS_OK;
      }
      void* args[2] = {const_cast<StepArgs<R>*>(&A), const_cast<CoopArgs<R>*>(&C)};
      CK(cudaLaunchCooperativeKernel((const void*)k, dim3(coop_tiles(h->G, S)), dim3(CN), args, CT::SMEM, h->stream));
      return SS_OK;
    }
  }
  static int coop_any(const ss_handle* h, int shape, const StepArgs<R>& A, const CoopArgs<R>& C, int* capacity) {
    constexpr int VW = 16 / (int)sizeof(R);
    switch (shape) {
      case 0: return h->tma ? launch_coop<0, VW>(h, A, C, capacity) : launch_coop<0, 1>(h, A, C, capacity);
      case 1: return h->tma ? launch_coop<1, VW>(h, A, C, capacity) : launch_coop<1, 1>(h, A, C, capacity);
    }
    return h->tma ? launch_coop<2, VW>(h, A, C, capacity) : launch_coop<2, 1>(h, A, C, capacity);
  }
  // whether the lattice's tiles of `shape` are all resident at once
  static bool coop_fits(const ss_handle* h, int shape) {
    const long long t = coop_tiles(h->G, shape);
    int cap = 0;
    return t <= COOP_MAX_TILES && coop_any(h, shape, StepArgs<R>{}, CoopArgs<R>{}, &cap) == SS_OK && t <= cap;
  }
  static int step_coop(ss_handle* h, int n, double prev, double* E_dev, double* err_dev, int* status_out) {
    StepArgs<R> A = step_args(h);
    // other work on the GPU may hold up a CTA of the grid
    A.wait_cycles = 16 * std::min(h->wait_cycles, std::numeric_limits<long long>::max() / 16);
    A.tx_extra = h->inject_timeout;  // the grid barrier expects one CTA more than there are
    h->inject_timeout = 0;
    CoopArgs<R> C;
    C.phi[0] = (R*)h->field;
    C.phi[1] = (R*)h->phi2;
    C.vel[0] = (R*)h->vel;
    C.vel[1] = (R*)h->vel2;
    C.l1 = (R*)h->l[0];
    C.l2 = (R*)h->l[1];
    C.status_out = status_out;
    for (int done = 0; done < n; done += C.n) {
      C.n = std::min(n - done, 4096);
      A.prev_energy = done ? NAN : prev;
      A.E_traj = E_dev ? E_dev + done : nullptr;
      A.err_traj = err_dev ? err_dev + done : nullptr;
      const int rc = coop_any(h, h->coop - 1, A, C, nullptr);
      if (rc) return rc;
    }
    return SS_OK;
  }

  static int launch_a2(const ss_handle* h, const StepArgs<R>& A) {
    constexpr size_t smem = step_smem<TH, R, PH_A, false>();
    using SH = StepShape<TH, R, PH_A, false>;
    const long long tiles = (long long)((h->G.X + SH::TX - 1) / SH::TX) * ((h->G.Y + TY - 1) / TY);
    auto go = [&](auto k, unsigned long long& done) -> int {
      set_smem(k, smem, done);
      k<<<(int)std::min<long long>(tiles, 2 * h->num_sms), SH::NT, smem, h->stream>>>(A);
      CK(cudaGetLastError());
      return SS_OK;
    };
    static unsigned long long done_fused = 0, done_plain = 0;
    return h->tma ? go(step_a2_kernel<TH, R, true>, done_fused) : go(step_a2_kernel<TH, R, false>, done_plain);
  }
  // flows whose energy rises (psi of the chiral magnet's demag field is maximised): nearly
  // every step is arrested, and phase A predicts it
  static bool saddle_flow(const ss_handle* h) {
    return h->P.k[0] && h->G.killkinen;
  }

  // n flow steps of the bound buffers, in place; trajectories to device arrays (nullable)
  // status_out (nullable, device-visible): the finish kernel copies the call's status there
  static int step(ss_handle* h, int n, double prev, double* E_dev, double* err_dev, int* status_out = nullptr) {
    if (n <= 0) return SS_OK;
    if (h->coop) return step_coop(h, n, prev, E_dev, err_dev, status_out);
    StepArgs<R> A = step_args(h);
    A.E_traj = E_dev;
    A.err_traj = err_dev;
    int rc, cur = 0;
    // An odd count would end in the other pair.  Its first phase A copies phi and V there on the
    // way, so that phase B writes the caller's buffers and nothing is copied back.  4096^2 chiral
    // magnet FP32, one-step call: phase A 244 -> 266 us, phase E 165 -> 122, finish 137 -> 6.
    const bool land = n & 1;
    for (int s = 0; s < n; ++s, cur ^= 1) {
      A.copy_phi = land && s == 0 ? (R*)h->phi2 : nullptr;
      A.copy_vel = land && s == 0 ? (R*)h->vel2 : nullptr;
      // A: l1, l2; energy of phi (the previous step's result) and its arrest test
      A.with_energy = A.arrest_update = s > 0;
      A.E_idx = s - 1;
      A.init_state = s == 0;
      A.prev_energy = prev;
      set_input(h, A, cur);
      if constexpr (std::is_same_v<TH, ChiralMagnet>) A.predict = s > 0 && saddle_flow(h);
      if ((rc = launch_phase<PH_A>(h, A))) return rc;
      A.init_state = 0;
      if constexpr (std::is_same_v<TH, ChiralMagnet>) {
        if (A.predict && (rc = launch_a2(h, A))) return rc;
      }
      if (A.copy_phi) cur = 1;
      // B: phi' and V' into the other pair, err
      A.err_idx = s;
      A.phi_out = (R*)(cur ? h->field : h->phi2);
      A.vel_out = (R*)(cur ? h->vel : h->vel2);
      set_input(h, A, cur);
      if ((rc = launch_phase<PH_B>(h, A))) return rc;
    }
    // trailing energy of the final field (cur is 0: the caller's) and its arrest test
    A.predict = 0;
    A.with_energy = A.arrest_update = 1;
    A.E_idx = n - 1;
    set_input(h, A, 0);
    if ((rc = launch_phase<PH_E>(h, A))) return rc;
    const long long nfN = (long long)h->nf * h->G.N;
    step_finish_kernel<R><<<grid_1d(nfN), 256, 0, h->stream>>>((R*)h->vel, nfN, h->st, status_out);
    CK(cudaGetLastError());
    return SS_OK;
  }

  // Time the step's two phases and the two staging variants of the gradient on the bound
  // buffers (the faster gradient variant is kept).  Writes only workspace scratch; the
  // energy reduction leaves the arrest state and the trajectories alone.
  static int autotune(ss_handle* h, int iters) {
    if (!h->tma) return SS_OK;
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    auto timed = [&](float& out, auto&& go) -> int {
      int rc = go();  // warm-up
      if (rc) return rc;
      CK(cudaEventRecord(e0, h->stream));
      for (int i = 0; i < iters && rc == SS_OK; ++i) rc = go();
      CK(cudaEventRecord(e1, h->stream));
      CK(cudaEventSynchronize(e1));
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, e0, e1));
      out = ms / iters;
      return rc;
    };
    StepArgs<R> A = step_args(h);
    A.with_energy = 1;
    A.phi_out = (R*)h->phi2;
    A.vel_out = (R*)h->vel2;
    int rc = SS_OK;
    for (int m : {(int)M_S1, (int)M_S4}) {
      const bool two = m == M_S4;
      for (int v = 0; v < 2 && !rc; ++v) {
        if (two) h->use_pipe[M_S3] = h->use_pipe[M_S4] = v;
        set_input(h, A, 0);
        if (v == 0 || two)
          rc = timed(h->tune_ms[m][v], [&]() { return m == M_S1 ? launch_phase<PH_A>(h, A) : launch_phase<PH_B>(h, A); });
        else
          h->tune_ms[m][1] = h->tune_ms[m][0];
      }
      if (two) h->use_pipe[M_S3] = h->use_pipe[M_S4] = h->tune_ms[m][1] <= h->tune_ms[m][0] ? 1 : 0;
      for (int v = 0; v < 2; ++v) h->tune_ms[m == M_S1 ? M_S2 : M_S3][v] = h->tune_ms[m][v];
    }
    for (int v = 0; v < 2; ++v) h->tune_ms[M_S23][v] = h->tune_ms[M_S1][0] + h->tune_ms[M_S4][h->use_pipe[M_S4]];
    if (uses_pipe(M_GRAD)) {
      FlowArgs<R> F = base_args(h);
      F.phi = (const R*)h->field;
      F.out_l = (R*)h->l[0];
      const bool tma = encode_tile_map(&F.tm_phi, F.phi, sizeof(R), h->G.X, h->G.Y, TH::NF);
      for (int v = 0; v < 2 && tma && !rc; ++v) {
        h->use_pipe[M_GRAD] = v;
        rc = timed(h->tune_ms[M_GRAD][v], [&]() { return launch(h, F, true); });
      }
      h->use_pipe[M_GRAD] = h->tune_ms[M_GRAD][1] <= h->tune_ms[M_GRAD][0] ? 1 : 0;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
  }

  static int gradient(ss_handle* h, const void* field, void* eg, void* l_out, int raw = 0,
                      const double* scale = nullptr) {
    FlowArgs<R> A = base_args(h);
    A.grad_raw = raw;
    A.scale = scale;
    A.phi = (const R*)field;
    A.out_eg = (R*)eg;
    A.out_l = (R*)l_out;
    A.G.pairs = site_pairs(h->G, sizeof(R), {eg, l_out});
    const bool tma = encode_tile_map(&A.tm_phi, field, sizeof(R), h->G.X, h->G.Y, TH::NF);
    return launch(h, A, tma);
  }

  // dE_h/dphi / dA of the discrete energy sum (true rows, unprojected), optionally
  // minus the flow's functional derivative in the same rows (FP64 fields)
  static int energy_gradient_exact(ss_handle* h, const void* field, double* out, double* q, double* sub) {
    if (sub) {
      int rc = Fused<TH, double>::gradient(h, field, sub, nullptr, 1);
      if (rc) return rc;
    }
    exact_partials_kernel<TH, R><<<grid_1d(h->G.N), 256, 0, h->stream>>>((const R*)field, out, q, h->G, h->P);
    CK(cudaGetLastError());
    exact_transpose_kernel<double><<<grid_1d((long long)TH::NF * h->G.N), 256, 0, h->stream>>>(out, q, sub, TH::NF,
                                                                                              h->G);
    CK(cudaGetLastError());
    return SS_OK;
  }

  // the observable: exact FP64 stencil of the stored values for every precision
  static int energy(ss_handle* h, const void* field) {
    if constexpr (sizeof(R) == 8) {  // the flow's own energy pass: FP64 jets are the exact differences
      StepArgs<R> S = step_args(h);
      S.with_energy = 1;
      S.phi = (const R*)field;
      CUtensorMap map{};
      const bool tma = encode_tile_map(&map, field, sizeof(R), h->G.X, h->G.Y, TH::NF, TXA, TY);
      return tma ? launch_energy(h, S, map) : launch_phase<false, PH_E>(h, S);
    }
    ObsList L{};
    L.n = 1;
    L.comps = ~0u;
    return observe(h, field, nullptr, true, L);
  }

  // FP64 energy of the sphere projection of `field` (element type R).  The FP64 copy
  // goes to the start of the l-buffer region, which holds at least 8 * nf * N bytes
  // for every precision (two FP32 l buffers, or one FP64 one) and is free between steps.
  static int energy_projected(ss_handle* h, const void* field) {
    double* copy = (double*)h->l[0];
    convert_kernel<R, double, TH::NF, TH::NMAG><<<grid_1d(h->G.N), 256, 0, h->stream>>>(
        (const R*)field, copy, h->G.N, TH::CONSTRAINED && h->G.unit_mag);
    CK(cudaGetLastError());
    return Fused<TH, double>::energy(h, copy);
  }

  static unsigned obs_comps(int kind, int which) {
    return kind == D_ENERGY ? ~0u : kind == D_CHARGE ? TH::charge_comps(which) : TH::coupling_comps(which);
  }
  // the quantities of L (comps filled in) of `field`: their sums (reduce) and, for one of
  // them, its density (nullable)
  static int observe(const ss_handle* h, const void* field, double* dens, bool reduce, const ObsList& L,
                     bool allow_tma = true) {
    CUtensorMap map{};
    const bool tma = allow_tma && encode_tile_map(&map, field, sizeof(R), h->G.X, h->G.Y, TH::NF);
    auto go = [&](auto k, unsigned long long& done) -> int {
      set_smem(k, BUF, done);
      k<<<h->nblocks, NT, BUF, h->stream>>>(map, (const R*)field, dens, reduce ? h->partial : nullptr, h->st, L, h->G,
                                            h->P, h->wait_cycles, take_injection(h, tma));
      CK(cudaGetLastError());
      return SS_OK;
    };
    static unsigned long long done[4] = {};  // one per instantiation
    if (L.n == 1)
      return tma ? go(observe_kernel<TH, R, TX, TY, NT, true, 1>, done[0])
                 : go(observe_kernel<TH, R, TX, TY, NT, false, 1>, done[1]);
    return tma ? go(observe_kernel<TH, R, TX, TY, NT, true, OBS_MAX>, done[2])
               : go(observe_kernel<TH, R, TX, TY, NT, false, OBS_MAX>, done[3]);
  }
  static int density(ss_handle* h, const void* field, double* dens, bool reduce, int kind, int which) {
    ObsList L{};
    L.n = 1;
    L.kind[0] = kind;
    L.which[0] = which;
    L.comps = obs_comps(kind, which);
    return observe(h, field, dens, reduce, L);
  }

  static int rk4_stage(ss_handle* h, void* k_out, const void* vel, const void* l_in, void* temp, const void* field,
                       const void* k_prev, double factor) {
    const long long n = (long long)h->nf * h->G.N;
    rk4_stage_kernel<R><<<grid_1d(n), 256, 0, h->stream>>>((R*)k_out, (const R*)vel, (const R*)l_in, (R*)temp,
                                                           (const R*)field, (const R*)k_prev, (R)factor, (R)h->G.dt, n);
    CK(cudaGetLastError());
    return SS_OK;
  }

  static int rk4_finalize(ss_handle* h, void* vel, void* field, const void* const* k, const void* const* l) {
    rk4_finalize_kernel<R, TH::NF, TH::NMAG><<<grid_1d(h->G.N), 256, 0, h->stream>>>(
        (R*)vel, (R*)field, (const R*)k[0], (const R*)k[1], (const R*)k[2], (const R*)k[3], (const R*)l[0],
        (const R*)l[1], (const R*)l[2], (const R*)l[3], h->G.N, TH::CONSTRAINED && h->G.unit_mag);
    CK(cudaGetLastError());
    return SS_OK;
  }
};

template <class TH>
struct Plain {
  static dim3 blocks(const ss_handle* h) { return dim3((h->G.X + 7) / 8, (h->G.Y + 7) / 8); }

  static int gradient(ss_handle* h, const double* F, double* l_out, double* eg) {
    plain_gradient_kernel<TH><<<blocks(h), dim3(8, 8), 0, h->stream>>>(l_out, F, h->d1, h->d2, eg, h->G, h->P);
    CK(cudaGetLastError());
    return SS_OK;
  }

  static int reduce(ss_handle* h, const double* var, long long size, int is_max, double* out) {
    const int nb = (int)((size + 1023) / 1024);
    plain_reduce_kernel<<<nb, 1024, 0, h->stream>>>(var, h->partial, size, is_max);
    CK(cudaGetLastError());
    h->host_partial.resize(nb);
    CK(cudaMemcpyAsync(h->host_partial.data(), h->partial, nb * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    double r = is_max ? -INFINITY : 0.0;
    for (int i = 0; i < nb; ++i) r = is_max ? std::max(r, h->host_partial[i]) : r + h->host_partial[i];
    *out = r;
    return SS_OK;
  }

  // observables.compute_energy (e.g. theories/chiral_magnet/observables.py:15-57)
  static int energy(ss_handle* h, const double* F, double* out) {
    plain_energy_kernel<TH><<<blocks(h), dim3(8, 8), 0, h->stream>>>(h->en, F, h->d1, h->G, h->P);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->stream));
    CK(cudaMemcpyAsync(h->entmp, h->en, h->G.N * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    int rc = reduce(h, h->entmp, h->G.N, 0, out);
    if (rc) return rc;
    CK(cudaMemsetAsync(h->entmp, 0, h->G.N * sizeof(double), h->stream));
    CK(cudaMemsetAsync(h->en, 0, h->G.N * sizeof(double), h->stream));
    return SS_OK;
  }

  // do_arrested_newton_flow (core/integrator.py:217-348), one host-driven step at a time
  static int step(ss_handle* h, int n, double prev, double* E_host, double* err_host) {
    double* F = (double*)h->field;
    double* V = (double*)h->vel;
    double** k = (double**)h->k;
    double** l = (double**)h->l;
    double* T = (double*)h->temp;
    double* EG = (double*)h->eg;
    const long long nfN = (long long)h->nf * h->G.N;
    double E = std::isnan(prev) ? h->E_last_host : prev;
    const double factors[4] = {0.0, 0.5, 0.5, 1.0};
    for (int s = 0; s < n; ++s) {
      for (int st = 0; st < 4; ++st) {
        const double* l_in = st == 0 ? V : l[st - 1];
        const double* k_prev = st == 0 ? F : k[st - 1];
        rk4_stage_kernel<double><<<grid_1d(nfN), 256, 0, h->stream>>>(k[st], V, l_in, T, F, k_prev, factors[st],
                                                                          h->G.dt, nfN);
        CK(cudaGetLastError());
        int rc = gradient(h, T, l[st], EG);
        if (rc) return rc;
      }
      rk4_finalize_kernel<double, TH::NF, TH::NMAG><<<grid_1d(h->G.N), 256, 0, h->stream>>>(
          V, F, k[0], k[1], k[2], k[3], l[0], l[1], l[2], l[3], h->G.N, TH::CONSTRAINED && h->G.unit_mag);
      CK(cudaGetLastError());
      CK(cudaStreamSynchronize(h->stream));
      double E_new = 0.0;
      int rc = energy(h, F, &E_new);
      if (rc) return rc;
      if (h->G.killkinen && E_new > E) {
        CK(cudaMemsetAsync(V, 0, nfN * sizeof(double), h->stream));
        CK(cudaStreamSynchronize(h->stream));
      }
      double err = 0.0;
      if ((rc = reduce(h, EG, nfN, 1, &err))) return rc;
      E = E_new;
      if (E_host) E_host[s] = E;
      if (err_host) err_host[s] = err;
      if (!std::isfinite(E)) {
        h->E_last_host = E;
        return fail(SS_ERR_NONFINITE, "non-finite energy at step %d", s);
      }
    }
    h->E_last_host = E;
    return SS_OK;
  }
};

// ---------------------------------------------------------------------------
// dispatch tables
// ---------------------------------------------------------------------------
template <class Fn>
int dispatch(const ss_handle* h, Fn&& fn) {
  switch (h->theory) {
    case SS_THEORY_CHIRAL_MAGNET: return fn((ChiralMagnet*)nullptr);
    case SS_THEORY_BABY_SKYRME: return fn((BabySkyrme*)nullptr);
    case SS_THEORY_GINZBURG_LANDAU: return fn((GinzburgLandau*)nullptr);
    case SS_THEORY_ANISOTROPIC: return fn((Anisotropic*)nullptr);
  }
  return fail(SS_ERR_ARG, "bad theory");
}

// rows of the step's phase tiles
void step_shape(const ss_handle* h, int& txa, int& txb) {
  dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    txa = h->precision == SS_FP32 ? StepShape<TH, float, PH_A>::TX : StepShape<TH, double, PH_A>::TX;
    txb = h->precision == SS_FP32 ? StepShape<TH, float, PH_B>::TX : StepShape<TH, double, PH_B>::TX;
    return SS_OK;
  });
}

// Whether (and in which tile shape) the handle's steps run cooperatively: 1 + shape, or 0.
// The first shape whose tiles are all resident: wherever one fits, the cooperative step was
// the faster.  us per step, two launches -> cooperative, by shape:
//                    8 x 32                      16 x 32                      16 x 64
//   FP32 chiral      320 x 320 25.1 -> 11.6      420 x 500 31.1 -> 16.1       512 x 560 30.8 -> 18.9
//        baby        320 x 320 26.2 -> 11.6      544 x 544 33.9 -> 20.4
//        Higgs       320 x 320 20.9 -> 11.4      420 x 500 27.1 -> 15.5       512 x 560 27.2 -> 19.6
//        s+id        256 x 256 24.3 -> 12.1      333 x 400 29.1 -> 20.3
//   FP64 chiral      256 x 256 29.4 -> 11.7                                   333 x 400 32.9 -> 20.1
//        baby        256 x 256 29.7 -> 11.9      333 x 400 31.8 -> 21.0
//        Higgs       256 x 256 25.1 -> 11.8                                   333 x 400 27.9 -> 20.0
//        s+id        128 x 128 27.2 -> 11.4      256 x 256 28.1 -> 27.0
// Of two shapes that fit the smaller tile (10.5 against 12.9 and 12.7, FP32 chiral 321 x 256).
int coop_plan(const ss_handle* h) {
  if (h->pinned) return 0;
  int dev = 0, ok = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&ok, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !ok)
    return 0;
  int got = 0;
  for (int s = 0; s < N_COOP_SHAPES && !got; ++s)
    dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      if (h->precision == SS_FP32 ? Fused<TH, float>::coop_fits(h, s) : Fused<TH, double>::coop_fits(h, s)) got = s + 1;
      return SS_OK;
    });
  return got;
}

static_assert(sizeof(StepState) <= 192, "fits behind the staged status");
int read_state(ss_handle* h, StepState* out) {
  // page-locked: the copy needs no intermediate buffer; pageable where no block can be had
  if (!h->stage.host && stage_take(h->stage) != cudaSuccess) cudaGetLastError();
  StepState* s = h->stage.host ? reinterpret_cast<StepState*>(h->stage.host + 2 * TRAJ_CAP + 8) : out;
  h->stage.busy = true;
  CK(cudaMemcpyAsync(s, h->st, sizeof(StepState), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->stage.busy = false;
  if (s != out) *out = *s;
  return SS_OK;
}

// error of a nonzero device status (read by the caller, with the stream idle), which is cleared on
// the device together with the counters a kernel that gave up leaves behind
int status_error(ss_handle* h, int status) {
  StepState s;
  int rc = read_state(h, &s);
  if (rc) return rc;
  s.status = 0;
  idle_counters(s);
  CK(cudaMemcpyAsync(h->st, &s, sizeof(s), cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  if (status == SS_ERR_TIMEOUT)
    return fail(SS_ERR_TIMEOUT, "a device-side wait timed out; re-bind the handle before further use");
  return fail(SS_ERR_NONFINITE, "a reduction produced a non-finite value");
}

int take_status(ss_handle* h) {
  StepState s;
  int rc = read_state(h, &s);
  if (rc) return rc;
  return s.status ? status_error(h, s.status) : SS_OK;
}

int fused_density(ss_handle* h, const void* field, double* dens, bool reduce, int kind, int which) {
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::density(h, field, dens, reduce, kind, which);
    return Fused<TH, double>::density(h, field, dens, reduce, kind, which);
  });
}

bool theory_has_charge(int theory, int which) {
  switch (theory) {
    case SS_THEORY_CHIRAL_MAGNET: return ChiralMagnet::has_charge(which);
    case SS_THEORY_BABY_SKYRME: return BabySkyrme::has_charge(which);
    case SS_THEORY_GINZBURG_LANDAU: return GinzburgLandau::has_charge(which);
    case SS_THEORY_ANISOTROPIC: return Anisotropic::has_charge(which);
  }
  return false;
}

bool theory_has_coupling(int theory, int which) {
  switch (theory) {
    case SS_THEORY_CHIRAL_MAGNET: return ChiralMagnet::has_coupling(which);
    case SS_THEORY_BABY_SKYRME: return BabySkyrme::has_coupling(which);
    case SS_THEORY_GINZBURG_LANDAU: return GinzburgLandau::has_coupling(which);
    case SS_THEORY_ANISOTROPIC: return Anisotropic::has_coupling(which);
  }
  return false;
}

int scalar_result(ss_handle* h, double* out) {
  StepState s;
  int rc = read_state(h, &s);
  if (rc) return rc;
  *out = s.scalar;
  if (s.status) return take_status(h);
  return SS_OK;
}

}  // namespace

// ===========================================================================
// exported entry points
// ===========================================================================
extern "C" {

int ss_abi_version(void) { return SS_ABI_VERSION; }

const char* ss_status_string(int status) {
  switch (status) {
    case SS_OK: return "ok";
    case SS_ERR_ARG: return "invalid argument";
    case SS_ERR_CUDA: return "CUDA error";
    case SS_ERR_NONFINITE: return "non-finite value";
    case SS_ERR_STATE: return "invalid call order";
    case SS_ERR_WORKSPACE: return "workspace too small or misaligned";
    case SS_ERR_TIMEOUT: return "device-side wait timed out";
  }
  return "unknown status";
}

const char* ss_last_error(void) { return g_err; }

int ss_create(int theory, const int32_t* p_i, int n_i, const double* p_f, int n_f, int precision, ss_handle** out) {
  if (!out) return fail(SS_ERR_ARG, "out must not be NULL");
  *out = nullptr;
  if (precision != SS_FP64 && precision != SS_FP32 && precision != SS_PLAIN_FP64)
    return fail(SS_ERR_ARG, "unknown precision %d", precision);
  ss_handle* h = new ss_handle();
  h->theory = theory;
  h->precision = precision;
  int rc = decode(h, theory, p_i, n_i, p_f, n_f);
  if (rc) {
    delete h;
    return rc;
  }
  h->elem = precision == SS_FP32 ? 4 : 8;
  // the step's phases tile at 8 rows where 16 do not fit: up to twice the tiles
  const long long tiles = (long long)((h->G.X + TX - 1) / TX) * ((h->G.Y + TY - 1) / TY);
  if (tiles > 0x1fffffffLL) {
    delete h;
    return fail(SS_ERR_ARG, "lattice too large");
  }
  h->nblocks = (int)tiles;
  h->plain_sum_blocks = (int)((h->G.N + 1023) / 1024);
  h->plain_max_blocks = (int)((h->G.N * h->nf + 1023) / 1024);
  *out = h;
  return SS_OK;
}

int ss_destroy(ss_handle* h) {
  delete h;
  return SS_OK;
}

int ss_workspace_bytes(const ss_handle* h, size_t* bytes) {
  if (!h || !bytes) return fail(SS_ERR_ARG, "NULL argument");
  ss_handle tmp = *h;
  tmp.graph = nullptr;  // the copy must not own the original's graph or staging
  tmp.stage = HostStage{};
  *bytes = layout(&tmp, nullptr);
  return SS_OK;
}

int ss_bind(ss_handle* h, void* field, void* velocity, void* workspace, size_t workspace_bytes, void* stream) {
  if (!h) return fail(SS_ERR_ARG, "NULL handle");
  if (!workspace) return fail(SS_ERR_ARG, "workspace must not be NULL");
  if (((uintptr_t)workspace) % ALIGN) return fail(SS_ERR_WORKSPACE, "workspace must be %zu-byte aligned", ALIGN);
  size_t need = 0;
  ss_workspace_bytes(h, &need);
  if (workspace_bytes < need) return fail(SS_ERR_WORKSPACE, "workspace has %zu bytes, needs %zu", workspace_bytes, need);
  h->field = field;
  h->vel = velocity;
  h->ws = (char*)workspace;
  h->ws_bytes = workspace_bytes;
  h->stream = (cudaStream_t)stream;
  h->G.pairs = site_pairs(h->G, h->elem, {field, velocity});
  layout(h, h->ws);
  StepState init;
  memset(&init, 0, sizeof(init));
  init.E_last = NAN;
  CK(cudaMemcpyAsync(h->st, &init, sizeof(init), cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->E_last_host = NAN;
  h->tma = false;
  if (h->precision != SS_PLAIN_FP64 && field && velocity) {
    const void* pairs[4] = {field, velocity, h->phi2, h->vel2};
    int txa = 0, txb = 0;
    step_shape(h, txa, txb);
    bool ok = true;
    for (int i = 0; i < 4 && ok; ++i)
      ok = encode_tile_map(&h->tm[TM_A + i], pairs[i], h->elem, h->G.X, h->G.Y, h->nf, txa, TY) &&
           encode_tile_map(&h->tm[TM_B + i], pairs[i], h->elem, h->G.X, h->G.Y, h->nf, txb, TY);
    for (int i = 0; i < 2 && ok; ++i)
      ok = encode_tile_map(&h->tm[TM_L + i], h->l[i], h->elem, h->G.X, h->G.Y, h->nf, txb, TY);
    h->tma = ok;
  }
  h->coop = 0;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
    h->num_sms = sms;
  if (h->precision != SS_PLAIN_FP64 && field && velocity) h->coop = coop_plan(h);
  return SS_OK;
}

int ss_step_form(const ss_handle* h) { return h ? h->coop : -1; }

int ss_tma_enabled(const ss_handle* h) { return h && h->tma ? 1 : 0; }

int ss_autotune(ss_handle* h, int iters, float* ms_out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!h->field || !h->vel) return fail(SS_ERR_STATE, "no Field/Velocity bound");
  if (h->precision == SS_PLAIN_FP64) return SS_OK;
  if (iters < 1) iters = 1;
  rc = dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::autotune(h, iters);
    return Fused<TH, double>::autotune(h, iters);
  });
  if (rc) return rc;
  if (ms_out)
    for (int m = 0; m < N_FLOW_MODES; ++m) {
      ms_out[2 * m] = h->tune_ms[m][0];
      ms_out[2 * m + 1] = h->tune_ms[m][1];
    }
  return take_status(h);
}

int ss_debug_wait_timeout(ss_handle* h, long long wait_cycles, int inject) {
  if (!h) return fail(SS_ERR_ARG, "NULL handle");
  if (wait_cycles <= 0) return fail(SS_ERR_ARG, "wait_cycles must be positive");
  h->wait_cycles = wait_cycles;
  h->inject_timeout = inject ? 1 : 0;
  return SS_OK;
}

int ss_get_variant(const ss_handle* h, int mode) {
  if (!h || mode < 0 || mode > 6) return -1;
  if (mode == M_S23) return h->fuse23;
  return h->use_pipe[mode];
}

int ss_set_variant(ss_handle* h, int mode, int variant) {
  if (!h) return fail(SS_ERR_ARG, "NULL handle");
  if (mode < 0 || mode > 6 || mode == 5)
    return fail(SS_ERR_ARG, "mode %d: 0 (gradient), 1..4 (stages) or 6 (stages 2+3 fused); the energy pass follows "
                "stage 1", mode);
  if (variant != 0 && variant != 1) return fail(SS_ERR_ARG, "variant %d: 0 (one tile per CTA) or 1 (pipelined)", variant);
  if (h->precision == SS_PLAIN_FP64) return fail(SS_ERR_ARG, "the plain FP64 form has no staging variants");
  if (variant == 1 && mode != M_S23) {
    if (!h->tma) return fail(SS_ERR_STATE, "the pipelined variant needs TMA-staged buffers (bind first; rows of 16-byte multiples)");
    const bool ok = dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      return h->precision == SS_FP32 ? Fused<TH, float>::uses_pipe(mode) : Fused<TH, double>::uses_pipe(mode);
    }) != 0;
    if (!ok) return fail(SS_ERR_ARG, "no pipelined variant of mode %d for this theory and precision", mode);
  }
  if (mode != M_GRAD) {  // the step's launches were asked for
    h->pinned = true;
    h->coop = 0;
  }
  if (mode == M_S23) {  // kept for the caller, chooses nothing
    h->fuse23 = variant;
    return SS_OK;
  }
  h->use_pipe[mode] = variant;
  if (mode == M_S1) h->use_pipe[M_ENERGY] = variant;  // reported only
  return SS_OK;
}

int ss_step_async(ss_handle* h, int n_steps, double prev_energy, double* energy_traj_dev, double* err_traj_dev) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (n_steps < 0) return fail(SS_ERR_ARG, "n_steps must be >= 0");
  if (!h->field || !h->vel) return fail(SS_ERR_STATE, "no Field/Velocity bound");
  if (h->precision == SS_PLAIN_FP64)
    return fail(SS_ERR_ARG, "the plain FP64 form arrests on the host; use ss_step");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::step(h, n_steps, prev_energy, energy_traj_dev, err_traj_dev);
    return Fused<TH, double>::step(h, n_steps, prev_energy, energy_traj_dev, err_traj_dev);
  });
}

int ss_step(ss_handle* h, int n_steps, double prev_energy, double* energy_traj, double* err_traj) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (n_steps < 0) return fail(SS_ERR_ARG, "n_steps must be >= 0");
  if (!h->field || !h->vel) return fail(SS_ERR_STATE, "no Field/Velocity bound");
  if (h->precision == SS_PLAIN_FP64) {
    return dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      return Plain<TH>::step(h, n_steps, prev_energy, energy_traj, err_traj);
    });
  }
  if (n_steps == 0) return take_status(h);
  // each chunk's trajectories and status are written by the kernels into mapped
  // page-locked memory: one synchronisation per chunk and no copies
  if (!h->stage.host) CK(stage_take(h->stage));
  double* hE = h->stage.host;
  double* hErr = h->stage.host + TRAJ_CAP;
  volatile int* hstatus = reinterpret_cast<volatile int*>(h->stage.host + 2 * TRAJ_CAP);
  int* dstatus = reinterpret_cast<int*>(h->stage.dev + 2 * TRAJ_CAP);
  double prev = prev_energy;
  for (int done = 0; done < n_steps; done += TRAJ_CAP) {
    const int k = std::min(TRAJ_CAP, n_steps - done);
    *hstatus = -1;
    h->stage.busy = true;
    rc = dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      double* dE = h->stage.dev;
      double* dErr = h->stage.dev + TRAJ_CAP;
      if (h->precision == SS_FP32) return Fused<TH, float>::step(h, k, prev, dE, dErr, dstatus);
      return Fused<TH, double>::step(h, k, prev, dE, dErr, dstatus);
    });
    if (rc) return rc;
    prev = NAN;
    CK(cudaStreamSynchronize(h->stream));
    h->stage.busy = false;
    if (energy_traj) memcpy(energy_traj + done, hE, k * sizeof(double));
    if (err_traj) memcpy(err_traj + done, hErr, k * sizeof(double));
    const int status = *hstatus;
    if (status < 0) return fail(SS_ERR_CUDA, "the step's status was not written");
    if (status) return status_error(h, status);
  }
  return SS_OK;
}

int ss_check_status(ss_handle* h) {
  int rc = check_bound(h);
  if (rc) return rc;
  return take_status(h);
}

int ss_gradient(ss_handle* h, const void* field, void* energy_gradient, void* l_out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field) return fail(SS_ERR_ARG, "field must not be NULL");
  if (h->precision == SS_PLAIN_FP64) {
    return dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      double* eg = energy_gradient ? (double*)energy_gradient : (double*)h->eg;
      double* l = l_out ? (double*)l_out : (double*)h->l[0];
      return Plain<TH>::gradient(h, (const double*)field, l, eg);
    });
  }
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::gradient(h, field, energy_gradient, l_out);
    return Fused<TH, double>::gradient(h, field, energy_gradient, l_out);
  });
}

int ss_energy_gradient(ss_handle* h, const void* field, void* grad) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !grad) return fail(SS_ERR_ARG, "NULL argument");
  if (h->precision == SS_PLAIN_FP64) return fail(SS_ERR_ARG, "ss_energy_gradient needs SS_FP32 or SS_FP64");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::gradient(h, field, grad, nullptr, 1);
    return Fused<TH, double>::gradient(h, field, grad, nullptr, 1);
  });
}

int ss_energy_vjp(ss_handle* h, const void* field, const double* grad_E, void* grad) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !grad || !grad_E) return fail(SS_ERR_ARG, "NULL argument");
  if (h->precision == SS_PLAIN_FP64) return fail(SS_ERR_ARG, "ss_energy_vjp needs SS_FP32 or SS_FP64");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::gradient(h, field, grad, nullptr, 1, grad_E);
    return Fused<TH, double>::gradient(h, field, grad, nullptr, 1, grad_E);
  });
}

int ss_energy_density(ss_handle* h, const void* field, double* density) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !density) return fail(SS_ERR_ARG, "NULL argument");
  return fused_density(h, field, density, false, D_ENERGY, 0);
}

int ss_energy(ss_handle* h, const void* field, double* out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !out) return fail(SS_ERR_ARG, "NULL argument");
  if (h->precision == SS_PLAIN_FP64) {
    return dispatch(h, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      return Plain<TH>::energy(h, (const double*)field, out);
    });
  }
  rc = dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::energy(h, field);
    return Fused<TH, double>::energy(h, field);
  });
  if (rc) return rc;
  return scalar_result(h, out);
}

namespace {
int launch_init(ss_handle* h, void* field, void* velocity, const InitArgs& A) {
  const long long N = (long long)A.X * A.Y;
  const unsigned blocks = (unsigned)((N + 255) / 256);
  auto go = [&](auto* tag) -> int {
    using R = std::remove_pointer_t<decltype(tag)>;
    R* F = (R*)field;
    R* V = (R*)velocity;
    switch (h->theory) {
      case 0: init_kernel<0, R><<<blocks, 256, 0, h->stream>>>(F, V, A); break;
      case 1: init_kernel<1, R><<<blocks, 256, 0, h->stream>>>(F, V, A); break;
      case 2: init_kernel<2, R><<<blocks, 256, 0, h->stream>>>(F, V, A); break;
      default: init_kernel<3, R><<<blocks, 256, 0, h->stream>>>(F, V, A); break;
    }
    CK(cudaGetLastError());
    return SS_OK;
  };
  return h->precision == SS_FP32 ? go((float*)nullptr) : go((double*)nullptr);
}

InitArgs init_args(const ss_handle* h, int mode) {
  InitArgs A;
  memset(&A, 0, sizeof(A));
  A.X = h->G.X;
  A.Y = h->G.Y;
  A.nf = h->nf;
  A.mode = mode;
  for (int i = 0; i < 32; ++i) A.pf[i] = h->pf_raw[i];
  return A;
}
}  // namespace

int ss_initialize(ss_handle* h, void* field, void* velocity, int mode, int ansatz, double rotation,
                  double vortex_number) {
  if (!h || !field) return fail(SS_ERR_ARG, "handle and field must not be NULL");
  if (mode != SS_INIT_GROUND && mode != SS_INIT_ANSATZ) return fail(SS_ERR_ARG, "unknown init mode %d", mode);
  if (ansatz < SS_ANSATZ_NONE || ansatz > SS_ANSATZ_ANTI) return fail(SS_ERR_ARG, "unknown ansatz %d", ansatz);
  InitArgs A = init_args(h, mode == SS_INIT_GROUND ? IM_GROUND : IM_ANSATZ);
  A.ansatz = ansatz;
  A.rotation = rotation;
  A.vortex_number = vortex_number;
  return launch_init(h, field, velocity, A);
}

int ss_insert_soliton(ss_handle* h, void* field, int pxi, int pxj, int ansatz, int vortex, double rotation) {
  if (!h || !field) return fail(SS_ERR_ARG, "handle and field must not be NULL");
  if (ansatz < SS_ANSATZ_NONE || ansatz > SS_ANSATZ_ANTI) return fail(SS_ERR_ARG, "unknown ansatz %d", ansatz);
  if (pxi < 0 || pxi >= h->G.X || pxj < 0 || pxj >= h->G.Y) return SS_OK;  // the reference's kernels ignore it
  InitArgs A = init_args(h, IM_INSERT);
  A.ansatz = ansatz;
  A.vortex = vortex ? 1 : 0;
  A.rotation = rotation;
  A.pxi = pxi;
  A.pxj = pxj;
  return launch_init(h, field, nullptr, A);
}

int ss_text_workspace_bytes(long long n, size_t* bytes) {
  if (!bytes || n < 0) return fail(SS_ERR_ARG, "bad arguments");
  const long long nb = (n + 1023) / 1024;
  *bytes = (size_t)(n + nb + 8) * sizeof(long long);
  return SS_OK;
}

int ss_format_text(const void* values, int precision, long long n, int digits, long long row, long long block,
                   char* out, size_t out_cap, long long* out_len, void* workspace, size_t workspace_bytes,
                   void* stream) {
  if (!values || !out_len || !workspace) return fail(SS_ERR_ARG, "values, out_len and workspace must not be NULL");
  if (precision != SS_FP32 && precision != SS_FP64) return fail(SS_ERR_ARG, "precision must be SS_FP32 or SS_FP64");
  if (n <= 0) return fail(SS_ERR_ARG, "n must be positive");
  if (digits < 1 || digits > TXT_MAX_P) return fail(SS_ERR_ARG, "digits must be 1..%d", TXT_MAX_P);
  if (row < 0 || block < 0) return fail(SS_ERR_ARG, "row and block must be >= 0");
  size_t need = 0;
  ss_text_workspace_bytes(n, &need);
  if (workspace_bytes < need) return fail(SS_ERR_WORKSPACE, "workspace of %zu bytes, need %zu", workspace_bytes, need);
  if ((reinterpret_cast<uintptr_t>(workspace) & 7u) != 0) return fail(SS_ERR_WORKSPACE, "workspace must be 8-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const long long nb = (n + 1023) / 1024;
  long long* off = (long long*)workspace;
  long long* sums = off + n;
  long long* total = sums + nb;
  const TextLayout L{n, row, block, digits};
  const unsigned g256 = (unsigned)((n + 255) / 256);
  if (precision == SS_FP32) text_len_kernel<float><<<g256, 256, 0, st>>>((const float*)values, L, off);
  else text_len_kernel<double><<<g256, 256, 0, st>>>((const double*)values, L, off);
  scan_block_kernel<<<(unsigned)nb, 1024, 0, st>>>(off, n, sums);
  scan_sums_kernel<<<1, 1024, 0, st>>>(sums, nb, total);
  scan_add_kernel<<<(unsigned)nb, 1024, 0, st>>>(off, n, sums);
  CK(cudaGetLastError());
  long long len = 0;
  CK(cudaMemcpyAsync(&len, total, sizeof(len), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  *out_len = len;
  if (!out) return SS_OK;  // size query
  if ((size_t)len > out_cap) return fail(SS_ERR_ARG, "text of %lld bytes does not fit the %zu-byte buffer", len, out_cap);
  if (precision == SS_FP32) text_write_kernel<float><<<g256, 256, 0, st>>>((const float*)values, L, off, out);
  else text_write_kernel<double><<<g256, 256, 0, st>>>((const double*)values, L, off, out);
  CK(cudaGetLastError());
  return SS_OK;
}

int ss_render_rgba(int kind, const void* src, int precision, int xlen, int ylen, double vmin, double vmax,
                   unsigned char* rgba, void* stream) {
  if (!src || !rgba) return fail(SS_ERR_ARG, "src and rgba must not be NULL");
  if (kind < SS_RENDER_JET || kind > SS_RENDER_MAGNETIZATION) return fail(SS_ERR_ARG, "unknown render kind %d", kind);
  if (precision != SS_FP32 && precision != SS_FP64)
    return fail(SS_ERR_ARG, "precision must be SS_FP32 or SS_FP64 (element type of src)");
  if (xlen <= 0 || ylen <= 0) return fail(SS_ERR_ARG, "xlen and ylen must be positive");
  if ((reinterpret_cast<uintptr_t>(rgba) & 3u) != 0) return fail(SS_ERR_ARG, "rgba must be 4-byte aligned");
  const dim3 grid((unsigned)((ylen + 31) / 32), (unsigned)((xlen + 31) / 32)), block(32, 8);
  if (grid.y > 65535u) return fail(SS_ERR_ARG, "xlen %d too large (at most %d)", xlen, 65535 * 32);
  cudaStream_t s = (cudaStream_t)stream;
  uint32_t* out = reinterpret_cast<uint32_t*>(rgba);
  auto go = [&](auto* tag) {
    using T = std::remove_pointer_t<decltype(tag)>;
    const T* p = (const T*)src;
    if (kind == SS_RENDER_JET) render_kernel<T, RK_JET><<<grid, block, 0, s>>>(p, xlen, ylen, vmin, vmax, out);
    else if (kind == SS_RENDER_GRAY) render_kernel<T, RK_GRAY><<<grid, block, 0, s>>>(p, xlen, ylen, vmin, vmax, out);
    else render_kernel<T, RK_MAGNETIZATION><<<grid, block, 0, s>>>(p, xlen, ylen, vmin, vmax, out);
  };
  if (precision == SS_FP32) go((float*)nullptr); else go((double*)nullptr);
  CK(cudaGetLastError());
  return SS_OK;
}

int ss_energy_projected(ss_handle* h, const void* field, double* out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !out) return fail(SS_ERR_ARG, "NULL argument");
  rc = dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::energy_projected(h, field);
    return Fused<TH, double>::energy_projected(h, field);
  });
  if (rc) return rc;
  return scalar_result(h, out);
}

int ss_charge_density(ss_handle* h, const void* field, int which, double* density) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !density) return fail(SS_ERR_ARG, "NULL argument");
  if (!theory_has_charge(h->theory, which)) return fail(SS_ERR_ARG, "charge %d not defined for theory %d", which, h->theory);
  return fused_density(h, field, density, false, D_CHARGE, which);
}

int ss_charge(ss_handle* h, const void* field, int which, double* out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !out) return fail(SS_ERR_ARG, "NULL argument");
  if (!theory_has_charge(h->theory, which)) return fail(SS_ERR_ARG, "charge %d not defined for theory %d", which, h->theory);
  rc = fused_density(h, field, nullptr, true, D_CHARGE, which);
  if (rc) return rc;
  return scalar_result(h, out);
}

int ss_observables(ss_handle* h, const void* field, int n, const int* kinds, const int* which, double* out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !kinds || !which || !out) return fail(SS_ERR_ARG, "NULL argument");
  if (n < 1 || n > OBS_MAX) return fail(SS_ERR_ARG, "n must be 1..%d", OBS_MAX);
  ObsList L{};
  for (int i = 0; i < n; ++i) {
    if (kinds[i] < SS_OBS_ENERGY || kinds[i] > SS_OBS_COUPLING) return fail(SS_ERR_ARG, "unknown kind %d", kinds[i]);
    if (kinds[i] == SS_OBS_CHARGE && !theory_has_charge(h->theory, which[i]))
      return fail(SS_ERR_ARG, "charge %d not defined for theory %d", which[i], h->theory);
    if (kinds[i] == SS_OBS_COUPLING && !theory_has_coupling(h->theory, which[i]))
      return fail(SS_ERR_ARG, "coupling %d not defined for theory %d", which[i], h->theory);
    if (h->precision != SS_FP32 && kinds[i] == SS_OBS_ENERGY) {
      // the flow's own FP64 energy (ss_energy): the two-launch step's to the last bit, a cooperative
      // step's to rounding (other tiles)
      if ((rc = ss_energy(h, field, out + i))) return rc;
      continue;
    }
    L.kind[L.n] = kinds[i];
    L.which[L.n++] = which[i];
  }
  if (!L.n) return SS_OK;
  rc = dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    for (int i = 0; i < L.n; ++i) L.comps |= Fused<TH, float>::obs_comps(L.kind[i], L.which[i]);
    if (h->precision == SS_FP32) return Fused<TH, float>::observe(h, field, nullptr, true, L);
    return Fused<TH, double>::observe(h, field, nullptr, true, L);
  });
  if (rc) return rc;
  StepState s;
  if ((rc = read_state(h, &s))) return rc;
  for (int i = 0, k = 0; i < n; ++i)
    if (!(h->precision != SS_FP32 && kinds[i] == SS_OBS_ENERGY)) out[i] = s.scalars[k++];
  return s.status ? take_status(h) : SS_OK;
}

int ss_coupling_grad(ss_handle* h, const void* field, int coupling, double* out) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !out) return fail(SS_ERR_ARG, "NULL argument");
  if (!theory_has_coupling(h->theory, coupling))
    return fail(SS_ERR_ARG, "coupling %d not defined for theory %d", coupling, h->theory);
  rc = fused_density(h, field, nullptr, true, D_COUPLING, coupling);
  if (rc) return rc;
  return scalar_result(h, out);
}

int ss_convert_field(ss_handle* h, const void* src, int src_precision, void* dst, int dst_precision, int project) {
  if (!h || !src || !dst) return fail(SS_ERR_ARG, "NULL argument");
  auto is_prec = [](int p) { return p == SS_FP32 || p == SS_FP64 || p == SS_PLAIN_FP64; };
  if (!is_prec(src_precision) || !is_prec(dst_precision)) return fail(SS_ERR_ARG, "unknown precision");
  const bool s32 = src_precision == SS_FP32, d32 = dst_precision == SS_FP32;
  if (src == dst && s32 != d32) return fail(SS_ERR_ARG, "in-place conversion needs equal element types");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    const int norm = project && TH::CONSTRAINED && h->G.unit_mag;
    const dim3 g = grid_1d(h->G.N);
    if (s32 && d32) convert_kernel<float, float, TH::NF, TH::NMAG><<<g, 256, 0, h->stream>>>((const float*)src, (float*)dst, h->G.N, norm);
    else if (s32) convert_kernel<float, double, TH::NF, TH::NMAG><<<g, 256, 0, h->stream>>>((const float*)src, (double*)dst, h->G.N, norm);
    else if (d32) convert_kernel<double, float, TH::NF, TH::NMAG><<<g, 256, 0, h->stream>>>((const double*)src, (float*)dst, h->G.N, norm);
    else convert_kernel<double, double, TH::NF, TH::NMAG><<<g, 256, 0, h->stream>>>((const double*)src, (double*)dst, h->G.N, norm);
    CK(cudaGetLastError());
    return SS_OK;
  });
}

int ss_energy_gradient_exact(ss_handle* h, const void* field, double* out, int minus_stencil) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!field || !out) return fail(SS_ERR_ARG, "NULL argument");
  if (h->precision == SS_PLAIN_FP64) return fail(SS_ERR_ARG, "ss_energy_gradient_exact needs SS_FP32 or SS_FP64");
  if (minus_stencil && h->precision != SS_FP64)
    return fail(SS_ERR_ARG, "the residual against the stencil gradient needs SS_FP64 fields");
  const size_t nfN = (size_t)h->nf * (size_t)h->G.N;
  const size_t q_bytes = align_up(2 * nfN * sizeof(double));
  const size_t need = q_bytes + (minus_stencil ? nfN * sizeof(double) : 0);
  char* region = (char*)h->l[0];
  if (!region || region + need > h->ws + h->ws_bytes)
    return fail(SS_ERR_WORKSPACE, "the workspace's flow buffers (%zu bytes) cannot hold the %zu bytes of scratch",
                (size_t)(h->ws + h->ws_bytes - region), need);
  double* q = (double*)region;
  double* sub = minus_stencil ? (double*)(region + q_bytes) : nullptr;
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::energy_gradient_exact(h, field, out, q, sub);
    return Fused<TH, double>::energy_gradient_exact(h, field, out, q, sub);
  });
}

int ss_set_forcing(ss_handle* h, const double* force) {
  if (!h) return fail(SS_ERR_ARG, "NULL handle");
  if (force && h->precision != SS_FP64) return fail(SS_ERR_ARG, "a forcing needs SS_FP64 fields");
  if (((uintptr_t)force) % 16) return fail(SS_ERR_ARG, "the forcing must be 16-byte aligned");
  h->force = force;
  return SS_OK;
}

int ss_field_density(ss_handle* h, const void* field, int kind, double* out) {
  if (!h || !field || !out) return fail(SS_ERR_ARG, "NULL argument");
  const bool ah = h->theory == SS_THEORY_GINZBURG_LANDAU, sid = h->theory == SS_THEORY_ANISOTROPIC;
  const bool ok = (kind == SS_DENSITY_HIGGS && ah) || (kind == SS_DENSITY_SUPERCURRENT && (ah || sid)) ||
                  ((kind == SS_DENSITY_HIGGS1 || kind == SS_DENSITY_HIGGS2 || kind == SS_DENSITY_PHASE_DIFFERENCE ||
                    kind == SS_DENSITY_MAGNETIC_FIELD) && sid);
  if (!ok) return fail(SS_ERR_ARG, "density kind %d not defined for theory %d", kind, h->theory);
  const double q = ah ? h->P.c[0] : h->P.c[1];
  if (h->precision == SS_FP32)
    field_density_kernel<float><<<grid_1d(h->G.N), 256, 0, h->stream>>>((const float*)field, out, kind, h->G, q);
  else
    field_density_kernel<double><<<grid_1d(h->G.N), 256, 0, h->stream>>>((const double*)field, out, kind, h->G, q);
  CK(cudaGetLastError());
  return SS_OK;
}

int ss_rk4_stage(ss_handle* h, void* k_out, const void* velocity, const void* l_in, void* temp, const void* field,
                 const void* k_prev, double factor) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (!k_out || !velocity || !l_in || !temp || !field || !k_prev) return fail(SS_ERR_ARG, "NULL argument");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::rk4_stage(h, k_out, velocity, l_in, temp, field, k_prev, factor);
    return Fused<TH, double>::rk4_stage(h, k_out, velocity, l_in, temp, field, k_prev, factor);
  });
}

int ss_rk4_finalize(ss_handle* h, void* velocity, void* field, const void* k1, const void* k2, const void* k3,
                    const void* k4, const void* l1, const void* l2, const void* l3, const void* l4) {
  int rc = check_bound(h);
  if (rc) return rc;
  const void* k[4] = {k1, k2, k3, k4};
  const void* l[4] = {l1, l2, l3, l4};
  for (int i = 0; i < 4; ++i)
    if (!k[i] || !l[i]) return fail(SS_ERR_ARG, "NULL argument");
  if (!velocity || !field) return fail(SS_ERR_ARG, "NULL argument");
  return dispatch(h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (h->precision == SS_FP32) return Fused<TH, float>::rk4_finalize(h, velocity, field, k, l);
    return Fused<TH, double>::rk4_finalize(h, velocity, field, k, l);
  });
}

}  // extern "C"

// ===========================================================================
// Total energy without any allocation.
//
// Some callers cannot allocate device memory at the point where they need an
// energy: hosts whose memory manager owns the whole device and forbids further
// allocations (a framework's caching allocator or a fixed memory pool), and
// interactive loops (a viewer's per-frame callback) that must not call cudaMalloc
// or cudaFree because those synchronise the device and stall the frame.  For them
// ss_energy_noalloc keeps its scratch (the per-block partial sums and the
// reduction state) in the file-scope array below, which every GPU that loads
// this library holds until exit.
// ===========================================================================
namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = 512 * 1024;   // 256 B state + up to 65504 block partials
__device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
// Device address of the array, per device.  Host threads calling concurrently on a
// device that has no entry yet may each look it up; they store the same address, and
// the atomic (relaxed ordering suffices) makes those concurrent stores well defined.
std::atomic<void*> g_noalloc_addr[64];

// Device address of the static scratch on the current device (looked up once per device,
// with that device current: in host code the array's name is only a host-side stand-in).
int noalloc_scratch(void** out) {
  int dev = -1;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(SS_ERR_ARG, "device ordinal %d out of range", dev);
  void* p = g_noalloc_addr[dev].load(std::memory_order_relaxed);
  if (!p) {
    CK(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_addr[dev].store(p, std::memory_order_relaxed);
  }
  *out = p;
  return SS_OK;
}

}  // namespace

extern "C" int ss_energy_noalloc(int theory, const int32_t* p_i, int n_i, const double* p_f, int n_f,
                                 int precision, const void* field, double* out, void* stream) {
  if (!field || !out) return fail(SS_ERR_ARG, "field and out must not be NULL");
  if (precision != SS_FP32 && precision != SS_FP64)
    return fail(SS_ERR_ARG, "ss_energy_noalloc supports SS_FP32 and SS_FP64 fields");
  ss_handle h;  // on the stack: decoding the parameters allocates nothing
  h.theory = theory;
  h.precision = precision;
  int rc = decode(&h, theory, p_i, n_i, p_f, n_f);
  if (rc) return rc;
  h.elem = precision == SS_FP32 ? 4 : 8;
  const long long tiles = (long long)((h.G.X + TX - 1) / TX) * ((h.G.Y + TY - 1) / TY);
  const size_t need = 256 + (size_t)tiles * sizeof(double);
  if (need > NOALLOC_SCRATCH_BYTES)
    return fail(SS_ERR_ARG,
                "lattice of %lld tiles (16 x 64 sites each) needs %zu bytes of scratch; the allocation-free "
                "entry point holds %zu (at most %zu tiles)",
                tiles, need, NOALLOC_SCRATCH_BYTES, (NOALLOC_SCRATCH_BYTES - 256) / sizeof(double));
  h.nblocks = (int)tiles;
  h.stream = (cudaStream_t)stream;
  void* scratch = nullptr;
  if ((rc = noalloc_scratch(&scratch))) return rc;
  h.st = (StepState*)scratch;
  h.partial = (double*)((char*)scratch + 256);
  // the last call's contents stay in the array: the reduction state must start at zero
  CK(cudaMemsetAsync(h.st, 0, sizeof(StepState), h.stream));
  rc = dispatch(&h, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    ObsList L{};
    L.n = 1;
    L.comps = ~0u;
    return precision == SS_FP32 ? Fused<TH, float>::observe(&h, field, nullptr, true, L, false)
                                : Fused<TH, double>::observe(&h, field, nullptr, true, L, false);
  });
  if (rc) return rc;
  StepState s;
  CK(cudaMemcpyAsync(&s, h.st, sizeof(StepState), cudaMemcpyDeviceToHost, h.stream));
  CK(cudaStreamSynchronize(h.stream));
  *out = s.scalar;
  if (s.status) return fail(SS_ERR_NONFINITE, "the energy reduction produced a non-finite value");
  return SS_OK;
}


// ===========================================================================
// Batched lattices: many independent relaxations of one theory per launch
// ===========================================================================
// Tile shapes of the batched phase kernels (BatchShape): the autotuner picks one per size
// class of lattices (ss_batch_autotune).  Shape 1 exists for TMA-staged FP32 batches.
constexpr int N_BATCH_SHAPES = 2;
constexpr int BSHAPE_TY[N_BATCH_SHAPES] = {64, 32};

struct ss_batch {
  int theory = 0, precision = 0, n = 0, nf = 0;
  size_t elem = 4;
  std::vector<ss_handle> inst;   // decoded parameters per lattice (host only)
  std::vector<int> shape;        // tile shape per lattice
  std::vector<int> max_tiles;    // tiles per lattice in its finest shape (partials are sized for it)
  int total_max = 0;             // sum of max_tiles: capacity of each tile list
  int group_tiles[N_BATCH_SHAPES][2] = {};  // tiles of the lattices of each shape and phase
  bool tma = false;
  cudaStream_t stream = nullptr;
  char* ws = nullptr;
  BatchInst* d_insts = nullptr;
  // lattice of each tile, per shape group and phase (A and E, B)
  int* d_tile_inst[N_BATCH_SHAPES][2] = {};
  float tune_ms[64][N_BATCH_SHAPES] = {};  // autotuner: per size class (first 64) and shape
  double* d_prev = nullptr;
  std::vector<BatchInst> h_insts;
  std::vector<void*> fields, vels;
  long long wait_cycles = WAIT_CYCLES;
  cudaGraphExec_t graph = nullptr;
  // per-lattice step states and trajectory rows, contiguous in the workspace (lattice i:
  // d_st[i], d_E / d_err rows i * TRAJ_CAP), so that one copy returns each for all lattices
  StepState* d_st = nullptr;
  double* d_E = nullptr;
  double* d_err = nullptr;
  char* h_stage = nullptr;  // page-locked staging of those copies (first ss_batch_step)
  ~ss_batch() {
    if (graph) cudaGraphExecDestroy(graph);
    if (h_stage) cudaFreeHost(h_stage);
  }
};

namespace {

size_t batch_layout(ss_batch* b, char* base) {
  size_t off = 0;
  auto take = [&](size_t bytes) -> char* {
    char* p = base ? base + off : nullptr;
    off = align_up(off + bytes);
    return p;
  };
  b->d_insts = (BatchInst*)take(sizeof(BatchInst) * b->n);
  for (int g = 0; g < N_BATCH_SHAPES; ++g)
    for (int p = 0; p < 2; ++p) b->d_tile_inst[g][p] = (int*)take(sizeof(int) * b->total_max);
  b->d_prev = (double*)take(sizeof(double) * b->n);
  b->d_st = (StepState*)take(sizeof(StepState) * b->n);
  b->d_E = (double*)take(sizeof(double) * TRAJ_CAP * b->n);
  b->d_err = (double*)take(sizeof(double) * TRAJ_CAP * b->n);
  b->h_insts.assign(b->n, BatchInst{});
  for (int i = 0; i < b->n; ++i) {
    BatchInst& I = b->h_insts[i];
    const size_t fb = b->elem * (size_t)b->nf * (size_t)b->inst[i].G.N;
    I.st = b->d_st ? b->d_st + i : nullptr;
    I.partial = (double*)take(sizeof(double) * b->max_tiles[i]);
    I.E_traj = b->d_E ? b->d_E + (size_t)i * TRAJ_CAP : nullptr;
    I.err_traj = b->d_err ? b->d_err + (size_t)i * TRAJ_CAP : nullptr;
    for (int k = BB_PHI2; k < BB_COUNT; ++k) I.buf[k] = take(fb);
  }
  return off;
}

template <class Fn>
int batch_dispatch(const ss_batch* b, Fn&& fn) {
  switch (b->theory) {
    case SS_THEORY_CHIRAL_MAGNET: return fn((ChiralMagnet*)nullptr);
    case SS_THEORY_BABY_SKYRME: return fn((BabySkyrme*)nullptr);
    case SS_THEORY_GINZBURG_LANDAU: return fn((GinzburgLandau*)nullptr);
    case SS_THEORY_ANISOTROPIC: return fn((Anisotropic*)nullptr);
  }
  return fail(SS_ERR_ARG, "bad theory");
}

template <class TH, typename R>
struct Batched {
  // one launch over the tiles of `tile_inst` (lattices of one tile shape)
  template <bool SMALL, bool TMA_, int PH>
  static int launch_shape(const ss_batch* b, const BatchStep& B, const int* tile_inst, int ntiles) {
    if (ntiles <= 0) return SS_OK;
    using SH = BatchShape<TH, R, PH, SMALL>;
    constexpr size_t smem = step_buffers<PH, TMA_>() * tile_buf_bytes<R, TH::NF, SH::TX, SH::TY>();
    auto k = batch_step_kernel<TH, R, SMALL, TMA_, PH>;
    static unsigned long long smem_done = 0;  // one per instantiation
    set_smem(k, smem, smem_done);
    k<<<ntiles, SH::NT, smem, b->stream>>>(b->d_insts, tile_inst, B);
    CK(cudaGetLastError());
    return SS_OK;
  }
  // a phase over every shape group (shape 1: TMA-staged FP32 batches only)
  template <int PH>
  static int launch(const ss_batch* b, const BatchStep& B) {
    constexpr int p = PH == PH_B ? 1 : 0;
    int rc = b->tma ? launch_shape<false, true, PH>(b, B, b->d_tile_inst[0][p], b->group_tiles[0][p])
                    : launch_shape<false, false, PH>(b, B, b->d_tile_inst[0][p], b->group_tiles[0][p]);
    if constexpr (sizeof(R) == 4) {
      if (!rc && b->tma) rc = launch_shape<true, true, PH>(b, B, b->d_tile_inst[1][p], b->group_tiles[1][p]);
    }
    return rc;
  }

  static int step(ss_batch* b, int n, bool use_prev) {
    if (n <= 0) return SS_OK;
    BatchStep B;
    memset(&B, 0, sizeof(B));
    B.wait_cycles = b->wait_cycles;
    B.E_idx = B.err_idx = -1;
    int rc;
    for (int s = 0; s < n; ++s, B.cur ^= 1) {
      B.with_energy = B.arrest_update = s > 0;
      B.init_state = s == 0;
      B.prev_energy = (s == 0 && use_prev) ? b->d_prev : nullptr;
      B.E_idx = s - 1;
      B.copy = s == 0 && (n & 1);  // as for a single lattice: the count ends in the caller's buffers
      if ((rc = launch<PH_A>(b, B))) return rc;
      if (B.copy) B.cur = 1;
      B.copy = 0;
      B.init_state = 0;
      B.prev_energy = nullptr;
      B.err_idx = s;
      if ((rc = launch<PH_B>(b, B))) return rc;
    }
    B.with_energy = B.arrest_update = 1;
    B.E_idx = n - 1;
    if ((rc = launch<PH_E>(b, B))) return rc;
    batch_finish_kernel<R, TH::NF><<<dim3(64, b->n), 256, 0, b->stream>>>(b->d_insts);
    CK(cudaGetLastError());
    return SS_OK;
  }

  // The launches of one step with every trajectory and arrest update off: reads the
  // current fields, writes only workspace scratch (l1, l2 and the second pair).
  static int timing_step(ss_batch* b) {
    BatchStep B;
    memset(&B, 0, sizeof(B));
    B.wait_cycles = b->wait_cycles;
    B.E_idx = -1;
    B.err_idx = -1;
    int rc = launch<PH_A>(b, B);
    if (!rc) rc = launch<PH_B>(b, B);
    return rc;
  }
};

// rows of a tile of shape `shape` in phase p (0: A and E, 1: B)
int batch_tx(const ss_batch* b, int shape, int p) {
  int tx = 0;
  batch_dispatch(b, [&](auto* tag) -> int {
    using TH = std::remove_pointer_t<decltype(tag)>;
    if (b->precision == SS_FP32)
      tx = shape ? (p ? BatchShape<TH, float, PH_B, true>::TX : BatchShape<TH, float, PH_A, true>::TX)
                 : (p ? BatchShape<TH, float, PH_B, false>::TX : BatchShape<TH, float, PH_A, false>::TX);
    else
      tx = p ? BatchShape<TH, double, PH_B, false>::TX : BatchShape<TH, double, PH_A, false>::TX;
    return SS_OK;
  });
  return tx;
}
// tiles of a lattice in tile shape `shape`, phase p
long long batch_tiles(const ss_batch* b, const Grid& G, int shape, int p) {
  const int tx = batch_tx(b, shape, p), ty = BSHAPE_TY[shape];
  return (long long)((G.X + tx - 1) / tx) * ((G.Y + ty - 1) / ty);
}

// TMA maps of lattice i for its current tile shape (buffers already set); false when
// a buffer or its row pitch is not 16-byte aligned
bool batch_encode(ss_batch* b, int i) {
  BatchInst& I = b->h_insts[i];
  const int sh = b->shape[i];
  bool ok = true;
  for (int k = 0; k < BT_COUNT && ok; ++k)
    ok = encode_tile_map(&I.tm[k], I.buf[BATCH_TM_BUF[k]], b->elem, I.G.X, I.G.Y, b->nf,
                         batch_tx(b, sh, k >= BT_B ? 1 : 0), BSHAPE_TY[sh]);
  return ok;
}

// Rebuild the per-shape tile lists from the lattices with include[i] (all when null),
// set each lattice's tile range and copy the descriptors and lists to the device.
int batch_upload(ss_batch* b, const std::vector<char>* include) {
  std::vector<int> lists[N_BATCH_SHAPES][2];
  for (int i = 0; i < b->n; ++i) {
    BatchInst& I = b->h_insts[i];
    const int sh = b->shape[i];
    for (int p = 0; p < 2; ++p) {
      std::vector<int>& L = lists[sh][p];
      I.ntiles[p] = (int)batch_tiles(b, I.G, sh, p);
      I.tile0[p] = (int)L.size();
      if (!include || (*include)[i]) L.insert(L.end(), (size_t)I.ntiles[p], i);
    }
  }
  for (int g = 0; g < N_BATCH_SHAPES; ++g)
    for (int p = 0; p < 2; ++p) {
      b->group_tiles[g][p] = (int)lists[g][p].size();
      if (!lists[g][p].empty())
        CK(cudaMemcpyAsync(b->d_tile_inst[g][p], lists[g][p].data(), sizeof(int) * lists[g][p].size(),
                           cudaMemcpyHostToDevice, b->stream));
    }
  CK(cudaMemcpyAsync(b->d_insts, b->h_insts.data(), sizeof(BatchInst) * b->n, cudaMemcpyHostToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return SS_OK;
}

}  // namespace

extern "C" {

int ss_batch_create(int theory, int n_lattices, const int32_t* p_i, int n_i, const double* p_f, int n_f,
                    int precision, ss_batch** out) {
  if (!out) return fail(SS_ERR_ARG, "out must not be NULL");
  *out = nullptr;
  if (n_lattices < 1) return fail(SS_ERR_ARG, "n_lattices must be >= 1");
  if (precision != SS_FP32 && precision != SS_FP64) return fail(SS_ERR_ARG, "batches support SS_FP32 and SS_FP64");
  ss_batch* b = new ss_batch();
  b->theory = theory;
  b->precision = precision;
  b->n = n_lattices;
  b->elem = precision == SS_FP32 ? 4 : 8;
  b->inst.resize(n_lattices);
  long long total = 0;
  for (int i = 0; i < n_lattices; ++i) {
    ss_handle& h = b->inst[i];
    int rc = decode(&h, theory, p_i + (size_t)i * n_i, n_i, p_f + (size_t)i * n_f, n_f);
    if (rc) {
      char msg[sizeof(g_err)];
      snprintf(msg, sizeof(msg), "%s", g_err);
      delete b;
      return fail(rc, "lattice %d: %s", i, msg);
    }
    // partials and tile lists are sized for the finest shape the precision may use
    long long t = 0;
    for (int sh = 0; sh < (precision == SS_FP32 ? N_BATCH_SHAPES : 1); ++sh)
      for (int p = 0; p < 2; ++p) t = std::max(t, batch_tiles(b, h.G, sh, p));
    b->max_tiles.push_back((int)std::min(t, 0x7fffffffLL));
    total += t;
  }
  if (total > 0x7fffffffLL) {
    delete b;
    return fail(SS_ERR_ARG, "batch too large");
  }
  b->total_max = (int)total;
  b->shape.assign(n_lattices, 0);
  b->nf = b->inst[0].nf;
  *out = b;
  return SS_OK;
}

int ss_batch_destroy(ss_batch* b) {
  delete b;
  return SS_OK;
}

int ss_batch_workspace_bytes(const ss_batch* b, size_t* bytes) {
  if (!b || !bytes) return fail(SS_ERR_ARG, "NULL argument");
  ss_batch tmp = *b;
  tmp.graph = nullptr;  // the copy must not own the original's graph or staging
  tmp.h_stage = nullptr;
  *bytes = batch_layout(&tmp, nullptr);
  return SS_OK;
}

int ss_batch_bind(ss_batch* b, void* const* fields, void* const* velocities, void* workspace, size_t workspace_bytes,
                  void* stream) {
  if (!b || !fields || !velocities || !workspace) return fail(SS_ERR_ARG, "NULL argument");
  if (((uintptr_t)workspace) % ALIGN) return fail(SS_ERR_WORKSPACE, "workspace must be %zu-byte aligned", ALIGN);
  size_t need = 0;
  ss_batch_workspace_bytes(b, &need);
  if (workspace_bytes < need) return fail(SS_ERR_WORKSPACE, "workspace has %zu bytes, needs %zu", workspace_bytes, need);
  b->ws = (char*)workspace;
  b->stream = (cudaStream_t)stream;
  batch_layout(b, b->ws);
  b->fields.assign(fields, fields + b->n);
  b->vels.assign(velocities, velocities + b->n);
  bool tma = true;
  for (int i = 0; i < b->n; ++i) {
    BatchInst& I = b->h_insts[i];
    if (!fields[i] || !velocities[i]) return fail(SS_ERR_ARG, "lattice %d: NULL field or velocity", i);
    I.G = b->inst[i].G;
    I.G.pairs = site_pairs(I.G, b->elem, {fields[i], velocities[i]});
    I.P = b->inst[i].P;
    I.buf[0] = fields[i];
    I.buf[1] = velocities[i];
    if (tma) tma = batch_encode(b, i);
  }
  b->tma = tma;
  if (!tma) b->shape.assign(b->n, 0);  // the small shape is built for TMA staging only
  StepState init;
  memset(&init, 0, sizeof(init));
  init.E_last = NAN;
  const std::vector<StepState> inits(b->n, init);  // pageable: staged before the call returns
  CK(cudaMemcpyAsync(b->d_st, inits.data(), sizeof(StepState) * b->n, cudaMemcpyHostToDevice, b->stream));
  return batch_upload(b, nullptr);
}

int ss_batch_step(ss_batch* b, int n_steps, const double* prev_energy, double* energy_traj, double* err_traj) {
  if (!b || !b->ws) return fail(SS_ERR_STATE, "batch not bound");
  if (n_steps < 0) return fail(SS_ERR_ARG, "n_steps must be >= 0");
  if (prev_energy)
    CK(cudaMemcpyAsync(b->d_prev, prev_energy, sizeof(double) * b->n, cudaMemcpyHostToDevice, b->stream));
  bool use_prev = prev_energy != nullptr;
  // trajectories (k columns of every lattice's row) and the step states come back through
  // page-locked staging: one 2-D copy each, one synchronisation per chunk
  const size_t nn = (size_t)b->n;
  if (!b->h_stage)
    CK(cudaHostAlloc((void**)&b->h_stage, 2 * nn * TRAJ_CAP * sizeof(double) + nn * sizeof(StepState),
                     cudaHostAllocDefault));
  double* hE = reinterpret_cast<double*>(b->h_stage);
  double* hErr = hE + nn * TRAJ_CAP;
  StepState* hst = reinterpret_cast<StepState*>(hErr + nn * TRAJ_CAP);
  for (int done = 0; done < n_steps; done += TRAJ_CAP) {
    const int k = std::min(TRAJ_CAP, n_steps - done);
    int rc = batch_dispatch(b, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      if (b->precision == SS_FP32) return Batched<TH, float>::step(b, k, use_prev);
      return Batched<TH, double>::step(b, k, use_prev);
    });
    if (rc) return rc;
    use_prev = false;
    const size_t row = k * sizeof(double), pitch = TRAJ_CAP * sizeof(double);
    if (energy_traj) CK(cudaMemcpy2DAsync(hE, row, b->d_E, pitch, row, nn, cudaMemcpyDeviceToHost, b->stream));
    if (err_traj) CK(cudaMemcpy2DAsync(hErr, row, b->d_err, pitch, row, nn, cudaMemcpyDeviceToHost, b->stream));
    CK(cudaStreamSynchronize(b->stream));
    for (size_t i = 0; i < nn; ++i) {
      if (energy_traj) memcpy(energy_traj + i * n_steps + done, hE + i * k, row);
      if (err_traj) memcpy(err_traj + i * n_steps + done, hErr + i * k, row);
    }
  }
  CK(cudaMemcpyAsync(hst, b->d_st, nn * sizeof(StepState), cudaMemcpyDeviceToHost, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  int worst = 0;
  for (size_t i = 0; i < nn; ++i) {
    if (hst[i].status) {
      worst = std::max(worst, hst[i].status);
      hst[i].status = 0;
      idle_counters(hst[i]);
      CK(cudaMemcpyAsync(&b->d_st[i], &hst[i], sizeof(StepState), cudaMemcpyHostToDevice, b->stream));
    }
  }
  if (worst) CK(cudaStreamSynchronize(b->stream));
  if (worst == SS_ERR_TIMEOUT) return fail(SS_ERR_TIMEOUT, "a device-side wait timed out; re-bind the batch");
  if (worst) return fail(SS_ERR_NONFINITE, "a lattice's energy became non-finite");
  return SS_OK;
}

int ss_batch_tma_enabled(const ss_batch* b) { return b && b->tma ? 1 : 0; }

int ss_batch_get_shape(const ss_batch* b, int lattice) {
  if (!b || lattice < 0 || lattice >= b->n) return -1;
  return b->shape[lattice];
}

int ss_batch_set_shape(ss_batch* b, int lattice, int shape) {
  if (!b || !b->ws) return fail(SS_ERR_STATE, "batch not bound");
  if (lattice < 0 || lattice >= b->n) return fail(SS_ERR_ARG, "lattice %d out of range", lattice);
  if (shape < 0 || shape >= N_BATCH_SHAPES) return fail(SS_ERR_ARG, "tile shape %d: 0 (16 x 64) or 1 (8 x 32)", shape);
  if (shape != 0 && (!b->tma || b->precision != SS_FP32))
    return fail(SS_ERR_ARG, "the 8 x 32 tile shape needs TMA-staged FP32 lattices");
  b->shape[lattice] = shape;
  if (!batch_encode(b, lattice)) return fail(SS_ERR_CUDA, "tensor map of lattice %d", lattice);
  return batch_upload(b, nullptr);
}

int ss_batch_autotune(ss_batch* b, int iters, float* ms_out) {
  if (!b || !b->ws) return fail(SS_ERR_STATE, "batch not bound");
  if (iters < 1) iters = 1;
  if (ms_out)
    for (int i = 0; i < 2 * b->n; ++i) ms_out[i] = 0.f;
  if (!b->tma || b->precision != SS_FP32) return SS_OK;  // one tile shape only
  // size classes: lattices of equal extents
  std::vector<int> cls(b->n, -1);
  std::vector<std::pair<int, int>> keys;
  for (int i = 0; i < b->n; ++i) {
    const std::pair<int, int> k(b->inst[i].G.X, b->inst[i].G.Y);
    size_t c = 0;
    while (c < keys.size() && keys[c] != k) ++c;
    if (c == keys.size()) keys.push_back(k);
    cls[i] = (int)c;
  }
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  std::vector<float> ms(keys.size() * N_BATCH_SHAPES, 0.f);
  int rc = SS_OK;
  for (size_t c = 0; c < keys.size() && rc == SS_OK; ++c) {
    std::vector<char> inc(b->n, 0);
    for (int i = 0; i < b->n; ++i) inc[i] = cls[i] == (int)c;
    for (int sh = 0; sh < N_BATCH_SHAPES && rc == SS_OK; ++sh) {
      for (int i = 0; i < b->n; ++i)
        if (inc[i]) {
          b->shape[i] = sh;
          batch_encode(b, i);
        }
      if ((rc = batch_upload(b, &inc))) break;
      auto time_steps = [&](int n) -> int {
        return batch_dispatch(b, [&](auto* tag) -> int {
          using TH = std::remove_pointer_t<decltype(tag)>;
          for (int k = 0; k < n; ++k) {
            const int r = Batched<TH, float>::timing_step(b);
            if (r) return r;
          }
          return SS_OK;
        });
      };
      if ((rc = time_steps(1))) break;  // warm-up
      if (cudaEventRecord(e0, b->stream) != cudaSuccess) { rc = fail(SS_ERR_CUDA, "cudaEventRecord"); break; }
      if ((rc = time_steps(iters))) break;
      if (cudaEventRecord(e1, b->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) {
        rc = fail(SS_ERR_CUDA, "timing the batch's tile shapes");
        break;
      }
      float t = 0.f;
      cudaEventElapsedTime(&t, e0, e1);
      ms[c * N_BATCH_SHAPES + sh] = t / iters;
    }
    const int best = ms[c * N_BATCH_SHAPES + 1] < ms[c * N_BATCH_SHAPES] ? 1 : 0;
    for (int i = 0; i < b->n; ++i)
      if (inc[i]) {
        b->shape[i] = rc == SS_OK ? best : 0;
        batch_encode(b, i);
      }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const int up = batch_upload(b, nullptr);
  if (rc) return rc;
  if (up) return up;
  if (ms_out)
    for (int i = 0; i < b->n; ++i)
      for (int sh = 0; sh < N_BATCH_SHAPES; ++sh) ms_out[2 * i + sh] = ms[cls[i] * N_BATCH_SHAPES + sh];
  // the timing steps ran the phases with every state update off; only the ticket and
  // err slots they reset were touched
  return SS_OK;
}

}  // extern "C"


// ===========================================================================
// CUDA graphs of whole relaxations
// ===========================================================================
namespace {

// Capture `issue` (which launches on *stream_slot) on a private stream into a graph.
template <class Issue>
int capture_graph(cudaStream_t* stream_slot, cudaGraphExec_t* out, Issue&& issue) {
  cudaStream_t cs;
  CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  cudaStream_t saved = *stream_slot;
  *stream_slot = cs;
  cudaGraph_t g = nullptr;
  int rc = SS_OK;
  cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed);
  if (e == cudaSuccess) {
    rc = issue();
    cudaError_t e2 = cudaStreamEndCapture(cs, &g);
    if (rc == SS_OK && e2 != cudaSuccess) rc = fail(SS_ERR_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(e2));
  } else {
    rc = fail(SS_ERR_CUDA, "cudaStreamBeginCapture: %s", cudaGetErrorString(e));
  }
  *stream_slot = saved;
  if (rc == SS_OK) {
    if (*out) cudaGraphExecDestroy(*out);
    *out = nullptr;
    e = cudaGraphInstantiate(out, g, 0);
    if (e != cudaSuccess) rc = fail(SS_ERR_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(e));
  }
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(cs);
  return rc;
}

}  // namespace

extern "C" {

int ss_graph_create(ss_handle* h, int n_steps, double* energy_traj_dev, double* err_traj_dev) {
  int rc = check_bound(h);
  if (rc) return rc;
  if (n_steps < 1) return fail(SS_ERR_ARG, "n_steps must be >= 1");
  if (h->precision == SS_PLAIN_FP64) return fail(SS_ERR_ARG, "the plain FP64 form arrests on the host");
  return capture_graph(&h->stream, &h->graph,
                       [&]() { return ss_step_async(h, n_steps, NAN, energy_traj_dev, err_traj_dev); });
}

int ss_graph_launch(ss_handle* h) {
  if (!h || !h->graph) return fail(SS_ERR_STATE, "no graph captured: call ss_graph_create");
  CK(cudaGraphLaunch(h->graph, h->stream));
  return SS_OK;
}

int ss_batch_graph_create(ss_batch* b, int n_steps) {
  if (!b || !b->ws) return fail(SS_ERR_STATE, "batch not bound");
  if (n_steps < 1 || n_steps > TRAJ_CAP) return fail(SS_ERR_ARG, "n_steps must be in 1..%d", TRAJ_CAP);
  return capture_graph(&b->stream, &b->graph, [&]() {
    return batch_dispatch(b, [&](auto* tag) -> int {
      using TH = std::remove_pointer_t<decltype(tag)>;
      if (b->precision == SS_FP32) return Batched<TH, float>::step(b, n_steps, false);
      return Batched<TH, double>::step(b, n_steps, false);
    });
  });
}

int ss_batch_graph_launch(ss_batch* b) {
  if (!b || !b->graph) return fail(SS_ERR_STATE, "no graph captured: call ss_batch_graph_create");
  CK(cudaGraphLaunch(b->graph, b->stream));
  return SS_OK;
}

int ss_batch_trajectory(ss_batch* b, int n_steps, double* energy_traj, double* err_traj) {
  if (!b || !b->ws) return fail(SS_ERR_STATE, "batch not bound");
  if (n_steps < 0 || n_steps > TRAJ_CAP) return fail(SS_ERR_ARG, "n_steps must be in 0..%d", TRAJ_CAP);
  const size_t row = n_steps * sizeof(double), pitch = TRAJ_CAP * sizeof(double);
  if (n_steps > 0 && energy_traj)
    CK(cudaMemcpy2DAsync(energy_traj, row, b->d_E, pitch, row, b->n, cudaMemcpyDeviceToHost, b->stream));
  if (n_steps > 0 && err_traj)
    CK(cudaMemcpy2DAsync(err_traj, row, b->d_err, pitch, row, b->n, cudaMemcpyDeviceToHost, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return SS_OK;
}

}  // extern "C"
