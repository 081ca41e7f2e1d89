// libafar host<->device boundary: the drop-in replacement of the reference's GPUevolve.{h,cu}
// (setDeviceFieldData x2, adjustTimeStep, GPUevolve, copyFieldDataDeviceToHost, freeFieldData),
// plus graph-captured multi-step runs and per-stage parity hooks.
//
// The caller hands over the reference's host arrays (include/afar.h afar_fieldPointer); the
// library re-lays them out on the device (slot-major per-cell lists, per-face geometry constants,
// policy-typed intermediates; see afar_kernels.cuh) and owns all device memory.
#include <cuda_runtime.h>

#include <cstring>
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <tuple>
#include <vector>

#include <cudaTypedefs.h>  // PFN_cuTensorMapEncodeTiled
#include <nvtx3/nvToolsExt.h>

#include "afar_internal.h"
#include "afar_kernels.cuh"
#include "afar_order.cuh"

namespace {
// A named NVTX range over an entry point (host-side tracing: it shows the library's calls on a
// profiler timeline beside their kernels; inert without a profiler attached).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
};
}  // namespace

using namespace afar;

#define AFAR_CUDA(call)                                                                      \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess) {                                                                 \
      set_error("%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
      return AFAR_ERR_CUDA;                                                                  \
    }                                                                                        \
  } while (0)

namespace {

constexpr int kCellBlock = 128;
constexpr size_t kMaxDynamicSmem = 227 * 1024;  // per CTA on sm_103a
constexpr int kFaceBlock = 256;
constexpr int kSMs = 152;  // GB300
const unsigned long long kDtArmed = 0x40F86A0000000000ull;  // the Courant minimum before a step: bits of 1e5
constexpr int kFaceBlock64 = 128;  // ref and fp64: smaller blocks, an evener last wave over the SMs' FP64 pipes
// GPUevolve.cu:223-225: the reference's truncated SSP-RK3 coefficients
constexpr double kBeta1[3] = {1.0, 0.75, 0.333333};
constexpr double kBeta2[3] = {0.0, 0.25, 0.666667};
constexpr double kBeta3[3] = {1.0, 0.25, 0.666667};

struct FaceRaw {
  double x, y, magSf, Sfx, Sfy;
};

// Runs body(first, last) over [0, n) on the host's cores: up to 16, each at least `grain` long.
template <class F>
void parallel_ranges(long long n, long long grain, F&& body) {
  const long long hw = std::max(1u, std::thread::hardware_concurrency());
  const int k = (int)std::max(1ll, std::min({hw, 16ll, n / grain}));
  std::thread t[16];
  for (int i = 1; i < k; ++i) {
    try {
      t[i] = std::thread([&, i] { body(n * i / k, n * (i + 1) / k); });
    } catch (const std::system_error&) {  // no more threads: this one does the range
      body(n * i / k, n * (i + 1) / k);
    }
  }
  body(0ll, n / k);
  for (auto& x : t)
    if (x.joinable()) x.join();
}


// setup kernels that only move the reference arrays into the device layout
// (in the device's cell and face order: the caller's cell of device cell c is o.cell(c), and so on)
__global__ void k_setup_lists(int Nc, int Nf, int ldc, int maxS, int maxM, int maxLB, const uint8_t* nS,
                              const uint8_t* nM, const uint16_t* localStencil, const int* extendStencil,
                              const int* cellFaces, int* sten, int* cf, DeviceOrder o) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= Nc) return;
  const int h = o.cell(c);
  const int blk = h / AFAR_BLOCKDIM;
  for (int i = 0; i < nS[c]; ++i) {
    const int loc = localStencil[(size_t)maxS * h + i];
    const int g =
        loc < AFAR_BLOCKDIM ? blk * AFAR_BLOCKDIM + loc : extendStencil[(size_t)(maxLB - AFAR_BLOCKDIM) * blk + (loc - AFAR_BLOCKDIM)];
    sten[(size_t)i * ldc + c] = o.inv && g < Nc ? o.inv[g] : g;
  }
  for (int i = 0; i < nM[c]; ++i) {
    const int f = cellFaces[(size_t)maxM * h + i];
    const int d = o.finv && abs(f) - 1 < Nf ? o.finv[abs(f) - 1] + 1 : abs(f);
    cf[(size_t)i * ldc + c] = f < 0 ? -d : d;
  }
}
__global__ void k_split_faces(int n, int Nf, const FaceRaw* raw, V4<double>* xy, V4<double>* s, DeviceOrder o) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n) return;
  const FaceRaw r = raw[f < Nf ? o.face(f) : f];
  xy[f] = V4<double>{r.x, r.y, 0.0, 0.0};
  s[f] = V4<double>{r.Sfx, r.Sfy, r.magSf, 0.0};
}

template <class T, class Src>
__global__ void k_setup_wts(int Nc, int Nf, int ldc, int maxS, const uint8_t* nS, const uint8_t* nM, const int* cf,
                            const Src* rbf, T* wts, DeviceOrder o) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= Nc) return;
  const size_t nmax = (size_t)maxS + 1;
  for (int fi = 0; fi < nM[c]; ++fi) {
    int f = cf[(size_t)fi * ldc + c];
    const int side = f < 0;
    f = abs(f) - 1;
    if (f >= Nf) continue;
    const Src* src = rbf + 2 * nmax * o.face(f) + side * nmax;
    T* dst = wts + (size_t)fi * nmax * ldc + c;
    for (int j = 0; j <= nS[c]; ++j) dst[(size_t)j * ldc] = (T)src[j];
  }
}

__global__ void k_set_write_interval(StepCtl* ctl, double interval) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    ctl->write_interval = interval;
    ctl->write_index = interval > 0.0 ? (long long)floor(ctl->t / interval * (1.0 + 1e-12)) : 0;
  }
}

__global__ void k_set_ctl(StepCtl* ctl, double dt_fixed, double cfl, double t_end) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    ctl->dt_fixed = dt_fixed;
    ctl->cfl = cfl;
    ctl->t_end = t_end;
  }
}

__global__ void k_init_ctl(StepCtl* ctl) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    ctl->dt_bits = (unsigned long long)__double_as_longlong(1e5);
    ctl->t = 0.0;
    ctl->t_end = 0.0;
    ctl->dt_fixed = 0.0;
    ctl->cfl = 0.5;
    ctl->last_dt = 0.0;
    ctl->steps = 0;
    ctl->err = 0;
    ctl->write_interval = 0.0;
    ctl->write_index = 0;
    ctl->tiles_done = 0;
  }
}

__global__ void k_reciprocal(int n, const double* in, double* out, float* outf, DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    const double r = 1.0 / in[o.cell(i)];
    if (out) out[i] = r;
    if (outf) outf[i] = (float)r;
  }
}

// The mixed policy's conserved state: double -> float pair, and back, between the caller's cell order
// and the device's.
__global__ void k_df_from_double(int n, const V4<double>* in, V4<double>* out, DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V4<double> v = in[o.cell(i)];
  DF4 d;
  d.hi = V4<float>{(float)v.x, (float)v.y, (float)v.z, (float)v.w};
  d.lo = V4<float>{(float)(v.x - (double)d.hi.x), (float)(v.y - (double)d.hi.y), (float)(v.z - (double)d.hi.z),
                   (float)(v.w - (double)d.hi.w)};
  reinterpret_cast<DF4*>(out)[i] = d;
}
__global__ void k_df_to_double(int n, const DF4* in, V4<double>* out, DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const DF4 d = in[i];
  out[o.cell(i)] = V4<double>{(double)d.hi.x + (double)d.lo.x, (double)d.hi.y + (double)d.lo.y,
                              (double)d.hi.z + (double)d.lo.z, (double)d.hi.w + (double)d.lo.w};
}
// The switch flags (two a cell) into the caller's cell order.
__global__ void k_flags_out(int Nc, int n, const int8_t* in, int8_t* out, DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) reinterpret_cast<char2*>(out)[i < Nc ? o.cell(i) : i] = reinterpret_cast<const char2*>(in)[i];
}

// the primitive state (cells, then ghosts) into the device's cell order and out of it
// (the ghosts also into the state's other buffers: those of label 6 are never written again)
__global__ void k_state_in(int Nc, int n, const V4<double>* in, V4<float>* out, V4<float>* b, V4<float>* c,
                           DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V4<double> v = in[i < Nc ? o.cell(i) : i];
  const V4<float> w{(float)v.x, (float)v.y, (float)v.z, (float)v.w};
  out[i] = w;
  if (i >= Nc) b[i] = c[i] = w;
}
// (and the switch flags with it, two a cell, where they are asked for)
__global__ void k_state_out(int Nc, int n, const V4<float>* in, V4<double>* out, const int8_t* si, int8_t* si_out,
                            DeviceOrder o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V4<float> v = in[i];
  const int at = i < Nc ? o.cell(i) : i;
  out[at] = V4<double>{(double)v.x, (double)v.y, (double)v.z, (double)v.w};
  if (si_out) reinterpret_cast<char2*>(si_out)[at] = reinterpret_cast<const char2*>(si)[i];
}

// A device buffer of one call.
struct Scratch {
  void* p = nullptr;
  ~Scratch() { cudaFree(p); }
};

inline int grid_for(long long n, int block) { return (int)((n + block - 1) / block); }

StageCoef stage_coef(int k) {
  StageCoef c;
  c.b1 = kBeta1[k];
  c.b2 = kBeta2[k];
  c.b3 = kBeta3[k];
  c.b1h = (float)c.b1;
  c.b1l = (float)(c.b1 - (double)c.b1h);
  c.b2h = (float)c.b2;
  c.b2l = (float)(c.b2 - (double)c.b2h);
  c.first = k == 0;
  c.last = k == 2;
  return c;
}

}  // namespace

struct afar_solver {
  int policy = AFAR_POLICY_REF;
  int device = 0;
  cudaStream_t stream = nullptr;
  // sizes
  int Nc = 0, Nf = 0, Nb = 0, patches = 0, maxS = 0, maxM = 0, maxLB = 0, maxCLB = 0, ldc = 0;
  bool have_fields = false, have_stencil = false;
  double R = 0.0, Cv = 0.0;  // of the captured graph
  // policy-independent device arrays
  V2<double>* cellC = nullptr;
  FaceRaw* faceRaw = nullptr;
  double* vol = nullptr;
  double* vinv = nullptr;
  float* vinvf = nullptr;  // mixed: 1/V as float
  V2<float>* dtgf = nullptr;  // mixed: Courant geometry as float
  double px = 0.0, py = 0.0;  // periods of a periodic mesh (afar_set_periodic)
  int recon_variant = 0;      // mixed reconstruct: 0 tile-staged, 1 register pass (autotuned)
  int recon_request = -1;     // afar_set_tuning: -1 autotune, else the variant to use
  // The step split for the reference-shaped loop: afar_adjustTimeStep runs the head (stage 1 up to
  // its flux, whose fused reduction is the Courant step) instead of a separate Courant pass, and the
  // afar_GPUevolve that follows runs the tail (the rest of the step) with the caller's step size.
  // head_pending: the head ran on the current state and nothing has touched the solver since.
  cudaGraphExec_t graph_head = nullptr, graph_tail = nullptr;
  bool head_pending = false;
  // The fused stage leaves the limiter untransformed, and its head the switch types of the step
  // before: the state buffer of the last stage whose BVD the accessors still have to run (-1: none).
  int bvd_pending = -1;
  float tune_ms[2] = {0.f, 0.f};  // the autotuner's measured launch times (0: decision from the cache)
  // Which ghosts the state's buffers hold, of all that were uploaded (mixed), and which the snapshot does.
  long long ghosts = 0, ghosts_next = 0, snap_ghosts = 0;
  void* xfer = nullptr;    // mixed: staging for double <-> device-format copies, 32 B x (Nc + Nb)
  // The mixed policy keeps its cells along a Hilbert curve, its internal faces by their first cell in
  // that order (see setup_cell_order); everything that crosses the boundary is in the caller's order.
  DeviceOrder order;
  // The fused stage tail (tail_body) of the mixed policy: its tiles, the state's other two buffers, and
  // whether the mesh has it (`tail_faces` the most faces of a tile).
  TailTile* tail = nullptr;
  int *thalo = nullptr, *textra = nullptr, *tlist = nullptr;
  int* thcode = nullptr;
  V2<float>* thsg = nullptr;
  uint16_t* tlf = nullptr;
  unsigned* wflag = nullptr;
  void* Wb[2] = {nullptr, nullptr};
  bool fused = false;
  int tail_faces = 0;
  int2* on = nullptr;
  uint8_t* btype = nullptr;
  uint8_t* nS = nullptr;
  uint8_t* nM = nullptr;
  uint8_t* tileS = nullptr;  // per 128-cell tile: its largest stencil size
  TileMaps* tmaps = nullptr;  // mixed: tensor maps of the operator rows (device memory)
  int* sten = nullptr;
  int* cf = nullptr;
  V4<double>* U = nullptr;
  V4<double>* U0 = nullptr;
  int8_t* si = nullptr;
  V2<double>* dtg = nullptr;
  V2<double>* bn = nullptr;
  V4<double>* res_dbg = nullptr;
  afar_batch* batch = nullptr;  // the batch this solver belongs to, if any
  StepCtl* ctl = nullptr;
  unsigned long long* dt_bits = nullptr;
  unsigned long long* counters = nullptr;  // four, of afar_switch_counts
  // policy-typed device arrays (element size depends on the policy)
  void* W = nullptr;
  void* fd = nullptr;
  void* fs = nullptr;
  void* lsm = nullptr;
  void* sg = nullptr;
  void* sr = nullptr;
  void* wts = nullptr;
  void* grad = nullptr;
  void* lim = nullptr;
  void* fv = nullptr;
  void* flux = nullptr;
  void* snap = nullptr;       // device snapshot of W, U, U0, step control
  // the optional multi-point face flux (afar_set_face_gauss_flux): points per face (0: off)
  int ng = 0;
  void* wg = nullptr;
  void* sgk = nullptr;
  void* fgk = nullptr;
  void* fvg = nullptr;
  double gw[4] = {0.0, 0.0, 0.0, 0.0};
  std::vector<double> rbf64;  // optional FP64 weights awaiting the stencil upload
  cudaGraphExec_t graph = nullptr;
  size_t bytes = 0;
  std::vector<void*> allocs;
  // the block that dalloc cuts from (alloc_all), and the sizes it adds up while measuring
  char* block = nullptr;
  size_t block_left = 0, measured = 0;
  bool measuring = false;
};

namespace {

// Device memory of the solver's life: from the current block where there is room, else of its own.
afar_status dalloc(afar_solver* s, void** p, size_t bytes) {
  *p = nullptr;
  bytes = (std::max<size_t>(bytes, 16) + 511) / 512 * 512;
  if (s->measuring) {
    s->measured += bytes;
    return AFAR_OK;
  }
  if (bytes <= s->block_left) {
    *p = s->block;
    s->block += bytes;
    s->block_left -= bytes;
    return AFAR_OK;
  }
  AFAR_CUDA(cudaMalloc(p, bytes));
  s->allocs.push_back(*p);
  s->bytes += bytes;
  return AFAR_OK;
}
// The allocations of `f` from one block of their total size: a cudaMalloc costs tens of microseconds
// and its cudaFree more, and a solver has 40 arrays (set-up and release of a mixed solver of 44k cells: 3.36 -> 1.66 ms,
// 10k cells: 1.40 -> 1.14).
template <class F>
afar_status alloc_all(afar_solver* s, F&& f) {
  s->measuring = true;
  s->measured = 0;
  f();
  s->measuring = false;
  AFAR_CUDA(cudaMalloc(reinterpret_cast<void**>(&s->block), s->measured));
  s->allocs.push_back(s->block);
  s->bytes += s->measured;
  s->block_left = s->measured;
  const afar_status st = f();
  s->block_left = 0;
  return st;
}
template <class T>
afar_status dalloc_t(afar_solver* s, T** p, size_t n) {
  return dalloc(s, reinterpret_cast<void**>(p), n * sizeof(T));
}

// Cells of a tile of the fused stage tail: as many as its 256 threads take with the halo in one pass (192
// triangles, 152 quads), fewer quads where a mesh is a few blocks and a block's time is the kernel's.  us a
// step at 96 / 152 / 192 cells: triangles 1.1k 41 / 43 / 41, 99k 72 / 73 / 68, 998k 588 / 512 / 497; quads 1.0k 42 / 45 / 58,
// 10k 46.5 / 47.2 / 61, 66k 70 / 62 / 72, 1.0M 670 / 584 / 631.  The line is where batches of such meshes begin to
// lose: 96 / 152 cells, 4096 quads alone 32.8 / 33.0, six, twelve and 24 members 40.7 / 41.0, 51.2 / 52.4, 85.8 / 84.0; 5041
// alone 32.8 / 34.8, six and twelve members 42.8 / 44.3, 66.4 / 55.3; 10k alone 33.4 / 34.8, six members 65.3 / 54.7.
int tail_cells(const afar_solver* s) { return tail_tile_cells(s->maxM, s->Nc); }

template <class P>
StageArgs<P> make_args(afar_solver* s) {
  StageArgs<P> a;
  using S = typename P::S;
  using G = typename P::G;
  a.Nc = s->Nc;
  a.Nf = s->Nf;
  a.Nb = s->Nb;
  a.ldc = s->ldc;
  a.maxS = s->maxS;
  a.maxM = s->maxM;
  a.cellC = s->cellC;
  a.on = s->on;
  a.fd = static_cast<const V4<G>*>(s->fd);
  a.fs = static_cast<const V4<G>*>(s->fs);
  a.dtg = s->dtg;
  a.bn = s->bn;
  a.btype = s->btype;
  a.vol = s->vol;
  a.nS = s->nS;
  a.tileS = s->tileS;
  a.nM = s->nM;
  a.sten = s->sten;
  a.cf = s->cf;
  a.lsm = static_cast<const V2<S>*>(s->lsm);
  a.sg = static_cast<const V2<G>*>(s->sg);
  a.sr = static_cast<const V2<S>*>(s->sr);
  a.wts = static_cast<const S*>(s->wts);
  a.tmaps = s->tmaps;
  a.W = static_cast<V4<typename P::W>*>(s->W);
  a.U = s->U;
  a.U0 = s->U0;
  a.grad = static_cast<V4<G>*>(s->grad);
  a.lim = static_cast<V4<S>*>(s->lim);
  a.si = s->si;
  a.fv = static_cast<V4<G>*>(s->fv);
  a.flux = static_cast<V4<typename P::F>*>(s->flux);
  a.vinv = s->vinv;
  a.ctl = s->ctl;
  a.res_dbg = nullptr;
  a.R = s->R;
  a.Cv = s->Cv;
  a.invR = s->R > 0.0 ? 1.0 / s->R : 0.0;
  a.gamma = s->Cv > 0.0 ? s->R / s->Cv + 1.0 : 0.0;
  a.Cp = s->Cv + s->R;
  a.gm1 = a.gamma - 1.0;
  a.gR = a.gamma * s->R;
  a.gm1f = (float)a.gm1;
  a.invRf = (float)a.invR;
  a.vinvf = s->vinvf;
  a.Rf = (float)s->R;
  a.Cvf = (float)s->Cv;
  a.gRf = (float)(a.gamma * s->R);
  a.dtgf = s->dtgf;
  a.px = s->px;
  a.py = s->py;
  a.tail = s->tail;
  a.thalo = s->thalo;
  a.thcode = s->thcode;
  a.thsg = reinterpret_cast<const V2<G>*>(s->thsg);
  a.textra = s->textra;
  a.tlf = s->tlf;
  a.tlist = s->tlist;
  a.wflag = s->wflag;
  a.W3[0] = a.W;
  for (int i = 0; i < 2; ++i) a.W3[i + 1] = static_cast<V4<typename P::W>*>(s->Wb[i]);
  a.tailT = tail_cells(s);
  a.nTail = (s->Nc + a.tailT - 1) / a.tailT;
  a.ng = s->ng;
  a.wg = static_cast<const S*>(s->wg);
  a.sgk = static_cast<const V2<G>*>(s->sgk);
  a.fgk = static_cast<const V2<G>*>(s->fgk);
  a.fvg = static_cast<V4<G>*>(s->fvg);
  for (int k = 0; k < 4; ++k) a.gw[k] = (G)s->gw[k];
  return a;
}

// cudaFuncAttributeMaxDynamicSharedMemorySize of a staged reconstruct kernel only grows (per
// device), so solvers and batches of different stencil sizes never lower one another's limit.
template <class K>
afar_status raise_smem_limit(K kernel, int device, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, size_t> done;
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = done[{reinterpret_cast<const void*>(kernel), device}];
  if (bytes > cur) {
    AFAR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cur = bytes;
  }
  return AFAR_OK;
}

// Threads a block of the single-solve kernels over n cells or faces.  The ref and fp64 kernels are
// bound by each SM's FP64 pipe, so a mesh too small to give every SM eight full blocks is cut into
// smaller ones until it reaches all SMs evenly: the pipe's time on the busiest SM is the kernel's.  us a
// step in blocks of 128 / 64 / 32: fp64, 41k triangles 267 / 242 / 237, 121k 553 / 545 / 550, 500k 1980 /
// 1966 / 1972; ref, 41k 333 / 294 / 281, 250k quads 1027 / 1022 / 1018.
template <class P>
int block_for(long long n, int full) {
  if constexpr (P::id == PolicyMixed::id) return full;
  int b = full;
  while (b > 32 && n < 8ll * kSMs * b) b /= 2;
  return b;
}

// Dynamic shared memory of the reconstruct: the mixed policy stages a whole 128-cell tile of
// operator rows (recon_tile_layout); ref stages the stencil values, fp64 the compact stencil's.
template <class P>
size_t recon_smem(const afar_solver* s, int block = kCellBlock) {
  if constexpr (P::id == PolicyMixed::id) return recon_tile_layout(s->maxM, s->maxS).bytes;
  const int rows = P::id == PolicyFP64::id ? s->maxM : s->maxS;  // fp64 stages the compact stencil only
  return (size_t)(rows > 0 ? rows : 1) * block * sizeof(V4<typename P::S>);
}

// mixed: the step runs as the fused stage (see enqueue_step)
inline bool fused_step(const afar_solver* s) { return s->fused && s->ng == 0; }

// One solve's stage launches, arguments by value.  The ref policy reconstructs in the staged
// kernel and runs the reference-layout flux; fp64 reconstructs staged, mixed in registers.
// The fused stage's kernels start before the one ahead is complete (pdl_next near its end): their
// barriers, lists and operator rows are on the way when its results are there.  us a step, without / with:
// 1k quads 43.6 / 39.2, 10k 47 / 41, 256k 161.6 / 155.7, 640k 361 / 354, 1.5M 784 / 778, 4.0M 1961 / 1954 (face-neighbour
// stencils 197.6 / 191.6, 422.6 / 419.5, 908 / 901, 2223 / 2217); 10k triangles 46 / 40, 202k 130 / 121, 2.0M 946 / 937.
// (Saying pdl_next first thing: 4.0M quads 2308, 2.0M triangles 1003: the next kernel's waiting blocks take the
// places of blocks that have work.)
// Not the tail where a quad mesh's reconstruct has 2 to 3.5 blocks a SM: its blocks crowd where that ends first.
// us a step with the tail early / on completion, edge- and face-neighbour stencils: 250 blocks 39.0 / 38.8 and
// 51.0 / 51.2, 300 41.7 / 39.8 and 54.0 / 51.9, 350 42.8 / 41.0 and 58.8 / 54.1, 400 45.4 / 45.1 and 59.9 / 57.4, 450 47.1 / 46.0
// and 61.7 / 57.4, 500 47.1 / 45.3 and 62.8 / 59.3, 549 47.2 / 49.2 and 64.0 / 61.3, 574 48.2 / 51.2 and 65.0 / 63.5,
// 600 48.8 / 51.2 and 65.2 / 65.3, 650 55.2 / 57.2 and 71.7 / 75.0, 800 70.6 / 73.8 and 87.9 / 90.3.
inline bool tail_early(int maxM, long long reconBlocks) {
  return maxM <= 3 || reconBlocks <= 2 * kSMs || 2 * reconBlocks > 7 * kSMs;
}

// Launches a kernel, with pdl as the programmatic dependent of the one before it on the stream.
template <class... A, class... B>
void launch(void (*kernel)(A...), int grid, int block, size_t smem, cudaStream_t stream, bool pdl, const B&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, A(args)...);
}

template <class P>
struct Stage {
  afar_solver* s;
  StageArgs<P> a;
  bool pdl = false;  // the launch may start before the one ahead of it is complete
  int bc() const { return block_for<P>(s->Nc, kCellBlock); }
  int gc() const { return grid_for(s->Nc, bc()); }

  // dt (mixed): also reduce the Courant step
  void reconstruct(bool dt = false) const {
    if constexpr (P::id == PolicyMixed::id) {
      const auto tile = s->maxM <= 3 ? (dt ? k_reconstruct_tile<P, 3, true> : k_reconstruct_tile<P, 3, false>)
                                     : (dt ? k_reconstruct_tile<P, 4, true> : k_reconstruct_tile<P, 4, false>);
      const auto reg = dt ? k_reconstruct_reg<P, true> : k_reconstruct_reg<P, false>;
      if (s->recon_variant == 1)
        launch(reg, gc(), kCellBlock, 0, s->stream, pdl, a);
      else
        launch(tile, gc(), kTile, recon_smem<P>(s), s->stream, pdl, a);
    } else
      k_reconstruct_staged<P><<<gc(), bc(), recon_smem<P>(s, bc()), s->stream>>>(a);
    if constexpr (P::id != PolicyRef::id) {
      if (s->ng > 0) k_reconstruct_gauss<P><<<gc(), bc(), 0, s->stream>>>(a);
    }
  }
  // mixed: everything after the reconstruct in one kernel where the mesh has its tiles
  bool fused() const { return P::id == PolicyMixed::id && fused_step(s); }
  // the reconstruct and the rest of stage k with the state in the k-th buffer
  Stage<P> at(int k) const {
    Stage<P> r = *this;
    r.a.W = a.W3[k];
    return r;
  }
  void tail(int k) const {
    if constexpr (P::id == PolicyMixed::id) {
      const auto f = s->maxM <= 3 ? k_tail<3> : k_tail<4>;
      launch(f, a.nTail, kTailThreads, tail_smem(s->tail_faces, tail_cells(s)).bytes, s->stream, pdl, a,
             a.W3[(k + 1) % 3], stage_coef(k));
    }
  }
  void bvd() const { k_bvd<P><<<gc(), bc(), 0, s->stream>>>(a); }
  // The face flux.  The ref policy computes the CFL step as a kernel of its own before the first
  // stage's flux, like the reference's setDeltaT; the other policies fuse it into that flux.
  void flux(bool dt_stage) const {
    const int bf = block_for<P>((long long)s->Nf + s->Nb, P::id == PolicyMixed::id ? kFaceBlock : kFaceBlock64);
    const int gf = grid_for((long long)s->Nf + s->Nb, bf);
    if constexpr (P::id == PolicyRef::id) {
      if (dt_stage && s->Nf > 0)
        k_delta_t<P><<<grid_for(s->Nf, bf), bf, 0, s->stream>>>(a, 0.0, &s->ctl->dt_bits, s->ctl);
      k_flux<P, false><<<gf, bf, 0, s->stream>>>(a);
    } else if (s->ng > 0) {  // the multi-point face flux; the Courant step as a kernel of its own
      if (dt_stage && s->Nf > 0)
        k_delta_t<P><<<grid_for(s->Nf, bf), bf, 0, s->stream>>>(a, 0.0, &s->ctl->dt_bits, s->ctl);
      k_flux_gauss<P><<<gf, bf, 0, s->stream>>>(a);
    } else {
      if (dt_stage)
        k_flux<P, true><<<gf, bf, 0, s->stream>>>(a);
      else
        k_flux<P, false><<<gf, bf, 0, s->stream>>>(a);
    }
  }
  void update(int k) const {
    k_update<P><<<gc(), bc(), 0, s->stream>>>(a, stage_coef(k));
  }
};

// Stage launcher of a solver; debug = true also writes the residual copy (afar_stage_debug).
template <class P>
afar_status make_stage(afar_solver* s, bool debug, Stage<P>* out) {
  out->s = s;
  out->a = make_args<P>(s);
  if (debug) out->a.res_dbg = s->res_dbg;
  return AFAR_OK;
}

// A step is its head (stage 1 as far as the Courant step) and its tail.  Fused (mixed): two kernels a
// stage, the head the first reconstruct.
template <class P>
void enqueue_head(const Stage<P>& st) {
  st.reconstruct(st.fused());
  if (st.fused()) return;
  st.bvd();
  st.flux(true);
}
template <class P>
void enqueue_tail(const Stage<P>& st) {
  if (st.fused()) {
    Stage<P> d = st;
    for (int k = 0; k < 3; ++k) {
      d.pdl = true;
      if (k > 0) d.at(k).reconstruct();
      d.pdl = tail_early(st.s->maxM, d.gc());
      d.at(k).tail(k);
    }
    return;
  }
  st.update(0);
  for (int k = 1; k < 3; ++k) {
    st.reconstruct();
    st.bvd();
    st.flux(false);
    st.update(k);
  }
  k_finish_step<<<1, 32, 0, st.s->stream>>>(st.s->ctl);
}

// What the separate BVD kernel leaves behind, after a fused stage: for the accessors of the limiter and
// of the switch types, and before anything replaces what it reads (a head's state, a stage's limiter, face
// values and flags).  A pending head no longer fits its tail then (the tail transforms the limiter).
afar_status settle_bvd(afar_solver* s) {
  if (s->bvd_pending < 0) return AFAR_OK;
  Stage<PolicyMixed> st;
  if (afar_status r = make_stage<PolicyMixed>(s, false, &st)) return r;
  st.at(s->bvd_pending).bvd();
  s->bvd_pending = -1;
  s->head_pending = false;
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  return AFAR_OK;
}

template <class P>
void enqueue_step(const Stage<P>& st) {
  enqueue_head(st);
  enqueue_tail(st);
}

template <class P>
afar_status setup_operators(afar_solver* s, const afar_fieldPointer* h, void* scratch) {
  using S = typename P::S;
  using G = typename P::G;
  const int Nc = s->Nc, Nf = s->Nf, Nb = s->Nb, ldc = s->ldc;
  afar_status st;
  AFAR_CUDA(cudaMemsetAsync(s->wts, 0, sizeof(S) * (size_t)s->maxM * (s->maxS + 1) * ldc, s->stream));
  AFAR_CUDA(cudaMemsetAsync(s->lsm, 0, sizeof(V2<S>) * (size_t)s->maxM * ldc, s->stream));

  // O3 weights: float reference layout (or the FP64 copy) -> slot-major
  const size_t nrbf = 2 * (size_t)(s->maxS + 1) * Nf;
  const int gc = grid_for(Nc, kCellBlock);
  if (std::is_same<S, double>::value && s->rbf64.size() == nrbf) {
    double* tmp = static_cast<double*>(scratch);
    AFAR_CUDA(cudaMemcpyAsync(tmp, s->rbf64.data(), sizeof(double) * nrbf, cudaMemcpyHostToDevice, s->stream));
    k_setup_wts<S, double><<<gc, kCellBlock, 0, s->stream>>>(Nc, Nf, ldc, s->maxS, s->nS, s->nM, s->cf, tmp,
                                                             static_cast<S*>(s->wts), s->order);
  } else {
    float* tmp = static_cast<float*>(scratch);
    AFAR_CUDA(cudaMemcpyAsync(tmp, h->RBFbasis, sizeof(float) * nrbf, cudaMemcpyHostToDevice, s->stream));
    k_setup_wts<S, float><<<gc, kCellBlock, 0, s->stream>>>(Nc, Nf, ldc, s->maxS, s->nS, s->nM, s->cf, tmp,
                                                            static_cast<S*>(s->wts), s->order);
  }
  V4<double>* fxy = static_cast<V4<double>*>(scratch);
  V4<double>* fsr = fxy + (Nf + Nb + 1);
  const int gF = grid_for((long long)Nf + Nb, kFaceBlock);
  k_split_faces<<<gF, kFaceBlock, 0, s->stream>>>(Nf + Nb, Nf, s->faceRaw, fxy, fsr, s->order);
  StageArgs<P> a = make_args<P>(s);
  k_setup_lsm<P><<<gc, kCellBlock, 0, s->stream>>>(a, static_cast<V2<S>*>(s->lsm), nullptr, 0, nullptr);
  k_setup_slot_geom<P><<<gc, kCellBlock, 0, s->stream>>>(a, fxy);
  k_setup_face_geom<P><<<gF, kFaceBlock, 0, s->stream>>>(a, fxy, fsr);
  if constexpr (P::id == PolicyMixed::id) {
  }
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  s->rbf64.clear();
  s->rbf64.shrink_to_fit();
  if constexpr (P::id != PolicyMixed::id) {
    return raise_smem_limit(k_reconstruct_staged<P>, s->device, recon_smem<P>(s));
  } else {
    if (recon_smem<P>(s) > kMaxDynamicSmem) {
      set_error("stencil too large for the reconstruct tile: %zu bytes of shared memory", recon_smem<P>(s));
      return AFAR_ERR_LIMIT;
    }
    if ((st = raise_smem_limit(k_reconstruct_tile<P, 3, false>, s->device, recon_smem<P>(s)))) return st;
    if ((st = raise_smem_limit(k_reconstruct_tile<P, 3, true>, s->device, recon_smem<P>(s)))) return st;
    if ((st = raise_smem_limit(k_reconstruct_tile<P, 4, false>, s->device, recon_smem<P>(s)))) return st;
    return raise_smem_limit(k_reconstruct_tile<P, 4, true>, s->device, recon_smem<P>(s));
  }
}

void destroy_graphs(afar_solver* s) {
  for (cudaGraphExec_t* g : {&s->graph, &s->graph_head, &s->graph_tail})
    if (*g) {
      cudaGraphExecDestroy(*g);
      *g = nullptr;
    }
  s->head_pending = false;
}

// One of the step's graphs: the whole step, its head, or its tail (the same launches split in two).
enum { kGraphStep, kGraphHead, kGraphTail };
afar_status capture_graph(afar_solver* s, int which) {
  cudaGraphExec_t* const out[3] = {&s->graph, &s->graph_head, &s->graph_tail};
  cudaGraph_t g = nullptr;
  auto capture = [&](auto tag) -> afar_status {
    using P = decltype(tag);
    Stage<P> st;
    afar_status r = make_stage<P>(s, false, &st);
    if (r) return r;
    AFAR_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    if (which == kGraphStep) enqueue_step<P>(st);
    if (which == kGraphHead) enqueue_head<P>(st);
    if (which == kGraphTail) enqueue_tail<P>(st);
    AFAR_CUDA(cudaStreamEndCapture(s->stream, &g));
    return AFAR_OK;
  };
  afar_status r;
  switch (s->policy) {
    case AFAR_POLICY_REF: r = capture(PolicyRef{}); break;
    case AFAR_POLICY_FP64: r = capture(PolicyFP64{}); break;
    default: r = capture(PolicyMixed{}); break;
  }
  if (r) return r;
  const cudaError_t e = cudaGraphInstantiate(out[which], g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    *out[which] = nullptr;
    set_error("cudaGraphInstantiate failed: %s", cudaGetErrorString(e));
    return AFAR_ERR_CUDA;
  }
  return AFAR_OK;
}

afar_status check_ready(afar_solver* s) {
  if (!s) {
    set_error("null solver");
    return AFAR_ERR_ARGUMENT;
  }
  s->head_pending = false;  // every call that goes through here may change what the head computed
  if (!s->have_fields || !s->have_stencil) {
    set_error("call afar_setDeviceFieldData and afar_setDeviceFieldDataStencil first");
    return AFAR_ERR_STATE;
  }
  AFAR_CUDA(cudaSetDevice(s->device));
  return AFAR_OK;
}

// Stepping a batch member on its own would race with (and desynchronise) the batch.
afar_status check_not_batched(afar_solver* s) {
  if (s->batch) {
    set_error("the solver belongs to a batch: step it with afar_batch_run or remove it first");
    return AFAR_ERR_STATE;
  }
  return AFAR_OK;
}

// Reads (and clears) the device error word after a wait: a bounded device wait that gave up marks
// the step's results invalid.
afar_status check_device_error(afar_solver* s) {
  unsigned err = 0;
  AFAR_CUDA(cudaMemcpyAsync(&err, &s->ctl->err, sizeof(err), cudaMemcpyDeviceToHost, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  if (err) {
    AFAR_CUDA(cudaMemsetAsync(&s->ctl->err, 0, sizeof(err), s->stream));
    AFAR_CUDA(cudaStreamSynchronize(s->stream));
    set_error("a device-side wait for a bulk copy timed out (error word %u); the state is not valid", err);
    return AFAR_ERR_CUDA;
  }
  return AFAR_OK;
}

size_t w_size(int policy) { return policy == AFAR_POLICY_MIXED ? sizeof(V4<float>) : sizeof(V4<double>); }

}  // namespace

// ------------------------------------------------------------------------------------------------
extern "C" afar_status afar_solver_create(afar_solver** out, int policy, int device) {
  if (!out || policy < AFAR_POLICY_REF || policy > AFAR_POLICY_MIXED) {
    set_error("afar_solver_create: null output or unknown policy %d", policy);
    return AFAR_ERR_ARGUMENT;
  }
  *out = nullptr;
  int n = 0;
  AFAR_CUDA(cudaGetDeviceCount(&n));
  if (device < 0 || device >= n) {
    set_error("afar_solver_create: device %d not present (%d devices)", device, n);
    return AFAR_ERR_ARGUMENT;
  }
  AFAR_CUDA(cudaSetDevice(device));
  afar_solver* s = new afar_solver();
  s->policy = policy;
  s->device = device;
  if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) {
    set_error("cudaStreamCreate failed");
    delete s;
    return AFAR_ERR_CUDA;
  }
  *out = s;
  return AFAR_OK;
}

// Host <-> device state in the reference's double layout, ordered on the solver's stream.  The
// mixed policy keeps W as float and U, Un as float pairs: the doubles are staged in `xfer` and
// converted on the device.
static afar_status put_state(afar_solver* s, const afar_basicFieldData* FD, const afar_conservedFieldData* cFD,
                      const afar_conservedFieldData* cFDold) {
  const size_t Nc = s->Nc, Nb = s->Nb;
  const bool mixed = s->policy == AFAR_POLICY_MIXED;
  if (FD && s->bvd_pending == 0) {  // (a later stage's state is in a buffer of its own)
    if (afar_status st = settle_bvd(s)) return st;
  }
  if (FD) {
    s->ghosts = ++s->ghosts_next;
    if (mixed) {
      AFAR_CUDA(cudaMemcpyAsync(s->xfer, FD, sizeof(V4<double>) * (Nc + Nb), cudaMemcpyHostToDevice, s->stream));
      k_state_in<<<grid_for(Nc + Nb, 256), 256, 0, s->stream>>>((int)Nc, (int)(Nc + Nb),
                                                                static_cast<const V4<double>*>(s->xfer),
                                                                static_cast<V4<float>*>(s->W),
                                                                static_cast<V4<float>*>(s->Wb[0]),
                                                                static_cast<V4<float>*>(s->Wb[1]), s->order);
    } else {
      AFAR_CUDA(cudaMemcpyAsync(s->W, FD, sizeof(V4<double>) * (Nc + Nb), cudaMemcpyHostToDevice, s->stream));
    }
  }
  const afar_conservedFieldData* src[2] = {cFD, cFDold};
  V4<double>* dst[2] = {s->U, s->U0};
  for (int i = 0; i < 2; ++i) {
    if (!src[i]) continue;
    if (i == 1 && cFDold == cFD) {  // the same host array twice: one upload, then a device copy
      AFAR_CUDA(cudaMemcpyAsync(s->U0, s->U, sizeof(V4<double>) * Nc, cudaMemcpyDeviceToDevice, s->stream));
      continue;
    }
    void* to = mixed ? s->xfer : dst[i];
    AFAR_CUDA(cudaMemcpyAsync(to, src[i], sizeof(V4<double>) * Nc, cudaMemcpyHostToDevice, s->stream));
    if (mixed)
      k_df_from_double<<<grid_for(Nc, 256), 256, 0, s->stream>>>((int)Nc, static_cast<const V4<double>*>(s->xfer),
                                                                 dst[i], s->order);
  }
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  return AFAR_OK;
}

// (the mixed policy's arrays leave through `xfer` one after another, in the stream's order)
static afar_status get_state(afar_solver* s, afar_basicFieldData* FD, afar_conservedFieldData* cFD, int8_t* si) {
  const size_t Nc = s->Nc, Nb = s->Nb, n = Nc + Nb;
  if (si && s->bvd_pending == 0) {  // a fused head: its stage's types
    if (afar_status st = settle_bvd(s)) return st;
  }
  const void *fd = s->W, *cfd = s->U;
  const int8_t* flags = s->si;
  const bool mixed = s->policy == AFAR_POLICY_MIXED;
  if (mixed) {
    int8_t* const to = si ? static_cast<int8_t*>(s->xfer) + sizeof(V4<double>) * n : nullptr;  // past the state's place
    if (FD)
      k_state_out<<<grid_for(n, 256), 256, 0, s->stream>>>((int)Nc, (int)n, static_cast<const V4<float>*>(s->W),
                                                           static_cast<V4<double>*>(s->xfer), s->si, to, s->order);
    else if (si)
      k_flags_out<<<grid_for(n, 256), 256, 0, s->stream>>>((int)Nc, (int)n, s->si, to, s->order);
    fd = cfd = s->xfer;
    flags = to;
  }
  if (FD) AFAR_CUDA(cudaMemcpyAsync(FD, fd, sizeof(V4<double>) * n, cudaMemcpyDeviceToHost, s->stream));
  if (si) AFAR_CUDA(cudaMemcpyAsync(si, flags, 2 * n, cudaMemcpyDeviceToHost, s->stream));
  if (cFD) {
    if (mixed)
      k_df_to_double<<<grid_for(Nc, 256), 256, 0, s->stream>>>((int)Nc, reinterpret_cast<const DF4*>(s->U),
                                                               static_cast<V4<double>*>(s->xfer), s->order);
    AFAR_CUDA(cudaMemcpyAsync(cFD, cfd, sizeof(V4<double>) * Nc, cudaMemcpyDeviceToHost, s->stream));
  }
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  return AFAR_OK;
}

// The project autotuner: the mixed reconstruct has two implementations whose speed depends on the
// mesh (stencil size, faces per cell, size): the tile-staged kernel (TMA loads of each 128-cell
// tile's operator rows into shared memory) and the register pass (no shared memory, more tiles per
// SM).  At the stencil upload each is timed on the solver's own data (one warm-up, best of three times
// the launches of a step, the first of a fused one with its Courant step; CUDA events on its stream; the
// launches only write the stage's intermediates and that minimum) and the faster kept.  Decisions are
// cached per device and mesh class (faces per cell, stencil size, cell count to a factor of two), so later
// solvers of the same class skip the timing.
// cuTensorMapEncodeTiled, looked up once through the runtime (the library links no driver API).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// The tensor maps of the mixed tile-staged reconstruct (TileMaps): built on the host after the
// operator rows are in place and copied to the solver's device memory.  Each map describes one
// slot-major array as rows of ldc elements (ldc a multiple of 32, so every row stride is a multiple
// of 128 bytes), with boxes of 128 cells.
static afar_status build_tile_maps(afar_solver* s) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return (set_error("cuTensorMapEncodeTiled is not available from the driver"), AFAR_ERR_CUDA);
  TileMaps h;
  std::memset(&h, 0, sizeof(h));
  const cuuint64_t ldc = (cuuint64_t)s->ldc, M = (cuuint64_t)s->maxM, S = (cuuint64_t)s->maxS;
  const cuuint32_t one[3] = {1, 1, 1};
  auto encode = [&](CUtensorMap* m, CUtensorMapDataType dt, cuuint32_t rank, void* base, const cuuint64_t* dims,
                    const cuuint64_t* strides, const cuuint32_t* box) -> afar_status {
    const CUresult r = enc(m, dt, rank, base, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return (set_error("cuTensorMapEncodeTiled failed (%d)", (int)r), AFAR_ERR_CUDA);
    return AFAR_OK;
  };
  afar_status st;
  {
    const cuuint64_t dims[2] = {ldc, M}, strides[1] = {ldc * 4};
    const cuuint32_t box[2] = {(cuuint32_t)kTile, (cuuint32_t)M};
    if ((st = encode(&h.cf, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, s->cf, dims, strides, box))) return st;
  }
  {
    const cuuint64_t dims[2] = {2 * ldc, M}, strides[1] = {ldc * 8};
    const cuuint32_t box[2] = {(cuuint32_t)(2 * kTile), (cuuint32_t)M};
    if ((st = encode(&h.lsm, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, s->lsm, dims, strides, box))) return st;
    if ((st = encode(&h.sg, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, s->sg, dims, strides, box))) return st;
    if ((st = encode(&h.sr, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, s->sr, dims, strides, box))) return st;
  }
  for (cuuint32_t k = 1; k <= (cuuint32_t)S; ++k) {
    const cuuint64_t dims[2] = {ldc, S}, strides[1] = {ldc * 4};
    const cuuint32_t box[2] = {(cuuint32_t)kTile, k};
    if ((st = encode(&h.sten[k - 1], CU_TENSOR_MAP_DATA_TYPE_INT32, 2, s->sten, dims, strides, box))) return st;
    const cuuint64_t wdims[3] = {ldc, S + 1, M}, wstrides[2] = {ldc * 4, ldc * 4 * (S + 1)};
    const cuuint32_t wbox[3] = {(cuuint32_t)kTile, k, (cuuint32_t)M};
    if ((st = encode(&h.wts[k - 1], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, s->wts, wdims, wstrides, wbox))) return st;
  }
  AFAR_CUDA(cudaMemcpy(s->tmaps, &h, sizeof(TileMaps), cudaMemcpyHostToDevice));
  return AFAR_OK;
}

static afar_status tune_reconstruct(afar_solver* s) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, int>, int> cache;
  if (s->recon_request >= 0) {
    s->recon_variant = s->recon_request;
    return AFAR_OK;
  }
  int lg = 0;
  while ((1 << (lg + 1)) <= s->Nc) ++lg;
  const auto key = std::make_tuple(s->device, s->maxM, s->maxS, lg);
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      s->recon_variant = it->second;
      s->tune_ms[0] = s->tune_ms[1] = 0.f;
      return AFAR_OK;
    }
  }
  Stage<PolicyMixed> sg;
  afar_status st = settle_bvd(s);
  if (st || (st = make_stage<PolicyMixed>(s, false, &sg))) return st;
  cudaEvent_t e0, e1;
  AFAR_CUDA(cudaEventCreate(&e0));
  AFAR_CUDA(cudaEventCreate(&e1));
  float best[2];
  for (int v = 0; v < 2; ++v) {
    s->recon_variant = v;
    const auto step = [&] {
      sg.reconstruct(sg.fused());
      for (int k = 1; k < 3; ++k) sg.reconstruct();
    };
    step();  // warm-up
    best[v] = 1e30f;
    for (int k = 0; k < 3; ++k) {
      AFAR_CUDA(cudaEventRecord(e0, s->stream));
      step();
      AFAR_CUDA(cudaEventRecord(e1, s->stream));
      AFAR_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      AFAR_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      best[v] = std::min(best[v], ms / 3.f);
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  AFAR_CUDA(cudaMemcpyAsync(&s->ctl->dt_bits, &kDtArmed, sizeof(kDtArmed), cudaMemcpyHostToDevice, s->stream));
  AFAR_CUDA(cudaGetLastError());
  if ((st = check_device_error(s))) return st;
  s->recon_variant = best[1] < best[0] ? 1 : 0;
  s->tune_ms[0] = best[0];
  s->tune_ms[1] = best[1];
  std::lock_guard<std::mutex> lock(mu);
  cache[key] = s->recon_variant;
  return AFAR_OK;
}

extern "C" afar_status afar_set_tuning(afar_solver* s, int reconVariant) {
  if (!s || reconVariant < -1 || reconVariant > 1) return (set_error("afar_set_tuning: variant -1, 0 or 1"), AFAR_ERR_ARGUMENT);
  s->recon_request = reconVariant;
  if (!s->have_stencil || s->policy != AFAR_POLICY_MIXED) return AFAR_OK;
  AFAR_CUDA(cudaSetDevice(s->device));
  afar_status st = tune_reconstruct(s);
  if (st) return st;
  destroy_graphs(s);  // the next step captures the launches of the variant
  return AFAR_OK;
}

extern "C" afar_status afar_get_tuning(afar_solver* s, int* reconVariant, float* msTile, float* msRegister) {
  if (!s || !reconVariant) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  *reconVariant = s->recon_variant;
  if (msTile) *msTile = s->tune_ms[0];
  if (msRegister) *msRegister = s->tune_ms[1];
  return AFAR_OK;
}

extern "C" afar_status afar_setDeviceFieldData(afar_solver* s, const afar_fieldPointer* h, int cellsNum, int facesNum,
                                               int totalBoundaryFacesNum) {
  if (!s || !h || !h->CELL || !h->FACE || !h->cellVolume || !h->FD || !h->cFD || cellsNum <= 0 || facesNum < 0 ||
      totalBoundaryFacesNum < 0) {
    set_error("afar_setDeviceFieldData: null array or bad size");
    return AFAR_ERR_ARGUMENT;
  }
  if (s->have_fields) {
    set_error("afar_setDeviceFieldData: already called on this solver");
    return AFAR_ERR_STATE;
  }
  AFAR_CUDA(cudaSetDevice(s->device));
  s->Nc = cellsNum;
  s->Nf = facesNum;
  s->Nb = totalBoundaryFacesNum;
  s->ldc = (cellsNum + 31) / 32 * 32;
  const size_t Nc = cellsNum, Nf = facesNum, Nb = totalBoundaryFacesNum;
  const size_t g = s->policy == AFAR_POLICY_MIXED ? sizeof(V4<float>) : sizeof(V4<double>);
  const size_t l = s->policy == AFAR_POLICY_FP64 ? sizeof(V4<double>) : sizeof(V4<float>);
  const bool mixed = s->policy == AFAR_POLICY_MIXED;
  int* perm = nullptr;
  afar_status st;
  if ((st = alloc_all(s, [&]() -> afar_status {
         afar_status st;
         if ((st = dalloc_t(s, &s->cellC, Nc + Nb))) return st;
         if ((st = dalloc_t(s, &s->faceRaw, Nf + Nb))) return st;
         if (mixed) {
           if ((st = dalloc_t(s, &s->vinvf, Nc))) return st;
           // (the flux of a fused solver's rare separate kernels too, see afar_setDeviceFieldDataStencil)
           if ((st = dalloc(s, &s->xfer, std::max({(sizeof(V4<double>) + 2) * (Nc + Nb), sizeof(V4<float>) * (Nf + Nb),
                                                   order_scratch(cellsNum)}))))
             return st;
           if ((st = dalloc_t(s, &perm, Nc))) return st;
           for (void*& w : s->Wb)
             if ((st = dalloc(s, &w, sizeof(V4<float>) * (Nc + Nb)))) return st;
         } else {
           if ((st = dalloc_t(s, &s->vol, Nc))) return st;
           if ((st = dalloc_t(s, &s->vinv, Nc))) return st;
           if ((st = dalloc(s, &s->flux, g * (Nf + Nb)))) return st;
           if ((st = dalloc_t(s, &s->dtg, Nf))) return st;
         }
         if ((st = dalloc_t(s, &s->U, Nc))) return st;
         if ((st = dalloc_t(s, &s->U0, Nc))) return st;
         if ((st = dalloc_t(s, &s->si, 2 * (Nc + Nb)))) return st;
         if ((st = dalloc_t(s, &s->ctl, 1))) return st;
         if ((st = dalloc_t(s, &s->dt_bits, 1))) return st;
         if ((st = dalloc_t(s, &s->counters, 4))) return st;
         if ((st = dalloc(s, &s->W, w_size(s->policy) * (Nc + Nb)))) return st;
         // intermediates
         if ((st = dalloc(s, &s->grad, g * 2 * Nc))) return st;
         if ((st = dalloc(s, &s->lim, l * Nc))) return st;
         if ((st = dalloc(s, &s->fv, g * 2 * Nf))) return st;
         return dalloc_t(s, &s->bn, Nb);
       })))
    return st;
  // mixed: the caller's centres and volumes go to the state's buffers first, which put_state fills below
  V2<double>* const centres = mixed ? static_cast<V2<double>*>(s->Wb[0]) : s->cellC;
  static_assert(sizeof(V2<double>) == sizeof(V4<float>), "a centre in a state's place");
  AFAR_CUDA(cudaMemcpyAsync(centres, h->CELL, sizeof(V2<double>) * (Nc + Nb), cudaMemcpyHostToDevice, s->stream));
  AFAR_CUDA(cudaMemcpyAsync(s->faceRaw, h->FACE, sizeof(FaceRaw) * (Nf + Nb), cudaMemcpyHostToDevice, s->stream));
  double* const vol = mixed ? reinterpret_cast<double*>(s->U0) : s->vol;
  AFAR_CUDA(cudaMemcpyAsync(vol, h->cellVolume, sizeof(double) * Nc, cudaMemcpyHostToDevice, s->stream));
  if (mixed) {
    // Cells along a Hilbert curve: a tile of consecutive cells is then a compact patch of the mesh,
    // whose stencils and faces reach few cells outside it, whatever order the caller numbers in
    // (reverse Cuthill-McKee fronts are strips: 128 cells reach ~620 others, a Hilbert patch ~96).
    // Each cell keeps its own order of stencil members and faces, so results do not change by a bit.
    // Step, 2.0M triangles in RCM order: the reconstruct 0.60 -> 0.51 ms a step, the step 1.20 -> 1.10;
    // 4.0M quads and triangles, whose fronts are compact already: 2.19 -> 2.22.
    hilbert_order(cellsNum, centres, perm, s->xfer, s->stream);
    s->order.perm = perm;
    k_gather<<<grid_for(Nc + Nb, 256), 256, 0, s->stream>>>((int)Nc, (int)(Nc + Nb), centres, s->cellC, s->order);
  }
  k_reciprocal<<<grid_for(Nc, 256), 256, 0, s->stream>>>((int)Nc, vol, s->vinv, s->vinvf, s->order);
  AFAR_CUDA(cudaMemsetAsync(s->si, 0, 2 * (Nc + Nb), s->stream));
  if ((st = put_state(s, reinterpret_cast<const afar_basicFieldData*>(h->FD),
                      reinterpret_cast<const afar_conservedFieldData*>(h->cFD),
                      reinterpret_cast<const afar_conservedFieldData*>(h->cFD))))
    return st;
  k_init_ctl<<<1, 32, 0, s->stream>>>(s->ctl);
  AFAR_CUDA(cudaMemsetAsync(s->fv, 0, g * 2 * Nf, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  AFAR_CUDA(cudaGetLastError());
  s->have_fields = true;
  return AFAR_OK;
}

extern "C" afar_status afar_set_rbf_basis64(afar_solver* s, const double* rbf, size_t count) {
  if (!s || (!rbf && count)) {
    set_error("afar_set_rbf_basis64: null argument");
    return AFAR_ERR_ARGUMENT;
  }
  s->head_pending = false;
  s->rbf64.assign(rbf, rbf + count);
  return AFAR_OK;
}

extern "C" afar_status afar_setDeviceFieldDataStencil(afar_solver* s, const afar_fieldPointer* h, int cellsNum,
                                                      int facesNum, int patchesNum, int totalBoundaryFacesNum,
                                                      int maxStencilSize, int maxCompactStencilSize,
                                                      int maxLocalBlockStencilSize,
                                                      int maxCompactLocalBlockStencilSize) {
  NvtxRange nvtx("afar_setDeviceFieldDataStencil");
  if (!s || !h) {
    set_error("afar_setDeviceFieldDataStencil: null argument");
    return AFAR_ERR_ARGUMENT;
  }
  if (!s->have_fields) {
    set_error("afar_setDeviceFieldDataStencil: call afar_setDeviceFieldData first");
    return AFAR_ERR_STATE;
  }
  if (s->have_stencil) {
    set_error("afar_setDeviceFieldDataStencil: already called on this solver");
    return AFAR_ERR_STATE;
  }
  if (cellsNum != s->Nc || facesNum != s->Nf || totalBoundaryFacesNum != s->Nb) {
    set_error("afar_setDeviceFieldDataStencil: sizes differ from afar_setDeviceFieldData");
    return AFAR_ERR_ARGUMENT;
  }
  if (maxStencilSize < 1 || maxStencilSize > AFAR_MAX_VALID_STENCIL_SIZE || maxCompactStencilSize < 1 ||
      maxCompactStencilSize > maxStencilSize || maxCompactStencilSize > kMaxFaces ||
      maxLocalBlockStencilSize < AFAR_BLOCKDIM ||
      maxCompactLocalBlockStencilSize < AFAR_BLOCKDIM || patchesNum < 0) {
    set_error("afar_setDeviceFieldDataStencil: stencil sizes out of range (maxS %d, maxM %d, maxLB %d)",
              maxStencilSize, maxCompactStencilSize, maxLocalBlockStencilSize);
    return AFAR_ERR_LIMIT;
  }
  if (!h->neighbour && facesNum > 0) return (set_error("neighbour is null"), AFAR_ERR_ARGUMENT);
  if (!h->stencilSize || !h->compactStencilSize || !h->localStencil || !h->cellFaces || !h->RBFbasis ||
      (totalBoundaryFacesNum > 0 && (!h->boundaryFaceNeiLabel || !h->boundaryFacesType)) ||
      (maxLocalBlockStencilSize > AFAR_BLOCKDIM && !h->extendStencil)) {
    set_error("afar_setDeviceFieldDataStencil: null stencil array");
    return AFAR_ERR_ARGUMENT;
  }
  AFAR_CUDA(cudaSetDevice(s->device));
  const int Nc = s->Nc, Nf = s->Nf, Nb = s->Nb;
  // host-side validation of everything a kernel indexes with: the cells on all cores, the first bad
  // one again to report it
  auto check_cell = [&](int c, bool* paired, long long* slots) -> afar_status {
    if (h->stencilSize[c] > maxStencilSize || h->compactStencilSize[c] > maxCompactStencilSize ||
        h->compactStencilSize[c] > h->stencilSize[c]) {
      set_error("cell %d: stencil sizes %d/%d exceed the declared maxima", c, h->stencilSize[c], h->compactStencilSize[c]);
      return AFAR_ERR_ARGUMENT;
    }
    int across[kMaxFaces] = {-1, -1, -1, -1};  // the cell across each internal face: the slot's stencil member
    for (int i = 0; i < h->compactStencilSize[c]; ++i) {
      const int fid = h->cellFaces[(size_t)maxCompactStencilSize * c + i];
      const int f = (fid < 0 ? -fid : fid) - 1;
      if (fid == 0 || f >= Nf + Nb || (f >= Nf && fid < 0)) {
        set_error("cell %d: cellFaces entry %d out of range", c, fid);
        return AFAR_ERR_ARGUMENT;
      }
      if (f < Nf) {  // this cell's side of the face, once
        ++*slots;
        if (h->neighbour[2 * (size_t)f + (fid < 0)] != c) *paired = false;
        for (int k = 0; k < i; ++k)
          if (h->cellFaces[(size_t)maxCompactStencilSize * c + k] == fid) *paired = false;
        across[i] = h->neighbour[2 * (size_t)f + (fid > 0)];
      }
    }
    const int blk = c / AFAR_BLOCKDIM;
    for (int i = 0; i < h->stencilSize[c]; ++i) {
      const int loc = h->localStencil[(size_t)maxStencilSize * c + i];
      if (loc >= maxLocalBlockStencilSize) {
        set_error("cell %d: localStencil entry %d out of range", c, loc);
        return AFAR_ERR_ARGUMENT;
      }
      const int g = loc < AFAR_BLOCKDIM ? blk * AFAR_BLOCKDIM + loc
                                        : h->extendStencil[(size_t)(maxLocalBlockStencilSize - AFAR_BLOCKDIM) * blk + (loc - AFAR_BLOCKDIM)];
      if (g < 0 || g >= Nc + Nb || (loc < AFAR_BLOCKDIM && g >= Nc)) {
        set_error("cell %d: stencil member %d out of range", c, g);
        return AFAR_ERR_ARGUMENT;
      }
      if (i < kMaxFaces && across[i] >= 0 && across[i] != g) *paired = false;
    }
    return AFAR_OK;
  };
  bool paired = true;  // every internal face is in the lists of both its cells, with the right sign and stencil member
  {
    std::mutex mu;
    int bad = Nc;
    long long slots = 0;
    parallel_ranges(Nc, 4096, [&](long long a, long long b) {
      bool p = true;
      long long n = 0;
      int c = (int)a;
      while (c < (int)b && check_cell(c, &p, &n) == AFAR_OK) ++c;
      std::lock_guard<std::mutex> lock(mu);
      if (c < (int)b) bad = std::min(bad, c);
      paired = paired && p;
      slots += n;
    });
    if (bad < Nc) return check_cell(bad, &paired, &slots);
    paired = paired && slots == 2ll * Nf;
  }
  for (int f = 0; f < Nf; ++f) {
    const int o = h->neighbour[2 * f], n = h->neighbour[2 * f + 1];
    if (o < 0 || o >= Nc || n < 0 || n >= Nc) {
      set_error("face %d: owner/neighbour (%d, %d) out of range", f, o, n);
      return AFAR_ERR_ARGUMENT;
    }
  }
  for (int b = 0; b < Nb; ++b) {
    if (h->boundaryFaceNeiLabel[b] < 0 || h->boundaryFaceNeiLabel[b] >= Nc) {
      set_error("boundary face %d: owner out of range", b);
      return AFAR_ERR_ARGUMENT;
    }
    if (h->boundaryFacesType[b] > AFAR_BC_FIXED_INITIAL) {
      set_error("boundary face %d: unknown boundary label %d (cudaEulerBCs 0-5, or 6)", b, h->boundaryFacesType[b]);
      return AFAR_ERR_ARGUMENT;
    }
  }
  s->patches = patchesNum;
  s->maxS = maxStencilSize;
  s->maxM = maxCompactStencilSize;
  s->maxLB = maxLocalBlockStencilSize;
  s->maxCLB = maxCompactLocalBlockStencilSize;
  const size_t ldc = s->ldc;
  const size_t wS = s->policy == AFAR_POLICY_FP64 ? 8 : 4, wG = s->policy == AFAR_POLICY_MIXED ? 4 : 8;
  const int ntile = (Nc + kTile - 1) / kTile;
  const size_t ntail = grid_for(Nc, tail_cells(s));
  int* fperm = nullptr;
  afar_status st;
  if ((st = alloc_all(s, [&]() -> afar_status {
         afar_status st;
         if ((st = dalloc_t(s, &s->on, (size_t)Nf))) return st;
         if ((st = dalloc_t(s, &s->btype, (size_t)Nb))) return st;
         if ((st = dalloc_t(s, &s->nS, (size_t)Nc))) return st;
         if ((st = dalloc_t(s, &s->nM, (size_t)Nc))) return st;
         if ((st = dalloc_t(s, &s->sten, (size_t)s->maxS * ldc))) return st;
         if ((st = dalloc_t(s, &s->cf, (size_t)s->maxM * ldc))) return st;
         if ((st = dalloc_t(s, &s->tileS, (size_t)ntile))) return st;
         if ((st = dalloc(s, &s->fd, 4 * wG * (size_t)Nf))) return st;
         if ((st = dalloc(s, &s->fs, 4 * wG * (size_t)(Nf + Nb)))) return st;
         if ((st = dalloc(s, &s->lsm, 2 * wS * (size_t)s->maxM * ldc))) return st;
         if ((st = dalloc(s, &s->sg, 2 * wG * (size_t)s->maxM * ldc))) return st;
         if ((st = dalloc(s, &s->sr, 2 * wS * (size_t)s->maxM * ldc))) return st;
         if ((st = dalloc(s, &s->wts, wS * (size_t)s->maxM * (s->maxS + 1) * ldc))) return st;
         if (s->policy == AFAR_POLICY_MIXED) {
           if ((st = dalloc_t(s, &s->dtgf, (size_t)Nf))) return st;
           if ((st = dalloc_t(s, &s->tmaps, 1))) return st;
           if ((st = dalloc_t(s, &fperm, (size_t)Nf))) return st;
           if ((st = dalloc_t(s, &s->tail, ntail))) return st;
           if ((st = dalloc_t(s, &s->thalo, ntail * kTailHalo))) return st;
           if ((st = dalloc_t(s, &s->thcode, ntail * 4 * kTailHalo))) return st;
           if ((st = dalloc_t(s, &s->thsg, ntail * 4 * kTailHalo))) return st;
           if ((st = dalloc_t(s, &s->textra, ntail * kTailExtra))) return st;
           if ((st = dalloc_t(s, &s->tlf, (size_t)s->maxM * ldc))) return st;
           if ((st = dalloc_t(s, &s->tlist, ntail * kTailList))) return st;
           if ((st = dalloc_t(s, &s->wflag, (size_t)ntile * 4))) return st;
         }
         return AFAR_OK;
       })))
    return st;
  // one scratch buffer for the set-up's steps, which follow one another on the stream
  const size_t nblk = (Nc + AFAR_BLOCKDIM - 1) / AFAR_BLOCKDIM;
  const size_t next = (size_t)(s->maxLB - AFAR_BLOCKDIM) * nblk;
  const size_t n_dls = (sizeof(uint16_t) * (size_t)s->maxS * Nc + 15) / 16 * 16, n_dext = (sizeof(int) * next + 15) / 16 * 16;
  const size_t nrbf = 2 * (size_t)(s->maxS + 1) * Nf;
  const size_t n_lists = n_dls + n_dext + (sizeof(int) * (size_t)s->maxM * Nc + 15) / 16 * 16;
  int tail_limits[2] = {0, 1};  // the most faces of a tile; a tile past the limits
  Scratch scratch;
  AFAR_CUDA(cudaMalloc(&scratch.p, std::max({n_lists + 12 * (size_t)Nf + 6 * (size_t)Nc, nrbf * wS,
                                             2 * sizeof(V4<double>) * (size_t)(Nf + Nb + 1)})));
  AFAR_CUDA(cudaMemsetAsync(s->sten, 0, sizeof(int) * s->maxS * ldc, s->stream));
  AFAR_CUDA(cudaMemsetAsync(s->cf, 0, sizeof(int) * s->maxM * ldc, s->stream));
  if (Nb) {
    AFAR_CUDA(cudaMemcpyAsync(s->btype, h->boundaryFacesType, Nb, cudaMemcpyHostToDevice, s->stream));
  }
  {
    char* at = static_cast<char*>(scratch.p);
    uint16_t* dls = reinterpret_cast<uint16_t*>(at);
    int* dext = reinterpret_cast<int*>(at + n_dls);
    int* dcf = reinterpret_cast<int*>(at + n_dls + n_dext);
    int* inv = reinterpret_cast<int*>(at + n_lists + sizeof(int2) * (size_t)Nf);  // then finv, for the set-up alone
    uint8_t* counts = reinterpret_cast<uint8_t*>(inv + (size_t)Nc + Nf);
    AFAR_CUDA(cudaMemcpyAsync(counts, h->stencilSize, Nc, cudaMemcpyHostToDevice, s->stream));
    AFAR_CUDA(cudaMemcpyAsync(counts + Nc, h->compactStencilSize, Nc, cudaMemcpyHostToDevice, s->stream));
    if (s->order.perm) s->order.inv = inv;
    k_setup_counts<<<ntile, kTile, 0, s->stream>>>(Nc, counts, counts + Nc, s->nS, s->nM, s->tileS,
                                                   s->order.perm ? inv : nullptr, s->order);
    AFAR_CUDA(cudaMemcpyAsync(dls, h->localStencil, sizeof(uint16_t) * (size_t)s->maxS * Nc, cudaMemcpyHostToDevice, s->stream));
    if (next) AFAR_CUDA(cudaMemcpyAsync(dext, h->extendStencil, sizeof(int) * next, cudaMemcpyHostToDevice, s->stream));
    AFAR_CUDA(cudaMemcpyAsync(dcf, h->cellFaces, sizeof(int) * (size_t)s->maxM * Nc, cudaMemcpyHostToDevice, s->stream));
    int2* raw = s->order.perm ? reinterpret_cast<int2*>(at + n_lists) : s->on;
    if (Nf) AFAR_CUDA(cudaMemcpyAsync(raw, h->neighbour, sizeof(int2) * Nf, cudaMemcpyHostToDevice, s->stream));
    if (s->order.perm && Nf) {
      if (paired) {  // (faces that are not keep the caller's order)
        int* start = static_cast<int*>(s->xfer);
        int* finv = inv + Nc;
        for (int pass = 0; pass < 2; ++pass) {
          k_face_order<<<grid_for(Nc, 256), 256, 0, s->stream>>>(Nc, Nf, s->maxM, s->nM, dcf,
                                                                 reinterpret_cast<const int*>(raw), s->order, start,
                                                                 fperm, finv, pass);
          if (pass == 0) device_scan(Nc, start, start + Nc, s->stream);
        }
        s->order.fperm = fperm;
        s->order.finv = finv;
      }
      k_setup_owners<<<grid_for(Nf, 256), 256, 0, s->stream>>>(Nf, raw, s->on, s->order);
    }
    k_setup_lists<<<grid_for(Nc, kCellBlock), kCellBlock, 0, s->stream>>>(Nc, Nf, s->ldc, s->maxS, s->maxM, s->maxLB,
                                                                           s->nS, s->nM, dls, dext, dcf, s->sten, s->cf,
                                                                           s->order);
    s->order.inv = s->order.finv = nullptr;
    if (s->policy == AFAR_POLICY_MIXED) {
      AFAR_CUDA(cudaMemsetAsync(s->wflag, 0, sizeof(unsigned) * (size_t)ntile * 4, s->stream));
    }
    AFAR_CUDA(cudaGetLastError());
  }
  switch (s->policy) {
    case AFAR_POLICY_REF: st = setup_operators<PolicyRef>(s, h, scratch.p); break;
    case AFAR_POLICY_FP64: st = setup_operators<PolicyFP64>(s, h, scratch.p); break;
    default: st = setup_operators<PolicyMixed>(s, h, scratch.p); break;
  }
  if (st) return st;
  if (s->policy == AFAR_POLICY_MIXED && paired && Nf > 0 && s->maxM >= 3) {
    int* start = static_cast<int*>(s->xfer);  // (of k_face_order)
    int* limits = start + Nc;
    StageArgs<PolicyMixed> a = make_args<PolicyMixed>(s);
    AFAR_CUDA(cudaMemsetAsync(limits, 0, 2 * sizeof(int), s->stream));
    k_tail_tiles<<<(int)ntail, 128, 0, s->stream>>>(a, start, s->tail, s->thalo, s->thcode, s->thsg, s->textra, s->tlf,
                                                    limits);
    k_tail_lists<<<(int)ntail, 128, 0, s->stream>>>(a, s->tail, s->thalo, s->tlist);
    AFAR_CUDA(cudaMemcpyAsync(tail_limits, limits, 2 * sizeof(int), cudaMemcpyDeviceToHost, s->stream));
  }
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  // meshes whose tiles are past the limits of the fused stage tail, or whose faces are not in the lists of
  // both their cells, or of cells with one or two faces, keep the separate kernels
  s->bvd_pending = -1;
  s->fused = tail_limits[1] == 0 && tail_smem(tail_limits[0], tail_cells(s)).bytes <= kMaxDynamicSmem - 2048;
  s->tail_faces = tail_limits[0];
  // The flux of the separate kernels: a solver that runs the fused stage has it in the transfer buffer, which
  // nothing else uses between a flux and its update (afar_stage_debug; a batch with block sizes of its own).
  if (s->policy == AFAR_POLICY_MIXED) {
    s->flux = s->xfer;
    if (!s->fused && (st = dalloc(s, &s->flux, sizeof(V4<float>) * (size_t)(Nf + Nb)))) return st;
  }
  if (s->fused) {
    if ((st = raise_smem_limit(k_tail<3>, s->device, tail_smem(s->tail_faces, tail_cells(s)).bytes))) return st;
    if ((st = raise_smem_limit(k_tail<4>, s->device, tail_smem(s->tail_faces, tail_cells(s)).bytes))) return st;
  }
  if (s->policy == AFAR_POLICY_MIXED && (st = build_tile_maps(s))) return st;
  if (s->policy == AFAR_POLICY_MIXED && (st = tune_reconstruct(s))) return st;
  s->have_stencil = true;
  return AFAR_OK;
}

// The gas constants, which the graphs hold: other ones drop the graphs.
static void set_gas(afar_solver* s, double R, double Cv) {
  if (s->R == R && s->Cv == Cv) return;
  s->R = R;
  s->Cv = Cv;
  destroy_graphs(s);
}
// Captures a graph that the solver does not have yet.
static afar_status ensure_graph(afar_solver* s, int which) {
  const cudaGraphExec_t g = which == kGraphStep ? s->graph : which == kGraphHead ? s->graph_head : s->graph_tail;
  return g ? AFAR_OK : capture_graph(s, which);
}

extern "C" afar_status afar_adjustTimeStep(afar_solver* s, int facesNum, double R, double Cv, double CFL, double* dt) {
  NvtxRange nvtx("afar_adjustTimeStep");
  afar_status st = check_ready(s);
  if (st) return st;
  if (!dt || facesNum != s->Nf || !(R > 0.0) || !(Cv > 0.0) || !(CFL > 0.0)) {
    set_error("afar_adjustTimeStep: bad argument");
    return AFAR_ERR_ARGUMENT;
  }
  // Outside a batch the Courant step comes from the head of the coming step -- stage 1 up to its
  // flux, whose fused reduction is the same Courant minimum over the internal faces (the ref
  // policy's head runs the reference-shaped Courant kernel itself) -- so no separate pass runs and
  // the afar_GPUevolve that follows runs only the tail of the step.
  if (!s->batch && s->Nf > 0) {
    set_gas(s, R, Cv);
    if ((st = ensure_graph(s, kGraphHead)) || (st = ensure_graph(s, kGraphTail))) return st;
    {
      k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, 0.0, CFL, 0.0);
      AFAR_CUDA(cudaGraphLaunch(s->graph_head, s->stream));
      s->bvd_pending = fused_step(s) ? 0 : -1;
      StepCtl c;
      AFAR_CUDA(cudaMemcpyAsync(&c, s->ctl, sizeof(c), cudaMemcpyDeviceToHost, s->stream));
      AFAR_CUDA(cudaStreamSynchronize(s->stream));
      AFAR_CUDA(cudaGetLastError());
      // the minimum is armed again at once, as at the end of a step: whichever step follows starts anew (the
      // tail has its step size from the caller)
      AFAR_CUDA(cudaMemcpyAsync(&s->ctl->dt_bits, &kDtArmed, sizeof(kDtArmed), cudaMemcpyHostToDevice, s->stream));
      if (c.err) {  // a bounded device wait gave up, in this head or in the step before it
        AFAR_CUDA(cudaMemsetAsync(&s->ctl->err, 0, sizeof(c.err), s->stream));
        AFAR_CUDA(cudaStreamSynchronize(s->stream));
        set_error("a device-side wait for a bulk copy timed out (error word %u); the state is not valid", c.err);
        return AFAR_ERR_CUDA;
      }
      std::memcpy(dt, &c.dt_bits, sizeof(double));
      s->head_pending = true;
      return AFAR_OK;
    }
  }
  AFAR_CUDA(cudaMemcpyAsync(s->dt_bits, &kDtArmed, sizeof(kDtArmed), cudaMemcpyHostToDevice, s->stream));
  const int gf = grid_for(s->Nf, kFaceBlock);
  if (s->Nf > 0) {
    switch (s->policy) {
      case AFAR_POLICY_REF: {
        StageArgs<PolicyRef> a = make_args<PolicyRef>(s);
        a.R = R;
        a.Cv = Cv;
        a.gR = (R / Cv + 1.0) * R;
        k_delta_t<PolicyRef><<<gf, kFaceBlock, 0, s->stream>>>(a, CFL, s->dt_bits, nullptr);
        break;
      }
      case AFAR_POLICY_FP64: {
        StageArgs<PolicyFP64> a = make_args<PolicyFP64>(s);
        a.gR = (R / Cv + 1.0) * R;
        k_delta_t<PolicyFP64><<<gf, kFaceBlock, 0, s->stream>>>(a, CFL, s->dt_bits, nullptr);
        break;
      }
      default: {  // the mixed policy's FP32 Courant estimate, as in its fused stage-1 flux
        StageArgs<PolicyMixed> a = make_args<PolicyMixed>(s);
        a.gRf = (float)((R / Cv + 1.0) * R);
        k_delta_t_mixed<<<gf, kFaceBlock, 0, s->stream>>>(a, (float)CFL, s->dt_bits);
        break;
      }
    }
  }
  unsigned long long bits = 0;
  AFAR_CUDA(cudaMemcpyAsync(&bits, s->dt_bits, sizeof(bits), cudaMemcpyDeviceToHost, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  AFAR_CUDA(cudaGetLastError());
  double v;
  std::memcpy(&v, &bits, sizeof(v));
  *dt = v;
  return AFAR_OK;
}

static afar_status run_impl(afar_solver* s, int nSteps, double dt, double CFL, double tEnd, bool wait) {
  NvtxRange nvtx("afar_run");
  afar_status st = check_ready(s);
  if (st || (st = check_not_batched(s))) return st;
  if (nSteps < 0 || (!(dt > 0.0) && !(CFL > 0.0))) {
    set_error("afar_run: nSteps must be >= 0 and either deltaT > 0 or CFL > 0");
    return AFAR_ERR_ARGUMENT;
  }
  if (!(s->R > 0.0)) return (set_error("call afar_set_gas (or afar_GPUevolve) first"), AFAR_ERR_STATE);
  if ((st = ensure_graph(s, kGraphStep))) return st;
  k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, dt > 0.0 ? dt : 0.0, CFL, tEnd);
  for (int i = 0; i < nSteps; ++i) AFAR_CUDA(cudaGraphLaunch(s->graph, s->stream));
  if (nSteps > 0) s->bvd_pending = fused_step(s) ? 2 : -1;
  AFAR_CUDA(cudaGetLastError());
  if (wait) return check_device_error(s);
  return AFAR_OK;
}

extern "C" afar_status afar_GPUevolve(afar_solver* s, double R, double Cv, double deltaT, int cellsNum, int facesNum,
                                      int totalBoundaryFacesNum, int maxStencilSize, int maxCompactStencilSize,
                                      int maxLocalBlockStencilSize, int maxCompactLocalBlockStencilSize) {
  NvtxRange nvtx("afar_GPUevolve");
  const bool head_done = s && s->head_pending;  // read before check_ready clears it
  afar_status st = check_ready(s);
  if (st) return st;
  if (cellsNum != s->Nc || facesNum != s->Nf || totalBoundaryFacesNum != s->Nb || maxStencilSize != s->maxS ||
      maxCompactStencilSize != s->maxM) {
    set_error("afar_GPUevolve: sizes differ from the uploaded fields");
    return AFAR_ERR_ARGUMENT;
  }
  (void)maxLocalBlockStencilSize;
  (void)maxCompactLocalBlockStencilSize;
  if (!(deltaT > 0.0) || !(R > 0.0) || !(Cv > 0.0)) {
    set_error("afar_GPUevolve: deltaT, R and Cv must be positive");
    return AFAR_ERR_ARGUMENT;
  }
  if (head_done && s->graph_tail && s->R == R && s->Cv == Cv) {
    // afar_adjustTimeStep ran this step's head on the current state: the tail with the caller's
    // step size completes it, the same kernels as the whole-step graph.  Enqueued, not waited
    // for: a device-side error of the step surfaces at the next call that waits.
    k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, deltaT, 1.0, 0.0);
    AFAR_CUDA(cudaGraphLaunch(s->graph_tail, s->stream));
    s->bvd_pending = fused_step(s) ? 2 : -1;
    AFAR_CUDA(cudaGetLastError());
    return AFAR_OK;
  }
  set_gas(s, R, Cv);
  return run_impl(s, 1, deltaT, 1.0, 0.0, true);
}

extern "C" afar_status afar_set_gas(afar_solver* s, double R, double Cv) {
  if (!s || !(R > 0.0) || !(Cv > 0.0)) {
    set_error("afar_set_gas: bad argument");
    return AFAR_ERR_ARGUMENT;
  }
  s->head_pending = false;
  set_gas(s, R, Cv);
  afar_status st = AFAR_OK;
  for (int g = kGraphStep; g <= kGraphTail && s->have_stencil && !st; ++g) st = ensure_graph(s, g);
  return st;
}

// The gas constants of a solver that is only ever stepped in a batch: no graphs of its own.
afar_status afar::set_gas_batched(afar_solver* s, double R, double Cv) {
  if (!s || !(R > 0.0) || !(Cv > 0.0)) {
    set_error("set_gas_batched: bad argument");
    return AFAR_ERR_ARGUMENT;
  }
  set_gas(s, R, Cv);
  return AFAR_OK;
}

extern "C" afar_status afar_run(afar_solver* s, int nSteps, double deltaT, double CFL, double tEnd) {
  return run_impl(s, nSteps, deltaT, CFL, tEnd, true);
}

extern "C" afar_status afar_run_async(afar_solver* s, int nSteps, double deltaT, double CFL, double tEnd) {
  return run_impl(s, nSteps, deltaT, CFL, tEnd, false);
}

extern "C" afar_status afar_run_timed(afar_solver* s, int nSteps, double dt, double CFL, double tEnd, float* ms) {
  afar_status st = check_ready(s);
  if (st || (st = check_not_batched(s))) return st;
  if (!ms) return (set_error("null output"), AFAR_ERR_ARGUMENT);
  if (!(s->R > 0.0)) return (set_error("call afar_set_gas (or afar_GPUevolve) first"), AFAR_ERR_STATE);
  if ((st = ensure_graph(s, kGraphStep))) return st;
  cudaEvent_t e0, e1;
  AFAR_CUDA(cudaEventCreate(&e0));
  AFAR_CUDA(cudaEventCreate(&e1));
  k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, dt > 0.0 ? dt : 0.0, CFL, tEnd);
  AFAR_CUDA(cudaEventRecord(e0, s->stream));
  for (int i = 0; i < nSteps; ++i) AFAR_CUDA(cudaGraphLaunch(s->graph, s->stream));
  if (nSteps > 0) s->bvd_pending = fused_step(s) ? 2 : -1;
  AFAR_CUDA(cudaEventRecord(e1, s->stream));
  AFAR_CUDA(cudaEventSynchronize(e1));
  AFAR_CUDA(cudaEventElapsedTime(ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  AFAR_CUDA(cudaGetLastError());
  return check_device_error(s);
}

extern "C" afar_status afar_profile_step(afar_solver* s, double dt, double CFL, float ms[5]) {
  afar_status st = check_ready(s);
  if (st || (st = check_not_batched(s))) return st;
  if (!ms) return (set_error("null output"), AFAR_ERR_ARGUMENT);
  if (!(s->R > 0.0)) return (set_error("call afar_set_gas (or afar_GPUevolve) first"), AFAR_ERR_STATE);
  cudaEvent_t ev[32];
  for (int i = 0; i < 32; ++i) AFAR_CUDA(cudaEventCreate(&ev[i]));
  k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, dt > 0.0 ? dt : 0.0, CFL, 0.0);
  int n = 0;
  int kind[32];
  auto mark = [&](int k) {
    cudaEventRecord(ev[n], s->stream);
    kind[n++] = k;
  };
  auto body = [&](auto tag) -> afar_status {
    using P = decltype(tag);
    Stage<P> sg;
    afar_status r = make_stage<P>(s, false, &sg);
    if (r) return r;
    mark(-1);
    for (int k = 0; k < 3; ++k) {
      if (sg.fused()) {
        sg.at(k).reconstruct(k == 0);
        mark(0);
        sg.at(k).tail(k);
        mark(3);
        s->bvd_pending = k;
        continue;
      }
      sg.reconstruct();
      mark(0);
      sg.bvd();
      mark(1);
      sg.flux(k == 0);
      mark(2);
      sg.update(k);
      mark(3);
    }
    if (!sg.fused()) {
      k_finish_step<<<1, 32, 0, s->stream>>>(s->ctl);
      mark(4);
    }
    return AFAR_OK;
  };
  switch (s->policy) {
    case AFAR_POLICY_REF: st = body(PolicyRef{}); break;
    case AFAR_POLICY_FP64: st = body(PolicyFP64{}); break;
    default: st = body(PolicyMixed{}); break;
  }
  if (st) return st;
  AFAR_CUDA(cudaEventSynchronize(ev[n - 1]));
  for (int k = 0; k < 5; ++k) ms[k] = 0.f;
  for (int i = 1; i < n; ++i) {
    float t = 0.f;
    AFAR_CUDA(cudaEventElapsedTime(&t, ev[i - 1], ev[i]));
    ms[kind[i]] += t;
  }
  for (int i = 0; i < 32; ++i) cudaEventDestroy(ev[i]);
  AFAR_CUDA(cudaGetLastError());
  return check_device_error(s);
}

extern "C" afar_status afar_synchronize(afar_solver* s) {
  if (!s) return (set_error("null solver"), AFAR_ERR_ARGUMENT);
  AFAR_CUDA(cudaSetDevice(s->device));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  AFAR_CUDA(cudaGetLastError());
  return AFAR_OK;
}

extern "C" afar_status afar_get_stream(afar_solver* s, void** stream) {
  if (!s || !stream) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  *stream = (void*)s->stream;
  return AFAR_OK;
}

extern "C" afar_status afar_get_time(afar_solver* s, double* t, double* lastDt, long long* steps) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  AFAR_CUDA(cudaSetDevice(s->device));
  StepCtl c;
  AFAR_CUDA(cudaMemcpyAsync(&c, s->ctl, sizeof(c), cudaMemcpyDeviceToHost, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  if (t) *t = c.t;
  if (lastDt) *lastDt = c.last_dt;
  if (steps) *steps = c.steps;
  return AFAR_OK;
}

extern "C" afar_status afar_set_time(afar_solver* s, double t) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  s->head_pending = false;
  AFAR_CUDA(cudaSetDevice(s->device));
  AFAR_CUDA(cudaMemcpyAsync(&s->ctl->t, &t, sizeof(double), cudaMemcpyHostToDevice, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  return AFAR_OK;
}

extern "C" afar_status afar_stage_debug(afar_solver* s, int stage, double deltaT, afar_fieldPointer* out) {
  afar_status st = check_ready(s);
  if (st || (st = check_not_batched(s))) return st;
  if (stage < 0 || stage > 2 || !(deltaT > 0.0) || !out) {
    set_error("afar_stage_debug: stage must be 0..2, deltaT > 0, out non-null");
    return AFAR_ERR_ARGUMENT;
  }
  if (!(s->R > 0.0)) return (set_error("call afar_set_gas (or afar_GPUevolve) first"), AFAR_ERR_STATE);
  k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, deltaT, 1.0, 0.0);
  const size_t Nc = s->Nc, Nf = s->Nf, Nb = s->Nb;
  const bool mixed = s->policy == AFAR_POLICY_MIXED;
  const bool f64 = s->policy == AFAR_POLICY_FP64;
  auto run = [&](auto tag) -> afar_status {
    using P = decltype(tag);
    Stage<P> sg;
    afar_status r = AFAR_OK;
    if (!s->res_dbg && (r = dalloc_t(s, &s->res_dbg, Nc))) return r;
    if ((r = make_stage<P>(s, true, &sg))) return r;
    s->bvd_pending = -1;
    sg.reconstruct();
    sg.bvd();
    sg.flux(false);
    sg.update(stage);
    return AFAR_OK;
  };
  switch (s->policy) {
    case AFAR_POLICY_REF: st = run(PolicyRef{}); break;
    case AFAR_POLICY_FP64: st = run(PolicyFP64{}); break;
    default: st = run(PolicyMixed{}); break;
  }
  if (st) return st;
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  // copy out in the reference layout and the caller's order: `group` entries for each cell or face of
  // `perm` (the caller's place of the device's; empty: the caller's order), the rest in place
  auto get4 = [&](auto* dst, const auto* src, size_t n, const std::vector<int>& perm, size_t group) -> afar_status {
    using D = std::remove_pointer_t<decltype(dst)>;
    using S = std::remove_const_t<std::remove_pointer_t<decltype(src)>>;
    if (std::is_same<D, S>::value && perm.empty()) {
      AFAR_CUDA(cudaMemcpy(dst, src, n * sizeof(S), cudaMemcpyDeviceToHost));
      return AFAR_OK;
    }
    std::unique_ptr<S[]> t(new S[n]);
    AFAR_CUDA(cudaMemcpy(t.get(), src, n * sizeof(S), cudaMemcpyDeviceToHost));
    parallel_ranges((long long)n, 16384, [&](long long i0, long long i1) {
      using E = decltype(dst->x);
      for (size_t i = (size_t)i0; i < (size_t)i1; ++i) {
        const size_t g = i / group;
        dst[g < perm.size() ? (size_t)perm[g] * group + i % group : i] = D{(E)t[i].x, (E)t[i].y, (E)t[i].z, (E)t[i].w};
      }
    });
    return AFAR_OK;
  };
  auto get = [&](void* dst, const void* src, size_t n, const std::vector<int>& perm, size_t group) {
    V4<double>* const d = static_cast<V4<double>*>(dst);
    return mixed ? get4(d, static_cast<const V4<float>*>(src), n, perm, group)
                 : get4(d, static_cast<const V4<double>*>(src), n, perm, group);
  };
  std::vector<int> perm, fperm;
  if (s->order.perm) {
    perm.resize(Nc);
    AFAR_CUDA(cudaMemcpy(perm.data(), s->order.perm, sizeof(int) * Nc, cudaMemcpyDeviceToHost));
  }
  if (s->order.fperm) {
    fperm.resize(Nf);
    AFAR_CUDA(cudaMemcpy(fperm.data(), s->order.fperm, sizeof(int) * Nf, cudaMemcpyDeviceToHost));
  }
  if (out->faceFD && (st = get(out->faceFD, s->fv, 2 * Nf, fperm, 2))) return st;
  if (out->gradFD && (st = get(out->gradFD, s->grad, 2 * Nc, perm, 2))) return st;
  if (out->Flux && (st = get(out->Flux, s->flux, Nf + Nb, fperm, 1))) return st;
  if ((out->FD || out->cFD || out->shockIndicator) &&
      (st = get_state(s, out->FD, reinterpret_cast<afar_conservedFieldData*>(out->cFD), out->shockIndicator)))
    return st;
  if (out->Res && (st = get4(reinterpret_cast<V4<double>*>(out->Res), s->res_dbg, Nc, perm, 1))) return st;
  V4<float>* const lim = reinterpret_cast<V4<float>*>(out->limiter);
  if (lim && (st = f64 ? get4(lim, static_cast<const V4<double>*>(s->lim), Nc, perm, 1)
                       : get4(lim, static_cast<const V4<float>*>(s->lim), Nc, perm, 1)))
    return st;
  return AFAR_OK;
}

extern "C" afar_status afar_debug_limiter64(afar_solver* s, double* lim) {
  afar_status st = check_ready(s);
  if (st) return st;
  if (!lim) return (set_error("null output"), AFAR_ERR_ARGUMENT);
  if ((st = settle_bvd(s))) return st;
  const size_t Nc = s->Nc;
  if (s->policy == AFAR_POLICY_FP64) {
    AFAR_CUDA(cudaMemcpy(lim, s->lim, Nc * sizeof(V4<double>), cudaMemcpyDeviceToHost));
  } else if (s->policy == AFAR_POLICY_MIXED) {
    k_state_out<<<grid_for((long long)Nc, 256), 256, 0, s->stream>>>((int)Nc, (int)Nc, static_cast<const V4<float>*>(s->lim),
                                                                     static_cast<V4<double>*>(s->xfer), nullptr, nullptr, s->order);
    AFAR_CUDA(cudaGetLastError());
    AFAR_CUDA(cudaMemcpyAsync(lim, s->xfer, Nc * sizeof(V4<double>), cudaMemcpyDeviceToHost, s->stream));
    AFAR_CUDA(cudaStreamSynchronize(s->stream));
  } else {
    std::vector<float> tmp(4 * Nc);
    AFAR_CUDA(cudaMemcpy(tmp.data(), s->lim, Nc * sizeof(V4<float>), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < 4 * Nc; ++i) lim[i] = tmp[i];
  }
  return AFAR_OK;
}

extern "C" afar_status afar_upload_state(afar_solver* s, const afar_basicFieldData* FD, const afar_conservedFieldData* cFD,
                                         const afar_conservedFieldData* cFDold) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  s->head_pending = false;
  AFAR_CUDA(cudaSetDevice(s->device));
  return put_state(s, FD, cFD, cFDold);
}

extern "C" afar_status afar_download_state(afar_solver* s, afar_basicFieldData* FD, afar_conservedFieldData* cFD,
                                           int8_t* shockIndicator) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  AFAR_CUDA(cudaSetDevice(s->device));
  return get_state(s, FD, cFD, shockIndicator);
}

extern "C" afar_status afar_copyFieldDataDeviceToHost(afar_fieldPointer* h, afar_solver* s, int cellsNum,
                                                      int totalBoundaryFacesNum) {
  if (!h || !s) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  if (cellsNum != s->Nc || totalBoundaryFacesNum != s->Nb) {
    set_error("afar_copyFieldDataDeviceToHost: sizes differ from the uploaded fields");
    return AFAR_ERR_ARGUMENT;
  }
  return afar_download_state(s, h->FD, nullptr, h->shockIndicator);
}

extern "C" afar_status afar_state_snapshot(afar_solver* s, int op) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  if (op != AFAR_SNAPSHOT_SAVE && op != AFAR_SNAPSHOT_RESTORE) return (set_error("unknown snapshot op %d", op), AFAR_ERR_ARGUMENT);
  if (op == AFAR_SNAPSHOT_RESTORE) s->head_pending = false;
  AFAR_CUDA(cudaSetDevice(s->device));
  const size_t wb = w_size(s->policy) * (size_t)(s->Nc + s->Nb);
  const size_t ub = sizeof(V4<double>) * (size_t)s->Nc;
  if (op == AFAR_SNAPSHOT_SAVE && !s->snap) {
    afar_status st = dalloc(s, &s->snap, wb + 2 * ub + sizeof(StepCtl));
    if (st) return st;
  }
  if (!s->snap) return (set_error("restore without a saved snapshot"), AFAR_ERR_STATE);
  if (op == AFAR_SNAPSHOT_RESTORE && s->bvd_pending == 0) {  // as in put_state
    if (afar_status st = settle_bvd(s)) return st;
  }
  char* p = static_cast<char*>(s->snap);
  void* dst[4] = {p, p + wb, p + wb + ub, p + wb + 2 * ub};
  void* src[4] = {s->W, s->U, s->U0, s->ctl};
  const size_t n[4] = {wb, ub, ub, sizeof(StepCtl)};
  for (int i = 0; i < 4; ++i) {
    if (op == AFAR_SNAPSHOT_SAVE)
      AFAR_CUDA(cudaMemcpyAsync(dst[i], src[i], n[i], cudaMemcpyDeviceToDevice, s->stream));
    else
      AFAR_CUDA(cudaMemcpyAsync(src[i], dst[i], n[i], cudaMemcpyDeviceToDevice, s->stream));
  }
  // The further buffers' ghosts are the last uploaded ones but for those that every stage writes.
  if (op == AFAR_SNAPSHOT_SAVE) s->snap_ghosts = s->ghosts;
  if (op == AFAR_SNAPSHOT_RESTORE && s->policy == AFAR_POLICY_MIXED && s->Nb && s->ghosts != s->snap_ghosts)
    for (void* b : s->Wb)
      AFAR_CUDA(cudaMemcpyAsync(static_cast<V4<float>*>(b) + s->Nc, static_cast<V4<float>*>(s->W) + s->Nc,
                                sizeof(V4<float>) * (size_t)s->Nb, cudaMemcpyDeviceToDevice, s->stream));
  if (op == AFAR_SNAPSHOT_RESTORE) s->ghosts = s->snap_ghosts;
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  return AFAR_OK;
}

extern "C" afar_status afar_download_ls_matrix(afar_solver* s, float* matrix) {
  afar_status st = check_ready(s);
  if (st) return st;
  if (!matrix) return (set_error("null output"), AFAR_ERR_ARGUMENT);
  float* d = nullptr;
  const size_t n = 2 * (size_t)s->maxM * s->Nc;
  AFAR_CUDA(cudaMalloc(&d, n * sizeof(float)));
  AFAR_CUDA(cudaMemsetAsync(d, 0, n * sizeof(float), s->stream));
  const int gc = grid_for(s->Nc, kCellBlock);
  void* scratch = nullptr;
  const size_t sl = (s->policy == AFAR_POLICY_FP64 ? sizeof(V2<double>) : sizeof(V2<float>)) * (size_t)s->maxM * s->ldc;
  AFAR_CUDA(cudaMalloc(&scratch, sl));
  switch (s->policy) {
    case AFAR_POLICY_REF:
      k_setup_lsm<PolicyRef><<<gc, kCellBlock, 0, s->stream>>>(make_args<PolicyRef>(s), static_cast<V2<float>*>(scratch), d, s->maxM, s->order.perm);
      break;
    case AFAR_POLICY_FP64:
      k_setup_lsm<PolicyFP64><<<gc, kCellBlock, 0, s->stream>>>(make_args<PolicyFP64>(s), static_cast<V2<double>*>(scratch), d, s->maxM, s->order.perm);
      break;
    default:
      k_setup_lsm<PolicyMixed><<<gc, kCellBlock, 0, s->stream>>>(make_args<PolicyMixed>(s), static_cast<V2<float>*>(scratch), d, s->maxM, s->order.perm);
      break;
  }
  AFAR_CUDA(cudaGetLastError());
  AFAR_CUDA(cudaMemcpyAsync(matrix, d, n * sizeof(float), cudaMemcpyDeviceToHost, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  cudaFree(d);
  cudaFree(scratch);
  return AFAR_OK;
}

namespace {
// Switch decisions of the last stage: troubled cells (si[2c] != 0), cells on the low-order TVD
// reconstruction (si[2c+1] == 1), shock cells (si[2c+1] < 0) and KFVS faces (a shock cell on either
// side).  Per-block counts in shared memory, one atomic per counter and block.
__global__ void k_switch_counts(int Nc, int Nf, const int8_t* si, const int2* on, unsigned long long* out) {
  __shared__ unsigned int cnt[4];
  if (threadIdx.x < 4) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < Nc) {
    if (si[2 * i] != 0) atomicAdd(&cnt[0], 1u);
    const int8_t f = si[2 * i + 1];
    if (f == 1) atomicAdd(&cnt[1], 1u);
    if (f < 0) atomicAdd(&cnt[2], 1u);
  }
  if (i < Nf) {
    const int2 p = on[i];
    if (si[2 * p.x + 1] < 0 || si[2 * p.y + 1] < 0) atomicAdd(&cnt[3], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 4 && cnt[threadIdx.x]) atomicAdd(&out[threadIdx.x], (unsigned long long)cnt[threadIdx.x]);
}
}  // namespace

extern "C" afar_status afar_switch_counts(afar_solver* s, long long counts[4]) {
  afar_status st = check_ready(s);
  if (st) return st;
  if (!counts) return (set_error("null output"), AFAR_ERR_ARGUMENT);
  if (s->bvd_pending == 0 && (st = settle_bvd(s))) return st;  // a fused head: its stage's types
  unsigned long long* const d = s->counters;
  AFAR_CUDA(cudaMemsetAsync(d, 0, 4 * sizeof(unsigned long long), s->stream));
  const int n = std::max(s->Nc, s->Nf);
  k_switch_counts<<<grid_for(n, 256), 256, 0, s->stream>>>(s->Nc, s->Nf, s->si, s->on, d);
  unsigned long long h[4];
  AFAR_CUDA(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s->stream));
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  for (int k = 0; k < 4; ++k) counts[k] = (long long)h[k];
  return AFAR_OK;
}

extern "C" afar_status afar_device_bytes(afar_solver* s, size_t* bytes) {
  if (!s || !bytes) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  *bytes = s->bytes;
  return AFAR_OK;
}

extern "C" int afar_launches_per_step(afar_solver* s) {
  if (!s) return 13;  // the face-centre step of the fp64 and mixed policies
  if (s->policy == AFAR_POLICY_REF) return 14;
  return s->ng > 0 ? 17 : 13;  // the multi-point flux: a Gauss-point reconstruct per stage, the Courant kernel
}

extern "C" int afar_step_launches(afar_solver* s) {
  return s && s->policy == AFAR_POLICY_MIXED && fused_step(s) ? 6 : afar_launches_per_step(s);
}

extern "C" afar_status afar_freeFieldData(afar_solver* s) {
  if (!s) return AFAR_OK;
  if (s->batch) afar_batch_remove(s->batch, s);  // the batch forgets a freed member
  cudaSetDevice(s->device);
  if (s->stream) cudaStreamSynchronize(s->stream);
  destroy_graphs(s);
  for (void* p : s->allocs) cudaFree(p);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return AFAR_OK;
}

// ------------------------------------------------------------------------------------------------
// step parameters and batches

extern "C" afar_status afar_set_step_params(afar_solver* s, double dt, double CFL, double tEnd) {
  afar_status st = check_ready(s);
  if (st) return st;
  if (!(dt > 0.0) && !(CFL > 0.0)) return (set_error("afar_set_step_params: deltaT or CFL must be positive"), AFAR_ERR_ARGUMENT);
  k_set_ctl<<<1, 32, 0, s->stream>>>(s->ctl, dt > 0.0 ? dt : 0.0, CFL, tEnd);
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  AFAR_CUDA(cudaGetLastError());
  return AFAR_OK;
}

extern "C" afar_status afar_set_periodic(afar_solver* s, double px, double py) {
  if (!s) return (set_error("null solver"), AFAR_ERR_ARGUMENT);
  if (s->have_stencil) return (set_error("afar_set_periodic: call it before afar_setDeviceFieldDataStencil"), AFAR_ERR_STATE);
  if (!(px >= 0.0) || !(py >= 0.0)) return (set_error("afar_set_periodic: negative period"), AFAR_ERR_ARGUMENT);
  if (s->policy == AFAR_POLICY_REF && (px > 0.0 || py > 0.0))
    return (set_error("afar_set_periodic: the ref policy takes raw cell centres in its flux (no periodic meshes)"),
            AFAR_ERR_ARGUMENT);
  s->px = px;
  s->py = py;
  return AFAR_OK;
}

extern "C" afar_status afar_set_write_interval(afar_solver* s, double writeInterval) {
  if (!s || !s->have_fields) return (set_error("solver not initialised"), AFAR_ERR_STATE);
  if (!(writeInterval >= 0.0)) return (set_error("afar_set_write_interval: negative interval"), AFAR_ERR_ARGUMENT);
  s->head_pending = false;
  AFAR_CUDA(cudaSetDevice(s->device));
  k_set_write_interval<<<1, 32, 0, s->stream>>>(s->ctl, writeInterval);
  AFAR_CUDA(cudaStreamSynchronize(s->stream));
  AFAR_CUDA(cudaGetLastError());
  return AFAR_OK;
}

// The batch's launch schedule: which reconstruct each member runs (the tile-staged one unless its
// solver forces the register pass, so a member's result never depends on its batch-mates) and the
// BVD and flux block sizes (timed on the whole batch; the results do not depend on them, every
// reduction being an exact minimum).
struct BatchSchedule {
  int bvd_block = 128, flux_block = 256;
  int tile_members = 0, reg_members = 0;
  float ms[5] = {0.f, 0.f, 0.f, 0.f, 0.f};  // BVD at 64, 128, 256; flux at 128, 256 (0: from the cache)
};

struct afar_batch {
  int policy = AFAR_POLICY_MIXED;
  int device = 0;
  cudaStream_t stream = nullptr;
  std::vector<afar_solver*> members;
  void* tab = nullptr;  // StageArgs<P>[members]
  size_t tab_bytes = 0;
  // block maps, (member, block within the member) per block, one after another in one buffer:
  // 128-cell blocks of the tile-reconstruct members, of the register-reconstruct members, of every
  // member (update; the fp64 reconstruct), BVD blocks, face blocks
  int2* maps = nullptr;
  size_t maps_n = 0;
  int n_tile = 0, n_reg = 0, n_cell = 0, n_bvd = 0, n_face = 0;
  size_t smem = 0;  // dynamic shared memory of the staged reconstruct (largest member)
  bool fused = false;  // mixed: the fused stage (two kernels a stage)
  BatchSchedule sched;
  int forced_bvd = 0, forced_flux = 0;  // afar_batch_set_schedule (0: autotune)
  cudaGraphExec_t graph = nullptr;
  size_t launches = 0;  // kernels of it
  bool dirty = true;
};

namespace {

// Blocks of `block` cells (or faces when faces) of each member in `which` (empty: all members).
void batch_map(const std::vector<afar_solver*>& members, int block, bool faces, const std::vector<int>* which,
               std::vector<int2>& out) {
  for (size_t i = 0; i < members.size(); ++i) {
    if (which && !(*which)[i]) continue;
    const afar_solver* s = members[i];
    const long long n = faces ? (long long)s->Nf + s->Nb : (long long)s->Nc;
    const int nb = grid_for(n, block);
    for (int k = 0; k < nb; ++k) out.push_back(int2{(int)i, k});
  }
}

template <class P>
void launch_bvd(int block, int nblocks, const StageArgs<P>* t, const int2* map, cudaStream_t st) {
  if (nblocks == 0) return;
  if (block == 64)
    kb_bvd<P, 64><<<nblocks, 64, 0, st>>>(t, map);
  else if (block == 256)
    kb_bvd<P, 256><<<nblocks, 256, 0, st>>>(t, map);
  else
    kb_bvd<P, 128><<<nblocks, 128, 0, st>>>(t, map);
}
template <class P, bool DT>
void launch_flux(int block, int nblocks, const StageArgs<P>* t, const int2* map, cudaStream_t st) {
  if (nblocks == 0) return;
  if (block == 128)
    kb_flux<P, DT, 128><<<nblocks, 128, 0, st>>>(t, map);
  else
    kb_flux<P, DT, 256><<<nblocks, 256, 0, st>>>(t, map);
}

// The batch autotuner's decisions, per device, policy and batch shape (cells and members, each to
// a factor of two): BVD and flux block sizes.
std::mutex g_batch_tune_mu;
std::map<std::tuple<int, int, int, int>, std::pair<int, int>> g_batch_tune;

// A chain of six kernels in a graph for up to a MemberTable's worth of members of a fused batch, after *end
// if that is a node; *end is its last kernel then.
template <int NF, bool EARLY>
afar_status add_fused_chain(cudaGraph_t graph, int device, const MemberTable<PolicyMixed>& cells,
                            const MemberTable<PolicyMixed>& tiles, size_t smem, size_t tail_bytes,
                            cudaGraphNode_t* end) {
  const auto recon = kp_reconstruct_tile<NF, false, EARLY>, recon_dt = kp_reconstruct_tile<NF, true, EARLY>;
  const auto tail_1 = kp_tail<NF, true, EARLY>, tail_23 = kp_tail<NF, false, EARLY>;
  afar_status st;
  if ((st = raise_smem_limit(recon, device, smem))) return st;
  if ((st = raise_smem_limit(recon_dt, device, smem))) return st;
  if ((st = raise_smem_limit(tail_1, device, tail_bytes))) return st;
  if ((st = raise_smem_limit(tail_23, device, tail_bytes))) return st;
  cudaGraphEdgeData edge{};
  if (EARLY) {
    edge.from_port = cudaGraphKernelNodePortProgrammatic;
    edge.type = cudaGraphDependencyTypeProgrammatic;
  }
  cudaGraphNode_t last = *end;
  for (int k = 0; k < 3; ++k) {
    StageCoef coef = stage_coef(k);
    void* recon_args[] = {const_cast<MemberTable<PolicyMixed>*>(&cells), &k};
    void* tail_args[] = {const_cast<MemberTable<PolicyMixed>*>(&tiles), &k, &coef};
    cudaKernelNodeParams np{};
    cudaGraphNode_t node;
    np.func = reinterpret_cast<void*>(k == 0 ? recon_dt : recon);
    np.gridDim = dim3(cells.first[cells.n]);
    np.blockDim = dim3(kTile);
    np.sharedMemBytes = (unsigned)smem;
    np.kernelParams = recon_args;
    AFAR_CUDA(cudaGraphAddKernelNode(&node, graph, nullptr, 0, &np));
    if (last) AFAR_CUDA(cudaGraphAddDependencies(graph, &last, &node, &edge, 1));
    np.func = reinterpret_cast<void*>(k == 0 ? tail_1 : tail_23);
    np.gridDim = dim3(tiles.first[tiles.n]);
    np.blockDim = dim3(kTailThreads);
    np.sharedMemBytes = (unsigned)tail_bytes;
    np.kernelParams = tail_args;
    AFAR_CUDA(cudaGraphAddKernelNode(&last, graph, nullptr, 0, &np));
    AFAR_CUDA(cudaGraphAddDependencies(graph, &node, &last, &edge, 1));
  }
  *end = last;
  return AFAR_OK;
}

// Whether a batch of members with wide stencils (quads with their neighbours' neighbours, 12 members: the order
// along the curve helps their reconstruct least) runs the fused stage: not many members of few cells, whose last
// tiles and borders are much of the work.  us a step, fused / separate: 128 members of 6k quads 679 / 653, 10k
// 1033 / 993, 20k 1870 / 1834; 256 of 4k 788 / 731, 6k 1344 / 1217, 10k 2053 / 1904; but 96 members of 4k 301 / 309, 10k 772 / 769,
// 20k 1397 / 1405, 26k 1753 / 1747, and 128 of 40k 3505 / 3685.  Nor where the tiles are those of 96 cells and more than two
// waves of them: 3.6k quads, 24 members 98 / 98, 48 190 / 170, 60 224 / 208.  Other stencils gain throughout: 256 members of
// 4k quads (8 members a stencil) 657 / 679, 96 of 10k 550 / 692, 60 of 40k 1368 / 1572; quads and triangles (15), 256 of
// 13k 2351 / 2379, 96 of 33k 2077 / 2221.
bool fused_pays(long long members, long long cells, long long tiles, bool wide) {
  if (!wide) return true;
  if (members > 2 * MemberTable<PolicyMixed>::kMembers && cells < 32000 * members) return false;
  return cells > 4096 * members || tiles <= 8 * kSMs;
}

// One fused step of a batch as a graph.  The chains work on different members: side by side they share their
// kernels' ends, one after another they leave the GPU to one kernel at a time.  us a step side by side / in turn, by
// the cells of a chain, wide stencils: 480k 486 / 524, 690k 667 / 691, 940k 890 / 898 (more members 1406 / 1384), 1.2M
// 1127 / 1127 (1790 / 1740), 1.9M 1768 / 1678; others: 480k 350 / 399, 940k 1056 / 1091, 1.2M 1342 / 1381, 1.9M 1375 / 1377; 256
// ramps of 5k to 200k quads 8930 / 8490.  Early starts (see
// tail_early) where the members together are no more than 4000 blocks of 128 cells; us a step without / with:
// four members of 4k quads 48 / 43, twelve of 41k triangles 296 / 292, twelve of 121k 727 / 731, ten of 160k quads 1%
// slower with.  The single solve's exception for quads is not one here: 450 to 480 blocks without / with, four
// members of 14k 56.1 / 56.8 (edge-neighbour stencils 49.2 / 48.2), six of 10k 55.3 / 53.1 (51.2 / 48.6).
afar_status capture_fused(afar_batch* b, const std::vector<StageArgs<PolicyMixed>>& tab, int nfmax, size_t smem,
                          size_t tail_bytes, bool wide, cudaGraph_t* graph) {
  using Table = MemberTable<PolicyMixed>;
  AFAR_CUDA(cudaGraphCreate(graph, 0));
  std::unique_ptr<Table> cells(new Table), tiles(new Table);
  long long blocks = 0;
  for (const auto& m : tab) blocks += grid_for(m.Nc, kTile);
  const bool early = blocks <= 4000;
  afar_status st = AFAR_OK;
  cudaGraphNode_t end = nullptr;
  for (size_t i0 = 0; i0 < tab.size() && !st; i0 += Table::kMembers) {
    const int n = (int)std::min<size_t>(Table::kMembers, tab.size() - i0);
    cells->n = tiles->n = n;
    cells->first[0] = tiles->first[0] = 0;
    for (int i = 0; i < n; ++i) {
      const StageArgs<PolicyMixed>& m = tab[i0 + i];
      cells->m[i] = tiles->m[i] = m;
      cells->first[i + 1] = cells->first[i] + grid_for(m.Nc, kTile);
      tiles->first[i + 1] = tiles->first[i] + m.nTail;
    }
    const auto chain = nfmax <= 3 ? (early ? add_fused_chain<3, true> : add_fused_chain<3, false>)
                                  : (early ? add_fused_chain<4, true> : add_fused_chain<4, false>);
    if (cells->first[n] <= (wide ? 7000 : 12000)) end = nullptr;  // side by side
    st = chain(*graph, b->device, *cells, *tiles, smem, tail_bytes, &end);
  }
  if (st) {
    cudaGraphDestroy(*graph);
    *graph = nullptr;
  }
  return st;
}

template <class P>
afar_status batch_build(afar_batch* b) {
  std::vector<StageArgs<P>> tab;
  size_t smem = 0;
  afar_status st;
  long long cells = 0;
  std::vector<int> is_tile(b->members.size(), 1), is_reg(b->members.size(), 0);
  for (size_t i = 0; i < b->members.size(); ++i) {
    afar_solver* s = b->members[i];
    tab.push_back(make_args<P>(s));
    smem = std::max(smem, recon_smem<P>(s));
    cells += s->Nc;
    if constexpr (P::id == PolicyMixed::id) {
      // the tile-staged reconstruct unless the member's solver forces the register pass
      // (afar_set_tuning): a member's solo autotuner times its mesh alone, where small meshes leave
      // the GPU idle and favour the register pass; in a full batch the tile kernel is faster
      // (14.2M cells in 256 members: 11.2 against 11.5 ms a step)
      is_reg[i] = s->recon_request == 1;
      is_tile[i] = !is_reg[i];
    }
  }
  // mixed: the fused stage (two kernels a stage) where every member has it, unless a member forces
  // the register pass or block sizes of the separate BVD and flux kernels are asked for, and where it
  // pays; the same bits either way
  bool fused = P::id == PolicyMixed::id && !b->forced_bvd && !b->forced_flux && !tab.empty();
  size_t tail_bytes = 0;
  long long tiles = 0;
  int maxS = 0, maxM = 0;
  for (size_t i = 0; i < b->members.size(); ++i) {
    const afar_solver* s = b->members[i];
    fused = fused && fused_step(s) && is_tile[i];
    if (fused) tail_bytes = std::max<size_t>(tail_bytes, tail_smem(s->tail_faces, tail_cells(s)).bytes);
    tiles += grid_for(s->Nc, tail_cells(s));
    maxS = std::max(maxS, s->maxS);
    maxM = std::max(maxM, s->maxM);
  }
  const bool wide = maxM > 3 && maxS > 8;  // quads with their neighbours' neighbours
  fused = fused && fused_pays((long long)b->members.size(), cells, tiles, wide);
  b->fused = fused;
  int lc = 0, lm = 0;
  while ((1ll << (lc + 1)) <= cells) ++lc;
  while ((1ll << (lm + 1)) <= (long long)b->members.size()) ++lm;
  const auto key = std::make_tuple(b->device, (int)P::id, lc, lm);
  BatchSchedule sc;
  for (size_t i = 0; i < b->members.size(); ++i) sc.tile_members += is_tile[i], sc.reg_members += is_reg[i];
  bool timed = true;
  if (fused) {
    timed = false;  // neither kernel runs: the schedule keeps its defaults
  } else if (b->forced_bvd || b->forced_flux) {
    sc.bvd_block = b->forced_bvd ? b->forced_bvd : 128;
    sc.flux_block = b->forced_flux ? b->forced_flux : 256;
    timed = false;
  } else {
    std::lock_guard<std::mutex> lock(g_batch_tune_mu);
    auto it = g_batch_tune.find(key);
    if (it != g_batch_tune.end()) {
      sc.bvd_block = it->second.first;
      sc.flux_block = it->second.second;
      timed = false;
    }
  }

  std::vector<int2> mp_tile, mp_reg, mp_cell;
  if (!fused) {  // (the fused stage finds its members from its own arguments)
    batch_map(b->members, kTile, false, &is_tile, mp_tile);
    batch_map(b->members, kTile, false, &is_reg, mp_reg);
    batch_map(b->members, kCellBlock, false, nullptr, mp_cell);
  }
  // candidate maps for the timing: BVD in 64/128/256-cell blocks, flux in 128/256-face blocks
  const int bvd_sizes[3] = {64, 128, 256}, flux_sizes[2] = {128, 256};
  std::vector<int2> mp_bvd[3], mp_face[2];
  for (int k = 0; k < 3; ++k)
    if (timed || (!fused && bvd_sizes[k] == sc.bvd_block)) batch_map(b->members, bvd_sizes[k], false, nullptr, mp_bvd[k]);
  for (int k = 0; k < 2; ++k)
    if (timed || (!fused && flux_sizes[k] == sc.flux_block)) batch_map(b->members, flux_sizes[k], true, nullptr, mp_face[k]);
  std::vector<int2> all;
  auto append = [&](const std::vector<int2>& v) {
    const size_t o = all.size();
    all.insert(all.end(), v.begin(), v.end());
    return o;
  };
  const size_t o_tile = append(mp_tile), o_reg = append(mp_reg), o_cell = append(mp_cell);
  size_t o_bvd[3], o_face[2];
  for (int k = 0; k < 3; ++k) o_bvd[k] = append(mp_bvd[k]);
  for (int k = 0; k < 2; ++k) o_face[k] = append(mp_face[k]);

  auto grow = [&](void** p, size_t* cap, size_t need) -> afar_status {
    if (need > *cap) {
      if (*p) cudaFree(*p);
      *p = nullptr;
      AFAR_CUDA(cudaMalloc(p, need));
      *cap = need;
    }
    return AFAR_OK;
  };
  size_t cap_m = b->maps_n * sizeof(int2);
  if ((st = grow(&b->tab, &b->tab_bytes, std::max<size_t>(1, tab.size()) * sizeof(StageArgs<P>)))) return st;
  if ((st = grow(reinterpret_cast<void**>(&b->maps), &cap_m, std::max<size_t>(1, all.size()) * sizeof(int2)))) return st;
  b->maps_n = cap_m / sizeof(int2);
  if (!tab.empty() && !fused) {
    AFAR_CUDA(cudaMemcpyAsync(b->tab, tab.data(), tab.size() * sizeof(StageArgs<P>), cudaMemcpyHostToDevice, b->stream));
    AFAR_CUDA(cudaMemcpyAsync(b->maps, all.data(), all.size() * sizeof(int2), cudaMemcpyHostToDevice, b->stream));
  }
  AFAR_CUDA(cudaStreamSynchronize(b->stream));
  b->smem = smem;
  int nfmax = 3;
  for (afar_solver* s : b->members) nfmax = std::max(nfmax, s->maxM);
  if constexpr (P::id != PolicyMixed::id) {
    if ((st = raise_smem_limit(kb_reconstruct_fp64, b->device, smem))) return st;
  } else {
    if ((st = raise_smem_limit(kb_reconstruct_tile<P, 3>, b->device, smem))) return st;
    if ((st = raise_smem_limit(kb_reconstruct_tile<P, 4>, b->device, smem))) return st;
  }
  if (b->graph) {
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
  }
  b->n_tile = (int)mp_tile.size();
  b->n_reg = (int)mp_reg.size();
  b->n_cell = (int)mp_cell.size();
  if (tab.empty()) {
    b->sched = sc;
    b->dirty = false;
    return AFAR_OK;
  }
  const StageArgs<P>* t = static_cast<const StageArgs<P>*>(b->tab);
  auto reconstruct = [&] {
    if constexpr (P::id == PolicyMixed::id) {
      const auto f = nfmax <= 3 ? kb_reconstruct_tile<P, 3> : kb_reconstruct_tile<P, 4>;
      if (b->n_tile) f<<<b->n_tile, kTile, b->smem, b->stream>>>(t, b->maps + o_tile);
      if (b->n_reg) kb_reconstruct_reg<P><<<b->n_reg, kCellBlock, 0, b->stream>>>(t, b->maps + o_reg);
    } else
      kb_reconstruct_fp64<<<b->n_cell, kCellBlock, b->smem, b->stream>>>(t, b->maps + o_cell);
  };

  if (timed) {
    // reconstruct once so that the BVD and flux read this step's intermediates, then time each
    // candidate: a warm-up and the best of three launches (both kernels are functions of the state
    // and the stage's intermediates; they change neither the state nor the step control)
    for (afar_solver* m : b->members)
      if ((st = settle_bvd(m))) return st;
    reconstruct();
    cudaEvent_t e0, e1;
    AFAR_CUDA(cudaEventCreate(&e0));
    AFAR_CUDA(cudaEventCreate(&e1));
    auto best_of = [&](auto&& launch) -> float {
      launch();
      float best = 1e30f;
      for (int r = 0; r < 3; ++r) {
        cudaEventRecord(e0, b->stream);
        launch();
        cudaEventRecord(e1, b->stream);
        cudaEventSynchronize(e1);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        best = std::min(best, ms);
      }
      return best;
    };
    for (int k = 0; k < 3; ++k)
      sc.ms[k] = best_of([&] { launch_bvd<P>(bvd_sizes[k], (int)mp_bvd[k].size(), t, b->maps + o_bvd[k], b->stream); });
    for (int k = 0; k < 2; ++k)
      sc.ms[3 + k] =
          best_of([&] { launch_flux<P, false>(flux_sizes[k], (int)mp_face[k].size(), t, b->maps + o_face[k], b->stream); });
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    AFAR_CUDA(cudaGetLastError());
    for (afar_solver* m : b->members)
      if ((st = check_device_error(m))) return st;
    sc.bvd_block = bvd_sizes[std::min_element(sc.ms, sc.ms + 3) - sc.ms];
    sc.flux_block = flux_sizes[std::min_element(sc.ms + 3, sc.ms + 5) - (sc.ms + 3)];
    std::lock_guard<std::mutex> lock(g_batch_tune_mu);
    g_batch_tune[key] = {sc.bvd_block, sc.flux_block};
  }
  const int kb = sc.bvd_block == 64 ? 0 : sc.bvd_block == 128 ? 1 : 2;
  const int kf = sc.flux_block == 128 ? 0 : 1;
  const int2* bmap = b->maps + o_bvd[kb];
  const int2* fmap = b->maps + o_face[kf];
  b->n_bvd = (int)mp_bvd[kb].size();
  b->n_face = (int)mp_face[kf].size();
  b->sched = sc;

  // capture one step of the whole batch
  cudaGraph_t g = nullptr;
  if constexpr (P::id == PolicyMixed::id) {
    if (fused) {
      if ((st = capture_fused(b, tab, nfmax, smem, tail_bytes, wide, &g))) return st;
    }
  }
  if (!fused) {
    AFAR_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < 3; ++k) {
      reconstruct();
      launch_bvd<P>(sc.bvd_block, b->n_bvd, t, bmap, b->stream);
      if (k == 0)
        launch_flux<P, true>(sc.flux_block, b->n_face, t, fmap, b->stream);
      else
        launch_flux<P, false>(sc.flux_block, b->n_face, t, fmap, b->stream);
      kb_update<P><<<b->n_cell, kCellBlock, 0, b->stream>>>(t, b->maps + o_cell, stage_coef(k));
    }
    kb_finish_step<P><<<grid_for((long long)tab.size(), 128), 128, 0, b->stream>>>(t, (int)tab.size());
    AFAR_CUDA(cudaStreamEndCapture(b->stream, &g));
  }
  cudaError_t e = cudaGraphGetNodes(g, nullptr, &b->launches);
  if (e == cudaSuccess) e = cudaGraphInstantiate(&b->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    b->graph = nullptr;
    set_error("batch graph instantiation failed: %s", cudaGetErrorString(e));
    return AFAR_ERR_CUDA;
  }
  b->dirty = false;
  return AFAR_OK;
}

}  // namespace

extern "C" afar_status afar_batch_create(afar_batch** out, int policy, int device) {
  if (!out || (policy != AFAR_POLICY_MIXED && policy != AFAR_POLICY_FP64)) {
    set_error("afar_batch_create: null output or policy other than fp64/mixed");
    return AFAR_ERR_ARGUMENT;
  }
  *out = nullptr;
  AFAR_CUDA(cudaSetDevice(device));
  afar_batch* b = new afar_batch();
  b->policy = policy;
  b->device = device;
  if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete b;
    set_error("cudaStreamCreate failed");
    return AFAR_ERR_CUDA;
  }
  *out = b;
  return AFAR_OK;
}

extern "C" afar_status afar_batch_add(afar_batch* b, afar_solver* s) {
  if (!b || !s) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  afar_status st = check_ready(s);
  if (st) return st;
  if (s->policy != b->policy || s->device != b->device)
    return (set_error("afar_batch_add: member policy/device differ from the batch's"), AFAR_ERR_ARGUMENT);
  if (!(s->R > 0.0)) return (set_error("afar_batch_add: call afar_set_gas on the member first"), AFAR_ERR_STATE);
  if (!s->have_stencil)
    return (set_error("afar_batch_add: upload the stencil (afar_setDeviceFieldDataStencil) first"), AFAR_ERR_STATE);
  if (s->batch) return (set_error("afar_batch_add: the solver already belongs to a batch"), AFAR_ERR_STATE);
  if (s->ng > 0)
    return (set_error("afar_batch_add: batches run the face-centre flux; the solver has the multi-point face flux"),
            AFAR_ERR_ARGUMENT);
  AFAR_CUDA(cudaStreamSynchronize(s->stream));  // no pending work of the member on its own stream
  b->members.push_back(s);
  s->batch = b;
  b->dirty = true;
  return AFAR_OK;
}

extern "C" afar_status afar_batch_remove(afar_batch* b, afar_solver* s) {
  if (!b || !s) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  for (size_t i = 0; i < b->members.size(); ++i)
    if (b->members[i] == s) {
      AFAR_CUDA(cudaSetDevice(b->device));
      AFAR_CUDA(cudaStreamSynchronize(b->stream));
      b->members.erase(b->members.begin() + i);
      s->batch = nullptr;
      b->dirty = true;
      return AFAR_OK;
    }
  set_error("afar_batch_remove: not a member");
  return AFAR_ERR_ARGUMENT;
}

extern "C" afar_status afar_batch_size(afar_batch* b, int* n) {
  if (!b || !n) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  *n = (int)b->members.size();
  return AFAR_OK;
}

extern "C" afar_status afar_batch_run(afar_batch* b, int nSteps, float* ms) {
  NvtxRange nvtx("afar_batch_run");
  if (!b || nSteps < 0) return (set_error("afar_batch_run: bad argument"), AFAR_ERR_ARGUMENT);
  AFAR_CUDA(cudaSetDevice(b->device));
  afar_status st;
  if (b->dirty) {
    st = b->policy == AFAR_POLICY_MIXED ? batch_build<PolicyMixed>(b) : batch_build<PolicyFP64>(b);
    if (st) return st;
  }
  if (ms) *ms = 0.f;
  if (b->members.empty() || nSteps == 0) return AFAR_OK;
  cudaEvent_t e0, e1;
  AFAR_CUDA(cudaEventCreate(&e0));
  AFAR_CUDA(cudaEventCreate(&e1));
  AFAR_CUDA(cudaEventRecord(e0, b->stream));
  for (int i = 0; i < nSteps; ++i) AFAR_CUDA(cudaGraphLaunch(b->graph, b->stream));
  for (afar_solver* m : b->members) m->bvd_pending = b->fused ? 2 : -1;
  AFAR_CUDA(cudaEventRecord(e1, b->stream));
  AFAR_CUDA(cudaEventSynchronize(e1));
  if (ms) AFAR_CUDA(cudaEventElapsedTime(ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  AFAR_CUDA(cudaGetLastError());
  for (afar_solver* m : b->members)
    if ((st = check_device_error(m))) return st;
  return AFAR_OK;
}

extern "C" afar_status afar_batch_destroy(afar_batch* b) {
  if (!b) return AFAR_OK;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (afar_solver* m : b->members) m->batch = nullptr;
  if (b->graph) cudaGraphExecDestroy(b->graph);
  if (b->tab) cudaFree(b->tab);
  if (b->maps) cudaFree(b->maps);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return AFAR_OK;
}

extern "C" afar_status afar_batch_set_schedule(afar_batch* b, int bvdBlock, int fluxBlock) {
  if (!b) return (set_error("null batch"), AFAR_ERR_ARGUMENT);
  if ((bvdBlock != 0 && bvdBlock != 64 && bvdBlock != 128 && bvdBlock != 256) ||
      (fluxBlock != 0 && fluxBlock != 128 && fluxBlock != 256))
    return (set_error("afar_batch_set_schedule: BVD block 0/64/128/256, flux block 0/128/256"), AFAR_ERR_ARGUMENT);
  b->forced_bvd = bvdBlock;
  b->forced_flux = fluxBlock;
  b->dirty = true;
  return AFAR_OK;
}

extern "C" afar_status afar_batch_get_schedule(afar_batch* b, int* tileMembers, int* registerMembers, int* bvdBlock,
                                               int* fluxBlock, float ms[5]) {
  if (!b) return (set_error("null batch"), AFAR_ERR_ARGUMENT);
  if (b->dirty) {
    AFAR_CUDA(cudaSetDevice(b->device));
    const afar_status st = b->policy == AFAR_POLICY_MIXED ? batch_build<PolicyMixed>(b) : batch_build<PolicyFP64>(b);
    if (st) return st;
  }
  if (tileMembers) *tileMembers = b->sched.tile_members;
  if (registerMembers) *registerMembers = b->sched.reg_members;
  if (bvdBlock) *bvdBlock = b->sched.bvd_block;
  if (fluxBlock) *fluxBlock = b->sched.flux_block;
  if (ms)
    for (int k = 0; k < 5; ++k) ms[k] = b->sched.ms[k];
  return AFAR_OK;
}

extern "C" afar_status afar_batch_step_launches(afar_batch* b, int* launches) {
  if (!b || !launches) return (set_error("null argument"), AFAR_ERR_ARGUMENT);
  *launches = 0;
  if (b->members.empty()) return AFAR_OK;
  if (b->dirty) {
    AFAR_CUDA(cudaSetDevice(b->device));
    const afar_status st = b->policy == AFAR_POLICY_MIXED ? batch_build<PolicyMixed>(b) : batch_build<PolicyFP64>(b);
    if (st) return st;
  }
  *launches = (int)b->launches;
  return AFAR_OK;
}

extern "C" afar_status afar_debug_wait_injection(int device, unsigned extraBytes, long long limitClocks) {
  return afar_debug_wait_injection_at(device, AFAR_WAIT_RECONSTRUCT_IDS, extraBytes, 0, limitClocks);
}

extern "C" afar_status afar_debug_wait_injection_at(int device, int where, unsigned extraBytes, int late,
                                                    long long limitClocks) {
  if (where < AFAR_WAIT_RECONSTRUCT_IDS || where > AFAR_WAIT_TAIL_STATES || (late && where != AFAR_WAIT_TAIL_FACES))
    return (set_error("afar_debug_wait_injection_at: unknown wait %d, or late at another than the tail's first", where),
            AFAR_ERR_ARGUMENT);
  AFAR_CUDA(cudaSetDevice(device));
  const long long lim = limitClocks > 0 ? limitClocks : (1ll << 31);
  unsigned extra[4] = {0, 0, 0, 0}, lateBytes = late ? extraBytes : 0;
  extra[where] = extraBytes;
  AFAR_CUDA(cudaMemcpyToSymbol(g_tile_extra_tx, extra, sizeof(extra)));
  AFAR_CUDA(cudaMemcpyToSymbol(g_tail_late_tx, &lateBytes, sizeof(lateBytes)));
  AFAR_CUDA(cudaMemcpyToSymbol(g_tile_wait_limit, &lim, sizeof(lim)));
  AFAR_CUDA(cudaDeviceSynchronize());
  return AFAR_OK;
}

extern "C" afar_status afar_set_face_gauss_flux(afar_solver* s, int nPoints, const double* points,
                                                const double* pointWeights, const double* rbfGauss) {
  afar_status st = check_ready(s);
  if (st || (st = check_not_batched(s))) return st;
  if (nPoints == 0) {
    s->ng = 0;
    destroy_graphs(s);
    return AFAR_OK;
  }
  if (s->policy == AFAR_POLICY_REF)
    return (set_error("afar_set_face_gauss_flux: the ref policy keeps the reference's face-centre flux"),
            AFAR_ERR_ARGUMENT);
  if (nPoints < 1 || nPoints > 4 || !points || !pointWeights || !rbfGauss)
    return (set_error("afar_set_face_gauss_flux: 1 to 4 points per face and non-null arrays"), AFAR_ERR_ARGUMENT);
  double wsum = 0.0;
  for (int k = 0; k < nPoints; ++k) {
    if (!(pointWeights[k] > 0.0)) return (set_error("afar_set_face_gauss_flux: non-positive point weight"), AFAR_ERR_ARGUMENT);
    wsum += pointWeights[k];
  }
  const int Nf = s->Nf, ng = nPoints, nmax = s->maxS + 1;
  const bool mixed = s->policy == AFAR_POLICY_MIXED;
  const size_t wS = mixed ? sizeof(float) : sizeof(double), wG = mixed ? sizeof(float) : sizeof(double);
  if ((st = dalloc(s, &s->wg, wS * (size_t)s->maxM * ng * nmax * s->ldc))) return st;
  AFAR_CUDA(cudaMemsetAsync(s->wg, 0, wS * (size_t)s->maxM * ng * nmax * s->ldc, s->stream));
  if ((st = dalloc(s, &s->sgk, 2 * wG * (size_t)s->maxM * ng * s->ldc))) return st;
  AFAR_CUDA(cudaMemsetAsync(s->sgk, 0, 2 * wG * (size_t)s->maxM * ng * s->ldc, s->stream));
  if ((st = dalloc(s, &s->fgk, 2 * wG * (size_t)Nf * ng))) return st;
  if ((st = dalloc(s, &s->fvg, 4 * wG * 2 * (size_t)Nf * ng))) return st;
  if (mixed && s->flux == s->xfer) {  // its steps have a flux between the calls of the reference-shaped loop
    void* flux = nullptr;
    if ((st = dalloc(s, &flux, sizeof(V4<float>) * (size_t)(Nf + s->Nb)))) return st;
    s->flux = flux;
  }
  if (mixed && !s->dtg && (st = dalloc_t(s, &s->dtg, (size_t)Nf))) return st;  // of its FP64 Courant step
  double *d_w = nullptr, *d_p = nullptr;
  V4<double>* fxy = nullptr;
  auto cleanup = [&]() {
    if (d_w) cudaFree(d_w);
    if (d_p) cudaFree(d_p);
    if (fxy) cudaFree(fxy);
  };
  const size_t nw = (size_t)Nf * 2 * ng * nmax, np = (size_t)Nf * ng * 2;
  if (cudaMalloc(&d_w, sizeof(double) * (nw ? nw : 1)) != cudaSuccess ||
      cudaMalloc(&d_p, sizeof(double) * (np ? np : 1)) != cudaSuccess ||
      cudaMalloc(&fxy, sizeof(V4<double>) * (size_t)(Nf + s->Nb + 1)) != cudaSuccess) {
    cleanup();
    set_error("afar_set_face_gauss_flux: out of device memory for the set-up");
    return AFAR_ERR_CUDA;
  }
  cudaMemcpyAsync(d_w, rbfGauss, sizeof(double) * nw, cudaMemcpyHostToDevice, s->stream);
  cudaMemcpyAsync(d_p, points, sizeof(double) * np, cudaMemcpyHostToDevice, s->stream);
  V4<double>* fsr = nullptr;
  if (cudaMalloc(&fsr, sizeof(V4<double>) * (size_t)(Nf + s->Nb + 1)) != cudaSuccess) {
    cleanup();
    set_error("afar_set_face_gauss_flux: out of device memory for the set-up");
    return AFAR_ERR_CUDA;
  }
  const int gF = grid_for((long long)Nf + s->Nb, kFaceBlock);
  k_split_faces<<<gF, kFaceBlock, 0, s->stream>>>(Nf + s->Nb, Nf, s->faceRaw, fxy, fsr, s->order);
  s->ng = ng;
  for (int k = 0; k < 4; ++k) s->gw[k] = k < ng ? pointWeights[k] / wsum : 0.0;
  auto setup = [&](auto tag) {
    using P = decltype(tag);
    StageArgs<P> a = make_args<P>(s);
    if (mixed) k_setup_face_geom<P><<<gF, kFaceBlock, 0, s->stream>>>(a, fxy, fsr);  // (the same again, and dtg)
    k_setup_gauss<P><<<grid_for(s->Nc, kCellBlock), kCellBlock, 0, s->stream>>>(a, d_w, d_p, s->order.fperm);
    if (Nf > 0) k_setup_gauss_faces<P><<<grid_for((long long)Nf * ng, 256), 256, 0, s->stream>>>(a, d_p, fxy, s->order.fperm);
  };
  if (mixed)
    setup(PolicyMixed{});
  else
    setup(PolicyFP64{});
  const cudaError_t e = cudaGetLastError();
  const cudaError_t e2 = cudaStreamSynchronize(s->stream);
  cleanup();
  cudaFree(fsr);
  if (e != cudaSuccess || e2 != cudaSuccess) {
    s->ng = 0;
    set_error("afar_set_face_gauss_flux: set-up failed: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    return AFAR_ERR_CUDA;
  }
  destroy_graphs(s);  // the next run captures the step with the multi-point flux
  return AFAR_OK;
}
