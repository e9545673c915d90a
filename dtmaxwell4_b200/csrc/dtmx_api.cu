// dtmx_api.cu -- host runtime behind the C ABI declared in include/dtmx.h.
//
// Owns every device allocation of a simulation context, validates the
// configuration (the reference's printf+exit checks in GeoParamsHost::set,
// DTmxw.cu:278-487, become status codes), builds the coefficient tables and
// launches the per-step kernel sequence on the context's stream.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>
#include <array>
#include <atomic>
#include <thread>

#include <cudaTypedefs.h>

#include "dtmx.h"
#include "dtmx_device.cuh"
#include "dtmx_aux.cuh"
#include "dtmx_torre.cuh"
#include "dtmx_adjoint.cuh"
#include "dtmx_fused.cuh"
#include "dtmx_adjsweep.cuh"

using namespace dtmx;

struct DftHost {
  DftDev d;
  int ncomp;
  double* omega = nullptr;
  double2* acc = nullptr;
  float* stage = nullptr;
  long long* sstep = nullptr;
};

// The device tables of a set of DFT planes that are sampled and folded
// together: their descriptors, the block map of the samples (tail_kernel) and
// the work units of a fold (dft_flush_kernel).
struct MonTable {
  DftDev* tab = nullptr;
  int2* map = nullptr;
  FlushUnit* unit = nullptr;
  int nmap = 0, nunit = 0;
  int nstaged = 0;          // samples staged since the last fold, the same for every plane
};

// Six DFT patches of the tangential E and H components on the faces of a box
// and the device buffer their flux reduction writes to.
struct FluxHost {
  int face[6];              // DFT ids: x lo, x hi, y lo, y hi, z lo, z hi
  // far field: tangential E and H of each face plane and H of the next plane,
  // on windows [lo, hi] of the in-plane axes (one more point than the flux windows)
  int ffe[6], ffh[6];
  double sgn_area[6];       // outward sign times the cell face area
  int nfreq;
  double* d_out = nullptr;  // [6][nfreq]
};

// A device array of a parkable context: a CUDA virtual-address reservation
// with its own physical allocation, so that dtmx_park can release the physical
// memory while the address (held in Params, TMA descriptors and graphs) stays
// reserved, and dtmx_unpark can map new memory at the same address.
struct VmmBlock {
  CUdeviceptr va = 0;
  size_t size = 0;
  CUmemGenericAllocationHandle h = 0;
  void* host = nullptr;       // pinned copy while parked
  bool dead = false;          // parked without a copy: refilled with zeros on unpark
  bool fixed = false;         // constant once the context has stepped (materials, tables)
  bool saved_prepared = false;  // the host copy was taken after the context first stepped
};

// the pieces of a streaming launch (plan_work)
struct WorkPlan {
  bool table = false, alone = false;   // alone: to be launched when the kernel ahead has finished
  int xchunk = 0, longest = 0;         // planes of equal pieces; of the longest piece
  dim3 grid;
  Work<true> work{};
};

struct dtmx_ctx {
  dtmx_config cfg{};
  int dev = 0;
  cudaStream_t stream = nullptr;
  Params P{};
  int nzp = 0;
  size_t nstore = 0;            // elements per component array (padded)
  size_t ncell = 0;             // nx*ny*nz
  std::vector<void*> allocs;
  std::vector<VmmBlock> vmm;    // the arrays of a parkable context (instead of allocs)
  bool parked = false;
  std::map<std::array<int, 4>, WorkPlan> work;   // by (kind, tile rows, planes per CTA asked for, early launches)
  WorkPlan work_once;                            // while the caller captures the stream
  bool early = false;           // launches may overlap their set-up with the kernel ahead (launch)
  // coefficient tables
  float* ctab[3][3] = {};
  // materials
  MatTable* d_mt = nullptr;
  MatTable h_mt{};
  dtmx_material mats[DTMX_MAX_MATERIALS]{};
  int nmat = 1;
  uint8_t* d_mat[3] = {};
  std::vector<uint8_t> h_mat[3];
  // sources
  std::vector<PointSrcDev> psrc;
  PointSrcDev* d_psrc = nullptr;   // the sources sorted by node (prepare)
  int2* d_psrc_run = nullptr;      // {first, count} of each node's (more sources than the tail's list holds)
  int nrun = 0;
  int has_tfsf = 0;
  dtmx_tfsf tfsf{};
  TfsfDev T{};
  int line_cap = 0;              // cells of line_e / line_h
  double* line_e = nullptr;
  double* line_h = nullptr;
  int line_src = 0;
  // monitors
  std::vector<ProbeDev> probes;
  ProbeDev* d_probes = nullptr;
  float* d_traces = nullptr;
  int probe_cap = 0;
  float* dense = nullptr;       // dense copy of a small field (DenseBlock)
  std::vector<DftHost> dfts;
  std::vector<FluxHost> fluxes;
  MonTable mon, objmon;         // tables of dfts and of the objective's plane
  unsigned* d_ticket = nullptr; // blocks of a tail launch that are done
  float* hist_out = nullptr;    // where the next step's design-region E goes (nullptr: not recorded)
  // state
  long long* d_step = nullptr;
  int* d_flag = nullptr;
  long long step = 0;
  long long launches = 0;
  bool prepared = false;
  bool profiling = false;
  cudaEvent_t ev[4] = {};
  double prof_ms_h = 0, prof_ms_e = 0;
  long long prof_count = 0;
  bool prof_pending = false;
  int engine = 0, tblock = 0;
  int xchunk = 0;               // planes per CTA of the per-step kernels (0: automatic)
  // 16 captured per-step launch sequences, one per field buffer holding the
  // current state (the single-sweep engine alternates them)
  cudaGraphExec_t graph16[2] = {};
  long long graph_launches[2] = {};
  TmaMaps maps{};
  // single-sweep engine (engine 3): the second field buffer and second set of
  // H auxiliaries (allocated on first use) and the maps reading each buffer
  // (its tiles are the per-step kernels' tiles and share their uniform-material
  // table).  P.f / P.ab.aux always point at the current state; the other set
  // is swapped in after every step.
  float* f_alt[6] = {};
  float* hax_alt[3][2] = {};
  TmaMaps maps_alt{};
  FusedMaps fmaps[2]{};               // 16-row tiles: [0] reads P.f, [1] reads f_alt (swapped with the buffers)
  FusedMaps fmaps8[2]{};              // the same for 8-row tiles
  int frows = 16;                     // tile rows of the single sweep (16 or 8; dtmx_set_tile_rows, dtmx_autotune)
  bool fused_ready = false;
  // The automatic choice's second set may be given back to whoever needs the
  // memory, another thread too, while no call on this context is using it.
  std::mutex run;
  std::atomic<std::thread::id> runner{};   // the thread that holds run
  bool lendable = false;              // registered in lenders()
  bool set_in_graph = false;          // a graph of the caller's uses the second set: it stays
  double fa_reserved = 0.0;           // bytes that fa_reserve has asked for
  bool spare_others = false;          // an allocation that is not worth another context's set
  bool pinned = false;                // the caller holds the fields' addresses: see step_engine
  bool graphs_stale = false;          // the step graphs were made before that
  bool auto_per_step = false;         // the automatic choice found no room for the second set
  int parity = 0;                     // 0: state in the buffers allocated first
  int* d_err = nullptr;
  bool has_gyro = false;
  // design region and the objective of dtmx_forward_adjoint
  float* d_des_ie[3] = {};
  std::vector<float> h_des_ie[3];
  bool monitors_off = false;  // probes and DFT planes paused (recomputed segments)
  bool obj_on = false;        // capture the objective's flux DFT each step
  long long adj_budget = -1;  // bytes of design-region history the adjoint may keep (-1: a quarter of free memory)
  DftHost obj{};
  int gcur = 0;              // gyrotropic current buffer holding J^{n-1/2}
  // wavefront engine
  TorreMaps tmaps{};
  bool tmaps_ok = false;
  int* d_ctr = nullptr;
  signed char* d_umat = nullptr;
  cudaError_t launch_err = cudaSuccess;   // the first launch that failed and has not been reported
  int fail_in[2] = {-1, -1};    // dtmx_fail_next: requests left before one is refused (-1: none)
  std::string err;
};

constexpr size_t kEarlyCells = (size_t)1 << 23;

// polls of one bounded device wait (mbarrier stages, wavefront neighbours / 16)
constexpr long long kWaitPolls = 1LL << 26;


// ---- large reads into pageable memory
// The driver's copy to pageable memory runs at 5 GB/s (151 MB of DFT
// accumulators: 30 ms), bound by one host thread that touches the caller's
// pages.  From 4 MB on, four threads copy instead: each has two pinned slots of
// 1 MB, lets the next piece come in while it moves the last one to the caller's
// buffer, and takes piece after piece until none is left.  The slots (8 MB)
// belong to the process, are used by one read at a time (another one meanwhile
// takes the driver's path) and are freed with the last context.  Pinning them
// takes 3 to 10 ms, as much as they save on 32 MB of fresh pages (8.4 MB 2.2 ms by
// the driver's copy, 1.05 through the slots) and more than they save where the
// caller's pages have been touched (0.45 and 0.4 to 0.6), so they are made by a read of 32
// MB, or by the one that brings the bytes read without them to 64 MB.
struct ReadSlots {
  std::mutex use, life;
  char* buf = nullptr;
  size_t plain = 0;             // bytes of large reads that took the driver's path for want of slots
  int contexts = 0;
};
constexpr size_t kReadPiece = 1 << 20, kReadMin = 4 << 20, kReadWorth = 32 << 20;
constexpr int kReadThreads = 4;
static ReadSlots& read_slots() {
  static ReadSlots s;
  return s;
}
static void read_slots_hold() {
  ReadSlots& S = read_slots();
  std::lock_guard<std::mutex> lk(S.life);
  S.contexts++;
}
static void read_slots_drop() {
  ReadSlots& S = read_slots();
  std::lock_guard<std::mutex> lk(S.life);
  if (--S.contexts > 0) return;
  std::lock_guard<std::mutex> us(S.use);
  if (S.buf) cudaFreeHost(S.buf);
  S.buf = nullptr;
  S.plain = 0;
}

// the calling thread's device while it uses another one
struct DeviceGuard {
  int was = -1;
  explicit DeviceGuard(int dev) {
    int cur = -1;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev && cudaSetDevice(dev) == cudaSuccess) was = cur;
  }
  ~DeviceGuard() {
    if (was >= 0) cudaSetDevice(was);
  }
};

// bytes of device memory to host memory, after the work queued on the stream; waits for it
static cudaError_t copy_to_host(int dev, cudaStream_t st, void* host, const void* devp, size_t bytes) {
  ReadSlots& S = read_slots();
  cudaPointerAttributes at{};
  bool direct = bytes < kReadMin;
  if (!direct) {
    if (cudaPointerGetAttributes(&at, host) == cudaSuccess) direct = at.type != cudaMemoryTypeUnregistered;
    else cudaGetLastError();
  }
  std::unique_lock<std::mutex> lk(S.use, std::defer_lock);
  if (!direct && !lk.try_lock()) direct = true;
  if (!direct && !S.buf && bytes < kReadWorth && (S.plain += bytes) < 2 * kReadWorth) direct = true;
  if (!direct && !S.buf && cudaHostAlloc((void**)&S.buf, kReadPiece * 2 * kReadThreads, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    S.buf = nullptr;
    direct = true;
  }
  if (direct && lk.owns_lock()) lk.unlock();
  cudaError_t e = cudaSuccess;
  if (!direct) {
    const size_t pieces = (bytes + kReadPiece - 1) / kReadPiece;
    std::atomic<size_t> next{0};
    std::atomic<int> bad{(int)cudaSuccess};
    auto work = [&](int w) {
      const DeviceGuard guard(dev);
      char* slot[2] = {S.buf + (size_t)w * 2 * kReadPiece, S.buf + (size_t)(w * 2 + 1) * kReadPiece};
      cudaEvent_t ev[2] = {};
      size_t at[2] = {pieces, pieces};
      cudaError_t r = cudaSuccess;
      for (int q = 0; q < 2 && r == cudaSuccess; q++) r = cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming);
      auto fetch = [&](int q) {
        at[q] = next.fetch_add(1);
        if (at[q] >= pieces) return;
        const size_t o = at[q] * kReadPiece;
        r = cudaMemcpyAsync(slot[q], (const char*)devp + o, std::min(kReadPiece, bytes - o), cudaMemcpyDeviceToHost, st);
        if (r == cudaSuccess) r = cudaEventRecord(ev[q], st);
      };
      for (int q = 0; q < 2 && r == cudaSuccess; q++) fetch(q);
      for (int q = 0; r == cudaSuccess && at[q] < pieces; q ^= 1) {
        if ((r = cudaEventSynchronize(ev[q])) != cudaSuccess) break;
        const size_t o = at[q] * kReadPiece;
        memcpy((char*)host + o, slot[q], std::min(kReadPiece, bytes - o));
        fetch(q);
      }
      if (r != cudaSuccess) { cudaGetLastError(); bad = (int)r; cudaStreamSynchronize(st); }   // no copy into the slots stays in flight
      for (auto v : ev)
        if (v) cudaEventDestroy(v);
    };
    std::vector<std::thread> th;
    try {
      th.reserve(kReadThreads);
      for (int w = 1; w < kReadThreads; w++) th.emplace_back(work, w);
    } catch (...) {
      // fewer threads: those that run, and this one, take all pieces
    }
    work(0);
    for (auto& t : th) t.join();
    e = (cudaError_t)bad.load();
    if (e == cudaSuccess) return cudaSuccess;
    // (a failure in a thread: once more, the plain way)
  }
  e = cudaMemcpyAsync(host, devp, bytes, cudaMemcpyDeviceToHost, st);
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}
static int copy_out(dtmx_ctx* ctx, void* host, const void* devp, size_t bytes);

// Field rows between the padded layout and a dense one (the driver's strided
// copy moves 55-float rows at 0.3 GB/s).
__global__ void dense_rows_kernel(const float* src, int sp, float* dst, int dp, long long rows, int nz) {
  for (long long r = blockIdx.x * 8LL + threadIdx.y; r < rows; r += gridDim.x * 8LL)
    for (int k = threadIdx.x; k < nz; k += 32) dst[r * dp + k] = src[r * sp + k];
}
// rows of a dense piece: at most 64 MB
static size_t dense_rows(int nz, size_t rows) { return std::min(rows, std::max<size_t>(1, ((size_t)64 << 20) / ((size_t)nz * 4))); }

static void drop_graphs(dtmx_ctx* ctx) {
  for (auto& g : ctx->graph16)
    if (g) { cudaGraphExecDestroy(g); g = nullptr; }
  ctx->graphs_stale = false;
}

static const char* kErrStr[] = {"ok", "invalid argument", "CUDA error", "out of device memory", "non-finite value",
                                "device wait timed out", "invalid state", "unsupported", "no CUDA device",
                                "input exceeds the fixed scratch size of the no-allocation entry point"};

#define CK(call)                                                                           \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess) {                                                               \
      if (ctx) ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);              \
      return e_ == cudaErrorMemoryAllocation ? DTMX_ERR_OOM : DTMX_ERR_CUDA;               \
    }                                                                                      \
  } while (0)

// is this request the one that dtmx_fail_next asked to refuse?
static bool refuse(dtmx_ctx* ctx, int what) { return ctx->fail_in[what] >= 0 && ctx->fail_in[what]-- == 0; }

// A launch; early: it may start its set-up before the kernel ahead of it on the
// stream has finished (pdl_wait in the kernel).  Captured into graphs like any
// other.  A context takes early launches up to 2^23 cells (kEarlyCells) and
// outside a batch, where the waiting CTAs take room from the other contexts
// (23.2 -> 23.7 ms).  Measured without and with them, us a step, a Drude sphere with
// TF/SF at order 2 / a gyrotropic layer / order 4 with TF/SF: 1 M cells 50.9 and 48.6 / 37.2 and
// 37.4 / 58.7 and 55.9; 8.0 M 163.5 and 162.7 / 174.8 and 177.3 / 223.6 and 222.0; 10.1 M 179.2 and
// 182.4 / 199.0 and 202.1 / 245.3 and 242.0; 16.8 M 237.7 and 253.9 / 267.7 and 271.5 / 326 and 324; a
// plain grid gains 1 to 2 % up to 1 M cells and nothing above.
// A launch that failed is kept in the context until launched() reports it.
template <class... P, class... A>
static cudaError_t launch(dtmx_ctx* ctx, bool early, void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid; c.blockDim = block; c.dynamicSmemBytes = smem; c.stream = st;
  c.attrs = at; c.numAttrs = early ? 1 : 0;
  const cudaError_t e = refuse(ctx, DTMX_FAIL_LAUNCH) ? cudaErrorLaunchOutOfResources : cudaLaunchKernelEx(&c, k, P(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (ctx->launch_err == cudaSuccess) ctx->launch_err = e;
  }
  return e;
}

static int fail(dtmx_ctx* ctx, int code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  return code;
}

// have all kernels been launched since the last call?
static int launched(dtmx_ctx* ctx) {
  const cudaError_t e = ctx->launch_err;
  ctx->launch_err = cudaSuccess;
  return e == cudaSuccess ? DTMX_OK : fail(ctx, DTMX_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
}

static int copy_out(dtmx_ctx* ctx, void* host, const void* devp, size_t bytes) {
  CK(copy_to_host(ctx->dev, ctx->stream, host, devp, bytes));
  return DTMX_OK;
}

// ---- parkable device memory (no reference counterpart) -----------------------
struct VmmApi {
  PFN_cuMemGetAllocationGranularity_v10020 gran = nullptr;
  PFN_cuMemAddressReserve_v10020 reserve = nullptr;
  PFN_cuMemAddressFree_v10020 vfree = nullptr;
  PFN_cuMemCreate_v10020 create = nullptr;
  PFN_cuMemRelease_v10020 release = nullptr;
  PFN_cuMemMap_v10020 map = nullptr;
  PFN_cuMemUnmap_v10020 unmap = nullptr;
  PFN_cuMemSetAccess_v10020 access = nullptr;
  bool ok = false;
};
static const VmmApi& vmm_api() {
  static const VmmApi api = [] {
    VmmApi v;
    auto get = [](const char* name, void** q) {
      cudaDriverEntryPointQueryResult qr;
      return cudaGetDriverEntryPoint(name, q, cudaEnableDefault, &qr) == cudaSuccess && qr == cudaDriverEntryPointSuccess;
    };
    v.ok = get("cuMemGetAllocationGranularity", (void**)&v.gran) && get("cuMemAddressReserve", (void**)&v.reserve) &&
           get("cuMemAddressFree", (void**)&v.vfree) && get("cuMemCreate", (void**)&v.create) &&
           get("cuMemRelease", (void**)&v.release) && get("cuMemMap", (void**)&v.map) &&
           get("cuMemUnmap", (void**)&v.unmap) && get("cuMemSetAccess", (void**)&v.access);
    return v;
  }();
  return api;
}
static CUmemAllocationProp vmm_prop(int dev) {
  CUmemAllocationProp prop{};
  prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
  prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  prop.location.id = dev;
  return prop;
}
// Physical allocations released by dtmx_park, kept per device for the next
// dtmx_unpark of a block of the same size (up to a byte limit, 0 by default:
// released at once).  Creating and releasing physical memory costs more than
// mapping it, so contexts that take turns on a device reuse each other's.
struct HandlePool {
  std::mutex mu;
  std::multimap<size_t, CUmemGenericAllocationHandle> free;
  size_t bytes = 0;
  long long limit = 0;          // < 0: unlimited
};
constexpr int kPoolDevices = 64;
static HandlePool& handle_pool(int dev) {
  static HandlePool pools[kPoolDevices];
  return pools[dev >= 0 && dev < kPoolDevices ? dev : 0];
}
static bool pool_take(int dev, size_t size, CUmemGenericAllocationHandle* h) {
  HandlePool& P = handle_pool(dev);
  std::lock_guard<std::mutex> lk(P.mu);
  auto it = P.free.find(size);
  if (it == P.free.end()) return false;
  *h = it->second;
  P.free.erase(it);
  P.bytes -= size;
  return true;
}
// keeps the handle (true) or leaves it to the caller to release (false)
static bool pool_put(int dev, size_t size, CUmemGenericAllocationHandle h) {
  HandlePool& P = handle_pool(dev);
  std::lock_guard<std::mutex> lk(P.mu);
  if (P.limit >= 0 && P.bytes + size > (size_t)P.limit) return false;
  P.free.insert({size, h});
  P.bytes += size;
  return true;
}
// physical memory for block b, mapped read-write at its reserved address
static CUresult vmm_back(int dev, VmmBlock& b) {
  const VmmApi& A = vmm_api();
  const CUmemAllocationProp prop = vmm_prop(dev);
  CUresult r = CUDA_SUCCESS;
  if (!pool_take(dev, b.size, &b.h) && (r = A.create(&b.h, b.size, &prop, 0)) != CUDA_SUCCESS) return r;
  if ((r = A.map(b.va, b.size, 0, b.h, 0)) != CUDA_SUCCESS) { A.release(b.h); return r; }
  CUmemAccessDesc acc{};
  acc.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
  acc.location.id = dev;
  acc.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
  if ((r = A.access(b.va, b.size, &acc, 1)) != CUDA_SUCCESS) { A.unmap(b.va, b.size); A.release(b.h); }
  return r;
}

// the caller captures the context's stream: no allocation, no wait
static bool capturing(const dtmx_ctx* ctx) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
}

// Calls that use a context's second set hold it while they run (again within
// the same thread: a batch holds all of its contexts).
struct Running {
  dtmx_ctx* c;
  explicit Running(dtmx_ctx* ctx) : c(ctx && ctx->runner.load() != std::this_thread::get_id() ? ctx : nullptr) {
    if (!c) return;
    c->run.lock();
    c->runner = std::this_thread::get_id();
  }
  ~Running() {
    if (!c) return;
    c->runner = std::thread::id();
    c->run.unlock();
  }
  Running(Running&& o) : c(o.c) { o.c = nullptr; }
};
// the contexts whose automatic choice has made a second set
struct Lenders {
  std::mutex mu;
  std::vector<dtmx_ctx*> list;
};
static Lenders& lenders() {
  static Lenders l;
  return l;
}
static bool fused_give_back(dtmx_ctx* ctx);
// Memory for a request of ctx that failed: the second set of this context (own: the
// request is not made in the middle of a step that uses it), else that of
// another one on the device that no other thread is using.  False: there is none.
static bool free_a_set(dtmx_ctx* ctx, bool own) {
  cudaGetLastError();
  if (ctx->spare_others) return false;
  if (own) {
    const Running running(ctx);
    if (fused_give_back(ctx)) return true;
  }
  Lenders& L = lenders();
  std::lock_guard<std::mutex> lk(L.mu);
  for (dtmx_ctx* h : L.list) {
    if (h == ctx || h->dev != ctx->dev) continue;
    const bool mine = h->runner.load() == std::this_thread::get_id();
    if (!mine && !h->run.try_lock()) continue;
    const bool got = fused_give_back(h);
    if (!mine) h->run.unlock();
    if (got) return true;
  }
  return false;
}

// device memory beside the context's own arrays (which dalloc makes); *p is nullptr without it
template <class T>
static cudaError_t dev_malloc(dtmx_ctx* ctx, T** p, size_t bytes, bool own = true) {
  *p = nullptr;
  cudaError_t e = refuse(ctx, DTMX_FAIL_ALLOC) ? cudaErrorMemoryAllocation : cudaMalloc((void**)p, bytes);
  while (e == cudaErrorMemoryAllocation && free_a_set(ctx, own)) e = cudaMalloc((void**)p, bytes);
  if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); *p = nullptr; }
  return e;
}

static bool vmm_back_or_free(dtmx_ctx* ctx, VmmBlock& b) {
  CUresult r = vmm_back(ctx->dev, b);
  while (r == CUDA_ERROR_OUT_OF_MEMORY && free_a_set(ctx, false)) r = vmm_back(ctx->dev, b);
  return r == CUDA_SUCCESS;
}

// an array of the context (made before the first step or in a step: its own second set stays)
template <class T>
static int dalloc(dtmx_ctx* ctx, T** p, size_t count, bool fixed = false) {
  if (ctx->cfg.parkable) {
    if (refuse(ctx, DTMX_FAIL_ALLOC)) return fail(ctx, DTMX_ERR_OOM, "device memory");
    const VmmApi& A = vmm_api();
    if (!A.ok) return fail(ctx, DTMX_ERR_CUDA, "CUDA virtual memory management is unavailable");
    const CUmemAllocationProp prop = vmm_prop(ctx->dev);
    size_t g = 0;
    if (A.gran(&g, &prop, CU_MEM_ALLOC_GRANULARITY_MINIMUM) != CUDA_SUCCESS || g == 0)
      return fail(ctx, DTMX_ERR_CUDA, "allocation granularity");
    VmmBlock b;
    const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
    b.size = (bytes + g - 1) / g * g;
    if (A.reserve(&b.va, b.size, 0, 0, 0) != CUDA_SUCCESS) return fail(ctx, DTMX_ERR_OOM, "address reservation");
    if (!vmm_back_or_free(ctx, b)) { A.vfree(b.va, b.size); return fail(ctx, DTMX_ERR_OOM, "device memory"); }
    b.fixed = fixed;
    ctx->vmm.push_back(b);
    CK(cudaMemsetAsync((void*)b.va, 0, b.size, ctx->stream));
    *p = (T*)b.va;
    return DTMX_OK;
  }
  void* q = nullptr;
  cudaError_t e = dev_malloc(ctx, &q, std::max<size_t>(count, 1) * sizeof(T), false);
  if (e != cudaSuccess) {
    ctx->err = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? DTMX_ERR_OOM : DTMX_ERR_CUDA;
  }
  e = cudaMemsetAsync(q, 0, std::max<size_t>(count, 1) * sizeof(T), ctx->stream);
  if (e != cudaSuccess) { ctx->err = cudaGetErrorString(e); return DTMX_ERR_CUDA; }
  ctx->allocs.push_back(q);
  *p = (T*)q;
  return DTMX_OK;
}

extern "C" int dtmx_version(void) { return DTMX_ABI_VERSION; }
extern "C" const char* dtmx_error_string(int code) {
  if (code < 0 || code > 9) return "unknown";
  return kErrStr[code];
}
extern "C" const char* dtmx_last_error(const dtmx_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

// ---------------------------------------------------------------- boundaries
static void setup_grid(dtmx_ctx* ctx) {
  Grid& g = ctx->P.g;
  const dtmx_config& c = ctx->cfg;
  int n[3] = {c.nx, c.ny, c.nz};
  for (int a = 0; a < 3; a++) g.n[a] = n[a];
  g.sy = ctx->nzp;
  g.sx = (long long)c.ny * ctx->nzp;
  for (int a = 0; a < 3; a++)
    for (int s = 0; s < 2; s++) { g.btype[a][s] = 0; g.bsE[a][s] = 1; g.bsH[a][s] = 1; }
  g.box = c.geometry == DTMX_GEOM_BOX;
  if (c.geometry == DTMX_GEOM_BOX) {
    for (int a = 0; a < 3; a++) { g.bplane[a][0] = -1; g.bplane[a][1] = 2 * n[a]; }
  } else {
    // x: isOutS zero planes (defs.h:40); y: I-kernel free reflection at 0 with H odd
    // (genAlg.py:166-168) and X-kernel even mirror at 6*Na-3 (genAlg.py:9,36);
    // z: Vrefl even mirrors at 0 and 2*Nv-1 (defs.h:76-81).
    g.bplane[0][0] = 3; g.bplane[0][1] = 2 * n[0] - 3;
    g.btype[1][0] = 1; g.bplane[1][0] = 0; g.bsH[1][0] = -1;
    g.btype[1][1] = 1; g.bplane[1][1] = 2 * n[1] - 3;
    g.btype[2][0] = 1; g.bplane[2][0] = 0;
    g.btype[2][1] = 1; g.bplane[2][1] = 2 * n[2] - 1;
  }
  for (int comp = 0; comp < 6; comp++)
    for (int a = 0; a < 3; a++) {
      int lo = 0, hi = n[a] - 1;
      for (; lo <= hi; lo++) {
        int H = 2 * lo + comp_off(comp, a);
        if (g.btype[a][0] == 0 ? H > g.bplane[a][0] : H >= g.bplane[a][0]) break;
      }
      for (; hi >= lo; hi--) {
        int H = 2 * hi + comp_off(comp, a);
        if (g.btype[a][1] == 0 ? H < g.bplane[a][1] : H <= g.bplane[a][1]) break;
      }
      g.live_lo[comp][a] = lo;
      g.live_hi[comp][a] = hi;
    }
  for (int a = 0; a < 3; a++) {
    g.all_lo[a] = 0; g.all_hi[a] = n[a] - 1;
    for (int comp = 0; comp < 6; comp++) {
      g.all_lo[a] = std::max(g.all_lo[a], g.live_lo[comp][a]);
      g.all_hi[a] = std::min(g.all_hi[a], g.live_hi[comp][a]);
    }
  }
}

// Does the (plane i, y tile ty, z tile tz) streaming tile intersect the design region?
static bool design_touches(const dtmx_ctx* ctx, int i, int ty, int tz) {
  const Params& P = ctx->P;
  if (!P.des_on) return false;
  return i >= P.des_lo[0] && i < P.des_lo[0] + P.des_n[0] && ty * TYT < P.des_lo[1] + P.des_n[1] &&
         ty * TYT + TYT > P.des_lo[1] && tz * TZ < P.des_lo[2] + P.des_n[2] && tz * TZ + TZ > P.des_lo[2];
}

// ---------------------------------------------------------------- TMA descriptors
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &qr) == cudaSuccess &&
        qr == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)q;
  }
  return fn;
}

// 3-D map over a padded field (or material) array: dims (nz, ny, nx), box (bz, by, 1)
static int make_map(dtmx_ctx* ctx, CUtensorMap* map, void* base, bool bytes, int bz, int by) {
  auto fn = encode_fn();
  if (!fn) return fail(ctx, DTMX_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
  const dtmx_config& c = ctx->cfg;
  const size_t es = bytes ? 1 : 4;
  cuuint64_t dims[3] = {(cuuint64_t)c.nz, (cuuint64_t)c.ny, (cuuint64_t)c.nx};
  cuuint64_t strides[2] = {(cuuint64_t)ctx->nzp * es, (cuuint64_t)ctx->nzp * c.ny * es};
  cuuint32_t box[3] = {(cuuint32_t)bz, (cuuint32_t)by, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, bytes ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(ctx, DTMX_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return DTMX_OK;
}

static int build_maps(dtmx_ctx* ctx) {
  const int R = ctx->cfg.order / 2;
  // source tiles: A and C components carry R (below) + R-1 (above) halo rows for
  // the H step and R-1 + R for the E step; B components no halo rows
  const int rows_h = TYT + 2 * R - 1, rows_e = TYT + 2 * R - 1;
  const int rows[6] = {rows_h, TYT, rows_h, rows_e, TYT, rows_e};
  int rc;
  for (int comp = 0; comp < 6; comp++) {
    if ((rc = make_map(ctx, &ctx->maps.src[comp], ctx->P.f[comp], false, TZ + 8, rows[comp]))) return rc;
    if ((rc = make_map(ctx, &ctx->maps.own[comp], ctx->P.f[comp], false, TZ, TYT))) return rc;
  }
  for (int comp = 0; comp < 3; comp++)
    if ((rc = make_map(ctx, &ctx->maps.mat[comp], ctx->d_mat[comp], true, TZ, TYT))) return rc;
  return DTMX_OK;
}

// Reference PMLgamma_func (DTmxw.cu:220-229).
static double ref_gamma(int i, int N, double dstep, double vmax) {
  if (i >= N - 3) return 0.0;
  if (i < 0) i = 0;
  N -= 3;
  const double att = 4.0;
  const double smax = vmax * std::log(10000.0) * ((att + 1.0) / (2.0 * (N * dstep * 0.5)));
  const double xmax = std::pow(smax, 1.0 / att);
  const double x = xmax - i * (xmax / N);
  return std::pow(x, att);
}

static int setup_absorber(dtmx_ctx* ctx) {
  const dtmx_config& c = ctx->cfg;
  Absorb& ab = ctx->P.ab;
  ab.kind = c.absorber;
  const int n[3] = {c.nx, c.ny, c.nz};
  const double d[3] = {c.dx, c.dy, c.dz};
  std::vector<float> t0[3], t1[3], t2[3];
  for (int a = 0; a < 3; a++) {
    const int H = 2 * n[a] + 2;
    t0[a].assign(H, 1.f); t1[a].assign(H, 0.f); t2[a].assign(H, 1.f);
    ab.L[a][0] = ab.L[a][1] = 0;
  }
  if (c.absorber == DTMX_ABS_CPML) {
    const double m = c.cpml_m > 0 ? c.cpml_m : 3.0;
    const double fac = c.cpml_sigma_factor > 0 ? c.cpml_sigma_factor : 1.0;
    const double kmax = c.cpml_kappa_max >= 1 ? c.cpml_kappa_max : 1.0;
    const double amax = c.cpml_alpha_max;
    for (int a = 0; a < 3; a++)
      for (int s = 0; s < 2; s++) {
        const int L = c.pml[a][s];
        ab.L[a][s] = L;
        if (L <= 0) continue;
        const double smax = fac * 0.8 * (m + 1.0) / d[a];
        for (int h = 0; h < 2 * n[a]; h++) {
          double dep = s == 0 ? (2.0 * L - 1.0 - h) * 0.5 : (h - (2.0 * n[a] - 2.0 * L)) * 0.5;
          if (dep <= 0) continue;
          dep = std::min<double>(dep, L);
          const double r = dep / L;
          const double sg = smax * std::pow(r, m);
          const double kp = 1.0 + (kmax - 1.0) * std::pow(r, m);
          const double al = amax * (1.0 - r);
          const double b = std::exp(-(sg / kp + al) * c.dt);
          const double aa = sg > 0 ? sg / (sg * kp + kp * kp * al) * (b - 1.0) : 0.0;
          t0[a][h] = (float)b; t1[a][h] = (float)aa; t2[a][h] = (float)(1.0 / kp);
        }
      }
  } else if (c.absorber == DTMX_ABS_SPLIT_PML) {
    // setPMLcoeffs (DTmxw.cu:250-265): K2 = 1/(1+dt/2*gamma), K1 = 2*K2-1;
    // K1 = K2 = 1 where gamma = 0
    for (int a = 0; a < 3; a++) t1[a].assign(2 * n[a] + 2, 1.f);
    const double V = c.spml_vmax;
    // table lengths KNpmlx = 2 Npmlx NDT, KNpmly = 2 Npmly NDT, KNpmlz = 2 Npmlz (params.h:106-108);
    // the slabs are Npmlx/2 and Npmly/2 rags of NDT cells and the Npmlz/2 top layers
    const int KX = 4 * c.pml[0][0], KY = 4 * c.pml[1][0], KZ = 4 * c.pml[2][1];
    const int XS = 2 * c.pml[0][0] - 3;                // inPMLsync (defs.h:45): Npmlx/2*2*NDT - NDT
    ab.L[0][0] = c.pml[0][0]; ab.L[0][1] = c.pml[0][1];
    ab.L[1][0] = c.pml[1][0]; ab.L[1][1] = c.pml[1][1];
    ab.L[2][0] = 0;           ab.L[2][1] = c.pml[2][1];
    for (int h = 0; h < 2 * n[0] + 2; h++) {
      int i = -1;
      if (h < XS) i = h;
      else if (h >= 2 * n[0] - XS) i = h - 2 * n[0] + KX;
      if (i < 0 || i >= KX) continue;
      const double k2 = 1.0 / (1.0 + 0.5 * c.dt * ref_gamma(KX / 2 - std::abs(i - KX / 2) - 3, KX / 2 - 3, c.dx, V));
      t1[0][h] = (float)k2; t0[0][h] = (float)(2.0 * k2 - 1.0);
    }
    for (int h = 0; h < 2 * n[1] + 2; h++) {
      int i = -1;
      if (h < KY / 2) i = h;
      else if (h >= 2 * n[1] - KY / 2) i = h - 2 * n[1] + KY;
      if (i < 0 || i >= KY) continue;
      const double k2 = 1.0 / (1.0 + 0.5 * c.dt * ref_gamma(i < KY / 2 ? i : KY - i - 3, KY / 2, c.dy, V));
      t1[1][h] = (float)k2; t0[1][h] = (float)(2.0 * k2 - 1.0);
    }
    for (int h = 0; h < 2 * n[2] + 2; h++) {
      const int i = h - 2 * n[2] + KZ;                 // top face only (DTmxw.cu:262)
      if (i < KZ / 2 || i >= KZ) continue;
      const double k2 = 1.0 / (1.0 + 0.5 * c.dt * ref_gamma(KZ - i - 1, KZ / 2, c.dz, V));
      t1[2][h] = (float)k2; t0[2][h] = (float)(2.0 * k2 - 1.0);
    }
  }
  for (int a = 0; a < 3; a++) {
    const int H = 2 * n[a] + 2;
    float* q[3];
    for (int t = 0; t < 3; t++) {
      int rc = dalloc(ctx, &q[t], H, true);
      if (rc) return rc;
    }
    CK(cudaMemcpyAsync(q[0], t0[a].data(), H * 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(q[1], t1[a].data(), H * 4, cudaMemcpyHostToDevice, ctx->stream));
    CK(cudaMemcpyAsync(q[2], t2[a].data(), H * 4, cudaMemcpyHostToDevice, ctx->stream));
    ab.c0[a] = q[0]; ab.c1[a] = q[1]; ab.c2[a] = q[2];
    const size_t th = (size_t)(ab.L[a][0] + ab.L[a][1]);
    for (int s = 0; s < 4; s++) ab.aux[a][s] = nullptr;
    if (!th || c.absorber == DTMX_ABS_NONE) continue;
    const size_t cnt = th * (ctx->ncell / (size_t)n[a]);
    if (cnt >= (size_t)INT32_MAX) return fail(ctx, DTMX_ERR_UNSUPPORTED, "absorber slab of more than 2^31 values");
    for (int s = 0; s < 4; s++) {
      int rc = dalloc(ctx, &ab.aux[a][s], cnt);
      if (rc) return rc;
    }
    // sync the coefficient vectors (host memory) before they go out of scope
    CK(cudaStreamSynchronize(ctx->stream));
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return DTMX_OK;
}

static int upload_mattable(dtmx_ctx* ctx) {
  dtmx_ctx* c = ctx;
  CK(cudaMemcpyAsync(c->d_mt, &c->h_mt, sizeof(MatTable), cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return DTMX_OK;
}

extern "C" int dtmx_create(const dtmx_config* cfg, dtmx_ctx** out) {
  if (!cfg || !out) return DTMX_ERR_INVALID;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return DTMX_ERR_NODEVICE;
  const dtmx_config& c = *cfg;
  if (c.nx < 8 || c.ny < 8 || c.nz < 8) return DTMX_ERR_INVALID;
  if (c.order != 2 && c.order != 4) return DTMX_ERR_INVALID;
  if (!(c.dx > 0 && c.dy > 0 && c.dz > 0 && c.dt > 0)) return DTMX_ERR_INVALID;
  // Courant limits: 1 for the Yee stencil, 6/7 for the (27,-1)/24 stencil (DTmxw.cu:332)
  const double cn = c.dt * std::sqrt(1 / (c.dx * c.dx) + 1 / (c.dy * c.dy) + 1 / (c.dz * c.dz));
  if (cn > (c.order == 4 ? 6.0 / 7.0 : 1.0)) return DTMX_ERR_INVALID;
  if (c.geometry != DTMX_GEOM_BOX && c.geometry != DTMX_GEOM_REFERENCE) return DTMX_ERR_INVALID;
  if (c.absorber == DTMX_ABS_CPML && c.geometry != DTMX_GEOM_BOX) return DTMX_ERR_UNSUPPORTED;
  if (c.absorber == DTMX_ABS_SPLIT_PML && c.geometry != DTMX_GEOM_REFERENCE) return DTMX_ERR_UNSUPPORTED;
  if (c.geometry == DTMX_GEOM_REFERENCE && (c.nx % 3 || c.ny % 3)) return DTMX_ERR_INVALID;  // DTmxw.cu:330-331
  // split PML: whole rags along x and y on both faces, the top z face only (Npmlx/2, Npmly/2 rags, Npmlz/2 layers)
  if (c.absorber == DTMX_ABS_SPLIT_PML &&
      (c.pml[0][0] != c.pml[0][1] || c.pml[1][0] != c.pml[1][1] || c.pml[0][0] % 3 || c.pml[1][0] % 3 ||
       c.pml[0][0] < 3 || c.pml[1][0] < 3 || c.pml[2][0] != 0 || c.pml[2][1] < 2))
    return DTMX_ERR_INVALID;
  const int n[3] = {c.nx, c.ny, c.nz};
  for (int a = 0; a < 3; a++)
    for (int s = 0; s < 2; s++)
      if (c.pml[a][s] < 0 || c.pml[a][0] + c.pml[a][1] > n[a] - 4) return DTMX_ERR_INVALID;

  dtmx_ctx* ctx = new dtmx_ctx();
  ctx->cfg = c;
  if (cudaGetDevice(&ctx->dev) != cudaSuccess) { delete ctx; return DTMX_ERR_CUDA; }
  if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) { delete ctx; return DTMX_ERR_CUDA; }
  read_slots_hold();
  ctx->nzp = (c.nz + 31) / 32 * 32;
  ctx->ncell = (size_t)c.nx * c.ny * c.nz;
  ctx->nstore = (size_t)c.nx * c.ny * ctx->nzp;
  ctx->early = ctx->ncell <= kEarlyCells;
  setup_grid(ctx);
  int rc = DTMX_OK;
  // 64 floats of slack: aligned 16-byte tile rows may read up to 3 floats past the last node
  for (int comp = 0; comp < 6 && !rc; comp++) rc = dalloc(ctx, &ctx->P.f[comp], ctx->nstore + 64);
  if (!rc) rc = setup_absorber(ctx);
  if (!rc) rc = dalloc(ctx, &ctx->d_mt, 1, true);
  if (!rc) rc = dalloc(ctx, &ctx->d_step, 1);
  if (!rc) rc = dalloc(ctx, &ctx->d_flag, 1);
  if (!rc) rc = dalloc(ctx, &ctx->d_ticket, 1);
  if (!rc) rc = dalloc(ctx, &ctx->d_err, 1);
  for (int comp = 0; comp < 3 && !rc; comp++) rc = dalloc(ctx, &ctx->d_mat[comp], ctx->nstore + 64, true);
  if (!rc) rc = build_maps(ctx);
  ctx->P.ntz = (c.nz + TZ - 1) / TZ;
  ctx->P.nty = (c.ny + TYT - 1) / TYT;
  if (!rc) rc = dalloc(ctx, &ctx->d_umat, (size_t)c.nx * ctx->P.nty * ctx->P.ntz, true);   // zeros: material 0 everywhere
  if (rc) { *out = ctx; return rc; }
  ctx->P.umat = ctx->d_umat;
  ctx->P.err = ctx->d_err;
  ctx->P.wait_limit = kWaitPolls;
  for (int comp = 0; comp < 3; comp++) ctx->P.mat[comp] = ctx->d_mat[comp];
  ctx->P.cdt[0] = (float)(c.dt / c.dx); ctx->P.cdt[1] = (float)(c.dt / c.dy); ctx->P.cdt[2] = (float)(c.dt / c.dz);
  // default material 0: vacuum
  dtmx_material vac{};
  vac.eps[0] = vac.eps[1] = vac.eps[2] = 1.0;
  ctx->mats[0] = vac;
  for (int comp = 0; comp < 3; comp++) ctx->h_mt.inv_eps[0][comp] = 1.f;
  ctx->P.mt = ctx->d_mt;
  rc = upload_mattable(ctx);
  if (rc) { *out = ctx; return rc; }
  ctx->probe_cap = c.probe_capacity > 0 ? c.probe_capacity : 4096;
  *out = ctx;
  return DTMX_OK;
}

static void dft_free(DftHost& h);
static void mon_free(MonTable& m) {
  cudaFree(m.tab); cudaFree(m.map); cudaFree(m.unit);
  m = MonTable{};
}

extern "C" void dtmx_destroy(dtmx_ctx* ctx) {
  if (!ctx) return;
  if (ctx->lendable) {
    std::lock_guard<std::mutex> lk(lenders().mu);
    auto& l = lenders().list;
    l.erase(std::find(l.begin(), l.end(), ctx));
  }
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  for (auto& g : ctx->graph16)
    if (g) cudaGraphExecDestroy(g);
  for (void* p : ctx->allocs) cudaFree(p);
  for (auto& b : ctx->vmm) {
    const VmmApi& A = vmm_api();
    if (!ctx->parked) { A.unmap(b.va, b.size); A.release(b.h); }
    A.vfree(b.va, b.size);
    if (b.host) cudaFreeHost(b.host);
  }
  cudaFree(ctx->dense);
  for (auto& d : ctx->dfts) dft_free(d);
  for (auto& fx : ctx->fluxes) cudaFree(fx.d_out);
  for (MonTable* m : {&ctx->mon, &ctx->objmon}) mon_free(*m);
  dft_free(ctx->obj);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  read_slots_drop();
  delete ctx;
}

// ---------------------------------------------------------------- materials
// DispStruct::set (dispersion.cpp:41-82), coefficients in double then stored in float.
static void disp_coeffs(const dtmx_material& M, double dt, MatTable& t, int mi) {
  double alpha[MAXPOLE], ksi[MAXPOLE], zetp[MAXPOLE], zetm[MAXPOLE], zet[MAXPOLE];
  double zms = 0, zps = 0, zs = 0;
  for (int i = 0; i < M.npoles; i++) {
    const double Deps = M.pole[i][0], wp = M.pole[i][1], gp = M.pole[i][2], gp_ = M.pole[i][3];
    const double a0 = Deps * wp * wp, a1 = Deps * gp_;
    const double b0 = M.pole_kind[i] == DTMX_POLE_DRUDE ? 0.0 : wp * wp, b1 = 2 * gp;
    alpha[i] = (4 - 2 * b0 * dt * dt) / (b1 * dt + 2);
    ksi[i] = (b1 * dt - 2) / (b1 * dt + 2);
    zetp[i] = (a0 * dt * dt + 2 * a1 * dt) / (b1 * dt + 2);
    zetm[i] = (-a0 * dt * dt + 2 * a1 * dt) / (b1 * dt + 2);
    zet[i] = -(4 * a1 * dt) / (b1 * dt + 2);
    zms += zetm[i]; zps += zetp[i]; zs += zet[i];
  }
  const double den = 2 * M.eps_inf + M.sigma * dt + zps;
  const double C1 = -zms / den, C2 = (2 * M.eps_inf - M.sigma * dt - zs) / den, C3 = 2 * dt / den;
  for (int xc = 0; xc < 3; xc++) {
    for (int i = 0; i < M.npoles; i++) {
      t.kJ[mi][xc][i][0] = (float)alpha[i]; t.kJ[mi][xc][i][1] = (float)ksi[i];
      t.kJ[mi][xc][i][2] = (float)(zetp[i] / dt); t.kJ[mi][xc][i][3] = (float)(zetm[i] / dt);
      t.kJ[mi][xc][i][4] = (float)(zet[i] / dt);
      t.kEJ[mi][xc][i][0] = (float)(C3 * 0.5 * (1 + alpha[i])); t.kEJ[mi][xc][i][1] = (float)(C3 * 0.5 * ksi[i]);
    }
    t.kE[mi][xc][0] = (float)C1; t.kE[mi][xc][1] = (float)C2; t.kE[mi][xc][2] = (float)(C3 / dt);
  }
}

static inline size_t store_index(const dtmx_ctx* ctx, int i, int j, int k) {
  return ((size_t)i * ctx->cfg.ny + j) * ctx->nzp + k;
}

// Per (plane, y tile, z tile): the common non-dispersive material of all
// three E components, -1 if mixed, dispersive, gyrotropic or in the design
// region (selects the simple path of the field kernels).
static int upload_umat(dtmx_ctx* ctx) {
  const dtmx_config& c = ctx->cfg;
  const int nty = ctx->P.nty, ntz = ctx->P.ntz;
  const bool have = !ctx->h_mat[0].empty();
  std::vector<signed char> um((size_t)c.nx * nty * ntz);
  for (int i = 0; i < c.nx; i++)
    for (int ty = 0; ty < nty; ty++)
      for (int tz = 0; tz < ntz; tz++) {
        int m0 = have ? -2 : 0;
        for (int j = ty * TYT; have && j < std::min(c.ny, ty * TYT + TYT) && m0 != -1; j++)
          for (int comp = 0; comp < 3 && m0 != -1; comp++) {
            const uint8_t* row = ctx->h_mat[comp].data() + store_index(ctx, i, j, 0);
            for (int k = tz * TZ; k < std::min(c.nz, tz * TZ + TZ); k++) {
              const int m = row[k];
              if (m0 == -2) m0 = m;
              // (a gyrotropic node takes the plain update with 1/eps_inf; its current is
              // subtracted by the post-pass, so a uniform gyrotropic tile stays uniform)
              if (m != m0 || ctx->mats[m].npoles > 0) { m0 = -1; break; }
            }
          }
        um[((size_t)i * nty + ty) * ntz + tz] = (signed char)(m0 < 0 || design_touches(ctx, i, ty, tz) ? -1 : m0);
      }
  CK(cudaMemcpyAsync(ctx->d_umat, um.data(), um.size(), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return DTMX_OK;
}

extern "C" int dtmx_set_materials(dtmx_ctx* ctx, const dtmx_material* table, int nmat, const uint8_t* idx_x,
                                  const uint8_t* idx_y, const uint8_t* idx_z) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !table || nmat < 1 || nmat > DTMX_MAX_MATERIALS || !idx_x) return fail(ctx, DTMX_ERR_INVALID, "bad material arguments");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "materials must be set before the first step");
  const uint8_t* src[3] = {idx_x, idx_y ? idx_y : idx_x, idx_z ? idx_z : idx_x};
  for (int m = 0; m < nmat; m++) {
    const dtmx_material& M = table[m];
    if (M.npoles < 0 || M.npoles > DTMX_MAX_POLES) return fail(ctx, DTMX_ERR_INVALID, "npoles out of range");
    if (M.npoles > 0 && !(M.eps_inf > 0)) return fail(ctx, DTMX_ERR_INVALID, "dispersive material needs eps_inf > 0");
    if (M.npoles == 0 && !(M.eps[0] > 0 && M.eps[1] > 0 && M.eps[2] > 0)) return fail(ctx, DTMX_ERR_INVALID, "eps must be > 0");
    if (M.gyro_wp < 0) return fail(ctx, DTMX_ERR_INVALID, "gyro_wp must be >= 0");
    if (M.gyro_wp > 0 && (M.npoles > 0 || !(M.eps_inf > 0)))
      return fail(ctx, DTMX_ERR_INVALID, "a gyrotropic material needs npoles = 0 and eps_inf > 0");
  }
  MatTable& t = ctx->h_mt;
  memset(&t, 0, sizeof(t));
  for (int m = 0; m < nmat; m++) {
    ctx->mats[m] = table[m];
    t.npoles[m] = table[m].npoles;
    for (int c = 0; c < 3; c++) t.inv_eps[m][c] = table[m].npoles > 0 ? -0.f : (float)(1.0 / table[m].eps[c]);
    if (table[m].npoles > 0) disp_coeffs(table[m], ctx->cfg.dt, t, m);
    if (table[m].gyro_wp > 0) {
      const double dt = ctx->cfg.dt;
      for (int c = 0; c < 3; c++) t.inv_eps[m][c] = (float)(1.0 / table[m].eps_inf);
      t.gA[m] = (float)std::exp(-table[m].gyro_gamma * dt);
      t.gC[m] = (float)std::cos(table[m].gyro_wc * dt);
      t.gS[m] = (float)std::sin(table[m].gyro_wc * dt);
      t.gB[m] = (float)(table[m].gyro_wp * table[m].gyro_wp * dt);
      t.gjc[m] = (float)(dt / table[m].eps_inf);
    }
  }
  ctx->nmat = nmat;
  const dtmx_config& c = ctx->cfg;
  int lo[3] = {c.nx, c.ny, c.nz}, hi[3] = {-1, -1, -1};
  for (int comp = 0; comp < 3; comp++) {
    ctx->h_mat[comp].assign(ctx->nstore, 0);
    for (int i = 0; i < c.nx; i++)
      for (int j = 0; j < c.ny; j++) {
        const uint8_t* row = src[comp] + ((size_t)i * c.ny + j) * c.nz;
        uint8_t* dst = ctx->h_mat[comp].data() + store_index(ctx, i, j, 0);
        for (int k = 0; k < c.nz; k++) {
          const uint8_t m = row[k];
          if (m >= nmat) return fail(ctx, DTMX_ERR_INVALID, "material index out of range");
          dst[k] = m;
          if (table[m].npoles > 0 || table[m].gyro_wp > 0) {
            const int v[3] = {i, j, k};
            for (int a = 0; a < 3; a++) { lo[a] = std::min(lo[a], v[a]); hi[a] = std::max(hi[a], v[a]); }
          }
        }
      }
    CK(cudaMemcpyAsync(ctx->d_mat[comp], ctx->h_mat[comp].data(), ctx->nstore, cudaMemcpyHostToDevice, ctx->stream));
    ctx->P.mat[comp] = ctx->d_mat[comp];
  }
  int rc = upload_mattable(ctx);
  if (rc) return rc;
  if ((rc = upload_umat(ctx))) return rc;
  Ade& A = ctx->P.ade;
  if (hi[0] >= 0) {
    size_t na = 1;
    for (int a = 0; a < 3; a++) { A.lo[a] = lo[a]; A.n[a] = hi[a] - lo[a] + 1; na *= A.n[a]; }
    int maxp = 0;
    bool gyro = false;
    for (int m = 0; m < nmat; m++) { maxp = std::max(maxp, table[m].npoles); gyro = gyro || table[m].gyro_wp > 0; }
    ctx->has_gyro = gyro;
    ctx->gcur = 0;
    for (int comp = 0; comp < 3 && gyro; comp++)
      for (int b = 0; b < 2; b++)
        if ((rc = dalloc(ctx, &A.Jg[b][comp], na))) return rc;
    for (int comp = 0; comp < 3; comp++) {
      if ((rc = dalloc(ctx, &A.Em[comp], na))) return rc;
      for (int q = 0; q < maxp; q++) {
        if ((rc = dalloc(ctx, &A.Jp[comp][q], na))) return rc;
        if ((rc = dalloc(ctx, &A.Jm[comp][q], na))) return rc;
      }
    }
  }
  CK(cudaStreamSynchronize(ctx->stream));
  return DTMX_OK;
}

static bool node_live(const dtmx_ctx* ctx, int comp, int i, int j, int k) {
  const Grid& g = ctx->P.g;
  return i >= g.live_lo[comp][0] && i <= g.live_hi[comp][0] && j >= g.live_lo[comp][1] && j <= g.live_hi[comp][1] &&
         k >= g.live_lo[comp][2] && k <= g.live_hi[comp][2];
}

extern "C" int dtmx_add_point_source(dtmx_ctx* ctx, const dtmx_point_source* s) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !s || s->comp < 0 || s->comp > 2) return fail(ctx, DTMX_ERR_INVALID, "bad point source");
  if (!node_live(ctx, s->comp, s->i, s->j, s->k)) return fail(ctx, DTMX_ERR_INVALID, "point source outside the live domain");
  if (!(s->tau > 0)) return fail(ctx, DTMX_ERR_INVALID, "point source tau must be > 0");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "sources must be added before the first step");
  PointSrcDev d;
  d.comp = s->comp;
  d.id = (long long)store_index(ctx, s->i, s->j, s->k);
  d.amp = s->amp; d.f0 = s->f0; d.tau = s->tau; d.t0 = s->t0;
  ctx->psrc.push_back(d);
  return DTMX_OK;
}

// inSF along one axis with the reference's float arithmetic (signal.hpp:153-160)
static void sf_range(double dstep, double bm, double bp, int hmax, int* lo, int* hi) {
  const float bmf = (float)bm, bpf = (float)bp, df = (float)dstep;
  *lo = 1; *hi = 0;
  bool first = true;
  for (int h = -8; h <= hmax + 8; h++) {
    const float sv = (float)((double)h * 0.5 * (double)df);
    if (sv > bmf && sv < bpf) { if (first) { *lo = h; first = false; } *hi = h; }
  }
}

extern "C" int dtmx_set_tfsf(dtmx_ctx* ctx, const dtmx_tfsf* s) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !s || (s->kind != DTMX_TFSF_DIPOLE && s->kind != DTMX_TFSF_PLANE_X)) return fail(ctx, DTMX_ERR_INVALID, "bad TF/SF source");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "TF/SF source must be set before the first step");
  const dtmx_config& c = ctx->cfg;
  // a slab of a larger grid: plane 0 is whole-grid cell xo of gnx
  const int xo = (int)s->x_origin;
  const int gnx = s->x_cells > 0 ? (int)s->x_cells : c.nx;
  if ((double)xo != s->x_origin || (s->x_cells > 0 && (double)gnx != s->x_cells) || xo < 0 || xo + c.nx > gnx ||
      (c.geometry != DTMX_GEOM_BOX && (xo != 0 || gnx != c.nx)))
    return fail(ctx, DTMX_ERR_INVALID, "TF/SF x_origin / x_cells do not place this grid inside a whole grid");
  TfsfDev& T = ctx->T;
  T = TfsfDev{};
  T.xo = xo;
  const double d[3] = {c.dx, c.dy, c.dz};
  const int n[3] = {c.nx, c.ny, c.nz};
  for (int a = 0; a < 3; a++) {
    sf_range(d[a], s->box_lo[a], s->box_hi[a], 2 * (a == 0 ? gnx : n[a]), &T.lo[a], &T.hi[a]);
    if (T.lo[a] > T.hi[a]) return fail(ctx, DTMX_ERR_INVALID, "TF/SF box contains no node");
    if (a == 0) { T.lo[0] -= 2 * xo; T.hi[0] -= 2 * xo; }
    // the correction shell (3 half cells around the surface) must stay inside the
    // live domain and clear of the absorber (along x: at the grid's uncut ends)
    const int clo = (T.lo[a] - 4) / 2 - 1, chi = (T.hi[a] + 4) / 2 + 1;
    const int alo = c.absorber == DTMX_ABS_NONE ? 0 : ctx->P.ab.L[a][0];
    const int ahi = c.absorber == DTMX_ABS_NONE ? 0 : ctx->P.ab.L[a][1];
    int llo = 0, lhi = n[a] - 1;
    for (int comp = 0; comp < 6; comp++) { llo = std::max(llo, ctx->P.g.live_lo[comp][a]); lhi = std::min(lhi, ctx->P.g.live_hi[comp][a]); }
    const bool lo_end = a != 0 || xo == 0, hi_end = a != 0 || xo + c.nx == gnx;
    if ((lo_end && clo < std::max(alo, llo) + 1) || (hi_end && chi > std::min(n[a] - 1 - ahi, lhi) - 1))
      return fail(ctx, DTMX_ERR_INVALID, "TF/SF box too close to the boundary or absorber");
  }
  T.active_cfg = 1;
  T.kind = s->kind;
  for (int a = 0; a < 3; a++) { T.ctr[a] = (s->box_lo[a] + s->box_hi[a]) * 0.5; T.hd[a] = d[a] * 0.5; }
  T.dt = c.dt; T.c = s->c; T.w = s->w; T.kenv = s->kenv; T.tstop = s->tstop;
  T.ntime = s->ntime > 0 ? s->ntime : 1;
  // correction jobs: per half step, component and curl term (axis a, source
  // component g), the nodes within 3 half cells of each face along a whose g
  // taps lie inside the box range on the other two axes
  for (int hs = 0; hs < 2; hs++) {
    T.njob[hs] = 0;
    for (int comp = hs * 3; comp < hs * 3 + 3; comp++) {
      int ax[2], gs[2];
      curl_terms(comp, ax[0], gs[0], ax[1], gs[1]);
      for (int term = 0; term < 2; term++) {
        const int a = ax[term], g = gs[term];
        if (s->kind == DTMX_TFSF_PLANE_X && g != 2 && g != 4) continue;
        for (int side = 0; side < 2; side++) {
          TfsfJob jb{};
          jb.c = comp;
          jb.a = a; jb.g = g; jb.sg = term == 0 ? 1 : -1;
          bool empty = false;
          for (int b = 0; b < 3; b++) {
            int X0, X1, o;
            if (b == a) { X0 = side ? T.hi[a] - 3 : T.lo[a] - 4; X1 = side ? T.hi[a] + 4 : T.lo[a] + 3; o = comp_off(comp, a); }
            else { X0 = T.lo[b]; X1 = T.hi[b]; o = comp_off(g, b); }
            // indices v with X0 <= 2v + o <= X1, clipped to the grid
            int v0 = (int)std::ceil((X0 - o) / 2.0), v1 = (int)std::floor((X1 - o) / 2.0);
            v0 = std::max(v0, 0); v1 = std::min(v1, n[b] - 1);
            if (b == a) {
              // along the curl axis keep only the indices where a tap of g actually
              // crosses the box surface (the other two axes agree for c and g)
              const int t0 = hs ? -2 : -1, qa = c.order == 4 ? 0 : 1, qb = c.order == 4 ? 3 : 2;
              auto crosses = [&](int v) {
                const int S = 2 * v + comp_off(comp, a);
                const bool sin_ = S >= T.lo[a] && S <= T.hi[a];
                for (int q = qa; q <= qb; q++) {
                  const int G = 2 * (v + t0 + q) + comp_off(g, a);
                  if ((G >= T.lo[a] && G <= T.hi[a]) != sin_) return true;
                }
                return false;
              };
              while (v0 <= v1 && !crosses(v0)) v0++;
              while (v1 >= v0 && !crosses(v1)) v1--;
            }
            if (v0 > v1) empty = true;
            jb.lo[b] = v0; jb.hi[b] = v1;
          }
          if (empty) continue;
          jb.cells = (long long)(jb.hi[0] - jb.lo[0] + 1) * (jb.hi[1] - jb.lo[1] + 1) * (jb.hi[2] - jb.lo[2] + 1);
          if (jb.cells >= (long long)INT32_MAX) return fail(ctx, DTMX_ERR_UNSUPPORTED, "TF/SF correction shell of more than 2^31 nodes");
          T.job[hs][T.njob[hs]++] = jb;
        }
      }
    }
  }
  if (s->kind == DTMX_TFSF_PLANE_X) {
    // the 1-D line spans the whole grid with 4096 cells beyond each end; plane 0
    // of this grid reads line cell xo + 4096, the source sits 10 cells before
    // the box's lower x face
    constexpr int kLinePad = 4096;
    T.line_M = kLinePad + xo;
    T.line_n = gnx + 2 * kLinePad;
    int rc;
    if (ctx->line_cap < T.line_n) {
      if ((rc = dalloc(ctx, &ctx->line_e, T.line_n))) return rc;
      if ((rc = dalloc(ctx, &ctx->line_h, T.line_n))) return rc;
      ctx->line_cap = T.line_n;
    }
    T.line_e = ctx->line_e; T.line_h = ctx->line_h;
    ctx->line_src = (T.lo[0] + 2 * xo - 1) / 2 - 10 + kLinePad;
  }
  ctx->tfsf = *s;
  ctx->has_tfsf = 1;
  CK(cudaStreamSynchronize(ctx->stream));
  return DTMX_OK;
}

extern "C" int dtmx_add_probe(dtmx_ctx* ctx, int comp, int i, int j, int k, int mode, int* id_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || comp < 0 || comp > 5 || (mode != DTMX_PROBE_NODE && mode != DTMX_PROBE_REFERENCE)) return fail(ctx, DTMX_ERR_INVALID, "bad probe");
  if (i < 0 || i >= ctx->cfg.nx || j < 0 || j >= ctx->cfg.ny || k < 0 || k >= ctx->cfg.nz) return fail(ctx, DTMX_ERR_INVALID, "probe outside the grid");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "probes must be added before the first step");
  ProbeDev p{comp, i, j, k, mode};
  ctx->probes.push_back(p);
  if (id_out) *id_out = (int)ctx->probes.size() - 1;
  return DTMX_OK;
}

extern "C" int dtmx_read_probes(dtmx_ctx* ctx, float* out, int max_samples, int* nsamples) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !out || max_samples < 0) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  const int every = ctx->cfg.probe_every > 0 ? ctx->cfg.probe_every : 1;
  const long long have = std::min<long long>(ctx->step / every, ctx->probe_cap);
  const int ns = (int)std::min<long long>(have, max_samples);
  CK(cudaStreamSynchronize(ctx->stream));
  if (ns > 0 && !ctx->probes.empty())
    CK(cudaMemcpy2D(out, (size_t)max_samples * 4, ctx->d_traces, (size_t)ctx->probe_cap * 4, (size_t)ns * 4,
                    ctx->probes.size(), cudaMemcpyDeviceToHost));
  if (nsamples) *nsamples = ns;
  return DTMX_OK;
}

static void dft_free(DftHost& h) {
  cudaFree(h.omega); cudaFree(h.acc); cudaFree(h.stage); cudaFree(h.sstep);
  h.omega = nullptr; h.acc = nullptr; h.stage = nullptr; h.sstep = nullptr;
}
// all four arrays of a DFT plane, or none of them
static bool dft_malloc(dtmx_ctx* ctx, DftHost& h, size_t nfreq, size_t nacc, size_t nstage) {
  if (dev_malloc(ctx, &h.omega, nfreq * sizeof(double)) == cudaSuccess && dev_malloc(ctx, &h.acc, nacc * sizeof(double2)) == cudaSuccess &&
      dev_malloc(ctx, &h.stage, nstage * sizeof(float)) == cudaSuccess && dev_malloc(ctx, &h.sstep, DFT_STAGE * sizeof(long long)) == cudaSuccess)
    return true;
  dft_free(h);
  return false;
}

extern "C" int dtmx_add_dft_patch(dtmx_ctx* ctx, int axis, int index, int lo1, int n1, int lo2, int n2, int comp_mask,
                                  int nfreq, const double* omegas, int* id_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || axis < 0 || axis > 2 || nfreq < 1 || nfreq > 64 || !omegas || (comp_mask & ~63) || !comp_mask)
    return fail(ctx, DTMX_ERR_INVALID, "bad DFT plane");
  const int n[3] = {ctx->cfg.nx, ctx->cfg.ny, ctx->cfg.nz};
  const int e1 = n[axis == 0 ? 1 : 0], e2 = n[axis == 2 ? 1 : 2];
  if (index < 0 || index >= n[axis]) return fail(ctx, DTMX_ERR_INVALID, "DFT plane index out of range");
  if (lo1 < 0 || n1 < 1 || lo1 + n1 > e1 || lo2 < 0 || n2 < 1 || lo2 + n2 > e2)
    return fail(ctx, DTMX_ERR_INVALID, "DFT patch outside the plane");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "DFT planes must be added before the first step");
  DftHost h{};
  h.d.axis = axis; h.d.index = index; h.d.comp_mask = comp_mask; h.d.nfreq = nfreq;
  h.d.lo1 = lo1; h.d.n1 = n1;
  h.d.lo2 = lo2; h.d.n2 = n2;
  h.ncomp = __builtin_popcount(comp_mask);
  const size_t nacc = (size_t)h.ncomp * nfreq * h.d.n1 * h.d.n2;
  const size_t nstage = (size_t)DFT_STAGE * h.ncomp * h.d.n1 * h.d.n2;
  if (!dft_malloc(ctx, h, nfreq, nacc, nstage)) return fail(ctx, DTMX_ERR_OOM, "DFT allocation");
  CK(cudaMemsetAsync(h.acc, 0, nacc * sizeof(double2), ctx->stream));
  CK(cudaMemcpyAsync(h.omega, omegas, nfreq * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  h.d.omega = h.omega; h.d.acc = h.acc; h.d.stage = h.stage; h.d.sstep = h.sstep;
  ctx->dfts.push_back(h);
  CK(cudaStreamSynchronize(ctx->stream));
  if (id_out) *id_out = (int)ctx->dfts.size() - 1;
  return DTMX_OK;
}

extern "C" int dtmx_add_dft_plane(dtmx_ctx* ctx, int axis, int index, int comp_mask, int nfreq, const double* omegas, int* id_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || axis < 0 || axis > 2) return fail(ctx, DTMX_ERR_INVALID, "bad DFT plane");
  const int n[3] = {ctx->cfg.nx, ctx->cfg.ny, ctx->cfg.nz};
  return dtmx_add_dft_patch(ctx, axis, index, 0, n[axis == 0 ? 1 : 0], 0, n[axis == 2 ? 1 : 2], comp_mask, nfreq, omegas,
                            id_out);
}

extern "C" int dtmx_add_flux_box(dtmx_ctx* ctx, const int lo[3], const int hi[3], int nfreq, const double* omegas,
                                 int* id_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !lo || !hi) return fail(ctx, DTMX_ERR_INVALID, "bad flux box");
  const int n[3] = {ctx->cfg.nx, ctx->cfg.ny, ctx->cfg.nz};
  const double ds[3] = {ctx->cfg.dx, ctx->cfg.dy, ctx->cfg.dz};
  for (int a = 0; a < 3; a++)
    if (lo[a] < 0 || hi[a] <= lo[a] || hi[a] + 1 >= n[a]) return fail(ctx, DTMX_ERR_INVALID, "flux box outside the grid");
  FluxHost fx{};
  fx.nfreq = nfreq;
  for (int a = 0; a < 3; a++) {
    // in-plane axes in (slow, fast) order and the tangential components
    const int s1 = a == 0 ? 1 : 0, s2 = a == 2 ? 1 : 2;
    const int b = (a + 1) % 3, c = (a + 2) % 3;
    const int mask = (1 << b) | (1 << c) | (1 << (3 + b)) | (1 << (3 + c));
    for (int side = 0; side < 2; side++) {
      int id = -1;
      const int rc = dtmx_add_dft_patch(ctx, a, side ? hi[a] : lo[a], lo[s1], hi[s1] - lo[s1], lo[s2], hi[s2] - lo[s2],
                                        mask, nfreq, omegas, &id);
      if (rc) return rc;
      fx.face[2 * a + side] = id;
      fx.sgn_area[2 * a + side] = (side ? 1.0 : -1.0) * ds[s1] * ds[s2];
      const int w = side ? hi[a] : lo[a];
      const int n1 = hi[s1] - lo[s1] + 1, n2 = hi[s2] - lo[s2] + 1;
      int eid = -1, hid = -1;
      int rc2 = dtmx_add_dft_patch(ctx, a, w, lo[s1], n1, lo[s2], n2, mask, nfreq, omegas, &eid);
      if (!rc2)
        rc2 = dtmx_add_dft_patch(ctx, a, w + 1, lo[s1], n1, lo[s2], n2, (1 << (3 + b)) | (1 << (3 + c)), nfreq,
                                 omegas, &hid);
      if (rc2) return rc2;
      fx.ffe[2 * a + side] = eid;
      fx.ffh[2 * a + side] = hid;
    }
  }
  if (dev_malloc(ctx, &fx.d_out, (size_t)6 * nfreq * sizeof(double)) != cudaSuccess)
    return fail(ctx, DTMX_ERR_OOM, "flux box allocation");
  ctx->fluxes.push_back(fx);
  if (id_out) *id_out = (int)ctx->fluxes.size() - 1;
  return DTMX_OK;
}

extern "C" int dtmx_flux_faces(dtmx_ctx* ctx, int id, int faces[6]) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || id < 0 || id >= (int)ctx->fluxes.size() || !faces) return fail(ctx, DTMX_ERR_INVALID, "bad flux box id");
  for (int q = 0; q < 6; q++) faces[q] = ctx->fluxes[id].face[q];
  return DTMX_OK;
}

// Tables of a set of DFT planes (made once: the planes are fixed from the first step on).
static int mon_build(dtmx_ctx* ctx, MonTable& m, const DftHost* h, int n) {
  mon_free(m);
  std::vector<DftDev> tab;
  std::vector<int2> map;
  std::vector<FlushUnit> unit;
  for (int q = 0; q < n; q++) {
    const DftDev& d = h[q].d;
    tab.push_back(d);
    const int nb = (int)(((long long)d.n1 * d.n2 + 255) / 256);
    for (int b = 0; b < nb; b++) map.push_back(make_int2(q, b));
    int slot = 0;
    for (int c = 0; c < 6; c++) {
      if (!(d.comp_mask & (1 << c))) continue;
      for (int f = 0; f < d.nfreq; f += DFT_FCHUNK)
        for (int b = 0; b < nb; b++) unit.push_back(FlushUnit{q, c, slot, f, b});
      slot++;
    }
  }
  if (tab.empty()) return DTMX_OK;
  if (dev_malloc(ctx, &m.tab, tab.size() * sizeof(DftDev)) != cudaSuccess || dev_malloc(ctx, &m.map, map.size() * sizeof(int2)) != cudaSuccess ||
      dev_malloc(ctx, &m.unit, unit.size() * sizeof(FlushUnit)) != cudaSuccess) {
    mon_free(m);
    return fail(ctx, DTMX_ERR_OOM, "DFT tables");
  }
  CK(cudaMemcpyAsync(m.tab, tab.data(), tab.size() * sizeof(DftDev), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(m.map, map.data(), map.size() * sizeof(int2), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(m.unit, unit.data(), unit.size() * sizeof(FlushUnit), cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  m.nmap = (int)map.size();
  m.nunit = (int)unit.size();
  return DTMX_OK;
}

// fold the staged samples of a set of planes into their accumulators
static void dft_flush(dtmx_ctx* ctx, MonTable& m) {
  if (m.nstaged == 0) return;
  const cudaError_t e = launch(ctx, false, dft_flush_kernel, m.nunit, 256, 0, ctx->stream, m.tab, m.unit, m.nstaged, ctx->cfg.dt);
  ctx->launches++;
  if (e == cudaSuccess || m.nstaged == DFT_STAGE) m.nstaged = 0;     // (a fold that did not start is made by the next one, while there is room)
}

extern "C" int dtmx_read_dft(dtmx_ctx* ctx, int id, double* out, size_t out_len) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || id < 0 || id >= (int)ctx->dfts.size() || !out) return fail(ctx, DTMX_ERR_INVALID, "bad DFT id");
  DftHost& h = ctx->dfts[id];
  const size_t n = (size_t)h.ncomp * h.d.nfreq * h.d.n1 * h.d.n2 * 2;
  if (out_len < n) return fail(ctx, DTMX_ERR_INVALID, "output buffer too small");
  dft_flush(ctx, ctx->mon);
  if (int rc = launched(ctx)) return rc;
  return copy_out(ctx, out, h.acc, n * sizeof(double));
}

extern "C" int dtmx_read_flux(dtmx_ctx* ctx, int id, double* out, size_t out_len) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || id < 0 || id >= (int)ctx->fluxes.size() || !out) return fail(ctx, DTMX_ERR_INVALID, "bad flux box id");
  FluxHost& fx = ctx->fluxes[id];
  const int nf = fx.nfreq;
  if (out_len < (size_t)7 * nf) return fail(ctx, DTMX_ERR_INVALID, "output buffer too small");
  dft_flush(ctx, ctx->mon);
  for (int q = 0; q < 6; q++) {
    DftHost& h = ctx->dfts[fx.face[q]];
    launch(ctx, false, flux_face_kernel, nf, FLUX_THREADS, 0, ctx->stream, h.d, fx.sgn_area[q], fx.d_out + (size_t)q * nf);
    ctx->launches++;
  }
  if (int rc = launched(ctx)) return rc;
  CK(cudaStreamSynchronize(ctx->stream));
  CK(cudaMemcpy(out, fx.d_out, (size_t)6 * nf * sizeof(double), cudaMemcpyDeviceToHost));
  for (int f = 0; f < nf; f++) {
    double t = 0.0;
    for (int q = 0; q < 6; q++) t += out[(size_t)q * nf + f];
    out[(size_t)6 * nf + f] = t;
  }
  return DTMX_OK;
}

extern "C" int dtmx_ntff(dtmx_ctx* ctx, int id, int ndir, const double* theta, const double* phi, const double* origin,
                         double* out, size_t out_len) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || id < 0 || id >= (int)ctx->fluxes.size() || ndir < 1 || !theta || !phi || !out)
    return fail(ctx, DTMX_ERR_INVALID, "bad far-field arguments");
  FluxHost& fx = ctx->fluxes[id];
  const int nf = fx.nfreq;
  if (out_len < (size_t)ndir * nf * 5) return fail(ctx, DTMX_ERR_INVALID, "output buffer too small");
  NtffFaces F{};
  const double ds[3] = {ctx->cfg.dx, ctx->cfg.dy, ctx->cfg.dz};
  dft_flush(ctx, ctx->mon);
  for (int q = 0; q < 6; q++) {
    F.f[q] = ctx->dfts[fx.ffe[q]].d;
    F.h[q] = ctx->dfts[fx.ffh[q]].d;
  }
  for (int a = 0; a < 3; a++) {
    F.ds[a] = ds[a];
    F.lo[a] = F.f[2 * a].index;
    F.hi[a] = F.f[2 * a + 1].index;
    // default origin: the centre of the E surface (box lo + 1/2 .. hi + 1/2)
    F.org[a] = origin ? origin[a] : (0.5 * (F.lo[a] + F.hi[a]) + 0.5) * ds[a];
  }
  double *dth = nullptr, *dph = nullptr, *dout = nullptr;
  const size_t nout = (size_t)ndir * nf * 5;
  if (dev_malloc(ctx, &dth, ndir * 8) != cudaSuccess || dev_malloc(ctx, &dph, ndir * 8) != cudaSuccess ||
      dev_malloc(ctx, &dout, nout * 8) != cudaSuccess) {
    cudaFree(dth); cudaFree(dph); cudaFree(dout);
    return fail(ctx, DTMX_ERR_OOM, "far-field allocation");
  }
  CK(cudaMemcpyAsync(dth, theta, ndir * 8, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemcpyAsync(dph, phi, ndir * 8, cudaMemcpyHostToDevice, ctx->stream));
  launch(ctx, false, ntff_kernel, dim3(ndir, nf), FLUX_THREADS, 0, ctx->stream, F, dth, dph, nf, dout);
  ctx->launches++;
  cudaError_t e = ctx->launch_err;
  ctx->launch_err = cudaSuccess;
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, dout, nout * 8, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(dth); cudaFree(dph); cudaFree(dout);
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("far field: ") + cudaGetErrorString(e));
  return DTMX_OK;
}

// ---------------------------------------------------------------- stepping
// How a streaming launch cuts the tile columns along x, one CTA a piece.
//   * One wave of the CTAs that fit, where that takes about a dozen planes a CTA:
//     small grids are bound by the latency of a CTA's walk, and a nearly empty last
//     wave costs as much as a full one (single sweep, 48^3: 9.4 us with pieces of one
//     plane, 26 with eight; per-step kernels, 64^3: 17.8 with four, 10.6 with one).
//   * With an absorber, in pieces of equal cost, not equal length: a plane next to a
//     slab costs about one interior plane more per slab axis, and on 128^3 in equal
//     pieces the busiest SM issued 1.43 times the average (single sweep 41.1 -> 36.3
//     us; per-step kernels 42.2 -> 37.4, 149x93x211 59.8 -> 50.0; adjoint sweep on
//     192x160x128 94 -> 86).  Such pieces serve one wave up to about 40 units (single
//     sweep, 192x160x128: 68.1 us in eight waves of equal pieces, 60.2 in one wave;
//     149x93x211 59.3 -> 52.5); above that several waves even out as well (384^3).
//     One wave has no slack for what the cost leaves out, nor for slots that other
//     kernels hold: the long pieces are not for the single sweep with a design region
//     (its tile-planes cost several others: the forward runs of a gradient on
//     192x160x128 18.8 -> 20.8 ms) or in a batch, and their launch waits for the
//     kernel ahead.  The single sweep's pieces below six planes stay equal: the lookup
//     ahead of the first copy costs them more than it evens out (96^3: 18.7 -> 20.7 us).
//     The order-4 per-step kernels stay at equal pieces (64.5 + 54.0 -> 75.1 + 55.3 us in
//     the reference geometry, 180x180x128; not measured on other grids).
//   * Otherwise several waves of equal pieces: of 6 to 32 planes for the single sweep
//     (192x160x128: 68 us with 6, 77 with 12; 384^3: 634 us with 32, 641 with 10, 669
//     with 64), 4 to 10 for the per-step kernels (384^3 712 us with 10, 830 with about 40).
// planes > 0: equal pieces of that many planes (dtmx_set_xchunk, dtmx_autotune).
static int tile_axes(const dtmx_ctx* ctx, int j0, int rows, int k0) {
  const Absorb& ab = ctx->P.ab;
  if (ab.kind == 0) return 0;
  const dtmx_config& c = ctx->cfg;
  return (j0 < ab.L[1][0] || j0 + rows > c.ny - ab.L[1][1] ? 1 : 0) + (k0 < ab.L[2][0] || k0 + TZ > c.nz - ab.L[2][1] ? 1 : 0);
}
// pieces of at most `budget` units: an interior plane is one, a piece's start two
static void work_cut(const dtmx_ctx* ctx, int rows, int budget, std::vector<int4>* out, long long* count) {
  const dtmx_config& c = ctx->cfg;
  const Absorb& ab = ctx->P.ab;
  constexpr int kStart = 2;
  std::vector<int> cuts[3];            // the cuts depend on the number of the column's slab axes alone
  for (int a = 0; a < 3; a++) {
    int cost = kStart, first = 0;
    cuts[a].push_back(0);
    for (int i = 0; i < c.nx; i++) {
      const int w = 1 + a + (ab.kind != 0 && (i < ab.L[0][0] || i >= c.nx - ab.L[0][1]) ? 1 : 0);
      if (i > first && (cost + w > budget || i - first >= FX_MAX)) { cuts[a].push_back(i); cost = kStart; first = i; }
      cost += w;
    }
    cuts[a].push_back(c.nx);
  }
  const int ntz = (c.nz + TZ - 1) / TZ, nty = (c.ny + rows - 1) / rows;
  size_t longest = 0;
  for (int a = 0; a < 3; a++) longest = std::max(longest, cuts[a].size() - 1);
  long long n = 0;
  // in order of their place along x, so that CTAs that start together share halos
  for (size_t q = 0; q < longest; q++)
    for (int ty = 0; ty < nty; ty++)
      for (int tz = 0; tz < ntz; tz++) {
        const std::vector<int>& cut = cuts[tile_axes(ctx, ty * rows, rows, tz * TZ)];
        if (q + 1 >= cut.size()) continue;
        n++;
        if (out) out->push_back(make_int4(tz, ty, cut[q], cut[q + 1]));
      }
  if (count) *count = n;
}
enum { WK_STREAM, WK_SWEEP, WK_ADJ };
constexpr int kOneWave = 40;            // most units of a piece in a single wave
// The plan of a launch; its table is made on first use, never while a stream is captured.
static int plan_work(dtmx_ctx* ctx, int kind, int rows, int per_sm, int planes, const WorkPlan** plan) {
  const dtmx_config& c = ctx->cfg;
  const int ntz = (c.nz + TZ - 1) / TZ, nty = (c.ny + rows - 1) / rows;
  const long long tiles = (long long)ntz * nty, fit = 148LL * per_sm;
  const bool many = ctx->early && !ctx->P.des_on;     // may take long pieces in one wave
  const std::array<int, 4> key{kind, rows, planes, many ? 1 : 0};
  auto it = ctx->work.find(key);
  if (it == ctx->work.end()) {
    WorkPlan w;
    std::vector<int4> v;
    bool keep = true;
    w.xchunk = planes;
    if (planes == 0) {
      const long long one = tiles <= fit ? (c.nx + fit / tiles - 1) / (fit / tiles) : c.nx;      // one wave of equal pieces
      int budget = kOneWave + 1;
      if (c.absorber != DTMX_ABS_NONE && rows == 16 && tiles <= fit && one >= (kind == WK_STREAM ? 5 : 6) && !(kind == WK_STREAM && c.order == 4) &&
          (kind != WK_SWEEP || one <= 12 || many)) {
        for (budget = 3; budget <= kOneWave; budget++) {
          long long n = 0;
          work_cut(ctx, rows, budget, nullptr, &n);
          if (n <= fit) break;
        }
      }
      int4* d = nullptr;
      if (budget <= kOneWave) {
        // no table while the caller captures the stream, nor without memory for one: equal pieces serve
        keep = !capturing(ctx);
        work_cut(ctx, rows, budget, &v, nullptr);
        if (keep && dalloc(ctx, &d, v.size(), true) != DTMX_OK) d = nullptr;
      }
      if (d) {
        CK(cudaMemcpyAsync(d, v.data(), v.size() * sizeof(int4), cudaMemcpyHostToDevice, ctx->stream));
        CK(cudaStreamSynchronize(ctx->stream));
        w.table = true;
        w.alone = kind == WK_SWEEP && one > 12;
        w.work.e = d;
        w.grid = dim3((unsigned)v.size());
      } else if (kind == WK_STREAM) {
        const long long chunks = std::max<long long>(1, (148LL * 8 * 3 + tiles - 1) / tiles), xc = (c.nx + chunks - 1) / chunks;
        w.xchunk = (int)(one <= 2 && c.order == 2 ? one : std::min<long long>(10, std::max<long long>(4, xc)));
      } else {
        const long long chunks = std::max<long long>(1, (8 * fit + tiles - 1) / tiles), xc = (c.nx + chunks - 1) / chunks;
        w.xchunk = (int)(one <= 12 ? one : std::min<long long>(32, std::max<long long>(6, xc)));
      }
    }
    if (!w.table) w.grid = dim3(ntz, nty, (c.nx + w.xchunk - 1) / w.xchunk);
    w.longest = std::min(w.xchunk, c.nx);
    for (const int4& e : v)
      if (w.table) w.longest = std::max(w.longest, e.w - e.z);
    if (!keep) {
      ctx->work_once = w;
      if (plan) *plan = &ctx->work_once;
      return DTMX_OK;
    }
    it = ctx->work.emplace(key, w).first;
  }
  if (plan) *plan = &it->second;
  return DTMX_OK;
}
static int plan_stream(dtmx_ctx* ctx, const WorkPlan** w) { return plan_work(ctx, WK_STREAM, TYT, ctx->cfg.order == 4 ? 3 : 4, ctx->xchunk, w); }
// Stages of the order-4 kernels' rings (h_kernel): 4 for launches of more than four waves
// of their CTAs and for walks of 8 planes and more, 3 otherwise.  In us a step, 3 and 4
// stages: 1024 CTAs of 4 planes (128^3) 39.4 and 41.5, 700 (100^3) 28.8 and 30.1; 2800 (192x160x224) 121.8
// and 115.8; 16 planes at 128^3 37.5 and 37.2, on 192x160x224 115.8 and 95.8.  Not with a
// design region nor where most cells lie in an absorber's slabs: their loads go
// through the L1 cache that the fourth stage takes (200^3 with a design region
// 220 and 227, 600x600x12 with slabs of 4 278 and 286).
static int stream_stages(const dtmx_ctx* ctx, const WorkPlan& w) {
  double inside = 1.0;
  for (int a = 0; a < 3; a++) inside *= 1.0 - (double)(ctx->P.ab.L[a][0] + ctx->P.ab.L[a][1]) / ctx->P.g.n[a];
  if (ctx->P.des_on || (ctx->P.ab.kind != 0 && inside < 0.5)) return 3;
  return (long long)w.grid.x * w.grid.y * w.grid.z > 4 * 148 * 3 || w.xchunk >= 8 ? 4 : 3;
}
static int plan_sweep(dtmx_ctx* ctx, const WorkPlan** w) {
  return plan_work(ctx, WK_SWEEP, ctx->frows, ctx->frows == 16 ? 3 : 5, std::min(ctx->xchunk, FX_MAX), w);
}

static int set_kernel_attributes() {
  static bool done = false;
  if (done) return 0;
  auto allow = [](const void* k, size_t smem) { cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); };
  allow((const void*)h_kernel<2, false, 3>, Pipe<2, true>::SMEM_BYTES);
  allow((const void*)h_kernel<2, true, 3>, Pipe<2, true>::SMEM_BYTES);
  allow((const void*)h_kernel<4, false, 3>, Pipe<4, true>::SMEM_BYTES);
  allow((const void*)h_kernel<4, false, 4>, Pipe<4, true, 4>::SMEM_BYTES);
  allow((const void*)e_kernel<2, false, 3>, Pipe<2, false>::SMEM_BYTES);
  allow((const void*)e_kernel<2, true, 3>, Pipe<2, false>::SMEM_BYTES);
  allow((const void*)e_kernel<4, false, 3>, Pipe<4, false>::SMEM_BYTES);
  allow((const void*)e_kernel<4, false, 4>, Pipe<4, false, 4>::SMEM_BYTES);
  done = true;
  return 0;
}

// The end of a step in one launch (two while the adjoint's objective is
// recorded next to other DFT planes): soft sources, probes, DFT samples, the
// design region's history, the step counter.  P.f is the state after the step.
static long long launch_tail(dtmx_ctx* ctx, const Params& P, cudaStream_t st) {
  const dtmx_config& c = ctx->cfg;
  long long nl = 0;
  TailArgs a{};
  a.dt = c.dt;
  a.ticket = ctx->d_ticket;
  const int ns = (int)ctx->psrc.size();
  if (ns > TAIL_SRC) {
    launch(ctx, ctx->early, point_source_kernel, (ctx->nrun + 63) / 64, 64, 0, st, P, ctx->d_psrc, ctx->d_psrc_run, ctx->nrun, ctx->d_step, c.dt);
    nl++;
  } else {
    a.src = ctx->d_psrc; a.ns = ns;
  }
  MonTable* sets[2] = {!ctx->monitors_off && ctx->mon.nmap ? &ctx->mon : nullptr, ctx->obj_on ? &ctx->objmon : nullptr};
  if (!sets[0]) { sets[0] = sets[1]; sets[1] = nullptr; }
  for (int q = 0; q < 2; q++) {
    if (q == 1 && !sets[1]) break;
    MonTable* m = sets[q];
    const bool end = q == 1 || !sets[1];
    TailArgs b = a;
    if (q == 0 && !ctx->probes.empty() && !ctx->monitors_off) {
      b.pr = ctx->d_probes; b.np = (int)ctx->probes.size();
      b.traces = ctx->d_traces; b.cap = ctx->probe_cap;
      b.every = c.probe_every > 0 ? c.probe_every : 1;
    }
    if (q == 1) b.ns = 0;                          // (the first launch has added the sources)
    if (m) { b.dft = m->tab; b.map = m->map; b.nmap = m->nmap; b.slot = m->nstaged; }
    if (end) {
      b.hist = ctx->hist_out;
      b.nd = P.des_on ? P.des_n[0] * P.des_n[1] * P.des_n[2] : 0;
      b.advance = 1;
    }
    const int blocks = std::max({1, b.nmap + (b.hist ? (3 * b.nd + 255) / 256 : 0), (b.np + 255) / 256});
    launch(ctx, ctx->early, tail_kernel, blocks, 256, 0, st, P, b, ctx->d_step);
    nl++;
    if (m && ++m->nstaged == DFT_STAGE) dft_flush(ctx, *m);
  }
  return nl;
}

// Nodes of a half step's dipole corrections up to which a node gets eight threads
// instead of one (tfsf_kernel).  Measured, us a step added by the corrections:
// order 2, 19 thousand nodes 12.6 with eight and 15.9 with one, 43 thousand 22 and 16,
// 307 thousand 126 and 30; order 4, whose nodes have up to two crossing taps of
// a term, 32 thousand 17 and 22, 58 thousand 28 and 23, 920 thousand 378 and 122.
constexpr long long kTapNodes2 = 28000, kTapNodes4 = 44000;
// TF/SF corrections of one half step, and the plane wave's line
static long long launch_tfsf(dtmx_ctx* ctx, const Params& P, cudaStream_t st, bool isH) {
  if (!ctx->has_tfsf) return 0;
  const TfsfDev& T = ctx->T;
  const int hs = isH ? 1 : 0;
  const bool o4 = ctx->cfg.order == 4;
  if (ctx->tfsf.kind == DTMX_TFSF_PLANE_X) {
    const dtmx_tfsf& s = ctx->tfsf;
    const LineDev l{ctx->line_e, ctx->line_h, T.line_n, ctx->line_src, ctx->cfg.dt / ctx->cfg.dx, ctx->cfg.dt, s.amp, s.f0, s.tau, s.t0};
    long long units = 64;                          // warps of a job (128 nodes each); at least 8 blocks for the line
    for (int r = 0; r < T.njob[hs]; r++) {
      const TfsfJob& jb = T.job[hs][r];
      const int la = jb.a == 2 ? 1 : 2;
      const long long nl = jb.hi[la] - jb.lo[la] + 1;
      units = std::max(units, jb.cells / nl * ((nl + 127) / 128));
    }
    const dim3 grd((unsigned)((units + 7) / 8), T.njob[hs] + 1);
    if (o4) launch(ctx, ctx->early, tfsf_plane_kernel<4>, grd, 256, 0, st, P, T, l, ctx->d_step, isH);
    else launch(ctx, ctx->early, tfsf_plane_kernel<2>, grd, 256, 0, st, P, T, l, ctx->d_step, isH);
    return 1;
  }
  long long mx = 1, all = 0;
  for (int r = 0; r < T.njob[hs]; r++) { mx = std::max(mx, T.job[hs][r].cells); all += T.job[hs][r].cells; }
  const bool taps = all <= (o4 ? kTapNodes4 : kTapNodes2);
  const dim3 grd((unsigned)((mx * (taps ? 8 : 1) + 255) / 256), std::max(1, T.njob[hs]));
  auto k = o4 ? (taps ? tfsf_kernel<4, 8> : tfsf_kernel<4, 1>) : (taps ? tfsf_kernel<2, 8> : tfsf_kernel<2, 1>);
  launch(ctx, ctx->early, k, grd, 256, 0, st, P, T, ctx->d_step, isH);
  return 1;
}
// grid of the passes over the ADE box (ade_cell)
static dim3 ade_grid(const Params& P) {
  return dim3((unsigned)(((long long)P.ade.n[1] * P.ade.n[2] + 255) / 256), std::max(1, P.ade.n[0]));
}

static int launch_step(dtmx_ctx* ctx) {
  set_kernel_attributes();
  const dtmx_config& c = ctx->cfg;
  Params P = ctx->P;
  const WorkPlan* wp;
  if (int rc = plan_stream(ctx, &wp)) return rc;
  const WorkPlan& plan = *wp;
  P.xchunk = plan.xchunk;
  const int blk = STREAM_NT;
  const dim3 grd = plan.grid;
  const bool o4 = c.order == 4, deep = o4 && stream_stages(ctx, plan) == 4;
  cudaStream_t st = ctx->stream;
  long long nl = 0;
  if (ctx->profiling) cudaEventRecord(ctx->ev[0], st);
  if (o4 && deep) launch(ctx, ctx->early, h_kernel<4, false, 4>, grd, blk, Pipe<4, true, 4>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  else if (o4) launch(ctx, ctx->early, h_kernel<4, false, 3>, grd, blk, Pipe<4, true>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  else if (plan.table) launch(ctx, ctx->early, h_kernel<2, true, 3>, grd, blk, Pipe<2, true>::SMEM_BYTES, st, P, ctx->maps, plan.work);
  else launch(ctx, ctx->early, h_kernel<2, false, 3>, grd, blk, Pipe<2, true>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  if (ctx->profiling) cudaEventRecord(ctx->ev[1], st);
  nl++;
  nl += launch_tfsf(ctx, P, st, true);
  const int cur = ctx->gcur;
  if (ctx->has_gyro) {
    launch(ctx, ctx->early, gyro_current_kernel, ade_grid(P), 256, 0, st, P, cur);
    ctx->gcur = 1 - cur;
    nl++;
  }
  if (ctx->profiling) cudaEventRecord(ctx->ev[2], st);
  if (o4 && deep) launch(ctx, ctx->early, e_kernel<4, false, 4>, grd, blk, Pipe<4, false, 4>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  else if (o4) launch(ctx, ctx->early, e_kernel<4, false, 3>, grd, blk, Pipe<4, false>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  else if (plan.table) launch(ctx, ctx->early, e_kernel<2, true, 3>, grd, blk, Pipe<2, false>::SMEM_BYTES, st, P, ctx->maps, plan.work);
  else launch(ctx, ctx->early, e_kernel<2, false, 3>, grd, blk, Pipe<2, false>::SMEM_BYTES, st, P, ctx->maps, Work<false>{});
  if (P.ade.Em[0] || ctx->has_gyro) {
    // dispersive and gyrotropic nodes of the E half step (e_kernel skipped them)
    const bool box = c.geometry == DTMX_GEOM_BOX;
    if (o4) { if (box) launch(ctx, ctx->early, ade_node_kernel<4, true, false>, ade_grid(P), 256, 0, st, P, cur); else launch(ctx, ctx->early, ade_node_kernel<4, false, false>, ade_grid(P), 256, 0, st, P, cur); }
    else { if (box) launch(ctx, ctx->early, ade_node_kernel<2, true, false>, ade_grid(P), 256, 0, st, P, cur); else launch(ctx, ctx->early, ade_node_kernel<2, false, false>, ade_grid(P), 256, 0, st, P, cur); }
    nl++;
  }
  if (ctx->profiling) {
    cudaEventRecord(ctx->ev[3], st);
    // read back this step's two kernel durations (keeps the events reusable)
    cudaEventSynchronize(ctx->ev[3]);
    float a = 0, b = 0;
    cudaEventElapsedTime(&a, ctx->ev[0], ctx->ev[1]);
    cudaEventElapsedTime(&b, ctx->ev[2], ctx->ev[3]);
    ctx->prof_ms_h += a; ctx->prof_ms_e += b; ctx->prof_count++;
  }
  nl++;
  nl += launch_tfsf(ctx, P, st, false);
  nl += launch_tail(ctx, P, st);
  ctx->launches += nl;
  return launched(ctx);
}

// First-step preparation: upload the source and probe lists, allocate the
// probe traces and check the TF/SF shell against the materials.
static int prepare(dtmx_ctx* ctx) {
  if (ctx->prepared) return DTMX_OK;
  int rc;
  std::vector<PointSrcDev> sorted = ctx->psrc;
  std::vector<int2> runs;
  if (!sorted.empty()) {
    // by node, sources on one node in the order they were given
    std::stable_sort(sorted.begin(), sorted.end(),
                     [](const PointSrcDev& a, const PointSrcDev& b) { return std::tie(a.comp, a.id) < std::tie(b.comp, b.id); });
    for (int q = 0; q < (int)sorted.size(); q++) {
      if (q > 0 && sorted[q].comp == sorted[q - 1].comp && sorted[q].id == sorted[q - 1].id) runs.back().y++;
      else runs.push_back(make_int2(q, 1));
    }
    if ((rc = dalloc(ctx, &ctx->d_psrc, sorted.size(), true))) return rc;
    CK(cudaMemcpyAsync(ctx->d_psrc, sorted.data(), sorted.size() * sizeof(PointSrcDev), cudaMemcpyHostToDevice, ctx->stream));
    if (sorted.size() > TAIL_SRC) {
      if ((rc = dalloc(ctx, &ctx->d_psrc_run, runs.size(), true))) return rc;
      CK(cudaMemcpyAsync(ctx->d_psrc_run, runs.data(), runs.size() * sizeof(int2), cudaMemcpyHostToDevice, ctx->stream));
      ctx->nrun = (int)runs.size();
    }
  }
  if (!ctx->probes.empty()) {
    if ((rc = dalloc(ctx, &ctx->d_probes, ctx->probes.size(), true))) return rc;
    CK(cudaMemcpyAsync(ctx->d_probes, ctx->probes.data(), ctx->probes.size() * sizeof(ProbeDev), cudaMemcpyHostToDevice, ctx->stream));
    if ((rc = dalloc(ctx, &ctx->d_traces, ctx->probes.size() * (size_t)ctx->probe_cap))) return rc;
  }
  if ((rc = mon_build(ctx, ctx->mon, ctx->dfts.data(), (int)ctx->dfts.size()))) return rc;
  if (ctx->has_tfsf && ctx->h_mat[0].size()) {
    // every E node that gets a correction, and the E nodes next to them, must be non-dispersive
    const TfsfDev& T = ctx->T;
    for (int r = 0; r < T.njob[0]; r++) {
      const TfsfJob& jb = T.job[0][r];
      for (int i = std::max(0, jb.lo[0] - 1); i <= std::min(ctx->cfg.nx - 1, jb.hi[0] + 1); i++)
        for (int j = std::max(0, jb.lo[1] - 1); j <= std::min(ctx->cfg.ny - 1, jb.hi[1] + 1); j++)
          for (int k = std::max(0, jb.lo[2] - 1); k <= std::min(ctx->cfg.nz - 1, jb.hi[2] + 1); k++)
            for (int comp = 0; comp < 3; comp++)
              if (ctx->mats[ctx->h_mat[comp][store_index(ctx, i, j, k)]].npoles > 0 ||
                  ctx->mats[ctx->h_mat[comp][store_index(ctx, i, j, k)]].gyro_wp > 0)
                return fail(ctx, DTMX_ERR_UNSUPPORTED, "dispersive or gyrotropic material on the TF/SF surface");
    }
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->prepared = true;
  return DTMX_OK;
}

// ---------------------------------------------------------------- wavefront engine
constexpr int TORRE_TY = 32;

static int build_torre_maps(dtmx_ctx* ctx) {
  if (ctx->tmaps_ok) return DTMX_OK;
  const int R2 = ctx->cfg.order - 1, TY = TORRE_TY;
  TorreMaps& m = ctx->tmaps;
  int rc;
  for (int h = 0; h < 2; h++) {
    const int c0 = 3 * h;
    if ((rc = make_map(ctx, &m.A[h], ctx->P.f[c0], false, 40, TY + R2))) return rc;
    if ((rc = make_map(ctx, &m.B[h], ctx->P.f[c0 + 1], false, 40, TY))) return rc;
    if ((rc = make_map(ctx, &m.C[h], ctx->P.f[c0 + 2], false, 32, TY + R2))) return rc;
  }
  for (int c = 0; c < 6; c++)
    if ((rc = make_map(ctx, &m.core[c], ctx->P.f[c], false, 32, TY))) return rc;
  for (int c = 0; c < 3; c++)
    if ((rc = make_map(ctx, &m.mat[c], ctx->d_mat[c], true, 32, TY))) return rc;
  ctx->tmaps_ok = true;
  return DTMX_OK;
}

using TorreFn = void (*)(const Params, const TorreMaps, const TorreArgs);

static TorreFn torre_fn(int order, int T, size_t* smem, int* nthr) {
  constexpr int TY = TORRE_TY;
#define DTMX_TORRE_CASE(O, TT)                                                         \
  if (order == O && T == TT) {                                                          \
    *smem = TorreLayout<O, TY>::SMEM; *nthr = TorreLayout<O, TY>::NTHR;                 \
    return torre_kernel<O, 2 * TT, TY>;                                                 \
  }
  DTMX_TORRE_CASE(2, 1) DTMX_TORRE_CASE(2, 2) DTMX_TORRE_CASE(2, 3) DTMX_TORRE_CASE(2, 4)
  DTMX_TORRE_CASE(4, 1) DTMX_TORRE_CASE(4, 2)
#undef DTMX_TORRE_CASE
  return nullptr;
}

// Can the wavefront engine run this context with T steps per launch?
static bool torre_usable(dtmx_ctx* ctx, int T, std::string* why) {
  const dtmx_config& c = ctx->cfg;
  size_t smem = 0;
  int nthr = 0;
  TorreFn fn = torre_fn(c.order, T, &smem, &nthr);
  if (!fn) { *why = "no kernel for order " + std::to_string(c.order) + " with " + std::to_string(T) + " steps per launch"; return false; }
  if (c.geometry != DTMX_GEOM_BOX) { *why = "needs the box geometry"; return false; }
  if (c.absorber == DTMX_ABS_SPLIT_PML) { *why = "split PML is not supported"; return false; }
  if (ctx->has_gyro) { *why = "gyrotropic materials need a current pass between half steps"; return false; }
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    *why = "shared memory attribute refused";
    return false;
  }
  int per_sm = 0, nsm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nthr, smem) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->dev) != cudaSuccess) {
    cudaGetLastError();
    *why = "occupancy query failed";
    return false;
  }
  const long long tiles = (long long)((c.nz + TT_Z - 1) / TT_Z) * ((c.ny + TORRE_TY - 1) / TORRE_TY);
  if (tiles > (long long)per_sm * nsm) {
    *why = std::to_string(tiles) + " tiles exceed the " + std::to_string(per_sm * nsm) + " co-resident CTAs";
    return false;
  }
  return true;
}

// features the wavefront engine does not carry inside its launch
static bool torre_features_ok(const dtmx_ctx* ctx, std::string* why) {
  if (ctx->has_gyro) { *why = "gyrotropic materials"; return false; }
  if (ctx->has_tfsf) { *why = "TF/SF source"; return false; }
  if (!ctx->psrc.empty()) { *why = "point sources"; return false; }
  if (!ctx->probes.empty()) { *why = "probes"; return false; }
  if (!ctx->dfts.empty()) { *why = "DFT planes"; return false; }
  return true;
}

__global__ void advance_step_by_kernel(long long* d_step, int n) { *d_step += n; }

static int launch_torre(dtmx_ctx* ctx, int T) {
  const dtmx_config& c = ctx->cfg;
  int rc = build_torre_maps(ctx);
  if (rc) return rc;
  size_t smem = 0;
  int nthr = 0;
  TorreFn fn = torre_fn(c.order, T, &smem, &nthr);
  const int ntz = (c.nz + TT_Z - 1) / TT_Z, nty = (c.ny + TORRE_TY - 1) / TORRE_TY;
  if (!ctx->d_ctr && (rc = dalloc(ctx, &ctx->d_ctr, (size_t)ntz * nty))) return rc;
  CK(cudaMemsetAsync(ctx->d_ctr, 0, sizeof(int) * ntz * nty, ctx->stream));
  Params P = ctx->P;
  P.x0 = 0; P.x1 = c.nx;
  TorreArgs ta;
  ta.ctr = ctx->d_ctr; ta.ntz = ntz; ta.nty = nty;
  ta.nsteps = c.nx + (c.order == 4 ? TorreGeom<4>::off(2 * T - 1) : TorreGeom<2>::off(2 * T - 1));
  void* args[] = {(void*)&P, (void*)&ctx->tmaps, (void*)&ta};
  if (ctx->profiling) cudaEventRecord(ctx->ev[0], ctx->stream);
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)fn, dim3(ntz, nty), dim3(nthr), args, smem, ctx->stream);
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("wavefront launch: ") + cudaGetErrorString(e));
  if (ctx->profiling) {
    cudaEventRecord(ctx->ev[1], ctx->stream);
    cudaEventSynchronize(ctx->ev[1]);
    float a = 0;
    cudaEventElapsedTime(&a, ctx->ev[0], ctx->ev[1]);
    ctx->prof_ms_h += a; ctx->prof_count += T;
  }
  launch(ctx, false, advance_step_by_kernel, 1, 1, 0, ctx->stream, ctx->d_step, T);
  ctx->launches += 2;
  if (int bad = launched(ctx)) return bad;
  ctx->step += T;
  return DTMX_OK;
}

// ---------------------------------------------------------------- single-sweep engine
// Applies to the box geometry with the Yee stencil and a CPML or no absorber;
// everything else the per-step engine covers.
static bool fused_usable(const dtmx_ctx* ctx, std::string* why) {
  const dtmx_config& c = ctx->cfg;
  if (c.geometry != DTMX_GEOM_BOX) { if (why) *why = "box geometry only"; return false; }
  if (c.order != 2) { if (why) *why = "order 2 only"; return false; }
  if (c.absorber == DTMX_ABS_SPLIT_PML) { if (why) *why = "no split PML"; return false; }
  return true;
}

template <int TY>
static int build_fused_maps(dtmx_ctx* ctx, FusedMaps& fm, float* const* f) {
  using L = FL<TY>;
  int rc;
  for (int c = 0; c < 3; c++) {
    if ((rc = make_map(ctx, &fm.e[c], f[c], false, FE_W, L::FE_R))) return rc;
    fm.mat[c] = ctx->maps.mat[c];
  }
  if ((rc = make_map(ctx, &fm.hx, f[3], false, FHX_W, L::FHX_R))) return rc;
  if ((rc = make_map(ctx, &fm.hy, f[4], false, FHY_W, L::FHY_R))) return rc;
  return make_map(ctx, &fm.hz, f[5], false, FHZ_W, L::FHZ_R);
}

// First use: the second buffer set, the maps reading each set, the tile table.
static int fused_prepare(dtmx_ctx* ctx) {
  if (ctx->fused_ready) return DTMX_OK;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(fused_kernel<16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL<16>::SMEM);
    cudaFuncSetAttribute(fused_kernel<16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL<16>::SMEM);
    cudaFuncSetAttribute(fused_kernel<8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL<8>::SMEM);
    attr = true;
  }
  // one allocation, cut up (twelve of them cost the first step of a 128^3 grid 3.6 ms), but for parkable contexts,
  // whose arrays are parked one by one; the first array's address is the block's (fused_release)
  float** arr[12];
  size_t len[12], total = 0;
  int na = 0, rc = DTMX_OK;
  auto want = [&](float** q, size_t n) { arr[na] = q; len[na++] = n; total += (n + 63) / 64 * 64; };
  for (int comp = 0; comp < 6; comp++) want(&ctx->f_alt[comp], ctx->nstore + 64);
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < 2; q++)
      if (ctx->P.ab.aux[a][2]) want(&ctx->hax_alt[a][q], (size_t)(ctx->P.ab.L[a][0] + ctx->P.ab.L[a][1]) * (ctx->ncell / (size_t)ctx->P.g.n[a]));
  if (ctx->cfg.parkable) {
    for (int q = 0; q < na && !rc; q++) rc = dalloc(ctx, arr[q], len[q]);
  } else {
    float* block = nullptr;
    rc = dalloc(ctx, &block, total);
    for (int q = 0; q < na && !rc; q++) { *arr[q] = block; block += (len[q] + 63) / 64 * 64; }
  }
  // maps of the per-step kernels over the second set, so either engine runs from either buffer
  if (!rc) {
    TmaMaps save = ctx->maps;
    float* fsave[6];
    for (int comp = 0; comp < 6; comp++) { fsave[comp] = ctx->P.f[comp]; ctx->P.f[comp] = ctx->f_alt[comp]; }
    rc = build_maps(ctx);
    ctx->maps_alt = ctx->maps;
    ctx->maps = save;
    for (int comp = 0; comp < 6; comp++) ctx->P.f[comp] = fsave[comp];
  }
  if (!rc) rc = build_fused_maps<16>(ctx, ctx->fmaps[0], ctx->P.f);
  if (!rc) rc = build_fused_maps<16>(ctx, ctx->fmaps[1], ctx->f_alt);
  if (!rc) rc = build_fused_maps<8>(ctx, ctx->fmaps8[0], ctx->P.f);
  if (!rc) rc = build_fused_maps<8>(ctx, ctx->fmaps8[1], ctx->f_alt);
  if (rc) return rc;
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->fused_ready = true;
  return DTMX_OK;
}

static double free_device_bytes() {
  size_t fr = 0, tot = 0;
  return cudaMemGetInfo(&fr, &tot) == cudaSuccess ? (double)fr : 0.0;
}

// device bytes of the second set
static double fused_set_bytes(const dtmx_ctx* ctx) {
  double n = 6.0 * (ctx->nstore + 64);
  for (int a = 0; a < 3; a++)
    if (ctx->P.ab.aux[a][2]) n += 2.0 * (ctx->P.ab.L[a][0] + ctx->P.ab.L[a][1]) * (double)(ctx->ncell / (size_t)ctx->P.g.n[a]);
  return 4.0 * n;
}

// Give the second set back, half-made or whole (plain allocations: the automatic choice leaves parkable
// contexts alone): the block, or after an odd number of swaps the arrays allocated first; pointers into a block free nothing.
static void fused_release(dtmx_ctx* ctx) {
  if (ctx->fused_ready) return;
  cudaStreamSynchronize(ctx->stream);
  auto drop = [&](float*& q) {
    if (!q) return;
    auto it = std::find(ctx->allocs.begin(), ctx->allocs.end(), (void*)q);
    if (it != ctx->allocs.end()) { cudaFree(q); ctx->allocs.erase(it); }
    q = nullptr;
  };
  for (auto& q : ctx->f_alt) drop(q);
  for (auto& a : ctx->hax_alt)
    for (auto& q : a) drop(q);
}

// The automatic choice's second set given back for another use of the memory:
// the context goes on with the per-step engine (the state is always in P.f).
// Not while the caller captures the stream: nothing may be freed then.
static bool fused_give_back(dtmx_ctx* ctx) {
  if (ctx->engine != 0 || !ctx->fused_ready || ctx->cfg.parkable || ctx->set_in_graph || capturing(ctx)) return false;
  cudaStreamSynchronize(ctx->stream);
  drop_graphs(ctx);
  ctx->fused_ready = false;
  ctx->auto_per_step = true;
  fused_release(ctx);
  return true;
}

// The state now lives in the other buffer set: swap the pointers (fields, H
// auxiliaries, the maps reading them) so that P and every pass see it.
static void fused_swap(dtmx_ctx* ctx) {
  for (int comp = 0; comp < 6; comp++) std::swap(ctx->P.f[comp], ctx->f_alt[comp]);
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < 2; q++) std::swap(ctx->P.ab.aux[a][2 + q], ctx->hax_alt[a][q]);
  std::swap(ctx->maps, ctx->maps_alt);
  std::swap(ctx->fmaps[0], ctx->fmaps[1]);
  std::swap(ctx->fmaps8[0], ctx->fmaps8[1]);
  ctx->parity ^= 1;
  ctx->tmaps_ok = false;          // the wavefront engine's maps are rebuilt for the current buffer
}

// One time step of the single-sweep engine: the side passes that act on the
// old state (TF/SF H correction, gyrotropic current), the sweep A -> B, the
// passes on the new state (dispersive nodes, sources, TF/SF E correction,
// monitors), then the buffer swap.
static int launch_fused_step(dtmx_ctx* ctx) {
  int rc = fused_prepare(ctx);
  if (rc) return rc;
  Params PA = ctx->P;
  const WorkPlan* wp;
  if ((rc = plan_sweep(ctx, &wp))) return rc;
  const WorkPlan& plan = *wp;
  PA.xchunk = plan.xchunk;
  Params PB = PA;
  FusedArgs fa{};
  for (int comp = 0; comp < 6; comp++) { PB.f[comp] = ctx->f_alt[comp]; fa.dst[comp] = ctx->f_alt[comp]; }
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < 2; q++) {
      fa.hsrc[a][q] = PA.ab.aux[a][2 + q];
      fa.hdst[a][q] = ctx->hax_alt[a][q];
      PB.ab.aux[a][2 + q] = ctx->hax_alt[a][q];
    }
  cudaStream_t st = ctx->stream;
  // TF/SF correction of H, added to the old H (the H update is linear in it)
  long long nl = launch_tfsf(ctx, PA, st, true);
  const dim3 grd = plan.grid;
  if (ctx->profiling) cudaEventRecord(ctx->ev[0], st);
  if (ctx->frows == 8) launch(ctx, ctx->early, fused_kernel<8, false>, grd, FL<8>::NT, FL<8>::SMEM, st, PA, fa, ctx->fmaps8[0], Work<false>{});
  else if (plan.table) launch(ctx, ctx->early && !plan.alone, fused_kernel<16, true>, grd, FL<16>::NT, FL<16>::SMEM, st, PA, fa, ctx->fmaps[0], plan.work);
  else launch(ctx, ctx->early, fused_kernel<16, false>, grd, FL<16>::NT, FL<16>::SMEM, st, PA, fa, ctx->fmaps[0], Work<false>{});
  if (ctx->profiling) cudaEventRecord(ctx->ev[1], st);
  nl++;
  if (PA.ade.Em[0] || ctx->has_gyro) {
    // dispersive nodes (left by the sweep) from the old E in A; on gyrotropic nodes the current from the
    // old E, then E -= dt/eps_inf J
    for (int comp = 0; comp < 3; comp++) PB.fe_old[comp] = PA.f[comp];
    if (ctx->has_gyro) {
      launch(ctx, ctx->early, ade_node_kernel<2, true, true>, ade_grid(PB), 256, 0, st, PB, ctx->gcur);
      ctx->gcur = 1 - ctx->gcur;
    } else {
      launch(ctx, ctx->early, ade_node_kernel<2, true, false>, ade_grid(PB), 256, 0, st, PB, 0);
    }
    nl++;
  }
  if (ctx->profiling) {
    cudaEventSynchronize(ctx->ev[1]);
    float a = 0;
    cudaEventElapsedTime(&a, ctx->ev[0], ctx->ev[1]);
    ctx->prof_ms_h += a; ctx->prof_count++;
  }
  nl += launch_tfsf(ctx, PB, st, false);
  nl += launch_tail(ctx, PB, st);
  ctx->launches += nl;
  if ((rc = launched(ctx))) return rc;
  fused_swap(ctx);
  return DTMX_OK;
}

// The engine of a step: 3 where it was chosen, and for engine 0 (automatic)
// wherever the single sweep applies: it was faster at every size measured
// (48^3 9.4 against 34.9 us a step, 128^3 40 against 66, 640x512x384 1.30
// against 1.79 ms).  The automatic choice stays with the per-step engine
//   * once the caller holds the fields' addresses, from dtmx_field_device_ptr
//     or in a graph that steps were captured into, which may be replayed any
//     number of times and between other steps (the single sweep alternates
//     between two sets of arrays, the per-step engine updates the one the caller
//     holds),
//   * while profiling (which times the H and the E kernel),
//   * for parkable contexts, where the second set would take more than an eighth
//     of the free device memory (or cannot be had), and once it has been given
//     back: it doubles the fields, and the memory left is the caller's.  A
//     request for device memory that fails, on this or another context, takes the
//     set (free_a_set); other allocators cannot, hence the eighth.
// Needs fused_prepare's allocations, so call it outside a capture.
static int step_engine(dtmx_ctx* ctx) {
  if (ctx->engine != 0) return ctx->engine == 3 ? 3 : 1;
  if (ctx->pinned || ctx->profiling || ctx->cfg.parkable || ctx->auto_per_step || !fused_usable(ctx, nullptr)) return 1;
  if (!ctx->fused_ready) {
    ctx->spare_others = true;
    const bool made = fused_set_bytes(ctx) <= 0.125 * free_device_bytes() && fused_prepare(ctx) == DTMX_OK;
    ctx->spare_others = false;
    if (!made) {
      fused_release(ctx);
      ctx->auto_per_step = true;
      return 1;
    }
  }
  if (!ctx->lendable) {
    std::lock_guard<std::mutex> lk(lenders().mu);
    lenders().list.push_back(ctx);
    ctx->lendable = true;
  }
  return 3;
}

// From here on the caller holds the addresses of the fields.  (The step graphs go
// later: this may be called while a stream is captured.)
static void pin_fields(dtmx_ctx* ctx) {
  if (ctx->pinned) return;
  ctx->pinned = true;
  ctx->graphs_stale = ctx->engine == 0;
}

// one time step of the selected per-step engine (per-step or single sweep)
static int launch_one(dtmx_ctx* ctx) { return step_engine(ctx) == 3 ? launch_fused_step(ctx) : launch_step(ctx); }

// Capture (once per field buffer) and launch 16 per-step launch sequences as
// one graph.  The host-side bookkeeping of the 16 steps (staging slots,
// flushes, buffer parities) is done during the capture; the captured kernels
// read the step number from the device counter, so the graph is valid at
// every 16-step boundary of an aligned run that starts from the same buffer
// (16 single-sweep steps come back to it).
static int graph_steps16(dtmx_ctx* ctx) {
  const int par = ctx->parity;
  if (ctx->graphs_stale) drop_graphs(ctx);
  if (!ctx->graph16[par]) {
    set_kernel_attributes();
    if (step_engine(ctx) == 3) {
      int rc = fused_prepare(ctx);
      if (!rc) rc = plan_sweep(ctx, nullptr);
      if (rc) return rc;
    } else if (int rc = plan_stream(ctx, nullptr)) {
      return rc;
    }
    const long long launches0 = ctx->launches;
    const int gcur0 = ctx->gcur;
    const int staged0 = ctx->mon.nstaged;
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
      return fail(ctx, DTMX_ERR_CUDA, "graph capture could not start");
    int rc = DTMX_OK;
    for (int q = 0; q < 16 && !rc; q++) rc = launch_one(ctx);
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    if (rc || e != cudaSuccess) {
      // nothing of it ran: the bookkeeping goes back too
      if (ctx->parity != par) fused_swap(ctx);
      ctx->gcur = gcur0;
      ctx->mon.nstaged = staged0;
      if (g) cudaGraphDestroy(g);
      if (e != cudaSuccess) cudaGetLastError();
      return rc ? rc : fail(ctx, DTMX_ERR_CUDA, "graph capture failed");
    }
    e = cudaGraphInstantiate(&ctx->graph16[par], g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) { ctx->graph16[par] = nullptr; cudaGetLastError(); return fail(ctx, DTMX_ERR_CUDA, "graph instantiation failed"); }
    // the capture ran the bookkeeping of 16 steps; the graph below executes them
    if (ctx->gcur != gcur0 || ctx->parity != par) return fail(ctx, DTMX_ERR_STATE, "graph capture: unexpected buffer parity");
    if (ctx->mon.nstaged != staged0) return fail(ctx, DTMX_ERR_STATE, "graph capture: staging not aligned");
    ctx->graph_launches[par] = ctx->launches - launches0;
  } else {
    ctx->launches += ctx->graph_launches[par];
  }
  CK(cudaGraphLaunch(ctx->graph16[par], ctx->stream));
  ctx->step += 16;
  return DTMX_OK;
}

extern "C" int dtmx_step(dtmx_ctx* ctx, int nsteps) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || nsteps < 0) return fail(ctx, DTMX_ERR_INVALID, "bad step count");
  const Running running(ctx);
  int rc0 = prepare(ctx);
  if (rc0) return rc0;
  int left = nsteps;
  if (int rc = launched(ctx)) return rc;         // (of an earlier call that ended with another error)
  // steps that the caller captures: with engine 0 in place, one by one; with engine 3 on both sets,
  // which then stay
  const bool any = (ctx->engine == 0 || ctx->engine == 3) && nsteps > 0 && capturing(ctx), captured = any && ctx->engine == 0;
  if (captured) pin_fields(ctx);
  if (any && ctx->engine == 3) ctx->set_in_graph = true;
  if (ctx->pinned) fused_give_back(ctx);
  if (ctx->engine == 2) {
    std::string why;
    if (!torre_features_ok(ctx, &why)) return fail(ctx, DTMX_ERR_UNSUPPORTED, "wavefront engine: " + why);
    while (left >= ctx->tblock) {
      int rc = launch_torre(ctx, ctx->tblock);
      if (rc) return rc;
      left -= ctx->tblock;
    }
  }
  if (ctx->engine == 3) {
    std::string why;
    if (!fused_usable(ctx, &why)) return fail(ctx, DTMX_ERR_UNSUPPORTED, "single-sweep engine: " + why);
  }
  while (left > 0) {
    // 16 steps as one CUDA graph when every DFT staging cycle is at its start
    // (the captured sequence then repeats exactly: staging slots, the flush
    // every 16 steps and the gyrotropic buffer parity)
    bool aligned = left >= 16 && !ctx->profiling && !ctx->monitors_off && ctx->engine != 2 && !captured;
    aligned = aligned && ctx->mon.nstaged == 0;
    if (aligned && !ctx->obj_on) {
      int rc = graph_steps16(ctx);
      if (rc) return rc;
      left -= 16;
      continue;
    }
    int rc = ctx->engine == 2 ? launch_step(ctx) : launch_one(ctx);
    if (rc) return rc;
    ctx->step++;
    left--;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  return DTMX_OK;
}

// ---------------------------------------------------------------- design region and adjoint
extern "C" int dtmx_set_design(dtmx_ctx* ctx, const int* lo, const int* n, const float* eps) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !lo || !n || !eps) return fail(ctx, DTMX_ERR_INVALID, "bad design region");
  const dtmx_config& c = ctx->cfg;
  const int dim[3] = {c.nx, c.ny, c.nz};
  for (int a = 0; a < 3; a++)
    if (n[a] < 1 || lo[a] < 0 || lo[a] + n[a] > dim[a]) return fail(ctx, DTMX_ERR_INVALID, "design region outside the grid");
  if (ctx->prepared) return fail(ctx, DTMX_ERR_STATE, "the design region must be set before the first step");
  const size_t nd = (size_t)n[0] * n[1] * n[2];
  for (int comp = 0; comp < 3; comp++) {
    ctx->h_des_ie[comp].resize(nd);
    for (size_t q = 0; q < nd; q++) {
      const float e = eps[comp * nd + q];
      if (!(e > 0)) return fail(ctx, DTMX_ERR_INVALID, "design permittivity must be > 0");
      ctx->h_des_ie[comp][q] = (float)(1.0 / (double)e);
    }
  }
  for (int comp = 0; comp < 3; comp++) {
    if (ctx->d_des_ie[comp] && (size_t)ctx->P.des_n[0] * ctx->P.des_n[1] * ctx->P.des_n[2] != nd) ctx->d_des_ie[comp] = nullptr;
    int rc;
    if (!ctx->d_des_ie[comp] && (rc = dalloc(ctx, &ctx->d_des_ie[comp], nd))) return rc;
    CK(cudaMemcpyAsync(ctx->d_des_ie[comp], ctx->h_des_ie[comp].data(), nd * 4, cudaMemcpyHostToDevice, ctx->stream));
    ctx->P.des_ie[comp] = ctx->d_des_ie[comp];
  }
  for (int a = 0; a < 3; a++) { ctx->P.des_lo[a] = lo[a]; ctx->P.des_n[a] = n[a]; }
  ctx->P.des_on = 1;
  return upload_umat(ctx);
}

// device buffers that make up the restartable state of a context
static void state_parts(dtmx_ctx* ctx, std::vector<std::pair<void*, size_t>>& parts) {
  parts.clear();
  for (int comp = 0; comp < 6; comp++) parts.push_back({ctx->P.f[comp], ctx->nstore * 4});
  for (int a = 0; a < 3; a++) {
    const size_t cnt = (size_t)(ctx->P.ab.L[a][0] + ctx->P.ab.L[a][1]) * (ctx->ncell / (size_t)ctx->P.g.n[a]);
    for (int q = 0; q < 4; q++)
      if (ctx->P.ab.aux[a][q]) parts.push_back({ctx->P.ab.aux[a][q], cnt * 4});
  }
  const Ade& A = ctx->P.ade;
  const size_t na = (size_t)A.n[0] * A.n[1] * A.n[2];
  for (int comp = 0; comp < 3 && na; comp++) {
    if (A.Em[comp]) parts.push_back({A.Em[comp], na * 4});
    for (int q = 0; q < MAXPOLE; q++) {
      if (A.Jp[comp][q]) parts.push_back({A.Jp[comp][q], na * 4});
      if (A.Jm[comp][q]) parts.push_back({A.Jm[comp][q], na * 4});
    }
    for (int b = 0; b < 2; b++)
      if (A.Jg[b][comp]) parts.push_back({A.Jg[b][comp], na * 4});
  }
  parts.push_back({ctx->d_step, sizeof(long long)});
  if (ctx->line_e) {
    parts.push_back({ctx->line_e, (size_t)ctx->T.line_n * 8});
    parts.push_back({ctx->line_h, (size_t)ctx->T.line_n * 8});
  }
}

static int state_copy(dtmx_ctx* ctx, char* ck, bool save) {
  std::vector<std::pair<void*, size_t>> parts;
  state_parts(ctx, parts);
  size_t off = 0;
  for (auto& pr : parts) {
    if (save) CK(cudaMemcpyAsync(ck + off, pr.first, pr.second, cudaMemcpyDeviceToDevice, ctx->stream));
    else CK(cudaMemcpyAsync(pr.first, ck + off, pr.second, cudaMemcpyDeviceToDevice, ctx->stream));
    off += (pr.second + 255) / 256 * 256;
  }
  return DTMX_OK;
}

static size_t state_bytes(dtmx_ctx* ctx) {
  std::vector<std::pair<void*, size_t>> parts;
  state_parts(ctx, parts);
  size_t off = 0;
  for (auto& pr : parts) off += (pr.second + 255) / 256 * 256;
  return off;
}

// Forward + adjoint run of one context, split into phases so that a batch of
// contexts can interleave them step by step (each context on its own stream).
struct FaRun {
  int N = 0, K = 0, nseg = 0, nd = 0, npl = 0, plane_x = 0;
  double omega = 0, J = 0;
  long long s0 = 0;
  int gcur0 = 0;              // gyrotropic current buffer at the start (it alternates every step)
  std::vector<char*> ck;
  AdjDev A{};
  float* hist = nullptr;
  double* dF = nullptr;
  int seg = -1, len = 0;
  bool full = false;          // the forward pass records the whole design history: no checkpoints, no recompute
  cudaStream_t st = nullptr;
  std::vector<void*> bufs;
  // single-sweep adjoint: A.lam / A.lpsi are the current set, these the other
  // one (swapped after every step), the maps read set 0 and set 1
  bool sweep = false;
  float* lam_alt[6] = {};
  float* lpsi_alt[3][4] = {};
  FusedMaps fm[2]{};
  // Device buffers of the run come from the device's stream-ordered pool:
  // released blocks stay in the pool (release threshold raised once per
  // process), so later runs -- on this context or a fresh one -- reuse them
  // without a device-wide synchronisation.
  void* take(dtmx_ctx* ctx, size_t bytes) {
    static const bool pool_kept = [] {
      int dev = 0;
      cudaMemPool_t pool;
      if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetDefaultMemPool(&pool, dev) != cudaSuccess) return false;
      uint64_t keep = ~0ull;
      return cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess;
    }();
    (void)pool_kept;
    st = ctx->stream;
    void* q = nullptr;
    cudaError_t e = refuse(ctx, DTMX_FAIL_ALLOC) ? cudaErrorMemoryAllocation : cudaMallocAsync(&q, bytes, ctx->stream);
    while (e != cudaSuccess && free_a_set(ctx, true)) e = cudaMallocAsync(&q, bytes, ctx->stream);
    if (e != cudaSuccess) { cudaGetLastError(); return nullptr; }
    bufs.push_back(q);
    return q;
  }
  void release() {
    for (void* q : bufs) cudaFreeAsync(q, st);
    bufs.clear();
    ck.clear();
  }
};

// Does the design-region E history of a whole run fit the context's budget?
// Then the forward pass records it and the adjoint needs no recomputation.
static double fa_history_bytes(const dtmx_ctx* ctx, int nsteps) {
  const Params& P = ctx->P;
  return (double)(nsteps + 1) * 3.0 * P.des_n[0] * P.des_n[1] * P.des_n[2] * 4.0;
}
// the bytes of an automatic second set: as good as free
static double lent_bytes(const dtmx_ctx* ctx) { return ctx->engine == 0 && ctx->fused_ready && !ctx->cfg.parkable ? fused_set_bytes(ctx) : 0.0; }
static bool fa_history_fits(dtmx_ctx* ctx, int nsteps) {
  const double bytes = fa_history_bytes(ctx, nsteps);
  if (ctx->adj_budget >= 0) return bytes <= (double)ctx->adj_budget;
  return bytes <= 0.25 * (free_device_bytes() + lent_bytes(ctx));
}

// The adjoint as one sweep a step (dtmx_adjsweep.cuh): the Yee stencil without
// gyrotropic material, and no dispersive node in a slab (its taps there would
// be stretched).  Never slower than the two-pass kernels where both apply.
static bool adj_sweep_usable(const dtmx_ctx* ctx) {
  const Params& P = ctx->P;
  if (ctx->cfg.order != 2 || ctx->has_gyro) return false;
  if (P.ade.Em[0])
    for (int a = 0; a < 3; a++)
      if (P.ade.lo[a] < P.ab.L[a][0] || P.ade.lo[a] + P.ade.n[a] > P.g.n[a] - P.ab.L[a][1]) return false;
  return true;
}

// Before a context's first run in a batch: the memory that it will take from the stream-ordered pool, once
// taken and given back on its stream.  The pool then hands it to that stream again; it would otherwise pass
// blocks from stream to stream while kernels run, and each stream waits for the other's (the first
// batch of 16 contexts of 48^3 took 47 ms, with this 22, later ones 11; 8 of 64^3 18.5 and 12).
static void fa_reserve(dtmx_ctx* ctx, int nsteps, bool full) {
  const Params& P = ctx->P;
  double bytes = 12.0 * (ctx->nstore + 64) * 4 + (full ? fa_history_bytes(ctx, nsteps) : 0.0);
  for (int a = 0; a < 3; a++)
    if (P.ab.aux[a][0]) bytes += 8.0 * (P.ab.L[a][0] + P.ab.L[a][1]) * (double)(ctx->ncell / (size_t)P.g.n[a]) * 4;
  if (bytes <= ctx->fa_reserved) return;
  ctx->fa_reserved = bytes;
  void* q = nullptr;
  if (cudaMallocAsync(&q, (size_t)bytes, ctx->stream) == cudaSuccess) cudaFreeAsync(q, ctx->stream);
  else cudaGetLastError();
}

static int fa_begin(dtmx_ctx* ctx, FaRun& R, int nsteps, int checkpoint_every, int plane_x, double omega, bool full) {
  const dtmx_config& c = ctx->cfg;
  Params& P = ctx->P;
  if (nsteps < 1 || checkpoint_every < 1) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  if (!P.des_on) return fail(ctx, DTMX_ERR_STATE, "no design region");
  if (plane_x < 0 || plane_x >= c.nx) return fail(ctx, DTMX_ERR_INVALID, "objective plane outside the grid");
  if (c.geometry != DTMX_GEOM_BOX || c.absorber == DTMX_ABS_SPLIT_PML)
    return fail(ctx, DTMX_ERR_UNSUPPORTED, "the adjoint needs the box geometry with CPML or no absorber");
  if (ctx->has_gyro && !ctx->h_mat[0].empty()) {
    // the design permittivity of a gyrotropic node would enter next to its current: not carried
    for (int comp = 0; comp < 3; comp++)
      for (int i = P.des_lo[0]; i < P.des_lo[0] + P.des_n[0]; i++)
        for (int j = P.des_lo[1]; j < P.des_lo[1] + P.des_n[1]; j++)
          for (int k = P.des_lo[2]; k < P.des_lo[2] + P.des_n[2]; k++)
            if (ctx->mats[ctx->h_mat[comp][store_index(ctx, i, j, k)]].gyro_wp > 0)
              return fail(ctx, DTMX_ERR_UNSUPPORTED, "the design region holds a gyrotropic node");
  }
  for (const auto& q : ctx->psrc) {
    const long long sz = ctx->nzp, sy = (long long)c.ny * sz;
    const int i = (int)(q.id / sy), j = (int)((q.id % sy) / sz), k = (int)(q.id % sz);
    if (design_index(P, i, j, k) >= 0) return fail(ctx, DTMX_ERR_INVALID, "a point source lies in the design region");
  }
  int rc = prepare(ctx);
  if (rc) return rc;
  R.full = full;
  R.N = nsteps; R.K = full ? nsteps : std::min(checkpoint_every, nsteps);
  R.nseg = (R.N + R.K - 1) / R.K;
  R.nd = P.des_n[0] * P.des_n[1] * P.des_n[2];
  R.npl = c.ny * c.nz;
  R.plane_x = plane_x; R.omega = omega;
  // objective flux DFT on the plane x = plane_x: Ey, Ez, Hy, Hz at omega
  DftHost& O = ctx->obj;
  if (!ctx->objmon.tab || O.d.index != plane_x) {
    mon_free(ctx->objmon);
    dft_free(O);
    O = DftHost{};
    O.d.axis = 0; O.d.index = plane_x; O.d.comp_mask = (1 << 1) | (1 << 2) | (1 << 4) | (1 << 5); O.d.nfreq = 1;
    O.d.n1 = c.ny; O.d.n2 = c.nz; O.ncomp = 4;
    if (!dft_malloc(ctx, O, 1, (size_t)4 * R.npl, (size_t)DFT_STAGE * 4 * R.npl)) return fail(ctx, DTMX_ERR_OOM, "objective DFT allocation");
    O.d.omega = O.omega; O.d.acc = O.acc; O.d.stage = O.stage; O.d.sstep = O.sstep;
    if ((rc = mon_build(ctx, ctx->objmon, &O, 1))) return rc;
  }
  CK(cudaMemcpyAsync(O.omega, &omega, 8, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaMemsetAsync(O.acc, 0, (size_t)4 * R.npl * sizeof(double2), ctx->stream));
  ctx->objmon.nstaged = 0;
  if (full) {
    // design-region history of every step: slot s holds E after s steps of the run
    void* h = R.take(ctx, (size_t)(R.N + 1) * 3 * R.nd * 4);
    if (!h) return fail(ctx, DTMX_ERR_OOM, "design history allocation");
    R.hist = (float*)h;
  } else {
    // checkpoints of the state every K steps plus the final state
    const size_t sb = state_bytes(ctx);
    R.ck.assign(R.nseg + 1, nullptr);
    for (auto& q : R.ck)
      if (!(q = (char*)R.take(ctx, sb))) { R.release(); return fail(ctx, DTMX_ERR_OOM, "checkpoint allocation"); }
  }
  R.s0 = ctx->step;
  R.gcur0 = ctx->gcur;
  ctx->obj_on = true;
  return DTMX_OK;
}

static unsigned design_blocks(const FaRun& R) { return (unsigned)((3 * R.nd + 255) / 256); }

// forward step st (0-based) of the run
static int fa_forward(dtmx_ctx* ctx, FaRun& R, int st) {
  if (R.full) {
    if (st == 0) {
      launch(ctx, false, design_capture_kernel, design_blocks(R), 256, 0, ctx->stream, ctx->P, R.hist, 0, R.nd);
      ctx->launches++;
    }
  } else if (st % R.K == 0) {
    state_copy(ctx, R.ck[st / R.K], true);
  }
  if (R.full) ctx->hist_out = R.hist + (size_t)(st + 1) * 3 * R.nd;
  int rc = launch_one(ctx);                      // (reports the launch above too)
  ctx->hist_out = nullptr;
  if (rc) return rc;
  ctx->step++;
  return DTMX_OK;
}

// end of the forward pass: objective, adjoint buffers (waits for the stream)
static int fa_forward_done(dtmx_ctx* ctx, FaRun& R) {
  Params& P = ctx->P;
  ctx->obj_on = false;
  if (!R.full) state_copy(ctx, R.ck[R.nseg], true);
  DftHost& O = ctx->obj;
  dft_flush(ctx, ctx->objmon);
  if (int rc = launched(ctx)) return rc;
  std::vector<double> F((size_t)8 * R.npl);
  CK(cudaMemcpyAsync(F.data(), O.acc, F.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  double J = 0;
  for (int u = 0; u < R.npl; u++) {
    const double *ey = &F[(0 * (size_t)R.npl + u) * 2], *ez = &F[(1 * (size_t)R.npl + u) * 2];
    const double *hy = &F[(2 * (size_t)R.npl + u) * 2], *hz = &F[(3 * (size_t)R.npl + u) * 2];
    J += ey[0] * hz[0] + ey[1] * hz[1] - (ez[0] * hy[0] + ez[1] * hy[1]);
  }
  R.J = J;
  AdjDev& A = R.A;
  A = AdjDev{};
  A.nd = R.nd;
  auto talloc = [&](void** q, size_t bytes) {
    if (!(*q = R.take(ctx, bytes))) return false;
    return cudaMemsetAsync(*q, 0, bytes, ctx->stream) == cudaSuccess;
  };
  bool ok = true;
  R.sweep = adj_sweep_usable(ctx);
  for (int comp = 0; comp < 6; comp++) ok = ok && talloc((void**)&A.lam[comp], (ctx->nstore + 64) * 4);
  for (int a = 0; a < 3; a++) {
    const size_t cnt = (size_t)(P.ab.L[a][0] + P.ab.L[a][1]) * (ctx->ncell / (size_t)P.g.n[a]);
    if (!P.ab.aux[a][0]) continue;
    for (int q = 0; q < 4; q++) ok = ok && talloc((void**)&A.lpsi[a][q], cnt * 4);
  }
  // six more field arrays: the sweep's second set, or the two-pass kernels' w
  float* six[6] = {};
  for (int comp = 0; comp < 6; comp++) ok = ok && talloc((void**)&six[comp], (ctx->nstore + 64) * 4);
  if (ctx->has_gyro) {
    const size_t na = (size_t)P.ade.n[0] * P.ade.n[1] * P.ade.n[2];
    for (int c3 = 0; c3 < 3; c3++) ok = ok && talloc((void**)&A.lJg[c3], na * 4) && talloc((void**)&A.lT[c3], na * 4);
  }
  if (P.ade.Em[0]) {
    // adjoint of the ADE state, over the ADE box
    const size_t na = (size_t)P.ade.n[0] * P.ade.n[1] * P.ade.n[2];
    for (int c3 = 0; c3 < 3; c3++) {
      ok = ok && talloc((void**)&A.lEm[c3], na * 4);
      for (int r = 0; r < MAXPOLE; r++)
        if (P.ade.Jp[c3][r]) ok = ok && talloc((void**)&A.lJp[c3][r], na * 4) && talloc((void**)&A.lJm[c3][r], na * 4);
    }
  }
  ok = ok && talloc((void**)&A.grad, (size_t)3 * R.nd * 8) && talloc((void**)&R.dF, F.size() * 8);
  if (!R.full) ok = ok && talloc((void**)&R.hist, (size_t)(R.K + 1) * 3 * R.nd * 4);
  if (!ok) { R.release(); return fail(ctx, DTMX_ERR_OOM, "adjoint allocation"); }
  // what the sweep needs beyond the two-pass kernels' arrays comes last: without room for it they serve
  for (int a = 0; a < 3 && R.sweep; a++)
    for (int q = 0; q < 4 && R.sweep && P.ab.aux[a][0]; q++)
      R.sweep = talloc((void**)&R.lpsi_alt[a][q], (size_t)(P.ab.L[a][0] + P.ab.L[a][1]) * (ctx->ncell / (size_t)P.g.n[a]) * 4);
  for (int c3 = 0; c3 < 3 && R.sweep && P.ade.Em[0]; c3++)
    R.sweep = talloc((void**)&A.lE[c3], (size_t)P.ade.n[0] * P.ade.n[1] * P.ade.n[2] * 4);
  for (int comp = 0; comp < 6; comp++) (R.sweep ? R.lam_alt[comp] : A.w[comp / 2][comp % 2]) = six[comp];
  A.hist = R.hist;
  if (R.sweep) {
    int rc;
    if ((rc = build_fused_maps<16>(ctx, R.fm[0], A.lam)) || (rc = build_fused_maps<16>(ctx, R.fm[1], R.lam_alt))) return rc;
    if (cudaFuncSetAttribute(adj_sweep_kernel<16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AL<16>::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(adj_sweep_kernel<16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AL<16>::SMEM) != cudaSuccess)
      return fail(ctx, DTMX_ERR_CUDA, "adjoint sweep: shared memory attribute");
  }
  CK(cudaMemcpyAsync(R.dF, F.data(), F.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->monitors_off = true;
  return DTMX_OK;
}

// restore checkpoint seg and record the design region of its first state
// (with the whole history recorded: the one segment is the run, nothing to restore)
static int fa_segment_begin(dtmx_ctx* ctx, FaRun& R, int seg) {
  R.seg = seg;
  const int start = seg * R.K;
  R.len = std::min(R.N, start + R.K) - start;
  if (R.full) return DTMX_OK;
  state_copy(ctx, R.ck[seg], false);
  ctx->step = R.s0 + start;
  ctx->gcur = R.gcur0 ^ (start & 1);
  launch(ctx, false, design_capture_kernel, design_blocks(R), 256, 0, ctx->stream, ctx->P, R.hist, 0, R.nd);
  return launched(ctx);
}

// recompute step q (1..len) of the current segment
static int fa_recompute(dtmx_ctx* ctx, FaRun& R, int q) {
  if (R.full) return DTMX_OK;
  ctx->hist_out = R.hist + (size_t)q * 3 * R.nd;
  int rc = launch_one(ctx);
  ctx->hist_out = nullptr;
  if (rc) return rc;
  ctx->step++;
  return DTMX_OK;
}

// adjoint of step q (len..1) of the current segment
static int fa_adjoint(dtmx_ctx* ctx, FaRun& R, int q) {
  const Params& P = ctx->P;
  const dtmx_config& c = ctx->cfg;
  AdjDev& A = R.A;
  cudaStream_t st = ctx->stream;
  if (R.sweep) {
    const long long s = R.s0 + (long long)R.seg * R.K + q;
    const int ns = (R.npl + 255) / 256, ng = (int)design_blocks(R);
    // the sources and the gradient share a launch unless the plane cuts the design region
    if (R.plane_x >= P.des_lo[0] && R.plane_x < P.des_lo[0] + P.des_n[0]) {
      launch(ctx, ctx->early, adj_pre_kernel, ns, 256, 0, st, P, A, R.dF, s, R.plane_x, R.omega, c.dt, ns, q);
      launch(ctx, ctx->early, adj_pre_kernel, ng, 256, 0, st, P, A, R.dF, s, R.plane_x, R.omega, c.dt, 0, q);
      ctx->launches++;
    } else {
      launch(ctx, ctx->early, adj_pre_kernel, ns + ng, 256, 0, st, P, A, R.dF, s, R.plane_x, R.omega, c.dt, ns, q);
    }
    if (P.ade.Em[0]) {
      launch(ctx, ctx->early, adj_ade_sweep_kernel, ade_grid(P), 256, 0, st, P, A);
      ctx->launches++;
    }
    Params PS = P;
    const WorkPlan* wp;
    if (int rc = plan_work(ctx, WK_ADJ, 16, 3, 0, &wp)) return rc;
    const WorkPlan& plan = *wp;
    PS.xchunk = plan.xchunk;
    AdjSweepArgs sa{};
    for (int comp = 0; comp < 6; comp++) sa.dst[comp] = R.lam_alt[comp];
    for (int a = 0; a < 3; a++)
      for (int k = 0; k < 4; k++) { sa.psrc[a][k] = A.lpsi[a][k]; sa.pdst[a][k] = R.lpsi_alt[a][k]; }
    const dim3 grd = plan.grid;
    if (plan.table) launch(ctx, ctx->early, adj_sweep_kernel<16, true>, grd, FL<16>::NT, AL<16>::SMEM, st, PS, sa, R.fm[0], plan.work);
    else launch(ctx, ctx->early, adj_sweep_kernel<16, false>, grd, FL<16>::NT, AL<16>::SMEM, st, PS, sa, R.fm[0], Work<false>{});
    ctx->launches += 2;
    for (int comp = 0; comp < 6; comp++) std::swap(A.lam[comp], R.lam_alt[comp]);
    for (int a = 0; a < 3; a++)
      for (int k = 0; k < 4; k++) std::swap(A.lpsi[a][k], R.lpsi_alt[a][k]);
    std::swap(R.fm[0], R.fm[1]);
    return launched(ctx);
  }
  launch(ctx, false, adj_source_kernel, (R.npl + 255) / 256, 256, 0, st, P, A, R.dF, R.s0 + (long long)R.seg * R.K + q, R.plane_x, R.omega, c.dt);
  launch(ctx, false, adj_grad_kernel, design_blocks(R), 256, 0, st, P, A, q);
  const dim3 blk(32, 8), grd((c.nz + 31) / 32, (c.ny + 7) / 8, c.nx);
  const dim3 wgrd((c.nz + 31) / 32, (c.ny + 7) / 8, (c.nx + ADJ_XP - 1) / ADJ_XP);   // adj_w: ADJ_XP planes per thread
  // the dispersive nodes' transposed ADE recursion replaces their w (after adj_w, before adj_curl);
  // the gyrotropic current's transposition reads lam_E' (after adj_w) and gathers over the box
  const bool ade = P.ade.Em[0] != nullptr;
  const bool gyro = ctx->has_gyro;
  const int ablk = 256;
  const dim3 agrd = ade_grid(P);
  if (c.order == 4) {
    launch(ctx, false, adj_w_kernel<4, 0>, wgrd, blk, 0, st, P, A);
    if (ade) launch(ctx, false, adj_ade_kernel, agrd, ablk, 0, st, P, A);
    if (gyro) { launch(ctx, false, adj_gyro_mu_kernel, agrd, ablk, 0, st, P, A); launch(ctx, false, adj_gyro_j_kernel, agrd, ablk, 0, st, P, A); }
    launch(ctx, false, adj_curl_kernel<4, 0>, grd, blk, 0, st, P, A);
    launch(ctx, false, adj_w_kernel<4, 1>, wgrd, blk, 0, st, P, A);
    launch(ctx, false, adj_curl_kernel<4, 1>, grd, blk, 0, st, P, A);
    ctx->launches += 6 + (ade ? 1 : 0) + (gyro ? 2 : 0);
  } else {
    launch(ctx, false, adj_w_kernel<2, 0>, wgrd, blk, 0, st, P, A);
    if (ade) launch(ctx, false, adj_ade_kernel, agrd, ablk, 0, st, P, A);
    if (gyro) { launch(ctx, false, adj_gyro_mu_kernel, agrd, ablk, 0, st, P, A); launch(ctx, false, adj_gyro_j_kernel, agrd, ablk, 0, st, P, A); }
    launch(ctx, false, adj_curl_kernel<2, 0>, grd, blk, 0, st, P, A);
    launch(ctx, false, adj_w_kernel<2, 1>, wgrd, blk, 0, st, P, A);
    launch(ctx, false, adj_curl_kernel<2, 1>, grd, blk, 0, st, P, A);
    ctx->launches += 6 + (ade ? 1 : 0) + (gyro ? 2 : 0);
  }
  return launched(ctx);
}

// final state back in place, gradient to the caller (waits for the stream)
static int fa_finish(dtmx_ctx* ctx, FaRun& R, double* objective, float* grad_eps) {
  ctx->monitors_off = false;
  if (!R.full) state_copy(ctx, R.ck[R.nseg], false);
  ctx->step = R.s0 + R.N;
  ctx->gcur = R.gcur0 ^ (R.N & 1);
  std::vector<double> g((size_t)3 * R.nd);
  CK(cudaMemcpyAsync(g.data(), R.A.grad, g.size() * 8, cudaMemcpyDeviceToHost, ctx->stream));
  cudaError_t e = cudaStreamSynchronize(ctx->stream);
  R.release();
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("adjoint: ") + cudaGetErrorString(e));
  for (int comp = 0; comp < 3; comp++)
    for (int q = 0; q < R.nd; q++) {
      const double ie = ctx->h_des_ie[comp][q];
      grad_eps[(size_t)comp * R.nd + q] = (float)(-ie * ie * g[(size_t)comp * R.nd + q]);
    }
  *objective = R.J;
  return DTMX_OK;
}

static void fa_abort(dtmx_ctx* ctx, FaRun& R) {
  cudaStreamSynchronize(ctx->stream);
  ctx->obj_on = false;
  ctx->monitors_off = false;
  R.release();
}

extern "C" int dtmx_forward_adjoint(dtmx_ctx* ctx, int nsteps, int checkpoint_every, int plane_x, double omega,
                                    double* objective, float* grad_eps) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !objective || !grad_eps) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  const Running running(ctx);
  FaRun R;
  if (nsteps < 1 || checkpoint_every < 1) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  int rc = fa_begin(ctx, R, nsteps, checkpoint_every, plane_x, omega, fa_history_fits(ctx, nsteps));
  if (rc) return rc;
  for (int st = 0; st < R.N && !rc; st++) rc = fa_forward(ctx, R, st);
  if (!rc) rc = fa_forward_done(ctx, R);
  for (int seg = R.nseg - 1; seg >= 0 && !rc; seg--) {
    rc = fa_segment_begin(ctx, R, seg);
    for (int q = 1; q <= R.len && !rc; q++) rc = fa_recompute(ctx, R, q);
    for (int q = R.len; q >= 1 && !rc; q--) rc = fa_adjoint(ctx, R, q);
  }
  if (rc) { fa_abort(ctx, R); return rc; }
  return fa_finish(ctx, R, objective, grad_eps);
}

extern "C" int dtmx_set_adjoint_memory(dtmx_ctx* ctx, int64_t bytes) {
  if (!ctx) return DTMX_ERR_INVALID;
  ctx->adj_budget = bytes < 0 ? -1 : (long long)bytes;
  return DTMX_OK;
}

// Batch of independent forward + adjoint runs: every phase is issued for all
// contexts step by step, each context on its own stream, so that the GPU runs
// the instances' kernels concurrently (instances of uneven sizes fill each
// other's gaps) and no instance waits on the host between its steps.
extern "C" int dtmx_batch_forward_adjoint(dtmx_ctx* const* ctxs, int n, int nsteps, int checkpoint_every,
                                          const int* plane_x, const double* omega, double* objectives,
                                          float* const* grads) {
  if (!ctxs || n < 1 || !plane_x || !omega || !objectives || !grads) return DTMX_ERR_INVALID;
  for (int b = 0; b < n; b++)
    if (ctxs[b] && ctxs[b]->parked) return fail(ctxs[b], DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  std::vector<Running> running;
  running.reserve(n);
  for (int b = 0; b < n; b++) running.emplace_back(ctxs[b]);
  std::vector<FaRun> R(n);
  // one context's early launches would hold room that another's kernels need
  struct Plain {
    dtmx_ctx* const* c;
    std::vector<char> was;
    Plain(dtmx_ctx* const* cs, int n) : c(cs), was(n) {
      for (int b = 0; b < n; b++)
        if (c[b]) { was[b] = c[b]->early; if (n > 1) c[b]->early = false; }
    }
    ~Plain() {
      for (size_t b = 0; b < was.size(); b++)
        if (c[b]) c[b]->early = was[b];
    }
  } plain(ctxs, n);
  int rc = DTMX_OK;
  auto abort_all = [&](int upto) {
    for (int b = 0; b < upto; b++) fa_abort(ctxs[b], R[b]);
  };
  // one mode for the whole batch (the segments advance in lock step)
  bool full = nsteps >= 1;
  double total = 0.0, lent = 0.0;
  bool automatic = true;
  for (int b = 0; b < n; b++) {
    full = full && ctxs[b] && fa_history_fits(ctxs[b], nsteps);
    if (!full) break;
    total += fa_history_bytes(ctxs[b], nsteps);
    lent += lent_bytes(ctxs[b]);
    automatic = automatic && ctxs[b]->adj_budget < 0;
  }
  if (full && automatic) full = total <= 0.25 * (free_device_bytes() + lent);
  for (int b = 0; b < n && n > 1; b++)
    if (ctxs[b]) fa_reserve(ctxs[b], nsteps, full);
  for (int b = 0; b < n; b++)
    if ((rc = fa_begin(ctxs[b], R[b], nsteps, checkpoint_every, plane_x[b], omega[b], full))) { abort_all(b); return rc; }
  for (int st = 0; st < nsteps && !rc; st++)
    for (int b = 0; b < n && !rc; b++) rc = fa_forward(ctxs[b], R[b], st);
  for (int b = 0; b < n && !rc; b++) rc = fa_forward_done(ctxs[b], R[b]);
  const int nseg = R[0].nseg;
  for (int seg = nseg - 1; seg >= 0 && !rc; seg--) {
    for (int b = 0; b < n && !rc; b++) rc = fa_segment_begin(ctxs[b], R[b], seg);
    const int len = R[0].len;
    for (int q = 1; q <= len && !rc; q++)
      for (int b = 0; b < n && !rc; b++) rc = fa_recompute(ctxs[b], R[b], q);
    for (int q = len; q >= 1 && !rc; q--)
      for (int b = 0; b < n && !rc; b++) rc = fa_adjoint(ctxs[b], R[b], q);
  }
  if (rc) { abort_all(n); return rc; }
  for (int b = 0; b < n; b++) {
    int r = fa_finish(ctxs[b], R[b], &objectives[b], grads[b]);
    if (r && !rc) rc = r;
  }
  return rc;
}

// ---------------------------------------------------------------- autotuner
// Times every applicable engine configuration for trial_steps steps from the
// current state (monitors paused, state restored after each trial) and keeps
// the fastest: the per-step engine with x chunks of {auto, 4, 8, 16, 32, 64}
// planes per CTA, and the wavefront engine with 1, 2 and 4 steps per launch.
// Results are cached per grid shape and feature set for the process.
struct TuneKey {
  int nx, ny, nz, order, absorber, geometry, feats;
  bool operator<(const TuneKey& o) const {
    return std::tie(nx, ny, nz, order, absorber, geometry, feats) < std::tie(o.nx, o.ny, o.nz, o.order, o.absorber, o.geometry, o.feats);
  }
};
struct TuneVal { int engine, tblock, xchunk; double ms; int rows = 16; };
static std::map<TuneKey, TuneVal>& tune_cache() {
  static std::map<TuneKey, TuneVal> m;
  return m;
}

extern "C" int dtmx_autotune(dtmx_ctx* ctx, int trial_steps, int* engine_out, int* tblock_out, int* xchunk_out,
                             double* ms_per_step_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || trial_steps < 1) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  const Running running(ctx);
  int rc = prepare(ctx);
  if (rc) return rc;
  const dtmx_config& c = ctx->cfg;
  const int feats = (ctx->has_tfsf ? 1 : 0) | (ctx->psrc.empty() ? 0 : 2) | (ctx->probes.empty() ? 0 : 4) |
                    (ctx->dfts.empty() ? 0 : 8) | (ctx->P.ade.Em[0] ? 16 : 0) | (ctx->has_gyro ? 32 : 0) |
                    (ctx->P.des_on ? 64 : 0);
  const TuneKey key{c.nx, c.ny, c.nz, c.order, c.absorber, c.geometry, feats};
  TuneVal best{1, 0, 0, 1e30};
  auto it = tune_cache().find(key);
  if (it != tune_cache().end()) {
    best = it->second;
  } else {
    char* ck = nullptr;
    if (dev_malloc(ctx, &ck, state_bytes(ctx)) != cudaSuccess) return fail(ctx, DTMX_ERR_OOM, "autotune state copy");
    state_copy(ctx, ck, true);
    const long long step0 = ctx->step;
    const int gcur0 = ctx->gcur, eng0 = ctx->engine, tb0 = ctx->tblock, xc0 = ctx->xchunk, fr0 = ctx->frows;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    std::vector<TuneVal> cand;
    for (int xc : {0, 4, 6, 8, 10, 12, 16, 24, 32, 64})
      if (xc <= c.nx) cand.push_back({1, 0, xc, 0});
    if (fused_usable(ctx, nullptr) && fused_prepare(ctx) == DTMX_OK)
      for (int rows : {16, 8})
        for (int xc : {0, 2, 4, 6, 8, 12, 16, 24, 32, 48, 64})
          if (xc <= c.nx) cand.push_back({3, 0, xc, 0, rows});
    std::string why;
    if (torre_features_ok(ctx, &why))
      for (int T : {1, 2, 4})
        if (trial_steps >= T && torre_usable(ctx, T, &why)) cand.push_back({2, T, 0, 0});
    ctx->monitors_off = true;
    for (auto& cd : cand) {
      ctx->xchunk = cd.xchunk;
      ctx->engine = cd.engine;
      ctx->frows = cd.rows;
      int r = DTMX_OK;
      const int n = cd.engine == 2 ? (trial_steps / cd.tblock) * cd.tblock : trial_steps;
      // (the work table is made outside the timed steps)
      if (cd.engine == 1) r = plan_stream(ctx, nullptr);
      else if (cd.engine == 3) r = plan_sweep(ctx, nullptr);
      cudaEventRecord(e0, ctx->stream);
      if (cd.engine == 2) {
        for (int q = 0; q < n && !r; q += cd.tblock) r = launch_torre(ctx, cd.tblock);
      } else {
        for (int q = 0; q < n && !r; q++) { r = launch_one(ctx); ctx->step++; }
      }
      cudaEventRecord(e1, ctx->stream);
      cudaEventSynchronize(e1);
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      cd.ms = r ? 1e30 : ms / n;
      if (r) cudaGetLastError();
      state_copy(ctx, ck, false);
      ctx->step = step0;
      ctx->gcur = gcur0;
      if (cd.ms < best.ms) best = cd;
    }
    ctx->monitors_off = false;
    CK(cudaStreamSynchronize(ctx->stream));
    cudaFree(ck);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    ctx->engine = eng0; ctx->tblock = tb0; ctx->xchunk = xc0; ctx->frows = fr0;
    tune_cache()[key] = best;
  }
  ctx->engine = best.engine;
  ctx->tblock = best.tblock;
  ctx->xchunk = best.xchunk;
  ctx->frows = best.rows;
  drop_graphs(ctx);
  if (engine_out) *engine_out = best.engine;
  if (tblock_out) *tblock_out = best.tblock;
  if (xchunk_out) *xchunk_out = best.xchunk;
  if (ms_per_step_out) *ms_per_step_out = best.ms;
  return DTMX_OK;
}

// ---------------------------------------------------------------- field and state files
// Field snapshot in the reference's .arr layout (drop.cu:84-107): int32 header
// {12, 0, 0, 0, 3, sizeof(float), nz, ny, nx} (a 12-byte comment of zeros, the
// rank, the element size and the extents, fastest first), then the values
// with z fastest and x slowest; dense cells instead of the reference's one
// value per rag.
extern "C" int dtmx_write_arr(dtmx_ctx* ctx, int comp, const char* path) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || comp < 0 || comp > 5 || !path) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  const dtmx_config& c = ctx->cfg;
  std::vector<float> buf((size_t)c.nx * c.ny * c.nz);
  int rc = dtmx_get_field(ctx, comp, buf.data());
  if (rc) return rc;
  FILE* f = fopen(path, "wb");
  if (!f) return fail(ctx, DTMX_ERR_INVALID, std::string("cannot open ") + path);
  const int32_t hdr[9] = {12, 0, 0, 0, 3, (int32_t)sizeof(float), c.nz, c.ny, c.nx};
  const bool ok = fwrite(hdr, sizeof(hdr), 1, f) == 1 && fwrite(buf.data(), 4, buf.size(), f) == buf.size();
  if (fclose(f) != 0 || !ok) return fail(ctx, DTMX_ERR_INVALID, std::string("write failed: ") + path);
  return DTMX_OK;
}

// Restartable state file: a header (magic, version, grid, order, geometry,
// absorber, step, byte count) and the device state of the context (fields,
// absorber and ADE state, step counter, plane-wave line), so that loading it
// into a context set up the same way and stepping on reproduces the saved run
// bit for bit.  Probe traces and DFT accumulators are not part of it.
struct StateHeader {
  char magic[8];
  int32_t version, nx, ny, nz, order, geometry, absorber, pad;
  int64_t step, bytes;
};

extern "C" int dtmx_save_state(dtmx_ctx* ctx, const char* path) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !path) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  int rc = prepare(ctx);
  if (rc) return rc;
  const Running running(ctx);
  const size_t sb = state_bytes(ctx);
  char* dev = nullptr;
  if (dev_malloc(ctx, &dev, sb) != cudaSuccess) return fail(ctx, DTMX_ERR_OOM, "state buffer");
  state_copy(ctx, dev, true);
  std::vector<char> host(sb);
  cudaError_t e = cudaMemcpyAsync(host.data(), dev, sb, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(dev);
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("state copy: ") + cudaGetErrorString(e));
  const dtmx_config& c = ctx->cfg;
  StateHeader h{};
  memcpy(h.magic, "DTMXSTAT", 8);
  h.version = 1; h.nx = c.nx; h.ny = c.ny; h.nz = c.nz; h.order = c.order; h.geometry = c.geometry;
  h.absorber = c.absorber; h.step = ctx->step; h.bytes = (int64_t)sb;
  FILE* f = fopen(path, "wb");
  if (!f) return fail(ctx, DTMX_ERR_INVALID, std::string("cannot open ") + path);
  const bool ok = fwrite(&h, sizeof(h), 1, f) == 1 && fwrite(host.data(), 1, sb, f) == sb;
  if (fclose(f) != 0 || !ok) return fail(ctx, DTMX_ERR_INVALID, std::string("write failed: ") + path);
  return DTMX_OK;
}

extern "C" int dtmx_load_state(dtmx_ctx* ctx, const char* path) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || !path) return fail(ctx, DTMX_ERR_INVALID, "bad arguments");
  int rc = prepare(ctx);
  if (rc) return rc;
  FILE* f = fopen(path, "rb");
  if (!f) return fail(ctx, DTMX_ERR_INVALID, std::string("cannot open ") + path);
  StateHeader h{};
  const size_t sb = state_bytes(ctx);
  const dtmx_config& c = ctx->cfg;
  if (fread(&h, sizeof(h), 1, f) != 1 || memcmp(h.magic, "DTMXSTAT", 8) != 0 || h.version != 1) {
    fclose(f);
    return fail(ctx, DTMX_ERR_INVALID, "not a state file");
  }
  if (h.nx != c.nx || h.ny != c.ny || h.nz != c.nz || h.order != c.order || h.geometry != c.geometry ||
      h.absorber != c.absorber || h.bytes != (int64_t)sb) {
    fclose(f);
    return fail(ctx, DTMX_ERR_INVALID, "state file does not match this context (grid, scheme or state layout)");
  }
  std::vector<char> host(sb);
  const bool ok = fread(host.data(), 1, sb, f) == sb;
  fclose(f);
  if (!ok) return fail(ctx, DTMX_ERR_INVALID, "truncated state file");
  const Running running(ctx);
  char* dev = nullptr;
  if (dev_malloc(ctx, &dev, sb) != cudaSuccess) return fail(ctx, DTMX_ERR_OOM, "state buffer");
  cudaError_t e = cudaMemcpyAsync(dev, host.data(), sb, cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) { state_copy(ctx, dev, false); e = cudaStreamSynchronize(ctx->stream); }
  cudaFree(dev);
  if (e != cudaSuccess) return fail(ctx, DTMX_ERR_CUDA, std::string("state copy: ") + cudaGetErrorString(e));
  ctx->step = h.step;
  // the host-side parity of the gyrotropic current buffers follows the step count
  if (ctx->has_gyro) ctx->gcur = (int)(h.step & 1);
  return DTMX_OK;
}

extern "C" int dtmx_sync(dtmx_ctx* ctx) {
  if (!ctx) return DTMX_ERR_INVALID;
  CK(cudaStreamSynchronize(ctx->stream));
  int err = 0;
  CK(cudaMemcpy(&err, ctx->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    CK(cudaMemset(ctx->d_err, 0, sizeof(int)));
    return fail(ctx, DTMX_ERR_TIMEOUT, err == 2 ? "a wavefront tile waited too long for its neighbours"
                                                : "a staged load did not arrive in time");
  }
  return DTMX_OK;
}

extern "C" int dtmx_get_step(const dtmx_ctx* ctx, int64_t* n) {
  if (!ctx || !n) return DTMX_ERR_INVALID;
  *n = ctx->step;
  return DTMX_OK;
}

// Device memory for the dense copy of a field whose rows are padded: up to 4 MB a
// block that the context keeps, above that one from the stream's pool, given
// back after the call.  (A block from the pool costs 0.4 ms a call, which a
// larger field's copy outweighs: set_field of 48^3 cells took 450 us with it,
// 160 by the driver's strided copy and 49 with the kept one, of 100^3 660, 1160 and
// 240; of 149x93x211, from the pool, 1.1 ms against 3.3.)
// No block: the strided copy.
constexpr size_t kDenseKept = 4 << 20;
struct DenseBlock {
  dtmx_ctx* ctx;
  float* p = nullptr;
  size_t rows;
  bool kept;
  DenseBlock(dtmx_ctx* c) : ctx(c), rows(dense_rows(c->cfg.nz, (size_t)c->cfg.nx * c->cfg.ny)) {
    const size_t bytes = rows * c->cfg.nz * 4;
    kept = bytes <= kDenseKept;
    if (kept && !c->dense) {
      const bool spare = c->spare_others;
      c->spare_others = true;
      dev_malloc(c, &c->dense, bytes);
      c->spare_others = spare;
    }
    if (kept) p = c->dense;
    else if (refuse(c, DTMX_FAIL_ALLOC) || cudaMallocAsync((void**)&p, bytes, c->stream) != cudaSuccess) { cudaGetLastError(); p = nullptr; }
  }
  ~DenseBlock() {
    if (p && !kept) cudaFreeAsync(p, ctx->stream);
  }
};

extern "C" int dtmx_get_field(dtmx_ctx* ctx, int comp, float* host_out) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || comp < 0 || comp > 5 || !host_out) return fail(ctx, DTMX_ERR_INVALID, "bad field request");
  const dtmx_config& c = ctx->cfg;
  const size_t rows = (size_t)c.nx * c.ny;
  const DeviceGuard guard(ctx->dev);
  if (c.nz == ctx->nzp) return copy_out(ctx, host_out, ctx->P.f[comp], rows * c.nz * 4);
  const DenseBlock block(ctx);
  float* const dense = block.p;
  const size_t per = block.rows;
  if (!dense) {
    CK(cudaStreamSynchronize(ctx->stream));
    CK(cudaMemcpy2D(host_out, (size_t)c.nz * 4, ctx->P.f[comp], (size_t)ctx->nzp * 4, (size_t)c.nz * 4, rows, cudaMemcpyDeviceToHost));
    return DTMX_OK;
  }
  int rc = DTMX_OK;
  for (size_t r = 0; r < rows && !rc; r += per) {
    const size_t n = std::min(per, rows - r);
    launch(ctx, false, dense_rows_kernel, 148 * 8, dim3(32, 8), 0, ctx->stream, ctx->P.f[comp] + r * ctx->nzp, ctx->nzp, dense, c.nz, (long long)n, c.nz);
    ctx->launches++;
    if (!(rc = launched(ctx))) rc = copy_out(ctx, host_out + r * c.nz, dense, n * c.nz * 4);
  }
  return rc;
}

extern "C" int dtmx_set_field(dtmx_ctx* ctx, int comp, const float* host_in) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || comp < 0 || comp > 5 || !host_in) return fail(ctx, DTMX_ERR_INVALID, "bad field request");
  const dtmx_config& c = ctx->cfg;
  const size_t rows = (size_t)c.nx * c.ny;
  if (c.nz != ctx->nzp) {
    const DenseBlock block(ctx);
    float* const dense = block.p;
    const size_t per = block.rows;
    cudaError_t e = cudaSuccess;
    if (!dense) e = cudaMemcpy2DAsync(ctx->P.f[comp], (size_t)ctx->nzp * 4, host_in, (size_t)c.nz * 4, (size_t)c.nz * 4, rows, cudaMemcpyHostToDevice, ctx->stream);
    for (size_t r = 0; dense && r < rows && e == cudaSuccess; r += per) {
      const size_t n = std::min(per, rows - r);
      e = cudaMemcpyAsync(dense, host_in + r * c.nz, n * c.nz * 4, cudaMemcpyHostToDevice, ctx->stream);
      launch(ctx, false, dense_rows_kernel, 148 * 8, dim3(32, 8), 0, ctx->stream, dense, c.nz, ctx->P.f[comp] + r * ctx->nzp, ctx->nzp, (long long)n, c.nz);
      ctx->launches++;
    }
    CK(e);
  } else {
    CK(cudaMemcpyAsync(ctx->P.f[comp], host_in, rows * c.nz * 4, cudaMemcpyHostToDevice, ctx->stream));
  }
  // non-live nodes are held at zero
  launch(ctx, false, mask_nonlive_kernel, 148 * 4, 256, 0, ctx->stream, ctx->P, comp, (long long)ctx->ncell);
  ctx->launches++;
  CK(cudaStreamSynchronize(ctx->stream));
  return launched(ctx);
}

extern "C" int dtmx_field_current_ptr(dtmx_ctx* ctx, int comp, void** dptr, int64_t strides[3]) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || comp < 0 || comp > 5 || !dptr) return fail(ctx, DTMX_ERR_INVALID, "bad field request");
  *dptr = ctx->P.f[comp];
  if (strides) { strides[0] = ctx->P.g.sx; strides[1] = ctx->P.g.sy; strides[2] = 1; }
  return DTMX_OK;
}

extern "C" int dtmx_field_device_ptr(dtmx_ctx* ctx, int comp, void** dptr, int64_t strides[3]) {
  const int rc = dtmx_field_current_ptr(ctx, comp, dptr, strides);
  // the caller may keep the address: the automatic engine choice leaves the arrays where they are from here on
  if (!rc) {
    const Running running(ctx);
    pin_fields(ctx);
    fused_give_back(ctx);
  }
  return rc;
}

extern "C" int dtmx_check_finite(dtmx_ctx* ctx) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx) return DTMX_ERR_INVALID;
  CK(cudaMemsetAsync(ctx->d_flag, 0, sizeof(int), ctx->stream));
  for (int comp = 0; comp < 6; comp++) {
    launch(ctx, false, nonfinite_kernel, 148 * 4, 256, 0, ctx->stream, ctx->P, comp, (long long)ctx->ncell, ctx->d_flag);
    ctx->launches++;
  }
  if (int rc = launched(ctx)) return rc;
  int flag = 0;
  CK(cudaMemcpyAsync(&flag, ctx->d_flag, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CK(cudaStreamSynchronize(ctx->stream));
  return flag ? fail(ctx, DTMX_ERR_NONFINITE, "non-finite field value") : DTMX_OK;
}

extern "C" int dtmx_kernel_launches(const dtmx_ctx* ctx, int64_t* n) {
  if (!ctx || !n) return DTMX_ERR_INVALID;
  *n = ctx->launches;
  return DTMX_OK;
}

extern "C" int dtmx_set_engine(dtmx_ctx* ctx, int engine, int time_block) {
  if (!ctx || engine < 0 || engine > 3 || time_block < 0) return fail(ctx, DTMX_ERR_INVALID, "bad engine");
  const Running running(ctx);
  if (engine == 3) {
    std::string why;
    if (!fused_usable(ctx, &why)) return fail(ctx, DTMX_ERR_UNSUPPORTED, "single-sweep engine: " + why);
    ctx->tblock = 0;
  } else if (engine == 2) {
    const int T = time_block > 0 ? time_block : 2;
    std::string why;
    if (!torre_usable(ctx, T, &why)) return fail(ctx, DTMX_ERR_UNSUPPORTED, "wavefront engine: " + why);
    ctx->tblock = T;
  } else {
    ctx->tblock = time_block;
  }
  // the per-step and wavefront engines have no use for an automatic choice's second set
  if (engine == 1 || engine == 2) fused_give_back(ctx);
  ctx->engine = engine;
  ctx->auto_per_step = false;
  drop_graphs(ctx);
  return DTMX_OK;
}

extern "C" int dtmx_park(dtmx_ctx* ctx) {
  if (!ctx) return DTMX_ERR_INVALID;
  if (!ctx->cfg.parkable) return fail(ctx, DTMX_ERR_STATE, "the context was not created parkable");
  if (ctx->parked) return DTMX_OK;
  CK(cudaStreamSynchronize(ctx->stream));
  const VmmApi& A = vmm_api();
  cudaFree(ctx->dense);                          // (a parked context holds no device memory for its fields)
  ctx->dense = nullptr;
  for (auto& b : ctx->vmm) {
    // the single sweep's output buffers hold nothing between steps: every
    // node they carry is written by the next step (zero where no step writes)
    b.dead = false;
    for (int comp = 0; comp < 6; comp++) b.dead = b.dead || b.va == (CUdeviceptr)ctx->f_alt[comp];
    for (int a = 0; a < 3; a++)
      for (int q = 0; q < 2; q++) b.dead = b.dead || b.va == (CUdeviceptr)ctx->hax_alt[a][q];
    if (b.dead) continue;
    // arrays fixed once the context has stepped keep the host copy of an earlier park
    if (b.fixed && b.host && ctx->prepared && b.saved_prepared) continue;
    if (!b.host) CK(cudaMallocHost(&b.host, b.size));
    CK(cudaMemcpyAsync(b.host, (void*)b.va, b.size, cudaMemcpyDeviceToHost, ctx->stream));
    b.saved_prepared = ctx->prepared;
  }
  CK(cudaStreamSynchronize(ctx->stream));
  for (auto& b : ctx->vmm) {
    if (A.unmap(b.va, b.size) != CUDA_SUCCESS || (!pool_put(ctx->dev, b.size, b.h) && A.release(b.h) != CUDA_SUCCESS))
      return fail(ctx, DTMX_ERR_CUDA, "releasing the device memory of a parked context");
    b.h = 0;
  }
  ctx->parked = true;
  return DTMX_OK;
}

extern "C" int dtmx_set_park_pool(int device, int64_t bytes) {
  if (device < 0 || device >= kPoolDevices) return DTMX_ERR_INVALID;
  const VmmApi& A = vmm_api();
  HandlePool& P = handle_pool(device);
  std::lock_guard<std::mutex> lk(P.mu);
  P.limit = bytes < 0 ? -1 : bytes;
  // release what the new limit does not hold, largest first
  while (P.limit >= 0 && P.bytes > (size_t)P.limit && !P.free.empty()) {
    auto it = std::prev(P.free.end());
    if (A.ok) A.release(it->second);
    P.bytes -= it->first;
    P.free.erase(it);
  }
  return DTMX_OK;
}

extern "C" int dtmx_unpark(dtmx_ctx* ctx) {
  if (!ctx) return DTMX_ERR_INVALID;
  if (!ctx->parked) return DTMX_OK;
  CK(cudaSetDevice(ctx->dev));
  for (size_t q = 0; q < ctx->vmm.size(); q++) {
    VmmBlock& b = ctx->vmm[q];
    if (!vmm_back_or_free(ctx, b)) {
      // keep the context consistent: release what was mapped again and stay parked
      const VmmApi& A = vmm_api();
      for (size_t r = 0; r < q; r++) { A.unmap(ctx->vmm[r].va, ctx->vmm[r].size); A.release(ctx->vmm[r].h); }
      return fail(ctx, DTMX_ERR_OOM, "device memory for an unparked context");
    }
  }
  for (auto& b : ctx->vmm) {
    if (b.dead) CK(cudaMemsetAsync((void*)b.va, 0, b.size, ctx->stream));
    else CK(cudaMemcpyAsync((void*)b.va, b.host, b.size, cudaMemcpyHostToDevice, ctx->stream));
  }
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->parked = false;
  return DTMX_OK;
}

// ---- plane state: fields, y/z CPML auxiliaries and ADE state of x planes,
// section-major in a dense host layout (the same for every context with the
// same y/z configuration and material table, whatever its ADE box).
static int plane_poles(const dtmx_ctx* ctx) {
  int p = 0;
  for (int m = 0; m < ctx->nmat; m++) p = std::max(p, ctx->mats[m].npoles);
  return p;
}

static size_t plane_floats(const dtmx_ctx* ctx) {
  const dtmx_config& c = ctx->cfg;
  const size_t nyz = (size_t)c.ny * c.nz;
  size_t n = 6 * nyz;
  if (ctx->P.ab.aux[1][0]) n += 4 * (size_t)(ctx->P.ab.L[1][0] + ctx->P.ab.L[1][1]) * c.nz;
  if (ctx->P.ab.aux[2][0]) n += 4 * (size_t)c.ny * (ctx->P.ab.L[2][0] + ctx->P.ab.L[2][1]);
  return n + (size_t)3 * (1 + 2 * plane_poles(ctx)) * nyz;
}

static int plane_refusal(dtmx_ctx* ctx) {
  if (ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (ctx->cfg.geometry != DTMX_GEOM_BOX || ctx->cfg.absorber == DTMX_ABS_SPLIT_PML)
    return fail(ctx, DTMX_ERR_UNSUPPORTED, "plane state: box geometry with a CPML or no absorber only");
  // (a TF/SF line is not per plane either, but every slab integrates the same one)
  if (ctx->has_gyro || ctx->P.des_on)
    return fail(ctx, DTMX_ERR_UNSUPPORTED, "plane state: gyrotropic materials and design regions are not per plane");
  return DTMX_OK;
}

static int plane_copy(dtmx_ctx* ctx, int x0, int np, float* host, bool read) {
  if (!ctx) return DTMX_ERR_INVALID;
  if (int rc = plane_refusal(ctx)) return rc;
  const dtmx_config& c = ctx->cfg;
  if (!host || np < 0 || x0 < 0 || x0 + np > c.nx) return fail(ctx, DTMX_ERR_INVALID, "planes outside the grid");
  const int xl = ctx->P.ab.aux[0][0] ? ctx->P.ab.L[0][0] : 0, xh = ctx->P.ab.aux[0][0] ? ctx->P.ab.L[0][1] : 0;
  if (np > 0 && (x0 < xl || x0 + np > c.nx - xh))
    return fail(ctx, DTMX_ERR_UNSUPPORTED, "planes inside an x absorber slab");
  if (np == 0) return DTMX_OK;
  const cudaMemcpyKind kind = read ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  const size_t nyz = (size_t)c.ny * c.nz;
  float* h = host;
  for (int comp = 0; comp < 6; comp++) {
    float* d = ctx->P.f[comp] + (size_t)x0 * ctx->P.g.sx;
    if (read) CK(cudaMemcpy2DAsync(h, (size_t)c.nz * 4, d, (size_t)ctx->nzp * 4, (size_t)c.nz * 4, (size_t)np * c.ny, kind, ctx->stream));
    else CK(cudaMemcpy2DAsync(d, (size_t)ctx->nzp * 4, h, (size_t)c.nz * 4, (size_t)c.nz * 4, (size_t)np * c.ny, kind, ctx->stream));
    h += (size_t)np * nyz;
  }
  for (int a = 1; a < 3; a++) {
    if (!ctx->P.ab.aux[a][0]) continue;
    const size_t th = (size_t)(ctx->P.ab.L[a][0] + ctx->P.ab.L[a][1]);
    const size_t pp = a == 1 ? th * c.nz : (size_t)c.ny * th;     // slab_index: x-major in both
    for (int q = 0; q < 4; q++) {
      float* d = ctx->P.ab.aux[a][q] + (size_t)x0 * pp;
      CK(cudaMemcpyAsync(read ? (void*)h : (void*)d, read ? (const void*)d : (const void*)h, (size_t)np * pp * 4, kind, ctx->stream));
      h += (size_t)np * pp;
    }
  }
  const Ade& A = ctx->P.ade;
  const int P = plane_poles(ctx);
  const int b0 = std::max(x0, A.lo[0]), b1 = std::min(x0 + np, A.lo[0] + A.n[0]);
  for (int comp = 0; comp < 3; comp++)
    for (int s = 0; s < 1 + 2 * P; s++) {
      float* arr = s == 0 ? A.Em[comp] : s <= P ? A.Jp[comp][s - 1] : A.Jm[comp][s - 1 - P];
      if (read) memset(h, 0, (size_t)np * nyz * 4);      // zero off the dispersive box
      if (arr && b0 < b1) {
        cudaMemcpy3DParms m = {};
        const cudaPitchedPtr dev = make_cudaPitchedPtr(arr, (size_t)A.n[2] * 4, A.n[2], A.n[1]);
        const cudaPitchedPtr hst = make_cudaPitchedPtr(h, (size_t)c.nz * 4, c.nz, c.ny);
        const cudaPos pd = make_cudaPos(0, 0, b0 - A.lo[0]), ph = make_cudaPos((size_t)A.lo[2] * 4, A.lo[1], b0 - x0);
        if (read) { m.srcPtr = dev; m.srcPos = pd; m.dstPtr = hst; m.dstPos = ph; }
        else { m.srcPtr = hst; m.srcPos = ph; m.dstPtr = dev; m.dstPos = pd; }
        m.extent = make_cudaExtent((size_t)A.n[2] * 4, A.n[1], b1 - b0);
        m.kind = kind;
        CK(cudaMemcpy3DAsync(&m, ctx->stream));
      }
      h += (size_t)np * nyz;
    }
  CK(cudaStreamSynchronize(ctx->stream));
  return DTMX_OK;
}

// Where array arr of ctx lives now: its device address, or while the context is
// parked, the same offset in its block's pinned host copy (nullptr if that block
// has no copy).  `bytes` from arr must lie inside the block.
static char* array_home(dtmx_ctx* ctx, const void* arr, size_t bytes) {
  if (!ctx->parked) return (char*)arr;
  const CUdeviceptr a = (CUdeviceptr)arr;
  for (const VmmBlock& b : ctx->vmm)
    if (a >= b.va && a + bytes <= b.va + b.size) return (b.host && !b.dead) ? (char*)b.host + (a - b.va) : nullptr;
  return nullptr;
}

// Plane state of planes [src_x0, src_x0 + n) of src into planes [dst_x0, ...)
// of dst, either of them parked (then its pinned host copy is read or written).
extern "C" int dtmx_copy_planes(dtmx_ctx* dst, int dst_x0, dtmx_ctx* src, int src_x0, int nplanes) {
  if (!dst || !src || dst == src) return fail(dst, DTMX_ERR_INVALID, "copy_planes needs two contexts");
  for (dtmx_ctx* x : {dst, src}) {
    if (x->cfg.geometry != DTMX_GEOM_BOX || x->cfg.absorber == DTMX_ABS_SPLIT_PML)
      return fail(dst, DTMX_ERR_UNSUPPORTED, "plane state: box geometry with a CPML or no absorber only");
    if (x->has_gyro || x->P.des_on)
      return fail(dst, DTMX_ERR_UNSUPPORTED, "plane state: gyrotropic materials and design regions are not per plane");
  }
  const dtmx_config &cd = dst->cfg, &cs = src->cfg;
  if (cd.ny != cs.ny || cd.nz != cs.nz || dst->nzp != src->nzp || plane_poles(dst) != plane_poles(src) ||
      plane_floats(dst) != plane_floats(src))
    return fail(dst, DTMX_ERR_INVALID, "copy_planes: contexts of different y/z configurations or material tables");
  for (int a = 1; a < 3; a++)
    if ((dst->P.ab.aux[a][0] != nullptr) != (src->P.ab.aux[a][0] != nullptr) || dst->P.ab.L[a][0] != src->P.ab.L[a][0] ||
        dst->P.ab.L[a][1] != src->P.ab.L[a][1])
      return fail(dst, DTMX_ERR_INVALID, "copy_planes: different y/z absorber slabs");
  const int np = nplanes;
  if (np < 0 || dst_x0 < 0 || src_x0 < 0 || dst_x0 + np > cd.nx || src_x0 + np > cs.nx)
    return fail(dst, DTMX_ERR_INVALID, "planes outside the grid");
  for (dtmx_ctx* x : {dst, src}) {
    const int x0 = x == dst ? dst_x0 : src_x0;
    const int xl = x->P.ab.aux[0][0] ? x->P.ab.L[0][0] : 0, xh = x->P.ab.aux[0][0] ? x->P.ab.L[0][1] : 0;
    if (np > 0 && (x0 < xl || x0 + np > x->cfg.nx - xh)) return fail(dst, DTMX_ERR_UNSUPPORTED, "planes inside an x absorber slab");
  }
  if (np == 0) return DTMX_OK;
  dtmx_ctx* ctx = dst;                          // errors of the copies are reported on dst
  CK(cudaStreamSynchronize(src->stream));
  cudaStream_t st = dst->stream;
  auto span = [&](dtmx_ctx* x, const float* arr, size_t off, size_t cnt) -> char* {
    // cnt floats from arr + off, inside the array's block
    return array_home(x, arr + off, cnt * 4);
  };
  // fields and y/z auxiliaries: the same per-plane layout in both contexts
  const size_t sx = (size_t)src->P.g.sx;
  for (int comp = 0; comp < 6; comp++) {
    char* d = span(dst, dst->P.f[comp], (size_t)dst_x0 * sx, (size_t)np * sx);
    char* h = span(src, src->P.f[comp], (size_t)src_x0 * sx, (size_t)np * sx);
    if (!d || !h) return fail(dst, DTMX_ERR_STATE, "copy_planes: a parked array has no host copy");
    CK(cudaMemcpyAsync(d, h, (size_t)np * sx * 4, cudaMemcpyDefault, st));
  }
  for (int a = 1; a < 3; a++) {
    if (!src->P.ab.aux[a][0]) continue;
    const size_t th = (size_t)(src->P.ab.L[a][0] + src->P.ab.L[a][1]);
    const size_t pp = a == 1 ? th * cs.nz : (size_t)cs.ny * th;
    for (int q = 0; q < 4; q++) {
      char* d = span(dst, dst->P.ab.aux[a][q], (size_t)dst_x0 * pp, (size_t)np * pp);
      char* h = span(src, src->P.ab.aux[a][q], (size_t)src_x0 * pp, (size_t)np * pp);
      if (!d || !h) return fail(dst, DTMX_ERR_STATE, "copy_planes: a parked array has no host copy");
      CK(cudaMemcpyAsync(d, h, (size_t)np * pp * 4, cudaMemcpyDefault, st));
    }
  }
  // ADE state over the intersection of the two boxes (a dispersive node of
  // the copied planes lies in both; the rest of either box holds zeros there)
  const Ade &As = src->P.ade, &Ad = dst->P.ade;
  const int P = plane_poles(src);
  const int p0 = std::max(std::max(0, As.lo[0] - src_x0), Ad.lo[0] - dst_x0);
  const int p1 = std::min(std::min(np, As.lo[0] + As.n[0] - src_x0), Ad.lo[0] + Ad.n[0] - dst_x0);
  const int y0 = std::max(As.lo[1], Ad.lo[1]), y1 = std::min(As.lo[1] + As.n[1], Ad.lo[1] + Ad.n[1]);
  const int z0 = std::max(As.lo[2], Ad.lo[2]), z1 = std::min(As.lo[2] + As.n[2], Ad.lo[2] + Ad.n[2]);
  for (int comp = 0; comp < 3; comp++)
    for (int q = 0; q < 1 + 2 * P; q++) {
      float* as = q == 0 ? As.Em[comp] : q <= P ? As.Jp[comp][q - 1] : As.Jm[comp][q - 1 - P];
      float* ad = q == 0 ? Ad.Em[comp] : q <= P ? Ad.Jp[comp][q - 1] : Ad.Jm[comp][q - 1 - P];
      if (!as || p0 >= p1 || y0 >= y1 || z0 >= z1) continue;       // nothing dispersive in the copied planes
      if (!ad) return fail(dst, DTMX_ERR_INVALID, "copy_planes: dispersive nodes the destination does not hold");
      const size_t ns = (size_t)As.n[0] * As.n[1] * As.n[2], nd = (size_t)Ad.n[0] * Ad.n[1] * Ad.n[2];
      char* hs = array_home(src, as, ns * 4);
      char* hd = array_home(dst, ad, nd * 4);
      if (!hs || !hd) return fail(dst, DTMX_ERR_STATE, "copy_planes: a parked array has no host copy");
      cudaMemcpy3DParms m = {};
      m.srcPtr = make_cudaPitchedPtr(hs, (size_t)As.n[2] * 4, As.n[2], As.n[1]);
      m.srcPos = make_cudaPos((size_t)(z0 - As.lo[2]) * 4, y0 - As.lo[1], src_x0 + p0 - As.lo[0]);
      m.dstPtr = make_cudaPitchedPtr(hd, (size_t)Ad.n[2] * 4, Ad.n[2], Ad.n[1]);
      m.dstPos = make_cudaPos((size_t)(z0 - Ad.lo[2]) * 4, y0 - Ad.lo[1], dst_x0 + p0 - Ad.lo[0]);
      m.extent = make_cudaExtent((size_t)(z1 - z0) * 4, y1 - y0, p1 - p0);
      m.kind = cudaMemcpyDefault;
      CK(cudaMemcpy3DAsync(&m, st));
    }
  CK(cudaStreamSynchronize(st));
  return DTMX_OK;
}

extern "C" int dtmx_plane_state_floats(dtmx_ctx* ctx, size_t* floats_per_plane) {
  if (!ctx || !floats_per_plane) return fail(ctx, DTMX_ERR_INVALID, "bad plane state request");
  if (int rc = plane_refusal(ctx)) return rc;
  *floats_per_plane = plane_floats(ctx);
  return DTMX_OK;
}

extern "C" int dtmx_read_planes(dtmx_ctx* ctx, int x0, int nplanes, float* host) {
  return plane_copy(ctx, x0, nplanes, host, true);
}

extern "C" int dtmx_write_planes(dtmx_ctx* ctx, int x0, int nplanes, const float* host) {
  return plane_copy(ctx, x0, nplanes, const_cast<float*>(host), false);
}

extern "C" int dtmx_set_tile_rows(dtmx_ctx* ctx, int rows) {
  if (!ctx || (rows != 0 && rows != 8 && rows != 16)) return fail(ctx, DTMX_ERR_INVALID, "tile rows must be 8 or 16");
  const Running running(ctx);
  ctx->frows = rows ? rows : 16;
  drop_graphs(ctx);
  return DTMX_OK;
}

extern "C" int dtmx_get_engine(dtmx_ctx* ctx, int* engine, int* time_block, int* xchunk, int* tile_rows) {
  if (!ctx) return DTMX_ERR_INVALID;
  if (engine) *engine = ctx->engine;
  if (time_block) *time_block = ctx->tblock;
  if (xchunk) *xchunk = ctx->xchunk;
  if (tile_rows) *tile_rows = ctx->frows;
  return DTMX_OK;
}

extern "C" int dtmx_set_xchunk(dtmx_ctx* ctx, int planes) {
  if (!ctx || planes < 0) return fail(ctx, DTMX_ERR_INVALID, "bad x chunk");
  const Running running(ctx);
  ctx->xchunk = planes;
  drop_graphs(ctx);
  return DTMX_OK;
}

extern "C" int dtmx_work_pieces(dtmx_ctx* ctx, int kernel, int* equal_cost, int* pieces, int* longest) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx || kernel < 0 || kernel > 2) return fail(ctx, DTMX_ERR_INVALID, "bad kernel");
  const Running running(ctx);
  const WorkPlan* w;
  const int rc = kernel == 0 ? plan_stream(ctx, &w) : kernel == 1 ? plan_sweep(ctx, &w) : plan_work(ctx, WK_ADJ, 16, 3, 0, &w);
  if (rc) return rc;
  if (equal_cost) *equal_cost = w->table ? 1 : 0;
  if (pieces) *pieces = (int)(w->grid.x * w->grid.y * w->grid.z);
  if (longest) *longest = w->longest;
  return DTMX_OK;
}

extern "C" int dtmx_set_wait_limit(dtmx_ctx* ctx, int64_t polls) {
  if (!ctx) return DTMX_ERR_INVALID;
  ctx->P.wait_limit = polls > 0 ? (long long)polls : kWaitPolls;
  return DTMX_OK;
}

extern "C" int dtmx_fail_next(dtmx_ctx* ctx, int what, int skip) {
  if (!ctx || (what != DTMX_FAIL_ALLOC && what != DTMX_FAIL_LAUNCH)) return fail(ctx, DTMX_ERR_INVALID, "bad failure request");
  ctx->fail_in[what] = skip < 0 ? -1 : skip;
  return DTMX_OK;
}

extern "C" int dtmx_get_stream(dtmx_ctx* ctx, void** stream) {
  if (!ctx || !stream) return DTMX_ERR_INVALID;
  *stream = (void*)ctx->stream;
  return DTMX_OK;
}

extern "C" int dtmx_set_profiling(dtmx_ctx* ctx, int enable) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx) return DTMX_ERR_INVALID;
  if (enable && !ctx->ev[0])
    for (int q = 0; q < 4; q++) CK(cudaEventCreate(&ctx->ev[q]));
  CK(cudaStreamSynchronize(ctx->stream));
  ctx->profiling = enable != 0;
  ctx->prof_ms_h = ctx->prof_ms_e = 0;
  ctx->prof_count = 0;
  ctx->prof_pending = false;
  return DTMX_OK;
}

extern "C" int dtmx_read_profile(dtmx_ctx* ctx, double* ms_h, double* ms_e, int64_t* count) {
  if (ctx && ctx->parked) return fail(ctx, DTMX_ERR_STATE, "the context is parked (dtmx_unpark first)");
  if (!ctx) return DTMX_ERR_INVALID;
  CK(cudaStreamSynchronize(ctx->stream));
  if (ms_h) *ms_h = ctx->prof_ms_h;
  if (ms_e) *ms_e = ctx->prof_ms_e;
  if (count) *count = ctx->prof_count;
  return DTMX_OK;
}

extern "C" int dtmx_abi_sizes(int64_t out[6]) {
  if (!out) return DTMX_ERR_INVALID;
  out[0] = sizeof(dtmx_config); out[1] = sizeof(dtmx_material);
  out[2] = sizeof(dtmx_point_source); out[3] = sizeof(dtmx_tfsf);
  out[4] = sizeof(dtmx_tfsfsrc); out[5] = sizeof(dtmx_ref_globals);
  return DTMX_OK;
}
