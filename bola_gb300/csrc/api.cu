// api.cu — library-wide state: error messages, SIMD-width setting, device info.
#include <cuda.h>

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <set>
#include <utility>

#include "common.cuh"

namespace bola {

namespace {
thread_local char g_msg[512] = "";
int g_lanes = 2;
}  // namespace

int fail(int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_msg, sizeof g_msg, fmt, ap);
  va_end(ap);
  return code;
}

int cuda_fail(cudaError_t e, const char *what) {
  return fail(BOLA_ERR_CUDA, "%s failed: %s", what, cudaGetErrorString(e));
}

int lanes() { return g_lanes; }

int num_sms() {
  static thread_local int dev = -1, sms = 0;
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) return 1;
  if (d != dev) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || v <= 0) v = 1;
    dev = d;
    sms = v;
  }
  return sms;
}

namespace {

// The calling thread's current context and its unique id (0 if none or unknown).
// The driver functions are reached through the runtime's entry-point query,
// so the library does not link the driver library directly.
unsigned long long current_context(CUcontext *out) {
  using GetCurrentFn = CUresult (*)(CUcontext *);
  using GetIdFn = CUresult (*)(CUcontext, unsigned long long *);
  static GetCurrentFn get_current = nullptr;
  static GetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrentFn>(p);
    p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetIdFn>(p);
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current == nullptr || get_id == nullptr || get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr ||
      get_id(ctx, &id) != CUDA_SUCCESS)
    return 0;
  *out = ctx;
  return id;
}

// Whether ctx, which is current, is its device's primary context.
bool is_primary(CUcontext ctx, int dev) {
  using RetainFn = CUresult (*)(CUcontext *, CUdevice);
  using ReleaseFn = CUresult (*)(CUdevice);
  using StateFn = CUresult (*)(CUdevice, unsigned *, int *);
  void *state = nullptr, *retain = nullptr, *release = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuDevicePrimaryCtxGetState", &state, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      cudaGetDriverEntryPointByVersion("cuDevicePrimaryCtxRetain", &retain, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      cudaGetDriverEntryPointByVersion("cuDevicePrimaryCtxRelease", &release, 12000, cudaEnableDefault, &q) != cudaSuccess)
    return true;  // (then nothing of its is given back)
  unsigned flags = 0;
  int active = 0;
  CUcontext primary = nullptr;
  if (reinterpret_cast<StateFn>(state)(dev, &flags, &active) != CUDA_SUCCESS) return true;
  if (!active) return false;
  if (reinterpret_cast<RetainFn>(retain)(&primary, dev) != CUDA_SUCCESS) return true;
  reinterpret_cast<ReleaseFn>(release)(dev);
  return primary == ctx;
}

constexpr int kMaxDevices = 64;
constexpr int kMaxPools = 8;  // per device: contexts that are served from a pool of their own
constexpr uint64_t kScratchKept = uint64_t(64) << 20;
std::mutex g_pool_mu;
struct PoolSlot {
  CUcontext ctx = nullptr;    // the context that the pool serves
  unsigned long long id = 0;  // and which one at that address
  bool primary = false;       // the device's primary context: a reset of the device ends the pool with it
  cudaMemPool_t pool = nullptr;
};
PoolSlot g_pool_slot[kMaxDevices][kMaxPools];

// Memory that graphs use: a block goes to one captured graph at a time and back
// to this list when CUDA says that the graph is gone (on a thread of its own,
// where no CUDA call may be made).  Blocks beyond MAX_FREE are given back to the
// device at the next capture that finds them.
struct GraphBlock {
  void *ptr = nullptr;
  size_t bytes = 0;
  unsigned long long ctx_id = 0;
  GraphBlock *next = nullptr;
};
constexpr int kMaxFreeBlocks = 16;
std::mutex g_graph_mu;
GraphBlock *g_graph_free = nullptr;
void CUDART_CB graph_gone(void *block) {
  std::lock_guard<std::mutex> lk(g_graph_mu);
  static_cast<GraphBlock *>(block)->next = g_graph_free;
  g_graph_free = static_cast<GraphBlock *>(block);
}
// Calls that allocate are allowed on this thread while one of its streams is captured.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace

unsigned long long context_id() {
  CUcontext ctx = nullptr;
  return current_context(&ctx);
}

int graph_memory(cudaStream_t s, size_t bytes, void **out) {
  *out = nullptr;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  BOLA_TRY_CUDA(cudaStreamGetCaptureInfo(s, &status, nullptr, &graph));
  if (status != cudaStreamCaptureStatusActive) return fail(BOLA_ERR_CUDA, "graph_memory: the stream is not being captured");
  size_t size = (size_t)64 << 10;
  while (size < bytes) size *= 2;
  CUcontext ctx = nullptr;
  const unsigned long long id = current_context(&ctx);
  RelaxedCapture relaxed;
  GraphBlock *block = nullptr, *extra = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_graph_mu);
    int kept = 0;
    for (GraphBlock **at = &g_graph_free; *at != nullptr;) {
      GraphBlock *b = *at;
      const bool take = block == nullptr && b->ctx_id == id && b->bytes == size;
      if (!take && (b->ctx_id != id || ++kept <= kMaxFreeBlocks)) {
        at = &b->next;
        continue;
      }
      *at = b->next;
      if (take) {
        block = b;
      } else {
        b->next = extra;
        extra = b;
      }
    }
  }
  while (extra != nullptr) {
    GraphBlock *b = extra;
    extra = b->next;
    cudaFree(b->ptr);
    delete b;
  }
  if (block == nullptr) {
    block = new (std::nothrow) GraphBlock();
    if (block == nullptr) return fail(BOLA_ERR_CUDA, "graph_memory: out of host memory");
    const cudaError_t e = cudaMalloc(&block->ptr, size);
    if (e != cudaSuccess) {
      delete block;
      return cuda_fail(e, "cudaMalloc(graph memory)");
    }
    block->bytes = size;
    block->ctx_id = id;
  }
  cudaUserObject_t owner = nullptr;
  cudaError_t e = cudaUserObjectCreate(&owner, block, graph_gone, 1, cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    graph_gone(block);
    return cuda_fail(e, "cudaUserObjectCreate");
  }
  e = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(owner, 1);
    return cuda_fail(e, "cudaGraphRetainUserObject");
  }
  *out = block->ptr;
  return 0;
}

int roomy(const void *kern) {
  int dev = 0;
  BOLA_TRY_CUDA(cudaGetDevice(&dev));
  static std::mutex mu;
  static std::set<std::pair<int, const void *>> done;
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, kern})) return 0;
  BOLA_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  try {
    done.insert({dev, kern});
  } catch (...) {  // (out of host memory: asked for again next time, and no exception leaves a C entry)
  }
  return 0;
}

cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  CUcontext ctx = nullptr;
  const unsigned long long id = current_context(&ctx);
  if (id == 0) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  // this context's slot, or a free one, or that of a context that was at this
  // address before (whose pool outlives it, and goes back here)
  PoolSlot *slot = nullptr;
  for (PoolSlot &s : g_pool_slot[dev]) {
    if (s.pool != nullptr && s.ctx != ctx) continue;
    if (s.pool != nullptr && s.id == id) return s.pool;
    slot = &s;
    break;
  }
  if (slot == nullptr) return nullptr;  // (the default pool serves further contexts)
  if (slot->pool != nullptr && !slot->primary) cudaMemPoolDestroy(slot->pool);
  slot->pool = nullptr;
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  uint64_t keep = kScratchKept;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    if (pool != nullptr) cudaMemPoolDestroy(pool);
    cudaGetLastError();
    return nullptr;
  }
  slot->ctx = ctx;
  slot->id = id;
  slot->primary = is_primary(ctx, dev);
  slot->pool = pool;
  return pool;
}

}  // namespace bola

extern "C" {

const char *bola_version(void) { return "bola_gb300 0.1.0 (sm_103a, BOLA 0.1.2 semantics)"; }

const char *bola_last_error(void) { return bola::g_msg; }

int bola_set_simd_lanes(int lanes) {
  if (lanes != 2 && lanes != 4) return -1;
  const int old = bola::g_lanes;
  bola::g_lanes = lanes;
  return old;
}

int bola_get_simd_lanes(void) { return bola::g_lanes; }

}  // extern "C"
