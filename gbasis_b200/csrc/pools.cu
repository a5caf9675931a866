// The process's pools: idle device blocks (block cache) and idle stream sets.
#include "pools.h"

#include <mutex>

#include "errors.h"

namespace gbx {

#define GBX_CUDA(call, what)                        \
  do {                                              \
    int _s = cuda_status((call), (what));           \
    if (_s != GBX_OK) return _s;                    \
  } while (0)

// ------------------------------------------------------------------- block cache
// Device blocks a basis gives back are kept for the next basis in the process, up to
// kBlockCacheBytes per device: the public full-tensor call builds and drops a basis every time,
// and cudaFree (which waits for the whole device) plus cudaMalloc of the compact store and the
// staging slabs cost milliseconds per call.  A block is reused for a request of at least half
// its size.  gbx_release_cached_memory() frees the cache, and so does an allocation that finds the
// device full: what would fit without the cache fits with it.
constexpr size_t kBlockCacheBytes = size_t(2) << 30;
struct CachedBlock {
  int device;
  void* p;
  size_t bytes;
};
static std::mutex g_block_mu;
static std::vector<CachedBlock> g_blocks;

static void* cache_take(int device, size_t bytes, size_t* got) {
  std::lock_guard<std::mutex> lk(g_block_mu);
  int best = -1;
  for (int i = 0; i < (int)g_blocks.size(); ++i) {
    const CachedBlock& b = g_blocks[i];
    if (b.device != device || b.bytes < bytes || b.bytes / 2 > bytes) continue;
    if (best < 0 || b.bytes < g_blocks[best].bytes) best = i;
  }
  if (best < 0) return nullptr;
  void* p = g_blocks[best].p;
  *got = g_blocks[best].bytes;
  g_blocks.erase(g_blocks.begin() + best);
  return p;
}

void block_give(int device, void* p, size_t bytes) {
  if (!p) return;
  {
    std::lock_guard<std::mutex> lk(g_block_mu);
    size_t held = 0;
    for (const CachedBlock& b : g_blocks)
      if (b.device == device) held += b.bytes;
    if (held + bytes <= kBlockCacheBytes) {
      g_blocks.push_back({device, p, bytes});
      return;
    }
  }
  cudaFree(p);
}

// Frees the idle blocks of a device (of all: device < 0); whether there were any.
static bool cache_drop(int device) {
  std::vector<CachedBlock> drop;
  {
    std::lock_guard<std::mutex> lk(g_block_mu);
    for (size_t i = g_blocks.size(); i-- > 0;)
      if (device < 0 || g_blocks[i].device == device) {
        drop.push_back(g_blocks[i]);
        g_blocks.erase(g_blocks.begin() + i);
      }
  }
  for (const CachedBlock& b : drop) {
    DeviceGuardLite g(b.device);
    cudaFree(b.p);
  }
  return !drop.empty();
}

int block_alloc(int device, void** p, size_t bytes, size_t* got, const char* what) {
  if (bytes == 0) bytes = 16;
  *p = cache_take(device, bytes, got);
  if (!*p) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation && cache_drop(device)) {
      cudaGetLastError();  // the failed attempt's error
      e = cudaMalloc(p, bytes);
    }
    GBX_CUDA(e, what);
    *got = bytes;
  }
  return GBX_OK;
}

// ------------------------------------------------------------------- stream pool
constexpr int kPooledStreamSets = 4;  // idle sets kept per device
// under g_block_mu; never destroyed (the driver may be gone when static destructors run)
static std::vector<std::unique_ptr<StreamSet>>& g_stream_sets =
    *new std::vector<std::unique_ptr<StreamSet>>;

int StreamSet::ensure_aux(int n) {
  while ((int)aux.size() < n) {
    cudaStream_t s = nullptr;
    cudaEvent_t e = nullptr;
    GBX_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "create event");
    const cudaError_t err = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    if (err != cudaSuccess) cudaEventDestroy(e);
    GBX_CUDA(err, "create stream");
    join.push_back(e);  // a stream and its event, or neither: the set may be used again after an error
    aux.push_back(s);
  }
  return GBX_OK;
}

StreamSet::~StreamSet() {
  DeviceGuardLite g(device);
  for (cudaStream_t s : aux) cudaStreamDestroy(s);
  for (cudaEvent_t e : join) cudaEventDestroy(e);
  for (cudaEvent_t e : {fork, in, out})
    if (e) cudaEventDestroy(e);
  if (copy) cudaStreamDestroy(copy);
  for (cudaEvent_t e : stage_ready)
    if (e) cudaEventDestroy(e);
  for (cudaEvent_t e : stage_free)
    if (e) cudaEventDestroy(e);
}

int streams_take(int device, std::unique_ptr<StreamSet>* out) {
  {
    std::lock_guard<std::mutex> lk(g_block_mu);
    for (size_t i = 0; i < g_stream_sets.size(); ++i)
      if (g_stream_sets[i]->device == device) {
        *out = std::move(g_stream_sets[i]);
        g_stream_sets.erase(g_stream_sets.begin() + i);
        return GBX_OK;
      }
  }
  auto set = std::make_unique<StreamSet>();
  set->device = device;
  for (cudaEvent_t* e : {&set->fork, &set->in, &set->out})
    GBX_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming), "create event");
  GBX_CUDA(cudaStreamCreateWithFlags(&set->copy, cudaStreamNonBlocking), "create stream");
  for (int k = 0; k < kStageBuffers; ++k) {
    GBX_CUDA(cudaEventCreateWithFlags(&set->stage_ready[k], cudaEventDisableTiming), "event");
    GBX_CUDA(cudaEventCreateWithFlags(&set->stage_free[k], cudaEventDisableTiming), "event");
  }
  *out = std::move(set);
  return GBX_OK;
}

void streams_give(std::unique_ptr<StreamSet> set, bool idle) {
  if (!set || !idle) return;  // a set that may still have work is destroyed, not shared
  std::lock_guard<std::mutex> lk(g_block_mu);
  int held = 0;
  for (const auto& s : g_stream_sets) held += s->device == set->device;
  if (held < kPooledStreamSets) g_stream_sets.push_back(std::move(set));
}

void release_pools() {
  std::vector<std::unique_ptr<StreamSet>> sets;  // destroyed at the end, outside the lock
  {
    std::lock_guard<std::mutex> lk(g_block_mu);
    sets.swap(g_stream_sets);
  }
  cache_drop(-1);
}

}  // namespace gbx
