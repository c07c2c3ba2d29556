// Library-wide device memory pool and stream sets (device_pool.h).
#include "device_pool.h"

#include <cuda.h>

#include <atomic>
#include <mutex>

namespace iqcp {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices] = {nullptr};
std::vector<StreamSet> g_idle[kMaxDevices];
// keeps the driver's segment for small blocks mapped: with nothing else from
// cudaMalloc in the process a 256-byte block costs 608 us, beside one 5 us
void* g_anchor[kMaxDevices] = {nullptr};
unsigned long long g_id[kMaxDevices] = {0};  // CUDA context that the above belong to
std::atomic<unsigned> g_epoch[kMaxDevices];

using CtxGetId = CUresult (*)(CUcontext, unsigned long long*);
CtxGetId ctx_get_id() {
  static const CtxGetId fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<CtxGetId>(p);
  }();
  return fn;
}

cudaError_t pool_of(int device, cudaMemPool_t* out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_pool[device]) {
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof(props));
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    unsigned long long keep = kPoolKeep;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    g_pool[device] = pool;
  }
  *out = g_pool[device];
  return cudaSuccess;
}

size_t round_up(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

cudaError_t device_refresh(int device, unsigned long long* id) {
  *id = 0;
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  cudaError_t e = cudaFree(nullptr);  // the primary context, made anew after a reset
  if (e != cudaSuccess) return e;
  const CtxGetId get = ctx_get_id();
  if (!get) return cudaErrorNotSupported;
  if (get(nullptr, id) != CUDA_SUCCESS) return cudaErrorDeviceUninitialized;
  std::lock_guard<std::mutex> lock(g_mu);
  if (g_id[device] != *id) {
    if (g_id[device]) g_epoch[device].fetch_add(1);
    g_id[device] = *id;
    g_pool[device] = nullptr;
    g_idle[device].clear();
    g_anchor[device] = nullptr;
  }
  return cudaSuccess;
}

unsigned device_epoch(int device) { return device >= 0 && device < kMaxDevices ? g_epoch[device].load() : 0; }

cudaError_t pool_alloc(int device, void** p, size_t bytes, cudaStream_t stream) {
  cudaMemPool_t pool = nullptr;
  const cudaError_t e = pool_of(device, &pool);
  if (e != cudaSuccess) return e;
  return cudaMallocFromPoolAsync(p, bytes > 0 ? bytes : 256, pool, stream);
}

void pool_free(void* p, cudaStream_t stream) {
  if (p) cudaFreeAsync(p, stream);
}

cudaError_t drain_block(int device, void** p) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  RelaxedCapture relaxed;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_anchor[device]) {
      const cudaError_t e = cudaMalloc(&g_anchor[device], 256);
      if (e != cudaSuccess) {
        g_anchor[device] = nullptr;
        return e;
      }
    }
  }
  return cudaMalloc(p, 256);
}

cudaError_t drain(void* block) {
  RelaxedCapture relaxed;
  return block ? cudaFree(block) : cudaErrorInvalidValue;
}

cudaError_t streams_take(int device, StreamSet* set) {
  *set = StreamSet();
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_idle[device].empty()) {
      *set = g_idle[device].back();
      g_idle[device].pop_back();
      return cudaSuccess;
    }
  }
  for (int i = 0; i < kSetStreams; ++i) {
    const cudaError_t e = cudaStreamCreateWithFlags(&set->s[i], cudaStreamNonBlocking);
    if (e != cudaSuccess) {
      for (int j = 0; j < i; ++j) cudaStreamDestroy(set->s[j]);
      *set = StreamSet();
      return e;
    }
  }
  return cudaSuccess;
}

void streams_give(int device, const StreamSet& set) {
  if (!set.s[0]) return;
  if (device >= 0 && device < kMaxDevices) {
    std::lock_guard<std::mutex> lock(g_mu);
    if (g_idle[device].size() < (size_t)kKeepStreams) {
      g_idle[device].push_back(set);
      return;
    }
  }
  for (int i = 0; i < kSetStreams; ++i) cudaStreamDestroy(set.s[i]);
}

cudaError_t DeviceBlock::alloc(int device, cudaStream_t stream) {
  size_t in = 0, total = 0;
  for (const Item& it : items_)
    if (it.src) in += round_up(it.bytes);
  total = in;
  for (const Item& it : items_)
    if (!it.src) total += round_up(it.bytes);
  pooled_ = total <= kPoolMax;
  cudaError_t e = pooled_ ? pool_alloc(device, &base_, total, stream) : cudaMalloc(&base_, total);
  if (e != cudaSuccess) {
    base_ = nullptr;
    return e;
  }
  char* base = static_cast<char*>(base_);
  std::vector<char> host(in);
  size_t a = 0, b = in;
  for (const Item& it : items_) {
    size_t& o = it.src ? a : b;
    *it.p = base + o;
    if (it.src && it.bytes) std::memcpy(host.data() + o, it.src, it.bytes);
    o += round_up(it.bytes);
  }
  items_.clear();
  // pageable source: the copy has left it when the call returns
  return in ? cudaMemcpyAsync(base, host.data(), in, cudaMemcpyHostToDevice, stream) : cudaSuccess;
}

void DeviceBlock::free(cudaStream_t stream) {
  if (pooled_) pool_free(base_, stream);
  else cudaFree(base_);
  base_ = nullptr;
}

}  // namespace iqcp
