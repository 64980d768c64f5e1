// pps_pool.cu -- see pps_pool.h.
#include "pps_pool.h"

#include <cuda.h>

#include <mutex>
#include <vector>

namespace pps {

namespace {

constexpr int kDevices = 64;

struct DevicePools {
  std::mutex mu;
  unsigned long long context = 0;  // what `idle` and `mem` belong to
  std::vector<PoolStream> idle;
  cudaMemPool_t mem = nullptr;
};

// never destroyed: a swarm may be closed while the process ends
DevicePools& pools(int device) {
  static DevicePools* p = new DevicePools[kDevices];
  return p[device];
}

bool known(int device) { return device >= 0 && device < kDevices; }

// The number of the current device's context: another one after a device reset,
// so handles of the context before it are told apart without touching them (a
// query of such a stream ends the process).  0: unknown.
unsigned long long context_number(int device) {
  using GetId = CUresult (*)(CUcontext, unsigned long long*);
  static const GetId get = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult r{};
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &r);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && r == cudaDriverEntryPointSuccess ? reinterpret_cast<GetId>(f) : nullptr;
  }();
  unsigned long long id = 0;
  if (!get) return 0;
  if (get(nullptr, &id) == CUDA_SUCCESS) return id;
  if (cudaSetDevice(device) != cudaSuccess) {  // makes the context that a reset took away
    cudaGetLastError();
    return 0;
  }
  return get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// The device's pools if they can serve its current context, locked by `lock`;
// what is left of a context before it is dropped, its handles being gone.
DevicePools* pools_of_context(int device, std::unique_lock<std::mutex>* lock) {
  const unsigned long long id = known(device) ? context_number(device) : 0;
  if (!id) return nullptr;
  DevicePools& d = pools(device);
  *lock = std::unique_lock<std::mutex>(d.mu);
  if (d.context != id) {
    d.idle.clear();
    d.mem = nullptr;
    d.context = id;
  }
  return &d;
}

void destroy(PoolStream* s) {
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  if (s->stream) cudaStreamDestroy(s->stream);
  *s = PoolStream{};
}

}  // namespace

cudaError_t pool_stream_get(int device, PoolStream* s) {
  *s = PoolStream{};
  {
    std::unique_lock<std::mutex> lock;
    DevicePools* d = pools_of_context(device, &lock);
    if (d && !d->idle.empty()) {
      *s = d->idle.back();
      d->idle.pop_back();
      return cudaSuccess;
    }
    if (d) s->context = d->context;
  }
  cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&s->ev1);
  if (e != cudaSuccess) destroy(s);
  return e;
}

void pool_stream_put(int device, PoolStream* s) {
  if (!s->stream) return destroy(s);
  const bool idle = cudaStreamSynchronize(s->stream) == cudaSuccess;
  if (idle) {
    std::unique_lock<std::mutex> lock;
    DevicePools* d = pools_of_context(device, &lock);
    if (d && s->context == d->context && (int)d->idle.size() < kPoolStreams) {
      d->idle.push_back(*s);
      *s = PoolStream{};
      return;
    }
  }
  destroy(s);
}

cudaError_t pool_alloc(int device, void** p, size_t bytes, cudaStream_t stream) {
  cudaMemPool_t mem = nullptr;
  {
    std::unique_lock<std::mutex> lock;
    DevicePools* d = pools_of_context(device, &lock);
    if (!d) return cudaMallocAsync(p, bytes, stream);
    if (!d->mem) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      unsigned long long keep = kPoolBytes;
      cudaMemPool_t fresh = nullptr;
      if (cudaMemPoolCreate(&fresh, &props) != cudaSuccess ||
          cudaMemPoolSetAttribute(fresh, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        if (fresh) cudaMemPoolDestroy(fresh);
        return cudaMallocAsync(p, bytes, stream);
      }
      d->mem = fresh;
    }
    mem = d->mem;
  }
  return cudaMallocFromPoolAsync(p, bytes, mem, stream);
}

}  // namespace pps
