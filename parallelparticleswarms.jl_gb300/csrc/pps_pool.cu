// pps_pool.cu -- see pps_pool.h.
#include "pps_pool.h"

#include <mutex>
#include <vector>

namespace pps {

namespace {

constexpr int kDevices = 64;

struct DevicePools {
  std::mutex mu;
  std::vector<PoolStream> idle;
  cudaMemPool_t mem = nullptr;
};

// never destroyed: a swarm may be closed while the process ends
DevicePools& pools(int device) {
  static DevicePools* p = new DevicePools[kDevices];
  return p[device];
}

bool known(int device) { return device >= 0 && device < kDevices; }

void destroy(PoolStream* s) {
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  if (s->stream) cudaStreamDestroy(s->stream);
  *s = PoolStream{};
}

}  // namespace

cudaError_t pool_stream_get(int device, PoolStream* s) {
  *s = PoolStream{};
  if (known(device)) {
    DevicePools& d = pools(device);
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.idle.empty()) {
      *s = d.idle.back();
      d.idle.pop_back();
      if (cudaStreamQuery(s->stream) == cudaSuccess) return cudaSuccess;
      cudaGetLastError();  // the device was reset meanwhile: its handles are gone
      d.idle.clear();
      *s = PoolStream{};
    }
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
  if (idle && known(device)) {
    DevicePools& d = pools(device);
    std::lock_guard<std::mutex> lock(d.mu);
    if ((int)d.idle.size() < kPoolStreams) {
      d.idle.push_back(*s);
      *s = PoolStream{};
      return;
    }
  }
  destroy(s);
}

cudaError_t pool_alloc(int device, void** p, size_t bytes, cudaStream_t stream) {
  if (!known(device)) return cudaMallocAsync(p, bytes, stream);
  DevicePools& d = pools(device);
  cudaMemPool_t mem;
  {
    std::lock_guard<std::mutex> lock(d.mu);
    if (!d.mem) {
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
      d.mem = fresh;
    }
    mem = d.mem;
  }
  const cudaError_t e = cudaMallocFromPoolAsync(p, bytes, mem, stream);
  if (e == cudaSuccess || e == cudaErrorMemoryAllocation) return e;
  cudaGetLastError();  // the pool is gone with a reset device
  {
    std::lock_guard<std::mutex> lock(d.mu);
    if (d.mem == mem) d.mem = nullptr;
  }
  return cudaMallocAsync(p, bytes, stream);
}

}  // namespace pps
