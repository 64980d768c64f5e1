// pps_pool.h -- driver objects that outlive one swarm, evaluation or snapshot:
// streams with a pair of timing events, and a memory pool for small blocks.
//
// Creating and destroying a stream, two events and a few kilobytes of device
// memory took most of a small solve (a swarm's create and close 209 us, an
// evaluation of one point 224 us, a position snapshot 149 us, against 1 ms of
// iterations for 1000 x 3-D, 500 iterations).  Both pools are per device, used
// from any thread, and bounded: at most kPoolStreams idle streams are kept
// (idle ones only: a stream is given back after it has been synchronised) and
// at most kPoolBytes of freed device memory; what is beyond is returned to the
// driver at once.
#pragma once
#include <cuda_runtime.h>

namespace pps {

constexpr int kPoolStreams = 16;
constexpr size_t kPoolBytes = (size_t)64 << 20;

struct PoolStream {
  cudaStream_t stream = nullptr;  // non-blocking
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  unsigned long long context = 0;  // the context it belongs to (0: it is not kept)
};

// a stream of the current device, idle
cudaError_t pool_stream_get(int device, PoolStream* s);
// gives a stream back after synchronising it (nullptr members are allowed)
void pool_stream_put(int device, PoolStream* s);
// `bytes` of the current device's memory in `stream`'s order; freed with cudaFreeAsync
cudaError_t pool_alloc(int device, void** p, size_t bytes, cudaStream_t stream);

}  // namespace pps
