// Double-buffered copies of a block stream: everything one block needs on the
// copy stream (order after the consumer of the buffer's last block, halo, new
// rows, order before the next consumer) in one call.
//
// What bounds a streamed operation over page-locked data is the host link, if
// the host keeps up: enqueueing a block through the framework's stream and
// event objects took about 90 us of host time, as long as the link needs for
// 5 MB; in one call it is 15 us.  Folding 262144 x 256 8-bit samples in 17 blocks
// of 4 MB: 1.97 -> 1.70 ms (1.23 ms for the same bytes in one copy); dedispersing
// 65536 x 256 in 5 blocks: 0.58 -> 0.52 ms.
#include <new>

#include "spp_common.cuh"

namespace spp {

struct Blocks {
  cudaStream_t copy = nullptr, compute = nullptr;
  cudaEvent_t copied[2] = {}, consumed[2] = {};
  int last = -1;  // buffer of the block being consumed
};

static void blocks_free(Blocks* b) {
  for (int k = 0; k < 2; ++k) {
    if (b->copied[k]) cudaEventDestroy(b->copied[k]);
    if (b->consumed[k]) cudaEventDestroy(b->consumed[k]);
  }
  delete b;
}

}  // namespace spp

using namespace spp;

extern "C" int spp_blocks_create(void** handle, void* copy_stream, void* compute_stream) {
  if (!handle) return fail(SPP_ERR_ARG, "spp_blocks_create: null pointer");
  *handle = nullptr;
  Blocks* b = new (std::nothrow) Blocks;
  if (!b) return fail(SPP_ERR_SIZE, "spp_blocks_create: out of host memory");
  b->copy = reinterpret_cast<cudaStream_t>(copy_stream);
  b->compute = reinterpret_cast<cudaStream_t>(compute_stream);
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
    e = cudaEventCreateWithFlags(&b->copied[k], cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->consumed[k], cudaEventDisableTiming);
    // the buffers may be memory that earlier work on the compute stream still uses
    if (e == cudaSuccess) e = cudaEventRecord(b->consumed[k], b->compute);
  }
  if (e != cudaSuccess) {
    blocks_free(b);
    return cuda_status(e, "block stream events");
  }
  *handle = b;
  return SPP_OK;
}

extern "C" int spp_blocks_put(void* handle, int k, void* dst, const void* halo, int64_t halo_bytes,
                              const void* src, int64_t bytes) {
  Blocks* b = static_cast<Blocks*>(handle);
  if (!b || (k != 0 && k != 1) || !dst || (halo_bytes > 0 && !halo) || (bytes > 0 && !src))
    return fail(SPP_ERR_ARG, "spp_blocks_put: bad argument");
  if (halo_bytes < 0 || bytes < 0) return fail(SPP_ERR_SIZE, "spp_blocks_put: negative size");
  cudaError_t e = cudaSuccess;
  if (b->last >= 0) e = cudaEventRecord(b->consumed[b->last], b->compute);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(b->copy, b->consumed[k], 0);
  if (e == cudaSuccess && halo_bytes > 0)
    e = cudaMemcpyAsync(dst, halo, (size_t)halo_bytes, cudaMemcpyDeviceToDevice, b->copy);
  if (e == cudaSuccess && bytes > 0)
    e = cudaMemcpyAsync(static_cast<char*>(dst) + halo_bytes, src, (size_t)bytes,
                        cudaMemcpyHostToDevice, b->copy);
  if (e == cudaSuccess) e = cudaEventRecord(b->copied[k], b->copy);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(b->compute, b->copied[k], 0);
  b->last = k;
  return cuda_status(e, "block copy");
}

extern "C" int spp_blocks_wait(void* handle, int k) {
  Blocks* b = static_cast<Blocks*>(handle);
  if (!b || (k != 0 && k != 1)) return fail(SPP_ERR_ARG, "spp_blocks_wait: bad argument");
  return cuda_status(cudaEventSynchronize(b->copied[k]), "block copy");
}

extern "C" int spp_blocks_destroy(void* handle) {
  Blocks* b = static_cast<Blocks*>(handle);
  if (!b) return SPP_OK;
  const cudaError_t e = cudaStreamSynchronize(b->copy);
  blocks_free(b);
  return cuda_status(e, "block copies");
}
