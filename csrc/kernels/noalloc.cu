// Allocation-free local AllReduce (see csrc/include/mccs_noalloc.h for who needs it
// and the rules). The kernel is the one-GPU AllReduce of one_gpu.cuh without a completion word:
// one pass over the buffers in an ordinary launch, no rank-to-rank protocol and so no signal
// pads, status blocks or other scratch to allocate, clear or share between calls. (The two-shot
// kernel it used before needed a cooperative launch, a memset of its pads in front and a grid
// small enough to be resident: 8 x 32 MiB bf16 took 106 us against 86 us.)
#include "../include/mccs_noalloc.h"

#include <cuda_runtime.h>
#include <string.h>

#include "dev_types.h"
#include "launch.h"

namespace {

static_assert(MCCS_NOALLOC_MAX_RANKS <= mccs::kMaxRanks, "more ranks than the kernels support");

bool overlap_without_identity(const void* a, const void* b, size_t bytes) {
  if (a == b) return false;
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return x < y ? y - x < bytes : x - y < bytes;
}

}  // namespace

extern "C" int mccsLocalAllReduceNoAllocPrepare(void) {
  using namespace mccs;
  // Asking for a kernel's attributes makes the runtime load its code now instead of at the
  // first launch.
  auto load = [](const void* fn) {
    cudaFuncAttributes attr;
    return fn ? cudaFuncGetAttributes(&attr, fn) : cudaErrorInvalidDeviceFunction;
  };
  for (int dt : {(int)kFloat32, (int)kFloat16, (int)kBfloat16})
    for (int n : {2, 4, MCCS_NOALLOC_MAX_RANKS})
      for (bool ragged : {false, true}) {
        cudaError_t e = load(one_gpu_function(kAllReduce, dt, kSum, n, ragged));
        if (e != cudaSuccess) return (int)e;
      }
  for (bool ragged : {false, true}) {   // one buffer: a copy
    cudaError_t e = load(local_copy_function(ragged));
    if (e != cudaSuccess) return (int)e;
  }
  return (int)cudaSuccess;
}

extern "C" int mccsLocalAllReduceNoAllocStatus(mccsNoAllocStatus_t* status, void* stream) {
  if (!status) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return (int)e;
  memset(status, 0, sizeof *status);   // nothing in the kernel waits, so there is no wait that could have run out
  return (int)cudaSuccess;
}

extern "C" int mccsLocalAllReduceNoAlloc(const void* const* in, void* const* out, int nranks, size_t count, int dtype,
                                         void* stream) {
  using namespace mccs;
  if (!in || !out || nranks < 1 || nranks > MCCS_NOALLOC_MAX_RANKS) return (int)cudaErrorInvalidValue;
  if (dtype != kFloat32 && dtype != kFloat16 && dtype != kBfloat16) return (int)cudaErrorInvalidValue;
  if (count == 0) return (int)cudaSuccess;
  const uint64_t bytes = (uint64_t)count * (uint64_t)dtype_size(dtype);
  for (int r = 0; r < nranks; r++)
    if (!in[r] || !out[r]) return (int)cudaErrorInvalidValue;
  // Identical buffers are fine (see the header); anything that overlaps partly is not.
  for (int r = 0; r < nranks; r++)
    for (int q = 0; q < nranks; q++) {
      if (overlap_without_identity(out[r], in[q], (size_t)bytes)) return (int)cudaErrorInvalidValue;
      if (q > r && (out[r] == out[q] || overlap_without_identity(out[r], out[q], (size_t)bytes))) return (int)cudaErrorInvalidValue;
    }
  CollArgs a;
  memset(&a, 0, sizeof a);
  a.rank = 0;
  a.nranks = nranks;
  a.dtype = dtype;
  a.op = kSum;
  a.variant = nranks > 1 ? kOneGpu : kLocalCopy;
  a.count = count;
  a.scale = 1.0f;
  for (int r = 0; r < nranks; r++) {
    a.send[r] = in[r];
    a.recv[r] = out[r];
  }
  if (nranks > 1) return (int)launch_one_gpu(kAllReduce, a, 0, false, stream);
  return (int)launch_collective(kAllReduce, a, LaunchDims{1, kCopyThreads}, stream);
}
