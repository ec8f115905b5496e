// Host-side entry to the collective kernels: kernel lookup by (variant, type, op)
// and the launch itself. The reference picks among five precompiled symbols
// (src/mccs/src/proxy/plan.rs:142-166) and launches grid = channels
// (plan.rs:637-669); here the grid is CTAs per rank, times ranks when one
// cooperative launch emulates every rank on a single GPU.
#pragma once
#include <cuda_runtime.h>

#include "dev_types.h"

namespace mccs {

const void* kernel_function(int variant, int dtype, int op);
cudaError_t launch_collective(int kind, const CollArgs& args, LaunchDims dims, void* stream);
// Largest CTA count per rank that keeps an emulated (cooperative) launch resident.
int max_cooperative_ctas(int variant, int dtype, int op, int threads, int nranks);

// Every rank of a communicator that shares one GPU, in one launch without rank-to-rank protocol
// (one_gpu.cuh): `args` as for an emulated launch_collective; `completion`: publish args.seq in
// the status blocks; `max_ctas` > 0 bounds the grid (in CTAs of 512 threads), otherwise it follows
// the message.
cudaError_t launch_one_gpu(int kind, const CollArgs& args, int max_ctas, bool completion, void* stream);
// The kernel such a launch runs; null when there is none for this type and operator.
const void* one_gpu_function(int kind, int dtype, int op, int nranks, bool ragged, bool batch = false);
// The copy of a communicator of one rank; `ragged`: not both buffers are 16-byte aligned.
const void* local_copy_function(bool ragged);
// Several such collectives in one launch, with a completion word (b.base.seq).
cudaError_t launch_one_gpu_batch(const BatchArgs& b, void* stream);

// Fused AllReduce (several members in one launch, see batch.cuh). Only the two-shot
// variants have a fused form; returns null / cudaErrorInvalidDeviceFunction otherwise.
const void* batch_kernel_function(int variant, int dtype, int op);
cudaError_t launch_batch(const BatchArgs& args, LaunchDims dims, void* stream);
int max_cooperative_batch_ctas(int variant, int dtype, int op, int threads, int nranks);

}  // namespace mccs
