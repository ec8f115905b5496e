#include "launch.h"

#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>

extern "C" {
const void* mccs_kfn_i8(int, int);
const void* mccs_kfn_u8(int, int);
const void* mccs_kfn_i32(int, int);
const void* mccs_kfn_u32(int, int);
const void* mccs_kfn_i64(int, int);
const void* mccs_kfn_u64(int, int);
const void* mccs_kfn_f16(int, int);
const void* mccs_kfn_f32(int, int);
const void* mccs_kfn_f64(int, int);
const void* mccs_kfn_bf16(int, int);
const void* mccs_kfn_untyped(int);
const void* mccs_kfn_local_copy_ragged();
const void* mccs_kfn_one_gpu_i8(int, int, int, int);
const void* mccs_kfn_one_gpu_u8(int, int, int, int);
const void* mccs_kfn_one_gpu_i32(int, int, int, int);
const void* mccs_kfn_one_gpu_u32(int, int, int, int);
const void* mccs_kfn_one_gpu_i64(int, int, int, int);
const void* mccs_kfn_one_gpu_u64(int, int, int, int);
const void* mccs_kfn_one_gpu_f16(int, int, int, int);
const void* mccs_kfn_one_gpu_f32(int, int, int, int);
const void* mccs_kfn_one_gpu_f64(int, int, int, int);
const void* mccs_kfn_one_gpu_bf16(int, int, int, int);
const void* mccs_kfn_group_gather(int, int, int);
const void* mccs_kfn_batch_i8(int, int);
const void* mccs_kfn_batch_u8(int, int);
const void* mccs_kfn_batch_i32(int, int);
const void* mccs_kfn_batch_u32(int, int);
const void* mccs_kfn_batch_i64(int, int);
const void* mccs_kfn_batch_u64(int, int);
const void* mccs_kfn_batch_f16(int, int);
const void* mccs_kfn_batch_f32(int, int);
const void* mccs_kfn_batch_f64(int, int);
const void* mccs_kfn_batch_bf16(int, int);
}

namespace mccs {

const void* batch_kernel_function(int variant, int dtype, int op);

const void* kernel_function(int variant, int dtype, int op) {
  if (variant == kOneGpu) return one_gpu_function(kAllReduce, dtype, op, 2, false);   // every type and operator has all forms
  if (variant == kArHybrid || variant == kRsDirect || variant == kRsNvls)
    return batch_kernel_function(variant, dtype, op);   // live with the newer kernels
  switch (variant) {
    case kAgPull: case kAgPush: case kAgNvls: case kAgRing: case kLocalCopy:
      return mccs_kfn_untyped(variant);
    default: break;
  }
  switch (dtype) {
    case kInt8: return mccs_kfn_i8(variant, op);
    case kUint8: return mccs_kfn_u8(variant, op);
    case kInt32: return mccs_kfn_i32(variant, op);
    case kUint32: return mccs_kfn_u32(variant, op);
    case kInt64: return mccs_kfn_i64(variant, op);
    case kUint64: return mccs_kfn_u64(variant, op);
    case kFloat16: return mccs_kfn_f16(variant, op);
    case kFloat32: return mccs_kfn_f32(variant, op);
    case kFloat64: return mccs_kfn_f64(variant, op);
    case kBfloat16: return mccs_kfn_bf16(variant, op);
  }
  return nullptr;
}

const void* batch_kernel_function(int variant, int dtype, int op) {
  switch (dtype) {
    case kInt8: return mccs_kfn_batch_i8(variant, op);
    case kUint8: return mccs_kfn_batch_u8(variant, op);
    case kInt32: return mccs_kfn_batch_i32(variant, op);
    case kUint32: return mccs_kfn_batch_u32(variant, op);
    case kInt64: return mccs_kfn_batch_i64(variant, op);
    case kUint64: return mccs_kfn_batch_u64(variant, op);
    case kFloat16: return mccs_kfn_batch_f16(variant, op);
    case kFloat32: return mccs_kfn_batch_f32(variant, op);
    case kFloat64: return mccs_kfn_batch_f64(variant, op);
    case kBfloat16: return mccs_kfn_batch_bf16(variant, op);
  }
  return nullptr;
}

const void* one_gpu_function(int kind, int dtype, int op, int nranks, bool ragged, bool batch) {
  if (kind == kAllGather) return mccs_kfn_group_gather(nranks, ragged, batch);
  switch (dtype) {
    case kInt8: return mccs_kfn_one_gpu_i8(nranks, op, ragged, batch);
    case kUint8: return mccs_kfn_one_gpu_u8(nranks, op, ragged, batch);
    case kInt32: return mccs_kfn_one_gpu_i32(nranks, op, ragged, batch);
    case kUint32: return mccs_kfn_one_gpu_u32(nranks, op, ragged, batch);
    case kInt64: return mccs_kfn_one_gpu_i64(nranks, op, ragged, batch);
    case kUint64: return mccs_kfn_one_gpu_u64(nranks, op, ragged, batch);
    case kFloat16: return mccs_kfn_one_gpu_f16(nranks, op, ragged, batch);
    case kFloat32: return mccs_kfn_one_gpu_f32(nranks, op, ragged, batch);
    case kFloat64: return mccs_kfn_one_gpu_f64(nranks, op, ragged, batch);
    case kBfloat16: return mccs_kfn_one_gpu_bf16(nranks, op, ragged, batch);
  }
  return nullptr;
}

const void* local_copy_function(bool ragged) { return ragged ? mccs_kfn_local_copy_ragged() : mccs_kfn_untyped(kLocalCopy); }

static int cooperative_fit(const void* fn, int threads, int nranks) {
  if (!fn || nranks <= 0) return 0;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess) return 0;
  return sms * per_sm / nranks;
}

int max_cooperative_batch_ctas(int variant, int dtype, int op, int threads, int nranks) {
  return cooperative_fit(batch_kernel_function(variant, dtype, op), threads, nranks);
}

cudaError_t launch_batch(const BatchArgs& args, LaunchDims dims, void* stream) {
  const CollArgs& a = args.base;
  const void* fn = batch_kernel_function(a.variant, a.dtype, a.op);
  if (!fn) return cudaErrorInvalidDeviceFunction;
  if (args.nops < 1 || args.nops > kMaxBatch) return cudaErrorInvalidValue;
  if (dims.ctas < 1 || dims.ctas > kMaxCtas || dims.threads < 32 || dims.threads > 512)
    return cudaErrorInvalidConfiguration;
  dim3 grid((unsigned)dims.ctas, a.emulated ? (unsigned)a.nranks : 1u, 1u);
  dim3 block((unsigned)dims.threads, 1u, 1u);
  BatchArgs b = args;
  void* params[] = {(void*)&b};
  if (a.emulated && a.nranks > 1) return cudaLaunchCooperativeKernel(fn, grid, block, params, 0, (cudaStream_t)stream);
  return cudaLaunchKernel(fn, grid, block, params, 0, (cudaStream_t)stream);
}

int max_cooperative_ctas(int variant, int dtype, int op, int threads, int nranks) {
  const void* fn = kernel_function(variant, dtype, op);
  if (!fn || nranks <= 0) return 0;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess) return 0;
  return sms * per_sm / nranks;
}

// Launch of a kernel that no other GPU takes part in. It may be set up while the kernel in front of
// it on the stream is still draining (it waits for that one's end in its first instruction): 1 to 2 us
// less between two kernels of a stream.
static cudaError_t launch_local(const void* fn, dim3 grid, dim3 block, void** params, void* stream) {
  cudaLaunchAttribute overlap;
  overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  overlap.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = (cudaStream_t)stream;
  cfg.attrs = &overlap;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, fn, params);
}

// Threads per CTA and packs of 16 bytes per thread and tile, for `packs` packs in all per group.
struct OneGpuTile { uint64_t threads, unroll; };
static OneGpuTile one_gpu_tile(int kind, int n, bool ragged, uint64_t packs) {
  const uint64_t groups = kind == kAllReduce ? 1 : (uint64_t)n;
  const uint64_t unroll = ragged ? 1
                          : kind == kAllGather ? (n <= 4 ? kGatherUnrollFew : kGatherUnrollMany)
                                               : (n <= 4 ? kReduceUnrollFew : 1);
  // 128 threads measured as fast as or faster than 256, as long as a CTA moves 16 KiB: the GPU
  // starts one CTA in about 2.7 ns, so smaller ones cannot keep up with the memory. The reduction
  // over more than four ranks needs the larger CTA for large messages (eight ranks scattering
  // 200 MiB each in blocks of 25 MiB: 273 us against 352 us) but not for a few waves, where what counts is how
  // evenly the last CTAs end. The shortest messages are spread until every SM has a CTA.
  const uint64_t buffers = (kind == kAllGather ? 1 : (uint64_t)n) + (kind == kReduceScatter ? 1 : (uint64_t)n);
  uint64_t threads = 128;
  if (threads * unroll * 16 * buffers < 16384 || (kind != kAllGather && n > 4 && packs * groups >= 16ull * kMaxCtas * kGroupThreads * unroll))
    threads = kGroupThreads;
  while (threads > 32 && packs * groups < (uint64_t)kMaxCtas * threads * unroll) threads /= 2;
  return {threads, unroll};
}

// Whether a collective's buffers or blocks leave the 16-byte grid.
static bool one_gpu_ragged(int kind, int n, uint64_t bytes, const void* const* send, void* const* recv) {
  uint64_t bits = kind == kAllReduce ? 0 : bytes;   // blocks start at multiples of their size
  for (int r = 0; r < n; r++) bits |= (uint64_t)send[r] | (uint64_t)recv[r];
  return (bits & 15u) != 0;
}

static void one_gpu_common(int kind, const CollArgs& args, bool completion, OneGpuArgs* a) {
  memset(a, 0, sizeof *a);
  for (int r = 0; r < args.nranks; r++) a->status[r] = args.status[r];
  a->nranks = args.nranks;
  a->kind = kind;
  a->op = args.op;
  a->trace = args.trace;
  a->scale = args.scale;
  a->seq = args.seq;
  a->counter = completion ? &args.pad[0]->pad_[kPadOneGpuCounter] : nullptr;
}

// The runtime loads a kernel's code at its first use, which takes milliseconds. Whoever launches one
// collective of a sort may soon have several go out together: that form is loaded at the first
// launch of the plain one, not in the middle of a stream of short kernels.
static void load_batch_form(int kind, int dtype, int op, int n, bool ragged) {
  constexpr int kDevices = 64;
  static std::atomic<bool> loaded[kDevices][kNumCollKinds][kNumDataTypes][kNumRedOps][3][2];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices || dtype < 0 || dtype >= kNumDataTypes || op < 0 || op >= kNumRedOps) return;
  std::atomic<bool>& done = loaded[dev][kind][dtype][op][n <= 2 ? 0 : n <= 4 ? 1 : 2][ragged ? 1 : 0];
  if (done.load(std::memory_order_relaxed)) return;
  cudaFuncAttributes attr;
  const void* fn = one_gpu_function(kind, dtype, op, n, ragged, true);
  if (fn && cudaFuncGetAttributes(&attr, fn) != cudaSuccess) cudaGetLastError();   // the batch's launch will report it
  done.store(true, std::memory_order_relaxed);
}

cudaError_t launch_one_gpu(int kind, const CollArgs& args, int max_ctas, bool completion, void* stream) {
  const int n = args.nranks;
  if (n < 2 || n > kMaxRanks) return cudaErrorInvalidValue;
  const uint64_t bytes = args.count * (uint64_t)(kind == kAllGather ? 1 : dtype_size(args.dtype));   // one rank's part, or one block
  OneGpuArgs a;
  one_gpu_common(kind, args, completion, &a);
  for (int r = 0; r < n; r++) {
    a.send[r] = args.send[r];
    a.recv[r] = args.recv[r];
  }
  a.count = args.count;
  const bool ragged = one_gpu_ragged(kind, n, bytes, a.send, a.recv);
  const void* fn = one_gpu_function(kind, args.dtype, args.op, n, ragged);
  if (!fn) return cudaErrorInvalidDeviceFunction;
  const uint64_t groups = kind == kAllReduce ? 1 : (uint64_t)n;
  const uint64_t packs = (bytes + 15) / 16;
  if (completion) load_batch_form(kind, args.dtype, args.op, n, ragged);
  OneGpuTile tile = one_gpu_tile(kind, n, ragged, packs);
  uint64_t ctas = (packs + tile.threads * tile.unroll - 1) / (tile.threads * tile.unroll);
  if (max_ctas > 0 && ctas * groups * tile.threads > (uint64_t)max_ctas * 512) {
    // A bounded grid (a tenant's share of the SMs, counted in CTAs of 512 threads) loops over the tiles.
    tile.threads = kGroupThreads;
    ctas = ((uint64_t)max_ctas * 512 / tile.threads + groups - 1) / groups;
  }
  if (ctas < 1) ctas = 1;
  if (ctas > 0x7fffffffull) ctas = 0x7fffffffull;
  void* params[] = {(void*)&a};
  return launch_local(fn, dim3((unsigned)ctas, (unsigned)groups, 1u), dim3((unsigned)tile.threads, 1u, 1u), params, stream);
}

cudaError_t launch_one_gpu_batch(const BatchArgs& b, void* stream) {
  const int n = b.base.nranks, kind = b.kind;
  if (n < 2 || n > kMaxRanks || b.nops < 1 || b.nops > kMaxBatch) return cudaErrorInvalidValue;
  const uint64_t esz = (uint64_t)(kind == kAllGather ? 1 : dtype_size(b.base.dtype));
  OneGpuBatchArgs a;
  memset(&a, 0, sizeof a);
  one_gpu_common(kind, b.base, true, &a.base);
  bool ragged = false;   // one member off the 16-byte grid makes it the ragged form for all
  uint64_t packs = 0;
  for (int k = 0; k < b.nops; k++) {
    OneGpuMember& m = a.member[k];
    for (int r = 0; r < n; r++) {
      m.send[r] = b.send[k][r];
      m.recv[r] = b.recv[k][r];
    }
    m.count = b.count[k];
    ragged |= one_gpu_ragged(kind, n, m.count * esz, m.send, m.recv);
    packs += (m.count * esz + 15) / 16;
  }
  const void* fn = one_gpu_function(kind, b.base.dtype, b.base.op, n, ragged, true);
  if (!fn) return cudaErrorInvalidDeviceFunction;
  const OneGpuTile tile = one_gpu_tile(kind, n, ragged, packs);
  const uint64_t per = tile.threads * tile.unroll * 16;
  uint64_t ctas = 0;
  for (int k = 0; k < kMaxBatch; k++) {
    a.first[k] = (uint32_t)ctas;
    if (k < b.nops) ctas += std::max<uint64_t>((b.count[k] * esz + per - 1) / per, 1);
    if (ctas > 0x7fffffffull) return cudaErrorInvalidValue;   // (members are bounded far below by what is worth fusing)
  }
  a.first[kMaxBatch] = (uint32_t)ctas;
  void* params[] = {(void*)&a};
  return launch_local(fn, dim3((unsigned)ctas, (unsigned)(kind == kAllReduce ? 1 : n), 1u), dim3((unsigned)tile.threads, 1u, 1u), params, stream);
}

cudaError_t launch_collective(int kind, const CollArgs& args, LaunchDims dims, void* stream) {
  CollArgs a = args;
  if (a.variant == kLocalCopy && kind_reduces(kind)) a.count = args.count * (uint64_t)dtype_size(args.dtype);
  const void* fn = kernel_function(a.variant, a.dtype, a.op);
  if (!fn) return cudaErrorInvalidDeviceFunction;
  if (dims.ctas < 1 || dims.ctas > kMaxCtas || dims.threads < 32 || dims.threads > 512)
    return cudaErrorInvalidConfiguration;
  if (variant_is_ring(a.variant) && dims.ctas > kMaxRingChannels) return cudaErrorInvalidConfiguration;
  if (a.variant == kLocalCopy) {
    // No CTA of a copy waits for another one, so the grid follows the message instead of the
    // plan: one CTA per tile (see local_copy_kernel), bounded so that the tile loop takes over
    // for messages beyond 16 GiB.
    const uint64_t tile = kCopyTileBytes;
    uint64_t ctas = (a.count + tile - 1) / tile;
    dims.ctas = (int32_t)(ctas < 1 ? 1 : ctas > (1u << 20) ? (1u << 20) : ctas);
    dims.threads = kCopyThreads;
  }
  dim3 grid((unsigned)dims.ctas, a.emulated ? (unsigned)a.nranks : 1u, 1u);
  dim3 block((unsigned)dims.threads, 1u, 1u);
  void* params[] = {(void*)&a};
  if (a.variant == kLocalCopy) {
    fn = local_copy_function((((uint64_t)a.send[a.rank] | (uint64_t)a.recv[a.rank]) & 15u) != 0);
    return launch_local(fn, grid, block, params, stream);
  }
  if (a.emulated && a.nranks > 1) {
    // All ranks' CTAs wait on one another, so they must be resident together.
    return cudaLaunchCooperativeKernel(fn, grid, block, params, 0, (cudaStream_t)stream);
  }
  return cudaLaunchKernel(fn, grid, block, params, 0, (cudaStream_t)stream);
}

}  // namespace mccs
