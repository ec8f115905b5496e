// Collectives of a communicator whose ranks all sit on ONE GPU, without any rank-to-rank
// protocol: the daemon launches one kernel for all ranks once every rank's input exists, and
// the kernel's end is the moment every rank's output exists, so neither a start nor a closing
// barrier (nor a cooperative launch, nor a grid that has to be resident at once) is needed.
// What is left is a stream over memory: every input byte is read once, every output byte is
// written once.
//
//   group_reduce_kernel : AllReduce (grid.y = 1: n sources, n destinations) and ReduceScatter
//                         (grid.y = block: n sources, one destination)
//   group_gather_kernel : AllGather (grid.y = source rank: one source, n destinations)
//
// Each also carries up to kMaxBatch collectives in one launch (OneGpuBatchArgs): a launch of its
// own costs a short collective about 4 us of idle memory (first loads, last stores, completion
// word). Two communicators of two ranks x 16 calls of 8 MiB fp32 in one group: 300 us one by one,
// 199 us together, 164 us at the measured copy rate.
//
// Bound: HBM. A CTA handles one tile of blockDim.x * U packs of 16 bytes of every source and
// ends; the grid follows the message. Measured on a B200, 4 x 512 MiB fp32 read and written:
// 624 us = 6.88 TB/s, against 730 us for a grid of 4 CTAs per SM that loops over the tiles with
// the same inner loop (CTAs that end and are replaced keep more loads in flight than a loop
// whose every trip waits for its own loads). What has to be kept small is the register count:
// it is the number of resident warps that hides the latency, not the loads per thread
// (8 x 32 MiB bf16: 116 us at 106 registers, 85 us at 64).
//
// Buffers need not be 16-byte aligned. The `ragged` forms start their packs on a 16-byte boundary
// of the destinations; a source that sits at another phase is read as two aligned packs that are
// shifted into place (the second one is the next thread's first, a hit in L1).
#pragma once
#include "collectives.cuh"

namespace mccs {
namespace dev {

// Completion word of the launch, as finish() in collectives.cuh, for the whole grid at once.
// Everything the kernel wrote is memory of this GPU, so order at GPU scope is enough: the counts carry it
// from every CTA's stores to the last CTA, whose word is then a plain store to host memory. (A
// system-scope fence in front of it and a release store made every launch 3 us longer.)
__device__ __forceinline__ void one_gpu_finish(const OneGpuArgs& a) {
  if (a.counter == nullptr) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned last = gridDim.x * gridDim.y - 1;
    if (count_off(a.counter, last) == last) {
      if (a.trace) {
        const uint64_t t = globaltimer_ns();
        for (int r = 0; r < a.nranks; r++) st_relaxed_sys_u64(&a.status[r]->end_ns, t);
        fence_sys();
      }
      for (int r = 0; r < a.nranks; r++) st_relaxed_sys_u64(&a.status[r]->done_seq, a.seq);
    }
  }
}

__device__ __forceinline__ void one_gpu_begin(const OneGpuArgs& a) {
  wait_for_previous_kernel();
  if (a.trace && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    const uint64_t t = globaltimer_ns();
    for (int r = 0; r < a.nranks; r++) st_relaxed_sys_u64(&a.status[r]->start_ns, t);
  }
}

// What a CTA works on: the launch's one collective, or the member of a batch it belongs to.
struct OneGpuWork {
  const void* const* send;
  void* const* recv;
  uint64_t count;
  unsigned cta, ctas;   // this CTA's number among those of the collective
};
__device__ __forceinline__ const OneGpuArgs& launch_args(const OneGpuArgs& a) { return a; }
__device__ __forceinline__ const OneGpuArgs& launch_args(const OneGpuBatchArgs& b) { return b.base; }
__device__ __forceinline__ OneGpuWork my_work(const OneGpuArgs& a) { return {a.send, a.recv, a.count, blockIdx.x, gridDim.x}; }
__device__ __forceinline__ OneGpuWork my_work(const OneGpuBatchArgs& b) {
  unsigned k = 0;   // independent comparisons with constants instead of a search: no chain of loads
#pragma unroll
  for (int j = 1; j < kMaxBatch; j++) k += blockIdx.x >= b.first[j] ? 1u : 0u;
  const OneGpuMember& m = b.member[k];
  return {m.send, m.recv, m.count, blockIdx.x - b.first[k], b.first[k + 1] - b.first[k]};
}

// Sum (Op) of one element or pack of every source, in source order, as reduce_store does it:
// the same bits as the kernels with one CTA set per rank.
template <typename T, typename Op, int BYTES, int MAXS>
__device__ __forceinline__ Raw<BYTES> reduce_packs(const Raw<BYTES> (&v)[MAXS], int nsrc, Scaler<typename AccOf<T>::type> sc) {
  using P = Pack<T, BYTES>;
  using Acc = typename P::Acc;
  Acc acc[P::kN];
  P::unpack(v[0], acc);
  if (sc.mode == 1) {
#pragma unroll
    for (int e = 0; e < P::kN; e++) acc[e] = sc.mul(acc[e]);
  }
#pragma unroll
  for (int s = 1; s < MAXS; s++) {
    if (s < nsrc) {
      Acc x[P::kN];
      P::unpack(v[s], x);
#pragma unroll
      for (int e = 0; e < P::kN; e++) acc[e] = Op::apply(acc[e], sc.mode == 1 ? sc.mul(x[e]) : x[e]);
    }
  }
  if (sc.mode == 2) {
#pragma unroll
    for (int e = 0; e < P::kN; e++) acc[e] = sc.div(acc[e]);
  }
  return P::pack(acc);
}

// MAXS: ranks an instantiation has registers for (2, 4 or 8). 64, 48 and 40 registers per
// thread (but for the 8-bit types, whose sixteen 32-bit sums need their own): measured best of
// 2 to 8 CTAs of 256 threads per SM.
template <typename T, typename Op, int MAXS, typename Args = OneGpuArgs>
__global__ void __launch_bounds__(kGroupThreads, sizeof(T) == 1 ? 3 : MAXS == 8 ? 4 : MAXS == 4 ? 5 : 6)
group_reduce_kernel(const __grid_constant__ Args args) {
  const OneGpuArgs& a = launch_args(args);
  const OneGpuWork w = my_work(args);
  constexpr int U = MAXS <= 4 ? kReduceUnrollFew : 1;
  constexpr uint64_t kN = 16 / sizeof(T);
  const int n = a.nranks;
  const bool scatter = a.kind == kReduceScatter;
  const uint64_t block = scatter ? (uint64_t)blockIdx.y * w.count * sizeof(T) : 0;   // this group's first byte in every source
  const Scaler<typename AccOf<T>::type> sc{scaler_mode(a.op), a.scale};
  one_gpu_begin(a);
  auto one = [&](uint64_t off, auto bytes) {
    constexpr int B = decltype(bytes)::value;
    Raw<B> v[MAXS];
#pragma unroll
    for (int s = 0; s < MAXS; s++)
      if (s < n) v[s] = ld_local<B>((const char*)w.send[s] + (block + off));
    const Raw<B> out = reduce_packs<T, Op, B, MAXS>(v, n, sc);
    if (scatter) {
      st_local<B>((char*)w.recv[blockIdx.y] + off, out);
    } else {
#pragma unroll
      for (int d = 0; d < MAXS; d++)
        if (d < n) st_local<B>((char*)w.recv[d] + off, out);
    }
  };
  const uint64_t packs = w.count / kN;
  const uint64_t step = (uint64_t)w.ctas * blockDim.x * U;
#pragma unroll 1
  for (uint64_t i = (uint64_t)w.cta * blockDim.x * U + threadIdx.x; i < packs; i += step) {
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i + u * blockDim.x < packs) one((i + u * blockDim.x) * 16, std::integral_constant<int, 16>{});
  }
  if (w.cta == 0 && threadIdx.x < w.count - packs * kN)
    one((packs * kN + threadIdx.x) * sizeof(T), std::integral_constant<int, (int)sizeof(T)>{});
  one_gpu_finish(a);
}

// The same for buffers or blocks that do not all start on 16-byte boundaries.
template <typename T, typename Op, int MAXS, typename Args = OneGpuArgs>
__global__ void __launch_bounds__(kGroupThreads, sizeof(T) == 1 ? 3 : 4) group_reduce_ragged_kernel(const __grid_constant__ Args args) {
  const OneGpuArgs& a = launch_args(args);
  const OneGpuWork w = my_work(args);
  constexpr uint64_t kN = 16 / sizeof(T);
  const int n = a.nranks;
  const bool scatter = a.kind == kReduceScatter;
  const uint64_t block = scatter ? (uint64_t)blockIdx.y * w.count * sizeof(T) : 0;
  const Scaler<typename AccOf<T>::type> sc{scaler_mode(a.op), a.scale};
  one_gpu_begin(a);
  const PackSplit ps = split_packs(w.recv + blockIdx.y, scatter ? 1 : n, 0, w.count, sizeof(T));
  auto one = [&](uint64_t off, auto bytes) {
    constexpr int B = decltype(bytes)::value;
    Raw<B> v[MAXS];
#pragma unroll
    for (int s = 0; s < MAXS; s++) {
      if (s < n) {
        const char* p = (const char*)w.send[s] + (block + off);
        if constexpr (B == 16) v[s] = ld_shifted(p, (uint32_t)(uintptr_t)p & 15u);
        else v[s] = ld_local<B>(p);
      }
    }
    const Raw<B> out = reduce_packs<T, Op, B, MAXS>(v, n, sc);
    if (scatter) {
      st_local<B>((char*)w.recv[blockIdx.y] + off, out);
    } else {
#pragma unroll
      for (int d = 0; d < MAXS; d++)
        if (d < n) st_local<B>((char*)w.recv[d] + off, out);
    }
  };
  const uint64_t first = (uint64_t)w.cta * blockDim.x + threadIdx.x;
  const uint64_t step = (uint64_t)w.ctas * blockDim.x;
#pragma unroll 1
  for (uint64_t i = first; i < ps.packs; i += step) one(ps.head * sizeof(T) + i * 16, std::integral_constant<int, 16>{});
  // Elements outside the packs: a few, or all of them when the destinations' phases differ.
  const uint64_t single = w.count - ps.packs * kN;
#pragma unroll 1
  for (uint64_t k = first; k < single; k += step)
    one((k < ps.head ? k : k + ps.packs * kN) * sizeof(T), std::integral_constant<int, (int)sizeof(T)>{});
  one_gpu_finish(a);
}

#ifdef MCCS_UNTYPED_KERNELS
// All loads of a tile go out before its first store: with few destinations four packs per
// thread, with up to eight two (4 x 64 MiB on each of four ranks: 209 us against 380 us with one
// pack per thread, where the rate at which CTAs start, one in about 2.7 ns, is what bounds it).
template <int MAXD, typename Args = OneGpuArgs>
__global__ void __launch_bounds__(kGroupThreads, 4) group_gather_kernel(const __grid_constant__ Args args) {
  const OneGpuArgs& a = launch_args(args);
  const OneGpuWork w = my_work(args);
  constexpr int U = MAXD <= 4 ? kGatherUnrollFew : kGatherUnrollMany;
  const int n = a.nranks, g = (int)blockIdx.y;
  const uint64_t at = (uint64_t)g * w.count;   // the source's place in every destination
  const char* const src = (const char*)w.send[g];
  const int skip = src == (const char*)w.recv[g] + at ? g : -1;
  one_gpu_begin(a);
  const uint64_t packs = w.count / 16;   // the launcher asks for this form when nothing is left over
  const uint64_t step = (uint64_t)w.ctas * blockDim.x * U;
#pragma unroll 1
  for (uint64_t i = (uint64_t)w.cta * blockDim.x * U + threadIdx.x; i < packs; i += step) {
    Raw<16> v[U];
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i + u * blockDim.x < packs) v[u] = ld_local<16>(src + (i + u * blockDim.x) * 16);
#pragma unroll
    for (int d = 0; d < MAXD; d++) {
      if (d < n && d != skip) {
#pragma unroll
        for (int u = 0; u < U; u++)
          if (i + u * blockDim.x < packs) st_local<16>((char*)w.recv[d] + (at + (i + u * blockDim.x) * 16), v[u]);
      }
    }
  }
  one_gpu_finish(a);
}

// The same for any byte count and any alignment.
template <int MAXD, typename Args = OneGpuArgs>
__global__ void __launch_bounds__(kGroupThreads, 6) group_gather_ragged_kernel(const __grid_constant__ Args args) {
  const OneGpuArgs& a = launch_args(args);
  const OneGpuWork w = my_work(args);
  const int n = a.nranks, g = (int)blockIdx.y;
  const uint64_t at = (uint64_t)g * w.count;
  const char* const src = (const char*)w.send[g];
  const int skip = src == (const char*)w.recv[g] + at ? g : -1;
  one_gpu_begin(a);
  const PackSplit ps = split_packs(w.recv, n, at, w.count, 1);
  const uint32_t shift = (uint32_t)((uintptr_t)src + ps.head) & 15u;
  const uint64_t first = (uint64_t)w.cta * blockDim.x + threadIdx.x;
  const uint64_t step = (uint64_t)w.ctas * blockDim.x;
  auto store = [&](uint64_t off, auto v) {
#pragma unroll
    for (int d = 0; d < MAXD; d++)
      if (d < n && d != skip) st_local<(int)sizeof(v)>((char*)w.recv[d] + (at + off), v);
  };
#pragma unroll 1
  for (uint64_t i = first; i < ps.packs; i += step) store(ps.head + i * 16, ld_shifted(src + ps.head + i * 16, shift));
  const uint64_t single = w.count - ps.packs * 16;
#pragma unroll 1
  for (uint64_t k = first; k < single; k += step) {
    const uint64_t off = k < ps.head ? k : k + ps.packs * 16;
    store(off, ld_local<1>(src + off));
  }
  one_gpu_finish(a);
}
#endif  // MCCS_UNTYPED_KERNELS

}  // namespace dev
}  // namespace mccs
