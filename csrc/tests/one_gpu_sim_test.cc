// The one-GPU kernels of kernels/one_gpu.cuh (the source the GPU build compiles) on the SIMT
// emulator, against plain loops: every rank count and register class, counts around the pack
// and tile edges, every combination of 16-byte phases, in place, bounded grids, several
// collectives in one launch. Guard bytes
// around every output catch a store outside it, the emulator a misaligned access.
#include "sim/simt_sim.h"

#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <random>
#include <type_traits>

#define MCCS_UNTYPED_KERNELS 1
#include "../kernels/one_gpu.cuh"

using namespace mccs;
using namespace mccs::dev;

namespace {

int g_cases = 0, g_failed = 0;
constexpr size_t kGuard = 64;

struct Block {   // `bytes` bytes at phase `off` of a 16-byte boundary, guard bytes on both sides
  std::vector<uint8_t> raw;
  size_t bytes, start;
  Block(size_t n, size_t off) : raw(n + 3 * kGuard + 16, 0xA5), bytes(n) {
    start = kGuard + (16 - ((uintptr_t)raw.data() + kGuard) % 16) % 16 + off;
  }
  uint8_t* p() { return raw.data() + start; }
  bool guards_intact() {
    for (size_t i = 0; i < raw.size(); i++)
      if ((i < start || i >= start + bytes) && raw[i] != 0xA5) return false;
    return true;
  }
};

template <typename T> double value(T v) { return (double)v; }
template <> double value(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> double value(__half v) { return __half2float(v); }
template <typename T> T made(double v) { return (T)v; }
template <> __nv_bfloat16 made(double v) { return __float2bfloat16_rn((float)v); }
template <> __half made(double v) { return __float2half_rn((float)v); }

template <typename Kernel, typename Args>
void launch(Kernel k, const Args& a, int ctas, int groups, int threads) {
  std::vector<std::thread> pool;
  sim::Dim3 grid;
  grid.x = (unsigned)ctas;
  grid.y = (unsigned)groups;
  sim::launch(k, grid, (unsigned)threads, a, &pool);
  sim::join_all(&pool);
}

template <typename T, typename Op, int MAXS>
void launch_reduce(const OneGpuArgs& a, bool ragged, int ctas, int groups, int threads) {
  if (ragged) launch(group_reduce_ragged_kernel<T, Op, MAXS>, a, ctas, groups, threads);
  else launch(group_reduce_kernel<T, Op, MAXS>, a, ctas, groups, threads);
}

// send_off / recv_off: phase of each rank's buffers, in elements.
template <typename T, typename Op>
void reduce_case(int kind, int n, size_t count, int op, const std::vector<size_t>& send_off, const std::vector<size_t>& recv_off, bool in_place,
                 int ctas, int threads, unsigned seed) {
  std::mt19937 rng(seed);
  const size_t esz = sizeof(T);
  const bool scatter = kind == kReduceScatter;
  const size_t in_elems = scatter ? count * (size_t)n : count;
  std::vector<Block> send, recv;
  std::vector<std::vector<double>> x((size_t)n);
  OneGpuArgs a;
  memset(&a, 0, sizeof a);
  uint64_t bits = scatter ? count * esz : 0;
  for (int r = 0; r < n; r++) {
    send.emplace_back(in_elems * esz, send_off[(size_t)r] * esz);
    recv.emplace_back(in_place ? 0 : count * esz, recv_off[(size_t)r] * esz);
  }
  std::vector<StatusBlock> status((size_t)n);
  uint32_t counter = 0;
  for (int r = 0; r < n; r++) {
    memset(&status[(size_t)r], 0, sizeof(StatusBlock));
    T* s = (T*)send[(size_t)r].p();
    for (size_t i = 0; i < in_elems; i++) {
      s[i] = made<T>((double)((int)(rng() % 17) - (std::is_unsigned<T>::value ? 0 : 8)) * (std::is_integral<T>::value ? 1.0 : 0.25));
      x[(size_t)r].push_back(value(s[i]));
    }
    a.send[r] = s;
    a.recv[r] = in_place ? (void*)(s + (scatter ? (size_t)r * count : 0)) : (void*)recv[(size_t)r].p();
    a.status[r] = &status[(size_t)r];
    bits |= (uint64_t)a.send[r] | (uint64_t)a.recv[r];
  }
  a.count = count; a.nranks = n; a.kind = kind; a.op = op; a.scale = op == kSumPostDiv ? 1.0f / (float)n : 2.0f;
  a.counter = &counter; a.seq = 77;
  const bool ragged = (bits & 15u) != 0;
  const int groups = scatter ? n : 1;
  if (n <= 2) launch_reduce<T, Op, 2>(a, ragged, ctas, groups, threads);
  else if (n <= 4) launch_reduce<T, Op, 4>(a, ragged, ctas, groups, threads);
  else launch_reduce<T, Op, 8>(a, ragged, ctas, groups, threads);
  bool good = counter == 0;
  for (int r = 0; r < n; r++) {
    const T* d = (const T*)a.recv[r];
    for (size_t i = 0; i < count; i++) {
      const size_t at = (scatter ? (size_t)r * count : 0) + i;
      double want = x[0][at] * (op == kPreMulSum ? 2.0 : 1.0);
      for (int q = 1; q < n; q++) want = (double)Op::apply(want, x[(size_t)q][at] * (op == kPreMulSum ? 2.0 : 1.0));
      if (op == kSumPostDiv) want = std::is_integral<T>::value ? (double)(int64_t)(want / n) : value(made<T>(want * (double)a.scale));
      if (value(d[i]) != value(made<T>(want))) good = false;
    }
    good &= send[(size_t)r].guards_intact() && recv[(size_t)r].guards_intact() && status[(size_t)r].done_seq == 77;
  }
  g_cases++;
  if (!good) {
    g_failed++;
    fprintf(stderr, "FAILED: kind %d n %d count %zu esz %zu op %d in_place %d ragged %d ctas %d\n", kind, n, count, esz, op, in_place, ragged, ctas);
  }
}

void gather_case(int n, size_t count, const std::vector<size_t>& send_off, const std::vector<size_t>& recv_off, bool in_place, int ctas, int threads) {
  std::vector<Block> send, recv;
  for (int r = 0; r < n; r++) {
    send.emplace_back(in_place ? 0 : count, send_off[(size_t)r]);
    recv.emplace_back(count * (size_t)n, recv_off[(size_t)r]);
  }
  OneGpuArgs a;
  memset(&a, 0, sizeof a);
  uint64_t bits = count;
  for (int r = 0; r < n; r++) {
    uint8_t* s = in_place ? recv[(size_t)r].p() + (size_t)r * count : send[(size_t)r].p();
    for (size_t i = 0; i < count; i++) s[i] = (uint8_t)(i * 7 + (size_t)r * 31);
    a.send[r] = s;
    a.recv[r] = recv[(size_t)r].p();
    bits |= (uint64_t)a.send[r] | (uint64_t)a.recv[r];
  }
  a.count = count; a.nranks = n; a.kind = kAllGather;
  const bool ragged = (bits & 15u) != 0;
  auto go = [&](auto plain, auto rag) { ragged ? launch(rag, a, ctas, n, threads) : launch(plain, a, ctas, n, threads); };
  if (n <= 2) go(group_gather_kernel<2>, group_gather_ragged_kernel<2>);
  else if (n <= 4) go(group_gather_kernel<4>, group_gather_ragged_kernel<4>);
  else go(group_gather_kernel<8>, group_gather_ragged_kernel<8>);
  bool good = true;
  for (int r = 0; r < n; r++) {
    for (int q = 0; q < n; q++)
      for (size_t i = 0; i < count; i++) good &= recv[(size_t)r].p()[(size_t)q * count + i] == (uint8_t)(i * 7 + (size_t)q * 31);
    good &= recv[(size_t)r].guards_intact() && send[(size_t)r].guards_intact();
  }
  g_cases++;
  if (!good) { g_failed++; fprintf(stderr, "FAILED: gather n %d count %zu in_place %d ragged %d ctas %d\n", n, count, in_place, ragged, ctas); }
}

void copy_case(size_t count, size_t send_off, size_t recv_off, int ctas, int threads) {
  Block in(count, send_off), out(count, recv_off);
  for (size_t i = 0; i < count; i++) in.p()[i] = (uint8_t)(i * 11 + 3);
  SignalPad* pad = (SignalPad*)aligned_alloc(128, sizeof(SignalPad));
  memset(pad, 0, sizeof *pad);
  StatusBlock status;
  memset(&status, 0, sizeof status);
  CollArgs a;
  memset(&a, 0, sizeof a);
  a.nranks = 1;
  a.count = count;
  a.seq = 5;
  a.send[0] = in.p(); a.recv[0] = out.p();
  a.pad[0] = pad; a.status[0] = &status;
  std::vector<std::thread> pool;
  sim::Dim3 grid;
  grid.x = (unsigned)ctas;
  sim::launch(local_copy_ragged_kernel, grid, (unsigned)threads, a, &pool);
  sim::join_all(&pool);
  g_cases++;
  if (memcmp(in.p(), out.p(), count) != 0 || !out.guards_intact() || status.done_seq != 5 || pad->pad_[kPadCtaCounter] != 0) {
    g_failed++;
    fprintf(stderr, "FAILED: ragged copy of %zu bytes, phases %zu -> %zu, %d CTAs\n", count, send_off, recv_off, ctas);
  }
  free(pad);
}

// Several collectives in one launch: each member against plain loops, whatever CTAs it has (first[]
// as the launcher fills it, one CTA at least, `per` packs' worth of bytes each).
void batch_case(int kind, int n, const std::vector<size_t>& counts, size_t send_off, size_t recv_off, size_t per, int threads) {
  const bool gather = kind == kAllGather, scatter = kind == kReduceScatter;
  const size_t esz = gather ? 1 : sizeof(float), nn = (size_t)n;
  std::vector<Block> send, recv;
  send.reserve(counts.size() * nn);   // (blocks must not move)
  recv.reserve(counts.size() * nn);
  OneGpuBatchArgs b;
  memset(&b, 0, sizeof b);
  uint64_t bits = 0;
  unsigned ctas = 0;
  for (size_t k = 0; k < (size_t)kMaxBatch; k++) {
    b.first[k] = ctas;
    if (k >= counts.size()) continue;
    const size_t c = counts[k];
    ctas += (unsigned)std::max<size_t>((c * esz + per - 1) / per, 1);
    b.member[k].count = c;
    bits |= kind == kAllReduce ? 0 : c * esz;
    for (int r = 0; r < n; r++) {
      send.emplace_back(c * esz * (scatter ? nn : 1), send_off * esz);
      recv.emplace_back(c * esz * (gather ? nn : 1), recv_off * esz);
      uint8_t* sp = send.back().p();
      for (size_t i = 0; i < send.back().bytes / esz; i++) {
        if (gather) sp[i] = (uint8_t)(i * 7 + (size_t)r * 31 + k);
        else ((float*)sp)[i] = (float)((i * 3 + (size_t)r * 5 + k) % 23);
      }
      b.member[k].send[r] = sp;
      b.member[k].recv[r] = recv.back().p();
      bits |= (uint64_t)sp | (uint64_t)recv.back().p();
    }
  }
  b.first[kMaxBatch] = ctas;
  std::vector<StatusBlock> status(nn);
  uint32_t counter = 0;
  for (int r = 0; r < n; r++) { memset(&status[(size_t)r], 0, sizeof(StatusBlock)); b.base.status[r] = &status[(size_t)r]; }
  b.base.nranks = n; b.base.kind = kind; b.base.op = kSum; b.base.scale = 1.0f; b.base.counter = &counter; b.base.seq = 9;
  const bool ragged = (bits & 15u) != 0;
  const int groups = kind == kAllReduce ? 1 : n;
  auto go = [&](auto plain, auto rag) { ragged ? launch(rag, b, (int)ctas, groups, threads) : launch(plain, b, (int)ctas, groups, threads); };
  using B = OneGpuBatchArgs;
  if (gather) {
    if (n <= 2) go(group_gather_kernel<2, B>, group_gather_ragged_kernel<2, B>);
    else if (n <= 4) go(group_gather_kernel<4, B>, group_gather_ragged_kernel<4, B>);
    else go(group_gather_kernel<8, B>, group_gather_ragged_kernel<8, B>);
  } else {
    if (n <= 2) go(group_reduce_kernel<float, OpSum, 2, B>, group_reduce_ragged_kernel<float, OpSum, 2, B>);
    else if (n <= 4) go(group_reduce_kernel<float, OpSum, 4, B>, group_reduce_ragged_kernel<float, OpSum, 4, B>);
    else go(group_reduce_kernel<float, OpSum, 8, B>, group_reduce_ragged_kernel<float, OpSum, 8, B>);
  }
  bool good = counter == 0;
  for (size_t k = 0; k < counts.size(); k++)
    for (size_t r = 0; r < nn; r++) {
      Block& out = recv[k * nn + r];
      for (size_t i = 0; i < out.bytes / esz; i++) {
        if (gather) {
          good &= out.p()[i] == send[k * nn + i / counts[k]].p()[i % counts[k]];
        } else {
          float want = 0;
          for (size_t q = 0; q < nn; q++) want += ((const float*)send[k * nn + q].p())[(scatter ? r * counts[k] : 0) + i];
          good &= ((const float*)out.p())[i] == want;
        }
      }
      good &= out.guards_intact() && status[r].done_seq == 9;
    }
  g_cases++;
  if (!good) { g_failed++; fprintf(stderr, "FAILED: batch kind %d n %d members %zu ragged %d per %zu\n", kind, n, counts.size(), ragged, per); }
}

template <typename T>
void type_cases() {
  const size_t per = 16 / sizeof(T);
  for (int n = 2; n <= 8; n++) {
    const std::vector<size_t> zero((size_t)n, 0);
    unsigned seed = (unsigned)n * 1000;
    for (size_t count : {(size_t)1, per - 1 ? per - 1 : 1, per, 32 * per, 64 * per + 1, 150 * per + per / 2}) {
      for (int kind : {(int)kAllReduce, (int)kReduceScatter}) {
        reduce_case<T, OpSum>(kind, n, count, kSum, zero, zero, false, 2, 32, seed++);
        reduce_case<T, OpSum>(kind, n, count, kSumPostDiv, zero, zero, true, 1, 32, seed++);
        std::vector<size_t> same((size_t)n, per / 2), mixed, other((size_t)n, per - 1);
        for (int r = 0; r < n; r++) mixed.push_back((size_t)(r * 3) % per);
        reduce_case<T, OpSum>(kind, n, count, kSum, same, same, false, 3, 32, seed++);    // one phase everywhere
        reduce_case<T, OpMax>(kind, n, count, kMax, same, other, false, 2, 32, seed++);   // sources behind the destinations
        reduce_case<T, OpSum>(kind, n, count, kPreMulSum, mixed, zero, false, 2, 64, seed++);   // a phase of its own per source
        reduce_case<T, OpMin>(kind, n, count, kMin, zero, mixed, false, 2, 32, seed++);   // destinations apart: element by element
        reduce_case<T, OpSum>(kind, n, count, kSum, same, same, true, 2, 32, seed++);
      }
    }
  }
}

}  // namespace

int main() {
  type_cases<float>();
  type_cases<__nv_bfloat16>();
  type_cases<__half>();
  type_cases<double>();
  type_cases<int8_t>();
  type_cases<int64_t>();
  for (int n = 2; n <= 8; n++)
    for (size_t count : {(size_t)1, (size_t)15, (size_t)16, (size_t)1024, (size_t)1025, (size_t)3003}) {
      const std::vector<size_t> zero((size_t)n, 0), same((size_t)n, 5);
      std::vector<size_t> mixed;
      for (int r = 0; r < n; r++) mixed.push_back((size_t)(r * 5) % 16);
      gather_case(n, count, zero, zero, false, 2, 32);
      gather_case(n, count, zero, zero, true, 1, 32);
      gather_case(n, count, same, zero, false, 2, 32);
      gather_case(n, count, mixed, same, false, 2, 64);
      gather_case(n, count, zero, mixed, true, 2, 32);
    }
  for (int kind : {(int)kAllReduce, (int)kAllGather, (int)kReduceScatter})
    for (int n : {2, 3, 4, 8})
      for (size_t per : {(size_t)512, (size_t)1024}) {   // the tile of 32 threads is 512 bytes (one pack each) or a multiple
        batch_case(kind, n, {64, 1024, 16, 512}, 0, 0, per, 32);
        batch_case(kind, n, {1, 130, 4099, 7, 1000, 33, 2048, 1}, 0, 0, per, 32);
        batch_case(kind, n, {515, 515}, 3, 1, per, 32);
        batch_case(kind, n, {48}, 0, 0, per, 32);
      }
  for (size_t count : {(size_t)1, (size_t)15, (size_t)16, (size_t)31, (size_t)2048, (size_t)2049, (size_t)5003})
    for (size_t so = 0; so < 16; so++)
      for (size_t ro : {(size_t)0, (size_t)1, (size_t)8, (size_t)15}) copy_case(count, so, ro, 2, 32);
  printf("one_gpu_sim_test: %d cases, %d failed\n", g_cases, g_failed);
  return g_failed ? 1 : 0;
}
