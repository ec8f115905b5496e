// Kernels that do not depend on the element type: AllGather (bytes), the ring
// AllGather and the single-rank copy, plus their lookup function.
#define MCCS_UNTYPED_KERNELS 1
#include "collectives.cuh"
#include "one_gpu.cuh"

namespace mccs {
namespace dev {

extern "C" const void* mccs_kfn_untyped(int variant) {
  switch (variant) {
    case kAgPull: return (const void*)&ag_direct_kernel<kAgModePull>;
    case kAgPush: return (const void*)&ag_direct_kernel<kAgModePush>;
    case kAgNvls: return (const void*)&ag_direct_kernel<kAgModeNvls>;
    case kAgRing: return (const void*)&ag_ring_kernel;
    case kLocalCopy: return (const void*)&local_copy_kernel;
  }
  return nullptr;
}

extern "C" const void* mccs_kfn_local_copy_ragged() { return (const void*)&local_copy_ragged_kernel; }

template <typename Args>
static const void* gather_by_ranks(int nranks, bool ragged) {
  if (nranks <= 2) return ragged ? (const void*)&group_gather_ragged_kernel<2, Args> : (const void*)&group_gather_kernel<2, Args>;
  if (nranks <= 4) return ragged ? (const void*)&group_gather_ragged_kernel<4, Args> : (const void*)&group_gather_kernel<4, Args>;
  return ragged ? (const void*)&group_gather_ragged_kernel<8, Args> : (const void*)&group_gather_kernel<8, Args>;
}
extern "C" const void* mccs_kfn_group_gather(int nranks, int ragged, int batch) {
  return batch ? gather_by_ranks<OneGpuBatchArgs>(nranks, ragged != 0) : gather_by_ranks<OneGpuArgs>(nranks, ragged != 0);
}

}  // namespace dev
}  // namespace mccs
