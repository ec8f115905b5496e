// One translation unit per element type (same -DMCCS_T / -DMCCS_TNAME scheme as
// inst_dtype.cu): instantiates the reducing kernels of one_gpu.cuh for up to two, four and eight
// ranks and exports their lookup function.
#include "one_gpu.cuh"

namespace mccs {
namespace dev {

#define MCCS_CAT2(a, b) a##b
#define MCCS_CAT(a, b) MCCS_CAT2(a, b)

template <typename Op, typename Args>
static const void* by_ranks(int nranks, bool ragged) {
  if (nranks <= 2) return ragged ? (const void*)&group_reduce_ragged_kernel<MCCS_T, Op, 2, Args> : (const void*)&group_reduce_kernel<MCCS_T, Op, 2, Args>;
  if (nranks <= 4) return ragged ? (const void*)&group_reduce_ragged_kernel<MCCS_T, Op, 4, Args> : (const void*)&group_reduce_kernel<MCCS_T, Op, 4, Args>;
  return ragged ? (const void*)&group_reduce_ragged_kernel<MCCS_T, Op, 8, Args> : (const void*)&group_reduce_kernel<MCCS_T, Op, 8, Args>;
}
template <typename Op>
static const void* by_form(int nranks, bool ragged, bool batch) {
  return batch ? by_ranks<Op, OneGpuBatchArgs>(nranks, ragged) : by_ranks<Op, OneGpuArgs>(nranks, ragged);
}

extern "C" const void* MCCS_CAT(mccs_kfn_one_gpu_, MCCS_TNAME)(int nranks, int op, int ragged, int batch) {
  switch (op) {
    case kSum: case kPreMulSum: case kSumPostDiv: return by_form<OpSum>(nranks, ragged != 0, batch != 0);
    case kProd: return by_form<OpProd>(nranks, ragged != 0, batch != 0);
    case kMax: return by_form<OpMax>(nranks, ragged != 0, batch != 0);
    case kMin: return by_form<OpMin>(nranks, ragged != 0, batch != 0);
  }
  return nullptr;
}

}  // namespace dev
}  // namespace mccs
