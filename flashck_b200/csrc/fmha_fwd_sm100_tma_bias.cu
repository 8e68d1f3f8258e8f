// Instances of the tcgen05 attention kernel: an elementwise bias tensor through shared memory.
#include "fmha_fwd_sm100.cuh"

namespace fck::sm100 {

FCK_SM100_TMA_BIAS(FCK_SM100_INST, __half) FCK_SM100_TMA_BIAS(FCK_SM100_INST, __nv_bfloat16)

}  // namespace fck::sm100
