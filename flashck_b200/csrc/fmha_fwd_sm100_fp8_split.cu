// Instances of the tcgen05 attention kernel: 8-bit operands, and the split modes.
#include "fmha_fwd_sm100.cuh"

namespace fck::sm100 {

FCK_SM100_FP8(FCK_SM100_INST, f8e4m3_t) FCK_SM100_FP8(FCK_SM100_INST, f8e5m2_t)
FCK_SM100_SPLIT(FCK_SM100_INST_SPLIT, __half) FCK_SM100_SPLIT(FCK_SM100_INST_SPLIT, __nv_bfloat16)

}  // namespace fck::sm100
