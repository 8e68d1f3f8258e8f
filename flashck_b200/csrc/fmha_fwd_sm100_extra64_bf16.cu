// Instances of the tcgen05 attention kernel: ALiBi and logits soft cap, hdim 64, bf16.
#include "fmha_fwd_sm100.cuh"

namespace fck::sm100 {

FCK_SM100_EXTRA64(FCK_SM100_INST, __nv_bfloat16)

}  // namespace fck::sm100
