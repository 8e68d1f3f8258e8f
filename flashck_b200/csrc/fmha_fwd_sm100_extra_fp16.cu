// Instances of the tcgen05 attention kernel: ALiBi and logits soft cap, hdim 128, fp16.
#include "fmha_fwd_sm100.cuh"

namespace fck::sm100 {

FCK_SM100_EXTRA(FCK_SM100_INST, __half)

}  // namespace fck::sm100
