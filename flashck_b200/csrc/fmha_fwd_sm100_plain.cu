// Instances of the tcgen05 attention kernel: no score additions, hdim 128 and 64.
#include "fmha_fwd_sm100.cuh"

namespace fck::sm100 {

FCK_SM100_PLAIN(FCK_SM100_INST, __half) FCK_SM100_PLAIN(FCK_SM100_INST, __nv_bfloat16)
FCK_SM100_HDIM64(FCK_SM100_INST, __half) FCK_SM100_HDIM64(FCK_SM100_INST, __nv_bfloat16)

}  // namespace fck::sm100
