// Tensor-core attention: head_dim 64, fp32 (hi + lo) queries, 2 query tiles per CTA.
#include "varq_attn_tc.cuh"

namespace varq {
const TcFile tc_d64_x2_q2 = {tc_launch_modes<64, 2, 2>, tc_file_status};
}
