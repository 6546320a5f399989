// Tensor-core attention: head_dim 64, 16-bit queries, 2 query tiles per CTA.
#include "varq_attn_tc.cuh"

namespace varq {
const TcFile tc_d64_x2_q1 = {tc_launch_modes<64, 1, 2>, tc_file_status};
}
