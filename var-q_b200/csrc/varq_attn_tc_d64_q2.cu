// Tensor-core attention: head_dim 64, fp32 (hi + lo) queries, 1 query tile per CTA.
#include "varq_attn_tc.cuh"

namespace varq {
const TcFile tc_d64_q2 = {tc_launch_modes<64, 2, 1>, tc_file_status};
}
