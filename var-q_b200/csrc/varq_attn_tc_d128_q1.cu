// Tensor-core attention: head_dim 128, 16-bit queries, 1 query tile per CTA.
#include "varq_attn_tc.cuh"

namespace varq {
const TcFile tc_d128_q1 = {tc_launch_modes<128, 1, 1>, tc_file_status};
}
