// Tensor-core attention: head_dim 128, fp32 (hi + lo) queries, 1 query tile per CTA.
#include "varq_attn_tc.cuh"

namespace varq {
const TcFile tc_d128_q2 = {tc_launch_modes<128, 2, 1>, tc_file_status};
}
