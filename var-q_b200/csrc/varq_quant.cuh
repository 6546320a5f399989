// What the quantize kernels share: group ranges, scale / zero-point of a range, the length of a row.
#pragma once
#include "varq_common.cuh"

namespace varq {

struct Range { uint32_t hi, lo; };      // hi = max f2ord(x or |x|), lo = max ~f2ord(x)

__device__ __forceinline__ void range_init(Range& r) { r.hi = 0u; r.lo = 0u; }
__device__ __forceinline__ void range_add(Range& r, float v, bool symmetric) {
    if (symmetric) {
        r.hi = max(r.hi, f2ord(fabsf(v)));
    } else {
        const uint32_t o = f2ord(v);
        r.hi = max(r.hi, o);
        r.lo = max(r.lo, ~o);
    }
}
__device__ __forceinline__ void range_merge(Range& r, const Range& o) { r.hi = max(r.hi, o.hi); r.lo = max(r.lo, o.lo); }

// scale / zero-point of a group from its range
__device__ __forceinline__ void params_from_range(const Range& r, int bits, bool symmetric, float eps, float& scale,
                                                  float& zp) {
    if (symmetric) {
        const float amax = ord2f(r.hi);
        scale = fmaxf(__fdiv_rn(amax, (float)((1 << (bits - 1)) - 1)), eps);
        zp = 0.0f;
    } else {
        const float mx = ord2f(r.hi), mn = ord2f(~r.lo);
        scale = fmaxf(__fdiv_rn(__fsub_rn(mx, mn), (float)((1 << bits) - 1)), eps);
        zp = __fadd_rn(rintf(__fsub_rn(-(float)(1 << (bits - 1)), __fdiv_rn(mn, scale))), 0.0f);
    }
}
constexpr float Q_MAGIC = 12582912.0f;       // 1.5 * 2^23: adding it rounds to an integer and leaves that in the low mantissa bits

// eight consecutive values of a row in registers: 16-bit inputs stay packed until they are needed
template <typename T> struct Vec8;
template <> struct Vec8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) { a = __ldg(reinterpret_cast<const float4*>(p)); b = __ldg(reinterpret_cast<const float4*>(p) + 1); }
    __device__ __forceinline__ void get(float (&v)[8]) const { v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w; }
};
template <> struct Vec8<__nv_bfloat16> {
    uint4 r;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ void get(float (&v)[8]) const {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
    }
};
template <> struct Vec8<__half> {
    uint4 r;
    __device__ __forceinline__ void load(const __half* p) { r = __ldg(reinterpret_cast<const uint4*>(p)); }
    __device__ __forceinline__ void get(float (&v)[8]) const {
        const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i])); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
    }
};
// max(||x||_2, eps) of a row held by `tpr` neighbouring lanes (8 or 16), eight values each.  Every kernel that normalises rows for the
// quantizers takes the sum in this order, so that they produce the same bits and the same codes.
__device__ __forceinline__ float row_length(const float (&v)[8], int tpr, float eps) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
    for (int m = 1; m < tpr; m <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
    return fmaxf(sqrtf(ss), eps);
}

// Quantize one or two tensors of a step in one launch where their groupings have a kernel for it (varq_append.cu); VARQ_ERR_UNSUPPORTED
// without a launch otherwise.  k_norm_eps >= 0: the first job's rows are L2-normalised on the way in.
int append_fast(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps, void* ws, size_t ws_bytes, cudaStream_t st);
size_t append_workspace_bytes(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps);

}  // namespace varq
