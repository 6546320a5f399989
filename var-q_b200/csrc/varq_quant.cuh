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
// max(||x||_2, eps) of a row of 64 or 128 values held by 8 or 16 neighbouring lanes (lane w of the row: values 8w .. 8w + 7).  The order of
// the sum is that of qk_norm_stats_kernel, in which warp lane i chains the values i, i + 32, ... and the lanes fold by 16, 8, 4, 2, 1: a length
// that rounds the other way moves the codes of values on a rounding boundary, and with 16-bit rows 1 in 10^4 packed words has one.  The
// chains take a transposition first, values travelling in pairs (one register per pair of 16-bit inputs), and every fold but the last
// ones halves what a lane holds: 9 shuffles for 16-bit rows of 128, against 4 for an arbitrary order.
template <typename T> struct Pair8 { uint32_t v; };
template <> struct Pair8<float> { float2 v; };
__device__ __forceinline__ Pair8<float> pair_xor(const Pair8<float>& p, int m) {
    Pair8<float> r;
    r.v.x = __shfl_xor_sync(0xffffffffu, p.v.x, m); r.v.y = __shfl_xor_sync(0xffffffffu, p.v.y, m);
    return r;
}
template <typename T> __device__ __forceinline__ Pair8<T> pair_xor(const Pair8<T>& p, int m) { return {__shfl_xor_sync(0xffffffffu, p.v, m)}; }
__device__ __forceinline__ float2 pair_values(const Pair8<float>& p) { return p.v; }
__device__ __forceinline__ float2 pair_values(const Pair8<__nv_bfloat16>& p) { return make_float2(__uint_as_float(p.v << 16), __uint_as_float(p.v & 0xffff0000u)); }
__device__ __forceinline__ float2 pair_values(const Pair8<__half>& p) { return __half22float2(*reinterpret_cast<const __half2*>(&p.v)); }
template <typename T> __device__ __forceinline__ void get_pairs(const Vec8<T>& x, Pair8<T> (&p)[4]) {
    if constexpr (sizeof(T) == 4) { p[0].v = {x.a.x, x.a.y}; p[1].v = {x.a.z, x.a.w}; p[2].v = {x.b.x, x.b.y}; p[3].v = {x.b.z, x.b.w}; }
    else { p[0].v = x.r.x; p[1].v = x.r.y; p[2].v = x.r.z; p[3].v = x.r.w; }
}
template <typename T> __device__ __forceinline__ float row_length(const Vec8<T>& x, int tpr, int w, float eps) {
    auto fold = [](float s, int m) { return s + __shfl_xor_sync(0xffffffffu, s, m); };
    auto halve = [](float a, float b, bool keep_b, int m) {      // the kept one, plus the partner's (which keeps the other)
        return (keep_b ? b : a) + __shfl_xor_sync(0xffffffffu, keep_b ? a : b, m);
    };
    Pair8<T> p[4], got[2], lo[2], hi[2];
    get_pairs(x, p);
    const int far = tpr >> 1;                                    // lanes w and w ^ far: the highest bit of the chain index w / 4
    const bool up = (w & far) != 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) got[i] = pair_xor(up ? p[i] : p[2 + i], far);
#pragma unroll
    for (int i = 0; i < 2; ++i) { lo[i] = up ? got[i] : p[i]; hi[i] = up ? p[2 + i] : got[i]; }
    float s;
    if (tpr == 16) {
        const bool odd = (w & 4) != 0;
        const Pair8<T> l_got = pair_xor(odd ? lo[0] : lo[1], 4), h_got = pair_xor(odd ? hi[0] : hi[1], 4);
        const float2 c[4] = {pair_values(odd ? l_got : lo[0]), pair_values(odd ? lo[1] : l_got), pair_values(odd ? h_got : hi[0]), pair_values(odd ? hi[1] : h_got)};
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) { s0 = fmaf(c[e].x, c[e].x, s0); s1 = fmaf(c[e].y, c[e].y, s1); }
        s = halve(s0, s1, (w & 2) != 0, 2);                      // 16
        s = fold(fold(fold(fold(s, 1), 8), 4), 2);               // 8, 4, 2, 1
    } else {
        float2 t[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float2 c0 = pair_values(lo[i]), c1 = pair_values(hi[i]);
            t[i] = make_float2(fmaf(c1.x, c1.x, c0.x * c0.x), fmaf(c1.y, c1.y, c0.y * c0.y));
        }
        const bool k2 = (w & 2) != 0;
        const float s0 = halve(t[0].x, t[1].x, k2, 2), s1 = halve(t[0].y, t[1].y, k2, 2);      // 16
        s = halve(s0, s1, (w & 1) != 0, 1);                      // 8
        s = fold(fold(fold(s, 4), 2), 1);                        // 4, 2, 1
    }
    return fmaxf(sqrtf(s), eps);
}

// Quantize one or two tensors of a step in one launch where their groupings have a kernel for it (varq_append.cu); VARQ_ERR_UNSUPPORTED
// without a launch otherwise.  k_norm_eps >= 0: the first job's rows are L2-normalised on the way in.
int append_fast(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps, void* ws, size_t ws_bytes, cudaStream_t st);
size_t append_workspace_bytes(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps);

}  // namespace varq
