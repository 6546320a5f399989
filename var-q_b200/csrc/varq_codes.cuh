// Packed codes as fp16 operands, shared by the tensor-core attention kernels.
#pragma once
#include "varq_common.cuh"

namespace varq {

// ---- packed integer codes -> fp16 without conversion instructions.
// 0x6400 | u is the fp16 number 1024 + u (0 <= u < 1024).  A field at bit position p of a 16-bit half gives 1024 + 2^p u without a
// shift; one packed multiply-add by 2^-p takes the factor and the zero-point out together (exact: all values are integers below
// 2048), so a word is unpacked with one logic operation per pair and one shift.  The pairs are then fields (i, i + 4) of a word of
// eight codes or (i, i + 8) of sixteen: operand tiles hold head_dim in that order, and the queries and outputs follow it.
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
    __half2 r = __hadd2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) {
    __half2 r = __hfma2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b), *reinterpret_cast<__half2*>(&c));
    return *reinterpret_cast<uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2_neg(uint32_t a) {       // an operand modifier of the instruction that takes it
    __half2 r = __hneg2(*reinterpret_cast<__half2*>(&a));
    return *reinterpret_cast<uint32_t*>(&r);
}
// head_dim index (inside a 16-code item) at operand position p
__host__ __device__ constexpr int code_at(int bits, int p) {
    return bits == 8 ? p : bits == 4 ? ((p & 8) | ((p & 1) << 2) | ((p & 7) >> 1)) : (((p & 1) << 3) | (p >> 1));
}
// and the operand position of head_dim index e
__host__ __device__ constexpr int code_pos(int bits, int e) {
    return bits == 8 ? e : bits == 4 ? ((e & 8) | ((e & 3) << 1) | ((e >> 2) & 1)) : (((e & 7) << 1) | (e >> 3));
}
__host__ __device__ constexpr int code_bias(int bits) { return bits == 8 ? 128 : bits == 4 ? 8 : 2; }
// The constants of the pairs as register values that the compiler cannot fold: (x & mask) ^ magic is one three-input logic instruction with
// the mask as its immediate only if the magic is in a register; with two known constants it became two instructions per pair, and
// logic instructions run at half rate.
static __constant__ uint32_t c_code_magic[3][4] = {{0x64026402u, 0x64086408u, 0x64206420u, 0x64806480u}, {0x64086408u, 0x64806480u, 0u, 0u}, {0x64646464u, 0u, 0u, 0u}};
template <int BITS> struct CodeMagic {
    static constexpr int N = BITS == 8 ? 1 : BITS == 4 ? 2 : 4;
    uint32_t m[N];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < N; ++i) {
            m[i] = c_code_magic[BITS == 2 ? 0 : BITS == 4 ? 1 : 2][i];
            asm volatile("" : "+r"(m[i]));
        }
    }
};
template <int BITS> struct Item {           // 16 consecutive codes of one key: 4, 2 or 1 packed words -> 8 pairs
    static constexpr int NW = BITS / 2;
    static constexpr int CLS = BITS == 8 ? 1 : BITS == 4 ? 2 : 4;      // classes of bit position: pair i has class i % CLS
    // pairs holding 1024 + 2^p (code + bias)
    static __device__ __forceinline__ void raw(const uint32_t* w, uint32_t (&h)[8], const CodeMagic<BITS>& cm) {
        if constexpr (BITS == 8) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t u = w[i] ^ 0x80808080u;
                h[2 * i] = __byte_perm(u, cm.m[0], 0x4140);
                h[2 * i + 1] = __byte_perm(u, cm.m[0], 0x4342);
            }
        } else if constexpr (BITS == 4) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint32_t x = w[i], y = w[i] >> 8;
                h[4 * i] = (x & 0x000F000Fu) ^ cm.m[0];
                h[4 * i + 1] = (x & 0x00F000F0u) ^ cm.m[1];
                h[4 * i + 2] = (y & 0x000F000Fu) ^ cm.m[0];
                h[4 * i + 3] = (y & 0x00F000F0u) ^ cm.m[1];
            }
        } else {
            const uint32_t x = w[0], y = w[0] >> 8;
            h[0] = (x & 0x00030003u) ^ cm.m[0]; h[1] = (x & 0x000C000Cu) ^ cm.m[1];
            h[2] = (x & 0x00300030u) ^ cm.m[2]; h[3] = (x & 0x00C000C0u) ^ cm.m[3];
            h[4] = (y & 0x00030003u) ^ cm.m[0]; h[5] = (y & 0x000C000Cu) ^ cm.m[1];
            h[6] = (y & 0x00300030u) ^ cm.m[2]; h[7] = (y & 0x00C000C0u) ^ cm.m[3];
        }
    }
    // -(1024 / 2^p + bias) of a class, before the zero-point
    static __host__ __device__ constexpr float neg_base(int cls) {
        return -(float)((BITS == 8 ? 1024 : BITS == 4 ? (cls == 0 ? 1024 : 64) : (cls == 0 ? 1024 : cls == 1 ? 256 : cls == 2 ? 64 : 16)) + code_bias(BITS));
    }
    // code - zp of pair i; nz[class] = -(1024 / 2^p + bias + zp) twice
    static __device__ __forceinline__ uint32_t minus_zp(uint32_t raw, int i, uint32_t nz) {
        const int cls = i % CLS;
        if (cls == 0) return h2_add(raw, nz);
        return h2_fma(raw, BITS == 4 ? 0x2C002C00u : cls == 1 ? 0x34003400u : cls == 2 ? 0x2C002C00u : 0x24002400u, nz);
    }
    // the classes' constants from that of class 0 (exact integers)
    static __device__ __forceinline__ void spread(uint32_t nz0, uint32_t (&nz)[CLS]) {
        nz[0] = nz0;
        if constexpr (BITS == 4) nz[1] = h2_add(nz0, 0x63806380u);                     // + 960
        if constexpr (BITS == 2) {
            nz[1] = h2_add(nz0, 0x62006200u);                                         // + 768
            nz[2] = h2_add(nz0, 0x63806380u);                                         // + 960
            nz[3] = h2_add(nz0, 0x63E063E0u);                                         // + 1008
        }
    }
};

}  // namespace varq
