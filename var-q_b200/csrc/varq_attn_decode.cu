// Attention of a few queries (up to eight per CTA) over a long packed cache: warp-level tensor-core instructions fed straight from
// global memory.
//
// The work is to stream the packed cache once, so the kernel is built around instructions per key: mma.sync m16n8k16 takes 16 keys x 16
// head_dim values of fp16 codes as its A operand, and its fragment layout lets every thread unpack whole words it loaded itself -- no
// shared memory, no conversion instructions.
//   S^T = K Q^T   A = 16 keys x codes: thread (g, c) of a warp (g = lane / 4, c = lane % 4) holds keys g and g + 8 and a quarter of the
//                 head_dim, contiguous in memory (the order of the contraction index is free as long as Q follows it);
//   O^T = V^T P^T A = codes x 16 keys: thread (g, c) holds an eighth of the head_dim of keys 2c, 2c + 1, 2c + 8, 2c + 9; pairs of keys
//                 are joined by byte permutes, and P^T is the transpose of S^T's fragment (movmatrix).
// The eight B columns are four queries as fp16 hi + lo: Q and P enter with 22 bits, codes are exact, scales and zero-points are applied
// in fp32 (K: s_k (acc - z_k sum q); V: the scale goes into P, the zero-point term is summed per query and taken off at the end), so the
// result has the accuracy of fp32 arithmetic.  NT column tiles share one unpacked K / V (NT = 2: eight queries).
// A warp walks over 16 keys at a time with the next tile's loads in flight; warps and CTAs (key ranges) are merged by the usual
// log-sum-exp rule, partial results of a split in the layout of the small-query kernel.
// Measured (B64 H16 c128, one bf16 query over 10 521 tokens, int4): 0.95 ms on the CUDA cores (254 instructions per four keys), see the
// figures at the dispatch rule for this kernel.  Bound by instruction issue at 2 and 4 bits, HBM at 8.
// Applies to one scale / zero-point per key (per token, per token and head) at head_dim 64 and 128.
#include <cfloat>
#include <type_traits>

#include "varq_attn.cuh"
#include "varq_codes.cuh"

namespace varq {

void attn_small_merge_launch(const AttnArgs& a, int n_qtiles, cudaStream_t st);

namespace {

constexpr int DC_WARPS = 4;
constexpr int DC_QT = 4;             // queries per column tile (matches the merge kernel's record layout)
constexpr float DC_LAZY = 8.f;       // a query keeps its reference maximum until a score exceeds it by this (log2 units)

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ float dc_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float dc_lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float dc_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// `BYTES` of a row -> words (two bytes: the low half of one word)
template <int BYTES> struct Raw {
    static constexpr int NW = BYTES < 4 ? 1 : BYTES / 4;
    uint32_t w[NW];
    __device__ __forceinline__ void load(const unsigned char* p) {
        if constexpr (BYTES == 2) w[0] = __ldg(reinterpret_cast<const unsigned short*>(p));
        else if constexpr (BYTES == 4) w[0] = __ldg(reinterpret_cast<const uint32_t*>(p));
        else if constexpr (BYTES == 8) { const uint2 v = __ldg(reinterpret_cast<const uint2*>(p)); w[0] = v.x; w[1] = v.y; }
        else {
#pragma unroll
            for (int i = 0; i < BYTES / 16; ++i) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(p) + i);
                w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
            }
        }
    }
};
// 8 pairs of raw halves -> signed codes: fp16 pairs of -(1024 / 2^p + bias) by bit position, as bit patterns (a conversion function would
// not be folded at compile time)
template <int BITS> __host__ __device__ constexpr uint32_t neg_base_h2(int cls) {
    return BITS == 8 ? 0xE480E480u : BITS == 4 ? (cls == 0 ? 0xE408E408u : 0xD480D480u)
                                               : (cls == 0 ? 0xE402E402u : cls == 1 ? 0xDC08DC08u : cls == 2 ? 0xD420D420u : 0xCC80CC80u);
}
template <int BITS> __device__ __forceinline__ void to_codes(uint32_t (&h)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = Item<BITS>::minus_zp(h[i], i, neg_base_h2<BITS>(i % Item<BITS>::CLS));
}
// the words of two keys -> words whose halves (bytes at 8 bits) alternate between the keys, so that unpacking them yields pairs
// (first key, second key) of one head_dim element each, in element order
template <int BITS, int NW> __device__ __forceinline__ void join_keys(const uint32_t (&a)[NW], const uint32_t (&b)[NW], uint32_t (&o)[2 * NW]) {
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        o[2 * i] = __byte_perm(a[i], b[i], BITS == 8 ? 0x5140 : 0x5410);
        o[2 * i + 1] = __byte_perm(a[i], b[i], BITS == 8 ? 0x7362 : 0x7632);
    }
}

template <int KB, int VB, int D, int NT, bool ZP>
__global__ void __launch_bounds__(DC_WARPS * 32, NT > 1 && D == 128 ? 2 : (KB == 8 || VB == 8 || NT > 1) ? 3 : 4) attn_decode_kernel(AttnArgs a, int keys_per_split, int q_tiles4) {
    constexpr int KBYTES = D / 4 * KB / 8, VBYTES = D / 8 * VB / 8;       // of a row and thread
    constexpr unsigned KROW = D * KB / 8, VROW = D * VB / 8;             // bytes between tokens
    constexpr int KITEMS = D / 64, VITEMS = D / 64;                       // 16-code items of K per row, 8-pair items of V per key pair
    constexpr int KSTEPS = D / 16, MT = D / 16;                          // contraction steps of S, row tiles of O
    __shared__ float s_part[DC_WARPS][DC_QT * NT][D + 2];

    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const unsigned blk = blockIdx.x;                        // query tile fastest, then key range, then (sample, head)
    const int qtile = (int)(blk % (unsigned)a.n_qtiles);
    const int split = (int)((blk / (unsigned)a.n_qtiles) % (unsigned)a.splits);
    const int bh = (int)(blk / ((unsigned)a.splits * (unsigned)a.n_qtiles)), b = bh / a.H, h = bh - b * a.H;
    const int q0 = qtile * (DC_QT * NT);

    // ---- Q fragments: column g = query g % 4 of the tile, hi (g < 4) or lo half; scaled by a power of two to use fp16's range
    uint32_t qf[NT][KSTEPS][2];
    float qfac[NT][2], qsum[NT][2];        // of this thread's two score columns (queries 2 (c % 2), + 1): scale_log2 / power of two, scale_log2 * sum q
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        float v[D / 4];
        const int qi = q0 + t * DC_QT + (g & 3);
        float mx = 0.f, sum = 0.f, ss = 0.f;
#pragma unroll
        for (int j = 0; j < D / 4; j += 8) {
            float e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (qi < a.Lq) load_q8(a.q, a.q_dtype, b * a.qs_b + (long long)qi * a.qs_l + h * a.qs_h + c * (D / 4) + j, e);
#pragma unroll
            for (int i = 0; i < 8; ++i) { v[j + i] = e[i]; mx = fmaxf(mx, fabsf(e[i])); sum += e[i]; ss = fmaf(e[i], e[i], ss); }
        }
        if (a.q_norm) {                 // x / max(||x||_2, eps) * scale_mul[h], on the way in
            ss += __shfl_xor_sync(0xffffffffu, ss, 1); ss += __shfl_xor_sync(0xffffffffu, ss, 2);
            const float f = (a.q_mul ? __ldg(a.q_mul + h) : 1.f) / fmaxf(sqrtf(ss), a.q_eps);
#pragma unroll
            for (int j = 0; j < D / 4; ++j) v[j] *= f;
            mx *= fabsf(f); sum *= f;
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1)); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        sum += __shfl_xor_sync(0xffffffffu, sum, 1); sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        // 2^(8 - exponent of the largest element), inside fp32's range
        const int ex = min(max((int)(__float_as_uint(mx) >> 23), 40), 240);
        const float f = __uint_as_float((uint32_t)(262 - ex) << 23), fi = __uint_as_float((uint32_t)(ex - 8) << 23);
#pragma unroll
        for (int s = 0; s < KSTEPS; ++s)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int p = 2 * s + r, d = (p >> 3) * 16;
                const float x0 = v[d + code_at(KB, 2 * (p & 7))] * f, x1 = v[d + code_at(KB, 2 * (p & 7) + 1)] * f;
                const __half2 hh = __floats2half2_rn(x0, x1);
                const float2 hf = __half22float2(hh);
                const __half2 hl = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
                qf[t][s][r] = g < 4 ? *reinterpret_cast<const uint32_t*>(&hh) : *reinterpret_cast<const uint32_t*>(&hl);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int src = (2 * (c & 1) + e) * 4;          // a lane of that query
            qfac[t][e] = __shfl_sync(0xffffffffu, fi, src) * a.scale_log2;
            qsum[t][e] = __shfl_sync(0xffffffffu, sum, src) * a.scale_log2;
        }
    }

    float o[NT][MT][4], m[NT][2], l[NT][2], corr[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
#pragma unroll
        for (int i = 0; i < MT; ++i) { o[t][i][0] = 0.f; o[t][i][1] = 0.f; o[t][i][2] = 0.f; o[t][i][3] = 0.f; }
#pragma unroll
        for (int e = 0; e < 2; ++e) { m[t][e] = -1e30f; l[t][e] = 0.f; corr[t][e] = 0.f; }
    }
    const unsigned char* kbase = reinterpret_cast<const unsigned char*>(a.kc + b * a.ks_b + h * a.ks_h) + c * KBYTES;
    const unsigned char* vbase = reinterpret_cast<const unsigned char*>(a.vc + b * a.vs_b + h * a.vs_h) + g * VBYTES;
    CodeMagic<KB> kmagic;
    CodeMagic<VB> vmagic;
    kmagic.init();
    vmagic.init();
    // per-token parameters of key g; a tensor without zero-points reads its scales in their place and drops them
    const long long kpar = a.kp.index(b, 0, h, 0), vpar = a.vp.index(b, 0, h, 0);
    const float *ksc = a.kp.scale + kpar, *vsc = a.vp.scale + vpar;
    const float *kzp = a.kp.zp ? a.kp.zp + kpar : ksc, *vzp = a.vp.zp ? a.vp.zp + vpar : vsc;
    const float kz_on = a.kp.zp ? 1.f : 0.f, vz_on = a.vp.zp ? 1.f : 0.f;
    const int ksr = (int)a.kp.sr, vsr = (int)a.vp.sr;

    const int k_begin = split * keys_per_split, k_end = min(a.Lk, k_begin + keys_per_split);
    struct Tile {
        Raw<KBYTES> k[2];                  // keys g, g + 8
        Raw<VBYTES> v[4];                  // keys 2c, 2c + 1, 2c + 8, 2c + 9
        float ks[2], kz[2], vs[2], vz[2];  // of keys g, g + 8
    };
    const int last = k_end - 1;
    // parameters of the two keys; a full tile needs no clamping, and its packed rows lie at constant offsets from one address
    auto fetch_par = [&](Tile& t, int key0, int key1) {
        const int k0_ = key0 * ksr, v0_ = key0 * vsr, k1_ = key1 * ksr, v1_ = key1 * vsr;
        t.ks[0] = __ldg(ksc + k0_); t.ks[1] = __ldg(ksc + k1_);
        t.vs[0] = __ldg(vsc + v0_); t.vs[1] = __ldg(vsc + v1_);
        if (ZP) {
            t.kz[0] = __ldg(kzp + k0_) * kz_on; t.kz[1] = __ldg(kzp + k1_) * kz_on;
            t.vz[0] = __ldg(vzp + v0_) * vz_on; t.vz[1] = __ldg(vzp + v1_) * vz_on;
        }
    };
    auto fetch = [&](Tile& t, int k0) {
        const unsigned char *kp = kbase + (unsigned)(k0 + g) * KROW, *vp = vbase + (unsigned)(k0 + 2 * c) * VROW;
        t.k[0].load(kp);
        t.k[1].load(kp + 8 * KROW);
        t.v[0].load(vp);
        t.v[1].load(vp + VROW);
        t.v[2].load(vp + 8 * VROW);
        t.v[3].load(vp + 9 * VROW);
        fetch_par(t, k0 + g, k0 + g + 8);
    };
    auto fetch_tail = [&](Tile& t, int k0) {
#pragma unroll
        for (int r = 0; r < 2; ++r) t.k[r].load(kbase + (unsigned)min(k0 + g + 8 * r, last) * KROW);
#pragma unroll
        for (int r = 0; r < 4; ++r) t.v[r].load(vbase + (unsigned)min(k0 + 2 * c + (r & 1) + 8 * (r >> 1), last) * VROW);
        fetch_par(t, min(k0 + g, last), min(k0 + g + 8, last));
    };
    auto process = [&](const Tile& cur, int k0, auto tail) {
        constexpr bool TAIL = decltype(tail)::value;
        // ---- S^T: 16 keys x 8 columns per tile
        float s[NT][4];
        {
            float s2[NT][2][4];
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int z = 0; z < 2; ++z) { s2[t][z][0] = 0.f; s2[t][z][1] = 0.f; s2[t][z][2] = 0.f; s2[t][z][3] = 0.f; }
#pragma unroll
            for (int it = 0; it < KITEMS; ++it) {
                uint32_t ka[8], kb[8];
                uint32_t w[Item<KB>::NW];
#pragma unroll
                for (int i = 0; i < Item<KB>::NW; ++i) w[i] = cur.k[0].w[it * Item<KB>::NW + i];
                Item<KB>::raw(w, ka, kmagic);
                to_codes<KB>(ka);
#pragma unroll
                for (int i = 0; i < Item<KB>::NW; ++i) w[i] = cur.k[1].w[it * Item<KB>::NW + i];
                Item<KB>::raw(w, kb, kmagic);
                to_codes<KB>(kb);
#pragma unroll
                for (int s4 = 0; s4 < 4; ++s4) {
                    const uint32_t af[4] = {ka[2 * s4], kb[2 * s4], ka[2 * s4 + 1], kb[2 * s4 + 1]};
#pragma unroll
                    for (int t = 0; t < NT; ++t) mma16816(s2[t][s4 & 1], af, qf[t][it * 4 + s4][0], qf[t][it * 4 + s4][1]);
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[t][i] = s2[t][0][i] + s2[t][1][i];
                    s[t][i] += __shfl_xor_sync(0xffffffffu, s[t][i], 2);          // hi + lo columns
                }
        }
        // ---- scores in the log2 domain with the V scale folded in, probabilities as fp16 hi (c < 2) or lo columns
        uint32_t pf[NT][2];
        float lv[2], rv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) { const float vs = fmaxf(cur.vs[r], 1e-30f); lv[r] = dc_lg2(vs); rv[r] = dc_rcp(vs); }
        bool over = false;
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float x = fmaf(cur.ks[r], ZP ? fmaf(s[t][2 * r + e], qfac[t][e], -cur.kz[r] * qsum[t][e]) : s[t][2 * r + e] * qfac[t][e], lv[r]);
                    s[t][2 * r + e] = !TAIL || k0 + g + 8 * r < k_end ? x : -1e30f;
                    over = over | (s[t][2 * r + e] > m[t][e] + DC_LAZY);
                }
        if (__any_sync(0xffffffffu, over)) {
            // rare after the first tile: new reference maxima, the same in every lane of a query, and everything accumulated is rescaled
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float x = fmaxf(s[t][e], s[t][2 + e]);
#pragma unroll
                    for (int z = 4; z < 32; z <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, z));
                    const float mn = fmaxf(m[t][e], x), alpha = dc_ex2(m[t][e] - mn);
                    m[t][e] = mn;
                    l[t][e] *= alpha; corr[t][e] *= alpha;
#pragma unroll
                    for (int i = 0; i < MT; ++i) { o[t][i][e] *= alpha; o[t][i][2 + e] *= alpha; }
                }
        }
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float p0 = dc_ex2(s[t][2 * r] - m[t][0]), p1 = dc_ex2(s[t][2 * r + 1] - m[t][1]);      // softmax weight x V scale
                l[t][0] = fmaf(p0, rv[r], l[t][0]); l[t][1] = fmaf(p1, rv[r], l[t][1]);
                if (ZP) { corr[t][0] = fmaf(p0, cur.vz[r], corr[t][0]); corr[t][1] = fmaf(p1, cur.vz[r], corr[t][1]); }
                const __half2 hh = __floats2half2_rn(p0, p1);
                const float2 hf = __half22float2(hh);
                const __half2 hl = __floats2half2_rn(p0 - hf.x, p1 - hf.y);
                pf[t][r] = transpose8x8(c < 2 ? *reinterpret_cast<const uint32_t*>(&hh) : *reinterpret_cast<const uint32_t*>(&hl));
            }
        // ---- O^T += V^T P^T
        uint32_t ja[2 * Raw<VBYTES>::NW], jb[2 * Raw<VBYTES>::NW];
        join_keys<VB>(cur.v[0].w, cur.v[1].w, ja);
        join_keys<VB>(cur.v[2].w, cur.v[3].w, jb);
#pragma unroll
        for (int it = 0; it < VITEMS; ++it) {
            uint32_t va[8], vb_[8];
            uint32_t w[Item<VB>::NW];
#pragma unroll
            for (int i = 0; i < Item<VB>::NW; ++i) w[i] = ja[it * Item<VB>::NW + i];
            Item<VB>::raw(w, va, vmagic);
            to_codes<VB>(va);
#pragma unroll
            for (int i = 0; i < Item<VB>::NW; ++i) w[i] = jb[it * Item<VB>::NW + i];
            Item<VB>::raw(w, vb_, vmagic);
            to_codes<VB>(vb_);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t af[4] = {va[2 * i], va[2 * i + 1], vb_[2 * i], vb_[2 * i + 1]};
#pragma unroll
                for (int t = 0; t < NT; ++t) mma16816(o[t][it * 4 + i], af, pf[t][0], pf[t][1]);
            }
        }
    };
    // full tiles in two buffers that take turns, the next one's loads in flight; then the ragged end
    constexpr int STEP = DC_WARPS * 16;
    const int full_end = k_begin + ((k_end - k_begin) & ~15);
    Tile ta, tb;
    int k0 = k_begin + warp * 16;
    if (k0 < full_end) fetch(ta, k0);
#pragma unroll 1
    while (k0 < full_end) {
        if (k0 + STEP < full_end) fetch(tb, k0 + STEP);
        process(ta, k0, std::false_type());
        k0 += STEP;
        if (k0 >= full_end) break;
        if (k0 + STEP < full_end) fetch(ta, k0 + STEP);
        process(tb, k0, std::false_type());
        k0 += STEP;
    }
    if (k0 < k_end) {
        fetch_tail(ta, k0);
        process(ta, k0, std::true_type());
    }
    // ---- a warp's partial result: hi + lo columns, sums over the keys of the lanes
#pragma unroll
    for (int t = 0; t < NT; ++t) {
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int z = 4; z < 32; z <<= 1) {
                l[t][e] += __shfl_xor_sync(0xffffffffu, l[t][e], z);
                corr[t][e] += __shfl_xor_sync(0xffffffffu, corr[t][e], z);
            }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                const float x = o[t][i][z] + __shfl_xor_sync(0xffffffffu, o[t][i][z], 2);
                // row g (z < 2) or g + 8 of row tile i = elements 2 i, 2 i + 1 of this thread's eighth of the head_dim
                if (c < 2) s_part[warp][t * DC_QT + 2 * c + (z & 1)][g * (D / 8) + 2 * i + (z >> 1)] = x - corr[t][z & 1];
            }
        if (g == 0 && c < 2) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                s_part[warp][t * DC_QT + 2 * c + e][D] = m[t][e];
                s_part[warp][t * DC_QT + 2 * c + e][D + 1] = l[t][e];
            }
        }
    }
    __syncthreads();
    // ---- merge the warps, then write the output or this split's partial record
    for (int i = threadIdx.x; i < DC_QT * NT * D; i += DC_WARPS * 32) {
        const int qi = i / D, d = i - qi * D;
        if (q0 + qi >= a.Lq) break;
        float M = -FLT_MAX;
#pragma unroll
        for (int w = 0; w < DC_WARPS; ++w) M = fmaxf(M, s_part[w][qi][D]);
        float num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < DC_WARPS; ++w) {
            const float wt = exp2f(s_part[w][qi][D] - M);
            num = fmaf(wt, s_part[w][qi][d], num);
            den = fmaf(wt, s_part[w][qi][D + 1], den);
        }
        if (a.splits == 1) {
            store_o_elem(a.out, a.o_dtype, b * a.os_b + (long long)(q0 + qi) * a.os_l + h * a.os_h + d, num / den);
        } else {
            const int t4 = qtile * NT + qi / DC_QT, q4 = qi % DC_QT;
            float* rec = a.ws + (((long long)bh * q_tiles4 + t4) * a.splits + split) * (DC_QT * (2 + D));
            rec[DC_QT * 2 + q4 * D + d] = num;
            if (d == 0) { rec[q4] = M; rec[DC_QT + q4] = den; }
        }
    }
}

// Key ranges per (sample, head): the count that makes the whole waves of CTAs (four per SM) shortest, a CTA costing its keys plus about 250
// keys' worth of set-up and merging.
int decode_splits(int B, int H, int Lq, int Lk, int& keys_per_split) {
    const int unit = DC_WARPS * 16;
    const long long base = (long long)B * H * ((Lq + 2 * DC_QT - 1) / (2 * DC_QT)), room = (long long)sm_count() * 4;
    long long best = 0;
    int splits = 1;
    for (int s = 1; s <= Lk / 256 || s == 1; ++s) {
        const long long kps = ((Lk + s - 1) / s + unit - 1) / unit * unit, cost = (base * s + room - 1) / room * (kps + 250);
        if (best == 0 || cost < best) { best = cost; splits = s; }
        if (base * s > 16 * room) break;
    }
    keys_per_split = (int)(((Lk + splits - 1) / splits + unit - 1) / unit) * unit;
    return (Lk + keys_per_split - 1) / keys_per_split;
}

template <int KB, int VB, int D, int NT>
int launch_decode(AttnArgs& a, int keys_per_split, cudaStream_t st) {
    const int n4 = (a.Lq + DC_QT - 1) / DC_QT;
    a.n_qtiles = (a.Lq + DC_QT * NT - 1) / (DC_QT * NT);
    const long long blocks = (long long)a.B * a.H * a.n_qtiles * a.splits;
    if (blocks > 0x7fffffffLL) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: more than 2^31 thread blocks");
    VARQ_CUDA_TRY(a.kp.zp || a.vp.zp ? launch_pdl(attn_decode_kernel<KB, VB, D, NT, true>, (unsigned)blocks, DC_WARPS * 32, 0, st, 1, a, keys_per_split, n4)
                                     : launch_pdl(attn_decode_kernel<KB, VB, D, NT, false>, (unsigned)blocks, DC_WARPS * 32, 0, st, 1, a, keys_per_split, n4));
    count_launches(1);
    if (a.splits > 1) {
        attn_small_merge_launch(a, n4, st);
        VARQ_CUDA_TRY(cudaGetLastError());
        count_launches(1);
    }
    return VARQ_OK;
}

}  // namespace

bool attn_decode_eligible(const AttnArgs& a, int kb, int vb) {
    (void)kb; (void)vb;
    return (a.D == 64 || a.D == 128) && a.kp.group == a.D && a.vp.group == a.D && a.k16 && a.v16 && a.ks_l == a.wk && a.vs_l == a.wv &&
           !a.kp.row_of_token && !a.vp.row_of_token && a.Lk * (a.kp.sr > a.vp.sr ? a.kp.sr : a.vp.sr) < (1ll << 31);
}

size_t attn_decode_workspace_bytes(int B, int H, int Lq, int Lk, int D) {
    int kps;
    const int splits = decode_splits(B, H, Lq, Lk, kps);
    if (splits <= 1 || Lq > 16) return 0;
    return (size_t)B * H * ((Lq + DC_QT - 1) / DC_QT) * splits * (DC_QT * (2 + D)) * sizeof(float);
}

int attn_decode_run(AttnArgs& a, int kb, int vb, void* ws, size_t ws_bytes, cudaStream_t st) {
    int kps = 0;
    a.splits = decode_splits(a.B, a.H, a.Lq, a.Lk, kps);
    if (a.splits > 1) {
        const size_t need = attn_decode_workspace_bytes(a.B, a.H, a.Lq, a.Lk, a.D);
        if (!ws || ws_bytes < need)
            return fail(VARQ_ERR_WORKSPACE, "varq_attn_fwd: workspace of %zu bytes needed, %zu given", need, ws_bytes);
        a.ws = reinterpret_cast<float*>(ws);
    }
#define GO(K_, V_)                                                                                                                     \
    if (kb == K_ && vb == V_) {                                                                                                        \
        if (a.D == 64) return a.Lq <= DC_QT ? launch_decode<K_, V_, 64, 1>(a, kps, st) : launch_decode<K_, V_, 64, 2>(a, kps, st);     \
        return a.Lq <= DC_QT ? launch_decode<K_, V_, 128, 1>(a, kps, st) : launch_decode<K_, V_, 128, 2>(a, kps, st);                  \
    }
    GO(8, 8) GO(8, 4) GO(8, 2) GO(4, 8) GO(4, 4) GO(4, 2) GO(2, 8) GO(2, 4) GO(2, 2)
#undef GO
    return fail(VARQ_ERR_ARG, "varq_attn_fwd: store bits must be 2, 4 or 8");
}

}  // namespace varq
