// Attention over the packed cache for the first scales of a schedule where the parameters vary along head_dim (per dim and step, or groups of
// fewer than 16): up to a few tens of queries over at most a few hundred tokens, everything in fp32.
//
// One CTA = one (sample, head) x 16 queries, four warps.  32 keys at a time go through shared memory: a thread keeps one word column of K and
// of V, so that the parameters of its head_dim values stay in registers while consecutive tokens belong to one step, and writes
// (code - zp) * scale, the reference's own fp32 values.  Scores: lane = key, warp = four queries (one 16-byte read of K and four broadcast reads of
// the queries for sixteen multiply-adds).  Softmax by warp reductions, weights through shared memory, output: a thread owns four head_dim
// values of two (four at head_dim 128) queries.
// Sums are kept in short chains (four partial sums of a score, even and odd keys of a chunk): the error stays below the general kernel's.
// Bound by latency: three dependent global round trips (step of a token, its parameters, the codes beside them) and three block barriers per
// 32 keys.  The general kernel (varq_attn_small.cu) stages 128 keys for four queries and reads the parameters of every (query, key) again.  us at B100
// H16 c64 int8, general / this, 1 / 4 / 9 / 16 queries over 1 / 5 / 14 / 30 tokens: 34 / 12, 36 / 13, 89 / 19, 130 / 26; B128 H30, K per dim int4:
// 61 / 24, 65 / 28, 187 / 39, 272 / 57.
// Where a word's codes share their parameters (ONE: groups of at least 4 to 16, one scale per key) a thread keeps one pair of them per column instead
// of one per code: 9 queries over 14 tokens, B64 H16 c64, int8 per head 13.4 -> 9.6, int4 per head 13.5 -> 8.6.
// CTAs per SM (23 KB of shared memory at c64, 37 KB at 128) against spilled registers, mean of 60 calls each (2 to 128 samples, 1 to 16 queries, 1 to 256
// tokens), relative: c64 per dim 7 (148 to 208 bytes spilled) 1, 6 (136 to 152) 1.02 int8 and 0.92 int4 but 1.13 to 1.29 where 7 make one wave less,
// 5 (44 to 120) 0.90 to 1.01 and up to 1.33; c128 per dim 5 (96 to 280) 1, 4 (0 to 80) 0.79 int4, 0.86 int8 but 1.08 where 5 make one wave less, 3 (none) 0.76
// and 0.88, up to 1.22; ONE at c64, 9 over 14 B64 int8: 8 (136 to 184) 12.4 us, 7 (8 to 80) 9.6 us, 6 11.6 us.
#include <cfloat>

#include "varq_attn.cuh"

namespace varq {

namespace {

constexpr int EA_THREADS = 128, EA_Q = 16, EA_KEYS = 32;

// Word column `w` of a thread: 32 / BITS consecutive head_dim values, parameters of the last step seen.  ONE: the word lies inside one group.
template <int BITS, bool ONE> struct EaColumn {
    static constexpr int N = 32 / BITS, NP = ONE ? 1 : N;
    float scale[NP], zp[NP];
    int row = -1;
    __device__ __forceinline__ void fetch(const ParamView& pv, long long base, int r, int d0) {
        if (r == row) return;
        row = r;
        const long long at = base + r * pv.sr;
        const float* sp = pv.scale + at + (long long)(d0 / pv.group) * pv.sg;
        const float* zq = pv.zp ? pv.zp + at + (long long)(d0 / pv.group) * pv.sg : nullptr;
        if constexpr (ONE) {
            scale[0] = __ldg(sp);
            zp[0] = zq ? __ldg(zq) : 0.f;
        } else if (pv.group == 1 && pv.sg == 1 && ((reinterpret_cast<uintptr_t>(sp) | reinterpret_cast<uintptr_t>(zq)) & 15u) == 0) {
#pragma unroll
            for (int j = 0; j < N; j += 4) {
                const float4 s = __ldg(reinterpret_cast<const float4*>(sp + j));
                const float4 z = zq ? __ldg(reinterpret_cast<const float4*>(zq + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
                scale[j] = s.x; scale[j + 1] = s.y; scale[j + 2] = s.z; scale[j + 3] = s.w;
                zp[j] = z.x; zp[j + 1] = z.y; zp[j + 2] = z.z; zp[j + 3] = z.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const long long i = at + (long long)((d0 + j) / pv.group) * pv.sg;
                scale[j] = __ldg(pv.scale + i);
                zp[j] = pv.zp ? __ldg(pv.zp + i) : 0.f;
            }
        }
    }
    // (code - zp) * scale; codes through the fp32 mantissa: 0x4B000000 | u is 2^23 + u
    __device__ __forceinline__ void store(float* dst, uint32_t word) const {
        constexpr uint32_t mask = BITS == 8 ? 0xffu : BITS == 4 ? 0xfu : 0x3u;
        constexpr float bias = 8388608.f + (float)(1 << (BITS - 1));
        const uint32_t x = word ^ (BITS == 8 ? 0x80808080u : BITS == 4 ? 0x88888888u : 0xAAAAAAAAu);
#pragma unroll
        for (int j = 0; j < N; j += 4) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = ((__uint_as_float(0x4B000000u | (x >> ((j + e) * BITS) & mask)) - bias) - zp[ONE ? 0 : j + e]) * scale[ONE ? 0 : j + e];
            *reinterpret_cast<float4*>(dst + j) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
};

template <int KB, int VB, int D, bool ONE>
__global__ void __launch_bounds__(EA_THREADS, D == 128 || (!ONE && (KB == 2 || VB == 2)) ? 4 : 7) attn_early_kernel(AttnArgs a) {
    constexpr int KW = D * KB / 32, VW = D * VB / 32;                          // words per row
    constexpr int KSTEP = EA_THREADS / KW, VSTEP = EA_THREADS / VW;            // keys per pass of the CTA (at least 4)
    constexpr int KIT = KSTEP < EA_KEYS ? EA_KEYS / KSTEP : 1, VIT = VSTEP < EA_KEYS ? EA_KEYS / VSTEP : 1;
    constexpr int KP = D + 4;                                                  // pitch of K: lanes on neighbouring keys read 16 bytes without conflicts
    constexpr int QPT = EA_Q * D / 4 / EA_THREADS;                             // queries per thread of the output
    __shared__ __align__(16) float sQ[EA_Q * D], sK[EA_KEYS * KP], sV[EA_KEYS * D], sP[EA_KEYS * EA_Q], sAlpha[EA_Q], sL[EA_Q];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int qt = (int)(blockIdx.x % (unsigned)a.n_qtiles), bh = (int)(blockIdx.x / (unsigned)a.n_qtiles), b = bh / a.H, h = bh - b * a.H;
    const int q0 = qt * EA_Q, nq = min(EA_Q, a.Lq - q0);
    const int32_t* kbase = a.kc + b * a.ks_b + h * a.ks_h;
    const int32_t* vbase = a.vc + b * a.vs_b + h * a.vs_h;
    const long long k_par = a.kp.index(b, 0, h, 0), v_par = a.vp.index(b, 0, h, 0);
    const int kw = tid % KW, kk0 = tid / KW, vw = tid % VW, vk0 = tid / VW;
    EaColumn<KB, ONE> kcol;
    EaColumn<VB, ONE> vcol;

    // ---- queries: a warp per query, scaled (and normalised) on the way in
    for (int q = warp; q < nq; q += EA_THREADS / 32) {
        const long long off = b * a.qs_b + (long long)(q0 + q) * a.qs_l + h * a.qs_h;
        float v[D / 32], ss = 0.f;
#pragma unroll
        for (int e = 0; e < D / 32; ++e) {
            v[e] = load_q_elem(a.q, a.q_dtype, off + lane + 32 * e);
            ss = fmaf(v[e], v[e], ss);
        }
        float mul = a.scale_log2;
        if (a.q_norm) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            mul *= (a.q_mul ? __ldg(a.q_mul + h) : 1.f) / fmaxf(sqrtf(ss), a.q_eps);
        }
#pragma unroll
        for (int e = 0; e < D / 32; ++e) sQ[q * D + lane + 32 * e] = v[e] * mul;
    }
    float m[4], l[4];                             // of the warp's four queries
#pragma unroll
    for (int u = 0; u < 4; ++u) { m[u] = -FLT_MAX; l[u] = 0.f; }
    const int d4 = tid % (D / 4) * 4, oq = tid / (D / 4) * QPT;
    float acc[QPT][4];
#pragma unroll
    for (int u = 0; u < QPT; ++u) { acc[u][0] = 0.f; acc[u][1] = 0.f; acc[u][2] = 0.f; acc[u][3] = 0.f; }

#pragma unroll 1
    for (int k0 = 0; k0 < a.Lk; k0 += EA_KEYS) {
        const int n = min(EA_KEYS, a.Lk - k0);
        uint32_t kwd[KIT], vwd[VIT];
        int krow[KIT], vrow[VIT];
#pragma unroll
        for (int i = 0; i < KIT; ++i) {
            const int key = kk0 + i * KSTEP;
            kwd[i] = 0u; krow[i] = 0;
            if (key < n) { kwd[i] = (uint32_t)__ldg(kbase + (long long)(k0 + key) * a.ks_l + kw); krow[i] = a.kp.row(k0 + key); }
        }
#pragma unroll
        for (int i = 0; i < VIT; ++i) {
            const int key = vk0 + i * VSTEP;
            vwd[i] = 0u; vrow[i] = 0;
            if (key < n) { vwd[i] = (uint32_t)__ldg(vbase + (long long)(k0 + key) * a.vs_l + vw); vrow[i] = a.vp.row(k0 + key); }
        }
        if (k0) __syncthreads();                  // the tiles of the chunk before are no longer read
#pragma unroll
        for (int i = 0; i < KIT; ++i) {
            const int key = kk0 + i * KSTEP;
            if (key < n) {
                kcol.fetch(a.kp, k_par, krow[i], kw * (32 / KB));
                kcol.store(sK + key * KP + kw * (32 / KB), kwd[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < VIT; ++i) {
            const int key = vk0 + i * VSTEP;
            if (key < n) {
                vcol.fetch(a.vp, v_par, vrow[i], vw * (32 / VB));
                vcol.store(sV + key * D + vw * (32 / VB), vwd[i]);
            }
        }
        __syncthreads();
        // ---- scores (log2 domain) and weights of four queries
        if (4 * warp < nq) {
            float s4[4][4] = {}, s[4];            // four partial sums: a shorter chain of roundings, and of latencies
            const float* kr = sK + min(lane, n - 1) * KP;
            const float* qr = sQ + 4 * warp * D;
#pragma unroll 8
            for (int d = 0; d < D; d += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 qv = *reinterpret_cast<const float4*>(qr + min(u, nq - 1 - 4 * warp) * D + d);
                    s4[u][0] = fmaf(kv.x, qv.x, s4[u][0]);
                    s4[u][1] = fmaf(kv.y, qv.y, s4[u][1]);
                    s4[u][2] = fmaf(kv.z, qv.z, s4[u][2]);
                    s4[u][3] = fmaf(kv.w, qv.w, s4[u][3]);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) s[u] = (s4[u][0] + s4[u][1]) + (s4[u][2] + s4[u][3]);
            float p[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float mx = lane < n ? s[u] : -FLT_MAX;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m[u], mx), al = exp2f(m[u] - m_new);
                m[u] = m_new;
                p[u] = lane < n ? exp2f(s[u] - m_new) : 0.f;
                float sum = p[u];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                l[u] = fmaf(l[u], al, sum);
                if (lane == 0) { sAlpha[4 * warp + u] = al; sL[4 * warp + u] = l[u]; }
            }
            *reinterpret_cast<float4*>(sP + lane * EA_Q + 4 * warp) = make_float4(p[0], p[1], p[2], p[3]);
        }
        __syncthreads();
        // ---- output
        if (oq < nq) {
            // even and odd keys of the chunk by themselves: short chains of roundings
            float part[2][QPT][4] = {};
            auto add_key = [&](int key, float (&into)[QPT][4]) {
                const float4 v = *reinterpret_cast<const float4*>(sV + key * D + d4);
                float p[QPT];
                if constexpr (QPT == 2) {
                    const float2 t = *reinterpret_cast<const float2*>(sP + key * EA_Q + oq);
                    p[0] = t.x; p[1] = t.y;
                } else {
                    const float4 t = *reinterpret_cast<const float4*>(sP + key * EA_Q + oq);
                    p[0] = t.x; p[1] = t.y; p[2] = t.z; p[3] = t.w;
                }
#pragma unroll
                for (int u = 0; u < QPT; ++u) {
                    into[u][0] = fmaf(p[u], v.x, into[u][0]);
                    into[u][1] = fmaf(p[u], v.y, into[u][1]);
                    into[u][2] = fmaf(p[u], v.z, into[u][2]);
                    into[u][3] = fmaf(p[u], v.w, into[u][3]);
                }
            };
            int key = 0;
#pragma unroll 2
            for (; key + 1 < n; key += 2) { add_key(key, part[0]); add_key(key + 1, part[1]); }
            if (key < n) add_key(key, part[0]);
#pragma unroll
            for (int u = 0; u < QPT; ++u) {
                const float al = sAlpha[oq + u];
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[u][e] = fmaf(acc[u][e], al, part[0][u][e] + part[1][u][e]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
        if (oq + u < nq) {
            const float inv = 1.f / sL[oq + u];
            const long long off = b * a.os_b + (long long)(q0 + oq + u) * a.os_l + h * a.os_h + d4;
#pragma unroll
            for (int e = 0; e < 4; ++e) store_o_elem(a.out, a.o_dtype, off + e, acc[u][e] * inv);
        }
    }
}

template <int KB, int VB, int D, bool ONE> int launch_early(const AttnArgs& a, cudaStream_t st) {
    VARQ_CUDA_TRY(launch_pdl(attn_early_kernel<KB, VB, D, ONE>, (unsigned)((long long)a.B * a.H * a.n_qtiles), EA_THREADS, 0, st, 1, a));
    count_launches(1);
    return VARQ_OK;
}

}  // namespace

bool attn_early_eligible(const AttnArgs& a) { return a.D == 64 || a.D == 128; }

int attn_early_run(AttnArgs& a, int kb, int vb, cudaStream_t st) {
    a.n_qtiles = (a.Lq + EA_Q - 1) / EA_Q;
    if ((long long)a.B * a.H * a.n_qtiles > 0x7fffffffLL) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: more than 2^31 thread blocks");
    const bool one = a.kp.group % (32 / kb) == 0 && a.vp.group % (32 / vb) == 0;
#define GO(K_, V_) if (kb == K_ && vb == V_) return one ? (a.D == 64 ? launch_early<K_, V_, 64, true>(a, st) : launch_early<K_, V_, 128, true>(a, st)) : a.D == 64 ? launch_early<K_, V_, 64, false>(a, st) : launch_early<K_, V_, 128, false>(a, st)
    GO(8, 8); GO(8, 4); GO(8, 2); GO(4, 8); GO(4, 4); GO(4, 2); GO(2, 8); GO(2, 4); GO(2, 2);
#undef GO
    return fail(VARQ_ERR_ARG, "varq_attn_fwd: store bits must be 2, 4 or 8");
}

}  // namespace varq
