// Quantize + pack of an appended step, K and V in one launch.
//
// Eight consecutive head_dim values per thread (one 16-byte load of 16-bit values, two of fp32) whatever the code width:
//   * rows     groups that keep (token, head) and are shared over the batch (per-token-per-head, with or without groups along
//              head_dim): a CTA holds every member of its groups in registers and reads the input once;
//   * planes   groups inside a plane of rows: one per head_dim element over batch and tokens of a head (per-dim), or one over batch, heads
//              and head_dim of a token (per-token).  Small planes: a cluster of CTAs owns one, every thread holds its rows in registers,
//              the statistics are folded through distributed shared memory -- one read, one launch.  Large planes: a statistics kernel
//              leaves column ranges per (plane, chunk of rows) in the workspace, the quantizing kernel folds the chunks of its plane and
//              reads the rows again, last chunks first (they are the likeliest to be in L2).
// Both optionally L2-normalise the rows on the way in (the K side of the attention hook), so a normalised K is never stored.
// Results are those of varq_quant.cu, bit for bit: fp32, true division, round-half-even, clamp after the round.
//
// What bounds them: short steps the launch and two dependent memory round trips, long ones HBM for fp32 and instruction issue for
// 16-bit inputs.  Hence per value: two multiply-adds that bracket the quotient, one comparison folded over eight values, one shift-add of
// the packing; only when a bracket disagrees (or a quotient is too large for the trick) the eight are redone with divisions.
#include <cooperative_groups.h>

#include "varq_quant.cuh"

namespace varq {
namespace {

namespace cg = cooperative_groups;

constexpr int AP_THREADS = 256;         // planes; rows: 256, or 512 when a group row of the batch needs them
constexpr int ROWS_MAX_THREADS = 512;

struct AppendJob {
    const void* x;
    long long xs_b, xs_l, xs_h;
    int32_t* codes;
    long long cs_b, cs_l, cs_h;
    float* scale;
    float* zp;                        // null: symmetric
    long long ps_r, ps_h, ps_g;       // strides of shared dims zero
    int32_t* row_of_token;            // per-step tables: entries of this step, or null
    int32_t* row_begin;               // [2]: first token of this step and of the next one
    int token0, row0;
    int kernel;                       // (dtype * 3 + log2(store bits) - 1) * 4 + symmetric * 2 + normalised
    int bits;
    float eps;
    float norm_eps;                   // normalised: x / max(||x||_2, norm_eps) is quantized
    int group;
    // rows kernel
    int bp, nv, ngr, h_fast;
    unsigned div_m, div_s;            // division by the inner extent as multiply-high + add + shift
    unsigned blocks;
    // planes
    long long xs_out, xs_in, cs_out, cs_in, ps_out;
    float* ranges;                    // large planes: workspace
    float* norms;
};
struct AppendArgs {
    AppendJob job[2];
    int n_jobs, B, L, H, D;
    // planes: `n_out` of them (heads, or tokens), each of B x n_in rows (tokens, or heads)
    int n_out, n_in, one_group;       // one_group: a plane is one group, else one per head_dim element
    int chunks, chunk_rows;           // large planes: row chunks
};

// ---- running range of a thread's values: one (rows) or one per value position (columns).  16-bit inputs are compared in packed pairs.
template <typename T, bool SYM> struct RangeAcc {               // fp32 values
    float hi[8], lo[8];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int j = 0; j < 8; ++j) { hi[j] = SYM ? 0.f : -INFINITY; lo[j] = INFINITY; }
    }
    __device__ __forceinline__ void add(const float (&v)[8]) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (SYM) hi[j] = fmaxf(hi[j], fabsf(v[j]));
            else { hi[j] = fmaxf(hi[j], v[j]); lo[j] = fminf(lo[j], v[j]); }
        }
    }
    __device__ __forceinline__ void add(const Vec8<float>& x) { float v[8]; x.get(v); add(v); }
    __device__ __forceinline__ void get(float (&h)[8], float (&l)[8]) const {
#pragma unroll
        for (int j = 0; j < 8; ++j) { h[j] = hi[j]; l[j] = lo[j]; }
    }
    __device__ __forceinline__ void fold(float& h, float& l) const {
        h = hi[0]; l = lo[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) { h = fmaxf(h, hi[j]); l = fminf(l, lo[j]); }
    }
};
template <typename T2, typename T, bool SYM> struct RangeAcc16 {
    T2 hi[4], lo[4];
    __device__ __forceinline__ static T2 bits(uint32_t u) { T2 t; memcpy(&t, &u, 4); return t; }
    __device__ __forceinline__ void add(const Vec8<T>& x) {
        const uint32_t w[4] = {x.r.x, x.r.y, x.r.z, x.r.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (SYM) hi[i] = __hmax2(hi[i], bits(w[i] & 0x7fff7fffu));
            else { hi[i] = __hmax2(hi[i], bits(w[i])); lo[i] = __hmin2(lo[i], bits(w[i])); }
        }
    }
    __device__ __forceinline__ void get(float (&h)[8], float (&l)[8]) const {
        Vec8<T> a, b;
        memcpy(&a.r, hi, 16);
        memcpy(&b.r, lo, 16);
        a.get(h);
        b.get(l);
    }
    __device__ __forceinline__ void fold(float& h, float& l) const {
        const T2 a = __hmax2(__hmax2(hi[0], hi[1]), __hmax2(hi[2], hi[3])), b = __hmin2(__hmin2(lo[0], lo[1]), __hmin2(lo[2], lo[3]));
        h = fmaxf(to_f32<T>(a.x), to_f32<T>(a.y)); l = fminf(to_f32<T>(b.x), to_f32<T>(b.y));
    }
};
template <bool SYM> struct RangeAcc<__nv_bfloat16, SYM> : RangeAcc16<__nv_bfloat162, __nv_bfloat16, SYM> {
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < 4; ++i) { this->hi[i] = this->bits(SYM ? 0u : 0xff80ff80u); this->lo[i] = this->bits(0x7f807f80u); }
    }
};
template <bool SYM> struct RangeAcc<__half, SYM> : RangeAcc16<__half2, __half, SYM> {
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int i = 0; i < 4; ++i) { this->hi[i] = this->bits(SYM ? 0u : 0xfc00fc00u); this->lo[i] = this->bits(0x7c007c00u); }
    }
};
// normalised rows are compared after the division, in fp32
template <typename T, bool SYM, bool NORM> struct PickAcc { using type = RangeAcc<T, SYM>; };
template <typename T, bool SYM> struct PickAcc<T, SYM, true> { using type = RangeAcc<float, SYM>; };

// ---- quantization of eight values.  RN(x / scale) lies strictly between x * rcp_lo and x * rcp_hi (rcp = RN(1 / scale), rcp_lo / hi =
// rcp (1 -/+ 2^-21)) and rint is monotonic: when both ends round to one integer, that is the code.  Adding 1.5 * 2^23 + zero-point
// rounds, adds the zero-point and leaves the two's-complement code in the low mantissa bits (an exact tie rounds by another parity than
// the quotient's own, but then the ends differ).  A normalised value enters as x * RN(1 / length), within 1.5 * 2^-23 of the rounded
// quotient x / length: with the other roundings still inside the bracket.
struct QPar { float lo, hi, magic; };
template <bool SYM> __device__ __forceinline__ QPar make_qpar(float scale, float zp, float mx, float mn) {
    const float rcp = __frcp_rn(scale);
    QPar q = {rcp * (1.0f - 4.76837158e-7f), rcp * (1.0f + 4.76837158e-7f), SYM ? Q_MAGIC : Q_MAGIC + zp};
    // an offset group whose quotients leave the trick's range is quantized by division: no bracket equals NaN
    if (!SYM && !(fmaxf(fabsf(mx), fabsf(mn)) * q.hi < 2097152.0f && fabsf(zp) < 2097152.0f)) q.lo = __int_as_float(0x7fc00000);
    return q;
}
// code of one value by division.  Out of line: the callers hold many values in registers and rarely come here.
__device__ __noinline__ float exact_code(float x, float length, float scale, float zp, float q_min, float q_max) {
    if (length > 0.f) x = __fdiv_rn(x, length);
    return fminf(fmaxf(__fadd_rn(rintf(__fdiv_rn(x, scale)), zp), q_min), q_max) + Q_MAGIC;
}
// Whether a code of an asymmetric group can leave its range before the clamp: codes grow with x, so the ends of the range decide (they
// only do when rounding takes zero-point and quotient apart).  Symmetric codes cannot: |x| <= amax.
__device__ __forceinline__ bool needs_clamp(float mx, float mn, float scale, float zp, int bits) {
    return !(rintf(__fdiv_rn(mx, scale)) + zp <= (float)((1 << (bits - 1)) - 1) && rintf(__fdiv_rn(mn, scale)) + zp >= -(float)(1 << (bits - 1)));
}
// y[8] (1.5 * 2^23 + code) -> packed fields: 8 bits two words, 4 bits one, 2 bits half a word.  The bit patterns are 0x4B400000 + code: a
// chain of shift-adds sums code << (bits * j) and a known constant, which is replaced by the offset that makes all fields
// non-negative, and the offset's bits are flipped back to two's complement.
template <int SB, int N> __device__ __forceinline__ uint32_t pack_fields(const float* y) {
    uint32_t acc = __float_as_uint(y[N - 1]);
    uint32_t ones = 1u;
#pragma unroll
    for (int j = N - 2; j >= 0; --j) { acc = (acc << SB) + __float_as_uint(y[j]); ones = (ones << SB) + 1u; }
    const uint32_t offset = ones * (1u << (SB - 1));
    return (acc + (offset - ones * 0x4B400000u)) ^ offset;
}
template <int SB> __device__ __forceinline__ uint2 pack8(const float (&y)[8]) {
    if constexpr (SB == 8) return make_uint2(pack_fields<8, 4>(y), pack_fields<8, 4>(y + 4));
    else return make_uint2(pack_fields<SB, 8>(y), 0u);
}
// Where the brackets disagree the quotient lies next to t = k + 1/2, k and k + 1 the two ends, and no division is needed: the residual
// r = x - t * scale is exact (t has few bits and the difference cancels), so its sign tells on which side of t the exact quotient lies,
// and the rounded quotient is t itself iff |r| <= scale * ulp(t) / 2; then the even end is the code.  (Below 1/2 floats are twice as
// dense, but both outcomes give 0 there.)  16-bit inputs of few distinct values hit such ties often.
__device__ __forceinline__ float settle(float x, float lo, float hi, float magic, float scale) {
    const float ka = fmaf(x, lo, magic) - magic, kb = fmaf(x, hi, magic) - magic;
    const float t = 0.5f * (ka + kb);
    const float r = fmaf(-t, scale, x), half_ulp = __uint_as_float(__float_as_uint(t) & 0x7f800000u) * 5.9604645e-8f;
    float k = (t + Q_MAGIC) - Q_MAGIC;                  // the ends agree: that integer; a tie: the even end
    if (ka != kb && fabsf(r) > scale * half_ulp) k = r > 0.f ? fmaxf(ka, kb) : fminf(ka, kb);
    return magic + k;
}
// PER_VALUE: parameters per value position (columns), else one set
template <int SB, bool SYM, bool NORM, bool PER_VALUE>
__device__ __forceinline__ uint2 quantize8(const float (&x)[8], float length, const float* lo, const float* hi, const float* magic, const float* scale,
                                           float q_min, float q_max, bool clamp) {
    float y[8];
    bool bad = false;
    const float rlen = NORM ? __frcp_rn(length) : 1.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int z = PER_VALUE ? j : 0;
        const float v = NORM ? x[j] * rlen : x[j];
        y[j] = fmaf(v, hi[z], magic[z]);
        bad = bad | (y[j] != fmaf(v, lo[z], magic[z]));
    }
    if (bad) {
        bool divide = NORM;
        if (!NORM && !SYM) {
#pragma unroll
            for (int z = 0; z < (PER_VALUE ? 8 : 1); ++z) divide = divide | (lo[z] != lo[z]);
        }
        if (divide) {
            float t[8];                                // indexed at run time: local memory, touched on this path only
#pragma unroll
            for (int j = 0; j < 8; ++j) t[j] = x[j];
#pragma unroll 1
            for (int j = 0; j < 8; ++j) {
                float m = magic[0];
                if (PER_VALUE) {
#pragma unroll
                    for (int z = 1; z < 8; ++z) m = j == z ? magic[z] : m;
                }
                t[j] = exact_code(t[j], NORM ? length : 0.f, scale[PER_VALUE ? j : 0], SYM ? 0.f : m - Q_MAGIC, q_min, q_max);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) y[j] = t[j];
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int z = PER_VALUE ? j : 0;
                y[j] = settle(x[j], lo[z], hi[z], magic[z], scale[z]);
            }
        }
    }
    if (!SYM && clamp) {
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j] = fminf(fmaxf(y[j], Q_MAGIC + q_min), Q_MAGIC + q_max);
    }
    return pack8<SB>(y);
}
// store the fields of thread w of a row (all lanes of the warp take part: 2-bit codes of two neighbours share a word)
template <int SB> __device__ __forceinline__ void store8(int32_t* row, int w, const uint2& p, bool ok) {
    if constexpr (SB == 8) { if (ok) *reinterpret_cast<uint2*>(row + 2 * w) = p; }
    else if constexpr (SB == 4) { if (ok) row[w] = (int32_t)p.x; }
    else {
        const uint32_t up = __shfl_down_sync(0xffffffffu, p.x, 1);
        if (ok && !(w & 1)) row[w >> 1] = (int32_t)(p.x | (up << 16));
    }
}

// =====================================================================================
// rows: one (token, head) row of every sample of the batch per D / 8 x bp threads
// =====================================================================================
constexpr int ROWS_NV = 4;              // samples per thread
// (token, head) of group row r
struct RowAt { long long l, h; };
__device__ __forceinline__ RowAt row_at(const AppendArgs& a, const AppendJob& jb, unsigned r) {
    const unsigned q = (unsigned)((__umulhi(r, jb.div_m) + (unsigned long long)r) >> jb.div_s), rem = r - q * (unsigned)(jb.h_fast ? a.H : a.L);
    return jb.h_fast ? RowAt{(long long)q, (long long)rem} : RowAt{(long long)rem, (long long)q};
}
struct RowsShared { uint32_t hi[ROWS_MAX_THREADS], lo[ROWS_MAX_THREADS]; float4 par[ROWS_MAX_THREADS]; };     // per group of the CTA
template <typename T, int SB, bool SYM, bool NORM>
__device__ __forceinline__ void rows_body(const AppendArgs& a, const AppendJob& jb, unsigned block, RowsShared& sh) {
    constexpr int NV = ROWS_NV;
    const int tid = threadIdx.x, tpr = a.D >> 3, lpg = jb.group >> 3, bsh = __ffs(tpr) - 1, psh = __ffs(jb.bp) - 1;
    const int w = tid & (tpr - 1), bl = (tid >> bsh) & (jb.bp - 1), g_local = tid >> (bsh + psh);
    const int gsh = bsh - (__ffs(lpg) - 1), n_groups = jb.ngr << gsh;      // groups per row (log2), of the CTA
    const unsigned n_gr = (unsigned)a.L * (unsigned)a.H, gr_ = block * (unsigned)jb.ngr + g_local;
    const bool in = gr_ < n_gr;
    // threads past the last group repeat it and store nothing
    const RowAt at = row_at(a, jb, in ? gr_ : n_gr - 1);
    const T* xp = reinterpret_cast<const T*>(jb.x) + at.l * jb.xs_l + at.h * jb.xs_h + w * 8;
    Vec8<T> x[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (k < jb.nv) x[k].load(xp + (long long)min(bl + k * jb.bp, a.B - 1) * jb.xs_b);      // past the batch: the last sample again
    const bool across_warps = tpr * jb.bp > 32;
    if (across_warps) {
        if (tid < n_groups) { sh.hi[tid] = 0u; sh.lo[tid] = 0u; }
        __syncthreads();
    }
    typename PickAcc<T, SYM, NORM>::type acc;
    acc.init();
    float len[NV];                                        // row lengths, when rows are normalised
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        len[k] = 0.f;
        if (k < jb.nv) {
            if constexpr (NORM) {
                float v[8];
                x[k].get(v);
                len[k] = row_length(x[k], tpr, w, jb.norm_eps);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __fdiv_rn(v[j], len[k]);
                acc.add(v);
            } else {
                acc.add(x[k]);
            }
        }
    }
    float hi, lo;
    acc.fold(hi, lo);
    for (int m = 1; m < lpg; m <<= 1) {
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, m));
        if (!SYM) lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, m));
    }
    for (int m = tpr; m < 32 && m < tpr * jb.bp; m <<= 1) {          // batch lanes of this warp
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, m));
        if (!SYM) lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, m));
    }
    const int g = (g_local << gsh) + (w >> (bsh - gsh));             // this thread's group inside the CTA
    if ((w & (lpg - 1)) == 0 && (across_warps ? (tid & 31) < tpr : bl == 0)) {
        if (across_warps) {
            atomicMax(&sh.hi[g], f2ord(hi));
            if (!SYM) atomicMax(&sh.lo[g], ~f2ord(lo));
        } else {
            sh.hi[g] = f2ord(hi);
            sh.lo[g] = SYM ? 0u : ~f2ord(lo);
        }
    }
    __syncthreads();
    // the divisions behind scale, zero-point and reciprocal once per group, by the first warps (done by every thread they were
    // half of the kernel's instructions)
    if (tid < n_groups) {
        const Range rg = {sh.hi[tid], sh.lo[tid]};
        float scale, zp;
        params_from_range(rg, jb.bits, SYM, jb.eps, scale, zp);
        const QPar q = make_qpar<SYM>(scale, zp, ord2f(rg.hi), ord2f(~rg.lo));
        // the sign of the scale says that the codes need their clamp
        sh.par[tid] = make_float4(q.lo, q.hi, q.magic, !SYM && needs_clamp(ord2f(rg.hi), ord2f(~rg.lo), scale, zp, jb.bits) ? -scale : scale);
        const unsigned r = block * (unsigned)jb.ngr + (unsigned)(tid >> gsh);
        if (r < n_gr) {
            const RowAt o = row_at(a, jb, r);
            const long long pi = o.l * jb.ps_r + o.h * jb.ps_h + (long long)(tid & ((1 << gsh) - 1)) * jb.ps_g;
            jb.scale[pi] = scale;
            if (!SYM) jb.zp[pi] = zp;
        }
    }
    __syncthreads();
    float4 q = sh.par[g];
    const bool clamp = !SYM && q.w < 0.f;
    q.w = fabsf(q.w);
    const float q_min = -(float)(1 << (jb.bits - 1)), q_max = (float)((1 << (jb.bits - 1)) - 1);
    int32_t* cp = jb.codes + at.l * jb.cs_l + at.h * jb.cs_h + (long long)bl * jb.cs_b;
    const long long c_step = (long long)jb.bp * jb.cs_b;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        if (k >= jb.nv) break;
        float v[8];
        x[k].get(v);
        const uint2 c = quantize8<SB, SYM, NORM, false>(v, NORM ? len[k] : 0.f, &q.x, &q.y, &q.z, &q.w, q_min, q_max, clamp);
        store8<SB>(cp, w, c, in && bl + k * jb.bp < a.B);
        cp += c_step;
    }
}

#define VARQ_AP_CASE4(BASE, T_, SB_)                                                                                   \
    case BASE: VARQ_BODY(T_, SB_, false, false); break;     case BASE + 1: VARQ_BODY(T_, SB_, false, true); break;     \
    case BASE + 2: VARQ_BODY(T_, SB_, true, false); break;  case BASE + 3: VARQ_BODY(T_, SB_, true, true); break;
#define VARQ_AP_SWITCH                                                                                                 \
    switch (jb.kernel) {                                                                                               \
        VARQ_AP_CASE4(0, float, 2) VARQ_AP_CASE4(4, float, 4) VARQ_AP_CASE4(8, float, 8)                               \
        VARQ_AP_CASE4(12, __half, 2) VARQ_AP_CASE4(16, __half, 4) VARQ_AP_CASE4(20, __half, 8)                         \
        VARQ_AP_CASE4(24, __nv_bfloat16, 2) VARQ_AP_CASE4(28, __nv_bfloat16, 4) VARQ_AP_CASE4(32, __nv_bfloat16, 8)    \
    }

template <int THREADS>
__global__ void __launch_bounds__(THREADS, 768 / THREADS) append_rows_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ RowsShared sh;
    pdl_trigger();
    pdl_wait();
    const int ji = a.n_jobs > 1 && blockIdx.x >= a.job[0].blocks ? 1 : 0;
    const AppendJob& jb = a.job[ji];
    const unsigned block = blockIdx.x - (ji ? a.job[0].blocks : 0u);
#define VARQ_BODY(T_, SB_, SYM_, NORM_) rows_body<T_, SB_, SYM_, NORM_>(a, jb, block, sh)
    VARQ_AP_SWITCH
#undef VARQ_BODY
}

// =====================================================================================
// planes: thread = eight head_dim columns, rows (sample, inner index) of a plane strided over CTAs
// =====================================================================================
// ranges of a thread's columns -> the CTA's, s_cta [2][D] (s_red: scratch of 16 D floats)
template <bool SYM>
__device__ __forceinline__ void fold_columns(float (&hi)[8], float (&lo)[8], int tpr, int w, int D, float* s_red, float* s_cta) {
    for (int m = tpr; m < 32; m <<= 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            hi[j] = fmaxf(hi[j], __shfl_xor_sync(0xffffffffu, hi[j], m));
            if (!SYM) lo[j] = fminf(lo[j], __shfl_xor_sync(0xffffffffu, lo[j], m));
        }
    }
    const int tid = threadIdx.x, warp = tid >> 5;
    if ((tid & 31) < tpr) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { s_red[(warp * 2) * D + w * 8 + j] = hi[j]; s_red[(warp * 2 + 1) * D + w * 8 + j] = lo[j]; }
    }
    __syncthreads();
    if (tid < D) {
        float a = s_red[tid], b = s_red[D + tid];
#pragma unroll
        for (int q = 1; q < AP_THREADS / 32; ++q) { a = fmaxf(a, s_red[q * 2 * D + tid]); b = fminf(b, s_red[(q * 2 + 1) * D + tid]); }
        s_cta[tid] = a; s_cta[D + tid] = b;
    }
}
// scale / zero-point and quantizer constants of column `d` from its range; s_par [5][D]: lo, hi, magic, scale, clamp
template <bool SYM>
__device__ __forceinline__ void column_params(const AppendJob& jb, int D, int plane, int d, float mx, float mn, bool write, float* s_par) {
    Range rg;
    rg.hi = f2ord(mx); rg.lo = SYM ? 0u : ~f2ord(mn);
    float scale, zp;
    params_from_range(rg, jb.bits, SYM, jb.eps, scale, zp);
    const QPar q = make_qpar<SYM>(scale, zp, mx, mn);
    s_par[d] = q.lo; s_par[D + d] = q.hi; s_par[2 * D + d] = q.magic; s_par[3 * D + d] = scale;
    if (!SYM) s_par[4 * D + d] = needs_clamp(mx, mn, scale, zp, jb.bits) ? 1.f : 0.f;
    if (write) {
        const long long pi = (long long)plane * jb.ps_out + (long long)d * jb.ps_g;
        jb.scale[pi] = scale;
        if (!SYM) jb.zp[pi] = zp;
    }
}
// one range for the whole plane: threads 0 .. D - 1 (whole warps) fold theirs; s_red: scratch.  Called by the whole CTA.
__device__ __forceinline__ void fold_plane(int D, float& mx, float& mn, float* s_red) {
    const int tid = threadIdx.x;
    __syncthreads();
    if (tid < D) {
        for (int m = 16; m; m >>= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, m));
        }
        if ((tid & 31) == 0) { s_red[tid >> 5] = mx; s_red[8 + (tid >> 5)] = mn; }
    }
    __syncthreads();
    if (tid < D)
        for (int q = 0; q < D / 32; ++q) { mx = fmaxf(mx, s_red[q]); mn = fminf(mn, s_red[8 + q]); }
}
template <bool SYM> struct ColQuant {
    float lo[8], hi[8], m[8], q_min, q_max;
    bool clamp;
    const float* scale;
    __device__ __forceinline__ void init(const AppendJob& jb, int D, int w, const float* s_par) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { lo[j] = s_par[w * 8 + j]; hi[j] = s_par[D + w * 8 + j]; m[j] = SYM ? Q_MAGIC : s_par[2 * D + w * 8 + j]; }
        q_min = -(float)(1 << (jb.bits - 1)); q_max = (float)((1 << (jb.bits - 1)) - 1);
        scale = s_par + 3 * D + w * 8;
        clamp = false;
        if (!SYM)
            for (int j = 0; j < 8; ++j) clamp = clamp | (scale[D + j] != 0.f);
    }
    template <int SB, bool NORM> __device__ __forceinline__ uint2 codes(const float (&v)[8], float length) const {
        return quantize8<SB, SYM, NORM, true>(v, length, lo, hi, m, scale, q_min, q_max, clamp);
    }
};
// (sample, inner index) of a thread's rows first, first + step, ...: one division at the start, then constant steps with a carry
struct RowWalk {
    unsigned b, l, L, step_b, step_l;
    __device__ __forceinline__ void init(unsigned r, unsigned L_, unsigned step) {
        L = L_; b = r / L; l = r - b * L; step_b = step / L; step_l = step - step_b * L;
    }
    __device__ __forceinline__ void next() { b += step_b; l += step_l; if (l >= L) { l -= L; ++b; } }
};
// the step's entries of the token -> row and row -> first token tables
__device__ __forceinline__ void write_step_rows(const AppendJob& jb, int L, int first, int stride) {
    if (!jb.row_of_token) return;
    for (int i = first; i < L; i += stride) jb.row_of_token[i] = jb.row0;
    if (first == 0) { jb.row_begin[0] = jb.token0; jb.row_begin[1] = jb.token0 + L; }
}

// ---- small planes: a cluster owns one, every thread holds all of its rows; statistics are folded through distributed shared memory
constexpr int HELD_ROWS = 4;
template <typename T, int SB, bool SYM, bool NORM>
__device__ __forceinline__ void cluster_body(const AppendArgs& a, const AppendJob& jb, int h, float* s_red, float* s_par) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), csize = (int)cl.num_blocks();
    const int tid = threadIdx.x, D = a.D, tpr = D >> 3, w = tid & (tpr - 1), rl = tid / tpr, nrl = AP_THREADS / tpr;
    const unsigned R = (unsigned)a.B * (unsigned)a.n_in, step = (unsigned)(nrl * csize), first = (unsigned)(rank * nrl + rl);
    const T* xh = reinterpret_cast<const T*>(jb.x) + (long long)h * jb.xs_out + w * 8;
    int32_t* ch = jb.codes + (long long)h * jb.cs_out;
    Vec8<T> x[HELD_ROWS];
    float len[HELD_ROWS];
    RowWalk k;
    k.init(first, (unsigned)a.n_in, step);
#pragma unroll
    for (int u = 0; u < HELD_ROWS; ++u) {
        if (k.b < (unsigned)a.B) x[u].load(xh + (long long)k.b * jb.xs_b + (long long)k.l * jb.xs_in);
        else x[u] = Vec8<T>{};
        k.next();
    }
    typename PickAcc<T, SYM, NORM>::type acc;
    acc.init();
#pragma unroll
    for (int u = 0; u < HELD_ROWS; ++u) {
        len[u] = 0.f;
        if ((unsigned)u * step < R) {
            const bool mine = first + (unsigned)u * step < R;
            if constexpr (NORM) {
                float v[8];
                x[u].get(v);
                len[u] = row_length(x[u], tpr, w, jb.norm_eps);
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __fdiv_rn(v[j], len[u]);
                if (mine) acc.add(v);
            } else if (mine) acc.add(x[u]);
        }
    }
    float hi[8], lo[8];
    acc.get(hi, lo);
    float* s_cta = s_red + 16 * D;                // [2][D]: this CTA's columns
    fold_columns<SYM>(hi, lo, tpr, w, D, s_red, s_cta);
    if (csize > 1) cl.sync(); else __syncthreads();
    float mx = 0.f, mn = 0.f;
    if (tid < D) {
        mx = s_cta[tid]; mn = s_cta[D + tid];
        for (int q = 1; q < csize; ++q) {
            const float* o = cl.map_shared_rank(s_cta, (rank + q) % csize);
            mx = fmaxf(mx, o[tid]); mn = fminf(mn, o[D + tid]);
        }
    }
    if (a.one_group) fold_plane(D, mx, mn, s_red);
    if (tid < D) column_params<SYM>(jb, D, h, tid, mx, mn, rank == 0 && (tid == 0 || !a.one_group), s_par);
    if (csize > 1) cl.sync(); else __syncthreads();      // parameters in place; nobody reads a neighbour's shared memory any more
    ColQuant<SYM> q;
    q.init(jb, D, w, s_par);
    k.init(first, (unsigned)a.n_in, step);
#pragma unroll
    for (int u = 0; u < HELD_ROWS; ++u) {
        if ((unsigned)u * step >= R) break;
        float v[8];
        x[u].get(v);
        const uint2 c = q.template codes<SB, NORM>(v, len[u]);
        store8<SB>(ch + (long long)k.b * jb.cs_b + (long long)k.l * jb.cs_in, w, c, k.b < (unsigned)a.B);
        k.next();
    }
}
__global__ void __launch_bounds__(AP_THREADS, 2) append_plane_cluster_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ float s_red[18 * 128], s_par[5 * 128];
    pdl_trigger();
    pdl_wait();
    const int csize = (int)cg::this_cluster().num_blocks();
    const int cluster = blockIdx.x / csize, ji = cluster / a.n_out, h = cluster - ji * a.n_out;
    const AppendJob& jb = a.job[ji];
    write_step_rows(jb, a.L, (h * csize + (int)(blockIdx.x % csize)) * AP_THREADS + threadIdx.x, a.n_out * csize * AP_THREADS);
#define VARQ_BODY(T_, SB_, SYM_, NORM_) cluster_body<T_, SB_, SYM_, NORM_>(a, jb, h, s_red, s_par)
    VARQ_AP_SWITCH
#undef VARQ_BODY
}

// ---- large planes: statistics of (plane, chunk of rows) to the workspace, then quantization.  CTAs of neighbouring planes run together
// (the plane index is fastest), so their pieces of a token's row come from the same DRAM pages.  Workspace: per job
// [planes][chunks][2][D] column ranges, then (normalised rows) [rows][planes] row lengths.
constexpr int COL_UNROLL = 4;        // rows in flight per thread
template <typename T, int SB, bool SYM, bool NORM>
__device__ __forceinline__ void plane_stats_body(const AppendArgs& a, const AppendJob& jb, int h, int chunk, float* s_red) {
    const int tid = threadIdx.x, D = a.D, tpr = D >> 3, w = tid & (tpr - 1), rl = tid / tpr, nrl = AP_THREADS / tpr;
    const unsigned R = (unsigned)a.B * (unsigned)a.n_in, r0 = (unsigned)chunk * (unsigned)a.chunk_rows, r1 = min(R, r0 + (unsigned)a.chunk_rows);
    const T* xh = reinterpret_cast<const T*>(jb.x) + (long long)h * jb.xs_out + w * 8;
    RowWalk k;
    k.init(r0 + rl, (unsigned)a.n_in, (unsigned)nrl);
    typename PickAcc<T, SYM, NORM>::type acc;
    acc.init();
    for (unsigned rr = r0; rr < r1; rr += COL_UNROLL * nrl) {            // uniform trip count: the rows' lanes shuffle together
        Vec8<T> x[COL_UNROLL];
#pragma unroll
        for (int u = 0; u < COL_UNROLL; ++u) {
            if (rr + u * nrl + rl < r1) x[u].load(xh + (long long)k.b * jb.xs_b + (long long)k.l * jb.xs_in);
            else x[u] = Vec8<T>{};
            k.next();
        }
#pragma unroll
        for (int u = 0; u < COL_UNROLL; ++u) {
            const unsigned r = rr + u * nrl + rl;
            if constexpr (NORM) {
                float v[8];
                x[u].get(v);
                const float d = row_length(x[u], tpr, w, jb.norm_eps);
                if (w == 0 && r < r1) jb.norms[(size_t)r * a.n_out + h] = d;
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __fdiv_rn(v[j], d);
                if (r < r1) acc.add(v);
            } else if (r < r1) acc.add(x[u]);
        }
    }
    float hi[8], lo[8];
    acc.get(hi, lo);
    float* s_cta = s_red + 16 * D;
    fold_columns<SYM>(hi, lo, tpr, w, D, s_red, s_cta);
    if (tid < D) {        // (written by this very thread)
        float* o = jb.ranges + ((size_t)h * a.chunks + chunk) * 2 * D;
        o[tid] = s_cta[tid]; o[D + tid] = s_cta[D + tid];
    }
}
template <typename T, int SB, bool SYM, bool NORM>
__device__ __forceinline__ void plane_apply_body(const AppendArgs& a, const AppendJob& jb, int h, int chunk, float* s_red, float* s_par) {
    const int tid = threadIdx.x, D = a.D, tpr = D >> 3, w = tid & (tpr - 1), rl = tid / tpr, nrl = AP_THREADS / tpr;
    {   // ranges of the plane's chunks, AP_THREADS / D of them at a time
        const int d = tid & (D - 1), part = tid / D, parts = AP_THREADS / D;
        const float* o = jb.ranges + (size_t)h * a.chunks * 2 * D + d;
        float mx = SYM ? 0.f : -INFINITY, mn = INFINITY;
#pragma unroll 4
        for (int q = part; q < a.chunks; q += parts) { mx = fmaxf(mx, __ldcg(o + (size_t)q * 2 * D)); mn = fminf(mn, __ldcg(o + (size_t)q * 2 * D + D)); }
        s_red[tid] = mx; s_red[AP_THREADS + tid] = mn;
        __syncthreads();
        if (tid < D)
            for (int q = 1; q < parts; ++q) { mx = fmaxf(mx, s_red[q * D + tid]); mn = fminf(mn, s_red[AP_THREADS + q * D + tid]); }
        if (a.one_group) fold_plane(D, mx, mn, s_red);
        if (tid < D) column_params<SYM>(jb, D, h, tid, mx, mn, chunk == 0 && (tid == 0 || !a.one_group), s_par);
        __syncthreads();
    }
    const unsigned R = (unsigned)a.B * (unsigned)a.n_in, r0 = (unsigned)chunk * (unsigned)a.chunk_rows, r1 = min(R, r0 + (unsigned)a.chunk_rows);
    const T* xh = reinterpret_cast<const T*>(jb.x) + (long long)h * jb.xs_out + w * 8;
    int32_t* ch = jb.codes + (long long)h * jb.cs_out;
    ColQuant<SYM> q;
    q.init(jb, D, w, s_par);
    RowWalk k, kc;
    k.init(r0 + rl, (unsigned)a.n_in, (unsigned)nrl);
    kc = k;
    for (unsigned rr = r0; rr < r1; rr += COL_UNROLL * nrl) {
        Vec8<T> x[COL_UNROLL];
        float d[COL_UNROLL];
#pragma unroll
        for (int u = 0; u < COL_UNROLL; ++u) {
            const unsigned r = rr + u * nrl + rl;
            d[u] = NORM ? 1.f : 0.f;
            if (r < r1) {
                x[u].load(xh + (long long)k.b * jb.xs_b + (long long)k.l * jb.xs_in);
                if (NORM) d[u] = jb.norms[(size_t)r * a.n_out + h];
            } else x[u] = Vec8<T>{};
            k.next();
        }
#pragma unroll
        for (int u = 0; u < COL_UNROLL; ++u) {
            float v[8];
            x[u].get(v);
            const uint2 c = q.template codes<SB, NORM>(v, d[u]);
            store8<SB>(ch + (long long)kc.b * jb.cs_b + (long long)kc.l * jb.cs_in, w, c, rr + u * nrl + rl < r1);
            kc.next();
        }
    }
}
__global__ void __launch_bounds__(AP_THREADS, 3) append_plane_stats_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ float s_red[18 * 128];
    pdl_trigger();
    pdl_wait();
    const unsigned t = blockIdx.x / (unsigned)a.n_out;
    const int h = blockIdx.x - t * a.n_out, ji = t / a.chunks, chunk = t - ji * a.chunks;
    const AppendJob& jb = a.job[ji];
#define VARQ_BODY(T_, SB_, SYM_, NORM_) plane_stats_body<T_, SB_, SYM_, NORM_>(a, jb, h, chunk, s_red)
    VARQ_AP_SWITCH
#undef VARQ_BODY
}
__global__ void __launch_bounds__(AP_THREADS, 2) append_plane_apply_kernel(const __grid_constant__ AppendArgs a) {
    __shared__ float s_red[2 * AP_THREADS], s_par[5 * 128];
    pdl_trigger();
    pdl_wait();
    const unsigned t = blockIdx.x / (unsigned)a.n_out;
    // chunks in reverse order: the ones read last by the statistics kernel are the likeliest to be in L2
    const int h = blockIdx.x - t * a.n_out, ji = a.n_jobs - 1 - (int)(t / a.chunks), chunk = a.chunks - 1 - (int)(t % a.chunks);
    const AppendJob& jb = a.job[ji];
    write_step_rows(jb, a.L, (chunk * a.n_out + h) * AP_THREADS + threadIdx.x, a.n_out * a.chunks * AP_THREADS);
#define VARQ_BODY(T_, SB_, SYM_, NORM_) plane_apply_body<T_, SB_, SYM_, NORM_>(a, jb, h, chunk, s_red, s_par)
    VARQ_AP_SWITCH
#undef VARQ_BODY
}

bool pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

// 2: groups of one head_dim element over batch and tokens, 3: groups of a token over batch, heads and head_dim, 0: neither
int plane_kind(const varq_qparams_t& p, int D) {
    if (!p.share_b || D < 32) return 0;
    if (p.share_l && !p.share_h && p.group == 1) return 2;
    if (!p.share_l && p.share_h && p.group == D) return 3;
    return 0;
}
// 1: rows kernel, 2: planes of a head, 3: planes of a token, 0: none of them
int plan_job(AppendJob& jb, const varq_append_job_t& in, int B, int L, int H, int D, float norm_eps) {
    const int es = dtype_size(in.x.dtype);
    auto al = [&](long long s) { return ((s * es) & 15) == 0; };
    if (D % 8 || !pow2(D / 8) || D > 128) return 0;
    if (norm_eps >= 0.f && D != 64 && D != 128) return 0;
    if ((reinterpret_cast<uintptr_t>(in.x.ptr) & 15) || !al(in.x.stride_b) || !al(in.x.stride_l) || !al(in.x.stride_h)) return 0;
    // 8-bit codes of a thread are two words, stored together
    if (in.store_bits == 8 && ((reinterpret_cast<uintptr_t>(in.codes.ptr) & 7) || ((in.codes.stride_b | in.codes.stride_l | in.codes.stride_h) & 1))) return 0;
    if (in.store_bits == 2 && D % 16) return 0;
    if (!in.p.share_b || (long long)B * L >= 0x7fffffffLL || (long long)L * H >= 0x7fffffffLL || (long long)B * H >= 0x7fffffffLL) return 0;
    jb.x = in.x.ptr; jb.xs_b = in.x.stride_b; jb.xs_l = in.x.stride_l; jb.xs_h = in.x.stride_h;
    jb.codes = (int32_t*)in.codes.ptr; jb.cs_b = in.codes.stride_b; jb.cs_l = in.codes.stride_l; jb.cs_h = in.codes.stride_h;
    jb.scale = in.p.scale; jb.zp = in.p.zp;
    jb.ps_r = in.p.share_l ? 0 : in.p.stride_r; jb.ps_h = in.p.stride_h; jb.ps_g = in.p.stride_g;
    jb.row_of_token = in.row_of_token; jb.row_begin = in.row_begin; jb.token0 = in.token0; jb.row0 = in.row0;
    jb.kernel = ((in.x.dtype == VARQ_F32 ? 0 : in.x.dtype == VARQ_F16 ? 3 : 6) + (in.store_bits == 8 ? 2 : in.store_bits == 4 ? 1 : 0)) * 4 +
                (in.p.zp == nullptr ? 2 : 0) + (norm_eps >= 0.f ? 1 : 0);
    jb.bits = in.bits; jb.eps = in.eps; jb.norm_eps = norm_eps; jb.group = in.p.group;
    jb.ranges = jb.norms = nullptr;
    jb.blocks = 0;
    if (in.p.share_l || in.p.share_h) {
        const int kind = plane_kind(in.p, D);
        const bool head = kind == 2;
        jb.xs_out = head ? jb.xs_h : jb.xs_l; jb.xs_in = head ? jb.xs_l : jb.xs_h;
        jb.cs_out = head ? jb.cs_h : jb.cs_l; jb.cs_in = head ? jb.cs_l : jb.cs_h;
        jb.ps_out = head ? jb.ps_h : jb.ps_r;
        return kind;
    }
    if (in.p.group % 8 || !pow2(in.p.group / 8) || (in.store_bits == 2 && in.p.group % 16) || D % in.p.group) return 0;
    const int tpr = D / 8;
    int bp = 1;
    while (bp * ROWS_NV < B) bp <<= 1;
    if (bp * tpr > ROWS_MAX_THREADS) return 0;
    jb.bp = bp;
    jb.nv = (B + bp - 1) / bp;
    jb.ngr = AP_THREADS / (tpr * bp) < 1 ? 1 : AP_THREADS / (tpr * bp);
    jb.h_fast = jb.xs_h <= jb.xs_l;
    const unsigned n_in = (unsigned)(jb.h_fast ? H : L);
    jb.div_s = 0;
    while ((1ull << jb.div_s) < n_in) ++jb.div_s;
    jb.div_m = (unsigned)(((1ull << 32) * ((1ull << jb.div_s) - n_in)) / n_in + 1);
    jb.blocks = (unsigned)(((long long)L * H + jb.ngr - 1) / jb.ngr);
    return 1;
}

// Planes: whether the cluster kernel holds `rows` rows in registers, and the cluster size
bool cluster_fits(long long rows, int D, int& cs) {
    const long long lanes = AP_THREADS / (D / 8);
    cs = 1;
    while (cs < 8 && cs * lanes < rows) cs <<= 1;        // one row per thread, then more
    return rows <= cs * lanes * HELD_ROWS;
}
// Row chunks per plane of the two-kernel path: about four CTAs per SM over both jobs
int plane_chunks(int n_jobs, long long rows, int planes) {
    long long c = ((long long)sm_count() * 4 + (long long)planes * n_jobs - 1) / ((long long)planes * n_jobs);
    if (c > 128) c = 128;
    if (c > (rows + 127) / 128) c = (rows + 127) / 128;
    return c < 1 ? 1 : (int)c;
}

}  // namespace

// (the larger of what one job alone and both jobs together use)
size_t append_workspace_bytes(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps) {
    size_t bytes = 0, lengths = 0;
    for (int i = 0; i < n_jobs; ++i) {
        const int kind = D <= 128 ? plane_kind(jobs[i].p, D) : 0;
        if (!kind) continue;
        const int planes = kind == 2 ? H : L;
        const long long rows = (long long)B * (kind == 2 ? L : H);
        int cs;
        if (cluster_fits(rows, D, cs)) continue;
        bytes += (size_t)planes * plane_chunks(1, rows, planes) * 2 * D * 4;
        if (i == 0 && k_norm_eps >= 0.f) lengths = (size_t)B * L * H * 4;
    }
    return bytes + lengths;
}

// Launches the jobs' step if kernels of this file take them: VARQ_OK, or VARQ_ERR_UNSUPPORTED without a launch.
int append_fast(const varq_append_job_t* jobs, int n_jobs, int B, int L, int H, int D, float k_norm_eps, void* ws, size_t ws_bytes, cudaStream_t st) {
    AppendArgs a;
    int kind[2] = {0, 0};
    for (int i = 0; i < n_jobs; ++i) kind[i] = plan_job(a.job[i], jobs[i], B, L, H, D, i == 0 ? k_norm_eps : -1.f);
    a.B = B; a.L = L; a.H = H; a.D = D;
    if (!kind[0] || (n_jobs > 1 && !kind[1])) return VARQ_ERR_UNSUPPORTED;
    const size_t need_ws = append_workspace_bytes(jobs, n_jobs, B, L, H, D, k_norm_eps);
    if (need_ws && (!ws || ws_bytes < need_ws)) return VARQ_ERR_UNSUPPORTED;
    const bool together = n_jobs == 1 || kind[0] == kind[1];
    for (int i = 0; i < (together ? 1 : n_jobs); ++i) {
        a.n_jobs = together ? n_jobs : 1;
        if (i == 1) a.job[0] = a.job[1];
        a.n_out = kind[i] == 3 ? L : H; a.n_in = kind[i] == 3 ? H : L; a.one_group = kind[i] == 3;
        a.chunks = a.chunk_rows = 0;
        const long long rows = (long long)B * a.n_in;
        int cs = 1;
        if (kind[i] == 1) {
            const int need = D / 8 * a.job[0].bp;            // (the same for both jobs)
            const unsigned blocks = a.job[0].blocks + (a.n_jobs > 1 ? a.job[1].blocks : 0u);
            VARQ_CUDA_TRY(need > AP_THREADS ? launch_pdl(append_rows_kernel<ROWS_MAX_THREADS>, blocks, ROWS_MAX_THREADS, 0, st, 1, a)
                                            : launch_pdl(append_rows_kernel<AP_THREADS>, blocks, AP_THREADS, 0, st, 1, a));
            count_launches(1);
        } else if (cluster_fits(rows, D, cs)) {
            VARQ_CUDA_TRY(launch_pdl(append_plane_cluster_kernel, (unsigned)(a.n_out * cs * a.n_jobs), AP_THREADS, 0, st, cs, a));
            count_launches(1);
        } else {
            a.chunks = plane_chunks(a.n_jobs, rows, a.n_out);
            a.chunk_rows = (int)((rows + a.chunks - 1) / a.chunks);
            float* p = reinterpret_cast<float*>(ws);
            for (int j = 0; j < a.n_jobs; ++j) { a.job[j].ranges = p; p += (size_t)a.n_out * a.chunks * 2 * D; }
            a.job[0].norms = p;
            const unsigned blocks = (unsigned)((long long)a.n_out * a.chunks * a.n_jobs);
            VARQ_CUDA_TRY(launch_pdl(append_plane_stats_kernel, blocks, AP_THREADS, 0, st, 1, a));
            VARQ_CUDA_TRY(launch_pdl(append_plane_apply_kernel, blocks, AP_THREADS, 0, st, 1, a));
            count_launches(2);
        }
    }
    return VARQ_OK;
}

}  // namespace varq
