// C entry points of attention over the packed cache: argument checks and kernel selection.
#include "varq_attn.cuh"

using namespace varq;

// Kernel choice pinned by varq_attn_force_path (0 = automatic).  A test hook, not a fallback switch: a pinned
// kernel that cannot take the call still yields to the general CUDA-core kernel.
static int g_forced_path = 0;

static bool words_aligned16(const varq_tensor_t* t, int words) {
    return (words % 4 == 0) && aligned16(t->ptr) && (t->stride_b % 4 == 0) && (t->stride_l % 4 == 0) &&
           (t->stride_h % 4 == 0);
}

extern "C" size_t varq_attn_workspace_bytes(int32_t B, int32_t H, int32_t Lq, int32_t Lk, int32_t D,
                                            int32_t k_store_bits, int32_t v_store_bits) {
    (void)k_store_bits; (void)v_store_bits;
    if (B <= 0 || H <= 0 || Lq <= 0 || Lk <= 0 || D <= 0) return 0;
    const size_t s1 = attn_small_workspace_bytes(B, H, Lq, Lk, D), s2 = attn_stream_workspace_bytes(B, H, Lq, Lk, D);
    const size_t s3 = attn_tc_workspace_bytes(B, H, Lq, Lk, D);
    const size_t s4 = D == 64 || D == 128 ? attn_decode_workspace_bytes(B, H, Lq, Lk, D) : 0;
    const size_t s12 = s1 > s2 ? s1 : s2, s34 = s3 > s4 ? s3 : s4;
    return s12 > s34 ? s12 : s34;
}

// 33 to 64 queries over a short cache, one scale per key, head_dim 64: one CTA of the warp-level kernel per (sample, head), four of which share an SM (three
// with fp32 queries), against two CTAs per SM of the tcgen05 kernel.  us at H16, int8, mid / tcgen05:
//     16-bit queries   33 over 40   48 over 64   64 over 64   36 over 91   64 over 128  48 over 200   fp32   33 over 40   48 over 64   36 over 91   64 over 128
//     batch  20       10.3 / 12.9  11.5 / 12.2  13.2 / 12.2  13.6 / 14.8  17.0 / 14.3  21.7 / 19.3          10.9 / 13.3  11.7 / 12.6  13.9 / 15.3  16.1 / 14.4
//            32       10.6 / 15.9  11.9 / 14.9  13.5 / 14.9  13.7 / 17.7  17.3 / 17.1  21.8 / 22.2          18.6 / 16.1  20.1 / 15.2  23.4 / 18.1  27.6 / 17.4
//            40       18.4 / 20.9  19.5 / 19.9  20.8 / 19.9  23.9 / 23.4  27.2 / 22.7  35.7 / 29.7          19.8 / 21.1  21.4 / 20.2  24.6 / 24.0  29.7 / 23.1
//            64       19.8 / 30.0  22.1 / 29.0  25.1 / 29.0  26.1 / 33.7  32.7 / 32.8  41.3 / 42.4          28.4 / 30.6  31.2 / 29.4  36.0 / 34.4  42.4 / 33.2
//            128      37.7 / 53.6  41.9 / 50.9  46.1 / 51.2  49.6 / 60.2  58.9 / 58.1  78.8 / 76.3          48.7 / 54.8  51.9 / 52.2  62.8 / 61.9  73.1 / 59.4
// (int4: mid 3 to 10 % less, 64 over 155 B64 34.2 / 39.2, 48 over 200 38.3 / 43.3.)  Up to two CTAs per SM tcgen05 is the faster one (33 over 40, batch 16:
// 10.2 / 8.2); beyond, what counts is how full the last wave of mid is and how little work a CTA has.  Both keep weights in fp16 and sums in fp32.
static bool mid_takes_64(bool fp32, bool narrow, long long heads, int Lq, int Lk) {
    if (heads <= 2 * sm_count()) return false;
    const long long wave = (fp32 ? 3 : 4) * sm_count(), waves = (heads + wave - 1) / wave;
    if (fp32 && waves > 1) return Lq <= 40 && Lk <= 64 && heads * 10 >= waves * wave * 7;
    const bool full = heads * 4 >= waves * wave * 3;
    return Lk <= 96 ? full || Lq <= 48 : full && narrow && !fp32 && Lk <= 208;       // narrow: K and V below 8 bits
}

static int attn_impl(const varq_tensor_t* q, const varq_tensor_t* k_codes, const varq_tensor_t* v_codes,
                     const varq_qparams_t* kp, const varq_qparams_t* vp, int32_t B, int32_t H, int32_t Lq,
                     int32_t Lk, int32_t D, int32_t kb, int32_t vb, float softmax_scale,
                     const varq_tensor_t* out, void* workspace, size_t workspace_bytes, void* stream, bool q_norm, const float* q_mul, float q_eps) {
    if (!q || !k_codes || !v_codes || !kp || !vp || !out) return fail(VARQ_ERR_ARG, "varq_attn_fwd: null descriptor");
    if ((kb != 2 && kb != 4 && kb != 8) || (vb != 2 && vb != 4 && vb != 8))
        return fail(VARQ_ERR_ARG, "varq_attn_fwd: store bits must be 2, 4 or 8 (got %d, %d)", kb, vb);
    if (B < 0 || H < 0 || Lq < 0 || Lk < 0 || D <= 0) return fail(VARQ_ERR_ARG, "varq_attn_fwd: bad shape");
    if (!dtype_ok(q->dtype) || !dtype_ok(out->dtype)) return fail(VARQ_ERR_ARG, "varq_attn_fwd: bad q/out dtype");
    if ((long long)B * H * Lq == 0) return VARQ_OK;
    if (Lk == 0) return fail(VARQ_ERR_ARG, "varq_attn_fwd: empty cache (Lk = 0)");
    if (!q->ptr || !out->ptr || !k_codes->ptr || !v_codes->ptr || !kp->scale || !vp->scale)
        return fail(VARQ_ERR_ARG, "varq_attn_fwd: null pointer");
    if (kp->group < 1 || kp->group > D || D % kp->group || vp->group < 1 || vp->group > D || D % vp->group)
        return fail(VARQ_ERR_ARG, "varq_attn_fwd: group must divide head_dim");
    const int kvw = 32 / kb, vvw = 32 / vb;
    if (D % kvw || D % vvw || D % 4) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: head_dim %d must be a multiple of the codes per word (%d, %d)", D, kvw, vvw);
    const int wk = D / kvw, wv = D / vvw;
    if (wv > 128 || (128 % wv) != 0)
        return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: V words per row (%d) must divide 128", wv);
    if (D > 256) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: head_dim %d > 256", D);

    AttnArgs a;
    a.q = q->ptr; a.q_dtype = q->dtype; a.qs_b = q->stride_b; a.qs_l = q->stride_l; a.qs_h = q->stride_h;
    a.out = out->ptr; a.o_dtype = out->dtype; a.os_b = out->stride_b; a.os_l = out->stride_l; a.os_h = out->stride_h;
    a.kc = (const int32_t*)k_codes->ptr; a.ks_b = k_codes->stride_b; a.ks_l = k_codes->stride_l; a.ks_h = k_codes->stride_h;
    a.vc = (const int32_t*)v_codes->ptr; a.vs_b = v_codes->stride_b; a.vs_l = v_codes->stride_l; a.vs_h = v_codes->stride_h;
    a.kp = make_param_view(kp);
    a.vp = make_param_view(vp);
    a.B = B; a.H = H; a.Lq = Lq; a.Lk = Lk; a.D = D;
    a.wk = wk; a.wv = wv; a.kpitch = wk;
    a.k16 = words_aligned16(k_codes, wk);
    a.v16 = words_aligned16(v_codes, wv);
    a.scale_log2 = softmax_scale * 1.4426950408889634f;
    a.splits = 1; a.tiles_per_split = 0; a.n_qtiles = 1; a.ws = reinterpret_cast<float*>(workspace);
    a.q_norm = q_norm ? 1 : 0; a.q_mul = q_mul; a.q_eps = q_eps;
    if (q_norm && !attn_tc_eligible(a, kb, vb)) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd_qnorm: no kernel normalises the queries of this shape or layout");
    // The CUDA-core streaming kernel is memory-bound only while its arithmetic (queries x keys x head_dim on the FMA pipe)
    // stays below the time to stream the packed cache: up to 4 queries at any cache length, and the 1-16-query first scales
    // of a schedule, whose caches are a few hundred tokens at most.  Everything else goes to the tensor cores, where a
    // 128-row tile with few live rows still finishes a long cache sooner.  Queries normalised on the way in follow the same rules as
    // queries that arrive normalised, so that few of them keep fp32 weights: on the tcgen05 kernel (weights and dequantised V in
    // fp16) the first scales of a per-dim or group-wise cache are 2e-4 away from the exact result, here 2e-7.
    const int force = __atomic_load_n(&g_forced_path, __ATOMIC_RELAXED);
    const bool small_q = Lq <= 4 || (Lq <= 16 && Lk <= 256);
    // head_dim 64 with one scale per key over at most 256 tokens (the early scales of a schedule), us at H16, int8:
    //               9 queries over 14 tokens                            12 over 30                                          16 over 30
    //               fp32                  16-bit                normal. fp32                  16-bit                normal. fp32                  16-bit                normal.
    //     batch     mid / decode / early  mid / decode / early  early   mid / decode / early  mid / decode / early  early   mid / decode / early  mid / decode / early  early
    //       2       9.4 /  3.9 /  6.1     8.8 /  3.9 /  6.6     7.2     9.7 /  3.9 /  7.8     9.1 /  4.0 /  8.4     8.9     9.6 /  4.1 /  8.2     9.0 /  4.2 /  8.8     9.5
    //      16      10.5 /  7.1 /  7.2    10.0 /  7.1 /  7.7     8.3    10.9 /  7.5 /  9.5    10.3 /  7.6 / 10.1    10.6    10.8 /  8.1 / 10.5    10.3 /  8.3 / 11.1    11.8
    //      32      10.9 / 10.3 /  8.1    11.4 / 10.3 /  8.6     8.9    11.3 / 11.2 / 10.6    11.9 / 11.2 / 11.2    11.9    11.2 / 12.2 / 11.5    11.8 / 12.2 / 12.2    13.4
    //      40      11.0 / 11.6 /  9.4    11.6 / 11.5 /  9.9    10.4    11.4 / 12.2 / 12.8    12.2 / 12.1 / 13.2    13.8    11.4 / 12.6 / 13.9    12.2 / 12.6 / 14.6    15.4
    //      64      19.3 / 17.3 /  9.6    11.8 / 17.2 / 10.0    10.6    19.9 / 18.7 / 13.0    12.4 / 18.6 / 13.4    14.1    19.7 / 19.9 / 14.2    12.4 / 19.9 / 14.8    15.6
    //     128      29.2 / 32.0 / 17.8    21.7 / 31.8 / 18.6    19.7    30.4 / 35.1 / 24.0    22.6 / 34.7 / 24.9    26.2    30.2 / 37.6 / 26.4    22.5 / 37.9 / 27.6    29.0
    // (decode on normalised queries 0.3 to 4 us more than on fp32, early at 30 heads or a batch of 30 up to 13 % more than between its neighbours.)  decode and early
    // keep weights to fp32's accuracy (1e-7 against 2e-4).  Over one chunk of keys early takes up to 12 queries, and 13 to 16 where mid would need fp32 operands
    // or cannot normalise, beyond 5 (sample, head) pairs per SM; from 3 per SM on only while half a chunk is enough.  13 to 16 queries of more than 512 pairs
    // that early leaves go to mid, everything else to decode, also over more keys: there mid is the faster one on 16-bit queries (16 over 64 B64
    // 13.2 / 21.2, 16 over 256 30.3 / 30.1) and decode keeps its accuracy.
    // 17 to 32 queries: mid where the tcgen05 kernel needs more than one wave (two CTAs per SM; 25 over 55, mid / tcgen05: B16 11.3 / 9.0, B32 12.9 / 16.9,
    // B64 22.7 / 30.9); up to 64: mid_takes_64.
    const long long heads = (long long)B * H;
    const bool key_scale = D == 64 && kp->group == D && vp->group == D, few = Lq > 8 && Lq <= 16 && Lk <= 256, mid_few = heads > 512 && Lk <= 32 && Lq > 12;
    const bool early_few = few && Lk <= 32 && (heads > 5 * sm_count() ? Lq <= 12 || q->dtype == VARQ_F32 || q_norm : heads > 3 * sm_count() && Lk <= 16);
    if (!force && key_scale && early_few && attn_early_eligible(a)) return attn_early_run(a, kb, vb, (cudaStream_t)stream);
    // A handful of queries over a long cache: warp-level tensor-core instructions fed from global memory, where one scale covers a key.
    // us at H16, int4, bf16 queries, decode / tcgen05 (the streaming kernel takes 1.8 to 6 times decode's time):
    //     B64 c64   8 x 300: 22 / 47, 16 x 300: 37 / 47, 16 x 2240: 205 / 179, 8 x 10521: 421 / 754, 16 x 10521: 763 / 757
    //     B64 c128  8 x 300: 42 / 75, 16 x 300: 73 / 75, 16 x 2240: 325 / 229, 8 x 10521: 660 / 893, 16 x 10521: 1199 / 902
    //     B2  c128  8 x 300: 10.4 / 10.0, 16 x 2240: 26 / 20, 16 x 10521: 50 / 44;   B2 c64  16 x 2240: 18 / 21, 16 x 10521: 39 / 56
    // Up to 8 queries (one CTA's worth) it is the faster one; from 9 to 16 it takes 0.6 to 1.4 times as long and stays for its
    // accuracy (3e-7 against 2e-4 for fp16 weights).
    const bool want_decode = force ? (force == VARQ_ATTN_PATH_DECODE) : Lq <= 16 && (Lk > 256 || (few && D == 64 && (q_norm || !mid_few)));
    if (want_decode && Lq <= 16 && attn_decode_eligible(a, kb, vb)) return attn_decode_run(a, kb, vb, workspace, workspace_bytes, (cudaStream_t)stream);
    const bool want_mid = force ? (force == VARQ_ATTN_PATH_MID) : few || (Lq > 16 && Lq <= 32 && Lk <= 256 && heads > 2 * sm_count())
                                                                                 || (Lq > 32 && Lq <= 64 && mid_takes_64(q->dtype == VARQ_F32, kb < 8 && vb < 8, heads, Lq, Lk));
    if (want_mid && !q_norm && attn_mid_eligible(a, kb, vb)) return attn_mid_run(a, kb, vb, (cudaStream_t)stream);
    const bool want_tc = force ? (force == VARQ_ATTN_PATH_TC) : !small_q;
    if (want_tc && attn_tc_eligible(a, kb, vb)) return attn_tc_run(a, kb, vb, workspace, workspace_bytes, (cudaStream_t)stream);
    const bool want_stream = force ? (force == VARQ_ATTN_PATH_STREAM) : small_q;
    if (want_stream && attn_stream_eligible(a, kb, vb)) return attn_stream_run(a, kb, vb, workspace, workspace_bytes, (cudaStream_t)stream);
    // Parameters that vary inside 16 head_dim values: up to 16 queries over at most 256 tokens have a kernel of their own.  us, general kernel /
    // early, int8 per dim, 4 / 9 / 16 queries over 5 / 14 / 30 tokens: B2 H16 c64 11.9 / 5.6, 12.5 / 7.0, 13.4 / 9.2; B64 H16 c64 24.8 / 8.4, 62 / 12,
    // 85 / 17; 16 queries over 256 tokens 283 / 84; c128 B6 H16 20.5 / 8.0 (4), 23.4 / 11.7 (16).  Relative L2 error 1.3e-7 / 1.1e-7.
    const bool want_early = force ? (force == VARQ_ATTN_PATH_EARLY) : Lq <= 16 && Lk <= 256;
    if (want_early && attn_early_eligible(a)) return attn_early_run(a, kb, vb, (cudaStream_t)stream);
    return attn_small_run(a, kb, vb, workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int varq_attn_fwd(const varq_tensor_t* q, const varq_tensor_t* k_codes, const varq_tensor_t* v_codes,
                             const varq_qparams_t* kp, const varq_qparams_t* vp, int32_t B, int32_t H, int32_t Lq,
                             int32_t Lk, int32_t D, int32_t kb, int32_t vb, float softmax_scale,
                             const varq_tensor_t* out, void* workspace, size_t workspace_bytes, void* stream) {
    return attn_impl(q, k_codes, v_codes, kp, vp, B, H, Lq, Lk, D, kb, vb, softmax_scale, out, workspace, workspace_bytes, stream, false, nullptr, 0.f);
}

extern "C" int varq_attn_fwd_qnorm(const varq_tensor_t* q, const varq_tensor_t* k_codes, const varq_tensor_t* v_codes,
                                   const varq_qparams_t* kp, const varq_qparams_t* vp, int32_t B, int32_t H, int32_t Lq,
                                   int32_t Lk, int32_t D, int32_t kb, int32_t vb, float softmax_scale, const float* q_mul, float q_eps,
                                   const varq_tensor_t* out, void* workspace, size_t workspace_bytes, void* stream) {
    return attn_impl(q, k_codes, v_codes, kp, vp, B, H, Lq, Lk, D, kb, vb, softmax_scale, out, workspace, workspace_bytes, stream, true, q_mul, q_eps);
}

extern "C" int varq_attn_force_path(int32_t path) {
    if (path < VARQ_ATTN_PATH_AUTO || path > VARQ_ATTN_PATH_EARLY) return fail(VARQ_ERR_ARG, "varq_attn_force_path: unknown path %d", path);
    __atomic_store_n(&g_forced_path, (int)path, __ATOMIC_RELAXED);
    return VARQ_OK;
}

extern "C" int varq_device_status(int32_t* status) {
    if (!status) return fail(VARQ_ERR_ARG, "varq_device_status: null pointer");
    int v = 0;
    if (int rc = attn_tc_status(&v)) return rc;
    *status = v;
    return VARQ_OK;
}
