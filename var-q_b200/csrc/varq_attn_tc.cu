// Tensor-core attention: choice of the instantiation, key splits and their merge, status.  The kernel is in varq_attn_tc.cuh.
#include "varq_attn_tc.cuh"

namespace varq {

// Partial rows of a split key range: one warp per (query row), lanes over head_dim.
__global__ void __launch_bounds__(256) attn_tc_merge_kernel(AttnArgs a, int tile_rows) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long row = blockIdx.x * 8ll + (threadIdx.x >> 5);
    if (row >= (long long)a.B * a.H * a.Lq) return;
    const int q = (int)(row % a.Lq);
    const int bh = (int)(row / a.Lq), b = bh / a.H, h = bh - b * a.H;
    const int qt = q / tile_rows, r = q - qt * tile_rows;
    const long long slots = (long long)a.B * a.H * a.splits * a.n_qtiles * tile_rows;
    auto slot = [&](int s) -> long long { return (((long long)bh * a.splits + s) * a.n_qtiles + qt) * tile_rows + r; };
    float m = -FLT_MAX;
    for (int s = 0; s < a.splits; ++s) m = fmaxf(m, a.ws[2 * slot(s)]);
    float den = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    const int per = a.D / 32;
    for (int s = 0; s < a.splits; ++s) {
        const long long sl = slot(s);
        const float w = ex2(a.ws[2 * sl] - m);
        den = fmaf(w, a.ws[2 * sl + 1], den);
        const float* o = a.ws + 2 * slots + sl * a.D + lane * per;
        for (int e = 0; e < per; ++e) acc[e] = fmaf(w, o[e], acc[e]);
    }
    const float inv = 1.f / den;
    for (int e = 0; e < per; ++e) store_o_elem(a.out, a.o_dtype, b * a.os_b + (long long)q * a.os_l + h * a.os_h + lane * per + e, acc[e] * inv);
}

// ---------------------------------------------------------------- host side
bool attn_tc_eligible(const AttnArgs& a, int kb, int vb) {
    if (a.D != 64 && a.D != 128) return false;
    if ((a.wk & 3) || (a.wv & 3)) return false;                // 16-byte rows for the bulk copies
    if (a.ks_l != a.wk || a.vs_l != a.wv) return false;        // tokens of one (sample, head) contiguous
    if (!a.k16 || !a.v16) return false;
    (void)kb; (void)vb;
    return true;
}

// Two query tiles per CTA share every converted K / V tile; a second tile needs queries to fill it.  Where such CTAs would fill at most half
// of the SMs, single tiles occupy twice as many.  One / two, int8 per head, int8 per dim and int4 in groups of 32, bf16 and fp32 queries, H16 and H30:
//   CTAs of two tiles      300 to 680 tokens   1024          2048          4096
//   38 to 72               0.78 to 1.00        0.78 to 0.97  0.78 to 1.00  0.77 to 1.01     (neither is split; 74 of 150 queries 0.84 to 1.02, fp32 per dim 1.04 to 1.12)
//   80 to 144              1.00 to 1.10        1.06 to 1.17  1.07 to 1.22  1.07 to 1.23     (two single tiles share an SM and convert everything twice)
//   20 to 37               0.63 to 0.91        0.83 to 1.02  1.13 to 1.39  1.57 to 1.81     (the key range of two tiles is split, that of one is not)
// In the last row one / two cross at 1100 to 1300 tokens.  With fewer CTAs still both are split: 0.81 to 0.97 for 256 queries of 16 pairs, but 1.09 for
// 169 over 424 tokens, per dim.
static int tc_query_tiles(int B, int H, int Lq, int Lk, int D) {
    if (D != 64 || Lq <= TC_M) return 1;
    const long long heads = (long long)B * H, one = heads * ((Lq + TC_M - 1) / TC_M), two = heads * ((Lq + 2 * TC_M - 1) / (2 * TC_M));
    const bool split = two * 4 <= sm_count();
    return two * 2 <= sm_count() && one * 4 > sm_count() && (!split || Lk <= 16 * TC_N) ? 1 : 2;
}

// Key range of a CTA.  Splitting pays when the CTAs of the unsplit grid leave most of the chip idle and every part still has a few
// tiles to hide its set-up behind (the merge is a second launch).
static int tc_splits(int B, int H, int Lq, int Lk, int D, int& tiles_per_split) {
    const int tiles = (Lk + TC_N - 1) / TC_N, rows = tc_query_tiles(B, H, Lq, Lk, D) * TC_M;
    const long long ctas = (long long)B * H * ((Lq + rows - 1) / rows);
    tiles_per_split = tiles;
    if (ctas * 4 > sm_count()) return 1;
    long long s = sm_count() / ctas;
    if (s > tiles / 3) s = tiles / 3;
    if (s <= 1) return 1;
    tiles_per_split = (int)((tiles + s - 1) / s);
    return (tiles + tiles_per_split - 1) / tiles_per_split;
}

size_t attn_tc_workspace_bytes(int B, int H, int Lq, int Lk, int D) {
    if (D != 64 && D != 128) return 0;
    int tps;
    const int splits = tc_splits(B, H, Lq, Lk, D, tps), rows = tc_query_tiles(B, H, Lq, Lk, D) * TC_M;
    if (splits == 1) return 256;
    return (size_t)B * H * splits * ((Lq + rows - 1) / rows) * rows * (D + 2) * sizeof(float) + 256;
}

// Step tables of at most this many bytes (K and V together) fit behind the fixed part of every plan of the head_dim: 66 steps of K and
// V at 64, 18 at 128 (the schedules of the models have 10 to 13).  Longer histories, and those whose number of steps is not given, have
// tables that move along (28 KB at both head_dims: at 64 two CTAs then share an SM).  B8 H16 c128, 256 bf16 queries over 2560 tokens in
// 18 / 40 / 64 steps of K and V, us: 117 / 150 / 180, and 537 for 40 and 64 on the fp32 routine.
constexpr int STEP_TABLE_BYTES_64 = 50 * 1024, STEP_TABLE_BYTES = 28 * 1024;
static int par_mode(const ParamView& pv, int D) {
    if (pv.group == D) return PM_EXACT;
    if (pv.group % 16 == 0 && (pv.group & (pv.group - 1)) == 0 && D / pv.group <= 4) return PM_GROUP;
    return pv.row_of_token ? PM_STEP : PM_SLOW;
}
static void step_tables(const AttnArgs& a, TcDyn& dy) {
    const bool ks = dy.k_mode == PM_STEP, vs = dy.v_mode == PM_STEP;
    const long long k = ks ? a.kp.n_rows : 0, v = vs ? a.vp.n_rows : 0;
    const bool known = (!ks || k > 0) && (!vs || v > 0);
    if (known && (k + v) * 3 * a.D * 2 <= (a.D == 64 ? STEP_TABLE_BYTES_64 : STEP_TABLE_BYTES)) { dy.k_rows = (int)k; dy.v_rows = (int)v; return; }
    const int room = STEP_TABLE_BYTES / (3 * a.D * 2);
    if (ks) { dy.k_mode = PM_WINDOW; dy.k_rows = vs ? room / 2 : room; }
    if (vs) { dy.v_mode = PM_WINDOW; dy.v_rows = room - dy.k_rows; }
}
static int bulk_params(const ParamView& pv, int D) {
    const int ng = D / pv.group;
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    return pv.row_of_token == nullptr && pv.sg == 1 && pv.sr == ng && (pv.sb & 3) == 0 && (pv.sh & 3) == 0 && al(pv.scale) && (!pv.zp || al(pv.zp));
}

int attn_tc_run(const AttnArgs& a0, int kb, int vb, void* ws, size_t ws_bytes, cudaStream_t st) {
    AttnArgs a = a0;
    // fp16 queries, and bf16 queries inside fp16's normal range (2^-14 <= |q| <= 65504), are exact in one fp16 term;
    // larger magnitudes saturate, smaller ones lose low bits (both far outside what a softmax can resolve)
    bool split_q = a.q_dtype == VARQ_F32 || a.q_norm;
    const size_t need = attn_tc_workspace_bytes(a.B, a.H, a.Lq, a.Lk, a.D);
    if (!ws || ws_bytes < need)
        return fail(VARQ_ERR_WORKSPACE, "varq_attn_fwd: workspace of %zu bytes needed, %zu given", need, ws_bytes);
    a.splits = tc_splits(a.B, a.H, a.Lq, a.Lk, a.D, a.tiles_per_split);
    a.ws = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(ws) + 15) & ~(uintptr_t)15);
    TcDyn dy = {};
    dy.k_mode = par_mode(a.kp, a.D);
    dy.v_mode = par_mode(a.vp, a.D);
    for (ParamView* pv : {&a.kp, &a.vp})
        if (pv->n_rows > a.Lk) pv->n_rows = 0;         // more rows than keys: read those that the keys name
    step_tables(a, dy);
    const bool window = dy.k_mode == PM_WINDOW || dy.v_mode == PM_WINDOW;
    const int qt = window ? 1 : tc_query_tiles(a.B, a.H, a.Lq, a.Lk, a.D), rows = qt * TC_M;       // (fewer rows of partials than the workspace is sized for)
    a.n_qtiles = (a.Lq + rows - 1) / rows;
    if ((long long)a.B * a.H * a.n_qtiles * a.splits * rows > 0x7fffffffLL) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: more than 2^31 query rows");
    dy.k_bulk = dy.k_mode == PM_GROUP && bulk_params(a.kp, a.D);
    dy.v_bulk = dy.v_mode == PM_GROUP && bulk_params(a.vp, a.D);
    split_q = split_q || window;
    const TcFile& f = a.D == 128 ? (split_q ? tc_d128_q2 : tc_d128_q1)
                    : qt == 2 ? (split_q ? tc_d64_x2_q2 : tc_d64_x2_q1) : (split_q ? tc_d64_q2 : tc_d64_q1);
    if (int rc = f.launch(a, dy, kb, vb, st)) return rc;
    if (a.splits > 1) {
        const long long q_rows = (long long)a.B * a.H * a.Lq;
        VARQ_CUDA_TRY(launch_pdl(attn_tc_merge_kernel, (unsigned)((q_rows + 7) / 8), 256, 0, st, 1, a, rows));
        count_launches(1);
    }
    return VARQ_OK;
}

int attn_tc_status(int* out) {
    *out = 0;
    // a symbol copy on the legacy default stream does not wait for kernels on non-blocking streams: wait for the device first
    VARQ_CUDA_TRY(cudaDeviceSynchronize());
    for (const TcFile* f : {&tc_d64_q1, &tc_d64_q2, &tc_d64_x2_q1, &tc_d64_x2_q2, &tc_d128_q1, &tc_d128_q2})
        if (int rc = f->status(out)) return rc;
    return VARQ_OK;
}

}  // namespace varq
