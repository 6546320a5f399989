// Attention over the packed cache on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a: the kernel template.
//
// One CTA = one (sample, head) x QT tiles of 128 queries, looping over tiles of 64 keys; everything that is not a packed code stays
// in tensor memory: the queries (fp16 hi [+ lo] halves, the A operand of S = Q K^T), the scores S, the probabilities P (fp16, written
// over the S columns they came from, the A operand of O += P V) and the output accumulators.  Shared memory then only feeds the
// B operands: with A in shared memory a 128 x 64 x 16 product costs 48 cycles of its bandwidth against 32 of the tensor pipe
// (measured), with A in tensor memory it runs at the pipe's rate.  Warps:
//   softmax    one thread per query row (= TMEM lane) at head_dim 64, two at 128.  A thread reads the scores of a key tile, applies the per-key
//              tables where K or V keep exact codes, exponentiates against a lazily updated reference, sums the rounded P in registers
//              and writes P back to tensor memory;
//   K and V converters: turn a tile's packed rows into 128B-swizzled fp16 operand tiles in shared memory.  K: exact integer codes
//              minus zero-point (one scale per key, applied to S in fp32), or an fp16 hi + lo pair of (code - zp) * scale when the scale
//              varies along head_dim.  V: codes minus zero-point (the per-key scale is folded into P through the exponent and taken out
//              of the row sum), or (code - zp) * scale rounded once to fp16;
//   MMA warp   waits converged; one elected lane issues tcgen05.mma and commits completion to mbarriers;
//   load warps one for K, one for V: a lane requests packed rows (and the raw scales of grouped parameters) up to three tiles ahead by
//              1-D bulk copies; all lanes fetch per-key parameters one tile ahead into registers and write them as records and
//              softmax tables.
// More than 128 queries share each converted tile (QT = 2, head_dim 64, all 512 TMEM columns); up to 128 queries run as two CTAs per SM of
// 256 columns each, one CTA's set-up and dependent waits under the other's tiles.  At head_dim 128 one CTA keeps three or four score
// tiles in flight.
// What bounds it, from builds that leave out arithmetic and keep every load, store, barrier and product (us a call: whole / no exponentials / constant
// operand tiles instead of conversion / neither; constant operands also draw less power):
//   c 64   B64 H16 256 x 10521, int2 group 32, bf16 queries       1237 /  853 / 1026 /  719
//          B32 H30 1024 x 2240, int4, K per dim, fp32 queries      1298 / 1150 / 1178 / 1072
//          B64 H16 256 x 680, int8 per head, fp32 queries          151 /  152 /  146 /  138
//   c 128  B4 H16 4096 x 10521, int4 and int2 group 32, fp32      2622 / 2591 / 1715 / 1425
//          B6 H16 1600 x 6000, int8 per dim, fp32                 1067 / 1063 /  653 /  630
//          B2 H16 4096 x 10521, int8 per head, bf16               1043 / 1083 /  952 /  943
// At head_dim 64 over long caches the softmax warps, two per sub-partition: 64 x 256 scores need 1024 cycles of the exponential unit, a tile takes 2100;
// over short ones what surrounds the tile loop.  At 128 the conversion of a dequantised K, in issue slots and in what its hi + lo operands draw (2250 cycles
// a tile at the full clock, 1024 of them the tensor pipe's; long calls run into the power limit).
// Few CTAs over a long cache: the key range is split across CTAs and a second kernel merges the partial rows.
// Numerics: integer codes are exact in fp16; an fp32 query is split into hi + lo fp16 halves, a dequantised K likewise (the lo x lo
// product is below fp32 resolution), so S has fp32-like accuracy; P and a dequantised V are rounded to fp16 once; sums are fp32.
// A V scale below 2^-20 is folded as 2^-20 (the error is below 127 * 2^-20 per unit of attention weight).
// Every wait is bounded: on expiry the kernel records a status code and all roles drain out.
#pragma once
#include <cfloat>

#include "varq_attn.cuh"
#include "varq_codes.cuh"

namespace varq {

constexpr int TC_M = 128;             // queries per tile
constexpr int TC_N = 64;              // keys per tile
constexpr uint32_t TC_WAIT_NS = 20000;         // one suspended try of a barrier wait
constexpr uint32_t TC_SPIN_LIMIT = 1u << 16;   // tries before a wait gives up (about a second)

static __device__ int g_tc_status = 0;   // first failure code of any launch of this file since the last read (0 = none)

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(TC_WAIT_NS) : "memory");
    return ok != 0;
}
// Most waits of a steady loop find their phase complete.  try_wait with a time limit costs a couple of hundred cycles even then
// (measured per wait site), test_wait a shared-memory round trip: it goes first.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when the limit expires or another thread has already given up.
// Everything is inline and small: a call here costs a few hundred cycles of register shuffling
// around it, at every one of the ~20 wait sites, and bloats the loops that hold them.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (mbar_test(bar, parity)) return true;
    uint32_t tries = 0;
#pragma unroll 1
    while (!mbar_try(bar, parity)) {     // a failed try_wait has already been suspended by the hardware for a while
        if (*abort_flag) return false;
        if (++tries >= TC_SPIN_LIMIT) {
            *abort_flag = 1;
            atomicCAS(&g_tc_status, 0, code);
            return false;
        }
    }
    return true;
}
// The same by a converged warp, which stays converged: all lanes poll and agree.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
    uint32_t tries = 0;
#pragma unroll 1
    while (!__all_sync(0xffffffffu, mbar_try(bar, parity))) {
        if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
        if (++tries >= TC_SPIN_LIMIT) {
            *abort_flag = 1;
            atomicCAS(&g_tc_status, 0, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Both are called by every lane of the MMA warp with the same operands and executed by one elected lane: the warp stays
// converged, so the descriptors are computed once in uniform registers, which is where the instruction takes them from.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[tmem] B[smem]; A holds two fp16 per 32-bit column, row = lane
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void sts128(void* p, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    *reinterpret_cast<uint4*>(p) = make_uint4(x, y, z, w);
}

// Shared-memory matrix descriptor, 128-byte swizzle, sm_100 format:
// [0,14) start >> 4 | [16,30) leading byte offset >> 4 | [32,46) stride byte offset >> 4 |
// [46,48) version = 1 | [61,64) layout type (2 = SWIZZLE_128B)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor, kind::f16: fp16 A and B, fp32 accumulator.
// [4,6) c format (1 = f32) | [7,10) a format (0 = f16) | [10,13) b format | 15 a major | 16 b major
// (0 = K-major, 1 = MN-major) | [17,23) N >> 3 | [24,29) M >> 4
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, int b_mn_major) {
    return (1u << 4) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// Byte offset of the 16-byte chunk `ch` (eight head_dim values) of key `key` in a 128B-swizzled tile of 64 keys: the 64-column blocks
// hold 64 rows of 128 bytes.  The same layout serves K (K-major B: row = N index, columns = contraction) and V (MN-major B: row =
// contraction index, columns = N).
__device__ __forceinline__ uint32_t chunk_off(int key, int ch) {
    return (uint32_t)((ch >> 3) * (TC_N * 128) + (key >> 3) * 1024 + (key & 7) * 128 + (((ch & 7) ^ (key & 7)) << 4));
}

// ---------------------------------------------------------------- how K / V parameters reach the converters
enum ParMode : int {
    PM_EXACT = 0,     // one scale / zero-point per key: integer codes, scale applied outside the product
    PM_GROUP = 1,     // raw (key, group) parameters of a tile in shared memory: groups of whole 16-code items, at most 4 per key
    PM_STEP = 2,      // per-dim parameters shared by the tokens of an appended step: a table [steps][3][D] in shared memory
    PM_WINDOW = 3,    // the same with more steps than such a table holds: it keeps consecutive steps and moves on where a tile needs others.
                      // A mode of its own, with one query tile and split queries only: in the kernels above the test per tile cost 4 %
    PM_SLOW = 4,      // anything else: fp32 parameters straight from global memory (runs in the PM_GROUP kernels)
};

__host__ __device__ constexpr bool per_step(int mode) { return mode == PM_STEP || mode == PM_WINDOW; }

template <int D, int NQ, int QT, int KM, int VM> struct TcPlan {
    static constexpr bool KX = KM == PM_EXACT, VX = VM == PM_EXACT;
    static constexpr int CTAS = (D == 64 && QT == 1) ? 2 : 1;  // resident CTAs per SM
    // converter warps: a tile is 64 * D / 16 items of 16 codes
    // Two threads per query row at head_dim 128.  ALT: they take the even and the odd key tiles, each with its own reference maximum and
    // accumulator in tensor memory, and meet in the epilogue, so the two warps of a sub-partition hide each other's latencies (score loads,
    // barriers).  Else each takes half of every tile's keys and they agree on one reference: with two query operands (hi + lo) the second
    // accumulator would leave room for two score tiles only, and the chain score product -> softmax -> output product then binds (B8 H16
    // Lq2048 Lk4096 int4, us: one operand 985 -> 814, two operands 1028 -> 1131, so those stay; dequantised K, 1035 -> 1032, is not bound by its softmax warps alone).
    static constexpr bool ALT = D == 128 && NQ == 1 && KX;
    static constexpr int KW = D == 128 ? (ALT ? 4 : 8) : 2 * QT, VW = D == 128 ? 4 : 2 * QT;
    static constexpr int KTHR = KW * 32, VTHR = VW * 32;
    static constexpr int HV = D == 128 ? 2 : 1;                // threads per query row
    static constexpr int K_WARP0 = 4 * HV * QT, V_WARP0 = K_WARP0 + KW, MMA_WARP = V_WARP0 + VW, LOAD_WARP = MMA_WARP + 2;     // one for K, one for V
    static constexpr int WARPS = MMA_WARP + 4, THREADS = WARPS * 32;      // roles are whole warpgroups
    // Registers per thread by role (setmaxnreg): the launch has REGS * THREADS of them
    static constexpr int REGS = (65536 / (THREADS * CTAS)) / 8 * 8;
    static constexpr int REGS_MISC = 48, REGS_CONV = D == 64 && QT == 1 ? 88 : 96;
    static constexpr int REGS_SOFT = ((REGS * WARPS - REGS_MISC * 4 - REGS_CONV * (KW + VW)) / (4 * HV * QT)) / 8 * 8;
    static_assert(K_WARP0 % 4 == 0 && MMA_WARP % 4 == 0, "warpgroup roles");
    static_assert(REGS_SOFT * 4 * HV * QT + REGS_CONV * (KW + VW) + REGS_MISC * 4 <= REGS * WARPS, "register plan");
    static constexpr int KT = KX ? 1 : 2;                     // K operand tiles per stage (hi, lo when K is dequantised)
    static constexpr int T_BYTES = TC_N * D * 2;              // one fp16 operand tile
    static constexpr int KST = CTAS == 2 ? 2 : 3, VST = KST;  // operand stages
    static constexpr int PST = D == 128 ? 2 : KST;            // packed stages (at most KST)
    static constexpr int SB = D == 64 ? 2 : ALT ? 3 : 4;    // score tiles in tensor memory, per query tile
    // The softmax of a tile: one block of exponentials, conversion and sum, behind which the reference may turn out to be too low, or the maximum
    // first.  At head_dim 128 the block takes issue slots from the converters of a dequantised K and from the other tile of ALT.  us, block / maximum
    // first, B2 H16 4096 x 10521: int8 in groups of 32 1460 / 1253, int8 per dim 1298 / 1285, ALT int8 per head 1050 / 986; exact K, two operands 1216 / 1490.
    static constexpr bool BLOCK = D == 64 || (KX && !ALT);
    static constexpr bool TAB = KX || VX;                     // per-key softmax tables
    static constexpr int TS = CTAS == 2 ? 8 : 16;             // table slots: more than PST + KST + SB tiles
    static constexpr int TAB_FLOATS = 4 * TC_N + 4;           // K scale, log2 V scale, 1 / V scale, K zero-point term; flag
    static constexpr int OFF_K = 0;
    static constexpr int OFF_V = OFF_K + KST * KT * T_BYTES;
    static constexpr int OFF_TAB = OFF_V + VST * T_BYTES;
    static constexpr int OFF_BAR = OFF_TAB + (TAB ? TS * TAB_FLOATS * 4 : 0);
    static constexpr int N_BARS = 38 + TS;
    static constexpr int OFF_MISC = OFF_BAR + N_BARS * 8;     // tmem base, abort flag
    static constexpr int OFF_PREF = OFF_MISC + 16;            // ParamRef [2]
    static constexpr int OFF_XCH = OFF_PREF + 2 * 48;         // float [4][QT * 128]: the two threads of a row, maxima and sums
    static constexpr int OFF_DYN = OFF_XCH + (HV == 2 ? 4 * QT * TC_M * 4 : 0);   // packed stages, records, step tables: sizes known at launch (TcDyn)
    // Queries that come in through shared memory: a warp reads contiguous pieces of rows and hands each lane its own (the V stages; the V converters
    // leave them alone until the queries are in place).  Every lane reading its row takes 32 sectors an instruction.  us per
    // call, lane by lane / so: head_dim 64, int8 B64 H16 256 x 680 155 / 149, int8 per dim B100 H16 228 / 217, int4 B64 H30 324 x 645 526 / 498, 16-bit
    // queries over exact int2 1044 x 505 85 / 80; head_dim 128, int8 per dim B16 H16 400 x 921 bf16 normalised 185 / 164, int8 per head B64 144 x 265 196 / 175.
    // Not so: 16-bit queries over a dequantised K, where the loop behind lost more to its changed schedule (c64 int2 group 32 1237 / 1278, c128 int8
    // 886 / 985), and up to 128 queries over grouped K at head_dim 64 (9 x 700 fp32 B48 H20 67 / 75, 100 x 255 B100 H16 68 / 74;
    // over 8, 4 and 2 bits, 32 to 1920 (sample, head) pairs, 17 to 128 queries and 121 to 5200 tokens it takes 1.02, 1.04 and 1.03 times as long on average: up to
    // 1.41 over long caches, 0.94 to 0.98 over two tiles of keys, 0.89 to 0.97 for 36 to 56 queries of 1280 pairs and more over 500 to 1800 tokens).
    static constexpr bool Q_STAGED = NQ == 2 ? D == 128 || QT == 2 || KM != PM_GROUP : D == 64 && KX;
    static constexpr int Q_STAGE = 32 * (D == 128 ? 144 : 80);           // bytes per softmax warp
    static_assert(K_WARP0 * Q_STAGE <= VST * T_BYTES, "query staging");
    static_assert(OFF_DYN % 16 == 0 && (OFF_TAB % 1024) == 0, "alignment");
    static_assert(QT * SB <= 4 && KST <= 3 && TS > PST + KST + SB, "barrier plan");
    // TMEM columns: queries, output accumulators, score tiles
    static constexpr int TMEM_COLS = CTAS == 2 ? 256 : 512;
    static constexpr int COL_Q = 0, COL_O = QT * NQ * D / 2, COL_S = COL_O + (ALT ? 2 : QT) * D;
    static_assert(COL_S + QT * SB * TC_N <= TMEM_COLS, "TMEM plan");
};
struct TcDyn {          // byte offsets of the launch-sized regions, from the aligned base of dynamic shared memory
    int pkk, pkv;       // packed rows: two stages each
    int krec, vrec;     // records: two stages each
    int ktab, vtab;     // step tables ...
    int k_rows, v_rows; // ... and the steps that they hold (PM_WINDOW: and one more row)
    int k_stage, v_stage, krec_stage, vrec_stage;
    int k_mode, v_mode;
    int k_bulk, v_bulk; // grouped parameters of consecutive tokens are contiguous and 16-byte aligned: bulk copies
};

// code - zp stays an exact fp16 integer and its product with the scale inside fp16's range
__device__ __forceinline__ bool par_in_bounds(float s, float z) { return fabsf(z) <= 512.f && s < 60.f; }
__device__ __forceinline__ uint32_t half_pair(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)) * 0x10001u; }
constexpr int STEPS_TO_MOVE = 16;                // a table moves for a tile of fewer steps (64 one-token steps per tile, us: 100 when it moved, 62 without)
constexpr uint32_t PAR_SLOW = 0x7e007e00u;        // NaN in place of a zero-point constant: the item takes the fp32 routine

// What the fp32 routine needs of a ParamView, with the (sample, head) part of the index folded into the pointers.
struct ParamRef {     // 40 bytes, kept in shared memory
    const float* scale;
    const float* zp;
    const int32_t* row_of_token;
    long long sr, sg;
    int group;
    __device__ __forceinline__ int row(int token) const { return row_of_token ? __ldg(row_of_token + token) : token; }
    __device__ __forceinline__ long long index(int r, int d) const { return r * sr + (long long)(d / group) * sg; }
};
__device__ __forceinline__ ParamRef param_ref(const ParamView& pv, int b, int h) {
    const long long base = pv.index(b, 0, h, 0);
    ParamRef r;
    r.scale = pv.scale + base;
    r.zp = pv.zp ? pv.zp + base : nullptr;
    r.row_of_token = pv.row_of_token;
    r.sr = pv.sr; r.sg = pv.sg; r.group = pv.group;
    return r;
}
// One item in fp32, parameters element by element: (code - zp) * scale as fp16 hi (+ lo when `lo_step` is not zero: the lo tile lies
// that many bytes behind).  Groupings without a faster mode, and parameters outside the packed-half arithmetic's bounds.
template <int BITS>
__device__ __noinline__ void slow_item(unsigned char* dst0, unsigned char* dst1, int lo_step, const uint32_t* words, const ParamRef* ref, int token, int d0) {
    constexpr int VPW = 32 / BITS;
    const ParamRef p = *ref;
    const int row = p.row(token);
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
        __half hh[8], hl[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int e = code_at(BITS, c * 8 + j);
            const long long pi = p.index(row, d0 + e);
            const float z = p.zp ? __ldg(p.zp + pi) : 0.f;
            const float v = ((float)(((int)(words[e / VPW] << (32 - BITS * (e % VPW + 1)))) >> (32 - BITS)) - z) * __ldg(p.scale + pi);
            hh[j] = __float2half_rn(v);
            hl[j] = __float2half_rn(v - __half2float(hh[j]));
        }
        unsigned char* dst = c ? dst1 : dst0;
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(hh);
        if (lo_step) *reinterpret_cast<uint4*>(dst + lo_step) = *reinterpret_cast<uint4*>(hl);
    }
}

// Packed-half arithmetic with (s_hi, s_lo), s_hi + s_lo = scale to 2^-22, on the exact integers d = code - zp:
//   k_hi = RN(d * s_hi),  k_lo = RN(d * s_lo + (d * s_hi - k_hi))      [the inner residual is exact in fp16]
// reproduce (code - zp) * scale to 2^-22; a single tile takes RN(d * s_hi + RN(d * s_lo)).
template <bool SPLIT>
__device__ __forceinline__ void scale_pair(uint32_t& d, uint32_t& lo, uint32_t sh, uint32_t sl) {
    if constexpr (SPLIT) {
        const uint32_t hi = h2_mul(d, sh);
        lo = h2_fma(d, sl, h2_fma(d, sh, h2_neg(hi)));
        d = hi;
    } else {
        d = h2_fma(d, sh, h2_mul(d, sl));
    }
}
template <int N> __device__ __forceinline__ void load_words(const uint32_t* p, uint32_t* w) {
    if constexpr (N == 4) { const uint4 v = *reinterpret_cast<const uint4*>(p); w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; }
    else if constexpr (N == 2) { const uint2 v = *reinterpret_cast<const uint2*>(p); w[0] = v.x; w[1] = v.y; }
    else w[0] = *p;
}
// The per-dim parameters of a thread's 16-wide head_dim slice, kept in registers while consecutive keys belong to one step
struct StepRegs { uint32_t sh[8], sl[8], nz[8]; int step; };
// Parameters of n steps from r0 on -> a table fp16 [n][3][D]: scale hi, scale lo, zero-point constant, in operand order (the
// zero-point constants of a 16-wide slice start with PAR_SLOW when one of its elements is out of bounds).  By nthr threads, a lane per
// element and eight elements' loads in flight: a CTA converts nothing before its table is there (a thread per slice, whose loads waited for one
// another: int8 per dim B100 H16 256 x 680 237 us, 221 so).
template <int D>
__device__ __forceinline__ void fill_steps(unsigned char* steptab, const ParamRef* ref, int r0, int n, int bits, int ptid, int nthr) {
    __half* tb = reinterpret_cast<__half*>(steptab);
    constexpr int U = 8;
    const int gs = __ffs(ref->group) - 1, lane = ptid & 31;       // the divisors of D are powers of two
#pragma unroll 1
    for (int e0 = ptid; e0 < n * D; e0 += U * nthr) {             // n * D elements: whole warps
        float sv[U], zv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = min(e0 + u * nthr, n * D - 32 + lane), row = r0 + e / D, d = e & (D - 1);
            const long long pi = row * ref->sr + (long long)(d >> gs) * ref->sg;
            sv[u] = __ldg(ref->scale + pi);
            zv[u] = ref->zp ? __ldg(ref->zp + pi) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * nthr, d = e & (D - 1), i = d & 15;
            if (e >= n * D) break;
            const int p = code_pos(bits, i), cls = p >> 1;
            const unsigned slow = __ballot_sync(0xffffffffu, !par_in_bounds(sv[u], zv[u])) >> (lane & 16) & 0xffffu;
            const float base = bits == 8 ? Item<8>::neg_base(0) : bits == 4 ? Item<4>::neg_base(cls & 1) : Item<2>::neg_base(cls & 3);
            const __half s_hi = __float2half_rn(sv[u]);
            __half* t = tb + (e / D) * 3 * D + (d & ~15) + p;
            t[0] = s_hi;
            t[D] = __float2half_rn(sv[u] - __half2float(s_hi));
            t[2 * D] = slow && p < 2 ? __ushort_as_half(PAR_SLOW & 0xffffu) : __float2half_rn(base - zv[u]);
        }
    }
}

// One operand tile by NTHR threads.  SPLIT: hi + lo tiles (K), otherwise one tile.  A thread keeps its head_dim slice and its place inside the
// swizzled rows (NTHR is a multiple of 8 keys' items), so its addresses advance by constants, and its packed words are all loaded before
// the first is used.  Rows past the keys are computed from whatever the stage holds; `zero` clears them (V: their P is zero, but 0 * NaN is not).
// An item is 16 codes of a key; with grouped parameters of narrow codes it is 32, which share a scale where the group has that many (the
// preparation of a scale is a third of a 16-code item's instructions).  Neighbouring lanes take the items of one key: contiguous reads, and
// a quarter-warp's 16-byte stores land in eight different bank groups; 32-code items do so when it takes two items of four keys.
template <int BITS, int D, int NTHR, int MODE, bool SPLIT>
__device__ __forceinline__ void convert_tile(unsigned char* tile, const unsigned char* packed, const unsigned char* rec, const unsigned char* steptab, StepRegs& sr,
                                             const ParamRef* ref, int mode, int n_valid, bool zero, int k0, int ptid, int gsh, int grp_shift, int zp_off, const CodeMagic<BITS>& cm) {
    constexpr int W = MODE == PM_GROUP && BITS < 8 ? 2 : 1;
    constexpr int IPK = D / (16 * W), NW = BITS / 2, NIT = TC_N * IPK / NTHR, KSTEP = NTHR / IPK;
    constexpr int LO = SPLIT ? TC_N * D * 2 : 0;
    constexpr int STEP_BYTES = KSTEP * 128;      // KSTEP keys further in the tile
    static_assert(TC_N * IPK % NTHR == 0 && KSTEP % 8 == 0, "items of a tile over the threads");
    const int item = W == 2 && IPK == 4 ? (ptid & 1) | (ptid >> 2 & 2) : ptid & (IPK - 1);
    const int key0 = W == 2 && IPK == 4 ? (ptid >> 1 & 3) | (ptid >> 2 & 4) | (ptid >> 5) * 8 : ptid / IPK, d0 = item * 16 * W;
    const uint32_t off0 = chunk_off(key0, 2 * W * item);
    auto dst = [&](int it, int ch) -> unsigned char* { return tile + (off0 ^ (uint32_t)(ch << 4)) + it * STEP_BYTES; };
    const uint32_t* src = reinterpret_cast<const uint32_t*>(packed) + (key0 * IPK + item) * (W * NW);
    uint32_t slow = 0;                       // 16-code slices to redo in fp32
    if (MODE == PM_GROUP && mode == PM_SLOW) {
        slow = (1u << (NIT * W)) - 1u;
    } else {
        uint32_t w[NIT][W * NW];
#pragma unroll
        for (int it = 0; it < NIT; ++it) load_words<W * NW>(src + it * NTHR * (W * NW), w[it]);
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int key = key0 + it * KSTEP;
            uint32_t sh = 0, sl = 0, nz[Item<BITS>::CLS];
            bool out = false;
#pragma unroll
            for (int u = 0; u < W; ++u) {
                uint32_t d[8], lo[8];
                Item<BITS>::raw(w[it] + u * NW, d, cm);
                if constexpr (MODE == PM_STEP) {
                    const int step = reinterpret_cast<const uint16_t*>(rec)[key];        // its slot in the table
                    if (step != sr.step) {
                        const uint4* t = reinterpret_cast<const uint4*>(steptab + (step * 3 * D + d0) * 2);
                        constexpr int TD = D * 2 / 16;      // uint4 per table row
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint4 a = t[i], b = t[TD + i], c = t[2 * TD + i];
                            sr.sh[4 * i] = a.x; sr.sh[4 * i + 1] = a.y; sr.sh[4 * i + 2] = a.z; sr.sh[4 * i + 3] = a.w;
                            sr.sl[4 * i] = b.x; sr.sl[4 * i + 1] = b.y; sr.sl[4 * i + 2] = b.z; sr.sl[4 * i + 3] = b.w;
                            sr.nz[4 * i] = c.x; sr.nz[4 * i + 1] = c.y; sr.nz[4 * i + 2] = c.z; sr.nz[4 * i + 3] = c.w;
                        }
                        sr.step = step;
                    }
                    if (sr.nz[0] == PAR_SLOW) slow |= 1u << it;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        d[i] = Item<BITS>::minus_zp(d[i], i, sr.nz[i]);
                        scale_pair<SPLIT>(d[i], lo[i], sr.sh[i], sr.sl[i]);
                    }
                } else if constexpr (MODE == PM_GROUP) {
                    if (u == 0 || grp_shift == 4) {
                        const float* par = reinterpret_cast<const float*>(rec) + (key << gsh) + ((d0 + 16 * u) >> grp_shift);
                        const float s = par[0], z = zp_off ? par[zp_off] : 0.f;
                        out = !par_in_bounds(s, z);
                        const __half s_hi = __float2half_rn(s);
                        sh = (uint32_t)__half_as_ushort(s_hi) * 0x10001u;
                        sl = half_pair(s - __half2float(s_hi));
                        Item<BITS>::spread(half_pair(Item<BITS>::neg_base(0) - z), nz);
                    }
                    if (out) slow |= 1u << (it * W + u);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        d[i] = Item<BITS>::minus_zp(d[i], i, nz[i % Item<BITS>::CLS]);
                        scale_pair<SPLIT>(d[i], lo[i], sh, sl);
                    }
                } else {
                    const uint32_t nz0 = reinterpret_cast<const uint32_t*>(rec)[key];
                    if (nz0 == PAR_SLOW) slow |= 1u << it;
                    Item<BITS>::spread(nz0, nz);
#pragma unroll
                    for (int i = 0; i < 8; ++i) d[i] = Item<BITS>::minus_zp(d[i], i, nz[i % Item<BITS>::CLS]);
                }
                sts128(dst(it, 2 * u), d[0], d[1], d[2], d[3]);
                sts128(dst(it, 2 * u + 1), d[4], d[5], d[6], d[7]);
                if constexpr (SPLIT) {
                    sts128(dst(it, 2 * u) + LO, lo[0], lo[1], lo[2], lo[3]);
                    sts128(dst(it, 2 * u + 1) + LO, lo[4], lo[5], lo[6], lo[7]);
                }
            }
        }
    }
    if (slow) {
#pragma unroll 1
        for (int e = 0; e < NIT * W; ++e) {
            const int it = e / W, u = e - it * W, key = key0 + it * KSTEP;
            if ((slow >> e & 1u) && key < n_valid)
                slow_item<BITS>(dst(it, 2 * u), dst(it, 2 * u + 1), LO, src + it * NTHR * (W * NW) + u * NW, ref, k0 + key, d0 + 16 * u);
        }
    }
    if (zero && n_valid < TC_N) {
#pragma unroll 1
        for (int it = 0; it < NIT; ++it)
            if (key0 + it * KSTEP >= n_valid) {
#pragma unroll
                for (int ch = 0; ch < 2 * W; ++ch) sts128(dst(it, ch), 0u, 0u, 0u, 0u);
            }
    }
}

// ---- softmax arithmetic
// A row keeps its reference until the weights of a tile add up to more than this: P stays below it in fp16 (largest finite value 65504)
// and the accumulators are rescaled rarely.
constexpr float TC_SUM_MAX = 32768.f;
constexpr float TC_LAZY = 12.f;       // the same for a maximum (log2 units)
constexpr float TC_VS_MIN = 9.5367431640625e-07f;     // 2^-20: smallest V scale folded into P as is
constexpr float TC_MASKED = -1e30f;
// |softmax scale| * log2(e) multiplies the scores; below this (a zero scale among them) it goes into the queries instead, so that
// a masked score stays masked
constexpr float TC_MIN_SCALE = 1e-18f;
__device__ __forceinline__ float tc_factor(float scale_log2) { const float c = fabsf(scale_log2); return c < TC_MIN_SCALE ? 1.f : c; }

// packed fp32 pairs (one instruction for two lanes of work on sm_100)
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0, float c1) {
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}
__device__ __forceinline__ void add2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float4 tab4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// d += the two halves of h
__device__ __forceinline__ void add_halves(float& d0, float& d1, uint32_t h) {
    asm("{\n\t.reg .f16 a, b;\n\tmov.b32 {a, b}, %2;\n\tadd.rn.f32.f16 %0, a, %0;\n\tadd.rn.f32.f16 %1, b, %1;\n\t}" : "+f"(d0), "+f"(d1) : "r"(h));
}
template <int N, int AT_LAUNCH> __device__ __forceinline__ void set_registers() {
    if constexpr (N > AT_LAUNCH) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
    else if constexpr (N < AT_LAUNCH) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int V> struct IntC { static constexpr int value = V; };

// 16 bytes of a query row from element `off` on (ES: bytes of an element); rows that do not lie on 16 bytes come element by element
template <int ES> __device__ __forceinline__ uint4 load_q16(const void* q, long long off) {
    const uintptr_t addr = reinterpret_cast<uintptr_t>(q) + (unsigned long long)off * ES;
    if ((addr & 15u) == 0) return __ldg(reinterpret_cast<const uint4*>(addr));
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if constexpr (ES == 4) w[i] = __ldg(reinterpret_cast<const uint32_t*>(addr) + i);
        else w[i] = (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(addr) + 2 * i) | (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(addr) + 2 * i + 1) << 16;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
// eight elements, as fp32
template <int ES> __device__ __forceinline__ void q8_floats(const uint4 (&r)[ES / 2], int dtype, float (&v)[8]) {
    if constexpr (ES == 4) {
        v[0] = __uint_as_float(r[0].x); v[1] = __uint_as_float(r[0].y); v[2] = __uint_as_float(r[0].z); v[3] = __uint_as_float(r[0].w);
        v[4] = __uint_as_float(r[1].x); v[5] = __uint_as_float(r[1].y); v[6] = __uint_as_float(r[1].z); v[7] = __uint_as_float(r[1].w);
    } else {
        const uint32_t w[4] = {r[0].x, r[0].y, r[0].z, r[0].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (dtype == VARQ_F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                v[2 * j] = f.x; v[2 * j + 1] = f.y;
            } else {                         // a bf16 is the upper half of an fp32
                v[2 * j] = __uint_as_float(w[j] << 16);
                v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
            }
        }
    }
}

template <int D, int NQ, int QT, int KM, int VM>
__global__ void __launch_bounds__(TcPlan<D, NQ, QT, KM, VM>::THREADS, TcPlan<D, NQ, QT, KM, VM>::CTAS) attn_tc_kernel(AttnArgs a, TcDyn dy, int kb, int vb) {
    using P = TcPlan<D, NQ, QT, KM, VM>;
    constexpr bool KX = P::KX, VX = P::VX;
    constexpr int KTHR = P::KTHR, VTHR = P::VTHR, MMA_WARP = P::MMA_WARP, SB = P::SB, HV = P::HV, KST = P::KST, VST = P::VST, PST = P::PST, TS = P::TS;
    constexpr int N = TC_N;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // swizzle atoms need 1024-byte alignment
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + P::OFF_BAR);
    // bars + 0, 1: [PM_WINDOW] the threads of a converter role, K and V, before and after their step table moves
    uint64_t* bar_pk = bars + 32;     // [PST] packed K rows (tx bytes) and records (load warp) of a tile in place
    uint64_t* bar_pv = bars + 35;     // [PST] the same for V
    uint64_t* bar_k = bars + 4;       // [KST] K operand tile written
    uint64_t* bar_v = bars + 7;       // [VST] V operand tile written
    uint64_t* bar_s = bars + 10;      // [QT][SB] S = Q K^T complete (tcgen05.commit)
    uint64_t* bar_p = bars + 14;      // [QT][SB] P written (the softmax threads that own real query rows)
    uint64_t* bar_o = bars + 18;      // [VST] O += P V complete (tcgen05.commit): V stage free
    uint64_t* bar_q = bars + 21;      // queries in tensor memory
    uint64_t* bar_end = bars + 22;    // all products complete
    uint64_t* bar_kf = bars + 24;     // [KST] every product that reads a K stage complete
    uint64_t* bar_sf = bars + 28;     // [SB] O += P V complete: the score columns are free (head_dim 128, where another warp issues S); QT = 2: [QT][2], the same
                                      // per query tile, for the softmax threads
    uint64_t* bar_t = bars + 38;      // [TS] softmax tables of tile i in place (slot i % TS)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + P::OFF_MISC);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + P::OFF_MISC + 4);

    const int tid = threadIdx.x, lane = tid & 31;
    // the warp index through a shuffle: the compiler then knows that it is the same in every lane, keeps the role branches
    // uniform and can hold addresses, descriptors and loop counters of a role in uniform registers
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // query tile fastest: the tiles of one (sample, head) run together and share its packed rows in L2
    const unsigned blk = blockIdx.x;
    const int qt = (int)(blk % (unsigned)a.n_qtiles);
    const int split = (int)((blk / (unsigned)a.n_qtiles) % (unsigned)a.splits);
    const int bh = (int)(blk / ((unsigned)a.n_qtiles * (unsigned)a.splits)), b = bh / a.H, h = bh - b * a.H;
    const int q0 = qt * (QT * TC_M);
    const int nq = min(QT * TC_M, a.Lq - q0);
    const int n_qt = QT == 1 ? 1 : (nq + TC_M - 1) / TC_M;                 // query tiles that hold real queries
    const int t0 = split * a.tiles_per_split;                              // first key tile of this CTA
    const int T = min(a.tiles_per_split, (a.Lk + N - 1) / N - t0);         // and how many
    auto tile_n = [&](int i) -> int { return min(N, a.Lk - (t0 + i) * N); };
    // the steps [x, y) that a step table starts with: from the first tile's on, as many as are known and fit
    auto first_steps = [&](const ParamView& pv, int tab_rows) {
        const int r = t0 == 0 ? 0 : pv.row(t0 * N);
        return make_int2(r, max(r, min(r + tab_rows, pv.n_rows)));
    };
    const int aq = (nq + 31) >> 5;                  // blocks of 32 rows that hold real queries, ...
    const int aq0 = min(aq, 4), aq1 = max(aq - 4, 0);    // ... per query tile

    if (warp == 0) {
        for (int i = lane; i < P::N_BARS; i += 32) {
            const uint32_t count = i >= 32 && i < 38 ? 33u : i == 1 ? (uint32_t)VTHR : i < 4 + 3 ? (uint32_t)KTHR : i < 10 ? (uint32_t)VTHR
                                 : i >= 14 && i < 18 ? (uint32_t)(32 * (P::ALT ? 1 : HV) * max(1, i - 14 < SB ? aq0 : aq1)) : i == 21 ? (uint32_t)(32 * HV * aq)
                                 : (i >= 18 && i < 21) || i == 22 || (i >= 24 && i < 27) ? (uint32_t)n_qt : i >= 38 ? 64u : 1u;
            mbar_init(&bars[i], count);
        }
        if (lane == 0) *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {   // TMEM allocation by one full warp
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)P::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pdl_wait();          // global memory is touched from here on only
    if (tid == P::K_WARP0 * 32) *reinterpret_cast<ParamRef*>(smem + P::OFF_PREF) = param_ref(a.kp, b, h);
    if (tid == P::V_WARP0 * 32) *reinterpret_cast<ParamRef*>(smem + P::OFF_PREF + 48) = param_ref(a.vp, b, h);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_trigger();       // behind the allocation: a CTA of a next launch must not take tensor memory that one of this launch still asks for
    const uint32_t tmem_base = *tmem_slot;

    if (warp < P::K_WARP0) {
        // =============================================================== softmax / epilogue
        set_registers<P::REGS_SOFT, P::REGS>();
        // Two threads share a query row at head_dim 128 (TcPlan::ALT says how): four (two) softmax warps per SM sub-partition keep the
        // exponential unit busy where one warp alone leaves it idle half of the time.  Without ALT the pair (two warps of one sub-partition)
        // agrees on the reference maximum by one barrier-with-reduction per tile.
        constexpr bool ALT = P::ALT;
        constexpr int NC = ALT ? N : N / HV, DH = D / HV;       // score columns and (queries, epilogue) head_dim values of a thread
        const int t = QT == 1 ? 0 : warp / (4 * HV), half = HV == 1 ? 0 : (warp >> 2) & 1, quarter = warp & 3;
        if (quarter < (t ? aq1 : aq0)) {
            const int r = t * TC_M + quarter * 32 + lane;       // query row of the CTA; TMEM lane = r % 128
            const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
            const uint32_t col_q = P::COL_Q + t * (NQ * D / 2), col_o = P::COL_O + t * D, col_s = P::COL_S + t * (SB * N);
            const bool live = r < nq;
            float* xch = reinterpret_cast<float*>(smem + P::OFF_XCH) + r;
            constexpr int XH = QT * TC_M;
            const int bar_id = 3 + t * 4 + quarter;
            auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(bar_id) : "memory"); };
            auto pair_any = [&](bool flag) -> bool {
                if (HV == 1 || ALT) return __any_sync(0xffffffffu, flag) != 0;
                uint32_t any;
                asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, %2, 64, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                             : "=r"(any) : "r"((uint32_t)flag), "r"(bar_id) : "memory");
                return any != 0;
            };
            auto pair_sum = [&](float v) -> float {      // both threads of a row get the sum of their values
                if (HV == 1) return v;
                xch[(2 + half) * XH] = v;
                pair_sync();
                const float w = v + xch[(2 + (half ^ 1)) * XH];
                pair_sync();
                return w;
            };
            // ---- queries -> tensor memory as fp16 hi [, lo]; the sign of the softmax scale goes with them
            float qsum = 0.f;
            {
                const long long q_own = b * a.qs_b + (long long)(q0 + (live ? r : 0)) * a.qs_l + h * a.qs_h + half * DH;
                const long long q_first = b * a.qs_b + (long long)q0 * a.qs_l + h * a.qs_h + half * DH;
                unsigned char* stage = smem + P::OFF_V + warp * P::Q_STAGE;
                float mul = a.scale_log2 < 0.f ? -1.f : 1.f;
                if (fabsf(a.scale_log2) < TC_MIN_SCALE) mul *= fabsf(a.scale_log2);
                // values of a row -> fp16 pairs in the order of the operands
                auto pack = [&](auto bits_c, auto n_c, const float* v, uint32_t* hi, uint32_t* lo) {
#pragma unroll
                    for (int e = 0; e < decltype(n_c)::value / 2; ++e) {
                        float y[2];
#pragma unroll
                        for (int z = 0; z < 2; ++z) {      // the operand is fp16: an element beyond its range saturates instead of becoming infinite
                            const int d = ((2 * e) & ~15) + code_at(decltype(bits_c)::value, (2 * e + z) & 15);
                            y[z] = fminf(fmaxf(v[d] * mul, -65504.f), 65504.f);
                        }
                        const __half2 hh = __floats2half2_rn(y[0], y[1]);
                        const float2 hf = __half22float2(hh);
                        hi[e] = *reinterpret_cast<const uint32_t*>(&hh);
                        if constexpr (NQ == 2) {
                            const __half2 hl = __floats2half2_rn(y[0] - hf.x, y[1] - hf.y);
                            lo[e] = *reinterpret_cast<const uint32_t*>(&hl);
                            if constexpr (KX) qsum += y[0] + y[1];
                        } else if constexpr (KX) qsum += hf.x + hf.y;
                    }
                };
                if constexpr (P::Q_STAGED && D == 128) {
                    // 128 bytes of a row at a time (a thread's half of a 16-bit row whole, read once even where it is normalised), and no more in registers than
                    // 16 values and their halves: with 32, and the next ones under way, every kernel of two operands spilled 164 to 312 bytes.  Calls whose
                    // only key tile hardly fills take 0.3 us longer than lane by lane (33 x 40 fp32 H20: 6.4 / 6.7 us).
                    const bool wide_q = a.q_dtype == VARQ_F32;
                    const int piece = wide_q ? 32 : 64;
                    auto stage_at = [&](int row, int ch) -> uint4* { return reinterpret_cast<uint4*>(stage + row * 144 + ch * 16); };
                    auto each16 = [&](bool staged, auto body) {      // body(head_dim value, 16 values from there on)
#pragma unroll 1
                        for (int c0 = 0; c0 < DH; c0 += piece) {
                            if (!staged) {
                                uint4 raw[8];
#pragma unroll
                                for (int p = 0; p < 8; ++p) {
                                    const int row = quarter * 32 + p * 4 + lane / 8;
                                    const long long off = q_first + (long long)(row < nq ? row : 0) * a.qs_l + c0;
                                    raw[p] = wide_q ? load_q16<4>(a.q, off + (lane & 7) * 4) : load_q16<2>(a.q, off + (lane & 7) * 8);
                                }
                                __syncwarp();
#pragma unroll
                                for (int p = 0; p < 8; ++p) *stage_at(p * 4 + lane / 8, lane & 7) = raw[p];
                                __syncwarp();
                            }
#pragma unroll 1
                            for (int u = 0; u < piece; u += 16) {
                                float v[16];
                                if (wide_q) {
#pragma unroll
                                    for (int e = 0; e < 4; ++e) {
                                        const uint4 w = *stage_at(lane, u / 4 + e);
                                        v[4 * e] = __uint_as_float(w.x); v[4 * e + 1] = __uint_as_float(w.y); v[4 * e + 2] = __uint_as_float(w.z); v[4 * e + 3] = __uint_as_float(w.w);
                                    }
                                } else {
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        const uint4 w[1] = {*stage_at(lane, u / 8 + e)};
                                        q8_floats<2>(w, a.q_dtype, *reinterpret_cast<float (*)[8]>(v + 8 * e));
                                    }
                                }
                                body(c0 + u, v);
                            }
                        }
                    };
                    bool staged = false;
                    if (a.q_norm) {       // x / max(||x||_2, eps) * scale_mul[h], on the way in
                        float ss = 0.f;
                        each16(false, [&](int, const float* v) {
#pragma unroll
                            for (int e = 0; e < 16; ++e) ss = fmaf(v[e], v[e], ss);
                        });
                        ss = pair_sum(ss);
                        mul *= (a.q_mul ? __ldg(a.q_mul + h) : 1.f) / fmaxf(sqrtf(ss), a.q_eps);
                        staged = !wide_q;
                    }
                    if (!live) mul = 0.f;
                    each16(staged, [&](int c, const float* v) {
                        uint32_t hi[8], lo[8];
                        if (kb == 8) pack(IntC<8>(), IntC<16>(), v, hi, lo); else if (kb == 4) pack(IntC<4>(), IntC<16>(), v, hi, lo); else pack(IntC<2>(), IntC<16>(), v, hi, lo);
                        tmem_st8(lane_base + col_q + (half * DH + c) / 2, hi);
                        tmem_st8(lane_base + col_q + D / 2 + (half * DH + c) / 2, lo);
                    });
                } else {
                    uint4 raw[8];
                    auto fetch = [&](auto es_c, int c0) {
                        constexpr int ES = decltype(es_c)::value;       // bytes of an element = lanes of a row segment of 16 elements
#pragma unroll
                        for (int p = 0; p < 2 * ES; ++p) {
                            const int row = t * TC_M + quarter * 32 + (p & (ES - 1)) * (32 / ES) + lane / ES;
                            raw[p] = load_q16<ES>(a.q, q_first + (long long)(row < nq ? row : 0) * a.qs_l + c0 + (p / ES) * 16 + (lane & (ES - 1)) * (16 / ES));
                        }
                    };
                    auto spread = [&](auto es_c, float (&v)[4][8]) {
                        constexpr int ES = decltype(es_c)::value, PITCH = 16 * ES + 16;
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            __syncwarp();
#pragma unroll
                            for (int p = 0; p < ES; ++p) *reinterpret_cast<uint4*>(stage + (p * (32 / ES) + lane / ES) * PITCH + (lane & (ES - 1)) * 16) = raw[u * ES + p];
                            __syncwarp();
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                uint4 w[ES / 2];
#pragma unroll
                                for (int p = 0; p < ES / 2; ++p) w[p] = *reinterpret_cast<const uint4*>(stage + lane * PITCH + (e * (ES / 2) + p) * 16);
                                q8_floats<ES>(w, a.q_dtype, v[2 * u + e]);
                            }
                        }
                    };
                    auto rows_at = [&](int c0, float (&v)[4][8]) {      // 32 head_dim values from c0 on; the next ones are requested
                        if constexpr (!P::Q_STAGED) {
#pragma unroll
                            for (int u = 0; u < 4; ++u) load_q8(a.q, a.q_dtype, q_own + c0 + 8 * u, v[u]);
                            return;
                        }
                        const int next = c0 + 32;
                        if (a.q_dtype == VARQ_F32) { if (c0 == 0) fetch(IntC<4>(), 0); spread(IntC<4>(), v); if (next < DH) fetch(IntC<4>(), next); }
                        else { if (c0 == 0) fetch(IntC<2>(), 0); spread(IntC<2>(), v); if (next < DH) fetch(IntC<2>(), next); }
                    };
                    if (a.q_norm) {       // x / max(||x||_2, eps) * scale_mul[h], on the way in
                        float ss = 0.f;
#pragma unroll 1
                        for (int c0 = 0; c0 < DH; c0 += 32) {
                            float v[4][8];
                            rows_at(c0, v);
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int e = 0; e < 8; ++e) ss = fmaf(v[u][e], v[u][e], ss);
                        }
                        ss = pair_sum(ss);
                        mul *= (a.q_mul ? __ldg(a.q_mul + h) : 1.f) / fmaxf(sqrtf(ss), a.q_eps);
                    }
                    if (!live) mul = 0.f;
#pragma unroll 1
                    for (int c0 = 0; c0 < DH; c0 += 32) {
                        float v[4][8];
                        rows_at(c0, v);
                        uint32_t hi[16], lo[16];
                        if (kb == 8) pack(IntC<8>(), IntC<32>(), &v[0][0], hi, lo); else if (kb == 4) pack(IntC<4>(), IntC<32>(), &v[0][0], hi, lo); else pack(IntC<2>(), IntC<32>(), &v[0][0], hi, lo);
                        tmem_st16(lane_base + col_q + (half * DH + c0) / 2, hi);
                        if constexpr (NQ == 2) tmem_st16(lane_base + col_q + D / 2 + (half * DH + c0) / 2, lo);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(bar_q);
                if constexpr (KX) qsum = pair_sum(qsum);
            }
            const float c = tc_factor(a.scale_log2);
            float m_used = -FLT_MAX;                            // reference (log2 domain): with ALT the thread's own, else the same in both threads of a row
            float l0 = 0.f, l1 = 0.f, l2 = 0.f, l3 = 0.f;       // row sum of this thread's softmax weights
            bool ok = true;
            const int first_col = ALT ? 0 : half * NC;          // of the tile's score columns
            const uint32_t col_acc = lane_base + col_o + (ALT ? half * D : 0);
            constexpr int STEP = ALT ? 2 : 1;
            // scores and tables of a tile in place?  Asked for the next tile while P of this one is on its way: the answer takes 130 cycles
            auto tile_ready = [&](int i) -> bool {
                const bool r = mbar_test(&bar_s[t * SB + i % SB], (i / SB) & 1);
                return P::TAB ? mbar_test(&bar_t[i % TS], (i / TS) & 1) && r : r;
            };
            bool ready = false;
            constexpr bool block = P::BLOCK;
            // The reference becomes `mt` (log2 domain) where that is higher, and what has been accumulated is rescaled (a factor 1 for the other rows)
            auto move_reference = [&](int i, float mt, float margin) -> bool {
                if (HV == 2 && !ALT) {
                    xch[half * XH] = mt;
                    pair_sync();
                    mt = fmaxf(mt, xch[(half ^ 1) * XH]);
                }
                const float m_new = mt > m_used + margin ? mt : m_used;
                const float alpha = ex2(m_used - m_new);    // 0 for a row without a reference yet
                const bool moved = !block || __any_sync(0xffffffffu, m_new > m_used);       // (the same in the other warp of a pair)
                m_used = m_new;
                l0 *= alpha; l1 *= alpha; l2 *= alpha; l3 *= alpha;
                if (i < STEP || !moved) return true;
                // The accumulator is stable.  With two query tiles bar_o waits for both, and the other may be so far behind that the parity
                // of an earlier phase answers: each has barriers of its own.
                const int o = i - STEP;
                ok = ok && (QT == 2 ? mbar_wait(&bar_sf[2 * t + (o & 1)], (o >> 1) & 1, abort_flag, 13) : mbar_wait(&bar_o[o % VST], (o / VST) & 1, abort_flag, 13));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) return false;
                tc_fence_after();
#pragma unroll 1
                for (int c0 = ALT ? 0 : half * DH; c0 < (ALT ? D : (half + 1) * DH); c0 += 16) {
                    uint32_t acc[16];
                    tmem_ld16(col_acc + c0, acc);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[j] = __float_as_uint(__uint_as_float(acc[j]) * alpha);
                    tmem_st16(col_acc + c0, acc);
                }
                tmem_wait_st();
                return true;
            };
            bool behind = true;        // (block) the reference has to follow this tile's scores before its P is computed
            // Once a wait has expired nothing is read or written any more, but a pair's barriers are still taken: without ALT both warps
            // run all iterations.
#pragma unroll 1
            for (int i = ALT ? half : 0; i < T;) {
                const int s = i % SB;
                if (!__all_sync(0xffffffffu, ready)) {
                    ok = ok && mbar_wait_warp(&bar_s[t * SB + s], (i / SB) & 1, abort_flag, 11);
                    if (P::TAB) ok = ok && mbar_wait_warp(&bar_t[i % TS], (i / TS) & 1, abort_flag, 12);
                    if (!ok) {
                        if (HV == 1 || ALT) break;
                        if constexpr (block) {
                            if (behind) pair_sync();
                            const bool again = pair_any(false), retry = again && !behind;
                            behind = again;
                            if (!retry) i += STEP;
                        } else {
                            if (pair_any(false)) pair_sync();
                            i += STEP;
                        }
                        continue;
                    }
                }
                const uint32_t s_addr = lane_base + col_s + s * N;
                const float* tab = reinterpret_cast<const float*>(smem + P::OFF_TAB) + (i % TS) * P::TAB_FLOATS + first_col;
                uint32_t x[NC], ph[NC / 2];
                const int nv = tile_n(i) - first_col;
                const bool wide = KX && __float_as_int(tab[4 * N - first_col]) != 0;        // a zero-point of this tile is too wide for the exact operand: its term in fp32
                tc_fence_after();
                tmem_ld32(s_addr + first_col, x);
                if constexpr (NC == 64) tmem_ld32(s_addr + 32, x + 32);
                tmem_wait_ld();
                if (wide || nv < NC) {          // and columns past the cache (the last tile) hold anything
#pragma unroll
                    for (int j = 0; j < NC; ++j) {
                        if (wide) x[j] = __float_as_uint(fmaf(-tab[3 * N + j], qsum, __uint_as_float(x[j])));
                        if (j >= nv) x[j] = __float_as_uint(TC_MASKED);
                    }
                }
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                auto to_half = [&](int j, const float (&y)[4]) {
                    const __half2 h01 = __floats2half2_rn(ex2(y[0]), ex2(y[1])), h23 = __floats2half2_rn(ex2(y[2]), ex2(y[3]));
                    ph[j / 2] = *reinterpret_cast<const uint32_t*>(&h01);
                    ph[j / 2 + 1] = *reinterpret_cast<const uint32_t*>(&h23);
                };
                // The row sum adds up the rounded P that multiplies V, so that a row dominated by one key stays exact
                auto sum_up = [&](int j) {
                    if constexpr (VX) {       // P carries the V scale: the softmax weight is P / V scale
                        const float4 v4 = tab4(tab + 2 * N + j);
                        const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&ph[j / 2])), f23 = __half22float2(*reinterpret_cast<const __half2*>(&ph[j / 2 + 1]));
                        fma2(s0, s1, f01.x, f01.y, v4.x, v4.y, s0, s1);
                        fma2(s2, s3, f23.x, f23.y, v4.z, v4.w, s2, s3);
                    } else {
                        add_halves(s0, s1, ph[j / 2]);
                        add_halves(s2, s3, ph[j / 2 + 1]);
                    }
                };
                auto store_p = [&]() {
                    if constexpr (NC == 64) tmem_st32(s_addr, ph); else tmem_st16(s_addr + half * 16, *reinterpret_cast<uint32_t (*)[16]>(ph));
                };
                // ---- P = 2^(score - reference), with the V scale where V keeps exact codes: fp16 pairs.
                if constexpr (!block) {
                    // The maximum first and the sum behind the store of P.  Nothing of it may move up into the waits for the scores (ALT, B8 H16 Lq2048 Lk4096
                    // int8: 872 us, 910 us where it did).
                    asm volatile("" ::: "memory");
                    float ma = -FLT_MAX, mb = -FLT_MAX;
#pragma unroll
                    for (int j = 0; j < NC; j += 4) {
                        if constexpr (P::TAB) {
                            const float4 k4 = KX ? tab4(tab + j) : make_float4(c, c, c, c), b4 = VX ? tab4(tab + N + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                            float y[4];
                            fma2(y[0], y[1], __uint_as_float(x[j]), __uint_as_float(x[j + 1]), k4.x, k4.y, b4.x, b4.y);
                            fma2(y[2], y[3], __uint_as_float(x[j + 2]), __uint_as_float(x[j + 3]), k4.z, k4.w, b4.z, b4.w);
#pragma unroll
                            for (int e = 0; e < 4; ++e) x[j + e] = __float_as_uint(y[e]);
                        }
                        ma = max3(ma, __uint_as_float(x[j]), __uint_as_float(x[j + 1]));
                        mb = max3(mb, __uint_as_float(x[j + 2]), __uint_as_float(x[j + 3]));
                    }
                    const float mt = fmaxf(ma, mb) * (P::TAB ? 1.f : c);
                    // (the vote: both threads of a row have read their scores before either stores P over them)
                    if (pair_any(mt > m_used + TC_LAZY) && !move_reference(i, mt, TC_LAZY)) { i += STEP; continue; }
                    const float nm = -m_used;
#pragma unroll
                    for (int j = 0; j < NC; j += 4) {
                        float y[4];
                        if constexpr (P::TAB) {
                            add2(y[0], y[1], __uint_as_float(x[j]), __uint_as_float(x[j + 1]), nm, nm);
                            add2(y[2], y[3], __uint_as_float(x[j + 2]), __uint_as_float(x[j + 3]), nm, nm);
                        } else {
                            fma2(y[0], y[1], __uint_as_float(x[j]), __uint_as_float(x[j + 1]), c, c, nm, nm);
                            fma2(y[2], y[3], __uint_as_float(x[j + 2]), __uint_as_float(x[j + 3]), c, c, nm, nm);
                        }
                        to_half(j, y);
                    }
                    store_p();
#pragma unroll
                    for (int j = 0; j < NC; j += 4) sum_up(j);
                } else {
                    const bool settled = behind;       // (both threads of a row have read their scores before either stores P over them: here and where they vote below)
                    if (behind) {
                        // The first tile, and where some row of these warps meets scores far above its reference
                        float mt = -FLT_MAX;
#pragma unroll
                        for (int j = 0; j < NC; j += 4) {
                            const float4 k4 = KX ? tab4(tab + j) : make_float4(c, c, c, c), b4 = VX ? tab4(tab + N + j) : make_float4(0.f, 0.f, 0.f, 0.f);
                            mt = max3(mt, fmaf(__uint_as_float(x[j]), k4.x, b4.x), fmaf(__uint_as_float(x[j + 1]), k4.y, b4.y));
                            mt = max3(mt, fmaf(__uint_as_float(x[j + 2]), k4.z, b4.z), fmaf(__uint_as_float(x[j + 3]), k4.w, b4.w));
                        }
                        if (!move_reference(i, mt, 0.f)) { behind = pair_any(false); ready = false; i += STEP; continue; }      // (the vote of the other warp's tile)
                    }
                    // One block of straight code: the exponential unit takes most of it, everything else fits in between
                    const float nm = -m_used;
#pragma unroll
                    for (int j = 0; j < NC; j += 4) {
                        const float4 k4 = KX ? tab4(tab + j) : make_float4(c, c, c, c);
                        float b0 = nm, b1 = nm, b2 = nm, b3 = nm, y[4];
                        if constexpr (VX) {
                            const float4 b4 = tab4(tab + N + j);
                            add2(b0, b1, b4.x, b4.y, nm, nm);
                            add2(b2, b3, b4.z, b4.w, nm, nm);
                        }
                        fma2(y[0], y[1], __uint_as_float(x[j]), __uint_as_float(x[j + 1]), k4.x, k4.y, b0, b1);
                        fma2(y[2], y[3], __uint_as_float(x[j + 2]), __uint_as_float(x[j + 3]), k4.z, k4.w, b2, b3);
                        to_half(j, y);
                        sum_up(j);
                    }
                    // P has room up to 65504: the sum of the tile's weights shows that none came close, without their maximum.  V scales: below the limit
                    // the largest of the tile may meet the heaviest weight.  Where heavy keys have far smaller ones the sum passes the limit and the
                    // reference stays: the next tile then begins with its maximum, and only the first of such tiles is computed twice (scales 10^4
                    // apart, B16 H16 256 x 2048 fp32, us: c64 173 when all were, 117 so, 90 with even scales; c128 298, 206, 164).
                    const float limit = VX ? tab[4 * N + 1 - first_col] : TC_SUM_MAX;
                    const bool again = pair_any(!((s0 + s1) + (s2 + s3) <= limit)), retry = again && !settled;
                    behind = again;
                    if (retry) { ready = true; continue; }
                    store_p();
                }
                l0 += s0; l1 += s1; l2 += s2; l3 += s3;
                i += STEP;
                ready = block && i < T && tile_ready(i);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bar_p[t * SB + s]);
            }
            // ---- output row: each thread writes half of its head_dim
            // (ALT) the accumulators of the two threads meet: f0 and f1 bring tiles of even and odd index to the common reference (0 where
            // a thread had no tile; the second accumulator is then not read either).
            float l = (l0 + l1) + (l2 + l3), f0 = 1.f, f1 = 0.f;
            if constexpr (!ALT) l = pair_sum(l);
            else {
                xch[half * XH] = m_used;
                pair_sync();
                const float m0 = xch[0], m1 = xch[XH];
                m_used = fmaxf(m0, m1);
                f0 = ex2(m0 - m_used);
                f1 = ex2(m1 - m_used);
                l = pair_sum(l * (half ? f1 : f0));
            }
            ok = ok && mbar_wait(bar_end, 0, abort_flag, 14);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                tc_fence_after();
                const float inv = a.splits == 1 ? 1.f / l : 1.f;
                const int row_slot = (int)blk * (QT * TC_M) + r;
                if (a.splits > 1 && live && half == 0) { a.ws[2 * (long long)row_slot] = m_used; a.ws[2 * (long long)row_slot + 1] = l; }
#pragma unroll 1
                for (int c0 = half * DH; c0 < (half + 1) * DH; c0 += 32) {
                    uint32_t o[32];
                    tmem_ld32(lane_base + col_o + c0, o);
                    tmem_wait_ld();
                    if constexpr (ALT) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f0);
                        if (T > 1) {
#pragma unroll
                            for (int u = 0; u < 32; u += 16) {
                                uint32_t o1[16];
                                tmem_ld16(lane_base + col_o + D + c0 + u, o1);
                                tmem_wait_ld();
#pragma unroll
                                for (int j = 0; j < 16; ++j) o[u + j] = __float_as_uint(fmaf(__uint_as_float(o1[j]), f1, __uint_as_float(o[u + j])));
                            }
                        }
                    }
                    if (live) {
                        auto put = [&](auto bits_c) {
                            float v[32];
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[(j & ~15) + code_at(decltype(bits_c)::value, j & 15)] = __uint_as_float(o[j]) * inv;
                            if (a.splits == 1) store_o_row32(a.out, a.o_dtype, b * a.os_b + (long long)(q0 + r) * a.os_l + h * a.os_h + c0, v);
                            else {
                                float4* dst = reinterpret_cast<float4*>(a.ws + 2 * (long long)gridDim.x * (QT * TC_M) + (long long)row_slot * D + c0);
#pragma unroll
                                for (int j = 0; j < 8; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            }
                        };
                        if (vb == 8) put(IntC<8>()); else if (vb == 4) put(IntC<4>()); else put(IntC<2>());
                    }
                }
            }
            tc_fence_before();
        }
    } else if (warp < MMA_WARP) {
        // =============================================================== converters
        set_registers<P::REGS_CONV, P::REGS>();
        const bool is_k = warp < P::V_WARP0;
        const int ptid = is_k ? tid - P::K_WARP0 * 32 : tid - P::V_WARP0 * 32;
        const ParamRef* ref = reinterpret_cast<const ParamRef*>(smem + P::OFF_PREF + (is_k ? 0 : 48));
        const int mode = is_k ? dy.k_mode : dy.v_mode, bits = is_k ? kb : vb;
        unsigned char* steptab = smem + (is_k ? dy.ktab : dy.vtab);
        if ((is_k ? KM : VM) == PM_STEP) {
            fill_steps<D>(steptab, ref, 0, is_k ? a.kp.n_rows : a.vp.n_rows, bits, ptid, is_k ? KTHR : VTHR);
            if (is_k) asm volatile("bar.sync 1, %0;" ::"n"(KTHR) : "memory");
            else asm volatile("bar.sync 2, %0;" ::"n"(VTHR) : "memory");
        }
        if ((is_k ? KM : VM) == PM_WINDOW) {       // the steps of the first tiles, and the row of the keys whose step is not there: their items take the fp32 routine
            const int rows = is_k ? dy.k_rows : dy.v_rows, nthr = is_k ? KTHR : VTHR;
            const int2 w = first_steps(is_k ? a.kp : a.vp, rows);
            fill_steps<D>(steptab, ref, w.x, w.y - w.x, bits, ptid, nthr);
            for (int d = ptid; d < D / 2; d += nthr) reinterpret_cast<uint32_t*>(steptab + (rows * 3 + 2) * D * 2)[d] = PAR_SLOW;
            if (is_k) asm volatile("bar.sync 1, %0;" ::"n"(KTHR) : "memory");
            else asm volatile("bar.sync 2, %0;" ::"n"(VTHR) : "memory");
        }
        const int group = is_k ? a.kp.group : a.vp.group, ng = D / group;
        const int gsh = __ffs(ng) - 1, grp_shift = __ffs(group) - 1;
        const int zp_off = (is_k ? a.kp.zp : a.vp.zp) ? N * ng : 0;       // raw zero-points behind the raw scales of a tile
        StepRegs sr;
        sr.step = -1;
        // A tile whose steps are not in the table: the load warp says which steps take their place.  All threads of the role meet before, when
        // they are through with the old ones, and after; on barriers with a limit, because a thread whose wait has expired does not come.
        auto move_table = [&](const int2 w, uint64_t* bar, int nthr) -> bool {
            mbar_arrive(bar);
            if (!mbar_wait(bar, 0, abort_flag, 25)) return false;
            fill_steps<D>(steptab, ref, w.x, w.y, bits, ptid, nthr);
            mbar_arrive(bar);
            sr = StepRegs{};
            sr.step = -1;
            return mbar_wait(bar, 1, abort_flag, 26);
        };
        if (is_k) {
            auto loop = [&](auto bits_c) {
                constexpr int BITS = decltype(bits_c)::value;
                CodeMagic<BITS> cm;
                cm.init();
#pragma unroll 1
                for (int i = 0; i < T; ++i) {
                    const int ps = i % PST, ks = i % KST;
                    bool ok = mbar_wait(&bar_pk[ps], (i / PST) & 1, abort_flag, 21);
                    if (ok && i >= KST) ok = mbar_wait(&bar_kf[ks], ((i - KST) / KST) & 1, abort_flag, 22);    // K stage is free
                    if (!ok) break;
                    const unsigned char* rec = smem + dy.krec + ps * dy.krec_stage;
                    if constexpr (KM == PM_WINDOW) {
                        const int2 w = *reinterpret_cast<const int2*>(rec + N * 2);
                        if (w.y > 0 && !move_table(w, &bars[0], KTHR)) break;
                    }
                    convert_tile<BITS, D, KTHR, KM == PM_WINDOW ? PM_STEP : KM, !KX>(smem + P::OFF_K + ks * P::KT * P::T_BYTES, smem + dy.pkk + ps * dy.k_stage, rec,
                                                         steptab, sr, ref, mode, tile_n(i), false, (t0 + i) * N, ptid, gsh, grp_shift, zp_off, cm);
                    fence_async_smem();
                    mbar_arrive(&bar_k[ks]);
                }
            };
            if (bits == 8) loop(IntC<8>()); else if (bits == 4) loop(IntC<4>()); else loop(IntC<2>());
        } else {
            auto loop = [&](auto bits_c) {
                constexpr int BITS = decltype(bits_c)::value;
                CodeMagic<BITS> cm;
                cm.init();
#pragma unroll 1
                for (int i = 0; i < T; ++i) {
                    const int ps = i % PST, vs = i % VST;
                    bool ok = (!P::Q_STAGED || i > 0 || mbar_wait(bar_q, 0, abort_flag, 27)) && mbar_wait(&bar_pv[ps], (i / PST) & 1, abort_flag, 23);
                    if (ok && i >= VST) ok = mbar_wait(&bar_o[vs], ((i - VST) / VST) & 1, abort_flag, 24);    // V stage is free
                    if (!ok) break;
                    const unsigned char* rec = smem + dy.vrec + ps * dy.vrec_stage;
                    if constexpr (VM == PM_WINDOW) {
                        const int2 w = *reinterpret_cast<const int2*>(rec + N * 2);
                        if (w.y > 0 && !move_table(w, &bars[1], VTHR)) break;
                    }
                    convert_tile<BITS, D, VTHR, VM == PM_WINDOW ? PM_STEP : VM, false>(smem + P::OFF_V + vs * P::T_BYTES, smem + dy.pkv + ps * dy.v_stage, rec,
                                                           steptab, sr, ref, mode, tile_n(i), true, (t0 + i) * N, ptid, gsh, grp_shift, zp_off, cm);
                    fence_async_smem();
                    mbar_arrive(&bar_v[vs]);
                }
            };
            if (bits == 8) loop(IntC<8>()); else if (bits == 4) loop(IntC<4>()); else loop(IntC<2>());
        }
    } else if (set_registers<P::REGS_MISC, P::REGS>(), warp < P::LOAD_WARP) {
        // =============================================================== MMA issue (the whole warp waits; one elected lane issues)
        // Per query tile: S(0) .. S(SB-1), then per key tile i: wait P(i) -> O += P(i) V(i) -> S(i + SB), which overwrites the columns of
        // S(i) / P(i).  A warp spends as long on the waits and the issue of a tile's products as the tensor pipe on the products, so
        // two warps share the work: one per query tile (QT = 2), or one for S and one for O (head_dim 128).
        constexpr bool ROLES = D == 128;
        const int mw = warp - MMA_WARP, t = ROLES ? 0 : mw;
        constexpr uint32_t IDESC_S = instr_desc(TC_M, N, 0), IDESC_O = instr_desc(TC_M, D, 1);
        const uint32_t col_o = tmem_base + P::COL_O + t * D, col_s = tmem_base + P::COL_S + t * (SB * N), col_q = tmem_base + P::COL_Q + t * (NQ * D / 2);
        const uint64_t kd0 = smem_desc(smem_u32(smem + P::OFF_K), 16, 1024);
        // MN-major: leading offset = between 64-column blocks, stride offset = between blocks of 8 keys
        const uint64_t vd0 = smem_desc(smem_u32(smem + P::OFF_V), N * 128, 1024);
        // exact codes: Q_hi K [+ Q_lo K]; dequantised K: Q_hi K_hi + Q_hi K_lo [+ Q_lo K_hi] (lo x lo is below fp32 resolution)
        auto issue_s = [&](int i) {
            const uint64_t kd = kd0 + (uint64_t)(((i % KST) * P::KT * P::T_BYTES) >> 4);
            const uint32_t d = col_s + (i % SB) * N;
            bool first = true;
#pragma unroll
            for (int qi = 0; qi < NQ; ++qi) {
#pragma unroll
                for (int ki = 0; ki < P::KT; ++ki) {
                    if (qi == 1 && ki == 1) continue;
#pragma unroll
                    for (int kk = 0; kk < D / 16; ++kk) {
                        tc_mma_ts(d, col_q + qi * (D / 2) + kk * 8, kd + (uint64_t)((ki * P::T_BYTES + (kk >> 2) * (N * 128) + (kk & 3) * 32) >> 4), IDESC_S, first ? 0u : 1u);
                        first = false;
                    }
                }
            }
            tc_commit(&bar_s[t * SB + i % SB]);
            tc_commit(&bar_kf[i % KST]);
        };
        auto issue_o = [&](int i) {
            const uint64_t vd = vd0 + (uint64_t)(((i % VST) * P::T_BYTES) >> 4);
            const uint32_t pa = col_s + (i % SB) * N, acc = col_o + (P::ALT ? (i & 1) * D : 0);
            const uint32_t more = i >= (P::ALT ? 2 : 1) ? 1u : 0u;
            const int n = tile_n(i);                     // P columns / V rows past the keys are never read
            tc_mma_ts(acc, pa, vd, IDESC_O, more);
            if (n > 48) {
#pragma unroll
                for (int kk = 1; kk < N / 16; ++kk) tc_mma_ts(acc, pa + kk * 8, vd + (uint64_t)((kk * 2048) >> 4), IDESC_O, 1u);
            } else {
                if (n > 16) tc_mma_ts(acc, pa + 8, vd + (uint64_t)(2048 >> 4), IDESC_O, 1u);
                if (n > 32) tc_mma_ts(acc, pa + 16, vd + (uint64_t)(4096 >> 4), IDESC_O, 1u);
            }
            tc_commit(&bar_o[i % VST]);
            if (ROLES) tc_commit(&bar_sf[i % SB]);
            else if (QT == 2) tc_commit(&bar_sf[2 * t + (i & 1)]);
        };
        if (t < n_qt && (mw == 0 || QT == 2 || ROLES)) {
            bool ok = mbar_wait_warp(bar_q, 0, abort_flag, 30);
            tc_fence_after();
            if (!ROLES || mw == 0) {
#pragma unroll 1
                for (int i = 0; i < T + (ROLES ? 0 : SB) && ok; ++i) {
                    if (!ROLES && i >= SB) {
                        ok = mbar_wait_warp(&bar_v[(i - SB) % VST], ((i - SB) / VST) & 1, abort_flag, 31) &&
                             mbar_wait_warp(&bar_p[t * SB + i % SB], ((i - SB) / SB) & 1, abort_flag, 32);
                        if (!ok) break;
                        tc_fence_after();
                        issue_o(i - SB);
                    }
                    if (i < T) {
                        ok = mbar_wait_warp(&bar_k[i % KST], (i / KST) & 1, abort_flag, 33);
                        if (ROLES && i >= SB) ok = ok && mbar_wait_warp(&bar_sf[i % SB], ((i - SB) / SB) & 1, abort_flag, 34);
                        if (!ok) break;
                        tc_fence_after();
                        issue_s(i);
                    }
                }
            } else {
#pragma unroll 1
                for (int i = 0; i < T && ok; ++i) {
                    ok = mbar_wait_warp(&bar_v[i % VST], (i / VST) & 1, abort_flag, 31) && mbar_wait_warp(&bar_p[i % SB], (i / SB) & 1, abort_flag, 32);
                    if (!ok) break;
                    tc_fence_after();
                    issue_o(i);
                }
            }
            if (ok && (!ROLES || mw == 1)) tc_commit(bar_end);
            tc_fence_before();
        }
    } else {
        // =============================================================== load warps
        const bool k = warp == P::LOAD_WARP;
        // Tile i goes into the packed stage of tile i - PST once the converters have arrived on that tile's operand barrier.  The table
        // slot of tile i was last read by the softmax of tile i - TS: K(i - PST) converted means S(i - PST - KST) is complete, which was
        // issued after P(i - PST - KST - SB), and TS exceeds that distance (V is converted later still).
        const long long k_par = a.kp.index(b, 0, h, 0), v_par = a.vp.index(b, 0, h, 0);     // (sample, head) part of the parameter index
        const int kng = D / a.kp.group, vng = D / a.vp.group;
        const float c = tc_factor(a.scale_log2);
        const int32_t* kbase = a.kc + b * a.ks_b + h * a.ks_h;
        const int32_t* vbase = a.vc + b * a.vs_b + h * a.vs_h;
        // one lane: the packed rows of tile i and, where they are contiguous, its raw grouped parameters.  Returns whether the other
        // lanes have to fetch the grouped parameters themselves (a ragged last tile, unaligned tables).
        auto copy = [&](int i) {
            const int ps = i % PST, n = tile_n(i);
            uint64_t* bar = k ? &bar_pk[ps] : &bar_pv[ps];
            const uint32_t bytes = (uint32_t)n * (k ? a.wk : a.wv) * 4;
            const int ng = k ? kng : vng;
            const ParamView& pv = k ? a.kp : a.vp;
            const bool bulk = (k ? dy.k_bulk : dy.v_bulk) && (n * ng & 3) == 0;
            const uint32_t pbytes = bulk ? (uint32_t)(n * ng * 4) : 0u;
            mbar_expect_tx(bar, bytes + (pv.zp ? 2 : 1) * pbytes);
            if (k) bulk_copy_g2s(smem + dy.pkk + ps * dy.k_stage, kbase + (long long)(t0 + i) * N * a.wk, bytes, bar);
            else bulk_copy_g2s(smem + dy.pkv + ps * dy.v_stage, vbase + (long long)(t0 + i) * N * a.wv, bytes, bar);
            if (bulk) {
                unsigned char* rec = smem + (k ? dy.krec + ps * dy.krec_stage : dy.vrec + ps * dy.vrec_stage);
                const long long off = (k ? k_par : v_par) + (long long)(t0 + i) * N * ng;
                bulk_copy_g2s(rec, pv.scale + off, pbytes, bar);
                if (pv.zp) bulk_copy_g2s(rec + N * ng * 4, pv.zp + off, pbytes, bar);
            }
        };
        // grouped parameters by ordinary loads, when they do not travel by bulk copy
        auto raw_params = [&](const ParamView& pv, long long base, int ng, bool bulk_tables, int i, float* rec) {
            const int n = tile_n(i);
            if (bulk_tables && (n * ng & 3) == 0) return;
            for (int e = lane; e < n * ng; e += 32) {
                const int key = e / ng, g = e - key * ng;
                const long long pi = base + pv.row((t0 + i) * N + key) * pv.sr + (long long)g * pv.sg;
                rec[e] = __ldg(pv.scale + pi);
                if (pv.zp) rec[N * ng + e] = __ldg(pv.zp + pi);
            }
        };
        // per-key parameters (or step indices) of two keys per lane, one tile ahead
        float ks_[2], kz_[2], vs_[2], vz_[2];
        auto fetch = [&](const ParamView& pv, long long base, bool step, int i, float (&sc)[2], float (&zp)[2]) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int row = pv.row(min((t0 + i) * N + lane + 32 * u, a.Lk - 1));
                if (step) { sc[u] = __int_as_float(row); continue; }
                const long long pi = base + row * pv.sr;
                sc[u] = __ldg(pv.scale + pi);
                zp[u] = pv.zp ? __ldg(pv.zp + pi) : 0.f;
            }
        };
        // Step record of a tile: the table slots of its keys, then the steps that the converters bring into the table first: (first, count), count
        // 0 where all are there.  The table moves on to the tile's first step and all that fit behind it.  For a tile of many steps it
        // stays where it is: keys of steps outside it get the slot of the fp32 routine.
        const ParamView& my = k ? a.kp : a.vp;
        const int tab_rows = k ? dy.k_rows : dy.v_rows;
        int2 win = (k ? KM : VM) == PM_WINDOW ? first_steps(my, tab_rows) : make_int2(0, 0);
        auto step_record = [&](unsigned char* rec, const float (&row)[2]) {
            const int r[2] = {__float_as_int(row[0]), __float_as_int(row[1])};
            const int lo = __reduce_min_sync(0xffffffffu, min(r[0], r[1])), hi = __reduce_max_sync(0xffffffffu, max(r[0], r[1]));
            const bool move = (lo < win.x || hi >= win.y) && hi - lo < min(tab_rows, STEPS_TO_MOVE);
            if (move) win = make_int2(lo, min(lo + tab_rows, max(my.n_rows, hi + 1)));
#pragma unroll
            for (int u = 0; u < 2; ++u) reinterpret_cast<uint16_t*>(rec)[lane + 32 * u] = (uint16_t)(r[u] >= win.x && r[u] < win.y ? r[u] - win.x : tab_rows);
            if (lane == 0) *reinterpret_cast<int2*>(rec + N * 2) = make_int2(win.x, move ? win.y - win.x : 0);
        };
        auto load_k = [&](int i) {
            const int ps = i % PST, n = tile_n(i);
            if (lane == 0) copy(i);
            float* tab = reinterpret_cast<float*>(smem + P::OFF_TAB) + (i % TS) * P::TAB_FLOATS;
            // ---- K records (and tables)
            unsigned char* krec = smem + dy.krec + ps * dy.krec_stage;
            if constexpr (KM == PM_EXACT) {
                bool wide = false;
                const float kbase0 = kb == 8 ? Item<8>::neg_base(0) : kb == 4 ? Item<4>::neg_base(0) : Item<2>::neg_base(0);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int key = lane + 32 * u;
                    const bool w = !(fabsf(kz_[u]) <= 512.f);       // code - zp is not exact in fp16: its term goes to the scores in fp32
                    reinterpret_cast<uint32_t*>(krec)[key] = half_pair(kbase0 - (w ? 0.f : kz_[u]));
                    tab[key] = key < n ? ks_[u] * c : 1.f;          // a masked score stays masked
                    tab[3 * N + key] = w ? kz_[u] : 0.f;
                    wide = wide || w;
                }
                wide = __any_sync(0xffffffffu, wide);
                if (lane == 0) tab[4 * N] = __int_as_float(wide ? 1 : 0);
            } else if constexpr (KM == PM_STEP) {
#pragma unroll
                for (int u = 0; u < 2; ++u) reinterpret_cast<uint16_t*>(krec)[lane + 32 * u] = (uint16_t)__float_as_int(ks_[u]);
            } else if constexpr (KM == PM_WINDOW) {
                step_record(krec, ks_);
            } else {
                if (dy.k_mode == PM_GROUP) raw_params(a.kp, k_par, kng, dy.k_bulk != 0, i, reinterpret_cast<float*>(krec));
            }
            mbar_arrive(&bar_pk[ps]);
            if (P::TAB) mbar_arrive(&bar_t[i % TS]);
            if (KM != PM_GROUP && i + 1 < T) fetch(a.kp, k_par, per_step(KM), i + 1, ks_, kz_);
        };
        auto load_v = [&](int i) {
            const int ps = i % PST;
            if (lane == 0) copy(i);
            float* tab = reinterpret_cast<float*>(smem + P::OFF_TAB) + (i % TS) * P::TAB_FLOATS;
            // ---- V records (and tables)
            unsigned char* vrec = smem + dy.vrec + ps * dy.vrec_stage;
            if constexpr (VM == PM_EXACT) {
                float least = FLT_MAX;          // of the weights' factors: P = weight / factor stays below TC_SUM_MAX while their sum is below that times this
                const float vbase0 = vb == 8 ? Item<8>::neg_base(0) : vb == 4 ? Item<4>::neg_base(0) : Item<2>::neg_base(0);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int key = lane + 32 * u;
                    const bool w = !(fabsf(vz_[u]) <= 512.f);       // such a key is dequantised in fp32 and rounded once; nothing is folded into P
                    const float s = w ? 1.f : fmaxf(vs_[u], TC_VS_MIN);
                    reinterpret_cast<uint32_t*>(vrec)[key] = w ? PAR_SLOW : half_pair(vbase0 - vz_[u]);
                    tab[N + key] = __log2f(s);
                    const float r = __frcp_rn(s);
                    tab[2 * N + key] = r;
                    least = fminf(least, r);
                }
                least = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(least)));
                if (lane == 0) tab[4 * N + 1] = TC_SUM_MAX * least;
            } else if constexpr (VM == PM_STEP) {
#pragma unroll
                for (int u = 0; u < 2; ++u) reinterpret_cast<uint16_t*>(vrec)[lane + 32 * u] = (uint16_t)__float_as_int(vs_[u]);
            } else if constexpr (VM == PM_WINDOW) {
                step_record(vrec, vs_);
            } else {
                if (dy.v_mode == PM_GROUP) raw_params(a.vp, v_par, vng, dy.v_bulk != 0, i, reinterpret_cast<float*>(vrec));
            }
            mbar_arrive(&bar_pv[ps]);
            if (P::TAB) mbar_arrive(&bar_t[i % TS]);
            if (VM != PM_GROUP && i + 1 < T) fetch(a.vp, v_par, per_step(VM), i + 1, vs_, vz_);
        };
        if (k) { if (KM != PM_GROUP) fetch(a.kp, k_par, per_step(KM), 0, ks_, kz_); }
        else if (VM != PM_GROUP) fetch(a.vp, v_par, per_step(VM), 0, vs_, vz_);
        int i = 0;
        bool ok = true;
#pragma unroll 1
        for (; i < T; ++i) {
            if (i >= PST) {
                ok = k ? mbar_wait_warp(&bar_k[(i - PST) % KST], ((i - PST) / KST) & 1, abort_flag, 41)
                       : mbar_wait_warp(&bar_v[(i - PST) % VST], ((i - PST) / VST) & 1, abort_flag, 42);
                if (!ok) break;
            }
            if (k) load_k(i); else load_v(i);
        }
        if (!ok && lane == 0) {
            // drain: bulk copies already issued must land before the CTA may exit
            for (int n = max(0, i - PST); n < i; ++n) {
                uint64_t* bar = k ? &bar_pk[n % PST] : &bar_pv[n % PST];
                for (uint32_t w = 0; w < TC_SPIN_LIMIT && !mbar_try(bar, (n / PST) & 1); ++w) {}
            }
        }
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)P::TMEM_COLS) : "memory");
    }
}


// smem layout of a launch, parameter modes, launch of one instantiation
template <int D, int NQ, int QT, int KM, int VM> int tc_launch_one(const AttnArgs& a, TcDyn dy, int kb, int vb, cudaStream_t st) {
    using P = TcPlan<D, NQ, QT, KM, VM>;
    auto tab_bytes = [](int mode, int rows) { return mode == PM_STEP ? rows * 3 * D * 2 : mode == PM_WINDOW ? (rows + 1) * 3 * D * 2 : 0; };
    auto rec_bytes = [](int mode, int ng) { return mode == PM_GROUP ? TC_N * ng * 8 : mode == PM_EXACT ? TC_N * 4 : mode == PM_STEP ? TC_N * 2 : mode == PM_WINDOW ? TC_N * 2 + 16 : 16; };
    dy.k_stage = TC_N * a.wk * 4; dy.v_stage = TC_N * a.wv * 4;
    dy.krec_stage = rec_bytes(dy.k_mode, D / a.kp.group); dy.vrec_stage = rec_bytes(dy.v_mode, D / a.vp.group);
    dy.pkk = P::OFF_DYN;
    dy.pkv = dy.pkk + P::PST * dy.k_stage;
    dy.krec = dy.pkv + P::PST * dy.v_stage;
    dy.vrec = dy.krec + P::PST * dy.krec_stage;
    dy.ktab = dy.vrec + P::PST * dy.vrec_stage;
    dy.vtab = dy.ktab + tab_bytes(KM, dy.k_rows);
    const size_t smem = (size_t)dy.vtab + tab_bytes(VM, dy.v_rows) + 1024;     // slack for the 1024-byte alignment of the swizzled tiles
    if (smem > 227 * 1024) return fail(VARQ_ERR_UNSUPPORTED, "varq_attn_fwd: %zu bytes of shared memory", smem);
    static bool configured[64] = {false};    // per device; the attribute is sticky, set it outside any stream capture
    int dev = 0;
    VARQ_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        VARQ_CUDA_TRY(cudaFuncSetAttribute(attn_tc_kernel<D, NQ, QT, KM, VM>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    VARQ_CUDA_TRY(launch_pdl(attn_tc_kernel<D, NQ, QT, KM, VM>, (unsigned)((long long)a.B * a.H * a.n_qtiles * a.splits), P::THREADS, smem, st, 1, a, dy, kb, vb));
    count_launches(1);
    return VARQ_OK;
}
template <int D, int NQ, int QT> int tc_launch_modes(const AttnArgs& a, const TcDyn& dy, int kb, int vb, cudaStream_t st) {
    const int km = dy.k_mode == PM_SLOW ? PM_GROUP : dy.k_mode, vm = dy.v_mode == PM_SLOW ? PM_GROUP : dy.v_mode;
#define VARQ_TC_GO(K_, V_) if (km == K_ && vm == V_) return tc_launch_one<D, NQ, QT, K_, V_>(a, dy, kb, vb, st)
    VARQ_TC_GO(PM_EXACT, PM_EXACT); VARQ_TC_GO(PM_EXACT, PM_GROUP); VARQ_TC_GO(PM_EXACT, PM_STEP);
    VARQ_TC_GO(PM_GROUP, PM_EXACT); VARQ_TC_GO(PM_GROUP, PM_GROUP); VARQ_TC_GO(PM_GROUP, PM_STEP);
    VARQ_TC_GO(PM_STEP, PM_EXACT); VARQ_TC_GO(PM_STEP, PM_GROUP); VARQ_TC_GO(PM_STEP, PM_STEP);
    if constexpr (NQ == 2 && QT == 1) {
        VARQ_TC_GO(PM_EXACT, PM_WINDOW); VARQ_TC_GO(PM_GROUP, PM_WINDOW); VARQ_TC_GO(PM_WINDOW, PM_EXACT); VARQ_TC_GO(PM_WINDOW, PM_GROUP); VARQ_TC_GO(PM_WINDOW, PM_WINDOW);
    }
#undef VARQ_TC_GO
    return fail(VARQ_ERR_ARG, "varq_attn_fwd: parameter mode");
}
// status word of this file's kernels
static int tc_file_status(int* out) {
    int v = 0;
    VARQ_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int)));
    if (v != 0) {
        const int zero = 0;
        VARQ_CUDA_TRY(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)));
    }
    if (*out == 0) *out = v;
    return VARQ_OK;
}
// one set per instantiation file
struct TcFile {
    int (*launch)(const AttnArgs&, const TcDyn&, int kb, int vb, cudaStream_t);
    int (*status)(int*);
};
extern const TcFile tc_d64_q1, tc_d64_q2, tc_d64_x2_q1, tc_d64_x2_q2, tc_d128_q1, tc_d128_q2;

}  // namespace varq
