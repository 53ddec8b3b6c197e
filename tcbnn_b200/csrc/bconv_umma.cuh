// Binary convolution on the 5th-generation tensor cores: tcgen05.mma kind::i8 with the
// accumulators in tensor memory.
//
// The layer is the same Conv128LayerFMT arithmetic (kernel.cuh:676-827) as the warp-MMA
// path in bnn_layers.cuh.  Here the packed input bits are expanded to +-1 bytes in shared
// memory and the contraction is an exact int8 x int8 -> int32 implicit GEMM, so the
// accumulator IS the reference's `C*R*S - exclude*C - 2*popc(a^w)`: out-of-frame taps are
// zero bytes and contribute nothing, no popcount identities or correction tables needed.
//
// Implicit GEMM without im2col.  Pixels of the whole batch are laid out in one "virtual"
// zero-padded raster of pitch PW = W + pad columns and VH = H + pad rows per image (one shared
// band of zeros between neighbouring rows / images).  A tile is 128 consecutive raster
// positions; the +-1 bytes of the positions it touches (tile + halo) sit in shared memory as
//     A[channel chunk of 16][raster position][16 bytes]
// which is the no-swizzle K-major core-matrix layout of the UMMA shared-memory descriptor
// (8 rows x 16 bytes contiguous, next 8 rows +128 B, next 16 channels +LBO).  In that layout
// filter tap (r, s) is nothing but a start-address offset of ((r*PW + s) * 16) bytes, so the
// nine taps reuse one expanded patch.  Positions that fall on the zero bands produce junk
// rows that are simply not stored.
//
// This header holds the PTX wrappers, descriptors and bit -> byte expansion shared by the kernels:
// bconv_umma_ws.cuh (filter-stationary), bconv_umma_as.cuh (activation-stationary),
// bconv_umma_pre.cuh (fed from a pre-expanded input), bgemm_umma.cuh (bit GEMM).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <climits>

namespace tcbnn {
namespace umma {

// ---- small PTX wrappers -------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Non-blocking form: a plain read of the barrier's phase, cheaper for a thread that expects the
// phase to be complete already.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// One lane of a converged warp (the whole warp must execute this).
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}
// Bounded wait: gives up after `limit` polls and reports failure instead of hanging.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* err_flag) {
    for (int i = 0; i < (1 << 22); i++)
        if (mbar_try_wait(bar, parity)) return true;
    if (err_flag) atomicExch(err_flag, 1);
    return false;
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {   // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_dst), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {    // whole warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc], int8 operands, int32 accumulate; one thread issues.
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Same instruction with the two descriptors handed over as (low, high) register pairs, so the
// issue loop only does 32-bit adds on the address field; no memory clobber (ordering against
// the data comes from the mbarrier waits and fences around the loop).
__device__ __forceinline__ void mma_i8_split(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi,
                                             uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %5, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar) : "memory");
}
// 32 lanes x 32 consecutive columns: thread t of the warp gets lane (base lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, int (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
// 16 lanes x 32 consecutive columns: thread t of the warp gets, for n = 0..3 and e = 0, 1, columns
// 8n + 2(t%4) + e of lane t/4 in r[4n + e] and of lane t/4 + 8 in r[4n + 2 + e].
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, int (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
// Same as tmem_ld32 for 16 and 8 columns.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The same wait, naming the registers it makes valid: keeps their uses behind it where a later load is
// issued before they are used.
__device__ __forceinline__ void tmem_ld_wait16(int (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :: "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle: rows 16 B apart inside a core matrix,
// `sbo` bytes between 8-row groups, `lbo` bytes between 16-byte K chunks.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor: int8 x int8 -> int32, both operands K-major, M = 128.
__host__ __device__ constexpr uint32_t idesc_i8(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

// 16 packed bits -> 16 bytes of +1 / -1.  Which bit lands in which byte is a fixed
// permutation; activations and filters both go through this function, so it cancels.
__device__ __forceinline__ uint4 expand16(uint32_t h) {
    uint32_t v[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const uint32_t nb = (h >> (4 * g)) & 0xFu;
        const uint32_t y = (nb * 0x00204081u) & 0x01010101u;      // one bit per byte
        v[g] = ~(y * 0xFEu);                                      // 1 -> 0x01, 0 -> 0xFF
    }
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// ---- 4-bit operands: tcgen05.mma kind::mxf4 ------------------------------------------------
// +1 / -1 are exact in e2m1 (0x2 / 0xA), zero is 0x0, and with unit ue8m0 block scales (byte 0x7F)
// the fp32 accumulator of a +-1 contraction is the exact integer sum (every partial sum is an
// integer far below 2^24).  An MMA is 128 x N x 64: twice the MAC rate of kind::i8 at half the
// operand bytes (measured by tcbnn_mma_peak kind 7).  Layout as for int8, K-major without
// swizzle, except that a 16-byte core-matrix row now holds 32 channels and one MMA spans two of
// them (`lbo` apart).
// 32 packed bits -> 16 bytes of +-1.0: bit 4*i + j of the word -> nibble i of .x/.y/.z/.w for j = 3..0
// (1 -> +1.0, 0 -> -1.0).  Which bit lands in which nibble is free -- activations and filters both go
// through this function, so the order inside a word cancels -- and this one costs a shift and a
// three-input logic operation per eight values (spreading a byte's bits in order takes four times that).
__host__ __device__ __forceinline__ uint4 expand32_f4(uint32_t w) {
    return make_uint4((w & 0x88888888u) ^ 0xAAAAAAAAu, ((w << 1) & 0x88888888u) ^ 0xAAAAAAAAu,
                      ((w << 2) & 0x88888888u) ^ 0xAAAAAAAAu, ((w << 3) & 0x88888888u) ^ 0xAAAAAAAAu);
}
// Output channel (within its 32) that column c of an accumulator holds.  A tcgen05.ld of shape 16x256b
// gives a thread columns 8n + 2q and 8n + 2q + 1 of its rows (q = lane % 4, n = 0..3); with this order
// those are two runs of four consecutive channels, 4q.. and 16 + 4q.., so that the four lanes of a
// quad move 64 (int32) or 32 (int16) consecutive bytes of an NHWC row.  The filter blob is laid out in
// this order (prepare_filter_f4), thresholds and bit positions follow it.
__host__ __device__ constexpr int f4_channel_of_column(int c) {
    return 16 * (c >> 4) + 4 * ((c >> 1) & 3) + 2 * ((c >> 3) & 1) + (c & 1);
}
__host__ __device__ constexpr int f4_column_of_channel(int ch) {
    return 8 * (2 * (ch >> 4) + ((ch >> 1) & 1)) + 2 * ((ch >> 2) & 3) + (ch & 1);
}
// Instruction descriptor of the block-scaled kinds: e2m1 x e2m1, ue8m0 scales, K-major, M = 128,
// K = 64, scale-factor ids 0.
__host__ __device__ constexpr uint32_t idesc_f4(int n) {
    return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((128u >> 4) << 24);
}
// D[tmem] (+)= A * B with the scale factors read from tensor memory at sfa / sfb; descriptors as
// (low, high) register pairs like mma_i8_split.
__device__ __forceinline__ void mma_f4_split(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi,
                                             uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                             uint32_t accumulate, uint32_t sfa, uint32_t sfb) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], da, db, %5, [%7], [%8], p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate),
          "r"(sfa), "r"(sfb));
}
// Runs of K MMAs (taps t[0..K-1] of one 64-channel block, B advancing by step_b per tap), each written
// as one block because of what the issuing warp does between two MMAs: the tensor pipe queues only
// two or three instructions, so whatever takes longer than that is time it idles.  The whole warp
// executes them, the lane with leader != 0 issues; the first MMA accumulates when acc != 0, the
// others always.
//   mma_f4_run      nothing but the MMAs
//   mma_f4_end      the last MMAs of a stage: two barrier tests in front of them whose results are
//                   read behind them, then the commits of the stage and of the accumulator.  A test
//                   takes 150-200 clocks to return while the MMAs keep the shared-memory port busy;
//                   asked for first and read last, that time is covered.  bar_c: 0 = no commit.
//                   Bit 0 / 1 of the result: phase par0 / par1 of barrier bar0 / bar1 is complete.
// Measured on groups of nine with one wait and one commit per group: 61.8 -> 48.0 clocks per MMA at
// N = 64, 70.7 -> 64.0 at N = 128, the pipe's own rate.
#define TCBNN_F4_MMA(G, AOFF, PRED)                                                                  \
    "add.u32 xa, %1, " AOFF ";\n\tmov.b64 da, {xa, %2};\n\tmov.b64 db, {xb, %4};\n\t"                \
    "@pl tcgen05.mma.cta_group::" G ".kind::mxf4.block_scale.block32 [%5], da, db, %6, [%8], [%9], " PRED ";\n\t" \
    "add.u32 xb, xb, %10;\n\t"
#define TCBNN_F4_HEAD                                                                                \
    ".reg .pred pq, pt, pl;\n\t.reg .b64 da, db;\n\t.reg .b32 xa, xb;\n\t"                           \
    "setp.ne.b32 pl, %0, 0;\n\tsetp.ne.b32 pq, %7, 0;\n\tsetp.eq.b32 pt, %0, %0;\n\tmov.u32 xb, %3;\n\t"
#define TCBNN_F4_IN                                                                                  \
    "r"(leader), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(d_tmem), "r"(idesc), "r"(acc), "r"(sfa), \
        "r"(sfb), "r"(step_b)
#define TCBNN_F4_RUN(G)                                                                              \
    if constexpr (K == 9)                                                                            \
        asm volatile("{\n\t" TCBNN_F4_HEAD TCBNN_F4_MMA(G, "%11", "pq") TCBNN_F4_MMA(G, "%12", "pt") TCBNN_F4_MMA(G, "%13", "pt") \
                     TCBNN_F4_MMA(G, "%14", "pt") TCBNN_F4_MMA(G, "%15", "pt") TCBNN_F4_MMA(G, "%16", "pt") \
                     TCBNN_F4_MMA(G, "%17", "pt") TCBNN_F4_MMA(G, "%18", "pt") TCBNN_F4_MMA(G, "%19", "pt") "}" \
                     ::TCBNN_F4_IN, "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), \
                       "r"(t[7]), "r"(t[8]) : "memory");                                             \
    else if constexpr (K == 5)                                                                       \
        asm volatile("{\n\t" TCBNN_F4_HEAD TCBNN_F4_MMA(G, "%11", "pq") TCBNN_F4_MMA(G, "%12", "pt") TCBNN_F4_MMA(G, "%13", "pt") \
                     TCBNN_F4_MMA(G, "%14", "pt") TCBNN_F4_MMA(G, "%15", "pt") "}"                   \
                     ::TCBNN_F4_IN, "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]) : "memory"); \
    else if constexpr (K == 4)                                                                       \
        asm volatile("{\n\t" TCBNN_F4_HEAD TCBNN_F4_MMA(G, "%11", "pq") TCBNN_F4_MMA(G, "%12", "pt") TCBNN_F4_MMA(G, "%13", "pt") \
                     TCBNN_F4_MMA(G, "%14", "pt") "}"                                                \
                     ::TCBNN_F4_IN, "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]) : "memory");          \
    else                                                                                             \
        asm volatile("{\n\t" TCBNN_F4_HEAD TCBNN_F4_MMA(G, "%11", "pq") "}" ::TCBNN_F4_IN, "r"(t[0]) : "memory")
template <int K, bool PAIR = false>
__device__ __forceinline__ void mma_f4_run(uint32_t leader, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi,
                                           uint32_t b_lo, uint32_t b_hi, uint32_t step_b, const uint32_t* t,
                                           uint32_t idesc, uint32_t acc, uint32_t sfa, uint32_t sfb) {
    static_assert(K == 1 || K == 4 || K == 5 || K == 9, "run lengths in use");
    if constexpr (PAIR) { TCBNN_F4_RUN("2"); } else { TCBNN_F4_RUN("1"); }
}
#undef TCBNN_F4_RUN
#undef TCBNN_F4_MMA
#undef TCBNN_F4_HEAD
#undef TCBNN_F4_IN
#define TCBNN_F4_MMA(G, AOFF, PRED)                                                                  \
    "add.u32 xa, %2, " AOFF ";\n\tmov.b64 da, {xa, %3};\n\tmov.b64 db, {xb, %5};\n\t"                \
    "@pl tcgen05.mma.cta_group::" G ".kind::mxf4.block_scale.block32 [%6], da, db, %7, [%9], [%10], " PRED ";\n\t" \
    "add.u32 xb, xb, %11;\n\t"
#define TCBNN_F4_HEAD(Q)                                                                             \
    "{\n\t.reg .b16 both;\n\tmov.b16 both, 3;\n\t.reg .pred p0, p1, pq, pt, pl, pc;\n\t.reg .b64 da, db;\n\t.reg .b32 xa, xb, r1;\n\t"       \
    "mbarrier.test_wait.parity" Q ".shared::cta.b64 p0, [%12], %13;\n\t"                            \
    "mbarrier.test_wait.parity" Q ".shared::cta.b64 p1, [%14], %15;\n\t"                            \
    "setp.ne.b32 pl, %1, 0;\n\tsetp.ne.b32 pq, %8, 0;\n\tsetp.eq.b32 pt, %1, %1;\n\tmov.u32 xb, %4;\n\t" \
    "setp.ne.and.b32 pc, %17, 0, pl;\n\t"
#define TCBNN_F4_TAIL(G, W, M)                                                                       \
    "@pl tcgen05.commit.cta_group::" G ".mbarrier::arrive::one.shared::cluster" W ".b64 [%16]" M ";\n\t" \
    "@pc tcgen05.commit.cta_group::" G ".mbarrier::arrive::one.shared::cluster" W ".b64 [%17]" M ";\n\t" \
    "selp.u32 %0, 1, 0, p0;\n\tselp.u32 r1, 2, 0, p1;\n\tor.b32 %0, %0, r1;\n\t}"
#define TCBNN_F4_IN                                                                                  \
    "r"(leader), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(d_tmem), "r"(idesc), "r"(acc), "r"(sfa), \
        "r"(sfb), "r"(step_b), "r"(bar0), "r"(par0), "r"(bar1), "r"(par1), "r"(bar_e), "r"(bar_c)
#define TCBNN_F4_END(G, Q, W, M)                                                                     \
    if constexpr (K == 4)                                                                            \
        asm volatile(TCBNN_F4_HEAD(Q) TCBNN_F4_MMA(G, "%18", "pq") TCBNN_F4_MMA(G, "%19", "pt") TCBNN_F4_MMA(G, "%20", "pt") \
                     TCBNN_F4_MMA(G, "%21", "pt") TCBNN_F4_TAIL(G, W, M)                             \
                     : "=&r"(ok) : TCBNN_F4_IN, "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]) : "memory"); \
    else if constexpr (K == 3)                                                                       \
        asm volatile(TCBNN_F4_HEAD(Q) TCBNN_F4_MMA(G, "%18", "pq") TCBNN_F4_MMA(G, "%19", "pt") TCBNN_F4_MMA(G, "%20", "pt") TCBNN_F4_TAIL(G, W, M) \
                     : "=&r"(ok) : TCBNN_F4_IN, "r"(t[0]), "r"(t[1]), "r"(t[2]) : "memory");         \
    else                                                                                             \
        asm volatile(TCBNN_F4_HEAD(Q) TCBNN_F4_MMA(G, "%18", "pq") TCBNN_F4_TAIL(G, W, M)            \
                     : "=&r"(ok) : TCBNN_F4_IN, "r"(t[0]) : "memory")
// (PAIR: the MMAs of a pair of CTAs, barriers of cluster scope, the commits arrive in both)
template <int K, bool PAIR = false>
__device__ __forceinline__ uint32_t mma_f4_end(uint32_t leader, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi,
                                               uint32_t b_lo, uint32_t b_hi, uint32_t step_b, const uint32_t* t,
                                               uint32_t idesc, uint32_t acc, uint32_t sfa, uint32_t sfb,
                                               uint32_t bar0, uint32_t par0, uint32_t bar1, uint32_t par1,
                                               uint32_t bar_e, uint32_t bar_c) {
    static_assert(K == 1 || K == 3 || K == 4, "run lengths in use");
    uint32_t ok;
    if constexpr (PAIR) { TCBNN_F4_END("2", ".acquire.cluster", ".multicast::cluster", ", both"); } else { TCBNN_F4_END("1", "", "", ""); }
    return ok;
}
#undef TCBNN_F4_END
#undef TCBNN_F4_MMA
#undef TCBNN_F4_HEAD
#undef TCBNN_F4_TAIL
#undef TCBNN_F4_IN
// Columns [col, col + 32) of the calling warp's 32 lanes of tensor memory := unit scales (every
// byte 0x7F), so a scale reads as 1.0 wherever in the region the hardware looks it up.  Whole
// warp; warps 0-3 of a warpgroup cover the 128 lanes between them (warp w -> lanes 32*(w%4)..).
__device__ __forceinline__ void tmem_fill_unit_scales(uint32_t tmem, uint32_t col) {
    const uint32_t base = tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + col;
#pragma unroll
    for (int c = 0; c < 32; c += 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};"
                     ::"r"(base + c), "r"(0x7F7F7F7Fu) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// fp32 accumulator holding an integer of magnitude below 2^22 -> that integer, exactly; the biased
// form leaves kF4Bias on it (its low 16 bits are those of the integer)
constexpr int kF4Bias = 0x4B400000;
__device__ __forceinline__ int f4_acc_to_biased(int raw) { return __float_as_int(__int_as_float(raw) + 12582912.0f); }
__device__ __forceinline__ int f4_acc_to_int(int raw) { return f4_acc_to_biased(raw) - kF4Bias; }

// Four consecutive residual channels (element index i, a multiple of 4) widened to int32.
__device__ __forceinline__ int4 ld_res4(const void* p, int bytes, size_t i) {
    if (bytes == 2) {
        const uint2 q = ld_dep(reinterpret_cast<const uint2*>(reinterpret_cast<const short*>(p) + i));
        return make_int4((int)(short)(q.x & 0xFFFFu), (int)(short)(q.x >> 16),
                         (int)(short)(q.y & 0xFFFFu), (int)(short)(q.y >> 16));
    }
    return ld_dep(reinterpret_cast<const int4*>(reinterpret_cast<const int*>(p) + i));
}
__device__ __forceinline__ int4 max4(int4 a, int4 b) {
    return make_int4(max(a.x, b.x), max(a.y, b.y), max(a.z, b.z), max(a.w, b.w));
}

}  // namespace umma
}  // namespace tcbnn
