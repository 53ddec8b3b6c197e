// Bit GEMM on tcgen05: C[m][n] = sum_k a[m][k] * w[n][k] over +-1 values, i.e. the reference's
// K - 2*popc(a ^ w) (bmm/tensorcore_kernel.cu:138-356; Fc128LayerFMT / Out128LayerFMT,
// kernel.cuh:174-280 on top of it), as an exact 4-bit MMA: tcgen05.mma kind::mxf4 on +-1.0 as e2m1
// nibbles with unit block scales (bconv_umma.cuh), fp32 accumulators holding exact integers.
//
// One streaming pass first writes both operands as +-1 nibbles (0 for padding: rows past the end,
// bits past K) in 4 KB units [128-row tile][64-bit k-block][32-bit chunk][row][16 B], the
// no-swizzle K-major operand layout, so that a unit is one bulk copy and one MMA operand.
// The GEMM is persistent: a CTA per SM walks over 128 x 128 tiles, or a pair of CTAs over 256 x 256
// tiles (PAIR), each over a range of k-blocks:
//
//   warps 0-7  epilogue : tcgen05.ld and either finish the layer (one split: int32 / threshold bits /
//                         scale + bias straight from the accumulator) or store int32 partial sums for
//                         gemm_splitk_finish.  128 x 128 tiles alternate between two accumulators, so
//                         that a tile is finished while the next one is computed
//   warp  8    loader A : one lane, one bulk copy (tensor copy in a pair) per stage (a stage holds up to
//                         kGemmKU consecutive k-blocks, contiguous in the expanded operand)
//   warp  9    MMA      : converged warp, elected lane: one MMA per k-block (the leader's, in a pair)
//   warp  10   loader W : one lane, one bulk copy per stage
//
// A 128 x 128 tile reads 8 KB of operands per k-block and has 8 KB copied in, which fills the
// shared-memory port for 128 clocks (136 measured) where its MMA takes 64.  A pair does four times the work on
// twice the SMs: each reads its 128 rows of A and half of W, 4 + 4 KB, and receives as much, for an MMA that
// takes 128 (133-153 measured).  8192 x 8192 x 8192 with threshold bits 204 -> 186 us against 256 x 128
// tiles on one SM (28 KB and 220 clocks per k-block); 174 by graph replay, the kernel 145 of it, 0.85 of the MMA rate.
//
// Loaders and issuer run ahead across tile boundaries, so set-up, first loads and epilogue of all
// but a CTA's last tile are hidden: as one CTA per tile (two per SM) the MLP's hidden layer, 8192 x 1024
// x 1024, spent 23 us on 3.3 us of MMAs.  W's rows are laid out in the order of
// f4_channel_of_column within each 32, so that integer and float results leave in whole sectors (the
// 16x256b read of the accumulator, see there).
//
// A thread that issues a bulk copy is busy for 100-200 clocks per copy whatever its size, and
// copies issued by different warps overlap (tcbnn_bulk_copy_rate measures both): hence few, large
// copies and one issuing warp per operand.
#pragma once
#include "bconv_umma_pre.cuh"

namespace tcbnn {
namespace umma {

constexpr int kGemmThreads = 352;
constexpr int kGemmUnit = 4096;                        // 128 rows x 64 k, 4 bits each
constexpr int kGemmKU = 4;                             // k-blocks per stage
// Ring depth and bytes of a stage (A and W).  One CTA per SM takes all of tensor memory: accumulators,
// then 32 columns of unit scales at the top.
constexpr int kGemmStages = 6;
constexpr int kGemmStageBytes = 2 * kGemmKU * kGemmUnit;
// ring, barriers, thresholds per epilogue warp
constexpr size_t kGemmSmem = (size_t)kGemmStages * kGemmStageBytes + 32 * 8 + 64 + 8 * 128 * 4;

struct GemmUmmaArgs {
    const unsigned char* ea;   // expanded A: [MT][KB] units
    const unsigned char* ew;   // expanded W: [NT][KB] units
    int M, N, KB, MT, NT, splits, per;   // per: k-blocks per split
    int32_t* partial;          // [splits][M][N], used when splits > 1
    // splits == 1: the layer is finished in the epilogue (GemmMode of bnn_layers.cuh)
    int mode; void* out; int ldo; const float* p0; const float* p1;
    uint4* nxt; int nxt_KB;    // threshold bits also as the next layer's expanded A operand, or null
    int* status;               // set to 1 when a bounded wait gives up
    long long* trace;          // null, or 16 counters: CTA 0 writes [9..15] (clocks; see the C header)
};

// zeroes the nibbles of the bits that are clear in m (nibble order of expand32_f4)
__device__ __forceinline__ uint4 keep32_f4(uint4 e, uint32_t m) {
    return make_uint4(e.x & (((m >> 3) & 0x11111111u) * 0xFu), e.y & (((m >> 2) & 0x11111111u) * 0xFu),
                      e.z & (((m >> 1) & 0x11111111u) * 0xFu), e.w & ((m & 0x11111111u) * 0xFu));
}

// Chunk c (32 bits of K) of row r of an expanded operand with KB k-blocks; `valid` elements exist, the rest
// is padding: 0, not -1.
__device__ __forceinline__ void store_unit_chunk(uint4* units, int KB, int r, int c, uint32_t word, int valid) {
    uint4 e = expand32_f4(word);
    if (valid < 32) e = keep32_f4(e, 0xFFFFFFFFu << (32 - valid));
    units[((size_t)(r >> 7) * KB + (c >> 1)) * 256 + (c & 1) * 128 + (r & 127)] = e;
}

// packed bits [rows][ld words] (bit k of a row at bit 31 - k%32 of word k/32) -> units.  A task is
// (128-row tile, group of four k-blocks): 256 threads, two per row, each reading the 16 bytes (four
// 32-bit chunks) of its row that fall into its half of the group -- a whole 32-byte sector per row -- and
// writing four 16-byte slots; for a given chunk the threads of a warp write two runs of 256 contiguous
// bytes.  ld is even, so the 8-byte loads are aligned.  W's rows go in the order of the accumulator's columns.
__device__ __forceinline__ void expand_rows_task(const uint32_t* bits, int rows, int ld, int K, int KB, int tk, bool isw, uint4* out) {
    const int KG = (KB + 3) >> 2;
    const int t = threadIdx.x, row = t >> 1, half = t & 1;
    const int rt = tk / KG, kg = tk - rt * KG;
    out += (size_t)rt * KB * 256;                                        // 256 slots of 16 bytes per unit
    const int r = rt * 128 + (isw ? (row & ~31) + f4_channel_of_column(row & 31) : row);
    const int w0 = kg * 8 + half * 4;                                    // first 32-bit chunk of this thread
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (r < rows) {
        const uint32_t* src = bits + (size_t)r * ld + w0;
        if (w0 + 1 < ld) { const uint2 q = ld_dep(reinterpret_cast<const uint2*>(src)); w[0] = q.x; w[1] = q.y; }
        else if (w0 < ld) w[0] = ld_dep(src);
        if (w0 + 3 < ld) { const uint2 q = ld_dep(reinterpret_cast<const uint2*>(src + 2)); w[2] = q.x; w[3] = q.y; }
        else if (w0 + 2 < ld) w[2] = ld_dep(src + 2);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = w0 + j, kb = c >> 1;                               // chunk -> k-block
        if (kb >= KB) break;
        const int k0 = c * 32;
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
        if (r < rows && k0 < K) {
            e = expand32_f4(w[j]);
            const int valid = K - k0;                                    // elements of this chunk that exist
            if (valid < 32) e = keep32_f4(e, 0xFFFFFFFFu << (32 - valid));   // the rest is padding: 0, not -1
        }
        out[(size_t)kb * 256 + (c & 1) * 128 + row] = e;
    }
}

// Both operands of a GEMM in one launch: tasks [0, RT_a * KG) belong to A, the rest to W (KG = groups per
// row tile).
__device__ __forceinline__ void expand_rows_pair(const uint32_t* a_bits, int a_rows, int a_ld, int RT_a,
                                                 const uint32_t* w_bits, int w_rows, int w_ld, int RT_w,
                                                 int K, int KB, uint4* out_a, uint4* out_w) {
    // the GEMM that consumes these units may be set up meanwhile (it waits before its first copy);
    // this pass itself is a programmatic dependent of whatever wrote A
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int KG = (KB + 3) >> 2;
    const int tasks = (RT_a + RT_w) * KG;
    for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
        const bool isw = task >= RT_a * KG;
        expand_rows_task(isw ? w_bits : a_bits, isw ? w_rows : a_rows, isw ? w_ld : a_ld, K, KB, isw ? task - RT_a * KG : task, isw,
                         isw ? out_w : out_a);
    }
}

// Weights that a pass over a chain of FC layers expands beside the packing of its input rows
// (tcbnn_pack_rows_w): tasks are those of expand_rows_task, weight i's from first[i] on.
constexpr int kMaxPassWeights = 8;
struct PassWeights {
    int n, first[kMaxPassWeights + 1];
    const uint32_t* bits[kMaxPassWeights];
    uint4* units[kMaxPassWeights];
    int rows[kMaxPassWeights], ld[kMaxPassWeights], K[kMaxPassWeights];
};
__device__ __forceinline__ void expand_pass_weights(const PassWeights& p, int block, int blocks) {
    for (int task = block; task < p.first[p.n]; task += blocks) {
        int i = 0;
        while (task >= p.first[i + 1]) i++;
        expand_rows_task(p.bits[i], p.rows[i], p.ld[i], p.K[i], (p.K[i] + 63) >> 6, task - p.first[i], true, p.units[i]);
    }
}

// ---- a pair of CTAs on one 256 x 256 tile (cta_group::2) ------------------------------------------
// Each CTA holds its 128 rows of A, half of W's 256 rows and its 128 x 256 accumulator; the leader (even
// rank) issues MMAs that read both shared memories.  The copies of both complete on the leader's barrier,
// which only a tensor copy of a pair may do (cta_group::2; no multicast): a thread of the second CTA that passed its
// CTA's completion on would have to do so with an arrival of cluster scope, 1400 clocks each, one at a
// time (8192 x 8192 x 8192 with threshold bits 174 us, 219 with three warps taking turns at it).
// One stage of an operand, kGemmKU units: rows of 1 KB of the expanded operand from `row` on.  (A stage
// that holds fewer k-blocks is followed by others' units or, behind the last, by zeros, which no MMA reads.)
__device__ __forceinline__ void tensor_g2s_pair(uint32_t dst, const CUtensorMap* map, int row, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(0), "r"(row), "r"(leader_bar) : "memory");
}
// K MMAs of 256 x 256 x 64, A and W advancing by `step` alike; with END what mma_f4_end does (the commits
// arrive in both CTAs).
#define TCBNN_F4_PAIR_MMA(PRED)                                                                      \
    "mov.b64 da, {xa, %3};\n\tmov.b64 db, {xb, %3};\n\t"                                            \
    "@pl tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%5], da, db, %6, [%8], [%9], " PRED ";\n\t" \
    "add.u32 xa, xa, %10;\n\tadd.u32 xb, xb, %10;\n\t"
#define TCBNN_F4_PAIR_HEAD                                                                           \
    "{\n\t.reg .pred p0, p1, pq, pt, pl, pc;\n\t.reg .b64 da, db;\n\t.reg .b32 xa, xb, r1;\n\t.reg .b16 both;\n\t" \
    "setp.ne.b32 pl, %1, 0;\n\tsetp.ne.b32 pq, %7, 0;\n\tsetp.eq.b32 pt, %1, %1;\n\t"              \
    "mov.u32 xa, %2;\n\tmov.u32 xb, %4;\n\t"
#define TCBNN_F4_PAIR_TEST                                                                           \
    "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p0, [%11], %12;\n\t"                 \
    "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p1, [%13], %14;\n\tsetp.ne.and.b32 pc, %16, 0, pl;\n\tmov.b16 both, 3;\n\t"
#define TCBNN_F4_PAIR_TAIL                                                                           \
    "@pl tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%15], both;\n\t" \
    "@pc tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%16], both;\n\t" \
    "selp.u32 %0, 1, 0, p0;\n\tselp.u32 r1, 2, 0, p1;\n\tor.b32 %0, %0, r1;\n\t}"
#define TCBNN_F4_PAIR_IN                                                                             \
    "r"(leader), "r"(a_lo), "r"(hi), "r"(b_lo), "r"(d_tmem), "r"(idesc), "r"(acc), "r"(sfa), "r"(sfb), "r"(step)
__device__ __forceinline__ void mma_f4_pair_run(uint32_t leader, uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi,
                                                uint32_t step, uint32_t idesc, uint32_t acc, uint32_t sfa, uint32_t sfb) {
    uint32_t none;
    asm volatile(TCBNN_F4_PAIR_HEAD TCBNN_F4_PAIR_MMA("pq") "mov.u32 %0, 0;\n\t}" : "=&r"(none) : TCBNN_F4_PAIR_IN : "memory");
}
template <int K>
__device__ __forceinline__ uint32_t mma_f4_pair_end(uint32_t leader, uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi,
                                                    uint32_t step, uint32_t idesc, uint32_t acc, uint32_t sfa, uint32_t sfb,
                                                    uint32_t bar0, uint32_t par0, uint32_t bar1, uint32_t par1, uint32_t bar_e,
                                                    uint32_t bar_c) {
    static_assert(K == 1 || K == 3, "run lengths in use");
    uint32_t ok;
    if constexpr (K == 3)
        asm volatile(TCBNN_F4_PAIR_HEAD TCBNN_F4_PAIR_TEST TCBNN_F4_PAIR_MMA("pq") TCBNN_F4_PAIR_MMA("pt") TCBNN_F4_PAIR_MMA("pt")
                     TCBNN_F4_PAIR_TAIL : "=&r"(ok) : TCBNN_F4_PAIR_IN, "r"(bar0), "r"(par0), "r"(bar1), "r"(par1), "r"(bar_e),
                     "r"(bar_c) : "memory");
    else
        asm volatile(TCBNN_F4_PAIR_HEAD TCBNN_F4_PAIR_TEST TCBNN_F4_PAIR_MMA("pq") TCBNN_F4_PAIR_TAIL
                     : "=&r"(ok) : TCBNN_F4_PAIR_IN, "r"(bar0), "r"(par0), "r"(bar1), "r"(par1), "r"(bar_e), "r"(bar_c) : "memory");
    return ok;
}
#undef TCBNN_F4_PAIR_MMA
#undef TCBNN_F4_PAIR_HEAD
#undef TCBNN_F4_PAIR_TEST
#undef TCBNN_F4_PAIR_TAIL
#undef TCBNN_F4_PAIR_IN

template <bool PAIR>
__device__ __forceinline__ void gemm_umma_cta(const GemmUmmaArgs& g, const CUtensorMap* map_a, const CUtensorMap* map_w, unsigned char* smem) {
    constexpr int STAGE = kGemmStageBytes, NST = kGemmStages;
    constexpr int NACC = PAIR ? 1 : 2;                  // accumulators of 256 / 128 columns
    constexpr uint32_t TM_COLS = 512, SF_COL = TM_COLS - 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long tr_cta0 = clock64();
    uint64_t* sBar = reinterpret_cast<uint64_t*>(smem + (size_t)NST * STAGE);
    // barriers: full[NST] | empty[NST] | acc_full[NACC] | acc_empty[NACC] | drain
    uint32_t* sTmem = reinterpret_cast<uint32_t*>(sBar + 2 * NST + 2 * NACC + 1);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sTmem + 1);
    float* sThr = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(sTmem + 2) + 15) & ~(uintptr_t)15);
    const uint32_t bar0 = smem_u32(sBar);
    auto BAR_FULL = [&](int s) { return bar0 + 8u * s; };
    auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (NST + s); };
    auto BAR_CFULL = [&](int b) { return bar0 + 8u * (2 * NST + b); };
    auto BAR_CEMPTY = [&](int b) { return bar0 + 8u * (2 * NST + NACC + b); };
    const uint32_t BAR_DRAIN = bar0 + 8u * (2 * NST + 2 * NACC);

    // tile t = (split * tiles_m + tm) * tiles_n + tn; both count pairs when PAIR, and a pair of CTAs walks
    // over the tiles together
    const int rank = PAIR ? (int)(blockIdx.x & 1u) : 0;
    const int t_first = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, t_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    const int tiles_m = PAIR ? (g.MT + 1) >> 1 : g.MT, tiles_n = PAIR ? (g.NT + 1) >> 1 : g.NT;
    const int ntiles = tiles_m * tiles_n * g.splits;
    struct Tile { int tn, rt, split, kb0, kb1; };
    auto tile = [&](int t) {
        Tile q;
        const int r = t / tiles_n, n = t - r * tiles_n;
        q.split = r / tiles_m;
        const int m = r - q.split * tiles_m;
        q.kb0 = q.split * g.per;
        q.kb1 = min(g.KB, q.kb0 + g.per);
        q.rt = PAIR ? m * 2 + rank : m;                 // this CTA's 128-row tile of A
        q.tn = PAIR ? n * 2 : n;                        // first 128-column tile
        return q;
    };

    if (tid == 0) {
        for (int s = 0; s < NST; s++) { mbar_init(BAR_FULL(s), 2); mbar_init(BAR_EMPTY(s), 1); }
        for (int b = 0; b < NACC; b++) { mbar_init(BAR_CFULL(b), 1); mbar_init(BAR_CEMPTY(b), PAIR ? 16 : 8); }
        mbar_init(BAR_DRAIN, 1);
        *sAbort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(sTmem)), "r"(TM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            tmem_alloc(smem_u32(sTmem), TM_COLS);
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *sTmem;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (not before the allocation: see bconv_umma_pre.cuh)
    if (warp < 4) tmem_fill_unit_scales(tmem, SF_COL);
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();                 // the partner's barriers and scales are set up as well
    tc_fence_after();
    const typename std::conditional<PAIR, PairWait, WsWait>::type wait{sAbort, g.status};
    // Launched as a programmatic dependent of the expansion pass, the CTA has come this far while
    // that pass was still running; its units are complete (and visible) once this returns.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr uint32_t OFF_W = kGemmKU * kGemmUnit;     // W's place inside a stage
    const bool tr = g.trace != nullptr && blockIdx.x == 0;

    if (warp == 8 || warp == 10) {
        // =============================== loaders ============================================
        if (lane == 0) {
            const bool isw = warp == 10;
            int s = 0;
            uint32_t ph = 0, issued = 0;
            bool ok = true;
            long long tr_w = 0;
            for (int t = t_first; t < ntiles && ok; t += t_step) {
                const Tile q = tile(t);
                const int tile128 = isw ? q.tn + rank : q.rt;
                const bool exists = tile128 < (isw ? g.NT : g.MT);   // (else: sums that nobody stores)
                const unsigned char* src = (isw ? g.ew : g.ea) + (size_t)tile128 * g.KB * kGemmUnit;
                for (int kb = q.kb0; kb < q.kb1; kb += kGemmKU) {
                    const uint32_t bytes = (uint32_t)min(kGemmKU, q.kb1 - kb) * kGemmUnit;
                    ok = tr ? wait.timed(BAR_EMPTY(s), ph ^ 1, tr_w) : wait(BAR_EMPTY(s), ph ^ 1);
                    if (!ok) break;
                    if constexpr (PAIR) {
                        constexpr uint32_t kStage = kGemmKU * kGemmUnit;
                        if (rank == 0)                   // (the leader's tile always exists)
                            mbar_expect_tx(BAR_FULL(s), tile128 + 1 < (isw ? g.NT : g.MT) ? 2 * kStage : kStage);
                        if (exists)
                            tensor_g2s_pair(smem_u32(smem + (size_t)s * STAGE) + (isw ? OFF_W : 0u), isw ? map_w : map_a,
                                            (tile128 * g.KB + kb) * (kGemmUnit / 1024), leader_address(BAR_FULL(s)));
                    } else {
                        mbar_expect_tx(BAR_FULL(s), bytes);
                        bulk_g2s(smem_u32(smem + (size_t)s * STAGE) + (isw ? OFF_W : 0u), src + (size_t)kb * kGemmUnit, bytes, BAR_FULL(s));
                    }
                    issued++;
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
            }
            if (tr && !isw) g.trace[10] = tr_w;
            if (!ok) {
                // giving up: wait (bounded) for the copies still in flight before the CTA exits.  A
                // stage's barrier completes once both loaders' copies have landed; if the other
                // loader never got that far the polls run out, which takes longer than any copy.  (A pair's
                // second CTA cannot poll the leader's barriers: it lets that time pass.)
                for (int s2 = 0; s2 < NST; s2++) {
                    const bool this_pass = s2 < s;
                    if (!this_pass && issued < (uint32_t)NST) continue;
                    for (int i = 0; i < (PAIR ? 1 << 16 : 1 << 20); i++)
                        if (PAIR ? rank == 0 && mbar_test_cluster(BAR_FULL(s2), this_pass ? ph : ph ^ 1) : mbar_try_wait(BAR_FULL(s2), this_pass ? ph : ph ^ 1)) break;
                        else if (PAIR) __nanosleep(20);
                }
            }
        }
        __syncwarp();
    } else if (PAIR && warp == 9 && rank == 1) {
        __syncwarp();                                   // (the leader issues for both)
    } else if (warp == 9) {
        // =============================== MMA issuer =========================================
        // (what the next stage needs is worked out and asked for while this one's MMAs are queued: the
        // same scheme as in bconv_umma_pre.cuh, reasons there)
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t IDESC = PAIR ? idesc_f4(256) + ((128u >> 4) << 24) : idesc_f4(128);   // (M = 256: one step up)
        const uint64_t desc0 = smem_desc(smem_u32(smem), 128 * 16, 128u);
        const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0;
        constexpr uint32_t stepStage = STAGE >> 4, stepUnit = kGemmUnit >> 4, offW = OFF_W >> 4;
        const uint32_t units[4] = {0u, stepUnit, 2 * stepUnit, 3 * stepUnit};
        const uint32_t sfa = tmem + SF_COL, sfb = tmem + SF_COL + 16;
        uint32_t s = 0, ph = 0, b = 0, bph = 0, ready = 0, need = 3u;
        bool ok = true;
        long long tr_w = 0;
        const long long tr_t0 = clock64();
        int t = t_first, tr_kb = 0;
        Tile q = tile(t < ntiles ? t : 0);
        int kb = q.kb0;
        while (t < ntiles) {
            if ((ready & need) != need) {
                if ((need & 2u) && !(ready & 2u)) {
                    ok = wait.spin(BAR_CEMPTY(b), bph ^ 1);
                    if (!ok) break;
                }
                if (!(ready & 1u)) {
                    ok = tr ? wait.timed(BAR_FULL(s), ph, tr_w) : wait.spin(BAR_FULL(s), ph);
                    if (!ok) break;
                }
            }
            tc_fence_after();
            const int nkb = min(kGemmKU, q.kb1 - kb);
            uint32_t acc = kb > q.kb0 ? 1u : 0u;
            const uint32_t d = tmem + b * 128;
            uint32_t aLo = lo0 + s * stepStage, bLo = aLo + offW;
            if constexpr (PAIR) {
                for (int j = 0; j < (nkb == kGemmKU ? 1 : nkb - 1); j++) {
                    mma_f4_pair_run(leader, d, aLo + j * stepUnit, bLo + j * stepUnit, hi, stepUnit, IDESC, acc, sfa, sfb);
                    acc = 1;
                }
            } else if (nkb == kGemmKU) {
                mma_f4_run<1>(leader, d, aLo, hi, bLo, hi, stepUnit, units, IDESC, acc, sfa, sfb);
            } else {
                for (int j = 0; j + 1 < nkb; j++) {
                    const uint32_t o = j * stepUnit;
                    mma_f4_run<1>(leader, d, aLo, hi, bLo + o, hi, stepUnit, &o, IDESC, acc, sfa, sfb);
                    acc = 1;
                }
            }
            asm volatile("" : "+r"(s), "+r"(b), "+r"(ph), "+r"(bph), "+r"(kb));   // what follows stays behind those MMAs
            tr_kb += nkb;
            const bool last = kb + nkb >= q.kb1;
            const uint32_t sc = s, bc = b;
            s = s + 1 == (uint32_t)NST ? 0u : s + 1;
            ph ^= s == 0 ? 1u : 0u;
            if (last) {
                b = b + 1 == (uint32_t)NACC ? 0u : b + 1;
                bph ^= b == 0 ? 1u : 0u;
            }
            const uint32_t bar_c = last ? BAR_CFULL(bc) : 0u;
            need = last ? 3u : 1u;
            // (while a tile is being issued, its own accumulator is what bar1 names; the answer counts
            // only at the first stage of a tile)
            const uint32_t o = (nkb - 1) * stepUnit;
            if constexpr (PAIR) {
                if (nkb == kGemmKU)
                    ready = mma_f4_pair_end<3>(leader, d, aLo + stepUnit, bLo + stepUnit, hi, stepUnit, IDESC, 1u, sfa, sfb,
                                               BAR_FULL(s), ph, BAR_CEMPTY(b), bph ^ 1u, BAR_EMPTY(sc), bar_c);
                else
                    ready = mma_f4_pair_end<1>(leader, d, aLo + o, bLo + o, hi, stepUnit, IDESC, acc, sfa, sfb,
                                               BAR_FULL(s), ph, BAR_CEMPTY(b), bph ^ 1u, BAR_EMPTY(sc), bar_c);
            } else if (nkb == kGemmKU) {
                ready = mma_f4_end<3>(leader, d, aLo, hi, bLo + stepUnit, hi, stepUnit, units + 1, IDESC, 1u, sfa, sfb,
                                      BAR_FULL(s), ph, BAR_CEMPTY(b), bph ^ 1u, BAR_EMPTY(sc), bar_c);
            } else {
                ready = mma_f4_end<1>(leader, d, aLo, hi, bLo + o, hi, stepUnit, &o, IDESC, acc, sfa, sfb,
                                      BAR_FULL(s), ph, BAR_CEMPTY(b), bph ^ 1u, BAR_EMPTY(sc), bar_c);
            }
            if (last) {
                t += t_step;
                if (t < ntiles) { q = tile(t); kb = q.kb0; }
            } else {
                kb += kGemmKU;
            }
        }
        if (tr && leader) { g.trace[11] = clock64() - tr_t0; g.trace[12] = tr_w; g.trace[14] = tr_kb; }
        if (!ok && leader) {
            // giving up: the MMAs already issued must have finished before tensor memory is freed
            if constexpr (PAIR)
                asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(BAR_DRAIN) : "memory");
            else
                mma_commit(BAR_DRAIN);
            for (int i = 0; i < (1 << 20); i++)
                if (PAIR ? mbar_test_cluster(BAR_DRAIN, 0) : mbar_try_wait(BAR_DRAIN, 0)) break;
        }
        __syncwarp();
    } else if (warp < 8) {
        // =============================== epilogue ===========================================
        const int quad = warp & 3, q4 = lane & 3;
        long long tr_w = 0, tr_body = 0;
        int b = 0;
        uint32_t bph = 0;
        for (int t = t_first; t < ntiles; t += t_step) {
            const Tile q = tile(t);
            const int sub = PAIR ? warp >> 2 : 0;       // pair: a warpgroup per 128 columns; alone: per 64
            const int nb0 = PAIR ? 0 : (warp >> 2) * 2, nb1 = PAIR ? 4 : nb0 + 2;
            const int m0 = q.rt * 128 + quad * 32, tn = q.tn + sub;          // this warp's rows, its column tile
            const bool have = !PAIR || (q.rt < g.MT && tn < g.NT);
            // thresholds of this warp's columns, in the accumulator's column order, while it is awaited
            // (a threshold per column straight from global memory costs a trip to L2 each: 6800 clocks
            // per tile).  NaN behind the last column: never reached.
            float* const thr = sThr + warp * 128;
            if (g.splits == 1 && g.mode == GEMM_FC_BITS) {
                constexpr int NB = PAIR ? 4 : 2;
                float tv[NB];
#pragma unroll
                for (int i = 0; i < NB; i++) {           // (all on their way before the first is stored)
                    const int n = tn * 128 + (nb0 + i) * 32 + f4_channel_of_column(lane);
                    tv[i] = n < g.N ? ld_dep(g.p0 + n) : __int_as_float(0x7FC00000);
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < NB; i++) thr[(nb0 + i) * 32 + lane] = tv[i];
                __syncwarp();
            }
            const long long e0 = clock64();
            if (!wait.relaxed(BAR_CFULL(b), bph)) break;
            const long long e1 = clock64();
            tr_w += e1 - e0;
            tc_fence_after();
            const uint32_t tcol = tmem + ((uint32_t)(quad * 32) << 16) + b * 128 + sub * 128;
            if (have) {
                const bool ints = g.splits > 1 || g.mode == GEMM_INT32;
                if (!ints && g.mode == GEMM_FC_BITS) {
                    const int m = m0 + lane;
#pragma unroll 1
                    for (int nb = nb0; nb < nb1; nb++) {
                        const int n0 = tn * 128 + nb * 32;
                        if (n0 >= g.N) break;
                        int v[32];
                        tmem_ld32(tcol + nb * 32, v);
                        tmem_ld_wait();
                        // (float)K - 2*(float)c >= thr[n] (kernel.cuh:210-213): the accumulator is that value
                        uint32_t word = 0;
                        const float4* t4 = reinterpret_cast<const float4*>(thr + nb * 32);
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const float4 th = t4[j];
                            if (__int_as_float(v[4 * j]) >= th.x) word |= 0x80000000u >> f4_channel_of_column(4 * j);
                            if (__int_as_float(v[4 * j + 1]) >= th.y) word |= 0x80000000u >> f4_channel_of_column(4 * j + 1);
                            if (__int_as_float(v[4 * j + 2]) >= th.z) word |= 0x80000000u >> f4_channel_of_column(4 * j + 2);
                            if (__int_as_float(v[4 * j + 3]) >= th.w) word |= 0x80000000u >> f4_channel_of_column(4 * j + 3);
                        }
                        if (m < g.M) {
                            reinterpret_cast<uint32_t*>(g.out)[(size_t)m * g.ldo + (n0 >> 5)] = word;
                            if (g.nxt) store_unit_chunk(g.nxt, g.nxt_KB, m, n0 >> 5, word, g.N - n0);
                        }
                    }
                } else {
                    // int32 sums (the split-K partials, or C itself), or scale and bias (kernel.cuh:270-273,
                    // fused multiply-add): rows of four consecutive columns per lane
                    uint32_t* dst = g.splits > 1 ? reinterpret_cast<uint32_t*>(g.partial) + (size_t)q.split * g.M * g.N
                                                 : reinterpret_cast<uint32_t*>(g.out);
                    const int ld = g.splits > 1 ? g.N : g.ldo;
                    const bool v4 = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll 1
                    for (int nb = nb0; nb < nb1; nb++) {
                        const int n0 = tn * 128 + nb * 32 + 4 * q4;
                        float4 sc[2], bi[2];
                        if (!ints) {
#pragma unroll
                            for (int gg = 0; gg < 2; gg++) {
                                const int n = n0 + 16 * gg;
                                sc[gg] = make_float4(n < g.N ? ld_dep(g.p0 + n) : 0.f, n + 1 < g.N ? ld_dep(g.p0 + n + 1) : 0.f,
                                                     n + 2 < g.N ? ld_dep(g.p0 + n + 2) : 0.f, n + 3 < g.N ? ld_dep(g.p0 + n + 3) : 0.f);
                                bi[gg] = make_float4(n < g.N ? ld_dep(g.p1 + n) : 0.f, n + 1 < g.N ? ld_dep(g.p1 + n + 1) : 0.f,
                                                     n + 2 < g.N ? ld_dep(g.p1 + n + 2) : 0.f, n + 3 < g.N ? ld_dep(g.p1 + n + 3) : 0.f);
                            }
                        }
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            int v[16];
                            tmem_ld_16x256b_x4(tcol + ((uint32_t)(16 * h) << 16) + nb * 32, v);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 2; i++) {
                                const int m = m0 + 16 * h + 8 * i + (lane >> 2);
                                if (m >= g.M) continue;
#pragma unroll
                                for (int gg = 0; gg < 2; gg++) {
                                    const int n = n0 + 16 * gg;
                                    const int r0 = v[8 * gg + 2 * i], r1 = v[8 * gg + 2 * i + 1];
                                    const int r2 = v[8 * gg + 4 + 2 * i], r3 = v[8 * gg + 4 + 2 * i + 1];
                                    uint4 w;
                                    if (ints)
                                        w = make_uint4((uint32_t)f4_acc_to_int(r0), (uint32_t)f4_acc_to_int(r1),
                                                       (uint32_t)f4_acc_to_int(r2), (uint32_t)f4_acc_to_int(r3));
                                    else
                                        w = make_uint4(__float_as_uint(fmaf(__int_as_float(r0), sc[gg].x, bi[gg].x)),
                                                       __float_as_uint(fmaf(__int_as_float(r1), sc[gg].y, bi[gg].y)),
                                                       __float_as_uint(fmaf(__int_as_float(r2), sc[gg].z, bi[gg].z)),
                                                       __float_as_uint(fmaf(__int_as_float(r3), sc[gg].w, bi[gg].w)));
                                    uint32_t* o = dst + (size_t)m * ld + n;
                                    if (v4 && n + 3 < g.N) {
                                        *reinterpret_cast<uint4*>(o) = w;
                                    } else {
                                        if (n < g.N) o[0] = w.x;
                                        if (n + 1 < g.N) o[1] = w.y;
                                        if (n + 2 < g.N) o[2] = w.z;
                                        if (n + 3 < g.N) o[3] = w.w;
                                    }
                                }
                            }
                        }
                    }
                }
            }
            tc_fence_before();                          // this warp is done with the accumulator
            __syncwarp();
            if (lane == 0) { if constexpr (PAIR) mbar_arrive_leader(BAR_CEMPTY(b)); else mbar_arrive(BAR_CEMPTY(b)); }
            tr_body += clock64() - e1;
            if (++b == NACC) { b = 0; bph ^= 1u; }
        }
        if (tr && tid == 0) { g.trace[13] = tr_w; g.trace[15] = tr_body; }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) {
        cluster_sync();                                 // nothing of the partner's reaches into this CTA any more
        if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM_COLS) : "memory");
    } else if (warp == 9) {
        tmem_dealloc(tmem, TM_COLS);
    }
    if (g.trace != nullptr && blockIdx.x == 0 && tid == 0) g.trace[9] = clock64() - tr_cta0;
}

}  // namespace umma
}  // namespace tcbnn
