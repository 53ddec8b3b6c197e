// Bit GEMM on tcgen05, fed from the packed bits: the arithmetic of bgemm_umma.cuh (tcgen05.mma kind::mxf4 on
// +-1 nibbles with unit block scales), with the bits expanded inside the GEMM instead of by a pass in
// front of it -- one launch, no scratch, and an eighth of the operand traffic.
//
// The roles of the operands are turned round: the MMA's 128 rows are rows of W (outputs), its columns rows
// of A (the batch).  W's rows are expanded straight into tensor memory (a lane per row, the MMA's A operand
// read from there), A's into shared memory.  Why so: the shared-memory port, 128 bytes per clock, is what
// bounds a GEMM whose operands both come through it (bgemm_umma.cuh: 136 clocks per 64-deep step of a 128 x 128
// tile whose MMA takes 64).  With one operand in tensor memory a step of 128 x n moves 32 n bytes in and
// 32 n out, n / 2 clocks together: the MMA's own time.  And with an output per lane, threshold, scale and
// bias are one register, integers and floats leave as whole lines, and n can be any multiple of 32: few
// rows cost few columns, and tiles can be cut to fill the last wave.
//
//   warps 0-7   epilogue    : lane = output; 32 x 32 blocks of bits are turned with shuffles
//   warps 8-15  W expanders : two groups of four (a warp reaches a quarter of the lanes), stages in turn
//   warps 16-23 A expanders : 32 rows each, in as many groups as fit, stages in turn
//   warp  24    MMA         : converged, elected lane
//
// A stage is 512 bits of K, 64 bytes of a row, which four lanes fetch together (cp.async): what the loads cost is
// the lines they touch, about two clocks each (a lane per row, 32 lines an instruction, took 1890 clocks per
// 256 bits of a 256-column tile whose MMAs take 512).  Each expander keeps two tiles of 32 rows in flight or in
// hand, in shared memory.  A stage costs 0.46 us at 32 and 64 columns, where an expander of W needs 1000 clocks for 112
// logic operations and 16 KB into tensor memory, and 0.95 at 256 (1024 clocks of MMAs), where only two stages fit and
// their hand-overs show.  Masking every word for the end of K, if-converted by the compiler, had doubled the expanders' time.
//
// Measured in one launch of a graph, before (expansion pass and GEMM, or the b1 kernel) and here: 1024 x 1024 x 4096
// 10.2 -> 8.4 us, 1024 x 25088 -> 512 21.0 -> 16.0, 32 x 25088 -> 4096 25.9 -> 12.5, 1024 x 512 -> 1000 11.2 -> 5.0, 2000 x 3000 x 64
// 41 -> 13, 4000 x 200 -> 8192 224 -> 23; 8192 x 8192 x 8192 173 -> 224, which is why large ones stay where they were.
//
// Where the tiles of M x N leave SMs idle, K is cut over a cluster's CTAs, whose sums meet in the first shared
// memory that the loop no longer needs; each CTA then finishes its share of the columns.
#pragma once
#include "bgemm_umma.cuh"

namespace tcbnn {
namespace umma {

constexpr int kBitsThreads = 800;
constexpr int kBitsMaxCols = 256;
constexpr int kBitsMaxStages = 6;
// 64 bits of K of A's rows, two planes of 16 bytes a row; the 16 bytes behind keep the four lanes of a row in
// different banks
__host__ __device__ inline uint32_t bits_unit(int cols) { return (uint32_t)cols * 32u + 16u; }
// 32 rows of a stage as they are fetched, and how many of them an expander has in flight or in hand
constexpr uint32_t kBitsTile = 2048;
constexpr int kBitsAhead = 2;
constexpr uint32_t kBitsRaw = 16 * kBitsAhead * kBitsTile;
// accumulators in front of W's ring in tensor memory (64 columns per stage), and the stages that the ring and
// shared memory hold
__host__ __device__ inline int bits_accumulators(int cols, int splits) { return splits == 1 && cols <= 128 ? 2 : 1; }
__host__ __device__ inline int bits_stages(int cols, int splits) {
    int n = (480 - bits_accumulators(cols, splits) * cols) / 64;
    while (n > 2 && n * 8 * bits_unit(cols) + kBitsRaw > 226 * 1024) n--;
    return n < kBitsMaxStages ? n : kBitsMaxStages;
}

struct GemmBitsArgs {
    const uint32_t* A; const uint32_t* W;              // [M][lda], [N][ldw] words; rows 16-byte aligned
    int M, N, K, lda, ldw;
    int cols;                                          // rows of A per tile: the MMA's N, a multiple of 32
    int tiles_m, tiles_n;                              // tiles of A's rows and of W's
    int stages, per;                                   // stages of K; per CTA of a cluster (none without any)
    int mode; void* out; int ldo; const float* p0; const float* p1;
    uint4* nxt; int nxt_KB;                            // threshold bits also expanded (store_unit_chunk), or null
    int settled;                                       // GemmArgs::settled
    int* status;
};
// (clusters exchange their sums through the ring)
__host__ __device__ inline size_t bits_ring_bytes(int cols, int splits) {
    const size_t ring = (size_t)bits_stages(cols, splits) * 8 * bits_unit(cols), sums = splits > 1 ? (size_t)cols * 512 : 0;
    return ((ring > sums ? ring : sums) + 127) & ~(size_t)127;
}
__host__ __device__ inline size_t bits_smem_bytes(int cols, int splits) { return bits_ring_bytes(cols, splits) + kBitsRaw + 32 * 8 + 64; }

// D[tmem] (+)= A[tmem] * B[smem desc], the unit scales at sf
__device__ __forceinline__ void mma_f4_ts(uint32_t leader, uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                          uint32_t sf, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred pa, pl;\n\t.reg .b64 db;\n\tmov.b64 db, {%2, %3};\n\tsetp.ne.b32 pa, %6, 0;\n\tsetp.ne.b32 pl, %7, 0;\n\t"
        "@pl tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%0], [%1], db, %4, [%5], [%5], pa;\n\t}"
        ::"r"(d), "r"(a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(sf), "r"(acc), "r"(leader) : "memory");
}
// Eight of them, A 8 columns and B `step` on each time, written as one block with the test of a barrier in front whose
// answer is read behind (see mma_f4_end): the issuing warp shares its scheduler with six that expand, and what it does
// between two MMAs is time the tensor pipe idles.
#define TCBNN_TS_MMA(PRED)                                                                           \
    "mov.b64 db, {xb, %4};\n\t"                                                                     \
    "@pl tcgen05.mma.cta_group::1.kind::mxf4.block_scale.block32 [%1], [xa], db, %5, [%6], [%6], " PRED ";\n\t" \
    "add.u32 xa, xa, 8;\n\tadd.u32 xb, xb, %9;\n\t"
__device__ __forceinline__ uint32_t mma_f4_ts_run8(uint32_t leader, uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t step,
                                                   uint32_t idesc, uint32_t sf, uint32_t acc, uint32_t next_bar, uint32_t next_parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred pa, pl, pt, p0;\n\t.reg .b64 db;\n\t.reg .b32 xa, xb;\n\t"
                 "setp.ne.b32 pa, %7, 0;\n\tsetp.ne.b32 pl, %8, 0;\n\tsetp.eq.b32 pt, %8, %8;\n\tmov.u32 xa, %2;\n\tmov.u32 xb, %3;\n\t"
                 TCBNN_TS_MMA("pa") TCBNN_TS_MMA("pt") TCBNN_TS_MMA("pt") TCBNN_TS_MMA("pt")
                 "mbarrier.test_wait.parity.shared::cta.b64 p0, [%10], %11;\n\t"
                 TCBNN_TS_MMA("pt") TCBNN_TS_MMA("pt") TCBNN_TS_MMA("pt") TCBNN_TS_MMA("pt") "selp.u32 %0, 1, 0, p0;\n\t}"
                 : "=&r"(ok) : "r"(d), "r"(a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(sf), "r"(acc), "r"(leader), "r"(step), "r"(next_bar),
                   "r"(next_parity) : "memory");
    return ok;
}
#undef TCBNN_TS_MMA
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4& a, const uint4& b) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}
__device__ __forceinline__ float4 ld_peer4(uint32_t shared, uint32_t rank) {
    uint32_t p;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(p) : "r"(shared), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p) : "memory");
    return v;
}
// 32 x 32 bits over a warp: bit 31 - i of lane j becomes bit 31 - j of lane i
__device__ __forceinline__ uint32_t transpose_bits(uint32_t w) {
    const int lane = threadIdx.x & 31;
    uint32_t mask = 0x0000FFFFu;
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const uint32_t o = __shfl_xor_sync(0xffffffffu, w, s);
        // lanes with bit s clear keep their high halves and take the partner's high halves as low ones
        w = (lane & s) ? (((o & mask) << s) | (w & mask)) : ((w & ~mask) | ((o & ~mask) >> s));
        mask ^= mask << (s >> 1);
    }
    return w;
}

// A stage of 32 rows, 64 bytes each, in 2 KB of shared memory: four 16-byte pieces a row, their order turned
// by the row so that neither a row's lanes nor a piece's have bank conflicts.
__device__ __forceinline__ uint32_t bits_piece(uint32_t tile, int row, int piece) { return tile + row * 64 + ((piece ^ ((row >> 1) & 3)) << 4); }
// Lane l asks for piece l % 4 of rows l / 4 + 8 i.  Words behind the rows' end and rows past the last one are zeros,
// for which nothing is read.  (The last row again instead: with 10 outputs every SM read the same line 118 times,
// 8192 x 1024 -> 10 6 -> 21 us.)
struct BitsSource {
    const uint32_t* row[4];
    int ld;
    __device__ __forceinline__ void set(const uint32_t* bits, int row0, int rows, int ld_) {
        const int lane = threadIdx.x & 31;
        ld = ld_;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = row0 + (lane >> 2) + 8 * i;
            row[i] = r < rows ? bits + (size_t)r * ld_ : nullptr;
        }
    }
    __device__ __forceinline__ void ask(uint32_t tile, int stage, const uint32_t* any) const {
        const int lane = threadIdx.x & 31, word = stage * 16 + (lane & 3) * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool in = row[i] && word < ld;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(bits_piece(tile, (lane >> 2) + 8 * i, lane & 3)),
                         "l"(in ? row[i] + word : any), "r"(in ? 16 : 0) : "memory");
        }
    }
};
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint4 (&e)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(e[0].x), "r"(e[0].y), "r"(e[0].z), "r"(e[0].w), "r"(e[1].x), "r"(e[1].y), "r"(e[1].z), "r"(e[1].w),
                   "r"(e[2].x), "r"(e[2].y), "r"(e[2].z), "r"(e[2].w), "r"(e[3].x), "r"(e[3].y), "r"(e[3].z), "r"(e[3].w),
                   "r"(e[4].x), "r"(e[4].y), "r"(e[4].z), "r"(e[4].w), "r"(e[5].x), "r"(e[5].y), "r"(e[5].z), "r"(e[5].w),
                   "r"(e[6].x), "r"(e[6].y), "r"(e[6].z), "r"(e[6].w), "r"(e[7].x), "r"(e[7].y), "r"(e[7].z), "r"(e[7].w) : "memory");
}
// row `lane` of a stage, expanded, into tensor memory: eight columns per 64 bits, of which `kblocks` are wanted
__device__ __forceinline__ void bits_to_tmem(uint32_t dst, const uint4 (&w)[4], int kblocks) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (4 * h >= kblocks) break;
        const uint4 e[8] = {expand32_f4(w[2 * h].x), expand32_f4(w[2 * h].y), expand32_f4(w[2 * h].z), expand32_f4(w[2 * h].w),
                            expand32_f4(w[2 * h + 1].x), expand32_f4(w[2 * h + 1].y), expand32_f4(w[2 * h + 1].z), expand32_f4(w[2 * h + 1].w)};
        if (4 * h + 4 <= kblocks) {
            tmem_st32(dst + h * 32, e);
        } else {
#pragma unroll
            for (int i = 0; i < 3; i++)
                if (4 * h + i < kblocks) tmem_st8(dst + h * 32 + i * 8, e[2 * i], e[2 * i + 1]);
        }
    }
}

template <bool CLUSTER>
__device__ __forceinline__ void gemm_bits_cta(const GemmBitsArgs& g, unsigned char* smem) {
    constexpr uint32_t TM_COLS = 512, SF_COL = TM_COLS - 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t nctas = CLUSTER ? [] { uint32_t n; asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n)); return n; }() : 1u;
    const uint32_t rank = CLUSTER ? [] { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }() : 0u;
    const int nacc = bits_accumulators(g.cols, (int)nctas), NST = bits_stages(g.cols, (int)nctas);
    const uint32_t unit = bits_unit(g.cols), stage_bytes = 8 * unit;
    const uint32_t ring_col = (uint32_t)(nacc * g.cols);                 // W's ring in tensor memory
    unsigned char* sRaw = smem + bits_ring_bytes(g.cols, (int)nctas);
    uint64_t* sBar = reinterpret_cast<uint64_t*>(sRaw + kBitsRaw);
    // barriers: full[NST] | empty[NST] | acc_full[2] | acc_empty[2] | drain
    uint32_t* sTmem = reinterpret_cast<uint32_t*>(sBar + 2 * NST + 5);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sTmem + 1);
    const uint32_t bar0 = smem_u32(sBar);
    auto BAR_FULL = [&](int s) { return bar0 + 8u * s; };
    auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (NST + s); };
    auto BAR_CFULL = [&](int b) { return bar0 + 8u * (2 * NST + b); };
    auto BAR_CEMPTY = [&](int b) { return bar0 + 8u * (2 * NST + 2 + b); };
    const uint32_t BAR_DRAIN = bar0 + 8u * (2 * NST + 4);

    const int t_first = CLUSTER ? (int)(blockIdx.x / nctas) : (int)blockIdx.x, t_step = CLUSTER ? (int)(gridDim.x / nctas) : (int)gridDim.x;
    const int ntiles = g.tiles_m * g.tiles_n;
    const int st0 = (int)rank * g.per, nst = max(0, min(g.per, g.stages - st0));          // this CTA's stages of K
    const int KB = (g.K + 63) >> 6;
    // A expanders: warps per 32 rows of the tile, and the groups that take stages in turn
    // (No more than NST groups: a group that waits for a slot has seen the release before last then, and
    // the barrier's parity names the last.)
    const int blocks = g.cols >> 5, width = blocks <= 2 ? 2 : blocks <= 4 ? 4 : 8, agroups = min(8 / width, NST);

    if (tid == 0) {
        for (int s = 0; s < NST; s++) { mbar_init(BAR_FULL(s), 4 + blocks); mbar_init(BAR_EMPTY(s), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(BAR_CFULL(b), 1); mbar_init(BAR_CEMPTY(b), 8); }
        mbar_init(BAR_DRAIN, 1);
        *sAbort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 24) tmem_alloc(smem_u32(sTmem), TM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *sTmem;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (not before the allocation: see bconv_umma_pre.cuh)
    if (warp < 4) tmem_fill_unit_scales(tmem, SF_COL);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const WsWait wait{sAbort, g.status};
    // W's expanders, and the epilogue's parameters, need not wait for the launch in front where nothing that it waited
    // for can still write them; what is stored waits all the same, for sums that need A.
    if (!g.settled || warp >= 16) asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp >= 8 && warp < 24) {
        // =============================== expanders ==========================================
        const bool isw = warp < 16;
        const int group = isw ? (warp - 8) >> 2 : (warp - 16) / width, groups = isw ? 2 : agroups;
        const int block = isw ? warp & 3 : (warp - 16) & (width - 1);
        const int ld = isw ? g.ldw : g.lda, rows = isw ? g.N : g.M;
        const uint32_t* bits = isw ? g.W : g.A;
        // position in the CTA's sequence of (tile, stage), `groups` at a time
        struct Pos { int t, st; };
        auto settle = [&](Pos& p) { while (p.st >= nst && p.t < ntiles) { p.st -= nst; p.t += t_step; } };
        const uint32_t raw = smem_u32(sRaw) + (uint32_t)(warp - 8) * kBitsAhead * kBitsTile;
        BitsSource src;
        int src_t = -1;                                  // the tile whose rows src names
        auto ask = [&](Pos& p, int slot) {               // p: the position to ask for next
            if (p.t < ntiles) {
                if (p.t != src_t) {
                    src_t = p.t;
                    const int tm = p.t / g.tiles_n, tn = p.t - tm * g.tiles_n;
                    src.set(bits, (isw ? tn * 128 : tm * g.cols) + block * 32, rows, ld);
                }
                src.ask(raw + slot * kBitsTile, st0 + p.st, bits);
                p.st += groups;
                settle(p);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (nst > 0 && block < (isw ? 4 : blocks) && group < groups) {
            Pos p{t_first, group};
            settle(p);
            Pos next = p;
            for (int i = 0; i < kBitsAhead; i++) ask(next, i);
            int s = group, slot = 0;
            uint32_t ph = 0;
            while (p.t < ntiles) {
                const int st = st0 + p.st;
                asm volatile("cp.async.wait_group %0;" ::"n"(kBitsAhead - 1) : "memory");
                __syncwarp();
                uint4 w[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    w[i] = lds128(isw ? bits_piece(raw + slot * kBitsTile, lane, i) : bits_piece(raw + slot * kBitsTile, (lane >> 2) + 8 * i, lane & 3));
                __syncwarp();
                ask(next, slot);
                slot = slot + 1 == kBitsAhead ? 0 : slot + 1;
                if (!wait(BAR_EMPTY(s), ph ^ 1)) break;
                if (isw) {
                    tc_fence_after();
                    bits_to_tmem(tmem + ((uint32_t)(block * 32) << 16) + ring_col + s * 64, w, KB - st * 8);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                } else {
                    // piece q of a row: 64-bit blocks 2q and 2q + 1
                    const int q = lane & 3, left = g.K - st * 512 - q * 128;      // bits of this piece that exist; the rest is 0, not -1
                    const uint32_t dst = smem_u32(smem) + s * stage_bytes + 2 * q * unit + (uint32_t)(block * 32 + (lane >> 2)) * 16u;
                    const uint32_t plane = (uint32_t)g.cols * 16u;
                    auto store = [&](int i, int j, const uint4& e) {
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (j >> 1) * unit + (j & 1) * plane + i * 128u),
                                     "r"(e.x), "r"(e.y), "r"(e.z), "r"(e.w) : "memory");
                    };
                    if (g.K - st * 512 >= 512) {         // (of the warp: all of the stage exists)
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            store(i, 0, expand32_f4(w[i].x)); store(i, 1, expand32_f4(w[i].y));
                            store(i, 2, expand32_f4(w[i].z)); store(i, 3, expand32_f4(w[i].w));
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const int valid = left - j * 32;
                            const uint32_t keep = valid >= 32 ? 0xFFFFFFFFu : valid <= 0 ? 0u : 0xFFFFFFFFu << (32 - valid);
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                store(i, j, keep32_f4(expand32_f4(j == 0 ? w[i].x : j == 1 ? w[i].y : j == 2 ? w[i].z : w[i].w), keep));
                        }
                    }
                    fence_proxy_async();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR_FULL(s));
                p.st += groups;
                settle(p);
                s += groups;
                if (s >= NST) { s -= NST; ph ^= 1; }     // (groups <= NST)
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");          // (where it gave up: nothing may land behind the CTA's end)
        }
        __syncwarp();
    } else if (warp == 24) {
        // =============================== MMA issuer =========================================
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t idesc = idesc_f4(g.cols), sf = tmem + SF_COL;
        const uint64_t desc0 = smem_desc(smem_u32(smem), (uint32_t)g.cols * 16u, 128u);
        const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0, step = unit >> 4;
        int s = 0, b = 0;
        uint32_t ph = 0, bph = 0, ready = 0;             // ready: this stage is known to be full
        bool ok = true;
        if (nst > 0)
            for (int t = t_first; t < ntiles && ok; t += t_step) {
                ok = wait.spin(BAR_CEMPTY(b), bph ^ 1);
                if (!ok) break;
                const uint32_t d = tmem + b * g.cols;
                for (int st = 0; st < nst; st++) {
                    if (!ready) ok = wait.spin(BAR_FULL(s), ph);
                    if (!ok) break;
                    tc_fence_after();
                    uint32_t a = tmem + ring_col + s * 64, lo = lo0 + (s * stage_bytes >> 4);
                    const int nkb = min(8, KB - (st0 + st) * 8), sn = s + 1 == NST ? 0 : s + 1;
                    ready = 0;
                    if (nkb == 8)
                        ready = mma_f4_ts_run8(leader, d, a, lo, hi, step, idesc, sf, st > 0, BAR_FULL(sn), sn ? ph : ph ^ 1u);
                    else
                        for (int j = 0; j < nkb; j++, a += 8, lo += step) mma_f4_ts(leader, d, a, lo, hi, idesc, sf, st > 0 || j > 0);
                    if (leader) {
                        mma_commit(BAR_EMPTY(s));
                        if (st + 1 == nst) mma_commit(BAR_CFULL(b));
                    }
                    __syncwarp();
                    if (++s == NST) { s = 0; ph ^= 1; }
                }
                if (++b == nacc) { b = 0; bph ^= 1; }
            }
        if (!ok && leader) {
            // giving up: the MMAs already issued must have finished before tensor memory is freed
            mma_commit(BAR_DRAIN);
            for (int i = 0; i < (1 << 20); i++)
                if (mbar_try_wait(BAR_DRAIN, 0)) break;
        }
        __syncwarp();
    } else if (warp < 8) {
        // =============================== epilogue ===========================================
        const int quad = warp & 3, half = warp >> 2;
        int b = 0;
        uint32_t bph = 0;
        bool ok = true;
        for (int t = t_first; t < ntiles && ok; t += t_step) {
            const int tm = t / g.tiles_n, tn = t - tm * g.tiles_n;
            const int n = tn * 128 + quad * 32 + lane;                   // this lane's output
            float p0 = 0.f, p1 = 0.f;
            // (NaN behind the last output: its bit is 0)
            if (g.mode == GEMM_FC_BITS) p0 = n < g.N ? ld_dep(g.p0 + n) : __int_as_float(0x7FC00000);
            if (g.mode == GEMM_OUT_AFFINE && n < g.N) { p0 = ld_dep(g.p0 + n); p1 = ld_dep(g.p1 + n); }
            if (nst > 0) ok = wait.relaxed(BAR_CFULL(b), bph);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tcol = tmem + ((uint32_t)(quad * 32) << 16) + b * g.cols;
            for (int c0 = half * 32; c0 < g.cols; c0 += 64) {
                const int m0 = tm * g.cols + c0;
                if (!CLUSTER && m0 >= g.M) break;
                int v[32];
                tmem_ld32(tcol + c0, v);
                tmem_ld_wait();
                if constexpr (CLUSTER) {
                    // sums for the cluster: [four columns][128 outputs][4]
                    float4* dst = reinterpret_cast<float4*>(smem) + (size_t)(c0 >> 2) * 128 + quad * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 8; j++)
                        dst[j * 128] = make_float4(__int_as_float(v[4 * j]), __int_as_float(v[4 * j + 1]), __int_as_float(v[4 * j + 2]), __int_as_float(v[4 * j + 3]));
                } else if (g.mode == GEMM_FC_BITS) {
                    uint32_t w = 0;                                      // (float)K - 2*(float)c >= thr[n] (kernel.cuh:210-213)
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (__int_as_float(v[j]) >= p0) w |= 0x80000000u >> j;
                    w = transpose_bits(w);                               // now: row m0 + lane, 32 outputs
                    const int m = m0 + lane, word = tn * 4 + quad;
                    if (m < g.M && word * 32 < g.N) {
                        reinterpret_cast<uint32_t*>(g.out)[(size_t)m * g.ldo + word] = w;
                        if (g.nxt) store_unit_chunk(g.nxt, g.nxt_KB, m, word, w, g.N - word * 32);
                    }
                } else if (n < g.N) {
                    uint32_t* dst = reinterpret_cast<uint32_t*>(g.out) + (size_t)m0 * g.ldo + n;
                    const int rows = min(32, g.M - m0);
#pragma unroll
                    for (int j = 0; j < 32; j++)                         // integers, or scale and bias (kernel.cuh:270-273)
                        if (j < rows) dst[(size_t)j * g.ldo] = g.mode == GEMM_INT32 ? (uint32_t)f4_acc_to_int(v[j])
                                                                                   : __float_as_uint(fmaf(__int_as_float(v[j]), p0, p1));
                }
            }
            tc_fence_before();                                           // this warp is done with the accumulator
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_CEMPTY(b));
            if (++b == nacc) { b = 0; bph ^= 1; }
        }
    }
    tc_fence_before();
    if constexpr (CLUSTER) {
        // One tile per cluster: every CTA finishes each nctas-th group of four columns.
        cluster_sync();
        if (warp < 8 && !*sAbort) {
            const int quad = warp & 3, half = warp >> 2, t = t_first, tm = t / g.tiles_n, tn = t - tm * g.tiles_n;
            const int n = tn * 128 + quad * 32 + lane, word = tn * 4 + quad;
            float p0 = 0.f, p1 = 0.f;
            if (g.mode == GEMM_FC_BITS) p0 = n < g.N ? ld_dep(g.p0 + n) : __int_as_float(0x7FC00000);
            if (g.mode == GEMM_OUT_AFFINE && n < g.N) { p0 = ld_dep(g.p0 + n); p1 = ld_dep(g.p1 + n); }
            const int cols = min(g.cols, g.M - tm * g.cols);
            const uint32_t src = smem_u32(smem) + (uint32_t)(quad * 32 + lane) * 16u;
            for (int c = 4 * ((int)rank + half * (int)nctas); c < cols; c += 8 * (int)nctas) {
                float4 part[8];
#pragma unroll
                for (uint32_t r = 0; r < 8; r++) part[r] = r < nctas ? ld_peer4(src + (uint32_t)c * 512u, r) : make_float4(0.f, 0.f, 0.f, 0.f);
                float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int r = 0; r < 8; r++) { v[0] += part[r].x; v[1] += part[r].y; v[2] += part[r].z; v[3] += part[r].w; }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int m = tm * g.cols + c + j;
                    if (g.mode == GEMM_FC_BITS) {
                        const uint32_t w = __brev(__ballot_sync(0xffffffffu, v[j] >= p0));
                        if (lane == 0 && c + j < cols && word * 32 < g.N) {
                            reinterpret_cast<uint32_t*>(g.out)[(size_t)m * g.ldo + word] = w;
                            if (g.nxt) store_unit_chunk(g.nxt, g.nxt_KB, m, word, w, g.N - word * 32);
                        }
                    } else if (n < g.N && c + j < cols) {
                        reinterpret_cast<uint32_t*>(g.out)[(size_t)m * g.ldo + n] =
                            g.mode == GEMM_INT32 ? (uint32_t)f4_acc_to_int(__float_as_int(v[j])) : __float_as_uint(fmaf(v[j], p0, p1));
                    }
                }
            }
            __syncwarp();
        }
        cluster_sync();                                                  // nobody reads this CTA's sums any more
    }
    __syncthreads();
    if (warp == 24) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace umma
}  // namespace tcbnn
