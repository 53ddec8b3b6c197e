// A whole MLP on a few rows in one launch: input packing, hidden FC layers and the output layer
// (In128LayerFMT, Fc128LayerFMT, Out128LayerFMT: kernel.cuh:153-280) by a cluster of eight CTAs per 16, 32 or 64 rows.
//
// A CTA owns 128 outputs of every layer.  Its weights are expanded into tensor memory (the MMA's A operand,
// bgemm_bits.cuh) while the input is still being packed and earlier layers run; a layer is a dozen MMAs of 128 x
// rows x 64, and its bits go as +-1 nibbles straight into the shared memory of the eight CTAs (st.async: the store
// itself completes the receiver's barrier, no release at cluster scope, which takes over a thousand clocks).
// What bounds it is that chain: 9000 clocks until the input has arrived everywhere (more of a cluster's rows, more of it), then 2700 a layer
// (16 MMAs at 80, reading the accumulator, turning its bits, sending them).  GPU time of MLP 784 -> 1024 -> 1024 -> 1024 -> 10, five
// launches (weights read ahead, operands packed) against this one: 64 rows 11.4 and 12.2 us, 100 14.8 and 12.5, 200 14.1 and 12.6, 400
// 15.6 and 15.2, 700 15.8 and 19.4; 256 -> 256 -> 256 -> 256 -> 10 on 100 rows 11.9 and 9.9; 784 -> 10 on 700 4.1 and 10.7.  So it is taken
// where an estimate of both says so (chain_pays).  8 rows 8.5 and 11.7: fewer than 64 stay with the layers' launches.
//
//   warps 0-3   epilogue of a quarter of the CTA's outputs each
//   warps 4-19  W expanders : four groups of four, 512 bits of K in turn
//   warp  20    MMA         : converged, elected lane
//   warps 0-19  pack the input first
#pragma once
#include "bgemm_bits.cuh"

namespace tcbnn {
namespace umma {

constexpr int kChainCtas = 8, kChainMaxLayers = 8, kChainGroups = 4;
constexpr int kChainThreads = (4 + 4 * kChainGroups + 1) * 32;
struct ChainLayer {
    const uint32_t* W; int ldw, K, N;      // [N][ldw] packed weights, rows 16-byte aligned
    const float* p0; const float* p1;      // thresholds | scale, bias of the last layer
    void* out; int ldo;                    // bit words | float [M][ldo] of the last layer
    int col, after;                        // first column of its weights in tensor memory; free once layer `after` is done (-1: from the start)
};
struct ChainArgs {
    const float* x; int M, K, ld; uint32_t* bits;        // input rows, packed to bits[M][ld]
    int rows;                                            // per cluster: 16, 32 or 64
    int n, units;                                        // layers; 64-bit blocks of the longest K
    ChainLayer layer[kChainMaxLayers];
    int* status;
};
__host__ __device__ inline size_t chain_smem_bytes(int rows, int units) {
    return (size_t)2 * units * rows * 32 + 4 * kChainGroups * kBitsAhead * kBitsTile + (4 * kChainMaxLayers + 2) * 8 + 64;
}
__host__ __device__ constexpr int chain_columns(int rows) { return 480 - rows; }        // of tensor memory, for weights

__device__ __forceinline__ uint32_t peer_address(uint32_t shared, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(shared), "r"(rank));
    return r;
}
__device__ __forceinline__ void store_peer(uint32_t addr, const uint4& v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar) : "memory");
}

__device__ __forceinline__ void fc_chain_cta(const ChainArgs& g, unsigned char* smem) {
    constexpr uint32_t TM_COLS = 512, SF_COL = TM_COLS - 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = blockIdx.x % kChainCtas;
    const int m0 = (int)(blockIdx.x / kChainCtas) * g.rows;
    const uint32_t unit = (uint32_t)g.rows * 32u, half_bytes = (uint32_t)g.units * unit;   // a 64-bit block of all rows; an input
    unsigned char* sRaw = smem + 2 * (size_t)half_bytes;
    uint64_t* sBar = reinterpret_cast<uint64_t*>(sRaw + 4 * kChainGroups * kBitsAhead * kBitsTile);
    uint32_t* sTmem = reinterpret_cast<uint32_t*>(sBar + 4 * kChainMaxLayers + 1);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sTmem + 1);
    const uint32_t bar0 = smem_u32(sBar), in0 = smem_u32(smem);
    auto BAR_IN = [&](int l) { return bar0 + 8u * l; };                                  // layer l's input has arrived
    auto BAR_W = [&](int l) { return bar0 + 8u * (kChainMaxLayers + l); };               // its weights are expanded
    auto BAR_DONE = [&](int l) { return bar0 + 8u * (2 * kChainMaxLayers + l); };        // its MMAs are done
    const uint32_t BAR_DRAIN = bar0 + 8u * (3 * kChainMaxLayers);
    const int n0 = (int)rank * 128;
    auto kblocks = [&](int k) { return (k + 63) >> 6; };

    // Before anything is set up: the weights' first tiles and the input are asked for.
    const int quad = warp & 3, group = warp < 4 ? 0 : (warp - 4) >> 2;
    struct Pos { int l, st; };
    auto settle = [&](Pos& p) {                                          // past the ends of layers
        for (; p.l < g.n; p.l++) {
            const int have = n0 < g.layer[p.l].N ? (g.layer[p.l].K + 511) >> 9 : 0;      // (none of a layer without outputs here)
            if (p.st < have) return;
            p.st -= have;
        }
    };
    const uint32_t raw = smem_u32(sRaw) + (uint32_t)(warp - 4) * kBitsAhead * kBitsTile;     // (W expanders)
    auto ask = [&](Pos& p, int slot) {                                   // p: the position to ask for next
        if (p.l < g.n) {
            const ChainLayer& y = g.layer[p.l];
            BitsSource src;
            src.set(y.W, n0 + quad * 32, y.N, y.ldw);
            src.ask(raw + slot * kBitsTile, p.st, y.W);
            p.st += kChainGroups;
            settle(p);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    Pos p{0, group}, next{0, 0};
    settle(p);
    next = p;
    if (warp >= 4 && warp < 20)
        for (int i = 0; i < kBitsAhead; i++) ask(next, i);
    // input: this CTA's eighth of the rows, a chunk (32 columns) per item
    const int per = g.rows / kChainCtas, chunks = 2 * kblocks(g.K), span = max(chunks, g.ld), items = per * span;
    constexpr int U = 4;
    auto pixel = [&](int i) {
        const int r = i / span, m = m0 + (int)rank * per + r, col = (i - r * span) * 32 + lane;
        return i < items && m < g.M && col < g.K ? __ldg(g.x + (size_t)m * g.K + col) : -1.0f;
    };
    float f[U];
#pragma unroll
    for (int u = 0; u < U; u++) f[u] = warp < 20 ? pixel(warp + 20 * u) : 0.f;

    if (tid == 0) {
        for (int l = 0; l < g.n; l++) {
            mbar_init(BAR_IN(l), 1); mbar_init(BAR_W(l), 4 * kChainGroups); mbar_init(BAR_DONE(l), 1);
        }
        mbar_init(BAR_DRAIN, 1);
        *sAbort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int l = 0; l < g.n; l++) mbar_expect_tx(BAR_IN(l), (uint32_t)kblocks(g.layer[l].K) * unit);
    }
    if (warp == 20) tmem_alloc(smem_u32(sTmem), TM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *sTmem;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");       // waited for before the first store to a peer
    if (warp < 4) tmem_fill_unit_scales(tmem, SF_COL);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t acc = tmem + chain_columns(g.rows);
    const WsWait wait{sAbort, g.status};
    // chunk c (32 bits of K) of row m of layer l's input, to all CTAs of the cluster: lane -> CTA
    auto push = [&](int l, int m, int c, const uint4& e, uint32_t to) {
        const uint32_t at = in0 + (uint32_t)(l & 1) * half_bytes + (uint32_t)(c >> 1) * unit + (uint32_t)((c & 1) * g.rows + m) * 16u;
        store_peer(peer_address(at, to), e, peer_address(BAR_IN(l), to));
    };
    auto masked = [&](uint32_t word, int valid) {        // `valid` of the word's bits exist, the rest is 0, not -1
        const uint4 e = expand32_f4(word);
        return valid >= 32 ? e : valid <= 0 ? make_uint4(0u, 0u, 0u, 0u) : keep32_f4(e, 0xFFFFFFFFu << (32 - valid));
    };

    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp < 20) {
        for (int i0 = warp; i0 < items; i0 += 20 * U) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 + 20 * u;
                if (i >= items) break;
                const int r = i / span, c = i - r * span, row = (int)rank * per + r, m = m0 + row;
                const uint32_t w = __brev(__ballot_sync(0xffffffffu, f[u] >= 0));
                if (c < g.ld && m < g.M && lane == 0) g.bits[(size_t)m * g.ld + c] = w;
                if (c < chunks && lane < kChainCtas) push(0, row, c, masked(w, m < g.M ? g.K - c * 32 : 0), (uint32_t)lane);
            }
#pragma unroll
            for (int u = 0; u < U; u++) f[u] = pixel(i0 + 20 * (U + u));
        }
    }
    if (warp < 4) {
        // =============================== epilogue ===========================================
        const int n = n0 + warp * 32 + lane;
        for (int l = 0; l < g.n; l++) {
            const ChainLayer& y = g.layer[l];
            const bool last = l + 1 == g.n;
            const int c = (n0 >> 5) + warp;                              // this warp's chunk of the next input
            if (n0 >= y.N || (last ? c * 32 >= y.N : c >= 2 * kblocks(y.N))) continue;
            float p0 = last ? 0.f : __int_as_float(0x7FC00000), p1 = 0.f;           // (NaN behind the last output: its bit is 0)
            if (n < y.N) { p0 = __ldg(y.p0 + n); if (last) p1 = __ldg(y.p1 + n); }
            if (!wait(BAR_DONE(l), 0)) break;
            tc_fence_after();
            for (int r0 = 0; r0 < g.rows; r0 += 16) {
                int v[16];
                tmem_ld16(acc + ((uint32_t)(warp * 32) << 16) + r0, v);
                tmem_ld_wait();
                tc_fence_before();                                       // (the next layer's MMAs wait for what is sent below)
                if (last) {                                              // scale and bias (kernel.cuh:270-273)
                    float* dst = reinterpret_cast<float*>(y.out) + (size_t)(m0 + r0) * y.ldo + n;
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (n < y.N && m0 + r0 + j < g.M) dst[(size_t)j * y.ldo] = fmaf(__int_as_float(v[j]), p0, p1);
                } else {                                                 // (float)K - 2*(float)c >= thr[n] (kernel.cuh:210-213)
                    uint32_t w = 0;
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (__int_as_float(v[j]) >= p0) w |= 0x80000000u >> j;
                    w = transpose_bits(w);                               // lane j < 16: row r0 + j
                    const int row = r0 + (lane & 15);
                    w = __shfl_sync(0xffffffffu, w, lane & 15);
                    if (lane < 16 && m0 + row < g.M && c * 32 < y.N) reinterpret_cast<uint32_t*>(y.out)[(size_t)(m0 + row) * y.ldo + c] = w;
                    const uint4 e = masked(w, y.N - c * 32);
#pragma unroll
                    for (int to = 0; to < kChainCtas; to += 2) push(l + 1, row, c, e, (uint32_t)(to + (lane >> 4)));
                }
            }
            __syncwarp();
        }
    } else if (warp < 20) {
        // =============================== W expanders ========================================
        int slot = 0;
        int told = 0;                                                    // layers whose barrier this warp has arrived at
        bool ok = true;
        auto tell = [&](int upto) {
            for (; told < upto; told++)
                if (n0 < g.layer[told].N && lane == 0) mbar_arrive(BAR_W(told));
        };
        while (p.l < g.n) {
            const ChainLayer& y = g.layer[p.l];
            tell(p.l);
            asm volatile("cp.async.wait_group %0;" ::"n"(kBitsAhead - 1) : "memory");
            __syncwarp();
            uint4 w[4];
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = lds128(bits_piece(raw + slot * kBitsTile, lane, i));
            __syncwarp();
            ask(next, slot);
            slot = slot + 1 == kBitsAhead ? 0 : slot + 1;
            int after = y.after;                                         // (the last of those with outputs here)
            while (after >= 0 && n0 >= g.layer[after].N) after--;
            if (after >= 0) {
                ok = wait(BAR_DONE(after), 0);
                if (!ok) break;
                tc_fence_after();
            }
            bits_to_tmem(tmem + ((uint32_t)(quad * 32) << 16) + y.col + p.st * 64, w, kblocks(y.K) - p.st * 8);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            p.st += kChainGroups;
            settle(p);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (ok) tell(g.n);
    } else {
        // =============================== MMA issuer =========================================
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t idesc = idesc_f4(g.rows), sf = tmem + SF_COL;
        const uint64_t desc0 = smem_desc(in0, (uint32_t)g.rows * 16u, 128u);
        const uint32_t hi = (uint32_t)(desc0 >> 32), lo0 = (uint32_t)desc0;
        bool ok = true;
        for (int l = 0; l < g.n && ok; l++) {
            const ChainLayer& y = g.layer[l];
            const bool mine = n0 < y.N;
            if (mine) ok = wait(BAR_W(l), 0);
            // (a CTA without outputs waits too: what is on its way to it must arrive before it ends)
            if (ok) {
                ok = false;
                for (int i = 0; i < (1 << 24) && !ok; i++) {
                    ok = mbar_test_cluster(BAR_IN(l), 0);
                    if ((i & 1023) == 1023 && *sAbort) break;
                }
                if (!ok) { *sAbort = 1; atomicExch(g.status, 1); }
            }
            if (!ok || !mine) continue;
            asm volatile("fence.proxy.async;" ::: "memory");             // written by stores, read by the MMAs
            tc_fence_after();
            const uint32_t a = tmem + y.col;
            uint32_t lo = lo0 + ((uint32_t)(l & 1) * half_bytes >> 4);
            for (int kb = 0; kb < kblocks(y.K); kb++, lo += unit >> 4) mma_f4_ts(leader, acc, a + kb * 8, lo, hi, idesc, sf, kb > 0);
            if (leader) mma_commit(BAR_DONE(l));
            __syncwarp();
        }
        if (!ok && leader) {
            // giving up: the MMAs already issued must have finished before tensor memory is freed
            mma_commit(BAR_DRAIN);
            for (int i = 0; i < (1 << 20); i++)
                if (mbar_try_wait(BAR_DRAIN, 0)) break;
        }
        __syncwarp();
    }
    tc_fence_before();
    cluster_sync();                                                      // (no CTA ends while a peer may still store into it)
    // The MMA warp has waited for all that peers send, unless this CTA gave up: the time of any store passes then.
    if (*sAbort)
        for (int i = 0; i < 5000; i++) __nanosleep(20);
    __syncwarp();
    if (warp == 20) tmem_dealloc(tmem, TM_COLS);
}

}  // namespace umma
}  // namespace tcbnn
