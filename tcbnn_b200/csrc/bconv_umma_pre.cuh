// tcgen05 binary convolution fed from a pre-expanded input (strides 1 and 2, C <= 512), 4-bit operands:
// tcgen05.mma kind::mxf4 on +-1.0 as e2m1 with unit block scales (bconv_umma.cuh), 128 x NT x 64
// per instruction -- one MMA per filter tap and 64-channel block.
//
// In bconv_umma_ws.cuh seven warps of every CTA turn packed bits into +-1 bytes, stage by
// stage, next to the epilogue warps; with 16 warps per SM that chain of dependent scalar
// instructions is what the layers wait for.  Here the expansion is done by whoever produces the
// input -- the previous layer's epilogue, or a separate streaming pass (expand_raster below: full
// occupancy, HBM-bound, 8 bytes in and 32 out per pixel and 64-channel block) -- which writes it
// as +-1 nibbles straight in the layout the MMA wants: for every 32-channel chunk a plane
// [raster position][16 bytes] over the zero-padded virtual raster of bconv_umma.cuh, zeros on the
// dead bands.  A tile's patch is then two contiguous runs per 64-channel block (and input parity, at
// stride 2), fetched with bulk asynchronous copies (cp.async.bulk + mbarrier complete_tx).  With half a byte
// per channel the filter block of 128 output channels stays resident up to 256 input channels
// (64 output channels at 512), so the wide layers run filter-stationary too.  The CTA becomes
//
//   warps 0-15  epilogue   : groups of four warps (eight at an n-tile of 128), each on a tile of its own
//   warp  16    loader     : up to eight lanes, bulk copies of the patch planes into the stage ring
//   warp  17    MMA issuer : converged, one elected lane
//
// (or 8 or 4 epilogue warps, see EPIW).  The planes come from the caller (tcbnn_conv_workspace_bytes).
#pragma once
#include "bconv_umma_as.cuh"
#include <cuda.h>
#include <type_traits>

namespace tcbnn {
namespace umma {

// One MMA-issuing warp.  (Two issuers on alternate tiles were tried and are wrong as well as no
// faster: an mbarrier wait names its phase by parity only, so a waiter must see every phase of a
// barrier; with two consumers alternating on the same ring slot the one that runs ahead finds the
// parity of the phase before last already complete and reads a slot that has not been refilled.)
//
// EPIW, the kernel's third template argument, is the number of epilogue warps: 16 (one CTA per SM,
// all of tensor memory), a single group of 4 or 8 (launches with one tile per CTA, where only latency
// counts: registers for all of a tile's residual at once, and the epilogue rehearsed) or 8 at an n-tile of
// 64 (two groups; the CTA allocates half of tensor memory and two CTAs share an SM -- twice the independent
// loader / issuer / epilogue pipelines, so that one CTA's barrier round trips and epilogue
// latency are covered by the other's work).
//
// PAIR, the fourth: a pair of CTAs shares an n-tile of 128 whose filter block neither could hold (more than 256 input
// channels) -- each holds half of its rows and the patch of its own tile; the leader issues MMAs of 256 x 128 x 64 that
// read both shared memories (cta_group::2), and each finishes its own 128 rows.
__host__ __device__ constexpr int pre_threads(int epiw) { return epiw * 32 + 64; }
constexpr int kPreMaxStages = 8;           // patch ring depth is chosen by the host from the shared memory left

// ---- a pair of CTAs on one tile (cta_group::2) ----------------------------------------------------
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t leader_address(uint32_t shared) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(shared));
    return r;
}
// The accumulator goes back to the leader's MMAs: tensor memory is ordered by the tcgen05 fences around
// the arrival and the wait, for which the arrival itself can be relaxed.
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_address(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// WsWait with the bound in clocks, about a second, as a CTA waits for its partner too.  Polls rather than
// suspends (360 clocks per k-block with try_wait).
struct PairWait {
    volatile int* abort;
    int* err;
    __device__ __forceinline__ bool poll(uint32_t bar, uint32_t parity, bool sleep) const {
        if (mbar_test_cluster(bar, parity)) return true;
        const long long t0 = clock64();
        for (int i = 0; i < (1 << 28); i++) {
            if (mbar_test_cluster(bar, parity)) return true;
            if (sleep) __nanosleep(64);
            if ((i & 63) == 63 && (*abort || clock64() - t0 > (1LL << 31))) break;
        }
        *abort = 1;
        atomicExch(err, 1);
        return false;
    }
    __device__ __forceinline__ bool operator()(uint32_t bar, uint32_t parity) const { return poll(bar, parity, false); }
    __device__ __forceinline__ bool spin(uint32_t bar, uint32_t parity) const { return poll(bar, parity, false); }
    __device__ __forceinline__ bool relaxed(uint32_t bar, uint32_t parity) const { return poll(bar, parity, true); }
    __device__ __forceinline__ bool timed(uint32_t bar, uint32_t parity, long long& acc) const {
        const long long t0 = clock64();
        const bool ok = poll(bar, parity, false);
        acc += clock64() - t0;
        return ok;
    }
    __device__ __forceinline__ bool relaxed_timed(uint32_t bar, uint32_t parity, uint32_t& acc) const {
        const uint32_t t0 = (uint32_t)clock64();
        const bool ok = poll(bar, parity, true);
        acc += (uint32_t)clock64() - t0;
        return ok;
    }
};
// A run of a plane, in elements of 8 bytes, to the calling CTA, completing on the leader's barrier.
__device__ __forceinline__ void tensor_g2s_pair_1d(uint32_t dst, const CUtensorMap* map, int at, uint32_t leader_bar) {
    asm volatile("cp.async.bulk.tensor.1d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2}], [%3];"
                 ::"r"(dst), "l"(map), "r"(at), "r"(leader_bar) : "memory");
}

// positions of zero padding in front of the planes (a tile's patch starts up to back_y*PW+back_x
// positions before its first output position) and the rounded-up plane length
__host__ __device__ inline long long pre_front(int back_y, int back_x, int PW) {
    return ((long long)back_y * PW + back_x + 7) & ~7LL;
}
__host__ __device__ inline long long pre_plane_positions(long long NV, int npos, long long front) {
    return ((front + ((NV + 127) / 128) * 128 + npos + 7) & ~7LL);
}
// nplane: 1 for stride 1, 4 for stride 2 (the input's four row / column parity planes)
// rows: of the filter block that the CTA holds (half the n-tile in a pair)
__host__ __device__ inline size_t pre_smem_bytes(int npos, int C, int RS, int nt, int stages, int nplane, int rows = 0) {
    return (size_t)stages * nplane * 2 * npos * 16 + (size_t)RS * C * (rows ? rows : nt) / 2 + nt * 8 + RS * 8 + 44 * 8 + 64;
}
// kEpiTileRes: one buffer per epilogue group for the injected residual of its next tile, [chunk][128
// pixels][16 B]
__host__ __device__ constexpr size_t pre_res_ring_bytes(int nt, int epiw) {
    return (size_t)(epiw / (nt <= 64 ? 4 : nt / 16)) * 128 * nt * 2 + 128;
}

// packed bits [B][H][W][C/32] -> planes [C/32][nplane][plane_positions][16 B] of +-1 nibbles, zero
// where the raster position is padding or outside the batch.  Stride 1: one plane, the raster of
// the input.  Stride 2: four planes, plane (py, px) holds input pixel (2*vr + py, 2*vx + px) at
// raster position (vr, vx) of the OUTPUT grid, so that a filter tap is again a fixed offset.
// A thread takes V words (32-channel chunks) of a position, blockIdx.y names the words and the plane.  HBM bounds
// it: 56 x 56 x 128 at batch 256 writes 53 MB.
template <int V>
__device__ __forceinline__ void expand_raster(const ConvWsArgs& a, uint4* planes, long long plane_positions,
                                              long long front) {
    // a programmatic dependent of the bits' producer; the convolution that follows is one of this pass,
    // and is let in only when all that came before this pass is complete (ConvWsArgs::filter_settled)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int Cw = a.C >> 5;
    const int nplane = a.stride == 2 ? 4 : 1;
    const int w0 = (int)(blockIdx.y / nplane) * V, pl = (int)(blockIdx.y % nplane);
    uint4* const dst = planes + ((size_t)w0 * nplane + pl) * plane_positions;
    // (positions fit 31 bits: prepared_layout)
    for (unsigned slot = blockIdx.x * blockDim.x + threadIdx.x; slot < (unsigned)plane_positions; slot += gridDim.x * blockDim.x) {
        const int gq = (int)slot - (int)front;
        uint32_t w[V];
        bool in = false;
        if (gq >= 0 && gq < (int)a.NV) {
            const int vy = fastdiv(gq, a.pw_mul, a.pw_sh), vx = gq - vy * a.PW;
            const int n = fastdiv(vy, a.vh_mul, a.vh_sh), vr = vy - n * a.VH;
            const int iy = nplane == 4 ? 2 * vr + (pl >> 1) : vr, ix = nplane == 4 ? 2 * vx + (pl & 1) : vx;
            if (vr < a.OHg && vx < a.OWg && iy < a.H && ix < a.W) {
                in = true;
                const uint32_t* src = a.in + ((size_t)(n * a.H + iy) * a.W + ix) * Cw + w0;
                if constexpr (V == 4) {
                    const uint4 q = ld_dep(reinterpret_cast<const uint4*>(src));
                    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
                } else {
                    const uint2 q = ld_dep(reinterpret_cast<const uint2*>(src));
                    w[0] = q.x; w[1] = q.y;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < V; i++)
            dst[(size_t)i * nplane * plane_positions + slot] = in ? expand32_f4(w[i]) : make_uint4(0u, 0u, 0u, 0u);
    }
}

// Epilogues.  A group of 4 warps (8 at an n-tile of 128) owns a whole tile and the groups take tiles in
// turn: a thread walks 64 columns (of one pixel, or of four pixels a quarter each) in passes of 32, so
// that the per-tile bookkeeping (raster position -> pixel, addresses, barrier waits: some 200
// instructions) is paid once per 64 outputs, and the groups work on different accumulators at the same
// time (NT = 64: 4 groups on 7 accumulators; NT = 128: 2 groups on 3).  EPI selects the epilogue the
// kernel is compiled with, so that each carries only its own registers: a thread has 96 with one CTA
// of 18 warps per SM or two of 10, and with nearly all of L1 taken as shared memory a spilled
// register costs a trip to L2 (28 x 28 x 128 with residuals at batch 512: eight spilled reloads per warp
// and tile kept every warp waiting for a third of its time).
//   kEpiTile      no residual, no integer output: the fp32 accumulator is compared with the fp32
//                 threshold as it is.  One thread per pixel.
//   kEpiTileRes   chunk-major int16 residuals in and / or out.  One thread per pixel: every tensor is
//                 touched in whole lines.  The live pixels of a tile are consecutive pixels of the
//                 tensor, so its incoming residual is one run of up to 2 KB per chunk; the group
//                 fetches these with bulk copies into a buffer of its own as soon as it has read the
//                 tile in front from it, so that they are in flight while it packs, stores and waits (a register-fed epilogue has 64 bytes per thread
//                 in flight, and only while it waits).
//   kEpiTilePool  the same with a pooled residual, or one whose buffers do not fit beside the filter
//                 block: read in place (four lines per pooled chunk).
//   kEpiRows2/4   everything else: NHWC residuals (int16 in: Rows2, int32 in: Rows4), NHWC saves,
//                 integer output, mixtures with the chunk-major layout.  The accumulator is read in
//                 the 16x256b shape: a quad of lanes holds 32 channels of four pixels, so it moves
//                 whole 32-byte sectors of an NHWC row (f4_channel_of_column), where a thread per pixel
//                 would move 16-byte pieces of 32 different rows.  What a later unit of work reads is
//                 requested before the one in front is computed.  Measured on 56 x 56 x 128 -> 128, batch
//                 256, int32 result saved (411 MB): 251 us with a thread per pixel.
constexpr int kEpiTile = 0, kEpiTileRes = 1, kEpiRows2 = 2, kEpiRows4 = 3, kEpiTilePool = 4;
template <int NT, int EPI, int EPIW, bool PAIR = false>
__device__ void conv_umma_pre_cta(const ConvWsArgs& a, unsigned char* smem, const CUtensorMap* map_head = nullptr,
                                  const CUtensorMap* map_tail = nullptr) {
    constexpr int kEpiThreads = EPIW * 32, kThreadsCta = pre_threads(EPIW);
    constexpr bool ROWS = EPI == kEpiRows2 || EPI == kEpiRows4;
    constexpr int CPT = NT < 64 ? NT : 64;            // columns of a tile per thread
    constexpr int WPG = 4 * (NT / CPT);               // warps of a group (all rows x all columns of a tile)
    constexpr int NG = EPIW / WPG;                    // groups, each on a tile of its own
    constexpr bool SINGLE = NG == 1;
    static_assert(EPIW == 16 || (EPIW == 8 && NT == 64) || (SINGLE && !ROWS), "forms in use");
    static_assert(!PAIR || (EPIW == 16 && NT == 128), "forms in use");
    constexpr int NB = PAIR ? NT / 2 : NT;             // filter rows (output channels) that this CTA holds
    // Tensor memory: accumulators (7 at NT = 64) below column 480, the unit block scales of the
    // 4-bit MMA above it; the patch ring is as deep as shared memory allows, so that no role waits
    // on another's latency.
    constexpr uint32_t TM_COLS = EPIW == 16 ? 512 : 256, SF_COL = TM_COLS - 32;
    constexpr int NACC = (SF_COL / NT) > 8 ? 8 : (SF_COL / NT);
    const int NSTAGE = a.pre_stages;
    constexpr int LOAD_WARP = EPIW, MMA_WARP = LOAD_WARP + 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int RS = a.R * a.S, NCB = a.C >> 6;
    const int NPLANE = a.stride == 2 ? 4 : 1;
    const uint32_t plane_bytes = 2u * a.NPOS * 16u;           // two 32-channel chunk planes
    const uint32_t block_bytes = NPLANE * plane_bytes;        // one 64-channel block of a tile's patch
    // A stage holds one, two or four blocks: the issuing thread's wait / commit round per stage is
    // time the tensor pipe idles, so layers with several blocks pay it once per 2 or 4 x RS MMAs.
    const int CBS = a.pre_cbs;
    const uint32_t stage_bytes = (uint32_t)CBS * block_bytes;

    unsigned char* sAraw = smem;
    uint4* sB = reinterpret_cast<uint4*>(smem + (size_t)NSTAGE * stage_bytes);
    int* sThr = reinterpret_cast<int*>(sB + (size_t)RS * (a.C >> 5) * NB);
    float* sThrF = reinterpret_cast<float*>(sThr + NT);       // the thresholds as given (fp32)
    uint32_t* sTapK = reinterpret_cast<uint32_t*>((reinterpret_cast<uintptr_t>(sThrF + NT) + 7) & ~(uintptr_t)7);
    uint64_t* sBar = reinterpret_cast<uint64_t*>(sTapK + 2 * RS);
    // barriers: a_full[8], a_empty[8], acc_full[8], acc_empty[8], drain, res_full[NG], res_empty[NG], filter
    uint32_t* sTmem = reinterpret_cast<uint32_t*>(sBar + 44);
    volatile int* sAbort = reinterpret_cast<volatile int*>(sTmem + 1);
    const uint32_t bar0 = smem_u32(sBar);
    const uint32_t BAR_DRAIN = bar0 + 8u * 32;         // MMAs still in flight when the issuer gives up
    volatile int* sP0 = reinterpret_cast<volatile int*>(sTmem + 2);      // first pixel in each group's residual buffer
    const uint32_t BAR_FILTER = bar0 + 8u * 41;        // the filter block has landed
    const uint32_t BAR_BOTH = bar0 + 8u * 42;          // (pair) ... the second CTA's, too
    unsigned char* sRes = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sTmem + 6) + 127) & ~(uintptr_t)127);
    auto BAR_AFULL = [&](int s) { return bar0 + 8u * s; };
    auto BAR_AEMPTY = [&](int s) { return bar0 + 8u * (8 + s); };
    auto BAR_CFULL = [&](int b) { return bar0 + 8u * (16 + b); };
    auto BAR_CEMPTY = [&](int b) { return bar0 + 8u * (24 + b); };

    // CTA -> (n-tile, first m-tile, stride over m-tiles).  Normally every n-tile gets the same
    // share of the grid; where only the first n-tiles carry the epilogue's expensive part (a pooled
    // residual injected into the first channels) the host gives those more CTAs each.
    int nt, mfirst, mstep;
    const int rank = PAIR ? (int)(blockIdx.x & 1u) : 0;
    if constexpr (PAIR) {
        const int pair = (int)(blockIdx.x >> 1);
        nt = pair % a.ntiles_n; mfirst = 2 * (pair / a.ntiles_n) + rank; mstep = 2 * ((int)(gridDim.x >> 1) / a.ntiles_n);
    } else if (a.nt_heavy > 0) {
        const int nh = a.nt_heavy * a.per_heavy;
        if ((int)blockIdx.x < nh) {
            nt = blockIdx.x % a.nt_heavy; mfirst = blockIdx.x / a.nt_heavy; mstep = a.per_heavy;
        } else {
            const int r = blockIdx.x - nh, nl = a.ntiles_n - a.nt_heavy;
            nt = a.nt_heavy + r % nl; mfirst = r / nl; mstep = a.per_light;
        }
    } else {
        nt = blockIdx.x % a.ntiles_n; mfirst = blockIdx.x / a.ntiles_n; mstep = gridDim.x / a.ntiles_n;
    }
    const int NV = (int)a.NV;
    const int mtiles = (NV + 127) / 128;
    // (a pair goes on while its first CTA has a tile: the second one's last may lie behind the batch, sums that
    // nobody stores)
    const int mend = PAIR ? ((mtiles + 1) & ~1) : mtiles;
    const int obase = nt * NT;

    // Launched as a programmatic dependent: everything up to griddepcontrol.wait may run while the
    // launch in front is still running, so it touches nothing but this CTA's own memory and a settled filter.
    if (tid == 0) {
        for (int s = 0; s < 8; s++) { mbar_init(BAR_AFULL(s), 1); mbar_init(BAR_AEMPTY(s), 1); }
        for (int b = 0; b < 8; b++) { mbar_init(BAR_CFULL(b), 1); mbar_init(BAR_CEMPTY(b), PAIR ? 2 * WPG : WPG); }
        mbar_init(BAR_DRAIN, 1);
        mbar_init(BAR_FILTER, 1);
        if constexpr (PAIR) mbar_init(BAR_BOTH, 1);
        for (int g = 0; g < NG; g++) { mbar_init(bar0 + 8u * (33 + g), WPG); mbar_init(bar0 + 8u * (37 + g), WPG); }
        *sAbort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(sTmem)), "r"(TM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            tmem_alloc(smem_u32(sTmem), TM_COLS);
        }
    }
    for (int t = tid; t < RS; t += kThreadsCta) {
        // offset of the tap's operand inside a stage, in 16-byte units
        const int r = t / a.S, sx = t % a.S;
        if (NPLANE == 4) {
            const int ty = r - a.pad_h, tx = sx - a.pad_w;
            const int py = ty & 1, px = tx & 1;
            const int dy = (ty - py) / 2, dx = (tx - px) / 2;
            sTapK[t] = (uint32_t)(py * 2 + px) * (plane_bytes >> 4) + (uint32_t)((dy + a.back_y) * a.PW + (dx + a.back_x));
        } else {
            sTapK[t] = (uint32_t)(r * a.PW + sx);
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *sTmem;
    // Only now that this CTA has its tensor memory may the next launch's CTAs come: one of them could
    // otherwise take it first and wait for this grid, which would wait for it.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp < 4) tmem_fill_unit_scales(tmem, SF_COL);
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) cluster_sync();                // the partner's barriers and scales are set up as well
    tc_fence_after();
    constexpr int kIssueLanes = 8;
    if (warp == LOAD_WARP) {
        // The filter block, in eight pieces (a multiple of 16 bytes each).  Where the caller's filter is
        // settled (ConvWsArgs::filter_settled) before the wait, under the launch in front.
        if (!a.filter_settled) asm volatile("griddepcontrol.wait;" ::: "memory");
        const uint32_t nB = (uint32_t)(RS * (a.C >> 5) * NB), part = (nB + kIssueLanes - 1) / kIssueLanes;
        if (lane == 0) mbar_expect_tx(BAR_FILTER, nB * 16u);
        __syncwarp();
        const uint32_t first = (uint32_t)lane * part;
        if (lane < kIssueLanes && first < nB)
            bulk_g2s(smem_u32(sB + first), a.wf4 + (size_t)(PAIR ? 2 * nt + rank : nt) * nB + first, min(part, nB - first) * 16u, BAR_FILTER);
    }
    // Rehearsal (single-group CTAs): the epilogue runs its loop once without effect (nothing read from or
    // written to global memory, no barrier touched) before it waits for the launch in front.  Its code
    // then comes from the instruction cache when it counts: fetching it from L2 as it is first executed
    // costs a microsecond and more of such a layer's 5 to 9.  `opaque` keeps the compiler from making a
    // copy of the loop body for it.  (The MMA issuer gains nothing by it; a CTA of several groups loses 7 %
    // in its residual epilogues to the extra predicates, on a long run of tiles.)
    auto opaque = [](uint32_t v) { asm volatile("" : "+r"(v)); return v; };
    // epilogue threads, behind their rehearsal
    auto epilogue_start = [&]() {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        // thresholds, in the accumulator's column order
        for (int i = tid; i < NT; i += kEpiThreads) {
            // integer form of  !((float)v < thr)  (kernel.cuh:795-796): v >= ceil(thr)
            int it = INT_MIN;
            float tf = __int_as_float(0x7FC00000);       // NaN: never "less", the bit is always set
            const int o = obase + (i & ~31) + f4_channel_of_column(i & 31);      // column i's channel
            if (o < a.O) {
                const float t = ld_dep(a.thr + o);
                tf = t;
                if (t == t) it = t >= 2147483520.0f ? INT_MAX : t <= -2147483648.0f ? INT_MIN : (int)ceilf(t);
            }
            // (the int16 epilogues compare values that still carry kF4Bias)
            sThr[i] = EPI == kEpiTileRes || EPI == kEpiTilePool ? kF4Bias + min(max(it, -(1 << 23)), 1 << 23) : it;
            sThrF[i] = tf;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
    };
    // an epilogue warp is done with accumulator b
    auto release = [&](int b) { if constexpr (PAIR) mbar_arrive_leader(BAR_CEMPTY(b)); else mbar_arrive(BAR_CEMPTY(b)); };
    const typename std::conditional<PAIR, PairWait, WsWait>::type wait{sAbort, a.err_flag};

    if (warp == LOAD_WARP) {
        // =============================== patch loader =======================================
        // Lane 0 waits for a free stage and announces the bytes; up to eight lanes then issue the
        // stage's bulk copies between them.  A thread is busy 100-200 clocks per copy whatever its
        // size, and a stage of a stride-2 layer is 8 to 32 copies (four parity planes x two chunks
        // per 64-channel block): one lane issuing them all took longer than the stage's MMAs.
        {
            const long long back = (long long)a.back_y * a.PW + a.back_x;
            const int ncopy = CBS * NPLANE * 2;
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t it = 0, sph = 0;
            int s = 0;
            bool ok = true;
            for (int m = mfirst; m - rank < mend && ok; m += mstep) {
                const long long slot0 = (long long)m * 128 - back + a.pre_front;
                for (int cb = 0; cb < NCB; cb += CBS, it++) {
                    // the ring is several tiles deep: lane 0 mostly waits for a slot, and sleeps
                    // between polls so that it does not take issue slots from the epilogue warps
                    if (lane == 0) ok = wait.relaxed(BAR_AEMPTY(s), sph ^ 1);
                    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
                    if (!ok) break;
                    const uint32_t dst = smem_u32(sAraw + (size_t)s * stage_bytes);
                    if constexpr (PAIR) {
                        // Both CTAs' copies complete on the leader's barrier, which only a tensor copy of a pair may do:
                        // a plane's run as up to 128 positions and what is left.
                        if (lane == 0 && rank == 0) mbar_expect_tx(BAR_AFULL(s), m + 1 < mtiles ? 2 * stage_bytes : stage_bytes);
                        __syncwarp();
                        if (m < mtiles && lane < kIssueLanes) {
                            for (int i = lane; i < 2 * ncopy; i += kIssueLanes) {
                                const int tail = i & 1, c = (i >> 1) & 1, sub = i >> 2;
                                const long long at = (long long)((cb + sub) * 2 + c) * a.pre_positions + slot0 + 128 * tail;
                                tensor_g2s_pair_1d(dst + (uint32_t)sub * block_bytes + (uint32_t)c * (uint32_t)a.NPOS * 16u + 2048u * tail,
                                                   tail ? map_tail : map_head, (int)(2 * at), leader_address(BAR_AFULL(s)));
                            }
                        }
                        __syncwarp();
                        if (++s == NSTAGE) { s = 0; sph ^= 1; }
                        continue;
                    }
                    if (lane == 0) mbar_expect_tx(BAR_AFULL(s), stage_bytes);
                    __syncwarp();
                    if (lane < kIssueLanes) {
                        for (int i = lane; i < ncopy; i += kIssueLanes) {
                            const int c = i & 1, pl = (i >> 1) % NPLANE, sub = (i >> 1) / NPLANE;
                            bulk_g2s(dst + (uint32_t)sub * block_bytes + (uint32_t)(pl * 2 + c) * (uint32_t)a.NPOS * 16u,
                                     a.pre + ((size_t)((cb + sub) * 2 + c) * NPLANE + pl) * a.pre_positions + slot0,
                                     (uint32_t)a.NPOS * 16u, BAR_AFULL(s));
                        }
                    }
                    if (++s == NSTAGE) { s = 0; sph ^= 1; }
                }
            }
            if (PAIR && !ok && lane == 0) {
                // giving up: the time of any copy passes (the second CTA's complete on the leader's barrier)
                for (int i = 0; i < (1 << 17); i++) __nanosleep(20);
            }
            if (!PAIR && !ok && lane == 0) {
                for (int i = 0; i < (1 << 20); i++)
                    if (mbar_try_wait(BAR_FILTER, 0)) break;
                // giving up: wait (bounded) for the copies still in flight before the CTA exits;
                // stages below `s` were last filled in this pass over the ring, the others in the one before
                for (int s2 = 0; s2 < NSTAGE; s2++) {
                    const bool this_pass = s2 < s;
                    if (!this_pass && it < (uint32_t)NSTAGE) continue;
                    for (int i = 0; i < (1 << 20); i++)
                        if (mbar_try_wait(BAR_AFULL(s2), this_pass ? sph : sph ^ 1)) break;
                }
            }
        }
        __syncwarp();
    } else if (PAIR && warp > LOAD_WARP && rank == 1) {
        // (the leader issues for both; it must know that this CTA's half of the filter is there)
        const bool landed = wait(BAR_FILTER, 0);
        if (landed && lane == 0)
            asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_address(BAR_BOTH)) : "memory");
        __syncwarp();
    } else if (warp > LOAD_WARP) {
        // =============================== MMA issuer =========================================
        // The whole warp runs the control flow converged and polls the barriers, and one elected
        // lane issues: what the issuing thread executes between two MMAs is time the tensor pipe
        // idles, and a lone lane in a diverged warp pays far more per branch and per wait.
        {
            const bool leader = elect_one();
            const uint32_t lboA = (uint32_t)a.NPOS * 16u, lboB = NB * 16u;
            const uint64_t descA0 = smem_desc(smem_u32(sAraw), lboA, 128u);
            const uint64_t descB0 = smem_desc(smem_u32(sB), lboB, 128u);
            const uint32_t aHi = (uint32_t)(descA0 >> 32), bHi = (uint32_t)(descB0 >> 32);
            const uint32_t aLo0 = (uint32_t)descA0, bLo0 = (uint32_t)descB0;
            const uint32_t stepB = (2u * lboB) >> 4, stepStage = stage_bytes >> 4;   // one tap = two chunks of B
            const uint32_t stepBlock = block_bytes >> 4;
            constexpr uint32_t IDESC = idesc_f4(NT) + (PAIR ? (128u >> 4) << 24 : 0u);       // (a pair: M = 256)
            const uint32_t sfa = tmem + SF_COL, sfb = tmem + SF_COL + 16;
            uint32_t tapk[9];                              // 3x3 filters: the tap offsets in registers
#pragma unroll
            for (int t = 0; t < 9; t++) tapk[t] = t < RS ? sTapK[t] : 0u;
            bool ok = true;
            long long tr_wc = 0, tr_wa = 0;
            const long long tr_t0 = clock64();
            // One pass per stage of the ring.  Ring slot, accumulator and their phases are running
            // counters (a division by the ring depth would sit between two groups of MMAs), and what
            // the next stage needs is worked out behind the stage's first MMAs, while these keep the
            // pipe busy: between the last MMA of a stage and the first of the next only a branch on
            // the outcome of tests made earlier is left.
            const uint32_t spt = (uint32_t)(NCB / CBS);    // stages per tile
            const uint32_t nit = mfirst < mend ? (uint32_t)((mend - mfirst + mstep - 1) / mstep) * spt : 0u;
            uint32_t s = 0, b = 0, sph = 0, bph = 0, left = spt;      // left: stages of this tile still to issue
            uint32_t acc = 0, bLo = bLo0, d = tmem, aLo = aLo0;
            // ready: bit 0 = this stage is known to be full, bit 1 = this tile's accumulator to be free,
            // asked while the stage in front was issued (mma_f4_end); waited for only where not yet so
            uint32_t ready = 0, need = 3u;
            const uint32_t tap_end = sTapK[RS - 1];
            ok = wait(BAR_FILTER, 0);
            if (PAIR && ok) ok = wait(BAR_BOTH, 0);
            for (uint32_t it = 0; it < nit && ok; it++) {
                if ((ready & need) != need) {
                    if ((need & 2u) && !(ready & 2u)) {
                        ok = a.trace ? wait.timed(BAR_CEMPTY(b), bph ^ 1, tr_wc) : wait.spin(BAR_CEMPTY(b), bph ^ 1);
                        if (!ok) break;
                    }
                    if (!(ready & 1u)) {
                        ok = a.trace ? wait.timed(BAR_AFULL(s), sph, tr_wa) : wait.spin(BAR_AFULL(s), sph);
                        if (!ok) break;
                    }
                }
                tc_fence_after();
                if (PAIR || RS == 9) {
                    for (int sub = 0; sub + 1 < CBS; sub++) {
                        mma_f4_run<9, PAIR>(leader, d, aLo, aHi, bLo, bHi, stepB, tapk, IDESC, acc, sfa, sfb);
                        bLo += 9 * stepB;
                        aLo += stepBlock;
                        acc = 1;
                    }
                    mma_f4_run<5, PAIR>(leader, d, aLo, aHi, bLo, bHi, stepB, tapk, IDESC, acc, sfa, sfb);
                    bLo += 5 * stepB;
                } else {
                    // other filters: taps in runs of five while they last, then one by one; the last is left
                    for (int sub = 0; sub < CBS; sub++) {
                        const int nt_ = sub + 1 == CBS ? RS - 1 : RS;
                        int t = 0;
                        uint32_t tk[5];                    // read one run ahead, for the same reason
#pragma unroll
                        for (int j = 0; j < 5; j++) tk[j] = sTapK[min(j, RS - 1)];
                        for (; t + 5 <= nt_; t += 5) {
                            uint32_t tn[5];
#pragma unroll
                            for (int j = 0; j < 5; j++) tn[j] = sTapK[min(t + 5 + j, RS - 1)];
                            mma_f4_run<5>(leader, d, aLo, aHi, bLo, bHi, stepB, tk, IDESC, acc, sfa, sfb);
                            bLo += 5 * stepB;
                            acc = 1;
#pragma unroll
                            for (int j = 0; j < 5; j++) tk[j] = tn[j];
                        }
                        for (; t < nt_; t++) {             // fewer than five: tk holds them
                            mma_f4_run<1>(leader, d, aLo, aHi, bLo, bHi, stepB, tk, IDESC, acc, sfa, sfb);
#pragma unroll
                            for (int j = 0; j < 4; j++) tk[j] = tk[j + 1];
                            bLo += stepB;
                            acc = 1;
                        }
                        if (sub + 1 < CBS) aLo += stepBlock;
                    }
                }
                asm volatile("" : "+r"(s), "+r"(b), "+r"(left), "+r"(sph), "+r"(bph));   // what follows stays behind those MMAs
                const bool last = left == 1;
                const bool swrap = s + 1 == (uint32_t)NSTAGE, bwrap = b + 1 == (uint32_t)NACC;
                const uint32_t sn = swrap ? 0u : s + 1, bn = bwrap ? 0u : b + 1;
                uint32_t sphn = swrap ? sph ^ 1u : sph, bphn = bwrap ? bph ^ 1u : bph;
                uint32_t bar_a = BAR_AFULL(sn), bar_b = BAR_CEMPTY(bn), par_b = bphn ^ 1u;
                uint32_t bar_e = BAR_AEMPTY(s), bar_c = last ? BAR_CFULL(b) : 0u;
                uint32_t aLon = aLo0 + sn * stepStage, dn = last ? tmem + bn * NT : d;
                uint32_t bLon = last ? bLo0 : bLo + (RS == 9 ? 4u : 1u) * stepB;
                need = last ? 3u : 1u;
                if (last) { b = bn; bph = bphn; }
                left = last ? spt : left - 1;
                s = sn;
                sph = sphn;
                const uint32_t acc_end = RS == 9 ? 1u : acc;
                acc = last ? 0u : 1u;
                asm volatile("" : "+r"(bar_a), "+r"(bar_b), "+r"(par_b), "+r"(bar_e), "+r"(bar_c), "+r"(aLon), "+r"(dn),
                                  "+r"(bLon), "+r"(need), "+r"(b), "+r"(bph), "+r"(left), "+r"(s), "+r"(sph), "+r"(acc));
                if (PAIR || RS == 9) {
                    ready = mma_f4_end<4, PAIR>(leader, d, aLo, aHi, bLo, bHi, stepB, tapk + 5, IDESC, acc_end, sfa, sfb,
                                          bar_a, sphn, bar_b, par_b, bar_e, bar_c);
                } else {
                    ready = mma_f4_end<1>(leader, d, aLo, aHi, bLo, bHi, stepB, &tap_end, IDESC, acc_end, sfa, sfb,
                                          bar_a, sphn, bar_b, par_b, bar_e, bar_c);
                }
                aLo = aLon;
                d = dn;
                bLo = bLon;
            }
            if (!ok && leader) {
                // giving up: the MMAs already issued must have finished before tensor memory is freed
                if constexpr (PAIR)
                    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(BAR_DRAIN) : "memory");
                else
                    mma_commit(BAR_DRAIN);
                for (int i = 0; i < (1 << 20); i++)
                    if (mbar_try_wait(BAR_DRAIN, 0)) break;
            }
            if (a.trace && blockIdx.x == 0 && leader) { a.trace[3] = clock64() - tr_t0; a.trace[4] = tr_wc; a.trace[5] = tr_wa; a.trace[2] = nit; }
        }
        __syncwarp();
    } else if (!ROWS && tid < kEpiThreads) {
        // =============================== epilogue, a thread per pixel ==========================
        constexpr bool RES = EPI == kEpiTileRes || EPI == kEpiTilePool, RING = EPI == kEpiTileRes;
        constexpr int PASSES = CPT / 32;
        const int grp = warp / WPG, wig = warp % WPG, quad = warp & 3, half = wig >> 2;
        const int row = quad * 32 + lane;
        const int Ow = (a.O + 31) >> 5;
        // Pass k of a thread covers the tile's 32-column block k (groups of 4 warps) or 2k + half
        // (groups of 8: the two halves interleave, so that a residual injected into the first
        // channels only -- the first block of a stage -- is shared between them).
        constexpr int HSTEP = WPG / 4;                     // 32-column blocks between a thread's passes
        const int o0 = obase + half * 32;                  // this thread's first output channel
        const int lim = (RES && a.res_in) ? min(a.residual_channels, a.res_in_ch) : 0;
        const bool has_in = RES && a.res_in && o0 < lim;
        const bool ring = RING && obase < lim;
        const uint4* rin = reinterpret_cast<const uint4*>(a.res_in) + (size_t)(o0 >> 3) * a.res_in_npix;
        uint4* rout = reinterpret_cast<uint4*>(a.res_out) + (size_t)(o0 >> 3) * a.res_out_npix;
        bool ok = true, overflow = false;
        const bool tr = a.trace != nullptr && blockIdx.x == 0;
        uint32_t tr_w = 0;
        const uint32_t tr_t0 = (uint32_t)clock64();
        // ---- the group's residual buffer -----------------------------------------------------
        const uint32_t bar_rf = bar0 + 8u * (33 + grp), bar_re = bar0 + 8u * (37 + grp);
        unsigned char* const rbuf = sRes + (size_t)grp * (128 * NT * 2);
        const int nchunk = ring ? min(NT, lim - obase) >> 3 : 0;
        // output pixels in front of raster position p
        auto live_before = [&](int p) -> int {
            if (p >= NV) return a.B * a.OHg * a.OWg;
            const int vy = fastdiv(p, a.pw_mul, a.pw_sh), x = p - vy * a.PW;
            const int n = fastdiv(vy, a.vh_mul, a.vh_sh), y = vy - n * a.VH;
            return (n * a.OHg + min(y, a.OHg)) * a.OWg + (y < a.OHg ? min(x, a.OWg) : 0);
        };
        // residual of m-tile `m` into the (free) buffer; the group's warps share the chunks, because a
        // warp that issues bulk copies is busy for 100-200 clocks with each of them
        auto request = [&](int m) {
            const int p0 = live_before(m * 128), nl = live_before(m * 128 + 128) - p0;
            const int mine = (nchunk - wig + WPG - 1) / WPG;             // chunks wig, wig + WPG, ..
            if (lane == 0) {
                if (wig == 0) sP0[grp] = p0;
                mbar_expect_tx(bar_rf, (uint32_t)(mine * nl) * 16u);
            }
            __syncwarp();
            if (nl > 0 && lane < mine)
                bulk_g2s(smem_u32(rbuf) + (uint32_t)(wig + lane * WPG) * 2048u,
                         reinterpret_cast<const uint4*>(a.res_in) + (size_t)((obase >> 3) + wig + lane * WPG) * a.res_in_npix + p0,
                         (uint32_t)nl * 16u, bar_rf);
        };
        uint32_t rph = 0;
        static_assert(NG <= NACC, "the accumulator counters below wrap at most once per tile");
        int b = grp;
        uint32_t bph = 0;
        uint32_t dry = SINGLE ? opaque(1u) : 0u;
        if (!SINGLE) {
            epilogue_start();
            if (ring && mfirst + grp * mstep < mtiles) request(mfirst + grp * mstep);
        }
#pragma unroll 1
        for (int m = mfirst + grp * mstep; (m - rank < mend || dry) && ok; m += NG * mstep, b += NG) {
            if (b >= NACC) { b -= NACC; bph ^= 1u; }
            // raster position -> output pixel
            const int p = m * 128 + row;
            bool live = false;
            int n = 0, y = 0, x = 0;
            if (p < NV && !dry) {
                const int vy = fastdiv(p, a.pw_mul, a.pw_sh);
                x = p - vy * a.PW;
                n = fastdiv(vy, a.vh_mul, a.vh_sh);
                y = vy - n * a.VH;
                live = x < a.OWg && y < a.OHg;
            }
            const int opix = (n * a.OHg + y) * a.OWg + x;
            // injected residual of step i (16 channels: half i & 1 of pass i >> 1): zeros where nothing
            // is injected; 2x2 max for pooled residuals (kernel.cuh:773-783)
            uint4 r[SINGLE ? 2 * PASSES : 1][2];
            auto fetch = [&](int i, uint4 (&r)[2]) {
                const uint4 z = make_uint4(0u, 0u, 0u, 0u);
                const size_t i00 = ((size_t)n * 2 * a.OHg + 2 * y) * 2 * a.OWg + 2 * x, rw = (size_t)2 * a.OWg;
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    r[j] = z;
                    const int oc = 32 * HSTEP * (i >> 1) + 16 * (i & 1) + 8 * j;
                    if (live && o0 + oc < lim) {
                        const uint4* q = rin + (size_t)(oc >> 3) * a.res_in_npix;
                        if (a.residual_pool) {
                            const uint4 w0 = ld_dep(q + i00), w1 = ld_dep(q + i00 + 1), w2 = ld_dep(q + i00 + rw), w3 = ld_dep(q + i00 + rw + 1);
                            r[j].x = __vmaxs2(__vmaxs2(w0.x, w1.x), __vmaxs2(w2.x, w3.x));
                            r[j].y = __vmaxs2(__vmaxs2(w0.y, w1.y), __vmaxs2(w2.y, w3.y));
                            r[j].z = __vmaxs2(__vmaxs2(w0.z, w1.z), __vmaxs2(w2.z, w3.z));
                            r[j].w = __vmaxs2(__vmaxs2(w0.w, w1.w), __vmaxs2(w2.w, w3.w));
                        } else {
                            r[j] = ld_dep(q + opix);
                        }
                    }
                }
            };
            if (EPI == kEpiTilePool && has_in) {           // flies while the accumulator is awaited
#pragma unroll
                for (int i = 0; i < (SINGLE ? 2 * PASSES : 1); i++) fetch(i, r[i]);
            }
            if (!dry) ok = tr ? wait.relaxed_timed(BAR_CFULL(b), bph, tr_w) : SINGLE ? wait(BAR_CFULL(b), bph) : wait.relaxed(BAR_CFULL(b), bph);
            if (!ok) break;
            uint32_t rslot = smem_u32(rbuf);
            if (ring && !dry) {
                ok = tr ? wait.relaxed_timed(bar_rf, rph, tr_w) : wait.relaxed(bar_rf, rph);
                if (!ok) break;
                rph ^= 1u;
                rslot = smem_u32(rbuf) + (uint32_t)(opix - sP0[grp]) * 16u;
            }
            tc_fence_after();
            int v0[16];                                    // (residual epilogues: the columns on their way)
#pragma unroll (SINGLE ? PASSES : 1)
            for (int k = 0; k < PASSES; k++) {
                const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + b * NT + (HSTEP * k + half) * 32;
                uint32_t word = 0;                         // channel c of the pass at bit 31 - c
                if constexpr (!RES) {
                    int v[32];
                    tmem_ld32(taddr, v);
                    tmem_ld_wait();
                    if (k == PASSES - 1) {
                        tc_fence_before();                 // this warp is done with the accumulator
                        __syncwarp();
                        if (lane == 0 && !dry) release(b);
                    }
                    // the reference's comparison as it stands, !((float)value < threshold)
                    // (kernel.cuh:795-796), on the fp32 accumulator
                    const float4* tf4 = reinterpret_cast<const float4*>(sThrF + (HSTEP * k + half) * 32);
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float4 th = tf4[j];
                        if (!(__int_as_float(v[4 * j]) < th.x)) word |= 0x80000000u >> f4_channel_of_column(4 * j);
                        if (!(__int_as_float(v[4 * j + 1]) < th.y)) word |= 0x80000000u >> f4_channel_of_column(4 * j + 1);
                        if (!(__int_as_float(v[4 * j + 2]) < th.z)) word |= 0x80000000u >> f4_channel_of_column(4 * j + 2);
                        if (!(__int_as_float(v[4 * j + 3]) < th.w)) word |= 0x80000000u >> f4_channel_of_column(4 * j + 3);
                    }
                } else {
                    // 16 columns (two chunks) at a time, the next 16 on their way meanwhile: fewer
                    // registers alive at once.  Values carry kF4Bias throughout.
                    auto step = [&](int (&v)[16], const int h) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = f4_acc_to_biased(v[j]);
                        auto add8 = [&](int j, const uint4& q) {
                            const uint32_t rw[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                            for (int e = 0; e < 8; e++)
                                v[f4_column_of_channel(8 * j + e)] += (e & 1) ? (int)rw[e >> 1] >> 16 : (int)(short)(rw[e >> 1] & 0xFFFFu);
                        };
                        const int c0 = (half + HSTEP * k) * 4 + 2 * h;       // first chunk of this step
                        if constexpr (RING) {
                            if (ring) {
                                if (live || dry) {
#pragma unroll
                                    for (int j = 0; j < 2; j++) {
                                        if (c0 + j < nchunk) {
                                            uint4 q;
                                            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                                                         : "r"(rslot + (uint32_t)(c0 + j) * 2048u) : "memory");
                                            add8(j, q);
                                        }
                                    }
                                }
                                if (h == 1 && k == PASSES - 1) {         // buffer read: refill it for the group's next tile
                                    __syncwarp();
                                    if (lane == 0 && !dry) mbar_arrive(bar_re);
                                    if (m + NG * mstep < mtiles && !dry) {
                                        ok = wait(bar_re, rph ^ 1u);
                                        if (ok) request(m + NG * mstep);
                                    }
                                }
                            }
                        } else if (has_in) {
#pragma unroll
                            for (int j = 0; j < 2; j++) add8(j, r[SINGLE ? 2 * k + h : 0][j]);
                            if (!SINGLE && 2 * k + h + 1 < 2 * PASSES) fetch(2 * k + h + 1, r[0]);   // flies during this step's arithmetic
                        }
                        const int4* th4 = reinterpret_cast<const int4*>(sThr + (HSTEP * k + half) * 32 + 16 * h);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const int4 th = th4[j];
                            if (v[4 * j] >= th.x) word |= 0x80000000u >> (16 * h + f4_channel_of_column(4 * j));
                            if (v[4 * j + 1] >= th.y) word |= 0x80000000u >> (16 * h + f4_channel_of_column(4 * j + 1));
                            if (v[4 * j + 2] >= th.z) word |= 0x80000000u >> (16 * h + f4_channel_of_column(4 * j + 2));
                            if (v[4 * j + 3] >= th.w) word |= 0x80000000u >> (16 * h + f4_channel_of_column(4 * j + 3));
                        }
                        if (a.res_out && (live || dry)) {
                            if (!a.res_out_proven) {       // a real branch: three instructions per value
                                uint32_t ovf = 0;          // |v| of every value ORed together
#pragma unroll
                                for (int j = 0; j < 16; j++) ovf |= (uint32_t)((v[j] - kF4Bias) ^ ((v[j] - kF4Bias) >> 31));
                                overflow |= ovf > 32767u && live;  // some value outside [-32768, 32767]
                            }
#pragma unroll
                            for (int j = 0; j < 2; j++) {
                                uint32_t w[4];
#pragma unroll
                                for (int kk = 0; kk < 4; kk++)
                                    w[kk] = __byte_perm((uint32_t)v[f4_column_of_channel(8 * j + 2 * kk)],
                                                        (uint32_t)v[f4_column_of_channel(8 * j + 2 * kk + 1)], 0x5410);
                                if (live) rout[(size_t)(4 * HSTEP * k + 2 * h + j) * a.res_out_npix + opix] = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                        }
                    };
                    int v1[16];
                    if (k == 0) tmem_ld16(taddr, v0);
                    tmem_ld_wait16(v0);
                    tmem_ld16(taddr + 16, v1);
                    step(v0, 0);
                    tmem_ld_wait16(v1);
                    if (k == PASSES - 1) {
                        tc_fence_before();                 // this warp is done with the accumulator
                        __syncwarp();
                        if (lane == 0 && !dry) release(b);
                    } else {
                        tmem_ld16(taddr + HSTEP * 32, v0);
                    }
                    step(v1, 1);
                }
                if (live) {
                    // bits of channel o live at bit 31 - o%32 of word o/32
                    a.out[(size_t)n * a.out_image_stride + ((size_t)y * a.OWg + x) * Ow + ((o0 + 32 * HSTEP * k) >> 5)] = word;
                    if (a.nxt) store_next_planes(a, n, y, x, o0 + 32 * HSTEP * k, word);
                }
            }
            if (dry) {
                dry = opaque(0u);
                epilogue_start();
                m = mfirst + (grp - NG) * mstep;
                b = grp - NG;
                if (ring && m + NG * mstep < mtiles) request(m + NG * mstep);
            }
        }
        if (ring && !ok) {
            // giving up: a request may be in flight; wait (bounded) for it before the CTA exits
            for (int i = 0; i < (1 << 20); i++)
                if (mbar_try_wait(bar_rf, rph)) break;
        }
        if (overflow) atomicExch(a.err_flag, 2);
        if (tr && tid == 0) {
            a.trace[6] = (uint32_t)clock64() - tr_t0;
            a.trace[7] = tr_w;
            a.trace[8] = mfirst < mtiles ? (mtiles - mfirst + NG * mstep - 1) / (NG * mstep) : 0;
        }
    } else if (ROWS && tid < kEpiThreads) {
        // =============================== epilogue, a quad per row piece ========================
        constexpr int RB = EPI == kEpiRows2 ? 2 : 4;       // bytes of an injected residual value
        constexpr int PASSES = CPT / 32, HSTEP = WPG / 4;
        // A unit of work is 16 rows x 32 columns, two per pass.  Residual values are requested one unit
        // ahead (int32, 16 registers) or two (int16, 8 registers each).
        constexpr int NU = 2 * PASSES, AHEAD = RB == 4 ? 1 : 2, RREG = 4 * RB;
        const int grp = warp / WPG, quad = warp & 3, half = (warp % WPG) >> 2;
        // the row whose packed word this lane ends up with, and the quad's four rows
        const int row = quad * 32 + (lane >> 2) + 8 * (lane & 3), q4 = lane & 3;
        const int Ow = (a.O + 31) >> 5;
        const int o0 = obase + half * 32;
        const int lim = a.res_in ? min(a.residual_channels, a.res_in_ch) : 0;
        // element (pixel, channel o): pixel * stride + o (NHWC), or chunk-major [o/8][pixel][8]
        const size_t in_ps = a.res_in_chunked ? 8 : (size_t)a.res_in_ch, out_ps = a.res_out_chunked ? 8 : (size_t)a.O;
        auto in_off = [&](int o) { return a.res_in_chunked ? (size_t)(o >> 3) * a.res_in_npix * 8 + (o & 7) : (size_t)o; };
        auto out_off = [&](int o) { return a.res_out_chunked ? (size_t)(o >> 3) * a.res_out_npix * 8 + (o & 7) : (size_t)o; };
        bool ok = true, overflow = false;
        const bool tr = a.trace != nullptr && blockIdx.x == 0;
        uint32_t tr_w = 0;
        const uint32_t tr_t0 = (uint32_t)clock64();
        int b = grp;
        uint32_t bph = 0;
        epilogue_start();
        for (int m = mfirst + grp * mstep; m - rank < mend && ok; m += NG * mstep, b += NG) {
            if (b >= NACC) { b -= NACC; bph ^= 1u; }
            const int p = m * 128 + row;
            bool live = false;
            int n = 0, y = 0, x = 0;
            if (p < NV) {
                const int vy = fastdiv(p, a.pw_mul, a.pw_sh);
                x = p - vy * a.PW;
                n = fastdiv(vy, a.vh_mul, a.vh_sh);
                y = vy - n * a.VH;
                live = x < a.OWg && y < a.OHg;
            }
            // pixel index of this lane's row (-1: not an output) and of the quad's rows; the same in
            // the residual's grid
            const int opix = live ? (n * a.OHg + y) * a.OWg + x : -1;
            const uint32_t ipix = a.residual_pool ? (uint32_t)((n * 2 * a.OHg + 2 * y) * 2) * a.OWg + 2 * x : (uint32_t)opix;
            auto orow = [&](int i) { return __shfl_sync(0xffffffffu, opix, (lane & ~3) | i); };
            auto irow = [&](int i) { return __shfl_sync(0xffffffffu, ipix, (lane & ~3) | i); };
            uint32_t r[AHEAD][RREG];
            // residual of unit u (rows 2(u&1), 2(u&1)+1 of the quad's four, pass u/2) into q
            auto fetch = [&](int u, uint32_t (&q)[RREG]) {
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const bool rlive = orow(2 * (u & 1) + i) >= 0;
                    const uint32_t rpix = irow(2 * (u & 1) + i);
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        const int o = o0 + 32 * HSTEP * (u >> 1) + 16 * g + 4 * q4;
                        const bool on = rlive && o < lim;
                        if constexpr (RB == 4) {
                            int4 w = make_int4(0, 0, 0, 0);
                            if (on) {
                                const int* src = reinterpret_cast<const int*>(a.res_in) + (size_t)rpix * in_ps + in_off(o);
                                if (a.residual_pool) {
                                    const size_t dn = (size_t)2 * a.OWg * in_ps;
                                    w = max4(max4(ld_res4(src, 4, 0), ld_res4(src, 4, in_ps)), max4(ld_res4(src, 4, dn), ld_res4(src, 4, dn + in_ps)));
                                } else {
                                    w = ld_res4(src, 4, 0);
                                }
                            }
                            q[i * 8 + g * 4] = w.x; q[i * 8 + g * 4 + 1] = w.y; q[i * 8 + g * 4 + 2] = w.z; q[i * 8 + g * 4 + 3] = w.w;
                        } else {
                            uint2 w = make_uint2(0u, 0u);
                            if (on) {
                                const short* src = reinterpret_cast<const short*>(a.res_in) + (size_t)rpix * in_ps + in_off(o);
                                auto ld = [&](size_t off) { return ld_dep(reinterpret_cast<const uint2*>(src + off)); };
                                w = ld(0);
                                if (a.residual_pool) {     // 2x2 max (kernel.cuh:773-783)
                                    const size_t dn = (size_t)2 * a.OWg * in_ps;
                                    const uint2 w1 = ld(in_ps), w2 = ld(dn), w3 = ld(dn + in_ps);
                                    w.x = __vmaxs2(__vmaxs2(w.x, w1.x), __vmaxs2(w2.x, w3.x));
                                    w.y = __vmaxs2(__vmaxs2(w.y, w1.y), __vmaxs2(w2.y, w3.y));
                                }
                            }
                            q[i * 4 + g * 2] = w.x; q[i * 4 + g * 2 + 1] = w.y;
                        }
                    }
                }
            };
            const bool has_in = o0 < lim;
            if (has_in) {                                  // flies while the accumulator is awaited
#pragma unroll
                for (int i = 0; i < AHEAD; i++)
                    if (i < NU) fetch(i, r[i]);
            }
            ok = tr ? wait.relaxed_timed(BAR_CFULL(b), bph, tr_w) : wait.relaxed(BAR_CFULL(b), bph);
            if (!ok) break;
            tc_fence_after();
            uint32_t w0 = 0, w1 = 0;                       // this lane's channels' bits of rows 0 and 1 of a pass
#pragma unroll 1
            for (int u = 0; u < NU; u++) {
                const int k = u >> 1, h = u & 1;
                const int cb = HSTEP * k + half;           // 32-column block of the accumulator
                const int o = o0 + 32 * HSTEP * k + 4 * q4;
                int v[16];
                tmem_ld_16x256b_x4(tmem + ((uint32_t)(quad * 32 + 16 * h) << 16) + b * NT + cb * 32, v);
                tmem_ld_wait();
                if (u == NU - 1) {
                    tc_fence_before();                     // this warp is done with the accumulator
                    __syncwarp();
                    if (lane == 0) release(b);
                }
                // values of row i of this unit, channel run g: four consecutive channels
                int4 c[2][2];
                const int op[2] = {orow(2 * h), orow(2 * h + 1)};
#pragma unroll
                for (int i = 0; i < 2; i++)
#pragma unroll
                    for (int g = 0; g < 2; g++) {
                        c[i][g] = make_int4(f4_acc_to_int(v[8 * g + 2 * i]), f4_acc_to_int(v[8 * g + 2 * i + 1]),
                                            f4_acc_to_int(v[8 * g + 4 + 2 * i]), f4_acc_to_int(v[8 * g + 4 + 2 * i + 1]));
                        if (a.acc_out && op[i] >= 0)
                            *reinterpret_cast<int4*>(a.acc_out + (size_t)op[i] * a.O + o + 16 * g) = c[i][g];
                        if (has_in) {
                            const uint32_t* q = r[0] + (i * 2 + g) * RB;
                            if constexpr (RB == 4) {
                                c[i][g].x += (int)q[0]; c[i][g].y += (int)q[1]; c[i][g].z += (int)q[2]; c[i][g].w += (int)q[3];
                            } else {
                                c[i][g].x += (int)(short)(q[0] & 0xFFFFu); c[i][g].y += (int)q[0] >> 16;
                                c[i][g].z += (int)(short)(q[1] & 0xFFFFu); c[i][g].w += (int)q[1] >> 16;
                            }
                        }
                    }
                if (has_in) {                              // a later unit's residual flies during what follows
                    if constexpr (AHEAD == 2) {
#pragma unroll
                        for (int j = 0; j < RREG; j++) r[0][j] = r[AHEAD - 1][j];
                    }
                    if (u + AHEAD < NU) fetch(u + AHEAD, r[AHEAD - 1]);
                }
                uint32_t w[2] = {0u, 0u};
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const int2 ta = *reinterpret_cast<const int2*>(sThr + cb * 32 + 16 * g + 2 * q4);
                    const int2 tb = *reinterpret_cast<const int2*>(sThr + cb * 32 + 16 * g + 8 + 2 * q4);
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        uint32_t nib = c[i][g].x >= ta.x ? 8u : 0u;
                        if (c[i][g].y >= ta.y) nib |= 4u;
                        if (c[i][g].z >= tb.x) nib |= 2u;
                        if (c[i][g].w >= tb.y) nib |= 1u;
                        w[i] |= nib << (28 - 16 * g - 4 * q4);
                    }
                }
                if (a.res_out) {
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        if (op[i] < 0) continue;
#pragma unroll
                        for (int g = 0; g < 2; g++) {
                            const size_t idx = (size_t)op[i] * out_ps + out_off(o + 16 * g);
                            if (a.res_out_bytes == 2) {
                                if (!a.res_out_proven) {
                                    const uint32_t ovf = (uint32_t)(c[i][g].x ^ (c[i][g].x >> 31)) | (uint32_t)(c[i][g].y ^ (c[i][g].y >> 31)) |
                                                         (uint32_t)(c[i][g].z ^ (c[i][g].z >> 31)) | (uint32_t)(c[i][g].w ^ (c[i][g].w >> 31));
                                    overflow |= ovf > 32767u;              // some value outside [-32768, 32767]
                                }
                                *reinterpret_cast<uint2*>(reinterpret_cast<short*>(a.res_out) + idx) =
                                    make_uint2(__byte_perm((uint32_t)c[i][g].x, (uint32_t)c[i][g].y, 0x5410),
                                               __byte_perm((uint32_t)c[i][g].z, (uint32_t)c[i][g].w, 0x5410));
                            } else {
                                *reinterpret_cast<int4*>(reinterpret_cast<int*>(a.res_out) + idx) = c[i][g];
                            }
                        }
                    }
                }
                if (h == 0) {
                    w0 = w[0]; w1 = w[1];
                    continue;
                }
                // every lane of a quad has its channels' bits of all four rows: lane i collects row i
                const bool up = (q4 & 2) != 0, odd = (q4 & 1) != 0;
                uint32_t k0 = up ? w[0] : w0, k1 = up ? w[1] : w1;
                k0 |= __shfl_xor_sync(0xffffffffu, up ? w0 : w[0], 2);
                k1 |= __shfl_xor_sync(0xffffffffu, up ? w1 : w[1], 2);
                uint32_t word = odd ? k1 : k0;
                word |= __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 1);
                if (live) {
                    a.out[(size_t)n * a.out_image_stride + ((size_t)y * a.OWg + x) * Ow + ((o0 + 32 * HSTEP * k) >> 5)] = word;
                    if (a.nxt) store_next_planes(a, n, y, x, o0 + 32 * HSTEP * k, word);
                }
            }
        }
        if (overflow) atomicExch(a.err_flag, 2);
        if (tr && tid == 0) {
            a.trace[6] = (uint32_t)clock64() - tr_t0;
            a.trace[7] = tr_w;
            a.trace[8] = mfirst < mtiles ? (mtiles - mfirst + NG * mstep - 1) / (NG * mstep) : 0;
        }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) {
        cluster_sync();                                 // nothing of the partner's reaches into this CTA any more
        if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM_COLS) : "memory");
    } else if (warp == MMA_WARP) {
        tmem_dealloc(tmem, TM_COLS);
    }
}

}  // namespace umma
}  // namespace tcbnn
