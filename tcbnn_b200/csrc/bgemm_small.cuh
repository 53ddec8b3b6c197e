// Bit GEMM for small problems on the warp-level b1 MMA (m16n8k256 AND-popc): the sizes below the
// tcgen05 path, where latency counts and the work is too little to fill the GPU with 32 x 32 tiles.
//
// A block owns (16 MT) rows x (8 NTL NW) columns; its warps are KW slices of K times NW column
// groups.  Slices are whole 256-bit steps, taken in turn, so that a warp's chain of loads and MMAs is
// K / (256 KW) long instead of K / 256; the slices' sums meet in shared memory and the block finishes
// the layer itself (int32, threshold bits or scale + bias), so there is one launch and no scratch.
// What bounds it: a b1 MMA occupies a sub-partition for about 195 clocks (390 TOP/s over the GPU), so
// the small tile's extra loads do not show; a launch of 8 x 1024 x 1024 took 14 us as 32 warps with the
// whole of K each.
#pragma once
#include "bnn_layers.cuh"

namespace tcbnn {

constexpr int kSmallMaxWarps = 16;

// AHEAD: W and the parameters are loaded in front of A, ahead of the wait for the launch in front where they are settled
// (GemmArgs::settled): a layer of an MLP on a few rows is a chain of latencies.  What it holds meanwhile costs the 16 x 8
// tile eight registers and one block of four per SM, see launch_gemm_small.
template <int MT, int NTL, bool AHEAD>
__device__ __forceinline__ void gemm_small_block(const GemmArgs& g, int KW, int NW, int* red) {
    constexpr int R = 16 * MT, C = 8 * NTL, CP = C + 2;    // rows, columns, padded row of the exchange buffer
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
    const int kw = warp % KW, nw = warp / KW;
    // bits are stored by whole 32-bit words: column groups past N write their zeros
    const int ncols = g.mode == GEMM_FC_BITS ? (g.N + 31) & ~31 : g.N;
    const int TN = (ncols + C * NW - 1) / (C * NW);
    const int m0 = (int)(blockIdx.x / TN) * R, nb = (int)(blockIdx.x % TN) * C * NW;
    const int n0 = nb + nw * C;
    const int KP = (g.K + 63) >> 6;                        // 64-bit pairs per row

    int acc[MT][NTL][4], sa[2 * MT], pw[NTL];
#pragma unroll
    for (int a = 0; a < MT; a++)
#pragma unroll
        for (int b = 0; b < NTL; b++)
#pragma unroll
            for (int c = 0; c < 4; c++) acc[a][b][c] = 0;
#pragma unroll
    for (int i = 0; i < 2 * MT; i++) sa[i] = 0;
#pragma unroll
    for (int j = 0; j < NTL; j++) pw[j] = 0;
    const uint32_t* wp[NTL];
    auto rows_w = [&] {
#pragma unroll
        for (int j = 0; j < NTL; j++) wp[j] = g.W + (size_t)min(n0 + j * 8 + gq, g.N - 1) * g.ldw;
    };
    // U steps' loads are issued together: the chain is the loads' latency
    constexpr int U = MT * NTL >= 4 ? 2 : 4;
    uint2 b[U][NTL];
    auto load_w = [&](int kb) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int kp = kb + u * KW * 4 + t;
#pragma unroll
            for (int j = 0; j < NTL; j++)
                b[u][j] = n0 < g.N && kp < KP ? ld_dep(reinterpret_cast<const uint2*>(wp[j] + 2 * kp)) : make_uint2(0u, 0u);
        }
    };
    // parameters of the first output that this thread finishes
    float f0 = 0.f, f1 = 0.f;
    auto load_p = [&](int e0) {
        const int e = e0 + threadIdx.x, c = e % C, w = e / (C * R), col = nb + w * C + c;
        if (e < NW * R * C && col < g.N && g.mode != GEMM_INT32) {
            f0 = ld_dep(g.p0 + col);
            if (g.mode == GEMM_OUT_AFFINE) f1 = ld_dep(g.p1 + col);
        }
    };
    if constexpr (AHEAD) {
        rows_w();
        if (g.settled) { load_w(kw * 4); load_p(0); }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");      // launched as a programmatic dependent
    if (AHEAD && !g.settled) { load_w(kw * 4); load_p(0); }
    if (n0 < g.N) {
        const uint32_t* ap[2 * MT];
#pragma unroll
        for (int i = 0; i < 2 * MT; i++) ap[i] = g.A + (size_t)min(m0 + i * 8 + gq, g.M - 1) * g.lda;   // rows past M re-read row M-1
        if constexpr (!AHEAD) rows_w();
        for (int kb = kw * 4; kb < KP; kb += KW * 4 * U) {
            uint2 a[U][2 * MT];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int kp = kb + u * KW * 4 + t;
#pragma unroll
                for (int i = 0; i < 2 * MT; i++) a[u][i] = kp < KP ? ld_dep(reinterpret_cast<const uint2*>(ap[i] + 2 * kp)) : make_uint2(0u, 0u);
                if constexpr (!AHEAD) {
#pragma unroll
                    for (int j = 0; j < NTL; j++) b[u][j] = kp < KP ? ld_dep(reinterpret_cast<const uint2*>(wp[j] + 2 * kp)) : make_uint2(0u, 0u);
                }
            }
            if (AHEAD && kb != kw * 4) load_w(kb);
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (kb + u * KW * 4 >= KP) break;
#pragma unroll
                for (int i = 0; i < 2 * MT; i++) sa[i] += __popc(a[u][i].x) + __popc(a[u][i].y);
#pragma unroll
                for (int j = 0; j < NTL; j++) {
                    pw[j] += __popc(b[u][j].x) + __popc(b[u][j].y);
#pragma unroll
                    for (int m = 0; m < MT; m++)
                        mma_b1_and(acc[m][j], a[u][2 * m].x, a[u][2 * m + 1].x, a[u][2 * m].y, a[u][2 * m + 1].y, b[u][j].x, b[u][j].y);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 2 * MT; i++) sa[i] = quad_sum(sa[i]);
    int* mine = red + (size_t)warp * R * CP;
#pragma unroll
    for (int j = 0; j < NTL; j++) {
        const int p = quad_sum(pw[j]);
        const int pw0 = __shfl_sync(0xffffffffu, p, (2 * t) * 4), pw1 = __shfl_sync(0xffffffffu, p, (2 * t + 1) * 4);
#pragma unroll
        for (int i = 0; i < 2 * MT; i++) {
            // -2 * popc(a ^ w) over this slice
            const int v0 = 4 * acc[i >> 1][j][2 * (i & 1)] - 2 * sa[i] - 2 * pw0;
            const int v1 = 4 * acc[i >> 1][j][2 * (i & 1) + 1] - 2 * sa[i] - 2 * pw1;
            *reinterpret_cast<int2*>(mine + (i * 8 + gq) * CP + j * 8 + 2 * t) = make_int2(v0, v1);
        }
    }
    __syncthreads();
    // one thread per output; eight consecutive threads hold eight consecutive columns of a row
    const int total = NW * R * C;
    for (int e0 = 0; e0 < total; e0 += blockDim.x) {
        const int e = e0 + threadIdx.x;
        const int c = e % C, r = (e / C) % R, w = e / (C * R);
        const int row = m0 + r, col = nb + w * C + c;
        const bool in = e < total && row < g.M && col < ncols;
        int v = g.K;
        if (AHEAD && e0 > 0) load_p(e0);
        if (in)
            for (int k = 0; k < KW; k++) v += red[(size_t)(w * KW + k) * R * CP + r * CP + c];
        if (g.mode == GEMM_FC_BITS) {
            // (float)K - 2*(float)c >= thr[n]  (kernel.cuh:210-213)
            const bool bit = in && col < g.N && (float)v >= (AHEAD ? f0 : ld_dep(g.p0 + col));
            const uint32_t bits = __ballot_sync(0xffffffffu, bit) >> (lane & 24);
            if (in && (lane & 7) == 0)                     // column `col` at bit 31 - col % 32 of its word
                reinterpret_cast<unsigned char*>((uint32_t*)g.out + (size_t)row * g.ldo + (col >> 5))[3 - ((col & 31) >> 3)] =
                    (unsigned char)(__brev(bits & 0xFFu) >> 24);
        } else if (in) {
            if (g.mode == GEMM_INT32) ((int32_t*)g.out)[(size_t)row * g.ldo + col] = v;
            else ((float*)g.out)[(size_t)row * g.ldo + col] = AHEAD ? __fmaf_rn((float)v, f0, f1) : __fmaf_rn((float)v, ld_dep(g.p0 + col), ld_dep(g.p1 + col));
        }
    }
}

}  // namespace tcbnn
