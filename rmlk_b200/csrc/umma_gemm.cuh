// Device side of the f16-kind tensor-core MatMul (see umma_gemm.cu for the overview).
#pragma once

#include "matmul_tc.cuh"
#include "umma_gemm.h"

namespace rmlk {
namespace umma {

using tc::cluster_ctarank;
using tc::cluster_sync_all;
using tc::fence_proxy_async;
using tc::mapa_shared;
using tc::mbar_arrive;
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::smem_desc_k128;
using tc::smem_u32;
using tc::tc_fence_after;
using tc::tc_fence_before;
using tc::tmem_ld_x32;

constexpr int BK = 64;     // f16 elements of K per block: one 128-byte row of an activation tile
constexpr int BN = 128;    // weight columns per CTA = MMA M per CTA = TMEM lanes
constexpr float LO_SCALE = 2048.f;            // the low parts are stored 2^11 times their size: their f16 exponent starts where the high part's ends

// Weight tile: two [64 k][64 n] blocks of 8 KB, n contiguous, 128-byte swizzled (what a SWIZZLE_128B box of 64 x 64 leaves in shared
// memory).  MN-major operand descriptor: 64-column blocks 8 KB apart (leading), groups of 8 k-rows 1 KB apart (stride).
constexpr uint32_t W_TILE = BN * BK * 2;
__device__ __forceinline__ uint64_t smem_desc_n128(uint32_t addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3fff);
    d |= static_cast<uint64_t>(8192 >> 4) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

template <int CG>
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 1)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// Arrives on `bar` (in both CTAs of the pair for CG = 2) when every MMA issued so far has completed.
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar) {
    if constexpr (CG == 1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                     "h"(static_cast<uint16_t>(3))
                     : "memory");
}

// 2-D box into this CTA's shared memory; the bytes are counted on `bar`, which for CG = 2 is the first CTA's barrier.
template <int CG>
__device__ __forceinline__ void load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    if constexpr (CG == 1)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                     "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
                     : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                     "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
                     : "memory");
}

__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

struct Params {
    void* out;               // f32 or f16 (OUT16); with ksplit > 1 the f32 slabs [ksplit][M][N]
    int64_t M, N, ldc;
    int n_tiles, m_tiles;    // tiles of CG * 128 columns x MT rows
    int m_group;             // row tiles that share a pass over the columns (tile order)
    int k_blocks, k_per_split, ksplit;
    int w_rows_per_tile;     // packed weights: rows of the tile map per block of 128 columns
    int x_lo_row;            // split activations: row of the low part of row 0 in the activation map
    const float* w_scale;    // split operands: per column / [chunk][x_scale_pitch] per row, exact powers of two, negative where
    const float* x_scale;    // pairs do not hold the column / the row; NULL: none
    int64_t x_scale_pitch;
    int chunk_blocks;        // k-blocks that share a row scale
    int w_static;            // nothing in flight writes the weights: their first loads may go out before the previous kernel has finished
    int* status;
    // Behind what every launch reads:
    int64_t K;               // split operands as they are, for the sums that are formed again (repair): W in its sources, X as fp32 rows
    WeightSources w_src;     // (all of them, or those that pairs do not hold) and as pairs
    int64_t w_col0, w_count, x_count;  // w_scale[w_count + ..], x_scale[x_count + ..]: how many values of a marked column, row are not held
    const float* x_full;
    int64_t x_full_ld, x_k_pad, x_low;
    int x_full_all;
    const void* x_pairs;
};

// CG: CTAs per tile (a pair shares one tile of 256 columns); SPLIT: operands are (high, low) pairs of f16; MT: activation rows per tile; ST: stages
template <int CG, bool SPLIT, int MT, int ST>
struct Layout {
    // Epilogue warps, two or four for each group of 32 TMEM lanes: at most 64 sums per thread, so that nothing spills.
    static constexpr int EPI_WARPS = MT >= 192 ? 16 : 8;
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;  // TMA warp, MMA warp, epilogue warps
    // Small tiles leave registers for the CTAs of the kernels before and behind, which overlap with this one: those of as many threads.
    static constexpr int REGS_FOR = !SPLIT || MT > 64 ? THREADS : MT == 64 ? 512 : 640;
    static constexpr int XR = MT / CG;  // activation rows that this CTA loads
    static constexpr uint32_t W_BYTES = W_TILE * (SPLIT ? 2 : 1);
    static constexpr uint32_t X_TILE = XR * BK * 2;
    static constexpr uint32_t X_BYTES = X_TILE * (SPLIT ? 2 : 1);
    static constexpr uint32_t STAGE = W_BYTES + X_BYTES;
    static constexpr int D_COLS = MT * (SPLIT ? 2 : 1);
    static constexpr int NBUF = D_COLS <= 256 ? 2 : 1;
    static constexpr uint32_t COLS_USED = D_COLS * NBUF;
    static constexpr uint32_t TMEM_COLS = COLS_USED <= 32 ? 32 : COLS_USED <= 64 ? 64 : COLS_USED <= 128 ? 128 : COLS_USED <= 256 ? 256 : 512;
    static constexpr uint32_t BAR_OFFSET = ST * STAGE;
    static constexpr uint32_t N_BARS = 2 * ST + 2 * NBUF;
    static constexpr uint32_t TOTAL = BAR_OFFSET + 8 * N_BARS + 32 + 1024;
    static_assert(COLS_USED <= 512 && TOTAL <= 227 * 1024, "TMEM or shared memory budget exceeded");
    static_assert(X_TILE % 1024 == 0, "a swizzled tile starts on a 1 KB boundary");
};

}  // namespace umma
}  // namespace rmlk
