// MatMul on tcgen05.mma kind::f16: f16 operands as they are, fp32 operands as pairs of f16.
//
// Orientation.  A CTA owns 128 columns of W - the MMA's M dimension, one TMEM lane per column - and a tile of MT rows of X, the
// MMA's N dimension; a pair of CTAs (cta_group::2) shares 256 columns, each holding its 128 columns of W and half of the rows of
// X.  The accumulator is C transposed, so that a warp of the epilogue writes 32 consecutive columns of a row at a time.
#include "umma_gemm.h"

#include <algorithm>
#include <mutex>

#include "umma_gemm_kernel.cuh"

namespace rmlk {
namespace umma {

static bool map_2d_f16(CUtensorMap* map, const void* ptr, uint64_t inner, uint64_t outer, uint64_t pitch, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle) {
    tc::EncodeTiledFn fn = tc::encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {pitch * 2};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CG, bool SPLIT, int MT, int ST, bool OUT16>
static int launch(cudaStream_t st, const CUtensorMap& tmW, const CUtensorMap& tmX, const Params& p) {
    using L = Layout<CG, SPLIT, MT, ST>;
    auto kernel = gemm_kernel<CG, SPLIT, MT, ST, OUT16>;
    static std::once_flag configured[64];  // the dynamic shared memory limit is raised once per device
    int dev = 0;
    cudaGetDevice(&dev);
    cudaError_t cfg_err = cudaSuccess;
    if (dev >= 0 && dev < 64)
        std::call_once(configured[dev], [&] { cfg_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL); });
    RMLK_CUDA(cfg_err);
    const int64_t items = static_cast<int64_t>(p.n_tiles) * p.m_tiles * p.ksplit;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(CG * std::min<int64_t>(items, sm_count() / CG)));
    cfg.blockDim = dim3(L::THREADS);
    cfg.dynamicSmemBytes = L::TOTAL;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    unsigned na = 0;
    if (CG == 2) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = 2;
        at[na].val.clusterDim.y = 1;
        at[na].val.clusterDim.z = 1;
        na++;
    }
    if (dep_launch_enabled()) {
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = at;
    cfg.numAttrs = na;
    RMLK_CUDA(cudaLaunchKernelEx(&cfg, kernel, tmW, tmX, p));
    RMLK_CHECK_LAUNCH("umma gemm_kernel");
    return RMLK_OK;
}

struct Plan {
    int cg, mt, ksplit;
};

// Tile shape for a product: the shape whose waves cost least, an item costing its k-blocks (the MMAs, or the bytes a CTA has to
// bring in where those take longer) plus what starting and storing a tile takes.  `products`: MMAs per product (3 for split operands).
static Plan plan_for(int64_t m, int64_t n, int64_t k, int products, bool may_split, bool chunks = false) {
    static const int shapes[][2] = {{1, 16}, {1, 32}, {1, 64}, {1, 128}, {2, 128}, {2, 192}, {2, 256}};
    const int64_t sms = sm_count(), kb = ceil_div64(k, BK);
    Plan best = {1, 16, 1};
    double best_cost = 1e30;
    for (const auto& s : shapes) {
        const int cg = s[0], mt = s[1];
        if (chunks && mt > 128) continue;  // the tall tiles take one scale per row
        const int64_t tiles = ceil_div64(n, BN * cg) * ceil_div64(m, mt), slots = sms / cg;
        int64_t ks = 1;
        // fewer than 16 k-blocks (K up to 960) are not split: adding up the parts costs more than the shorter loop saves
        if (may_split && tiles < slots && kb >= 16) {
            ks = std::min<int64_t>(slots / tiles, std::max<int64_t>(1, kb / 4));
            ks = ceil_div64(kb, ceil_div64(kb, ks));
        }
        const double per_block = std::max(products * 2.0 * mt, (BN + mt / cg) * BK * 2.0 * (products > 1 ? 2 : 1) / 40.0);
        const double item = ceil_div64(kb, ks) * per_block + 1200 + 6.0 * mt;
        const double cost = ceil_div64(tiles * ks, slots) * item + (ks > 1 ? 1500.0 + 4.0 * m * n * ks / 4000.0 : 0.0);
        if (cost < best_cost) {
            best_cost = cost;
            best = {cg, mt, static_cast<int>(ks)};
        }
    }
    return best;
}

template <bool SPLIT, bool OUT16>
static int dispatch(cudaStream_t st, const Plan& pl, const CUtensorMap& tmW, const CUtensorMap& tmX, const Params& p) {
    if (pl.cg == 1) switch (pl.mt) {
        case 16: return launch<1, SPLIT, 16, SPLIT ? 5 : 10, OUT16>(st, tmW, tmX, p);
        case 32: return launch<1, SPLIT, 32, SPLIT ? 5 : 8, OUT16>(st, tmW, tmX, p);
        case 64: return launch<1, SPLIT, 64, SPLIT ? 4 : 8, OUT16>(st, tmW, tmX, p);
        default: return launch<1, SPLIT, 128, SPLIT ? 3 : 6, OUT16>(st, tmW, tmX, p);
    }
    switch (pl.mt) {
        case 128: return launch<2, SPLIT, 128, SPLIT ? 4 : 8, OUT16>(st, tmW, tmX, p);
        case 192: return launch<2, SPLIT, 192, SPLIT ? 3 : 7, OUT16>(st, tmW, tmX, p);
        default: return launch<2, SPLIT, 256, SPLIT ? 3 : 6, OUT16>(st, tmW, tmX, p);
    }
}

static void fill_tiles(Params& p, const Plan& pl, int64_t m, int64_t n, int64_t k) {
    p.M = m;
    p.N = n;
    p.n_tiles = static_cast<int>(ceil_div64(n, BN * pl.cg));
    p.m_tiles = static_cast<int>(ceil_div64(m, pl.mt));
    p.m_group = std::min(p.m_tiles, 8);
    p.k_blocks = static_cast<int>(ceil_div64(k, BK));
    p.k_per_split = static_cast<int>(ceil_div64(p.k_blocks, pl.ksplit));
    p.ksplit = static_cast<int>(ceil_div64(p.k_blocks, p.k_per_split));
}

}  // namespace umma

bool umma_f16_eligible(int64_t m, int64_t n, int64_t k, const void* a, const void* b) {
    // TMA: rows of both operands on 16-byte boundaries; tile counts in 32 bits
    return tc_enabled() && m >= 1 && n % 8 == 0 && k % 8 == 0 && k > 0 && aligned_to(a, 16) && aligned_to(b, 16) && m < (1ll << 24) && n < (1ll << 30) &&
           k < (1ll << 30) && ceil_div64(n, 128) * ceil_div64(m, 16) < (1ll << 30) && tc::encode_fn() != nullptr;
}

int umma_f16(cudaStream_t st, int64_t m, int64_t n, int64_t k, const void* a, const void* b, void* c, int* status) {
    using namespace umma;
    const Plan pl = plan_for(m, n, k, 1, false);
    CUtensorMap tmW, tmX;
    if (!map_2d_f16(&tmW, b, n, k, n, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B) || !map_2d_f16(&tmX, a, k, m, k, BK, pl.mt / pl.cg, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(RMLK_ERR_INTERNAL, "matmul f16: cuTensorMapEncodeTiled failed");
    Params p = {};
    fill_tiles(p, pl, m, n, k);
    p.out = c;
    p.ldc = n;
    p.chunk_blocks = p.k_blocks;
    p.status = status;
    return dispatch<false, true>(st, pl, tmW, tmX, p);
}

int umma_split_parts(int64_t m, int64_t n, int64_t k, bool short_sums) { return umma::plan_for(m, n, k, 3, true, short_sums).ksplit; }

constexpr int SHORT_BLOCKS = 4;
int umma_split(cudaStream_t st, const SplitRows& x, const SplitWeights& w, float* out, int64_t ldc, float* slabs, size_t slab_bytes, int* status, int flags, bool short_sums,
               int* parts) {
    using namespace umma;
    const bool scales = static_cast<int64_t>(x.chunk_blocks) * BK < x.k_pad;  // a scale per chunk of a row
    const bool chunks = scales || short_sums;
    Plan pl = plan_for(x.m, w.n, x.k, 3, parts != nullptr, chunks);
    if (pl.ksplit > 1 && slab_bytes < static_cast<size_t>(pl.ksplit) * x.m * w.n * sizeof(float)) pl = plan_for(x.m, w.n, x.k, 3, false, chunks);
    CUtensorMap tmW, tmX;
    if (!map_2d_f16(&tmW, w.tiles, 64, static_cast<uint64_t>(w.n_blocks) * w.k_blocks * 256, 64, 64, 256, CU_TENSOR_MAP_SWIZZLE_NONE) ||
        !map_2d_f16(&tmX, x.data, x.k_pad, 2 * x.m_pad, x.k_pad, BK, pl.mt / pl.cg, CU_TENSOR_MAP_SWIZZLE_128B))
        return fail(RMLK_ERR_INTERNAL, "matmul: cuTensorMapEncodeTiled failed");
    Params p = {};
    fill_tiles(p, pl, x.m, w.n, x.k);
    p.out = p.ksplit > 1 ? slabs : out;
    p.ldc = p.ksplit > 1 ? w.n : ldc;
    p.w_rows_per_tile = static_cast<int>(w.k_blocks * 256);
    p.x_lo_row = static_cast<int>(x.m_pad);
    p.w_scale = w.scale;
    p.x_scale = x.scale;
    p.K = x.k;
    p.w_src = w.src;
    p.w_col0 = w.col0;
    p.w_count = w.count;
    p.x_count = x.count;
    p.x_full = x.full;
    p.x_full_ld = x.full_ld;
    p.x_full_all = x.full_all ? 1 : 0;
    p.x_pairs = x.data;
    p.x_k_pad = x.k_pad;
    p.x_low = x.m_pad * x.k_pad;
    p.x_scale_pitch = scales ? x.scale_pitch : 0;  // one scale per row: every chunk reads the same one
    p.chunk_blocks = scales || !short_sums ? x.chunk_blocks : SHORT_BLOCKS;
    p.w_static = (flags & RMLK_MATMUL_B_STATIC) ? 1 : 0;
    p.status = status;
    if (parts) *parts = p.ksplit;
    return dispatch<true, false>(st, pl, tmW, tmX, p);
}

}  // namespace rmlk
