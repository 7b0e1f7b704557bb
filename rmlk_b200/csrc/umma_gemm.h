// Host entry points of umma_gemm.cu, for the other translation units of the library.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace rmlk {

namespace tc {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn();  // matmul_tc.cu: the driver's tensor-map encoder, NULL if the driver has none
}  // namespace tc
bool tc_enabled();

// C[m, n] = A[m, k] x B[k, n], row-major f16, fp32 accumulation, one rounding.
bool umma_f16_eligible(int64_t m, int64_t n, int64_t k, const void* a, const void* b);
int umma_f16(cudaStream_t st, int64_t m, int64_t n, int64_t k, const void* a, const void* b, void* c, int* status);

// ---- fp32 operands as pairs of f16 (umma_pack.cu) ----
// Up to 4 row-major [k][n_j] matrices laid side by side.
struct WeightSources {
    int count;
    const float* w[4];
    int64_t n[4], col0[4];
    int vec[4];  // rows are 16-byte aligned
};
struct SplitWeights {
    void* tiles;   // [n_blocks][k_blocks][2][16 KB]
    float* scale;  // per column, padded to whole blocks, negative where pairs do not hold the column; behind it the scratch of the packing kernels
    int64_t n, k, n_blocks, k_blocks;
    WeightSources src;  // the fp32 matrices, which have to stay: a column that pairs do not hold is read from them
    int64_t col0;       // first column of a window
    int64_t count;      // scale[count + n]: values of a marked column that pairs do not hold, as a float
};
size_t split_weights_bytes(int64_t n, int64_t k);
SplitWeights split_weights_at(void* buf, int64_t n, int64_t k);  // buf: 1 KB aligned
SplitWeights split_weights_window(const SplitWeights& w, int64_t n0, int64_t n);  // columns [n0, n0 + n), n0 a multiple of 128
int split_weights_pack(cudaStream_t st, const WeightSources& src, SplitWeights& w);

struct SplitRows {
    void* data;    // f16 [2][m_pad][k_pad]: high parts over low parts; rows behind m are never read into a result
    float* scale;  // [chunks][scale_pitch], negative where pairs do not hold the values of the row in the chunk
    int64_t m, k, m_pad, k_pad, scale_pitch;
    int chunk_blocks;  // blocks of 64 k that share a scale
    int64_t count;     // scale[count + ...]: for a negative scale, the values that pairs do not hold, as a float
    float* full;       // rows of k fp32 values, full_ld apart: all of them (full_all), or those that pairs do not hold
    int64_t full_ld;
    bool full_all;
};
// chunk_blocks 0: one scale per row.  keep_full: with room for the fp32 values of rows that pairs do not hold, for a producer to write.
size_t split_rows_bytes(int64_t m, int64_t k, int chunk_blocks, bool keep_full);
SplitRows split_rows_at(void* buf, int64_t m, int64_t k, int chunk_blocks, bool keep_full);
int split_rows_pack(cudaStream_t st, const float* x, int64_t ldx, SplitRows& dst);  // one scale per row; x has to stay, it is dst.full

// out[m, n] = x w.  With `parts` the K splits may be left as f32 slabs [*parts][m][n] in `slabs` (*parts = 1: out holds the result);
// without it, or without room for the slabs, K is not split.
// short_sums: the accumulator, which truncates, takes at most 256 k before it is added to fp32 sums in registers - for products that would
// otherwise run on FMA chains (N no multiple of 128, K none of 32, unaligned operands), so that they lose no accuracy
// ([1000,777] x [777,1003]: 2-norm error 9.7e-7 with one accumulation over K, 3.5e-7 so, 5.0e-7 on the FMA kernel).
int umma_split(cudaStream_t st, const SplitRows& x, const SplitWeights& w, float* out, int64_t ldc, float* slabs, size_t slab_bytes, int* status, int flags, bool short_sums,
               int* parts);
int umma_split_parts(int64_t m, int64_t n, int64_t k, bool short_sums);  // K splits that the plan would take

// ---- producers that write their result as pairs (fused.cu, attention.cu) ----
// RMSNorm of x, or of x + b (b: b_parts split-K slabs [b_parts][rows][cols]; the sum goes to `sum`)
bool rmsnorm_pairs_supported(int64_t rows, int64_t cols, const float* x, const float* b, int b_parts, const float* weight);
int rmsnorm_pairs(cudaStream_t st, int64_t rows, int64_t cols, const float* x, const float* b, int b_parts, float exponent, float eps, const float* weight, float* sum,
                  const SplitRows& out);
// SwiGLU gate read from K slabs (cols, pitches and part_stride multiples of 4, 16-byte aligned)
int swiglu_slabs(cudaStream_t st, int64_t rows, int64_t cols, const float* gate, int64_t ldg, const float* up, int64_t ldu, int parts, int64_t part_stride, float* out);
bool swiglu_pairs_supported(int64_t rows, int64_t cols);
int swiglu_pairs(cudaStream_t st, int64_t rows, int64_t cols, const float* gate, int64_t ldg, const float* up, int64_t ldu, const SplitRows& out);
// Decode attention (rmlk_b200_gqa_decode_attention) whose result is row b, columns [h rows D, (h + 1) rows D) of `out` for KV head h of batch
// entry b: one scale per KV head (out.chunk_blocks * 64 == rows * D)
int gqa_decode_attention_pairs(cudaStream_t st, int64_t problems, int64_t rows, int64_t head_dim, int64_t keys, int64_t kv_heads, const float* q, const float* k,
                               int64_t kb, const float* v, int64_t vb, float scale, const float* mask, int64_t ms_b, int64_t ms_h, const SplitRows& out);

}  // namespace rmlk
