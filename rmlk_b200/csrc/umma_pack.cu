// fp32 operands of the tensor-core MatMul as pairs of f16.
//
// x = (hi + lo / 2^11) * 2^-e: a power of two per column of W (per row of X) brings the largest value of the column to [2^14, 2^15),
// hi is x * 2^e rounded to f16 (11 significant bits), lo the exact rest times 2^11, again rounded to f16.  Together they hold 22 to
// 23 significant bits of every value down to 2^-29 of its column's largest, and at least 2^-51 of that largest below - more
// than the two TF32 terms (21 bits) of the kernel that splits in flight, at twice its MMA rate.  A column or row with values below
// 2^-28 of its largest is marked by the sign of its scale: the product then looks at each of its sums, and forms those again in fp32 in which
// what pairs lost could show (a table read by one-hot rows with one entry of the lowest float in a column, say).
//
// Weights go into blocks of [64 k][128 n], the high and the low tile of a block behind one another (32 KB that one TMA request
// brings in), each laid out as the MMA reads it from shared memory: two [64 k][64 n] parts, 128-byte rows, 16-byte units swizzled by
// the row.  K is padded to a multiple of 64 and N to a multiple of 128 with zeros, so any size is taken.
// Rows go into two plain row-major f16 matrices (high over low) that TMA swizzles on its way in.
#include <algorithm>

#include "split_pair.cuh"

namespace rmlk {
namespace umma {

// Eight consecutive columns of row k of the matrices laid side by side
__device__ __forceinline__ void load8(const WeightSources& s, int64_t k, int64_t n0, float (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = 0.f;
    int j = 0;
    while (j + 1 < s.count && n0 >= s.col0[j + 1]) j++;
    const int64_t c = n0 - s.col0[j];
    const float* row = s.w[j] + k * s.n[j];
    if (s.vec[j] && c + 8 <= s.n[j]) {
        const float4 a = *reinterpret_cast<const float4*>(row + c), b = *reinterpret_cast<const float4*>(row + c + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        int64_t n = n0 + i;
        int q = j;
        while (q + 1 < s.count && n >= s.col0[q + 1]) q++;
        if (n < s.col0[q] + s.n[q]) x[i] = s.w[q][k * s.n[q] + n - s.col0[q]];
    }
}

// Largest finite magnitude of every column, and its smallest one that is not zero.  Grid: blocks of 128 columns x ranges of rows; 16 threads of 8 columns times 16 rows.
__global__ void __launch_bounds__(256) column_range_kernel(WeightSources s, int64_t K, int64_t rows_per_block, uint32_t* __restrict__ colmax, uint32_t* __restrict__ collow) {
    dep_sync();
    __shared__ uint32_t sm[128], sl[128];
    const int c8 = threadIdx.x & 15, r = threadIdx.x >> 4;
    const int64_t n0 = static_cast<int64_t>(blockIdx.x) * 128 + c8 * 8;
    const int64_t k0 = static_cast<int64_t>(blockIdx.y) * rows_per_block, k1 = min(K, k0 + rows_per_block);
    if (threadIdx.x < 128) {
        sm[threadIdx.x] = 0;
        sl[threadIdx.x] = 0xffffffffu;
    }
    __syncthreads();
    uint32_t mx[8], low[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        mx[i] = 0;
        low[i] = 0xffffffffu;
    }
#pragma unroll 4
    for (int64_t k = k0 + r; k < k1; k += 16) {
        float x[8];
        load8(s, k, n0, x);
#pragma unroll
        for (int i = 0; i < 8; i++) {
            mx[i] = max(mx[i], finite_abs_bits(x[i]));
            low[i] = min(low[i], nonzero_low(x[i]));
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        atomicMax(&sm[c8 * 8 + i], mx[i]);
        atomicMin(&sl[c8 * 8 + i], low[i]);
    }
    __syncthreads();
    if (threadIdx.x < 128 && sm[threadIdx.x]) {
        atomicMax(colmax + static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x, sm[threadIdx.x]);
        atomicMax(collow + static_cast<int64_t>(blockIdx.x) * 128 + threadIdx.x, ~sl[threadIdx.x]);  // inverted: one memset clears both
    }
}

// Grid: blocks of 128 columns x blocks of 64 rows.
__global__ void __launch_bounds__(256) pack_weights_kernel(WeightSources s, int64_t K, const uint32_t* __restrict__ colmax, const uint32_t* __restrict__ collow,
                                                           float* __restrict__ colcount, uint8_t* __restrict__ tiles, float* __restrict__ w_scale) {
    dep_sync();
    const int c8 = threadIdx.x & 15, r0 = threadIdx.x >> 4;
    const int64_t nb = blockIdx.x, n0 = nb * 128 + c8 * 8;
    const int64_t kb = blockIdx.y;
    uint8_t* tile = tiles + (nb * gridDim.y + kb) * 32768;
    int e[8];
#pragma unroll
    for (int i = 0; i < 8; i++) e[i] = scale_exponent(colmax[n0 + i]);
    uint32_t marked = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) marked |= pairs_hold(colmax[n0 + i], ~collow[n0 + i]) ? 0u : 1u << i;
    if (kb == 0 && r0 == 0) {
#pragma unroll
        for (int i = 0; i < 8; i++) w_scale[n0 + i] = marked >> i & 1 ? -exp2_int(-e[i]) : exp2_int(-e[i]);
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const int r = r0 + p * 16;
        const int64_t k = kb * 64 + r;
        float x[8];
        if (k < K) {
            load8(s, k, n0, x);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] *= exp2_int(e[i]);
        if (marked) {
#pragma unroll
            for (int i = 0; i < 8; i++)
                if ((marked >> i & 1) && is_lossy(x[i])) atomicAdd(colcount + n0 + i, 1.f);
        }
        uint4 hi, lo;
        split8(x, 1.f, hi, lo);
        const uint32_t off = (c8 >> 3) * 8192 + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(tile + off) = hi;
        *reinterpret_cast<uint4*>(tile + 16384 + off) = lo;
    }
}

// One CTA per row: its largest magnitude, then both parts.  A row is read twice, the second time from L1 / L2.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, int64_t ldx, int64_t K, int64_t k_pad, int64_t m_pad, __half* __restrict__ out,
                                                         float* __restrict__ x_scale, int64_t count, int vec) {
    dep_sync();
    __shared__ uint32_t sm, sl;
    const int64_t m = blockIdx.x;
    const float* row = x + m * ldx;
    if (threadIdx.x == 0) {
        sm = 0;
        sl = 0xffffffffu;
    }
    __syncthreads();
    uint32_t mx = 0, low = 0xffffffffu;
    if (vec) {
        for (int64_t k = threadIdx.x * 4; k < K; k += 1024) {
            const float4 v = *reinterpret_cast<const float4*>(row + k);
            mx = max(max(mx, max(finite_abs_bits(v.x), finite_abs_bits(v.y))), max(finite_abs_bits(v.z), finite_abs_bits(v.w)));
            low = min(min(low, min(nonzero_low(v.x), nonzero_low(v.y))), min(nonzero_low(v.z), nonzero_low(v.w)));
        }
    } else {
        for (int64_t k = threadIdx.x; k < K; k += 256) {
            mx = max(mx, finite_abs_bits(row[k]));
            low = min(low, nonzero_low(row[k]));
        }
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    low = __reduce_min_sync(0xffffffffu, low);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&sm, mx);
        atomicMin(&sl, low);
    }
    __syncthreads();
    const int e = scale_exponent(sm);
    const float scale = exp2_int(e);
    const bool hold = pairs_hold(sm, sl);
    if (threadIdx.x == 0) x_scale[m] = hold ? exp2_int(-e) : -exp2_int(-e);
    int lossy = 0;
    __half* hrow = out + m * k_pad;
    __half* lrow = hrow + m_pad * k_pad;
    for (int64_t k = threadIdx.x * 8; k < k_pad; k += 2048) {
        float v[8];
        if (vec && k + 8 <= K) {
            const float4 a = *reinterpret_cast<const float4*>(row + k), b = *reinterpret_cast<const float4*>(row + k + 4);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = k + i < K ? row[k + i] : 0.f;
        }
        uint4 hi, lo;
        split8(v, scale, hi, lo);
        *reinterpret_cast<uint4*>(hrow + k) = hi;
        *reinterpret_cast<uint4*>(lrow + k) = lo;
        if (!hold) {
#pragma unroll
            for (int i = 0; i < 8; i++) lossy += is_lossy(v[i] * scale);
        }
    }
    if (!hold) {  // the same in every thread
        __shared__ int total;
        if (threadIdx.x == 0) total = 0;
        __syncthreads();
        lossy = __reduce_add_sync(0xffffffffu, lossy);
        if ((threadIdx.x & 31) == 0) atomicAdd(&total, lossy);
        __syncthreads();
        if (threadIdx.x == 0) x_scale[count + m] = static_cast<float>(total);
    }
}

}  // namespace umma

static int64_t pad_to(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

size_t split_weights_bytes(int64_t n, int64_t k) {
    const int64_t nb = ceil_div64(n, 128), kb = ceil_div64(k, 64);
    return static_cast<size_t>(nb) * kb * 32768 + static_cast<size_t>(nb) * 128 * 16;
}

SplitWeights split_weights_at(void* buf, int64_t n, int64_t k) {
    SplitWeights w = {};
    w.n = n;
    w.k = k;
    w.n_blocks = ceil_div64(n, 128);
    w.k_blocks = ceil_div64(k, 64);
    w.tiles = buf;
    w.scale = reinterpret_cast<float*>(static_cast<char*>(buf) + static_cast<size_t>(w.n_blocks) * w.k_blocks * 32768);
    w.count = 3 * w.n_blocks * 128;
    return w;
}

SplitWeights split_weights_window(const SplitWeights& w, int64_t n0, int64_t n) {
    SplitWeights r = w;
    r.n = n;
    r.n_blocks = ceil_div64(n, 128);
    r.tiles = static_cast<char*>(w.tiles) + (n0 / 128) * w.k_blocks * 32768;
    r.scale = w.scale + n0;
    r.col0 = w.col0 + n0;
    return r;
}

int split_weights_pack(cudaStream_t st, const WeightSources& src, SplitWeights& w) {
    if (w.n_blocks > 0x7fffffffll || w.k_blocks > 65535) return fail(RMLK_ERR_INVALID_ARG, "matmul: weights too large to pack");
    w.src = src;
    uint32_t* colmax = reinterpret_cast<uint32_t*>(w.scale + w.n_blocks * 128);
    uint32_t* collow = colmax + w.n_blocks * 128;
    RMLK_CUDA(cudaMemsetAsync(colmax, 0, static_cast<size_t>(w.n_blocks) * 1536, st));
    // about 8 CTAs per SM
    int64_t ranges = std::max<int64_t>(1, std::min<int64_t>(ceil_div64(8ll * sm_count(), w.n_blocks), ceil_div64(w.k, 64)));
    const int64_t rows = ceil_div64(w.k, ranges);
    ranges = ceil_div64(w.k, rows);
    launch_dep(umma::column_range_kernel, dim3(static_cast<unsigned>(w.n_blocks), static_cast<unsigned>(ranges)), dim3(256), 0, st, src, w.k, rows, colmax, collow);
    RMLK_CHECK_LAUNCH("column_range_kernel");
    launch_dep(umma::pack_weights_kernel, dim3(static_cast<unsigned>(w.n_blocks), static_cast<unsigned>(w.k_blocks)), dim3(256), 0, st, src, w.k,
               static_cast<const uint32_t*>(colmax), static_cast<const uint32_t*>(collow), w.scale + w.count, static_cast<uint8_t*>(w.tiles), w.scale);
    RMLK_CHECK_LAUNCH("pack_weights_kernel");
    return RMLK_OK;
}

SplitRows split_rows_at(void* buf, int64_t m, int64_t k, int chunk_blocks, bool keep_full) {
    SplitRows x = {};
    x.m = m;
    x.k = k;
    x.m_pad = pad_to(m, 64);
    x.k_pad = pad_to(k, 64);
    x.chunk_blocks = chunk_blocks > 0 ? chunk_blocks : static_cast<int>(x.k_pad / 64);
    x.scale_pitch = x.m_pad + 256;  // a tile of up to 256 rows may read scales behind the last row
    x.data = buf;
    x.scale = reinterpret_cast<float*>(static_cast<char*>(buf) + static_cast<size_t>(x.m_pad) * x.k_pad * 4);
    x.count = ceil_div64(x.k_pad / 64, x.chunk_blocks) * x.scale_pitch;
    if (keep_full) {
        x.full = x.scale + 2 * x.count;
        x.full_ld = k;
    }
    return x;
}

size_t split_rows_bytes(int64_t m, int64_t k, int chunk_blocks, bool keep_full) {
    const SplitRows x = split_rows_at(nullptr, m, k, chunk_blocks, keep_full);
    return static_cast<size_t>(x.m_pad) * x.k_pad * 4 + static_cast<size_t>(x.count) * 8 +
           (keep_full ? static_cast<size_t>(m) * k * 4 : 0);
}

int split_rows_pack(cudaStream_t st, const float* x, int64_t ldx, SplitRows& dst) {
    dst.full = const_cast<float*>(x);
    dst.full_ld = ldx;
    dst.full_all = true;
    if (dst.m > 0x7fffffffll) return fail(RMLK_ERR_INVALID_ARG, "matmul: too many rows");
    const int vec = aligned_to(x, 16) && ldx % 4 == 0 && dst.k % 4 == 0;
    launch_dep(umma::split_rows_kernel, dim3(static_cast<unsigned>(dst.m)), dim3(256), 0, st, x, ldx, dst.k, dst.k_pad, dst.m_pad, static_cast<__half*>(dst.data),
               dst.scale, dst.count, vec);
    RMLK_CHECK_LAUNCH("split_rows_kernel");
    return RMLK_OK;
}

}  // namespace rmlk
