// Attention of many query tokens (a prompt, or new tokens behind a cache) in one launch: softmax(q K^T scale + mask) V in fp32.
//
// Op by op this was: the keys copied out transposed and repeated per query head, a SIMT product of 64-wide rows, the softmax chain over a
// [B, H, S, T] tensor in HBM and a second SIMT product - the FMA pipe bounds the products, HBM the rest.  Here a CTA keeps 128 query
// rows of one KV head (the rows of the query heads that share it lie behind one another, so short prompts fill the tile too) and walks
// over the keys in blocks of 64.  Both contractions run on tcgen05.mma kind::f16 over pairs of f16 (split_pair.cuh: 22-23 bits), high x high
// and the two mixed products in accumulators of their own; scores and probabilities never leave the SM.  One thread owns one row: scores
// come out of TMEM into its registers, the running maximum and sum and the 64 output sums stay in registers in fp32, and the
// probabilities go back through shared memory as pairs.
//
// What bounds it: the chain of one block - mask and keys in, scores, softmax, probabilities, values - through which a CTA goes step by step; issue
// slots are 32 % busy.  Two CTAs per SM (98 KB, 256 TMEM columns, 255 registers) overlap their chains.  [4, 32 heads, 512] queries over 512 keys
// take 110 us, with 2-norm error 2.1e-7 (fp32 products and softmax op by op: 2.7e-7).
// Prompts of 16 x 512 tokens 80.9 -> 60.5 ms, of 3 x 187 tokens 5.5 -> 5.2 ms.
// A block of keys whose mask is the lowest fp32 value (or -inf) for every row of the tile contributes exactly zero once a row has seen a
// score of ordinary size; such a block is passed over when all its values are finite and of ordinary size.
// (Fetching it costs most of what a block costs: the causal mask above measured no faster than one that hides nothing.)
#include <mutex>

#include "split_pair.cuh"
#include "umma_gemm.cuh"

namespace rmlk {
namespace prefill {

using namespace umma;

constexpr int D = 64;          // head size
constexpr int QT = 128;        // query rows per CTA = MMA M = threads
constexpr int KT = 64;         // keys per block
constexpr uint32_t QH = 0, QL = 16384, KH = 32768, VH = 49152, PH = 65536, PL = 81920;  // low tiles of K and V lie 8 KB behind the high ones
constexpr uint32_t ROW_OFF = 98304, RED = ROW_OFF + QT * 8, BARS = RED + 4 * 16 + 16, TOTAL = BARS + 32 + 1024;
constexpr float P_SCALE = 16384.f;  // probabilities are at most 1
// Queries of a tile share a scale, keys of a block do, values of a block do.  Values far below the largest are held to 2^-50 of that:
// Scores are off by less than 2^-43 |q|max |k|max scale through it, less than a rounding of the exponent's argument up to here; above, or where the
// values of the blocks span more than pairs hold and a result is too small to hide it, the tile is left to rows_in_fp32.
constexpr float SCORES_MOST = 65536.f;

struct Params {
    const float *q, *k, *v, *mask;
    float* out;
    int64_t kb, vb;              // problem strides of K and V
    int64_t ms_b, ms_h, ms_s;    // mask strides per batch entry, head and query
    int64_t os_b, os_h, os_s;    // output strides
    int rows, S, G, T, kv_heads, tiles;
    int mask_vec;                // rows of the mask are 16-byte aligned
    float scale;
    int* status;
};

// 16-byte unit c of row r in a tile of 128-byte rows, 128-byte swizzle
__device__ __forceinline__ uint32_t unit(int r, int c) { return static_cast<uint32_t>(r * 128 + ((c ^ (r & 7)) << 4)); }

struct Mags {
    uint32_t finite, any;  // bits of the largest finite magnitude, of the largest magnitude
    __device__ __forceinline__ void add(float4 x) {
        one(x.x); one(x.y); one(x.z); one(x.w);
    }
    __device__ __forceinline__ void one(float x) {
        finite = max(finite, finite_abs_bits(x));
        any = max(any, __float_as_uint(x) & 0x7fffffffu);
    }
    __device__ __forceinline__ void warp_max() {
        finite = __reduce_max_sync(0xffffffffu, finite);
        any = __reduce_max_sync(0xffffffffu, any);
    }
};

// four values of row r, columns 4 c4 .. 4 c4 + 3, as pairs; the low tile `low` bytes behind the high one
__device__ __forceinline__ void put_pairs(uint8_t* tile, uint32_t low, int r, int c4, float4 x, float up) {
    uint2 hi, lo;
    split2(x.x * up, x.y * up, hi.x, lo.x);
    split2(x.z * up, x.w * up, hi.y, lo.y);
    uint8_t* at = tile + unit(r, c4 >> 1) + (c4 & 1) * 8;
    *reinterpret_cast<uint2*>(at) = hi;
    *reinterpret_cast<uint2*>(at + low) = lo;
}

// high x high + 2^-11 (the mixed products); a sum that is not finite is what the fp32 product would be (see umma_gemm_kernel.cuh)
__device__ __forceinline__ float joined(uint32_t high, uint32_t low) {
    const float h = __uint_as_float(high);
    return fabsf(h) < INFINITY ? fmaf(__uint_as_float(low), 1.f / LO_SCALE, h) : h;
}

// The tile's rows one per thread in fp32.  512 keys: one tile 353 us (58 us on pairs), all tiles of [4, 32 heads, 512] queries 876 us (107 us).
__device__ __noinline__ void rows_in_fp32(const Params& p, int64_t prob, int row0, int64_t mask_row) {
    const int row = row0 + threadIdx.x;
    if (row >= p.rows) return;
    const int64_t b = prob / p.kv_heads;
    const int g = row / p.S, s_at = row - g * p.S;
    const int64_t h = (prob - b * p.kv_heads) * p.G + g;
    const float4* Q = reinterpret_cast<const float4*>(p.q + (prob * p.rows + row) * D);
    const float4* K = reinterpret_cast<const float4*>(p.k + prob * p.kb);
    const float4* V = reinterpret_cast<const float4*>(p.v + prob * p.vb);
    float4 q[D / 4], acc[D / 4];
#pragma unroll
    for (int j = 0; j < D / 4; j++) {
        q[j] = Q[j];
        acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float top = -INFINITY, sum = 0.f;
#pragma unroll 1
    for (int64_t t = 0; t < p.T; t++) {
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < D / 4; j++) {
            const float4 k = K[t * (D / 4) + j];
            d.x = fmaf(q[j].x, k.x, d.x);
            d.y = fmaf(q[j].y, k.y, d.y);
            d.z = fmaf(q[j].z, k.z, d.z);
            d.w = fmaf(q[j].w, k.w, d.w);
        }
        float x = __fmul_rn((d.x + d.y) + (d.z + d.w), p.scale);
        if (p.mask) x = __fadd_rn(x, p.mask[mask_row + t]);
        if (x > top) {
            const float corr = top == -INFINITY ? 0.f : expf(top - x);
            top = x;
            sum *= corr;
#pragma unroll
            for (int j = 0; j < D / 4; j++) acc[j] = make_float4(acc[j].x * corr, acc[j].y * corr, acc[j].z * corr, acc[j].w * corr);
        }
        const float e = expf(x - (top == -INFINITY ? 0.f : top));
        sum += e;
#pragma unroll
        for (int j = 0; j < D / 4; j++) {
            const float4 v = V[t * (D / 4) + j];
            acc[j] = make_float4(fmaf(e, v.x, acc[j].x), fmaf(e, v.y, acc[j].y), fmaf(e, v.z, acc[j].z), fmaf(e, v.w, acc[j].w));
        }
    }
    float4* o = reinterpret_cast<float4*>(p.out + b * p.os_b + h * p.os_h + s_at * p.os_s);
#pragma unroll
    for (int j = 0; j < D / 4; j++) o[j] = make_float4(acc[j].x / sum, acc[j].y / sum, acc[j].z / sum, acc[j].w / sum);
}

__global__ void __launch_bounds__(QT, 2) attention_kernel(const __grid_constant__ Params p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - smem_u32(smem_raw));
    int64_t* s_row = reinterpret_cast<int64_t*>(sm + ROW_OFF);
    uint4* s_red = reinterpret_cast<uint4*>(sm + RED);
    uint32_t* s_low = reinterpret_cast<uint32_t*>(sm + RED + 64);
    const uint32_t bar_s = base + BARS, bar_o = bar_s + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + BARS + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + BARS + 20);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // TMEM is asked for when the kernel in front has given back its own, and the kernel behind may start once this one has it: neither can
    // hold columns that another one needs in order to finish.
    dep_wait();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(bar_s, 1);
        mbar_init(bar_o, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    const int64_t prob = blockIdx.x / p.tiles;
    const int row0 = static_cast<int>(blockIdx.x - prob * p.tiles) * QT;
    const int64_t b = prob / p.kv_heads;
    const int row = row0 + tid, row_in = min(row, p.rows - 1);
    const int g = row_in / p.S, s_at = row_in - g * p.S;
    const int64_t h = (prob - b * p.kv_heads) * p.G + g;
    s_row[tid] = b * p.ms_b + h * p.ms_h + s_at * p.ms_s;
    const float* Kp = p.k + prob * p.kb;
    const float* Vp = p.v + prob * p.vb;
    const int c4 = tid & 15, r8 = tid >> 4;  // loads: 16 threads per row, 8 rows at a time
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);

    // ---- queries ----
    int qe;
    bool q_plain;
    float k_most;  // scores stay below SCORES_MOST with keys up to this
    {
        float4 x[16];
        const float* Qp = p.q + (prob * p.rows + row0) * D;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int r = r8 + 8 * i;
            x[i] = row0 + r < p.rows ? *reinterpret_cast<const float4*>(Qp + static_cast<int64_t>(r) * D + 4 * c4) : zero4;
        }
        Mags m = {0, 0};
#pragma unroll
        for (int i = 0; i < 16; i++) m.add(x[i]);
        m.warp_max();
        if (lane == 0) s_red[warp] = make_uint4(m.finite, m.any, 0, 0);
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
#pragma unroll
        for (int w = 0; w < 4; w++) {
            m.finite = max(m.finite, s_red[w].x);
            m.any = max(m.any, s_red[w].y);
        }
        qe = scale_exponent(m.finite);
        q_plain = m.any < 0x58800000u;  // 2^50
        k_most = SCORES_MOST / (__uint_as_float(m.finite) * fabsf(p.scale));  // (infinite where all queries are zero)
        const float up = exp2_int(qe);
#pragma unroll
        for (int i = 0; i < 16; i++) put_pairs(sm + QH, QL - QH, r8 + 8 * i, c4, x[i], up);
    }
    const uint32_t tmem = *tmem_slot;
    __syncthreads();  // every thread has read s_red; all of the grid's TMEM requests of this CTA are served
    dep_trigger();

    float4 kx[8], vx[8];
    auto load_kv = [&](int key0) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int t = key0 + r8 + 8 * i;
            const bool in = t < p.T;
            kx[i] = in ? *reinterpret_cast<const float4*>(Kp + static_cast<int64_t>(t) * D + 4 * c4) : zero4;
            vx[i] = in ? *reinterpret_cast<const float4*>(Vp + static_cast<int64_t>(t) * D + 4 * c4) : zero4;
        }
    };
    load_kv(0);

    // idesc: f16 x f16 -> f32, M = 128; the second operand of P V is n-major
    constexpr uint32_t idesc = (1u << 4) | ((KT >> 3) << 17) | ((QT >> 4) << 24), idesc_wide = (1u << 4) | (((2 * KT) >> 3) << 17) | ((QT >> 4) << 24);
    constexpr uint32_t B_N_MAJOR = 1u << 16;
    const uint64_t qh = smem_desc_k128(base + QH), ql = smem_desc_k128(base + QL), kd = smem_desc_k128(base + KH);
    const uint64_t ph = smem_desc_k128(base + PH), pl = smem_desc_k128(base + PL), vd = smem_desc_n128(base + VH);
    const uint32_t lanes = static_cast<uint32_t>(warp * 32) << 16;

    float acc[D];
#pragma unroll
    for (int j = 0; j < D; j++) acc[j] = 0.f;
    float top = -INFINITY, sum = 0.f;
    uint32_t phase = 0;
    bool ok = true, plain = true;  // plain: pairs do
    uint32_t v_max = 0, v_low = 0xffffffffu;
    for (int key0 = 0; key0 < p.T; key0 += KT) {
        // The mask of the block goes where the probabilities will be: the row's first 32 values into its 128 bytes of the high tile, the others into
        // the low tile's, so that a thread overwrites nothing but what it has read.
        if (p.mask && p.mask_vec) {
#pragma unroll 4
            for (int i = 0; i < 16; i++) {
                const int r = r8 + 8 * i, t = key0 + 4 * c4;
                const uint32_t at = PH + (c4 >> 3) * (PL - PH) + unit(r, c4 & 7);
                if (t < p.T) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + at), "l"(p.mask + s_row[r] + t) : "memory");
                else *reinterpret_cast<float4*>(sm + at) = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            }
        } else {
#pragma unroll 4
            for (int i = 0; i < QT * KT / QT; i++) {
                const int e = tid + i * QT, r = e / KT, c = e % KT, t = key0 + c;
                const uint32_t at = PH + (c >> 5) * (PL - PH) + unit(r, (c & 31) >> 2) + (c & 3) * 4;
                if (p.mask && t < p.T) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(base + at), "l"(p.mask + s_row[r] + t) : "memory");
                else *reinterpret_cast<float*>(sm + at) = t < p.T ? 0.f : -INFINITY;
            }
        }
        Mags km = {0, 0}, vm = {0, 0};
        uint32_t low = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            km.add(kx[i]);
            vm.add(vx[i]);
            low = min(min(low, min(nonzero_low(vx[i].x), nonzero_low(vx[i].y))), min(nonzero_low(vx[i].z), nonzero_low(vx[i].w)));
        }
        km.warp_max();
        vm.warp_max();
        low = __reduce_min_sync(0xffffffffu, low);
        if (lane == 0) {
            s_red[warp] = make_uint4(km.finite, km.any, vm.finite, vm.any);
            s_low[warp] = low;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
#pragma unroll
        for (int w = 0; w < 4; w++) {
            const uint4 x = s_red[w];
            km.finite = max(km.finite, x.x);
            km.any = max(km.any, x.y);
            vm.finite = max(vm.finite, x.z);
            vm.any = max(vm.any, x.w);
            low = min(low, s_low[w]);
        }
        if (key0 > 0 && p.mask) {
            float most = -INFINITY;
#pragma unroll
            for (int c = 0; c < 16; c++) {
                const float4 x = *reinterpret_cast<const float4*>(sm + PH + (c >> 3) * (PL - PH) + unit(tid, c & 7));
                // (written so that a NaN in the mask keeps the block)
                most = !(x.x <= most) ? x.x : most;
                most = !(x.y <= most) ? x.y : most;
                most = !(x.z <= most) ? x.z : most;
                most = !(x.w <= most) ? x.w : most;
                if (!(most <= -1e38f)) break;
            }
            const bool nothing = most <= -1e38f && top > -1e30f && top < 1e30f && fabsf(p.scale) < 1e6f;
            if (__syncthreads_and((nothing || row >= p.rows) && q_plain && km.any < 0x58800000u && vm.any < 0x7f800000u)) {
                load_kv(key0 + KT);
                continue;
            }
        }
        v_max = max(v_max, vm.finite);
        v_low = min(v_low, low);
        if (!(__uint_as_float(km.finite) <= k_most)) {
            plain = false;
            break;
        }
        const int ke = scale_exponent(km.finite), ve = scale_exponent(vm.finite);
        {
            const float ku = exp2_int(ke), vu = exp2_int(ve);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                put_pairs(sm + KH, 8192, r8 + 8 * i, c4, kx[i], ku);
                put_pairs(sm + VH, 8192, r8 + 8 * i, c4, vx[i], vu);
            }
        }
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                mma_f16<1>(tmem, qh + kk * 2, kd + kk * 2, idesc_wide, kk > 0);  // the low rows of K follow the high ones: one MMA of twice the width
                mma_f16<1>(tmem + KT, ql + kk * 2, kd + kk * 2, idesc, 1u);
            }
            commit<1>(bar_s);
        }
        load_kv(key0 + KT);
        // q k: 2^-(qe + ke); formed first where it is a normal number, so that neither alone takes a score out of range
        const float a = exp2_int(-qe), t2 = exp2_int(-ke), both = a * t2;
        const bool normal = both >= 1.17549435e-38f && both < INFINITY;
        const float f1 = normal ? both : a, f2 = normal ? p.scale : t2 * p.scale;

        ok = mbar_wait(bar_s, phase, abort_flag, p.status) && ok;
        __syncwarp();
        tc_fence_after();
        float s[KT];
        float most = -INFINITY;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            uint32_t hi[32], lo[32];
            tmem_ld_x32(tmem + lanes + half * 32, hi);
            tmem_ld_x32(tmem + lanes + KT + half * 32, lo);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const float4 x = *reinterpret_cast<const float4*>(sm + PH + half * (PL - PH) + unit(tid, c));
                const int j = 4 * c;
                s[32 * half + j] = __fadd_rn(__fmul_rn(joined(hi[j], lo[j]) * f1, f2), x.x);
                s[32 * half + j + 1] = __fadd_rn(__fmul_rn(joined(hi[j + 1], lo[j + 1]) * f1, f2), x.y);
                s[32 * half + j + 2] = __fadd_rn(__fmul_rn(joined(hi[j + 2], lo[j + 2]) * f1, f2), x.z);
                s[32 * half + j + 3] = __fadd_rn(__fmul_rn(joined(hi[j + 3], lo[j + 3]) * f1, f2), x.w);
            }
        }
#pragma unroll
        for (int j = 0; j < KT; j++) most = fmaxf(most, s[j]);
        most = fmaxf(most, top);
        const float shift = most == -INFINITY ? 0.f : most;  // nothing but -inf so far: every weight is zero
        const float corr = top == -INFINITY ? 0.f : expf(top - most);
        top = most;
        float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 8; c++) {
            float e[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                e[j] = expf(s[8 * c + j] - shift);
                part[j & 3] += e[j];
            }
            uint4 hi, lo;
            split8(e, P_SCALE, hi, lo);
            *reinterpret_cast<uint4*>(sm + PH + unit(tid, c)) = hi;
            *reinterpret_cast<uint4*>(sm + PL + unit(tid, c)) = lo;
        }
        sum = fmaf(sum, corr, (part[0] + part[1]) + (part[2] + part[3]));
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                mma_f16<1>(tmem + 128, ph + kk * 2, vd + kk * 128, idesc_wide | B_N_MAJOR, kk > 0);
                mma_f16<1>(tmem + 128 + D, pl + kk * 2, vd + kk * 128, idesc | B_N_MAJOR, 1u);
            }
            commit<1>(bar_o);
        }
        const float fv = exp2_int(-ve) * (1.f / P_SCALE);
        ok = mbar_wait(bar_o, phase, abort_flag, p.status) && ok;
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int half = 0; half < 2; half++) {
            uint32_t hi[32], lo[32];
            tmem_ld_x32(tmem + lanes + 128 + half * 32, hi);
            tmem_ld_x32(tmem + lanes + 128 + D + half * 32, lo);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; j++) acc[32 * half + j] = fmaf(acc[32 * half + j], corr, joined(hi[j], lo[j]) * fv);
        }
        tc_fence_before();
        phase ^= 1;
    }
    const bool bad = __syncthreads_or(!ok);
    if (plain && !pairs_hold(v_max, v_low)) {  // the same in every thread
        // each block's share is off by less than 2^-43 of the largest value: by 2^-21 of a result that is not below this
        const float least = __uint_as_float(v_max) * (1.f / 4194304.f) * static_cast<float>(p.T / KT + 1);
        bool small = false;
#pragma unroll
        for (int j = 0; j < D; j++) small = small || fabsf(acc[j]) < least;
        plain = !__syncthreads_or(small && row < p.rows);
    }
    if (!plain && !bad) {
        rows_in_fp32(p, prob, row0, s_row[tid]);
    } else if (row < p.rows) {
        float4* o = reinterpret_cast<float4*>(p.out + b * p.os_b + h * p.os_h + s_at * p.os_s);
        const float nan = __int_as_float(0x7fc00000);
#pragma unroll
        for (int j = 0; j < D / 4; j++)
            o[j] = bad ? make_float4(nan, nan, nan, nan) : make_float4(acc[4 * j] / sum, acc[4 * j + 1] / sum, acc[4 * j + 2] / sum, acc[4 * j + 3] / sum);
    }
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
    }
}

}  // namespace prefill
}  // namespace rmlk

using namespace rmlk;

extern "C" int rmlk_b200_gqa_prefill_attention_supported(int64_t queries, int64_t rows, int64_t head_dim, int64_t keys) {
    return tc_enabled() && queries >= 1 && rows >= 1 && queries < (1ll << 24) && rows < (1ll << 20) && queries * rows < (1ll << 30) && head_dim == prefill::D && keys >= 1 &&
           keys < (1ll << 30);
}

extern "C" int rmlk_b200_gqa_prefill_attention(rmlk_stream_t stream, int dtype, int64_t problems, int64_t rows, int64_t queries, int64_t head_dim, int64_t keys,
                                               int64_t kv_heads, const void* q, const void* k, int64_t k_problem_stride, const void* v, int64_t v_problem_stride,
                                               float scale, const void* mask, const int64_t* mask_strides, void* out, const int64_t* out_strides, int* status) {
    if (dtype != RMLK_F32) return fail(RMLK_ERR_UNSUPPORTED_DTYPE, "unsupported data type for gqa_prefill_attention (f32 only)");
    if (problems < 0 || kv_heads <= 0) return fail(RMLK_ERR_INVALID_ARG, "gqa_prefill_attention: bad extent");
    if (!rmlk_b200_gqa_prefill_attention_supported(queries, rows, head_dim, keys)) return fail(RMLK_ERR_INVALID_ARG, "gqa_prefill_attention: needs head_dim 64");
    if (problems == 0) return RMLK_OK;
    if (!q || !k || !v || !out || !out_strides || (mask && !mask_strides)) return fail(RMLK_ERR_INVALID_ARG, "gqa_prefill_attention: NULL pointer");
    if (!aligned_to(q, 16) || !aligned_to(k, 16) || !aligned_to(v, 16) || !aligned_to(out, 16) || k_problem_stride % 4 || v_problem_stride % 4 || out_strides[0] % 4 ||
        out_strides[1] % 4 || out_strides[2] % 4)
        return fail(RMLK_ERR_INVALID_ARG, "gqa_prefill_attention: operands must be 16-byte aligned");
    prefill::Params p = {};
    p.q = static_cast<const float*>(q);
    p.k = static_cast<const float*>(k);
    p.v = static_cast<const float*>(v);
    p.mask = static_cast<const float*>(mask);
    p.out = static_cast<float*>(out);
    p.kb = k_problem_stride;
    p.vb = v_problem_stride;
    if (mask) {
        p.ms_b = mask_strides[0];
        p.ms_h = mask_strides[1];
        p.ms_s = mask_strides[2];
        p.mask_vec = aligned_to(mask, 16) && keys % 4 == 0 && p.ms_b % 4 == 0 && p.ms_h % 4 == 0 && p.ms_s % 4 == 0;
    }
    p.os_b = out_strides[0];
    p.os_h = out_strides[1];
    p.os_s = out_strides[2];
    p.rows = static_cast<int>(rows * queries);
    p.S = static_cast<int>(queries);
    p.G = static_cast<int>(rows);
    p.T = static_cast<int>(keys);
    p.kv_heads = static_cast<int>(kv_heads);
    p.tiles = static_cast<int>(ceil_div64(p.rows, prefill::QT));
    p.scale = scale;
    p.status = status;
    if (problems * p.tiles > 0x7fffffffll) return fail(RMLK_ERR_INVALID_ARG, "gqa_prefill_attention: too many problems");
    static std::once_flag configured[64];  // the dynamic shared memory limit is raised once per device
    int dev = 0;
    cudaGetDevice(&dev);
    cudaError_t cfg_err = cudaSuccess;
    if (dev >= 0 && dev < 64)
        std::call_once(configured[dev], [&] { cfg_err = cudaFuncSetAttribute(prefill::attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, prefill::TOTAL); });
    RMLK_CUDA(cfg_err);
    launch_dep(prefill::attention_kernel, dim3(static_cast<unsigned>(problems * p.tiles)), dim3(prefill::QT), prefill::TOTAL, as_stream(stream), p);
    RMLK_CHECK_LAUNCH("prefill attention_kernel");
    return RMLK_OK;
}
