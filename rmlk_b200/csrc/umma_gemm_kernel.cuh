// gemm_kernel: out[m][n] = sum_k X[m][k] W[k][n] on tcgen05.mma kind::f16.
#pragma once

#include "umma_gemm.cuh"

namespace rmlk {
namespace umma {

__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
template <int W>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* r) {
    if constexpr (W == 32) {
        tmem_ld_x16(taddr, r);
        tmem_ld_x16(taddr + 16, r + 16);
    } else if constexpr (W == 16) {
        tmem_ld_x16(taddr, r);
    } else {
        static_assert(W == 8, "");
        tmem_ld_x8(taddr, r);
    }
}

// high x high + 2^-11 (high x low + low x high).  Where an operand is infinite or NaN its low part is NaN, and an infinity times a low
// part of zero is one too: the high product alone then says what the fp32 product is.
__device__ __forceinline__ float add_low(float high, float low) {
    return fabsf(high) < INFINITY ? fmaf(low, 1.f / LO_SCALE, high) : high;
}
// v 2^a 2^b for the scales of a row and a column.  Their product is formed first where it is a normal number - v times one of them alone
// may overflow although the result does not; where it is not, both have the same sign of exponent and the order does not matter.
__device__ __forceinline__ float unscale(float v, float a, float b) {
    const float t = a * b;
    return t >= 1.17549435e-38f && t < INFINITY ? v * t : v * a * b;
}

struct Item {
    int n_tile, m_tile, split;
};
// Tile order: passes over all column tiles with `m_group` row tiles each, so that concurrently running tiles share weights and
// activations in L2; the K splits of a tile come one after the other.
__device__ __forceinline__ Item item_at(int w, const Params& p) {
    Item it;
    it.split = w % p.ksplit;
    const int t = w / p.ksplit;
    const int per_pass = p.m_group * p.n_tiles;
    const int pass = t / per_pass, r = t - pass * per_pass;
    const int m_first = pass * p.m_group;
    const int rows = min(p.m_group, p.m_tiles - m_first);
    it.n_tile = r / rows;
    it.m_tile = m_first + r - it.n_tile * rows;
    return it;
}

// Pairs keep an element of a row or column to 2^-50 of its largest at worst: of the lossy ones, lx in the row and lw in the column, each moves
// a sum by less than 2^-36 2^15 sx sw (largest values are below 2^15 sx, 2^15 sw).  That is 2^-21 of the sum where it is lx + lw of sx sw or more,
// which ordinary sums are (they measure in the tens of millions).  The smallest sum of a thread's tile is kept, chunk by chunk, as the sums come out
// of TMEM; where a tile has a marked row or column and a sum below the line - a column of a table whose largest entry no row asks for, a row
// whose large values meet zeros - such sums are formed again here from the fp32 operands.  One warp, columns n of its lanes, rows m_base ..
// m_base + rows; behind all tiles, so that nothing waits for it.  (Few registers: what it needs is added to what the product's kernel needs.  A
// look at every sum inside the epilogue cost each product 0.6 us, by its mere size.)  64 rows whose every row is marked (SwiGLU of two
// equal operands) x [8192, 2048]: 20.0 us, 19.6 with ordinary rows; [4096,4096] x [4096,4096] with nearly every sum below the line: 31 ms, 0.35.
__device__ __noinline__ void repair(const Params& p, int rows, int split, int64_t m_base, int64_t n) {
    constexpr int R = 4;
    const int lane = threadIdx.x & 31;
    const int kb0 = split * p.k_per_split, nk = min(p.k_per_split, p.k_blocks - kb0);
    const int k0 = kb0 * BK, k1 = static_cast<int>(min(p.K, static_cast<int64_t>(k0) + nk * BK));
    const int c_first = p.x_scale_pitch ? kb0 / p.chunk_blocks : 0, c_last = p.x_scale_pitch ? (kb0 + nk - 1) / p.chunk_blocks : 0;
    const bool in = n < p.N;
    const float ws = in ? p.w_scale[n] : 1.f;
    const float lw = in && ws < 0.f ? fminf(p.w_scale[p.w_count + n], static_cast<float>(k1 - k0)) : 0.f;
    float* out = static_cast<float*>(p.out) + (p.ksplit > 1 ? static_cast<int64_t>(split) * p.M * p.N : 0) + n;
    const float* w = nullptr;  // column n of W in fp32, ldw apart
    int64_t ldw = 0;
    if (in) {
        const int64_t c = n + p.w_col0;
        int j = 0;
        while (j + 1 < p.w_src.count && c >= p.w_src.col0[j + 1]) j++;
        w = p.w_src.w[j] + c - p.w_src.col0[j];
        ldw = p.w_src.n[j];
    }
    auto chunk_at = [&](int k) { return p.x_scale_pitch ? k / BK / p.chunk_blocks * p.x_scale_pitch : 0; };
    auto x_at = [&](int64_t m, int k, int64_t chunk) {
        const float s = p.x_scale[chunk + m];
        if (p.x_full_all || s < 0.f) return p.x_full[m * p.x_full_ld + k];
        const __half* h = static_cast<const __half*>(p.x_pairs) + m * p.x_k_pad + k;
        return fmaf(__half2float(h[p.x_low]), 1.f / LO_SCALE, __half2float(h[0])) * s;
    };
    rows = static_cast<int>(min(static_cast<int64_t>(rows), p.M - m_base));
    uint64_t which = 0;  // rows to look at: the marked ones, or all of them where the column of a lane is marked
    const bool any_col = __any_sync(0xffffffffu, lw > 0.f);
    for (int h = 0; h < 64; h += 32) {
        bool marked = false;
        if (h + lane < rows)
            for (int c = c_first; c <= c_last; c++) marked = marked || any_col || p.x_scale[c * p.x_scale_pitch + m_base + h + lane] < 0.f;
        which |= static_cast<uint64_t>(__ballot_sync(0xffffffffu, marked)) << h;
    }
#pragma unroll 1
    for (int j0 = 0; j0 < rows; j0 += R) {
        if ((which >> j0 & 15) == 0) continue;
        float v[R], most[R], lx[R];
#pragma unroll
        for (int j = 0; j < R; j++) {
            most[j] = lx[j] = 0.f;
            v[j] = in && j0 + j < rows ? out[(m_base + j0 + j) * p.ldc] : 0.f;
        }
#pragma unroll 1
        for (int c = c_first; c <= c_last; c++) {
#pragma unroll
            for (int j = 0; j < R; j++) {
                const int64_t at = c * p.x_scale_pitch + m_base + min(j0 + j, rows - 1);
                const float s = p.x_scale[at];
                most[j] = fmaxf(most[j], fabsf(s));
                if (s < 0.f) lx[j] -= s * fminf(p.x_scale[p.x_count + at], static_cast<float>(k1 - k0));
            }
        }
        uint32_t lanes[R];
        int total = 0;
#pragma unroll
        for (int j = 0; j < R; j++) {
            lanes[j] = __ballot_sync(0xffffffffu, in && j0 + j < rows && fabsf(v[j]) < (lx[j] + lw * most[j]) * fabsf(ws));
            total += __popc(lanes[j]);
        }
        if (total == 0) continue;
        if (total <= 12) {  // a sum at a time, the lanes along k
#pragma unroll 1
            for (int j = 0; j < R; j++) {
                const int64_t m = m_base + j0 + j;
                for (uint32_t left = j == 0 ? lanes[0] : j == 1 ? lanes[1] : j == 2 ? lanes[2] : lanes[3]; left; left &= left - 1) {
                    const int l = __ffs(left) - 1;
                    const float* wl = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<uint64_t>(w), l));
                    const int64_t ld = __shfl_sync(0xffffffffu, ldw, l);
                    float sum = 0.f;
#pragma unroll 4
                    for (int k = k0 + lane; k < k1; k += 32) sum = fmaf(x_at(m, k, chunk_at(k)), wl[k * ld], sum);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == l) out[m * p.ldc] = sum;
                }
            }
            continue;
        }
        // a column per lane, four rows
        float sum[R] = {0.f, 0.f, 0.f, 0.f};
        int k = k0;
        if (p.x_full_all) {
            const float* x = p.x_full + (m_base + j0) * p.x_full_ld;
            const int64_t last = p.M - 1 - (m_base + j0);
#pragma unroll 1
            for (; k + 4 <= k1; k += 4) {
                float wv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) wv[i] = in ? w[(k + i) * ldw] : 0.f;
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const float* row = x + min(static_cast<int64_t>(j), last) * p.x_full_ld + k;
#pragma unroll
                    for (int i = 0; i < 4; i++) sum[j] = fmaf(row[i], wv[i], sum[j]);
                }
            }
        }
#pragma unroll 1
        for (; k < k1; k++) {
            const float wv = in ? w[k * ldw] : 0.f;
#pragma unroll
            for (int j = 0; j < R; j++)
                if (lanes[j]) sum[j] = fmaf(x_at(m_base + j0 + j, k, chunk_at(k)), wv, sum[j]);
        }
#pragma unroll
        for (int j = 0; j < R; j++)
            if (lanes[j] >> lane & 1) out[(m_base + j0 + j) * p.ldc] = sum[j];
    }
}

template <int CG, bool SPLIT, int MT, int ST, bool OUT16>
__global__ void __launch_bounds__(Layout<CG, SPLIT, MT, ST>::REGS_FOR, 1) gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                                                     const __grid_constant__ Params p) {
    using L = Layout<CG, SPLIT, MT, ST>;
    dep_trigger();
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + L::BAR_OFFSET;
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (ST + s); };
    auto acc_full = [&](int b) { return bars + 8u * (2 * ST + b); };
    auto acc_empty = [&](int b) { return bars + 8u * (2 * ST + L::NBUF + b); };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(base_ptr + L::BAR_OFFSET + 8 * L::N_BARS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + L::BAR_OFFSET + 8 * L::N_BARS + 8);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = CG == 2 ? cluster_ctarank() : 0;
    const int first = CG == 2 ? blockIdx.x >> 1 : blockIdx.x, stride = CG == 2 ? gridDim.x >> 1 : gridDim.x;
    const int items = p.n_tiles * p.m_tiles * p.ksplit;

    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < L::NBUF; b++) {
            mbar_init(acc_full(b), 1);
            mbar_init(acc_empty(b), CG * L::EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if constexpr (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(L::TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(L::TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    if constexpr (CG == 2) cluster_sync_all();  // the pair's barriers exist and both have their TMEM
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ---------------- loads ----------------
        if (lane == 0) {
            const uint32_t pair_bar = CG == 2 ? mapa_shared(bars, 0) : bars;  // the pair's full barriers live in its first CTA
            bool waited = false;
            if (!p.w_static) {
                dep_wait();
                waited = true;
            }
            auto load_w = [&](int s, int n_tile, int kb) {
                const uint32_t dst = base + s * L::STAGE, bar = pair_bar + 8u * s;
                const int nb = n_tile * CG + static_cast<int>(rank);  // block of 128 columns
                if constexpr (SPLIT) {  // packed: the high and the low tile of a block lie behind one another
                    load_2d<CG>(dst, &tmW, 0, nb * p.w_rows_per_tile + kb * 256, bar);
                } else {
                    load_2d<CG>(dst, &tmW, nb * BN, kb * BK, bar);
                    load_2d<CG>(dst + 8192, &tmW, nb * BN + 64, kb * BK, bar);
                }
            };
            auto load_x = [&](int s, int m_tile, int kb) {
                const uint32_t dst = base + s * L::STAGE + L::W_BYTES, bar = pair_bar + 8u * s;
                const int row = m_tile * MT + static_cast<int>(rank) * L::XR;
                load_2d<CG>(dst, &tmX, kb * BK, row, bar);
                if constexpr (SPLIT) load_2d<CG>(dst + L::X_TILE, &tmX, kb * BK, row + p.x_lo_row, bar);
            };
            // The weights of the first stages do not depend on the kernel before this one: they are requested while it still
            // runs (this grid may have been scheduled early), the activations behind its end.
            int early = 0;
            if (!waited && first < items) {
                const Item it = item_at(first, p);
                const int kb0 = it.split * p.k_per_split, nk = min(p.k_per_split, p.k_blocks - kb0);
                early = min(ST, nk);
                for (int s = 0; s < early; s++) {
                    if (rank == 0) mbar_expect_tx(full(s), CG * L::STAGE);
                    load_w(s, it.n_tile, kb0 + s);
                }
                dep_wait();
                for (int s = 0; s < early; s++) load_x(s, it.m_tile, kb0 + s);
            } else if (!waited) {
                dep_wait();
            }
            int s = 0, done = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int w = first; w < items && ok; w += stride) {
                const Item it = item_at(w, p);
                const int kb0 = it.split * p.k_per_split, nk = min(p.k_per_split, p.k_blocks - kb0);
                for (int kb = 0; kb < nk && ok; kb++) {
                    if (done >= early) {
                        if (done >= ST) ok = mbar_wait(empty(s), phase ^ 1, abort_flag, p.status);
                        if (!ok) break;
                        if (rank == 0) mbar_expect_tx(full(s), CG * L::STAGE);
                        load_w(s, it.n_tile, kb0 + kb);
                        load_x(s, it.m_tile, kb0 + kb);
                    }
                    done++;
                    if (++s == ST) {
                        s = 0;
                        phase ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMAs: one thread of the pair's first CTA ----------------
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = (1u << 4) | (1u << 15) | ((MT >> 3) << 17) | ((CG * BN >> 4) << 24);  // f16 x f16 -> f32, weights n-major
            constexpr uint32_t idesc_wide = (1u << 4) | (1u << 15) | (((2 * MT) >> 3) << 17) | ((CG * BN >> 4) << 24);
            const uint64_t w_desc0 = smem_desc_n128(base), x_desc0 = smem_desc_k128(base + L::W_BYTES);
            int s = 0, buf = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int w = first; w < items && ok; w += stride) {
                const Item it = item_at(w, p);
                const int kb0 = it.split * p.k_per_split, nk = min(p.k_per_split, p.k_blocks - kb0);
                for (int kb = 0; kb < nk && ok; kb++) {
                    const int in_chunk = (kb0 + kb) % p.chunk_blocks;
                    const bool fresh = kb == 0 || in_chunk == 0;
                    if (fresh) {
                        ok = mbar_wait(acc_empty(buf), acc_phase ^ 1, abort_flag, p.status);  // its first use passes at once
                        if (!ok) break;
                    }
                    ok = mbar_wait(full(s), phase, abort_flag, p.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t d = tmem + buf * L::D_COLS;
                    const uint64_t w_hi = w_desc0 + ((s * L::STAGE) >> 4), x_hi = x_desc0 + ((s * L::STAGE) >> 4);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++) {
                        const uint32_t acc = (fresh && kk == 0) ? 0u : 1u;
                        const uint64_t wh = w_hi + kk * 128, xh = x_hi + kk * 2;  // 16 k: 2 KB of the weight tile, 32 bytes inside the activation rows
                        if constexpr (!SPLIT) {
                            mma_f16<CG>(d, wh, xh, idesc, acc);
                        } else {
                            // high x high in columns [0, MT), high x low and low x high in [MT, 2 MT): the small products stay out of the
                            // large sums.  low x low (below 2^-22 of the product) is dropped.
                            const uint64_t wl = wh + (W_TILE >> 4), xl = xh + (L::X_TILE >> 4);
                            if constexpr (CG == 1) {  // the low activation tile follows the high one: one MMA of twice the width
                                mma_f16<CG>(d, wh, xh, idesc_wide, acc);
                            } else {
                                mma_f16<CG>(d, wh, xh, idesc, acc);
                                mma_f16<CG>(d + MT, wh, xl, idesc, acc);
                            }
                            mma_f16<CG>(d + MT, wl, xh, idesc, 1u);
                        }
                    }
                    commit<CG>(empty(s));
                    if (++s == ST) {
                        s = 0;
                        phase ^= 1;
                    }
                    if (kb + 1 == nk || in_chunk + 1 == p.chunk_blocks) {
                        commit<CG>(acc_full(buf));
                        if (++buf == L::NBUF) {
                            buf = 0;
                            acc_phase ^= 1;
                        }
                    }
                }
            }
        }
    } else {
        // ---------------- epilogue ----------------
        // Several warps per group of 32 TMEM lanes (= columns of the output), each with its part of the tile's rows.  A chunk's sums move from
        // TMEM to registers (scaled and added up there), the accumulator goes back to the MMA thread, and the stores follow under
        // the next tile's MMAs.
        constexpr int HM = MT / (L::EPI_WARPS / 4), STEP = HM < 16 ? HM : 16;
        constexpr bool ONE_CHUNK = MT > 128;  // tall tiles take one scale per row
        const int sub = warp & 3, part = (warp - 2) >> 2;
        const uint32_t lane_field = static_cast<uint32_t>(sub * 32) << 16;
        const uint32_t pair_empty = CG == 2 ? mapa_shared(acc_empty(0), 0) : acc_empty(0);
        dep_wait();  // scales and outputs may belong to kernels before this one
        int buf = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        int again_at = -1;  // tile with sums that have to be formed again (repair), -2: several
        for (int w = first; w < items && ok; w += stride) {
            const Item it = item_at(w, p);
            const int kb0 = it.split * p.k_per_split, nk = min(p.k_per_split, p.k_blocks - kb0);
            const int64_t n = (static_cast<int64_t>(it.n_tile) * CG + rank) * BN + sub * 32 + lane;
            const bool in = n < p.N;
            float ws = 0.f;
            float low = INFINITY;       // smallest sum over a chunk
            bool col_marked = false, row_marked = false;  // this column; one of the tile's rows that this lane has the scale of
            if constexpr (SPLIT) {
                const float w_scale = in ? __ldg(p.w_scale + n) : 0.f;
                col_marked = w_scale < 0.f;
                if constexpr (!ONE_CHUNK) ws = fabsf(w_scale);
            }
            const int64_t m_base = static_cast<int64_t>(it.m_tile) * MT + part * HM;
            const int valid = static_cast<int>(min(static_cast<int64_t>(HM), p.M - m_base));  // rows of this warp (what lies behind them is no data)
            float acc[HM];
            float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
            auto row_scale = [&](int j) {
                return __shfl_sync(0xffffffffu, (j & 3) == 0 ? s4.x : (j & 3) == 1 ? s4.y : (j & 3) == 2 ? s4.z : s4.w, j >> 2);
            };
            const int c_first = kb0 / p.chunk_blocks, c_last = (kb0 + nk - 1) / p.chunk_blocks;
            for (int c = c_first; c <= c_last && ok; c++) {
                // the scales of this warp's rows, four per lane, handed round by shuffles when they are needed
                if constexpr (SPLIT) {
                    if (4 * lane < HM) {
                        s4 = __ldg(reinterpret_cast<const float4*>(p.x_scale + c * p.x_scale_pitch + m_base) + lane);
                        const int left = valid - 4 * lane;
                        if (left < 4) s4 = make_float4(left > 0 ? s4.x : 1.f, left > 1 ? s4.y : 1.f, left > 2 ? s4.z : 1.f, 1.f);
                        row_marked = row_marked || fminf(fminf(s4.x, s4.y), fminf(s4.z, s4.w)) < 0.f;
                    }
                }
                ok = __all_sync(0xffffffffu, mbar_wait(acc_full(buf), acc_phase, abort_flag, p.status));  // (one lane's limit may run out before another's)
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + lane_field + buf * L::D_COLS + part * HM;
                if constexpr (!SPLIT || ONE_CHUNK) {
#pragma unroll
                    for (int j0 = 0; j0 < HM; j0 += STEP) tmem_ld<STEP>(d + j0, reinterpret_cast<uint32_t*>(acc) + j0);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if constexpr (SPLIT) {
#pragma unroll
                        for (int j0 = 0; j0 < HM; j0 += STEP) {
                            uint32_t q[STEP];
                            tmem_ld<STEP>(d + MT + j0, q);
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                            for (int j = 0; j < STEP; j++) {
                                acc[j0 + j] = add_low(acc[j0 + j], __uint_as_float(q[j]));
                                if (j0 + j < valid) low = fminf(low, fabsf(acc[j0 + j]));
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int j0 = 0; j0 < HM; j0 += STEP) {
                        uint32_t r[STEP], q[STEP];
                        tmem_ld<STEP>(d + j0, r);
                        tmem_ld<STEP>(d + MT + j0, q);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < STEP; j++) {
                            float v = add_low(__uint_as_float(r[j]), __uint_as_float(q[j]));
                            if (j0 + j < valid) low = fminf(low, fabsf(v));
                            v = unscale(v, fabsf(row_scale(j0 + j)), ws);
                            acc[j0 + j] = c == c_first ? v : acc[j0 + j] + v;
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (CG == 2) arrive_cluster(pair_empty + 8u * buf);
                    else mbar_arrive(acc_empty(buf));
                }
                if (++buf == L::NBUF) {
                    buf = 0;
                    acc_phase ^= 1;
                }
            }
            if (!ok) break;
            if constexpr (SPLIT && ONE_CHUNK) ws = in ? fabsf(__ldg(p.w_scale + n)) : 0.f;
            if constexpr (SPLIT) {
                if (__any_sync(0xffffffffu, col_marked || row_marked)) {
                    const float all = static_cast<float>(BK * min(p.chunk_blocks, nk));
                    float line = c_first < c_last ? all : 0.f;
                    if (row_marked && c_first == c_last) {
                        const float* count = p.x_scale + p.x_count + c_first * p.x_scale_pitch + m_base + 4 * lane;
                        line = fmaxf(fmaxf(s4.x < 0.f ? count[0] : 0.f, s4.y < 0.f ? count[1] : 0.f), fmaxf(s4.z < 0.f ? count[2] : 0.f, s4.w < 0.f ? count[3] : 0.f));
                        line = fminf(fmaxf(line, 1.f), all);
                    }
                    line = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(line)));
                    if (col_marked) line += fminf(p.w_scale[p.w_count + n], all);
                    if (__any_sync(0xffffffffu, in && low < line)) again_at = again_at == -1 ? w : -2;
                }
            }
            using Out = typename std::conditional<OUT16, __half, float>::type;
            Out* o = static_cast<Out*>(p.out) + (p.ksplit > 1 ? static_cast<int64_t>(it.split) * p.M * p.N : 0) + m_base * p.ldc + n;
            const int64_t rows = in ? p.M - m_base : 0;
#pragma unroll
            for (int j = 0; j < HM; j++) {
                float v = acc[j];
                if constexpr (SPLIT && ONE_CHUNK) v = unscale(v, fabsf(row_scale(j)), ws);
                if (j < rows) {
                    if constexpr (OUT16) *o = __float2half_rn(v);
                    else *o = v;
                }
                o += p.ldc;
                asm volatile("" : "+l"(o)::"memory");  // one row after the other: addresses and scales of all 128 rows would not fit in registers beside the sums
            }
        }
        if constexpr (SPLIT)
            if (ok && again_at != -1) {
                for (int w = again_at >= 0 ? again_at : first; w < items; w = again_at >= 0 ? items : w + stride) {
                    const Item it = item_at(w, p);
                    repair(p, HM, it.split, static_cast<int64_t>(it.m_tile) * MT + part * HM, (static_cast<int64_t>(it.n_tile) * CG + rank) * BN + sub * 32 + lane);
                }
            }
    }
    tc_fence_before();
    if constexpr (CG == 2) cluster_sync_all();  // no CTA of the pair leaves while the other may still signal its barriers or read its tiles
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if constexpr (CG == 1)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
    }
}

}  // namespace umma
}  // namespace rmlk
