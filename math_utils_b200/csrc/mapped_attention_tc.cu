// Prompt steps of the attention with score maps (mapped_attention.cu says what it computes) on the 5th-generation tensor
// cores: bfloat16, a block a tile of up to 128 consecutive tokens of one sequence and one head, both products of a cache
// page of 64 positions as tcgen05.mma with their accumulators in tensor memory.
//   S = Q K^T   queries [128][dim] and a page's keys [64][dim] by TMA, K-major, 64 columns a box;
//   O = P V     a page's values lie position-major in the cache row, so they are the right operand MN-major ([64 positions]
//               [64 columns] a box, 128-byte swizzle); P is written by the softmax threads as two bfloat16 terms (the
//               rounded weight and what the rounding left: some 16 bits of mantissa), two products a page.
// Two streams of softmax, four warps each, a thread a query row: with two score maps a stream a map, with one the streams
// take the pages in turns; each has a score buffer, a pair of P tiles and an output accumulator in tensor memory.  A row's
// reference for exp2 is a running maximum that moves only when a page exceeds it by more than 8 (weights stay below 2^8, sums
// and outputs are float32), so the accumulator is rescaled rarely: by the row's own warp, when the product before is
// complete.  At the end the first stream's threads read both accumulators and join them (the maps' difference, or the two
// halves of the pages under a common maximum), with the options of mapped_attention.cu; `head_sink` (one score per head, not
// scaled) is one more key without a value whose score is learned.
// Roles: warp 0 loads queries and keys, warp 3 values, warp 1 owns tensor memory and issues S, warp 2 issues P V.  Waits are
// bounded; one that runs out sets *status (5 loads, 6 products, 7 softmax) and the block leaves without storing.
//
// Sizes: pages of 64; maps * dim a multiple of 16 up to 256, vdim a multiple of 16 up to 128, rows in steps of 8 entries.
// What bounds it: the softmax's chain per page and stream (64 columns a thread); the products take a fraction of it.
// Measured (B200, 2 x 1,024 tokens, 8 heads): two maps of 64, values of 128, window 512: 91 -> 33 us beside the mma.sync
// kernel (64 queries a block, four warps that multiply and exponentiate in turn); the layer around it 136 -> 79 us.  Latent
// attention's prompts over expanded rows (2,048 tokens of three sequences, 16 heads of 128 + 64, values of 128): 41 us, and
// 20 for the product that expands them, where the kernel in latent space took 295; the layer 443 -> 147 us.
#include "tcgen05.cuh"

#include <math.h>

namespace mu {

constexpr int MT_Q = 128, MT_K = 64, MT_THREADS = 384, MT_MAX_STAGES = 4;
constexpr int MT_BOX = 64 * 64 * 2;                    // bytes of a box of 64 rows x 64 columns

struct MtBars {
    uint64_t q_full, k_full[MT_MAX_STAGES], k_empty[MT_MAX_STAGES], v_full[MT_MAX_STAGES], v_empty[MT_MAX_STAGES];
    uint64_t s_full[2], s_free[2], p_full[2], pv_done[2], x_full;
    float hand_ml[MT_Q][2];                            // the second stream's references and sums
    uint32_t tmem_base;
    int failed;
};

struct MtArgs {
    const int *block_table, *tok_pos, *tok_seq, *tiles;
    int max_pages, n_heads, n_kv_heads, maps, dim, vdim, window, chunk, keep, stages, unit_rms, sink, gate_each;
    int key_tiles, val_boxes, val_at;                  // boxes of keys and of values a page; column of kv head 0's values
    int val_step;                                      // columns from one kv head's values to the next one's
    int key_step, key_split, split_at;                 // columns between kv heads' keys; boxes from key_split on lie at split_at
    float scale, lambda, out_scale, eps, softcap;
    const float *head_scale, *slopes, *head_sink;
    const __nv_bfloat16* gate;
    long long ldg, ldo;
    __nv_bfloat16* out;
    int* status;
    const __nv_bfloat16 *q, *rows;                     // what the maps stand for (mt_row_alone)
    long long ldq;
    int row_width;
};

__device__ __forceinline__ float mt_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Right operand, MN-major: rows (k) of 64 columns in 128 swizzled bytes, groups of 8 rows 1024 bytes apart, the next 64
// columns one box further.
__device__ __forceinline__ uint64_t mt_desc_mn(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(MT_BOX >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void mt_tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}

// What a row's two accumulators are multiplied by, out = w0 O0 + w1 O1, from their references (in units of log2) and sums: the
// maps' difference, or (one map) both streams under a common maximum; with a sink's share in the sums.
__device__ __forceinline__ float2 mt_join(const MtArgs& a, int h, float ref0, float sum0, float ref1, float sum1) {
    constexpr float LOG2E = 1.4426950408889634f;
    const bool sinks = a.sink || a.head_sink;
    const float sink = a.head_sink ? a.head_sink[h] * LOG2E : a.sink ? 0.0f : -INFINITY;
    float2 w;
    if (a.maps == 2) {
        const float t0 = fmaxf(ref0, sink), t1 = fmaxf(ref1, sink);
        const float f0 = ref0 == -INFINITY ? 0.0f : mt_exp2(ref0 - t0), f1 = ref1 == -INFINITY ? 0.0f : mt_exp2(ref1 - t1);
        const float l0 = sum0 * f0 + (sinks ? mt_exp2(sink - t0) : 0.0f), l1 = sum1 * f1 + (sinks ? mt_exp2(sink - t1) : 0.0f);
        w.x = l0 > 0.0f ? f0 / l0 : 0.0f;
        w.y = l1 > 0.0f ? -a.lambda * (f1 / l1) : 0.0f;
    } else {
        const float t = fmaxf(fmaxf(ref0, ref1), sink);
        const float f0 = ref0 == -INFINITY ? 0.0f : mt_exp2(ref0 - t), f1 = ref1 == -INFINITY ? 0.0f : mt_exp2(ref1 - t);
        const float l = sum0 * f0 + sum1 * f1 + (sinks ? mt_exp2(sink - t) : 0.0f);
        w.x = l > 0.0f ? f0 / l : 0.0f;
        w.y = l > 0.0f ? f1 / l : 0.0f;
    }
    return w;
}

// One query's result over exactly the keys that it sees, by a warp: for rows that came out infinite or NaN.  A weight of
// zero does not keep an infinite or NaN value out of a product, and a tile's rows meet all pages of the tile: those with later
// tokens, and what lies in the last page behind the sequence's end.  Finite rows pay one multiply-add a pair of values for the check.
// A row whose scores hold a NaN is NaN throughout and stops there.
// (Everything is worked out anew from the tile and the row, so that nothing is kept in registers for it.)
__device__ __noinline__ void mt_row_alone(const MtArgs& a, int row) {
    constexpr float LOG2E = 1.4426950408889634f;
    const int lane = threadIdx.x & 31, kw = a.maps * a.dim;
    const int tile = blockIdx.x / a.n_heads, h = blockIdx.x % a.n_heads, g = h / (a.n_heads / a.n_kv_heads);
    const int flat0 = a.tiles[2 * tile], flat = flat0 + row, pos0 = a.tok_pos[flat0], pos = pos0 + row;
    const int last = (pos0 + min(a.tiles[2 * tile + 1], MT_Q) - 1) / MT_K;
    const int page_lo = (a.chunk > 0 ? pos0 - pos0 % a.chunk : a.window > 0 ? max(0, pos0 - a.window + 1) : 0) / MT_K;
    const int kept_pages = min((a.keep + MT_K - 1) / MT_K, page_lo), n_pages = kept_pages + last - page_lo + 1;
    const int* pages = a.block_table + (long long)a.tok_seq[flat0] * a.max_pages;
    const int lo = a.chunk > 0 ? pos - pos % a.chunk : a.window > 0 ? pos - a.window + 1 : 0;
    const float scale = a.head_scale ? a.scale * a.head_scale[h] : a.scale;
    const float inv_cap = a.softcap > 0.0f ? 1.0f / a.softcap : 0.0f, slope = a.slopes ? a.slopes[h] * LOG2E : 0.0f;
    float acc[2][4] = {}, ref[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};      // columns lane + 32 c
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (m == a.maps) break;
        const __nv_bfloat16* q = a.q + (long long)flat * a.ldq + (long long)h * kw + m * a.dim;
        for (int i = 0; i < 2 * n_pages; ++i) {                                         // 32 keys at a time
            const int page = i / 2 < kept_pages ? i / 2 : page_lo + i / 2 - kept_pages, key = page * MT_K + (i & 1) * 32 + lane;
            const bool seen = key <= pos && (key >= lo || key < a.keep);
            const unsigned some = __ballot_sync(0xffffffffu, seen);
            if (!some) continue;
            const __nv_bfloat16* rows = a.rows + ((long long)pages[page] * MT_K + (i & 1) * 32) * a.row_width;
            float x = -INFINITY;
            if (seen) {
                const __nv_bfloat16* row = rows + (long long)lane * a.row_width;
                x = 0.0f;
                for (int e = 0; e < a.dim; e += 2) {
                    const int col = m * a.dim + e, far = col - 64 * a.key_split;
                    const float2 k = __bfloat1622float2(
                        *reinterpret_cast<const __nv_bfloat162*>(row + (far < 0 ? g * a.key_step + col : a.split_at + far)));
                    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(q + e));
                    x = fmaf(k.y, y.y, fmaf(k.x, y.x, x));
                }
                x *= scale;
                if (a.softcap > 0.0f) x = softcap_fast(x, a.softcap, inv_cap);
                x = x * LOG2E - slope * (float)(pos - key);
            }
            const float top = fmaxf(ref[m], warp_max(x)), from = top == -INFINITY ? 0.0f : top, f = mt_exp2(ref[m] - from);
            const float p = seen ? mt_exp2(x - from) : 0.0f;
            ref[m] = top;
            sum[m] = sum[m] * f + warp_sum(p);
            if (isnan(sum[m])) {
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[m][c] = NAN;
                break;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[m][c] *= f;
            for (int j = 0; j < 32; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j);
                if (!(some >> j & 1u)) continue;
                const __nv_bfloat16* value = rows + (long long)j * a.row_width + a.val_at + g * a.val_step;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (lane + 32 * c < a.vdim) acc[m][c] = fmaf(pj, __bfloat162float(value[lane + 32 * c]), acc[m][c]);
            }
        }
    }
    const float2 w = mt_join(a, h, ref[0], sum[0], ref[1], sum[1]);
    float v[4], sq = 0.0f, times = a.out_scale;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        v[c] = acc[0][c] * w.x;
        if (a.maps == 2) v[c] += acc[1][c] * w.y;
        if (lane + 32 * c < a.vdim) sq = fmaf(v[c], v[c], sq);
    }
    if (a.unit_rms) times *= 1.0f / sqrtf(warp_sum(sq) / (float)a.vdim + a.eps);
    const __nv_bfloat16* gate = a.gate ? a.gate + (long long)flat * a.ldg : nullptr;
    if (gate && !a.gate_each) times *= 1.0f / (1.0f + expf(-__bfloat162float(gate[h])));
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int d = lane + 32 * c;
        if (d >= a.vdim) break;
        float y = v[c] * times;
        if (a.gate_each) y = __fdividef(y, 1.0f + __expf(-__bfloat162float(gate[(long long)h * a.vdim + d])));
        a.out[(long long)flat * a.ldo + (long long)h * a.vdim + d] = __float2bfloat16_rn(y);
    }
}

__global__ void __launch_bounds__(MT_THREADS)
mapped_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_rows,
                           const __grid_constant__ MtArgs a) {
    extern __shared__ unsigned char mt_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)mt_raw + 1023) & ~(uintptr_t)1023);
    const int key_bytes = a.key_tiles * MT_BOX, val_bytes = a.val_boxes * MT_BOX;
    unsigned char* sq = base;                                              // [key_tiles][128 rows x 64 columns]
    unsigned char* sp = sq + a.key_tiles * 2 * MT_BOX;                     // per stream: P rounded, P rest [128 x 64] each
    unsigned char* sk = sp + 4 * 2 * MT_BOX;                               // [stages] pages of keys
    unsigned char* sv = sk + a.stages * key_bytes;                         // [stages] pages of values
    MtBars& sm = *reinterpret_cast<MtBars*>(sv + a.stages * val_bytes);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int tile = blockIdx.x / a.n_heads, h = blockIdx.x % a.n_heads, g = h / (a.n_heads / a.n_kv_heads);
    const int kw = a.maps * a.dim, stages = a.stages;
    constexpr uint32_t TMEM_COLS = 512;              // scores of stream i at 64 i, its output at 128 + 128 i

    if (threadIdx.x == 0) {
        tma_prefetch_map(&map_q);
        tma_prefetch_map(&map_rows);
        mbar_init(&sm.q_full, 1);
        for (int s = 0; s < MT_MAX_STAGES; ++s) {
            mbar_init(&sm.k_full[s], 1); mbar_init(&sm.k_empty[s], 1);
            mbar_init(&sm.v_full[s], 1); mbar_init(&sm.v_empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sm.s_full[i], 1); mbar_init(&sm.s_free[i], 4);
            mbar_init(&sm.p_full[i], 4); mbar_init(&sm.pv_done[i], 1);
        }
        mbar_init(&sm.x_full, 4);
        sm.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&sm.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = sm.tmem_base;
    pdl_trigger();
    pdl_wait();

    const int flat0 = a.tiles[2 * tile], count = min(a.tiles[2 * tile + 1], MT_Q);
    const int pos0 = a.tok_pos[flat0];
    const int* pages = a.block_table + (long long)a.tok_seq[flat0] * a.max_pages;
    const int last_key = pos0 + count - 1;
    const int first_key = a.chunk > 0 ? pos0 - pos0 % a.chunk : a.window > 0 ? max(0, pos0 - a.window + 1) : 0;
    const int page_lo = first_key / MT_K, page_hi = last_key / MT_K;
    // the pages in their order: those before the window that hold kept positions, then the window's
    const int kept_pages = min((a.keep + MT_K - 1) / MT_K, page_lo), n_pages = kept_pages + page_hi - page_lo + 1;
    auto page_at = [&](int i) { return i < kept_pages ? i : page_lo + i - kept_pages; };
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(&sm.q_full, a.key_tiles * 2 * MT_BOX);
            for (int t = 0; t < a.key_tiles; ++t) tma_load_2d(sq + t * 2 * MT_BOX, &map_q, h * kw + 64 * t, flat0, &sm.q_full);
            int issued = 0;
            for (int j = 0; j < n_pages; ++j) {
                const int s = j % stages, row = pages[page_at(j)] * MT_K;
                ok = mbar_wait_poll(&sm.k_empty[s], (uint32_t)(((j / stages) & 1) ^ 1));
                if (!ok) break;
                mbar_expect_tx(&sm.k_full[s], key_bytes);
                for (int t = 0; t < a.key_tiles; ++t)
                    tma_load_2d(sk + s * key_bytes + t * MT_BOX, &map_rows,
                                t < a.key_split ? g * a.key_step + 64 * t : a.split_at + 64 * (t - a.key_split), row, &sm.k_full[s]);
                issued = j + 1;
            }
            if (!ok) {
                atomicExch(a.status, 5);
                sm.failed = 1;
            }
            mbar_wait(&sm.q_full, 0);                        // every copy has landed before the block may go away
            for (int j = issued > stages ? issued - stages : 0; j < issued; ++j)
                mbar_wait(&sm.k_full[j % stages], (uint32_t)((j / stages) & 1));
        }
    } else if (warp == 3) {
        if (lane == 0) {
            int issued = 0;
            for (int j = 0; j < n_pages; ++j) {
                const int s = j % stages, row = pages[page_at(j)] * MT_K;
                ok = mbar_wait_poll(&sm.v_empty[s], (uint32_t)(((j / stages) & 1) ^ 1));
                if (!ok) break;
                mbar_expect_tx(&sm.v_full[s], val_bytes);
                for (int t = 0; t < a.val_boxes; ++t)
                    tma_load_2d(sv + s * val_bytes + t * MT_BOX, &map_rows, a.val_at + g * a.val_step + 64 * t, row, &sm.v_full[s]);
                issued = j + 1;
            }
            if (!ok) {
                atomicExch(a.status, 5);
                sm.failed = 1;
            }
            for (int j = issued > stages ? issued - stages : 0; j < issued; ++j)
                mbar_wait(&sm.v_full[j % stages], (uint32_t)((j / stages) & 1));
        }
    } else if (warp == 1) {
        {
            const bool one = elect_one();
            constexpr uint32_t idesc = idesc_bf16(MT_Q, MT_K);
            const uint64_t q_desc = smem_desc_sw128(smem_u32(sq)), k_desc = smem_desc_sw128(smem_u32(sk));
            ok = mbar_wait_poll(&sm.q_full, 0);
            for (int j = 0; j < n_pages && ok; ++j) {
                const int s = j % stages;
                ok = mbar_wait_poll(&sm.k_full[s], (uint32_t)((j / stages) & 1));
                for (int m = 0; m < a.maps && ok; ++m) {
                    const int i = a.maps == 2 ? m : j & 1, u = a.maps == 2 ? j : j >> 1;       // stream, its u-th page
                    ok = mbar_wait_poll(&sm.s_free[i], (uint32_t)((u & 1) ^ 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (!one) continue;
                    for (int kk = 0; kk < a.dim / 16; ++kk) {
                        const int col = m * a.dim + 16 * kk, t = col >> 6, in = (col & 63) >> 3;      // box, 16-byte piece in its rows
                        umma_bf16(tmem_base + 64 * i, q_desc + (uint64_t)(t * (2 * MT_BOX / 16) + in),
                                  k_desc + (uint64_t)((s * key_bytes + t * MT_BOX) / 16 + in), idesc, kk > 0 ? 1u : 0u);
                    }
                    umma_commit(&sm.s_full[i]);
                }
                if (ok && one) umma_commit(&sm.k_empty[s]);         // the keys are free once these products have read them
            }
            if (!ok && one) {
                atomicExch(a.status, 6);
                sm.failed = 1;
            }
        }
    } else if (warp == 2) {
        {
            const bool one = elect_one();
            const uint32_t idesc = idesc_bf16(MT_Q, a.vdim) | (1u << 16);                     // the right operand is MN-major
            const uint64_t p_desc = smem_desc_sw128(smem_u32(sp)), v_desc = mt_desc_mn(smem_u32(sv));
            for (int j = 0; j < n_pages && ok; ++j) {
                const int s = j % stages;
                ok = mbar_wait_poll(&sm.v_full[s], (uint32_t)((j / stages) & 1));
                for (int m = 0; m < a.maps && ok; ++m) {
                    const int i = a.maps == 2 ? m : j & 1, u = a.maps == 2 ? j : j >> 1;
                    ok = mbar_wait_poll(&sm.p_full[i], (uint32_t)(u & 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (!one) continue;
#pragma unroll
                    for (int term = 0; term < 2; ++term)
#pragma unroll
                        for (int kk = 0; kk < MT_K / 16; ++kk)
                            umma_bf16(tmem_base + 128 + 128 * i, p_desc + (uint64_t)((2 * i + term) * (2 * MT_BOX / 16) + 2 * kk),
                                      v_desc + (uint64_t)((s * val_bytes + kk * 2048) / 16), idesc,
                                      u > 0 || term > 0 || kk > 0 ? 1u : 0u);
                    umma_commit(&sm.pv_done[i]);
                }
                if (ok && one) umma_commit(&sm.v_empty[s]);
            }
            if (!ok && one) {
                atomicExch(a.status, 6);
                sm.failed = 1;
            }
        }
    } else {
        const int quad = warp & 3, stream = (warp - 4) >> 2, row = quad * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint32_t s_col = lane_base + 64 * stream, o_col = lane_base + 128 + 128 * stream;
        constexpr float LOG2E = 1.4426950408889634f;
        const int qpos = pos0 + row;
        const bool real = row < count;
        // the positions the row sees: lo .. hi, and those before `keep`
        const int hi = real ? qpos : -1, lo = a.chunk > 0 ? qpos - qpos % a.chunk : a.window > 0 ? qpos - a.window + 1 : 0;
        const float scale = a.head_scale ? a.scale * a.head_scale[h] : a.scale;
        const float inv_cap = a.softcap > 0.0f ? 1.0f / a.softcap : 0.0f, slope = a.slopes ? a.slopes[h] * LOG2E : 0.0f;
        const float mult = a.softcap > 0.0f ? LOG2E : scale * LOG2E;
        float ref = -INFINITY, sum = 0.0f;                   // in units of log2
        const int n_mine = a.maps == 2 ? n_pages : n_pages > stream ? (n_pages - stream + 1) / 2 : 0;
        for (int u = 0; u < n_mine; ++u) {
            const int key0 = page_at(a.maps == 2 ? u : 2 * u + stream) * MT_K;
            ok = mbar_wait(&sm.s_full[stream], (uint32_t)(u & 1));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t r[2][32];
            tmem_ld_32x32_nowait(s_col, r[0]);
            tmem_ld_32x32_nowait(s_col + 32, r[1]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 32; ++c) asm volatile("" : "+r"(r[0][c]), "+r"(r[1][c]));        // not read before that wait
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.s_free[stream]);
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            const int see_hi = hi - key0, see_lo = lo - key0, see_keep = a.keep - key0;          // seen: c <= hi and (c >= lo or c < keep)
            const bool whole = see_hi >= MT_K - 1 && (see_lo <= 0 || see_keep >= MT_K);
            if (a.softcap > 0.0f) {
#pragma unroll
                for (int c = 0; c < 64; ++c)
                    r[c >> 5][c & 31] = __float_as_uint(softcap_fast(__uint_as_float(r[c >> 5][c & 31]) * scale, a.softcap, inv_cap));
            }
            const float far = slope * (float)(qpos - key0);
#pragma unroll
            for (int c = 0; c < 64; ++c) {
                float x = __uint_as_float(r[c >> 5][c & 31]) * mult;
                if (a.slopes) x -= far - slope * (float)c;
                if (!whole && !(c <= see_hi && (c >= see_lo || c < see_keep))) x = -INFINITY;
                r[c >> 5][c & 31] = __float_as_uint(x);
                top[c & 3] = fmaxf(top[c & 3], x);
            }
            const float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            // the P tiles and the accumulator are this warp's own rows' once the product before is complete
            if (u > 0) {
                ok = mbar_wait(&sm.pv_done[stream], (uint32_t)((u - 1) & 1));
                if (!ok) break;
            }
            const bool grow = mx > ref + 8.0f || (ref == -INFINITY && mx > -INFINITY);
            if (__any_sync(0xffffffffu, grow)) {
                const float next = grow ? mx : ref;
                const float f = grow ? mt_exp2(ref - next) : 1.0f;                               // (0 for a row that had seen nothing)
                ref = next;
                sum *= f;
                if (u > 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int c = 0; c < a.vdim; c += 32) {
                        uint32_t o[32];
                        tmem_ld_32x32(o_col + c, o);
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                        mt_tmem_st_32x32(o_col + c, o);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                }
            }
            const float from = ref == -INFINITY ? 0.0f : ref;
            float sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            unsigned char* p_hi = sp + (2 * stream) * 2 * MT_BOX + row * 128;
            unsigned char* p_lo = p_hi + 2 * MT_BOX;
#pragma unroll
            for (int c = 0; c < 64; c += 8) {
                uint32_t hw[4], lw[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float p0 = mt_exp2(__uint_as_float(r[c >> 5][(c & 31) + 2 * e]) - from);
                    const float p1 = mt_exp2(__uint_as_float(r[c >> 5][(c & 31) + 2 * e + 1]) - from);
                    sums[e] += p0 + p1;
                    const __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
                    const __nv_bfloat162 ll = __floats2bfloat162_rn(p0 - __low2float(hh), p1 - __high2float(hh));
                    hw[e] = *reinterpret_cast<const uint32_t*>(&hh);
                    lw[e] = *reinterpret_cast<const uint32_t*>(&ll);
                }
                const int piece = 16 * ((c >> 3) ^ (row & 7));            // where the swizzle puts a row's 16-byte piece
                *reinterpret_cast<uint4*>(p_hi + piece) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                *reinterpret_cast<uint4*>(p_lo + piece) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
            }
            sum += (sums[0] + sums[1]) + (sums[2] + sums[3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read P through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_full[stream]);
        }
        if (ok && n_mine > 0) ok = mbar_wait(&sm.pv_done[stream], (uint32_t)((n_mine - 1) & 1));
        if (!ok && lane == 0) {
            atomicExch(a.status, 7);
            sm.failed = 1;
        }
        if (stream == 1) {
            sm.hand_ml[row][0] = ref;
            sm.hand_ml[row][1] = sum;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.x_full);
        } else {
            if (ok) ok = mbar_wait(&sm.x_full, 0);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (__all_sync(0xffffffffu, ok && !sm.failed)) {
                const float2 w = mt_join(a, h, ref, sum, sm.hand_ml[row][0], sm.hand_ml[row][1]);
                const float w0 = w.x, w1 = w.y;
                const bool two = a.maps == 2 || n_pages > 1;              // (else the second accumulator was never written)
                auto columns = [&](int c, float (&v)[32]) {
                    uint32_t x[32], y[32];
                    tmem_ld_32x32(o_col + c, x);
                    if (two) tmem_ld_32x32(o_col + 128 + c, y);
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        v[i] = __uint_as_float(x[i]) * w0 + (two ? __uint_as_float(y[i]) * w1 : 0.0f);
                };
                float times = a.out_scale;
                if (a.unit_rms) {
                    float sq = 0.0f;
                    for (int c = 0; c < a.vdim; c += 32) {
                        float v[32];
                        columns(c, v);
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c + i < a.vdim) sq = fmaf(v[i], v[i], sq);
                    }
                    times *= 1.0f / sqrtf(sq / (float)a.vdim + a.eps);
                }
                const __nv_bfloat16* gate = a.gate ? a.gate + (long long)(flat0 + min(row, count - 1)) * a.ldg : nullptr;
                if (gate && !a.gate_each) times *= 1.0f / (1.0f + expf(-__bfloat162float(gate[h])));
                __nv_bfloat16* dst = a.out + (long long)(flat0 + row) * a.ldo + (long long)h * a.vdim;
                const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
                __nv_bfloat162 odd[4] = {zero, zero, zero, zero};          // NaN from the first value that is not finite on
                for (int c = 0; c < a.vdim; c += 32) {
                    float v[32];
                    __syncwarp();
                    columns(c, v);
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        if (!real || c + i >= a.vdim) break;
                        uint32_t word[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            float y0 = v[i + 2 * e] * times, y1 = v[i + 2 * e + 1] * times;
                            if (a.gate_each) {
                                const __nv_bfloat162 z = *reinterpret_cast<const __nv_bfloat162*>(gate + (long long)h * a.vdim + c + i + 2 * e);
                                y0 = __fdividef(y0, 1.0f + __expf(-__low2float(z)));
                                y1 = __fdividef(y1, 1.0f + __expf(-__high2float(z)));
                            }
                            const __nv_bfloat162 b = __floats2bfloat162_rn(y0, y1);
                            odd[e] = __hfma2(b, zero, odd[e]);
                            word[e] = *reinterpret_cast<const uint32_t*>(&b);
                        }
                        *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(word[0], word[1], word[2], word[3]);
                    }
                }
                const float2 some = __bfloat1622float2(__hadd2(__hadd2(odd[0], odd[1]), __hadd2(odd[2], odd[3])));
                for (unsigned todo = __ballot_sync(0xffffffffu, isnan(some.x + some.y)); todo; todo &= todo - 1) {
                    mt_row_alone(a, ((int)threadIdx.x >> 5 & 3) * 32 + __ffs(todo) - 1);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

static size_t mt_smem(int key_tiles, int val_boxes, int stages) {
    return (size_t)MT_BOX * (2 * key_tiles + 8 + stages * (key_tiles + val_boxes)) + sizeof(MtBars) + 1024;
}
constexpr size_t MT_MOST = 227 * 1024;

}  // namespace mu

// Whether the kernel takes these sizes.
MU_EXPORT int mu_mapped_attention_tc_fits(int n_kv_heads, int maps, int dim, int vdim, int page_tokens, int shared) {
    const long long width = (long long)n_kv_heads * (maps * dim + (shared ? 0 : vdim));
    return page_tokens == mu::MT_K && (maps == 1 || maps == 2) && dim > 0 && dim % 16 == 0 && maps * dim <= 256 && vdim > 0 &&
           vdim % 16 == 0 && vdim <= 128 && width % 8 == 0 && width <= 0x3fffffff;
}

// As mu_mapped_attention_mma, for tiles of up to 128 tokens.  n_tokens: rows of q; n_pages: pages of the cache; out rows in
// whole 16-byte pieces; head_sink (may be null; not with sink): a score per head, not scaled, of one more key without a value;
// split_keys k > 0 (a multiple of 64): a row holds the heads' first k key entries, their values, and the dim - k entries that
// all heads' keys end with.
MU_EXPORT int mu_mapped_attention_tc(const void* q, long long ldq, int n_tokens, const void* rows, long long n_pages,
                                     const int* block_table, int max_pages, int page_tokens, const int* tok_pos,
                                     const int* tok_seq, const int* tiles, int n_tiles, int n_heads, int n_kv_heads, int maps,
                                     int dim, int vdim, float scale, int window, float lambda, float out_scale, float eps,
                                     int unit_rms, void* out, long long ldo, int* status, void* stream, const float* head_scale,
                                     int sink, const void* gate, long long ldg, int chunk, const float* slopes, int keep,
                                     float softcap, int gate_each, int shared, const float* head_sink, int split_keys) {
    if (n_tiles <= 0) return MU_OK;
    if (keep < 0 || (gate_each && !gate) || (shared && (maps != 1 || vdim != dim)) || (sink && head_sink)) return MU_ERR_BAD_ARGUMENT;
    if (gate_each && (ldg % 2 || ((uintptr_t)gate & 3))) return MU_ERR_ALIGNMENT;
    if (!q || !rows || !block_table || !tok_pos || !tok_seq || !tiles || !out || !status || n_tokens <= 0 || n_pages <= 0 ||
        n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads || window < 0 || chunk < 0 || ldq < (long long)n_heads * maps * dim)
        return MU_ERR_BAD_ARGUMENT;
    if (!mu_mapped_attention_tc_fits(n_kv_heads, maps, dim, vdim, page_tokens, shared)) return MU_ERR_UNSUPPORTED_SIZE;
    if (((uintptr_t)q & 15) || ((uintptr_t)rows & 15) || ((uintptr_t)out & 15) || ldq % 8 || ldo % 8) return MU_ERR_ALIGNMENT;
    const int kw = maps * dim;
    if (split_keys && (maps != 1 || shared || split_keys % 64 || split_keys <= 0 || split_keys >= kw)) return MU_ERR_BAD_ARGUMENT;
    const int width = split_keys ? n_kv_heads * (split_keys + vdim) + kw - split_keys : n_kv_heads * (kw + (shared ? 0 : vdim));
    const long long items = (long long)n_tiles * n_heads;
    if (n_pages * mu::MT_K > 0x7fffffffll || items > 0x7fffffffll || (long long)n_heads * kw > 0x3fffffff) return MU_ERR_UNSUPPORTED_SIZE;
    CUtensorMap map_q, map_rows;
    if (!mu::tensor_map_bf16(&map_q, q, n_tokens, n_heads * kw, ldq, mu::MT_Q) ||
        !mu::tensor_map_bf16(&map_rows, rows, n_pages * mu::MT_K, width, width, mu::MT_K))
        return MU_ERR_LAUNCH;
    mu::MtArgs a = {};
    a.block_table = block_table, a.tok_pos = tok_pos, a.tok_seq = tok_seq, a.tiles = tiles, a.max_pages = max_pages;
    a.n_heads = n_heads, a.n_kv_heads = n_kv_heads, a.maps = maps, a.dim = dim, a.vdim = vdim, a.window = window, a.chunk = chunk;
    a.keep = keep, a.unit_rms = unit_rms, a.sink = sink, a.gate_each = gate_each, a.scale = scale, a.lambda = lambda;
    a.out_scale = out_scale, a.eps = eps, a.softcap = softcap, a.head_scale = head_scale, a.slopes = slopes, a.head_sink = head_sink;
    a.q = (const __nv_bfloat16*)q, a.ldq = ldq, a.rows = (const __nv_bfloat16*)rows, a.row_width = width;
    a.gate = (const __nv_bfloat16*)gate, a.ldg = ldg, a.ldo = ldo, a.out = (__nv_bfloat16*)out, a.status = status;
    a.key_tiles = (kw + 63) / 64, a.val_boxes = (vdim + 63) / 64;
    a.key_step = kw, a.key_split = a.key_tiles;
    a.val_at = shared ? 0 : n_kv_heads * kw, a.val_step = vdim;
    if (split_keys) {                                  // [keys without their shared part | values | the part all heads share]
        a.key_step = split_keys, a.key_split = split_keys / 64;
        a.val_at = n_kv_heads * split_keys, a.split_at = n_kv_heads * (split_keys + vdim);
    }
    a.stages = mu::MT_MAX_STAGES;
    while (a.stages > 2 && mu::mt_smem(a.key_tiles, a.val_boxes, a.stages) > mu::MT_MOST) --a.stages;
    const size_t smem = mu::mt_smem(a.key_tiles, a.val_boxes, a.stages);
    if (smem > mu::MT_MOST) return MU_ERR_UNSUPPORTED_SIZE;
    const void* kernel = reinterpret_cast<const void*>(mu::mapped_attention_tc_kernel);
    if (!mu::allow_shared(kernel, mu::MT_MOST)) return MU_ERR_LAUNCH;
    mu::prefer_shared_memory(kernel);
    return mu::launch_pdl(mu::mapped_attention_tc_kernel, dim3((unsigned)items), dim3(mu::MT_THREADS), smem, (cudaStream_t)stream, 1,
                          map_q, map_rows, a);
}
