// The experts' products, and products per head, on the 5th-generation tensor cores (bfloat16, float32 accumulation).
//
// mu_moe_gather    the experts' input rows in the order of their slots: xs[slot] = x[pair / top].
// mu_moe_gemm_tc   for every tile of up to 128 slots of one expert: out[slot] = act(W1[e] xs[slot]), or with a second weight
//                  stack silu(W1[e] xs[slot]) * W2[e] xs[slot]; a row weight multiplies the products first.
// mu_heads_gemm_tc out[t, g, :] = W[g] x[t, g, :] for every row t and group (head) g.
//
// One kernel: the persistent product of gemm_tc_kernel.cuh (a loader thread, an issuing thread, eight epilogue warps, a
// ring of TMA stages that runs on across tiles, two accumulators in tensor memory that take turns) over a LIST of tiles
// instead of a grid.  The list is on the device and its length is read there, so nothing is known to the host.  A tile's
// 128 rows of A begin at its first slot; what follows an expert's last slot belongs to the next one (or lies past the
// matrix and is zero), is multiplied along and never stored: a row of the accumulator depends on its own row of A alone.
// The rows are gathered by a launch of their own, which costs what reading and writing them once costs and lets TMA fetch
// whole boxes.  The items' order (tiles_first) keeps an expert's tiles close together, so the weights cross from
// memory once.
//
// What bounds it: with few rows an expert the weights' bytes; with hundreds the operands' way from the L2, 48 KB for every 128 x
// 256 x 64 step, some 11 TB/s, a quarter of the tiles' rows empty.  Measured (B200): 64 experts of 2,048 x 1,408 x 3, 12,288
// pairs, the same number for every expert, both products: mma.sync with 64 rows a block 943 us; tiles of 128 slots 338 (220 + 119),
// tile by tile 297 (190 + 106; the weights' bytes alone take 113 + 56); the gather ~10 us; 48 pairs over those
// experts with two matrices each, the whole feed-forward 136 -> 93 us.  Tiles of 256 slots by pairs of SMs (cta_group::2)
// took 263 us with equal experts, but where routing loads them unequally their emptier tiles cost what the feeding saves
// (the whole feed-forward 447 us against 436).  Per head, 16 heads, 2,048 rows, the launch alone: 512 x 128 36 -> 25 us, 128 x 512 26 -> 9;
// at 300 rows 8.3 -> 8.5 and 14.5 -> 6.0.
#include "gemm_tc_kernel.cuh"

#include <math.h>

namespace mu {

// NB: 128-row boxes of weights a stage; GATED: the two boxes are the same columns of the two stacks.
template <int NB, bool GATED, typename TC>
__global__ void __launch_bounds__(TC_THREADS)
grouped_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w1,
                  const __grid_constant__ CUtensorMap map_w2, const int* __restrict__ tile_info,
                  const int* __restrict__ n_tiles, const int* __restrict__ pair_of, const float* __restrict__ row_weight,
                  int n, int k, TC* __restrict__ out, long long ldo, int act, int* status, int n_rows, int n_groups,
                  int x_group_offset, long long out_group_offset, const __nv_bfloat16* __restrict__ gate, long long ldg, int tile_first) {
    constexpr int BN = 128 * NB, STAGES = NB == 2 ? 4 : 3, KSUB = NB == 2 ? 1 : 2, OUT_COLS = GATED ? 128 : BN;
    typedef TcSmem<BN, STAGES, KSUB> Smem;
    extern __shared__ unsigned char tc_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(((uintptr_t)tc_raw + 1023) & ~(uintptr_t)1023);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    // (a sub-tile that would begin past k is neither fetched nor multiplied: by head there lies the gap after the slice, or the
    // next head's slice, and zeros of the weights do not make a product with an infinity or a NaN zero)
    const int num_kb = (k + KSUB * TC_BK - 1) / (KSUB * TC_BK);
    auto sub_tiles = [&](int kb) { return min(KSUB, (k + TC_BK - 1) / TC_BK - kb * KSUB); };
    constexpr uint32_t SUB_BYTES = (TC_BM + BN) * TC_BK * sizeof(__nv_bfloat16);
    constexpr uint32_t TMEM_COLS = 2 * BN;
    bool ok = true;
    if (threadIdx.x == 0) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_w1);
        if (GATED) tma_prefetch_map(&map_w2);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&sm.acc_full[b], 1); mbar_init(&sm.acc_empty[b], TC_EPI_WARPS); }
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

    const bool by_head = tile_info == nullptr;
    const int tiles = by_head ? (n_rows + TC_BM - 1) / TC_BM : n_tiles[0];
    const int n_blocks = (n + OUT_COLS - 1) / OUT_COLS;
    const int items = tiles * n_blocks * (by_head ? n_groups : 1);
    struct Item { int group, row0, rows, n0; };
    auto item_at = [&](int item) {
        Item w;
        if (by_head) {
            const int tile = item % tiles, rest = item / tiles;
            w.group = rest / n_blocks, w.row0 = tile * TC_BM, w.rows = min(TC_BM, n_rows - w.row0);
            w.n0 = rest % n_blocks * OUT_COLS;
        } else {
            const int* info = tile_info + 3 * (tile_first ? item / n_blocks : item % tiles);
            w.group = info[0], w.row0 = info[1], w.rows = info[2];
            w.n0 = (tile_first ? item % n_blocks : item / tiles) * OUT_COLS;
        }
        return w;
    };

    if (warp == 0) {
        if (lane == 0) {
            long long it = 0, issued = 0;
            Item w = {};
            if ((int)blockIdx.x < items) w = item_at(blockIdx.x);
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
                Item next = {};
                if (item + (int)gridDim.x < items) next = item_at(item + gridDim.x);      // on its way while this tile loads
                const int ax = by_head ? w.group * x_group_offset : 0, wy = w.group * n + w.n0;
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = (int)(it % STAGES);
                    ok = mbar_wait(&sm.empty[s], (uint32_t)(((it / STAGES) & 1) ^ 1));
                    if (!ok) break;
                    const int subs = sub_tiles(kb);
                    mbar_expect_tx(&sm.full[s], subs * SUB_BYTES);
#pragma unroll
                    for (int u = 0; u < KSUB; ++u) {
                        if (u > 0 && u >= subs) break;
                        const int x = (kb * KSUB + u) * TC_BK;
                        tma_load_2d(sm.a[s][u], &map_a, ax + x, w.row0, &sm.full[s]);
                        tma_load_2d(sm.b[s][u], &map_w1, x, wy, &sm.full[s]);
                        if (NB == 2) {
                            if (GATED) tma_load_2d(sm.b[s][u] + 128 * TC_BK, &map_w2, x, wy, &sm.full[s]);
                            else tma_load_2d(sm.b[s][u] + 128 * TC_BK, &map_w1, x, wy + 128, &sm.full[s]);
                        }
                    }
                    issued = it + 1;
                }
                w = next;
            }
            if (!ok) {
                atomicExch(status, 1);
                for (long long j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)      // copies under way land first
                    mbar_wait(&sm.full[j % STAGES], (uint32_t)((j / STAGES) & 1));
            }
        }
    } else if (warp == 1) {
        {
            const bool one = elect_one();
            constexpr uint32_t idesc = idesc_bf16(TC_BM, BN);
            const uint64_t a_desc0 = smem_desc_sw128(smem_u32(sm.a[0][0]));
            const uint64_t b_desc0 = smem_desc_sw128(smem_u32(sm.b[0][0]));
            constexpr uint32_t A_SUB = TC_BM * TC_BK * sizeof(__nv_bfloat16) / 16, B_SUB = BN * TC_BK * sizeof(__nv_bfloat16) / 16;
            long long it = 0;
            int local = 0;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++local) {
                const int buf = local & 1;
                ok = mbar_wait(&sm.acc_empty[buf], (uint32_t)(((local >> 1) & 1) ^ 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = (int)(it % STAGES);
                    ok = mbar_wait(&sm.full[s], (uint32_t)((it / STAGES) & 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t a_stage = a_desc0 + (uint64_t)((uint32_t)s * (KSUB * A_SUB));
                    const uint64_t b_stage = b_desc0 + (uint64_t)((uint32_t)s * (KSUB * B_SUB));
                    const int subs = sub_tiles(kb);
                    if (!one) continue;
#pragma unroll
                    for (int u = 0; u < KSUB; ++u) {
                        if (u > 0 && u >= subs) break;
#pragma unroll
                        for (int kk = 0; kk < TC_BK / 16; ++kk)
                            umma_bf16(tmem_d, a_stage + (uint64_t)(u * A_SUB + 2 * kk), b_stage + (uint64_t)(u * B_SUB + 2 * kk),
                                      idesc, (kb > 0 || u > 0 || kk > 0) ? 1u : 0u);
                    }
                    umma_commit(&sm.empty[s]);
                }
                if (ok && one) umma_commit(&sm.acc_full[buf]);
            }
            if (!ok && one) atomicExch(status, 2);
        }
    } else {
        const int quad = warp & 3, half = (warp - 2) / 4;       // 32 rows and half of the columns a warp, as in gemm_tc
        constexpr int COLS = OUT_COLS / (TC_EPI_WARPS / 4), CHUNKS = COLS / 32;
        float* patch = sm.patch[warp - 2];
        const float no_bias[8] = {};
        const bool vec_ok = sizeof(TC) == 2 && (ldo * sizeof(TC)) % 16 == 0 && ((uintptr_t)out) % 16 == 0 &&
                            (out_group_offset * sizeof(TC)) % 16 == 0;
        int local = 0;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x, ++local) {
            const int buf = local & 1;
            const Item w = item_at(item);
            const int row0 = w.row0 + quad * 32, limit = w.row0 + w.rows, row = min(row0 + lane, limit - 1);
            const float f = row_weight ? row_weight[pair_of ? pair_of[row] : row] : 1.0f;
            TC* dst = out + (by_head ? w.group * out_group_offset : 0);
            const __nv_bfloat16* gate_row = gate ? gate + w.group * out_group_offset + (long long)row * ldg : nullptr;
            ok = mbar_wait(&sm.acc_full[buf], (uint32_t)((local >> 1) & 1));
            if (!ok) {
                if (lane == 0) atomicExch(status, 3);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN + half * COLS);
#pragma unroll
            for (int q = 0; q < CHUNKS; ++q) {
                uint32_t r[32];
                if constexpr (GATED) {
                    uint32_t up[32];
                    tmem_ld_32x32_nowait(acc_addr + 32 * q, r);
                    tmem_ld_32x32(acc_addr + 128 + 32 * q, up);                   // (waits for both)
#pragma unroll
                    for (int i = 0; i < 32; ++i) asm volatile("" : "+r"(r[i]));   // not read before that wait
                    if (q == CHUNKS - 1) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) mbar_arrive(&sm.acc_empty[buf]);
                    }
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float z = __uint_as_float(r[i]) * f;
                        r[i] = __float_as_uint(z / (1.0f + expf(-z)) * (__uint_as_float(up[i]) * f));
                    }
                } else {
                    tmem_ld_32x32(acc_addr + 32 * q, r);
                    if (q == CHUNKS - 1) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) mbar_arrive(&sm.acc_empty[buf]);
                    }
                    if (row_weight) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
                    }
                }
                const int nb = w.n0 + half * COLS + 32 * q;
                if (row0 >= limit || nb >= n) continue;                           // the same for the whole warp
                if (gate_row) {                                                   // out *= sigmoid(gate), in float32
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (nb + i < n)
                            r[i] = __float_as_uint(__uint_as_float(r[i]) / (1.0f + expf(-__bfloat162float(gate_row[nb + i]))));
                }
                const bool packed = vec_ok && nb + 32 <= n;
                if (act == ACT_RELU2)
                    tc_finish_block<ACT_RELU2, TC>(r, patch, lane, nullptr, no_bias, nullptr, dst, limit, n, row0, nb, ldo, 0, packed);
                else
                    tc_finish_block<ACT_NONE, TC>(r, patch, lane, nullptr, no_bias, nullptr, dst, limit, n, row0, nb, ldo, 0, packed);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// The order of the items.  One column block after another for all tiles reads every expert's tiles side by side, and the rows once
// a column block; once these no longer stay in the L2 beside the weights that pass through it they come from memory each time,
// and the items go tile by tile, all its column blocks together (an expert's tiles still follow one another).  64 experts
// of 2,048 x 1,408 x 3, pairs and their rows' megabytes, microseconds of the first product by column blocks and by tiles:
// 1,024 (4) 132 and 131, 4,096 (17) 138 and 131, 6,144 (25) 146 and 136, 12,288 (50) 220 and 191; of two matrices 68 and 70,
// 72 and 76, 82 and 72, 128 and 109.  The line, an eighth of the L2, lies between the two middle ones; seven other shapes (8 to 48
// experts of 768 to 4,096 x 512 to 4,096, rows of 4 to 98 MB) in two forms took 0.99 to 1.19 times less than by column blocks.
constexpr long long GROUPED_ROWS_KEPT = 17000000;
inline bool tiles_first(long long rows, int k) { return rows * k * 2 > GROUPED_ROWS_KEPT; }

template <int NB, bool GATED, typename TC>
static int launch_grouped(const void* x, long long x_rows, int x_cols, long long ldx, const void* w1, const void* w2,
                          long long w_rows, long long ldw, const int* tile_info, const int* n_tiles, const int* pair_of,
                          const float* row_weight, int n, int k, TC* out, long long ldo, int act, int* status, int n_rows,
                          int n_groups, int x_group_offset, long long out_group_offset, const void* gate, long long ldg,
                          long long most_items, cudaStream_t s) {
    constexpr int BN = 128 * NB, STAGES = NB == 2 ? 4 : 3, KSUB = NB == 2 ? 1 : 2;
    CUtensorMap a, b1, b2;
    if (!tensor_map_bf16(&a, x, x_rows, x_cols, ldx, TC_BM) || !tensor_map_bf16(&b1, w1, w_rows, k, ldw, 128))
        return MU_ERR_LAUNCH;
    b2 = b1;
    if (GATED && !tensor_map_bf16(&b2, w2, w_rows, k, ldw, 128)) return MU_ERR_LAUNCH;
    auto kernel = grouped_tc_kernel<NB, GATED, TC>;
    const size_t smem = sizeof(TcSmem<BN, STAGES, KSUB>) + 1024;
    if (!allow_shared(reinterpret_cast<const void*>(kernel), smem)) return MU_ERR_LAUNCH;
    prefer_shared_memory(reinterpret_cast<const void*>(kernel));
    const int sms = sm_count();
    if (sms <= 0) return MU_ERR_LAUNCH;
    const dim3 grid((unsigned)(most_items < sms ? most_items : sms));
    return launch_pdl(kernel, grid, dim3(TC_THREADS), smem, s, 1, a, b1, b2, tile_info, n_tiles, pair_of, row_weight, n, k, out,
                      ldo, act, status, n_rows, n_groups, x_group_offset, out_group_offset, (const __nv_bfloat16*)gate, ldg, (int)tiles_first(x_rows, k));
}

// A warp a pair: its token's row to the pair's slot, sixteen bytes a lane at a time.
__global__ void moe_gather_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ slot_of,
                                  int n_pairs, int top, int pieces, __nv_bfloat16* __restrict__ xs) {
    pdl_trigger();
    pdl_wait();
    const int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= n_pairs) return;
    const int slot = slot_of[p];
    if (slot < 0) return;                                        // an identity expert's pair
    const uint4* src = reinterpret_cast<const uint4*>(x + (long long)(p / top) * ldx);
    uint4* dst = reinterpret_cast<uint4*>(xs) + (long long)slot * pieces;
    for (int i = lane; i < pieces; i += 128) {
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + 32 * j < pieces) v[j] = src[i + 32 * j];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + 32 * j < pieces) dst[i + 32 * j] = v[j];
    }
}

}  // namespace mu

MU_EXPORT int mu_moe_gather(const void* x, long long ldx, const int* slot_of, int n_pairs, int top, int width, void* xs,
                            void* stream) {
    if (n_pairs <= 0) return MU_OK;
    if (!x || !slot_of || !xs || top <= 0 || width <= 0) return MU_ERR_BAD_ARGUMENT;
    if (width % 8 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)xs & 15)) return MU_ERR_ALIGNMENT;
    return mu::launch_pdl(mu::moe_gather_kernel, dim3((n_pairs + 7) / 8), dim3(256), 0, (cudaStream_t)stream, 1,
                          (const __nv_bfloat16*)x, ldx, slot_of, n_pairs, top, width / 8, (__nv_bfloat16*)xs);
}

// xs [xs_rows, k] (rows by slot), w1 / w2 [n_experts, n, k] contiguous, tiles of up to 128 slots; bfloat16, k and ldx
// multiples of 8, bases 16-byte aligned.  status: as for mu_gemm_tc.
MU_EXPORT int mu_moe_gemm_tc(const void* xs, long long xs_rows, long long ldx, const int* pair_of, const void* w1, const void* w2,
                             int n_experts, const int* tile_info, const int* n_tiles, int max_tiles, int n, int k, void* out,
                             long long ldo, int out_bf16, int act, const float* row_weight, int* status, void* stream) {
    if (max_tiles <= 0 || xs_rows <= 0) return MU_OK;
    if (!xs || !w1 || !tile_info || !n_tiles || !out || !status || n <= 0 || k <= 0 || n_experts <= 0 || ldx < k || ldo < n)
        return MU_ERR_BAD_ARGUMENT;
    if (k % 8 || ldx % 8 || ((uintptr_t)xs & 15) || ((uintptr_t)w1 & 15) || ((uintptr_t)w2 & 15)) return MU_ERR_ALIGNMENT;
    if ((long long)n_experts * n > 0x7fffffffll || xs_rows > 0x7fffffffll || (act != mu::ACT_NONE && act != mu::ACT_RELU2) ||
        (w2 && act != mu::ACT_NONE))
        return MU_ERR_BAD_ARGUMENT;
    const int sms = mu::sm_count();
    if (sms <= 0) return MU_ERR_LAUNCH;
    // Columns of an item: 256 do more products per byte of A and per issued instruction; where the tiles are few the
    // weights' bytes decide, and items of 128 columns share them out more evenly.
    const bool wide = !w2 && (long long)max_tiles * ((n + 255) / 256) >= 4ll * sms;
    const int cols = w2 ? 128 : wide ? 256 : 128;
    const long long items = (long long)max_tiles * ((n + cols - 1) / cols);
    if (items > 0x7fffffffll) return MU_ERR_UNSUPPORTED_SIZE;
    typedef __nv_bfloat16 bf;
#define MU_GR(NB, G, TC)                                                                                                   \
    return mu::launch_grouped<NB, G, TC>(xs, xs_rows, k, ldx, w1, w2, (long long)n_experts * n, k, tile_info, n_tiles, pair_of, \
                                         row_weight, n, k, (TC*)out, ldo, act, status, 0, 1, 0, 0, nullptr, 0, items,       \
                                         (cudaStream_t)stream)
    if (w2) {
        if (out_bf16) MU_GR(2, true, bf);
        MU_GR(2, true, float);
    }
    if (wide) {
        if (out_bf16) MU_GR(2, false, bf);
        MU_GR(2, false, float);
    }
    if (out_bf16) MU_GR(1, false, bf);
    MU_GR(1, false, float);
#undef MU_GR
}

// As mu_heads_gemm (moe_mma.cu), for contiguous weights and k a multiple of 64 (a slice's stages of 64 then end where the
// slice ends).  x_cols: columns of x's rows that may be read (the last group's slice must end within them).
MU_EXPORT int mu_heads_gemm_tc(const void* x, int x_cols, long long ldx, long long x_group_offset, const void* w, int n_rows,
                               int n_groups, int n, int k, void* out, long long ldo, long long out_group_offset, int out_bf16,
                               const void* gate, long long ldg, int* status, void* stream) {
    if (n_rows <= 0 || n_groups <= 0) return MU_OK;
    if (!x || !w || !out || !status || n <= 0 || k <= 0 || x_cols < (n_groups - 1) * x_group_offset + k || ldx < x_cols)
        return MU_ERR_BAD_ARGUMENT;
    if (k % 64 || ldx % 8 || x_group_offset % 8 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15)) return MU_ERR_ALIGNMENT;
    const int cols = n > 128 ? 256 : 128;
    const long long items = (long long)((n_rows + 127) / 128) * ((n + cols - 1) / cols) * n_groups;
    if (items > 0x7fffffffll || (long long)n_groups * n > 0x7fffffffll || x_cols > 0x3fffffff) return MU_ERR_UNSUPPORTED_SIZE;
    typedef __nv_bfloat16 bf;
#define MU_HG(NB, TC)                                                                                                       \
    return mu::launch_grouped<NB, false, TC>(x, n_rows, x_cols, ldx, w, nullptr, (long long)n_groups * n, k, nullptr, nullptr, \
                                             nullptr, nullptr, n, k, (TC*)out, ldo, mu::ACT_NONE, status, n_rows, n_groups,  \
                                             (int)x_group_offset, out_group_offset, gate, ldg, items, (cudaStream_t)stream)
    if (cols == 256) {
        if (out_bf16) MU_HG(2, bf);
        MU_HG(2, float);
    }
    if (out_bf16) MU_HG(1, bf);
    MU_HG(1, float);
#undef MU_HG
}
