// C[M, N] = act(A[M, K] . W[N, K]^T + bias) (+ residual) by pairs of SMs: the product of gemm_tc_kernel.cuh (bfloat16 in, float32
// accumulators, the same epilogue) in tiles of 256 x BN, of which each block of a cluster of two computes 128 rows.
//
// What bounds the one-SM product at these sizes is the bytes an SM takes in from the L2 (16 KB of A and BN x 128 bytes of W for
// 64 of k).  In a pair every SM loads its own rows of A and HALF of W's rows, and tcgen05.mma.cta_group::2, which the first
// block issues, reads both halves: 32 KB for 128 x 256 x 64 instead of 48.  4,096 x 4,096 x 2,048
// in one launch of each: tensor pipe active in 81 % of the SMs' cycles, by single SMs in 74.  A pair's launch costs about 1 us
// more, so small products stay with one SM (the rule, with both sides: gemm_tc.cu).
//
// Roles in each block: warp 0 loads its share of every stage; both blocks' copies count on the FIRST block's "full" barrier.  Warp
// 1 allocates tensor memory (all 128 lanes of both SMs, two accumulators of BN columns); the first block's warp 1 issues
// the products and commits every stage to both blocks' "empty" barriers and every accumulator to both "acc_full".  Warps 2-9
// read the block's own 128 rows and finish them; both blocks' warps give an accumulator back on the first block's
// "acc_empty".  Waits are bounded as in gemm_tc_kernel.cuh; the blocks leave together.
#include "gemm_pair.cuh"

namespace mu {

template <int BN, int STAGES, typename TC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                 const __grid_constant__ CUtensorMap map_c, const float* __restrict__ bias, const float* residual, TC* C,
                 int M, int N, int K, long long ldc, long long ldr, int act, int* status, int bulk_out) {
    extern __shared__ unsigned char pair_raw[];
    PairSmem<BN, STAGES>& sm = *reinterpret_cast<PairSmem<BN, STAGES>*>(((uintptr_t)pair_raw + 1023) & ~(uintptr_t)1023);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int num_kb = (K + TC_BK - 1) / TC_BK;
    const int m_tiles = (M + 2 * TC_BM - 1) / (2 * TC_BM), n_tiles = (N + BN - 1) / BN, tiles = m_tiles * n_tiles;
    constexpr uint32_t STAGE_BYTES = (TC_BM + BN / 2) * TC_BK * sizeof(__nv_bfloat16);
    constexpr uint32_t TMEM_COLS = 2 * BN <= 256 ? 256 : 512;
    bool ok = true;

    if (threadIdx.x == 0) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_w);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&sm.acc_full[b], 1); mbar_init(&sm.acc_empty[b], 2 * TC_EPI_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&sm.tmem_base)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                          // both blocks' barriers and tensor memory are there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = sm.tmem_base;
    pdl_trigger();
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            long long it = 0, issued = 0;
            for (int tile = blockIdx.x >> 1; tile < tiles && ok; tile += gridDim.x >> 1) {
                const int m0 = (tile % m_tiles) * 2 * TC_BM + (int)rank * TC_BM, n0 = (tile / m_tiles) * BN + (int)rank * (BN / 2);
                for (int kb = 0; kb < num_kb; ++kb, ++it) {
                    const int s = (int)(it % STAGES);
                    ok = mbar_wait(&sm.empty[s], (uint32_t)(((it / STAGES) & 1) ^ 1));
                    if (!ok) break;
                    const uint32_t bar = in_first_block(&sm.full[s]);
                    if (rank == 0) mbar_expect_tx(&sm.full[s], 2 * STAGE_BYTES);
                    tma_load_2d_pair(sm.a[s], &map_a, kb * TC_BK, m0, bar);
                    tma_load_2d_pair(sm.b[s], &map_w, kb * TC_BK, n0, bar);
                    issued = it + 1;
                }
            }
            if (!ok) {
                atomicExch(status, 1);
                if (rank == 0)                               // copies under way land first (the other block waits below)
                    for (long long j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)
                        mbar_wait(&sm.full[j % STAGES], (uint32_t)((j / STAGES) & 1));
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            constexpr uint32_t idesc = idesc_bf16(2 * TC_BM, BN);
            constexpr uint32_t A_STAGE = TC_BM * TC_BK * sizeof(__nv_bfloat16) / 16, B_STAGE = BN / 2 * TC_BK * sizeof(__nv_bfloat16) / 16;
            const bool one = elect_one();
            const uint64_t a_desc0 = smem_desc_sw128(smem_u32(sm.a[0])), b_desc0 = smem_desc_sw128(smem_u32(sm.b[0]));
            long long it = 0;
            int local = 0;
            for (int tile = blockIdx.x >> 1; tile < tiles && ok; tile += gridDim.x >> 1, ++local) {
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
                    const uint64_t a_desc = a_desc0 + (uint64_t)(s * A_STAGE), b_desc = b_desc0 + (uint64_t)(s * B_STAGE);
                    if (!one) continue;
#pragma unroll
                    for (int k = 0; k < TC_BK / 16; ++k)
                        umma_bf16_pair(tmem_d, a_desc + 2 * k, b_desc + 2 * k, idesc, kb > 0 || k > 0 ? 1u : 0u);
                    umma_commit_pair(&sm.empty[s]);
                }
                if (ok && one) umma_commit_pair(&sm.acc_full[buf]);
            }
            if (!ok && one) atomicExch(status, 2);
        }
    } else {
        const int quad = warp & 3, half = (warp - 2) / 4;
        constexpr int COLS = BN / 2, CHUNKS = COLS / 32;
        float* patch = sm.patch[warp - 2];
        const bool vec_ok = sizeof(TC) == 2 && ((ldc * sizeof(TC)) % 16 == 0) && (((uintptr_t)C) % 16 == 0) && !residual &&
                            (((uintptr_t)bias) % 16 == 0);
        int local = 0;
        for (int tile = blockIdx.x >> 1; tile < tiles; tile += gridDim.x >> 1, ++local) {
            const int buf = local & 1;
            const int row0 = (tile % m_tiles) * 2 * TC_BM + (int)rank * TC_BM + quad * 32, n0 = (tile / m_tiles) * BN;
            ok = mbar_wait(&sm.acc_full[buf], (uint32_t)((local >> 1) & 1));
            if (!ok) {
                if (lane == 0) atomicExch(status, 3);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc_addr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN + half * COLS);
            const bool last = tile + (int)(gridDim.x >> 1) >= tiles;
            float* ring = reinterpret_cast<float*>(sm.a[0]) + (warp - 2) * (CHUNKS * 1024);
#pragma unroll
            for (int q = 0; q < CHUNKS; ++q) {
                const int nb = n0 + half * COLS + 32 * q;
                uint32_t r[32];
                tmem_ld_32x32(acc_addr + 32 * q, r);
                if (q == CHUNKS - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    if (lane == 0) mbar_arrive_cluster(in_first_block(&sm.acc_empty[buf]));
                }
                if (row0 >= M || nb >= N) continue;                   // the same for the whole warp
                if (bulk_out) {
                    if (act == ACT_GELU_NEW)
                        tc_finish_block_bulk<ACT_GELU_NEW, TC>(r, last ? ring + q * 1024 : patch, lane, bias, &map_c, N, row0, nb, bulk_out == 2, !last);
                    else if (act == ACT_GELU_ERF)
                        tc_finish_block_bulk<ACT_GELU_ERF, TC>(r, last ? ring + q * 1024 : patch, lane, bias, &map_c, N, row0, nb, bulk_out == 2, !last);
                    else if (act == ACT_RELU2)
                        tc_finish_block_bulk<ACT_RELU2, TC>(r, last ? ring + q * 1024 : patch, lane, bias, &map_c, N, row0, nb, bulk_out == 2, !last);
                    else
                        tc_finish_block_bulk<0, TC>(r, last ? ring + q * 1024 : patch, lane, bias, &map_c, N, row0, nb, bulk_out == 2, !last);
                    continue;
                }
                const bool packed = vec_ok && nb + 32 <= N;
                float bias_col[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int n = packed ? nb + 8 * (lane & 3) + e : nb + lane;
                    bias_col[e] = bias && n < N ? bias[n] : 0.0f;
                }
                if (act == ACT_GELU_NEW)
                    tc_finish_block<ACT_GELU_NEW, TC>(r, patch, lane, bias, bias_col, residual, C, M, N, row0, nb, ldc, ldr, packed);
                else if (act == ACT_GELU_ERF)
                    tc_finish_block<ACT_GELU_ERF, TC>(r, patch, lane, bias, bias_col, residual, C, M, N, row0, nb, ldc, ldr, packed);
                else if (act == ACT_RELU2)
                    tc_finish_block<ACT_RELU2, TC>(r, patch, lane, bias, bias_col, residual, C, M, N, row0, nb, ldc, ldr, packed);
                else
                    tc_finish_block<0, TC>(r, patch, lane, bias, bias_col, residual, C, M, N, row0, nb, ldc, ldr, packed);
            }
        }
    }
    if (bulk_out && warp >= 2 && lane == 0) tma_store_wait_all();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                          // neither block leaves while the other reads or signals it
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

template <int BN, int STAGES, typename TC>
static int launch_pair(const void* A, const void* W, const float* bias, const float* residual, TC* C, int M, int N, int K,
                       long long lda, long long ldw, long long ldc, long long ldr, int act, int* status, cudaStream_t s) {
    CUtensorMap map_a, map_w, map_c;
    if (!tensor_map_bf16(&map_a, A, M, K, lda, TC_BM) || !tensor_map_bf16(&map_w, W, N, K, ldw, BN / 2)) return MU_ERR_LAUNCH;
    int bulk_out = 0;                                        // as in launch_tc
    if ((((uintptr_t)C) & 15) == 0 && (ldc * (long long)sizeof(TC)) % 16 == 0 &&
        (residual == nullptr || (sizeof(TC) == 4 && (const void*)residual == (const void*)C && ldr == ldc)) &&
        tensor_map_out(&map_c, C, M, N, ldc, sizeof(TC) == 2))
        bulk_out = residual ? 2 : 1;
    if (!bulk_out) map_c = map_a;
    auto kernel = gemm_pair_kernel<BN, STAGES, TC>;
    const size_t smem = sizeof(PairSmem<BN, STAGES>) + 1024;
    if (!allow_shared(reinterpret_cast<const void*>(kernel), smem)) return MU_ERR_LAUNCH;
    prefer_shared_memory(reinterpret_cast<const void*>(kernel));
    const int pairs = sm_count() / 2;
    if (pairs <= 0) return MU_ERR_LAUNCH;
    const long long tiles = (long long)((M + 2 * TC_BM - 1) / (2 * TC_BM)) * ((N + BN - 1) / BN);
    return launch_pdl(kernel, dim3(2 * (unsigned)(tiles < pairs ? tiles : pairs)), dim3(TC_THREADS), smem, s, 1, map_a, map_w, map_c,
                      bias, residual, C, M, N, K, ldc, ldr, act, status, bulk_out);
}

// bn: 128, 192 or 256; the arguments as mu_gemm_tc has checked them.
int launch_gemm_pair(int bn, const void* A, const void* W, const float* bias, const float* residual, void* C, int M, int N, int K,
                     long long lda, long long ldw, long long ldc, long long ldr, int act, int out_bf16, int* status,
                     cudaStream_t s) {
#define MU_PAIR(BN, ST)                                                                                                       \
    case BN:                                                                                                                  \
        return out_bf16 ? launch_pair<BN, ST, __nv_bfloat16>(A, W, bias, residual, (__nv_bfloat16*)C, M, N, K, lda, ldw, ldc, \
                                                             ldr, act, status, s)                                             \
                        : launch_pair<BN, ST, float>(A, W, bias, residual, (float*)C, M, N, K, lda, ldw, ldc, ldr, act, status, s)
    switch (bn) {
        MU_PAIR(128, 7);
        MU_PAIR(192, 6);
        MU_PAIR(256, 5);
    }
#undef MU_PAIR
    return MU_ERR_BAD_ARGUMENT;
}

}  // namespace mu
