// C[M, N] = act(A[M, K] . W[N, K]^T + bias) (+ residual), float32 in and out, on the 5th-generation tensor cores: the 32-bit
// path's products over a long K.
//
// Every operand is two TF32 numbers, hi = x rounded to 11 bits and lo = x - hi rounded to 11 bits (together 22 to 23 bits of
// x's 24), and a product three: lo hi + hi lo + hi hi.  What tensor cores lose of a sum is not in the operands but in the
// accumulator, which they cut off instead of rounding it; so an accumulator only ever holds 32 of k (twelve products, the
// small ones first), and warps add it to the tile's float32 sums in registers, rounded.  Error against float64 (2-norm, normal
// values; float32 multiply-adds, gemm_simt.cu, in brackets): k = 192 1.13e-7 (1.32e-7), 768 1.37e-7 (2.52e-7), 3072 1.43e-7
// (4.98e-7); all values positive: 4.6e-8 (6.6e-8), 7.6e-8 (1.11e-7), 5.7e-8 (2.08e-7).
//
// A block per SM walks over tiles of 128 x BN.  Warp 0 issues the TMA loads of 32 of k (128 rows of A, BN of W, 128-byte
// swizzle).  Sixteen warps split them: A's parts go to tensor memory (a row a lane), W's hi part back to where it came from and
// its lo part beside it, which keeps the swizzle.  Warp 1 issues the products with A from tensor memory and W from shared
// memory into one of two accumulators; the sixteen warps meanwhile add the other to their sums (32 rows x BN / 4 columns a
// warp).  With A's operands in shared memory as well a step would move 252 KB through it instead of 172 (BN = 160), at 128
// bytes a cycle more than its products take; as it is both take about as long.  What is left is the warps' chain from load
// to arrival: a step of 32 took 0.42 us (32 columns), 0.67 (96), 0.80 (128) and 1.0 (160) whatever of the splitting,
// the products or the sums was left out alone, so two teams of eight warps split every other step.  Measured (B200,
// microseconds; the multiply-adds in brackets): 777 x 3072 x 768 30 (121), 777 x 768 x 3072 40 (129), 2048 x 4096 x 4096 412
// (1,700; 167 TFLOP/s), 8 x 3072 x 768 14 (19), 8 x 768 x 3072 12.5 (66).
//
// A tile's sum is, for every run of k, the sum of its steps in order, and then the runs' sums in order; how long a run is
// follows from k alone.  A product of few tiles is cut into those runs (CUT): a cluster of blocks has a tile, each block
// a run, and every block adds the runs of its share of the columns, in order, as they lie in the other blocks' shared memory.  So
// a row's result is the same bits whatever the cut, the tile's width and the rest of the step are, and no launch keeps
// anything in device memory that another one, on another stream, could meet.
//
// A value that is infinite, or NaN, or rounds to infinity in 11 bits, has parts that make NaN where float32 gives
// an infinity; so a sum that comes out not finite is made once more by multiply-adds, by the lane that stores it.
#include "tcgen05.cuh"

#include <atomic>

namespace mu {

constexpr int FC_BM = 128, FC_BK = 32, FC_WORKERS = 16, FC_THREADS = 64 + 32 * FC_WORKERS;
constexpr int FC_RUN = 24, FC_RUNS = 8;                  // a run's steps of 32, if k has no more than that many runs
// Steps of a run: runs of one length, as few as FC_RUN allows (a cluster has eight blocks).
inline int fc_group(int steps) {
    const int runs = (steps + FC_RUN - 1) / FC_RUN;
    return (steps + (runs < FC_RUNS ? runs : FC_RUNS) - 1) / (runs < FC_RUNS ? runs : FC_RUNS);
}
constexpr int FC_TEAM = FC_WORKERS / 2;                  // two teams of warps split every other step
// What tensor cores cut off of an accumulator's four large additions is 2^-23 of it on average; it is given back.
constexpr float FC_GIVE_BACK = 1.0f + 1.1920929e-7f;
constexpr int FC_PITCH = 9;                              // floats a row of an epilogue patch (32 rows x 8 columns)

bool tensor_map_f32(CUtensorMap* map, const void* base, long long rows, int cols, long long ld, int box_rows);

// Instruction descriptor of kind::tf32: float32 accumulator, TF32 operands (2 at bits 7 and 10), both K-major.
__host__ __device__ constexpr uint32_t idesc_tf32(int m, int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld_x8_nowait(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// x to 11 bits, ties away from zero (a NaN may lose its mark here: its other part, x - hi, keeps it).
__device__ __forceinline__ uint32_t tf32_bits(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
__device__ __forceinline__ void tf32_parts(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_bits(x);
    lo = __float_as_uint(x - __uint_as_float(hi));       // (exact; the tensor cores read its first 11 bits)
}
__device__ __forceinline__ bool is_finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

template <int BN> constexpr int fc_room(bool runs) { return runs && BN * 8 > 32 * FC_PITCH ? BN * 8 : 32 * FC_PITCH; }

template <int BN, int STAGES, bool RUNS>
struct FcSmem {
    float a[STAGES][FC_BM * FC_BK];                      // rows of 128 bytes, 128-byte swizzle, each tile 1024-byte aligned
    float w_hi[STAGES][BN * FC_BK];                      // W as it came, then its hi parts
    float w_lo[STAGES][BN * FC_BK];
    float patch[FC_WORKERS][fc_room<BN>(RUNS)];          // a warp's patch, and before that (RUNS) its sum of the runs so far
    uint64_t full[STAGES], split[STAGES], empty[STAGES]; // loaded; split into parts; read by the products
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem_base;
};

// The sum once more by multiply-adds in the order of k.
__device__ __noinline__ float fc_plain_sum(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.0f;
    for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
    return s;
}

struct FcArgs {
    const float *A, *W, *bias, *residual;
    float* C;
    int M, N, K;
    long long lda, ldw, ldc, ldr;
    int* status;
    int group, runs;                                     // steps of a run, runs of k
};

template <int ACT> __device__ __forceinline__ float fc_act(float x) {
    if (ACT == ACT_GELU_NEW) return gelu_new(x);
    if (ACT == ACT_GELU_ERF) return gelu_erf(x);
    if (ACT == ACT_RELU2) return relu2(x);
    return x;
}

// A warp's 32 rows x CW columns to C: through its patch eight columns at a time, so that an instruction touches four rows'
// 32 bytes.
template <int ACT, int CW>
__device__ __forceinline__ void fc_finish(const FcArgs& g, const float* sum, float* patch, int lane, int row0, int col0) {
    const int c = lane & 7, r0 = lane >> 3, n_rows = min(32, g.M - row0);
#pragma unroll
    for (int p = 0; p < CW / 8; ++p) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) patch[lane * FC_PITCH + i] = sum[8 * p + i];
        __syncwarp();
        const int n = col0 + 8 * p + c;
        const bool live = n < g.N;
        const float b = g.bias && live ? g.bias[n] : 0.0f;
        float res[8];
#pragma unroll
        for (int it = 0; it < 8; ++it)
            res[it] = g.residual && live && 4 * it + r0 < n_rows ? g.residual[(long long)(row0 + 4 * it + r0) * g.ldr + n] : 0.0f;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const int r = 4 * it + r0;
            if (!live || r >= n_rows) continue;
            float v = patch[r * FC_PITCH + c];
            if (!is_finite_bits(v)) v = fc_plain_sum(g.A + (long long)(row0 + r) * g.lda, g.W + (long long)n * g.ldw, g.K);
            g.C[(long long)(row0 + r) * g.ldc + n] = fc_act<ACT>(v + b) + res[it];
        }
    }
}

__device__ __forceinline__ void fc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 fc_load_remote(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// RUNS: a block sums several runs of a tile.  CUT: a cluster's blocks (along y) have a run of one tile each.
template <int BN, int STAGES, bool RUNS, bool CUT>
__global__ void __launch_bounds__(FC_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const FcArgs g, int act) {
    extern __shared__ unsigned char fc_raw[];
    FcSmem<BN, STAGES, RUNS>& sm = *reinterpret_cast<FcSmem<BN, STAGES, RUNS>*>(((uintptr_t)fc_raw + 1023) & ~(uintptr_t)1023);
    constexpr int CW = BN / 4, COL_A = 2 * BN, COLS = COL_A + 64 * STAGES;
    constexpr uint32_t TMEM_COLS = COLS <= 128 ? 128 : COLS <= 256 ? 256 : 512;
    static_assert(COLS <= 512 && BN % 32 == 0, "tensor memory");
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int steps = (g.K + FC_BK - 1) / FC_BK;
    const int m_tiles = (g.M + FC_BM - 1) / FC_BM, n_tiles = (g.N + BN - 1) / BN;
    const int tiles = m_tiles * n_tiles;
    const int begin = CUT ? (int)blockIdx.y * g.group : 0, end = CUT ? min(steps, begin + g.group) : steps;      // this block's steps
    bool ok = true;

    if (threadIdx.x == 0) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_w);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&sm.full[s], 1); mbar_init(&sm.split[s], FC_TEAM); mbar_init(&sm.empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&sm.acc_full[b], 1); mbar_init(&sm.acc_empty[b], FC_WORKERS); }
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
    const uint32_t tmem = sm.tmem_base;
    pdl_trigger();
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int it = 0, issued = 0;
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                const int m0 = tile % m_tiles * FC_BM, n0 = tile / m_tiles * BN;
                for (int st = begin; st < end; ++st, ++it) {
                    const int s = it % STAGES;
                    ok = mbar_wait(&sm.empty[s], (uint32_t)((it / STAGES & 1) ^ 1));
                    if (!ok) break;
                    mbar_expect_tx(&sm.full[s], (FC_BM + BN) * FC_BK * sizeof(float));
                    tma_load_2d(sm.a[s], &map_a, st * FC_BK, m0, &sm.full[s]);
                    tma_load_2d(sm.w_hi[s], &map_w, st * FC_BK, n0, &sm.full[s]);
                    issued = it + 1;
                }
            }
            if (!ok) {
                atomicExch(g.status, 1);
                for (int j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)      // copies under way land first
                    mbar_wait(&sm.full[j % STAGES], (uint32_t)(j / STAGES & 1));
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = idesc_tf32(FC_BM, BN), STAGE16 = BN * FC_BK * sizeof(float) / 16;
        const bool one = elect_one();
        const uint64_t hi0 = smem_desc_sw128(smem_u32(sm.w_hi[0])), lo0 = smem_desc_sw128(smem_u32(sm.w_lo[0]));
        int it = 0;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            for (int st = begin; st < end; ++st, ++it) {
                const int s = it % STAGES, buf = it & 1;
                ok = mbar_wait(&sm.split[s], (uint32_t)(it / STAGES & 1)) &&
                     mbar_wait(&sm.acc_empty[buf], (uint32_t)((it >> 1 & 1) ^ 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(buf * BN), a_hi = tmem + (uint32_t)(COL_A + 64 * s), a_lo = a_hi + 32;
                const uint64_t w_hi = hi0 + (uint64_t)(s * STAGE16), w_lo = lo0 + (uint64_t)(s * STAGE16);
                if (!one) continue;
#pragma unroll
                for (int k = 0; k < 4; ++k) {            // 8 of k: 8 columns, 32 bytes
                    umma_tf32_ts(d, a_lo + 8 * k, w_hi + 2 * k, idesc, k > 0);
                    umma_tf32_ts(d, a_hi + 8 * k, w_lo + 2 * k, idesc, 1);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) umma_tf32_ts(d, a_hi + 8 * k, w_hi + 2 * k, idesc, 1);
                umma_commit(&sm.empty[s]);
                umma_commit(&sm.acc_full[buf]);
            }
        }
        if (!ok && lane == 0) atomicExch(g.status, 2);
    } else {
        const int quad = warp & 3, part = (warp - 2) >> 2, tid = threadIdx.x - 64;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const bool rows_here = g.M > quad * 32;          // a single row of tiles may leave whole warps without rows
        float* patch = sm.patch[warp - 2];
        const int total = ((int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0) * (end - begin);
        auto split = [&](int it) {                       // this warp's share of a step: 32 rows x 16 of k of A, an eighth of W
            const int s = it % STAGES;
            if (!mbar_wait(&sm.full[s], (uint32_t)(it / STAGES & 1))) return false;
            constexpr int THREADS = 32 * FC_TEAM, PIECES = (BN * 8 + THREADS - 1) / THREADS, QUARTERS = 4;
            constexpr bool EVEN = BN * 8 % THREADS == 0;
            const int row = quad * 32 + lane, at = tid & (THREADS - 1), k4 = (part & 1) * QUARTERS;
            float4 x[QUARTERS], w[PIECES];               // all are asked for before any is split
#pragma unroll
            for (int j = 0; j < QUARTERS; ++j)
                x[j] = *reinterpret_cast<const float4*>(sm.a[s] + row * FC_BK + (((k4 + j) ^ (row & 7)) << 2));
            float4* w_at = reinterpret_cast<float4*>(sm.w_hi[s]) + at;
            uint4* lo_at = reinterpret_cast<uint4*>(sm.w_lo[s]) + at;
#pragma unroll
            for (int i = 0; i < PIECES; ++i)
                if (EVEN || at + i * THREADS < BN * 8) w[i] = w_at[i * THREADS];
            if (rows_here) {
#pragma unroll
                for (int h = 0; h < QUARTERS / 2; ++h) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float4 v = x[2 * h + j];
                        tf32_parts(v.x, hi[4 * j], lo[4 * j]); tf32_parts(v.y, hi[4 * j + 1], lo[4 * j + 1]);
                        tf32_parts(v.z, hi[4 * j + 2], lo[4 * j + 2]); tf32_parts(v.w, hi[4 * j + 3], lo[4 * j + 3]);
                    }
                    tmem_st_x8(lanes + (uint32_t)(COL_A + 64 * s + 4 * k4 + 8 * h), hi);
                    tmem_st_x8(lanes + (uint32_t)(COL_A + 64 * s + 32 + 4 * k4 + 8 * h), lo);
                }
            }
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                if (EVEN || at + i * THREADS < BN * 8) {
                    uint4 hi, lo;
                    tf32_parts(w[i].x, hi.x, lo.x); tf32_parts(w[i].y, hi.y, lo.y);
                    tf32_parts(w[i].z, hi.z, lo.z); tf32_parts(w[i].w, hi.w, lo.w);
                    *reinterpret_cast<uint4*>(w_at + i * THREADS) = hi;
                    lo_at[i * THREADS] = lo;
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.split[s]);
            return true;
        };
        const int team = part >> 1;
        int it = 0;
        if (total > 0 && team == 0) ok = split(0);
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            float2x sum[CW / 2];
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) sum[i] = 0ull;
            int run_end = begin + g.group;
            for (int st = begin; st < end; ++st, ++it) {
                if (it + 1 < total && team == ((it + 1) & 1)) ok = split(it + 1);
                const int buf = it & 1;
                ok = ok && mbar_wait(&sm.acc_full[buf], (uint32_t)(it >> 1 & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (rows_here) {
                    uint32_t r[CW];
#pragma unroll
                    for (int c = 0; c < CW; c += 8) tmem_ld_x8_nowait(lanes + (uint32_t)(buf * BN + part * CW + c), r + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < CW / 2; ++i)
                        sum[i] = pair_fma(pair_of_floats(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])),
                                          pair_of_floats(FC_GIVE_BACK, FC_GIVE_BACK), sum[i]);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.acc_empty[buf]);
                if (RUNS && st + 1 == run_end && st + 1 != end) {                // a run is complete: onto those before it
                    float2x* at = reinterpret_cast<float2x*>(patch) + lane;
#pragma unroll
                    for (int i = 0; i < CW / 2; ++i) {
                        at[32 * i] = run_end == g.group ? sum[i] : pair_add(at[32 * i], sum[i]);
                        sum[i] = 0ull;
                    }
                    run_end += g.group;
                }
            }
            if (!ok) break;
            if (RUNS && g.runs > 1) {
                const float2x* at = reinterpret_cast<const float2x*>(patch) + lane;
#pragma unroll
                for (int i = 0; i < CW / 2; ++i) sum[i] = pair_add(at[32 * i], sum[i]);
            }
            float out[CW];
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) {
                const float2 two = floats_of_pair(sum[i]);
                out[2 * i] = two.x;
                out[2 * i + 1] = two.y;
            }
            const int row0 = tile % m_tiles * FC_BM + quad * 32, col0 = tile / m_tiles * BN + part * CW;
            if constexpr (CUT) {
                // The run's sums to where the operands lay (every product has read them): four columns of 32 rows side by side,
                // warp after warp.
                float4* mine = reinterpret_cast<float4*>(sm.a[0]) + (warp - 2) * (CW / 4) * 32 + lane;
#pragma unroll
                for (int j = 0; j < CW / 4; ++j) mine[32 * j] = make_float4(out[4 * j], out[4 * j + 1], out[4 * j + 2], out[4 * j + 3]);
                continue;                                // (a block has one tile)
            }
            if (row0 < g.M && col0 < g.N) {
                if (act == ACT_GELU_NEW) fc_finish<ACT_GELU_NEW, CW>(g, out, patch, lane, row0, col0);
                else if (act == ACT_GELU_ERF) fc_finish<ACT_GELU_ERF, CW>(g, out, patch, lane, row0, col0);
                else if (act == ACT_RELU2) fc_finish<ACT_RELU2, CW>(g, out, patch, lane, row0, col0);
                else fc_finish<0, CW>(g, out, patch, lane, row0, col0);
            }
        }
        if (!ok && lane == 0) atomicExch(g.status, 3);
    }
    if constexpr (CUT) {
        static_assert(sizeof(sm.a) + sizeof(sm.w_hi) + sizeof(sm.w_lo) >= FC_BM * BN * sizeof(float), "room for a run's sums");
        ok = __all_sync(0xffffffffu, ok);
        fc_cluster_sync();                               // every run's sums are in its block's shared memory
        if (warp >= 2 && ok) {
            // Eight columns of 32 rows at a time, dealt out to the cluster's blocks and their warps.
            constexpr int EIGHTS = CW / 8;
            const int m0 = (int)blockIdx.x % m_tiles * FC_BM, n0 = (int)blockIdx.x / m_tiles * BN;
            for (int p = (int)blockIdx.y + (warp - 2) * g.runs; p < FC_WORKERS * EIGHTS; p += FC_WORKERS * g.runs) {
                const int owner = p / EIGHTS, row0 = m0 + ((owner + 2) & 3) * 32, col0 = n0 + (owner >> 2) * CW + p % EIGHTS * 8;
                if (row0 >= g.M || col0 >= g.N) continue;
                const uint32_t at = smem_u32(reinterpret_cast<const float4*>(sm.a[0]) + 2 * p * 32 + lane);
                float out[8];
                for (int r = 0; r < g.runs; ++r) {
                    uint32_t there;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(r));
                    const float4 x = fc_load_remote(there), y = fc_load_remote(there + 32 * sizeof(float4));
                    const float more[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                    for (int j = 0; j < 8; ++j) out[j] = r ? out[j] + more[j] : more[j];
                }
                float* patch = sm.patch[warp - 2];
                if (act == ACT_GELU_NEW) fc_finish<ACT_GELU_NEW, 8>(g, out, patch, lane, row0, col0);
                else if (act == ACT_GELU_ERF) fc_finish<ACT_GELU_ERF, 8>(g, out, patch, lane, row0, col0);
                else if (act == ACT_RELU2) fc_finish<ACT_RELU2, 8>(g, out, patch, lane, row0, col0);
                else fc_finish<0, 8>(g, out, patch, lane, row0, col0);
            }
        }
        __syncwarp();
        fc_cluster_sync();                               // no block leaves while another reads its sums
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

template <int BN, int STAGES, bool RUNS, bool CUT>
int launch_f32_tc(const FcArgs& g, int act, int sms, cudaStream_t s) {
    CUtensorMap map_a, map_w;
    if (!tensor_map_f32(&map_a, g.A, g.M, g.K, g.lda, FC_BM) || !tensor_map_f32(&map_w, g.W, g.N, g.K, g.ldw, BN)) return MU_ERR_LAUNCH;
    auto kernel = gemm_f32_tc_kernel<BN, STAGES, RUNS, CUT>;
    const size_t smem = sizeof(FcSmem<BN, STAGES, RUNS>) + 1024;
    if (!allow_shared(reinterpret_cast<const void*>(kernel), smem)) return MU_ERR_LAUNCH;
    prefer_shared_memory(reinterpret_cast<const void*>(kernel));
    const long long tiles = (long long)((g.M + FC_BM - 1) / FC_BM) * ((g.N + BN - 1) / BN);
    const dim3 grid((unsigned)(CUT || tiles < sms ? tiles : sms), CUT ? g.runs : 1);
    return launch_pdl(kernel, grid, dim3(FC_THREADS), smem, s, CUT ? g.runs : 1, map_a, map_w, g, act);
}

// Tiles that are worked on at once if each is cut into `runs`: clusters that the device takes at a time (asked for once).
template <int BN, int STAGES>
int fc_clusters(int runs) {
    static std::atomic<int> known[FC_RUNS + 1];
    int n = known[runs].load(std::memory_order_relaxed);
    if (n != 0) return n;
    auto kernel = gemm_f32_tc_kernel<BN, STAGES, false, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, runs);
    cfg.blockDim = dim3(FC_THREADS);
    cfg.dynamicSmemBytes = sizeof(FcSmem<BN, STAGES, false>) + 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = (unsigned)runs;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (!allow_shared(reinterpret_cast<const void*>(kernel), cfg.dynamicSmemBytes) ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = -1;                                          // (never cut)
    }
    known[runs].store(n, std::memory_order_relaxed);
    return n;
}

}  // namespace mu

// float32 A [M, K] (lda), W [N, K] (ldw): K, lda, ldw multiples of 4, bases 16-byte aligned.  C float32 (ldc); residual
// float32 (ldr), may be C itself.  `status`: as mu_gemm_tc's.  tile: width of the tiles (0: chosen here); cut: 0 never, 1
// wherever K has several runs, -1 chosen here.  Neither changes a bit of the result.
MU_EXPORT int mu_gemm_f32_tc(const void* A, const void* W, const float* bias, const float* residual, void* C, int M, int N,
                             int K, long long lda, long long ldw, long long ldc, long long ldr, int act, int tile, int cut,
                             int* status, void* stream) {
    if (M <= 0 || N <= 0) return MU_OK;
    if (K <= 0 || !A || !W || !C || !status) return MU_ERR_BAD_ARGUMENT;
    if (K % 4 != 0 || lda % 4 != 0 || ldw % 4 != 0 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return MU_ERR_ALIGNMENT;
    if (lda < K || ldw < K || ldc < N || (residual && ldr < N) || cut < -1 || cut > 1) return MU_ERR_BAD_ARGUMENT;
    if (tile != 0 && tile != 32 && tile != 64 && tile != 96 && tile != 128 && tile != 160) return MU_ERR_BAD_ARGUMENT;
    const int sms = mu::sm_count();
    if (sms <= 0) return MU_ERR_LAUNCH;
    const long long m_tiles = (M + mu::FC_BM - 1) / mu::FC_BM;
    if (m_tiles * ((N + 31) / 32) > (1LL << 30)) return MU_ERR_UNSUPPORTED_SIZE;
    const int steps = (K + mu::FC_BK - 1) / mu::FC_BK, group = mu::fc_group(steps), runs = (steps + group - 1) / group;
    const mu::FcArgs g = {(const float*)A, (const float*)W, bias, residual, (float*)C, M, N, K, lda, ldw, ldc, ldr, status,
                          group, runs};
    cudaStream_t s = (cudaStream_t)stream;
#define MU_FC_ALL(DO) DO(32, 7, 6) DO(64, 6, 5) DO(96, 5, 4) DO(128, 4, 3) DO(160, 3, 3)
    // The width, and whether to cut, by what the SM that ends last has to do, in microseconds: a step took 0.42 (32 columns), 0.67
    // (96), 0.80 (128) and 1.0 (160), handing the sums over 4.
    int best = 0, best_cut = 0;
    double best_cost = 0.0;
    const int widths[5] = {32, 64, 96, 128, 160};
    for (int i = 0; i < 5; ++i) {
        const int bn = widths[i];
        if (tile ? bn != tile : bn > 32 && bn - 32 >= N) continue;
        const long long tiles = m_tiles * ((N + bn - 1) / bn);
        for (int c = 0; c < 2; ++c) {
            if (c == 1 && (cut == 0 || runs == 1)) continue;
            if (c == 0 && runs > 1 && bn == 160) continue;           // (no registers for both sums)
            long long at_once = sms;
            if (c == 1) {
#define MU_FC_CLUSTERS(BN, ST, ST_RUNS) if (bn == BN) at_once = mu::fc_clusters<BN, ST>(runs);
                MU_FC_ALL(MU_FC_CLUSTERS)
#undef MU_FC_CLUSTERS
                if (at_once <= 0) continue;
            }
            const long long rounds = (tiles + at_once - 1) / at_once;
            double cost = rounds * ((c ? group : steps) * (0.28 + 0.0045 * bn) + 1.0 + 0.01 * bn) + (c ? 4.0 : 0.0);
            if (c == 1 && cut == 1) cost *= 1e-6;
            if (best == 0 || cost < best_cost) best = bn, best_cut = c, best_cost = cost;
        }
    }
    if (best == 0) best = tile == 160 ? 128 : tile, best_cut = 0;
#define MU_FC(BN, ST, ST_RUNS)                                                                                         \
    if (best == BN) {                                                                                                  \
        if (best_cut) return mu::launch_f32_tc<BN, ST, false, true>(g, act, sms, s);                                   \
        if (runs == 1) return mu::launch_f32_tc<BN, ST, false, false>(g, act, sms, s);                                 \
        if constexpr (BN < 160) return mu::launch_f32_tc<BN, ST_RUNS, true, false>(g, act, sms, s);                    \
    }
    MU_FC_ALL(MU_FC)
#undef MU_FC
#undef MU_FC_ALL
    return MU_ERR_BAD_ARGUMENT;
}
