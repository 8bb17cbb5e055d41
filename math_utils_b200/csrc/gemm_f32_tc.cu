// C[M, N] = act(A[M, K] . W[N, K]^T + bias) (+ residual), float32 in and out, on the 5th-generation tensor cores: the 32-bit
// path's products over a long K.
//
// Every operand is three bfloat16 numbers that are together exactly it (8 bits each of its 24, each rounded from what those
// before left), and a product eight: all but lo lo, which is 2^-36 of it at most.  What is left to lose is in the accumulators, which
// tensor cores cut off instead of rounding.  So the large products, hi hi (16 bits each), have an accumulator of their own that
// holds 32 of k (two instructions) and is added to the tile's float32 sums in registers, rounded; the seven others, 2^-8 and
// less of these, run on in a second one and are added at the end of a run of k (below), where what they were cut by is nothing.
// A product that float32 holds is exact, and so are sums of whole numbers up to 2^24; entries below 2^-109 lose their last bits
// (bfloat16 has none below 2^-133).
// Error against float64, rms over the outputs of |error| / (|a| . |w|) (float32 multiply-adds, gemm_simt.cu, in brackets): normal
// values k = 384 5.8e-9 (1.45e-8), 768 4.9e-9 (1.42e-8), 3072 3.2e-9 (1.41e-8); positive ones 768 6.1e-8 (1.11e-7), 3072 6.3e-8
// (2.11e-7); rows of 1, 4, 16 and 64 values, k = 768, 2.53e-8 (2.53e-8), 2.40e-8 (2.95e-8), 1.49e-8 (2.21e-8), 9.7e-9 (1.66e-8);
// log-normal factors of sigma 2 and any sign 4.2e-8 (9.9e-8).  Further off than multiply-adds only where both rows are
// positive and a few terms carry the sum (log-normal factors of sigma 2, none negative: k = 384 1.34 times, 512 1.22, 768 1.10, from
// 1536 on less over whole rows), and by 8 % where k has eight runs and a row two positive values in each.
//
// A block per SM walks over tiles of 128 x BN.  Warp 0 issues the TMA loads of 32 of k (128 rows of A, BN of W, 128-byte
// swizzle).  Sixteen warps split them: A's parts go to tensor memory (a row a lane), W's hi and mid parts back to where the row
// came from and its lo parts beside it.  Warp 1 issues the products with A from tensor memory and W from shared memory; the
// sixteen warps add what is complete to their sums (32 rows x BN / 4 columns a warp).  A step of 32 of k and 128 columns takes
// 0.79 us, some 1,500 cycles: its products need 1,024, its bytes through shared memory 1,190 at 128 a cycle (fill, split, W's
// parts eight times), its instructions about half; none is the bound alone (tensor pipe active in 36 to 46 % of a whole launch's
// cycles, issue in 46 to 52 %).  The warps' chain from load to arrival lies over them: two teams of eight split every other step,
// two steps ahead (one step ahead: 0.92).  Eighteen warps leave 96 registers each: uncut tiles of 128 columns spill 128 bytes, of 64
// 36 and of 160 20, cut ones of the same steps, whose ends take eight columns a warp at a time, 4 bytes at most.  Others: 0.48 us (32 columns), 0.56 (64), 0.71 (96), 1.04 (160).  Measured (B200, microseconds; the multiply-adds in
// brackets): 777 x 3072 x 768 37 (121), 777 x 768 x 768 15.4 (34), 777 x 768 x 3072 44 (129), 2048 x 4096 x 4096 475 (1,700; 145
// TFLOP/s), 8 x 3072 x 768 11.6 (17.5), 8 x 768 x 3072 14 (66).
//
// A tile's sum is, for every run of k, the sum of its steps in order, and then the runs' sums in order; how long a run is
// follows from k alone.  A product of few tiles is cut into those runs (CUT): a cluster of blocks has a tile, each block
// a run, and every block adds the runs of its share of the columns, in order, as they lie in the other blocks' shared memory.  So
// a row's result is the same bits whatever the cut, the tile's width and the rest of the step are, and no launch keeps
// anything in device memory that another one, on another stream, could meet.
//
// A value that is infinite, or NaN, or rounds to infinity in 8 bits, has parts that make NaN where float32 gives
// an infinity; so a sum that comes out not finite is made once more by multiply-adds, by the lane that stores it, up to where it is NaN.
// 777 x 3072 x 768 takes 37 us, with a NaN early in one row 39, in all rows 61 (to the end of every sum: 150 and 3,065), with one
// row infinite 186 and with all 2,350.
#include "tcgen05.cuh"

#include <atomic>

namespace mu {

constexpr int FC_BM = 128, FC_BK = 32, FC_WORKERS = 16, FC_THREADS = 64 + 32 * FC_WORKERS;
// k in runs of one length: two, more where they would be longer than FC_RUN steps of 32, up to the eight blocks of a cluster.  One
// sum over all of k rounds at its full size at every step, and rows of 32 to 256 positive values (k = 768) came out up to
// 1.28 times as far off as by multiply-adds, which keep four sums; two runs 0.88 times.  768 of k are some 20 us of a block (128
// columns), against 3 for a cluster's start and handing over, and every run more is a rounding more of sums of few values.
constexpr int FC_RUN = 24, FC_RUNS = 8;
inline int fc_group(int steps) {
    const int most = (steps + FC_RUN - 1) / FC_RUN, runs = most < 2 ? 2 : most < FC_RUNS ? most : FC_RUNS;
    return (steps + runs - 1) / runs;
}
constexpr int FC_TEAM = FC_WORKERS / 2;                  // two teams of warps split every other step
constexpr int FC_PITCH = 9;                              // floats a row of an epilogue patch (32 rows x 8 columns)

bool tensor_map_f32(CUtensorMap* map, const void* base, long long rows, int cols, long long ld, int box_rows);

// K-major operand in rows of 64 bytes with the 64-byte swizzle, groups of 8 rows 512 bytes apart (mode 4; the rest as smem_desc_sw128).
__device__ __forceinline__ uint64_t fc_desc_sw64(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
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
// Two values as three pairs of bfloat16 (the first in the low half), each rounded from what those before it left: exactly the
// values, down to 2^-109 (where the third falls below bfloat16's range).
__device__ __forceinline__ void fc_parts(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
    x -= __uint_as_float(hi << 16), y -= __uint_as_float(hi & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(y), "f"(x));
    x -= __uint_as_float(mid << 16), y -= __uint_as_float(mid & 0xffff0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(y), "f"(x));
}
__device__ __forceinline__ bool is_finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

template <int BN> constexpr int fc_room(bool cut) { return !cut && BN * 8 > 32 * FC_PITCH ? BN * 8 : 32 * FC_PITCH; }

template <int BN, int STAGES, bool CUT>
struct FcSmem {
    float a[STAGES][FC_BM * FC_BK];                      // rows of 128 bytes, 128-byte swizzle, each tile 1024-byte aligned
    float w[STAGES][BN * FC_BK];                         // W as it came, then a row's hi parts and its mid parts, 64 bytes each
    __nv_bfloat16 w_lo[STAGES][BN * FC_BK];              // rows of 64 bytes, 64-byte swizzle
    float patch[FC_WORKERS][fc_room<BN>(CUT)];           // a warp's patch, and before that (uncut) its sum of the runs so far
    uint64_t full[STAGES], split[STAGES], empty[STAGES]; // loaded; split into parts; read by the products
    uint64_t acc_full, acc_empty, small_empty[2];
    uint32_t tmem_base;
};

// The sum once more by multiply-adds in the order of k, to its end or until it is NaN, which it stays.
__device__ __noinline__ float fc_plain_sum(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.0f;
    for (int k = 0; k < K && s == s; k += 4) {               // (rows are whole 16-byte pieces)
        const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
    }
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

// CUT: a cluster's blocks (along y) have a run of one tile each; otherwise a block sums all runs of its tiles.
template <int BN, int STAGES, bool CUT>
__global__ void __launch_bounds__(FC_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const FcArgs g, int act) {
    extern __shared__ unsigned char fc_raw[];
    FcSmem<BN, STAGES, CUT>& sm = *reinterpret_cast<FcSmem<BN, STAGES, CUT>*>(((uintptr_t)fc_raw + 1023) & ~(uintptr_t)1023);
    // tensor memory: sums of the large products, of the small ones (SMALL buffers), A's parts of AHEAD + 1 steps
    constexpr int CW = BN / 4, AHEAD = 2, SMALL = BN <= 96 ? 2 : 1, COL_SMALL = BN;
    constexpr int COL_A = COL_SMALL + SMALL * BN, COLS = COL_A + (AHEAD + 1) * 48;
    constexpr uint32_t TMEM_COLS = COLS <= 256 ? 256 : 512;
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
        mbar_init(&sm.acc_full, 1);
        mbar_init(&sm.acc_empty, FC_WORKERS);
        for (int b = 0; b < 2; ++b) mbar_init(&sm.small_empty[b], FC_WORKERS);
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
                    tma_load_2d(sm.w[s], &map_w, st * FC_BK, n0, &sm.full[s]);
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
        constexpr uint32_t idesc = idesc_bf16(FC_BM, BN), W_STAGE = BN * FC_BK * sizeof(float) / 16, LO_STAGE = W_STAGE / 2;
        const bool one = elect_one();
        const uint64_t w0 = smem_desc_sw128(smem_u32(sm.w[0])), lo0 = fc_desc_sw64(smem_u32(sm.w_lo[0]));
        int it = 0, run = -1;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            int run_at = begin;                          // the step that begins a run
            for (int st = begin; st < end; ++st, ++it) {
                const int s = it % STAGES;
                const bool first = st == run_at;
                if (first) run_at += g.group, ++run;
                const int small = run % SMALL;
                ok = mbar_wait(&sm.split[s], (uint32_t)(it / STAGES & 1));
                if (ok && first) ok = mbar_wait(&sm.small_empty[small], (uint32_t)((run / SMALL & 1) ^ 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_hi = tmem + (uint32_t)(COL_A + 48 * (it % (AHEAD + 1))), a_mid = a_hi + 16, a_lo = a_hi + 32;
                const uint64_t w_hi = w0 + (uint64_t)(s * W_STAGE), w_mid = w_hi + 4, w_lo = lo0 + (uint64_t)(s * LO_STAGE);
                if (one) {
                    const uint32_t d = tmem + (uint32_t)(COL_SMALL + small * BN);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {        // 16 of k: 8 columns, 32 bytes
                        umma_bf16_ts(d, a_lo + 8 * k, w_mid + 2 * k, idesc, k > 0 || !first);
                        umma_bf16_ts(d, a_mid + 8 * k, w_lo + 2 * k, idesc, 1);
                        umma_bf16_ts(d, a_lo + 8 * k, w_hi + 2 * k, idesc, 1);
                        umma_bf16_ts(d, a_hi + 8 * k, w_lo + 2 * k, idesc, 1);
                        umma_bf16_ts(d, a_mid + 8 * k, w_mid + 2 * k, idesc, 1);
                        umma_bf16_ts(d, a_mid + 8 * k, w_hi + 2 * k, idesc, 1);
                        umma_bf16_ts(d, a_hi + 8 * k, w_mid + 2 * k, idesc, 1);
                    }
                }
                __syncwarp();
                ok = mbar_wait(&sm.acc_empty, (uint32_t)((it & 1) ^ 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (one) {
#pragma unroll
                    for (int k = 0; k < 2; ++k) umma_bf16_ts(tmem, a_hi + 8 * k, w_hi + 2 * k, idesc, k > 0);
                    umma_commit(&sm.empty[s]);
                    umma_commit(&sm.acc_full);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) atomicExch(g.status, 2);
    } else {
        const int quad = warp & 3, part = (warp - 2) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(quad * 32) << 16);
        const bool rows_here = g.M > quad * 32;          // a single row of tiles may leave whole warps without rows
        float* patch = sm.patch[warp - 2];
        const int total = ((int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0) * (end - begin);
        // This warp's share of a step's parts: 32 rows x 16 of k of A, and rows of W, eight at a time.  Lanes take eight of k of a
        // row; those that touch shared memory together are of rows r and r ^ 5, whose pieces lie in other banks both as they
        // came and as the parts lie (hi | mid).
        auto split = [&](int it) {
            const int s = it % STAGES;
            if (!mbar_wait(&sm.full[s], (uint32_t)(it / STAGES & 1))) return false;
            constexpr int EIGHTS = BN / 8, PIECES = (EIGHTS + FC_TEAM - 1) / FC_TEAM;
            constexpr bool EVEN = EIGHTS % FC_TEAM == 0;
            const int row = quad * 32 + lane, k4 = (part & 1) * 4, eight0 = (warp - 2) & (FC_TEAM - 1);
            const int r8 = lane >> 3 ^ (lane & 4 ? 5 : 0), j8 = lane & 3;
            float4 x[4], w[PIECES][2];                   // all are asked for before any is split
#pragma unroll
            for (int j = 0; j < 4; ++j)
                x[j] = *reinterpret_cast<const float4*>(sm.a[s] + row * FC_BK + (((k4 + j) ^ (row & 7)) << 2));
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                if (!EVEN && eight0 + i * FC_TEAM >= EIGHTS) continue;
                const float4* from = reinterpret_cast<const float4*>(sm.w[s]) + (8 * (eight0 + i * FC_TEAM) + r8) * 8;
                w[i][0] = from[(2 * j8) ^ r8], w[i][1] = from[(2 * j8 + 1) ^ r8];
            }
            if (rows_here) {
                uint32_t hi[8], mid[8], lo[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fc_parts(x[j].x, x[j].y, hi[2 * j], mid[2 * j], lo[2 * j]);
                    fc_parts(x[j].z, x[j].w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
                }
                const uint32_t at = lanes + (uint32_t)(COL_A + 48 * (it % (AHEAD + 1)) + 2 * k4);
                tmem_st_x8(at, hi);
                tmem_st_x8(at + 16, mid);
                tmem_st_x8(at + 32, lo);
            }
            __syncwarp();                                // a row's lanes have read it
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                if (!EVEN && eight0 + i * FC_TEAM >= EIGHTS) continue;
                const int wrow = 8 * (eight0 + i * FC_TEAM) + r8;
                uint4 hi, mid, lo;
                fc_parts(w[i][0].x, w[i][0].y, hi.x, mid.x, lo.x);
                fc_parts(w[i][0].z, w[i][0].w, hi.y, mid.y, lo.y);
                fc_parts(w[i][1].x, w[i][1].y, hi.z, mid.z, lo.z);
                fc_parts(w[i][1].z, w[i][1].w, hi.w, mid.w, lo.w);
                uint4* to = reinterpret_cast<uint4*>(sm.w[s]) + wrow * 8;
                to[j8 ^ r8] = hi;
                to[(4 + j8) ^ r8] = mid;
                reinterpret_cast<uint4*>(sm.w_lo[s])[wrow * 4 + (j8 ^ (r8 >> 1 & 3))] = lo;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.split[s]);
            return true;
        };
        const int team = part >> 1;
        int it = 0, run = 0;
        if (team < total) ok = split(team);
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            float2x sum[CW / 2];
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) sum[i] = 0ull;
            int run_end = begin + g.group;
            for (int st = begin; st < end; ++st, ++it) {
                if (it + AHEAD < total && team == (it & 1)) ok = split(it + AHEAD);
                ok = ok && mbar_wait(&sm.acc_full, (uint32_t)(it & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                auto add = [&](uint32_t column) {        // an accumulator's columns of this warp onto the sums
                    if (!rows_here) return;
                    uint32_t r[CW];
#pragma unroll
                    for (int c = 0; c < CW; c += 8) tmem_ld_x8_nowait(lanes + column + (uint32_t)(part * CW + c), r + c);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < CW / 2; ++i)
                        sum[i] = pair_add(sum[i], pair_of_floats(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])));
                };
                add(0u);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.acc_empty);
                if (st + 1 == run_end || st + 1 == end) {                        // a run is complete: its small products
                    add((uint32_t)(COL_SMALL + run % SMALL * BN));
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sm.small_empty[run % SMALL]);
                    ++run;
                }
                if (!CUT && st + 1 == run_end && st + 1 != end) {                // onto the runs before it
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
            if (!CUT && g.runs > 1) {
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
        static_assert(sizeof(sm.a) + sizeof(sm.w) + sizeof(sm.w_lo) >= FC_BM * BN * sizeof(float), "room for a run's sums");
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

template <int BN, int STAGES, bool CUT>
int launch_f32_tc(const FcArgs& g, int act, int sms, cudaStream_t s) {
    CUtensorMap map_a, map_w;
    if (!tensor_map_f32(&map_a, g.A, g.M, g.K, g.lda, FC_BM) || !tensor_map_f32(&map_w, g.W, g.N, g.K, g.ldw, BN)) return MU_ERR_LAUNCH;
    auto kernel = gemm_f32_tc_kernel<BN, STAGES, CUT>;
    const size_t smem = sizeof(FcSmem<BN, STAGES, CUT>) + 1024;
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
    auto kernel = gemm_f32_tc_kernel<BN, STAGES, true>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, runs);
    cfg.blockDim = dim3(FC_THREADS);
    cfg.dynamicSmemBytes = sizeof(FcSmem<BN, STAGES, true>) + 1024;
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
    // (columns of a tile, stages of the ring if it is cut and if not)
#define MU_FC_ALL(DO) DO(32, 8, 8) DO(64, 7, 6) DO(96, 6, 5) DO(128, 5, 4) DO(160, 4, 3)
    // The width, and whether to cut, by what the SM that ends last has to do, in microseconds: a step and a tile's end as below, a
    // launch 3, a further round of clusters 2.5 (fitted to one to three rounds of 192 to 768 of k; a cut tile's end, spread over its
    // cluster, is 0.6 of it; uncut tiles of 160 have three stages for three steps).  777 x 3,072 x 768 takes 37 us of 160, uncut,
    // and 48 of the next best form, 777 x 768 x 768 15.4 of 96, cut, and 20, 8 x 3,072 x 768 11.5 of 64, cut, and 16.
    int best = 0, best_cut = 0;
    double best_cost = 0.0;
    const struct { int width; double step, step_cut, end; } forms[5] = {
        {32, 0.50, 0.48, 1.4}, {64, 0.63, 0.56, 2.6}, {96, 0.75, 0.71, 4.2}, {128, 0.86, 0.79, 4.4}, {160, 1.20, 1.04, 7.3}};
    for (int i = 0; i < 5; ++i) {
        const int bn = forms[i].width;
        if (tile ? bn != tile : bn > 32 && bn - 32 >= N) continue;
        const long long tiles = m_tiles * ((N + bn - 1) / bn);
        for (int c = 0; c < 2; ++c) {
            if (c == 1 && (cut == 0 || runs == 1)) continue;
            long long at_once = sms;
            if (c == 1) {
#define MU_FC_CLUSTERS(BN, ST_CUT, ST) if (bn == BN) at_once = mu::fc_clusters<BN, ST_CUT>(runs);
                MU_FC_ALL(MU_FC_CLUSTERS)
#undef MU_FC_CLUSTERS
                if (at_once <= 0) continue;
            }
            const double rounds = (double)((tiles + at_once - 1) / at_once);
            double cost = c ? rounds * (group * forms[i].step_cut + 0.6 * forms[i].end + 2.5) + 0.5
                            : rounds * (steps * forms[i].step + forms[i].end) + 3.0;
            if (c == 1 && cut == 1) cost *= 1e-6;
            if (best == 0 || cost < best_cost) best = bn, best_cut = c, best_cost = cost;
        }
    }
#define MU_FC(BN, ST_CUT, ST)                                                                                          \
    if (best == BN)                                                                                                    \
        return best_cut ? mu::launch_f32_tc<BN, ST_CUT, true>(g, act, sms, s) : mu::launch_f32_tc<BN, ST, false>(g, act, sms, s);
    MU_FC_ALL(MU_FC)
#undef MU_FC
#undef MU_FC_ALL
    return MU_ERR_BAD_ARGUMENT;
}
