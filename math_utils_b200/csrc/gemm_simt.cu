// C[M, N] = act(A[M, K] . W[N, K]^T + bias[N]) (+ residual[M, N]) on CUDA cores.
//
// This is the 32-bit matrix product of the library in float32 multiply-adds (for
// short k and any shape; from 384 of k on gemm_f32_tc.cu has it) and also the
// any-shape fallback of the bfloat16 path.  Every output element is one
// running sum over k = 0..K-1 in order, whatever M is and wherever the row
// lies in the batch, so a row's result does not depend on what else is in the
// step.  The reference's counterpart is `apply` over matmulNT/matmulTiled
// (include/ai/LocalModel.hpp:1052-1126; include/ai/Kernels.hpp:184-207, 315-430).
//
// That is the first kernel, which takes any type, stride and size.  The second (gemm_f32_tile) takes float32 operands whose
// rows are whole 16-byte pieces: the 32-bit path's products up to k = 380.  Its sums are four, over the k of every fourth
// run of eight, added in order at the end: as independent of the rest of the step, and no less exact.  It is bound by the
// FMA pipes (2 m n k / 73 TFLOP/s) and next by how few warps share a scheduler: a small thread tile needs too many
// shared-memory reads, and the large one that needs few leaves two (80 rows) to four of them, which issue in 45 to 59 % of the
// cycles and wait for fixed latencies and the pipe otherwise, not for shared memory (50 to 66 % busy).  So a thread owns TM x 8 outputs
// (pairs of columns, fma.rn.f32x2: two FMAs an instruction, each rounded as its scalar form), and four groups of warps
// share every staged tile, each taking a quarter of its k.  Operands lie k-major in shared memory; the next 32 of k are on
// their way from global memory meanwhile.  Measured (B200, microseconds; the first kernel's in brackets): 777 x 3072 x 768 120
// (186), 777 x 768 x 3072 128 (313), 2048 x 4096 x 4096 1,705 (2,664; 40 TFLOP/s), 8 x 3072 x 768 17 (55).  Two blocks an
// SM up to 64 rows; a tile of 80 rows fills the registers of one, and is taken where it saves a wave (128 us against 196
// with 48 rows for 777 x 768 x 3072).
#include "common.cuh"

namespace mu {

constexpr int FT_BN = 64, FT_GROUPS = 4, FT_RUN = 8, FT_BK = FT_GROUPS * FT_RUN, FT_THREADS = 64 * FT_GROUPS;
constexpr int FT_PW = FT_BN + 4;                         // floats a row of W's stage, and of the sums handed over

template <int TM> constexpr size_t ft_smem() {
    return sizeof(float) * (2 * FT_BK * (8 * TM + 2 + FT_PW) > FT_GROUPS * 8 * TM * FT_PW ? 2 * FT_BK * (8 * TM + 2 + FT_PW)
                                                                                          : FT_GROUPS * 8 * TM * FT_PW);
}

// A block computes BM = 8 TM rows x 64 columns.  A group's 64 threads are 8 along m (row pairs 2 tm + 16 i) and 8 along n
// (column pairs 2 tn + 16 j), a warp 4 x 8.  Operands are read 8 bytes at a time: such a load, of four or eight different
// places, is one pass over the banks, where a 16-byte load takes four whatever its lanes share.  Column n of W's stage lies
// at (n + 2 (k & ~3)) mod 64, which spreads the transposing stores over all banks, as A's pitch does for its rows.
template <int TM>
__global__ void __launch_bounds__(FT_THREADS, TM <= 8 ? 2 : 1)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     const float* residual, float* C, int M, int N, int K, long long lda, long long ldw, long long ldc,
                     long long ldr, int act) {
    constexpr int BM = 8 * TM, PA = BM + 2, STAGE = FT_BK * (PA + FT_PW);
    constexpr int ROWS4 = 4 * (BM + FT_BN);              // 16-byte pieces of half a stage's k
    constexpr int LOADS = (2 * ROWS4 + FT_THREADS - 1) / FT_THREADS;
    extern __shared__ __align__(16) float ft_sm[];       // two stages of [k][BM + 2] | [k][68]; at the end the groups' sums
    const int tid = threadIdx.x, group = tid >> 6, tm = (tid & 63) >> 3, tn = tid & 7;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * FT_BN;
    float4 next[LOADS];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LOADS; ++i) {
            const int r = (tid + i * FT_THREADS) % ROWS4 >> 2, k = k0 + (tid + i * FT_THREADS) / ROWS4 * 16 + (tid & 3) * 4;
            next[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (tid + i * FT_THREADS >= 2 * ROWS4 || k >= K) continue;
            if (r < BM) {
                if (m0 + r < M) next[i] = *reinterpret_cast<const float4*>(A + (long long)(m0 + r) * lda + k);
            } else if (n0 + r - BM < N) {
                next[i] = *reinterpret_cast<const float4*>(W + (long long)(n0 + r - BM) * ldw + k);
            }
        }
    };
    auto lay = [&](int s) {
#pragma unroll
        for (int i = 0; i < LOADS; ++i) {
            const int r = (tid + i * FT_THREADS) % ROWS4 >> 2, k = (tid + i * FT_THREADS) / ROWS4 * 16 + (tid & 3) * 4;
            if (tid + i * FT_THREADS >= 2 * ROWS4) continue;
            const int pitch = r < BM ? PA : FT_PW;
            float* dst = ft_sm + s * STAGE + k * pitch + (r < BM ? r : FT_BK * PA + ((r - BM + 2 * k) & (FT_BN - 1)));
            dst[0] = next[i].x; dst[pitch] = next[i].y; dst[2 * pitch] = next[i].z; dst[3 * pitch] = next[i].w;
        }
    };
    float2x acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    const int steps = (K + FT_BK - 1) / FT_BK;
    fetch(0);
    lay(0);
    __syncthreads();
    for (int st = 0; st < steps; ++st) {
        if (st + 1 < steps) fetch((st + 1) * FT_BK);
        const float* sa = ft_sm + (st & 1) * STAGE + group * FT_RUN * PA + 2 * tm;
        const float* sw = ft_sm + (st & 1) * STAGE + FT_BK * PA + group * FT_RUN * FT_PW;
#pragma unroll
        for (int kk = 0; kk < FT_RUN; ++kk) {
            float2x w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                w[j] = *reinterpret_cast<const float2x*>(
                    sw + kk * FT_PW + ((2 * tn + 16 * j + 2 * (group * FT_RUN + (kk & 4))) & (FT_BN - 1)));
#pragma unroll
            for (int i = 0; i < TM; i += 2) {
                const float2 a = *reinterpret_cast<const float2*>(sa + kk * PA + 8 * i);
                const float2x lo = pair_of_floats(a.x, a.x), hi = pair_of_floats(a.y, a.y);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = pair_fma(lo, w[j], acc[i][j]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i + 1][j] = pair_fma(hi, w[j], acc[i + 1][j]);
            }
        }
        if (st + 1 < steps) lay((st + 1) & 1);           // (that buffer's readers passed the barrier of the step before)
        __syncthreads();
    }
    // the groups' sums meet in shared memory, and all threads finish the tile, four columns of a row at a time
    float* mine = ft_sm + (group * BM) * FT_PW + 2 * tn;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        float* row = mine + (2 * tm + 8 * (i & ~1) + (i & 1)) * FT_PW;
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float2x*>(row + 16 * j) = acc[i][j];
    }
    __syncthreads();
    const int n = n0 + (tid & 15) * 4;
    if (n >= N) return;
    float b4[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) b4[e] = bias && n + e < N ? bias[n + e] : 0.0f;
    const bool wide = n + 3 < N && ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
    for (int r = tid >> 4; r < BM && m0 + r < M; r += FT_THREADS / 16) {
        const float* src = ft_sm + r * FT_PW + (tid & 15) * 4;
        float4 sum = *reinterpret_cast<const float4*>(src);
#pragma unroll
        for (int g = 1; g < FT_GROUPS; ++g) {
            const float4 part = *reinterpret_cast<const float4*>(src + g * BM * FT_PW);
            sum.x += part.x; sum.y += part.y; sum.z += part.z; sum.w += part.w;
        }
        float v[4] = {sum.x, sum.y, sum.z, sum.w};
        const long long m = m0 + r;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[e] = apply_act(v[e] + b4[e], act);
            if (residual && n + e < N) v[e] += residual[m * ldr + n + e];
        }
        float* dst = C + m * ldc + n;
        if (wide) {
            *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < N) dst[e] = v[e];
        }
    }
}

// Rows a thread, hence the tile's height 16, 32 .. 80: the one whose last wave wastes least.  The SM that ends last has
// ceil(tiles / SMs) tiles behind it, each of its rows plus a fixed part worth some 12 of them.  (The height does not change
// a sum, so the choice may depend on M.)
inline int pick_rows(int M, int N, int sms) {
    int best = 2;
    long long best_cost = -1;
    for (int tm = 2; tm <= 10; tm += 2) {
        const long long tiles = (long long)((M + 8 * tm - 1) / (8 * tm)) * ((N + FT_BN - 1) / FT_BN);
        const long long cost = ((tiles + sms - 1) / sms) * (8 * tm + 12);
        if (best_cost < 0 || cost <= best_cost) best = tm, best_cost = cost;
    }
    return best;
}

template <int TM, typename... Args>
int launch_f32_tile(int M, int N, cudaStream_t s, Args... args) {
    const dim3 grid((N + FT_BN - 1) / FT_BN, (M + 8 * TM - 1) / (8 * TM));
    if (grid.y > 65535) return MU_ERR_UNSUPPORTED_SIZE;
    if (!allow_shared(reinterpret_cast<const void*>(gemm_f32_tile_kernel<TM>), ft_smem<TM>())) return MU_ERR_LAUNCH;
    prefer_shared_memory(reinterpret_cast<const void*>(gemm_f32_tile_kernel<TM>));          // room for two blocks an SM
    // (in plain stream order: started early, the blocks would be dealt into the room the kernel before has left, some of
    // them two to an SM while others stay idle)
    return launch_after(gemm_f32_tile_kernel<TM>, grid, dim3(FT_THREADS), ft_smem<TM>(), s, args...);
}

constexpr int SG_BM = 64, SG_BN = 64, SG_BK = 16, SG_THREADS = 256;

template <typename TA, typename TC>
__global__ void __launch_bounds__(SG_THREADS)
gemm_simt_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias,
                 const float* residual, TC* C, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, long long ldr, int act) {
    __shared__ float As[SG_BK][SG_BM + 4];
    __shared__ float Ws[SG_BK][SG_BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * SG_BM, n0 = blockIdx.x * SG_BN;
    const int tx = tid % 16, ty = tid / 16;          // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    // each thread loads 4 elements of A and 4 of W per k-block: row = tid / 4, k = (tid % 4) * 4 ..
    const int lr = tid / 4, lk = (tid % 4) * 4;
    for (int k0 = 0; k0 < K; k0 += SG_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int am = m0 + lr, wn = n0 + lr;
            As[lk + i][lr] = (am < M && k < K) ? to_float(A[(long long)am * lda + k]) : 0.0f;
            Ws[lk + i][lr] = (wn < N && k < K) ? to_float(W[(long long)wn * ldw + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < SG_BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            v = apply_act(v, act);
            if (residual) v += residual[(long long)m * ldr + n];
            C[(long long)m * ldc + n] = from_float<TC>(v);
        }
    }
}

}  // namespace mu

// in_bf16: A and W hold bfloat16 (else float32); out_bf16: C holds bfloat16 (else float32).
// residual (float32, leading dimension ldr) may be C itself when C is float32.
MU_EXPORT int mu_gemm_simt(const void* A, const void* W, const float* bias, const float* residual,
                           void* C, int M, int N, int K, long long lda, long long ldw,
                           long long ldc, long long ldr, int act, int in_bf16, int out_bf16,
                           void* stream) {
    if (M <= 0 || N <= 0) return MU_OK;
    if (K <= 0 || !A || !W || !C) return MU_ERR_BAD_ARGUMENT;
    if (lda < K || ldw < K || ldc < N || (residual && ldr < N)) return MU_ERR_BAD_ARGUMENT;
    dim3 grid((N + mu::SG_BN - 1) / mu::SG_BN, (M + mu::SG_BM - 1) / mu::SG_BM);
    if (grid.y > 65535) return MU_ERR_UNSUPPORTED_SIZE;
    cudaStream_t s = (cudaStream_t)stream;
    if (!in_bf16 && !out_bf16 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 &&
        ((uintptr_t)W & 15) == 0) {
        const int sms = mu::sm_count();
        if (sms <= 0) return MU_ERR_LAUNCH;
#define MU_TILE(TM)                                                                                                    \
    case TM:                                                                                                           \
        return mu::launch_f32_tile<TM>(M, N, s, (const float*)A, (const float*)W, bias, residual, (float*)C, M, N, K, lda, \
                                       ldw, ldc, ldr, act)
        switch (mu::pick_rows(M, N, sms)) {
            MU_TILE(2);
            MU_TILE(4);
            MU_TILE(6);
            MU_TILE(8);
            MU_TILE(10);
        }
#undef MU_TILE
    }
#define MU_LAUNCH(TA, TC)                                                                     \
    mu::gemm_simt_kernel<TA, TC><<<grid, mu::SG_THREADS, 0, s>>>(                              \
        (const TA*)A, (const TA*)W, bias, residual, (TC*)C, M, N, K, lda, ldw, ldc, ldr, act)
    if (in_bf16 && out_bf16) MU_LAUNCH(__nv_bfloat16, __nv_bfloat16);
    else if (in_bf16) MU_LAUNCH(__nv_bfloat16, float);
    else if (out_bf16) MU_LAUNCH(float, __nv_bfloat16);
    else MU_LAUNCH(float, float);
#undef MU_LAUNCH
    MU_CHECK_LAUNCH();
    return MU_OK;
}
