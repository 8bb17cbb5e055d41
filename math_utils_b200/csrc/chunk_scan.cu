// Prompt steps of the recurrences that write a matrix state per head without reading it first, chunk by chunk on tensor
// cores, with errors of the size that their token-by-token forms (linear_scan.cu, ssd.cu) have in float32 (cs_products):
//     S_t = a_t S_(t-1) + b_t k_t v_t^T,   o_t = scale S_t^T q_t (+ D v_t),
// a and b one number each per token and head.  Two mixers use it:
//   the matrix memory of xLSTM (gates given), with a normalizer n_t = a_t n_(t-1) + b_t k_t read out as scale n . q;
//   the state-space mixer (k = B, q = C, v = x, b = dt = softplus(raw + bias), a = exp(-exp(A_log) dt)).
//
// A sequence's tokens of the step are cut into chunks of 64.  With S the state before a chunk of n tokens and L_t the sum of
// log a over the chunk's tokens up to t,
//     o_t = exp(L_t) S^T q_t + sum_{s <= t} exp(L_t - L_s) b_s (q_t . k_s) v_s,
//     S'  = exp(L_(n-1)) S + sum_s exp(L_(n-1) - L_s) b_s k_s v_s^T,
// so all chunks of all sequences and heads work at once but for the states between them.  Three launches: chunk_sums (a
// chunk's own sum, to scratch), chunk_states (walks over a sequence's chunks entry by entry, leaves each one's starting
// state, moves the slot's state on), chunk_outputs.
//
// Products are mma.sync.m16n8k8 on TF32 operands, every float32 operand as two terms (x rounded to TF32, and the rest so
// rounded: 22 bits) in three products, so that an element acts to some 2^-22; two steps' products at a time are summed apart
// and added to the running sum by ordinary additions (cs_products).  L is summed
// in float64 and kept as two floats, since exp(L_t - L_s) of neighbours takes the difference of two large numbers.
//
// What bounds it: dependent products of three warps a scheduler, which issue in half of the cycles and wait for fixed latencies
// and the pipe otherwise; the token-by-token forms are bound by the chain of 1,024 tokens a sequence.  Measured (B200,
// 2 x 1,024 tokens): the state-space layer of 16 heads of 128 x 64 by key 365 us token by token, 123 in chunks, the matrix memory's
// of 8 heads of 128 x 128 with normalizer over 2,018 tokens 265 and 146; one sequence of some 300
// tokens gains half, wide batches of the matrix memory nothing (matrix_lstm.py has the rule).
#include "common.cuh"

#include <math.h>

namespace mu {

constexpr int CS_TOK = 64, CS_COLS = 64, CS_THREADS = 256;
constexpr int CS_PP = CS_TOK + 8;                             // a row of the weights in shared memory: 8 banks apart

// Where a chunk's part of the scratch lies (as lightning_prompt.cu): no two chunks of a step share a place.
__device__ __forceinline__ long long cs_place(int flat0, int s, int first) { return first / CS_TOK + s + (flat0 - first) / CS_TOK; }

struct ChunkArgs {
    const float* q;              // [T] rows ld apart; head h's slice starts at (h / heads_per_key) * dk
    const float* k;
    const float* v;              // head h's slice starts at h * dv
    long long ld;
    const float4* gates;         // [T][heads] (a, b, -, -); or null, and then:
    const void* dt_raw;          // [T] rows lddt apart, one per head
    long long lddt;
    const float* dt_bias;
    const float* a_log;
    const float* skip;           // D per head, or null
    const int* tiles;            // [n_tiles][2]: first flat token, count <= 64
    const int* tok_seq;
    const int* seq_first;
    const int* seq_slots;
    int n_heads, heads_per_key, dk, dv;
    float scale;
    float* sums;                 // [places][heads][dk * dv], in the order of the state
    float* norm_sums;            // [places][heads][dk], or null: no normalizer
    float* decays;               // [places][heads]
    float* state;                // a slot's S: heads x [dv][dk], or [dk][dv] (BY_KEY); the normalizers heads x [dk] behind
    long long state_stride, state_offset;
    float* out;                  // [T] rows ldo apart
    long long ldo;
    float* norm_out;             // [T][heads]
};

__device__ __forceinline__ void cs_copy16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cs_copy8(float* dst, const float* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(there ? 8 : 0) : "memory");
}
// x rounded to TF32 (to nearest, ties away from zero) as two integer operations: the conversion instruction gives the same bits at
// a fraction of their rate (with the rest's conversion as it was: state space 140 -> 132 us, matrix memory 161 -> 153).  A NaN
// of all ones comes out as zero; what that leaves of it is NaN, which the instruction keeps.
__device__ __forceinline__ uint32_t cs_tf32(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
// x as two TF32 terms: the rounded value, and what the rounding left.
__device__ __forceinline__ void cs_split(float x, uint32_t& hi, uint32_t& lo) {
    hi = cs_tf32(x);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(x - __uint_as_float(hi)));
}
__device__ __forceinline__ void cs_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// What a sum that the tensor cores made has lost, as a share of it: they cut it off after 24 bits, half of the last one on
// average over mantissas (2^-24 (1 - 1/2) / ln 2).
constexpr float CS_CUT = 4.3e-8f;

// x as two TF32 terms that are together longer than x by that share.
__device__ __forceinline__ void cs_split_more(float x, uint32_t& hi, uint32_t& lo) {
    hi = cs_tf32(x);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(fmaf(x, CS_CUT, x - __uint_as_float(hi))));
}

// d += the product over two steps of 8 (a: their two-term fragments; b: slots tig, tig + 4 of each).  Six products go into
// a sum of their own, the small ones first, which joins d by an ordinary addition: the tensor cores cut a running sum off
// where an addition rounds it, and what the cut takes on average the right operand brings along.  Measured against float64
// over the layers' sizes (of the outputs): 8 heads of 128 x 128 1.47e-7, token by token in float32 1.64e-7, without
// the share 1.87e-7; 16 heads of 64 x 128 by key 0.85e-7, 0.77e-7 and 1.03e-7; the states 1.0e-7, 1.5e-7 and 1.2e-7.  (A second
// sum for the products of the large terms: 1.55e-7 and 0.88e-7; the product of the two small terms as well: 1.42e-7 and
// 0.83e-7 in 6 % more time.)
__device__ __forceinline__ void cs_products(float (&d)[4], const uint32_t (&ah)[2][4], const uint32_t (&al)[2][4], float b0,
                                            float b1, float b2, float b3) {
    uint32_t h0, l0, h1, l1, h2, l2, h3, l3;
    cs_split_more(b0, h0, l0);
    cs_split_more(b1, h1, l1);
    cs_split_more(b2, h2, l2);
    cs_split_more(b3, h3, l3);
    float t[4] = {};
    cs_mma(t, al[0], h0, h1);
    cs_mma(t, ah[0], l0, l1);
    cs_mma(t, al[1], h2, h3);
    cs_mma(t, ah[1], l2, l3);
    cs_mma(t, ah[0], h0, h1);
    cs_mma(t, ah[1], h2, h3);
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] += t[i];
}

// Rows flat0 .. flat0 + count - 1 of `src` (row stride ld), `width` floats of each, to [64][pitch]; zeros for the rows past
// the chunk's and for the floats past the width up to `padded` (both multiples of 4).
__device__ __forceinline__ void cs_stage(float* dst, int pitch, const float* src, long long ld, int flat0, int count, int width,
                                         int padded) {
    const int pieces = padded >> 2;
    for (int i = threadIdx.x; i < CS_TOK * pieces; i += CS_THREADS) {
        const int r = i / pieces, c = 4 * (i - r * pieces);
        const bool there = r < count && c < width;
        cs_copy16(dst + r * pitch + c, there ? src + (long long)(flat0 + r) * ld + c : src, there);
    }
}

// One warp: log a and b of the chunk's tokens, L as two floats (from the chunk's end on: its last value, b = 0).
template <typename TD>
__device__ __forceinline__ void cs_gates(const ChunkArgs& a, int h, int flat0, int count, float* l_hi, float* l_lo, float* b) {
    const int lane = threadIdx.x & 31;
    double run[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int t = 2 * lane + j;
        float la = 0.0f, take = 0.0f;
        if (t < count) {
            if (a.gates) {
                const float4 g = a.gates[(long long)(flat0 + t) * a.n_heads + h];
                la = logf(g.x), take = g.y;
            } else {
                const TD* raw = reinterpret_cast<const TD*>(a.dt_raw);
                take = softplus(to_float(raw[(long long)(flat0 + t) * a.lddt + h]) + a.dt_bias[h]);
                la = -expf(a.a_log[h]) * take;
            }
            if (la < -200.0f) la = -200.0f;                  // exp of it is zero either way, and sums of it stay finite
        }
        b[t] = take;
        run[j] = la;
    }
    run[1] += run[0];
    double upto = run[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += other;
    }
    const double before = upto - run[1];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const double L = before + run[j];
        const float hi = (float)L;
        l_hi[2 * lane + j] = hi;
        l_lo[2 * lane + j] = (float)(L - (double)hi);
    }
}

// The sum of a chunk in the order of the state: out[m][n] = sum_s A[s][m] (w_s B[s][n]) with (A, B) = (v, k), or (k, v) where
// the state lies by key (BY_KEY).  A warp takes 16 rows m at a time and 64 columns n of them.
template <bool BY_KEY, typename TD>
__global__ void __launch_bounds__(CS_THREADS)
chunk_sums_kernel(const __grid_constant__ ChunkArgs a) {
    extern __shared__ __align__(16) float cs_sm[];
    __shared__ float l_hi[CS_TOK], l_lo[CS_TOK], b[CS_TOK], w[CS_TOK];
    const int M = BY_KEY ? a.dk : a.dv, N = BY_KEY ? a.dv : a.dk;
    const int ap = (M + 31) / 32 * 32 + 8, bp = (N + 63) / 64 * 64 + 8;        // 8 banks a row apart
    float* As = cs_sm;
    float* Bs = As + CS_TOK * ap;
    pdl_trigger();
    pdl_wait();
    const int flat0 = a.tiles[2 * blockIdx.x], count = min(a.tiles[2 * blockIdx.x + 1], CS_TOK), h = blockIdx.y;
    const int s = a.tok_seq[flat0];
    const long long at = cs_place(flat0, s, a.seq_first[s]) * a.n_heads + h;
    const float* ks = a.k + (long long)(h / a.heads_per_key) * a.dk;
    const float* vs = a.v + (long long)h * a.dv;
    cs_stage(As, ap, BY_KEY ? ks : vs, a.ld, flat0, count, M, M);
    cs_stage(Bs, bp, BY_KEY ? vs : ks, a.ld, flat0, count, N, (N + 7) / 8 * 8);
    copy_async_commit();
    if (threadIdx.x < 32) cs_gates<TD>(a, h, flat0, count, l_hi, l_lo, b);
    __syncthreads();
    if (threadIdx.x < CS_TOK) {
        const int t = threadIdx.x;
        w[t] = expf((l_hi[CS_TOK - 1] - l_hi[t]) + (l_lo[CS_TOK - 1] - l_lo[t])) * b[t];
        if (t == 0) a.decays[at] = expf(l_hi[CS_TOK - 1] + l_lo[CS_TOK - 1]);
    }
    copy_async_wait<0>();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    float* dst = a.sums + at * (long long)a.dk * a.dv;
    for (int item = warp; item < (M + 15) / 16 * ((N + 63) / 64); item += CS_THREADS / 32) {
        const int m0 = item % ((M + 15) / 16) * 16, n0 = item / ((M + 15) / 16) * 64;
        float sum[8][4] = {};
        const int tiles = min(8, (N - n0 + 7) / 8);
        for (int t0 = 0; t0 < count; t0 += 16) {              // (rows past the chunk's end are zero)
            uint32_t ah[2][4], al[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int s0 = t0 + 8 * u + tig, s1 = s0 + 4;
                cs_split(As[s0 * ap + m0 + gid] * w[s0], ah[u][0], al[u][0]);
                cs_split(As[s0 * ap + m0 + gid + 8] * w[s0], ah[u][1], al[u][1]);
                cs_split(As[s1 * ap + m0 + gid] * w[s1], ah[u][2], al[u][2]);
                cs_split(As[s1 * ap + m0 + gid + 8] * w[s1], ah[u][3], al[u][3]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (j >= tiles) break;
                const float* src = Bs + (t0 + tig) * bp + n0 + 8 * j + gid;
                cs_products(sum[j], ah, al, src[0], src[4 * bp], src[8 * bp], src[12 * bp]);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + 8 * j + 2 * tig;
            if (n >= N) continue;                             // (N is a multiple of 4: a pair is in or out)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int m = m0 + gid + 8 * r;
                if (m < M)
                    *reinterpret_cast<float2*>(dst + (long long)m * N + n) =
                        make_float2(sum[j][2 * r], sum[j][2 * r + 1]);
            }
        }
    }
    if (a.norm_sums) {                                        // (only with the state by value: Bs holds the keys)
        for (int n = threadIdx.x; n < a.dk; n += CS_THREADS) {
            float sum = 0.0f;
            for (int t = 0; t < count; ++t) sum = fmaf(w[t], Bs[t * bp + n], sum);
            a.norm_sums[at * a.dk + n] = sum;
        }
    }
}

constexpr int CS_AHEAD = 8;      // chunks whose sums are on their way at once

__global__ void __launch_bounds__(128)
chunk_states_kernel(const __grid_constant__ ChunkArgs a) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.z, h = blockIdx.y, entries = a.dk * a.dv;
    const int i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    const bool norm = i >= entries;                           // the entries behind S are the normalizer's
    if (i >= entries + (a.norm_sums ? a.dk : 0)) return;
    const int first = a.seq_first[s], count = a.seq_first[s + 1] - first;
    if (count <= 0) return;
    const int chunks = (count + CS_TOK - 1) / CS_TOK, per = norm ? a.dk : entries, in = norm ? i - entries : i;
    const long long place = cs_place(first, s, first) * a.n_heads + h, step = (long long)a.n_heads * per;
    float* u = (norm ? a.norm_sums : a.sums) + place * per + in;
    const float* decay = a.decays + place;
    float4* kept = reinterpret_cast<float4*>(a.state + (long long)a.seq_slots[s] * a.state_stride + a.state_offset +
                                             (norm ? (long long)a.n_heads * entries : 0) + (long long)h * per + in);
    float4 S = *kept;
    for (int c0 = 0; c0 < chunks; c0 += CS_AHEAD) {
        float4 x[CS_AHEAD];
        float d[CS_AHEAD];
#pragma unroll
        for (int j = 0; j < CS_AHEAD; ++j) {
            const int c = min(c0 + j, chunks - 1);
            x[j] = *reinterpret_cast<const float4*>(u + c * step);
            d[j] = decay[(long long)c * a.n_heads];
        }
#pragma unroll
        for (int j = 0; j < CS_AHEAD; ++j) {
            if (c0 + j >= chunks) break;
            *reinterpret_cast<float4*>(u + (c0 + j) * step) = S;
            S = make_float4(fmaf(d[j], S.x, x[j].x), fmaf(d[j], S.y, x[j].y), fmaf(d[j], S.z, x[j].z), fmaf(d[j], S.w, x[j].w));
        }
    }
    *kept = S;
}

// A block takes a chunk, a head and 64 value columns; a warp 16 tokens and 32 of the columns.  The two warps of the same tokens
// make the weights of half of their keys each and find the rest in shared memory (each made all of them before: state space
// 132 -> 123 us, matrix memory 153 -> 146).
// Along dk the lanes take
// their entries four at a time (lane tig's k slots of two steps of 8 are entries 4 tig .. 4 tig + 3 of 16), so queries come
// as 16-byte loads from global memory and keys and states by value as 16-byte loads from shared memory.
template <bool BY_KEY, typename TD>
__global__ void __launch_bounds__(CS_THREADS, 2)
chunk_outputs_kernel(const __grid_constant__ ChunkArgs a) {
    constexpr int VP = CS_COLS + 4, SP = CS_COLS + 2;          // (2 VP and 4 SP are 8 banks apart)
    extern __shared__ __align__(16) float cs_sm[];
    __shared__ float l_hi[CS_TOK], l_lo[CS_TOK], b[CS_TOK];
    const int kp = (a.dk + 31) / 32 * 32 + 16;
    float* Ks = cs_sm;                                         // [64 tokens][kp]
    float* Vs = Ks + CS_TOK * kp;                              // [64 tokens][VP]
    float* Ps = Vs + CS_TOK * VP;                              // [64 tokens][PP] weights of the keys
    float* Ss = Ps + CS_TOK * CS_PP;                           // [64 columns][kp], or by key [dk][SP]
    pdl_trigger();
    pdl_wait();
    const int flat0 = a.tiles[2 * blockIdx.x], count = min(a.tiles[2 * blockIdx.x + 1], CS_TOK), h = blockIdx.y;
    const int col0 = blockIdx.z * CS_COLS, cols = min(CS_COLS, a.dv - col0), dk = a.dk;
    const int s = a.tok_seq[flat0];
    const long long at = cs_place(flat0, s, a.seq_first[s]) * a.n_heads + h;
    const int key_at = h / a.heads_per_key * dk;
    const float* S = a.sums + at * (long long)dk * a.dv;
    cs_stage(Ks, kp, a.k + key_at, a.ld, flat0, count, dk, dk);
    cs_stage(Vs, VP, a.v + (long long)h * a.dv + col0, a.ld, flat0, count, cols, CS_COLS);
    if (BY_KEY) {
        for (int i = threadIdx.x; i < dk * (CS_COLS / 2); i += CS_THREADS) {
            const int r = i / (CS_COLS / 2), c = i % (CS_COLS / 2) * 2;
            cs_copy8(Ss + r * SP + c, c < cols ? S + (long long)r * a.dv + col0 + c : S, c < cols);
        }
    } else {
        for (int i = threadIdx.x; i < CS_COLS * (dk / 4); i += CS_THREADS) {
            const int r = i / (dk / 4), c = (i - r * (dk / 4)) * 4;
            cs_copy16(Ss + r * kp + c, r < cols ? S + (long long)(col0 + r) * dk + c : S, r < cols);
        }
    }
    copy_async_commit();
    if (threadIdx.x < 32) cs_gates<TD>(a, h, flat0, count, l_hi, l_lo, b);
    copy_async_wait<0>();
    __syncthreads();
    const int warp = (threadIdx.x >> 5) & 3, half0 = (threadIdx.x >> 7) * 32;
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const bool norm = a.norm_sums != nullptr && col0 == 0 && half0 == 0;
    const bool mine = warp * 16 < count;
    // The last sixteen keys of a warp are its own tokens: those after a token have the weight zero, which does not keep an
    // infinite or NaN value out of a product.  With such a value among them they are added key by key.
    float odd = 0.0f;                                          // NaN from the first value that is not finite on
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(Vs + (warp * 16 + 4 * i + (lane >> 3)) * VP + half0 + 4 * (lane & 7));
        odd = fmaf(x.x, 0.0f, fmaf(x.y, 0.0f, fmaf(x.z, 0.0f, fmaf(x.w, 0.0f, odd))));
    }
    const bool plain = !__any_sync(0xffffffffu, isnan(odd));
    const int t0 = warp * 16 + gid, t1 = t0 + 8;               // this thread's two tokens
    const float* q0 = a.q + (long long)(flat0 + min(t0, count - 1)) * a.ld + key_at + 4 * tig;
    const float* q1 = a.q + (long long)(flat0 + min(t1, count - 1)) * a.ld + key_at + 4 * tig;
    const float* nrow = norm ? a.norm_sums + at * dk + 4 * tig : q0;
    const int key_tiles = 2 * (warp + 1), own_tiles = warp + 1;         // runs of 8 keys that these tokens see, and this warp's
    const int own0 = half0 ? 8 * own_tiles : 0;                // the first of its keys
    float o[4][4] = {}, w[CS_TOK / 16][4] = {}, den0 = 0.0f, den1 = 0.0f;
    float4 x0 = *reinterpret_cast<const float4*>(q0), x1 = *reinterpret_cast<const float4*>(q1);
    float4 nv = *reinterpret_cast<const float4*>(nrow);
    for (int k0 = 0; mine && k0 < dk; k0 += 16) {
        const float4 c0 = x0, c1 = x1, cn = nv;
        const int next = k0 + 16 < dk ? k0 + 16 : k0;
        x0 = *reinterpret_cast<const float4*>(q0 + next);
        x1 = *reinterpret_cast<const float4*>(q1 + next);
        nv = *reinterpret_cast<const float4*>(nrow + next);
        uint32_t ah[2][4], al[2][4];
        cs_split(c0.x, ah[0][0], al[0][0]);
        cs_split(c1.x, ah[0][1], al[0][1]);
        cs_split(c0.y, ah[0][2], al[0][2]);
        cs_split(c1.y, ah[0][3], al[0][3]);
        cs_split(c0.z, ah[1][0], al[1][0]);
        cs_split(c1.z, ah[1][1], al[1][1]);
        cs_split(c0.w, ah[1][2], al[1][2]);
        cs_split(c1.w, ah[1][3], al[1][3]);
        if (norm) {
            den0 += c0.x * cn.x + c0.y * cn.y + c0.z * cn.z + c0.w * cn.w;
            den1 += c1.x * cn.x + c1.y * cn.y + c1.z * cn.z + c1.w * cn.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 f;
            if (BY_KEY) {
                const float* src = Ss + (k0 + 4 * tig) * SP + half0 + 8 * j + gid;
                f = make_float4(src[0], src[SP], src[2 * SP], src[3 * SP]);
            } else {
                f = *reinterpret_cast<const float4*>(Ss + (half0 + 8 * j + gid) * kp + k0 + 4 * tig);
            }
            cs_products(o[j], ah, al, f.x, f.y, f.z, f.w);
        }
#pragma unroll
        for (int j = 0; j < CS_TOK / 16; ++j) {
            if (j >= own_tiles) break;
            const float4 f = *reinterpret_cast<const float4*>(Ks + (own0 + 8 * j + gid) * kp + k0 + 4 * tig);
            cs_products(w[j], ah, al, f.x, f.y, f.z, f.w);
        }
    }
    const float h0 = l_hi[t0], e0 = l_lo[t0], h1 = l_hi[t1], e1 = l_lo[t1];
    const float f0 = expf(h0 + e0), f1 = expf(h1 + e1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        o[j][0] *= f0, o[j][1] *= f0;
        o[j][2] *= f1, o[j][3] *= f1;
    }
    den0 *= f0, den1 *= f1;
    if (mine) {
#pragma unroll
        for (int j = 0; j < CS_TOK / 16; ++j) {
            if (j >= own_tiles) break;
            const int s0 = own0 + 8 * j + 2 * tig, s1 = s0 + 1;
            const float (&x)[4] = w[j];
            const float p0 = s0 <= t0 ? x[0] * (expf((h0 - l_hi[s0]) + (e0 - l_lo[s0])) * b[s0]) : 0.0f;
            const float p1 = s1 <= t0 ? x[1] * (expf((h0 - l_hi[s1]) + (e0 - l_lo[s1])) * b[s1]) : 0.0f;
            const float p2 = s0 <= t1 ? x[2] * (expf((h1 - l_hi[s0]) + (e1 - l_lo[s0])) * b[s0]) : 0.0f;
            const float p3 = s1 <= t1 ? x[3] * (expf((h1 - l_hi[s1]) + (e1 - l_lo[s1])) * b[s1]) : 0.0f;
            *reinterpret_cast<float2*>(Ps + t0 * CS_PP + s0) = make_float2(p0, p1);
            *reinterpret_cast<float2*>(Ps + t1 * CS_PP + s0) = make_float2(p2, p3);
        }
    }
    __syncthreads();
    if (!mine || half0 >= cols) return;
#pragma unroll
    for (int n = 0; n < CS_TOK / 8; n += 2) {
        if (n >= key_tiles) break;
        uint32_t ph[2][4], pl[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            // a pair of keys a lane: its slots of this step are keys 2 tig and 2 tig + 1 of the eight
            const float2 pa = *reinterpret_cast<const float2*>(Ps + t0 * CS_PP + 8 * (n + u) + 2 * tig);
            const float2 pb = *reinterpret_cast<const float2*>(Ps + t1 * CS_PP + 8 * (n + u) + 2 * tig);
            den0 += pa.x + pa.y;
            den1 += pb.x + pb.y;
            cs_split(pa.x, ph[u][0], pl[u][0]);
            cs_split(pb.x, ph[u][1], pl[u][1]);
            cs_split(pa.y, ph[u][2], pl[u][2]);
            cs_split(pb.y, ph[u][3], pl[u][3]);
        }
        if (plain || n + 2 < key_tiles) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float* src = Vs + (8 * n + 2 * tig) * VP + half0 + 8 * j + gid;
                cs_products(o[j], ph, pl, src[0], src[VP], src[8 * VP], src[9 * VP]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {                      // key by key, seen keys alone
                const int s = 8 * n + i, u = i >> 3, from = (lane & ~3) | ((i & 7) >> 1), f = 2 * (i & 1);
                const float p = __uint_as_float(ph[u][f]) + __uint_as_float(pl[u][f]);
                const float r = __uint_as_float(ph[u][f + 1]) + __uint_as_float(pl[u][f + 1]);
                const float p0 = __shfl_sync(0xffffffffu, p, from), p1 = __shfl_sync(0xffffffffu, r, from);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float* src = Vs + s * VP + half0 + 8 * j + 2 * tig;
                    if (s <= t0) o[j][0] = fmaf(p0, src[0], o[j][0]), o[j][1] = fmaf(p0, src[1], o[j][1]);
                    if (s <= t1) o[j][2] = fmaf(p1, src[0], o[j][2]), o[j][3] = fmaf(p1, src[1], o[j][3]);
                }
            }
        }
    }
    const float d_skip = a.skip ? a.skip[h] : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int c = half0 + 8 * j + 2 * tig;
        if (c >= cols) continue;                                // (cols is a multiple of 4)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = r ? t1 : t0;
            if (t >= count) continue;
            float y0 = a.scale * o[j][2 * r], y1 = a.scale * o[j][2 * r + 1];
            if (a.skip) y0 = fmaf(d_skip, Vs[t * VP + c], y0), y1 = fmaf(d_skip, Vs[t * VP + c + 1], y1);
            *reinterpret_cast<float2*>(a.out + (long long)(flat0 + t) * a.ldo + (long long)h * a.dv + col0 + c) = make_float2(y0, y1);
        }
    }
    if (norm) {
#pragma unroll
        for (int o2 = 1; o2 < 4; o2 <<= 1) {
            den0 += __shfl_xor_sync(0xffffffffu, den0, o2);
            den1 += __shfl_xor_sync(0xffffffffu, den1, o2);
        }
        if (tig == 0) {
            if (t0 < count) a.norm_out[(long long)(flat0 + t0) * a.n_heads + h] = a.scale * den0;
            if (t1 < count) a.norm_out[(long long)(flat0 + t1) * a.n_heads + h] = a.scale * den1;
        }
    }
}

template <bool BY_KEY, typename TD>
static int launch_chunks(const ChunkArgs& a, int n_tiles, int n_seqs, cudaStream_t s) {
    const int M = BY_KEY ? a.dk : a.dv, N = BY_KEY ? a.dv : a.dk;
    const size_t smem1 = sizeof(float) * CS_TOK * ((M + 31) / 32 * 32 + 8 + (N + 63) / 64 * 64 + 8);
    const int kp = (a.dk + 31) / 32 * 32 + 16;
    const size_t smem3 = sizeof(float) * (CS_TOK * kp + CS_TOK * (CS_COLS + 4) + CS_TOK * CS_PP + (BY_KEY ? a.dk * (CS_COLS + 2) : CS_COLS * kp));
    auto k1 = chunk_sums_kernel<BY_KEY, TD>;
    auto k3 = chunk_outputs_kernel<BY_KEY, TD>;
    if (!allow_shared((const void*)k1, 140 * 1024) || !allow_shared((const void*)k3, 112 * 1024) || smem1 > 140 * 1024 ||
        smem3 > 112 * 1024)
        return MU_ERR_LAUNCH;
    prefer_shared_memory((const void*)k1);
    prefer_shared_memory((const void*)k3);
    if (int e = launch_pdl(k1, dim3(n_tiles, a.n_heads), dim3(CS_THREADS), smem1, s, 1, a)) return e;
    const int entries = a.dk * a.dv + (a.norm_sums ? a.dk : 0);
    if (int e = launch_pdl(chunk_states_kernel, dim3((entries / 4 + 127) / 128, a.n_heads, n_seqs), dim3(128), 0, s, 1, a)) return e;
    return launch_pdl(k3, dim3(n_tiles, a.n_heads, (a.dv + CS_COLS - 1) / CS_COLS), dim3(CS_THREADS), smem3, s, 1, a);
}

}  // namespace mu

// Whether the chunked form takes these sizes: keys in steps of 16 up to 128 (queries are read, and a chunk's keys and states
// staged, in such steps), values in steps of 4 up to 256 (whole 16-byte pieces; a chunk's staged rows fit).
MU_EXPORT int mu_chunk_scan_fits(int dk, int dv) { return dk >= 16 && dk <= 128 && dk % 16 == 0 && dv >= 4 && dv <= 256 && dv % 4 == 0; }

// Floats of scratch for a step of n_tokens tokens of n_seqs sequences.
MU_EXPORT long long mu_chunk_scan_scratch(int n_tokens, int n_seqs, int n_heads, int dk, int dv) {
    return ((long long)n_tokens / mu::CS_TOK + n_seqs + 1) * n_heads * ((long long)dk * dv + dk + 4);
}

// As mu_linear_scan with gates per token and head ([T][heads][4] = (a, b, -, -)), for steps of many tokens.  tiles:
// [n_tiles][2] = (first flat token, count <= 64), every sequence cut from its first token of the step on.
MU_EXPORT int mu_linear_scan_chunks(const float* q, const float* k, const float* v, long long ld, const float* gates,
                                    const int* tiles, int n_tiles, const int* tok_seq, int n_tokens, int n_seqs, int n_heads,
                                    int dk, int dv, float scale, const int* seq_first, const int* seq_slots, float* scratch,
                                    float* state, long long state_stride, long long state_offset, float* out, long long ldo,
                                    float* norm_out, void* stream) {
    if (n_tiles <= 0 || n_seqs <= 0) return MU_OK;
    if (!q || !k || !v || !gates || !tiles || !tok_seq || !seq_first || !seq_slots || !scratch || !state || !out || n_heads <= 0)
        return MU_ERR_BAD_ARGUMENT;
    if (!mu_chunk_scan_fits(dk, dv) || n_heads > 65535 || n_seqs > 65535) return MU_ERR_UNSUPPORTED_SIZE;
    if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)gates | (uintptr_t)scratch | (uintptr_t)state) & 15 ||
        ((uintptr_t)out & 7) || ld % 4 || ldo % 2 || state_stride % 4 || state_offset % 4)
        return MU_ERR_ALIGNMENT;
    mu::ChunkArgs a = {};
    const long long places = (long long)n_tokens / mu::CS_TOK + n_seqs + 1;
    a.q = q, a.k = k, a.v = v, a.ld = ld, a.gates = (const float4*)gates;
    a.tiles = tiles, a.tok_seq = tok_seq, a.seq_first = seq_first, a.seq_slots = seq_slots;
    a.n_heads = n_heads, a.heads_per_key = 1, a.dk = dk, a.dv = dv, a.scale = scale;
    a.sums = scratch, a.decays = scratch + places * n_heads * ((long long)dk * dv + dk);
    a.norm_sums = norm_out ? scratch + places * n_heads * (long long)dk * dv : nullptr;
    a.state = state, a.state_stride = state_stride, a.state_offset = state_offset, a.out = out, a.ldo = ldo, a.norm_out = norm_out;
    return mu::launch_chunks<false, float>(a, n_tiles, n_seqs, (cudaStream_t)stream);
}

// As mu_ssd_scan, for steps of many tokens (tiles as above).
MU_EXPORT int mu_ssd_scan_chunks(const float* xbc, int channels, const void* dt_raw, long long lddt, int dt_bf16,
                                 const float* dt_bias, const float* a_log, const float* skip, const int* tiles, int n_tiles,
                                 const int* tok_seq, int n_tokens, int n_seqs, int n_heads, int P, int N, int groups,
                                 const int* seq_first, const int* seq_slots, float* scratch, float* state, long long state_stride,
                                 long long state_offset, float* y, void* stream) {
    if (n_tiles <= 0 || n_seqs <= 0) return MU_OK;
    if (!xbc || !dt_raw || !dt_bias || !a_log || !skip || !tiles || !tok_seq || !seq_first || !seq_slots || !scratch || !state ||
        !y || n_heads <= 0 || groups <= 0 || n_heads % groups || channels < n_heads * P + 2 * groups * N)
        return MU_ERR_BAD_ARGUMENT;
    if (!mu_chunk_scan_fits(N, P) || n_heads > 65535 || n_seqs > 65535) return MU_ERR_UNSUPPORTED_SIZE;
    const int inner = n_heads * P;
    if (((uintptr_t)xbc | (uintptr_t)scratch | (uintptr_t)state) & 15 || ((uintptr_t)y & 7) || channels % 4 || inner % 4 ||
        state_stride % 4 || state_offset % 4)
        return MU_ERR_ALIGNMENT;
    mu::ChunkArgs a = {};
    const long long places = (long long)n_tokens / mu::CS_TOK + n_seqs + 1;
    a.q = xbc + inner + groups * N, a.k = xbc + inner, a.v = xbc, a.ld = channels;
    a.dt_raw = dt_raw, a.lddt = lddt, a.dt_bias = dt_bias, a.a_log = a_log, a.skip = skip;
    a.tiles = tiles, a.tok_seq = tok_seq, a.seq_first = seq_first, a.seq_slots = seq_slots;
    a.n_heads = n_heads, a.heads_per_key = n_heads / groups, a.dk = N, a.dv = P, a.scale = 1.0f;
    a.sums = scratch, a.decays = scratch + places * n_heads * ((long long)N * P + N);
    a.state = state, a.state_stride = state_stride, a.state_offset = state_offset, a.out = y, a.ldo = inner;
    return dt_bf16 ? mu::launch_chunks<true, __nv_bfloat16>(a, n_tiles, n_seqs, (cudaStream_t)stream)
                   : mu::launch_chunks<true, float>(a, n_tiles, n_seqs, (cudaStream_t)stream);
}
