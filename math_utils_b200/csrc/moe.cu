// A feed-forward of routed experts: router, grouping of (token, expert) pairs by expert, the experts'
// products over each expert's rows, and the weighted sum per token.  Nothing is read back by the host,
// so a step with these kernels can be recorded in a CUDA graph: grids are sized for the worst case and
// blocks without work leave at once.
//
// mu_moe_route    z = W_r h in float32; s = sigmoid(z) (or softmax over the experts); the `top` experts with
//                 the largest s + correction are chosen (ties: the lower index); weight = s * scale
//                 (optionally divided by the chosen experts' sum).  A block per token, or per eight in prompt steps.
// mu_moe_group    counts the pairs of each expert, gives every pair a slot so that an expert's slots are
//                 contiguous, and lists tiles of TM slots that never straddle two experts.
// mu_moe_gemm     for every tile: out[slot, :] = act(W1[e] x[row]) (* W2[e] x[row]) on CUDA cores, one running
//                 sum per output over k in order, so a row's result does not depend on which rows share its
//                 tile.  Rows of x are gathered through the slot's pair (token = pair / top) or are the slots
//                 themselves.
// mu_moe_combine  y[t, :] = sum over the token's pairs, in the order of its choices, of weight * out[slot, :].
//
// Options for other designs.  Identity experts: the router's outputs from `n_real` on have no matrices; their
// pairs get no slot (slot_of = -1) and no tile, and the combine takes the token's own input row for them.  The
// router can divide the chosen weights by (their sum + renorm_eps), and compute one more number per token,
// sigmoid(gate_w . h), which the combine multiplies a shared expert's row by before adding it.  The experts'
// product takes an activation code (mu::ACT_*) for experts of the form W2 act(W1 x).  The combine can add its
// result to what `out` holds.  A design whose weights act on the experts' INPUT gives them to the first product
// (`row_weight`, one per pair: a row's products are multiplied by it before the activation, which is the product of
// the weighted row), and none to the combine.
#include "common.cuh"

#include <math.h>

namespace mu {

constexpr int MOE_TM = 32, MOE_TN = 64, MOE_TK = 32;

constexpr size_t ROUTE_SMEM = 100 * 1024;

// A block takes TOK consecutive tokens: their rows are staged in shared memory as they are, the warps share the
// experts (each logit one warp's sum over the row, lanes striding along it; a router row is read once for the
// block's tokens), then warp i scores and chooses for token i.  A token's sums run in the same order whatever TOK
// is and whichever tokens share its block.
//
// Many tokens: NE router rows a pass, so that a staged piece serves them all; a bfloat16 row stays bfloat16 in shared memory (half
// the passes over its banks) and becomes float32 in registers.  Seven tokens a block leave registers to ask for four pieces of
// each row at a time; eight do not, and are taken where they save a round of blocks.  64 experts, hidden 2,048, routers out of the L2: 2,048 tokens
// 44 -> 38 us; 128 experts, hidden 4,096, 900 tokens 106 -> 55.  It still waits for the rows and the sums' exchanges (the
// multiply-adds take 7).
// Few tokens (SHARED): the blocks of a cluster share a token's experts, since a block alone waits row after row for memory, and
// hand their logits to the first, which chooses: 8 tokens of 72 experts 17 -> 7 us, 128 experts of 4,096 78 -> 10; up to 16
// experts a block alone is no slower.
template <typename T, int TOK, int WARPS, int NE, bool SHARED>
__global__ void __launch_bounds__(WARPS * 32)
moe_route_kernel(const T* __restrict__ h, long long ldh, const float* __restrict__ router,
                 const float* __restrict__ correction, int n_tokens, int hidden, int n_experts, int top,
                 float scale, int softmax, int renormalize, int* __restrict__ expert_of,
                 float* __restrict__ weight_of, float renorm_eps, const float* __restrict__ gate_w,
                 float* __restrict__ gate_out) {
    extern __shared__ __align__(16) float sm[];        // rows [TOK][hidden], scores [TOK][n_experts], choice [TOK][n_experts]
    if (SHARED) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = blockIdx.x * TOK, nt = min(TOK, n_tokens - t0);
    const int shares = SHARED ? gridDim.y : 1, share = SHARED ? blockIdx.y : 0;      // (the cluster is a token's grid.y blocks)
    T* hrow = reinterpret_cast<T*>(sm);
    float* score_all = sm + ((size_t)TOK * hidden * sizeof(T) + 15) / 16 * 4;
    float* choice_all = score_all + TOK * n_experts;
    if (hidden % (16 / sizeof(T)) == 0 && ldh % (16 / sizeof(T)) == 0 && ((uintptr_t)h & 15) == 0) {
        const int pieces = hidden / (16 / (int)sizeof(T));
        for (int j = threadIdx.x; j < TOK * pieces; j += blockDim.x) {
            const int i = j / pieces, c = j % pieces;
            uint4 raw = make_uint4(0u, 0u, 0u, 0u);
            if (i < nt) raw = reinterpret_cast<const uint4*>(h + (long long)(t0 + i) * ldh)[c];
            reinterpret_cast<uint4*>(hrow)[j] = raw;
        }
    } else {
        for (int i = 0; i < TOK; ++i) {
            const T* row = h + (long long)(t0 + i) * ldh;
            for (int d = threadIdx.x; d < hidden; d += blockDim.x) hrow[i * hidden + d] = i < nt ? row[d] : from_float<T>(0.0f);
        }
    }
    __syncthreads();
    const bool wide = hidden % 4 == 0 && ((uintptr_t)router & 15) == 0 &&
                      ((uintptr_t)gate_w & 15) == 0;                          // rows of the router in 16-byte pieces
    // (with gate_w: one more sum, over the shared expert's gate row, by the warp whose turn it is)
    const int rows = n_experts + (gate_w ? 1 : 0);
    auto row_of = [&](int e) { return e < n_experts ? router + (long long)e * hidden : gate_w; };
    auto put = [&](int e, const float (&z)[TOK]) {
#pragma unroll
        for (int i = 0; i < TOK; ++i) {
            const float zi = warp_sum(z[i]);
            if (lane == 0 && i < nt) {
                if (e >= n_experts) {
                    gate_out[t0 + i] = 1.0f / (1.0f + expf(-zi));
                } else if (SHARED) {
                    uint32_t there;                          // the first block's copy of the scores
                    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(there)
                                 : "r"((uint32_t)__cvta_generic_to_shared(score_all + i * n_experts + e)));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(there), "f"(zi) : "memory");
                } else {
                    score_all[i * n_experts + e] = zi;
                }
            }
        }
    };
    // Four entries of a staged row, as pairs of float32.
    auto piece = [&](int i, int d) {
        if (sizeof(T) == 4) return reinterpret_cast<const ulonglong2*>(hrow)[i * (hidden / 4) + d];
        const uint2 raw = reinterpret_cast<const uint2*>(hrow)[i * (hidden / 4) + d];
        return make_ulonglong2(pair_of_floats(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u)),
                               pair_of_floats(__uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u)));
    };
    // One router row: the lane's part of every token's sum.
    auto sum_row = [&](const float* w, float (&z)[TOK]) {
        if (wide) {
            const ulonglong2* w4 = reinterpret_cast<const ulonglong2*>(w);
            const int n4 = hidden / 4;
            float2x z01[TOK], z23[TOK];                                      // a lane's sum in four parts, then in order
#pragma unroll
            for (int i = 0; i < TOK; ++i) z01[i] = z23[i] = 0ull;
#pragma unroll (SHARED ? 16 : 8)
            for (int d = lane; d < n4; d += 32) {                            // (unrolled: the row's loads go out together)
                const ulonglong2 b = w4[d];
#pragma unroll
                for (int i = 0; i < TOK; ++i) {
                    const ulonglong2 a = piece(i, d);
                    z01[i] = pair_fma(a.x, b.x, z01[i]);
                    z23[i] = pair_fma(a.y, b.y, z23[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < TOK; ++i) {
                const float2 lo = floats_of_pair(z01[i]), hi = floats_of_pair(z23[i]);
                z[i] = (lo.x + lo.y) + (hi.x + hi.y);
            }
        } else {
#pragma unroll
            for (int i = 0; i < TOK; ++i) z[i] = 0.0f;
            for (int d = lane; d < hidden; d += 32) {
                const float b = w[d];
#pragma unroll
                for (int i = 0; i < TOK; ++i) z[i] += to_float(hrow[i * hidden + d]) * b;
            }
        }
    };
    if (SHARED) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");      // the first block runs: its memory may be written
    constexpr int AHEAD = 4;
    const int step = WARPS * shares;
    for (int e0 = warp * shares + share; e0 < rows; e0 += NE * step) {
        if (NE > 1 && wide) {
            const ulonglong2* w4[NE];
#pragma unroll
            for (int n = 0; n < NE; ++n) w4[n] = reinterpret_cast<const ulonglong2*>(row_of(min(e0 + n * step, rows - 1)));
            const int n4 = hidden / 4, live = min(NE, (rows - e0 + step - 1) / step);
            float2x z01[NE][TOK], z23[NE][TOK];                              // a lane's sum in four parts, then in order
#pragma unroll
            for (int n = 0; n < NE; ++n)
#pragma unroll
                for (int i = 0; i < TOK; ++i) z01[n][i] = z23[n][i] = 0ull;
            auto add = [&](int d, const ulonglong2 (&b)[NE]) {
#pragma unroll
                for (int i = 0; i < TOK; ++i) {
                    const ulonglong2 a = piece(i, d);
#pragma unroll
                    for (int n = 0; n < NE; ++n) {
                        z01[n][i] = pair_fma(a.x, b[n].x, z01[n][i]);
                        z23[n][i] = pair_fma(a.y, b[n].y, z23[n][i]);
                    }
                }
            };
            int d = lane;
            for (; d - lane + 32 * AHEAD <= n4; d += 32 * AHEAD) {           // (AHEAD of the rows' pieces are asked for together)
                ulonglong2 b[AHEAD][NE];
#pragma unroll
                for (int p = 0; p < AHEAD; ++p)
#pragma unroll
                    for (int n = 0; n < NE; ++n) b[p][n] = w4[n][d + 32 * p];
#pragma unroll
                for (int p = 0; p < AHEAD; ++p) add(d + 32 * p, b[p]);
            }
            for (; d < n4; d += 32) {
                ulonglong2 b[NE];
#pragma unroll
                for (int n = 0; n < NE; ++n) b[n] = w4[n][d];
                add(d, b);
            }
#pragma unroll
            for (int n = 0; n < NE; ++n) {
                if (n >= live) continue;
                float z[TOK];
#pragma unroll
                for (int i = 0; i < TOK; ++i) {
                    const float2 lo = floats_of_pair(z01[n][i]), hi = floats_of_pair(z23[n][i]);
                    z[i] = (lo.x + lo.y) + (hi.x + hi.y);
                }
                put(e0 + n * step, z);
            }
        } else {
#pragma unroll
            for (int n = 0; n < NE; ++n) {
                const int e = e0 + n * step;
                if (n > 0 && e >= rows) break;
                float z[TOK];
                sum_row(row_of(e), z);
                put(e, z);
            }
        }
    }
    if (SHARED) {                                            // every block's logits are with the first one
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (share != 0) return;
    }
    __syncthreads();
    if (warp >= nt) return;
    const int t = t0 + warp;
    float* score = score_all + warp * n_experts;
    float* choice = choice_all + warp * n_experts;
    if (softmax) {
        float top_z = -INFINITY, sum = 0.0f;
        for (int e = lane; e < n_experts; e += 32) top_z = fmaxf(top_z, score[e]);
        top_z = warp_max(top_z);
        for (int e = lane; e < n_experts; e += 32) sum += expf(score[e] - top_z);
        sum = warp_sum(sum);
        for (int e = lane; e < n_experts; e += 32) score[e] = expf(score[e] - top_z) / sum;
    } else {
        for (int e = lane; e < n_experts; e += 32) score[e] = 1.0f / (1.0f + expf(-score[e]));
    }
    for (int e = lane; e < n_experts; e += 32) choice[e] = score[e] + (correction ? correction[e] : 0.0f);
    __syncwarp();
    float kept = 0.0f;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int arg = n_experts;
        for (int e = lane; e < n_experts; e += 32)
            if (choice[e] > best) { best = choice[e]; arg = e; }       // first maximum of the lane's experts
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
        }
        if (arg >= n_experts) arg = 0;                                 // (not a number everywhere)
        if (lane == 0) {
            expert_of[(long long)t * top + k] = arg;
            weight_of[(long long)t * top + k] = score[arg];
            choice[arg] = -INFINITY;
        }
        kept += score[arg];
        __syncwarp();
    }
    const float f = renormalize ? scale / (kept + renorm_eps) : scale;
    for (int k = lane; k < top; k += 32) weight_of[(long long)t * top + k] *= f;
}

// One block.  slot_of[pair], pair_of[slot], and the tile list: tile_info[3 i] = expert, [3 i + 1] = first slot,
// [3 i + 2] = rows; n_tiles[0] = how many.  It is a chain of latencies (read, count, sum up, write), so each is gone through
// once: a thread's pairs are read together and stay in registers (GROUP_KEPT a thread; what is beyond is read again), the
// count of a pair's expert hands it its place within the expert, and a warp sums the counts up.  (Which pair of an expert
// gets which slot changes no result: every row is computed by itself.)  With the router's pass above, two rows of it at a
// time: the layer of 64 experts of 2,048 x 1,408 x 3 over 12,288 pairs 502 us -> 470.
constexpr int GROUP_KEPT = 16;

__global__ void __launch_bounds__(1024)
moe_group_kernel(const int* __restrict__ expert_of, int n_pairs, int n_experts, int* __restrict__ slot_of,
                 int* __restrict__ pair_of, int* __restrict__ tile_info, int* __restrict__ n_tiles, int tile_rows, int n_real) {
    extern __shared__ int smi[];                       // count [n_experts], first [n_experts + 1], tile0 [n_experts + 1]
    int* count = smi;
    int* first = smi + n_experts;
    int* tile0 = first + n_experts + 1;
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) count[e] = 0;
    pdl_trigger();
    pdl_wait();
    __syncthreads();
    const int kept = GROUP_KEPT * blockDim.x;
    int expert[GROUP_KEPT], place[GROUP_KEPT];
#pragma unroll
    for (int i = 0; i < GROUP_KEPT; ++i) {
        const int p = threadIdx.x + i * blockDim.x;
        expert[i] = p < n_pairs ? expert_of[p] : n_real;
    }
#pragma unroll
    for (int i = 0; i < GROUP_KEPT; ++i) place[i] = expert[i] < n_real ? atomicAdd(&count[expert[i]], 1) : -1;
    __syncthreads();
    if (n_pairs > kept) {                              // (these take places from the end of their experts' slots, below)
        for (int p = kept + threadIdx.x; p < n_pairs; p += blockDim.x)
            if (expert_of[p] < n_real) atomicAdd(&count[expert_of[p]], 1);
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        int at = 0, tiles = 0;
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int e = e0 + threadIdx.x, n = e < n_experts ? count[e] : 0, t = (n + tile_rows - 1) / tile_rows;
            int upto_n = n, upto_t = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int on = __shfl_up_sync(0xffffffffu, upto_n, o), ot = __shfl_up_sync(0xffffffffu, upto_t, o);
                if ((int)threadIdx.x >= o) upto_n += on, upto_t += ot;
            }
            if (e < n_experts) first[e] = at + upto_n - n, tile0[e] = tiles + upto_t - t;
            at += __shfl_sync(0xffffffffu, upto_n, 31);
            tiles += __shfl_sync(0xffffffffu, upto_t, 31);
        }
        if (threadIdx.x == 0) n_tiles[0] = tiles;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < GROUP_KEPT; ++i) {
        const int p = threadIdx.x + i * blockDim.x;
        if (p < n_pairs) {
            const int slot = place[i] < 0 ? -1 : first[expert[i]] + place[i];   // (-1: an identity expert, nothing to compute)
            slot_of[p] = slot;
            if (slot >= 0) pair_of[slot] = p;
        }
    }
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) {
        const int n = count[e];
        for (int i = 0, k = tile0[e]; i < n; i += tile_rows, ++k) {
            tile_info[3 * k] = e;
            tile_info[3 * k + 1] = first[e] + i;
            tile_info[3 * k + 2] = min(tile_rows, n - i);
        }
    }
    if (n_pairs <= kept) return;
    __syncthreads();
    for (int p = kept + threadIdx.x; p < n_pairs; p += blockDim.x) {
        const int e = expert_of[p];
        int slot = -1;
        if (e < n_real) {
            slot = first[e] + atomicSub(&count[e], 1) - 1;
            pair_of[slot] = p;
        }
        slot_of[p] = slot;
    }
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// GATED: out = silu(W1 x) * (W2 x); else out = W1 x.  x rows: pair_of[slot] / top if pair_of, else slot.
template <typename T, typename TO, bool GATED>
__global__ void __launch_bounds__(256)
moe_gemm_kernel(const T* __restrict__ x, long long ldx, const int* __restrict__ pair_of, int top,
                const T* __restrict__ w1, const T* __restrict__ w2, long long expert_stride, long long ldw,
                const int* __restrict__ tile_info, const int* __restrict__ n_tiles, int n, int k,
                TO* __restrict__ out, long long ldo, int act, const float* __restrict__ row_weight) {
    __shared__ float sa[MOE_TM][MOE_TK + 1];
    __shared__ float sw1[MOE_TN][MOE_TK + 1];
    __shared__ float sw2[GATED ? MOE_TN : 1][MOE_TK + 1];
    __shared__ int src_row[MOE_TM];
    pdl_trigger();
    pdl_wait();
    const int tile = blockIdx.x;
    if (tile >= n_tiles[0]) return;
    const int e = tile_info[3 * tile], slot0 = tile_info[3 * tile + 1], rows = tile_info[3 * tile + 2];
    const int n0 = blockIdx.y * MOE_TN;
    const T* w1e = w1 + (long long)e * expert_stride;
    const T* w2e = GATED ? w2 + (long long)e * expert_stride : nullptr;
    if (threadIdx.x < MOE_TM) {
        const int r = threadIdx.x;
        src_row[r] = r < rows ? (pair_of ? pair_of[slot0 + r] / top : slot0 + r) : -1;
    }
    __syncthreads();
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;     // rows 2 ty, 2 ty + 1; columns tx + 16 j
    float a1[2][4] = {}, a2[2][4] = {};
    for (int k0 = 0; k0 < k; k0 += MOE_TK) {
        for (int i = threadIdx.x; i < MOE_TM * MOE_TK; i += 256) {
            const int r = i / MOE_TK, c = i % MOE_TK;
            const int row = src_row[r];
            sa[r][c] = (row >= 0 && k0 + c < k) ? to_float(x[(long long)row * ldx + k0 + c]) : 0.0f;
        }
        for (int i = threadIdx.x; i < MOE_TN * MOE_TK; i += 256) {
            const int r = i / MOE_TK, c = i % MOE_TK;
            const bool in = n0 + r < n && k0 + c < k;
            sw1[r][c] = in ? to_float(w1e[(long long)(n0 + r) * ldw + k0 + c]) : 0.0f;
            if (GATED) sw2[r][c] = in ? to_float(w2e[(long long)(n0 + r) * ldw + k0 + c]) : 0.0f;
        }
        __syncthreads();
#pragma unroll 8
        for (int c = 0; c < MOE_TK; ++c) {
            const float x0 = sa[2 * ty][c], x1 = sa[2 * ty + 1][c];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float u = sw1[tx + 16 * j][c];
                a1[0][j] += x0 * u;
                a1[1][j] += x1 * u;
                if (GATED) {
                    const float v = sw2[tx + 16 * j][c];
                    a2[0][j] += x0 * v;
                    a2[1][j] += x1 * v;
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = 2 * ty + i;
        if (r >= rows) continue;
        if (row_weight) {
            const float f = row_weight[pair_of ? pair_of[slot0 + r] : slot0 + r];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                a1[i][j] *= f;
                a2[i][j] *= f;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = n0 + tx + 16 * j;
            if (col >= n) continue;
            const float v = GATED ? silu(a1[i][j]) * a2[i][j] : apply_act(a1[i][j], act);
            out[(long long)(slot0 + r) * ldo + col] = from_float<TO>(v);
        }
    }
}

// x (may be null): the rows the experts read, for pairs without a slot; shared / shared_gate (may be null): a row
// per token that every token gets, times the token's gate.
template <typename TX>
__global__ void moe_combine_kernel(const float* __restrict__ y, long long ldy, const int* __restrict__ slot_of,
                                   const float* __restrict__ weight_of, int top, int width, float* __restrict__ out,
                                   long long ldo, const TX* __restrict__ x, long long ldx,
                                   const float* __restrict__ shared, long long lds,
                                   const float* __restrict__ shared_gate, int add) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float v = 0.0f;
        for (int k = 0; k < top; ++k) {
            const int slot = slot_of[(long long)t * top + k];
            const float row = slot >= 0 ? y[(long long)slot * ldy + d] : to_float(x[(long long)t * ldx + d]);
            v += (weight_of ? weight_of[(long long)t * top + k] : 1.0f) * row;
        }
        if (shared) v += (shared_gate ? shared_gate[t] : 1.0f) * shared[(long long)t * lds + d];
        if (add) v += out[(long long)t * ldo + d];
        out[(long long)t * ldo + d] = v;
    }
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// The same for rows that are whole 16-byte pieces: four entries a thread, every row's piece asked for before the
// first is used.  TOP > 0: the number of choices at compile time (the loads of all choices are in flight together).
template <typename TX, int TOP>
__global__ void moe_combine_vec_kernel(const float* __restrict__ y, long long ldy, const int* __restrict__ slot_of,
                                       const float* __restrict__ weight_of, int top, int width, float* __restrict__ out,
                                       long long ldo, const TX* __restrict__ x, long long ldx,
                                       const float* __restrict__ shared, long long lds,
                                       const float* __restrict__ shared_gate, int add) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    if (TOP > 0) top = TOP;
    for (int d = 4 * threadIdx.x; d < width; d += 4 * blockDim.x) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (TOP > 0) {
            float4 row[TOP > 0 ? TOP : 1];
            float w[TOP > 0 ? TOP : 1];
#pragma unroll
            for (int k = 0; k < TOP; ++k) {
                const int slot = slot_of[(long long)t * TOP + k];
                w[k] = weight_of ? weight_of[(long long)t * TOP + k] : 1.0f;
                row[k] = slot >= 0 ? load4(y + (long long)slot * ldy + d) : load4(x + (long long)t * ldx + d);
            }
#pragma unroll
            for (int k = 0; k < TOP; ++k) {                                // in the order of the choices
                v.x += w[k] * row[k].x; v.y += w[k] * row[k].y; v.z += w[k] * row[k].z; v.w += w[k] * row[k].w;
            }
        } else {
            for (int k = 0; k < top; ++k) {
                const int slot = slot_of[(long long)t * top + k];
                const float w = weight_of ? weight_of[(long long)t * top + k] : 1.0f;
                const float4 row = slot >= 0 ? load4(y + (long long)slot * ldy + d) : load4(x + (long long)t * ldx + d);
                v.x += w * row.x; v.y += w * row.y; v.z += w * row.z; v.w += w * row.w;
            }
        }
        if (shared) {
            const float g = shared_gate ? shared_gate[t] : 1.0f;
            const float4 sh = load4(shared + (long long)t * lds + d);
            v.x += g * sh.x; v.y += g * sh.y; v.z += g * sh.z; v.w += g * sh.w;
        }
        float* dst = out + (long long)t * ldo + d;
        if (add) {
            const float4 old = load4(dst);
            v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
        }
        *reinterpret_cast<float4*>(dst) = v;
    }
}

// The same sum, normed and added into the residual stream: out[t, :] += tanh(alpha v) w + b with v the token's sum.
__global__ void moe_combine_tanh_kernel(const float* __restrict__ y, long long ldy, const int* __restrict__ slot_of,
                                        const float* __restrict__ weight_of, int top, int width,
                                        const float* __restrict__ w, const float* __restrict__ b,
                                        const float* __restrict__ alpha, float* __restrict__ out, long long ldo) {
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x;
    const float a = alpha[0];
    for (int d = threadIdx.x; d < width; d += blockDim.x) {
        float v = 0.0f;
        for (int k = 0; k < top; ++k)
            v += weight_of[(long long)t * top + k] * y[(long long)slot_of[(long long)t * top + k] * ldy + d];
        out[(long long)t * ldo + d] += tanhf(a * v) * w[d] + (b ? b[d] : 0.0f);
    }
}

}  // namespace mu

MU_EXPORT int mu_moe_combine_tanh(const float* y, long long ldy, const int* slot_of, const float* weight_of, int n_tokens,
                                  int top, int width, const float* w, const float* b, const float* alpha, float* out,
                                  long long ldo, void* stream) {
    if (n_tokens <= 0) return MU_OK;
    if (!y || !slot_of || !weight_of || !out || !w || !alpha || top <= 0 || width <= 0) return MU_ERR_BAD_ARGUMENT;
    return mu::launch_pdl(mu::moe_combine_tanh_kernel, dim3(n_tokens), dim3(width >= 1024 ? 256 : 128), 0,
                          (cudaStream_t)stream, 1, y, ldy, slot_of, weight_of, top, width, w, b, alpha, out, ldo);
}

MU_EXPORT int mu_moe_tile_rows() { return mu::MOE_TM; }

MU_EXPORT int mu_moe_route(const void* h, long long ldh, int h_bf16, const float* router, const float* correction,
                           int n_tokens, int hidden, int n_experts, int top, float scale, int softmax, int renormalize,
                           int* expert_of, float* weight_of, void* stream, float renorm_eps, const float* gate_w,
                           float* gate_out) {
    if (n_tokens <= 0) return MU_OK;
    if (!h || !router || !expert_of || !weight_of || hidden <= 0 || n_experts <= 0 || top <= 0 || top > n_experts ||
        (gate_w != nullptr) != (gate_out != nullptr))
        return MU_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    typedef __nv_bfloat16 bf;
    auto limit = [&](int tok) { return (size_t)tok * (hidden + 2 * n_experts) * sizeof(float); };
    auto room = [&](int tok) {                               // as the kernel lays it out: the rows end on a 16-byte boundary
        return ((size_t)tok * hidden * (h_bf16 ? 2 : 4) + 15) / 16 * 16 + (size_t)tok * 2 * n_experts * sizeof(float);
    };
#define MU_ROUTE(T, TOK, WARPS, NE, SHARED, GRID, CLUSTER)                                                             \
    do {                                                                                                               \
        auto kernel = mu::moe_route_kernel<T, TOK, WARPS, NE, SHARED>;                                                 \
        if (!mu::allow_shared(reinterpret_cast<const void*>(kernel), (TOK > 1 ? mu::ROUTE_SMEM : 48 * 1024) + 16)) return MU_ERR_LAUNCH; \
        return mu::launch_pdl(kernel, GRID, dim3(WARPS * 32), room(TOK), s, CLUSTER, (const T*)h, ldh, router, correction, \
                              n_tokens, hidden, n_experts, top, scale, softmax, renormalize, expert_of, weight_of, renorm_eps, \
                              gate_w, gate_out);                                                                       \
    } while (0)
#define MU_ROUTE_MANY(TOK, WARPS, NE)                                                                                  \
    do {                                                                                                               \
        const dim3 grid((n_tokens + TOK - 1) / TOK);                                                                   \
        if (h_bf16) MU_ROUTE(bf, TOK, WARPS, NE, false, grid, 1);                                                      \
        MU_ROUTE(float, TOK, WARPS, NE, false, grid, 1);                                                               \
    } while (0)
    // prompt steps: several tokens a block, so that the router's rows are read once for all of them (with a block a
    // token the router came out of the L2 once per token), as many as there is room for
    const int sms = mu::sm_count();
    if (sms <= 0) return MU_ERR_LAUNCH;
    // widths: what one token in 48 KB as float32, or two of many in ROUTE_SMEM, leave room for (16 bytes more where a row's end is
    // rounded up), whatever the rows' type
    const bool many = n_tokens >= 4 * sms;
    if (many ? limit(2) > mu::ROUTE_SMEM : limit(1) > 48 * 1024) return MU_ERR_UNSUPPORTED_SIZE;
    if (many) {
        // (a block an SM at a time: eight tokens, with registers spilled, where that saves a round; 64 experts of 2,048, 2,100 tokens:
        // 42 us with eight, 54 with seven; 2,048: 44 and 38)
        const int rounds8 = (n_tokens + 8 * sms - 1) / (8 * sms), rounds7 = (n_tokens + 7 * sms - 1) / (7 * sms);
        if (room(8) <= mu::ROUTE_SMEM && rounds8 < rounds7) MU_ROUTE_MANY(8, 16, 2);
        if (room(7) <= mu::ROUTE_SMEM) MU_ROUTE_MANY(7, 16, 2);
        if (room(4) <= mu::ROUTE_SMEM) MU_ROUTE_MANY(4, 16, 2);
        MU_ROUTE_MANY(2, 16, 1);
    }
    // few tokens: a block each, or a cluster of blocks that share the experts while these blocks find an SM
    const int rows = n_experts + (gate_w ? 1 : 0);
    const int shares = rows <= 16 ? 1 : n_tokens <= sms / 2 ? 8 : n_tokens <= sms ? 4 : 1;
    if (shares > 1) {
        const dim3 grid(n_tokens, shares);
        if (h_bf16) MU_ROUTE(bf, 1, 16, 1, true, grid, shares);
        MU_ROUTE(float, 1, 16, 1, true, grid, shares);
    }
    MU_ROUTE_MANY(1, 16, 1);
#undef MU_ROUTE_MANY
#undef MU_ROUTE
}

// tile_info needs 3 * (n_pairs / tile_rows + n_experts) ints.  tile_rows: the CUDA-core product takes tiles of
// mu_moe_tile_rows() slots, the tensor-core product of 32 or 64.
// n_real (0: all of them): experts from n_real on are identity experts.
MU_EXPORT int mu_moe_group(const int* expert_of, int n_pairs, int n_experts, int* slot_of, int* pair_of, int* tile_info,
                           int* n_tiles, int tile_rows, void* stream, int n_real) {
    if (n_pairs <= 0) return MU_OK;
    if (!expert_of || !slot_of || !pair_of || !tile_info || !n_tiles || n_experts <= 0 || tile_rows <= 0)
        return MU_ERR_BAD_ARGUMENT;
    const size_t smem = (size_t)(3 * n_experts + 2) * sizeof(int);
    if (smem > 48 * 1024) return MU_ERR_UNSUPPORTED_SIZE;
    if (n_real < 0 || n_real > n_experts) return MU_ERR_BAD_ARGUMENT;
    // (a block of 1,024 takes a whole SM's registers and waits for an empty one: 288 pairs, the layer around them, 86 us so, 81
    // with fewer)
    const int threads = n_pairs <= 256 ? 128 : n_pairs <= 1024 ? 256 : 1024;
    return mu::launch_pdl(mu::moe_group_kernel, dim3(1), dim3(threads), smem, (cudaStream_t)stream, 1, expert_of, n_pairs,
                          n_experts, slot_of, pair_of, tile_info, n_tiles, tile_rows, n_real > 0 ? n_real : n_experts);
}

// w1 (and w2 when gated): [n_experts][n][k] with row stride ldw and expert stride `expert_stride` elements.
// max_tiles: the bound the grid is sized for (n_pairs / tile_rows + n_experts covers every grouping).
MU_EXPORT int mu_moe_gemm(const void* x, long long ldx, const int* pair_of, int top, const void* w1, const void* w2,
                          long long expert_stride, long long ldw, const int* tile_info, const int* n_tiles,
                          int max_tiles, int n, int k, void* out, long long ldo, int is_bf16, int out_bf16,
                          void* stream, int act, const float* row_weight) {
    if (max_tiles <= 0) return MU_OK;
    if (!x || !w1 || !tile_info || !n_tiles || !out || n <= 0 || k <= 0 || (pair_of && top <= 0))
        return MU_ERR_BAD_ARGUMENT;
    if (is_bf16 != out_bf16 && !(is_bf16 && !out_bf16)) return MU_ERR_BAD_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 grid(max_tiles, (n + mu::MOE_TN - 1) / mu::MOE_TN), block(256);
    typedef __nv_bfloat16 bf;
#define MU_MOE(T, TO, G)                                                                                             \
    return mu::launch_pdl(mu::moe_gemm_kernel<T, TO, G>, grid, block, 0, s, 1, (const T*)x, ldx, pair_of, top,        \
                          (const T*)w1, (const T*)w2, expert_stride, ldw, tile_info, n_tiles, n, k, (TO*)out, ldo, act, row_weight)
    if (w2) {
        if (is_bf16 && out_bf16) MU_MOE(bf, bf, true);
        if (is_bf16) MU_MOE(bf, float, true);
        MU_MOE(float, float, true);
    }
    if (is_bf16 && out_bf16) MU_MOE(bf, bf, false);
    if (is_bf16) MU_MOE(bf, float, false);
    MU_MOE(float, float, false);
#undef MU_MOE
}

// x (the experts' input rows, bfloat16 if x_bf16 else float32) is needed when a pair may have no slot; weight_of null:
// every choice counts once.
MU_EXPORT int mu_moe_combine(const float* y, long long ldy, const int* slot_of, const float* weight_of, int n_tokens,
                             int top, int width, float* out, long long ldo, void* stream, const void* x, long long ldx,
                             int x_bf16, const float* shared, long long lds, const float* shared_gate, int add) {
    if (n_tokens <= 0) return MU_OK;
    if (!y || !slot_of || !out || top <= 0 || width <= 0) return MU_ERR_BAD_ARGUMENT;
    const dim3 grid(n_tokens), block(width >= 1024 ? 256 : 128);
    const bool vec = width % 4 == 0 && ldy % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)y & 15) == 0 && ((uintptr_t)out & 15) == 0 &&
                     (!x || (ldx % 4 == 0 && ((uintptr_t)x & (x_bf16 ? 7 : 15)) == 0)) &&
                     (!shared || (lds % 4 == 0 && ((uintptr_t)shared & 15) == 0));
    if (vec) {
        const dim3 vblock(width >= 1024 ? 256 : width >= 512 ? 128 : 64);
#define MU_COMBINE(TX, TOP)                                                                                            \
    return mu::launch_pdl(mu::moe_combine_vec_kernel<TX, TOP>, grid, vblock, 0, (cudaStream_t)stream, 1, y, ldy, slot_of, \
                          weight_of, top, width, out, ldo, (const TX*)x, ldx, shared, lds, shared_gate, add)
        if (x_bf16) {
            if (top == 1) MU_COMBINE(__nv_bfloat16, 1);
            if (top == 2) MU_COMBINE(__nv_bfloat16, 2);
            if (top == 4) MU_COMBINE(__nv_bfloat16, 4);
            if (top == 6) MU_COMBINE(__nv_bfloat16, 6);
            if (top == 8) MU_COMBINE(__nv_bfloat16, 8);
            MU_COMBINE(__nv_bfloat16, 0);
        }
        if (top == 1) MU_COMBINE(float, 1);
        if (top == 2) MU_COMBINE(float, 2);
        if (top == 4) MU_COMBINE(float, 4);
        if (top == 6) MU_COMBINE(float, 6);
        if (top == 8) MU_COMBINE(float, 8);
        MU_COMBINE(float, 0);
#undef MU_COMBINE
    }
    if (x_bf16)
        return mu::launch_pdl(mu::moe_combine_kernel<__nv_bfloat16>, grid, block, 0, (cudaStream_t)stream, 1, y, ldy,
                              slot_of, weight_of, top, width, out, ldo, (const __nv_bfloat16*)x, ldx, shared, lds,
                              shared_gate, add);
    return mu::launch_pdl(mu::moe_combine_kernel<float>, grid, block, 0, (cudaStream_t)stream, 1, y, ldy, slot_of,
                          weight_of, top, width, out, ldo, (const float*)x, ldx, shared, lds, shared_gate, add);
}
