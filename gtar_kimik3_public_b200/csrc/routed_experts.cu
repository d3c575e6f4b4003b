// A feed-forward of many small gated experts of which every token uses a few.
//
//   route        z = W_r h in 32-bit (a warp per token and eight experts), then, a warp per token: s = sigmoid(z),
//                choice = s + correction.  The experts form equal groups of neighbours; a group's score is the sum of its
//                two largest choice scores and only the experts of the best `keep` groups may be chosen.  The `top`
//                largest choice scores among them are chosen (ties: the lower index); a chosen expert's weight is its s
//                (without the correction) times a constant.
//                With the flag for logits the score is the logit itself plus a stored bias, s = z + b (no sigmoid, choice by s),
//                and the chosen experts' weights are the softmax over the chosen scores alone, times the constant.
//                Further rules (flags): s = softmax(z) over all experts; a group's score is its largest choice score; the
//                chosen experts' s are divided by their sum (plus 1e-20) before the constant.
//                A shared expert that every token runs, weighted by the sigmoid of a number of its own: that number's row
//                stands behind the router's rows (z has E + 1 entries), and the sigmoid is either the weight of one more
//                pair (token, expert E) behind the token's chosen ones, or an output of its own.
//   experts_up   act[pair] = silu(W_gate[e] h_t) * (W_up[e] h_t) for every pair (token, chosen expert)
//   experts_down (and experts_join behind it) out_t = add_t (times a number per token, where one is given) + sum over the token's pairs, in the order they were chosen, of weight * W_down[e] act[pair]
//                (32-bit result: it is what goes into the residual stream)
//
// This is the path of few-token steps, of 32-bit runs and of sizes the sorted path does not take.  Its kernels come in two forms with
// the same sums: an expert's pairs together, so that its rows are fetched once for several of them, and, where the pairs' experts
// are nearly all different or small, a pair and a token by itself (`experts` below).  A token's result depends on the token alone.
//
//   sort, gather_rows, combine   many-token steps: the pairs put in the order of their experts, the tokens' rows copied
//                into that order (each expert's rows then go through one tensor-core product, made by the caller), and
//                the weighted sum of a token's expert outputs in the order the experts were chosen

#include <algorithm>
#include <cmath>

#include "tensor_map.cuh"

namespace {

constexpr int ROUTE_WARPS = 4;

__device__ __forceinline__ void score_copy16(void* smem, const void* gmem, bool in) {  // zeros where `in` is false
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}


// Loads of several elements want their address on as many bytes: a row length that is a multiple of them says so only where the
// matrix starts on them (a view into a larger buffer may start anywhere).
__device__ __forceinline__ bool starts_on(const void* p, int bytes) { return ((uintptr_t)p & (bytes - 1)) == 0; }

// four neighbouring numbers of a row (which start on four elements), zeros where `in` is false
template <typename T>
__device__ __forceinline__ void load_four(const T* p, bool in, float (&v)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 x = in ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    } else {
        const uint2 raw = in ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        v[0] = lo.x, v[1] = lo.y, v[2] = hi.x, v[3] = hi.y;
    }
}

// z[t, e] = h_t . w_router[e] in 32-bit.  One warp per (SCORE_TOKENS tokens, SCORE_EXPERTS experts): four and eight where
// tokens are many (a router row is fetched once for four tokens; eight tokens a warp measured slower: 66 against 60 us
// for 2,048 tokens of 1,024 and 32 experts), four and two where they are few and the launch would otherwise be a handful
// of warps; a lane sums its elements of a row in index order and the lanes meet in the fixed order of warp_sum, so a
// score depends on the token's row alone.
template <typename T, int SCORE_EXPERTS, int SCORE_TOKENS>
__global__ void __launch_bounds__(ROUTE_WARPS * 32) route_scores_kernel(const T* __restrict__ h, const float* __restrict__ w_router,
                                                                        float* __restrict__ z, int n_tokens, int width, int n_experts) {
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int parts = (n_experts + SCORE_EXPERTS - 1) / SCORE_EXPERTS;
    const int token_groups = (n_tokens + SCORE_TOKENS - 1) / SCORE_TOKENS;
    const long long unit = (long long)blockIdx.x * ROUTE_WARPS + warp;
    if (unit >= (long long)token_groups * parts) return;
    const int t0 = (int)(unit / parts) * SCORE_TOKENS, e0 = (int)(unit % parts) * SCORE_EXPERTS;
    float acc[SCORE_TOKENS][SCORE_EXPERTS];
#pragma unroll
    for (int a = 0; a < SCORE_TOKENS; ++a)
#pragma unroll
        for (int j = 0; j < SCORE_EXPERTS; ++j) acc[a][j] = 0.f;
    if (width % 4 == 0 && starts_on(h, 4 * sizeof(T)) && starts_on(w_router, 16)) {  // four neighbouring elements a lane and turn
#pragma unroll (SCORE_EXPERTS == 2 ? 4 : 2)
        for (int i = lane * 4; i < width; i += 128) {
            float xv[SCORE_TOKENS][4], wv[SCORE_EXPERTS][4];
#pragma unroll
            for (int a = 0; a < SCORE_TOKENS; ++a) load_four(h + (size_t)(t0 + a) * width + i, t0 + a < n_tokens, xv[a]);
#pragma unroll
            for (int j = 0; j < SCORE_EXPERTS; ++j) load_four(w_router + (size_t)(e0 + j) * width + i, e0 + j < n_experts, wv[j]);
#pragma unroll
            for (int a = 0; a < SCORE_TOKENS; ++a)
#pragma unroll
                for (int j = 0; j < SCORE_EXPERTS; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[a][j] = fmaf(xv[a][e], wv[j][e], acc[a][j]);
        }
    } else
#pragma unroll 4
    for (int i = lane; i < width; i += 32) {
        float xv[SCORE_TOKENS], wv[SCORE_EXPERTS];
#pragma unroll
        for (int a = 0; a < SCORE_TOKENS; ++a) xv[a] = t0 + a < n_tokens ? to_float(h[(size_t)(t0 + a) * width + i]) : 0.f;
#pragma unroll
        for (int j = 0; j < SCORE_EXPERTS; ++j) wv[j] = e0 + j < n_experts ? w_router[(size_t)(e0 + j) * width + i] : 0.f;
#pragma unroll
        for (int a = 0; a < SCORE_TOKENS; ++a)
#pragma unroll
            for (int j = 0; j < SCORE_EXPERTS; ++j) acc[a][j] = fmaf(xv[a], wv[j], acc[a][j]);
    }
#pragma unroll
    for (int a = 0; a < SCORE_TOKENS; ++a)
#pragma unroll
        for (int j = 0; j < SCORE_EXPERTS; ++j) {
            const float sum = warp_sum(acc[a][j]);
            if (lane == 0 && t0 + a < n_tokens && e0 + j < n_experts) z[(size_t)(t0 + a) * n_experts + e0 + j] = sum;
        }
}

// The same where tokens are few: a block has eight tokens and two rows of the router, all of which it asks for at once (the kernel
// above goes back to memory for every fourth of a row, on a handful of SMs), a warp four tokens and one row.  Rows of a multiple
// of eight entries; the sums are those of the kernel above bit for bit.  Bound by its launch and one trip to memory.
// Measured (us, scores and choice, cold, 1 to 128 tokens; the kernel above / here): 64 experts of 2,048: 23.6 / 13.3, 32 of 1,024: 17.4 /
// 11.3, 16 of 4,096: 32 / 11.3; 8 of 256: 11.3 / 9.2.
constexpr int FEW_TOKENS = 8, FEW_EXPERTS = 2;
template <typename T>
__global__ void __launch_bounds__(128) route_scores_few_kernel(const T* __restrict__ h, const float* __restrict__ w_router, float* __restrict__ z,
                                                               int n_tokens, int width, int n_experts) {
    extern __shared__ __align__(16) unsigned char few_smem[];  // router rows [FEW_EXPERTS][width], tokens [FEW_TOKENS][width]
    float* ws = reinterpret_cast<float*>(few_smem);
    T* xs = reinterpret_cast<T*>(ws + FEW_EXPERTS * width);
    pdl_launch_dependents();
    const int e0 = blockIdx.x * FEW_EXPERTS, t0 = blockIdx.y * FEW_TOKENS, tokens = min(FEW_TOKENS, n_tokens - t0), rows = min(FEW_EXPERTS, n_experts - e0);
    for (int i = threadIdx.x * 4; i < rows * width; i += 128 * 4) cp_async_16(ws + i, w_router + (size_t)e0 * width + i);  // no kernel in flight writes them
    pdl_wait();
    constexpr int PIECE = 16 / sizeof(T);
    for (int i = threadIdx.x * PIECE; i < tokens * width; i += 128 * PIECE) cp_async_16(xs + i, h + (size_t)t0 * width + i);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = warp & 1, first = (warp >> 1) * 4;
    if (row >= rows || first >= tokens) return;
    const float* w = ws + row * width;
    const T* x = xs + first * width;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int i = lane * 4; i < width; i += 128) {
        float wv[4], xv[4][4];
        load_four(w + i, true, wv);
#pragma unroll
        for (int a = 0; a < 4; ++a) load_four(x + a * width + i, first + a < tokens, xv[a]);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[a] = fmaf(xv[a][e], wv[e], acc[a]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const float sum = warp_sum(acc[a]);
        if (lane == 0 && first + a < tokens) z[(size_t)(t0 + first + a) * n_experts + e0 + row] = sum;
    }
}

// The same for many bfloat16 tokens: a block has 16 tokens and 16 NJ rows of the router, the reduction in pieces of 64 entries
// that come through a two-stage cp.async ring.  Its threads are four groups of 64 that take a quarter of every piece each, a
// thread 4 tokens x NJ rows; the groups' sums meet at the end in their order.  A score depends on the token's row alone.
constexpr int SCORE_K = 64, SCORE_ROWS = 16, SCORE_LDW = SCORE_K + 4, SCORE_LDH = SCORE_K + 8;


template <int NJ>
__global__ void __launch_bounds__(256) route_scores_tiled_kernel(const __nv_bfloat16* __restrict__ h, const float* __restrict__ w_router,
                                                                 float* __restrict__ z, int n_tokens, int width, int n_rows) {
    constexpr int BN = 16 * NJ;
    __shared__ __align__(16) float ws[2][BN * SCORE_LDW];
    __shared__ __align__(16) __nv_bfloat16 hs[2][SCORE_ROWS * SCORE_LDH];
    const int tid = threadIdx.x, kg = tid >> 6, eg = tid & 15, tg = (tid >> 4) & 3;
    const int t0 = blockIdx.x * SCORE_ROWS, n0 = blockIdx.y * BN;
    pdl_launch_dependents();
    const int pieces = (width + SCORE_K - 1) / SCORE_K;
    auto issue_weights = [&](int p) {
        for (int i = tid; i < BN * (SCORE_K / 4); i += 256) {
            const int row = i / (SCORE_K / 4), k = (i % (SCORE_K / 4)) * 4, at = p * SCORE_K + k;
            const bool in = n0 + row < n_rows && at < width;
            score_copy16(&ws[p & 1][row * SCORE_LDW + k], in ? w_router + (size_t)(n0 + row) * width + at : w_router, in);
        }
    };
    auto issue_tokens = [&](int p) {
        if (tid < SCORE_ROWS * (SCORE_K / 8)) {
            const int row = tid / (SCORE_K / 8), k = (tid % (SCORE_K / 8)) * 8, at = p * SCORE_K + k;
            const bool in = t0 + row < n_tokens && at < width;
            score_copy16(&hs[p & 1][row * SCORE_LDH + k], in ? h + (size_t)(t0 + row) * width + at : h, in);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue_weights(0);  // no kernel in flight writes them
    pdl_wait();
    issue_tokens(0);
    float acc[4][NJ];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[a][j] = 0.f;
    for (int p = 0; p < pieces; ++p) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (p + 1 < pieces) {
            issue_weights(p + 1);
            issue_tokens(p + 1);
        }
        const float* wp = &ws[p & 1][eg * SCORE_LDW + kg * 16];
        const __nv_bfloat16* hp = &hs[p & 1][tg * 4 * SCORE_LDH + kg * 16];
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
            float x[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const uint2 raw = *reinterpret_cast<const uint2*>(hp + a * SCORE_LDH + k);
                const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
                const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
                x[a][0] = lo.x, x[a][1] = lo.y, x[a][2] = hi.x, x[a][3] = hi.y;
            }
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(wp + j * 16 * SCORE_LDW + k);
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    acc[a][j] = fmaf(x[a][0], w.x, acc[a][j]);
                    acc[a][j] = fmaf(x[a][1], w.y, acc[a][j]);
                    acc[a][j] = fmaf(x[a][2], w.z, acc[a][j]);
                    acc[a][j] = fmaf(x[a][3], w.w, acc[a][j]);
                }
            }
        }
        // the next turn's first barrier stands before anything is written into this stage again
    }
    __syncthreads();
    float* sums = &ws[0][0];  // [4][SCORE_ROWS][BN]
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int j = 0; j < NJ; ++j) sums[(kg * SCORE_ROWS + tg * 4 + a) * BN + eg + 16 * j] = acc[a][j];
    __syncthreads();
    for (int i = tid; i < SCORE_ROWS * BN; i += 256) {
        const int t = t0 + i / BN, n = n0 + i % BN;
        if (t < n_tokens && n < n_rows)
            z[(size_t)t * n_rows + n] = ((sums[i] + sums[SCORE_ROWS * BN + i]) + sums[2 * SCORE_ROWS * BN + i]) + sums[3 * SCORE_ROWS * BN + i];
    }
}

enum RouteFlags : int { ROUTE_LOGITS = 1, ROUTE_SOFTMAX = 2, ROUTE_GROUP_BEST = 4, ROUTE_RENORMALISE = 8 };

// The choice from the scores: one warp per token.  z has n_scores = n_experts or n_experts + 1 entries a token; ids and
// weights have ld_pairs.
__global__ void __launch_bounds__(ROUTE_WARPS * 32) route_choose_kernel(
    const float* __restrict__ z, const float* __restrict__ correction, int* __restrict__ ids, float* __restrict__ weights,
    int n_tokens, int n_experts, int top, int n_groups, int keep, float scale, int flags, int n_scores, int ld_pairs,
    float* __restrict__ shared_weight) {
    extern __shared__ float route_smem[];  // per warp: s [E] | choice [E] | group score [n_groups]
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * ROUTE_WARPS + warp;
    if (t >= n_tokens) return;
    float* s = route_smem + (size_t)warp * (2 * n_experts + n_groups);
    float* choice = s + n_experts;
    float* group_score = choice + n_experts;
    const bool logits = (flags & ROUTE_LOGITS) != 0, softmax = (flags & ROUTE_SOFTMAX) != 0;
    float largest_z = -INFINITY, denom = 0.f;
    if (softmax) {
        for (int e = lane; e < n_experts; e += 32) largest_z = fmaxf(largest_z, z[(size_t)t * n_scores + e]);
        largest_z = warp_max(largest_z);
        for (int e = lane; e < n_experts; e += 32) denom += expf(z[(size_t)t * n_scores + e] - largest_z);
        denom = warp_sum(denom);
    }
    for (int e = lane; e < n_experts; e += 32) {
        const float ze = z[(size_t)t * n_scores + e];
        const float sg = logits ? ze + correction[e] : softmax ? expf(ze - largest_z) / denom : 1.f / (1.f + expf(-ze));
        s[e] = sg;
        choice[e] = logits ? sg : sg + correction[e];
    }
    if (n_scores > n_experts && lane == 0) {
        const float share = 1.f / (1.f + expf(-z[(size_t)t * n_scores + n_experts]));
        if (shared_weight != nullptr) shared_weight[t] = share;
        else {
            ids[(size_t)t * ld_pairs + top] = n_experts;
            weights[(size_t)t * ld_pairs + top] = share;
        }
    }
    __syncwarp();
    const int per = n_experts / n_groups;
    if (n_groups > 1 && keep < n_groups) {
        for (int gidx = lane; gidx < n_groups; gidx += 32) {
            float first = -INFINITY, second = -INFINITY;
#pragma unroll 8
            for (int e = gidx * per; e < (gidx + 1) * per; ++e) {
                const float c = choice[e];
                if (c > first) { second = first; first = c; }
                else if (c > second) second = c;
            }
            group_score[gidx] = per > 1 && !(flags & ROUTE_GROUP_BEST) ? first + second : first;
        }
        __syncwarp();
        // the groups that are not among the best `keep` lose their experts
        for (int gidx = lane; gidx < n_groups; gidx += 32) {
            int better = 0;
#pragma unroll 8
            for (int o = 0; o < n_groups; ++o)
                better += (group_score[o] > group_score[gidx]) || (group_score[o] == group_score[gidx] && o < gidx);
            if (better >= keep)
                for (int e = gidx * per; e < (gidx + 1) * per; ++e) choice[e] = -INFINITY;
        }
        __syncwarp();
    }
    // A lane keeps the best of its own experts, as a number that orders like the score (zero: none left); two reductions of the warp
    // find the largest and, where several are equal, the lowest expert.
    unsigned int best = 0;
    int arg = 0x7fffffff;
    const auto own_best = [&]() {
        best = 0, arg = 0x7fffffff;
        for (int e = lane; e < n_experts; e += 32) {
            const float c = choice[e] + 0.f;  // one zero
            const unsigned int bits = __float_as_uint(c), key = c > -INFINITY ? (bits & 0x80000000u ? ~bits : bits | 0x80000000u) : 0u;
            if (key > best) best = key, arg = e;
        }
    };
    own_best();
    for (int pick = 0; pick < top; ++pick) {
        const unsigned int most = __reduce_max_sync(0xffffffffu, best);
        int chosen = (int)__reduce_min_sync(0xffffffffu, best == most ? (unsigned int)arg : 0x7fffffffu);
        if (chosen == 0x7fffffff) chosen = 0;  // nothing left to choose from: cannot happen when top <= allowed experts
        if (lane == 0) {
            ids[(size_t)t * ld_pairs + pick] = chosen;
            weights[(size_t)t * ld_pairs + pick] = logits || (flags & ROUTE_RENORMALISE) ? s[chosen] : s[chosen] * scale;
        }
        if (lane == (chosen & 31)) {
            choice[chosen] = -INFINITY;
            own_best();
        }
    }
    __syncwarp();
    if ((flags & ROUTE_RENORMALISE) && lane == 0) {
        float* w = weights + (size_t)t * ld_pairs;
        float sum = 0.f;
        for (int pick = 0; pick < top; ++pick) sum += w[pick];
        for (int pick = 0; pick < top; ++pick) w[pick] = w[pick] / (sum + 1e-20f) * scale;
    }
    if (logits && lane == 0) {
        // softmax over the chosen scores, in the order they were chosen (the first is the largest)
        float* w = weights + (size_t)t * ld_pairs;
        const float largest = w[0];
        float sum = 0.f;
        for (int pick = 0; pick < top; ++pick) sum += expf(w[pick] - largest);
        for (int pick = 0; pick < top; ++pick) w[pick] = expf(w[pick] - largest) / sum * scale;
    }
}

template <typename TW>
__device__ __forceinline__ bool wide_rows(const TW* matrix, int n) { return n % (16 / (int)sizeof(TW)) == 0 && starts_on(matrix, 16); }

// A lane's share of the dot products of NR rows in memory with NT vectors in shared memory (`stride` apart), each summed in
// index order; the rows' loads are independent, so all of them are on their way together, and a piece of a vector is read once
// for all rows.  `wide` (wide_rows): 16-byte loads.  The caller finishes each with warp_sum.
template <typename TW, int NR, int NT>
__device__ __forceinline__ void dot_many(const float* __restrict__ x, int stride, const TW* const (&rows)[NR], int n, bool wide, int lane, float (&acc)[NT][NR]) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < NR; ++j) acc[t][j] = 0.f;
    constexpr int VEC = 16 / sizeof(TW);
    if (wide) {
#pragma unroll 2
        for (int i = lane * VEC; i < n; i += 32 * VEC) {
            uint4 raw[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) raw[j] = *reinterpret_cast<const uint4*>(rows[j] + i);
            float w[NR][VEC];
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                if constexpr (sizeof(TW) == 2) {
                    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float2 f = __bfloat1622float2(p[c]);
                        w[j][2 * c] = f.x, w[j][2 * c + 1] = f.y;
                    }
                } else {
                    const float* f = reinterpret_cast<const float*>(&raw[j]);
#pragma unroll
                    for (int c = 0; c < VEC; ++c) w[j][c] = f[c];
                }
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
#pragma unroll
                for (int c = 0; c < VEC; c += 4) {
                    const float4 xv = *reinterpret_cast<const float4*>(x + t * stride + i + c);
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        acc[t][j] = fmaf(xv.x, w[j][c], acc[t][j]);
                        acc[t][j] = fmaf(xv.y, w[j][c + 1], acc[t][j]);
                        acc[t][j] = fmaf(xv.z, w[j][c + 2], acc[t][j]);
                        acc[t][j] = fmaf(xv.w, w[j][c + 3], acc[t][j]);
                    }
                }
            }
        }
    } else {
        for (int i = lane; i < n; i += 32)
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                const float w = to_float(rows[j][i]);
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[t][j] = fmaf(x[t * stride + i], w, acc[t][j]);
            }
    }
}

constexpr int UP_WARPS = 8, LIST = 1024, MAX_NT = 4;

// The pairs of one expert among the LIST pairs from `first` on, in their order.  A block asks for the expert `blockIdx.x`
// (by_expert) or for that of pair `blockIdx.x`; in the second form only the block of the expert's first pair goes on.
// Returns how many there are (0: nothing to do), the same in all threads.
template <int WARPS>
__device__ __forceinline__ int list_pairs(const int* __restrict__ ids, int n_pairs, int first, bool by_expert, int& expert, int* list, int* scratch) {
    expert = by_expert ? (int)blockIdx.x : ids[blockIdx.x];
    const int last = min(first + LIST, n_pairs), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int count = 0;
    for (int i0 = first; i0 < last; i0 += WARPS * 32) {
        const int i = i0 + threadIdx.x;
        const bool mine = i < last && ids[i] == expert;
        const unsigned int found = __ballot_sync(0xffffffffu, mine);
        if (lane == 0) scratch[warp] = __popc(found);
        __syncthreads();
        int before = count;
        for (int w = 0; w < WARPS; ++w) {
            if (w < warp) before += scratch[w];
            count += scratch[w];
        }
        if (mine) list[before + __popc(found & ((1u << lane) - 1))] = i;
        __syncthreads();
    }
    if (!by_expert && count > 0 && list[0] != (int)blockIdx.x) count = 0;
    return count;
}

// act[pair] = silu(gate) * up for NT pairs of one expert (their tokens' rows in `xs`), rows f0 .. f_end - 1
template <typename T, typename TW, int NT, bool LISTED = true>
__device__ __forceinline__ void up_rows(const float* xs, const int* pairs, int count, const TW* wg, const TW* wu, T* __restrict__ act, int width, int ff, bool wide, int f0, int f_end) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int f = f0 + warp;
    for (; f + UP_WARPS < f_end; f += 2 * UP_WARPS) {  // two rows of gate and of up at once: four rows' loads in flight
        const TW* const rows[4] = {wg + (size_t)f * width, wu + (size_t)f * width, wg + (size_t)(f + UP_WARPS) * width,
                                   wu + (size_t)(f + UP_WARPS) * width};
        float part[NT][4];
        dot_many<TW, 4, NT>(xs, width, rows, width, LISTED ? wide : wide_rows(rows[0], width), lane, part);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int j = 0; j < 4; ++j) part[t][j] = warp_sum(part[t][j]);
            if (lane == 0 && t < count) {
                T* to = act + (size_t)pairs[t] * ff + f;
                to[0] = from_float<T>(part[t][0] / (1.f + expf(-part[t][0])) * part[t][1]);
                to[UP_WARPS] = from_float<T>(part[t][2] / (1.f + expf(-part[t][2])) * part[t][3]);
            }
        }
    }
    for (; f < f_end; f += UP_WARPS) {
        const TW* const rows[2] = {wg + (size_t)f * width, wu + (size_t)f * width};
        float part[NT][2];
        dot_many<TW, 2, NT>(xs, width, rows, width, LISTED ? wide : wide_rows(rows[0], width), lane, part);
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float gate = warp_sum(part[t][0]), up = warp_sum(part[t][1]);
            if (lane == 0 && t < count) act[(size_t)pairs[t] * ff + f] = from_float<T>(gate / (1.f + expf(-gate)) * up);
        }
    }
}

// grid (experts or pairs, chunks of ff, lists of pairs): w_gate_up [E, 2, ff, width] (gate rows then up rows of an expert).
// An expert's rows are fetched once for `at_once` of the tokens that chose it (more tokens take the rows again, out of L2).
template <typename T, typename TW>
__global__ void __launch_bounds__(UP_WARPS * 32) experts_up_kernel(
    const T* __restrict__ h, const TW* __restrict__ w_gate_up, const int* __restrict__ ids, T* __restrict__ act, int n_pairs, int width,
    int ff, int top, int rows_per_block, int by_expert, int at_once) {
    extern __shared__ __align__(16) unsigned char expert_smem[];
    float* xs = reinterpret_cast<float*>(expert_smem);  // [at_once][width]
    __shared__ int list[LIST], scratch[UP_WARPS];
    pdl_launch_dependents();
    pdl_wait();
    int e;
    const int n = list_pairs<UP_WARPS>(ids, n_pairs, blockIdx.z * LIST, by_expert != 0, e, list, scratch);
    const TW* wg = w_gate_up + (size_t)e * 2 * ff * width;
    const TW* wu = wg + (size_t)ff * width;
    const int f0 = blockIdx.y * rows_per_block, f_end = min(ff, f0 + rows_per_block);
    const bool wide = wide_rows(w_gate_up, width);
    for (int at = 0; at < n; at += at_once) {
        const int count = min(at_once, n - at);
        __syncthreads();
        for (int k = 0; k < count; ++k) {
            const T* x = h + (size_t)(list[at + k] / top) * width;
            for (int i = threadIdx.x; i < width; i += UP_WARPS * 32) xs[k * width + i] = to_float(x[i]);
        }
        __syncthreads();
        if (count == 1) up_rows<T, TW, 1>(xs, list + at, count, wg, wu, act, width, ff, wide, f0, f_end);
        else if (count == 2) up_rows<T, TW, 2>(xs, list + at, count, wg, wu, act, width, ff, wide, f0, f_end);
        else up_rows<T, TW, MAX_NT>(xs, list + at, count, wg, wu, act, width, ff, wide, f0, f_end);
    }
}

template <typename TW, int NT>
__device__ __forceinline__ void down_rows(const float* as, const int* pairs, int count, const TW* w, float* __restrict__ parts, int width, int ff, bool wide, int c0, int c_end) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int c = c0 + 4 * warp; c < c_end; c += 4 * UP_WARPS) {
        if (c + 4 <= c_end) {  // four rows' loads in flight
            const TW* const rows[4] = {w + (size_t)c * ff, w + (size_t)(c + 1) * ff, w + (size_t)(c + 2) * ff, w + (size_t)(c + 3) * ff};
            float part[NT][4];
            dot_many<TW, 4, NT>(as, ff, rows, ff, wide, lane, part);
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                float mine = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float sum = warp_sum(part[t][j]);
                    if (lane == j) mine = sum;
                }
                if (lane < 4 && t < count) parts[(size_t)pairs[t] * width + c + lane] = mine;
            }
        } else {  // what is left of a chunk that is no multiple of four
            for (int cc = c; cc < c_end; ++cc) {
                const TW* const rows[1] = {w + (size_t)cc * ff};
                float part[NT][1];
                dot_many<TW, 1, NT>(as, ff, rows, ff, wide, lane, part);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const float sum = warp_sum(part[t][0]);
                    if (lane == 0 && t < count) parts[(size_t)pairs[t] * width + cc] = sum;
                }
            }
        }
    }
}

// grid as experts_up: w_down [E, width, ff], parts [pairs, width] = the pairs' unweighted outputs, which experts_join adds up.
template <typename T, typename TW>
__global__ void __launch_bounds__(UP_WARPS * 32) experts_down_kernel(
    const T* __restrict__ act, const TW* __restrict__ w_down, const int* __restrict__ ids, float* __restrict__ parts, int n_pairs, int width,
    int ff, int rows_per_block, int by_expert, int at_once) {
    extern __shared__ __align__(16) unsigned char expert_smem[];
    float* as = reinterpret_cast<float*>(expert_smem);  // [at_once][ff]
    __shared__ int list[LIST], scratch[UP_WARPS];
    pdl_launch_dependents();
    pdl_wait();
    int e;
    const int n = list_pairs<UP_WARPS>(ids, n_pairs, blockIdx.z * LIST, by_expert != 0, e, list, scratch);
    const TW* w = w_down + (size_t)e * width * ff;
    const int c0 = blockIdx.y * rows_per_block, c_end = min(width, c0 + rows_per_block);
    const bool wide = wide_rows(w_down, ff);
    for (int at = 0; at < n; at += at_once) {
        const int count = min(at_once, n - at);
        __syncthreads();
        for (int k = 0; k < count; ++k) {
            const T* x = act + (size_t)list[at + k] * ff;
            for (int i = threadIdx.x; i < ff; i += UP_WARPS * 32) as[k * ff + i] = to_float(x[i]);
        }
        __syncthreads();
        if (count == 1) down_rows<TW, 1>(as, list + at, count, w, parts, width, ff, wide, c0, c_end);
        else if (count == 2) down_rows<TW, 2>(as, list + at, count, w, parts, width, ff, wide, c0, c_end);
        else down_rows<TW, MAX_NT>(as, list + at, count, w, parts, width, ff, wide, c0, c_end);
    }
}

// ---- a pair, a token at a time: every pair streams its expert's rows by itself.  The sums are those of the kernels above.  Measured
// (us, lists / here): 64 tokens, 2 of 6 experts of 70 x 30: 55 / 5.9; 256 tokens, 2 of 8 of 256 x 128, 32-bit: 111 / 33.

// grid (pairs, chunks of ff)
template <typename T, typename TW>
__global__ void __launch_bounds__(UP_WARPS * 32, 4) pair_up_kernel(const T* __restrict__ h, const TW* __restrict__ w_gate_up, const int* __restrict__ ids,
                                                                T* __restrict__ act, int width, int ff, int top, int rows_per_block) {
    extern __shared__ __align__(16) unsigned char expert_smem[];
    float* xs = reinterpret_cast<float*>(expert_smem);  // [width]
    pdl_launch_dependents();
    pdl_wait();
    const int pair = blockIdx.x;
    const TW* wg = w_gate_up + (size_t)ids[pair] * 2 * ff * width;
    const T* x = h + (size_t)(pair / top) * width;
    for (int i = threadIdx.x; i < width; i += UP_WARPS * 32) xs[i] = to_float(x[i]);
    __syncthreads();
    const int f0 = blockIdx.y * rows_per_block;
    up_rows<T, TW, 1, false>(xs, &pair, 1, wg, wg + (size_t)ff * width, act, width, ff, false, f0, min(ff, f0 + rows_per_block));
}

// The dot products of NR vectors in shared memory, `stride` apart, with a row of their own each (dot_many's order).
template <typename TW, int NR>
__device__ __forceinline__ void dot_pairs(const float* __restrict__ x, int stride, const TW* const (&rows)[NR], int n, int lane, float (&acc)[NR]) {
#pragma unroll
    for (int j = 0; j < NR; ++j) acc[j] = 0.f;
    constexpr int VEC = 16 / sizeof(TW);
    if (n % VEC == 0 && starts_on(rows[0], 16)) {  // the other rows are whole rows away
#pragma unroll 2
        for (int i = lane * VEC; i < n; i += 32 * VEC) {
            uint4 raw[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) raw[j] = *reinterpret_cast<const uint4*>(rows[j] + i);
#pragma unroll
            for (int j = 0; j < NR; ++j) {
                const float* xj = x + j * stride + i;
                if constexpr (sizeof(TW) == 2) {
                    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw[j]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float2 f = __bfloat1622float2(p[c]);
                        acc[j] = fmaf(xj[2 * c], f.x, acc[j]);
                        acc[j] = fmaf(xj[2 * c + 1], f.y, acc[j]);
                    }
                } else {
                    const float* f = reinterpret_cast<const float*>(&raw[j]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[j] = fmaf(xj[c], f[c], acc[j]);
                }
            }
        }
    } else {
        for (int i = lane; i < n; i += 32)
#pragma unroll
            for (int j = 0; j < NR; ++j) acc[j] = fmaf(x[j * stride + i], to_float(rows[j][i]), acc[j]);
    }
}

template <int N>
struct Count {
    static constexpr int value = N;
};

// grid (tokens, chunks of width): the down product of a token's pairs and their sum
template <typename T, typename TW>
__global__ void __launch_bounds__(UP_WARPS * 32) token_down_kernel(const T* __restrict__ act, const TW* __restrict__ w_down, const int* __restrict__ ids,
                                                                   const float* __restrict__ weights, const T* __restrict__ add,
                                                                   const float* __restrict__ add_weight, float* __restrict__ out, int width, int ff,
                                                                   int top, int rows_per_block) {
    extern __shared__ __align__(16) unsigned char expert_smem[];
    float* as = reinterpret_cast<float*>(expert_smem);  // [top][ff]
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    for (int i = threadIdx.x; i < top * ff; i += UP_WARPS * 32) as[i] = to_float(act[t * top * ff + i]);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = blockIdx.y * rows_per_block;
    for (int c = c0 + warp; c < min(width, c0 + rows_per_block); c += UP_WARPS) {
        float acc = add != nullptr ? to_float(add[t * width + c]) : 0.f;
        if (add_weight != nullptr) acc *= add_weight[t];
        int kk = 0;
        const auto add_pairs = [&](auto count) {  // their rows in flight together; the sum still takes them in the order they were chosen
            constexpr int NR = decltype(count)::value;
            const TW* rows[NR];
            float part[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) rows[j] = w_down + ((size_t)ids[t * top + kk + j] * width + c) * ff;
            dot_pairs<TW, NR>(as + (size_t)kk * ff, ff, rows, ff, lane, part);
#pragma unroll
            for (int j = 0; j < NR; ++j) acc = fmaf(weights[t * top + kk + j], warp_sum(part[j]), acc);
            kk += NR;
        };
        while (kk + 4 <= top) add_pairs(Count<4>{});
        if (kk + 2 <= top) add_pairs(Count<2>{});
        if (kk < top) add_pairs(Count<1>{});
        if (lane == 0) out[t * width + c] = acc;
    }
}

// ---- the same products on the tensor cores, for bfloat16 rows and weights of sizes in whole tiles (mma.sync m16n8k16, 32-bit sums)
//
// A block has sixteen rows of an expert's matrix at a time (of gate and of up together), each of its four warps a quarter of
// the reduction, and the tokens that chose the expert are the product's columns, eight or sixteen of them.  The order in which
// a product walks k is free as long as both operands take the same one, so a lane reads eight neighbouring entries of its row
// at once (16 bytes) and they serve as its fragments of two products; the tokens' rows lie in shared memory and are read the
// same way.  What remains is the stream of the weights, an expert's rows once for sixteen of its tokens (for eight where rows are longer
// than some 1,500 entries: two blocks an SM would not hold sixteen) and for every list of 512 pairs.  Blocks stay
// and take equal runs of (expert, sixteen rows) units: the experts that were chosen are listed by every block for itself.  (One block a pair
// and chunk of rows, most of which found that another had their expert, spent their time in the chain ids - list - weights - tokens.)
//
// The weights come by TMA, boxes of sixteen rows x 64 entries into a ring of every warp's own that runs on across the ends of units, in two to
// four blocks an SM.  (Loads into registers had four pieces in flight that ended with every unit, and went through
// the load unit 64 bytes of a row at a time: 400 cycles a piece and warp, which also held for copies of 16 bytes into a ring.)
// (Tensor-memory products would want 128 rows a tile, for a step that does next to no arithmetic.)
// Measured (us, cold; up, down and join; loads into registers / here): 6 of 64 experts of 2,048 x 1,024: 8 tokens 125 / 95, 42: 232 / 172; 4 of
// 32 of 1,024 x 768: 16 tokens 54 / 42, 63: 68 / 55; 2 of 16 of 4,096 x 1,536: 16 tokens 178 / 120, 120: 346 / 228; of 1,024 x 4,096, 120: 191 / 177.
// Every pair by itself on the FP32 pipes: 8 tokens 170 and 43, 42 and 63 tokens 763 and 265.  Bound by the weights (4.7 TB/s of them in the
// whole call of 8 tokens) with 6 us of launch and list before the first of them, by the tokens' products where an expert has sixteen and more.
constexpr int MMA_WARPS = 4, MMA_TOKENS = 16, MMA_LIST = 512;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// bytes from one token's row in shared memory to the next: 64 beyond a multiple of 128, so that the eight lanes that read
// together (two rows, four pieces) fall into different banks
__host__ __device__ constexpr int mma_stride(int k) { return (k * 2 + 127) / 128 * 128 + 64; }

// rows of `source` (`divide` pairs share one) for pairs[0 .. count - 1] into shared memory; what stands in the rows behind them
// is multiplied into columns that nobody reads
__device__ __forceinline__ void mma_stage(unsigned char* xs, int stride, const __nv_bfloat16* __restrict__ source, const int* pairs, int count, int divide, int k) {
    const int pieces = k / 8;
#pragma unroll 8
    for (int i = threadIdx.x; i < count * pieces; i += MMA_WARPS * 32) {
        const int t = i / pieces, c = i - t * pieces;
        *reinterpret_cast<uint4*>(xs + t * stride + c * 16) = *reinterpret_cast<const uint4*>(source + (size_t)(pairs[t] / divide) * k + c * 8);
    }
}

// ---- TMA: a warp's boxes of sixteen rows, each waited for on a barrier of its own; waits are bounded
constexpr uint32_t EXPERT_SPINS = 1u << 24;

__device__ __forceinline__ uint32_t smem_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool box_wait(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < EXPERT_SPINS; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_address(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// A warp's boxes of 16 rows x `box_k` entries (64, or 32 where rows have no more) of NM matrices, DEPTH of them ahead of the products
// and across the ends of units.
template <int NM, int DEPTH>
struct BoxRing {
    static constexpr int SLOT = NM * 16 * 128;  // bytes
    unsigned char* slots;
    uint64_t* full;
    int asked = 0, taken = 0, put = 0, take = 0;
    uint32_t phase = 0;
    bool ok = true;
    // one lane asks; the whole warp has read what stood in the place before.  Behind a wait that was given up nothing more is asked for.
    __device__ __forceinline__ void ask(const CUtensorMap* map, int k, int row, int rows_apart, int box_k, bool elected) {
        if (elected) {
            const uint32_t bar = smem_address(full + put);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(NM * 16 * box_k * 2) : "memory");
#pragma unroll
            for (int m = 0; m < NM; ++m)
                asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                                 smem_address(slots + put * SLOT + m * 16 * 128)),
                             "l"(reinterpret_cast<uint64_t>(map)), "r"(k), "r"(row + m * rows_apart), "r"(bar)
                             : "memory");
        }
        ++asked;
        put = put + 1 == DEPTH ? 0 : put + 1;
    }
    // Every lane waits for itself; one that gave up stays at the box that it gave up, so that drain() waits for it again.
    __device__ __forceinline__ const unsigned char* next() {
        if (ok) ok = box_wait(full + take, phase);
        return slots + take * SLOT;
    }
    __device__ __forceinline__ void pass() {
        ++taken;
        take = take + 1 == DEPTH ? 0 : take + 1;
        if (take == 0) phase ^= 1;
    }
    __device__ __forceinline__ void done() {
        if (ok) pass();
    }
    __device__ __forceinline__ void drain() {  // nothing may land in shared memory after the block is gone
        for (; taken < asked; pass()) box_wait(full + take, phase);
    }
};

// the sum of one entry over the warps
template <int N>
__device__ __forceinline__ float mma_sum(const float (*part)[N][32], int entry, int lane) {
    return ((part[0][entry][lane] + part[1][entry][lane]) + part[2][entry][lane]) + part[3][entry][lane];
}

// A run of up to `at_once` pairs of one expert: places `start` .. of the pairs in the order of their experts.
struct MmaRun {
    int expert, start, count;
};

// The pairs ids[first .. last - 1] (at most MMA_LIST) in the order of their experts, an expert's in their own order, and their runs:
// all blocks come to the same list, so that each may take some of a run's rows.  `counts`: 2 n_experts + MMA_LIST ints of shared
// memory.  Returns the number of runs.
__device__ __forceinline__ int mma_list(const int* __restrict__ ids, int first, int last, int n_experts, int at_once, int* counts, int* list, MmaRun* runs, int* n_runs) {
    constexpr int THREADS = MMA_WARPS * 32;
    if (last - first <= 32) {  // a few tokens: one warp, a lane a pair, the experts in the order of their first pairs
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x, i = first + lane, e = i < last ? ids[i] : -1 - lane;
            const unsigned int same = __match_any_sync(0xffffffffu, e);
            const int rank = __popc(same & ((1u << lane) - 1)), leader = __ffs(same) - 1;
            const int mine = i < last && rank == 0 ? __popc(same) : 0, mine_runs = (mine + at_once - 1) / at_once;
            int upto = mine, upto_runs = mine_runs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, upto, o), b = __shfl_up_sync(0xffffffffu, upto_runs, o);
                if (lane >= o) upto += a, upto_runs += b;
            }
            const int start = __shfl_sync(0xffffffffu, upto - mine, leader);
            if (i < last) list[start + rank] = i;
            for (int r = 0; r < mine_runs; ++r) runs[upto_runs - mine_runs + r] = MmaRun{e, start + r * at_once, min(at_once, mine - r * at_once)};
            if (lane == 31) *n_runs = upto_runs;
        }
        __syncthreads();
        return *n_runs;
    }
    int *starts = counts + n_experts, *expert_of = starts + n_experts;
    for (int e = threadIdx.x; e < n_experts; e += THREADS) counts[e] = 0;
    __syncthreads();
    for (int i = first + threadIdx.x; i < last; i += THREADS) {
        expert_of[i - first] = ids[i];
        atomicAdd(&counts[ids[i]], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int pairs = 0, all = 0;  // of the experts before
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int e = e0 + lane, mine = e < n_experts ? counts[e] : 0, mine_runs = (mine + at_once - 1) / at_once;
            int upto = mine, upto_runs = mine_runs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int a = __shfl_up_sync(0xffffffffu, upto, o), b = __shfl_up_sync(0xffffffffu, upto_runs, o);
                if (lane >= o) upto += a, upto_runs += b;
            }
            const int start = pairs + upto - mine;
            if (e < n_experts) starts[e] = start;
            for (int r = 0; r < mine_runs; ++r) runs[all + upto_runs - mine_runs + r] = MmaRun{e, start + r * at_once, min(at_once, mine - r * at_once)};
            pairs += __shfl_sync(0xffffffffu, upto, 31);
            all += __shfl_sync(0xffffffffu, upto_runs, 31);
        }
        if (lane == 0) *n_runs = all;
        __syncwarp();
        for (int i0 = first; i0 < last; i0 += 32) {
            const int i = i0 + lane;
            const unsigned int there = __ballot_sync(0xffffffffu, i < last);
            if (i < last) {
                const int e = expert_of[i - first];
                const unsigned int same = __match_any_sync(there, e);
                const int before = __popc(same & ((1u << lane) - 1)), at = starts[e];
                list[at + before] = i;
                __syncwarp(there);
                if (before == 0) starts[e] = at + __popc(same);
            }
            __syncwarp();
        }
    }
    __syncthreads();
    return *n_runs;
}

// UP: gate and up rows, act[pair] = silu(gate) * up; else rows of w_down, parts[pair].  k entries a row, n_rows rows a matrix; `map`: all
// experts' rows one after another.
template <bool UP, int DEPTH>
__global__ void __launch_bounds__(MMA_WARPS * 32) experts_mma_kernel(
    const __grid_constant__ CUtensorMap map, const __nv_bfloat16* __restrict__ source, const int* __restrict__ ids, __nv_bfloat16* __restrict__ act,
    float* __restrict__ parts, int n_pairs, int k, int n_rows, int divide, int n_experts, int at_once, int box_k, int* error_flag) {
    constexpr int NM = UP ? 2 : 1, ENTRIES = NM * MMA_TOKENS / 8 * 4;
    extern __shared__ __align__(128) unsigned char ring_smem[];  // the rings [MMA_WARPS][DEPTH]; the tokens' rows [at_once][stride], before that counts
    __shared__ int list[MMA_LIST], n_runs;
    __shared__ MmaRun runs[MMA_LIST];
    __shared__ float part[MMA_WARPS][ENTRIES][32];
    __shared__ __align__(8) uint64_t full[MMA_WARPS][DEPTH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    if (threadIdx.x < MMA_WARPS * DEPTH) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_address(&full[0][0] + threadIdx.x)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    pdl_launch_dependents();
    pdl_wait();
    unsigned char* staged_rows = ring_smem + MMA_WARPS * DEPTH * BoxRing<NM, DEPTH>::SLOT;
    const int first_pair = blockIdx.z * MMA_LIST, last_pair = min(first_pair + MMA_LIST, n_pairs);
    const int tiles = n_rows / 16;
    // (a barrier of the block stands in here)
    const long long units = (long long)mma_list(ids, first_pair, last_pair, n_experts, at_once, (int*)staged_rows, list, runs, &n_runs) * tiles;
    const int stride = mma_stride(k), pieces = k / 32, share = (pieces + MMA_WARPS - 1) / MMA_WARPS, per = box_k / 32, pitch = box_k * 2;
    const int begin = min(warp * share, pieces), end = min(begin + share, pieces);
    int unit = (int)(units * blockIdx.x / gridDim.x);
    const int unit_end = (int)(units * (blockIdx.x + 1) / gridDim.x);
    BoxRing<NM, DEPTH> ring{ring_smem + warp * DEPTH * BoxRing<NM, DEPTH>::SLOT, full[warp]};
    int ahead = begin < end ? unit : unit_end, piece = begin, row = 0;  // what is asked for next
    const auto point = [&]() {
        if (ahead < unit_end) row = runs[ahead / tiles].expert * NM * n_rows + (ahead % tiles) * 16;
    };
    const auto ask = [&]() {
        if (ahead >= unit_end || !ring.ok) return;
        ring.ask(&map, piece * 32, row, n_rows, box_k, lane == 0);
        piece += per;
        if (piece >= end) {
            piece = begin;
            ++ahead;
            point();
        }
    };
    point();
    for (int i = 0; i < DEPTH; ++i) ask();
    for (int staged = -1; unit < unit_end; ++unit) {
        const int at = unit / tiles, tile = unit % tiles, count = runs[at].count, NB = count <= 8 ? 1 : 2;
        const int* pairs = list + runs[at].start;
        if (at != staged) {  // all warps are through with the rows of before: they stand behind the barrier after their sums
            mma_stage(staged_rows, stride, source, pairs, count, divide, k);
            staged = at;
        }
        __syncthreads();
        const unsigned char* x = staged_rows + g * stride + q * 16;
        float sums[NM][2][4];
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int e = 0; e < 4; ++e) sums[m][b][e] = 0.f;
        for (int i = begin; i < end; i += per) {
            const unsigned char* box = ring.next() + g * pitch + q * 16;
            const int here = min(per, end - i);
            uint4 lo[2][NM], hi[2][NM], v[2][2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u >= here) continue;
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    lo[u][m] = *reinterpret_cast<const uint4*>(box + m * 16 * 128 + u * 64);
                    hi[u][m] = *reinterpret_cast<const uint4*>(box + m * 16 * 128 + u * 64 + 8 * pitch);
                }
                v[u][0] = *reinterpret_cast<const uint4*>(x + (i + u) * 64);
                if (NB == 2) v[u][1] = *reinterpret_cast<const uint4*>(x + (i + u) * 64 + 8 * stride);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (u >= here) continue;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (b >= NB) continue;
#pragma unroll
                    for (int m = 0; m < NM; ++m) {
                        mma_bf16(sums[m][b], lo[u][m].x, hi[u][m].x, lo[u][m].y, hi[u][m].y, v[u][b].x, v[u][b].y);
                        mma_bf16(sums[m][b], lo[u][m].z, hi[u][m].z, lo[u][m].w, hi[u][m].w, v[u][b].z, v[u][b].w);
                    }
                }
            }
            ring.done();
            __syncwarp();  // the place is free
            ask();
        }
#pragma unroll
        for (int m = 0; m < NM; ++m)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (b < NB) part[warp][(m * NB + b) * 4 + e][lane] = sums[m][b][e];
        __syncthreads();
        // entry (b, i) of lane (g, q): token 8 b + 2 q + i % 2, row g + 8 (i / 2)
        for (int entry = warp; entry < NB * 4; entry += MMA_WARPS) {
            const int t = (entry >> 2) * 8 + q * 2 + (entry & 1), row_out = tile * 16 + g + ((entry >> 1) & 1) * 8;
            if (t >= count) continue;
            const float sum = mma_sum<ENTRIES>(part, entry, lane);
            if constexpr (UP) act[(size_t)pairs[t] * n_rows + row_out] = __float2bfloat16_rn(sum / (1.f + expf(-sum)) * mma_sum<ENTRIES>(part, NB * 4 + entry, lane));
            else parts[(size_t)pairs[t] * n_rows + row_out] = sum;
        }
        // the next unit's first barrier stands before `part` is written again
    }
    if (!__all_sync(0xffffffffu, ring.ok) && lane == 0) atomicExch(error_flag, 71);
    ring.drain();
}

// ---- the same for so few pairs that their experts are nearly all different: no list, no third kernel, and a pair's row is the
// product's column (all eight of them).  A column's sums are those of the kernel above, so a token's result does not depend on
// which of the two its step takes.  Bound by two launches and the chain ids - rows - sums in each of them; a block asks for all of
// its rows (64 KB of gate and up at 1,024) at once.
// Measured (us), every pair by itself on the FP32 pipes / lists / here: 4 of 32 experts of 1,024 x 768: one token 9.4 / 11.7 / 8.4, 3:
// 18.5 / 19.4 / 13.4; 6 of 64 of 2,048 x 1,024, one token: 26.6 / 21.4 / 19.1; 2 of 8 of 256 x 128: one token 4.3 / 8.8 / 4.5, 64: 12.7 /
// 13.5 / 10.2.

// This warp's quarter of sixteen rows of NM matrices (row0: this lane's row of each) times one vector: the sums of column 0 come to
// rest in lanes 0, 4, ... 28, rows lane / 4 and lane / 4 + 8.
template <int NM>
__device__ __forceinline__ void mma_column(const __nv_bfloat16* const (&row0)[NM], const __nv_bfloat16* __restrict__ x, int k, int begin, int end, float (&sums)[NM][4]) {
    constexpr int STEPS = 4;
    const __nv_bfloat16* x_at = x + (threadIdx.x & 3) * 8;
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) sums[m][e] = 0.f;
    for (int i = begin; i < end; i += STEPS) {
        uint4 lo[STEPS][NM], hi[STEPS][NM], xv[STEPS];
#pragma unroll
        for (int u = 0; u < STEPS; ++u)
            if (i + u < end) {
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    const __nv_bfloat16* at = row0[m] + (i + u) * 32;
                    lo[u][m] = *reinterpret_cast<const uint4*>(at);
                    hi[u][m] = *reinterpret_cast<const uint4*>(at + (size_t)8 * k);
                }
                xv[u] = *reinterpret_cast<const uint4*>(x_at + (i + u) * 32);
            }
#pragma unroll
        for (int u = 0; u < STEPS; ++u)
            if (i + u < end) {
#pragma unroll
                for (int m = 0; m < NM; ++m) {
                    mma_bf16(sums[m], lo[u][m].x, hi[u][m].x, lo[u][m].y, hi[u][m].y, xv[u].x, xv[u].y);
                    mma_bf16(sums[m], lo[u][m].z, hi[u][m].z, lo[u][m].w, hi[u][m].w, xv[u].z, xv[u].w);
                }
            }
    }
}

// grid (pairs, tiles of sixteen rows)
__global__ void __launch_bounds__(MMA_WARPS * 32) pair_up_mma_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ weights,
                                                                     const int* __restrict__ ids, __nv_bfloat16* __restrict__ act, int k, int n_rows, int top) {
    __shared__ float part[MMA_WARPS][2][16];
    pdl_launch_dependents();
    pdl_wait();
    const int pair = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int pieces = k / 32, share = (pieces + MMA_WARPS - 1) / MMA_WARPS, begin = min(warp * share, pieces), end = min(begin + share, pieces);
    const __nv_bfloat16* gate = weights + (size_t)ids[pair] * 2 * n_rows * k + (size_t)(blockIdx.y * 16 + g) * k + q * 8;
    const __nv_bfloat16* const rows[2] = {gate, gate + (size_t)n_rows * k};
    float sums[2][4];
    mma_column<2>(rows, h + (size_t)(pair / top) * k, k, begin, end, sums);
    if (q == 0) {
#pragma unroll
        for (int m = 0; m < 2; ++m) part[warp][m][g] = sums[m][0], part[warp][m][g + 8] = sums[m][2];
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        const int r = threadIdx.x;
        const float z = ((part[0][0][r] + part[1][0][r]) + part[2][0][r]) + part[3][0][r], up = ((part[0][1][r] + part[1][1][r]) + part[2][1][r]) + part[3][1][r];
        act[(size_t)pair * n_rows + blockIdx.y * 16 + r] = __float2bfloat16_rn(z / (1.f + expf(-z)) * up);
    }
}

// grid (tokens, tiles of sixteen columns of the result): four warps a pair, up to TOKEN_PAIRS pairs of the token at a time
constexpr int TOKEN_PAIRS = 4;
__global__ void __launch_bounds__(TOKEN_PAIRS * MMA_WARPS * 32) token_down_mma_kernel(
    const __nv_bfloat16* __restrict__ act, const __nv_bfloat16* __restrict__ weights, const int* __restrict__ ids, const float* __restrict__ pair_weights,
    const __nv_bfloat16* __restrict__ add, const float* __restrict__ add_weight, float* __restrict__ out, int k, int n_rows, int top) {
    __shared__ float part[2][TOKEN_PAIRS][MMA_WARPS][16];
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    const int lane = threadIdx.x & 31, group = threadIdx.x / (MMA_WARPS * 32), groups = blockDim.x / (MMA_WARPS * 32), warp = (threadIdx.x >> 5) % MMA_WARPS;
    const int g = lane >> 2, q = lane & 3, column = blockIdx.y * 16 + threadIdx.x;
    const int pieces = k / 32, share = (pieces + MMA_WARPS - 1) / MMA_WARPS, begin = min(warp * share, pieces), end = min(begin + share, pieces);
    float acc = 0.f;
    if (threadIdx.x < 16 && add != nullptr) acc = to_float(add[t * n_rows + column]);
    if (threadIdx.x < 16 && add_weight != nullptr) acc *= add_weight[t];
    for (int kk0 = 0, turn = 0; kk0 < top; kk0 += groups, turn ^= 1) {
        const int kk = kk0 + group;
        if (kk < top) {
            const __nv_bfloat16* const rows[1] = {weights + (size_t)ids[t * top + kk] * n_rows * k + (size_t)(blockIdx.y * 16 + g) * k + q * 8};
            float sums[1][4];
            mma_column<1>(rows, act + (t * top + kk) * k, k, begin, end, sums);
            if (q == 0) part[turn][group][warp][g] = sums[0][0], part[turn][group][warp][g + 8] = sums[0][2];
        }
        __syncthreads();  // two sets of parts in turn: one barrier a turn
        if (threadIdx.x < 16)
            for (int j = 0; j < groups && kk0 + j < top; ++j) {
                const float (*p)[16] = part[turn][j];
                const int r = threadIdx.x;
                acc = fmaf(pair_weights[t * top + kk0 + j], ((p[0][r] + p[1][r]) + p[2][r]) + p[3][r], acc);
            }
    }
    if (threadIdx.x < 16) out[t * n_rows + column] = acc;
}

// out_t = add_t (times add_weight_t) + the token's parts times their weights, in the order they were chosen
template <typename T>
__global__ void experts_join_kernel(const float* __restrict__ parts, const float* __restrict__ weights, const T* __restrict__ add,
                                    const float* __restrict__ add_weight, float* __restrict__ out, int width, int top) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= width) return;
    float acc = add != nullptr ? to_float(add[t * width + c]) : 0.f;
    if (add_weight != nullptr) acc *= add_weight[t];
    const float* p = parts + t * top * width + c;
#pragma unroll 4
    for (int kk = 0; kk < top; ++kk) acc = fmaf(weights[t * top + kk], p[(size_t)kk * width], acc);
    out[t * width + c] = acc;
}

// ---- pairs in the order of their experts, for products that take all rows of an expert at once
// One block.  ends[e] = one past the last place of expert e (cumulative counts); place_of[pair] = the pair's place in
// that order; pair_at[place] = the pair that stands there.  Which of an expert's pairs gets which of its places is
// settled by atomic counters and may differ from run to run; a row's product does not depend on its place.
constexpr int SORT_THREADS = 1024;

__global__ void __launch_bounds__(SORT_THREADS) experts_sort_kernel(const int* __restrict__ ids, int n_pairs, int n_experts,
                                                                    int* __restrict__ ends, int* __restrict__ place_of,
                                                                    int* __restrict__ pair_at) {
    extern __shared__ int sort_smem[];  // counts [E] | starts [E]
    pdl_launch_dependents();
    int* counts = sort_smem;
    int* starts = sort_smem + n_experts;
    for (int e = threadIdx.x; e < n_experts; e += SORT_THREADS) counts[e] = 0;
    __syncthreads();
    pdl_wait();
    for (int i = threadIdx.x; i < n_pairs; i += SORT_THREADS) atomicAdd(&counts[ids[i]], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0;
        for (int e = 0; e < n_experts; ++e) {
            starts[e] = at;
            at += counts[e];
            ends[e] = at;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_pairs; i += SORT_THREADS) {
        const int place = atomicAdd(&starts[ids[i]], 1);
        place_of[i] = place;
        pair_at[place] = i;
    }
}

// out[place] = x[pair_at[place] / top]: the rows of the tokens in the order of their experts
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ x, const int* __restrict__ pair_at, T* __restrict__ out, int width, int top) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t place = blockIdx.x;
    const T* src = x + (size_t)(pair_at[place] / top) * width;
    T* dst = out + place * width;
    if ((width * sizeof(T)) % 16 == 0 && starts_on(x, 16) && starts_on(out, 16)) {
        const int n16 = width * (int)sizeof(T) / 16;
        for (int i = threadIdx.x; i < n16; i += blockDim.x) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    } else {
        for (int i = threadIdx.x; i < width; i += blockDim.x) dst[i] = src[i];
    }
}

// out_t = add_t + sum_k weights[t, k] * y[place_of[t, k]] in the order the experts were chosen (32-bit)
template <typename T>
__global__ void experts_combine_kernel(const T* __restrict__ y, const int* __restrict__ place_of, const float* __restrict__ weights,
                                       const T* __restrict__ add, const float* __restrict__ add_weight, float* __restrict__ out,
                                       int width, int top) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t t = blockIdx.x;
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
        float acc = add != nullptr ? to_float(add[t * width + c]) : 0.f;
        if (add_weight != nullptr) acc *= add_weight[t];
        for (int kk = 0; kk < top; ++kk)
            acc = fmaf(weights[t * top + kk], to_float(y[(size_t)place_of[t * top + kk] * width + c]), acc);
        out[t * width + c] = acc;
    }
}

}  // namespace

GK_EXPORT int gk_experts_sort(const int* ids, int n_pairs, int n_experts, int* ends, int* place_of, int* pair_at, void* stream) {
    GK_REQUIRE(n_pairs >= 0 && n_experts > 0 && n_experts <= 4096, "experts_sort: bad sizes");
    gk_launch(experts_sort_kernel, dim3(1), dim3(SORT_THREADS), (size_t)2 * n_experts * sizeof(int), (cudaStream_t)stream, ids, n_pairs,
              n_experts, ends, place_of, pair_at);
    GK_CHECK_LAUNCH("experts_sort");
    return GK_OK;
}

GK_EXPORT int gk_gather_rows(const void* x, int dtype, const int* pair_at, void* out, int n_places, int width, int top, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(dtype) && width > 0 && top > 0, "gather_rows: bad arguments");
    if (n_places == 0) return GK_OK;
    GK_DISPATCH_DTYPE(dtype, T, {
        gk_launch(gather_rows_kernel<T>, dim3(n_places), dim3(128), 0, (cudaStream_t)stream, (const T*)x, pair_at, (T*)out, width, top);
    })
    GK_CHECK_LAUNCH("gather_rows");
    return GK_OK;
}

GK_EXPORT int gk_experts_combine(const void* y, int dtype, const int* place_of, const float* weights, const void* add,
                                 const float* add_weight, float* out, int n_tokens, int width, int top, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(dtype) && width > 0 && top > 0 && (add != nullptr || add_weight == nullptr), "experts_combine: bad arguments");
    if (n_tokens == 0) return GK_OK;
    GK_DISPATCH_DTYPE(dtype, T, {
        gk_launch(experts_combine_kernel<T>, dim3(n_tokens), dim3(256), 0, (cudaStream_t)stream, (const T*)y, place_of, weights,
                  (const T*)add, add_weight, out, width, top);
    })
    GK_CHECK_LAUNCH("experts_combine");
    return GK_OK;
}

// shared: w_router and z have one row more, the shared expert's number; its sigmoid goes to shared_weight [T] or, where that is
// null, to one more pair a token (ids and weights [T, top + 1]).
GK_EXPORT int gk_route_groups(const void* h, int dtype, const float* w_router, const float* correction, float* z, int* ids,
                              float* weights, int n_tokens, int width, int n_experts, int top, int n_groups, int keep, float scale, int flags,
                              int shared, float* shared_weight, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(dtype), "route_groups: bad dtype %d", dtype);
    GK_REQUIRE(n_experts > 0 && top > 0 && top <= n_experts, "route_groups: %d of %d experts", top, n_experts);
    GK_REQUIRE(n_groups >= 1 && n_experts % n_groups == 0 && keep >= 1 && keep <= n_groups, "route_groups: %d groups, %d kept, %d experts",
               n_groups, keep, n_experts);
    GK_REQUIRE(top <= keep * (n_experts / n_groups), "route_groups: %d experts cannot come from %d groups of %d", top, keep,
               n_experts / n_groups);
    GK_REQUIRE(!(flags & ROUTE_LOGITS) || !(flags & (ROUTE_SOFTMAX | ROUTE_RENORMALISE)), "route_groups: logits have a rule of their own");
    if (n_tokens == 0) return GK_OK;
    const size_t smem = (size_t)ROUTE_WARPS * (2 * n_experts + n_groups) * sizeof(float);
    GK_REQUIRE(smem <= 48 * 1024, "route_groups: too many experts (%d)", n_experts);
    cudaStream_t s = (cudaStream_t)stream;
    const bool many = (long long)((n_tokens + 7) / 8) * ((n_experts + 7) / 8) >= 512;
    const int per_warp = many ? 8 : 2;
    const int token_groups = (n_tokens + 3) / 4;
    const int n_scores = n_experts + (shared ? 1 : 0), ld_pairs = top + (shared && shared_weight == nullptr ? 1 : 0);
    const long long units = (long long)token_groups * ((n_scores + per_warp - 1) / per_warp);
    GK_REQUIRE(units / ROUTE_WARPS < 2147483647LL, "route_groups: too many tokens");
    const dim3 score_grid((unsigned)((units + ROUTE_WARPS - 1) / ROUTE_WARPS));
    if (dtype == GK_BF16 && n_tokens >= 256 && width % 8 == 0 && (((uintptr_t)h | (uintptr_t)w_router) & 15) == 0) {
        const int tiles = (n_scores + 63) / 64, nj = ((n_scores + tiles - 1) / tiles + 15) / 16;
        const dim3 grid((n_tokens + SCORE_ROWS - 1) / SCORE_ROWS, tiles);
#define GK_TILED(NJ) \
    gk_launch(route_scores_tiled_kernel<NJ>, grid, dim3(256), 0, s, (const __nv_bfloat16*)h, w_router, z, n_tokens, width, n_scores)
        if (nj == 1) GK_TILED(1);
        else if (nj == 2) GK_TILED(2);
        else if (nj == 3) GK_TILED(3);
        else GK_TILED(4);
#undef GK_TILED
    } else GK_DISPATCH_DTYPE(dtype, T, {
        const size_t few = (size_t)width * (FEW_EXPERTS * sizeof(float) + FEW_TOKENS * sizeof(T));
        if (!many && width % 8 == 0 && (((uintptr_t)h | (uintptr_t)w_router) & 15) == 0 && few <= 160 * 1024) {
            if (few > 48 * 1024) cudaFuncSetAttribute(route_scores_few_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
            gk_launch(route_scores_few_kernel<T>, dim3((n_scores + FEW_EXPERTS - 1) / FEW_EXPERTS, (n_tokens + FEW_TOKENS - 1) / FEW_TOKENS), dim3(128), few, s,
                      (const T*)h, w_router, z, n_tokens, width, n_scores);
        } else if (per_warp == 8)
            gk_launch(route_scores_kernel<T, 8, 4>, score_grid, dim3(ROUTE_WARPS * 32), 0, s, (const T*)h, w_router, z, n_tokens, width, n_scores);
        else
            gk_launch(route_scores_kernel<T, 2, 4>, score_grid, dim3(ROUTE_WARPS * 32), 0, s, (const T*)h, w_router, z, n_tokens, width, n_scores);
    })
    GK_CHECK_LAUNCH("route_scores");
    gk_launch_behind(route_choose_kernel, dim3((n_tokens + ROUTE_WARPS - 1) / ROUTE_WARPS), dim3(ROUTE_WARPS * 32), smem, s, (const float*)z,
              correction, ids, weights, n_tokens, n_experts, top, n_groups, keep, scale, flags, n_scores, ld_pairs, shared_weight);
    GK_CHECK_LAUNCH("route_groups");
    return GK_OK;
}

namespace {

int sm_count() {
    static const int sms = [] {
        int device = 0, n = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) n = 148;
        return n;
    }();
    return sms;
}

// How the pairs of a step are dealt to blocks: by pair where those are fewer than the experts (blocks of an expert's later pairs
// leave at once), else by expert; an expert's rows are cut into chunks so that every SM finds some blocks' worth of work even if
// half of the pairs share their experts.
struct ExpertGrid {
    dim3 grid;
    int rows, by_expert, at_once;
    size_t smem;
    long long blocks() const { return (long long)grid.x * grid.y; }
};
constexpr int UP_ROWS = 2 * UP_WARPS, DOWN_ROWS = 4 * UP_WARPS;  // the least of a chunk: every warp has its rows in flight

ExpertGrid expert_grid(long long pairs, int n_experts, int n_rows, int row_length, int least_rows) {
    ExpertGrid g;
    g.by_expert = pairs > n_experts || pairs > LIST;
    const long long items = g.by_expert ? n_experts : pairs;
    int chunks = 1;
    while (items * chunks < 1184 && n_rows / (chunks * 2) >= least_rows) chunks *= 2;
    g.rows = (n_rows + chunks - 1) / chunks;
    g.grid = dim3((unsigned)items, (n_rows + g.rows - 1) / g.rows, (unsigned)((pairs + LIST - 1) / LIST));
    g.at_once = MAX_NT;
    while (g.at_once > 1 && (size_t)g.at_once * row_length * sizeof(float) > 64 * 1024) g.at_once /= 2;
    g.smem = (size_t)g.at_once * row_length * sizeof(float);
    return g;
}

// Whole tiles: rows of k entries in pieces of 32, sixteen rows a tile; eight tokens' rows fit in shared memory, and so do
// the experts' counts.
bool mma_suits(int k, int n_rows, int n_experts) {
    return k % 32 == 0 && n_rows % 16 == 0 && 8 * (size_t)mma_stride(k) <= 160 * 1024 && n_experts <= 4096;
}

constexpr size_t ring_bytes(bool up, int depth) { return (size_t)MMA_WARPS * depth * (up ? 2 : 1) * 16 * 128; }
// at most the shared memory of a block beside its rings and its tokens' rows: whole pieces of 128 bytes, and what the device keeps for itself
constexpr size_t mma_static_bytes(bool up, int depth) {
    return MMA_LIST * (sizeof(int) + sizeof(MmaRun)) + MMA_WARPS * ((up ? 2 : 1) * (MMA_TOKENS / 8 * 4) * 32 * sizeof(float) + depth * sizeof(uint64_t)) + 128 + 1024;
}

struct MmaStep {
    const void *source, *weights;
    const int* ids;
    void* act;
    float* parts;
    long long pairs;
    int n_tokens, k, n_rows, divide, n_experts;
    int* error_flag;
};

template <bool UP, int DEPTH>
int launch_ring(const MmaStep& p, int at_once, size_t staged, int blocks, cudaStream_t s) {
    CUtensorMap map;
    const int box_k = p.k < 64 ? 32 : 64;
    const int status = gk_matrix_map(&map, p.weights, (long long)p.n_experts * (UP ? 2 : 1) * p.n_rows, p.k, p.k, box_k, 16, false);
    if (status) return status;
    const long long most = std::min(p.pairs, (long long)MMA_LIST) * (p.n_rows / 16);
    cudaFuncSetAttribute(experts_mma_kernel<UP, DEPTH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(228 * 1024 - mma_static_bytes(UP, DEPTH)));
    // the down product stands behind the up product of the same call
    gk_launch_with(gk_early(!UP || t_gk_chain == 2), experts_mma_kernel<UP, DEPTH>,
                   dim3((unsigned)std::min(most, (long long)blocks * sm_count()), 1, (unsigned)((p.pairs + MMA_LIST - 1) / MMA_LIST)), dim3(MMA_WARPS * 32),
                   staged + ring_bytes(UP, DEPTH), s, dim3(1, 1, 1), map, (const __nv_bfloat16*)p.source, p.ids, (__nv_bfloat16*)p.act, p.parts, (int)p.pairs,
                   p.k, p.n_rows, p.divide, p.n_experts, at_once, box_k, p.error_flag);
    return GK_OK;
}

template <bool UP>
int launch_mma(const MmaStep& p, cudaStream_t s) {
    const int at_once = p.n_tokens > 8 && MMA_TOKENS * (size_t)mma_stride(p.k) <= 48 * 1024 ? MMA_TOKENS : 8;
    const size_t rows = (size_t)at_once * mma_stride(p.k), counts = (2 * (size_t)p.n_experts + MMA_LIST) * 4, staged = ((rows > counts ? rows : counts) + 127) / 128 * 128;
    // As many blocks an SM as find room beside the tokens' rows, up to three (up) and four (down), with rings as deep as that leaves; one block
    // with 128 KB of rings only where two do not fit.  What a block has to do for a box (a warp a scheduler) weighs more than the boxes in
    // flight.  Measured (us, whole call; two blocks with rings of 48 KB, or one with 128 KB where rows are 4,096 / here): 2 of 16 experts of 4,096
    // x 1,536: 16 tokens 158 / 118, 63: 245 / 169; of 1,024 x 4,096: 120 tokens 226 / 182; 2 of 64 of 4,096 x 512: 63 tokens 221 / 149; 4 of 64 of
    // 2,048 x 1,024: 16 tokens 130 / 117; 4 of 16 of 512 x 2,048: 63 tokens 73 / 60.
    const auto fits = [&](int blocks, int depth) { return blocks * (staged + ring_bytes(UP, depth) + mma_static_bytes(UP, depth)) <= 228 * 1024; };
    for (int blocks = UP ? 3 : 4; blocks >= 2; --blocks) {
        if (!fits(blocks, 2)) continue;
        if constexpr (UP) return fits(blocks, 3) ? launch_ring<UP, 3>(p, at_once, staged, blocks, s) : launch_ring<UP, 2>(p, at_once, staged, blocks, s);
        else return fits(blocks, 4) ? launch_ring<UP, 4>(p, at_once, staged, blocks, s) : launch_ring<UP, 2>(p, at_once, staged, blocks, s);
    }
    constexpr int DEEP = UP ? 8 : 16, FLAT = UP ? 2 : 4;
    return fits(1, DEEP) ? launch_ring<UP, DEEP>(p, at_once, staged, 1, s) : launch_ring<UP, FLAT>(p, at_once, staged, 1, s);
}

// Megabytes of weights that the pairs of a step fetch and that they would not if every expert came once (a token's experts are all
// different, two tokens' are chosen independently).
double repeated_megabytes(int n_tokens, int top, int n_experts, double expert_bytes) {
    const double different = n_experts * (1.0 - std::pow(1.0 - std::min(1.0, (double)top / n_experts), (double)n_tokens));
    return ((double)n_tokens * top - different) * expert_bytes * 1e-6;
}

struct ExpertStep {
    const void *h, *w_gate_up, *w_down;
    int dtype, w_dtype;
    const int* ids;
    const float* weights;
    const void* add;
    const float* add_weight;
    float* parts;  // 32-bit scratch [n_tokens * top, width]
    void* act;     // [n_tokens * top, ff] in the run's type
    float* out;
    int n_tokens, width, ff, top, n_experts;
    int* error_flag;
};

template <typename T>
void launch_join(const ExpertStep& p, cudaStream_t s) {
    gk_launch_behind(experts_join_kernel<T>, dim3(p.n_tokens, (p.width + 255) / 256), dim3(256), 0, s, (const float*)p.parts, p.weights, (const T*)p.add,
              p.add_weight, p.out, p.width, p.top);
}

// up: inner values of all pairs; down: their products and the sums.  Each on the tensor cores where its sizes are whole tiles, and
// each either a pair by itself or an expert's pairs together.
int up_mma(const ExpertStep& p, bool few, cudaStream_t s) {
    const long long pairs = (long long)p.n_tokens * p.top;
    if (!few) return launch_mma<true>(MmaStep{p.h, p.w_gate_up, p.ids, p.act, nullptr, pairs, p.n_tokens, p.width, p.ff, p.top, p.n_experts, p.error_flag}, s);
    gk_launch(pair_up_mma_kernel, dim3((unsigned)pairs, p.ff / 16), dim3(MMA_WARPS * 32), 0, s, (const __nv_bfloat16*)p.h, (const __nv_bfloat16*)p.w_gate_up,
              p.ids, (__nv_bfloat16*)p.act, p.width, p.ff, p.top);
    return GK_OK;
}

int down_mma(const ExpertStep& p, bool few, cudaStream_t s) {
    if (few) {
        const int turns = (p.top + TOKEN_PAIRS - 1) / TOKEN_PAIRS, groups = (p.top + turns - 1) / turns;
        gk_launch(token_down_mma_kernel, dim3(p.n_tokens, p.width / 16), dim3(groups * MMA_WARPS * 32), 0, s, (const __nv_bfloat16*)p.act,
                  (const __nv_bfloat16*)p.w_down, p.ids, p.weights, (const __nv_bfloat16*)p.add, p.add_weight, p.out, p.ff, p.width, p.top);
        return GK_OK;
    }
    const int status = launch_mma<false>(MmaStep{p.act, p.w_down, p.ids, nullptr, p.parts, (long long)p.n_tokens * p.top, p.n_tokens, p.ff, p.width, 1, p.n_experts, p.error_flag}, s);
    if (status) return status;
    launch_join<__nv_bfloat16>(p, s);
    return GK_OK;
}

template <typename T, typename TW>
void up_fp32(const ExpertStep& p, bool few, cudaStream_t s) {
    const long long pairs = (long long)p.n_tokens * p.top;
    if (few) {  // cut the experts' rows over more blocks, so that a single token still finds every SM a share
        int chunks = 1;
        while (pairs * chunks < 592 && p.ff / (chunks * 2) >= UP_WARPS) chunks *= 2;
        const int rows = (p.ff + chunks - 1) / chunks;
        const size_t smem = (size_t)p.width * sizeof(float);
        if (smem > 48 * 1024) cudaFuncSetAttribute(pair_up_kernel<T, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        gk_launch(pair_up_kernel<T, TW>, dim3((unsigned)pairs, (p.ff + rows - 1) / rows), dim3(UP_WARPS * 32), smem, s, (const T*)p.h, (const TW*)p.w_gate_up, p.ids,
                  (T*)p.act, p.width, p.ff, p.top, rows);
        return;
    }
    const ExpertGrid g = expert_grid(pairs, p.n_experts, p.ff, p.width, UP_ROWS);
    if (g.smem > 40 * 1024) cudaFuncSetAttribute(experts_up_kernel<T, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    gk_launch(experts_up_kernel<T, TW>, g.grid, dim3(UP_WARPS * 32), g.smem, s, (const T*)p.h, (const TW*)p.w_gate_up, p.ids, (T*)p.act, (int)pairs, p.width,
              p.ff, p.top, g.rows, g.by_expert, g.at_once);
}

template <typename T, typename TW>
void down_fp32(const ExpertStep& p, bool few, cudaStream_t s) {
    if (few) {
        int chunks = 1;
        while ((long long)p.n_tokens * chunks < 592 && p.width / (chunks * 2) >= UP_WARPS) chunks *= 2;
        const int rows = (p.width + chunks - 1) / chunks;
        const size_t smem = (size_t)p.top * p.ff * sizeof(float);
        if (smem > 48 * 1024) cudaFuncSetAttribute(token_down_kernel<T, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        gk_launch(token_down_kernel<T, TW>, dim3(p.n_tokens, (p.width + rows - 1) / rows), dim3(UP_WARPS * 32), smem, s, (const T*)p.act, (const TW*)p.w_down, p.ids,
                  p.weights, (const T*)p.add, p.add_weight, p.out, p.width, p.ff, p.top, rows);
        return;
    }
    const long long pairs = (long long)p.n_tokens * p.top;
    const ExpertGrid g = expert_grid(pairs, p.n_experts, p.width, p.ff, DOWN_ROWS);
    if (g.smem > 40 * 1024) cudaFuncSetAttribute(experts_down_kernel<T, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    gk_launch(experts_down_kernel<T, TW>, g.grid, dim3(UP_WARPS * 32), g.smem, s, (const T*)p.act, (const TW*)p.w_down, p.ids, p.parts, (int)pairs, p.width,
              p.ff, g.rows, g.by_expert, g.at_once);
    launch_join<T>(p, s);
}

int experts(const ExpertStep& p, cudaStream_t s) {
    const bool bf16 = p.dtype == GK_BF16 && p.w_dtype == GK_BF16;
    const bool mma_up = bf16 && mma_suits(p.width, p.ff, p.n_experts) && (((uintptr_t)p.h | (uintptr_t)p.w_gate_up) & 15) == 0;
    const bool mma_down = bf16 && mma_suits(p.ff, p.width, p.n_experts) && (((uintptr_t)p.act | (uintptr_t)p.w_down) & 15) == 0;
    const long long pairs = (long long)p.n_tokens * p.top;
    const double third = (double)p.ff * p.width * (p.w_dtype == GK_F32 ? 4 : 2), repeated = repeated_megabytes(p.n_tokens, p.top, p.n_experts, 3 * third);
    // A pair by itself where hardly any expert has two, or where the pairs' rows are little in all.  The lists cost some 4 us, as
    // much as fetching 8 MB again.  Measured (us, by itself / lists; tensor cores): 3 tokens, 5 of 33 experts of 1,024 x 768 (10 MB
    // again): 16.7 / 18.9, 4 tokens (19 MB): 20.4 / 19.6; 3 tokens, 6 of 64 of 2,048 x 1,024 (21 MB): 75.7 / 71.9.  On the FP32 pipes a
    // list serves four tokens at a time and wins later, and not where its blocks are few: 4 tokens, 6 of 64 of 2,048 x 1,024 in 32
    // bits (80 MB): 126.7 / 116; 3 tokens (40 MB): 88.6 / 100; 1,024 tokens, 2 of 8 of 256 x 128: 106 / 217.
    const bool few_mma = (repeated <= 8 || (double)pairs * 3e-6 * third <= 32) && p.width / 16 <= 65535 && p.ff / 16 <= 65535;
    const bool few_up = repeated <= 64 || expert_grid(pairs, p.n_experts, p.ff, p.width, UP_ROWS).blocks() < 2LL * sm_count();
    const bool few_down = repeated <= 64 || expert_grid(pairs, p.n_experts, p.width, p.ff, DOWN_ROWS).blocks() < 2LL * sm_count();
    int status = GK_OK;
    if (mma_up) status = up_mma(p, few_mma, s);
    else GK_DISPATCH_DTYPE(p.dtype, T, { GK_DISPATCH_DTYPE(p.w_dtype, TW, { up_fp32<T, TW>(p, few_up, s); }) })
    if (status) return status;
    if (mma_down) status = down_mma(p, few_mma, s);
    else GK_DISPATCH_DTYPE(p.dtype, T, { GK_DISPATCH_DTYPE(p.w_dtype, TW, { down_fp32<T, TW>(p, few_down, s); }) })
    if (status) return status;
    GK_CHECK_LAUNCH("experts");
    return GK_OK;
}

}  // namespace

// The whole routed feed-forward behind the router.  `work`: scratch of `at_once` times top * (4 width + ff * the type's size) bytes; more
// tokens than that go in several turns.
GK_EXPORT int gk_experts(const void* h, int dtype, const void* w_gate_up, const void* w_down, int w_dtype, const int* ids, const float* weights,
                         const void* add, const float* add_weight, float* work, float* out, int n_tokens, int at_once, int width, int ff, int top,
                         int n_experts, int* error_flag, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(dtype) && GK_VALID_DTYPE(w_dtype), "experts: bad dtype");
    GK_REQUIRE(at_once > 0 && width > 0 && ff > 0 && top > 0 && n_experts > 0 && (add != nullptr || add_weight == nullptr), "experts: bad sizes");
    GK_REQUIRE(error_flag != nullptr, "experts: error_flag is required");
    if (n_tokens == 0) return GK_OK;
    // a token's inner values stand in shared memory in the down product of few pairs
    GK_REQUIRE((size_t)width * sizeof(float) <= 200 * 1024, "experts: rows of %d are longer than the kernels stage", width);
    GK_REQUIRE((size_t)top * ff * sizeof(float) <= 200 * 1024, "experts: %d experts of %d are more than the kernels stage", top, ff);
    GK_REQUIRE((long long)std::min(at_once, n_tokens) * top <= 65535LL * MMA_LIST, "experts: too many pairs at once");
    const size_t size = dtype == GK_F32 ? 4 : 2;
    for (int at = 0; at < n_tokens; at += at_once) {
        const size_t row = (size_t)at * width;
        const ExpertStep p{(const char*)h + row * size, w_gate_up, w_down, dtype, w_dtype, ids + (size_t)at * top, weights + (size_t)at * top,
                           add ? (const char*)add + row * size : nullptr, add_weight ? add_weight + at : nullptr, work, work + (size_t)at_once * top * width,
                           out + row, std::min(at_once, n_tokens - at), width, ff, top, n_experts, error_flag};
        const int status = experts(p, (cudaStream_t)stream);
        if (status != GK_OK) return status;
    }
    return GK_OK;
}
