// Causal grouped-query attention over the paged cache, any head size, any dtype: the exact
// kernel.  It is the 32-bit path's attention and the fallback of the bfloat16 path for head
// sizes the tensor-core kernels do not take.
//
// For a token at position pos of its sequence, query head hq, kv head hk = hq / (n_q / n_kv):
//   s_j = (q . k_j) * scale      for the visible keys j <= pos (and j > pos - window, if a window is set)
//   o   = sum_j softmax(s)_j v_j
// With `sink` the softmax has one more term in its denominator, a key of score 0 that has no value:
//   p_j = exp(s_j) / (1 + sum_i exp(s_i)).
// which is the rule  key j visible to query i iff j <= past + i  of the reference
// (src/layers/attention.py:116-119) with consecutive query heads sharing a kv head
// (src/ops/flash_attention_2.py:33-34), scale = head_dim^-0.5 (flash_attention_2.py:216).
//
// Keys are taken in blocks of 32 from key 0 upward (from the block of the first key in a window), with a running maximum
// and sum (all 32-bit, expf); a score is one chain over the head's entries, a block's sum of exponentials the butterfly of
// warp_sum, and an entry of the read-out one chain over the keys.  The sequence of operations for a (token, head) depends
// only on its own position and keys: results are bit-equal however the tokens are cut into steps or batched.  Three
// kernels carry out these same operations:
//   tile    many tokens, heads of up to 128: 64 (token, head) rows that share a kv head walk its keys together, eight rows a
//           warp; a block of keys is fetched once for all of them, and a 16-byte read of a key or value out of shared
//           memory serves eight rows
//   single  few tokens, heads of up to 128: a cluster a (token, kv head) whose blocks share the scores of 1,024 keys at a
//           time and then carry a slice of the read-out's entries each, so that a step of few sequences spreads over the
//           device; what is left serial is the chain over the keys, 4 cycles each
//   warp    other sizes: one warp a (token, head), one key a lane

#include "common.cuh"

namespace {

constexpr int WARPS = 4;
constexpr int MAX_ACC = 16;  // head_dim <= 512
constexpr int KEYS = 32;     // keys of a block

__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void read4(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void read4(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    v[0] = lo.x, v[1] = lo.y, v[2] = hi.x, v[3] = hi.y;
}

struct Exact {
    const void *q, *k_pages, *v_pages;
    void* out;
    const int *tok_pos, *tok_seq, *slots, *block_table;
    int n_tokens, n_q, n_kv, head_dim, max_pages, page_size;
    float scale;
    int window, sink;
};

// ------------------------------------------------------------------ tile
constexpr int TILE_WARPS = 8, TILE_R = 8, TILE_ROWS = TILE_WARPS * TILE_R, TILE_MAX_D = 128;

template <typename T>
size_t tile_smem(int d) {
    return (size_t)TILE_ROWS * d * 4 + 2 * (size_t)KEYS * ((d + 16 / sizeof(T)) + d) * sizeof(T) + (size_t)TILE_ROWS * KEYS * 4;
}

// Rows of a block: tokens t0 .. t0 + TQ - 1, the heads of one group; row r is token r / group, head r % group.  The tile's
// tokens are walked sequence by sequence (tokens of a sequence lie side by side).  A prompt of 2,048 tokens, 16/8 heads of
// 128, 32-bit: 983 us (the warp kernel: 7,495); bound by the FP32 pipes and shared memory.
template <typename T>
__global__ void __launch_bounds__(TILE_WARPS * 32, 2) attention_exact_tile_kernel(const Exact p, int TQ) {
    constexpr int R = TILE_R, PAD = 16 / sizeof(T);
    extern __shared__ __align__(16) unsigned char smem[];
    const int d = p.head_dim, ldk = d + PAD, group = p.n_q / p.n_kv;
    float* qs = reinterpret_cast<float*>(smem);                            // [ROWS][d]
    float* ps = qs + (size_t)TILE_ROWS * d;                                // [ROWS][KEYS]
    T* ks = reinterpret_cast<T*>(ps + TILE_ROWS * KEYS);                   // [2][KEYS][ldk]
    T* vs = ks + 2 * KEYS * ldk;                                           // [2][KEYS][d]
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hk = blockIdx.y;
    const int tiles = (p.n_tokens + TQ - 1) / TQ;
    const int t0 = (tiles - 1 - (int)blockIdx.x) * TQ;  // the last tokens of a prompt have the most keys: they start first
    const int t_end = min(t0 + TQ, p.n_tokens);
    const T* q = (const T*)p.q;
    T* out = (T*)p.out;
    for (int i = tid; i < TILE_ROWS * d; i += TILE_WARPS * 32) {
        const int r = i / d, c = i - r * d, t = t0 + r / group;
        qs[i] = t < t_end && r < TQ * group ? to_float(q[((size_t)t * p.n_q + hk * group + r % group) * d + c]) : 0.f;
    }
    const int chunks = d / PAD;  // 16-byte pieces of a row
    for (int ts = t0; ts < t_end;) {
        const int seq = p.tok_seq[ts];
        int te = ts, last = 0, first = 0x7fffffff;
        for (; te < t_end && p.tok_seq[te] == seq; ++te) {
            const int pos = p.tok_pos[te];
            last = max(last, pos);
            first = min(first, (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0);
        }
        const int* pages = p.block_table + (size_t)p.slots[seq] * p.max_pages;
        int pos[R], lo[R];
        float m[R], l[R], acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = warp * R + r, t = t0 + row / group;
            const bool mine = row < TQ * group && t >= ts && t < te;
            pos[r] = mine ? p.tok_pos[t] : -1;
            lo[r] = mine && p.window > 0 && pos[r] - p.window + 1 > 0 ? pos[r] - p.window + 1 : 0;
            m[r] = -INFINITY;
            l[r] = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][e] = 0.f;
        }
        auto fetch = [&](int j0, int buf) {
            const size_t base = (((size_t)pages[j0 / p.page_size] * p.n_kv + hk) * p.page_size + j0 % p.page_size) * d;
            const T* kp = (const T*)p.k_pages + base;
            const T* vp = (const T*)p.v_pages + base;
            for (int i = tid; i < KEYS * chunks; i += TILE_WARPS * 32) {
                const int r = i / chunks, c = (i - r * chunks) * PAD;
                copy16(ks + (buf * KEYS + r) * ldk + c, kp + (size_t)r * d + c);
                copy16(vs + (buf * KEYS + r) * d + c, vp + (size_t)r * d + c);
            }
        };
        int j0 = (first >> 5) << 5, buf = 0;
        fetch(j0, 0);
        copy_commit();
        for (; j0 <= last; j0 += KEYS, buf ^= 1) {
            if (j0 + KEYS <= last) fetch(j0 + KEYS, buf ^ 1);
            copy_commit();
            copy_wait<1>();
            __syncthreads();
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
            const T* k_at = ks + (buf * KEYS + lane) * ldk;
            const float* q_at = qs + warp * R * d;
#pragma unroll 2
            for (int i = 0; i < d; i += 4) {
                float kv[4];
                read4(k_at + i, kv);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    float qv[4];
                    read4(q_at + r * d + i, qv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[r] = fmaf(qv[e], kv[e], s[r]);
                }
            }
            const int j = j0 + lane;
            int here[R];  // keys of this block that the row's chains take
            bool full = true;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float pr = 0.f;
                here[r] = 0;
                if (j0 <= pos[r] && j0 >= (lo[r] >> 5) << 5) {
                    const bool valid = j <= pos[r] && j >= lo[r];
                    const float sv = valid ? __fmul_rn(s[r], p.scale) : -INFINITY;
                    const float m_new = fmaxf(m[r], warp_max(sv));
                    pr = valid ? expf(sv - m_new) : 0.f;
                    const float corr = expf(m[r] - m_new);
                    l[r] = fmaf(l[r], corr, warp_sum(pr));
                    m[r] = m_new;
                    here[r] = min(KEYS, pos[r] - j0 + 1);
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[r][e] *= corr;
                }
                full = full && here[r] == KEYS;
                ps[(warp * R + r) * KEYS + lane] = pr;
            }
            __syncwarp();
            if (lane * 4 < d) {
                const T* v_at = vs + buf * KEYS * d + lane * 4;
                const float* p_at = ps + warp * R * KEYS;
                if (full) {
#pragma unroll 2
                    for (int jj = 0; jj < KEYS; jj += 4) {
                        float vv[4][4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) read4(v_at + (jj + u) * d, vv[u]);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            float pv[4];
                            read4(p_at + r * KEYS + jj, pv);
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int e = 0; e < 4; ++e) acc[r][e] = fmaf(pv[u], vv[u][e], acc[r][e]);
                        }
                    }
                } else {  // a key beyond a row's position must not enter its chain, whatever stands there
                    for (int jj = 0; jj < KEYS; ++jj) {
                        float vv[4];
                        read4(v_at + jj * d, vv);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            if (jj >= here[r]) continue;
                            const float pj = p_at[r * KEYS + jj];
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[r][e] = fmaf(pj, vv[e], acc[r][e]);
                        }
                    }
                }
            }
            __syncthreads();  // the other stage may be overwritten
        }
        copy_wait<0>();
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (pos[r] < 0 || lane * 4 >= d) continue;
            const int row = warp * R + r;
            const float sum = p.sink ? l[r] + expf(-m[r]) : l[r];  // the term of score 0, against the same reference exponent
            T* o = out + ((size_t)(t0 + row / group) * p.n_q + hk * group + row % group) * d + lane * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = from_float<T>(acc[r][e] / sum);
        }
        ts = te;
    }
}

// ------------------------------------------------------------------ single
constexpr int SINGLE_WARPS = 8, SPAN = 1024, SPAN_BLOCKS = SPAN / KEYS, V_KEYS = 128, V_STAGES = 3, K_PIECE = 32, MAX_GROUP = 16;

__host__ __device__ inline int single_ranks(int d) { return d <= 32 ? 1 : d <= 64 ? 2 : 4; }
__host__ __device__ inline int single_slice(int d) { return (((d + single_ranks(d) - 1) / single_ranks(d)) + 7) / 8 * 8; }

template <typename T>
size_t single_smem(int d, int group) {
    const int own = SPAN / single_ranks(d);
    return (size_t)group * d * 4 + (size_t)group * (SPAN + own) * 4 + (size_t)group * 3 * SPAN_BLOCKS * 4 +
           (size_t)SINGLE_WARPS * 2 * KEYS * (K_PIECE + 16 / sizeof(T)) * sizeof(T) + (size_t)V_STAGES * V_KEYS * single_slice(d) * sizeof(T);
}

// A cluster of 1, 2 or 4 blocks a (token, kv head).  1,024 keys at a time: a block forms the scores of every rank-th block
// of keys (a warp a block of keys, one key a lane, the keys through the warp's own ring in pieces of 32 entries), all blocks
// fetch all scores through distributed shared memory and form maxima, exponentials and sums, and a warp a head carries the
// chains of the block's slice of entries, the values through a ring that all threads fill.  GP: heads of a group, rounded up.
// Bound by the chain over the keys where sequences are few.  Single tokens after 2,047, 16/8 heads of 128, 32-bit: one
// sequence 52 us (the warp kernel: 846), eight 105 (1,646).
template <typename T, int GP>
__global__ void __launch_bounds__(SINGLE_WARPS * 32) attention_exact_single_kernel(const Exact p) {
    constexpr int PAD = 16 / sizeof(T), LDK = K_PIECE + PAD, THREADS = SINGLE_WARPS * 32;
    extern __shared__ __align__(16) unsigned char smem[];
    const int d = p.head_dim, group = p.n_q / p.n_kv, ranks = single_ranks(d), slice = single_slice(d), own_keys = SPAN / ranks;
    float* qs = reinterpret_cast<float*>(smem);           // [group][d]
    float* sc = qs + (size_t)group * d;                   // [group][SPAN]: scores, then weights
    float* own = sc + (size_t)group * SPAN;               // [group][own_keys]: what this block's warps formed
    float* block_m = own + (size_t)group * own_keys;      // [group][SPAN_BLOCKS]: maxima, then running maxima
    float* block_c = block_m + group * SPAN_BLOCKS;       // corrections
    float* block_l = block_c + group * SPAN_BLOCKS;       // sums of the weights
    T* ks = reinterpret_cast<T*>(block_l + group * SPAN_BLOCKS);  // [warps][2][KEYS][LDK]
    T* vs = ks + SINGLE_WARPS * 2 * KEYS * LDK;                   // [V_STAGES][V_KEYS][slice]
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = (int)(blockIdx.x % ranks), unit = (int)(blockIdx.x / ranks);  // a cluster's blocks are consecutive
    const int t = unit / p.n_kv, hk = unit % p.n_kv;
    const int pos = p.tok_pos[t];
    const int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    const int* pages = p.block_table + (size_t)p.slots[p.tok_seq[t]] * p.max_pages;
    const T* q = (const T*)p.q + ((size_t)t * p.n_q + hk * group) * d;
    const T* k_pages = (const T*)p.k_pages;
    const T* v_pages = (const T*)p.v_pages;
    const int dim0 = rank * slice, dims = max(0, min(slice, d - dim0)), v_chunks = dims / PAD;
    for (int i = tid; i < group * d; i += THREADS) qs[i] = to_float(q[i]);
    const auto row_of = [&](int j) { return ((size_t)pages[j / p.page_size] * p.n_kv + hk) * p.page_size + j % p.page_size; };

    constexpr int HEADS = (GP + SINGLE_WARPS - 1) / SINGLE_WARPS;  // heads whose chains a warp carries
    float m_run[HEADS], l_run[HEADS], acc[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; ++h) m_run[h] = -INFINITY, l_run[h] = 0.f, acc[h] = 0.f;
    __syncthreads();

    for (int j0 = (lo >> 5) << 5; j0 <= pos; j0 += SPAN) {
        const int n_keys = min(SPAN, pos - j0 + 1), n_blocks = (n_keys + KEYS - 1) / KEYS, v_steps = (n_keys + V_KEYS - 1) / V_KEYS;
        const auto fetch_v = [&](int step) {
            const int first = step * V_KEYS, count = min(V_KEYS, n_keys - first);
            T* dst = vs + (step % V_STAGES) * V_KEYS * slice;
            for (int i = tid; i < count * v_chunks; i += THREADS) {
                const int r = i / v_chunks, c = (i - r * v_chunks) * PAD;
                copy16(dst + r * slice + c, v_pages + row_of(j0 + first + r) * d + dim0 + c);
            }
        };
        // scores of key blocks rank, rank + ranks, ...
        for (int kb = rank + ranks * warp; kb < n_blocks; kb += ranks * SINGLE_WARPS) {
            const size_t row = row_of(j0 + kb * KEYS);  // page sizes are multiples of 32: a block of keys lies in one page
            T* mine = ks + warp * 2 * KEYS * LDK;
            const int pieces = (d + K_PIECE - 1) / K_PIECE;
            const auto fetch_k = [&](int piece) {
                const int width = min(K_PIECE, d - piece * K_PIECE) / PAD;
                for (int i = lane; i < KEYS * width; i += 32) {
                    const int r = i / width, c = (i - r * width) * PAD;
                    copy16(mine + ((piece & 1) * KEYS + r) * LDK + c, k_pages + (row + r) * d + piece * K_PIECE + c);
                }
                copy_commit();
            };
            float s[GP];
#pragma unroll
            for (int g = 0; g < GP; ++g) s[g] = 0.f;
            fetch_k(0);
            for (int piece = 0; piece < pieces; ++piece) {
                if (piece + 1 < pieces) {
                    fetch_k(piece + 1);
                    copy_wait<1>();
                } else {
                    copy_wait<0>();
                }
                __syncwarp();
                const int width = min(K_PIECE, d - piece * K_PIECE);
                const T* k_at = mine + ((piece & 1) * KEYS + lane) * LDK;
                const float* q_at = qs + piece * K_PIECE;
#pragma unroll 4
                for (int i = 0; i < width; i += 4) {
                    float kv[4];
                    read4(k_at + i, kv);
#pragma unroll
                    for (int g = 0; g < GP; ++g) {
                        if (g >= group) break;
                        float qv[4];
                        read4(q_at + g * d + i, qv);
#pragma unroll
                        for (int e = 0; e < 4; ++e) s[g] = fmaf(qv[e], kv[e], s[g]);
                    }
                }
                __syncwarp();  // the piece's stage may be filled again
            }
            const int j = j0 + kb * KEYS + lane;
            const bool valid = j <= pos && j >= lo;
#pragma unroll
            for (int g = 0; g < GP; ++g)
                if (g < group) own[g * own_keys + (kb / ranks) * KEYS + lane] = valid ? __fmul_rn(s[g], p.scale) : -INFINITY;
        }
        for (int step = 0; step < V_STAGES - 1; ++step) {  // the first values come while the scores are exchanged
            if (step < v_steps) fetch_v(step);
            copy_commit();
        }
        cluster_barrier();
        for (int i = tid; i < group * n_blocks * KEYS; i += THREADS) {
            const int g = i / (n_blocks * KEYS), at = i - g * n_blocks * KEYS, kb = at / KEYS;
            const uint32_t local = (uint32_t)__cvta_generic_to_shared(own + g * own_keys + (kb / ranks) * KEYS + at % KEYS);
            uint32_t remote;
            float v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(kb % ranks));
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
            sc[g * SPAN + at] = v;
        }
        cluster_barrier();  // the blocks' own scores may be overwritten from here on (and their blocks may leave)
        for (int i = warp; i < group * n_blocks; i += SINGLE_WARPS) {
            const int g = i / n_blocks, kb = i - g * n_blocks;
            const float best = warp_max(sc[g * SPAN + kb * KEYS + lane]);
            if (lane == 0) block_m[g * SPAN_BLOCKS + kb] = best;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < HEADS; ++h) {  // running maxima and corrections: a warp a head, a lane a block of keys
            const int g = warp + h * SINGLE_WARPS;
            if (g >= group) continue;
            float best = lane < n_blocks ? block_m[g * SPAN_BLOCKS + lane] : -INFINITY;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float other = __shfl_up_sync(0xffffffffu, best, o);
                if (lane >= o) best = fmaxf(other, best);
            }
            best = fmaxf(m_run[h], best);
            float before = __shfl_up_sync(0xffffffffu, best, 1);
            if (lane == 0) before = m_run[h];
            if (lane < n_blocks) {
                block_m[g * SPAN_BLOCKS + lane] = best;
                block_c[g * SPAN_BLOCKS + lane] = expf(before - best);
            }
            m_run[h] = __shfl_sync(0xffffffffu, best, n_blocks - 1);
        }
        __syncthreads();
        for (int i = warp; i < group * n_blocks; i += SINGLE_WARPS) {
            const int g = i / n_blocks, kb = i - g * n_blocks, j = j0 + kb * KEYS + lane;
            float* at = sc + g * SPAN + kb * KEYS + lane;
            const float w = j <= pos && j >= lo ? expf(*at - block_m[g * SPAN_BLOCKS + kb]) : 0.f;
            *at = w;
            const float sum = warp_sum(w);
            if (lane == 0) block_l[g * SPAN_BLOCKS + kb] = sum;
        }
        __syncthreads();
        for (int step = 0; step < v_steps; ++step) {
            copy_wait<V_STAGES - 2>();
            __syncthreads();
            if (step + V_STAGES - 1 < v_steps) fetch_v(step + V_STAGES - 1);
            copy_commit();
            const T* stage = vs + (step % V_STAGES) * V_KEYS * slice + min(lane, max(dims, 1) - 1);
#pragma unroll
            for (int h = 0; h < HEADS; ++h) {
                const int g = warp + h * SINGLE_WARPS;
                if (g >= group) continue;
                for (int b = 0; b < V_KEYS / KEYS; ++b) {
                    const int kb = step * (V_KEYS / KEYS) + b;
                    if (kb >= n_blocks) break;
                    const float corr = block_c[g * SPAN_BLOCKS + kb];
                    l_run[h] = fmaf(l_run[h], corr, block_l[g * SPAN_BLOCKS + kb]);
                    float a = acc[h] * corr;
                    const float* w_at = sc + g * SPAN + kb * KEYS;
                    const T* v_at = stage + b * KEYS * slice;
                    const int here = min(KEYS, n_keys - kb * KEYS);
                    if (here == KEYS) {
#pragma unroll
                        for (int jj = 0; jj < KEYS; jj += 4) {
                            float w[4];
                            read4(w_at + jj, w);
#pragma unroll
                            for (int u = 0; u < 4; ++u) a = fmaf(w[u], to_float(v_at[(jj + u) * slice]), a);
                        }
                    } else {
                        for (int jj = 0; jj < here; ++jj) a = fmaf(w_at[jj], to_float(v_at[jj * slice]), a);
                    }
                    acc[h] = a;
                }
            }
        }
        copy_wait<0>();
        __syncthreads();  // scores and values may be overwritten
    }
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
        const int g = warp + h * SINGLE_WARPS;
        if (g >= group || lane >= dims) continue;
        const float sum = p.sink ? l_run[h] + expf(-m_run[h]) : l_run[h];
        ((T*)p.out)[((size_t)t * p.n_q + hk * group + g) * d + dim0 + lane] = from_float<T>(acc[h] / sum);
    }
}

// ------------------------------------------------------------------ warp
template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q, const T* __restrict__ k, int d);

template <>
__device__ __forceinline__ float dot_row<float>(const float* __restrict__ q, const float* __restrict__ k, int d) {
    float acc = 0.f;
    for (int i = 0; i < d; i += 4) {
        const float4 kv = *reinterpret_cast<const float4*>(k + i);
        acc = fmaf(q[i], kv.x, acc);
        acc = fmaf(q[i + 1], kv.y, acc);
        acc = fmaf(q[i + 2], kv.z, acc);
        acc = fmaf(q[i + 3], kv.w, acc);
    }
    return acc;
}

template <>
__device__ __forceinline__ float dot_row<__nv_bfloat16>(const float* __restrict__ q,
                                                        const __nv_bfloat16* __restrict__ k, int d) {
    float acc = 0.f;
    for (int i = 0; i < d; i += 8) {
        const uint4 raw = *reinterpret_cast<const uint4*>(k + i);
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float2 f = __bfloat1622float2(p[c]);
            acc = fmaf(q[i + 2 * c], f.x, acc);
            acc = fmaf(q[i + 2 * c + 1], f.y, acc);
        }
    }
    return acc;
}

template <typename T>
__global__ void __launch_bounds__(WARPS * 32) attention_exact_kernel(
    const T* __restrict__ q, const T* __restrict__ k_pages, const T* __restrict__ v_pages, T* __restrict__ out,
    const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, const int* __restrict__ slots,
    const int* __restrict__ block_table, int n_tokens, int n_q, int n_kv, int head_dim, int max_pages, int page_size,
    float scale, int window, int sink) {
    extern __shared__ float q_smem[];  // WARPS * head_dim
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long wid = (long long)blockIdx.x * WARPS + warp;
    if (wid >= (long long)n_tokens * n_q) return;  // whole warp leaves together; no block-wide sync below
    const int t = (int)(wid / n_q);
    const int hq = (int)(wid - (long long)t * n_q);
    const int hk = hq / (n_q / n_kv);
    const int pos = tok_pos[t];
    const int slot = slots[tok_seq[t]];
    const int* pages = block_table + (size_t)slot * max_pages;
    float* qs = q_smem + warp * head_dim;
    const T* qrow = q + ((size_t)t * n_q + hq) * head_dim;
    for (int i = lane; i < head_dim; i += 32) qs[i] = to_float(qrow[i]);
    __syncwarp();

    const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    float m = -INFINITY, l = 0.f;
    float acc[MAX_ACC];
#pragma unroll
    for (int c = 0; c < MAX_ACC; ++c) acc[c] = 0.f;
    const int n_acc = (head_dim + 31) >> 5;

    for (int j0 = (lo >> 5) << 5; j0 <= pos; j0 += 32) {
        const int page = pages[j0 / page_size];  // page_size is a multiple of 32: one page per block
        const int in_page = j0 % page_size;
        const size_t base = (((size_t)page * n_kv + hk) * page_size + in_page) * head_dim;
        const int j = j0 + lane;
        const bool valid = j <= pos && j >= lo;
        float s = -INFINITY;
        if (valid) s = __fmul_rn(dot_row<T>(qs, k_pages + base + (size_t)lane * head_dim, head_dim), scale);
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = fmaf(l, corr, warp_sum(p));
        const int n_here = min(32, pos - j0 + 1);
#pragma unroll
        for (int c = 0; c < MAX_ACC; ++c)
            if (c < n_acc) acc[c] *= corr;
        for (int jj = 0; jj < n_here; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const T* vrow = v_pages + base + (size_t)jj * head_dim;
#pragma unroll
            for (int c = 0; c < MAX_ACC; ++c) {
                const int dim = lane + 32 * c;
                if (c < n_acc && dim < head_dim) acc[c] = fmaf(pj, to_float(vrow[dim]), acc[c]);
            }
        }
        m = m_new;
    }
    if (sink) l += expf(-m);  // the term of score 0, against the same reference exponent as the others
    T* orow = out + ((size_t)t * n_q + hq) * head_dim;
#pragma unroll
    for (int c = 0; c < MAX_ACC; ++c) {
        const int dim = lane + 32 * c;
        if (c < n_acc && dim < head_dim) orow[dim] = from_float<T>(acc[c] / l);
    }
}

// `single` for steps of about one token a sequence, and for so few tokens that its blocks (one set a token) are still fewer
// than the tile's serial walk is long.  Measured (us, single / tile; 16/8 heads of 128, 32-bit, tokens after 1,000): 16
// tokens: 104 / 290, 32: 222 / 290, 64: 488 / 294.  The warp kernel, which took all of them before: 431, 444, 500.
constexpr long long SINGLE_BLOCKS = 1024;
constexpr size_t MAX_SMEM = 227 * 1024;

template <typename T>
void launch_tile(const Exact& p, cudaStream_t s) {
    const int TQ = TILE_ROWS / (p.n_q / p.n_kv);
    const size_t smem = tile_smem<T>(p.head_dim);
    if (smem > 48 * 1024) cudaFuncSetAttribute((const void*)attention_exact_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gk_launch(attention_exact_tile_kernel<T>, dim3((p.n_tokens + TQ - 1) / TQ, p.n_kv), dim3(TILE_WARPS * 32), smem, s, p, TQ);
}

template <typename T, int GP>
void launch_single(const Exact& p, cudaStream_t s) {
    const int ranks = single_ranks(p.head_dim);
    const size_t smem = single_smem<T>(p.head_dim, p.n_q / p.n_kv);
    if (smem > 48 * 1024) cudaFuncSetAttribute((const void*)attention_exact_single_kernel<T, GP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gk_launch_cluster(attention_exact_single_kernel<T, GP>, dim3((unsigned)((long long)p.n_tokens * p.n_kv * ranks)), dim3(SINGLE_WARPS * 32), smem, s,
                      dim3(ranks, 1, 1), p);
}

}  // namespace

// `n_seqs` (how many sequences the tokens belong to) is read by the choice of the kernel alone.
GK_EXPORT int gk_attention_exact(const void* q, const void* k_pages, const void* v_pages, void* out, int dtype,
                                 const int* tok_pos, const int* tok_seq, const int* slots, const int* block_table,
                                 int n_tokens, int n_q, int n_kv, int head_dim, int max_pages, int page_size,
                                 float scale, int window, int sink, int n_seqs, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(dtype), "attention_exact: bad dtype %d", dtype);
    GK_REQUIRE(n_tokens >= 0 && n_q > 0 && n_kv > 0 && n_q % n_kv == 0, "attention_exact: bad head counts %d/%d", n_q,
               n_kv);
    GK_REQUIRE(head_dim > 0 && head_dim % 8 == 0 && head_dim <= 32 * MAX_ACC,
               "attention_exact: head_dim %d must be a multiple of 8 and at most %d", head_dim, 32 * MAX_ACC);
    GK_REQUIRE(page_size > 0 && page_size % 32 == 0, "attention_exact: page_size %d must be a multiple of 32",
               page_size);
    GK_REQUIRE(window >= 0, "attention_exact: window must be >= 0 (0 = none)");
    if (n_tokens == 0) return GK_OK;
    const long long warps = (long long)n_tokens * n_q;
    const long long blocks = (warps + WARPS - 1) / WARPS;
    GK_REQUIRE(blocks < 2147483647LL, "attention_exact: too many tokens");
    const size_t smem = (size_t)WARPS * head_dim * sizeof(float);
    cudaStream_t s = (cudaStream_t)stream;
    const int group = n_q / n_kv;
    // pages on 16 bytes (a head's row is a multiple of them)
    if (head_dim <= TILE_MAX_D && group <= MAX_GROUP && n_kv <= 65535 && (((uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0) {
        const Exact p{q, k_pages, v_pages, out, tok_pos, tok_seq, slots, block_table, n_tokens, n_q, n_kv, head_dim, max_pages, page_size, scale, window, sink};
        const long long singles = (long long)n_tokens * n_kv * single_ranks(head_dim);
        const bool few = n_tokens <= 2LL * n_seqs || singles <= SINGLE_BLOCKS;
        const size_t needs = dtype == GK_F32 ? single_smem<float>(head_dim, group) : single_smem<__nv_bfloat16>(head_dim, group);
        if (few && needs <= MAX_SMEM && singles < 2147483647LL) {
            GK_DISPATCH_DTYPE(dtype, T, {
                if (group == 1) launch_single<T, 1>(p, s);
                else if (group == 2) launch_single<T, 2>(p, s);
                else if (group <= 4) launch_single<T, 4>(p, s);
                else if (group <= 8) launch_single<T, 8>(p, s);
                else launch_single<T, 16>(p, s);
            })
            GK_CHECK_LAUNCH("attention_exact");
            return GK_OK;
        }
        if (!few) {
            GK_DISPATCH_DTYPE(dtype, T, { launch_tile<T>(p, s); })
            GK_CHECK_LAUNCH("attention_exact");
            return GK_OK;
        }
    }
    GK_DISPATCH_DTYPE(dtype, T, {
        gk_launch(attention_exact_kernel<T>, dim3((unsigned)blocks), dim3(WARPS * 32), smem, s,
            (const T*)q, (const T*)k_pages, (const T*)v_pages, (T*)out, tok_pos, tok_seq, slots, block_table, n_tokens,
            n_q, n_kv, head_dim, max_pages, page_size, scale, window, sink);
    })
    GK_CHECK_LAUNCH("attention_exact");
    return GK_OK;
}
