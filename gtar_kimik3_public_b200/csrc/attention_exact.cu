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
// only on its own position and keys: results are bit-equal however the tokens are cut into steps or batched.  Heads of up to 128
// have three ways to carry out these same operations, others the last:
//   tile    runs of many tokens of a sequence: 64 (token, head) rows that share a kv head walk its keys together, eight rows a
//           warp; a block of keys is fetched once for all of them, and a 16-byte read of a key or value out of shared
//           memory serves eight rows
//   warp    tokens that stand alone or in short runs, many of them: a warp a (token, up to four heads of a kv head)
//   single  so few tokens that warps would leave the device idle: a cluster a (token, kv head) whose blocks share the scores of
//           1,024 keys at a time and then carry a slice of the read-out's entries each
//   wide    other sizes: one warp a (token, head), one key a lane
// Tiles and warps are blocks of one launch (`rows`), which look at the step's own runs of tokens: how many tokens of which sequence
// a captured step will bring is not known when it is captured.

#include <algorithm>

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

// ------------------------------------------------------------------ warp
__device__ __forceinline__ void load16(const float* p, float (&v)[4]) { read4(p, v); }
__device__ __forceinline__ void load16(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float2 f = __bfloat1622float2(pairs[c]);
        v[2 * c] = f.x, v[2 * c + 1] = f.y;
    }
}

// floats of shared memory a warp works in: the heads' queries and a block of keys' weights
__host__ __device__ inline int warp_floats(int heads, int d) { return heads * (d + KEYS); }

// Heads g0 .. g0 + heads - 1 (up to HC) of kv head hk of token t.  A lane has a key of the block for the scores and four entries for
// the read-out; keys and values come straight from memory, sixteen bytes a load and eight loads in flight.  Bound by latency (0.2 us
// a key with a warp or two an SM) and, with many warps, by the lanes' keys, each in a line of its own.  Measured (us; 16/8 heads of
// 128, 32-bit; the wide kernel / a cluster each / here): 64 single tokens after 10: 10 / 141 / 7, after 1,000: 815 / 418 / 223; 512 after
// 100: 323 / 1,270 / 130.
template <typename T, int HC>
__device__ __forceinline__ void warp_rows(const Exact& p, int t, int hk, int g0, int heads, float* mine) {
    constexpr int PER = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, d = p.head_dim, group = p.n_q / p.n_kv;
    float* qs = mine;            // [HC][d]
    float* ps = mine + HC * d;  // [HC][KEYS]
    const int pos = p.tok_pos[t];
    const int lo = (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0;
    const int* pages = p.block_table + (size_t)p.slots[p.tok_seq[t]] * p.max_pages;
    const size_t first = ((size_t)t * p.n_q + hk * group + g0) * d;
    const T* q = (const T*)p.q + first;
    __syncwarp();
    for (int i = lane; i < HC * d; i += 32) qs[i] = i < heads * d ? to_float(q[i]) : 0.f;
    __syncwarp();
    const bool carries = lane * 4 < d;
    float m[HC], l[HC], acc[HC][4];
#pragma unroll
    for (int h = 0; h < HC; ++h) {
        m[h] = -INFINITY, l[h] = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[h][e] = 0.f;
    }
    for (int j0 = (lo >> 5) << 5; j0 <= pos; j0 += KEYS) {
        const size_t base = (((size_t)pages[j0 / p.page_size] * p.n_kv + hk) * p.page_size + j0 % p.page_size) * d;  // in one page
        const T* k_at = (const T*)p.k_pages + base + (size_t)lane * d;
        float s[HC];
#pragma unroll
        for (int h = 0; h < HC; ++h) s[h] = 0.f;
#pragma unroll 8
        for (int i = 0; i < d; i += PER) {
            float kv[PER];
            load16(k_at + i, kv);
#pragma unroll
            for (int h = 0; h < HC; ++h)
#pragma unroll
                for (int c = 0; c < PER; c += 4) {
                    float qv[4];
                    read4(qs + h * d + i + c, qv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) s[h] = fmaf(qv[e], kv[c + e], s[h]);
                }
        }
        const int j = j0 + lane;
        const bool valid = j <= pos && j >= lo;
#pragma unroll
        for (int h = 0; h < HC; ++h) {
            const float sv = valid ? __fmul_rn(s[h], p.scale) : -INFINITY;
            const float m_new = fmaxf(m[h], warp_max(sv));
            const float pr = valid ? expf(sv - m_new) : 0.f;
            const float corr = expf(m[h] - m_new);
            l[h] = fmaf(l[h], corr, warp_sum(pr));
            m[h] = m_new;
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[h][e] *= corr;
            ps[h * KEYS + lane] = pr;
        }
        __syncwarp();
        const int here = min(KEYS, pos - j0 + 1);  // a key beyond the token must not enter its chain, whatever stands there
        if (carries) {
            const T* v_at = (const T*)p.v_pages + base + lane * 4;
            constexpr int AT_ONCE = 8;
            int jj = 0;
            for (; jj + AT_ONCE <= here; jj += AT_ONCE) {
                float vv[AT_ONCE][4];
#pragma unroll
                for (int u = 0; u < AT_ONCE; ++u) read4(v_at + (size_t)(jj + u) * d, vv[u]);
#pragma unroll
                for (int h = 0; h < HC; ++h)
#pragma unroll
                    for (int u0 = 0; u0 < AT_ONCE; u0 += 4) {
                        float pv[4];
                        read4(ps + h * KEYS + jj + u0, pv);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[h][e] = fmaf(pv[u], vv[u0 + u][e], acc[h][e]);
                    }
            }
            for (; jj < here; ++jj) {
                float vv[4];
                read4(v_at + (size_t)jj * d, vv);
#pragma unroll
                for (int h = 0; h < HC; ++h) {
                    const float pj = ps[h * KEYS + jj];
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[h][e] = fmaf(pj, vv[e], acc[h][e]);
                }
            }
        }
        __syncwarp();  // the weights may be overwritten
    }
    if (!carries) return;
#pragma unroll
    for (int h = 0; h < HC; ++h) {
        if (h >= heads) break;
        const float sum = p.sink ? l[h] + expf(-m[h]) : l[h];  // the term of score 0, against the same reference exponent
        T* o = (T*)p.out + first + (size_t)h * d + lane * 4;
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = from_float<T>(acc[h][e] / sum);
    }
}

constexpr int ROW_WARPS = 8;
constexpr int LIST = 1024;  // tokens that the warps' blocks look at together
constexpr int TILE_WARPS = 8, TILE_R = 8, TILE_ROWS = TILE_WARPS * TILE_R, TILE_MAX_D = 128;

// A tile walks its runs of tokens one after another, all where they are one or two, else those of at least min_run tokens: the
// others would each cost a walk for a few of its rows.  min_run 0: everything.
constexpr int RUNS_TOGETHER = 2;

// The tokens that no tile walks (min_run 0: there are no tiles), by a warp a (token, HC heads).  Every block makes the same list
// of them, LIST tokens at a time; the units are spread over the blocks before a block takes a second one.
template <typename T, int HC>
__global__ void __launch_bounds__(ROW_WARPS * 32, 2) attention_exact_warp_kernel(const Exact p, int TQ, int min_run) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int seqs[LIST], list[LIST], counts[ROW_WARPS], runs[LIST / 4];  // a tile has at least four tokens
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = p.n_q / p.n_kv, parts = (group + HC - 1) / HC;
    float* mine = reinterpret_cast<float*>(smem) + warp * warp_floats(HC, p.head_dim);
    const int step = min_run > 0 ? LIST / TQ * TQ : p.n_tokens;
    for (int c0 = 0; c0 < p.n_tokens; c0 += step) {
        const int in_step = min(step, p.n_tokens - c0);
        int n = in_step;
        if (min_run > 0) {
            __syncthreads();  // the list of before has been used
            for (int i = tid; i < in_step; i += ROW_WARPS * 32) seqs[i] = p.tok_seq[c0 + i];
            for (int i = tid; i < LIST / 4; i += ROW_WARPS * 32) runs[i] = 0;
            __syncthreads();
            for (int i = tid; i < in_step; i += ROW_WARPS * 32)
                if (i % TQ == 0 || seqs[i] != seqs[i - 1]) atomicAdd(&runs[i / TQ], 1);
            __syncthreads();
            n = 0;
            for (int i0 = 0; i0 < in_step; i0 += ROW_WARPS * 32) {
                const int i = i0 + tid;
                bool alone = false;
                if (i < in_step && runs[i / TQ] > RUNS_TOGETHER) {
                    const int begin = i / TQ * TQ, end = min(begin + TQ, in_step);
                    int run = 1;
                    for (int j = i - 1; j >= begin && run < min_run && seqs[j] == seqs[i]; --j) ++run;
                    for (int j = i + 1; j < end && run < min_run && seqs[j] == seqs[i]; ++j) ++run;
                    alone = run < min_run;
                }
                const unsigned int those = __ballot_sync(0xffffffffu, alone);
                if (lane == 0) counts[warp] = __popc(those);
                __syncthreads();
                int before = n;
                for (int w = 0; w < ROW_WARPS; ++w) {
                    if (w < warp) before += counts[w];
                    n += counts[w];
                }
                if (alone) list[before + __popc(those & ((1u << lane) - 1))] = i;
                __syncthreads();
            }
        }
        const long long units = (long long)n * p.n_kv * parts;
        const int at_once = (int)min((long long)ROW_WARPS, (units + gridDim.x - 1) / gridDim.x);  // neighbours share keys where tokens do
        if (warp >= at_once) continue;
        for (long long u = (long long)blockIdx.x * at_once + warp; u < units; u += (long long)gridDim.x * at_once) {
            const int i = (int)(u % n), part = (int)(u / n), hk = part / parts, g0 = part % parts * HC;
            warp_rows<T, HC>(p, c0 + (min_run > 0 ? list[i] : i), hk, g0, min(HC, group - g0), mine);
        }
    }
}

// ------------------------------------------------------------------ tile
template <typename T>
size_t tile_smem(int d) {
    return (size_t)TILE_ROWS * d * 4 + 2 * (size_t)KEYS * ((d + 16 / sizeof(T)) + d) * sizeof(T) + (size_t)TILE_ROWS * KEYS * 4;
}

// Rows of a block: tokens t0 .. t0 + TQ - 1, the heads of one group; row r is token r / group, head r % group.  A prompt of 2,048
// tokens, 16/8 heads of 128, 32-bit: 983 us (the wide kernel: 7,495); bound by the FP32 pipes and shared memory.
template <typename T>
__global__ void __launch_bounds__(TILE_WARPS * 32, 2) attention_exact_tile_kernel(const Exact p, int TQ, int min_run) {
    constexpr int R = TILE_R, PAD = 16 / sizeof(T), NOT_MINE = -0x7fffffff - 1;
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
    int shortest = 0;
    if (min_run > 0) {
        int runs = 1;
        for (int t = t0 + 1; t < t_end; ++t) runs += p.tok_seq[t] != p.tok_seq[t - 1];
        if (runs > RUNS_TOGETHER) shortest = min_run;
    }
    for (int ts = t0; ts < t_end;) {
        const int seq = p.tok_seq[ts];
        int te = ts, last = -1, first = 0x7fffffff;
        for (; te < t_end && p.tok_seq[te] == seq; ++te) {
            const int pos = p.tok_pos[te];
            last = max(last, pos);
            first = min(first, (p.window > 0 && pos - p.window + 1 > 0) ? pos - p.window + 1 : 0);
        }
        if (te - ts < shortest) {  // the warp kernel's tokens
            ts = te;
            continue;
        }
        const int* pages = p.block_table + (size_t)p.slots[seq] * p.max_pages;
        int pos[R], lo[R];
        float m[R], l[R], acc[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = warp * R + r, t = t0 + row / group;
            const bool mine = row < TQ * group && t >= ts && t < te;
            pos[r] = mine ? p.tok_pos[t] : NOT_MINE;
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
        if (j0 <= last) fetch(j0, 0);
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
            if (pos[r] == NOT_MINE || lane * 4 >= d) continue;
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
constexpr int SINGLE_WARPS = 8, SPAN = 1024, SPAN_BLOCKS = SPAN / KEYS, V_KEYS = 128, V_STAGES = 3, K_PIECE = 32, MAX_GROUP = 16, SHORT_KEYS = 32;

__host__ __device__ inline int single_ranks(int d) { return d <= 32 ? 1 : d <= 64 ? 2 : 4; }
__host__ __device__ inline int single_slice(int d) { return (((d + single_ranks(d) - 1) / single_ranks(d)) + 7) / 8 * 8; }

template <typename T>
size_t single_smem(int d, int group) {
    const int own = SPAN / single_ranks(d);
    const size_t keys = (size_t)SINGLE_WARPS * 2 * KEYS * (K_PIECE + 16 / sizeof(T)) * sizeof(T), values = (size_t)V_STAGES * V_KEYS * single_slice(d) * sizeof(T);
    return (size_t)group * d * 4 + (size_t)group * (SPAN + own) * 4 + (size_t)group * 3 * SPAN_BLOCKS * 4 + std::max(keys, values);
}

// A cluster of 1, 2 or 4 blocks a (token, kv head).  1,024 keys at a time: a block forms the scores of every rank-th block
// of keys (a warp a block of keys, one key a lane, the keys through the warp's own ring in pieces of 32 entries), all blocks
// fetch all scores through distributed shared memory and form maxima, exponentials and sums, and a warp a head carries the
// chains of the block's slice of entries, the values through a ring that all threads fill.  GP: heads of a group, rounded up.
// Some 25 us a span of 1,024 keys (16/8 heads of 128, 32-bit), 2 of them the chain over the keys, 4 cycles each; the others are
// the scores of one block of keys a warp, the exchange and its barriers, and the wait for the values.  Keys and values share a
// place in shared memory, so that two blocks (three in bfloat16) are on an SM.  Measured (us; the wide kernel / here): one token after
// 3,000: 1,262 / 73; sixteen: 2,451 / 183.  A token whose keys lie in one block of them
// takes a warp a head; with two blocks that is slower (a prompt of 64, 6/2 heads of 32: 6.9 against 6.2).
template <typename T, int GP>
__global__ void __launch_bounds__(SINGLE_WARPS * 32, GP <= 8 ? 3 : 2) attention_exact_single_kernel(const Exact p) {
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
    T* vs = ks;                                                   // [V_STAGES][V_KEYS][slice], once the keys have been used
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
    if (pos - ((lo >> 5) << 5) < SHORT_KEYS) {  // a warp a head, in all blocks of the cluster alike
        float* mine = reinterpret_cast<float*>(smem) + warp * warp_floats(1, d);
        for (int g = rank * SINGLE_WARPS + warp; g < group; g += ranks * SINGLE_WARPS) warp_rows<T, 1>(p, t, hk, g, 1, mine);
        return;
    }
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
        __syncthreads();  // all warps are through with the keys, whose place the values take
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

// ------------------------------------------------------------------ wide
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

constexpr size_t MAX_SMEM = 227 * 1024;

template <typename T>
void launch_tile(const Exact& p, int min_run, cudaStream_t s) {
    const int TQ = TILE_ROWS / (p.n_q / p.n_kv);
    const size_t smem = tile_smem<T>(p.head_dim);
    if (smem > 48 * 1024) cudaFuncSetAttribute((const void*)attention_exact_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gk_launch(attention_exact_tile_kernel<T>, dim3((p.n_tokens + TQ - 1) / TQ, p.n_kv), dim3(TILE_WARPS * 32), smem, s, p, TQ, min_run);
}

template <typename T, int HC>
void launch_warps(const Exact& p, int min_run, int blocks, cudaStream_t s) {
    const int TQ = TILE_ROWS / (p.n_q / p.n_kv);
    const size_t smem = (size_t)ROW_WARPS * warp_floats(HC, p.head_dim) * sizeof(float);
    gk_launch(attention_exact_warp_kernel<T, HC>, dim3(blocks), dim3(ROW_WARPS * 32), smem, s, p, TQ, min_run);
}

template <typename T, int GP>
void launch_single(const Exact& p, cudaStream_t s) {
    const int ranks = single_ranks(p.head_dim);
    const size_t smem = single_smem<T>(p.head_dim, p.n_q / p.n_kv);
    if (smem > 48 * 1024) cudaFuncSetAttribute((const void*)attention_exact_single_kernel<T, GP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gk_launch_cluster(attention_exact_single_kernel<T, GP>, dim3((unsigned)((long long)p.n_tokens * p.n_kv * ranks)), dim3(SINGLE_WARPS * 32), smem, s,
                      dim3(ranks, 1, 1), p);
}

int sm_count() {
    static const int sms = [] {
        int device = 0, n = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) n = 148;
        return n;
    }();
    return sms;
}

// Which kernels a step of heads of up to 128 takes, from what is known when it is captured: numbers of tokens and sequences, and
// the most tokens of one sequence where the caller knows (0: it does not).  Lengths are not known; a kernel that is the better one
// for long contexts has to bear short ones and the other way round.
struct Route {
    int single, tiles, min_run, warp_blocks;
};

// single: up to two and a half turns of the clusters that are on the device at once.  Measured (us, single / warps; 16/8 heads of 128,
//   32-bit; 16 tokens after 10, 1,000 and 3,000): 10.3, 64, 183 / 5.9, 202, 588; 32/8 heads of 64, bfloat16, 64 tokens after 10, 1,000
//   and 3,000: 13.5, 115, 332 / 7.0, 158, 460.
// tiles:  for steps beyond 16 warp units or 32 rows an SM, where a run can be long enough to fill tiles.  Measured (us, tiles /
//   warps; 16/8 heads of 128, 32-bit): 512 tokens after 1,000: 372 / 975; 64 single tokens after 1,000 and a prompt of 512: 376 / 660;
//   640 tokens in 16 runs of 40: 63 / 42; 16/1 heads of 128, 512 after 1,000: 381 / 559; 6/2 heads of 32, the same: 257 / 176.
// The mixed step took 7,477 us with tiles that walk every run of theirs, 64 tokens after 10 141 us with a cluster each (here 7), and
// the wide kernel for all of them 881 and 10.
Route exact_route(long long n_tokens, long long n_seqs, long long longest_run, int n_q, int n_kv, int head_dim, int dtype, int sms) {
    const int group = n_q / n_kv, TQ = TILE_ROWS / group, heads_a_warp = group >= 3 ? 4 : group;
    const size_t needs = dtype == GK_F32 ? single_smem<float>(head_dim, group) : single_smem<__nv_bfloat16>(head_dim, group);
    const long long resident = sms * std::min(group <= 8 ? 3LL : 2LL, (long long)(MAX_SMEM / (needs + 1024)));
    Route r{};
    if (2 * n_tokens * n_kv * single_ranks(head_dim) <= 5 * resident) {
        r.single = 1;
        return r;
    }
    const long long units = n_tokens * n_kv * ((group + heads_a_warp - 1) / heads_a_warp);
    const int least = (TQ + 1) / 2;
    r.tiles = (units > 16LL * sms || n_tokens * n_q > 32LL * sms) && n_tokens - (n_seqs - 1) >= least && (longest_run == 0 || longest_run >= 2 * TQ);
    r.min_run = r.tiles && n_seqs > 1 ? least : 0;
    if (!r.tiles || n_seqs > 1) r.warp_blocks = (int)std::min(2LL * sms, units);
    return r;
}

}  // namespace

// What exact_route answers, for tests: bit 0 single, bit 1 tiles, bit 2 warps.
GK_EXPORT int gk_attention_exact_route(int n_tokens, int n_seqs, int longest_run, int n_q, int n_kv, int head_dim, int dtype, int sms) {
    const Route r = exact_route(n_tokens, n_seqs, longest_run, n_q, n_kv, head_dim, dtype, sms);
    return r.single | r.tiles << 1 | (r.warp_blocks > 0) << 2;
}

// `n_seqs` (how many sequences the tokens belong to) and `longest_run` (the most tokens of one sequence, 0 where the caller does not
// know) are read by the choice of the kernels alone.
GK_EXPORT int gk_attention_exact(const void* q, const void* k_pages, const void* v_pages, void* out, int dtype,
                                 const int* tok_pos, const int* tok_seq, const int* slots, const int* block_table,
                                 int n_tokens, int n_q, int n_kv, int head_dim, int max_pages, int page_size,
                                 float scale, int window, int sink, int n_seqs, int longest_run, void* stream) {
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
        const Route r = exact_route(n_tokens, n_seqs, longest_run, n_q, n_kv, head_dim, dtype, sm_count());
        if (r.single) {
            GK_DISPATCH_DTYPE(dtype, T, {
                if (group == 1) launch_single<T, 1>(p, s);
                else if (group == 2) launch_single<T, 2>(p, s);
                else if (group <= 4) launch_single<T, 4>(p, s);
                else if (group <= 8) launch_single<T, 8>(p, s);
                else launch_single<T, 16>(p, s);
            })
            GK_CHECK_LAUNCH("attention_exact");
        }
        if (r.tiles) {
            GK_DISPATCH_DTYPE(dtype, T, { launch_tile<T>(p, r.min_run, s); })
            GK_CHECK_LAUNCH("attention_exact");
        }
        if (r.warp_blocks > 0) {
            GK_DISPATCH_DTYPE(dtype, T, {
                if (group == 1) launch_warps<T, 1>(p, r.min_run, r.warp_blocks, s);
                else if (group == 2) launch_warps<T, 2>(p, r.min_run, r.warp_blocks, s);
                else launch_warps<T, 4>(p, r.min_run, r.warp_blocks, s);
            })
            GK_CHECK_LAUNCH("attention_exact");
        }
        return GK_OK;
    }
    GK_DISPATCH_DTYPE(dtype, T, {
        gk_launch(attention_exact_kernel<T>, dim3((unsigned)blocks), dim3(WARPS * 32), smem, s,
            (const T*)q, (const T*)k_pages, (const T*)v_pages, (T*)out, tok_pos, tok_seq, slots, block_table, n_tokens,
            n_q, n_kv, head_dim, max_pages, page_size, scale, window, sink);
    })
    GK_CHECK_LAUNCH("attention_exact");
    return GK_OK;
}
