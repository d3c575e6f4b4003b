// Token choice from 32-bit logits: greedy argmax, and temperature (+ top-k) sampling.
//
// The reference samples with  logits / temperature -> optional top-k mask (values below the
// k-th largest become -inf, ties at the threshold survive) -> softmax -> multinomial
// (src/engine.py:5-12).  Here the multinomial draw is done with the Gumbel-max rule, which
// draws from exactly the same distribution: token = argmax_i (logit_i / T + g_i),
// g_i = -log(-log(u_i)), u_i uniform in (0,1).  u_i comes from a counter-based generator keyed by
// (seed, request, step, i), so a request's tokens do not depend on what else is in the batch
// and a host implementation can reproduce them.
//
// Ties go to the lowest index in both kernels.

#include <cstddef>

#include "common.cuh"

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 30;
    x *= 0xBF58476D1CE4E5B9ULL;
    x ^= x >> 27;
    x *= 0x94D049BB133111EBULL;
    x ^= x >> 31;
    return x;
}

__device__ __forceinline__ float uniform_open(unsigned long long seed, unsigned long long request,
                                              unsigned long long step, unsigned long long index) {
    unsigned long long x = seed * 0x9E3779B97F4A7C15ULL + request * 0xBF58476D1CE4E5B9ULL +
                           step * 0x94D049BB133111EBULL + index;
    x = mix64(x);
    return ((float)(x >> 41) + 0.5f) * (1.0f / 8388608.0f);
}

// Order-preserving map float -> uint32 (larger float, larger key).
__device__ __forceinline__ unsigned int float_key(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_float(unsigned int key) { return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key); }

struct Best {
    float value;
    int index;
};

__device__ __forceinline__ Best better(Best a, Best b) {
    if (b.value > a.value || (b.value == a.value && b.index < a.index)) return b;
    return a;
}

__device__ __forceinline__ Best block_best(Best mine, Best* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best other;
        other.value = __shfl_xor_sync(0xffffffffu, mine.value, o);
        other.index = __shfl_xor_sync(0xffffffffu, mine.index, o);
        mine = better(mine, other);
    }
    if (lane == 0) scratch[warp] = mine;
    __syncthreads();
    if (warp == 0) {
        Best t = lane < n_warps ? scratch[lane] : Best{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            Best other;
            other.value = __shfl_xor_sync(0xffffffffu, t.value, o);
            other.index = __shfl_xor_sync(0xffffffffu, t.index, o);
            t = better(t, other);
        }
        if (lane == 0) scratch[0] = t;
    }
    __syncthreads();
    return scratch[0];
}

// Every element of row[begin .. end) goes to `visit(value, index)`: the elements up to the first 16-byte
// boundary one by one, then four at a time with several loads of a thread in flight (a thread that waits for
// each element before it asks for the next scans at a few GB/s), then the rest.
template <typename Visit>
__device__ __forceinline__ void scan_slice(const float* __restrict__ row, int begin, int end, Visit visit) {
    const int lead = min((int)((16 - ((uintptr_t)(row + begin) & 15)) & 15) / 4, max(end - begin, 0));
    if ((int)threadIdx.x < lead) visit(row[begin + threadIdx.x], begin + (int)threadIdx.x);
    const int vec_begin = begin + lead, n_vec = max(end - vec_begin, 0) / 4;
    const float4* vec = reinterpret_cast<const float4*>(row + vec_begin);
    constexpr int IN_FLIGHT = 4;
    for (int v0 = threadIdx.x; v0 < n_vec; v0 += blockDim.x * IN_FLIGHT) {
        float4 got[IN_FLIGHT];
#pragma unroll
        for (int u = 0; u < IN_FLIGHT; ++u) {
            const int v = v0 + u * (int)blockDim.x;
            if (v < n_vec) got[u] = vec[v];
        }
#pragma unroll
        for (int u = 0; u < IN_FLIGHT; ++u) {
            const int v = v0 + u * (int)blockDim.x;
            if (v < n_vec) {
                const int i = vec_begin + 4 * v;
                visit(got[u].x, i);
                visit(got[u].y, i + 1);
                visit(got[u].z, i + 2);
                visit(got[u].w, i + 3);
            }
        }
    }
    for (int i = vec_begin + 4 * n_vec + threadIdx.x; i < end; i += blockDim.x) visit(row[i], i);
}

// What a scan of the whole slice leaves for one of its few large elements: the largest key of each thread's turns of sixteen
// elements, `per` turns together, [MARKS][blockDim.x] in shared memory.
constexpr int MARKS = 8;
__device__ __forceinline__ int turns_a_mark(int n_vec) { return (n_vec + (int)blockDim.x * 4 * MARKS - 1) / ((int)blockDim.x * 4 * MARKS); }

// The largest key among the thread's elements of row[begin .. end), and of each group of its turns.
__device__ __forceinline__ unsigned int scan_largest(const float* __restrict__ row, int begin, int end, unsigned int* marks) {
    const int lead = min((int)((16 - ((uintptr_t)(row + begin) & 15)) & 15) / 4, max(end - begin, 0));
    const int vec_begin = begin + lead, n_vec = max(end - vec_begin, 0) / 4, rest = vec_begin + 4 * n_vec, per = turns_a_mark(n_vec);
    const float4* vec = reinterpret_cast<const float4*>(row + vec_begin);
    unsigned int largest = 0, group = 0;
    if ((int)threadIdx.x < lead) largest = float_key(row[begin + threadIdx.x]);
    if ((int)threadIdx.x < end - rest) largest = max(largest, float_key(row[rest + threadIdx.x]));
    int left = per;
    unsigned int* mark = marks + threadIdx.x;
    for (int v0 = threadIdx.x; v0 < n_vec; v0 += blockDim.x * 4) {
        float4 got[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int v = v0 + u * (int)blockDim.x;
            if (v < n_vec) got[u] = vec[v];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (v0 + u * (int)blockDim.x < n_vec)
                group = max(group, max(max(float_key(got[u].x), float_key(got[u].y)), max(float_key(got[u].z), float_key(got[u].w))));
        if (--left == 0) {
            *mark = group;
            mark += blockDim.x;
            largest = max(largest, group);
            group = 0, left = per;
        }
    }
    if (left != per) *mark = group;
    return max(largest, group);
}

// The same for the elements whose key reaches `least`, of which there are few: what is done with one stands in the code once and
// fetches it again, instead of sixteen times behind the loads.  With `marks` (scan_largest's) only the turns among which there is one
// are fetched.
template <typename Visit>
__device__ __forceinline__ void scan_reaching(const float* __restrict__ row, int begin, int end, unsigned int least, Visit visit, const unsigned int* marks = nullptr) {
    const int lead = min((int)((16 - ((uintptr_t)(row + begin) & 15)) & 15) / 4, max(end - begin, 0));
    const int vec_begin = begin + lead, n_vec = max(end - vec_begin, 0) / 4, rest = vec_begin + 4 * n_vec;
    const float4* vec = reinterpret_cast<const float4*>(row + vec_begin);
    const float least_value = key_float(least);
    const auto maybe = [&](float x) { return !(x < least_value); };  // true for all that reach it, for a zero of the other sign and for NaN
    constexpr int IN_FLIGHT = 4;
    const int per = marks != nullptr ? turns_a_mark(n_vec) : 0;
    int turn = 0;
    // the last turn of all threads is for the elements beside the whole pieces: at most three in front and three behind
    for (int v0 = threadIdx.x;; v0 += blockDim.x * IN_FLIGHT, ++turn) {
        unsigned int hits = 0;
        int first = vec_begin + 4 * v0, step = 4 * (int)blockDim.x;
        const bool last = v0 >= n_vec;
        if (marks != nullptr && !last && marks[turn / per * (int)blockDim.x + (int)threadIdx.x] < least) continue;
        if (!last) {
            float4 got[IN_FLIGHT];
#pragma unroll
            for (int u = 0; u < IN_FLIGHT; ++u) {
                const int v = v0 + u * (int)blockDim.x;
                if (v < n_vec) got[u] = vec[v];
            }
#pragma unroll
            for (int u = 0; u < IN_FLIGHT; ++u) {
                if (maybe(got[u].x)) hits |= 1u << (4 * u);
                if (maybe(got[u].y)) hits |= 2u << (4 * u);
                if (maybe(got[u].z)) hits |= 4u << (4 * u);
                if (maybe(got[u].w)) hits |= 8u << (4 * u);
            }
            if (v0 + (IN_FLIGHT - 1) * (int)blockDim.x >= n_vec)  // what was not loaded
#pragma unroll
                for (int u = 1; u < IN_FLIGHT; ++u)
                    if (v0 + u * (int)blockDim.x >= n_vec) hits &= ~(15u << (4 * u));
        } else {
            if ((int)threadIdx.x < lead) hits |= 1u;
            if ((int)threadIdx.x < end - rest) hits |= 1u << 4;
            first = begin + (int)threadIdx.x, step = rest - begin;
        }
        for (; hits != 0; hits &= hits - 1) {
            const int bit = __ffs(hits) - 1, i = first + (bit >> 2) * step + (bit & 3);
            const float x = row[i];
            if (float_key(x) >= least) visit(x, i);
        }
        if (last) break;
    }
}

// Grid (parts, rows): block (p, r) scans its slice of row r and leaves its best (value, index) in
// `partial[r * parts + p]`; with one part it writes the answer itself.
__global__ void argmax_kernel(const float* __restrict__ logits, long long row_stride, int vocab,
                              int* __restrict__ out, Best* __restrict__ partial) {
    __shared__ Best scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const int parts = gridDim.x, part = blockIdx.x, r = blockIdx.y;
    const float* row = logits + (size_t)r * row_stride;
    const int per = (vocab + parts - 1) / parts;
    const int begin = part * per, end = min(begin + per, vocab);
    Best mine{-INFINITY, 0x7fffffff};
    scan_slice(row, begin, end, [&](float x, int i) { mine = better(mine, Best{x, i}); });
    Best b = block_best(mine, scratch);
    if (threadIdx.x == 0) {
        if (parts == 1) out[r] = b.index == 0x7fffffff ? 0 : b.index;
        else partial[(size_t)r * parts + part] = b;
    }
}

// One warp per row picks among the parts' results; `steps` (sampling only) is advanced here, once per row.
__global__ void best_merge_kernel(const Best* __restrict__ partial, int parts, int* __restrict__ out, int* __restrict__ steps) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x;
    Best mine{-INFINITY, 0x7fffffff};
    for (int p = threadIdx.x; p < parts; p += 32) mine = better(mine, partial[(size_t)r * parts + p]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Best other;
        other.value = __shfl_xor_sync(0xffffffffu, mine.value, o);
        other.index = __shfl_xor_sync(0xffffffffu, mine.index, o);
        mine = better(mine, other);
    }
    if (threadIdx.x == 0) {
        out[r] = mine.index == 0x7fffffff ? 0 : mine.index;
        if (steps) steps[r] += 1;
    }
}

// ---- top-k: the choice among the logits that reach the row's k-th largest, in one kernel.
//
// A cluster of up to SELECT_BLOCKS blocks shares a row (top_k up to half of MAX_KEYS).  The lanes of a warp, or a
// half, a quarter ... of them where k is larger, form a group, at least two groups for each of the k; of all groups' largest logits
// the k-th largest is a bound that at least k logits reach, and hardly more do (of random rows about 63 with 128 groups and k =
// 50).  The scan also leaves the largest key of every few turns of a thread, so that the second one, which lists the logits that reach the
// bound, fetches hardly anything; the cluster's first block gathers the blocks' lists, finds the k-th largest among them and draws.  So
// noise is formed for the candidates alone.  (With a second scan out of L2, and a request of the first block's list for every few
// candidates: 22.5 us instead of 22.0 for 64 rows of 151,936, k = 50, new logits every time.)  Where more logits reach the bound than
// a list holds, they are listed no further; if fewer than k of them are above it (rows of equal numbers, rows masked down to
// fewer than k), the bound is the k-th largest and a third scan draws.  Else (rows in order), as for larger k: a radix select over the
// order-preserving keys, eight bits a scan, with the blocks' histograms added up through distributed shared memory, and a last scan
// that draws.
// Bound by the scan (10 us of new logits) and the cluster's barriers behind it.  A block has 40 registers a thread (three blocks an SM, a few of
// them spilled): with four blocks an SM and 32 registers 64 rows of 151,936 took 22.0 us instead of 17.4.
constexpr int SELECT_BLOCKS = 8, SELECT_THREADS = 512, MAX_KEYS = 512, CANDIDATES = 2048;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t remote_address(const void* mine, int rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
    return remote;
}
__device__ __forceinline__ unsigned int remote_read(const void* mine, int rank) {
    unsigned int v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote_address(mine, rank)) : "memory");
    return v;
}

struct Draw {
    float temperature;
    unsigned long long seed, request, step;
    __device__ __forceinline__ Best of(float x, int i) const {
        if (x == -INFINITY) return Best{x, i};  // whatever the noise
        const float u = uniform_open(seed, request, step, (unsigned long long)i);
        const float g = -logf(-logf(u));
        return Best{x / temperature + g, i};
    }
};

struct CandidateList {
    int2 entries[CANDIDATES];  // a logit's bits and its index
    unsigned int count;
};

struct SelectShared {
    unsigned int hist[2][256], total[256], sel_prefix, sel_remaining;
};

// The key of the row's k-th largest logit, by the long way.  Two histograms in turn, so that a block may clear the next one
// while others still read this one.  Lanes that meet in a bin add to it once.  `least`: a key that is not above the k-th largest.
__device__ __noinline__ unsigned int radix_threshold(const float* __restrict__ row, int begin, int end, int top_k, int n_ranks, unsigned int least,
                                                     SelectShared& sh) {
    const int lane = threadIdx.x & 31;
    unsigned int prefix = 0, mask = 0;
    if (threadIdx.x == 0) sh.sel_remaining = (unsigned)top_k;
    if (threadIdx.x < 256) sh.hist[0][threadIdx.x] = 0;
    __syncthreads();
    int pass = 0;
    for (int shift = 24; shift >= 0; shift -= 8, ++pass) {
        unsigned int* mine = sh.hist[pass & 1];
        scan_slice(row, begin, end, [&](float x, int) {
            const unsigned int key = float_key(x);
            if ((key & mask) == prefix && key >= least) {
                const unsigned int bin = (key >> shift) & 255u;
                const unsigned int same = __match_any_sync(__activemask(), bin);
                if (lane == __ffs(same) - 1) atomicAdd(&mine[bin], (unsigned)__popc(same));
            }
        });
        cluster_barrier();  // every block's counts of this pass are complete
        if (threadIdx.x < 256) {
            unsigned int sum = 0;
            for (int b = 0; b < n_ranks; ++b) sum += remote_read(&mine[threadIdx.x], b);
            sh.total[threadIdx.x] = sum;
            sh.hist[(pass + 1) & 1][threadIdx.x] = 0;  // last read a pass ago, before the barrier above
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            // from the highest bin down: lane l sums bins 255 - 8l .. 248 - 8l, the warp finds the lane in whose
            // bins the count reaches what is still wanted, and that lane finds the bin
            const unsigned int remaining = sh.sel_remaining;
            unsigned int own = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) own += sh.total[255 - 8 * lane - j];
            unsigned int upto = own;  // inclusive sum over lanes 0 .. lane
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int other = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += other;
            }
            const unsigned int reached = __ballot_sync(0xffffffffu, upto >= remaining);
            const int owner = reached ? __ffs(reached) - 1 : 31;
            if (lane == owner) {
                unsigned int cum = upto - own;
                int chosen = 248 - 8 * lane;
                for (int j = 0; j < 8; ++j) {
                    const int b = 255 - 8 * lane - j;
                    if (cum + sh.total[b] >= remaining) {
                        chosen = b;
                        break;
                    }
                    cum += sh.total[b];
                }
                sh.sel_remaining = remaining - cum;
                sh.sel_prefix = prefix | ((unsigned)chosen << shift);
            }
        }
        __syncthreads();
        prefix = sh.sel_prefix;
        mask |= 255u << shift;
    }
    return prefix;
}

// The least of keys[first .. first + count - 1] (up to MAX_KEYS of them) in front of which fewer than k of keys[0 .. n - 1] stand
// (larger ones): over all n keys that is the k-th largest.  As many threads a key as there are take a run of the n each, a warp
// the same run, four keys a load.  `in_front` holds zeros and `*least` all ones before and `in_front` zeros afterwards; a barrier
// stands between that and the call.  (One thread for each of 512 keys, which goes through all of them, took 29 of 43 us for 64 rows of
// 32,000 with k = 65.)
__device__ __noinline__ unsigned int least_of_first(const unsigned int* keys, int n, int k, int first, int count, unsigned int* in_front, unsigned int* least) {
    if (n <= 128) {  // first = 0, count = n: a thread a key, and whoever stands on the k-th place says so
        if ((int)threadIdx.x < n) {
            const unsigned int mine = keys[threadIdx.x];
            int front = 0;
#pragma unroll 8
            for (int j = 0; j < n; ++j) front += keys[j] > mine || (keys[j] == mine && j < (int)threadIdx.x);
            if (front == k - 1) *least = mine;
        }
        __syncthreads();
        return *least;
    }
    const int padded = (count + 31) & ~31, runs = SELECT_THREADS / padded, run = (int)threadIdx.x / padded, at = (int)threadIdx.x - run * padded;
    const int length = ((n + runs - 1) / runs + 3) & ~3, end = min(n, (run + 1) * length);
    if (run < runs) {
        const unsigned int mine = at < count ? keys[first + at] : 0u;
        unsigned int larger = 0;
        int j = run * length;
#pragma unroll 4
        for (; j + 4 <= end; j += 4) {
            const uint4 four = *reinterpret_cast<const uint4*>(keys + j);
            larger += (four.x > mine) + (four.y > mine) + (four.z > mine) + (four.w > mine);
        }
        for (; j < end; ++j) larger += keys[j] > mine;
        if (at < count) atomicAdd(&in_front[at], larger);
    }
    __syncthreads();
    if ((int)threadIdx.x < padded) {
        const unsigned int mine = (int)threadIdx.x < count && in_front[threadIdx.x] < (unsigned int)k ? keys[first + threadIdx.x] : 0xffffffffu;
        const unsigned int of_warp = __reduce_min_sync(0xffffffffu, mine);
        if ((threadIdx.x & 31) == 0) atomicMin(least, of_warp);
        in_front[threadIdx.x] = 0;
    }
    __syncthreads();
    return *least;
}

// The k-th largest of keys[0 .. n - 1] (n >= k), the same in all threads: the largest number that k keys reach, four bits a turn,
// each of sixteen warps counting for one value of the four.  For lists where counting all pairs takes longer.
__device__ __noinline__ unsigned int kth_of_many(const unsigned int* keys, int n, int k, unsigned int (*enough)[16]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int reached = 0;
    int turn = 0;
    for (int shift = 28; shift >= 0; shift -= 4, turn ^= 1) {
        const unsigned int wanted = reached | ((unsigned int)warp << shift);
        unsigned int count = 0;
        for (int i = lane; i < n; i += 32) count += keys[i] >= wanted;
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0) enough[turn][warp] = count >= (unsigned int)k;
        __syncthreads();  // two sets of answers in turn: one barrier a turn
        const unsigned int those = __ballot_sync(0xffffffffu, enough[turn][lane & 15] != 0) & 0xffffu;
        reached |= (31u - __clz(those)) << shift;
    }
    return reached;
}

// The thresholds of all rows, for sample_kernel.
__global__ void __launch_bounds__(1024, 1) top_k_threshold_kernel(const float* __restrict__ logits, long long row_stride, int vocab, int top_k,
                                                                  unsigned int* __restrict__ threshold) {
    __shared__ SelectShared sh;
    pdl_launch_dependents();
    pdl_wait();
    uint32_t n_ranks;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_ranks));
    const int r = blockIdx.x / (int)n_ranks, rank = blockIdx.x % (int)n_ranks;  // the cluster's blocks are consecutive
    const int per = (vocab + (int)n_ranks - 1) / (int)n_ranks;
    const int begin = min(rank * per, vocab), end = min(begin + per, vocab);
    const unsigned int found = radix_threshold(logits + (size_t)r * row_stride, begin, end, top_k, (int)n_ranks, 0u, sh);
    if (threadIdx.x == 0 && rank == 0) threshold[r] = found;
    cluster_barrier();  // nobody leaves while its histogram may still be read
}

__global__ void __launch_bounds__(SELECT_THREADS, 3) sample_top_k_kernel(
    const float* __restrict__ logits, long long row_stride, int vocab, int top_k, float temperature, unsigned long long seed,
    const int* __restrict__ request_ids, int* __restrict__ steps, int advance_steps, int* __restrict__ out) {
    __shared__ SelectShared sh;
    __shared__ Best scratch[32], block_result;
    __shared__ __align__(16) unsigned int keys[CANDIDATES];  // first the groups' largest keys, then the candidates' keys
    __shared__ unsigned int own_keys[MAX_KEYS], enough[2][16], in_front[MAX_KEYS], bounds[2], n_above, counts[SELECT_BLOCKS];
    __shared__ CandidateList list;
    __shared__ unsigned int marks[MARKS * SELECT_THREADS];
    pdl_launch_dependents();
    pdl_wait();
    uint32_t n_ranks_raw;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n_ranks_raw));
    const int n_ranks = (int)n_ranks_raw, r = blockIdx.x / n_ranks, rank = blockIdx.x % n_ranks;  // the cluster's blocks are consecutive
    const float* row = logits + (size_t)r * row_stride;
    const int per = (vocab + n_ranks - 1) / n_ranks;
    const int begin = min(rank * per, vocab), end = min(begin + per, vocab);
    const auto key_of_row = [&] { return Draw{temperature, seed, (unsigned long long)(unsigned int)request_ids[r], (unsigned long long)(unsigned int)steps[r]}; };
    Best mine{-INFINITY, 0x7fffffff};
    bool settled = false, known = false;  // the same in all blocks of the cluster
    unsigned int threshold = 0;           // the k-th largest key, where it is known
    int lanes = 32;                       // of a group
    while (lanes > 1 && 2 * top_k > n_ranks * (SELECT_THREADS / lanes) && n_ranks * (SELECT_THREADS / lanes) < MAX_KEYS) lanes /= 2;
    const int groups = SELECT_THREADS / lanes;  // in a block
    unsigned int least = 0;  // no smaller key can be the k-th largest
    if (2 * top_k <= n_ranks * groups) {  // so it is for every top_k that comes here, up to half of MAX_KEYS
        if (threadIdx.x == 0) list.count = 0, n_above = 0, bounds[0] = bounds[1] = 0xffffffffu;
        in_front[threadIdx.x] = 0;
        unsigned int largest = scan_largest(row, begin, end, marks);
        for (int o = 1; o < lanes; o <<= 1) largest = max(largest, __shfl_xor_sync(0xffffffffu, largest, o));
        if (threadIdx.x % lanes == 0) own_keys[threadIdx.x / lanes] = largest;
        cluster_barrier();
        for (int i = threadIdx.x; i < n_ranks * groups; i += SELECT_THREADS) keys[i] = remote_read(&own_keys[i % groups], i / groups);
        __syncthreads();
        const int n_keys = n_ranks * groups;
        unsigned int reach;
        if (n_keys <= 256) {
            reach = least_of_first(keys, n_keys, top_k, 0, n_keys, in_front, &bounds[0]);
        } else {  // every block looks among its own groups' keys
            least_of_first(keys, n_keys, top_k, rank * groups, groups, in_front, &bounds[0]);
            cluster_barrier();
            reach = 0xffffffffu;
            for (int b = 0; b < n_ranks; ++b) reach = min(reach, remote_read(&bounds[0], b));
        }
        // into the block's own list: a request of another SM for every few of them would be most of this scan
        bool full = false;
        unsigned int above = 0;
        scan_reaching(row, begin, end, reach, [&](float x, int i) {
            above += float_key(x) > reach;
            if (full) return;
            const unsigned int at = atomicAdd(&list.count, 1u);
            if (at < CANDIDATES) list.entries[at] = make_int2(__float_as_int(x), i);
            else full = true;
        }, marks);
        for (int o = 1; o < 32; o <<= 1) above += __shfl_xor_sync(0xffffffffu, above, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(&n_above, above);
        cluster_barrier();
        if ((int)threadIdx.x < n_ranks) counts[threadIdx.x] = remote_read(&list.count, threadIdx.x);
        __syncthreads();
        int n = 0;
        for (int b = 0; b < n_ranks; ++b) n += (int)counts[b];
        settled = n <= CANDIDATES;
        if (settled && rank == 0) {  // the others' lists behind this block's own
            for (int i = threadIdx.x; i < n; i += SELECT_THREADS) {
                int b = 0, at = i;
                while (at >= (int)counts[b]) at -= (int)counts[b++];
                if (b > 0) list.entries[i] = make_int2((int)remote_read(&list.entries[at].x, b), (int)remote_read(&list.entries[at].y, b));
                keys[i] = float_key(__int_as_float(list.entries[i].x));
            }
            __syncthreads();
            const unsigned int kth = n <= MAX_KEYS ? least_of_first(keys, n, top_k, 0, n, in_front, &bounds[1]) : kth_of_many(keys, n, top_k, enough);
            const Draw draw = key_of_row();
            for (int i = threadIdx.x; i < n; i += SELECT_THREADS)
                if (keys[i] >= kth) mine = better(mine, draw.of(__int_as_float(list.entries[i].x), list.entries[i].y));
        }
        if (!settled) {  // fewer than k logits above the bound, which at least k reach: it is the k-th largest itself
            unsigned int all = 0;
            for (int b = 0; b < n_ranks; ++b) all += remote_read(&n_above, b);
            known = all < (unsigned int)top_k;
            threshold = least = reach;
        }
    }
    if (!settled) {
        if (!known) threshold = radix_threshold(row, begin, end, top_k, n_ranks, least, sh);
        const Draw draw = key_of_row();
        scan_reaching(row, begin, end, threshold, [&](float x, int i) { mine = better(mine, draw.of(x, i)); });
    }
    if (!settled || rank == 0) {
        const Best b = block_best(mine, scratch);
        if (threadIdx.x == 0) block_result = b;
    }
    cluster_barrier();  // the blocks' results are there, and nobody reads another block's histogram or list any more
    if (rank == 0 && threadIdx.x == 0) {
        Best b = block_result;
        if (!settled)
            for (int o = 1; o < n_ranks; ++o) b = better(b, Best{__uint_as_float(remote_read(&block_result.value, o)), (int)remote_read(&block_result.index, o)});
        out[r] = b.index == 0x7fffffff ? 0 : b.index;
        if (advance_steps) steps[r] += 1;
    }
    cluster_barrier();  // nobody leaves while its result may still be read
}

// Grid (parts, rows): the best of  logit / T + Gumbel noise  over the block's slice of the row, among the logits whose key reaches
// the row's threshold (`threshold` null: all).
__global__ void sample_kernel(const float* __restrict__ logits, long long row_stride, int vocab, float temperature,
                              const unsigned int* __restrict__ threshold, unsigned long long seed,
                              const int* __restrict__ request_ids, int* __restrict__ steps, int advance_steps,
                              int* __restrict__ out, Best* __restrict__ partial) {
    __shared__ Best scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const int parts = gridDim.x, part = blockIdx.x, r = blockIdx.y;
    const float* row = logits + (size_t)r * row_stride;
    const int per = (vocab + parts - 1) / parts;
    const int begin = part * per, end = min(begin + per, vocab);
    const Draw draw{temperature, seed, (unsigned long long)(unsigned int)request_ids[r], (unsigned long long)(unsigned int)steps[r]};
    Best mine{-INFINITY, 0x7fffffff};
    const unsigned int least = threshold != nullptr ? threshold[r] : 0u;
    scan_slice(row, begin, end, [&](float x, int i) {
        if (float_key(x) >= least) mine = better(mine, draw.of(x, i));
    });
    Best b = block_best(mine, scratch);
    if (threadIdx.x == 0) {
        if (parts == 1) {
            out[r] = b.index == 0x7fffffff ? 0 : b.index;
            if (advance_steps) steps[r] = (int)draw.step + 1;
        } else {
            partial[(size_t)r * parts + part] = b;
        }
    }
}

}  // namespace

// `scratch` (8 bytes * n_rows * parts) is needed when `parts` > 1: a row is then scanned by that many
// blocks and a second kernel picks among their results (ties still go to the lowest index).
GK_EXPORT int gk_argmax(const float* logits, long long row_stride, int n_rows, int vocab, int* out, int parts,
                        void* scratch, void* stream) {
    GK_REQUIRE(n_rows >= 0 && vocab > 0 && row_stride >= vocab, "argmax: bad sizes rows=%d vocab=%d", n_rows, vocab);
    GK_REQUIRE(parts >= 1 && parts <= 1024 && n_rows <= 65535, "argmax: bad split %d of %d rows", parts, n_rows);
    GK_REQUIRE(parts == 1 || scratch, "argmax: scratch is needed when a row is split");
    if (n_rows == 0) return GK_OK;
    gk_launch(argmax_kernel, dim3(parts, n_rows), dim3(parts == 1 ? 1024 : 256), 0, (cudaStream_t)stream, logits,
              row_stride, vocab, out, (Best*)scratch);
    GK_CHECK_LAUNCH("argmax");
    if (parts > 1) {
        gk_launch(best_merge_kernel, dim3(n_rows), dim3(32), 0, (cudaStream_t)stream, (const Best*)scratch, parts, out, (int*)nullptr);
        GK_CHECK_LAUNCH("argmax_merge");
    }
    return GK_OK;
}

// `scratch`: 4 bytes * n_rows for thresholds (rounded up to 8), then 8 bytes * n_rows * parts for the parts' results; not read with
// a top_k of up to half of MAX_KEYS.
GK_EXPORT int gk_sample(const float* logits, long long row_stride, int n_rows, int vocab, float temperature, int top_k,
                        unsigned long long seed, const int* request_ids, int* steps, int advance_steps, int* out,
                        int parts, void* scratch, void* stream) {
    GK_REQUIRE(n_rows >= 0 && vocab > 0 && row_stride >= vocab, "sample: bad sizes rows=%d vocab=%d", n_rows, vocab);
    GK_REQUIRE(temperature > 0.f, "sample: temperature must be positive (0 means greedy: call argmax)");
    GK_REQUIRE(top_k >= 0, "sample: top_k must be >= 0 (0 = off)");
    GK_REQUIRE(parts >= 1 && parts <= 1024 && n_rows <= 65535, "sample: bad split %d of %d rows", parts, n_rows);
    const bool select = top_k > 0 && top_k < vocab, short_way = select && top_k <= MAX_KEYS / 2;
    GK_REQUIRE((parts == 1 && !select) || short_way || scratch, "sample: scratch is needed for a large top_k and when a row is split");
    if (n_rows == 0) return GK_OK;
    cudaStream_t s = (cudaStream_t)stream;
    static const int n_sms = [] {
        int device = 0, n = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) n = 148;
        return n;
    }();
    int blocks = SELECT_BLOCKS;
    if (short_way) {
        // As many blocks a row as leaves all of them on the GPU at once (three of 512 threads fit an SM).  Measured (us; the threshold by
        // four counting scans, a scan that draws and a join in three kernels / here): 64 rows of 151,936, k = 50: 65.4 / 17.4, k = 200:
        // 66.8 / 24.6; 64 rows of 32,000, k = 200: 30.0 / 17.0; one row of 151,936, k = 50: 24.6 / 10.7.  Rows of equal numbers: 64: 101 /
        // 86, one: 29.8 / 36 (its eight blocks form all the noise, which the three kernels spread); rows masked down to 25: 64: 116 / 59,
        // one: 32.4 / 28.  Larger k: the three kernels; in one kernel a row of 151,936 took 32 instead of 24.6 us with k = 257.
        while (blocks > 1 && (long long)n_rows * blocks > 3LL * n_sms) blocks /= 2;
        gk_launch_cluster(sample_top_k_kernel, dim3(n_rows * blocks), dim3(SELECT_THREADS), 0, s, dim3(blocks, 1, 1), logits, row_stride,
                          vocab, top_k, temperature, seed, request_ids, steps, advance_steps, out);
        GK_CHECK_LAUNCH("sample_top_k");
        return GK_OK;
    }
    unsigned int* threshold = select ? (unsigned int*)scratch : nullptr;
    Best* partial = (Best*)((char*)scratch + 8 * (((size_t)n_rows + 1) / 2));  // 8-byte aligned, after the thresholds
    if (select) {
        while (blocks > 1 && (long long)n_rows * blocks > 2LL * n_sms) blocks /= 2;  // two of 1,024 threads fit an SM
        gk_launch_cluster(top_k_threshold_kernel, dim3(n_rows * blocks), dim3(1024), 0, s, dim3(blocks, 1, 1), logits, row_stride, vocab, top_k,
                          threshold);
        GK_CHECK_LAUNCH("top_k_threshold");
    }
    gk_launch(sample_kernel, dim3(parts, n_rows), dim3(256), 0, s, logits, row_stride, vocab, temperature, (const unsigned int*)threshold, seed,
              request_ids, steps, advance_steps, out, partial);
    GK_CHECK_LAUNCH("sample");
    if (parts > 1) {
        gk_launch(best_merge_kernel, dim3(n_rows), dim3(32), 0, s, (const Best*)partial, parts, out, advance_steps ? steps : (int*)nullptr);
        GK_CHECK_LAUNCH("sample_merge");
    }
    return GK_OK;
}
