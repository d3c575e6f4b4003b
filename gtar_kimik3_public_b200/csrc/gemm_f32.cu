// True 32-bit matrix product  C[M,N] = A[M,K] * W[N,K]^T  on the FP32 pipes (FFMA only: no
// tensor cores, no TF32, no reduced-precision accumulation).  nn.Linear without bias, as
// every projection of the reference is (src/layers/attention.py:62-65, src/layers/swiglu.py:9-11).
//
// Each output element is one chain  acc = fma(a[k], w[k], acc)  for k = 0..K-1 in order.  The
// chain does not depend on M, on the tile the element falls in, or on the other rows, so a
// token's result is bit-equal however the tokens are cut into steps or batches.
//
// A may be float or bfloat16 (converted exactly), C float or bfloat16 (rounded once).
//
// Three kernels form the same chains:
//   tile   many tokens: BM x BN outputs a block, TM x TN chains a thread, operands through a ring of cp.async stages
//          in shared memory as they lie in memory (rows of BK), so that a thread reads four steps of k of a row with
//          one 16-byte load and the lanes' rows (BK + 4 floats apart) fall into different banks.
//   wide   many tokens times many rows: 8 x 8 chains a thread, two in an instruction, operands turned on their way into shared memory
//   few    up to 16 tokens: a warp per eight rows of W, lane = (row, token), so that a step's chains spread over all SMs;
//          bound by the chain itself (4 cycles a step of k: 2.1 us for K = 1,024) beside the fetch of the weights, which
//          starts before the kernel in front has finished.

#include "common.cuh"

namespace {

__device__ __forceinline__ void copy16(void* smem, const void* gmem, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Rows row0 .. row0 + ROWS - 1 of a matrix, columns k0 .. k0 + BK - 1, into `dst` (rows STRIDE elements apart); what lies
// outside the matrix becomes zero.  VEC: every row starts on 16 bytes.
template <typename T, int ROWS, int BK, int STRIDE, int THREADS, bool VEC>
__device__ __forceinline__ void stage_rows(T* dst, const T* __restrict__ src, long long ld, int row0, int n_rows, int k0, int K, int tid) {
    if constexpr (VEC) {
        constexpr int PER = 16 / sizeof(T), CHUNKS = BK / PER;
        if (row0 + ROWS <= n_rows && k0 + BK <= K) {  // inside the matrix: no bounds to work out for every piece
            const T* from = src + (size_t)row0 * ld + k0;
#pragma unroll
            for (int i = tid; i < ROWS * CHUNKS; i += THREADS) copy16(dst + (i / CHUNKS) * STRIDE + (i % CHUNKS) * PER, from + (size_t)(i / CHUNKS) * ld + (i % CHUNKS) * PER, 16);
            return;
        }
#pragma unroll
        for (int i = tid; i < ROWS * CHUNKS; i += THREADS) {
            const int r = i / CHUNKS, k = (i % CHUNKS) * PER;
            const int left = row0 + r < n_rows ? K - (k0 + k) : 0;
            const int bytes = left <= 0 ? 0 : left >= PER ? 16 : left * (int)sizeof(T);
            copy16(dst + r * STRIDE + k, bytes > 0 ? src + (size_t)(row0 + r) * ld + k0 + k : src, bytes);
        }
    } else {
        for (int i = tid; i < ROWS * BK; i += THREADS) {
            const int r = i / BK, k = i % BK;
            dst[r * STRIDE + k] = row0 + r < n_rows && k0 + k < K ? src[(size_t)(row0 + r) * ld + k0 + k] : from_float<T>(0.f);
        }
    }
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

struct Product {
    const void* A;
    const float* W;
    void* C;
    int M, N, K;
    long long lda, ldw, ldc, batch_a, batch_w, batch_c;
};

constexpr int TILE_BK = 32, TILE_STAGES = 3;

template <typename TA, int BM, int BN>
constexpr size_t tile_smem() {
    return (size_t)TILE_STAGES * (BM * (TILE_BK + 16 / sizeof(TA)) * sizeof(TA) + BN * (TILE_BK + 4) * sizeof(float));
}

// Bound by the FP32 pipes, at a little over half of what two-number multiply-adds reach: one chain step an instruction, with the
// 16-byte reads of both operands beside them.  41 TFLOP/s at 2,048 x 4,096 x 4,096.  What it measured, and what the one tile of
// 128 x 128 with plain loads between two barriers measured before, stands at the launch rule.
template <typename TA, typename TC, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_f32_tile_kernel(const Product p) {
    constexpr int THREADS = (BM / TM) * (BN / TN), BK = TILE_BK, S = TILE_STAGES;
    constexpr int LDA = BK + 16 / sizeof(TA), LDW = BK + 4, RM = BM / TM, RN = BN / TN;
    extern __shared__ __align__(16) unsigned char smem[];
    float* ws = reinterpret_cast<float*>(smem);                   // [S][BN][LDW]
    TA* as = reinterpret_cast<TA*>(smem + (size_t)S * BN * LDW * sizeof(float));  // [S][BM][LDA]
    pdl_launch_dependents();
    const TA* A = (const TA*)p.A + (size_t)blockIdx.z * p.batch_a;  // a batch of products: one per grid plane
    const float* W = p.W + (size_t)blockIdx.z * p.batch_w;
    TC* C = (TC*)p.C + (size_t)blockIdx.z * p.batch_c;
    const int tid = threadIdx.x, tiles_m = (p.M + BM - 1) / BM;
    const int m0 = (int)(blockIdx.x % tiles_m) * BM, n0 = (int)(blockIdx.x / tiles_m) * BN;  // blocks side by side share rows of W
    const int tx = tid % RN, ty = tid / RN;
    const int steps = (p.K + BK - 1) / BK;
    // weights are written by no kernel in flight; activations may be
#pragma unroll
    for (int s = 0; s < S - 1; ++s)
        if (s < steps) stage_rows<float, BN, BK, LDW, THREADS, VEC>(ws + s * BN * LDW, W, p.ldw, n0, p.N, s * BK, p.K, tid);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (s < steps) stage_rows<TA, BM, BK, LDA, THREADS, VEC>(as + s * BM * LDA, A, p.lda, m0, p.M, s * BK, p.K, tid);
        copy_commit();
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    int at = 0, next = S - 1;
    for (int step = 0; step < steps; ++step) {
        copy_wait<S - 2>();
        __syncthreads();
        if (step + S - 1 < steps) {
            stage_rows<float, BN, BK, LDW, THREADS, VEC>(ws + next * BN * LDW, W, p.ldw, n0, p.N, (step + S - 1) * BK, p.K, tid);
            stage_rows<TA, BM, BK, LDA, THREADS, VEC>(as + next * BM * LDA, A, p.lda, m0, p.M, (step + S - 1) * BK, p.K, tid);
        }
        copy_commit();
        const float* w_at = ws + at * BN * LDW + tx * LDW;
        const TA* a_at = as + at * BM * LDA + ty * LDA;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float w[TN][4];
#pragma unroll
            for (int j = 0; j < TN; ++j) read4(w_at + j * RN * LDW + k, w[j]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float a[4];
                read4(a_at + i * RM * LDA + k, a);
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[e], w[j][e], acc[i][j]);
            }
        }
        at = at + 1 == S ? 0 : at + 1;
        next = next + 1 == S ? 0 : next + 1;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + i * RM;
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * RN;
            if (n < p.N) C[(size_t)m * p.ldc + n] = from_float<TC>(acc[i][j]);
        }
    }
}

// Two chains of neighbouring columns in one instruction, each rounded as by itself.
__device__ __forceinline__ void fma_two(unsigned long long& acc, unsigned long long a, unsigned long long w) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(w));
}
__device__ __forceinline__ unsigned long long twice(float a) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
    return d;
}

// Four entries of row `row` from k0 on, zeros where the row is not there and behind its end.
template <bool VEC, typename T>
__device__ __forceinline__ void fetch4(const T* __restrict__ src, long long ld, int row, bool there, int k0, int K, float (&v)[4]) {
    if (VEC && there && k0 + 4 <= K) {
        read4(src + (size_t)row * ld + k0, v);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = there && k0 + e < K ? to_float(src[(size_t)row * ld + k0 + e]) : 0.f;
}

constexpr int WIDE_BK = 16;

// A thread has TM rows of A and TN of W, as TM x TN / 2 pairs of chains.  Operands go through registers into shared memory, turned (a step
// of k is a row there), so that a 16-byte read brings four rows' entries of one step: what shared memory delivers, 128 bytes a clock
// whether lanes ask for the same ones or not, is TM + TN numbers a thread for TM TN chain steps.  N is a multiple of BN (the launch's rule).
template <typename TA, typename TC, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_f32_wide_kernel(const Product p) {
    constexpr int RN = BN / TN, THREADS = (BM / TM) * RN, BK = WIDE_BK, LDA = BM + 4, LDW = BN + 4;
    constexpr int NA = BM * BK / 4 / THREADS, NW = BN * BK / 4 / THREADS;  // pieces of four entries a thread fetches
    static_assert(BM * BK / 4 % THREADS == 0 && BN * BK / 4 % THREADS == 0 && TM % 4 == 0 && TN % 4 == 0, "whole pieces");
    __shared__ __align__(16) float as[2][BK][LDA], ws[2][BK][LDW];
    pdl_launch_dependents();
    const TA* A = (const TA*)p.A + (size_t)blockIdx.z * p.batch_a;  // a batch of products: one per grid plane
    const float* W = p.W + (size_t)blockIdx.z * p.batch_w;
    TC* C = (TC*)p.C + (size_t)blockIdx.z * p.batch_c;
    const int tid = threadIdx.x, tiles_m = (p.M + BM - 1) / BM;
    const int m0 = (int)(blockIdx.x % tiles_m) * BM, n0 = (int)(blockIdx.x / tiles_m) * BN;  // blocks side by side share rows of W
    const int tx = tid % RN, ty = tid / RN, row = tid / 4, piece = (tid % 4) * 4;
    const int steps = (p.K + BK - 1) / BK;
    float va[NA][4], vw[NW][4];
    const auto fetch_w = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NW; ++i) fetch4<VEC>(W, p.ldw, n0 + row + i * (THREADS / 4), true, k0 + piece, p.K, vw[i]);
    };
    const auto fetch_a = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int m = m0 + row + i * (THREADS / 4);
            fetch4<VEC>(A, p.lda, m, m < p.M, k0 + piece, p.K, va[i]);
        }
    };
    const auto put = [&](int half) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
            for (int i = 0; i < NW; ++i) ws[half][piece + e][row + i * (THREADS / 4)] = vw[i][e];
#pragma unroll
            for (int i = 0; i < NA; ++i) as[half][piece + e][row + i * (THREADS / 4)] = va[i][e];
        }
    };
    fetch_w(0);  // weights are written by no kernel in flight; activations may be
    pdl_wait();
    fetch_a(0);
    put(0);
    __syncthreads();
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
    for (int step = 0; step < steps; ++step) {
        const int half = step & 1;
        const bool more = step + 1 < steps;
        if (more) {
            fetch_w((step + 1) * BK);
            fetch_a((step + 1) * BK);
        }
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            ulonglong2 w[TN / 4];
            float4 a[TM / 4];
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(&ws[half][k][j * (BN / (TN / 4)) + 4 * tx]);
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) a[i] = *reinterpret_cast<const float4*>(&as[half][k][ty * TM + 4 * i]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 four = a[i / 4];
                const unsigned long long both = twice(i % 4 == 0 ? four.x : i % 4 == 1 ? four.y : i % 4 == 2 ? four.z : four.w);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma_two(acc[i][j], both, j & 1 ? w[j / 2].y : w[j / 2].x);
            }
        }
        if (more) put(half ^ 1);  // last read a step ago, in front of the barrier
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            const int n = n0 + j * (BN / (TN / 4)) + 4 * tx;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = __uint_as_float((uint32_t)(acc[i][2 * j + (e >> 1)] >> (32 * (e & 1))));
            TC* to = C + (size_t)m * p.ldc + n;
            if (sizeof(TC) == 4 && ((uintptr_t)to & 15) == 0) {
                *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
                continue;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) to[e] = from_float<TC>(v[e]);
        }
    }
}

constexpr int FEW_BK = 128, FEW_STAGES = 5, FEW_TOKENS = 16, FEW_ROWS = 8;

template <typename TA, int MI>
constexpr size_t few_smem() {
    return (size_t)FEW_STAGES * (FEW_ROWS * (FEW_BK + 4) * sizeof(float) + 4 * MI * (FEW_BK + 16 / sizeof(TA)) * sizeof(TA));
}

// One warp: eight rows of W, 4 MI tokens; a lane holds row lane % 8 and the tokens lane / 8 + 4 i.  Its own ring of five
// stages keeps 16 KB of weights on their way, so that a few warps an SM ask for enough of the memory's bandwidth.  Sixteen
// rows a warp (two a lane) were slower at every size tried, also where there are more warps than schedulers: 174 against
// 147 us for 8 tokens of 4,096 and 24,576 rows, 32 against 11 us for 3 tokens of 2,048 and 1,024 rows.
// Measured (us for 3 tokens; K x N), before / now: 1,024 x 4,096: 168 / 8.5, 3,072 x 1,024: 518 / 15.
template <typename TA, typename TC, int MI, bool VEC, bool WHOLE>
__global__ void __launch_bounds__(32) gemm_f32_few_kernel(const Product p) {
    constexpr int BK = FEW_BK, S = FEW_STAGES, LDA = BK + 16 / sizeof(TA), LDW = BK + 4, ROWS = FEW_ROWS, G = 4;
    extern __shared__ __align__(16) unsigned char smem[];
    float* ws = reinterpret_cast<float*>(smem);                                      // [S][ROWS][LDW]
    TA* as = reinterpret_cast<TA*>(smem + (size_t)S * ROWS * LDW * sizeof(float));  // [S][4 MI][LDA]
    pdl_launch_dependents();
    const TA* A = (const TA*)p.A + (size_t)blockIdx.z * p.batch_a;
    const float* W = p.W + (size_t)blockIdx.z * p.batch_w;
    TC* C = (TC*)p.C + (size_t)blockIdx.z * p.batch_c;
    const int lane = threadIdx.x, n0 = (int)blockIdx.x * ROWS;
    const int steps = (p.K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < S - 1; ++s)
        if (s < steps) stage_rows<float, ROWS, BK, LDW, 32, VEC>(ws + s * ROWS * LDW, W, p.ldw, n0, p.N, s * BK, p.K, lane);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (s < steps) stage_rows<TA, 4 * MI, BK, LDA, 32, VEC>(as + s * 4 * MI * LDA, A, p.lda, 0, p.M, s * BK, p.K, lane);
        copy_commit();
    }
    const int col = lane & 7, tok = lane >> 3;
    float acc[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) acc[i] = 0.f;
    int slot = 0, next = S - 1;
    if constexpr (WHOLE) {
        // The chain of multiply-adds is all that a warp should wait for, so nothing stands between two of them that can branch or
        // wait.  The next sixteen entries are read under the multiply-adds of these, across the ends of stages too, and a stage's copies
        // are asked for a quarter at a time between them (with no bytes behind the end).
        constexpr int CA = BK * sizeof(TA) / 16, AR = 4 * MI * CA / 32;  // 16-byte pieces of a token's row, and pieces a lane copies of all
        const float* w_from = W + (size_t)n0 * p.ldw + (S - 1) * BK + lane * 4;
        const TA* a_from[AR];
        int a_bytes[AR], a_to[AR];
#pragma unroll
        for (int i = 0; i < AR; ++i) {
            const int r = (lane + 32 * i) / CA, c = (lane + 32 * i) % CA * (16 / (int)sizeof(TA));
            a_bytes[i] = r < p.M ? 16 : 0;
            a_from[i] = A + (r < p.M ? (size_t)r * p.lda : 0) + (S - 1) * BK + c;
            a_to[i] = r * LDA + c;
        }
        float w[2][G][4], a[2][G][MI][4];
        const auto read = [&](int half, int from, int k) {
            const float* w_at = ws + (from * ROWS + col) * LDW + k;
            const TA* a_at = as + (from * 4 * MI + tok) * LDA + k;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                read4(w_at + 4 * g, w[half][g]);
#pragma unroll
                for (int i = 0; i < MI; ++i) read4(a_at + 4 * i * LDA + 4 * g, a[half][g][i]);
            }
        };
        constexpr int TURNS = BK / (4 * G);
        copy_wait<S - 2>();
        __syncwarp();
        read(0, 0, 0);
        for (int step = 0; step < steps; ++step) {
            const int after = slot + 1 == S ? 0 : slot + 1;
            const bool more = step + S - 1 < steps;
            float* w_to = ws + next * ROWS * LDW + lane * 4;
            TA* a_dst = as + next * 4 * MI * LDA;
#pragma unroll
            for (int h = 0; h < TURNS; ++h) {
                if (h + 1 < TURNS) {
                    read((h + 1) & 1, slot, (h + 1) * 4 * G);
                } else {
                    copy_wait<S - 2>();  // the next stage, of what was asked for (behind the last one: nothing)
                    __syncwarp();
                    read((h + 1) & 1, after, 0);
                }
#pragma unroll
                for (int r = h * 2; r < h * 2 + 2 && r < ROWS; ++r) copy16(w_to + r * LDW, more ? w_from + (size_t)r * p.ldw : W, more ? 16 : 0);
#pragma unroll
                for (int i = 0; i < AR; ++i)
                    if (i % 4 == h) copy16(a_dst + a_to[i], more ? a_from[i] : A, more ? a_bytes[i] : 0);
                if (h == 4) copy_commit();
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int i = 0; i < MI; ++i) acc[i] = fmaf(a[h & 1][g][i][e], w[h & 1][g][e], acc[i]);
            }
            w_from += BK;
#pragma unroll
            for (int i = 0; i < AR; ++i) a_from[i] += BK;
            slot = after;
            next = next + 1 == S ? 0 : next + 1;
        }
        copy_wait<0>();
    } else {
        for (int step = 0; step < steps; ++step) {
            copy_wait<S - 2>();
            __syncwarp();
            if (step + S - 1 < steps) {
                stage_rows<float, ROWS, BK, LDW, 32, VEC>(ws + next * ROWS * LDW, W, p.ldw, n0, p.N, (step + S - 1) * BK, p.K, lane);
                stage_rows<TA, 4 * MI, BK, LDA, 32, VEC>(as + next * 4 * MI * LDA, A, p.lda, 0, p.M, (step + S - 1) * BK, p.K, lane);
            }
            copy_commit();
            const float* w_at = ws + (slot * ROWS + col) * LDW;
            const TA* a_at = as + (slot * 4 * MI + tok) * LDA;
            float w[2][G][4], a[2][G][MI][4];
            const auto read = [&](int half, int k) {
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    read4(w_at + k + 4 * g, w[half][g]);
#pragma unroll
                    for (int i = 0; i < MI; ++i) read4(a_at + 4 * i * LDA + k + 4 * g, a[half][g][i]);
                }
            };
            read(0, 0);
#pragma unroll
            for (int k = 0; k < BK; k += 4 * G) {
                const int half = (k / (4 * G)) & 1;
                if (k + 4 * G < BK) read(half ^ 1, k + 4 * G);
#pragma unroll
                for (int g = 0; g < G; ++g)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
#pragma unroll
                        for (int i = 0; i < MI; ++i) acc[i] = fmaf(a[half][g][i][e], w[half][g][e], acc[i]);
            }
            slot = slot + 1 == S ? 0 : slot + 1;
            next = next + 1 == S ? 0 : next + 1;
        }
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int m = tok + 4 * i, n = n0 + col;
        if (m < p.M && n < p.N) C[(size_t)m * p.ldc + n] = from_float<TC>(acc[i]);
    }
}

template <typename K>
void launch_with_smem(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t s, const Product& p) {
    if (smem > 48 * 1024) cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    gk_launch(kernel, grid, dim3(threads), smem, s, p);
}

template <typename TA, typename TC, bool VEC, int MI>
void launch_few(const Product& p, int batch, int sms, cudaStream_t s) {
    const dim3 grid((p.N + FEW_ROWS - 1) / FEW_ROWS, 1, batch);
    // Whole stages of whole groups of rows, where the chains are what a launch waits for: up to two warps an SM, or four chains a lane.
    // Measured (us, K x N, the general form / here): 3 tokens: 3,072 x 1,024: 13.9 / 10.4, 2,048 x 1,024: 9.8 / 7.8, 1,024 x 6,144 (five warps
    // an SM): 11.4 / 11.8; 8 tokens, 1,024 x 6,144: 15.2 / 15.9; 16 tokens: 3,072 x 1,024: 26.7 / 20.6, 1,024 x 6,144: 26.1 / 23.0.
    if constexpr (VEC) {
        if (p.K % FEW_BK == 0 && p.N % FEW_ROWS == 0 && (MI == 4 || (long long)grid.x * batch <= 2LL * sms)) {
            launch_with_smem(gemm_f32_few_kernel<TA, TC, MI, true, true>, grid, 32, few_smem<TA, MI>(), s, p);
            return;
        }
    }
    launch_with_smem(gemm_f32_few_kernel<TA, TC, MI, VEC, false>, grid, 32, few_smem<TA, MI>(), s, p);
}

template <typename TA, typename TC, bool VEC, int BM, int BN, int TM, int TN>
void launch_tile(const Product& p, int batch, cudaStream_t s) {
    const unsigned tiles = (unsigned)((p.M + BM - 1) / BM) * (unsigned)((p.N + BN - 1) / BN);
    launch_with_smem(gemm_f32_tile_kernel<TA, TC, BM, BN, TM, TN, VEC>, dim3(tiles, 1, batch), (BM / TM) * (BN / TN), tile_smem<TA, BM, BN>(), s, p);
}

template <typename TA, typename TC, bool VEC, int BM, int BN, int TM, int TN>
void launch_wide(const Product& p, int batch, cudaStream_t s) {
    const unsigned tiles = (unsigned)((p.M + BM - 1) / BM) * (unsigned)((p.N + BN - 1) / BN);
    gk_launch(gemm_f32_wide_kernel<TA, TC, BM, BN, TM, TN, VEC>, dim3(tiles, 1, batch), dim3((BM / TM) * (BN / TN)), 0, s, p);
}

template <typename TA, typename TC, bool VEC>
void launch_product(const Product& p, int batch, cudaStream_t s) {
    static const int sms = [] {
        int device = 0, n = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
        return n > 0 ? n : 148;
    }();
    if (p.M <= 4) launch_few<TA, TC, VEC, 1>(p, batch, sms, s);
    else if (p.M <= 8) launch_few<TA, TC, VEC, 2>(p, batch, sms, s);
    else if (p.M <= FEW_TOKENS) launch_few<TA, TC, VEC, 4>(p, batch, sms, s);
    // Tiles of 64 x 64 (8 x 4 chains a thread) where there are two for every SM, else of 32 x 32 (4 x 4 chains), which lose a
    // fifth to shared memory but spread.  Measured (us, 64 / 32; tokens x N x K): 2,048 x 4,096 x 4,096: 1,669 / 1,986;
    // 805 x 6,144 x 1,024: 275 / 307; 805 x 1,024 x 2,048 (208 tiles of 64): 127 / 114; 128 x 6,144 x 1,024 (192): 65 / 59;
    // 33 x 4,096 x 1,024 (64): 41 / 26.  Tiles of 128 x 128 lose at all of these (8 x 16 chains a thread: 1,955 at the first).
    // Before, with tiles of 128 x 128 alone: 3,247, 695, 424, 221 and 176.
    // Tiles of 64 x 128 (8 x 8 chains a thread, in pairs) where an SM has some two of them or more and their columns are whole.  Measured (us,
    // tiles of 64 x 64 below / here): 2,048 x 4,096 x 4,096: 1,632 / 1,414; 805 x 6,144 x 1,024 (624 tiles): 272 / 258; 805 x 4,096 x 1,024: 184 /
    // 159; 384 x 6,144 x 1,024 (288): 123 / 113; 805 x 3,000 x 1,024 (312, the last half empty): 159 / 161; 128 x 6,144 x 1,024 (96): 58 / 72.
    // 8 x 16 chains a thread: 1,523 to 1,586 at the first (two warps a scheduler are too few for its reads).
    else if (p.N % 128 == 0 && 4 * (long long)((p.M + 63) / 64) * (p.N / 128) * batch >= 7LL * sms) launch_wide<TA, TC, VEC, 64, 128, 8, 8>(p, batch, s);
    else if ((long long)((p.M + 63) / 64) * ((p.N + 63) / 64) * batch >= 2LL * sms) launch_tile<TA, TC, VEC, 64, 64, 8, 4>(p, batch, s);
    else launch_tile<TA, TC, VEC, 32, 32, 4, 4>(p, batch, s);
}

// Copies of 16 bytes want every row of both operands on 16 bytes.
bool rows_aligned(const Product& p, size_t size_a) {
    const auto whole = [](long long elements, size_t size) { return (elements * (long long)size) % 16 == 0; };
    return (((uintptr_t)p.A | (uintptr_t)p.W) & 15) == 0 && whole(p.lda, size_a) && whole(p.batch_a, size_a) && whole(p.ldw, 4) && whole(p.batch_w, 4);
}

void dispatch_product(const Product& p, int a_dtype, int c_dtype, int batch, cudaStream_t s) {
    GK_DISPATCH_DTYPE(a_dtype, TA, {
        GK_DISPATCH_DTYPE(c_dtype, TC, {
            if (rows_aligned(p, sizeof(TA))) launch_product<TA, TC, true>(p, batch, s);
            else launch_product<TA, TC, false>(p, batch, s);
        })
    })
}

}  // namespace

GK_EXPORT int gk_gemm_f32(const void* A, int a_dtype, const float* W, void* C, int c_dtype, int M, int N, int K,
                          long long lda, long long ldw, long long ldc, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(a_dtype) && GK_VALID_DTYPE(c_dtype), "gemm_f32: bad dtype code");
    GK_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    GK_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: a leading dimension is shorter than its row");
    if (M == 0) return GK_OK;
    GK_REQUIRE((M + 127) / 128 <= 65535, "gemm_f32: M=%d needs more than 65535 row tiles", M);
    dispatch_product(Product{A, W, C, M, N, K, lda, ldw, ldc, 0, 0, 0}, a_dtype, c_dtype, 1, (cudaStream_t)stream);
    GK_CHECK_LAUNCH("gemm_f32");
    return GK_OK;
}

// `batch` products at once: product b reads A + b * batch_a and W + b * batch_w and writes C + b * batch_c (strides in
// elements).  Rows may be strided (lda, ldw, ldc), so heads that lie side by side in a row are products of one batch.
GK_EXPORT int gk_gemm_f32_batched(const void* A, int a_dtype, const float* W, void* C, int c_dtype, int batch, int M, int N,
                                  int K, long long lda, long long ldw, long long ldc, long long batch_a, long long batch_w,
                                  long long batch_c, void* stream) {
    GK_REQUIRE(GK_VALID_DTYPE(a_dtype) && GK_VALID_DTYPE(c_dtype), "gemm_f32_batched: bad dtype code");
    GK_REQUIRE(batch > 0 && batch <= 65535 && M >= 0 && N > 0 && K > 0, "gemm_f32_batched: bad sizes batch=%d M=%d N=%d K=%d",
               batch, M, N, K);
    GK_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32_batched: a leading dimension is shorter than its row");
    if (M == 0) return GK_OK;
    GK_REQUIRE((M + 127) / 128 <= 65535, "gemm_f32_batched: M=%d needs more than 65535 row tiles", M);
    dispatch_product(Product{A, W, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c}, a_dtype, c_dtype, batch, (cudaStream_t)stream);
    GK_CHECK_LAUNCH("gemm_f32_batched");
    return GK_OK;
}
