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
// Two kernels form the same chains:
//   tile   many tokens: BM x BN outputs a block, TM x TN chains a thread, operands through a ring of cp.async stages
//          in shared memory as they lie in memory (rows of BK), so that a thread reads four steps of k of a row with
//          one 16-byte load and the lanes' rows (BK + 4 floats apart) fall into different banks.
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
template <typename TA, typename TC, int MI, bool VEC>
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
void launch_few(const Product& p, int batch, cudaStream_t s) {
    launch_with_smem(gemm_f32_few_kernel<TA, TC, MI, VEC>, dim3((p.N + FEW_ROWS - 1) / FEW_ROWS, 1, batch), 32, few_smem<TA, MI>(), s, p);
}

template <typename TA, typename TC, bool VEC, int BM, int BN, int TM, int TN>
void launch_tile(const Product& p, int batch, cudaStream_t s) {
    const unsigned tiles = (unsigned)((p.M + BM - 1) / BM) * (unsigned)((p.N + BN - 1) / BN);
    launch_with_smem(gemm_f32_tile_kernel<TA, TC, BM, BN, TM, TN, VEC>, dim3(tiles, 1, batch), (BM / TM) * (BN / TN), tile_smem<TA, BM, BN>(), s, p);
}

template <typename TA, typename TC, bool VEC>
void launch_product(const Product& p, int batch, cudaStream_t s) {
    static const int sms = [] {
        int device = 0, n = 0;
        cudaGetDevice(&device);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
        return n > 0 ? n : 148;
    }();
    if (p.M <= 4) launch_few<TA, TC, VEC, 1>(p, batch, s);
    else if (p.M <= 8) launch_few<TA, TC, VEC, 2>(p, batch, s);
    else if (p.M <= FEW_TOKENS) launch_few<TA, TC, VEC, 4>(p, batch, s);
    // Tiles of 64 x 64 (8 x 4 chains a thread) where there are two for every SM, else of 32 x 32 (4 x 4 chains), which lose a
    // fifth to shared memory but spread.  Measured (us, 64 / 32; tokens x N x K): 2,048 x 4,096 x 4,096: 1,669 / 1,986;
    // 805 x 6,144 x 1,024: 275 / 307; 805 x 1,024 x 2,048 (208 tiles of 64): 127 / 114; 128 x 6,144 x 1,024 (192): 65 / 59;
    // 33 x 4,096 x 1,024 (64): 41 / 26.  Tiles of 128 x 128 lose at all of these (8 x 16 chains a thread: 1,955 at the first).
    // Before, with tiles of 128 x 128 alone: 3,247, 695, 424, 221 and 176.
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
