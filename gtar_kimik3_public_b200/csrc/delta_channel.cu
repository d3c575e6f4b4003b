// The gated delta rule with a decay per head and key channel (see delta_rule.cu) over many tokens at once, for bfloat16 steps:
// everything between the layer's input projections and its output projection in three kernels.
//
// With S0 the state before a chunk of 64 tokens and G_t = g_0 * .. * g_t per channel, the writes u_t solve
//     u_t = beta_t (v_t - (k_t G_t)^T S0 - sum_{j<t} (k_t . (k_j g_{j+1} .. g_t)) u_j)
// so with A_tj = beta_t sum_c k_tc k_jc g_{j+1,c} .. g_tc below the diagonal
//     u  = U - W S0                   U = (1 + A)^-1 diag(beta) V,   W = (1 + A)^-1 diag(beta) (K o G)
//     o  = (Q o G) S0 + P u           P_tj = sum_c q_tc k_jc g_{j+1,c} .. g_tc for j <= t
//     S1 = diag(G_last) S0 + (K o g_{t+1} .. g_last)^T u
// (the chunked form of the delta rule: S. Yang, B. Wang, Y. Zhang, Y. Shen, Y. Kim, "Parallelizing Linear Transformers with the
// Delta Rule over Sequence Length"; decays per channel by blocks inside a chunk: S. Yang, B. Wang, Y. Shen, R. Panda, Y. Kim, "Gated
// Linear Attention Transformers with Hardware-Efficient Training".)
//
// Products of decays are never divided: between two blocks of 16 tokens a term's decays are (from the later block's start to t) x
// (whole blocks between) x (from j to the end of j's block), all at most one; inside a block they are multiplied up token by token.
// So nothing overflows however strong the decays, and no logarithm is taken.
//
//   inner   a block per chunk and head: convolutions, SiLU, unit lengths, decays, beta; A, P, W, U and the scaled keys and queries
//   walk    a block per head and 8 value columns, the chunks in sequence: 128 x 8 numbers of state in the accumulators of eight warps
//   read    a block per chunk and head: o, RMS norm over a head, weight and gate
//
// Every matrix product takes 32-bit operands: each number is split into three bfloat16 numbers whose sum it is, six mma.sync a product
// (G. Henry, P. T. P. Tang, A. Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations");
// what is left out is at most 2^-24 of a product, 2^-27.5 root mean square.  The large parts are added up by 32-bit additions outside the
// tensor core, whose own sums are cut and not rounded (H. Ootomo, R. Yokota, "Recovering single precision accuracy from Tensor Cores while
// surpassing the FP32 theoretical peak performance"); of their products of 16 bits little is cut.  FFMA instead would be bound by what
// shared memory can deliver.
//
// Error of the states against 64 bits, relative, the kernels that go token by token / here (heads of 128; activations and decays are formed
// alike): one prompt of 2,048, 8 heads: 5.35e-7 / 5.15e-7; 1,024 + 500 + 77, 16 heads: 4.76e-7 / 4.62e-7; 192 after a state: 2.78e-7 / 2.70e-7;
// smaller in each of 20 drawn steps of 33 to 1,100 tokens, by 3 to 10%; of the bfloat16 read-outs 1.66e-3 both ways.  Where decays leave
// hardly anything of the token before (e^-2.7 a token) u has one rounding more: 1.20e-7 / 1.26e-7.  (Two TF32 numbers and three products, the same number
// of instructions: 137 us instead of 146 at the first, but 2.93e-7 at the third.)
// Measured (us, token by token / here): 2,048 tokens, 8 heads: 620 / 146; 1,024 + 500 + 77, 16 heads: 539 / 295; 512 + 300, 8 heads: 179 / 94.
// `inner` is bound by latency (some 50 us of the 146: its phases follow one another, two blocks an SM), `walk` by its two products and three
// barriers a chunk (1.5 us).

#include "common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int CHUNK = 64, SUB = 16, STRIP = 8;
constexpr int THREADS = 256;
constexpr int MAX_TAPS = 4;
constexpr int TILE16 = SUB * SUB;

// 32-bit numbers a chunk and head leaves in the workspace
template <int D>
struct Unit {
    static constexpr int W = 0;                    // left operand of the walk's first product, in fragments [4][D/8][32] of four
    static constexpr int K = W + CHUNK * D;        // left operand of its second product, in fragments [D/16][8][32]
    static constexpr int Q = K + CHUNK * D;        // left operand of the read-out, in fragments [4][D/8][32]
    static constexpr int P = Q + CHUNK * D;        // and within the chunk, in fragments [4][8][32]; what lies above the diagonal is not written
    static constexpr int G = P + CHUNK * CHUNK;    // decays over the whole chunk
    static constexpr int U = G + D;                // [64][dv]: U, then u
    static constexpr int S = U + CHUNK * D;        // [D][dv]: the state before the chunk
    static constexpr int SIZE = S + D * D;
};

// As in the kernels that go token by token
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two 32-bit numbers as three pairs of bfloat16 numbers: the nearest one, the nearest one to the rest, and what then remains, which is one.
// A NaN stays one; an infinity leaves NaN as its rest, so that it becomes NaN in every sum.
__device__ __forceinline__ uint32_t bf16_pair(float x, float y) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(y), "f"(x));
    return d;
}
__device__ __forceinline__ void split(float x, float y, uint32_t (&part)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        part[i] = bf16_pair(x, y);
        x -= __uint_as_float(part[i] << 16);
        y -= __uint_as_float(part[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// the same with nothing to add to
__device__ __forceinline__ void mma_alone(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// Left operand, two pieces of 16 x 8: of a piece lane 4 r + c holds rows r, r + 8 of two columns, in the order (r, first), (r + 8, first), (r,
// second), (r + 8, second).  Which two columns is free as long as the right operand's two rows are the same ones: 2c and 2c + 1 where an
// accumulator becomes an operand (no exchange between lanes), c and c + 4 where rows lie four banks apart.  The instruction's pairs of
// columns are one of each piece, so that where a thread has rows r and r + 8 of a right operand they are a pair.
struct Left {
    uint32_t part[3][4];
    __device__ __forceinline__ Left(const float4& a, const float4& b) {
        const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t p[3];
            split(x[i], y[i], p);
            part[0][i] = p[0], part[1][i] = p[1], part[2][i] = p[2];
        }
    }
};
struct Right {
    uint32_t part[3][2];
    __device__ __forceinline__ Right() {}
    // the two rows of the first piece, then those of the second
    __device__ __forceinline__ Right(float a0, float a1, float b0, float b1) {
        uint32_t p[3], q[3];
        split(a0, b0, p);
        split(a1, b1, q);
#pragma unroll
        for (int i = 0; i < 3; ++i) part[i][0] = p[i], part[i][1] = q[i];
    }
};
// CHAINS: of the small parts' products, which the tensor core adds up itself, one after another
template <int CHAINS>
struct SumOf {
    float acc[4], low[CHAINS][4];
    __device__ __forceinline__ SumOf() {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc[i] = 0.f;
#pragma unroll
            for (int j = 0; j < CHAINS; ++j) low[j][i] = 0.f;
        }
    }
    __device__ __forceinline__ void add(const Left& a, const Right& b) {
        float c[4];
        mma_alone(c, a.part[0], b.part[0]);
        mma(low[0], a.part[0], b.part[1]);
        mma(low[CHAINS - 1], a.part[1], b.part[0]);
        mma(low[0], a.part[0], b.part[2]);
        mma(low[CHAINS - 1], a.part[2], b.part[0]);
        mma(low[0], a.part[1], b.part[1]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] += c[i];
    }
    __device__ __forceinline__ float at(int i) const { return acc[i] + (CHAINS > 1 ? low[0][i] + low[CHAINS - 1][i] : low[0][i]); }
};
typedef SumOf<1> Sum;

// entry (t, j) of a 16 x 16 block in shared memory: pairs of columns turned so that eight rows' pairs fall into different banks
__device__ __forceinline__ int at16(int t, int j) { return t * SUB + 2 * ((j >> 1) ^ (((t >> 1) & 1) << 2)) + (j & 1); }

// N (4 or 2) bfloat16 numbers as they lie in memory
template <int N>
struct Raw {
    uint32_t pairs[N / 2];
    __device__ __forceinline__ void numbers(float (&x)[N]) const {
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pairs[i]));
            x[2 * i] = f.x, x[2 * i + 1] = f.y;
        }
    }
};
template <>
struct __align__(8) Raw<4> {
    uint32_t pairs[2];
    __device__ __forceinline__ void numbers(float (&x)[4]) const {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pairs[i]));
            x[2 * i] = f.x, x[2 * i + 1] = f.y;
        }
    }
};

template <int N>
__device__ __forceinline__ void load_row(const float* src, float (&x)[N]) {
    if constexpr (N == 4) {
        const float4 a = *reinterpret_cast<const float4*>(src);
        x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w;
    } else {
        const float2 a = *reinterpret_cast<const float2*>(src);
        x[0] = a.x, x[1] = a.y;
    }
}
template <int N>
__device__ __forceinline__ void store_row(float* dst, const float (&x)[N]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
    else *reinterpret_cast<float2*>(dst) = make_float2(x[0], x[1]);
}

struct Inputs {
    const bf16* proj;        // [T, ld]: q | k | v | b
    const float* low;        // [T, ld_low]: decays | gate
    const float* conv_w;     // [channels, taps]
    float* conv_state;       // [slots, taps - 1, channels]
    const float *a_log, *dt_bias, *norm;
    const int *cu_q, *slots;
    long long ld, ld_low;
    int n_heads, n_kv, dv, taps, chunk0, wave;
};

// Eight consecutive tokens' convolution and SiLU of N neighbouring channels from column c on; s0: the first token's place in the
// step, `live` of the eight are there.  Inputs before the step come from the sequence's convolution state.
template <int N, bool USUAL>
__device__ __forceinline__ void conv_eight(const Inputs& in, int tok, int s0, int live, size_t slot, int c, int channels, float (&y)[8][N]) {
    const int taps = USUAL ? MAX_TAPS : in.taps;
    constexpr int ROWS = 8 + MAX_TAPS - 1;
    float w[MAX_TAPS][N], x[ROWS][N];
    Raw<N> raw[ROWS];  // all of them asked for before the first is looked at
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int back = i - (MAX_TAPS - 1);
        const bool there = back < live && -back < taps && s0 + back >= 0;
        raw[i] = there ? *reinterpret_cast<const Raw<N>*>(in.proj + (long long)(tok + back) * in.ld + c) : Raw<N>{};
    }
    if (USUAL) {
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const float4 four = *reinterpret_cast<const float4*>(in.conv_w + (size_t)(c + e) * MAX_TAPS);
            w[3][e] = four.x, w[2][e] = four.y, w[1][e] = four.z, w[0][e] = four.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < MAX_TAPS; ++j)
#pragma unroll
            for (int e = 0; e < N; ++e) w[j][e] = j < taps ? in.conv_w[(size_t)(c + e) * taps + taps - 1 - j] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i) raw[i].numbers(x[i]);
    if (s0 < taps - 1 && live > 0) {  // the step's first tokens
#pragma unroll
        for (int i = 0; i < MAX_TAPS - 1; ++i) {
            const int s = s0 + i - (MAX_TAPS - 1);
            if (s < 0 && taps - 1 + s >= 0) load_row<N>(in.conv_state + (slot * (taps - 1) + (taps - 1 + s)) * channels + c, x[i]);
        }
    }
#pragma unroll
    for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int e = 0; e < N; ++e) {
            float z = 0.f;
#pragma unroll
            for (int j = 0; j < MAX_TAPS; ++j)
                if (j < taps) z = fmaf(w[j][e], x[t + MAX_TAPS - 1 - j][e], z);
            y[t][e] = t < live ? silu_f(z) : 0.f;
        }
}

template <int D>
struct InnerSmem {
    static constexpr int LD = D + 4;  // rows four banks apart
    float k[CHUNK][LD], g[CHUNK][LD], q[CHUNK][LD];
    float blk[10][TILE16];            // (1 + A)^-1 - 1 of the four blocks on the diagonal, then the six of A below it
    float total[5][D];                // decays over a block, and ones
    float beta[CHUNK];
};

// USUAL: four taps, values as wide as keys and tap weights on 16 bytes, known when the kernel is built: without branches on them a thread's
// loads are asked for together.
template <int D, bool USUAL>
__global__ void __launch_bounds__(THREADS, 2) channel_inner_kernel(Inputs in, float* __restrict__ work) {
    constexpr int N = D / 32, KS = D / 8, LD = InnerSmem<D>::LD;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    InnerSmem<D>& sm = *reinterpret_cast<InnerSmem<D>*>(smem_raw);
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, hk = head / (in.n_heads / in.n_kv), dv = USUAL ? D : in.dv;
    const int t0 = in.cu_q[seq], len = in.cu_q[seq + 1] - t0;
    const int first = (in.chunk0 + blockIdx.x) * CHUNK;
    if (first >= len) return;
    const int n = min(CHUNK, len - first), tok0 = t0 + first;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c2 = lane & 3;
    const int qk = in.n_kv * D, channels = 2 * qk + in.n_heads * dv;
    const size_t slot = in.slots[seq];
    float* mine = work + (((size_t)seq * in.wave + blockIdx.x) * in.n_heads + head) * Unit<D>::SIZE;

    // ---- queries, keys, values, decays, beta: a warp has eight tokens, a lane N channels.  (Loops stay loops wherever registers allow:
    //      the kernel runs through its code once, and code that is not in the instruction cache yet costs more than the branches.)
    for (int i = tid; i < CHUNK * D / 4; i += THREADS) {  // what the decays are made of, on its way meanwhile
        const int t = i / (D / 4), c = i % (D / 4) * 4;
        if (t < n) cp_async_16(&sm.g[t][c], in.low + (long long)(tok0 + t) * in.ld_low + head * D + c);
    }
    cp_async_commit();
    {
        const int w0 = warp * 8, live = min(8, n - w0), at = lane * N;
#pragma unroll 1
        for (int part = 0; part < 3; ++part) {
            const bool values = part == 2;
            if (values && at >= dv) break;
            float y[8][N];
            conv_eight<N, USUAL>(in, tok0 + w0, first + w0, live, slot, (values ? 2 * qk + head * dv : part * qk + hk * D) + at, channels, y);
            if (values) {  // for now where their solutions will be
#pragma unroll
                for (int t = 0; t < 8; ++t) store_row<N>(mine + Unit<D>::U + (w0 + t) * dv + at, y[t]);
                break;
            }
            float* to = (part == 0 ? &sm.q[w0][0] : &sm.k[w0][0]) + at;
            float squares = 0.f;  // of token `lane`
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                float ss = 0.f;
#pragma unroll
                for (int e = 0; e < N; ++e) ss = fmaf(y[t][e], y[t][e], ss);
                ss = warp_sum(ss);
                if (lane == t) squares = ss;
            }
            float unit = 1.f / sqrtf(squares + 1e-6f);
            if (part == 0) unit *= 1.f / sqrtf((float)D);
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float mine_t = __shfl_sync(0xffffffffu, unit, t);
#pragma unroll
                for (int e = 0; e < N; ++e) y[t][e] *= mine_t;
                store_row<N>(to + t * LD, y[t]);
            }
        }
        if (tid < D) sm.total[4][tid] = 1.f;
        if (tid < CHUNK) sm.beta[tid] = tid < n ? sigmoid_f(to_float(in.proj[(long long)(tok0 + tid) * in.ld + channels + head])) : 0.f;
    }
    cp_async_wait<0>();
    __syncthreads();
    {
        const float rate = -expf(in.a_log[head]);
        const int c = tid % D;
        const float bias = in.dt_bias[head * D + c];
#pragma unroll 4
        for (int t = tid / D; t < CHUNK; t += THREADS / D) sm.g[t][c] = t < n ? expf(rate * softplus_f(sm.g[t][c] + bias)) : 1.f;
    }
    __syncthreads();

    // ---- blocks on the diagonal, token by token: a warp has every other key of a block, decayed on from token to token
    {
        const int b = warp >> 1, odd = warp & 1, at = lane * N;
        float held[8][N];
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
            for (int e = 0; e < N; ++e) held[m][e] = 0.f;
        const int value = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
        const int j = 2 * (value & 7) + odd;
#pragma unroll 2
        for (int t = 0; t < SUB; ++t) {
            float g[N], k[N], q[N], v[16];
            load_row<N>(&sm.g[b * SUB + t][at], g);
            load_row<N>(&sm.k[b * SUB + t][at], k);
            load_row<N>(&sm.q[b * SUB + t][at], q);
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                v[m] = v[8 + m] = 0.f;
                const bool meets = 2 * m + odd == t;  // zero until then
#pragma unroll
                for (int e = 0; e < N; ++e) {
                    held[m][e] = meets ? k[e] : held[m][e] * g[e];
                    v[m] = fmaf(k[e], held[m][e], v[m]);
                    v[8 + m] = fmaf(q[e], held[m][e], v[8 + m]);
                }
            }
            // sixteen sums over the lanes: a lane keeps half of its values at every exchange
#pragma unroll
            for (int o = 16, half = 8; half >= 1; o >>= 1, half >>= 1) {
                const bool upper = (lane & o) != 0;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const float send = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
            if ((lane & 1) == 0) {
                if (value < 8) sm.blk[b][at16(t, j)] = j < t ? sm.beta[b * SUB + t] * v[0] : 0.f;
                else mine[Unit<D>::P + ((b * 8 + 2 * b + (j >> 3)) * 32 + (t & 7) * 4 + ((j & 7) >> 1)) * 4 + (j & 1) * 2 + (t >> 3)] = v[0];
            }
        }
    }
    __syncthreads();
    if (warp < 4) {  // (1 + A)^-1 of a block, a column a lane
        float x[SUB];
        float* A = sm.blk[warp];
#pragma unroll
        for (int i = 0; i < SUB; ++i) {
            float p[2] = {0.f, 0.f};
#pragma unroll
            for (int j = 0; j < i; j += 2) {
                const float2 a = *reinterpret_cast<const float2*>(A + at16(i, j));
                p[0] = fmaf(a.x, x[j], p[0]);
                if (j + 1 < i) p[1] = fmaf(a.y, x[j + 1], p[1]);
            }
            x[i] = (i == (lane & 15) ? 1.f : 0.f) - (p[0] + p[1]);
        }
        __syncwarp();
        if (lane < SUB)
#pragma unroll
            for (int i = 0; i < SUB; ++i) A[at16(i, lane)] = i == lane ? 0.f : x[i];  // the ones on the diagonal are added where it is used
    } else {  // decays from a block's start into keys and queries, and keys with the decays to the block's end in the place of the decays
        for (int item = tid - 128; item < 4 * D; item += 128) {
            const int c = item % D, b = item / D;
            float g[SUB], k[SUB], run = 1.f;
#pragma unroll
            for (int t = 0; t < SUB; ++t) {
                g[t] = sm.g[b * SUB + t][c];
                k[t] = sm.k[b * SUB + t][c];
            }
#pragma unroll
            for (int t = 0; t < SUB; ++t) {
                run *= g[t];
                sm.k[b * SUB + t][c] = k[t] * run;
                sm.q[b * SUB + t][c] *= run;
            }
            sm.total[b][c] = run;
            run = 1.f;
#pragma unroll
            for (int t = SUB - 1; t >= 0; --t) {
                sm.g[b * SUB + t][c] = k[t] * run;
                run *= g[t];
            }
        }
    }
    __syncthreads();

    // ---- blocks below the diagonal: 24 products of 16 x 8 (six blocks, two halves, keys and queries), three a warp
#pragma unroll 1
    for (int task = warp; task < 24; task += 8) {
        const bool queries = task >= 12;
        const int pair = (task % 12) >> 1, nt = task & 1;
        const int I = pair == 0 ? 1 : pair < 3 ? 2 : 3, J = pair - I * (I - 1) / 2;
        const float* a = (queries ? &sm.q[I * SUB + r][0] : &sm.k[I * SUB + r][0]) + c2;
        const float* b = &sm.g[J * SUB + nt * 8 + r][0] + c2;
        const float *f1 = sm.total[I - J > 1 ? J + 1 : 4] + c2, *f2 = sm.total[I - J > 2 ? J + 2 : 4] + c2;  // the blocks between
        SumOf<2> s;
        const auto left = [&](int c) { return make_float4(a[c], a[c + 8 * LD], a[c + 4], a[c + 8 * LD + 4]); };
        const auto right = [&](int c) { return b[c] * f1[c] * f2[c]; };
#pragma unroll 2
        for (int c = 0; c < D; c += 16) s.add(Left(left(c), left(c + 8)), Right(right(c), right(c + 4), right(c + 8), right(c + 12)));
        if (queries) {
            reinterpret_cast<float4*>(mine + Unit<D>::P)[(I * 8 + J * 2 + nt) * 32 + lane] = make_float4(s.at(0), s.at(2), s.at(1), s.at(3));
        } else {
            float* to = sm.blk[4 + pair];
            const float b0 = sm.beta[I * SUB + r], b1 = sm.beta[I * SUB + r + 8];
            const int j = nt * 8 + 2 * c2;
            *reinterpret_cast<float2*>(to + at16(r, j)) = make_float2(b0 * s.at(0), b0 * s.at(1));
            *reinterpret_cast<float2*>(to + at16(r + 8, j)) = make_float2(b1 * s.at(2), b1 * s.at(3));
        }
    }
    // ---- queries and keys with their decays, in the order of the operands they become
    for (int i = warp; i < 4 * KS; i += 8) {
        const int I = i / KS, c = (i % KS) * 8 + 2 * c2;
        float2 x = *reinterpret_cast<const float2*>(&sm.q[I * SUB + r][c]), y = *reinterpret_cast<const float2*>(&sm.q[I * SUB + r + 8][c]);
        for (int b = 0; b < I; ++b) {
            const float2 f = *reinterpret_cast<const float2*>(&sm.total[b][c]);
            x.x *= f.x, x.y *= f.y, y.x *= f.x, y.y *= f.y;
        }
        reinterpret_cast<float4*>(mine + Unit<D>::Q)[i * 32 + lane] = make_float4(x.x, y.x, x.y, y.y);
    }
    for (int i = warp; i < D / 16 * 8; i += 8) {
        const int c = (i >> 3) * 16 + r, t = (i & 7) * 8 + 2 * c2;
        float x[4] = {sm.g[t][c], sm.g[t][c + 8], sm.g[t + 1][c], sm.g[t + 1][c + 8]};
        for (int b = (t >> 4) + 1; b < 4; ++b) {
            const float f0 = sm.total[b][c], f1 = sm.total[b][c + 8];
            x[0] *= f0, x[1] *= f1, x[2] *= f0, x[3] *= f1;
        }
        reinterpret_cast<float4*>(mine + Unit<D>::K)[i * 32 + lane] = make_float4(x[0], x[1], x[2], x[3]);
    }
    if (tid < D) mine[Unit<D>::G + tid] = sm.total[0][tid] * sm.total[1][tid] * sm.total[2][tid] * sm.total[3][tid];
    __syncthreads();

    // ---- (1 + A)^-1 of beta K G and of beta V, block after block: a warp has 16 columns of each, which meet no others.  The transposed
    //      system: an accumulator is the next product's left operand as it stands
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
        if (warp * 16 >= (part == 0 ? D : dv)) continue;
        const int c = warp * 16 + r;
        const float* src = part == 0 ? &sm.k[0][0] : mine + Unit<D>::U;
        const int ld_src = part == 0 ? LD : dv;
        float pre[2] = {1.f, 1.f}, x[8][4];
        const auto turned = [](const float(&a)[4], const float(&b)[4]) { return Left(make_float4(a[0], a[2], a[1], a[3]), make_float4(b[0], b[2], b[1], b[3])); };
        const auto block = [&](int which, int nt) {
            const float2 a = *reinterpret_cast<const float2*>(&sm.blk[which][at16(nt * 8 + r, 2 * c2)]);
            const float2 b = *reinterpret_cast<const float2*>(&sm.blk[which][at16(nt * 8 + r, 8 + 2 * c2)]);
            return Right(a.x, a.y, b.x, b.y);
        };
#pragma unroll
        for (int I = 0; I < 4; ++I) {
            float rest[2][4];
            {
                Sum s[2];
#pragma unroll
                for (int J = 0; J < I; ++J) {
                    const Left a = turned(x[2 * J], x[2 * J + 1]);
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt) s[nt].add(a, block(4 + I * (I - 1) / 2 + J, nt));
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = I * SUB + nt * 8 + 2 * c2 + (e & 1);
                        rest[nt][e] = src[t * ld_src + c + 8 * (e >> 1)] * pre[e >> 1] * sm.beta[t] - s[nt].at(e);
                    }
            }
            // what is no number from a token on (a zero above the block's diagonal times it would be none for the tokens in front)
            int from[2] = {SUB, SUB};
            bool numbers = true;
#pragma unroll
            for (int i = 0; i < 8; ++i) numbers = numbers && finite(rest[i >> 2][i & 3]);
            const bool broken = __any_sync(0xffffffffu, !numbers);
            if (broken) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int i = 3; i >= 0; --i) {
                        float& x_t = rest[i >> 1][2 * h + (i & 1)];
                        if (!finite(x_t)) from[h] = (i >> 1) * 8 + 2 * c2 + (i & 1), x_t = 0.f;
                    }
                    from[h] = min(from[h], __shfl_xor_sync(0xffffffffu, from[h], 1));
                    from[h] = min(from[h], __shfl_xor_sync(0xffffffffu, from[h], 2));
                }
            }
            Sum s[2];
            const Left a = turned(rest[0], rest[1]);
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                s[nt].add(a, block(I, nt));
#pragma unroll
                for (int e = 0; e < 4; ++e) x[2 * I + nt][e] = rest[nt][e] + s[nt].at(e);
            }
            if (broken)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (nt * 8 + 2 * c2 + (e & 1) >= from[e >> 1]) x[2 * I + nt][e] = NAN;
            if (part == 0) {
                pre[0] *= sm.total[I][c];
                pre[1] *= sm.total[I][c + 8];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = i * 8 + 2 * c2 + (e & 1), col = c + 8 * (e >> 1);
                if (part == 0) sm.k[t][col] = x[i][e];  // nobody else reads these columns
                else mine[Unit<D>::U + t * dv + col] = x[i][e];
            }
    }
    __syncthreads();
    for (int i = warp; i < 4 * KS; i += 8) {
        const int t = (i / KS) * SUB + r, c = (i % KS) * 8 + 2 * c2;
        const float2 x = *reinterpret_cast<const float2*>(&sm.k[t][c]), y = *reinterpret_cast<const float2*>(&sm.k[t + 8][c]);
        reinterpret_cast<float4*>(mine + Unit<D>::W)[i * 32 + lane] = make_float4(x.x, y.x, x.y, y.y);
    }
}

// Sixteen rows of a column whose words are pairs already, the three parts `apart` bytes from one another.
__device__ __forceinline__ Right right_at(const uint32_t* words, size_t apart) {
    Right b;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint2 two = *reinterpret_cast<const uint2*>(words + p * apart / 4);
        b.part[p][0] = two.x, b.part[p][1] = two.y;
    }
    return b;
}

// RING: tiles that a warp's pieces of are in flight or in use: six where a block has an SM to itself, three where two share one
template <int D, int RING>
struct WalkSmem {
    float4 ring[RING][8][8][32];             // a warp's pieces of the tiles: a lane reads back what it copied itself
    // rows of value columns, eight banks apart, in three parts: a word is channels (tokens) r and r + 8 of sixteen
    uint32_t state[3][STRIP][D / 2 + 8];
    uint32_t u[3][STRIP][CHUNK / 2 + 8];
    float4 part[4][32];                      // the second half of the first product's sums
};

template <int D, int RING>
__global__ void __launch_bounds__(THREADS, RING == 3 ? 2 : 1) channel_walk_kernel(Inputs in, float* __restrict__ work, float* __restrict__ state) {
    constexpr int HALF = D / 16;  // steps of eight channels that a warp has of the first product
    extern __shared__ __align__(128) unsigned char smem_raw[];
    WalkSmem<D, RING>& sm = *reinterpret_cast<WalkSmem<D, RING>*>(smem_raw);
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, v0 = blockIdx.x * STRIP, dv = in.dv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c2 = lane & 3;
    const int t0 = in.cu_q[seq], len = in.cu_q[seq + 1] - t0;
    const size_t slot = in.slots[seq];
    if (in.chunk0 == 0 && in.taps > 1 && len > 0) {
        // the convolution state moves on by the step's inputs: a channel a thread, rows upward, so every row is read before it is written
        const int rows = in.taps - 1, channels = 2 * in.n_kv * D + in.n_heads * dv;
        for (int c = (blockIdx.y * gridDim.x + blockIdx.x) * THREADS + threadIdx.x; c < channels; c += gridDim.x * gridDim.y * THREADS) {
            float* mine = in.conv_state + slot * rows * channels + c;
            for (int i = 0; i < rows; ++i) {
                const int at = len - rows + i;
                mine[(size_t)i * channels] = at >= 0 ? to_float(in.proj[(long long)(t0 + at) * in.ld + c]) : mine[(size_t)(i + len) * channels];
            }
        }
    }
    const int here = min(in.wave, (len + CHUNK - 1) / CHUNK - in.chunk0);
    if (here <= 0) return;
    const size_t step = (size_t)in.n_heads * Unit<D>::SIZE;
    float* unit = work + ((size_t)seq * in.wave * in.n_heads + head) * Unit<D>::SIZE;
    const bool owns = warp < D / 16;       // of the state: channels 16 warp + r and + 8, columns 2 c2 and + 1
    const int mt = warp & 3, kh = warp >> 2;
    auto issue = [&](int i) {
        if (i < 2 * here) {
            const float* u = unit + (i >> 1) * step;
            if ((i & 1) == 0) {
                const float4* src = reinterpret_cast<const float4*>(u + Unit<D>::W) + (mt * (D / 8) + kh * HALF) * 32 + lane;
#pragma unroll
                for (int ks = 0; ks < HALF; ++ks) cp_async_16(&sm.ring[i % RING][warp][ks][lane], src + ks * 32);
            } else if (owns) {
                const float4* src = reinterpret_cast<const float4*>(u + Unit<D>::K) + warp * 8 * 32 + lane;
#pragma unroll
                for (int ks = 0; ks < 8; ++ks) cp_async_16(&sm.ring[i % RING][warp][ks][lane], src + ks * 32);
            }
        }
        cp_async_commit();
    };
    for (int i = 0; i < RING - 1; ++i) issue(i);
    float* saved = state + (slot * in.n_heads + head) * (size_t)D * dv + v0 + 2 * c2;
    float S[4] = {0.f, 0.f, 0.f, 0.f};
    const int ch = warp * 16 + r;
    if (owns) {
        const float2 a = *reinterpret_cast<const float2*>(saved + (size_t)ch * dv), b = *reinterpret_cast<const float2*>(saved + (size_t)(ch + 8) * dv);
        S[0] = a.x, S[1] = a.y, S[2] = b.x, S[3] = b.y;
    }
    const int tok = mt * 16 + r;
    float2 next_u[2] = {};
    float next_g[2] = {};
    auto fetch = [&](int i) {  // what the chunk needs beside its tiles
        if (i >= here) return;
        const float* u = unit + i * step;
        if (kh == 0) {
            next_u[0] = *reinterpret_cast<const float2*>(u + Unit<D>::U + tok * dv + v0 + 2 * c2);
            next_u[1] = *reinterpret_cast<const float2*>(u + Unit<D>::U + (tok + 8) * dv + v0 + 2 * c2);
        }
        if (owns) {
            next_g[0] = u[Unit<D>::G + ch];
            next_g[1] = u[Unit<D>::G + ch + 8];
        }
    };
    fetch(0);
    for (int i = 0; i < here; ++i) {
        float* mine = unit + i * step;
        if (owns) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t part[3];
                split(S[e], S[2 + e], part);
#pragma unroll
                for (int h = 0; h < 3; ++h) sm.state[h][2 * c2 + e][warp * 8 + r] = part[h];
            }
            *reinterpret_cast<float2*>(mine + Unit<D>::S + ch * dv + v0 + 2 * c2) = make_float2(S[0], S[1]);
            *reinterpret_cast<float2*>(mine + Unit<D>::S + (ch + 8) * dv + v0 + 2 * c2) = make_float2(S[2], S[3]);
        }
        const float2 u0 = next_u[0], u1 = next_u[1];
        const float g0 = next_g[0], g1 = next_g[1];
        fetch(i + 1);
        issue(2 * i + RING - 1);
        cp_async_wait<RING - 1>();
        __syncthreads();  // the state before the chunk is there
        {
            SumOf<2> s;
#pragma unroll
            for (int ks = 0; ks < HALF; ks += 2)
                s.add(Left(sm.ring[(2 * i) % RING][warp][ks][lane], sm.ring[(2 * i) % RING][warp][ks + 1][lane]), right_at(&sm.state[0][r][(kh * HALF + ks) * 4 + 2 * c2], sizeof(sm.state[0])));
            // the two halves meet: 64 threads a barrier
            if (kh == 1) {
                sm.part[mt][lane] = make_float4(s.at(0), s.at(1), s.at(2), s.at(3));
                asm volatile("bar.arrive %0, 64;" ::"r"(1 + mt) : "memory");
            } else {
                asm volatile("bar.sync %0, 64;" ::"r"(1 + mt) : "memory");
                const float4 p = sm.part[mt][lane];
                const float u[4] = {u0.x - (s.at(0) + p.x), u0.y - (s.at(1) + p.y), u1.x - (s.at(2) + p.z), u1.y - (s.at(3) + p.w)};
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    uint32_t part[3];
                    split(u[e], u[2 + e], part);
#pragma unroll
                    for (int h = 0; h < 3; ++h) sm.u[h][2 * c2 + e][mt * 8 + r] = part[h];
                }
                *reinterpret_cast<float2*>(mine + Unit<D>::U + tok * dv + v0 + 2 * c2) = make_float2(u[0], u[1]);
                *reinterpret_cast<float2*>(mine + Unit<D>::U + (tok + 8) * dv + v0 + 2 * c2) = make_float2(u[2], u[3]);
            }
        }
        issue(2 * i + RING);
        cp_async_wait<RING - 1>();
        __syncthreads();  // u is there, and nobody reads the state before the chunk any more
        if (owns) {
            SumOf<2> s;
#pragma unroll
            for (int ks = 0; ks < 8; ks += 2)
                s.add(Left(sm.ring[(2 * i + 1) % RING][warp][ks][lane], sm.ring[(2 * i + 1) % RING][warp][ks + 1][lane]), right_at(&sm.u[0][r][ks * 4 + 2 * c2], sizeof(sm.u[0])));
            S[0] = fmaf(S[0], g0, s.at(0));
            S[1] = fmaf(S[1], g0, s.at(1));
            S[2] = fmaf(S[2], g1, s.at(2));
            S[3] = fmaf(S[3], g1, s.at(3));
        }
    }
    cp_async_wait<0>();
    if (owns) {
        *reinterpret_cast<float2*>(saved + (size_t)ch * dv) = make_float2(S[0], S[1]);
        *reinterpret_cast<float2*>(saved + (size_t)(ch + 8) * dv) = make_float2(S[2], S[3]);
    }
}

template <int D>
struct ReadSmem {
    static constexpr int LD = 132;  // two rows are eight banks apart
    float state[D][LD], u[CHUNK][LD];
    float squares[2][CHUNK];
};

template <int D, bool USUAL>
__global__ void __launch_bounds__(THREADS, 2) channel_read_kernel(Inputs in, const float* __restrict__ work, bf16* __restrict__ out, float eps) {
    constexpr int LD = ReadSmem<D>::LD;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    ReadSmem<D>& sm = *reinterpret_cast<ReadSmem<D>*>(smem_raw);
    pdl_launch_dependents();
    pdl_wait();
    const int head = blockIdx.y, seq = blockIdx.z, dv = USUAL ? D : in.dv;
    const int t0 = in.cu_q[seq], len = in.cu_q[seq + 1] - t0;
    const int first = (in.chunk0 + blockIdx.x) * CHUNK;
    if (first >= len) return;
    const int n = min(CHUNK, len - first), tok0 = t0 + first;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, c2 = lane & 3, mt = warp & 3, nh = warp >> 2;
    const float* mine = work + (((size_t)seq * in.wave + blockIdx.x) * in.n_heads + head) * Unit<D>::SIZE;
    const int pieces = dv / 4;
    for (int i = threadIdx.x; i < D * pieces; i += THREADS) cp_async_16(&sm.state[i / pieces][(i % pieces) * 4], mine + Unit<D>::S + i * 4);
    for (int i = threadIdx.x; i < CHUNK * pieces; i += THREADS) cp_async_16(&sm.u[i / pieces][(i % pieces) * 4], mine + Unit<D>::U + i * 4);
    cp_async_commit();
    const int tiles = dv / 16, v0 = nh * (dv / 2);
    Sum s[8];
    cp_async_wait<0>();
    __syncthreads();
    // last: the sixteen tokens on the diagonal, where a zero times what is no number would be none for the tokens in front of it
    bool numbers = true;
    auto product = [&](const float4* left, int steps, const float(*right)[LD], bool last) {
        float4 ahead[4];  // from L2, four steps ahead
#pragma unroll
        for (int i = 0; i < 4; ++i) ahead[i] = i < steps ? left[i * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int k4 = 0; k4 < steps; k4 += 4)
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const int ks = k4 + i;
                if (ks >= steps) break;
                const Left a(ahead[i], ahead[i + 1]);
                if (ks + 4 < steps) ahead[i] = left[(ks + 4) * 32 + lane], ahead[i + 1] = left[(ks + 5) * 32 + lane];
                const float *b0 = &right[ks * 8 + 2 * c2][v0 + r], *b1 = b0 + LD;
#pragma unroll
                for (int nt = 0; nt < 8; ++nt)
                    if (nt < tiles) {
                        float x[4] = {b0[nt * 8], b1[nt * 8], b0[nt * 8 + 8 * LD], b1[nt * 8 + 8 * LD]};
                        if (last)
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const bool number = finite(x[e]);
                                numbers = numbers && number;
                                x[e] = number ? x[e] : 0.f;
                            }
                        s[nt].add(a, Right(x[0], x[1], x[2], x[3]));
                    }
            }
    };
    product(reinterpret_cast<const float4*>(mine + Unit<D>::Q) + mt * (D / 8) * 32, D / 8, sm.state, false);
    const float4* within = reinterpret_cast<const float4*>(mine + Unit<D>::P) + mt * 8 * 32;
    product(within, 2 * mt, sm.u, false);
    product(within + 2 * mt * 32, 2, sm.u + mt * SUB, true);
    if (__any_sync(0xffffffffu, !numbers)) {
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (nt < tiles)
#pragma unroll 1
                    for (int j = 0; j <= r + 8 * (e >> 1); ++j)
                        if (!finite(sm.u[mt * SUB + j][v0 + nt * 8 + 2 * c2 + (e & 1)])) s[nt].acc[e] = NAN;
    }
    float ss[2] = {0.f, 0.f};
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s[nt].acc[e] = nt < tiles ? s[nt].at(e) : 0.f;
            ss[e >> 1] = fmaf(s[nt].acc[e], s[nt].acc[e], ss[e >> 1]);
        }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        ss[h] += __shfl_xor_sync(0xffffffffu, ss[h], 1);
        ss[h] += __shfl_xor_sync(0xffffffffu, ss[h], 2);
        if (c2 == 0) sm.squares[nh][mt * 16 + r + 8 * h] = ss[h];
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int t = mt * 16 + r + 8 * h;
        if (t >= n) continue;
        const float unit = 1.f / sqrtf((sm.squares[0][t] + sm.squares[1][t]) / (float)dv + eps);
        const float* gate = in.low + (long long)(tok0 + t) * in.ld_low + (long long)in.n_heads * D + head * dv + v0 + 2 * c2;
        bf16* to = out + ((size_t)(tok0 + t) * in.n_heads + head) * dv + v0 + 2 * c2;
        float2 z[8], w[8];  // all asked for before the first is used
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
            if (nt < tiles) {
                z[nt] = *reinterpret_cast<const float2*>(gate + nt * 8);
                w[nt] = *reinterpret_cast<const float2*>(in.norm + v0 + nt * 8 + 2 * c2);
            }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
            if (nt < tiles) {
                const float x = s[nt].acc[2 * h] * unit * w[nt].x * sigmoid_f(z[nt].x), y = s[nt].acc[2 * h + 1] * unit * w[nt].y * sigmoid_f(z[nt].y);
                *reinterpret_cast<__nv_bfloat162*>(to + nt * 8) = __floats2bfloat162_rn(x, y);
            }
    }
}

}  // namespace

static bool channel_fits(int d, int dv, int taps) { return (d == 64 || d == 128) && dv > 0 && dv % 16 == 0 && dv <= d && taps >= 1 && taps <= MAX_TAPS; }
GK_EXPORT int gk_delta_channel_fits(int d, int dv, int taps) { return channel_fits(d, dv, taps); }
// 32-bit numbers of workspace per sequence, chunk of a wave and head
GK_EXPORT int gk_delta_channel_work(int d) { return d == 64 ? Unit<64>::SIZE : Unit<128>::SIZE; }

// proj [T, ld] bfloat16: q (G d) | k (G d) | v (H dv) | b (H) | ..; low [T, ld_low] 32-bit: a (H d) | gate (H dv); out [T, H dv] bfloat16;
// state [slots, H, d, dv] and conv_state [slots, taps - 1, channels] are moved on by the step's tokens.  max_len bounds the sequences'
// token counts; `wave` chunks of every sequence are in flight at a time.
GK_EXPORT int gk_delta_channel(const void* proj, long long ld, const float* low, long long ld_low, const float* conv_w, float* conv_state,
                               const float* a_log, const float* dt_bias, const float* norm, float eps, float* state, float* work, void* out,
                               const int* cu_q, const int* slots, int n_seqs, int n_heads, int n_kv, int d, int dv, int taps, int max_len,
                               int wave, void* stream) {
    GK_REQUIRE(n_heads > 0 && n_heads <= 65535 && n_kv > 0 && n_heads % n_kv == 0 && n_seqs >= 0 && n_seqs <= 65535, "delta_channel: bad counts");
    GK_REQUIRE(channel_fits(d, dv, taps), "delta_channel: heads of %d / %d with %d taps do not fit", d, dv, taps);
    GK_REQUIRE(taps == 1 || conv_state != nullptr, "delta_channel: a convolution of several taps needs its state");
    GK_REQUIRE(max_len >= 0 && wave > 0 && work != nullptr, "delta_channel: bad sizes");
    GK_REQUIRE(ld % 8 == 0 && ld_low % 4 == 0, "delta_channel: rows must start on 16 bytes");
    GK_REQUIRE((((uintptr_t)proj | (uintptr_t)low | (uintptr_t)work | (uintptr_t)state | (uintptr_t)conv_state | (uintptr_t)dt_bias | (uintptr_t)norm |
                 (uintptr_t)out) & 15) == 0, "delta_channel: tensors must start on 16 bytes");
    if (n_seqs == 0 || max_len == 0) return GK_OK;
    static int sms = 0;
    if (sms == 0) {
#define GK_ATTR(KERNEL, BYTES)                                                                                  \
    if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(BYTES)) != cudaSuccess) \
        return gk_fail(GK_CUDA_ERROR, "delta_channel: shared memory")
#define GK_ATTRS(D)                                                  \
    GK_ATTR((channel_inner_kernel<D, false>), sizeof(InnerSmem<D>)); \
    GK_ATTR((channel_inner_kernel<D, true>), sizeof(InnerSmem<D>));  \
    GK_ATTR((channel_walk_kernel<D, 3>), sizeof(WalkSmem<D, 3>));    \
    GK_ATTR((channel_walk_kernel<D, 6>), sizeof(WalkSmem<D, 6>));    \
    GK_ATTR((channel_read_kernel<D, false>), sizeof(ReadSmem<D>));   \
    GK_ATTR((channel_read_kernel<D, true>), sizeof(ReadSmem<D>))
        GK_ATTRS(64);
        GK_ATTRS(128);
#undef GK_ATTRS
#undef GK_ATTR
        int device = 0, n = 0;
        if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) n = 148;
        sms = n;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int chunks = (max_len + CHUNK - 1) / CHUNK;
    const bool usual = taps == MAX_TAPS && dv == d && ((uintptr_t)conv_w & 15) == 0;
    const dim3 strips(dv / STRIP, n_heads, n_seqs);
    const bool alone = (long long)strips.x * strips.y * strips.z <= sms;
    for (int chunk0 = 0; chunk0 < chunks; chunk0 += wave) {
        const int here = chunks - chunk0 < wave ? chunks - chunk0 : wave;
        const Inputs in{(const bf16*)proj, low, conv_w, conv_state, a_log, dt_bias, norm, cu_q, slots, ld, ld_low, n_heads, n_kv, dv, taps, chunk0, wave};
        const dim3 units(here, n_heads, n_seqs);
#define GK_INNER(D, USUAL) gk_launch(channel_inner_kernel<D, USUAL>, units, dim3(THREADS), sizeof(InnerSmem<D>), s, in, work)
#define GK_WALK(D, RING) gk_launch_behind(channel_walk_kernel<D, RING>, strips, dim3(THREADS), sizeof(WalkSmem<D, RING>), s, in, work, state)
#define GK_READ(D, USUAL) gk_launch_behind(channel_read_kernel<D, USUAL>, units, dim3(THREADS), sizeof(ReadSmem<D>), s, in, (const float*)work, (bf16*)out, eps)
#define GK_CHANNEL(D)              \
    if (usual) GK_INNER(D, true);  \
    else GK_INNER(D, false);       \
    if (alone) GK_WALK(D, 6);      \
    else GK_WALK(D, 3);            \
    if (usual) GK_READ(D, true);   \
    else GK_READ(D, false)
        if (d == 64) {
            GK_CHANNEL(64);
        } else {
            GK_CHANNEL(128);
        }
#undef GK_CHANNEL
#undef GK_READ
#undef GK_WALK
#undef GK_INNER
    }
    GK_CHECK_LAUNCH("delta_channel");
    return GK_OK;
}
