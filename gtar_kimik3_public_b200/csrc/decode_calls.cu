// The attention layer of a decode step as one call from the host: the q|k|v product of a few tokens, attention with norm, rotation and
// cache write in its input stage, and the output product.  The three kernels are those of their own entry points; what is saved is
// the host's part of two further calls (checks, two more buffers and argument conversion, some 8 us each), which is what a layer called
// outside a captured step waits for.  Measured: a layer of 4B sizes at 8 sequences of 255 to 4,095 49.6 us by three calls, 40.5 by this one.

#include "common.cuh"

GK_EXPORT int gk_gemv_bf16(const void* w, int n, int k, long long ldw, const void* x, int tokens, long long ldx, void* out, int out_dtype,
                           int swiglu, float act_a, float act_b, void* stream);
GK_EXPORT int gk_attention_decode_fused_bf16(const void* qkv, const void* wq, const void* wk, int weight_dtype, int use_norm, float eps,
                                             const float* cos_table, const float* sin_table, int table_positions, int max_position,
                                             int write_kv, void* k_pages, void* v_pages, void* out, float* part_o, float* part_ml,
                                             const int* kv_len, const int* slots, const int* block_table, int n_seqs, int n_q, int n_kv,
                                             int head_dim, int max_pages, int page_size, float scale, int window, int n_splits, void* stream);

// x [tokens, hidden], out [tokens, out_width] bfloat16, one token a sequence; `scratch`: tokens * (2 n_q + 2 n_kv) * head_dim bfloat16 numbers.
GK_EXPORT int gk_attention_decode_layer_bf16(const void* x, int tokens, int hidden, const void* w_qkv, const void* w_o, int out_width, void* scratch,
                                             void* out, const void* wq, const void* wk, int weight_dtype, int use_norm, float eps,
                                             const float* cos_table, const float* sin_table, int table_positions, int max_position,
                                             int write_kv, void* k_pages, void* v_pages, const int* kv_len, const int* slots,
                                             const int* block_table, int n_q, int n_kv, int head_dim, int max_pages, int page_size,
                                             float scale, int window, int n_splits, void* stream) {
    GK_REQUIRE(n_splits >= 1 && n_splits <= 8, "attention_decode_layer: takes at most 8 splits");
    const int rows = (n_q + 2 * n_kv) * head_dim, read = n_q * head_dim;
    __nv_bfloat16* qkv = (__nv_bfloat16*)scratch;
    __nv_bfloat16* o = qkv + (size_t)tokens * rows;
    int status = gk_gemv_bf16(w_qkv, rows, hidden, hidden, x, tokens, hidden, qkv, GK_BF16, 0, 0.f, 0.f, stream);
    if (status == GK_OK)
        status = gk_attention_decode_fused_bf16(qkv, wq, wk, weight_dtype, use_norm, eps, cos_table, sin_table, table_positions, max_position,
                                                write_kv, k_pages, v_pages, o, nullptr, nullptr, kv_len, slots, block_table, tokens, n_q, n_kv,
                                                head_dim, max_pages, page_size, scale, window, n_splits, stream);
    if (status == GK_OK) status = gk_gemv_bf16(w_o, out_width, read, read, o, tokens, read, out, GK_BF16, 0, 0.f, 0.f, stream);
    return status;
}
