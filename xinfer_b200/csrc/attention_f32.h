// Float32 attention over the paged cache, by tiles of queries (attention_f32.cu).
#pragma once
#include <cuda_runtime.h>

// The arguments of xb_attention_plain (generic.cu), where they are explained.
struct XbAttentionF32 {
    float* out;
    const float *q, *k_cache, *v_cache, *sink;
    const int *positions, *req_of_token, *block_table;
    int* err;
    long long q_ts, q_hs, ldo;
    int k_stride, v_stride, table_stride, requests, tokens, nh, nkv, d, dv, page_size, num_pages, window, keep, chunk;
    float scale, softcap, slope_exp, out_scale;
};

// Whether the kernel takes these sizes, strides and addresses (never a question of how many tokens there are).
bool xb_attention_f32_takes(const XbAttentionF32& p);
int xb_attention_f32(const XbAttentionF32& p, cudaStream_t stream);
