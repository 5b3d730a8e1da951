// Attention with talking heads for single tokens (talking_decode.cu).
#pragma once
#include <cuda_runtime.h>

// As TalkMmaArgs (talking_attention_mma.cu), of which this is what single tokens need.
struct XbTalkDecode {
    const int *q_start, *start_pos, *block_table;
    const float* talk;
    float *part_o, *part_ml;
    int num_entries, table_stride, nh, nkv, page_size, num_pages, window, sink, parts, ldo;
    float scale, out_scale;
    int* err;
};
bool xb_talk_decode_takes(int nh, int nkv, int d, int dv);
int xb_talk_decode(void* out, const void* q, const void* k_pages, const void* v_pages, const XbTalkDecode& a, int tokens, int d, cudaStream_t stream);
