// The layers of a pre-norm stack queued by one native call: norm, q/k/v product, head preparation and cache write, attention,
// output product, norm, gate/up product, gate, down product - the kernels that the parts launch one by one, in the same order with
// the same arguments.  Queued from Python a launch costs some 20 us of host time, more than most of these kernels run: three
// prompts of up to 777 tokens beside sixteen decoding requests (0.6B sizes, eight layers) took 1,750 us and take 1,030 now.
// No device code here.
#include <cublas_v2.h>

#include "common.cuh"

// the kernels' entry points, explained where they are defined
XB_EXPORT int xb_rmsnorm_bf16(void* out, void* sum_out, const void* x, const void* branch, const int* rows, const float* w, int nrows, int dim,
                              int src_rows, float eps, float offset, int* err, cudaStream_t stream);
XB_EXPORT int xb_gemm_skinny_tc(void* out, int out_f32, const void* x, const void* w, int M, int N, int K, int splits, int* err, cudaStream_t stream);
XB_EXPORT int xb_qk_norm_rope_write_bf16(void* q_out, void* k_cache, void* v_cache, const void* qkv, const float* q_w, const float* k_w,
                                         const float* cos_t, const float* sin_t, const int* positions, const int* req_of_token,
                                         const int* block_table, int table_stride, int tokens, int nh, int nkv, int d, int rot, int interleaved,
                                         int page_size, int num_pages, int max_pos, float eps, int write_kv, int* err, cudaStream_t stream);
XB_EXPORT int xb_attn_prefill_tc(void* out, const void* q, const void* kc, const void* vc, const int* q_start, const int* start_pos, const int* table,
                                 int stride, int tokens, int nh, int nkv, int d, int dv, long long ldo, int ps, int num_pages, int window, int keep,
                                 float scale, float softcap, float slope_exp, const float* sink, float out_scale, const int* work, int ctas, int* err,
                                 cudaStream_t stream);
XB_EXPORT int xb_attn_decode_tc(void* out, float* part_o, float* part_ml, const void* q, const void* kc, const void* vc, const int* plan,
                                const int* table, int stride, int q_rows, int nh, int nkv, int d, int dv, long long ldo, int ps, int num_pages,
                                int keep, float scale, float softcap, float slope_exp, const float* sink, float out_scale, int dec_max,
                                int splits_max, int tokens, int ctas, int* tickets, int overlap, int* err, cudaStream_t stream);
XB_EXPORT int xb_swiglu_bf16(void* out, const void* gu, int tokens, int inter, int act, float p0, float p1, cudaStream_t stream);
XB_EXPORT int xb_swiglu_rows_bf16(void* out, const void* gu, int tokens, int inter, int act, float p0, float p1, cudaStream_t stream);

typedef cublasStatus_t (*GemmEx)(cublasHandle_t, cublasOperation_t, cublasOperation_t, int, int, int, const void*, const void*, cudaDataType, int,
                                 const void*, cudaDataType, int, const void*, void*, cudaDataType, int, cublasComputeType_t, cublasGemmAlgo_t);

// What all layers share and what a layer has of its own; the Python side mirrors both field by field.
struct XbDenseStep {
    void *x, *h, *qkv, *q, *o, *attn_out, *gate_up, *act, *ffn_out;
    const int *positions, *req_of_token, *table, *q_start, *start_pos;
    const float *cos_t, *sin_t;
    const int *work, *plan;
    float *part_o, *part_ml;
    int *tickets, *err;
    void *gemm_ex, *blas;                   // cublasGemmEx and the current handle, for steps of more tokens than `skinny`
    int tokens, hidden, nh, nkv, d, inter, table_stride, page_size, num_pages, max_pos, rot, interleaved, window;
    int prefill_ctas, decode_ctas, splits_max, small, dec_max, overlap, skinny, many_rows, activation;
    float eps1, offset1, eps2, offset2, qk_eps, scale, p0, p1;
};
struct XbDenseLayer {
    const void *w_qkv, *w_o, *w_gate_up, *w_down;
    const float *norm1, *norm2, *q_norm, *k_norm;
    void *k_pages, *v_pages;
};

XB_EXPORT int xb_dense_step_size() { return (int)sizeof(XbDenseStep); }

// Leaves the last layer's feed-forward output in ffn_out, still to be added to x.
// `library`: receives the number of products that went to the library.
XB_EXPORT int xb_dense_layers(const XbDenseStep* step, const XbDenseLayer* layers, int count, int* library, cudaStream_t stream) {
    const XbDenseStep& S = *step;
    const int T = S.tokens, qd = S.nh * S.d, width = (S.nh + 2 * S.nkv) * S.d;
    *library = 0;
    auto product = [&](void* out, const void* in, const void* w, int N, int K) -> int {
        if (T <= S.skinny) {
            const int rc = xb_gemm_skinny_tc(out, 0, in, w, T, N, K, 0, S.err, stream);
            if (rc != (int)cudaErrorNotSupported) return rc;
        }
        const float one = 1.f, zero = 0.f;
        ++*library;
        const cublasStatus_t rc = reinterpret_cast<GemmEx>(S.gemm_ex)(
            (cublasHandle_t)S.blas, CUBLAS_OP_T, CUBLAS_OP_N, N, T, K, &one, w, CUDA_R_16BF, K, in, CUDA_R_16BF, K, &zero, out, CUDA_R_16BF, N,
            CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
        return rc == CUBLAS_STATUS_SUCCESS ? 0 : (int)cudaErrorUnknown;
    };
    for (int i = 0; i < count; ++i) {
        const XbDenseLayer& L = layers[i];
        int rc = xb_rmsnorm_bf16(S.h, i ? S.x : nullptr, S.x, i ? S.ffn_out : nullptr, nullptr, L.norm1, T, S.hidden, T, S.eps1, S.offset1, S.err, stream);
        if (!rc) rc = product(S.qkv, S.h, L.w_qkv, width, S.hidden);
        if (!rc)
            rc = xb_qk_norm_rope_write_bf16(S.q, L.k_pages, L.v_pages, S.qkv, L.q_norm, L.k_norm, S.cos_t, S.sin_t, S.positions, S.req_of_token,
                                            S.table, S.table_stride, T, S.nh, S.nkv, S.d, S.rot, S.interleaved, S.page_size, S.num_pages, S.max_pos,
                                            S.qk_eps, 1, S.err, stream);
        if (!rc && S.prefill_ctas > 0)
            rc = xb_attn_prefill_tc(S.o, S.q, L.k_pages, L.v_pages, S.q_start, S.start_pos, S.table, S.table_stride, T, S.nh, S.nkv, S.d, S.d, qd,
                                    S.page_size, S.num_pages, S.window, 0, S.scale, 0.f, 0.f, nullptr, 1.f, S.work, S.prefill_ctas, S.err, stream);
        if (!rc && S.small > 0)
            rc = xb_attn_decode_tc(S.o, S.part_o, S.part_ml, S.q, L.k_pages, L.v_pages, S.plan, S.table, S.table_stride, T, S.nh, S.nkv, S.d, S.d, qd,
                                   S.page_size, S.num_pages, 0, S.scale, 0.f, 0.f, nullptr, 1.f, S.dec_max, S.splits_max, S.small, S.decode_ctas,
                                   S.tickets, S.overlap, S.err, stream);
        if (!rc) rc = product(S.attn_out, S.o, L.w_o, S.hidden, qd);
        if (!rc) rc = xb_rmsnorm_bf16(S.h, S.x, S.x, S.attn_out, nullptr, L.norm2, T, S.hidden, T, S.eps2, S.offset2, S.err, stream);
        if (!rc) rc = product(S.gate_up, S.h, L.w_gate_up, 2 * S.inter, S.hidden);
        if (!rc)
            rc = T >= S.many_rows ? xb_swiglu_rows_bf16(S.act, S.gate_up, T, S.inter, S.activation, S.p0, S.p1, stream)
                                  : xb_swiglu_bf16(S.act, S.gate_up, T, S.inter, S.activation, S.p0, S.p1, stream);
        if (!rc) rc = product(S.ffn_out, S.act, L.w_down, S.hidden, S.inter);
        if (rc) return rc;
    }
    return 0;
}
