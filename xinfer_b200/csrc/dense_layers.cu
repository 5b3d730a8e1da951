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

// What all layers share, what a layer has of its own, and what has been queued.  The Python side lays out its mirrors by the
// descriptions that xb_dense_fields gives, so the two cannot differ.
#define XB_DENSE_STEP(F)                                                                                                                     \
    F(ptr, x) F(ptr, h) F(ptr, qkv) F(ptr, q) F(ptr, o) F(ptr, attn_out) F(ptr, gate_up) F(ptr, act) F(ptr, ffn_out)                         \
    F(ptr, positions) F(ptr, req_of_token) F(ptr, table) F(ptr, q_start) F(ptr, start_pos) F(ptr, cos_t) F(ptr, sin_t)                       \
    F(ptr, work) F(ptr, plan) F(ptr, part_o) F(ptr, part_ml) F(ptr, tickets) F(ptr, err)                                                     \
    F(ptr, gemm_ex) F(ptr, blas) /* cublasGemmEx and the current handle, for steps of more tokens than `skinny` */                           \
    F(int, tokens) F(int, hidden) F(int, nh) F(int, nkv) F(int, d) F(int, inter) F(int, table_stride) F(int, page_size) F(int, num_pages)    \
    F(int, max_pos) F(int, rot) F(int, interleaved) F(int, window) F(int, prefill_ctas) F(int, decode_ctas) F(int, splits_max) F(int, small) \
    F(int, dec_max) F(int, overlap) F(int, skinny) F(int, many_rows) F(int, activation)                                                      \
    F(float, eps1) F(float, offset1) F(float, eps2) F(float, offset2) F(float, qk_eps) F(float, scale) F(float, p0) F(float, p1)
#define XB_DENSE_LAYER(F)                                                                                                                    \
    F(ptr, w_qkv) F(ptr, w_o) F(ptr, w_gate_up) F(ptr, w_down) F(ptr, norm1) F(ptr, norm2) F(ptr, q_norm) F(ptr, k_norm) F(ptr, k_pages)     \
    F(ptr, v_pages)
// `half`: the half layer that the call stopped in; `launch`: what it stopped at (XbDenseLaunch), `blas_status` if that was the
// library; then how many launches of each kind have been queued, in the order of XbDenseLaunch
#define XB_DENSE_DONE(F)                                                                                                                     \
    F(int, half) F(int, launch) F(int, blas_status) F(int, norms) F(int, skinny) F(int, library) F(int, ropes) F(int, prefill) F(int, decode) F(int, gates)
typedef void* ptr;
#define XB_MEMBER(type, name) type name;
#define XB_DESCRIBED(type, name) #type " " #name ";"
struct XbDenseStep { XB_DENSE_STEP(XB_MEMBER) };
struct XbDenseLayer { XB_DENSE_LAYER(XB_MEMBER) };
struct XbDenseDone { XB_DENSE_DONE(XB_MEMBER) };
enum XbDenseLaunch { NORM, SKINNY, LIBRARY, ROPE, PREFILL, DECODE, GATE };

XB_EXPORT const char* xb_dense_fields(int which) {
    return which == 0 ? XB_DENSE_STEP(XB_DESCRIBED) : which == 1 ? XB_DENSE_LAYER(XB_DESCRIBED) : XB_DENSE_DONE(XB_DESCRIBED);
}

// Half layers [begin, end): 2 i is layer i up to its attention, 2 i + 1 the rest of it.  The last one leaves the layer's feed-forward output in
// ffn_out, still to be added to x.  cudaErrorNotSupported: everything before the attention of half layer done->half is queued, and
// an attention kernel does not take the step; the caller attends with another one and goes on at done->half + 1.
XB_EXPORT int xb_dense_layers(const XbDenseStep* step, const XbDenseLayer* layers, int begin, int end, XbDenseDone* done, cudaStream_t stream) {
    const XbDenseStep& S = *step;
    const int T = S.tokens, qd = S.nh * S.d, width = (S.nh + 2 * S.nkv) * S.d;
    typedef const int* cip;
    typedef const float* cfp;
    cfp cos_t = (cfp)S.cos_t, sin_t = (cfp)S.sin_t;
    cip positions = (cip)S.positions, requests = (cip)S.req_of_token, table = (cip)S.table;
    int* err = (int*)S.err;
    *done = XbDenseDone{};
    auto queued = [&](XbDenseLaunch what, int rc) -> int {
        if (rc) done->launch = what;
        else ++(&done->norms)[what];
        return rc;
    };
    auto product = [&](void* out, const void* in, const void* w, int N, int K) -> int {
        if (T <= S.skinny) {
            const int rc = xb_gemm_skinny_tc(out, 0, in, w, T, N, K, 0, err, stream);
            if (rc != (int)cudaErrorNotSupported) return queued(SKINNY, rc);
        }
        const float one = 1.f, zero = 0.f;
        done->blas_status = reinterpret_cast<GemmEx>(S.gemm_ex)(
            (cublasHandle_t)S.blas, CUBLAS_OP_T, CUBLAS_OP_N, N, T, K, &one, w, CUDA_R_16BF, K, in, CUDA_R_16BF, K, &zero, out, CUDA_R_16BF, N,
            CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
        return queued(LIBRARY, done->blas_status == CUBLAS_STATUS_SUCCESS ? 0 : (int)cudaErrorUnknown);
    };
    for (int half = begin; half < end; ++half) {
        const int i = half / 2;
        const XbDenseLayer& L = layers[i];
        int rc = 0;
        done->half = half;
        if (half % 2 == 0) {
            rc = queued(NORM, xb_rmsnorm_bf16(S.h, i ? S.x : nullptr, S.x, i ? S.ffn_out : nullptr, nullptr, (cfp)L.norm1, T, S.hidden, T, S.eps1,
                                              S.offset1, err, stream));
            if (!rc) rc = product(S.qkv, S.h, L.w_qkv, width, S.hidden);
            if (!rc)
                rc = queued(ROPE, xb_qk_norm_rope_write_bf16(S.q, L.k_pages, L.v_pages, S.qkv, (cfp)L.q_norm, (cfp)L.k_norm, cos_t, sin_t, positions,
                                                             requests, table, S.table_stride, T, S.nh, S.nkv, S.d, S.rot, S.interleaved, S.page_size,
                                                             S.num_pages, S.max_pos, S.qk_eps, 1, err, stream));
            if (!rc && S.prefill_ctas > 0)
                rc = queued(PREFILL, xb_attn_prefill_tc(S.o, S.q, L.k_pages, L.v_pages, (cip)S.q_start, (cip)S.start_pos, table, S.table_stride, T, S.nh,
                                                        S.nkv, S.d, S.d, qd, S.page_size, S.num_pages, S.window, 0, S.scale, 0.f, 0.f, nullptr, 1.f,
                                                        (cip)S.work, S.prefill_ctas, err, stream));
            if (!rc && S.small > 0)
                rc = queued(DECODE, xb_attn_decode_tc(S.o, (float*)S.part_o, (float*)S.part_ml, S.q, L.k_pages, L.v_pages, (cip)S.plan, table,
                                                      S.table_stride, T, S.nh, S.nkv, S.d, S.d, qd, S.page_size, S.num_pages, 0, S.scale, 0.f, 0.f,
                                                      nullptr, 1.f, S.dec_max, S.splits_max, S.small, S.decode_ctas, (int*)S.tickets, S.overlap, err,
                                                      stream));
        } else {
            rc = product(S.attn_out, S.o, L.w_o, S.hidden, qd);
            if (!rc)
                rc = queued(NORM, xb_rmsnorm_bf16(S.h, S.x, S.x, S.attn_out, nullptr, (cfp)L.norm2, T, S.hidden, T, S.eps2, S.offset2, err, stream));
            if (!rc) rc = product(S.gate_up, S.h, L.w_gate_up, 2 * S.inter, S.hidden);
            if (!rc)
                rc = queued(GATE, T >= S.many_rows ? xb_swiglu_rows_bf16(S.act, S.gate_up, T, S.inter, S.activation, S.p0, S.p1, stream)
                                                   : xb_swiglu_bf16(S.act, S.gate_up, T, S.inter, S.activation, S.p0, S.p1, stream));
            if (!rc) rc = product(S.ffn_out, S.act, L.w_down, S.hidden, S.inter);
        }
        if (rc) return rc;
    }
    return 0;
}
