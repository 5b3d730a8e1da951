// Shared device helpers for the engine's kernels (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

// Bits of the device-side error word that kernels set instead of faulting.
#define XB_ERR_BAD_TOKEN 1   // a token id outside [0, vocab)
#define XB_ERR_BAD_PAGE 2    // a block-table entry outside [0, num_pages)
#define XB_ERR_WAIT 4        // a bounded wait on an mbarrier gave up
#define XB_ERR_BAD_ROW 8     // a requested row outside [0, tokens)
#define XB_ERR_SCRATCH 16    // scratch memory that a kernel must find zeroed was not
#define XB_ERR_BAD_POSITION 32  // a token position outside the position table

// Element type codes shared with the Python side.
#define XB_F32 0
#define XB_BF16 1

#define XB_EXPORT extern "C" __attribute__((visibility("default")))

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result.  The order of the
// additions is fixed by the thread layout, so the result does not depend on what else runs.
__device__ __forceinline__ float block_sum(float v, float* scratch /* >= 33 floats */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < nwarps ? scratch[lane] : 0.f;
        t = warp_sum(t);
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// silu(g) * u for bfloat16 activations: the exponential and the quotient by the fast intrinsics, whose
// error (a few units in the last place of float32) is far below half a unit of the bfloat16 result.
// Every bfloat16 kernel that forms this product uses this function, so that they agree bit for bit;
// the float32 path divides and exponentiates exactly.
__device__ __forceinline__ float silu_mul_bf16(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }

// Activations of a gated feed-forward, act(g) * f(u), by code (shared with the Python side).  Two of them take
// parameters p0 and p1:
//   relu           max(g, 0) * u
//   clamped swish  with a = min(g, p0) and b = clamp(u, -p0, p0):  a * sigmoid(p1 * a) * (b + 1)
#define XB_ACT_SILU 0
#define XB_ACT_GELU_TANH 1
#define XB_ACT_RELU 2
#define XB_ACT_SWISH_CLAMP 3
// gelu in its tanh form: 0.5 z (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))), float32 throughout
__device__ __forceinline__ float gelu_tanh_f32(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float swish_clamp_f32(float g, float u, float limit, float alpha) {
    const float a = fminf(g, limit), b = fminf(fmaxf(u, -limit), limit);
    return a / (1.f + expf(-alpha * a)) * (b + 1.f);
}
template <int ACT>
__device__ __forceinline__ float gate_mul_bf16(float g, float u, float p0 = 0.f, float p1 = 0.f) {
    if (ACT == XB_ACT_RELU) return fmaxf(g, 0.f) * u;
    if (ACT == XB_ACT_SWISH_CLAMP) return swish_clamp_f32(g, u, p0, p1);
    return ACT == XB_ACT_GELU_TANH ? gelu_tanh_f32(g) * u : silu_mul_bf16(g, u);
}
template <int ACT>
__device__ __forceinline__ float gate_mul_f32(float g, float u, float p0 = 0.f, float p1 = 0.f) {
    if (ACT == XB_ACT_RELU) return fmaxf(g, 0.f) * u;
    if (ACT == XB_ACT_SWISH_CLAMP) return swish_clamp_f32(g, u, p0, p1);
    return ACT == XB_ACT_GELU_TANH ? gelu_tanh_f32(g) * u : g / (1.f + expf(-g)) * u;
}
// the same by a code known only at run time (epilogues of products, where the branch costs nothing)
__device__ __forceinline__ float gate_mul_any(int act, float g, float u, float p0, float p1) {
    switch (act) {
        case XB_ACT_GELU_TANH: return gelu_tanh_f32(g) * u;
        case XB_ACT_RELU: return fmaxf(g, 0.f) * u;
        case XB_ACT_SWISH_CLAMP: return swish_clamp_f32(g, u, p0, p1);
        default: return g / (1.f + expf(-g)) * u;
    }
}

// Last CUDA error of a launch as an int for the caller (0 = ok).
static inline int xb_launch_status() { return (int)cudaGetLastError(); }

// Programmatic dependent launch: a kernel launched through xb_launch may be scheduled while the
// kernel before it in the stream is still running; it calls pdl_wait() before it touches anything
// that kernel may have written (or still reads), and pdl_launch_dependents() as early as it likes
// to let the kernel after it do the same.  Both are no-ops in a kernel launched the plain way.
// What a predecessor writes is read through pointers without __restrict__: that word promises that nobody else writes there
// while the kernel runs, so that the compiler may load in front of the wait.
// A kernel that allocates tensor memory lets the next one start only once every thread block has its columns (and a block
// that allocates none, where it leaves): the next kernel's blocks hold theirs while they wait for this grid's end, so a block
// of this grid that still waited for columns on the same processor would wait for ever, and so would they.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

#include <cstdlib>
static inline bool xb_pdl_enabled() {   // XINFER_B200_PDL=0 switches the overlap off
    static int v = -1;
    if (v < 0) {
        const char* e = getenv("XINFER_B200_PDL");
        v = (e && e[0] == '0') ? 0 : 1;
    }
    return v != 0;
}

// `overlap` false: the kernel starts only when the one before it has completed (its pdl_wait() is then a no-op).
template <typename... KArgs, typename... Args>
static inline int xb_launch_opt(bool overlap, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap && xb_pdl_enabled() ? 1 : 0;
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
    return rc != cudaSuccess ? (int)rc : xb_launch_status();
}
template <typename... KArgs, typename... Args>
static inline int xb_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    return xb_launch_opt(true, kernel, grid, block, smem, stream, args...);
}
// For the small kernels between the large ones: overlapped with their neighbours while the grid is no more than one block per
// processor, as in decode steps, whose launches then hide each other's start-up.  In a prompt a kernel that starts early finds
// its neighbour's blocks on most processors and crowds its own onto the others.  Such a kernel begins with pdl_overlap_few().
constexpr unsigned long long XB_FEW_BLOCKS = 148;
constexpr int XB_FEW_TOKENS = 8;            // a kernel that walks a request's tokens lets its successor start at this many or fewer
__device__ __forceinline__ void pdl_overlap_few() {
    if ((unsigned long long)gridDim.x * gridDim.y * gridDim.z <= XB_FEW_BLOCKS) pdl_launch_dependents();
    pdl_wait();
}
template <typename... KArgs, typename... Args>
static inline int xb_launch_few(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    const bool few = (unsigned long long)grid.x * grid.y * grid.z <= XB_FEW_BLOCKS;
    return xb_launch_opt(few, kernel, grid, block, smem, stream, args...);
}
