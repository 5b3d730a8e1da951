// RMS norm that takes the residual arithmetic around it into one pass over a row of the float32 stream:
//
//   br  = branch[src]                                      (either type; absent: no addition)
//   br' = bw ? br * rsqrt(mean(br^2) + beps) * (boffset + bw) : br        the branch's own RMS norm
//   s   = x[src] + bscale * gain * br'                      gain: a learned vector (absent: ones)
//   out = w ? s * rsqrt(mean(s^2) + eps) * (offset + w) : s                in TO; out absent: only the sum
//
// sum_out (float32, nullable) receives s; it may be x itself when no rows are gathered.  Sums and statistics are
// float32; a row is reduced in an order fixed by the thread layout, so a row's result does not depend on the batch.
// Also here: the sum of two RMS-normed branches, a bias added to rows, and the gated activation with biases.
#include "common.cuh"

template <typename TB, typename TO>
__global__ void rms_chain_kernel(TO* __restrict__ out, float* sum_out, const float* x, const TB* branch,
                                 const int* __restrict__ rows, const float* __restrict__ w, const float* __restrict__ bw,
                                 const float* __restrict__ gain, int dim, int src_rows, float eps, float offset, float beps,
                                 float boffset, float bscale, int* err) {
    pdl_overlap_few();
    __shared__ float scratch[33];
    extern __shared__ float srow[];
    const int r = blockIdx.x;
    int src = rows ? rows[r] : r;
    if (src < 0 || src >= src_rows) {
        if (threadIdx.x == 0) atomicOr(err, XB_ERR_BAD_ROW);
        src = 0;
    }
    const float* xr = x + (size_t)src * dim;
    const TB* br = branch ? branch + (size_t)src * dim : nullptr;
    float binv = 1.f;
    if (br && bw) {
        float sb = 0.f;
        for (int i = threadIdx.x; i < dim; i += blockDim.x) {
            const float v = to_f32<TB>(br[i]);
            srow[i] = v;
            sb += v * v;
        }
        binv = 1.f / sqrtf(block_sum(sb, scratch) / (float)dim + beps);
    }
    float ss = 0.f;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        float v = xr[i];
        if (br) {
            float b = bw ? srow[i] * binv * (boffset + bw[i]) : to_f32<TB>(br[i]);
            if (gain) b *= gain[i];
            v = bscale == 1.f ? v + b : fmaf(bscale, b, v);
        }
        srow[i] = v;
        ss += v * v;
    }
    float inv = 1.f;
    if (out && w) inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)dim + eps);
    TO* o = out ? out + (size_t)r * dim : nullptr;
    float* so = sum_out ? sum_out + (size_t)r * dim : nullptr;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        const float v = srow[i];
        if (so) so[i] = v;
        if (o) o[i] = from_f32<TO>(w ? v * inv * (offset + w[i]) : v);
    }
}

// The same for rows in fours whose pieces start on vector boundaries: a thread keeps VPT vectors of its row in registers, all loads
// of a row are in flight at once, and what no kernel writes is fetched before the wait for the kernel before.  What bounded the form
// above were its three walks over the row, each waiting for the one before: four rows of 4,096 took 9.5 us of a decode
// step, 2.6 to 3.3 now; 1,798 rows of 1,024 12.9 us, 7.2 now.
template <typename T>
__device__ __forceinline__ float4 chain_load4(const T* p);
template <>
__device__ __forceinline__ float4 chain_load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 chain_load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
__device__ __forceinline__ void chain_store4(__nv_bfloat16* p, const float4& v) {
    uint2 u;
    *reinterpret_cast<__nv_bfloat162*>(&u.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162*>(&u.y) = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = u;
}

template <typename TB, int VPT>
__global__ void __launch_bounds__(512) rms_chain4_kernel(__nv_bfloat16* __restrict__ out, float* sum_out, const float* x, const TB* branch,
                                                         const int* __restrict__ rows, const float* __restrict__ w, const float* __restrict__ bw,
                                                         const float* __restrict__ gain, int dim, int src_rows, float eps, float offset, float beps,
                                                         float boffset, float bscale, int* err) {
    if ((unsigned long long)gridDim.x <= XB_FEW_BLOCKS) pdl_launch_dependents();
    __shared__ float scratch[33];
    const int nvec = dim / 4;
    float4 wv[VPT], bv[VPT], gv[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int v = threadIdx.x + i * blockDim.x;
        wv[i] = bv[i] = gv[i] = make_float4(1.f, 1.f, 1.f, 1.f);
        if (v >= nvec) continue;
        if (w) wv[i] = reinterpret_cast<const float4*>(w)[v];
        if (branch && bw) bv[i] = reinterpret_cast<const float4*>(bw)[v];
        if (branch && gain) gv[i] = reinterpret_cast<const float4*>(gain)[v];
    }
    const int r = blockIdx.x;
    pdl_wait();
    int src = rows ? rows[r] : r;
    if (src < 0 || src >= src_rows) {
        if (threadIdx.x == 0) atomicOr(err, XB_ERR_BAD_ROW);
        src = 0;
    }
    const float* xr = x + (size_t)src * dim;
    const TB* br = branch ? branch + (size_t)src * dim : nullptr;
    float4 s[VPT], b[VPT];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int v = threadIdx.x + i * blockDim.x;
        s[i] = b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (v >= nvec) continue;
        s[i] = chain_load4<float>(xr + v * 4);
        if (br) b[i] = chain_load4<TB>(br + v * 4);
    }
    if (br) {
        float binv = 1.f;
        if (bw) {
            float sb = 0.f;
#pragma unroll
            for (int i = 0; i < VPT; ++i) sb += b[i].x * b[i].x + b[i].y * b[i].y + (b[i].z * b[i].z + b[i].w * b[i].w);
            binv = 1.f / sqrtf(block_sum(sb, scratch) / (float)dim + beps);
        }
        auto add = [&](float& v, float u, float nw, float g) {
            if (bw) u = u * binv * (boffset + nw);
            if (gain) u *= g;
            v = bscale == 1.f ? v + u : fmaf(bscale, u, v);
        };
#pragma unroll
        for (int i = 0; i < VPT; ++i) {
            if (threadIdx.x + i * blockDim.x >= nvec) continue;
            add(s[i].x, b[i].x, bv[i].x, gv[i].x);
            add(s[i].y, b[i].y, bv[i].y, gv[i].y);
            add(s[i].z, b[i].z, bv[i].z, gv[i].z);
            add(s[i].w, b[i].w, bv[i].w, gv[i].w);
        }
    }
    float inv = 1.f;
    if (w) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < VPT; ++i) ss += s[i].x * s[i].x + s[i].y * s[i].y + (s[i].z * s[i].z + s[i].w * s[i].w);
        inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)dim + eps);
    }
    __nv_bfloat16* o = out + (size_t)r * dim;
    float* so = sum_out ? sum_out + (size_t)r * dim : nullptr;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
        const int v = threadIdx.x + i * blockDim.x;
        if (v >= nvec) continue;
        if (so) reinterpret_cast<float4*>(so)[v] = s[i];
        float4 y = s[i];
        if (w) y = make_float4(y.x * inv * (offset + wv[i].x), y.y * inv * (offset + wv[i].y), y.z * inv * (offset + wv[i].z), y.w * inv * (offset + wv[i].w));
        chain_store4(o + v * 4, y);
    }
}

template <typename TB, typename TO>
static int rms_chain_launch(void* out, float* sum_out, const float* x, const void* branch, const int* rows, const float* w,
                            const float* bw, const float* gain, int nrows, int dim, int src_rows, float eps, float offset,
                            float beps, float boffset, float bscale, int* err, cudaStream_t stream) {
    const uintptr_t wide = (uintptr_t)sum_out | (uintptr_t)x | (uintptr_t)w | (uintptr_t)bw | (uintptr_t)gain;
    // (rows that leave in bfloat16: a float32 engine keeps the order of its sums)
    if (sizeof(TO) == 2 && out && dim % 4 == 0 && dim <= 8192 && !(wide & 15) && !((uintptr_t)out & 7) && !((uintptr_t)branch & (4 * sizeof(TB) - 1))) {
        int threads = 64;
        while (threads < 512 && threads * 8 < dim) threads *= 2;      // two vectors a thread, more where 512 threads are not enough
        const int vpt = (dim / 4 + threads - 1) / threads;
#define XB_GO4(V)                                                                                                                       \
    return xb_launch_few(rms_chain4_kernel<TB, V>, dim3(nrows), dim3(threads), 0, stream, (__nv_bfloat16*)out, sum_out, x, (const TB*)branch, rows, w, \
                         bw, gain, dim, src_rows, eps, offset, beps, boffset, bscale, err)
        if (vpt <= 2) XB_GO4(2);
        XB_GO4(4);
#undef XB_GO4
    }
    const size_t smem = (size_t)dim * sizeof(float);
    if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
    if (smem > 48 * 1024) cudaFuncSetAttribute(rms_chain_kernel<TB, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int threads = dim >= 2048 ? 512 : (dim >= 512 ? 256 : 128);
    xb_launch_few(rms_chain_kernel<TB, TO>, dim3(nrows), dim3(threads), smem, stream, (TO*)out, sum_out, x, (const TB*)branch, rows, w, bw, gain, dim,
                                                              src_rows, eps, offset, beps, boffset, bscale, err);
    return xb_launch_status();
}

XB_EXPORT int xb_rms_chain(int branch_dtype, int out_dtype, void* out, float* sum_out, const float* x, const void* branch,
                           const int* rows, const float* w, const float* bw, const float* gain, int nrows, int dim,
                           int src_rows, float eps, float offset, float beps, float boffset, float bscale, int* err,
                           cudaStream_t stream) {
    if (nrows <= 0) return 0;
    typedef __nv_bfloat16 bf;
#define XB_ARGS out, sum_out, x, branch, rows, w, bw, gain, nrows, dim, src_rows, eps, offset, beps, boffset, bscale, err, stream
    if (branch_dtype == XB_F32) return out_dtype == XB_F32 ? rms_chain_launch<float, float>(XB_ARGS) : rms_chain_launch<float, bf>(XB_ARGS);
    return out_dtype == XB_F32 ? rms_chain_launch<bf, float>(XB_ARGS) : rms_chain_launch<bf, bf>(XB_ARGS);
#undef XB_ARGS
}

// out = sl * l * rsqrt(mean(l^2) + eps) * (offset + wl) + sr * r * rsqrt(mean(r^2) + eps) * (offset + wr), row by row
template <typename T>
__global__ void dual_rms_sum_kernel(T* __restrict__ out, const T* l, const T* r,
                                    const float* __restrict__ wl, const float* __restrict__ wr, int dim, float eps,
                                    float offset, float sl, float sr) {
    pdl_overlap_few();
    __shared__ float scratch[33];
    const size_t base = (size_t)blockIdx.x * dim;
    float a = 0.f, b = 0.f;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        const float u = to_f32<T>(l[base + i]), v = to_f32<T>(r[base + i]);
        a += u * u;
        b += v * v;
    }
    const float il = 1.f / sqrtf(block_sum(a, scratch) / (float)dim + eps);
    const float ir = 1.f / sqrtf(block_sum(b, scratch) / (float)dim + eps);
    for (int i = threadIdx.x; i < dim; i += blockDim.x) {
        const float u = to_f32<T>(l[base + i]) * il * (offset + wl[i]);
        const float v = to_f32<T>(r[base + i]) * ir * (offset + wr[i]);
        out[base + i] = from_f32<T>(sl * u + sr * v);
    }
}

XB_EXPORT int xb_dual_rms_sum(int dtype, void* out, const void* l, const void* r, const float* wl, const float* wr, int rows,
                              int dim, float eps, float offset, float sl, float sr, cudaStream_t stream) {
    if (rows <= 0) return 0;
    const int threads = dim >= 2048 ? 512 : (dim >= 512 ? 256 : 128);
    if (dtype == XB_F32)
        xb_launch_few(dual_rms_sum_kernel<float>, dim3(rows), dim3(threads), 0, stream, (float*)out, (const float*)l, (const float*)r, wl, wr, dim, eps, offset, sl, sr);
    else
        xb_launch_few(dual_rms_sum_kernel<__nv_bfloat16>, dim3(rows), dim3(threads), 0, stream, (__nv_bfloat16*)out, (const __nv_bfloat16*)l,
                                                                        (const __nv_bfloat16*)r, wl, wr, dim, eps, offset, sl, sr);
    return xb_launch_status();
}

// x[t, i] += bias[i]
template <typename T>
__global__ void add_bias_kernel(T* x, const float* __restrict__ bias, size_t n, int dim) {
    pdl_overlap_few();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = from_f32<T>(to_f32<T>(x[i]) + bias[i % dim]);
}

XB_EXPORT int xb_add_bias(int dtype, void* x, const float* bias, int rows, int dim, cudaStream_t stream) {
    const size_t n = (size_t)rows * dim;
    if (n == 0) return 0;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (dtype == XB_F32)
        xb_launch_few(add_bias_kernel<float>, dim3(blocks), dim3(256), 0, stream, (float*)x, bias, n, dim);
    else
        xb_launch_few(add_bias_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (__nv_bfloat16*)x, bias, n, dim);
    return xb_launch_status();
}

// out[t, i] = act(gu[t, i] + bias[i]) * (gu[t, I + i] + bias[I + i])    (float32 arithmetic, exact exponential)
template <typename TI, typename TO, int ACT>
__global__ void swiglu_bias_kernel(TO* __restrict__ out, const TI* gu, const float* __restrict__ bias, int I,
                                   size_t n) {
    pdl_overlap_few();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t t = i / I;
    const int c = (int)(i % I);
    const float g = to_f32<TI>(gu[t * 2 * I + c]) + bias[c];
    const float u = to_f32<TI>(gu[t * 2 * I + I + c]) + bias[I + c];
    out[i] = from_f32<TO>(gate_mul_f32<ACT>(g, u));
}

// The same arithmetic for many float32 rows that leave in bfloat16, in fours: a block walks over rows with its columns' biases in
// registers.  A value a thread, with a division for its row, took 23 us for 1,802 rows of 3,072 (55 MB), this 9.3.
template <int ACT>
__global__ void __launch_bounds__(256) swiglu_bias_rows_kernel(__nv_bfloat16* __restrict__ out, const float* gu, const float* __restrict__ bias, int I, int rows) {
    pdl_overlap_few();
    const int c = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (c >= I) return;
    const float4 bg = *reinterpret_cast<const float4*>(bias + c), bu = *reinterpret_cast<const float4*>(bias + I + c);
#pragma unroll 4
    for (int t = blockIdx.y; t < rows; t += gridDim.y) {
        const float* row = gu + (size_t)t * 2 * I + c;
        const float4 g = *reinterpret_cast<const float4*>(row), u = *reinterpret_cast<const float4*>(row + I);
        chain_store4(out + (size_t)t * I + c,
                     make_float4(gate_mul_f32<ACT>(g.x + bg.x, u.x + bu.x), gate_mul_f32<ACT>(g.y + bg.y, u.y + bu.y),
                                 gate_mul_f32<ACT>(g.z + bg.z, u.z + bu.z), gate_mul_f32<ACT>(g.w + bg.w, u.w + bu.w)));
    }
}

template <typename TI, typename TO>
static int swiglu_bias_launch(void* out, const void* gu, const float* bias, int rows, int I, int act, cudaStream_t stream) {
    const size_t n = (size_t)rows * I;
    if (sizeof(TI) == 4 && sizeof(TO) == 2 && rows > 64 && I % 4 == 0 && !(((uintptr_t)gu | (uintptr_t)bias) & 15) && !((uintptr_t)out & 7)) {
        // about eight blocks a processor, each with at least four rows where there are that many
        const unsigned bx = (unsigned)((I / 4 + 255) / 256), want = (148 * 8 + bx - 1) / bx, most = (unsigned)((rows + 3) / 4);
        const dim3 grid(bx, want < most ? want : most);
        if (act == XB_ACT_GELU_TANH)
            return xb_launch_few(swiglu_bias_rows_kernel<XB_ACT_GELU_TANH>, grid, dim3(256), 0, stream, (__nv_bfloat16*)out, (const float*)gu, bias, I, rows);
        return xb_launch_few(swiglu_bias_rows_kernel<XB_ACT_SILU>, grid, dim3(256), 0, stream, (__nv_bfloat16*)out, (const float*)gu, bias, I, rows);
    }
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (act == XB_ACT_GELU_TANH)
        xb_launch_few(swiglu_bias_kernel<TI, TO, XB_ACT_GELU_TANH>, dim3(blocks), dim3(256), 0, stream, (TO*)out, (const TI*)gu, bias, I, n);
    else
        xb_launch_few(swiglu_bias_kernel<TI, TO, XB_ACT_SILU>, dim3(blocks), dim3(256), 0, stream, (TO*)out, (const TI*)gu, bias, I, n);
    return xb_launch_status();
}

XB_EXPORT int xb_swiglu_bias(int in_dtype, int out_dtype, void* out, const void* gu, const float* bias, int rows, int I, int act,
                             cudaStream_t stream) {
    if (rows <= 0 || I <= 0) return 0;
    typedef __nv_bfloat16 bf;
    if (in_dtype == XB_F32)
        return out_dtype == XB_F32 ? swiglu_bias_launch<float, float>(out, gu, bias, rows, I, act, stream)
                                   : swiglu_bias_launch<float, bf>(out, gu, bias, rows, I, act, stream);
    return out_dtype == XB_F32 ? swiglu_bias_launch<bf, float>(out, gu, bias, rows, I, act, stream)
                               : swiglu_bias_launch<bf, bf>(out, gu, bias, rows, I, act, stream);
}
