// Float32 attention over the paged cache by tiles of queries (the plain kernel of generic.cu takes one warp per query).
#include "attention_f32.h"

#include "common.cuh"

namespace {

// ------------------------------------------------------------------------------------------
// A block takes up to 16 query rows that read the same key/value head - consecutive tokens times the heads of a group - and
// walks over their keys in groups of 32 (positions 32 c .. 32 c + 31), which it brings to shared memory once for all rows:
// the values while the scores are formed, the next keys while the values are summed.  One buffer of each lets four blocks
// share a processor and hide each other's waits (with two of each and two blocks: 113 us).  A warp holds up to four rows.  Scores: a lane per key, four sums of every fourth
// channel each; softmax: the group's maximum and sum over the warp; values: a lane per four channels, keys in order.
// A row visits the groups that hold a key it sees and no others, each in the same way, so its result depends on its own
// position and keys alone, not on how many rows run beside it.  A block's rows are of one run: neighbouring tokens of a request.
// What bounded the kernel with a warp per query were the five shuffles, two exponentials and two dependent loads of every
// key; here these are shared by 32 keys and by the rows, and the loads of the keys by the rows.  Two prompts of 301 and
// 145 tokens, 16 heads over 8, head size 128: 292 us a layer before, 58 us now.
// ------------------------------------------------------------------------------------------
constexpr int KEYS = 32, ROWS = 16, WARPS = 4;

__device__ __forceinline__ unsigned long long af_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long af_mul(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long af_pack(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 af_unpack(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ void af_copy16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 16 : 0) : "memory");
}

// The tokens [t0, t0 + tokens) of request b, neighbours in the step; R: rows of a warp, tokens * heads <= R * WARPS.
template <int R>
__device__ __forceinline__ void attend_run(const XbAttentionF32& p, int t0, int tokens, int b, float* af_smem) {
    const int ldk = p.d + 4, ldv = p.dv;          // a lane per key: rows 16 bytes apart from a multiple of all banks
    float* sk = af_smem;                          // [KEYS][ldk]
    float* sv = sk + KEYS * ldk;                  // [KEYS][ldv]
    float* sp = sv + KEYS * ldv;                  // [R * WARPS][KEYS] weights
    float* sq = sp + R * WARPS * KEYS;            // [R * WARPS][d], scaled
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = p.nh / p.nkv, g = blockIdx.y, h0 = blockIdx.z * ROWS, heads = min(group - h0, ROWS), rows = tokens * heads;
    if (b >= 0)
        for (int i = threadIdx.x; i < rows * p.d; i += WARPS * 32) {
            const int r = i / p.d, c = i - r * p.d;
            sq[i] = p.q[(size_t)(t0 + r / heads) * p.q_ts + (size_t)(g * group + h0 + r % heads) * p.q_hs + c] * p.scale;
        }
    // row i * WARPS + warp of the run: its token's position (-1: no row), the first key beside the kept ones that it sees
    int pos[R], lo[R];
    float m[R], l[R], slope[R];
    unsigned long long acc[R][2];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = i * WARPS + warp;
        pos[i] = -1;
        lo[i] = 0;
        m[i] = -INFINITY;
        l[i] = slope[i] = 0.f;
        acc[i][0] = acc[i][1] = 0ull;
        if (r < rows) {
            const int t = t0 + r / heads, h = g * group + h0 + r % heads;
            pos[i] = p.positions[t];
            lo[i] = p.window > 0 ? max(pos[i] - p.window + 1, 0) : 0;
            if (p.chunk > 0) lo[i] = max(lo[i], pos[i] / p.chunk * p.chunk);
            if (p.slope_exp > 0.f) slope[i] = exp2f(-p.slope_exp * (float)(h + 1) / (float)p.nh);
            if (p.sink) {      // the entry without a key: exp(sink - m) with m = sink
                m[i] = p.sink[h];
                l[i] = 1.f;
            }
        }
    }
    if (b >= 0) {                                 // (else padding)
        int hi = -1, first = 0x7fffffff;
        for (int t = t0; t < t0 + tokens; ++t) {
            const int ps = p.positions[t];
            int low = p.window > 0 ? max(ps - p.window + 1, 0) : 0;
            if (p.chunk > 0) low = max(low, ps / p.chunk * p.chunk);
            hi = max(hi, ps);
            first = min(first, low);
        }
        const int* table = p.block_table + (size_t)b * p.table_stride;
        const int last = hi / KEYS, begin = first / KEYS;
        const int kept = min(p.keep, first);                     // positions before `first` that some row may see
        const int kept_groups = min((kept + KEYS - 1) / KEYS, begin);
        const int steps = kept_groups + last - begin + 1;
        auto group_of = [&](int n) { return n < kept_groups ? n : begin + n - kept_groups; };
        // row of the caches that key `lane` of group n has, -1 for none (behind the last key, or a page that does not exist)
        auto row_of = [&](int n) -> long long {
            const int j = n < steps ? group_of(n) * KEYS + lane : hi + 1;
            if (j > hi) return -1;
            const int page = table[j / p.page_size];
            return page < 0 || page >= p.num_pages ? -1 : ((long long)page * p.nkv + g) * p.page_size + j % p.page_size;
        };
        auto bring = [&](float* dst, int ld, const float* src, int stride, int width, long long rows_of_lanes) {
#pragma unroll
            for (int i = 0; i < KEYS / WARPS; ++i) {
                const int k = warp + i * WARPS;
                const long long row = __shfl_sync(0xffffffffu, rows_of_lanes, k);
                if (lane * 4 < width) af_copy16(dst + k * ld + lane * 4, src + (row < 0 ? 0 : row * stride) + lane * 4, row >= 0);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        long long rows_now = row_of(0);
        bring(sk, ldk, p.k_cache, p.k_stride, p.d, rows_now);
        for (int n = 0; n < steps; ++n) {
            const int j = group_of(n) * KEYS + lane;
            unsigned vis[R], any = 0u, all = 0xffffffffu;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const bool sees = j <= pos[i] && (j >= lo[i] || j < p.keep);
                if (sees && rows_now < 0) atomicOr(p.err, XB_ERR_BAD_PAGE);
                vis[i] = __ballot_sync(0xffffffffu, sees && rows_now >= 0);
                any |= vis[i];
                all &= vis[i];
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();                       // the keys have landed, the values before them have been read
            bring(sv, ldv, p.v_cache, p.v_stride, p.dv, rows_now);
            unsigned long long sum[R][2];
#pragma unroll
            for (int i = 0; i < R; ++i) sum[i][0] = sum[i][1] = 0ull;
            if (any) {
                const float* kr = sk + lane * ldk;
                const float* qb = sq + warp * p.d;
#pragma unroll 8
                for (int x = 0; x < p.d; x += 4) {
                    const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(kr + x);
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qb + i * WARPS * p.d + x);
                        sum[i][0] = af_fma(qv.x, kv.x, sum[i][0]);
                        sum[i][1] = af_fma(qv.y, kv.y, sum[i][1]);
                    }
                }
            }
            __syncthreads();                       // the keys have been read
            rows_now = row_of(n + 1);
            bring(sk, ldk, p.k_cache, p.k_stride, p.d, rows_now);
            float* pb = sp + warp * KEYS;
            if (any) {
                float sc[R], most[R], total[R], corr[R];      // (sums of products spelled out: the same for every R)
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const float2 s01 = af_unpack(sum[i][0]), s23 = af_unpack(sum[i][1]);
                    sc[i] = (s01.x + s01.y) + (s23.x + s23.y);
                    if (p.softcap > 0.f) sc[i] = p.softcap * tanhf(sc[i] / p.softcap);
                    sc[i] = fmaf(-slope[i], (float)(pos[i] - j), sc[i]);
                    most[i] = vis[i] >> lane & 1u ? sc[i] : -INFINITY;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < R; ++i) most[i] = fmaxf(most[i], __shfl_xor_sync(0xffffffffu, most[i], o));
#pragma unroll
                for (int i = 0; i < R; ++i) {      // (a row that sees no key of the group: times 1, plus 0)
                    const float m_new = fmaxf(m[i], most[i]);
                    corr[i] = vis[i] ? expf(m[i] - m_new) : 1.f;      // exp(-inf) = 0 on the first key
                    total[i] = vis[i] >> lane & 1u ? expf(sc[i] - m_new) : 0.f;
                    pb[i * WARPS * KEYS + lane] = total[i];
                    const unsigned long long c2 = af_pack(corr[i], corr[i]);
                    acc[i][0] = af_mul(acc[i][0], c2);
                    acc[i][1] = af_mul(acc[i][1], c2);
                    m[i] = m_new;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int i = 0; i < R; ++i) total[i] += __shfl_xor_sync(0xffffffffu, total[i], o);
#pragma unroll
                for (int i = 0; i < R; ++i) l[i] = fmaf(l[i], corr[i], total[i]);
            }
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();                       // the values have landed
            if (any && lane * 4 < p.dv) {
                const float* vb = sv + lane * 4;
                if (all == 0xffffffffu) {
#pragma unroll 2
                    for (int k = 0; k < KEYS; k += 4) {
                        float4 w4[R];
#pragma unroll
                        for (int i = 0; i < R; ++i) w4[i] = *reinterpret_cast<const float4*>(pb + i * WARPS * KEYS + k);
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(vb + (k + kk) * ldv);
#pragma unroll
                            for (int i = 0; i < R; ++i) {
                                const float w = kk == 0 ? w4[i].x : kk == 1 ? w4[i].y : kk == 2 ? w4[i].z : w4[i].w;
                                const unsigned long long w2 = af_pack(w, w);
                                acc[i][0] = af_fma(w2, vv.x, acc[i][0]);
                                acc[i][1] = af_fma(w2, vv.y, acc[i][1]);
                            }
                        }
                    }
                } else {       // keys that a row does not see take no part in its sums, whatever their values are
                    for (int k = 0; k < KEYS; ++k) {
                        const ulonglong2 vv = *reinterpret_cast<const ulonglong2*>(vb + k * ldv);
#pragma unroll
                        for (int i = 0; i < R; ++i)
                            if (vis[i] >> k & 1u) {
                                const float w = pb[i * WARPS * KEYS + k];
                                const unsigned long long w2 = af_pack(w, w);
                                acc[i][0] = af_fma(w2, vv.x, acc[i][0]);
                                acc[i][1] = af_fma(w2, vv.y, acc[i][1]);
                            }
                    }
                }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                           // the buffers are free for the next run's keys
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int r = i * WARPS + warp;
        if (r >= rows || lane * 4 >= p.dv) continue;
        const float inv = l[i] > 0.f ? p.out_scale / l[i] : 0.f;
        float* o = p.out + (size_t)(t0 + r / heads) * p.ldo + (size_t)(g * group + h0 + r % heads) * p.dv + lane * 4;
        const float2 a = af_unpack(acc[i][0]), c = af_unpack(acc[i][1]);
        const float v[4] = {a.x, a.y, c.x, c.y};
#pragma unroll
        for (int x = 0; x < 4; ++x) o[x] = b < 0 ? 0.f : v[x] * inv;
    }
}

// The first token of the k-th run that does not start a tile, -1 if there are fewer.
__device__ __forceinline__ int further_run(const XbAttentionF32& p, int tile, int k) {
    for (int base = 0; base < p.tokens; base += 32) {
        const int t = base + (int)(threadIdx.x & 31);
        unsigned starts = __ballot_sync(0xffffffffu, t < p.tokens && t % tile && p.req_of_token[t] != p.req_of_token[t - 1]);
        const int here = __popc(starts);
        if (k < here) {
            for (; k > 0; --k) starts &= starts - 1;
            return base + __ffs(starts) - 1;
        }
        k -= here;
    }
    return -1;
}

// How many tokens the run has in its tile.
__device__ __forceinline__ int run_length(const XbAttentionF32& p, int tile, int t0) {
    const int b = p.req_of_token[t0], end = min(t0 / tile * tile + tile, p.tokens);
    int t = t0 + 1;
    while (t < end && p.req_of_token[t] == b) ++t;
    return t - t0;
}

// The runs from the k-th on, one after the other (a step with more runs than requests).
template <int R>
__device__ __noinline__ void attend_rest(const XbAttentionF32& p, int tile, int k, float* af_smem) {
    for (int t0; (t0 = further_run(p, tile, k)) >= 0; ++k) attend_run<R>(p, t0, run_length(p, tile, t0), p.req_of_token[t0], af_smem);
}

// The first `tiles` blocks of a grid take the run that starts their tile of `tile` tokens (at most ROWS / min(group, ROWS)), the
// others the further ones, one each, so that the requests of a decode step are attended side by side; a run of few rows takes
// the form with one row to a warp.  With the runs of a tile one after the other in its block, 16 tokens at context 1,024 took
// 1,758 us (8 heads of their own) and 896 (16 over 8), a warp per query 1,221 and 1,225; now 65 each.  (1,500 tokens of one
// request: 547 and 555; 32 heads of 64 channels 760 and 786.)  A loop over runs around the one call made its steps 8 % longer.
template <int R>
__global__ void __launch_bounds__(WARPS * 32, 4) attention_f32_kernel(const __grid_constant__ XbAttentionF32 p, int tile, int tiles) {
    extern __shared__ __align__(16) float af_smem[];
    const int heads = min(p.nh / p.nkv - (int)blockIdx.z * ROWS, ROWS);
    const int k = (int)blockIdx.x - tiles;
    const int t0 = k < 0 ? blockIdx.x * tile : further_run(p, tile, k);
    if (t0 < 0) return;
    const int n = run_length(p, tile, t0);
    if (R == 1 || n * heads > WARPS) attend_run<R>(p, t0, n, p.req_of_token[t0], af_smem);
    else attend_run<1>(p, t0, n, p.req_of_token[t0], af_smem);
    if (k >= 0 && blockIdx.x + 1 == gridDim.x) attend_rest<R>(p, tile, k + 1, af_smem);
}

template <int R>
int launch(const XbAttentionF32& p, int tile, cudaStream_t stream) {
    const int group = p.nh / p.nkv, tiles = (p.tokens + tile - 1) / tile;
    const int others = min(max(p.requests - 1, 1), p.tokens - tiles);      // (`requests` may be wrong: then a block takes several runs, or none)
    const int smem = (KEYS * (p.d + 4) + KEYS * p.dv + R * WARPS * (p.d + KEYS)) * 4;
    cudaFuncSetAttribute(attention_f32_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attention_f32_kernel<R><<<dim3(tiles + others, p.nkv, (group + ROWS - 1) / ROWS), WARPS * 32, smem, stream>>>(p, tile, tiles);
    return xb_launch_status();
}

}  // namespace

// Rows of keys and values by 16-byte copies, four value channels a lane.  The rule does not look at the number of tokens: the
// two kernels sum in different orders, and a token's result must not depend on the step that it came in.
bool xb_attention_f32_takes(const XbAttentionF32& p) {
    return p.d % 4 == 0 && p.d <= 128 && p.dv % 4 == 0 && p.dv <= 128 && p.k_stride % 4 == 0 && p.v_stride % 4 == 0 &&
           !(((uintptr_t)p.k_cache | (uintptr_t)p.v_cache) & 15) && p.nkv <= 65535;
}

int xb_attention_f32(const XbAttentionF32& p, cudaStream_t stream) {
    const int heads = min(p.nh / p.nkv, ROWS);
    // Shorter tiles while their blocks are at most two a processor: keys are then read more often, but by more processors.  64
    // tokens behind 2,048: 228 us in whole tiles, 160 so (16 heads over 8); 32 heads of 64 channels 242 and 170, with a limit of four
    // blocks a processor 206.
    const long long columns = (long long)p.nkv * ((p.nh / p.nkv + ROWS - 1) / ROWS);
    int tile = max(1, min(ROWS / heads, p.tokens));
    while (tile > 1 && (p.tokens + tile / 2 - 1) / (tile / 2) * columns <= 296) tile /= 2;
    const int rows = tile * heads;
    if (rows <= WARPS) return launch<1>(p, tile, stream);
    if (rows <= 2 * WARPS) return launch<2>(p, tile, stream);
    return launch<4>(p, tile, stream);
}
