// Attention with talking heads for single tokens (the arithmetic is described in talking_attention.cu): a block takes one token
// and a range of its keys, 16 of them at a time.
//
//   a. a warp per key/value head: raw scores by mma.sync, keys as rows, the group's query heads as columns; keys come from the
//      pages straight into the operand's registers, the next 16 while these are worked on
//   b. a thread per key and heads / 16 heads: the mix across heads, float32 FMA
//   c. a warp per key/value head again: softmax, value sums by mma.sync (values as rows, heads as columns), values in registers
//      since before b.  Nothing of a key or a value passes through shared memory, only scores do.
//
// The kernel that holds tiles of 32 keys of all heads in shared memory (talking_attention_mma.cu) waits for its 130 KB tile
// between its steps and has one block a processor: eight tokens at 2,048 keys, 16 heads over 8 of 128 channels (67 MB),
// 33.6 us a layer; here, with two blocks a processor, 20.5.  (Started before its predecessor's end, with the first keys
// on their way, the step is 4 % longer: its blocks take the processors that the next product's would start on.)
// Weights are rounded once, in front of their product, and the rounded ones are summed; everything else is float32.
#include "common.cuh"
#include "mma_sync.cuh"
#include "talking_decode.h"

namespace {

typedef __nv_bfloat16 bf;
constexpr int KEYS = 16, MAX_GROUPS = 8, MAX_HEADS = 64;

__device__ __forceinline__ void mma_keys(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    const uint32_t a[4] = {a0, a1, a2, a3};
    xbmma::mma_bf16(c, a, b0, b1);
}
// 8 x 8 values of 16 bits: lane (row, pair of columns) gets what was in lane (column, pair of rows)
__device__ __forceinline__ unsigned transposed(unsigned v) {
    unsigned r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ unsigned pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&v);
}
__device__ __forceinline__ float2 unpack2(unsigned u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }

__device__ __forceinline__ unsigned word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// H: room for heads, ALL: all of it taken (else zeros lie there, which change no sum); D: channels of a head.
template <int H, bool ALL, int D>
__global__ void __launch_bounds__(256, 2) talk_decode_kernel(bf* __restrict__ out, const bf* q, const bf* k_pages, const bf* v_pages,
                                                             const XbTalkDecode a) {
    pdl_overlap_few();
    constexpr int LDS = H + 4, LDM = KEYS + 1, Q_BYTES = D * 2 + 16, KS = D / 32, VS = D / 64, SUMS = D / 16;
    __shared__ __align__(16) float raw[KEYS * LDS];            // [key][head]
    __shared__ float mixed[H * LDM];                           // [head][key]
    __shared__ __align__(16) float talk[H * H];
    __shared__ __align__(16) unsigned char qs[H * Q_BYTES];
    __shared__ int s_entry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, j = lane & 3;
    const int heads = ALL ? H : a.nh, G = a.nkv, rep = heads / G, t = blockIdx.x;
    if (tid == 0) s_entry = -1;
    __syncthreads();
    for (int e = tid; e < a.num_entries; e += 256)
        if (a.q_start[e] <= t && t < a.q_start[e + 1]) s_entry = e;
    for (int i = tid; i < H * H; i += 256) {
        const int to = i / H, from = i % H;
        talk[i] = to >= heads || from >= heads ? 0.f : a.talk ? a.talk[to * heads + from] : to == from ? 1.f : 0.f;
    }
    if (heads < H)
        for (int i = tid; i < KEYS * LDS; i += 256) raw[i] = 0.f;
    __syncthreads();
    const int b = s_entry;
    if (b < 0) return;
    const int pos = a.start_pos[b] + t - a.q_start[b];
    const int* table = a.block_table + (size_t)b * a.table_stride;
    int lo = a.window > 0 ? max(pos - a.window + 1, 0) : 0, hi = pos + 1;
    if (a.parts > 1) {
        const int base = lo / KEYS, chunks = (hi + KEYS - 1) / KEYS - base, per = (chunks + a.parts - 1) / a.parts;
        const int first = (base + (int)blockIdx.y * per) * KEYS;
        lo = max(lo, first);
        hi = min(hi, first + per * KEYS);
    }
    const bool first_part = blockIdx.y == 0, works = warp < G;
    float m[2], l[2], o[SUMS][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        m[e] = a.sink && first_part ? 0.f : -INFINITY;
        l[e] = 0.f;                                            // (of this lane's keys; the sink's 1 is added at the end)
    }
#pragma unroll
    for (int i = 0; i < SUMS; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    // row of the pages that key `lane & 15` of a chunk has, -1 for none
    auto row_of = [&](int c) -> int {
        const int key = c * KEYS + (lane & 15);
        if (key < lo || key >= hi) return -1;
        const int page = table[key / a.page_size];
        if (page < 0 || page >= a.num_pages) {
            atomicOr(a.err, XB_ERR_BAD_PAGE);
            return -1;
        }
        return (page * G + warp) * a.page_size + key % a.page_size;
    };
    uint4 k[2][KS], v[VS][4];
    auto fetch_keys = [&](int rows) {                          // keys g and g + 8 (a key that is not there: any row, its score is not used)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int row = __shfl_sync(0xffffffffu, rows, u * 8 + g);
            const uint4* src = reinterpret_cast<const uint4*>(k_pages) + (size_t)max(row, 0) * (D / 8) + j;
#pragma unroll
            for (int s = 0; s < KS; ++s) k[u][s] = src[s * 4];
        }
    };
    const int c_lo = lo / KEYS, c_hi = hi > lo ? (hi + KEYS - 1) / KEYS : c_lo;
    int rows = -1, rows_next = -1;
    if (works && c_lo < c_hi) {
        rows = row_of(c_lo);
        fetch_keys(rows);
        if (c_lo + 1 < c_hi) rows_next = row_of(c_lo + 1);
    }
    for (int i = tid; i < heads * (D / 8); i += 256) {
        const int h = i / (D / 8), c = i % (D / 8);
        *reinterpret_cast<uint4*>(qs + h * Q_BYTES + c * 16) = *reinterpret_cast<const uint4*>(q + ((size_t)t * heads + h) * D + c * 8);
    }
    __syncthreads();
#pragma unroll 1
    for (int c = c_lo; c < c_hi; ++c) {
        unsigned there = 0;
        if (works) {
            there = __ballot_sync(0xffffffffu, rows >= 0);
            float sc[4] = {0.f, 0.f, 0.f, 0.f};                // (key g, head 2 j), (g, 2 j + 1), (g + 8, 2 j), (g + 8, 2 j + 1)
#pragma unroll
            for (int s = 0; s < KS; ++s) {
                uint4 qv = make_uint4(0u, 0u, 0u, 0u);
                if (g < rep) qv = *reinterpret_cast<const uint4*>(qs + (warp * rep + g) * Q_BYTES + s * 64 + j * 16);
                mma_keys(sc, k[0][s].x, k[1][s].x, k[0][s].y, k[1][s].y, qv.x, qv.y);
                mma_keys(sc, k[0][s].z, k[1][s].z, k[0][s].w, k[1][s].w, qv.z, qv.w);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * j + e < rep) {
                    raw[g * LDS + warp * rep + 2 * j + e] = sc[e] * a.scale;
                    raw[(g + 8) * LDS + warp * rep + 2 * j + e] = sc[2 + e] * a.scale;
                }
#pragma unroll
            for (int e = 0; e < 4; ++e) {                      // keys 2 j, 2 j + 1, 2 j + 8, 2 j + 9: eight values of every 64
                const int row = __shfl_sync(0xffffffffu, rows, 2 * j + (e & 1) + (e >> 1) * 8);
                const uint4* src = reinterpret_cast<const uint4*>(v_pages) + (size_t)max(row, 0) * (D / 8) + g;
#pragma unroll
                for (int s = 0; s < VS; ++s) {
                    v[s][e] = src[s * 8];
                    if (row < 0) v[s][e] = make_uint4(0u, 0u, 0u, 0u);            // (0 times what lies there could be NaN)
                }
            }
            if (c + 1 < c_hi) {
                rows = rows_next;
                fetch_keys(rows);
                if (c + 2 < c_hi) rows_next = row_of(c + 2);
            }
        }
        __syncthreads();
        {
            const int key = tid & 15;
            const float4* sr = reinterpret_cast<const float4*>(raw + key * LDS);
#pragma unroll 1
            for (int h = tid >> 4; h < heads; h += 16) {
                const float4* tr = reinterpret_cast<const float4*>(talk + h * H);
                float m0 = 0.f, m1 = 0.f, m2 = 0.f, m3 = 0.f;
#pragma unroll 4
                for (int i = 0; i < H / 4; ++i) {
                    const float4 w = tr[i], s = sr[i];
                    m0 = fmaf(w.x, s.x, m0);
                    m1 = fmaf(w.y, s.y, m1);
                    m2 = fmaf(w.z, s.z, m2);
                    m3 = fmaf(w.w, s.w, m3);
                }
                mixed[h * LDM + key] = (m0 + m1) + (m2 + m3);
            }
        }
        __syncthreads();
        if (works) {
            float p[4], corr[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float* row = mixed + (warp * rep + min(2 * j + e, rep - 1)) * LDM;
                const bool mine = 2 * j + e < rep;
                const float s0 = mine && (there >> g & 1u) ? row[g] : -INFINITY, s1 = mine && (there >> (g + 8) & 1u) ? row[g + 8] : -INFINITY;
                float most = fmaxf(s0, s1);
                most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 4));
                most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 8));
                most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 16));
                const float m_new = fmaxf(m[e], most), base = m_new == -INFINITY ? 0.f : m_new;
                corr[e] = __expf(m[e] - base);
                m[e] = m_new;
                p[e] = __expf(s0 - base);
                p[e + 2] = __expf(s1 - base);
            }
            const unsigned p0 = pack2(p[0], p[1]), p1 = pack2(p[2], p[3]);
            const float2 f0 = unpack2(p0), f1 = unpack2(p1);
            l[0] = l[0] * corr[0] + (f0.x + f1.x);             // as the product sees them
            l[1] = l[1] * corr[1] + (f0.y + f1.y);
            if (a.sink && first_part && c == c_lo && g == 0) { // the entry of score 0 without a key
                l[0] += corr[0];
                l[1] += corr[1];
            }
            const unsigned b0 = transposed(p0), b1 = transposed(p1);
#pragma unroll
            for (int w = 0; w < SUMS / 2; ++w) {
                // rows g of the product: two of the lane's first values; rows g + 8: of the other 64 channels, or of the last four
                const int wy = VS == 2 ? w : w + 2;
                const unsigned x0 = word(v[0][0], w), x1 = word(v[0][1], w), x2 = word(v[0][2], w), x3 = word(v[0][3], w);
                const unsigned y0 = word(v[VS - 1][0], wy), y1 = word(v[VS - 1][1], wy), y2 = word(v[VS - 1][2], wy), y3 = word(v[VS - 1][3], wy);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float(&acc)[4] = o[w * 2 + e];
                    acc[0] *= corr[0], acc[1] *= corr[1], acc[2] *= corr[0], acc[3] *= corr[1];
                    const unsigned pick = e ? 0x7632u : 0x5410u;
                    mma_keys(acc, __byte_perm(x0, x1, pick), __byte_perm(y0, y1, pick), __byte_perm(x2, x3, pick), __byte_perm(y2, y3, pick), b0, b1);
                }
            }
        }
    }
    if (!works) return;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
        if (c_lo >= c_hi && a.sink && first_part) l[e] = 1.f;
        if (2 * j + e >= rep) continue;
        const int h = warp * rep + 2 * j + e;
        // sum i holds values g * 8 + i and 64 + g * 8 + i of the lane's two heads (of 64 channels: g * 8 + i and g * 8 + 4 + i)
        constexpr int OTHER = VS == 2 ? 64 : 4;
        if (a.parts > 1) {
            const size_t at = ((size_t)t * a.parts + blockIdx.y) * heads + h;
#pragma unroll
            for (int hd = 0; hd < 2; ++hd)
#pragma unroll
                for (int i = 0; i < SUMS; i += 4)
                    *reinterpret_cast<float4*>(a.part_o + at * D + hd * OTHER + g * 8 + i) =
                        make_float4(o[i][hd * 2 + e], o[i + 1][hd * 2 + e], o[i + 2][hd * 2 + e], o[i + 3][hd * 2 + e]);
            if (g == 0) *reinterpret_cast<float2*>(a.part_ml + at * 2) = make_float2(m[e], l[e]);
        } else {
            const float f = l[e] > 0.f ? a.out_scale / l[e] : 0.f;
            bf* dst = out + (size_t)t * a.ldo + (size_t)h * D + g * 8;
#pragma unroll
            for (int hd = 0; hd < 2; ++hd)
#pragma unroll
                for (int i = 0; i < SUMS; i += 2)
                    *reinterpret_cast<unsigned*>(dst + hd * OTHER + i) = pack2(o[i][hd * 2 + e] * f, o[i + 1][hd * 2 + e] * f);
        }
    }
}

template <int H>
int launch(bf* out, const bf* q, const bf* k_pages, const bf* v_pages, const XbTalkDecode& a, int tokens, int d, cudaStream_t stream) {
    const dim3 grid(tokens, a.parts);
#define XB_GO(ALL, D) return xb_launch_few(talk_decode_kernel<H, ALL, D>, grid, dim3(256), 0, stream, out, q, k_pages, v_pages, a)
    if (d == 64) {
        if (a.nh == H) XB_GO(true, 64);
        XB_GO(false, 64);
    }
    if (a.nh == H) XB_GO(true, 128);
    XB_GO(false, 128);
#undef XB_GO
}

}  // namespace

// Heads of 64 or 128 channels (eight values a lane of every 64), keys and values alike; a warp for each of at most eight key/value heads,
// with at most eight heads each (the eight columns of an mma.sync).  Against the kernel with tiles in shared memory, us, eight tokens at 2,048
// keys and one at 700: 16 heads over 8 of 128 channels 42.0 -> 33.8 and 44.0 -> 25.7, 64 over 8 66.6 -> 58.4 and 72.7 -> 42.0, 24 over 3 of 64
// channels 42.0 -> 25.7 and 42.0 -> 23.6, 8 over 1 of 64 27.6 -> 21.5 and 25.6 -> 21.5; nowhere slower.
bool xb_talk_decode_takes(int nh, int nkv, int d, int dv) {
    return d == dv && (d == 64 || d == 128) && nkv >= 1 && nkv <= MAX_GROUPS && nh <= MAX_HEADS && nh % nkv == 0 && nh / nkv >= 1 && nh / nkv <= 8;
}

int xb_talk_decode(void* out, const void* q, const void* k_pages, const void* v_pages, const XbTalkDecode& a, int tokens, int d, cudaStream_t stream) {
    bf* o = (bf*)out;
    const bf *qs = (const bf*)q, *ks = (const bf*)k_pages, *vs = (const bf*)v_pages;
    return a.nh <= 16 ? launch<16>(o, qs, ks, vs, a, tokens, d, stream)
           : a.nh <= 32 ? launch<32>(o, qs, ks, vs, a, tokens, d, stream)
                        : launch<64>(o, qs, ks, vs, a, tokens, d, stream);
}
