// Float32 matrix product  out[M, N] = a[M, K] . w[N, K]^T  on the tensor cores, with float32's own precision.
//
// Every operand is cut into three bfloat16 numbers that add up to it exactly, each rounded to nearest.  The second and third are kept
// 2^8 and 2^16 times as large, so that no digit of a small operand falls below the smallest bfloat16.  Of the nine products the
// six largest are formed; what is left out is below 2^-24 of the whole (of an operand below 2^-126: below its last digit, 2^-149,
// times the other one):
//     w0 a0 + 2^-8 ((w0 a1 + w1 a0) + 2^-8 (w1 a1 + w0 a2 + w2 a0)).
// Tensor memory rounds a running sum towards zero, so little stays there: of 32 terms at a time the products w0 a0, whose digits
// fit, go to one column, and the small ones, whose cut-off digits do not count, to another; these two are added in registers,
// to nearest, and so are the sums of 32 terms.  The four 16 terms of a panel are taken as first and third, second and fourth, so that
// up to 32 terms nothing is added to a large sum in tensor memory.  (Splitting a number into parts whose products are exact is Dekker's,
// 1971.)
// An output's sum has that one form whatever M, the tile or the operands' alignment is, so a row's result does not depend on
// what else is in the step.  A sum that is not finite is formed again term by term (an infinity times a part of 0 is no number).
//
// Relative error against 64 bits (2-norm), by float32 multiply-adds of 16 terms and so: normal operands, K = 64 8.4e-8 and 5.5e-8,
// 1,024 1.65e-7 and 1.16e-7, 3,072 2.6e-7 and 1.8e-7; operands near 2^-124 the same; one term 1,000 times the others, K = 1,024
// 1.85e-7 and 1.50e-7.  Where it is larger: the tensor cores cut every product off near 2^-25 of the largest of its 16, so short
// sums of one sign, K = 64 5.0e-8 and 5.6e-8, the more the more one term stands out (1,000 times the others, all of one sign, K =
// 64 9.3e-8 and 2.2e-7, 1,024 1.55e-7 and 1.75e-7; 10^6 times, 1,024 1.9e-7 and 3.7e-7).
// With the leading part cut off instead of rounded, parts not scaled and all products in one column (and 446 x 4,096 x 1,024 41
// instead of 46 us): a single product 5.6e-8, where this has 2.5e-8 as multiply-adds have, operands near 2^-116 3.2e-6.
//
// The cut rows of W go to tensor memory, from where an operand A costs no bytes of shared memory; that holds the panels as they come
// and the cut rows of A (with the cut rows of W there too, a panel of 64 k took 1,730 cycles at 16 tokens instead of 1,500).  What
// bounds the kernel then at 64 tokens is instructions, 2.9 to 3.1 of four a cycle (the tensor pipe a third of the time): cutting, and
// the adding warps' reads, of which the small sums are 13 of 215 us at 2,048 x 6,144 x 1,024.  At 16 tokens, 2.7 a cycle while memory
// is read at half its rate, it is the time from a panel to its sums, which two teams of cutting warps and two stages overlap: 48
// panels of 1,024 rows 46.1 -> 38.9 us with one team -> with two.
// Measured, float32 multiply-adds and now: 446 x 4,096 x 1,024 145 -> 47 us, 446 x 1,024 x 3,072 209 -> 49 us, 2,048 x 6,144 x
// 1,024 786 -> 215 us (120 TFLOP/s), one row of 6,144 x 1,024 21.2 -> 20.5 us, two of 151,936 x 1,024 123 -> 121 us, one of 24,576 x
// 4,096 90 -> 98 us (4,100 GB/s; 117 with one team and all tiles 128 rows high).
//
// Roles of a block (persistent, a tile of up to 128 rows of W and TOK of A after another): one thread asks for panels by TMA, a ring
// of them ahead; sixteen warps cut the panels, a thread 16 k (or 32 of every other panel) of a row of W; two warps issue the products,
// of 32 k each; four or eight warps add up the sums, through a ring of column buffers, and write the tile.
#include "common.cuh"
#include "gemm_f32_tc.h"
#include "tc_common.cuh"

namespace {

using namespace xbtc;

constexpr int TILE_W = 128, PANEL = 64, HALF = 32, TERMS = 32, CUTTERS = 16, ISSUERS = PANEL / TERMS;

template <int TOK>
struct Shape {
    static constexpr int ADDERS = TOK > 32 ? 8 : 4, WIDTH = TOK / (ADDERS / 4);      // columns of an adding warp
    static constexpr int THREADS = (CUTTERS + ISSUERS + ADDERS + 1) * 32;
    static constexpr int A_BYTES = TOK * 128, STAGE = 3 * A_BYTES, STAGES = 2;       // the cut rows of A: three parts
    static constexpr int RAW = (TILE_W + TOK) * PANEL * 4, RAWS = TOK <= 32 ? 4 : 3;
    // Two teams of cutting warps take every other panel, so that one cuts while the other waits.  A barrier of the ring then has one
    // team only, which waits for its phases one after the other (a phase that nobody of a team waits for could be taken for the next).
    static constexpr int TEAMS = RAWS % 2 == 0 ? 2 : 1;
    static constexpr int SMEM = RAWS * RAW + STAGES * STAGE + 1024;
    // columns of tensor memory: the cut rows of W (two numbers a column), then the sums
    static constexpr int W_COLS = 3 * (PANEL / 2), SUMS = STAGES * W_COLS, BUF = 2 * TOK, BUFS = TOK <= 16 ? 8 : TOK <= 32 ? 4 : 2;
    static_assert(SUMS + BUFS * BUF <= 512 && BUFS % ISSUERS == 0, "columns");
    static constexpr int AT_ONCE = TOK <= 32 ? 16 : 8;                               // columns of either sum that an adding warp reads at once
};

// one lane of the warp, the same one every time
__device__ __forceinline__ bool elect_one() {
    uint32_t is;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(is));
    return is != 0;
}

// an output whose sum is not finite: its terms one by one, in float32
__device__ __noinline__ float term_by_term(const float* a, const float* w, int K) {
    float sum = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        float part = 0.f;
        for (int k = k0; k < min(k0 + 16, K); ++k) part = fmaf(a[k], w[k], part);
        sum += part;
    }
    return sum;
}

__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// the three parts of two numbers, the second and third 2^8 and 2^16 times their value
__device__ __forceinline__ void cut2(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const f32x2 minus = pack2(-1.f, -1.f), up = pack2(256.f, 256.f);
    auto halves = [](uint32_t v) { return pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); };
    float r0, r1;
    hi = pack_bf16(x, y);
    const f32x2 r = mul2(fma2(halves(hi), minus, pack2(x, y)), up);      // (no digit of a difference is lost)
    unpack2(r, r0, r1);
    mid = pack_bf16(r0, r1);
    unpack2(mul2(fma2(halves(mid), minus, r), up), r0, r1);
    lo = __byte_perm(__float_as_uint(r0), __float_as_uint(r1), 0x7632);  // (what is left has no more than eight bits)
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld_nowait(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_nowait(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
// umma_bf16_ta onto 2^-SHIFT times what is there
template <int SHIFT>
__device__ __forceinline__ void umma_bf16_ta_scaled(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "n"(SHIFT) : "memory");
}
// four numbers of a panel's row as TMA leaves them: halves of 32 numbers, rows of 128 bytes, swizzled
__device__ __forceinline__ float4 raw4(const unsigned char* rows, int row, int chunk) {
    return *reinterpret_cast<const float4*>(rows + row * 128 + ((chunk ^ (row & 7)) << 4));
}
// the same from a row that is not aligned, `left` numbers of which are there
__device__ __forceinline__ float4 any4(const float* p, int left) {
    return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}

// BY_TMA: the operands' rows start on 16-byte boundaries; else the cutters read them from global memory themselves.
template <int TOK, bool BY_TMA>
__global__ void __launch_bounds__(Shape<TOK>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, float* out, const float* a,
                   const float* w, int M, int N, int K, int height, int* err) {
    typedef Shape<TOK> S;
    extern __shared__ unsigned char gf_smem[];
    __shared__ unsigned long long s_full[S::STAGES], s_empty[S::STAGES], s_sum[S::BUFS], s_free[S::BUFS], s_raw[S::RAWS], s_read[S::RAWS];
    __shared__ uint32_t s_tmem;
    const uint32_t base = (smem_u32(gf_smem) + 1023u) & ~1023u;
    unsigned char* mem = gf_smem + (base - smem_u32(gf_smem));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 32) {
        for (int i = 0; i < S::STAGES; ++i) {
            mbar_init(smem_u32(&s_full[i]), CUTTERS / S::TEAMS);
            mbar_init(smem_u32(&s_empty[i]), ISSUERS);
        }
        for (int i = 0; i < S::BUFS; ++i) {
            mbar_init(smem_u32(&s_sum[i]), 1);
            mbar_init(smem_u32(&s_free[i]), S::ADDERS);
        }
        for (int i = 0; i < S::RAWS; ++i) {
            mbar_init(smem_u32(&s_raw[i]), 1);
            mbar_init(smem_u32(&s_read[i]), CUTTERS / S::TEAMS);
        }
        mbar_init_fence();
    }
    if (warp == 0) tmem_alloc(&s_tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    pdl_launch_dependents();   // only now: see pdl_launch_dependents on tensor memory
    pdl_wait();
    const int across = (M + TOK - 1) / TOK, tiles = (N + height - 1) / height * across, panels = (K + PANEL - 1) / PANEL;

    if (warp < CUTTERS) {
        // 16 k of a row of W for every team, in the quarter of tensor memory's lanes that a warp of this number may write, and eight of a
        // row of A
        constexpr int TEAMS = S::TEAMS, WARPS = CUTTERS / TEAMS;
        const int team = warp / WARPS, row = (warp & 3) * 32 + lane, part0 = ((warp % WARPS) >> 2) * TEAMS;
        const int r = (threadIdx.x % (WARPS * 32)) >> 3, c = threadIdx.x & 7, all_k = panels * PANEL;
        const bool has_a = r < TOK, has_w = (warp & 3) * 32 < height;      // (rows behind the tile's are not cut: what is there reaches no result)
        int stage = team % S::STAGES, raw = team, tile = blockIdx.x, k0 = team * PANEL;
        uint32_t parity = 1, raw_parity = 0;                      // (a fresh barrier's phase before its first counts as over)
        for (;; k0 += TEAMS * PANEL) {
            for (; k0 >= all_k; k0 -= all_k) tile += gridDim.x;
            if (tile >= tiles) break;
            float4 v[TEAMS][4], u[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
            if (BY_TMA) {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_raw[raw]), raw_parity, err, true))) break;
                const unsigned char* src = mem + raw * S::RAW;
#pragma unroll
                for (int t = 0; t < TEAMS; ++t)
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[t][i] = raw4(src + ((part0 + t) >> 1) * (TILE_W * 128), row, ((part0 + t) & 1) * 4 + i);
                src += TILE_W * PANEL * 4;
                if (has_a) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) u[i] = raw4(src + (c >> 2) * (TOK * 128), r, (c & 3) * 2 + i);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_read[raw]));
                raw += TEAMS;
                if (raw >= S::RAWS) {
                    raw -= S::RAWS;
                    raw_parity ^= 1;
                }
            } else {
                const int n = tile / across * height + row, m = tile % across * TOK + r, ka = k0 + c * 8;
#pragma unroll
                for (int t = 0; t < TEAMS; ++t)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int kw = k0 + (part0 + t) * 16 + i * 4;
                        v[t][i] = any4(w + (size_t)n * K + kw, n < N ? K - kw : 0);
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i) u[i] = any4(a + (size_t)m * K + ka + i * 4, has_a && m < M ? K - ka - i * 4 : 0);
            }
#pragma unroll
            for (int t = 0; t < TEAMS; ++t) {
                uint32_t hi[8], mid[8], lo[8];
                if (!has_w) {
                    if (t == 0 && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[stage]), parity, err, true))) goto done;
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    cut2(v[t][i].x, v[t][i].y, hi[2 * i], mid[2 * i], lo[2 * i]);
                    cut2(v[t][i].z, v[t][i].w, hi[2 * i + 1], mid[2 * i + 1], lo[2 * i + 1]);
                }
                if (t == 0) {
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_empty[stage]), parity, err, true))) goto done;
                    tc_fence_after();
                }
                const uint32_t to = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(stage * S::W_COLS + (part0 + t) * 8);
                tmem_st8(to, hi);
                tmem_st8(to + PANEL / 2, mid);
                tmem_st8(to + PANEL, lo);
            }
            if (has_a) {
                unsigned char* dst = mem + S::RAWS * S::RAW + stage * S::STAGE + r * 128 + ((c ^ (r & 7)) << 4);
                uint4 h, md, l;
                cut2(u[0].x, u[0].y, h.x, md.x, l.x);
                cut2(u[0].z, u[0].w, h.y, md.y, l.y);
                cut2(u[1].x, u[1].y, h.z, md.z, l.z);
                cut2(u[1].z, u[1].w, h.w, md.w, l.w);
                *reinterpret_cast<uint4*>(dst) = h;
                *reinterpret_cast<uint4*>(dst + S::A_BYTES) = md;
                *reinterpret_cast<uint4*>(dst + 2 * S::A_BYTES) = l;
            }
            tmem_st_wait();
            tc_fence_before();
            fence_async_shared();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&s_full[stage]));
            stage += TEAMS;
            if (stage >= S::STAGES) {
                stage -= S::STAGES;
                parity ^= 1;
            }
        }
    done:;
    } else if (warp < CUTTERS + ISSUERS) {
        // Issuer q takes the q-th and the (q + 2)-th 16 terms of every panel; the whole warp walks along, so that the descriptors are the same in
        // all lanes, and one lane issues.
        const uint32_t idesc = umma_idesc(TOK);
        const int q = __shfl_sync(0xffffffffu, warp, 0) - CUTTERS;
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), mem0 = __shfl_sync(0xffffffffu, base, 0);
        int stage = 0, buf = q, last = -1;
        uint32_t parity = 0, free_parity = 1, last_parity = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
            for (int k0 = 0; k0 < K; k0 += PANEL) {
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[stage]), parity, err, true) &&
                                                 mbar_wait(smem_u32(&s_free[buf]), free_parity, err, true));
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tm + (uint32_t)(S::SUMS + buf * S::BUF), sa = mem0 + S::RAWS * S::RAW + stage * S::STAGE + q * TERMS;
                const uint32_t w0 = tm + (uint32_t)(stage * S::W_COLS + q * (TERMS / 4)), w1 = w0 + PANEL / 2, w2 = w0 + PANEL;
                const uint64_t a0 = umma_desc(sa), a1 = umma_desc(sa + S::A_BYTES), a2 = umma_desc(sa + 2 * S::A_BYTES);
                if (elect_one()) {                                // 16 terms are 8 columns and 32 bytes of a row, the next 16 of the issuer's twice that further
                    const uint32_t small = d + TOK;
                    umma_bf16_ta(small, w2, a0, idesc, 0u);
                    umma_bf16_ta(small, w0, a2, idesc, 1u);
                    umma_bf16_ta(small, w1, a1, idesc, 1u);
                    umma_bf16_ta(small, w2 + 16, a0 + 4, idesc, 1u);
                    umma_bf16_ta(small, w0 + 16, a2 + 4, idesc, 1u);
                    umma_bf16_ta(small, w1 + 16, a1 + 4, idesc, 1u);
                    umma_bf16_ta_scaled<8>(small, w1, a0, idesc);
                    umma_bf16_ta(small, w0, a1, idesc, 1u);
                    umma_bf16_ta(small, w1 + 16, a0 + 4, idesc, 1u);
                    umma_bf16_ta(small, w0 + 16, a1 + 4, idesc, 1u);
                    umma_bf16_ta(d, w0, a0, idesc, 0u);
                    umma_bf16_ta(d, w0 + 16, a0 + 4, idesc, 1u);
                    umma_commit(smem_u32(&s_sum[buf]));
                    umma_commit(smem_u32(&s_empty[stage]));
                }
                __syncwarp();
                last = stage, last_parity = parity;
                buf += ISSUERS;
                if (buf >= S::BUFS) {
                    buf = q;
                    free_parity ^= 1;
                }
                if (++stage == S::STAGES) {
                    stage = 0;
                    parity ^= 1;
                }
            }
        // (the last arrivals must find the block still there)
        if (last >= 0 && ok) mbar_wait(smem_u32(&s_empty[last]), last_parity, err);
        __syncwarp();
    } else if (warp < CUTTERS + ISSUERS + S::ADDERS) {
        const int quarter = warp & 3;                             // (the quarter of tensor memory's lanes that a warp of this number may read)
        const int c0 = (warp - CUTTERS - ISSUERS) / 4 * S::WIDTH, steps = panels * ISSUERS;
        int buf = 0;
        uint32_t parity = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            float acc[S::WIDTH];
#pragma unroll
            for (int i = 0; i < S::WIDTH; ++i) acc[i] = 0.f;
            for (int s = 0; s < steps; ++s) {
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&s_sum[buf]), parity, err, true));
                if (!ok) break;
                tc_fence_after();
                const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(S::SUMS + buf * S::BUF + c0);
#pragma unroll
                for (int c = 0; c < S::WIDTH; c += S::AT_ONCE) {
                    uint32_t large[S::AT_ONCE], small[S::AT_ONCE];
                    tmem_ld_nowait(from + c, large);
                    tmem_ld_nowait(from + TOK + c, small);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < S::AT_ONCE; ++i) acc[c + i] += fmaf(__uint_as_float(small[i]), 0x1p-8f, __uint_as_float(large[i]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&s_free[buf]));
                if (++buf == S::BUFS) {
                    buf = 0;
                    parity ^= 1;
                }
            }
            const int n = tile / across * height + quarter * 32 + lane, m0 = tile % across * TOK + c0;
            if (ok && n < N && quarter * 32 + lane < height) {
#pragma unroll
                for (int i = 0; i < S::WIDTH; ++i)
                    if (m0 + i < M) {
                        float v = acc[i];
                        if (!(fabsf(v) <= 3.402823466e38f)) v = term_by_term(a + (size_t)(m0 + i) * K, w + (size_t)n * K, K);
                        out[(size_t)(m0 + i) * N + n] = v;
                    }
            }
        }
    } else if (BY_TMA && lane == 0) {
        int raw = 0, issued = 0;
        uint32_t parity = 1;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const int n0 = tile / across * height, m0 = tile % across * TOK;
            for (int k0 = 0; k0 < K; k0 += PANEL) {
                ok = mbar_wait(smem_u32(&s_read[raw]), parity, err, true);
                if (!ok) break;
                const uint32_t dst = base + raw * S::RAW, bar = smem_u32(&s_raw[raw]);
                mbar_expect_tx(bar, (height + TOK) * PANEL * 4);  // (what lies outside an operand arrives as zeros)
                for (int h = 0; h < 2; ++h) {
                    tma_load_2d(dst + h * (TILE_W * 128), &map_w, k0 + h * HALF, n0, bar);
                    tma_load_2d(dst + TILE_W * PANEL * 4 + h * (TOK * 128), &map_a, k0 + h * HALF, m0, bar);
                }
                ++issued;
                if (++raw == S::RAWS) {
                    raw = 0;
                    parity ^= 1;
                }
            }
        }
        for (int back = min(issued, S::RAWS); back > 0; --back) { // no copy may land after the block has left
            const int i = raw >= back ? raw - back : raw - back + S::RAWS;
            mbar_wait(smem_u32(&s_raw[i]), raw >= back ? parity ^ 1 : parity, err, true);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free(tmem, 512);
}

int processors() {
    int device = 0, n = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    return n;
}

// rows of K floats through boxes of `box_rows` x HALF with the 128-byte swizzle, what lies outside as zeros
bool rows_map(CUtensorMap* map, const float* p, int rows, int K, int box_rows) {
    const EncodeTiledFn fn = encode_fn();
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {HALF, (cuuint32_t)box_rows}, ones[2] = {1, 1};
    return fn && fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(p), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TOK, bool BY_TMA>
int launch(float* out, const float* a, const float* w, int M, int N, int K, int height, int* err, int sms, cudaStream_t stream) {
    const cudaError_t rc = cudaFuncSetAttribute(gemm_f32_tc_kernel<TOK, BY_TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<TOK>::SMEM);
    if (rc != cudaSuccess) return (int)rc;
    CUtensorMap map_w = {}, map_a = {};
    if (BY_TMA && !(rows_map(&map_w, w, N, K, height) && rows_map(&map_a, a, M, K, TOK))) return (int)cudaErrorInvalidValue;
    const long long tiles = (long long)((N + height - 1) / height) * ((M + TOK - 1) / TOK);
    if (tiles > 0x7fffffffLL - sms) return (int)cudaErrorInvalidValue;
    return xb_launch(gemm_f32_tc_kernel<TOK, BY_TMA>, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(Shape<TOK>::THREADS), Shape<TOK>::SMEM, stream, map_w,
                     map_a, out, a, w, M, N, K, height, err);
}

}  // namespace

int xb_gemm_f32_tc(float* out, const float* a, const float* w, int M, int N, int K, int* err, cudaStream_t stream) {
    const int sms = processors();
    if (sms < 1) return (int)cudaErrorInvalidDevice;
    const bool by_tma = K % 4 == 0 && !(((uintptr_t)a | (uintptr_t)w) & 15);
    // tokens of a tile: what takes the fewest rounds of blocks, a round taken to cost 1 at 16 tokens, 1.15 at 32 and
    // 1.5 at 64 (48 panels: 38.9, 45.1 and 57.4 us; 128 with all processors at work: 98, 111 and 143)
    auto cost = [&](int tok, float round) {
        const long long tiles = (long long)((N + TILE_W - 1) / TILE_W) * ((M + tok - 1) / tok);
        return (float)((tiles + sms - 1) / sms) * round;
    };
    const float c16 = cost(16, 1.f), c32 = cost(32, 1.15f), c64 = cost(64, 1.5f);
    // rows of W of a tile: as few as the number of rounds allows, so that the last round has work for every processor
    // (one row of 24,576 x 4,096, 192 tiles of 128 rows or 280 of 88: 111 and 98 us)
    auto height = [&](int tok) {
        const long long across = (M + tok - 1) / tok, rounds = ((long long)((N + TILE_W - 1) / TILE_W) * across + sms - 1) / sms, most = rounds * sms / across;
        const int rows = (int)((N + most - 1) / most);
        return rows <= 32 ? 32 : (rows + 7) / 8 * 8;
    };
#define XB_GF(TOK) (by_tma ? launch<TOK, true>(out, a, w, M, N, K, height(TOK), err, sms, stream) : launch<TOK, false>(out, a, w, M, N, K, height(TOK), err, sms, stream))
    if (c16 <= c32 && c16 <= c64) return XB_GF(16);
    if (c32 <= c64) return XB_GF(32);
    return XB_GF(64);
#undef XB_GF
}
