// Attention of prompt portions over a cached latent, with the keys and values of every head formed for the step.
//
// A cached row [c | k_r] stands for the keys k_h = [W_uk,h c | k_r] and values v_h = W_uv,h c of all heads.  Working on
// the rows themselves (latent_attention_mma.cu) costs 2 (2 rank + rot) operations per head, query and key; on the
// heads' own keys and values it is 2 (d + rot + dv): 640 against 2,176 at rank 512, d = dv = 128, rot 64.  Forming them
// costs 2 rank (d + dv) per head and key, once for all queries of the step, so it pays from a few dozen queries on.
// The tensor cores bound the kernel at long prompts, the exponentials of the softmax beside them.  It replaces the
// mma.sync kernel over the rows for portions of more than four tokens: at rank 512, 32 heads and a prompt of 2,048
// tokens 1,570 us (91 TFLOP/s) before, now 55 us for the attention where the product has just left keys and values in the L2
// cache (782 TFLOP/s of its 43 GFLOP; 66 us after a flush), 18 us for the product that forms them and 4 us for the gathering,
// without the 33 us of maps into and out of the latent space; at rank 256 and 16 heads 626 us before, 37 + 9 us now (47 us
// after a flush).
//
//   latent_gather_kernel   the rows a step's portions can see, out of their pages, in runs of 64 rows per portion that
//                          begin at a multiple of 64 positions; rows no query of the portion sees are zeros.  The matrix
//                          product [rows, rank] x [W_uk | W_uv] then gives all keys and values, token-major.
//   attn_rows_tc_kernel    128 or 256 queries of one head per work item against that head's keys and values: tcgen05.mma
//                          with scores, probabilities and accumulators in tensor memory, TMA-fed rings, one softmax row
//                          per thread.  Two tiles of 128 queries share every key/value tile.
//
// A cached row whose latent holds an infinity or no number must not reach queries that do not see it (a weight of 0 times its
// values would): the gathering kernel leaves zeros in its place and marks it, and the attention makes the result of every query
// that sees it no number.
#include "attention_common.cuh"
#include "tc_common.cuh"

namespace {

using namespace xbtc;

constexpr int QT = 128, KT = 64;
constexpr int STAGES = 3;
constexpr int THREADS = 384;
constexpr int ITEM_INTS = 4;            // portion, first query of it, head | tiles << 16, row of the position 0
constexpr float RESCALE_STEP = 8.f;     // the row maximum moves only when it grows by more than 2^8

struct Item {
    int h, nt, t0, p0, row0;            // head, query tiles, first row of q / out, its position, row of position 0
    int rows[2], lo[2], hi[2];          // of each query tile: queries, first and last key tile
};

__device__ __forceinline__ Item item_of(const int* __restrict__ it, const int* __restrict__ q_start,
                                        const int* __restrict__ start_pos, int window) {
    Item w;
    const int b = it[0], first = it[1];
    w.h = it[2] & 0xffff;
    w.nt = (it[2] >> 16) == 2 ? 2 : 1;
    w.row0 = it[3];
    const int n = q_start[b + 1] - q_start[b];
    w.t0 = q_start[b] + first;
    w.p0 = start_pos[b] + first;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        w.rows[i] = max(0, min(QT, n - first - i * QT));
        const int p = w.p0 + i * QT;
        w.lo[i] = first_visible(p, window) / KT;
        w.hi[i] = (p + w.rows[i] - 1) / KT;
    }
    return w;
}

// One warp per row of the gathered buffer, eight rows a block.  blocks: (portion, first position) of every run of 64 rows.  `bad`
// (a bit per row): rows whose first `checked` pieces hold something that is not finite; they are gathered as zeros.
__global__ void latent_gather_kernel(uint4* __restrict__ out, const uint4* pages, const int* __restrict__ blocks,
                                     int rows, const int* __restrict__ q_start, const int* __restrict__ start_pos,
                                     const int* __restrict__ table, int table_stride, int page_size, int num_pages, int window,
                                     int pieces, int checked, unsigned char* bad, int* err) {
    pdl_overlap_few();
    __shared__ int s_off[8];
    const int warp = threadIdx.x >> 5, row = blockIdx.x * 8 + warp, lane = threadIdx.x & 31;      // rows: a multiple of 64
    const int b = blocks[2 * (row >> 6)], j = blocks[2 * (row >> 6) + 1] + (row & 63);
    const int start = start_pos[b], end = start + q_start[b + 1] - q_start[b];
    const uint4* src = nullptr;
    if (j >= first_visible(start, window) && j < end) {
        const int page = table[(size_t)b * table_stride + j / page_size];
        if (page < 0 || page >= num_pages) {
            if (lane == 0) atomicOr(err, XB_ERR_BAD_PAGE);
        } else {
            src = pages + ((size_t)page * page_size + j % page_size) * pieces;
        }
    }
    bool off = false;
    if (bad != nullptr && src != nullptr)
        for (int c = lane; c < checked; c += 32) off |= bf16_not_finite(src[c]);
    if (__any_sync(0xffffffffu, off)) src = nullptr, off = true;
    for (int c = lane; c < pieces; c += 32) out[(size_t)row * pieces + c] = src ? src[c] : make_uint4(0, 0, 0, 0);
    if (bad != nullptr) {
        if (lane == 0) s_off[warp] = off ? 1 << warp : 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            int bits = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) bits |= s_off[i];
            bad[blockIdx.x] = (unsigned char)bits;
        }
    }
}

// NKC: 64-channel pieces of a key (the last one is the part all heads share when TAIL), DVC: of a value.
// Roles as in the prefill kernel over pages: warps 0..3 and 4..7 softmax of the two query tiles, warp 8 loads keys,
// warp 10 values, warp 9 loads queries and issues S = Q K^T, warp 11 issues O += P V.
// Shared memory: Q [2][NKC][128][64], STAGES x (K [NKC][64][64], V [DVC][64][64]), all 128-byte swizzled; barriers.
// Tensor memory: S of tile 0 at 0 and 64, of tile 1 at 128 and 192; O at 256 and 384.
template <int NKC, int DVC, bool TAIL>
__global__ void __launch_bounds__(THREADS)
attn_rows_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                    const __grid_constant__ CUtensorMap map_tail, __nv_bfloat16* __restrict__ out, long long ldo,
                    const int* __restrict__ q_start, const int* __restrict__ start_pos, int nh, int rank, int window,
                    float scale_log2, const float* __restrict__ sink, const int* __restrict__ work, const unsigned long long* bad,
                    int* err) {
    constexpr int D = 64 * (NKC - (TAIL ? 1 : 0)), DV = 64 * DVC;
    constexpr uint32_t Q_ONE = NKC * QT * 128, Q_BYTES = 2 * Q_ONE;
    constexpr uint32_t PIECE = KT * 128, K_BYTES = NKC * PIECE, STAGE_BYTES = (NKC + DVC) * PIECE;
    constexpr uint32_t BAR_OFF = Q_BYTES + STAGES * STAGE_BYTES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = smem_u32(smem_raw), q_sm = base, kv_sm = base + Q_BYTES, bars = base + BAR_OFF;
    const uint32_t k_full0 = bars, k_empty0 = bars + 32, v_full0 = bars + 64, v_empty0 = bars + 96;
    const uint32_t s_ready0 = bars + 128, pv_done0 = bars + 160, p_ready0 = bars + 192, o_done0 = bars + 208;
    const uint32_t q_full = bars + 224, q_empty = bars + 232;
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem_raw + BAR_OFF + 240);   // where tensor memory begins
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int ctas = (int)gridDim.x;
    const int item_begin = work[blockIdx.x];
    int item_end = work[blockIdx.x + 1];
    const int* const items = work + ctas + 1;
    if (threadIdx.x == 0) {
        if (base & 1023u) atomicOr(err, XB_ERR_WAIT);
        for (int i = 0; i < 16; ++i) mbar_init(bars + 8 * i, 1);            // k_full, k_empty, v_full, v_empty
        for (int i = 0; i < 4; ++i) {
            mbar_init(s_ready0 + 8 * i, 1);
            mbar_init(pv_done0 + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(p_ready0 + 8 * i, 128);
            mbar_init(o_done0 + 8 * i, 1);
        }
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        mbar_init_fence();
    }
    if (*reinterpret_cast<volatile int*>(err) & XB_ERR_WAIT) item_end = item_begin;   // an earlier CTA gave up
    __syncthreads();
    if (item_end <= item_begin || (base & 1023u)) {
        pdl_launch_dependents();
        pdl_wait();
        return;
    }
    if (warp == 0) tmem_alloc(const_cast<uint32_t*>(&words[0]), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = words[0];
    pdl_launch_dependents();    // only now: see pdl_launch_dependents on tensor memory
    pdl_wait();

    auto item_at = [&](int k) { return item_of(items + (size_t)k * ITEM_INTS, q_start, start_pos, window); };
    if (warp == 8 || warp == 10) {
        // ---- producers of keys (warp 8) and values (warp 10): one lane per 64-channel piece of a tile
        const bool is_v = warp == 10;
        const uint32_t full0 = is_v ? v_full0 : k_full0, empty0 = is_v ? v_empty0 : k_empty0;
        const int pieces = is_v ? DVC : NKC;
        int s = 0;
        uint32_t ph = 0;
        bool rounds = false, ok = true;
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            const int last = w.nt == 2 ? w.hi[1] : w.hi[0];
            for (int kt = w.lo[0]; kt <= last; ++kt) {
                if (rounds && !__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1u, err))) {
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_expect_tx(full0 + 8 * s, pieces * PIECE);
                __syncwarp();
                if (lane < pieces) {
                    const uint32_t dst = kv_sm + s * STAGE_BYTES + (is_v ? K_BYTES : 0u) + lane * PIECE;
                    const int y = w.row0 + kt * KT;
                    if (is_v) tma_load_2d(dst, &map_kv, nh * D + w.h * DV + lane * 64, y, full0 + 8 * s);
                    else if (TAIL && lane == NKC - 1) tma_load_2d(dst, &map_tail, rank, y, full0 + 8 * s);
                    else tma_load_2d(dst, &map_kv, w.h * D + lane * 64, y, full0 + 8 * s);
                }
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                    rounds = true;
                }
            }
        }
    } else if (warp == 9) {
        // ---- queries and S = Q K^T of both tiles
        const bool leader = lane == 0;
        const uint32_t idesc = umma_idesc(KT, 0);
        const uint64_t dq0 = umma_desc(q_sm, 16, 1024), dk0 = umma_desc(kv_sm, 16, 1024);
        auto load_q = [&](const Item& w) {
            if (leader) {
                mbar_expect_tx(q_full, (uint32_t)w.nt * Q_ONE);
                for (int i = 0; i < w.nt; ++i)
#pragma unroll
                    for (int c = 0; c < NKC; ++c)
                        tma_load_3d(q_sm + i * Q_ONE + c * QT * 128, &map_q, c * 64, w.h, w.t0 + i * QT, q_full);
            }
            __syncwarp();
        };
        int s = 0, Th[2] = {0, 0};
        uint32_t ph = 0;
        bool ok = true;
        Item w = item_at(item_begin);
        load_q(w);
        for (int k = item_begin; k < item_end && ok; ++k) {
            ok = __all_sync(0xffffffffu, mbar_wait(q_full, (uint32_t)(k - item_begin) & 1u, err, true));
            const int last = w.nt == 2 ? w.hi[1] : w.hi[0];
            for (int kt = w.lo[0]; kt <= last && ok; ++kt) {
                ok = __all_sync(0xffffffffu, mbar_wait(k_full0 + 8 * s, ph, err, true));
                const uint64_t dk = dk0 + (uint64_t)((s * STAGE_BYTES) >> 4);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (!ok || i >= w.nt || kt < w.lo[i] || kt > w.hi[i]) continue;
                    const int th = Th[i]++, sb = th & 1;
                    // this buffer held the scores and then P of the tile's key tile th - 2: that P V must have read it
                    ok = th < 2 || __all_sync(0xffffffffu, mbar_wait(pv_done0 + 8 * (2 * i + sb), ((th >> 1) - 1) & 1, err, true));
                    if (!ok) continue;
                    tc_fence_after();
                    const uint64_t dq = dq0 + (uint64_t)((i * Q_ONE) >> 4);
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < NKC * 4; ++kk) {
                            const uint32_t off = (kk >> 2), inner = (kk & 3) * 32;
                            umma_bf16(tmem + (uint32_t)(i * 128 + sb * 64), dq + (uint64_t)((off * QT * 128 + inner) >> 4),
                                      dk + (uint64_t)((off * PIECE + inner) >> 4), idesc, kk ? 1u : 0u);
                        }
                        umma_commit(s_ready0 + 8 * (2 * i + sb));
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (leader) umma_commit(k_empty0 + 8 * s);
                __syncwarp();
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (ok && k + 1 < item_end) {
                // the next item's queries go where these lie, once every product that reads them has completed
                if (leader) umma_commit(q_empty);
                __syncwarp();
                ok = __all_sync(0xffffffffu, mbar_wait(q_empty, (uint32_t)(k - item_begin) & 1u, err, true));
                if (ok) {
                    w = item_at(k + 1);
                    load_q(w);
                }
            }
        }
    } else if (warp == 11) {
        // ---- O += P V of both tiles: P in tensor memory over the scores it came from, V MN-major
        const bool leader = lane == 0;
        const uint32_t idesc = umma_idesc(DV, 1);
        const uint64_t dv0 = umma_desc(kv_sm + K_BYTES, PIECE, 1024);
        int s = 0, Th[2] = {0, 0};
        uint32_t ph = 0;
        bool ok = true;
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            const int last = w.nt == 2 ? w.hi[1] : w.hi[0];
            for (int kt = w.lo[0]; kt <= last && ok; ++kt) {
                ok = __all_sync(0xffffffffu, mbar_wait(v_full0 + 8 * s, ph, err, true));
                const uint64_t dv = dv0 + (uint64_t)((s * STAGE_BYTES) >> 4);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (!ok || i >= w.nt || kt < w.lo[i] || kt > w.hi[i]) continue;
                    const int th = Th[i]++, sb = th & 1;
                    ok = __all_sync(0xffffffffu, mbar_wait(p_ready0 + 8 * i, th & 1, err, true));
                    if (!ok) continue;
                    tc_fence_after();
                    const uint32_t tp = tmem + (uint32_t)(i * 128 + sb * 64);
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < KT / 16; ++kk)
                            umma_bf16_ta(tmem + (uint32_t)(256 + i * 128), tp + (uint32_t)(kk * 8), dv + (uint64_t)((kk * 2048) >> 4),
                                         idesc, (kt > w.lo[i] || kk) ? 1u : 0u);
                        umma_commit(pv_done0 + 8 * (2 * i + sb));
                        if (kt == w.hi[i]) umma_commit(o_done0 + 8 * i);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (leader) umma_commit(v_empty0 + 8 * s);
                __syncwarp();
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp < 8) {
        // ---- softmax: one query per thread
        const int i = warp >> 2, r = (int)threadIdx.x & 127;
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tmem_s = tmem + (uint32_t)(i * 128) + lane_addr, tmem_o = tmem + (uint32_t)(256 + i * 128) + lane_addr;
        const uint32_t my_s_ready = s_ready0 + 16 * i, my_p_ready = p_ready0 + 8 * i, my_pv_done = pv_done0 + 16 * i;
        int th = 0, done = 0;
        bool alive = true;
        for (int k = item_begin; k < item_end && alive; ++k) {
            const Item w = item_at(k);
            if (i >= w.nt) continue;    // an item of one tile: the second warpgroup sits it out
            const int rows = i ? w.rows[1] : w.rows[0], lo = i ? w.lo[1] : w.lo[0], hi = i ? w.hi[1] : w.hi[0];
            const int p_first = w.p0 + i * QT, my_pos = p_first + r, last_key = p_first + rows - 1;
            const int my_lo = first_visible(my_pos, window), edge_lo = first_visible(p_first + QT - 1, window);
            float m_ref = -INFINITY, l = 0.f;
            for (int kt = lo; kt <= hi; ++kt, ++th) {
                const int sb = th & 1, key0 = kt * KT;
                const unsigned long long off = bad != nullptr ? bad[(w.row0 + key0) / KT] : 0ull;
                if (!__all_sync(0xffffffffu, mbar_wait(my_s_ready + 8 * sb, (th >> 1) & 1, err))) {
                    alive = false;
                    break;
                }
                tc_fence_after();
                float sc[64];
                {
                    uint32_t ra[32], rb[32];
                    tmem_ld32_nowait(tmem_s + sb * 64, ra);
                    tmem_ld32_nowait(tmem_s + sb * 64 + 32, rb);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        sc[c] = __uint_as_float(ra[c]);
                        sc[32 + c] = __uint_as_float(rb[c]);
                    }
                }
                if (key0 + KT - 1 > p_first || key0 + KT - 1 > last_key || key0 < edge_lo) {
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        const int j = key0 + c;
                        sc[c] = (j <= my_pos && j <= last_key && j >= my_lo) ? sc[c] : -INFINITY;
                    }
                }
                if (off != 0ull) {      // (rare) rows of the tile that were not finite: no number for the queries that see them
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        const int j = key0 + c;
                        if (((off >> c) & 1ull) && j <= my_pos && j <= last_key && j >= my_lo) sc[c] = NAN;
                    }
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 64; c += 8) {
                    mx4[0] = max3(mx4[0], sc[c], sc[c + 1]);
                    mx4[1] = max3(mx4[1], sc[c + 2], sc[c + 3]);
                    mx4[2] = max3(mx4[2], sc[c + 4], sc[c + 5]);
                    mx4[3] = max3(mx4[3], sc[c + 6], sc[c + 7]);
                }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
                float corr = 1.f;
                int moved = 0;
                if (mx > m_ref + RESCALE_STEP) {
                    corr = m_ref == -INFINITY ? 0.f : ex2(m_ref - mx);
                    m_ref = mx;
                    moved = kt > lo;
                }
                const float m_neg = m_ref == -INFINITY ? 0.f : -m_ref;
                const f32x2 scale2 = pack2(scale_log2, scale_log2), mneg2 = pack2(m_neg, m_neg);
                f32x2 sum_a = pack2(0.f, 0.f), sum_b = pack2(0.f, 0.f);
                uint32_t pk[32];
#pragma unroll
                for (int c8 = 0; c8 < 8; ++c8) {
                    float x[8], e[8];
#pragma unroll
                    for (int c = 0; c < 8; c += 2)
                        unpack2(fma2(pack2(sc[c8 * 8 + c], sc[c8 * 8 + c + 1]), scale2, mneg2), x[c], x[c + 1]);
#pragma unroll
                    for (int c = 0; c < 8; ++c) e[c] = ex2(x[c]);
                    sum_a = add2(sum_a, add2(pack2(e[0], e[1]), pack2(e[2], e[3])));
                    sum_b = add2(sum_b, add2(pack2(e[4], e[5]), pack2(e[6], e[7])));
                    pk[c8 * 4] = pack_bf16(e[0], e[1]);
                    pk[c8 * 4 + 1] = pack_bf16(e[2], e[3]);
                    pk[c8 * 4 + 2] = pack_bf16(e[4], e[5]);
                    pk[c8 * 4 + 3] = pack_bf16(e[6], e[7]);
                }
                float s0, s1, s2, s3;
                unpack2(sum_a, s0, s1);
                unpack2(sum_b, s2, s3);
                l = l * corr + ((s0 + s1) + (s2 + s3));
                tmem_st32_u(tmem_s + sb * 64, pk);
                // the product before must be complete before O is touched, and before this tile is announced: the issuer
                // waits for the announcements by their parity, so a tile must never be two of them ahead of it
                if (kt > lo && !__all_sync(0xffffffffu, mbar_wait(my_pv_done + 8 * (sb ^ 1), ((th - 1) >> 1) & 1, err))) {
                    alive = false;
                    break;
                }
                if (__any_sync(0xffffffffu, moved)) {
                    tc_fence_after();
                    const float f = moved ? corr : 1.f;
#pragma unroll
                    for (int c0 = 0; c0 < DV; c0 += 32) {
                        float o[32];
                        tmem_ld32(tmem_o + c0, o);
#pragma unroll
                        for (int c = 0; c < 32; ++c) o[c] *= f;
                        tmem_st32(tmem_o + c0, o);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(my_p_ready);
            }
            if (alive) alive = mbar_wait(o_done0 + 8 * i, (uint32_t)done & 1u, err);
            ++done;
            alive = __all_sync(0xffffffffu, alive);
            tc_fence_after();
            if (sink != nullptr) l += exp2f(fmaf(sink[w.h], 1.4426950408889634f, -m_ref));
            const float inv = l > 0.f ? 1.f / l : 0.f;
            if (alive) {
                __nv_bfloat16* dst = out + (size_t)(w.t0 + i * QT + r) * ldo + (size_t)w.h * DV;
#pragma unroll
                for (int c0 = 0; c0 < DV; c0 += 32) {
                    float o[32];
                    tmem_ld32(tmem_o + c0, o);      // warp-wide, whatever the row
                    if (r < rows) {
#pragma unroll
                        for (int c8 = 0; c8 < 4; ++c8) {
                            uint4 v;
                            v.x = pack_bf16(o[c8 * 8] * inv, o[c8 * 8 + 1] * inv);
                            v.y = pack_bf16(o[c8 * 8 + 2] * inv, o[c8 * 8 + 3] * inv);
                            v.z = pack_bf16(o[c8 * 8 + 4] * inv, o[c8 * 8 + 5] * inv);
                            v.w = pack_bf16(o[c8 * 8 + 6] * inv, o[c8 * 8 + 7] * inv);
                            *reinterpret_cast<uint4*>(dst + c0 + c8 * 8) = v;
                        }
                    }
                }
            }
            // these reads of O come before this tile's next announcement, and so before the product that overwrites it
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

template <int NKC, int DVC, bool TAIL>
int launch(const CUtensorMap& mq, const CUtensorMap& mkv, const CUtensorMap& mt, void* out, long long ldo, const int* q_start,
           const int* start_pos, int nh, int rank, int window, float sl2, const float* sink, const int* work, int ctas,
           const unsigned long long* bad, int* err, cudaStream_t stream) {
    constexpr size_t smem = (size_t)2 * NKC * QT * 128 + (size_t)STAGES * (NKC + DVC) * KT * 128 + 1024;
    const auto kernel = attn_rows_tc_kernel<NKC, DVC, TAIL>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return xb_launch(kernel, dim3(ctas), dim3(THREADS), smem, stream, mq, mkv, mt, (__nv_bfloat16*)out, ldo, q_start, start_pos,
                     nh, rank, window, sl2, sink, work, bad, err);
}

}  // namespace

// Rows of `width` bfloat16 (a multiple of 8) from their pages [pages, page_size, width] into out [rows, width], rows a
// multiple of 64: run i of 64 rows holds portion blocks[2 i]'s positions from blocks[2 i + 1] on.  `bad` (rows / 8 bytes, or none):
// see latent_gather_kernel; `rank` channels are looked at.
XB_EXPORT int xb_latent_gather(void* out, const void* pages, const int* blocks, int rows, const int* q_start,
                               const int* start_pos, const int* table, int table_stride, int page_size, int num_pages,
                               int window, int width, int rank, void* bad, int* err, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (width % 8 || rows % 64 || page_size <= 0 || window < 0 || rank % 8 || rank < 0 || rank > width) return (int)cudaErrorInvalidValue;
    xb_launch_few(latent_gather_kernel, dim3(rows / 8), dim3(256), 0, stream, (uint4*)out, (const uint4*)pages, blocks, rows, q_start, start_pos,
                  table, table_stride, page_size, num_pages, window, width / 8, rank / 8, (unsigned char*)bad, err);
    return xb_launch_status();
}

// Whether xb_attn_rows_tc takes these sizes: key channels of a head's own (d) and shared by all heads (rd), value channels.
XB_EXPORT int xb_attn_rows_tc_takes(int d, int rd, int dv, int rank) {
    return (d == 64 || d == 128) && (dv == 64 || dv == 128) && rd >= 0 && rd <= 64 && rd % 8 == 0 && rank > 0 && rank % 8 == 0;
}

// q: head h of token t at q + t * q_ts + h * (d + rd) [d + rd]; kv [rows, nh * (d + dv)]: all heads' keys, then all
// heads' values; tail [rows, width]: channels rank .. rank + rd - 1 are the key part all heads share; out: head h of
// token t at out + t * ldo + h * dv.  `work` comes from xb_latent_prefill_work (host library) for the same step, heads
// and window; `bad` from xb_latent_gather (or none).  Returns cudaErrorNotSupported, having done nothing, for sizes or strides it does not take.
XB_EXPORT int xb_attn_rows_tc(void* out, long long ldo, const void* q, long long q_ts, const void* kv, const void* tail,
                              int tokens, int rows, int nh, int d, int rd, int dv, int rank, int width, const int* q_start,
                              const int* start_pos, int window, float scale, const float* sink, const int* work, int ctas,
                              const void* bad, int* err, cudaStream_t stream) {
    if (ctas <= 0) return 0;
    if (!xb_attn_rows_tc_takes(d, rd, dv, rank) || nh <= 0 || nh > 65535 || q_ts % 8 || width % 8 || width < rank + rd || ldo % 8 ||
        rows % 64 || window < 0 || (((uintptr_t)out | (uintptr_t)q | (uintptr_t)kv | (uintptr_t)tail) & 15) || ((uintptr_t)bad & 7))
        return (int)cudaErrorNotSupported;
    CUtensorMap mq, mkv, mt;
    const long long qd[3] = {d + rd, nh, tokens}, qs[2] = {d + rd, q_ts};
    const int qb[3] = {64, 1, QT};
    // the shared key part ends at rank + rd: what a box asks for beyond it reads as zero
    const long long td[2] = {rank + rd, rows}, ts[1] = {width};
    const int tb[2] = {64, KT};
    if (!tensor_map_bf16(&mq, q, 3, qd, qs, qb) || !tensor_map_2d(&mkv, kv, rows, (long long)nh * (d + dv), KT) ||
        !tensor_map_bf16(&mt, tail, 2, td, ts, tb))
        return (int)cudaErrorNotSupported;
    const float sl2 = scale * 1.4426950408889634f;
#define XB_GO(N, V, T) return launch<N, V, T>(mq, mkv, mt, out, ldo, q_start, start_pos, nh, rank, window, sl2, sink, work, ctas, (const unsigned long long*)bad, err, stream)
    if (d == 128) {
        if (dv == 128) { if (rd) XB_GO(3, 2, true); else XB_GO(2, 2, false); }
        if (rd) XB_GO(3, 1, true); else XB_GO(2, 1, false);
    }
    if (dv == 128) { if (rd) XB_GO(2, 2, true); else XB_GO(1, 2, false); }
    if (rd) XB_GO(2, 1, true); else XB_GO(1, 1, false);
#undef XB_GO
}
