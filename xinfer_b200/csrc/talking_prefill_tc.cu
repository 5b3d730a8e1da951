// Attention with talking heads for steps of many tokens, on the 5th-generation tensor cores (the arithmetic is described
// in talking_attention.cu).  Every head's score of a (query, key) pair enters every head's softmax, so no head can be
// worked on alone; a block that keeps the scores, the accumulators and the rows of all heads together has room for 16
// queries only, and its steps - products, mix, softmax, value sums - wait for one another (talking_attention_mma.cu:
// 1,890 us for a prompt of 2,048 tokens and 32 heads, 29 us for 16 queries x 32 keys x 32 heads).  Here the step is cut
// where the heads part again:
//
//   talk_scores_tc_kernel   raw scores of all heads by tcgen05.mma into tensor memory, mixed in float32 on the FMA units,
//                           written as float32 tiles of 128 queries x 32 keys per head.  Bound by the mix: heads^2
//                           multiply-adds per pair, 4.3 GFLOP at 2,048 tokens and 32 heads, 58 us at the FMA units' rate.
//   talk_values_tc_kernel   softmax rows over those tiles and O += P V by tcgen05.mma, two heads of a key/value head per
//                           work item.  Bound by reading the tiles: 4 bytes per pair and head, 280 MB at 2,048 tokens.
//
// 2,048 tokens: 1,890 us -> 135 + 64 us with 32 heads, 1,088 us -> 51 + 43 us with 16.
// What is rounded is what talking_attention_mma.cu rounds: the weights, once, in front of their product with the values, and it
// is the rounded ones that are summed; the mixed scores leave as float32.  Steps whose tiles would not fit the scratch memory run
// as several pairs of launches over fewer queries each.  A value that is not finite must not reach queries that do not see it (a
// weight of 0 times it would): in tiles that some query sees in part it is a 0 for the product, and is added to the results of the
// queries that see it.
#include "attention_common.cuh"
#include "tc_common.cuh"

namespace {

using namespace xbtc;

constexpr int QB_ROWS = 128;             // queries of a block of score tiles
constexpr int TILE_KEYS = 32;            // keys of a score tile
constexpr int TILE_FLOATS = QB_ROWS * TILE_KEYS;
constexpr int BLOCK_INTS = 6;            // portion, first query of it, first 32-key tile, 32-key tiles, first score tile, -
constexpr int ITEM_INTS = 4;
constexpr float RESCALE_STEP = 8.f;

struct TalkBlock {
    int b, first, kb0, nkb, rows, t0, p0;
    long long tile0;
};
__device__ __forceinline__ TalkBlock talk_block(const int* __restrict__ blk, const int* __restrict__ q_start, const int* __restrict__ start_pos) {
    TalkBlock w;
    w.b = blk[0];
    w.first = blk[1];
    w.kb0 = blk[2];
    w.nkb = blk[3];
    w.tile0 = blk[4];
    const int n = q_start[w.b + 1] - q_start[w.b];
    w.rows = min(QB_ROWS, n - w.first);
    w.t0 = q_start[w.b] + w.first;
    w.p0 = start_pos[w.b] + w.first;
    return w;
}

// 32x32b.xN: lane = row, registers = N columns
template <int N>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, float* v);
template <>
__device__ __forceinline__ void tmem_ld_cols<4>(uint32_t taddr, float* v) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_ld_cols<8>(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_ld_cols<16>(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---- scores -----------------------------------------------------------------------------------------------------------
// A work item is QN = 512 / heads queries of one block and a run of 128-key tiles.  Keys are the rows of the product (a
// lane of tensor memory each), (head, query) its columns: a tile fills all 512 of them, and a thread that owns a key finds
// all heads' raw scores of a query in its own lane.  The other way round (queries as rows) the queries would have to be
// loaded again for every 16 keys: 1 MB against 256 KB of keys.  The queries of all heads stay in shared memory (128 KB)
// for the whole item, the keys of one key/value head after the other come through two stages of 32 KB.
//   warps 0..7 mix (lane = key; warps 4..7 the second half of the queries): 128 raw scores of 128 / heads queries in
//   registers, packed by pairs of queries.  The matrix comes from shared memory, four entries per load, the next head's row
//   while this head's sums are formed: loads bound the mix otherwise (entries stored twice, as ready operands: 191 us per
//   launch at 2,048 tokens and 32 heads; once: 160 us; with the row loaded ahead, which takes 224 registers: 135 us; as
//   operands of the constant bank 296 us, though 64 against 72 us at 16 heads, where now it is 51 us).  The last raw
//   scores are in registers before they are mixed, so the next tile's products run meanwhile.
//   warp 8 loads queries and keys (one lane per page box), warp 9 issues the products.
constexpr int S_THREADS = 384;
// Registers: the launch gives each of the twelve warps 168; the mixing warpgroups take 224, the third keeps 56.
constexpr int S_MIX_REGS = 224, S_AUX_REGS = 56;
constexpr int S_KEYS = 128;

// The matrix, times the scale and log2(e).  It travels with the launch and is copied to shared memory, where the mix reads it.
template <int H>
struct TalkMatrix {
    float t[H * H];
};

template <int H, int HALVES /* 64-channel pieces of a key */>
struct ScoresSmem {
    static constexpr uint32_t Q_BYTES = 512 * HALVES * 128, K_STAGE = HALVES * S_KEYS * 128;
    static constexpr uint32_t TALK_OFF = Q_BYTES + 2 * K_STAGE, BAR_OFF = TALK_OFF + H * H * 4, TOTAL = BAR_OFF + 128;
};

template <int H, int HALVES>
__global__ void __launch_bounds__(S_THREADS, 1)
talk_scores_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      float* __restrict__ scores, const __grid_constant__ TalkMatrix<H> talk, const int* __restrict__ blocks,
                      const int* __restrict__ work, const int* __restrict__ q_start, const int* __restrict__ start_pos,
                      const int* __restrict__ block_table, int table_stride, int nkv, int ps, int ps_shift, int num_pages,
                      int window, int* err) {
    using L = ScoresSmem<H, HALVES>;
    constexpr int QN = 512 / H, QB = 128 / H;       // queries of an item; queries mixed at a time
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = smem_u32(smem_raw), k_sm = base + L::Q_BYTES, bars = base + L::BAR_OFF;
    const uint32_t k_full0 = bars, k_empty0 = bars + 16, d_full = bars + 32, d_empty = bars + 40, q_full = bars + 48, q_empty = bars + 56;
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem_raw + L::BAR_OFF + 64);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rep = H / nkv;
    const int ctas = (int)gridDim.x;
    const int item_begin = work[blockIdx.x];
    int item_end = work[blockIdx.x + 1];
    const int* const items = work + ctas + 1;
    if (threadIdx.x == 0) {
        if (base & 1023u) atomicOr(err, XB_ERR_WAIT);
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full0 + 8 * i, 1);
            mbar_init(k_empty0 + 8 * i, 1);
        }
        mbar_init(d_full, 1);
        mbar_init(d_empty, 8);
        mbar_init(q_full, 1);
        mbar_init(q_empty, 1);
        mbar_init_fence();
    }
    for (int i = threadIdx.x; i < H * H; i += S_THREADS) reinterpret_cast<float*>(smem_raw + L::TALK_OFF)[i] = talk.t[i];
    if (*reinterpret_cast<volatile int*>(err) & XB_ERR_WAIT) item_end = item_begin;
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
    pdl_wait();     // queries and new keys come from the kernel before; the tiles were read by the one before that

    if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S_MIX_REGS));
        // ---- the mix: lane = key
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        int tiles = 0;
        bool alive = true;
        for (int k = item_begin; k < item_end && alive; ++k) {
            const int* it = items + (size_t)k * ITEM_INTS;
            const TalkBlock w = talk_block(blocks + (size_t)it[0] * BLOCK_INTS, q_start, start_pos);
            const int first = it[1] * QN, rows = min(QN, w.rows - first), last_key = w.p0 + first + rows - 1;
            for (int kt = it[2]; kt < it[2] + it[3]; ++kt, ++tiles) {
                alive = __all_sync(0xffffffffu, mbar_wait(d_full, (uint32_t)tiles & 1u, err));
                if (!alive) break;
                tc_fence_after();
                const int kb = kt * 4 + quarter;                            // this warp's 32-key tile
                // queries of this half that exist, as long as any of them sees a key of the warp
                const int q_end = kb * 32 > last_key ? 0 : min(rows, (half + 1) * (QN / 2));
                float* tile = scores + (w.tile0 + (kb - w.kb0)) * TILE_FLOATS + (lane & 3);
                bool released = false;
                for (int q0 = half * (QN / 2); q0 < q_end; q0 += QB) {
                    float raw[H][QB];
#pragma unroll
                    for (int h = 0; h < H; ++h) tmem_ld_cols<QB>(tmem + lane_addr + (uint32_t)(h * QN + q0), raw[h]);
                    tmem_ld_wait();
                    if (q0 + QB >= q_end) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(d_empty);
                        released = true;
                    }
                    int dst[QB];
#pragma unroll
                    for (int q = 0; q < QB; ++q) {
                        const int r = first + q0 + q;
                        dst[q] = r * TILE_KEYS + (((lane >> 2) ^ (r & 7)) << 2);
                    }
                    float* to = tile;
                    // the row of the matrix for the next head is on its way while this head's sums are formed
                    const float4* row = reinterpret_cast<const float4*>(smem_raw + L::TALK_OFF);
                    float4 cur[H / 4], nxt[H / 4];
#pragma unroll
                    for (int i = 0; i < H / 4; ++i) cur[i] = row[i];
                    auto head = [&](const float4 (&c)[H / 4]) {
                        f32x2 acc[QB / 2];
#pragma unroll
                        for (int q = 0; q < QB / 2; ++q) acc[q] = pack2(0.f, 0.f);
#pragma unroll
                        for (int g = 0; g < H; ++g) {
                            const float4 v = c[g / 4];
                            const float f = (g & 3) == 0 ? v.x : (g & 3) == 1 ? v.y : (g & 3) == 2 ? v.z : v.w;
#pragma unroll
                            for (int q = 0; q < QB / 2; ++q)
                                acc[q] = fma2(pack2(f, f), pack2(raw[g][2 * q], raw[g][2 * q + 1]), acc[q]);
                        }
#pragma unroll
                        for (int q = 0; q < QB / 2; ++q) {      // 128 bytes of a tile's row per warp and store
                            float a, b;
                            unpack2(acc[q], a, b);
                            to[dst[2 * q]] = a;
                            to[dst[2 * q + 1]] = b;
                        }
                        to += (size_t)w.nkb * TILE_FLOATS;
                    };
#pragma unroll 1
                    for (int h = 0; h < H; h += 2) {
#pragma unroll
                        for (int i = 0; i < H / 4; ++i) nxt[i] = row[(h + 1) * (H / 4) + i];
                        head(cur);
                        const int h2 = h + 2 < H ? h + 2 : 0;
#pragma unroll
                        for (int i = 0; i < H / 4; ++i) cur[i] = row[h2 * (H / 4) + i];
                        head(nxt);
                    }
                }
                if (!released) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S_AUX_REGS));
        if (warp == 8) {
            // ---- queries and keys
            const int box_rows = ps < S_KEYS ? ps : S_KEYS, boxes = (S_KEYS / box_rows) * HALVES;   // at most 32
            const int bi = lane / HALVES, hf = lane % HALVES;
            int s = 0;
            uint32_t ph = 0;
            bool rounds = false, ok = true;
            for (int k = item_begin; k < item_end && ok; ++k) {
                const int* it = items + (size_t)k * ITEM_INTS;
                const TalkBlock w = talk_block(blocks + (size_t)it[0] * BLOCK_INTS, q_start, start_pos);
                const int first = it[1] * QN, rows = min(QN, w.rows - first), p0 = w.p0 + first;
                const int first_key = first_visible(p0, window), last_key = p0 + rows - 1;
                if (k > item_begin) ok = __all_sync(0xffffffffu, mbar_wait(q_empty, (uint32_t)(k - item_begin - 1) & 1u, err));
                if (!ok) break;
                if (lane == 0) mbar_expect_tx(q_full, L::Q_BYTES);
                __syncwarp();
                // head h = c * rep + g: rows g * QN .. of the c-th group of 512 / nkv rows
                for (int h = lane; h < H; h += 32)
#pragma unroll
                    for (int f = 0; f < HALVES; ++f)
                        tma_load_3d(base + (h / rep) * ((512 / nkv) * HALVES * 128) + f * (512 / nkv) * 128 + (h % rep) * QN * 128, &map_q,
                                    f * 64, h, w.t0 + first, q_full);
                const int* table = block_table + (size_t)w.b * table_stride;
                for (int kt = it[2]; kt < it[2] + it[3] && ok; ++kt) {
                    const int j = kt * S_KEYS + bi * box_rows;
                    int page = -1;
                    if (lane < boxes && j <= last_key && j + box_rows - 1 >= first_key) {
                        page = table[j >> ps_shift];
                        if (page < 0 || page >= num_pages) {
                            atomicOr(err, XB_ERR_BAD_PAGE);
                            page = -1;
                        }
                    }
                    const uint32_t nb = __popc(__ballot_sync(0xffffffffu, page >= 0));
                    for (int c = 0; c < nkv; ++c) {
                        if (rounds && !__all_sync(0xffffffffu, mbar_wait(k_empty0 + 8 * s, ph ^ 1u, err))) {
                            ok = false;
                            break;
                        }
                        if (lane == 0) mbar_expect_tx(k_full0 + 8 * s, nb * box_rows * 128);
                        __syncwarp();
                        // keys without a page stay what they were: their scores are masked by the kernel that reads them
                        if (page >= 0)
                            tma_load_2d(k_sm + s * L::K_STAGE + hf * S_KEYS * 128 + bi * box_rows * 128, &map_k, hf * 64,
                                        (page * nkv + c) * ps + (j & (ps - 1)), k_full0 + 8 * s);
                        if (++s == 2) {
                            s = 0;
                            ph ^= 1u;
                            rounds = true;
                        }
                    }
                }
            }
        } else if (warp == 9) {
            // ---- products: for every key/value head [128 keys x d] x [d x its heads' queries]
            const bool leader = lane == 0;
            const int n = 512 / nkv;
            const uint32_t idesc = umma_idesc(n, 0);
            const uint64_t dq0 = umma_desc(base, 16, 1024), dk0 = umma_desc(k_sm, 16, 1024);
            int s = 0, tiles = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int k = item_begin; k < item_end && ok; ++k) {
                const int nt = items[(size_t)k * ITEM_INTS + 3];
                ok = __all_sync(0xffffffffu, mbar_wait(q_full, (uint32_t)(k - item_begin) & 1u, err, true));
                for (int t = 0; t < nt && ok; ++t, ++tiles) {
                    // the raw scores of the tile before have been read
                    if (tiles > 0) ok = __all_sync(0xffffffffu, mbar_wait(d_empty, (uint32_t)(tiles - 1) & 1u, err, true));
                    for (int c = 0; c < nkv && ok; ++c) {
                        ok = __all_sync(0xffffffffu, mbar_wait(k_full0 + 8 * s, ph, err, true));
                        if (!ok) break;
                        tc_fence_after();
                        if (leader) {
#pragma unroll
                            for (int kk = 0; kk < HALVES * 4; ++kk)
                                umma_bf16(tmem + (uint32_t)(c * n),
                                          dk0 + (uint64_t)((s * L::K_STAGE + (kk >> 2) * S_KEYS * 128 + (kk & 3) * 32) >> 4),
                                          dq0 + (uint64_t)((c * n * HALVES * 128 + (kk >> 2) * n * 128 + (kk & 3) * 32) >> 4), idesc, kk ? 1u : 0u);
                            umma_commit(k_empty0 + 8 * s);
                            if (c == nkv - 1) umma_commit(d_full);
                        }
                        __syncwarp();
                        if (++s == 2) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                }
                if (leader) umma_commit(q_empty);
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

// ---- softmax and value sums ---------------------------------------------------------------------------------------------
// A work item is a block's 128 queries and two heads of one key/value head (or one).  Per 64 keys and head two score
// tiles of 16 KB lie side by side in memory and come as one bulk copy into one of three stages; a thread reads its row, whose 16-byte pieces the
// kernel before has laid out XOR-ed with row & 7.  The roles and waits are those of the prefill kernel over pages, with
// scores from shared memory in place of a product.
//   warps 0..3, 4..7 softmax of the two heads, warp 8 loads score tiles, warp 10 value pages, warp 9 clears in them what must not
//   meet a weight of 0, warp 11 issues O += P V.
// Tensor memory: P of head A at 0 and 32, of head B at 64 and 96 (two buffers each); O at 128 and 256.
constexpr int V_THREADS = 384;
constexpr int V_KEYS = 64;
constexpr int S_STAGES = 3, V_STAGES = 2;       // of scores (64 KB each) and of values (16 KB)
constexpr uint32_t V_SCORES = 2 * TILE_FLOATS * 4;       // one head's scores of a stage

// Whether some of the queries from position p0 on do not see all of the 64 keys from key0 on; edge_lo: the first key that the last
// of them sees.
__device__ __forceinline__ bool seen_in_part(int key0, int p0, int edge_lo) { return key0 + V_KEYS - 1 > p0 || key0 < edge_lo; }

// An element of a value row that holds an infinity or no number.
__device__ __forceinline__ bool bf16_bits_not_finite(uint32_t b) { return (b & 0x7f80u) == 0x7f80u; }

// (Rare.)  To one query's result of one head: the values that are not finite, of the keys from `first` to `last` (those it sees) in
// tiles that were cleared of them.
__device__ __noinline__ void add_not_finite(__nv_bfloat16* dst, const __nv_bfloat16* vc, const int* table, int nkv, int g, int ps, int ps_shift,
                                            int num_pages, int dv, int first, int last, int p0, int edge_lo, float out_scale) {
    for (int j = first; j <= last; ++j) {
        const int key0 = j / V_KEYS * V_KEYS;
        if (!seen_in_part(key0, p0, edge_lo)) {
            j = key0 + V_KEYS - 1;
            continue;
        }
        const int page = table[j >> ps_shift];
        if (page < 0 || page >= num_pages) continue;
        const uint4* row = reinterpret_cast<const uint4*>(vc + ((size_t)(page * nkv + g) * ps + (j & (ps - 1))) * dv);
        for (int c8 = 0; c8 < dv / 8; ++c8) {
            const uint4 v = row[c8];
            if (!bf16_not_finite(v)) continue;
            for (int c = 0; c < 8; ++c) {
                const uint32_t w = c < 2 ? v.x : c < 4 ? v.y : c < 6 ? v.z : v.w, b = (c & 1) ? w >> 16 : w & 0xffffu;
                if (bf16_bits_not_finite(b))
                    dst[c8 * 8 + c] = __float2bfloat16(__bfloat162float(dst[c8 * 8 + c]) + out_scale * __uint_as_float(b << 16));
            }
        }
    }
}

template <int DVC>
__global__ void __launch_bounds__(V_THREADS)
talk_values_tc_kernel(const __grid_constant__ CUtensorMap map_v, const __nv_bfloat16* vc, const float* scores, __nv_bfloat16* __restrict__ out,
                      long long ldo, const int* __restrict__ blocks, const int* __restrict__ work, const int* __restrict__ q_start,
                      const int* __restrict__ start_pos, const int* __restrict__ block_table, int table_stride, int nh, int nkv,
                      int ps, int ps_shift, int num_pages, int window, int sink, float out_scale, int* err) {
    constexpr int DV = 64 * DVC;
    constexpr uint32_t PIECE = V_KEYS * 128, V_BYTES = DVC * PIECE, V_OFF = S_STAGES * 2 * V_SCORES, BAR_OFF = V_OFF + V_STAGES * V_BYTES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t base = smem_u32(smem_raw), bars = base + BAR_OFF;
    // v_full[stage] v_empty[stage] pv_done[head][2] p_ready[head] o_done[head] s_full[head][stage] s_empty[head][stage]
    const uint32_t v_full0 = bars, v_empty0 = bars + 16, pv_done0 = bars + 32, p_ready0 = bars + 64, o_done0 = bars + 80;
    const uint32_t s_full0 = bars + 96, s_empty0 = bars + 96 + 16 * S_STAGES, v_clear0 = bars + 96 + 32 * S_STAGES;      // v_clear[stage]
    volatile uint32_t* marks = reinterpret_cast<volatile uint32_t*>(smem_raw + BAR_OFF + 112 + 32 * S_STAGES);      // of four items in turn
    volatile uint32_t* words = reinterpret_cast<volatile uint32_t*>(smem_raw + BAR_OFF + 240);
    static_assert(112 + 32 * S_STAGES + 16 <= 240, "room for the barriers");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ctas = (int)gridDim.x;
    const int item_begin = work[blockIdx.x];
    int item_end = work[blockIdx.x + 1];
    const int* const items = work + ctas + 1;
    if (threadIdx.x == 0) {
        if (base & 1023u) atomicOr(err, XB_ERR_WAIT);
        for (int i = 0; i < 2 * S_STAGES; ++i) {
            mbar_init(s_full0 + 8 * i, 1);
            mbar_init(s_empty0 + 8 * i, 4);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(v_full0 + 8 * i, 1);      // v_full, v_empty
            mbar_init(pv_done0 + 8 * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(p_ready0 + 8 * i, 128);
            mbar_init(o_done0 + 8 * i, 1);
            mbar_init(v_clear0 + 8 * i, 32);
        }
        mbar_init_fence();
    }
    if (*reinterpret_cast<volatile int*>(err) & XB_ERR_WAIT) item_end = item_begin;
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

    struct Item {
        TalkBlock blk;
        int h0, nhd, g, lo, hi, first_key, last_key;
    };
    auto item_at = [&](int k) {
        const int* it = items + (size_t)k * ITEM_INTS;
        Item w;
        w.blk = talk_block(blocks + (size_t)it[0] * BLOCK_INTS, q_start, start_pos);
        w.h0 = it[1];
        w.nhd = it[2] == 2 ? 2 : 1;
        w.g = w.h0 / (nh / nkv);
        w.first_key = first_visible(w.blk.p0, window);
        w.last_key = w.blk.p0 + w.blk.rows - 1;
        w.lo = w.first_key / V_KEYS;
        w.hi = w.last_key / V_KEYS;
        return w;
    };
    if (warp == 8) {
        // ---- score tiles
        bool ok = true;
        // each head's own ring: the stage of its next tile, the parity of its rounds, whether there was one (a head may sit
        // an item out)
        int st[2] = {0, 0};
        uint32_t ph[2] = {0, 0};
        bool rounds[2] = {false, false};
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            for (int kt = w.lo; kt <= w.hi && ok; ++kt) {
#pragma unroll
                for (int hd = 0; hd < 2; ++hd) {
                    if (hd >= w.nhd || !ok) continue;
                    const uint32_t at = S_STAGES * hd + st[hd];
                    if (rounds[hd]) ok = __all_sync(0xffffffffu, mbar_wait(s_empty0 + 8 * at, ph[hd] ^ 1u, err));
                    if (!ok) continue;
                    if (lane == 0) {
                        const uint32_t bar = s_full0 + 8 * at;
                        mbar_expect_tx(bar, V_SCORES);
                        const float* src = scores + (w.blk.tile0 + (long long)(w.h0 + hd) * w.blk.nkb + (kt * 2 - w.blk.kb0)) * TILE_FLOATS;
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                     ::"r"(base + at * V_SCORES), "l"(src), "r"(V_SCORES), "r"(bar) : "memory");
                    }
                    __syncwarp();
                    if (++st[hd] == S_STAGES) {
                        st[hd] = 0;
                        ph[hd] ^= 1u;
                        rounds[hd] = true;
                    }
                }
            }
        }
    } else if (warp == 10) {
        // ---- value pages: one lane per page box
        const int box_rows = ps < V_KEYS ? ps : V_KEYS, boxes = (V_KEYS / box_rows) * DVC;      // at most 16
        const int bi = lane / DVC, hf = lane % DVC;
        int s = 0;
        uint32_t ph = 0;
        bool rounds = false, ok = true;
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            const int* table = block_table + (size_t)w.blk.b * table_stride;
            for (int kt = w.lo; kt <= w.hi; ++kt) {
                const int j = kt * V_KEYS + bi * box_rows;
                int page = -1;
                if (lane < boxes && j <= w.last_key && j + box_rows - 1 >= w.first_key) {
                    page = table[j >> ps_shift];
                    if (page < 0 || page >= num_pages) {
                        atomicOr(err, XB_ERR_BAD_PAGE);
                        page = -1;
                    }
                }
                if (rounds && !__all_sync(0xffffffffu, mbar_wait(v_empty0 + 8 * s, ph ^ 1u, err))) {
                    ok = false;
                    break;
                }
                const uint32_t nb = __popc(__ballot_sync(0xffffffffu, page >= 0));
                if (lane == 0) mbar_expect_tx(v_full0 + 8 * s, nb * box_rows * 128);
                __syncwarp();
                if (page >= 0)
                    tma_load_2d(base + V_OFF + s * V_BYTES + hf * PIECE + bi * box_rows * 128, &map_v, hf * 64,
                                (page * nkv + w.g) * ps + (j & (ps - 1)), v_full0 + 8 * s);
                if (++s == V_STAGES) {
                    s = 0;
                    ph ^= 1u;
                    rounds = true;
                }
            }
        }
    } else if (warp == 9) {
        // ---- values that must not meet a weight of 0, in tiles that some query sees in part: rows that no query of the block
        // sees (their pages were not loaded, or hold anything) become zeros, and so do elements that are not finite; whether
        // there were any of those is the item's mark.  The product waits for this warp at every tile.
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            const int edge_lo = first_visible(w.blk.p0 + QB_ROWS - 1, window);
            bool any = false;
            if (lane == 0) marks[k & 3] = 0;
            for (int kt = w.lo; kt <= w.hi; ++kt) {
                if (!__all_sync(0xffffffffu, mbar_wait(v_full0 + 8 * s, ph, err))) {
                    ok = false;
                    break;
                }
                const int key0 = kt * V_KEYS;
                if (seen_in_part(key0, w.blk.p0, edge_lo)) {
                    uint4* tile = reinterpret_cast<uint4*>(smem_raw + V_OFF + s * V_BYTES);
#pragma unroll 4
                    for (int i = lane; i < (int)V_BYTES / 16; i += 32) {       // a row is 8 pieces of 16 bytes, in any order
                        const int j = key0 + ((i >> 3) & (V_KEYS - 1));
                        const bool out_of = j < w.first_key || j > w.last_key;
                        uint4 v = tile[i];
                        if (out_of) {
                            tile[i] = make_uint4(0, 0, 0, 0);
                        } else if (bf16_not_finite(v)) {
                            auto clear = [](uint32_t x) {
                                return (bf16_bits_not_finite(x) ? 0u : x & 0xffffu) | (bf16_bits_not_finite(x >> 16) ? 0u : x & 0xffff0000u);
                            };
                            tile[i] = make_uint4(clear(v.x), clear(v.y), clear(v.z), clear(v.w));
                            any = true;
                        }
                    }
                    fence_async_shared();
                    any = __any_sync(0xffffffffu, any);
                    if (any && lane == 0) marks[k & 3] = 1;
                }
                mbar_arrive(v_clear0 + 8 * s);
                if (++s == V_STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 11) {
        // ---- O += P V
        const bool leader = lane == 0;
        const uint32_t idesc = umma_idesc(DV, 1);
        const uint64_t dv0 = umma_desc(base + V_OFF, PIECE, 1024);
        int s = 0, Th[2] = {0, 0};
        uint32_t ph = 0;
        bool ok = true;
        for (int k = item_begin; k < item_end && ok; ++k) {
            const Item w = item_at(k);
            for (int kt = w.lo; kt <= w.hi && ok; ++kt) {
                ok = __all_sync(0xffffffffu, mbar_wait(v_clear0 + 8 * s, ph, err, true));
                const uint64_t dv = dv0 + (uint64_t)((s * V_BYTES) >> 4);
#pragma unroll
                for (int hd = 0; hd < 2; ++hd) {
                    if (!ok || hd >= w.nhd) continue;
                    const int th = Th[hd]++, sb = th & 1;
                    ok = __all_sync(0xffffffffu, mbar_wait(p_ready0 + 8 * hd, th & 1, err, true));
                    if (!ok) continue;
                    tc_fence_after();
                    if (leader) {
#pragma unroll
                        for (int kk = 0; kk < V_KEYS / 16; ++kk)
                            umma_bf16_ta(tmem + (uint32_t)(128 + hd * 128), tmem + (uint32_t)(hd * 64 + sb * 32 + kk * 8),
                                         dv + (uint64_t)((kk * 2048) >> 4), idesc, (kt > w.lo || kk) ? 1u : 0u);
                        umma_commit(pv_done0 + 8 * (2 * hd + sb));
                        if (kt == w.hi) umma_commit(o_done0 + 8 * hd);
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (leader) umma_commit(v_empty0 + 8 * s);
                __syncwarp();
                if (++s == V_STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp < 8) {
        // ---- softmax: one query per thread
        const int hd = warp >> 2, r = (int)threadIdx.x & 127;
        const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tmem_p = tmem + (uint32_t)(hd * 64) + lane_addr, tmem_o = tmem + (uint32_t)(128 + hd * 128) + lane_addr;
        const uint32_t my_p_ready = p_ready0 + 8 * hd, my_pv_done = pv_done0 + 16 * hd;
        int th = 0, done = 0;      // key tiles of this head, items of this head
        uint32_t ss = 0, sph = 0;           // stage of this head's next scores, parity of the rounds
        bool alive = true;
        for (int k = item_begin; k < item_end && alive; ++k) {
            const Item w = item_at(k);
            if (hd >= w.nhd) continue;
            const int p0 = w.blk.p0, my_pos = p0 + r, last_key = w.last_key, lo = w.lo, hi = w.hi;
            const int my_lo = first_visible(my_pos, window), edge_lo = first_visible(p0 + QB_ROWS - 1, window);
            float m_ref = sink ? 0.f : -INFINITY, l = sink ? 1.f : 0.f;      // the silent entry: score 0
            for (int kt = lo; kt <= hi; ++kt, ++th) {
                const int sb = th & 1, key0 = kt * V_KEYS;
                if (!__all_sync(0xffffffffu, mbar_wait(s_full0 + 8 * (S_STAGES * hd + ss), sph, err))) {
                    alive = false;
                    break;
                }
                float sc[64];
                {
                    const unsigned char* row = smem_raw + (S_STAGES * hd + ss) * V_SCORES + r * 128;
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(row + (c >> 3) * (TILE_FLOATS * 4) + (((c & 7) ^ (r & 7)) << 4));
                        sc[c * 4] = v.x; sc[c * 4 + 1] = v.y; sc[c * 4 + 2] = v.z; sc[c * 4 + 3] = v.w;
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(s_empty0 + 8 * (S_STAGES * hd + ss));
                if (++ss == S_STAGES) {
                    ss = 0;
                    sph ^= 1u;
                }
                if (seen_in_part(key0, p0, edge_lo)) {
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        const int j = key0 + c;
                        sc[c] = (j <= my_pos && j <= last_key && j >= my_lo) ? sc[c] : -INFINITY;
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
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                float corr = 1.f;
                int moved = 0;
                if (mx > m_ref + RESCALE_STEP) {
                    corr = m_ref == -INFINITY ? 0.f : ex2(m_ref - mx);
                    m_ref = mx;
                    moved = kt > lo;
                }
                const float m_neg = m_ref == -INFINITY ? 0.f : -m_ref;
                const f32x2 mneg2 = pack2(m_neg, m_neg);
                f32x2 sum_a = pack2(0.f, 0.f), sum_b = pack2(0.f, 0.f);
                uint32_t pk[32];
#pragma unroll
                for (int c8 = 0; c8 < 8; ++c8) {
                    float x[8], e[8];
#pragma unroll
                    for (int c = 0; c < 8; c += 2) unpack2(add2(pack2(sc[c8 * 8 + c], sc[c8 * 8 + c + 1]), mneg2), x[c], x[c + 1]);
#pragma unroll
                    for (int c = 0; c < 8; ++c) e[c] = ex2(x[c]);
                    // the sum is that of the weights as the product sees them
                    f32x2 w[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t two = pack_bf16(e[2 * c], e[2 * c + 1]);
                        pk[c8 * 4 + c] = two;
                        w[c] = pack2(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u));
                    }
                    sum_a = add2(sum_a, add2(w[0], w[1]));
                    sum_b = add2(sum_b, add2(w[2], w[3]));
                }
                float s0, s1, s2, s3;
                unpack2(sum_a, s0, s1);
                unpack2(sum_b, s2, s3);
                l = l * corr + ((s0 + s1) + (s2 + s3));
                // P's buffer was read two tiles ago: by the product whose end was waited for one tile ago, or one before it
                tmem_st32_u(tmem_p + sb * 32, pk);
                // the product before must be complete before O is touched, and before this tile is announced
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
            if (alive) alive = mbar_wait(o_done0 + 8 * hd, (uint32_t)done & 1u, err);
            ++done;
            alive = __all_sync(0xffffffffu, alive);
            tc_fence_after();
            const float inv = l > 0.f ? out_scale / l : 0.f;
            if (alive) {
                __nv_bfloat16* dst = out + (size_t)(w.blk.t0 + r) * ldo + (size_t)(w.h0 + hd) * DV;
#pragma unroll
                for (int c0 = 0; c0 < DV; c0 += 32) {
                    float o[32];
                    tmem_ld32(tmem_o + c0, o);
                    if (r < w.blk.rows) {
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
                if (marks[k & 3] != 0 && r < w.blk.rows)        // (the item's tiles have all been looked at: its products are done)
                    add_not_finite(dst, vc, block_table + (size_t)w.blk.b * table_stride, nkv, w.g, ps, ps_shift, num_pages, DV, my_lo, my_pos, p0,
                                   edge_lo, out_scale);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_free(tmem, 512);
}

template <int H, int HALVES>
int launch_scores(const CUtensorMap& mq, const CUtensorMap& mk, float* scores, const float* talk_host, const int* blocks, const int* work,
                  int ctas, const int* q_start, const int* start_pos, const int* table, int stride, int nkv, int ps, int shift,
                  int num_pages, int window, float sl2, int* err, cudaStream_t stream) {
    constexpr size_t smem = ScoresSmem<H, HALVES>::TOTAL;
    const auto kernel = talk_scores_tc_kernel<H, HALVES>;
    TalkMatrix<H> talk;
    for (int i = 0; i < H * H; ++i) talk.t[i] = talk_host[i] * sl2;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return xb_launch(kernel, dim3(ctas), dim3(S_THREADS), smem, stream, mq, mk, scores, talk, blocks, work, q_start, start_pos, table,
                     stride, nkv, ps, shift, num_pages, window, err);
}
template <int DVC>
int launch_values(const CUtensorMap& mv, const void* vc, const float* scores, void* out, long long ldo, const int* blocks, const int* work, int ctas,
                  const int* q_start, const int* start_pos, const int* table, int stride, int nh, int nkv, int ps, int shift,
                  int num_pages, int window, int sink, float out_scale, int* err, cudaStream_t stream) {
    constexpr size_t smem = (size_t)S_STAGES * 2 * V_SCORES + V_STAGES * DVC * V_KEYS * 128 + 256;
    const auto kernel = talk_values_tc_kernel<DVC>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return xb_launch(kernel, dim3(ctas), dim3(V_THREADS), smem, stream, mv, (const __nv_bfloat16*)vc, scores, (__nv_bfloat16*)out, ldo, blocks, work, q_start,
                     start_pos, table, stride, nh, nkv, ps, shift, num_pages, window, sink, out_scale, err);
}

}  // namespace

// Whether xb_attn_talking_tc takes these sizes: a tile of scores fills tensor memory, so heads divide 512 columns into at
// least 16 queries each, and the queries of a key/value head are one product of at most 128 columns; page boxes are at most
// a lane each.
XB_EXPORT int xb_attn_talking_tc_takes(int nh, int nkv, int d, int dv, int ps) {
    return (nh == 8 || nh == 16 || nh == 32) && (nkv == 4 || nkv == 8 || nkv == 16) && nh % nkv == 0 && (d == 64 || d == 128) &&
           (dv == 64 || dv == 128) && ps >= 8 && (ps & (ps - 1)) == 0;
}

// One pair of launches over the blocks of a chunk (xb_talk_work of the host library): scores of `heads` heads into
// `scores`, then softmax and value sums into out (rows ldo elements apart, times out_scale).  `talk` [heads, heads]
// lies in HOST memory.
XB_EXPORT int xb_attn_talking_tc(void* out, long long ldo, const void* q, const void* kc, const void* vc, const float* talk,
                                 float* scores, const int* blocks, const int* work1, int ctas1, const int* work2, int ctas2,
                                 const int* q_start, const int* start_pos, const int* table, int stride, int tokens, int nh, int nkv,
                                 int d, int dv, int ps, int num_pages, int window, float scale, int sink, float out_scale, int* err,
                                 cudaStream_t stream) {
    if (ctas1 <= 0 || ctas2 <= 0) return 0;
    if (!xb_attn_talking_tc_takes(nh, nkv, d, dv, ps) || ldo % 8 || window < 0 ||
        (((uintptr_t)out | (uintptr_t)q | (uintptr_t)kc | (uintptr_t)vc | (uintptr_t)scores) & 15) || !talk)
        return (int)cudaErrorNotSupported;
    int shift = 3;
    while ((1 << shift) < ps) ++shift;
    CUtensorMap mq, mk, mv;
    const int qn = 512 / nh;
    const long long qd[3] = {d, nh, tokens}, qs[2] = {d, (long long)nh * d}, rows = (long long)num_pages * nkv * ps;
    const int qb[3] = {64, 1, qn};
    if (!tensor_map_bf16(&mq, q, 3, qd, qs, qb) || !tensor_map_2d(&mk, kc, rows, d, ps < S_KEYS ? ps : S_KEYS) ||
        !tensor_map_2d(&mv, vc, rows, dv, ps < V_KEYS ? ps : V_KEYS))
        return (int)cudaErrorNotSupported;
    const float sl2 = scale * 1.4426950408889634f;
    int rc;
#define XB_S(N, F) rc = launch_scores<N, F>(mq, mk, scores, talk, blocks, work1, ctas1, q_start, start_pos, table, stride, nkv, ps, shift, num_pages, window, sl2, err, stream)
#define XB_SH(N) do { if (d == 128) XB_S(N, 2); else XB_S(N, 1); } while (0)
    if (nh == 8) XB_SH(8);
    else if (nh == 16) XB_SH(16);
    else XB_SH(32);
#undef XB_SH
#undef XB_S
    if (rc != 0) return rc;
#define XB_V(N) launch_values<N>(mv, vc, scores, out, ldo, blocks, work2, ctas2, q_start, start_pos, table, stride, nh, nkv, ps, shift, num_pages, window, sink, out_scale, err, stream)
    return dv == 128 ? XB_V(2) : XB_V(1);
#undef XB_V
}
