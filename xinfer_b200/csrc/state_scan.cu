// Recurrences whose state is a matrix per head, carried per request in float32:
//
//   selective_scan_kernel   (state-space duality)   S[N, P]:  S <- exp(-A dt) S + dt B x^T,   y = S^T C + D x
//   delta_rule_kernel       (gated delta rule)      S[d, dv]: S <- diag(g) S,  u = beta (v - S^T k),  S <- S + k u^T,
//                                                             o = S^T q      (read after the token's own update)
//   linear_scan_kernel      (gated linear attention)  S[d, dv]: S <- diag(alpha) S + k v^T,  o = scale S^T q
//   matrix_memory_kernel    (xLSTM's mLSTM)         S[d, dv]: S <- e^(f+m-m') S + e^(i-m') k v^T, n[d] likewise with k alone,
//                                                             o = S^T q and the divisor max(|n . q|, e^(-m')) + eps
//   low_rank_decay_kernel   alpha = sigmoid(W_a2 low + b)^(1 / tau) for it, per token and key channel
//   gated_head_norm_kernel  the gate and the RMS norm over a head (or a group of channels) behind either
//
// Layout of the scans: a block takes one (request, head) and a tile of the state's columns (columns never mix).
// Its first warps compute: a lane keeps kRows rows of two neighbouring columns in registers; DS lanes of a warp
// share a column pair and fold their sums over rows with shuffles.  Its last warps feed them: tokens of a request
// are walked in order, a tile of TT tokens at a time, and while the computing warps work on one tile the feeding
// warps bring the ones after it into shared memory with asynchronous copies, work out what every column needs alike
// (step sizes, decays, unit vectors, beta) once per token, and write the tile before to memory.  The step loop
// reads broadcast vectors from shared memory only.  One block barrier per tile hands the buffers over.  The state
// is read from state[slot] at the step's first token and left there after its last, so a cut between steps changes
// nothing but when the state crosses memory.  Everything is float32: decays, softplus, exponentials, step sizes,
// unit norms, gates.
//
// What bounds them is the issue of the multiply-adds of a token and, in the chain from token to token, the shuffles that fold
// the sums: rows are worked on in pairs (one packed instruction for two), the sums of four tokens are folded by the same
// shuffles, and a finer column tile is taken while processors would be idle.  2,048 tokens, 32 heads of 128 x 128 states:
// selective 563 -> 414 us, delta rule 690 -> 471 us and 94 us of delta_prepare_kernel, linear 418 -> 356 us; matrix memory
// 437 -> 368 us.
#include "common.cuh"

__device__ __forceinline__ float softplus_f32(float v) { return v > 20.f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float sigmoid_exact(float v) { return 1.f / (1.f + expf(-v)); }

namespace {
// State rows a lane keeps per column.  (8, which spreads a column's work over twice the lanes, made 2,048 tokens of 16 heads of
// 128 x 128 states 4 % faster, but doubles the shuffles: 32 heads were 4 to 18 % slower, a decode step's scans 1.5 times.)
constexpr int kRows = 16;
constexpr int kRowsPad = kRows + 4;  // the same rows in shared memory, spaced so that row groups fall on different banks
constexpr int kScanTile = 16;        // tokens per tile, at most
constexpr int kStages = 3;           // tiles in shared memory: one is worked on, one lands, one is asked for

__device__ __forceinline__ void scan_cp4(float* dst, const float* src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
}
__device__ __forceinline__ void scan_cp16(float* dst, const float* src) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}
// A tile's copies are one group of the copying thread; the tile before the newest has landed.
__device__ __forceinline__ void scan_cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void scan_cp_land() {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncwarp();
}

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// Two float32 in one 64-bit register: state rows are kept and worked on in pairs, as a 16-byte load of a row vector brings them.
typedef unsigned long long pair2;
__device__ __forceinline__ pair2 pr_make(float a, float b) {
    pair2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void pr_split(pair2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ float pr_sum(pair2 v) {
    float a, b;
    pr_split(v, a, b);
    return a + b;
}
__device__ __forceinline__ pair2 pr_fma(pair2 a, pair2 b, pair2 c) {
    pair2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ pair2 pr_mul(pair2 a, pair2 b) {
    pair2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
constexpr int kPairs = kRows / 2;
// A group of N tokens that are worked on together.  Whole: its code then has no branch between the tokens, and the loads of one
// can overlap the arithmetic of another.
template <int N, bool WHOLE>
struct Group {
    static constexpr int tokens = N;
    static constexpr bool whole = WHOLE;
};
// Where no request brings more than this many tokens the kernels take them one by one: there is no chain to hide, and the code
// needs 128 registers instead of 140 to 166, with which two blocks of eight warps fit a processor.  256 requests of one token, 8
// heads of 64 x 64 states: linear 42 -> 27 us, selective 43 -> 28 us; 32 requests of five tokens, 13 -> 11 us.  (At 40 tokens groups
// of four are 1.1 to 1.2 times as fast.)  The sums are the same bits either way.
constexpr int kFewTokens = 16;

// The feeding warps' walk over the tiles, in step with the computing warps (one block barrier per tile): while tile t is
// worked on, the copies of t + 2 are asked for, t + 1 has landed and is finished, and the results of t - 1 leave: the copies have
// a whole tile's time to land, and the memory's latency is not part of a tile's.
template <typename Bring, typename Finish, typename Leave>
__device__ __forceinline__ void feed(int ntiles, Bring bring, Finish finish, Leave leave) {
    bring(0);
    scan_cp_commit();
    if (ntiles > 1) bring(1);
    scan_cp_commit();
    finish(0);
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        if (tile + 2 < ntiles) bring(tile + 2);
        scan_cp_commit();
        if (tile + 1 < ntiles) finish(tile + 1);
        if (tile > 0) leave(tile - 1);
        __syncthreads();
    }
}
// Four pairs of rows at once from shared memory (16-byte loads).
__device__ __forceinline__ void load_pairs(const float* src, pair2 (&v)[kPairs]) {
    const ulonglong2* p = reinterpret_cast<const ulonglong2*>(src);
#pragma unroll
    for (int i = 0; i < kPairs / 2; ++i) {
        const ulonglong2 t = p[i];
        v[2 * i] = t.x;
        v[2 * i + 1] = t.y;
    }
}

// Sums over the row groups of N values a lane holds, for all of them at once: a step halves the values a lane keeps as long
// as it has several, so that N = 8 sums over 8 row groups are 7 shuffles and one round of waiting where one value after the
// other took 24 and eight.  Afterwards a lane holds the sums of values first .. first + (returned count) - 1 in v[0 ..];
// lanes that differ only in row-group bits beyond those hold the same ones.  (Lanes of a warp are laid out [DS row groups]
// [32 / DS column pairs].)
template <int DS, int N>
__device__ __forceinline__ int fold_many(float (&v)[N], int ds, int& first) {
    constexpr int CGW = 32 / DS;
    int width = N;
    first = 0;
#pragma unroll
    for (int bit = DS / 2; bit >= 1; bit >>= 1) {
        if (width > 1) {
            const int half = width / 2;
            const bool upper = (ds & bit) != 0;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i >= half) break;
                const float send = upper ? v[i] : v[i + half], keep = upper ? v[i + half] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit * CGW);
            }
            first += upper ? half : 0;
            width = half;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], bit * CGW);
        }
    }
    return width;
}
// Behind fold_many: every lane gets the sums of all N values.
template <int DS, int N>
__device__ __forceinline__ void spread_many(float (&v)[N], int ds) {
    constexpr int CGW = 32 / DS, LAST = DS > N ? DS / N : 1;     // the lowest row-group bit that halved the values
    int width = DS >= N ? 1 : N / DS;
#pragma unroll
    for (int bit = LAST; bit < DS; bit <<= 1) {
        if (width >= N) break;
        const bool upper = (ds & bit) != 0;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if (i >= width) break;
            const float other = __shfl_xor_sync(0xffffffffu, v[i], bit * CGW), own = v[i];
            v[i] = upper ? other : own;
            v[i + width] = upper ? own : other;
        }
        width *= 2;
    }
}
// Whether this lane writes what fold_many left it with: one lane of those that hold the same sums.
template <int DS, int N>
__device__ __forceinline__ bool fold_writes(int ds) {
    return DS <= N || (ds & (DS / N - 1)) == 0;
}
__device__ __forceinline__ int padded_row(int j) { return (j / kRows) * kRowsPad + (j % kRows); }

// A row vector of `len` floats (rows up to `padded` are zero) into the padded layout; `vec` says that source and
// length allow 16-byte copies.
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int len, int padded, int lane, bool vec) {
    if (vec) {
        for (int j = lane * 4; j < padded; j += 128) {
            if (j < len)
                scan_cp16(dst + padded_row(j), src + j);
            else
                *reinterpret_cast<float4*>(dst + padded_row(j)) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        for (int j = lane; j < padded; j += 32) {
            if (j < len)
                scan_cp4(dst + padded_row(j), src + j);
            else
                dst[padded_row(j)] = 0.f;
        }
    }
}
// The block's columns [c_base, c_base + VT) of a row of `cols` columns; the ones past the end are zero.
__device__ __forceinline__ void stage_cols(float* dst, const float* src, int c_base, int cols, int VT, int lane, bool vec) {
    if (vec) {
        for (int c = lane * 4; c < VT; c += 128) {
            if (c_base + c < cols)
                scan_cp16(dst + c, src + c_base + c);
            else
                *reinterpret_cast<float4*>(dst + c) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
        for (int c = lane; c < VT; c += 32) {
            if (c_base + c < cols)
                scan_cp4(dst + c, src + c_base + c);
            else
                dst[c] = 0.f;
        }
    }
}
}  // namespace

// xbc[t] = [x: H*P | B: G*N | C: G*N] after the short convolution; dt is column dt_off + h of proj[t] (before
// the bias and the softplus).  state [slots, H, N, P].  y [T, H*P].  Shared memory: three stages of
// B[TT][NP] C[TT][NP] x[TT][VT] dt[TT] dec[TT], then two tiles y[TT][VT].  `cw` of the block's warps compute.
template <int DS, bool FEW>
__global__ void __launch_bounds__(FEW ? 256 : 384, FEW ? 2 : 1) selective_scan_kernel(float* __restrict__ y, const float* xbc, int C,
                                                             const float* proj, long long ldp, int dt_off,
                                                             const float* __restrict__ dt_bias,
                                                             const float* __restrict__ A_log, const float* __restrict__ Dv,
                                                             float* state, const int* __restrict__ q_start,
                                                             const int* __restrict__ slots, int H, int P, int N, int G,
                                                             int TT, int stage, int cw, int vec) {
    pdl_wait();
    extern __shared__ __align__(16) float scan_smem[];
    constexpr int CGW = 32 / DS, NP = DS * kRowsPad, NR = DS * kRows;
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int VT = cw * CGW * 2, c_base = blockIdx.z * VT;
    const int slot = slots[b];
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 - t0 <= XB_FEW_TOKENS) pdl_launch_dependents();
    if (slot < 0 || t1 <= t0) return;
    const int inner = H * P, g = h / (H / G);
    const int ntiles = (t1 - t0 + TT - 1) / TT;
    float* sy = scan_smem + kStages * stage;
    if (w >= cw) {
        // feeding warps: warp `pi` of `pw` takes tokens pi, pi + pw, ... of every tile
        const int pi = w - cw, pw = (blockDim.x >> 5) - cw;
        const float A = expf(A_log[h]), dtb = dt_bias[h];
        auto bring = [&](int tile) {
            float* sB = scan_smem + (tile % kStages) * stage;
            float* sC = sB + TT * NP;
            float* sx = sC + TT * NP;
            float* sdt = sx + TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw) {
                const float* row = xbc + (size_t)(tb + tt) * C;
                stage_rows(sB + tt * NP, row + inner + g * N, N, NR, lane, vec);
                stage_rows(sC + tt * NP, row + inner + (G + g) * N, N, NR, lane, vec);
                stage_cols(sx + tt * VT, row + h * P, c_base, P, VT, lane, vec);
            }
            const int mine = pi + lane * pw;
            if (mine < nt) scan_cp4(sdt + mine, proj + (size_t)(tb + mine) * ldp + dt_off + h);
        };
        auto finish = [&](int tile) {
            float* sdt = scan_smem + (tile % kStages) * stage + 2 * TT * NP + TT * VT;
            const int nt = min(TT, t1 - t0 - tile * TT), mine = pi + lane * pw;
            scan_cp_land();
            if (mine < nt) {
                const float dt = softplus_f32(sdt[mine] + dtb);
                sdt[mine] = dt;
                sdt[TT + mine] = expf(-A * dt);
            }
        };
        auto leave = [&](int tile) {
            const float* src = sy + (tile & 1) * TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw)
                for (int c = lane; c < VT; c += 32)
                    if (c_base + c < P) y[(size_t)(tb + tt) * inner + h * P + c_base + c] = src[tt * VT + c];
        };
        feed(ntiles, bring, finish, leave);
        leave(ntiles - 1);
        return;
    }
    const int ds = lane / CGW, cl = (w * CGW + lane % CGW) * 2, p0 = c_base + cl;
    const float Dh = Dv[h];
    pair2 S0[kPairs], S1[kPairs];
    float* st = state + ((size_t)slot * H + h) * N * P;
    auto at = [&](int n, int p) { return n < N && p < P ? st[(size_t)n * P + p] : 0.f; };
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int n = ds * kRows + 2 * i;
        S0[i] = pr_make(at(n, p0), at(n + 1, p0));
        S1[i] = pr_make(at(n, p0 + 1), at(n + 1, p0 + 1));
    }
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        const float* sB = scan_smem + (tile % kStages) * stage + ds * kRowsPad;
        const float* sC = sB + TT * NP;
        const float* sx = scan_smem + (tile % kStages) * stage + 2 * TT * NP;
        const float* sdt = sx + TT * VT;
        sx += cl;
        float* out = sy + (tile & 1) * TT * VT + cl;
        const int nt = min(TT, t1 - t0 - tile * TT);
        // four tokens at a time: the state's updates of one token hide the sums over the row groups of the others
        auto group = [&](int tt, auto grp) {
            constexpr int NG = decltype(grp)::tokens;
            constexpr bool whole = decltype(grp)::whole;
            float v[2 * NG];
#pragma unroll
            for (int k = 0; k < NG; ++k) {
                v[2 * k] = v[2 * k + 1] = 0.f;
                if (!whole && tt + k >= nt) continue;
                const float dt = sdt[tt + k], dec = sdt[TT + tt + k];
                const float2 xv = *reinterpret_cast<const float2*>(sx + (tt + k) * VT);
                const pair2 d0 = pr_make(dt * xv.x, dt * xv.x), d1 = pr_make(dt * xv.y, dt * xv.y), keep = pr_make(dec, dec);
                pair2 B[kPairs], Cv[kPairs], a0 = 0ull, a1 = 0ull;
                load_pairs(sB + (tt + k) * NP, B);
                load_pairs(sC + (tt + k) * NP, Cv);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    S0[i] = pr_fma(keep, S0[i], pr_mul(B[i], d0));
                    S1[i] = pr_fma(keep, S1[i], pr_mul(B[i], d1));
                    a0 = pr_fma(S0[i], Cv[i], a0);
                    a1 = pr_fma(S1[i], Cv[i], a1);
                }
                v[2 * k] = pr_sum(a0);
                v[2 * k + 1] = pr_sum(a1);
            }
            int first;
            const int n = fold_many<DS, 2 * NG>(v, ds, first);
            if (fold_writes<DS, 2 * NG>(ds)) {
#pragma unroll
                for (int i = 0; i < 2 * NG; ++i) {
                    const int k = (first + i) >> 1, c = (first + i) & 1;
                    if (i < n && (whole || tt + k < nt)) out[(tt + k) * VT + c] = fmaf(Dh, sx[(tt + k) * VT + c], v[i]);
                }
            }
        };
        if constexpr (FEW) {
            for (int tt = 0; tt < nt; ++tt) group(tt, Group<1, true>{});
        } else {
            int done = 0;
            for (; done + 4 <= nt; done += 4) group(done, Group<4, true>{});
            if (done < nt) group(done, Group<4, false>{});
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        float u[4];
        pr_split(S0[i], u[0], u[1]);
        pr_split(S1[i], u[2], u[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int n = ds * kRows + 2 * i + (e & 1), p = p0 + (e >> 1);
            if (n < N && p < P) st[(size_t)n * P + p] = u[e];
        }
    }
}

// qkv[t] = [q: G*d | k: G*d | v: H*dv] after the short convolution; beta is column beta_off + h of proj[t] before
// the sigmoid; ag[t] holds the decay's pre-activation for (head, key channel) at its front.  q and k become unit
// vectors over a head (q also times d^-1/2); g = exp(-exp(A_log_h) softplus(a + dt_bias)) per (head, key channel).
// state [slots, H, d, dv].  o [T, H*dv].
//
// Four tokens of a request are taken at a time, so that the chain from token to token - an inner product over the state's
// rows, its sum over the row groups, an update - is walked once for them: with G_i the product of the decays up to token i
// of the four, E_j that of those behind token j, and S the state before them,
//     u_i = beta_i (v_i - S^T (G_i k_i) - sum_{j<i} A_ij u_j),      A_ij = sum_r k_i (G_i / G_j) k_j,
//     o_i = S^T (G_i q_i) + sum_{j<=i} B_ij u_j,                    B_ij = sum_r q_i (G_i / G_j) k_j,
//     S  <- G_3 S + sum_j (E_j k_j) u_j^T.
// The quotients are products of the decays between the two tokens, never divided.  A request's last tokens are filled up by
// ones that change nothing.  What needs no column of the state - unit vectors, decays, their products, A and B - is formed
// once per head by delta_prepare_kernel, a warp per (four tokens, head): formed by the feeding warps of every column tile's
// block it took those 0.34 us a token (690 us for 2,048 tokens of 16 heads of 128 x 128), whatever the computing warps did.
// prep: [T][H][G q | G k | E k][d], then per (four tokens, head) [G_3: d | A, B: 16]; the place of four tokens that begin at
// token t of request b is t / 4 + b.
__device__ __forceinline__ const float* delta_group(const float* prep, long long tokens, int H, int d, int t, int b, int h) {
    return prep + tokens * H * 3 * d + ((long long)((t >> 2) + b) * H + h) * (d + 16);
}
// V = 4: a lane takes four neighbouring channels with 16-byte accesses, where the rows allow it (2,048 tokens of 32 heads of
// 128: 136 -> 94 us).
template <int V>
__global__ void __launch_bounds__(128) delta_prepare_kernel(float* __restrict__ prep, const float* qkv, int Cq,
                                                            const float* ag, long long ldag,
                                                            const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                                                            const int* __restrict__ q_start, int entries, int tokens, int H, int G,
                                                            int d, float unit_eps) {
    pdl_overlap_few();
    const int lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (h >= H) return;
    int grp = blockIdx.x, b = 0, t = 0, n = 0;
    for (; b < entries; ++b) {
        const int t0 = q_start[b], groups = (q_start[b + 1] - t0 + 3) / 4;
        if (grp < groups) {
            t = t0 + grp * 4;
            n = min(4, q_start[b + 1] - t);
            break;
        }
        grp -= groups;
    }
    if (n <= 0) return;
    const int kvh = h / (H / G);
    const float A = expf(A_log[h]), qk_scale = 1.f / sqrtf((float)d);
    const float* qr = qkv + (size_t)t * Cq + kvh * d;
    const float* kr = qr + G * d;
    const float* ar = ag + (size_t)t * ldag + h * d;
    float qs[4], ks[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) qs[i] = ks[i] = 0.f;
    auto fetch = [](const float* p, float (&x)[V]) {
        if (V == 4) {
            const float4 v = *reinterpret_cast<const float4*>(p);
            x[0] = v.x; x[V > 1 ? 1 : 0] = v.y; x[V > 2 ? 2 : 0] = v.z; x[V > 3 ? 3 : 0] = v.w;
        } else {
            x[0] = *p;
        }
    };
    auto put = [](float* p, const float (&x)[V]) {
        if (V == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[V > 1 ? 1 : 0], x[V > 2 ? 2 : 0], x[V > 3 ? 3 : 0]);
        else *p = x[0];
    };
    for (int j = lane * V; j < d; j += 32 * V)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= n) break;
            float q[V], k[V];
            fetch(qr + (size_t)i * Cq + j, q);
            fetch(kr + (size_t)i * Cq + j, k);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                qs[i] = fmaf(q[e], q[e], qs[i]);
                ks[i] = fmaf(k[e], k[e], ks[i]);
            }
        }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        qs[i] = qk_scale / sqrtf(warp_total(qs[i]) + unit_eps);
        ks[i] = 1.f / sqrtf(warp_total(ks[i]) + unit_eps);
    }
    float ab[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) ab[i] = 0.f;
    float* dst = prep + ((size_t)t * H + h) * 3 * d;
    const size_t step = (size_t)H * 3 * d;
    float* group = const_cast<float*>(delta_group(prep, tokens, H, d, t, b, h));
    for (int j = lane * V; j < d; j += 32 * V) {
        float g[4][V], kv[4][V], qv[4][V], e4[4][V], last[V], bias[V];
        fetch(dt_bias + (size_t)h * d + j, bias);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i < n) {
                fetch(qr + (size_t)i * Cq + j, qv[i]);
                fetch(kr + (size_t)i * Cq + j, kv[i]);
                fetch(ar + (size_t)i * ldag + j, g[i]);
            }
#pragma unroll
            for (int e = 0; e < V; ++e) {
                qv[i][e] = i < n ? qv[i][e] * qs[i] : 0.f;
                kv[i][e] = i < n ? kv[i][e] * ks[i] : 0.f;
                g[i][e] = i < n ? expf(-A * softplus_f32(g[i][e] + bias[e])) : 1.f;
            }
        }
#pragma unroll
        for (int e = 0; e < V; ++e) {
            // decays between two tokens, and the keys carried over them
            const float c10 = g[1][e], c21 = g[2][e], c32 = g[3][e], c20 = c10 * c21, c31 = c21 * c32, c30 = c20 * c32;
            const float k10 = c10 * kv[0][e], k20 = c20 * kv[0][e], k30 = c30 * kv[0][e], k21 = c21 * kv[1][e],
                        k31 = c31 * kv[1][e], k32 = c32 * kv[2][e];
            ab[0] = fmaf(kv[1][e], k10, ab[0]);
            ab[1] = fmaf(kv[2][e], k20, ab[1]);
            ab[2] = fmaf(kv[2][e], k21, ab[2]);
            ab[3] = fmaf(kv[3][e], k30, ab[3]);
            ab[4] = fmaf(kv[3][e], k31, ab[4]);
            ab[5] = fmaf(kv[3][e], k32, ab[5]);
            ab[6] = fmaf(qv[0][e], kv[0][e], ab[6]);
            ab[7] = fmaf(qv[1][e], k10, ab[7]);
            ab[8] = fmaf(qv[1][e], kv[1][e], ab[8]);
            ab[9] = fmaf(qv[2][e], k20, ab[9]);
            ab[10] = fmaf(qv[2][e], k21, ab[10]);
            ab[11] = fmaf(qv[2][e], kv[2][e], ab[11]);
            ab[12] = fmaf(qv[3][e], k30, ab[12]);
            ab[13] = fmaf(qv[3][e], k31, ab[13]);
            ab[14] = fmaf(qv[3][e], k32, ab[14]);
            ab[15] = fmaf(qv[3][e], kv[3][e], ab[15]);
            const float g1 = g[0][e] * g[1][e], g2 = g1 * g[2][e], g3 = g2 * g[3][e], all[4] = {g[0][e], g1, g2, g3};
            e4[0][e] = k30;
            e4[1][e] = k31;
            e4[2][e] = k32;
            e4[3][e] = kv[3][e];
            last[e] = g3;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                qv[i][e] *= all[i];
                kv[i][e] *= all[i];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < n) {
                put(dst + i * step + j, qv[i]);
                put(dst + i * step + d + j, kv[i]);
                put(dst + i * step + 2 * d + j, e4[i]);
            }
        put(group + j, last);
    }
    int first;
    fold_many<32, 16>(ab, lane, first);      // two neighbouring lanes hold the same sum
    if ((lane & 1) == 0) group[d + first] = ab[0];
}

// Shared memory: three stages of Gq[TT][DP] Gk[TT][DP] Ek[TT][DP] v[TT][VT] beta[TT] A, B[TT/4][16] G_3[TT/4][DP], then two
// tiles o[TT][VT].
template <int DS>
__global__ void __launch_bounds__(384, 1) delta_rule_kernel(float* __restrict__ o, const float* prep,
                                                         const float* vals, int ldv, const float* proj,
                                                         long long ldp, int beta_off, float* state,
                                                         const int* __restrict__ q_start, const int* __restrict__ slots, int tokens,
                                                         int H, int d, int dv, int TT, int stage, int cw, int vec) {
    pdl_wait();
    extern __shared__ __align__(16) float scan_smem[];
    constexpr int CGW = 32 / DS, DP = DS * kRowsPad, NR = DS * kRows;
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int VT = cw * CGW * 2, c_base = blockIdx.z * VT;
    const int slot = slots[b];
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 - t0 <= XB_FEW_TOKENS) pdl_launch_dependents();
    if (slot < 0 || t1 <= t0) return;
    const int ntiles = (t1 - t0 + TT - 1) / TT;
    float* so = scan_smem + kStages * stage;
    if (w >= cw) {
        // feeding warps: warp `pi` of `pw` takes tokens pi, pi + pw, ... of every tile
        const int pi = w - cw, pw = (blockDim.x >> 5) - cw;
        auto bring = [&](int tile) {
            float* sq = scan_smem + (tile % kStages) * stage;
            float* sk = sq + TT * DP;
            float* se = sk + TT * DP;
            float* sv = se + TT * DP;
            float* sbeta = sv + TT * VT;
            float* sab = sbeta + TT;
            float* slast = sab + TT * 4;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < ((nt + 3) & ~3); tt += pw) {
                const int len = tt < nt ? d : 0;         // tokens that fill up the last four: zeros
                const float* row = prep + ((size_t)(tb + tt) * H + h) * 3 * d;
                stage_rows(sq + tt * DP, row, len, NR, lane, vec);
                stage_rows(sk + tt * DP, row + d, len, NR, lane, vec);
                stage_rows(se + tt * DP, row + 2 * d, len, NR, lane, vec);
                if (tt >= nt) continue;
                stage_cols(sv + tt * VT, vals + (size_t)(tb + tt) * ldv + h * dv, c_base, dv, VT, lane, vec);
                if (lane == 0) scan_cp4(sbeta + tt, proj + (size_t)(tb + tt) * ldp + beta_off + h);
            }
            for (int grp = pi; grp * 4 < nt; grp += pw) {
                const float* src = delta_group(prep, tokens, H, d, tb + grp * 4, b, h);
                stage_rows(slast + grp * DP, src, d, NR, lane, vec);
                if (lane < 16) scan_cp4(sab + grp * 16 + lane, src + d + lane);
            }
        };
        auto finish = [&](int tile) {
            float* sbeta = scan_smem + (tile % kStages) * stage + 3 * TT * DP + TT * VT;
            const int nt = min(TT, t1 - t0 - tile * TT);
            scan_cp_land();
            if (lane == 0)
                for (int tt = pi; tt < nt; tt += pw) sbeta[tt] = sigmoid_exact(sbeta[tt]);
        };
        auto leave = [&](int tile) {
            const float* src = so + (tile & 1) * TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw)
                for (int c = lane; c < VT; c += 32)
                    if (c_base + c < dv) o[((size_t)(tb + tt) * H + h) * dv + c_base + c] = src[tt * VT + c];
        };
        feed(ntiles, bring, finish, leave);
        leave(ntiles - 1);
        return;
    }
    const int ds = lane / CGW, cl = (w * CGW + lane % CGW) * 2, v0 = c_base + cl;
    pair2 S0[kPairs], S1[kPairs];
    float* st = state + ((size_t)slot * H + h) * d * dv;
    auto at = [&](int j, int c) { return j < d && c < dv ? st[(size_t)j * dv + c] : 0.f; };
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int j = ds * kRows + 2 * i;
        S0[i] = pr_make(at(j, v0), at(j + 1, v0));
        S1[i] = pr_make(at(j, v0 + 1), at(j + 1, v0 + 1));
    }
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        const float* sq = scan_smem + (tile % kStages) * stage + ds * kRowsPad;
        const float* sk = sq + TT * DP;
        const float* se = sk + TT * DP;
        const float* sv = scan_smem + (tile % kStages) * stage + 3 * TT * DP;
        const float* sbeta = sv + TT * VT;
        const float* sab = sbeta + TT;
        const float* slast = sab + TT * 4 + ds * kRowsPad;
        sv += cl;
        float* out = so + (tile & 1) * TT * VT + cl;
        const int nt = min(TT, t1 - t0 - tile * TT);
        for (int tt = 0; tt < nt; tt += 4) {
            float pk[8], pq[8];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                pair2 kv[kPairs], qv[kPairs], k0 = 0ull, k1 = 0ull, q0 = 0ull, q1 = 0ull;
                load_pairs(sk + (tt + k) * DP, kv);
                load_pairs(sq + (tt + k) * DP, qv);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    k0 = pr_fma(S0[i], kv[i], k0);
                    k1 = pr_fma(S1[i], kv[i], k1);
                    q0 = pr_fma(S0[i], qv[i], q0);
                    q1 = pr_fma(S1[i], qv[i], q1);
                }
                pk[2 * k] = pr_sum(k0);
                pk[2 * k + 1] = pr_sum(k1);
                pq[2 * k] = pr_sum(q0);
                pq[2 * k + 1] = pr_sum(q1);
            }
            int first;
            fold_many<DS, 8>(pk, ds, first);
            const int n = fold_many<DS, 8>(pq, ds, first);
            spread_many<DS, 8>(pk, ds);
            float ab[16], u[4][2];
            {
                const float4* p4 = reinterpret_cast<const float4*>(sab + tt * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 x = p4[i];
                    ab[4 * i] = x.x; ab[4 * i + 1] = x.y; ab[4 * i + 2] = x.z; ab[4 * i + 3] = x.w;
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                // (a token that fills up the four has neither value nor beta: whatever lies there is not used)
                const bool real = tt + k < nt;
                const float beta = sbeta[tt + k];
                const float2 vv = *reinterpret_cast<const float2*>(sv + (tt + k) * VT);
                float r0 = vv.x - pk[2 * k], r1 = vv.y - pk[2 * k + 1];
#pragma unroll
                for (int j = 0; j < k; ++j) {
                    const float a = ab[k * (k - 1) / 2 + j];
                    r0 = fmaf(-a, u[j][0], r0);
                    r1 = fmaf(-a, u[j][1], r1);
                }
                u[k][0] = real ? beta * r0 : 0.f;
                u[k][1] = real ? beta * r1 : 0.f;
            }
            {
                pair2 g[kPairs];
                load_pairs(slast + (tt / 4) * DP, g);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    S0[i] = pr_mul(S0[i], g[i]);
                    S1[i] = pr_mul(S1[i], g[i]);
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                pair2 e[kPairs];
                load_pairs(se + (tt + k) * DP, e);
                const pair2 u0 = pr_make(u[k][0], u[k][0]), u1 = pr_make(u[k][1], u[k][1]);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    S0[i] = pr_fma(e[i], u0, S0[i]);
                    S1[i] = pr_fma(e[i], u1, S1[i]);
                }
            }
            if (fold_writes<DS, 8>(ds)) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        float add = 0.f;
#pragma unroll
                        for (int j = 0; j <= k; ++j) add = fmaf(ab[6 + k * (k + 1) / 2 + j], u[j][c], add);
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (i < n && first + i == 2 * k + c && tt + k < nt) out[(tt + k) * VT + c] = pq[i] + add;
                    }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        float w4[4];
        pr_split(S0[i], w4[0], w4[1]);
        pr_split(S1[i], w4[2], w4[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = ds * kRows + 2 * i + (e & 1), c = v0 + (e >> 1);
            if (j < d && c < dv) st[(size_t)j * dv + c] = w4[e];
        }
    }
}

// The delta rule where every request brings few tokens (delta_few): one at a time, with unit vectors and decays formed by the
// feeding warps, since a launch in front of it costs more than it saves.  With gS the decayed state, o = (gS)^T q + u (k . q).
// Shared memory: three stages of q[TT][DP] k[TT][DP] g[TT][DP] v[TT][VT] beta[TT] kq[TT], then two tiles o[TT][VT].
// One token of 16 heads of 128 x 128, 1 and 8 requests: 15 and 26 us with the kernel in front, 11 and 18 us so.  A small state's
// chain is short beside that kernel: 8 heads of 64 x 64, 32 requests of five tokens 28 and 15 us, eight of 40 tokens 28 and 20 us, one
// of 128 tokens 48 and 47 us, of 600 tokens 161 and 185 us; of 128 x 128, eight of 40 tokens 52 and 65 us.
constexpr int kFewTokensSmall = 96;
static inline bool delta_few(int longest, int d) { return longest <= (d <= 64 ? kFewTokensSmall : kFewTokens); }
template <int DS>
__global__ void __launch_bounds__(384, 1) delta_few_kernel(float* __restrict__ o, const float* qkv, int Cq,
                                                        const float* proj, long long ldp, int beta_off,
                                                        const float* ag, long long ldag,
                                                        const float* __restrict__ dt_bias, const float* __restrict__ A_log,
                                                        float* state, const int* __restrict__ q_start,
                                                        const int* __restrict__ slots, int H, int G, int d, int dv,
                                                        float unit_eps, int TT, int stage, int cw, int vec) {
    pdl_wait();
    extern __shared__ __align__(16) float scan_smem[];
    constexpr int CGW = 32 / DS, DP = DS * kRowsPad, NR = DS * kRows;
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int VT = cw * CGW * 2, c_base = blockIdx.z * VT;
    const int slot = slots[b];
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 - t0 <= XB_FEW_TOKENS) pdl_launch_dependents();
    if (slot < 0 || t1 <= t0) return;
    const int kvh = h / (H / G);
    const int ntiles = (t1 - t0 + TT - 1) / TT;
    float* so = scan_smem + kStages * stage;
    if (w >= cw) {
        // feeding warps: warp `pi` of `pw` takes tokens pi, pi + pw, ... of every tile
        const int pi = w - cw, pw = (blockDim.x >> 5) - cw;
        const float A = expf(A_log[h]);
        const float qk_scale = 1.f / sqrtf((float)d);
        const float* bias = dt_bias + (size_t)h * d;
        auto bring = [&](int tile) {
            float* sq = scan_smem + (tile % kStages) * stage;
            float* sk = sq + TT * DP;
            float* sg = sk + TT * DP;
            float* sv = sg + TT * DP;
            float* sbeta = sv + TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw) {
                const float* row = qkv + (size_t)(tb + tt) * Cq;
                stage_rows(sq + tt * DP, row + kvh * d, d, NR, lane, vec);
                stage_rows(sk + tt * DP, row + (G + kvh) * d, d, NR, lane, vec);
                stage_rows(sg + tt * DP, ag + (size_t)(tb + tt) * ldag + h * d, d, NR, lane, vec);
                stage_cols(sv + tt * VT, row + 2 * G * d + h * dv, c_base, dv, VT, lane, vec);
                if (lane == 0) scan_cp4(sbeta + tt, proj + (size_t)(tb + tt) * ldp + beta_off + h);
            }
        };
        auto finish = [&](int tile) {
            float* sq = scan_smem + (tile % kStages) * stage;
            float* sk = sq + TT * DP;
            float* sg = sk + TT * DP;
            float* sbeta = sg + TT * DP + TT * VT;
            const int nt = min(TT, t1 - t0 - tile * TT);
            scan_cp_land();
            for (int tt = pi; tt < nt; tt += pw) {
                float* q = sq + tt * DP;
                float* k = sk + tt * DP;
                float* gd = sg + tt * DP;
                float qq = 0.f, kk = 0.f;
                for (int j = lane; j < d; j += 32) {
                    const int at = padded_row(j);
                    qq = fmaf(q[at], q[at], qq);
                    kk = fmaf(k[at], k[at], kk);
                }
                qq = warp_total(qq);
                kk = warp_total(kk);
                const float qs = qk_scale / sqrtf(qq + unit_eps), ks = 1.f / sqrtf(kk + unit_eps);
                float kq = 0.f;
                for (int j = lane; j < d; j += 32) {
                    const int at = padded_row(j);
                    const float qn = q[at] * qs, kn = k[at] * ks;
                    q[at] = qn;
                    k[at] = kn;
                    kq = fmaf(kn, qn, kq);
                    gd[at] = expf(-A * softplus_f32(gd[at] + bias[j]));
                }
                kq = warp_total(kq);
                if (lane == 0) {
                    sbeta[TT + tt] = kq;
                    sbeta[tt] = sigmoid_exact(sbeta[tt]);
                }
            }
        };
        auto leave = [&](int tile) {
            const float* src = so + (tile & 1) * TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw)
                for (int c = lane; c < VT; c += 32)
                    if (c_base + c < dv) o[((size_t)(tb + tt) * H + h) * dv + c_base + c] = src[tt * VT + c];
        };
        feed(ntiles, bring, finish, leave);
        leave(ntiles - 1);
        return;
    }
    const int ds = lane / CGW, cl = (w * CGW + lane % CGW) * 2, v0 = c_base + cl;
    float S0[kRows], S1[kRows];
    float* st = state + ((size_t)slot * H + h) * d * dv;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int j = ds * kRows + r;
        S0[r] = j < d && v0 < dv ? st[(size_t)j * dv + v0] : 0.f;
        S1[r] = j < d && v0 + 1 < dv ? st[(size_t)j * dv + v0 + 1] : 0.f;
    }
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        const float* sq = scan_smem + (tile % kStages) * stage + ds * kRowsPad;
        const float* sk = sq + TT * DP;
        const float* sg = sk + TT * DP;
        const float* sv = scan_smem + (tile % kStages) * stage + 3 * TT * DP;
        const float* sbeta = sv + TT * VT;
        sv += cl;
        float* out = so + (tile & 1) * TT * VT + cl;
        const int nt = min(TT, t1 - t0 - tile * TT);
        for (int tt = 0; tt < nt; ++tt, sq += DP, sk += DP, sg += DP, sv += VT, out += VT) {
            const float beta = sbeta[tt];
            const float2 vv = *reinterpret_cast<const float2*>(sv);
            const float4* qp = reinterpret_cast<const float4*>(sq);
            const float4* kp = reinterpret_cast<const float4*>(sk);
            const float4* gp = reinterpret_cast<const float4*>(sg);
            float kr[kRows], a[4] = {0.f, 0.f, 0.f, 0.f};     // (gS)^T k and (gS)^T q of the two columns
#pragma unroll
            for (int i = 0; i < kRows / 4; ++i) {
                const float4 g4 = gp[i], k4 = kp[i], q4 = qp[i];
                const float ge[4] = {g4.x, g4.y, g4.z, g4.w}, ke[4] = {k4.x, k4.y, k4.z, k4.w}, qe[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = 4 * i + e;
                    S0[r] *= ge[e];
                    S1[r] *= ge[e];
                    a[0] = fmaf(S0[r], ke[e], a[0]);
                    a[1] = fmaf(S1[r], ke[e], a[1]);
                    a[2] = fmaf(S0[r], qe[e], a[2]);
                    a[3] = fmaf(S1[r], qe[e], a[3]);
                    kr[r] = ke[e];
                }
            }
#pragma unroll
            for (int bit = 16; bit >= CGW; bit >>= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], bit);
            const float u0 = beta * (vv.x - a[0]), u1 = beta * (vv.y - a[1]);
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                S0[r] = fmaf(kr[r], u0, S0[r]);
                S1[r] = fmaf(kr[r], u1, S1[r]);
            }
            if (ds == 0) *reinterpret_cast<float2*>(out) = make_float2(fmaf(u0, sbeta[TT + tt], a[2]), fmaf(u1, sbeta[TT + tt], a[3]));
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const int j = ds * kRows + r;
        if (j < d && v0 < dv) st[(size_t)j * dv + v0] = S0[r];
        if (j < d && v0 + 1 < dv) st[(size_t)j * dv + v0 + 1] = S1[r];
    }
}

// proj[t] holds q (H*d from column 0), k (H*d behind it) and v (H*dv behind that) of a token; alpha[t] the decay of
// every (head, key channel).  state [slots, H, d, dv].  o [T, H*dv] = scale * S^T q after the token's own write.  Shared
// memory: three stages of q[TT][DP] k[TT][DP] alpha[TT][DP] v[TT][VT], then two tiles o[TT][VT].
template <int DS, bool FEW>
__global__ void __launch_bounds__(FEW ? 256 : 384, FEW ? 2 : 1) linear_scan_kernel(float* __restrict__ o, const float* proj,
                                                             long long ldp, const float* alpha,
                                                             float* state, const int* __restrict__ q_start,
                                                             const int* __restrict__ slots, int H, int d, int dv, float scale,
                                                             int TT, int stage, int cw, int vec) {
    pdl_wait();
    extern __shared__ __align__(16) float scan_smem[];
    constexpr int CGW = 32 / DS, DP = DS * kRowsPad, NR = DS * kRows;
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int VT = cw * CGW * 2, c_base = blockIdx.z * VT;
    const int slot = slots[b];
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 - t0 <= XB_FEW_TOKENS) pdl_launch_dependents();
    if (slot < 0 || t1 <= t0) return;
    const int ntiles = (t1 - t0 + TT - 1) / TT;
    float* so = scan_smem + kStages * stage;
    if (w >= cw) {
        // feeding warps: warp `pi` of `pw` takes tokens pi, pi + pw, ... of every tile
        const int pi = w - cw, pw = (blockDim.x >> 5) - cw;
        auto bring = [&](int tile) {
            float* sq = scan_smem + (tile % kStages) * stage;
            float* sk = sq + TT * DP;
            float* sa = sk + TT * DP;
            float* sv = sa + TT * DP;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw) {
                const float* row = proj + (size_t)(tb + tt) * ldp;
                stage_rows(sq + tt * DP, row + h * d, d, NR, lane, vec);
                stage_rows(sk + tt * DP, row + (H + h) * d, d, NR, lane, vec);
                stage_rows(sa + tt * DP, alpha + ((size_t)(tb + tt) * H + h) * d, d, NR, lane, vec);
                stage_cols(sv + tt * VT, row + 2 * H * d + h * dv, c_base, dv, VT, lane, vec);
            }
        };
        auto finish = [&](int) { scan_cp_land(); };
        auto leave = [&](int tile) {
            const float* src = so + (tile & 1) * TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw)
                for (int c = lane; c < VT; c += 32)
                    if (c_base + c < dv) o[((size_t)(tb + tt) * H + h) * dv + c_base + c] = src[tt * VT + c];
        };
        feed(ntiles, bring, finish, leave);
        leave(ntiles - 1);
        return;
    }
    const int ds = lane / CGW, cl = (w * CGW + lane % CGW) * 2, v0 = c_base + cl;
    pair2 S0[kPairs], S1[kPairs];
    float* st = state + ((size_t)slot * H + h) * d * dv;
    auto at = [&](int j, int c) { return j < d && c < dv ? st[(size_t)j * dv + c] : 0.f; };
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int j = ds * kRows + 2 * i;
        S0[i] = pr_make(at(j, v0), at(j + 1, v0));
        S1[i] = pr_make(at(j, v0 + 1), at(j + 1, v0 + 1));
    }
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        const float* sq = scan_smem + (tile % kStages) * stage + ds * kRowsPad;
        const float* sk = sq + TT * DP;
        const float* sa = sk + TT * DP;
        const float* sv = scan_smem + (tile % kStages) * stage + 3 * TT * DP + cl;
        float* out = so + (tile & 1) * TT * VT + cl;
        const int nt = min(TT, t1 - t0 - tile * TT);
        auto group = [&](int tt, auto grp) {        // as in selective_scan_kernel
            constexpr int NG = decltype(grp)::tokens;
            constexpr bool whole = decltype(grp)::whole;
            float v[2 * NG];
#pragma unroll
            for (int k = 0; k < NG; ++k) {
                v[2 * k] = v[2 * k + 1] = 0.f;
                if (!whole && tt + k >= nt) continue;
                const float2 vv = *reinterpret_cast<const float2*>(sv + (tt + k) * VT);
                pair2 q[kPairs], kv[kPairs], a0 = 0ull, a1 = 0ull;
                load_pairs(sq + (tt + k) * DP, q);
                load_pairs(sk + (tt + k) * DP, kv);
                const pair2 x0 = pr_make(vv.x, vv.x), x1 = pr_make(vv.y, vv.y);
                pair2 keep[kPairs];
                load_pairs(sa + (tt + k) * DP, keep);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    S0[i] = pr_fma(keep[i], S0[i], pr_mul(kv[i], x0));
                    S1[i] = pr_fma(keep[i], S1[i], pr_mul(kv[i], x1));
                    a0 = pr_fma(S0[i], q[i], a0);
                    a1 = pr_fma(S1[i], q[i], a1);
                }
                v[2 * k] = pr_sum(a0);
                v[2 * k + 1] = pr_sum(a1);
            }
            int first;
            const int n = fold_many<DS, 2 * NG>(v, ds, first);
            if (fold_writes<DS, 2 * NG>(ds)) {
#pragma unroll
                for (int i = 0; i < 2 * NG; ++i) {
                    const int k = (first + i) >> 1, c = (first + i) & 1;
                    if (i < n && (whole || tt + k < nt)) out[(tt + k) * VT + c] = scale * v[i];
                }
            }
        };
        if constexpr (FEW) {
            for (int tt = 0; tt < nt; ++tt) group(tt, Group<1, true>{});
        } else {
            int done = 0;
            for (; done + 4 <= nt; done += 4) group(done, Group<4, true>{});
            if (done < nt) group(done, Group<4, false>{});
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        float u[4];
        pr_split(S0[i], u[0], u[1]);
        pr_split(S1[i], u[2], u[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = ds * kRows + 2 * i + (e & 1), c = v0 + (e >> 1);
            if (j < d && c < dv) st[(size_t)j * dv + c] = u[e];
        }
    }
}

// proj[t] holds q (H*d from column 0), k (H*d behind it), v (H*dv behind that) and at gate_off the input gates' and the
// forget gates' pre-activations (H each, without their biases).  With i = cap tanh((z_i + b_i) / cap) and
// f = -softplus(-cap tanh((z_f + b_f) / cap)):
//   m' = max(f + m, i);  a = e^(f + m - m');  b = e^(i - m');   S <- a S + b k v^T;   n <- a n + b k
//   o[t, h*dv ..] = scale S^T q,   div[t, h] = max(|scale n . q|, e^(-m')) + div_eps          after the token's own write
// state_s [slots, H, d, dv], state_n [slots, H, d].  The running maximum m is read by every block of a head but left by
// one of them, so it has two places: state_m [slots, H, 2, 2] holds (tokens it stands behind, m) twice; a step reads the
// place that stands behind its start and writes the other one.  Zeros are a request's start.
// Shared memory: three stages of q[TT][DP] k[TT][DP] v[TT][VT] a[TT] b[TT] e^(-m')[TT], then two tiles o[TT][VT].  Besides
// the computing and the feeding warps there is one (warp `cw`) that carries n where the block has the head's first
// columns; the first feeding warp works out the gates, a lane per token, and walks m over the tile.
template <int DS, bool FEW>
__global__ void __launch_bounds__(384, 1) matrix_memory_kernel(
    float* __restrict__ o, float* __restrict__ div, const float* proj, long long ldp, int gate_off,
    const float* __restrict__ bi, const float* __restrict__ bf, float cap, float* state_s,
    float* state_n, float* state_m, const int* __restrict__ q_start, const int* __restrict__ start_pos,
    const int* __restrict__ slots, int H, int d, int dv, float scale, float div_eps, int TT, int stage, int cw, int vec) {
    pdl_wait();
    extern __shared__ __align__(16) float scan_smem[];
    constexpr int CGW = 32 / DS, DP = DS * kRowsPad, NR = DS * kRows;
    const int b = blockIdx.x, h = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int VT = cw * CGW * 2, c_base = blockIdx.z * VT;
    const int slot = slots[b];
    const int t0 = q_start[b], t1 = q_start[b + 1];
    if (t1 - t0 <= XB_FEW_TOKENS) pdl_launch_dependents();
    if (slot < 0 || t1 <= t0) return;
    const int ntiles = (t1 - t0 + TT - 1) / TT;
    float* so = scan_smem + kStages * stage;
    if (w > cw) {
        // feeding warps: warp `pi` of `pw` takes tokens pi, pi + pw, ... of every tile
        const int pi = w - cw - 1, pw = (blockDim.x >> 5) - cw - 1;
        float* place = state_m + ((size_t)slot * H + h) * 4;
        const float at_start = (float)start_pos[b];
        const int from = place[0] == at_start ? 0 : 1;
        float m = place[2 * from + 1];
        const float b_i = bi[h], b_f = bf[h];
        float zi_next = 0.f, zf_next = 0.f;
        auto gates = [&](int tile) {
            const int tt = tile * TT + lane;
            if (pi == 0 && lane < TT && t0 + tt < t1) {
                const float* g = proj + (size_t)(t0 + tt) * ldp + gate_off + h;
                zi_next = g[0];
                zf_next = g[H];
            }
        };
        gates(0);
        auto bring = [&](int tile) {
            float* sq = scan_smem + (tile % kStages) * stage;
            float* sk = sq + TT * DP;
            float* sv = sk + TT * DP;
            float* sg = sv + TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            const float zi = zi_next, zf = zf_next;      // asked for a tile ago
            gates(tile + 1);
            for (int tt = pi; tt < nt; tt += pw) {
                const float* row = proj + (size_t)(tb + tt) * ldp;
                stage_rows(sq + tt * DP, row + h * d, d, NR, lane, vec);
                stage_rows(sk + tt * DP, row + (H + h) * d, d, NR, lane, vec);
                stage_cols(sv + tt * VT, row + 2 * H * d + h * dv, c_base, dv, VT, lane, vec);
            }
            if (pi == 0) {
                const float gi = cap * tanhf((zi + b_i) / cap), y = cap * tanhf((zf + b_f) / cap);
                const float gf = fminf(y, 0.f) - log1pf(expf(-fabsf(y)));      // log of the sigmoid
                float before = m, after = m;
                for (int tt = 0; tt < nt; ++tt) {
                    const float f_t = __shfl_sync(0xffffffffu, gf, tt), i_t = __shfl_sync(0xffffffffu, gi, tt);
                    const float next = fmaxf(f_t + m, i_t);
                    if (lane == tt) {
                        before = m;
                        after = next;
                    }
                    m = next;
                }
                if (lane < nt) {
                    sg[lane] = expf(gf + before - after);
                    sg[TT + lane] = expf(gi - after);
                    sg[2 * TT + lane] = expf(-after);
                }
            }
        };
        auto finish = [&](int) { scan_cp_land(); };
        auto leave = [&](int tile) {
            const float* src = so + (tile & 1) * TT * VT;
            const int tb = t0 + tile * TT, nt = min(TT, t1 - tb);
            for (int tt = pi; tt < nt; tt += pw)
                for (int c = lane; c < VT; c += 32)
                    if (c_base + c < dv) o[((size_t)(tb + tt) * H + h) * dv + c_base + c] = src[tt * VT + c];
        };
        feed(ntiles, bring, finish, leave);
        leave(ntiles - 1);
        if (pi == 0 && lane == 0 && blockIdx.z == 0) {
            place[2 * (from ^ 1)] = at_start + (float)(t1 - t0);
            place[2 * (from ^ 1) + 1] = m;
        }
        return;
    }
    if (w == cw) {
        // n and the divisors; a lane keeps rows lane, lane + 32, ...
        constexpr int NN = (NR + 31) / 32;
        const bool mine = blockIdx.z == 0;
        float n[NN];
        float* sn = state_n + ((size_t)slot * H + h) * d;
#pragma unroll
        for (int r = 0; r < NN; ++r) n[r] = mine && lane + 32 * r < d ? sn[lane + 32 * r] : 0.f;
        __syncthreads();
        for (int tile = 0; tile < ntiles; ++tile) {
            if (mine) {
                const float* sq = scan_smem + (tile % kStages) * stage;
                const float* sk = sq + TT * DP;
                const float* sg = scan_smem + (tile % kStages) * stage + 2 * TT * DP + TT * VT;
                const int nt = min(TT, t1 - t0 - tile * TT);
                float* dst = div + (size_t)(t0 + tile * TT) * H + h;
#pragma unroll 4
                for (int tt = 0; tt < nt; ++tt) {
                    const float a = sg[tt], bb = sg[TT + tt];
                    float acc = 0.f;
#pragma unroll
                    for (int r = 0; r < NN; ++r) {
                        if (lane + 32 * r >= NR) break;
                        const int at = tt * DP + padded_row(lane + 32 * r);
                        n[r] = fmaf(a, n[r], bb * sk[at]);
                        acc = fmaf(n[r], sq[at], acc);
                    }
                    acc = warp_total(acc);
                    if (lane == 0) dst[(size_t)tt * H] = fmaxf(fabsf(scale * acc), sg[2 * TT + tt]) + div_eps;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < NN; ++r)
            if (mine && lane + 32 * r < d) sn[lane + 32 * r] = n[r];
        return;
    }
    const int ds = lane / CGW, cl = (w * CGW + lane % CGW) * 2, v0 = c_base + cl;
    pair2 S0[kPairs], S1[kPairs];
    float* st = state_s + ((size_t)slot * H + h) * d * dv;
    auto at = [&](int j, int c) { return j < d && c < dv ? st[(size_t)j * dv + c] : 0.f; };
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        const int j = ds * kRows + 2 * i;
        S0[i] = pr_make(at(j, v0), at(j + 1, v0));
        S1[i] = pr_make(at(j, v0 + 1), at(j + 1, v0 + 1));
    }
    __syncthreads();
    for (int tile = 0; tile < ntiles; ++tile) {
        const float* sq = scan_smem + (tile % kStages) * stage + ds * kRowsPad;
        const float* sk = sq + TT * DP;
        const float* sv = scan_smem + (tile % kStages) * stage + 2 * TT * DP;
        const float* sg = sv + TT * VT;
        sv += cl;
        float* out = so + (tile & 1) * TT * VT + cl;
        const int nt = min(TT, t1 - t0 - tile * TT);
        auto group = [&](int tt, auto grp) {        // as in selective_scan_kernel
            constexpr int NG = decltype(grp)::tokens;
            constexpr bool whole = decltype(grp)::whole;
            float v[2 * NG];
#pragma unroll
            for (int k = 0; k < NG; ++k) {
                v[2 * k] = v[2 * k + 1] = 0.f;
                if (!whole && tt + k >= nt) continue;
                const float2 vv = *reinterpret_cast<const float2*>(sv + (tt + k) * VT);
                pair2 q[kPairs], kv[kPairs], a0 = 0ull, a1 = 0ull;
                load_pairs(sq + (tt + k) * DP, q);
                load_pairs(sk + (tt + k) * DP, kv);
                const float dec = sg[tt + k], in = sg[TT + tt + k];
                const pair2 x0 = pr_make(in * vv.x, in * vv.x), x1 = pr_make(in * vv.y, in * vv.y), keep = pr_make(dec, dec);
#pragma unroll
                for (int i = 0; i < kPairs; ++i) {
                    S0[i] = pr_fma(keep, S0[i], pr_mul(kv[i], x0));
                    S1[i] = pr_fma(keep, S1[i], pr_mul(kv[i], x1));
                    a0 = pr_fma(S0[i], q[i], a0);
                    a1 = pr_fma(S1[i], q[i], a1);
                }
                v[2 * k] = pr_sum(a0);
                v[2 * k + 1] = pr_sum(a1);
            }
            int first;
            const int n = fold_many<DS, 2 * NG>(v, ds, first);
            if (fold_writes<DS, 2 * NG>(ds)) {
#pragma unroll
                for (int i = 0; i < 2 * NG; ++i) {
                    const int k = (first + i) >> 1, c = (first + i) & 1;
                    if (i < n && (whole || tt + k < nt)) out[(tt + k) * VT + c] = scale * v[i];
                }
            }
        };
        if constexpr (FEW) {
            for (int tt = 0; tt < nt; ++tt) group(tt, Group<1, true>{});
        } else {
            int done = 0;
            for (; done + 4 <= nt; done += 4) group(done, Group<4, true>{});
            if (done < nt) group(done, Group<4, false>{});
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
        float u[4];
        pr_split(S0[i], u[0], u[1]);
        pr_split(S1[i], u[2], u[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int j = ds * kRows + 2 * i + (e & 1), c = v0 + (e >> 1);
            if (j < d && c < dv) st[(size_t)j * dv + c] = u[e];
        }
    }
}

// alpha[t, c] = sigmoid(z)^(1 / tau) = exp(-softplus(-z) / tau),  z = bias[c] + sum_r w[c, r] low[t, r].  low is a
// column range of wider float32 rows.  A block takes a tile of tokens and 128 channels, a thread one channel of all its
// tokens; both operands pass through shared memory, so that memory is read in order; r in order for every output.
constexpr int kDecayTokens = 16, kDecayRanks = 16, kDecayChannels = 128;
__global__ void __launch_bounds__(kDecayChannels) low_rank_decay_kernel(float* __restrict__ alpha, const float* low,
                                                                        long long ldl, const float* __restrict__ w,
                                                                        const float* __restrict__ bias, int tokens, int C, int R,
                                                                        float inv_tau) {
    pdl_overlap_few();
    __shared__ __align__(16) float sl[kDecayRanks][kDecayTokens];
    __shared__ float sw[kDecayRanks][kDecayChannels + 1];
    const int tb = blockIdx.x * kDecayTokens, nt = min(kDecayTokens, tokens - tb);
    const int c0 = blockIdx.y * kDecayChannels, c = c0 + threadIdx.x;
    float z[kDecayTokens];
    const float b = c < C ? bias[c] : 0.f;
#pragma unroll
    for (int i = 0; i < kDecayTokens; ++i) z[i] = b;
    for (int r0 = 0; r0 < R; r0 += kDecayRanks) {
        if (r0 > 0) __syncthreads();
        for (int i = threadIdx.x; i < kDecayRanks * kDecayTokens; i += kDecayChannels) {
            const int tt = i / kDecayRanks, r = i % kDecayRanks;
            sl[r][tt] = (tt < nt && r0 + r < R) ? low[(size_t)(tb + tt) * ldl + r0 + r] : 0.f;
        }
        for (int i = threadIdx.x; i < kDecayRanks * kDecayChannels; i += kDecayChannels) {
            const int cc = i / kDecayRanks, r = i % kDecayRanks;
            sw[r][cc] = (c0 + cc < C && r0 + r < R) ? w[(size_t)(c0 + cc) * R + r0 + r] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kDecayRanks; ++r) {
            const float wv = sw[r][threadIdx.x];
#pragma unroll
            for (int i = 0; i < kDecayTokens; i += 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(&sl[r][i]);
                z[i] = fmaf(wv, l4.x, z[i]);
                z[i + 1] = fmaf(wv, l4.y, z[i + 1]);
                z[i + 2] = fmaf(wv, l4.z, z[i + 2]);
                z[i + 3] = fmaf(wv, l4.w, z[i + 3]);
            }
        }
    }
    if (c >= C) return;
#pragma unroll
    for (int i = 0; i < kDecayTokens; ++i)
        if (i < nt) {
            const float sp = fmaxf(-z[i], 0.f) + log1pf(expf(-fabsf(z[i])));      // softplus(-z), for any z without a branch
            alpha[(size_t)(tb + i) * C + c] = expf(-sp * inv_tau);
        }
}

// Row groups per column pair: the smallest power of two with DS * kRows >= rows.
static inline int scan_row_groups(int rows) {
    int ds = 1;
    while (ds * kRows < rows) ds *= 2;
    return ds;
}

// Computing warps per block: enough to cover the columns (at most 8; 4 where two blocks are to share a processor), fewer (down to
// 2) while the grid would leave a third of the processors idle and the finer one still runs as one block per processor.  Every
// block of a head repeats the feeding warps' copies, so column tiles are not cut finer than that.
static inline int scan_warps(int cols, int ds, long long heads_total, int most = 8) {
    const int per_warp = (32 / ds) * 2;
    int warps = 1;
    while (warps < most && warps * per_warp < cols) warps *= 2;
    auto blocks = [&](int n) { return heads_total * ((cols + n * per_warp - 1) / (n * per_warp)); };
    while (warps > 2 && blocks(warps) < 100 && blocks(warps / 2) <= 148) warps /= 2;      // (a block fills an SM)
    return warps;
}

static inline bool scan_aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Floats of one stage (`vectors` row vectors and a few scalars per token beside the column tile), rounded so that
// the stages stay 16-byte aligned; the tile shrinks until they and two output tiles fit.
static inline void scan_tile(int vectors, int ds, int vt, int& tt, int& stage, size_t& bytes, int scalars = 2) {
    for (tt = kScanTile;; tt /= 2) {
        stage = (tt * (vectors * ds * kRowsPad + vt + scalars) + 3) & ~3;
        bytes = ((size_t)kStages * stage + (size_t)2 * tt * vt) * sizeof(float);
        if (bytes <= 200 * 1024 || tt == 1) return;
    }
}

template <typename K>
static inline int scan_smem_opt_in(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return 0;
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

#define XB_SCAN_DISPATCH(KERNEL, DSV, ...)                                                      \
    switch (DSV) {                                                                              \
        case 1: XB_SCAN_LAUNCH((KERNEL<1>), __VA_ARGS__) break;                                 \
        case 2: XB_SCAN_LAUNCH((KERNEL<2>), __VA_ARGS__) break;                                 \
        case 4: XB_SCAN_LAUNCH((KERNEL<4>), __VA_ARGS__) break;                                 \
        case 8: XB_SCAN_LAUNCH((KERNEL<8>), __VA_ARGS__) break;                                 \
        case 16: XB_SCAN_LAUNCH((KERNEL<16>), __VA_ARGS__) break;                               \
        default: XB_SCAN_LAUNCH((KERNEL<32>), __VA_ARGS__) break;                               \
    }
#define XB_SCAN_DISPATCH_FEW(KERNEL, DSV, FEW, ...)                                             \
    switch ((DSV) * 2 + ((FEW) ? 1 : 0)) {                                                      \
        case 2: XB_SCAN_LAUNCH((KERNEL<1, false>), __VA_ARGS__) break;                          \
        case 3: XB_SCAN_LAUNCH((KERNEL<1, true>), __VA_ARGS__) break;                           \
        case 4: XB_SCAN_LAUNCH((KERNEL<2, false>), __VA_ARGS__) break;                          \
        case 5: XB_SCAN_LAUNCH((KERNEL<2, true>), __VA_ARGS__) break;                           \
        case 8: XB_SCAN_LAUNCH((KERNEL<4, false>), __VA_ARGS__) break;                          \
        case 9: XB_SCAN_LAUNCH((KERNEL<4, true>), __VA_ARGS__) break;                           \
        case 16: XB_SCAN_LAUNCH((KERNEL<8, false>), __VA_ARGS__) break;                         \
        case 17: XB_SCAN_LAUNCH((KERNEL<8, true>), __VA_ARGS__) break;                          \
        case 32: XB_SCAN_LAUNCH((KERNEL<16, false>), __VA_ARGS__) break;                        \
        case 33: XB_SCAN_LAUNCH((KERNEL<16, true>), __VA_ARGS__) break;                         \
        case 65: XB_SCAN_LAUNCH((KERNEL<32, true>), __VA_ARGS__) break;                         \
        default: XB_SCAN_LAUNCH((KERNEL<32, false>), __VA_ARGS__) break;                        \
    }
#define XB_SCAN_LAUNCH(K, ...)                                  \
    {                                                           \
        const int rc = scan_smem_opt_in(K, bytes);              \
        if (rc) return rc;                                      \
        xb_launch_few(K, dim3(grid), dim3(threads), bytes, stream, __VA_ARGS__); \
    }

// `longest`, here and below: tokens of the request that brings most, as far as the caller knows; only the choice between the
// forms of a kernel depends on it.
XB_EXPORT int xb_selective_scan(float* y, const float* xbc, int C, const float* proj, long long ldp, int dt_off,
                                const float* dt_bias, const float* A_log, const float* Dv, float* state, const int* q_start,
                                const int* slots, int entries, int longest, int H, int P, int N, int G, cudaStream_t stream) {
    if (entries <= 0) return 0;
    if (N < 1 || N > 32 * kRows || P < 1 || G < 1 || H % G || H > 65535) return (int)cudaErrorInvalidValue;
    const int ds = scan_row_groups(N);
    const int warps = scan_warps(P, ds, (long long)entries * H, longest <= kFewTokens ? 4 : 8);
    const int vt = warps * (32 / ds) * 2;
    int tt, stage;
    size_t bytes;
    scan_tile(2, ds, vt, tt, stage, bytes);
    const dim3 grid(entries, H, (P + vt - 1) / vt);
    const int threads = (warps + 4) * 32;  // four feeding warps
    const int vec = scan_aligned16(xbc) && C % 4 == 0 && P % 4 == 0 && N % 4 == 0 && vt % 4 == 0;
    XB_SCAN_DISPATCH_FEW(selective_scan_kernel, ds, longest <= kFewTokens, y, xbc, C, proj, ldp, dt_off, dt_bias, A_log, Dv, state, q_start, slots, H, P, N,
                     G, tt, stage, warps, vec)
    return xb_launch_status();
}

// Floats of `prep` for that many tokens and entries (none where every request brings few).
XB_EXPORT long long xb_delta_prep_floats(int tokens, int entries, int longest, int H, int d) {
    return delta_few(longest, d) ? 0 : (long long)tokens * H * 3 * d + (long long)(tokens / 4 + entries + 1) * H * (d + 16);
}

XB_EXPORT int xb_delta_rule(float* o, const float* qkv, int Cq, const float* proj, long long ldp, int beta_off, const float* ag,
                            long long ldag, const float* dt_bias, const float* A_log, float* state, const int* q_start,
                            const int* slots, int entries, int tokens, int longest, int H, int G, int d, int dv, float unit_eps,
                            float* prep, cudaStream_t stream) {
    if (entries <= 0 || tokens <= 0) return 0;
    const bool few = delta_few(longest, d);
    if (d < 1 || d > 32 * kRows || dv < 1 || G < 1 || H % G || H > 65535 || (!few && !prep)) return (int)cudaErrorInvalidValue;
    const int ds = scan_row_groups(d);
    const int warps = scan_warps(dv, ds, (long long)entries * H);
    const int vt = warps * (32 / ds) * 2;
    int tt, stage;
    size_t bytes;
    if (few) {
        scan_tile(3, ds, vt, tt, stage, bytes);
        const dim3 grid(entries, H, (dv + vt - 1) / vt);
        // the unit vectors and decays are the feeding warps' work: eight of them where the block has room, else four
        const int threads = (warps + (warps <= 4 ? 8 : 4)) * 32;
        const int vec = scan_aligned16(qkv) && scan_aligned16(ag) && Cq % 4 == 0 && ldag % 4 == 0 && d % 4 == 0 && dv % 4 == 0 &&
                        vt % 4 == 0;
        XB_SCAN_DISPATCH(delta_few_kernel, ds, o, qkv, Cq, proj, ldp, beta_off, ag, ldag, dt_bias, A_log, state, q_start, slots, H,
                         G, d, dv, unit_eps, tt, stage, warps, vec)
        return xb_launch_status();
    }
    scan_tile(3, ds, vt, tt, stage, bytes, 5 + ds * kRowsPad / 4);      // beta, A and B, a quarter of a row vector
    if (tt < 4) return (int)cudaErrorInvalidValue;                       // (a tile holds whole groups of four tokens)
    // every request adds at most one group of fewer than four tokens
    const bool fours = scan_aligned16(prep) && scan_aligned16(qkv) && scan_aligned16(ag) && scan_aligned16(dt_bias) && Cq % 4 == 0 &&
                       ldag % 4 == 0 && d % 4 == 0;
    const auto prepare = fours ? delta_prepare_kernel<4> : delta_prepare_kernel<1>;
    xb_launch_few(prepare, dim3(dim3(tokens / 4 + entries, (H + 3) / 4)), dim3(128), 0, stream, prep, qkv, Cq, ag, ldag, dt_bias, A_log, q_start, entries,
                                                                         tokens, H, G, d, unit_eps);
    const int rc0 = xb_launch_status();
    if (rc0) return rc0;
    const dim3 grid(entries, H, (dv + vt - 1) / vt);
    const int threads = (warps + 4) * 32;  // four feeding warps: they only copy
    const float* vals = qkv + 2 * G * d;
    const int vec = scan_aligned16(prep) && scan_aligned16(vals) && Cq % 4 == 0 && d % 4 == 0 && dv % 4 == 0 && vt % 4 == 0;
    XB_SCAN_DISPATCH(delta_rule_kernel, ds, o, prep, vals, Cq, proj, ldp, beta_off, state, q_start, slots, tokens, H, d, dv, tt, stage,
                     warps, vec)
    return xb_launch_status();
}

XB_EXPORT int xb_linear_scan(float* o, const float* proj, long long ldp, const float* alpha, float* state, const int* q_start,
                             const int* slots, int entries, int longest, int H, int d, int dv, float scale, cudaStream_t stream) {
    if (entries <= 0) return 0;
    if (d < 1 || d > 32 * kRows || dv < 1 || H < 1 || H > 65535) return (int)cudaErrorInvalidValue;
    const int ds = scan_row_groups(d);
    const int warps = scan_warps(dv, ds, (long long)entries * H, longest <= kFewTokens ? 4 : 8);
    const int vt = warps * (32 / ds) * 2;
    int tt, stage;
    size_t bytes;
    scan_tile(3, ds, vt, tt, stage, bytes);
    const dim3 grid(entries, H, (dv + vt - 1) / vt);
    const int threads = (warps + 4) * 32;  // four feeding warps: they only copy
    const int vec = scan_aligned16(proj) && scan_aligned16(alpha) && ldp % 4 == 0 && d % 4 == 0 && dv % 4 == 0 && vt % 4 == 0;
    XB_SCAN_DISPATCH_FEW(linear_scan_kernel, ds, longest <= kFewTokens, o, proj, ldp, alpha, state, q_start, slots, H, d, dv, scale, tt, stage, warps, vec)
    return xb_launch_status();
}

XB_EXPORT int xb_matrix_memory(float* o, float* div, const float* proj, long long ldp, int gate_off, const float* bi,
                               const float* bf, float cap, float* state_s, float* state_n, float* state_m, const int* q_start,
                               const int* start_pos, const int* slots, int entries, int longest, int H, int d, int dv, float scale,
                               float div_eps, cudaStream_t stream) {
    if (entries <= 0) return 0;
    if (d < 1 || d > 32 * kRows || dv < 1 || H < 1 || H > 65535 || !(cap > 0.f)) return (int)cudaErrorInvalidValue;
    const int ds = scan_row_groups(d);
    const int warps = scan_warps(dv, ds, (long long)entries * H);
    const int vt = warps * (32 / ds) * 2;
    int tt, stage;
    size_t bytes;
    scan_tile(2, ds, vt, tt, stage, bytes, 3);
    const dim3 grid(entries, H, (dv + vt - 1) / vt);
    const int threads = (warps + 1 + (warps == 8 ? 3 : 4)) * 32;   // the warp of n, then three or four feeding warps
    const int vec = scan_aligned16(proj) && ldp % 4 == 0 && d % 4 == 0 && dv % 4 == 0 && vt % 4 == 0;
    XB_SCAN_DISPATCH_FEW(matrix_memory_kernel, ds, longest <= kFewTokens, o, div, proj, ldp, gate_off, bi, bf, cap, state_s, state_n, state_m, q_start,
                     start_pos, slots, H, d, dv, scale, div_eps, tt, stage, warps, vec)
    return xb_launch_status();
}

XB_EXPORT int xb_low_rank_decay(float* alpha, const float* low, long long ldl, const float* w, const float* bias, int tokens,
                                int C, int R, float tau, cudaStream_t stream) {
    if (tokens <= 0 || C <= 0) return 0;
    const int cols = (C + kDecayChannels - 1) / kDecayChannels;
    if (R < 1 || !(tau > 0.f) || cols > 65535) return (int)cudaErrorInvalidValue;
    const dim3 grid((tokens + kDecayTokens - 1) / kDecayTokens, cols);
    xb_launch_few(low_rank_decay_kernel, dim3(grid), dim3(kDecayChannels), 0, stream, alpha, low, ldl, w, bias, tokens, C, R, 1.f / tau);
    return xb_launch_status();
}

// One block per (token, group of `part` consecutive channels of the W):
//   mode 0:  v = y * silu(gate);  out = v * rsqrt(mean(v^2) + eps) * w[c mod w_len]          (gate before the norm)
//   mode 1:  out = y * rsqrt(mean(y^2) + eps) * w[c mod w_len] * sigmoid(gate)               (gate behind it)
//   mode 2:  the same with silu(gate)
// gate is column g_off + c of a wider float32 row.  div (nullable): every y of a part is first divided by div[t, part].
// out's rows lie ldo apart and receive out_scale times the result.
template <typename TO>
__global__ void gated_head_norm_kernel(TO* __restrict__ out, const float* y, const float* gate,
                                       long long ldg, int g_off, const float* __restrict__ w, int w_len, int W, int part,
                                       float eps, int mode, const float* div, long long ldo, float out_scale) {
    pdl_overlap_few();
    __shared__ float scratch[33];
    const int t = blockIdx.x, c0 = blockIdx.y * part;
    const float* yr = y + (size_t)t * W + c0;
    const float* gr = gate + (size_t)t * ldg + g_off + c0;
    float dv = div ? div[(size_t)t * gridDim.y + blockIdx.y] : 1.f;
    if (dv == 0.f) dv = 1.f;        // (a padding token's, which nothing has written)
    float ss = 0.f;
    for (int i = threadIdx.x; i < part; i += blockDim.x) {
        float v = yr[i] / dv;
        if (mode == 0) {
            const float z = gr[i];
            v *= z / (1.f + expf(-z));
        }
        ss = fmaf(v, v, ss);
    }
    const float inv = 1.f / sqrtf(block_sum(ss, scratch) / (float)part + eps);
    TO* o = out + (size_t)t * ldo + c0;
    for (int i = threadIdx.x; i < part; i += blockDim.x) {
        const float z = gr[i];
        float v = yr[i] / dv;
        if (mode == 0)
            v = v * (z / (1.f + expf(-z))) * inv * w[(c0 + i) % w_len];
        else
            v = v * inv * w[(c0 + i) % w_len] * (mode == 2 ? z * sigmoid_exact(z) : sigmoid_exact(z));
        o[i] = from_f32<TO>(out_scale * v);
    }
}

// The same for parts of at most 32 * NV channels: a warp per (token, part) keeps its channels in registers, one pass
// over memory, sums by shuffles; a block's warps take neighbouring parts of a token.
template <typename TO, int NV>
__global__ void __launch_bounds__(256) gated_head_norm_warp_kernel(TO* __restrict__ out, const float* y,
                                                                   const float* gate, long long ldg, int g_off,
                                                                   const float* __restrict__ w, int w_len, int W, int part,
                                                                   float eps, int mode, const float* div,
                                                                   long long ldo, float out_scale, long long units) {
    pdl_overlap_few();
    const int lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (unit >= units) return;
    const int parts = W / part;
    const long long t = unit / parts;
    const int c0 = (int)(unit % parts) * part;
    const float* yr = y + (size_t)t * W + c0;
    const float* gr = gate + (size_t)t * ldg + g_off + c0;
    float v[NV], z[NV];
    float dv = div ? div[unit] : 1.f;
    if (dv == 0.f) dv = 1.f;        // (a padding token's, which nothing has written)
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = lane + 32 * k;
        v[k] = i < part ? yr[i] : 0.f;
        z[k] = i < part ? gr[i] : 0.f;
        if (div) v[k] /= dv;
        if (mode == 0) v[k] *= z[k] / (1.f + expf(-z[k]));
        ss = fmaf(v[k], v[k], ss);
    }
    const float inv = 1.f / sqrtf(warp_total(ss) / (float)part + eps);
    TO* o = out + (size_t)t * ldo + c0;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = lane + 32 * k;
        if (i >= part) continue;
        float r = v[k] * inv * w[(c0 + i) % w_len];
        if (mode != 0) r *= mode == 2 ? z[k] * sigmoid_exact(z[k]) : sigmoid_exact(z[k]);
        o[i] = from_f32<TO>(out_scale * r);
    }
}

// The same for parts of a multiple of four channels that leave in bfloat16, with 16-byte loads that are all in flight before the
// first is used: a warp per (token, part) up to 512 channels, a block of 256 threads above, NV times four channels a thread.
// Bound by latency, not bytes: 1,802 rows of 2,048 channels (37 MB) took 24.6 us in parts of 1,024, where a part's gates were
// read twice, and 16.5 us in parts of 128, a value a load; this 12.5 and 12.3 (4,096 rows of 4,096 in parts of 512: 111 and 43).
template <int NV, bool BLOCK>
__global__ void __launch_bounds__(256) gated_head_norm4_kernel(__nv_bfloat16* __restrict__ out, const float* y, const float* gate,
                                                               long long ldg, int g_off, const float* __restrict__ w, int w_len,
                                                               int W, int part, float eps, int mode, const float* div,
                                                               long long ldo, float out_scale, unsigned units) {
    pdl_overlap_few();
    __shared__ float scratch[33];
    constexpr int L = BLOCK ? 256 : 32;
    const unsigned unit = BLOCK ? blockIdx.x : blockIdx.x * 8 + (threadIdx.x >> 5), parts = (unsigned)(W / part);
    if (unit >= units) return;
    const int lane = BLOCK ? threadIdx.x : threadIdx.x & 31;
    const unsigned t = unit / parts;
    const int c0 = (int)(unit % parts) * part;
    const float* yr = y + (size_t)t * W + c0;
    const float* gr = gate + (size_t)t * ldg + g_off + c0;
    float4 v[NV], z[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (lane + L * k) * 4;
        v[k] = i < part ? *reinterpret_cast<const float4*>(yr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        z[k] = i < part ? *reinterpret_cast<const float4*>(gr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float dv = div ? div[unit] : 1.f;
    if (dv == 0.f) dv = 1.f;        // (a padding token's, which nothing has written)
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        float* vk = reinterpret_cast<float*>(&v[k]);
        const float* zk = reinterpret_cast<const float*>(&z[k]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (div) vk[e] /= dv;
            if (mode == 0) vk[e] *= zk[e] / (1.f + expf(-zk[e]));
            ss = fmaf(vk[e], vk[e], ss);
        }
    }
    const float inv = 1.f / sqrtf((BLOCK ? block_sum(ss, scratch) : warp_total(ss)) / (float)part + eps);
    __nv_bfloat16* o = out + (size_t)t * ldo + c0;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (lane + L * k) * 4;
        if (i >= part) continue;
        const float4 wv = *reinterpret_cast<const float4*>(w + (c0 + i) % w_len);
        const float* vk = reinterpret_cast<const float*>(&v[k]);
        const float* zk = reinterpret_cast<const float*>(&z[k]);
        const float* wk = reinterpret_cast<const float*>(&wv);
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            r[e] = vk[e] * inv * wk[e];
            if (mode != 0) r[e] *= mode == 2 ? zk[e] * sigmoid_exact(zk[e]) : sigmoid_exact(zk[e]);
            r[e] *= out_scale;
        }
        const __nv_bfloat162 a = __floats2bfloat162_rn(r[0], r[1]), b = __floats2bfloat162_rn(r[2], r[3]);
        uint2 q;
        q.x = *reinterpret_cast<const unsigned*>(&a);
        q.y = *reinterpret_cast<const unsigned*>(&b);
        *reinterpret_cast<uint2*>(o + i) = q;
    }
}

// Whether the kernel above takes the call: what its 16-byte loads and 8-byte stores need, and up to 4,096 channels a part.
static bool gated_head_norm4(__nv_bfloat16* out, const float* y, const float* gate, long long ldg, int g_off, const float* w,
                             int w_len, int tokens, int W, int part, float eps, int mode, const float* div, long long ldo,
                             float out_scale, cudaStream_t stream) {
    const long long units = (long long)tokens * (W / part);
    if (part % 4 || part > 4096 || ldg % 4 || g_off % 4 || w_len % 4 || ldo % 4 || units > INT_MAX) return false;
    if ((((uintptr_t)y | (uintptr_t)gate | (uintptr_t)w) & 15) || ((uintptr_t)out & 7)) return false;
#define XB_HEAD_NORM4(NVV, BLOCKV)                                                                                        \
    xb_launch_few(gated_head_norm4_kernel<NVV, BLOCKV>, dim3((unsigned)(BLOCKV ? units : (units + 7) / 8)), dim3(256), 0, stream, out, y, gate, ldg, \
                  g_off, w, w_len, W, part, eps, mode, div, ldo, out_scale, (unsigned)units)
    if (part <= 128) XB_HEAD_NORM4(1, false);
    else if (part <= 256) XB_HEAD_NORM4(2, false);
    else if (part <= 512) XB_HEAD_NORM4(4, false);
    else if (part <= 1024) XB_HEAD_NORM4(1, true);
    else if (part <= 2048) XB_HEAD_NORM4(2, true);
    else XB_HEAD_NORM4(4, true);
#undef XB_HEAD_NORM4
    return true;
}
static bool gated_head_norm4(float*, const float*, const float*, long long, int, const float*, int, int, int, int, float, int,
                             const float*, long long, float, cudaStream_t) {
    return false;       // float32 rows keep the order of their sums
}

template <typename TO>
static void gated_head_norm_launch(TO* out, const float* y, const float* gate, long long ldg, int g_off, const float* w,
                                   int w_len, int tokens, int W, int part, float eps, int mode, const float* div,
                                   long long ldo, float out_scale, cudaStream_t stream) {
    if (gated_head_norm4(out, y, gate, ldg, g_off, w, w_len, tokens, W, part, eps, mode, div, ldo, out_scale, stream)) return;
    const long long units = (long long)tokens * (W / part);
    const int warps = 8;
    const unsigned blocks = (unsigned)((units + warps - 1) / warps);
#define XB_HEAD_NORM_NV(NVV)                                                                                              \
    xb_launch_few(gated_head_norm_warp_kernel<TO, NVV>, dim3(blocks), dim3(warps * 32), 0, stream, out, y, gate, ldg, g_off, w, w_len, W, part, \
                                                                            eps, mode, div, ldo, out_scale, units)
    if (part <= 32) XB_HEAD_NORM_NV(1);
    else if (part <= 64) XB_HEAD_NORM_NV(2);
    else if (part <= 128) XB_HEAD_NORM_NV(4);
    else if (part <= 256) XB_HEAD_NORM_NV(8);
    else if (part <= 512) XB_HEAD_NORM_NV(16);
    else {
        const dim3 grid(tokens, W / part);
        const int threads = part >= 1024 ? 256 : 128;
        xb_launch_few(gated_head_norm_kernel<TO>, dim3(grid), dim3(threads), 0, stream, out, y, gate, ldg, g_off, w, w_len, W, part, eps, mode, div, ldo,
                                                             out_scale);
    }
#undef XB_HEAD_NORM_NV
}

XB_EXPORT int xb_gated_head_norm(int out_dtype, void* out, const float* y, const float* gate, long long ldg, int g_off,
                                 const float* w, int w_len, int tokens, int W, int part, float eps, int mode,
                                 const float* div, long long ldo, float out_scale, cudaStream_t stream) {
    if (tokens <= 0 || W <= 0) return 0;
    if (part <= 0 || W % part || W / part > 65535) return (int)cudaErrorInvalidValue;
    if (out_dtype == XB_F32)
        gated_head_norm_launch<float>((float*)out, y, gate, ldg, g_off, w, w_len, tokens, W, part, eps, mode, div, ldo,
                                      out_scale, stream);
    else
        gated_head_norm_launch<__nv_bfloat16>((__nv_bfloat16*)out, y, gate, ldg, g_off, w, w_len, tokens, W, part, eps, mode,
                                              div, ldo, out_scale, stream);
    return xb_launch_status();
}
