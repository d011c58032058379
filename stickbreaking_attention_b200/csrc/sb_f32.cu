// Kernels of float32 precision: forward, backward-dq and backward-dk/dv.
//
// They serve float32 inputs (whose products must not be rounded to bf16/tf32), head dims other than 32, 64 and
// 128, and tensors whose strides the TMA path cannot take.  Structure mirrors the tensor-core kernels:
//   * forward walks the key tiles of one query block right to left and carries, per row, the running
//     product W = prod(1 - beta) of everything to the right (the reference carries its log,
//     stickbreaking_attention/sb_varlen/sb_varlen_fwd.py:53-66,155-193);
//   * the value of W at every 32-key boundary is saved ("carry_w") so that the backward can enter any quarter
//     directly instead of subtracting from the row total as the reference does (sb_varlen_bwd.py:396-445);
//   * backward-dq walks left to right carrying the prefix sum of g = A * dA (sb_varlen_bwd.py:438-449) and saves
//     it at every boundary ("carry_c");
//   * backward-dk/dv keeps one 64-key tile stationary and walks the query blocks below it, entering each
//     32-key quarter with the two saved carries; dk and dv are accumulated in registers and stored once, so there is no
//     atomic or lock on the data (the reference uses a spin lock per key tile, sb_varlen_bwd.py:11-53).
//
// Arithmetic.  A value is written as a sum of bf16 terms: x = x0 + x1 + x2 with x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1).
// One term holds a bf16 value, two an f16 value, three the 24 bits of a float32, all exactly.  Every product runs on the tensor
// cores as the sum of the term products x_i y_j with i + j <= 2, accumulated in float32: what is left out, x1 y2 and smaller, is
// below 2^-25 |x y|, a unit of which float32 multiply-adds lose as much in every addition.  Weights and score gradients are
// float32 values and enter the second products in three terms.  exp and division are the accurate ones (no fast math here; on tcgen05 the division
// is an approximate reciprocal and a step of Newton's method, as accurate).
// Three kinds of values do not divide into terms: infinities, magnitudes that round to one in bf16, and magnitudes below 2^-100, whose
// later terms lie below the smallest bf16.  They show in a block's results, which then are NaN (terms of the first two kinds are), or
// tiny: such a block starts over and forms its sums with ordinary multiply-adds on the values as they are ("direct" below;
// several times slower; a block that does not need it looks at its results and no more).
//
// This file: head dims above 64 and short sequences, on warp-level mma.  (The others: sb_f32_tc.cu; the rule is on_tcgen05 below.)
// What bounds them: the latency of the chain load -> scores -> scan -> second product of a tile, with the issue slots of the per-score
// arithmetic behind it.  (warp-level mma takes 1024 multiply-adds per clock and SM, measured: a 64 x 64 x 64 product costs 256
// clocks for bf16 inputs, 768 where one side is float32 and 1536 where both are.  tcgen05 takes a quarter; at head dims above 64 its planes of three
// terms do not fit shared memory in the backward.)  So a block has eight warps where registers allow it, and the keys of
// a tile are stored in an order that makes the keys of a thread neighbours: the scan along a row is a serial one in registers
// and one over four lanes.
#include <type_traits>

#include "sb_f32.cuh"

namespace sb {

namespace {

template <typename T, int DP>
__global__ void __launch_bounds__(256, DP > 64 ? 1 : 2) f32_fwd_kernel(const __grid_constant__ KArgs a) {
    extern __shared__ __align__(16) __nv_bfloat16 tiles[];
    __shared__ float xs[2][kBM];
    __shared__ OwnTables own;
    pdl_wait();
    if (a.own_tables) {
        if (threadIdx.x < 32) build_own_tables(a, &own, threadIdx.x);
        __syncthreads();
    }
    const int covered_end = a.own_tables ? own.covered_end : a.hdr->covered_end;
    if (a.zero_tail && covered_end < a.tokens) zero_tail_rows<T>(a, covered_end, linear_thread(), all_threads());
    const BlockIdx bi = block_idx();
    if (bi.item >= (a.own_tables ? own.n_items : a.hdr->n_items)) return;
    const auto item = [&]() { return a.own_tables ? item_ctx(own.items, own.seqs, bi.item) : item_ctx(a, bi.item); };
    const ItemCtx c = item();
    if (c.qt * kTileQ + bi.part * kBM >= c.len) return;
    // (16-bit types look their item up again instead of keeping it: the loop has no register to spare for it.  At sizes that take tcgen05 by now,
    // 35.8 -> 35.3 us on 4 x 8 heads x 500 tokens, head dim 50; float32 loses by it, 132 -> 137 us on 8 heads, 4096 tokens, head dim 64)
    if (fwd_block<T, DP, kTerms>(a, c, bi, tiles, xs)) fwd_block<T, DP, kValuesInPlace>(a, sizeof(T) == 2 ? item() : c, bi, tiles, xs);
}

template <typename T, int DP>
__global__ void __launch_bounds__(256, DP > 64 ? 1 : 2) f32_bwd_dq_kernel(const __grid_constant__ KArgs a) {
    extern __shared__ __align__(16) __nv_bfloat16 tiles[];
    __shared__ float xs[2][kBM];
    pdl_wait();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) zero_tail_grads<T>(a, a.hdr->covered_end, linear_thread(), all_threads());
    const BlockIdx bi = block_idx();
    if (bi.item >= a.hdr->n_items) return;
    const ItemCtx c = item_ctx(a, bi.item);
    if (c.qt * kTileQ + bi.part * kBM >= c.len) return;
    if (dq_block<T, DP, kTerms>(a, c, bi, tiles, xs)) dq_block<T, DP, kValuesInPlace>(a, c, bi, tiles, xs);
}

// Scores transposed (rows = keys).  kQ queries per step.  First half of a step: two 32-key quarters (each entered with its own carries) x
// groups of 8 queries; P^T and dS^T go to shared memory as three terms each.  Second half: four groups of 16 keys x {dv, dk} (x the
// two halves of the columns with sixteen warps, so that a thread accumulates 16 or 32 values only).  (With P^T and dS^T kept in
// registers four warps had to hold dk and dv of 32 keys each, 255 registers and 8 warps per SM: 311 against 255 us on 8 heads, 4096 float32 tokens, head dim
// 64, which take tcgen05 by now.)
// Sixteen warps, one block per SM, take steps of 64 queries, or of 32 where the tiles would not fit otherwise (float32 at D > 64; eight
// of the warps then sit out the first half; forward + backward of 8 heads, 4096 tokens, head dim 128: 1638 us with four warps
// that kept P^T and dS^T in registers, 1163 us so).  kBuf = 2, where shared memory has the room: the next step's Q and dO travel during
// the second half and go to the other buffer at its end, which takes a barrier and the whole load out of the step (265 -> 255 us on the same).
// Eight warps, two blocks per SM, take steps of 32: one block's loads and scans run under the other's products.  From six blocks for each SM on, where a short
// last wave does not matter (64 sequences of 64 float32 tokens, 8 heads: 42 -> 36 us).  Over the lengths that these kernels still take (head dims up to 64,
// all types, 40 to 700 tokens each) the whole backward takes 1.01 to 1.24 times as long with sixteen warps at 6 to 24 blocks per SM, 1.01 to 1.2 at 3 to 5, and 0.78
// to 0.94 at one and less; in between it goes by the last wave, 0.81 to 1.1: a line at three blocks would serve these lengths better.
template <typename T, int DP, int kWarps, int kQ, int kBuf>
__global__ void __launch_bounds__(32 * kWarps, 16 / kWarps) f32_bwd_dkdv_kernel(const __grid_constant__ KArgs a) {
    constexpr int kT = 32 * kWarps, kN = Terms<T>::n;
    constexpr int kDC = kWarps == 16 && DP >= 32 ? DP / 2 : DP;  // columns of dk or dv per warp
    constexpr int kNC = kDC < 32 ? kDC / 8 : 4;                  // column blocks at a time
    constexpr int kPP = kQ + 8, kPPlane = 64 * kPP;  // P^T, dS^T: [64 keys][kQ queries], three planes each
    constexpr int kQTile = kN * kQ * kPitch<DP>;     // Q, dO: kQ rows
    constexpr bool kEarly = kBuf == 2 || (kWarps == 8 && sizeof(T) == 2);  // loads a step ahead; float32 lacks the registers otherwise
    extern __shared__ __align__(16) __nv_bfloat16 tiles[];
    __nv_bfloat16* sK = tiles;
    __nv_bfloat16* sV = sK + kTileElems<T, DP>;
    __nv_bfloat16* const tiles_q = sV + kTileElems<T, DP>;
    __nv_bfloat16 *sQ = tiles_q, *sG = sQ + kQTile;
    __nv_bfloat16* sP = sQ + 2 * kBuf * kQTile;
    __nv_bfloat16* sS = sP + kWTerms * kPPlane;
    pdl_wait();
    const BlockIdx bi = block_idx();
    const int n_items = a.hdr->n_items;
    if (bi.item >= n_items) return;
    // the table is heaviest-first for query tiles; key tiles are heaviest at the other end
    const ItemCtx c = item_ctx(a, n_items - 1 - bi.item);
    const int h = bi.h, D = a.head_dim;
    const int key0 = c.qt * kTileQ + bi.part * kBN;
    if (key0 >= c.len) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int kq = warp & 1, q0 = 8 * (warp >> 1);                                     // first half of a step
    const int kg = warp & 3, col0 = (warp >> 3) * kDC;                                 // second half
    const bool is_dk = (warp >> 2) & 1, second = col0 < DP;                            // (head dim 16: the columns are not split)
    const int keys_valid = min(kBN, c.len - key0);
    load_tile<kT, T, DP, kKeyRows>(sK, a.k, D, c.b, h, c.start + key0, keys_valid);
    load_tile<kT, T, DP, kKeyRows>(sV, a.v, D, c.b, h, c.start + key0, keys_valid);
    const int quarter = key0 / 32 + kq;            // of the sequence
    const float* cw = a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ;
    const float* cc = a.carry_c + ((int64_t)h * a.slot_cap) * kTileQ;
    float acc[kDC / 8][4];

    const int uq = unit<T>(a.q, D), ug = unit<T>(a.d_o, D);
    Rows<kT, T, DP, kQ> rq, rg;
    auto fetch = [&](int row0) {
        const int n = min(kQ, c.len - row0);
        rq.fetch(a.q, uq, D, c.b, h, c.start + row0, n);
        rg.fetch(a.d_o, ug, D, c.b, h, c.start + row0, n);
    };
    const auto sweep = [&](auto direct) {
        constexpr bool kDirect = decltype(direct)::value;
        float* const fP = (float*)sP;  // direct: P^T and dS^T as they are, one after the other
        float* const fS = fP + kPPlane;
        static_assert(2 * sizeof(float) * kPPlane <= 2 * kWTerms * sizeof(__nv_bfloat16) * kPPlane, "P^T and dS^T in the place of their terms");
#pragma unroll
        for (int n = 0; n < kDC / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
        if (kEarly && !kDirect) fetch(key0);
        if (kBuf == 2 && !kDirect) {
            rq.template put<kPlain>(sQ, uq);
            rg.template put<kPlain>(sG, ug);
        }
        for (int row0 = key0; row0 < c.len; row0 += kQ) {
            const int rows_valid = min(kQ, c.len - row0);
            if (kDirect) {
                __syncthreads();
            } else if (kBuf == 1) {
                if (!kEarly) fetch(row0);
                __syncthreads();
                rq.template put<kPlain>(sQ, uq);
                rg.template put<kPlain>(sG, ug);
            }
            const int64_t slot = carry_slot32(c.slot_base, row0 / kTileQ, quarter) * kTileQ + row0 % kTileQ;
            float W[2] = {0.f, 0.f}, cr[2] = {0.f, 0.f}, drem[2] = {0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int q = q0 + 2 * t + e;
                if (q < rows_valid) {
                    W[e] = cw[slot + q];
                    cr[e] = cc[slot + q];
                    drem[e] = to_f32<T>(((const T*)a.d_rem.ptr)[(int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + (int64_t)(c.start + row0 + q) * a.d_rem.st]);
                }
            }
            __syncthreads();
            const bool edge = row0 < key0 + kBN || keys_valid < kBN || rows_valid < kQ;
            if (q0 < kQ) {
                float s[2][1][4], dp[2][1][4];
                if (kDirect) {
                    const int key = 32 * kq + 4 * g, q = q0 + 2 * t;
                    direct_scores_t<T>(s, row_of<T>(a.k, c, h, key0 + key), a.k.st, keys_valid - key, row_of<T>(a.q, c, h, row0 + q), a.q.st, rows_valid - q, D);
                    direct_scores_t<T>(dp, row_of<T>(a.v, c, h, key0 + key), a.v.st, keys_valid - key, row_of<T>(a.d_o, c, h, row0 + q), a.d_o.st, rows_valid - q, D);
                } else {
                    product_nt<kN, DP, 2, 1, kQ>(s, sK + 32 * kq * kPitch<DP>, sQ + q0 * kPitch<DP>, D, lane);
                    product_nt<kN, DP, 2, 1, kQ>(dp, sV + 32 * kq * kPitch<DP>, sG + q0 * kPitch<DP>, D, lane);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float* const ps[4] = {&s[0][0][e], &s[0][0][2 + e], &s[1][0][e], &s[1][0][2 + e]};
                    float* const pd[4] = {&dp[0][0][e], &dp[0][0][2 + e], &dp[1][0][e], &dp[1][0][2 + e]};
                    const int q = q0 + 2 * t + e;
                    // a query behind the end of the sequence sees no key: its zeros against an infinite or NaN key would make NaNs
                    const int lim = q < rows_valid ? min(keys_valid, row0 + q + a.attend_current - key0) : 0;
                    column(ps, pd, a.inv_temp, edge, lim - 32 * kq - 4 * g, W[e], cr[e], drem[e], g);
                }
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const int at = (32 * kq + 16 * m + 8 * hh + g) * kPP + q0 + 2 * t;
                        if (kDirect) {
                            *(float2*)(fP + at) = make_float2(s[m][0][2 * hh], s[m][0][2 * hh + 1]);
                            *(float2*)(fS + at) = make_float2(dp[m][0][2 * hh], dp[m][0][2 * hh + 1]);
                            continue;
                        }
                        uint32_t tp[kWTerms], ts[kWTerms];
                        split_pair<kWTerms>(s[m][0][2 * hh], s[m][0][2 * hh + 1], tp);
                        split_pair<kWTerms>(dp[m][0][2 * hh], dp[m][0][2 * hh + 1], ts);
#pragma unroll
                        for (int i = 0; i < kWTerms; ++i) {
                            *(uint32_t*)(sP + i * kPPlane + at) = tp[i];
                            *(uint32_t*)(sS + i * kPPlane + at) = ts[i];
                        }
                    }
            }
            __syncthreads();
            if (kEarly && !kDirect && row0 + kQ < c.len) fetch(row0 + kQ);
            if (kDirect && second) {
                const MatView& mx = is_dk ? a.q : a.d_o;
                const T* x = row_of<T>(mx, c, h, row0) + col0 + 2 * t;
                const float* pa = (is_dk ? fS : fP) + (16 * kg + g) * kPP;
#pragma unroll 1
                for (int q = 0; q < rows_valid; ++q) {
                    const float p0 = pa[q], p1 = pa[8 * kPP + q];
#pragma unroll
                    for (int n = 0; n < kDC / 8; ++n)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float v = col0 + 8 * n + 2 * t + e < D ? to_f32<T>(x[(int64_t)q * mx.st + 8 * n + e]) : 0.f;
                            acc[n][e] = fmaf(p0, v, acc[n][e]);
                            acc[n][2 + e] = fmaf(p1, v, acc[n][2 + e]);
                        }
                }
            }
            if (!kDirect && second) {
                const __nv_bfloat16* pa = (is_dk ? sS : sP) + (16 * kg + (lane & 15)) * kPP + (lane >> 4) * 8;
                const __nv_bfloat16* px = (is_dk ? sQ : sG) + ((lane & 7) + ((lane >> 3) & 1) * 8) * kPitch<DP> + (lane >> 4) * 8 + col0;
#pragma unroll
                for (int n0 = 0; n0 < kDC / 8; n0 += kNC) {
                    float big[kNC][4] = {}, small[kNC][4] = {};
#pragma unroll
                    for (int k = 0; k < kQ / 16; ++k) {
                        uint32_t fa[kWTerms][4];
#pragma unroll
                        for (int i = 0; i < kWTerms; ++i) ldsm4(fa[i], pa + i * kPPlane + 16 * k);
#pragma unroll
                        for (int j = 0; j < kN; ++j) {
                            uint32_t fb[kNC / 2][4];
#pragma unroll
                            for (int n2 = 0; n2 < kNC / 2; ++n2)
                                ldsm4_t(fb[n2], px + j * kQ * kPitch<DP> + k * 16 * kPitch<DP> + n0 * 8 + n2 * 16);
#pragma unroll
                            for (int i = 0; i < kWTerms; ++i) {
                                if (i + j > 2) continue;
#pragma unroll
                                for (int n = 0; n < kNC; ++n) mma(i + j == 0 ? big[n] : small[n], fa[i], fb[n >> 1][2 * (n & 1)], fb[n >> 1][2 * (n & 1) + 1]);
                            }
                        }
                    }
#pragma unroll
                    for (int n = 0; n < kNC; ++n)
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[n0 + n][i] += big[n][i] + small[n][i];
                }
            }
            if (kBuf == 2 && !kDirect && row0 + kQ < c.len) {
                sQ = tiles_q + (sQ == tiles_q ? 2 * kQTile : 0);
                sG = sQ + kQTile;
                rq.template put<kPlain>(sQ, uq);
                rg.template put<kPlain>(sG, ug);
            }
        }
        return __syncthreads_or(asks_for_direct(acc, 0) || asks_for_direct(acc, 2));
    };
    if (sweep(std::false_type{})) sweep(std::true_type{});
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    if (!second) return;
    if (a.fused && !is_dk) {  // dv += rem * do
        const T* d_o = (const T*)a.d_o.ptr + (int64_t)c.b * a.d_o.sb + (int64_t)h * a.d_o.sh + (int64_t)(c.start + key0) * a.d_o.st;
        const T* rem = (const T*)a.rem.ptr + (int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + (int64_t)(c.start + key0) * a.rem.st;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int row = 32 * (kg >> 1) + 4 * g + 2 * (kg & 1) + hh;
            if (row < keys_valid) add_row<T, kDC>(acc, 2 * hh, to_f32<T>(rem[(int64_t)row * a.rem.st]), d_o + (int64_t)row * a.d_o.st, D, col0, t);
        }
    }
    const MatView m = is_dk ? a.dk : a.dv;
    const bool pairs = units_ok<T>(m, D, 2);
    T* base = (T*)m.ptr + (int64_t)c.b * m.sb + (int64_t)h * m.sh + (int64_t)(c.start + key0) * m.st;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int row = 32 * (kg >> 1) + 4 * g + 2 * (kg & 1) + hh;
        if (row < keys_valid) store_row<T, kDC>(acc, 2 * hh, is_dk ? a.inv_temp : 1.f, m, pairs, D, col0, base, row, t);
    }
}

template <typename T, int DP>
int launch_one(void (*kernel)(KArgs), int threads, int tiles, int more, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    const int smem = tiles * kTileElems<T, DP> * 2 + more;
    const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
    if (e != 0) return e;
    return launch_kernel(kernel, block_grid(L.max_items, a.heads), dim3(threads), smem, st, a);
}
template <typename T, int DP, int kQ, int kBuf>
constexpr int dkdv_smem() {
    return 2 * (2 * kTileElems<T, DP> + kBuf * 2 * Terms<T>::n * kQ * kPitch<DP> + 2 * kWTerms * 64 * (kQ + 8));
}
template <typename T, int DP, int kWarps, int kQ, int kBuf>
int launch_dkdv(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    return launch_one<T, DP>(f32_bwd_dkdv_kernel<T, DP, kWarps, kQ, kBuf>, 32 * kWarps, 2, dkdv_smem<T, DP, kQ, kBuf>() - 4 * kTileElems<T, DP>, L, a, st);
}
template <typename T, int DP>
int launch_d(bool backward, const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    if (!backward) return launch_one<T, DP>(f32_fwd_kernel<T, DP>, 256, 3, 0, L, a, st);
    if (phases != SBATTN_BWD_DKDV) {
        const int e = launch_one<T, DP>(f32_bwd_dq_kernel<T, DP>, 256, 4, 0, L, a, st);
        if (e != 0) return e;
    }
    if (phases == SBATTN_BWD_DQ) return 0;
    if constexpr (DP <= 64) {  // six blocks for each SM: see the kernel
        if ((int64_t)L.max_items * a.heads * 2 >= 6 * sm_count()) return launch_dkdv<T, DP, 8, 32, 1>(L, a, st);
    }
    constexpr int kQ = DP > 64 && Terms<T>::n == 3 ? 32 : 64;
    return launch_dkdv<T, DP, 16, kQ, dkdv_smem<T, DP, kQ, 2>() <= kMaxSmem ? 2 : 1>(L, a, st);
}
template <typename T>
int launch_t(bool backward, const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    if (a.head_dim > 64) return launch_d<T, 128>(backward, L, a, phases, st);
    if (a.head_dim > 32) return launch_d<T, 64>(backward, L, a, phases, st);
    return a.head_dim > 16 ? launch_d<T, 32>(backward, L, a, phases, st) : launch_d<T, 16>(backward, L, a, phases, st);
}
int launch_any(const SbParams& p, bool backward, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    if (L.max_items <= 0) return 0;
    switch (p.dtype) {
        case SBATTN_BF16: return launch_t<__nv_bfloat16>(backward, L, a, p.bwd_phases, st);
        case SBATTN_F16: return launch_t<__half>(backward, L, a, p.bwd_phases, st);
        default: return launch_t<float>(backward, L, a, p.bwd_phases, st);
    }
}

}  // namespace

// Whether the kernels on tcgen05 (sb_f32_tc.cu) take a pass.  They work on 128-row tiles, a block per SM, with ~6 us around an item's steps, and on
// 64 columns whatever the head dim: long sequences, by the average length of a pack.  Forward + backward in us, warp-level / tcgen05 kernels, 8 heads,
// 8192 tokens in sequences of equal length:
//   head dim 64, float32:  64 each 176 / 236, 128: 229 / 201, 256: 324 / 239, 1024: 901 / 457, 4096: 3267 / 1348
//   head dim 50, bf16:     192: 180 / 195, 1024: 577 / 353, 4096: 2049 / 1047
//   head dim 32, float32:  192: 178 / 213, 256: 216 / 200, 384: 274 / 226, 4096: 2137 / 1275;   18, bf16: 256: 164 / 162, 384: 208 / 183, 4096: 1555 / 1007
//   head dim 16, float32:  384: 215 / 220, 512: 264 / 256, 1024: 457 / 396, 4096: 1644 / 1240;  16, bf16: 512: 209 / 205, 1024: 358 / 312, 4096: 1261 / 958
// The bounds lie above some lengths at which they gain up to 10 % with 8 heads: with 32 they do not.
// Lengths around the average (log-normal, sigma 0.7) only help, since the long ones have the work: at the bounds forward 1.0 ... 1.6 and backward 1.0 ... 1.7 times
// as fast.  Sequences of nearly equal length, though, all have a last tile as full as the average says, and where that is half a tile or less the rows
// that do not exist cost more than the units gain up to a second bound, as soon as three blocks and more follow one another on an SM (up to there the shorter
// chain of a block counts: 1.05 ... 1.5 times as fast).  Warp-level / tcgen05 there, forward and backward apart, 8 heads (32 alike):
//   float32, head dim 64: 140 each forward 90.8 / 83.5, backward 227 / 244;  161: 80.3 / 73.3, 228 / 221
//   bf16, 50:             257: 78.8 / 73.8, 190 / 193;   300: 70.7 / 64.5, 183 / 173;   f16: 257: 103 / 82, 248 / 229
//   float32, 32:          320: 65.7 / 63.8, 171 / 183;   385: 91.9 / 80.0, 240 / 238
//   bf16, 18:             320: 52.9 / 55.4, 128 / 145;   385: 72.6 / 69.0, 175 / 189;   448: 64.0 / 58.3, 163 / 161;  f16, 20: 320: 59.7 / 59.2, 152 / 165
//   float32, 16:          800: 102 / 90, 276 / 284;      bf16, 16: 1.05 and 0.97 times as fast at 800, 1.10 and 1.01 at 897
//   bf16, 9:              800: 86.4 / 91.5, 235 / 253;   897: 99.7 / 101, 277 / 287;    1000: 99.6 / 95.3, 287 / 268
// (A form of theirs in which one block per SM draws item after item, and with 32 columns, gains up to 25 % below these lines, where it still loses, and
// costs 9-20 % above them: a drawn item is bound to its block, a block that the hardware starts is not.)
// A sequence's last bits depend on its pack thereby: the average, the longest length and, between the two bounds, the number of blocks choose the family.
bool on_tcgen05(const SbParams& p, const WsLayout& L, bool backward) {
    const int D = p.head_dim;
    if (D > 64) return false;
    const int64_t seqs = p.batch > 0 ? 1 : (p.num_seqs > 0 ? p.num_seqs : 1), average = p.tokens / seqs;
    const bool f32 = p.dtype == SBATTN_F32, bf16 = p.dtype == SBATTN_BF16;
    const int bound = D > 32 ? (f32 ? 128 : 224) : D > 16 ? 320 : 768;
    if (average < bound) return false;
    const int64_t longest = p.batch == 0 && p.max_seqlen > 0 && p.max_seqlen < p.tokens ? p.max_seqlen : p.tokens;
    if (longest > average + average / 16 || (average - 1) % kTileQ >= kTileQ / 2 || (int64_t)L.max_items * p.heads <= 3 * sm_count()) return true;
    if (backward) return average >= (D > 32 ? (f32 ? 160 : bf16 ? 288 : 224) : D > 16 ? 416 : 961);
    return !bf16 || D > 32 || average >= (D > 16 ? 384 : D % 2 == 0 ? 768 : 961);  // odd head dims: rows are loaded one element at a time
}
int launch_f32_fwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    return on_tcgen05(p, L, false) ? launch_f32tc(p, false, L, a, st) : launch_any(p, false, L, a, st);
}
int launch_f32_bwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    return on_tcgen05(p, L, true) ? launch_f32tc(p, true, L, a, st) : launch_any(p, true, L, a, st);
}

}  // namespace sb
