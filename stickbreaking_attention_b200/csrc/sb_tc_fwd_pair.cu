// Tensor-core forward (sm_100a), two query tiles of a sequence at a time: head dim 128, sequences of one length with enough work for every SM
// (use_pairs in sb_tc_fwd.cu).  The results and carries of sb_tc_fwd.cu to rounding (the reference's _forward_one_row,
// stickbreaking_attention/sb_varlen/sb_varlen_fwd.py:155-193): here the carry enters a chunk's chain of reciprocals at its start, there it is multiplied in at
// the end, and here P V sums the right half of a tile first.
//
// One work item = (head, sequence, pair of neighbouring 128-row query tiles); the lowest tile of an odd number stands alone.  The pair
// walks the key tiles right to left together, so a K or V tile is loaded once for both.  Each tile has its own row warps, scores and
// accumulator, and the two take turns: while the row threads of one turn scores into weights, the tensor cores form O += P V and the next
// S of the other.
//
// Warps of a block (352 threads, three per scheduler, so that a thread may hold 168 registers):
//   0-3 / 4-7  row warps of the upper / lower tile: a thread owns one query row, all 128 keys of a step, as four chunks of 32 from right
//              to left.  The carry W (product of 1 - beta over everything to the right) stays in a register and nothing is exchanged between
//              warps.  The scores of a chunk travel while the chunk before is swept, and its weights are finished while the next one is.
//   8 / 10     TMA producers: warp 8 draws the items and loads Q (three slots, so that the next item's first tile is there in time) and
//              the K tiles (two stages), warp 10 the V tiles (two stages).
//   9          issues tcgen05.mma.  P V of a tile in two halves of 64 keys, each as soon as its weights exist.
// Tensor memory (512 columns): S of the upper / lower tile at 0 / 128 (P overwrites the right half of its S: a thread has read the
// columns that it writes), O at 256 / 384.
//
// What bounds it: power, then the row threads.  A step of one tile takes 3 190 cycles (clock readings around its parts), 1 910 of them row work
// (1 152 of the special-function unit) and 1 280 between P and the next S, in which the other tile has the scheduler to itself: 1 595
// cycles for 128 x 128 scores against 2 100 in sb_tc_fwd.cu.  In back-to-back calls the SM clock falls to about 1.7 GHz with either kernel.
// Forward of 32 heads, 8192 tokens in one sequence, bf16, calls back to back: 557 -> 520 us when written (cuBLAS at its sustained rate would need 397 us
// for the same operations), 535 -> 534 us against sb_tc_fwd.cu with its early reads of items; 8 heads, 65 536 tokens 7 920 -> 7 640 us.  With P V in parts
// of 96 and 32 keys 528 us.
#include "sb_tc_fwd_common.cuh"

namespace sb {

using namespace sm100;
using namespace fwd;

namespace {

constexpr int kThreads = 352;
constexpr int kBM = 128, kBN = 128;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kColS = 0, kColO = 256, kColPOff = 64;  // of tile t: + 128 t
constexpr int kQSlots = 3;
enum PairBar { Q_FULL0, Q_FULL1, Q_FULL2, Q_EMPTY0, Q_EMPTY1, Q_EMPTY2, K_FULL0, K_FULL1, K_EMPTY0, K_EMPTY1, V_FULL0, V_FULL1, V_EMPTY0, V_EMPTY1,
               S_READY0, S_READY1, P_RIGHT0, P_RIGHT1, P_LEFT0, P_LEFT1, O_READY0, O_READY1, O_FREE0, O_FREE1,
               WORK_FULL0, WORK_FULL1, WORK_EMPTY0, WORK_EMPTY1, kNumBars };

__device__ __forceinline__ void store_carry(float* p, float v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"((int)on) : "memory");
}

// a whole step of an unmasked tile; s_base: this thread's lane of S
template <bool kF16>
__device__ __forceinline__ void step_full(uint32_t s_base, float scale, float& W, float* cw, bool save, uint64_t* right_ready) {
    uint32_t u[2][32], packed[16];
    float2 pw[2][2][8], run[2], f[2][2];
    tmem_ld32(s_base + 96, u[0]);
    tmem_wait_ld(u[0]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = 3 - i;  // chunk of 32 keys
        if (i < 3) tmem_ld32(s_base + 32 * (c - 1), u[(i + 1) & 1]);
        fwd_sweep<false>(u[i & 1], scale, 0, 0, pw[i & 1], run);
        if (i > 0) {  // the weights of the chunk before
            fwd_finish<kF16>(pw[(i - 1) & 1], f[(i - 1) & 1], 1.f, packed);
            tmem_st16(s_base + kColPOff + 16 * (c + 1), packed);
        }
        if (i == 2) {
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(right_ready);
        }
        store_carry(cw + c * kTileQ, W, save);  // the carry at the chunk's right edge
        fwd_carries(run, W, f[i & 1]);
        if (i < 3) tmem_wait_ld(u[(i + 1) & 1]);
    }
    fwd_finish<kF16>(pw[1], f[1], 1.f, packed);
    tmem_st16(s_base + kColPOff, packed);
}
// the diagonal tile: chunks to the right of the warp's rows hold no visible key
template <bool kF16>
__device__ __forceinline__ void step_diagonal(uint32_t s_base, float scale, int lim, int row_chunk, float& W, float* cw, bool save,
                                              uint64_t* right_ready) {
#pragma unroll 1
    for (int c = 3; c >= 0; --c) {
        uint32_t packed[16];
        store_carry(cw + c * kTileQ, W, save);
        if (c > row_chunk) {
#pragma unroll
            for (int i = 0; i < 16; ++i) packed[i] = 0u;
        } else {
            uint32_t u[32];
            float2 pw[2][8], run[2], f[2];
            tmem_ld32(s_base + 32 * c, u);
            tmem_wait_ld(u);
            fwd_sweep<true>(u, scale, 32 * c, lim, pw, run);
            fwd_carries(run, W, f);
            fwd_finish<kF16>(pw, f, 1.f, packed);
        }
        tmem_st16(s_base + kColPOff + 16 * c, packed);
        if (c == 2) {
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(right_ready);
        }
    }
}

template <bool kF16, bool kFused>
__global__ void __launch_bounds__(kThreads, 1)
tc_fwd_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const __grid_constant__ KArgs a) {
    constexpr int D = kMaxHeadDim, kTileBytes = kBM * D * 2;
    constexpr int kBoxBytes = 128 * 128;  // one TMA box: 128 rows of 64 elements
    constexpr int kBoxes = D / 64;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                        // kQSlots tiles
    uint8_t* sK = sQ + kQSlots * kTileBytes;   // two tiles
    uint8_t* sV = sK + 2 * kTileBytes;         // two tiles
    uint64_t* bars = (uint64_t*)(sV + 2 * kTileBytes);
    SchedRing<Work>* ring = (SchedRing<Work>*)(bars + kNumBars);
    uint32_t* tmem_slot = (uint32_t*)(ring + 1);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kNumBars; ++i) {
            uint32_t cnt = 1;
            if (i >= P_RIGHT0 && i <= P_LEFT1) cnt = 128;
            if (i == O_FREE0 || i == O_FREE1) cnt = 128;
            if (i == WORK_EMPTY0 || i == WORK_EMPTY1) cnt = 258;  // MMA warp (one lane), V producer, 256 row threads
            mbar_init(&bars[i], cnt);
        }
        *abort_flag = (smem_u32(smem) & 1023u) ? 1u : 0u;  // the swizzled tiles need a 1024-byte aligned base
        fence_barrier_init();
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    if (warp == 8 && lane == 0) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) {
        const int64_t me = (int64_t)blockIdx.x * kThreads + tid, all = (int64_t)gridDim.x * kThreads;
        if (kF16) zero_tail_rows<__half>(a, a.hdr->covered_end, me, all);
        else zero_tail_rows<__nv_bfloat16>(a, a.hdr->covered_end, me, all);
    }
    const int n_items = a.hdr->n_items;
    const int n_work = *abort_flag ? 0 : n_items * a.heads;

    if (warp == 8) {
        // ------------------------------------------------------------------ TMA producer: items, Q and K
        if (lane == 0) {
            uint32_t ph_qe = 7, qs = 0;  // bit i: Q slot i ("empty" barriers start released); slot of the next tile
            uint32_t kv = 0;
            bool ok = true, first = true;
            uint32_t ph_we = 3, ri = 0;
            // Heads that do not fill the groups go first: the longest pair of a last group that is too small for all SMs would end the kernel
            // alone.  One sequence of 16 384 tokens, 16 heads (groups of five), against one tile at a time: 9 % slower with the
            // one head of the remainder last, 8 % faster with it first; 17 heads 10 % slower and 2 % faster.
            const int missing = (a.head_group - a.heads % a.head_group) % a.head_group;
            const auto wait_q_slot = [&]() {
                ok = mbar_wait_idle(&bars[Q_EMPTY0 + qs], (ph_qe >> qs) & 1, abort_flag);
                ph_qe ^= 1u << qs;
                return ok;
            };
            while (ok) {
                const uint32_t sl = ri++ & 1;
                ok = mbar_wait(&bars[WORK_EMPTY0 + sl], (ph_we >> sl) & 1, abort_flag);
                ph_we ^= 1u << sl;
                if (!ok) break;
                // The table lists single tiles; the upper tile of a pair is the one an even number of tiles below the sequence's
                // end, and the draws of the others are passed over.
                int w;
                Work wk{};
                while (true) {
                    w = first ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(a.sched + 0, 1);
                    first = false;
                    if (w >= n_work) { w = -1; break; }
                    wk = fetch_work(a, a.items, a.seqs, n_items, w, missing);
                    if (((((wk.len + kBM - 1) / kBM) - 1 - wk.qt) & 1) == 0) break;
                }
                if (w >= 0) ring->work[sl] = wk;
                ring->slot[sl] = w;
                mbar_arrive(&bars[WORK_FULL0 + sl]);
                if (w < 0) break;
                for (int kt = wk.qt; ok && kt >= 0; --kt, ++kv) {
                    const int t = wk.qt - kt;  // the first two steps bring the tiles of Q: the upper one, then the lower one
                    if (t < 2) {
                        if (!wait_q_slot()) break;
                        mbar_expect_tx(&bars[Q_FULL0 + qs], kTileBytes);
#pragma unroll
                        for (int bx = 0; bx < kBoxes; ++bx)
                            tma_load_4d(sQ + qs * kTileBytes + bx * kBoxBytes, &map_q, &bars[Q_FULL0 + qs], bx * 64, wk.start + kt * kBM, wk.h, wk.b);
                        qs = qs == kQSlots - 1 ? 0 : qs + 1;
                    }
                    const uint32_t st = kv & 1;
                    ok = mbar_wait_idle(&bars[K_EMPTY0 + st], ((kv >> 1) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&bars[K_FULL0 + st], kTileBytes);
#pragma unroll
                    for (int bx = 0; bx < kBoxes; ++bx)
                        tma_load_4d(sK + st * kTileBytes + bx * kBoxBytes, &map_k, &bars[K_FULL0 + st], bx * 64, wk.start + kt * kBN, wk.h, wk.b);
                }
            }
        }
    } else if (warp == 10) {
        // ------------------------------------------------------------------ TMA producer: V
        if (lane == 0) {
            uint32_t kv = 0;
            bool ok = true;
            SchedConsumer sched;
            int w;
            Work wk;
            while (ok && (w = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, wk)) >= 0) {
                for (int kt = wk.qt; kt >= 0; --kt, ++kv) {
                    const uint32_t st = kv & 1;
                    ok = mbar_wait_idle(&bars[V_EMPTY0 + st], ((kv >> 1) & 1) ^ 1, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(&bars[V_FULL0 + st], kTileBytes);
#pragma unroll
                    for (int bx = 0; bx < kBoxes; ++bx)
                        tma_load_4d(sV + st * kTileBytes + bx * kBoxBytes, &map_v, &bars[V_FULL0 + st], bx * 64, wk.start + kt * kBN, wk.h, wk.b);
                }
            }
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------------ MMA issuer
        const bool leader = elect_one();  // the whole warp runs the loops; one lane issues
        constexpr uint32_t idesc_s = make_idesc(kBM, kBN, kF16 ? 0 : 1, 0, 0);
        constexpr uint32_t idesc_o = make_idesc(kBM, D, kF16 ? 0 : 1, 0, 1);
        const SmemDesc desc_q = make_desc(smem_u32(sQ), 0, 1024);          // K-major operands of S
        const SmemDesc desc_k = make_desc(smem_u32(sK), 0, 1024);
        const SmemDesc desc_v = make_desc(smem_u32(sV), kBoxBytes, 1024);  // MN-major operand of P V
        uint32_t ph_qf = 0, ph_of = 3;   // bit i: Q slot i / bit t: O_FREE of tile t
        uint32_t ph_p = 0;               // bit t: parity of P_RIGHT and P_LEFT of tile t
        uint32_t next_slot = 0;          // Q slot of the next tile to come
        uint32_t kbase = 0;              // K / V tiles of all items before the current one
        bool ok = true;
        // S of one tile from Q slot qs and the k-th K tile overall.  The tile's own P has been consumed by contractions issued before.
        const auto issue_s = [&](uint32_t t, uint32_t qs, uint32_t k, bool last_use_of_k, bool last_use_of_q) {
            const uint32_t st = k & 1;
            ok = mbar_wait(&bars[K_FULL0 + st], (k >> 1) & 1, abort_flag);
            if (!ok) return;
            tc_fence_after();
            const SmemDesc dq = {desc_q.lo + qs * (kTileBytes >> 4), desc_q.hi};
            const SmemDesc dk = {desc_k.lo + st * (kTileBytes >> 4), desc_k.hi};
#pragma unroll
            for (int i = 0; i < D / 16; ++i) {
                const uint32_t off = (i >> 2) * kBoxBytes + (i & 3) * 32;
                if (i == 0) mma_ss<false>(leader, tmem + kColS + 128 * t, dq, off, dk, off, idesc_s);
                else mma_ss<true>(leader, tmem + kColS + 128 * t, dq, off, dk, off, idesc_s);
            }
            mma_commit(leader, &bars[S_READY0 + t]);
            if (last_use_of_k) mma_commit(leader, &bars[K_EMPTY0 + st]);
            if (last_use_of_q) mma_commit(leader, &bars[Q_EMPTY0 + qs]);
        };
        const auto wait_q = [&](uint32_t qs) {
            ok = mbar_wait(&bars[Q_FULL0 + qs], (ph_qf >> qs) & 1, abort_flag);
            ph_qf ^= 1u << qs;
        };
        // O += P V of one tile with the v-th V tile overall
        const auto issue_pv = [&](uint32_t t, uint32_t v, bool first, int vrows, bool last_use_of_v) {
            const uint32_t st = v & 1;
            const uint32_t d_o = tmem + kColO + 128 * t, a_p = tmem + kColS + 128 * t + kColPOff;
            const SmemDesc dv = {desc_v.lo + st * (kTileBytes >> 4), desc_v.hi};
            ok = mbar_wait(&bars[V_FULL0 + st], (v >> 1) & 1, abort_flag) && mbar_wait(&bars[P_RIGHT0 + t], (ph_p >> t) & 1, abort_flag);
            if (!ok) return;
            if (first) {  // the tile's previous O must have been read out
                ok = mbar_wait(&bars[O_FREE0 + t], (ph_of >> t) & 1, abort_flag) && mbar_wait(&bars[P_LEFT0 + t], (ph_p >> t) & 1, abort_flag);
                ph_of ^= 1u << t;
                if (!ok) return;
                // Ragged end of the sequence (upper tile only): the slices of 16 keys behind the end are not issued, the rows between the
                // end and the next multiple of 16 are set to zero: they meet weights of zero, which do not silence a NaN.
                if (vrows < kBN && (vrows & 15)) {
                    zero_rows_to_16(sV + st * kTileBytes, kBoxes, kBoxBytes, vrows, lane);
                    zero_rows_done();
                }
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < kBN / 16; ++i) {
                    if (i == 0) mma_ts<false>(leader, d_o, a_p, dv, 0, idesc_o);
                    else if (16 * i < vrows) mma_ts<true>(leader, d_o, a_p + i * 8, dv, i * 2048, idesc_o);
                }
            } else {
                tc_fence_after();
#pragma unroll
                for (int i = 4; i < 8; ++i) mma_ts<true>(leader, d_o, a_p + i * 8, dv, i * 2048, idesc_o);
                ok = mbar_wait(&bars[P_LEFT0 + t], (ph_p >> t) & 1, abort_flag);
                if (!ok) return;
                tc_fence_after();
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_ts<true>(leader, d_o, a_p + i * 8, dv, i * 2048, idesc_o);
            }
            ph_p ^= 1u << t;
            if (last_use_of_v) mma_commit(leader, &bars[V_EMPTY0 + st]);
        };
        SchedConsumer sched;
        Work wk, nx;
        bool have = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, wk, leader, true) >= 0;
        // Upper tile: step r meets K and V tile kbase + r.  Lower tile: step r meets tile kbase + r + 1, half a round before the upper one.
        uint32_t q0 = 0, q1 = 0;
        // S of the first step of an item, lower tile / upper tile
        const auto begin_lower = [&](const Work& e, uint32_t kb) {
            q1 = next_slot == kQSlots - 1 ? 0 : next_slot + 1;
            wait_q(q1);
            if (ok) issue_s(1, q1, kb + 1, false, e.qt == 1);
        };
        const auto begin_upper = [&](const Work& e, uint32_t kb) {
            q0 = next_slot;
            const uint32_t used = e.qt > 0 ? 2u : 1u;
            next_slot += used;
            if (next_slot >= kQSlots) next_slot -= kQSlots;
            wait_q(q0);
            if (ok) issue_s(0, q0, kb, true, e.qt == 0);
        };
        if (have) {
            // (begin_lower looks at next_slot, which begin_upper moves on)
            if (wk.qt > 0) begin_lower(wk, 0);
            if (ok) begin_upper(wk, 0);
        }
        while (ok && have) {
            const int n = wk.qt + 1;  // steps of the upper tile; the lower one has n - 1
            bool more = false;
            for (int r = 0; ok && r < n; ++r) {
                if (r + 1 == n) {  // the lower tile is through: its next item begins
                    more = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, nx, leader, true) >= 0;
                    if (more && nx.qt > 0) begin_lower(nx, kbase + n);
                    if (!ok) break;
                }
                issue_pv(0, kbase + r, r == 0, r == 0 ? wk.len - wk.qt * kBM : kBN, true);
                if (!ok) break;
                if (r + 1 < n) {
                    issue_s(0, q0, kbase + r + 1, true, r + 2 == n);
                    if (!ok) break;
                    issue_pv(1, kbase + r + 1, r == 0, kBN, false);
                    if (!ok) break;
                    if (r + 2 < n) issue_s(1, q1, kbase + r + 2, false, r + 3 == n);
                    else mma_commit(leader, &bars[O_READY1]);
                }
            }
            if (!ok) break;
            mma_commit(leader, &bars[O_READY0]);
            kbase += n;
            have = more;
            wk = nx;
            if (have) begin_upper(wk, kbase);
        }
    } else {
        // ------------------------------------------------------------------ row threads
        const int tile = warp >> 2;            // 0: upper tile of the pair, 1: lower
        const int r = (warp & 3) * 32 + lane;  // row of the tile == TMEM lane
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t s_base = lane_base + kColS + 128 * tile, o_base = lane_base + kColO + 128 * tile;
        const float scale = a.inv_temp * kLog2e;
        const int lim = a.attend_current ? r + 1 : r;  // diagonal tile: columns < lim are visible
        const bool save = a.carry_w != nullptr;
        uint32_t g = 0, items = 0;  // steps and items of this tile so far
        bool ok = true;
        SchedConsumer sched;
        Work wk;
        int w = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, wk, false);
        while (ok && w >= 0) {
            sched.release(&bars[WORK_EMPTY0]);
            const int qt = wk.qt - tile;
            if (qt < 0) {
                w = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, wk, false);
                continue;
            }
            const int qi = qt * kBM + r;
            const bool row_ok = qi < wk.len;
            float* cw = save ? a.carry_w + ((int64_t)wk.h * a.slot_cap + carry_slot32(wk.slot_base, qt, 4 * qt)) * kTileQ + r : nullptr;
            float W = 1.f;
            for (int kt = qt; kt >= 0; --kt, ++g) {
                ok = mbar_wait(&bars[S_READY0 + tile], g & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                if (kt == qt) step_diagonal<kF16>(s_base, scale, lim, warp & 3, W, cw, save, &bars[P_RIGHT0 + tile]);
                else step_full<kF16>(s_base, scale, W, cw, save, &bars[P_RIGHT0 + tile]);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars[P_LEFT0 + tile]);
                cw -= 4 * kTileQ;
            }
            if (!ok) break;
            const int64_t tok = wk.start + qi;
            // the row of v, a chunk of 32 columns ahead of its use
            const char* vrow = a.v.ptr + 2 * ((int64_t)wk.b * a.v.sb + (int64_t)wk.h * a.v.sh + (row_ok ? tok : wk.start) * a.v.st);
            Row32 vx;
            if (kFused) vx.load(vrow);
            if (row_ok) {
                char* rp = a.rem.ptr + 2 * ((int64_t)wk.b * a.rem.sb + (int64_t)wk.h * a.rem.sh + tok * a.rem.st);
                if (kF16) *(__half*)rp = __float2half_rn(W);
                else *(__nv_bfloat16*)rp = __float2bfloat16_rn(W);
                ((float*)a.nla.ptr)[(int64_t)wk.b * a.nla.sb + (int64_t)wk.h * a.nla.sh + tok * a.nla.st] = lg2_approx(W);
            }
            char* orow = a.o.ptr + 2 * ((int64_t)wk.b * a.o.sb + (int64_t)wk.h * a.o.sh + tok * a.o.st);
            // the next item is read from the ring while this one's last contraction completes
            w = sched.next(ring, &bars[WORK_FULL0], &bars[WORK_EMPTY0], abort_flag, wk, false);
            ok = mbar_wait(&bars[O_READY0 + tile], items & 1, abort_flag);
            ++items;
            if (!ok) break;
            tc_fence_after();
            const float remf = round16<kF16>(W);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                uint32_t v[32];
                tmem_ld32(o_base + 32 * c, v);
                tmem_wait_ld(v);
                if (c == D / 32 - 1) {
                    tc_fence_before();
                    mbar_arrive(&bars[O_FREE0 + tile]);
                }
                if (kFused) {  // out = o + rem * v, rem rounded to the output type first
                    float x[32];
                    unpack_row32<kF16>(vx, x);
                    if (c + 1 < D / 32) vx.load(vrow + 64 * (c + 1));
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(fmaf(remf, x[i], __uint_as_float(v[i])));
                }
                store_row32_pairs<kF16>(orow + 64 * c, v, 1.f, (int64_t)a.o.st * 2, row_ok, lane);
            }
        }
    }
    tc_teardown(abort_flag, a.status, tmem, kTmemCols, 9);
    sched_finish(a.sched + 0);
}

template <bool kF16>
int launch_t(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    CUtensorMap mq, mk, mv;
    const int kind = kF16 ? 2 : 0;
    const int64_t B = p.batch > 0 ? p.batch : 1;
    const int hd = p.head_dim;
    if (encode_tile_map(&mq, p.q.ptr, kind, hd, p.tokens, p.heads, B, p.q.stride_t, p.q.stride_h, p.q.stride_b, kBM) ||
        encode_tile_map(&mk, p.k.ptr, kind, hd, p.tokens, p.heads, B, p.k.stride_t, p.k.stride_h, p.k.stride_b, kBN) ||
        encode_tile_map(&mv, p.v.ptr, kind, hd, p.tokens, p.heads, B, p.v.stride_t, p.v.stride_h, p.v.stride_b, kBN))
        return kMapEncodeFailed;
    constexpr int smem = (kQSlots + 4) * kBM * kMaxHeadDim * 2 + 1024;  // tiles, barriers and the scheduler's ring: one block per SM
    static_assert(smem <= 232448, "shared memory of a block");
    static_assert(kNumBars * 8 + sizeof(SchedRing<Work>) + 16 <= 1024, "small data");
    const auto launch = [&](auto kernel) {
        const int e = ensure_kernel_attrs((const void*)kernel, smem, false);
        if (e != 0) return e;
        return launch_kernel(kernel, dim3(persistent_grid((int64_t)L.max_items * p.heads)), dim3(kThreads), smem, st, mq, mk, mv, a);
    };
    return a.fused ? launch(tc_fwd_pair_kernel<kF16, true>) : launch(tc_fwd_pair_kernel<kF16, false>);
}

}  // namespace

int launch_tensor_fwd_pair(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    return p.dtype == SBATTN_F16 ? launch_t<true>(p, L, a, st) : launch_t<false>(p, L, a, st);
}

}  // namespace sb
