// Tensor-core backward (sm_100a) for packs whose sequences have at most 128 tokens: dq, dk and dv in one kernel.
//
// A sequence is one 128 x 128 tile of scores then, so nothing crosses between tiles: the scores, the weights and the gradients of
// the scores are formed once, all five contractions of the tile follow, and q, k, v, do are read once (the two kernels of
// sb_tc_bwd.cu read them twice).  Same arithmetic as there (the reference's _backward_one_row,
// stickbreaking_attention/sb_varlen/sb_varlen_bwd.py:401-473).
//
// What bounds it is memory: seven matrices per item, 224 KB at head dim 128, ~10 000 cycles of the SM's share of the DRAM
// bandwidth.  Contractions, arithmetic, read-out and stores of an item take about as long one after the other, so the loads,
// S and dP of the next item run while the results of this one are stored, and the row threads read the next item and its scalars (the carry, drem)
// before these stores: at the item's start the ring, the table entry and two dependent loads cost 3 000 of 14 000 cycles.  32 heads, 512 sequences of
// 128 tokens, bf16, head dim 128: 757 -> 640 us for this kernel (575 at the copy bandwidth), forward + backward 1.32 -> 1.23 ms (1.76 ms with the two
// kernels).  Two slots for q and k, with p in the place of v, were slower (757 -> 833, with the early reads 640 -> 665).
//
// One persistent block of 576 threads per SM: warps 0-15 row warps (a thread owns one query row and 32 keys, warps 0-3 the
// rightmost quarter ... 12-15 the leftmost), warp 16 TMA producer, warp 17 issues tcgen05.mma.
// Tensor memory (512 columns): S, dP (dQ takes its place), dK, dV.
#include "sb_tc_bwd_common.cuh"

namespace sb {

using namespace sm100;
using namespace bwd;

namespace {

constexpr int kThreads = 576;  // 18 warps put five on one scheduler, which caps a thread at 96 registers
template <int D> constexpr int kTileStages = D > 64 ? 1 : 2;  // slots for q, k, v, do
constexpr int kSmall = 4096;                                  // bytes behind the tiles: exchange slots, barriers, scheduler ring
enum TileBar { T_Q_FULL0, T_Q_FULL1, T_V_FULL0, T_V_FULL1,    // q and k / v and do have arrived (per slot)
               T_Q_EMPTY0, T_Q_EMPTY1, T_K_EMPTY0, T_K_EMPTY1, T_V_EMPTY0, T_V_EMPTY1, T_DO_EMPTY0, T_DO_EMPTY1,
               T_SDP_READY, T_P_READY, T_DS_READY, T_DQ_READY, T_DQ_FREE, T_DKV_READY, T_DKV_FREE,
               T_WORK_FULL0, T_WORK_FULL1, T_WORK_EMPTY0, T_WORK_EMPTY1,
               T_X0,  // 12 barriers for the totals of g: [quarter 0 ... 2][warp & 3]
               kNumTileBars = T_X0 + 12 };

// Right to left over 32 columns: s <- 1 - beta, dp <- g = p * (dp - drem), pp <- the weights p = W * beta; returns the sum of g
template <bool kF16>
__device__ __forceinline__ float tile_grads(uint32_t (&s)[32], uint32_t (&dp)[32], float scale, int col0, int lim, float drem, float W,
                                            uint32_t (&pp)[16]) {
    float2 tot = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 7; q >= 0; --q) {
        float2 om[2];
        stick4<true, false>(__uint_as_float(s[4 * q]), __uint_as_float(s[4 * q + 1]), __uint_as_float(s[4 * q + 2]), __uint_as_float(s[4 * q + 3]),
                            scale, col0 + 4 * q, lim, om[0], om[1]);
#pragma unroll
        for (int h = 1; h >= 0; --h) {
            const int jj = 2 * q + h;
            const float2 t = __fadd2_rn(make_float2(__uint_as_float(dp[2 * jj]), __uint_as_float(dp[2 * jj + 1])), make_float2(-drem, -drem));
            const float w1 = W * om[h].y, p1 = W - w1;
            const float w0 = w1 * om[h].x, p0 = w1 - w0;
            W = w0;
            const float2 g = __fmul2_rn(make_float2(p0, p1), t);
            tot = __fadd2_rn(tot, g);
            pp[jj] = pack16<kF16>(p0, p1);
            s[2 * jj] = __float_as_uint(om[h].x);
            s[2 * jj + 1] = __float_as_uint(om[h].y);
            dp[2 * jj] = __float_as_uint(g.x);
            dp[2 * jj + 1] = __float_as_uint(g.y);
        }
    }
    return tot.x + tot.y;
}
// ds = g - beta * c = om * c - (c - g), right to left; c enters as the inclusive prefix of g at the right edge
template <bool kF16>
__device__ __forceinline__ void tile_ds(const uint32_t (&om)[32], const uint32_t (&g)[32], float c, uint32_t (&ps)[16]) {
#pragma unroll
    for (int jj = 15; jj >= 0; --jj) {
        const float c1 = c - __uint_as_float(g[2 * jj + 1]);
        const float ds1 = fmaf(__uint_as_float(om[2 * jj + 1]), c, -c1);
        const float c0 = c1 - __uint_as_float(g[2 * jj]);
        const float ds0 = fmaf(__uint_as_float(om[2 * jj]), c1, -c0);
        c = c0;
        ps[jj] = pack16<kF16>(ds0, ds1);
    }
}

template <int D, bool kF16, bool kFused>
__global__ void __launch_bounds__(608, 1)
tc_bwd_tile_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ CUtensorMap map_do, const __grid_constant__ KArgs a) {
    constexpr int kBoxes = D / 64;
    constexpr int kTile = kBM * D * 2;   // a 128-row tile of Q, dO, K or V
    constexpr int kPBytes = 2 * kQBox;   // 128 query rows x 128 keys, 16-bit, as two 64-key blocks
    constexpr int kSt = kTileStages<D>;
    constexpr uint32_t kColS = 0, kColDP = 128, kColDK = 256, kColDV = 256 + D, kCols = 512;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;  // kSt slots of each
    uint8_t* sK = sQ + kSt * kTile;
    uint8_t* sV = sK + kSt * kTile;
    uint8_t* sDO = sV + kSt * kTile;
    uint8_t* sP = sDO + kSt * kTile;
    uint8_t* sDS = sP + kPBytes;
    float* xg = (float*)(sDS + kPBytes);  // [quarter 0 ... 2][128 rows]: the totals of g
    uint64_t* bars = (uint64_t*)(xg + 384);
    uint32_t* tmem_slot = (uint32_t*)(bars + kNumTileBars);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    SchedRing<KvWork>* ring = (SchedRing<KvWork>*)(tmem_slot + 2);
    static_assert(4 * 384 + 8 * kNumTileBars + 8 + sizeof(SchedRing<KvWork>) <= kSmall, "the small arrays do not fit their place");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kNumTileBars; ++i) {
            uint32_t cnt = 1;
            if (i == T_P_READY || i == T_DS_READY || i == T_DQ_FREE || i == T_DKV_FREE) cnt = 512;
            if (i >= T_X0) cnt = 32;
            if (i == T_WORK_EMPTY0 || i == T_WORK_EMPTY1) cnt = 17;  // MMA warp, 16 row warps
            mbar_init(&bars[i], cnt);
        }
        *abort_flag = (smem_u32(smem) & 1023u) ? 1u : 0u;  // the swizzled tiles need a 1024-byte aligned base
        fence_barrier_init();
    }
    if (warp == 17) {
        tmem_alloc(tmem_slot, kCols);
        tmem_relinquish();
    }
    if (warp == 16 && lane == 0) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        tma_prefetch_desc(&map_do);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_wait();
    pdl_launch_dependents();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) {
        const int64_t me = (int64_t)blockIdx.x * kThreads + tid, all = (int64_t)gridDim.x * kThreads;
        if (kF16) zero_tail_grads<__half>(a, a.hdr->covered_end, me, all);
        else zero_tail_grads<__nv_bfloat16>(a, a.hdr->covered_end, me, all);
    }
    const int n_items = a.hdr->n_items;
    const int n_work = *abort_flag ? 0 : n_items * a.heads;
    // i counts the items of this block: item i uses slot i % kSt for the (i / kSt)-th time; a barrier that completes once per item is
    // in phase i & 1.

    if (warp == 16) {
        // ------------------------------------------------------------------ TMA producer: in the order in which the slots fall free
        if (lane == 0) {
            bool ok = true;
            SchedProducer sched;
            int w;
            KvWork wk;
            const auto fetch = [&](int w_) { return fetch_kv_work(a, n_items, w_); };
            for (uint32_t i = 0; ok && (w = sched.next(a.sched + 4, n_work, ring, &bars[T_WORK_FULL0], &bars[T_WORK_EMPTY0], abort_flag, fetch, wk)) >= 0; ++i) {
                const uint32_t st = i % kSt, ph = ((i / kSt) & 1) ^ 1;
                const auto load = [&](uint8_t* base, const CUtensorMap* m, int empty, int full) {
                    ok = ok && mbar_wait_idle(&bars[empty + st], ph, abort_flag);
                    if (!ok) return;
#pragma unroll
                    for (int bx = 0; bx < kBoxes; ++bx)
                        tma_load_4d(base + st * kTile + bx * kQBox, m, &bars[full + st], bx * 64, wk.start, wk.h, wk.b);
                };
                ok = mbar_wait_idle(&bars[T_V_EMPTY0 + st], ph, abort_flag);
                if (!ok) break;
                mbar_expect_tx(&bars[T_V_FULL0 + st], 2 * kTile);
                load(sV, &map_v, T_V_EMPTY0, T_V_FULL0);
                load(sDO, &map_do, T_DO_EMPTY0, T_V_FULL0);
                if (ok) ok = mbar_wait_idle(&bars[T_K_EMPTY0 + st], ph, abort_flag);
                if (!ok) break;
                mbar_expect_tx(&bars[T_Q_FULL0 + st], 2 * kTile);
                load(sK, &map_k, T_K_EMPTY0, T_Q_FULL0);
                load(sQ, &map_q, T_Q_EMPTY0, T_Q_FULL0);
            }
        }
    } else if (warp == 17) {
        // ------------------------------------------------------------------ MMA issuer
        {
            const bool leader = elect_one();  // the whole warp runs the loops; one lane issues
            constexpr uint32_t idesc_s = make_idesc(kBM, kKT, kF16 ? 0 : 1, 0, 0);
            constexpr uint32_t idesc_t = make_idesc(kKT, D, kF16 ? 0 : 1, 1, 1);   // (P^T or dS^T)[128 keys x q] * (dO or Q)[q x D]
            constexpr uint32_t idesc_dq = make_idesc(kBM, D, kF16 ? 0 : 1, 0, 1);  // dS[q x keys] * K[keys x D]
            const SmemDesc desc_q = make_desc(smem_u32(sQ), 0, 1024), desc_do = make_desc(smem_u32(sDO), 0, 1024);  // K-major
            const SmemDesc desc_k = make_desc(smem_u32(sK), 0, 1024), desc_v = make_desc(smem_u32(sV), 0, 1024);
            const SmemDesc desc_qmn = make_desc(smem_u32(sQ), kQBox, 1024), desc_domn = make_desc(smem_u32(sDO), kQBox, 1024);  // MN-major
            const SmemDesc desc_kmn = make_desc(smem_u32(sK), kQBox, 1024);
            const SmemDesc desc_pt = make_desc(smem_u32(sP), kQBox, 1024), desc_dst = make_desc(smem_u32(sDS), kQBox, 1024);
            const SmemDesc desc_ds = make_desc(smem_u32(sDS), 0, 1024);
            const auto at = [](SmemDesc d, uint32_t slot) { return SmemDesc{d.lo + slot * (uint32_t)(kTile >> 4), d.hi}; };
            bool ok = true;
            SchedConsumer sched;
            int w;
            KvWork wk;
            for (uint32_t i = 0; ok && (w = sched.next(ring, &bars[T_WORK_FULL0], &bars[T_WORK_EMPTY0], abort_flag, wk, leader, true)) >= 0; ++i) {
                const uint32_t st = i % kSt, use = (i / kSt) & 1, ph = i & 1;
                const int rows = wk.len;  // 1 ... 128
                // Rows of the tiles behind the end of the sequence belong to the next sequence or to nobody, and a zero weight does not
                // silence a NaN.  K, V: set to zero.  Q, dO: dk, dv contract over query rows in slices of 16; slices behind the end
                // are not issued, the rows between the end and the next multiple of 16 are set to zero (S, dP, p, ds of them are
                // zero then).
                ok = mbar_wait(&bars[T_V_FULL0 + st], use, abort_flag);
                if (!ok) break;
                if (rows < kBM) {
                    zero_rows(sV + st * kTile, kBoxes, kQBox, rows, kBM, lane);
                    if (rows & 15) zero_rows_to_16(sDO + st * kTile, kBoxes, kQBox, rows, lane);
                    zero_rows_done();
                }
                ok = mbar_wait(&bars[T_DQ_FREE], ph ^ 1, abort_flag);  // the previous dQ, in the columns of dP, has been read out
                if (!ok) break;
                tc_fence_after();
                {
                    const SmemDesc x = at(desc_do, st), y = at(desc_v, st);
#pragma unroll
                    for (int k = 0; k < D / 16; ++k) {
                        const uint32_t o = (k >> 2) * kQBox + (k & 3) * 32;
                        if (k == 0) mma_ss<false>(leader, tmem + kColDP, x, o, y, o, idesc_s);
                        else mma_ss<true>(leader, tmem + kColDP, x, o, y, o, idesc_s);
                    }
                    mma_commit(leader, &bars[T_V_EMPTY0 + st]);
                }
                ok = mbar_wait(&bars[T_Q_FULL0 + st], use, abort_flag);
                if (!ok) break;
                if (rows < kBM) {
                    zero_rows(sK + st * kTile, kBoxes, kQBox, rows, kBM, lane);
                    if (rows & 15) zero_rows_to_16(sQ + st * kTile, kBoxes, kQBox, rows, lane);
                    zero_rows_done();
                }
                tc_fence_after();  // S: the previous scores were in registers before dQ was issued
                {
                    const SmemDesc x = at(desc_q, st), y = at(desc_k, st);
#pragma unroll
                    for (int k = 0; k < D / 16; ++k) {
                        const uint32_t o = (k >> 2) * kQBox + (k & 3) * 32;
                        if (k == 0) mma_ss<false>(leader, tmem + kColS, x, o, y, o, idesc_s);
                        else mma_ss<true>(leader, tmem + kColS, x, o, y, o, idesc_s);
                    }
                    mma_commit(leader, &bars[T_SDP_READY]);
                }
                ok = mbar_wait(&bars[T_P_READY], ph, abort_flag) && mbar_wait(&bars[T_DKV_FREE], ph ^ 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                {
                    const SmemDesc y = at(desc_domn, st);
#pragma unroll
                    for (int k = 0; k < kBM / 16; ++k) {
                        if (k == 0) mma_ss<false>(leader, tmem + kColDV, desc_pt, 0, y, 0, idesc_t);
                        else if (16 * k < rows) mma_ss<true>(leader, tmem + kColDV, desc_pt, k * 2048, y, k * 2048, idesc_t);
                    }
                    mma_commit(leader, &bars[T_DO_EMPTY0 + st]);
                }
                ok = mbar_wait(&bars[T_DS_READY], ph, abort_flag);
                if (!ok) break;
                tc_fence_after();
                {
                    const SmemDesc y = at(desc_kmn, st);
#pragma unroll
                    for (int k = 0; k < kKT / 16; ++k) {
                        const uint32_t o = (k >> 2) * kQBox + (k & 3) * 32;
                        if (k == 0) mma_ss<false>(leader, tmem + kColDP, desc_ds, o, y, 0, idesc_dq);
                        else if (16 * k < rows) mma_ss<true>(leader, tmem + kColDP, desc_ds, o, y, k * 2048, idesc_dq);
                    }
                    mma_commit(leader, &bars[T_DQ_READY]);
                    mma_commit(leader, &bars[T_K_EMPTY0 + st]);
                }
                {
                    const SmemDesc y = at(desc_qmn, st);
#pragma unroll
                    for (int k = 0; k < kBM / 16; ++k) {
                        if (k == 0) mma_ss<false>(leader, tmem + kColDK, desc_dst, 0, y, 0, idesc_t);
                        else if (16 * k < rows) mma_ss<true>(leader, tmem + kColDK, desc_dst, k * 2048, y, k * 2048, idesc_t);
                    }
                    mma_commit(leader, &bars[T_DKV_READY]);
                    mma_commit(leader, &bars[T_Q_EMPTY0 + st]);
                }
            }
        }
    } else if (warp < 16) {
        // ------------------------------------------------------------------ row threads
        const int kq = 3 - (warp >> 2);        // 32-key quarter of the tile this thread owns
        const int hf = kq >> 1, sub = kq & 1;  // its 64-key half (a block of the P / dS buffers) and the quarter inside it
        const int r = (warp & 3) * 32 + lane;
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const float scale = a.inv_temp * kLog2e;
        uint8_t* prow = sP + hf * kQBox + r * 128;
        uint8_t* srow = sDS + hf * kQBox + r * 128;
        const int kv_chunks = max(0, min(D / 64, a.head_dim / 32 - hf * (D / 64)));  // 32-column chunks of dk / dv this thread stores
        bool ok = true;
        SchedConsumer sched;
        int w;
        KvWork wk, nx;
        // The next item and its scalars are fetched as soon as this one's gradients of the scores are out, and arrive under its stores
        float W = 0.f;
        uint32_t drem_raw = 0u;  // drem stays as it was loaded until it is used: a conversion behind the load would wait for it
        const auto next_item = [&]() {
            w = sched.next(ring, &bars[T_WORK_FULL0], &bars[T_WORK_EMPTY0], abort_flag, nx, false, true);
            W = 0.f;
            drem_raw = 0u;
            if (w < 0 || r >= nx.len) return;
            // a quarter behind the end of the sequence (in a half whose carry slots do not exist) has no visible key: any W does
            if (64 * hf < nx.len) W = __ldg(a.carry_w + ((int64_t)nx.h * a.slot_cap + carry_slot32(nx.slot_base, 0, kq)) * kTileQ + r);
            const int64_t tok = nx.start + r;
            if (kFused) {  // drem + do . v
                drem_raw = __ldg((const uint32_t*)a.drem_eff + (int64_t)nx.h * a.drem_rows + (int64_t)nx.b * a.tokens + tok);
            } else {
                const char* dp = a.d_rem.ptr + 2 * ((int64_t)nx.b * a.d_rem.sb + (int64_t)nx.h * a.d_rem.sh + tok * a.d_rem.st);
                drem_raw = __ldg((const unsigned short*)dp);
            }
        };
        next_item();
        for (uint32_t i = 0; ok && w >= 0; ++i) {
            const uint32_t ph = i & 1;
            wk = nx;
            if (lane == 0) sched.release(&bars[T_WORK_EMPTY0]);
            const bool row_ok = r < wk.len;
            const int64_t tok = wk.start + r;
            // Columns < lim of the quarter are visible.  None to a row behind the end of the sequence: its zero query against an infinite
            // or NaN key would make a NaN of every weight to the left, and dk, dv contract over such rows up to a multiple of 16.
            const int lim = row_ok ? r + a.attend_current - 32 * kq : 0;
            ok = mbar_wait(&bars[T_SDP_READY], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            uint32_t om[32], gv[32];
            tmem_ld32(lane_base + kColS + 32 * kq, om);
            tmem_ld32(lane_base + kColDP + 32 * kq, gv);
            tmem_wait_ld(om, gv);
            tc_fence_before();
            const float drem = kFused ? __uint_as_float(drem_raw) : kF16 ? __half2float(__ushort_as_half((unsigned short)drem_raw)) : __uint_as_float(drem_raw << 16);
            float tot;
            {
                uint32_t pp[16];
                tot = tile_grads<kF16>(om, gv, scale, 0, lim, drem, W, pp);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch)
                    *(uint4*)(prow + (((4 * sub + ch) ^ (r & 7)) << 4)) = make_uint4(pp[4 * ch], pp[4 * ch + 1], pp[4 * ch + 2], pp[4 * ch + 3]);
                fence_async_smem();
                mbar_arrive(&bars[T_P_READY]);
            }
            // prefix of g through the quarter's right edge: the totals of the quarters to the left, and its own
            float c = tot;
            if (kq < 3) {
                xg[kq * 128 + r] = tot;
                mbar_arrive(&bars[T_X0 + 4 * kq + (warp & 3)]);
            }
            for (int q = 0; ok && q < kq; ++q) {
                ok = mbar_wait(&bars[T_X0 + 4 * q + (warp & 3)], ph, abort_flag);
                if (ok) c += xg[q * 128 + r];
            }
            if (!ok) break;
            {
                uint32_t ps[16];
                tile_ds<kF16>(om, gv, c, ps);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch)
                    *(uint4*)(srow + (((4 * sub + ch) ^ (r & 7)) << 4)) = make_uint4(ps[4 * ch], ps[4 * ch + 1], ps[4 * ch + 2], ps[4 * ch + 3]);
                fence_async_smem();
                mbar_arrive(&bars[T_DS_READY]);
            }
            next_item();
            // dq: a quarter of the columns per thread; then the next item's dP may overwrite it
            ok = mbar_wait(&bars[T_DQ_READY], ph, abort_flag);
            if (!ok) break;
            tc_fence_after();
            char* orow = a.dq.ptr + 2 * ((int64_t)wk.b * a.dq.sb + (int64_t)wk.h * a.dq.sh + tok * a.dq.st);
            if (kq < D / 32) {
                uint32_t v[32];
                tmem_ld32(lane_base + kColDP + 32 * kq, v);
                tmem_wait_ld(v);
                tc_fence_before();
                mbar_arrive(&bars[T_DQ_FREE]);
                store_row32_pairs<kF16>(orow + 64 * kq, v, a.inv_temp, (int64_t)a.dq.st * 2, row_ok && (D == 128 || a.head_dim > 32 * kq), lane);
            } else {
                mbar_arrive(&bars[T_DQ_FREE]);
            }
            ok = mbar_wait(&bars[T_DKV_READY], ph, abort_flag);
            if (!ok) break;
            kv_store_rows_inl<D, kF16, kFused>(a, sub == 1, wk, r, lane_base + (sub == 0 ? kColDK : kColDV), hf * (D / 64), kv_chunks);
            mbar_arrive(&bars[T_DKV_FREE]);
        }
    }
    tc_teardown(abort_flag, a.status, tmem, kCols, 17);
    sched_finish(a.sched + 4);
}

template <int D, bool kF16>
int launch_t(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    CUtensorMap mq, mk, mv, mdo;
    const int kind = kF16 ? 2 : 0;
    const int64_t B = p.batch > 0 ? p.batch : 1;
    const int hd = p.head_dim;  // the maps carry the true head dim; TMA fills the columns up to D with zeros
    if (encode_tile_map(&mq, p.q.ptr, kind, hd, p.tokens, p.heads, B, p.q.stride_t, p.q.stride_h, p.q.stride_b, kBM) ||
        encode_tile_map(&mk, p.k.ptr, kind, hd, p.tokens, p.heads, B, p.k.stride_t, p.k.stride_h, p.k.stride_b, kBM) ||
        encode_tile_map(&mv, p.v.ptr, kind, hd, p.tokens, p.heads, B, p.v.stride_t, p.v.stride_h, p.v.stride_b, kBM) ||
        encode_tile_map(&mdo, p.d_o.ptr, kind, hd, p.tokens, p.heads, B, p.d_o.stride_t, p.d_o.stride_h, p.d_o.stride_b, kBM))
        return kMapEncodeFailed;
    if (a.fused) {
        const int e = launch_drem(p, a, st);
        if (e != 0) return e;
    }
    constexpr int smem = 4 * kTileStages<D> * kBM * D * 2 + 2 * 2 * kQBox + kSmall;
    const auto launch = [&](auto kernel) {
        const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
        if (e != 0) return e;
        return launch_kernel(kernel, dim3(persistent_grid((int64_t)L.max_items * p.heads)), dim3(kThreads), smem, st, mq, mk, mv, mdo, a);
    };
    return a.fused ? launch(tc_bwd_tile_kernel<D, kF16, true>) : launch(tc_bwd_tile_kernel<D, kF16, false>);
}

}  // namespace

int launch_tensor_bwd_tile(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    const bool f16 = p.dtype == SBATTN_F16;
    if (p.head_dim > 64) return f16 ? launch_t<128, true>(p, L, a, st) : launch_t<128, false>(p, L, a, st);
    return f16 ? launch_t<64, true>(p, L, a, st) : launch_t<64, false>(p, L, a, st);
}

}  // namespace sb
