// Shared by the backward kernels: the per-score arithmetic, the (head, sequence, key tile) work items and the epilogue of dk, dv.
#pragma once

#include "sb_tc_common.cuh"

namespace sb {

namespace bwd {

using namespace sm100;

constexpr int kBM = 128;  // query rows per tile
constexpr int kBK = 64;   // keys per half of a step: the unit of masking and a 128-byte row of the p / ds buffers
constexpr int kKT = 128;  // keys per stationary tile
constexpr int kQBox = 128 * 128;  // bytes of one TMA box of a 128-row tile (64 elements wide)
constexpr int kKBox = 64 * 128;   // bytes of one TMA box of a 64-row tile

// Element-wise core shared by the backward kernels, four adjacent scores at a time: om = 1 - beta = 1 / (1 + 2^(s * scale));
// masked keys get om = 1 (no stick broken, weight 0).  The operations without a dependency along the row are packed
// fp32x2 instructions, and the four reciprocals cost one MUFU operation: with d_i = 1 + e_i,
// 1 / d_i = (product of the other three) / (d_0 d_1 d_2 d_3).  The exponent is clamped at 30 so that the product of four
// stays finite (om = 2^-30 instead of something smaller: no visible difference).
template <bool kMasked, bool kGrouped = true>
__device__ __forceinline__ void stick4(float s0, float s1, float s2, float s3, float scale, int col, int lim, float2& om01,
                                       float2& om23) {
    float2 x01 = __fmul2_rn(make_float2(s0, s1), make_float2(scale, scale));
    float2 x23 = __fmul2_rn(make_float2(s2, s3), make_float2(scale, scale));
    if (kGrouped) {
        x01.x = fminf(x01.x, 30.f);
        x01.y = fminf(x01.y, 30.f);
        x23.x = fminf(x23.x, 30.f);
        x23.y = fminf(x23.y, 30.f);
    }
    if (kMasked) {
        if (col >= lim) x01.x = -INFINITY;
        if (col + 1 >= lim) x01.y = -INFINITY;
        if (col + 2 >= lim) x23.x = -INFINITY;
        if (col + 3 >= lim) x23.y = -INFINITY;
    }
    const float2 d01 = __fadd2_rn(make_float2(ex2_approx(x01.x), ex2_approx(x01.y)), make_float2(1.f, 1.f));
    const float2 d23 = __fadd2_rn(make_float2(ex2_approx(x23.x), ex2_approx(x23.y)), make_float2(1.f, 1.f));
    if (!kGrouped) {
        om01 = make_float2(rcp_approx(d01.x), rcp_approx(d01.y));
        om23 = make_float2(rcp_approx(d23.x), rcp_approx(d23.y));
        return;
    }
    const float2 m = __fmul2_rn(d01, d23);  // (d0 d2, d1 d3)
    const float r = rcp_approx(m.x * m.y);
    const float2 rm = make_float2(r * m.y, r * m.x);  // (1 / (d0 d2), 1 / (d1 d3))
    om01 = __fmul2_rn(rm, d23);
    om23 = __fmul2_rn(rm, d01);
}

struct KvWork {
    int h, b, start, len, kt, slot_base, n_qt;
};
__device__ __forceinline__ KvWork fetch_kv_work(const KArgs& a, int n_items, int w) {
    // groups of head_group heads; inside a group the 128-key tiles heaviest first (key tiles are heaviest where
    // query tiles are lightest: the item table is walked backwards), the heads of the group innermost
    const int per_group = n_items * a.head_group;
    const int g = w / per_group, rest = w - g * per_group;
    const int hg = min(a.head_group, a.heads - g * a.head_group);
    const int idx = rest / hg;
    const int2 it = a.items[n_items - 1 - idx];
    const SeqInfo s = a.seqs[it.x];
    KvWork k;
    k.h = g * a.head_group + rest - idx * hg;
    k.b = s.batch; k.start = s.start; k.len = s.len; k.slot_base = s.slot_base;
    k.kt = it.y;
    k.n_qt = (s.len + kBM - 1) / kBM;
    return k;
}

// dk or dv of a finished item out of tensor memory: a thread holds one key row and D / 2 columns of the head dim, from
// chunk0 * 32 on.
// Not inlined: it runs once per item, and inside the step loop it would only dilute the instruction cache.
// With the fused remainder dv also receives rem * do of its own row: the direct path of out = o + rem * v.
template <int D, bool kF16, bool kFused>
__device__ __forceinline__ void kv_store_rows_inl(const KArgs& a, bool is_dv, const KvWork e, int r, uint32_t taddr, int chunk0,
                                                  int n_chunks) {
    tc_fence_after();
    const MatView m = is_dv ? a.dv : a.dk;
    const float sc = is_dv ? 1.f : a.inv_temp;
    const bool key_ok = e.kt * kKT + r < e.len;
    const int64_t tok = e.start + e.kt * kKT + r;
    char* orow = m.ptr + 2 * ((int64_t)e.b * m.sb + (int64_t)e.h * m.sh + tok * m.st);
    const char* add = nullptr;
    float mul = 0.f;
    if (kFused && is_dv && key_ok) {
        add = a.d_o.ptr + 2 * ((int64_t)e.b * a.d_o.sb + (int64_t)e.h * a.d_o.sh + tok * a.d_o.st);
        const char* rp = a.rem.ptr + 2 * ((int64_t)e.b * a.rem.sb + (int64_t)e.h * a.rem.sh + tok * a.rem.st);
        mul = kF16 ? __half2float(*(const __half*)rp) : __bfloat162float(*(const __nv_bfloat16*)rp);
    }
#pragma unroll
    for (int cc = 0; cc < D / 64; ++cc) {  // this thread's half of the head dim, 32 columns at a time
        const int cidx = chunk0 + cc;
        uint32_t v[32];
        tmem_ld32(taddr + cidx * 32, v);
        tmem_wait_ld(v);
        if (!(kFused && is_dv)) {  // two rows per lane pair: -7 % on a pack of 128-token sequences, -0.6 % on long ones
            // (in the forward, whose threads store half as much, it gains at head dim 64 only)
            store_row32_pairs<kF16>(orow + cidx * 64, v, sc, (int64_t)m.st * 2, key_ok && (D == 128 || cc < n_chunks), (int)(threadIdx.x & 31));
        } else if (key_ok && (D == 128 || cc < n_chunks)) {  // D == 64 serves head dim 32 as well: then fewer chunks exist
            if (kFused && add) {
                float x[32];
                load_row32<kF16>(add + cidx * 64, x);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(fmaf(mul, x[i], __uint_as_float(v[i])));
                store_row32<kF16>(orow + cidx * 64, v, 1.f);
            } else {
                store_row32<kF16>(orow + cidx * 64, v, sc);
            }
        }
    }
    tc_fence_before();
}
template <int D, bool kF16, bool kFused>
__device__ __noinline__ void kv_store_rows(const KArgs& a, bool is_dv, const KvWork e, int r, uint32_t taddr, int chunk0, int n_chunks) {
    kv_store_rows_inl<D, kF16, kFused>(a, is_dv, e, r, taddr, chunk0, n_chunks);
}

}  // namespace bwd

}  // namespace sb
