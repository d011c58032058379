// Shared by the tensor-core forward kernels: scores to weights for chunks of 32 keys of one row.
#pragma once

#include "sb_tc_common.cuh"

namespace sb {

namespace fwd {

// With e = exp(s) and d = 1 + e:  beta = e / d,  1 - beta = 1 / d.  For key m of a group of 8 keys entered with the
// carry W (product of 1 - beta over everything to its right)
//     p_m = beta_m * W * prod_{m' > m in group} 1/d_m'  =  e_m * (prod_{m' < m in group} d_m') * W / (prod over the group of d)
// which needs one reciprocal per GROUP instead of one per key.  Scores are clamped at 2^15 (beta = 1 - 3e-5 there)
// so that the product of 8 factors stays below 2^127.  Masked keys get e = 0: weight 0 and no stick broken.
//
// First pass over a chunk of 32 keys: p <- e * (product of d over the keys of its group to the LEFT); run <- product of d over
// the group.  The four groups are swept side by side so that their chains overlap, and in pairs: p[h][m] holds key m of groups 2h
// and 2h + 1, so that every multiplication of the chains is one packed fp32x2 instruction for two keys (the exponentials deliver
// their results into whatever register the pairing wants).
template <bool kMasked>
__device__ __forceinline__ void fwd_sweep(const uint32_t (&s)[32], float scale, int col0, int lim, float2 (&p)[2][8], float2 (&run)[2]) {
    run[0] = run[1] = make_float2(1.f, 1.f);
#pragma unroll
    for (int m = 0; m < 8; m += 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i0 = 16 * h + m, i1 = i0 + 8;  // two adjacent keys of either group: the scaling is a packed multiply too
            const float2 x0 = __fmul2_rn(make_float2(__uint_as_float(s[i0]), __uint_as_float(s[i0 + 1])), make_float2(scale, scale));
            const float2 x1 = __fmul2_rn(make_float2(__uint_as_float(s[i1]), __uint_as_float(s[i1 + 1])), make_float2(scale, scale));
            float2 ea = make_float2(ex2_approx(fminf(x0.x, 15.f)), ex2_approx(fminf(x1.x, 15.f)));
            float2 eb = make_float2(ex2_approx(fminf(x0.y, 15.f)), ex2_approx(fminf(x1.y, 15.f)));
            if (kMasked) {
                if (col0 + i0 >= lim) ea.x = 0.f;
                if (col0 + i1 >= lim) ea.y = 0.f;
                if (col0 + i0 + 1 >= lim) eb.x = 0.f;
                if (col0 + i1 + 1 >= lim) eb.y = 0.f;
            }
            p[h][m] = __fmul2_rn(ea, run[h]);
            run[h] = __ffma2_rn(run[h], ea, run[h]);
            p[h][m + 1] = __fmul2_rn(eb, run[h]);
            run[h] = __ffma2_rn(run[h], eb, run[h]);
        }
    }
}
// carry entering each group from the right: f[h] = (W / (product of d over groups 2h..3), W / (product over groups 2h+1..3));
// W <- the chunk's exit carry
__device__ __forceinline__ void fwd_carries(const float2 (&run)[2], float& W, float2 (&f)[2]) {
    f[1].y = W * rcp_approx(run[1].y);
    f[1].x = f[1].y * rcp_approx(run[1].x);
    f[0].y = f[1].x * rcp_approx(run[0].y);
    f[0].x = f[0].y * rcp_approx(run[0].x);
    W = f[0].x;
}
template <bool kF16>
__device__ __forceinline__ void fwd_finish(const float2 (&p)[2][8], const float2 (&f)[2], float mul, uint32_t (&packed)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 fm = __fmul2_rn(f[h], make_float2(mul, mul));
#pragma unroll
        for (int m = 0; m < 8; m += 2) {
            const float2 a = __fmul2_rn(p[h][m], fm), b = __fmul2_rn(p[h][m + 1], fm);
            packed[8 * h + m / 2] = pack16<kF16>(a.x, b.x);
            packed[8 * h + 4 + m / 2] = pack16<kF16>(a.y, b.y);
        }
    }
}

}  // namespace fwd

}  // namespace sb
