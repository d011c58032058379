// Kernels of float32 precision on tcgen05, head dims up to 64: forward, backward-dq and backward-dk/dv.  (Larger head dims: sb_f32.cu, whose
// arithmetic this is: every value a sum of bf16 terms, every product the sum of the term products x_i y_j with i + j <= 2.)
//
// One block works on a 128-row tile (dk/dv: a 64-key tile) in steps of 128 queries x 64 keys.  Operands lie in shared memory as planes, one per
// term, of 64 columns with the 128-byte swizzle; whatever the head dim, type, strides or alignment, threads load rows themselves, split them and store
// the planes.  Weights and score gradients go back as three planes: to tensor memory (operand of O += P V and dQ += dS K) or, as
// queries are the contracted index there, to shared memory (dK, dV).
//   warps 0-7  a thread owns a query row and 32 keys of a step.  It reads its scores from tensor memory, so the scan along the keys is
//              serial in registers; the two threads of a row exchange one number per step (forward: the product of 1 - beta, dq: the sum of g;
//              dk/dv: nothing, the carries of both are saved at every 32-key boundary).  It also loads and splits the next tiles.
//   warp 8     issues the products.
// Sums: the tensor core rounds every accumulation towards zero, so a leading product is accumulated from zero over at most 64 indices, the smaller
// term products in accumulators of their own, and the row threads add both to registers in float32 (o, dq, dk, dv over steps likewise).
// A plane of B follows the plane before, so that one instruction takes a term of A through two or three of them (N = 128 or 192): an instruction with
// N = 64 costs what one with N = 128 does.  In dk/dv one product [P | dS]^T [dO | Q] forms both (half of its results are unused, but M = 128
// and N = 128 are full).
//
// Errors against float64 sums (norm of the difference / norm, 8 heads, 4096 float32 tokens; warp-level kernels before): o 8.3e-8 (9.2e-8), dq 1.4e-7
// (1.5e-7), dk 1.6e-7 (3.6e-7), dv 1.0e-7 (1.0e-7).
//
// us per kernel, forward / dq / dk,dv (the warp-level kernels of sb_f32.cu before); medians of 30 training calls in a row under the PyTorch profiler, where
// kernels do not overlap as they do in a stream (the first call takes 264 us without it):
//   8 heads, 4096 float32 tokens in 4 sequences, head dim 64:    56 /  75 / 134 (134 / 174 / 251)
//   4 x 8 heads x 500 tokens, bf16, head dim 50:                  24 /  27 /  35 (36 / 43 / 45)
//   4 heads, 512 float32 tokens, head dim 64:                     13 /  17 /  18 (19 / 23 / 25)
// What bounds them: the row threads.  A forward step takes 4 150 cycles (float32; clock readings around its parts): 1 650 the weights (25 instructions per
// score, issue-bound), 800 splitting the next K and V, 570 splitting the weights, 450 sums of accumulators, the rest barriers (~100 each).  dk/dv: 10 700 for
// twice the scores, 4 900 of them until its products are there: shared memory has no room for a second tile of Q and dO.  Counters (16 heads): tensor
// pipe 27 / 31 / 32 % active, issue slots 46 / 42 / 33 %.
// Sixteen row warps of 16 keys per thread were slower (56 / 90 / 168 us): 96 registers a thread, and with 28 KB left for the L1 every spilled
// value came back from the L2 at ~300 cycles.  Hence eight warps, and the registers that the last group of warps does without.
#include "sb_f32.cuh"
#include "sb_sm100.cuh"
#include "sb_tc_common.cuh"

namespace sb {

using namespace sm100;

namespace {

constexpr int kRowThreads = 256, kThreads = 384;  // warps 0-7: a row and 32 keys of a step per thread; warp 8 issues; 9-11 make up its group
constexpr int kQPlane = 128 * 128;  // a term of 128 rows of 64 columns: 128 bytes per row
constexpr int kKPlane = 64 * 128;   // a term of 64 rows

// The row threads take over registers of the last group: 384 x 168 at launch, 256 x 216 + 128 x 72 afterwards.
constexpr int kRowRegs = 216, kOtherRegs = 72;
static_assert(kRowThreads * kRowRegs + (kThreads - kRowThreads) * kOtherRegs <= kThreads * 168, "registers of the launch");
__device__ __forceinline__ void take_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRowRegs)); }
__device__ __forceinline__ void give_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs)); }
// whether any of the row threads says so
__device__ __forceinline__ bool any_row_thread(bool x) {
    int y;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 11, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(y) : "r"((int)x), "n"(kRowThreads) : "memory");
    return y != 0;
}
// the halves of a tile (bit 0: rows 0-63, bit 1: 64-127) in which a row thread says so
__device__ __forceinline__ int halves_where(bool x, int row) {
    return any_row_thread(x) ? (int)any_row_thread(x && row < 64) | (int)any_row_thread(x && row >= 64) << 1 : 0;
}

// ------------------------------------------------------------------------------------------ operand tiles
// loads without branches; zeros where ok is 0
__device__ __forceinline__ void load_if(uint32_t (&x)[4], const void* p, int ok) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                 "@q ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}" : "=&r"(x[0]), "=&r"(x[1]), "=&r"(x[2]), "=&r"(x[3]) : "l"(p), "r"(ok));
}
__device__ __forceinline__ void load_if(uint32_t (&x)[2], const void* p, int ok) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@q ld.global.v2.b32 {%0, %1}, [%2];\n\t}"
                 : "=&r"(x[0]), "=&r"(x[1]) : "l"(p), "r"(ok));
}
__device__ __forceinline__ void load_if(uint32_t (&x)[1], const void* p, int ok) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.b32 %0, [%1];\n\t}" : "=&r"(x[0]) : "l"(p), "r"(ok));
}
__device__ __forceinline__ void load_if(uint32_t& x, const float* p, int ok) { load_if((uint32_t(&)[1])x, (const void*)p, ok); }
template <typename T>
__device__ __forceinline__ void load_if(uint32_t& x, const T* p, int ok) {
    unsigned short v;
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b16 %0, 0;\n\t@q ld.global.b16 %0, [%1];\n\t}" : "=&h"(v) : "l"(p), "r"(ok));
    x = v;
}
// kRows rows of a [.., T, D] tensor on their way into planes of terms (128-byte swizzle, zeros behind the valid rows and columns).  fetch()
// issues the loads, put() splits and stores.  kU: 4 a load takes four elements, 2 two, 1 one.  kPlaneRows: rows
// of a plane, where these are a part of it.
template <typename T, int kU, int kRows, int kPlaneRows = kRows>
struct Tile {
    static constexpr int kN = Terms<T>::n, kE = kU == 4 ? 4 : 2, kPer = 64 / kE, kStep = kRowThreads / kPer, kPasses = kRows / kStep;
    static constexpr int kWords = sizeof(T) == 4 || kU == 1 ? kE : kE / 2;
    uint32_t x[kPasses][kWords];

    // this thread's first element of a tile, of which it takes rows kStep apart
    static __device__ __forceinline__ const T* first(const MatView& m, const ItemCtx& c, int h, int row) {
        return row_of<T>(m, c, h, row + (int)threadIdx.x / kPer) + kE * ((int)threadIdx.x % kPer);
    }
    // p: first(), st: elements between rows
    __device__ __forceinline__ void fetch(const T* p, int64_t st, int D, int rows_valid) {
        const int left = kE * ((int)threadIdx.x % kPer) < D ? rows_valid - (int)threadIdx.x / kPer : 0;
#pragma unroll
        for (int i = 0; i < kPasses; ++i, p += (int64_t)kStep * st) {
            const int ok = i * kStep < left;
            if constexpr (kU == 1) {
                load_if(x[i][0], p, ok);
                load_if(x[i][1], p + 1, ok && kE * ((int)threadIdx.x % kPer) + 1 < D);
            } else {
                load_if(x[i], p, ok);
            }
        }
    }
    __device__ __forceinline__ void put(uint8_t* dst) const {
        const int d = kE * ((int)threadIdx.x % kPer), r0 = (int)threadIdx.x / kPer;
        uint8_t* p = dst + r0 * 128 + (((d >> 3) ^ (r0 & 7)) << 4) + ((d * 2) & 15);
#pragma unroll
        for (int i = 0; i < kPasses; ++i, p += kStep * 128) {
            uint32_t w[kE / 2][kN];
#pragma unroll
            for (int u = 0; u < kE / 2; ++u) {
                if constexpr (sizeof(T) == 4) {
                    split_pair<kN>(__uint_as_float(x[i][2 * u]), __uint_as_float(x[i][2 * u + 1]), w[u]);
                } else {
                    const uint32_t v = kU == 1 ? x[i][0] | x[i][kWords - 1] << 16 : x[i][u];
                    if constexpr (kN == 1) {
                        w[u][0] = v;
                    } else {
                        const float2 f = __half22float2(*(const __half2*)&v);
                        split_pair<kN>(f.x, f.y, w[u]);
                    }
                }
            }
#pragma unroll
            for (int n = 0; n < kN; ++n) {
                if constexpr (kE == 4) *(uint2*)(p + n * kPlaneRows * 128) = make_uint2(w[0][n], w[1][n]);
                else *(uint32_t*)(p + n * kPlaneRows * 128) = w[0][n];
            }
        }
    }
};
// A 64-row tile on its way into planes through shared memory, where it waits as it is: a thread copies asynchronously into slots of its own and
// splits what it has copied itself.  (Waiting in registers, the tiles made the compiler spill registers that loads were still under way to.)
template <typename T, int kU>
struct Staged {
    static constexpr bool kPacked = sizeof(T) == 2 && kU == 1;  // no asynchronous copy of two bytes: loaded and stored
    using Regs = Tile<T, kPacked ? 2 : kU, 64>;
    static constexpr int kWords = Regs::kWords, kBytes = Regs::kPasses * kWords * 4 * kRowThreads;
    static __device__ __forceinline__ uint32_t* slot(uint8_t* stage, int i) { return (uint32_t*)stage + (i * kRowThreads + (int)threadIdx.x) * kWords; }
    static __device__ __forceinline__ void fetch(uint8_t* stage, const T* p, int64_t st, int D, int rows_valid) {
        const int d = Regs::kE * ((int)threadIdx.x % Regs::kPer), left = d < D ? rows_valid - (int)threadIdx.x / Regs::kPer : 0;
#pragma unroll
        for (int i = 0; i < Regs::kPasses; ++i, p += (int64_t)Regs::kStep * st) {
            const bool ok = i * Regs::kStep < left;
            const uint32_t dst = smem_u32(slot(stage, i));
            if constexpr (kPacked) {
                uint32_t x, y;
                load_if(x, p, ok);
                load_if(y, p + 1, ok && d + 1 < D);
                *slot(stage, i) = x | y << 16;
            } else if constexpr (kU == 1) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(p), "r"(ok ? 4 : 0) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4), "l"(p + 1), "r"(ok && d + 1 < D ? 4 : 0) : "memory");
            } else if constexpr (kWords == 4) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p), "r"(ok ? 16 : 0) : "memory");
            } else {
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(p), "n"(4 * kWords), "r"(ok ? 4 * kWords : 0) : "memory");
            }
        }
    }
    static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    // all but this thread's last kPending commits are in place
    template <int kPending>
    static __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory"); }
    static __device__ __forceinline__ void put(uint8_t* stage, uint8_t* dst) {
        Regs t;
#pragma unroll
        for (int i = 0; i < Regs::kPasses; ++i) {
            if constexpr (kWords == 4) {
                const uint4 v = *(const uint4*)slot(stage, i);
                t.x[i][0] = v.x; t.x[i][1] = v.y; t.x[i][2] = v.z; t.x[i][3] = v.w;
            } else if constexpr (kWords == 2) {
                const uint2 v = *(const uint2*)slot(stage, i);
                t.x[i][0] = v.x; t.x[i][1] = v.y;
            } else {
                t.x[i][0] = *slot(stage, i);
            }
        }
        t.put(dst);
    }
};

// ------------------------------------------------------------------------------------------ products
// Sum of the term products A_i B_j, i + j <= 2, into kBlocks accumulators of 64 columns: i + j = 0 (the leading one), 1, 2 (what
// lies beyond the last goes there).  The planes of B lie one after the other, so that one instruction takes A_i through several of
// them: N = 64 costs as much as N = 128.  kA: terms of A, kB: of B.  mma(columns, A's term, B's term, N, first in these columns).
template <int kA, int kB, int kBlocks, typename F>
__device__ __forceinline__ void term_products(F mma) {
#pragma unroll
    for (int i = 0; i < kA; ++i) {
        const int m = kB < 3 - i ? kB : 3 - i;
        const int wide = m < kBlocks - i ? m : kBlocks - i;
        if (wide > 0) mma(64 * i, i, 0, 64 * wide, i == 0 || kB == 1);
#pragma unroll
        for (int j = 0; j < m; ++j)
            if (j >= wide) mma(64 * (kBlocks - 1), i, j, 64, false);
    }
}
// 32 columns: the sum of kBlocks accumulators, small ones first, (kAdd) added to x; 16 columns at a time, which keeps registers
template <int kBlocks, bool kAdd = false>
__device__ __forceinline__ void load_sum(const uint32_t (&at)[kBlocks], float (&x)[32]) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t b[kBlocks][16];
#pragma unroll
        for (int i = 0; i < kBlocks; ++i) tmem_ld16(at[i] + 16 * half, b[i]);
#pragma unroll
        for (int i = 0; i < kBlocks; ++i) tmem_wait_ld(b[i]);
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            float2 v = make_float2(__uint_as_float(b[kBlocks - 1][c]), __uint_as_float(b[kBlocks - 1][c + 1]));
#pragma unroll
            for (int i = kBlocks - 2; i >= 0; --i) v = __fadd2_rn(v, make_float2(__uint_as_float(b[i][c]), __uint_as_float(b[i][c + 1])));
            if (kAdd) v = __fadd2_rn(make_float2(x[16 * half + c], x[16 * half + c + 1]), v);
            x[16 * half + c] = v.x;
            x[16 * half + c + 1] = v.y;
        }
    }
}
// of accumulators 64 columns apart
template <int kBlocks>
__device__ __forceinline__ void load_scores(uint32_t taddr, float (&x)[32]) {
    if constexpr (kBlocks == 1) load_sum<1>({taddr}, x);
    else if constexpr (kBlocks == 2) load_sum<2>({taddr, taddr + 64}, x);
    else load_sum<3>({taddr, taddr + 64, taddr + 128}, x);
}
// 32 values of a row as the terms of an operand in tensor memory: 16 columns of each plane, planes 32 columns apart
__device__ __forceinline__ void store_terms(uint32_t taddr, const float (&x)[32]) {
    uint32_t w[kWTerms][16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        uint32_t t[kWTerms];
        split_pair<kWTerms>(x[2 * i], x[2 * i + 1], t);
#pragma unroll
        for (int k = 0; k < kWTerms; ++k) w[k][i] = t[k];
    }
#pragma unroll
    for (int k = 0; k < kWTerms; ++k) tmem_st16(taddr + 32 * k, w[k]);
}

// ------------------------------------------------------------------------------------------ per-score arithmetic
// beta = sigmoid(x) and 1 - beta of two scores with full relative accuracy on both sides and no branches: 1 / (1 + e), whose divisor lies
// in [1, 2], is the hardware's approximate reciprocal after one step of Newton's method.
__device__ __forceinline__ void sigmoid2(float s0, float s1, float inv_temp, float2& beta, float2& om) {
    const float2 x = __fmul2_rn(make_float2(s0, s1), make_float2(inv_temp, inv_temp));
    const float2 e = make_float2(expf(-fabsf(x.x)), expf(-fabsf(x.y)));
    const float2 nd = __ffma2_rn(e, make_float2(-1.f, -1.f), make_float2(-1.f, -1.f));  // -(1 + e)
    float2 y = make_float2(rcp_approx(-nd.x), rcp_approx(-nd.y));
    y = __ffma2_rn(y, __ffma2_rn(nd, y, make_float2(1.f, 1.f)), y);
    const float2 z = __fmul2_rn(e, y);
    beta = make_float2(x.x >= 0.f ? y.x : z.x, x.y >= 0.f ? y.y : z.y);
    om = make_float2(x.x >= 0.f ? z.x : y.x, x.y >= 0.f ? z.y : y.y);
}
template <bool kMasked>
__device__ __forceinline__ void mask2(int i, int lim, float2& beta, float2& om) {
    if (!kMasked) return;
    if (i >= lim) { beta.x = 0.f; om.x = 1.f; }
    if (i + 1 >= lim) { beta.y = 0.f; om.y = 1.f; }
}
// forward, right to left, entered with 1: s <- weights; run <- product of 1 - beta.  Keys >= lim are not visible.
template <bool kMasked>
__device__ __forceinline__ void weights(float (&s)[32], float inv_temp, int lim, float& run) {
    run = 1.f;
#pragma unroll
    for (int i = 30; i >= 0; i -= 2) {
        float2 beta, om;
        sigmoid2(s[i], s[i + 1], inv_temp, beta, om);
        mask2<kMasked>(i, lim, beta, om);
        s[i + 1] = beta.y * run;
        run *= om.y;
        s[i] = beta.x * run;
        run *= om.x;
    }
}
// backward, right to left, entered with the product of 1 - beta to the right: b <- beta, s <- weights p (dk/dv), dp <- g = p (dp - drem),
// sum <- sum of g
template <bool kMasked>
__device__ __forceinline__ void score_grads(float (&s)[32], float (&dp)[32], float (&b)[32], float inv_temp, int lim, float drem, float run, float& sum) {
    sum = 0.f;
#pragma unroll
    for (int i = 30; i >= 0; i -= 2) {
        float2 beta, om;
        sigmoid2(s[i], s[i + 1], inv_temp, beta, om);
        mask2<kMasked>(i, lim, beta, om);
        const float2 d = __fadd2_rn(make_float2(dp[i], dp[i + 1]), make_float2(-drem, -drem));
        s[i + 1] = beta.y * run;
        run *= om.y;
        s[i] = beta.x * run;
        run *= om.x;
        const float2 g = __fmul2_rn(make_float2(s[i], s[i + 1]), d);
        b[i] = beta.x;
        b[i + 1] = beta.y;
        dp[i] = g.x;
        dp[i + 1] = g.y;
        sum += g.y;
        sum += g.x;
    }
}
// left to right: dp <- ds = g - beta (sum of g through the key), c: the sum left of the first.  (From the sum through the right edge and what lies
// right of a key the same takes one pass less, but dq is off by 3.0e-7 instead of 1.4e-7 of its norm, dk by 4.1e-7 instead of 2e-7.)
__device__ __forceinline__ void finish_ds(float (&dp)[32], const float (&beta)[32], float c) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const float g = dp[i];
        c += g;
        dp[i] = fmaf(-beta[i], c, g);
    }
}

// ------------------------------------------------------------------------------------------ results
// 32 columns of a row, n of them valid.  unit: of the tensor
template <typename T>
__device__ __forceinline__ void store32(const float (&x)[32], float scale, T* dst, int unit, int n) {
    if (n >= 32 && unit == 4) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            T v[4] = {from_f32<T>(x[i] * scale), from_f32<T>(x[i + 1] * scale), from_f32<T>(x[i + 2] * scale), from_f32<T>(x[i + 3] * scale)};
            if constexpr (sizeof(T) == 4) *(float4*)(dst + i) = make_float4(v[0], v[1], v[2], v[3]);
            else *(uint2*)(dst + i) = *(const uint2*)v;
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
        T v[2] = {from_f32<T>(x[i] * scale), from_f32<T>(x[i + 1] * scale)};
        if (unit > 1) {
            if (i < n) {
                if constexpr (sizeof(T) == 4) *(float2*)(dst + i) = make_float2(v[0], v[1]);
                else *(uint32_t*)(dst + i) = *(const uint32_t*)v;
            }
        } else {
            if (i < n) dst[i] = v[0];
            if (i + 1 < n) dst[i + 1] = v[1];
        }
    }
}
// x += f * y, each operation rounded by itself
template <typename T>
__device__ __forceinline__ void add32(float (&x)[32], float f, const T* y, int n) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i < n) x[i] = __fadd_rn(x[i], __fmul_rn(f, to_f32<T>(y[i])));
}
// whether these results ask for multiply-adds: a NaN, or a magnitude below 2^-100 other than zero.  (asks_for_direct wants all of a thread's to be small.  Here
// a thread has 32 neighbouring columns, and a tiny column among ordinary ones would lose its later terms.)
__device__ __forceinline__ bool row_asks_for_direct(const float (&x)[32], int n) {
    bool asks = false;
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (i < n) asks |= !(fabsf(x[i]) >= 0x1p-100f || x[i] == 0.f);
    return asks;
}
// this block's work item
__device__ __forceinline__ int block_item() { return (int)min(blockIdx.z * gridDim.y + blockIdx.y, 0x7fffffffu); }
// Sums by multiply-adds, by the eight row warps.  Forward and dq redo the 64-row halves of a tile that ask for it (bits of `halves`), one after the other;
// they look up again what they need instead of having the kernels keep it (registers).  One block has the SM, and was bound by the latency of its loads where it read
// the values in place, so they are copied to shared memory as float32 first.  8 heads, four sequences of 1024 tokens, one infinite value per head, forward /
// backward in us, in place, here and on the warp-level kernels: float32 head dim 64 863 / 2388, 342 / 741, 514 / 2163; bf16 50 977 / 2583, 343 / 697, 513 / 2150;
// float32 16 456 / 1010, 184 / 385, 235 / 672.  (Four loads of the values in place at a time: 772 / 2508 and 1242 / 2956 for the first two.)
template <typename T, int DP>
__device__ __forceinline__ void direct_fwd_halves(const KArgs& a, const ItemCtx& c, int halves, uint8_t* tiles, float (*xs)[kBM]) {
#pragma unroll 1
    for (int part = 0; part < 2; ++part)
        if (halves >> part & 1) {
            rows_sync<kStaged>();  // the half before has read its tiles
            fwd_block<T, DP, kStaged>(a, c, BlockIdx{0, (int)blockIdx.x, part}, (__nv_bfloat16*)tiles, xs);
        }
}
template <typename T>
__device__ __noinline__ void direct_fwd(const KArgs& a, const OwnTables& own, int halves, uint8_t* tiles, float (*xs)[kBM]) {
    const ItemCtx c = a.own_tables ? item_ctx(own.items, own.seqs, block_item()) : item_ctx(a, block_item());
    if (a.head_dim > 32) direct_fwd_halves<T, 64>(a, c, halves, tiles, xs);
    else if (a.head_dim > 16) direct_fwd_halves<T, 32>(a, c, halves, tiles, xs);
    else direct_fwd_halves<T, 16>(a, c, halves, tiles, xs);
}
template <typename T, int DP>
__device__ __forceinline__ void direct_dq_halves(const KArgs& a, const ItemCtx& c, int halves, uint8_t* tiles, float (*xs)[kBM]) {
#pragma unroll 1
    for (int part = 0; part < 2; ++part)
        if (halves >> part & 1) {
            rows_sync<kStaged>();  // the half before has read its tiles
            dq_block<T, DP, kStaged>(a, c, BlockIdx{0, (int)blockIdx.x, part}, (__nv_bfloat16*)tiles, xs);
        }
}
template <typename T>
__device__ __noinline__ void direct_dq(const KArgs& a, int halves, uint8_t* tiles, float (*xs)[kBM]) {
    const ItemCtx c = item_ctx(a, block_item());
    if (a.head_dim > 32) direct_dq_halves<T, 64>(a, c, halves, tiles, xs);
    else if (a.head_dim > 16) direct_dq_halves<T, 32>(a, c, halves, tiles, xs);
    else direct_dq_halves<T, 16>(a, c, halves, tiles, xs);
}
// dk and dv of a 64-key tile, 32 queries per step
constexpr int kDirectQ = 32, kDirectP = kDirectQ + 8;
template <int DP> constexpr int kDirectKv = 3 * kValues<DP> + 2 * 64 * kDirectP;  // floats
template <typename T, int DP>
__device__ __forceinline__ void direct_dkdv_tile(const KArgs& a, const ItemCtx& c, const BlockIdx& bi, float* tiles) {
    constexpr int kQ = kDirectQ, kPP = kDirectP;
    float *const vK = tiles, *const vV = vK + kValues<DP>, *const vQ = vV + kValues<DP>, *const vG = vQ + kValues<DP> / 2;
    float *const fP = vG + kValues<DP> / 2, *const fS = fP + 64 * kPP;  // weights and score gradients, [64 keys][kQ queries]
    const int h = bi.h, D = a.head_dim, key0 = c.qt * kTileQ + bi.part * kBN, keys_valid = min(kBN, c.len - key0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int kq = warp & 1, q0 = 8 * (warp >> 1);  // first half of a step: 32 keys and 8 queries
    const int kg = warp & 3;                        // second half: 16 keys of dk or dv
    const bool is_dk = warp >> 2;
    const float* cw = a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ;
    const float* cc = a.carry_c + ((int64_t)h * a.slot_cap) * kTileQ;
    float acc[DP / 8][4] = {};
    stage_values<T, DP, kBN>(vK, row_of<T>(a.k, c, h, key0), a.k.st, D, keys_valid);
    stage_values<T, DP, kBN>(vV, row_of<T>(a.v, c, h, key0), a.v.st, D, keys_valid);
    for (int row0 = key0; row0 < c.len; row0 += kQ) {
        const int rows_valid = min(kQ, c.len - row0);
        const int64_t slot = carry_slot32(c.slot_base, row0 / kTileQ, key0 / 32 + kq) * kTileQ + row0 % kTileQ;
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
        rows_sync<kStaged>();
        stage_values<T, DP, kQ>(vQ, row_of<T>(a.q, c, h, row0), a.q.st, D, rows_valid);
        stage_values<T, DP, kQ>(vG, row_of<T>(a.d_o, c, h, row0), a.d_o.st, D, rows_valid);
        rows_sync<kStaged>();
        {
            float s[2][1][4], dp[2][1][4];
            const int key = 32 * kq + 4 * g, qq = q0 + 2 * t;
            values_scores_t<DP>(s, vK + value_row<DP>(key), vQ + value_row<DP>(qq), D);
            values_scores_t<DP>(dp, vV + value_row<DP>(key), vG + value_row<DP>(qq), D);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float* const ps[4] = {&s[0][0][e], &s[0][0][2 + e], &s[1][0][e], &s[1][0][2 + e]};
                float* const pd[4] = {&dp[0][0][e], &dp[0][0][2 + e], &dp[1][0][e], &dp[1][0][2 + e]};
                const int q = qq + e;
                const int lim = q < rows_valid ? min(keys_valid, row0 + q + a.attend_current - key0) : 0;
                column(ps, pd, a.inv_temp, true, lim - key, W[e], cr[e], drem[e], g);
            }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    const int at = (32 * kq + 16 * m + 8 * hh + g) * kPP + q0 + 2 * t;
                    *(float2*)(fP + at) = make_float2(s[m][0][2 * hh], s[m][0][2 * hh + 1]);
                    *(float2*)(fS + at) = make_float2(dp[m][0][2 * hh], dp[m][0][2 * hh + 1]);
                }
        }
        rows_sync<kStaged>();
        const float* x = (is_dk ? vQ : vG) + 2 * t;
        const float* pa = (is_dk ? fS : fP) + (16 * kg + g) * kPP;
#pragma unroll 2
        for (int q = 0; q < rows_valid; ++q) {
            const float p0 = pa[q], p1 = pa[8 * kPP + q];
#pragma unroll
            for (int n = 0; n < DP / 8; ++n) {
                const float2 v = *(const float2*)(x + value_row<DP>(q) + 8 * n);
                acc[n][0] = fmaf(p0, v.x, acc[n][0]);
                acc[n][1] = fmaf(p0, v.y, acc[n][1]);
                acc[n][2] = fmaf(p1, v.x, acc[n][2]);
                acc[n][3] = fmaf(p1, v.y, acc[n][3]);
            }
        }
    }
    const MatView m = is_dk ? a.dk : a.dv;
    const bool pairs = units_ok<T>(m, D, 2);
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int row = 32 * (kg >> 1) + 4 * g + 2 * (kg & 1) + hh;
        if (row >= keys_valid) continue;
        if (a.fused && !is_dk)  // dv += rem * do
            add_row<T, DP>(acc, 2 * hh, to_f32<T>(((const T*)a.rem.ptr)[(int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + (int64_t)(c.start + key0 + row) * a.rem.st]),
                           row_of<T>(a.d_o, c, h, key0 + row), D, 0, t);
        store_row<T, DP>(acc, 2 * hh, is_dk ? a.inv_temp : 1.f, m, pairs, D, 0, (T*)row_of<T>(m, c, h, key0), row, t);
    }
}

template <typename T>
__device__ __noinline__ void direct_dkdv(const KArgs& a, uint8_t* tiles) {
    const ItemCtx c = item_ctx(a, a.hdr->n_items - 1 - block_item());
    const BlockIdx bi{0, (int)(blockIdx.x >> 1), (int)(blockIdx.x & 1)};
    if (a.head_dim > 32) direct_dkdv_tile<T, 64>(a, c, bi, (float*)tiles);
    else if (a.head_dim > 16) direct_dkdv_tile<T, 32>(a, c, bi, (float*)tiles);
    else direct_dkdv_tile<T, 16>(a, c, bi, (float*)tiles);
}

// bytes of a kernel's tiles, which share their place with the float32 values of the direct forms
constexpr int tiles_size(int bytes, int values) { return bytes > 4 * values ? bytes : 4 * values; }
// start and end common to the kernels
struct Shared {
    uint32_t tmem, abort;
};
__device__ __forceinline__ void block_start(uint8_t* smem, Shared& sh, int warp) {
    if (threadIdx.x == 0) {
        sh.abort = (smem_u32(smem) & 1023u) ? 1u : 0u;  // the swizzled planes need a 1024-byte aligned base
        fence_barrier_init();
    }
    if (warp == 8) {
        tmem_alloc(&sh.tmem, 512);
        tmem_relinquish();
    }
}

// ------------------------------------------------------------------------------------------ forward
enum FwdBar { F_S_READY, F_S_FREE, F_P_READY, F_O_READY, F_X, kFwdBars = F_X + 8 };  // F_X: exchange along rows, [32 rows][step parity]
struct FwdShared : Shared {
    uint64_t bars[kFwdBars];
    float xs[2][2][128];  // [step parity][half][row]: product of 1 - beta over 32 keys
    OwnTables own;
};
template <typename T, int kU>
constexpr int kFwdTiles = tiles_size(Terms<T>::n * (kQPlane + 2 * kKPlane) + 2 * Staged<T, kU>::kBytes, 3 * kValues<64>);
template <typename T, int kU>
constexpr int fwd_smem() { return kFwdTiles<T, kU> + (int)sizeof(FwdShared) + 1024; }

template <typename T, int kU>
__global__ void __launch_bounds__(kThreads, 1) f32tc_fwd_kernel(const __grid_constant__ KArgs a) {
    constexpr int kN = Terms<T>::n, kSB = kN > 1 ? 2 : 1, kOB = 2;
    constexpr uint32_t kColS = 0, kColP = 128, kColO = 224;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + kN * kQPlane;
    uint8_t* sV = sK + kN * kKPlane;
    uint8_t* stage_k = sV + kN * kKPlane;
    uint8_t* stage_v = stage_k + Staged<T, kU>::kBytes;
    FwdShared& sh = *(FwdShared*)(smem + kFwdTiles<T, kU>);
    uint64_t* bars = sh.bars;
    volatile uint32_t* abort_flag = &sh.abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0)
        for (int i = 0; i < kFwdBars; ++i) mbar_init(&bars[i], i == F_S_FREE || i == F_P_READY ? kRowThreads : i >= F_X ? 64 : 1);
    block_start(smem, sh, warp);
    pdl_wait();
    if (a.own_tables && warp == 0) build_own_tables(a, &sh.own, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    const int covered_end = a.own_tables ? sh.own.covered_end : a.hdr->covered_end;
    if (a.zero_tail && covered_end < a.tokens) zero_tail_rows<T>(a, covered_end, linear_thread(), all_threads());
    const int item = block_item(), h = blockIdx.x, D = a.head_dim;
    const bool mine = item < (a.own_tables ? sh.own.n_items : a.hdr->n_items) && !*abort_flag;
    const ItemCtx c = !mine ? ItemCtx{} : a.own_tables ? item_ctx(sh.own.items, sh.own.seqs, item) : item_ctx(a, item);
    const int row0 = c.qt * kTileQ, rows_valid = min(kTileQ, c.len - row0);
    const int n = mine ? min(2 * c.qt + 1, (c.len - 1) / 64) + 1 : 0;  // 64-key steps, right to left
    const int r = (warp & 3) * 32 + lane, q = (warp >> 2) & 1;  // row threads: a row and a half (32 keys, 0 the left one) of a step
    if (mine) {
        float o[32], W = 1.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) o[i] = 0.f;
        using KTile = Staged<T, kU>;
        const T *pk = KTile::Regs::first(a.k, c, h, 64 * (n - 1)), *pv = KTile::Regs::first(a.v, c, h, 64 * (n - 1));  // next tile to load
        const int64_t back_k = 64 * a.k.st, back_v = 64 * a.v.st;
        if (warp < 8) {
            KTile::fetch(stage_k, pk, a.k.st, D, c.len - 64 * (n - 1));
            KTile::commit();
            Tile<T, kU, 128> tq;
            tq.fetch(tq.first(a.q, c, h, row0), a.q.st, D, rows_valid);
            tq.put(sQ);
            KTile::template wait<0>();
            KTile::put(stage_k, sK);
            pk -= back_k;
            if (n > 1) KTile::fetch(stage_k, pk, a.k.st, D, 64);
            KTile::commit();
            KTile::fetch(stage_v, pv, a.v.st, D, c.len - 64 * (n - 1));
            KTile::commit();
            fence_async_smem();
        }
        __syncthreads();
        if (warp >= 8) {
            give_registers();
            if (warp == 8) {
                // ---------------------------------------------------------------- issuing warp
                const bool leader = elect_one();
                const SmemDesc dq = make_desc(smem_u32(sQ), 0, 1024), dk = make_desc(smem_u32(sK), 0, 1024), dv = make_desc(smem_u32(sV), kKPlane, 1024);
                const auto issue_s = [&]() {
                    term_products<kN, kN, kSB>([&](int col, int i, int jb, int cols, bool first) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 0);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (16 * k < D) mma_ss_dyn(leader, tmem + kColS + col, dq, i * kQPlane + 32 * k, dk, jb * kKPlane + 32 * k, idesc, !(first && k == 0));
                    });
                    mma_commit(leader, &bars[F_S_READY]);
                };
                issue_s();
                for (int j = 0; j < n; ++j) {
                    if (j + 1 < n) {
                        if (!mbar_wait(&bars[F_S_FREE], j & 1, abort_flag)) break;
                        tc_fence_after();
                        issue_s();
                    }
                    if (!mbar_wait(&bars[F_P_READY], j & 1, abort_flag)) break;
                    tc_fence_after();
                    term_products<kWTerms, kN, kOB>([&](int col, int i, int jb, int cols, bool first) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 1);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            mma_ts_dyn(leader, tmem + kColO + col, tmem + kColP + 32 * i + 8 * k, dv, jb * kKPlane + 2048 * k, idesc, !(first && k == 0));
                    });
                    mma_commit(leader, &bars[F_O_READY]);
                }
            }
        } else {
            // ---------------------------------------------------------------- row threads
            take_registers();
            const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16), base = lane_base + 32 * q;
            // the carry at the right edge of this thread's keys
            float* cw = a.carry_w ? a.carry_w + ((int64_t)h * a.slot_cap + carry_slot32(c.slot_base, c.qt, 2 * (n - 1) + q)) * kTileQ + r : nullptr;
            bool ok = true;
            for (int j = 0; j < n; ++j) {
                ok = mbar_wait(&bars[F_S_READY], j & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                float s[32], run;
                load_scores<kSB>(base + kColS, s);
                tc_fence_before();
                if (j + 1 < n) {  // the next keys
                    KTile::template wait<1>();
                    KTile::put(stage_k, sK);
                    fence_async_smem();
                }
                mbar_arrive(&bars[F_S_FREE]);
                pk -= back_k;
                if (j + 2 < n) KTile::fetch(stage_k, pk, a.k.st, D, 64);
                KTile::commit();
                const int kh = n - 1 - j;
                if (kh >= 2 * c.qt) weights<true>(s, a.inv_temp, min(c.len, row0 + r + a.attend_current) - 64 * kh - 32 * q, run);
                else weights<false>(s, a.inv_temp, 32, run);
                float(*xs)[128] = sh.xs[j & 1];
                xs[q][r] = run;
                uint64_t* bx = &bars[F_X + 2 * (warp & 3) + (j & 1)];
                mbar_arrive(bx);
                if (j > 0) {  // the product before has read its weights and its V
                    ok = mbar_wait(&bars[F_O_READY], (j - 1) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    load_sum<2, true>({base + kColO, base + kColO + 64}, o);
                }
                KTile::template wait<1>();
                KTile::put(stage_v, sV);
                pv -= back_v;
                if (j + 1 < n) KTile::fetch(stage_v, pv, a.v.st, D, 64);
                KTile::commit();
                fence_async_smem();
                ok = mbar_wait(bx, (j >> 1) & 1, abort_flag);
                if (!ok) break;
                const float right = W * xs[1][r], win = q ? W : right;
                W = right * xs[0][r];
                if (cw) {
                    *cw = win;
                    cw -= 2 * kTileQ;
                }
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float2 v = __fmul2_rn(make_float2(s[i], s[i + 1]), make_float2(win, win));
                    s[i] = v.x;
                    s[i + 1] = v.y;
                }
                store_terms(lane_base + kColP + 16 * q, s);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars[F_P_READY]);
            }
            if (ok && mbar_wait(&bars[F_O_READY], (n - 1) & 1, abort_flag)) {
                tc_fence_after();
                load_sum<2, true>({base + kColO, base + kColO + 64}, o);
            }
            const int cols = D - 32 * q;  // of this thread's 32, that exist
            const bool in_rows = r < rows_valid;
            const int again = halves_where(in_rows && (row_asks_for_direct(o, cols) || W != W), r);
            pdl_launch_dependents();
            if (!*abort_flag && in_rows && !(again >> (r >> 6) & 1)) {
                // out = o + rem * v: the same bits as the expression outside for float32
                if (a.fused) add32<T>(o, to_f32<T>(from_f32<T>(W)), row_of<T>(a.v, c, h, row0 + r) + 32 * q, cols);
                if (cols > 0) store32<T>(o, 1.f, (T*)row_of<T>(a.o, c, h, row0 + r) + 32 * q, unit<T>(a.o, D), cols);
                if (q == 0) {
                    const int64_t tok = c.start + row0 + r;
                    ((T*)a.rem.ptr)[(int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + tok * a.rem.st] = from_f32<T>(W);
                    ((float*)a.nla.ptr)[(int64_t)c.b * a.nla.sb + (int64_t)h * a.nla.sh + tok * a.nla.st] = log2f(W);
                }
            }
            if (again && !*abort_flag) direct_fwd<T>(a, sh.own, again, smem, (float(*)[kBM])sh.xs);
        }
    }
    tc_teardown(abort_flag, a.status, tmem, 512, 8);
}

// ------------------------------------------------------------------------------------------ backward: dq
enum DqBar { A_READY, A_FREE, A_KEYS, A_DS, A_DQ, A_X, kDqBars = A_X + 8 };
struct DqShared : Shared {
    uint64_t bars[kDqBars];
    float xg[2][2][128];  // [step parity][half][row]: sum of g over 32 keys
};
template <typename T, int kU>
constexpr int kDqTiles = tiles_size(Terms<T>::n * (2 * kQPlane + 3 * kKPlane) + 2 * Staged<T, kU>::kBytes, 4 * kValues<64>);
template <typename T, int kU>
constexpr int dq_smem() { return kDqTiles<T, kU> + (int)sizeof(DqShared) + 1024; }

template <typename T, int kU>
__global__ void __launch_bounds__(kThreads, 1) f32tc_bwd_dq_kernel(const __grid_constant__ KArgs a) {
    constexpr int kN = Terms<T>::n, kSB = kN > 1 ? 2 : 1;
    constexpr uint32_t kColS = 0, kColDP = 128, kColDS = 256, kColDQ = 352;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sG = sQ + kN * kQPlane;      // dO
    uint8_t* sK = sG + kN * kQPlane;      // two tiles: step j's is read by the last product of that step
    uint8_t* sV = sK + 2 * kN * kKPlane;
    uint8_t* stage_k = sV + kN * kKPlane;
    uint8_t* stage_v = stage_k + Staged<T, kU>::kBytes;
    DqShared& sh = *(DqShared*)(smem + kDqTiles<T, kU>);
    uint64_t* bars = sh.bars;
    volatile uint32_t* abort_flag = &sh.abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0)
        for (int i = 0; i < kDqBars; ++i) mbar_init(&bars[i], i == A_FREE || i == A_KEYS || i == A_DS ? kRowThreads : i >= A_X ? 64 : 1);
    block_start(smem, sh, warp);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    pdl_wait();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) zero_tail_grads<T>(a, a.hdr->covered_end, linear_thread(), all_threads());
    const int item = block_item(), h = blockIdx.x, D = a.head_dim;
    const bool mine = item < a.hdr->n_items && !*abort_flag;
    const ItemCtx c = !mine ? ItemCtx{} : item_ctx(a, item);
    const int row0 = c.qt * kTileQ, rows_valid = min(kTileQ, c.len - row0);
    const int n = mine ? min(2 * c.qt + 1, (c.len - 1) / 64) + 1 : 0;  // 64-key steps, left to right
    const int r = (warp & 3) * 32 + lane, q = (warp >> 2) & 1;
    if (mine) {
        float acc[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
        const auto valid = [&](int j) { return c.len - 64 * j; };
        using KTile = Staged<T, kU>;
        const T *pk = KTile::Regs::first(a.k, c, h, 0), *pv = KTile::Regs::first(a.v, c, h, 0);  // next tile to load
        const int64_t step_k = 64 * a.k.st, step_v = 64 * a.v.st;
        if (warp < 8) {
            KTile::fetch(stage_k, pk, a.k.st, D, valid(0));
            KTile::fetch(stage_v, pv, a.v.st, D, valid(0));
            KTile::commit();
            Tile<T, kU, 128> tq;
            tq.fetch(tq.first(a.q, c, h, row0), a.q.st, D, rows_valid);
            tq.put(sQ);
            tq.fetch(tq.first(a.d_o, c, h, row0), a.d_o.st, D, rows_valid);
            KTile::template wait<0>();
            KTile::put(stage_k, sK);
            KTile::put(stage_v, sV);
            pk += step_k;
            pv += step_v;
            if (n > 1) KTile::fetch(stage_v, pv, a.v.st, D, valid(1));
            KTile::commit();
            if (n > 1) KTile::fetch(stage_k, pk, a.k.st, D, valid(1));
            KTile::commit();
            tq.put(sG);
            fence_async_smem();
        }
        __syncthreads();
        if (warp >= 8) {
            give_registers();
            if (warp == 8) {
                const bool leader = elect_one();
                const SmemDesc dq = make_desc(smem_u32(sQ), 0, 1024), dg = make_desc(smem_u32(sG), 0, 1024), dk = make_desc(smem_u32(sK), 0, 1024),
                               dv = make_desc(smem_u32(sV), 0, 1024), dkm = make_desc(smem_u32(sK), kKPlane, 1024);
                const auto issue_dp = [&]() {
                    term_products<kN, kN, kSB>([&](int col, int i, int jb, int cols, bool first) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 0);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (16 * k < D) mma_ss_dyn(leader, tmem + kColDP + col, dg, i * kQPlane + 32 * k, dv, jb * kKPlane + 32 * k, idesc, !(first && k == 0));
                    });
                };
                const auto issue_s = [&](int j) {
                    const uint32_t ko = (j & 1) * kN * kKPlane;
                    term_products<kN, kN, kSB>([&](int col, int i, int jb, int cols, bool first) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 0);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (16 * k < D) mma_ss_dyn(leader, tmem + kColS + col, dq, i * kQPlane + 32 * k, dk, ko + jb * kKPlane + 32 * k, idesc, !(first && k == 0));
                    });
                    mma_commit(leader, &bars[A_READY]);  // of both
                };
                issue_dp();
                issue_s(0);
                for (int j = 0; j < n; ++j) {
                    if (j + 1 < n) {
                        if (!mbar_wait(&bars[A_FREE], j & 1, abort_flag)) break;
                        tc_fence_after();
                        issue_dp();
                        if (!mbar_wait(&bars[A_KEYS], j & 1, abort_flag)) break;
                        tc_fence_after();
                        issue_s(j + 1);
                    }
                    if (!mbar_wait(&bars[A_DS], j & 1, abort_flag)) break;
                    tc_fence_after();
                    const uint32_t ko = (j & 1) * kN * kKPlane;
                    term_products<kWTerms, kN, 2>([&](int col, int i, int jb, int cols, bool first) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 1);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            mma_ts_dyn(leader, tmem + kColDQ + col, tmem + kColDS + 32 * i + 8 * k, dkm, ko + jb * kKPlane + 2048 * k, idesc, !(first && k == 0));
                    });
                    mma_commit(leader, &bars[A_DQ]);
                }
            }
        } else {
            take_registers();
            const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16), base = lane_base + 32 * q;
            const int64_t slot = ((int64_t)h * a.slot_cap + carry_slot32(c.slot_base, c.qt, q)) * kTileQ + r;
            const float* cw = a.carry_w + slot;
            float* cc = a.carry_c + slot;
            const bool row_ok = r < rows_valid;
            const float drem = row_ok ? to_f32<T>(((const T*)a.d_rem.ptr)[(int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + (int64_t)(c.start + row0 + r) * a.d_rem.st]) : 0.f;
            float prefix = 0.f;  // sum of g over all keys left of the step
            bool ok = true;
            float W = row_ok ? *cw : 0.f;  // of the step to come
            for (int j = 0; j < n; ++j) {
                ok = mbar_wait(&bars[A_READY], j & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                float s[32], dp[32], b[32], mine_g;
                load_scores<kSB>(base + kColS, s);
                load_scores<kSB>(base + kColDP, dp);
                tc_fence_before();
                if (j + 1 < n) {  // the next V
                    KTile::template wait<1>();
                    KTile::put(stage_v, sV);
                    fence_async_smem();
                }
                mbar_arrive(&bars[A_FREE]);
                pv += step_v;
                if (j + 2 < n) KTile::fetch(stage_v, pv, a.v.st, D, valid(j + 2));
                KTile::commit();
                if (j >= 2 * c.qt) score_grads<true>(s, dp, b, a.inv_temp, min(c.len, row0 + r + a.attend_current) - 64 * j - 32 * q, drem, W, mine_g);
                else score_grads<false>(s, dp, b, a.inv_temp, 32, drem, W, mine_g);
                float(*xg)[128] = sh.xg[j & 1];
                xg[q][r] = mine_g;
                uint64_t* bx = &bars[A_X + 2 * (warp & 3) + (j & 1)];
                mbar_arrive(bx);
                cw += 2 * kTileQ;
                if (j + 1 < n) W = row_ok ? *cw : 0.f;
                if (j > 0) {  // the product before has read its ds and its keys
                    ok = mbar_wait(&bars[A_DQ], (j - 1) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    load_sum<2, true>({base + kColDQ, base + kColDQ + 64}, acc);
                }
                if (j + 1 < n) {  // the next keys
                    KTile::template wait<1>();
                    KTile::put(stage_k, sK + ((j + 1) & 1) * kN * kKPlane);
                    fence_async_smem();
                }
                mbar_arrive(&bars[A_KEYS]);
                pk += step_k;
                if (j + 2 < n) KTile::fetch(stage_k, pk, a.k.st, D, valid(j + 2));
                KTile::commit();
                ok = mbar_wait(bx, (j >> 1) & 1, abort_flag);
                if (!ok) break;
                const float left = q ? prefix + xg[0][r] : prefix;
                prefix = prefix + xg[0][r] + xg[1][r];
                if (row_ok) *cc = left + mine_g;  // sum of g through this half's right edge
                cc += 2 * kTileQ;
                finish_ds(dp, b, left);
                store_terms(lane_base + kColDS + 16 * q, dp);
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars[A_DS]);
            }
            if (ok && mbar_wait(&bars[A_DQ], (n - 1) & 1, abort_flag)) {
                tc_fence_after();
                load_sum<2, true>({base + kColDQ, base + kColDQ + 64}, acc);
            }
            const int cols = D - 32 * q;
            const bool in_rows = r < rows_valid;
            const int again = halves_where(in_rows && row_asks_for_direct(acc, cols), r);
            pdl_launch_dependents();
            if (!*abort_flag && in_rows && cols > 0 && !(again >> (r >> 6) & 1))
                store32<T>(acc, a.inv_temp, (T*)row_of<T>(a.dq, c, h, row0 + r) + 32 * q, unit<T>(a.dq, D), cols);
            if (again && !*abort_flag) direct_dq<T>(a, again, smem, (float(*)[kBM])sh.xg);
        }
    }
    tc_teardown(abort_flag, a.status, tmem, 512, 8);
}

// ------------------------------------------------------------------------------------------ backward: dk, dv
enum KvBar { B_LOADED, B_READY, B_FREE, B_W0, B_RING = B_W0 + 4, B_A0, B_A1, kKvBars };  // B_W0 ...: of the four chunks of 32 queries
struct KvShared : Shared {
    uint64_t bars[kKvBars];
};
constexpr int kChunk = kWTerms * 2 * 32 * 128;  // 32 queries: terms of [weights | ds], 64 keys each
template <typename T>
constexpr int kKvTiles = tiles_size(Terms<T>::n * (2 * kQPlane + 2 * kKPlane) + 3 * kChunk, kDirectKv<64>);
template <typename T>
constexpr int kv_smem() { return kKvTiles<T> + (int)sizeof(KvShared) + 1024; }

template <typename T, int kU>
__global__ void __launch_bounds__(kThreads, 1) f32tc_bwd_dkdv_kernel(const __grid_constant__ KArgs a) {
    constexpr int kN = Terms<T>::n;
    constexpr uint32_t kColS = 0, kColDP = 192, kColA[2] = {384, 0}, kColSmall[2] = {128, 256};  // accumulators lie over the scores
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;
    uint8_t* sV = sK + kN * kKPlane;
    uint8_t* sG = sV + kN * kKPlane;  // dO
    uint8_t* sQ = sG + kN * kQPlane;
    uint8_t* sW = sQ + kN * kQPlane;  // three chunks
    KvShared& sh = *(KvShared*)(smem + kKvTiles<T>);
    uint64_t* bars = sh.bars;
    volatile uint32_t* abort_flag = &sh.abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0)
        for (int i = 0; i < kKvBars; ++i) mbar_init(&bars[i], i == B_LOADED || i == B_FREE ? kRowThreads : i >= B_W0 && i < B_RING ? 64 : 1);
    block_start(smem, sh, warp);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem;
    pdl_wait();
    const int item = block_item(), h = blockIdx.x >> 1, part = blockIdx.x & 1, D = a.head_dim;
    const int n_items = a.hdr->n_items;
    bool mine = item < n_items && !*abort_flag;
    // the table is heaviest-first for query tiles; key tiles are heaviest at the other end
    const ItemCtx c = !mine ? ItemCtx{} : item_ctx(a, n_items - 1 - item);
    const int key0 = c.qt * kTileQ + part * 64, keys_valid = min(64, c.len - key0);
    mine = mine && key0 < c.len;
    const int first = c.qt * kTileQ;  // query rows of step j: first + 128 j ...
    const int n = mine ? (c.len - first + 127) / 128 : 0;
    const int r = (warp & 3) * 32 + lane, q = (warp >> 2) & 1;
    if (mine) {
        float acc[32];  // rows 0-63: dv of key r, 64-127: dk of key r - 64; 32 columns
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = 0.f;
        const auto valid = [&](int j) { return min(128, c.len - first - 128 * j); };
        // Chunks of 32 queries of step j that see a key and exist: [lo, hi), never empty.  Chunks 0, 1 and 2, 3 have accumulators of their own.
        const auto lo = [&](int j) { return j == 0 ? 2 * part : 0; };
        const auto hi = [&](int j) { return (valid(j) + 31) >> 5; };
        if (warp >= 8) {
            give_registers();
            if (warp == 8) {
                const bool leader = elect_one();
                const SmemDesc dq = make_desc(smem_u32(sQ), 0, 1024), dg = make_desc(smem_u32(sG), 0, 1024), dk = make_desc(smem_u32(sK), 0, 1024),
                               dv = make_desc(smem_u32(sV), 0, 1024), dw = make_desc(smem_u32(sW), 32 * 128, 1024), dgq = make_desc(smem_u32(sG), kN * kQPlane, 1024);
                uint32_t uses = 0;  // bit i: parity of the next use of chunk i's barrier
                bool ok = true;
                for (int j = 0; ok && j < n; ++j) {
                    ok = mbar_wait(&bars[B_LOADED], j & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    term_products<kN, kN, kN>([&](int col, int i, int jb, int cols, bool fresh) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 0);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (16 * k < D) mma_ss_dyn(leader, tmem + kColS + col, dq, i * kQPlane + 32 * k, dk, jb * kKPlane + 32 * k, idesc, !(fresh && k == 0));
                    });
                    term_products<kN, kN, kN>([&](int col, int i, int jb, int cols, bool fresh) {
                        const uint32_t idesc = make_idesc(128, cols, 1, 0, 0);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (16 * k < D) mma_ss_dyn(leader, tmem + kColDP + col, dg, i * kQPlane + 32 * k, dv, jb * kKPlane + 32 * k, idesc, !(fresh && k == 0));
                    });
                    mma_commit(leader, &bars[B_READY]);
                    ok = mbar_wait(&bars[B_FREE], j & 1, abort_flag);  // scores are in registers
                    if (!ok) break;
                    const int c0 = lo(j), c1 = hi(j);
                    for (int ch = c0; ch < c1; ++ch) {
                        ok = mbar_wait(&bars[B_W0 + ch], (uses >> ch) & 1, abort_flag);
                        if (!ok) break;
                        uses ^= 1u << ch;
                        tc_fence_after();
                        // [weights | ds]^T [dO | Q]: the blocks on the diagonal are dv and dk
                        constexpr uint32_t idesc = make_idesc(128, 128, 1, 1, 1);
                        const uint32_t lead = tmem + (ch < 2 ? kColA[0] : kColA[1]), small = tmem + (ch < 2 ? kColSmall[0] : kColSmall[1]);
                        const uint32_t wo = (ch == 3 ? 0 : ch) * kChunk;
                        const bool add = (ch & 1) && ch > c0;  // to what the chunk before has left there
#pragma unroll
                        for (int order = 2; order >= 0; --order)
#pragma unroll
                            for (int i = 0; i < kWTerms; ++i) {
                                const int jb = order - i;
                                if (jb < 0 || jb >= kN) continue;
                                const bool fresh = order == 0 || (order == 2 && i == (kN == 1 ? 2 : kN == 2 ? 1 : 0));
#pragma unroll
                                for (int k = 0; k < 2; ++k)
                                    mma_ss_dyn(leader, order ? small : lead, dw, wo + i * 2 * 32 * 128 + 2048 * k, dgq, jb * kQPlane + ch * 32 * 128 + 2048 * k, idesc, add || !(fresh && k == 0));
                            }
                        if (ch == 0) mma_commit(leader, &bars[B_RING]);
                        if (ch == 1 || (ch == 0 && c1 == 1)) mma_commit(leader, &bars[B_A0]);
                        if (ch == 3 || (ch == 2 && c1 == 3)) mma_commit(leader, &bars[B_A1]);
                    }
                }
            }
        } else {
            take_registers();
            const int chunk = warp & 3;
            const uint32_t lane_base = tmem + ((uint32_t)(chunk * 32) << 16), base = lane_base + 32 * q;
            const int64_t slot = ((int64_t)h * a.slot_cap) * kTileQ + r;
            const T* drems = (const T*)a.d_rem.ptr + (int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + (int64_t)(c.start + first + r) * a.d_rem.st;
            const int q32 = 2 * (key0 / 64) + q;  // 32-key quarter of the sequence
            bool ok = true;
            uint32_t uses = 0;  // bits 0, 1: parity of the accumulators' barriers, bit 2: of B_RING
            Tile<T, kU, 64, 128> tq, tg;  // half of a step: more of them have no registers
            const T *pq = tq.first(a.q, c, h, first), *pg = tg.first(a.d_o, c, h, first);
            const auto fetch = [&](int rows_left) {
                tq.fetch(pq, a.q.st, D, rows_left);
                tg.fetch(pg, a.d_o.st, D, rows_left);
                pq += 64 * a.q.st;
                pg += 64 * a.d_o.st;
            };
            const auto put = [&](int half) {
                tq.put(sQ + half * 64 * 128);
                tg.put(sG + half * 64 * 128);
            };
            {
                Tile<T, kU, 64> tk, tv;
                tk.fetch(tk.first(a.k, c, h, key0), a.k.st, D, keys_valid);
                tv.fetch(tv.first(a.v, c, h, key0), a.v.st, D, keys_valid);
                fetch(valid(0));
                tk.put(sK);
                tv.put(sV);
                put(0);
                fetch(valid(0) - 64);
                put(1);
            }
            for (int j = 0; j < n; ++j) {
                fence_async_smem();
                tc_fence_before();
                mbar_arrive(&bars[B_LOADED]);
                const bool row_ok = r < valid(j);
                const int64_t at32 = slot + carry_slot32(c.slot_base, c.qt + j, q32) * kTileQ;
                const float W = row_ok ? a.carry_w[at32] : 0.f;
                const float left = row_ok && q32 > 0 ? a.carry_c[at32 - kTileQ] : 0.f;  // through the right edge of the keys to the left
                const float drem = row_ok ? to_f32<T>(drems[(int64_t)128 * j * a.d_rem.st]) : 0.f;
                ok = mbar_wait(&bars[B_READY], j & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                float s[32], dp[32], b[32], sum;
                load_scores<kN>(base + kColS, s);
                load_scores<kN>(base + kColDP, dp);
                tc_fence_before();
                mbar_arrive(&bars[B_FREE]);
                // a query behind the end of the sequence sees no key: its zeros against an infinite or NaN key would make NaNs
                const int lim = row_ok ? min(keys_valid, first + 128 * j + r + a.attend_current - key0) - 32 * q : 0;
                if (j == 0 || keys_valid < 64 || valid(j) < 128) score_grads<true>(s, dp, b, a.inv_temp, lim, drem, W, sum);
                else score_grads<false>(s, dp, b, a.inv_temp, 32, drem, W, sum);
                finish_ds(dp, b, left);
                const int c0 = lo(j), c1 = hi(j);
                if (chunk >= c0 && chunk < c1) {
                    if (chunk == 3 && c0 == 0) {  // takes the place of chunk 0
                        ok = mbar_wait(&bars[B_RING], (uses >> 2) & 1, abort_flag);
                        if (!ok) break;
                    }
                    uint8_t* dst = sW + (chunk == 3 ? 0 : chunk) * kChunk + lane * 128;
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int v = 0; v < 4; ++v) {  // 8 keys: 16 bytes
                            uint32_t w[kWTerms][4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int x = 8 * v + 2 * i;
                                uint32_t t[kWTerms];
                                if (m) split_pair<kWTerms>(dp[x], dp[x + 1], t);
                                else split_pair<kWTerms>(s[x], s[x + 1], t);
#pragma unroll
                                for (int k = 0; k < kWTerms; ++k) w[k][i] = t[k];
                            }
#pragma unroll
                            for (int k = 0; k < kWTerms; ++k)
                                *(uint4*)(dst + (2 * k + m) * 32 * 128 + (((4 * q + v) ^ (lane & 7)) << 4)) = make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
                        }
                    fence_async_smem();
                    mbar_arrive(&bars[B_W0 + chunk]);
                }
                if (c0 == 0) uses ^= 4;
                if (j + 1 < n) fetch(valid(j + 1));
                const uint32_t at = base + (chunk & 2 ? 64 : 0);  // dv: columns 0-63, dk: 64-127
                if (c0 < 2) {
                    ok = mbar_wait(&bars[B_A0], uses & 1, abort_flag);
                    if (!ok) break;
                    uses ^= 1;
                    tc_fence_after();
                    load_sum<2, true>({at + kColA[0], at + kColSmall[0]}, acc);
                }
                if (j + 1 < n) {
                    put(0);
                    fetch(valid(j + 1) - 64);
                }
                if (c1 > 2) {
                    ok = mbar_wait(&bars[B_A1], (uses >> 1) & 1, abort_flag);
                    if (!ok) break;
                    uses ^= 2;
                    tc_fence_after();
                    load_sum<2, true>({at + kColA[1], at + kColSmall[1]}, acc);
                }
                if (j + 1 < n) put(1);
            }
            const int cols = D - 32 * q, key = r & 63;
            const bool is_dk = r >= 64, key_ok = key < keys_valid;
            const bool again = any_row_thread(key_ok && row_asks_for_direct(acc, cols));
            pdl_launch_dependents();
            if (*abort_flag) {
            } else if (again) {
                direct_dkdv<T>(a, smem);
            } else if (key_ok && cols > 0) {
                if (a.fused && !is_dk)  // dv += rem * do
                    add32<T>(acc, to_f32<T>(((const T*)a.rem.ptr)[(int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + (int64_t)(c.start + key0 + key) * a.rem.st]),
                             row_of<T>(a.d_o, c, h, key0 + key) + 32 * q, cols);
                const MatView& m = is_dk ? a.dk : a.dv;
                store32<T>(acc, is_dk ? a.inv_temp : 1.f, (T*)row_of<T>(m, c, h, key0 + key) + 32 * q, unit<T>(m, D), cols);
            }
        }
    }
    tc_teardown(abort_flag, a.status, tmem, 512, 8);
}

// ------------------------------------------------------------------------------------------ launches
dim3 item_grid(int items, int x) {  // heads innermost: the heavy items of all heads start first
    const unsigned y = items < 65535 ? items : 65535;
    return dim3(x, y, (items + y - 1) / y);
}
int launch(void (*kernel)(KArgs), int smem, dim3 grid, const KArgs& a, cudaStream_t st) {
    const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
    return e != 0 ? e : launch_kernel(kernel, grid, dim3(kThreads), smem, st, a);
}
template <typename T>
int host_unit(const MatView& m, int D) {
    const auto ok = [&](int u) { return ((D | m.st | m.sh | m.sb) & (u - 1)) == 0 && ((uintptr_t)m.ptr & (u * sizeof(T) - 1)) == 0; };
    return ok(4) ? 4 : ok(2) ? 2 : 1;
}
template <typename T, int kU>
int launch_u(bool backward, const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    if (!backward) return launch(f32tc_fwd_kernel<T, kU>, fwd_smem<T, kU>(), item_grid(L.max_items, a.heads), a, st);
    if (phases != SBATTN_BWD_DKDV) {
        const int e = launch(f32tc_bwd_dq_kernel<T, kU>, dq_smem<T, kU>(), item_grid(L.max_items, a.heads), a, st);
        if (e != 0) return e;
    }
    if (phases == SBATTN_BWD_DQ) return 0;
    return launch(f32tc_bwd_dkdv_kernel<T, kU>, kv_smem<T>(), item_grid(L.max_items, 2 * a.heads), a, st);
}
template <typename T>
int launch_t(bool backward, const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    int u = 4;
    const auto look = [&](const MatView& m) { const int x = host_unit<T>(m, a.head_dim); u = x < u ? x : u; };
    look(a.q);
    look(a.k);
    look(a.v);
    if (backward) look(a.d_o);
    return u == 4 ? launch_u<T, 4>(backward, L, a, phases, st) : u == 2 ? launch_u<T, 2>(backward, L, a, phases, st) : launch_u<T, 1>(backward, L, a, phases, st);
}

}  // namespace

int launch_f32tc(const SbParams& p, bool backward, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    if (L.max_items <= 0) return 0;
    switch (p.dtype) {
        case SBATTN_BF16: return launch_t<__nv_bfloat16>(backward, L, a, p.bwd_phases, st);
        case SBATTN_F16: return launch_t<__half>(backward, L, a, p.bwd_phases, st);
        default: return launch_t<float>(backward, L, a, p.bwd_phases, st);
    }
}

}  // namespace sb
