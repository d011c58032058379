// Kernels of float32 precision: arithmetic on sums of bf16 terms, tile loads, warp-level products, and the blocks that form their sums by
// ordinary multiply-adds.  Shared by sb_f32.cu (warp-level mma) and sb_f32_tc.cu (tcgen05); compiled without fast math.
#pragma once

#include "sb_common.cuh"

namespace sb {

namespace {

constexpr int kMaxSmem = 227 * 1024;
constexpr int kBM = 64;   // query rows per block
constexpr int kBN = 64;   // keys per tile

template <typename T> struct Terms;
template <> struct Terms<__nv_bfloat16> { static constexpr int n = 1; };
template <> struct Terms<__half> { static constexpr int n = 2; };
template <> struct Terms<float> { static constexpr int n = 3; };
constexpr int kWTerms = 3;  // weights and score gradients

// An operand tile in shared memory: N planes (terms) of 64 rows of DP bf16 values; rows are 16 bytes longer, which spreads the
// eight rows of a matrix load over all banks.
template <int DP> constexpr int kPitch = DP + 8;
template <int DP> constexpr int kPlane = 64 * kPitch<DP>;
template <typename T, int DP> constexpr int kTileElems = Terms<T>::n * kPlane<DP>;

// Where row r of a tile is stored.  A lane = 4 g + t holds of a 16 x 8 accumulator block the elements (g, 2t), (g, 2t + 1), (g + 8, 2t),
// (g + 8, 2t + 1).
enum Order { kPlain, kKeyColumns, kKeyRows };
template <int kOrder>
__device__ __forceinline__ int stored_row(int r) {
    const int k = r & 31;
    // keys along the columns of four blocks (32 keys): key 8 t + 2 n + e in block n, column 2 t + e: a thread has eight neighbours
    if (kOrder == kKeyColumns) return (r & 32) + 8 * ((k >> 1) & 3) + 2 * (k >> 3) + (k & 1);
    // keys along the rows of two blocks: key 4 g + 2 m + h in block m, row 8 h + g: a thread has four neighbours
    if (kOrder == kKeyRows) return (r & 32) + 16 * ((k >> 1) & 1) + 8 * (k & 1) + (k >> 2);
    return r;
}

// two values -> N packed terms.  An infinity, or a value that rounds to one, leaves a NaN in a later term.
template <int N>
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&t)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        t[i] = *(const uint32_t*)&h;
        if (i + 1 < N) {
            x -= __uint_as_float(t[i] << 16);
            y -= __uint_as_float(t[i] & 0xffff0000u);
        }
    }
}

// whether rows can be read or written in units of u elements
template <typename T>
__device__ __forceinline__ bool units_ok(const MatView& m, int D, int u) {
    return ((D | m.st | m.sh | m.sb) & (u - 1)) == 0 && ((uintptr_t)m.ptr & (u * sizeof(T) - 1)) == 0;
}

// kRows rows of a [.., T, D] tensor on their way into a tile: fetch() issues the loads, put() splits and stores them, with zeros
// behind the valid rows and columns.  Between the two lie a barrier and, where registers allow, the work on the tile before.  A
// thread keeps its columns and walks the rows.
template <int kT, typename T, int DP, int kRows = 64, int kTileRows = kRows>
struct Rows {
    uint32_t w[kRows * DP / kT > 4 ? kRows * DP / kT : 4];

    template <int kU>  // elements per load
    struct Map {
        static constexpr int kPer = DP / kU;                      // threads per row
        static constexpr int kStep = kT / kPer;                   // rows per pass
        static constexpr int kPasses = kRows / kStep > 0 ? kRows / kStep : 1;
        static constexpr int kWords = sizeof(T) == 4 ? kU : (kU + 1) / 2;
    };
    template <int kU>
    __device__ __forceinline__ void fetch_u(const T* base, int64_t st, int D, int rows_valid) {
        using M = Map<kU>;
        const int d = kU * ((int)threadIdx.x % M::kPer), r0 = (int)threadIdx.x / M::kPer;
        const T* src = base + r0 * st + d;
        const bool col_ok = d < D;
#pragma unroll
        for (int i = 0; i < M::kPasses; ++i) {
            uint32_t* x = w + i * M::kWords;
#pragma unroll
            for (int u = 0; u < M::kWords; ++u) x[u] = 0;
            if (!col_ok || r0 + i * M::kStep >= rows_valid) continue;
            const T* p = src + (int64_t)i * M::kStep * st;
            if constexpr (M::kWords == 4) {
                const uint4 v = *(const uint4*)p;
                x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
            } else if constexpr (M::kWords == 2) {
                const uint2 v = *(const uint2*)p;
                x[0] = v.x; x[1] = v.y;
            } else if constexpr (sizeof(T) * kU == 4) {
                x[0] = *(const uint32_t*)p;
            } else {
                x[0] = *(const unsigned short*)p;
            }
        }
    }
    template <int kOrder, int kU>
    __device__ __forceinline__ void put_u(__nv_bfloat16* dst, int first = 0) const {
        using M = Map<kU>;
        constexpr int kN = Terms<T>::n;
        const int d = kU * ((int)threadIdx.x % M::kPer), r0 = (int)threadIdx.x / M::kPer;
#pragma unroll
        for (int i = 0; i < M::kPasses; ++i) {
            const uint32_t* x = w + i * M::kWords;
            const int r = r0 + i * M::kStep;
            if (M::kStep > kRows && r >= kRows) continue;
            uint32_t t[kU > 1 ? kU / 2 : 1][kN];
#pragma unroll
            for (int u = 0; u < (kU > 1 ? kU / 2 : 1); ++u) {
                if constexpr (kN == 1) {
                    t[u][0] = x[u];
                } else if constexpr (sizeof(T) == 4) {
                    split_pair<kN>(__uint_as_float(x[kU > 1 ? 2 * u : 0]), kU > 1 ? __uint_as_float(x[kU > 1 ? 2 * u + 1 : 0]) : 0.f, t[u]);
                } else {
                    const float2 v = __half22float2(*(const __half2*)&x[u]);
                    split_pair<kN>(v.x, v.y, t[u]);
                }
            }
            __nv_bfloat16* p = dst + stored_row<kOrder>(first + r) * kPitch<DP> + d;
#pragma unroll
            for (int n = 0; n < kN; ++n) {
                if constexpr (kU == 4) *(uint2*)(p + n * kTileRows * kPitch<DP>) = make_uint2(t[0][n], t[1][n]);
                else if constexpr (kU == 2) *(uint32_t*)(p + n * kTileRows * kPitch<DP>) = t[0][n];
                else *(unsigned short*)(p + n * kTileRows * kPitch<DP>) = (unsigned short)t[0][n];
            }
        }
    }
    // u: what unit() says of the tensor
    __device__ __forceinline__ void fetch(const MatView& m, int u, int D, int b, int h, int row0, int rows_valid) {
        const T* base = (const T*)m.ptr + (int64_t)b * m.sb + (int64_t)h * m.sh + (int64_t)row0 * m.st;
        if (u == 4) fetch_u<4>(base, m.st, D, rows_valid);
        else if (u == 2) fetch_u<2>(base, m.st, D, rows_valid);
        else fetch_u<1>(base, m.st, D, rows_valid);
    }
    template <int kOrder>
    __device__ __forceinline__ void put(__nv_bfloat16* dst, int u) const {
        if (u == 4) put_u<kOrder, 4>(dst);
        else if (u == 2) put_u<kOrder, 2>(dst);
        else put_u<kOrder, 1>(dst);
    }
};
template <typename T>
__device__ __forceinline__ int unit(const MatView& m, int D) { return units_ok<T>(m, D, 4) ? 4 : units_ok<T>(m, D, 2) ? 2 : 1; }
template <int kT, typename T, int DP, int kOrder>
__device__ __forceinline__ void load_tile(__nv_bfloat16* dst, const MatView& m, int D, int b, int h, int row0, int rows_valid) {
    const T* base = (const T*)m.ptr + (int64_t)b * m.sb + (int64_t)h * m.sh + (int64_t)row0 * m.st;
    Rows<kT, T, DP> x;
    if (units_ok<T>(m, D, 4)) {
        x.template fetch_u<4>(base, m.st, D, rows_valid);
        x.template put_u<kOrder, 4>(dst);
    } else if (units_ok<T>(m, D, 2)) {
        x.template fetch_u<2>(base, m.st, D, rows_valid);
        x.template put_u<kOrder, 2>(dst);
    } else {
        Rows<kT, T, DP, 32, 64> y;
#pragma unroll 1
        for (int r = 0; r < 64; r += 32) {
            y.template fetch_u<1>(base + r * m.st, m.st, D, rows_valid - r);
            y.template put_u<kOrder, 1>(dst, r);
        }
    }
}

// ------------------------------------------------------------------------------------------ warp-level matrix instructions
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];"
                 : "=r"(r[0]), "=r"(r[1])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const __nv_bfloat16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p))
                 : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The tensor cores round every accumulation towards zero, so sums are kept short: the leading products x0 y0 of at most 64 indices
// are accumulated from zero, all smaller ones (whose rounding does not matter) in a second accumulator, and the two are added
// with ordinary float32 additions.  Longer sums are float32 additions of such pieces.  Independent accumulators are innermost
// in the loops: a chain of dependent mma runs at a fraction of the rate.

// c[mb][nb] = A[16 kMB rows] * B[8 kNB rows]^T over D columns; A and B tiles, `a` and `b` at their first rows, B of kRowsB rows
template <int kN, int DP, int kMB, int kNB, int kRowsB = 64>
__device__ __forceinline__ void product_nt(float (&c)[kMB][kNB][4], const __nv_bfloat16* a, const __nv_bfloat16* b, int D, int lane) {
    const __nv_bfloat16* pa = a + (lane & 15) * kPitch<DP> + (lane >> 4) * 8;
    const __nv_bfloat16* pb = b + ((lane & 7) + ((lane >> 4) << 3)) * kPitch<DP> + ((lane >> 3) & 1) * 8;
    float small[kMB][kNB][4], first[kMB][kNB][4];  // first: the leading products of the first 64 indices, D > 64
#pragma unroll
    for (int m = 0; m < kMB; ++m)
#pragma unroll
        for (int n = 0; n < kNB; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) c[m][n][i] = small[m][n][i] = first[m][n][i] = 0.f;
#pragma unroll 1
    for (int k = 0; k < D; k += 16) {
        uint32_t fa[kMB][kN][4];
#pragma unroll
        for (int m = 0; m < kMB; ++m)
#pragma unroll
            for (int i = 0; i < kN; ++i) ldsm4(fa[m][i], pa + i * kPlane<DP> + m * 16 * kPitch<DP> + k);
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            uint32_t fb[(kNB + 1) / 2][4];
            if constexpr (kNB == 1) ldsm2(fb[0], pb + j * kRowsB * kPitch<DP> + k);
#pragma unroll
            for (int n2 = 0; n2 < kNB / 2; ++n2) ldsm4(fb[n2], pb + j * kRowsB * kPitch<DP> + n2 * 16 * kPitch<DP> + k);
#pragma unroll
            for (int i = 0; i < kN; ++i) {
                if (i + j > 2) continue;
#pragma unroll
                for (int n = 0; n < kNB; ++n)
#pragma unroll
                    for (int m = 0; m < kMB; ++m)
                        mma(i + j == 0 ? c[m][n] : small[m][n], fa[m][i], fb[n >> 1][2 * (n & 1)], fb[n >> 1][2 * (n & 1) + 1]);
            }
        }
        if (DP > 64 && k + 16 == 64) {  // 64 indices are the longest sum: the second 64 start anew
#pragma unroll
            for (int m = 0; m < kMB; ++m)
#pragma unroll
                for (int n = 0; n < kNB; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        first[m][n][i] = c[m][n][i];
                        c[m][n][i] = 0.f;
                    }
        }
    }
    if (kN > 1 || DP > 64)
#pragma unroll
        for (int m = 0; m < kMB; ++m)
#pragma unroll
            for (int n = 0; n < kNB; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) c[m][n][i] += DP > 64 ? first[m][n][i] + small[m][n][i] : small[m][n][i];
}

// acc[mb][DC / 8] += P * X: P = kMB x kNB accumulator blocks in registers (float32, three terms), X a tile whose rows are the contracted
// index (`x` at the first row and column), DC columns of it, 32 at a time
template <int kN, int DP, int DC, int kMB, int kNB>
__device__ __forceinline__ void product_px(float (&acc)[kMB][DC / 8][4], const float (&p)[kMB][kNB][4], const __nv_bfloat16* x, int lane) {
    constexpr int kNC = DC < 32 ? DC / 8 : 4;  // column blocks at a time
    const __nv_bfloat16* px = x + ((lane & 7) + ((lane >> 3) & 1) * 8) * kPitch<DP> + (lane >> 4) * 8;
    uint32_t fa[kNB / 2][kMB][kWTerms][4];
#pragma unroll
    for (int k = 0; k < kNB / 2; ++k)
#pragma unroll
        for (int m = 0; m < kMB; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float* v = p[m][2 * k + (e >> 1)];
                uint32_t t[kWTerms];
                split_pair<kWTerms>(v[2 * (e & 1)], v[2 * (e & 1) + 1], t);
#pragma unroll
                for (int i = 0; i < kWTerms; ++i) fa[k][m][i][e] = t[i];
            }
#pragma unroll
    for (int n0 = 0; n0 < DC / 8; n0 += kNC) {
        float big[kMB][kNC][4] = {}, small[kMB][kNC][4] = {};
#pragma unroll
        for (int k = 0; k < kNB / 2; ++k) {
#pragma unroll
            for (int j = 0; j < kN; ++j) {
                uint32_t fb[kNC / 2][4];
#pragma unroll
                for (int n2 = 0; n2 < kNC / 2; ++n2) ldsm4_t(fb[n2], px + j * kPlane<DP> + k * 16 * kPitch<DP> + n0 * 8 + n2 * 16);
#pragma unroll
                for (int i = 0; i < kWTerms; ++i) {
                    if (i + j > 2) continue;
#pragma unroll
                    for (int n = 0; n < kNC; ++n)
#pragma unroll
                        for (int m = 0; m < kMB; ++m)
                            mma(i + j == 0 ? big[m][n] : small[m][n], fa[k][m][i], fb[n >> 1][2 * (n & 1)], fb[n >> 1][2 * (n & 1) + 1]);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < kMB; ++m)
#pragma unroll
            for (int n = 0; n < kNC; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[m][n0 + n][i] += big[m][n][i] + small[m][n][i];
    }
}

// ------------------------------------------------------------------------------------------ the same products on the values themselves
// whether a thread's results (elements i0, i0 + 1 of its accumulator blocks: one row, every fourth pair of columns) ask for them: a NaN, or nothing but
// magnitudes below 2^-100
template <int kN>
__device__ __forceinline__ bool asks_for_direct(const float (&acc)[kN][4], int i0) {
    float most = 0.f;
    bool nan = false;
#pragma unroll
    for (int n = 0; n < kN; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            nan |= acc[n][i0 + e] != acc[n][i0 + e];
            most = fmaxf(most, fabsf(acc[n][i0 + e]));
        }
    return nan || (most > 0.f && most < 0x1p-100f);
}
// c[r][j] = row r of A (na of them valid) . row j of B (nb valid)
template <typename T, int kR, int kC>
__device__ __forceinline__ void direct_nt(float (&c)[kR][kC], const T* a, int64_t sa, int na, const T* b, int64_t sb, int nb, int D) {
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int j = 0; j < kC; ++j) c[r][j] = 0.f;
#pragma unroll 1
    for (int d = 0; d < D; ++d) {
        float x[kR], y[kC];
#pragma unroll
        for (int r = 0; r < kR; ++r) x[r] = r < na ? to_f32<T>(a[r * sa + d]) : 0.f;
#pragma unroll
        for (int j = 0; j < kC; ++j) y[j] = j < nb ? to_f32<T>(b[j * sb + d]) : 0.f;
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int j = 0; j < kC; ++j) c[r][j] = fmaf(x[r], y[j], c[r][j]);
    }
}
// scores of forward and dq: this lane's rows (r, r + 8) against its eight neighbouring keys
template <typename T>
__device__ __forceinline__ void direct_scores(float (&s)[1][4][4], const T* a, int64_t sa, int rows, const T* b, int64_t sb, int keys, int D) {
    float c[2][8];
    direct_nt<T>(c, a, 8 * sa, rows > 8 ? 2 : rows > 0, b, sb, keys, D);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[0][j >> 1][2 * r + (j & 1)] = c[r][j];
}
// scores of dk/dv: four neighbouring keys against this lane's two queries
template <typename T>
__device__ __forceinline__ void direct_scores_t(float (&s)[2][1][4], const T* a, int64_t sa, int keys, const T* b, int64_t sb, int rows, int D) {
    float c[4][2];
    direct_nt<T>(c, a, sa, keys, b, sb, rows, D);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) s[k >> 1][0][2 * (k & 1) + e] = c[k][e];
}
// acc += P * X over the 32 keys of a half, `keys` of them valid; P in registers as the forward and dq hold it
template <typename T, int DP>
__device__ __forceinline__ void direct_px(float (&acc)[1][DP / 8][4], const float (&p)[1][4][4], const T* x, int64_t st, int keys, int D, int lane) {
    const int t = lane & 3;
#pragma unroll 1
    for (int from = 0; from < 4; ++from) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float p0 = __shfl_sync(0xffffffffu, p[0][j >> 1][j & 1], (lane & ~3) | from);
            const float p1 = __shfl_sync(0xffffffffu, p[0][j >> 1][2 + (j & 1)], (lane & ~3) | from);
            const int k = 8 * from + j;
            if (k >= keys) continue;
#pragma unroll
            for (int n = 0; n < DP / 8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int d = 8 * n + 2 * t + e;
                    const float v = d < D ? to_f32<T>(x[k * st + d]) : 0.f;
                    acc[0][n][e] = fmaf(p0, v, acc[0][n][e]);
                    acc[0][n][2 + e] = fmaf(p1, v, acc[0][n][2 + e]);
                }
        }
    }
}

// The same three on tiles of float32 values in shared memory: rows of DP columns, 16 bytes longer, and 16 more after every eighth, so that rows next to each other
// and rows eight apart start in different banks; zeros behind the valid rows and columns.  Four columns at a time; sums in the same order.
template <int DP> constexpr int kValuePitch = DP + 4;               // inside eight rows
template <int DP> constexpr int kValueEight = 8 * kValuePitch<DP> + 4;
template <int DP> constexpr int kValues = 8 * kValueEight<DP>;  // of a tile
template <int DP>
__device__ __forceinline__ int value_row(int r) { return (r >> 3) * kValueEight<DP> + (r & 7) * kValuePitch<DP>; }
template <typename T, int DP, int kRows>
__device__ __forceinline__ void stage_values(float* dst, const T* src, int64_t st, int D, int rows_valid) {  // 256 threads
    constexpr int kStep = 256 / DP, kPasses = kRows / kStep, kBatch = kPasses < 8 ? kPasses : 8;  // loads under way at a time: the stores may alias them
    const int d = threadIdx.x % DP, r0 = threadIdx.x / DP, left = d < D ? rows_valid - r0 : 0;
    src += r0 * st + d;
#pragma unroll
    for (int i0 = 0; i0 < kPasses; i0 += kBatch) {
        float v[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) v[i] = (i0 + i) * kStep < left ? to_f32<T>(src[(i0 + i) * kStep * st]) : 0.f;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) dst[value_row<DP>(r0 + (i0 + i) * kStep) + d] = v[i];
    }
}
template <int DP, int kR, int kC>
__device__ __forceinline__ void values_nt(float (&c)[kR][kC], const float* a, int sa, const float* b, int sb, int D) {
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
        for (int j = 0; j < kC; ++j) c[r][j] = 0.f;
#pragma unroll 1
    for (int d = 0; d < D; d += 4) {
        float4 x[kR], y[kC];
#pragma unroll
        for (int r = 0; r < kR; ++r) x[r] = *(const float4*)(a + r * sa + d);
#pragma unroll
        for (int j = 0; j < kC; ++j) y[j] = *(const float4*)(b + j * sb + d);
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int j = 0; j < kC; ++j) c[r][j] = fmaf(x[r].w, y[j].w, fmaf(x[r].z, y[j].z, fmaf(x[r].y, y[j].y, fmaf(x[r].x, y[j].x, c[r][j]))));
    }
}
template <int DP>
__device__ __forceinline__ void values_scores(float (&s)[1][4][4], const float* a, const float* b, int D) {
    float c[2][8];
    values_nt<DP>(c, a, kValueEight<DP>, b, kValuePitch<DP>, D);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[0][j >> 1][2 * r + (j & 1)] = c[r][j];
}
template <int DP>
__device__ __forceinline__ void values_scores_t(float (&s)[2][1][4], const float* a, const float* b, int D) {
    float c[4][2];
    values_nt<DP>(c, a, kValuePitch<DP>, b, kValuePitch<DP>, D);
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) s[k >> 1][0][2 * (k & 1) + e] = c[k][e];
}
template <int DP>
__device__ __forceinline__ void values_px(float (&acc)[1][DP / 8][4], const float (&p)[1][4][4], const float* x, int keys, int lane) {
    const int t = lane & 3;
#pragma unroll 1
    for (int from = 0; from < 4; ++from) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float p0 = __shfl_sync(0xffffffffu, p[0][j >> 1][j & 1], (lane & ~3) | from);
            const float p1 = __shfl_sync(0xffffffffu, p[0][j >> 1][2 + (j & 1)], (lane & ~3) | from);
            const int k = 8 * from + j;
            if (k >= keys) continue;
#pragma unroll
            for (int n = 0; n < DP / 8; ++n) {
                const float2 v = *(const float2*)(x + from * kValueEight<DP> + j * kValuePitch<DP> + 8 * n + 2 * t);
                acc[0][n][0] = fmaf(p0, v.x, acc[0][n][0]);
                acc[0][n][1] = fmaf(p0, v.y, acc[0][n][1]);
                acc[0][n][2] = fmaf(p1, v.x, acc[0][n][2]);
                acc[0][n][3] = fmaf(p1, v.y, acc[0][n][3]);
            }
        }
    }
}

// a row of accumulator blocks (elements i0, i0 + 1 of each) into row `row` of a [.., T, D] tensor
template <typename T, int DC>
__device__ __forceinline__ void store_row(const float (&acc)[DC / 8][4], int i0, float scale, const MatView& m, bool pairs, int D, int col0, T* base,
                                          int row, int t) {
    T* dst = base + (int64_t)row * m.st;
#pragma unroll
    for (int n = 0; n < DC / 8; ++n) {
        const int d = col0 + 8 * n + 2 * t;
        T v[2] = {from_f32<T>(acc[n][i0] * scale), from_f32<T>(acc[n][i0 + 1] * scale)};
        if (pairs) {
            if (d < D) {
                if constexpr (sizeof(T) == 4) *(float2*)(dst + d) = make_float2(v[0], v[1]);
                else *(uint32_t*)(dst + d) = *(const uint32_t*)v;
            }
        } else {
            if (d < D) dst[d] = v[0];
            if (d + 1 < D) dst[d + 1] = v[1];
        }
    }
}

// the same elements += f * x
template <typename T, int DC>
__device__ __forceinline__ void add_row(float (&acc)[DC / 8][4], int i0, float f, const T* x, int D, int col0, int t) {
#pragma unroll
    for (int n = 0; n < DC / 8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int d = col0 + 8 * n + 2 * t + e;
            if (d < D) acc[n][i0 + e] = __fadd_rn(acc[n][i0 + e], __fmul_rn(f, to_f32<T>(x[d])));
        }
}

// sigmoid pieces with full relative accuracy on both sides: beta = sigmoid(s), r = 1 - beta
__device__ __forceinline__ void sigmoid_pair(float s, float& beta, float& r) {
    const float e = expf(-fabsf(s));
    const float inv = 1.0f / (1.0f + e);
    const float big = inv, small = e * inv;
    beta = s >= 0.f ? big : small;
    r = s >= 0.f ? small : big;
}

// One step of a scan over lanes: combine with the value `off` lanes to the right (left) where there is one.  kSeg: clamp and segment
// operand of the shuffle (0x1c1f: four lanes, towards larger; 0x1c00: four lanes, towards smaller; 0x1f: the warp).
template <int kSeg>
__device__ __forceinline__ float mul_right(float x, int off) {
    asm("{\n\t.reg .pred p;\n\t.reg .f32 y;\n\t"
        "shfl.sync.down.b32 y|p, %0, %1, %2, 0xffffffff;\n\t"
        "@p mul.rn.f32 %0, %0, y;\n\t}" : "+f"(x) : "r"(off), "n"(kSeg));
    return x;
}
template <int kSeg>
__device__ __forceinline__ float add_right(float x, int off) {
    asm("{\n\t.reg .pred p;\n\t.reg .f32 y;\n\t"
        "shfl.sync.down.b32 y|p, %0, %1, %2, 0xffffffff;\n\t"
        "@p add.rn.f32 %0, %0, y;\n\t}" : "+f"(x) : "r"(off), "n"(kSeg));
    return x;
}
template <int kSeg>
__device__ __forceinline__ float add_left(float x, int off) {
    asm("{\n\t.reg .pred p;\n\t.reg .f32 y;\n\t"
        "shfl.sync.up.b32 y|p, %0, %1, %2, 0xffffffff;\n\t"
        "@p add.rn.f32 %0, %0, y;\n\t}" : "+f"(x) : "r"(off), "n"(kSeg));
    return x;
}
constexpr int kQuadRight = 0x1c1f, kQuadLeft = 0x1c00, kWarpRight = 0x1f;

// the two warps that share 16 query rows
__device__ __forceinline__ void pair_sync(int group) { asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory"); }
// How a 64-row block forms its sums: of terms; by multiply-adds on the values where they lie; or on copies of them in shared memory (blocks that have an SM
// to themselves: room for the copies, and too few warps for the latency of the loads)
enum Sums { kTerms, kValuesInPlace, kStaged };
// the 256 threads of a 64-row block: a thread block, or (kStaged) the first ones of a larger one
template <int kSums>
__device__ __forceinline__ void rows_sync() {
    if (kSums == kStaged) asm volatile("bar.sync 9, 256;" ::: "memory");
    else __syncthreads();
}

struct ItemCtx {
    int qt, b, start, len, slot_base;
};
__device__ inline ItemCtx item_ctx(const int2* items, const SeqInfo* seqs, int item) {
    const int2 it = items[item];
    const SeqInfo s = seqs[it.x];
    return ItemCtx{it.y, s.batch, s.start, s.len, s.slot_base};
}
__device__ inline ItemCtx item_ctx(const KArgs& a, int item) { return item_ctx(a.items, a.seqs, item); }
// row `i` of the item's sequence
template <typename T>
__device__ __forceinline__ const T* row_of(const MatView& m, const ItemCtx& c, int h, int i) {
    return (const T*)m.ptr + (int64_t)c.b * m.sb + (int64_t)h * m.sh + (int64_t)(c.start + i) * m.st;
}
// Blocks in the order of the item table (heaviest first), the heads and the halves of a 128-row tile innermost: the hardware
// deals blocks out in this order, so the heavy ones of all heads start first.  Items along y and z (together more than an axis takes,
// and more blocks than x alone would).
struct BlockIdx {
    int item, h, part;
};
inline dim3 block_grid(int items, int heads) {
    const unsigned y = items < 65535 ? items : 65535;
    return dim3(2u * heads, y, (items + y - 1) / y);
}
__device__ __forceinline__ BlockIdx block_idx() {
    return BlockIdx{(int)min(blockIdx.z * gridDim.y + blockIdx.y, 0x7fffffffu), (int)(blockIdx.x >> 1), (int)(blockIdx.x & 1)};
}
__device__ __forceinline__ int64_t linear_thread() {
    return (((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ int64_t all_threads() { return (int64_t)gridDim.x * gridDim.y * gridDim.z * blockDim.x; }

// ------------------------------------------------------------------------------------------ forward
// Eight warps: four groups of 16 query rows x the two 32-key halves of a tile.  The halves exchange their products once per tile; o
// is summed over the halves at the end.
// kSums: how the sums are formed; returns whether multiply-adds have to (nothing is stored then).
// xs: product of 1 - beta over a half, per row.
template <typename T, int DP, int kSums>
__device__ __forceinline__ bool fwd_block(const KArgs& a, const ItemCtx& c, const BlockIdx& bi, __nv_bfloat16* tiles, float (*xs)[kBM]) {
    constexpr int kT = 256, kN = Terms<T>::n;
    constexpr bool kDirect = kSums != kTerms;
    constexpr bool kEarly = sizeof(T) == 2 && !kDirect;  // loads a tile ahead; the 32 words of two float32 tiles cost more registers than they gain
    float* const vQ = (float*)tiles;  // kStaged
    float *const vK = vQ + kValues<DP>, *const vV = vK + kValues<DP>;
    __nv_bfloat16* sQ = tiles;
    __nv_bfloat16* sK = sQ + kTileElems<T, DP>;
    __nv_bfloat16* sV = sK + kTileElems<T, DP>;
    const int h = bi.h, D = a.head_dim;
    const int row0 = c.qt * kTileQ + bi.part * kBM;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int rg = warp & 3, hf = warp >> 2;  // hf 0: the left 32 keys, 1: the right
    const int rows_valid = min(kBM, c.len - row0);
    if (kSums == kStaged) stage_values<T, DP, kBM>(vQ, row_of<T>(a.q, c, h, row0), a.q.st, D, rows_valid);
    if (!kDirect) load_tile<kT, T, DP, kPlain>(sQ, a.q, D, c.b, h, c.start + row0, rows_valid);
    const int wrow = 16 * rg + g;  // this lane's rows of the block: wrow, wrow + 8
    float W[2] = {1.f, 1.f};
    float o[1][DP / 8][4] = {};
    float* cw = a.carry_w ? a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ + bi.part * kBM + wrow : nullptr;
    const int last = (row0 + rows_valid - 1) / kBN;
    // key tiles of the 128-key diagonal tile that lie right of these rows: a tensor-core backward may follow, and it reads the
    // carry of every quarter of its tile
    if (cw && t == 0)
        for (int kh = last + 1; kh <= 2 * c.qt + 1 && kh * kBN < c.len; ++kh)
#pragma unroll
            for (int r = 0; r < 2; ++r) cw[carry_slot32(c.slot_base, c.qt, 2 * kh + hf) * kTileQ + 8 * r] = 1.f;

    const int uk = unit<T>(a.k, D), uv = unit<T>(a.v, D);
    Rows<kT, T, DP> rk, rv;
    auto fetch = [&](int kh) {
        const int n = min(kBN, c.len - kh * kBN);
        rk.fetch(a.k, uk, D, c.b, h, c.start + kh * kBN, n);
        rv.fetch(a.v, uv, D, c.b, h, c.start + kh * kBN, n);
    };
    if (kEarly) fetch(last);
    for (int kh = last; kh >= 0; --kh) {
        const int key0 = kh * kBN;
        const int keys_valid = min(kBN, c.len - key0);
        rows_sync<kSums>();
        if (kSums == kStaged) {
            stage_values<T, DP, kBN>(vK, row_of<T>(a.k, c, h, key0), a.k.st, D, keys_valid);
            stage_values<T, DP, kBN>(vV, row_of<T>(a.v, c, h, key0), a.v.st, D, keys_valid);
        } else if (kDirect) {
        } else if (kEarly) {
            rk.template put<kKeyColumns>(sK, uk);
            rv.template put<kKeyColumns>(sV, uv);
        } else {
            load_tile<kT, T, DP, kKeyColumns>(sK, a.k, D, c.b, h, c.start + key0, keys_valid);
            load_tile<kT, T, DP, kKeyColumns>(sV, a.v, D, c.b, h, c.start + key0, keys_valid);
        }
        rows_sync<kSums>();
        float s[1][4][4], om[2][8], excl[2];
        if (kSums == kStaged) values_scores<DP>(s, vQ + value_row<DP>(wrow), vK + (4 * hf + t) * kValueEight<DP>, D);
        else if (kDirect) direct_scores<T>(s, row_of<T>(a.q, c, h, row0 + wrow), a.q.st, rows_valid - wrow, row_of<T>(a.k, c, h, key0 + 32 * hf + 8 * t), a.k.st, keys_valid - 32 * hf - 8 * t, D);
        else product_nt<kN, DP, 1, 4>(s, sQ + 16 * rg * kPitch<DP>, sK + 32 * hf * kPitch<DP>, D, lane);
        const bool edge = kh == last || keys_valid < kBN;  // some pair of the tile is not visible
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float beta[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) sigmoid_pair(s[0][j >> 1][2 * r + (j & 1)] * a.inv_temp, beta[j], om[r][j]);
            if (edge) {
                const int lim = min(keys_valid, row0 + wrow + 8 * r + a.attend_current - key0) - 32 * hf - 8 * t;  // keys < lim of this lane are visible
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j >= lim) { beta[j] = 0.f; om[r][j] = 1.f; }
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s[0][j >> 1][2 * r + (j & 1)] = beta[j];
            float incl = ((om[r][0] * om[r][1]) * (om[r][2] * om[r][3])) * ((om[r][4] * om[r][5]) * (om[r][6] * om[r][7]));
            incl = mul_right<kQuadRight>(incl, 1);
            incl = mul_right<kQuadRight>(incl, 2);
            const float y = __shfl_down_sync(0xffffffffu, incl, 1, 4);
            excl[r] = t == 3 ? 1.f : y;
            if (t == 0) xs[hf][wrow + 8 * r] = incl;  // over the whole half
        }
        pair_sync(rg);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float right = xs[1][wrow + 8 * r], left = xs[0][wrow + 8 * r];
            const float win = hf ? W[r] : W[r] * right;  // at the right edge of this half
            if (cw && t == 0) cw[carry_slot32(c.slot_base, c.qt, 2 * kh + hf) * kTileQ + 8 * r] = win;
            float run = win * excl[r];
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                s[0][j >> 1][2 * r + (j & 1)] *= run;
                run *= om[r][j];
            }
            W[r] = W[r] * right * left;
        }
        if (kEarly && kh > 0) fetch(kh - 1);
        if (kSums == kStaged) values_px<DP>(o, s, vV + 4 * hf * kValueEight<DP>, keys_valid - 32 * hf, lane);
        else if (kDirect) direct_px<T, DP>(o, s, row_of<T>(a.v, c, h, key0 + 32 * hf), a.v.st, keys_valid - 32 * hf, D, lane);
        else product_px<kN, DP, DP, 1, 4>(o, s, sV + 32 * hf * kPitch<DP>, lane);
    }
    float* x = (float*)tiles;
    rows_sync<kSums>();
    if (hf == 1) {
#pragma unroll
        for (int n = 0; n < DP / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[((rg * (DP / 8) + n) * 4 + e) * 32 + lane] = o[0][n][e];
    }
    rows_sync<kSums>();
    bool again = false;
    if (hf == 0) {
#pragma unroll
        for (int n = 0; n < DP / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[0][n][e] += x[((rg * (DP / 8) + n) * 4 + e) * 32 + lane];
#pragma unroll
        for (int r = 0; r < 2; ++r) again |= wrow + 8 * r < rows_valid && (asks_for_direct(o[0], 2 * r) || W[r] != W[r]);
    }
    if (!kDirect && __syncthreads_or(again)) return true;
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    if (hf == 1) return false;
    if (a.fused) {  // out = o + rem * v, each operation rounded by itself: the same bits as the expression outside for float32
        const T* v = (const T*)a.v.ptr + (int64_t)c.b * a.v.sb + (int64_t)h * a.v.sh + (int64_t)(c.start + row0) * a.v.st;
#pragma unroll
        for (int r = 0; r < 2; ++r)
            if (wrow + 8 * r < rows_valid) add_row<T, DP>(o[0], 2 * r, to_f32<T>(from_f32<T>(W[r])), v + (int64_t)(wrow + 8 * r) * a.v.st, D, 0, t);
    }
    const bool pairs = units_ok<T>(a.o, D, 2);
    T* base = (T*)a.o.ptr + (int64_t)c.b * a.o.sb + (int64_t)h * a.o.sh + (int64_t)(c.start + row0) * a.o.st;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (wrow + 8 * r >= rows_valid) continue;
        store_row<T, DP>(o[0], 2 * r, 1.f, a.o, pairs, D, 0, base, wrow + 8 * r, t);
        if (t == 0) {
            const int64_t tok = c.start + row0 + wrow + 8 * r;
            ((T*)a.rem.ptr)[(int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + tok * a.rem.st] = from_f32<T>(W[r]);
            ((float*)a.nla.ptr)[(int64_t)c.b * a.nla.sb + (int64_t)h * a.nla.sh + tok * a.nla.st] = log2f(W[r]);
        }
    }
    return false;
}
// ------------------------------------------------------------------------------------------ backward: dq
// Warps as in the forward; W comes from the forward's carries, the halves exchange their sums of g.
// xs: sum of g over a half, per row.
template <typename T, int DP, int kSums>
__device__ __forceinline__ bool dq_block(const KArgs& a, const ItemCtx& c, const BlockIdx& bi, __nv_bfloat16* tiles, float (*xs)[kBM]) {
    constexpr int kT = 256, kN = Terms<T>::n;
    constexpr bool kDirect = kSums != kTerms;
    constexpr bool kEarly = (kN == 1 || (kN == 2 && DP < 64)) && !kDirect;  // loads a tile ahead, where registers allow
    float* const vQ = (float*)tiles;  // kStaged
    float *const vG = vQ + kValues<DP>, *const vK = vG + kValues<DP>, *const vV = vK + kValues<DP>;
    __nv_bfloat16* sQ = tiles;
    __nv_bfloat16* sG = sQ + kTileElems<T, DP>;  // dO
    __nv_bfloat16* sK = sG + kTileElems<T, DP>;
    __nv_bfloat16* sV = sK + kTileElems<T, DP>;
    const int h = bi.h, D = a.head_dim;
    const int row0 = c.qt * kTileQ + bi.part * kBM;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int rg = warp & 3, hf = warp >> 2;
    const int rows_valid = min(kBM, c.len - row0);
    if (kSums == kStaged) {
        stage_values<T, DP, kBM>(vQ, row_of<T>(a.q, c, h, row0), a.q.st, D, rows_valid);
        stage_values<T, DP, kBM>(vG, row_of<T>(a.d_o, c, h, row0), a.d_o.st, D, rows_valid);
    }
    if (!kDirect) {
        load_tile<kT, T, DP, kPlain>(sQ, a.q, D, c.b, h, c.start + row0, rows_valid);
        load_tile<kT, T, DP, kPlain>(sG, a.d_o, D, c.b, h, c.start + row0, rows_valid);
    }
    const int wrow = 16 * rg + g;
    float drem[2], prefix[2] = {0.f, 0.f};  // prefix: sum of g over all keys left of the current tile
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int64_t tok = c.start + row0 + wrow + 8 * r;
        drem[r] = wrow + 8 * r < rows_valid ? to_f32<T>(((const T*)a.d_rem.ptr)[(int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + tok * a.d_rem.st]) : 0.f;
    }
    const float* cw = a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ + bi.part * kBM + wrow;
    float* cc = a.carry_c + ((int64_t)h * a.slot_cap) * kTileQ + bi.part * kBM + wrow;
    float o[1][DP / 8][4] = {};
    const int last = (row0 + rows_valid - 1) / kBN;

    const int uk = unit<T>(a.k, D), uv = unit<T>(a.v, D);
    Rows<kT, T, DP> rk, rv;
    auto fetch = [&](int kh) {
        const int n = min(kBN, c.len - kh * kBN);
        rk.fetch(a.k, uk, D, c.b, h, c.start + kh * kBN, n);
        rv.fetch(a.v, uv, D, c.b, h, c.start + kh * kBN, n);
    };
    if (kEarly) fetch(0);
    for (int kh = 0; kh <= last; ++kh) {
        const int key0 = kh * kBN;
        const int keys_valid = min(kBN, c.len - key0);
        rows_sync<kSums>();
        if (kSums == kStaged) {
            stage_values<T, DP, kBN>(vK, row_of<T>(a.k, c, h, key0), a.k.st, D, keys_valid);
            stage_values<T, DP, kBN>(vV, row_of<T>(a.v, c, h, key0), a.v.st, D, keys_valid);
        } else if (kDirect) {
        } else if (kEarly) {
            rk.template put<kKeyColumns>(sK, uk);
            rv.template put<kKeyColumns>(sV, uv);
        } else {
            load_tile<kT, T, DP, kKeyColumns>(sK, a.k, D, c.b, h, c.start + key0, keys_valid);
            load_tile<kT, T, DP, kKeyColumns>(sV, a.v, D, c.b, h, c.start + key0, keys_valid);
        }
        const int64_t slot = carry_slot32(c.slot_base, c.qt, 2 * kh + hf) * kTileQ;
        float W[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) W[r] = wrow + 8 * r < rows_valid ? cw[slot + 8 * r] : 0.f;
        rows_sync<kSums>();
        float s[1][4][4], dp[1][4][4], excl[2];
        if (kSums == kStaged) {
            values_scores<DP>(s, vQ + value_row<DP>(wrow), vK + (4 * hf + t) * kValueEight<DP>, D);
            values_scores<DP>(dp, vG + value_row<DP>(wrow), vV + (4 * hf + t) * kValueEight<DP>, D);
        } else if (kDirect) {
            const int key = key0 + 32 * hf + 8 * t, keys = keys_valid - 32 * hf - 8 * t;
            direct_scores<T>(s, row_of<T>(a.q, c, h, row0 + wrow), a.q.st, rows_valid - wrow, row_of<T>(a.k, c, h, key), a.k.st, keys, D);
            direct_scores<T>(dp, row_of<T>(a.d_o, c, h, row0 + wrow), a.d_o.st, rows_valid - wrow, row_of<T>(a.v, c, h, key), a.v.st, keys, D);
        } else {
            product_nt<kN, DP, 1, 4>(s, sQ + 16 * rg * kPitch<DP>, sK + 32 * hf * kPitch<DP>, D, lane);
            product_nt<kN, DP, 1, 4>(dp, sG + 16 * rg * kPitch<DP>, sV + 32 * hf * kPitch<DP>, D, lane);
        }
        const bool edge = kh == last || keys_valid < kBN;
        // right to left: s <- beta, dp <- g
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float beta[8], om[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) sigmoid_pair(s[0][j >> 1][2 * r + (j & 1)] * a.inv_temp, beta[j], om[j]);
            if (edge) {
                const int lim = min(keys_valid, row0 + wrow + 8 * r + a.attend_current - key0) - 32 * hf - 8 * t;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j >= lim) { beta[j] = 0.f; om[j] = 1.f; }
            }
            float incl = ((om[0] * om[1]) * (om[2] * om[3])) * ((om[4] * om[5]) * (om[6] * om[7]));
            incl = mul_right<kQuadRight>(incl, 1);
            incl = mul_right<kQuadRight>(incl, 2);
            const float y = __shfl_down_sync(0xffffffffu, incl, 1, 4);
            float run = W[r] * (t == 3 ? 1.f : y);
            float sum = 0.f;
#pragma unroll
            for (int j = 7; j >= 0; --j) {
                float& d = dp[0][j >> 1][2 * r + (j & 1)];
                d = beta[j] * run * (d - drem[r]);
                sum += d;
                run *= om[j];
                s[0][j >> 1][2 * r + (j & 1)] = beta[j];
            }
            float upto = add_left<kQuadLeft>(sum, 1);
            upto = add_left<kQuadLeft>(upto, 2);
            const float z = __shfl_up_sync(0xffffffffu, upto, 1, 4);
            excl[r] = t == 0 ? 0.f : z;
            if (t == 3) xs[hf][wrow + 8 * r] = upto;  // over the whole half
        }
        pair_sync(rg);
        // left to right: s <- ds = g - beta * (prefix of g including the key)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float right = xs[1][wrow + 8 * r], left = xs[0][wrow + 8 * r];
            const float base = hf ? prefix[r] + left : prefix[r];  // at the left edge of this half
            if (t == 0 && wrow + 8 * r < rows_valid) cc[slot + 8 * r] = base + (hf ? right : left);  // prefix through the half's right edge
            float cin = base + excl[r];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float gj = dp[0][j >> 1][2 * r + (j & 1)];
                float& sj = s[0][j >> 1][2 * r + (j & 1)];
                cin += gj;
                sj = gj - sj * cin;
            }
            prefix[r] = prefix[r] + left + right;
        }
        if (kEarly && kh < last) fetch(kh + 1);
        if (kSums == kStaged) values_px<DP>(o, s, vK + 4 * hf * kValueEight<DP>, keys_valid - 32 * hf, lane);
        else if (kDirect) direct_px<T, DP>(o, s, row_of<T>(a.k, c, h, key0 + 32 * hf), a.k.st, keys_valid - 32 * hf, D, lane);
        else product_px<kN, DP, DP, 1, 4>(o, s, sK + 32 * hf * kPitch<DP>, lane);
    }
    float* x = (float*)tiles;
    rows_sync<kSums>();
    if (hf == 1) {
#pragma unroll
        for (int n = 0; n < DP / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[((rg * (DP / 8) + n) * 4 + e) * 32 + lane] = o[0][n][e];
    }
    rows_sync<kSums>();
    bool again = false;
    if (hf == 0) {
#pragma unroll
        for (int n = 0; n < DP / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[0][n][e] += x[((rg * (DP / 8) + n) * 4 + e) * 32 + lane];
#pragma unroll
        for (int r = 0; r < 2; ++r) again |= wrow + 8 * r < rows_valid && asks_for_direct(o[0], 2 * r);
    }
    if (!kDirect && __syncthreads_or(again)) return true;
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    if (hf == 1) return false;
    const bool pairs = units_ok<T>(a.dq, D, 2);
    T* base = (T*)a.dq.ptr + (int64_t)c.b * a.dq.sb + (int64_t)h * a.dq.sh + (int64_t)(c.start + row0) * a.dq.st;
#pragma unroll
    for (int r = 0; r < 2; ++r)
        if (wrow + 8 * r < rows_valid) store_row<T, DP>(o[0], 2 * r, a.inv_temp, a.dq, pairs, D, 0, base, wrow + 8 * r, t);
    return false;
}
// ------------------------------------------------------------------------------------------ backward: dk, dv
// One query column of a block of transposed scores, keys 4 g ... 4 g + 3 of a quarter: s <- weights, dp <- ds.  W and cr enter at the
// quarter's right edge (product of 1 - beta to the right, sum of g through it); keys >= lim of the lane's four are not visible.
__device__ __forceinline__ void column(float* const (&s)[4], float* const (&dp)[4], float inv_temp, bool edge, int lim, float W, float cr, float drem, int g) {
    float beta[4], om[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) sigmoid_pair(*s[k] * inv_temp, beta[k], om[k]);
    if (edge) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k >= lim) { beta[k] = 0.f; om[k] = 1.f; }
    }
    float incl = (om[0] * om[1]) * (om[2] * om[3]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) incl = mul_right<kWarpRight>(incl, off);
    const float y = __shfl_down_sync(0xffffffffu, incl, 4);
    float run = W * (g == 7 ? 1.f : y);
    float gk[4];
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        const float p = beta[k] * run;
        run *= om[k];
        gk[k] = p * (*dp[k] - drem);
        *s[k] = p;
    }
    float from = (gk[0] + gk[1]) + (gk[2] + gk[3]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) from = add_right<kWarpRight>(from, off);
    const float z = __shfl_down_sync(0xffffffffu, from, 4);
    // inclusive prefix at a key = (prefix through the quarter's right edge) - (sum of g right of it)
    float cin = cr - (g == 7 ? 0.f : z);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        *dp[k] = gk[k] - beta[k] * cin;
        cin -= gk[k];
    }
}

}  // namespace

}  // namespace sb
