// fp32-arithmetic kernels (no tensor cores): forward, backward-dq and backward-dk/dv.
//
// They serve float32 inputs (where products must not be rounded to bf16/tf32), head dims other than 32, 64 and
// 128, and tensors whose strides the TMA path cannot take.  Structure mirrors the tensor-core kernels:
//   * forward walks the key tiles of one query block right to left and carries, per row, the running
//     product W = prod(1 - beta) of everything to the right (the reference carries its log,
//     stickbreaking_attention/sb_varlen/sb_varlen_fwd.py:53-66,155-193);
//   * the value of W at every 32-key boundary is saved ("carry_w") so that the backward can enter any tile
//     directly instead of subtracting from the row total as the reference does (sb_varlen_bwd.py:396-445);
//   * backward-dq walks left to right carrying the prefix sum of g = A * dA (sb_varlen_bwd.py:438-449) and saves
//     it at every boundary ("carry_c");
//   * backward-dk/dv keeps one 64-key tile stationary and walks the query blocks below it, entering each
//     tile with the two saved carries; dk and dv are accumulated in registers and stored once, so there is no
//     atomic or lock on the data (the reference uses a spin lock per key tile, sb_varlen_bwd.py:11-53).
//
// What bounds them is the FMA pipes (128 per clock and SM), so everything else is kept out of their way: a thread owns a
// register tile of 4 rows x 4 columns of every product in packed fp32x2 multiply-adds, operands come from shared memory in 16-byte
// pieces, scores never leave the registers (the 16 lanes of a row exchange their products and sums by shuffles), and only
// the weights pass through shared memory on their way into the second product.  us per kernel, forward / dq / dk,dv, with scalar
// loads and the scores in shared memory -> now (tiles of 8 x 4 need a quarter fewer instructions but leave 8 to 12 warps per SM,
// too few to hide their latencies: 255 / 378 / 388 in the first line):
//   8 heads, 4096 float32 tokens in 4 sequences, head dim 64:   642 / 825 / 1028 -> 201 / 297 / 363
//   4 x 8 heads x 500 tokens, bf16, head dim 50:                186 / 235 / 280  ->  76 / 106 / 119
//   4 heads, 512 float32 tokens, head dim 64:                    53 / 72 / 82    ->  27 / 37 / 31
#include "sb_common.cuh"

namespace sb {

namespace {

constexpr int kBN = 64;         // keys per tile (and query rows per tile of the dk/dv kernel)

// An operand tile in shared memory, transposed: [DP][kW] floats, element (row, d) in row d of the tile.  The 16-byte pieces of
// a row are permuted by a function of d so that neither the transposing stores (lanes along d) nor the loads (lanes along the
// piece index, or along d with a fixed piece) pile up on a bank: (d ^ d / 4) is a permutation of 0 ... 15 both over
// 16 consecutive d and over 16 d that are 4 apart.
template <int kW>
__device__ __forceinline__ int piece(int d, int c) {
    return d * kW + (((c ^ d ^ (d >> 2)) & (kW / 4 - 1)) << 2);
}

// kU consecutive elements as float32
template <typename T, int kU>
__device__ __forceinline__ void load_unit(const T* src, float (&x)[kU]) {
    if constexpr (sizeof(T) == 4) {
        if constexpr (kU == 4) {
            const float4 v = *(const float4*)src;
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else if constexpr (kU == 2) {
            const float2 v = *(const float2*)src;
            x[0] = v.x; x[1] = v.y;
        } else {
            x[0] = to_f32<T>(*src);
        }
    } else {
        T v[kU];
        if constexpr (kU == 4) *(uint2*)v = *(const uint2*)src;
        else if constexpr (kU == 2) *(uint32_t*)v = *(const uint32_t*)src;
        else v[0] = *src;
#pragma unroll
        for (int i = 0; i < kU; ++i) x[i] = to_f32<T>(v[i]);
    }
}
// whether rows can be read in units of u elements
template <typename T>
__device__ __forceinline__ bool units_ok(const MatView& m, int D, int u) {
    return ((D | m.st | m.sh | m.sb) & (u - 1)) == 0 && ((uintptr_t)m.ptr & (u * sizeof(T) - 1)) == 0;
}

// kRows rows of a [.., T, D] tensor into a transposed tile (see piece) as float32, zeros behind the valid rows and columns.
// A thread keeps its columns and walks the rows, several loads in flight.
template <int kT, typename T, int DP, int kRows, int kU>
__device__ __forceinline__ void load_tile_u(float* dst, const T* base, int64_t st, int D, int rows_valid) {
    constexpr int kPer = DP / kU;                   // threads per row
    constexpr int kStep = kT / kPer;                // rows per pass
    constexpr int kN = kRows / kStep > 0 ? kRows / kStep : 1;
    constexpr int kMax = 32 / kU < 8 ? 8 : 32 / kU, kBatch = kN < kMax ? kN : kMax;
    const int d = kU * ((int)threadIdx.x % kPer), r0 = (int)threadIdx.x / kPer;
    const T* src = base + r0 * st + d;
    const bool col_ok = d < D;
#pragma unroll 1
    for (int i0 = 0; i0 < kN; i0 += kBatch) {
        float x[kBatch][kU];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int r = r0 + (i0 + i) * kStep;
#pragma unroll
            for (int u = 0; u < kU; ++u) x[i][u] = 0.f;
            if (col_ok && r < rows_valid) load_unit<T, kU>(src + (int64_t)(i0 + i) * kStep * st, x[i]);
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
            const int r = r0 + (i0 + i) * kStep;
            if (kRows < kStep && r >= kRows) continue;
#pragma unroll
            for (int u = 0; u < kU; ++u) dst[piece<kRows>(d + u, r >> 2) + (r & 3)] = x[i][u];
        }
    }
}
template <int kT, typename T, int DP, int kRows>
__device__ __forceinline__ void load_tile(float* dst, const MatView& m, int D, int b, int h, int row0, int rows_valid) {
    const T* base = (const T*)m.ptr + (int64_t)b * m.sb + (int64_t)h * m.sh + (int64_t)row0 * m.st;
    if (units_ok<T>(m, D, 4)) load_tile_u<kT, T, DP, kRows, 4>(dst, base, m.st, D, rows_valid);
    else if (units_ok<T>(m, D, 2)) load_tile_u<kT, T, DP, kRows, 2>(dst, base, m.st, D, rows_valid);
    else load_tile_u<kT, T, DP, kRows, 1>(dst, base, m.st, D, rows_valid);
}

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }

// column of the head dim that accumulator column c of lane group tx stands for
template <int DP>
__device__ __forceinline__ int col_of(int c, int tx) {
    return DP >= 64 ? (c >> 2) * 64 + 4 * tx + (c & 3) : (DP / 16) * tx + c;
}

// s[rows of ty x kJ keys of tx] = A (kR rows per thread, tile width kWA) * B^T (16 * kJ keys), both transposed tiles
template <int kR, int kWA, int kJ>
__device__ __forceinline__ void product_nt(float2 (&s)[kR / 2][kJ], const float* A, const float* B, int ty, int tx, int D) {
#pragma unroll
    for (int i = 0; i < kR / 2; ++i)
#pragma unroll
        for (int j = 0; j < kJ; ++j) s[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int d = 0; d < D; ++d) {
        float4 x[kR / 4];
#pragma unroll
        for (int i = 0; i < kR / 4; ++i) x[i] = *(const float4*)(A + piece<kWA>(d, ty * (kR / 4) + i));
        float2 kk[kJ];
        if constexpr (kJ == 4) {
            const float4 k = *(const float4*)(B + piece<64>(d, tx));
            kk[0] = dup(k.x); kk[1] = dup(k.y); kk[2] = dup(k.z); kk[3] = dup(k.w);
        } else {
            const float2 k = *(const float2*)(B + piece<32>(d, tx >> 1) + 2 * (tx & 1));
            kk[0] = dup(k.x); kk[1] = dup(k.y);
        }
#pragma unroll
        for (int i = 0; i < kR / 4; ++i)
#pragma unroll
            for (int j = 0; j < kJ; ++j) {
                s[2 * i][j] = __ffma2_rn(make_float2(x[i].x, x[i].y), kk[j], s[2 * i][j]);
                s[2 * i + 1][j] = __ffma2_rn(make_float2(x[i].z, x[i].w), kk[j], s[2 * i + 1][j]);
            }
    }
}

// acc[kR rows x DP/16 columns] += P * X: P in shared memory with the contracted index along its rows (row j: 16-byte pieces of
// rows, permuted by kSwz ? j / 4 : 0), X a transposed tile [d][contracted index]; four contracted indices at a time
template <int DP, int kR, int kWP, bool kSwz>
__device__ __forceinline__ void product_px(float2 (&acc)[kR / 2][DP / 16], const float* P, const float* X, int ty, int tx) {
    constexpr int kNC = DP / 16;
#pragma unroll 2
    for (int j4 = 0; j4 < 16; ++j4) {
        float4 x[kNC];
#pragma unroll
        for (int c = 0; c < kNC; ++c) x[c] = *(const float4*)(X + piece<64>(col_of<DP>(c, tx), j4));
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
            float2 p[kR / 2];
            if constexpr (kR == 2) {
                p[0] = *(const float2*)(P + (4 * j4 + jj) * kWP + 2 * ty);
            } else {
#pragma unroll
                for (int i = 0; i < kR / 4; ++i) {
                    const int c = ty * (kR / 4) + i;
                    const float4 q = *(const float4*)(P + (4 * j4 + jj) * kWP + ((kSwz ? ((c ^ j4) & (kWP / 4 - 1)) : c) << 2));
                    p[2 * i] = make_float2(q.x, q.y);
                    p[2 * i + 1] = make_float2(q.z, q.w);
                }
            }
#pragma unroll
            for (int c = 0; c < kNC; ++c) {
                const float2 xx = dup(jj == 0 ? x[c].x : jj == 1 ? x[c].y : jj == 2 ? x[c].z : x[c].w);
#pragma unroll
                for (int i = 0; i < kR / 2; ++i) acc[i][c] = __ffma2_rn(p[i], xx, acc[i][c]);
            }
        }
    }
}

// four keys of kR rows into the [key][row] tile that product_px<kSwz> reads
template <int kR, int kW>
__device__ __forceinline__ void put_weights(float* P, const float2 (&p)[kR / 2][4], int ty, int tx) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < kR / 4; ++i)
            *(float4*)(P + (4 * tx + j) * kW + (((ty * (kR / 4) + i) ^ tx) & (kW / 4 - 1)) * 4) =
                make_float4(p[2 * i][j].x, p[2 * i][j].y, p[2 * i + 1][j].x, p[2 * i + 1][j].y);
}

template <typename T, int DP, int kR>
__device__ __forceinline__ void store_acc(const float2 (&acc)[kR / 2][DP / 16], float scale, const MatView& m, int D, int b, int h, int row0,
                                          int rows_valid, int ty, int tx) {
    constexpr int kNC = DP / 16;
    T* base = (T*)m.ptr + (int64_t)b * m.sb + (int64_t)h * m.sh + (int64_t)row0 * m.st;
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        const int row = ty * kR + r;
        if (row >= rows_valid) continue;
#pragma unroll
        for (int c = 0; c < kNC; ++c) {
            const int d = col_of<DP>(c, tx);
            const float x = (r & 1) ? acc[r >> 1][c].y : acc[r >> 1][c].x;
            if (d < D) base[(int64_t)row * m.st + d] = from_f32<T>(x * scale);
        }
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

// A row's 64 keys lie in 16 consecutive lanes, four each.  Inclusive product (sum) over this lane and those to its right (left).
__device__ __forceinline__ float right_prod(float x, int tx) {
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
        const float y = __shfl_down_sync(0xffffffffu, x, off, 16);
        x *= tx + off < 16 ? y : 1.f;
    }
    return x;
}
__device__ __forceinline__ float right_sum(float x, int tx) {
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
        const float y = __shfl_down_sync(0xffffffffu, x, off, 16);
        x += tx + off < 16 ? y : 0.f;
    }
    return x;
}
__device__ __forceinline__ float left_sum(float x, int tx) {
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, x, off, 16);
        x += tx >= off ? y : 0.f;
    }
    return x;
}

__device__ __forceinline__ float& pick(float2& v, int odd) { return odd ? v.y : v.x; }

struct ItemCtx {
    int seq, qt, b, start, len, slot_base;
};
__device__ inline bool fetch_item(const KArgs& a, int item, ItemCtx& c) {
    if (item >= a.hdr->n_items) return false;
    const int2 it = a.items[item];
    const SeqInfo s = a.seqs[it.x];
    c.seq = it.x; c.qt = it.y; c.b = s.batch; c.start = s.start; c.len = s.len; c.slot_base = s.slot_base;
    return true;
}

// Blocks in the order of the item table (heaviest first), the heads and the parts of a 128-row tile innermost: the hardware
// deals blocks out in this order, so the heavy ones of all heads start first.
struct BlockIdx {
    int item, h, part;
};
__device__ __forceinline__ BlockIdx block_idx(int heads, int parts) {
    const int per = heads * parts, item = (int)blockIdx.x / per, rest = (int)blockIdx.x - item * per;
    return BlockIdx{item, rest / parts, rest % parts};
}
__device__ __forceinline__ int64_t linear_thread() { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int64_t all_threads() { return (int64_t)gridDim.x * blockDim.x; }

// ------------------------------------------------------------------------------------------ forward
// kT / 16 groups of 4 query rows: blocks of 64 rows, or 32 where the problem is small (the host chooses)
template <typename T, int DP, int kT>
__global__ void __launch_bounds__(kT, DP > 64 ? 1 : kT > 128 ? 2 : 4) simt_fwd_kernel(const __grid_constant__ KArgs a) {
    constexpr int kR = 4, kBM = kT / 16 * kR;
    extern __shared__ __align__(16) float smem[];
    float* Qt = smem;             // [DP][kBM]
    float* Kt = Qt + DP * kBM;    // [DP][64]
    float* Vt = Kt + DP * kBN;    // [DP][64]
    float* Ps = Vt + DP * kBN;    // [64 keys][kBM]
    pdl_wait();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) zero_tail_rows<T>(a, a.hdr->covered_end, linear_thread(), all_threads());
    ItemCtx c;
    const BlockIdx bi = block_idx(a.heads, kTileQ / kBM);
    if (!fetch_item(a, bi.item, c)) return;
    const int h = bi.h, D = a.head_dim;
    const int sub = bi.part * kBM;  // first row inside the 128-row tile
    const int row0 = c.qt * kTileQ + sub;
    if (row0 >= c.len) return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int rows_valid = min(kBM, c.len - row0);
    load_tile<kT, T, DP, kBM>(Qt, a.q, D, c.b, h, c.start + row0, rows_valid);
    float W[kR];
    float2 o[kR / 2][DP / 16];
#pragma unroll
    for (int r = 0; r < kR; ++r) W[r] = 1.f;
#pragma unroll
    for (int i = 0; i < kR / 2; ++i)
#pragma unroll
        for (int j = 0; j < DP / 16; ++j) o[i][j] = make_float2(0.f, 0.f);
    float* cw = a.carry_w ? a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ + sub + ty * kR : nullptr;
    const int last = (min(row0 + kBM, c.len) - 1) / kBN;
    // key tiles of the 128-key diagonal tile that lie right of these rows: a tensor-core backward may follow, and it reads the
    // carry of every quarter of its tile
    if (cw && tx == 0)
        for (int kh = last + 1; kh <= 2 * c.qt + 1 && kh * kBN < c.len; ++kh)
#pragma unroll
            for (int r = 0; r < kR; ++r) {
                cw[carry_slot(c.slot_base, c.qt, kh) * kTileQ + r] = 1.f;
                cw[carry_slot32(c.slot_base, c.qt, 2 * kh) * kTileQ + r] = 1.f;
            }

    for (int kh = last; kh >= 0; --kh) {
        const int key0 = kh * kBN;
        const int keys_valid = min(kBN, c.len - key0);
        __syncthreads();
        load_tile<kT, T, DP, kBN>(Kt, a.k, D, c.b, h, c.start + key0, keys_valid);
        load_tile<kT, T, DP, kBN>(Vt, a.v, D, c.b, h, c.start + key0, keys_valid);
        __syncthreads();
        float2 s[kR / 2][4];
        product_nt<kR, kBM>(s, Qt, Kt, ty, tx, D);
        const bool edge = key0 + kBN > row0 || keys_valid < kBN;  // some pair of the tile is not visible
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int lim = edge ? min(keys_valid, row0 + ty * kR + r + a.attend_current - key0) : kBN;  // keys < lim are visible
            float beta[4], om[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sigmoid_pair(pick(s[r >> 1][j], r & 1) * a.inv_temp, beta[j], om[j]);
                if (4 * tx + j >= lim) { beta[j] = 0.f; om[j] = 1.f; }
            }
            const float incl = right_prod((om[0] * om[1]) * (om[2] * om[3]), tx);
            float right = __shfl_down_sync(0xffffffffu, incl, 1, 16);
            if (tx == 15) right = 1.f;
            float run = W[r] * right;
            if (cw) {  // W at the right edges of the two 32-key quarters
                if (tx == 15) cw[carry_slot(c.slot_base, c.qt, kh) * kTileQ + r] = run;
                if (tx == 7) cw[carry_slot32(c.slot_base, c.qt, 2 * kh) * kTileQ + r] = run;
            }
            W[r] *= __shfl_sync(0xffffffffu, incl, 0, 16);
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                pick(s[r >> 1][j], r & 1) = beta[j] * run;
                run *= om[j];
            }
        }
        put_weights<kR, kBM>(Ps, s, ty, tx);
        __syncthreads();
        product_px<DP, kR, kBM, true>(o, Ps, Vt, ty, tx);
    }
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    store_acc<T, DP, kR>(o, 1.f, a.o, D, c.b, h, c.start + row0, rows_valid, ty, tx);
    if (tx == 0) {
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            if (ty * kR + r >= rows_valid) continue;
            const int64_t t = c.start + row0 + ty * kR + r;
            ((T*)a.rem.ptr)[(int64_t)c.b * a.rem.sb + (int64_t)h * a.rem.sh + t * a.rem.st] = from_f32<T>(W[r]);
            ((float*)a.nla.ptr)[(int64_t)c.b * a.nla.sb + (int64_t)h * a.nla.sh + t * a.nla.st] = log2f(W[r]);
        }
    }
}

// ------------------------------------------------------------------------------------------ backward: dq
template <typename T, int DP, int kT>
__global__ void __launch_bounds__(kT, DP > 64 ? 1 : kT > 128 ? 2 : 3) simt_bwd_dq_kernel(const __grid_constant__ KArgs a) {
    constexpr int kR = 4, kBM = kT / 16 * kR;
    constexpr bool kShare = DP >= kBM;  // dS takes the place of V, which is done with
    extern __shared__ __align__(16) float smem[];
    float* Qt = smem;
    float* Gt = Qt + DP * kBM;  // dO
    float* Kt = Gt + DP * kBM;
    float* Vt = Kt + DP * kBN;
    float* Ss = kShare ? Vt : Vt + DP * kBN;  // dS, [64 keys][kBM]
    pdl_wait();
    if (a.zero_tail && a.hdr->covered_end < a.tokens) zero_tail_grads<T>(a, a.hdr->covered_end, linear_thread(), all_threads());
    ItemCtx c;
    const BlockIdx bi = block_idx(a.heads, kTileQ / kBM);
    if (!fetch_item(a, bi.item, c)) return;
    const int h = bi.h, D = a.head_dim;
    const int sub = bi.part * kBM;
    const int row0 = c.qt * kTileQ + sub;
    if (row0 >= c.len) return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int rows_valid = min(kBM, c.len - row0);
    load_tile<kT, T, DP, kBM>(Qt, a.q, D, c.b, h, c.start + row0, rows_valid);
    load_tile<kT, T, DP, kBM>(Gt, a.d_o, D, c.b, h, c.start + row0, rows_valid);
    float drem[kR], prefix[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
        const int64_t t = c.start + row0 + ty * kR + r;
        drem[r] = ty * kR + r < rows_valid ? to_f32<T>(((const T*)a.d_rem.ptr)[(int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + t * a.d_rem.st]) : 0.f;
        prefix[r] = 0.f;  // sum of g over all keys left of the current tile
    }
    const float* cw = a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ + sub + ty * kR;
    float* cc = a.carry_c + ((int64_t)h * a.slot_cap) * kTileQ + sub + ty * kR;
    float2 o[kR / 2][DP / 16];
#pragma unroll
    for (int i = 0; i < kR / 2; ++i)
#pragma unroll
        for (int j = 0; j < DP / 16; ++j) o[i][j] = make_float2(0.f, 0.f);
    const int last = (min(row0 + kBM, c.len) - 1) / kBN;

    for (int kh = 0; kh <= last; ++kh) {
        const int key0 = kh * kBN;
        const int keys_valid = min(kBN, c.len - key0);
        __syncthreads();
        load_tile<kT, T, DP, kBN>(Kt, a.k, D, c.b, h, c.start + key0, keys_valid);
        load_tile<kT, T, DP, kBN>(Vt, a.v, D, c.b, h, c.start + key0, keys_valid);
        const int64_t slot = carry_slot(c.slot_base, c.qt, kh) * kTileQ;
        float Win[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) Win[r] = ty * kR + r < rows_valid ? cw[slot + r] : 0.f;
        __syncthreads();
        float2 s[kR / 2][4], dp[kR / 2][4];
        product_nt<kR, kBM>(s, Qt, Kt, ty, tx, D);
        product_nt<kR, kBM>(dp, Gt, Vt, ty, tx, D);
        const bool edge = key0 + kBN > row0 || keys_valid < kBN;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int lim = edge ? min(keys_valid, row0 + ty * kR + r + a.attend_current - key0) : kBN;
            float beta[4], om[4], g[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                sigmoid_pair(pick(s[r >> 1][j], r & 1) * a.inv_temp, beta[j], om[j]);
                if (4 * tx + j >= lim) { beta[j] = 0.f; om[j] = 1.f; }
            }
            const float incl = right_prod((om[0] * om[1]) * (om[2] * om[3]), tx);
            float right = __shfl_down_sync(0xffffffffu, incl, 1, 16);
            if (tx == 15) right = 1.f;
            float run = Win[r] * right;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                g[j] = beta[j] * run * (pick(dp[r >> 1][j], r & 1) - drem[r]);
                run *= om[j];
            }
            const float mine = (g[0] + g[1]) + (g[2] + g[3]);
            const float upto = left_sum(mine, tx);  // through this lane's keys
            float cin = prefix[r] + (upto - mine);
            prefix[r] += __shfl_sync(0xffffffffu, upto, 15, 16);
            if (ty * kR + r < rows_valid) {  // prefixes through the right edges of the two 32-key quarters
                if (tx == 15) cc[slot + r] = prefix[r];
                if (tx == 7) cc[slot - kTileQ + r] = cin + mine;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                cin += g[j];
                pick(s[r >> 1][j], r & 1) = g[j] - beta[j] * cin;
            }
        }
        if (kShare) __syncthreads();  // everybody has read V
        put_weights<kR, kBM>(Ss, s, ty, tx);
        __syncthreads();
        product_px<DP, kR, kBM, true>(o, Ss, Kt, ty, tx);
    }
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    store_acc<T, DP, kR>(o, a.inv_temp, a.dq, D, c.b, h, c.start + row0, rows_valid, ty, tx);
}

// ------------------------------------------------------------------------------------------ backward: dk, dv
// kJ keys per lane: stationary tiles of 16 * kJ keys (64, or 32 for small problems)
template <typename T, int DP, int kJ>
__global__ void __launch_bounds__(256, DP > 64 ? 1 : 2) simt_bwd_dkdv_kernel(const __grid_constant__ KArgs a) {
    constexpr int kT = 256, kR = 4, kBM = 64, kKeys = 16 * kJ, kRK = kKeys / 16;
    extern __shared__ __align__(16) float smem[];
    float* Qt = smem;
    float* Gt = Qt + DP * kBM;
    float* Kt = Gt + DP * kBM;
    float* Vt = Kt + DP * kKeys;
    float* Ps = Vt + DP * kKeys;   // P, [64 queries][kKeys]
    float* Ss = Ps + kBM * kKeys;  // dS
    pdl_wait();
    ItemCtx c;
    const int n_items = a.hdr->n_items;
    const BlockIdx bi = block_idx(a.heads, kTileQ / kKeys);
    if (bi.item >= n_items) return;
    // the table is heaviest-first for query tiles; key tiles are heaviest at the other end
    if (!fetch_item(a, n_items - 1 - bi.item, c)) return;
    const int h = bi.h, D = a.head_dim;
    const int key0 = c.qt * kTileQ + bi.part * kKeys;
    const int edge_slot = key0 / 32 + kKeys / 32 - 1;  // the 32-key quarter at the tile's right edge
    if (key0 >= c.len) return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int keys_valid = min(kKeys, c.len - key0);
    load_tile<kT, T, DP, kKeys>(Kt, a.k, D, c.b, h, c.start + key0, keys_valid);
    load_tile<kT, T, DP, kKeys>(Vt, a.v, D, c.b, h, c.start + key0, keys_valid);
    const float* cw = a.carry_w + ((int64_t)h * a.slot_cap) * kTileQ;
    const float* cc = a.carry_c + ((int64_t)h * a.slot_cap) * kTileQ;
    float2 ok[kRK / 2][DP / 16], ov[kRK / 2][DP / 16];
#pragma unroll
    for (int i = 0; i < kRK / 2; ++i)
#pragma unroll
        for (int j = 0; j < DP / 16; ++j) ok[i][j] = ov[i][j] = make_float2(0.f, 0.f);
    const int n_qb = (c.len + kBM - 1) / kBM;

    for (int qb = key0 / kBM; qb < n_qb; ++qb) {
        const int row0 = qb * kBM;
        const int rows_valid = min(kBM, c.len - row0);
        __syncthreads();
        load_tile<kT, T, DP, kBM>(Qt, a.q, D, c.b, h, c.start + row0, rows_valid);
        load_tile<kT, T, DP, kBM>(Gt, a.d_o, D, c.b, h, c.start + row0, rows_valid);
        const int64_t slot = carry_slot32(c.slot_base, qb >> 1, edge_slot) * kTileQ + (qb & 1) * kBM + ty * kR;
        float Win[kR], cright[kR], drem[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const bool row_ok = ty * kR + r < rows_valid;
            const int64_t t = c.start + row0 + ty * kR + r;
            Win[r] = row_ok ? cw[slot + r] : 0.f;
            cright[r] = row_ok ? cc[slot + r] : 0.f;
            drem[r] = row_ok ? to_f32<T>(((const T*)a.d_rem.ptr)[(int64_t)c.b * a.d_rem.sb + (int64_t)h * a.d_rem.sh + t * a.d_rem.st]) : 0.f;
        }
        __syncthreads();
        float2 s[kR / 2][kJ], dp[kR / 2][kJ];
        product_nt<kR, kBM>(s, Qt, Kt, ty, tx, D);
        product_nt<kR, kBM>(dp, Gt, Vt, ty, tx, D);
        const bool edge = qb == key0 / kBM || keys_valid < kKeys;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int lim = edge ? min(keys_valid, row0 + ty * kR + r + a.attend_current - key0) : kKeys;
            float beta[kJ], om[kJ], g[kJ], p[kJ];
#pragma unroll
            for (int j = 0; j < kJ; ++j) {
                sigmoid_pair(pick(s[r >> 1][j], r & 1) * a.inv_temp, beta[j], om[j]);
                if (kJ * tx + j >= lim) { beta[j] = 0.f; om[j] = 1.f; }
            }
            const float incl = right_prod(kJ == 4 ? (om[0] * om[1]) * (om[kJ - 2] * om[kJ - 1]) : om[0] * om[1], tx);
            float right = __shfl_down_sync(0xffffffffu, incl, 1, 16);
            if (tx == 15) right = 1.f;
            float run = Win[r] * right;
#pragma unroll
            for (int j = kJ - 1; j >= 0; --j) {
                p[j] = beta[j] * run;
                g[j] = p[j] * (pick(dp[r >> 1][j], r & 1) - drem[r]);
                run *= om[j];
            }
            const float from = right_sum(kJ == 4 ? (g[0] + g[1]) + (g[kJ - 2] + g[kJ - 1]) : g[0] + g[1], tx);
            float behind = __shfl_down_sync(0xffffffffu, from, 1, 16);  // sum of g right of this lane's keys
            if (tx == 15) behind = 0.f;
            // inclusive prefix at key j = (prefix through the tile's right edge) - (sum of g right of j)
            float cin = cright[r] - behind;
#pragma unroll
            for (int j = kJ - 1; j >= 0; --j) {
                pick(s[r >> 1][j], r & 1) = p[j];
                pick(dp[r >> 1][j], r & 1) = g[j] - beta[j] * cin;
                cin -= g[j];
            }
        }
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int q = ty * kR + r;
            if constexpr (kJ == 4) {
                *(float4*)(Ps + q * kKeys + 4 * tx) = make_float4(pick(s[r >> 1][0], r & 1), pick(s[r >> 1][1], r & 1), pick(s[r >> 1][2], r & 1), pick(s[r >> 1][3], r & 1));
                *(float4*)(Ss + q * kKeys + 4 * tx) = make_float4(pick(dp[r >> 1][0], r & 1), pick(dp[r >> 1][1], r & 1), pick(dp[r >> 1][2], r & 1), pick(dp[r >> 1][3], r & 1));
            } else {
                *(float2*)(Ps + q * kKeys + 2 * tx) = make_float2(pick(s[r >> 1][0], r & 1), pick(s[r >> 1][1], r & 1));
                *(float2*)(Ss + q * kKeys + 2 * tx) = make_float2(pick(dp[r >> 1][0], r & 1), pick(dp[r >> 1][1], r & 1));
            }
        }
        __syncthreads();
        product_px<DP, kRK, kKeys, false>(ov, Ps, Gt, ty, tx);
        product_px<DP, kRK, kKeys, false>(ok, Ss, Qt, ty, tx);
    }
    pdl_launch_dependents();  // not earlier: waiting blocks would take the places of this kernel's own and spread unevenly
    store_acc<T, DP, kRK>(ok, a.inv_temp, a.dk, D, c.b, h, c.start + key0, keys_valid, ty, tx);
    store_acc<T, DP, kRK>(ov, 1.f, a.dv, D, c.b, h, c.start + key0, keys_valid, ty, tx);
}

// Blocks of 32 query rows (key tiles of 32) where 64-row ones, `items * heads * 2` at most, would not give every SM one: half the
// work per block, at the price of loading every key (query) tile for half as many rows.  float32, 4 heads, 512 tokens: 96.7 -> 88
// us per step; from two blocks per SM on, 64 rows are faster in each kernel (below: 76 / 106 / 119 against 90 / 114 / 132).
bool small_problem(const WsLayout& L, const KArgs& a) { return (int64_t)L.max_items * a.heads * 2 <= 148; }

template <typename T, int DP, int kT>
int launch_fwd_k(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    constexpr int kBM = kT / 4;
    const int smem = (int)sizeof(float) * (DP * kBM + 2 * DP * kBN + kBN * kBM);
    const auto kernel = simt_fwd_kernel<T, DP, kT>;
    const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
    if (e != 0) return e;
    return launch_kernel(kernel, dim3((unsigned)L.max_items * a.heads * (kTileQ / kBM)), dim3(kT), smem, st, a);
}
template <typename T, int DP, int kT>
int launch_dq_k(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    constexpr int kBM = kT / 4;
    const int smem = (int)sizeof(float) * (2 * DP * kBM + 2 * DP * kBN + (DP >= kBM ? 0 : kBN * kBM));
    const auto kernel = simt_bwd_dq_kernel<T, DP, kT>;
    const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
    if (e != 0) return e;
    return launch_kernel(kernel, dim3((unsigned)L.max_items * a.heads * (kTileQ / kBM)), dim3(kT), smem, st, a);
}
template <typename T, int DP, int kJ>
int launch_dkdv_k(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    const int smem = (int)sizeof(float) * (2 * DP * (64 + 16 * kJ) + 2 * 64 * 16 * kJ);
    const auto kernel = simt_bwd_dkdv_kernel<T, DP, kJ>;
    const int e = ensure_kernel_attrs((const void*)kernel, smem, true);
    if (e != 0) return e;
    return launch_kernel(kernel, dim3((unsigned)L.max_items * a.heads * (8 / kJ)), dim3(256), smem, st, a);
}

template <typename T, int DP>
int launch_fwd_d(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    return small_problem(L, a) ? launch_fwd_k<T, DP, 128>(L, a, st) : launch_fwd_k<T, DP, 256>(L, a, st);
}
template <typename T, int DP>
int launch_bwd_d(const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    if (phases != SBATTN_BWD_DKDV) {
        const int e = small_problem(L, a) ? launch_dq_k<T, DP, 128>(L, a, st) : launch_dq_k<T, DP, 256>(L, a, st);
        if (e != 0) return e;
    }
    if (phases == SBATTN_BWD_DQ) return 0;
    return small_problem(L, a) ? launch_dkdv_k<T, DP, 2>(L, a, st) : launch_dkdv_k<T, DP, 4>(L, a, st);
}

template <typename T>
int launch_fwd_t(const WsLayout& L, const KArgs& a, cudaStream_t st) {
    if (a.head_dim > 64) return launch_fwd_d<T, 128>(L, a, st);
    if (a.head_dim > 32) return launch_fwd_d<T, 64>(L, a, st);
    return a.head_dim > 16 ? launch_fwd_d<T, 32>(L, a, st) : launch_fwd_d<T, 16>(L, a, st);
}
template <typename T>
int launch_bwd_t(const WsLayout& L, const KArgs& a, int phases, cudaStream_t st) {
    if (a.head_dim > 64) return launch_bwd_d<T, 128>(L, a, phases, st);
    if (a.head_dim > 32) return launch_bwd_d<T, 64>(L, a, phases, st);
    return a.head_dim > 16 ? launch_bwd_d<T, 32>(L, a, phases, st) : launch_bwd_d<T, 16>(L, a, phases, st);
}

}  // namespace

int launch_simt_fwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    if (L.max_items <= 0) return 0;
    switch (p.dtype) {
        case SBATTN_BF16: return launch_fwd_t<__nv_bfloat16>(L, a, st);
        case SBATTN_F16: return launch_fwd_t<__half>(L, a, st);
        default: return launch_fwd_t<float>(L, a, st);
    }
}

int launch_simt_bwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st) {
    if (L.max_items <= 0) return 0;
    switch (p.dtype) {
        case SBATTN_BF16: return launch_bwd_t<__nv_bfloat16>(L, a, p.bwd_phases, st);
        case SBATTN_F16: return launch_bwd_t<__half>(L, a, p.bwd_phases, st);
        default: return launch_bwd_t<float>(L, a, p.bwd_phases, st);
    }
}

}  // namespace sb
