// Prep kernel: turns the sequence ends on the device into the tables every attention kernel walks -- one
// SeqInfo per sequence and the list of (sequence, 128-row tile) work items ordered heaviest first (a tile's
// cost is the number of key tiles to its left, i.e. its index inside the sequence + 1).  Runs as a single
// thread block on the caller's stream, so no host synchronisation is needed to learn the sequence lengths.
//
// Reference counterpart: the grid computation of varlen_fwd (stickbreaking_attention/sb_varlen/sb_varlen_fwd.py
// :476-479), which sizes the grid by max_seqlens and lets programs of short sequences exit early, and the
// per-program lookup of the sequence bounds (:283-288).
#include "sb_common.cuh"

namespace sb {

namespace {

constexpr int kPrepThreads = 1024;

__device__ inline int64_t read_end(const void* cu, int width, int i) {
    return width == 8 ? ((const int64_t*)cu)[i] : (int64_t)((const int32_t*)cu)[i];
}

// Inclusive block scan of two ints per thread (warp shuffles, then one warp over the warps' totals); the totals of the block
// come back in tot_a, tot_b.  `sh` holds 2 x 33 ints.
__device__ inline void block_scan2(int& a, int& b, int (*sh)[33], int& tot_a, int& tot_b) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int va = __shfl_up_sync(0xffffffffu, a, off), vb = __shfl_up_sync(0xffffffffu, b, off);
        if (lane >= off) { a += va; b += vb; }
    }
    __syncthreads();  // the previous scan's totals have been read
    if (lane == 31) { sh[0][warp] = a; sh[1][warp] = b; }
    __syncthreads();
    if (warp == 0) {
        int x = sh[0][lane], y = sh[1][lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int vx = __shfl_up_sync(0xffffffffu, x, off), vy = __shfl_up_sync(0xffffffffu, y, off);
            if (lane >= off) { x += vx; y += vy; }
        }
        sh[0][lane] = x;
        sh[1][lane] = y;
    }
    __syncthreads();
    tot_a = sh[0][31];
    tot_b = sh[1][31];
    if (warp > 0) { a += sh[0][warp - 1]; b += sh[1][warp - 1]; }
}

// One block.  What bounds it is latency: the launch, the read of the ends, two block scans, the writes of the tables.  The
// per-class counters live in shared memory where they fit (up to kSharedBins tiles in the longest sequence, else in the
// workspace), the counts per class are scans instead of serial loops, and the items of a sequence are written by a group of up to
// 32 lanes.  With one thread per sequence and one for the classes the kernel took 31 us for one sequence of 8192 tokens and 19 us
// for four of 1000 ... 3000.
constexpr int kSharedBins = 4096;

__global__ void __launch_bounds__(kPrepThreads, 1)
prep_kernel(WsHeader* hdr, SeqInfo* seqs, int2* items, int32_t* bins, const void* cu, int cu_width, int n_seqs,
            int batch, int tokens, int max_len, int n_max, int max_items, int64_t slot_cap, uint32_t* status) {
    __shared__ int sh[2][33];
    __shared__ int sh_bad;
    __shared__ int sh_bins[kSharedBins + 2];
    const int t = threadIdx.x;
    int* cursor = n_max <= kSharedBins ? sh_bins : bins;  // [n_max+2]: sequences per tile count, then write position per cost class
    if (t == 0) sh_bad = 0;
    pdl_wait();  // before anything is written to the workspace, whose memory an earlier kernel may still be reading
    pdl_launch_dependents();
    for (int i = t; i < n_max + 2; i += kPrepThreads) cursor[i] = 0;
    if (t < 8) hdr->sched[t] = 0;
    __syncthreads();

    // pass 1: sequence table, running offsets
    int item_carry = 0, slot_carry = 0;
    for (int base = 0; base < n_seqs; base += kPrepThreads) {
        const int s = base + t;
        int len = 0, start = 0, b = 0, bad = 0;
        if (s < n_seqs) {
            if (batch > 0) {
                b = s; start = 0; len = tokens;
            } else {
                const int64_t e1 = read_end(cu, cu_width, s);
                const int64_t e0 = s > 0 ? read_end(cu, cu_width, s - 1) : 0;
                if (e0 < 0 || e1 < e0 || e1 > tokens || e1 - e0 > max_len) bad = 1;
                start = (int)e0;
                len = bad ? 0 : (int)(e1 - e0);
                if (s == n_seqs - 1) hdr->covered_end = (int)e1;  // a rejected table: overwritten below
            }
        }
        if (bad) sh_bad = 1;
        const int n = (len + kTileQ - 1) / kTileQ;
        int a_items = n, a_slots = n * (n + 1), tot_i, tot_s;
        block_scan2(a_items, a_slots, sh, tot_i, tot_s);
        if (s < n_seqs) {
            seqs[s] = SeqInfo{b, start, len, slot_carry + a_slots - n * (n + 1)};
            if (n > 0) atomicAdd(&cursor[n], 1);
        }
        item_carry += tot_i;
        slot_carry += tot_s;
    }
    __syncthreads();
    const bool bad = sh_bad != 0 || item_carry > max_items || (int64_t)slot_carry > slot_cap;

    // pass 2: items of cost c (tile index c-1) = sequences with at least c tiles; heaviest class first: two scans from the
    // largest c downwards
    int seqs_carry = 0, pos_carry = 0;
    for (int base = 0; base < n_max; base += kPrepThreads) {
        const int c = n_max - base - t;
        int n_with = c >= 1 ? cursor[c] : 0, none = 0, tot_n, tot_p, tot_x;
        block_scan2(n_with, none, sh, tot_n, tot_x);  // sequences with at least c tiles
        n_with += seqs_carry;
        int pos = c >= 1 ? n_with : 0;
        none = 0;
        block_scan2(pos, none, sh, tot_p, tot_x);
        if (c >= 1) cursor[c] = pos_carry + pos - n_with;
        seqs_carry += tot_n;
        pos_carry += tot_p;
    }
    if (t == 0) {
        hdr->n_items = bad ? 0 : item_carry;
        hdr->n_seqs = n_seqs;
        hdr->total_slots = slot_carry;
        hdr->bad = bad ? 1 : 0;
        if (batch > 0) hdr->covered_end = tokens;
        else if (bad || n_seqs == 0) hdr->covered_end = 0;
        if (bad) atomicOr(status, SBATTN_ST_BAD_SEQLENS);
    }
    __syncthreads();
    if (bad) return;
    int group = 1;  // lanes per sequence
    while (group < 32 && group < n_max) group <<= 1;
    for (int s = t / group; s < n_seqs; s += kPrepThreads / group) {
        const int n = (seqs[s].len + kTileQ - 1) / kTileQ;
        for (int qt = t & (group - 1); qt < n; qt += group) items[atomicAdd(&cursor[qt + 1], 1)] = make_int2(s, qt);
    }
}

// Fused-remainder backward: drem_eff = drem + do . v per row (out = o + rem * v sends do . v into rem), float32.  16 bytes of do
// and v per lane, the D / 8 lanes of a row add up by shuffles, four rows in flight per group.  Bound by memory: 2 x 2 D bytes per row.
// (In the dq kernel, where every row thread read its two rows itself, 256 bytes apart from its neighbours', this cost 0.7 ms
// of 4.3 ms on 12 heads x 4 x 8192 tokens.)
template <typename T>
__global__ void __launch_bounds__(256) drem_kernel(const __grid_constant__ KArgs a, int entries) {
    constexpr int kInFlight = 4;
    pdl_wait();
    pdl_launch_dependents();
    const int lanes = a.head_dim >> 3, per_block = 256 / lanes;  // 4, 8 or 16 lanes per row
    const int col = ((int)threadIdx.x & (lanes - 1)) * 8;
    const int t0 = (int)blockIdx.x * per_block * kInFlight + (int)threadIdx.x / lanes;
    for (int bh = blockIdx.y; bh < entries; bh += gridDim.y) {  // no divisions per row
        const int b = bh / a.heads, h = bh - b * a.heads;
        const T* pd = (const T*)a.d_o.ptr + (int64_t)b * a.d_o.sb + (int64_t)h * a.d_o.sh + col;
        const T* pv = (const T*)a.v.ptr + (int64_t)b * a.v.sb + (int64_t)h * a.v.sh + col;
        const T* pr = (const T*)a.d_rem.ptr + (int64_t)b * a.d_rem.sb + (int64_t)h * a.d_rem.sh;
        uint4 x[kInFlight], y[kInFlight];
        float add[kInFlight];
#pragma unroll
        for (int i = 0; i < kInFlight; ++i) {
            const int t = t0 + i * per_block;
            x[i] = y[i] = make_uint4(0u, 0u, 0u, 0u);
            add[i] = 0.f;
            if (t < a.tokens) {
                x[i] = __ldg((const uint4*)(pd + (int64_t)t * a.d_o.st));
                y[i] = __ldg((const uint4*)(pv + (int64_t)t * a.v.st));
                add[i] = to_f32<T>(pr[(int64_t)t * a.d_rem.st]);
            }
        }
#pragma unroll
        for (int i = 0; i < kInFlight; ++i) {
            const int t = t0 + i * per_block;
            const T* xe = (const T*)&x[i];
            const T* ye = (const T*)&y[i];
            float dot = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) dot = fmaf(to_f32<T>(xe[e]), to_f32<T>(ye[e]), dot);
            for (int off = lanes >> 1; off; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
            if (t < a.tokens && col == 0) a.drem_eff[(int64_t)h * a.drem_rows + (int64_t)b * a.tokens + t] = add[i] + dot;
        }
    }
}

// First entry and largest difference of cumulative ends, written to pinned host memory: out[0], out[1], then out[2] = 1.  The host
// waits for that word: 15 -> 10 us against a copy and a stream synchronisation.
template <typename I>
__global__ void __launch_bounds__(256) seq_bounds_kernel(const I* cu, int64_t n, int leading, int64_t* out) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ int64_t part[8];
    int64_t m = INT64_MIN;
    for (int64_t i = leading + threadIdx.x; i < n; i += 256) {
        const int64_t d = (int64_t)cu[i] - (i > 0 ? (int64_t)cu[i - 1] : 0);
        m = d > m ? d : m;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int64_t y = __shfl_xor_sync(0xffffffffu, m, off);
        m = y > m ? y : m;
    }
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) m = part[w] > m ? part[w] : m;
    out[0] = (int64_t)cu[0];
    out[1] = n > leading ? m : 0;
    __threadfence_system();
    *(volatile int64_t*)(out + 2) = 1;
}

}  // namespace

int launch_drem(const SbParams& p, const KArgs& a, cudaStream_t st) {
    const int entries = (p.batch > 0 ? p.batch : 1) * p.heads, per_block = 4 * 256 / (p.head_dim / 8);
    const dim3 grid((unsigned)((p.tokens + per_block - 1) / per_block), (unsigned)(entries < 65535 ? entries : 65535));
    if (p.dtype == SBATTN_F16) return launch_kernel(drem_kernel<__half>, grid, dim3(256), 0, st, a, entries);
    return launch_kernel(drem_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, a, entries);
}

int launch_prep(const SbParams& p, const WsLayout& L, cudaStream_t st) {
    char* ws = (char*)p.fwd_workspace;
    const int max_len = p.batch > 0 ? p.tokens : (p.max_seqlen > 0 ? p.max_seqlen : p.tokens);
    return launch_kernel(prep_kernel, dim3(1), dim3(kPrepThreads), 0, st, (WsHeader*)ws, (SeqInfo*)(ws + L.off_seqs),
                         (int2*)(ws + L.off_items), (int32_t*)(ws + L.off_bins), p.cu_seqlens, (int)p.cu_width, (int)L.n_seqs, (int)p.batch,
                         (int)p.tokens, max_len, (int)L.n_max, (int)L.max_items, L.slot_cap, p.status);
}

}  // namespace sb

extern "C" int sbattn_seq_bounds(const void* cu, int cu_width, int64_t n, int leading, int64_t* out, void* stream) {
    if (!cu || !out) return SBATTN_ENULL;
    if ((cu_width != 4 && cu_width != 8) || n < 1 || leading < 0 || leading > 1) return SBATTN_EINVAL;
    const cudaStream_t st = (cudaStream_t)stream;
    const int e = cu_width == 8 ? sb::launch_kernel(sb::seq_bounds_kernel<int64_t>, dim3(1), dim3(256), 0, st, (const int64_t*)cu, n, leading, out)
                                : sb::launch_kernel(sb::seq_bounds_kernel<int32_t>, dim3(1), dim3(256), 0, st, (const int32_t*)cu, n, leading, out);
    return e == 0 ? SBATTN_OK : SBATTN_ECUDA;
}
