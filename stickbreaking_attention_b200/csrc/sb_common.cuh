// Shared host/device definitions of the stick-breaking attention library: workspace layout, the work-item
// table that every kernel walks, and small device helpers.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <atomic>
#include <mutex>
#include <unordered_map>
#include <utility>

#include "../../include/sbattn.h"

namespace sb {

constexpr int kTileQ = 128;    // query rows per work item
constexpr int kTileKV = 64;    // keys per slot of the slot count (each slot holds two 32-key carries)
constexpr int kMaxHeadDim = 128;

// One sequence of the pack (or one batch entry of the batched layout).
struct SeqInfo {
    int32_t batch;      // index along B (0 for the packed layout)
    int32_t start;      // first token along T
    int32_t len;        // tokens
    int32_t slot_base;  // first carry slot of this sequence (per head)
};

// Start of the forward workspace.  The prep kernel fills it; all later kernels only read it.
struct WsHeader {
    int32_t n_items;      // work items per head = sum over sequences of ceil(len/128)
    int32_t n_seqs;
    int32_t total_slots;  // carry slots per head actually used
    int32_t bad;          // non-zero: sequence table rejected, n_items is 0
    // work counters of the persistent kernels (forward, backward dq, backward dk/dv): [2k] next work index,
    // [2k+1] blocks that have finished; zeroed by the prep kernel, reset by the last block of every launch
    int32_t sched[8];
    int32_t covered_end;  // packed layout: end of the last sequence (tokens beyond it belong to no sequence)
    int32_t pad[51];
};
static_assert(sizeof(WsHeader) == 256, "header is one 256-byte line");

// Host-side description of where things live inside the workspaces (all offsets in bytes).
struct WsLayout {
    int32_t n_seqs;      // sequences (packed: num_seqs, batched: B)
    int32_t n_max;       // max 128-row tiles of one sequence
    int32_t max_items;   // upper bound on items per head
    int64_t slot_cap;    // upper bound on 64-key carry slots per head
    int32_t hb;          // heads (batched: heads; the batch index comes from the sequence)
    size_t off_seqs, off_items, off_bins, off_carry;
    size_t off_drem;     // inside the backward workspace
    size_t fwd_bytes;    // with carries if save_carries
    size_t bwd_bytes;
};

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

inline WsLayout make_layout(const SbParams& p) {
    WsLayout L{};
    const bool batched = p.batch > 0;
    L.n_seqs = batched ? p.batch : p.num_seqs;
    const int64_t maxlen = batched ? p.tokens : (p.max_seqlen > 0 ? (p.max_seqlen < p.tokens ? p.max_seqlen : p.tokens) : p.tokens);
    L.n_max = (int32_t)((maxlen + kTileQ - 1) / kTileQ);
    if (L.n_max < 1) L.n_max = 1;
    if (batched) {
        L.max_items = L.n_seqs * L.n_max;
        L.slot_cap = (int64_t)L.n_seqs * L.n_max * (L.n_max + 1);
    } else {
        // sum ceil(len/128) <= T/128 + S ; sum n(n+1) <= (n_max+1) * sum n
        const int64_t items = p.tokens / kTileQ + L.n_seqs;
        L.max_items = (int32_t)items;
        L.slot_cap = items * (L.n_max + 1);
    }
    L.hb = p.heads;
    size_t off = sizeof(WsHeader);
    L.off_seqs = off;
    off = align_up(off + sizeof(SeqInfo) * (size_t)L.n_seqs, 256);
    L.off_items = off;
    off = align_up(off + sizeof(int2) * (size_t)L.max_items, 256);
    L.off_bins = off;
    off = align_up(off + sizeof(int32_t) * (size_t)(2 * (L.n_max + 2)), 256);
    L.off_carry = off;
    const size_t carry = sizeof(float) * (size_t)L.hb * (size_t)(2 * L.slot_cap) * kTileQ;  // two 32-key carries per slot
    L.fwd_bytes = off + (p.save_carries ? carry : 0);
    L.off_drem = align_up(carry, 256);  // after carry_c: drem + do . v per (head, token), fused-remainder backward
    L.bwd_bytes = L.off_drem + align_up(sizeof(float) * (size_t)p.heads * (size_t)p.tokens * (size_t)(batched ? p.batch : 1), 256);
    return L;
}

// What the kernels need of a [B,H,T,D] tensor.
struct MatView {
    char* ptr;
    int64_t sb, sh, st;  // element strides
};
struct VecView {
    char* ptr;
    int64_t sb, sh, st;
};
inline MatView view(const SbMat& m) { return MatView{(char*)m.ptr, m.stride_b, m.stride_h, m.stride_t}; }
inline VecView view(const SbVec& m) { return VecView{(char*)m.ptr, m.stride_b, m.stride_h, m.stride_t}; }

// Arguments common to every attention kernel.
struct KArgs {
    const WsHeader* hdr;
    const SeqInfo* seqs;
    const int2* items;      // (sequence, 128-row tile), heaviest first
    float* carry_w;         // forward carries  [heads][slot_cap][128], may be null in a no-grad forward; slot_cap: 32-key slots
    float* carry_c;         // backward carries [heads][slot_cap][128]
    int64_t slot_cap;
    int32_t heads, head_dim, attend_current;
    int32_t fused;          // SBATTN_FLAG_FUSED_REMAINDER, SBATTN_FLAG_REMAINDER_IN_DV
    int32_t tokens;         // tokens per batch entry (row index of drem_eff: batch * tokens + token)
    float* drem_eff;        // [heads][drem_rows]: drem + do . v (fused-remainder backward)
    int64_t drem_rows;      // batch * tokens (tokens for the packed layout)
    int32_t head_group;     // heads whose work is interleaved (sized so that their K and V stay in L2)
    int32_t zero_tail;      // packed layout: clear the result rows of tokens behind the last sequence
    // forward of small problems: every block builds the work-item table itself (no prep kernel)
    int32_t own_tables, cu_width, n_seqs, batch, max_len, n_max, max_items;
    const void* cu_seqlens;
    int32_t* sched;         // WsHeader::sched
    float inv_temp;
    MatView q, k, v, o, d_o, dq, dk, dv;
    VecView rem, nla, d_rem;
    uint32_t* status;
};

// Carries exist at every 32-key boundary.  carry_slot32: (128-row tile qt of a sequence, 32-key quarter kq in [0, 4*qt+3]),
// the value at the quarter's right edge.  slot_base and WsLayout::slot_cap count 64-key slots, KArgs::slot_cap 32-key slots.
__host__ __device__ inline int64_t carry_slot32(int32_t slot_base, int32_t qt, int32_t kq) {
    return 2 * ((int64_t)slot_base + (int64_t)qt * (qt + 1)) + kq;
}

template <typename T> __device__ inline float to_f32(T x);
template <> __device__ inline float to_f32<float>(float x) { return x; }
template <> __device__ inline float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }
template <> __device__ inline float to_f32<__half>(__half x) { return __half2float(x); }
template <typename T> __device__ inline T from_f32(float x);
template <> __device__ inline float from_f32<float>(float x) { return x; }
template <> __device__ inline __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ inline __half from_f32<__half>(float x) { return __float2half_rn(x); }

// Kernel launches made by the library in this process (sbattn_launch_count); every launch site calls count_launch().
extern unsigned long long g_launch_count;
inline void count_launch() { __atomic_fetch_add(&g_launch_count, 1ull, __ATOMIC_RELAXED); }

// Programmatic dependent launch: every kernel of the library may start while the kernel before it in the stream drains, sets up
// what needs no global memory, and then waits here for that kernel's completion (and with it, since every kernel of
// the library waits, for everything before).  A kernel that lets its successor start early calls pdl_launch_dependents().
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgsT, typename... ArgsT>
inline int launch_kernel(void (*kernel)(KArgsT...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, ArgsT&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<ArgsT>(args)...);
    count_launch();
    return (int)(e == cudaSuccess ? cudaGetLastError() : e);
}

// streaming multiprocessors of the current device
inline int sm_count() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int n = cache[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cache[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Dynamic shared memory size (and the carve-out preference) of a kernel, set once per kernel and device instead of on
// every launch: the two driver calls cost more than the launch itself for small problems.
inline int ensure_kernel_attrs(const void* kernel, int smem_bytes, bool prefer_shared) {
    static std::mutex mu;
    static std::unordered_map<const void*, uint64_t> done;  // bit d: set on device d
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return (int)cudaErrorInvalidDevice;
    const bool tracked = dev >= 0 && dev < 64;
    if (tracked) {
        std::lock_guard<std::mutex> lock(mu);
        auto it = done.find(kernel);
        if (it != done.end() && ((it->second >> dev) & 1)) return 0;
    }
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (e != cudaSuccess) return (int)e;
    if (prefer_shared) cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (tracked) {
        std::lock_guard<std::mutex> lock(mu);
        done[kernel] |= 1ull << dev;
    }
    return 0;
}

// The tables of prep_kernel for at most 32 sequences and kOwnItems items, built by one warp in shared memory; the launch of that
// kernel is a quarter of a small forward.  Every block comes to the same order (heaviest first; inside a class by sequence).
// Block 0 leaves the tables in the workspace for the backward.
constexpr int kOwnSeqs = 32, kOwnItems = 256;
struct OwnTables {
    SeqInfo seqs[kOwnSeqs];
    int2 items[kOwnItems];
    int n_items, covered_end;
};
__device__ inline void build_own_tables(const KArgs& a, OwnTables* t, int lane) {
    const auto end_of = [&](int s) { return a.cu_width == 8 ? ((const int64_t*)a.cu_seqlens)[s] : (int64_t)((const int32_t*)a.cu_seqlens)[s]; };
    int b = 0, start = 0, len = 0, end = 0;
    bool bad = false;
    if (lane < a.n_seqs) {
        if (a.batch > 0) {
            b = lane;
            len = a.tokens;
        } else {
            const int64_t e1 = end_of(lane), e0 = lane > 0 ? end_of(lane - 1) : 0;
            bad = e0 < 0 || e1 < e0 || e1 > a.tokens || e1 - e0 > a.max_len;
            start = (int)e0;
            len = bad ? 0 : (int)(e1 - e0);
            end = (int)e1;
        }
    }
    const int n = (len + kTileQ - 1) / kTileQ;
    int slots = n * (n + 1), total = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, slots, off), y = __shfl_up_sync(0xffffffffu, total, off);
        if (lane >= off) {
            slots += x;
            total += y;
        }
    }
    const int total_slots = __shfl_sync(0xffffffffu, slots, 31);
    total = __shfl_sync(0xffffffffu, total, 31);
    bad = __any_sync(0xffffffffu, bad) || total > a.max_items || 2 * (int64_t)total_slots > a.slot_cap;
    const SeqInfo mine{b, start, len, slots - n * (n + 1)};
    if (lane < a.n_seqs) t->seqs[lane] = mine;
    end = __shfl_sync(0xffffffffu, end, max(a.n_seqs - 1, 0));
    const bool out = blockIdx.x == 0;
    int pos = 0;
    for (int c = bad ? 0 : a.n_max; c >= 1; --c) {  // sequences with at least c tiles have a tile c - 1
        const unsigned has = __ballot_sync(0xffffffffu, n >= c);
        if (n >= c) {
            const int at = pos + __popc(has & ((1u << lane) - 1u));
            t->items[at] = make_int2(lane, c - 1);
            if (out) const_cast<int2*>(a.items)[at] = make_int2(lane, c - 1);
        }
        pos += __popc(has);
    }
    if (lane == 0) {
        t->n_items = bad ? 0 : total;
        t->covered_end = a.batch > 0 ? a.tokens : bad ? 0 : end;
    }
    if (out) {
        WsHeader* hdr = const_cast<WsHeader*>(a.hdr);
        if (lane < a.n_seqs) const_cast<SeqInfo*>(a.seqs)[lane] = mine;
        if (lane < 8) hdr->sched[lane] = 0;
        if (lane == 0) {
            hdr->n_items = bad ? 0 : total;
            hdr->n_seqs = a.n_seqs;
            hdr->total_slots = total_slots;
            hdr->bad = bad ? 1 : 0;
            hdr->covered_end = a.batch > 0 ? a.tokens : bad ? 0 : end;
            if (bad) atomicOr(a.status, SBATTN_ST_BAD_SEQLENS);
        }
    }
}

// Result rows of tokens that belong to no sequence (a pack whose last end is below T), shared out over all threads of the grid:
// every other row is written by the attention kernels, so the caller need not clear anything.  rem and neg_log_acc are
// zero there (what the reference's zero-initialised outputs hold, sb_varlen_fwd.py:418-419), and so are the gradients.
template <typename T>
__device__ inline void zero_tail_rows(const KArgs& a, int first, int64_t thread, int64_t n_threads) {
    const int64_t total = (int64_t)(a.tokens - first) * a.heads;
    for (int64_t i = thread; i < total; i += n_threads) {
        const int h = (int)(i % a.heads);
        const int64_t t = first + i / a.heads;
        ((T*)a.rem.ptr)[h * a.rem.sh + t * a.rem.st] = T(0.f);
        ((float*)a.nla.ptr)[h * a.nla.sh + t * a.nla.st] = 0.f;
    }
}
template <typename T>
__device__ inline void zero_tail_grads(const KArgs& a, int first, int64_t thread, int64_t n_threads) {
    const int D = a.head_dim;
    const int64_t total = (int64_t)(a.tokens - first) * a.heads * D;
    for (int64_t i = thread; i < total; i += n_threads) {
        const int d = (int)(i % D);
        const int64_t rh = i / D;
        const int h = (int)(rh % a.heads);
        const int64_t t = first + rh / a.heads;
        ((T*)a.dq.ptr)[h * a.dq.sh + t * a.dq.st + d] = T(0.f);
        ((T*)a.dk.ptr)[h * a.dk.sh + t * a.dk.st + d] = T(0.f);
        ((T*)a.dv.ptr)[h * a.dv.sh + t * a.dv.st + d] = T(0.f);
    }
}

// launchers implemented in the .cu files (each returns a cudaError_t as int; the tensor-core launchers return
// kMapEncodeFailed when a tensor map could not be encoded, before anything has been launched)
constexpr int kMapEncodeFailed = -1000;
int launch_prep(const SbParams& p, const WsLayout& L, cudaStream_t st);
int launch_drem(const SbParams& p, const KArgs& a, cudaStream_t st);
int launch_f32_fwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);
int launch_f32tc(const SbParams& p, bool backward, const WsLayout& L, const KArgs& a, cudaStream_t st);  // head dims up to 64
int launch_f32_bwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);
bool tensor_path_eligible(const SbParams& p, bool backward, int* why);
int launch_tensor_fwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);
int launch_tensor_fwd_pair(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);  // two query tiles at a time
int launch_tensor_bwd_tile(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);  // sequences of one tile
int launch_tensor_bwd(const SbParams& p, const WsLayout& L, const KArgs& a, cudaStream_t st);
int launch_weights(const SbParams& p, float* w, int64_t stride_b, int64_t stride_h, int64_t stride_m, cudaStream_t st);

}  // namespace sb
