// Fused five-GEMM attention backward for sm_100a.
//
// One CTA owns one (batch, KV head, 128-key tile) and walks every 128-row query
// tile that can see those keys, for each of the G query heads that share the
// KV head.  dK and dV stay in tensor memory for the whole walk, so a GQA group
// is reduced inside the kernel and written once.  Per query tile ("step"):
//
//     S^T  = K  Q^T        [key j on TMEM lanes, query i on columns]   SS MMA
//     dP^T = V  dO^T                                                    SS MMA
//     P^T  = exp2(S^T * scale*log2e - m_i) * r_i      (CUDA cores, -> TMEM b16)
//     dV  += P^T dO        A = P^T from TMEM, B = dO (MN-major)         TS MMA
//     dS^T = P^T o (dP^T - delta_i)                   (CUDA cores, -> smem b16)
//     dK  += dS^T Q        A = dS^T (K-major), B = Q (MN-major)         SS MMA
//     dQ   = dS K          A = dS^T read MN-major, B = K (MN-major)     SS MMA
//     dQacc[tile] += dQ    TMEM -> regs -> smem -> TMA reduce-add (fp32)
//
// The softmax scale is applied once at the end (dK in the epilogue, dQ in the
// convert kernel) instead of per element of dS.
//
// Epilogue: when the last MMA has completed, every softmax warp stages its 32 key rows of dK
// (scaled) or dV in shared memory and stores them in whole lines.  On problems too small to fill the GPU the query steps
// of a key tile are cut into chunks, one CTA each (a table in the kernel parameters says which,
// longest chunks first); such a CTA stores its partial dK / dV to its own slab and the convert
// kernel adds the slabs of a tile in chunk order.
//
// Warp roles (512 threads, four warpgroups): warp 0 = TMA producer, warp 1 = MMA
// issuer and TMEM owner, warp 2 = row statistics, warp 3 = which tile; warps 4-7 and 8-11 = two softmax / dS warpgroups (thread
// j of each owns TMEM lane j = key j; the first takes queries 0-63 of the tile,
// the second queries 64-127); warps 12-15 = dQ drain warpgroup.  Registers are
// re-split with setmaxnreg (96 / 120 / 120 / 176 per thread at D=128).  All hand-offs go
// through mbarriers; every wait is bounded and a time-out raises an error flag
// instead of hanging.  (The longest that a correct run needs is that for the next tile, over a whole tile: kMostStepsTakenOver.)
//
// Tiles (kPersist): a CTA that is about to finish its tile asks for the block index of a CTA that has not started, warp 3
// works out what that is and hands it to the other roles in shared memory, and the roles, rings and hand-offs run on: K, V, Q
// and dO of the next tile are loaded and its first S is computed beside the epilogue, and the set-up (barriers, tensor memory,
// cold instruction cache: 1300-2800 clk until the first loads, 3000-5000 until they have landed) is paid once.  Where every SM
// has several tiles; the rule and what it measured stand in cta_order.h.  One warp works the tile out for all, in either
// form, because the index arithmetic inlined in five roles was 1400 clk of cold code in front of the first loads.
//
// Tensor-memory ledger (512 columns x 128 lanes x 32 bit):
//     D = 128:  dK [0,128)  dV [128,256)  S/P [256,384)  dP and dQ share [384,512)
//     D =  64:  dK [0,64)   dV [64,128)   S/P [128,256)  dP [256,384)  dQ [384,448)
// P^T (16-bit, two per column) is written over S^T in place: queries 0-63 on the
// first 32 columns of the S region, queries 64-127 on columns 64-95, so that each
// softmax warpgroup only overwrites columns it has already read itself.
//
// Shared-memory ledger (bytes; every tile is made of 16 KiB boxes of
// [128 rows][64 x 16 bit] in the 128-byte swizzle):
//     K, V            2 x D*256            resident for the CTA
//     Q               2 stages (D=128) or 3 (D=64) x D*256
//     dO              1 stage (D=128) or 2 stages (D=64) x D*256
//     dS^T            32 KiB               [128 keys][128 queries]
//     dQ staging      32 KiB               4 warps x 2 boxes of [32 rows][32 fp32]
//     row statistics  2 KiB                {log2 r - m, -delta} x 128 rows x 2 buffers
//     mbarriers       256
//     work of a tile  256                  two buffers
//     total           231,936 (D=128) / 182,784 (D=64)   of 232,448 available
//
// What bounds it: at D=64 the softmax / dS warpgroups (2650 clk per step, 1664 of MMA): one instruction per two
// elements wherever packed arithmetic allows, statistics brought by a warp of their own, one arrival per warp
// and uniform votes at the barriers took the step from 2980; B=4,H=16,S=4096 full, kernel alone after a pause:
// 859-867 -> 788 us.  At D=128 the copy engine (64 KB of loads and 64 KB of fp32 reduce-adds per step, 2400-3000 clk
// for the latter) and the chain dS -> dQ -> drain -> dP -> dS, 3800-4000 clk per step (2560 of MMA): 1197 -> 1188 us for
// the same shape, 1270-1320 both under the power limit, which holds the clock near 1.55 GHz.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "geometry.h"
#include "ptx.cuh"

namespace fa3b200 {

enum DeviceError : int {
    kDevOk = 0,
    kDevWaitTimeout = 1,
    kDevSmemMisaligned = 2,
};

// First error raised by any kernel since the flag was last cleared.
__device__ int g_device_error = 0;

#ifdef FA3B200_TRACE
// Instrumented builds only: cycle stamps of every CTA, by role (0 producer, 1 MMA warp,
// 2 first softmax warp, 3 first drain warp) and event slot.
constexpr int kTraceCtas = 1024;
constexpr int kTraceEvents = 64;
__device__ long long g_trace[kTraceCtas][4][kTraceEvents];
__device__ long long g_trace_rowwise[4];  // {delta first start, delta last end, convert first start, convert last end} (globaltimer)
__device__ __forceinline__ long long trace_globaltimer() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define TRACE(role, ev) do { if ((threadIdx.x & 31) == 0 && blockIdx.x < kTraceCtas && (ev) < kTraceEvents) g_trace[blockIdx.x][role][ev] = clock64(); } while (0)
#define TRACE_GT(role, ev) do { if ((threadIdx.x & 31) == 0 && blockIdx.x < kTraceCtas) g_trace[blockIdx.x][role][ev] = trace_globaltimer(); } while (0)
#define TRACE_VALUE(role, ev, v) do { if ((threadIdx.x & 31) == 0 && blockIdx.x < kTraceCtas) g_trace[blockIdx.x][role][ev] = (v); } while (0)
#else
#define TRACE(role, ev) do {} while (0)
#define TRACE_GT(role, ev) do {} while (0)
#define TRACE_VALUE(role, ev, v) do {} while (0)
#endif

struct FusedArgs {
    // Row statistics of query row i, one of the two: {log2 r - m, -delta} as [B,Hq,Sq,2] (packed sequences:
    // [Hq,total_q,2]), what the v2 call's delta stage leaves, or the packed sidecar {m, r, delta} as
    // [B,Hq,Sq,3] of the component entry points.
    const float2* stats;
    const float* sidecar;
    void* dk;              // [B,Hkv,Sk,D] or [B,Sk,Hkv,D], see kv_strides
    void* dv;
    void* dkv_slabs;       // split tiles: a CTA writes its partial dK (scaled) to slab 2x and dV to slab 2x+1,
                           // each [128 rows][D], fp32 or (slabs_f16, fp16 inputs only) fp16; the convert
                           // kernel adds the slabs of a tile
    int slabs_f16;
    TensorStrides kv_strides;  // element strides of dk / dv
    int batch;
    int heads_q;
    int heads_kv;
    Band band;             // sequence lengths and the visible band (geometry.h); with packed
                           // sequences the lengths are the maxima and each CTA reads its own
    const int* cu_seqlens_q;  // non-null: sequences are packed ([total, H, D] tensors) and sequence b
    const int* cu_seqlens_k;  // owns rows cu[b] .. cu[b+1]-1; the tensor maps then have batch = 1
    const int* seqused_q;     // non-null: only the first seqused[b] rows of batch entry b take part; the
    const int* seqused_k;     // gradient rows behind them, up to the end of the entry's slot, are zero
    int sidecar_rows;      // rows per head of the sidecar / accumulators (seqlen_q, or total_q when packed)
    float scale;
    float scale_log2;
    // softcap variant: the scaled scores go through softcap * tanh(x / softcap) before the softmax;
    // in log2 units that is softcap_post * tanh(score * softcap_pre), softcap_pre = scale / softcap,
    // softcap_post = softcap * log2(e)
    float softcap_pre;
    float softcap_post;
    FastDiv per_group;     // key tiles * head_group
    FastDiv in_group;      // head_group
    FastDiv kv_heads;      // heads_kv
    FastDiv chunks;        // chunks_per_head
    int group;             // heads_q / heads_kv
    int order_mode;        // see cta_order.h
    int order_width;
    int head_group;        // heads per scheduling group: block = (group * n_tiles + tile slot) * head_group + head
    int chunk_steps;       // > 0: the steps of a key tile are cut into chunks of this many steps, one CTA
                           // per chunk, and the partial dK/dV of every chunk go to its own slabs
    int chunks_per_head;   // number of chunks of one (batch, KV head) when chunk_steps > 0
    // chunk_steps > 0: which chunk CTA x runs, longest chunks first.  Entry = key tile | chunk index
    // inside the tile << 8 | slab << 16, where slab = (batch, KV head) * chunks_per_head + the chunk's
    // place in the head's list (key tile 0 first): the CTA's partial dK goes to slab 2*slab, dV to 2*slab+1.
    uint32_t cta_table[kMaxSplitCtas];
};

__host__ __device__ inline int remap_k_tile(int physical, int count, int mode, int width) {
    if (mode == 0) return physical;                 // heaviest (lowest index) first
    if (mode == 1) return count - 1 - physical;     // lightest first
    // mode 2: serpentine inside rounds of `width` tiles
    const int round = physical / width;
    const int base = round * width;
    const int slot = physical - base;
    int span = count - base;
    if (span > width) span = width;
    return base + ((round & 1) == 0 ? slot : span - 1 - slot);
}

template <int D, bool kSoftcap = false>
struct FusedCfg {
    static constexpr int kTile = 128;
    static constexpr int kThreads = 512;
    static constexpr int kBoxBytes = 128 * 128;
    static constexpr int kBoxes = D / 64;
    static constexpr int kOperandBytes = kBoxes * kBoxBytes;
    // (a third Q stage at D=64: us per call of B=4,H=16,S=4096 full, back to back, 877-899 with two and 873 with three;
    // the kernel alone after a pause 782 and 788; a fourth, or a third of dO, no more)
    static constexpr int kQStages = D == 64 ? 3 : 2;
    static constexpr int kDoStages = D == 128 ? 1 : 2;
    static constexpr int kDsBytes = 2 * kBoxBytes;
    static constexpr int kStageBoxBytes = 32 * 128;
    static constexpr int kStageBytes = 4 * 2 * kStageBoxBytes;

    static constexpr int kOffK = 0;
    static constexpr int kOffV = kOffK + kOperandBytes;
    static constexpr int kOffQ = kOffV + kOperandBytes;
    static constexpr int kOffDO = kOffQ + kQStages * kOperandBytes;
    static constexpr int kOffDS = kOffDO + kDoStages * kOperandBytes;
    static constexpr int kOffStage = kOffDS + kDsBytes;
    static constexpr int kOffStats = kOffStage + kStageBytes;
    // Row statistics: two buffers of 128 x {log2 r - m}, then two of 128 x {-delta}
    static constexpr int kOffBar = kOffStats + 2 * 1024;
    static constexpr int kOffWork = kOffBar + 256;  // two buffers
    static constexpr int kSmemBytes = kOffWork + 256;
    static_assert(kSmemBytes <= 232448, "shared-memory ledger exceeds 227 KiB");
    static_assert(kOffStage % 1024 == 0 && kOffDS % 1024 == 0, "swizzled regions need 1 KiB alignment");

    // setmaxnreg split per warpgroup (producer+MMA / softmax x2 / drain); sums to <= 512.  (Capped scores hold P (1 - t^2) in 48
    // registers instead of P in 32.)
    static constexpr int kRegsControl = kSoftcap && D == 128 ? 80 : 96;
    static constexpr int kRegsCompute = (D == 128 ? 120 : 136) + (kSoftcap ? 8 : 0);
    static constexpr int kRegsDrain = D == 128 ? 176 : kSoftcap ? 128 : 136;
    static constexpr int kRegsComputeNoDq = 160;  // without dQ the drain warpgroup idles at kRegsControl
    static_assert(kRegsControl + 2 * kRegsCompute + kRegsDrain <= 512, "register file over-committed");
    static_assert(2 * kRegsControl + 2 * kRegsComputeNoDq <= 512, "register file over-committed");

    // Capped scores: of every 8 pairs of tanh, how many go to the FMA pipe (tanh_mixed).  us of the first gradients named there for 2,
    // 3, 4, 5, 8 of 8: 144, 141, 140, 140, 147; of the last 352, 339, 335, 328, 340.
    static constexpr int kTanhFmaPairs = 5;

    static constexpr int kTmemCols = 512;
    static constexpr int kColDK = 0;
    static constexpr int kColDV = D;
    static constexpr int kColS = 2 * D;
    static constexpr int kColDP = 2 * D + 128;
    static constexpr int kColDQ = D == 128 ? kColDP : kColDP + 128;
    static_assert(kColDQ + D <= kTmemCols, "tensor-memory ledger exceeds 512 columns");
    static_assert(8 * 32 * D * 4 <= kOffStage - kOffQ, "epilogue staging does not fit");
};

enum Bar : int {
    kKvFull = 0,
    kQFull = 1,        // up to 3 stages
    kQEmpty = 4,       // up to 3 stages
    kDoFull = 7,       // up to 2 stages
    kDoEmpty = 9,      // up to 2 stages
    kSFull = 11,
    kDpFull = 12,
    kPReady = 13,
    kDsReady = 14,
    kDqFull = 15,
    kDqEmpty = 16,
    kDkvFull = 17,
    kStatsFull = 18,   // 2 buffers
    kStatsEmpty = 20,  // 2 buffers
    kAnswer = 22,      // which block comes next
    kWorkFull = 23,    // 2 buffers: the work of a block
    kWorkEmpty = 25,   // 2 buffers
    kNumBars = 27,
};

constexpr uint32_t kWaitTimeoutCycles = 2000000000u;  // about one second, of a 32-bit cycle counter

// Bounded mbarrier wait of a single thread (the TMA producer).  Returns false when the wait timed out
// here or was abandoned because another thread of the CTA timed out (abort_flag: its shared-memory address).
__device__ __forceinline__ uint32_t flag_value(uint32_t flag) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(flag) : "memory");
    return v;
}
__device__ __forceinline__ void flag_set(uint32_t flag, uint32_t v) {
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(flag), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t clock_lo() {
    uint32_t c;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(c));
    return c;
}
template <bool kBackoff = false>
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
    if (ptx::mbar_try_wait(bar, parity)) return true;
    const uint32_t start = clock_lo();
#pragma unroll 1
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            if (ptx::mbar_try_wait(bar, parity)) return true;
            if (kBackoff) __nanosleep(32);  // keep a waiting warp off the issue ports
        }
        if (flag_value(abort_flag) != 0) return false;
        if (clock_lo() - start > kWaitTimeoutCycles) {
            flag_set(abort_flag, 1);
            atomicCAS(&g_device_error, kDevOk, kDevWaitTimeout);
            return false;
        }
    }
}

// The same for a converged warp.  The votes make every branch uniform: a wait for a barrier that has
// completed costs one round trip to the barrier (97 clk; 107-153 beside busy math warps), where per-lane
// polling with a vote behind it costs the reconvergence of a divergent loop on top (174 clk, 189-262).
template <bool kBackoff = true>
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t abort_flag) {
    constexpr uint32_t kAll = 0xffffffffu;
    if (__all_sync(kAll, ptx::mbar_try_wait(bar, parity))) return true;
    const uint32_t start = clock_lo();
#pragma unroll 1
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            if (__all_sync(kAll, ptx::mbar_try_wait(bar, parity))) return true;
            if (kBackoff) __nanosleep(32);
        }
        if (__any_sync(kAll, flag_value(abort_flag) != 0)) return false;
        if (__any_sync(kAll, clock_lo() - start > kWaitTimeoutCycles)) {
            flag_set(abort_flag, 1);
            atomicCAS(&g_device_error, kDevOk, kDevWaitTimeout);
            return false;
        }
    }
}

// Two barriers at once (one round trip when both have completed).
__device__ __forceinline__ bool warp_wait2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1, uint32_t abort_flag) {
    const bool d0 = ptx::mbar_try_wait(bar0, parity0);
    const bool d1 = ptx::mbar_try_wait(bar1, parity1);
    if (__all_sync(0xffffffffu, d0 && d1)) return true;
    return warp_wait(bar0, parity0, abort_flag) && warp_wait(bar1, parity1, abort_flag);
}

// Which key tile and which of its steps a CTA works on.  One warp works it out and hands it to the others in shared memory.
struct alignas(16) FusedWork {
    int block;            // place in the launch order, -1: there is none
    int kt, b, kvh, slab;
    Band band;            // this batch entry's own lengths
    int q_base, k_base, b_coord;
    int slot_k;           // rows of dK / dV this batch entry owns
    int q_tiles;          // query tiles of the sequence
    int q_begin;          // first query tile that sees the key tile
    int steps_per_head;
    int first_head;       // first query head of the KV head's group
    int t_begin, n_steps; // this CTA's share of the tile's steps (all of them unless the tile is split)
    int rotation;
};
// (the forward's work, too)
template <typename W>
__device__ __forceinline__ void store_work(uint32_t addr, const W& w) {
    static_assert(sizeof(W) == 96, "six 16-byte words");
    const uint32_t* v = reinterpret_cast<const uint32_t*>(&w);
#pragma unroll
    for (int i = 0; i < 24; i += 4)
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr + 4 * i), "r"(v[i]), "r"(v[i + 1]), "r"(v[i + 2]), "r"(v[i + 3]) : "memory");
}
template <typename W = FusedWork>
__device__ __forceinline__ W load_work(uint32_t addr) {
    W w;
    uint32_t* v = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
    for (int i = 0; i < 24; i += 4)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[i]), "=r"(v[i + 1]), "=r"(v[i + 2]), "=r"(v[i + 3]) : "r"(addr + 4 * i) : "memory");
    return w;
}

// A value that all lanes of a warp hold, in a form that tells the compiler so: what comes from shared memory might differ between them,
// and loops and branches on it are compiled for that.  us, without and with it, on what the loops of the math warps and the
// MMA warp test: forward, D=64, 11 x 2 heads x 4970 full 190 and 185.5, 4 x 8192 93.0 and 91.6, B=8, 32 x 512 35.9 and 35.2, D=128, B=8,
// 32 x 300 causal 33.3 and 32.0; backward, D=64, 8 x 4096 causal 66.6 and 65.1, 4 x 16384 455 and 438, D=128, B=8, 32 x 300 79.3 and 78.0.
// (All of the work handed over so: slower.)
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }

template <bool kCausal>
__device__ __forceinline__ FusedWork fused_work(const FusedArgs& a, int block) {
    FusedWork w;
    w.block = block;
    const int n_tiles = tiles_of(a.band.seqlen_k);      // key tiles (of the longest sequence)
    const int bh_count = a.batch * a.heads_kv;
    const bool split = a.chunk_steps > 0;
    const int group = a.group;
    int bhi;
    w.t_begin = w.slab = 0;
    if (!split) {
        // groups of head_group heads; inside a group tile slot major, head minor (see cta_order.h)
        const int hg = fast_div(block, a.per_group);
        const int rem = block - hg * a.per_group.divisor;
        const int heads_here = min(a.head_group, bh_count - hg * a.head_group);
        const int tile_slot = heads_here == a.head_group ? fast_div(rem, a.in_group) : rem / heads_here;
        bhi = hg * a.head_group + (rem - tile_slot * heads_here);
        w.kt = remap_k_tile(tile_slot, n_tiles, a.order_mode, a.order_width);
    } else {
        const uint32_t entry = a.cta_table[block];
        w.kt = int(entry & 0xffu);
        w.t_begin = int((entry >> 8) & 0xffu) * a.chunk_steps;
        w.slab = int(entry >> 16);
        bhi = fast_div(w.slab, a.chunks);
    }
    w.b = fast_div(bhi, a.kv_heads);
    w.kvh = bhi - w.b * a.heads_kv;
    w.first_head = w.kvh * group;
    // Packed sequences: this batch entry's own lengths and first rows; tensors are addressed as one
    // batch of `total` rows, so rows past the end of a sequence belong to its neighbour (or read as
    // zero past the end of the tensor) and are masked like any ragged tile end.
    Band band = a.band;
    w.q_base = w.k_base = 0;
    w.b_coord = w.b;
    if (a.cu_seqlens_q != nullptr) {
        w.q_base = a.cu_seqlens_q[w.b];
        w.k_base = a.cu_seqlens_k[w.b];
        band.seqlen_q = a.cu_seqlens_q[w.b + 1] - w.q_base;
        band.seqlen_k = a.cu_seqlens_k[w.b + 1] - w.k_base;
        band.off = band.seqlen_k - band.seqlen_q;
        w.b_coord = 0;
    }
    w.slot_k = band.seqlen_k;
    if (a.seqused_q != nullptr || a.seqused_k != nullptr) {
        if (a.seqused_q != nullptr) band.seqlen_q = max(0, min(band.seqlen_q, a.seqused_q[w.b]));
        if (a.seqused_k != nullptr) band.seqlen_k = max(0, min(band.seqlen_k, a.seqused_k[w.b]));
        band.off = band.seqlen_k - band.seqlen_q;
    }
    w.band = band;
    w.q_tiles = tiles_of(band.seqlen_q);
    const bool tile_exists = w.kt * kTileRows < band.seqlen_k;  // false only with packed sequences
    w.q_begin = first_q_tile(w.kt, band);
    w.steps_per_head = tile_exists ? q_tiles_of_k_tile(w.kt, band) : 0;
    const int total_steps = group * w.steps_per_head;
    w.n_steps = (split ? min(total_steps, w.t_begin + a.chunk_steps) : total_steps) - w.t_begin;
    // Query tiles are visited in ascending order starting at the diagonal (causal) or at a
    // per-CTA rotation (non-causal), so that CTAs of one head that run together add into
    // different dQ tiles at any moment.
    w.rotation = (kCausal || w.q_tiles == 0) ? 0 : w.kt < w.q_tiles ? w.kt : w.kt % w.q_tiles;
    return w;
}

// The walk over a CTA's steps: query head, query tile, place inside the head.
template <bool kCausal>
struct StepWalk {
    int hq, qt, r;
    __device__ __forceinline__ explicit StepWalk(const FusedWork& w) {
        const int g = w.t_begin < w.steps_per_head || w.steps_per_head == 0 ? 0 : w.t_begin / w.steps_per_head;
        hq = w.first_head + g;
        r = w.t_begin - g * w.steps_per_head;
        qt = r + (kCausal ? w.q_begin : w.rotation);
        if (!kCausal && qt >= w.q_tiles) qt -= w.q_tiles;
    }
    __device__ __forceinline__ void next(const FusedWork& w) {
        ++r;
        ++qt;
        if (!kCausal && qt == w.q_tiles) qt = 0;
        if (r == w.steps_per_head) {
            r = 0;
            ++hq;
            qt = kCausal ? w.q_begin : w.rotation;
        }
    }
};

// kCausal: general form -- the visible band may be bounded (causal mask, sliding window) and the
// sequence lengths need not be multiples of 128; tiles that need it are masked in registers and the
// query tiles of a key tile are walked in ascending order from the first one that sees it.
// false = full attention over whole tiles only: no masking code at all, query sweep rotated per CTA
// (measured: carrying the unused masking code costs the D=64 full-attention kernel 6 %).
// T: storage type of Q/K/V/dO (__half or __nv_bfloat16).  TOut: type of the dK
// and dV outputs (T for the fused path, float for the split path).  kWithDq:
// false turns the kernel into the four-GEMM dK/dV half of the split path.
// kPersist: CTAs take over the tiles of CTAs that have not started (see above).
// kSoftcap: softcapped scores (general form only).  dS then carries the slope 1 - t^2 of the cap, t the tanh: the second
// softmax phase needs P only in that product, so P (1 - t^2) is what it is handed in registers, in P's place.  In 24 bits: P itself
// rounds to 16 almost exactly in a row that few keys dominate, and the product does not, nor does fp16 hold it where the
// scores are far above the cap (S=8192, D=128, cap 15, scores of spread 40, fp16: dQ 9.8e-4 from exact with 16 bits, 3.1e-4 so;
// 130 and 134 us, B=1, Hq=16, Hkv=8, S=4096, D=128, window 1024, cap 30, with the tanh as it was then).
template <typename T, int D, bool kCausal, bool kWithDq, typename TOut, bool kSoftcap = false, bool kPersist = false>
__global__ void __launch_bounds__(512, 1)
fused_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                 const __grid_constant__ CUtensorMap tm_dqacc, const __grid_constant__ FusedArgs a) {
    using C = FusedCfg<D, kSoftcap>;
    static_assert(!kSoftcap || !kPersist, "with capped scores the epilogue reads the work of the first tile again");
    constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wg = warp >> 2;
    auto bar = [&](int i) -> uint32_t { return sbase + C::kOffBar + 8 * i; };
    const uint32_t tmem_slot = sbase + C::kOffBar + 8 * kNumBars;
    const uint32_t abort_flag = tmem_slot + 4;
    const uint32_t answer = sbase + C::kOffBar + 240;
    static_assert(8 * kNumBars + 8 <= 240, "barriers and the answer share 256 bytes");
    const uint32_t work = sbase + C::kOffWork;
    // (a converged warp) the first tile, and the tile after this one; n: how many this CTA has done before
    auto first_tile = [&]() -> FusedWork {
        const FusedWork w = load_work(work);
        __syncwarp();
        if (kPersist && lane == 0) ptx::mbar_arrive(bar(kWorkEmpty));
        return w;
    };
    auto next_tile = [&](uint32_t n, FusedWork* w) -> bool {
        if (!kPersist) return false;
        const uint32_t buf = (n + 1) & 1;
        if (!warp_wait(bar(kWorkFull + buf), (n >> 1) & 1, abort_flag)) return false;
        *w = load_work(work + 128 * buf);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(kWorkEmpty + buf));
        return w->block >= 0;
    };

    if (threadIdx.x == 0) {
        TRACE(0, 0);
        TRACE_GT(0, 1);
    }
    const bool misaligned = (sbase & 1023u) != 0;
    if (threadIdx.x == 0) {
        if (misaligned) atomicCAS(&g_device_error, kDevOk, kDevSmemMisaligned);
        ptx::mbar_init(bar(kKvFull), 1);
        for (int s = 0; s < C::kQStages; ++s) {
            ptx::mbar_init(bar(kQFull + s), 1);
            ptx::mbar_init(bar(kQEmpty + s), 1);
        }
        for (int s = 0; s < C::kDoStages; ++s) {
            ptx::mbar_init(bar(kDoFull + s), 1);
            ptx::mbar_init(bar(kDoEmpty + s), 1);
        }
        // (the math warps arrive once per warp)
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(bar(kStatsFull + s), 1);
            ptx::mbar_init(bar(kStatsEmpty + s), 8);
            ptx::mbar_init(bar(kWorkFull + s), 1);
            ptx::mbar_init(bar(kWorkEmpty + s), kWithDq ? 15 : 11);  // every warp that does the work
        }
        ptx::mbar_init(bar(kAnswer), 1);
        ptx::mbar_init(bar(kSFull), 1);
        ptx::mbar_init(bar(kDpFull), 1);
        ptx::mbar_init(bar(kPReady), 8);
        ptx::mbar_init(bar(kDsReady), 8);
        ptx::mbar_init(bar(kDqFull), 1);
        ptx::mbar_init(bar(kDqEmpty), 4);
        ptx::mbar_init(bar(kDkvFull), 1);
        flag_set(abort_flag, 0);
        ptx::fence_mbar_init();
        TRACE(0, 2);
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, C::kTmemCols);
        ptx::tmem_relinquish();
    }
    // The kernel behind this one (dQ convert) may begin to launch; it waits for our completion itself.  (The dQ kernel
    // of the split path does not: it is let go by the statistics warp, below, once the delta stage has completed.)
    if (kWithDq) ptx::launch_dependents();
    // (all threads: barriers initialised, tensor memory allocated, first tile known)
    auto set_up_done = [&] {
        ptx::tc_fence_before();
        asm volatile("bar.sync 0;" ::: "memory");
        ptx::tc_fence_after();
    };

    // Every role walks the tiles of this CTA, and keeps count of the steps of all of them (g0 in front of a tile): the rings and
    // hand-offs run on from tile to tile.
    if (wg == 0) {
        ptx::setmaxnreg_dec<C::kRegsControl>();
        if (warp == 0) {
            // =================================================== TMA producer
            set_up_done();
            FusedWork w = first_tile();
            uint32_t n = 0, used = 0;  // tiles, tiles with steps
            int g0 = 0;
#pragma unroll 1
            for (bool more = !misaligned; more; ++n) {
                if (lane == 0) {
                    // K and V, when the MMAs of the tile before have completed.  (Tensor maps are [batch][head][row][D]; rows
                    // past the end of a sequence read as zero.)
                    if (w.n_steps > 0 && (used == 0 || bounded_wait<true>(bar(kDkvFull), (used - 1) & 1, abort_flag))) {
                        ptx::mbar_arrive_expect_tx(bar(kKvFull), 2 * C::kOperandBytes);
#pragma unroll
                        for (int bx = 0; bx < C::kBoxes; ++bx) {
                            ptx::tma_load_4d(sbase + C::kOffK + bx * C::kBoxBytes, &tm_k, bar(kKvFull), bx * 64,
                                             w.k_base + w.kt * C::kTile, w.kvh, w.b_coord);
                            ptx::tma_load_4d(sbase + C::kOffV + bx * C::kBoxBytes, &tm_v, bar(kKvFull), bx * 64,
                                             w.k_base + w.kt * C::kTile, w.kvh, w.b_coord);
                        }
                    }
                    if (n == 0) TRACE(0, 3);
                    StepWalk<kCausal> st(w);
#pragma unroll 1
                    for (int t = 0; t < w.n_steps; ++t, st.next(w)) {
                        const int hq = st.hq;
                        const int q_row = w.q_base + st.qt * C::kTile;
                        const int g = g0 + t;
                        const int s = g % C::kQStages;
                        if (!bounded_wait<true>(bar(kQEmpty + s), ((g / C::kQStages) & 1) ^ 1, abort_flag)) break;
                        ptx::mbar_arrive_expect_tx(bar(kQFull + s), C::kOperandBytes);
#pragma unroll
                        for (int bx = 0; bx < C::kBoxes; ++bx) {
                            ptx::tma_load_4d(sbase + C::kOffQ + s * C::kOperandBytes + bx * C::kBoxBytes, &tm_q,
                                             bar(kQFull + s), bx * 64, q_row, hq, w.b_coord);
                        }
                        const int sd = g % C::kDoStages;
                        if (!bounded_wait<true>(bar(kDoEmpty + sd), ((g / C::kDoStages) & 1) ^ 1, abort_flag)) break;
                        ptx::mbar_arrive_expect_tx(bar(kDoFull + sd), C::kOperandBytes);
#pragma unroll
                        for (int bx = 0; bx < C::kBoxes; ++bx) {
                            ptx::tma_load_4d(sbase + C::kOffDO + sd * C::kOperandBytes + bx * C::kBoxBytes, &tm_do,
                                             bar(kDoFull + sd), bx * 64, q_row, hq, w.b_coord);
                        }
                    }
                }
                __syncwarp();
                g0 += w.n_steps;
                used += w.n_steps > 0 ? 1 : 0;
                more = next_tile(n, &w);
            }
        } else if (warp == 1) {
            // ===================================================== MMA issuer
            // The whole warp runs this role converged; MMAs and commits elect their lane inside the asm.
            set_up_done();
            const uint32_t tmem = flag_value(tmem_slot);
            FusedWork w = first_tile();
            TRACE(1, 0);
            constexpr uint32_t kIdSdP = ptx::instr_desc_f16(kBf16, 128, 128, false, false);
            constexpr uint32_t kIdDkv = ptx::instr_desc_f16(kBf16, 128, D, false, true);
            constexpr uint32_t kIdDq = ptx::instr_desc_f16(kBf16, 128, D, true, true);
            // Descriptor low words (address >> 4 | LBO) of every operand tile.
            const uint32_t loK_k = ptx::desc_lo_k_major(sbase + C::kOffK);
            const uint32_t loV_k = ptx::desc_lo_k_major(sbase + C::kOffV);
            const uint32_t loDS_k = ptx::desc_lo_k_major(sbase + C::kOffDS);
            const uint32_t loK_mn = ptx::desc_lo_mn_major(sbase + C::kOffK, C::kBoxBytes);
            const uint32_t loDS_mn = ptx::desc_lo_mn_major(sbase + C::kOffDS, C::kBoxBytes);
            // (g: step counted over all tiles)
            auto sQ = [&](int g) { return sbase + C::kOffQ + (g % C::kQStages) * C::kOperandBytes; };
            auto sDO = [&](int g) { return sbase + C::kOffDO + (g % C::kDoStages) * C::kOperandBytes; };
            auto wait_q = [&](int g) { return warp_wait<false>(bar(kQFull + g % C::kQStages), (g / C::kQStages) & 1, abort_flag); };
            auto wait_do = [&](int g) { return warp_wait<false>(bar(kDoFull + g % C::kDoStages), (g / C::kDoStages) & 1, abort_flag); };
            auto issue_s = [&](int g) {
                const uint32_t loQ = ptx::desc_lo_k_major(sQ(g));
                ptx::mma_ss<D / 16, ptx::KMajor, ptx::KMajor>(tmem + C::kColS, loK_k, loQ, kIdSdP, 0);
                ptx::tc_commit_elect(bar(kSFull));
            };
            auto issue_dp = [&](int g) {
                const uint32_t loDO = ptx::desc_lo_k_major(sDO(g));
                ptx::mma_ss<D / 16, ptx::KMajor, ptx::KMajor>(tmem + C::kColDP, loV_k, loDO, kIdSdP, 0);
                ptx::tc_commit_elect(bar(kDpFull));
            };
            // Asks for the next tile, in front of the last dK and dQ of this one: late enough that tiles go to the CTAs in the order in
            // which these become free, early enough that its K and V, which wait for those MMAs, are there when dK and dV are
            // stored.  (Warp 3 has used the answer before.  Asked for when the last Q and dO were requested, one or two steps
            // earlier: us, causal, 80 heads x 512, D=128 45.3 and 44.4, B=8, 32 x 300 84.2 and 80.9, packed 9 x 2048, 16 heads 277 and 271;
            // full, 80 x 512 56.3 and 57.1; with a mask at D=64 slower than one CTA per tile, now faster.)
            auto request = [&] {
                if constexpr (kPersist) {
                    if (lane == 0) {
                        ptx::mbar_arrive_expect_tx(bar(kAnswer), 16);
                        ptx::request_block(answer, bar(kAnswer));
                    }
                    __syncwarp();
                }
            };
            uint32_t n = 0, used = 0;
            int g0 = 0;
            bool ok = true;
#pragma unroll 1
            for (bool next = !misaligned; next; ++n) {
                const int n_steps = uniform(w.n_steps);
                if (n_steps == 0) request();
                if (n_steps > 0) {
                    ok = warp_wait<false>(bar(kKvFull), used & 1, abort_flag) && wait_q(g0);
                    if (n == 0) TRACE(1, 1);
                    if (ok) {
                        ptx::tc_fence_after();
                        issue_s(g0);
                        if (n == 0) TRACE(1, 2);
                        ok = wait_do(g0);
                        // (dP takes the columns of dQ of the last step)
                        if (kWithDq && D == 128) ok = ok && warp_wait<false>(bar(kDqEmpty), (g0 & 1) ^ 1, abort_flag);
                    }
                    if (ok) {
                        ptx::tc_fence_after();
                        issue_dp(g0);
                        if (n == 0) TRACE(1, 4);
                    }
                    ++used;
                }
#pragma unroll 1
                for (int t = 0; ok && t < n_steps; ++t) {
                    const int g = g0 + t;
                    const bool more = t + 1 < n_steps;
                    const bool traced = n == 0 && t < 6;
                    // dV += P^T dO.  P^T of queries 0-63 sits on columns [0,32) of the S
                    // region, of queries 64-127 on columns [64,96).
                    // (the softmax warps have stored dK / dV of the tile before when they hand over their first P)
                    if (!(ok = warp_wait<false>(bar(kPReady), g & 1, abort_flag))) break;
                    if (traced) TRACE(1, 8 + 8 * t + 0);
                    ptx::tc_fence_after();
                    {
                        const uint32_t loDO = ptx::desc_lo_mn_major(sDO(g), C::kBoxBytes);
                        ptx::mma_ts_8<ptx::TmemHalves, ptx::MnMajor>(tmem + C::kColDV, tmem + C::kColS, loDO, kIdDkv, t > 0 ? 1u : 0u);
                    }
                    ptx::tc_commit_elect(bar(kDoEmpty + g % C::kDoStages));
                    if (traced) TRACE(1, 8 + 8 * t + 1);
                    // S of the next step may overwrite S/P of this one: MMAs execute in issue order.
                    if (more) {
                        if (!(ok = wait_q(g + 1))) break;
                        ptx::tc_fence_after();
                        issue_s(g + 1);
                    }
                    if (traced) TRACE(1, 8 + 8 * t + 2);
                    // dK += dS^T Q
                    if (!(ok = warp_wait<false>(bar(kDsReady), g & 1, abort_flag))) break;
                    if (traced) TRACE(1, 8 + 8 * t + 3);
                    if (!more) request();
                    ptx::tc_fence_after();
                    {
                        const uint32_t loQ = ptx::desc_lo_mn_major(sQ(g), C::kBoxBytes);
                        ptx::mma_ss_8<ptx::KMajor, ptx::MnMajor>(tmem + C::kColDK, loDS_k, loQ, kIdDkv, t > 0 ? 1u : 0u);
                    }
                    ptx::tc_commit_elect(bar(kQEmpty + g % C::kQStages));
                    if (kWithDq) {
                        if (D == 64) {  // own dQ region: wait for the drain of the step before
                            if (!(ok = warp_wait<false>(bar(kDqEmpty), (g & 1) ^ 1, abort_flag))) break;
                            ptx::tc_fence_after();
                        }
                        // dQ = dS K  (overwrites dP when D = 128: it was consumed before kDsReady)
                        ptx::mma_ss_8<ptx::MnMajor, ptx::MnMajor>(tmem + C::kColDQ, loDS_mn, loK_mn, kIdDq, 0);
                        ptx::tc_commit_elect(bar(kDqFull));
                    }
                    if (traced) TRACE(1, 8 + 8 * t + 4);
                    if (more) {
                        if (!(ok = wait_do(g + 1))) break;
                        if (traced) TRACE(1, 8 + 8 * t + 5);
                        if (kWithDq && D == 128) {  // dP of the next step reuses the dQ columns
                            if (!(ok = warp_wait<false>(bar(kDqEmpty), g & 1, abort_flag))) break;
                        }
                        if (traced) TRACE(1, 8 + 8 * t + 6);
                        ptx::tc_fence_after();
                        issue_dp(g + 1);
                        if (traced) TRACE(1, 8 + 8 * t + 7);
                    }
                }
                if (!ok) break;
                if (n_steps > 0) ptx::tc_commit_elect(bar(kDkvFull));
                if (n == 0) TRACE(1, 62);
                g0 += n_steps;
                next = next_tile(n, &w);
            }
            TRACE_VALUE(1, 63, n);  // tiles of this CTA (every other stamp but the drain's last and the CTA's end is of the first)
        } else if (warp == 2) {
            // ============================================== row statistics
            // One warp fetches the statistics of the next step's 128 query rows while the math warps work and
            // hands them over in shared memory, two steps deep.  (A softmax warpgroup that fetched its own spent
            // 300-700 clk of every step on it.)  P = exp2(x - m) * r = exp2(x + (log2 r - m)); a row past the end
            // of the sequence gets -inf, which makes its P, and with it dS, exactly zero.
            // The statistics come from the delta kernel, which may still be running (programmatic launch); Q, K,
            // V, dO are inputs of the call, so the TMA and MMA warps did not have to wait.
            float* stats = reinterpret_cast<float*>(smem + C::kOffStats);
            float neg[4], ndel[4];
            auto fetch = [&](const FusedWork& w, const StepWalk<kCausal>& st) {
                const int64_t row0 = int64_t(w.b_coord * a.heads_q + st.hq) * a.sidecar_rows + w.q_base;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int qi = st.qt * C::kTile + k * 32 + lane;
                    const bool valid = !kCausal || qi < w.band.seqlen_q;
                    neg[k] = -INFINITY;
                    ndel[k] = 0.0f;
                    if (valid && a.stats != nullptr) {
                        const float2 v = a.stats[row0 + qi];
                        neg[k] = v.x;
                        ndel[k] = v.y;
                    } else if (valid) {
                        const float* v = a.sidecar + (row0 + qi) * 3;
                        neg[k] = __log2f(v[1]) - v[0];
                        ndel[k] = -v[2];
                    }
                }
            };
            if (lane == 0) {
                ptx::prefetch_tensormap(&tm_k);
                ptx::prefetch_tensormap(&tm_v);
                ptx::prefetch_tensormap(&tm_q);
                ptx::prefetch_tensormap(&tm_do);
            }
            __syncwarp();
            set_up_done();
            FusedWork w = first_tile();
            ptx::grid_dependency_wait();
            if (!kWithDq) ptx::launch_dependents();
            uint32_t n = 0;
            int g = 0;
            bool ok = true;
#pragma unroll 1
            for (bool more = !misaligned; more; ++n) {
                StepWalk<kCausal> st(w);
                if (w.n_steps > 0) fetch(w, st);
#pragma unroll 1
                for (int t = 0; t < w.n_steps; ++t, ++g) {
                    const int buf = g & 1;
                    if (!(ok = warp_wait(bar(kStatsEmpty + buf), ((g >> 1) & 1) ^ 1, abort_flag))) break;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        stats[buf * 128 + k * 32 + lane] = neg[k];
                        stats[256 + buf * 128 + k * 32 + lane] = ndel[k];
                    }
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(bar(kStatsFull + buf));
                    if (t + 1 < w.n_steps) {
                        st.next(w);
                        fetch(w, st);
                    }
                }
                if (!ok) break;
                more = next_tile(n, &w);
            }
        } else {
            // ================================================== which tile next
            {
                const FusedWork w = fused_work<kCausal>(a, int(blockIdx.x));
                if (lane == 0) store_work(work, w);
            }
            set_up_done();
            if (kPersist && !misaligned) {
#pragma unroll 1
                for (uint32_t n = 0, answers = 0;; ++n) {  // the work of tile n + 1
                    const uint32_t buf = (n + 1) & 1;
                    FusedWork w;
                    bool ok;
                    while ((ok = warp_wait(bar(kAnswer), answers & 1, abort_flag))) {
                        ++answers;
                        const int block = ptx::answered_block(answer);
                        ptx::fence_proxy_async_smem();  // (it is written through the async proxy again)
                        if (block >= 0) w = fused_work<kCausal>(a, block);
                        w.block = block;
                        // (packed sequences: the grid is sized for the longest one, and many blocks have no rows)
                        if (block < 0 || w.kt * C::kTile < w.slot_k) break;
                        __syncwarp();
                        if (lane == 0) {
                            ptx::mbar_arrive_expect_tx(bar(kAnswer), 16);
                            ptx::request_block(answer, bar(kAnswer));
                        }
                    }
                    // (that of tile n - 1 has been read)
                    if (!ok || (n >= 1 && !warp_wait(bar(kWorkEmpty + buf), ((n - 1) >> 1) & 1, abort_flag))) break;
                    if (lane == 0) store_work(work + 128 * buf, w);
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(bar(kWorkFull + buf));
                    if (w.block < 0) break;
                }
            }
        }
    } else if (wg == 1 || wg == 2) {
        // ============================================ softmax / dS warpgroups
        if (!kWithDq) ptx::setmaxnreg_inc<C::kRegsComputeNoDq>();
        else if (C::kRegsCompute < 128) ptx::setmaxnreg_dec<C::kRegsCompute>();
        else if (C::kRegsCompute > 128) ptx::setmaxnreg_inc<C::kRegsCompute>();
        set_up_done();
        const uint32_t tmem = flag_value(tmem_slot);
        FusedWork w = first_tile();
        {
            const int half = wg - 1;          // which 64 queries of the tile
            const int j = threadIdx.x & 127;  // key row inside the tile == TMEM lane
            const uint32_t tl = tmem + (uint32_t((warp & 3) * 32) << 16);
            const uint32_t s_cols = tl + C::kColS + half * 64;
            const uint32_t dp_cols = tl + C::kColDP + half * 64;
            const uint32_t stats = sbase + C::kOffStats + half * 256;  // this half's 64 queries
            const uint64_t scale2 = ptx::f2_pack(a.scale_log2, a.scale_log2);
            const uint64_t post2 = ptx::f2_pack(a.softcap_post, a.softcap_post);
            const uint64_t pre2 = ptx::f2_pack(a.softcap_pre * ptx::kTanhArg, a.softcap_pre * ptx::kTanhArg);
            // what dP - delta is multiplied with: P as it is handed to the MMA, in 16 bits, or P (1 - t^2), in 24 (pack24)
            uint32_t ppk[kSoftcap ? 48 : 32];
            // one arrival per warp: every lane's accesses are ordered before it by the fence and the warp barrier
            auto arrive = [&](int which) {
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar(which));
            };
            bool ok = true;
            uint32_t n = 0, used = 0;
            int g = 0;  // step, counted over all tiles
#pragma unroll 1
            for (bool more = !misaligned; more; ++n) {
                w.n_steps = uniform(w.n_steps);
                w.kt = uniform(w.kt);
                w.q_begin = uniform(w.q_begin);
                w.steps_per_head = uniform(w.steps_per_head);
                w.rotation = uniform(w.rotation);
                w.q_tiles = uniform(w.q_tiles);
                StepWalk<kCausal> st(w);
#pragma unroll 1
                for (int t = 0; t < w.n_steps; ++t, ++g, st.next(w)) {
                    const bool traced = warp == 4 && n == 0 && t < 7;
                    if (traced && t == 3) TRACE(2, 0);
                    const int qt = st.qt;
                    const int buf = g & 1;
                    const uint32_t negp = stats + buf * 512;
                    const uint32_t delp = stats + 1024 + buf * 512;
                    if (!(ok = warp_wait2(bar(kStatsFull + buf), (g >> 1) & 1, bar(kSFull), g & 1, abort_flag))) break;
                    if (traced) TRACE(2, 4 + 8 * t + 1);
                    ptx::tc_fence_after();
                    // A tile that crosses an edge of the band or holds keys past the end of the sequence is
                    // masked: element (key j, query i) survives iff mask_from <= i <= mask_to.
                    const bool diagonal = kCausal && tile_needs_mask(w.kt, qt, w.band);
                    int mask_from = 0, mask_to = 0;  // set only on masked tiles
                    // ---- P^T = exp2(S^T * scale_log2 + neg_i), masked as above: 32 scores from column `first` of this half on;
                    // p: their P, two in a register
                    // (two copies of the code, so that unmasked tiles carry no per-element test)
                    auto softmax_cols = [&](int first, const uint32_t* r, uint32_t* p, auto masked_tag) {
                        constexpr bool kMasked = decltype(masked_tag)::value;
#pragma unroll
                        for (int e = 0; e < 32; e += 4) {
                            float slope_p[4];
                            const ptx::F4Pairs n4 = ptx::f2_ld_shared(negp + (first + e) * 4);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const uint64_t neg2 = h == 0 ? n4.lo : n4.hi;
                                const int el = e + 2 * h;
                                // score in log2 units, relative to the row's reference: s * scale*log2e + (log2 r - m), or the
                                // capped score + (log2 r - m)
                                const uint64_t s2 = ptx::f2_pack(__uint_as_float(r[el]), __uint_as_float(r[el + 1]));
                                uint64_t t2 = 0;
                                if constexpr (kSoftcap) t2 = ptx::tanh_mixed<C::kTanhFmaPairs>(ptx::f2_mul(s2, pre2), el / 2);
                                // (exp2_poly for a part of these changed nothing: B=4,H=16,S=4096,D=64 791, 792, 795, 810 us for 0 to 3
                                // pairs of 8)
                                float2 p2 = ptx::f2_unpack(kSoftcap ? ptx::f2_fma(t2, post2, neg2) : ptx::f2_fma(s2, scale2, neg2));
                                p2.x = ptx::ex2_approx(p2.x);
                                p2.y = ptx::ex2_approx(p2.y);
                                float2 w2;
                                if constexpr (kSoftcap) {
                                    const float2 tt = ptx::f2_unpack(t2);
                                    w2 = ptx::f2_unpack(ptx::f2_mul(ptx::f2_pack(p2.x, p2.y),
                                                                    ptx::f2_pack(fmaf(-tt.x, tt.x, 1.0f), fmaf(-tt.y, tt.y, 1.0f))));
                                }
                                if (kMasked) {
                                    const int i = half * 64 + first + el;
                                    const bool sees0 = i + 0 >= mask_from && i + 0 <= mask_to, sees1 = i + 1 >= mask_from && i + 1 <= mask_to;
                                    p2.x = sees0 ? p2.x : 0.0f;
                                    p2.y = sees1 ? p2.y : 0.0f;
                                    if constexpr (kSoftcap) {
                                        w2.x = sees0 ? w2.x : 0.0f;
                                        w2.y = sees1 ? w2.y : 0.0f;
                                    }
                                }
                                p[el / 2] = ptx::Pack2<T>::pack(p2.x, p2.y);
                                if constexpr (kSoftcap) {
                                    slope_p[2 * h] = w2.x;
                                    slope_p[2 * h + 1] = w2.y;
                                }
                            }
                            if constexpr (kSoftcap) ptx::pack24(slope_p, &ppk[(first + e) / 4 * 3]);
                        }
                    };
                    auto softmax_phase = [&](auto masked_tag) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            uint32_t r[32], capped_p[16];  // (capped_p: P where ppk holds P (1 - t^2))
                            uint32_t* p = kSoftcap ? capped_p : &ppk[c * 16];
                            ptx::tmem_ld32(s_cols + c * 32, r);
                            ptx::tmem_ld_wait();
                            softmax_cols(c * 32, r, p, masked_tag);
                            ptx::tmem_st16(s_cols + c * 16, p);  // P chunk c -> columns [16c, 16c+16) of this half's S columns (already read)
                        }
                    };
                    if (diagonal) {
                        query_range_of_key(w.kt * C::kTile + j, qt * C::kTile, w.band, &mask_from, &mask_to);
                        softmax_phase(std::true_type{});
                    } else {
                        softmax_phase(std::false_type{});
                    }
                    if (traced) TRACE(2, 4 + 8 * t + 2);
                    ptx::tmem_st_wait();
                    arrive(kPReady);
                    if (traced) TRACE(2, 4 + 8 * t + 3);
                    // ---- dS^T = P^T * (dP^T - delta_i), stored [key][query] in the 128-byte swizzle
                    if (!(ok = warp_wait(bar(kDpFull), g & 1, abort_flag))) break;
                    if (traced) TRACE(2, 4 + 8 * t + 4);
                    // (the dS buffer is free: dP was issued behind dK and dQ of the step before, the readers of its dS,
                    // and the barrier just passed completes only when every MMA issued before it has)
                    ptx::tc_fence_after();
                    const uint32_t ds_row = sbase + C::kOffDS + half * C::kBoxBytes + j * 128;
                    auto ds_chunk = [&](int c, const uint32_t* r) {
#pragma unroll
                        for (int e = 0; e < 32; e += 8) {
                            uint32_t o[4];
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const ptx::F4Pairs d4 = ptx::f2_ld_shared(delp + (c * 32 + e + 4 * h) * 4);  // -delta
                                const int el = e + 4 * h;
                                float slope_p[4];
                                if constexpr (kSoftcap) ptx::unpack24(&ppk[c * 24 + el / 4 * 3], slope_p);
#pragma unroll
                                for (int g = 0; g < 2; ++g) {
                                    const float2 p = kSoftcap ? make_float2(slope_p[2 * g], slope_p[2 * g + 1]) : ptx::Pack2<T>::unpack(ppk[c * 16 + el / 2 + g]);
                                    const uint64_t dp2 = ptx::f2_pack(__uint_as_float(r[el + 2 * g]), __uint_as_float(r[el + 2 * g + 1]));
                                    const float2 ds = ptx::f2_unpack(ptx::f2_mul(ptx::f2_pack(p.x, p.y), ptx::f2_add(dp2, g == 0 ? d4.lo : d4.hi)));
                                    o[2 * h + g] = ptx::Pack2<T>::pack(ds.x, ds.y);
                                }
                            }
                            const int chunk = c * 4 + e / 8;  // 16-byte chunk inside this half's box
                            const uint32_t addr = ds_row + ((chunk ^ (j & 7)) << 4);
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(o[0]),
                                         "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                        }
                    };
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        uint32_t r[32];
                        ptx::tmem_ld32(dp_cols + c * 32, r);
                        ptx::tmem_ld_wait();
                        ds_chunk(c, r);
                    }
                    if (traced) TRACE(2, 4 + 8 * t + 6);
                    ptx::fence_proxy_async_smem();
                    arrive(kDsReady);
                    if (lane == 0) ptx::mbar_arrive(bar(kStatsEmpty + buf));
                    if (traced) TRACE(2, 4 + 8 * t + 7);
                }
                // ---- epilogue: the first warpgroup writes dK (scaled), the second dV
                if (!ok) break;
                if constexpr (kSoftcap) w = load_work(work);  // (what only the epilogue needs is not held in registers before)
                const int w4 = warp & 3;  // which 32 rows of the tile
                const bool has_steps = w.n_steps > 0;
                const int64_t slab = int64_t(w.slab * 2 + half) * (C::kTile * D) + w4 * 32 * D;
                const int rows = w.slot_k - (w.kt * C::kTile + w4 * 32);
                // (rows between the used length and the end of the slot hold exact zeros)
                TOut* out = reinterpret_cast<TOut*>(half == 0 ? a.dk : a.dv) + w.b_coord * a.kv_strides.batch +
                            w.kvh * a.kv_strides.head + int64_t(w.k_base + w.kt * C::kTile + w4 * 32) * a.kv_strides.row;
                more = next_tile(n, &w);  // (while the last MMAs of this one run)
                if (has_steps && !(ok = warp_wait(bar(kDkvFull), used & 1, abort_flag))) break;
                if (warp == 4 && n == 0) TRACE(2, 60);
                if (has_steps) {
                    // Every MMA of the tile has completed.  Each warp stages its 32 key rows in shared memory and stores them again in
                    // whole lines: over the dead Q / dO / dS^T buffers, 512 contiguous bytes (or two rows) per instruction, or, where
                    // the next tile's Q and dO are being loaded, over its own rows of dS^T, 128 bytes of each row at a time.
                    // (Stores through the copy engine queue behind the drain's last reduce-adds, about 2700 clk at D=128; a thread
                    // storing its own row straight from registers writes 16 bytes per line and instruction.)
                    ++used;
                    ptx::tc_fence_after();
                    const float mul = half == 0 ? a.scale : 1.0f;
                    const uint32_t col0 = tl + (half == 0 ? C::kColDK : C::kColDV);
                    // rows of element type O at dst, `pitch` elements apart, of which the first `rows_here` are written
                    auto store_rows = [&](auto tag, void* dst_rows, int64_t pitch, int rows_here) {
                        using O = decltype(tag);
                        constexpr int kPass = kPersist ? 128 : D * int(sizeof(O));  // bytes of a row
                        constexpr int kCols = kPass / int(sizeof(O));
                        constexpr int kChunks = kPass / 16;
                        constexpr int kPerLoad = 32 * int(sizeof(O)) / 16;  // 16-byte chunks of 32 columns
                        constexpr int kRowsAtOnce = 32 / kChunks;
                        const uint32_t scratch = sbase + (kPersist ? C::kOffDS + half * C::kBoxBytes + w4 * 32 * kPass
                                                                   : C::kOffQ + (half * 4 + w4) * 32 * kPass);
                        const int sub = lane / kChunks, ch = lane % kChunks;
                        O* dst = static_cast<O*>(dst_rows) + ch * (16 / int(sizeof(O)));
#pragma unroll 1
                        for (int col = 0; col < D; col += kCols) {
#pragma unroll
                            for (int c = 0; c < kCols / 32; ++c) {
                                uint32_t r[32];
                                ptx::tmem_ld32(col0 + col + c * 32, r);
                                ptx::tmem_ld_wait();
#pragma unroll
                                for (int e = 0; e < kPerLoad; ++e) {
                                    uint32_t o[4];
#pragma unroll
                                    for (int h = 0; h < 4; ++h) {
                                        if constexpr (sizeof(O) == 4) {
                                            o[h] = __float_as_uint(__uint_as_float(r[4 * e + h]) * mul);
                                        } else {
                                            o[h] = ptx::Pack2<O>::pack(__uint_as_float(r[8 * e + 2 * h]) * mul, __uint_as_float(r[8 * e + 2 * h + 1]) * mul);
                                        }
                                    }
                                    const int chunk = (c * kPerLoad + e) ^ (lane & 7);  // (spread over the banks)
                                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                                 ::"r"(scratch + lane * kPass + chunk * 16), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                                }
                            }
                            __syncwarp();
#pragma unroll 8
                            for (int row = sub; row < 32; row += kRowsAtOnce) {
                                uint4 v;
                                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                             : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                                             : "r"(scratch + row * kPass + ((ch ^ (row & 7)) << 4)) : "memory");
                                if (row < rows_here) *reinterpret_cast<uint4*>(dst + row * pitch + col) = v;
                            }
                            __syncwarp();
                        }
                    };
                    if (kWithDq && a.chunk_steps > 0) {
                        // a share of a split tile: the partial sums go to this CTA's slabs (slab 2x: dK, 2x+1: dV).  fp32, but
                        // fp16 for fp16 inputs where the tiles are fewer than the SMs: the bytes written, not the arithmetic,
                        // bound this epilogue.  (With as many tiles as SMs, fp16 slabs had taken dK and dV, whose sums stay in
                        // tensor memory when their tile is not split, 1.16 and 1.23 times as far from the exact values.)
                        if (!kBf16 && a.slabs_f16) store_rows(__half{}, static_cast<__half*>(a.dkv_slabs) + slab, D, 32);
                        else store_rows(float{}, static_cast<float*>(a.dkv_slabs) + slab, D, 32);
                    } else {
                        store_rows(TOut{}, out, a.kv_strides.row, rows);
                    }
                } else if (a.chunk_steps == 0) {
                    // nobody attends to these keys (possible with a left-bounded window), but dK / dV still owe zeros
                    if (lane < rows) {
                        uint4* d4 = reinterpret_cast<uint4*>(out + lane * a.kv_strides.row);
#pragma unroll
                        for (int e = 0; e < int(D * sizeof(TOut) / 16); ++e) d4[e] = make_uint4(0u, 0u, 0u, 0u);
                    }
                }
                if (warp == 4 && n == 0) TRACE(2, 61);
            }
        }
    } else {
        // ==================================================== dQ drain warpgroup
        if (!kWithDq) {
            ptx::setmaxnreg_dec<C::kRegsControl>();
            set_up_done();
        } else {
            if (C::kRegsDrain > 128) ptx::setmaxnreg_inc<C::kRegsDrain>();
            set_up_done();
            const uint32_t tmem = flag_value(tmem_slot);
            FusedWork w = first_tile();
            {
                const int qd = warp & 3;
                const uint32_t tl = tmem + (uint32_t(qd * 32) << 16);
                const uint32_t stage = sbase + C::kOffStage + qd * 2 * C::kStageBoxBytes;
                bool pending = false;
                // the accumulators are cleared by the delta kernel: do not add into them before it is done
                ptx::grid_dependency_wait();
                bool ok = true;
                uint32_t n = 0;
                int g = 0;
#pragma unroll 1
                for (bool more = !misaligned; more; ++n) {
                    StepWalk<kCausal> st(w);
#pragma unroll 1
                    for (int t = 0; t < w.n_steps; ++t, ++g, st.next(w)) {
                        const bool traced = warp == 12 && n == 0 && t < 12;
                        const int q_row = st.qt * C::kTile + qd * 32;  // row inside the head
                        const int q_head = w.b_coord * a.heads_q + st.hq;
                        if (!(ok = warp_wait(bar(kDqFull), g & 1, abort_flag))) break;
                        if (traced) TRACE(3, 4 + 4 * t + 0);
                        ptx::tc_fence_after();
                        // pull the whole dQ tile row into registers and hand the columns back at once
                        uint32_t r[D / 32][32];
#pragma unroll
                        for (int c = 0; c < D / 32; ++c) ptx::tmem_ld32(tl + C::kColDQ + c * 32, r[c]);
                        ptx::tmem_ld_wait();
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(bar(kDqEmpty));
                        if (traced) TRACE(3, 4 + 4 * t + 1);
#pragma unroll
                        for (int hf = 0; hf < D / 64; ++hf) {
                            if (pending) {
                                if (lane == 0) ptx::bulk_wait_group_read<0>();
                                __syncwarp();
                            }
#pragma unroll
                            for (int bx = 0; bx < 2; ++bx) {
                                const uint32_t row_addr = stage + bx * C::kStageBoxBytes + lane * 128;
#pragma unroll
                                for (int c = 0; c < 8; ++c) {
                                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                                 ::"r"(row_addr + ((c ^ (lane & 7)) << 4)), "r"(r[hf * 2 + bx][4 * c]),
                                                   "r"(r[hf * 2 + bx][4 * c + 1]), "r"(r[hf * 2 + bx][4 * c + 2]),
                                                   "r"(r[hf * 2 + bx][4 * c + 3])
                                                 : "memory");
                                }
                            }
                            ptx::fence_proxy_async_smem();
                            __syncwarp();
                            // accumulator map: [batch*head][row][D]; rows past the sequence end are dropped
                            if (lane == 0 && q_row < w.band.seqlen_q) {
                                ptx::tma_reduce_add_3d(&tm_dqacc, stage, hf * 64, w.q_base + q_row, q_head);
                                ptx::tma_reduce_add_3d(&tm_dqacc, stage + C::kStageBoxBytes, hf * 64 + 32, w.q_base + q_row, q_head);
                                ptx::bulk_commit_group();
                            }
                            pending = true;
                        }
                        if (traced) TRACE(3, 4 + 4 * t + 2);
                    }
                    if (!ok) break;
                    more = next_tile(n, &w);
                }
                if (lane == 0) ptx::bulk_wait_group<0>();
                if (warp == 12) TRACE(3, 59);
            }
        }
    }

    // ---- teardown: everybody meets, then the allocating warp frees TMEM
    if (threadIdx.x == 0) ptx::grid_dependency_wait();
    __syncwarp();
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(flag_value(tmem_slot), C::kTmemCols);
    }
    if (threadIdx.x == 0) {
        TRACE(0, 63);
        TRACE_GT(0, 62);
    }
}

}  // namespace fa3b200
