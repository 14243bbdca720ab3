// Attention forward for sm_100a: O = softmax(Q K^T * scale) V and the log-sum-exp of every row, the
// two tensors the backward needs next to Q, K, V.  Same tile geometry, masks, layouts and packed
// sequences as the backward kernels (geometry.h).
//
// One CTA owns one (batch, query head) and TWO neighbouring 128-row query tiles, A and B.  Both Q tiles
// stay in shared memory, K and V tiles stream through rings and are used by both query tiles, and each
// query tile has its own softmax warpgroup, score buffer and output accumulator in tensor memory.  Per
// key tile and query tile:
//
//     S  = Q K^T          [query i on TMEM lanes, key j on columns]           SS MMA
//     m  = max(m, rowmax S),  P = exp2((S - m) * scale*log2e),  l = l*alpha + rowsum P
//          (thread i owns query row i: no shuffles; P goes back to tensor memory as 16-bit pairs)
//     O += P V            A = P from TMEM, B = V (MN-major)                   TS MMA
//
// The two query tiles alternate on the tensor pipe: while the softmax warpgroup of tile A works on
// S_A(t), the pipe computes S_B(t) and P_B V, and the other way round.  At D=128 P is written over S, so
// S(t+1) follows P(t) V; at D=64 P has columns of its own and S(t+1) is computed while the softmax of
// step t runs.  P V starts on the first 64 keys while the exponentials of the others are computed.
// The running maximum is updated lazily: a row keeps its reference maximum until the new maximum
// exceeds it by more than 2^8, so P stays below 256 and the accumulator only has to be rescaled
// (tensor memory -> registers -> tensor memory) on the rare steps where some row of a warp moves
// its reference.  The result is exact: O and l carry the same factor, which cancels in O / l.
//
// What bounds it: the chain S -> softmax -> P V of a tile.  An iteration (both tiles, one key tile) takes 3030
// clk at D=128 (2048 of MMA) and 2500 at D=64 (1280 of MMA, 2048 of exponentials at 16 per clk).  A lone
// busy warp of a scheduler issues an instruction every 1.9 clk, so the softmax is written for few
// instructions: packed two-value arithmetic, three-input maxima, at D=64 every eighth exponential on the FMA
// pipe (more of them cost more issue slots than they free), votes instead of divergent polling at the
// barriers (see warp_wait), P's barrier asked for ahead of its use.  TFLOP/s, back to back, before and
// after: B=4, H=16, S=4096 full, D=64 567 and 823, D=128 930-990 and 1155-1170 (there the power limit holds the
// clock near 1.6 GHz); B=2, Hq=32, Hkv=8, S=8192 causal, D=128 857 and 1063.
//
// With at least two pairs of query tiles per SM (kPersist) CTAs take over the pairs of CTAs that have not started, as in the
// backward; the rule and what it measured stand in cta_order.h.
//
// When the pairs are too few to fill the GPU a cluster of 2, 4 or 8 CTAs shares the key tiles of a pair
// (plan_fwd) and merges the partial outputs through distributed shared memory.
//
// Tensor-memory ledger: S_A [0,128)  S_B [128,256)  O_A [256,256+D)  O_B [256+D,256+2D); at D=64 also
// P_A [384,448)  P_B [448,512).
// Shared-memory ledger: Q_A, Q_B resident (2 x D*256), K and V rings of two stages (D=128) or three (D=64),
// partial row statistics 2 KiB, mbarriers 288, work of a pair 256: 199,200 bytes at D=128, 133,664 at D=64; with pairs taken over
// 32 KiB more for their O: 232,448 and 166,912.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "fused_bwd_kernel.cuh"
#include "geometry.h"
#include "ptx.cuh"

namespace fa3b200 {

struct FwdArgs {
    void* out;                // [B,Hq,Sq,D] or [B,Sq,Hq,D] (or [total_q,Hq,D]), see o_strides
    float* lse;               // [B,Hq,Sq] natural log ([Hq,total_q] when packed)
    TensorStrides o_strides;  // element strides of out
    int batch;
    int heads_q;
    int heads_kv;
    Band band;                // sequence lengths and the visible band; maxima when packed
    const int* cu_seqlens_q;  // non-null: packed sequences, see FusedArgs
    const int* cu_seqlens_k;
    const int* seqused_q;     // non-null: used lengths per batch entry, see FusedArgs; rows behind them
    const int* seqused_k;     // get out = 0 and lse = -inf
    int lse_rows;             // rows per head of lse (seqlen_q, or total_q when packed)
    float scale_log2;         // softmax scale * log2(e)
    float softcap_pre;        // softcap variant: scores become softcap_post * tanh(score * softcap_pre),
    float softcap_post;       // with softcap_pre = scale / softcap and softcap_post = softcap * log2(e)
    FastDiv bh;               // batch * heads_q
    FastDiv heads;            // heads_q
    FastDiv group;            // heads_q / heads_kv
    int split_shift;          // log2(splits)
    int splits;               // CTAs per pair of query tiles: a cluster of so many shares its key tiles
    int fold;                 // pairs are the last and the first query tile, the last but one and the second, ... (no split)
    int staged_store;         // out goes through tm_o (not packed: the copy engine cannot clip at a sequence's end)
};

template <int D>
struct FwdCfg {
    static constexpr int kTile = 128;
    static constexpr int kThreads = 384;
    static constexpr int kBoxBytes = 128 * 128;
    static constexpr int kBoxes = D / 64;
    static constexpr int kOperandBytes = kBoxes * kBoxBytes;
    static constexpr int kStages = D == 64 ? 3 : 2;
    static constexpr int kOffQ = 0;                                  // two query tiles
    static constexpr int kOffK = 2 * kOperandBytes;
    static constexpr int kOffV = kOffK + kStages * kOperandBytes;
    static constexpr int kOffMerge = kOffK;                          // split: [2 tiles][128 rows][D] fp32 over the dead rings
    static constexpr int kOffStats = kOffV + kStages * kOperandBytes;  // split: [2 tiles][128 rows] {m, l}
    static constexpr int kOffBar = kOffStats + 2 * 128 * 8;
    static constexpr int kOffWork = kOffBar + 288;                   // two buffers
    static constexpr int kOffOut = kOffBar + 1024;                   // tiles taken over: [8 warps][32 rows][64 columns] of O
    static constexpr int kSmemBytes = kOffWork + 256;
    static constexpr int kSmemBytesPersist = kOffOut + 8 * 4096;
    static_assert(kOffOut % 1024 == 0, "swizzled region");
    static_assert(kSmemBytesPersist <= 232448, "shared-memory ledger exceeds 227 KiB");
    static_assert(2 * 128 * D * 4 <= kOffStats - kOffMerge, "partial outputs do not fit over the rings");
    // P in columns of its own where they are free (D=64): the scores of the next key tile are then computed
    // while the exponentials of this one are, because the score columns are free once they are in registers
    static constexpr bool kOwnP = D == 64;
    static constexpr int kTmemCols = 512;
    static constexpr int kColS = 0;                     // + 128 per query tile
    static constexpr int kColO = 256;                   // + D per query tile
    static constexpr int kColP = kOwnP ? 384 : kColS;   // + kPStride per query tile
    static constexpr int kPStride = kOwnP ? 64 : 128;
    static_assert(kColO + 2 * D <= (kOwnP ? kColP : kTmemCols) && kColP + 2 * 64 <= kTmemCols, "tensor-memory ledger exceeds 512 columns");
    static constexpr float kRescaleThreshold = 8.0f;  // log2 units
    // Of every 8 pairs of exponentials, how many go to the FMA pipe (exp2_poly) instead of the special-function unit.
    // us per call of B=4, H=16, S=4096 full for 0, 1, 2, 3 of 8: D=64 348, 338, 355, 371; D=128 486, 492, 490, 500.
    static constexpr int kPolyPairs = D == 64 ? 1 : 0;
    // ... and of every 8 pairs of tanh of capped scores (tanh_mixed): us of the forwards named there for 2, 4, 5, 8 of 8: 84.5, 81,
    // 80, 87; 247, 227, 228, 259 (before the loop was compiled as uniform: 78.5 and 222 now).  6 of 8 spill at D=128.
    static constexpr int kTanhFmaPairs = 5;
    // setmaxnreg split: the kernel starts with 168 registers per thread (384 threads); the producer /
    // MMA warpgroup gives most of its share to the two softmax warpgroups, which hold a whole score
    // row (128 values) in registers
    static constexpr int kRegsControl = 72;
    static constexpr int kRegsSoftmax = 216;
    static_assert(kRegsControl + 2 * kRegsSoftmax <= 504, "more registers than the CTA was launched with (168 x 384)");
};

enum FwdBar : int {
    kFwdQFull = 0,    // per query tile
    kFwdKFull = 2,    // up to 3 stages
    kFwdKEmpty = 5,   // up to 3 stages
    kFwdVFull = 8,    // up to 3 stages
    kFwdVEmpty = 11,  // up to 3 stages
    kFwdSFull = 14,   // per query tile
    kFwdSFree = 16,   // per query tile: the scores are in registers (kOwnP)
    kFwdPFirst = 18,  // per query tile: the first half of P is written
    kFwdPReady = 20,  // per query tile: all of P is written
    kFwdPvDone = 22,  // per query tile
    kFwdAllDone = 24, // every MMA of the CTA has completed
    kFwdAnswer = 25,     // tiles taken over, as in the backward: which block comes next
    kFwdWorkFull = 26,   // 2 buffers
    kFwdWorkEmpty = 28,  // 2 buffers
    kFwdQEmpty = 30,     // per query tile: its last scores have been computed
    kFwdNum = 32,
};

// Which query tiles and keys a CTA works on.  One warp works it out and hands it to the others in shared memory.
struct alignas(16) FwdWork {
    int block;           // place in the launch order, -1: there is none
    int rank, hq, kvh, b, b_coord, q_base, k_base;
    int tile[2];         // query tiles A and B
    int slot_q;          // rows of out this batch entry owns
    int t_begin, n_iter; // the CTA walks key tiles t_begin .. t_begin + n_iter - 1;
    int lo[2], hi[2];    // query tile x takes part in iterations lo[x] .. hi[x] - 1 (none when it sees no key or
                         // lies past the end of its sequence)
    Band band;
    __device__ __forceinline__ bool active(int x, int it) const { return it >= lo[x] && it < hi[x]; }
};

// (behind grid_dependency_wait)
template <bool kMasked>
__device__ __forceinline__ FwdWork fwd_work(const FwdArgs& a, int block) {
    FwdWork w;
    w.block = block;
    const int unit = block >> a.split_shift;
    w.rank = block & (a.splits - 1);        // == rank in the cluster
    const int slot = fast_div(unit, a.bh);
    // heaviest query tiles (most visible keys) are launched first (packed: of the longest sequence)
    const TilePair tiles = tile_pair_of_slot(slot, tiles_of(a.band.seqlen_q), kMasked, kMasked && a.fold);
    w.tile[0] = tiles.a;
    w.tile[1] = tiles.b;
    const int bhi = unit - slot * a.bh.divisor;
    w.b = fast_div(bhi, a.heads);
    w.hq = bhi - w.b * a.heads_q;
    w.kvh = fast_div(w.hq, a.group);
    // packed sequences: this batch entry's own lengths and first rows
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
    w.slot_q = band.seqlen_q;
    if (a.seqused_q != nullptr || a.seqused_k != nullptr) {
        if (a.seqused_q != nullptr) band.seqlen_q = max(0, min(band.seqlen_q, a.seqused_q[w.b]));
        if (a.seqused_k != nullptr) band.seqlen_k = max(0, min(band.seqlen_k, a.seqused_k[w.b]));
        band.off = band.seqlen_k - band.seqlen_q;
    }
    // Query tile x (0 = A, 1 = B) visits key tiles first[x] .. first[x] + count[x] - 1; count is 0 when
    // no key is visible or the tile lies past the end of this sequence.  The CTA walks the union, or its
    // share of it when a cluster splits the keys.
    int first[2], count[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int qt = w.tile[x];
        first[x] = first_k_tile(qt, band);
        count[x] = qt * kTileRows < band.seqlen_q ? k_tiles_of_q_tile(qt, band) : 0;
    }
    int t_begin = 0, t_end = -1;  // inclusive range of key tiles
    if (count[0] > 0 && count[1] > 0) {
        t_begin = min(first[0], first[1]);
        t_end = max(first[0] + count[0], first[1] + count[1]) - 1;
    } else if (count[0] > 0) {
        t_begin = first[0];
        t_end = first[0] + count[0] - 1;
    } else if (count[1] > 0) {
        t_begin = first[1];
        t_end = first[1] + count[1] - 1;
    }
    if (a.splits > 1) {
        const int share = (t_end - t_begin + a.splits) >> a.split_shift;  // ceil(tiles / splits)
        t_begin += w.rank * share;
        t_end = min(t_end, t_begin + share - 1);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int lo = max(first[x], t_begin), hi = min(first[x] + count[x] - 1, t_end);
            first[x] = lo;
            count[x] = max(0, hi - lo + 1);
        }
    }
    w.t_begin = t_begin;
    w.n_iter = max(0, t_end - t_begin + 1);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        w.lo[x] = first[x] - t_begin;
        w.hi[x] = w.lo[x] + count[x];
    }
    w.band = band;
    return w;
}

// The 256 softmax threads finish 256 / kSplits rows of the pair of query tiles from the cluster's kSplits partial
// outputs, which they read through distributed shared memory.  All reads of a row are requested before the first
// is used: one after the other, they cost 10 us per call at four CTAs per pair.
template <typename T, int D, int kSplits>
__device__ __forceinline__ void fwd_merge(const FwdArgs& a, const FwdWork& w, uint32_t sbase) {
    using C = FwdCfg<D>;
    constexpr int kLanes = D / 8;  // threads per row: columns 4*col .. 4*col+3 of either half (a warp reads whole lines)
    constexpr int kRows = 256 / kSplits;
    const int tid = threadIdx.x - 128;
    const int col = tid % kLanes;
    uint32_t peer[kSplits];
#pragma unroll
    for (int s = 0; s < kSplits; ++s) peer[s] = ptx::map_to_cta(sbase, s);
#pragma unroll 1
    for (int rr = tid / kLanes; rr < kRows; rr += 256 / kLanes) {
        const int row = w.rank * kRows + rr;  // row of the pair
        const int qi = w.tile[0] * kTileRows + row;  // (split pairs are neighbours)
        if (qi >= w.slot_q) break;
        float2 ml[kSplits];
        float4 part[kSplits][2];
#pragma unroll
        for (int s = 0; s < kSplits; ++s) {
            const uint32_t base = peer[s] + C::kOffMerge + row * (D * 4);
            ml[s] = ptx::ld_cluster_f2(peer[s] + C::kOffStats + row * 8);
            part[s][0] = ptx::ld_cluster_f4(base + ((col ^ (row & 7)) << 4));
            part[s][1] = ptx::ld_cluster_f4(base + (((kLanes + col) ^ (row & 7)) << 4));
        }
        float m = ml[0].x;
#pragma unroll
        for (int s = 1; s < kSplits; ++s) m = fmaxf(m, ml[s].x);
        float l = 0.0f, acc[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = 0.0f;
#pragma unroll
        for (int s = 0; s < kSplits; ++s) {
            const float f = m == -INFINITY ? 0.0f : ptx::ex2_approx(ml[s].x - m);
            l = fmaf(f, ml[s].y, l);
            acc[0] = fmaf(f, part[s][0].x, acc[0]); acc[1] = fmaf(f, part[s][0].y, acc[1]);
            acc[2] = fmaf(f, part[s][0].z, acc[2]); acc[3] = fmaf(f, part[s][0].w, acc[3]);
            acc[4] = fmaf(f, part[s][1].x, acc[4]); acc[5] = fmaf(f, part[s][1].y, acc[5]);
            acc[6] = fmaf(f, part[s][1].z, acc[6]); acc[7] = fmaf(f, part[s][1].w, acc[7]);
        }
        const float inv = l == 0.0f ? 0.0f : 1.0f / l;  // (l = 0: no visible key, or behind the used length; NaN stays)
        uint4 o;
        o.x = ptx::Pack2<T>::pack(acc[0] * inv, acc[1] * inv);
        o.y = ptx::Pack2<T>::pack(acc[2] * inv, acc[3] * inv);
        o.z = ptx::Pack2<T>::pack(acc[4] * inv, acc[5] * inv);
        o.w = ptx::Pack2<T>::pack(acc[6] * inv, acc[7] * inv);
        T* dst = reinterpret_cast<T*>(a.out) + w.b_coord * a.o_strides.batch + w.hq * a.o_strides.head +
                 int64_t(w.q_base + qi) * a.o_strides.row + col * 4;
        *reinterpret_cast<uint2*>(dst) = make_uint2(o.x, o.y);
        *reinterpret_cast<uint2*>(dst + D / 2) = make_uint2(o.z, o.w);
        if (col == 0)
            a.lse[int64_t(w.b_coord * a.heads_q + w.hq) * a.lse_rows + w.q_base + qi] =
                l == 0.0f ? -INFINITY : (m + __log2f(l)) * 0.69314718055994531f;
    }
}

// kSoftcap: the scaled scores go through softcap * tanh(x / softcap) before the softmax.
// kPersist: CTAs take over the tiles of CTAs that have not started (no clusters).  K, V and Q of the next tile are loaded and its
// first scores computed beside the output of this one, which is staged in a region of its own.
template <typename T, int D, bool kMasked, bool kSoftcap = false, bool kPersist = false>
__global__ void __launch_bounds__(384, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
           const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
           const __grid_constant__ FwdArgs a) {
    using C = FwdCfg<D>;
    static_assert(!kSoftcap || !kPersist, "with capped scores the output reads the work of the first tile again");
    constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = ptx::smem_u32(smem);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    auto bar = [&](int i) -> uint32_t { return sbase + C::kOffBar + 8 * i; };
    const uint32_t tmem_slot = sbase + C::kOffBar + 8 * kFwdNum;
    const uint32_t abort_flag = tmem_slot + 4;

    // Packed sequences: the grid is sized for the longest one, so many CTAs have no rows; they leave before any set-up.
    if (a.cu_seqlens_q != nullptr) {
        ptx::grid_dependency_wait();
        const int slot = fast_div(int(blockIdx.x) >> a.split_shift, a.bh);
        const int first_tile = tile_pair_of_slot(slot, tiles_of(a.band.seqlen_q), kMasked, false).a;
        const int entry = fast_div((int(blockIdx.x) >> a.split_shift) - slot * a.bh.divisor, a.heads);
        if (first_tile * C::kTile >= a.cu_seqlens_q[entry + 1] - a.cu_seqlens_q[entry]) return;
    }

    const uint32_t answer = sbase + C::kOffBar + 272;
    static_assert(8 * kFwdNum + 8 <= 272, "barriers, then the answer");
    const uint32_t work = sbase + C::kOffWork;
    // (a converged warp) the first tile, and the tile after this one; n: how many this CTA has done before
    auto first_tile = [&]() -> FwdWork {
        const FwdWork w = load_work<FwdWork>(work);
        __syncwarp();
        if (kPersist && lane == 0) ptx::mbar_arrive(bar(kFwdWorkEmpty));
        return w;
    };
    auto next_tile = [&](uint32_t n, FwdWork* w) -> bool {
        if (!kPersist) return false;
        const uint32_t buf = (n + 1) & 1;
        if (!warp_wait<false>(bar(kFwdWorkFull + buf), (n >> 1) & 1, abort_flag)) return false;
        *w = load_work<FwdWork>(work + 128 * buf);
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(bar(kFwdWorkEmpty + buf));
        return w->block >= 0;
    };

    // Set-up first: launched programmatically, it overlaps the end of the kernel in front, which
    // grid_dependency_wait() below waits for before any of its outputs is read.
    const bool misaligned = (sbase & 1023u) != 0;
    if (threadIdx.x == 0) {
        if (misaligned) atomicCAS(&g_device_error, kDevOk, kDevSmemMisaligned);
        for (int x = 0; x < 2; ++x) {
            ptx::mbar_init(bar(kFwdQFull + x), 1);
            ptx::mbar_init(bar(kFwdSFull + x), 1);
            ptx::mbar_init(bar(kFwdSFree + x), 4);
            ptx::mbar_init(bar(kFwdPFirst + x), 4);
            ptx::mbar_init(bar(kFwdPReady + x), 4);
            ptx::mbar_init(bar(kFwdPvDone + x), 1);
            ptx::mbar_init(bar(kFwdQEmpty + x), 1);
        }
        for (int s = 0; s < C::kStages; ++s) {
            ptx::mbar_init(bar(kFwdKFull + s), 1);
            ptx::mbar_init(bar(kFwdKEmpty + s), 1);
            ptx::mbar_init(bar(kFwdVFull + s), 1);
            ptx::mbar_init(bar(kFwdVEmpty + s), 1);
        }
        ptx::mbar_init(bar(kFwdAllDone), 1);
        ptx::mbar_init(bar(kFwdAnswer), 1);
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(bar(kFwdWorkFull + s), 1);
            ptx::mbar_init(bar(kFwdWorkEmpty + s), 10);  // producer, MMA issuer, softmax warps
        }
        flag_set(abort_flag, 0);
        ptx::fence_mbar_init();
    }
    if (warp == 0 && lane == 0) {
        ptx::prefetch_tensormap(&tm_q);
        ptx::prefetch_tensormap(&tm_k);
        ptx::prefetch_tensormap(&tm_v);
    }
    if (warp == 1) {
        ptx::tmem_alloc(tmem_slot, C::kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::launch_dependents();

    // (all threads: barriers initialised, tensor memory allocated, first tile known)
    auto set_up_done = [&] {
        ptx::grid_dependency_wait();
        ptx::tc_fence_before();
        asm volatile("bar.sync 0;" ::: "memory");
        ptx::tc_fence_after();
        return flag_value(tmem_slot);
    };

    // (each role changes its register budget at the top of its own branch, where the compiler can see
    // which code runs under which budget)
    if (warp < 4) {
        ptx::setmaxnreg_dec<C::kRegsControl>();
        if (warp == 2) {
            ptx::grid_dependency_wait();
            const FwdWork w = fwd_work<kMasked>(a, int(blockIdx.x));
            if (lane == 0) store_work(work, w);
            __syncwarp();
        }
        const uint32_t tmem = set_up_done();
        if (misaligned) {
            // nothing to do
        } else if (warp == 0) {
            // TMA producer, converged like the MMA issuer
            FwdWork w = first_tile();
            uint32_t n = 0;
            int g0 = 0, used[2] = {0, 0};  // iterations of the tiles before; how often Q of either query tile was loaded
            bool ok = true;
#pragma unroll 1
            for (bool more = true; ok && more; ++n) {
                auto load_k = [&](int it) {
                    const int g = g0 + it, s = g % C::kStages;
                    if (!warp_wait(bar(kFwdKEmpty + s), ((g / C::kStages) & 1) ^ 1, abort_flag)) return false;
                    ptx::tma_load_tile_elect<C::kBoxes>(sbase + C::kOffK + s * C::kOperandBytes, &tm_k, bar(kFwdKFull + s),
                                                        w.k_base + (w.t_begin + it) * C::kTile, w.kvh, w.b_coord);
                    return true;
                };
                auto load_v = [&](int it) {
                    const int g = g0 + it, s = g % C::kStages;
                    if (!warp_wait(bar(kFwdVEmpty + s), ((g / C::kStages) & 1) ^ 1, abort_flag)) return false;
                    ptx::tma_load_tile_elect<C::kBoxes>(sbase + C::kOffV + s * C::kOperandBytes, &tm_v, bar(kFwdVFull + s),
                                                        w.k_base + (w.t_begin + it) * C::kTile, w.kvh, w.b_coord);
                    return true;
                };
                if (n > 0 && w.n_iter > 0) ok = load_k(0);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    if (w.lo[x] >= w.hi[x] || !ok) continue;  // nothing is loaded for a tile that sees no key
                    if (used[x] > 0) ok = warp_wait(bar(kFwdQEmpty + x), (used[x] - 1) & 1, abort_flag);
                    if (ok) ptx::tma_load_tile_elect<C::kBoxes>(sbase + C::kOffQ + x * C::kOperandBytes, &tm_q, bar(kFwdQFull + x),
                                                                w.q_base + w.tile[x] * C::kTile, w.hq, w.b_coord);
                    ++used[x];
                }
#pragma unroll 1
                for (int it = 0; ok && it < w.n_iter; ++it) ok = ((n > 0 && it == 0) || load_k(it)) && load_v(it);
                if (!ok) break;
                g0 += w.n_iter;
                more = next_tile(n, &w);
            }
        } else if (warp == 1) {
            // MMA issuer: the whole warp runs the role converged; the issue forms and the commits elect their
            // lane inside the asm.
            constexpr uint32_t kIdS = ptx::instr_desc_f16(kBf16, 128, 128, false, false);
            constexpr uint32_t kIdO = ptx::instr_desc_f16(kBf16, 128, D, false, true);
            FwdWork w = first_tile();
            uint32_t n = 0;
            int g0 = 0, c[2] = {0, 0}, used[2] = {0, 0};  // ... and how often Q of either query tile was loaded
            // S of query tile x against the key tile of iteration `it`
            auto issue_s = [&](int x, int it) {
                const uint32_t loQ = ptx::desc_lo_k_major(sbase + C::kOffQ + x * C::kOperandBytes);
                const uint32_t loK = ptx::desc_lo_k_major(sbase + C::kOffK + ((g0 + it) % C::kStages) * C::kOperandBytes);
                const uint32_t dst = tmem + C::kColS + x * 128;
                ptx::mma_ss<D / 16, ptx::KMajor, ptx::KMajor>(dst, loQ, loK, kIdS, 0);
                ptx::tc_commit_elect(bar(kFwdSFull + x));
                if (kPersist && it == w.hi[x] - 1) ptx::tc_commit_elect(bar(kFwdQEmpty + x));
            };
            auto wait_k = [&](int it) { return warp_wait<false>(bar(kFwdKFull + (g0 + it) % C::kStages), ((g0 + it) / C::kStages) & 1, abort_flag); };
            auto wait_v = [&](int it) { return warp_wait<false>(bar(kFwdVFull + (g0 + it) % C::kStages), ((g0 + it) / C::kStages) & 1, abort_flag); };
            // O of query tile x += P V of iteration `it`: on the first part of P as soon as it is there, then on the rest
            auto issue_pv = [&](int x, int it) {
                const uint32_t loV = ptx::desc_lo_mn_major(sbase + C::kOffV + ((g0 + it) % C::kStages) * C::kOperandBytes, C::kBoxBytes);
                const uint32_t p_cols = tmem + C::kColP + x * C::kPStride;
                const uint32_t o_cols = tmem + C::kColO + x * D;
                const uint32_t parity = (c[x] + it - w.lo[x]) & 1;
                const uint32_t accumulate = it > w.lo[x] ? 1u : 0u;
                if (!warp_wait<false>(bar(kFwdPFirst + x), parity, abort_flag)) return false;
                ptx::tc_fence_after();
                ptx::mma_ts_4<0, ptx::TmemPacked, ptx::MnMajor>(o_cols, p_cols, loV, kIdO, accumulate);
                if (!warp_wait<false>(bar(kFwdPReady + x), parity, abort_flag)) return false;
                ptx::tc_fence_after();
                ptx::mma_ts_4<4, ptx::TmemPacked, ptx::MnMajor>(o_cols, p_cols, loV, kIdO, 1);
                ptx::tc_commit_elect(bar(kFwdPvDone + x));
                return true;
            };
            // (own P) the scores in front of those of iteration `it` are in registers
            auto wait_s_free = [&](int x, int it) {
                const int before = c[x] + it - w.lo[x];
                return before == 0 || warp_wait<false>(bar(kFwdSFree + x), (before - 1) & 1, abort_flag);
            };
            // Asks for the next tile, in front of the last P V of this one: late enough that tiles go to the CTAs in the order in
            // which these become free, early enough that its K and V are there when this one's output is.  (Warp 2 has used
            // the answer before.)
            auto request = [&] {
                if constexpr (kPersist) {
                    if (lane == 0) {
                        ptx::mbar_arrive_expect_tx(bar(kFwdAnswer), 16);
                        ptx::request_block(answer, bar(kFwdAnswer));
                    }
                    __syncwarp();
                }
            };
            bool ok = true;
#pragma unroll 1
            for (bool next = true; ok && next; ++n) {
                const int n_iter = w.n_iter;
                if (n_iter == 0) request();
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    if (ok && w.lo[x] < w.hi[x]) ok = warp_wait<false>(bar(kFwdQFull + x), used[x]++ & 1, abort_flag);
                }
                if (ok && n_iter > 0) ok = wait_k(0);
                if (ok && n_iter > 0) {
                    ptx::tc_fence_after();
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (ok && w.active(x, 0)) {
                            if (C::kOwnP) {
                                ok = wait_s_free(x, 0);
                                ptx::tc_fence_after();
                            }
                            if (ok) issue_s(x, 0);
                        }
                    }
                    ptx::tc_commit_elect(bar(kFwdKEmpty + g0 % C::kStages));
                }
                if constexpr (!C::kOwnP) {
#pragma unroll 1
                    for (int it = 0; ok && it < n_iter; ++it) {
                        const bool more = it + 1 < n_iter;
                        if (!more) request();
                        bool v_ready = false, k_ready = false;
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            if (w.active(x, it)) {
                                if (!v_ready) {
                                    if (!(ok = wait_v(it))) break;
                                    v_ready = true;
                                }
                                if (!(ok = issue_pv(x, it))) break;
                            }
                            // S of the next key tile goes over P of this one: it follows P V in the pipe
                            if (more && w.active(x, it + 1)) {
                                if (!k_ready) {
                                    if (!(ok = wait_k(it + 1))) break;
                                    k_ready = true;
                                    ptx::tc_fence_after();
                                }
                                issue_s(x, it + 1);
                            }
                        }
                        if (!ok) break;
                        if (more) ptx::tc_commit_elect(bar(kFwdKEmpty + (g0 + it + 1) % C::kStages));
                        ptx::tc_commit_elect(bar(kFwdVEmpty + (g0 + it) % C::kStages));
                    }
                } else {
                    // S(x, it+1) needs only "scores (x, it) in registers"; P V of tile B is issued one half
                    // iteration late, because the two softmax warpgroups settle half an iteration apart
#pragma unroll 1
                    for (int it = 0; ok && n_iter > 0 && it <= n_iter; ++it) {
                        const bool more = it + 1 < n_iter;
                        if (it == n_iter - 1) request();
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            if (more && w.active(x, it + 1)) {
                                ok = wait_s_free(x, it + 1);
                                if (!(ok = ok && wait_k(it + 1))) break;
                                ptx::tc_fence_after();
                                issue_s(x, it + 1);
                            }
                            // x = 0: P V of tile B, previous iteration; x = 1: P V of tile A, this iteration
                            const int pv = it - (x == 0 ? 1 : 0);
                            const int y = x ^ 1;
                            if (pv < n_iter && w.active(y, pv)) {
                                if (!(ok = wait_v(pv) && issue_pv(y, pv))) break;
                            }
                            if (x == 0 && it > 0) ptx::tc_commit_elect(bar(kFwdVEmpty + (g0 + it - 1) % C::kStages));
                        }
                        if (!ok) break;
                        if (more) ptx::tc_commit_elect(bar(kFwdKEmpty + (g0 + it + 1) % C::kStages));
                    }
                }
                if (!ok) break;
                if (n_iter > 0) ptx::tc_commit_elect(bar(kFwdAllDone));  // (waited for with one tile per CTA)
                g0 += n_iter;
#pragma unroll
                for (int x = 0; x < 2; ++x) c[x] += max(0, w.hi[x] - w.lo[x]);
                next = next_tile(n, &w);
            }
        } else if (warp == 2 && kPersist) {
            // which tile next
#pragma unroll 1
            for (uint32_t n = 0, answers = 0;; ++n) {  // the work of tile n + 1
                const uint32_t buf = (n + 1) & 1;
                FwdWork w;
                bool ok;
                while ((ok = warp_wait(bar(kFwdAnswer), answers & 1, abort_flag))) {
                    ++answers;
                    const int block = ptx::answered_block(answer);
                    ptx::fence_proxy_async_smem();  // (it is written through the async proxy again)
                    if (block >= 0) w = fwd_work<kMasked>(a, block);
                    w.block = block;
                    // (packed sequences: blocks without rows)
                    if (block < 0 || min(w.tile[0], w.tile[1]) * C::kTile < w.slot_q) break;
                    __syncwarp();
                    if (lane == 0) {
                        ptx::mbar_arrive_expect_tx(bar(kFwdAnswer), 16);
                        ptx::request_block(answer, bar(kFwdAnswer));
                    }
                }
                // (that of tile n - 1 has been read)
                if (!ok || (n >= 1 && !warp_wait(bar(kFwdWorkEmpty + buf), ((n - 1) >> 1) & 1, abort_flag))) break;
                if (lane == 0) store_work(work + 128 * buf, w);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(bar(kFwdWorkFull + buf));
                if (w.block < 0) break;
            }
        }
        if (a.splits > 1) {  // (the softmax warps meet their peers around the merge)
            __syncwarp();
            ptx::cluster_sync();
            ptx::cluster_sync();
        }
    } else {
        ptx::setmaxnreg_inc<C::kRegsSoftmax>();
        const uint32_t tmem = set_up_done();
        if (misaligned) {
            if (a.splits > 1) {
                ptx::cluster_sync();
                ptx::cluster_sync();
            }
        } else {
            const int x = (warp - 4) >> 2;      // which query tile
            const int i = threadIdx.x & 127;    // query row inside the tile == TMEM lane
            FwdWork w = first_tile();
            uint32_t n = 0;
            int c0 = 0;  // steps of the tiles before
            bool more = true;
#pragma unroll 1
            for (; more; ++n) {
                // (selects, not indexing: no local array; uniform: see there)
                const int qt = uniform(x == 0 ? w.tile[0] : w.tile[1]);
                const int n_steps = uniform(x == 0 ? w.hi[0] - w.lo[0] : w.hi[1] - w.lo[1]);
                const int k_begin = w.t_begin + (x == 0 ? w.lo[0] : w.lo[1]);
                const uint32_t tl = tmem + (uint32_t((warp & 3) * 32) << 16);
                const uint32_t s_cols = tl + C::kColS + x * 128;
                const uint32_t p_cols = tl + C::kColP + x * C::kPStride;
                const uint32_t o_cols = tl + C::kColO + x * D;
                const int qi = qt * C::kTile + i;  // query row inside the head
                const bool q_valid = qi < w.band.seqlen_q;
                float m_ref = -INFINITY;  // reference maximum (raw scores) the exponentials are taken against
                float l = 0.0f;           // sum of the exponentials, in units of exp2(m_ref * scale_log2)
                const float sl = kSoftcap ? a.softcap_post : a.scale_log2;  // log2 units per unit of (transformed) score
                const uint64_t sl2 = ptx::f2_pack(sl, sl);
                // one arrival per warp: every lane's accesses are ordered before it by the fence and the warp barrier
                auto arrive = [&](int which) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(bar(which + x));
                };
                // key j of key tile k_begin + u survives for query i iff mask_from <= j <= mask_to
                int mask_from = 0, mask_to = 0;
                if (kMasked) key_range_of_query(qi, k_begin * C::kTile, w.band, &mask_from, &mask_to);
                bool ok = true;
#pragma unroll 1
                for (int u = 0; u < n_steps; ++u) {
                    if (!(ok = warp_wait<false>(bar(kFwdSFull + x), (c0 + u) & 1, abort_flag))) break;
                    ptx::tc_fence_after();
                    const bool diagonal = kMasked && __any_sync(0xffffffffu, mask_from > 0 || mask_to < C::kTile - 1);
                    // ---- the whole score row of this tile goes to registers in one round trip
                    uint32_t r[4][32];
#pragma unroll
                    for (int c = 0; c < 4; ++c) ptx::tmem_ld32(s_cols + c * 32, r[c]);
                    // (asked ahead of its use: has P V of the previous key tile completed?)
                    const bool p_free = !C::kOwnP || u == 0 || ptx::mbar_test_wait(bar(kFwdPvDone + x), (c0 + u - 1) & 1);
                    ptx::tmem_ld_wait();
                    if (C::kOwnP) arrive(kFwdSFree);
                    if (kSoftcap) {
                        // from here on the scores are the tanh, and their scale the cap
                        const float pre = a.softcap_pre * ptx::kTanhArg;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
#pragma unroll
                            for (int e = 0; e < 32; e += 2) {
                                const uint64_t s2 = ptx::f2_pack(__uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1]));
                                const float2 t = ptx::f2_unpack(ptx::tanh_mixed<C::kTanhFmaPairs>(ptx::f2_mul(s2, ptx::f2_pack(pre, pre)), e / 2));
                                r[c][e] = __float_as_uint(t.x);
                                r[c][e + 1] = __float_as_uint(t.y);
                            }
                        }
                    }
                    if (diagonal) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
#pragma unroll
                            for (int e = 0; e < 32; ++e) {
                                const int j = c * 32 + e;
                                if (j < mask_from || j > mask_to) r[c][e] = 0xff800000u;  // -inf
                            }
                        }
                    }
                    // four chains of three-input maxima; a NaN among the visible scores makes the maximum NaN
                    float mx[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) mx[c] = ptx::max_nan(__uint_as_float(r[c][0]), __uint_as_float(r[c][1]));
#pragma unroll
                    for (int e = 2; e < 32; e += 2) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) mx[c] = ptx::max3_nan(mx[c], __uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1]));
                    }
                    const float mt = ptx::max_nan(ptx::max3_nan(mx[0], mx[1], mx[2]), mx[3]);
                    // ---- move the reference maximum only when it is more than 2^8 too small (or NaN)
                    const bool move = m_ref == -INFINITY ? mt != -INFINITY : !((mt - m_ref) * sl <= C::kRescaleThreshold);
                    if (__any_sync(0xffffffffu, move)) {
                        // exp2(-inf) = 0 on the first move
                        const float alpha = move ? ptx::ex2_approx((m_ref - mt) * sl) : 1.0f;
                        if (move) m_ref = mt;
                        // a NaN or +inf score makes l, and by it O and the log-sum-exp, NaN (mt - mt): not every exponential
                        // of such a row would be NaN (exp2_poly)
                        l = fmaf(l, alpha, move ? mt - mt : 0.0f);
                        if (u > 0) {
                            // O carries the old reference: wait for P V of step u-1, then rescale these 32 rows (16
                            // columns at a time: the score row is still held in registers)
                            if (!(ok = warp_wait<false>(bar(kFwdPvDone + x), (c0 + u - 1) & 1, abort_flag))) break;
                            ptx::tc_fence_after();
#pragma unroll 1
                            for (int c = 0; c < D / 16; ++c) {
                                uint32_t acc[16];
                                ptx::tmem_ld16(o_cols + c * 16, acc);
                                ptx::tmem_ld_wait();
#pragma unroll
                                for (int e = 0; e < 16; ++e) acc[e] = __float_as_uint(__uint_as_float(acc[e]) * alpha);
                                ptx::tmem_st16(o_cols + c * 16, acc);
                            }
                            ptx::tmem_st_wait();
                        }
                    }
                    // ---- P = exp2((S - m_ref) * scale_log2), written as 16-bit pairs (over S, every column of which
                    // has been read by now, where P has no columns of its own)
                    if (C::kOwnP) {
                        // P of the previous key tile must have been used before it is overwritten
                        if (!__all_sync(0xffffffffu, p_free) && !(ok = warp_wait<false>(bar(kFwdPvDone + x), (c0 + u - 1) & 1, abort_flag))) break;
                        ptx::tc_fence_after();
                    }
                    const float neg = m_ref == -INFINITY ? 0.0f : -m_ref * sl;
                    const uint64_t neg2 = ptx::f2_pack(neg, neg);
                    uint64_t sum2[2] = {0, 0};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[16];
#pragma unroll
                        for (int e = 0; e < 32; e += 2) {
                            const uint64_t x2 = ptx::f2_fma(ptx::f2_pack(__uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1])), sl2, neg2);
                            float2 pr;
                            // (the pairs that take the polynomial are spread evenly over the row)
                            if (((e / 2) * C::kPolyPairs) % 8 + C::kPolyPairs >= 8 && C::kPolyPairs > 0) {
                                pr = ptx::exp2_poly(x2);
                            } else {
                                pr = ptx::f2_unpack(x2);
                                pr.x = ptx::ex2_approx(pr.x);
                                pr.y = ptx::ex2_approx(pr.y);
                            }
                            sum2[(e / 2) & 1] = ptx::f2_add(sum2[(e / 2) & 1], ptx::f2_pack(pr.x, pr.y));
                            o[e / 2] = ptx::Pack2<T>::pack(pr.x, pr.y);
                        }
                        ptx::tmem_st16(p_cols + c * 16, o);
                        if (c == 1) {
                            ptx::tmem_st_wait();
                            arrive(kFwdPFirst);
                        }
                    }
                    ptx::tmem_st_wait();
                    arrive(kFwdPReady);
                    const float2 sum = ptx::f2_unpack(ptx::f2_add(sum2[0], sum2[1]));
                    l += sum.x + sum.y;
                    mask_from -= C::kTile;
                    mask_to -= C::kTile;
                }
                if constexpr (kSoftcap) w = load_work<FwdWork>(work);  // (what only the output needs is not held in registers before)
                // (m_ref, not l, says whether the row saw a key: exp2_poly leaves 2^-126 on a masked one)
                const bool any_key = q_valid && m_ref != -INFINITY;
                const float inv = any_key ? 1.0f / l : 0.0f;
                // ln(sum exp(s*scale)) = (m_ref*scale_log2 + log2 l) * ln 2
                float* lse_dst = a.lse + int64_t(w.b_coord * a.heads_q + w.hq) * a.lse_rows + w.q_base + qi;
                if (!kPersist && a.splits > 1) {
                    // This CTA's share of the keys: unnormalised O, fp32, and {m in log2 units, l} go to shared
                    // memory, over the K / V rings, for the merge below.
                    if (ok && w.n_iter > 0) ok = warp_wait(bar(kFwdAllDone), 0, abort_flag);
                    ptx::tc_fence_after();
                    *reinterpret_cast<float2*>(smem + C::kOffStats + (x * 128 + i) * 8) =
                        make_float2(any_key ? m_ref * sl : -INFINITY, any_key ? l : 0.0f);
                    const uint32_t row_addr = sbase + C::kOffMerge + (x * 128 + i) * (D * 4);
#pragma unroll 1
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t r[32];
                        if (n_steps > 0) {
                            ptx::tmem_ld32(o_cols + c * 32, r);
                            ptx::tmem_ld_wait();
                        }
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int chunk = (c * 8 + e) ^ (i & 7);  // (rows are 256 or 512 bytes apart: spread over the banks)
                            const bool keep = n_steps > 0 && any_key;
                            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                         ::"r"(row_addr + chunk * 16), "r"(keep ? r[4 * e] : 0u), "r"(keep ? r[4 * e + 1] : 0u),
                                           "r"(keep ? r[4 * e + 2] : 0u), "r"(keep ? r[4 * e + 3] : 0u) : "memory");
                        }
                    }
                } else {
                    if (ok && n_steps > 0) ok = warp_wait(bar(kFwdPvDone + x), (c0 + n_steps - 1) & 1, abort_flag);
                    T* dst = reinterpret_cast<T*>(a.out) + w.b_coord * a.o_strides.batch + w.hq * a.o_strides.head +
                             int64_t(w.q_base + qi) * a.o_strides.row;
                    if (ok && ((q_valid && n_steps == 0) || (!q_valid && qi < w.slot_q))) {
                        // no visible key at all, or a row behind the used length: O = 0, lse = -inf
                        uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
                        for (int e = 0; e < D / 8; ++e) d4[e] = make_uint4(0u, 0u, 0u, 0u);
                        *lse_dst = -INFINITY;
                    }
                    __syncwarp();
                    if (ok && n_steps > 0) {
                        // (tensor-memory loads are warp-wide: every lane runs them, only the stores of query rows
                        // past the end of the sequence are skipped)
                        ptx::tc_fence_after();
                        if (q_valid) *lse_dst = any_key ? (m_ref * sl + __log2f(l)) * 0.69314718055994531f : -INFINITY;
                        if (a.staged_store) {
                            // through shared memory (the Q tile is dead: its last S completed before this O) and the copy
                            // engine: whole lines instead of 16 bytes of 32 rows per instruction, rows past the end clipped
                            const int w4 = warp & 3;
                            const uint32_t stage = kPersist ? sbase + C::kOffOut + (x * 4 + w4) * 4096 : sbase + C::kOffQ + x * C::kOperandBytes + w4 * (C::kBoxes * 4096);
                            const bool in_range = qt * C::kTile + w4 * 32 < w.slot_q;
                            const float scale_row = q_valid ? inv : 0.0f;  // (rows behind a used length hold zeros)
#pragma unroll
                            for (int c = 0; c < D / 32; ++c) {
                                uint32_t r[32];
                                ptx::tmem_ld32(o_cols + c * 32, r);
                                ptx::tmem_ld_wait();
                                const uint32_t row_addr = stage + (kPersist ? 0 : c >> 1) * 4096 + lane * 128;
                                if (kPersist && (c & 1) == 0) {  // (its 64 columns before have been read)
                                    if (lane == 0) ptx::bulk_wait_group_read<0>();
                                    __syncwarp();
                                }
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    uint32_t o[4];
#pragma unroll
                                    for (int h = 0; h < 4; ++h) {
                                        const float lo = __uint_as_float(r[8 * e + 2 * h]) * scale_row, hi = __uint_as_float(r[8 * e + 2 * h + 1]) * scale_row;
                                        o[h] = scale_row != 0.0f ? ptx::Pack2<T>::pack(lo, hi) : 0u;
                                    }
                                    const int chunk = ((c & 1) * 4 + e) ^ (lane & 7);
                                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};"
                                                 ::"r"(row_addr + (chunk << 4)), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                                }
                                if (kPersist && (c & 1) == 1) {
                                    ptx::fence_proxy_async_smem();
                                    __syncwarp();
                                    if (lane == 0 && in_range) {
                                        ptx::tma_store_4d(&tm_o, stage, (c >> 1) * 64, qt * C::kTile + w4 * 32, w.hq, w.b);
                                        ptx::bulk_commit_group();
                                    }
                                }
                            }
                            if (!kPersist) {
                                ptx::fence_proxy_async_smem();
                                __syncwarp();
                                if (lane == 0 && in_range) {
#pragma unroll
                                    for (int bx = 0; bx < C::kBoxes; ++bx)
                                        ptx::tma_store_4d(&tm_o, stage + bx * 4096, bx * 64, qt * C::kTile + w4 * 32, w.hq, w.b);
                                    ptx::bulk_commit_group();
                                    ptx::bulk_wait_group_read<0>();
                                }
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < D / 32; ++c) {
                                uint32_t r[32];
                                ptx::tmem_ld32(o_cols + c * 32, r);
                                ptx::tmem_ld_wait();
                                if (q_valid) {
                                    uint4* d4 = reinterpret_cast<uint4*>(dst + c * 32);
#pragma unroll
                                    for (int e = 0; e < 4; ++e) {
                                        uint4 o;
                                        o.x = ptx::Pack2<T>::pack(__uint_as_float(r[8 * e + 0]) * inv, __uint_as_float(r[8 * e + 1]) * inv);
                                        o.y = ptx::Pack2<T>::pack(__uint_as_float(r[8 * e + 2]) * inv, __uint_as_float(r[8 * e + 3]) * inv);
                                        o.z = ptx::Pack2<T>::pack(__uint_as_float(r[8 * e + 4]) * inv, __uint_as_float(r[8 * e + 5]) * inv);
                                        o.w = ptx::Pack2<T>::pack(__uint_as_float(r[8 * e + 6]) * inv, __uint_as_float(r[8 * e + 7]) * inv);
                                        d4[e] = o;
                                    }
                                }
                                __syncwarp();  // reconverge before the next warp-wide load
                            }
                        }
                    }
                }
                if (kPersist) {
                    __syncwarp();
                    if (!ok) break;
                    c0 += max(0, n_steps);
                }
                if (!kPersist && a.splits > 1) {
                    // ---- merge of the cluster's shares: every CTA finishes 256 / splits of the pair's rows, reading
                    // the partial outputs of all peers through distributed shared memory
                    __syncwarp();
                    ptx::cluster_sync();
                    if (a.splits == 2) fwd_merge<T, D, 2>(a, w, sbase);
                    else if (a.splits == 4) fwd_merge<T, D, 4>(a, w, sbase);
                    else fwd_merge<T, D, 8>(a, w, sbase);
                    __syncwarp();
                    ptx::cluster_sync();  // the peers read this CTA's shared memory until here
                }
                more = next_tile(n, &w);
            }
            if (kPersist && lane == 0) ptx::bulk_wait_group_read<0>();  // (shared memory is not given back before)
        }
    }

    __syncwarp();
    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(flag_value(tmem_slot), C::kTmemCols);
    }
}

}  // namespace fa3b200
