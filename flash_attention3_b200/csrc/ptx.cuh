// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (bulk tensor copies and
// bulk tensor reduce-add), tcgen05 (TMEM allocation, MMA, commit, ld/st) and
// the UMMA shared-memory / instruction descriptors.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ------------------------------------------------------------------ mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// The same question without waiting.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Generic-proxy writes to shared memory -> visible to the async proxy (TMA,
// tcgen05.mma operand reads).
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------- TMA
// 4-D tiled load (coordinates innermost first); rows outside the tensor read as zero.
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* map, uint32_t bar, int c0,
                                            int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
// The producer's step for a converged warp (one lane is elected): expect the bytes of kBoxes boxes of
// [128 rows][64 x 16 bit] on the barrier and request them, boxes 64 columns and 16 KiB apart.
template <int kBoxes>
__device__ __forceinline__ void tma_load_tile_elect(uint32_t dst, const void* map, uint32_t bar, int row, int head, int batch) {
    static_assert(kBoxes == 1 || kBoxes == 2, "head dimension 64 or 128");
    if (kBoxes == 1) {
        asm volatile(
            "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
            "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], 16384;\n\t"
            "@q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%6, %3, %4, %5}], [%2];\n\t}"
            ::"r"(dst), "l"(map), "r"(bar), "r"(row), "r"(head), "r"(batch), "r"(0) : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
            "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], 32768;\n\t"
            "@q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%6, %3, %4, %5}], [%2];\n\t"
            "@q cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%8], [%1, {%7, %3, %4, %5}], [%2];\n\t}"
            ::"r"(dst), "l"(map), "r"(bar), "r"(row), "r"(head), "r"(batch), "r"(0), "r"(64), "r"(dst + 16384) : "memory");
    }
}
// 3-D tiled reduce-add shared -> global; elements outside the tensor are dropped.
__device__ __forceinline__ void tma_reduce_add_3d(const void* map, uint32_t src, int c0, int c1,
                                                  int c2) {
    asm volatile(
        "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group"
        " [%0, {%2, %3, %4}], [%1];"
        ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// 4-D tiled store shared -> global; elements outside the tensor are dropped.
__device__ __forceinline__ void tma_store_4d(const void* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
        ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void bulk_commit_group() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_group_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void bulk_wait_group() {
    asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const void* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ------------------------------------------------------------------- tcgen05
// All of these are warp-wide (.sync.aligned) unless noted.
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Whole converged warp: the elected lane arrives on an mbarrier when all MMAs it issued so far
// have completed (the election is deterministic, so it is the lane the MMA forms below elect).
__device__ __forceinline__ void tc_commit_elect(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar) : "memory");
}
// Issue forms for the MMA-issuing warp.  They are executed by the whole, converged warp and elect the
// issuing lane inside the asm block: with a converged warp the descriptors live in uniform registers and
// one MMA costs a couple of issue slots, whereas a single divergent lane needs many more and is starved by
// the math warps that share its scheduler.  One block issues the whole chain of K steps of a tile behind
// one election: with two busy math warps on every scheduler, M128 N128 K16 MMAs go out every 64.2 cycles,
// the rate of the pipe, against 79.6 when every MMA elects and builds its descriptors for itself.
// A descriptor is passed as its low 32 bits (start address >> 4 | LBO field); the high half (SBO, version,
// swizzle) is one constant, and a K step adds a compile-time constant.
constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024 B, version 1, 128-B swizzle
__host__ __device__ constexpr uint32_t desc_lo_k_major(uint32_t addr) { return ((addr & 0x3FFFF) >> 4) | (1u << 16); }
__host__ __device__ constexpr uint32_t desc_lo_mn_major(uint32_t addr, uint32_t lbo_bytes) {
    return ((addr & 0x3FFFF) >> 4) | (((lbo_bytes >> 4) & 0x3FFF) << 16);
}
// What K step kk (16 elements) adds to an operand: a K-major tile of [128 rows][64 columns] boxes, an
// MN-major tile, and a 16-bit operand in tensor memory (two elements per column, contiguous or with columns
// 64-127 of the tile 64 columns on).
struct KMajor { __host__ __device__ static constexpr int step(int kk) { return (kk >> 2) * ((128 * 128) >> 4) + (kk & 3) * 2; } };
struct MnMajor { __host__ __device__ static constexpr int step(int kk) { return kk * 128; } };
struct TmemPacked { __host__ __device__ static constexpr int step(int kk) { return kk * 8; } };
struct TmemHalves { __host__ __device__ static constexpr int step(int kk) { return (kk >> 2) * 64 + (kk & 3) * 8; } };

#define FA3_MMA_SS_STEP(A, B) \
    "add.s64 ea, da, %" A ";\n\tadd.s64 eb, db, %" B ";\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], ea, eb, %4, t;\n\t"
// D[tmem] (+)= A[smem] * B[smem] over K steps 0..7 (or 0..3); accumulate = 0: the first one overwrites D.
template <typename A, typename B>
__device__ __forceinline__ void mma_ss_8(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 da, db, ea, eb;\n\telect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
        FA3_MMA_SS_STEP("6", "7") FA3_MMA_SS_STEP("8", "9") FA3_MMA_SS_STEP("10", "11") FA3_MMA_SS_STEP("12", "13")
        FA3_MMA_SS_STEP("14", "15") FA3_MMA_SS_STEP("16", "17") FA3_MMA_SS_STEP("18", "19") "}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate),
          "n"(A::step(1)), "n"(B::step(1)), "n"(A::step(2)), "n"(B::step(2)), "n"(A::step(3)), "n"(B::step(3)), "n"(A::step(4)),
          "n"(B::step(4)), "n"(A::step(5)), "n"(B::step(5)), "n"(A::step(6)), "n"(B::step(6)), "n"(A::step(7)), "n"(B::step(7))
        : "memory");
}
template <typename A, typename B>
__device__ __forceinline__ void mma_ss_4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 da, db, ea, eb;\n\telect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tmov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t"
        FA3_MMA_SS_STEP("6", "7") FA3_MMA_SS_STEP("8", "9") FA3_MMA_SS_STEP("10", "11") "}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kDescHiSw128), "r"(idesc), "r"(accumulate),
          "n"(A::step(1)), "n"(B::step(1)), "n"(A::step(2)), "n"(B::step(2)), "n"(A::step(3)), "n"(B::step(3))
        : "memory");
}
// K = 16 * kSteps elements.
template <int kSteps, typename A, typename B>
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    static_assert(kSteps == 4 || kSteps == 8, "K of 64 or 128");
    if (kSteps == 8) mma_ss_8<A, B>(d_tmem, a_lo, b_lo, idesc, accumulate);
    else mma_ss_4<A, B>(d_tmem, a_lo, b_lo, idesc, accumulate);
}
#undef FA3_MMA_SS_STEP

#define FA3_MMA_TS_STEP(A, B) \
    "add.u32 ea, %1, %" A ";\n\tadd.s64 eb, db, %" B ";\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [ea], eb, %4, t;\n\t"
// D[tmem] (+)= A[tmem] * B[smem] over the K steps kFirst .. kFirst + 3 of 16 elements.
template <int kFirst, typename A, typename B>
__device__ __forceinline__ void mma_ts_4(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 db, eb;\n\t.reg .b32 ea;\n\telect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %3, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tmov.b64 db, {%2, %5};\n\t"
        "add.u32 ea, %1, %6;\n\tadd.s64 eb, db, %7;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [ea], eb, %4, p;\n\t"
        FA3_MMA_TS_STEP("8", "9") FA3_MMA_TS_STEP("10", "11") FA3_MMA_TS_STEP("12", "13") "}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(accumulate), "r"(idesc), "r"(kDescHiSw128),
          "n"(A::step(kFirst)), "n"(B::step(kFirst)), "n"(A::step(kFirst + 1)), "n"(B::step(kFirst + 1)),
          "n"(A::step(kFirst + 2)), "n"(B::step(kFirst + 2)), "n"(A::step(kFirst + 3)), "n"(B::step(kFirst + 3))
        : "memory");
}
// ... over the eight K steps of 128 elements.
template <typename A, typename B>
__device__ __forceinline__ void mma_ts_8(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 db, eb;\n\t.reg .b32 ea;\n\telect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %3, 0;\n\tsetp.eq.u32 t, 0, 0;\n\tmov.b64 db, {%2, %5};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t"
        FA3_MMA_TS_STEP("6", "7") FA3_MMA_TS_STEP("8", "9") FA3_MMA_TS_STEP("10", "11") FA3_MMA_TS_STEP("12", "13")
        FA3_MMA_TS_STEP("14", "15") FA3_MMA_TS_STEP("16", "17") FA3_MMA_TS_STEP("18", "19") "}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(accumulate), "r"(idesc), "r"(kDescHiSw128),
          "n"(A::step(1)), "n"(B::step(1)), "n"(A::step(2)), "n"(B::step(2)), "n"(A::step(3)), "n"(B::step(3)), "n"(A::step(4)),
          "n"(B::step(4)), "n"(A::step(5)), "n"(B::step(5)), "n"(A::step(6)), "n"(B::step(6)), "n"(A::step(7)), "n"(B::step(7))
        : "memory");
}
#undef FA3_MMA_TS_STEP

// 32 lanes x 32 consecutive 32-bit columns: thread l of the warp receives the
// 32 columns of TMEM lane (lane_base + l).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// 32 lanes x 16 columns load.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 32 lanes x 16 columns store (one register per column).
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
          "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]),
          "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// --------------------------------------------------------------- descriptors
// 64-bit shared-memory matrix descriptor, 128-byte swizzle, version 1 (kDescHiSw128 and desc_lo_* above are its halves).
//   bits  0-13  start address >> 4
//   bits 16-29  leading-dimension byte offset >> 4
//   bits 32-45  stride-dimension byte offset >> 4
//   bits 46-47  descriptor version (1 on sm_100)
//   bits 61-63  swizzle mode (2 = 128 B)
// Tiles are stored as boxes of [rows][64 x 16-bit] = rows x 128 B, each box
// written by TMA (or by threads) with the 128-byte swizzle, 1024-B aligned.
//  K-major operand (the 64 contiguous elements run along the MMA K
//    dimension): SBO = 1024 (next 8 rows); LBO unused.  K advances by 32 B per
//    16 elements inside a box and by one box per 64.
//  MN-major operand (the 64 contiguous elements run along M or N): LBO = box
//    bytes (next 64 M/N elements), SBO = 1024 (next 8 K rows).  K advances by
//    2048 B per 16 rows.

// 32-bit instruction descriptor for kind::f16, fp32 accumulate.
//   bits 4-5 D format (1 = f32); 7-9 A format; 10-12 B format (0 f16, 1 bf16);
//   bit 15 A major; bit 16 B major (0 = K, 1 = MN); 17-22 N >> 3; 24-28 M >> 4.
__host__ __device__ constexpr uint32_t instr_desc_f16(bool bf16, int m, int n, bool a_mn_major,
                                                      bool b_mn_major) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) |
           ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

// Programmatic dependent launch: a kernel launched with the programmatic-serialisation
// attribute may start while its predecessor in the stream still runs; grid_dependency_wait()
// blocks until the predecessor has completed and its writes are visible, and
// launch_dependents() lets the successor's CTAs begin to launch.  Both are no-ops for a kernel
// launched without the attribute.
__device__ __forceinline__ void grid_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Taking over the work of a block that has not started (a running block asks for the index of one; the block that had it is
// never launched).  The answer, 16 bytes in shared memory, is counted by the barrier; after a refusal nothing more is asked.
__device__ __forceinline__ void request_block(uint32_t answer, uint32_t bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                 ::"r"(answer), "r"(bar) : "memory");
}
// blockIdx.x of the block taken over, -1 for a refusal.
__device__ __forceinline__ int answered_block(uint32_t answer) {
    uint32_t taken, x;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\tld.shared.b128 r, [%2];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\tselp.u32 %0, 1, 0, p;\n\tmov.u32 %1, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, r;\n\t}"
        : "=r"(taken), "=r"(x) : "r"(answer) : "memory");
    return taken != 0 ? int(x) : -1;
}

// Thread-block clusters.
// All threads of all CTAs of the cluster; shared-memory writes before it are visible to the peers after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Address of this CTA's shared-memory location `addr` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t d;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

// Per-warpgroup register re-allocation (all 128 threads of the warpgroup).
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// ---------------------------------------------------------------- misc math
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Two fp32 values in one 64-bit register: one issue slot for both (the FMA pipe takes two cycles).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t d) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(d));
    return v;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// Four consecutive fp32 values in shared memory, as two pairs.
struct F4Pairs {
    uint64_t lo, hi;
};
__device__ __forceinline__ F4Pairs f2_ld_shared(uint32_t addr) {
    F4Pairs v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(addr) : "memory");
    return v;
}
// Maxima that are NaN if any operand is (fmaxf drops a NaN).
__device__ __forceinline__ float max_nan(float a, float b) {
    float d;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// 2^x of two values on the FMA and integer pipes, for code that the special-function unit bounds (a warp's
// ex2 keeps it busy for 8 cycles, these 24 instructions for two values keep the FMA pipe busy for 16).
// x = n + f with n the nearest integer (rounded by adding 1.5 * 2^23, which also leaves n in the low bits),
// 2^f by a polynomial of degree 5 on [-1/2, 1/2] (Remez exchange on the relative error: 7.5e-8, or 2.2e-7 with
// coefficients and arithmetic in fp32; ex2.approx is good to 2.4e-7), then n added to the exponent field.  x above
// 127 and NaN are not expected (the forward treats a row with such a score by its sum); below -126 the result stays
// at 2^-126.
__device__ __forceinline__ float2 exp2_poly(uint64_t x2) {
    const float kMagic = 12582912.0f;
    float2 x = f2_unpack(x2);
    x2 = f2_pack(fmaxf(x.x, -126.0f), fmaxf(x.y, -126.0f));
    const uint64_t t2 = f2_add(x2, f2_pack(kMagic, kMagic));
    const uint64_t f2 = f2_add(x2, f2_fma(t2, f2_pack(-1.0f, -1.0f), f2_pack(kMagic, kMagic)));  // x - n
    uint64_t p2 = f2_pack(0x1.5c08e6p-10f, 0x1.5c08e6p-10f);
    p2 = f2_fma(p2, f2, f2_pack(0x1.3d0c52p-7f, 0x1.3d0c52p-7f));
    p2 = f2_fma(p2, f2, f2_pack(0x1.c6b6e4p-5f, 0x1.c6b6e4p-5f));
    p2 = f2_fma(p2, f2, f2_pack(0x1.ebf918p-3f, 0x1.ebf918p-3f));
    p2 = f2_fma(p2, f2, f2_pack(0x1.62e428p-1f, 0x1.62e428p-1f));
    p2 = f2_fma(p2, f2, f2_pack(0x1.000002p+0f, 0x1.000002p+0f));
    const float2 t = f2_unpack(t2), p = f2_unpack(p2);
    return make_float2(__uint_as_float(__float_as_uint(p.x) + (__float_as_uint(t.x) << 23)),
                       __uint_as_float(__float_as_uint(p.y) + (__float_as_uint(t.y) << 23)));
}

// tanh of two values, 1 - 2 / (exp(2x) + 1), absolute error at most 2.3e-7; the argument is x * kTanhArg.  A NaN
// stays a NaN, and neither value depends on the other (one of the two may be masked).
// (tanh.approx.f32 has a relative error of 2^-11; the softcap multiplies it by softcap*log2(e), which for a cap
// of 50 already costs P a quarter of a percent.  One reciprocal for both values, 1/a = b * 1/(ab), is 4 % faster, 238
// against 247 us for forward and gradients of B=1, Hq=16, Hkv=8, S=4096, D=128, window 1024, but the rounded product takes
// the error to 3.6e-7, and the Newton step that brings it back costs what the reciprocal saved.)
constexpr float kTanhArg = 2.8853900817779268f;  // 2 * log2(e)
__device__ __forceinline__ uint64_t tanh_pair(uint64_t x_arg2) {
    const float2 x = f2_unpack(x_arg2);
    const float2 d = f2_unpack(f2_add(f2_pack(ex2_approx(x.x), ex2_approx(x.y)), f2_pack(1.0f, 1.0f)));
    float rx, ry;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ry) : "f"(d.y));
    return f2_fma(f2_pack(rx, ry), f2_pack(-2.0f, -2.0f), f2_pack(1.0f, 1.0f));
}
// The same on the FMA pipe but for one exponential per value: sign(x) (1 - z) / (1 + z), z = exp(-2|x|).  1 / (1 + z) by a
// polynomial of degree 3 (relative error e up to 1.7e-3) and one step of third order, r + r (e + e^2).  Absolute error at most 1.9e-7.
__device__ __forceinline__ uint64_t tanh_pair_fma(uint64_t x_arg2) {
    const float2 x = f2_unpack(x_arg2);
    const uint64_t one2 = f2_pack(1.0f, 1.0f), minus2 = f2_pack(-1.0f, -1.0f);
    const uint64_t z2 = f2_pack(ex2_approx(-fabsf(x.x)), ex2_approx(-fabsf(x.y)));
    uint64_t r2 = f2_pack(-0x1.c6527ep-3f, -0x1.c6527ep-3f);
    r2 = f2_fma(r2, z2, f2_pack(0x1.54bde2p-1f, 0x1.54bde2p-1f));
    r2 = f2_fma(r2, z2, f2_pack(-0x1.e2b7aep-1f, -0x1.e2b7aep-1f));
    r2 = f2_fma(r2, z2, f2_pack(0x1.ff1cd6p-1f, 0x1.ff1cd6p-1f));
    const uint64_t e2 = f2_fma(f2_fma(z2, minus2, minus2), r2, one2);  // 1 - (1 + z) r
    r2 = f2_fma(r2, f2_fma(e2, e2, e2), r2);
    const float2 t = f2_unpack(f2_mul(f2_fma(z2, minus2, one2), r2));
    return f2_pack(copysignf(t.x, x.x), copysignf(t.y, x.y));
}
// tanh of the `pair`-th pair of values of a thread: of every 8 pairs kFmaPairs take the second form.  The first keeps the
// special-function unit busy for 32 cycles (the exponential of the softmax for 16 more), the second for 16 and the FMA pipe for
// 20; a mix keeps both busy.  Which form a value takes depends on its place alone, and the time not on the scores.
// us, all of the first form and so: B=1, Hq=16, Hkv=8, S=4096, D=128, window 1024, cap 30 forward 89.8 and 78.5, gradients 157 and 138,
// reproducible 204 and 177; B=4, 16 x 2048 full, D=64, cap 50 262 and 222, 397 and 327, 684 and 569 (with P (1 - tanh^2) handed to the dS
// phase instead of taken from log2 of P).  A polynomial on the FMA pipe alone where all of a warp's 32 x 32 scores are below
// the cap, and both forms where some are not, measured 76, 134, 178 and 232, 311, 537 without such scores, but 114, 199, 240 and 334,
// 491, 808 with one in a thousand above the cap, and 111, 171, 228 and 329, 432, 738 with four in ten.
template <int kFmaPairs>
__device__ __forceinline__ uint64_t tanh_mixed(uint64_t x_arg2, int pair) {
    return (pair * kFmaPairs) % 8 + kFmaPairs >= 8 ? tanh_pair_fma(x_arg2) : tanh_pair(x_arg2);
}

// Four fp32 values in three registers, the upper 24 bits of each (15 bits of significand, to within 2^-15 and without a bias: the
// byte that is missing is taken to be like the one above it, which keeps 0, infinities and NaN as they are).
__device__ __forceinline__ uint32_t byte_perm(uint32_t a, uint32_t b, uint32_t selector) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
    return d;
}
__device__ __forceinline__ void pack24(const float* v, uint32_t* o) {
    const uint32_t last = __float_as_uint(v[3]);
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = byte_perm(__float_as_uint(v[i]), last, 0x3215u + i);
}
__device__ __forceinline__ void unpack24(const uint32_t* o, float* v) {
#pragma unroll
    for (int i = 0; i < 3; ++i) v[i] = __uint_as_float(byte_perm(o[i], 0u, 0x3211u));
    v[3] = __uint_as_float(byte_perm(byte_perm(o[0], o[1], 0x0400u), o[2], 0x4211u));
}

template <typename T>
struct Pack2;
template <>
struct Pack2<__half> {
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t u) {
        return __half22float2(*reinterpret_cast<__half2*>(&u));
    }
};
template <>
struct Pack2<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
        __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&h);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t u) {
        return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
    }
};

}  // namespace ptx
