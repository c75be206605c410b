// int8 x int8 -> int32 convolution as an implicit GEMM on the sm_100a tensor cores.
//
//   GEMM view   M = N*OH*OW output pixels, N = O output channels, K = KH*KW*Cp  (k ordered kh, kw, c)
//   A operand   activations, int8 [N][H][W][Cp]; one TMA im2col load per (filter tap, channel block) brings the
//               128 x BK tile of a 128-pixel run of output positions -- halo, stride, dilation and zero padding
//               are resolved by the tensor map, nothing is materialised in memory
//   B operand   weights, int8 [O][KH][KW][Cp]; plain 2-D TMA tiles of BN x BK
//   MMA         tcgen05.mma kind::i8, 128 x BN x 32 per instruction, int32 accumulators in tensor memory,
//               issued by two warps on alternate tiles; up to four accumulator buffers, so the epilogue of a
//               tile overlaps the main loops of the next ones
//   epilogue    sixteen warps read the accumulators with tcgen05.ld and apply dequantize / bias / residual /
//               activation / requantize in registers, then store fp32 (NCHW or NHWC) and/or int8, or hand
//               them to four copy warps in shared-memory tiles (staged class)
//
// Warp roles in a CTA of 608 threads (736 in the staged class): warp 0 = TMA producer, warps 1 and 2 = MMA issuers (warp 1
// owns tensor memory), warps 3..18 = epilogue, warps 19..22 = the staged class's copies.  The kernel is persistent:
// gridDim.x CTAs walk the tile list with stride gridDim.x, or, with resident weights, each a range of it.
//
// Every wait on an mbarrier is bounded; a wait that runs out records a code in *status, raises a CTA-wide
// abort flag and all roles fall through to the common exit, where tensor memory is released.
// (barrier.cluster.wait, in split-K, has no bound of its own: see there.)
#pragma once

#include "conv_common.cuh"
#include "conv_tc.h"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cstdlib>

namespace tsb {
namespace tc {

constexpr int kBM = 128;
constexpr int kIssuers = 2;                              // warps that issue MMAs, on alternate tiles
constexpr int kEpiWarp0 = 1 + kIssuers;                  // first epilogue warp
constexpr int kEpiThreads = 512;                         // sixteen epilogue warps
constexpr int kCopyWarp0 = kEpiWarp0 + kEpiThreads / 32; // staged epilogue: the first of its four copy warps
constexpr int kMaxAccBufs = 4;                           // accumulator buffers in tensor memory (512 columns / BN, at most 4)
constexpr uint32_t kSmemBudget = 216 * 1024;  // stages and staged tiles; the rest of the 227 KB holds barriers and epilogue tables

// ---------------------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

// Bounded wait.  Returns false when the CTA is aborting or ~2 s of polling went by.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t spin = 0;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 255u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > 4000000000LL) return false;
        }
    }
}

// The same for a whole warp, with an answer that the compiler knows to be the same in every lane.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// True in one lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(on));
    return on != 0;
}

// ---- clusters (split-K): CTAs that write to each other's shared memory
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the address of `addr` (this CTA's shared memory) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
    return out;
}
__device__ __forceinline__ void sts128_cluster(uint32_t addr, int a, int b, int c, int d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// an arrival on another CTA's barrier that publishes what the cluster can see of this thread's writes
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// mbar_wait that sees what the other CTAs of the cluster wrote before they arrived
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    const long long t0 = clock64();
    for (uint32_t spin = 0;; ++spin) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
        if ((spin & 255u) == 255u) {
            if (*abort_flag) return false;
            if (clock64() - t0 > 4000000000LL) return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}

// plain (untiled) bulk copy global -> shared; both addresses and the size are multiples of 16 bytes
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int w, int h, int n) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int w, int h) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h) : "memory");
}
// tile stores shared -> global (bulk async group of the issuing thread); out-of-range parts of the box are not written
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap *map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, uint32_t src, int x, int y, int z, int w) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the stores of this thread's groups have finished READING shared memory (the source may be overwritten)
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// generic-proxy writes to shared memory become visible to the async proxy (TMA) of this CTA
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_load_im2col_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c, int w,
                                                   int h, int n, uint16_t off_w, uint16_t off_h) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h) : "memory");
}

// Brings a box of a tensor into L2 without a destination in shared memory (no barrier, nothing to wait for).
__device__ __forceinline__ void tma_prefetch_l2_2d(const CUtensorMap *map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}

// Brings a tensor map (a kernel parameter) into the copy engine's descriptor cache.
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The same, executed only when `on` is non-zero -- a predicated instruction, not a branch.  What an issuing warp spends between two MMAs is
// not hidden, so its MMA sequences are straight-line code in which inactive slots (a filter row outside the image, a tap beyond
// the filter) are switched off by predicate.
__device__ __forceinline__ void mma_i8_if(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t on) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(on));
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, int (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const int (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
        ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are one swizzle span (BK bytes) wide: 8-row groups are
// group_stride_bytes apart (8*BK in a tile that is packed; more under a patch, whose rows a window skips); leading byte offset unused;
// version 1; swizzle 128B (2) or 64B (4).  The swizzle is a function of the absolute shared-memory address (measured: any
// 128-byte-aligned start and any group stride read back what a tensor-map copy with the same swizzle wrote; the base-offset
// field stays 0), so a start need not be 1024-byte aligned.
// Everything but the 14-bit start-address field is loop-invariant, so a loop keeps the invariant part in a register and ORs in
// (address >> 4) -- shared-memory addresses stay below 2^18, so the field never overflows into its neighbours, and stepping along K
// inside a swizzle span or to another filter tap is a plain add on that field.
template <int BK>
__device__ __forceinline__ constexpr uint64_t smem_desc_hi(uint32_t group_stride_bytes) {
    return ((uint64_t)1 << 16) | ((uint64_t)(group_stride_bytes >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)(BK == 128 ? 2 : (BK == 64 ? 4 : 6)) << 61);
}

// A descriptor from its two 32-bit halves (a register pair: no instruction).  The issuing thread keeps the high half and
// the leading-offset bits of the low half loop-invariant and steps only the 14-bit address field: `lo` below is
// (address >> 4) | (1 << 16), and adding a few 16-byte units to it never carries out of the field.
__device__ __forceinline__ uint64_t desc_pair(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | (uint64_t)lo; }
constexpr uint32_t kDescLbo = 1u << 16;   // leading byte offset 16 (unused for swizzled K-major operands, set as before)

// Descriptor of a pixel operand whose rows OVERLAP in shared memory (raw-row mode): no swizzle, K-major.  In that canonical
// layout row r, 16-byte K chunk j sits at (r % 8) * 16 + (r / 8) * SBO + j * LBO; with SBO = 128 and LBO = 16 that is
// r * 16 + j * 16: pixel r reads the bytes that start 16 bytes after pixel r-1's, which is exactly a convolution window
// sliding by one pixel stride over one staged image row.
__device__ __forceinline__ uint64_t smem_desc_sliding(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(16 >> 4) << 16;               // leading byte offset: next 16-byte chunk along K
    d |= (uint64_t)(128 >> 4) << 32;              // stride byte offset: next group of 8 rows
    d |= (uint64_t)1 << 46;                       // descriptor version of this architecture
    return d;                                     // layout 0: no swizzle
}

// Instruction descriptor: int32 accumulate, signed 8-bit A and B, both K-major, M = 128, N = BN.
template <int BN>
__device__ __forceinline__ constexpr uint32_t instr_desc() {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}


// ---------------------------------------------------------------------------------------------------------
// epilogue: 32 accumulator columns of one output pixel (one thread) at a time
// ---------------------------------------------------------------------------------------------------------
// Which one a launch takes is a template parameter of the kernel (EPI): an instance holds the code of one class only.  With all
// classes in one kernel every class paid for the others: 700 bytes of spills in all of them (now at most 32, 48 in the
// staged class, 304 in the pixel-major one of raw rows), and a variant more cost the layers that never ran it 3-8 %.  Measured with the
// classes apart: the five sweep layers at batch 32 126 -> 115 us, a ResNet-50 pass of 64 images 1.42 -> 1.35 ms.
constexpr int kEpiGeneric = 0;   // any combination of outputs, element by element
constexpr int kEpiF32Nchw = 1;   // fp32 NCHW output only (the operator's own output)
constexpr int kEpiI8Nhwc = 2;    // requantized int8 NHWC_PAD output only, one scale for the batch (half to even) or per image (half away from zero)
constexpr int kEpiNhwc = 3;      // fp32 [N][P][O] residual in and/or fp32 [N][P][O] out and/or int8 NHWC_PAD out, from registers (swapped orientation;
                                 // raw rows whose weights leave no room for the staged class)
constexpr int kEpiStaged = 4;    // the same outputs through shared-memory tiles and tensor-map loads / stores (normal orientation)
constexpr int kEpiStagedAfter = 5;   // ... with the residual added after the activation
__host__ __device__ constexpr bool is_staged(int epi) { return epi == kEpiStaged || epi == kEpiStagedAfter; }
// producer warp, issuer warps, sixteen epilogue warps and, in the staged class, four copy warps
__host__ __device__ constexpr int cta_threads(int epi) { return 32 * (kCopyWarp0 + (is_staged(epi) ? 4 : 0)); }
constexpr uint32_t kStageF32Bytes = kBM * 32 * 4;   // one staged fp32 tile: 128 pixels x 32 channels, 128-byte rows, swizzle 128B
constexpr uint32_t kStageI8Bytes = kBM * 32;        // one staged int8 tile: 128 pixels x 32 channels, 32-byte rows
constexpr int kSplit = 4;                           // CTAs that share the K blocks of a tile in split-K mode
constexpr int kQuads = 4;                           // the sixteen epilogue warps form four quads of one warp per lane quarter

// (a layer without a bias adds a zero: the same value up to the sign of a zero, which the operators' results are compared up
// to anyway)
template <int ACT>
__device__ __forceinline__ float epi_value(int acc, float dq, float bias, float leaky) {
    float f = __fadd_rn(__fmul_rn(__int2float_rn(acc), dq), bias);
    if (ACT == TSB_ACT_RELU) f = fmaxf(f, 0.0f);   // finite values only: same result as x > 0 ? x : 0
    if (ACT == TSB_ACT_LEAKY_RELU) f = f > 0.0f ? f : __fmul_rn(f, leaky);
    return f;
}

// Round-half-away of an already scaled value t, as a signed 32-bit integer (three instructions per value):
// floor(|t| + 0.5) is obtained exactly as trunc(round_toward_zero(|t| + 0.5)) -- a round-to-nearest sum would be wrong
// for |t| just below 0.5 -- and the sign is put back before the (saturating) conversion.
__device__ __forceinline__ int half_away_s32(float t) {
    const float mag = __fadd_rz(fabsf(t), 0.5f);
    const float signed_mag = __int_as_float((__float_as_int(mag) & 0x7fffffff) | (__float_as_int(t) & 0x80000000));
    return __float2int_rz(signed_mag);
}

// The rounding of a requantize, as a signed 32-bit integer: half-to-even where one scale covers the tensor (a batch of one;
// the last count % 8 elements excepted, see fix_tail), half away from zero otherwise.  A compile-time choice: one conversion
// per value either way.  (Element by element, as single-scale outputs once went, a 128 x 64 tile took 15 us where this takes 2: a
// CSPDarknet53-shaped pass of one 608 x 608 image 2.65 -> 0.61 ms.)
template <bool EVEN>
__device__ __forceinline__ int round_s32(float t) {
    if (EVEN) return __float2int_rn(t);
    return half_away_s32(t);
}
// ... and as a saturated int8
template <bool EVEN>
__device__ __forceinline__ int round_s8(float t) {
    int q;
    if (EVEN) {
        asm("cvt.rni.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(t));
    } else {
        const float mag = __fadd_rz(fabsf(t), 0.5f);
        const float sm = __int_as_float((__float_as_int(mag) & 0x7fffffff) | (__float_as_int(t) & 0x80000000));
        asm("cvt.rzi.sat.s8.f32 %0, %1;" : "=r"(q) : "f"(sm));
    }
    return q;
}

// four signed integers -> four int8 with saturation to [-128,127], v0 in the lowest byte
__device__ __forceinline__ uint32_t pack_sat_s8(int v0, int v1, int v2, int v3) {
    uint32_t hi, out;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(v3), "r"(v2), "r"(0));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(v1), "r"(v0), "r"(hi));
    return out;
}

// max that keeps a NaN once it has seen one
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// the same over three values (one instruction on this architecture)
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// ---- fast paths, normal orientation: the thread owns one PIXEL (its tensor-memory lane) and 32 consecutive channels
template <int ACT, int W>
__device__ __forceinline__ void store_f32_nchw_t(const int (&v)[W], const float *__restrict__ dq,
                                                 const float *__restrict__ bias, float leaky, float *__restrict__ dst,
                                                 uint32_t stride, int channels) {
    if (channels < W) {    // the last chunk of a channel count that is no multiple of 32
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < channels) dst[(uint32_t)j * stride] = epi_value<ACT>(v[j], dq[j], bias[j], leaky);
        return;
    }
#pragma unroll
    for (int j4 = 0; j4 < W / 4; ++j4) {
        const float4 d4 = *reinterpret_cast<const float4 *>(dq + 4 * j4);
        const float4 b4 = *reinterpret_cast<const float4 *>(bias + 4 * j4);
        dst[(uint32_t)(4 * j4 + 0) * stride] = epi_value<ACT>(v[4 * j4 + 0], d4.x, b4.x, leaky);
        dst[(uint32_t)(4 * j4 + 1) * stride] = epi_value<ACT>(v[4 * j4 + 1], d4.y, b4.y, leaky);
        dst[(uint32_t)(4 * j4 + 2) * stride] = epi_value<ACT>(v[4 * j4 + 2], d4.z, b4.z, leaky);
        dst[(uint32_t)(4 * j4 + 3) * stride] = epi_value<ACT>(v[4 * j4 + 3], d4.w, b4.w, leaky);
    }
}

// The same with an fp32 NCHW residual (operator "add" between add_bias and the activation, or after the activation): the
// residual is read where the result is written, so a warp's 32 pixels make one coalesced line per channel either way.
template <int ACT, int W, bool AFTER>
__device__ __forceinline__ void store_f32_nchw_res_t(const int (&v)[W], const float *__restrict__ dq,
                                                     const float *__restrict__ bias, float leaky, const float *__restrict__ res,
                                                     float *__restrict__ dst, uint32_t stride, int channels) {
#pragma unroll
    for (int j8 = 0; j8 < W / 8; ++j8) {
        float r[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) r[k] = 8 * j8 + k < channels ? __ldg(res + (uint32_t)(8 * j8 + k) * stride) : 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = 8 * j8 + k;
            float t = __fadd_rn(__fmul_rn(__int2float_rn(v[j]), dq[j]), bias[j]);
            if (!AFTER) t = __fadd_rn(t, r[k]);
            if (ACT == TSB_ACT_RELU) t = fmaxf(t, 0.0f);
            if (ACT == TSB_ACT_LEAKY_RELU) t = t > 0.0f ? t : __fmul_rn(t, leaky);
            if (AFTER) t = __fadd_rn(t, r[k]);
            if (j < channels) dst[(uint32_t)j * stride] = t;
        }
    }
}

// Requantized int8 output.  Returns false when a scaled value was NaN or beyond the int32 range -- those quantize to
// -128 in the reference (x86 integer-indefinite), which the saturating fast path does not reproduce; the caller
// then redoes the chunk element by element.
// (columns at or beyond O have zero weights, scale and bias, so they come out as the zeros that the layout's padding channels
// hold; `bytes` says how much of the chunk lies inside the padded row)
template <int ACT, bool EVEN, int W>
__device__ __forceinline__ bool store_i8_nhwc_t(const int (&v)[W], const float *__restrict__ dq,
                                                const float *__restrict__ bias, float leaky, float rs,
                                                int8_t *__restrict__ dst, int bytes) {
    uint32_t q[W / 4];
    float worst = 0.0f;
#pragma unroll
    for (int j4 = 0; j4 < W / 4; ++j4) {
        const float4 d4 = *reinterpret_cast<const float4 *>(dq + 4 * j4);
        const float4 b4 = *reinterpret_cast<const float4 *>(bias + 4 * j4);
        const float t0 = __fmul_rn(epi_value<ACT>(v[4 * j4 + 0], d4.x, b4.x, leaky), rs);
        const float t1 = __fmul_rn(epi_value<ACT>(v[4 * j4 + 1], d4.y, b4.y, leaky), rs);
        const float t2 = __fmul_rn(epi_value<ACT>(v[4 * j4 + 2], d4.z, b4.z, leaky), rs);
        const float t3 = __fmul_rn(epi_value<ACT>(v[4 * j4 + 3], d4.w, b4.w, leaky), rs);
        worst = max3_nan(max3_nan(worst, fabsf(t0), fabsf(t1)), fabsf(t2), fabsf(t3));
        q[j4] = pack_sat_s8(round_s32<EVEN>(t0), round_s32<EVEN>(t1), round_s32<EVEN>(t2), round_s32<EVEN>(t3));
    }
    if (!(worst < 2147483648.0f)) return false;
#pragma unroll
    for (int h = 0; h < W / 16; ++h)
        if (16 * h < bytes) *reinterpret_cast<int4 *>(dst + 16 * h) = make_int4(q[4 * h], q[4 * h + 1], q[4 * h + 2], q[4 * h + 3]);
    return true;
}

// Pixel-major fp32 tensors from a thread that owns a pixel: its 32 channels are contiguous, 16-byte loads and stores (rows of O floats
// with O % 4 == 0).  For raw rows whose weights and image rows leave no room for the staged class below; the staged class is the faster one
// where it fits (a thread's stores go to rows far apart).
// Measured, 5x5 3 -> 96 at 200 x 416, 4 images: 78 us, element by element 312 (NCHW 38).
template <int ACT, bool EVEN, bool AFTER>
__device__ __forceinline__ bool store_nhwc_t(const int (&v)[32], const float *__restrict__ dq, const float *__restrict__ bias, float leaky,
                                             const float *__restrict__ res, float *__restrict__ out_f32, int8_t *__restrict__ out_i8,
                                             float rs, int channels, int bytes) {
    uint32_t q[8];
    float worst = 0.0f;
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
        const float4 d4 = *reinterpret_cast<const float4 *>(dq + 4 * j4);
        const float4 b4 = *reinterpret_cast<const float4 *>(bias + 4 * j4);
        float4 r4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (res && 4 * j4 < channels) r4 = __ldg(reinterpret_cast<const float4 *>(res) + j4);
        float f[4];
        const float dd[4] = {d4.x, d4.y, d4.z, d4.w}, bb[4] = {b4.x, b4.y, b4.z, b4.w}, rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float t = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + k]), dd[k]), bb[k]);
            if (!AFTER) t = __fadd_rn(t, rr[k]);
            if (ACT == TSB_ACT_RELU) t = fmaxf(t, 0.0f);
            if (ACT == TSB_ACT_LEAKY_RELU) t = t > 0.0f ? t : __fmul_rn(t, leaky);
            if (AFTER) t = __fadd_rn(t, rr[k]);
            f[k] = t;
        }
        if (out_f32 && 4 * j4 < channels) reinterpret_cast<float4 *>(out_f32)[j4] = make_float4(f[0], f[1], f[2], f[3]);
        if (out_i8) {
            const float t0 = __fmul_rn(f[0], rs), t1 = __fmul_rn(f[1], rs), t2 = __fmul_rn(f[2], rs), t3 = __fmul_rn(f[3], rs);
            worst = max3_nan(max3_nan(worst, fabsf(t0), fabsf(t1)), fabsf(t2), fabsf(t3));
            q[j4] = pack_sat_s8(round_s32<EVEN>(t0), round_s32<EVEN>(t1), round_s32<EVEN>(t2), round_s32<EVEN>(t3));
        }
    }
    if (out_i8) {
        if (!(worst < 2147483648.0f)) return false;
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (16 * h < bytes) *reinterpret_cast<int4 *>(out_i8 + 16 * h) = make_int4(q[4 * h], q[4 * h + 1], q[4 * h + 2], q[4 * h + 3]);
    }
    return true;
}

// Block-output epilogue of a residual network: v = act(dq*acc + bias + residual); fp32 copy for the next residual and
// int8 copy for the next convolution, each optional.  The thread's 32 channels of residual come from its row of a shared-memory
// tile that a tensor-map load filled (128-byte rows, 128B swizzle: 16-byte chunk i of row r sits at chunk i ^ (r & 7)), the
// fp32 results go back into the same places and the int8 results into the thread's 32-byte row of a second tile; tensor-
// map stores carry both tiles to global memory.  No global address arithmetic, every shared-memory access 16 bytes wide.
// r_row: shared-memory address of the row, its swizzle key folded in, so that chunk i is at r_row ^ (i * 16).
__device__ __forceinline__ float4 lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Returns false when an int8 value needs the exact conversion (NaN, beyond the int32 range).  q: the packed int8 results.
template <int ACT, bool EVEN, bool AFTER>
__device__ __forceinline__ bool staged_chunk_t(const int (&v)[32], const float *__restrict__ dq, const float *__restrict__ bias,
                                               float leaky, uint32_t r_row, bool has_res, bool has_i8, float rs, uint32_t (&q)[8]) {
    float worst = 0.0f;
#pragma unroll
    for (int j4 = 0; j4 < 8; ++j4) {
        const float4 d4 = *reinterpret_cast<const float4 *>(dq + 4 * j4);
        const float4 b4 = *reinterpret_cast<const float4 *>(bias + 4 * j4);
        float4 r4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (has_res) r4 = lds128(r_row ^ (uint32_t)(j4 * 16));
        float f[4];
        const float dd[4] = {d4.x, d4.y, d4.z, d4.w}, bb[4] = {b4.x, b4.y, b4.z, b4.w}, rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float t = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + k]), dd[k]), bb[k]);
            // without a residual rr is zero: adding it changes nothing but the sign of a negative zero, which the
            // operators' results are compared up to anyway (relu and leaky_relu do not pin it either)
            if (!AFTER) t = __fadd_rn(t, rr[k]);
            if (ACT == TSB_ACT_RELU) t = fmaxf(t, 0.0f);
            if (ACT == TSB_ACT_LEAKY_RELU) t = t > 0.0f ? t : __fmul_rn(t, leaky);
            if (AFTER) t = __fadd_rn(t, rr[k]);
            f[k] = t;
        }
        sts128(r_row ^ (uint32_t)(j4 * 16), make_float4(f[0], f[1], f[2], f[3]));
        if (has_i8) {
            const float t0 = __fmul_rn(f[0], rs), t1 = __fmul_rn(f[1], rs), t2 = __fmul_rn(f[2], rs), t3 = __fmul_rn(f[3], rs);
            worst = max3_nan(max3_nan(worst, fabsf(t0), fabsf(t1)), fabsf(t2), fabsf(t3));
            q[j4] = pack_sat_s8(round_s32<EVEN>(t0), round_s32<EVEN>(t1), round_s32<EVEN>(t2), round_s32<EVEN>(t3));
        }
    }
    return worst < 2147483648.0f;
}

// ---- fast paths, swapped orientation: the thread owns one CHANNEL (its lane) and 32 consecutive pixels; dq and bias
// are per-thread scalars
template <int ACT>
__device__ __forceinline__ void swap_f32_run(const int (&v)[32], float dq, float bias, float leaky, float *__restrict__ dst) {
    // 32 consecutive pixels of one channel plane: 128 contiguous bytes
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
            float4 o;
            o.x = epi_value<ACT>(v[4 * j4 + 0], dq, bias, leaky);
            o.y = epi_value<ACT>(v[4 * j4 + 1], dq, bias, leaky);
            o.z = epi_value<ACT>(v[4 * j4 + 2], dq, bias, leaky);
            o.w = epi_value<ACT>(v[4 * j4 + 3], dq, bias, leaky);
            reinterpret_cast<float4 *>(dst)[j4] = o;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) dst[j] = epi_value<ACT>(v[j], dq, bias, leaky);
    }
}

// The same where the chunk ends the tensor (npix < 32) or crosses an image boundary: pixels from `split` on belong to the next
// image, `jump` floats further on.  For images of at least 32 pixels (one boundary at most).
template <int ACT>
__device__ __forceinline__ void swap_f32_split_run(const int (&v)[32], float dq, float bias, float leaky, float *__restrict__ dst,
                                                   int npix, int split, uint32_t jump) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
        if (j < npix) dst[(uint32_t)j + (j >= split ? jump : 0u)] = epi_value<ACT>(v[j], dq, bias, leaky);
}

// int8 NHWC_PAD output: for one pixel the 32 lanes of the warp hold 32 consecutive channels, so each byte store
// instruction of the warp writes one full 32-byte sector.  The first `split` pixels use rs0, the rest rs1 (the chunk
// crosses at most one image boundary).
// Returns false if a value needs the slow path (NaN / beyond int32); the decision is uniform over the warp.
template <int ACT, bool EVEN>
__device__ __forceinline__ bool swap_i8_run(const int (&v)[32], float dq, float bias, float leaky, float rs0, float rs1,
                                            int split, bool write, int8_t *__restrict__ dst, uint32_t pixel_stride, int npix) {
    float worst = 0.0f;
    int q[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const float t = __fmul_rn(epi_value<ACT>(v[j], dq, bias, leaky), j < split ? rs0 : rs1);
        worst = max_nan(worst, fabsf(t));
        q[j] = round_s8<EVEN>(t);
    }
    if (__any_sync(0xffffffffu, !(worst < 2147483648.0f))) return false;
    if (write) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if (j < npix) dst[(uint32_t)j * pixel_stride] = (int8_t)q[j];
    }
    return true;
}

// Patch mode, swapped orientation: the 32 accumulators of a chunk are 4 tile rows of 8 pixels of one channel.
// rows_live / cols_live say how much of that 4 x 8 block lies inside the image (uniform over the warp).
template <int ACT, bool EVEN>
__device__ __forceinline__ bool patch_i8_run(const int (&v)[32], float dq, float bias, float leaky, float rs, bool write,
                                             int8_t *__restrict__ dst, uint32_t pixel_stride, uint32_t row_stride,
                                             int rows_live, int cols_live) {
    float worst = 0.0f;
    int q[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const float t = __fmul_rn(epi_value<ACT>(v[j], dq, bias, leaky), rs);
        const bool live = (j >> 3) < rows_live && (j & 7) < cols_live;
        worst = max_nan(worst, live ? fabsf(t) : 0.0f);
        q[j] = round_s8<EVEN>(t);
    }
    if (__any_sync(0xffffffffu, !(worst < 2147483648.0f))) return false;
    if (write) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
            if ((j >> 3) < rows_live && (j & 7) < cols_live) dst[(uint32_t)(j >> 3) * row_stride + (uint32_t)(j & 7) * pixel_stride] = (int8_t)q[j];
    }
    return true;
}
template <int ACT>
__device__ __forceinline__ void patch_f32_run(const int (&v)[32], float dq, float bias, float leaky, float *__restrict__ dst,
                                              uint32_t row_stride, int rows_live, int cols_live) {
    // fp32 NCHW: each tile row is 8 consecutive floats of one channel plane
    const bool vec = cols_live == 8 && ((reinterpret_cast<uintptr_t>(dst) | ((uintptr_t)row_stride * 4)) & 15) == 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (r >= rows_live) break;
        float *row = dst + (size_t)r * row_stride;
        if (vec) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float4 o;
                o.x = epi_value<ACT>(v[8 * r + 4 * h + 0], dq, bias, leaky);
                o.y = epi_value<ACT>(v[8 * r + 4 * h + 1], dq, bias, leaky);
                o.z = epi_value<ACT>(v[8 * r + 4 * h + 2], dq, bias, leaky);
                o.w = epi_value<ACT>(v[8 * r + 4 * h + 3], dq, bias, leaky);
                reinterpret_cast<float4 *>(row)[h] = o;
            }
        } else {
#pragma unroll
            for (int cidx = 0; cidx < 8; ++cidx)
                if (cidx < cols_live) row[cidx] = epi_value<ACT>(v[8 * r + cidx], dq, bias, leaky);
        }
    }
}

// Pixel-major fp32 tensors in the swapped orientation: for one pixel the warp's 32 lanes touch 32 consecutive floats
// (residual read, fp32 write) and 32 consecutive int8 (requantized write): every access is one coalesced line.
template <int ACT, bool EVEN, bool AFTER>
__device__ __forceinline__ bool swap_nhwc_run(const int (&v)[32], float dq, float bias, float leaky,
                                              const float *__restrict__ res, float *__restrict__ out_f32,
                                              int8_t *__restrict__ out_i8, bool write_i8, float rs0, float rs1, int split,
                                              uint32_t O, uint32_t out_cp, bool ch_live) {
    float worst = 0.0f;
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 8) {
        float r[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) r[k] = (res && ch_live) ? __ldg(res + (uint32_t)(j0 + k) * O) : 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int j = j0 + k;
            float t = __fadd_rn(__fmul_rn(__int2float_rn(v[j]), dq), bias);
            if (res && !AFTER) t = __fadd_rn(t, r[k]);
            if (ACT == TSB_ACT_RELU) t = fmaxf(t, 0.0f);
            if (ACT == TSB_ACT_LEAKY_RELU) t = t > 0.0f ? t : __fmul_rn(t, leaky);
            if (res && AFTER) t = __fadd_rn(t, r[k]);
            if (out_f32 && ch_live) out_f32[(uint32_t)j * O] = t;
            if (out_i8) {
                const float u = __fmul_rn(t, j < split ? rs0 : rs1);
                worst = max_nan(worst, fabsf(u));
                const int q = round_s8<EVEN>(u);
                if (write_i8) out_i8[(uint32_t)j * out_cp] = (int8_t)q;   // redone by the caller if the check below fails
            }
        }
    }
    return !__any_sync(0xffffffffu, !(worst < 2147483648.0f));
}

// Calls f(activation) / f(activation, half-to-even) / ... with the run-time choices as compile-time constants.
template <typename F>
__device__ __forceinline__ void with_act(int act, F f) {
    if (act == TSB_ACT_RELU) f(std::integral_constant<int, TSB_ACT_RELU>());
    else if (act == TSB_ACT_LEAKY_RELU) f(std::integral_constant<int, TSB_ACT_LEAKY_RELU>());
    else f(std::integral_constant<int, TSB_ACT_NONE>());
}
template <typename F>
__device__ __forceinline__ void with_act_flag(int act, int flag, F f) {
    if (flag) with_act(act, [&](auto a) { f(a, std::true_type()); });
    else with_act(act, [&](auto a) { f(a, std::false_type()); });
}
template <typename F>
__device__ __forceinline__ void with_act_flags(int act, int flag, int flag2, F f) {
    if (flag2) with_act_flag(act, flag, [&](auto a, auto e) { f(a, e, std::true_type()); });
    else with_act_flag(act, flag, [&](auto a, auto e) { f(a, e, std::false_type()); });
}
// (the constant behind such an argument)
#define TSB_VAL(x) decltype(x)::value

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ldw(uint32_t taddr, int (&v)[32]) { tmem_ld32(taddr, v); }
__device__ __forceinline__ void tmem_ldw(uint32_t taddr, int (&v)[16]) { tmem_ld16(taddr, v); }

// one tensor-memory column of this warp's 32 lanes (used by the rolled, element-by-element paths)
__device__ __forceinline__ int tmem_ld1(uint32_t taddr) {
    int r;
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    return r;
}

// One scale rounds half to even, except the last count % 8 elements of the tensor (in NCHW order), which round half away from
// zero (epi.tail says whether there are any).  The fast paths round everything half to even; this redoes, element by element, the few
// columns of a chunk that hold such an element.  n_of(j), o_of(j), p_of(j): image, channel and pixel of this thread's column j;
// ok(j): whether the column is one of its outputs.  Called by whole warps.
template <typename Ok, typename N, typename O, typename P>
__device__ __forceinline__ void fix_tail(const EpiParams &epi, uint32_t taddr, Ok ok, N n_of, O o_of, P p_of) {
#pragma unroll 1
    for (int j = 0; j < 32; ++j) {
        const bool mine = ok(j) && ((uint32_t)(n_of(j) * epi.O + o_of(j)) * (uint32_t)epi.P + (uint32_t)p_of(j)) >= epi.rne_limit;
        if (!__any_sync(0xffffffffu, mine)) continue;
        const int a = tmem_ld1(taddr + (uint32_t)j);
        if (mine) epilogue_store_one(epi, n_of(j), o_of(j), p_of(j), a);
    }
}

// ---------------------------------------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------------------------------------
// Division by a divisor known at launch time as multiply-high, add and shift (round-up method for 32-bit unsigned
// numerators below 2^31): the role threads divide once or twice per tile and a hardware-less 32-bit division costs them
// more than a hundred cycles each.
struct FastDiv {
    uint32_t mul = 0, shr = 0;
    FastDiv() = default;
    explicit FastDiv(uint32_t d) {
        uint32_t l = 0;
        while ((1ull << l) < d) ++l;
        shr = l;
        mul = (uint32_t)((((1ull << 32) * ((1ull << l) - d)) / d) + 1);
    }
    __device__ __forceinline__ int div(int n) const {
        return (int)(((uint64_t)__umulhi((uint32_t)n, mul) + (uint32_t)n) >> shr);
    }
};

struct KernelParams {
    int M_total;     // N*OH*OW
    int OW, P;       // P = OH*OW
    int KH, KW;
    int sh, sw, dh, dw, pad_t, pad_l;
    int Cp;          // channels of the staged input per filter tap
    int num_m_tiles, num_n_tiles;   // pixel tiles, channel tiles
    FastDiv d_P, d_OW, d_m_tiles, d_n_tiles, d_segs, d_OH, d_dh;   // dividers by P, OW, num_m_tiles, num_n_tiles, rows_segs, rows_OH, dh
    int a_tiled;           // activations are a plain [M][Cp] matrix (1x1, stride 1, no padding): 2-D tile loads
    // shared-memory plan (bytes from the 1024-aligned base)
    int stages;            // pipeline stages (<= kMaxStages)
    uint32_t stage_bytes;  // one stage: kgroup units of (pixel tile, followed by the weight tile unless the weights are resident)
    int kgroup;            // general mode: K blocks per stage (1, 2 or 4; divides the K blocks of a tile): one barrier wait
                           // and one commit of the MMA issuer serve kgroup * BK/32 MMAs
    uint32_t unit_bytes;   // one K block inside a stage
    int b_resident;        // all K blocks of this CTA's weight tile stay in shared memory; only activations stream
    uint32_t b_off;        // offset of the resident weights
    uint32_t bar_off;      // offset of the mbarriers; tensor-memory slot, abort flag and epilogue tables follow
    uint32_t stg_off;      // staged epilogue: offset of its tiles (1024-aligned): the quads' fp32 tiles, then one int8 tile per quad
    int stg_tiles;         // fp32 tiles per quad: 1 or 2
    int stg_groups;        // groups of epilogue warps, each on its own tile (1, 2 or 4; fewer where the CTA has fewer tiles)
    // raw-row mode (rows_segs > 0): a tile is up to 128 consecutive pixels of ONE output row; per filter row the
    // producer copies the staged bytes under those pixels once, and the MMA reads them through a sliding descriptor
    int rows_segs;         // tiles per output row (0: mode off)
    int rows_OH, rows_H;   // output rows per image, staged input rows per image
    uint32_t rows_bytes;   // bytes copied per tile and filter row
    long long rows_stride_h, rows_stride_n;   // bytes between staged rows / images
    const int8_t *rows_x;  // the folded staging
    // patch mode (patch != 0; filters with several taps, of stride 1 or, patch == 2, stride 2 and 64 padded channels): a tile is 8 pixels wide and PIX/8 pixels high; ONE
    // tiled tensor-map load per channel block brings the input patch under it, halo included, and every filter tap reads
    // its shifted window out of that patch through a descriptor whose start is moved by whole pixels
    int patch;
    int patch_tiles_w, patch_tiles_hw;        // tiles across an image, tiles per image
    int patch_pw;                             // patch width in pixels (8 + (KW-1)*dw) or pixel pairs
    int patch_left;                           // columns (pairs) of the patch left of the tile's first pixel (of its pair): pad_l or (pad_l+1)/2
    uint32_t patch_bytes;                     // bytes of one patch (one channel block)
    int OH;
    FastDiv d_tiles_w, d_tiles_hw;
    int res_prefetch;      // swapped orientation: the residual tensor has a tensor map (map_r), by which the epilogue prefetches boxes of it into
                           // L2 two chunks ahead of the registers' loads, so that those find the data on chip
    int *status;     // device word: 0 ok, else the code of the wait that ran out
    unsigned long long *trace;  // profiling builds: timeline of CTA 0, 8 stamps per tile, 32 tiles (null otherwise)
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
#ifdef TSB_ENABLE_TRACE
#define TSB_TRACE(tile_index, slot)                                                              \
    do {                                                                                         \
        if (kp.trace && blockIdx.x == 0 && (tile_index) < 32) kp.trace[(tile_index) * 8 + (slot)] = global_ns(); \
    } while (0)
// cycle accounting of the MMA issuer (profiling builds): where its time goes, summed over the CTA's tiles
#define TSB_CYC_DECL long long cyc_full = 0, cyc_tempty = 0, cyc_issue = 0, cyc_commit = 0, cyc_t0 = clock64(), cyc_tmp = 0; int cyc_waits = 0
#define TSB_CYC_START cyc_tmp = clock64()
#define TSB_CYC_ADD(which) do { which += clock64() - cyc_tmp; } while (0)
#define TSB_CYC_REPORT(ntiles)                                                                   \
    do {                                                                                         \
        if (kp.trace && blockIdx.x == 0) {                                                       \
            kp.trace[31 * 8 + 0] = (unsigned long long)(clock64() - cyc_t0);                     \
            kp.trace[31 * 8 + 1] = (unsigned long long)cyc_full;                                 \
            kp.trace[31 * 8 + 2] = (unsigned long long)cyc_tempty;                               \
            kp.trace[31 * 8 + 3] = (unsigned long long)(ntiles);                                 \
            kp.trace[31 * 8 + 4] = (unsigned long long)cyc_waits;                                \
            kp.trace[31 * 8 + 5] = (unsigned long long)cyc_issue;                                \
            kp.trace[31 * 8 + 6] = (unsigned long long)cyc_commit;                               \
        }                                                                                        \
    } while (0)
#else
#define TSB_TRACE(tile_index, slot) do { } while (0)
#define TSB_CYC_DECL do { } while (0)
#define TSB_CYC_START do { } while (0)
#define TSB_CYC_ADD(which) do { } while (0)
#define TSB_CYC_REPORT(ntiles) do { } while (0)
#endif

// raw-row mode: the filter rows kh_lo..kh_hi that meet an input row for output row oh (a contiguous, non-empty range)
__device__ __forceinline__ void rows_span(const KernelParams &kp, int oh, int &kh_lo, int &kh_hi) {
    const int top = oh * kp.sh - kp.pad_t;                 // input row under filter row 0
    kh_lo = top >= 0 ? 0 : kp.d_dh.div(-top + kp.dh - 1);
    kh_hi = min(kp.KH - 1, kp.d_dh.div(kp.rows_H - 1 - top));
}

// Patch mode: distance of filter tap (kh, kw)'s window from the start of a patch, in bytes.  In a patch of pixel pairs (stride 2) a row of
// shared memory is an even and an odd pixel of 64 channels each, so a tap takes one half of the pair it falls on.
template <int BK>
__device__ __forceinline__ uint32_t patch_tap(const KernelParams &kp, int kh, int kw) {
    if (kp.patch == 2) {
        const int col = kw - kp.pad_l;
        return (uint32_t)((kh * kp.patch_pw + (col >> 1) + kp.patch_left) * 128 + (col & 1) * 64);
    }
    return (uint32_t)((kh * kp.dh * kp.patch_pw + kw * kp.dw) * BK);
}

// kModeSplit: as kModeGeneral, but the K blocks of a tile are shared out over the kSplit CTAs of a cluster, for layers whose tiles
// leave most of the GPU idle: one SM takes in its operands at about 60 bytes a cycle however many there are.  BN = 128 only: each of the
// four CTAs adds up and finishes one 32-channel chunk of the tile (int32 sums are exact in any order).
constexpr int kModeGeneral = 0, kModeRows = 1, kModePatch = 2, kModeSplit = 3;

// Projected-shortcut kernels (DUAL): a second, 1x1 convolution over the same output pixels (the projection shortcut of a
// residual block: its own input, weights, dequantize scales and bias) runs in the same tile, into a second accumulator,
// ahead of the main convolution; the epilogue dequantizes it (+ bias) and uses the result as the main convolution's
// residual.  The projection's fp32 output never exists in global memory.
struct alignas(64) DualParams {
    CUtensorMap map_a2, map_b2;   // the projection's activations ([M][Cp2] tiles or a 1x1 im2col walk with its stride) and weights
    const float *dq2, *bias2;     // its dequantize scales and (optional) bias, per output channel
    int k2_iters;                 // its K blocks per tile: Cp2 / BK
    int Cp2, a2_tiled, sh2, sw2;
    int concat;                   // 1: no second accumulator and no residual -- the second convolution's K blocks are summed into
                                  // the main accumulator, i.e. ONE convolution over the channel concatenation of the two inputs
                                  // (int32 sums are exact in any order); dq2 / bias2 are unused
};
struct NoDual {};
constexpr int kMaxStages = 24;
constexpr uint32_t kMaxDynamicSmem = 227 * 1024;

// barriers, in this order: full[stages], empty[stages], tmem_full[4], tmem_empty[4], b_full, b_free, and for the staged
// epilogue's tiles ready[4 quads][2], full[4][2], int8_free[4]; split-K: the partial sums of the other CTAs are here
__host__ __device__ constexpr uint32_t num_barriers(int stages) { return 2u * (uint32_t)stages + 2u * kMaxAccBufs + 2u + 5u * kQuads + 1u; }

// PIX pixels x CH channels per tile.  Normal orientation: the pixel tile is the MMA's A operand (M = 128 pixels), the
// weight tile its B operand (N = BN channels).  Swapped orientation: the weight tile is A (M = 128 channels, rows
// beyond O zero-filled by the tensor map) and the pixel tile is B (N = BN pixels).  An MMA instruction takes the tensor core 128 cycles at
// N = 256, 64 at 128 and 48 at 64, but the issuing warp 77-115 whatever its N, so narrow multi-tap layers run swapped: N = 256 pixels
// where N = O would leave the tensor core waiting.
// MODE: how activations reach shared memory -- kModeGeneral (im2col or plain 2-D tile loads), kModeSplit (the same, K shared out over a
// cluster), kModeRows (raw-row), kModePatch.
// A compile-time parameter: the role loops of each mode stay short and keep their registers.
template <int BN, int BK, bool SWAP, int MODE, int EPI, bool DUAL>
__global__ void __launch_bounds__(cta_threads(EPI), 1)
conv_i8_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_of,
                  const __grid_constant__ CUtensorMap map_oi, const __grid_constant__ KernelParams kp,
                  const __grid_constant__ EpiParams epi,
                  const __grid_constant__ std::conditional_t<DUAL, DualParams, NoDual> dual) {
    constexpr bool SPLIT = MODE == kModeSplit;
    static_assert(!SPLIT || (!SWAP && BN == 32 * kSplit), "split-K: one 32-channel chunk of the tile per CTA of the cluster");
    static_assert(!DUAL || (!SWAP && MODE == kModeGeneral), "projected-shortcut kernels: normal orientation, general mode");
    static_assert(SWAP ? !is_staged(EPI) : (EPI != kEpiNhwc || MODE == kModeRows), "pixel-major fp32 tensors: staged tiles where a thread owns a pixel");
    constexpr int PIX = SWAP ? BN : kBM;      // pixels per tile
    constexpr int CH = SWAP ? kBM : BN;       // output channels per tile
    constexpr uint32_t kPixBytes = PIX * BK, kWgtBytes = CH * BK;
    constexpr int kBufs = 512 / BN < kMaxAccBufs ? 512 / BN : kMaxAccBufs;   // accumulator buffers: 2 for BN = 256, else 4
    constexpr uint32_t kTmemCols = 512;                                       // one CTA per SM: all of tensor memory
    const int kStages = kp.stages;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *base_ptr = smem_raw + (base - raw);
    const uint32_t bar_full = base + kp.bar_off;
    const uint32_t bar_empty = bar_full + 8 * kStages;
    const uint32_t bar_tfull = bar_empty + 8 * kStages;
    const uint32_t bar_tempty = bar_tfull + 8 * kMaxAccBufs;
    const uint32_t bar_bfull = bar_tempty + 8 * kMaxAccBufs;
    const uint32_t bar_bfree = bar_bfull + 8;
    const uint32_t bar_stg = bar_bfree + 8;     // the staged epilogue's
    const uint32_t bar_parts = bar_stg + 8 * 5 * kQuads;    // split-K
    const uint32_t slot_off = kp.bar_off + 8 * num_barriers(kStages);
    volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(base_ptr + slot_off);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(base_ptr + slot_off + 4);
    float *table = reinterpret_cast<float *>(base_ptr + ((slot_off + 8 + 15) & ~15u));
    // patch mode: (byte offset >> 4) of every filter tap's window inside a patch, for the MMA issuer
    uint32_t *tap16 = reinterpret_cast<uint32_t *>(table + kMaxAccBufs * 2 * BN);
    const uint32_t w_res = base + kp.b_off;   // resident weights

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (known to be uniform)
    const int total_tiles = kp.num_m_tiles * kp.num_n_tiles;
    const int k_iters = kp.KH * kp.KW * (kp.Cp / BK);
    int k_sc = 0;                              // K blocks of the projection, which come first in every tile
    bool concat = false;
    if constexpr (DUAL) { k_sc = dual.k2_iters; concat = dual.concat != 0; }
    // This CTA's tiles.  Streaming weights: tiles blockIdx.x, +gridDim.x, ... with the channel tile running fastest.
    // Resident weights: one contiguous range of the channel-major tile order, so the weight tile changes at most a
    // few times.
    const int rank = SPLIT ? (int)blockIdx.x % kSplit : 0;                     // split-K: the CTA of its cluster (clusters are consecutive CTAs)
    const int k_lo = SPLIT ? k_iters * rank / kSplit : 0, k_hi = SPLIT ? k_iters * (rank + 1) / kSplit : k_iters;
    const int tile_lo = kp.b_resident ? (int)((long long)blockIdx.x * total_tiles / gridDim.x) : 0;
    const int tile_hi = kp.b_resident ? (int)((long long)(blockIdx.x + 1) * total_tiles / gridDim.x) : 0;
    const int my_tiles = SPLIT ? 1 : kp.b_resident ? tile_hi - tile_lo : (total_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    // Accumulator buffers in use = epilogue groups: as many as tensor memory holds (kBufs), but no more than this CTA has
    // tiles -- a CTA with a single tile puts all sixteen epilogue warps on it.
    // (a projected-shortcut tile holds two accumulators: buffers 2a and 2a+1 of logical buffer a)
    const int nbuf = DUAL ? ((kBufs >= 4 && my_tiles >= 2) ? 2 : 1) : (my_tiles >= 4 && kBufs >= 4 ? 4 : (my_tiles >= 2 ? 2 : 1));
    // Epilogue groups: one per buffer, each on its own tile; in the staged class as many as the configuration says.
    const int groups = is_staged(EPI) ? min(kp.stg_groups, nbuf) : nbuf;
    auto decode = [&](int i, int &m_tile, int &n_tile) {   // m_tile: pixel tile, n_tile: channel tile
        if (kp.b_resident) {
            const int t = tile_lo + i;
            n_tile = kp.d_m_tiles.div(t); m_tile = t - n_tile * kp.num_m_tiles;
        } else {
            const int t = SPLIT ? (int)blockIdx.x / kSplit : (int)blockIdx.x + i * (int)gridDim.x;
            m_tile = kp.d_n_tiles.div(t); n_tile = t - m_tile * kp.num_n_tiles;
        }
    };

    // raw rows of several tiles: both issuers consume one ring (below)
    const bool shared_ring = MODE == kModeRows && kp.rows_segs > 1;
    if (threadIdx.x == 0) TSB_TRACE(0, 7);
    if (warp == 0) {
        // one barrier per lane and step (a single thread takes 0.3 us for the eighty of them); the descriptors' first fetch
        // overlaps the wait for the previous kernel
        for (int i = lane; i < (int)num_barriers(kStages); i += 32) {
            const int t = i - 2 * kStages;                                            // full, empty: one arrival each (empty: one per issuer of a shared ring)
            const bool tempty = t >= kMaxAccBufs && t < 2 * kMaxAccBufs;
            const int stg = t - (2 * kMaxAccBufs + 2);                                // staged tiles: ready, full, int8 free
            const bool full = stg >= 2 * kQuads && stg < 4 * kQuads;
            const bool parts_in = stg == 5 * kQuads;                                  // four warps of each of the other CTAs
            const bool empty = i >= kStages && t < 0;
            mbar_init(bar_full + 8 * i, empty ? (shared_ring ? kIssuers : 1) : tempty ? kEpiThreads / groups : (full ? 4 : (parts_in ? 4 * (kSplit - 1) : 1)));
        }
        if (lane == 0) {
            *abort_flag = 0;
            if (MODE != kModeRows) prefetch_tensormap(&map_a);
            prefetch_tensormap(&map_b);
            if constexpr (DUAL) { prefetch_tensormap(&dual.map_a2); prefetch_tensormap(&dual.map_b2); }
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t *>(tmem_slot)), kTmemCols);
        tmem_relinquish();
    }
    if (MODE == kModePatch && threadIdx.x >= 32 * kEpiWarp0) {
        for (int t = (int)threadIdx.x - 32 * kEpiWarp0; t < kp.KH * kp.KW; t += kEpiThreads) {
            const int kh = t / kp.KW, kw = t - kh * kp.KW;
            tap16[t] = patch_tap<BK>(kp, kh, kw) >> 4;
        }
    }
    // How many warps issue MMAs, each for every such tile of the CTA.  One where tiles share state that one thread has to order --
    // resident weights that are replaced inside this CTA's tile range -- and where the ring of stages has no room for a tile of each issuer.
    // Each issuer has a ring of stages of its own (stages [i * kStages / issuers, ...) for issuer i), which the producer fills for
    // that issuer's tiles.  A barrier wait names a phase by its parity only; in a ring that nobody else consumes, an issuer
    // has itself seen the round before the one it waits for.  (With one ring for both, an issuer could arrive at a stage while the
    // other issuer's tile of the round before was still being loaded -- loads complete out of order -- and pass its wait.)
    // (Raw-row stages that several tiles of an output row share are the exception: there both issuers walk all rows through one ring,
    // and a stage is free when both have said so -- each sees every fill.)
    int issuers = 1;
    if (my_tiles > 1 && warp <= kIssuers) {
        const int spt = MODE == kModePatch ? kp.Cp / BK : (MODE == kModeRows ? 1 : (k_iters + k_sc) / kp.kgroup);   // stages a tile consumes
        bool shared_state = false;
        if (kp.b_resident && kp.num_n_tiles > 1) {
            int first_m, first_n, last_m, last_n;
            decode(0, first_m, first_n);
            decode(my_tiles - 1, last_m, last_n);
            shared_state = first_n != last_n;
        }
        // (an issuer must also own its accumulator buffers: with a single logical buffer one thread takes every tile)
        if (!shared_state && (shared_ring || kStages >= kIssuers * spt) && !(DUAL && nbuf < kIssuers)) issuers = kIssuers;
    }
    const int ring = issuers > 1 && !shared_ring ? kStages / kIssuers : kStages;
    tc_fence_before();
    __syncthreads();
    if constexpr (SPLIT) cluster_arrive();      // this CTA's barriers are initialised
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    pdl_sync();   // everything above touched only shared and tensor memory

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        // Like the issuers below, the whole warp walks the tiles and one elected lane issues: 64 images of ResNet-50 1.155 -> 1.137 ms, 8 images
        // 0.424 -> 0.404; CSPDarknet53, 16 images 2.58 -> 2.46 ms, one image 0.570 -> 0.534.
        {
            int stage = 0, stage_lo = 0, stage_alt = ring;                  // absolute stage, first stage of its ring; the other ring's
            uint32_t phase = 0, phase_alt = 0;
            auto next_stage = [&]() { if (++stage == stage_lo + ring) { stage = stage_lo; phase ^= 1u; } };
            bool ok = true;
            int cur_n = -1, w_loads = 0;
            const uint32_t tx_bytes = (uint32_t)kp.kgroup * (kp.b_resident ? kPixBytes : kPixBytes + kWgtBytes);
            for (int i = 0; i < my_tiles && ok; ++i) {
                if (i > 0 && issuers > 1 && !shared_ring) {                              // the next tile is the other issuer's
                    const int s = stage; stage = stage_alt; stage_alt = s;
                    const uint32_t p = phase; phase = phase_alt; phase_alt = p;
                    stage_lo = ring - stage_lo;
                }
                TSB_TRACE(i, 0);
                int m_tile, n_tile;
                decode(i, m_tile, n_tile);
                const int m0 = m_tile * PIX;
                const int img = kp.d_P.div(m0), rem = m0 - img * kp.P;
                const int oh = kp.d_OW.div(rem), ow = rem - oh * kp.OW;
                const int wc = ow * kp.sw - kp.pad_l, hc = oh * kp.sh - kp.pad_t;
                if (kp.b_resident && n_tile != cur_n) {
                    // (re)load the whole weight tile; wait until the MMAs that read the previous one are done
                    if (w_loads > 0 && !mbar_wait_warp(bar_bfree, (uint32_t)(w_loads - 1) & 1u, abort_flag)) {
                        if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 5); }
                        break;
                    }
                    if (elect_one()) {
                        mbar_arrive_expect_tx(bar_bfull, (uint32_t)(k_iters + k_sc) * kWgtBytes);
                        if constexpr (DUAL)
                            for (int it = 0; it < k_sc; ++it)
                                tma_load_2d(w_res + (uint32_t)it * kWgtBytes, &dual.map_b2, bar_bfull, it * BK, n_tile * CH);
                        for (int it = 0; it < k_iters; ++it)
                            tma_load_2d(w_res + (uint32_t)(k_sc + it) * kWgtBytes, &map_b, bar_bfull, it * BK, n_tile * CH);
                    }
                    cur_n = n_tile;
                    ++w_loads;
                }
                if (MODE == kModePatch) {
                    const int p_img = kp.d_tiles_hw.div(m_tile), p_rem = m_tile - p_img * kp.patch_tiles_hw;
                    const int p_r = kp.d_tiles_w.div(p_rem), p_c = p_rem - p_r * kp.patch_tiles_w;
                    const int h0 = p_r * (PIX / 8) * kp.sh - kp.pad_t, w0 = p_c * 8 - kp.patch_left;
                    for (int cb = 0; cb < kp.Cp && ok; cb += BK) {
                        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
                            if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 1); }
                            ok = false;
                            break;
                        }
                        if (elect_one()) {
                            mbar_arrive_expect_tx(bar_full + 8 * stage, kp.patch_bytes);
                            tma_load_4d(base + stage * kp.stage_bytes, &map_a, bar_full + 8 * stage, cb, w0, h0, p_img);
                        }
                        next_stage();
                    }
                } else if (MODE == kModeRows) {
                    // One copy per output row (per run of its segments that this CTA owns): the staged bytes from the
                    // first to the last input row the filter meets, from this segment to the end of the row.  The
                    // following tiles of the same output row read the same stage at +2048 bytes per segment.
                    const int row_id = kp.d_segs.div(m_tile), seg = m_tile - row_id * kp.rows_segs;
                    if (seg == 0 || i == 0) {
                        const int r_img = kp.d_OH.div(row_id), r_oh = row_id - r_img * kp.rows_OH;
                        int kh_lo, kh_hi;
                        rows_span(kp, r_oh, kh_lo, kh_hi);
                        if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
                            if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 1); }
                            break;
                        }
                        const int ih_lo = r_oh * kp.sh - kp.pad_t + kh_lo * kp.dh;
                        const uint32_t bytes = (uint32_t)((kh_hi - kh_lo) * kp.dh) * (uint32_t)kp.rows_stride_h +
                                               (uint32_t)(kp.rows_segs - 1 - seg) * (PIX * 16) + kp.rows_bytes;
                        if (elect_one()) {
                            mbar_arrive_expect_tx(bar_full + 8 * stage, bytes);
                            bulk_load(base + stage * kp.stage_bytes,
                                      kp.rows_x + r_img * kp.rows_stride_n + ih_lo * kp.rows_stride_h + (long long)seg * (PIX * 16),
                                      bytes, bar_full + 8 * stage);
                        }
                        next_stage();
                    }
                } else {
                    int gk = 0;   // K block inside the current stage
                    if constexpr (DUAL) {
                        const int wc2 = ow * dual.sw2, hc2 = oh * dual.sh2;   // the projection: 1x1, no padding
                        for (int cb = 0; cb < dual.Cp2; cb += BK) {
                            if (gk == 0) {
                                if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
                                    if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 1); }
                                    ok = false;
                                    break;
                                }
                            }
                            const uint32_t sp = base + stage * kp.stage_bytes + (uint32_t)gk * kp.unit_bytes, sw = sp + kPixBytes;
                            if (elect_one()) {
                                if (gk == 0) mbar_arrive_expect_tx(bar_full + 8 * stage, tx_bytes);
                                if (dual.a2_tiled) tma_load_2d(sp, &dual.map_a2, bar_full + 8 * stage, cb, m0);
                                else tma_load_im2col_4d(sp, &dual.map_a2, bar_full + 8 * stage, cb, wc2, hc2, img, (uint16_t)0, (uint16_t)0);
                                if (!kp.b_resident) tma_load_2d(sw, &dual.map_b2, bar_full + 8 * stage, cb, n_tile * CH);
                            }
                            if (++gk == kp.kgroup) {
                                gk = 0;
                                next_stage();
                            }
                        }
                    }
                    int kh_0 = 0, kw_0 = 0, cb_0 = 0, left = k_hi - k_lo;       // (split-K: from the middle of a tap to the middle of another)
                    if constexpr (SPLIT) {
                        const int blocks = kp.Cp / BK, tap = k_lo / blocks;
                        kh_0 = tap / kp.KW; kw_0 = tap - kh_0 * kp.KW; cb_0 = (k_lo - tap * blocks) * BK;
                    }
                    for (int kh = kh_0; kh < kp.KH && ok; ++kh, kw_0 = 0)
                        for (int kw = kw_0; kw < kp.KW && ok; ++kw, cb_0 = 0)
                            for (int cb = cb_0; cb < kp.Cp; cb += BK) {
                                if (SPLIT && left-- == 0) { ok = false; break; }
                                if (gk == 0) {
                                    if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1u, abort_flag)) {
                                        if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 1); }
                                        ok = false;
                                        break;
                                    }
                                }
                                const uint32_t sp = base + stage * kp.stage_bytes + (uint32_t)gk * kp.unit_bytes, sw = sp + kPixBytes;
                                if (elect_one()) {
                                    if (gk == 0) mbar_arrive_expect_tx(bar_full + 8 * stage, tx_bytes);
                                    if (kp.a_tiled)
                                        tma_load_2d(sp, &map_a, bar_full + 8 * stage, cb, m0);
                                    else
                                        tma_load_im2col_4d(sp, &map_a, bar_full + 8 * stage, cb, wc, hc, img,
                                                           (uint16_t)(kw * kp.dw), (uint16_t)(kh * kp.dh));
                                    if (!kp.b_resident)
                                        tma_load_2d(sw, &map_b, bar_full + 8 * stage, (kh * kp.KW + kw) * kp.Cp + cb, n_tile * CH);
                                }
                                if (++gk == kp.kgroup) {
                                    gk = 0;
                                    next_stage();
                                }
                            }
                }
                TSB_TRACE(i, 1);
            }
        }
    } else if (warp <= kIssuers) {
        // ------------------------------------------------------------------ MMA issuers
        // One thread at a time feeds the tensor core, but its whole warp walks the tiles: an MMA takes its descriptors from uniform registers,
        // and where the code is known to run converged (waits that answer through a vote, the issuing lane chosen by elect.sync) they are
        // computed there; a lane that runs alone moves every operand over instead.  64 images: ResNet-50 1.20 -> 1.15 ms, 8 images
        // 0.452 -> 0.424 ms; CSPDarknet53, 16 images 2.71 -> 2.58 ms, one image 0.609 -> 0.570 ms.
        // The MMAs of a stage are straight-line code; descriptors are a loop-invariant high word plus a 14-bit address field (in
        // 16-byte units) that takes one add; slots that do not apply are switched off by predicate; and one barrier wait / one
        // commit serve as many MMAs as the stage holds.  What is spent between two MMAs is not hidden behind the tensor core's work on the
        // earlier one, so kIssuers warps issue, each for every kIssuers-th tile of the CTA: while one computes, waits and commits, the
        // tensor core runs the other's MMAs.  A tile's stages, accumulator buffer and barriers belong to the issuer of that
        // tile alone.
        {
            constexpr uint32_t idesc = instr_desc<BN>();
            constexpr uint64_t dhi = smem_desc_hi<BK>(8 * BK);
            constexpr uint32_t kWgt16 = kWgtBytes >> 4, kPix16 = kPixBytes >> 4;
            constexpr int kMmaPerBlock = BK / 32;
            const uint32_t base16 = base >> 4, stage16 = kp.stage_bytes >> 4, wres16 = w_res >> 4, unit16 = kp.unit_bytes >> 4;
            const int resident = kp.b_resident;
            bool ok = true;
            const int me = warp - 1, stage_lo = shared_ring ? 0 : me * ring;
            int stage = stage_lo; uint32_t phase = 0;
            // raw rows: the output row whose stage comes next, the segment its copy starts at, whether it is there; the last row of this CTA
            int rows_next = 0, rows_seg_first = 0, rows_last = 0;
            bool rows_held = false;
            if (shared_ring) {
                int m_tile, n_tile;
                decode(0, m_tile, n_tile);
                rows_next = kp.d_segs.div(m_tile); rows_seg_first = m_tile - rows_next * kp.rows_segs;
                decode(my_tiles - 1, m_tile, n_tile);
                rows_last = kp.d_segs.div(m_tile);
            }
            auto rows_pass = [&]() {            // on to the next row; this one's stage is free when the MMAs have read it
                if (elect_one()) {
                    tc_commit(bar_empty + 8 * stage);
                    if (shared_ring && issuers == 1) tc_commit(bar_empty + 8 * stage);      // for the issuer that is not there
                }
                if (++stage == stage_lo + ring) { stage = stage_lo; phase ^= 1u; }
                ++rows_next;
                rows_held = false;
                rows_seg_first = 0;
            };
            auto rows_wait = [&]() {
                if (!rows_held && !mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
                    if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 3); }
                    return false;
                }
                rows_held = true;
                return true;
            };
            int w_loads = resident ? 1 : 0;   // without shared state the resident weights are loaded exactly once
            int cur_n = -1;
            // patch mode with up to nine filter taps (3x3, 1x3 ...): the taps' window offsets live in registers
            const int taps = kp.KH * kp.KW;
            uint32_t tapreg[9];
            {
                int kh = 0, kw = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    tapreg[t] = (MODE == kModePatch && t < taps) ? patch_tap<BK>(kp, kh, kw) >> 4 : 0u;
                    if (++kw == kp.KW) { kw = 0; ++kh; }
                }
            }
            TSB_CYC_DECL;
            for (int local = me; local < my_tiles && ok && me < issuers; local += issuers) {
                int m_tile, n_tile;
                decode(local, m_tile, n_tile);
                uint32_t st16 = base16 + (uint32_t)stage * stage16;    // (address >> 4) of the current stage
                const int acc = local & (nbuf - 1);
                const uint32_t acc_phase = (uint32_t)(local / nbuf) & 1u;
                TSB_CYC_START;
                if (!mbar_wait_warp(bar_tempty + 8 * acc, acc_phase ^ 1u, abort_flag)) {
                    if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 2); }
                    break;
                }
                TSB_CYC_ADD(cyc_tempty);
                if (resident && n_tile != cur_n) {
                    // the (w_loads)-th load of resident weights: completes phase (w_loads - 1) of its barrier
                    if (!mbar_wait_warp(bar_bfull, (uint32_t)(w_loads - 1) & 1u, abort_flag)) {
                        if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 6); }
                        break;
                    }
                    cur_n = n_tile;
                    ++w_loads;
                }
                tc_fence_after();
                if (me == 0) TSB_TRACE(local, 2);
                uint32_t d_tmem = tmem_base + (uint32_t)(DUAL ? (2 * acc + (concat ? 0 : 1)) * BN : acc * BN);   // DUAL: the projection's accumulator first
                uint32_t accumulate = 0;
                if (MODE == kModePatch) {
                    const int n_cb = kp.Cp / BK;
                    // next tile row = next patch row, or the next but one of pixel pairs
                    const uint64_t dhi_patch = kp.patch == 2 ? smem_desc_hi<128>(2u * (uint32_t)kp.patch_pw * 128u) : smem_desc_hi<BK>((uint32_t)kp.patch_pw * BK);
                    const uint32_t hi_patch = (uint32_t)(dhi_patch >> 32), hi_plain = (uint32_t)(dhi >> 32);
                    const uint32_t wtap16 = (uint32_t)n_cb * kWgt16;                          // next tap of the resident weights
                    for (int cbi = 0; cbi < n_cb && ok; ++cbi) {
                        TSB_CYC_START;
                        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
                            if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 3); }
                            ok = false;
                            break;
                        }
                        TSB_CYC_ADD(cyc_full);
                        tc_fence_after();
                        if (cbi == 0 && me == 0) TSB_TRACE(local, 3);
                        uint32_t w16 = wres16 + (uint32_t)cbi * kWgt16;
                        TSB_CYC_START;
                        if (elect_one()) {
                        if (taps == 9) {
                            // 3x3: eighteen or thirty-six MMAs, two adds each
                            const uint32_t p_lo = st16 | kDescLbo;
#pragma unroll
                            for (int t = 0; t < 9; ++t) {
                                const uint32_t a_lo = p_lo + tapreg[t], w_lo = (w16 | kDescLbo) + (uint32_t)t * wtap16;
#pragma unroll
                                for (int k = 0; k < kMmaPerBlock; ++k) {
                                    const uint64_t dp = desc_pair(hi_patch, a_lo + 2u * k), dw = desc_pair(hi_plain, w_lo + 2u * k);
                                    mma_i8(d_tmem, SWAP ? dw : dp, SWAP ? dp : dw, idesc, (t | k) ? 1u : accumulate);
                                }
                            }
                            accumulate = 1u;
                        } else if (taps < 9) {
#pragma unroll
                            for (int t = 0; t < 9; ++t) {
                                const uint64_t dp = dhi_patch | (uint64_t)(st16 + tapreg[t]);
                                const uint64_t dw = dhi | (uint64_t)w16;
                                const uint64_t da = SWAP ? dw : dp, db = SWAP ? dp : dw;
                                const uint32_t on = t < taps ? 1u : 0u;
#pragma unroll
                                for (int k = 0; k < kMmaPerBlock; ++k)
                                    mma_i8_if(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (t | k) ? 1u : accumulate, on);
                                w16 += wtap16;
                            }
                            accumulate = 1u;
                        } else {
                            for (int t = 0; t < taps; ++t) {
                                const uint64_t dp = dhi_patch | (uint64_t)(st16 + tap16[t]);
                                const uint64_t dw = dhi | (uint64_t)w16;
                                const uint64_t da = SWAP ? dw : dp, db = SWAP ? dp : dw;
#pragma unroll
                                for (int k = 0; k < kMmaPerBlock; ++k) {
                                    mma_i8(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, accumulate);
                                    accumulate = 1u;
                                }
                                w16 += wtap16;
                            }
                        }
                        tc_commit(bar_empty + 8 * stage);
                        }
                        accumulate = 1u;
                        TSB_CYC_ADD(cyc_issue);
                        st16 += stage16;
                        if (++stage == stage_lo + ring) { stage = stage_lo; phase ^= 1u; st16 = base16 + (uint32_t)stage_lo * stage16; }
                    }
                } else if (!SWAP && MODE == kModeRows) {
                    const int row_id = kp.d_segs.div(m_tile), seg = m_tile - row_id * kp.rows_segs;
                    int kh_lo, kh_hi;
                    rows_span(kp, row_id - kp.d_OH.div(row_id) * kp.rows_OH, kh_lo, kh_hi);
                    if (shared_ring) {
                        // a row without a tile of this issuer (the CTA's first, with a single tile, of the other's) is passed by
                        while (issuers > 1 && ok && rows_next < row_id) {
                            ok = rows_wait();
                            if (ok) rows_pass();
                        }
                        st16 = base16 + (uint32_t)stage * stage16;
                    }
                    ok = ok && rows_wait();
                    if (!ok) break;
                    tc_fence_after();
                    if (me == 0) TSB_TRACE(local, 3);
                    // sliding descriptor (no swizzle, LBO 16, SBO 128): only its address field changes from row to row
                    const uint64_t dslide = smem_desc_sliding(0);
                    const uint32_t row16 = (uint32_t)kp.dh * (uint32_t)(kp.rows_stride_h >> 4);
                    // filter row kh reads the staged row (kh - kh_lo); rows outside [kh_lo, kh_hi] meet no input row
                    const uint32_t a16_0 = st16 + (uint32_t)(seg - rows_seg_first) * PIX - (uint32_t)kh_lo * row16;
                    const bool row_done = seg + issuers >= kp.rows_segs || local + issuers >= my_tiles;    // this issuer's last tile of the row
                    if (elect_one()) {
                    if (kp.KH <= 8) {
                        // straight-line code for the filter heights in use (a predicated-off MMA still costs the issuing
                        // thread some 50 cycles, so the sequence is as long as the filter is high, not always eight)
                        auto issue_rows = [&](auto height) {
                            constexpr int kH = decltype(height)::value;
                            if (kh_lo == 0 && kh_hi == kH - 1) {
                                // every filter row meets an input row (all output rows but those at the image's edge): no
                                // predicates, accumulate flags known at compile time
#pragma unroll
                                for (int kh = 0; kh < kH; ++kh) {
                                    const uint64_t da = dslide | (uint64_t)((a16_0 + (uint32_t)kh * row16) & 0x3FFFu);
                                    const uint64_t db = dhi | (uint64_t)(wres16 + (uint32_t)kh * kWgt16);
#pragma unroll
                                    for (int k = 0; k < kMmaPerBlock; ++k)
                                        mma_i8(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kh | k) ? 1u : 0u);
                                }
                                return;
                            }
#pragma unroll
                            for (int kh = 0; kh < kH; ++kh) {
                                const uint64_t da = dslide | (uint64_t)((a16_0 + (uint32_t)kh * row16) & 0x3FFFu);
                                const uint64_t db = dhi | (uint64_t)(wres16 + (uint32_t)kh * kWgt16);
                                const uint32_t on = (kh >= kh_lo && kh <= kh_hi && kh < kp.KH) ? 1u : 0u;
#pragma unroll
                                for (int k = 0; k < kMmaPerBlock; ++k)
                                    mma_i8_if(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (kh > kh_lo || k > 0) ? 1u : 0u, on);
                            }
                        };
                        if (kp.KH <= 3) issue_rows(std::integral_constant<int, 3>());
                        else if (kp.KH <= 5) issue_rows(std::integral_constant<int, 5>());
                        else if (kp.KH <= 7) issue_rows(std::integral_constant<int, 7>());
                        else issue_rows(std::integral_constant<int, 8>());
                    } else {
                        for (int kh = kh_lo; kh <= kh_hi; ++kh) {
                            const uint64_t da = dslide | (uint64_t)(a16_0 + (uint32_t)kh * row16);
                            const uint64_t db = dhi | (uint64_t)(wres16 + (uint32_t)kh * kWgt16);
#pragma unroll
                            for (int k = 0; k < kMmaPerBlock; ++k) {
                                mma_i8(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, accumulate);
                                accumulate = 1u;
                            }
                        }
                    }
                    }
                    if (row_done) rows_pass();
                } else {
                    // general mode: a stage holds kgroup K blocks; one wait, kgroup * BK/32 MMAs in a row, one commit
                    uint32_t w16 = wres16;
                    const int G = kp.kgroup;
                    const uint32_t hi_plain = (uint32_t)(dhi >> 32);
                    auto issue_stage = [&](auto group) {      // the MMAs of one stage as straight-line code
                        constexpr int kG = decltype(group)::value;
#pragma unroll
                        for (int g = 0; g < kG; ++g) {
                            const uint32_t a_lo = (st16 | kDescLbo) + (uint32_t)g * unit16;
                            const uint32_t w_lo = resident ? (w16 | kDescLbo) + (uint32_t)g * kWgt16 : a_lo + kPix16;
#pragma unroll
                            for (int k = 0; k < kMmaPerBlock; ++k) {
                                // +32 bytes along K = +2 in the descriptor's 16-byte address units (inside the swizzle span)
                                const uint64_t dp = desc_pair(hi_plain, a_lo + 2u * k), dw = desc_pair(hi_plain, w_lo + 2u * k);
                                mma_i8(d_tmem, SWAP ? dw : dp, SWAP ? dp : dw, idesc, (g | k) ? 1u : accumulate);
                            }
                        }
                    };
                    for (int it = k_lo; it < k_hi + k_sc; it += G) {
                        if (DUAL && it == k_sc && !concat) { d_tmem -= BN; accumulate = 0u; }   // the main convolution's accumulator
                        TSB_CYC_START;
                        if (!mbar_wait_warp(bar_full + 8 * stage, phase, abort_flag)) {
                            if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 3); }
                            ok = false;
                            break;
                        }
                        TSB_CYC_ADD(cyc_full);
                        tc_fence_after();
                        if (it == k_lo && me == 0) TSB_TRACE(local, 3);
                        TSB_CYC_START;
                        if (elect_one()) {
                            if (G == 4) issue_stage(std::integral_constant<int, 4>());
                            else if (G == 2) issue_stage(std::integral_constant<int, 2>());
                            else issue_stage(std::integral_constant<int, 1>());
                            tc_commit(bar_empty + 8 * stage);  // frees the stage once these MMAs have read it
                        }
                        TSB_CYC_ADD(cyc_issue);
                        accumulate = 1u;
                        w16 += (uint32_t)G * kWgt16;
                        st16 += stage16;
                        if (++stage == stage_lo + ring) { stage = stage_lo; phase ^= 1u; st16 = base16 + (uint32_t)stage_lo * stage16; }
                    }
                }
                TSB_CYC_START;
                if (ok && elect_one()) tc_commit(bar_tfull + 8 * acc);  // accumulator complete
                TSB_CYC_ADD(cyc_commit);
                if (ok && resident && issuers == 1) {
                    int nm = 0, nn = -1;
                    if (local + 1 < my_tiles) decode(local + 1, nm, nn);
                    if (nn != cur_n && elect_one()) tc_commit(bar_bfree);  // the resident weights may be replaced
                }
                if (me == 0) TSB_TRACE(local, 4);
            }
            // ... and so is the last one
            while (shared_ring && issuers > 1 && ok && rows_next <= rows_last) {
                ok = rows_wait();
                if (ok) rows_pass();
            }
            if (me == 0) TSB_CYC_REPORT((my_tiles + issuers - 1) / issuers);
        }
    } else if (is_staged(EPI) && warp >= kCopyWarp0) {
        // ------------------------------------------------------------------ staged epilogue: copies
        // One thread per quad moves the quad's tiles, so that the arithmetic warps neither issue copies nor wait for them.  A tile
        // is loaded (residual), worked on and stored; with two tiles per quad the store of one chunk and the load of the next
        // but one run under the arithmetic of the chunk between them.  What is left is what the copies themselves cost: tensor-map
        // copies alone (a box in, a box out, 412 MB) run at 5.3-5.5 TB/s here, 64 -> 256 channels at 56 x 56 with a residual (474 MB,
        // 64 images) at 4.8.  (With the quad's first warp issuing the copies and one
        // tile, a chunk of 128 pixels x 32 channels took 7700 cycles, of which the arithmetic was 1900, waiting for the residual
        // 1260, issuing copies 550, waiting until a store had read the tile 700, barriers and the rest 1200.)
        if (lane == 0) {
            const int quad = warp - kCopyWarp0, parts = kQuads / groups, group = quad / parts, part = quad % parts;
            const int tiles = kp.stg_tiles;
            const bool has_res = epi.residual != nullptr, has_f32 = epi.out_f32 != nullptr, has_i8 = epi.out_i8 != nullptr;
            const uint32_t f_tile = base + kp.stg_off + (uint32_t)(quad * tiles) * kStageF32Bytes;
            const uint32_t q_tile = base + kp.stg_off + (uint32_t)(kQuads * tiles) * kStageF32Bytes + (uint32_t)quad * kStageI8Bytes;
            const uint32_t ready = bar_stg + 8 * (quad * 2), full = bar_stg + 8 * (2 * kQuads + quad * 2), q_free = bar_stg + 8 * (4 * kQuads + quad);
            if (has_res) prefetch_tensormap(&map_r);
            if (has_f32) prefetch_tensormap(&map_of);
            if (has_i8) prefetch_tensormap(&map_oi);
            // a walk over the quad's chunks: tile coordinates (innermost: the channel) and the position in the channel tile
            struct Walk { int local, c, nchunks, o_base, c1, c2, c3; };
            auto enter = [&](Walk &w) {            // at the first chunk of tile w.local
                if (w.local >= my_tiles) return;
                int m_tile, n_tile;
                decode(w.local, m_tile, n_tile);
                w.o_base = n_tile * CH;
                const int ch_end = min(w.o_base + BN, max(epi.O, has_i8 ? epi.out_cp : 0));
                w.nchunks = ch_end > w.o_base ? (ch_end - w.o_base + 31) >> 5 : 0;
                w.c = part;
                if (SPLIT && part != rank) w.nchunks = 0;                       // another CTA of the cluster finishes this chunk
                w.c1 = m_tile * PIX; w.c2 = 0; w.c3 = 0;                          // general: [pixel][channel]
                if (MODE == kModeRows) {                                        // [image row][ow][channel]
                    const int row_id = kp.d_segs.div(m_tile);
                    w.c1 = (m_tile - row_id * kp.rows_segs) * PIX; w.c2 = row_id;
                }
                if (MODE == kModePatch) {                                       // [image][oh][ow][channel]
                    const int p_img = kp.d_tiles_hw.div(m_tile), p_rem = m_tile - p_img * kp.patch_tiles_hw;
                    const int p_r = kp.d_tiles_w.div(p_rem), p_c = p_rem - p_r * kp.patch_tiles_w;
                    w.c1 = p_c * 8; w.c2 = p_r * (PIX / 8); w.c3 = p_img;
                }
            };
            auto settle = [&](Walk &w) {           // skip tiles in which this quad has no chunk (left)
                while (w.local < my_tiles && w.c >= w.nchunks) { w.local += groups; enter(w); }
            };
            // makes tile t ready for the chunk at w and moves w on
            auto load = [&](Walk &w, int t) {
                if (w.local >= my_tiles) return;
                const int ch = w.o_base + w.c * 32;
                const uint32_t bar = ready + 8 * t;
                if (has_res && ch < epi.O) {
                    const uint32_t dst = f_tile + (uint32_t)t * kStageF32Bytes;
                    mbar_arrive_expect_tx(bar, kStageF32Bytes);
                    if (MODE == kModePatch) tma_load_4d(dst, &map_r, bar, ch, w.c1, w.c2, w.c3);
                    else if (MODE == kModeRows) tma_load_3d(dst, &map_r, bar, ch, w.c1, w.c2);
                    else tma_load_2d(dst, &map_r, bar, ch, w.c1);
                } else {
                    mbar_arrive(bar);
                }
                w.c += parts;
                settle(w);
            };
            auto store = [&](const CUtensorMap *map, uint32_t src, const Walk &w, int ch) {
                if (MODE == kModePatch) tma_store_4d(map, src, ch, w.c1, w.c2, w.c3);
                else if (MODE == kModeRows) tma_store_3d(map, src, ch, w.c1, w.c2);
                else tma_store_2d(map, src, ch, w.c1);
            };
            Walk in, out;
            in.local = group; in.c = in.nchunks = in.o_base = in.c1 = in.c2 = in.c3 = 0;
            enter(in);
            settle(in);
            out = in;
            for (int t = 0; t < tiles; ++t) load(in, t);
            for (int i = 0; out.local < my_tiles; ++i) {
                const int t = i & (tiles - 1);
                if (!mbar_wait(full + 8 * t, (uint32_t)(tiles == 2 ? i >> 1 : i) & 1u, abort_flag)) {
                    if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 8); }
                    break;
                }
                const int ch = out.o_base + out.c * 32;
                if (has_f32 && ch < epi.O) store(&map_of, f_tile + (uint32_t)t * kStageF32Bytes, out, ch);
                if (has_i8) store(&map_oi, q_tile, out, ch);
                bulk_commit();
                bulk_wait_read();                                    // the tiles may be overwritten
                if (has_i8) mbar_arrive(q_free);
                load(in, t);
                out.c += parts;
                settle(out);
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (sixteen warps)
        // A warp may read only the 32 tensor-memory lanes of its quarter (warp id mod 4); four warps share a
        // quarter and split the tile's columns between them in chunks of 32.
        // The sixteen warps form groups (of four, eight or all sixteen warps); group g takes the tiles local = g, g + groups, ...
        // One tile's epilogue is a chain of latencies (barrier, tensor-memory
        // load, arithmetic, stores); with the groups on different tiles those chains overlap.
        const int group_warps = 16 / groups;                       // 4, 8 or 16
        const int group_threads = 32 * group_warps;
        const int parts = group_warps / 4;                       // warps of a group per lane quarter: 1, 2 or 4
        const int quarter = warp & 3;
        const int group = (warp - kEpiWarp0) / group_warps;
        const int part = ((warp - kEpiWarp0) % group_warps) >> 2;        // 0 .. parts-1
        const int et = (int)threadIdx.x - 32 * kEpiWarp0 - group * group_threads;   // thread index inside the group
        const int row = quarter * 32 + lane;     // tensor-memory lane this thread reads
        constexpr int kChunks = BN / 32;
        constexpr int CW = 32;                   // normal orientation: columns a warp takes per step
        const int act = epi.activation;
        int stg_count = 0;                       // staged epilogue: chunks this quad has worked through
        int table_n = -1;                        // channel tile this group's scale / bias table holds
        for (int local = group; local < my_tiles; local += groups) {
            const int acc = local & (nbuf - 1);
            const uint32_t acc_phase = (uint32_t)(local / nbuf) & 1u;
            int m_tile, n_tile;
            decode(local, m_tile, n_tile);
            const int o_base = n_tile * CH;
            const int slot = DUAL ? 2 * acc : acc;          // first accumulator buffer of this tile
            // ... and those of the other CTAs, to which partial sums will go.  (A barrier without a bound: the CTAs of a cluster start together and
            // arrive before any other wait than that for tensor memory, which a kernel before this one gives back when it ends.)
            if constexpr (SPLIT) cluster_wait();
            float *t_dq = table + (DUAL ? 2 * group : group) * 2 * BN, *t_bias = t_dq + BN;
            if (!SWAP && n_tile != table_n) {
                // this group's table of per-channel scales and biases: rebuilt only when the channel tile changes (never, for
                // layers of at most BN channels), between two barriers of the group
                if (table_n >= 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(group_threads) : "memory");
                for (int j = et; j < BN; j += group_threads) {
                    const int o = o_base + j;
                    t_dq[j] = o < epi.O ? epi.dq[o] : 0.0f;
                    t_bias[j] = (o < epi.O && epi.bias) ? epi.bias[o] : 0.0f;
                    if constexpr (DUAL) {                   // the projection's table: the next slot
                        t_dq[2 * BN + j] = (o < epi.O && dual.dq2) ? dual.dq2[o] : 0.0f;
                        t_dq[3 * BN + j] = (o < epi.O && dual.bias2) ? dual.bias2[o] : 0.0f;
                    }
                }
                asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(group_threads) : "memory");
                table_n = n_tile;
            }
            // every warp waits for the accumulator on its own; one that gives up raises the CTA's abort flag, which ends
            // the other warps' waits as well
            if (!mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag)) {
                if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 4); }
                break;
            }
            tc_fence_after();
            if (et == 0 && local < 32) TSB_TRACE(local, 5);
#ifdef TSB_ENABLE_TRACE
            // profiling experiment: with trace[255] set, the epilogue warps hand the accumulator back without touching it
            // (outputs are then garbage) -- shows how fast the other two roles run when left alone
            if (kp.trace && kp.trace[255] != 0) { tc_fence_before(); mbar_arrive(bar_tempty + 8 * acc); continue; }
#endif
            const uint32_t taddr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(slot * BN);
            if constexpr (SPLIT) {
                // The sixteen warps hold one tile: part = chunk = the CTA that finishes it.  A warp whose chunk another CTA finishes sends
                // its 32 x 32 partial sums there, into the slot of this CTA (16-byte pieces of consecutive rows side by side), and
                // is done; the warps of this CTA's chunk add the three slots to their own accumulators, in tensor memory, and go on.
                // (Slot i lies in the fp32 tile of quad i, which the staged epilogue does not use here unless i is this CTA.)
                int v[32];
                tmem_ld32(taddr0 + (uint32_t)(part * 32), v);
                tmem_ld_wait();
                const uint32_t slots = base + kp.stg_off + (uint32_t)row * 16u;
                if (part != rank) {
                    const uint32_t to = map_to_rank(slots + (uint32_t)rank * kStageF32Bytes, (uint32_t)part);
#pragma unroll
                    for (int j = 0; j < 8; ++j) sts128_cluster(to + (uint32_t)j * (kBM * 16), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(map_to_rank(bar_parts, (uint32_t)part));
                    continue;
                }
                if (!__all_sync(0xffffffffu, mbar_wait_cluster(bar_parts, 0u, abort_flag))) {
                    if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 9); }
                    break;
                }
                for (int q = 0; q < kSplit; ++q) {
                    if (q == rank) continue;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int4 a = *reinterpret_cast<const int4 *>(base_ptr + kp.stg_off + (uint32_t)q * kStageF32Bytes + (uint32_t)(j * kBM + row) * 16u);
                        v[4 * j] += a.x; v[4 * j + 1] += a.y; v[4 * j + 2] += a.z; v[4 * j + 3] += a.w;
                    }
                }
                tmem_st32(taddr0 + (uint32_t)(part * 32), v);
            }
            if constexpr (!SWAP) {
                int m = m_tile * PIX + row;
                bool live = m < kp.M_total;
                if (MODE == kModeRows) {
                    const int row_id = kp.d_segs.div(m_tile), ow = (m_tile - row_id * kp.rows_segs) * PIX + row;
                    live = ow < kp.OW;
                    m = row_id * kp.OW + ow;
                }
                if (MODE == kModePatch) {
                    const int p_img = kp.d_tiles_hw.div(m_tile), p_rem = m_tile - p_img * kp.patch_tiles_hw;
                    const int p_r = kp.d_tiles_w.div(p_rem), p_c = p_rem - p_r * kp.patch_tiles_w;
                    const int oh = p_r * (PIX / 8) + (row >> 3), ow = p_c * 8 + (row & 7);
                    live = oh < kp.OH && ow < kp.OW;
                    m = p_img * kp.P + oh * kp.OW + ow;
                }
                const int img = live ? kp.d_P.div(m) : 0;
                const int p = live ? m - img * kp.P : 0;
                if constexpr (is_staged(EPI)) {
                    // ---- staged epilogue, the arithmetic: residual tile -> result tiles, all in shared memory.
                    // A quad (the four warps of this group that share `part`, one per lane quarter = the tile's 128
                    // pixels) works through its 32-channel chunks; its copy warp brings the residual tiles and carries the
                    // result tiles off (below).  The warps of a quad do not wait for each other.
                    const int quad = group * parts + part;
                    const uint32_t q_row = base + kp.stg_off + (uint32_t)(kQuads * kp.stg_tiles) * kStageF32Bytes + (uint32_t)quad * kStageI8Bytes + (uint32_t)row * 32u;
                    const bool has_res = epi.residual != nullptr, has_i8 = epi.out_i8 != nullptr;
                    // channels this tile has to cover: the real ones, and for an int8 output its zero padding as well
                    const int ch_end = min(o_base + BN, max(epi.O, has_i8 ? epi.out_cp : 0));
                    const int nchunks = ch_end > o_base ? (ch_end - o_base + 31) >> 5 : 0;
                    const float rs = epi.nscales == 1 ? epi.rq_scales[0] : epi.rq_scales[min(img, epi.nscales - 1)];
                    bool stg_ok = true;
#pragma unroll 1
                    for (int c = part; c < nchunks; c += parts, ++stg_count) {
                        const int col0 = c * 32;
                        const bool real = o_base + col0 < epi.O;      // false: nothing but the int8 output's channel padding
                        const int t = stg_count & (kp.stg_tiles - 1);
                        const uint32_t r_row = base + kp.stg_off + (uint32_t)(quad * kp.stg_tiles + t) * kStageF32Bytes + (uint32_t)row * 128u + (uint32_t)(row & 7) * 16u;
                        const uint32_t tile_phase = (uint32_t)(kp.stg_tiles == 2 ? stg_count >> 1 : stg_count) & 1u;
                        int v[32];
                        if (real) tmem_ld32(taddr0 + (uint32_t)(DUAL && !concat ? BN + col0 : col0), v);
                        // the tile is free, and holds the residual if there is one
                        stg_ok = __all_sync(0xffffffffu, mbar_wait(bar_stg + 8 * (quad * 2 + t), tile_phase, abort_flag));
                        if (!stg_ok) { tmem_ld_wait(); break; }
                        if constexpr (DUAL) {
                            // the projection's 32 channels of this pixel, dequantized (+ bias), into the thread's own row of
                            // the fp32 tile -- where a tensor-map load would have put a residual
                            if (real && !concat) {
                                tmem_ld_wait();
#pragma unroll
                                for (int j4 = 0; j4 < 8; ++j4) {
                                    const float4 d4 = *reinterpret_cast<const float4 *>(t_dq + 2 * BN + col0 + 4 * j4);
                                    const float4 b4 = *reinterpret_cast<const float4 *>(t_dq + 3 * BN + col0 + 4 * j4);
                                    float4 f;
                                    f.x = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + 0]), d4.x), b4.x);
                                    f.y = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + 1]), d4.y), b4.y);
                                    f.z = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + 2]), d4.z), b4.z);
                                    f.w = __fadd_rn(__fmul_rn(__int2float_rn(v[4 * j4 + 3]), d4.w), b4.w);
                                    sts128(r_row ^ (uint32_t)(j4 * 16), f);
                                }
                                tmem_ld32(taddr0 + (uint32_t)col0, v);
                            }
                        }
                        uint32_t q[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
                        bool fine = true;
                        if (real) {
                            tmem_ld_wait();
                            with_act_flag(act, epi.even, [&](auto a, auto even) {
                                fine = staged_chunk_t<TSB_VAL(a), TSB_VAL(even), EPI == kEpiStagedAfter>(v, t_dq + col0, t_bias + col0, epi.leaky, r_row, has_res || (DUAL && !concat), has_i8, rs, q);
                            });
                        }
                        if (has_i8) {
                            // the previous chunk's int8 tile has been read
                            stg_ok = __all_sync(0xffffffffu, mbar_wait(bar_stg + 8 * (4 * kQuads + quad), (uint32_t)(stg_count + 1) & 1u, abort_flag));
                            if (!stg_ok) break;
                            sts128(q_row, q[0], q[1], q[2], q[3]);
                            sts128(q_row + 16, q[4], q[5], q[6], q[7]);
                            const uint32_t nchw0 = (uint32_t)(img * epi.O + o_base + col0) * (uint32_t)epi.P + (uint32_t)p;
                            if (real && live && (!fine || (epi.tail && nchw0 + 31u * (uint32_t)epi.P >= epi.rne_limit))) {
                                // NaN or a value beyond the int32 range (they quantize to -128 in the reference), or an
                                // element of the tensor's tail, which rounds the other way: exactly, from the fp32 results
                                for (int j = 0; j < 32 && o_base + col0 + j < epi.O; ++j) {
                                    float f;
                                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"((r_row ^ (uint32_t)((j >> 2) * 16)) + (uint32_t)(j & 3) * 4u) : "memory");
                                    const int b = q8(f, rs, epi.even && nchw0 + (uint32_t)j * (uint32_t)epi.P < epi.rne_limit);
                                    asm volatile("st.shared.u8 [%0], %1;" ::"r"(q_row + (uint32_t)j), "r"(b) : "memory");
                                }
                            }
                        }
                        fence_async_smem();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_stg + 8 * (2 * kQuads + quad * 2 + t));     // this warp's rows are written
                    }
                    if (!stg_ok) {
                        if (!*abort_flag) { *abort_flag = 1; atomicExch(kp.status, 7); }
                        break;
                    }
                } else {
#pragma unroll 1
                for (int c = part; c < BN / CW; c += parts) {
                    const int col0 = c * CW;
                    if (o_base + col0 >= epi.O) {
                        // nothing but channel padding in this step: no accumulators to read, only the zero bytes the
                        // NHWC_PAD layout wants in its padding channels
                        if (live && epi.out_i8 && epi.i8_nhwc) {
#pragma unroll
                            for (int u = 0; u < CW; u += 16)
                                if (o_base + col0 + u < epi.out_cp)
                                    *reinterpret_cast<int4 *>(epi.out_i8 + (size_t)m * epi.out_cp + o_base + col0 + u) = make_int4(0, 0, 0, 0);
                        }
                        continue;
                    }
                    const int channels = min(CW, epi.O - (o_base + col0));
                    bool done = false;
                    if constexpr (EPI != kEpiGeneric) {
                        int v[CW];
                        tmem_ldw(taddr0 + (uint32_t)col0, v);
                        tmem_ld_wait();
                        if constexpr (EPI == kEpiF32Nchw) {
                            if (live) {
                                const size_t off = (size_t)(img * epi.O + o_base + col0) * (size_t)epi.P + (size_t)p;
                                float *dst = epi.out_f32 + off;
                                if (epi.residual) with_act_flag(act, epi.res_after, [&](auto a, auto after) {
                                    store_f32_nchw_res_t<TSB_VAL(a), CW, TSB_VAL(after)>(v, t_dq + col0, t_bias + col0, epi.leaky, epi.residual + off, dst, (uint32_t)epi.P, channels);
                                });
                                else with_act(act, [&](auto a) {
                                    store_f32_nchw_t<TSB_VAL(a), CW>(v, t_dq + col0, t_bias + col0, epi.leaky, dst, (uint32_t)epi.P, channels);
                                });
                            }
                            done = true;
                        } else if constexpr (EPI == kEpiNhwc) {
                            const float rs = epi.nscales == 1 ? epi.rq_scales[0] : epi.rq_scales[min(img, epi.nscales - 1)];
                            const size_t f_off = (size_t)m * epi.O + o_base + col0;
                            const float *res = epi.residual ? epi.residual + f_off : nullptr;
                            float *of = epi.out_f32 ? epi.out_f32 + f_off : nullptr;
                            int8_t *oi = epi.out_i8 ? epi.out_i8 + (size_t)m * epi.out_cp + o_base + col0 : nullptr;
                            bool fine = true;
                            if (live) with_act_flags(act, epi.even, epi.res_after, [&](auto a, auto even, auto after) {
                                fine = store_nhwc_t<TSB_VAL(a), TSB_VAL(even), TSB_VAL(after)>(v, t_dq + col0, t_bias + col0, epi.leaky, res, of, oi, rs, channels,
                                                                                              epi.out_cp - (o_base + col0));
                            });
                            done = !__any_sync(0xffffffffu, !fine);
                        } else {
                            const float rs = epi.nscales == 1 ? epi.rq_scales[0] : epi.rq_scales[img];
                            int8_t *dst = epi.out_i8 + (size_t)m * epi.out_cp + o_base + col0;
                            bool fine = true;
                            if (live) with_act_flag(act, epi.even, [&](auto a, auto even) {
                                fine = store_i8_nhwc_t<TSB_VAL(a), TSB_VAL(even), CW>(v, t_dq + col0, t_bias + col0, epi.leaky, rs, dst, epi.out_cp - (o_base + col0));
                            });
                            done = !__any_sync(0xffffffffu, !fine);
                        }
                        if (EPI != kEpiF32Nchw && epi.tail && done &&
                            __any_sync(0xffffffffu, live && ((uint32_t)(img * epi.O + o_base + col0 + channels - 1) * (uint32_t)epi.P + (uint32_t)p) >= epi.rne_limit))
                            fix_tail(epi, taddr0 + (uint32_t)col0, [&](int j) { return live && j < channels; }, [&](int) { return img; },
                                     [&](int j) { return o_base + col0 + j; }, [&](int) { return p; });
                    }
                    if (!done) {
                        // element by element: any combination of outputs, residual, partial channel chunks
                        for (int j = 0; j < CW; ++j) {
                            const int a = tmem_ld1(taddr0 + (uint32_t)(col0 + j));
                            const int o = o_base + col0 + j;
                            if (!live) continue;
                            if (o < epi.O) epilogue_store_one(epi, img, o, p, a);
                            else if (epi.out_i8 && epi.i8_nhwc && o < epi.out_cp) epi.out_i8[(size_t)m * epi.out_cp + o] = 0;
                        }
                    }
                }
                }   // not staged
            } else {
                // this thread's channel; its scale and bias live in registers
                const int o = o_base + row;
                const bool ch_live = o < epi.O;
                const bool quarter_live = o_base + quarter * 32 < max(epi.O, epi.out_i8 && epi.i8_nhwc ? epi.out_cp : 0);
                const float my_dq = ch_live ? epi.dq[o] : 0.0f;
                const float my_bias = (ch_live && epi.bias) ? epi.bias[o] : 0.0f;
                int p_img = 0, p_r = 0, p_c = 0;
                if (MODE == kModePatch) {
                    p_img = kp.d_tiles_hw.div(m_tile);
                    const int p_rem = m_tile - p_img * kp.patch_tiles_hw;
                    p_r = kp.d_tiles_w.div(p_rem);
                    p_c = p_rem - p_r * kp.patch_tiles_w;
                }
                // residual boxes of this thread quad ({128 channels, 32 pixels} each), two chunks ahead of their use
                const bool prefetcher = EPI == kEpiNhwc && kp.res_prefetch && MODE != kModePatch && quarter == 0 && lane == 0;
                if (prefetcher) {
                    if (m_tile * PIX + part * 32 < kp.M_total) tma_prefetch_l2_2d(&map_r, o_base, m_tile * PIX + part * 32);
                    if (part + parts < kChunks && m_tile * PIX + (part + parts) * 32 < kp.M_total) tma_prefetch_l2_2d(&map_r, o_base, m_tile * PIX + (part + parts) * 32);
                }
#pragma unroll 1
                for (int c = part; c < kChunks && quarter_live; c += parts) {
                    const int col0 = c * 32;
                    if (prefetcher && c + 2 * parts < kChunks && m_tile * PIX + (c + 2 * parts) * 32 < kp.M_total)
                        tma_prefetch_l2_2d(&map_r, o_base, m_tile * PIX + (c + 2 * parts) * 32);
                    if (MODE == kModePatch) {
                        // this chunk: tile rows col0/8 .. col0/8+3, 8 pixels each
                        const int oh0 = p_r * (PIX / 8) + (col0 >> 3), ow0 = p_c * 8;
                        if (oh0 >= kp.OH) break;                         // uniform over the warp; later chunks lie lower still
                        const int rows_live = min(4, kp.OH - oh0), cols_live = min(8, kp.OW - ow0);
                        const int p0 = oh0 * kp.OW + ow0;
                        bool done = false;
                        if constexpr (EPI == kEpiF32Nchw || EPI == kEpiI8Nhwc) {
                            int v[32];
                            tmem_ld32(taddr0 + (uint32_t)col0, v);
                            tmem_ld_wait();
                            if constexpr (EPI == kEpiF32Nchw) {
                                if (ch_live) {
                                    float *dst = epi.out_f32 + ((size_t)(p_img * epi.O + o) * (size_t)epi.P + (size_t)p0);
                                    with_act(act, [&](auto a) { patch_f32_run<TSB_VAL(a)>(v, my_dq, my_bias, epi.leaky, dst, (uint32_t)kp.OW, rows_live, cols_live); });
                                }
                                done = true;
                            } else {
                                const float rs = epi.nscales == 1 ? epi.rq_scales[0] : epi.rq_scales[p_img];
                                int8_t *dst = epi.out_i8 + ((size_t)p_img * epi.P + p0) * epi.out_cp + o;
                                with_act_flag(act, epi.even, [&](auto a, auto even) {
                                    done = patch_i8_run<TSB_VAL(a), TSB_VAL(even)>(v, my_dq, my_bias, epi.leaky, rs, o < epi.out_cp, dst, (uint32_t)epi.out_cp,
                                                                                   (uint32_t)(kp.OW * epi.out_cp), rows_live, cols_live);
                                });
                                const int p_top = p0 + (rows_live - 1) * kp.OW + cols_live - 1;
                                if (epi.tail && done && __any_sync(0xffffffffu, ch_live && ((uint32_t)(p_img * epi.O + o) * (uint32_t)epi.P + (uint32_t)p_top) >= epi.rne_limit))
                                    fix_tail(epi, taddr0 + (uint32_t)col0, [&](int j) { return ch_live && (j >> 3) < rows_live && (j & 7) < cols_live; },
                                             [&](int) { return p_img; }, [&](int) { return o; }, [&](int j) { return p0 + (j >> 3) * kp.OW + (j & 7); });
                            }
                        }
                        if (!done) {
                            for (int j = 0; j < 32; ++j) {
                                if ((j >> 3) >= rows_live || (j & 7) >= cols_live) continue;   // uniform over the warp
                                const int a = tmem_ld1(taddr0 + (uint32_t)(col0 + j));
                                const int pj = p0 + (j >> 3) * kp.OW + (j & 7);
                                if (ch_live) epilogue_store_one(epi, p_img, o, pj, a);
                                else if (epi.out_i8 && epi.i8_nhwc && o < epi.out_cp)
                                    epi.out_i8[((size_t)p_img * epi.P + pj) * epi.out_cp + o] = 0;
                            }
                        }
                        continue;
                    }
                    const int mfirst = m_tile * PIX + col0;              // first pixel of this chunk
                    if (mfirst >= kp.M_total) break;                     // uniform over the warp
                    const int npix = min(32, kp.M_total - mfirst);
                    const int img0 = kp.d_P.div(mfirst), p0 = mfirst - img0 * kp.P;
                    const int split = kp.P - p0;                           // pixels j >= split belong to the next image
                    const bool one_image = npix == 32 && split >= 32;
                    // pixel-major outputs are linear in the pixel index: an image boundary inside the chunk only switches
                    // the requantize scale (at most once when an image has at least 32 pixels)
                    const bool linear_ok = (npix == 32 || EPI != kEpiNhwc) && kp.P >= 32;
                    bool done = false;
                    if (EPI != kEpiGeneric && (linear_ok || one_image)) {
                        int v[32];
                        tmem_ld32(taddr0 + (uint32_t)col0, v);
                        tmem_ld_wait();
                        const float rs0 = epi.nscales == 1 ? epi.rq_scales[0] : epi.rq_scales[img0];
                        const float rs1 = epi.nscales == 1 ? rs0 : epi.rq_scales[min(img0 + 1, epi.nscales - 1)];
                        if constexpr (EPI == kEpiF32Nchw) {
                            if (ch_live) {
                                float *dst = epi.out_f32 + ((size_t)(img0 * epi.O + o) * (size_t)epi.P + (size_t)p0);
                                if (one_image) with_act(act, [&](auto a) { swap_f32_run<TSB_VAL(a)>(v, my_dq, my_bias, epi.leaky, dst); });
                                else with_act(act, [&](auto a) { swap_f32_split_run<TSB_VAL(a)>(v, my_dq, my_bias, epi.leaky, dst, npix, split, (uint32_t)((epi.O - 1) * epi.P)); });
                            }
                            done = true;
                        } else if constexpr (EPI == kEpiI8Nhwc) {
                            int8_t *dst = epi.out_i8 + (size_t)mfirst * epi.out_cp + o;
                            with_act_flag(act, epi.even, [&](auto a, auto even) {
                                done = swap_i8_run<TSB_VAL(a), TSB_VAL(even)>(v, my_dq, my_bias, epi.leaky, rs0, rs1, split, o < epi.out_cp, dst, (uint32_t)epi.out_cp, npix);
                            });
                        } else if constexpr (EPI == kEpiNhwc) {
                            const size_t f_off = (size_t)mfirst * epi.O + (ch_live ? o : 0);
                            const float *res = epi.residual ? epi.residual + f_off : nullptr;
                            float *of = epi.out_f32 ? epi.out_f32 + f_off : nullptr;
                            int8_t *oi = epi.out_i8 ? epi.out_i8 + (size_t)mfirst * epi.out_cp + o : nullptr;
                            with_act_flags(act, epi.even, epi.res_after, [&](auto a, auto even, auto after) {
                                done = swap_nhwc_run<TSB_VAL(a), TSB_VAL(even), TSB_VAL(after)>(v, my_dq, my_bias, epi.leaky, res, of, oi, o < epi.out_cp, rs0, rs1, split,
                                                                                               (uint32_t)epi.O, (uint32_t)epi.out_cp, ch_live);
                            });
                        }
                        if (EPI != kEpiF32Nchw && epi.tail && done) {       // (one scale: the batch may still have several images)
                            auto img_of = [&](int j) { return kp.d_P.div(mfirst + j); };
                            const int last = kp.d_P.div(mfirst + npix - 1), p_last = mfirst + npix - 1 - last * kp.P;
                            if (__any_sync(0xffffffffu, ch_live && ((uint32_t)(last * epi.O + o) * (uint32_t)epi.P + (uint32_t)p_last) >= epi.rne_limit))
                                fix_tail(epi, taddr0 + (uint32_t)col0, [&](int j) { return ch_live && j < npix; }, img_of, [&](int) { return o; },
                                         [&](int j) { return mfirst + j - img_of(j) * kp.P; });
                        }
                    }
                    if (!done) {
                        int img = img0, p = p0;
                        for (int j = 0; j < npix; ++j) {
                            const int a = tmem_ld1(taddr0 + (uint32_t)(col0 + j));
                            if (ch_live) epilogue_store_one(epi, img, o, p, a);
                            else if (epi.out_i8 && epi.i8_nhwc && o < epi.out_cp)
                                epi.out_i8[(size_t)(img * epi.P + p) * epi.out_cp + o] = 0;
                            if (++p == kp.P) { p = 0; ++img; }
                        }
                    }
                }
            }
            tc_fence_before();
            mbar_arrive(bar_tempty + 8 * acc);
            if (et == 0) TSB_TRACE(local, 6);
        }
    }

    // common exit: everybody meets here, then the allocating warp releases tensor memory
    if (*abort_flag) {
        // give copies that may still be in flight time to land before shared memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) { __nanosleep(1000); }
    }
    tc_fence_before();
    __syncthreads();
    if constexpr (SPLIT) {
        // Nobody may write to, or arrive in, a CTA that has left.  One that has its partial sums gets no more of either; one that gave up
        // stays until the others have left or given up (threads that have exited count as arrived), which their own bounded waits see to.
        if (warp < kEpiWarp0 || warp >= kCopyWarp0) cluster_wait();     // (the epilogue warps have done so above)
        if (*abort_flag) { cluster_arrive(); cluster_wait(); }
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// Launches one instance.
template <int BN, int BK, bool SWAP, int MODE, int EPI, bool DUAL>
int launch(const Config &cfg, const CUtensorMap &ma, const CUtensorMap &mb, const CUtensorMap &mr, const CUtensorMap &mof,
           const CUtensorMap &moi, const KernelParams &kp, const EpiParams &epi, cudaStream_t stream,
           const std::conditional_t<DUAL, DualParams, NoDual> &dual) {
    // The shared-memory limit of a kernel is a per-device attribute: one process may drive several GPUs (one TenniS
    // Workbench per device, each on its own thread), so the "already raised" note is kept per device.
    static std::atomic<uint64_t> configured{0};
    auto kernel = conv_i8_tc_kernel<BN, BK, SWAP, MODE, EPI, DUAL>;
    int dev = 0;
    TSB_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        TSB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynamicSmem));
        configured.fetch_or(bit, std::memory_order_release);
    }
    TSB_CUDA(launch_pdl_cluster(MODE == kModeSplit ? kSplit : 1, kernel, dim3(cfg.grid), dim3(cta_threads(EPI)), cfg.dyn_smem, stream, ma, mb, mr, mof, moi,
                                kp, epi, dual));
    TSB_LAUNCHED("conv_i8_tc_kernel");
    return TSB_OK;
}

// The instances of the kernel, in groups that are compiled side by side (one object file of conv_tc_inst.cu per group).
// X(BN, BK, SWAP, MODE, EPI, DUAL)
#define TSB_TC_NORMAL(X, BN_, BK_, MODE_)                                                                                    \
    X(BN_, BK_, false, MODE_, kEpiGeneric, false) X(BN_, BK_, false, MODE_, kEpiF32Nchw, false)                             \
    X(BN_, BK_, false, MODE_, kEpiI8Nhwc, false) X(BN_, BK_, false, MODE_, kEpiStaged, false)                                 \
    X(BN_, BK_, false, MODE_, kEpiStagedAfter, false)
#define TSB_TC_SWAPPED(X, BN_, BK_)                                                                                          \
    X(BN_, BK_, true, kModeGeneral, kEpiGeneric, false) X(BN_, BK_, true, kModeGeneral, kEpiF32Nchw, false)                 \
    X(BN_, BK_, true, kModeGeneral, kEpiI8Nhwc, false) X(BN_, BK_, true, kModeGeneral, kEpiNhwc, false)                     \
    X(BN_, BK_, true, kModePatch, kEpiGeneric, false) X(BN_, BK_, true, kModePatch, kEpiF32Nchw, false)                     \
    X(BN_, BK_, true, kModePatch, kEpiI8Nhwc, false)
#define TSB_TC_PAIR(X, BN_, BK_)                                                                                             \
    X(BN_, BK_, false, kModeGeneral, kEpiStaged, true) X(BN_, BK_, false, kModeGeneral, kEpiStagedAfter, true) X(BN_, BK_, false, kModeGeneral, kEpiI8Nhwc, true)
#define TSB_TC_PART_0(X) TSB_TC_NORMAL(X, 64, 64, kModeGeneral) TSB_TC_NORMAL(X, 64, 128, kModeGeneral) TSB_TC_NORMAL(X, 64, 64, kModePatch)
#define TSB_TC_PART_1(X) TSB_TC_NORMAL(X, 128, 64, kModeGeneral) TSB_TC_NORMAL(X, 128, 128, kModeGeneral) TSB_TC_NORMAL(X, 64, 128, kModePatch)
#define TSB_TC_PART_2(X) TSB_TC_NORMAL(X, 256, 64, kModeGeneral) TSB_TC_NORMAL(X, 256, 128, kModeGeneral)
#define TSB_TC_PART_3(X) TSB_TC_NORMAL(X, 128, 64, kModePatch) TSB_TC_NORMAL(X, 128, 128, kModePatch)
#define TSB_TC_PART_4(X) TSB_TC_NORMAL(X, 256, 64, kModePatch) TSB_TC_NORMAL(X, 256, 128, kModePatch)
#define TSB_TC_ROWS(X, BN_, BK_) TSB_TC_NORMAL(X, BN_, BK_, kModeRows) X(BN_, BK_, false, kModeRows, kEpiNhwc, false)
#define TSB_TC_PART_5(X) TSB_TC_ROWS(X, 64, 64) TSB_TC_ROWS(X, 128, 64) TSB_TC_ROWS(X, 256, 64)
#define TSB_TC_PART_6(X) TSB_TC_ROWS(X, 64, 128) TSB_TC_ROWS(X, 128, 128) TSB_TC_ROWS(X, 256, 128)
#define TSB_TC_PART_7(X) TSB_TC_SWAPPED(X, 128, 64) TSB_TC_SWAPPED(X, 128, 128)
#define TSB_TC_PART_8(X) TSB_TC_SWAPPED(X, 256, 64) TSB_TC_SWAPPED(X, 256, 128)
#define TSB_TC_PART_9(X)                                                                                                     \
    TSB_TC_PAIR(X, 64, 64) TSB_TC_PAIR(X, 64, 128) TSB_TC_PAIR(X, 128, 64) TSB_TC_PAIR(X, 128, 128) TSB_TC_PAIR(X, 256, 64) TSB_TC_PAIR(X, 256, 128)
#define TSB_TC_PART_10(X) TSB_TC_NORMAL(X, 128, 64, kModeSplit) TSB_TC_NORMAL(X, 128, 128, kModeSplit)
#define TSB_TC_ALL(X)                                                                                                        \
    TSB_TC_PART_0(X) TSB_TC_PART_1(X) TSB_TC_PART_2(X) TSB_TC_PART_3(X) TSB_TC_PART_4(X) TSB_TC_PART_5(X) TSB_TC_PART_6(X)  \
    TSB_TC_PART_7(X) TSB_TC_PART_8(X) TSB_TC_PART_9(X) TSB_TC_PART_10(X)

}  // namespace tc
}  // namespace tsb
