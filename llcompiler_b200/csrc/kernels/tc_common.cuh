// PTX building blocks for the 5th-generation tensor-core kernels: mbarriers with bounded
// waits, TMA tiled loads, tensor-memory allocation, tcgen05.mma issue / commit / load.
//
// Every wait on an mbarrier is bounded: after kSpinLimit polls the waiter records a code in the
// status word (tcStatusWord) and carries on, so that a wrong byte count or a lost arrive can never
// hang the GPU; the result of that launch is then wrong and the host reports the status.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace llc {
namespace tc {

constexpr uint32_t kSpinLimit = 1u << 21;

__device__ __forceinline__ uint32_t smemAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count));
}
__device__ __forceinline__ void fenceBarrierInit() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbarExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbarArrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory");
}
// Returns false when the wait gave up.  `abortWord` is a CTA-wide flag in shared memory: the first
// wait that gives up sets it, and every other wait of the CTA then returns at its next check, so a
// CTA whose pipeline broke drains in milliseconds instead of timing out once per remaining tile.
__device__ __forceinline__ bool mbarWait(uint64_t* bar, uint32_t parity, volatile int* abortWord) {
  uint32_t addr = smemAddr(bar);
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && *abortWord) return false;
  }
  *abortWord = 1;
  return false;
}

// The same for a barrier that threads or MMAs of the other CTA of a pair arrive on: what they wrote before is visible after it.
__device__ __forceinline__ bool mbarWaitCluster(uint64_t* bar, uint32_t parity, volatile int* abortWord) {
  uint32_t addr = smemAddr(bar);
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && *abortWord) return false;
  }
  *abortWord = 1;
  return false;
}

// generic-proxy writes to shared memory -> visible to the async proxy (tensor core, TMA)
__device__ __forceinline__ void fenceProxyAsync() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- CTA pairs (clusters of two) ---------------------------------------------------------------
__device__ __forceinline__ uint32_t clusterCtaRank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// Barrier over every thread of the cluster, with release / acquire of what was written before it.
__device__ __forceinline__ void clusterSync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrives on the barrier at the same place in CTA 0 of the pair (its own CTA for CTA 0).  What the arrival hands over has
// its own fences (tcgen05.fence for accumulators, fence.proxy.async for operand tiles); a cluster-scope release on top
// would wait for every store of the thread (1600 cycles in the GEMM's epilogue).
__device__ __forceinline__ void mbarArriveLeader(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 a;\n\t"
      "mapa.shared::cluster.u32 a, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}"
      ::"r"(smemAddr(bar)) : "memory");
}
// The shared::cluster address of the same place in CTA 0 of the pair.
__device__ __forceinline__ uint32_t leaderAddr(const void* p) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smemAddr(p)));
  return a;
}
// Tiled / im2col loads into this CTA's shared memory whose bytes are counted by the barrier of CTA 0 of the pair.
__device__ __forceinline__ void tmaLoadPair4d(void* smemDst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smemAddr(smemDst)), "l"((uint64_t)map), "r"(leaderAddr(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tmaLoadPairIm2col4d(void* smemDst, const CUtensorMap* map, uint64_t* bar, int c, int w, int h, int n, uint16_t offW, uint16_t offH) {
  asm volatile(
      "cp.async.bulk.tensor.4d.im2col.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      ::"r"(smemAddr(smemDst)), "l"((uint64_t)map), "r"(leaderAddr(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"(offW), "h"(offH)
      : "memory");
}

__device__ __forceinline__ void tmaLoad4d(void* smemDst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smemAddr(smemDst)), "l"((uint64_t)map), "r"(smemAddr(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// Im2col-mode load of an NHWC activation tensor: `pixelsPerColumn` (tensor map) consecutive output positions starting at
// the input pixel (w, h) of image n, walked in w -> h -> n order inside the map's bounding box with its traversal
// strides; every pixel is displaced by the filter-tap offset (offW, offH); c is the first channel.  Pixels that fall
// outside the tensor are filled with zeros (padding).
__device__ __forceinline__ void tmaLoadIm2col4d(void* smemDst, const CUtensorMap* map, uint64_t* bar, int c, int w, int h, int n, uint16_t offW,
                                                uint16_t offH) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};"
      ::"r"(smemAddr(smemDst)), "l"((uint64_t)map), "r"(smemAddr(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"(offW), "h"(offH)
      : "memory");
}
// Tile store from shared memory (bulk-group completion).  Elements of the box that lie past the
// tensor's extents are not written, which is how M and N tails are clipped.
__device__ __forceinline__ void tmaStore4d(const CUtensorMap* map, const void* smemSrc, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"((uint64_t)map), "r"(smemAddr(smemSrc)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void bulkCommit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Waits until the bulk stores this thread committed have finished reading shared memory.
__device__ __forceinline__ void bulkWaitRead() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// Same, but lets the most recent store still read: with two staging slots used in turn, the slot about to be
// rewritten belongs to the store before the last one.
__device__ __forceinline__ void bulkWaitRead1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulkWaitRead3() { asm volatile("cp.async.bulk.wait_group.read 3;" ::: "memory"); }   // four slots
__device__ __forceinline__ void prefetchTensorMap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

// (x0, x1) = (x0, x1) * (s0, s1) + (b0, b1), two fp32 multiply-adds in one instruction.
__device__ __forceinline__ void fma2(float& x0, float& x1, float s0, float s1, float b0, float b1) {
  asm("{\n\t.reg .b64 x, s, b;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 s, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "fma.rn.f32x2 x, x, s, b;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+f"(x0), "+f"(x1) : "f"(s0), "f"(s1), "f"(b0), "f"(b1));
}
// geluTanhBf16 (common.cuh) of two values, the same operations on packed pairs.
__device__ __forceinline__ void geluTanhBf16x2(float& x0, float& x1) {
  float u0, u1, h0, h1;
  asm("{\n\t.reg .b64 x, u, a, b, h;\n\tmov.b64 x, {%4, %5};\n\tmov.b64 a, {%6, %6};\n\tmov.b64 b, {%7, %7};\n\tmov.b64 h, {%8, %8};\n\t"
      "mul.rn.f32x2 u, x, x;\n\tfma.rn.f32x2 u, u, a, b;\n\tmul.rn.f32x2 u, x, u;\n\tmul.rn.f32x2 h, x, h;\n\t"
      "mov.b64 {%0, %1}, u;\n\tmov.b64 {%2, %3}, h;\n\t}"
      : "=f"(u0), "=f"(u1), "=f"(h0), "=f"(h1) : "f"(x0), "f"(x1), "f"(0.0356774081f), "f"(0.7978845608f), "f"(0.5f));
  asm("tanh.approx.f32 %0, %1;" : "=f"(u0) : "f"(u0));
  asm("tanh.approx.f32 %0, %1;" : "=f"(u1) : "f"(u1));
  fma2(h0, h1, u0, u1, h0, h1);
  x0 = h0; x1 = h1;
}

// ---- tensor memory ------------------------------------------------------------------------------
// Executed by one full warp.  `cols` is a power of two >= 32.
__device__ __forceinline__ void tmemAlloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemDealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// The same for both CTAs of a pair at once (executed by the same warp of each).
__device__ __forceinline__ void tmemAllocPair(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmemDeallocPair(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tcFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tcFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major operand tile stored as rows of 128 bytes with the
// 128-byte swizzle (what a TMA load with CU_TENSOR_MAP_SWIZZLE_128B writes): 8-row groups are
// 1024 bytes apart (stride byte offset), the leading byte offset is not used by this layout.
__device__ __forceinline__ uint64_t smemDescKMajorSw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);        // start address, 16-byte units
  d |= (uint64_t)1 << 16;                         // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;               // stride byte offset
  d |= (uint64_t)1 << 46;                         // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                         // layout: SWIZZLE_128B
  return d;
}
// MN-major operand tile: 64-element (128-byte) column slabs of K rows each, 8-row groups 1024 bytes
// apart (stride byte offset); consecutive slabs along N are `slabBytes` apart (leading byte offset).
__device__ __forceinline__ uint64_t smemDescMnMajorSw128(uint32_t saddr, uint32_t slabBytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((slabBytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor for kind::f16 / kind::tf32 with fp32 accumulation.
// fmt: 0 = f16, 1 = bf16, 2 = tf32.
__host__ __device__ constexpr uint32_t instrDesc(int fmt, int m, int n, int aMnMajor, int bMnMajor) {
  return (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)aMnMajor << 15) | ((uint32_t)bMnMajor << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

template <bool TF32>
__device__ __forceinline__ void mmaSS(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
  if (TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// One MMA over a CTA pair: M = 256, CTA r holds rows 128 r..+127 of A and of the accumulator and half r of the rows of B;
// issued by CTA 0 with descriptors that name the same places in both CTAs.
template <bool TF32>
__device__ __forceinline__ void mmaPairSS(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
  if (TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate) : "memory");
  }
}
// Arrives on the barriers at this place in both CTAs of the pair once every pair MMA issued so far has completed.
__device__ __forceinline__ void mmaCommitPair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smemAddr(bar)), "h"((uint16_t)3) : "memory");
}
// Arrives on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mmaCommit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smemAddr(bar)) : "memory");
}

// 32 lanes x 32 consecutive fp32 columns: thread i of the warp receives row (lane base + i).
__device__ __forceinline__ void tmemLoad32x32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
        "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// The same load split in two, so that the next chunk's load can be in flight while this chunk is worked on:
// tmemIssue32 starts it (the registers are not valid yet), tmemWait32 waits for every load issued so far and names the
// registers as read-write operands, which keeps the compiler from moving any use of them above the wait.
__device__ __forceinline__ void tmemIssue32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
        "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmemWait32(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]),
                 "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :: "memory");
}

// 32 lanes x N consecutive fp32 columns (N = 16 or 32).
template <int N> __device__ __forceinline__ void tmemLoadCols(uint32_t taddr, float* v);
template <> __device__ __forceinline__ void tmemLoadCols<32>(uint32_t taddr, float* v) { tmemLoad32x32(taddr, v); }
template <> __device__ __forceinline__ void tmemLoadCols<16>(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace tc
}  // namespace llc
