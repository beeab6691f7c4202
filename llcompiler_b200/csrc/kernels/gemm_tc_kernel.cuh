// Tensor-core GEMM and implicit-GEMM convolution for sm_100a: tcgen05.mma with accumulators in
// tensor memory, TMA-fed operands, persistent warp-specialised CTAs, fused epilogue.  Serves
// llc_cuda_gemm / llc_cuda_conv2d for bf16 operands and for fp32 operands at precision tf32 (one
// pass) or tf32x3 (three passes, fp32-grade accuracy).
//
// One CTA per SM loops over 128 x BN output tiles (BN = 64, 128 or 256).  Roles, by warp:
//   warp 0      TMA producer: per K block waits for a free stage, arms its mbarrier with the byte
//               count and issues the tile loads (B: BN rows x 128 bytes; dense GEMM also A: 128 rows
//               x 128 bytes; K-major, 128-byte swizzle; rows/columns past the edge are zero-filled
//               by TMA, which is how M, N and K tails are handled).
//   warp 1      MMA issuer: one lane waits for the stage, issues BK/UMMA_K tcgen05.mma (fp32
//               accumulation into one of two TMEM accumulators), commits the stage back to the
//               producer; after the last K block commits the accumulator to the epilogue.
//               Allocates and frees tensor memory.
//   warps 2-9   epilogue: tcgen05.ld (32 lanes x 32 columns per warp and step, the next step's load in
//               flight; a warp owns one lane quarter and one column half), alpha*scale[n]*acc + shift[n]
//               + res, activation, rows staged in one of two swizzled slots and written by TMA stores;
//               releases the accumulator as soon as it is in registers so that the next tile's MMAs
//               overlap the stores.
//   next 8      convolution only: im2col gather of the A tile (NHWC activations) with 16-byte
//               cp.async into the swizzled layout, zero-filling padding taps.
//   next 4      tf32x3 only: split each landed fp32 tile into its low-order part x - tf32(x)
//               (same swizzled position in a second buffer) and hand the stage to the issuer.
// CTA pairs (CG = 2, bf16 and tf32, BN = 256): two CTAs of a cluster work on a 256 x 256 tile.  Each loads its 128 rows of A
// and half of the rows of B (32 KB a stage instead of 48), CTA 0 issues cta_group::2 MMAs that read both CTAs' shared memory
// and leave each CTA its 128 rows of the accumulator, so that the epilogue is the single CTA's.
// tf32x3: acc = A_hi*B_hi + A_lo*B_hi + A_hi*B_lo.  The tensor core reads only the upper 19 bits
// of an fp32 operand, so A_hi is the raw tile and A_lo = A - truncate_to_tf32(A) is exact.
//
// Bound: tensor pipe.  Algorithmic FLOPs 2*M*N*K per batch entry; HBM bytes (M*K + N*K + M*N)
// elements; A is re-read once per column of tiles and B once per row of tiles (L2 hits).
// With K <= 768 the epilogue competes with the main loop: the tile walk without divisions, the column factors in shared
// memory, the packed GELU and the pair tiles together took (98304 rows, bf16, CUDA events) 2304 x 768 + bias 0.301 -> 0.250
// ms, 768 x 768 + residual 0.123 -> 0.103, 3072 x 768 + GELU 0.449 -> 0.368, 768 x 3072 + residual 0.371 -> 0.323.
#pragma once
#include "common.cuh"
#include "tc_common.cuh"

namespace llc {
namespace tcgemm {

using namespace tc;


constexpr int BM = 128;
constexpr int kTileKBytes = 128;          // one swizzle atom along K

struct TcArgs {
  int* status;              // non-zero after a bounded wait gave up: 1 producer, 2 issuer, 3 split, 4 epilogue, 5 gather
  void* out; const float* scale; const float* shift; const void* res;
  int out_dtype, res_dtype, act; float alpha;
  long long M, N, K;
  long long o_s0, o_s1, o_sm, r_s0, r_s1, r_sm, r_sn;
  int b1; int kBlocks; int vecOut;
  int resTile;              // the residual can be fetched as 32-row x 64-byte units with 16-byte loads
  int splits;               // K is cut into this many slices, each a CTA of its own; partial tiles meet in `ws`
  float* ws; int* counters; // workspace: parked partial tiles, and one arrival counter per tile (zero between launches)
  int accs, accBlocks;      // accumulators a unit's K loop is spread over, added up in the epilogue; bf16 / tf32: each sums this many K blocks in a row
  int hasBLo;               // tf32x3: the low-order part of B comes from memory (mapBLo) instead of the split warps
  int tmaOut;               // 0, or the bytes per row of the output box the epilogue stores through TMA (64)
  int aZ0, aZ1, bZ0, bZ1;   // 1: the operand has this batch dim, 0: it is broadcast (coordinate 0)
  int rZ0, rZ1;             // the same for the residual (RES kernels: it is loaded through a tensor map)
  int mTiles, nTiles; long long tiles;
  // convolution (A gathered from NHWC activations)
  const void* x; int H, W, C, KH, KW, OH, OW, sh, sw, ph, pw, dh, dw;
  long long xs_n, xs_h, xs_w;   // element strides of x along image, row and pixel (dense NHWC: H*W*C, W*C, C)
};

// RES: the epilogue adds a residual tile that TMA loads fetch ahead of time into a ring of four units per epilogue warp
// (the ring also stages the output); without it a warp has two output slots.
constexpr int kEpiWarps = 8;

template <int BN, int KIND, bool RES, int CG> struct Smem {
  static constexpr int kABytes = BM * kTileKBytes, kBBytes = BN / CG * kTileKBytes;   // a CTA pair splits the rows of B
  static constexpr int kStageBytes = (kABytes + kBBytes) * (KIND == 2 ? 2 : 1);
  static constexpr int kSlots = RES || CG == 2 ? 4 : 2;   // units of 32 rows x 64 bytes each epilogue warp owns
  static constexpr int kStagingPerWarp = kSlots * 2048;
  static constexpr int kStagingBytes = kEpiWarps * kStagingPerWarp;
  static constexpr int kStageBudget = 224 * 1024 - kStagingBytes;
  static constexpr int kStages = kStageBudget / kStageBytes > 8 ? 8 : kStageBudget / kStageBytes;
  static constexpr int kBarrierBytes = 1024;
  static constexpr int kVecBytes = 2048;    // per column half: alpha * scale[n] and shift[n] of the tile's columns
  static constexpr int kTotal = kStages * kStageBytes + kBarrierBytes + kStagingBytes + kVecBytes;
  static_assert(kTotal <= 227 * 1024, "shared memory of one CTA");
};

__device__ __forceinline__ void cpAsync16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;   // src-size 0: the 16 destination bytes are zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// The barrier receives one arrival (counted against its expected count) when every cp.async this
// thread has issued so far has landed: the thread itself never waits for its copies.
__device__ __forceinline__ void cpAsyncArriveOn(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smemAddr(bar)) : "memory");
}

// Where a work unit lies: K slice, column tile, row tile, batch.  A CTA (pair) takes every step-th unit; the position is
// carried along without a division (64-bit divisions per tile and role cost the epilogue 2000 of its 6500 cycles).
struct UnitWalk {
  int s, n, m, z1, z0, ds, dn, dm, d1, d0;
  __device__ __forceinline__ UnitWalk(const TcArgs& p, uint32_t first, uint32_t step) {
    const uint32_t sp = (uint32_t)p.splits, nt = (uint32_t)p.nTiles, mt = (uint32_t)p.mTiles, b1 = (uint32_t)p.b1;
    uint32_t q = first / sp; s = (int)(first - q * sp); first = q;
    q = first / nt; n = (int)(first - q * nt); first = q;
    q = first / mt; m = (int)(first - q * mt); first = q;
    q = first / b1; z1 = (int)(first - q * b1); z0 = (int)q;
    q = step / sp; ds = (int)(step - q * sp); step = q;
    q = step / nt; dn = (int)(step - q * nt); step = q;
    q = step / mt; dm = (int)(step - q * mt); step = q;
    q = step / b1; d1 = (int)(step - q * b1); d0 = (int)q;
  }
  __device__ __forceinline__ void next(const TcArgs& p) {
    s += ds; int c = s >= p.splits; s -= c ? p.splits : 0;
    n += dn + c; c = n >= p.nTiles; n -= c ? p.nTiles : 0;
    m += dm + c; c = m >= p.mTiles; m -= c ? p.mTiles : 0;
    z1 += d1 + c; c = z1 >= p.b1; z1 -= c ? p.b1 : 0;
    z0 += d0 + c;
  }
};

// KIND: 0 bf16, 1 tf32, 2 tf32x3.  BMN: B is stored [k][n] (unit stride along n) instead of [n][k].
// Threads of a CTA: producer, issuer, 8 epilogue warps, 8 gather warps (MODE 1), 4 split warps (tf32x3).
__host__ __device__ constexpr int tcThreads(int kind, int mode) { return (2 + kEpiWarps + (mode == 1 ? 8 : 0) + (kind == 2 ? 4 : 0)) * 32; }

// MODE: 0 dense GEMM (A by tiled TMA), 1 convolution with A gathered by warps (any channel count that keeps a
// 16-byte chunk inside one filter tap), 2 convolution with A loaded by TMA in im2col mode (a K block of 128
// bytes lies inside one filter tap: channels * element size is a multiple of 128).  (A variant with sixteen epilogue
// warps and one pipeline stage less was measured 1.2 to 1.9 times slower on every shape tried and is not kept.)
// CG: 1, a CTA works for itself on 128 x BN tiles; 2, a cluster of two CTAs works on 256 x BN tiles with cta_group::2 MMAs.
// CUT: calls of few tiles, one unit per CTA: K cut into slices that meet in the workspace, or sums spread over more accumulators
// than the set has, or both.  A variant of its own, because the code for it in the others' epilogue cost them 2 % (bottleneck
// block, 256 images 451 -> 459 us).
template <int BN, int KIND, int MODE, bool BMN, bool RES, int CG, bool CUT>
__global__ void __launch_bounds__(tcThreads(KIND, MODE), 1)
tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ CUtensorMap mapO,
          const __grid_constant__ CUtensorMap mapBLo, const __grid_constant__ CUtensorMap mapR, const TcArgs p) {
  constexpr bool X3 = KIND == 2;
  constexpr bool TF32 = KIND != 0;
  constexpr bool CONV = MODE == 1;      // the gather warps exist
  constexpr bool IM2COL = MODE == 2;
  constexpr bool PAIR = CG == 2;
  using S = Smem<BN, KIND, RES, CG>;
  static_assert(!PAIR || (MODE != 1 && !BMN && KIND != 2), "CTA pairs take TMA-fed K-major bf16 / tf32 operands");
  static_assert(!CUT || (MODE != 1 && !BMN && !RES && !PAIR), "one-CTA tiles of TMA-fed K-major operands can be cut along K");
  static_assert(!RES || (KIND != 2 && MODE != 1 && !BMN), "the residual ring exists for bf16 / tf32 kernels with TMA-fed operands");
  constexpr int kStages = S::kStages;
  constexpr int kElemBytes = TF32 ? 4 : 2;
  constexpr int BK = kTileKBytes / kElemBytes;          // 64 bf16 / 32 tf32
  constexpr int UMMA_K = 32 / kElemBytes;               // 16 bf16 / 8 tf32 (32 bytes of K per instruction)
  constexpr uint32_t kIdesc = instrDesc(TF32 ? 2 : 1, CG * BM, BN, 0, BMN ? 1 : 0);
  // Two accumulator sets (double buffering).  The tensor core truncates when it adds into its fp32 accumulator, so shorter
  // chains mean a smaller (K-proportional) rounding bias: tf32x3 spreads the K loop over kChains accumulators per set and
  // adds them in the epilogue; the CUT kernels spread it over p.accs of them (chooseTile says how many), past the first set,
  // which nothing else uses where a CTA has one unit.
  constexpr int kChains = X3 ? 256 / BN : 1;
  constexpr int kSetCols = X3 ? 256 : BN;
  const int accs = CUT ? p.accs : kChains;
  uint32_t accCols = 2 * kSetCols;                             // tensor memory to hold (twice as much cost 0.2 us a launch)
  if (CUT) while ((int)accCols < accs * BN) accCols *= 2;
  static_assert(!X3 || BN <= 128, "tf32x3 uses BN <= 128");
  constexpr int kAtomN = kTileKBytes / kElemBytes;      // BMN: elements of n per 128-byte slab row
  constexpr int kSlabBytes = BK * 128;                  // BMN: one slab = BK rows of k x 128 bytes of n
  constexpr int kGatherWarps = 8;
  constexpr int kGatherWarp0 = 2 + kEpiWarps, kSplitWarp0 = kGatherWarp0 + (CONV ? kGatherWarps : 0);
  constexpr int kFullCount = CONV ? kGatherWarps * 32 + 1 : 1;   // gather threads + the TMA arm

  extern __shared__ __align__(1024) uint8_t smem[];   // the swizzled tiles want 1024-byte boundaries
  uint8_t* tiles = smem;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * S::kStageBytes);
  uint64_t* full = bars;                    // [kStages] operands landed
  uint64_t* empty = bars + kStages;         // [kStages] MMAs that read the stage are done
  uint64_t* split = bars + 2 * kStages;     // [kStages] low-order tiles written (tf32x3)
  uint64_t* accFull = bars + 3 * kStages;   // [2] accumulator complete
  uint64_t* accEmpty = bars + 3 * kStages + 2;  // [2] accumulator drained by the epilogue
  uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bars + 3 * kStages + 4);
  volatile int* abortWord = reinterpret_cast<volatile int*>(tmemSlot + 1);
  volatile int* lastFlag = reinterpret_cast<volatile int*>(tmemSlot + 2);   // split-K: this CTA's slice arrived last
  uint64_t* resFull = bars + 32;                // [8 epilogue warps][4]: a unit of the residual has landed (RES)
  uint8_t* staging = smem + kStages * S::kStageBytes + S::kBarrierBytes;   // 1024-byte aligned
  constexpr int kStagingPerWarp = S::kStagingPerWarp;
  float* tileVec = reinterpret_cast<float*>(staging + S::kStagingBytes);   // [column half][alpha * scale, shift][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // The CTA (pair)'s share of the work, and the rows of a tile this CTA holds.  In a pair the barriers the issuer waits on
  // (full, accEmpty) are those of CTA 0, the issuer's; what the MMAs signal (empty, accFull) reaches both CTAs.
  const int rank = PAIR ? (int)clusterCtaRank() : 0;
  const uint32_t unit0 = blockIdx.x / CG, unitStep = gridDim.x / CG;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbarInit(&full[s], kFullCount); mbarInit(&empty[s], 1); mbarInit(&split[s], 4); }
    for (int a = 0; a < 2; ++a) { mbarInit(&accFull[a], 1); mbarInit(&accEmpty[a], kEpiWarps * CG); }
    if (RES) for (int i = 0; i < kEpiWarps * 4; ++i) mbarInit(&resFull[i], 1);
    *abortWord = 0;
    fenceBarrierInit();
  }
  if (warp == 1) { if constexpr (PAIR) tmemAllocPair(tmemSlot, accCols); else tmemAlloc(tmemSlot, accCols); }
  tcFenceBefore();
  if (PAIR) clusterSync(); else __syncthreads();
  tcFenceAfter();
  const uint32_t tmemBase = *tmemSlot;

  auto stageA = [&](int s) { return tiles + s * S::kStageBytes; };
  auto stageB = [&](int s) { return tiles + s * S::kStageBytes + S::kABytes; };
  auto stageALo = [&](int s) { return tiles + s * S::kStageBytes + S::kABytes + S::kBBytes; };
  auto stageBLo = [&](int s) { return tiles + s * S::kStageBytes + 2 * S::kABytes + S::kBBytes; };
  // Work units: (tile, K slice); fewer than 2^31 of them.  Without split-K a unit is a tile and its slice the whole K loop.
  const uint32_t units = (uint32_t)(p.tiles * p.splits);
  const int kPer = (p.kBlocks + p.splits - 1) / p.splits;
  auto kRange = [&](const UnitWalk& w, int& kb0, int& kb1) { kb0 = w.s * kPer; kb1 = kb0 + kPer < p.kBlocks ? kb0 + kPer : p.kBlocks; };

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      if (!CONV) prefetchTensorMap(&mapA);
      int ow0 = 0, oh0 = 0, img0 = 0;
      prefetchTensorMap(&mapB);
      uint32_t it = 0;
      bool ok = true;
      UnitWalk w(p, unit0, unitStep);
      for (uint32_t u = unit0; u < units && ok; u += unitStep, w.next(p)) {
        int kb0, kb1; kRange(w, kb0, kb1);
        const int tileM = w.m, tileN = w.n, zb0 = w.z0, zb1 = w.z1;
        int tapR = 0, tapS = 0, cc = 0;                      // im2col: filter tap and first channel of the K block
        if (IM2COL && kb0 > 0) { const long long k0 = (long long)kb0 * BK; const int tap = (int)(k0 / p.C); cc = (int)(k0 - (long long)tap * p.C); tapR = tap / p.KW; tapS = tap - tapR * p.KW; }
        if (IM2COL) {
          const uint32_t m0 = (uint32_t)(tileM * CG + rank) * BM;   // first output pixel of this CTA's rows (fewer than 2^31 pixels)
          const uint32_t t2 = m0 / (uint32_t)p.OW; ow0 = (int)(m0 - t2 * (uint32_t)p.OW);
          img0 = (int)(t2 / (uint32_t)p.OH); oh0 = (int)(t2 - (uint32_t)img0 * (uint32_t)p.OH);
        }
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % kStages; const uint32_t ph = (it / kStages) & 1;
          if (!mbarWait(&empty[s], ph ^ 1, abortWord)) { atomicExch(p.status, 1); ok = false; break; }
          if (rank == 0) mbarExpectTx(&full[s], ((CONV ? S::kBBytes : S::kABytes + S::kBBytes) + ((X3 && p.hasBLo) ? S::kBBytes : 0)) * CG);
          const int rowA = (tileM * CG + rank) * BM, rowB = tileN * BN + rank * (BN / CG);
          if (MODE == 0) {
            if constexpr (PAIR) tmaLoadPair4d(stageA(s), &mapA, &full[s], kb * BK, rowA, zb1 * p.aZ1, zb0 * p.aZ0);
            else tmaLoad4d(stageA(s), &mapA, &full[s], kb * BK, rowA, zb1 * p.aZ1, zb0 * p.aZ0);
          }
          if (IM2COL) {
            // 128 output pixels from (img0, oh0, ow0) on, in w -> h -> n order; the coordinates name the input pixel
            // under filter tap (0, 0), the offsets select the tap
            if constexpr (PAIR) tmaLoadPairIm2col4d(stageA(s), &mapA, &full[s], cc, ow0 * p.sw - p.pw, oh0 * p.sh - p.ph, img0, (uint16_t)(tapS * p.dw), (uint16_t)(tapR * p.dh));
            else tmaLoadIm2col4d(stageA(s), &mapA, &full[s], cc, ow0 * p.sw - p.pw, oh0 * p.sh - p.ph, img0, (uint16_t)(tapS * p.dw), (uint16_t)(tapR * p.dh));
            cc += BK;
            if (cc >= p.C) { cc = 0; if (++tapS == p.KW) { tapS = 0; ++tapR; } }
          }
          if (BMN) {
#pragma unroll
            for (int a = 0; a < BN / kAtomN; ++a)
              tmaLoad4d(stageB(s) + a * kSlabBytes, &mapB, &full[s], tileN * BN + a * kAtomN, kb * BK, zb1 * p.bZ1, zb0 * p.bZ0);
          } else {
            if constexpr (PAIR) tmaLoadPair4d(stageB(s), &mapB, &full[s], kb * BK, rowB, zb1 * p.bZ1, zb0 * p.bZ0);
            else tmaLoad4d(stageB(s), &mapB, &full[s], kb * BK, rowB, zb1 * p.bZ1, zb0 * p.bZ0);
            if (X3 && p.hasBLo) tmaLoad4d(stageBLo(s), &mapBLo, &full[s], kb * BK, rowB, zb1 * p.bZ1, zb0 * p.bZ0);
          }
        }
      }
      if (PAIR) {   // the MMAs' arrivals on this CTA's `empty` barriers have all come before it may leave
        for (uint32_t j = 0; j < (uint32_t)kStages && j < it && ok; ++j) {
          const uint32_t use = it - 1 - j;
          if (!mbarWait(&empty[use % kStages], (use / kStages) & 1, abortWord)) { atomicExch(p.status, 1); ok = false; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (lane == 0 && rank == 0) {
      auto commit = [](uint64_t* bar) { if constexpr (PAIR) mmaCommitPair(bar); else mmaCommit(bar); };
      auto mma = [](uint32_t d, uint64_t a, uint64_t b, uint32_t acc) { if constexpr (PAIR) mmaPairSS<TF32>(d, a, b, kIdesc, acc); else mmaSS<TF32>(d, a, b, kIdesc, acc); };
      auto waitIssuer = [&](uint64_t* bar, uint32_t parity) { return PAIR ? mbarWaitCluster(bar, parity, abortWord) : mbarWait(bar, parity, abortWord); };
      uint32_t it = 0, tcount = 0;
      bool ok = true;
      UnitWalk w(p, unit0, unitStep);
      for (uint32_t u = unit0; u < units && ok; u += unitStep, ++tcount, w.next(p)) {
        int kb0, kb1; kRange(w, kb0, kb1);
        const int ab = tcount & 1; const uint32_t aph = (tcount >> 1) & 1;
        if (!waitIssuer(&accEmpty[ab], aph ^ 1)) { atomicExch(p.status, 2); ok = false; break; }
        tcFenceAfter();
        const uint32_t accSet = tmemBase + (uint32_t)(ab * kSetCols);
        uint32_t cutAcc = accSet; int inChain = 0;          // CUT: where this K block's accumulator lies (divisions here held the MMAs up, 17 -> 20 us for 300 x 256 x 4096 tf32)
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % kStages; const uint32_t ph = (it / kStages) & 1;
          if (!waitIssuer(X3 ? &split[s] : &full[s], ph)) { atomicExch(p.status, 2); ok = false; break; }
          if (CONV && !X3) fenceProxyAsync();               // the gathered A tile was written through the generic proxy
          tcFenceAfter();
          const uint32_t acc = CUT ? cutAcc : accSet + (uint32_t)(((kb - kb0) % kChains) * BN);
          const bool fresh = X3 || !CUT ? kb - kb0 < accs : inChain == 0;      // first K block of this chain: overwrite
          if constexpr (CUT) {                              // tf32x3 takes the accumulators in turn, the other kinds one after the other
            ++inChain;
            if (X3) { cutAcc += BN; if (inChain == accs) { inChain = 0; cutAcc = accSet; } }
            else if (inChain == p.accBlocks) { inChain = 0; cutAcc += BN; }
          }
          const uint64_t dA = smemDescKMajorSw128(smemAddr(stageA(s)));
          const uint64_t dB = BMN ? smemDescMnMajorSw128(smemAddr(stageB(s)), kSlabBytes) : smemDescKMajorSw128(smemAddr(stageB(s)));
          constexpr uint64_t kAdvA = (UMMA_K * kElemBytes) >> 4;                      // 32 bytes of K inside the swizzle atom
          constexpr uint64_t kAdvB = BMN ? (uint64_t)(UMMA_K * 128) >> 4 : kAdvA;     // BMN: UMMA_K rows of 128 bytes
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            mma(acc, dA + k * kAdvA, dB + k * kAdvB, (!fresh || k > 0) ? 1u : 0u);
          if (X3) {
            const uint64_t dAl = smemDescKMajorSw128(smemAddr(stageALo(s)));
            const uint64_t dBl = BMN ? smemDescMnMajorSw128(smemAddr(stageBLo(s)), kSlabBytes) : smemDescKMajorSw128(smemAddr(stageBLo(s)));
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k) {
              mma(acc, dAl + k * kAdvA, dB + k * kAdvB, 1u);
              mma(acc, dA + k * kAdvA, dBl + k * kAdvB, 1u);
            }
          }
          commit(&empty[s]);
        }
        commit(&accFull[ab]);   // also reached after a failed wait so that the epilogue does not spin out
      }
    }
  } else if (warp < 2 + kEpiWarps) {
    // ---------------------------------------------------------------- epilogue
    // Warp w reads TMEM lanes 32*(w%4)..+31 (a hardware rule) and the column share (w-2)/4 of the tile, in chunks of 32
    // columns; the accumulator load of chunk i+1 is in flight while chunk i is worked on.  Results leave as units of
    // 32 rows x 64 bytes (32 bf16 or 16 fp32 columns, 64-byte swizzle), each staged in shared memory and written by one
    // TMA store, so that the store of a unit overlaps the arithmetic of the next.
    //   RES kernels: a warp owns a ring of four unit buffers.  The residual of a unit is loaded into its buffer by TMA
    //   three units ahead (across tile boundaries: it depends on nothing the MMAs produce), the lane adds its row,
    //   writes the result back into the same buffer and the store takes it from there.
    //   Other kernels: two (pairs: four) output slots used in turn; a residual, if any, comes through registers (below).
    // The per-column factors alpha * scale[n] and shift[n] reach the epilogue through shared memory: the 128 threads of a
    // column half load the next tile's while they work on this one's.  Loaded from global memory where they are used, they
    // waited behind the tile loads in every chunk (98304 x 2304 x 768 bf16 with a bias: 0.301 ms, without one 0.266).
    const int q = warp & 3, half = (warp - 2) >> 2;
    constexpr int kColsPerWarp = BN / (kEpiWarps / 4);
    constexpr int kChunks = kColsPerWarp / 32;
    constexpr bool kPrefetch = kChains == 1 && !CONV && !CUT;   // tf32x3 and CUT add several sums per chunk, and the gather form has no registers to spare
    constexpr uint32_t kRing = (uint32_t)S::kSlots;
    char* outBase = reinterpret_cast<char*>(p.out);
    const bool outF32 = p.out_dtype == LLC_FLOAT32;
    const bool tma = RES || p.tmaOut != 0;
    const int esz = outF32 ? 4 : 2;
    const int unitCols = 64 / esz;                              // columns of one staged unit
    const int nUnits = kColsPerWarp / unitCols;                 // units of this warp per tile
    uint8_t* const warpStaging = staging + (warp - 2) * kStagingPerWarp;
    const uint32_t slotBase = smemAddr(warpStaging);
    uint64_t* const myResFull = resFull + (warp - 2) * 4;
    uint32_t slotIt = 0;                                        // units this warp has staged so far; the buffer in use is slotIt % kRing
    // 16-byte piece c of row r of a unit buffer (64-byte swizzle: the piece index is XORed with bits 1-2 of the row)
    auto pieceAddr = [&](uint32_t slot, uint32_t r, uint32_t c) { return slotBase + (slot << 11) + r * 64u + ((c ^ ((r >> 1) & 3u)) << 4); };
    auto acquireSlot = [&]() { if (lane == 0) { if constexpr (kRing == 4) bulkWaitRead3(); else bulkWaitRead1(); } __syncwarp(); };   // the store kRing units ago has read its slot
    // RES (lane 0): starts the TMA load of the residual of this warp's next unit not requested yet, the m-th over all its
    // tiles, into buffer m % 4; past this CTA's last tile nothing is loaded and nobody waits.
    UnitWalk w(p, unit0, unitStep), resWalk = w;
    uint32_t resU = unit0, resM = 0; int resG = 0;
    auto loadResUnit = [&]() {
      if (resU >= units) return;
      uint64_t* bar = &myResFull[resM & 3u];
      mbarExpectTx(bar, 2048);
      tmaLoad4d(warpStaging + ((resM & 3u) << 11), &mapR, bar, resWalk.n * BN + half * kColsPerWarp + resG * unitCols, (resWalk.m * CG + rank) * BM + q * 32,
                resWalk.z1 * p.rZ1, resWalk.z0 * p.rZ0);
      ++resM;
      if (++resG == nUnits) { resG = 0; resU += unitStep; resWalk.next(p); }
    };
    if (RES && lane == 0) { prefetchTensorMap(&mapR); loadResUnit(); loadResUnit(); loadResUnit(); }
    if (tma && lane == 0) prefetchTensorMap(&mapO);
    const bool scaled = p.scale || p.alpha != 1.f, affine = scaled || p.shift;
    float* const myVec = tileVec + half * 2 * kColsPerWarp;
    const int vecCol = q * 32 + lane;                           // the column (of this half) whose factors this thread fetches
    float nextScale = 0.f, nextShift = 0.f;
    auto fetchVec = [&](int tileCol) {
      if (!affine || vecCol >= kColsPerWarp) return;
      const long long n = (long long)tileCol * BN + half * kColsPerWarp + vecCol;
      nextScale = p.alpha; nextShift = 0.f;
      if (n < p.N) { if (p.scale) nextScale *= __ldg(p.scale + n); if (p.shift) nextShift = __ldg(p.shift + n); }
    };
    fetchVec(w.n);
    uint32_t tcount = 0;
    for (uint32_t u = unit0; u < units; u += unitStep, ++tcount) {
      int kb0, kb1; kRange(w, kb0, kb1);
      const int tileM = w.m, tileN = w.n, zb0 = w.z0, zb1 = w.z1, sliceIdx = w.s;
      w.next(p);
      if (affine) {
        asm volatile("bar.sync %0, 128;" ::"r"(3 + half) : "memory");      // the previous tile's factors have been read
        if (vecCol < kColsPerWarp) { myVec[vecCol] = nextScale; myVec[kColsPerWarp + vecCol] = nextShift; }
        asm volatile("bar.sync %0, 128;" ::"r"(3 + half) : "memory");
        fetchVec(w.n);
      }
      const int ab = tcount & 1; const uint32_t aph = (tcount >> 1) & 1;
      const long long row0 = ((long long)tileM * CG + rank) * BM;
      const long long gm = row0 + q * 32 + lane;
      const bool rowOk = gm < p.M;
      const bool rowsInside = row0 + q * 32 < p.M;          // this warp's 32 rows are not all past the edge
      const long long oRow = zb0 * p.o_s0 + zb1 * p.o_s1 + gm * p.o_sm;
      const long long rRow = zb0 * p.r_s0 + zb1 * p.r_s1 + gm * p.r_sm;
      // Residual through registers (kernels without the ring).  A unit of the residual (32 rows x 64 bytes, the box
      // the output store writes) is fetched with coalesced 16-byte loads (four lanes per row, eight rows per
      // instruction), passed through the staging slot and read back one row per lane: lane = row is how the
      // accumulator arrives, but loading global memory that way touches 32 lines per instruction.  The loads of unit
      // g + 1 are issued when unit g is taken over, those of unit 0 while the MMAs still run.
      const bool resTile = !RES && !CONV && p.resTile && tma;    // (the gather kernel has no registers to spare and its layers no residual)
      uint4 rA[4];
      auto issueRes = [&](int g) {
        const int piece = lane & 3, r0 = lane >> 2;
        const long long gcol = (long long)tileN * BN + half * kColsPerWarp + (long long)g * unitCols + piece * (16 / esz);
        const char* base = reinterpret_cast<const char*>(p.res) + (zb0 * p.r_s0 + zb1 * p.r_s1 + gcol) * esz;
        const bool colOk = gcol < p.N;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const long long gr = row0 + q * 32 + j * 8 + r0;
          rA[j] = (gr < p.M && colOk) ? __ldg(reinterpret_cast<const uint4*>(base + gr * p.r_sm * esz)) : make_uint4(0u, 0u, 0u, 0u);
        }
      };
      // The lane's own row of the residual of the unit in buffer `slot`, as four 16-byte pieces.
      auto ownRow = [&](uint32_t slot, uint4* own) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(own[c].x), "=r"(own[c].y), "=r"(own[c].z), "=r"(own[c].w)
                       : "r"(pieceAddr(slot, (uint32_t)lane, (uint32_t)c)) : "memory");
      };
      // Takes unit g over (register path): the residual rows go through the acquired slot, the next unit's loads start.
      auto residualRow = [&](int g, uint4* own) {
        const uint32_t slot = slotIt % kRing;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 r = rA[j];
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(pieceAddr(slot, (uint32_t)(j * 8 + (lane >> 2)), (uint32_t)(lane & 3))), "r"(r.x), "r"(r.y),
                       "r"(r.z), "r"(r.w) : "memory");
        }
        __syncwarp();                                            // from here on every lane touches only its own row
        if (g + 1 < nUnits) issueRes(g + 1);
        ownRow(slot, own);
      };
      // Ring path: waits for the residual of the current unit to land and reads the lane's row.
      auto ringRow = [&](uint4* own) {
        if (!mbarWait(&myResFull[slotIt & 3u], (slotIt >> 2) & 1u, abortWord)) atomicExch(p.status, 4);
        ownRow(slotIt & 3u, own);
      };
      // Hands the staged unit to the TMA store (columns from x0 on; rows past M and columns past N are clipped by the
      // store).  A group is committed even when nothing is stored, so that "all but the latest group" always means
      // "every unit before this one".  RES: the buffer of the unit before this one is then free for the residual of
      // the unit three ahead.
      auto storeUnit = [&](long long x0) {
        fenceProxyAsync();
        __syncwarp();
        if (lane == 0) {
          if (rowsInside && x0 < p.N) tmaStore4d(&mapO, warpStaging + ((slotIt % kRing) << 11), (int)x0, (int)row0 + q * 32, zb1, zb0);
          bulkCommit();
          if (RES) { bulkWaitRead1(); loadResUnit(); }
        }
        ++slotIt;
      };
      auto stageF32 = [&](const float* w) {                      // 16 fp32 values -> the lane's row of the current buffer
        const uint32_t slot = slotIt % kRing;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(pieceAddr(slot, (uint32_t)lane, (uint32_t)c)), "f"(w[4 * c]), "f"(w[4 * c + 1]),
                       "f"(w[4 * c + 2]), "f"(w[4 * c + 3]) : "memory");
      };
      auto stageBf16 = [&](const float* w) {                     // 32 fp32 values, rounded to bf16
        const uint32_t slot = slotIt % kRing;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const __nv_bfloat162 a0 = __floats2bfloat162_rn(w[8 * c], w[8 * c + 1]), a1 = __floats2bfloat162_rn(w[8 * c + 2], w[8 * c + 3]);
          const __nv_bfloat162 a2 = __floats2bfloat162_rn(w[8 * c + 4], w[8 * c + 5]), a3 = __floats2bfloat162_rn(w[8 * c + 6], w[8 * c + 7]);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(pieceAddr(slot, (uint32_t)lane, (uint32_t)c)),
                       "r"(*reinterpret_cast<const unsigned*>(&a0)), "r"(*reinterpret_cast<const unsigned*>(&a1)), "r"(*reinterpret_cast<const unsigned*>(&a2)),
                       "r"(*reinterpret_cast<const unsigned*>(&a3)) : "memory");
        }
      };
      const bool splitK = CUT && p.splits > 1;
      if (resTile && !splitK) issueRes(0);
      if (!mbarWait(&accFull[ab], aph, abortWord)) atomicExch(p.status, 4);   // carry on with whatever is there: every warp must still reach the barriers below
      tcFenceAfter();
      const uint32_t acc = tmemBase + (uint32_t)(ab * kSetCols) + ((uint32_t)(q * 32) << 16);
      const int usedAccs = X3 ? (kb1 - kb0 < accs ? kb1 - kb0 : accs) : CUT ? (kb1 - kb0 + p.accBlocks - 1) / p.accBlocks : 1;
      auto loadAccs = [&](int c0, float* v) {           // the unit's sums, 32 columns from c0 on (the load is warp-collective)
        __syncwarp();
        tmemLoad32x32(acc + (uint32_t)c0, v);
        if (X3 || CUT) {
          int a = 1;
          if constexpr (!X3) {                          // two loads in flight
#pragma unroll 1
            for (; a + 1 < usedAccs; a += 2) {
              uint32_t w2[32], w3[32];
              tmemIssue32(acc + (uint32_t)(a * BN + c0), w2);
              tmemIssue32(acc + (uint32_t)((a + 1) * BN + c0), w3);
              tmemWait32(w2); tmemWait32(w3);
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = v[j] + __uint_as_float(w2[j]) + __uint_as_float(w3[j]);
            }
          }
#pragma unroll 1
          for (; a < usedAccs; ++a) {
            float w2[32];
            tmemLoad32x32(acc + (uint32_t)(a * BN + c0), w2);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += w2[j];
          }
        }
      };
      // Split-K: every slice parks its partial tile (fp32, this lane's row) in the workspace; the one that arrives last at
      // the tile's counter adds the slices up in order and runs the epilogue.  The slices of a tile run on different CTAs at
      // the same time (the grid holds every unit), so nobody waits for anybody.  Layout of a parked tile: [epilogue warp]
      // [32-column chunk][float4 of the chunk][lane], writer and reader being the same (warp, lane) of their CTAs, so that
      // one store or load of a warp covers 512 contiguous bytes.  (Clusters that meet in distributed shared memory instead
      // measured the same, 128 x 768 x 3072 bf16 11.1 against 11.4 us, and 48 clusters of three do not run at once.)
      const float4* const slices = reinterpret_cast<const float4*>(p.ws) + (size_t)(u - (uint32_t)sliceIdx) * (BM * BN / 4) +
                                   (size_t)((half * 4 + q) * (kColsPerWarp / 4)) * 32 + lane;        // slice 0 of this tile
      if (splitK) {
        float4* const mine = const_cast<float4*>(slices) + (size_t)sliceIdx * (BM * BN / 4);
#pragma unroll 1
        for (int ci = 0; ci < kChunks; ++ci) {
          const int c0 = half * kColsPerWarp + ci * 32;
          float v[32];
          loadAccs(c0, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) __stcg(mine + (ci * 8 + j) * 32, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
        }
        if (resTile) issueRes(0);                          // (lands under the meeting; the slices that come first need none of it)
        tcFenceBefore();
        __syncwarp();
        if (lane == 0) mbarArrive(&accEmpty[ab]);
        __threadfence();                                   // the partial tile is visible before the arrival is counted
        asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
        if (warp == 2 && lane == 0) {
          const int tile = (int)(u / (uint32_t)p.splits), before = atomicAdd(&p.counters[tile], 1);
          if (before == p.splits - 1) p.counters[tile] = 0;   // everyone has arrived: zero again for the next launch
          *lastFlag = before == p.splits - 1;
        }
        asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * 32) : "memory");
        if (!*lastFlag) continue;
        __threadfence();
      }
      constexpr bool pipelined = kPrefetch;
      uint32_t raw[32];
      if (pipelined) { __syncwarp(); tmemIssue32(acc + (uint32_t)(half * kColsPerWarp), raw); }
#pragma unroll 1
      for (int ci = 0; ci < kChunks; ++ci) {
        const int c0 = half * kColsPerWarp + ci * 32;
        float v[32];
        if (splitK) {                                   // the partial sums of all two to four slices in order (from L2), two slices in flight
          float4 even[8], odd[8];
          auto fetch = [&](int sl, float4* f) {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = __ldcg(slices + (size_t)sl * (BM * BN / 4) + (ci * 8 + j) * 32);
          };
          auto add = [&](const float4* f) {
#pragma unroll
            for (int j = 0; j < 8; ++j) { v[4 * j] += f[j].x; v[4 * j + 1] += f[j].y; v[4 * j + 2] += f[j].z; v[4 * j + 3] += f[j].w; }
          };
          fetch(0, even);
          if (!X3) fetch(1, odd);                       // (the split warps leave tf32x3 no registers for it)
#pragma unroll
          for (int j = 0; j < 8; ++j) { v[4 * j] = even[j].x; v[4 * j + 1] = even[j].y; v[4 * j + 2] = even[j].z; v[4 * j + 3] = even[j].w; }
          if constexpr (X3) {
#pragma unroll 1
            for (int sl = 1; sl < p.splits; ++sl) { fetch(sl, odd); add(odd); }
          } else {
            if (p.splits > 2) fetch(2, even);
            add(odd);
            if (p.splits > 3) fetch(3, odd);
            if (p.splits > 2) add(even);
            if (p.splits > 3) add(odd);
          }
        } else if (pipelined) {
          tmemWait32(raw);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(raw[j]);
          if (ci + 1 < kChunks) { __syncwarp(); tmemIssue32(acc + (uint32_t)(c0 + 32), raw); }
        } else {
          loadAccs(c0, v);
        }
        if (ci == kChunks - 1 && !splitK) {             // this warp's share is in registers: hand the accumulator back
          tcFenceBefore();
          __syncwarp();
          if (lane == 0) { if constexpr (PAIR) mbarArriveLeader(&accEmpty[ab]); else mbarArrive(&accEmpty[ab]); }
        }
        const long long gn0 = (long long)tileN * BN + c0;
        const bool inside = gn0 < p.N;
        const bool whole = p.vecOut && gn0 + 32 <= p.N;
        const int g0 = (ci * 32) / unitCols;              // first unit of this chunk
        // v = alpha * scale[n] * v + shift[n] (columns past the edge: alpha and 0, never stored)
        if (affine && inside) {
          const float4* sc = reinterpret_cast<const float4*>(myVec + ci * 32);
          const float4* sh = sc + kColsPerWarp / 4;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 b4 = sh[j];
            if (scaled) {
              const float4 s4 = sc[j];
              fma2(v[4 * j], v[4 * j + 1], s4.x, s4.y, b4.x, b4.y); fma2(v[4 * j + 2], v[4 * j + 3], s4.z, s4.w, b4.z, b4.w);
            } else {
              v[4 * j] += b4.x; v[4 * j + 1] += b4.y; v[4 * j + 2] += b4.z; v[4 * j + 3] += b4.w;
            }
          }
        }
        auto activate = [&](float* w, int count) {
          if (p.act == LLC_ACT_RELU) {
#pragma unroll
            for (int j = 0; j < 32; ++j) if (j < count) w[j] = fmaxf(w[j], 0.f);
          } else if (p.act == LLC_ACT_GELU) {
            if (outF32) {
#pragma unroll
              for (int j = 0; j < 32; ++j) if (j < count) w[j] = geluFast(w[j]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; j += 2) if (j < count) geluTanhBf16x2(w[j], w[j + 1]);
            }
          }
        };
        if constexpr (RES) {
          // every unit of every tile goes through the ring, inside the matrix or not (loads past the edge read zeros,
          // stores past the edge write nothing), so that buffers and barrier phases advance uniformly
          if (outF32) {
#pragma unroll
            for (int un = 0; un < 2; ++un) {
              uint4 own[4];
              ringRow(own);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                v[un * 16 + 4 * c] += __uint_as_float(own[c].x); v[un * 16 + 4 * c + 1] += __uint_as_float(own[c].y);
                v[un * 16 + 4 * c + 2] += __uint_as_float(own[c].z); v[un * 16 + 4 * c + 3] += __uint_as_float(own[c].w);
              }
              activate(v + un * 16, 16);
              stageF32(v + un * 16);
              storeUnit(gn0 + un * 16);
            }
          } else {
            uint4 own[4];
            ringRow(own);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&own[c]);
#pragma unroll
              for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); v[8 * c + 2 * e] += f.x; v[8 * c + 2 * e + 1] += f.y; }
            }
            activate(v, 32);
            stageBf16(v);
            storeUnit(gn0);
          }
        } else if (whole) {
          // residual, in fp32 (one rounding for the sum, whatever the storage type)
          bool slotHeld = false;                            // bf16: the unit's slot was acquired for the residual already
          if (resTile) {
            if (!outF32) {
              uint4 own[4];
              acquireSlot(); residualRow(g0, own); slotHeld = true;
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&own[c]);
#pragma unroll
                for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); v[8 * c + 2 * e] += f.x; v[8 * c + 2 * e + 1] += f.y; }
              }
            }                                               // fp32: two units per chunk, each takes its residual below
          } else if (p.res && rowOk) {
            if (p.r_sn == 1 && p.res_dtype == LLC_BFLOAT16 && ((rRow + gn0) & 3) == 0) {
              const __nv_bfloat16* rp = reinterpret_cast<const __nv_bfloat16*>(p.res) + rRow + gn0;
#pragma unroll
              for (int j = 0; j < 8; ++j) { float4 r4 = Vec4<__nv_bfloat16>::load(rp + 4 * j); v[4 * j] += r4.x; v[4 * j + 1] += r4.y; v[4 * j + 2] += r4.z; v[4 * j + 3] += r4.w; }
            } else if (p.r_sn == 1 && p.res_dtype == LLC_FLOAT32 && ((rRow + gn0) & 3) == 0) {
              const float* rp = reinterpret_cast<const float*>(p.res) + rRow + gn0;
#pragma unroll
              for (int j = 0; j < 8; ++j) { float4 r4 = Vec4<float>::load(rp + 4 * j); v[4 * j] += r4.x; v[4 * j + 1] += r4.y; v[4 * j + 2] += r4.z; v[4 * j + 3] += r4.w; }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += loadAs(p.res, rRow + (gn0 + j) * p.r_sn, p.res_dtype);
            }
          }
          // (with fp32 output and a residual tile the activation follows the residual, unit by unit, below)
          if (!(resTile && outF32)) activate(v, 32);
          if (tma) {
            if (outF32) {
#pragma unroll
              for (int un = 0; un < 2; ++un) {
                acquireSlot();
                if (resTile) {
                  uint4 own[4];
                  residualRow(g0 + un, own);
#pragma unroll
                  for (int c = 0; c < 4; ++c) {
                    v[un * 16 + 4 * c] += __uint_as_float(own[c].x); v[un * 16 + 4 * c + 1] += __uint_as_float(own[c].y);
                    v[un * 16 + 4 * c + 2] += __uint_as_float(own[c].z); v[un * 16 + 4 * c + 3] += __uint_as_float(own[c].w);
                  }
                  activate(v + un * 16, 16);
                }
                stageF32(v + un * 16);
                storeUnit(gn0 + un * 16);
              }
            } else {
              if (!slotHeld) acquireSlot();
              stageBf16(v);
              storeUnit(gn0);
            }
          } else if (rowOk) {
            if (outF32) {
              float* dst = reinterpret_cast<float*>(outBase) + oRow + gn0;
#pragma unroll
              for (int j = 0; j < 32; j += 4) Vec4<float>::store(dst + j, make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
            } else {
              uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(outBase) + oRow + gn0);
              const bool al16 = ((oRow + gn0) & 7) == 0;
              if (al16) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  __nv_bfloat162 a0 = __floats2bfloat162_rn(v[8 * j], v[8 * j + 1]), a1 = __floats2bfloat162_rn(v[8 * j + 2], v[8 * j + 3]);
                  __nv_bfloat162 a2 = __floats2bfloat162_rn(v[8 * j + 4], v[8 * j + 5]), a3 = __floats2bfloat162_rn(v[8 * j + 6], v[8 * j + 7]);
                  uint4 pk; pk.x = *reinterpret_cast<unsigned*>(&a0); pk.y = *reinterpret_cast<unsigned*>(&a1); pk.z = *reinterpret_cast<unsigned*>(&a2); pk.w = *reinterpret_cast<unsigned*>(&a3);
                  dst[j] = pk;
                }
              } else {
                __nv_bfloat16* d2 = reinterpret_cast<__nv_bfloat16*>(outBase) + oRow + gn0;
#pragma unroll
                for (int j = 0; j < 32; j += 4) Vec4<__nv_bfloat16>::store(d2 + j, make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]));
              }
            }
          }
        } else if (inside) {
          // ragged edge, continued: residual and activation element by element, then staged units or scalar stores
          if (rowOk) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const long long n = gn0 + j;
              if (n < p.N) {
                float x = v[j];
                if (p.res) x += loadAs(p.res, rRow + n * p.r_sn, p.res_dtype);
                v[j] = applyAct(x, p.act);
              }
            }
          }
          if (tma) {
            if (outF32) {
#pragma unroll
              for (int un = 0; un < 2; ++un) {
                if (gn0 + un * 16 < p.N) { acquireSlot(); stageF32(v + un * 16); storeUnit(gn0 + un * 16); }
              }
            } else {
              acquireSlot(); stageBf16(v); storeUnit(gn0);
            }
          } else if (rowOk) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (gn0 + j < p.N) storeAs(p.out, oRow + gn0 + j, p.out_dtype, v[j]);
          }
        }
      }
    }
    if (tma && lane == 0) bulkWaitRead();   // shared memory stays valid until the last store has read it
  } else if (CONV && warp < kGatherWarp0 + kGatherWarps) {
    // ---------------------------------------------------------------- im2col gather of A (convolution)
    // 256 threads; thread g owns 16-byte chunk (g & 7) of tile rows (g >> 3) + 32*j, j = 0..3, so that
    // eight neighbouring lanes fetch one row's 128 contiguous bytes.  A chunk never straddles a filter
    // tap (C * element size is a multiple of 16), so it is one load from x[n, ih, iw, c..] or zeros.
    // The tap of a chunk depends only on the K block, not on the row: it is tracked incrementally.
    constexpr int kChunkElems = 16 / kElemBytes;
    const int g = threadIdx.x - kGatherWarp0 * 32;
    const int chunk = g & 7, row0 = g >> 3;
    const char* X = reinterpret_cast<const char*>(p.x);
    const uint32_t dstOff = (uint32_t)(row0 * 128 + ((chunk ^ (row0 & 7)) << 4));   // (row0 + 32 j) & 7 == row0 & 7
    const int tapsPerBlock = (p.C <= BK && BK % p.C == 0) ? BK / p.C : 0;          // whole taps per K block
    uint32_t it = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {      // (the gathered form is never split along K)
      const int tileM = (int)(t / p.nTiles);                               // (one batch entry)
      long long rowBase[4]; int ih0[4], iw0[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long gm = (long long)tileM * BM + row0 + 32 * j;
        if (gm < p.M) {
          const int ow = (int)(gm % p.OW); const long long t2 = gm / p.OW; const int oh = (int)(t2 % p.OH); const long long img = t2 / p.OH;
          ih0[j] = oh * p.sh - p.ph; iw0[j] = ow * p.sw - p.pw;
          rowBase[j] = img * p.xs_n + (long long)ih0[j] * p.xs_h + (long long)iw0[j] * p.xs_w;
        } else { ih0[j] = -(1 << 28); iw0[j] = 0; rowBase[j] = 0; }   // never in range: the row is zero-filled
      }
      int tapR = 0, tapS = 0, cc = chunk * kChunkElems;       // filter tap and channel of this thread's chunk
      while (cc >= p.C) { cc -= p.C; if (++tapS == p.KW) { tapS = 0; ++tapR; } }
      for (int kb = 0; kb < p.kBlocks; ++kb, ++it) {
        const int s = it % kStages; const uint32_t ph = (it / kStages) & 1;
        if (!mbarWait(&empty[s], ph ^ 1, abortWord)) { atomicExch(p.status, 5); ok = false; break; }
        const int dIh = tapR * p.dh, dIw = tapS * p.dw;
        const long long tapOff = (long long)dIh * p.xs_h + (long long)dIw * p.xs_w + cc;
        const bool tapOk = tapR < p.KH;                        // past the last tap: K tail, zero-filled
        const uint32_t dst = smemAddr(stageA(s)) + dstOff;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool valid = tapOk && (unsigned)(ih0[j] + dIh) < (unsigned)p.H && (unsigned)(iw0[j] + dIw) < (unsigned)p.W;
          cpAsync16(dst + j * 32 * 128, X + (valid ? (rowBase[j] + tapOff) * kElemBytes : 0), valid);
        }
        cpAsyncArriveOn(&full[s]);                           // arrives when the four copies above have landed
        // next K block: 128 bytes further along K.  Narrow channel counts (the padded stem) step over several taps at once.
        if (tapsPerBlock > 0) { tapS += tapsPerBlock; while (tapS >= p.KW) { tapS -= p.KW; ++tapR; } }
        else { cc += BK; while (cc >= p.C) { cc -= p.C; if (++tapS == p.KW) { tapS = 0; ++tapR; } } }
      }
    }
    cpAsyncCommit();
    cpAsyncWait<0>();                                          // nothing of this thread is in flight at exit
  } else if (X3 && warp >= kSplitWarp0) {
    // ---------------------------------------------------------------- low-order tiles (tf32x3)
    // elementwise, so every 16-byte chunk keeps its swizzled position
    const int et = threadIdx.x - kSplitWarp0 * 32;
    uint32_t it = 0;
    bool ok = true;
    UnitWalk w(p, unit0, unitStep);
    for (uint32_t u = unit0; u < units && ok; u += unitStep, w.next(p)) {
      int kb0, kb1; kRange(w, kb0, kb1);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int s = it % kStages; const uint32_t ph = (it / kStages) & 1;
        if (!mbarWait(&full[s], ph, abortWord)) { atomicExch(p.status, 3); ok = false; break; }
        const float4* srcA = reinterpret_cast<const float4*>(stageA(s)); float4* dstA = reinterpret_cast<float4*>(stageALo(s));
        const float4* srcB = reinterpret_cast<const float4*>(stageB(s)); float4* dstB = reinterpret_cast<float4*>(stageBLo(s));
        auto lo = [](float x) { return x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u); };
#pragma unroll 4
        for (int i = et; i < S::kABytes / 16; i += 128) { float4 v = srcA[i]; dstA[i] = make_float4(lo(v.x), lo(v.y), lo(v.z), lo(v.w)); }
        if (!p.hasBLo) {
#pragma unroll 4
          for (int i = et; i < S::kBBytes / 16; i += 128) { float4 v = srcB[i]; dstB[i] = make_float4(lo(v.x), lo(v.y), lo(v.z), lo(v.w)); }
        }
        fenceProxyAsync();
        __syncwarp();
        if (lane == 0) mbarArrive(&split[s]);
      }
    }
  }
  tcFenceBefore();
  __syncwarp();
  // (neither CTA of a pair leaves while the other's MMAs may read its shared memory or arrive on its barriers)
  if (PAIR) clusterSync(); else __syncthreads();
  if (warp == 1) { tcFenceAfter(); if constexpr (PAIR) tmemDeallocPair(tmemBase, accCols); else tmemDealloc(tmemBase, accCols); }
}

// The tile a call is cut into: width, K slices, CTAs per tile, accumulators per unit, and whether the CUT kernels take it.
struct TilePlan { int bn; int splits; int cg; int accs; bool cut; };
struct TcMaps { CUtensorMap a, b, out, bLo, res; };

// Launches the kernel for one MODE and KIND (see tc_kernel); each pair is compiled in a file of its own.  `res`: the variant
// whose epilogue fetches the residual through a ring of TMA loads (bf16 / tf32, TMA-fed operands).  BMN: see tc_kernel.
template <int MODE, int KIND> int dispatchTc(const TilePlan& plan, bool res, const TcMaps& m, const TcArgs& a, long long batch, cudaStream_t st);
#define LLC_TC_DECLARE(MODE_, KIND_) template <> int dispatchTc<MODE_, KIND_>(const TilePlan& plan, bool res, const TcMaps& m, const TcArgs& a, long long batch, cudaStream_t st);
LLC_TC_DECLARE(0, 0) LLC_TC_DECLARE(0, 1) LLC_TC_DECLARE(0, 2) LLC_TC_DECLARE(1, 0) LLC_TC_DECLARE(1, 1) LLC_TC_DECLARE(1, 2)
LLC_TC_DECLARE(2, 0) LLC_TC_DECLARE(2, 1) LLC_TC_DECLARE(2, 2)
#undef LLC_TC_DECLARE
int dispatchTcMn(const TilePlan& plan, const TcMaps& m, const TcArgs& a, long long batch, cudaStream_t st);

// One instantiation: set up once per device, then launched.  CG == 2: clusters of two CTAs, one pair per two SMs.
template <int BN, int KIND, int MODE, bool BMN, bool RES, int CG, bool CUT>
int launchTc(const TcMaps& m, TcArgs a, long long batch, cudaStream_t st) {
  using S = Smem<BN, KIND, RES, CG>;
  static_assert(S::kStages >= 2, "at least two pipeline stages");
  static DeviceOnce configured;                          // the shared-memory opt-in is kept per device
  const int dev = currentDevice();
  auto kernel = tc_kernel<BN, KIND, MODE, BMN, RES, CG, CUT>;
  if (!configured.test(dev)) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (e != cudaSuccess) return cudaFail(e, "cudaFuncSetAttribute(tc_kernel)");
    configured.set(dev);
  }
  a.mTiles = (int)((a.M + CG * BM - 1) / (CG * BM)); a.nTiles = (int)((a.N + BN - 1) / BN);
  a.tiles = (long long)a.mTiles * a.nTiles * batch;
  if (!CUT) a.splits = 1;
  const long long units = a.tiles * a.splits, slots = deviceSMs() / CG;
  if (CUT && (units > slots || a.accs < 1 || a.accs * BN > 512)) return setError(LLC_ERR_INTERNAL, "llc internal: a call cut along K has one unit per CTA");
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((units < slots ? units : slots) * CG));
  cfg.blockDim = dim3(tcThreads(KIND, MODE));
  cfg.dynamicSmemBytes = S::kTotal;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if (CG == 2) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
  }
  LLC_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, m.a, m.b, m.out, m.bLo, m.res, a));
  return LLC_OK;
}

#define LLC_TC_CASE(BN_, R_, CG_) if (plan.bn == BN_ && res == R_ && plan.cg == CG_ && !plan.cut) return launchTc<BN_, KIND, MODE, false, R_, CG_, false>(m, a, batch, st);
#define LLC_TC_CUT(BN_) if (plan.bn == BN_ && plan.cut) return launchTc<BN_, KIND, MODE, false, false, 1, true>(m, a, batch, st);
#define LLC_TC_DISPATCH(MODE_, KIND_, CASES)                                                                                                             \
  template <> int dispatchTc<MODE_, KIND_>(const TilePlan& plan, bool res, const TcMaps& m, const TcArgs& a, long long batch, cudaStream_t st) {          \
    constexpr int MODE = MODE_, KIND = KIND_;                                                                                                            \
    CASES                                                                                                                                                \
    return setError(LLC_ERR_INTERNAL, "llc internal: no tensor-core kernel for this tile");                                                              \
  }
#define LLC_TC_WIDTHS(R_, CG_) LLC_TC_CASE(64, R_, CG_) LLC_TC_CASE(128, R_, CG_) LLC_TC_CASE(256, R_, CG_)

}  // namespace tcgemm
}  // namespace llc
