// Host side of the tensor-core GEMM and convolution: tensor maps, the choice of tile, the calls that go there.
// The kernel is in gemm_tc_kernel.cuh, its instantiations in gemm_tc_{dense,im2col}_*.cu and gemm_tc_gather.cu.
#include "gemm_tc_kernel.cuh"

namespace llc {

__device__ int g_tcStatus = 0;   // see TcArgs::status

// Device address of the status word on the current device (for the kernels, and for callers that copy it back on their own stream).
int* tcStatusAddress() {
  static std::atomic<int*> cache[64];
  const int dev = currentDevice();
  if (dev >= 0 && dev < 64) { int* c = cache[dev].load(std::memory_order_acquire); if (c) return c; }
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_tcStatus) != cudaSuccess) return nullptr;
  if (dev >= 0 && dev < 64) cache[dev].store(static_cast<int*>(p), std::memory_order_release);
  return static_cast<int*>(p);
}

namespace {

using namespace tcgemm;

// ---- host side ------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encodeTiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// K-major operand [b0, b1, rows, K] with unit stride along K -> 4-D tensor map, box = 128 bytes of K x boxRows rows.
bool makeMap(CUtensorMap* map, const void* base, bool f32, long long K, long long rows, long long b1, long long b0, long long sRow, long long s1,
             long long s0, int boxRows) {
  EncodeTiledFn enc = encodeTiled();
  if (!enc) return false;
  const int eb = f32 ? 4 : 2;
  // a broadcast batch dim (stride 0) or a unit extent becomes extent 1 with any legal stride
  const bool has1 = b1 > 1 && s1 > 0, has0 = b0 > 1 && s0 > 0;
  const long long dense = sRow * rows;
  cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)(has1 ? b1 : 1), (cuuint64_t)(has0 ? b0 : 1)};
  cuuint64_t strides[3] = {(cuuint64_t)(sRow * eb), (cuuint64_t)((has1 ? s1 : dense) * eb), (cuuint64_t)((has0 ? s0 : dense) * eb)};
  cuuint32_t box[4] = {(cuuint32_t)(kTileKBytes / eb), (cuuint32_t)boxRows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const int*, const int*,
                                   cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                   CUtensorMapFloatOOBfill);
EncodeIm2colFn encodeIm2col() {
  static EncodeIm2colFn fn = []() -> EncodeIm2colFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<EncodeIm2colFn>(p);
  }();
  return fn;
}

// NHWC activations -> im2col tensor map: a load brings 128 output positions x 128 bytes of channels for one filter tap.
// The bounding box is the set of input pixels that sit under tap (0, 0) of some output position: it starts `pad` pixels
// before the image and ends (kernel extent - 1 - pad) pixels before its end; the traversal strides are the convolution's.
bool makeIm2colMap(CUtensorMap* map, const LlcConvParams* p, bool f32) {
  EncodeIm2colFn enc = encodeIm2col();
  if (!enc) return false;
  const int eb = f32 ? 4 : 2;
  cuuint64_t dims[4] = {(cuuint64_t)p->c, (cuuint64_t)p->w_in, (cuuint64_t)p->h, (cuuint64_t)p->n};
  const bool dense = p->x_sn == 0 && p->x_sh == 0 && p->x_sw == 0;
  cuuint64_t strides[3] = {(cuuint64_t)((dense ? p->c : p->x_sw) * eb), (cuuint64_t)((dense ? p->w_in * p->c : p->x_sh) * eb),
                           (cuuint64_t)((dense ? p->h * p->w_in * p->c : p->x_sn) * eb)};
  int lower[2] = {-p->pad_w, -p->pad_h};
  int upper[2] = {p->pad_w - (int)(p->kw - 1) * p->dil_w, p->pad_h - (int)(p->kh - 1) * p->dil_h};
  cuuint32_t estr[4] = {1, (cuuint32_t)p->stride_w, (cuuint32_t)p->stride_h, 1};
  CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(p->x), dims, strides, lower, upper,
                   (cuuint32_t)(kTileKBytes / eb), (cuuint32_t)BM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}
// Whether the im2col load can serve this convolution: a K block inside one tap, corners and tap offsets inside the
// ranges the 4-D descriptor and instruction encode, and the output extents exactly those the bounding box yields.
bool im2colEligible(const LlcConvParams* p, bool f32) {
  const int eb = f32 ? 4 : 2;
  static const bool off = []() { const char* e = getenv("LLC_TC_CONV_GATHER"); return e && e[0] == '1'; }();
  if (off || (p->c * eb) % kTileKBytes != 0) return false;
  const int lowW = -p->pad_w, lowH = -p->pad_h;
  const int upW = p->pad_w - (int)(p->kw - 1) * p->dil_w, upH = p->pad_h - (int)(p->kh - 1) * p->dil_h;
  auto in8 = [](int v) { return v >= -128 && v <= 127; };
  if (!in8(lowW) || !in8(lowH) || !in8(upW) || !in8(upH)) return false;
  if ((p->kw - 1) * p->dil_w > 255 || (p->kh - 1) * p->dil_h > 255) return false;
  if (p->stride_w < 1 || p->stride_w > 8 || p->stride_h < 1 || p->stride_h > 8) return false;
  const long long extW = p->w_in + upW - lowW, extH = p->h + upH - lowH;     // base positions per row / column
  if (extW < 1 || extH < 1) return false;
  if ((extW - 1) / p->stride_w + 1 != p->ow || (extH - 1) / p->stride_h + 1 != p->oh) return false;
  if (p->n * p->oh * p->ow > (1LL << 31)) return false;
  return encodeIm2col() != nullptr;
}

// MN-major operand [b0, b1, K, N] with unit stride along N -> 4-D tensor map, box = 128 bytes of N x boxK rows of K.
bool makeMapMn(CUtensorMap* map, const void* base, bool f32, long long N, long long K, long long b1, long long b0, long long sK, long long s1,
               long long s0, int boxK) {
  EncodeTiledFn enc = encodeTiled();
  if (!enc) return false;
  const int eb = f32 ? 4 : 2;
  const bool has1 = b1 > 1 && s1 > 0, has0 = b0 > 1 && s0 > 0;
  const long long dense = sK * K;
  cuuint64_t dims[4] = {(cuuint64_t)N, (cuuint64_t)K, (cuuint64_t)(has1 ? b1 : 1), (cuuint64_t)(has0 ? b0 : 1)};
  cuuint64_t strides[3] = {(cuuint64_t)(sK * eb), (cuuint64_t)((has1 ? s1 : dense) * eb), (cuuint64_t)((has0 ? s0 : dense) * eb)};
  cuuint32_t box[4] = {(cuuint32_t)(kTileKBytes / eb), (cuuint32_t)boxK, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Output [b0, b1, M, N] with unit stride along N -> 4-D tensor map for the epilogue's stores; box = rowBytes of N x 32 rows,
// swizzle span = rowBytes (64 or 128).  Returns false when the layout cannot be described (the epilogue then stores directly).
bool makeOutMap(CUtensorMap* map, void* base, bool f32, long long N, long long M, long long b1, long long b0, long long sRow, long long s1,
                long long s0, int rowBytes) {
  EncodeTiledFn enc = encodeTiled();
  if (!enc) return false;
  const int eb = f32 ? 4 : 2;
  const bool has1 = b1 > 1, has0 = b0 > 1;
  auto ok16 = [&](long long s) { return s > 0 && (s * eb) % 16 == 0; };
  if ((reinterpret_cast<uintptr_t>(base) & 15) || !ok16(sRow) || sRow < N || (has1 && !ok16(s1)) || (has0 && !ok16(s0))) return false;
  if (N > (1LL << 31) || M > (1LL << 31)) return false;
  const long long dense = sRow * M;
  cuuint64_t dims[4] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)(has1 ? b1 : 1), (cuuint64_t)(has0 ? b0 : 1)};
  cuuint64_t strides[3] = {(cuuint64_t)(sRow * eb), (cuuint64_t)((has1 ? s1 : dense) * eb), (cuuint64_t)((has0 ? s0 : dense) * eb)};
  cuuint32_t box[4] = {(cuuint32_t)(rowBytes / eb), 32, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, rowBytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}
// Residual [b0, b1, M, N] (unit stride along N, batch dims possibly broadcast) -> the same 64-byte x 32-row boxes as the
// output map, for the ring of TMA loads in the RES kernels.  `has1` / `has0` tell whether the batch coordinates apply.
bool makeResMap(CUtensorMap* map, const void* base, bool f32, long long N, long long M, long long b1, long long b0, long long sRow, long long s1,
                long long s0, bool* has1Out, bool* has0Out) {
  EncodeTiledFn enc = encodeTiled();
  if (!enc) return false;
  const int eb = f32 ? 4 : 2;
  const bool has1 = b1 > 1 && s1 > 0, has0 = b0 > 1 && s0 > 0;
  auto ok16 = [&](long long s) { return s > 0 && (s * eb) % 16 == 0; };
  if ((reinterpret_cast<uintptr_t>(base) & 15) || !ok16(sRow) || sRow < N || (has1 && !ok16(s1)) || (has0 && !ok16(s0))) return false;
  if ((b1 > 1 && s1 < 0) || (b0 > 1 && s0 < 0) || N > (1LL << 31) || M > (1LL << 31)) return false;
  const long long dense = sRow * M;
  cuuint64_t dims[4] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)(has1 ? b1 : 1), (cuuint64_t)(has0 ? b0 : 1)};
  cuuint64_t strides[3] = {(cuuint64_t)(sRow * eb), (cuuint64_t)((has1 ? s1 : dense) * eb), (cuuint64_t)((has0 ? s0 : dense) * eb)};
  cuuint32_t box[4] = {(cuuint32_t)(64 / eb), 32, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  *has1Out = has1; *has0Out = has0;
  return enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// LLC_TC_RES_RING=0 keeps residuals on the register path (used to compare the two).
bool resRingEnabled() {
  static const bool on = []() { const char* e = getenv("LLC_TC_RES_RING"); return !(e && e[0] == '0'); }();
  return on;
}
// Bytes per row of the output box the epilogue stages and stores: 32 bf16 or 16 fp32 columns.
constexpr int kOutBoxBytes = 64;

int numSMs() { return deviceSMs(); }

// LLC_TC_SPLITK=0 keeps every K loop in one piece (2 is accepted and means the default: split wherever SMs would idle).
int splitKMode() {
  const char* e = getenv("LLC_TC_SPLITK");
  return e && *e ? atoi(e) : 1;
}
bool splitKEnabled() { return splitKMode() != 0; }

// LLC_TC_DIRECT_STORES=1 keeps the epilogue on direct global stores (used to compare the two paths).
bool tmaEpilogueEnabled() {
  static const bool on = []() { const char* e = getenv("LLC_TC_DIRECT_STORES"); return !(e && e[0] == '1'); }();
  return on;
}

// LLC_TC_PAIR=0 keeps every tile on one CTA, 2 takes CTA pairs wherever they can run (the tests use it to send small shapes there).
int pairModeEnv() {
  const char* e = getenv("LLC_TC_PAIR");
  return e && *e ? atoi(e) : 1;
}

// LLC_TC_SLICES=n cuts K into n slices wherever they can run (the tests use it to reach every way of meeting).
int slicesEnv() {
  const char* e = getenv("LLC_TC_SLICES");
  return e && *e ? atoi(e) : 0;
}

int ceilDiv(long long a, long long b) { return (int)((a + b - 1) / b); }
// Accumulators a unit always has: tf32x3 spreads its K blocks over 256 columns of tensor memory.
int setAccs(int kind, int bn) { return kind == 2 ? 256 / bn : 1; }

// Workspace of a call cut into K slices: 4096 bytes of arrival counters and the parked partial tiles.
long long parkedBytes(long long tiles, int splits, int bn) { return 4096 + tiles * splits * (long long)BM * bn * 4; }

// K blocks one accumulator may sum up.  The tensor core truncates what it adds, so the error of a result grows with the
// length of its sums (64 x 128 x 1024 bf16 against float64: 1.0e-6 of the result as one sum, 2.3e-7 as four), and a plan
// that is chosen by time alone would trade accuracy for it.  The line: a call whose tiles leave at least half of the SMs idle
// sums what up to four K slices over the idle SMs would, of at least four K blocks, at the width that is fastest when
// slices meet in memory at 10 us a tile.  chooseTile reaches it by slices or by accumulators.
int longestChain(long long M, long long N, long long batch, bool allow256, int kind, int kBlocks, long long wsBytes) {
  static const float kBlockUs[3][3] = {{0.22f, 0.25f, 0.40f}, {0.28f, 0.33f, 0.50f}, {0.60f, 0.75f, 0.f}};   // [kind][width]
  static const float epilogueUs[3] = {0.8f, 1.2f, 2.0f};
  int chain = kBlocks; float bestCost = 0.f;
  for (int i = 0; i < 3; ++i) {
    const int bn = 64 << i;
    if (bn == 256 && (!allow256 || kind == 2)) continue;
    if (i > 0 && N <= bn / 2) continue;
    const long long tiles = (M + BM - 1) / BM * ((N + bn - 1) / bn) * batch;
    int splits = 1;
    if (wsBytes > 0 && tiles * 2 <= numSMs() && kBlocks >= 8) {
      splits = (int)(numSMs() / tiles < 4 ? numSMs() / tiles : 4);
      while (splits > 1 && (kBlocks / splits < 4 || parkedBytes(tiles, splits, bn) > wsBytes)) --splits;
    }
    const float loop = ceilDiv(kBlocks, splits) * kBlockUs[kind][i];
    const float cost = (float)((tiles * splits + numSMs() - 1) / numSMs()) * ((loop > epilogueUs[i] ? loop : epilogueUs[i]) + 0.3f) + (splits > 1 ? 10.f : 0.f);
    if (i == 0 || cost <= bestCost) { chain = ceilDiv(ceilDiv(kBlocks, splits), setAccs(kind, bn)); bestCost = cost; }
  }
  return chain;
}

// Tile by a cost model: a persistent CTA (pair) works through ceil(tiles / slots) tiles, and a tile costs the longer of its
// main loop (K blocks x a per-block time that grows slowly with the width, because narrow tiles are bound by operand
// traffic and latency rather than by the tensor pipe) and its epilogue.  Times in microseconds, measured on B200.
// CTA pairs (256 x 256 tiles) exist for bf16 and tf32: each CTA fetches half of B, so a K block takes 0.42 us instead of
// 0.46 (tf32 0.45 / 0.54), at 0.6 us more for setting up the pair.  98304 x 768 x 3072 bf16 0.372 -> 0.323 ms, 98304 x 2304 x
// 768 0.264 -> 0.250, 4096 x 768 x 3072 tf32 58 -> 48 us; 6144 x 768 x 768 (one round either way) 19.4 against 21.4 us, which
// is what the 0.6 is for.  Narrower pair tiles and tf32x3 pairs measured equal to single CTAs and are not built.
// `wsBytes` > 0 allows slices: where the tiles leave SMs idle, K may be cut into up to four that run side by side, one unit
// per CTA, and meet in the workspace, 3.5 to 13 us by the bytes that are parked.  (As clusters that met in distributed
// shared memory 1024 x 768 x 3072 tf32x3 had only two slices and took 44.5 us; in three, through memory, 34.7.)
TilePlan chooseTile(long long M, long long N, long long batch, bool allow256, int kind, int kBlocks, long long wsBytes, bool allowPair) {
  static const float kBlockUs[3][3] = {{0.32f, 0.36f, 0.46f}, {0.33f, 0.37f, 0.54f}, {0.66f, 0.80f, 0.f}};   // [kind][width]
  static const float kPairUs[2] = {0.42f, 0.45f};
  static const float epilogueUs[3] = {0.8f, 1.2f, 2.0f};
  static const float meetingUs[3] = {2.5f, 2.5f, 3.f}, parkUs[3] = {0.5f, 1.f, 2.6f};
  const int pairMode = kind == 2 || !allowPair || !allow256 ? 0 : pairModeEnv(), forced = wsBytes > 0 ? slicesEnv() : 0;
  const int chain = longestChain(M, N, batch, allow256, kind, kBlocks, wsBytes);
  const long long mT = (M + BM - 1) / BM;
  TilePlan best{64, 1, 1, setAccs(kind, 64), false}; float bestCost = 0.f;
  for (int i = 0; i < 3; ++i) {
    const int bn = 64 << i;
    if (bn == 256 && (!allow256 || kind == 2)) continue;
    if (i > 0 && N <= bn / 2) continue;                    // at least half of the tile's columns exist
    const long long tiles = mT * ((N + bn - 1) / bn) * batch;
    for (int splits = 1; splits <= 4; ++splits) {
      if (splits > 1 && (kBlocks / splits < 4 || tiles * splits > numSMs())) break;      // (four K blocks a slice also mean that none is empty)
      if (splits > 1 && parkedBytes(tiles, splits, bn) > wsBytes) break;
      if (forced && splits != forced) continue;
      const int perSlice = ceilDiv(kBlocks, splits), set = setAccs(kind, bn);
      const int accs = ceilDiv(perSlice, chain) > set ? ceilDiv(perSlice, chain) : set;
      if (accs > set && (wsBytes <= 0 || tiles * splits > numSMs() || accs * bn > 512)) continue;        // accumulators beyond the set's: one unit per CTA
      const long long rounds = (tiles * splits + numSMs() - 1) / numSMs();
      const float loop = perSlice * kBlockUs[kind][i];
      const float cost = (float)rounds * ((loop > epilogueUs[i] ? loop : epilogueUs[i]) + 0.3f) + (splits > 1 ? meetingUs[i] + parkUs[i] * (float)splits : 0.f);
      if (bestCost == 0.f || cost <= bestCost) { best = TilePlan{bn, splits, 1, accs, splits > 1 || accs > set}; bestCost = cost; }
    }
  }
  if (pairMode != 0 && !forced && (N > 128 || pairMode == 2)) {
    const long long tiles = ((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256) * batch, slots = numSMs() / 2;
    const float loop = kBlocks * kPairUs[kind];
    const float cost = (float)((tiles + slots - 1) / slots) * ((loop > epilogueUs[2] ? loop : epilogueUs[2]) + 0.3f) + 0.6f;
    if (pairMode == 2 || (chain >= kBlocks && cost <= bestCost)) best = TilePlan{256, 1, 2, 1, false};
  }
  return best;
}

// The plan as the kernel reads it.
void setPlan(TcArgs& a, const TilePlan& plan, void* workspace) {
  a.splits = plan.splits; a.accs = plan.accs; a.accBlocks = ceilDiv(ceilDiv(a.kBlocks, plan.splits), plan.accs);
  if (plan.splits > 1) { a.counters = reinterpret_cast<int*>(workspace); a.ws = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + 4096); }
}
// Bytes of a caller's workspace that slices can meet in.
long long usableWorkspace(const void* workspace, long long bytes) {
  return workspace && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0 && splitKEnabled() ? bytes : 0;
}

}  // namespace

// Whether the tensor-core kernel takes this call (otherwise the FMA kernel does).
bool tcGemmSupported(const LlcGemmParams* p) {
  const bool f32 = p->in_dtype == LLC_FLOAT32;
  if (!f32 && p->in_dtype != LLC_BFLOAT16) return false;
  if (f32 && p->precision != LLC_PREC_TF32 && p->precision != LLC_PREC_TF32X3) return false;
  const bool bmn = p->b_sk != 1;                        // B stored [k][n]
  if (bmn && p->b_sn != 1) return false;
  if (bmn && f32) return false;                         // 32-bit operands are taken K-major only (an MN-major tf32 B produced zeros on B200)
  const int eb = f32 ? 4 : 2;
  auto ok16 = [&](long long s) { return (s * eb) % 16 == 0; };
  if (!ok16(p->a_sm) || !ok16(p->a_s0) || !ok16(p->a_s1) || !ok16(bmn ? p->b_sk : p->b_sn) || !ok16(p->b_s0) || !ok16(p->b_s1)) return false;
  if (p->a_sm < p->k || (bmn ? p->b_sk < p->n : p->b_sn < p->k)) return false;   // overlapping rows are not expressible as a tensor map
  if (p->a_s0 < 0 || p->a_s1 < 0 || p->b_s0 < 0 || p->b_s1 < 0) return false;
  if ((reinterpret_cast<uintptr_t>(p->a) | reinterpret_cast<uintptr_t>(p->b)) & 15) return false;
  if (p->m < 1 || p->n < 1 || p->k < 1) return false;
  // (work units are counted in 32 bits: 128 x 64 tiles, at most four K slices each)
  if (((p->m + BM - 1) / BM) * ((p->n + 63) / 64) > (1LL << 28) / ((p->b0 > 0 ? p->b0 : 1) * (p->b1 > 0 ? p->b1 : 1))) return false;
  if (p->b0 > (1 << 30) || p->b1 > (1 << 30) || p->m > (1LL << 31) * 64 || p->n > (1LL << 31)) return false;
  // tiny problems: the FMA kernel has less fixed cost.  For 32-bit operands the break-even measured near 2^25
  // multiply-adds (64x512x784 took 20 us on either kernel, 64x10x512 19 us against 27 us); LLC_TC_MIN_MACS_LOG2 moves it.
  const char* minEnv = getenv("LLC_TC_MIN_MACS_LOG2");
  int minLog2F32 = minEnv && *minEnv ? atoi(minEnv) : 25;
  minLog2F32 = minLog2F32 < 0 ? 0 : (minLog2F32 > 40 ? 40 : minLog2F32);
  const long long macs = p->m * p->n * p->k * (p->b0 > 0 ? p->b0 : 1) * (p->b1 > 0 ? p->b1 : 1);
  if (p->m * p->n * p->k < (1LL << 18) || (f32 && macs < (1LL << minLog2F32))) return false;
  return encodeTiled() != nullptr;
}

int tcGemm(const LlcGemmParams* p, cudaStream_t st) {
  const bool f32 = p->in_dtype == LLC_FLOAT32;
  const int eb = f32 ? 4 : 2;
  const int bk = kTileKBytes / eb;
  const long long batch = p->b0 * p->b1;
  const bool bmn = p->b_sk != 1;
  const int kind = !f32 ? 0 : (p->precision == LLC_PREC_TF32X3 ? 2 : 1);
  const TilePlan plan = chooseTile(p->m, p->n, batch, !bmn, kind, (int)((p->k + bk - 1) / bk), bmn ? 0 : usableWorkspace(p->workspace, p->workspace_bytes), !bmn);
  const int bn = plan.bn;
  CUtensorMap ma, mb;
  bool okMaps = makeMap(&ma, p->a, f32, p->k, p->m, p->b1, p->b0, p->a_sm, p->a_s1, p->a_s0, BM);
  okMaps = okMaps && (bmn ? makeMapMn(&mb, p->b, f32, p->n, p->k, p->b1, p->b0, p->b_sk, p->b_s1, p->b_s0, bk)
                          : makeMap(&mb, p->b, f32, p->k, p->n, p->b1, p->b0, p->b_sn, p->b_s1, p->b_s0, bn / plan.cg));
  if (!okMaps) return setError(LLC_ERR_CUDA, "llc cuda: cuTensorMapEncodeTiled rejected the GEMM operands");
  TcArgs a{};
  a.status = tcStatusAddress();
  if (!a.status) return setError(LLC_ERR_CUDA, "llc cuda: the status word of the tensor-core kernels has no address");
  a.out = p->out; a.scale = p->scale; a.shift = p->shift; a.res = p->res;
  a.out_dtype = p->out_dtype; a.res_dtype = p->res_dtype; a.act = p->act; a.alpha = p->alpha;
  a.M = p->m; a.N = p->n; a.K = p->k;
  a.o_s0 = p->o_s0; a.o_s1 = p->o_s1; a.o_sm = p->o_sm; a.r_s0 = p->r_s0; a.r_s1 = p->r_s1; a.r_sm = p->r_sm; a.r_sn = p->r_sn;
  a.b1 = (int)p->b1; a.kBlocks = (int)((p->k + bk - 1) / bk);
  setPlan(a, plan, p->workspace);
  a.aZ0 = p->b0 > 1 && p->a_s0 > 0; a.aZ1 = p->b1 > 1 && p->a_s1 > 0; a.bZ0 = p->b0 > 1 && p->b_s0 > 0; a.bZ1 = p->b1 > 1 && p->b_s1 > 0;
  const int ob = p->out_dtype == LLC_FLOAT32 ? 4 : 2;
  a.vecOut = (reinterpret_cast<uintptr_t>(p->out) % (ob * 4)) == 0 && p->o_sm % 4 == 0 && p->o_s0 % 4 == 0 && p->o_s1 % 4 == 0;
  CUtensorMap mo = ma;   // a valid map even when unused
  if (tmaEpilogueEnabled() && makeOutMap(&mo, p->out, ob == 4, p->n, p->m, p->b1, p->b0, p->o_sm, p->o_s1, p->o_s0, kOutBoxBytes)) a.tmaOut = kOutBoxBytes;
  auto r16 = [&](long long st) { return st >= 0 && (st * ob) % 16 == 0; };
  a.resTile = p->res && p->r_sn == 1 && p->res_dtype == p->out_dtype && (reinterpret_cast<uintptr_t>(p->res) & 15) == 0 && r16(p->r_sm) && r16(p->r_s0) &&
              r16(p->r_s1) && p->n % (16 / ob) == 0;
  CUtensorMap mbl = mb;
  if (kind == 2 && !bmn && p->b_lo && (reinterpret_cast<uintptr_t>(p->b_lo) & 15) == 0 &&
      makeMap(&mbl, p->b_lo, f32, p->k, p->n, p->b1, p->b0, p->b_sn, p->b_s1, p->b_s0, bn / plan.cg))
    a.hasBLo = 1;
  // the residual through a ring of TMA loads: whole tiles only (no split-K), same element type as the output
  CUtensorMap mr = mo;
  bool resRing = false;
  if (a.resTile && a.tmaOut && !plan.cut && kind != 2 && !bmn && resRingEnabled()) {
    bool h1 = false, h0 = false;
    if (makeResMap(&mr, p->res, ob == 4, p->n, p->m, p->b1, p->b0, p->r_sm, p->r_s1, p->r_s0, &h1, &h0)) { resRing = true; a.rZ1 = h1; a.rZ0 = h0; }
  }
  const TcMaps maps{ma, mb, mo, mbl, mr};
  if (bmn) return dispatchTcMn(plan, maps, a, batch, st);
  return kind == 0 ? dispatchTc<0, 0>(plan, resRing, maps, a, batch, st) : kind == 1 ? dispatchTc<0, 1>(plan, resRing, maps, a, batch, st) : dispatchTc<0, 2>(plan, false, maps, a, batch, st);
}

bool tcConvSupported(const LlcConvParams* p) {
  const bool f32 = p->in_dtype == LLC_FLOAT32;
  if (!f32 && p->in_dtype != LLC_BFLOAT16) return false;
  if (f32 && p->precision != LLC_PREC_TF32 && p->precision != LLC_PREC_TF32X3) return false;
  const int eb = f32 ? 4 : 2;
  if ((p->c * eb) % 16 != 0) return false;              // a 16-byte chunk must stay inside one filter tap
  if ((p->x_sn * eb) % 16 != 0 || (p->x_sh * eb) % 16 != 0 || (p->x_sw * eb) % 16 != 0 || p->x_sn < 0 || p->x_sh < 0 || p->x_sw < 0) return false;
  if ((reinterpret_cast<uintptr_t>(p->x) | reinterpret_cast<uintptr_t>(p->w)) & 15) return false;
  const long long M = p->n * p->oh * p->ow, K = p->kh * p->kw * p->c;
  if (M * p->f * K < (1LL << 18)) return false;
  if (((M + BM - 1) / BM) * ((p->f + 63) / 64) > (1LL << 28)) return false;      // (work units are counted in 32 bits)
  return encodeTiled() != nullptr;
}

int tcConv(const LlcConvParams* p, cudaStream_t st) {
  const bool f32 = p->in_dtype == LLC_FLOAT32;
  const int eb = f32 ? 4 : 2;
  const int bk = kTileKBytes / eb;
  const long long M = p->n * p->oh * p->ow, K = p->kh * p->kw * p->c;
  const int kind = !f32 ? 0 : (p->precision == LLC_PREC_TF32X3 ? 2 : 1);
  // the plan comes after the map: a refused one leaves the gathered form, whose tiles are not cut and not paired
  CUtensorMap ma, mb;
  const bool im2col = im2colEligible(p, f32) && makeIm2colMap(&ma, p, f32);
  const TilePlan plan = chooseTile(M, p->f, 1, true, kind, (int)((K + bk - 1) / bk), im2col ? usableWorkspace(p->workspace, p->workspace_bytes) : 0, im2col);
  const int bn = plan.bn;
  if (!makeMap(&mb, p->w, f32, K, p->f, 1, 1, K, 0, 0, bn / plan.cg))
    return setError(LLC_ERR_CUDA, "llc cuda: cuTensorMapEncodeTiled rejected the convolution weights");
  TcArgs a{};
  a.status = tcStatusAddress();
  if (!a.status) return setError(LLC_ERR_CUDA, "llc cuda: the status word of the tensor-core kernels has no address");
  a.out = p->out; a.scale = p->scale; a.shift = p->shift; a.res = p->res;
  a.out_dtype = p->out_dtype; a.res_dtype = p->res_dtype; a.act = p->act; a.alpha = p->alpha;
  a.M = M; a.N = p->f; a.K = K; a.o_sm = p->f; a.r_sm = p->f; a.r_sn = 1; a.b1 = 1;
  a.kBlocks = (int)((K + bk - 1) / bk);
  setPlan(a, plan, p->workspace);
  const int ob = p->out_dtype == LLC_FLOAT32 ? 4 : 2;
  a.vecOut = (reinterpret_cast<uintptr_t>(p->out) % (ob * 4)) == 0 && p->f % 4 == 0;
  a.x = p->x; a.H = (int)p->h; a.W = (int)p->w_in; a.C = (int)p->c; a.KH = (int)p->kh; a.KW = (int)p->kw; a.OH = (int)p->oh; a.OW = (int)p->ow;
  a.sh = p->stride_h; a.sw = p->stride_w; a.ph = p->pad_h; a.pw = p->pad_w; a.dh = p->dil_h; a.dw = p->dil_w;
  {
    const bool dense = p->x_sn == 0 && p->x_sh == 0 && p->x_sw == 0;
    a.xs_w = dense ? p->c : p->x_sw; a.xs_h = dense ? p->w_in * p->c : p->x_sh; a.xs_n = dense ? p->h * p->w_in * p->c : p->x_sn;
  }
  CUtensorMap mo = mb;
  if (tmaEpilogueEnabled() && makeOutMap(&mo, p->out, ob == 4, p->f, M, 1, 1, p->f, 0, 0, kOutBoxBytes)) a.tmaOut = kOutBoxBytes;
  a.resTile = p->res && p->res_dtype == p->out_dtype && (reinterpret_cast<uintptr_t>(p->res) & 15) == 0 && (p->f * ob) % 16 == 0;
  CUtensorMap mbl = mb;
  if (kind == 2 && p->w_lo && (reinterpret_cast<uintptr_t>(p->w_lo) & 15) == 0 && makeMap(&mbl, p->w_lo, f32, K, p->f, 1, 1, K, 0, 0, bn / plan.cg)) a.hasBLo = 1;
  if (im2col) {
    CUtensorMap mr = mo;
    bool resRing = false;
    if (a.resTile && a.tmaOut && !plan.cut && kind != 2 && resRingEnabled()) {
      bool h1 = false, h0 = false;
      if (makeResMap(&mr, p->res, ob == 4, p->f, M, 1, 1, p->f, 0, 0, &h1, &h0)) resRing = true;
    }
    const TcMaps maps{ma, mb, mo, mbl, mr};
    return kind == 0 ? dispatchTc<2, 0>(plan, resRing, maps, a, 1, st) : kind == 1 ? dispatchTc<2, 1>(plan, resRing, maps, a, 1, st) : dispatchTc<2, 2>(plan, false, maps, a, 1, st);
  }
  const TcMaps maps{mb, mb, mo, mbl, mo};
  return kind == 0 ? dispatchTc<1, 0>(plan, false, maps, a, 1, st) : kind == 1 ? dispatchTc<1, 1>(plan, false, maps, a, 1, st) : dispatchTc<1, 2>(plan, false, maps, a, 1, st);
}

// Reads and clears the status word the bounded waits write (0 = no wait ever gave up).
int tcStatus() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_tcStatus, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_tcStatus, &zero, sizeof(int));
  return v;
}

}  // namespace llc
