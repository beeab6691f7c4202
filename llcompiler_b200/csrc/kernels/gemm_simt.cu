// FMA (CUDA-core) GEMM for problems of few tiles: the fp32-exact path (precision "fp32") of llc_cuda_gemm and the fallback for
// shapes the tensor-core kernels do not take, fp32 or bf16 operands, fp32 accumulation.  igemm_simt.cu has the one for the
// others and asks this one first (clusterGemm).
//
// A CTA of 256 threads computes a BM x BN tile over a slice of K; up to eight CTAs along K form a cluster, meet in
// distributed shared memory (each adds up one slice of the rows, the partial tiles in K order, so results are
// bit-reproducible) and run the epilogue on it: no scratch in global memory, no counters, no second launch.  K is walked in
// blocks of 32, fetched a block ahead into registers and stored k-major in one of two shared buffers, so that a thread
// reads its fragments as float4 and one barrier per block is enough.
// Bound: latency (a CTA alone on its SM needs 62 ns per k where the FMAs take 33), which is why the K loop is cut.  Against
// igemm_simt_kernel (us a launch, back to back): 64 x 512 x 784 14.5 -> 11.2, 64 x 10 x 512 15.2 -> 6.5, 1021 x 512 x 784
// 45.5 -> 36.9, 2048 x 2048 x 256 114 -> 86.
#include "common.cuh"

namespace llc {
namespace {

struct SimtArgs {
  const void* a; const void* b; void* out; const float* scale; const float* shift; const void* res;
  int out_dtype, res_dtype, act; float alpha;
  long long M, N, K;
  long long a_s0, a_s1, a_sm, b_s0, b_s1, b_sk, b_sn, o_s0, o_s1, o_sm, r_s0, r_s1, r_sm, r_sn;
  int b1; int vecOut;
  int slices; long long kPer;      // CTAs along K (= cluster size along z) and the length of their slices
};

constexpr int BK = 32;

__device__ __forceinline__ void clusterBarrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Four floats at the same place of another CTA of the cluster (clusters extend along z only, so z is the rank).
__device__ __forceinline__ float4 loadPeer4(const float* p, uint32_t rank) {
  float4 v; uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

template <int BM, int BN> struct SimtSmem {
  static constexpr int kStride = BM + 4, kStrideB = BN + 4;
  static constexpr int kTiles = 2 * BK * (kStride + kStrideB) * 4, kPartial = BM * BN * 4;
  static constexpr int kBytes = kTiles > kPartial ? kTiles : kPartial;
};

// Threads form a 16 x 16 grid; a thread owns (BM / 16) x (BN / 16) results in groups of four rows and four columns.
template <typename T, int BM, int BN, bool VEC>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const __grid_constant__ SimtArgs p) {
  constexpr int TM = BM / 16, TN = BN / 16;
  constexpr int kB4 = BN * BK / 4;                             // float4 loads of a K block of B (fewer than there are threads for 16 columns)
  constexpr int AV = BM * BK / 1024, BV = (kB4 + 255) / 256;   // float4 loads per thread and K block
  constexpr int AS = SimtSmem<BM, BN>::kStride, BS = SimtSmem<BM, BN>::kStrideB;
  extern __shared__ __align__(16) float smem[];
  float* const As = smem;                                      // [2][BK][AS]
  float* const Bs = smem + 2 * BK * AS;                        // [2][BK][BS]

  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long long m0 = (long long)blockIdx.x * BM, n0 = (long long)blockIdx.y * BN;
  const int kz = (int)(blockIdx.z % (unsigned)p.slices), z = (int)(blockIdx.z / (unsigned)p.slices), zb0 = z / p.b1, zb1 = z % p.b1;
  const long long kBeg = (long long)kz * p.kPer;
  const long long kEnd = kBeg + p.kPer < p.K ? kBeg + p.kPer : p.K;
  const T* A = reinterpret_cast<const T*>(p.a) + zb0 * p.a_s0 + zb1 * p.a_s1;
  const T* B = reinterpret_cast<const T*>(p.b) + zb0 * p.b_s0 + zb1 * p.b_s1;
  const bool bKMajor = p.b_sk == 1;

  float4 ra[AV], rb[BV];
  // four consecutive k of one row (zeros past the slice's end or the matrix's last row)
  auto load4k = [&](const T* base, long long row, long long rows, long long stride, long long kStride, long long k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows) {
      const T* src = base + row * stride + k * kStride;
      if (VEC) { if (k < kEnd) v = Vec4<T>::load(src); }
      else {
        if (k < kEnd) v.x = toFloat<T>(src[0]);
        if (k + 1 < kEnd) v.y = toFloat<T>(src[kStride]);
        if (k + 2 < kEnd) v.z = toFloat<T>(src[2 * kStride]);
        if (k + 3 < kEnd) v.w = toFloat<T>(src[3 * kStride]);
      }
    }
    return v;
  };
  // Neighbouring lanes take neighbouring rows: their transposing stores hit different banks, and the 16-byte reads of one
  // row's 128 bytes come close enough together to share its sectors in L1.
  auto loadTile = [&](long long k0) {
#pragma unroll
    for (int i = 0; i < AV; ++i) { const int e = tid + i * 256; ra[i] = load4k(A, m0 + e % BM, p.M, p.a_sm, 1, k0 + e / BM * 4); }
    if (VEC && !bKMajor) {                                      // B rows along n: four columns of one k
#pragma unroll
      for (int i = 0; i < BV; ++i) {
        const int e = tid + i * 256;
        const long long k = k0 + e / (BN / 4), n = n0 + e % (BN / 4) * 4;
        rb[i] = (e < kB4 && n < p.N && k < kEnd) ? Vec4<T>::load(B + k * p.b_sk + n) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    } else {
#pragma unroll
      for (int i = 0; i < BV; ++i) { const int e = tid + i * 256; if (e < kB4) rb[i] = load4k(B, n0 + e % BN, p.N, p.b_sn, p.b_sk, k0 + e / BN * 4); }
    }
  };
  auto storeTile = [&](int buf) {
    float* as = As + buf * BK * AS;
    float* bs = Bs + buf * BK * BS;
#pragma unroll
    for (int i = 0; i < AV; ++i) {
      const int e = tid + i * 256, row = e % BM, k = e / BM * 4;
      as[k * AS + row] = ra[i].x; as[(k + 1) * AS + row] = ra[i].y; as[(k + 2) * AS + row] = ra[i].z; as[(k + 3) * AS + row] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < BV; ++i) {
      const int e = tid + i * 256;
      if (e >= kB4) continue;
      if (VEC && !bKMajor) *reinterpret_cast<float4*>(bs + e / (BN / 4) * BS + e % (BN / 4) * 4) = rb[i];
      else {
        const int row = e % BN, k = e / BN * 4;
        bs[k * BS + row] = rb[i].x; bs[(k + 1) * BS + row] = rb[i].y; bs[(k + 2) * BS + row] = rb[i].z; bs[(k + 3) * BS + row] = rb[i].w;
      }
    }
  };
  // fragment of T values: rows (columns) g * 64 + 4 * t .. + 3; a tile of 16 or 32 columns gives a thread 1 or 2
  auto fragment = [&](const float* row, int t, auto& v) {
    constexpr int W = sizeof(v) / sizeof(float);
    if constexpr (W >= 4) {
#pragma unroll
      for (int g = 0; g < W / 4; ++g) {
        const float4 f = *reinterpret_cast<const float4*>(row + g * 64 + t * 4);
        v[4 * g] = f.x; v[4 * g + 1] = f.y; v[4 * g + 2] = f.z; v[4 * g + 3] = f.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < W; ++j) v[j] = row[t * W + j];
    }
  };

  // Sums of 128 products are added up in `total`: the K slices of problems with few tiles have always been that short, and
  // one sum over an eighth of K was off by twice as much (64 x 10 x 25088: 1.0e-6 of the result against 5.1e-7).  128 x 128
  // tiles, which have no registers for it, are never cut into longer slices than igemm_simt_kernel would cut them into.
  constexpr bool kShortSums = TM * TN <= 16;
  constexpr int kSumBlocks = 128 / BK;
  float acc[TM][TN], total[kShortSums ? TM : 1][kShortSums ? TN : 1];
  auto closeSums = [&](bool last) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        if (last) acc[i][j] += total[i][j];
        else { total[i][j] += acc[i][j]; acc[i][j] = 0.f; }
      }
  };
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) { acc[i][j] = 0.f; if constexpr (kShortSums) total[i][j] = 0.f; }

  const int nk = kEnd > kBeg ? (int)((kEnd - kBeg + BK - 1) / BK) : 0;
  if (nk > 0) { loadTile(kBeg); storeTile(0); }
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int buf = kt & 1;
    if (kt + 1 < nk) loadTile(kBeg + (long long)(kt + 1) * BK);
    const float* as = As + buf * BK * AS;
    const float* bs = Bs + buf * BK * BS;
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
      fragment(as + kk * AS, ty, a);
      fragment(bs + kk * BS, tx, b);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (kt + 1 < nk) {
      storeTile(buf ^ 1);
      if constexpr (kShortSums) { if (kt % kSumBlocks == kSumBlocks - 1) closeSums(false); }
    }
    __syncthreads();
  }

  if constexpr (kShortSums) closeSums(true);

  // The partial (or whole) tile goes through shared memory, so that the epilogue works on whole rows.
  auto rowOf = [&](int i) { return (i >> 2) * 64 + ty * 4 + (i & 3); };
  auto colOf = [&](int j) { return TN >= 4 ? (j >> 2) * 64 + tx * 4 + (j & 3) : tx * TN + j; };
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    float* row = smem + rowOf(i) * BN;
    if constexpr (TN >= 4) {
#pragma unroll
      for (int j = 0; j < TN; j += 4) *reinterpret_cast<float4*>(row + colOf(j)) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < TN; ++j) row[colOf(j)] = acc[i][j];
    }
  }
  const bool split = p.slices > 1;
  if (split) clusterBarrier(); else __syncthreads();

  // epilogue of this CTA's share of the rows: alpha * scale[n] * sum + shift[n] + res, activation, store
  const int rowsPer = BM / p.slices, r0 = kz * rowsPer;
  const long long oOff = zb0 * p.o_s0 + zb1 * p.o_s1, rOff = zb0 * p.r_s0 + zb1 * p.r_s1;
  for (int e = tid; e < rowsPer * (BN / 4); e += 256) {
    const int row = r0 + e / (BN / 4), col = e % (BN / 4) * 4;
    const long long gm = m0 + row, gn = n0 + col;
    if (gm >= p.M || gn >= p.N) continue;
    const float* src = smem + row * BN + col;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (split) {
      for (int q0 = 0; q0 < p.slices; q0 += 2) {                // (two to eight slices, a power of two)
        const float4 x = loadPeer4(src, (uint32_t)q0), y = loadPeer4(src, (uint32_t)q0 + 1);
        s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
        s.x += y.x; s.y += y.y; s.z += y.z; s.w += y.w;
      }
    } else s = *reinterpret_cast<const float4*>(src);
    float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const long long n = gn + j;
      float x = v[j] * p.alpha;
      if (n < p.N) {
        if (p.scale) x *= p.scale[n];
        if (p.shift) x += p.shift[n];
        if (p.res) x += loadAs(p.res, rOff + gm * p.r_sm + n * p.r_sn, p.res_dtype);
      }
      v[j] = applyAct(x, p.act);
    }
    const long long o = oOff + gm * p.o_sm + gn;
    if (p.vecOut && gn + 3 < p.N) {
      if (p.out_dtype == LLC_FLOAT32) Vec4<float>::store(reinterpret_cast<float*>(p.out) + o, make_float4(v[0], v[1], v[2], v[3]));
      else Vec4<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(p.out) + o, make_float4(v[0], v[1], v[2], v[3]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) if (gn + j < p.N) storeAs(p.out, o + j, p.out_dtype, v[j]);
    }
  }
  if (split) clusterBarrier();                                   // no CTA leaves while another reads its partial tile
}

// Tile and number of K slices by estimated time, us: a constant for the launch and the epilogue, and K of a slice times what a k
// takes on an SM that holds `c` CTAs (measured; from four on the CTAs' L1 is too small for the rows they read 16 bytes at a
// time).  Clusters do not fill the chip: of four CTAs 33 run at once, of eight 14.  Rows that cannot be read as vectors
// take 15 % longer (10 % in the other kernel).  Over 234 shapes (1 to 4096 rows, 8 to 4096 columns, K 32 to 30000) the two
// kernels chosen so take 0.71 of what igemm_simt_kernel takes alone, geometric mean, and no shape more than 1.08.  (The first choice of tiles counted no
// neighbours on an SM: 4096 x 512 x 784 105 -> 190 us, 64 x 10 x 25088 46 -> 110.)
struct SimtPlan { int bn, slices; float us; };   // bn 128: 128 x 128 tiles, otherwise 64 x bn
SimtPlan choosePlan(long long M, long long N, long long K, long long batch, bool vec) {
  static const struct { int bm, bn; float fixedUs, perK; } tiles[] = {{64, 16, 4.f, 0.0345f}, {64, 64, 4.f, 0.0625f}, {128, 128, 10.f, 0.131f}};
  SimtPlan best{0, 0, 0.f};
  for (const auto& t : tiles) {
    if (t.bn == 16 ? N > 64 : t.bn == 128 && (M <= 64 || N <= 64)) continue;
    const long long nTiles = (N + t.bn - 1) / t.bn, n = (M + t.bm - 1) / t.bm * nTiles * batch;
    if (nTiles > 65535) continue;                        // (the grid's y extent)
    for (int s = 1; s <= 8; s *= 2) {
      if (s > 1 && (K / s < BK || n * s > 2 * kNumSMs || batch * s > 65535)) break;
      const long long atOnce = s == 8 ? 112 : s == 4 ? 132 : kNumSMs, per = t.bn == 128 ? atOnce : kNumSMs, sms = (n * s + per - 1) / per;
      const float c = n * s <= atOnce ? 1.f : sms < 2 ? 2.f : (float)sms;
      const float share = c == 1.f ? 1.f : t.bn == 16 ? 0.95f * c : t.bn == 128 ? c : c == 2.f ? (sms < 2 ? 1.4f : 1.6f) : c == 3.f ? 2.3f : 1.1f * c;
      const float us = t.fixedUs + (s > 1 ? 0.7f : 0.f) + (float)((K + s - 1) / s) * t.perK * share * (vec ? 1.f : 1.15f);
      if (!best.bn || us < best.us) best = SimtPlan{t.bn, s, us};
    }
  }
  return best;
}

template <typename T, int BM, int BN, bool VEC> int launchTile(const SimtArgs& a, long long batch, cudaStream_t st) {
  constexpr int kBytes = SimtSmem<BM, BN>::kBytes;
  auto kernel = gemm_simt_kernel<T, BM, BN, VEC>;
  if (kBytes > 48 * 1024) {
    static DeviceOnce configured;                          // the shared-memory opt-in is kept per device
    const int dev = currentDevice();
    if (!configured.test(dev)) {
      LLC_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes));
      configured.set(dev);
    }
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((a.M + BM - 1) / BM), (unsigned)((a.N + BN - 1) / BN), (unsigned)(batch * a.slices));
  cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = kBytes; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = (unsigned)a.slices;
  cfg.attrs = attr; cfg.numAttrs = a.slices > 1 ? 1 : 0;
  LLC_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, a));
  return LLC_OK;
}

template <typename T, bool VEC> int launchGemm(SimtArgs a, const SimtPlan& plan, long long batch, cudaStream_t st) {
  a.slices = plan.slices;
  a.kPer = (((a.K + plan.slices - 1) / plan.slices) + 3) / 4 * 4;
  if (plan.bn == 128) return launchTile<T, 128, 128, VEC>(a, batch, st);
  return plan.bn == 64 ? launchTile<T, 64, 64, VEC>(a, batch, st) : launchTile<T, 64, 16, VEC>(a, batch, st);
}

bool aligned(const void* p, int bytes) { return (reinterpret_cast<uintptr_t>(p) % bytes) == 0; }

}  // namespace

// Runs the GEMM (arguments checked by the caller, nothing empty) if it is done clearly before `otherUs`; *taken tells.
int clusterGemm(const LlcGemmParams* p, float otherUs, cudaStream_t st, bool* taken) {
  *taken = false;
  const int eb = p->in_dtype == LLC_FLOAT32 ? 4 : 2, ob = p->out_dtype == LLC_FLOAT32 ? 4 : 2;
  const bool vec = p->k % 4 == 0 && p->a_sm % 4 == 0 && p->a_s0 % 4 == 0 && p->a_s1 % 4 == 0 && aligned(p->a, eb * 4) && aligned(p->b, eb * 4) &&
                   p->b_s0 % 4 == 0 && p->b_s1 % 4 == 0 && (p->b_sk == 1 ? p->b_sn % 4 == 0 : (p->n % 4 == 0 && p->b_sk % 4 == 0));
  const long long batch = p->b0 * p->b1;
  if ((p->b_sk != 1 && p->b_sn != 1) || batch > 65535) return LLC_OK;      // (what the caller refuses)
  const SimtPlan plan = choosePlan(p->m, p->n, p->k, batch, vec);
  if (!plan.bn || plan.us >= 0.95f * otherUs * (vec ? 1.f : 1.1f)) return LLC_OK;
  SimtArgs a{};
  a.a = p->a; a.b = p->b; a.out = p->out; a.scale = p->scale; a.shift = p->shift; a.res = p->res;
  a.out_dtype = p->out_dtype; a.res_dtype = p->res_dtype; a.act = p->act; a.alpha = p->alpha;
  a.M = p->m; a.N = p->n; a.K = p->k;
  a.a_s0 = p->a_s0; a.a_s1 = p->a_s1; a.a_sm = p->a_sm;
  a.b_s0 = p->b_s0; a.b_s1 = p->b_s1; a.b_sk = p->b_sk; a.b_sn = p->b_sn;
  a.o_s0 = p->o_s0; a.o_s1 = p->o_s1; a.o_sm = p->o_sm;
  a.r_s0 = p->r_s0; a.r_s1 = p->r_s1; a.r_sm = p->r_sm; a.r_sn = p->r_sn;
  a.b1 = (int)p->b1;
  a.vecOut = aligned(p->out, ob * 4) && p->o_sm % 4 == 0 && p->o_s0 % 4 == 0 && p->o_s1 % 4 == 0;
  *taken = true;
  if (p->in_dtype == LLC_FLOAT32) return vec ? launchGemm<float, true>(a, plan, batch, st) : launchGemm<float, false>(a, plan, batch, st);
  return vec ? launchGemm<__nv_bfloat16, true>(a, plan, batch, st) : launchGemm<__nv_bfloat16, false>(a, plan, batch, st);
}

}  // namespace llc
