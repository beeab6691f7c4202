// Elementwise chains: the kernels behind llc_cuda_eltwise for programs in chain form (eltwise_prog.cuh).
//   chain_rows_kernel   every operand dense or broadcast along the output's innermost dim: eight or sixteen elements per
//                       thread in 16-byte pieces, no division for two dims or fewer.
//   chain_tile_kernel   at least one operand is dense along another dim than the output (an NHWC activation read by a step
//                       that writes NCHW, or the other way round): 64 x 64 tiles of that operand go through shared memory.
// Bound: HBM.  Algorithmic bytes: every operand element once, the output once.  Against the general kernels, which these
// programs went to before (CUDA events, one B200): NHWC + NCHW -> ReLU -> NCHW on 256x512x28x28 bf16 1.018 -> 0.140 ms
// (4.4 TB/s), NHWC -> NCHW copy of 256x64x56x56 bf16 0.396 -> 0.045 ms (4.5), NCHW -> NHWC of 256x512x28x28 0.259 ->
// 0.099 ms (4.2), `a + b[row]` on 98304 x 768 bf16 0.113 -> 0.062 ms (4.9).
#include "eltwise_prog.cuh"

namespace llc {
namespace elt {
namespace {

// V neighbouring elements (along the output's innermost dim) of a dense, strided or broadcast operand, in two halves:
// loadRaw only requests them, unpack turns them into floats.  A conversion right behind its load would make the loads of a
// thread wait for one another (`a + b[row]` on 98304 x 768 bf16: 0.123 ms that way).  Operands whose offsets are multiples
// of V elements and whose base is aligned take the vector form (`vec`).
template <int V> struct Raw { uint32_t w[V]; };
template <int V> __device__ __forceinline__ void loadRaw(const void* base, int dt, long long off, long long stride, bool vec, Raw<V>& r) {
  if constexpr (V >= 4) {
    if (vec && stride == 1 && dt == LLC_BFLOAT16) {
      const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(base) + off;
      if constexpr (V == 8) { const uint4 q = __ldg(reinterpret_cast<const uint4*>(p)); r.w[0] = q.x; r.w[1] = q.y; r.w[2] = q.z; r.w[3] = q.w; }
      else { const uint2 q = __ldg(reinterpret_cast<const uint2*>(p)); r.w[0] = q.x; r.w[1] = q.y; }
      return;
    }
    if (vec && stride == 1 && dt == LLC_FLOAT32) {
      const float* p = reinterpret_cast<const float*>(base) + off;
#pragma unroll
      for (int h = 0; h < V / 4; ++h) { const uint4 q = __ldg(reinterpret_cast<const uint4*>(p) + h); r.w[4 * h] = q.x; r.w[4 * h + 1] = q.y; r.w[4 * h + 2] = q.z; r.w[4 * h + 3] = q.w; }
      return;
    }
  }
  if (stride == 0) {
    r.w[0] = __float_as_uint(loadAs(base, off, dt));
    return;
  }
#pragma unroll
  for (int e = 0; e < V; ++e) r.w[e] = __float_as_uint(loadAs(base, off + e * stride, dt));
}
template <int V> __device__ __forceinline__ void unpack(const Raw<V>& r, int dt, long long stride, bool vec, float* v) {
  if (stride == 0) {
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = __uint_as_float(r.w[0]);
  } else if (V >= 4 && vec && stride == 1 && dt == LLC_BFLOAT16) {
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = __uint_as_float((e & 1) ? r.w[e / 2] & 0xffff0000u : r.w[e / 2] << 16);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e) v[e] = __uint_as_float(r.w[e]);
  }
}
template <int V> __device__ __forceinline__ void storeResult(void* base, int dt, long long off, const float* v) {
  if constexpr (V >= 4) {                       // the launcher gives V > 1 to f32 and bf16 outputs only
    if (dt == LLC_FLOAT32) {
      float* p = reinterpret_cast<float*>(base) + off;
#pragma unroll
      for (int e = 0; e < V; e += 4) Vec4<float>::store(p + e, make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]));
    } else if constexpr (V == 8) {
      uint4 q; __nv_bfloat162 h;
      h = __floats2bfloat162_rn(v[0], v[1]); q.x = *reinterpret_cast<unsigned*>(&h); h = __floats2bfloat162_rn(v[2], v[3]); q.y = *reinterpret_cast<unsigned*>(&h);
      h = __floats2bfloat162_rn(v[4], v[5]); q.z = *reinterpret_cast<unsigned*>(&h); h = __floats2bfloat162_rn(v[6], v[7]); q.w = *reinterpret_cast<unsigned*>(&h);
      *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(base) + off) = q;
    } else {
      Vec4<__nv_bfloat16>::store(reinterpret_cast<__nv_bfloat16*>(base) + off, make_float4(v[0], v[1], v[2], v[3]));
    }
  } else {
    storeAs(base, off, dt, v[0]);
  }
}

// The operands in the order the chain consumes them ("slots": an operand that is read twice has two), so that a kernel
// knows at compile time which registers a step reads; picking them by index at run time cost more than the arithmetic
// (`a + b[row]` on 98304 x 768 bf16: 0.151 ms that way, 0.123 ms with slots, before the loads were taken apart as above).
constexpr int kMaxSlots = 3;
struct SlotArgs {
  void* out; int odt; int rank; long long total;
  long long shape[kMaxRank], ostr[kMaxRank];
  const void* in[kMaxSlots]; int idt[kMaxSlots]; long long istr[kMaxSlots][kMaxRank];
  EltChain c;
};

// The programs most large steps consist of have kernels of their own: the general chain's branches and the calls behind
// them made the kernels wait for instructions (NHWC + NCHW -> ReLU -> NCHW on 256x512x28x28 bf16: issue slots 77 % busy).
// P_ONE: one step of any kind, its op decoded once per thread and inline (as a chain of one step, with a call per element for
// the transcendental ops, 64 x 512 bf16 GELU took 5.1 us where it had taken 3.2, a division 4.6 for 2.6).
enum ChainProg { P_CHAIN = 0, P_COPY, P_ADD, P_ADD_RELU, P_ONE };

// acc = op(acc, y) (or op(y, acc) when `swap`) for E elements.
template <int E> __device__ __forceinline__ void oneStep(int op, float* acc, const float* y, bool swap) {
  float a[E], b[E];
#pragma unroll
  for (int e = 0; e < E; ++e) { a[e] = swap ? y[e] : acc[e]; b[e] = swap ? acc[e] : y[e]; }
  switch (op) {
#define LLC_ONE(OP) case OP: _Pragma("unroll") for (int e = 0; e < E; ++e) acc[e] = evalOp(OP, a[e], b[e], 0.f, 0.f); break;
    LLC_ONE(E_ADD) LLC_ONE(E_SUB) LLC_ONE(E_MUL) LLC_ONE(E_DIV) LLC_ONE(E_MAX) LLC_ONE(E_MIN) LLC_ONE(E_POW) LLC_ONE(E_RELU) LLC_ONE(E_ABS) LLC_ONE(E_SQRT)
    LLC_ONE(E_RSQRT) LLC_ONE(E_EXP) LLC_ONE(E_GELU) LLC_ONE(E_TANH) LLC_ONE(E_ERF) LLC_ONE(E_SIGMOID) LLC_ONE(E_NEG) LLC_ONE(E_TRUNC) LLC_ONE(E_TF32LO)
    LLC_ONE(E_EQ) LLC_ONE(E_NE) LLC_ONE(E_GE) LLC_ONE(E_GT) LLC_ONE(E_LE) LLC_ONE(E_LT)
#undef LLC_ONE
    default: break;                              // E_CAST
  }
}

// Runs the chain on E elements; v[j] holds slot j.
template <int PROG, int NIN, int E> __device__ __forceinline__ void runChain(const EltChain& c, float (*v)[E], float* acc) {
  if constexpr (PROG == P_COPY) {
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = v[0][e];
    return;
  }
  if constexpr (PROG == P_ADD || PROG == P_ADD_RELU) {
#pragma unroll
    for (int e = 0; e < E; ++e) { const float x = v[0][e] + v[1][e]; acc[e] = PROG == P_ADD ? x : fmaxf(x, 0.f); }
    return;
  }
  if constexpr (PROG == P_ONE) {                 // the operand is the other slot, a constant or the value itself
    float y[E];
#pragma unroll
    for (int e = 0; e < E; ++e) { acc[e] = v[0][e]; y[e] = NIN == 2 ? v[NIN - 1][e] : c.src[0] == C_IMM ? c.imm[0] : v[0][e]; }
    oneStep<E>(c.op[0], acc, y, c.swap[0] != 0);
    return;
  }
  int s = 0;
  auto plain = [&]() {                           // a step whose operand is a constant, the running value or nothing
    if (c.src[s] == C_SELF) {
      float y[E];
#pragma unroll
      for (int e = 0; e < E; ++e) y[e] = acc[e];
      chainStep<E>(c.op[s], acc, y, c.swap[s] != 0);
    } else {
      float y[E];
#pragma unroll
      for (int e = 0; e < E; ++e) y[e] = c.imm[s];
      chainStep<E>(c.op[s], acc, y, c.swap[s] != 0);
    }
    ++s;
  };
  int j0 = 0;
  if (c.startSrc == C_INPUT) {
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = v[0][e];
    j0 = 1;
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = c.startImm;
  }
#pragma unroll
  for (int j = 0; j < NIN; ++j) {
    if (j < j0) continue;
    while (c.src[s] != C_INPUT) plain();
    chainStep<E>(c.op[s], acc, v[j], c.swap[s] != 0);
    ++s;
  }
  while (s < c.n) plain();
}

struct RowsArgs {
  SlotArgs e;
  int pieces; long long rows;      // two dims or fewer: rows x pieces of eight elements
};

// TWO: at most two dims - a block is blockDim.y rows by one part of a row, no thread divides.  Otherwise the linear piece
// index is decomposed over the dims.  A thread takes U pieces: two, so that twice the loads are in flight, or one where two
// would leave SMs without a block (rowPieces).
template <bool TWO, int U, int PROG, int NIN>
__global__ void __launch_bounds__(256, NIN == 3 ? 3 : NIN == 2 || PROG == P_ONE ? 4 : 6) chain_rows_kernel(const __grid_constant__ RowsArgs p) {
  const SlotArgs& e = p.e;
  const int last = e.rank - 1;
  long long oOff[U], iOff[U][NIN];
  bool in[U];
  if constexpr (TWO) {
    const int part = (int)blockIdx.y;
    const long long row = (long long)blockIdx.x * blockDim.y + threadIdx.y;
    if (row >= p.rows) return;
    const bool two = e.rank == 2;
    const long long oRow = two ? row * e.ostr[0] : 0;
    long long iRow[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) iRow[k] = two ? row * e.istr[k][0] : 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int piece = (part * U + u) * (int)blockDim.x + (int)threadIdx.x;
      in[u] = piece < p.pieces;
      const long long col = (long long)(in[u] ? piece : 0) * 8;
      oOff[u] = col + oRow;
#pragma unroll
      for (int k = 0; k < NIN; ++k) iOff[u][k] = iRow[k] + (e.istr[k][last] ? col : 0);
    }
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long piece = ((long long)blockIdx.x * U + u) * 256 + threadIdx.x;
      in[u] = piece * 8 < e.total;
      long long rem = in[u] ? piece * 8 : 0;
      oOff[u] = 0;
#pragma unroll
      for (int k = 0; k < NIN; ++k) iOff[u][k] = 0;
      for (int d = last; d >= 0; --d) {
        const unsigned long long ext = (unsigned long long)e.shape[d];
        long long c;
        if ((unsigned long long)rem < (1ull << 32) && ext < (1ull << 32)) { const unsigned q = (unsigned)rem / (unsigned)ext; c = (unsigned)rem - q * (unsigned)ext; rem = q; }
        else { const long long q = rem / (long long)ext; c = rem - q * (long long)ext; rem = q; }
        oOff[u] += c * e.ostr[d];
#pragma unroll
        for (int k = 0; k < NIN; ++k) iOff[u][k] += c * e.istr[k][d];
      }
    }
  }
  Raw<8> raw[NIN][U];
#pragma unroll
  for (int k = 0; k < NIN; ++k)
#pragma unroll
    for (int u = 0; u < U; ++u) loadRaw<8>(e.in[k], e.idt[k], iOff[u][k], e.istr[k][last], true, raw[k][u]);
  // one piece at a time from here on: the floats of both would take registers that more resident blocks make better use of
#pragma unroll
  for (int u = 0; u < U; ++u) {
    float v[NIN][8], acc[8];
#pragma unroll
    for (int k = 0; k < NIN; ++k) unpack<8>(raw[k][u], e.idt[k], e.istr[k][last], true, v[k]);
    runChain<PROG, NIN, 8>(e.c, v, acc);
    if (in[u]) storeResult<8>(e.out, e.odt, oOff[u], acc);
  }
}

// ---- transposing tiles ---------------------------------------------------------------------------
constexpr int kT = 64;                           // tile: 64 positions of the output's innermost dim (p) x 64 of the operand's (c)
struct TileArgs {
  SlotArgs e;
  int cDim; unsigned tilesP;                     // blockIdx.x: outer index * tilesP + tile along p; blockIdx.y: tile along c
  int oC, iP[kMaxSlots], iC[kMaxSlots];          // strides inside a tile (64 steps of any of them stay below 2^31)
  int tileOf[kMaxSlots];                         // which shared-memory tile a slot reads, -1: straight from memory
  int first[2]; int nT;                          // the slot each tile is filled from
  int vin;                                       // tiles are filled with 16-byte reads along c
};

// ES: bytes per element of the transposed operands.  V: elements per thread along p for the other operands and the output.
// A tile row is 128 (2-byte types) or 256 (fp32) bytes in both directions, whole sectors either way.  In shared memory a
// row is one c: 64 p positions plus one word, which leaves the transposing writes and the reads without bank conflicts;
// 2-byte elements are paired along p so that every access is a word.  The operands that need no transposing are requested
// before the tiles are filled.  (The fp32 variants of three operands spill 140 bytes at three blocks per SM; at two, without
// spills, 32 x 512 x 28 x 28 took 55 us for 48.)
template <int ES, int V, int PROG, int NIN>
__global__ void __launch_bounds__(256, NIN == 1 ? 5 : NIN == 2 ? 4 : 3) chain_tile_kernel(const __grid_constant__ TileArgs p) {
  constexpr int kWords = kT * ES / 4, kRow = kWords + 1;
  extern __shared__ uint32_t tiles[];            // nT x [64][kRow]
  const SlotArgs& e = p.e;
  const int last = e.rank - 1;
  unsigned t = blockIdx.x / p.tilesP;
  const unsigned tp = blockIdx.x - t * p.tilesP;
  const long long p0 = (long long)tp * kT, c0 = (long long)blockIdx.y * kT;
  long long oBase = p0 + c0 * p.oC, iBase[NIN];
#pragma unroll
  for (int k = 0; k < NIN; ++k) iBase[k] = p0 * p.iP[k] + c0 * p.iC[k];
  for (int d = last - 1, left = e.rank - 2; left > 0; --d) {
    if (d == p.cDim) continue;
    unsigned x = t;
    if (--left > 0) { const unsigned q = t / (unsigned)e.shape[d]; x = t - q * (unsigned)e.shape[d]; t = q; }
    oBase += x * e.ostr[d];
#pragma unroll
    for (int k = 0; k < NIN; ++k) iBase[k] += x * e.istr[k][d];
  }
  const int nP = (int)min((long long)kT, e.shape[last] - p0), nC = (int)min((long long)kT, e.shape[p.cDim] - c0);
  constexpr int kPv = kT / V, kItems = kT * kPv / 256;            // pieces of V elements per thread
  constexpr int kBatch = kItems < 8 ? kItems : 8;                 // pieces whose operands are held at a time (one at a time left a chain of sixteen where V is 1)
  auto pieceOf = [&](int i, int& pv, int& c) { const int x = (int)threadIdx.x + i * 256; pv = (x % kPv) * V; c = x / kPv; return pv < nP && c < nC; };
  Raw<V> raw[NIN][kBatch];
  auto fetchDirect = [&](int i0) {
#pragma unroll
    for (int k = 0; k < NIN; ++k) {
      if (p.tileOf[k] >= 0) continue;
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
        int pv, c;
        if (pieceOf(i0 + b, pv, c))
          loadRaw<V>(e.in[k], e.idt[k], iBase[k] + (pv * p.iP[k] + c * p.iC[k]), p.iP[k], true, raw[k][b]);
      }
    }
  };
  fetchDirect(0);
#pragma unroll
  for (int k = 0; k < NIN; ++k) {
    const int m = p.tileOf[k];
    if (m < 0 || p.first[m] != k) continue;
    const int sp = p.iP[k];
    uint32_t* tl = tiles + m * (kT * kRow);
    if constexpr (ES == 2) {
      const uint16_t* src = reinterpret_cast<const uint16_t*>(e.in[k]) + iBase[k];
      if (p.vin) {
        // a thread takes eight c of two neighbouring p; a warp 4 groups of c x 8 pairs of p (conflict-free word writes)
        const int cg = (threadIdx.x & 3) + ((threadIdx.x >> 5) & 1) * 4, pp = ((threadIdx.x >> 2) & 7) + (threadIdx.x >> 6) * 8;
        uint4 a = make_uint4(0, 0, 0, 0), b = a;
        if (cg * 8 < nC) {
          if (2 * pp < nP) a = __ldg(reinterpret_cast<const uint4*>(src + (2 * pp) * sp + cg * 8));
          if (2 * pp + 1 < nP) b = __ldg(reinterpret_cast<const uint4*>(src + (2 * pp + 1) * sp + cg * 8));
        }
        const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          tl[(cg * 8 + 2 * j) * kRow + pp] = __byte_perm(aw[j], bw[j], 0x5410);
          tl[(cg * 8 + 2 * j + 1) * kRow + pp] = __byte_perm(aw[j], bw[j], 0x7632);
        }
      } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < kT * kT / 2; i += 256) {
          const int c = i & 63, pp = i >> 6;
          uint32_t lo = 0, hi = 0;
          if (c < nC) {
            if (2 * pp < nP) lo = src[(2 * pp) * sp + c];
            if (2 * pp + 1 < nP) hi = src[(2 * pp + 1) * sp + c];
          }
          tl[c * kRow + pp] = lo | (hi << 16);
        }
      }
    } else {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(e.in[k]) + iBase[k];
      if (p.vin) {
        uint4 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int cg = (threadIdx.x & 7) + (i & 1) * 8, pq = (threadIdx.x >> 3) + (i >> 1) * 32;
          if (cg * 4 < nC && pq < nP) a[i] = __ldg(reinterpret_cast<const uint4*>(src + pq * sp + cg * 4));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int cg = (threadIdx.x & 7) + (i & 1) * 8, pq = (threadIdx.x >> 3) + (i >> 1) * 32;
          if (cg * 4 < nC && pq < nP) {
            tl[(cg * 4) * kRow + pq] = a[i].x; tl[(cg * 4 + 1) * kRow + pq] = a[i].y; tl[(cg * 4 + 2) * kRow + pq] = a[i].z; tl[(cg * 4 + 3) * kRow + pq] = a[i].w;
          }
        }
      } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < kT * kT; i += 256) {
          const int c = i & 63, pq = i >> 6;
          if (c < nC && pq < nP) tl[c * kRow + pq] = src[pq * sp + c];
        }
      }
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int i0 = 0; i0 < kItems; i0 += kBatch) {
    if (i0 > 0) fetchDirect(i0);
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      int pv, c;
      const bool inside = pieceOf(i0 + b, pv, c);
      float v[NIN][V], acc[V];
#pragma unroll
      for (int k = 0; k < NIN; ++k) {
        if (p.tileOf[k] < 0) { unpack<V>(raw[k][b], e.idt[k], p.iP[k], true, v[k]); continue; }
        const bool half = ES == 2 && e.idt[k] == LLC_FLOAT16;
        const uint32_t* row = tiles + p.tileOf[k] * (kT * kRow) + c * kRow;      // (inside the tile for every thread)
#pragma unroll
        for (int x = 0; x < V; ++x) {
          if constexpr (ES == 4) v[k][x] = __uint_as_float(row[pv + x]);
          else {
            const uint32_t w = row[(pv + x) >> 1];
            const uint32_t h = ((pv + x) & 1) ? w >> 16 : w & 0xffffu;
            v[k][x] = half ? __half2float(__ushort_as_half((unsigned short)h)) : __uint_as_float(h << 16);
          }
        }
      }
      runChain<PROG, NIN, V>(e.c, v, acc);
      if (inside) storeResult<V>(e.out, e.odt, oBase + (pv + c * p.oC), acc);   // (V > 1 only where the extent is a multiple of V)
    }
  }
}

bool isVecType(int dt) { return dt == LLC_FLOAT32 || dt == LLC_BFLOAT16; }
bool alignedTo(const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % (uintptr_t)bytes == 0; }

// The operands of `a` as slots of its chain; false when there are more than the kernels hold.
bool makeSlots(const EltArgs& a, const EltChain& chain, SlotArgs& s, int* nin) {
  s = SlotArgs{};
  s.out = a.out; s.odt = a.odt; s.rank = a.rank; s.total = a.total; s.c = chain;
  for (int d = 0; d < a.rank; ++d) { s.shape[d] = a.shape[d]; s.ostr[d] = a.ostr[d]; }
  int n = 0;
  auto take = [&](int k) {
    if (n == kMaxSlots) return false;
    s.in[n] = a.in[k]; s.idt[n] = a.idt[k];
    for (int d = 0; d < a.rank; ++d) s.istr[n][d] = a.istr[k][d];
    ++n;
    return true;
  };
  if (chain.startSrc == C_INPUT && !take(chain.startIn)) return false;
  for (int i = 0; i < chain.n; ++i) if (chain.src[i] == C_INPUT && !take(chain.in[i])) return false;
  *nin = n;
  return n > 0;
}

ChainProg progOf(const EltChain& c) {
  if (c.startSrc != C_INPUT) return P_CHAIN;
  if (c.n == 0) return P_COPY;
  const bool add = c.op[0] == E_ADD && c.src[0] == C_INPUT;
  if (c.n == 1) return add ? P_ADD : c.op[0] == E_CAST ? P_COPY : P_ONE;
  return add && c.n == 2 && c.op[1] == E_RELU ? P_ADD_RELU : P_CHAIN;
}

// Pieces of eight elements per thread.  Below two blocks of 16 x 256 elements per SM the second piece only lengthens a thread;
// fp32 results, 32 bytes a piece, have enough loads in flight with one for longer.
int rowPieces(long long total, int odt) { return total < (odt == LLC_FLOAT32 ? 6LL : 2LL) * kNumSMs * 256 * 16 ? 1 : 2; }

// Steps that are an instruction or two in a chain as well: on large tensors the chain kernels' smaller register count counts
// for more (98304 x 768 bf16 ReLU 53 against 63 us), on small ones the decoding does (64 x 512 2.3 against 2.0).
bool cheapStep(int op) {
  return op == E_SUB || op == E_MUL || op == E_MAX || op == E_MIN || op == E_RELU || op == E_NEG || op == E_ABS || op == E_TF32LO;
}

template <bool TWO, int U> int launchRows(int nin, const RowsArgs& p, dim3 blocks, dim3 threads, cudaStream_t st) {
  const ChainProg prog = progOf(p.e.c);
  switch (U == 2 && prog == P_ONE && cheapStep(p.e.c.op[0]) ? P_CHAIN : prog) {
    case P_COPY: chain_rows_kernel<TWO, U, P_COPY, 1><<<blocks, threads, 0, st>>>(p); break;
    case P_ADD: chain_rows_kernel<TWO, U, P_ADD, 2><<<blocks, threads, 0, st>>>(p); break;
    case P_ADD_RELU: chain_rows_kernel<TWO, U, P_ADD_RELU, 2><<<blocks, threads, 0, st>>>(p); break;
    case P_ONE:
      if (nin == 1) chain_rows_kernel<TWO, U, P_ONE, 1><<<blocks, threads, 0, st>>>(p);
      else chain_rows_kernel<TWO, U, P_ONE, 2><<<blocks, threads, 0, st>>>(p);
      break;
    default:
      if (nin == 1) chain_rows_kernel<TWO, U, P_CHAIN, 1><<<blocks, threads, 0, st>>>(p);
      else if (nin == 2) chain_rows_kernel<TWO, U, P_CHAIN, 2><<<blocks, threads, 0, st>>>(p);
      else chain_rows_kernel<TWO, U, P_CHAIN, 3><<<blocks, threads, 0, st>>>(p);
  }
  LLC_LAUNCH_CHECK("chain_rows_kernel");
  return LLC_OK;
}
template <int ES, int V> int launchTile(int nin, const TileArgs& t, dim3 blocks, cudaStream_t st) {
  const size_t smem = (size_t)t.nT * kT * (kT * ES / 4 + 1) * 4;
  switch (progOf(t.e.c)) {
    case P_COPY: chain_tile_kernel<ES, V, P_COPY, 1><<<blocks, 256, smem, st>>>(t); break;
    case P_ADD: chain_tile_kernel<ES, V, P_ADD, 2><<<blocks, 256, smem, st>>>(t); break;
    case P_ADD_RELU: chain_tile_kernel<ES, V, P_ADD_RELU, 2><<<blocks, 256, smem, st>>>(t); break;
    default:
      if (nin == 1) chain_tile_kernel<ES, V, P_CHAIN, 1><<<blocks, 256, smem, st>>>(t);
      else if (nin == 2) chain_tile_kernel<ES, V, P_CHAIN, 2><<<blocks, 256, smem, st>>>(t);
      else chain_tile_kernel<ES, V, P_CHAIN, 3><<<blocks, 256, smem, st>>>(t);
  }
  LLC_LAUNCH_CHECK("chain_tile_kernel");
  return LLC_OK;
}

}  // namespace

bool makeChain(const EltProgram& prog, EltChain& c) {
  struct Rev { int op, leaf; bool self, swap; } rev[kMaxChain];
  auto isLeaf = [&](int r) { return prog.op[r] == E_LD || prog.op[r] == E_IMM; };
  auto isUnary = [&](int op) { return op == E_RELU || op == E_ABS || op == E_SQRT || op == E_RSQRT || op == E_EXP || op == E_GELU || op == E_TANH || op == E_ERF ||
                                      op == E_SIGMOID || op == E_NEG || op == E_CAST || op == E_TRUNC || op == E_TF32LO; };
  int cur = prog.n - 1, n = 0;
  while (!isLeaf(cur)) {
    if (n == kMaxChain || prog.op[cur] == E_WHERE) return false;
    const int op = prog.op[cur], a = prog.a[cur], b = prog.b[cur];
    if (isUnary(op)) { rev[n++] = {op, -1, false, false}; cur = a; continue; }
    if (a == b) { rev[n++] = {op, -1, true, false}; cur = a; }
    else if (isLeaf(b)) { rev[n++] = {op, b, false, false}; cur = a; }
    else if (isLeaf(a)) { rev[n++] = {op, a, false, true}; cur = b; }
    else return false;
  }
  c = EltChain{};
  c.startSrc = prog.op[cur] == E_LD ? C_INPUT : C_IMM; c.startIn = prog.a[cur]; c.startImm = prog.imm[cur];
  c.n = n;
  for (int i = 0; i < n; ++i) {
    const Rev& r = rev[n - 1 - i];
    c.op[i] = (unsigned char)r.op; c.swap[i] = r.swap; c.src[i] = r.self ? C_SELF : C_NONE;
    if (r.leaf >= 0) { c.src[i] = prog.op[r.leaf] == E_LD ? C_INPUT : C_IMM; c.in[i] = prog.a[r.leaf]; c.imm[i] = prog.imm[r.leaf]; }
  }
  return true;
}

int launchChain(const EltArgs& a, cudaStream_t st, bool* taken) {
  *taken = false;
  const int r = a.rank, last = r - 1;
  const long long inner = a.shape[last];
  if (a.ostr[last] != 1 && inner != 1) return LLC_OK;
  EltChain chain; SlotArgs e; int nin = 0;
  if (!makeChain(a.prog, chain) || !makeSlots(a, chain, e, &nin)) return LLC_OK;
  // ---- rows: every operand dense (16-byte aligned, eight elements at a time) or broadcast along the innermost dim
  bool rowsOk = inner % 8 == 0 && isVecType(a.odt) && alignedTo(a.out, 16);
  for (int d = 0; d < last && rowsOk; ++d) rowsOk = a.ostr[d] % 8 == 0;
  for (int k = 0; k < nin && rowsOk; ++k) {
    const long long s = e.istr[k][last];
    if (s == 0) continue;
    rowsOk = s == 1;
    if (!isVecType(e.idt[k])) continue;            // other types (an integer mask) are read element by element
    rowsOk = rowsOk && alignedTo(e.in[k], 16);
    for (int d = 0; d < last && rowsOk; ++d) rowsOk = e.istr[k][d] % 8 == 0;
  }
  if (rowsOk) {
    RowsArgs p; p.e = e; p.pieces = 0; p.rows = 1;
    const long long pieces = inner / 8;
    const int u = rowPieces(a.total, a.odt);
    if ((r == 1 || (r == 2 && pieces >= 48)) && pieces <= 0x7FFFFFFFLL / 16) {      // (short rows would leave most of a warp idle)
      // threads along a row: the row's pieces (or pairs of pieces) split into equal parts of at most 256, rounded up to whole warps
      p.rows = r == 2 ? a.shape[0] : 1; p.pieces = (int)pieces;
      const long long pairs = (pieces + u - 1) / u, parts = (pairs + 255) / 256;
      const int tx = (int)((((pairs + parts - 1) / parts) + 31) / 32 * 32);
      const int ty = (int)(256 / tx < 1 ? 1 : (256 / tx < p.rows ? 256 / tx : p.rows));
      const long long blocks = (p.rows + ty - 1) / ty;
      if (blocks <= 0x7FFFFFFFLL && parts <= 65535) {
        *taken = true;
        const dim3 grid((unsigned)blocks, (unsigned)parts), threads((unsigned)tx, (unsigned)ty);
        return u == 1 ? launchRows<true, 1>(nin, p, grid, threads, st) : launchRows<true, 2>(nin, p, grid, threads, st);
      }
    }
    const long long blocks = (a.total / 8 + 256 * u - 1) / (256 * u);
    if (blocks > 0x7FFFFFFFLL) return LLC_OK;
    *taken = true;
    return u == 1 ? launchRows<false, 1>(nin, p, dim3((unsigned)blocks), dim3(256), st) : launchRows<false, 2>(nin, p, dim3((unsigned)blocks), dim3(256), st);
  }
  // ---- tiles: one or two operands dense along one and the same other dim
  TileArgs t; t.cDim = -1; t.nT = 0; t.first[0] = t.first[1] = 0;
  int es = 0;
  for (int k = 0; k < nin; ++k) {
    t.tileOf[k] = -1;
    const long long s = e.istr[k][last];
    if (s == 0 || s == 1) continue;
    int cd = -1;
    for (int d = 0; d < last; ++d) if (e.istr[k][d] == 1 && a.shape[d] > 1) cd = d;
    const int b = e.idt[k] == LLC_FLOAT32 ? 4 : (e.idt[k] == LLC_BFLOAT16 || e.idt[k] == LLC_FLOAT16) ? 2 : 0;
    if (cd < 0 || b == 0) continue;                // a strided operand of another kind is read element by element
    if ((t.cDim >= 0 && t.cDim != cd) || (es && es != b)) return LLC_OK;
    t.cDim = cd; es = b;
    for (int j = 0; j < k; ++j) {                  // the same tensor once more: it shares the tile
      bool same = t.tileOf[j] >= 0 && e.in[j] == e.in[k] && e.idt[j] == e.idt[k];
      for (int d = 0; d < r && same; ++d) same = e.istr[j][d] == e.istr[k][d];
      if (same) t.tileOf[k] = t.tileOf[j];
    }
    if (t.tileOf[k] >= 0) continue;
    if (t.nT == 2) return LLC_OK;
    t.first[t.nT] = k; t.tileOf[k] = t.nT++;
  }
  // Below 32 x 8 a tile is mostly empty and the general kernels read few enough lines per warp.
  if (t.nT == 0 || a.shape[t.cDim] < 32 || inner < 8) return LLC_OK;
  if (!isVecType(a.odt) && a.odt != LLC_FLOAT16) return LLC_OK;
  bool vin = true;
  for (int m = 0; m < t.nT; ++m) {
    const int k = t.first[m], ve = 16 / es;
    vin = vin && alignedTo(e.in[k], 16) && a.shape[t.cDim] % ve == 0;
    for (int d = 0; d < r; ++d) if (d != t.cDim && a.shape[d] > 1) vin = vin && e.istr[k][d] % ve == 0;
  }
  t.vin = vin;
  auto vecOk = [&](int v) {
    bool ok = isVecType(a.odt) && inner % v == 0 && alignedTo(a.out, a.odt == LLC_FLOAT32 ? 16 : 2 * v);
    for (int d = 0; d < last; ++d) if (a.shape[d] > 1) ok = ok && a.ostr[d] % v == 0;
    for (int k = 0; k < nin && ok; ++k) {
      if (t.tileOf[k] >= 0 || e.istr[k][last] != 1 || !isVecType(e.idt[k])) continue;
      ok = alignedTo(e.in[k], e.idt[k] == LLC_FLOAT32 ? 16 : 2 * v);
      for (int d = 0; d < last; ++d) if (a.shape[d] > 1) ok = ok && e.istr[k][d] % v == 0;
    }
    return ok;
  };
  const int v = vecOk(8) ? 8 : vecOk(4) ? 4 : 1;
  const long long tilesP = (inner + kT - 1) / kT, tilesC = (a.shape[t.cDim] + kT - 1) / kT;
  const long long blocksX = tilesP * (a.total / (inner * a.shape[t.cDim])), blocks = blocksX * tilesC;
  if (blocksX > 0x7FFFFFFFLL || tilesC > 65535) return LLC_OK;
  auto inTile = [](long long s) { return s >= 0 && s < (1LL << 24); };
  if (!inTile(a.ostr[t.cDim])) return LLC_OK;
  t.oC = (int)a.ostr[t.cDim];
  for (int k = 0; k < nin; ++k) {
    if (!inTile(e.istr[k][last]) || !inTile(e.istr[k][t.cDim])) return LLC_OK;
    t.iP[k] = (int)e.istr[k][last]; t.iC[k] = (int)e.istr[k][t.cDim];
  }
  // Element-wise tiles (odd extents) take sixteen elements per thread: with less than a tile per SM the general kernel, one
  // element per thread, is done sooner (64 x 41 x 41 bf16, 27 tiles: 8.7 against 10.8 us; 64 x 2048 x 7 x 7: 87 against 25 us).
  if (v == 1 && blocks < kNumSMs) return LLC_OK;
  t.e = e; t.tilesP = (unsigned)tilesP;
  const dim3 grid((unsigned)blocksX, (unsigned)tilesC);
  *taken = true;
  if (es == 2) return v == 8 ? launchTile<2, 8>(nin, t, grid, st) : v == 4 ? launchTile<2, 4>(nin, t, grid, st) : launchTile<2, 1>(nin, t, grid, st);
  return v == 8 ? launchTile<4, 8>(nin, t, grid, st) : v == 4 ? launchTile<4, 4>(nin, t, grid, st) : launchTile<4, 1>(nin, t, grid, st);
}

}  // namespace elt
}  // namespace llc
