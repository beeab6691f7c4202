// The register program of the elementwise kernels and its linear ("chain") form, shared by eltwise.cu and eltwise_chain.cu.
#pragma once
#include "common.cuh"

namespace llc {
namespace elt {

constexpr int kMaxInstr = 48;
constexpr int kMaxRank = 6;
constexpr int kMaxIn = 8;

enum EltOp : int {
  E_LD = 0, E_IMM, E_ADD, E_SUB, E_MUL, E_DIV, E_MAX, E_MIN, E_POW, E_RELU, E_ABS, E_SQRT, E_RSQRT, E_EXP, E_GELU, E_TANH,
  E_ERF, E_SIGMOID, E_NEG, E_CAST, E_TRUNC, E_TF32LO, E_WHERE, E_EQ, E_NE, E_GE, E_GT, E_LE, E_LT
};

struct EltProgram {
  int n;
  unsigned char op[kMaxInstr], a[kMaxInstr], b[kMaxInstr], c[kMaxInstr];
  float imm[kMaxInstr];
};

struct EltArgs {
  void* out; int odt; int rank; int nin;
  long long shape[kMaxRank], ostr[kMaxRank];
  const void* in[kMaxIn]; int idt[kMaxIn]; long long istr[kMaxIn][kMaxRank];
  long long total;      // number of output elements
  int innerVec;         // elements handled per thread along the innermost dim (1 or 4)
  EltProgram prog;
};

__device__ __forceinline__ float evalOp(int op, float x, float y, float z, float imm) {
  switch (op) {
    case E_IMM: return imm;
    case E_ADD: return x + y;
    case E_SUB: return x - y;
    case E_MUL: return x * y;
    case E_DIV: return x / y;
    case E_MAX: return fmaxf(x, y);
    case E_MIN: return fminf(x, y);
    case E_POW: return powf(x, y);
    case E_RELU: return fmaxf(x, 0.f);
    case E_ABS: return fabsf(x);
    case E_SQRT: return sqrtf(x);
    case E_RSQRT: return rsqrtf(x);
    case E_EXP: return expf(x);
    case E_GELU: return geluErf(x);
    case E_TANH: return tanhf(x);
    case E_ERF: return erff(x);
    case E_SIGMOID: return 1.f / (1.f + expf(-x));
    case E_NEG: return -x;
    case E_CAST: return x;
    case E_TRUNC: return truncf(x);
    case E_TF32LO: return x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);   // what a tf32 operand read drops
    case E_WHERE: return x != 0.f ? y : z;
    case E_EQ: return x == y ? 1.f : 0.f;
    case E_NE: return x != y ? 1.f : 0.f;
    case E_GE: return x >= y ? 1.f : 0.f;
    case E_GT: return x > y ? 1.f : 0.f;
    case E_LE: return x <= y ? 1.f : 0.f;
    case E_LT: return x < y ? 1.f : 0.f;
  }
  return 0.f;
}

template <typename T> __device__ __forceinline__ void load8(const T* p, float* v);
template <> __device__ __forceinline__ void load8<float>(const float* p, float* v) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float* v) {
  const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p));
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); v[2 * e] = f.x; v[2 * e + 1] = f.y; }
}

// A program whose every step combines the running value with a loaded operand, a constant or itself: acc = start; then
// acc = op(acc, operand) (or op(operand, acc) when `swap`), in the program's order and with the same fp32 operations, so the
// result is the program's bit for bit.  Almost every step a graph produces is one (copies, casts, residual adds, scales,
// ReLU behind them); it needs no register file, so the op is decoded once per thread instead of once per element.
enum ChainSrc : unsigned char { C_NONE = 0, C_INPUT, C_IMM, C_SELF };
constexpr int kMaxChain = 12;
struct EltChain {
  int n;                               // steps after the start
  unsigned char startSrc, startIn;     // C_INPUT or C_IMM
  float startImm;
  unsigned char op[kMaxChain], src[kMaxChain], in[kMaxChain], swap[kMaxChain];
  float imm[kMaxChain];
};

static __device__ __noinline__ float evalRare(int op, float x, float y) { return evalOp(op, x, y, 0.f, 0.f); }

// acc = op(acc, y) for V elements; the cheap ops inline, the transcendental ones through one call each.
template <int V> __device__ __forceinline__ void chainStep(int op, float* acc, const float* y, bool swap) {
  switch (op) {
#define LLC_CH(OP, EXPR) case OP: _Pragma("unroll") for (int v = 0; v < V; ++v) { const float a = acc[v], b = y[v]; (void)a; (void)b; acc[v] = EXPR; } break;
    LLC_CH(E_ADD, a + b) LLC_CH(E_MUL, a * b) LLC_CH(E_SUB, swap ? b - a : a - b)
    LLC_CH(E_MAX, swap ? fmaxf(b, a) : fmaxf(a, b)) LLC_CH(E_MIN, swap ? fminf(b, a) : fminf(a, b))
    LLC_CH(E_RELU, fmaxf(a, 0.f)) LLC_CH(E_NEG, -a) LLC_CH(E_ABS, fabsf(a))
    LLC_CH(E_TF32LO, a - __uint_as_float(__float_as_uint(a) & 0xFFFFE000u))
#undef LLC_CH
    case E_CAST: break;
    default:
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] = swap ? evalRare(op, y[v], acc[v]) : evalRare(op, acc[v], y[v]);
  }
}

// Host: the chain form of a program, or false.
bool makeChain(const EltProgram& prog, EltChain& c);
// Host: launches the chain kernels when the shapes suit them; *taken tells whether anything was launched.
int launchChain(const EltArgs& a, cudaStream_t st, bool* taken);

}  // namespace elt
}  // namespace llc
