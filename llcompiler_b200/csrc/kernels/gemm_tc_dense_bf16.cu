#include "gemm_tc_kernel.cuh"

namespace llc {
namespace tcgemm {

LLC_TC_DISPATCH(0, 0, LLC_TC_WIDTHS(false, 1) LLC_TC_WIDTHS(true, 1) LLC_TC_CASE(256, false, 2) LLC_TC_CASE(256, true, 2) LLC_TC_CUT(64) LLC_TC_CUT(128) LLC_TC_CUT(256))

// B stored [k][n] (bf16 only).
int dispatchTcMn(const TilePlan& plan, const TcMaps& m, const TcArgs& a, long long batch, cudaStream_t st) {
  if (plan.bn == 64) return launchTc<64, 0, 0, true, false, 1, false>(m, a, batch, st);
  return launchTc<128, 0, 0, true, false, 1, false>(m, a, batch, st);
}

}  // namespace tcgemm
}  // namespace llc
