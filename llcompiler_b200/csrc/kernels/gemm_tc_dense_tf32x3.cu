#include "gemm_tc_kernel.cuh"

namespace llc {
namespace tcgemm {

LLC_TC_DISPATCH(0, 2, LLC_TC_CASE(64, false, 1) LLC_TC_CASE(128, false, 1) LLC_TC_CUT(64) LLC_TC_CUT(128))

}  // namespace tcgemm
}  // namespace llc
