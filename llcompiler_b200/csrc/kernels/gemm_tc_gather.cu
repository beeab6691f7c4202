#include "gemm_tc_kernel.cuh"

namespace llc {
namespace tcgemm {

LLC_TC_DISPATCH(1, 0, LLC_TC_WIDTHS(false, 1))
LLC_TC_DISPATCH(1, 1, LLC_TC_WIDTHS(false, 1))
LLC_TC_DISPATCH(1, 2, LLC_TC_CASE(64, false, 1) LLC_TC_CASE(128, false, 1))

}  // namespace tcgemm
}  // namespace llc
