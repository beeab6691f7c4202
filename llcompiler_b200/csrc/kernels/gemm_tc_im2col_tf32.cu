#include "gemm_tc_kernel.cuh"

namespace llc {
namespace tcgemm {

LLC_TC_DISPATCH(2, 1, LLC_TC_WIDTHS(false, 1) LLC_TC_WIDTHS(true, 1) LLC_TC_CASE(256, false, 2) LLC_TC_CASE(256, true, 2) LLC_TC_CUT(64) LLC_TC_CUT(128) LLC_TC_CUT(256))

}  // namespace tcgemm
}  // namespace llc
