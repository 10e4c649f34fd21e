// rpl_xyw_f64u.cu -- instances of the y-walk x/y pass (rpl_xyw.cuh): FP64 models with an odd count of kappa bins.
#include "rpl_xyw.cuh"

namespace rpl {
namespace xyw {
RPL_XYW_INSTANCES(, double, false, 32)
}  // namespace xyw
}  // namespace rpl
