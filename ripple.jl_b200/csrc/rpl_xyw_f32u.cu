// rpl_xyw_f32u.cu -- instances of the y-walk x/y pass (rpl_xyw.cuh): FP32 models with any other count of kappa bins.
#include "rpl_xyw.cuh"

namespace rpl {
namespace xyw {
RPL_XYW_INSTANCES(, float, false, 8)
}  // namespace xyw
}  // namespace rpl
