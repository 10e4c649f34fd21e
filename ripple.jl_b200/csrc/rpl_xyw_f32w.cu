// rpl_xyw_f32w.cu -- instances of the y-walk x/y pass (rpl_xyw.cuh): FP32 models with 33 to 64 kappa bins.
#include "rpl_xyw.cuh"

namespace rpl {
namespace xyw {
RPL_XYW_INSTANCES(, float, false, 16)
}  // namespace xyw
}  // namespace rpl
