// rpl_xyw_f32.cu -- instances of the y-walk x/y pass (rpl_xyw.cuh): FP32 models whose kappa bins are whole lane vectors.
#include "rpl_xyw.cuh"

namespace rpl {
namespace xyw {
RPL_XYW_INSTANCES(, float, true, 8)
}  // namespace xyw
}  // namespace rpl
