// rpl_xyw_f64.cu -- instances of the y-walk x/y pass (rpl_xyw.cuh): FP64 models whose kappa bins are whole lane vectors.
#include "rpl_xyw.cuh"

namespace rpl {
namespace xyw {
RPL_XYW_INSTANCES(, double, true, 32)
}  // namespace xyw
}  // namespace rpl
