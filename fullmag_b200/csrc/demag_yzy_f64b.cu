// demag_yzy_f64b.cu — F64 instantiations of the fused kx-plane pass, 5 <= nz <= 8.
#define YZY_HALF 1
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f64b(Backend &b) { return yzy_configure_t<double>(b); }
bool yzy_launch_f64b(Backend &b, const DemagArgs<double> &a) { return yzy_launch_t<double>(b, a); }

}  // namespace fm
