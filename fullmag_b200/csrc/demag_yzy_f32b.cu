// demag_yzy_f32b.cu — F32 instantiations of the fused kx-plane pass, 5 <= nz <= 8.
#define YZY_HALF 1
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f32b(Backend &b) { return yzy_configure_t<float>(b); }
bool yzy_launch_f32b(Backend &b, const DemagArgs<float> &a) { return yzy_launch_t<float>(b, a); }

}  // namespace fm
