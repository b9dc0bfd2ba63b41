// demag_yzy_f32.cu — F32 instantiations of the fused kx-plane pass (demag_yzy.cuh),
// nz <= 4, and the pass's entry points.
#define YZY_HALF 0
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f32b(Backend &b);
bool yzy_launch_f32b(Backend &b, const DemagArgs<float> &a);

bool yzy_configure_f32(Backend &b) { return b.nz <= 4 ? yzy_configure_t<float>(b) : yzy_configure_f32b(b); }
bool yzy_launch(Backend &b, const DemagArgs<float> &a) { return b.nz <= 4 ? yzy_launch_t<float>(b, a) : yzy_launch_f32b(b, a); }
int yzy_table_values_f32(int Ly) { return yzy_table_row<float>(Ly); }
void yzy_table_row_f32(int Ly, const double *src, double sign, float *dst) { yzy_table(Ly, src, sign, dst); }

}  // namespace fm
