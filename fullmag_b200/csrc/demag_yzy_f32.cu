// demag_yzy_f32.cu — F32 instantiations of the fused kx-plane pass (demag_yzy.cuh).
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f32(Backend &b) { return yzy_configure_t<float>(b); }
bool yzy_launch(Backend &b, const DemagArgs<float> &a) { return yzy_launch_t<float>(b, a); }
int yzy_table_values_f32(int Ly) { return yzy_table_row<float>(Ly); }
void yzy_table_row_f32(int Ly, const double *src, double sign, float *dst) { yzy_table(Ly, src, sign, dst); }

}  // namespace fm
