// demag_yzy_f64.cu — F64 instantiations of the fused kx-plane pass (demag_yzy.cuh).
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f64(Backend &b) { return yzy_configure_t<double>(b); }
bool yzy_launch(Backend &b, const DemagArgs<double> &a) { return yzy_launch_t<double>(b, a); }
int yzy_table_values_f64(int Ly) { return yzy_table_row<double>(Ly); }
void yzy_table_row_f64(int Ly, const double *src, double sign, double *dst) { yzy_table(Ly, src, sign, dst); }

}  // namespace fm
