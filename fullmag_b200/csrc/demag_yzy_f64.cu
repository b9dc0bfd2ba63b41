// demag_yzy_f64.cu — F64 instantiations of the fused kx-plane pass (demag_yzy.cuh),
// nz <= 4, and the pass's entry points.
#define YZY_HALF 0
#include "demag_yzy.cuh"

namespace fm {

bool yzy_configure_f64b(Backend &b);
bool yzy_launch_f64b(Backend &b, const DemagArgs<double> &a);

bool yzy_configure_f64(Backend &b) { return b.nz <= 4 ? yzy_configure_t<double>(b) : yzy_configure_f64b(b); }
bool yzy_launch(Backend &b, const DemagArgs<double> &a) { return b.nz <= 4 ? yzy_launch_t<double>(b, a) : yzy_launch_f64b(b, a); }
int yzy_table_values_f64(int Ly) { return yzy_table_row<double>(Ly); }
void yzy_table_row_f64(int Ly, const double *src, double sign, double *dst) { yzy_table(Ly, src, sign, dst); }

}  // namespace fm
