// demag_line_f64.cu — the line-FFT demag passes (demag_line.cuh) in FP64.
#include "demag_line.cuh"

namespace fm {
FM_LINE_INSTANCES(double);
}  // namespace fm
