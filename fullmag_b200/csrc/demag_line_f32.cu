// demag_line_f32.cu — the line-FFT demag passes (demag_line.cuh) in FP32.
#include "demag_line.cuh"

namespace fm {
FM_LINE_INSTANCES(float);
}  // namespace fm
