// demag_line.hpp — launch interface of the register line-FFT demag passes
// (demag_line.cuh), compiled once per precision.
#pragma once

#include <cuda_runtime.h>

#include "demag.cuh"

namespace fm {

// Block shapes of the passes for one grid (line_setup).
struct LineCfg {
    int Lx = 0, Ly = 0;
    bool pdl = true;                         // programmatic dependent launches (pdl.cuh)
    int lines_x = 0, te_x = 0, thr_x = 0;    // x passes: row pairs per block, line stride
    size_t smem_x = 0;
    int lines_y = 0, thr_y = 0;              // y passes: lines per block
    size_t smem_y = 0;
    int kb_y = 0, thr_yc = 0;                // thin films: kx columns per block
    size_t smem_yc = 0;
};

// Fill the shapes for padded in-plane lengths Lx, Ly (line_length values) and set
// the kernels' attributes; cudaErrorInvalidValue when a length is not one of them.
template <typename T> cudaError_t line_setup(LineCfg &c, int Lx, int Ly, bool thin, int ny, int nz, int nkx);
// x forward: Ms m -> S1; y forward: S1 -> S2; y inverse: S2 -> S1; thin films' y
// convolution on S1; x inverse: S1 -> H_d
template <typename T> void line_x_fwd(const LineCfg &c, DemagArgs<T> a, cudaStream_t st);
template <typename T> void line_x_inv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st);
template <typename T> void line_y_fwd(const LineCfg &c, DemagArgs<T> a, cudaStream_t st);
template <typename T> void line_y_inv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st);
template <typename T> void line_y_conv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st);

}  // namespace fm
