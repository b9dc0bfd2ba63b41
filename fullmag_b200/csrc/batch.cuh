// batch.cuh — persistent kernels over many independent problems (the batched
// ensemble, fullmag_fdm_batch_*; no counterpart in the reference).
//
// Every stage of a step is one launch for the whole batch: the blocks walk a
// work list of (problem, block coordinates) items in grid-stride order and
// run the same block bodies as the single-problem kernels (demag_line.cuh,
// stages.cuh) on that problem's arguments.  The padded FFT lengths differ per
// problem, so each item dispatches on its problem's length; the switch is
// uniform across the block.  Work lists, per-problem arguments and the grid
// sizes (chosen by the batch autotuner) are set up by batch.cu.
#pragma once

#include "demag_line.cuh"
#include "demag_reg.cuh"
#include "stages.cuh"

namespace fm {

// Blocks of 256 threads per SM the x / y kernels' registers are cut for.  A kernel holds
// the registers of its longest line, so batches without lines over 512 points take
// the form without them (LONG = false: FP32 80 registers, 24 warps per SM).
template <typename T, bool LONG> __host__ __device__ constexpr int batch_min_blocks() {
    return sizeof(T) == 4 ? (LONG ? 2 : 3) : 1;
}

// x passes: item (p, bx, z, c); lines_x = threads / G lines per block for each problem;
// Lx one of the line-FFT lengths 16..1024 (batch.cu pads every in-plane axis to them)
template <typename T, bool INV, bool LONG>
__global__ void __launch_bounds__(256, (batch_min_blocks<T, LONG>())) k_batch_x(const DemagArgs<T> *__restrict__ A,
                                                                                 const int4 *__restrict__ work, int nwork) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 it = work[w];
        const DemagArgs<T> &a = A[it.x];
        switch (a.Lx) {
#define FM_B(L)                                                                  \
    case L:                                                                      \
        if (INV) lx_inv_body<T, L, true>(a, it.y, it.z, it.w, smem_raw);  \
        else lx_fwd_body<T, L, true>(a, it.y, it.z, it.w, smem_raw);      \
        break;
            FM_B(16) FM_B(32) FM_B(64) FM_B(96) FM_B(128) FM_B(192) FM_B(256) FM_B(384) FM_B(512)
            default:
                if constexpr (LONG) {
                    switch (a.Lx) {
                        FM_B(768) FM_B(1024)
                        default: break;
                    }
                }
                break;
#undef FM_B
        }
        __syncthreads();  // the next item reuses the line tiles
    }
}

// y passes: item (p, bx); lines_y = threads / G lines per block
template <typename T, bool INV, bool LONG>
__global__ void __launch_bounds__(256, (batch_min_blocks<T, LONG>())) k_batch_y(const DemagArgs<T> *__restrict__ A,
                                                                                 const int4 *__restrict__ work, int nwork) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 it = work[w];
        const DemagArgs<T> &a = A[it.x];
        switch (a.Ly) {
#define FM_B(L)                                                                  \
    case L:                                                                      \
        if (INV) ly_inv_body<T, L>(a, it.y, smem_raw);  \
        else ly_fwd_body<T, L>(a, it.y, smem_raw);      \
        break;
            FM_B(16) FM_B(32) FM_B(64) FM_B(96) FM_B(128) FM_B(192) FM_B(256) FM_B(384) FM_B(512)
            default:
                if constexpr (LONG) {
                    switch (a.Ly) {
                        FM_B(768) FM_B(1024)
                        default: break;
                    }
                }
                break;
#undef FM_B
        }
        __syncthreads();  // the next item reuses the line tiles
    }
}

// z convolution: item (p, chunk) of 128 column tasks; 128 threads.  DIRECT: the
// direct sum per column for nz <= NZMAX (the kernel's registers are those of
// its largest case, so batches whose problems all have nz <= 4 take NZMAX = 4),
// else the z FFT pass (zc_task; with Lz = 16 a thread pair per column)
template <typename T, bool DIRECT, int NZMAX = 8>
__global__ void __launch_bounds__(128) k_batch_z(const DemagArgs<T> *__restrict__ A, const int4 *__restrict__ work,
                                                 int nwork) {
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 it = work[w];
        const DemagArgs<T> &a = A[it.x];
        const int tid = it.y * 128 + threadIdx.x;
        if constexpr (DIRECT) {
            switch (a.nz) {
                case 1: zd_col<T, 1>(a, tid); break;
                case 2: zd_col<T, 2>(a, tid); break;
                case 3: zd_col<T, 3>(a, tid); break;
                case 4: zd_col<T, 4>(a, tid); break;
                default:
                    if constexpr (NZMAX > 4) {
                        switch (a.nz) {
                            case 5: zd_col<T, 5>(a, tid); break;
                            case 6: zd_col<T, 6>(a, tid); break;
                            case 7: zd_col<T, 7>(a, tid); break;
                            case 8: zd_col<T, 8>(a, tid); break;
                            default: break;
                        }
                    }
                    break;
            }
        } else {
            switch (a.Lz) {
                case 2: zc_task<T, 2, 1>(a, tid, 0); break;
                case 4: zc_task<T, 4, 1>(a, tid, 0); break;
                case 8: zc_task<T, 8, 1>(a, tid, 0); break;
                case 16: zc_task<T, 16, 2>(a, tid, threadIdx.x & 1); break;
                default: break;
            }
        }
    }
}

// stage kernel: item (p, bx, by, bz), block (32, 4); zb[p] planes per thread;
// no diagnostics (the batch reports states, not per-step statistics)
template <typename T, int MODE>
__global__ void __launch_bounds__(128, 4) k_batch_stage(const StageArgs<T> *__restrict__ S,
                                                        const int *__restrict__ zb,
                                                        const int4 *__restrict__ work, int nwork) {
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 it = work[w];
        double acc[NQ] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // unused: no diagnostics
        stage_plain_body<T, MODE>(S[it.x], zb[it.x], it.y, it.z, it.w, acc);
    }
}

// predictor combine: item (p, chunk) of 256 cells
template <typename T>
__global__ void __launch_bounds__(256) k_batch_combine(const CombineArgs<T> *__restrict__ A,
                                                       const int4 *__restrict__ work, int nwork) {
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 it = work[w];
        const CombineArgs<T> &a = A[it.x];
        const long long i = (long long)it.y * 256 + threadIdx.x;
        if (i < a.n) combine_cell(a, i);
    }
}

// A problem's state, SoA in T, as AoS FP64: 48 problems, 1.36 M cells, read back in 7.6 ms;
// with the words turned round one by one on the host 10.6 ms.
template <typename T>
__global__ void __launch_bounds__(256) k_batch_aos(const T *__restrict__ m, double *__restrict__ out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        out[3 * i] = (double)m[i];
        out[3 * i + 1] = (double)m[n + i];
        out[3 * i + 2] = (double)m[2 * n + i];
    }
}

}  // namespace fm
