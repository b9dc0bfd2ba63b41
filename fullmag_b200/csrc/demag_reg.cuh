// demag_reg.cuh — the z passes of the demag convolution in registers: direct sums
// (k_zd) and the z FFT with the tensor product (k_zc_r), on S2 [c][z][kx][ky] of the
// line-FFT passes (demag_line.cuh); and the line strides of the opt-in row pass.
#pragma once

#include "cpasync.cuh"
#include "demag.cuh"
#include "fftreg.cuh"
#include "pdl.cuh"
#include "zsum.cuh"

namespace fm {

// Per-line shared-memory region (tile, then the line's outputs), padded by one
// element so that consecutive lines start in different banks.
template <int L1, int L2> __host__ __device__ constexpr int line_region() {
    return (tile_elems(L1, L2) > L1 * L2 ? tile_elems(L1, L2) : L1 * L2) + 1;
}

// Line stride of the x passes whose threads each handle a pair of rows (the x
// inverse's gather, the pipelined x forward's transposed store): a warp touches
// 4 lines x 8 kx (FP32) or a quarter-warp 4 lines x 2 kx (FP64) at once, and a
// stride of 4 mod 16 (FP32) or 2 mod 8 (FP64) complex elements puts each phase
// in distinct banks (line_region's 1 mod 16 made them collide).  Lines of 32
// threads only: a warp then holds one line inside fft4step.
template <typename T, int L1, int L2> __host__ __device__ constexpr int pair_stride() {
    return L2 == 32 ? line_region<L1, L2>() + (sizeof(T) == 8 ? 1 : 3) : line_region<L1, L2>();
}
// ---------------------------------------------------------------------------
// z convolution (3-D): P threads per (kx, ky) column hold the three
// components' z lines in registers: forward FFT, H = -N M per kz, inverse FFT,
// keep z < nz.  With P = 2 the zero padding (x[z] = 0 for z >= nz = LZ/2) is
// used to split the transform by the parity h of kz:
//   X[2m + h] = FFT_nz(x[z] W_LZ^{h z})[m],
//   x'[z]     = sum_h W_LZ^{-h z} IFFT_nz(X'_h)[z]        (z < nz),
// so each thread of the pair holds 3 x nz values and the two halves are summed
// with one shuffle exchange.
// ---------------------------------------------------------------------------
// One column task tid (tid / P = column, h = tid % P = kz parity, passed in by
// the caller: it is the lane parity, invariant over the caller's loop); the task
// index of a warp's lanes must be contiguous and start at a multiple of 32.
template <typename T, int LZ, int P>
__device__ __forceinline__ void zc_task(const DemagArgs<T> &a, int tid, int h) {
    using C = cx<T>;
    constexpr int NZL = LZ / P;  // points per thread
    static_assert(P == 1 || P == 2, "z split");
    // nkx * Ly < 2^31 for every supported grid: 32-bit index math
    const int cols = a.nkx * a.Ly;
    const int nz = a.nz, Ly = a.Ly, nkx = a.nkx;
    const long long cs = (long long)nz * nkx * Ly;  // component stride in S2
    const long long zs = (long long)nkx * Ly;
    {
        const int col = tid / P;
        const bool valid = col < cols;
        const int kx = valid ? col / Ly : 0;
        const int ky = valid ? col - kx * Ly : 0;
        C *base = a.s2 + (long long)kx * Ly + ky;
        C vx[NZL], vy[NZL], vz[NZL];
#pragma unroll
        for (int z = 0; z < NZL; ++z) {
            const bool in = valid && z < nz;
            vx[z] = in ? base[z * zs] : mk<T>(0, 0);
            vy[z] = in ? base[cs + z * zs] : mk<T>(0, 0);
            vz[z] = in ? base[2 * cs + z * zs] : mk<T>(0, 0);
            if (P == 2 && h == 1 && z > 0) {
                const C w = tw64<C>(z * (64 / LZ));  // W_LZ^z
                vx[z] = cmul(vx[z], w); vy[z] = cmul(vy[z], w); vz[z] = cmul(vz[z], w);
            }
        }
        fft_reg<NZL, false>(vx);
        fft_reg<NZL, false>(vy);
        fft_reg<NZL, false>(vz);
        if (valid) {
            // tensor_apply for one (kx, ky) column: the ky mirror, its sign and the
            // column's offset in a kz plane of the octant are hoisted out of the kz
            // loop; 32-bit offsets (6 KZ nkx KY < 2^31 for every supported grid)
            const int KY = a.KY, plane_z = nkx * KY, cstr = a.KZ * plane_z;
            const bool ymir = ky > Ly / 2;
            const T sy = ymir ? T(-1) : T(1);
            const T *sp = a.spec + (kx * KY + (ymir ? Ly - ky : ky));
#pragma unroll
            for (int p = 0; p < NZL; ++p) {
                const int kz = P * brev<NZL>(p) + h;
                const bool zmir = kz > LZ / 2;
                const T sz = zmir ? T(-1) : T(1);
                const T *q = sp + (zmir ? LZ - kz : kz) * plane_z;
                const T nxx = q[0], nyy = q[cstr], nzz = q[2 * cstr];
                const T nxy = q[3 * cstr] * sy, nxz = q[4 * cstr] * sz, nyz = q[5 * cstr] * (sy * sz);
                const C mx = vx[p], my = vy[p], mz = vz[p];
                vx[p].x = -((nxx * mx.x + nxy * my.x) + nxz * mz.x);
                vx[p].y = -((nxx * mx.y + nxy * my.y) + nxz * mz.y);
                vy[p].x = -((nxy * mx.x + nyy * my.x) + nyz * mz.x);
                vy[p].y = -((nxy * mx.y + nyy * my.y) + nyz * mz.y);
                vz[p].x = -((nxz * mx.x + nyz * my.x) + nzz * mz.x);
                vz[p].y = -((nxz * mx.y + nyz * my.y) + nzz * mz.y);
            }
        }
        fft_reg_dit<NZL, true>(vx);
        fft_reg_dit<NZL, true>(vy);
        fft_reg_dit<NZL, true>(vz);
        if constexpr (P == 1) {
            if (valid) {
#pragma unroll
                for (int z = 0; z < NZL; ++z) {
                    if (z < nz) {
                        base[z * zs] = vx[z];
                        base[cs + z * zs] = vy[z];
                        base[2 * cs + z * zs] = vz[z];
                    }
                }
            }
        } else {
            // thread h keeps z in [h nz/2, (h+1) nz/2); the partner's half arrives by shuffle
#pragma unroll
            for (int zz = 0; zz < NZL / 2; ++zz) {
                // register selection by h without dynamic indexing
                const int zlo = zz, zhi = zz + NZL / 2;
                const int zmine = h ? zhi : zlo;
                C ox = h ? vx[zhi] : vx[zlo], oy = h ? vy[zhi] : vy[zlo], oz = h ? vz[zhi] : vz[zlo];
                C sx = h ? vx[zlo] : vx[zhi], sy = h ? vy[zlo] : vy[zhi], sz = h ? vz[zlo] : vz[zhi];
                if (h == 1) {
                    // this thread's values carry W_LZ^{-z}
                    const C w1 = tw64<C>(zhi * (64 / LZ));
                    ox = cmulc(ox, w1); oy = cmulc(oy, w1); oz = cmulc(oz, w1);
                    const C w2 = tw64<C>(zlo * (64 / LZ));
                    sx = cmulc(sx, w2); sy = cmulc(sy, w2); sz = cmulc(sz, w2);
                }
                C rx, ry, rz;
                rx.x = __shfl_xor_sync(0xffffffffu, sx.x, 1); rx.y = __shfl_xor_sync(0xffffffffu, sx.y, 1);
                ry.x = __shfl_xor_sync(0xffffffffu, sy.x, 1); ry.y = __shfl_xor_sync(0xffffffffu, sy.y, 1);
                rz.x = __shfl_xor_sync(0xffffffffu, sz.x, 1); rz.y = __shfl_xor_sync(0xffffffffu, sz.y, 1);
                if (valid && zmine < nz) {
                    base[zmine * zs] = cadd(ox, rx);
                    base[cs + zmine * zs] = cadd(oy, ry);
                    base[2 * cs + zmine * zs] = cadd(oz, rz);
                }
            }
        }
    }
}

template <typename T, int LZ, int P>
__global__ void __launch_bounds__(128) k_zc_r(DemagArgs<T> a) {
    const int span = ((a.nkx * a.Ly * P + 127) / 128) * 128;  // whole pairs and warps iterate together
    const int h = (P == 2) ? (threadIdx.x & 1) : 0;
    pdl_wait();
    for (int tid = blockIdx.x * blockDim.x + threadIdx.x; tid < span; tid += gridDim.x * blockDim.x)
        zc_task<T, LZ, P>(a, tid, h);
}

// ---------------------------------------------------------------------------
// z convolution by direct summation (3-D, nz <= 8).  With the zero padding the
// FFT pass computes, per (kx, ky) column, the linear convolution
//   H(z) = -sum_{z' < nz} n(z - z') M(z'),   n(d) = sum_kz N(kx, ky, kz) W_Lz^{-kz d},
// and only offsets |d| < nz reach a kept output, so the same sum is taken here
// directly (zsum.cuh): nz^2 / 2 3x3 tensor products per column instead of the two
// z FFTs, no twiddles and no padded points.  The table (built on the host from the
// octant, newell_host.hpp octant_to_z_direct) holds n(d) for d in [0, nz):
// components even in z are real; xz and yz are i tau(d) with tau real and odd
// in d.  With Mz' = -i Mz and Hz' = -i Hz the product is a real matrix on
// complex vectors,
//   (Hx, Hy, Hz') = [[-nxx, -nxy, tau_xz], [-nxy, -nyy, tau_yz],
//                    [-tau_xz, -tau_yz, -nzz]] (Mx, My, Mz'),
// stored as tab[c][d][kx][ky'] = (-nxx, -nyy, -nzz, -nxy, tau_xz, tau_yz) / 2 for
// ky' <= Ly/2.  ky > Ly/2 reads the mirror with the sign of the components odd
// in y (xy, yz); d < 0 flips the components odd in z (xz, yz).
// ---------------------------------------------------------------------------
// Persistent threads, one column per thread per iteration; the
// next column's inputs and table entries are copied into the thread's own
// shared-memory slots (cp.async, double buffer) while the current one is
// summed, so the loads of one column overlap the arithmetic of the previous.
// A thread only reads back what it copied itself: no block barrier.
// Shared memory per thread: 2 x (3 nz complex + 6 nz reals), item-major with
// the thread index fastest (conflict-free).
template <typename T, int NZ>
__host__ __device__ constexpr size_t zd_smem_per_thread() {
    return 2 * (3 * NZ * sizeof(cx<T>) + 6 * NZ * sizeof(T));
}
template <typename T> __host__ __device__ constexpr int zd_threads() { return sizeof(T) == 8 ? 64 : 128; }

template <typename T, int NZ>
__global__ void __launch_bounds__(zd_threads<T>()) k_zd(DemagArgs<T> a) {
    using C = cx<T>;
    constexpr int NM = 3 * NZ, NT = 6 * NZ, BT = zd_threads<T>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    C *mb0 = reinterpret_cast<C *>(smem_raw);
    T *tb0 = reinterpret_cast<T *>(mb0 + 2 * NM * BT);
    // 3 NZ nkx Ly and 6 NZ nkx KY < 2^31 for every supported grid: 32-bit offsets
    const int Ly = a.Ly, KY = a.KY, cols = a.nkx * Ly;
    const int cs = NZ * cols, dstr = a.nkx * KY, tstr = NZ * dstr;
    auto prefetch = [&](int col, int buf) {
        const int kx = col / Ly, ky = col - kx * Ly;
        const C *src = a.s2 + col;
        const unsigned dm = (unsigned)__cvta_generic_to_shared(mb0 + buf * NM * BT + tid);
#pragma unroll
        for (int s = 0; s < NM; ++s)
            cp_async_elem<sizeof(C)>(dm + s * BT * (unsigned)sizeof(C), src + (s / NZ) * cs + (s % NZ) * cols);
        const T *tp = a.spec + (kx * KY + (ky > Ly / 2 ? Ly - ky : ky));
        const unsigned dt = (unsigned)__cvta_generic_to_shared(tb0 + buf * NT * BT + tid);
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
            for (int d = 0; d < NZ; ++d)
                if (c < 4 || d > 0)  // tau(0) = 0 is not read
                    cp_async_elem<sizeof(T)>(dt + (c * NZ + d) * BT * (unsigned)sizeof(T), tp + c * tstr + d * dstr);
    };
    pdl_wait();
    const int stride = gridDim.x * BT;
    int col = blockIdx.x * BT + tid, buf = 0;
    if (col < cols) prefetch(col, 0);
    cp_async_commit();
    for (; col < cols; col += stride, buf ^= 1) {
        if (col + stride < cols) prefetch(col + stride, buf ^ 1);
        cp_async_commit();  // possibly empty: "all but the newest" is this column
        cp_async_wait_all_but_one();
        const C *sm = mb0 + buf * NM * BT + tid;
        const T *st = tb0 + buf * NT * BT + tid;
        const int kx = col / Ly, ky = col - kx * Ly;
        const T sy = ky > Ly / 2 ? T(-1) : T(1);
        C mx[NZ], my[NZ], mz[NZ];
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
            mx[z] = sm[z * BT];
            my[z] = sm[(NZ + z) * BT];
            my[z].x *= sy; my[z].y *= sy;  // xy and yz change sign with ky: so do My and Hy
            const C v = sm[(2 * NZ + z) * BT];
            mz[z] = mk<T>(v.y, -v.x);  // -i Mz
        }
        zsum_column<NZ, T>(mx, my, mz, [&](int e, int d) { return st[(e * NZ + d) * BT]; });
        C *base = a.s2 + col;
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
            base[z * cols] = mx[z];
            base[cs + z * cols] = mk<T>(my[z].x * sy, my[z].y * sy);
            base[2 * cs + z * cols] = mk<T>(-mz[z].y, mz[z].x);  // Hz = i Hz'
        }
    }
    cp_async_wait_all();
}

}  // namespace fm
