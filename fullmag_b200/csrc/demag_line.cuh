// demag_line.cuh — the x and y passes of the demag convolution on the line FFTs
// of linefft.cuh: buffers and data flow of demag.cuh (S1 [c][z][kx][y],
// S2 [c][z][kx][ky]), padded in-plane lengths any line_length() >= 2n.
#pragma once

#include <algorithm>

#include "demag.cuh"
#include "demag_line.hpp"
#include "linefft.cuh"
#include "pdl.cuh"
#include "zsum.cuh"

namespace fm {

// Most threads of a block: 256, or one 4-line block of 2048 points (512)
template <typename T, int L> __host__ __device__ constexpr int line_max_threads() { return Lf<T, L>::G >= 128 ? 512 : 256; }
// Blocks per SM the register budget is cut for: 32 warps per SM in FP32 (64
// registers; 24 values per thread: 80, 32: 128), 16 in FP64 (24 with 8 to 12 values)
template <typename T, int L> __host__ __device__ constexpr int line_min_blocks() {
    constexpr int V = L / Lf<T, L>::G;
    constexpr int warps = sizeof(T) == 4 ? (V > 24 ? 16 : V > 16 ? 24 : 32) : (V > 16 ? 8 : V > 12 ? 16 : 24);
    return warps * 32 / line_max_threads<T, L>() > 0 ? warps * 32 / line_max_threads<T, L>() : 1;
}

// The twiddles on their way to L1 while the kernel before still runs, then its results.
template <typename T, int L> __device__ __forceinline__ void line_begin(const cx<T> *tw) {
    if constexpr (Lf<T, L>::NP > 1) warm_lines(tw, Lf<T, L>::TW * (int)sizeof(cx<T>));
    pdl_wait();
}

// ---------------------------------------------------------------------------
// x forward: two rows of Ms m per complex line, R2C, transposed store.
// grid (ceil(ny / 2 lines_x), nz, 3), lines_x groups of G threads.
// ---------------------------------------------------------------------------
// Block body (row block bx, plane z, component c); UNI: no mask, Ms map, volume
// fraction or unit source (the batched kernels, batch.cuh).
template <typename T, int L, bool UNI = false>
__device__ __forceinline__ void lx_fwd_body(const DemagArgs<T> &a, int bx, int z, int c, unsigned char *smem_raw) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G;
    C *region = reinterpret_cast<C *>(smem_raw);
    const int LP = a.lines_x, TE = a.te_x, RB = 2 * LP;
    const int y0 = bx * RB, nx = a.nx, ny = a.ny;
    const int q = threadIdx.x / G, t = threadIdx.x % G;
    const int ya = y0 + 2 * q, yb = ya + 1;
    // rows past the grid read row ny - 1 and are zeroed
    const long long rowa = ((long long)z * ny + min(ya, ny - 1)) * nx, rowb = ((long long)z * ny + min(yb, ny - 1)) * nx;
    const T *ma = a.m + (long long)c * a.n + rowa, *mb = a.m + (long long)c * a.n + rowb;
    C *line = region + q * TE;
    auto out = [&](int k, C v) { line[line_slot<T, L>(k)] = v; };
    if (UNI || (!a.mask && !a.ms_map && !a.vf)) {
        // M = Ms m in the storage precision
        const T msT = a.unit_source ? T(1) : (T)a.ms;
        const T sa = ya < ny ? msT : T(0), sb = yb < ny ? msT : T(0);
        auto in = [&](int j) -> C { return j < nx ? mk<T>(ma[j] * sa, mb[j] * sb) : mk<T>(0, 0); };
        line_fwd<L, true>(t, q, a.twx4, line, in, out);
    } else if (a.vf) {
        // boundary tiers: (phi Ms) m over every cell
        auto in = [&](int j) -> C {
            if (j >= nx) return mk<T>(0, 0);
            C v = mk<T>((T)((a.vf[rowa + j] * a.ms) * (double)ma[j]), (T)((a.vf[rowb + j] * a.ms) * (double)mb[j]));
            if (ya >= ny) v.x = T(0);
            if (yb >= ny) v.y = T(0);
            return v;
        };
        line_fwd<L, true>(t, q, a.twx4, line, in, out);
    } else {
        // Ms_i m on active cells (demag_source); every operand is loaded before any
        // is tested, so that a thread's loads are all in flight together
        auto in = [&](int j) -> C {
            if (j >= nx) return mk<T>(0, 0);
            const T va = ma[j], vb = mb[j];
            const double msa = a.ms_map ? a.ms_map[rowa + j] : a.ms, msb = a.ms_map ? a.ms_map[rowb + j] : a.ms;
            const bool ka = a.mask ? a.mask[rowa + j] != 0 : true, kb = a.mask ? a.mask[rowb + j] != 0 : true;
            const T wa = a.unit_source ? va : (T)((double)va * msa), wb = a.unit_source ? vb : (T)((double)vb * msb);
            return mk<T>(ka && msa > 0.0 && ya < ny ? wa : T(0), kb && msb > 0.0 && yb < ny ? wb : T(0));
        };
        line_fwd<L, true>(t, q, a.twx4, line, in, out);
    }
    __syncthreads();
    const int nkx = a.nkx;
    C *s1row = a.s1 + ((long long)c * a.nz + z) * nkx * ny;
    // a thread splits one line pair at one kx: A = (Z[k] + conj Z[-k]) / 2,
    // B = -i (Z[k] - conj Z[-k]) / 2, adjacent in S1
    const int qq = threadIdx.x % LP, kstep = blockDim.x / LP, y = y0 + 2 * qq;
    if (y >= ny) return;
    const C *ln = region + qq * TE;
    const bool both = y + 1 < ny, vec = ny % 2 == 0;
    for (int k = threadIdx.x / LP; k < nkx; k += kstep) {
        const C zk = ln[line_slot<T, L>(k)], zm = ln[line_slot<T, L>(k == 0 ? 0 : L - k)];
        C o0, o1;
        o0.x = T(0.5) * (zk.x + zm.x); o0.y = T(0.5) * (zk.y - zm.y);
        o1.x = T(0.5) * (zk.y + zm.y); o1.y = T(-0.5) * (zk.x - zm.x);
        C *d = s1row + (long long)k * ny + y;
        if (sizeof(C) == 8 && vec) {
            *reinterpret_cast<float4 *>(d) = make_float4((float)o0.x, (float)o0.y, (float)o1.x, (float)o1.y);
        } else {
            d[0] = o0;
            if (both) d[1] = o1;
        }
    }
}

template <typename T, int L>
__global__ void __launch_bounds__((line_max_threads<T, L>()), (line_min_blocks<T, L>())) k_lx_fwd(DemagArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    line_begin<T, L>(a.twx4);
    lx_fwd_body<T, L>(a, blockIdx.x, blockIdx.y, blockIdx.z, smem_raw);
}

// ---------------------------------------------------------------------------
// x inverse: gather the half spectra of the line's two rows, Z = A + iB on the
// full circle (DC and Nyquist taken as real), C2R, crop, 1/P, mask.
// ---------------------------------------------------------------------------
template <typename T, int L, bool UNI = false>
__device__ __forceinline__ void lx_inv_body(const DemagArgs<T> &a, int bx, int z, int c, unsigned char *smem_raw) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G, U = sizeof(T) == 4 ? 8 : 4;  // loads in flight per thread
    C *region = reinterpret_cast<C *>(smem_raw);
    const int LP = a.lines_x, TE = a.te_x, RB = 2 * LP;
    const int y0 = bx * RB, nx = a.nx, ny = a.ny, nkx = a.nkx;
    const int q = threadIdx.x / G, t = threadIdx.x % G;
    const int ya = y0 + 2 * q, yb = ya + 1;
    const bool oka = ya < ny, okb = yb < ny;
    const long long rowa = ((long long)z * ny + ya) * nx, rowb = rowa + nx;
    // activity of the cells this thread will write, loaded before the gather so that the
    // mask's latency is not paid after the transform
    constexpr int NB = line_out_count<T, L, true>();
    static_assert(NB <= 32, "activity bits");
    unsigned acta = 0u, actb = 0u;
    if (!UNI && (a.mask || a.ms_map)) {
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int n = line_out_index<T, L, true>(t, i);
            double msi;
            if (n < nx && oka && cell_active(a, rowa + n, msi)) acta |= 1u << i;
            if (n < nx && okb && cell_active(a, rowb + n, msi)) actb |= 1u << i;
        }
    }
    {
        const C *s1row = a.s1 + ((long long)c * a.nz + z) * nkx * ny;
        const int qq = threadIdx.x % LP, kstep = blockDim.x / LP, k0 = threadIdx.x / LP, y = y0 + 2 * qq;
        const bool on = y < ny, both = y + 1 < ny, vec = ny % 2 == 0;
        C *ln = region + qq * TE;
        for (int kk = k0; kk < nkx; kk += U * kstep) {
            C va[U], vb[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = kk + u * kstep;
                va[u] = mk<T>(0, 0);
                vb[u] = mk<T>(0, 0);
                if (k < nkx && on) {
                    const C *p = s1row + (long long)k * ny + y;
                    if (sizeof(C) == 8 && vec) {
                        const float4 v = *reinterpret_cast<const float4 *>(p);
                        va[u] = mk<T>((T)v.x, (T)v.y);
                        vb[u] = mk<T>((T)v.z, (T)v.w);
                    } else {
                        va[u] = p[0];
                        if (both) vb[u] = p[1];
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = kk + u * kstep;
                if (k < nkx) {
                    const C A = va[u], B = vb[u];
                    if (k == 0 || k == L / 2) {
                        ln[line_slot<T, L>(k)] = mk<T>(A.x, B.x);
                    } else {
                        ln[line_slot<T, L>(k)] = mk<T>(A.x - B.y, A.y + B.x);
                        ln[line_slot<T, L>(L - k)] = mk<T>(A.x + B.y, -A.y + B.x);
                    }
                }
            }
        }
    }
    __syncthreads();
    C *line = region + q * TE;
    const T nrm = (T)a.norm;
    T *ha = a.hd + (long long)c * a.n + rowa, *hb = ha + nx;
    auto in = [&](int k) -> C { return line[line_slot<T, L>(k)]; };
    if (UNI || (!a.mask && !a.ms_map)) {
        const T sc = a.ms > 0.0 ? nrm : T(0);  // no mask, no Ms map: every cell active when Ms > 0
        auto out = [&](int n, C v) {
            if (n >= nx) return;
            if (oka) ha[n] = v.x * sc;
            if (okb) hb[n] = v.y * sc;
        };
        line_inv<L, true>(t, q, a.twx4, line, in, out);
    } else {
        auto out = [&](int n, int i, C v) {
            if (n >= nx) return;
            if (oka) ha[n] = (acta >> i) & 1u ? v.x * nrm : T(0);
            if (okb) hb[n] = (actb >> i) & 1u ? v.y * nrm : T(0);
        };
        line_inv<L, true>(t, q, a.twx4, line, in, out);
    }
}

template <typename T, int L>
__global__ void __launch_bounds__((line_max_threads<T, L>()), (line_min_blocks<T, L>())) k_lx_inv(DemagArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    line_begin<T, L>(a.twx4);
    lx_inv_body<T, L>(a, blockIdx.x, blockIdx.y, blockIdx.z, smem_raw);
}

// ---------------------------------------------------------------------------
// y forward S1 -> S2 and inverse S2 -> S1 (3-D): line g = (c, z, kx),
// lines_y groups of G threads per block; no block barrier
// ---------------------------------------------------------------------------
template <typename T, int L>
__device__ __forceinline__ void ly_fwd_body(const DemagArgs<T> &a, int bx, unsigned char *smem_raw) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G, TE = Lf<T, L>::TILE;
    const int q = threadIdx.x / G, t = threadIdx.x % G, ny = a.ny;
    const long long total = 3LL * a.nz * a.nkx, g = (long long)bx * a.lines_y + q;
    const bool valid = g < total;
    const C *src = a.s1 + (valid ? g : 0) * ny;
    C *dst = a.s2 + g * L;
    auto in = [&](int j) -> C { return j < ny ? src[j] : mk<T>(0, 0); };
    auto out = [&](int k, C v) { if (valid) dst[k] = v; };
    line_fwd<L, true>(t, q, a.twy4, reinterpret_cast<C *>(smem_raw) + q * TE, in, out);
}

template <typename T, int L>
__global__ void __launch_bounds__((line_max_threads<T, L>()), (line_min_blocks<T, L>())) k_ly_fwd(DemagArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    line_begin<T, L>(a.twy4);
    ly_fwd_body<T, L>(a, blockIdx.x, smem_raw);
}

template <typename T, int L>
__device__ __forceinline__ void ly_inv_body(const DemagArgs<T> &a, int bx, unsigned char *smem_raw) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G, TE = Lf<T, L>::TILE;
    const int q = threadIdx.x / G, t = threadIdx.x % G, ny = a.ny;
    const long long total = 3LL * a.nz * a.nkx, g = (long long)bx * a.lines_y + q;
    const bool valid = g < total;
    const C *src = a.s2 + (valid ? g : 0) * L;
    C *dst = a.s1 + g * ny;
    auto in = [&](int k) -> C { return src[k]; };
    auto out = [&](int n, C v) { if (valid && n < ny) dst[n] = v; };
    line_inv<L, true>(t, q, a.twy4, reinterpret_cast<C *>(smem_raw) + q * TE, in, out);
}

template <typename T, int L>
__global__ void __launch_bounds__((line_max_threads<T, L>()), (line_min_blocks<T, L>())) k_ly_inv(DemagArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    line_begin<T, L>(a.twy4);
    ly_inv_body<T, L>(a, blockIdx.x, smem_raw);
}

// ---------------------------------------------------------------------------
// y convolution (2-D thin film): kb_y kx columns x 3 components per block;
// forward y, product with N(kx, ky, 0) where the spectrum lies, inverse y
// ---------------------------------------------------------------------------
template <typename T, int L>
__device__ __forceinline__ void ly_conv_body(const DemagArgs<T> &a, int bx, unsigned char *smem_raw) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G, TE = Lf<T, L>::TILE;
    C *region = reinterpret_cast<C *>(smem_raw);
    const int KB = a.kb_y, ny = a.ny, nkx = a.nkx;
    const int q = threadIdx.x / G, t = threadIdx.x % G;
    const int comp = q / KB, kxl = q - comp * KB;
    const int kx0 = bx * KB, kx = kx0 + kxl;
    const bool valid = kx < nkx;
    C *line = region + q * TE;
    C *g = a.s1 + ((long long)comp * nkx + (valid ? kx : 0)) * ny;
    auto in_g = [&](int j) -> C { return j < ny ? g[j] : mk<T>(0, 0); };
    auto out_s = [&](int k, C v) { line[line_slot<T, L>(k)] = v; };
    line_fwd<L, true>(t, q, a.twy4, line, in_g, out_s);
    __syncthreads();
    for (int u = threadIdx.x; u < KB * L; u += blockDim.x) {
        const int kl = u / L, ky = u % L, s = line_slot<T, L>(ky);
        if (kx0 + kl >= nkx) continue;
        C *lx = region + kl * TE + s, *ly = lx + KB * TE, *lz = ly + KB * TE;
        C mx = *lx, my = *ly, mz = *lz;
        const bool mir = ky > L / 2;
        const T *sp = a.spec + (long long)(kx0 + kl) * a.KY + (mir ? L - ky : ky);
        const long long plane = (long long)nkx * a.KY;
        const T nxx = sp[0], nyy = sp[plane], nzz = sp[2 * plane], nxy = mir ? -sp[3 * plane] : sp[3 * plane];
        if (!a.thin6) {  // a film's xz and yz are zero (odd in z): 4 of 6 tensor planes read
            lx->x = -(nxx * mx.x + nxy * my.x);
            lx->y = -(nxx * mx.y + nxy * my.y);
            ly->x = -(nxy * mx.x + nyy * my.x);
            ly->y = -(nxy * mx.y + nyy * my.y);
            lz->x = -(nzz * mz.x);
            lz->y = -(nzz * mz.y);
        } else {  // an octant of the caller's that has them
            const T nxz = sp[4 * plane], nyz = mir ? -sp[5 * plane] : sp[5 * plane];
            lx->x = -((nxx * mx.x + nxy * my.x) + nxz * mz.x);
            lx->y = -((nxx * mx.y + nxy * my.y) + nxz * mz.y);
            ly->x = -((nxy * mx.x + nyy * my.x) + nyz * mz.x);
            ly->y = -((nxy * mx.y + nyy * my.y) + nyz * mz.y);
            lz->x = -((nxz * mx.x + nyz * my.x) + nzz * mz.x);
            lz->y = -((nxz * mx.y + nyz * my.y) + nzz * mz.y);
        }
    }
    __syncthreads();
    auto in_s = [&](int k) -> C { return line[line_slot<T, L>(k)]; };
    auto out_g = [&](int n, C v) { if (valid && n < ny) g[n] = v; };
    line_inv<L, true>(t, q, a.twy4, line, in_s, out_g);
}

template <typename T, int L>
__global__ void __launch_bounds__((line_max_threads<T, L>() * 3 / 2)) k_ly_conv(DemagArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // the block's columns of the tensor (xx, yy, zz, xy; with thin6 also xz, yz)
    const int kx0 = blockIdx.x * a.kb_y, kb = min(a.kb_y, a.nkx - kx0);
    for (int e = 0; e < (a.thin6 ? 6 : 4); ++e)
        warm_lines(a.spec + ((long long)e * a.nkx + kx0) * a.KY, kb * a.KY * (int)sizeof(T));
    line_begin<T, L>(a.twy4);
    ly_conv_body<T, L>(a, blockIdx.x, smem_raw);
}

// ---------------------------------------------------------------------------
// Direct z sum of one column (col = kx Ly + ky; the batched kernels) with the table of
// octant_to_z_direct: the arithmetic of k_zd (zsum.cuh),
// inputs and table entries read straight from global memory.
template <typename T, int NZ>
__device__ __forceinline__ void zd_col(const DemagArgs<T> &a, int col) {
    using C = cx<T>;
    const int Ly = a.Ly, KY = a.KY, cols = a.nkx * Ly;
    if (col >= cols) return;
    const int cs = NZ * cols, dstr = a.nkx * KY, tstr = NZ * dstr;
    const int kx = col / Ly, ky = col - kx * Ly;
    const bool ymir = ky > Ly / 2;
    const T sy = ymir ? T(-1) : T(1);
    const T *tp = a.spec + (kx * KY + (ymir ? Ly - ky : ky));
    C *base = a.s2 + col;
    C mx[NZ], my[NZ], mz[NZ];
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
        mx[z] = base[z * cols];
        my[z] = base[cs + z * cols];
        my[z].x *= sy; my[z].y *= sy;  // xy and yz change sign with ky: so do My and Hy
        const C v = base[2 * cs + z * cols];
        mz[z] = mk<T>(v.y, -v.x);  // -i Mz
    }
    T tab[6][NZ];
#pragma unroll
    for (int e = 0; e < 6; ++e)
#pragma unroll
        for (int d = 0; d < NZ; ++d) tab[e][d] = e < 4 || d > 0 ? tp[e * tstr + d * dstr] : T(0);
    zsum_column<NZ, T>(mx, my, mz, [&](int e, int d) { return tab[e][d]; });
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
        base[z * cols] = mx[z];
        base[cs + z * cols] = mk<T>(my[z].x * sy, my[z].y * sy);
        base[2 * cs + z * cols] = mk<T>(-mz[z].y, mz[z].x);  // Hz = i Hz'
    }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
// The limit on a kernel's dynamic shared memory is one value per kernel and device, so
// it is set to the most any grid asks of that kernel: a handle with smaller blocks,
// created later, must not lower it for the others.
template <typename K>
cudaError_t line_smem(K kern, size_t most) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}
// most lines per x or y block, and kx columns per thin-film block
template <typename T, int L> constexpr int line_most() {
    constexpr int G = Lf<T, L>::G, lp = line_max_threads<T, L>() / G;
    return lp < 1 ? 1 : G > 32 && lp > 8 ? 8 : lp;
}
template <typename T, int L> constexpr int line_most_kb() {
    constexpr int G = Lf<T, L>::G, least = G >= 32 ? 1 : 32 / G;  // whole warps
    constexpr int kb = line_max_threads<T, L>() / (3 * G) / least * least;
    return kb < least ? least : kb;
}

// Line stride of an x block of lp lines: they start 16 / lp (FP32; 8 / lp in FP64) banks
// apart, so the threads that split or gather them at neighbouring kx do not collide.
template <typename T, int L> int line_stride(int lp) {
    const int banks = sizeof(T) == 4 ? 16 : 8, want = banks / std::min(lp, banks);
    int te = Lf<T, L>::TILE;
    while (te % banks != want % banks) ++te;
    return te;
}

// Lines per block: 256 threads (4 lines of 1024 points: 64-byte segments of S1 per
// kx in FP32), fewer while the grid would leave SMs without a block, never less
// than a warp.
template <typename T>
cudaError_t line_setup(LineCfg &c, int Lx, int Ly, bool thin, int ny, int nz, int nkx) {
    constexpr int kSms = 148;
    c = LineCfg{};
    c.Lx = Lx;
    c.Ly = Ly;
    cudaError_t err = cudaErrorInvalidValue;
    const bool okx = with_line(Lx, [&](auto l) {
        constexpr int L = decltype(l)::value, G = Lf<T, L>::G;
        const int pairs = (ny + 1) / 2, least = std::max(1, 32 / G);
        int lp = line_most<T, L>();
        while (lp > least && (pairs + lp - 1) / lp * nz * 3 < 2 * kSms) lp /= 2;
        const int te = line_stride<T, L>(lp);
        c.lines_x = lp;
        c.te_x = te;
        c.thr_x = lp * G;
        c.smem_x = (size_t)lp * te * sizeof(cx<T>);
        const size_t most = (size_t)line_most<T, L>() * (Lf<T, L>::TILE + 15) * sizeof(cx<T>);
        err = line_smem(k_lx_fwd<T, L>, most);
        if (err == cudaSuccess) err = line_smem(k_lx_inv<T, L>, most);
    });
    if (!okx || err != cudaSuccess) return err;
    err = cudaErrorInvalidValue;
    with_line(Ly, [&](auto l) {
        constexpr int L = decltype(l)::value, G = Lf<T, L>::G;
        const size_t line = (size_t)Lf<T, L>::TILE * sizeof(cx<T>);
        if (thin) {
            const int least = G >= 32 ? 1 : 32 / G;  // whole warps
            int kb = line_most_kb<T, L>();
            while (kb > least && (nkx + kb - 1) / kb < kSms) kb = std::max(least, kb / 2 / least * least);
            c.kb_y = kb;
            c.thr_yc = 3 * kb * G;
            c.smem_yc = 3 * kb * line;
            err = line_smem(k_ly_conv<T, L>, 3 * line_most_kb<T, L>() * line);
        } else {
            const int least = std::max(1, 32 / G);
            const long long lines = 3LL * nz * nkx;
            int lp = line_most<T, L>();
            while (lp > least && (lines + lp - 1) / lp < 4 * kSms) lp /= 2;
            c.lines_y = lp;
            c.thr_y = lp * G;
            c.smem_y = lp * line;
            err = line_smem(k_ly_fwd<T, L>, line_most<T, L>() * line);
            if (err == cudaSuccess) err = line_smem(k_ly_inv<T, L>, line_most<T, L>() * line);
        }
    });
    return err;
}

template <typename K, typename T>
void line_launch(const LineCfg &c, K kern, dim3 g, int threads, size_t smem, cudaStream_t st, const DemagArgs<T> &a) {
    if (c.pdl) pdl_launch(kern, g, dim3((unsigned)threads), smem, st, a);
    else kern<<<g, threads, smem, st>>>(a);
}

template <typename T>
void line_x_fwd(const LineCfg &c, DemagArgs<T> a, cudaStream_t st) {
    a.lines_x = c.lines_x;
    a.te_x = c.te_x;
    const dim3 g((a.ny + 2 * c.lines_x - 1) / (2 * c.lines_x), a.nz, 3);
    with_line(c.Lx, [&](auto l) { line_launch(c, k_lx_fwd<T, decltype(l)::value>, g, c.thr_x, c.smem_x, st, a); });
}

template <typename T>
void line_x_inv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st) {
    a.lines_x = c.lines_x;
    a.te_x = c.te_x;
    const dim3 g((a.ny + 2 * c.lines_x - 1) / (2 * c.lines_x), a.nz, 3);
    with_line(c.Lx, [&](auto l) { line_launch(c, k_lx_inv<T, decltype(l)::value>, g, c.thr_x, c.smem_x, st, a); });
}

template <typename T>
void line_y_fwd(const LineCfg &c, DemagArgs<T> a, cudaStream_t st) {
    a.lines_y = c.lines_y;
    const unsigned g = (unsigned)((3LL * a.nz * a.nkx + c.lines_y - 1) / c.lines_y);
    with_line(c.Ly, [&](auto l) { line_launch(c, k_ly_fwd<T, decltype(l)::value>, g, c.thr_y, c.smem_y, st, a); });
}

template <typename T>
void line_y_inv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st) {
    a.lines_y = c.lines_y;
    const unsigned g = (unsigned)((3LL * a.nz * a.nkx + c.lines_y - 1) / c.lines_y);
    with_line(c.Ly, [&](auto l) { line_launch(c, k_ly_inv<T, decltype(l)::value>, g, c.thr_y, c.smem_y, st, a); });
}

template <typename T>
void line_y_conv(const LineCfg &c, DemagArgs<T> a, cudaStream_t st) {
    a.kb_y = c.kb_y;
    const unsigned g = (unsigned)((a.nkx + c.kb_y - 1) / c.kb_y);
    with_line(c.Ly, [&](auto l) { line_launch(c, k_ly_conv<T, decltype(l)::value>, g, c.thr_yc, c.smem_yc, st, a); });
}

#define FM_LINE_INSTANCES(T)                                                                     \
    template cudaError_t line_setup<T>(LineCfg &, int, int, bool, int, int, int);                \
    template void line_x_fwd<T>(const LineCfg &, DemagArgs<T>, cudaStream_t);                    \
    template void line_x_inv<T>(const LineCfg &, DemagArgs<T>, cudaStream_t);                    \
    template void line_y_fwd<T>(const LineCfg &, DemagArgs<T>, cudaStream_t);                    \
    template void line_y_inv<T>(const LineCfg &, DemagArgs<T>, cudaStream_t);                    \
    template void line_y_conv<T>(const LineCfg &, DemagArgs<T>, cudaStream_t)

}  // namespace fm
