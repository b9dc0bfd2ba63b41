// demag_yzy.cuh — fused y forward, direct z convolution and y inverse of one kx
// plane per cluster of P CTAs (3-D grids with nz <= 8, direct z table).
//
// The three split kernels move the plane's y spectrum S2 through HBM three
// times (written by the y forward pass, read and written by the z sum, read
// by the y inverse pass).  Here the 3 nz lines (c, z) of plane kx stay in the
// shared memory of one thread-block cluster from the y forward FFT to the y
// inverse FFT.  CTA h of the cluster owns lines [h NLH, (h + 1) NLH):
//   1. one group of threads per owned line: forward y (line_fwd, the zero-padded
//      half of the input pruned) from S1 into the line's row, left in slot order;
//   2. cluster barrier; CTA h sums the direct z convolution of the ky columns
//      [h Ly/P, (h + 1) Ly/P), reading each column's 3 nz values from the
//      owners' rows (distributed shared memory for the other CTAs' lines) and
//      writing the results back there (k_zd's loop, all three components at once;
//      one component at a time measured 104.6 against 99.4 us at 512 x 512 x 8);
//   3. cluster barrier; inverse y (line_inv) from the owned rows back into S1,
//      keeping y < ny.
// The sums are those of k_zd, in the same order per output, and the FFTs are
// those of k_ly_fwd and k_ly_inv, so the result is bitwise the split path's.
// Shared memory per CTA: NLH rows of a line's tile, then the twiddles.  P = 1 is one
// CTA per plane.  No TMA; the remote rows are read and written with plain loads and
// stores.
//
// The spectrum stays in the slots the transforms leave it in (linefft.cuh), and the z
// table is uploaded in the same order (yzy_table), so the lanes of the z sum read
// neighbouring slots of every row and neighbouring table values.
//
// Measured at 512 x 512 x 8 (FP32, P = 2): 106 us with 3-pass lines of 64 threads and
// named barriers, 100 us with the two-pass lines of one warp each (P = 1 with 384
// threads 114 us); a half plane's CTA then took 12.4 kcycles for the forward lines, 16.8
// for the z sum and 8 for the inverse.  With the z sum over even and odd halves: 88 us
// (P = 1 90.5, P = 4 120, P = 8 128; the split kernels 31 + 54 + 31).  What bounds it now:
// 12 warps per SM (162 registers, 107 KB per CTA) in chains of shared and cluster memory
// and dependent arithmetic: issue 41 % active, FMA pipe 28 %, LSU 22 %, DRAM 15 %; its
// bytes would take 24 us, its multiply-adds of the z sum 8.
// Two units per precision (demag_yzy_f32.cu, demag_yzy_f32b.cu, ..: nz <= 4 and
// above), so that they compile in parallel.
#pragma once
#include <cooperative_groups.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "backend_impl.hpp"
#include "demag.cuh"
#include "demag_reg.cuh"
#include "linefft.cuh"
#include "pdl.cuh"
#include "demag_yzy.hpp"

namespace cg = cooperative_groups;

namespace fm {

// table values per (component, offset, kx): tile rows k0 <= R0 / 2
template <typename T, int L> __host__ __device__ constexpr int yzy_row() { return (Lf<T, L>::R0 / 2 + 1) * (L / Lf<T, L>::R0); }
// lines owned by one CTA of a P-CTA cluster
template <int NZ, int P> __host__ __device__ constexpr int yzy_nlh() { return (3 * NZ + P - 1) / P; }
// lines per FFT pass: at most 384 threads in FP32 for a whole plane, 192 for a cluster's
// share of one (168 registers each, the z sum's need, so that two CTAs of 107 KB fit per
// SM), 384 in FP64
template <typename T, int L2, int NZ, int P> __host__ __device__ constexpr int yzy_lpp() {
    constexpr int most = sizeof(T) == 4 && P > 1 ? 192 : 384;
    constexpr int cap = L2 > 32 ? (most / L2 < 15 ? most / L2 : 15) : most / L2;  // named barriers
    constexpr int l = yzy_nlh<NZ, P>() < cap ? yzy_nlh<NZ, P>() : cap;
    constexpr int unit = L2 < 32 ? 32 / L2 : 1;  // whole warps
    return (l + unit - 1) / unit * unit;
}
// rows: the owned lines rounded up to whole passes (the idle line groups of a
// last, partial pass use their own rows as 4-step scratch)
template <typename T, int L2, int NZ, int P> __host__ __device__ constexpr int yzy_rows() {
    return (yzy_nlh<NZ, P>() + yzy_lpp<T, L2, NZ, P>() - 1) / yzy_lpp<T, L2, NZ, P>() * yzy_lpp<T, L2, NZ, P>();
}
template <typename T, int L, int NZ, int P>
__host__ __device__ constexpr size_t yzy_smem() {
    return ((size_t)yzy_rows<T, Lf<T, L>::G, NZ, P>() * Lf<T, L>::TILE + (size_t)Lf<T, L>::TW) * sizeof(cx<T>);
}
constexpr size_t kYzySmemMax = 227 * 1024;
template <typename T, int L, int NZ, int P>
__host__ __device__ constexpr bool yzy_fits() {
    return yzy_smem<T, L, NZ, P>() <= kYzySmemMax;
}
template <typename T, int L, int NZ, int P> __host__ __device__ constexpr int yzy_threads() {
    return yzy_lpp<T, Lf<T, L>::G, NZ, P>() * Lf<T, L>::G;
}

// CTAs per SM: as many as fit the shared memory, registers cut to match
template <typename T, int L, int NZ, int P> __host__ __device__ constexpr int yzy_min_blocks() {
    constexpr int by_smem = (int)(kYzySmemMax / (yzy_smem<T, L, NZ, P>() + 1024));
    constexpr int by_thr = 65536 / (yzy_threads<T, L, NZ, P>() * 168);
    constexpr int m = by_smem < by_thr ? by_smem : by_thr;
    return m < 1 ? 1 : m;
}

template <typename T, int L, int NZ, int P>
__global__ void __launch_bounds__((yzy_threads<T, L, NZ, P>()), (yzy_min_blocks<T, L, NZ, P>())) k_yzy(DemagArgs<T> a) {
    using C = cx<T>;
    constexpr int G = Lf<T, L>::G, TE = Lf<T, L>::TILE, NL = 3 * NZ, NLH = yzy_nlh<NZ, P>();
    constexpr int LPP = yzy_lpp<T, G, NZ, P>(), ROWS = yzy_rows<T, G, NZ, P>(), BT = LPP * G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *S = reinterpret_cast<C *>(smem_raw);
    C *tws = S + ROWS * TE;
    const int h = P > 1 ? (int)cg::this_cluster().block_rank() : 0;
    auto cluster_sync = [&]() {
        if constexpr (P > 1) cg::this_cluster().sync();
        else __syncthreads();
    };
    for (int k = threadIdx.x; k < Lf<T, L>::TW; k += BT) tws[k] = a.twy4[k];
    __syncthreads();  // the transforms have no block barrier
    const int kx = blockIdx.x / P, nkx = a.nkx, ny = a.ny;
    const int qg = threadIdx.x / G, t = threadIdx.x % G;
    {   // only the z sum reads the plane's table (6 NZ rows of yzy_row<T, L>() values): bring
        // it into L2 while the y forward FFTs run, the rows split over the cluster's CTAs
        constexpr int LN = 128 / (int)sizeof(T), ROW = yzy_row<T, L>(), NLN = (ROW + LN - 1) / LN;
        const T *t0 = a.spec + (long long)kx * ROW;
        for (int i = h * BT + threadIdx.x; i < 6 * NZ * NLN; i += P * BT) {
            const int r = i / NLN, j = i - r * NLN;
            const T *p = t0 + (long long)r * nkx * ROW + min(j * LN, ROW - 1);
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        }
    }
    pdl_wait();
    // 1. forward y, LPP lines per pass: inputs y < ny (= L/2; the upper half is the
    // zero padding).  Every thread takes part in every pass (the lines' barriers).
#pragma unroll 1
    for (int r0 = 0; r0 < ROWS; r0 += LPP) {
        const int lr = r0 + qg, q = h * NLH + lr;  // local row, line q = c nz + z
        const bool valid = lr < NLH && q < NL;     // spare rows are scratch
        const C *line1 = a.s1 + ((long long)(valid ? q : 0) * nkx + kx) * ny;  // S1 [c][z][kx][y]
        C *row = S + lr * TE;
        auto in1 = [&](int j) -> C { return j < ny ? line1[j] : mk<T>(0, 0); };
        auto out1 = [&](int k, C v) { row[line_slot<T, L>(k)] = v; };
        line_fwd<L, true>(t, qg, tws, row, in1, out1);
    }
    cluster_sync();
    // 2. direct z convolution of this CTA's ky columns (table and signs as in k_zd)
    {
        C *own[P];  // row 0 of every CTA of the cluster
#pragma unroll
        for (int r = 0; r < P; ++r) {
            if constexpr (P > 1) own[r] = cg::this_cluster().map_shared_rank(S, r);
            else own[r] = S;
        }
        auto cell = [&](int line, int s) -> C & { return own[line / NLH][(line % NLH) * TE + s]; };
        // column i of the plane in slot order: tile row k0 = i / M0, place i % M0.  The
        // table (yzy_table) holds the rows k0 <= R0 / 2 in the same order; a row above is
        // the mirror ky -> L - ky of row R0 - k0, read backwards, with the components odd
        // in y negated.  So neighbouring lanes read neighbouring table values and
        // neighbouring slots of every line.
        constexpr int R0 = Lf<T, L>::R0, M0 = L / R0, LD = Lf<T, L>::LD, ROW = yzy_row<T, L>();
        const int dstr = nkx * ROW, tstr = NZ * dstr;
        constexpr int KC = L / P;  // columns per CTA
        for (int kk = threadIdx.x; kk < KC; kk += BT) {
            const int i = h * KC + kk, k0 = i / M0, idx = i % M0, sl = Lf<T, L>::NP == 1 ? i : k0 * LD + idx;
            const bool mir = 2 * k0 > R0;
            const T sy = mir ? T(-1) : T(1);
            const T *tp = a.spec + ((long long)kx * ROW + (mir ? (R0 - k0) * M0 + (M0 - 1 - idx) : i));
            T tab[6][NZ];  // the column's table entries, all in flight at once
#pragma unroll
            for (int e = 0; e < 6; ++e)
#pragma unroll
                for (int d = 0; d < NZ; ++d) tab[e][d] = e < 4 || d > 0 ? __ldg(tp + e * tstr + d * dstr) : T(0);
            C mx[NZ], my[NZ], mz[NZ];
#pragma unroll
            for (int z = 0; z < NZ; ++z) {
                mx[z] = cell(z, sl);
                my[z] = cell(NZ + z, sl);
                my[z].x *= sy; my[z].y *= sy;  // xy and yz change sign with ky: so do My and Hy
                const C v = cell(2 * NZ + z, sl);
                mz[z] = mk<T>(v.y, -v.x);  // -i Mz
            }
            zsum_column<NZ, T>(mx, my, mz, [&](int e, int d) { return tab[e][d]; });
#pragma unroll
            for (int z = 0; z < NZ; ++z) {
                cell(z, sl) = mx[z];
                cell(NZ + z, sl) = mk<T>(my[z].x * sy, my[z].y * sy);
                cell(2 * NZ + z, sl) = mk<T>(-mz[z].y, mz[z].x);  // Hz = i Hz'
            }
        }
    }
    cluster_sync();  // after this no CTA touches another's shared memory
    // 3. inverse y, keep y < ny
#pragma unroll 1
    for (int r0 = 0; r0 < ROWS; r0 += LPP) {
        const int lr = r0 + qg, q = h * NLH + lr;
        const bool valid = lr < NLH && q < NL;
        C *line1 = a.s1 + ((long long)(valid ? q : 0) * nkx + kx) * ny;
        C *row = S + lr * TE;
        auto in3 = [&](int k) -> C { return row[line_slot<T, L>(k)]; };
        auto out3 = [&](int n, C v) { if (valid && n < ny) line1[n] = v; };
        line_inv<L, true>(t, qg, tws, row, in3, out3);
    }
}

template <int N> using YzyIC = std::integral_constant<int, N>;

// Ly in 256..1024 and NZ of nz as compile-time values: nz <= 4 in the units with
// YZY_HALF 0, above in those with 1
// static: the two halves have different bodies
template <class F>
static void yzy_dispatch(int Ly, int nz, F &&f) {
    auto nzs = [&](auto l) {
        switch (nz) {
#if YZY_HALF == 0
            case 1: f(l, YzyIC<1>{}); break;
            case 2: f(l, YzyIC<2>{}); break;
            case 3: f(l, YzyIC<3>{}); break;
            case 4: f(l, YzyIC<4>{}); break;
#else
            case 5: f(l, YzyIC<5>{}); break;
            case 6: f(l, YzyIC<6>{}); break;
            case 7: f(l, YzyIC<7>{}); break;
            case 8: f(l, YzyIC<8>{}); break;
#endif
            default: break;
        }
    };
    switch (Ly) {
        case 256: nzs(YzyIC<256>{}); break;
        case 512: nzs(YzyIC<512>{}); break;
        case 1024: nzs(YzyIC<1024>{}); break;
        default: break;  // other lengths: the split kernels
    }
}

template <class F>
void yzy_with_p(int P, F &&f) {
    switch (P) {
        case 1: f(YzyIC<1>{}); break;
        case 2: f(YzyIC<2>{}); break;
        case 4: f(YzyIC<4>{}); break;
        case 8: f(YzyIC<8>{}); break;
        default: break;
    }
}

template <typename T, int L, int NZ, int P>
cudaLaunchConfig_t yzy_config(const Backend &b, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(b.nkx * P));
    cfg.blockDim = dim3((unsigned)yzy_threads<T, L, NZ, P>());
    cfg.dynamicSmemBytes = yzy_smem<T, L, NZ, P>();
    cfg.stream = b.stream;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = P > 1 ? attr : attr + 1;
    cfg.numAttrs = P > 1 ? 2 : 1;
    return cfg;
}

template <typename T>
static bool yzy_configure_t(Backend &b) {
    b.use_yzy = false;
    b.yzy_P = 0;
    const char *off = std::getenv("FULLMAG_FDM_YZY");
    if (b.thin || !b.zdirect || (off && std::strcmp(off, "off") == 0)) return true;
    // cluster size: FULLMAG_FDM_YZY_P, else the smallest P whose CTA fits twice per SM
    int want = 0;
    if (const char *p = std::getenv("FULLMAG_FDM_YZY_P")) want = std::atoi(p);
    // FP64 only on request: at 512 x 512 x 8 it takes 329, 415 and 387 us with P = 2, 4 and
    // 8 (P = 1 does not fit) against 216 us for the three split kernels, at 256 x 256 x 8
    // 88 us with P = 1 against 65; only 4 planes and fewer, where one CTA holds the plane,
    // are faster fused (512 x 512 x 4: 88 against 111 us)
    if (sizeof(T) == 8 && !want) return true;
    yzy_dispatch(b.Ly, b.nz, [&](auto l, auto nzc) {
        constexpr int L = decltype(l)::value, NZ = decltype(nzc)::value;
        for (int P : {1, 2, 4, 8}) {
            if (b.use_yzy || (want && P != want)) continue;
            yzy_with_p(P, [&](auto pc) {
                constexpr int PP = decltype(pc)::value;
                if constexpr (yzy_fits<T, L, NZ, PP>()) {
                    constexpr size_t smem = yzy_smem<T, L, NZ, PP>();
                    if (!want && PP < 8 && smem > kYzySmemMax / 2) return;  // one CTA per SM: try a larger cluster
                    auto kern = k_yzy<T, L, NZ, PP>;
                    // the largest shared-memory carveout, so that two CTAs fit per SM
                    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
                        cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                             (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess) {
                        cudaGetLastError();
                        return;
                    }
                    if constexpr (PP > 1) {
                        cudaLaunchAttribute attr[2];
                        cudaLaunchConfig_t cfg = yzy_config<T, L, NZ, PP>(b, attr);
                        int nclusters = 0;
                        if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) != cudaSuccess || nclusters < 1) {
                            cudaGetLastError();
                            return;
                        }
                    }
                    b.yzy_P = PP;
                    b.use_yzy = true;
                }
            });
        }
    });
    return true;
}

template <typename T>
static bool yzy_launch_t(Backend &b, const DemagArgs<T> &a) {
    yzy_dispatch(b.Ly, b.nz, [&](auto l, auto nzc) {
        constexpr int L = decltype(l)::value, NZ = decltype(nzc)::value;
        yzy_with_p(b.yzy_P, [&](auto pc) {
            constexpr int PP = decltype(pc)::value;
            if constexpr (yzy_fits<T, L, NZ, PP>()) {
                cudaLaunchAttribute attr[2];
                cudaLaunchConfig_t cfg = yzy_config<T, L, NZ, PP>(b, attr);
                cudaLaunchKernelEx(&cfg, k_yzy<T, L, NZ, PP>, a);
            }
        });
    });
    return true;
}

// Values per row of the fused pass's z table for length Ly (0: other lengths).
template <typename T> static int yzy_table_row(int Ly) {
    int r = 0;
    yzy_dispatch(Ly, 1, [&](auto l, auto) { r = yzy_row<T, decltype(l)::value>(); });
    return r;
}

// One row of the direct z table (ky = 0..Ly/2) in the order k_yzy reads it: place
// i = k0 M0 + idx of tile row k0 <= R0 / 2 holds the frequency in that slot, those
// above Ly / 2 by the ky mirror with `sign` (-1 for components odd in y).
template <typename T>
static void yzy_table(int Ly, const double *src, double sign, T *dst) {
    yzy_dispatch(Ly, 1, [&](auto l, auto) {
        constexpr int L = decltype(l)::value, R0 = Lf<T, L>::R0, M0 = L / R0, M1 = Lf<T, L>::NP == 3 ? Lf<T, L>::M1 : 1;
        constexpr int R1 = M0 / M1;
        for (int k0 = 0; k0 <= R0 / 2; ++k0)
            for (int idx = 0; idx < M0; ++idx) {
                const int ky = k0 + R0 * (idx / M1 + R1 * (idx % M1));
                dst[k0 * M0 + idx] = (T)(ky > L / 2 ? sign * src[L - ky] : src[ky]);
            }
    });
}

}  // namespace fm
