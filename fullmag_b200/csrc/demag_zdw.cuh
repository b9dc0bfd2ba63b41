// demag_zdw.cuh — direct z convolution for 8 < nz <= 16 in FP32 (the split
// y / z / y path of 3-D grids whose z lines are too long for one thread).
//
// k_zd (demag_reg.cuh) sums the whole column in one thread, which for nz = 16
// would be 192 FP32 registers of inputs and outputs alone.  Here the two sets of
// zsum.cuh go to two warps of the block, each with 3 nz/2 inputs and as many sums:
//   - a block of 4 warps takes 64 consecutive columns (col = kx Ly + ky) per
//     iteration of its persistent loop; warps 0-1 sum set S of columns
//     [c0, c0 + 64), warps 2-3 set A of the same columns;
//   - the 64 columns' inputs (3 nz complex) and table entries (6 nz reals) are
//     copied into shared memory with cp.async by all 128 threads, double
//     buffered: the next batch's copies run while this batch is summed, and
//     both sets read one copy; the sums are exchanged in the input slots.
// The sums and their order are k_zd's, so the outputs are bitwise its own.
// What bounds it (1024 x 512 x 16, 250 us, 3.9 TB/s): 8 warps per SM (204 registers, 99 KiB
// per block) whose largest stall is the fetch of the two sets' unrolled code, then
// dependent arithmetic; issue 39 % active, FMA pipe 26 %, DRAM 46 %.  Its bytes would take
// 155 us, its multiply-adds 67.
// Shared memory: 2 buffers x 64 columns x (3 nz complex + 6 nz reals),
// 96 KiB at nz = 16 (99 KiB in the window form below): two blocks per SM.
// No TMA; plain cp.async copies.
//
// Window form (WIN, Ly a multiple of 128): the table is uploaded with its rows
// padded to kyp = KY rounded up to 4 values, and a batch of 64 columns lies in
// one kx row on one side of the ky mirror.  Its entries of one table slot are
// then one window of 68 values that starts on a 16-byte boundary (ky' from ky0,
// or from Ly - ky0 - 64 for a mirrored batch), so every copy of the batch is a
// 16-byte cp.async.cg (no L1 allocation): 12 input and 13 table copies per
// thread in place of 24 + 47 element copies.
#pragma once

#include <algorithm>
#include <type_traits>

#include "backend_impl.hpp"
#include "cpasync.cuh"
#include "demag.cuh"
#include "demag_reg.cuh"
#include "demag_zdw.hpp"

namespace fm {

constexpr int kZdwCols = 64;     // columns per batch
constexpr int kZdwThreads = 128; // 4 warps: 2 column groups of 32 x 2 output halves

constexpr int kZdwWin = 68;      // table window per slot in the window form (values)

// table values per slot in shared memory
template <bool WIN> __host__ __device__ constexpr int zdw_ts() { return WIN ? kZdwWin : kZdwCols; }
template <int NZ, bool WIN> __host__ __device__ constexpr size_t zdw_buf_bytes() {
    return (size_t)kZdwCols * 3 * NZ * sizeof(float2) + (size_t)6 * NZ * zdw_ts<WIN>() * sizeof(float);
}
template <int NZ, bool WIN> __host__ __device__ constexpr size_t zdw_smem() { return 2 * zdw_buf_bytes<NZ, WIN>(); }

// One set (zsum.cuh) of one column: the thread of set S or A reads the column's
// inputs and table entries from the batch buffer (si, st: slot strides kZdwCols and
// TS), the two exchange their sums through the column's input slots, and S stores
// the outputs z < H (and the middle one's x and y for odd nz), A those above (and the
// middle z).  bar: the named barrier of the 64 threads that share 32 columns.
template <int NZ, int TS, bool SETA>
__device__ __forceinline__ void zdw_col(float2 *si, const float *st, float sy, float2 *base, int cols, bool store,
                                        int bar) {
    constexpr int H = NZ / 2, CS = kZdwCols;
    auto group_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory"); };
    float2 x[H + 1], y[H + 1], z[H + 1], mid[3];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        const float2 xa = si[j * CS], xb = si[(NZ - 1 - j) * CS];
        float2 ya = si[(NZ + j) * CS], yb = si[(2 * NZ - 1 - j) * CS];
        const float2 va = si[(2 * NZ + j) * CS], vb = si[(3 * NZ - 1 - j) * CS];
        ya.x *= sy; ya.y *= sy; yb.x *= sy; yb.y *= sy;  // xy and yz change sign with ky: so do My and Hy
        const float2 za = make_float2(va.y, -va.x), zb = make_float2(vb.y, -vb.x);  // -i Mz
        x[j] = SETA ? zs_sub(xa, xb) : zs_add(xa, xb);
        y[j] = SETA ? zs_sub(ya, yb) : zs_add(ya, yb);
        z[j] = SETA ? zs_neg(zs_add(za, zb)) : zs_sub(za, zb);
    }
    if (NZ & 1) {
        mid[0] = si[H * CS];
        mid[1] = si[(NZ + H) * CS];
        mid[1].x *= sy; mid[1].y *= sy;
        const float2 v = si[(2 * NZ + H) * CS];
        mid[2] = make_float2(v.y, -v.x);
    }
    float2 X[H + 1], Y[H + 1], Z[H + 1];
    zsum_set<SETA, NZ, float>(x, y, z, X, Y, Z, mid, [&](int e, int d) { return st[(e * NZ + d) * TS]; });
    group_sync();  // both sets have read the inputs: their slots carry the sums
    float2 *mine = si + (SETA ? 3 * H * CS : 0), *other = si + (SETA ? 0 : 3 * H * CS);
#pragma unroll
    for (int i = 0; i < H; ++i) {
        mine[i * CS] = X[i];
        mine[(H + i) * CS] = Y[i];
        mine[(2 * H + i) * CS] = Z[i];
    }
    group_sync();
    if (!store) return;
    const int cs = NZ * cols;
#pragma unroll
    for (int i = 0; i < H; ++i) {
        const float2 ox = other[i * CS], oy = other[(H + i) * CS], oz = other[(2 * H + i) * CS];
        // S: (S_x + A_x, S_y + A_y, A_z + S_z) at i; A: (S_x - A_x, S_y - A_y, S_z - A_z) at nz - 1 - i; Z of A = -S_z
        const float2 hx = SETA ? zs_sub(ox, X[i]) : zs_add(X[i], ox);
        const float2 hy = SETA ? zs_sub(oy, Y[i]) : zs_add(Y[i], oy);
        const float2 hz = SETA ? zs_neg(zs_add(Z[i], oz)) : zs_sub(Z[i], oz);
        const int o = SETA ? NZ - 1 - i : i;
        base[o * cols] = hx;
        base[cs + o * cols] = make_float2(hy.x * sy, hy.y * sy);
        base[2 * cs + o * cols] = make_float2(-hz.y, hz.x);  // Hz = i Hz'
    }
    if (NZ & 1) {
        if (SETA) {
            base[2 * cs + H * cols] = make_float2(-mid[2].y, mid[2].x);
        } else {
            base[H * cols] = mid[0];
            base[cs + H * cols] = make_float2(mid[1].x * sy, mid[1].y * sy);
        }
    }
}

template <int NZ, bool WIN>
__global__ void __launch_bounds__(kZdwThreads, 2) k_zdw(DemagArgs<float> a, int kyp) {
    constexpr int NM = 3 * NZ, NT = 6 * NZ, CS = kZdwCols, TS = zdw_ts<WIN>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    // 3 NZ nkx Ly and 6 NZ nkx kyp < 2^31 for every supported grid: 32-bit offsets
    const int Ly = a.Ly, KY = a.KY, nkx = a.nkx, cols = nkx * Ly;
    const int dstr = nkx * KY, tstr = NZ * dstr;
    const int nbat = (cols + CS - 1) / CS;
    auto in_buf = [&](int buf) { return reinterpret_cast<float2 *>(smem_raw + buf * zdw_buf_bytes<NZ, WIN>()); };
    auto tab_buf = [&](int buf) { return reinterpret_cast<float *>(in_buf(buf) + NM * CS); };
    auto issue = [&](int bt, int buf) {
        const int c0 = bt * CS;
        if constexpr (WIN) {
            // Ly % 128 == 0: the batch is whole (cols % 64 == 0), in one kx row
            // and on one side of the mirror; inputs: 3 NZ slots x 32 chunks of
            // 16 bytes; table: 6 NZ slots x 17 chunks of its window
            const int kx = c0 / Ly, ky0 = c0 - kx * Ly;
            const int wstart = ky0 >= Ly / 2 ? Ly - ky0 - CS : ky0;
            float2 *di = in_buf(buf);
            for (int q = tid; q < NM * (CS / 2); q += kZdwThreads) {
                const int s = q / (CS / 2), p = q - s * (CS / 2);
                cp_async16(di + s * CS + 2 * p, a.s2 + (s * cols + c0 + 2 * p));
            }
            float *dt = tab_buf(buf);
            for (int q = tid; q < NT * (kZdwWin / 4); q += kZdwThreads) {
                const int t = q / (kZdwWin / 4), p = q - t * (kZdwWin / 4);
                cp_async16(dt + t * kZdwWin + 4 * p, a.spec + ((t * nkx + kx) * kyp + wstart + 4 * p));
            }
        } else {
            // element e = tid + 128 i has column e % 64 = tid % 64 and slot
            // e / 64 = tid / 64 + 2 i; columns past the end are left uncopied
            // (their sums are not stored)
            const int cl_copy = tid % CS, s0 = tid / CS;
            const int col = c0 + cl_copy;
            if (col >= cols) return;
            const int kx = col / Ly, ky = col - kx * Ly;
            const float2 *src = a.s2 + col;
            const unsigned di = (unsigned)__cvta_generic_to_shared(in_buf(buf) + cl_copy);
#pragma unroll
            for (int s = s0; s < NM; s += kZdwThreads / CS)
                cp_async_elem<8>(di + s * CS * (unsigned)sizeof(float2), src + s * cols);
            const float *tp = a.spec + (kx * KY + (ky > Ly / 2 ? Ly - ky : ky));
            const unsigned dt = (unsigned)__cvta_generic_to_shared(tab_buf(buf) + cl_copy);
#pragma unroll
            for (int s = s0; s < NT; s += kZdwThreads / CS) {
                const int c = s / NZ, d = s - c * NZ;
                if (c < 4 || d > 0)  // tau(0) = 0 is not read
                    cp_async_elem<4>(dt + s * CS * (unsigned)sizeof(float), tp + c * tstr + d * dstr);
            }
        }
    };
    const int warp = tid >> 5, lane = tid & 31;
    const int cl = (warp & 1) * 32 + lane, half = warp >> 1;
    pdl_wait();
    int bt = blockIdx.x, buf = 0;
    if (bt < nbat) issue(bt, 0);
    cp_async_commit();
    for (; bt < nbat; bt += gridDim.x, buf ^= 1) {
        if (bt + (int)gridDim.x < nbat) issue(bt + gridDim.x, buf ^ 1);
        cp_async_commit();  // possibly empty: "all but the newest" is this batch
        cp_async_wait_all_but_one();
        __syncthreads();  // every thread's copies of this batch are visible
        const int col = bt * CS + cl;
        const bool ok = col < cols;
        const int kx = ok ? col / Ly : 0, ky = ok ? col - kx * Ly : 0;
        // the column's table entries: its own slot position, or in the window
        // form ky' - wstart (64 - cl for a mirrored batch)
        const int ti = WIN ? ((ky - cl) >= Ly / 2 ? CS - cl : cl) : cl;
        float2 *si = in_buf(buf) + cl;
        const float *st = tab_buf(buf) + ti;
        float2 *base = a.s2 + (ok ? col : 0);
        if (half == 0) zdw_col<NZ, TS, false>(si, st, ky > Ly / 2 ? -1.f : 1.f, base, cols, ok, 1 + (warp & 1));
        else zdw_col<NZ, TS, true>(si, st, ky > Ly / 2 ? -1.f : 1.f, base, cols, ok, 1 + (warp & 1));
        __syncthreads();  // this buffer is refilled by the next iteration's copies
    }
    cp_async_wait_all();
}

template <int N> using ZdwIC = std::integral_constant<int, N>;

// nz = 11 and 13 never get here: their padded length 2 nz has a prime factor > 7
template <class F>
bool zdw_with_nz(int nz, F &&f) {
    switch (nz) {
        case 8: f(ZdwIC<8>{}); return true;
        case 9: f(ZdwIC<9>{}); return true;
        case 10: f(ZdwIC<10>{}); return true;
        case 12: f(ZdwIC<12>{}); return true;
        case 14: f(ZdwIC<14>{}); return true;
        case 15: f(ZdwIC<15>{}); return true;
        case 16: f(ZdwIC<16>{}); return true;
        default: return false;
    }
}

}  // namespace fm
