// zsum.cuh — the direct z convolution of one (kx, ky) column, summed over the
// even and odd parts of the column.
//
//   H(z) = sum_{z' < N} A(z - z') M(z'),  A = [[c_xx, c_xy, c_xz], [c_xy, c_yy, c_yz],
//                                              [-c_xz, -c_yz, c_zz]] on (Mx, My, -i Mz)
// with c_xx, c_yy, c_zz, c_xy even and c_xz, c_yz odd in z - z' (demag_reg.cuh).
// Reversing z leaves the even part of the matrix alone and negates the odd one,
// so the sums split into two independent halves of N / 2 each: with
// s_j = M(j) + M(N-1-j), a_j = M(j) - M(N-1-j) (j < N/2), the set S takes
// (s_x, s_y, a_z) to (S_x, S_y, A_z) and the set A takes (a_x, a_y, s_z) to
// (A_x, A_y, S_z), H(i), H(N-1-i) = (S_i +- A_i) / 2.  An entry of a half is
// c(i-j) +- c(N-1-i-j), formed on the fly: for N = 8 a column takes 288
// multiply-adds of a real with a complex number, 104 additions of entries and 48
// complex additions instead of 576 multiply-adds; for N = 16 1152 instead of
// 2304.  Halving them took 11 % off k_yzy and 8 % off k_zdw: at 2.05 cycles per complex
// one and scheduler (packed or not) they are 8 of k_yzy's 88 us at 512 x 512 x 8 and 67 of
// k_zdw's 250 at 1024 x 512 x 16, and what bounds those kernels stands there.
// FP32: an entry formed as c(i-j) +- c(N-1-i-j) is rounded once more, the sums half as
// often; the field's rms error against FP64 is 0.81 to 0.99 of the plain sum's (8 grids of
// unchanged lengths, nz = 4 to 16), single maxima 0.82 to 1.08.
// The table holds c / 2 (newell_host.hpp octant_to_z_direct): no scaling here.
//
// For odd N the middle row and column (index N/2) join S (x, y) and A (z).
//
// Entries are visited with i + j = sg ascending over the even sg, then the odd
// ones, and j - i ascending within: the c(j - i) of one parity stay in registers
// and every c(N-1-sg) is read once.  Every kernel that uses these functions gets
// the same bits.
#pragma once

#include "common.cuh"

namespace fm {

__device__ __forceinline__ void zs_fma(float2 &h, float c, float2 m) { h = __ffma2_rn(make_float2(c, c), m, h); }
__device__ __forceinline__ void zs_fma(double2 &h, double c, double2 m) {
    h.x = __fma_rn(c, m.x, h.x);
    h.y = __fma_rn(c, m.y, h.y);
}
__device__ __forceinline__ float zs_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double zs_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float2 zs_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ double2 zs_add(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
template <typename C> __device__ __forceinline__ C zs_neg(C a) { a.x = -a.x; a.y = -a.y; return a; }
template <typename C> __device__ __forceinline__ C zs_sub(C a, C b) { return zs_add(a, zs_neg(b)); }

// One set on its inputs (x, y, z)[j], j < H, into outputs (X, Y, Z)[i]; set S:
// (s_x, s_y, a_z) -> (S_x, S_y, A_z), set A: (a_x, a_y, -s_z) -> (A_x, A_y, -S_z).
// tab(e, d): half the table's entry e (xx, yy, zz, xy, xz, yz) at offset d < N.
// For odd N: S also takes the middle (x, y) in mid[0..1] and gives the middle's
// (Hx, Hy) there, A the middle z in mid[2] and gives its Hz.
template <bool SETA, int N, typename T, typename C, class Tab>
__device__ __forceinline__ void zsum_set(const C (&x)[N / 2 + 1], const C (&y)[N / 2 + 1], const C (&z)[N / 2 + 1],
                                         C (&X)[N / 2 + 1], C (&Y)[N / 2 + 1], C (&Z)[N / 2 + 1], C (&mid)[3],
                                         Tab tab) {
    constexpr int H = N / 2;
    const C zero = mk<T>(T(0), T(0));
#pragma unroll
    for (int i = 0; i <= H; ++i) { X[i] = zero; Y[i] = zero; Z[i] = zero; }
#pragma unroll
    for (int par = 0; par < 2; ++par) {
        T t1[H / 2 + 1][6];  // c(d1) / 2, d1 = par, par + 2, ..
#pragma unroll
        for (int d1 = par; d1 < H; d1 += 2)
#pragma unroll
            for (int e = 0; e < 6; ++e) t1[d1 / 2][e] = (e < 4 || d1 > 0) ? tab(e, d1) : T(0);
#pragma unroll
        for (int sg = par; sg <= 2 * H - 2; sg += 2) {
            const int d2 = N - 1 - sg;
            T t2[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) t2[e] = tab(e, d2);
#pragma unroll
            for (int d1 = par; d1 < H; d1 += 2) {
                if (d1 > sg || d1 > 2 * H - 2 - sg) continue;
                const int i = (sg - d1) / 2, j = (sg + d1) / 2;
                const T *t = t1[d1 / 2];
                // even entries: the sum where S -> S or A -> A of the even kind, else the difference
                const T cxx = zs_add(t[0], SETA ? -t2[0] : t2[0]), cyy = zs_add(t[1], SETA ? -t2[1] : t2[1]);
                const T cxy = zs_add(t[3], SETA ? -t2[3] : t2[3]), czz = zs_add(t[2], SETA ? t2[2] : -t2[2]);
                // odd entries: u = c(d2) + c(d1), v = c(d2) - c(d1)
                const T ux = d1 ? zs_add(t2[4], t[4]) : t2[4], vx = d1 ? zs_add(t2[4], -t[4]) : t2[4];
                const T uy = d1 ? zs_add(t2[5], t[5]) : t2[5], vy = d1 ? zs_add(t2[5], -t[5]) : t2[5];
                {   // outputs i from inputs j
                    const T ax = SETA ? ux : vx, ay = SETA ? uy : vy, bx = SETA ? vx : ux, by = SETA ? vy : uy;
                    zs_fma(X[i], cxx, x[j]); zs_fma(X[i], cxy, y[j]); zs_fma(X[i], ax, z[j]);
                    zs_fma(Y[i], cxy, x[j]); zs_fma(Y[i], cyy, y[j]); zs_fma(Y[i], ay, z[j]);
                    zs_fma(Z[i], bx, x[j]); zs_fma(Z[i], by, y[j]); zs_fma(Z[i], czz, z[j]);
                }
                if (d1 > 0) {  // outputs j from inputs i
                    const T ax = SETA ? vx : ux, ay = SETA ? vy : uy, bx = SETA ? ux : vx, by = SETA ? uy : vy;
                    zs_fma(X[j], cxx, x[i]); zs_fma(X[j], cxy, y[i]); zs_fma(X[j], ax, z[i]);
                    zs_fma(Y[j], cxy, x[i]); zs_fma(Y[j], cyy, y[i]); zs_fma(Y[j], ay, z[i]);
                    zs_fma(Z[j], bx, x[i]); zs_fma(Z[j], by, y[i]); zs_fma(Z[j], czz, z[i]);
                }
            }
        }
    }
    if constexpr (N % 2 == 1) {
        // the middle row and column: full entries c(H - j) = twice the table's
        if constexpr (!SETA) {
            const C mx = mid[0], my = mid[1];
            C hx = zero, hy = zero;
            {
                const T cxx = T(2) * tab(0, 0), cyy = T(2) * tab(1, 0), cxy = T(2) * tab(3, 0);
                zs_fma(hx, cxx, mx); zs_fma(hx, cxy, my);
                zs_fma(hy, cxy, mx); zs_fma(hy, cyy, my);
            }
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const int d = H - j;
                const T cxx = T(2) * tab(0, d), cyy = T(2) * tab(1, d), cxy = T(2) * tab(3, d);
                const T cxz = T(2) * tab(4, d), cyz = T(2) * tab(5, d);
                zs_fma(hx, cxx, x[j]); zs_fma(hx, cxy, y[j]); zs_fma(hx, cxz, z[j]);
                zs_fma(hy, cxy, x[j]); zs_fma(hy, cyy, y[j]); zs_fma(hy, cyz, z[j]);
                zs_fma(X[j], cxx, mx); zs_fma(X[j], cxy, my);
                zs_fma(Y[j], cxy, mx); zs_fma(Y[j], cyy, my);
                zs_fma(Z[j], cxz, mx); zs_fma(Z[j], cyz, my);
            }
            mid[0] = hx;
            mid[1] = hy;
        } else {
            const C nmz = zs_neg(mid[2]);
            C hz = zero;  // minus Hz, as z holds minus s_z
            zs_fma(hz, T(2) * tab(2, 0), nmz);
#pragma unroll
            for (int j = 0; j < H; ++j) {
                const int d = H - j;
                const T czz = T(2) * tab(2, d), cxz = T(2) * tab(4, d), cyz = T(2) * tab(5, d);
                zs_fma(hz, cxz, x[j]); zs_fma(hz, cyz, y[j]); zs_fma(hz, czz, z[j]);
                zs_fma(X[j], cxz, nmz); zs_fma(Y[j], cyz, nmz);
                zs_fma(Z[j], czz, nmz);
            }
            mid[2] = zs_neg(hz);
        }
    }
}

// A whole column in one thread: (mx, my, -i Mz) in, (hx, hy, -i Hz) out in place.
template <int N, typename T, typename C, class Tab>
__device__ __forceinline__ void zsum_column(C (&mx)[N], C (&my)[N], C (&mz)[N], Tab tab) {
    constexpr int H = N / 2;
    C mid[3] = {mx[H], my[H], mz[H]};  // used for odd N
    C x[H + 1], y[H + 1], z[H + 1], SX[H + 1], SY[H + 1], SZ[H + 1];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        x[j] = zs_add(mx[j], mx[N - 1 - j]);
        y[j] = zs_add(my[j], my[N - 1 - j]);
        z[j] = zs_sub(mz[j], mz[N - 1 - j]);
    }
    zsum_set<false, N, T>(x, y, z, SX, SY, SZ, mid, tab);
#pragma unroll
    for (int j = 0; j < H; ++j) {
        x[j] = zs_sub(mx[j], mx[N - 1 - j]);
        y[j] = zs_sub(my[j], my[N - 1 - j]);
        z[j] = zs_neg(zs_add(mz[j], mz[N - 1 - j]));
    }
    C AX[H + 1], AY[H + 1], AZ[H + 1];
    zsum_set<true, N, T>(x, y, z, AX, AY, AZ, mid, tab);
#pragma unroll
    for (int i = 0; i < H; ++i) {
        mx[i] = zs_add(SX[i], AX[i]);
        mx[N - 1 - i] = zs_sub(SX[i], AX[i]);
        my[i] = zs_add(SY[i], AY[i]);
        my[N - 1 - i] = zs_sub(SY[i], AY[i]);
        mz[i] = zs_sub(SZ[i], AZ[i]);                  // A_z + S_z, AZ = -S_z
        mz[N - 1 - i] = zs_neg(zs_add(AZ[i], SZ[i]));  // S_z - A_z
    }
    if constexpr (N % 2 == 1) { mx[H] = mid[0]; my[H] = mid[1]; mz[H] = mid[2]; }
}

}  // namespace fm
