// linefft.cuh — complex line FFTs of 2..4096 points, a few values per thread.
//
// A line of L = R0 R1 R2 points (R1 = R2 = 1 for the shortest) is transformed
// by a group of G threads in one to three passes of register DFTs of sizes R0,
// R1, R2 (powers of two, or three times one, at most 32), with the values
// exchanged in place in the line's shared-memory tile:
//   forward (decimation in frequency), n = j + M0 i, M0 = R1 R2, M1 = R2:
//     pass 0  y[k0][j]      = W_L^{j k0}   sum_i x[j + M0 i] W_R0^{i k0}
//     pass 1  z[k0][k1][j'] = W_M0^{j' k1} sum_i y[k0][j' + M1 i] W_R1^{i k1}
//     pass 2  X[k0 + R0 (k1 + R1 k2)] = sum_j' z[k0][k1][j'] W_R2^{j' k2}
//   inverse (decimation in time): the transposed network, passes 2, 1, 0.
// Every pass reads and writes the slots of its own items, so a pass needs one
// barrier of the line's G threads before the next (a warp barrier for G <= 32,
// a named barrier for longer lines) and never one of the whole block.  The
// forward transform may leave the spectrum where it lies (frequency k at
// line_slot(k)) and the inverse starts from there, which saves the reordering
// round trip wherever the product with the tensor is taken in shared memory.
//
// 4 to 16 values per thread (24 at 1536 points, 32 at FP32's 1024) instead of 32 to
// 64: the transforms are bound by latency (shared-memory and FP chains), not by issue
// slots or bandwidth, so what counts is the number of warps an SM can hold; at 2048 FP32
// points a thread needs 61 to 64 registers where the two-pass 64 x 32 form needed 168 to 242.
//
// Zero padding: HALF inputs n >= L/2 are zero and HALF outputs n >= L/2 are not
// wanted; both fold away at compile time (R0 is even).
//
// All arithmetic is written with explicitly rounded operations, so every kernel
// that runs one of these transforms gives the same bits.
#pragma once

#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace fm {

// ---------------------------------------------------------------------------
// compile-time cos / sin (2 pi k / n) by octant reduction and Taylor series
// ---------------------------------------------------------------------------
constexpr double ct_taylor_cos(double x) {
    double s = 0.0, t = 1.0;
    const double x2 = x * x;
    double term[12] = {};
    for (int i = 0; i < 12; ++i) { term[i] = t; t = -t * x2 / (double)((2 * i + 1) * (2 * i + 2)); }
    for (int i = 11; i >= 0; --i) s += term[i];
    return s;
}
constexpr double ct_taylor_sin(double x) {
    double s = 0.0, t = x;
    const double x2 = x * x;
    double term[12] = {};
    for (int i = 0; i < 12; ++i) { term[i] = t; t = -t * x2 / (double)((2 * i + 2) * (2 * i + 3)); }
    for (int i = 11; i >= 0; --i) s += term[i];
    return s;
}
// cos(2 pi p / q), 0 <= p / q <= 1/4
constexpr double ct_cos_q(int p, int q) {
    return 8 * p <= q ? ct_taylor_cos(2.0 * kPi * (double)p / (double)q)
                      : ct_taylor_sin(2.0 * kPi * (double)(q - 4 * p) / (double)(4 * q));
}
constexpr double ct_cos(int k, int n) {
    k = ((k % n) + n) % n;
    if (2 * k > n) k = n - k;
    return 4 * k <= n ? ct_cos_q(k, n) : -ct_cos_q(n - 2 * k, 2 * n);
}
constexpr double ct_sin(int k, int n) { return ct_cos(4 * k - n, 4 * n); }  // cos(a - pi / 2)

// explicitly rounded complex arithmetic
__device__ __forceinline__ float lf_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double lf_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float lf_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double lf_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float2 lf_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 lf_sub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ double2 lf_add(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 lf_sub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
// a w (forward) or a conj(w) (inverse)
template <bool INV, typename C, typename T>
__device__ __forceinline__ C lf_mulw(C a, T wx, T wy) {
    C r;
    if (INV) {
        r.x = lf_fma(a.x, wx, lf_mul(a.y, wy));
        r.y = lf_fma(a.y, wx, -lf_mul(a.x, wy));
    } else {
        r.x = lf_fma(a.x, wx, -lf_mul(a.y, wy));
        r.y = lf_fma(a.y, wx, lf_mul(a.x, wy));
    }
    return r;
}


template <int R> __host__ __device__ constexpr bool lf_pow2() { return (R & (R - 1)) == 0; }
template <int R> __host__ __device__ constexpr int lf_log2() { return R <= 1 ? 0 : 1 + lf_log2<R / 2>(); }

// position of output k after lf_dft<R>
template <int R> __host__ __device__ constexpr int lf_perm(int k) {
    if constexpr (R == 1) return 0;
    else if constexpr (lf_pow2<R>()) {
        int r = 0;
        for (int b = 0; b < lf_log2<R>(); ++b) r |= ((k >> b) & 1) << (lf_log2<R>() - 1 - b);
        return r;
    } else {
        return (k % 3) * (R / 3) + lf_perm<R / 3>(k / 3);
    }
}


template <int N, int K, bool INV, typename C>
__device__ __forceinline__ C lf_tw(C v) {
    using T = decltype(v.x);
    if constexpr (K == 0) return v;
    else if constexpr (4 * K == N) return rot_i<INV>(v);
    else if constexpr (2 * K == N) { C r; r.x = -v.x; r.y = -v.y; return r; }
    else if constexpr (4 * K == 3 * N) return rot_i<!INV>(v);
    else {
        constexpr double cw = ct_cos(K, N), sw = -ct_sin(K, N);
        return lf_mulw<INV>(v, (T)cw, (T)sw);
    }
}

// compile-time loop
template <int I, int N, class F>
__device__ __forceinline__ void lf_for(F &&f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        lf_for<I + 1, N>(f);
    }
}

// R-point DFT in registers, output k at position lf_perm<R>(k).  Powers of two:
// radix-2 decimation in frequency; R = 3 M: a radix-3 level, then M-point DFTs.
template <int R, int O, bool INV, int S, typename C>
__device__ __forceinline__ void lf_dft_at(C (&v)[S]) {
    using T = decltype(v[0].x);
    if constexpr (R == 1) {
    } else if constexpr (lf_pow2<R>()) {
        constexpr int H = R / 2;
        lf_for<0, H>([&](auto j) {
            constexpr int J = decltype(j)::value;
            const C a = v[O + J], b = v[O + J + H];
            v[O + J] = lf_add(a, b);
            v[O + J + H] = lf_tw<R, J, INV>(lf_sub(a, b));
        });
        lf_dft_at<H, O, INV, S>(v);
        lf_dft_at<H, O + H, INV, S>(v);
    } else {
        constexpr int M = R / 3;
        constexpr double hs = 0.86602540378443864676;  // sin(pi / 3)
        lf_for<0, M>([&](auto j) {
            constexpr int J = decltype(j)::value;
            const C a = v[O + J], b = v[O + J + M], c = v[O + J + 2 * M];
            const C sm = lf_add(b, c), df = rot_i<INV>(lf_sub(b, c));
            C t, x1, x2;
            t.x = lf_fma(T(-0.5), sm.x, a.x);
            t.y = lf_fma(T(-0.5), sm.y, a.y);
            x1.x = lf_fma((T)hs, df.x, t.x);
            x1.y = lf_fma((T)hs, df.y, t.y);
            x2.x = lf_fma((T)-hs, df.x, t.x);
            x2.y = lf_fma((T)-hs, df.y, t.y);
            v[O + J] = lf_add(a, sm);
            v[O + J + M] = lf_tw<R, J, INV>(x1);
            v[O + J + 2 * M] = lf_tw<R, (2 * J) % R, INV>(x2);
        });
        lf_dft_at<M, O, INV, S>(v);
        lf_dft_at<M, O + M, INV, S>(v);
        lf_dft_at<M, O + 2 * M, INV, S>(v);
    }
}
template <int R, bool INV, typename C>
__device__ __forceinline__ void lf_dft(C (&v)[R]) { lf_dft_at<R, 0, INV, R>(v); }

// ---------------------------------------------------------------------------
// plans: passes R0 x R1 x R2 and threads per line.  G <= 32 divides 32 (a line
// lies in one warp); V = L / G values per thread.
// ---------------------------------------------------------------------------
// Longer chains of values per thread cost latency on grids that do not fill the chip,
// fewer cost a third pass; measured per length and precision:
// - FP32 at 1024 points: two passes of 32 values in one warp.  At 512 x 512 x 8 against
//   16 x 8 x 8 on 64 threads: y passes 31.2 against 33.2 us, x forward 24.2 / 25.6, x
//   inverse 29.2 / 27.5, the fused plane pass 100 / 106 (its lines then need no barrier).
// - FP32 at 256: 16 x 16 on 16 threads; 4 x 8 x 8 on 32 the same alone, but 14.7 against
//   10.7 us in the fused plane pass of 128 x 128 x 8.
// - elsewhere 8 to 12 values per thread against 16 to 24: 300 x 180 x 5 masked FP32 143 ->
//   116 us per Heun step, 256 x 256 FP32 54 -> 37, 90 x 90 x 4 FP32 56 -> 42, 384 x 384 x 8
//   FP64 528 -> 430; 256 x 256 x 8 FP32 105 -> 101.
// - 3072: without it 1025 to 1536 cells went to 4096. Heun step and handle at 4096 and here:
//   1050 x 1050 FP32 510 -> 450 us, 272 -> 215 MB, FP64 976 -> 732 us; 1050 x 1050 x 4 FP32
//   2329 -> 1643 us, 1994 -> 1369 MB (at 2n = 2100: 5431 us, 928 MB).
template <typename T, int L> struct LfPlan;
#define FM_LF_PLAN(L_, R0_, R1_, R2_, G_) \
    template <typename T> struct LfPlan<T, L_> { static constexpr int L = L_, R0 = R0_, R1 = R1_, R2 = R2_, G = G_; }
FM_LF_PLAN(2, 2, 1, 1, 1);
FM_LF_PLAN(4, 4, 1, 1, 1);
FM_LF_PLAN(8, 8, 1, 1, 1);
FM_LF_PLAN(16, 4, 4, 1, 4);
FM_LF_PLAN(32, 8, 4, 1, 4);
FM_LF_PLAN(64, 8, 8, 1, 8);
FM_LF_PLAN(96, 6, 4, 4, 16);
FM_LF_PLAN(128, 4, 4, 8, 16);
FM_LF_PLAN(192, 6, 4, 8, 32);
FM_LF_PLAN(256, 4, 8, 8, 32);
FM_LF_PLAN(384, 6, 8, 8, 32);
FM_LF_PLAN(512, 8, 8, 8, 64);
FM_LF_PLAN(768, 12, 8, 8, 64);
FM_LF_PLAN(1024, 16, 8, 8, 64);
FM_LF_PLAN(1536, 24, 8, 8, 64);
FM_LF_PLAN(2048, 16, 16, 8, 128);
FM_LF_PLAN(3072, 12, 16, 16, 256);
FM_LF_PLAN(4096, 16, 16, 16, 256);
#undef FM_LF_PLAN
template <> struct LfPlan<float, 256> { static constexpr int L = 256, R0 = 16, R1 = 16, R2 = 1, G = 16; };
template <> struct LfPlan<float, 1024> { static constexpr int L = 1024, R0 = 32, R1 = 32, R2 = 1, G = 32; };

// The lengths above; any length >= 2n - 1 gives the linear convolution of n cells.
constexpr int kLfLengths[] = {2, 4, 8, 16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096};
// the smallest of them >= v, or 0
inline int line_length(int v) {
    for (int L : kLfLengths)
        if (L >= v) return L;
    return 0;
}
template <int V> using LfIC = std::integral_constant<int, V>;
// f(integral_constant L); false for other lengths
template <class F>
inline bool with_line(int L, F &&f) {
    switch (L) {
        case 2: f(LfIC<2>{}); return true;
        case 4: f(LfIC<4>{}); return true;
        case 8: f(LfIC<8>{}); return true;
        case 16: f(LfIC<16>{}); return true;
        case 32: f(LfIC<32>{}); return true;
        case 64: f(LfIC<64>{}); return true;
        case 96: f(LfIC<96>{}); return true;
        case 128: f(LfIC<128>{}); return true;
        case 192: f(LfIC<192>{}); return true;
        case 256: f(LfIC<256>{}); return true;
        case 384: f(LfIC<384>{}); return true;
        case 512: f(LfIC<512>{}); return true;
        case 768: f(LfIC<768>{}); return true;
        case 1024: f(LfIC<1024>{}); return true;
        case 1536: f(LfIC<1536>{}); return true;
        case 2048: f(LfIC<2048>{}); return true;
        case 3072: f(LfIC<3072>{}); return true;
        case 4096: f(LfIC<4096>{}); return true;
        default: return false;
    }
}

template <typename T, int L> struct Lf : LfPlan<T, L> {
    using P = LfPlan<T, L>;
    static_assert(P::R0 * P::R1 * P::R2 == L, "line plan");
    static constexpr int NP = P::R1 == 1 ? 1 : P::R2 == 1 ? 2 : 3;  // passes
    static constexpr int M0 = P::R1 * P::R2, M1 = P::R2;
    static constexpr int LD = NP == 1 ? 1 : M0 + 1;                  // tile row stride (odd: distinct banks)
    static constexpr int TILE = NP == 1 ? L : P::R0 * LD;            // complex elements of a line's tile
    static constexpr int TW = L + (NP == 3 ? M0 : 0);                // twiddle table: W_L^{j k0} [k0][j], then W_M0^{j' k1} [k1][j']
};

// where frequency k lies in a line's tile
template <typename T, int L> __device__ __forceinline__ int line_slot(int k) {
    using F = Lf<T, L>;
    if constexpr (F::NP == 1) return k;
    else if constexpr (F::NP == 2) return (k % F::R0) * F::LD + k / F::R0;
    else return (k % F::R0) * F::LD + (k / F::R0 % F::R1) * F::M1 + k / (F::R0 * F::R1);
}

// host: the twiddle table of a length (Lf<T, L>::TW elements)
template <typename T>
inline std::vector<cx<T>> line_twiddles(int L) {
    std::vector<cx<T>> t;
    with_line(L, [&](auto l) {
        using F = Lf<T, decltype(l)::value>;
        t.assign(F::TW, mk<T>(T(1), T(0)));
        for (int k0 = 0; k0 < F::R0; ++k0)
            for (int j = 0; j < F::M0; ++j) {
                const double a = 2.0 * kPi * (double)(k0 * j) / (double)F::L;
                t[k0 * F::M0 + j] = mk<T>((T)std::cos(a), (T)(-std::sin(a)));
            }
        if constexpr (F::NP == 3) {
            for (int k1 = 0; k1 < F::R1; ++k1)
                for (int j = 0; j < F::M1; ++j) {
                    const double a = 2.0 * kPi * (double)(k1 * j) / (double)F::M0;
                    t[F::L + k1 * F::M1 + j] = mk<T>((T)std::cos(a), (T)(-std::sin(a)));
                }
        }
    });
    return t;
}
template <typename T>
inline int line_twiddle_count(int L) {
    int n = 0;
    with_line(L, [&](auto l) { n = Lf<T, decltype(l)::value>::TW; });
    return n;
}

// barrier of the G threads of line group q (of at most 15 groups when G > 32)
template <int G> __device__ __forceinline__ void line_sync(int q) {
    if constexpr (G <= 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(q + 1), "n"(G) : "memory");
}

// Forward: x[n] = in(n), out(k, X[k]); thread t of line group q, the line's tile
// and the twiddle table tw.  HALF: x[n] = 0 for n >= L/2 (in is not called there).
// The tile's previous contents must not be needed by anyone (in may not read it).
template <int L, bool HALF, typename C, class In, class Out>
__device__ __forceinline__ void line_fwd(int t, int q, const C *__restrict__ tw, C *tile, In in, Out out) {
    using T = decltype(C::x);
    using F = Lf<T, L>;
    constexpr int R0 = F::R0, R1 = F::R1, R2 = F::R2, G = F::G, M0 = F::M0, M1 = F::M1, LD = F::LD;
    constexpr int NI = HALF ? R0 / 2 : R0;
    if constexpr (F::NP == 1) {
        C v[R0];
#pragma unroll
        for (int i = 0; i < R0; ++i) { if (i < NI) v[i] = in(i); else { v[i].x = 0; v[i].y = 0; } }
        lf_dft<R0, false>(v);
#pragma unroll
        for (int k = 0; k < R0; ++k) out(k, v[lf_perm<R0>(k)]);
    } else {
        constexpr int B0 = (M0 + G - 1) / G;
        C v[B0][R0];
#pragma unroll
        for (int b = 0; b < B0; ++b) {
            const int j = t + G * b;
#pragma unroll
            for (int i = 0; i < R0; ++i) {
                if (i < NI && (M0 % G == 0 || j < M0)) v[b][i] = in(j + M0 * i);
                else { v[b][i].x = 0; v[b][i].y = 0; }
            }
        }
#pragma unroll
        for (int b = 0; b < B0; ++b) {
            const int j = t + G * b;
            if (M0 % G != 0 && j >= M0) continue;
            lf_dft<R0, false>(v[b]);
#pragma unroll
            for (int k0 = 0; k0 < R0; ++k0) {
                C x = v[b][lf_perm<R0>(k0)];
                if (k0 != 0) {
                    const C w = tw[k0 * M0 + j];
                    x = lf_mulw<false>(x, w.x, w.y);
                }
                tile[k0 * LD + j] = x;
            }
        }
        line_sync<G>(q);
        if constexpr (F::NP == 3) {
            constexpr int NB = R0 * M1, B1 = (NB + G - 1) / G;
#pragma unroll
            for (int b = 0; b < B1; ++b) {
                const int u = t + G * b;
                if (NB % G != 0 && u >= NB) continue;
                const int k0 = u % R0, j = u / R0;
                C *p = tile + k0 * LD + j;
                C y[R1];
#pragma unroll
                for (int i = 0; i < R1; ++i) y[i] = p[M1 * i];
                lf_dft<R1, false>(y);
#pragma unroll
                for (int k1 = 0; k1 < R1; ++k1) {
                    C x = y[lf_perm<R1>(k1)];
                    if (k1 != 0) {
                        const C w = tw[L + k1 * M1 + j];
                        x = lf_mulw<false>(x, w.x, w.y);
                    }
                    p[M1 * k1] = x;
                }
            }
            line_sync<G>(q);
        }
        constexpr int RL = F::NP == 3 ? R2 : R1, NL = L / RL, BL = (NL + G - 1) / G;
#pragma unroll
        for (int b = 0; b < BL; ++b) {
            const int u = t + G * b;
            if (NL % G != 0 && u >= NL) continue;
            const C *p = tile + (F::NP == 3 ? (u % R0) * LD + (u / R0) * M1 : u * LD);
            C y[RL];
#pragma unroll
            for (int i = 0; i < RL; ++i) y[i] = p[i];
            lf_dft<RL, false>(y);
#pragma unroll
            for (int k = 0; k < RL; ++k) out(u + NL * k, y[lf_perm<RL>(k)]);
        }
    }
}

// out(n, x) or, where it takes the output's index within the thread too, out(n, i, x):
// line_out_count<T, L, HALF>() outputs per thread, output i at n = line_out_index(t, i).
template <class Out, typename C>
__device__ __forceinline__ void line_emit(Out &out, int n, int i, C x) {
    if constexpr (std::is_invocable_v<Out &, int, int, C>) out(n, i, x);
    else out(n, x);
}
template <typename T, int L, bool HALF> __host__ __device__ constexpr int line_out_count() {
    using F = Lf<T, L>;
    return (F::NP == 1 ? 1 : (F::M0 + F::G - 1) / F::G) * (HALF ? F::R0 / 2 : F::R0);
}
template <typename T, int L, bool HALF> __device__ __forceinline__ int line_out_index(int t, int i) {
    using F = Lf<T, L>;
    constexpr int NO = HALF ? F::R0 / 2 : F::R0;
    return F::NP == 1 ? i : t + F::G * (i / NO) + F::M0 * (i % NO);
}

// Inverse (unnormalised): X[k] = in(k), out(n, x[n]) for n < L/2 with HALF, else
// all n.  in(k) may read the tile at line_slot(k).
template <int L, bool HALF, typename C, class In, class Out>
__device__ __forceinline__ void line_inv(int t, int q, const C *__restrict__ tw, C *tile, In in, Out out) {
    using T = decltype(C::x);
    using F = Lf<T, L>;
    constexpr int R0 = F::R0, R1 = F::R1, R2 = F::R2, G = F::G, M0 = F::M0, M1 = F::M1, LD = F::LD;
    constexpr int NO = HALF ? R0 / 2 : R0;
    if constexpr (F::NP == 1) {
        C v[R0];
#pragma unroll
        for (int i = 0; i < R0; ++i) v[i] = in(i);
        lf_dft<R0, true>(v);
#pragma unroll
        for (int n = 0; n < NO; ++n) line_emit(out, n, n, v[lf_perm<R0>(n)]);
    } else {
        constexpr int RL = F::NP == 3 ? R2 : R1, NL = L / RL, BL = (NL + G - 1) / G;
        {
            C y[BL][RL];
#pragma unroll
            for (int b = 0; b < BL; ++b) {
                const int u = t + G * b;
#pragma unroll
                for (int k = 0; k < RL; ++k) {
                    if (NL % G == 0 || u < NL) y[b][k] = in(u + NL * k);
                    else { y[b][k].x = 0; y[b][k].y = 0; }
                }
            }
#pragma unroll
            for (int b = 0; b < BL; ++b) {
                const int u = t + G * b;
                if (NL % G != 0 && u >= NL) continue;
                C *p = tile + (F::NP == 3 ? (u % R0) * LD + (u / R0) * M1 : u * LD);
                lf_dft<RL, true>(y[b]);
#pragma unroll
                for (int i = 0; i < RL; ++i) p[i] = y[b][lf_perm<RL>(i)];
            }
        }
        line_sync<G>(q);
        if constexpr (F::NP == 3) {
            constexpr int NB = R0 * M1, B1 = (NB + G - 1) / G;
#pragma unroll
            for (int b = 0; b < B1; ++b) {
                const int u = t + G * b;
                if (NB % G != 0 && u >= NB) continue;
                const int k0 = u % R0, j = u / R0;
                C *p = tile + k0 * LD + j;
                C y[R1];
#pragma unroll
                for (int k1 = 0; k1 < R1; ++k1) {
                    y[k1] = p[M1 * k1];
                    if (k1 != 0) {
                        const C w = tw[L + k1 * M1 + j];
                        y[k1] = lf_mulw<true>(y[k1], w.x, w.y);
                    }
                }
                lf_dft<R1, true>(y);
#pragma unroll
                for (int i = 0; i < R1; ++i) p[M1 * i] = y[lf_perm<R1>(i)];
            }
            line_sync<G>(q);
        }
        constexpr int B0 = (M0 + G - 1) / G;
#pragma unroll
        for (int b = 0; b < B0; ++b) {
            const int j = t + G * b;
            if (M0 % G != 0 && j >= M0) continue;
            C v[R0];
#pragma unroll
            for (int k0 = 0; k0 < R0; ++k0) {
                v[k0] = tile[k0 * LD + j];
                if (k0 != 0) {
                    const C w = tw[k0 * M0 + j];
                    v[k0] = lf_mulw<true>(v[k0], w.x, w.y);
                }
            }
            lf_dft<R0, true>(v);
#pragma unroll
            for (int i = 0; i < NO; ++i) line_emit(out, j + M0 * i, b * NO + i, v[lf_perm<R0>(i)]);
        }
    }
}

}  // namespace fm
