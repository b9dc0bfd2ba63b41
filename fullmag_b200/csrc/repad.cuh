// repad.cuh — an octant's in-plane lengths changed from 2n to the line-FFT lengths, on
// the device, when a handle is created.
//
// One axis of a table [r][k <= n] of spectra of length 2n, even or odd in k: back to the
// offsets |d| < n (the wrapped entry d = n reaches no physical cell), zeros between, and
// forward at length L >= 2n to [r][k <= L/2].  Both transforms are shared-memory FFTs
// (fft.cuh) in FP64 of two rows at once: even rows have real transforms, odd ones
// imaginary, so a pair packed as real and imaginary part comes apart without a sum.
// Creating an FP32 handle from supplied spectra, with these transforms by host FFTs, here,
// and without padding: 160 x 160 x 16 411, 31 and 25 ms; 2000 x 2000 x 4 9.5, 0.94 and
// 0.73 s; 1280 x 1280 x 12 19.9, 1.0 and 0.75 s.
#pragma once

#include "fft.cuh"

namespace fm {

struct RepadArgs {
    const double *src;
    double *dst;
    LinePlan p0, p1;       // lengths 2n and L
    int n, odd, lines;     // lines: row pairs per block
    long long rows;
    int inner, st;         // row r starts at (r / inner) so + r % inner; entries st apart
    long long so, dso;     // so: of src, dso: of dst
};

__global__ void __launch_bounds__(256) k_repad(RepadArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = a.n, L0 = 2 * n, L = a.p1.L, ld = L + 1, R = 2 * a.lines;
    double2 *tw = reinterpret_cast<double2 *>(smem_raw);
    double2 *A = tw + L, *B = A + a.lines * ld;
    const long long r0 = (long long)blockIdx.x * R;
    const int nr = (int)min((long long)R, a.rows - r0);
    auto twiddles = [&](int len) {
        for (int k = threadIdx.x; k < len; k += blockDim.x) {
            double s, c;
            sincospi(2.0 * (double)k / (double)len, &s, &c);
            tw[k] = mk<double>(c, -s);
        }
    };
    // entry (r, k) of item u of R rows of m entries: neighbouring threads at neighbouring addresses
    auto item = [&](int u, int m, int &r, int &k) {
        if (a.st == 1) { r = u / m; k = u - r * m; }
        else { k = u / R; r = u - k * R; }
    };
    auto at = [&](int r, long long so) { const long long g = r0 + r; return (g / a.inner) * so + g % a.inner; };

    twiddles(L0);
    for (int u = threadIdx.x; u < R * (n + 1); u += blockDim.x) {
        int r, k;
        item(u, n + 1, r, k);
        const bool edge = k == 0 || k == n;
        double v = 0.0;
        if (r < nr && !(a.odd && edge)) v = a.src[at(r, a.so) + (long long)k * a.st];
        double *line = reinterpret_cast<double *>(A + (r >> 1) * ld) + (r & 1);
        line[2 * k] = v;
        if (!edge) line[2 * (L0 - k)] = a.odd ? -v : v;
    }
    __syncthreads();
    double2 *f = fft_lines<false>(A, B, a.p0, a.lines, ld, tw), *g = f == A ? B : A;
    twiddles(L);  // the transform ended with a barrier
    const double s = 1.0 / (double)L0;
    for (int u = threadIdx.x; u < a.lines * L; u += blockDim.x) {
        const int q = u / L, d = u - q * L, e = d < n ? d : L - d;
        double2 v = mk<double>(0.0, 0.0);
        if (e < n && !(a.odd && d == 0)) {
            const double2 z = f[q * ld + e];
            const double so = d < n ? s : -s;  // odd rows: the pair's transform is i F_a - F_b
            v = a.odd ? mk<double>(-z.y * so, z.x * so) : mk<double>(z.x * s, z.y * s);
        }
        g[q * ld + d] = v;
    }
    __syncthreads();
    const double2 *o = fft_lines<false>(g, f, a.p1, a.lines, ld, tw);
    const int m = L / 2 + 1;
    for (int u = threadIdx.x; u < R * m; u += blockDim.x) {
        int r, k;
        item(u, m, r, k);
        if (r >= nr) continue;
        const double2 z = o[(r >> 1) * ld + k];
        double v = (r & 1) ? z.y : z.x;
        if (a.odd) v = (k == 0 || k == L / 2) ? 0.0 : ((r & 1) ? z.x : -z.y);  // -i S_a + S_b
        a.dst[at(r, a.dso) + (long long)k * a.st] = v;
    }
}

// Rows [r][ky < KY] -> the passes' table rows of W values: place i holds entry |map[i]| - 1
// (negated where map[i] < 0 and `neg`), or 0 where map[i] = 0.
template <typename T>
__global__ void __launch_bounds__(256) k_table_rows(const double *src, T *out, const int *map, int KY, int W,
                                                    long long rows, bool neg) {
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < rows * W; u += (long long)gridDim.x * blockDim.x) {
        const long long r = u / W;
        const int e = map[u - r * W];
        double v = 0.0;
        if (e != 0) v = src[r * KY + (e < 0 ? -e : e) - 1];
        out[u] = (T)(e < 0 && neg ? -v : v);
    }
}

}  // namespace fm
