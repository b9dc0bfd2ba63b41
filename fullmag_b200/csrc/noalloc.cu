// noalloc.cu — the demag field for callers that cannot allocate device memory.
//
// fullmag_fdm_demag_field_f64_noalloc computes H_demag = -IFFT(N(k) FFT(Ms m))
// exactly like the stepper's FP64 demag passes (demag_line.cuh), but it makes
// no device allocation: the FFT work arrays (two half-spectrum buffers) live in
// g_fft_scratch, a file-scope __device__ array of
// kNoAllocScratchBytes (32 MiB).  Every GPU that loads this library holds that
// array until the process exits.  The caller owns and passes the inputs (m,
// the Newell octant) and the output (H); the library only launches kernels.
//
// Who needs this: code that runs inside a host framework which owns the
// whole device-memory budget and forbids allocations outside its own
// allocator, and latency-critical loops that must not pay the implicit device
// synchronisation cudaMalloc / cudaFree bring.  Such callers cannot use
// fullmag_fdm_backend_create, which allocates its arena.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <type_traits>

#include "demag_line.hpp"
#include "demag_reg.cuh"
#include "fullmag_fdm.h"
#include "fullmag_fdm_ext.h"
#include "linefft.cuh"

namespace fm {
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;
constexpr int kMaxDevices = 64;

// FFT work arrays of the allocation-free entry point (shared by every call).
static __device__ __align__(256) unsigned char g_fft_scratch[kNoAllocScratchBytes];

// Line-FFT twiddles (linefft.cuh) of every in-plane length this entry point takes,
// filled with the radix-64 constants when a device is set up: as constants they cost a
// call nothing (five fill launches per call took 12 of the 62 us of a 128 x 128 x 8
// field).
constexpr int kTwLengths[] = {2, 4, 8, 16, 32, 64, 128, 256, 512, 1024};
constexpr int kTwElems = 4096;  // >= the sum of their line_twiddle_count
static __device__ double2 g_line_tw[kTwElems];
int tw_offset(int L) {
    int o = 0;
    for (int l : kTwLengths) {
        if (l == L) return o;
        o += line_twiddle_count<double>(l);
    }
    return -1;
}

struct DeviceSlot {
    bool ready = false;
    unsigned char *scratch = nullptr;  // device address of g_fft_scratch on that device
    double2 *tw = nullptr;             // ... and of g_line_tw
};
std::mutex g_mu;
DeviceSlot g_slots[kMaxDevices];

void put_error(char *buf, uint64_t len, const char *msg) {
    if (buf && len > 0) {
        std::strncpy(buf, msg, (size_t)len - 1);
        buf[len - 1] = '\0';
    }
}

// With the device current: resolve the arrays' device addresses (the host-side
// symbols are only stand-ins) on every call, which is cheap, and once per
// device (again if an address changed) fill this file's copies of the radix-64
// and line-FFT twiddle tables.  The upload goes through the legacy default stream from
// pageable memory, which may return before the data reach the device, and a
// caller's non-blocking stream is not ordered after it: the device is
// synchronised once here, before the first kernel can read the tables.
bool setup_device(int dev, unsigned char **out, double2 **tw_out, char *err, uint64_t errlen) {
    std::lock_guard<std::mutex> lock(g_mu);
    DeviceSlot &s = g_slots[dev];
    void *p = nullptr;
    void *ptw = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_fft_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&ptw, g_line_tw);
    if (e != cudaSuccess) {
        char m[256];
        std::snprintf(m, sizeof(m), "cudaGetSymbolAddress(g_fft_scratch): %s", cudaGetErrorString(e));
        put_error(err, errlen, m);
        return false;
    }
    if (!s.ready || s.scratch != p || s.tw != ptw) {
        s.ready = false;
        double2 d[64];
        float2 f[64];
        for (int k = 0; k < 64; ++k) {
            const double a = 2.0 * kPi * (double)k / 64.0;
            d[k] = make_double2(std::cos(a), -std::sin(a));
            f[k] = make_float2((float)d[k].x, (float)d[k].y);
        }
        e = cudaMemcpyToSymbol(c_tw64d, d, sizeof(d));
        if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tw64f, f, sizeof(f));
        try {  // the tables are built in vectors; no exception leaves a C entry
            for (int L : kTwLengths) {
                const std::vector<double2> t = line_twiddles<double>(L);
                if (e == cudaSuccess)
                    e = cudaMemcpyToSymbol(g_line_tw, t.data(), t.size() * sizeof(double2), (size_t)tw_offset(L) * sizeof(double2));
            }
        } catch (const std::bad_alloc &) {
            e = cudaErrorMemoryAllocation;
        }
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            char m[256];
            std::snprintf(m, sizeof(m), "twiddle table upload: %s", cudaGetErrorString(e));
            put_error(err, errlen, m);
            return false;
        }
        s.scratch = static_cast<unsigned char *>(p);
        s.tw = static_cast<double2 *>(ptw);
        s.ready = true;
    }
    *out = s.scratch;
    *tw_out = s.tw;
    return true;
}

bool pow2(int L) { return L >= 2 && (L & (L - 1)) == 0; }

}  // namespace
}  // namespace fm

extern "C" int fullmag_fdm_demag_field_f64_noalloc(uint32_t nx, uint32_t ny, uint32_t nz,
                                                   int thin_film_2d, const double *octant,
                                                   const double *m, double ms, double *h,
                                                   void *stream, char *error_out,
                                                   uint64_t error_out_len) {
    using namespace fm;
    using C = double2;
    if (!octant || !m || !h || nx == 0 || ny == 0 || nz == 0 || !(ms > 0.0)) {
        put_error(error_out, error_out_len, "null pointer, empty grid or non-positive Ms");
        return FULLMAG_FDM_ERR_INVALID;
    }
    // range first, so that the doubled lengths below cannot overflow
    if (nx > 512 || ny > 512 || nz > 8) {
        put_error(error_out, error_out_len,
                  "grid not supported: 2nx and 2ny must be powers of two <= 1024 and 2nz <= 16 (or nz = 1)");
        return FULLMAG_FDM_ERR_INVALID;
    }
    const bool thin = thin_film_2d && nz == 1;
    const int Lx = 2 * (int)nx, Ly = 2 * (int)ny, Lz = thin ? 1 : 2 * (int)nz;
    if (!pow2(Lx) || !pow2(Ly) || Lx > 1024 || Ly > 1024 || (!thin && (!pow2(Lz) || Lz > 16))) {
        put_error(error_out, error_out_len,
                  "grid not supported: 2nx and 2ny must be powers of two <= 1024 and 2nz <= 16 (or nz = 1)");
        return FULLMAG_FDM_ERR_INVALID;
    }
    const int nkx = (int)nx + 1;
    // scratch layout (complex elements): S1 | S2.  The limit also counts 2 Lx + 2 Ly + Lz
    // elements of tables, so that it does not depend on where those are kept
    const size_t s1 = (size_t)3 * nz * nkx * ny, s2 = thin ? 0 : (size_t)3 * nz * nkx * Ly;
    const size_t elems = (size_t)2 * Lx + 2 * Ly + Lz + s1 + s2 + 16;
    const size_t need = elems * sizeof(C);
    if (need > kNoAllocScratchBytes) {
        char msg[256];
        std::snprintf(msg, sizeof(msg),
                      "grid %ux%ux%u needs %zu bytes of FFT scratch; the allocation-free entry point "
                      "holds at most %zu bytes",
                      nx, ny, nz, need, kNoAllocScratchBytes);
        put_error(error_out, error_out_len, msg);
        return FULLMAG_FDM_ERR_INVALID;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        put_error(error_out, error_out_len, "no current CUDA device");
        return FULLMAG_FDM_ERR_CUDA;
    }
    unsigned char *base = nullptr;
    C *tw = nullptr;
    if (!setup_device(dev, &base, &tw, error_out, error_out_len)) return FULLMAG_FDM_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // a launch error left by earlier, unrelated work is not this call's: clear
    // it, so that the check after the launches reports only this call's own
    (void)cudaGetLastError();

    C *ps1 = reinterpret_cast<C *>(base);
    C *ps2 = ps1 + s1;

    DemagArgs<double> a{};
    a.nx = nx; a.ny = ny; a.nz = nz;
    a.n = (long long)nx * ny * nz;
    a.Lx = Lx; a.Ly = Ly; a.Lz = Lz; a.nkx = nkx;
    a.KZ = thin ? 1 : (int)nz + 1;
    a.KY = (int)ny + 1;
    a.twx4 = tw + tw_offset(Lx);
    a.twy4 = tw + tw_offset(Ly);
    a.s1 = ps1; a.s2 = thin ? nullptr : ps2;
    a.spec = octant;
    a.thin6 = thin;  // the octant is the caller's: all six components
    a.m = m;
    a.mask = nullptr;
    a.ms_map = nullptr;
    a.ms = ms;
    a.hd = h;
    a.norm = 1.0 / ((double)Lx * (double)Ly * (double)Lz);

    LineCfg line;
    if (line_setup<double>(line, Lx, Ly, thin, (int)ny, (int)nz, nkx) != cudaSuccess) {
        put_error(error_out, error_out_len, "cudaFuncSetAttribute failed");
        return FULLMAG_FDM_ERR_CUDA;
    }
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    line.pdl = cudaStreamIsCapturing(st, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone;
    line_x_fwd<double>(line, a, st);
    if (thin) {
        line_y_conv<double>(line, a, st);
    } else {
        line_y_fwd<double>(line, a, st);
        const int cols = nkx * Ly;
        const int P = Lz > 8 ? 2 : 1;
        const unsigned gz = (unsigned)std::min<long long>(((long long)cols * P + 127) / 128, 148LL * 64);
        switch (Lz * 10 + P) {
            case 21: k_zc_r<double, 2, 1><<<gz, 128, 0, st>>>(a); break;
            case 41: k_zc_r<double, 4, 1><<<gz, 128, 0, st>>>(a); break;
            case 81: k_zc_r<double, 8, 1><<<gz, 128, 0, st>>>(a); break;
            case 162: k_zc_r<double, 16, 2><<<gz, 128, 0, st>>>(a); break;
            default: break;
        }
        line_y_inv<double>(line, a, st);
    }
    line_x_inv<double>(line, a, st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        char msg[256];
        std::snprintf(msg, sizeof(msg), "kernel launch: %s", cudaGetErrorString(e));
        put_error(error_out, error_out_len, msg);
        return FULLMAG_FDM_ERR_CUDA;
    }
    return FULLMAG_FDM_OK;
}
