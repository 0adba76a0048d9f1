// common.hpp — shared host/device definitions of the B200 SIMPLE solver.
#pragma once

#include "../../include/sgpu.h"

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define SGPU_HD __host__ __device__
#else
#define SGPU_HD
#endif

namespace sgpu {

// ---- errors ----

// Exception carrying an sgpu status code; converted to a return value at the C ABI.
struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void set_last_error(const std::string& msg);
int fail(int code, const std::string& msg); // sets the message, returns code
// Kernel launches issued by this library (process-wide, for the benchmark's launch count).
void count_launch();

void params_defaults(sgpu_params_t& p);
void params_finalize(sgpu_params_t& p);
void params_from_config(const std::string& text, sgpu_params_t& p);

#ifdef __CUDACC__
#define SGPU_CUDA(x)                                                                          \
    do {                                                                                      \
        cudaError_t e_ = (x);                                                                 \
        if (e_ != cudaSuccess)                                                                \
            throw ::sgpu::Error(e_ == cudaErrorMemoryAllocation ? SGPU_E_NOMEM : SGPU_E_CUDA, \
                                std::string("GPU error: ") + cudaGetErrorString(e_) +         \
                                    " in " #x);                                               \
    } while (0)
#define SGPU_LAUNCH()                                                                         \
    do {                                                                                      \
        ::sgpu::count_launch();                                                               \
        SGPU_CUDA(cudaGetLastError());                                                        \
    } while (0)

// Once-per-device set-up of a kernel: function attributes (cudaFuncSetAttribute) and occupancy
// queries. CUDA keeps a function's attributes in each device's context, so a process that runs on
// several GPUs must set them on every one. The state is one bit per device ordinal; the first call
// on a device runs init() with that device current, under a mutex, so first calls from several
// host threads are safe. init() returns an int that later calls on that device get back (e.g. the
// resident blocks per SM).
struct PerDeviceOnce {
    static constexpr int kMaxDevices = 64;
    std::mutex mu;
    std::atomic<std::uint64_t> done{0};
    int value[kMaxDevices] = {};
    template <class F> int get(F&& init) {
        int dev = 0;
        SGPU_CUDA(cudaGetDevice(&dev));
        if (dev < 0 || dev >= kMaxDevices) throw Error(SGPU_E_INVALID, "device ordinal above 63");
        const std::uint64_t bit = std::uint64_t{1} << dev;
        if (done.load(std::memory_order_acquire) & bit) return value[dev];
        std::lock_guard<std::mutex> lock(mu);
        if (!(done.load(std::memory_order_relaxed) & bit)) {
            value[dev] = init();
            done.fetch_or(bit, std::memory_order_release);
        }
        return value[dev];
    }
};
#endif

// ---- device layout ----
//
// Every full-grid field is stored row-major with a padded row pitch: element (i, j) of the
// reference's nrows x ncols Field2D is at [i * pitch + j]. The pitch is a multiple of 32 doubles, so
// each row starts on a 256-byte boundary; the padding columns are never read as cells.
struct Grid {
    int nrows = 0, ncols = 0, pitch = 0;
    std::size_t elems() const { return static_cast<std::size_t>(nrows) * pitch; }
    std::size_t bytes() const { return elems() * sizeof(double); }
};

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Inclusive cell range [i0, i1] x [j0, j1] of a kernel, in global (i, j) indices.
struct Range {
    int i0, i1, j0, j1;
    SGPU_HD int rows() const { return i1 >= i0 ? i1 - i0 + 1 : 0; }
    SGPU_HD int cols() const { return j1 >= j0 ? j1 - j0 + 1 : 0; }
};

// What the kernels read from the parameters. The diffusive coefficients depend only on whether a
// cell is in the boundary band, so the host evaluates both variants once (with the expressions of
// diffusive_coefficients, src/coefficients.cpp:41-63; IEEE-exact, no contraction) and the kernels
// add them to the per-cell convective part.
struct DevParams {
    int NX, NY, H, Hx, Hy, nrows, ncols, pitch;
    int ncol;  // momentum colours: 5, or 2 for UDS + order 2 (momentum_u.cpp:70-72)
    int uds;   // convection_scheme == UDS
    int order; // diffusion_order
    double dx, dy, nu, au, av, ap;
    double dband[9]; // diffusive coefficients in the boundary band (and for order 2)
    double dint[9];  // diffusive coefficients elsewhere (order 4)
};

// Multigrid level view (the reference's MGView, include/simple/multigrid.hpp:59-66): element
// (I, J), 0 <= I < nx, 0 <= J < ny, of each array is ptr[I * stride + J]; the pointers address
// interior cell (0, 0) and every neighbour of an interior cell lies inside the allocation.
#ifdef __CUDACC__
// The red-black update value of multigrid.cpp:61-63, x = b / AP; x += nb / AP. The double
// instances keep the reference's two divisions (bit parity); the float instances (the mixed-precision
// V-cycle, where no bit parity applies) divide once, (b + nb) / AP, with the fast single-precision
// division (__fdividef, a reciprocal and a multiply: within 2 ulp for AP of any magnitude the
// operator holds). A smoother of a correction solve inside FP64 defect correction needs no correctly
// rounded quotient, and the IEEE division's instruction sequence is a sizeable share of the level
// kernels' issue slots.
// The double division takes a long path (444 cycles against 116, measured) when any lane's dividend is
// zero, and every first half sweep from x = 0 divides nothing but zeros, so div_sum divides 1 there and
// takes the zero itself: +-0 / AP is that zero for AP > 0. (A red-black pair solve whose idle lanes
// divided 0 by 1 took 1285 cycles a sweep: double tail at 32^2 57 -> 42 us, 37^2 solve 286 -> 176 us.)
__device__ __forceinline__ double div_sum(double t, double nb, double ap) {
    const bool zero = nb == 0.0 && ap > 0.0;
    double n = zero ? 1.0 : nb;
    asm("" : "+d"(n)); // keeps the compiler from seeing that the quotient of a zero is not used
    const double q = n / ap;
    return t + (zero ? nb : q);
}
__device__ __forceinline__ double rb_value(double b, double nb, double ap) { return div_sum(b / ap, nb, ap); }
// Division by an AP that is divided by more than once, from y = inverse(ap) = 1 / AP: if y is correctly
// rounded, q within an ulp of a / AP and r = a - AP q exact, then fma(r, y, q) is a / AP correctly rounded
// (P. Markstein, IBM J. Res. Dev. 34(1), 1990); a y can be two ulps off, so the step is taken twice, the
// first bringing q within one. Five dependent operations, 41 cycles against the division's 113, and no
// branch that keeps two of them from overlapping. The exponent bounds keep y, q and r normal numbers;
// outside them (inverse returns 0 for such an AP), and for infinities and NaN, see quotient_rare.
__device__ __forceinline__ double inverse(double ap) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(ap)); // the sign bit fails the test too
    return (hi >> 20) - 923u <= 200u ? 1.0 / ap : 0.0;             // 2^-100 <= AP < 2^101
}
// The quotient, or slow set where it takes quotient_rare.
__device__ __forceinline__ double quotient_try(double a, double ap, double y, bool& slow) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(a));
    const bool zero = ((hi << 1) | static_cast<unsigned>(__double2loint(a))) == 0u;
    const bool mid = ((hi >> 20) & 0x7ffu) - 123u <= 1800u; // 2^-900 <= |a| < 2^901
    double q = a * y;
    q = __fma_rn(__fma_rn(-ap, q, a), y, q);
    q = __fma_rn(__fma_rn(-ap, q, a), y, q);
    slow |= !(mid || zero) || __double2hiint(y) == 0;
    return zero ? a : q; // AP > 0 keeps a zero's sign
}
// The quotient where quotient_try gave none. A red-black solve of a cavity started from rest has p' falling off
// over hundreds of decades ahead of what the sweeps have reached, so dividends too small for the steps above are
// common there, and the division takes its long path for them (in the level sweeps three in a row: a red-black
// iteration on 1024 x 128, UDS, 20 to 60 iterations from rest 275 -> 243 us, QUICK 400 -> 360). So they are scaled: a 2^300 and its quotient q are normal
// numbers, q 2^-300 rounds once more only where it is subnormal, and that gives another number than one rounding
// only from a q half way between two subnormal ones (q is the rounded quotient and such a point is a number
// itself, so any other q lies on the quotient's side of it), where it divides.
__device__ __forceinline__ double quotient_rare(double a, double ap, double y) {
    asm volatile("" : "+d"(a)); // stays inside the caller's branch
    const unsigned hi = static_cast<unsigned>(__double2hiint(a));
    if (((hi >> 20) & 0x7ffu) < 123u && __double2hiint(y) != 0) {
        const double s = a * 0x1p300;
        double q = s * y;
        q = __fma_rn(__fma_rn(-ap, q, s), y, q);
        q = __fma_rn(__fma_rn(-ap, q, s), y, q);
        const double r = q * 0x1p-300;
        if (fabs(q - r * 0x1p300) != 0x1p-775) return a == 0.0 ? a : r;
    }
    return a / ap;
}
__device__ __forceinline__ double quotient(double a, double ap, double y) {
    bool slow = false;
    double q = quotient_try(a, ap, y, slow);
    if (slow) q = quotient_rare(a, ap, y);
    return q;
}
__device__ __forceinline__ float rb_value(float b, float nb, float ap) {
    return __fdividef(b + nb, ap);
}
#endif

// The four links of one FP32 multigrid cell, read with one 128-bit load.
struct alignas(16) Link4 {
    float e, w, n, s;
};

// One multigrid level (interior origin at AE..r, row stride `stride`). Double levels (the reference's
// bits) keep the links in the arrays AE, AW, AN, AS; float levels (the mixed-precision V-cycle) keep
// them in L4, one record per cell, and leave those four arrays null.
template <class T> struct LevelViewT {
    int nx, ny, stride;
    T *AE, *AW, *AN, *AS, *AP, *b, *x, *r;
    Link4* L4 = nullptr;
};
using LevelView = LevelViewT<double>;
using LevelView32 = LevelViewT<float>;

#ifdef __CUDACC__
template <class T> struct Links {
    T e, w, n, s;
};
// Through the read-only path: for operators that the running kernel does not write.
__device__ __forceinline__ Links<double> links(const LevelViewT<double>& L, int q) {
    return {__ldg(L.AE + q), __ldg(L.AW + q), __ldg(L.AN + q), __ldg(L.AS + q)};
}
__device__ __forceinline__ Links<float> links(const LevelViewT<float>& L, int q) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(L.L4) + q);
    return {v.x, v.y, v.z, v.w};
}
// With plain loads: for operators that the running kernel may itself have formed (set_links).
__device__ __forceinline__ Links<double> links_written(const LevelViewT<double>& L, int q) {
    return {L.AE[q], L.AW[q], L.AN[q], L.AS[q]};
}
__device__ __forceinline__ Links<float> links_written(const LevelViewT<float>& L, int q) {
    const float4 v = reinterpret_cast<const float4*>(L.L4)[q];
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ void set_links(const LevelViewT<double>& L, int q, double e, double w, double n,
                                          double s) {
    L.AE[q] = e;
    L.AW[q] = w;
    L.AN[q] = n;
    L.AS[q] = s;
}
__device__ __forceinline__ void set_links(const LevelViewT<float>& L, int q, float e, float w, float n, float s) {
    reinterpret_cast<float4*>(L.L4)[q] = make_float4(e, w, n, s);
}
#endif

} // namespace sgpu
