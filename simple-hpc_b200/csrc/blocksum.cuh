// blocksum.cuh — deterministic block sums in FP64 (the mixed-precision path's residual sums), and the serial
// chain of the ordered ones.
//
// A fixed xor-shuffle tree inside each warp, then thread 0 adds the warps' sums in warp order. At
// each tree step lane i forms v_i + v_(i^o) and its partner v_(i^o) + v_i, the same bits, so every
// lane of a warp ends with the same value and the result depends only on the inputs and the block
// shape: repeated runs give the same bits, independent of scheduling. No atomics are involved.
#pragma once

namespace sgpu {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum of v over a block of NW full warps (tid: the linear thread index); valid in thread 0.
// s: NW doubles of shared memory. Every thread of the block must call it.
template <int NW>
__device__ __forceinline__ double block_sum(double v, double* s, int tid) {
    v = warp_sum(v);
    if ((tid & 31) == 0) s[tid >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (tid == 0) {
#pragma unroll
        for (int w = 0; w < NW; ++w) t += s[w];
    }
    return t;
}

// The sum of part[0 .. n) as k_sum_partials forms it (value v goes to thread v mod 1024 of 32 warps), by a
// block of 256 threads, each standing for four of those threads: the same bits. Valid in every thread; s: 33
// doubles of shared memory. A kernel whose blocks each need a sum of few partial sums forms it itself
// instead of waiting for a launch that does.
__device__ __forceinline__ double partials_sum256(const double* __restrict__ part, int n, double* s, int tid) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        double a = 0.0;
        for (int i = tid + 256 * k; i < n; i += 1024) a += part[i];
        a = warp_sum(a);
        if ((tid & 31) == 0) s[8 * k + (tid >> 5)] = a;
    }
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 32; ++w) t += s[w];
        s[32] = t;
    }
    __syncthreads();
    return s[32];
}

// The serial sum of v[0 .. n) (ABS: of |v|) continued from a, the reference's order within a row; v is
// 16-byte aligned shared memory. 16 values are loaded, two at a time, while 16 are added.
template <bool ABS = false> __device__ __forceinline__ double ordered_chain(double a, const double* v, int n) {
    double x[16], y[16];
    auto load = [](double (&to)[16], const double* from) {
#pragma unroll
        for (int u = 0; u < 16; u += 2) {
            const double2 d = *reinterpret_cast<const double2*>(from + u);
            to[u] = d.x;
            to[u + 1] = d.y;
        }
    };
    auto add = [&](const double (&from)[16]) {
#pragma unroll
        for (int u = 0; u < 16; ++u) a += ABS ? fabs(from[u]) : from[u];
    };
    int t = 0;
    if (n >= 16) {
        load(x, v);
        for (; t + 48 <= n; t += 32) {
            load(y, v + t + 16);
            add(x);
            load(x, v + t + 32);
            add(y);
        }
        add(x);
        t += 16;
    }
    for (; t < n; ++t) a += ABS ? fabs(v[t]) : v[t];
    return a;
}

} // namespace sgpu
