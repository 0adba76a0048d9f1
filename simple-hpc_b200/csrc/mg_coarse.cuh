// mg_coarse.cuh — the coarsest multigrid level (coarse_solve, multigrid.cpp:120-140) with a cell pair
// per thread in registers: remove the mean of b, red-black sweeps until ||b - A x|| < tol ||b|| or 200
// sweeps, remove the mean of x. Included by mg.cu in the double and the float unit.
//
// What bounds it is latency: up to 200 sweeps of two dependent colour passes over few cells. So
//  * each thread owns one cell of each colour, its links, AP and b in registers; only x is in shared
//    memory, one array per colour (the neighbours of 32 consecutive cells of a row are consecutive in
//    the other colour's array: no bank conflicts);
//  * a sweep has two barriers. The neighbour sum that a colour-0 update needs is the one that the
//    residual of the sweep before needs, and a colour-1 cell's residual takes the sum of its own
//    update, so the residual adds no pass;
//  * the stopping test needs no sum while any cell has |r| >= tol ||b||: the sum of squares, in any
//    order, is then at least r^2 (adding non-negative terms never rounds below one of them). That
//    vote rides on the barrier of the next colour-0 pass, whose update is undone when it fails; only
//    then is the norm formed, in the reference's order (each row left to right, then the rows,
//    det_sum, multigrid.cpp:18-34), and compared as the reference compares it. Sweep counts and, in
//    FP64, all bits are the reference's.
// Measured on the float tail at 128^2 (an 8 x 8 solve in one warp, 24 sweeps): 53 -> 37 us for the whole
// tail, and on the double tail at 32^2 (4 x 4, 48 sweeps): 94 -> 63 us, against one warp that formed the
// norm after every sweep; large levels: see the launcher's comment in mg.cu.
#pragma once

#include "common.hpp"

#include <cooperative_groups.h>

namespace sgpu {
namespace {

constexpr int kCoarseSweeps = 200; // the reference's cap (multigrid.cpp:128)

// Layout of the solve's shared memory for a band of `rows` rows of ny cells (of a level of nx rows):
// the row sums, the two broadcast words, the band's values for an ordered sum, x of both colours.
template <class T> struct CoarseSmem {
    double* sums;   // nx row sums
    double* bcast;  // [0] the result of an ordered sum, [1] (as an int) the sweep of the last vote
    double* vals;   // rows x vstride
    T* x[2];        // (rows + 2) x xstride per colour, zero ring included
    int vstride, xstride;
};
__host__ __device__ inline int coarse_hp(int ny) { return (ny + 1) / 2; } // cells of a colour per row, at most
// Threads the solve takes for `rows` rows: one per row and cell pair, in whole warps.
__host__ __device__ inline int coarse_threads(int rows, int ny) { return (rows * coarse_hp(ny) + 31) / 32 * 32; }
template <class T> __host__ __device__ inline int coarse_smem_bytes(int nx, int rows, int ny) {
    return (nx + 2 + rows * (ny | 1)) * 8 + 2 * (rows + 2) * (coarse_hp(ny) + 2) * static_cast<int>(sizeof(T));
}
template <class T> __device__ inline CoarseSmem<T> coarse_smem(void* base, int nx, int rows, int ny) {
    CoarseSmem<T> s;
    s.vstride = ny | 1; // odd: lanes on consecutive rows read distinct banks
    s.xstride = coarse_hp(ny) + 2;
    s.sums = static_cast<double*>(base);
    s.bcast = s.sums + nx;
    s.vals = s.bcast + 2;
    s.x[0] = reinterpret_cast<T*>(s.vals + rows * s.vstride);
    s.x[1] = s.x[0] + (rows + 2) * s.xstride;
    return s;
}

// The threads that solve together: the first nt threads of one CTA (a whole warp, or several on a
// named barrier, so the CTA's other warps need not take part), or every thread of a cluster.
struct CoarseCta {
    static constexpr bool kCluster = false;
    int nt;
    __device__ __forceinline__ void sync() const {
        if (nt == 32) __syncwarp();
        else asm volatile("bar.sync 1, %0;\n" ::"r"(nt) : "memory");
    }
    // a barrier that also tells whether v holds for any thread
    __device__ __forceinline__ bool vote(bool v, int, double*) const {
        if (nt == 32) {
            const bool any = __any_sync(0xffffffffu, v) != 0;
            __syncwarp(); // a vote alone orders no memory
            return any;
        }
        unsigned o;
        asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n"
                     " selp.u32 %0, 1, 0, q;\n}\n"
                     : "=r"(o)
                     : "r"(v ? 1u : 0u), "r"(nt)
                     : "memory");
        return o != 0;
    }
    template <class T> __device__ __forceinline__ T* at(T* p, int) const { return p; }
    __device__ __forceinline__ int rank() const { return 0; }
    __device__ __forceinline__ int size() const { return 1; }
};
struct CoarseCluster {
    static constexpr bool kCluster = true;
    int nt;
    __device__ __forceinline__ void sync() const { cooperative_groups::this_cluster().sync(); }
    // The CTA's vote, then (if it holds) the sweep's number into every CTA's word before the cluster
    // barrier: a word that is not this sweep's was not written in it.
    __device__ __forceinline__ bool vote(bool v, int sweep, double* bcast) const {
        int* word = reinterpret_cast<int*>(bcast + 1);
        const int any = __syncthreads_or(v ? 1 : 0);
        if (any && static_cast<int>(threadIdx.x) < size()) *at(word, static_cast<int>(threadIdx.x)) = sweep;
        sync();
        return *reinterpret_cast<volatile int*>(word) == sweep;
    }
    template <class T> __device__ __forceinline__ T* at(T* p, int r) const {
        return cooperative_groups::this_cluster().map_shared_rank(p, r);
    }
    __device__ __forceinline__ int rank() const {
        return static_cast<int>(cooperative_groups::this_cluster().block_rank());
    }
    __device__ __forceinline__ int size() const {
        return static_cast<int>(cooperative_groups::this_cluster().num_blocks());
    }
};

template <class T> struct CoarseCell {
    T e, w, n, s, ap, b, x;
};

// The update value of a cell from its neighbour sum. Double: b / AP (t0, formed once) + nb / AP, the
// two statements of multigrid.cpp:61-63, y = inverse(AP); float: as rb_value.
__device__ __forceinline__ double coarse_value(double t0, double, double nb, double ap, double y) {
    return t0 + quotient(nb, ap, y);
}
__device__ __forceinline__ float coarse_value(float, float b, float nb, float ap, float) { return rb_value(b, nb, ap); }
__device__ __forceinline__ double coarse_inverse(double ap) { return inverse(ap); }
__device__ __forceinline__ float coarse_inverse(float) { return 0.0f; }
__device__ __forceinline__ double coarse_t0(double b, double ap) { return b / ap; }
__device__ __forceinline__ float coarse_t0(float, float) { return 0.0f; }

// Solve a level of nx x ny cells, this CTA holding rows [i0, i0 + m) (all of them for CoarseCta; at
// least one), `up` the rows of the band above. Every thread of the team calls it. load(I, J) gives a
// cell, store(I, J, x, b) takes the results.
// The caller has made the inputs visible to the team, and syncs before it reads the results.
template <class T, class Team, class Load, class Store>
__device__ void coarse_solve(const Team& tm, int nx, int ny, int i0, int m, int up, double tol,
                             const CoarseSmem<T>& sm, Load load, Store store, int* sweeps_out) {
    const int tid = static_cast<int>(threadIdx.x), hp = coarse_hp(ny);
    const int Il = tid / hp, jj = tid - Il * hp, I = i0 + Il;
    const int J[2] = {2 * jj + (I & 1), 2 * jj + ((I + 1) & 1)}; // this thread's cell of each colour
    const bool ok[2] = {Il < m && J[0] < ny, Il < m && J[1] < ny};
    const int R = tm.size(), rank = tm.rank();
    CoarseCell<T> c[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (ok[k]) c[k] = load(I, J[k]);
        else c[k] = {T(0), T(0), T(0), T(0), T(1), T(0), T(0)};
    }
    tm.sync(); // the loads are done: the shared memory may hold what they read
    for (int q = tid; q < 2 * (m + 2) * sm.xstride; q += tm.nt) sm.x[0][q] = T(0);
    if (tid == 0) *reinterpret_cast<int*>(sm.bcast + 1) = -1;

    // Ordered sum of v (a value per own cell) over the level.
    auto ordered_sum = [&](double va, double vb) {
        if (ok[0]) sm.vals[Il * sm.vstride + J[0]] = va;
        if (ok[1]) sm.vals[Il * sm.vstride + J[1]] = vb;
        tm.sync();
        for (int r = tid; r < m; r += tm.nt) {
            const double* q = sm.vals + r * sm.vstride;
            double a = 0.0;
#pragma unroll 4
            for (int j = 0; j < ny; ++j) a += q[j];
            *tm.at(sm.sums + i0 + r, 0) = a;
        }
        tm.sync();
        if (rank == 0 && tid == 0) {
            double a = 0.0;
#pragma unroll 4
            for (int r = 0; r < nx; ++r) a += sm.sums[r];
            for (int r = 0; r < R; ++r) *tm.at(sm.bcast, r) = a;
        }
        tm.sync();
        return *const_cast<volatile double*>(sm.bcast);
    };
    const double dn = static_cast<double>(nx) * ny;
    const double mb = ordered_sum(c[0].b, c[1].b) / dn;
    c[0].b = static_cast<T>(c[0].b - mb);
    c[1].b = static_cast<T>(c[1].b - mb);
    auto square = [](T v) { return static_cast<double>(v) * static_cast<double>(v); };
    const double bb = ordered_sum(square(c[0].b), square(c[1].b));
    int sweeps = 0;
    if (bb > 0.0) {
        const double bn = sqrt(bb), thr = tol * bn;
        // |r| >= big in any cell: sqrt of the sum of squares is not below thr (the margin covers the
        // rounding of the squares, the sum and the root; the float one that of the bound too). That needs
        // squares of normal size and a bound that T holds: below, the norm is formed after every sweep.
        const T big = thr >= (sizeof(T) == 8 ? 1e-140 : 1e-30)
                          ? static_cast<T>(thr * (sizeof(T) == 8 ? 1.0 + 1e-9 : 1.0 + 1e-6))
                          : static_cast<T>(INFINITY);
        const T t0[2] = {coarse_t0(c[0].b, c[0].ap), coarse_t0(c[1].b, c[1].ap)};
        const T y[2] = {coarse_inverse(c[0].ap), coarse_inverse(c[1].ap)};
        // This thread's cells are element o of each colour's array; the neighbours are o + odd (east),
        // o + odd - 1 (west), o + xstride (south) and o - xstride (north) of the other colour's.
        const int xs = sm.xstride, cs = static_cast<int>(sm.x[1] - sm.x[0]);
        T* const x = sm.x[0];
        const int o = Il < m ? (Il + 1) * xs + jj + 1 : xs + 1;
        const int odd = J[0] & 1;
        // the copies of a band's edge rows in the neighbouring bands
        T *gup = nullptr, *gdn = nullptr;
        if (Team::kCluster && Il == 0 && m > 0 && rank > 0) gup = tm.at(x + (up + 1) * xs + jj + 1, rank - 1);
        if (Team::kCluster && Il == m - 1 && rank < R - 1) gdn = tm.at(x + jj + 1, rank + 1);
        auto put = [&](int k, T v) {
            if (!ok[k]) return;
            x[o + k * cs] = v;
            if (Team::kCluster && gup) gup[k * cs] = v;
            if (Team::kCluster && gdn) gdn[k * cs] = v;
        };
        auto flow = [&](int k) {
            const T* q = x + o + (1 - k) * cs;
            const int e = k ? 1 - odd : odd;
            return c[k].e * q[e] + c[k].w * q[e - 1] + c[k].s * q[xs] + c[k].n * q[-xs];
        };
        put(0, c[0].x);
        put(1, c[1].x);
        tm.sync();
        T f0 = flow(0), r0 = T(0), r1 = T(0);
        while (true) {
            // colour 0 of sweep sweeps + 1, and the test of sweep `sweeps`
            const T v0 = coarse_value(t0[0], c[0].b, f0, c[0].ap, y[0]);
            put(0, v0);
            const bool above = (ok[0] && !(fabs(r0) < big)) || (ok[1] && !(fabs(r1) < big));
            if (!tm.vote(sweeps == 0 || above, sweeps, sm.bcast)) {
                if (sqrt(ordered_sum(square(r0), square(r1))) < thr) break; // x of sweep `sweeps`: colour 0 is not taken over
            }
            c[0].x = v0;
            const T f1 = flow(1);
            c[1].x = coarse_value(t0[1], c[1].b, f1, c[1].ap, y[1]);
            put(1, c[1].x);
            tm.sync();
            if (++sweeps == kCoarseSweeps) break;
            f0 = flow(0);
            r0 = c[0].b - (c[0].ap * c[0].x - f0);
            r1 = c[1].b - (c[1].ap * c[1].x - f1);
        }
    }
    const double mx = ordered_sum(c[0].x, c[1].x) / dn;
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (ok[k]) store(I, J[k], static_cast<T>(c[k].x - mx), c[k].b);
    if (rank == 0 && tid == 0 && sweeps_out) *sweeps_out = sweeps;
}

} // namespace
} // namespace sgpu
