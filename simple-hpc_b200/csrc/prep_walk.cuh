// prep_walk.cuh — the walk of a momentum assembly (prep) over a strip of 32 columns, by sweep step.
//
// A prep pass reads 13 values of x, the other component and p per cell, works through a long chain and
// writes records that the sweeps read by step: cell (i, j) of colour c at step row i + 2c. So the block's eight
// warps walk down the strip eight steps at a time, a warp per step row and a lane per column: the lane's cell is
// row step - 2c, and the records go out as whole rows straight from registers. The inputs come through
// rings of rows in shared memory, each row copied once per strip, eight steps ahead; what is stored by field row
// (AP, |R|) is collected in a ring and written when a row's last step is done. A lane's row differs from
// its neighbour's by an even number, and two ring rows are a multiple of the 32 banks: no conflicts.
// (Before, a block assembled a tile of field rows from global memory and staged its records in shared memory:
// 23 cycles per issued instruction at 30 warps an SM, waiting for loads; the same with the inputs
// copied ahead was bound by shared-memory wavefronts, twice as many as here, and slower still.)
#pragma once

#include "stencil.cuh"

namespace sgpu {
namespace {

constexpr int kPrepSteps = 8; // step rows per round: the warps of a block
constexpr int kPrepRing = 32; // rows: a round reads 20 and eight more are on their way
constexpr int kPrepPitch = 40;

// OUT: what a cell leaves by field row (a plain struct of up to 16 bytes).
template <bool V, class OUT> struct PrepWalk {
    double x[kPrepRing][kPrepPitch], o[kPrepRing][kPrepPitch], f[kPrepRing][kPrepPitch]; // from columns j0 - 2, j0 + D and j0
    OUT out[kPrepRing][32];
    static constexpr int D = V ? -1 : 0; // v cells read u at j - 1 and j, u cells v at j and j + 1

    // Walks rows [R0, R1) of the columns j0 .. of the update range ur. cell(step, i, j, coefficients,
    // neighbour sum, pressure term, own value) returns the cell's OUT; row(i, j, OUT) stores it.
    template <int NCOL, class Cell, class Row>
    __device__ __forceinline__ void run(const DevParams& p, const double* __restrict__ gx, const double* __restrict__ go,
                                        const double* __restrict__ gf, const Range& ur, int j0, int R0, int R1, Cell cell,
                                        Row row) {
        const int lane = static_cast<int>(threadIdx.x), wy = static_cast<int>(threadIdx.y), j = j0 + lane;
        // the rows that the cells of field row m are the first to read
        auto fetch = [&](int m) {
            if (m + 2 >= R0 - 2 && m + 2 <= R1 + 1) copy_row(x[(m + 2) & (kPrepRing - 1)], 36, gx, p.pitch, m + 2, j0 - 2, ur.j0 - 2, ur.j1 + 2);
            const int mo = m + 1 + D;
            if (mo >= R0 + D && mo <= R1 + D) copy_row(o[mo & (kPrepRing - 1)], 33, go, p.pitch, mo, j0 + D, ur.j0 + D, ur.j1 + 1 + D);
            if (m >= R0 + D && m < R1) copy_row(f[m & (kPrepRing - 1)], 33, gf, p.pitch, m, j0, ur.j0, ur.j1 + 1 + D);
        };
        auto store = [&](int i) {
            if (i >= R0 && i < R1 && j >= ur.j0 && j <= ur.j1) row(i, j, out[i & (kPrepRing - 1)][lane]);
        };
        if (wy < 4) fetch(R0 - 4 + wy);
        fetch(R0 + wy);
        commit();
        int s0 = R0;
        int c = NCOL == 5 ? (2 * (s0 + wy) + j) % 5 : (s0 + wy + j) & 1; // the colour of step s0 + wy in column j
        const int last = R1 - 1 + 2 * (NCOL - 1);
        for (; s0 <= last; s0 += kPrepSteps) {
            wait();
            __syncthreads();
            fetch(s0 + kPrepSteps + wy);
            commit();
            store(s0 - 2 * kPrepSteps + wy); // rows up to s0 - 9 had their last step in the round before
            const int st = s0 + wy, i = st - 2 * c;
            if (j >= ur.j0 && j <= ur.j1 && i >= R0 && i < R1) {
                auto at = [&](double (&a)[kPrepRing][kPrepPitch], int r, int k) { return &a[r & (kPrepRing - 1)][lane + k]; };
                const double *q = at(x, i, 2), *qn = at(x, i - 1, 2), *qs = at(x, i + 1, 2);
                double ue, uw, vn, vs, pt;
                if (!V) { // assemble_u, momentum_u.cpp:12-19, and the pressure term, momentum_u.cpp:51
                    const double *a = at(o, i, 0), *b = at(o, i + 1, 0), *g = at(f, i, 0);
                    ue = (q[0] + q[1]) / 2;
                    uw = (q[0] + q[-1]) / 2;
                    vn = (a[0] + a[1]) / 2;
                    vs = (b[0] + b[1]) / 2;
                    pt = (g[0] - g[1]) * p.dy;
                } else { // assemble_v, momentum_v.cpp:13-19, and :43-47
                    const double *a = at(o, i - 1, 0), *b = at(o, i, 0);
                    ue = (a[1] + b[1]) / 2;
                    uw = (b[0] + a[0]) / 2;
                    vn = (q[0] + qn[0]) / 2;
                    vs = (q[0] + qs[0]) / 2;
                    pt = (*at(f, i, 0) - *at(f, i - 1, 0)) * p.dx;
                }
                const Coef9 k = momentum_coef(p, ue, uw, vn, vs, i, j);
                // nb_sum, momentum_u.cpp:36-41
                const double nb = (k.AE * q[1] + k.AW * q[-1] + k.AN * qn[0] + k.AS * qs[0]) +
                                  (k.AEE * q[2] + k.AWW * q[-2] + k.ANN * *at(x, i - 2, 2) + k.ASS * *at(x, i + 2, 2));
                out[i & (kPrepRing - 1)][lane] = cell(st, i, j, k, nb, pt, q[0]);
            }
            if (NCOL == 5) c = c == 4 ? 0 : c + 1; // 2 * 8 steps on, mod 5
        }
        wait();
        __syncthreads();
        store(s0 - 2 * kPrepSteps + wy);
        store(s0 - kPrepSteps + wy);
    }

private:
    static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
    static __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
    // Columns j .. of row i, as many as the ring row holds and jmax allows: a warp's copies.
    static __device__ __forceinline__ void copy_row(double* dst, int width, const double* src, int pitch, int i, int j, int jmin, int jmax) {
        const int lane = static_cast<int>(threadIdx.x);
        const double* s = src + static_cast<std::size_t>(i) * pitch + j + lane;
        const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst + lane));
        if (j + lane >= jmin && j + lane <= jmax) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(s) : "memory");
        if (32 + lane < width && j + 32 + lane <= jmax)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d + 256), "l"(s + 32) : "memory");
    }
};

// The strips start at a multiple of four columns: whole 32-byte sectors of every array, so that no sector
// is written by two strips, which the L2 would have to complete from memory (4096^2 doubles: 352 us, with strips from
// the range's first column 395).
__host__ __device__ inline int prep_first(const Range& ur) { return ur.j0 & ~3; }
inline int prep_strips(const Range& ur) { return (ur.j1 + 1 - prep_first(ur) + 31) / 32; }
// Rows a block walks: one wave of `resident` blocks, at least a sixteenth of the grid's and 8 to 32:
// short walks on a small grid, which is bound by the latency of each, longer ones on grids that a batch runs
// side by side, where the skew rows count (20 cavities of 64 to 512 cells a side: 53.9 ms, at least 8 rows for all 54.7).
// The rule takes nothing but the grid and the device, since the sums of |R| are formed by block. More and shorter segments
// cost skew rows and spread the writes (4096^2 doubles: 1024 rows 352 us, 512 363, 128 400; 1024^2: 57 rows 28.3 us,
// 28 28.0, 128 27.7).
inline int prep_rows(const Range& ur, int resident) {
    const int want = resident / prep_strips(ur) > 0 ? resident / prep_strips(ur) : 1;
    const int rows = (ur.rows() + want - 1) / want;
    const int least = ur.rows() / 16 > 32 ? 32 : ur.rows() / 16 < kPrepSteps ? kPrepSteps : ur.rows() / 16;
    return rows < least ? least : rows;
}
// Sets the kernel's shared memory on the current device (once per device) and returns the blocks of 256
// threads resident there.
template <class K> int prep_resident(K kernel, int smem, PerDeviceOnce& once) {
    return once.get([&] {
        int dev = 0, sms = 0, n = 0;
        SGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        SGPU_CUDA(cudaGetDevice(&dev));
        SGPU_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        SGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, smem));
        return (n < 1 ? 1 : n) * sms;
    });
}

} // namespace
} // namespace sgpu
