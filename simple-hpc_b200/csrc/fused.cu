// fused.cu — the fast FP64 outer iteration: same bits as the reference, a fraction of the traffic.
//
// Momentum phase (assemble + bc + residual + maxit_inner multicolour sweeps, momentum_u.cpp /
// momentum_v.cpp) without the 9 coefficient arrays:
//  * k_mom_prep computes each cell's coefficients from the velocity at assembly time, writes the
//    residual |R| (ordered sum afterwards), the AP coefficient (the only one assemble_p and correct
//    read) and a frozen copy xF of the velocity, from which every later sweep recomputes the
//    coefficients (convective_coefficients + diffusive_coefficients, coefficients.cpp:15-63).
//  * k_mom_stream runs one whole multicolour sweep (all colours) in one pass over memory. A CTA
//    owns a strip of columns plus a halo and walks it top to bottom; cell (r, j) of colour c is
//    updated at step t = r + 2c. Every stencil neighbour of a cell is updated at least two steps
//    before it (if its colour comes first) or two steps after it (if later), so the update order
//    of each cell relative to its neighbours is exactly the reference's colour order. Rows stream
//    through a shared-memory ring filled by cp.async; halo cells are updated redundantly and only
//    the owned block is written, to a second buffer.
//  * k_mom_prep_rec and k_mom_rec_stream are the same pair with the coefficients stored instead, once per
//    component, in records laid out by sweep step: the sweep reads them (80 B/cell) and is left with a
//    third of the instructions.
//  * k_mom_cluster does both for a small grid, in the shared memory of one thread-block cluster.
// Pressure assembly (assemble_p, pressure.cpp:14-54) is one kernel with the wall zeros folded in.
#include "kernels.hpp"
#include "bulk.cuh"
#include "prep_walk.cuh"
#include "stencil.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <climits>

namespace sgpu {

namespace {

__device__ __forceinline__ std::size_t ix(const DevParams& p, int i, int j) {
    return static_cast<std::size_t>(i) * p.pitch + j;
}

// Coefficients of a u cell (assemble_u, momentum_u.cpp:12-19) from the frozen u and from v.
__device__ __forceinline__ Coef9 coef_u(const DevParams& p, const double* __restrict__ uF,
                                        const double* __restrict__ v, int i, int j) {
    const std::size_t q = ix(p, i, j), ld = p.pitch;
    const double ue = (uF[q] + uF[q + 1]) / 2;
    const double uw = (uF[q] + uF[q - 1]) / 2;
    const double vn = (v[q] + v[q + 1]) / 2;
    const double vs = (v[q + ld] + v[q + ld + 1]) / 2;
    return momentum_coef(p, ue, uw, vn, vs, i, j);
}

// Coefficients of a v cell (assemble_v, momentum_v.cpp:13-19) from u and the frozen v.
__device__ __forceinline__ Coef9 coef_v(const DevParams& p, const double* __restrict__ u,
                                        const double* __restrict__ vF, int i, int j) {
    const std::size_t q = ix(p, i, j), ld = p.pitch;
    const double ue = (u[q - ld] + u[q]) / 2;
    const double uw = (u[q - 1] + u[q - ld - 1]) / 2;
    const double vn = (vF[q] + vF[q - ld]) / 2;
    const double vs = (vF[q] + vF[q + ld]) / 2;
    return momentum_coef(p, ue, uw, vn, vs, i, j);
}

// Residual / copy pass. Grid over the copy range cr (the update range ur widened by the cells the
// coefficient recomputation reads); cells of ur also get |R| and AP.
template <bool V>
__global__ void k_mom_prep(DevParams p, const double* __restrict__ x, const double* __restrict__ oth,
                           const double* __restrict__ pf, double* __restrict__ xF,
                           double* __restrict__ AP, double* __restrict__ cells, Range ur, Range cr) {
    const int j = cr.j0 + static_cast<int>(blockIdx.x * 32 + threadIdx.x);
    const int i = cr.i0 + static_cast<int>(blockIdx.y * 8 + threadIdx.y);
    if (i > cr.i1 || j > cr.j1) return;
    const std::size_t q = ix(p, i, j), ld = p.pitch;
    xF[q] = x[q];
    if (i < ur.i0 || i > ur.i1 || j < ur.j0 || j > ur.j1) return;
    const Coef9 c = V ? coef_v(p, oth, x, i, j) : coef_u(p, x, oth, i, j);
    // nb_sum (momentum_u.cpp:36-41); residual_u / residual_v (momentum_u.cpp:51, momentum_v.cpp:43-47).
    const double nb = (c.AE * x[q + 1] + c.AW * x[q - 1] + c.AN * x[q - ld] + c.AS * x[q + ld]) +
                      (c.AEE * x[q + 2] + c.AWW * x[q - 2] + c.ANN * x[q - 2 * ld] +
                       c.ASS * x[q + 2 * ld]);
    const double pt = V ? (pf[q] - pf[q - ld]) * p.dx : (pf[q] - pf[q + 1]) * p.dy;
    const double R = nb + pt - c.AP * x[q];
    cells[static_cast<std::size_t>(i - ur.i0) * ur.cols() + (j - ur.j0)] = fabs(R);
    AP[q] = c.AP;
}

constexpr int kRing = 32;    // rows held in the shared-memory ring (power of two)
constexpr int kPrefetch = 8; // rows the cp.async ring runs ahead of the rows being read
#ifndef SGPU_STREAM_PF
#define SGPU_STREAM_PF 0
#endif
constexpr int kStreamPF = SGPU_STREAM_PF; // input staging of k_mom_stream (see the kernel)

// The 9 global inputs of one cell's coefficient recomputation and pressure term, read through
// per-thread column pointers (xF, oth, pf already offset by the thread's column) at row offset o.
//   u cell: uF(r, j-1), uF(r, j), uF(r, j+1), v(r, j), v(r, j+1), v(r+1, j), v(r+1, j+1),
//           p(r, j), p(r, j+1)
//   v cell: u(r-1, j), u(r, j), u(r, j-1), u(r-1, j-1), vF(r, j), vF(r-1, j), vF(r+1, j),
//           p(r, j), p(r-1, j)
template <bool V>
__device__ __forceinline__ void load_inputs(const double* __restrict__ xF,
                                            const double* __restrict__ oth,
                                            const double* __restrict__ pf, int o, int ld,
                                            double a[9]) {
    if (!V) {
        const double* f = xF + o;
        const double* g = oth + o;
        const double* h = pf + o;
        a[0] = __ldg(f - 1); a[1] = __ldg(f); a[2] = __ldg(f + 1);
        a[3] = __ldg(g); a[4] = __ldg(g + 1); a[5] = __ldg(g + ld); a[6] = __ldg(g + ld + 1);
        a[7] = __ldg(h); a[8] = __ldg(h + 1);
    } else {
        const double* f = xF + o;
        const double* g = oth + o;
        const double* h = pf + o;
        a[0] = __ldg(g - ld); a[1] = __ldg(g); a[2] = __ldg(g - 1); a[3] = __ldg(g - ld - 1);
        a[4] = __ldg(f); a[5] = __ldg(f - ld); a[6] = __ldg(f + ld);
        a[7] = __ldg(h); a[8] = __ldg(h - ld);
    }
}

// max(0, a) for the coefficient recomputation. The reference's std::max(0.0, a) returns +0.0 for
// a = -0.0, where fmax may return either zero; the sign of that zero never reaches a coefficient,
// because every coefficient adds its diffusive part, which is non-zero or +0.0, to the convective
// part last (coefficients.cpp:5-8), and x + d == x' + d for the two zeros x, x'. NaN gives 0.0 in
// both forms.
__device__ __forceinline__ double mxf(double a) { return fmax(a, 0.0); }

// The 9 coefficients of a momentum cell from its face velocities: convective_coefficients
// (coefficients.cpp:15-39) plus the precomputed diffusive ones (:41-63), specialised on the scheme
// and the diffusion order. Band cells (rare: two rows and two columns) take the UDS / 2nd-order
// branch like the reference; warp_has_band (the same for the whole warp) keeps every other warp
// off that path.
template <bool QUICK, int ORDER>
__device__ __forceinline__ Coef9 coef_spec(const DevParams& p, double ue, double uw, double vn,
                                           double vs, bool band, bool warp_has_band) {
    const double dx = p.dx, dy = p.dy;
    Coef9 c;
    if (QUICK) {
        c.AE = -dy * (-0.75 * mxf(-ue) + 0.375 * mxf(ue) - 0.125 * mxf(-uw));
        c.AW = -dy * (-0.125 * mxf(ue) + 0.375 * mxf(-uw) - 0.75 * mxf(uw));
        c.AN = -dx * (-0.75 * mxf(-vn) + 0.375 * mxf(vn) - 0.125 * mxf(-vs));
        c.AS = -dx * (-0.125 * mxf(vn) + 0.375 * mxf(-vn) - 0.75 * mxf(vs));
        c.AEE = -0.125 * dy * mxf(-ue);
        c.AWW = -0.125 * dy * mxf(uw);
        c.ANN = -0.125 * dx * mxf(-vn);
        c.ASS = -0.125 * dx * mxf(vs);
    } else {
        c.AE = dy * mxf(-ue);
        c.AW = dy * mxf(uw);
        c.AN = dx * mxf(-vn);
        c.AS = dx * mxf(vs);
        c.AEE = c.AWW = c.ANN = c.ASS = 0.0;
    }
    // Diffusive part: the 2nd-order (band) values for ORDER 2, else the 4th-order ones. Indexed
    // directly so the parameter arrays stay in constant space.
#define SGPU_D(k) (ORDER == 2 ? p.dband[k] : p.dint[k])
    c.AP = c.AS + c.AW + c.AN + c.AE + c.ASS + c.AWW + c.ANN + c.AEE;
    c.AE += SGPU_D(0);
    c.AW += SGPU_D(1);
    c.AN += SGPU_D(2);
    c.AS += SGPU_D(3);
    c.AEE += SGPU_D(4);
    c.AWW += SGPU_D(5);
    c.ANN += SGPU_D(6);
    c.ASS += SGPU_D(7);
    c.AP += SGPU_D(8);
#undef SGPU_D
    if (QUICK || ORDER == 4) {
        if (warp_has_band && band) {
            // in_boundary_band: UDS convection and 2nd-order diffusion (coefficients.cpp:20-27, 45-51).
            c.AE = dy * mxf(-ue);
            c.AW = dy * mxf(uw);
            c.AN = dx * mxf(-vn);
            c.AS = dx * mxf(vs);
            c.AP = c.AS + c.AW + c.AN + c.AE + 0.0 + 0.0 + 0.0 + 0.0;
            c.AE += p.dband[0];
            c.AW += p.dband[1];
            c.AN += p.dband[2];
            c.AS += p.dband[3];
            c.AEE = 0.0 + p.dband[4];
            c.AWW = 0.0 + p.dband[5];
            c.ANN = 0.0 + p.dband[6];
            c.ASS = 0.0 + p.dband[7];
            c.AP += p.dband[8];
        }
    }
    return c;
}

__device__ __forceinline__ void prefetch_l1(const double* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// One multicolour sweep of u (V = false) or v (V = true) from xin to xout. NT threads per CTA, one
// column each; the CTA owns W = NT - 4 * NCOL columns starting at blockIdx.x * W and rows
// [blockIdx.y * seg_rows, + seg_rows). For five colours every dependency between two updates is at
// least two steps apart, so two steps run between barriers (SPB = 2). PF selects how the cells'
// global inputs are brought in: 0 = loaded into registers one super-step ahead, 1 = loaded when
// used (more CTAs per SM hide the latency), 2 = their cache lines prefetched into L1 one
// super-step ahead and loaded when used.
template <int NCOL, bool V, int NT, bool QUICK, int ORDER, int PF>
__global__ void __launch_bounds__(NT, PF == 0 ? 2 : 3)
    k_mom_stream(DevParams p, const double* __restrict__ xin, double* __restrict__ xout,
                 const double* __restrict__ xF, const double* __restrict__ oth,
                 const double* __restrict__ pf, int seg_rows) {
    constexpr int SPB = NCOL == 5 ? 2 : 1;       // steps per barrier
    constexpr int HC = 2 * NCOL;                 // halo: a sweep's dependency reach
    constexpr int W = NT - 2 * HC;
    constexpr int A = kPrefetch + SPB + 2;       // rows issued ahead of the first super-step
    static_assert(kPrefetch + 2 * SPB + 1 < kRing - 2 * NCOL, "ring too small for the prefetch");
    extern __shared__ double ring_mem[];
    __shared__ int s_rmin[NCOL], s_rmax[NCOL];
    const int tid = threadIdx.x;
    const int j0 = blockIdx.x * W;
    const int C0 = j0 - HC, C1 = j0 + W + HC; // loaded columns [C0, C1)
    const int col = C0 + tid;
    const int R0 = blockIdx.y * seg_rows;
    const int R1 = min(R0 + seg_rows, p.nrows);
    const int L0 = max(R0 - HC, 0), L1 = min(R1 + HC, p.nrows); // loaded rows [L0, L1)
    const int ld = p.pitch;
    const bool col_in = col >= 0 && col < p.ncols;
    const bool col_out = col_in && col >= j0 && col < j0 + W;
    const int H = p.H;
    // Per colour: the rows a cell of that colour may be updated at (the update range clipped to
    // the window's dependency cone; only cut sides constrain).
    if (tid < NCOL) {
        const int c = tid;
        int lo = V ? H + 1 : H, hi = p.NX + H - 1;
        if (L0 > 0) lo = max(lo, L0 + 2 + 2 * c);
        if (L1 < p.nrows) hi = min(hi, L1 - 3 - 2 * c);
        s_rmin[c] = lo;
        s_rmax[c] = hi;
    }
    // Colours for which this column is updatable (update range and cut columns).
    unsigned colmask = 0;
    {
        const int ju0 = H + 1, ju1 = V ? p.NY + H : p.NY + H - 1;
#pragma unroll
        for (int c = 0; c < NCOL; ++c) {
            bool ok = col >= ju0 && col <= ju1;
            if (C0 > 0) ok = ok && col >= C0 + 2 + 2 * c;
            if (C1 < p.ncols) ok = ok && col <= C1 - 3 - 2 * c;
            colmask |= (ok ? 1u : 0u) << c;
        }
    }
    // Band tests need global indices: in_boundary_band (coefficients.cpp:10-13).
    const bool col_band = col == p.Hy + 1 || col == p.NY + p.Hy;
    const int band_r0 = p.Hx, band_r1 = p.NX + p.Hx - 1;
    const double relax = V ? p.av : p.au;
    const double omr = 1 - relax;
    const double* xFc = xF + col;
    const double* othc = oth + col;
    const double* pfc = pf + col;
    double* ringc = ring_mem + tid; // column tid of ring row k at ringc[k * NT]
    const double* xinc = xin + col;

    int next = L0;
    auto issue = [&]() {
        if (next < L1 && col_in) cp_async(ringc + (next & (kRing - 1)) * NT, xinc + next * ld);
        cp_async_commit();
        ++next;
    };
    auto step_cell = [&](int c, int t, int& r) -> bool {
        r = t - 2 * c;
        return ((colmask >> c) & 1u) && r >= s_rmin[c] && r <= s_rmax[c];
    };
    auto prefetch_cell = [&](int r) {
        const int o = r * ld;
        if (!V) {
            prefetch_l1(xFc + o);
            prefetch_l1(othc + o);
            prefetch_l1(othc + o + ld);
            prefetch_l1(pfc + o);
        } else {
            prefetch_l1(othc + o - ld);
            prefetch_l1(othc + o);
            prefetch_l1(xFc + o - ld);
            prefetch_l1(xFc + o);
            prefetch_l1(xFc + o + ld);
            prefetch_l1(pfc + o - ld);
            prefetch_l1(pfc + o);
        }
    };
    auto is_band = [&](bool ok, int r) { return ok && (col_band || r == band_r1 || r == band_r0); };
    auto update = [&](int r, const double a[9], bool warp_has_band) {
        double ue, uw, vn, vs, pt;
        if (!V) {
            ue = (a[1] + a[2]) / 2;
            uw = (a[1] + a[0]) / 2;
            vn = (a[3] + a[4]) / 2;
            vs = (a[5] + a[6]) / 2;
            pt = (a[7] - a[8]) * p.dy;
        } else {
            ue = (a[0] + a[1]) / 2;
            uw = (a[2] + a[3]) / 2;
            vn = (a[4] + a[5]) / 2;
            vs = (a[4] + a[6]) / 2;
            pt = (a[7] - a[8]) * p.dx;
        }
        const bool band = col_band || r == band_r1 || r == band_r0;
        const Coef9 k = coef_spec<QUICK, ORDER>(p, ue, uw, vn, vs, band, warp_has_band);
        double* rc = ringc + (r & (kRing - 1)) * NT;
        const double xe = rc[1], xw = rc[-1];
        const double xn = ringc[((r - 1) & (kRing - 1)) * NT];
        const double xs = ringc[((r + 1) & (kRing - 1)) * NT];
        // near_sum for two colours (momentum_u.cpp:84-87), nb_sum for five (:36-41).
        double nb = k.AE * xe + k.AW * xw + k.AN * xn + k.AS * xs;
        if (NCOL == 5) {
            const double xee = rc[2], xww = rc[-2];
            const double xnn = ringc[((r - 2) & (kRing - 1)) * NT];
            const double xss = ringc[((r + 2) & (kRing - 1)) * NT];
            nb = nb + (k.AEE * xee + k.AWW * xww + k.ANN * xnn + k.ASS * xss);
        }
        const double xo = rc[0];
        rc[0] = relax * (nb + pt) / k.AP + omr * xo;
    };

    for (int k = 0; k < A; ++k) issue(); // rows L0 .. L0 + A - 1
    __syncthreads();                     // s_rmin / s_rmax

    const int c_start = NCOL == 5 ? (2 * L0 + col + 1000) % 5 : (L0 + col + 1000) & 1;
    auto next_colour = [&](int c, int steps) {
        return NCOL == 5 ? (c + 2 * steps) % 5 : (c + steps) & 1;
    };
    // Row R1 - 1 is written back by the super-step starting at R1 + 2 NCOL - 2 or one later.
    const int t_last = R1 + 2 * NCOL - 2 + (SPB - 1);

    auto write_back = [&](int t) {
#pragma unroll
        for (int s = 0; s < SPB; ++s) {
            const int rw = t - 2 * NCOL + 1 - (SPB - 1) + s;
            if (rw >= R0 && rw < R1 && col_out) xout[col + rw * ld] = ringc[(rw & (kRing - 1)) * NT];
        }
    };

    if (PF == 0) {
        // Register prefetch: two register sets, alternating between consecutive super-steps.
        double bufA[SPB][9], bufB[SPB][9];
        int rA[SPB], rB[SPB];
        bool okA[SPB], okB[SPB];
#pragma unroll
        for (int s = 0; s < SPB; ++s) {
            okA[s] = step_cell(next_colour(c_start, s), L0 + s, rA[s]);
            if (okA[s]) load_inputs<V>(xFc, othc, pfc, rA[s] * ld, ld, bufA[s]);
        }
        auto super_step = [&](int t, int c0, double (&cur)[SPB][9], const int (&rcur)[SPB],
                              const bool (&okcur)[SPB], double (&nxt)[SPB][9], int (&rnxt)[SPB],
                              bool (&oknxt)[SPB]) {
            cp_async_wait<kPrefetch>(); // rows <= t + SPB + 1 have landed (this thread's copies)
            __syncthreads();            // ... everyone's, and the previous super-step's updates
#pragma unroll
            for (int s = 0; s < SPB; ++s) issue();
            const int cn = next_colour(c0, SPB);
#pragma unroll
            for (int s = 0; s < SPB; ++s) {
                oknxt[s] = step_cell(next_colour(cn, s), t + SPB + s, rnxt[s]);
                if (oknxt[s]) load_inputs<V>(xFc, othc, pfc, rnxt[s] * ld, ld, nxt[s]);
            }
#pragma unroll
            for (int s = 0; s < SPB; ++s) {
                const bool wb = __any_sync(0xffffffffu, is_band(okcur[s], rcur[s]));
                if (okcur[s]) update(rcur[s], cur[s], wb);
            }
            write_back(t);
            return cn;
        };
        int c0 = c_start;
        for (int t = L0; t <= t_last; t += 2 * SPB) {
            c0 = super_step(t, c0, bufA, rA, okA, bufB, rB, okB);
            if (t + SPB <= t_last) c0 = super_step(t + SPB, c0, bufB, rB, okB, bufA, rA, okA);
        }
    } else {
        int c0 = c_start;
        if (PF == 2) {
#pragma unroll
            for (int s = 0; s < SPB; ++s) {
                int r;
                if (step_cell(next_colour(c0, s), L0 + s, r)) prefetch_cell(r);
            }
        }
        for (int t = L0; t <= t_last; t += SPB) {
            cp_async_wait<kPrefetch>();
            __syncthreads();
#pragma unroll
            for (int s = 0; s < SPB; ++s) issue();
            const int cn = next_colour(c0, SPB);
            if (PF == 2) {
#pragma unroll
                for (int s = 0; s < SPB; ++s) {
                    int r;
                    if (step_cell(next_colour(cn, s), t + SPB + s, r)) prefetch_cell(r);
                }
            }
            int r[SPB];
            bool ok[SPB];
            double a[SPB][9];
#pragma unroll
            for (int s = 0; s < SPB; ++s) {
                ok[s] = step_cell(next_colour(c0, s), t + s, r[s]);
                if (ok[s]) load_inputs<V>(xFc, othc, pfc, r[s] * ld, ld, a[s]);
            }
#pragma unroll
            for (int s = 0; s < SPB; ++s) {
                const bool wb = __any_sync(0xffffffffu, is_band(ok[s], r[s]));
                if (ok[s]) update(r[s], a[s], wb);
            }
            write_back(t);
            c0 = cn;
        }
    }
    cp_async_wait<0>();
}

// ---- stored coefficients ----
//
// The recomputing sweep is bound by instruction issue (about 400 a cell, half of the slots busy, DRAM at
// 17%), and its CTAs' halo and skew rows cost as much as their own. Records cost 72 B/cell once per
// component and 56 B/cell more per sweep, but a third of the instructions, and up to about 1024^2 they
// stay in L2. Measured, prep and four sweeps of one component: 175 us at 1024^2 and 1400 us at 4096^2,
// against 206 and 1810 us (a sweep: 37 and 262 us against 47 and 390; the prep
// 27 and 350 us against 18 and 260).

// Prep over the update range: |R|, AP and the records (prep_walk.cuh), 350 us at 4096^2
// and 27 at 1024^2; from tiles assembled in global memory 505 and 31. It is bound by memory now (120 B a cell:
// 307 us).
template <int NCOL, bool V>
__global__ void __launch_bounds__(256, 4)
    k_mom_prep_rec(DevParams p, const double* __restrict__ x, const double* __restrict__ oth,
                   const double* __restrict__ pf, double* __restrict__ AP, double* __restrict__ cells, MomRec64 rec,
                   Range ur, int rows) {
    extern __shared__ __align__(16) unsigned char prep_sm[];
    PrepWalk<V, double2>& walk = *reinterpret_cast<PrepWalk<V, double2>*>(prep_sm);
    const int R0 = ur.i0 + static_cast<int>(blockIdx.y) * rows, R1 = min(R0 + rows, ur.i1 + 1);
    walk.template run<NCOL>(
        p, x, oth, pf, ur, prep_first(ur) + static_cast<int>(blockIdx.x) * 32, R0, R1,
        [&](int st, int, int j, const Coef9& c, double nb, double pt, double own) {
            const std::size_t q = static_cast<std::size_t>(st) * p.pitch + j;
            rec.r[0][q] = make_double2(c.AE, c.AW);
            rec.r[1][q] = make_double2(c.AN, c.AS);
            if (NCOL == 5) {
                rec.r[2][q] = make_double2(c.AEE, c.AWW);
                rec.r[3][q] = make_double2(c.ANN, c.ASS);
            }
            rec.r[4][q] = make_double2(c.AP, pt);
            return make_double2(c.AP, fabs(nb + pt - c.AP * own));
        },
        [&](int i, int j, const double2& v) {
            AP[ix(p, i, j)] = v.x;
            cells[static_cast<std::size_t>(i - ur.i0) * ur.cols() + (j - ur.j0)] = v.y;
        });
}

// Threads of the record sweep's CTAs, and the resident CTAs its registers are bounded for: the x ring and
// two record slot sets of 224 columns take 98 KB, so two CTAs fit an SM.
constexpr int kMomRecNT = 224, kMomRecMinb = 2;
constexpr int kMomRecRing = 16; // x rows: a super-step reads down to 2 NCOL behind it, 6 rows ahead are issued
constexpr int kMomRecAhead = 2; // record slot sets (super-steps in flight)

template <int NCOL, int NT> struct MomRecSmem {
    static constexpr int SPB = NCOL == 5 ? 2 : 1;
    static constexpr int NK = NCOL == 5 ? 5 : 3;
    static constexpr int slots = kMomRecAhead * SPB;
    static constexpr int ring = kMomRecRing * NT * 8;
    static constexpr int bytes = ring + NK * slots * NT * 16;
    static constexpr unsigned row_bytes = NK * NT * 16; // bytes one step row of records brings in
};

// One multicolour sweep xin -> xout from the records: the schedule of k_mom_stream (cell (r, j) of colour
// c at step r + 2c, SPB steps per barrier, strip halo of 2 per colour). The records of one step for the
// CTA's columns are NK contiguous row segments; thread 0 fetches a super-step's with bulk copies into one
// of kMomRecAhead slot sets, completing on its `full` mbarrier, and refills a set once every thread has
// arrived on its `empty` mbarrier. x rows are per-thread cp.async copies, one group per super-step. Waits
// are bounded; a give-up sets *err, the next barrier stops the CTA, no further copy is issued, and thread
// 0 waits (bounded) for its copies in flight before it exits.
template <int NCOL, bool V, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_mom_rec_stream(DevParams p, const double* __restrict__ xin, double* __restrict__ xout, MomRec64 rec, int seg_rows,
                     unsigned* err) {
    using S = MomRecSmem<NCOL, NT>;
    constexpr int SPB = S::SPB, NK = S::NK;
    constexpr int HC = 2 * NCOL;
    constexpr int W = NT - 2 * HC;
    constexpr int D = kMomRecAhead;
    constexpr int E0 = SPB * D + 2; // x rows issued before the first super-step
    constexpr int MASK = kMomRecRing - 1;
    static_assert(D == 2, "the step loop is unrolled over the two record slot sets");
    extern __shared__ __align__(16) unsigned char mr_mem[];
    double* ring_mem = reinterpret_cast<double*>(mr_mem);
    double2* s_rec = reinterpret_cast<double2*>(mr_mem + S::ring); // [array][slot][column]
    __shared__ int s_rmin[NCOL], s_rmax[NCOL];
    __shared__ __align__(8) unsigned long long full[D], empty[D];
    const int tid = threadIdx.x;
    const int j0 = blockIdx.x * W;
    const int C0 = j0 - HC, C1 = j0 + W + HC;
    const int col = C0 + tid;
    const int R0 = blockIdx.y * seg_rows;
    const int R1 = min(R0 + seg_rows, p.nrows);
    const int L0 = max(R0 - HC, 0), L1 = min(R1 + HC, p.nrows);
    const int ld = p.pitch, H = p.H;
    const bool col_in = col >= 0 && col < p.ncols;
    const bool col_out = col_in && col >= j0 && col < j0 + W;
    if (tid < NCOL) { // the rows a cell of colour tid may be updated at (k_mom_stream)
        int lo = V ? H + 1 : H, hi = p.NX + H - 1;
        if (L0 > 0) lo = max(lo, L0 + 2 + 2 * tid);
        if (L1 < p.nrows) hi = min(hi, L1 - 3 - 2 * tid);
        s_rmin[tid] = lo;
        s_rmax[tid] = hi;
    }
    if (tid == 0) {
        for (int d = 0; d < D; ++d) {
            mbar_init(&full[d], 1);
            mbar_init(&empty[d], NT);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    unsigned colmask = 0;
    {
        const int ju0 = H + 1, ju1 = V ? p.NY + H : p.NY + H - 1;
#pragma unroll
        for (int c = 0; c < NCOL; ++c) {
            bool ok = col >= ju0 && col <= ju1;
            if (C0 > 0) ok = ok && col >= C0 + 2 + 2 * c;
            if (C1 < p.ncols) ok = ok && col <= C1 - 3 - 2 * c;
            colmask |= (ok ? 1u : 0u) << c;
        }
    }
    const double relax = V ? p.av : p.au;
    const double omr = 1 - relax;
    double* ringc = ring_mem + tid;
    int next = L0;
    const double* xo = xin + col + static_cast<std::ptrdiff_t>(L0) * ld; // the next row to issue
    double* wo = xout + col + static_cast<std::ptrdiff_t>(L0 - 2 * NCOL + 1 - (SPB - 1)) * ld; // ... to write
    auto issue_row = [&]() {
        if (next < L1 && col_in) cp_async(ringc + (next & MASK) * NT, xo);
        ++next;
        xo += ld;
    };
    auto step_cell = [&](int c, int t, int& r) -> bool {
        r = t - 2 * c;
        return ((colmask >> c) & 1u) && r >= s_rmin[c] && r <= s_rmax[c];
    };
    auto next_colour = [&](int c, int steps) { return NCOL == 5 ? (c + 2 * steps) % 5 : (c + steps) & 1; };
    const int rec_rows = p.nrows + kRecExtraRows;
    unsigned inflight = 0, inflight_parity = 0; // thread 0: the slot sets whose copies it has not seen land
    auto fill = [&](int slot, int t, unsigned parity) {
        inflight |= 1u << slot;
        inflight_parity = (inflight_parity & ~(1u << slot)) | (parity << slot);
        unsigned bytes = 0;
#pragma unroll
        for (int s = 0; s < SPB; ++s)
            if (t + s < rec_rows) bytes += S::row_bytes;
        mbar_arrive_expect(&full[slot], bytes);
#pragma unroll
        for (int s = 0; s < SPB; ++s) {
            if (t + s >= rec_rows) continue;
            const std::ptrdiff_t o = static_cast<std::ptrdiff_t>(t + s) * ld + C0;
#pragma unroll
            for (int k = 0; k < NK; ++k)
                bulk_load(s_rec + (k * S::slots + slot * SPB + s) * NT, rec.r[NK == 5 ? k : (k == 2 ? 4 : k)] + o,
                          NT * 16, &full[slot]);
        }
    };
    auto update = [&](int r, int q) {
        double* rc = ringc + (r & MASK) * NT;
        const double2 ew = s_rec[q], ns = s_rec[S::slots * NT + q], d = s_rec[(NK - 1) * S::slots * NT + q];
        const double xn = ringc[((r - 1) & MASK) * NT], xs = ringc[((r + 1) & MASK) * NT];
        double nb = ew.x * rc[1] + ew.y * rc[-1] + ns.x * xn + ns.y * xs;
        if (NCOL == 5) {
            const double2 fe = s_rec[2 * S::slots * NT + q], fn = s_rec[(NK - 2) * S::slots * NT + q];
            const double xnn = ringc[((r - 2) & MASK) * NT], xss = ringc[((r + 2) & MASK) * NT];
            nb = nb + (fe.x * rc[2] + fe.y * rc[-2] + fn.x * xnn + fn.y * xss);
        }
        rc[0] = relax * (nb + d.y) / d.x + omr * rc[0];
    };

    __syncthreads(); // s_rmin / s_rmax and the initialised mbarriers
    const int c_start = NCOL == 5 ? (2 * L0 + col + 1000) % 5 : (L0 + col + 1000) & 1;
    const int t_last = R1 + 2 * NCOL - 2 + (SPB - 1);
    for (int i = 0; i < E0; ++i) issue_row();
    cp_async_commit();
    cp_async_commit();
    if (tid == 0) {
        fill(0, L0, 0u);
        if (L0 + SPB <= t_last) fill(1, L0 + SPB, 0u);
    }
    int c_cur = c_start;
    bool gave_up = false;
    auto super_step = [&](int t, int slot, unsigned parity) -> bool {
        cp_async_wait<D - 1>(); // this thread's x rows for this super-step
        if (mbar_wait(&full[slot], parity, err)) {
            if (tid == 0) inflight &= ~(1u << slot);
        } else {
            gave_up = true;
        }
        if (__syncthreads_or(gave_up ? 1 : 0)) return false; // ... and everyone's
#pragma unroll
        for (int s = 0; s < SPB; ++s) {
            int r;
            if (step_cell(next_colour(c_cur, s), t + s, r)) update(r, (slot * SPB + s) * NT + tid);
        }
        mbar_arrive(&empty[slot]);
#pragma unroll
        for (int s = 0; s < SPB; ++s) {
            const int rw = t - 2 * NCOL + 1 - (SPB - 1) + s;
            if (rw >= R0 && rw < R1 && col_out) wo[s * ld] = ringc[(rw & MASK) * NT];
        }
        wo += SPB * ld;
#pragma unroll
        for (int s = 0; s < SPB; ++s) issue_row();
        cp_async_commit();
        c_cur = next_colour(c_cur, SPB);
        if (tid == 0 && t + SPB * D <= t_last) {
            if (mbar_wait(&empty[slot], parity, err)) fill(slot, t + SPB * D, parity ^ 1u);
            else gave_up = true; // not refilled: the next super-step's barrier stops the CTA
        }
        return true;
    };
    unsigned parity = 0;
    for (int t = L0; t <= t_last; t += 2 * SPB) {
        if (!super_step(t, 0, parity)) break;
        if (t + SPB <= t_last && !super_step(t + SPB, 1, parity)) break;
        parity ^= 1u;
    }
    if (tid == 0) // after a give-up only
        for (int sl = 0; sl < D; ++sl)
            if ((inflight >> sl) & 1u) mbar_wait(&full[sl], (inflight_parity >> sl) & 1u, err);
    cp_async_wait<0>();
}

// ---- small grids: a component's assembly, residual and sweeps on one thread-block cluster ----
//
// A grid of a few strips leaves the streaming sweep waiting: each CTA walks its rows, halo and colour
// skew at a block barrier per step, 23 us a sweep whatever the size. Where the component's
// coefficients, pressure term and velocity fit the shared memory of at most 16 CTAs (10 doubles and
// one per cell, 6 and one with two colours), the update range's rows are split into bands, each CTA
// forms its band's coefficients once (k_mom_prep's expressions; |R| and AP go to memory as there) and
// the sweeps go colour by colour, as the reference's. Colours are flattened over (row, cell of the
// colour), so narrow rows fill warps. A cell in the first or last two rows of a band is also stored
// into the neighbour's ghost rows (distributed shared memory): no cell of a colour reads another of
// it, so one barrier per colour is enough. One launch instead of 1 + maxit_inner.
// Measured, prep and four sweeps of one component: 19 us at 32^2 and 31 us at 128^2, against 96
// and 109 us.
constexpr int kMomCluster = 16; // CTAs at most
constexpr int kMomGhost = 2;
constexpr int kMomThreads = 512;
constexpr int kMomSmem = 227 * 1024;

struct MomClusterPlan {
    int ctas;
    int band[kMomCluster + 1]; // first row of each CTA's band (band[ctas]: one past the last)
    int rows;                  // rows of the largest band
    int bytes;                 // dynamic shared memory per CTA
};

template <int NCOL, bool V>
__global__ void __launch_bounds__(kMomThreads)
    k_mom_cluster(DevParams p, double* __restrict__ x, const double* __restrict__ oth, const double* __restrict__ pf,
                  double* __restrict__ AP, double* __restrict__ cells, Range ur, MomClusterPlan pl, int nsweeps) {
    namespace cg = cooperative_groups;
    constexpr int G = kMomGhost;
    constexpr int NK = NCOL == 5 ? 8 : 4; // links
    extern __shared__ double mc_mem[];
    cg::cluster_group cl = cg::this_cluster();
    const int R = pl.ctas, rank = R > 1 ? static_cast<int>(cl.block_rank()) : 0;
    auto sync = [&] {
        if (R > 1) cl.sync();
        else __syncthreads();
    };
    const int tid = static_cast<int>(threadIdx.x);
    const int nc = p.ncols, nu = ur.cols(), i0 = pl.band[rank], m = pl.band[rank + 1] - i0;
    const int plane = pl.rows * nu;
    double* xs = mc_mem;                        // rows -G .. rows + G - 1 of the band, all columns
    double* k = xs + (pl.rows + 2 * G) * nc;    // links, AP, pressure term: a plane each
    double* ap = k + NK * plane;
    double* pt = ap + plane;
    const std::size_t ld = p.pitch;
    for (int q = tid; q < (m + 2 * G) * nc; q += kMomThreads) {
        const int r = q / nc, j = q - r * nc;
        xs[q] = x[ix(p, i0 - G + r, j)];
    }
    __syncthreads();
    for (int q = tid; q < m * nu; q += kMomThreads) {
        const int r = q / nu, i = i0 + r, j = ur.j0 + (q - r * nu);
        const std::size_t g = ix(p, i, j);
        const double* c = xs + (r + G) * nc + j;
        double ue, uw, vn, vs, f;
        if (!V) { // coef_u
            ue = (c[0] + c[1]) / 2;
            uw = (c[0] + c[-1]) / 2;
            vn = (oth[g] + oth[g + 1]) / 2;
            vs = (oth[g + ld] + oth[g + ld + 1]) / 2;
            f = (pf[g] - pf[g + 1]) * p.dy;
        } else { // coef_v
            ue = (oth[g - ld] + oth[g]) / 2;
            uw = (oth[g - 1] + oth[g - ld - 1]) / 2;
            vn = (c[0] + c[-nc]) / 2;
            vs = (c[0] + c[nc]) / 2;
            f = (pf[g] - pf[g - ld]) * p.dx;
        }
        const Coef9 a = momentum_coef(p, ue, uw, vn, vs, i, j);
        const double nb = (a.AE * c[1] + a.AW * c[-1] + a.AN * c[-nc] + a.AS * c[nc]) +
                          (a.AEE * c[2] + a.AWW * c[-2] + a.ANN * c[-2 * nc] + a.ASS * c[2 * nc]);
        cells[static_cast<std::size_t>(i - ur.i0) * nu + (j - ur.j0)] = fabs(nb + f - a.AP * c[0]);
        AP[g] = a.AP;
        k[q] = a.AE;
        k[plane + q] = a.AW;
        k[2 * plane + q] = a.AN;
        k[3 * plane + q] = a.AS;
        if (NCOL == 5) {
            k[4 * plane + q] = a.AEE;
            k[5 * plane + q] = a.AWW;
            k[6 * plane + q] = a.ANN;
            k[7 * plane + q] = a.ASS;
        }
        ap[q] = a.AP;
        pt[q] = f;
    }
    // The band above holds our rows 0 .. G-1 as its rows mup .. mup + G - 1, the band below our last G
    // rows as its rows -G .. -1.
    double* xup = R > 1 && rank > 0 ? cl.map_shared_rank(xs, rank - 1) : nullptr;
    double* xdn = R > 1 && rank < R - 1 ? cl.map_shared_rank(xs, rank + 1) : nullptr;
    const int mup = rank > 0 ? i0 - pl.band[rank - 1] : 0;
    const double relax = V ? p.av : p.au, omr = 1 - relax;
    const int spr = (nu + NCOL - 1) / NCOL; // cells of one colour per row, at most
    const int r_first = tid / spr, c_first = tid - r_first * spr;
    sync(); // every CTA of the cluster runs and has loaded before any ghost row is written
    for (int sw = 0; sw < nsweeps; ++sw)
        for (int col = 0; col < NCOL; ++col) {
            int r = r_first, cell = c_first;
            for (int s = tid; s < m * spr; s += kMomThreads) {
                if (s != tid) {
                    r = s / spr;
                    cell = s - r * spr;
                }
                const int i = i0 + r;
                // colour = (i + 3 j) mod 5, or (i + j) mod 2: j = 2 (col - i) mod 5, or (col - i) mod 2
                const int res = NCOL == 5 ? (2 * (col - i - 3 * ur.j0) % 5 + 5) % 5 : ((col - i - ur.j0) & 1);
                const int jj = res + NCOL * cell;
                if (jj >= nu) continue;
                const int q = r * nu + jj, j = ur.j0 + jj;
                double* c = xs + (r + G) * nc + j;
                double nb = k[q] * c[1] + k[plane + q] * c[-1] + k[2 * plane + q] * c[-nc] + k[3 * plane + q] * c[nc];
                if (NCOL == 5)
                    nb = nb + (k[4 * plane + q] * c[2] + k[5 * plane + q] * c[-2] + k[6 * plane + q] * c[-2 * nc] +
                               k[7 * plane + q] * c[2 * nc]);
                const double v = relax * (nb + pt[q]) / ap[q] + omr * c[0];
                c[0] = v;
                if (r < G && xup) xup[(mup + G + r) * nc + j] = v;
                if (r >= m - G && xdn) xdn[(r - m + G) * nc + j] = v;
            }
            sync();
        }
    for (int q = tid; q < m * nu; q += kMomThreads) {
        const int r = q / nu, j = ur.j0 + (q - r * nu);
        x[ix(p, i0 + r, j)] = xs[(r + G) * nc + j];
    }
}

// assemble_p (pressure.cpp:14-54) in one pass: links with the wall zeros, APP, b, |b| and b. Each
// thread assembles the two cells (j, j + 1) of a column pair (j even; the pitch is even): the FP64
// inputs and outputs move as 16-byte pairs (a single store where only one of the two is a cell).
// The per-cell expressions are the reference's.
__device__ __forceinline__ double2 ld2(const double* q) { return *reinterpret_cast<const double2*>(q); }
__global__ void k_assemble_p(DevParams p, const double* __restrict__ APU,
                             const double* __restrict__ APV, const double* __restrict__ u,
                             const double* __restrict__ v, PressurePtr w, double* __restrict__ cabs,
                             double* __restrict__ cb) {
    const int H = p.H;
    const int j = ((H + 1) & ~1) + 2 * static_cast<int>(blockIdx.x * 32 + threadIdx.x);
    const int i = H + static_cast<int>(blockIdx.y * 8 + threadIdx.y);
    if (i > p.NX + H - 1 || j > p.NY + H) return;
    const std::size_t q = ix(p, i, j), ld = p.pitch;
    const double dx = p.dx, dy = p.dy;
    const double2 apu = ld2(APU + q), apv = ld2(APV + q), apvs = ld2(APV + q + ld);
    const double2 uu = ld2(u + q), vv = ld2(v + q), vs = ld2(v + q + ld);
    const double apuw = APU[q - 1], uw = u[q - 1];
    const double apu_e[2] = {apu.x, apu.y}, apu_w[2] = {apuw, apu.x};
    const double apv_n[2] = {apv.x, apv.y}, apv_s[2] = {apvs.x, apvs.y};
    const double u_e[2] = {uu.x, uu.y}, u_w[2] = {uw, uu.x};
    const double v_n[2] = {vv.x, vv.y}, v_s[2] = {vs.x, vs.y};
    double ae[2], aw[2], an[2], as[2], ap[2], bb[2];
    bool cell[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int jj = j + e;
        cell[e] = jj >= H + 1 && jj <= p.NY + H;
        if (!cell[e]) continue;
        ae[e] = (jj == p.NY + H) ? 0.0 : dy * dy / apu_e[e];
        aw[e] = (jj == H + 1) ? 0.0 : dy * dy / apu_w[e];
        an[e] = (i == H) ? 0.0 : dx * dx / apv_n[e];
        as[e] = (i == p.NX + H - 1) ? 0.0 : dx * dx / apv_s[e];
        ap[e] = ae[e] + aw[e] + an[e] + as[e];
        bb[e] = -dx * (-v_s[e] + v_n[e]) - dy * (-u_w[e] + u_e[e]);
        const std::size_t c = static_cast<std::size_t>(i - H) * p.NY + (jj - H - 1);
        if (cabs) cabs[c] = fabs(bb[e]);
        if (cb) cb[c] = bb[e];
    }
    auto put = [&](double* dst, const double* val) {
        if (cell[0] && cell[1]) *reinterpret_cast<double2*>(dst + q) = make_double2(val[0], val[1]);
        else if (cell[0]) dst[q] = val[0];
        else if (cell[1]) dst[q + 1] = val[1];
    };
    put(w.AEP, ae);
    put(w.AWP, aw);
    put(w.ANP, an);
    put(w.ASP, as);
    put(w.APP, ap);
    put(w.b, bb);
}

template <bool V>
void prep_ranges(const DevParams& p, Range& ur, Range& cr) {
    const int H = p.H;
    if (!V) {
        ur = {H, p.NX + H - 1, H + 1, p.NY + H - 1};
        cr = {ur.i0, ur.i1, ur.j0 - 1, ur.j1 + 1}; // coef_u reads uF at j - 1 .. j + 1
    } else {
        ur = {H + 1, p.NX + H - 1, H + 1, p.NY + H};
        cr = {ur.i0 - 1, ur.i1 + 1, ur.j0, ur.j1}; // coef_v reads vF at i - 1 .. i + 1
    }
}

template <int NCOL, bool V, int NT, bool QUICK, int ORDER, int PF>
void launch_stream(const DevParams& p, const double* xin, double* xout, const double* xF,
                   const double* oth, const double* pf, int seg_rows, cudaStream_t st) {
    constexpr int W = NT - 4 * NCOL;
    const dim3 grid((p.ncols + W - 1) / W, (p.nrows + seg_rows - 1) / seg_rows);
    constexpr int smem = kRing * NT * static_cast<int>(sizeof(double));
    static PerDeviceOnce attr; // the attribute lives in each device's context
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_mom_stream<NCOL, V, NT, QUICK, ORDER, PF>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        return 0;
    });
    k_mom_stream<NCOL, V, NT, QUICK, ORDER, PF><<<grid, NT, smem, st>>>(p, xin, xout, xF, oth, pf, seg_rows);
    SGPU_LAUNCH();
}

template <bool V, int PF>
void launch_stream_v(const DevParams& p, const double* xin, double* xout, const double* xF,
                     const double* oth, const double* pf, int seg_rows, cudaStream_t st) {
    if (p.uds && p.order == 2) launch_stream<2, V, 256, false, 2, PF>(p, xin, xout, xF, oth, pf, seg_rows, st);
    else if (p.uds) launch_stream<5, V, 256, false, 4, PF>(p, xin, xout, xF, oth, pf, seg_rows, st);
    else if (p.order == 2) launch_stream<5, V, 256, true, 2, PF>(p, xin, xout, xF, oth, pf, seg_rows, st);
    else launch_stream<5, V, 256, true, 4, PF>(p, xin, xout, xF, oth, pf, seg_rows, st);
}

// The cluster's plan: the fewest CTAs (a power of two, at least kMomGhost rows each) whose shared memory
// holds the component, and whose threads hold a colour of it where 16 CTAs can; false where it does not
// fit. Fewer CTAs make a barrier cheaper, more than one cell per thread and colour makes a pass longer.
bool mom_cluster_plan(const DevParams& p, const Range& ur, MomClusterPlan& pl) {
    const int n = ur.rows(), nu = ur.cols();
    if (n < 1 || nu < 1) return false;
    bool found = false;
    for (int c = 1; c <= kMomCluster && (c == 1 || n >= kMomGhost * c); c *= 2) {
        const int rows = (n + c - 1) / c;
        const long long bytes = 8LL * ((rows + 2 * kMomGhost) * static_cast<long long>(p.ncols) +
                                       static_cast<long long>(rows) * nu * (p.ncol == 5 ? 10 : 6));
        if (bytes > kMomSmem) continue;
        found = true;
        pl.ctas = c;
        pl.rows = rows;
        pl.bytes = static_cast<int>(bytes);
        for (int r = 0; r <= c; ++r) pl.band[r] = ur.i0 + static_cast<int>(static_cast<long long>(r) * n / c);
        if (rows * ((nu + p.ncol - 1) / p.ncol) <= kMomThreads) break;
    }
    return found;
}

// Clusters of 16 such CTAs that this device runs (its kernels' attributes set once per device); 0: none.
template <int NCOL, bool V> int mom_cluster_available() {
    static PerDeviceOnce once;
    return once.get([] {
        auto kernel = k_mom_cluster<NCOL, V>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMomCluster);
        cfg.blockDim = dim3(kMomThreads);
        cfg.dynamicSmemBytes = kMomSmem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kMomCluster;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMomSmem) != cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            (void)cudaGetLastError(); // a device that refuses them runs the streaming kernels
            return 0;
        }
        return n;
    });
}

template <int NCOL, bool V>
void launch_mom_cluster_t(const DevParams& p, double* x, const double* oth, const double* pf, double* AP, double* cells,
                          const Range& ur, const MomClusterPlan& pl, int nsweeps, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.ctas);
    cfg.blockDim = dim3(kMomThreads);
    cfg.dynamicSmemBytes = static_cast<std::size_t>(pl.bytes);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(pl.ctas);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SGPU_CUDA(cudaLaunchKernelEx(&cfg, k_mom_cluster<NCOL, V>, p, x, oth, pf, AP, cells, ur, pl, nsweeps));
    SGPU_LAUNCH();
}

template <int NCOL, bool V>
void launch_rec_stream(const DevParams& p, const double* xin, double* xout, MomRec64 rec, int seg_rows, unsigned* err,
                       cudaStream_t st) {
    // A bulk copy starts at record (t * pitch + first column), 16 bytes each: aligned when the arrays are.
    for (int k = 0; k < 5; ++k)
        if (mom_rec_used(NCOL, k) && (!rec.r[k] || (reinterpret_cast<std::uintptr_t>(rec.r[k]) & 15u)))
            throw Error(SGPU_E_INVALID, "momentum sweep: records missing or not aligned for bulk copies");
    constexpr int NT = kMomRecNT, W = NT - 4 * NCOL;
    static_assert(2 * NCOL <= kRecFrontCols && NT <= kRecBackCols, "copy windows must stay in the margins");
    using S = MomRecSmem<NCOL, NT>;
    static PerDeviceOnce attr;
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_mom_rec_stream<NCOL, V, NT, kMomRecMinb>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, S::bytes));
        return 0;
    });
    const dim3 grid((p.ncols + W - 1) / W, (p.nrows + seg_rows - 1) / seg_rows);
    k_mom_rec_stream<NCOL, V, NT, kMomRecMinb><<<grid, NT, S::bytes, st>>>(p, xin, xout, rec, seg_rows, err);
    SGPU_LAUNCH();
}

} // namespace

// Rows per CTA segment of the streaming sweep: enough segments to fill the GPU with one wave of
// 2 CTAs per SM, but never so short that the 2 * NCOL-row halo dominates.
int stream_seg_rows(const DevParams& p, int sms, int blocks_per_sm, int min_seg, int nt) {
    const int W = nt - 4 * p.ncol;
    const int strips = (p.ncols + W - 1) / W;
    const int want = std::max(1, (blocks_per_sm * sms) / strips); // one wave of resident CTAs
    int seg = (p.nrows + want - 1) / want;
    const int lo = min_seg > 0 ? min_seg : 8 * p.ncol;
    if (seg < lo) seg = lo;
    return seg;
}

void launch_mom_prep(const DevParams& p, bool v_component, const double* x, const double* oth,
                     const double* pf, double* xF, double* AP, double* cells, cudaStream_t st) {
    Range ur, cr;
    if (v_component) prep_ranges<true>(p, ur, cr);
    else prep_ranges<false>(p, ur, cr);
    if (cr.rows() <= 0 || cr.cols() <= 0) return;
    const dim3 grid((cr.cols() + 31) / 32, (cr.rows() + 7) / 8);
    if (v_component) k_mom_prep<true><<<grid, dim3(32, 8), 0, st>>>(p, x, oth, pf, xF, AP, cells, ur, cr);
    else k_mom_prep<false><<<grid, dim3(32, 8), 0, st>>>(p, x, oth, pf, xF, AP, cells, ur, cr);
    SGPU_LAUNCH();
}

bool mom_cluster_fits(const DevParams& p, bool v_component) {
    Range ur, cr;
    if (v_component) prep_ranges<true>(p, ur, cr);
    else prep_ranges<false>(p, ur, cr);
    MomClusterPlan pl{};
    if (!mom_cluster_plan(p, ur, pl)) return false;
    if (p.ncol == 5) return (v_component ? mom_cluster_available<5, true>() : mom_cluster_available<5, false>()) > 0;
    return (v_component ? mom_cluster_available<2, true>() : mom_cluster_available<2, false>()) > 0;
}

void launch_mom_cluster(const DevParams& p, bool v_component, double* x, const double* oth, const double* pf,
                        double* AP, double* cells, int nsweeps, cudaStream_t st) {
    Range ur, cr;
    if (v_component) prep_ranges<true>(p, ur, cr);
    else prep_ranges<false>(p, ur, cr);
    MomClusterPlan pl{};
    mom_cluster_plan(p, ur, pl);
    if (p.ncol == 5) {
        if (v_component) launch_mom_cluster_t<5, true>(p, x, oth, pf, AP, cells, ur, pl, nsweeps, st);
        else launch_mom_cluster_t<5, false>(p, x, oth, pf, AP, cells, ur, pl, nsweeps, st);
    } else {
        if (v_component) launch_mom_cluster_t<2, true>(p, x, oth, pf, AP, cells, ur, pl, nsweeps, st);
        else launch_mom_cluster_t<2, false>(p, x, oth, pf, AP, cells, ur, pl, nsweeps, st);
    }
}

void launch_mom_sweep(const DevParams& p, bool v_component, const double* xin, double* xout,
                      const double* xF, const double* oth, const double* pf, int seg_rows,
                      cudaStream_t st) {
    if (v_component) launch_stream_v<true, kStreamPF>(p, xin, xout, xF, oth, pf, seg_rows, st);
    else launch_stream_v<false, kStreamPF>(p, xin, xout, xF, oth, pf, seg_rows, st);
}

namespace {
template <int NCOL, bool V>
void launch_prep_rec(const DevParams& p, const double* x, const double* oth, const double* pf, double* AP, double* cells,
                     MomRec64 rec, const Range& ur, cudaStream_t st) {
    constexpr int smem = sizeof(PrepWalk<V, double2>);
    static PerDeviceOnce once;
    const int rows = prep_rows(ur, prep_resident(k_mom_prep_rec<NCOL, V>, smem, once));
    const dim3 grid(prep_strips(ur), (ur.rows() + rows - 1) / rows);
    k_mom_prep_rec<NCOL, V><<<grid, dim3(32, kPrepSteps), smem, st>>>(p, x, oth, pf, AP, cells, rec, ur, rows);
    SGPU_LAUNCH();
}
} // namespace
void launch_mom_prep_rec(const DevParams& p, bool v_component, const double* x, const double* oth, const double* pf,
                         double* AP, double* cells, MomRec64 rec, cudaStream_t st) {
    Range ur, cr;
    if (v_component) prep_ranges<true>(p, ur, cr);
    else prep_ranges<false>(p, ur, cr);
    if (ur.rows() <= 0 || ur.cols() <= 0) return;
    if (p.ncol == 5) {
        if (v_component) launch_prep_rec<5, true>(p, x, oth, pf, AP, cells, rec, ur, st);
        else launch_prep_rec<5, false>(p, x, oth, pf, AP, cells, rec, ur, st);
    } else {
        if (v_component) launch_prep_rec<2, true>(p, x, oth, pf, AP, cells, rec, ur, st);
        else launch_prep_rec<2, false>(p, x, oth, pf, AP, cells, rec, ur, st);
    }
}

void launch_mom_sweep_rec(const DevParams& p, bool v_component, const double* xin, double* xout, MomRec64 rec,
                          int seg_rows, unsigned* err, cudaStream_t st) {
    if (p.ncol == 5) {
        if (v_component) launch_rec_stream<5, true>(p, xin, xout, rec, seg_rows, err, st);
        else launch_rec_stream<5, false>(p, xin, xout, rec, seg_rows, err, st);
    } else {
        if (v_component) launch_rec_stream<2, true>(p, xin, xout, rec, seg_rows, err, st);
        else launch_rec_stream<2, false>(p, xin, xout, rec, seg_rows, err, st);
    }
}

int mom_rec_threads() { return kMomRecNT; }
int mom_rec_blocks_per_sm(int ncol) {
    static PerDeviceOnce five, two;
    auto resident = [](auto kernel, int smem) {
        int n = 0;
        SGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        SGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kMomRecNT, smem));
        return std::max(n, 1);
    };
    if (ncol == 5)
        return five.get([&] { return resident(k_mom_rec_stream<5, false, kMomRecNT, kMomRecMinb>, MomRecSmem<5, kMomRecNT>::bytes); });
    return two.get([&] { return resident(k_mom_rec_stream<2, false, kMomRecNT, kMomRecMinb>, MomRecSmem<2, kMomRecNT>::bytes); });
}

void launch_assemble_p_fused(const DevParams& p, const double* APU, const double* APV,
                             const double* u, const double* v, PressurePtr w, double* cabs,
                             double* cb, cudaStream_t st) {
    const int pairs = (p.NY + p.H - ((p.H + 1) & ~1)) / 2 + 1; // column pairs over j = H + 1 .. NY + H
    const dim3 grid((pairs + 31) / 32, (p.NX + 7) / 8);
    k_assemble_p<<<grid, dim3(32, 8), 0, st>>>(p, APU, APV, u, v, w, cabs, cb);
    SGPU_LAUNCH();
}

} // namespace sgpu
