// mg.cu — geometric multigrid for p' on the device, bit-identical to the reference in FP64.
//
// The reference runs multigrid on the CPU only (src/multigrid.cpp). These kernels restate each of
// its loops with the same per-cell expression order: the Galerkin 2x2 build (mg_build, :232-261),
// the red-black two-statement smoother (smooth, :46-70), residual (:73-87), restriction (:90-103),
// prolongation with over-correction (:106-116), and the coarsest-level solve with its fixed-order
// norms (coarse_solve, :120-140), which runs inside one CTA so its data-dependent sweep count
// needs no host round trip. Every kernel is a template on the element type: double gives the
// reference's bits; float is the mixed-precision mode's V-cycle (sums and norms still in double).
// The small levels of the streaming V-cycle run in one kernel, the tail: in the shared memory of a
// thread-block cluster (k_mg_tail_cluster) or of one CTA (k_mg_tail_smem), or on global memory in one
// CTA (k_mg_tail). The coarsest solve has a kernel of its own, and a device function inside the
// tails, with a cell pair per thread in registers (mg_coarse.cuh).
#include "kernels.hpp"
#include "mg_coarse.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

namespace sgpu {

namespace {

constexpr int BX = 32, BY = 8;

dim3 grid2(int nx, int ny) { return dim3((ny + BX - 1) / BX, (nx + BY - 1) / BY); }

// Coarse cell c of mg_build from its four fine cells' links.
template <class T>
__device__ __forceinline__ void build_cell(const LevelViewT<T>& C, int c, Links<T> k00, Links<T> k01, Links<T> k10,
                                           Links<T> k11) {
    const T ae = k01.e + k11.e;
    const T aw = k00.w + k10.w;
    const T an = k00.n + k01.n;
    const T as = k10.s + k11.s;
    set_links(C, c, ae, aw, an, as);
    C.AP[c] = ae + aw + an + as;
}

// mg_build: coarse links are the sums of the two fine links crossing each coarse face.
template <class T> __global__ void k_mg_build(LevelViewT<T> F, LevelViewT<T> C) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= C.nx || J >= C.ny) return;
    const int fs = F.stride;
    const int f = 2 * I * fs + 2 * J, c = I * C.stride + J;
    build_cell(C, c, links(F, f), links(F, f + 1), links(F, f + fs), links(F, f + fs + 1));
}

// One colour of smooth: colour (I + J) & 1, update x = b/AP; x += (E W S N)/AP.
template <class T> __global__ void k_mg_smooth(LevelViewT<T> L, int colour) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= L.nx || J >= L.ny || ((I + J) & 1) != colour) return;
    const int s = L.stride, q = I * s + J;
    T* x = L.x;
    const Links<T> k = links(L, q);
    x[q] = rb_value(L.b[q], k.e * x[q + 1] + k.w * x[q - 1] + k.s * x[q + s] + k.n * x[q - s], L.AP[q]);
}

template <class T> __global__ void k_mg_residual(LevelViewT<T> L) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= L.nx || J >= L.ny) return;
    const int s = L.stride, q = I * s + J;
    const T* x = L.x;
    const Links<T> k = links(L, q);
    L.r[q] = L.b[q] - (L.AP[q] * x[q] - (k.e * x[q + 1] + k.w * x[q - 1] + k.s * x[q + s] + k.n * x[q - s]));
}

template <class T> __global__ void k_mg_restrict(LevelViewT<T> F, LevelViewT<T> C) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= F.nx / 2 || J >= F.ny / 2) return;
    const int fs = F.stride, f = 2 * I * fs + 2 * J, c = I * C.stride + J;
    C.b[c] = F.r[f] + F.r[f + 1] + F.r[f + fs] + F.r[f + fs + 1];
    C.x[c] = T(0);
}

template <class T> __global__ void k_mg_prolong(LevelViewT<T> C, LevelViewT<T> F, double omega) {
    const int j = blockIdx.x * BX + threadIdx.x, i = blockIdx.y * BY + threadIdx.y;
    if (i >= F.nx || j >= F.ny) return;
    F.x[i * F.stride + j] += static_cast<T>(omega) * C.x[(i / 2) * C.stride + j / 2];
}

// Squares of the level residual r = b - A x (multigrid.cpp:84-85 form), in FP64, one per cell of a
// compact nx x ny plane, for the ordered norm of the tolerance-driven V-cycle loop.
template <class T> __global__ void k_mg_residual_sq(LevelViewT<T> L, double* cells) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= L.nx || J >= L.ny) return;
    const int s = L.stride, q = I * s + J;
    const T* x = L.x;
    const Links<T> k = links(L, q);
    const double r = static_cast<double>(L.b[q]) -
                     (static_cast<double>(L.AP[q]) * x[q] -
                      (static_cast<double>(k.e) * x[q + 1] + static_cast<double>(k.w) * x[q - 1] +
                       static_cast<double>(k.s) * x[q + s] + static_cast<double>(k.n) * x[q - s]));
    cells[static_cast<std::size_t>(I) * L.ny + J] = r * r;
}

// Squares of b, for ||b|| of the same loop.
template <class T> __global__ void k_mg_b_sq(LevelViewT<T> L, double* cells) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= L.nx || J >= L.ny) return;
    const double b = L.b[I * L.stride + J];
    cells[static_cast<std::size_t>(I) * L.ny + J] = b * b;
}

__global__ void k_mg_sub_mean(LevelView L, double* x, const double* sum) {
    const int J = blockIdx.x * BX + threadIdx.x, I = blockIdx.y * BY + threadIdx.y;
    if (I >= L.nx || J >= L.ny) return;
    const double m = *sum / (static_cast<double>(L.nx) * L.ny);
    x[I * L.stride + J] -= m;
}

// ---- levels inside one CTA ----

constexpr int kCoarseThreads = 512;

// det_sum (multigrid.cpp:18-34) of f(q) in one CTA: one thread per row chain, then row order.
// Accumulates in double for both element types.
template <class T, class F>
__device__ double cta_det_sum(const LevelViewT<T>& L, double* rowbuf, F f) {
    for (int I = threadIdx.x; I < L.nx; I += blockDim.x) {
        double s = 0.0;
        for (int J = 0; J < L.ny; ++J) s += f(I * L.stride + J);
        rowbuf[I] = s;
    }
    __syncthreads();
    __shared__ double total;
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int I = 0; I < L.nx; ++I) s += rowbuf[I];
        total = s;
    }
    __syncthreads();
    const double t = total;
    __syncthreads();
    return t;
}

template <class T> __device__ void cta_remove_mean(const LevelViewT<T>& L, double* rowbuf, T* x) {
    const double m = cta_det_sum(L, rowbuf, [x](int q) { return static_cast<double>(x[q]); }) /
                     (static_cast<double>(L.nx) * L.ny);
    const int n = L.nx * L.ny;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int I = k / L.ny, J = k % L.ny;
        x[I * L.stride + J] = static_cast<T>(x[I * L.stride + J] - m);
    }
    __syncthreads();
}

template <class T> __device__ void cta_smooth_colour(const LevelViewT<T>& L, int colour) {
    const int n = L.nx * L.ny, s = L.stride;
    T* x = L.x;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int I = k / L.ny, J = k % L.ny;
        if (((I + J) & 1) != colour) continue;
        const int q = I * s + J;
        const Links<T> k4 = links_written(L, q);
        x[q] = rb_value(L.b[q], k4.e * x[q + 1] + k4.w * x[q - 1] + k4.s * x[q + s] + k4.n * x[q - s], L.AP[q]);
    }
    __syncthreads();
}

template <class T> __device__ void cta_residual(const LevelViewT<T>& L) {
    const int n = L.nx * L.ny, s = L.stride;
    const T* x = L.x;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int I = k / L.ny, J = k % L.ny, q = I * s + J;
        const Links<T> k4 = links_written(L, q);
        L.r[q] = L.b[q] - (L.AP[q] * x[q] - (k4.e * x[q + 1] + k4.w * x[q - 1] + k4.s * x[q + s] + k4.n * x[q - s]));
    }
    __syncthreads();
}

// restrict_residual (multigrid.cpp:90-103) inside one CTA.
template <class T> __device__ void cta_restrict(const LevelViewT<T>& F, const LevelViewT<T>& C) {
    const int n = C.nx * C.ny, fs = F.stride;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int I = k / C.ny, J = k % C.ny;
        const int f = 2 * I * fs + 2 * J, c = I * C.stride + J;
        C.b[c] = F.r[f] + F.r[f + 1] + F.r[f + fs] + F.r[f + fs + 1];
        C.x[c] = T(0);
    }
    __syncthreads();
}

// mg_build (multigrid.cpp:232-261) inside one CTA.
template <class T> __device__ void cta_build(const LevelViewT<T>& F, const LevelViewT<T>& C) {
    const int n = C.nx * C.ny, fs = F.stride;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int I = k / C.ny, J = k % C.ny, f = 2 * I * fs + 2 * J;
        build_cell(C, I * C.stride + J, links_written(F, f), links_written(F, f + 1),
                   links_written(F, f + fs), links_written(F, f + fs + 1));
    }
    __syncthreads();
}

// prolong (multigrid.cpp:106-116) inside one CTA.
template <class T>
__device__ void cta_prolong(const LevelViewT<T>& C, const LevelViewT<T>& F, double omega) {
    const int n = F.nx * F.ny;
    const T om = static_cast<T>(omega);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int i = k / F.ny, j = k % F.ny;
        F.x[i * F.stride + j] += om * C.x[(i / 2) * C.stride + j / 2];
    }
    __syncthreads();
}

// coarse_solve (multigrid.cpp:120-140): remove the mean of b; red-black sweeps until
// ||b - A x|| < tol ||b|| (tol = 1e-10 in the reference) or 200 sweeps; remove the mean of x.
template <class T>
__device__ void cta_coarse_solve(const LevelViewT<T>& L, double* rowbuf, double tol, int* sweeps_out) {
    cta_remove_mean(L, rowbuf, L.b);
    const T* b = L.b;
    const double bb = cta_det_sum(L, rowbuf, [b](int q) {
        const double v = b[q];
        return v * v;
    });
    int sweeps = 0;
    if (bb > 0.0) {
        const double bn = sqrt(bb);
        const T* r = L.r;
        while (sweeps < 200) {
            cta_smooth_colour(L, 0);
            cta_smooth_colour(L, 1);
            ++sweeps;
            cta_residual(L);
            const double rr = cta_det_sum(L, rowbuf, [r](int q) {
                const double v = r[q];
                return v * v;
            });
            if (sqrt(rr) < tol * bn) break;
        }
    }
    cta_remove_mean(L, rowbuf, L.x);
    if (threadIdx.x == 0 && sweeps_out) *sweeps_out = sweeps;
}

// A level held in shared memory: (nx + 2) x (ny + 2) cells with the zero ring, row stride S, interior
// cell (I, J) at index (I + 1) * S + J + 1; links {e, w, n, s}, AP, b and x per cell.
template <class T> struct alignas(16) Link4T {
    T e, w, n, s;
};
template <class T> struct SLevel {
    int nx, ny, S;
    Link4T<T>* l4;
    T *x, *b, *ap;
    __device__ int at(int I, int J) const { return (I + 1) * S + J + 1; }
    __device__ T flow(int q) const {
        const Link4T<T> a = l4[q];
        return a.e * x[q + 1] + a.w * x[q - 1] + a.s * x[q + S] + a.n * x[q - S];
    }
};
// Bytes of one SLevel block (links first, 16-byte aligned).
template <class T> __host__ __device__ inline int slevel_bytes(int nx, int ny) {
    const int n2 = (nx + 2) * (ny + 2);
    return (n2 * 7 * static_cast<int>(sizeof(T)) + 15) / 16 * 16;
}
template <class T> __device__ inline SLevel<T> slevel_at(unsigned char* base, int nx, int ny) {
    const int n2 = (nx + 2) * (ny + 2);
    SLevel<T> v;
    v.nx = nx;
    v.ny = ny;
    v.S = ny + 2;
    v.l4 = reinterpret_cast<Link4T<T>*>(base);
    v.x = reinterpret_cast<T*>(base) + 4 * n2;
    v.b = v.x + n2;
    v.ap = v.b + n2;
    return v;
}

// The block's threads over rows of `width` cells: a power of two of them per row, so that short rows
// share a warp and no row index takes a division.
struct RowWalk {
    int r, dr, c, dc;
    __device__ explicit RowWalk(int width) {
        const int nt = static_cast<int>(blockDim.x), tid = static_cast<int>(threadIdx.x);
        int sh = width > 1 ? 32 - __clz(width - 1) : 0;
        while ((1 << sh) > nt) --sh;
        dc = 1 << sh;
        dr = nt >> sh;
        c = tid & (dc - 1);
        r = tid >> sh;
        if (r >= dr) r = 1 << 29; // threads past the last whole row (a block that is no power of two)
    }
};

// The coarsest solve on a shared level by the first coarse_threads() threads of the block: its scratch
// is the level's own link array, which the solve has read into registers before it writes there (for
// every level the links take more than the scratch).
template <class T> __device__ void s_coarse_solve(const SLevel<T>& L, double tol, int* sweeps_out) {
    const CoarseCta team{coarse_threads(L.nx, L.ny)};
    if (static_cast<int>(threadIdx.x) < team.nt)
        coarse_solve<T>(
            team, L.nx, L.ny, 0, L.nx, 0, tol, coarse_smem<T>(L.l4, L.nx, L.nx, L.ny),
            [&](int I, int J) {
                const int q = L.at(I, J);
                const Link4T<T> a = L.l4[q];
                return CoarseCell<T>{a.e, a.w, a.n, a.s, L.ap[q], L.b[q], L.x[q]};
            },
            [&](int I, int J, T x, T b) {
                const int q = L.at(I, J);
                L.x[q] = x;
                L.b[q] = b;
            },
            sweeps_out);
    __syncthreads();
}

// Rows [g0, g0 + s.nx) of the global level L into the shared band s, by all threads of the block:
// links and AP with `links`, b and x (its ghost rows too) with `values`; zero elsewhere.
template <class T> __device__ void slevel_load(const LevelViewT<T>& L, const SLevel<T>& s, int g0, bool link, bool values) {
    const int n2 = (s.nx + 2) * s.S;
    for (int k = threadIdx.x; k < n2; k += blockDim.x) {
        const int I = k / s.S - 1, J = k % s.S - 1, g = g0 + I;
        const bool cin = J >= 0 && J < L.ny, own = cin && I >= 0 && I < s.nx;
        const int q = g * L.stride + J;
        Link4T<T> l{T(0), T(0), T(0), T(0)};
        if (own && link) {
            const Links<T> a = links(L, q);
            l = {a.e, a.w, a.n, a.s};
        }
        s.l4[k] = l;
        s.ap[k] = own && link ? L.AP[q] : T(0);
        s.b[k] = (own && values) ? L.b[q] : T(0);
        s.x[k] = (values && cin && g >= 0 && g < L.nx) ? L.x[q] : T(0);
    }
}
// The band's interior x back to rows g0 on of L.
template <class T> __device__ void slevel_store_x(const LevelViewT<T>& L, const SLevel<T>& s, int g0) {
    const RowWalk w(L.ny);
    for (int I = w.r; I < s.nx; I += w.dr)
        for (int J = w.c; J < L.ny; J += w.dc) L.x[(g0 + I) * L.stride + J] = s.x[s.at(I, J)];
}

// mg_build (multigrid.cpp:232-261) of the band F into rows c0 on of the coarse level C. No barrier.
template <class T> __device__ void s_build(const SLevel<T>& F, const SLevel<T>& C, int c0) {
    const RowWalk w(C.ny);
    for (int I = w.r; I < F.nx / 2; I += w.dr)
        for (int J = w.c; J < C.ny; J += w.dc) {
            const int f = F.at(2 * I, 2 * J), c = C.at(c0 + I, J), S = F.S;
            const Link4T<T> k00 = F.l4[f], k01 = F.l4[f + 1], k10 = F.l4[f + S], k11 = F.l4[f + S + 1];
            const Link4T<T> k{k01.e + k11.e, k00.w + k10.w, k00.n + k01.n, k10.s + k11.s};
            C.l4[c] = k;
            C.ap[c] = k.e + k.w + k.n + k.s;
        }
}

// ---- the tail with every level in the shared memory of one CTA ----

// Byte offset of each tail level's SLevel block in dynamic shared memory, and the total.
struct TailSmem {
    int off[24];
    int bytes;
};

// One colour of smooth on a shared level.
template <class T> __device__ void s_smooth(const SLevel<T>& L, int colour) {
    const RowWalk w((L.ny + 1) / 2);
    for (int I = w.r; I < L.nx; I += w.dr)
        for (int J = ((I + colour) & 1) + 2 * w.c; J < L.ny; J += 2 * w.dc) {
            const int q = L.at(I, J);
            L.x[q] = rb_value(L.b[q], L.flow(q), L.ap[q]);
        }
    __syncthreads();
}
// Residual of F (multigrid.cpp:84-85 form) restricted 2x2 (multigrid.cpp:90-103) into rows c0 on of C, C.x = 0.
template <class T> __device__ void s_restrict_rows(const SLevel<T>& F, const SLevel<T>& C, int c0) {
    const RowWalk w(C.ny);
    const int S = F.S;
    auto r = [&](int q) { return F.b[q] - (F.ap[q] * F.x[q] - F.flow(q)); };
    for (int I = w.r; I < F.nx / 2; I += w.dr)
        for (int J = w.c; J < C.ny; J += w.dc) {
            const int f = F.at(2 * I, 2 * J), c = C.at(c0 + I, J);
            C.b[c] = r(f) + r(f + 1) + r(f + S) + r(f + S + 1);
            C.x[c] = T(0);
        }
}
// prolong (multigrid.cpp:106-116): F.x += omega * C.x of the parent cell.
template <class T> __device__ void s_prolong(const SLevel<T>& C, const SLevel<T>& F, T om) {
    const RowWalk w(F.ny);
    for (int i = w.r; i < F.nx; i += w.dr)
        for (int j = w.c; j < F.ny; j += w.dc) F.x[F.at(i, j)] += om * C.x[C.at(i >> 1, j >> 1)];
    __syncthreads();
}

// Levels [first, nl) of one V-cycle (mg_vcycle, multigrid.cpp:299-323) in one CTA with every level in
// shared memory: the links, AP, b and x of the first tail level are read once, the coarser operators
// built from them (build) or read, the passes run against shared memory with a block barrier between
// them, and x of the first level is written back. Same passes and per-cell expressions as k_mg_tail.
template <class T>
__global__ void __launch_bounds__(kCoarseThreads)
    k_mg_tail_smem(MgLevelsT<T> lv, int first, int pre, int post, double omega, double tol, TailSmem ts, int build,
                   int* sweeps_out) {
    extern __shared__ __align__(16) unsigned char tail_sm[];
    const int nl = lv.n;
    auto sl = [&](int l) { return slevel_at<T>(tail_sm + ts.off[l], lv.L[l].nx, lv.L[l].ny); };
    for (int l = first; l < nl; ++l) slevel_load(lv.L[l], sl(l), 0, l == first || !build, l == first);
    __syncthreads();
    for (int l = first; l + 1 < nl; ++l) {
        const SLevel<T> L = sl(l);
        for (int s = 0; s < pre; ++s) {
            s_smooth(L, 0);
            s_smooth(L, 1);
        }
        s_restrict_rows(L, sl(l + 1), 0);
        if (build) s_build(L, sl(l + 1), 0);
        __syncthreads();
    }
    s_coarse_solve(sl(nl - 1), tol, sweeps_out);
    const T om = static_cast<T>(omega);
    for (int l = nl - 2; l >= first; --l) {
        const SLevel<T> L = sl(l);
        s_prolong(sl(l + 1), L, om);
        for (int s = 0; s < post; ++s) {
            s_smooth(L, 0);
            s_smooth(L, 1);
        }
    }
    slevel_store_x(lv.L[first], sl(first), 0);
}

// ---- the tail on a thread-block cluster ----
//
// Levels [first, lg) of the V-cycle are split by rows over the kClusterTail CTAs of one cluster, each
// CTA's band of a level held in its shared memory as an SLevel whose ring rows are ghost copies of the
// neighbouring bands' edge rows; levels [lg, nl) (at most kGatherCells cells each) and the coarsest
// solve run on CTA 0 as in k_mg_tail_smem. The passes and per-cell expressions are k_mg_tail_smem's,
// with a cluster barrier between passes instead of a block barrier. Levels halve exactly
// (mg_level_dims halves only even sizes), and the bands of the coarsest split level start at even rows,
// so every band of every split level starts at an even row: a 2 x 2 restriction block, a coarse
// operator's block and a prolongation parent lie in the CTA's own bands, and the red-black colour of a
// cell is the parity of its local row plus column. A pass that updates a band's first or last row also
// stores the value into the ghost row of the neighbouring band (distributed shared memory). In a
// colour pass the neighbours read only the other colour's ghost cells, and a prolongation reads no
// ghost cell, so the stores race with no read, and one cluster barrier per pass publishes them.
// With `build` the coarse operators are formed here, beside the restriction of each level, from the
// first level's links (mg_build's sums): no launch per level before the cycle.
// It is bound by latency: about 0.6 us per pass, 77 us for the double tail from 128^2 against
// 112 + 50 us for the single-CTA tail from 64^2 and the streamed level above it.
constexpr int kClusterTail = 16;   // CTAs per cluster (a non-portable size)
constexpr int kGatherCells = 1024; // levels of at most this many cells run on CTA 0
// The cluster tail takes levels of at most this many cells (its shared memory: 7 values per cell).
template <class T> constexpr int kClusterTailCells = sizeof(T) == 4 ? 65536 : 16384;

struct ClusterTailPlan {
    int first, lg, nl;             // split levels [first, lg), gathered levels [lg, nl)
    int band[kClusterTail + 1];    // band starts of level lg - 1 for ranks 0 .. R (band[R] = its nx)
    int off[24];                   // byte offset of each level's block in every CTA's shared memory
    int rows[24];                  // rows allocated per split level (its largest band)
    int bytes;                     // dynamic shared memory per CTA
};

namespace cg = cooperative_groups;

// One colour of smooth on a band; xup / xdn: the x arrays of the bands above / below (null at the
// cluster's ends), mup: the rows of the band above (its bottom ghost row mirrors our row 0).
template <class T> __device__ void c_smooth(const SLevel<T>& L, T* xup, int mup, T* xdn, int colour) {
    const RowWalk w((L.ny + 1) / 2);
    const int S = L.S;
    for (int I = w.r; I < L.nx; I += w.dr)
        for (int J = ((I + colour) & 1) + 2 * w.c; J < L.ny; J += 2 * w.dc) {
            const int q = L.at(I, J);
            const T v = rb_value(L.b[q], L.flow(q), L.ap[q]);
            L.x[q] = v;
            if (I == 0 && xup) xup[(mup + 1) * S + J + 1] = v;
            if (I == L.nx - 1 && xdn) xdn[J + 1] = v;
        }
    cg::this_cluster().sync();
}
// prolong into the band F from rows c0 + I / 2 of the coarse level C (this CTA's band, c0 = 0, or
// the gathered level on CTA 0), with the ghost stores of c_smooth.
template <class T>
__device__ void c_prolong(const SLevel<T>& C, int c0, const SLevel<T>& F, T* xup, int mup, T* xdn, T om) {
    const RowWalk w(F.ny);
    const int S = F.S;
    for (int I = w.r; I < F.nx; I += w.dr)
        for (int J = w.c; J < F.ny; J += w.dc) {
            const int q = F.at(I, J);
            const T v = F.x[q] + om * C.x[C.at(c0 + (I >> 1), J >> 1)];
            F.x[q] = v;
            if (I == 0 && xup) xup[(mup + 1) * S + J + 1] = v;
            if (I == F.nx - 1 && xdn) xdn[J + 1] = v;
        }
    cg::this_cluster().sync();
}

template <class T>
__global__ void __launch_bounds__(kCoarseThreads)
    k_mg_tail_cluster(MgLevelsT<T> lv, ClusterTailPlan pl, int pre, int post, double omega, double tol, int build,
                      int* sweeps_out) {
    extern __shared__ __align__(16) unsigned char tail_sm[];
    cg::cluster_group cl = cg::this_cluster();
    const int R = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    const int first = pl.first, lg = pl.lg, nl = pl.nl, Lc = lg - 1;
    auto start = [&](int l, int rr) { return pl.band[rr] << (Lc - l); }; // band start of rank rr
    // this CTA's band of split level l (laid out for the level's largest band: the same offsets in
    // every CTA, so a neighbour's arrays are this CTA's mapped to its rank)
    auto band = [&](int l) {
        SLevel<T> s = slevel_at<T>(tail_sm + pl.off[l], pl.rows[l], lv.L[l].ny);
        s.nx = start(l, rank + 1) - start(l, rank);
        return s;
    };
    auto xup = [&](const SLevel<T>& s) { return rank > 0 ? cl.map_shared_rank(s.x, rank - 1) : nullptr; };
    auto xdn = [&](const SLevel<T>& s) { return rank < R - 1 ? cl.map_shared_rank(s.x, rank + 1) : nullptr; };
    auto mup = [&](int l) { return rank > 0 ? start(l, rank) - start(l, rank - 1) : 0; };
    auto gathered = [&](int l) { return slevel_at<T>(tail_sm + pl.off[l], lv.L[l].nx, lv.L[l].ny); };
    auto gathered0 = [&](int l) { // the gathered level l in CTA 0's shared memory
        SLevel<T> s = gathered(l);
        s.l4 = cl.map_shared_rank(s.l4, 0);
        s.x = cl.map_shared_rank(s.x, 0);
        s.b = cl.map_shared_rank(s.b, 0);
        s.ap = cl.map_shared_rank(s.ap, 0);
        return s;
    };
    for (int l = first; l < lg; ++l) // the bands, with their ghost rows of x
        slevel_load(lv.L[l], band(l), start(l, rank), l == first || !build, l == first);
    if (rank == 0)
        for (int l = lg; l < nl; ++l) slevel_load(lv.L[l], gathered(l), 0, !build, false);
    cl.sync(); // every CTA of the cluster has loaded before any touches another's shared memory
    const T om = static_cast<T>(omega);
    for (int l = first; l < lg; ++l) {
        const SLevel<T> s = band(l);
        for (int k = 0; k < pre; ++k) {
            c_smooth(s, xup(s), mup(l), xdn(s), 0);
            c_smooth(s, xup(s), mup(l), xdn(s), 1);
        }
        const SLevel<T> c = l + 1 < lg ? band(l + 1) : gathered0(lg);
        const int c0 = l + 1 < lg ? 0 : start(l, rank) / 2;
        s_restrict_rows(s, c, c0);
        if (build) s_build(s, c, c0);
        cl.sync();
    }
    if (rank == 0) { // the gathered levels and the coarsest solve, as k_mg_tail_smem
        for (int l = lg; l + 1 < nl; ++l) {
            const SLevel<T> L = gathered(l);
            for (int k = 0; k < pre; ++k) {
                s_smooth(L, 0);
                s_smooth(L, 1);
            }
            s_restrict_rows(L, gathered(l + 1), 0);
            if (build) s_build(L, gathered(l + 1), 0);
            __syncthreads();
        }
        s_coarse_solve(gathered(nl - 1), tol, sweeps_out);
        for (int l = nl - 2; l >= lg; --l) {
            const SLevel<T> L = gathered(l);
            s_prolong(gathered(l + 1), L, om);
            for (int k = 0; k < post; ++k) {
                s_smooth(L, 0);
                s_smooth(L, 1);
            }
        }
    }
    cl.sync();
    for (int l = lg - 1; l >= first; --l) {
        const SLevel<T> s = band(l);
        if (l + 1 < lg) c_prolong(band(l + 1), 0, s, xup(s), mup(l), xdn(s), om);
        else c_prolong(gathered0(lg), start(l, rank) / 2, s, xup(s), mup(l), xdn(s), om);
        for (int k = 0; k < post; ++k) {
            c_smooth(s, xup(s), mup(l), xdn(s), 0);
            c_smooth(s, xup(s), mup(l), xdn(s), 1);
        }
    }
    slevel_store_x(lv.L[first], band(first), start(first, rank));
}

// A level in global memory as coarse_solve's cells.
template <class T> __device__ CoarseCell<T> coarse_load(const LevelViewT<T>& L, int I, int J) {
    const int q = I * L.stride + J;
    const Links<T> k = links_written(L, q);
    return {k.e, k.w, k.n, k.s, L.AP[q], L.b[q], L.x[q]};
}

// The coarsest level alone, a cell pair per thread: one CTA, or a cluster of them with the rows split
// into bands.
struct CoarseBands {
    int band[17]; // first row of each CTA's band (band[number of CTAs] = nx)
    int rows;     // rows of the largest band
};
template <class T, class Team>
__global__ void __launch_bounds__(1024) k_mg_coarse_pairs(LevelViewT<T> L, CoarseBands pl, double tol, int* sweeps_out) {
    extern __shared__ __align__(16) unsigned char tail_dyn[];
    const Team team{static_cast<int>(blockDim.x)};
    const int rank = team.rank(), i0 = pl.band[rank];
    coarse_solve<T>(
        team, L.nx, L.ny, i0, pl.band[rank + 1] - i0, rank > 0 ? i0 - pl.band[rank - 1] : 0, tol,
        coarse_smem<T>(tail_dyn, L.nx, pl.rows, L.ny), [&](int I, int J) { return coarse_load(L, I, J); },
        [&](int I, int J, T x, T b) {
            const int q = I * L.stride + J;
            L.x[q] = x;
            L.b[q] = b;
        },
        sweeps_out);
}

template <class T>
__global__ void __launch_bounds__(kCoarseThreads) k_mg_coarse(LevelViewT<T> L, double* rowbuf,
                                                              double tol, int* sweeps_out) {
    cta_coarse_solve(L, rowbuf, tol, sweeps_out);
}

// Levels [first, nl) of one V-cycle (mg_vcycle, multigrid.cpp:299-323) in one CTA: the small
// levels are latency-bound, so they run back to back with a block barrier between passes.
template <class T>
__global__ void __launch_bounds__(kCoarseThreads)
    k_mg_tail(MgLevelsT<T> lv, int first, int pre, int post, double omega, double tol,
              double* rowbuf, int* sweeps_out, int pairs, int build) {
    extern __shared__ __align__(16) unsigned char tail_dyn[];
    const int nl = lv.n;
    for (int l = first; l + 1 < nl; ++l) {
        if (build) cta_build(lv.L[l], lv.L[l + 1]);
        for (int s = 0; s < pre; ++s) {
            cta_smooth_colour(lv.L[l], 0);
            cta_smooth_colour(lv.L[l], 1);
        }
        cta_residual(lv.L[l]);
        cta_restrict(lv.L[l], lv.L[l + 1]);
    }
    if (pairs) {
        const LevelViewT<T>& L = lv.L[nl - 1];
        const CoarseCta team{coarse_threads(L.nx, L.ny)};
        __syncthreads();
        if (static_cast<int>(threadIdx.x) < team.nt)
            coarse_solve<T>(
                team, L.nx, L.ny, 0, L.nx, 0, tol, coarse_smem<T>(tail_dyn, L.nx, L.nx, L.ny),
                [&](int I, int J) { return coarse_load(L, I, J); },
                [&](int I, int J, T x, T b) {
                    const int q = I * L.stride + J;
                    L.x[q] = x;
                    L.b[q] = b;
                },
                sweeps_out);
        __syncthreads();
    } else {
        cta_coarse_solve(lv.L[nl - 1], rowbuf, tol, sweeps_out);
    }
    for (int l = nl - 2; l >= first; --l) {
        cta_prolong(lv.L[l + 1], lv.L[l], omega);
        for (int s = 0; s < post; ++s) {
            cta_smooth_colour(lv.L[l], 0);
            cta_smooth_colour(lv.L[l], 1);
        }
    }
}

} // namespace

// The tail runs with every level in shared memory when they fit (the 64^2-and-below float levels of a
// square grid take about 170 KB, the 32^2-and-below double ones 100 KB); otherwise through global memory.
constexpr int kTailSmemMax = 200 * 1024;
// Shared memory of a pair solve: any level of 1024 threads per CTA takes less.
constexpr int kCoarseSmemMax = 160 * 1024;

// The coarsest level alone, where its pairs fit: one CTA up to 1024 threads (about 2048 cells), then a
// cluster of 8 CTAs, then of 16 (about 32768 cells); beyond that (or fewer rows than CTAs) false. One
// CTA's block barrier is a fraction of a cluster barrier, so it goes first; 8 CTAs are the largest
// portable cluster. 37 x 37 FP64, 200 sweeps: 0.28 ms (one warp on shared memory: 6.31 ms); 75 x 125
// FP32, 200 sweeps: 0.23 ms in a cluster of 8 (one CTA on global memory: 5.63 ms).
template <class T>
bool launch_coarse_pairs(const LevelViewT<T>& L, bool clusters, double tol, int* sweeps_out, cudaStream_t st) {
    CoarseBands pl{};
    auto plan = [&](int ctas) {
        pl.rows = (L.nx + ctas - 1) / ctas;
        for (int r = 0; r <= ctas; ++r) pl.band[r] = static_cast<int>(static_cast<long long>(r) * L.nx / ctas);
        return L.nx >= ctas && static_cast<long long>(pl.rows) * coarse_hp(L.ny) <= 1024 &&
               coarse_smem_bytes<T>(L.nx, pl.rows, L.ny) <= kCoarseSmemMax;
    };
    if (plan(1)) {
        static PerDeviceOnce attr;
        attr.get([] {
            SGPU_CUDA(cudaFuncSetAttribute(k_mg_coarse_pairs<T, CoarseCta>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, kCoarseSmemMax));
            return 0;
        });
        k_mg_coarse_pairs<T, CoarseCta><<<1, coarse_threads(L.nx, L.ny), coarse_smem_bytes<T>(L.nx, L.nx, L.ny), st>>>(
            L, pl, tol, sweeps_out);
        SGPU_LAUNCH();
        return true;
    }
    if (!clusters) return false;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // clusters of this size that this device runs (0: none), its attributes set once per device
    auto available = [&](int ctas) {
        static PerDeviceOnce attr, fit8, fit16;
        const int ok = attr.get([] {
            const bool set = cudaFuncSetAttribute(k_mg_coarse_pairs<T, CoarseCluster>,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  kCoarseSmemMax) == cudaSuccess &&
                             cudaFuncSetAttribute(k_mg_coarse_pairs<T, CoarseCluster>,
                                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
            if (!set) (void)cudaGetLastError();
            return set ? 1 : 0;
        });
        return ok && (ctas == 8 ? fit8 : fit16).get([&] {
            cfg.gridDim = dim3(ctas);
            cfg.blockDim = dim3(1024);
            cfg.dynamicSmemBytes = kCoarseSmemMax;
            at[0].val.clusterDim.x = static_cast<unsigned>(ctas);
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k_mg_coarse_pairs<T, CoarseCluster>, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
            return n;
        }) > 0;
    };
    for (int ctas : {8, 16}) {
        if (!plan(ctas) || !available(ctas)) continue;
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(coarse_threads(pl.rows, L.ny));
        cfg.dynamicSmemBytes = static_cast<std::size_t>(coarse_smem_bytes<T>(L.nx, pl.rows, L.ny));
        cfg.stream = st;
        at[0].val.clusterDim.x = static_cast<unsigned>(ctas);
        SGPU_CUDA(cudaLaunchKernelEx(&cfg, k_mg_coarse_pairs<T, CoarseCluster>, L, pl, tol, sweeps_out));
        SGPU_LAUNCH();
        return true;
    }
    return false;
}

template <class T>
void launch_mg_tail(const MgLevelsT<T>& lv, int first, int pre, int post, double omega, double tol,
                    double* rowbuf, int* sweeps_out, cudaStream_t st, bool build) {
    const LevelViewT<T>& Lc = lv.L[lv.n - 1];
    if (first == lv.n - 1 && launch_coarse_pairs(Lc, lv.clusters, tol, sweeps_out, st)) return;
    // pair solve inside the tail: a thread of the block per pair
    const bool pairs = static_cast<long long>(Lc.nx) * coarse_hp(Lc.ny) <= kCoarseThreads;
    TailSmem ts{};
    long long bytes = 0;
    for (int l = first; l < lv.n && l < 24 && bytes <= kTailSmemMax; ++l) {
        ts.off[l] = static_cast<int>(bytes);
        bytes += static_cast<long long>(lv.L[l].nx + 2) * (lv.L[l].ny + 2) * 7 * static_cast<int>(sizeof(T)) + 16;
        bytes = bytes / 16 * 16;
    }
    if (lv.n <= 24 && bytes <= kTailSmemMax && pairs) {
        static PerDeviceOnce attr; // the attribute lives in each device's context
        attr.get([] {
            SGPU_CUDA(cudaFuncSetAttribute(k_mg_tail_smem<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kTailSmemMax));
            return 0;
        });
        ts.bytes = static_cast<int>(bytes);
        k_mg_tail_smem<T><<<1, kCoarseThreads, ts.bytes, st>>>(lv, first, pre, post, omega, tol, ts, build ? 1 : 0,
                                                               sweeps_out);
        SGPU_LAUNCH();
        return;
    }
    static PerDeviceOnce attr;
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_mg_tail<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kCoarseSmemMax));
        return 0;
    });
    const int dyn = pairs ? coarse_smem_bytes<T>(Lc.nx, Lc.nx, Lc.ny) : 0;
    k_mg_tail<T><<<1, kCoarseThreads, dyn, st>>>(lv, first, pre, post, omega, tol, rowbuf, sweeps_out, pairs ? 1 : 0,
                                                 build ? 1 : 0);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_build(const LevelViewT<T>& F, const LevelViewT<T>& C, cudaStream_t st) {
    k_mg_build<T><<<grid2(C.nx, C.ny), dim3(BX, BY), 0, st>>>(F, C);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_smooth_colour(const LevelViewT<T>& L, int colour, cudaStream_t st) {
    k_mg_smooth<T><<<grid2(L.nx, L.ny), dim3(BX, BY), 0, st>>>(L, colour);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_residual(const LevelViewT<T>& L, cudaStream_t st) {
    k_mg_residual<T><<<grid2(L.nx, L.ny), dim3(BX, BY), 0, st>>>(L);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_restrict(const LevelViewT<T>& F, const LevelViewT<T>& C, cudaStream_t st) {
    k_mg_restrict<T><<<grid2(F.nx / 2, F.ny / 2), dim3(BX, BY), 0, st>>>(F, C);
    SGPU_LAUNCH();
}
template <class T>
void launch_mg_prolong(const LevelViewT<T>& C, const LevelViewT<T>& F, double omega, cudaStream_t st) {
    k_mg_prolong<T><<<grid2(F.nx, F.ny), dim3(BX, BY), 0, st>>>(C, F, omega);
    SGPU_LAUNCH();
}
template <class T>
void launch_mg_coarse(const LevelViewT<T>& L, double* rowbuf, double tol, int* sweeps_out, cudaStream_t st) {
    k_mg_coarse<T><<<1, kCoarseThreads, 0, st>>>(L, rowbuf, tol, sweeps_out);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_residual_sq(const LevelViewT<T>& L, double* cells, cudaStream_t st) {
    k_mg_residual_sq<T><<<grid2(L.nx, L.ny), dim3(BX, BY), 0, st>>>(L, cells);
    SGPU_LAUNCH();
}
template <class T> void launch_mg_b_sq(const LevelViewT<T>& L, double* cells, cudaStream_t st) {
    k_mg_b_sq<T><<<grid2(L.nx, L.ny), dim3(BX, BY), 0, st>>>(L, cells);
    SGPU_LAUNCH();
}
#ifndef SGPU_FLOAT_UNIT
void launch_mg_sub_mean(const LevelView& L, double* x, const double* sum, cudaStream_t st) {
    k_mg_sub_mean<<<grid2(L.nx, L.ny), dim3(BX, BY), 0, st>>>(L, x, sum);
    SGPU_LAUNCH();
}
namespace {
__global__ void k_quotient(const double* a, const double* ap, int n, double* out) {
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) out[i] = quotient(a[i], ap[i], inverse(ap[i]));
}
} // namespace
void launch_quotient(const double* a, const double* ap, int n, double* out, cudaStream_t st) {
    if (n <= 0) return;
    k_quotient<<<(n + 255) / 256, 256, 0, st>>>(a, ap, n, out);
    SGPU_LAUNCH();
}
bool mg_clusters_enabled() {
    const char* e = std::getenv("SGPU_MG_CLUSTER");
    return !e || std::atoi(e) != 0;
}
#endif

namespace {
// Dynamic shared memory per CTA of the cluster tail (the 227 KB a CTA may have).
constexpr int kClusterSmemMax = 227 * 1024;

// The cluster tail's plan from level `first`; false where it does not apply: fewer than one split
// level, a split level that does not halve exactly into the next, a coarsest split level of fewer
// than 2 rows per CTA, or more shared memory per CTA than kClusterSmemMax.
template <class T> bool cluster_tail_plan(const MgLevelsT<T>& lv, int first, ClusterTailPlan& pl) {
    const int nl = lv.n;
    if (nl > 24 || first < 0 || first >= nl - 1) return false;
    int lg = first;
    while (lg < nl - 1 && lv.L[lg].nx * lv.L[lg].ny > kGatherCells) ++lg;
    if (lg == first || lv.L[lg].nx * lv.L[lg].ny > kGatherCells) return false;
    if (lv.L[nl - 1].nx * coarse_hp(lv.L[nl - 1].ny) > kCoarseThreads) return false; // the coarse solve's pairs
    for (int l = first; l < lg; ++l)
        if (lv.L[l].nx != 2 * lv.L[l + 1].nx || lv.L[l].ny != 2 * lv.L[l + 1].ny) return false;
    const int Lc = lg - 1, nxc = lv.L[Lc].nx;
    if (nxc < 2 * kClusterTail) return false;
    pl.first = first;
    pl.lg = lg;
    pl.nl = nl;
    for (int r = 0; r < kClusterTail; ++r) pl.band[r] = 2 * ((r * (nxc / 2)) / kClusterTail);
    pl.band[kClusterTail] = nxc;
    if (lv.L[first].nx * lv.L[first].ny > kClusterTailCells<T>) return false;
    int bytes = 0;
    for (int l = first; l < lg; ++l) {
        int rows = 0;
        for (int r = 0; r < kClusterTail; ++r) rows = std::max(rows, (pl.band[r + 1] - pl.band[r]) << (Lc - l));
        pl.rows[l] = rows;
        pl.off[l] = bytes;
        bytes += slevel_bytes<T>(rows, lv.L[l].ny);
    }
    for (int l = lg; l < nl; ++l) {
        pl.off[l] = bytes;
        bytes += slevel_bytes<T>(lv.L[l].nx, lv.L[l].ny);
    }
    pl.bytes = bytes;
    return bytes <= kClusterSmemMax;
}

// Whether this device runs the cluster tail: its function attributes set (the dynamic shared memory
// and the non-portable cluster size, once per device) and at least one such cluster resident.
template <class T> bool cluster_tail_available() {
    static PerDeviceOnce once;
    return once.get([] {
        // a device that refuses either attribute runs the kernels without a cluster
        if (cudaFuncSetAttribute(k_mg_tail_cluster<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmemMax) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_mg_tail_cluster<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterTail);
        cfg.blockDim = dim3(kCoarseThreads);
        cfg.dynamicSmemBytes = kClusterSmemMax;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClusterTail;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k_mg_tail_cluster<T>, &cfg) != cudaSuccess) {
            (void)cudaGetLastError(); // not supported here: the clear-up of the failed query
            return 0;
        }
        return n > 0 ? 1 : 0;
    }) != 0;
}
} // namespace

template <class T> int mg_cluster_tail_first(const MgLevelsT<T>& lv, int fallback) {
    if (!lv.clusters || !cluster_tail_available<T>()) return fallback;
    int t = 0;
    while (t < lv.n - 1 && lv.L[t].nx * lv.L[t].ny > kClusterTailCells<T>) ++t;
    ClusterTailPlan pl{};
    for (; t < fallback; ++t)
        if (cluster_tail_plan(lv, t, pl)) return t;
    return fallback;
}

template <class T>
bool launch_mg_tail_cluster(const MgLevelsT<T>& lv, int first, int pre, int post, double omega, double tol,
                            int* sweeps_out, cudaStream_t st, bool build) {
    ClusterTailPlan pl{};
    if (!cluster_tail_plan(lv, first, pl)) return false;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterTail);
    cfg.blockDim = dim3(kCoarseThreads);
    cfg.dynamicSmemBytes = static_cast<std::size_t>(pl.bytes);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClusterTail;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SGPU_CUDA(cudaLaunchKernelEx(&cfg, k_mg_tail_cluster<T>, lv, pl, pre, post, omega, tol, build ? 1 : 0,
                                 sweeps_out));
    SGPU_LAUNCH();
    return true;
}
#define SGPU_MG_INST(T)                                                                            \
    template void launch_mg_tail<T>(const MgLevelsT<T>&, int, int, int, double, double, double*,   \
                                    int*, cudaStream_t, bool);                                     \
    template int mg_cluster_tail_first<T>(const MgLevelsT<T>&, int);                               \
    template bool launch_mg_tail_cluster<T>(const MgLevelsT<T>&, int, int, int, double, double,    \
                                            int*, cudaStream_t, bool);                             \
    template void launch_mg_build<T>(const LevelViewT<T>&, const LevelViewT<T>&, cudaStream_t);    \
    template void launch_mg_smooth_colour<T>(const LevelViewT<T>&, int, cudaStream_t);             \
    template void launch_mg_residual<T>(const LevelViewT<T>&, cudaStream_t);                       \
    template void launch_mg_restrict<T>(const LevelViewT<T>&, const LevelViewT<T>&, cudaStream_t); \
    template void launch_mg_prolong<T>(const LevelViewT<T>&, const LevelViewT<T>&, double,         \
                                       cudaStream_t);                                              \
    template void launch_mg_coarse<T>(const LevelViewT<T>&, double*, double, int*, cudaStream_t);  \
    template void launch_mg_residual_sq<T>(const LevelViewT<T>&, double*, cudaStream_t);           \
    template void launch_mg_b_sq<T>(const LevelViewT<T>&, double*, cudaStream_t);
// This file alone instantiates the double kernels (built without contraction: the reference's
// bits); mg32.cu includes it with SGPU_FLOAT_UNIT for the float ones (contraction allowed).
#ifndef SGPU_FLOAT_UNIT
SGPU_MG_INST(double)
#else
SGPU_MG_INST(float)
#endif
#undef SGPU_MG_INST

} // namespace sgpu
