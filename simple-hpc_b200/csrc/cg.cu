// cg.cu — Jacobi-preconditioned conjugate gradient for p' on the device (solve_pc_cg,
// src/pressure.cpp:208-317), FP64 and bit-identical to the reference.
//
// The scalars (alpha, beta, the mean corrections, the stopping test) live in device memory and are
// updated by one-thread kernels between the per-cell passes, so an iteration needs no host round
// trip; once the solve stops, every later kernel of the launch sequence sees `done` and returns.
// Sums of per-cell values go through the ordered reduction (reduce.cu) in CellSums order.
// Grids whose rows fit the shared memory of one CTA per SM run the whole solve in one cooperative kernel
// instead (k_cg_persist); the pass-by-pass kernels take the others.
#include "kernels.hpp"
#include "blocksum.cuh"

#include <algorithm>

namespace sgpu {

namespace {

constexpr int BX = 32, BY = 8;

__device__ __forceinline__ bool cell_p(const DevParams& p, int& i, int& j) {
    j = p.H + 1 + static_cast<int>(blockIdx.x * BX + threadIdx.x);
    i = p.H + static_cast<int>(blockIdx.y * BY + threadIdx.y);
    return i <= p.NX + p.H - 1 && j <= p.NY + p.H;
}

dim3 grid_p(const DevParams& p) { return dim3((p.NY + BX - 1) / BX, (p.NX + BY - 1) / BY); }

// Plane offset of cell (i, j) in the compact NX x NY cell buffer.
__device__ __forceinline__ std::size_t cell_ix(const DevParams& p, int i, int j) {
    return static_cast<std::size_t>(i - p.H) * p.NY + (j - p.H - 1);
}

// r = b - mb, z = r / APP; values rr, z, r.z, r (pressure.cpp:230-245).
__global__ void k_cg_init(DevParams p, PressurePtr w, CgPtr cg, const CgScalars* sc,
                          double* cells, std::size_t plane) {
    int i, j;
    if (!cell_p(p, i, j)) return;
    const std::size_t q = static_cast<std::size_t>(i) * p.pitch + j, c = cell_ix(p, i, j);
    const double ri = w.b[q] - sc->mb;
    cg.r[q] = ri;
    const double zi = ri / w.APP[q];
    cg.z[q] = zi;
    cells[c] = ri * ri;
    cells[plane + c] = zi;
    cells[2 * plane + c] = ri * zi;
    cells[3 * plane + c] = ri;
}

// d = z - mz (pressure.cpp:253-256).
__global__ void k_cg_dinit(DevParams p, CgPtr cg, const CgScalars* sc) {
    if (sc->done) return;
    int i, j;
    if (!cell_p(p, i, j)) return;
    const std::size_t q = static_cast<std::size_t>(i) * p.pitch + j;
    cg.d[q] = cg.z[q] - sc->mz;
}

// q = A d, value d.q (pressure.cpp:263-274).
__global__ void k_cg_dq(DevParams p, PressurePtr w, CgPtr cg, const CgScalars* sc, double* cells) {
    if (sc->done) return;
    int i, j;
    if (!cell_p(p, i, j)) return;
    const std::size_t q = static_cast<std::size_t>(i) * p.pitch + j, ld = p.pitch;
    const double* d = cg.d;
    const double qi = w.APP[q] * d[q] -
                      (w.AEP[q] * d[q + 1] + w.AWP[q] * d[q - 1] + w.ASP[q] * d[q + ld] +
                       w.ANP[q] * d[q - ld]);
    cg.q[q] = qi;
    cells[cell_ix(p, i, j)] = d[q] * qi;
}

// x += alpha d; r -= alpha q; z = r / APP; values rr, z, r.z, r (pressure.cpp:278-292).
__global__ void k_cg_update(DevParams p, PressurePtr w, CgPtr cg, const CgScalars* sc,
                            double* cells, std::size_t plane) {
    if (sc->done) return;
    int i, j;
    if (!cell_p(p, i, j)) return;
    const std::size_t q = static_cast<std::size_t>(i) * p.pitch + j, c = cell_ix(p, i, j);
    const double alpha = sc->alpha;
    w.pc[q] += alpha * cg.d[q];
    const double ri = cg.r[q] - alpha * cg.q[q];
    cg.r[q] = ri;
    const double zi = ri / w.APP[q];
    cg.z[q] = zi;
    cells[c] = ri * ri;
    cells[plane + c] = zi;
    cells[2 * plane + c] = ri * zi;
    cells[3 * plane + c] = ri;
}

// d = (z - mz) + beta d (pressure.cpp:306-309).
__global__ void k_cg_dir(DevParams p, CgPtr cg, const CgScalars* sc) {
    if (sc->done) return;
    int i, j;
    if (!cell_p(p, i, j)) return;
    const std::size_t q = static_cast<std::size_t>(i) * p.pitch + j;
    cg.d[q] = (cg.z[q] - sc->mz) + sc->beta * cg.d[q];
}

// Scalar steps between the passes. sums holds the ordered sums of the preceding pass.
//  0: mb = sum(b) / n                                  (pressure.cpp:226-228)
//  1: after the init pass: rr == 0 -> done; nb, mz, rz (pressure.cpp:246-252)
//  2: after the d.q pass: breakdown test, alpha        (pressure.cpp:275-277)
//  3: after the update pass: k, rel, stop test, beta   (pressure.cpp:293-305)
__global__ void k_cg_scalars(int stage, CgScalars* sc, const double* sums) {
    if (stage == 0) {
        sc->k = 0;
        sc->done = 0;
        sc->rel = 0.0;
        sc->mb = sums[0] / sc->n;
        return;
    }
    if (sc->done) return;
    if (stage == 1) {
        const double rr = sums[0], sz = sums[1], rz = sums[2], sr = sums[3];
        if (rr == 0.0) {
            sc->done = 1; // ||b|| == 0: p' = 0
            return;
        }
        sc->nb = sqrt(rr);
        sc->mz = sz / sc->n;
        sc->rz = rz - sc->mz * sr;
        sc->rel = 1.0;
        if (sc->maxit <= 0) sc->done = 1;
    } else if (stage == 2) {
        const double dq = sums[0];
        if (!(dq > 0.0)) {
            sc->done = 1; // breakdown: stop with the current x
            return;
        }
        sc->alpha = sc->rz / dq;
    } else {
        const double rr = sums[0], sz = sums[1], sr = sums[3];
        double rzn = sums[2];
        sc->k += 1;
        sc->rel = sqrt(rr) / sc->nb;
        if (sc->rel <= sc->tol) {
            sc->done = 1;
            return;
        }
        sc->mz = sz / sc->n;
        rzn -= sc->mz * sr;
        sc->beta = rzn / sc->rz;
        sc->rz = rzn;
        // The reference still updates d before its loop test fails; d is not read afterwards.
        if (sc->k >= sc->maxit) sc->done = 2;
    }
}

// ---- the whole solve in one kernel ----
//
// An iteration has two sums over the grid, each a chain of nc adds per row and then one of nr adds over
// the rows: at 8 cycles an add (the order is the reference's, so they cannot be split) 2 (nc + nr) adds
// are a floor of 9 us at 512^2. The pass-by-pass kernels took 59 us there: seven launches and their gaps,
// the chains waiting behind passes over memory. Here one CTA per SM owns R rows for the whole solve and
// an iteration is two phases:
//   A  d = (z - mz) + beta d on the own rows and one halo row each side (shared memory; the halo needs
//      only the neighbours' z), q = A d, values d q;
//   B  x += alpha d, r -= alpha q, z = r / APP, values r r, z, r z, r.
// Eight warps form a phase's values in chunks of columns (128, or 32 or 64 on narrow grids) in a ring of shared-memory buffers, and
// `cw` further warps, a lane per row and plane, add them in column order while the next chunks are
// formed: the passes hide behind the chains, as far as their arrays fit the shared memory too (CgArray; all
// at 512^2, none at 1200^2). The row sums then go to memory, and every CTA waits for all of them, adds
// them (a lane per plane) and forms the scalars: that wait is the grid's only synchronisation. A row sum
// is its own flag: an entry holds kCgEmpty, a signalling NaN that no arithmetic produces, until its sum is
// stored (release; read with acquire). Three buffers take turns: the lane that stores a sum in phase p has
// seen every sum of phase p - 1, so every CTA has read phase p - 2, and it empties its entry of that
// buffer, the one of phase p + 1, first.
// The per-cell expressions and the scalars' are those of the kernels above.
// Waits are bounded: a CTA that gives up sets *err, which ends every other wait, and the kernel returns.
// Measured at 512^2 (UDS, 1e-6): 20 us an iteration against 59.
constexpr int kCgBufs = 3, kCgWork = 256;
constexpr int kCgSpin = 1 << 22;
constexpr int kCgSmem = 220 * 1024;

struct CgPlan {
    int R, G, cw; // rows per CTA, CTAs, chain warps
    int sh;       // log2 of the columns of a chunk
    int dld;      // row stride of d in shared memory
    int held;     // how many of the arrays of CgArray, in its order, are in shared memory
    int bytes;    // dynamic shared memory
};

// The per-cell arrays of the solve, in the order in which they take what shared memory is left: those
// written every iteration first.
enum CgArray { kCgZ, kCgR, kCgQ, kCgX, kCgAPP, kCgE, kCgW, kCgS, kCgN, kCgArrays };

constexpr unsigned long long kCgEmpty = 0xFFF7C6C6C6C6C6C6ull; // (see above)
__global__ void k_cg_empty(unsigned long long* sums, int n) {
    for (int k = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x); k < n; k += static_cast<int>(gridDim.x * blockDim.x))
        sums[k] = kCgEmpty;
}

__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory"); }

__global__ void __launch_bounds__(kCgWork + 128)
    k_cg_persist(DevParams p, PressurePtr w, CgPtr cg, CgScalars* sc, unsigned long long* sums, unsigned* err,
                 CgPlan pl) {
    extern __shared__ __align__(16) double cg_mem[];
    __shared__ double tot[4];
    __shared__ int stop;
    const int nr = p.NX, nc = p.NY, R = pl.R, H = p.H;
    const int tid = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    const bool work = tid < kCgWork;
    const int r0 = static_cast<int>(blockIdx.x) * R, m = min(R, nr - r0);
    const int cc = 1 << pl.sh, nch = (nc + cc - 1) >> pl.sh;
    const int tc = tid & (cc - 1), tr = tid >> pl.sh, rstep = kCgWork >> pl.sh; // column, first row, row step
    const int sld = cc + 2; // staged row stride: lanes of the chain read distinct banks, 16 bytes each
    double* stage = cg_mem;                                // kCgBufs x 4 planes x R rows
    double* fin = stage;                                   // all row sums of up to 4 planes, between phases
    const int nrp = (nr + 1) & ~1;                         // ... a plane of them
    double* ds = stage + max(kCgBufs * 4 * R * sld, 4 * nrp); // d on rows -1 .. R, columns -1 .. nc
    auto dat = [&](int r, int c) -> double& { return ds[(r + 1) * pl.dld + c + 1]; };
    const int ld = p.pitch;
    const std::size_t origin = static_cast<std::size_t>(H + r0) * ld + (H + 1); // this CTA's first cell
    // Each array as a base and a row stride, in shared memory or where it lies.
    double* base[kCgArrays] = {cg.z + origin,  cg.r + origin,  cg.q + origin,  w.pc + origin, w.APP + origin,
                               w.AEP + origin, w.AWP + origin, w.ASP + origin, w.ANP + origin};
    int stride[kCgArrays];
    {
        double* held = ds + (R + 2) * pl.dld;
#pragma unroll
        for (int k = 0; k < kCgArrays; ++k) {
            stride[k] = ld;
            if (k < pl.held) {
                double* dst = held + k * R * nc;
                for (int r = 0; r < m; ++r)
                    for (int c = tid; c < nc; c += nt) dst[r * nc + c] = base[k][static_cast<std::size_t>(r) * ld + c];
                base[k] = dst;
                stride[k] = nc;
            }
        }
    }
    auto val = [&](int k, int r, int c) -> double& { return base[k][static_cast<std::size_t>(r) * stride[k] + c]; };
    // z of the own rows, and of the first and last of them in memory for the neighbours' halo rows
    auto zat = [&](int r, int c) { return cg.z + origin + static_cast<std::ptrdiff_t>(r) * ld + c; };
    auto put_z = [&](int r, int c, double z) {
        val(kCgZ, r, c) = z;
        if (pl.held && (r == 0 || r == m - 1)) *zat(r, c) = z;
    };
    int turn = 0; // the buffer of this phase
    if (tid == 0) stop = 0;
    for (int q = tid; q < (R + 2) * pl.dld; q += nt) ds[q] = 0.0;
    __syncthreads();

    // One phase: form(chunk, buffer) by the working warps, K ordered sums over the grid into tot; false
    // when a wait has given up.
    // beside: what the working warps do while the row sums are added.
    auto phase = [&](int K, auto form, auto beside) -> bool {
        unsigned long long* now = sums + static_cast<std::size_t>(turn) * 4 * nr;
        turn = turn == 2 ? 0 : turn + 1;
        unsigned long long* next = sums + static_cast<std::size_t>(turn) * 4 * nr;
        if (work) {
            for (int c = 0; c < nch; ++c) {
                const int b = c % kCgBufs;
                __syncwarp();
                if (c >= kCgBufs) named_sync(4 + b, nt);
                form(c, stage + b * 4 * R * sld);
                __syncwarp();
                named_arrive(1 + b, nt);
            }
        } else {
            const int l = tid - kCgWork, r = l / K, k = l - r * K;
            const bool on = r < m;
            double a = 0.0;
            for (int c = 0; c < nch; ++c) {
                const int b = c % kCgBufs;
                __syncwarp();
                named_sync(1 + b, nt);
                if (on) a = ordered_chain(a, stage + (b * 4 * R + k * R + r) * sld, min(cc, nc - c * cc));
                __syncwarp();
                if (c + kCgBufs < nch) named_arrive(4 + b, nt);
            }
            if (on) {
                const int row = r0 + r;
                for (int e = k; e < 4; e += K) next[static_cast<std::size_t>(e) * nr + row] = kCgEmpty;
                asm volatile("st.release.gpu.global.u64 [%0], %1;\n" ::"l"(now + static_cast<std::size_t>(k) * nr + row),
                             "l"(__double_as_longlong(a))
                             : "memory");
            }
        }
        __syncthreads(); // the staging buffers are free
        const int all = K * nr;
        for (int q0 = tid; q0 < all; q0 += 8 * nt) { // eight loads in flight
            unsigned long long x[8];
            bool wait = true;
            for (int it = 0; wait; ++it) {
                wait = false;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (q0 + u * nt >= all || (it && x[u] != kCgEmpty)) continue;
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(x[u]) : "l"(now + q0 + u * nt) : "memory");
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) wait = wait || (q0 + u * nt < all && x[u] == kCgEmpty);
                if (wait && (it & 63) == 63) {
                    unsigned e;
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(e) : "l"(err) : "memory");
                    if (e || it > kCgSpin) {
                        atomicOr(err, 1u);
                        stop = 1;
                        break;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int q = q0 + u * nt, k = q / nr;
                if (q < all) fin[k * nrp + (q - k * nr)] = __longlong_as_double(static_cast<long long>(x[u]));
            }
        }
        __threadfence(); // with the relaxed loads: an acquire
        __syncthreads();
        if (stop) return false;
        if (work) beside();
        else if (tid - kCgWork < K) tot[tid - kCgWork] = ordered_chain(0.0, fin + (tid - kCgWork) * nrp, nr);
        __syncthreads();
        return true;
    };
    // This thread's cells of a chunk, two at a time: load(row, column, i) for both, then form(row, column, i,
    // its staged values), so that the loads of both are in flight together.
    auto cells = [&](int c, double* st, auto load, auto form) {
        const int col = c * cc + tc;
        if (col >= nc) return;
        for (int r = tr; r < m; r += 2 * rstep) {
            const bool two = r + rstep < m;
            load(r, col, 0);
            if (two) load(r + rstep, col, 1);
            form(r, col, 0, st + r * sld + tc);
            if (two) form(r + rstep, col, 1, st + (r + rstep) * sld + tc);
        }
    };
    double a0[2], a1[2], a2[2], a3[2], a4[2];
    const int plane = R * sld;
    auto values4 = [&](double* v, double ri, double zi) { // r r, z, r z, r
        v[0] = ri * ri;
        v[plane] = zi;
        v[2 * plane] = ri * zi;
        v[3 * plane] = ri;
    };

    const double n = sc->n, tol = sc->tol;
    const int maxit = sc->maxit;
    int k = 0, done = 0;
    double rel = 0.0;
    // z of the halo rows at this thread's first two columns (u >> 1; u & 1: the row below), fetched while the
    // chain warps add the row sums that say it is final.
    double hz[4] = {0.0, 0.0, 0.0, 0.0};
    auto halo_at = [&](int u, int c) { return c < nc && (u & 1 ? r0 + m < nr : r0 > 0); };
    auto fetch_halo = [&] {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = tid + (u >> 1) * kCgWork;
            if (halo_at(u, c)) hz[u] = __ldcg(zat(u & 1 ? m : -1, c));
        }
    };
    auto load_b = [&](int r, int c, int i) { a0[i] = w.b[origin + static_cast<std::size_t>(r) * ld + c]; };
    auto nothing = [] {};
    bool live = phase(1, [&](int c, double* st) { cells(c, st, load_b, [&](int, int, int i, double* v) { *v = a0[i]; }); }, nothing);
    const double mb = live ? tot[0] / n : 0.0;
    if (live)
        live = phase(4, [&](int c, double* st) {
            cells(
                c, st,
                [&](int r, int col, int i) {
                    load_b(r, col, i);
                    a1[i] = val(kCgAPP, r, col);
                },
                [&](int r, int col, int i, double* v) {
                    const double ri = a0[i] - mb, zi = ri / a1[i];
                    val(kCgR, r, col) = ri;
                    put_z(r, col, zi);
                    values4(v, ri, zi);
                });
        }, fetch_halo);
    double nb = 0.0, mz = 0.0, rz = 0.0, alpha = 0.0, beta = 0.0;
    if (live) {
        const double rr = tot[0], sz = tot[1], srz = tot[2], sr = tot[3];
        if (rr == 0.0) done = 1; // ||b|| == 0: p' = 0
        else {
            nb = sqrt(rr);
            mz = sz / n;
            rz = srz - mz * sr;
            rel = 1.0;
            if (maxit <= 0) done = 1;
        }
    }
    while (live && !done) {
        const bool first = k == 0;
        auto next_d = [&](double& d, double z) { d = first ? z - mz : (z - mz) + beta * d; };
        auto dir = [&](int c) { // d of chunk c on the own rows
            const int col = c * cc + tc;
            if (c < nch && col < nc)
                for (int r = tr; r < m; r += rstep) next_d(dat(r, col), val(kCgZ, r, col));
        };
        auto halo = [&] { // d on the halo rows
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (halo_at(u, tid + (u >> 1) * kCgWork)) next_d(dat(u & 1 ? m : -1, tid + (u >> 1) * kCgWork), hz[u]);
            for (int c = tid + 2 * kCgWork; c < nc; c += kCgWork)
                for (int u = 0; u < 2; ++u)
                    if (halo_at(u, c)) next_d(dat(u ? m : -1, c), __ldcg(zat(u ? m : -1, c)));
        };
        live = phase(1, [&](int c, double* st) {
            if (c == 0) {
                halo();
                dir(0);
            }
            dir(c + 1);
            __syncwarp();
            named_sync(7, kCgWork);
            cells(
                c, st,
                [&](int r, int col, int i) {
                    a0[i] = val(kCgAPP, r, col);
                    a1[i] = val(kCgE, r, col);
                    a2[i] = val(kCgW, r, col);
                    a3[i] = val(kCgS, r, col);
                    a4[i] = val(kCgN, r, col);
                },
                [&](int r, int col, int i, double* v) {
                    const double d = dat(r, col);
                    const double qi = a0[i] * d - (a1[i] * dat(r, col + 1) + a2[i] * dat(r, col - 1) +
                                                   a3[i] * dat(r + 1, col) + a4[i] * dat(r - 1, col));
                    val(kCgQ, r, col) = qi;
                    *v = d * qi;
                });
        }, nothing);
        if (!live) break;
        const double dq = tot[0];
        if (!(dq > 0.0)) { // breakdown: stop with the current x
            done = 1;
            break;
        }
        alpha = rz / dq;
        live = phase(4, [&](int c, double* st) {
            cells(
                c, st,
                [&](int r, int col, int i) {
                    a0[i] = val(kCgX, r, col);
                    a1[i] = val(kCgR, r, col);
                    a2[i] = val(kCgQ, r, col);
                    a3[i] = val(kCgAPP, r, col);
                },
                [&](int r, int col, int i, double* v) {
                    val(kCgX, r, col) = a0[i] + alpha * dat(r, col);
                    const double ri = a1[i] - alpha * a2[i];
                    val(kCgR, r, col) = ri;
                    const double zi = ri / a3[i];
                    put_z(r, col, zi);
                    values4(v, ri, zi);
                });
        }, fetch_halo);
        if (!live) break;
        const double rr = tot[0], sz = tot[1], sr = tot[3];
        double rzn = tot[2];
        ++k;
        rel = sqrt(rr) / nb;
        if (rel <= tol) {
            done = 1;
            break;
        }
        mz = sz / n;
        rzn -= mz * sr;
        beta = rzn / rz;
        rz = rzn;
        if (k >= maxit) done = 2;
    }
    auto load_x = [&](int r, int c, int i) { a0[i] = val(kCgX, r, c); };
    if (live) // remove the mean of the solution (pressure.cpp:311-316)
        live = phase(1, [&](int c, double* st) { cells(c, st, load_x, [&](int, int, int i, double* v) { *v = a0[i]; }); }, nothing);
    if (live && work) {
        const double mx = tot[0] / n;
        for (int c = 0; c < nch; ++c)
            cells(c, stage, load_x, [&](int r, int col, int i, double*) {
                w.pc[origin + static_cast<std::size_t>(r) * ld + col] = a0[i] - mx;
            });
    }
    if (blockIdx.x == 0 && tid == 0) {
        sc->k = k;
        sc->done = done ? done : 1;
        sc->rel = rel;
    }
}

// Rows per CTA, CTAs and shared memory of k_cg_persist for this grid on `sms` SMs; false where a CTA's rows
// do not fit (from about 1300^2). About 1024 cells per CTA where they do: a barrier over fewer CTAs is
// cheaper than rows spread thin.
bool cg_plan(const DevParams& p, int sms, CgPlan& pl) {
    const long long cells = static_cast<long long>(p.NX) * p.NY;
    pl.sh = p.NY <= 32 ? 5 : p.NY <= 64 ? 6 : 7;
    pl.dld = (p.NY + 2) | 1;
    const int most = std::min(sms, p.NX);
    for (long long ctas = std::max(1LL, std::min<long long>((cells + 1023) / 1024, most));; ctas = std::min<long long>(2 * ctas, most)) {
        pl.R = static_cast<int>((p.NX + ctas - 1) / ctas);
        pl.G = (p.NX + pl.R - 1) / pl.R;
        pl.cw = (4 * pl.R + 31) / 32;
        const long long stage = std::max<long long>(kCgBufs * 4LL * pl.R * ((1 << pl.sh) + 2), 4LL * (p.NX + 1));
        const long long bytes = 8 * (static_cast<long long>(pl.R + 2) * pl.dld + stage);
        if (pl.cw <= 4 && bytes <= kCgSmem) { // four chain warps: a lane per row and plane of 32 rows
            const long long array = 8LL * pl.R * p.NY; // what is left holds the solve's own arrays
            pl.held = static_cast<int>(std::min<long long>(kCgArrays, (kCgSmem - bytes) / array));
            pl.bytes = static_cast<int>(bytes + pl.held * array);
            return true;
        }
        if (ctas == most) return false;
    }
}

} // namespace

void launch_cg_init(const DevParams& p, PressurePtr w, CgPtr cg, CgScalars* sc, double* cells,
                    std::size_t plane, cudaStream_t st) {
    k_cg_init<<<grid_p(p), dim3(BX, BY), 0, st>>>(p, w, cg, sc, cells, plane);
    SGPU_LAUNCH();
}
void launch_cg_scalars(int stage, CgScalars* sc, const double* sums, cudaStream_t st) {
    k_cg_scalars<<<1, 1, 0, st>>>(stage, sc, sums);
    SGPU_LAUNCH();
}
void launch_cg_dinit(const DevParams& p, CgPtr cg, const CgScalars* sc, cudaStream_t st) {
    k_cg_dinit<<<grid_p(p), dim3(BX, BY), 0, st>>>(p, cg, sc);
    SGPU_LAUNCH();
}
void launch_cg_dq(const DevParams& p, PressurePtr w, CgPtr cg, const CgScalars* sc, double* cells,
                  cudaStream_t st) {
    k_cg_dq<<<grid_p(p), dim3(BX, BY), 0, st>>>(p, w, cg, sc, cells);
    SGPU_LAUNCH();
}
void launch_cg_update(const DevParams& p, PressurePtr w, CgPtr cg, const CgScalars* sc,
                      double* cells, std::size_t plane, cudaStream_t st) {
    k_cg_update<<<grid_p(p), dim3(BX, BY), 0, st>>>(p, w, cg, sc, cells, plane);
    SGPU_LAUNCH();
}
void launch_cg_dir(const DevParams& p, CgPtr cg, const CgScalars* sc, cudaStream_t st) {
    k_cg_dir<<<grid_p(p), dim3(BX, BY), 0, st>>>(p, cg, sc);
    SGPU_LAUNCH();
}

bool launch_cg_solve(const DevParams& p, PressurePtr w, CgPtr cg, CgScalars* sc, unsigned long long* sums, unsigned* err,
                     int sms, cudaStream_t st) {
    CgPlan pl{};
    if (!cg_plan(p, sms, pl)) return false;
    static PerDeviceOnce once;
    const int ok = once.get([] { // cooperative launches, one CTA per SM with the most shared memory and threads
        int dev = 0, coop = 0, blocks = 0;
        SGPU_CUDA(cudaGetDevice(&dev));
        SGPU_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop || cudaFuncSetAttribute(k_cg_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, kCgSmem) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_cg_persist, kCgWork + 128, kCgSmem) != cudaSuccess) {
            (void)cudaGetLastError();
            return 0;
        }
        return blocks;
    });
    if (ok < 1) return false;
    const int entries = 12 * p.NX;
    k_cg_empty<<<std::min(148, (entries + 255) / 256), 256, 0, st>>>(sums, entries);
    SGPU_LAUNCH();
    void* args[] = {const_cast<DevParams*>(&p), &w, &cg, &sc, &sums, &err, &pl};
    SGPU_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(&k_cg_persist), dim3(pl.G), dim3(kCgWork + 32 * pl.cw), args,
                                          static_cast<std::size_t>(pl.bytes), st));
    SGPU_LAUNCH();
    return true;
}

} // namespace sgpu
