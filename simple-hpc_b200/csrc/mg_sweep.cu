// mg_sweep.cu — two red-black sweeps of a double level from its symmetric operator, in one streaming pass.
//
// The pass is mg_fast.cu's (a CTA walks a strip of columns top to bottom; the cell of colour c in row I is
// updated by sweep s at step I + 2c + 4s, so the update order of every cell against its neighbours is the
// reference's; halo cells are updated redundantly and the iterate goes to a second buffer), around the same
// three jobs: the descent (sweeps from x or zero, residual, restriction, coarse operator), the ascent
// (prolongation, sweeps) and plain sweeps. What differs is where the operator comes from:
//  * AW(I, J) = AE(I, J - 1), AS(I, J) = AN(I + 1, J) and AP = AE + AW + AN + AS, bit for bit, in the
//    operators of assemble_p (both sides divide the same values) and in those mg_build forms from them. So
//    AE, AN and b are all that is read: 24 B a cell instead of 48.
//  * they come into shared memory once, rows ahead by asynchronous copies, beside x. mg_fast.cu's kernels
//    load the six inputs of each of their two updates and the residual into registers instead, 144 B a cell
//    of L2 traffic and 128 registers, and then wait for each update's division in turn: 3000 cycles a step
//    at 16 warps an SM.
//  * an update's two divisions, and the next sweep's, go through one inverse of AP (quotient() in
//    common.hpp), which a cell's first sweep forms and passes to its second in registers, and a step reads
//    all it needs before it stores (its cells' neighbours lie on rows and columns that no thread updates in
//    the same step), so the two sweeps' chains overlap.
// Measured, the streamed levels of a V(2,2) cycle at 4096^2: descent 670 -> 460 us, ascent 540 -> 395 us; 8 sweeps
// of the red-black solver at 1531 x 2047: 470 us (16 launches, a colour each) -> 192 us. It is now bound by
// issue slots and shared-memory wavefronts (60% of each; DRAM 25%).
#include "kernels.hpp"

#include <algorithm>

namespace sgpu {

namespace {

constexpr int kNT = 128;        // threads: loaded columns of a strip
constexpr int kRing = 16;       // rows of the x ring
constexpr int kHalo = 6;        // of a strip: one cell per colour pass, one for the residual, kept even
constexpr int kLag = 8;         // rows between a step and the row whose two sweeps it completes

enum Job { kDown, kUp, kPlain };
// Rows of the rings of AE, AN and b: without a residual they are last read two rows behind the step. With
// them at 8 rows four CTAs fit an SM (41 KB each), otherwise three (65 KB).
__host__ __device__ constexpr int coef_ring(Job j) { return j == kDown ? 16 : 8; }
__host__ __device__ constexpr int ctas(Job j) { return j == kDown ? 3 : 4; }
// and a pad: the first column's west neighbour
__host__ __device__ constexpr int smem_bytes(Job j) { return ((kRing + 3 * coef_ring(j)) * kNT + 2) * 8; }

__device__ __forceinline__ void cp_async(double* smem, const double* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// What a cell's first sweep leaves for its second, four steps later.
struct Swept {
    double e, w, n, s, ap, y, t0;
};

// parity: 0 where the first colour is the cells with I + J even, 1 where it is the others.
template <Job JOB>
__global__ void __launch_bounds__(kNT, ctas(JOB))
    k_level_sweeps(LevelView L, LevelView C, const double* __restrict__ xin, double* __restrict__ xout,
                   double omega, int x_zero, int parity, int seg_rows, int build) {
    // Rows copied beyond the ones a step reads: a step refills the slot of a row last read before it.
    constexpr int LA = JOB == kUp ? 2 : 1, RC = coef_ring(JOB), PF = JOB == kDown ? 4 : JOB == kUp ? 2 : 3;
    extern __shared__ __align__(16) double sm[];
    double* const X = sm + 2;
    double* const AE = X + kRing * kNT;
    double* const AN = AE + RC * kNT;
    double* const B = AN + RC * kNT;
    const int tid = threadIdx.x, nx = L.nx, ny = L.ny, ls = L.stride;
    constexpr int W = kNT - 2 * kHalo;
    const int R0 = blockIdx.y * seg_rows, R1 = min(R0 + seg_rows, nx);            // owned rows
    const int L0 = max(R0 - kHalo, -1), L1 = min(R1 + kHalo, nx + 1);             // loaded rows [L0, L1)
    const int J0 = blockIdx.x * W, C0 = J0 - kHalo, Jc = C0 + tid;                // owned, loaded, own column
    const bool cload = Jc >= -1 && Jc <= ny, cint = Jc >= 0 && Jc < ny;
    const bool cown = cint && Jc >= J0 && Jc < J0 + W;
    // Pass k (colour k & 1 of sweep k / 2; 4: the residual) is computable k + 1 cells inside a cut edge.
    const bool cut_top = L0 > -1, cut_bot = L1 < nx + 1, cut_left = C0 > -1, cut_right = C0 + kNT < ny + 1;
    unsigned cols = 0;
    for (int k = 0; k <= 4; ++k)
        if (cint && (!cut_left || tid >= 1 + k) && (!cut_right || tid <= kNT - 2 - k)) cols |= 1u << k;
    const int lo = cut_top ? L0 + 1 : 0, hi = cut_bot ? L1 - 2 : nx - 1;
    auto ok = [&](int I, int k) {
        return ((cols >> k) & 1u) && I >= lo + (cut_top ? k : 0) && I <= hi - (cut_bot ? k : 0);
    };
    auto at = [&](int I) { return (I & (kRing - 1)) * kNT + tid; };
    auto cat = [&](int I) { return (I & (RC - 1)) * kNT + tid; };

    int next = L0;
    auto issue = [&]() {
        if (next < L1 && cload) {
            const int q = at(next), k = cat(next);
            const bool in = cint && next >= 0 && next < nx;
            const long long c = static_cast<long long>(next) * ls + Jc;
            if (x_zero || (JOB == kPlain && !in)) X[q] = 0.0;
            else cp_async(X + q, xin + c);
            if (in) {
                cp_async(AE + k, L.AE + c);
                cp_async(AN + k, L.AN + c);
                cp_async(B + k, L.b + c);
            } else { // the west and south links of the cells along the walls
                AE[k] = 0.0;
                AN[k] = 0.0;
            }
        }
        cp_async_commit();
        ++next;
    };
    for (int k = 0; k < LA + 1 + PF; ++k) issue();

    const int t0 = JOB == kUp ? L0 - 2 : L0;
    Swept Q[4];
    double cx[4]; // kUp: the coarse correction of row t + 2 for the steps ahead
    auto coarse_at = [&](int I) {
        return cint && I >= 0 && I < nx && I < L1 ? __ldg(C.x + static_cast<long long>(I >> 1) * C.stride + (Jc >> 1)) : 0.0;
    };
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        Q[d] = {0.0, 0.0, 0.0, 0.0, 1.0, 1.0, 0.0};
        if (JOB == kUp) cx[d] = coarse_at(t0 + d + 2);
    }
    double r_prev = 0.0, lp_e = 0.0, lp_w = 0.0, lp_n = 0.0; // kDown: of the residual row before

    auto step = [&](int t, Swept& sw, double& cxt) {
        if (JOB == kUp && t < L0) cp_async_wait<PF + 1>();
        else cp_async_wait<PF>(); // rows <= t + LA have landed
        __syncthreads();
        if (JOB != kUp || t >= L0) issue();
        if (JOB == kUp) { // prolongation of row t + 2 (read first at step t + 1)
            const int I = t + 2;
            if (cint && I >= 0 && I < nx && I < L1) X[at(I)] += omega * cxt;
        }
        const int c = (t + Jc + parity) & 1;
        const int I0 = t - 2 * c, I1 = I0 - 4;
        const bool ok0 = ok(I0, c), ok1 = ok(I1, 2 + c);
        const int q0 = at(I0), q0n = at(I0 - 1), q0s = at(I0 + 1);
        const int q1 = at(I1), q1n = at(I1 - 1), q1s = at(I1 + 1);
        Swept z;
        const int k0 = cat(I0);
        z.e = AE[k0];
        z.w = AE[k0 - 1];
        z.n = AN[k0];
        z.s = AN[cat(I0 + 1)];
        const double b0 = B[k0];
        const double nb0 = z.e * X[q0 + 1] + z.w * X[q0 - 1] + z.s * X[q0s] + z.n * X[q0n];
        const double nb1 = sw.e * X[q1 + 1] + sw.w * X[q1 - 1] + sw.s * X[q1s] + sw.n * X[q1n];
        z.ap = ok0 ? z.e + z.w + z.n + z.s : 1.0;
        z.y = inverse(z.ap);
        bool slow0 = false, slow1 = false;
        z.t0 = quotient_try(b0, z.ap, z.y, slow0);
        double v0 = quotient_try(nb0, z.ap, z.y, slow0), v1 = quotient_try(nb1, sw.ap, sw.y, slow1);
        if ((ok0 && slow0) || (ok1 && slow1)) {
            z.t0 = divided(b0, z.ap);
            v0 = divided(nb0, z.ap);
            v1 = divided(nb1, sw.ap);
        }
        if (ok0) X[q0] = z.t0 + v0;
        if (ok1) X[q1] = sw.t0 + v1;
        sw = z;
        if (JOB == kDown) {
            // Residual of row Ir (multigrid.cpp:84-85); its neighbours' updates are earlier steps'.
            const int Ir = t - kLag, q = at(Ir), qn = at(Ir - 1), qs = at(Ir + 1);
            double r = 0.0, e = 0.0, w = 0.0, n = 0.0, s = 0.0;
            if (ok(Ir, 4)) {
                e = AE[q];
                w = AE[q - 1];
                n = AN[q];
                s = AN[qs];
                r = B[q] - ((e + w + n + s) * X[q] - (e * X[q + 1] + w * X[q - 1] + s * X[qs] + n * X[qn]));
            }
            // Restriction of the rows Ir - 1 and Ir, C.b = r[f] + r[f+1] + r[f+fs] + r[f+fs+1], and with
            // build the coarse cell's links as mg_build adds them (the odd column from the next lane).
            if ((Ir & 1) && Ir >= 1) { // uniform over the CTA
                const double rp_odd = __shfl_down_sync(0xffffffffu, r_prev, 1), r_odd = __shfl_down_sync(0xffffffffu, r, 1);
                double ep_odd = 0.0, e_odd = 0.0, np_odd = 0.0, s_odd = 0.0;
                if (build) {
                    ep_odd = __shfl_down_sync(0xffffffffu, lp_e, 1);
                    e_odd = __shfl_down_sync(0xffffffffu, e, 1);
                    np_odd = __shfl_down_sync(0xffffffffu, lp_n, 1);
                    s_odd = __shfl_down_sync(0xffffffffu, s, 1);
                }
                const int Rc = Ir >> 1;
                if (cown && !(Jc & 1) && Ir - 1 >= R0 && Ir < R1 && Rc < C.nx) {
                    const int cq = Rc * C.stride + (Jc >> 1);
                    C.b[cq] = r_prev + rp_odd + r + r_odd;
                    C.x[cq] = 0.0;
                    if (build) {
                        const double ae = ep_odd + e_odd, aw = lp_w + w, an = lp_n + np_odd, as = s + s_odd;
                        set_links(C, cq, ae, aw, an, as);
                        C.AP[cq] = ae + aw + an + as;
                    }
                }
            }
            r_prev = r;
            lp_e = e;
            lp_w = w;
            lp_n = n;
        }
        const int rw = t - kLag + 1; // had its last update at step t - 1
        if (cown && rw >= R0 && rw < R1) xout[static_cast<long long>(rw) * ls + Jc] = X[at(rw)];
        if (JOB == kUp) cxt = coarse_at(t + 4 + 2);
    };
    const int t_last = R1 - 1 + kLag;
    for (int t = t0; t <= t_last; t += 4) {
#pragma unroll
        for (int d = 0; d < 4; ++d)
            if (t + d <= t_last) step(t + d, Q[d], cx[d]);
    }
    cp_async_wait<0>();
}

// Rows per CTA: one wave of resident CTAs, at least min_seg rows (min_seg <= 0: enough that the halo and
// skew rows a CTA walks are about half of its steps), even so that restriction pairs stay in one CTA.
template <Job JOB>
void launch(const LevelView& L, const LevelView& C, const double* xin, double* xout, double omega, bool x_zero,
            int parity, bool build, int sms, int min_seg, cudaStream_t st) {
    auto kernel = k_level_sweeps<JOB>;
    static PerDeviceOnce once;
    const int blocks = once.get([&] {
        SGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(JOB)));
        int n = 0;
        SGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kNT, smem_bytes(JOB)));
        return n < 1 ? 1 : n;
    });
    constexpr int W = kNT - 2 * kHalo;
    const int strips = (L.ny + W - 1) / W, want = std::max(1, blocks * sms / strips);
    int seg = ((L.nx + want - 1) / want + 1) & ~1;
    seg = std::max(seg, min_seg > 0 ? std::max(2, min_seg & ~1) : 2 * kHalo + 8);
    kernel<<<dim3(strips, (L.nx + seg - 1) / seg), kNT, smem_bytes(JOB), st>>>(L, C, xin, xout, omega, x_zero ? 1 : 0, parity, seg,
                                                                   build ? 1 : 0);
    SGPU_LAUNCH();
}

} // namespace

void launch_sweeps_down(const LevelView& F, const LevelView& C, double* xout, bool x_zero, int sms, int min_seg,
                        cudaStream_t st, bool build) {
    launch<kDown>(F, C, F.x, xout, 0.0, x_zero, 0, build, sms, min_seg, st);
}
void launch_sweeps_up(const LevelView& C, const LevelView& F, const double* xin, double* xout, double omega, int sms,
                      int min_seg, cudaStream_t st) {
    launch<kUp>(F, C, xin, xout, omega, false, 0, false, sms, min_seg, st);
}
void launch_sweeps_plain(const LevelView& L, const double* xin, double* xout, bool x_zero, int parity, int sms,
                         int min_seg, cudaStream_t st) {
    launch<kPlain>(L, L, xin, xout, 0.0, x_zero, parity, false, sms, min_seg, st);
}

} // namespace sgpu
