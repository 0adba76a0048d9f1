// mg_sweep.cu — two red-black sweeps of a level in one streaming pass, its operator through shared memory.
//
// The pass is mg_fast.cu's (a CTA walks a strip of columns top to bottom; the cell of colour c in row I is
// updated by sweep s at step I + 2c + 4s, so the update order of every cell against its neighbours is the
// reference's; halo cells are updated redundantly and the iterate goes to a second buffer), around the same
// three jobs: the descent (sweeps from x or zero, residual, restriction, coarse operator), the ascent
// (prolongation, sweeps) and, in double, plain sweeps. What differs is where the operator comes from:
//  * each row's comes into shared memory once, rows ahead by asynchronous copies, beside x. mg_fast.cu's kernels
//    load the six inputs of each of their two updates and of the residual into registers instead, from L2
//    each time, and in double then wait for each update's division in turn: 3000 cycles a step at 16 warps
//    an SM.
//  * in double it is AE and AN alone: AW(I, J) = AE(I, J - 1), AS(I, J) = AN(I + 1, J) and AP = AE + AW + AN + AS,
//    bit for bit, in the operators of assemble_p (both sides divide the same values) and in those mg_build
//    forms from them. 24 B a cell with b instead of 48. (In float the links are one 16-byte record, and AP
//    is rounded from the double one.)
//  * a cell's second sweep takes links and AP from its first in registers; in double the first forms an inverse
//    of AP there and every division goes through it (quotient() in common.hpp). A step reads all it needs
//    before it stores (its cells' neighbours lie on rows and columns that no thread updates in the same
//    step), so the two sweeps' chains overlap.
// Measured, the streamed levels of a V(2,2) cycle at 4096^2: double, descent 670 -> 448 us and ascent 540 ->
// 381 us; float, 309 -> 260 and 263 -> 219 us; float at 1024^2, 51 -> 31 and 47 -> 36 us. 8 sweeps of the
// red-black solver at 1531 x 2047: 470 us (16 launches, a colour each) -> 184 us. The passes are bound by issue
// slots (float: 3.0 instructions a cycle; double: 2.4, and 60% of the shared-memory wavefronts; DRAM 25%).
#include "kernels.hpp"

#include <algorithm>

namespace sgpu {

namespace {

constexpr int kNT = 128;        // threads: loaded columns of a strip (a power of two: ring elements wrap by a mask)
constexpr int kRing = 16;       // rows of the x ring
constexpr int kHalo = 6;        // of a strip: one cell per colour pass, one for the residual, kept even
constexpr int kLag = 8;         // rows between a step and the row whose two sweeps it completes

enum Job { kDown, kUp, kPlain };
// Rows of the rings of the operator and b: without a residual they are last read two rows behind the step. In
// double three blocks fit an SM with 16 rows (65 KB each) and four with 8 (41 KB; the registers' bound), in
// float three (57 KB) and six (33 KB).
template <class T, Job JOB> struct Shape {
    static constexpr int coef_rows = JOB == kDown ? 16 : 8;
    static constexpr int ctas = JOB == kDown ? 3 : sizeof(T) == 8 ? 4 : 6;
    // per cell: AE, AN and b, or the four links, AP and b; 16 bytes before x: the first column's west neighbour
    static constexpr int smem = 16 + (kRing * static_cast<int>(sizeof(T)) + coef_rows * 24) * kNT;
};

template <class V> __device__ __forceinline__ void cp_async(V* smem, const V* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    if constexpr (sizeof(V) == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(sizeof(V)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// What a cell's first sweep leaves for its second, four steps later (float: y unused, t0 is b).
template <class T> struct Swept {
    T e, w, n, s, ap, y, t0;
};

// The operator and b of the rows at hand: the links, AP and b of the cell at ring index k (own row) of which
// ks is the index one row down.
template <class T, int RC> struct Operator;
template <int RC> struct Operator<double, RC> {
    double *AE, *AN, *B;
    __device__ explicit Operator(double* p) : AE(p), AN(p + RC * kNT), B(p + 2 * RC * kNT) {}
    __device__ __forceinline__ void fetch(const LevelView& L, int k, int c, bool in) const {
        if (in) {
            cp_async(AE + k, L.AE + c);
            cp_async(AN + k, L.AN + c);
            cp_async(B + k, L.b + c);
        } else { // the west and south links of the cells along the walls
            AE[k] = 0.0;
            AN[k] = 0.0;
        }
    }
    __device__ __forceinline__ void links(int k, int ks, double& e, double& w, double& n, double& s) const {
        e = AE[k];
        w = AE[k - 1];
        n = AN[k];
        s = AN[ks];
    }
    __device__ __forceinline__ double ap(int, double e, double w, double n, double s) const { return e + w + n + s; }
};
template <int RC> struct Operator<float, RC> {
    float4* K;
    float *P, *B;
    __device__ explicit Operator(float* p) : K(reinterpret_cast<float4*>(p)), P(p + 4 * RC * kNT), B(p + 5 * RC * kNT) {}
    __device__ __forceinline__ void fetch(const LevelView32& L, int k, int c, bool in) const {
        if (!in) return;
        cp_async(K + k, reinterpret_cast<const float4*>(L.L4) + c);
        cp_async(P + k, static_cast<const float*>(L.AP) + c);
        cp_async(B + k, static_cast<const float*>(L.b) + c);
    }
    __device__ __forceinline__ void links(int k, int, float& e, float& w, float& n, float& s) const {
        const float4 v = K[k];
        e = v.x;
        w = v.y;
        n = v.z;
        s = v.w;
    }
    __device__ __forceinline__ float ap(int k, float, float, float, float) const { return P[k]; }
};

// The updates of a step's two cells (multigrid.cpp:61-63) from their neighbour sums: of z, in its first sweep, whose
// b is given, and of sw, in its second.
template <class T>
__device__ __forceinline__ void update(bool ok0, bool ok1, T b0, T nb0, T nb1, Swept<T>& z, const Swept<T>& sw, T& v0, T& v1) {
    if constexpr (sizeof(T) == 8) {
        if (!ok0) z.ap = 1.0; // not a cell of this pass: nothing that would take the division's long path
        z.y = inverse(z.ap);
        bool slow0 = false, slow1 = false;
        z.t0 = quotient_try(b0, z.ap, z.y, slow0);
        v0 = quotient_try(nb0, z.ap, z.y, slow0);
        v1 = quotient_try(nb1, sw.ap, sw.y, slow1);
        if ((ok0 && slow0) || (ok1 && slow1)) {
            z.t0 = quotient_rare(b0, z.ap, z.y);
            v0 = quotient_rare(nb0, z.ap, z.y);
            v1 = quotient_rare(nb1, sw.ap, sw.y);
        }
        v0 = z.t0 + v0;
        v1 = sw.t0 + v1;
    } else {
        z.t0 = b0;
        v0 = rb_value(b0, nb0, z.ap);
        v1 = rb_value(sw.t0, nb1, sw.ap);
    }
}

// parity: 0 where the first colour is the cells with I + J even, 1 where it is the others.
template <class T, Job JOB>
__global__ void __launch_bounds__(kNT, (Shape<T, JOB>::ctas))
    k_level_sweeps(LevelViewT<T> L, LevelViewT<T> C, const T* __restrict__ xin, T* __restrict__ xout,
                   double omega, int x_zero, int parity, int seg_rows, int build) {
    // Rows copied beyond the ones a step reads: a step refills the slot of a row last read before it.
    constexpr int LA = JOB == kUp ? 2 : 1, RC = Shape<T, JOB>::coef_rows, PF = JOB == kDown ? 4 : JOB == kUp ? 2 : 3;
    extern __shared__ __align__(16) unsigned char sweep_sm[];
    T* const X = reinterpret_cast<T*>(sweep_sm + 16);
    const Operator<T, RC> A(X + kRing * kNT);
    const T om = static_cast<T>(omega);
    const int tid = threadIdx.x, nx = L.nx, ny = L.ny, ls = L.stride;
    constexpr int W = kNT - 2 * kHalo;
    const int R0 = blockIdx.y * seg_rows, R1 = min(R0 + seg_rows, nx);            // owned rows
    const int L0 = max(R0 - kHalo, -1), L1 = min(R1 + kHalo, nx + 1);             // loaded rows [L0, L1)
    const int J0 = blockIdx.x * W, C0 = J0 - kHalo, Jc = C0 + tid;                // owned, loaded, own column
    const bool cload = Jc >= -1 && Jc <= ny, cint = Jc >= 0 && Jc < ny;
    const bool cown = cint && Jc >= J0 && Jc < J0 + W;
    // Pass k (colour k & 1 of sweep k / 2; 4: the residual) is computable k + 1 cells inside a cut edge: the
    // thread's steps for it are the span's, of a column where it never is none. All of a step's tests are one
    // subtraction and one unsigned comparison, and what differs between a thread's two colours is formed here,
    // since the instructions of a step are what bounds the pass.
    const bool cut_top = L0 > -1, cut_bot = L1 < nx + 1, cut_left = C0 > -1, cut_right = C0 + kNT < ny + 1;
    const int lo = cut_top ? L0 + 1 : 0, hi = cut_bot ? L1 - 2 : nx - 1;
    struct Span {
        int first;
        unsigned len;
        __device__ __forceinline__ bool has(int t) const { return static_cast<unsigned>(t - first) < len; }
    };
    auto span = [&](int k, int lag) { // the cell of step t is in row t - lag
        const bool col = cint && (!cut_left || tid >= 1 + k) && (!cut_right || tid <= kNT - 2 - k);
        const int a = lo + (cut_top ? k : 0), n = hi - (cut_bot ? k : 0) + 1 - a;
        return Span{a + lag, col && n > 0 ? static_cast<unsigned>(n) : 0u};
    };
    auto rows = [&](bool col, int a, int b, int lag) { return Span{a + lag, col && b > a ? static_cast<unsigned>(b - a) : 0u}; };
    auto wrap = [&](int e) { return e & (kRing * kNT - 1); };  // ring element of row I, column J: wrap(I * kNT + J)
    auto cwrap = [&](int e) { return e & (RC * kNT - 1); };

    const Span loaded = rows(cload, L0, L1, 0), inside = rows(cint, 0, nx, 0);
    int next = L0, c = L0 * ls + Jc; // the row to copy next, and its element of the level's arrays
    auto issue = [&]() {
        if (loaded.has(next)) {
            const int e = next * kNT + tid;
            const bool in = inside.has(next);
            if (x_zero || (JOB == kPlain && !in)) X[wrap(e)] = T(0);
            else cp_async(X + wrap(e), xin + c);
            A.fetch(L, cwrap(e), c, in);
        }
        cp_async_commit();
        ++next;
        c += ls;
    };
    for (int k = 0; k < LA + 1 + PF; ++k) issue();

    const int t0 = JOB == kUp ? L0 - 2 : L0;
    Swept<T> Q[4];
    T cx[4]; // kUp: the coarse correction of row t + 2 for the steps ahead
    const Span raised = rows(cint, 0, min(nx, L1), -2); // rows t + 2
    auto coarse_at = [&](int t) {
        return raised.has(t) ? __ldg(C.x + ((t + 2) >> 1) * C.stride + (Jc >> 1)) : T(0);
    };
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        Q[d] = {T(0), T(0), T(0), T(0), T(1), T(1), T(0)};
        if (JOB == kUp) cx[d] = coarse_at(t0 + d);
    }
    T r_prev = T(0), lp_e = T(0), lp_w = T(0), lp_n = T(0); // kDown: of the residual row before

    // of the steps t0, t0 + 2, ..: colour col[0]; of the others: the other
    const int col[2] = {(t0 + Jc + parity) & 1, (t0 + 1 + Jc + parity) & 1};
    Span sp[2][2]; // first and second sweep
    int ofs[2];    // ring element of the first sweep's cell, less t * kNT
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        sp[k][0] = span(col[k], 2 * col[k]);
        sp[k][1] = span(2 + col[k], 2 * col[k] + 4);
        ofs[k] = tid - 2 * col[k] * kNT;
    }
    const Span sp_res = span(4, kLag), sp_out = rows(cown, R0, R1, kLag - 1);

    auto step = [&](int t, int d, Swept<T>& sw, T& cxt) {
        if (JOB == kUp && t < L0) cp_async_wait<PF + 1>();
        else cp_async_wait<PF>(); // rows <= t + LA have landed
        __syncthreads();
        if (JOB != kUp || t >= L0) issue();
        if (JOB == kUp) { // prolongation of row t + 2 (read first at step t + 1)
            if (raised.has(t)) X[wrap((t + 2) * kNT + tid)] += om * cxt;
        }
        const bool ok0 = sp[d & 1][0].has(t), ok1 = sp[d & 1][1].has(t);
        const int e = t * kNT + ofs[d & 1];
        const int q0 = wrap(e), q0n = wrap(e - kNT), q0s = wrap(e + kNT);
        const int q1 = wrap(e - 4 * kNT), q1n = wrap(e - 5 * kNT), q1s = wrap(e - 3 * kNT);
        Swept<T> z;
        const int k0 = cwrap(e);
        A.links(k0, cwrap(e + kNT), z.e, z.w, z.n, z.s);
        z.ap = A.ap(k0, z.e, z.w, z.n, z.s);
        const T nb0 = z.e * X[q0 + 1] + z.w * X[q0 - 1] + z.s * X[q0s] + z.n * X[q0n];
        const T nb1 = sw.e * X[q1 + 1] + sw.w * X[q1 - 1] + sw.s * X[q1s] + sw.n * X[q1n];
        T v0, v1;
        update(ok0, ok1, A.B[k0], nb0, nb1, z, sw, v0, v1);
        if (ok0) X[q0] = v0;
        if (ok1) X[q1] = v1;
        sw = z;
        if (JOB == kDown) {
            // Residual of row Ir (multigrid.cpp:84-85); its neighbours' updates are earlier steps'.
            const int Ir = t - kLag, er = Ir * kNT + tid, q = wrap(er), qn = wrap(er - kNT), qs = wrap(er + kNT);
            T r = T(0), ke = T(0), kw = T(0), kn = T(0), ks = T(0);
            if (sp_res.has(t)) {
                A.links(q, qs, ke, kw, kn, ks); // the rings are of the same height here
                const T ap = A.ap(q, ke, kw, kn, ks);
                r = A.B[q] - (ap * X[q] - (ke * X[q + 1] + kw * X[q - 1] + ks * X[qs] + kn * X[qn]));
            }
            // Restriction of the rows Ir - 1 and Ir, C.b = r[f] + r[f+1] + r[f+fs] + r[f+fs+1], and with
            // build the coarse cell's links as mg_build adds them (the odd column from the next lane).
            if ((Ir & 1) && Ir >= 1) { // uniform over the CTA
                const T rp_odd = __shfl_down_sync(0xffffffffu, r_prev, 1), r_odd = __shfl_down_sync(0xffffffffu, r, 1);
                T ep_odd = T(0), e_odd = T(0), np_odd = T(0), s_odd = T(0);
                if (build) {
                    ep_odd = __shfl_down_sync(0xffffffffu, lp_e, 1);
                    e_odd = __shfl_down_sync(0xffffffffu, ke, 1);
                    np_odd = __shfl_down_sync(0xffffffffu, lp_n, 1);
                    s_odd = __shfl_down_sync(0xffffffffu, ks, 1);
                }
                const int Rc = Ir >> 1;
                if (cown && !(Jc & 1) && Ir - 1 >= R0 && Ir < R1 && Rc < C.nx) {
                    const int cq = Rc * C.stride + (Jc >> 1);
                    C.b[cq] = r_prev + rp_odd + r + r_odd;
                    C.x[cq] = T(0);
                    if (build) {
                        const T ae = ep_odd + e_odd, aw = lp_w + kw, an = lp_n + np_odd, as = ks + s_odd;
                        set_links(C, cq, ae, aw, an, as);
                        C.AP[cq] = ae + aw + an + as;
                    }
                }
            }
            r_prev = r;
            lp_e = ke;
            lp_w = kw;
            lp_n = kn;
        }
        // row t - kLag + 1 had its last update at step t - 1
        if (sp_out.has(t)) xout[(t - kLag + 1) * ls + Jc] = X[wrap((t - kLag + 1) * kNT + tid)];
        if (JOB == kUp) cxt = coarse_at(t + 4);
    };
    const int t_last = R1 - 1 + kLag;
    for (int t = t0; t <= t_last; t += 4) {
#pragma unroll
        for (int d = 0; d < 4; ++d)
            if (t + d <= t_last) step(t + d, d, Q[d], cx[d]);
    }
    cp_async_wait<0>();
}

// Rows per CTA: one wave of resident CTAs, at least min_seg rows (min_seg <= 0: enough that the halo and
// skew rows a CTA walks are about half of its steps), even so that restriction pairs stay in one CTA.
template <class T, Job JOB>
void launch(const LevelViewT<T>& L, const LevelViewT<T>& C, const T* xin, T* xout, double omega, bool x_zero,
            int parity, bool build, int sms, int min_seg, cudaStream_t st) {
    auto kernel = k_level_sweeps<T, JOB>;
    constexpr int smem = Shape<T, JOB>::smem;
    static PerDeviceOnce once;
    const int blocks = once.get([&] {
        SGPU_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        int n = 0;
        SGPU_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kNT, smem));
        return n < 1 ? 1 : n;
    });
    constexpr int W = kNT - 2 * kHalo;
    const int strips = (L.ny + W - 1) / W, want = std::max(1, blocks * sms / strips);
    int seg = ((L.nx + want - 1) / want + 1) & ~1;
    seg = std::max(seg, min_seg > 0 ? std::max(2, min_seg & ~1) : 2 * kHalo + 8);
    kernel<<<dim3(strips, (L.nx + seg - 1) / seg), kNT, smem, st>>>(L, C, xin, xout, omega, x_zero ? 1 : 0, parity, seg,
                                                                   build ? 1 : 0);
    SGPU_LAUNCH();
}

} // namespace

template <class T>
void launch_sweeps_down(const LevelViewT<T>& F, const LevelViewT<T>& C, T* xout, bool x_zero, int sms, int min_seg,
                        cudaStream_t st, bool build) {
    launch<T, kDown>(F, C, F.x, xout, 0.0, x_zero, 0, build, sms, min_seg, st);
}
template <class T>
void launch_sweeps_up(const LevelViewT<T>& C, const LevelViewT<T>& F, const T* xin, T* xout, double omega, int sms,
                      int min_seg, cudaStream_t st) {
    launch<T, kUp>(F, C, xin, xout, omega, false, 0, false, sms, min_seg, st);
}
// This file alone instantiates the double kernels (built without contraction: the reference's bits);
// mg_sweep32.cu includes it with SGPU_FLOAT_UNIT for the float ones (contraction allowed).
#ifndef SGPU_FLOAT_UNIT
template void launch_sweeps_down<double>(const LevelView&, const LevelView&, double*, bool, int, int, cudaStream_t, bool);
template void launch_sweeps_up<double>(const LevelView&, const LevelView&, const double*, double*, double, int, int,
                                       cudaStream_t);
void launch_sweeps_plain(const LevelView& L, const double* xin, double* xout, bool x_zero, int parity, int sms,
                         int min_seg, cudaStream_t st) {
    launch<double, kPlain>(L, L, xin, xout, 0.0, x_zero, parity, false, sms, min_seg, st);
}
#else
template void launch_sweeps_down<float>(const LevelView32&, const LevelView32&, float*, bool, int, int, cudaStream_t, bool);
template void launch_sweeps_up<float>(const LevelView32&, const LevelView32&, const float*, float*, double, int, int,
                                      cudaStream_t);
#endif

} // namespace sgpu
