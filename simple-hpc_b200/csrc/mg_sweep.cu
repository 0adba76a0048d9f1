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
// Measured, the streamed levels of a V(2,2) cycle at 4096^2: double, descent 670 -> 460 us and ascent 540 ->
// 395 us; float, 309 -> 262 and 263 -> 244 us; float at 1024^2, 51 -> 32 and 47 -> 38 us. 8 sweeps of the
// red-black solver at 1531 x 2047: 470 us (16 launches, a colour each) -> 192 us. The double passes are bound
// by issue slots and shared-memory wavefronts (60% of each; DRAM 25%).
#include "kernels.hpp"

#include <algorithm>

namespace sgpu {

namespace {

constexpr int kNT = 128;        // threads: loaded columns of a strip
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
    __device__ __forceinline__ void fetch(const LevelView& L, int k, long long c, bool in) const {
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
    __device__ __forceinline__ void fetch(const LevelView32& L, int k, long long c, bool in) const {
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
__device__ __forceinline__ void update(bool ok0, bool ok1, double b0, double nb0, double nb1, Swept<double>& z,
                                       const Swept<double>& sw, double& v0, double& v1) {
    if (!ok0) z.ap = 1.0; // not a cell of this pass: nothing that would take the division's long path
    z.y = inverse(z.ap);
    bool slow0 = false, slow1 = false;
    z.t0 = quotient_try(b0, z.ap, z.y, slow0);
    v0 = quotient_try(nb0, z.ap, z.y, slow0);
    v1 = quotient_try(nb1, sw.ap, sw.y, slow1);
    if ((ok0 && slow0) || (ok1 && slow1)) {
        z.t0 = divided(b0, z.ap);
        v0 = divided(nb0, z.ap);
        v1 = divided(nb1, sw.ap);
    }
    v0 = z.t0 + v0;
    v1 = sw.t0 + v1;
}
__device__ __forceinline__ void update(bool, bool, float b0, float nb0, float nb1, Swept<float>& z, const Swept<float>& sw,
                                       float& v0, float& v1) {
    z.t0 = b0;
    v0 = rb_value(b0, nb0, z.ap);
    v1 = rb_value(sw.t0, nb1, sw.ap);
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
            if (x_zero || (JOB == kPlain && !in)) X[q] = T(0);
            else cp_async(X + q, xin + c);
            A.fetch(L, k, c, in);
        }
        cp_async_commit();
        ++next;
    };
    for (int k = 0; k < LA + 1 + PF; ++k) issue();

    const int t0 = JOB == kUp ? L0 - 2 : L0;
    Swept<T> Q[4];
    T cx[4]; // kUp: the coarse correction of row t + 2 for the steps ahead
    auto coarse_at = [&](int I) {
        return cint && I >= 0 && I < nx && I < L1 ? __ldg(C.x + static_cast<long long>(I >> 1) * C.stride + (Jc >> 1)) : T(0);
    };
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        Q[d] = {T(0), T(0), T(0), T(0), T(1), T(1), T(0)};
        if (JOB == kUp) cx[d] = coarse_at(t0 + d + 2);
    }
    T r_prev = T(0), lp_e = T(0), lp_w = T(0), lp_n = T(0); // kDown: of the residual row before

    auto step = [&](int t, Swept<T>& sw, T& cxt) {
        if (JOB == kUp && t < L0) cp_async_wait<PF + 1>();
        else cp_async_wait<PF>(); // rows <= t + LA have landed
        __syncthreads();
        if (JOB != kUp || t >= L0) issue();
        if (JOB == kUp) { // prolongation of row t + 2 (read first at step t + 1)
            const int I = t + 2;
            if (cint && I >= 0 && I < nx && I < L1) X[at(I)] += om * cxt;
        }
        const int c = (t + Jc + parity) & 1;
        const int I0 = t - 2 * c, I1 = I0 - 4;
        const bool ok0 = ok(I0, c), ok1 = ok(I1, 2 + c);
        const int q0 = at(I0), q0n = at(I0 - 1), q0s = at(I0 + 1);
        const int q1 = at(I1), q1n = at(I1 - 1), q1s = at(I1 + 1);
        Swept<T> z;
        const int k0 = cat(I0);
        A.links(k0, cat(I0 + 1), z.e, z.w, z.n, z.s);
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
            const int Ir = t - kLag, q = at(Ir), qn = at(Ir - 1), qs = at(Ir + 1);
            T r = T(0), e = T(0), w = T(0), n = T(0), s = T(0);
            if (ok(Ir, 4)) {
                A.links(q, qs, e, w, n, s); // the rings are of the same height here
                const T ap = A.ap(q, e, w, n, s);
                r = A.B[q] - (ap * X[q] - (e * X[q + 1] + w * X[q - 1] + s * X[qs] + n * X[qn]));
            }
            // Restriction of the rows Ir - 1 and Ir, C.b = r[f] + r[f+1] + r[f+fs] + r[f+fs+1], and with
            // build the coarse cell's links as mg_build adds them (the odd column from the next lane).
            if ((Ir & 1) && Ir >= 1) { // uniform over the CTA
                const T rp_odd = __shfl_down_sync(0xffffffffu, r_prev, 1), r_odd = __shfl_down_sync(0xffffffffu, r, 1);
                T ep_odd = T(0), e_odd = T(0), np_odd = T(0), s_odd = T(0);
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
                    C.x[cq] = T(0);
                    if (build) {
                        const T ae = ep_odd + e_odd, aw = lp_w + w, an = lp_n + np_odd, as = s + s_odd;
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
