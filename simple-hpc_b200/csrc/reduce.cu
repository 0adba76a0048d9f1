// reduce.cu — ordered (bit-reproducible) sums on the device.
//
// The reference sums a per-cell quantity by adding each row left to right from 0.0 and then the
// row sums top to bottom from 0.0 (CellSums::sum and add_rows, src/decomp.cpp:176-205; det_sum,
// src/multigrid.cpp:18-34). Floating-point addition is not associative, so the same bits need the
// same chain: one dependent chain per row, then one chain over the rows.
//
// A CTA owns kRows rows. Its four warps copy tiles of kRows x kCols values into a ring in shared memory,
// several tiles ahead, and one of them adds them, a lane per row (for two sums of a row, two do). The adds
// are the floor, 8 cycles each, nc of them and then nr over the rows by the last CTA to finish; few rows
// per CTA spread the memory stream over the SMs and long tile rows leave a barrier per 128 adds. Measured:
// one sum 16.6 us at 1024^2 and 71 us at 4096^2, a pair 17.5 and 89, against 27.8 and 100, 28.8 and 106 with
// 32 rows per warp and 32-column tiles.
#include "kernels.hpp"
#include "blocksum.cuh"

#include <algorithm>

namespace sgpu {

namespace {

constexpr int kRows = 8, kCols = 128; // of a tile
constexpr int kPitch = kCols + 2;     // tile row: 16-byte aligned, lanes on distinct banks
constexpr int kStages = 5;            // tiles in the ring: 5 CTAs per SM, one wave up to 5900 rows
constexpr int kLeanStages = 3;        // the lean variant: little shared memory, to run beside other kernels

__device__ __forceinline__ void cp_async(double* smem, const double* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The grid covers ceil(nr / kRows) x K planes. PAIR: one plane, two sums in one pass (out[0] = sum of |v|,
// out[1] = sum of v, each in the same order).
template <int STAGES, bool PAIR>
__global__ void __launch_bounds__(kCols)
    k_ordered_sum(const double* __restrict__ vals, std::size_t plane_stride, int ld, int nr, int nc,
                  double* __restrict__ rows, unsigned int* counter, double* __restrict__ out, const int* skip) {
    if (skip && *skip) return;
    extern __shared__ __align__(16) double ring[]; // STAGES tiles
    __shared__ bool last_block;
    const int m = blockIdx.y, tid = threadIdx.x;
    const int r0 = blockIdx.x * kRows, nrow = min(kRows, nr - r0);
    const double* src = vals + m * plane_stride + static_cast<std::size_t>(r0) * ld;
    const int ntiles = (nc + kCols - 1) / kCols;
    auto issue = [&](int k) {
        const int c = k * kCols + tid;
        if (c < nc) {
            double* t = ring + (k % STAGES) * kRows * kPitch + tid;
            for (int r = 0; r < nrow; ++r) cp_async(t + r * kPitch, src + static_cast<std::size_t>(r) * ld + c);
        }
        cp_async_commit();
    };
    for (int k = 0; k < STAGES - 1; ++k) issue(k);
    const int warp = tid / 32, r = tid % 32; // the first warp adds v, the second one |v|
    const bool adds = r < nrow && warp < (PAIR ? 2 : 1), absolute = PAIR && warp == 1;
    double s = 0.0;
    for (int k = 0; k < ntiles; ++k) {
        cp_async_wait<STAGES - 2>(); // tile k has landed (this thread's copies)
        __syncthreads();             // ... and everyone's; tile k - 1 has been added
        issue(k + STAGES - 1);
        if (adds) {
            const double* t = ring + (k % STAGES) * kRows * kPitch + r * kPitch;
            const int n = min(kCols, nc - k * kCols);
            s = absolute ? ordered_chain<true>(s, t, n) : ordered_chain(s, t, n);
        }
    }
    cp_async_wait<0>();
    if (adds) rows[static_cast<std::size_t>(PAIR ? (absolute ? 0 : 1) : m) * nr + r0 + r] = s;

    // The last CTA to finish adds every plane's row sums in row order, a chunk at a time from shared memory.
    __threadfence();
    __syncthreads();
    if (tid == 0) last_block = atomicAdd(counter, 1u) == gridDim.x * gridDim.y - 1;
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    const int K = PAIR ? 2 : static_cast<int>(gridDim.y);
    const int cap = (STAGES * kRows * kPitch / K) & ~1; // row sums of a plane in the ring at once
    double acc = 0.0;
    for (int c0 = 0; c0 < nr; c0 += cap) {
        const int n = min(cap, nr - c0);
        __syncthreads();
        for (int p = 0; p < K; ++p)
            for (int q0 = tid; q0 < n; q0 += 8 * kCols) { // eight loads in flight; L2: other CTAs wrote them
                double x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    x[u] = q0 + u * kCols < n ? __ldcg(rows + static_cast<std::size_t>(p) * nr + c0 + q0 + u * kCols) : 0.0;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (q0 + u * kCols < n) ring[p * cap + q0 + u * kCols] = x[u];
            }
        __syncthreads();
        if (tid < K) acc = ordered_chain(acc, ring + tid * cap, n);
    }
    if (tid < K) out[tid] = acc;
    if (tid == 0) *counter = 0u; // ready for the next launch on this stream
}

template <int STAGES, bool PAIR = false>
void launch_sum(const double* vals, std::size_t plane_stride, int ld, int nr, int nc, int K,
                double* out, const SumScratch& s, const int* skip, cudaStream_t st) {
    const int kout = PAIR ? 2 : K;
    if (K < 1 || K > 32 || kout > s.max_k || nr > s.max_rows || (PAIR && K != 1))
        throw Error(SGPU_E_INVALID, "ordered sum: sizes exceed the scratch");
    if (nr <= 0) {
        SGPU_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * kout, st));
        return;
    }
    const dim3 grid((nr + kRows - 1) / kRows, K);
    constexpr int smem = STAGES * kRows * kPitch * static_cast<int>(sizeof(double));
    static PerDeviceOnce attr; // the attribute lives in each device's context
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_ordered_sum<STAGES, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        return 0;
    });
    k_ordered_sum<STAGES, PAIR><<<grid, kCols, smem, st>>>(vals, plane_stride, ld, nr, nc, s.rows, s.counter, out, skip);
    SGPU_LAUNCH();
}

// ---- deterministic FP64 tree sums (the mixed-precision path) ----

// Block k: *jobs.out[k] = the sum of the jobs.n[k] partial sums at jobs.part[k]: thread t adds values t,
// t + 1024, ... in order, then the block tree.
__global__ void __launch_bounds__(1024) k_sum_partials(SumJobs jobs) {
    __shared__ double s[32];
    const double* src = jobs.part[blockIdx.x];
    const int n = jobs.n[blockIdx.x];
    double a = 0.0;
#pragma unroll 8
    for (int i = static_cast<int>(threadIdx.x); i < n; i += 1024) a += src[i];
    const double t = block_sum<32>(a, s, static_cast<int>(threadIdx.x));
    if (threadIdx.x == 0) *jobs.out[blockIdx.x] = t;
}

constexpr int kTileRows = 32; // rows per block of k_tile_sum

// Block (bx, by) of an nr x nc array (row stride ld): columns 256 bx .. +255, rows 32 by .. +31.
// Each thread adds its column's values top to bottom in FP64, then the block tree; one partial sum
// per block.
template <class T>
__global__ void __launch_bounds__(256)
    k_tile_sum(const T* __restrict__ vals, int ld, int nr, int nc, double* __restrict__ part) {
    __shared__ double s[8];
    const int c = static_cast<int>(blockIdx.x * 256 + threadIdx.x);
    const int r0 = static_cast<int>(blockIdx.y) * kTileRows, r1 = min(r0 + kTileRows, nr);
    double a = 0.0;
    if (c < nc) {
        const T* src = vals + static_cast<std::size_t>(r0) * ld + c;
#pragma unroll 8
        for (int r = r0; r < r1; ++r, src += ld) a += static_cast<double>(*src);
    }
    const double t = block_sum<8>(a, s, static_cast<int>(threadIdx.x));
    if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = t;
}

} // namespace

void launch_sum_partials(const SumJobs& jobs, cudaStream_t st) {
    if (jobs.count < 1 || jobs.count > SumJobs::kMax) throw Error(SGPU_E_INVALID, "partial sums: 1 to 4 jobs");
    k_sum_partials<<<jobs.count, 1024, 0, st>>>(jobs);
    SGPU_LAUNCH();
}

void launch_sum_partials(const double* part, int n, int K, int plane, double* out0, double* out1,
                         cudaStream_t st) {
    if (K < 1 || K > 2 || (K == 2 && !out1)) throw Error(SGPU_E_INVALID, "partial sums: 1 or 2 planes");
    SumJobs jobs;
    jobs.add(part, n, out0);
    if (K == 2) jobs.add(part + plane, n, out1);
    launch_sum_partials(jobs, st);
}

int tree_sum_partials(int nr, int nc) {
    return ((nc + 255) / 256) * ((nr + kTileRows - 1) / kTileRows);
}

void launch_tree_sum(const float* vals, int ld, int nr, int nc, double* part, double* out, cudaStream_t st) {
    if (nr <= 0 || nc <= 0) {
        if (out) SGPU_CUDA(cudaMemsetAsync(out, 0, sizeof(double), st));
        return;
    }
    const dim3 grid((nc + 255) / 256, (nr + kTileRows - 1) / kTileRows);
    k_tile_sum<float><<<grid, 256, 0, st>>>(vals, ld, nr, nc, part);
    SGPU_LAUNCH();
    if (out) launch_sum_partials(part, static_cast<int>(grid.x * grid.y), 1, 0, out, nullptr, st);
}

void launch_ordered_sum(const double* vals, std::size_t plane_stride, int ld, int nr, int nc, int K,
                        double* out, const SumScratch& s, const int* skip, cudaStream_t st) {
    launch_sum<kStages>(vals, plane_stride, ld, nr, nc, K, out, s, skip, st);
}

void launch_ordered_sum_abs_pair(const double* vals, int ld, int nr, int nc, double* out, const SumScratch& s,
                                 cudaStream_t st) {
    launch_sum<kStages, true>(vals, 0, ld, nr, nc, 1, out, s, nullptr, st);
}

void launch_ordered_sum_lean(const double* vals, int ld, int nr, int nc, double* out, const SumScratch& s,
                             cudaStream_t st) {
    launch_sum<kLeanStages>(vals, 0, ld, nr, nc, 1, out, s, nullptr, st);
}

} // namespace sgpu
