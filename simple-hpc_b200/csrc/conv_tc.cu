// conv_tc.cu — the warm-start network's 3x3 convolutions on the Blackwell tensor cores (tcgen05).
//
// Implicit GEMM: Y[p, co] = sum over taps t and input channels ci of X[p + t, ci] W[co, t, ci], with
// M = pixels in blocks of 128 (the accumulator's TMEM lanes), N = output channels (FP32 accumulator
// columns in TMEM) and K = 9 taps x Cin. See k_conv_tc (forward and input gradient) and k_conv_wgrad_tc
// (weight gradient). Every mbarrier wait is bounded: a give-up sets *err, no further MMA is issued,
// outstanding commits are waited for (bounded again), TMEM is freed and the CTA returns.
#include "cnn.hpp"

#include <algorithm>
#include <cstdint>

namespace sgpu {

namespace {

using bf16 = __nv_bfloat16;

constexpr int kM = 128;          // accumulator rows = TMEM lanes
constexpr int kThreadsTc = 128;  // 4 warps: warp w owns TMEM lanes 32w .. 32w + 31
constexpr int kSpinTc = 1 << 22; // mbarrier polls before a wait gives up

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bar_init(uint64_t* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ bool bar_test(uint64_t* b, unsigned parity) {
    unsigned done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(smem_addr(b)), "r"(parity)
                 : "memory");
    return done != 0;
}
// Bounded wait for phase `parity` of b; false (and *err set) on a give-up.
__device__ __forceinline__ bool bar_wait(uint64_t* b, unsigned parity, unsigned* err) {
    for (int it = 0; !bar_test(b, parity); ++it)
        if (it >= kSpinTc) {
            atomicOr(err, 2u);
            return false;
        }
    return true;
}

// Shared-memory matrix descriptor (tcgen05): start address, leading and stride byte offsets (all
// >> 4), the fixed field 0b001 at bits 46-48, base offset 0, no swizzling.
__device__ __forceinline__ uint64_t smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, N and M.
__host__ __device__ constexpr uint32_t instr_desc(int n, int m) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void mma_issue(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                     smem_addr(b))
                 : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// Generic-proxy shared-memory writes made visible to the tensor cores' (async proxy) reads.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// 16 FP32 accumulator columns [col, col + 16) of this warp's 32 TMEM lanes: lane i of the warp gets
// row 32 (warp % 4) + i.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                 "%12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// 16-byte asynchronous copy global -> shared; src_bytes 0 writes zeros (no global read).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, unsigned src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// ---- forward and input gradient ----
//
// Tiles are stored as they lie in memory, a plane per 8 channels and 16 bytes per pixel, which is the
// K-major layout without swizzling (core matrices of 8 pixels x 16 bytes, 128 bytes apart in M, a plane
// apart in K). So the CTA brings its input tile in once, with plain 16-byte copies, and a tap is only
// another start address: the pixels of a tile are numbered with a pitch of cw + 2 (one halo column on
// each side), M block b of tap (dy, dx) starts at pixel 128 b + dy (cw + 2) + dx, and the rows of the
// product that fall on halo columns or past the tile are not stored. (Gathering a tile per tap instead,
// nine reads of the input, is what bound this kernel before.) Weights sit beside it, a tile per tap.
// The order of the MMAs of an output is chunk, tap, channel, whatever the tile.
// mask (the input gradient of a pair's second convolution): the output of the layer whose gradient this
// is; the gradient is zeroed where that layer's ReLU was off, and db[co] += its sum over the pixels, so
// neither takes a pass of its own.
// Measured: the 14 convolutions of a forward pass on one 256^2 image, 169 us against 276 us; the 27
// of a training step on 8 images, 0.78 ms against 1.63 ms.
constexpr int kThreadsConv = 256; // two warps per TMEM lane quarter

// g where the post-activation outputs y (two BF16) are positive, else 0.
__device__ __forceinline__ __nv_bfloat162 relu_mask(uint32_t y, __nv_bfloat162 g) {
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&y);
    const __nv_bfloat16 zero = __float2bfloat16(0.0f);
    return {__low2float(v) > 0.0f ? g.x : zero, __high2float(v) > 0.0f ? g.y : zero};
}

struct ConvPlan {
    int cw, rb, tb;       // columns and rows of output pixels per CTA; M blocks of 128
    int nt;               // output channels per CTA
    int kc, chunks;       // channels brought in at a time (divides Cin), and how often
    int ctiles, rchunks;  // column tiles and row chunks per image
    unsigned x_plane;     // bytes of one 8-channel plane of the input tile
    int smem;
    uint32_t tmem_cols;
};

__global__ void __launch_bounds__(kThreadsConv)
    k_conv_tc(const bf16* __restrict__ X, int H, int W, int Cin, const bf16* __restrict__ Wt,
              const float* __restrict__ bias, bf16* __restrict__ Y, int Cout, int relu, const bf16* __restrict__ mask,
              float* __restrict__ db, ConvPlan pl, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    __shared__ float s_db[256];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    s_db[tid] = 0.0f;
    int bx = static_cast<int>(blockIdx.x);
    const int x0 = (bx % pl.ctiles) * pl.cw;
    bx /= pl.ctiles;
    const int y0 = (bx % pl.rchunks) * pl.rb;
    const long image = static_cast<long>(bx / pl.rchunks) * H * W;
    const int co0 = static_cast<int>(blockIdx.y) * pl.nt;
    const int P = pl.cw + 2, gk = pl.kc / 8;
    unsigned char* const wtile = smem + gk * pl.x_plane;
    const unsigned w_plane = static_cast<unsigned>(pl.nt) * 16u;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(pl.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        bar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }

    auto load = [&](int c0) { // channels [c0, c0 + kc) of the input tile and of the weights
        const int step_g = 32 % gk, step_c = 32 / gk;
        for (int r = warp; r < pl.rb + 2; r += kThreadsConv / 32) {
            const int y = y0 + r - 1;
            const bool yin = y >= 0 && y < H;
            const bf16* row = X + (image + static_cast<long>(yin ? y : 0) * W) * Cin + c0;
            unsigned char* dst = smem + r * P * 16;
            int c = lane / gk, g = lane - c * gk;
            while (c < P) {
                const int x = x0 + c - 1;
                const bool in = yin && x >= 0 && x < W;
                cp_async16(dst + g * pl.x_plane + c * 16, in ? row + static_cast<long>(x) * Cin + 8 * g : X,
                           in ? 16u : 0u);
                c += step_c;
                g += step_g;
                if (g >= gk) {
                    g -= gk;
                    ++c;
                }
            }
        }
        const int cnt = pl.nt * 9 * gk;
        for (int u = tid; u < cnt; u += kThreadsConv) {
            const int row = u / gk, g = u - row * gk, co = row / 9, t = row - 9 * co;
            cp_async16(wtile + (t * gk + g) * w_plane + co * 16,
                       Wt + (static_cast<long>(co0 + co) * 9 + t) * Cin + c0 + 8 * g, 16u);
        }
        cp_async_commit();
    };

    load(0);
    fence_before();
    __syncthreads(); // the TMEM address and the initialised mbarrier
    fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = instr_desc(pl.nt, kM);
    bool gave_up = false;
    int committed = 0; // chunks
    for (int ch = 0; ch < pl.chunks && !gave_up; ++ch) {
        cp_async_wait<0>(); // this thread's copies
        fence_async_smem();
        __syncthreads(); // ... and everyone's
        if (tid == 0) {
            fence_after();
            const unsigned xa = smem_addr(smem), wa = smem_addr(wtile);
            for (int b = 0; b < pl.tb; ++b) {
                const uint32_t d = tmem + static_cast<uint32_t>(b * pl.nt);
                for (int t = 0; t < 9; ++t) {
                    const unsigned a0 = xa + static_cast<unsigned>(128 * b + (t / 3) * P + t % 3) * 16u;
                    const unsigned w0 = wa + static_cast<unsigned>(t * gk) * w_plane;
                    for (int k = 0; k < gk; k += 2)
                        mma_issue(d, smem_desc(a0 + k * pl.x_plane, pl.x_plane, 128u),
                                  smem_desc(w0 + k * w_plane, w_plane, 128u), idesc,
                                  (ch > 0 || t > 0 || k > 0) ? 1u : 0u);
                }
            }
            mma_commit(&bar);
        }
        committed = ch + 1;
        // every thread waits for the chunk's MMAs (phase ch): the tiles are then free, the sums formed
        if (!bar_wait(&bar, static_cast<unsigned>(ch & 1), err)) gave_up = true;
        if (__syncthreads_or(gave_up ? 1 : 0)) gave_up = true;
        else if (ch + 1 < pl.chunks) load((ch + 1) * pl.kc);
    }
    if (gave_up) {
        // what is in flight, before TMEM and shared memory are given back (bounded)
        if (tid == 0) bar_wait(&bar, static_cast<unsigned>((committed - 1) & 1), err);
    } else {
        fence_after();
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        for (int k0 = 0; k0 < pl.nt; k0 += 16) {
            float sum[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) sum[k] = 0.0f;
            for (int b = warp >> 2; b < pl.tb; b += kThreadsConv / 128) {
                const int m = 128 * b + (warp & 3) * 32 + lane, r = m / P, c = m - r * P;
                const bool live = r < pl.rb && c < pl.cw && y0 + r < H && x0 + c < W;
                const long o = (image + static_cast<long>(y0 + r) * W + x0 + c) * Cout + co0 + k0;
                float v[16];
                __syncwarp(); // tcgen05.ld takes the whole warp, converged
                tmem_ld16(tmem + lane_base + static_cast<uint32_t>(b * pl.nt + k0), v);
                if (live) {
                    uint4 q[2], y[2];
                    if (mask) {
                        y[0] = __ldg(reinterpret_cast<const uint4*>(mask + o));
                        y[1] = __ldg(reinterpret_cast<const uint4*>(mask + o) + 1);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        float v0 = v[2 * k] + (bias ? bias[co0 + k0 + 2 * k] : 0.0f);
                        float v1 = v[2 * k + 1] + (bias ? bias[co0 + k0 + 2 * k + 1] : 0.0f);
                        if (relu) {
                            v0 = fmaxf(v0, 0.0f);
                            v1 = fmaxf(v1, 0.0f);
                        }
                        __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
                        if (mask) {
                            h = relu_mask((&y[0].x)[k], h);
                            sum[2 * k] += __low2float(h);
                            sum[2 * k + 1] += __high2float(h);
                        }
                        (&q[0].x)[k] = *reinterpret_cast<const uint32_t*>(&h);
                    }
                    uint4* dst = reinterpret_cast<uint4*>(Y + o);
                    dst[0] = q[0];
                    dst[1] = q[1];
                }
            }
            if (mask) { // (uniform) the bias gradient of the masked output
#pragma unroll
                for (int k = 0; k < 16; ++k)
                    for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
                if (lane == 0)
#pragma unroll
                    for (int k = 0; k < 16; ++k) atomicAdd(&s_db[k0 + k], sum[k]);
            }
        }
        if (mask) {
            __syncthreads();
            if (tid < pl.nt) atomicAdd(db + co0 + tid, s_db[tid]);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(pl.tmem_cols)
                     : "memory");
}

// Weight gradient of a 3x3 convolution: dW[co, t, ci] += sum over pixels p of dZ[p, co] X[p + t, ci].
// A GEMM with M = output channels (128 lanes; rows from Cout on are whatever lies behind the tile and
// are never read back), N = Cin per tap (taps side by side in TMEM) and K = pixels.
//  * Layout. Both operands are stored as they lie in memory, channels innermost ("MN-major"): a plane
//    per 8 channels, 16 bytes per pixel, pixels of a row contiguous. So a tile row is filled with plain
//    16-byte copies, and a tap is only another start address: one pixel to the side is 16 bytes, one
//    row up or down another ring slot. X is brought in once for its nine taps (the gather into K-major
//    tiles that this replaces read it nine times and transposed it with 4-byte stores: that bound it).
//  * Split. A CTA takes `cw` columns (a multiple of 16, zero-filled past the image), `rows` rows of one
//    image and `nt` taps (nt Cin <= 512 TMEM columns); it walks down its rows with a ring of kWgAhead + 3
//    rows of X and kWgAhead + 1 of dZ, filled by cp.async kWgAhead rows ahead of the MMAs. At most 4096
//    pixels are accumulated before the FP32 adds into dW (vector reductions).
// Measured: the 14 weight gradients of a training step on 8 images of 256^2, 0.91 ms against 8.42 ms.
constexpr int kWgAhead = 2;
constexpr int kWgXRows = kWgAhead + 3, kWgZRows = kWgAhead + 1;

struct WgradPlan {
    int cw, rows, nt;         // columns, rows and taps per CTA
    int ctiles, rchunks;      // column tiles and row chunks per image
    unsigned z_plane, x_plane; // bytes of one 8-channel plane of a tile row
    unsigned z_row, x_row;     // bytes of one tile row (all planes)
    int smem;
};

// Shared-memory descriptor of an MN-major tile without swizzling: `k8` bytes between groups of 8
// pixels, `mn8` between planes of 8 channels.
__device__ __forceinline__ uint64_t smem_desc_mn(unsigned addr, unsigned k8, unsigned mn8) {
    return smem_desc(addr, k8, mn8);
}

__global__ void __launch_bounds__(kThreadsTc)
    k_conv_wgrad_tc(const bf16* __restrict__ X, const bf16* __restrict__ dZ, int H, int W, int Cin, int Cout,
                    WgradPlan pl, float* __restrict__ dW, uint32_t tmem_cols, unsigned* err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[3]; // stages in turn; [2] the end of all MMAs
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int t0 = blockIdx.y * pl.nt, nt = min(pl.nt, 9 - t0);
    int bx = static_cast<int>(blockIdx.x);
    const int x0 = (bx % pl.ctiles) * pl.cw;
    bx /= pl.ctiles;
    const int y0 = (bx % pl.rchunks) * pl.rows, n = bx / pl.rchunks;
    const int nrows = min(pl.rows, H - y0);
    unsigned char* const xring = smem + kWgZRows * pl.z_row;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                         smem_addr(&tmem_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        bar_init(&bars[0], 1);
        bar_init(&bars[1], 1);
        bar_init(&bars[2], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;

    const int gz = Cout / 8, gx = Cin / 8;
    const long image = static_cast<long>(n) * H * W;
    // row y of X, columns x0 - 1 .. x0 + cw, into its ring slot (zeros outside the image)
    auto load_x = [&](int y) {
        unsigned char* dst = xring + ((y + 1) % kWgXRows) * pl.x_row;
        const bool yin = y >= 0 && y < H;
        const int cnt = (pl.cw + 2) * gx;
        for (int u = tid; u < cnt; u += kThreadsTc) {
            const int px = u / gx, g = u - px * gx, x = x0 + px - 1;
            const bool in = yin && x >= 0 && x < W;
            cp_async16(dst + g * pl.x_plane + px * 16, in ? X + (image + static_cast<long>(y) * W + x) * Cin + 8 * g : X,
                       in ? 16u : 0u);
        }
    };
    auto load_z = [&](int s) {
        unsigned char* dst = smem + (s % kWgZRows) * pl.z_row;
        const int cnt = pl.cw * gz;
        for (int u = tid; u < cnt; u += kThreadsTc) {
            const int px = u / gz, g = u - px * gz, x = x0 + px;
            const bool in = x < W;
            cp_async16(dst + g * pl.z_plane + px * 16,
                       in ? dZ + (image + static_cast<long>(y0 + s) * W + x) * Cout + 8 * g : dZ, in ? 16u : 0u);
        }
    };
    auto issue = [&](int s) { // what stage s (row y0 + s) adds to the rings; one group per stage
        if (s < nrows) {
            if (s == 0) {
                load_x(y0 - 1);
                load_x(y0);
            }
            load_x(y0 + s + 1);
            load_z(s);
        }
        cp_async_commit();
    };

    const uint32_t idesc = instr_desc(Cin, kM) | (1u << 15) | (1u << 16); // A and B MN-major
    bool gave_up = false;
    int issued = 0;
    for (int s = 0; s < kWgAhead; ++s) issue(s);
    for (int s = 0; s < nrows; ++s) {
        cp_async_wait<kWgAhead - 1>(); // this thread's copies of stage s have landed
        fence_async_smem();
        if (__syncthreads_or(gave_up ? 1 : 0)) {
            gave_up = true;
            break;
        }
        if (tid == 0) {
            fence_after();
            const unsigned za = smem_addr(smem + (s % kWgZRows) * pl.z_row);
            for (int tl = 0; tl < nt; ++tl) {
                const int t = t0 + tl;
                // tap t of pixel x: row y0 + s + t / 3 - 1, ring column x - x0 + 1 + t % 3 - 1
                const unsigned xa =
                    smem_addr(xring + ((y0 + s + t / 3) % kWgXRows) * pl.x_row) + static_cast<unsigned>(t % 3) * 16u;
                for (int k = 0; k < pl.cw / 16; ++k)
                    mma_issue(tmem + static_cast<uint32_t>(tl * Cin), smem_desc_mn(za + 256u * k, 128u, pl.z_plane),
                              smem_desc_mn(xa + 256u * k, 128u, pl.x_plane), idesc, (s > 0 || k > 0) ? 1u : 0u);
            }
            mma_commit(&bars[s & 1]);
            if (s == nrows - 1) mma_commit(&bars[2]);
        }
        issued = s + 1;
        // stage s + kWgAhead refills the slots that stage s - 1 read last
        if (s >= 1 && s + kWgAhead < nrows &&
            !bar_wait(&bars[(s - 1) & 1], static_cast<unsigned>(((s - 1) >> 1) & 1), err))
            gave_up = true;
        if (!gave_up) issue(s + kWgAhead);
        else cp_async_commit();
    }
    cp_async_wait<0>();
    if (!gave_up && !bar_wait(&bars[2], 0u, err)) gave_up = true;
    if (__syncthreads_or(gave_up ? 1 : 0)) {
        // wait (bounded) for what is in flight before TMEM and shared memory are given back
        if (tid == 0 && issued > 0) {
            if (issued < nrows) mma_commit(&bars[2]);
            bar_wait(&bars[2], 0u, err);
        }
    } else if (issued > 0) {
        fence_after();
        const int co = warp * 32 + (tid & 31);
        const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
        if (warp * 32 < Cout) // uniform in the warp
            for (int c0 = 0; c0 < nt * Cin; c0 += 16) { // 16 columns of one tap (Cin is a multiple of 16)
                float v[16];
                __syncwarp(); // (as above)
                tmem_ld16(tmem + lane_base + static_cast<uint32_t>(c0), v);
                if (co < Cout) {
                    float* dst = dW + (static_cast<long>(co) * 9 + t0) * Cin + c0;
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst + e), "f"(v[e]),
                                     "f"(v[e + 1]), "f"(v[e + 2]), "f"(v[e + 3])
                                     : "memory");
                }
            }
    }
    fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(tmem_cols)
                     : "memory");
}

// Kernel shared memory available for the stage ring (one CTA's share of an SM).
constexpr int kConvSmemMax = 200 * 1024;
constexpr int kWgSmemPair = 110 * 1024; // the weight gradient's share with two CTAs on an SM

// The tile of a convolution. Channels come in at once up to 128 (more: the largest multiple of 16 that
// divides Cin and is at most 128). Among the column widths, M blocks and output channel splits that fit,
// the one of least estimated time: per wave of resident CTAs a latency of about 2 us (allocation, copies
// in flight, first MMA, epilogue), per CTA its bytes at about 60 B/ns, its MMAs (an MMA reads its 4 KB of
// A in about 20 ns, more with many output channels) and its stores. Narrow tiles waste product rows on
// halo columns, wide or tall ones leave SMs idle on a single image.
// Where the weights of all output channels do not fit beside a tile (128 -> 128), that leaves one CTA of few
// output channels on an SM, whose copies wait for nobody's MMAs. There 16 channels at a time, for 64 output
// channels or more, are tried too: small tiles, several CTAs on an SM, one's copies beside another's MMAs, at
// about 0.6 us a chunk; taken where the estimate is well below the other's. A base of 128 channels, one level,
// us a forward call, all channels at once / 16 at a time: 2 x 16 x 1024 200 / 161, 1 x 128^2 138 / 126,
// 1 x 256^2 291 / 217, 1 x 512^2 944 / 685 (8 x 32^2: 132 either way, all at once).
ConvPlan conv_plan(int N, int H, int W, int cin, int cout) {
    int whole = cin;
    if (whole > 128)
        for (whole = 128; cin % whole; whole -= 16) {}
    const int wr = (W + 7) / 8 * 8;
    // the best plan that brings in kc channels at a time and forms at least nt_min output channels; its time in ns
    auto search = [&](int kc, int nt_min, double& best_ns) {
        ConvPlan best{};
        best_ns = 1e30;
        for (int cw : {8, 16, 32, 48, 64, 96, 128}) {
            if (cw > wr && cw != 8) continue;
            const int P = cw + 2;
            for (int tb : {1, 2, 3, 4, 6, 8}) {
                const int rb = std::min(H, 128 * tb / P);
                if (rb < 1 || (tb > 1 && 128 * (tb - 1) >= rb * P)) continue;
                for (int nt = cout; nt >= nt_min; nt = nt % 32 ? nt - 16 : nt / 2) {
                    if (cout % nt || tb * nt > 512) continue;
                    const long lp = 128L * tb + 2 * P + 2; // pixels a shifted block may read
                    const long smem = lp * 16 * (kc / 8) + 9L * kc * nt * 2;
                    if (smem > kConvSmemMax) continue;
                    uint32_t cols = 32;
                    while (cols < static_cast<uint32_t>(tb * nt)) cols <<= 1;
                    const long occ = std::min({227L * 1024 / (smem + 1024), 512L / cols, 8L});
                    const long ct = (W + cw - 1) / cw, rc = (H + rb - 1) / rb;
                    const long ctas = ct * rc * N * (cout / nt), chunks = cin / kc;
                    const double copies = static_cast<double>((rb + 2) * P * 2L * cin + 18L * cin * nt) / 60.0;
                    const double mma = 9.0 * (cin / 16) * tb * std::max(20.0, 0.3 * nt);
                    const double waves = static_cast<double>((ctas + 148 * occ - 1) / (148 * occ));
                    const double per_sm = static_cast<double>((ctas + 147) / 148);
                    const double together = std::min(static_cast<double>(occ), per_sm);
                    const double ns =
                        (kc == whole ? waves * (1000.0 + 1000.0 * chunks) + per_sm * (copies + mma)
                                     : waves * std::max(1000.0 + 600.0 * chunks + copies + mma, together * std::max(copies, mma))) +
                        per_sm * (tb * nt * 2.0);
                    if (ns < best_ns) {
                        best_ns = ns;
                        best = {cw, rb, tb, nt, kc, static_cast<int>(chunks), static_cast<int>(ct), static_cast<int>(rc),
                                static_cast<unsigned>(lp * 16), static_cast<int>(smem), cols};
                    }
                }
            }
        }
        return best;
    };
    double ns = 0.0, ns16 = 0.0;
    ConvPlan best = search(whole, 16, ns);
    if (whole > 16 && 9L * whole * cout * 2 > kConvSmemMax) {
        const ConvPlan chunked = search(16, 64, ns16);
        if (ns16 < 0.7 * ns) best = chunked;
    }
    return best;
}

} // namespace

void launch_conv_wgrad_tc(const bf16* X, const bf16* dZ, int N, int H, int W, int Cin, int Cout, float* dW,
                          unsigned* err, cudaStream_t st) {
    if (Cin < 16 || Cin > 256 || Cin % 16 || Cout < 16 || Cout > kM || Cout % 16 || !err)
        throw Error(SGPU_E_INVALID, "tensor-core weight gradient: channels must be multiples of 16, Cout <= 128");
    const auto misaligned = [](const void* q) { return (reinterpret_cast<std::uintptr_t>(q) & 15u) != 0; };
    if (misaligned(X) || misaligned(dZ))
        throw Error(SGPU_E_INVALID, "tensor-core weight gradient: operands must be 16-byte aligned");
    if (reinterpret_cast<std::uintptr_t>(dW) & 15u)
        throw Error(SGPU_E_INVALID, "tensor-core weight gradient: dW must be 16-byte aligned");
    if (static_cast<long>(N) * H * W <= 0) return;
    WgradPlan pl{};
    pl.nt = std::min(9, 512 / Cin); // Cin <= 256: two taps at least
    pl.nt = (9 + (9 + pl.nt - 1) / pl.nt - 1) / ((9 + pl.nt - 1) / pl.nt); // even groups
    // the widest column tile whose rings fit (two CTAs per SM where that still leaves 64 columns)
    auto size = [&](int cw) {
        pl.cw = cw;
        pl.z_plane = static_cast<unsigned>(cw) * 16u;
        pl.x_plane = static_cast<unsigned>(cw + 2) * 16u;
        pl.z_row = pl.z_plane * (Cout / 8);
        pl.x_row = pl.x_plane * (Cin / 8);
        // the A descriptor spans 16 planes from any dZ slot, whatever Cout is
        const unsigned rings = kWgZRows * pl.z_row + kWgXRows * pl.x_row;
        pl.smem = static_cast<int>(std::max(rings, (kWgZRows - 1) * pl.z_row + 16u * pl.z_plane));
        return pl.smem;
    };
    int cw = std::min(256, (W + 15) / 16 * 16);
    while (cw > 16 && size(cw) > (cw > 64 ? kWgSmemPair : kConvSmemMax)) cw = (cw / 2 + 15) / 16 * 16;
    if (size(cw) > kConvSmemMax)
        throw Error(SGPU_E_INVALID, "tensor-core weight gradient: row ring exceeds shared memory");
    pl.ctiles = (W + cw - 1) / cw;
    // rows per CTA: about two CTAs per SM over the layer, at most 4096 pixels each
    const long want = std::max(1L, 296L / ((9 + pl.nt - 1) / pl.nt) / pl.ctiles);
    pl.rows = static_cast<int>(std::max(1L, std::min<long>(4096 / cw, (static_cast<long>(N) * H + want - 1) / want)));
    pl.rows = std::min(pl.rows, H);
    pl.rchunks = (H + pl.rows - 1) / pl.rows;
    uint32_t cols = 32;
    while (cols < static_cast<uint32_t>(pl.nt * Cin)) cols <<= 1;
    static PerDeviceOnce attr;
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_conv_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmemMax));
        return 0;
    });
    const dim3 grid(static_cast<unsigned>(static_cast<long>(N) * pl.rchunks * pl.ctiles),
                    static_cast<unsigned>((9 + pl.nt - 1) / pl.nt));
    k_conv_wgrad_tc<<<grid, kThreadsTc, pl.smem, st>>>(X, dZ, H, W, Cin, Cout, pl, dW, cols, err);
    SGPU_LAUNCH();
}

void launch_conv_tc(const bf16* X, int N, int H, int W, int Cin, const bf16* Wt, const float* bias, bf16* Y,
                    int Cout, int relu, unsigned* err, cudaStream_t st, const bf16* mask, float* db) {
    if (Cin < 16 || Cin % 16 || Cout < 16 || Cout > 256 || Cout % 16 || !err)
        throw Error(SGPU_E_INVALID, "tensor-core convolution: channels must be multiples of 16, Cout <= 256");
    const auto misaligned = [](const void* q) { return (reinterpret_cast<std::uintptr_t>(q) & 15u) != 0; };
    if (misaligned(X) || misaligned(Wt) || misaligned(Y) || misaligned(mask) || (mask && !db))
        throw Error(SGPU_E_INVALID, "tensor-core convolution: operands must be 16-byte aligned");
    const long npix = static_cast<long>(N) * H * W;
    if (npix <= 0) return;
    const ConvPlan pl = conv_plan(N, H, W, Cin, Cout);
    if (pl.smem <= 0) throw Error(SGPU_E_INVALID, "tensor-core convolution: no tile fits shared memory");
    static PerDeviceOnce attr;
    attr.get([] {
        SGPU_CUDA(cudaFuncSetAttribute(k_conv_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmemMax));
        return 0;
    });
    const dim3 grid(static_cast<unsigned>(static_cast<long>(N) * pl.ctiles * pl.rchunks),
                    static_cast<unsigned>(Cout / pl.nt));
    k_conv_tc<<<grid, kThreadsConv, pl.smem, st>>>(X, H, W, Cin, Wt, bias, Y, Cout, relu, mask, db, pl, err);
    SGPU_LAUNCH();
}

} // namespace sgpu
