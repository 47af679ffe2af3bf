// One-kernel transforms of 2^13 and 2^14 values: persistent blocks, the next transform's bulk copy in
// flight while the current one computes.
#include "fft_tma.cuh"

namespace ofb {

cudaError_t set_expire_waits_long(int on) {
    const int v = on ? 1 : 0;
    return cudaMemcpyToSymbol(g_expire_waits, &v, sizeof v);
}

// A transform of n = B 4096 values (B = 2, 4) as B transforms of the 4096-value sub-sequences
// x[B i + s], three radix-16 stages each, and one radix-B stage over them: k_batched's Stockham
// schedule for n, stage for stage (the same operations on the same values, so the same bits), but
// with all B sub-sequences of a butterfly lane in ONE thread, 16 B values, so that
//  - the last stage needs no exchange (2 instead of 3);
//  - a thread loads each stage twiddle once for its B butterflies;
//  - an exchange moves the B re (then im) parts of a lane as one 8- or 16-byte word. Half the
//    values' bytes at a time leaves room for the landing buffer: the next transform arrives by one
//    bulk copy while this one computes.
// What bounds it: the shared-memory pipe (46-55 % busy, ncu) and the arithmetic between the block's
// barriers, on the 8 (2^14) or 16 (2^13) warps per SM that registers allow; HBM runs at 60-80 % of
// the copy rate. Against k_batched's one block of 16 values per thread (B200, forward, calls back to
// back): 4096 x 2^13 124 -> 104 us, 1000 x 2^13 34.4 -> 32.0, 2048 x 2^14 153 -> 135, 1021 x 2^14
// 81 -> 70, 300 x 2^14 33.4 -> 29.5. Measured and left out: stage tables in shared memory (2^14
// 69 -> 76 us: the pipe is the bound), last-stage twiddles loaded early or past L1 (slower), the
// first exchange within half-warps in place of the landing buffer, which needs 256 padded row
// copies instead of one (2^13 55 -> 93 us for 2048: about 50 cycles per bulk copy).
template <int B>
struct Lanes;  // B FP32 values as one shared-memory word
template <>
struct Lanes<2> {
    using T = float2;
};
template <>
struct Lanes<4> {
    using T = float4;
};
template <int B>
struct Long {
    static constexpr int LOG_B = B == 2 ? 1 : 2, LOG_N = 12 + LOG_B, N = 1 << LOG_N, THREADS = 256;
    static constexpr int EX_OFF = 8 * N;                     // bytes; the landing buffer comes first
    static constexpr int EX_WORDS = 4096 + 256;              // of 4 B bytes; one pad word every 16
    static constexpr int BAR_OFF = EX_OFF + 4 * B * EX_WORDS;
    static constexpr int SMEM = BAR_OFF + 16;
};

__device__ __forceinline__ float2 gather_x(const float2 (&v)[2][16], int k) { return make_float2(v[0][k].x, v[1][k].x); }
__device__ __forceinline__ float2 gather_y(const float2 (&v)[2][16], int k) { return make_float2(v[0][k].y, v[1][k].y); }
__device__ __forceinline__ float4 gather_x(const float2 (&v)[4][16], int k) {
    return make_float4(v[0][k].x, v[1][k].x, v[2][k].x, v[3][k].x);
}
__device__ __forceinline__ float4 gather_y(const float2 (&v)[4][16], int k) {
    return make_float4(v[0][k].y, v[1][k].y, v[2][k].y, v[3][k].y);
}
__device__ __forceinline__ void scatter_x(float2 (&v)[2][16], int k, float2 w) { v[0][k].x = w.x, v[1][k].x = w.y; }
__device__ __forceinline__ void scatter_y(float2 (&v)[2][16], int k, float2 w) { v[0][k].y = w.x, v[1][k].y = w.y; }
__device__ __forceinline__ void scatter_x(float2 (&v)[4][16], int k, float4 w) {
    v[0][k].x = w.x, v[1][k].x = w.y, v[2][k].x = w.z, v[3][k].x = w.w;
}
__device__ __forceinline__ void scatter_y(float2 (&v)[4][16], int k, float4 w) {
    v[0][k].y = w.x, v[1][k].y = w.y, v[2][k].y = w.z, v[3][k].y = w.w;
}

// Stages S .. 2 of the B sub-transforms of 4096 values, lane j of 256. The block has been
// synchronised since the exchange buffer was last read.
template <int B, int S>
__device__ __forceinline__ void long_stages(float2 (&v)[B][16], int j, const float2* __restrict__ stw,
                                            typename Lanes<B>::T* ex) {
    constexpr int LNS = Stages<12>::log2_ns(S), NS = 1 << LNS;
    if (S > 0) {
        const float2* tw = stw + Stages<12>::tw_offset(S) + (j & (NS - 1));
#pragma unroll
        for (int q = 1; q < 16; ++q) {
            const float2 w = __ldg(tw + (q - 1) * NS);
#pragma unroll
            for (int s = 0; s < B; ++s) v[s][q] = cmul(v[s][q], w);
        }
    }
#pragma unroll
    for (int s = 0; s < B; ++s) dft16(v[s]);
    if constexpr (S < 2) {
        typename Lanes<B>::T* w = ex + spad(((j >> LNS) << (4 + LNS)) + (j & (NS - 1)));
        const typename Lanes<B>::T* r = ex + spad(j);
        if (S > 0) __syncthreads();  // the previous exchange's reads are done
#pragma unroll
        for (int p = 0; p < 16; ++p) w[padc(p * NS)] = gather_x(v, p);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) scatter_x(v, k, r[padc(k * 256)]);
        __syncthreads();
#pragma unroll
        for (int p = 0; p < 16; ++p) w[padc(p * NS)] = gather_y(v, p);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) scatter_y(v, k, r[padc(k * 256)]);
        long_stages<B, S + 1>(v, j, stw, ex);
    }
}

template <int B, int INV, bool W>
__global__ void __launch_bounds__(256, B == 2 ? 2 : 1)
    k_batched_long(const float2* __restrict__ in, float2* __restrict__ out, long long batch,
                   const float2* __restrict__ stw, unsigned* err, const float2* __restrict__ pre,
                   const float2* __restrict__ post) {
    using G = Long<B>;
    constexpr int LOG_N = G::LOG_N;
    constexpr unsigned BYTES = 8u * G::N;
    extern __shared__ __align__(1024) unsigned char long_smem[];
    const float2* land = reinterpret_cast<const float2*>(long_smem);
    auto* ex = reinterpret_cast<typename Lanes<B>::T*>(long_smem + G::EX_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(long_smem + G::BAR_OFF);
    const int j = threadIdx.x;
    long long b = blockIdx.x;
    unsigned parity = 0;
    if (j == 0) {
        mbar_init(bar, 1);
        dependent_wait();  // the other threads touch the caller's buffers only after the copy landed
        mbar_expect_tx(bar, BYTES);
        bulk_load(long_smem, in + (b << LOG_N), BYTES, bar);
    }
    __syncthreads();  // the barrier is initialised before anyone waits on it
    for (; b < batch; b += gridDim.x, parity ^= 1u) {
        const bool ok = !g_expire_waits && mbar_wait(bar, parity);
        float2 v[B][16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int i = B * (j + 256 * k);
#pragma unroll
            for (int s = 0; s < B; s += 2) {
                const float4 x = *reinterpret_cast<const float4*>(land + i + s);
                v[s][k] = make_float2(x.x, x.y);
                v[s + 1][k] = make_float2(x.z, x.w);
            }
#pragma unroll
            for (int s = 0; s < B; ++s) {
                if constexpr (W) {
                    if (pre) v[s][k] = cmul(v[s][k], __ldg(pre + i + s));
                }
                if (INV) v[s][k] = swap_ri(v[s][k]);
            }
        }
        if (__syncthreads_or(!ok)) {
            if (j == 0) {
                *(volatile unsigned*)err = 4u;
                mbar_wait(bar, parity);  // let the copy land before the block's memory is released
            }
            return;
        }
        // every value is in registers: the landing buffer takes the next transform
        if (j == 0 && b + gridDim.x < batch) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(bar, BYTES);
            bulk_load(long_smem, in + ((b + gridDim.x) << LOG_N), BYTES, bar);
        }
        long_stages<B, 0>(v, j, stw, ex);
        // the radix-B stage: butterfly r = j + 256 k, output p at r + 4096 p
        float2* dst = out + (b << LOG_N) + j;
        const float2* tw = stw + Stages<LOG_N>::tw_offset(3) + j;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float2 x[B];
            x[0] = v[0][k];
#pragma unroll
            for (int s = 1; s < B; ++s) x[s] = cmul(v[s][k], __ldg(tw + (s - 1) * 4096 + 256 * k));
            dft<B>(x);
#pragma unroll
            for (int p = 0; p < B; ++p) {
                float2 y = INV ? swap_ri(x[p]) : x[p];
                if constexpr (W) {
                    if (post) y = cmul(y, __ldg(post + j + 256 * k + 4096 * p));
                }
                dst[256 * k + 4096 * p] = y;
            }
        }
    }
}

// ---- host side ----------------------------------------------------------------------------------

bool batched_long_supported(int log2n) { return log2n == 13 || log2n == 14; }

template <int B, int INV, bool W>
static cudaError_t launch_long_w(const float2* in, float2* out, long long batch, const float2* stw, unsigned* err,
                                 cudaStream_t stream, const float2* pre, const float2* post) {
    using G = Long<B>;
    auto kernel = k_batched_long<B, INV, W>;
    static std::atomic<unsigned long long> done{0};
    cudaError_t e = smem_limit((const void*)kernel, G::SMEM, done);
    if (e != cudaSuccess) return e;
    // persistent grid: the blocks that fit on the device at once (per device, computed once)
    static std::atomic<int> grid_of[64];
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    int grid = grid_of[dev & 63].load(std::memory_order_relaxed);
    if (grid == 0) {
        int per_sm = 0, sms = 0;
        if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, G::THREADS, G::SMEM)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        grid = per_sm * sms > 0 ? per_sm * sms : 1;
        grid_of[dev & 63].store(grid, std::memory_order_relaxed);
    }
    if ((long long)grid > batch) grid = (int)batch;
    return launch_kernel<!W>(kernel, dim3((unsigned)grid), G::THREADS, G::SMEM, stream, in, out, batch, stw, err, pre, post);
}

template <int B>
static cudaError_t launch_long_t(const float2* in, float2* out, long long batch, const float2* stw, int inverse,
                                 unsigned* err, cudaStream_t stream, const float2* pre, const float2* post) {
    if (pre || post)
        return inverse ? launch_long_w<B, 1, true>(in, out, batch, stw, err, stream, pre, post)
                       : launch_long_w<B, 0, true>(in, out, batch, stw, err, stream, pre, post);
    return inverse ? launch_long_w<B, 1, false>(in, out, batch, stw, err, stream, nullptr, nullptr)
                   : launch_long_w<B, 0, false>(in, out, batch, stw, err, stream, nullptr, nullptr);
}

cudaError_t launch_batched_long(int log2n, const float2* in, float2* out, long long batch, const float2* stw,
                                int inverse, unsigned* err, cudaStream_t stream, const float2* pre, const float2* post) {
    if (batch <= 0) return cudaSuccess;
    if ((uintptr_t)in & 15) return cudaErrorInvalidValue;  // bulk copies start on 16-byte boundaries
    switch (log2n) {
    case 13: return launch_long_t<2>(in, out, batch, stw, inverse, err, stream, pre, post);
    case 14: return launch_long_t<4>(in, out, batch, stw, inverse, err, stream, pre, post);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace ofb
