// Large batches of 2^15 values per transform in ONE trip through HBM: a cluster of two blocks keeps a
// whole transform on chip.
#include "fft_pair.cuh"
#include "fft_tma.cuh"

namespace ofb {

cudaError_t set_expire_waits_cluster(int on) {
    const int v = on ? 1 : 0;
    return cudaMemcpyToSymbol(g_expire_waits, &v, sizeof v);
}

// n = 256 B, B = 64 Q for a cluster of Q blocks (2^15 = 256 x 128, Q = 2): the two passes of the tuned
// two-pass split, with the same arithmetic on the same values (so the same bits), but the array
// between them goes from block to block through distributed shared memory.
//  - Block r of the cluster transforms columns 64 r .. 64 r + 63 (256 values each, one bulk tensor
//    copy, 128 KiB), 32 values per thread: first one butterfly lane of two columns, after the
//    exchange two adjacent lanes of one column, i.e. results k0, k0 + 1.
//  - Those pairs go, 16 bytes each, to the block that owns row k0 (rows (256 / Q) s .. in block s),
//    into its landing buffer, whose values are in registers by then.
//  - Block s transforms its rows (B values each) two adjacent rows a thread, and stores 16-byte pairs:
//    512 contiguous bytes a warp.
// The next transform's copy is issued when a block has read its rows, half a transform ahead.
// Two cluster barriers a transform: one says that every landing buffer is free (arrived at early, waited
// for late), one that the rows have arrived. The first arrival releases this thread's reads of its
// landing buffer to the peers that overwrite it, and nothing else (cluster_arrive_shared). A block's
// columns are the same for every transform it takes, so the inter-pass factors are computed once per
// launch.
//
// Measured on a B200, warm, against the two passes: 2000 x 2^15 293 us against 351, 512 x 2^15 86
// against 95 (two trips of 268 MB through HBM at the board's power limit). What bounds it: a block's
// load, two transforms and exchanges follow each other (one block an SM, 10.4 us a transform), so it
// needs many transforms per cluster: 160 x 2^15 (three rounds of 72 clusters) 40 us against 29. The same
// with four blocks for 2^16 was slower than two passes (1000 transforms 405 us against 372; 33 clusters
// fit the device, and three quarters of the values cross blocks) and is not built.
template <int Q>
struct Cluster {
    static_assert(Q == 2, "rows of 128 values");
    static constexpr int LOG_Q = 1, LOG_B = 6 + LOG_Q, LOG_N = 8 + LOG_B, B = 1 << LOG_B;
    static constexpr int THREADS = 512, ROWS = 256 / Q, PAIRS = ROWS / 2, TB = B / 16;
    // landing buffer: 256 rows of 64 columns, then row pairs [pair][j1] of 16 bytes; the odd pad
    // spreads the readers, a pair apart, over the banks
    static constexpr int PAD = B + 1;
    static constexpr int EX_OFF = PAIRS * PAD * 16 > 131072 ? PAIRS * PAD * 16 : 131072;
    static constexpr int TW_OFF = EX_OFF + 65536;  // exchange: one 8-byte word per two values
    static constexpr int BAR_OFF = TW_OFF + 64 * 17 * 8;
    static constexpr int SMEM = BAR_OFF + 16;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
// The same for this thread's accesses to its own block's shared memory only: a relaxed arrival orders
// nothing by itself, so the fence before it does, without the full release's wait for this thread's
// writes to global memory (the previous transform's output: 2000 transforms 293 us with the fence, 324 with a full release).
__device__ __forceinline__ void cluster_arrive_shared() {
    asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_map(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

template <int Q, bool INV, bool W>
__global__ void __cluster_dims__(Q, 1, 1) __launch_bounds__(512, 1)
    k_cluster(PassArgs a, const float2* __restrict__ stw_b, const __grid_constant__ CUtensorMap tin, long long batch) {
    using G = Cluster<Q>;
    extern __shared__ __align__(1024) unsigned char cl_smem[];
    const float2* land = reinterpret_cast<const float2*>(cl_smem);
    float2* ex = reinterpret_cast<float2*>(cl_smem + G::EX_OFF);
    float2* tws = reinterpret_cast<float2*>(cl_smem + G::TW_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(cl_smem + G::BAR_OFF);
    unsigned* failed = reinterpret_cast<unsigned*>(cl_smem + G::BAR_OFF + 8);  // a wait of the cluster expired
    const int tid = threadIdx.x;
    unsigned rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int stride = (int)gridDim.x / Q;
    long long t = blockIdx.x / Q;  // the same for the whole cluster; the grid has no more clusters than transforms
    auto load = [&](long long b) {
        mbar_expect_tx(bar, 131072u);
        tma_load_4d(cl_smem, &tin, (int)rank * 64, 0, 0, (int)b, bar);
    };
    if (tid == 0) {
        *failed = 0;
        mbar_init(bar, 1);
        dependent_wait();  // the other threads touch the caller's buffers only after the copy landed
        load(t);
    }
    const float2 *pre = nullptr, *post = nullptr;
    if constexpr (W) pre = a.pre, post = a.post;
    // first pass: loads and stage 0 as lane j of columns 2 p, 2 p + 1; stage 1 as lanes 2 u, 2 u + 1 of
    // column c
    const int p = tid & 31, j = tid >> 5, c = tid & 63, u = tid >> 6;
    // second pass: lane m of rows 2 q, 2 q + 1
    const int q = tid & (G::PAIRS - 1), m = tid / G::PAIRS;
    pass_twiddle_rows<8, 6, 0>(a, rank * 64, tws, tid, G::THREADS);
    const float2 wl[2] = {pass_twiddle_lane<8>(a, rank * 64 + c, 2 * u), pass_twiddle_lane<8>(a, rank * 64 + c, 2 * u + 1)};
    const unsigned rows = smem_u32(cl_smem) + (unsigned)(u * G::PAD + (int)rank * 64 + c) * 16;
    cluster_arrive();  // every block of the cluster runs and has cleared its flag before another sets it
    cluster_wait();
    unsigned parity = 0;
    for (; t < batch; t += stride, parity ^= 1u) {
        const bool ok = !g_expire_waits && mbar_wait(bar, parity);
        float2 v[2][16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(land + (j + 16 * k) * 64 + 2 * p);
            v[0][k] = make_float2(x.x, x.y);
            v[1][k] = make_float2(x.z, x.w);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if constexpr (W) {
                    if (pre) v[i][k] = cmul(v[i][k], __ldg(pre + (j + 16 * k) * G::B + (int)rank * 64 + 2 * p + i));
                }
                if (INV) v[i][k] = swap_ri(v[i][k]);
            }
        }
        if (__syncthreads_or(!ok) && tid == 0) {
            *(volatile unsigned*)a.err = 1u;
            mbar_wait(bar, parity);  // let a late copy land before the memory is reused
#pragma unroll
            for (int s = 0; s < Q; ++s)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_map(smem_u32(failed), s)), "r"(1u) : "memory");
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
        }
        cluster_arrive_shared();  // this thread's reads of the landing buffer are done
        pair_stage<8, 0>(v, j, a.stw);
        {
            float2* w = ex + 16 * j * 32 + p;
            const float* r = reinterpret_cast<const float*>(ex) + 2 * u * 64 + c;
#pragma unroll
            for (int k = 0; k < 16; ++k) w[k * 32] = make_float2(v[0][k].x, v[1][k].x);
            __syncthreads();
            float x[2][16];
#pragma unroll
            for (int k = 0; k < 16; ++k) x[0][k] = r[k * 1024], x[1][k] = r[k * 1024 + 64];
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) w[k * 32] = make_float2(v[0][k].y, v[1][k].y);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) v[0][k] = make_float2(x[0][k], r[k * 1024]), v[1][k] = make_float2(x[1][k], r[k * 1024 + 64]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            stage_compute<8, 1>(v[i], 2 * u + i, a.stw);
#pragma unroll
            for (int k = 0; k < 16; ++k) v[i][k] = cmul(v[i][k], cmul(wl[i], tws[c * 17 + k]));
        }
        cluster_wait();  // every landing buffer is free, every block's flag is final
        if (*(volatile unsigned*)failed) return;  // the same in all blocks; nothing is in flight between them
        // results k0 = 2 u + 16 k, k0 + 1: row pair u + 8 (k mod (16 / Q)) of block k / (16 / Q)
#pragma unroll
        for (int s = 0; s < Q; ++s) {
            const unsigned to = cluster_map(rows, s);
#pragma unroll
            for (int i = 0; i < 16 / Q; ++i) {
                const int k = s * (16 / Q) + i;
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 8 * i * G::PAD * 16), "f"(v[0][k].x),
                             "f"(v[0][k].y), "f"(v[1][k].x), "f"(v[1][k].y)
                             : "memory");
            }
        }
        cluster_arrive();
        cluster_wait();  // the rows have arrived
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(cl_smem + (q * G::PAD + m + G::TB * k) * 16);
            v[0][k] = make_float2(x.x, x.y);
            v[1][k] = make_float2(x.z, x.w);
        }
        __syncthreads();  // the rows are in registers: the landing buffer takes the next transform
        if (tid == 0 && t + stride < batch) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            load(t + stride);
        }
        pair_stage<G::LOG_B, 0>(v, m, stw_b);
        {
            float2* w = ex + 16 * m * G::PAIRS + q;
            const float2* r = ex + m * G::PAIRS + q;
#pragma unroll
            for (int k = 0; k < 16; ++k) w[k * G::PAIRS] = make_float2(v[0][k].x, v[1][k].x);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float2 x = r[k * G::TB * G::PAIRS];
                v[0][k].x = x.x, v[1][k].x = x.y;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) w[k * G::PAIRS] = make_float2(v[0][k].y, v[1][k].y);
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float2 x = r[k * G::TB * G::PAIRS];
                v[0][k].y = x.x, v[1][k].y = x.y;
            }
        }
        pair_stage<G::LOG_B, 1>(v, m, stw_b);
        // output k0 + 256 k1, k1 = m + TB k
        const int o = m * 256 + (int)rank * G::ROWS + 2 * q;
        float2* dst = a.out + (t << G::LOG_N) + o;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float2 y[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                y[i] = INV ? swap_ri(v[i][k]) : v[i][k];
                if constexpr (W) {
                    if (post) y[i] = cmul(y[i], __ldg(post + o + 256 * G::TB * k + i));
                }
            }
            *reinterpret_cast<float4*>(dst + 256 * G::TB * k) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
        }
        // (the next transform writes the exchange buffer only after two block barriers)
    }
}

// ---- host side ----------------------------------------------------------------------------------

template <int Q, bool INV, bool W>
static cudaError_t launch_cluster_w(const PassArgs& a, const float2* stw_b, long long batch, cudaStream_t stream) {
    using G = Cluster<Q>;
    auto kernel = k_cluster<Q, INV, W>;
    static std::atomic<unsigned long long> done{0};
    cudaError_t e = smem_limit((const void*)kernel, G::SMEM, done);
    if (e != cudaSuccess) return e;
    // persistent grid: the clusters that fit on the device at once (per device, computed once)
    static std::atomic<int> clusters_of[64];
    int dev = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    int clusters = clusters_of[dev & 63].load(std::memory_order_relaxed);
    if (clusters == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(Q);
        cfg.blockDim = dim3(G::THREADS);
        cfg.dynamicSmemBytes = G::SMEM;
        if ((e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg)) != cudaSuccess) return e;
        if (clusters < 1) return cudaErrorInvalidConfiguration;
        clusters_of[dev & 63].store(clusters, std::memory_order_relaxed);
    }
    if ((long long)clusters > batch) clusters = (int)batch;
    CUtensorMap tin;
    if (!make_map(&tin, a.in, 0, G::LOG_N, 8, 6, G::LOG_B, (int)batch)) return cudaErrorInvalidValue;
    return launch_kernel<!W>(kernel, dim3((unsigned)(clusters * Q)), G::THREADS, G::SMEM, stream, a, stw_b, tin, batch);
}

cudaError_t launch_cluster(const PassArgs& a, const float2* stw_b, int inverse, long long batch, cudaStream_t stream) {
    if (a.log2n != Cluster<2>::LOG_N) return cudaErrorInvalidValue;
    if (a.pre || a.post)
        return inverse ? launch_cluster_w<2, true, true>(a, stw_b, batch, stream)
                       : launch_cluster_w<2, false, true>(a, stw_b, batch, stream);
    return inverse ? launch_cluster_w<2, true, false>(a, stw_b, batch, stream)
                   : launch_cluster_w<2, false, false>(a, stw_b, batch, stream);
}

}  // namespace ofb
