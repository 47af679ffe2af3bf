// Wide-tile pass kernels (sm_100a): one pass of a two- or three-pass transform by persistent blocks,
// one tile of 2^14 (or two of 2^13) values per SM, with the next tile's bulk tensor copy in flight
// while the current one computes. Same arithmetic as k_pass and k_pass_tma on the same values.
//
// Why beside k_pass_tma (one tile per block, 16 values per thread): its tiles of 2^11 .. 2^12
// values need many blocks per SM to hide their copies, which registers allow only for short columns:
// at 2048 or 4096 values a column, one or two blocks ran and waited. So 2^22 .. 2^24 took three
// passes of short columns over HBM; here two passes of long ones are faster. A thread owns one
// butterfly lane of TWO adjacent columns, 32 values: it loads each stage twiddle once for both,
// moves 16-byte pieces from the landing buffer and to strided outputs, and 8-byte words (two columns'
// re parts, then their im parts) through the exchange buffer, which with half the bytes per round
// leaves the room for the landing buffer. The first pass regroups its threads in the last exchange,
// so that it stores contiguous runs straight from registers (k_pass_tma transposes once more).
//
// What bounds it (B200, a pass over 2^24 values, 268 MB moved, 41 us at the copy rate): the tile's
// load, arithmetic and store between the block's barriers. First pass, columns x values: 2 x 4096
// 65 us, 4 x 2048 59, 8 x 1024 56, 16 x 512 52, 32 x 256 50; last pass 4 x 4096 69 (without its
// 32-byte store pieces 61), 8 x 2048 62, 16 x 1024 60, 16 x 512 50. Loads and stores alone, no
// arithmetic: 58, 50, 48, 48, 46; 55, 52, 50, 45. Sustained, the HBM traffic of a plain copy alone draws
// the board's 1000 W, so arithmetic beside it lowers the clock: fewer passes pay twice.
//
// Measured and left out: inter-pass powers shared by the block (the extra latency costs what the
// FP64 work saves), stage twiddles loaded before the exchange that precedes their stage (no
// change), strided last passes of 8 columns at strides of 512 KiB and more (64-byte pieces: 2^27
// 1478 us; 1213 with 16 columns).
#include "fft_pair.cuh"
#include "fft_tma.cuh"

namespace ofb {

cudaError_t set_expire_waits_wide(int on) {
    const int v = on ? 1 : 0;
    return cudaMemcpyToSymbol(g_expire_waits, &v, sizeof v);
}

// Geometry of a tile of C = 2^LOG_C columns of L = 2^LOG_L values. A thread owns one of the T = L / 16
// butterfly lanes of TWO adjacent columns: it loads each stage twiddle once for both, and moves the
// two columns' re (then im) parts through the exchange buffer as one 8-byte word.
template <int LOG_L, int LOG_C>
struct Wide {
    static constexpr int L = 1 << LOG_L, C = 1 << LOG_C, P = C / 2, T = L / 16, THREADS = T * P;
    static constexpr int VALUES = L * C;
    // Exchange buffer, in 8-byte words: rows [e][p] of the column pairs with one pad row every 16, or
    // whole columns [p][e] for the exchange that regroups the threads by column (padded alike, and
    // offset so that the writers, 16 / P lanes of each pair, meet distinct banks).
    static constexpr int COL = L + L / 16 + 16 / P;
    static_assert(P <= 16 && (L / 16) % 16 == 0, "bank layout");
    static constexpr int ROW_WORDS = (L + L / 16) * P, COL_WORDS = COL * P;
    static constexpr int EX_WORDS = ROW_WORDS > COL_WORDS ? ROW_WORDS : COL_WORDS;
    static constexpr int EX_OFF = 8 * VALUES;                     // bytes; the landing buffer comes first
    static constexpr int TW_OFF = EX_OFF + 8 * EX_WORDS;          // 2 x C x 17 inter-pass factors
    static constexpr int BAR_OFF = TW_OFF + 2 * C * 17 * 8;
    static constexpr int SMEM = BAR_OFF + 16;
};

// The exchange between stages S and S + 1 (tile_fft's): output p of lane j goes to element
// E0(j) + p Ns of pair c, and element jr + T k of pair cr is read back, re and im parts one after
// the other. COLUMNS: the buffer holds whole columns, so that the readers can run along a column
// where the writers ran across columns. The block has been synchronised since the buffer was last
// read.
template <int LOG_L, int LOG_C, int S, bool COLUMNS>
__device__ __forceinline__ void pair_exchange(float2 (&v)[2][16], int j, int c, int jr, int cr, float2* ex) {
    using G = Wide<LOG_L, LOG_C>;
    constexpr int LNS = Stages<LOG_L>::log2_ns(S), NS = 1 << LNS;
    constexpr int STEP = COLUMNS ? 1 : G::P;
    const int e0 = ((j >> LNS) << (4 + LNS)) + (j & (NS - 1));
    float2* w = ex + (COLUMNS ? c * G::COL + spad(e0) : spad(e0) * STEP + c);
    const float2* r = ex + (COLUMNS ? cr * G::COL + spad(jr) : spad(jr) * STEP + cr);
#pragma unroll
    for (int p = 0; p < 16; ++p) w[padc(p * NS) * STEP] = make_float2(v[0][p].x, v[1][p].x);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 x = r[padc(k * G::T) * STEP];
        v[0][k].x = x.x, v[1][k].x = x.y;
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 16; ++p) w[padc(p * NS) * STEP] = make_float2(v[0][p].y, v[1][p].y);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 x = r[padc(k * G::T) * STEP];
        v[0][k].y = x.x, v[1][k].y = x.y;
    }
}

// Stages S .. of the tile; the last one runs on lane jl of pair cl.
template <int LOG_L, int LOG_C, int S, bool REGROUP>
__device__ __forceinline__ void pair_stages(float2 (&v)[2][16], int j, int c, int jl, int cl,
                                            const float2* __restrict__ stw, float2* ex) {
    constexpr int COUNT = Stages<LOG_L>::COUNT;
    pair_stage<LOG_L, S>(v, S + 1 == COUNT ? jl : j, stw);
    if constexpr (S + 1 < COUNT) {
        constexpr bool TO_LAST = S + 2 == COUNT;
        if constexpr (S > 0) __syncthreads();  // the previous exchange's reads are done
        pair_exchange<LOG_L, LOG_C, S, TO_LAST && REGROUP>(v, j, c, TO_LAST ? jl : j, TO_LAST ? cl : c, ex);
        pair_stages<LOG_L, LOG_C, S + 1, REGROUP>(v, j, c, jl, cl, stw, ex);
    }
}

// SWAP: the first pass exchanges re/im on load, the last on store. W: the first pass multiplies its input by
// PassArgs::pre (not NULL). X: a
// pass of a column transform (PassArgs' column fields, as tma_tile; re/im exchanges at run time): the
// tile of a.in, the column factors, and the first pass with colstore or the last pass writing the
// column layout.
template <int LOG_L, int LOG_C, int MODE, bool SWAP, bool W, bool X = false>
__global__ void __launch_bounds__(Wide<LOG_L, LOG_C>::THREADS, LOG_L + LOG_C >= 14 ? 1 : LOG_L + LOG_C == 13 ? 2 : 4)
    k_pass_wide(PassArgs a, const __grid_constant__ CUtensorMap tin, unsigned tiles, int log_tiles) {
    using G = Wide<LOG_L, LOG_C>;
    extern __shared__ __align__(1024) unsigned char wide_smem[];
    const float2* land = reinterpret_cast<const float2*>(wide_smem);
    float2* ex = reinterpret_cast<float2*>(wide_smem + G::EX_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(wide_smem + G::BAR_OFF);
    const int tid = threadIdx.x;
    if (smem_u32(wide_smem) & 127) {  // bulk tensor copies need a 128-byte aligned destination
        if (tid == 0) *(volatile unsigned*)a.err = 2u;
        return;
    }
    // loads, first stages and strided stores run across the columns, contiguous stores along them
    const int c = tid & (G::P - 1), j = tid / G::P;
    const int cl = MODE == 0 ? tid / G::T : c, jl = MODE == 0 ? tid & (G::T - 1) : j;
    auto load = [&](unsigned t) {
        const int b = (int)(t >> log_tiles);
        const unsigned col0 = (t & ((1u << log_tiles) - 1)) << LOG_C;
        mbar_expect_tx(bar, (unsigned)(G::VALUES * sizeof(float2)));
        if (MODE == 0) tma_load_4d(wide_smem, &tin, (int)col0, 0, 0, b, bar);
        else tma_load_5d(wide_smem, &tin, (int)(col0 & ((1u << a.log_s) - 1)), 0, 0, (int)(col0 >> a.log_s), b, bar);
    };
    unsigned t = blockIdx.x, parity = 0;
    if (t >= tiles) return;
    if (tid == 0) {
        mbar_init(bar, 1);
        dependent_wait();  // the other threads touch the caller's buffers only after the copy landed
        load(t);
    }
    if constexpr (W) dependent_wait();  // every thread reads the caller's weights
    __syncthreads();  // the barrier is initialised before anyone waits on it
    for (; t < tiles; t += gridDim.x, parity ^= 1u) {
        const unsigned col0 = (t & ((1u << log_tiles) - 1)) << LOG_C;
        const long long toff = (long long)(t >> log_tiles) << a.log2n;
        // inter-pass factors (as pass_tile) while the copy is in flight; the rows alternate between
        // two buffers, since slower threads may still read the previous tile's
        float2* tws = reinterpret_cast<float2*>(wide_smem + G::TW_OFF) + parity * (G::C * 17);
        float2 wl[2];
        bool twiddled = MODE != 2;
        if constexpr (X) {
            twiddled = a.tw_lo != nullptr;  // the same for the whole block
            if (twiddled) {
                column_twiddle_rows<LOG_L, LOG_C, MODE>(a, col0, tws, tid, G::THREADS);
                wl[0] = column_twiddle_lane<LOG_L, MODE>(a, col0, 2 * cl, jl);
                wl[1] = column_twiddle_lane<LOG_L, MODE>(a, col0, 2 * cl + 1, jl);
            }
        } else if (MODE != 2) {
            pass_twiddle_rows<LOG_L, LOG_C, MODE>(a, col0, tws, tid, G::THREADS);
            const unsigned f = MODE == 0 ? col0 + 2 * cl : (col0 >> a.log_s) << a.log_s;
            wl[0] = pass_twiddle_lane<LOG_L>(a, f, jl);
            wl[1] = MODE == 0 ? pass_twiddle_lane<LOG_L>(a, f + 1, jl) : wl[0];
        }
        float2 v[2][16];
        if constexpr (W) {  // the weights first, in the registers of the values they multiply
            const float2* w = a.pre + col0 + 2 * c + ((unsigned)j << a.log_s);
            const unsigned step = (unsigned)G::T << a.log_s;
            if (((uintptr_t)a.pre & 15) == 0) {
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const float4 x = ld_stream4(w + k * step);
                    v[0][k] = make_float2(x.x, x.y);
                    v[1][k] = make_float2(x.z, x.w);
                }
            } else {
#pragma unroll
                for (int k = 0; k < 16; ++k) v[0][k] = ld_stream(w + k * step), v[1][k] = ld_stream(w + k * step + 1);
            }
        }
        const bool ok = !g_expire_waits && mbar_wait(bar, parity);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(land + (j + G::T * k) * G::C + 2 * c);
            if constexpr (W) {
                v[0][k] = cmul(make_float2(x.x, x.y), v[0][k]);
                v[1][k] = cmul(make_float2(x.z, x.w), v[1][k]);
            } else {
                v[0][k] = make_float2(x.x, x.y);
                v[1][k] = make_float2(x.z, x.w);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (X ? a.swap_in : SWAP && MODE == 0) v[i][k] = swap_ri(v[i][k]);
            }
        }
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                *(volatile unsigned*)a.err = 1u;
                mbar_wait(bar, parity);  // let a late copy land before the memory is released
            }
            return;
        }
        // every value is in registers: the landing buffer takes the next tile
        if (tid == 0 && t + gridDim.x < tiles) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            load(t + gridDim.x);
        }
        pair_stages<LOG_L, LOG_C, 0, MODE == 0>(v, j, c, jl, cl, a.stw, ex);
        if (twiddled) {
            const float2* tw = tws + (MODE == 0 ? 2 * cl * 17 : 0);
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                v[0][k] = cmul(v[0][k], cmul(wl[0], tw[k]));
                v[1][k] = cmul(v[1][k], cmul(wl[1], tw[MODE == 0 ? 17 + k : k]));
            }
        }
        // Column layout (column_dst), for blocks of at least the 16th part of the output's extent: output
        // k + (16th part) i of transform b goes to its block's row b, i's part of the offset being the
        // same for all threads.
        const int log_part = LOG_L - 4 + (MODE == 0 ? 0 : a.log_s);
        auto part = [&](int i) {
            const unsigned long long k = (unsigned long long)i << log_part;
            return ((k >> a.xlog_blk) << (a.xlog_cols + a.xlog_blk)) + (k & ((1ull << a.xlog_blk) - 1));
        };
        if (X && MODE == 0 && a.colstore) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float2* q = a.out + ((unsigned long long)(col0 + 2 * cl + i) << a.xlog_blk) + jl;
#pragma unroll
                for (int k = 0; k < 16; ++k) q[part(k)] = a.swap_out ? swap_ri(v[i][k]) : v[i][k];
            }
        } else if (MODE == 0) {
            // contiguous column runs at their digit-reversed place, as k_pass
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const unsigned rr = col0 + 2 * cl + i, j2 = rr & ((1u << a.rev_b2) - 1), j1 = rr >> a.rev_b2;
                float2* q = a.out + toff + (((j1 + (j2 << a.rev_b1)) << LOG_L) + jl);
#pragma unroll
                for (int k = 0; k < 16; ++k) q[G::T * k] = v[i][k];
            }
        } else {
            const unsigned q0 = col0 & ((1u << a.log_s) - 1), h = col0 >> a.log_s;
            const unsigned base = q0 + 2 * c + (h << (a.log_s + LOG_L));
            float2* qx = X ? a.out + ((unsigned long long)h << a.xlog_blk) + q0 + 2 * c + ((unsigned)j << a.log_s) : nullptr;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const unsigned e = base + ((unsigned)(j + G::T * k) << a.log_s);
                float2 y[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) y[i] = (X ? a.swap_out : SWAP && MODE == 2) ? swap_ri(v[i][k]) : v[i][k];
                *reinterpret_cast<float4*>(X ? qx + part(k) : a.out + toff + e) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
            }
        }
    }
}

template <int LOG_L, int LOG_C, int MODE, bool SWAP, bool W, bool X = false>
static cudaError_t launch_wide_w(const PassArgs& a, int batch, cudaStream_t stream) {
    using G = Wide<LOG_L, LOG_C>;
    auto kernel = k_pass_wide<LOG_L, LOG_C, MODE, SWAP, W, X>;
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
    CUtensorMap tin;
    if (!make_map(&tin, MODE == 0 || X ? a.in : a.out, MODE, a.log2n, LOG_L, LOG_C, a.log_s, batch))
        return cudaErrorInvalidValue;
    const int log_tiles = a.log2n - LOG_L - LOG_C;
    const unsigned tiles = (unsigned)batch << log_tiles;
    if ((unsigned)grid > tiles) grid = (int)tiles;
    return launch_kernel<true>(kernel, dim3((unsigned)grid), G::THREADS, G::SMEM, stream, a, tin, tiles, log_tiles);
}

// Weights cost a persistent block of one tile an SM more than the small blocks of k_pass_tma: their 16- to
// 64-byte row pieces arrive by per-thread loads, which nothing overlaps but the tile's own copy. First passes of
// up to 2^10 values take them (128-byte pieces, loaded while the copy is in flight); longer first passes and all
// last ones go to k_pass_tma. Wide against k_pass_tma for the weighted pass, us (B200, warm): input weights,
// 16 x 2^21 299 / 288, 2^22 48.1 / 43.0, 4 x 2^23 424 / 351, 2^24 224 / 190 (2^20, which stays: 32 x 255 / 266);
// output weights, 64 x 2^19 283 / 238, 32 x 2^20 298 / 268, 16 x 2^21 322 / 290, 2^22 48.5 / 43.4, 2^23 107 / 92,
// 2^24 221 / 201, 2^28 3392 / 3367.
constexpr int kWideWeightsLog2 = 10;
bool pass_wide_weights(int mode, int log_l, const PassArgs& a) {
    return mode == 0 ? !a.pre || log_l <= kWideWeightsLog2 : mode == 1 || !a.post;
}

template <int LOG_L, int LOG_C, int MODE>
static cudaError_t launch_wide_t(const PassArgs& a, int batch, cudaStream_t stream) {
    const bool swap = MODE == 0 ? a.swap_in : a.swap_out;
    if constexpr (MODE == 0 && LOG_L <= kWideWeightsLog2) {
        if (a.pre)
            return swap ? launch_wide_w<LOG_L, LOG_C, MODE, true, true>(a, batch, stream)
                        : launch_wide_w<LOG_L, LOG_C, MODE, false, true>(a, batch, stream);
    }
    if (!pass_wide_weights(MODE, LOG_L, a)) return cudaErrorInvalidValue;
    if constexpr (MODE != 1) {
        if (swap) return launch_wide_w<LOG_L, LOG_C, MODE, true, false>(a, batch, stream);
    }
    return launch_wide_w<LOG_L, LOG_C, MODE, false, false>(a, batch, stream);
}

// Tile shapes (log2 values, log2 columns) with a wide kernel, by pass: those the tuned table uses.
#define OFB_WIDE_FIRST(X) X(12, 1) X(11, 2) X(10, 4) X(10, 3) X(9, 4)
#define OFB_WIDE_MIDDLE(X) X(10, 4) X(9, 4)
#define OFB_WIDE_LAST(X) X(12, 2) X(11, 3) X(10, 4) X(10, 3) X(8, 4)

cudaError_t launch_pass_wide(int mode, int log_l, int log_c, const PassArgs& a, int batch, cudaStream_t stream) {
#define OFB_WIDE_CASE0(LL, LC) \
    if (mode == 0 && log_l == LL && log_c == LC) return launch_wide_t<LL, LC, 0>(a, batch, stream);
#define OFB_WIDE_CASE1(LL, LC) \
    if (mode == 1 && log_l == LL && log_c == LC) return launch_wide_t<LL, LC, 1>(a, batch, stream);
#define OFB_WIDE_CASE2(LL, LC) \
    if (mode == 2 && log_l == LL && log_c == LC) return launch_wide_t<LL, LC, 2>(a, batch, stream);
    OFB_WIDE_FIRST(OFB_WIDE_CASE0)
    OFB_WIDE_MIDDLE(OFB_WIDE_CASE1)
    OFB_WIDE_LAST(OFB_WIDE_CASE2)
#undef OFB_WIDE_CASE0
#undef OFB_WIDE_CASE1
#undef OFB_WIDE_CASE2
    return cudaErrorInvalidValue;
}

// ---- column transforms ----------------------------------------------------------------------------

// Tile width (log2 columns) of a column-transform pass, -1: none. First passes of 2^8 .. 2^10 values stay
// with k_pass_tma, whose regrouped tiles are faster at the full clock (B200, 2^27 values, one pass of
// 2^10 418 us against 453, 2^9 401 against 437) and level at the power-limited one (498 / 492, 473 / 476).
// The others, wide against k_pass_tma's, power-limited: one pass of 2^11 572 -> 513 us, 2^12 619 -> 563
// (555 -> 494 at the full clock), two passes with a wide second one 2^18 930 -> 885, 2^20 1008 -> 914 (863 ->
// 822). Last passes of 2^8 and 2^9 values take tiles of 32 and 16 columns, which leave SMs idle on
// small matrices: from 2^25 values on.
static constexpr int column_wide_log_c(int mode, int log_l) {
    return log_l == 12 ? (mode == 0 ? 1 : 2) : log_l == 11 ? (mode == 0 ? 2 : 3) : mode == 0 ? -1
           : log_l == 10 ? 4 : log_l == 9 ? 4 : log_l == 8 ? 5 : -1;
}

bool pass_columns_wide_supported(int mode, int log_l, const PassArgs& a) {
    const int c = column_wide_log_c(mode, log_l);
    return c >= 0 && (log_l >= 10 || a.log2n >= 25) && a.log2n >= log_l + c && (mode == 0 || a.log_s >= c) &&
           (!a.colstore || a.xlog_blk >= log_l - 4 + (mode == 0 ? 0 : a.log_s)) && ((uintptr_t)a.out & 15) == 0;
}

cudaError_t launch_pass_columns_wide(int mode, int log_l, const PassArgs& a, cudaStream_t stream) {
#define OFB_WIDE_COLUMNS(LL, M) \
    if (log_l == LL && mode == M) return launch_wide_w<LL, column_wide_log_c(M, LL), M, false, false, true>(a, 1, stream);
    OFB_WIDE_COLUMNS(12, 0)
    OFB_WIDE_COLUMNS(11, 0)
    OFB_WIDE_COLUMNS(12, 2)
    OFB_WIDE_COLUMNS(11, 2)
    OFB_WIDE_COLUMNS(10, 2)
    OFB_WIDE_COLUMNS(9, 2)
    OFB_WIDE_COLUMNS(8, 2)
#undef OFB_WIDE_COLUMNS
    return cudaErrorInvalidValue;
}

}  // namespace ofb
