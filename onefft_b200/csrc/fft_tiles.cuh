// Tile bodies shared by the stand-alone kernels (fft_kernels.cu) and the persistent uneven-batch
// kernel (uneven.cu): the same arithmetic in both, so an uneven batch reproduces the plain
// per-size path.
#pragma once

#include "fft_device.cuh"
#include "fft_launch.h"
#include "fft_tc.cuh"

namespace ofb {

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}

// w_n^t for t < n from the two-level tables, in FP64.
__device__ __forceinline__ double2 big_twiddle_f64(const double2* __restrict__ lo, const double2* __restrict__ hi,
                                                   int lo_bits, unsigned t) {
    return zmul(__ldg(lo + (t & ((1u << lo_bits) - 1))), __ldg(hi + (t >> lo_bits)));
}

// w^e for e < 2^BITS by square-and-multiply in FP64. With w from the two-level tables (error
// ~1e-16), the result is within ~BITS * 2^(BITS+1) * 1e-16 of exact, far below FP32 rounding.
template <int BITS>
__device__ __forceinline__ double2 zpow(double2 w, unsigned e) {
    double2 r = make_double2(1.0, 0.0);
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        if ((e >> b) & 1u) r = zmul(r, w);
        if (b + 1 < BITS) w = zmul(w, w);
    }
    return r;
}

// Inter-pass twiddles of a pass tile: output j + T kk of a column with factor F (first pass:
// the column index; middle pass: S h) is multiplied by w_n^(F j) * w_n^(F T kk), each factor
// rounded once to FP32. Both factors are powers of ONE table product per column (w_n^F and
// w_n^(F T)), so a tile reads the FP64 tables at C addresses instead of once per factor.
// The 16 factors w_n^(F T kk) of each column go to shared memory (rows of 17).
template <int LOG_L, int LOG_C, int MODE>
__device__ __forceinline__ void pass_twiddle_rows(const PassArgs& a, unsigned col0, float2* tws, int tid, int nthreads) {
    constexpr unsigned T = 1u << (LOG_L - 4);
    constexpr int C = 1 << LOG_C;
    const unsigned hs = (col0 >> a.log_s) << a.log_s;
    for (int i = tid; i < (MODE == 0 ? C : 1) * 16; i += nthreads) {
        const int cc = i >> 4, kk = i & 15;
        const unsigned f = MODE == 0 ? col0 + cc : hs;
        const double2 w = zpow<4>(big_twiddle_f64(a.tw_lo, a.tw_hi, a.lo_bits, f * T), (unsigned)kk);
        tws[cc * 17 + kk] = make_float2((float)w.x, (float)w.y);
    }
}
// ... and the thread's own factor w_n^(F j).
template <int LOG_L>
__device__ __forceinline__ float2 pass_twiddle_lane(const PassArgs& a, unsigned f, int j) {
    const double2 w = zpow<LOG_L - 4>(big_twiddle_f64(a.tw_lo, a.tw_hi, a.lo_bits, f), (unsigned)j);
    return make_float2((float)w.x, (float)w.y);
}

// Column transforms (PassArgs' column fields): w_N^t, N = 2^a.xlog2n <= 2^40, for any 64-bit t
// (reduced mod N; unsigned products wrap mod 2^64, a multiple of N).
__device__ __forceinline__ double2 wide_twiddle_f64(const PassArgs& a, unsigned long long t) {
    t &= (1ull << a.xlog2n) - 1;
    return zmul(__ldg(a.tw_lo + (t & ((1ull << a.lo_bits) - 1))), __ldg(a.tw_hi + (t >> a.lo_bits)));
}
// The factors of a column-transform tile, split like the inter-pass twiddles above (one FP32
// rounding per factor). First pass: output j + T kk of column col gets w_N^(F (j + T kk)),
// F = xcol0 + (col >> tw_shift): rows w_N^(F T kk) per column, lane w_N^(F j). Last pass: output
// k = q + 2^log_s (j + T kk) of transform h = col >> log_s (q = col mod 2^log_s) gets
// w_N^((xcol0 + h) k): rows w_N^((xcol0 + h) 2^log_s T kk), one per tile (a tile's columns share
// h), lane w_N^((xcol0 + h)(q + 2^log_s j)).
template <int LOG_L, int LOG_C, int MODE>
__device__ __forceinline__ void column_twiddle_rows(const PassArgs& a, unsigned col0, float2* tws, int tid, int nthreads) {
    constexpr unsigned long long T = 1ull << (LOG_L - 4);
    constexpr int C = 1 << LOG_C;
    for (int i = tid; i < (MODE == 0 ? C : 1) * 16; i += nthreads) {
        const int cc = i >> 4, kk = i & 15;
        const unsigned long long step = MODE == 0 ? (a.xcol0 + ((col0 + cc) >> a.tw_shift)) * T
                                                  : ((a.xcol0 + (col0 >> a.log_s)) << a.log_s) * T;
        const double2 w = zpow<4>(wide_twiddle_f64(a, step), (unsigned)kk);
        tws[cc * 17 + kk] = make_float2((float)w.x, (float)w.y);
    }
}
template <int LOG_L, int MODE>
__device__ __forceinline__ float2 column_twiddle_lane(const PassArgs& a, unsigned col0, int c, int j) {
    double2 w;
    if (MODE == 0) {
        w = zpow<LOG_L - 4>(wide_twiddle_f64(a, a.xcol0 + ((col0 + c) >> a.tw_shift)), (unsigned)j);
    } else {
        const unsigned long long f = a.xcol0 + (col0 >> a.log_s);
        const unsigned long long q = (col0 & ((1u << a.log_s) - 1)) + c;
        w = wide_twiddle_f64(a, f * (q + ((unsigned long long)j << a.log_s)));
    }
    return make_float2((float)w.x, (float)w.y);
}
// Destination of output k of transform b in the column layout (PassArgs::colstore).
__device__ __forceinline__ long long column_dst(const PassArgs& a, unsigned long long b, unsigned long long k) {
    return (long long)(((((k >> a.xlog_blk) << a.xlog_cols) + b) << a.xlog_blk) + (k & ((1ull << a.xlog_blk) - 1)));
}

// Loads of the caller's data, through L2 only. The next kernel of the stream may be resident on this SM
// already (dependent_launch) and reads its input once dependent_wait() has returned; if a block of this
// kernel, or of one before it, had left a copy of that 32-byte sector in this SM's L1 before another SM
// wrote the sector, the read could find the copy. That takes a kernel that reads and writes one
// sector: the in-place passes on buffers that are only 8-byte aligned, an input that ends or begins
// in the sector where the output begins or ends. Whether the wait alone discards such copies is not
// established here; with no such data in L1 it does not matter. Volatile: none moves above the wait.
// ld_cached is for kernels whose SMs hold no older copy: ordinary launches, and the uneven kernel, which
// fences after its wait. They gain from L1 where a warp reads pieces shorter than a line.
// Pointwise weights of the one-kernel sizes are read by every block and belong in L1 (through L2 only, a
// batch of 2^24 values in transforms of 4 took 234 us instead of 52, in transforms of 2^14 154 instead of
// 94): they are __ldg loads, and those kernels are launched as ordinary successors (launch_kernel<false>).
// A pass reads each weight once per transform: ld_stream.
__device__ __forceinline__ float2 ld_stream(const float2* p) {
    float2 v;
    asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_stream4(const float2* p) {  // 16-byte aligned
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_cached(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
// The array between passes may be kept in L2 for the next pass (evict last).
__device__ __forceinline__ unsigned long long policy_evict_last() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void st_policy(float2* p, float2 v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(v.x), "f"(v.y), "l"(pol)
                 : "memory");
}

// Bounded wait until *p >= target (acquire at GPU scope), for counters that other blocks of the
// same launch advance: ~1 us per poll, about a second in all.
constexpr unsigned kCountWaitLimit = 1u << 20;
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned target) {
    for (unsigned i = 0; i < kCountWaitLimit; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= target) return true;
        __nanosleep(128);
    }
    return false;
}

// As wait_count, also giving up as soon as *abort is non-zero (another block's wait ran out).
__device__ __forceinline__ bool wait_count_or_abort(const unsigned* p, unsigned target, const unsigned* abort) {
    for (unsigned i = 0; i < kCountWaitLimit; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        if (v >= target) return true;
        if (*(const volatile unsigned*)abort) return false;
        __nanosleep(128);
    }
    return false;
}

// Shared memory (bytes) of a tile of 2^log_c columns of length 2^log_l, with padding.
__host__ __device__ constexpr int smem_bytes(int log_l, int log_c) {
    return (int)sizeof(float2) * ((1 << (log_l + log_c)) + (1 << (log_l + log_c - 4)));
}
// Slots (float2) of a pass tile's exchange memory: a first pass of two or more stages regroups its
// threads in its last exchange (tile_fft_regroup).
__host__ __device__ constexpr bool pass_regroups(int log_l, int mode) { return mode == 0 && log_l > 4; }
__host__ __device__ constexpr int pass_slots(int log_l, int log_c, int mode) {
    return pass_regroups(log_l, mode) ? regroup_slots(log_l, log_c) : (1 << (log_l + log_c)) + (1 << (log_l + log_c - 4));
}
// Shared memory of a pass tile: the exchange memory plus the inter-pass twiddle factors (17 per column).
__host__ __device__ constexpr int pass_smem_bytes(int log_l, int log_c, int mode) {
    return (int)sizeof(float2) * (pass_slots(log_l, log_c, mode == 2 ? 2 : 0) + (mode == 2 ? 0 : 17 * (1 << log_c)));
}

// ---- n <= 8: one transform per thread -------------------------------------------------------------

// W: pointwise weights of the input and output (either pointer NULL), out = post * T(pre * in);
// without W the weights are not compiled in at all.
template <int LOG_N, bool W = false>
__device__ __forceinline__ void tiny_transform(const float2* __restrict__ src, float2* __restrict__ dst, int inverse,
                                               const float2* __restrict__ pre = nullptr,
                                               const float2* __restrict__ post = nullptr) {
    constexpr int N = 1 << LOG_N;
    float2 a[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        a[i] = ld_cached(src + i);
        if constexpr (W) {
            if (pre) a[i] = cmul(a[i], __ldg(pre + i));
        }
        if (inverse) a[i] = swap_ri(a[i]);
    }
    dft<N>(a);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float2 y = inverse ? swap_ri(a[i]) : a[i];
        if constexpr (W) {
            if (post) y = cmul(y, __ldg(post + i));
        }
        dst[i] = y;
    }
}

// ---- one block of whole transforms, n = 16 .. 2^14 --------------------------------------------------
//
// 2^LOG_C transforms of length L = 2^LOG_L, 16 values per thread, thread tid owns column
// c = tid / (L/16) and butterfly lane j = tid mod (L/16). src / dst point at this thread's
// transform; inactive columns (past the end of a batch) compute on zeros and store nothing.
// TC: 0 = FP32 stages; 3 or 6 = the split-BF16 tensor-core stages with that many product terms
// (fft_tc.cuh). W, pre, post as tiny_transform. L1: the loads may be cached there (ld_cached).
template <int LOG_L, int LOG_C, bool L1, int TC = 0, bool W = false>
__device__ __forceinline__ void batched_tile(const float2* __restrict__ src, float2* __restrict__ dst, bool active,
                                             int inverse, const float2* __restrict__ stw, float2* smem, int tid,
                                             const float2* __restrict__ pre = nullptr,
                                             const float2* __restrict__ post = nullptr) {
    constexpr int L = 1 << LOG_L, T = L / 16;
    const int j = tid & (T - 1);
    const int c = tid >> (LOG_L - 4);
    src += j;
    dst += j;
    float2 v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) 
        v[k] = !active ? make_float2(0.f, 0.f) : L1 ? ld_cached(src + T * k) : ld_stream(src + T * k);
    if constexpr (W) {  // after all loads: a test of `pre` between them would keep them apart
        if (pre) {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = cmul(v[k], __ldg(pre + j + T * k));
        }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = inverse ? swap_ri(v[k]) : v[k];
    if constexpr (TC != 0) tile_fft_tc<LOG_L, LOG_C, 1, TC>(v, j, stw, smem, c << LOG_L, tid);
    else tile_fft<LOG_L, 1>(v, j, stw, smem, c << LOG_L);
    if (active) {
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float2 y = inverse ? swap_ri(v[k]) : v[k];
            if constexpr (W) {
                if (post) y = cmul(y, __ldg(post + j + T * k));
            }
            dst[T * k] = y;
        }
    }
}

// ---- one tile of a pass of the multi-pass decomposition -----------------------------------------
//
// MODE 0: first pass, in -> out with digit-reversed contiguous column runs and w_n^(r k).
// MODE 1: middle pass, in place on out, twiddle w_n^((h k) S).
// MODE 2: last pass, in place on out, no twiddle.
// Tile t covers 2^LOG_C adjacent columns of the transform at element offset `toff`; tid runs
// over the 2^LOG_C L / 16 threads of the tile.
// W: the first pass multiplies its input by a.pre, the last pass its output by a.post (see
// PassArgs; the pointer the pass uses is not NULL); without W they are not compiled in.
// CG: later passes load through L2 only (ld_stream), for data that other blocks may have written while
// this SM's L1 holds an older copy.
// X: a pass of a column transform (PassArgs' column fields): MODE 0 takes its inter-pass factor
// from the column fields and, with colstore, writes the column layout (and a.swap_out: it is
// then the only pass); MODE 2 reads a.in, multiplies by the larger transform's factors and
// writes the column layout to a.out. One matrix per launch (toff 0).
template <int LOG_L, int LOG_C, int MODE, int TC = 0, bool W = false, bool CG = false, bool X = false>
__device__ __forceinline__ void pass_tile(const PassArgs& a, unsigned t, long long toff, float2* smem, int tid) {
    constexpr int L = 1 << LOG_L, T = L / 16, C = 1 << LOG_C;
    const int c = tid & (C - 1);
    const int j = tid >> LOG_C;
    const unsigned col0 = a.tli >= 31 ? (t << LOG_C)
                                      : ((a.outer_base + (t >> a.tli)) << a.outer_shift) + a.inner_base +
                                            ((t & ((1u << a.tli) - 1)) << LOG_C);
    unsigned base;  // element e of this thread's column is at base + (e << a.log_s)
    if (MODE == 0) {
        base = col0 + c;
    } else {
        unsigned q = (col0 & ((1u << a.log_s) - 1)) + c;
        unsigned h = col0 >> a.log_s;
        base = q + (h << (a.log_s + LOG_L));
    }
    // Inter-pass twiddles w_n^(F (j + T kk)) for this thread's outputs, F = r (first pass,
    // per column) or S h (middle pass, per tile), split as w^(F j) * w^(F T kk): the factors
    // w^(F T kk) of each column in shared memory (rows padded to 17 so the columns of a warp hit
    // distinct banks), w^(F j) per thread; each rounded once to FP32, their product applied in
    // FP32 (pass_twiddle_rows / pass_twiddle_lane).
    // REGROUP: after the last exchange the thread holds lane jl of column cl.
    constexpr bool REGROUP = pass_regroups(LOG_L, MODE) && TC == 0;
    const int cl = REGROUP ? tid >> (LOG_L - 4) : c, jl = REGROUP ? tid & (T - 1) : j;
    float2* tws = smem + pass_slots(LOG_L, LOG_C, MODE);
    float2 wjf = make_float2(1.f, 0.f);
    bool twiddled = MODE != 2;
    if constexpr (X) {
        twiddled = MODE != 1 && a.tw_lo != nullptr;  // the same for the whole block
        if (twiddled) {
            column_twiddle_rows<LOG_L, LOG_C, MODE>(a, col0, tws, tid, C * T);
            wjf = column_twiddle_lane<LOG_L, MODE>(a, col0, cl, jl);
        }
    } else if (MODE != 2) {
        pass_twiddle_rows<LOG_L, LOG_C, MODE>(a, col0, tws, tid, C * T);
        wjf = pass_twiddle_lane<LOG_L>(a, MODE == 0 ? col0 + cl : (col0 >> a.log_s) << a.log_s, jl);
    }
    dependent_wait();  // (the uneven kernel has waited already)
    // element j + T k of the column: p0 + k * estep
    const long long estep = (long long)T << a.log_s;
    const long long off0 = toff + base + ((long long)j << a.log_s);
    float2 v[16];
    {
        const float2* p0 = a.in + off0;
        if constexpr (W && MODE == 0) {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = ld_stream(a.pre + (off0 - toff) + k * estep);
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            // The first pass streams the input; later passes read and write `out` in place.
            float2 x = MODE == 0 || CG ? ld_stream(p0 + k * estep) : p0[k * estep];
            if constexpr (W && MODE == 0) x = cmul(x, v[k]);
            v[k] = a.swap_in ? swap_ri(x) : x;
        }
    }
    if constexpr (TC != 0) tile_fft_tc<LOG_L, LOG_C, C, TC>(v, j, a.stw, smem, c, tid);
    else if constexpr (REGROUP) tile_fft_regroup<LOG_L, LOG_C>(v, j, c, jl, cl, a.stw, smem);
    else tile_fft<LOG_L, C>(v, j, a.stw, smem, c);
    if (twiddled) {
        if (Stages<LOG_L>::COUNT == 1) __syncthreads();  // tile_fft had no barrier to publish tws
        const float2* tw = tws + (MODE == 0 ? cl * 17 : 0);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = cmul(v[k], cmul(wjf, tw[k]));
    }
    const unsigned long long keep = a.l2_keep ? policy_evict_last() : 0ull;
    if (MODE == 0) {
        // Each column's L results leave as one contiguous, coalesced run at its digit-reversed place:
        // thread tid stores values kk0 + T i (i = 0..15) of column cc = tid / T, which it holds
        // (REGROUP) or gets through shared memory.
        const int cc = tid >> (LOG_L - 4), kk0 = tid & (T - 1);
        if constexpr (!REGROUP) {
            float2* w = smem + spad(j * C + c);
#pragma unroll
            for (int k = 0; k < 16; ++k) w[padc(k * T * C)] = v[k];
            __syncthreads();
            const float2* r = smem + spad(kk0 * C + cc);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = r[padc(i * T * C)];
        }
        const unsigned rr = col0 + cc;
        if (X && a.colstore) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                a.out[column_dst(a, rr, (unsigned)(kk0 + i * T))] = a.swap_out ? swap_ri(v[i]) : v[i];
            return;
        }
        const unsigned j2 = rr & ((1u << a.rev_b2) - 1), j1 = rr >> a.rev_b2;
        float2* q = a.out + toff + (((j1 + (j2 << a.rev_b1)) << LOG_L) + kk0);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (a.l2_keep) st_policy(q + i * T, v[i], keep);
            else q[i * T] = v[i];
        }
    } else if (X && MODE == 2) {
        const unsigned long long h = col0 >> a.log_s, q = (col0 & ((1u << a.log_s) - 1)) + c;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 x = a.swap_out ? swap_ri(v[k]) : v[k];
            a.out[column_dst(a, h, q + ((unsigned long long)(j + T * k) << a.log_s))] = x;
        }
    } else {
        float2* p0 = a.out + off0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            float2 x = a.swap_out ? swap_ri(v[k]) : v[k];
            if constexpr (W && MODE == 2) x = cmul(x, ld_stream(a.post + (off0 - toff) + k * estep));
            if (MODE == 1 && a.l2_keep) st_policy(p0 + k * estep, x, keep);
            else p0[k * estep] = x;
        }
    }
}

}  // namespace ofb
