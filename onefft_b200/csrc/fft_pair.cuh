// Two columns per thread: the radix stages shared by the wide-tile passes (fft_wide.cu) and the
// cluster transforms (fft_cluster.cu).
#pragma once

#include "fft_device.cuh"

namespace ofb {

// Stage S on lane j of both columns (stage_compute, with each twiddle loaded once).
template <int LOG_L, int S>
__device__ __forceinline__ void pair_stage(float2 (&v)[2][16], int j, const float2* __restrict__ stw) {
    using St = Stages<LOG_L>;
    constexpr int LR = St::log2_radix(S), R = 1 << LR, NS = 1 << St::log2_ns(S), BPT = 16 / R;
#pragma unroll
    for (int i = 0; i < BPT; ++i) {
        float2 a[2][R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[0][q] = v[0][i + BPT * q], a[1][q] = v[1][i + BPT * q];
        if (S > 0) {
            const float2* tw = stw + St::tw_offset(S) + ((j + St::T * i) & (NS - 1));
#pragma unroll
            for (int q = 1; q < R; ++q) {
                const float2 w = __ldg(tw + (q - 1) * NS);
                a[0][q] = cmul(a[0][q], w);
                a[1][q] = cmul(a[1][q], w);
            }
        }
        dft<R>(a[0]);
        dft<R>(a[1]);
#pragma unroll
        for (int p = 0; p < R; ++p) v[0][i + BPT * p] = a[0][p], v[1][i + BPT * p] = a[1][p];
    }
}

}  // namespace ofb
