// Shared parts of the anti-diagonal kernels (band_wave.cu, traceback.cu): the
// score table, the packed helpers and the letters entering a lane's windows.
#pragma once
#include <cuda_runtime.h>

#include "band_common.cuh"

namespace saber {

constexpr int kWaveRow = kWaveRowBytes;   // bytes per row of either score table
constexpr int kWaveSent = 24;             // row / column of the sentinel score
constexpr int kWaveAhead = 4;             // pairs of steps between a letter's load and its use

__device__ __forceinline__ uint32_t wv_prmt(uint32_t x, uint32_t y, uint32_t sel) { return __byte_perm(x, y, sel); }
__device__ __forceinline__ uint32_t wv_pk2(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x10001u; }

// Row word of query position i: byte offset of its table row | bias << 16;
// the sentinel row outside [0, m).
__device__ __forceinline__ uint32_t wv_row(const uint32_t* __restrict__ qrow, int i, int m) {
    return (unsigned)i < (unsigned)m ? __ldg(qrow + i) : (uint32_t)(kWaveSent * kWaveRow);
}
// Residue code of window column c, the sentinel code outside [0, n).
__device__ __forceinline__ uint32_t wv_col(const uint8_t* __restrict__ win, int c, int n) {
    return (unsigned)c < (unsigned)n ? (uint32_t)__ldg(win + c) : (uint32_t)kWaveSent;
}

// The score table: 24 x 24 matrix + gap open as int16, the sentinel in row and
// column 24, in 25 rows at the pitch of the pair table (a query's row words
// serve both without a multiply between a letter and its score's read: 40
// windows 257 -> 250 us).
__device__ __forceinline__ void wv_table(int16_t* tab, const int32_t* __restrict__ matrix, int go) {
    for (int t = threadIdx.x; t < 25 * 25; t += blockDim.x) {
        const int r = t / 25, c = t - r * 25;
        tab[r * (kWaveRow / 2) + c] =
            r < 24 && c < 24 ? (int16_t)(matrix[r * 24 + c] + go) : (int16_t)kSent16;
    }
}
// The pair table of a scheme whose scores + gap open fit int8: for row code q
// and two neighbouring column codes c, d the bytes S(q, c) + go, S(q, d) + go at
// kWaveRow q + 50 c + 2 d (sentinel -128), so that one 16-bit read gives a
// row's scores of an even and the following odd step.
constexpr int kWavePairBytes = 25 * kWaveRow;
static_assert(kWaveRow == 25 * 25 * 2, "a row holds every pair of column codes");
cudaError_t launch_wave_pairs(cudaStream_t s, const int32_t* matrix, int go, uint8_t* pairs);  // band_wave.cu

// Packed scores of two cells (low, high) plus the row pair's biases.
__device__ __forceinline__ uint32_t wv_sub(const uint8_t* tab, uint32_t ra, uint32_t ca, uint32_t rb, uint32_t cb,
                                           uint32_t bias) {
    const uint32_t x = *reinterpret_cast<const uint16_t*>(tab + ra + ca);
    const uint32_t y = *reinterpret_cast<const uint16_t*>(tab + rb + cb);
    return __vadd2(wv_prmt(x, y, 0x5410), bias);
}

// Anti-diagonals s = 2 i + k of the window cells of an m x n job with clipped
// band lo .. lo + w - 1: the even s to start at, and the pairs of steps.
__host__ __device__ inline void wv_span(int m, int n, int lo, int w, int& s0, int& nit) {
    const int hi = lo + w - 1;
    const int first = hi < 0 ? -hi : 0;
    int last = n - 1 - lo;
    if (last > m - 1) last = m - 1;
    const int s_min = 2 * first + (-lo - first > 0 ? -lo - first : 0);
    const int k_end = n - 1 - lo - last;
    const int s_max = 2 * last + (k_end < w - 1 ? k_end : w - 1);
    s0 = s_min & ~1;
    nit = (s_max - s0) / 2 + 1;
}

}  // namespace saber
