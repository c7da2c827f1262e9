// transpose.cuh — A transposed for the kernels that read it [k][slot]
// (compute_stage_kmajor), by 64 x 64 tiles through shared memory.  HBM-bound:
// coalesced on both sides, 16 KB in flight per block.
#pragma once

#include <cstdint>

namespace sgb {
namespace ffma {

// A [m x lda] -> [k][ld]: row r at slot r, or, for 7-row threads, in groups of
// 28 rows per 32 slots whose last 12 rows sit 3 to 4 slots (Cfg::SLOTS).
struct TransposeJob {
    const float* src;
    float* dst;
    int m, k, ld_src, ld_dst;
    int sevens;  // 7-row slots
    int vec;     // 16-byte aligned rows: float4 loads
    int blocks;  // blocks of the launch that work on it (0: none)
};

constexpr int kTrTile = 64;  // transposed by 64 x 64 tiles, 256 threads each

__device__ __forceinline__ int slot_of(int row, int sevens) {
    if (!sevens) return row;
    const int q = row % 28;
    return row / 28 * 32 + (q < 16 ? q : 16 + (q - 16) / 3 * 4 + (q - 16) % 3);
}

// Tile t of the job.
__device__ __forceinline__ void transpose_tile(const TransposeJob& j, int t,
                                               float (&tile)[kTrTile][kTrTile + 1]) {
    const int tk = (j.k + kTrTile - 1) / kTrTile;
    const int c4 = threadIdx.x % 16, r0 = threadIdx.x / 16;  // 16 float4 columns x 16 rows
    const int k0 = t % tk * kTrTile, m0 = t / tk * kTrTile;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int row = m0 + r0 + 16 * i, k = k0 + 4 * c4;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row >= j.m) continue;
        const float* p = j.src + (int64_t)row * j.ld_src + k;
        if (j.vec && k + 3 < j.k) {
            v[i] = *reinterpret_cast<const float4*>(p);
        } else {
            if (k < j.k) v[i].x = p[0];
            if (k + 1 < j.k) v[i].y = p[1];
            if (k + 2 < j.k) v[i].z = p[2];
            if (k + 3 < j.k) v[i].w = p[3];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = r0 + 16 * i;
        tile[4 * c4][r] = v[i].x;
        tile[4 * c4 + 1][r] = v[i].y;
        tile[4 * c4 + 2][r] = v[i].z;
        tile[4 * c4 + 3][r] = v[i].w;
    }
    __syncthreads();
    const int row = m0 + threadIdx.x % 64;
    const int slot = slot_of(row, j.sevens);
    if (row < j.m) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int kk = threadIdx.x / 64 + 4 * i;
            if (k0 + kk < j.k)
                j.dst[(int64_t)(k0 + kk) * j.ld_dst + slot] = tile[kk][threadIdx.x % 64];
        }
    }
}

}  // namespace ffma
}  // namespace sgb
