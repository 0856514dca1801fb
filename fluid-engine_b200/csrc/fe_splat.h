// fe_splat.h — density splat into a headless voxel grid (fe_splat.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace fe {

constexpr int kSplatRadius = 8;
constexpr int kSplatSide = 2 * kSplatRadius + 1;  // 17 offsets per axis
constexpr int kSplatMaxD2 = 53;                   // largest d^2 whose weight is not 0

// The weight per d^2 (sums of two squares and a third up to 7^2 may be looked
// up: 0 beyond kSplatMaxD2).
struct SplatWeights {
    uint32_t w[kSplatMaxD2 + 50];
};

// The integer weight of every voxel offset, [kSplatSide^3] with x fastest.
cudaError_t splat_weights(uint32_t* d_weights, cudaStream_t stream);

// What the water pass asks of the grid: bit x % 32 of word [z][y][x / 32] tells
// whether texel x is above kSurfaceCount (bits beyond the grid are 0).
constexpr uint32_t kSurfaceCount = 300;
inline size_t splat_bit_words(int3 res) { return (size_t)((res.x + 31) / 32) * res.y * res.z; }

// The splat as a convolution: hist[(rz+1)][(ry+1)][(rx+1)] counts the
// particles per centre voxel (centres run 0..res inclusive; cleared by the
// caller), then every grid voxel v gets sum_t weight_t * hist[v - offset_t]
// (exact in integers), and `bits` the grid's bits.  Tiles without particles in
// reach are skipped (the caller cleared grid and bits).
cudaError_t splat_histogram(const float4* pos, uint32_t n, float3 box_min, float3 box_max,
                            int3 res, uint32_t* hist, cudaStream_t stream);
cudaError_t splat_convolve(const uint32_t* hist, int3 res, const SplatWeights& w, uint32_t* grid,
                           uint32_t* bits, cudaStream_t stream);

// The bits of a grid that came from elsewhere.
cudaError_t splat_bits(const uint32_t* grid, int3 res, uint32_t* bits, cudaStream_t stream);

}  // namespace fe
