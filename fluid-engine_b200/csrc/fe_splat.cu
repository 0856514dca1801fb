// fe_splat.cu — splat_density.comp:11-51 as a headless voxel grid.
//
// Each particle inside the box adds uint(200 (1 - (d/8)^2)^3) to every voxel
// at integer offset (x, y, z), d = |(x, y, z)| < 8, from its centre voxel
// ivec3(uvw * grid_res), uvw = (p - box_min) / (box_max - box_min).  The
// weight depends on d^2 alone, so it is evaluated once per d^2 (in the shader's
// FP32 operation order; 1,647 offsets, d^2 <= 53, have one that is not 0), and
// the grid is the convolution of the per-centre-voxel particle counts with it:
// grid[v] = sum_t w_t * count[v - d_t].  Integer sums do not depend on order,
// so the grid is bit-identical to the shader's scatter of atomic adds.
// (Scattering per particle with global reductions, or accumulating per tile
// with shared-memory atomics, did the same sums 2.4x and 2.7x slower at 1M
// particles on 128^3 than a plain convolution.)
//
// The weight depends on (y, z) through s = y^2 + z^2 alone, so the rows of
// counts along x with the same s (up to 12 of the 169) are added up first and
// then convolved along x once, with the weights of +x and -x together, eight
// voxels a thread: per voxel some 340 additions and 400 multiply-adds on
// registers and 100 16-byte shared loads, where the plain convolution's one
// shared load and multiply-add per tap (1,647 of each) made it wait for shared
// memory.
#include "fe_splat.h"

#include "fe_common.cuh"

namespace fe {

namespace {

// GLSL uint(x) for the splat's weights, which lie in [0, 200]: truncation.
__device__ __forceinline__ uint32_t glsl_uint(float x) { return __float2uint_rz(x); }
// GLSL int(x) with the conversion convention of the rest of the step:
// truncation, saturating, NaN -> 0 (cvt.rzi).
__device__ __forceinline__ int glsl_int(float x) { return __float2int_rz(x); }

__global__ void k_splat_weights(uint32_t* __restrict__ w) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kSplatSide * kSplatSide * kSplatSide) return;
    const int x = t % kSplatSide - kSplatRadius;
    const int y = (t / kSplatSide) % kSplatSide - kSplatRadius;
    const int z = t / (kSplatSide * kSplatSide) - kSplatRadius;
    const float r = (float)kSplatRadius;
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    const float dist = sqrtf((fx * fx + fy * fy) + fz * fz);   // length(vec3(x, y, z))
    uint32_t c = 0;
    if (dist < r) {
        const float x_norm = dist / r;
        float weight = 1.0f - x_norm * x_norm;
        weight = (weight * weight) * weight;
        c = glsl_uint(weight * 200.0f);
    }
    w[t] = c;
}

// The centre voxel of a particle, or false outside the box (the shader's
// early return).
__device__ __forceinline__ bool centre_voxel(float4 p, float3 bmin, float3 bmax, int3 res,
                                             int* cx, int* cy, int* cz) {
    const float sx = bmax.x - bmin.x, sy = bmax.y - bmin.y, sz = bmax.z - bmin.z;
    const float u = (p.x - bmin.x) / sx, v = (p.y - bmin.y) / sy, w = (p.z - bmin.z) / sz;
    if (u < 0.0f || v < 0.0f || w < 0.0f || u > 1.0f || v > 1.0f || w > 1.0f) return false;
    *cx = glsl_int(u * (float)res.x);
    *cy = glsl_int(v * (float)res.y);
    *cz = glsl_int(w * (float)res.z);
    return true;
}

// A block's output tile, and the window of counts it needs: 7 voxels around
// it (the weights are 0 beyond), x rounded out to whole 16-byte groups and
// padded so that the 16-byte loads of a quarter warp fall into different banks.
constexpr int kTileX = 32, kTileY = 8, kTileZ = 8;
constexpr int kReach = 7;
constexpr int kPer = 8;                           // voxels along x per thread
constexpr int kThreads = kTileX / kPer * kTileY * kTileZ;
constexpr int kWinX = kTileX + 16, kWinY = kTileY + 2 * kReach, kWinZ = kTileZ + 2 * kReach;
constexpr int kRow = kWinX + 4;                   // words from row to row
constexpr size_t kWinBytes = (size_t)kRow * kWinY * kWinZ * 4;

// The rows (y, z) with y^2 + z^2 <= kSplatMaxD2 sorted by that sum: one class
// per sum, its rows as offsets in words into the window.
struct RowClasses {
    int n, rows;
    int s[54], first[55], offset[192];
};
constexpr RowClasses make_classes() {
    RowClasses c{};
    for (int s = 0; s <= kSplatMaxD2; ++s) {
        const int before = c.rows;
        for (int z = -kReach; z <= kReach; ++z)
            for (int y = -kReach; y <= kReach; ++y)
                if (y * y + z * z == s) c.offset[c.rows++] = (z * kWinY + y) * kRow;
        if (c.rows == before) continue;
        c.s[c.n] = s;
        c.first[c.n++] = before;
    }
    c.first[c.n] = c.rows;
    return c;
}
constexpr RowClasses kClassTable = make_classes();
__constant__ RowClasses kClasses = kClassTable;
// Classes from here on reach at most 4 voxels along x.
constexpr int first_narrow() {
    int k = 0;
    while (kClassTable.s[k] + 25 <= kSplatMaxD2) ++k;
    return k;
}
constexpr int kNarrow = first_narrow();

// Classes [c0, c1): adds up their rows from kReachX voxels left of the thread's
// first one to kReachX right of its last (whole 16-byte groups) and convolves
// along x.  `at`: the thread's first voxel in the window.
template <int kReachX>
__device__ __forceinline__ void add_classes(uint32_t (&acc)[kPer], const uint32_t* at, int c0,
                                            int c1, const SplatWeights& W) {
    constexpr int kSide = (kReachX + 3) / 4 * 4, kWords = kPer + 2 * kSide;
    static_assert(kSide <= 8, "inside the window");
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
        uint32_t row[kWords];
#pragma unroll
        for (int i = 0; i < kWords; ++i) row[i] = 0u;
        const int end = kClasses.first[c + 1];
#pragma unroll 2
        for (int r = kClasses.first[c]; r < end; ++r) {
            const uint4* p = reinterpret_cast<const uint4*>(at + kClasses.offset[r] - kSide);
#pragma unroll
            for (int i = 0; i < kWords; i += 4) {
                const uint4 v = p[i / 4];
                row[i] += v.x;
                row[i + 1] += v.y;
                row[i + 2] += v.z;
                row[i + 3] += v.w;
            }
        }
        const int s = kClasses.s[c];
#pragma unroll
        for (int k = 0; k <= kReachX; ++k) {
            const uint32_t w = W.w[s + k * k];
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                acc[i] += w * (k ? row[kSide + i - k] + row[kSide + i + k] : row[kSide + i]);
        }
    }
}

__global__ void __launch_bounds__(256) k_splat_hist(const float4* __restrict__ pos, uint32_t n,
                                                    float3 bmin, float3 bmax, int3 res,
                                                    uint32_t* __restrict__ hist) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int cx, cy, cz;
    if (!centre_voxel(__ldg(pos + i), bmin, bmax, res, &cx, &cy, &cz)) return;
    cx = min(max(cx, 0), res.x);
    cy = min(max(cy, 0), res.y);
    cz = min(max(cz, 0), res.z);
    atomicAdd(hist + ((size_t)cz * (res.y + 1) + cy) * (res.x + 1) + cx, 1u);
}

// One block per output tile; a window without particles leaves the grid at 0.
// The bits of kSurfaceCount go out with the grid: the water pass would read 32
// times as much to find them (512^3 voxels: 0.48 ms).
__global__ void __launch_bounds__(kThreads, 2) k_splat_conv(const uint32_t* __restrict__ hist,
                                                            int3 res, SplatWeights W,
                                                            uint32_t* __restrict__ grid,
                                                            uint32_t* __restrict__ bits) {
    extern __shared__ __align__(16) uint32_t win[];  // [kWinZ][kWinY][kRow]
    const int tdx = (res.x + kTileX - 1) / kTileX, tdy = (res.y + kTileY - 1) / kTileY;
    const int tx = blockIdx.x % tdx, ty = (blockIdx.x / tdx) % tdy, tz = blockIdx.x / (tdx * tdy);
    const int ox = tx * kTileX - 8, oy = ty * kTileY - kReach, oz = tz * kTileZ - kReach;
    const int hx = res.x + 1, hy = res.y + 1, hz = res.z + 1;   // hist extent
    int any = 0;
#pragma unroll 4
    for (int v = threadIdx.x; v < kWinX * kWinY * kWinZ; v += kThreads) {
        const int wx = v % kWinX, wr = v / kWinX;
        const int x = ox + wx, y = oy + wr % kWinY, z = oz + wr / kWinY;
        uint32_t c = 0u;
        if (x >= 0 && y >= 0 && z >= 0 && x < hx && y < hy && z < hz)
            c = __ldg(hist + ((size_t)z * hy + y) * hx + x);
        win[wr * kRow + wx] = c;
        any |= c != 0u;
    }
    if (!__syncthreads_or(any)) return;
    const int lx = threadIdx.x % (kTileX / kPer) * kPer, ly = threadIdx.x / (kTileX / kPer) % kTileY,
              lz = threadIdx.x / (kTileX / kPer * kTileY);
    const uint32_t* at = win + ((lz + kReach) * kWinY + ly + kReach) * kRow + lx + 8;
    uint32_t acc[kPer] = {};
    add_classes<kReach>(acc, at, 0, kNarrow, W);
    add_classes<4>(acc, at, kNarrow, kClassTable.n, W);
    const int x = tx * kTileX + lx, y = ty * kTileY + ly, z = tz * kTileZ + lz;
    // a row of the tile is one word of bits, four threads' bytes
    static_assert(kTileX == 32 && kPer == 8, "a tile row per word");
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
        word |= (x + i < res.x && acc[i] > kSurfaceCount ? 1u : 0u) << (lx + i);
    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1);
    word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2);
    if (y >= res.y || z >= res.z) return;
    if (lx == 0) bits[((size_t)z * res.y + y) * tdx + tx] = word;
    uint32_t* out = grid + ((size_t)z * res.y + y) * res.x + x;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
        if (x + i < res.x) out[i] = acc[i];
}

__global__ void __launch_bounds__(256) k_splat_bits(const uint32_t* __restrict__ grid, int3 res,
                                                    uint32_t* __restrict__ bits) {
    const int words = (res.x + 31) / 32;
    const size_t w = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= (size_t)words * res.y * res.z) return;
    const int x = (int)(w % words) * 32 + (int)(threadIdx.x & 31u);
    const bool above = x < res.x && __ldg(grid + w / words * res.x + x) > kSurfaceCount;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, above);
    if ((threadIdx.x & 31u) == 0) bits[w] = b;
}

}  // namespace

cudaError_t splat_histogram(const float4* pos, uint32_t n, float3 box_min, float3 box_max,
                            int3 res, uint32_t* hist, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    k_splat_hist<<<(n + 255) / 256, 256, 0, stream>>>(pos, n, box_min, box_max, res, hist);
    return cudaGetLastError();
}

cudaError_t splat_convolve(const uint32_t* hist, int3 res, const SplatWeights& w, uint32_t* grid,
                           uint32_t* bits, cudaStream_t stream) {
    const int tdx = (res.x + kTileX - 1) / kTileX, tdy = (res.y + kTileY - 1) / kTileY,
              tdz = (res.z + kTileZ - 1) / kTileZ;
    cudaError_t e = cudaFuncSetAttribute(k_splat_conv, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kWinBytes);
    if (e != cudaSuccess) return e;
    k_splat_conv<<<tdx * tdy * tdz, kThreads, kWinBytes, stream>>>(hist, res, w, grid, bits);
    return cudaGetLastError();
}

cudaError_t splat_bits(const uint32_t* grid, int3 res, uint32_t* bits, cudaStream_t stream) {
    const size_t words = splat_bit_words(res);
    k_splat_bits<<<(unsigned)((words + 7) / 8), 256, 0, stream>>>(grid, res, bits);
    return cudaGetLastError();
}

cudaError_t splat_weights(uint32_t* d_weights, cudaStream_t stream) {
    const int total = kSplatSide * kSplatSide * kSplatSide;
    k_splat_weights<<<(total + 255) / 256, 256, 0, stream>>>(d_weights);
    return cudaGetLastError();
}

}  // namespace fe
