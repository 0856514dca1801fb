// fe_neighbors.cuh — particle/chunk mapping and the neighbour iteration
// shared by the DFSPH passes (fe_kernels.cu) and the learned warm start
// (fe_learned.cu).
#pragma once

#include "fe_common.cuh"

namespace fe {

__device__ __forceinline__ bool chunk_of(const Bufs& B, uint32_t& i, uint32_t& s,
                                         uint32_t& chunk) {
    chunk = blockIdx.x;
    uint4 c = B.chunks[chunk];
    s = c.z;
    i = c.x + threadIdx.x;
    return threadIdx.x < c.y;
}

// The shape of the neighbour passes for few particles: blocks of 64 threads, a
// quarter of a chunk each, so that the particles spread over all SMs, and
// deep batches of list entries (for_each_entry).
template <int kThreads>
constexpr int kEntryBatch = kThreads == kFewThreads ? 12 : 4;
template <int kThreads>
constexpr bool kEntryAhead = kThreads == kFewThreads;

// Block-size-agnostic particle loop of the neighbour kernels over the chunk
// table (the scene-offset table: every chunk is <= 256 consecutive particles
// of one scene).  A block of kThreads threads takes kThreads / 256 chunks at a
// time (512), or one chunk in 256 / kThreads passes (128); a grid smaller
// than the chunk count makes the kernel persistent: each block strides over
// the chunks until all are done.  Every warp covers 32 consecutive particles
// of one chunk, so warp-level cooperation and per-particle results are the
// same for every shape.  f(i, scene, live) is called by every thread of a
// warp together (live: i is a particle of the chunk).
template <int kThreads>
struct ParticleLoop {
    static_assert(kThreads == kFewThreads || kThreads == 128 || kThreads == 256 ||
                      kThreads == 512,
                  "block size");
    static constexpr uint32_t kChunksPerStep = kThreads >= kBlock ? kThreads / kBlock : 1;
    static constexpr uint32_t kPasses = kThreads >= kBlock ? 1 : kBlock / kThreads;
};

// kPersist = false: the grid has one block per chunk step and the loop
// below runs once (compiled without the loop state).
template <int kThreads, bool kPersist, class F>
__device__ __forceinline__ void for_each_particle(const Bufs& B, F&& f) {
    using L = ParticleLoop<kThreads>;
    if constexpr (kThreads == kFewThreads) {
        static_assert(!kPersist, "one block per quarter chunk");
        constexpr uint32_t per = kBlock / kFewThreads;
        if (B.n_scenes == 1) {   // chunk c starts at 256 c: no table read
            const uint32_t i = blockIdx.x * kFewThreads + threadIdx.x;
            f(i, 0u, i < B.n_total);
        } else {
            const uint4 cc = B.chunks[blockIdx.x / per];
            const uint32_t off = (blockIdx.x % per) * kFewThreads + threadIdx.x;
            f(cc.x + off, cc.z, off < cc.y);
        }
        return;
    }
    const uint32_t sub = kThreads >= kBlock ? threadIdx.x / kBlock : 0u;
    const uint32_t t = kThreads >= kBlock ? threadIdx.x % kBlock : threadIdx.x;
    auto step = [&](uint32_t c0) {
        const uint32_t c = c0 + sub;
        if (c >= B.n_chunks) return;   // whole warps: sub is uniform per 256 threads
        const uint4 cc = B.chunks[c];
#pragma unroll 1
        for (uint32_t k = 0; k < L::kPasses; ++k) {
            const uint32_t off = k * kThreads + t;
            f(cc.x + off, cc.z, off < cc.y);
        }
    };
    if constexpr (kPersist) {
        for (uint32_t c0 = blockIdx.x * L::kChunksPerStep; c0 < B.n_chunks;
             c0 += gridDim.x * L::kChunksPerStep)
            step(c0);
    } else {
        step(blockIdx.x * L::kChunksPerStep);
    }
}

// The bucket walk of the shaders (e.g. density_and_alpha.comp:31-63) over the
// {start, end} table.  f(j, r_vec, r2) is called for each candidate with
// r2 <= h*h, in walk order.  kCoherent: see for_each_neighbor (the table is
// the search's, so its loads are read-only ones either way).
template <bool kCoherent = false, class F>
__device__ __forceinline__ void walk(const Bufs& B, const DevParams& P, f3 pi, F&& f) {
    const float h = P.h;
    const float h2 = h * h;
    const int cx = cell_coord(pi.x, h), cy = cell_coord(pi.y, h), cz = cell_coord(pi.z, h);
    for (int z = -1; z <= 1; ++z)
        for (int y = -1; y <= 1; ++y)
            for (int x = -1; x <= 1; ++x) {
                uint32_t k = P.table_base +
                             cell_hash_pow2((int)((uint32_t)cx + (uint32_t)x),
                                            (int)((uint32_t)cy + (uint32_t)y),
                                            (int)((uint32_t)cz + (uint32_t)z), P.T - 1u);
                const uint2 cell = __ldg(B.cells + k);
                if (cell.x == kEmpty) continue;
                for (uint32_t j = cell.x; j < cell.y; ++j) {
                    f3 rv = sub(pi, xyz(kCoherent ? *posb(B, j) : __ldg(posb(B, j))));
                    float r2 = dot(rv, rv);
                    if (r2 > h2) continue;
                    f(j, rv, r2);
                }
            }
}

// The same with the next candidate's position and load(j) on their way while this
// one's terms are computed, f(r_vec, r2, load(j)): for few particles, whose threads
// have nothing else to wait with.  20 + 20 iterations of 2.3k and 8.2k particles at
// h = 2.6 spacings (73 neighbours each, more than the list holds): 13.2 and 15.1 ms
// in k_solve_resident with the walk above, 9.8 and 10.4 with this one; as passes
// of 256 threads a block 11.7 and 14.0.
template <bool kCoherent, class Load, class F>
__device__ __forceinline__ void walk_ahead(const Bufs& B, const DevParams& P, f3 pi, Load&& load,
                                           F&& f) {
    auto position = [&](uint32_t j) { return kCoherent ? *posb(B, j) : __ldg(posb(B, j)); };
    const float h2 = P.h * P.h;
    const int cx = cell_coord(pi.x, P.h), cy = cell_coord(pi.y, P.h), cz = cell_coord(pi.z, P.h);
#pragma unroll 1
    for (int z = -1; z <= 1; ++z)
#pragma unroll 1
        for (int y = -1; y <= 1; ++y)
#pragma unroll 1
            for (int x = -1; x <= 1; ++x) {
                const uint2 cell =
                    __ldg(B.cells + P.table_base +
                          cell_hash_pow2((int)((uint32_t)cx + (uint32_t)x),
                                         (int)((uint32_t)cy + (uint32_t)y),
                                         (int)((uint32_t)cz + (uint32_t)z), P.T - 1u));
                if (cell.x == kEmpty) continue;
                float4 pj = position(cell.x);
                auto d = load(cell.x);
#pragma unroll 1
                for (uint32_t j = cell.x; j < cell.y; ++j) {
                    const f3 rv = sub(pi, xyz(pj));
                    const auto d0 = d;
                    if (j + 1 < cell.y) {
                        pj = position(j + 1);
                        d = load(j + 1);
                    }
                    const float r2 = dot(rv, rv);
                    if (!(r2 > h2)) f(rv, r2, d0);
                }
            }
}

// Streaming read of a neighbour-list entry: read once per pass, so it
// bypasses L1 and carries an evict-first L2 policy, leaving the caches to the
// gathered neighbour data.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

__device__ __forceinline__ uint2 ld_list(const uint2* p, uint64_t pol) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
                 : "=r"(v.x), "=r"(v.y)
                 : "l"(p), "l"(pol));
    return v;
}

// The list entries of particle i in order: f(entry, load(entry.x)).  kBatch
// entries at a time, all their loads issued before the arithmetic, which runs
// strictly in list order.
// kAhead: also the next batch's list words are loaded before this batch's
// gathers are used.  The shape for few particles (see few() in fe_api.cu), where a
// pass is one chain of load latencies per thread and nothing else hides them;
// with many particles the passes are bound by the gathers' throughput and the
// registers cost more than the order gains.
template <int kBatch, bool kAhead, class Load, class F>
__device__ __forceinline__ void for_each_entry(const Bufs& B, uint32_t i, uint32_t cnt,
                                               Load&& load, F&& f) {
    const uint2* e = B.nbr + i;
    const size_t stride = B.n_total;
    const uint64_t pol = evict_first_policy();
    uint2 v[kBatch];
    decltype(load(0u)) d[kBatch];
    if constexpr (kAhead) {
        uint2 next[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            if (q < cnt) next[q] = ld_list(e + q * stride, pol);
        for (uint32_t k = 0; k < cnt; k += kBatch) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                v[q] = next[q];
                if (k + q < cnt) d[q] = load(v[q].x);
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (k + kBatch + q < cnt) next[q] = ld_list(e + (k + kBatch + q) * stride, pol);
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (k + q < cnt) f(v[q], d[q]);
        }
    } else {
        uint32_t k = 0;
        for (; k + kBatch <= cnt; k += kBatch) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q) v[q] = ld_list(e + (k + q) * stride, pol);
#pragma unroll
            for (int q = 0; q < kBatch; ++q) d[q] = load(v[q].x);
#pragma unroll
            for (int q = 0; q < kBatch; ++q) f(v[q], d[q]);
        }
        for (; k < cnt; ++k) {
            v[0] = ld_list(e + k * stride, pol);
            f(v[0], load(v[0].x));
        }
    }
}

// The walk of a pass in this shape: f(r_vec, r2, load(j)).
template <int kThreads, bool kCoherent, class Load, class F>
__device__ __forceinline__ void walk_for(const Bufs& B, const DevParams& P, f3 pi, Load&& load,
                                         F&& f) {
    if constexpr (kEntryAhead<kThreads>)
        walk_ahead<kCoherent>(B, P, pi, load, f);
    else
        walk<kCoherent>(B, P, pi, [&](uint32_t j, f3 rv, float r2) { f(rv, r2, load(j)); });
}

// Neighbours with r > 1e-6 in walk order: f(r_vec, grad_scale, pos_j), where
// pos_j = pos_b[j] (w = p_j / rho_j^2).  kCoherent: other blocks of the same
// launch write what is gathered (between grid barriers), so the loads are not
// read-only ones.
template <int kThreads, bool kCoherent = false, class F>
__device__ __forceinline__ void for_each_neighbor(const Bufs& B, const DevParams& P, uint32_t i,
                                                  f3 pi, F&& f) {
    const uint32_t cnt = B.nbr_count[i];
    if (cnt <= kNbrCap) {
        for_each_entry<kEntryBatch<kThreads>, kEntryAhead<kThreads>>(
            B, i, cnt, [&](uint32_t j) { return kCoherent ? *posb(B, j) : __ldg(posb(B, j)); },
            [&](uint2 v, float4 q) { f(sub(pi, xyz(q)), __uint_as_float(v.y), q); });
    } else {
        const float h = P.h;
        auto load = [&](uint32_t j) { return kCoherent ? *posb(B, j) : __ldg(posb(B, j)); };
        walk_for<kThreads, kCoherent>(B, P, pi, load, [&](f3 rv, float r2, float4 q) {
            const float r = sqrtf(r2);
            if (r > kEpsR) f(rv, kernel_grad_scale(r, h), q);
        });
    }
}

// As for_each_neighbor, over a 32-byte record array whose first half of
// record j is a copy of position_b: f(r_vec, grad_scale, second_half_j), with
// both halves of j fetched by one 256-bit load.  B.rec (position,
// acceleration) for pressure_update, B.pv (position, velocity_b) for
// viscosity and the FIXED-mode divergence source, B.pa (position,
// velocity_a) for the density source and the REFERENCE-mode divergence source.
struct Pair {
    float4 pos, data;
};
template <int kThreads, bool kCoherent = false, class F>
__device__ __forceinline__ void for_each_neighbor_pair(const Bufs& B, const DevParams& P,
                                                       uint32_t i, f3 pi, const float4* recs,
                                                       F&& f) {
    const uint32_t cnt = B.nbr_count[i];
    if (cnt <= kNbrCap) {
        for_each_entry<kEntryBatch<kThreads>, kEntryAhead<kThreads>>(
            B, i, cnt,
            [&](uint32_t j) {
                Pair p;
                if (kCoherent)
                    ld_pair_coherent(recs, j, p.pos, p.data);
                else
                    ld_pair(recs, j, p.pos, p.data);
                return p;
            },
            [&](uint2 v, const Pair& p) {
                f(sub(pi, xyz(p.pos)), __uint_as_float(v.y), p.data);
            });
    } else {
        const float h = P.h;
        auto load = [&](uint32_t j) {
            const float4* data = recs + 2 * (size_t)j + 1;
            return kCoherent ? *data : __ldg(data);
        };
        walk_for<kThreads, kCoherent>(B, P, pi, load, [&](f3 rv, float r2, float4 d) {
            const float r = sqrtf(r2);
            if (r > kEpsR) f(rv, kernel_grad_scale(r, h), d);
        });
    }
}

}  // namespace fe
