// fe_kernels.cu — the DFSPH passes as sm_100a kernels.
//
// One 256-thread block per chunk of <= 256 particles of one scene.  Each
// kernel restates one reference shader (cited per kernel); arithmetic is in
// the shader's order with no contraction (see fe_common.cuh), so results
// equal the host oracle bit for bit.
//
// Neighbour access.  density_alpha walks the 27 hash buckets exactly like the
// shaders (z, y, x offsets; bucket walk in sorted order; r^2 <= h^2) and, in
// the same pass, records for every particle the neighbours with r > 1e-6 in
// walk order together with the gradient scale grad_factor / (h r) of
// kernel_grad.  Positions do not move until the next neighbour search, so the
// ~18 later neighbour passes of the substep read this list (8 bytes per pair,
// coalesced: entry k of particle i at k * n_total + i) instead of re-walking
// ~216 candidates; they visit the same pairs in the same order and therefore
// produce identical sums.  A particle with more than kNbrCap neighbours keeps
// walking the buckets in every pass.
#include <cuda_fp16.h>

#include "fe_common.cuh"
#include "fe_features.cuh"
#include "fe_kernels.h"
#include "fe_neighbors.cuh"
#include "fe_pressure.cuh"

namespace fe {

// ---------------------------------------------------------------------------
// Neighbour search: spatial_hash.comp, grid_offsets.comp, reorder.comp.
// ---------------------------------------------------------------------------
__global__ void k_fill_u32(uint32_t* p, uint32_t v, size_t count) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) p[i] = v;
}

__global__ void k_fill_cells(uint2* p, size_t count) {
    stage_begin();
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride)
        p[i] = make_uint2(kEmpty, kEmpty);
}

// spatial_hash.comp:23-36 (the sentinel tail is written once at creation and
// never changes).
__global__ void __launch_bounds__(kBlock) k_hash(Bufs B) {
    stage_begin();
    uint32_t i, s, c;
    if (!chunk_of(B, i, s, c)) return;
    const DevParams& P = B.P[s];
    float4 p = __ldg(B.pos_a + i);
    const float h = P.h;
    B.keys[i] = P.table_base + cell_hash_pow2(cell_coord(p.x, h), cell_coord(p.y, h),
                                              cell_coord(p.z, h), P.T - 1u);
    B.vals[i] = i;
}

// grid_offsets.comp:20-33, also recording where each bucket ends so that the
// walk needs no hash comparison.
__global__ void k_offsets(Bufs B) {
    stage_begin();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.n_total) return;
    uint32_t key = B.keys[i];
    if (key >= B.T_total) return;
    uint32_t prev = i == 0 ? kEmpty : B.keys[i - 1];
    uint32_t next = i + 1 == B.n_total ? kEmpty : B.keys[i + 1];
    if (key != prev) B.cells[key].x = i;
    if (key != next) B.cells[key].y = i + 1;
}

// reorder.comp:37-46.  FIXED mode also gathers the pressures into prs_tmp.
// The neighbour list of the old order is invalidated: until density_alpha
// rebuilds it, the neighbour passes walk the new buckets.
// kCarry: the learned warm start's per-particle state is gathered too.
// Every store is a whole aligned vector of a fully written array (no
// read-modify-write of pos_b, no half-written record): partial sectors
// made this pass about twice as slow.
template <bool kCarry>
__device__ __forceinline__ void reorder_slot(const Bufs& B, int carry_pressure,
                                             const LearnArgs& L, uint32_t i, uint32_t src) {
    B.nbr_count[i] = kNbrCap + 1;
    // pos_b.w holds p / rho^2 of slot i (pressures and densities are not
    // permuted here): the value every pass that writes p or rho maintains,
    // recomputed from them.  The records' position half is written by
    // pressure_force, the only pass before pressure_update that needs it.
    float4 p = __ldg(B.pos_a + src);
    p.w = pressure_over_rho2(B.prs[i], B.rho[i]);
    *posb(B, i) = p;
    // position copy + velocity_b; then this slot's velocity_a record with the
    // new position copy (its velocity half is rewritten unchanged, so the
    // gathers of other threads read the same bytes either way)
    st_pair(B.pv, i, p, *vela(B, src));
    st_pair(B.pa, i, p, *vela(B, i));
    if (carry_pressure) B.prs_tmp[i] = B.prs[src];
    if (kCarry) {
        L.carry_tmp[i] = L.carry[src];
        L.mom_tmp[i] = L.mom[src];
    }
}

template <bool kCarry>
__device__ __forceinline__ void reorder_body(const Bufs& B, int carry_pressure,
                                             const LearnArgs& L) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.n_total) return;
    uint32_t src = B.vals[i];
    if (src >= B.n_total) src = i;  // unreachable for a valid permutation
    reorder_slot<kCarry>(B, carry_pressure, L, i, src);
}

__global__ void __launch_bounds__(kBlock) k_reorder(Bufs B, int carry_pressure) {
    stage_begin();
    reorder_body<false>(B, carry_pressure, LearnArgs{});
}
__global__ void __launch_bounds__(kBlock) k_reorder_carry(Bufs B, int carry_pressure,
                                                          LearnArgs L) {
    stage_begin();
    reorder_body<true>(B, carry_pressure, L);
}

// ---------------------------------------------------------------------------
// The search by cell counts (radix selected): the stable sort of the cell
// hashes as a counting sort over the table itself, which also yields the
// bucket bounds.
//   k_cell_count    hash of every particle; its cell's counter gives it a
//                   place among the cell's particles, in no particular order
//   k_cell_scan     exclusive sum over the table: {start, end} per slot
//   k_cell_scatter  particle indices to start + place
//   k_cell_reorder  each entry finds its rank among its cell's indices (so
//                   the order is the stable sort's) and takes the particle's
//                   state to that slot
// Four launches instead of hash, scratch fill, histogram, 2-4 radix passes,
// table fill, offsets and reorder, and 4 bytes moved per particle and pass
// instead of 16.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t particle_key(const DevParams& P, f3 p) {
    const float h = P.h;
    return P.table_base + cell_hash_pow2(cell_coord(p.x, h), cell_coord(p.y, h),
                                         cell_coord(p.z, h), P.T - 1u);
}

// The warp's particles come in the last search's order, so neighbours in the
// warp mostly share a cell: one atomic per run of equal keys.  All 32 lanes.
__device__ __forceinline__ void cell_count(const CellSort& C, uint32_t i, uint32_t key,
                                           bool live) {
    const uint32_t lane = threadIdx.x & 31u;
    if (!live) key = kEmpty;
    const uint32_t prev = __shfl_up_sync(kFull, key, 1);
    const bool head = lane == 0 || prev != key;
    const uint32_t heads = __ballot_sync(kFull, head);
    const uint32_t mine = 31u - __clz(heads & (kFull >> (31u - lane)));  // head of my run
    const uint32_t after = heads & ~(kFull >> (31u - lane));
    const uint32_t next = after ? __ffs(after) - 1u : 32u;
    uint32_t place = 0;
    if (head && live) place = atomicAdd(C.count + key, next - lane);
    place = __shfl_sync(kFull, place, mine) + (lane - mine);
    if (!live) return;
    C.key[i] = key;
    C.place[i] = place;
}

__global__ void __launch_bounds__(kBlock) k_cell_count(Bufs B, CellSort C) {
    stage_begin();
    uint32_t i, s, c;
    const bool live = chunk_of(B, i, s, c);
    const DevParams& P = B.P[s];
    const float4 p = live ? __ldg(B.pos_a + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    cell_count(C, i, particle_key(P, xyz(p)), live);
}

// Single-pass scan with decoupled look-back: a tile of kScanTile slots per
// block, taken in ticket order.  A status word holds the launch's number next
// to its state, so nothing has to be cleared between searches; the counters
// are left at zero for the next one.
constexpr unsigned long long kScanSum = 1ull << 32, kScanPrefix = 2ull << 32;

// The sum of the tiles before `tile` of this launch: 32 status words at a time,
// nearest last, until one holds a whole prefix.  A word that has not come within
// `limit` looks raises the flag and ends the wait.  One warp.
__device__ __forceinline__ uint32_t scan_look_back(const volatile unsigned long long* st, int tile,
                                                   unsigned long long epoch, int limit,
                                                   uint32_t* flags) {
    const int lane = lane_id();
    uint32_t base = 0;
    int spins = 0;
    for (int last = tile - 1; last >= 0;) {
        const int pred = last - lane;
        unsigned long long v = epoch | kScanPrefix;   // before tile 0: 0
        if (pred >= 0) v = st[pred];
        const bool ready = (v >> 34) == (epoch >> 34);
        const uint32_t not_ready = __ballot_sync(kFull, !ready);
        const uint32_t whole = __ballot_sync(kFull, ready && (v & kScanPrefix));
        // usable: the words up to the nearest whole prefix, or up to the
        // first one that is not there yet
        const uint32_t stop = whole ? __ffs(whole) : 33u;           // count to take
        const uint32_t gap = not_ready ? __ffs(not_ready) - 1u : 32u;
        const uint32_t take = min(stop, gap);
        uint32_t part = (uint32_t)lane < take ? (uint32_t)v : 0u;
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) part += __shfl_xor_sync(kFull, part, m);
        base += part;
        if (stop <= gap) break;
        last -= (int)take;
        if (take == 0) {
            if (++spins > limit) {
                if (lane == 0) atomicOr(flags, 0x4u);
                break;
            }
            __nanosleep(32);
        }
    }
    return base;
}

// A thread owns 8 slots, 32 bytes of counters and 64 of bounds, so every access
// is to whole sectors (16 slots a thread: 15.7 us at 2^20 slots; 8: 9 us).
__global__ void __launch_bounds__(kScanThreads) k_cell_scan(Bufs B, CellSort C) {
    stage_begin();
    constexpr int kWarps = kScanThreads / 32;
    __shared__ uint32_t s_warp[kWarps], s_base;
    __shared__ unsigned long long s_ticket;
    if (threadIdx.x == 0) s_ticket = atomicAdd(C.ticket, 1ull);
    __syncthreads();
    const uint32_t tile = (uint32_t)(s_ticket % gridDim.x);
    const unsigned long long epoch = ((s_ticket / gridDim.x) + 1ull) << 34;
    constexpr int kPer = kScanTile / kScanThreads;
    static_assert(kPer == 8, "two 16-byte loads and two 32-byte stores per thread");
    const uint32_t k0 = tile * kScanTile + threadIdx.x * kPer;
    uint32_t cnt[kPer], sum = 0;
    if (k0 + kPer <= B.T_total) {
#pragma unroll
        for (int q = 0; q < kPer; q += 4) {
            uint4* p = reinterpret_cast<uint4*>(C.count + k0 + q);
            const uint4 v = *p;
            *p = make_uint4(0u, 0u, 0u, 0u);
            cnt[q] = v.x; cnt[q + 1] = v.y; cnt[q + 2] = v.z; cnt[q + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            cnt[q] = 0;
            if (k0 + q < B.T_total) {
                cnt[q] = C.count[k0 + q];
                C.count[k0 + q] = 0;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) sum += cnt[q];
    // exclusive sum over the block
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kWarps ? s_warp[lane] : 0u, total = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, total, o);
            if (lane >= o) total += y;
        }
        if (lane < kWarps) s_warp[lane] = total - w;
        total = __shfl_sync(kFull, total, 31);
        // this tile's sum, then the sums of the tiles before it
        volatile unsigned long long* st = C.status;
        if (lane == 0) {
            st[tile] = epoch | (tile == 0 ? kScanPrefix : kScanSum) | total;
        }
        const uint32_t base = scan_look_back(st, (int)tile, epoch, kScanSpins, &B.G->flags);
        if (lane == 0) {
            if (tile) st[tile] = epoch | kScanPrefix | (unsigned long long)(base + total);
            s_base = base;
        }
    }
    __syncthreads();
    uint32_t start = s_base + s_warp[warp] + (x - sum);
    uint2 cell[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        cell[q] = cnt[q] ? make_uint2(start, start + cnt[q]) : make_uint2(kEmpty, kEmpty);
        start += cnt[q];
    }
    if (k0 + kPer <= B.T_total) {
#pragma unroll
        for (int q = 0; q < kPer; q += 4)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(
                             B.cells + k0 + q),
                         "r"(cell[q].x), "r"(cell[q].y), "r"(cell[q + 1].x), "r"(cell[q + 1].y),
                         "r"(cell[q + 2].x), "r"(cell[q + 2].y), "r"(cell[q + 3].x),
                         "r"(cell[q + 3].y)
                         : "memory");
    } else {
#pragma unroll
        for (int q = 0; q < kPer; ++q)
            if (k0 + q < B.T_total) B.cells[k0 + q] = cell[q];
    }
}

// Waits for the tile before tile 1, which nothing publishes.
__global__ void k_scan_selftest(const unsigned long long* status, uint32_t* flags, int limit) {
    scan_look_back(status, 1, 1ull << 34, limit, flags);
}
cudaError_t scan_wait_on(const unsigned long long* status, uint32_t* flags, int limit,
                         cudaStream_t stream) {
    k_scan_selftest<<<1, 32, 0, stream>>>(status, flags, limit < kScanSpins ? limit : kScanSpins);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(kBlock) k_cell_scatter(Bufs B, CellSort C) {
    stage_begin();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.n_total) return;
    const uint32_t at = B.cells[C.key[i]].x + C.place[i];
    if (at < B.n_total) C.slot[at] = i;  // always, unless a scan's wait gave up
}

template <bool kCarry>
__device__ __forceinline__ void cell_reorder(const Bufs& B, const CellSort& C, int carry_pressure,
                                             const LearnArgs& L, uint32_t t) {
    uint32_t src = __ldcg(C.slot + t);
    if (src >= B.n_total) src = t;  // unreachable, unless a scan's wait gave up
    const uint32_t key = C.key[src];
    const uint2 cell = B.cells[key];
    uint32_t i = t;
    if (cell.x <= t && t < cell.y && cell.y <= B.n_total) {
        uint32_t rank = 0;
        for (uint32_t q = cell.x; q < cell.y; ++q) rank += C.slot[q] < src;
        i = cell.x + rank;
    }
    if (i >= B.n_total) return;
    B.keys[i] = key;
    B.vals[i] = src;
    reorder_slot<kCarry>(B, carry_pressure, L, i, src);
}
__global__ void __launch_bounds__(kBlock) k_cell_reorder(Bufs B, CellSort C, int carry_pressure) {
    stage_begin();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < B.n_total) cell_reorder<false>(B, C, carry_pressure, LearnArgs{}, t);
}
__global__ void __launch_bounds__(kBlock) k_cell_reorder_carry(Bufs B, CellSort C,
                                                               int carry_pressure, LearnArgs L) {
    stage_begin();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < B.n_total) cell_reorder<true>(B, C, carry_pressure, L, t);
}

// FIXED mode: the gathered pressures become current; pr = p / rho^2 keeps
// matching the (not yet recomputed) densities.  kCarry: the gathered learned
// state too.
template <bool kCarry>
__device__ __forceinline__ void take_pressure_body(const Bufs& B, const LearnArgs& L) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B.n_total) return;
    float p = B.prs_tmp[i];
    B.prs[i] = p;
    posb(B, i)->w = pressure_over_rho2(p, B.rho[i]);
    if (kCarry) {
        L.carry[i] = L.carry_tmp[i];
    }
}

__global__ void __launch_bounds__(kBlock) k_take_pressure(Bufs B) {
    stage_begin();
    take_pressure_body<false>(B, LearnArgs{});
}
__global__ void __launch_bounds__(kBlock) k_take_pressure_carry(Bufs B, LearnArgs L) {
    stage_begin();
    take_pressure_body<true>(B, L);
}

// Snapshot of a float4 field for fe_download_async: element i of a field
// whose elements lie `stride` float4 apart, with w replaced by `w` when
// fix_w (the reference's w of that field; the device keeps other data there).
__global__ void __launch_bounds__(kBlock) k_snapshot4(float4* dst, const float4* src,
                                                      uint32_t stride, uint32_t n, int fix_w,
                                                      float w) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = src[(size_t)i * stride];
    if (fix_w) v.w = w;
    dst[i] = v;
}

// pr = p / rho^2, velocity_b's w = m / rho and velocity_a's w = the density
// residual t for all particles (after a host upload of p, rho, position_b or
// a velocity).  One block per chunk (t needs the scene's rho0).
__global__ void __launch_bounds__(kBlock) k_refresh_pr(Bufs B) {
    uint32_t i, s, c;
    if (!chunk_of(B, i, s, c)) return;
    posb(B, i)->w = pressure_over_rho2(B.prs[i], B.rho[i]);
    velb(B, i)->w = B.P[s].mass / B.rho[i];
    vela(B, i)->w = density_residual_t(B.rho[i], B.P[s].rho0);
}

// ---------------------------------------------------------------------------
// density_and_alpha.comp:14-72 + neighbour list.
//
// Two phases with the shader's summation order.  Phase 1 finds the in-range
// candidates (r^2 <= h^2, the shader's test) in walk order; phase 2 visits
// them in that order and does the expensive part (sqrt, kernel, gradient,
// list entry) with the lanes in lockstep.
//
// Phase 1 takes one of two forms, chosen per warp.  The lanes of a warp hold
// consecutive particles of the sorted order, and a run of lanes whose
// particles share a cell also shares that cell's 27 buckets.
//  * Few runs (bulk fluid, several particles per cell): cell-cooperative.  A
//    run's buckets laid end to end in walk order (z, y, x offsets, each
//    bucket's entries in sorted order) are its row of candidates.  The rows
//    are taken a window of kMaxSlabs slabs at a time, phase 1 and 2 for each
//    (mostly there is one).  Of a window the warp takes all its runs'
//    candidates a slab of 32 at a time: it stages the
//    slab's positions (each loaded once per run) in shared memory, and every
//    lane then tests its own particle against the 32 candidates of its run
//    and keeps the mask.  The test is a superset of the exact one, in packed
//    half precision relative to the run's first particle (see kNearHalf);
//    phase 2 applies the exact test.  In phase 2 the set bits of a particle's
//    masks, slab by slab and bit by bit, are its candidates in walk order; a
//    bit mask of where buckets start in the slab turns a bit back into a
//    particle index.
//  * Many runs (spray, sparse cells): each lane walks its own 27 buckets and
//    records its in-range candidates, kStage of them at a time.
// ---------------------------------------------------------------------------
// In-range candidates a lane can keep in the per-lane form; window and runs of
// the cooperative form: what fits 5.6 KB per warp, 32 warps an SM.  A
// moving dam break has 5 to 8 runs in the mean warp and more than 10 in 5 to
// 15 % of them; its rows are 70 to 320 candidates long.  Rows longer than a window
// come with a denser fluid, a larger h, and buckets that cells share (12,000
// particles at rest, 0.1 % of them with 385 to 392 candidates: 89 us when those
// walked in one phase, 36 in windows).  1M particles in motion, ms, walked /
// windows: h of 2.0 spacings 0.41 / 0.40, 2.42 1.62 / 0.71, 2.9 1.31 / 0.95.  Only
// where every candidate is in range, thousands of particles on one spot, does the
// test cost more than it saves (16k there: 5.7 / 7.1).
constexpr int kStage = 44;
constexpr int kMaxSlabs = 12;
constexpr uint32_t kWindow = kMaxSlabs * 32;
constexpr int kCoopRuns = 10;

// The near test in half precision, in units of h, relative to the first
// particle of the run.  A particle of the run lies within 1 of it on each axis
// and a candidate within 2, so rounding moves a coordinate difference by at
// most 2^-12 + 2^-11 + 2^-11, the sum of squares by at most 4.3e-3 where it
// is 1, and its three roundings add 1.5e-3: no pair with r <= h exceeds
// 1.0058.  Coordinates beyond half's range become Inf (rejected, as such a
// pair is far apart) or, Inf - Inf and NaN, pass on to the exact test.
constexpr float kNearHalf = 1.0078125f;
// h for which the scaled coordinates and h^2 stay far from FP32's limits.
constexpr float kCoopMinH = 1e-15f, kCoopMaxH = 1e15f;

// Per-warp scratch: one form or the other.
union DensityScratch {
    struct {
        uint32_t mask[kMaxSlabs][32];
        // the window of each run's row: where non-empty buckets start (bit c of
        // word w: at candidate 32 w + c; a bucket that goes on from the window
        // before starts at 0), how many start before a word, each bucket's
        // first entry minus its place in the window, and the candidates in it
        uint32_t starts[kCoopRuns][kMaxSlabs];
        uint8_t before[kCoopRuns][kMaxSlabs];
        uint32_t first[kCoopRuns][27];
        uint32_t total[kCoopRuns];
        int3 cell[kCoopRuns];
        alignas(16) float4 head[kCoopRuns];   // position of the run's first particle
        // a slab of each run: x, y, z as 16 pairs (candidate k, candidate
        // k + 16).  208 bytes apart, so that eight runs' 16-byte reads fall
        // into different banks
        alignas(16) __half near[kCoopRuns][104];
    };
    uint32_t cand[kStage][32];
};

struct DensityAcc {
    float density = 0.0f, sum_grad_sq = 0.0f;
    f3 grad_sum = {0.0f, 0.0f, 0.0f};
    uint32_t cnt = 0;
    float div = 0.0f;   // kDiv: the divergence source's sum
    uint2* op = nullptr;   // the particle's next list slot
};

// kn = kernel_norm(h); q = r / h is shared by W and grad W.  The list entry
// goes to a.op, the particle's next slot (a.op advances by one row).  kDiv != 0 also
// sums divergence_source_term.comp's m (v_i - v_j) . grad W over the same
// pairs in the same order (vi, vj: the velocities that pass binds).
template <int kDiv>
__device__ __forceinline__ void density_term(DensityAcc& a, float m, const DevParams& P, float kn,
                                             uint32_t j, f3 rv, float r2, uint32_t stride,
                                             f3 vi, float4 vj) {
    const float h = P.h;
    float r = sqrtf(r2);
    float q = div_h(r, h, P.inv_h, P.h_recip_exact);
    float w = kernel_w_q(q, kn);
    a.density += m * w;
    if (r > kEpsR) {
        float g = 0.0f;   // kernel_grad_scale_q with r > 1e-6 known
        if (!(q >= 1.0f)) {
            const float inner = kn * (18.0f * q * q - 12.0f * q);
            const float omq = 1.0f - q;
            const float outer = kn * -6.0f * omq * omq;
            const float gf = q <= 0.5f ? inner : outer;
            g = gf / (h * r);
        }
        f3 grad = scale(g, rv);
        f3 mg = scale(m, grad);
        a.grad_sum = add(a.grad_sum, mg);
        a.sum_grad_sq += dot(mg, mg);
        if (kDiv) {
            f3 vd = sub(vi, xyz(vj));
            a.div += m * dot(vd, grad);
        }
        if (a.cnt < kNbrCap) {
            *a.op = make_uint2(j, __float_as_uint(g));
            a.op += stride;
        }
        ++a.cnt;
    }
}

// Neighbour j's position (and, kDiv, the velocity the fused divergence
// source binds: velocity_b's record in FIXED mode, velocity_a's in
// REFERENCE mode; both records start with a copy of position_b).
template <int kDiv>
__device__ __forceinline__ f3 neighbour_pos(const Bufs& B, uint32_t j, float4& vj) {
    if (kDiv == 0) return xyz(__ldg(posb(B, j)));
    float4 q;
    ld_pair(kDiv == 1 ? B.pv : B.pa, j, q, vj);
    return xyz(q);
}

// A row's candidate c in slab `sl` (c = 32 sl + bit) as a particle index.
__device__ __forceinline__ uint32_t row_entry(const uint32_t* first, uint32_t starts,
                                              uint32_t before, uint32_t sl, uint32_t bit) {
    const uint32_t slot = before + __popc(starts & ((2u << bit) - 1u)) - 1u;
    return first[slot] + (sl << 5) + bit;
}

// Candidates [from, from + kWindow) of the rows of the warp's runs (see above;
// S.cell and S.head are set): the calling lane's masks, and in n_in the number
// that passed the near test.  Returns whether a row goes on.  All 32 lanes.
__device__ __forceinline__ bool coop_candidates(const Bufs& B, const DevParams& P,
                                                DensityScratch& S, int runs, int run, bool live,
                                                float4 p4, uint32_t from, uint32_t& n_in) {
    constexpr int kGroup = 4;   // runs whose loads are in flight together
    const uint32_t lane = (uint32_t)lane_id();
    const uint32_t lt_mask = (1u << lane) - 1u;
    bool more = false;
    n_in = 0;
    for (uint32_t t = lane; t < kCoopRuns * kMaxSlabs; t += 32) (&S.starts[0][0])[t] = 0u;
    __syncwarp();
#pragma unroll 1
    for (int r0 = 0; r0 < runs; r0 += kGroup) {
        uint32_t start[kGroup], len[kGroup];
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
            start[q] = len[q] = 0;
            if (r0 + q >= runs) continue;
            const int3 cell3 = S.cell[r0 + q];
            if (lane < 27u) {   // lane t: bucket t of the walk
                const int t = (int)lane;
                const int x = t % 3 - 1, y = (t / 3) % 3 - 1, z = t / 9 - 1;
                const uint2 cell = B.cells[P.table_base +
                                           cell_hash_pow2((int)((uint32_t)cell3.x + (uint32_t)x),
                                                          (int)((uint32_t)cell3.y + (uint32_t)y),
                                                          (int)((uint32_t)cell3.z + (uint32_t)z),
                                                          P.T - 1u)];
                start[q] = cell.x;
                len[q] = cell.x != kEmpty ? cell.y - cell.x : 0u;
            }
        }
#pragma unroll
        for (int q = 0; q < kGroup; ++q) {
            const int r = r0 + q;
            if (r >= runs) continue;
            uint32_t incl = len[q];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(kFull, incl, d);
                if (lane >= (uint32_t)d) incl += v;
            }
            const uint32_t total = __shfl_sync(kFull, incl, 31);
            more |= total > from + kWindow;
            // this lane's bucket within the window: places [a, b)
            const uint32_t excl = incl - len[q];
            const uint32_t a = max(excl, from) - from, b = min(incl, from + kWindow);
            const bool in = max(excl, from) < b;
            const uint32_t nonempty = __ballot_sync(kFull, in);
            if (in) {
                const uint32_t slot = __popc(nonempty & lt_mask), end = b - from;
                S.first[r][slot] = start[q] - excl + from;
                atomicOr(&S.starts[r][a >> 5], 1u << (a & 31u));
                // words that begin after this bucket's first entry and not
                // after its last have slot + 1 starts before them
                for (uint32_t k = (a >> 5) + 1; k <= end >> 5 && k < kMaxSlabs; ++k)
                    S.before[r][k] = (uint8_t)(slot + 1);
            }
            if (lane == 0) {
                S.total[r] = total > from ? min(total - from, kWindow) : 0u;
                S.before[r][0] = 0;
            }
        }
    }
    __syncwarp();
    const uint32_t my_total = live ? S.total[run] : 0u;
    const uint32_t my_slabs = (my_total + 31u) >> 5;
    const uint32_t slabs = __reduce_max_sync(kFull, my_slabs);
    const float inv_h = P.inv_h;
    const float4 o = live ? S.head[run] : p4;
    const __half2 ax = __float2half2_rn((p4.x - o.x) * inv_h),
                  ay = __float2half2_rn((p4.y - o.y) * inv_h),
                  az = __float2half2_rn((p4.z - o.z) * inv_h);
    const __half2 bound = __float2half2_rn(kNearHalf);
    const uint32_t at = 2u * (lane & 15u) + (lane >> 4);   // my candidate's place in `near`
#pragma unroll 1
    for (uint32_t sl = 0; sl < slabs; ++sl) {
        const uint32_t c = (sl << 5) + lane;
        {
#pragma unroll 1
            for (int r0 = 0; r0 < runs; r0 += kGroup) {
                float4 q[kGroup];
#pragma unroll
                for (int k = 0; k < kGroup; ++k) {
                    const int r = r0 + k;
                    q[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    // (a lane past the row's end stages anything: its bit is masked)
                    if (r < runs && c < S.total[r])
                        q[k] = __ldg(posb(B, row_entry(S.first[r], S.starts[r][sl],
                                                       S.before[r][sl], sl, lane)));
                }
#pragma unroll
                for (int k = 0; k < kGroup; ++k) {
                    if (r0 + k >= runs) continue;
                    __half* near = S.near[r0 + k];
                    const float4 o = S.head[r0 + k];
                    near[at] = __float2half_rn((q[k].x - o.x) * inv_h);
                    near[32 + at] = __float2half_rn((q[k].y - o.y) * inv_h);
                    near[64 + at] = __float2half_rn((q[k].z - o.z) * inv_h);
                }
            }
            __syncwarp();
            if (sl < my_slabs) {
                const uint4* near = reinterpret_cast<const uint4*>(S.near[run]);
                uint32_t far = 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const uint4 x4 = near[g], y4 = near[4 + g], z4 = near[8 + g];
                    const uint32_t xs[4] = {x4.x, x4.y, x4.z, x4.w},
                                   ys[4] = {y4.x, y4.y, y4.z, y4.w},
                                   zs[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const __half2 dx = __hsub2(ax, *reinterpret_cast<const __half2*>(&xs[k]));
                        const __half2 dy = __hsub2(ay, *reinterpret_cast<const __half2*>(&ys[k]));
                        const __half2 dz = __hsub2(az, *reinterpret_cast<const __half2*>(&zs[k]));
                        const __half2 r2 = __hfma2(dx, dx, __hfma2(dy, dy, __hmul2(dz, dz)));
                        far |= __hgt2_mask(r2, bound) & (0x00010001u << (4 * g + k));
                    }
                }
                const uint32_t rest = my_total - (sl << 5);
                const uint32_t bits = ~far & (rest < 32u ? (1u << rest) - 1u : kFull);
                S.mask[sl][lane] = bits;
                n_in += __popc(bits);
            }
            __syncwarp();
        }
    }
    return more;
}

// The per-lane form: the next in-range candidates of the lane's walk, at most
// kStage, to S.cand; returns their number.  t: the bucket to go on with (27: none
// left), next: the candidate in it (0: its first).
__device__ __forceinline__ uint32_t lane_candidates(const Bufs& B, const DevParams& P,
                                                    DensityScratch& S, f3 pi, int cx, int cy,
                                                    int cz, uint32_t& t, uint32_t& next) {
    const float h2 = P.h * P.h;
    const int lane = lane_id();
    uint32_t n = 0;
#pragma unroll 1
    for (uint32_t r = t / 3u; r < 9u; ++r) {   // three buckets' bounds in flight
        const uint32_t y = (uint32_t)cy + r % 3u - 1u, z = (uint32_t)cz + r / 3u - 1u;
        uint2 cell[3];
#pragma unroll
        for (uint32_t x = 0; x < 3u; ++x)
            cell[x] = __ldg(B.cells + P.table_base +
                            cell_hash_pow2((int)((uint32_t)cx + x - 1u), (int)y, (int)z, P.T - 1u));
#pragma unroll
        for (uint32_t x = 0; x < 3u; ++x) {
            uint32_t j = cell[x].x, end = j == kEmpty ? 0u : cell[x].y;
            if (3u * r + x < t) continue;
            if (next) {
                j = next;
                next = 0;
            }
            for (; j < end; ++j) {
                const f3 rv = sub(pi, xyz(__ldg(posb(B, j))));
                if (dot(rv, rv) > h2) continue;
                S.cand[n][lane] = j;
                if (++n == (uint32_t)kStage) {
                    t = 3u * r + x;
                    next = j + 1;
                    return n;
                }
            }
        }
    }
    t = 27u;
    return n;
}

// The candidates of a lane that passed the near test, in walk order.
struct RowWalk {
    uint32_t sl = 0, bits = 0, starts = 0, before = 0;
    __device__ __forceinline__ RowWalk(const DensityScratch& S, int run, int lane) {
        bits = S.mask[0][lane];
        starts = S.starts[run][0];
    }
    // the next one (there is one)
    __device__ __forceinline__ uint32_t next(const DensityScratch& S, int run, int lane) {
        while (bits == 0) {
            bits = S.mask[++sl][lane];
            starts = S.starts[run][sl];
            before = S.before[run][sl];
        }
        const uint32_t bit = __ffs(bits) - 1;
        bits &= bits - 1;
        return row_entry(S.first[run], starts, before, sl, bit);
    }
};

// Blocks per SM the launch bounds ask for: 1024 resident threads per SM
// (at most 64 registers per thread), for every block size.
// (the shape for few particles takes the registers for its loads in flight)
template <int kThreads>
constexpr int kMinBlocks = kThreads == kFewThreads ? 5 : 1024 / kThreads;

// Two warps a block, whatever the tuned shape: warps differ by a factor of two
// and more in their runs and candidates, and a block keeps its shared memory
// until its last warp is done.  On 1M particles 40 frames into a fall, 256
// threads take 0.50 ms, 64 threads 0.46.
constexpr int kDensityThreads = kFewThreads;
constexpr int kDensityBlocks = 16;   // 64 registers a thread

// kDiv: 0 density and alpha only; 1 also the FIXED-mode divergence source
// (velocity_b), 2 also the REFERENCE-mode one (velocity_a) -- see
// density_term.
// kLearn (with kDiv): also the divergence solve's feature row, from this
// pass's density, factor, count and source and the moments carried from
// the substep's density source.
template <int kDiv, bool kLearn>
__device__ __forceinline__ void density_alpha_particle(const Bufs& B, DensityScratch& S,
                                                       uint32_t i, uint32_t s, bool live,
                                                       const LearnArgs& L) {
    const DevParams& P = B.P[s];
    const float m = P.mass, h = P.h;
    const float kn = kernel_norm(h);
    const int lane = lane_id();
    const float4 p4 = live ? __ldg(posb(B, i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const f3 pi = xyz(p4);
    const int cx = cell_coord(pi.x, h), cy = cell_coord(pi.y, h), cz = cell_coord(pi.z, h);

    // Runs: live lanes form a prefix; a run starts where the cell changes.
    const int px = __shfl_up_sync(kFull, cx, 1), py = __shfl_up_sync(kFull, cy, 1),
              pz = __shfl_up_sync(kFull, cz, 1);
    const bool head = live && (lane == 0 || cx != px || cy != py || cz != pz);
    const uint32_t heads = __ballot_sync(kFull, head);
    const int runs = __popc(heads);
    const bool coop = runs <= kCoopRuns && h > kCoopMinH && h < kCoopMaxH;
    const uint32_t stride = B.n_total;
    DensityAcc a;
    // (the particle's velocity and next list slot are fetched again for every
    // batch of pairs: kept through phase 1, they are registers it needs)
    auto velocity = [&] {
        return kDiv ? xyz(__ldg(kDiv == 1 ? velb(B, i) : vela(B, i))) : f3{0.0f, 0.0f, 0.0f};
    };
    float4 vj = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // n candidates in order, the next one's position on its way while this one's
    // terms are computed
    auto sums = [&](uint32_t n, auto&& next) {
        if (n == 0) return;
        const f3 vi = velocity();
        a.op = B.nbr + i + (size_t)min(a.cnt, kNbrCap) * stride;
        uint32_t j = next();
        f3 pj = neighbour_pos<kDiv>(B, j, vj);
        for (uint32_t k = 1; k <= n; ++k) {
            const uint32_t j0 = j;
            const f3 p0 = pj;
            const float4 v0 = vj;
            if (k < n) {
                j = next();
                pj = neighbour_pos<kDiv>(B, j, vj);
            }
            const f3 rv = sub(pi, p0);
            const float r2 = dot(rv, rv);
            if (r2 > h * h) continue;   // the shader's test (phase 1 may pass a superset)
            density_term<kDiv>(a, m, P, kn, j0, rv, r2, stride, vi, v0);
        }
    };
    uint32_t n1 = 0;
    if (coop) {
        const int run = __popc(heads & ((2u << lane) - 1u)) - 1;
        if (head) {
            S.cell[run] = make_int3(cx, cy, cz);
            S.head[run] = p4;
        }
        __syncwarp();
        bool more = true;
#pragma unroll 1
        for (uint32_t from = 0; more; from += kWindow) {
            more = coop_candidates(B, P, S, runs, run, live, p4, from, n1);
            __syncwarp();
            if (live && n1) {
                RowWalk w(S, run, lane);
                sums(n1, [&] { return w.next(S, run, lane); });
            }
            __syncwarp();
        }
    } else {
        if (live)
            walk(B, P, pi, [&](uint32_t j, f3, float) {
                if (n1 < (uint32_t)kStage) S.cand[n1][lane] = j;
                ++n1;
            });
        // A lane with more than fit starts again, kStage at a time, going on with
        // its walk where it left it.  (Walking from the start for every kStage of
        // them took 118 ms beside cells of 4000 particles, this 16; a walk that
        // stops at kStage from the beginning is slower for the lanes with fewer.)
        uint32_t t = n1 > (uint32_t)kStage ? 0u : 27u, next = 0;
        if (t == 0u) n1 = 0;
        for (;;) {
            __syncwarp();
            uint32_t k = 0;
            sums(n1, [&] { return S.cand[k++][lane]; });
            if (!__any_sync(kFull, t < 27u)) break;
            n1 = lane_candidates(B, P, S, pi, cx, cy, cz, t, next);
        }
    }
    if (!live) return;
    if (kDiv) B.src[i] = -a.div;   // divergence_source_term.comp:58-60
    B.rho[i] = a.density;
    // velocity_b.w carries m / rho (the factor viscosity applies to each
    // neighbour's velocity, the same division done once per particle)
    velb(B, i)->w = m / a.density;
    float al = a.sum_grad_sq + dot(a.grad_sum, a.grad_sum);
    B.alpha[i] = al > kEpsR ? al : 0.0f;
    B.nbr_count[i] = a.cnt;
    // After the substep's re-sort this pass also makes the gathered state
    // current (what a separate copy pass did before): FIXED mode's pressure,
    // and the learned warm start's carry.
    float p_i;
    if (kDiv == 1) {
        p_i = B.prs_tmp[i];
        B.prs[i] = p_i;
    } else {
        p_i = B.prs[i];
    }
    posb(B, i)->w = pressure_over_rho2(p_i, a.density);
    if (a.cnt > kNbrCap) atomicOr(&B.G->flags, 0x2u);
    if (kLearn) {
        const float4 cr = L.carry_tmp[i];
        L.carry[i] = cr;
        // the substep's density-source moments, as the re-sort gathered them
        const float4 m4 = L.mom_tmp[i];
        const float fm[kMoments] = {m4.x, m4.y, m4.z, m4.w, cr.z};
        emit_features(B, L, P, i, s, 1, a.div, velocity(), fm);
    }
}

// kLanes: particles per warp, in its first lanes.  A warp's time is a chain of
// some 8000 instructions and their latencies whatever its number of
// particles, so with few particles 8 or 16 of them per warp make more, and
// shorter, chains (fewer cells each) where the SMs would otherwise idle.
template <int kLanes, class F>
__device__ __forceinline__ void density_particle(const Bufs& B, F&& f) {
    constexpr uint32_t per = kBlock / kLanes;   // warps per chunk
    const uint32_t unit = blockIdx.x * (kDensityThreads / 32) + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31u;
    if (B.n_scenes == 1) {   // chunk c starts at 256 c: no table read
        const uint32_t i = unit * kLanes + lane;
        f(i, 0u, lane < kLanes && i < B.n_total);
    } else {
        const uint4 cc = B.chunks[unit / per];
        const uint32_t off = (unit % per) * kLanes + lane;
        f(cc.x + off, cc.z, lane < kLanes && off < cc.y);
    }
}

template <int kLanes>
__global__ void __launch_bounds__(kDensityThreads, kDensityBlocks) k_density_alpha(Bufs B) {
    stage_begin();
    __shared__ DensityScratch scratch[kDensityThreads / 32];
    DensityScratch& S = scratch[threadIdx.x >> 5];
    density_particle<kLanes>(B, [&](uint32_t i, uint32_t s, bool live) {
        density_alpha_particle<0, false>(B, S, i, s, live, LearnArgs{});
    });
}

// density_alpha with the (plain) divergence source of the same substep
// summed in its pair loop: the divergence source needs exactly these pairs,
// gradients and order, and the neighbour's velocity shares a 32-byte record
// with the position copy the loop loads.  kDiv: 1 FIXED mode (velocity_b),
// 2 REFERENCE mode (velocity_a); a kernel each, since with both in one the
// compiler no longer inlines them (2079 -> 2437 us a 1M frame).  It runs right after the substep's
// re-sort and takes over that search's last copy: FIXED mode's gathered
// pressures (prs_tmp) become current here.
template <int kLanes, int kDiv>
__global__ void __launch_bounds__(kDensityThreads, kDensityBlocks) k_density_alpha_div(Bufs B) {
    __shared__ DensityScratch scratch[kDensityThreads / 32];
    DensityScratch& S = scratch[threadIdx.x >> 5];
    density_particle<kLanes>(B, [&](uint32_t i, uint32_t s, bool live) {
        density_alpha_particle<kDiv, false>(B, S, i, s, live, LearnArgs{});
    });
}

// The same with the learned state: also the divergence solve's features,
// and the gathered carry (carry_tmp) becomes current here in both modes.
template <int kLanes, int kDiv>
__global__ void __launch_bounds__(kDensityThreads, kDensityBlocks)
    k_density_alpha_div_learn(Bufs B, LearnArgs L) {
    __shared__ DensityScratch scratch[kDensityThreads / 32];
    DensityScratch& S = scratch[threadIdx.x >> 5];
    density_particle<kLanes>(B, [&](uint32_t i, uint32_t s, bool live) {
        density_alpha_particle<kDiv, true>(B, S, i, s, live, L);
    });
}

// ---------------------------------------------------------------------------
// viscosity.comp:17-66: velocity_b in, velocity_a out.
// ---------------------------------------------------------------------------
template <int kThreads>
__device__ __forceinline__ void viscosity_particle(const Bufs& B, uint32_t i, uint32_t s) {
    const DevParams& P = B.P[s];
    const float h = P.h;
    const float kn = kernel_norm(h), inv_h = P.inv_h;
    const uint32_t exact = P.h_recip_exact;
    const f3 pi = xyz(__ldg(posb(B, i)));
    const f3 vi = xyz(__ldg(velb(B, i)));
    f3 sum = {0.0f, 0.0f, 0.0f};
    // velocity_b.w = m / rho_j (written by density_alpha): one 256-bit load of
    // the position/velocity record per neighbour
    for_each_neighbor_pair<kThreads>(
        B, P, i, pi, B.pv, [&](f3 rv, float, float4 vj) {
            float r2 = dot(rv, rv);
            float r = sqrtf(r2);
            float w = kernel_w_q(div_h(r, h, inv_h, exact), kn);
            f3 vd = sub(xyz(vj), vi);
            sum = add(sum, scale_r(scale(vj.w, vd), w));
        });
    f3 vv = add(vi, scale(P.visc, sum));
    f3 g = {P.gx, P.gy, P.gz};
    f3 vf = add(vv, scale_r(g, P.dt));
    // the whole position/velocity_a record; w = the slot's density residual
    // t (density_residual_t) for the learned density source
    st_pair(B.pa, i, make_float4(pi.x, pi.y, pi.z, 0.0f),
            make_float4(vf.x, vf.y, vf.z, density_residual_t(B.rho[i], P.rho0)));
}

template <int kThreads, bool kPersist>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kThreads>) k_viscosity(Bufs B) {
    stage_begin();
    for_each_particle<kThreads, kPersist>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (live) viscosity_particle<kThreads>(B, i, s);
    });
}

// ---------------------------------------------------------------------------
// density_source_term.comp:16-74 (velocities = velocity_a).  The kLearn
// variant also emits the warm-start features (same arithmetic for s and p).
// ---------------------------------------------------------------------------
template <int kThreads, bool kLearn>
__device__ __forceinline__ void density_source_body(const Bufs& B, const LearnArgs& L,
                                                    uint32_t i, uint32_t s) {
    const DevParams& P = B.P[s];
    const float m = P.mass, dt = P.dt;
    const f3 pi = xyz(__ldg(posb(B, i)));
    const f3 vi = xyz(__ldg(vela(B, i)));
    float div = 0.0f;
    Moments mo;
    // velocity_a and (w) the density residual t of j from one load of its record
    for_each_neighbor_pair<kThreads>(B, P, i, pi, B.pa, [&](f3 rv, float g, float4 vj) {
        f3 grad = scale(g, rv);
        f3 vd = sub(vi, xyz(vj));
        div += m * dot(vd, grad);
        if (kLearn) mo.add_t(g, vj.w);   // velocity_a's w: the residual t of j
    });
    // for k_pressure_first: a gradient of this particle that is not finite
    // leaves the sum above not finite
    if (!isfinite(div)) atomicOr(&B.G->src_nonfinite, 1u);
    float rho_i = B.rho[i];
    float source = 0.0f;
    if (dt > kEpsR) source = ((P.rho0 - rho_i) / dt) - div;
    B.src[i] = source;
    B.prs[i] = 0.0f;
    posb(B, i)->w = pressure_over_rho2(0.0f, rho_i);
    if (kLearn) {
        float fm[kMoments];
        moment_features(mo, fm);
        emit_features(B, L, P, i, s, 0, div, vi, fm);
    }
}

template <int kThreads, bool kPersist>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kThreads>) k_density_source(Bufs B) {
    stage_begin();
    for_each_particle<kThreads, kPersist>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (live) density_source_body<kThreads, false>(B, LearnArgs{}, i, s);
    });
}
template <int kThreads, bool kPersist>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kThreads>)
    k_density_source_learn(Bufs B, LearnArgs L) {
    for_each_particle<kThreads, kPersist>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (live) density_source_body<kThreads, true>(B, L, i, s);
    });
}

// ---------------------------------------------------------------------------
// divergence_source_term.comp:14-61 (velocities = velocity_a in REFERENCE
// mode, velocity_b in FIXED mode).
// ---------------------------------------------------------------------------
template <int kThreads>
__device__ __forceinline__ void divergence_source_body(const Bufs& B, int fixed, uint32_t i,
                                                       uint32_t s) {
    const DevParams& P = B.P[s];
    const float m = P.mass;
    const f3 pi = xyz(__ldg(posb(B, i)));
    const f3 vi = xyz(__ldg(fixed ? velb(B, i) : vela(B, i)));
    float div = 0.0f;
    // both velocities sit in records that start with the position
    for_each_neighbor_pair<kThreads>(B, P, i, pi, fixed ? B.pv : B.pa,
                                     [&](f3 rv, float g, float4 vj) {
                                         f3 grad = scale(g, rv);
                                         f3 vd = sub(vi, xyz(vj));
                                         div += m * dot(vd, grad);
                                     });
    B.src[i] = -div;
}

// The stand-alone pass (the stage call; a frame sums it inside
// density_alpha, k_density_alpha_div).
template <int kThreads, bool kPersist>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kThreads>) k_divergence_source(Bufs B,
                                                                                      int fixed) {
    stage_begin();
    for_each_particle<kThreads, kPersist>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (live) divergence_source_body<kThreads>(B, fixed, i, s);
    });
}

// ---------------------------------------------------------------------------
// pressure_force.comp:15-78.  pr[j] = p_j / rho_j^2 (NaN when rho_j <= 1e-6)
// is maintained by every pass that writes p or rho.
// ---------------------------------------------------------------------------
template <int kThreads, bool kPersist>
__global__ void __launch_bounds__(kThreads, kMinBlocks<kThreads>) k_pressure_force(Bufs B,
                                                                                   int which) {
    stage_begin();
    for_each_particle<kThreads, kPersist>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (live && !(which >= 0 && B.S[s].solve[which].done))
            pressure_force_particle<kThreads>(B, i, s);
    });
}

// ---------------------------------------------------------------------------
// pressure_update.comp:18-84, plus the solver control of the tolerance loop.
// which = 0 (density solve), 1 (divergence solve), -1 (a bare stage call:
// no control).  The per-particle error of the pressure *before* this update
// is the projected-Jacobi step in residual units, with r_i = s_i - Ap_i:
// |r_i| where the update stays positive, p_i |a_ii| / omega where it clamps
// to 0 (0 for a particle at p = 0 that would go negative, i.e. complementary
// expansion), and 0 for rows the solver cannot act on (alpha or rho <= 1e-6).
// It vanishes only at the solution of the clamped system, so an over-
// estimated pressure counts as error as well as a missing one.  Times dt for
// the density solve, it is summed in the fixed FP64 order; the last block
// turns the per-scene sums into the metric, advances the iteration count and
// sets the loop condition.
// ---------------------------------------------------------------------------
// Index of scene sc's first chunk (chunks are laid out scene by scene): a
// block-wide sum of the chunk counts of the scenes before it.  `tmp` holds 8
// words.  Whole block.
__device__ __forceinline__ uint32_t scene_chunk_base(const Bufs& B, uint32_t sc, uint32_t* tmp) {
    uint32_t t = 0;
    for (uint32_t k = threadIdx.x; k < sc; k += kBlock) t += (B.P[k].n + kBlock - 1) / kBlock;
    for (int m = 16; m >= 1; m >>= 1) t += __shfl_xor_sync(kFull, t, m);
    if (lane_id() == 0) tmp[threadIdx.x >> 5] = t;
    __syncthreads();
    uint32_t r = 0;
    for (int w = 0; w < 8; ++w) r += tmp[w];
    __syncthreads();
    return r;
}

// Solver control of scene s after an iteration (whole block): the final
// fixed-order sum of its chunk partials, the metric, iteration count and
// done flag.  c0 = the scene's first chunk.
__device__ void solve_finish_scene(Bufs& B, int which, uint32_t s, uint32_t c0, double* smem) {
    const DevParams& P = B.P[s];
    SolveCtl& ctl = B.S[s].solve[which];
    uint32_t nchunks = (P.n + kBlock - 1) / kBlock;
    bool active = !ctl.done;
    double sum = 0.0, mx = 0.0;
    if (active && P.solver == 1u) {
        sum = block_final_sum(B.partials + c0, nchunks, smem);
        double m = 0.0;
        for (uint32_t k = threadIdx.x; k < nchunks; k += kBlock)
            m = fmax(m, __ldcg(B.partials + B.n_chunks + c0 + k));
        mx = block_max256(m, smem);
    }
    if (threadIdx.x == 0 && active) {
        ctl.iter += 1;
        if (P.solver == 1u) {
            double avg = sum / (double)P.n;
            if (which == 1) avg = avg * (double)P.dt;
            double metric = avg / (double)P.rho0;
            double metric_max = (which == 1 ? mx * (double)P.dt : mx) / (double)P.rho0;
            ctl.metric = metric;
            ctl.metric_max = metric_max;
            float tol = which == 0 ? P.tol_d : P.tol_v;
            if (ctl.iter >= P.min_it && metric <= (double)tol) {
                ctl.done = 1;
            } else if (ctl.iter >= P.max_it) {
                ctl.done = 1;
                ctl.cap_hit = 1;
            }
        } else {
            if (ctl.iter >= ctl.K) ctl.done = 1;
        }
    }
    __syncthreads();
}

// Sets the loop condition from every scene's done flag (whole block).
__device__ __forceinline__ void solve_set_condition(Bufs& B, int which,
                                                    cudaGraphConditionalHandle handle,
                                                    int use_handle) {
    int any_open = 0;
    for (uint32_t s = threadIdx.x; s < B.n_scenes; s += blockDim.x)
        if (!__ldcg(&B.S[s].solve[which].done)) any_open = 1;
    any_open = __syncthreads_or(any_open);
    if (threadIdx.x != 0) return;
    B.G->cond[which] = (uint32_t)any_open;
    if (use_handle) cudaGraphSetConditional(handle, (unsigned)any_open);
}

// Multi-scene contexts: the per-scene finish in parallel, one block per
// scene (the same per-scene code, so the same sums); the last block sets the
// loop condition.
__global__ void __launch_bounds__(kBlock) k_solve_finish(Bufs B, int which,
                                                         cudaGraphConditionalHandle handle,
                                                         int use_handle, int first) {
    __shared__ double smem[8];
    __shared__ uint32_t tmp[8];
    const uint32_t s = blockIdx.x;
    const uint32_t c0 = scene_chunk_base(B, s, tmp);
    // after k_pressure_first: unless that pass had to stand aside
    if (!first || B.G->src_nonfinite == 0u) solve_finish_scene(B, which, s, c0, smem);
    if (last_block_done(&B.G->tickets[kTicketSolve], gridDim.x)) {
        solve_set_condition(B, which, handle, use_handle);
        if (threadIdx.x == 0) B.G->tickets[kTicketSolve] = 0;
    }
}

// The stage call for few particles: no control, so no chunk partials.
__global__ void __launch_bounds__(kFewThreads, kMinBlocks<kFewThreads>)
    k_pressure_update_few(Bufs B) {
    stage_begin();
    for_each_particle<kFewThreads, false>(B, [&](uint32_t i, uint32_t s, bool live) {
        if (!live) return;
        const DevParams& P = B.P[s];
        pressure_update_particle(B, P, i, -1, pressure_update_sum<kFewThreads>(B, P, i));
    });
}

// One block per chunk, or a persistent grid whose blocks stride over the
// chunks (the per-chunk partials, and so the sums, are the same).
// kShape: the shape whose batches of list entries are used (the block has 256
// threads either way: its partials are per chunk).
template <int kShape>
__global__ void __launch_bounds__(kBlock) k_pressure_update(Bufs B, int which,
                                                            cudaGraphConditionalHandle handle,
                                                            int use_handle) {
    __shared__ double smem[8];
    const bool control = which >= 0;
    for (uint32_t c = blockIdx.x; c < B.n_chunks; c += gridDim.x) {
        const uint4 cc = B.chunks[c];
        const uint32_t i = cc.x + threadIdx.x, s = cc.z;
        const bool valid = threadIdx.x < cc.y;
        const DevParams& P = B.P[s];
        const bool skip = control && B.S[s].solve[which].done;
        double e_sum_in = 0.0;
        if (valid && !skip) {
            e_sum_in = pressure_update_particle(B, P, i, which,
                                                pressure_update_sum<kShape>(B, P, i));
        }
        if (control && !skip && P.solver == 1u) solve_chunk_partials(B, c, e_sum_in, smem);
    }
    if (!control) return;
    // One scene: its last block finishes the iteration.  Several scenes:
    // k_solve_finish does, one block per scene.
    if (B.n_scenes == 1 && last_block_done(&B.G->tickets[kTicketSolve], gridDim.x)) {
        solve_finish_scene(B, which, 0, 0, smem);
        solve_set_condition(B, which, handle, use_handle);
        if (threadIdx.x == 0) B.G->tickets[kTicketSolve] = 0;
    }
}

// Starts a solve: resets scene s's control; whether the scene is open.
__device__ __forceinline__ bool solve_begin_scene(const Bufs& B, int which, uint32_t s,
                                                  uint32_t& cap) {
    const DevParams& P = B.P[s];
    SolveCtl& ctl = B.S[s].solve[which];
    const uint32_t K = which == 0 ? B.S[s].iters_rho : B.S[s].iters_div;
    const uint32_t want = (P.solver == 1u) ? P.max_it : K;
    cap = want > cap ? want : cap;
    ctl.iter = 0;
    ctl.cap_hit = 0;
    ctl.metric = 0.0;
    ctl.metric_max = 0.0;
    ctl.K = K;
    ctl.done = want == 0u;
    return want != 0u;
}

// Starts a solve: resets the per-scene control and sets the loop condition.
// One block, scenes spread over its threads: a scene's control is a chain of
// dependent loads from its parameter block, and one thread walking 256 scenes
// took 248 us of a batch frame (about 4 us this way).
__global__ void __launch_bounds__(kBlock) k_solve_begin(Bufs B, int which,
                                                        cudaGraphConditionalHandle handle,
                                                        int use_handle) {
    __shared__ uint32_t s_cap;
    if (threadIdx.x == 0) s_cap = 0;
    __syncthreads();
    int any_open = 0;
    uint32_t cap = 0;
    for (uint32_t s = threadIdx.x; s < B.n_scenes; s += blockDim.x)
        if (solve_begin_scene(B, which, s, cap)) any_open = 1;
    if (cap) atomicMax(&s_cap, cap);
    any_open = __syncthreads_or(any_open);
    if (threadIdx.x != 0) return;
    B.G->cond[which] = (uint32_t)any_open;
    B.G->body_runs[which] = 0;
    B.G->body_cap[which] = s_cap + 2;
    if (which == 1) B.G->src_nonfinite = 0;   // for the next density source
    if (use_handle) cudaGraphSetConditional(handle, (unsigned)any_open);
}

// ---------------------------------------------------------------------------
// The density solve's first iteration without its two neighbour loops.  The
// density source has just set every pressure to 0 (and the plain start keeps
// it), so pressure_force sums m (0 + 0) grad W over the neighbours: +0 in
// every component while the gradients are finite, hence an acceleration of
// -0; and pressure_update then sums m (-0 - -0) . grad W: +0.  What remains
// is the update of each particle from its own source term.  The density
// source, which visits the same pairs, flags a sum that is not finite (the
// only way a gradient can be Inf or NaN); then this pass does nothing and
// the loop runs that iteration too.
// Bound by HBM (100 B per particle); at 1M it takes the place of 0.098 +
// 0.134 ms of list passes.
// Single scene: also begins the solve (its k_solve_begin), in the last block.
// Several scenes: k_solve_begin runs before, k_solve_finish after.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock) k_pressure_first(Bufs B,
                                                           cudaGraphConditionalHandle handle,
                                                           int use_handle) {
    __shared__ double smem[8];
    const bool usable = B.G->src_nonfinite == 0u;
    const uint32_t c = blockIdx.x;
    const uint4 cc = B.chunks[c];
    const uint32_t i = cc.x + threadIdx.x, s = cc.z;
    const DevParams& P = B.P[s];
    const uint32_t want = (P.solver == 1u) ? P.max_it : B.S[s].iters_rho;
    const bool run = usable && want != 0u;
    double e = 0.0;
    if (run && threadIdx.x < cc.y) {
        st_record(B, i, *posb(B, i), make_float4(-0.0f, -0.0f, -0.0f, 0.0f));
        e = pressure_update_particle(B, P, i, 0, 0.0f);
    }
    if (run && P.solver == 1u) solve_chunk_partials(B, c, e, smem);
    if (B.n_scenes != 1 || !last_block_done(&B.G->tickets[kTicketSolve], gridDim.x)) return;
    if (threadIdx.x == 0) {
        uint32_t cap = 0;
        solve_begin_scene(B, 0, 0, cap);
        B.G->body_runs[0] = 0;
        B.G->body_cap[0] = cap + 2;
        B.G->tickets[kTicketSolve] = 0;
    }
    __syncthreads();
    if (run) solve_finish_scene(B, 0, 0, 0, smem);
    solve_set_condition(B, 0, handle, use_handle);
}

// Last node of a WHILE body: counts executions and ends the loop after a
// hard bound even if the solver control above misbehaved, so a frame graph
// always terminates.  Raises FE_STATS_LOOKBACK_TIMEOUT when it has to act.
__global__ void k_loop_guard(Bufs B, int which, cudaGraphConditionalHandle handle) {
    if (threadIdx.x != 0) return;
    uint32_t runs = ++B.G->body_runs[which];
    if (runs >= B.G->body_cap[which]) {
        cudaGraphSetConditional(handle, 0);
        B.G->cond[which] = 0;
        atomicOr(&B.G->flags, 0x4u);
    }
}

// Ends a solve: records iterations used, residual and cap hits (scenes over
// the threads of one block, as k_solve_begin: 214 us before at 256 scenes).
__global__ void __launch_bounds__(kBlock) k_solve_end(Bufs B, int which) {
    for (uint32_t s = threadIdx.x; s < B.n_scenes; s += blockDim.x) {
        SceneState& S = B.S[s];
        SolveCtl& ctl = S.solve[which];
        S.last_iters[which] = ctl.iter;
        S.last_metric[which] = ctl.metric;
        S.last_metric_max[which] = ctl.metric_max;
        S.total_iters[which] += ctl.iter;
        if (ctl.cap_hit) {
            S.cap_hits += 1;
            atomicOr(&B.G->flags, 0x1u);
        }
    }
}

// ---------------------------------------------------------------------------
// pressure_integration.comp:16-77: position_b in, position_a and velocity_a
// out.
// ---------------------------------------------------------------------------
template <bool kLearn>
__device__ __forceinline__ void pressure_integration_body(const Bufs& B, const LearnArgs& L) {
    uint32_t i, s, c;
    if (!chunk_of(B, i, s, c)) return;
    const DevParams& P = B.P[s];
    const float dt = P.dt, r = P.radius;
    const float rest = 0.5f, fric = 0.95f, eps = 0.001f;
    f3 pos = xyz(__ldg(posb(B, i)));
    const float4 v0 = *vela(B, i);
    f3 vel = xyz(v0);
    f3 ap = xyz(*accp(B, i));
    f3 nv = add(vel, scale_r(ap, dt));
    f3 np = add(pos, scale_r(nv, dt));
    if (np.y < P.bminy + r) {
        np.y = P.bminy + r + eps; nv.y *= -rest; nv.x *= fric; nv.z *= fric;
    } else if (np.y > P.bmaxy - r) {
        np.y = P.bmaxy - r - eps; nv.y *= -rest; nv.x *= fric; nv.z *= fric;
    }
    if (np.x < P.bminx + r) {
        np.x = P.bminx + r + eps; nv.x *= -rest; nv.y *= fric; nv.z *= fric;
    } else if (np.x > P.bmaxx - r) {
        np.x = P.bmaxx - r - eps; nv.x *= -rest; nv.y *= fric; nv.z *= fric;
    }
    if (np.z < P.bminz + r) {
        np.z = P.bminz + r + eps; nv.z *= -rest; nv.x *= fric; nv.y *= fric;
    } else if (np.z > P.bmaxz - r) {
        np.z = P.bmaxz - r - eps; nv.z *= -rest; nv.x *= fric; nv.y *= fric;
    }
    B.pos_a[i] = make_float4(np.x, np.y, np.z, 1.0f);
    *vela(B, i) = make_float4(nv.x, nv.y, nv.z, v0.w);
    if (kLearn) after_solve_particle(B, L, P, i, 0);
}

__global__ void __launch_bounds__(kBlock) k_pressure_integration(Bufs B) {
    stage_begin();
    pressure_integration_body<false>(B, LearnArgs{});
}
// + the density solve's after-solve bookkeeping of the learned warm start
__global__ void __launch_bounds__(kBlock) k_pressure_integration_learn(Bufs B, LearnArgs L) {
    pressure_integration_body<true>(B, L);
}

// divergence_integration.comp:14-43 (velocity; colour is render-only).
template <bool kLearn>
__device__ __forceinline__ void divergence_integration_body(const Bufs& B, int fixed,
                                                            const LearnArgs& L) {
    uint32_t i, s, c;
    if (!chunk_of(B, i, s, c)) return;
    const DevParams& P = B.P[s];
    float4* vel = fixed ? velb(B, i) : vela(B, i);
    const float4 v0 = *vel;
    f3 nv = add(xyz(v0), scale_r(xyz(*accp(B, i)), P.dt));
    *vel = make_float4(nv.x, nv.y, nv.z, v0.w);  // w (the density) is kept
    if (kLearn) after_solve_particle(B, L, P, i, 1);
}

__global__ void __launch_bounds__(kBlock) k_divergence_integration(Bufs B, int fixed) {
    stage_begin();
    divergence_integration_body<false>(B, fixed, LearnArgs{});
}
__global__ void __launch_bounds__(kBlock) k_divergence_integration_learn(Bufs B, int fixed,
                                                                          LearnArgs L) {
    divergence_integration_body<true>(B, fixed, L);
}

// ---------------------------------------------------------------------------
// stats.comp:18-30 + FP64 means.  Per-chunk partials, combined per scene by
// the last block (no fill pass needed, order fixed).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t fixed_point(float x, float scale) {
    float v = x * scale;
    if (!(v > 0.0f)) return 0u;
    if (v >= 10000.0f) return 10000u;
    return (uint32_t)v;
}

// The stats of scene sc from its chunk partials (whole block): two FP64
// sums in the fixed order, integer max and sums.  c0 = its first chunk.
__device__ void stats_finish_scene(Bufs& B, const uint4* upart, uint32_t sc, uint32_t c0,
                                   double* smem, uint32_t (*s_u)[8]) {
    const DevParams& Q = B.P[sc];
    uint32_t nch = (Q.n + kBlock - 1) / kBlock;
    // Two FP64 sums in the fixed order over this scene's chunks.
    double t1 = 0.0, t2 = 0.0;
    for (uint32_t k = threadIdx.x; k < nch; k += kBlock) {
        t1 = t1 + __ldcg(B.partials + 2 * (c0 + k));
        t2 = t2 + __ldcg(B.partials + 2 * (c0 + k) + 1);
    }
    double f1 = block_tree256(t1, smem);
    double f2 = block_tree256(t2, smem);
    // integer partials: max and wrapping sums, order-free
    uint32_t a = 0, b = 0, d = 0;
    for (uint32_t k = threadIdx.x; k < nch; k += kBlock) {
        uint4 u = __ldcg(upart + c0 + k);
        a = max(a, u.x);
        b += u.y;
        d += u.z;
    }
    for (int m = 16; m >= 1; m >>= 1) {
        a = max(a, __shfl_xor_sync(kFull, a, m));
        b += __shfl_xor_sync(kFull, b, m);
        d += __shfl_xor_sync(kFull, d, m);
    }
    if (lane_id() == 0) {
        s_u[0][threadIdx.x >> 5] = a;
        s_u[1][threadIdx.x >> 5] = b;
        s_u[2][threadIdx.x >> 5] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = b = d = 0;
        for (int w = 0; w < 8; ++w) {
            a = max(a, s_u[0][w]);
            b += s_u[1][w];
            d += s_u[2][w];
        }
        SceneState& S = B.S[sc];
        S.stats[0] = a;
        S.stats[1] = b;
        S.stats[2] = d;
        S.stats_f64[0] = f1 / (double)Q.n;
        S.stats_f64[1] = f2 / (double)Q.n;
    }
    __syncthreads();
}

// The stats of one chunk (whole block): v = particle i's velocity (the one
// the pass binds), read by the caller.
__device__ __forceinline__ void stats_chunk(Bufs B, uint4* upart, bool valid, uint32_t i,
                                            uint32_t s, uint32_t c, float4 v) {
    __shared__ double smem[8];
    __shared__ uint32_t s_u[3][8];
    const DevParams& P = B.P[s];
    uint32_t mx = 0, s1 = 0, s2 = 0, bad = 0;
    double d1 = 0.0, d2 = 0.0;
    if (valid) {
        float speed = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
        mx = __float_as_uint(speed);
        float rho = B.rho[i], src = B.src[i];
        s1 = fixed_point(fabsf(rho - P.rho0), 1.0f);
        s2 = fixed_point(fabsf(src), 10.0f);
        d1 = fabs((double)rho - (double)P.rho0);
        d2 = fabs((double)src);
        bad = !(isfinite(speed) && isfinite(rho) && isfinite(src));
    }
    // integer parts: order-free
    for (int m = 16; m >= 1; m >>= 1) {
        mx = max(mx, __shfl_xor_sync(kFull, mx, m));
        s1 += __shfl_xor_sync(kFull, s1, m);
        s2 += __shfl_xor_sync(kFull, s2, m);
        bad |= __shfl_xor_sync(kFull, bad, m);
    }
    const int warp = threadIdx.x >> 5;
    if (lane_id() == 0) {
        s_u[0][warp] = mx;
        s_u[1][warp] = s1;
        s_u[2][warp] = s2;
    }
    if (bad) atomicOr(&B.S[s].nonfinite, 1u);
    double p1 = block_tree256(d1, smem);
    double p2 = block_tree256(d2, smem);
    if (threadIdx.x == 0) {
        uint32_t a = 0, b = 0, d = 0;
        for (int w = 0; w < 8; ++w) {
            a = max(a, s_u[0][w]);
            b += s_u[1][w];
            d += s_u[2][w];
        }
        upart[c] = make_uint4(a, b, d, 0);
        B.partials[2 * c] = p1;
        B.partials[2 * c + 1] = p2;
    }
    // One scene: its last block finishes.  Several scenes: k_stats_finish
    // does, one block per scene.
    if (B.n_scenes == 1 && last_block_done(&B.G->tickets[kTicketStats], gridDim.x)) {
        stats_finish_scene(B, upart, 0, 0, smem, s_u);
        if (threadIdx.x == 0) B.G->tickets[kTicketStats] = 0;
    }
}

__global__ void __launch_bounds__(kBlock) k_stats(Bufs B, int fixed, uint4* upart) {
    stage_begin();
    uint32_t i, s, c;
    const bool valid = chunk_of(B, i, s, c);
    const float4* vel = fixed ? velb(B, 0) : vela(B, 0);
    stats_chunk(B, upart, valid, i, s, c,
                valid ? vel[(size_t)i * 2u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f));
}

// The substep's last divergence integration and the frame's stats in one
// pass: the stats read the velocity this pass has just written (the same
// value the stats pass would read back), and every other input of the stats
// is final by then.
template <bool kLearn>
__device__ __forceinline__ void divergence_integration_stats_body(const Bufs& B, int fixed,
                                                                  const LearnArgs& L,
                                                                  uint4* upart) {
    uint32_t i, s, c;
    const bool valid = chunk_of(B, i, s, c);
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (valid) {
        const DevParams& P = B.P[s];
        float4* vel = fixed ? velb(B, i) : vela(B, i);
        const float4 v0 = *vel;
        const f3 nv = add(xyz(v0), scale_r(xyz(*accp(B, i)), P.dt));
        v = make_float4(nv.x, nv.y, nv.z, v0.w);
        *vel = v;
        if (kLearn) after_solve_particle(B, L, P, i, 1);
    }
    stats_chunk(B, upart, valid, i, s, c, v);
}

__global__ void __launch_bounds__(kBlock) k_divergence_integration_stats(Bufs B, int fixed,
                                                                         uint4* upart) {
    divergence_integration_stats_body<false>(B, fixed, LearnArgs{}, upart);
}
__global__ void __launch_bounds__(kBlock) k_divergence_integration_stats_learn(Bufs B, int fixed,
                                                                               LearnArgs L,
                                                                               uint4* upart) {
    divergence_integration_stats_body<true>(B, fixed, L, upart);
}

__global__ void __launch_bounds__(kBlock) k_stats_finish(Bufs B, uint4* upart) {
    stage_begin();
    __shared__ double smem[8];
    __shared__ uint32_t s_u[3][8];
    const uint32_t sc = blockIdx.x;
    const uint32_t c0 = scene_chunk_base(B, sc, s_u[0]);
    stats_finish_scene(B, upart, sc, c0, smem, s_u);
}

// ---------------------------------------------------------------------------
// Frame prologue (renderer/mod.rs:231-267): adaptive CFL dt and early-exit
// iteration choice from the previous frame's stats.  One thread per scene.
// ---------------------------------------------------------------------------
__global__ void k_frame_prologue(Bufs B) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= B.n_scenes) return;
    DevParams& P = B.P[s];
    SceneState& S = B.S[s];
    float n = (float)P.n;
    float max_speed = __uint_as_float(S.stats[0]);
    float avg_de = (float)S.stats[1] / (1.0f * n);
    float avg_ve = (float)S.stats[2] / (10.0f * n);
    if (P.use_cfl && max_speed > 0.01f) {
        float cfl = (P.cfl_lambda * P.h) / max_speed;
        if (cfl < P.cfl_min) cfl = P.cfl_min;
        if (cfl > P.cfl_max) cfl = P.cfl_max;
        P.dt = fminf(cfl, P.dt * P.cfl_growth);
    }
    float rho0 = P.rho0;
    float thr_d = P.eta_d_pct / 100.0f * rho0;
    float thr_v = P.eta_v_pct / 100.0f * rho0;
    bool early = P.use_thr && P.solver == 0u;
    S.iters_rho = (early && avg_de < thr_d) ? 2u : P.k_rho;
    S.iters_div = (early && avg_ve < thr_v) ? 1u : P.k_div;
}

// fe_read_stats_async: scene `scene`'s stats, the global flags and its dt,
// in stream order, into mapped host memory (one thread; a few hundred
// bytes).
__global__ void k_stats_snapshot(Bufs B, StatsSnapshot* dst, uint32_t scene) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    dst->S = B.S[scene];
    dst->G = *B.G;
    dst->dt = B.P[scene].dt;
    dst->n = B.P[scene].n;
    __threadfence_system();
}

__global__ void k_count_substep(Bufs B) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < B.n_scenes) B.S[s].substeps += 1;
}

// The block sizes the autotuner chooses from.
#define FE_NBR_INSTANTIATE(T, P)                                                      \
    template __global__ void k_viscosity<T, P>(Bufs);                                 \
    template __global__ void k_density_source<T, P>(Bufs);                            \
    template __global__ void k_density_source_learn<T, P>(Bufs, LearnArgs);           \
    template __global__ void k_divergence_source<T, P>(Bufs, int);                    \
    template __global__ void k_pressure_force<T, P>(Bufs, int);
FE_NBR_INSTANTIATE(kFewThreads, false)
FE_NBR_INSTANTIATE(128, false)
FE_NBR_INSTANTIATE(256, false)
FE_NBR_INSTANTIATE(512, false)
FE_NBR_INSTANTIATE(128, true)
FE_NBR_INSTANTIATE(256, true)
FE_NBR_INSTANTIATE(512, true)
#define FE_DENSITY_INSTANTIATE(L)                                              \
    template __global__ void k_density_alpha<L>(Bufs);                         \
    template __global__ void k_density_alpha_div<L, 1>(Bufs);                  \
    template __global__ void k_density_alpha_div<L, 2>(Bufs);                  \
    template __global__ void k_density_alpha_div_learn<L, 1>(Bufs, LearnArgs); \
    template __global__ void k_density_alpha_div_learn<L, 2>(Bufs, LearnArgs);
FE_DENSITY_INSTANTIATE(8)
FE_DENSITY_INSTANTIATE(16)
FE_DENSITY_INSTANTIATE(32)
template __global__ void k_pressure_update<kBlock>(Bufs, int, cudaGraphConditionalHandle, int);
template __global__ void k_pressure_update<kFewThreads>(Bufs, int, cudaGraphConditionalHandle, int);

}  // namespace fe
