// fe_resident.cu — a whole Jacobi solve of few particles as one kernel.
//
// With few particles an iteration is all waiting: pressure_force and
// pressure_update each take some 7 us of which 2 are the launch and most of the
// rest the chain parameters -> count -> list words -> neighbours, and the graph's
// WHILE node adds 7 us between iterations (16k particles: 24 us an iteration,
// with a particle per thread 8.6).
// Here every particle keeps a thread for all the iterations.  The pair
// gradients, which do not change during a solve, stay in shared memory with the
// neighbours' indices, so an iteration is two gathers (4 bytes of p / rho^2, 16
// of acceleration), a thread's loads in flight together, and two grid-wide
// barriers: 4.1k particles' frame of 4 + 4 iterations 232 -> 133 us.  More
// particles take chunks (k_solve_resident_many): 16k 262 -> 207 us, 32k 282 ->
// 218.  How far each goes is decided in choose_resident.
//
// The arithmetic is that of k_pressure_force and k_pressure_update in the same
// order (the same bits), and so are the tolerance solver's FP64 sums, which
// every block adds up for itself from the warps' sums after each iteration.
//
// The launch is cooperative (all blocks resident); a barrier that does not
// come about within kBarrierSpins polls raises FE_STATS_LOOKBACK_TIMEOUT and
// ends the kernel.
#include "fe_common.cuh"
#include "fe_kernels.h"
#include "fe_neighbors.cuh"
#include "fe_pressure.cuh"

namespace fe {

namespace {

constexpr int kBarrierSpins = 1 << 22;

// Barrier number `k` (1, 2, ...) of the launch over all blocks.  False, with
// the flag raised, if it did not come about within `limit` polls.  Whole block.
// Every thread's stores before it come before every thread's loads after it
// (release and acquire by one thread, bar.sync for the others), so the gathers
// are plain loads, which the neighbours that a cell's particles share make L1
// hits (through L2 alone an iteration took 14.0 us instead of 11.2 at 37k
// particles).
__device__ __forceinline__ bool grid_barrier(uint32_t* flags, uint32_t* count, uint32_t k,
                                             int limit = kBarrierSpins) {
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        const uint32_t target = k * gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        int spins = 0;
        uint32_t seen;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
            if (seen >= target) break;
            if (++spins > limit) {
                atomicOr(flags, 0x4u);
                ok = 0;
                break;
            }
        }
    }
    return __syncthreads_and(ok || threadIdx.x != 0);
}

struct Particle {
    const float4* cache;   // [cnt][kResidentThreads]: gradient, neighbour index
    uint32_t i, cnt;
    f3 pi;
};

// f(gradient, load(j)) over particle q's neighbours in list order, kBatch loads
// in flight.
template <int kBatch, class Load, class F>
__device__ __forceinline__ void for_each_cached(const Bufs& B, const DevParams& P,
                                                const Particle& q, Load&& load, F&& f) {
    if (q.cnt > kNbrCap) {
        const float h = P.h;
        walk_ahead<true>(B, P, q.pi, load, [&](f3 rv, float r2, auto d) {
            const float r = sqrtf(r2);
            if (r > kEpsR) f(scale(kernel_grad_scale(r, h), rv), d);
        });
        return;
    }
    for (uint32_t k = 0; k < q.cnt; k += kBatch) {
        float4 e[kBatch];
        decltype(load(0u)) d[kBatch];
#pragma unroll
        for (int t = 0; t < kBatch; ++t)
            if (k + t < q.cnt) {
                e[t] = q.cache[(k + t) * kResidentThreads];
                d[t] = load(__float_as_uint(e[t].w));
            }
#pragma unroll
        for (int t = 0; t < kBatch; ++t)
            if (k + t < q.cnt) f(xyz(e[t]), d[t]);
    }
}

// The 8 sums of a chunk's warps, and of the final 8, as block_tree256 adds them.
__device__ __forceinline__ double tree8(const double* w) {
    return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
}

// The fixed-order sum and the largest of the warps' values (block_final_sum
// over chunk partials), in every thread.  s: 16 doubles.  Whole block.
__device__ __forceinline__ void sum_warps(const double* sums, const double* maxes, uint32_t chunks,
                                          double* s, double& sum, double& mx) {
    const int lane = lane_id();
    for (int vw = threadIdx.x >> 5; vw < 8; vw += blockDim.x >> 5) {
        double a = 0.0, b = 0.0;
        for (uint32_t c = vw * 32 + lane; c < chunks; c += 256) {
            double w[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                w[k] = __ldcg(sums + 8 * c + k);
                b = fmax(b, __ldcg(maxes + 8 * c + k));
            }
            a = a + tree8(w);
        }
        for (int m = 16; m >= 1; m >>= 1) {
            a = a + __shfl_xor_sync(kFull, a, m);
            b = fmax(b, __shfl_xor_sync(kFull, b, m));
        }
        if (lane == 0) {
            s[vw] = a;
            s[8 + vw] = b;
        }
    }
    __syncthreads();
    sum = tree8(s);
    mx = 0.0;
    for (int k = 0; k < 8; ++k) mx = fmax(mx, s[8 + k]);
    __syncthreads();
}

// The metric of an iteration from its sum and largest error (solve_finish_scene).
__device__ __forceinline__ void finish_metric(const DevParams& P, int which, double sum, double mx,
                                              double& metric, double& metric_max) {
    double avg = sum / (double)P.n;
    if (which == 1) {
        avg = avg * (double)P.dt;
        mx = mx * (double)P.dt;
    }
    metric = avg / (double)P.rho0;
    metric_max = mx / (double)P.rho0;
}

// The fixed-order sum and the largest of the chunks' partials, in every thread
// of a block of 256.
__device__ __forceinline__ void sum_chunks(const Bufs& B, double* smem, double& sum, double& mx) {
    __shared__ double s_result[2];
    const double a = block_final_sum(B.partials, B.n_chunks, smem);
    double m = 0.0;
    for (uint32_t k = threadIdx.x; k < B.n_chunks; k += kBlock)
        m = fmax(m, __ldcg(B.partials + B.n_chunks + k));
    m = block_max256(m, smem);
    if (threadIdx.x == 0) {
        s_result[0] = a;
        s_result[1] = m;
    }
    __syncthreads();
    sum = s_result[0];
    mx = s_result[1];
    __syncthreads();
}

// Scene s's control as its solve leaves it, and what k_solve_end records.
__device__ __forceinline__ void end_scene(const Bufs& B, int which, uint32_t s, uint32_t K,
                                          uint32_t iter, bool done, bool cap_hit, double metric,
                                          double metric_max) {
    SceneState& S = B.S[s];
    SolveCtl& ctl = S.solve[which];
    ctl.iter = iter;
    ctl.K = K;
    ctl.done = done;
    ctl.cap_hit = cap_hit;
    ctl.metric = metric;
    ctl.metric_max = metric_max;
    S.last_iters[which] = iter;
    S.last_metric[which] = metric;
    S.last_metric_max[which] = metric_max;
    S.total_iters[which] += iter;
    if (cap_hit) {
        S.cap_hits += 1;
        atomicOr(&B.G->flags, 0x1u);
    }
}
__device__ __forceinline__ void end_solve(const Bufs& B, int which) {
    B.G->cond[which] = 0;
    if (which == 1) B.G->src_nonfinite = 0;   // for the next density source
}

// The last block to leave resets the barrier for the next launch.
__device__ __forceinline__ void leave(uint32_t* barrier) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(barrier + 1, 1u) == gridDim.x - 1) {
        barrier[0] = 0;
        barrier[1] = 0;
    }
}

}  // namespace

// A solve of a single-scene context: iterations from the current pressures (or
// from where k_pressure_first left the density solve: begun != 0) until the
// solver's control says done.
// 16 entries at a time in the force and 8 in the update; all 36 and 18 at once
// made an iteration 2.8 us longer at 16k particles (more predicated
// instructions than latencies saved).
__global__ void __launch_bounds__(kResidentThreads, 3)
    k_solve_resident(Bufs B, ResidentScratch R, int which, int begun) {
    constexpr int kForceBatch = 16, kUpdateBatch = 8;
    extern __shared__ float4 s_cache[];
    __shared__ double s_sum[16];
    const DevParams& P = B.P[0];
    SceneState& S = B.S[0];
    SolveCtl& ctl = S.solve[which];
    const bool tolerance = P.solver == 1u;
    const uint32_t K = which == 0 ? S.iters_rho : S.iters_div;
    const uint32_t limit = tolerance ? P.max_it : K, min_it = P.min_it;
    const double tol = (double)(which == 0 ? P.tol_d : P.tol_v);
    const float m = P.mass, dt = P.dt, omega = P.omega;
    uint32_t iter = begun ? ctl.iter : 0u;
    bool done = begun ? ctl.done != 0u : limit == 0u;
    double metric = begun ? ctl.metric : 0.0, metric_max = begun ? ctl.metric_max : 0.0;
    bool cap_hit = begun && ctl.cap_hit != 0u;
    const uint32_t first_iter = iter;

    Particle q;
    q.i = blockIdx.x * blockDim.x + threadIdx.x;
    q.cache = s_cache + threadIdx.x;
    const uint32_t i = q.i;
    const bool live = i < B.n_total;
    q.cnt = 0;
    float4 p4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float rho_i = 0.0f, alpha_i = 0.0f, s_i = 0.0f, p_i = 0.0f;
    uint32_t barrier = 0;
    bool ok = true;
    const uint32_t chunks = B.n_chunks;
    if (blockIdx.x == 0 && tolerance)   // warps of the last chunk without particles
        for (uint32_t w = (B.n_total + 31) / 32 + threadIdx.x; w < 8 * chunks; w += blockDim.x)
            R.sums[w] = R.maxes[w] = 0.0;
    f3 acc = {0.0f, 0.0f, 0.0f};
    float pr_before = 0.0f;   // p / rho^2 as the last force saw it
    auto p_over_rho2 = [&] { return rho_i > kEpsR ? p_i / (rho_i * rho_i) : 0.0f; };
    if (!done && live) {
        p4 = *posb(B, i);
        q.pi = xyz(p4);
        q.cnt = B.nbr_count[i];
        rho_i = B.rho[i];
        alpha_i = B.alpha[i];
        s_i = B.src[i];
        p_i = B.prs[i];
        // the gradients to shared memory; the first force on the way, while
        // the neighbours' p / rho^2 come with their positions
        const float pr_i = p_over_rho2();
        pr_before = p4.w;
        auto force = [&](f3 grad, float pr_j) {
            if (pr_j == pr_j) acc = add(acc, scale(m * (pr_i + pr_j), grad));
        };
        if (q.cnt <= kNbrCap) {
            uint32_t k = 0;
            for_each_entry<8, true>(
                B, i, q.cnt, [&](uint32_t j) { return *posb(B, j); },
                [&](uint2 v, float4 pj) {
                    const f3 grad = scale(__uint_as_float(v.y), sub(q.pi, xyz(pj)));
                    s_cache[k * kResidentThreads + threadIdx.x] =
                        make_float4(grad.x, grad.y, grad.z, __uint_as_float(v.x));
                    ++k;
                    force(grad, pj.w);
                });
        } else {
            for_each_cached<1>(B, P, q, [&](uint32_t j) { return posb(B, j)->w; }, force);
        }
    }
    while (!done) {
        // every thread has its acceleration from the current pressures
        const f3 ai = {-acc.x, -acc.y, -acc.z};
        if (live) *accp(B, i) = make_float4(ai.x, ai.y, ai.z, 0.0f);
        if (!(ok = grid_barrier(&B.G->flags, R.barrier, ++barrier))) break;
        double e_sum = 0.0;
        if (live) {
            float sum_ap = 0.0f;
            for_each_cached<kUpdateBatch>(
                B, P, q, [&](uint32_t j) { return *accp(B, j); },
                [&](f3 grad, float4 aj) {
                    const f3 ad = sub(ai, xyz(aj));
                    sum_ap += m * dot(ad, grad);
                });
            const float ap_i = dt * sum_ap;
            const float error = s_i - ap_i;
            float e = 0.0f;
            if (alpha_i > kEpsR && rho_i > kEpsR) {
                const float a_ii = -(dt / (rho_i * rho_i)) * alpha_i;
                if (fabsf(a_ii) > 1e-20f) {
                    const float corr = (omega * error) / a_ii;
                    const float np = p_i + corr;
                    e = np > 0.0f ? fabsf(error) : (p_i * fabsf(a_ii)) / omega;
                    p_i = np > 0.0f ? np : 0.0f;
                }
            }
            if (iter != first_iter) pr_before = R.pr[i];
            R.pr[i] = pressure_over_rho2(p_i, rho_i);
            if (which == 0) e = dt * e;
            e_sum = e > 0.0f ? (double)e : 0.0;  // NaN -> 0
        }
        if (tolerance) {
            double a = e_sum, b = e_sum;
            for (int k = 16; k >= 1; k >>= 1) {
                a = a + __shfl_xor_sync(kFull, a, k);
                b = fmax(b, __shfl_xor_sync(kFull, b, k));
            }
            if (lane_id() == 0 && (i >> 5) < 8 * chunks) {
                R.sums[i >> 5] = a;
                R.maxes[i >> 5] = b;
            }
        }
        if (!(ok = grid_barrier(&B.G->flags, R.barrier, ++barrier))) break;
        ++iter;
        if (tolerance) {
            double sum, mx;
            sum_warps(R.sums, R.maxes, chunks, s_sum, sum, mx);
            finish_metric(P, which, sum, mx, metric, metric_max);
            if (iter >= min_it && metric <= tol) {
                done = true;
            } else if (iter >= limit) {
                done = true;
                cap_hit = true;
            }
        } else {
            done = iter >= K;
        }
        if (done || !live) continue;
        acc = {0.0f, 0.0f, 0.0f};
        const float pr_i = p_over_rho2();
        for_each_cached<kForceBatch>(
            B, P, q, [&](uint32_t j) { return R.pr[j]; },
            [&](f3 grad, float pr_j) {
                if (pr_j == pr_j) acc = add(acc, scale(m * (pr_i + pr_j), grad));
            });
    }
    // What the passes leave behind: pressure, p / rho^2, and the record's
    // position half as the last force wrote it.
    if (live && iter != first_iter) {
        B.prs[i] = p_i;
        *rec_pos(B, i) = make_float4(p4.x, p4.y, p4.z, pr_before);
        posb(B, i)->w = pressure_over_rho2(p_i, rho_i);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        end_scene(B, which, 0, K, iter, done, cap_hit, metric, metric_max);
        end_solve(B, which);
    }
    leave(R.barrier);
}

// The same for any number of particles: a grid of resident blocks strides over
// the chunks in each half iteration, with the passes' own list loops, and two
// grid barriers take the place of two launches and the WHILE node between
// iterations.  One scene, or several that all iterate a fixed number of times
// (then begun: k_pressure_first has run for them, without control).
__global__ void __launch_bounds__(kBlock, kResidentBlocks)
    k_solve_resident_many(Bufs B, ResidentScratch R, int which, int begun) {
    __shared__ double smem[8];
    __shared__ uint32_t s_limit;
    const bool one = B.n_scenes == 1;
    const DevParams& P0 = B.P[0];
    SolveCtl& ctl = B.S[0].solve[which];
    const bool tolerance = one && P0.solver == 1u;
    auto wanted = [&](uint32_t s) {
        if (one && tolerance) return P0.max_it;
        return which == 0 ? B.S[s].iters_rho : B.S[s].iters_div;
    };
    if (threadIdx.x == 0) s_limit = 0;
    __syncthreads();
    uint32_t most = 0;
    for (uint32_t s = threadIdx.x; s < B.n_scenes; s += kBlock) most = max(most, wanted(s));
    atomicMax(&s_limit, most);
    __syncthreads();
    const uint32_t limit = s_limit;
    uint32_t iter = 0;
    bool done = limit == 0u, cap_hit = false;
    double metric = 0.0, metric_max = 0.0;
    if (begun && one) {
        iter = ctl.iter;
        done = ctl.done != 0u;
        cap_hit = ctl.cap_hit != 0u;
        metric = ctl.metric;
        metric_max = ctl.metric_max;
    } else if (begun) {
        iter = limit != 0u && B.G->src_nonfinite == 0u ? 1u : 0u;
        done = iter >= limit;
    }
    uint32_t barrier = 0;
    while (!done) {
        for (uint32_t c = blockIdx.x; c < B.n_chunks; c += gridDim.x) {
            const uint4 cc = B.chunks[c];
            if (threadIdx.x < cc.y && (one || iter < wanted(cc.z)))
                pressure_force_particle<kBlock, true>(B, cc.x + threadIdx.x, cc.z);
        }
        if (!grid_barrier(&B.G->flags, R.barrier, ++barrier)) break;
        for (uint32_t c = blockIdx.x; c < B.n_chunks; c += gridDim.x) {
            const uint4 cc = B.chunks[c];
            const uint32_t i = cc.x + threadIdx.x;
            double e = 0.0;
            if (threadIdx.x < cc.y && (one || iter < wanted(cc.z)))
                e = pressure_update_particle(B, B.P[cc.z], i, which,
                                             pressure_update_sum<kBlock, true>(B, B.P[cc.z], i));
            if (tolerance) solve_chunk_partials(B, c, e, smem);
        }
        if (!grid_barrier(&B.G->flags, R.barrier, ++barrier)) break;
        ++iter;
        done = iter >= limit;
        if (tolerance) {
            double sum, mx;
            sum_chunks(B, smem, sum, mx);
            finish_metric(P0, which, sum, mx, metric, metric_max);
            if (iter >= P0.min_it && metric <= (double)(which == 0 ? P0.tol_d : P0.tol_v))
                done = true;
            else
                cap_hit = done;
        }
    }
    if (blockIdx.x == 0) {
        for (uint32_t s = threadIdx.x; s < B.n_scenes; s += kBlock) {
            const uint32_t K = which == 0 ? B.S[s].iters_rho : B.S[s].iters_div;
            end_scene(B, which, s, K, one ? iter : min(iter, K), done, cap_hit, metric, metric_max);
        }
        if (threadIdx.x == 0) end_solve(B, which);
    }
    leave(R.barrier);
}

namespace {
// Waits for a barrier that this launch alone cannot complete.
__global__ void k_barrier_selftest(uint32_t* count, uint32_t* flags, int limit) {
    grid_barrier(flags, count, 2, limit);
}
}  // namespace

cudaError_t grid_barrier_wait_on(uint32_t* count, uint32_t* flags, int limit, cudaStream_t stream) {
    k_barrier_selftest<<<1, kResidentThreads, 0, stream>>>(
        count, flags, limit < kBarrierSpins ? limit : kBarrierSpins);
    return cudaGetLastError();
}

}  // namespace fe
