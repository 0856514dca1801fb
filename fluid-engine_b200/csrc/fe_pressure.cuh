// fe_pressure.cuh — the two halves of a Jacobi iteration for one particle,
// shared by the passes (fe_kernels.cu) and the resident solves (fe_resident.cu).
// kCoherent: see for_each_neighbor.
#pragma once

#include "fe_neighbors.cuh"

namespace fe {

// pressure_force.comp:15-78.
template <int kThreads, bool kCoherent = false>
__device__ __forceinline__ void pressure_force_particle(const Bufs& B, uint32_t i, uint32_t s) {
    const DevParams& P = B.P[s];
    const float m = P.mass;
    const float4 p4 = kCoherent ? *posb(B, i) : __ldg(posb(B, i));
    const f3 pi = xyz(p4);
    const float rho_i = B.rho[i], p_i = B.prs[i];
    float p_rho_i = 0.0f;
    if (rho_i > kEpsR) p_rho_i = p_i / (rho_i * rho_i);
    f3 acc = {0.0f, 0.0f, 0.0f};
    for_each_neighbor<kThreads, kCoherent>(B, P, i, pi, [&](f3 rv, float g, float4 qj) {
        float p_rho_j = qj.w;  // p_j / rho_j^2, NaN when rho_j <= 1e-6
        if (p_rho_j == p_rho_j) {
            f3 grad = scale(g, rv);
            float term = p_rho_i + p_rho_j;
            acc = add(acc, scale(m * term, grad));
        }
    });
    // the whole record: this particle's position for pressure_update's
    // gathers and its acceleration
    st_record(B, i, p4, make_float4(-acc.x, -acc.y, -acc.z, 0.0f));
}

// The Jacobi update of particle i from its sum over the pairs; returns its
// term of the tolerance metric (0 without control).
__device__ __forceinline__ double pressure_update_particle(const Bufs& B, const DevParams& P,
                                                           uint32_t i, int which, float sum_ap) {
    const float dt = P.dt, omega = P.omega;
    const float alpha_i = B.alpha[i], rho_i = B.rho[i], s_i = B.src[i], p_i = B.prs[i];
    float ap_i = dt * sum_ap;
    float error = s_i - ap_i;
    float p_new = p_i;
    float e = 0.0f;
    if (alpha_i > kEpsR && rho_i > kEpsR) {
        float a_ii = -(dt / (rho_i * rho_i)) * alpha_i;
        if (fabsf(a_ii) > 1e-20f) {
            float corr = (omega * error) / a_ii;
            float np = p_i + corr;
            p_new = np > 0.0f ? np : 0.0f;
            B.prs[i] = p_new;
            e = np > 0.0f ? fabsf(error) : (p_i * fabsf(a_ii)) / omega;
        }
    }
    posb(B, i)->w = pressure_over_rho2(p_new, rho_i);
    if (which < 0 || P.solver != 1u) return 0.0;
    if (which == 0) e = dt * e;
    return e > 0.0f ? (double)e : 0.0;  // NaN -> 0
}

// The sum of particle i's pairs in the update.
template <int kThreads, bool kCoherent = false>
__device__ __forceinline__ float pressure_update_sum(const Bufs& B, const DevParams& P,
                                                     uint32_t i) {
    const float m = P.mass;
    const f3 pi = xyz(*posb(B, i));
    const f3 ai = xyz(*accp(B, i));
    float sum_ap = 0.0f;
    for_each_neighbor_pair<kThreads, kCoherent>(B, P, i, pi, B.rec, [&](f3 rv, float g, float4 aj) {
        f3 grad = scale(g, rv);
        f3 ad = sub(ai, xyz(aj));
        sum_ap += m * dot(ad, grad);
    });
    return sum_ap;
}

// Chunk c's partial of the fixed-order sum and its largest error (whole
// block).
__device__ __forceinline__ void solve_chunk_partials(const Bufs& B, uint32_t c, double e,
                                                     double* smem) {
    double part = block_tree256(e, smem);
    double mx = block_max256(e, smem);
    if (threadIdx.x == 0) {
        B.partials[c] = part;
        B.partials[B.n_chunks + c] = mx;
    }
}

}  // namespace fe
