// qew_team.cuh -- the group of threads that runs one device-resident solve:
// one CTA (CtaTeam) or one thread-block cluster (ClusterTeam: up to 16 CTAs
// on as many SMs, sharing a line). A team gives every thread its first index
// and stride over the line, broadcast reductions whose result is identical in
// every thread, and a barrier after which writes of any team thread are
// visible.
//   * CtaTeam: exactly the CTA primitives of qew_block.cuh (warp butterflies,
//     warp partials added in warp order, __syncthreads).
//   * ClusterTeam: indices and the cluster barrier; its reductions are the
//     batched ones of qew_lbfgs_gram.cuh. Loads of vectors that the team
//     shares bypass L1 (ld.global.cg): another SM may have written them.
#pragma once

#include <cooperative_groups.h>

#include "qew_block.cuh"

constexpr int kTeamMaxCtas = 16;

template <int BS>
struct CtaTeam {
    static constexpr bool kCluster = false;
    static constexpr int kBS = BS;
    double *s_w;  // >= 96 doubles of shared memory
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int stride() const { return BS; }
    __device__ __forceinline__ unsigned rank() const { return 0; }
    __device__ __forceinline__ unsigned size() const { return 1; }
    __device__ __forceinline__ double sum(double v) const { return bsum_all<BS>(v, s_w); }
    __device__ __forceinline__ double max(double v) const { return bmax_all<BS>(v, s_w); }
    __device__ __forceinline__ void sum3(double &a, double &b, double &c) const {
        bsum3_all<BS>(a, b, c, s_w);
    }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ double ld(const double *p) const { return *p; }
    __device__ __forceinline__ float ld(const float *p) const { return *p; }
};

template <int BS>
struct ClusterTeam {
    static constexpr bool kCluster = true;
    static constexpr int kBS = BS;
    unsigned r, sz;
    __device__ __forceinline__ int tid() const { return (int)r * BS + threadIdx.x; }
    __device__ __forceinline__ int stride() const { return BS * (int)sz; }
    __device__ __forceinline__ unsigned rank() const { return r; }
    __device__ __forceinline__ unsigned size() const { return sz; }
    __device__ __forceinline__ void sync() const { cooperative_groups::this_cluster().sync(); }
    __device__ __forceinline__ double ld(const double *p) const { return __ldcg(p); }
    __device__ __forceinline__ float ld(const float *p) const { return __ldcg(p); }
};

// gradient() of a whole line by a team (qew_model.h:149-193): edge pass into
// ev/es, barrier, site combine into g, barrier.
template <class Noise, class Team, class R>
__device__ void team_gradient(Team &T, const Noise &nz, const double *__restrict__ h, int n,
                              const LineDx &dx, double lt, double f, bool arc, R *ev, R *es,
                              R *g) {
    for (int e = T.tid(); e < n; e += T.stride()) {
        const int ep = (e + 1 == n) ? 0 : e + 1;
        double dv, sl;
        edge_gradient(nz, e, n, T.ld(h + e), T.ld(h + ep), dx, arc, dv, sl);
        ev[e] = (R)dv;
        es[e] = (R)sl;
    }
    T.sync();
    for (int i = T.tid(); i < n; i += T.stride()) {
        const int ip = (i + 1 == n) ? 0 : i + 1;
        const int im = (i == 0) ? n - 1 : i - 1;
        g[i] = (R)site_gradient<Noise>(T.ld(h + im), T.ld(h + i), T.ld(h + ip), (double)T.ld(ev + im),
                                (double)T.ld(ev + i), (double)T.ld(es + im), (double)T.ld(es + i),
                                dx, lt, f, arc);
    }
    T.sync();
}

// objective() at x0 + alpha*d by a team.
template <class Noise, class Team, class R>
__device__ double team_objective(Team &T, const Noise &nz, const double *__restrict__ x0,
                                 const R *__restrict__ d, double alpha, int n,
                                 const LineDx &dx, double lt, double f, int model) {
    double acc = 0.0;
    for (int i = T.tid(); i < n; i += T.stride()) {
        const int ip = (i + 1 == n) ? 0 : i + 1;
        const double hi = T.ld(x0 + i) + alpha * (double)T.ld(d + i);
        const double hip = T.ld(x0 + ip) + alpha * (double)T.ld(d + ip);
        acc += edge_energy(nz, i, ip, hi, hip, dx, lt, f, model);
    }
    return T.sum(acc);
}
