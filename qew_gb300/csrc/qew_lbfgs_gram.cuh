// qew_lbfgs_gram.cuh -- the FP64 lbfgs_minimize (lbfgs.h:94-287) of one line by
// a team of threads (one CTA, or one thread-block cluster), with the
// reductions of an iteration in three batches.
//
// What bound the loop written out as in the reference: 2 m + 4 broadcast
// reductions an iteration, each a barrier round trip and some 14 dependent
// FP64 additions (64 cycles apiece) behind the last, with the vectors fetched
// and stored between them. Here:
//   * the two-loop recursion runs on inner products. With S_i, Y_i the pairs
//     (i = 0 oldest) and q_i the vector before step i,
//       a_i = rho_i (S_i.g - sum_{j newer} a_j S_i.Y_j),  q = g - sum a_i Y_i,
//       b_i = rho_i (Y_i.d0 + sum_{j older} (a_j - b_j) Y_i.S_j),  d0 = M^-1 q,
//       d = -(d0 + sum (a_i - b_i) S_i),
//     the same recursion term by term: only products of an older S with a newer
//     Y enter, one new row an iteration, taken with s.y, s.s, y.y and S_i.g in
//     one batch after the step; Y_i.d0 and g.d0 are the second batch; the trial
//     energy is the third. Both triangular recursions are solved by one warp.
//   * a batch is folded eight values at a time (9 additions for eight values
//     instead of 40), then over the warps and the cluster's CTAs by butterflies.
//   * a thread owns consecutive points, so the preconditioner's recurrences
//     need scans only, and every vector but the line is private to its thread.
//     Boundary values of d travel once an iteration; the neighbours' heights
//     are advanced from them.
//   * a trial evaluates energy and dV/dy from one gather, so an accepted trial
//     needs no second one.
// One line of 4096 points (preconditioned, m = 10, 16 CTAs): 10.4-15.1 -> 2.5 ms
// a solve, 52 k cycles an iteration, most of them latencies: the two
// recurrences 8 k, the products 12 k, the trial 10 k. 768 lines of 256 to 4096
// points on all SMs: 68 -> 45 ms (two CTAs of 256 threads an SM; the long
// lines' vectors lie in L2 and memory, and their products take half the time).
#pragma once

#include "qew_team.cuh"
#include "qew_lbfgs_resident.cuh"

constexpr int kGramVals = 2 * kLbfgsMaxM + 8;  // values of the largest batch, rounded to 8

template <int BS>
struct GramShared {
    static constexpr int NW = BS / 32;
    double part[NW][kGramVals];
    unsigned long long pmax[NW];
    double red[kGramVals];
    double sy[kLbfgsMaxM][kLbfgsMaxM + 1];  // S_i.Y_j by row, older i, newer j
    double rho[kLbfgsMaxM], sg[kLbfgsMaxM], coef[kLbfgsMaxM];
    double scal[2];
    int slots[kLbfgsMaxM], sbuf[kLbfgsMaxM], ybuf[kLbfgsMaxM];
    int so[kLbfgsMaxM], yo[kLbfgsMaxM];  // sbuf, ybuf in chronological order
    int nslots, stmp, ytmp;
    double wagg[2][NW];        // warp aggregates of the scans
    double bd[2][NW + 1][4];   // boundary values between warps
    double z, inv, zl[5], zw[4], zc[4], zlane[32], zwarp[NW], zown, unpad;
};
template <bool kCluster>
struct GramExchange {};
template <>
struct GramExchange<true> {
    double val[2][kGramVals][kTeamMaxCtas];
    unsigned long long mx[2][kTeamMaxCtas];
    double agg[2][kTeamMaxCtas];
    double bd[2][4];
};

template <class Noise, class Team>
struct Gram {
    static constexpr int BS = Team::kBS;
    static constexpr int NW = BS / 32;
    static constexpr bool kCluster = Team::kCluster;
    Team &T;
    GramShared<BS> &s;
    GramExchange<kCluster> &x;
    int n, c, p0, cnt, na;  // points per thread, first point, points, active threads
    int lane, w, gt, G;
    double *zb_f, *zb_r;    // this thread's powers
    int ph = 0;             // buffer of the next exchange

    __device__ __forceinline__ void cta_or_cluster_sync() { T.sync(); }
    template <class V>
    __device__ __forceinline__ V *remote(V *p, int rank) {
        if constexpr (kCluster)
            return cooperative_groups::this_cluster().map_shared_rank(p, rank);
        else
            return p;
    }

    // ---- batched sums: put() groups of eight, then finish(K)
    __device__ __forceinline__ void put(double a[8], int g) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool up = lane & 16;
            const double send = up ? a[q] : a[q + 4], keep = up ? a[q + 4] : a[q];
            a[q] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const bool up = lane & 8;
            const double send = up ? a[q] : a[q + 2], keep = up ? a[q + 2] : a[q];
            a[q] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        {
            const bool up = lane & 4;
            const double send = up ? a[0] : a[1], keep = up ? a[1] : a[0];
            a[0] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
        }
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
        if ((lane & 3) == 0) s.part[w][8 * g + (lane >> 2)] = a[0];
    }
    __device__ __forceinline__ void put1(double a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) s.part[w][0] = a;
    }
    // largest of non-negative doubles by their bits
    static __device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
        const unsigned hi = (unsigned)(v >> 32);
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)v : 0u);
        return ((unsigned long long)mh << 32) | ml;
    }
    __device__ __forceinline__ void put_max(unsigned long long v) {
        v = warp_max(v);
        if (lane == 0) s.pmax[w] = v;
    }
    // Sums of the K values put, into s.red (every thread may read it after);
    // with_max: also the largest of put_max's, returned.
    __device__ __forceinline__ double finish(int K, bool with_max) {
        __syncthreads();
        constexpr int PER = 32;  // values a pass: NW lanes each
        const int v0 = threadIdx.x / NW, q = threadIdx.x % NW;
        for (int b = 0; b < K; b += PER) {
            const int v = b + v0;
            double a = v < K ? s.part[q][v] : 0.0;
#pragma unroll
            for (int o = NW / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            if (v < K) {
                if constexpr (kCluster) {
                    for (unsigned r = q; r < T.size(); r += NW) remote(&x.val[ph][v][T.rank()], r)[0] = a;
                } else if (q == 0) {
                    s.red[v] = a;
                }
            }
        }
        unsigned long long m = 0;
        if (with_max) {
            m = warp_max(lane < NW ? s.pmax[lane] : 0ull);
            if constexpr (kCluster) {
                if (threadIdx.x < T.size()) remote(&x.mx[ph][T.rank()], threadIdx.x)[0] = m;
            }
        }
        cta_or_cluster_sync();
        if constexpr (kCluster) {
            const int r = threadIdx.x % kTeamMaxCtas;
            for (int b = 0; b < K; b += BS / kTeamMaxCtas) {
                const int v = b + threadIdx.x / kTeamMaxCtas;
                double a = (v < K && r < (int)T.size()) ? x.val[ph][v][r] : 0.0;
#pragma unroll
                for (int o = kTeamMaxCtas / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (v < K && r == 0) s.red[v] = a;
            }
            if (with_max) m = warp_max(lane < (int)T.size() ? x.mx[ph][lane] : 0ull);
            ph ^= 1;
            __syncthreads();
        }
        return __longlong_as_double((long long)m);
    }
    __device__ __forceinline__ double sum1(double v) {
        put1(v);
        finish(1, false);
        return s.red[0];
    }

    // ---- boundary values: prev = the preceding thread's `last`, next = the
    // following thread's `first` (threads in a ring of the na active ones)
    __device__ __forceinline__ void neighbours(double first, double last, double &prev,
                                               double &next) {
        const int b = ph;
        const int lw = BS / 32 - 1;
        prev = __shfl_up_sync(0xffffffffu, last, 1);
        next = __shfl_down_sync(0xffffffffu, first, 1);
        const bool is_last = gt == na - 1;
        if (cnt > 0) {
            if (lane == 31 || is_last) {  // `last` to the next warp, CTA, or the ring's start
                if (is_last) {
                    if constexpr (kCluster) remote(&x.bd[b][0], 0)[0] = last;
                    else s.bd[b][0][0] = last;
                } else if (w == lw) {
                    if constexpr (kCluster) remote(&x.bd[b][0], (int)T.rank() + 1)[0] = last;
                } else {
                    s.bd[b][w + 1][0] = last;
                }
            }
            if (lane == 0) {  // `first` to the warp, CTA before, or the ring's end
                if (gt == 0) {
                    if constexpr (kCluster) remote(&x.bd[b][2], (na - 1) / BS)[0] = first;
                    else s.bd[b][NW][2] = first;
                } else if (w == 0) {
                    if constexpr (kCluster) remote(&x.bd[b][1], (int)T.rank() - 1)[0] = first;
                } else {
                    s.bd[b][w][1] = first;
                }
            }
        }
        cta_or_cluster_sync();
        if (lane == 0) {
            if (w == 0) {
                if constexpr (kCluster) prev = x.bd[b][0];
                else prev = s.bd[b][0][0];
            } else {
                prev = s.bd[b][w][0];
            }
        }
        if (is_last) {
            if constexpr (kCluster) next = x.bd[b][2];
            else next = s.bd[b][NW][2];
        } else if (lane == 31) {
            if (w == lw) {
                if constexpr (kCluster) next = x.bd[b][1];
            } else {
                next = s.bd[b][w + 1][1];
            }
        }
        ph ^= 1;
    }
    // the preceding thread's two values
    __device__ __forceinline__ void from_prev(double v0, double v1, double &r0, double &r1) {
        const int b = ph;
        r0 = __shfl_up_sync(0xffffffffu, v0, 1);
        r1 = __shfl_up_sync(0xffffffffu, v1, 1);
        const bool is_last = gt == na - 1;
        if (cnt > 0 && (lane == 31 || is_last)) {
            double *to;
            if (is_last) {
                if constexpr (kCluster) to = remote(&x.bd[b][0], 0);
                else to = &s.bd[b][0][0];
            } else if (w == BS / 32 - 1) {
                if constexpr (kCluster) to = remote(&x.bd[b][0], (int)T.rank() + 1);
                else to = &s.bd[b][0][0];  // unreached: the CTA's last thread is the ring's last
            } else {
                to = &s.bd[b][w + 1][0];
            }
            to[0] = v0;
            to[3] = v1;
        }
        cta_or_cluster_sync();
        if (lane == 0) {
            const double *from;
            if (w == 0) {
                if constexpr (kCluster) from = &x.bd[b][0];
                else from = &s.bd[b][0][0];
            } else {
                from = &s.bd[b][w][0];
            }
            r0 = from[0];
            r1 = from[3];
        }
        ph ^= 1;
    }

    // ---- the periodic recurrence y_k = x_k + z y_(k-1) over the points in
    // order (rev: in reverse order), in place on the thread's own values v (stride
    // ps), times gain.
    // Powers of z (GramShared): zl[j] = z^(c 2^j), a warp's scan multipliers;
    // zw[j] = z^(32 c 2^j); zc[j] = z^(BS c 2^j); zlane, zwarp of the points of
    // the threads before in the warp, of the warps before in the CTA; zown of
    // the last chunk; zb of all points before a thread's, in either order. Every thread's chunk
    // counts c points, the last ones' missing points as zero input; the
    // periodic value comes from the last point's owner.
    __device__ __forceinline__ void make_scan(const PrecondCoef &pc) {
        auto pw = [&](double k) { return exp(k * pc.logz); };
        const int t = threadIdx.x;
        if (t < 5) s.zl[t] = pw((double)c * (1 << t));
        if (t < 4) {
            s.zw[t] = pw(32.0 * c * (1 << t));
            s.zc[t] = pw((double)BS * c * (1 << t));
        }
        if (t < 32) s.zlane[t] = pw((double)c * t);
        if (t < NW) s.zwarp[t] = pw(32.0 * c * t);
        if (t == 0) {
            s.z = pc.z;
            s.inv = pc.inv_1mzn;
            s.zown = pw((double)(n - (na - 1) * c));
            const double missing = (double)c * G - (double)n;
            s.unpad = -missing * pc.logz < 500.0 ? pw(-missing) : 0.0;
        }
        zb_f[0] = pw(p0);
        zb_r[0] = pw((double)n - p0 - cnt);
    }
    __device__ __forceinline__ void recurrence(double *v, int ps, bool rev, double gain) {
        const double z = s.z;
        double B = 0.0;
        for (int k = 0; k < cnt; ++k) B = fma(z, B, v[(rev ? cnt - 1 - k : k) * ps]);
        // threads in scan order: idx 0..na-1 (rev: from the ring's end)
        const double own = B;
        if (cnt < c && !rev)
            for (int k = cnt; k < c; ++k) B *= z;
        // Reverse order: the last active thread is first and may be short; it
        // then simply covers fewer points, which its zero start makes exact.
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            const double p = rev ? __shfl_down_sync(0xffffffffu, B, 1 << j)
                                 : __shfl_up_sync(0xffffffffu, B, 1 << j);
            const bool in = rev ? lane + (1 << j) < 32 : lane >= (1 << j);
            if (in) B = fma(s.zl[j], p, B);
        }
        double before = rev ? __shfl_down_sync(0xffffffffu, B, 1) : __shfl_up_sync(0xffffffffu, B, 1);
        if (lane == (rev ? 31 : 0)) before = 0.0;
        const int b = ph;
        if (lane == (rev ? 0 : 31)) s.wagg[b][w] = B;
        __syncthreads();
        // inclusive value at the end of every warp of the CTA, by lanes
        double A = lane < NW ? s.wagg[b][rev ? NW - 1 - lane : lane] : 0.0;
#pragma unroll
        for (int j = 0; (1 << j) < NW; ++j) {
            const double p = __shfl_up_sync(0xffffffffu, A, 1 << j);
            if (lane >= (1 << j)) A = fma(s.zw[j], p, A);
        }
        const int wi = rev ? NW - 1 - w : w;  // warp in scan order
        double wbefore = __shfl_sync(0xffffffffu, A, wi > 0 ? wi - 1 : 0);
        if (wi == 0) wbefore = 0.0;
        double cbefore = 0.0, total = __shfl_sync(0xffffffffu, A, NW - 1);
        if constexpr (kCluster) {
            if (threadIdx.x < T.size()) remote(&x.agg[b][T.rank()], threadIdx.x)[0] = total;
            T.sync();
            const int sz = (int)T.size();
            double Q = lane < sz ? x.agg[b][rev ? sz - 1 - lane : lane] : 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double p = __shfl_up_sync(0xffffffffu, Q, 1 << j);
                if (lane >= (1 << j)) Q = fma(s.zc[j], p, Q);
            }
            const int ci = rev ? sz - 1 - (int)T.rank() : (int)T.rank();
            cbefore = __shfl_sync(0xffffffffu, Q, ci > 0 ? ci - 1 : 0);
            if (ci == 0) cbefore = 0.0;
            total = __shfl_sync(0xffffffffu, Q, sz - 1);
        }
        // zero-start value before this thread's chunk: thread in warp, warps, CTAs
        const double start = fma(s.zlane[rev ? 31 - lane : lane],
                                 fma(s.zwarp[wi], cbefore, wbefore), before);
        // the periodic start: the zero-start value at the last point. In reverse
        // order it is the scan's total; forward, the total of the padded ring,
        // which ran on for the missing points (unpad = z^-missing), or, where
        // that could underflow, the last point's owner's.
        double yend;
        if (rev || s.unpad > 0.0) {
            yend = rev ? total : s.unpad * total;
        } else {
            if (gt == na - 1) s_end(b, fma(s.zown, start, own));
            cta_or_cluster_sync();
            yend = end_value(b);
        }
        const double P = s.inv * yend;
        // z^(points before this chunk)
        double y = fma(rev ? *zb_r : *zb_f, P, start);
        for (int k = 0; k < cnt; ++k) {
            double *q = v + (rev ? cnt - 1 - k : k) * ps;
            y = fma(z, y, *q);
            *q = gain * y;
        }
        ph ^= 1;
    }
    __device__ __forceinline__ void s_end(int b, double v) {
        if constexpr (kCluster) {
            for (unsigned r = 0; r < T.size(); ++r) remote(&x.bd[b][3], r)[0] = v;
        } else {
            s.bd[b][NW][3] = v;
        }
    }
    __device__ __forceinline__ double end_value(int b) const {
        if constexpr (kCluster) return x.bd[b][3];
        else return s.bd[b][NW][3];
    }
};

// Padded length of a solver vector: ceil(n / G) points for each of G threads.
__host__ __device__ __forceinline__ size_t gram_npad(int n, int G) {
    return (size_t)((n + G - 1) / G) * (size_t)G;
}

// lbfgs_minimize by team T. ws: this CTA's part of the solver's vectors, each
// ceil(n / G) x BS doubles (point k of thread t at k BS + t; nothing but its
// owner reads it), in shared memory where it fits, else in global memory.
template <class Noise, class Team>
__device__ qew_lbfgs_result lbfgs_gram(Team &T, const Noise &nz, double *__restrict__ h, const int n,
                                       const qew_params P, const LbfgsCfg cfg, const PrecondCoef pc,
                                       double *ws) {
    __shared__ GramShared<Team::kBS> sh;
    __shared__ GramExchange<Team::kCluster> shx;
    Gram<Noise, Team> W{T, sh, shx};
    const int lane = threadIdx.x & 31;
    const int gt = T.tid(), G = T.stride();
    W.n = n;
    W.lane = lane;
    W.w = threadIdx.x >> 5;
    W.gt = gt;
    W.G = G;
    const int c = W.c = (n + G - 1) / G;
    const int p0 = W.p0 = min(gt * c, n);
    const int cnt = W.cnt = min(c, n - p0);
    W.na = (n + c - 1) / c;
    const LineDx L = make_line_dx(P.physical_size, n, P.line_tension, P.driving_force);
    const double lt = P.line_tension;
    const bool arc = (P.model == QEW_MODEL_ARCLENGTH);
    const int m = cfg.m;
    constexpr int PS = Team::kBS;
    const int len = c * PS;
    auto vec = [&](int b) { return ws + (size_t)b * len + threadIdx.x; };
    double *g = vec(0), *gn = vec(1), *d = vec(2), *ev = vec(5), *es = vec(6);
    auto row = [&](int b) { return vec(kLbfgsVecs + b); };
    auto at = [&](int k) { return k * PS; };
    if (threadIdx.x == 0) {
        sh.nslots = 0;
        for (int k = 0; k < m; ++k) {
            sh.sbuf[k] = k;
            sh.ybuf[k] = m + 1 + k;
        }
        sh.stmp = m;
        sh.ytmp = 2 * m + 1;
    }
    W.zb_f = vec(3);
    W.zb_r = vec(4);
    if (cfg.precondition && !pc.scalar) W.make_scan(pc);
    // the neighbours' heights, advanced with theirs from here on
    double hl = cnt ? T.ld(h + (p0 == 0 ? n - 1 : p0 - 1)) : 0.0;
    double hr = cnt ? T.ld(h + (p0 + cnt == n ? 0 : p0 + cnt)) : 0.0;
    T.sync();

    // energy and dV/dy (ev, es) of the own edges on the line h + alpha d
    auto trial = [&](double alpha, double dr) {
        double acc = 0.0;
        double x0 = cnt ? fma(alpha, d[at(0)], h[p0]) : 0.0;
        for (int k = 0; k < cnt; ++k) {
            const double x1 = k + 1 < cnt ? fma(alpha, d[at(k + 1)], h[p0 + k + 1]) : fma(alpha, dr, hr);
            const int e = p0 + k, ep = e + 1 == n ? 0 : e + 1;
            double v, dv;
            noise_both_edge(nz, e, EdgeX{e + ep, L.dx}, x0 + x1, v, dv);
            const double dh = L.slope(x1 - x0);
            double el;
            if (arc) {
                const double w = fx_invroot(dh);
                es[at(k)] = dh * w;
                el = lt * fma(fma(dh, dh, 1.0), w, -1.0);
            } else {
                el = 0.5 * lt * dh * dh;
            }
            ev[at(k)] = dv;
            acc += fma(-P.driving_force, x0, el + v);
            x0 = x1;
        }
        return W.sum1(acc) * L.dx;
    };
    // gradient into o from the edges of the last trial(alpha, dr) (dl: the left
    // neighbour's d)
    auto gradient = [&](double alpha, double dl, double dr, double *o) {
        double dvl, sll;
        W.from_prev(cnt ? ev[at(cnt - 1)] : 0.0, cnt && arc ? es[at(cnt - 1)] : 0.0, dvl, sll);
        double xm = fma(alpha, dl, hl), x0 = cnt ? fma(alpha, d[at(0)], h[p0]) : 0.0;
        for (int k = 0; k < cnt; ++k) {
            const double x1 = k + 1 < cnt ? fma(alpha, d[at(k + 1)], h[p0 + k + 1]) : fma(alpha, dr, hr);
            const double dv = ev[at(k)], sl = arc ? es[at(k)] : 0.0;
            o[at(k)] = site_gradient<Noise>(xm, x0, x1, dvl, dv, sll, sl, L, lt, 0.0, arc);
            xm = x0;
            x0 = x1;
            dvl = dv;
            sll = sl;
        }
    };
    // |v| in an order of its bits; a NaN does not count, as with fmax
    auto abs_bits = [](double v) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
        return b > 0x7FF0000000000000ull ? 0ull : b;
    };

    qew_lbfgs_result res;
    res.iterations = 0;
    res.max_force = 0;
    res.converged = 0;
    res.n_func_evals = 0;
    res.n_curvature_skips = 0;
    res.n_ls_restarts = 0;
    double phi = 0.0, gmax = 0.0;
    int ls_fail_streak = 0;
    bool done = false;

    for (int k = 0; k < cnt; ++k) d[at(k)] = 0.0;
    const double phi_first = trial(0.0, 0.0);
    gradient(0.0, 0.0, 0.0, g);
    {
        unsigned long long mx = 0;
        for (int k = 0; k < cnt; ++k) mx = max(mx, abs_bits(g[at(k)]));
        W.put_max(mx);
        gmax = W.finish(0, true);
    }
    for (int it = 0; it < cfg.max_iter; ++it) {
        if (gmax < cfg.ftol) {  // lbfgs.h:155-161
            res.iterations = it;
            res.max_force = gmax;
            res.converged = 1;
            done = true;
            break;
        }
        // two-loop recursion, lbfgs.h:163-191, on inner products
        const int hs = sh.nslots;
        if (W.w == 0 && hs > 0) {  // lane i: slot i in chronological order
            const int r = lane < hs ? sh.slots[lane] : 0;
            double t = lane < hs ? sh.sg[r] : 0.0, mine = 0.0;
            const double rho = lane < hs ? sh.rho[r] : 0.0;
            for (int j = hs - 1; j >= 0; --j) {
                const double a = __shfl_sync(0xffffffffu, rho * t, j);
                if (lane == j) mine = a;
                if (lane < j) t = fma(-a, sh.sy[r][sh.slots[j]], t);
            }
            if (lane < hs) sh.coef[lane] = mine;
        }
        __syncthreads();
        for (int k = 0; k < cnt; ++k) {
            double q = g[at(k)];
            for (int i = hs - 1; i >= 0; --i)
                q = fma(-sh.coef[i], row(sh.yo[i])[at(k)], q);
            if (!cfg.precondition)
                q *= (hs == 0) ? 1.0 : sh.scal[1];
            else if (pc.scalar)
                q *= pc.inv_sigma;
            d[at(k)] = q;
        }
        if (cfg.precondition && !pc.scalar) {
            W.recurrence(d, PS, false, 1.0);
            W.recurrence(d, PS, true, pc.gain);
        }
        // g.d0 and Y_i.d0
        for (int gi = 0; gi * 8 < hs + 1; ++gi) {
            double a[8] = {};
            for (int k = 0; k < cnt; ++k) {
                const double dv = d[at(k)];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int v = 8 * gi + q;
                    if (v <= hs)
                        a[q] = fma(v == 0 ? g[at(k)] : row(sh.yo[v - 1])[at(k)], dv, a[q]);
                }
            }
            W.put(a, gi);
        }
        W.finish(hs + 1, false);
        if (W.w == 0) {
            const int r = lane < hs ? sh.slots[lane] : 0;
            double t = lane < hs ? sh.red[1 + lane] : 0.0;
            const double rho = lane < hs ? sh.rho[r] : 0.0, a = lane < hs ? sh.coef[lane] : 0.0;
            double mine = 0.0;
            for (int j = 0; j < hs; ++j) {
                const double cj = __shfl_sync(0xffffffffu, fma(-rho, t, a), j);
                if (lane == j) mine = cj;
                if (lane > j && lane < hs) t = fma(cj, sh.sy[sh.slots[j]][r], t);
            }
            double e = lane < hs ? mine * sh.sg[r] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            __syncwarp();
            if (lane < hs) sh.coef[lane] = mine;
            if (lane == 0) sh.scal[0] = -(sh.red[0] + e);  // g.d
        }
        __syncthreads();
        double dphi0 = sh.scal[0];
        bool empty = (hs == 0);
        if (dphi0 >= 0) {  // steepest-descent fallback, lbfgs.h:195-200
            empty = true;
            double gg = 0.0;
            for (int k = 0; k < cnt; ++k) {
                const double v = g[at(k)];
                d[at(k)] = -v;
                gg = fma(v, v, gg);
            }
            dphi0 = -W.sum1(gg);
            if (threadIdx.x == 0) sh.nslots = 0;
        } else {
            for (int k = 0; k < cnt; ++k) {
                double v = -d[at(k)];
                for (int i = 0; i < hs; ++i)
                    v = fma(-sh.coef[i], row(sh.so[i])[at(k)], v);
                d[at(k)] = v;
            }
        }
        double dl, dr;
        W.neighbours(cnt ? d[at(0)] : 0.0, cnt ? d[at(cnt - 1)] : 0.0, dl, dr);
        // Armijo backtracking, lbfgs.h:202-238
        if (it == 0) {
            phi = phi_first;
            ++res.n_func_evals;
        }
        const double phi0 = phi;
        double alpha = 1.0;
        if (!cfg.precondition && empty) {
            double gg = 0.0;
            for (int k = 0; k < cnt; ++k) gg = fma(g[at(k)], g[at(k)], gg);
            alpha = 1.0 / fmax(1.0, sqrt(W.sum1(gg)));
        }
        bool ok = false, have_gn = false;
        for (int ls = 0; ls < cfg.max_ls; ++ls) {
            const double pt = trial(alpha, dr);
            ++res.n_func_evals;
            if (pt <= phi0 + cfg.c1 * alpha * dphi0) {
                phi = pt;
                ok = true;
                break;
            }
            if (cfg.ls_fallback) {  // slope test at the trial point
                gradient(alpha, dl, dr, gn);
                double sd = 0.0;
                for (int k = 0; k < cnt; ++k) sd = fma(gn[at(k)], d[at(k)], sd);
                const double dphia = W.sum1(sd);
                ++res.n_func_evals;
                if (dphia >= kAwSigma * dphi0 && dphia <= (2.0 * kAwDelta - 1.0) * dphi0 &&
                    pt <= phi0 + kAwEps * fabs(phi0)) {
                    phi = pt;
                    ok = true;
                    have_gn = true;  // gn already holds the gradient at the new point
                    break;
                }
            }
            alpha *= cfg.ls_shrink;
        }
        if (!ok) {
            if (empty || ++ls_fail_streak > 2) {
                res.iterations = it;
                res.max_force = gmax;
                res.converged = 0;
                done = true;
                break;
            }
            __syncthreads();
            if (threadIdx.x == 0) sh.nslots = 0;
            ++res.n_ls_restarts;
            __syncthreads();
            continue;
        }
        ls_fail_streak = 0;
        if (!have_gn) gradient(alpha, dl, dr, gn);
        for (int k = 0; k < cnt; ++k) h[p0 + k] = fma(alpha, d[at(k)], h[p0 + k]);  // lbfgs.h:243-244
        hl = fma(alpha, dl, hl);
        hr = fma(alpha, dr, hr);
        // the new pair and its products, lbfgs.h:250-261, with S_i.g, S_i.y
        double *sT = row(sh.stmp), *yT = row(sh.ytmp);
        const int hs2 = sh.nslots;
        {
            double a[8] = {};
            unsigned long long mx = 0;
            const double *S0 = hs2 > 0 ? row(sh.so[0]) : nullptr;
            const double *S1 = hs2 > 1 ? row(sh.so[1]) : nullptr;
            for (int k = 0; k < cnt; ++k) {
                const double gk = gn[at(k)];
                const double sv = alpha * d[at(k)], y = gk - g[at(k)];
                sT[at(k)] = sv;
                yT[at(k)] = y;
                mx = max(mx, abs_bits(gk));
                a[0] = fma(sv, y, a[0]);
                a[1] = fma(sv, sv, a[1]);
                a[2] = fma(y, y, a[2]);
                a[3] = fma(sv, gk, a[3]);
                if (S0) {
                    const double q = S0[at(k)];
                    a[4] = fma(q, gk, a[4]);
                    a[5] = fma(q, y, a[5]);
                }
                if (S1) {
                    const double q = S1[at(k)];
                    a[6] = fma(q, gk, a[6]);
                    a[7] = fma(q, y, a[7]);
                }
            }
            W.put(a, 0);
            W.put_max(mx);
        }
        for (int gi = 1; 4 * gi - 2 < hs2; ++gi) {
            double a[8] = {};
            for (int k = 0; k < cnt; ++k) {
                const double gk = gn[at(k)], y = yT[at(k)];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int i = 4 * gi - 2 + q;
                    if (i < hs2) {
                        const double sv = row(sh.so[i])[at(k)];
                        a[2 * q] = fma(sv, gk, a[2 * q]);
                        a[2 * q + 1] = fma(sv, y, a[2 * q + 1]);
                    }
                }
            }
            W.put(a, gi);
        }
        gmax = W.finish(4 + 2 * hs2, true);
        if (W.w == 0) {
            const double sy = sh.red[0], ss = sh.red[1], yy = sh.red[2];
            const bool keep = sy > cfg.curvature_eps * sqrt(ss * yy);  // lbfgs.h:262-279
            if (!keep) ++res.n_curvature_skips;
            if (lane < hs2) sh.sg[sh.slots[lane]] = sh.red[4 + 2 * lane];
            __syncwarp();
            if (keep) {
                const bool full = hs2 == m;
                const int r = full ? sh.slots[0] : hs2;
                const int mine = lane + (full ? 1 : 0) < hs2 ? sh.slots[lane + (full ? 1 : 0)] : -1;
                const double q = mine >= 0 ? sh.red[5 + 2 * (lane + (full ? 1 : 0))] : 0.0;
                __syncwarp();
                if (mine >= 0) {
                    sh.slots[lane] = mine;
                    sh.sy[mine][r] = q;
                }
                if (lane == 0) {
                    int tmp = sh.sbuf[r];
                    sh.sbuf[r] = sh.stmp;
                    sh.stmp = tmp;
                    tmp = sh.ybuf[r];
                    sh.ybuf[r] = sh.ytmp;
                    sh.ytmp = tmp;
                    sh.rho[r] = 1.0 / sy;
                    if (!cfg.precondition) sh.scal[1] = sy / yy;
                    sh.sg[r] = sh.red[3];
                    const int last = full ? hs2 - 1 : hs2;
                    sh.slots[last] = r;
                    sh.nslots = last + 1;
                }
                __syncwarp();
                if (lane < sh.nslots) {
                    sh.so[lane] = sh.sbuf[sh.slots[lane]];
                    sh.yo[lane] = sh.ybuf[sh.slots[lane]];
                }
            }
        }
        __syncthreads();
        double *tg = g;
        g = gn;
        gn = tg;
    }
    if (!done) {  // lbfgs.h:283-286
        res.iterations = cfg.max_iter;
        res.max_force = gmax;
        res.converged = 0;
    }
    return res;  // warp 0's counts the skipped pairs
}

// Doubles of one CTA's part of the vectors.
__host__ __device__ __forceinline__ size_t gram_ws(int n, int G, int bs, int m) {
    return (size_t)((n + G - 1) / G) * (size_t)bs * (size_t)(kLbfgsVecs + 2 * (m + 1));
}

// One CTA runs the whole solve.
template <class Noise, int BS>
__device__ qew_lbfgs_result lbfgs_gram_block(const Noise &nz, double *__restrict__ h, const int n,
                                             const qew_params P, const LbfgsCfg cfg,
                                             const PrecondCoef pc, double *ws) {
    CtaTeam<BS> T{nullptr};
    return lbfgs_gram<Noise, CtaTeam<BS>>(T, nz, h, n, P, cfg, pc, ws);
}
