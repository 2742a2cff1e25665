// qew_rk_device.cuh -- device functions of the Rosso-Krauth construction
// (rosso_krauth.h:51-124): the single-site velocity and the nearest forward
// velocity zero (march, then bisect).
#pragma once

#include "qew_internal.cuh"
#include "qew_model_kernels.cuh"

struct RkP {
    double dstep, max_advance, root_tol, sweep_tol, runaway;
    int max_sweeps;
};

inline RkP rkp_from(const qew_rk_params *rp) {
    return RkP{rp->dstep, rp->max_advance, rp->root_tol, rp->sweep_tol, rp->runaway, rp->max_sweeps};
}

// The elastic force of a site as the reference evaluates it (unfused where a
// contraction would change 1 + s^2; the rest rounds the same either way), for
// the reference-exact velocity.
__device__ __forceinline__ double rk_line_force_ref(double dx, double lt, int model, double hi,
                                                    double hl, double hr) {
    if (model == QEW_MODEL_LINEAR) return -lt * (hl + hr - 2.0 * hi) / (dx * dx);
    const double dhr = (hr - hi) / dx;
    const double dhl = (hi - hl) / dx;
    return lt *
           (dhl / sqrt(__dadd_rn(1.0, __dmul_rn(dhl, dhl))) -
            dhr / sqrt(__dadd_rn(1.0, __dmul_rn(dhr, dhr)))) /
           dx;
}

// rk_site_velocity, rosso_krauth.h:51-82: exactly -gradient_i, from the two
// edges' dV/dy. Every operation is written out, so that each kernel gets the
// same bits; with the reference-exact functor they are the reference's.
template <class Noise>
__device__ __forceinline__ double rk_velocity_of(double dvl, double dvr, const LineDx &L, double lt,
                                                 double f, int model, double hi, double hl,
                                                 double hr) {
    if constexpr (noise_is_ref<Noise>::value) {
        const double grad = L.dx * (rk_line_force_ref(L.dx, lt, model, hi, hl, hr) +
                                    0.5 * (dvl + dvr) - f);
        return -grad;
    } else {
        const double rest = fma(L.half_dx, __dadd_rn(dvl, dvr), -L.fdx);
        if (model == QEW_MODEL_LINEAR) return -fma(L.c_el, fma(-2.0, hi, __dadd_rn(hl, hr)), rest);
        const double sll = fx_slope(L.slope(__dsub_rn(hi, hl)));
        const double slr = fx_slope(L.slope(__dsub_rn(hr, hi)));
        return -fma(lt, __dsub_rn(sll, slr), rest);
    }
}

template <class Noise>
__device__ __forceinline__ double rk_site_velocity(const Noise &nz, int i, int n, const LineDx &L,
                                                   double lt, double f, int model, double hi,
                                                   double hl, double hr) {
    const int im = (i == 0) ? n - 1 : i - 1;
    const int ip = (i + 1 == n) ? 0 : i + 1;
    const EdgeX xcl{im + i, L.dx}, xcr{i + ip, L.dx};
    const double dvl = noise_dvdy_edge(nz, im, xcl, __dadd_rn(hl, hi));  // edge (im, i)
    const double dvr = noise_dvdy_edge(nz, i, xcr, __dadd_rn(hi, hr));   // edge (i, ip)
    return rk_velocity_of<Noise>(dvl, dvr, L, lt, f, model, hi, hl, hr);
}

// rk_forward_zero, rosso_krauth.h:88-124. The march is bounded by
// max_advance/dstep steps, the bisection by 60.
template <class Noise>
__device__ __forceinline__ double rk_forward_zero(const Noise &nz, int i, int n, const LineDx &dx,
                                                  double lt, double f, int model, double hi,
                                                  double hl, double hr, const RkP &rp,
                                                  bool &found) {
    const double v0 = rk_site_velocity(nz, i, n, dx, lt, f, model, hi, hl, hr);
    if (v0 <= 0) {
        found = true;
        return hi;
    }
    double a = hi;
    double advanced = 0;
    while (advanced < rp.max_advance) {
        const double b = a + rp.dstep;
        const double vb = rk_site_velocity(nz, i, n, dx, lt, f, model, b, hl, hr);
        if (vb <= 0) {
            double lo = a, hc = b;
            for (int k = 0; k < 60 && (hc - lo) > rp.root_tol; ++k) {
                const double mid = 0.5 * (lo + hc);
                const double vm = rk_site_velocity(nz, i, n, dx, lt, f, model, mid, hl, hr);
                if (vm > 0)
                    lo = mid;
                else
                    hc = mid;
            }
            found = true;
            return 0.5 * (lo + hc);
        }
        a = b;
        advanced += rp.dstep;
    }
    found = false;
    return a;
}

// rk_forward_zero evaluated by a group of G lanes (G = 2, 4, 8, 16 or 32; the
// G lanes of one aligned G-lane slice of the warp, `lane` = 0..G-1 within it,
// all with the same site and neighbours). It returns exactly what
// rk_forward_zero returns: every velocity it compares is computed from the
// same operands by the same code, and the search is replayed step by step
// from those comparisons; only the evaluations are spread over the lanes.
//   * march: lane j evaluates the point the serial loop reaches after j + 1
//     steps of a round (each lane redoes the round's additions of dstep, so
//     its point is the serial one bit for bit); the first lane with v <= 0
//     brackets the zero, as the serial loop would have found it;
//   * bisection: lane j (1 <= j < G) evaluates node j of the next
//     log2(G)-level subtree of midpoints (heap order, each node's interval
//     replayed from the root with the serial midpoint formula); the walk down
//     the subtree then applies the serial loop's test and update per level.
template <int G, class Noise>
__device__ __forceinline__ double rk_forward_zero_group(const Noise &nz, int i, int n, const LineDx &dx,
                                                        double lt, double f, int model, double hi,
                                                        double hl, double hr, const RkP &rp,
                                                        bool &found, int lane, unsigned gmask) {
    static_assert(G >= 2 && G <= 32 && (G & (G - 1)) == 0, "G must be a power of two <= 32");
    constexpr int kLevels = (G >= 32) ? 5 : (G >= 16) ? 4 : (G >= 8) ? 3 : (G >= 4) ? 2 : 1;
    const double v0 = rk_site_velocity(nz, i, n, dx, lt, f, model, hi, hl, hr);
    if (v0 <= 0) {
        found = true;
        return hi;
    }
    double a = hi, advanced = 0.0;
    double lo = 0.0, hc = 0.0;
    bool bracketed = false;
    // The serial march takes at most ceil(max_advance / dstep) steps
    // (validated on the host), so this loop ends.
    while (!bracketed) {
        // this lane's point: j + 1 serial steps from (a, advanced)
        double la = a, ladv = advanced, b = a;
        bool valid = true;
        for (int t = 0; t <= lane; ++t) {
            if (!(ladv < rp.max_advance)) {
                valid = false;
                break;
            }
            b = la + rp.dstep;
            if (t < lane) {
                la = b;
                ladv += rp.dstep;
            }
        }
        const double vb = valid ? rk_site_velocity(nz, i, n, dx, lt, f, model, b, hl, hr) : 1.0;
        const unsigned shift = (unsigned)(threadIdx.x & 31) & ~(unsigned)(G - 1);
        const unsigned okm = (__ballot_sync(gmask, valid) >> shift) & ((G == 32) ? ~0u : ((1u << G) - 1));
        const unsigned hitm = (__ballot_sync(gmask, valid && vb <= 0) >> shift) &
                              ((G == 32) ? ~0u : ((1u << G) - 1));
        if (hitm) {
            const int j = __ffs(hitm) - 1;
            lo = __shfl_sync(gmask, la, j, G);
            hc = __shfl_sync(gmask, b, j, G);
            bracketed = true;
        } else {
            const bool all_ok = okm == ((G == 32) ? ~0u : ((1u << G) - 1));
            if (!all_ok) {
                // the march ran out of max_advance: the serial loop returns the
                // last point it stepped to (or a, when no step was possible)
                found = false;
                if (okm == 0) return a;
                const int last = 31 - __clz(okm);
                return __shfl_sync(gmask, b, last, G);
            }
            a = __shfl_sync(gmask, b, G - 1, G);
            advanced = __shfl_sync(gmask, ladv + rp.dstep, G - 1, G);
        }
    }
    // bisection: for (k = 0; k < 60 && (hc - lo) > root_tol; ++k)
    int k = 0;
    while (true) {
        // node `lane` (1..G-1) of the subtree rooted at the current interval
        double vm = 0.0;
        if (lane >= 1) {
            const int depth = 31 - __clz(lane);
            double l2 = lo, h2 = hc;
            for (int d = depth - 1; d >= 0; --d) {
                const double mid = 0.5 * (l2 + h2);
                if ((lane >> d) & 1)
                    l2 = mid;
                else
                    h2 = mid;
            }
            vm = rk_site_velocity(nz, i, n, dx, lt, f, model, 0.5 * (l2 + h2), hl, hr);
        }
        int node = 1;
        bool done = false;
        for (int level = 0; level < kLevels; ++level) {
            if (!(k < 60 && (hc - lo) > rp.root_tol)) {
                done = true;
                break;
            }
            const double mid = 0.5 * (lo + hc);
            const double v = __shfl_sync(gmask, vm, node, G);
            if (v > 0) {
                lo = mid;
                node = 2 * node + 1;
            } else {
                hc = mid;
                node = 2 * node;
            }
            ++k;
        }
        if (done || !(k < 60 && (hc - lo) > rp.root_tol)) break;
    }
    found = true;
    return 0.5 * (lo + hc);
}

// rk_site_velocity evaluated by a lane pair (lanes `lane` = 0 and 1 of an
// aligned pair, same site and heights): each lane gathers one of the two edge
// midpoints, the other one's value comes by shuffle, and both finish the
// same expression -- the value is rk_site_velocity's bit for bit.
template <class Noise>
__device__ __forceinline__ double rk_site_velocity_pair(const Noise &nz, int i, int n,
                                                        const LineDx &L, double lt, double f,
                                                        int model, double hi, double hl, double hr,
                                                        int lane, unsigned pmask) {
    const int im = (i == 0) ? n - 1 : i - 1;
    const int ip = (i + 1 == n) ? 0 : i + 1;
    const EdgeX xc{lane ? i + ip : im + i, L.dx};
    const double mine =
        noise_dvdy_edge(nz, lane ? i : im, xc, lane ? __dadd_rn(hi, hr) : __dadd_rn(hl, hi));
    const double other = __shfl_xor_sync(pmask, mine, 1);
    return rk_velocity_of<Noise>(lane ? other : mine, lane ? mine : other, L, lt, f, model, hi, hl,
                                 hr);
}

// rk_forward_zero with every velocity evaluated by a lane pair
// (rk_site_velocity_pair): the serial march and bisection, run identically by
// both lanes, with each evaluation's two gathers side by side. Same result as
// rk_forward_zero.
template <class Noise>
__device__ __forceinline__ double rk_forward_zero_pair(const Noise &nz, int i, int n, const LineDx &dx,
                                                       double lt, double f, int model, double hi,
                                                       double hl, double hr, const RkP &rp,
                                                       bool &found, int lane, unsigned pmask) {
    const double v0 = rk_site_velocity_pair(nz, i, n, dx, lt, f, model, hi, hl, hr, lane, pmask);
    if (v0 <= 0) {
        found = true;
        return hi;
    }
    double a = hi;
    double advanced = 0;
    while (advanced < rp.max_advance) {
        const double b = a + rp.dstep;
        const double vb = rk_site_velocity_pair(nz, i, n, dx, lt, f, model, b, hl, hr, lane, pmask);
        if (vb <= 0) {
            double lo = a, hc = b;
            for (int k = 0; k < 60 && (hc - lo) > rp.root_tol; ++k) {
                const double mid = 0.5 * (lo + hc);
                const double vm =
                    rk_site_velocity_pair(nz, i, n, dx, lt, f, model, mid, hl, hr, lane, pmask);
                if (vm > 0)
                    lo = mid;
                else
                    hc = mid;
            }
            found = true;
            return 0.5 * (lo + hc);
        }
        a = b;
        advanced += rp.dstep;
    }
    found = false;
    return a;
}

// ---------------------------------------------------------- the fast search
// rk_forward_zero for the linear model on the fixed-point gather, by a group
// of G lanes: its result bit for bit, from three rounds of evaluations instead
// of the march and some 33 bisection levels. A search is one chain of
// dependent work on a nearly idle scheduler, so its cycles are latencies: what
// counts is the number of rounds, the loads, and FP64 instructions.
//   * The rows of two cells on either edge (the midpoints' cells at the start
//     and the next ones) are summed by the group's lanes side by side, once;
//     every evaluation below is arithmetic on them.
//   * March: lane j evaluates the point j serial steps ahead (lane 0 the
//     start, so the first round holds v(h_i) too); the first v <= 0 brackets
//     the zero between it and the point before.
//   * Within a cell v is a quadratic, so both ends of its slope there follow
//     from the cell's cubic. Where the bound over the bracket's cells
//     is positive (-dv/dh >= s > 0: the elastic slope 2 Gamma / dx outweighs
//     the field's curvature), v falls all along and has one zero. A secant and
//     a Newton step find it to about 1e-8, two evaluations either side bracket
//     it, and a line between them gives it up to the slope's change there and
//     the rounding of v, which grows with each edge's own slope (the edges' may
//     cancel in s) times the rounding of its height sum.
//   * Bisection then only asks on which side of the zero its midpoints lie. In
//     integers of the bracket's binade the midpoints are a grid where the width
//     halves without a remainder (else the levels are replayed); a midpoint
//     nearer to the zero than v's rounding errors over s is evaluated.
// Anything else (a steep field, a bracket out of the two cells) takes the generic
// search. 200 sweeps of
// a 2048-point line (16 taps): 39.0 -> 5.9 ms.
struct RkEdge {     // one edge's cubics in row cells iy and iy + 1
    long long p[2], u2[2], w[2];
    int d[2];  // the cells' units' orders below the field's (FxCubic)
    int iy;
    double unit;
};

// Index (0, 1) of the midpoint's cell in the window, or -1.
__device__ __forceinline__ int rk_cell(const NoiseBSpline64 &nz, const RkEdge &ed, double a,
                                       FxFrac &t) {
    int iy;
    if (!nz.fx_row(a, iy, t)) return -1;
    if (iy == ed.iy) return 0;
    return (iy == ed.iy + 1 || (iy == 0 && ed.iy + 1 == nz.ny)) ? 1 : -1;
}

struct RkFast {
    RkEdge l, r;
    double hl, hr;
    // -dv/dh = slope0 + bl q_l + br q_r, q = d(2 dV/dt)/dt in units of 2^32 of the
    // cell's unit, b by window cell
    float slope0, bl[2], br[2];
};

// b 2^-d for a cell's d (from 252 orders on it is far below any slope that counts).
__device__ __forceinline__ float rk_scale(float b, int d) {
    d = min(d, 252);
    const int half = d >> 1;
    return b * __int_as_float((127 - half) << 23) * __int_as_float((127 - d + half) << 23);
}

// An edge's b q over the window cells from k0 to k1: its smallest value, the
// largest of its magnitude and of its change along a cell.
struct RkSlope {
    float lo, mag, bend;
};
__device__ __forceinline__ RkSlope rk_slope(const RkEdge &ed, const float b[2], int k0, int k1) {
    RkSlope r{0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float q0 = (float)(int)(ed.u2[k] >> 32), q1 = (float)(int)((ed.u2[k] + 2 * ed.w[k]) >> 32);
        const float s0 = b[k] * q0, s1 = b[k] * q1;
        const bool first = k == k0, used = first || k == k1;
        const float lo = fminf(s0, s1);
        r.lo = used ? (first ? lo : fminf(r.lo, lo)) : r.lo;
        r.mag = used ? fmaxf(r.mag, fmaxf(fabsf(s0), fabsf(s1))) : r.mag;
        r.bend = used ? fmaxf(r.bend, fabsf(s1 - s0)) : r.bend;
    }
    return r;
}

// v(h) as rk_site_velocity gives it; s: -dv/dh; cl, cr: the window cells (-1:
// outside, v unset).
__device__ __forceinline__ double rk_fast_velocity(const NoiseBSpline64 &nz, const RkFast &F,
                                                   const LineDx &L, double h, float &s, int &cl,
                                                   int &cr) {
    FxFrac tl, tr;
    cl = rk_cell(nz, F.l, __dadd_rn(F.hl, h), tl);
    cr = rk_cell(nz, F.r, __dadd_rn(h, F.hr), tr);
    const bool l1 = cl == 1, r1 = cr == 1;
    const long long wl = l1 ? F.l.w[1] : F.l.w[0], wr = r1 ? F.r.w[1] : F.r.w[0];
    const long long ul = l1 ? F.l.u2[1] : F.l.u2[0], ur = r1 ? F.r.u2[1] : F.r.u2[0];
    const long long twl = fx_mul(wl, tl), twr = fx_mul(wr, tr);
    const long long Rl = (l1 ? F.l.p[1] : F.l.p[0]) + fx_mul(ul + twl, tl);
    const long long Rr = (r1 ? F.r.p[1] : F.r.p[0]) + fx_mul(ur + twr, tr);
    s = fmaf(l1 ? F.bl[1] : F.bl[0], (float)(int)((ul + 2 * twl) >> 32),
             fmaf(r1 ? F.br[1] : F.br[0], (float)(int)((ur + 2 * twr) >> 32), F.slope0));
    const double dvl = __dmul_rn(fx_to_double(Rl, -(l1 ? F.l.d[1] : F.l.d[0])), F.l.unit);
    const double dvr = __dmul_rn(fx_to_double(Rr, -(r1 ? F.r.d[1] : F.r.d[0])), F.r.unit);
    return rk_velocity_of<NoiseBSpline64>(dvl, dvr, L, 0.0, 0.0, QEW_MODEL_LINEAR, h, F.hl, F.hr);
}

// One edge's place: its column, and general x weights where it needs them.
struct RkPlace {
    int e, iy;
    bool cst;
    FxFrac fx;
};
__device__ __forceinline__ bool rk_place(const NoiseBSpline64 &nz, RkPlace &q, int e, EdgeX xc,
                                         double a) {
    FxFrac t;
    q.e = e;
    q.cst = nz.fx_const(q.e);
    if (!nz.fx_row(a, q.iy, t)) return false;
    return q.cst || nz.fx_locate(xc, nz.dx, nz.inv_dx, nz.kx, nz.nx, q.e, q.fx);
}

// The windows of both edges, by the group's lanes.
template <int G>
__device__ __forceinline__ void rk_window(const NoiseBSpline64 &nz, RkFast &F, const RkPlace &ql,
                                          const RkPlace &qr, int lane, unsigned gmask) {
    F.l.iy = ql.iy;
    F.r.iy = qr.iy;
    F.l.unit = ql.cst ? nz.fx_dv_c : nz.fx_dv_g;
    F.r.unit = qr.cst ? nz.fx_dv_c : nz.fx_dv_g;
    if (nz.poly && ql.cst && qr.cst) {
        const int l1 = ql.iy + 1 == nz.ny ? 0 : ql.iy + 1, r1 = qr.iy + 1 == nz.ny ? 0 : qr.iy + 1;
        const FxCubic a = nz.fx_const_cell(ql.e, ql.iy), b = nz.fx_const_cell(ql.e, l1);
        const FxCubic c = nz.fx_const_cell(qr.e, qr.iy), d = nz.fx_const_cell(qr.e, r1);
        F.l.p[0] = a.p, F.l.u2[0] = a.u2, F.l.w[0] = a.w, F.l.d[0] = a.d;
        F.l.p[1] = b.p, F.l.u2[1] = b.u2, F.l.w[1] = b.w, F.l.d[1] = b.d;
        F.r.p[0] = c.p, F.r.u2[0] = c.u2, F.r.w[0] = c.w, F.r.d[0] = c.d;
        F.r.p[1] = d.p, F.r.u2[1] = d.u2, F.r.w[1] = d.w, F.r.d[1] = d.d;
        return;
    }
    // row sums 0..4 of the left edge's rows iy - 1 .. iy + 3, 5..9 of the right's
    constexpr int kPass = (10 + G - 1) / G;
    long long mine[kPass];
    int kmine[kPass];
#pragma unroll
    for (int p = 0; p < kPass; ++p) {
        const int k = min(p * G + lane, 9);
        const bool right = k >= 5;
        const int e = right ? qr.e : ql.e, rr = k - (right ? 5 : 0) - 1;
        int y = (right ? qr.iy : ql.iy) + rr;
        if (y < 0) y += nz.ny;
        while (y >= nz.ny) y -= nz.ny;  // at most 3 times
        int xs[4];
        wrap4(e, nz.nx, xs);
        const double x[4] = {nz.c(xs[0], y), nz.c(xs[1], y), nz.c(xs[2], y), nz.c(xs[3], y)};
        if (right ? qr.cst : ql.cst) {
            mine[p] = fx_row_const(x, nz.kb, kmine[p]);
        } else {
            FxFrac wx[4];
            fx_weights(right ? qr.fx : ql.fx, wx);
            mine[p] = fx_row_sum(x, wx, nz.kb, kmine[p]);
        }
    }
    long long E[10];
    int kr[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
        E[k] = __shfl_sync(gmask, mine[k / G], k % G, G);
        kr[k] = __shfl_sync(gmask, kmine[k / G], k % G, G);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const FxCubic a = fx_cubic(E + k, kr + k, nz.kb), b = fx_cubic(E + 5 + k, kr + 5 + k, nz.kb);
        F.l.p[k] = a.p, F.l.u2[k] = a.u2, F.l.w[k] = a.w, F.l.d[k] = a.d;
        F.r.p[k] = b.p, F.r.u2[k] = b.u2, F.r.w[k] = b.w, F.r.d[k] = b.d;
    }
}

// False (found and the result unset): the generic search has to decide.
template <int G>
__device__ __forceinline__ bool rk_forward_zero_fast(const NoiseBSpline64 &nz, int i, int n,
                                                     const LineDx &L, int model, double hi,
                                                     double hl, double hr, const RkP &rp,
                                                     bool &found, double &result, int lane,
                                                     unsigned gmask) {
    static_assert(G >= 2, "the march advances at least a step a round");
    if (model != QEW_MODEL_LINEAR || nz.kb < 0) return false;
    const unsigned all = (G == 32) ? ~0u : ((1u << G) - 1u);
    const unsigned shift = (unsigned)(threadIdx.x & 31) & ~(unsigned)(G - 1);
    auto votes = [&](bool b) { return (__ballot_sync(gmask, b) >> shift) & all; };
    RkFast F;
    const int im = (i == 0) ? n - 1 : i - 1, ip = (i + 1 == n) ? 0 : i + 1;
    const EdgeX xl{im + i, L.dx}, xr{i + ip, L.dx};
    F.hl = hl;
    F.hr = hr;
    F.slope0 = (float)(-2.0 * L.c_el);
    // the slopes are compared as floats, far from their range's ends
    if (!(F.slope0 >= 1e-20f && F.slope0 <= 1e20f)) return false;
    double a = hi, advanced = 0.0, lo = 0.0, hc = 0.0, vlo = 0.0, vhc = 0.0;
    float s, smin, bend, mag_l, mag_r;
    int cl, cr;
    // The march takes at most ceil(max_advance / dstep) steps (validated on
    // the host), at least one a round.
    for (bool first = true;; first = false) {
        RkPlace ql, qr;
        if (!rk_place(nz, ql, im, xl, __dadd_rn(hl, a)) || !rk_place(nz, qr, i, xr, __dadd_rn(a, hr)))
            return false;
        rk_window<G>(nz, F, ql, qr, lane, gmask);
        const float bl = (float)(0.5 * L.half_dx * F.l.unit * nz.inv_dy * 0x1p32);
        const float br = (float)(0.5 * L.half_dx * F.r.unit * nz.inv_dy * 0x1p32);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            F.bl[k] = rk_scale(bl, F.l.d[k]);
            F.br[k] = rk_scale(br, F.r.d[k]);
        }
        double b = a, adv = advanced;
        bool valid = true;
        if (advanced + 1.001 * G * rp.dstep < rp.max_advance) {
            for (int t = 0; t < lane; ++t) b = __dadd_rn(b, rp.dstep);
        } else {
            for (int t = 0; t < lane; ++t) {
                if (!(adv < rp.max_advance)) {
                    valid = false;
                    break;
                }
                b = __dadd_rn(b, rp.dstep);
                adv = __dadd_rn(adv, rp.dstep);
            }
        }
        const double v = rk_fast_velocity(nz, F, L, b, s, cl, cr);
        const unsigned okm = votes(valid), in = votes(valid && cl >= 0 && cr >= 0);
        const unsigned hit = votes(valid && cl >= 0 && cr >= 0 && v <= 0);
        const int last = __ffs(~in & (all << 1 | 1u)) ? __ffs(~in) - 2 : G - 1;  // last point of the run of cells in the window
        if (last < 0) return false;
        if (first && (hit & 1u)) {
            found = true;
            result = hi;
            return true;
        }
        const int j = hit ? __ffs(hit) - 1 : 0;
        if (j && j <= last) {
            lo = __shfl_sync(gmask, b, j - 1, G);
            hc = __shfl_sync(gmask, b, j, G);
            vlo = __shfl_sync(gmask, v, j - 1, G);
            vhc = __shfl_sync(gmask, v, j, G);
            const int l0 = __shfl_sync(gmask, cl, j - 1, G), l1 = __shfl_sync(gmask, cl, j, G);
            const int r0 = __shfl_sync(gmask, cr, j - 1, G), r1 = __shfl_sync(gmask, cr, j, G);
            const RkSlope sl = rk_slope(F.l, F.bl, l0, l1), sr = rk_slope(F.r, F.br, r0, r1);
            mag_l = sl.mag;
            mag_r = sr.mag;
            bend = sl.bend + sr.bend;
            // less what the floats round and the integers' upper halves leave out
            smin = F.slope0 + sl.lo + sr.lo -
                   (1.0e-6f * (F.slope0 + mag_l + mag_r) +
                    2.0f * (fmaxf(F.bl[0], F.bl[1]) + fmaxf(F.br[0], F.br[1])));
            // a step as long as a period of the field could skip cells
            if (!(l0 <= l1 && r0 <= r1 && rp.dstep < 2.0 * nz.dy && smin > 0.25f * F.slope0 &&
                  smin < 1e25f))
                return false;
            break;
        }
        if (okm != all && last + 1 >= 32 - __clz(okm)) {  // out of max_advance: the last point stepped to
            found = false;
            result = __shfl_sync(gmask, b, 31 - __clz(okm), G);
            return true;
        }
        if (last == 0) return false;
        a = __shfl_sync(gmask, b, last, G);
        for (int t = 0; t < last; ++t) advanced = __dadd_rn(advanced, rp.dstep);
    }
    long long bl = __double_as_longlong(lo), bh = __double_as_longlong(hc);
    int ex = (int)(bl >> 52);  // positive, of ordinary size
    if (ex <= 200 || bh < bl || bh >= (1800ll << 52)) return false;
    const double ulp = __longlong_as_double((long long)(ex - 52) << 52);
    // the zero: a secant and a Newton step, then a line through two points
    // either side (lanes 0 and 1)
    const float width = (float)(hc - lo);
    double x = fma((double)((float)vlo / (float)(vlo - vhc)), hc - lo, lo);
    {
        const double v = rk_fast_velocity(nz, F, L, x, s, cl, cr);
        x = __dadd_rn(x, (double)((float)v / s));
    }
    const double gap = (double)(width * 1.0e-7f) + 64.0 * ulp;
    const double side = (lane & 1) ? x + gap : x - gap;
    const double vs = rk_fast_velocity(nz, F, L, side, s, cl, cr);
    if (votes(!(cl >= 0 && cr >= 0 && ((lane & 1) ? vs <= 0 : vs > 0)))) return false;
    const double v0 = __shfl_sync(gmask, vs, 0, G), v1 = __shfl_sync(gmask, vs, 1, G);
    const double x0 = __shfl_sync(gmask, side, 0, G);
    // what follows is in floats, far from their range's ends
    const float fall = (float)(v0 - v1);
    if (!(fall >= 1e-28f && fall <= 1e28f && width >= 1e-30f)) return false;
    const double z = fma((double)((float)v0 / fall), 2.0 * gap, x0);
    // v's rounding errors, at most, each within 2^-53 of its number (1.7e-16: and
    // a half more): the sums of heights in the elastic part; each edge's
    // midpoint (the sum, its quotient by the spacing, the fold of a negative one
    // into the period) times that edge's own slope, the field's weight of which
    // s knows only the sum; the force; and the integers' units and the
    // conversions and products of dV/dy (R below 2^60: 700 units in all).
    const float ah = (float)fabs(hc), al = (float)fabs(hl), ar = (float)fabs(hr);
    const float period = 2.0f * (float)nz.ny * (float)nz.dy;
    const float unit = (float)(2.0 * nz.dy * 0x1p-32) *
                       fmaxf(fmaxf(F.bl[0], F.bl[1]), fmaxf(F.br[0], F.br[1]));
    const float eps = 1.7e-16f * (2.0f * (float)fabs(L.c_el) * (al + ar + ah) + (float)fabs(L.fdx) +
                                  mag_l * (2.0f * (al + ah) + period) +
                                  mag_r * (2.0f * (ar + ah) + period)) +
                      700.0f * unit;
    // The line's zero is off by v's errors at its two points over s, by the
    // change of the slope between them (bend / 2 dy a unit of height: half of
    // that times gap^2 over s) and by the floats' quotient.
    const float gf = (float)gap;
    const double g = (double)((3.0f * eps + bend * (float)(0.25 * nz.inv_dy) * gf * gf) / smin) +
                     4.0 * ulp + 4.0e-7 * gap;
    // v > 0 up to z0, v <= 0 from z1 on; the bracket's own ends are known. (A
    // site within its rounding of the zero, z0 <= bl, is what a line near its
    // critical force is made of.)
    if (!(z + g > 0.0)) return false;
    const long long zl = __double_as_longlong(z - g), zh = __double_as_longlong(z + g);
    const long long z0 = min(max(zl, bl), bh - 1), z1 = max(min(zh, bh), z0);
    // levels across a binade's end, as the serial loop takes them
    int k0 = 0;
    for (; k0 < 60 && (int)(bh >> 52) != (int)(bl >> 52); ++k0) {
        lo = __longlong_as_double(bl);
        hc = __longlong_as_double(bh);
        if (!(hc - lo > rp.root_tol)) return false;  // ends here: leave it to the serial loop
        const long long M = __double_as_longlong(0.5 * (lo + hc));
        if (M <= z0)
            bl = M;
        else if (M >= z1)
            bh = M;
        else
            return false;
    }
    ex = (int)(bl >> 52);
    const int levels = 60 - k0;
    // (hc - lo) > root_tol in units of the binade's ulp; levels until it fails
    const double tu = rp.root_tol * __longlong_as_double((long long)(2098 - ex) << 52);
    const long long tol = tu < 0 ? -1 : tu < 4.6e18 ? (long long)tu : (1ll << 62);
    const long long W = bh - bl;
    int k = 0;
    while (k < levels && (W >> k) > tol && !((W >> k) & 1)) ++k;
    const long long wk = W >> k;
    if (k < levels && wk > tol) {  // an odd width: midpoints round, level by level
        long long A = bl, B = bh;
        for (k = 0; k < levels && B - A > tol; ++k) {
            const long long D = B - A, M0 = A + (D >> 1), M = M0 + (D & M0 & 1);  // ties to even
            bool pos = M <= z0;
            if (!pos && M < z1) {
                pos = rk_fast_velocity(nz, F, L, __longlong_as_double(M), s, cl, cr) > 0;
                if (cl < 0 || cr < 0) return false;
            }
            if (pos)
                A = M;
            else
                B = M;
        }
        found = true;
        result = 0.5 * (__longlong_as_double(A) + __longlong_as_double(B));
        return true;
    }
    // the grid interval about the zero
    long long q0, q1;
    if ((wk & (wk - 1)) == 0) {
        const int sft = 63 - __clzll(wk);
        q0 = (z0 - bl) >> sft;
        q1 = (z1 - bl) >> sft;
    } else {
        q0 = (z0 - bl) / wk;
        q1 = (z1 - bl) / wk;
    }
    if (q1 > q0 + 1) return false;
    if (q1 > q0) {  // a midpoint at the zero
        const double v = rk_fast_velocity(nz, F, L, __longlong_as_double(bl + q1 * wk), s, cl, cr);
        if (cl < 0 || cr < 0) return false;
        if (v > 0) q0 = q1;
    }
    found = true;
    result = 0.5 * (__longlong_as_double(bl + q0 * wk) + __longlong_as_double(bl + (q0 + 1) * wk));
    return true;
}
