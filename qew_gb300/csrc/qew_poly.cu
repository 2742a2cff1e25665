// qew_poly.cu -- FP64 gradient on the cell-polynomial store (QEW_STORE_FP64_POLY).
//
// gradient() (qew_model.h:149-193) of lines with one point per field column,
// heights and gradients in FP64: the edge pass reads one 32-byte cell of the
// store per edge (the x-filtered field's cubic in the row fraction, built
// once with the field) and evaluates dV/dy in 64-bit fixed point; the
// per-site combine is the reference's, with its factors folded:
//   grad_i = dx (F_el,i + (dv_{i-1} + dv_i)/2 - f)
//          = c_el d2h_i + (dx/2)(dv_{i-1} + dv_i) - dx f        (linear,
//            c_el = -Gamma/dx)
//          = Gamma (s_{i-1} - s_i) + (dx/2)(dv_{i-1} + dv_i) - dx f  (arclength).
//
// Three kernels:
//   k_gradient_poly_walk  the linear model: every step up to the last two
//     multiply-adds in integers (below);
//   k_gradient_poly_walk_host  the same for lines in host memory;
//   k_gradient_poly       arclength: FP64 heights and combine, the cell and
//     the slope's root in fixed point.
#include <algorithm>
#include <climits>
#include <cmath>

#include <math_constants.h>

#include "qew_internal.cuh"
#include "qew_model_kernels.cuh"
#include "qew_poly.cuh"
#include "qew_tune.cuh"

namespace {

constexpr int kBS = 256;
constexpr int kMinCtas = 4;  // 64 registers a thread: up to 4 resident CTAs per SM

struct PolyGeom {
    NoiseBSpline64 nz;    // the store, and the 16-tap path of the wrap edge
    int n;
    int ky;               // (h_e + h_ep) [* recip] * 2^ky = midpoint in row cells
    FxFrac recip;         // mantissa of 1 / (2 dy) in [1/2, 1) (not a power of two)
    LineDx L;
    double lt;            // Gamma
    double half_unit;     // dx / 2 * the unit of an edge's integer dV/dy
    float inv_ny;
};

// dV/dy of an edge that the store does not cover (the wrap edge): out of line,
// so that its general path takes no registers of the kernels' loops.
__device__ __noinline__ double walk_edge_rare(const PolyGeom &g, int e, double sum) {
    const int ep = (e + 1 == g.n) ? 0 : e + 1;
    return g.nz.dvdy_edge_sum(e, EdgeX{e + ep, g.L.dx}, sum);
}

// 8-byte asynchronous global -> shared copy.
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Persistent, batched (lines stored n apart), one CTA per resident slot; each
// CTA walks tiles of kTile sites gridDim.x apart and copies the next tile's
// heights into its spare shared buffer with cp.async while the current
// tile's gathers are in flight. Bound about equally by 10 FP64 instructions a
// point and by issue: 8 lines of 2^20 points 269 -> 181 us.
template <int kItems>
__global__ void __launch_bounds__(kBS, kMinCtas)
k_gradient_poly(const double *__restrict__ h, const __grid_constant__ PolyGeom g,
                double *__restrict__ grad, int count) {
    constexpr int kTile = kBS * kItems;
    __shared__ double s_h[2][kTile + 2];
    __shared__ double s_dv[kTile + 1];
    __shared__ double s_sl[kTile + 1];
    const int n = g.n;
    const int per_line = (n + kTile - 1) / kTile;
    const int t = threadIdx.x;
    // This CTA's tiles are blockIdx.x + k * gridDim.x in line-major order;
    // (line, index in line) advance by a fixed step, one division per CTA.
    const int step_l = (int)gridDim.x / per_line;
    const int step_i = (int)gridDim.x - step_l * per_line;
    auto fetch = [&](int line, int idx, int buf) {  // a tile's heights (+ halo) into buffer buf
        const int base = idx * kTile;
        const int cnt = min(kTile, n - base);
        const double *hl = h + (size_t)line * (size_t)n;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int j = t + k * kBS;
            if (j < cnt) cp_async8(&s_h[buf][j + 1], hl + base + j);
        }
        if (t == 0) {
            cp_async8(&s_h[buf][0], hl + (base == 0 ? n - 1 : base - 1));
        } else if (t == kBS - 1) {
            cp_async8(&s_h[buf][cnt + 1], hl + ((base + cnt == n) ? 0 : base + cnt));
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    int line = (int)blockIdx.x / per_line;
    int idx = (int)blockIdx.x - line * per_line;
    if (line < count) fetch(line, idx, 0);
    for (int buf = 0; line < count; buf ^= 1) {
        int nline = line + step_l, nidx = idx + step_i;
        if (nidx >= per_line) {
            nidx -= per_line;
            ++nline;
        }
        const int base = idx * kTile;
        const int cnt = min(kTile, n - base);
        const double *sh = s_h[buf];
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        // Barrier A: this tile's heights are in place, and every thread has
        // left the previous tile, whose buffer may now be refilled and whose
        // edge values may be rewritten.
        __syncthreads();
        if (nline < count) fetch(nline, nidx, buf ^ 1);
        auto edge = [&](int e, int slot) {
            slot = QEW_IDX(slot, kTile + 1, g.nz.oob);
            const double he = sh[slot], hep = sh[slot + 1];
            s_dv[slot] = e + 1 < n ? g.nz.dvdy_edge_store(e, hep + he) : walk_edge_rare(g, e, hep + he);
            s_sl[slot] = fx_slope(g.L.slope(hep - he));
        };
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int j = t + k * kBS;
            if (j < cnt) edge(base + j, j + 1);
        }
        if (t == kBS - 1) edge(base == 0 ? n - 1 : base - 1, 0);
        __syncthreads();  // barrier B: edge values in place
        double *out = grad + (size_t)line * (size_t)n + base;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int j = QEW_IDX(t + k * kBS, kTile, g.nz.oob);
            if (t + k * kBS >= cnt) break;
            __stcs(out + j, site_gradient<NoiseBSpline64>(
                                sh[j], sh[j + 1], sh[j + 2], s_dv[j], s_dv[j + 1], s_sl[j],
                                s_sl[j + 1], g.L, g.lt, 0.0, true));
        }
        line = nline;
        idx = nidx;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// ------------------------------------------------------------ integer walk
// The linear gradient with the heights themselves as integers. A warp takes
// chunks of 255 consecutive sites, the 256 edges about them in 8 steps of 32;
// the chunk's 257 heights become signed integers in the unit 2^-8 of the ulp
// of the largest one: exactly down to 2^-8 of it, smaller ones cut at that
// unit, which FP64's sum with a neighbour rounds coarser as long as one of the
// two is above 2^-7 of the largest. The midpoint sum, its row cell (folded into the field's period) and
// fraction, dV/dy and the second difference of the heights are then integer
// sums and products, and a site takes two FP64 instructions (the combine)
// for seven before:
//   grad = c_el d2h + (half_unit (R_l + R_r) - dx f).
// A chunk with two neighbours below that, a non-finite height, or heights too
// small or too large beside the row spacing (a flat line at 0) takes FP64 sums
// (walk_chunk_fp64). Chunks start at
// multiples of 255 of their line, whatever the launch, so every launch shape
// and batch gives the same bits.
constexpr int kWalkSteps = 8;
constexpr int kWalkEdges = 32 * kWalkSteps;
constexpr int kWalkSites = kWalkEdges - 1;
constexpr int kWalkGuard = 8;

// R = dV/dy of edge e < n - 1 in the unit of its cell, d orders below the
// store's, from the integer sum a of its heights, whose midpoint in row cells is a 2^-sh, |a 2^-sh| < 2^22.
// kPow2: a power-of-two row spacing; else a is first multiplied by the
// spacing's reciprocal mantissa (62 bits).
template <bool kPow2>
__device__ __forceinline__ long long walk_edge(const PolyGeom &g, int e, long long a, int sh,
                                               int &d) {
    if (!kPow2) a = fx_mul(a, g.recip);
    int c = (int)(a >> sh);  // floor
    const FxFrac t = fx_frac((unsigned long long)a << (64 - sh));
    if ((unsigned)c >= (unsigned)g.nz.ny) {  // fold into the period: the quotient is off by 1 at most
        c -= __float2int_rd((float)c * g.inv_ny) * g.nz.ny;
        if (c < 0) c += g.nz.ny;
        if (c >= g.nz.ny) c -= g.nz.ny;
    }
    c = QEW_IDX(c, g.nz.ny, g.nz.oob);
    e = QEW_IDX(e, g.nz.nx, g.nz.oob);
    const FxCubic q = fx_load_cell(g.nz.poly + ((size_t)c * (size_t)g.nz.nx + (size_t)e) * 4);
    d = q.d;
    return fx_dt2(q, t);
}

// v of the next lane; the last lane gets `wrap` of the first one.
template <class T>
__device__ __forceinline__ T lane_next(T v, T wrap, int lane) {
    return __shfl_sync(0xffffffffu, lane == 0 ? wrap : v, (lane + 1) & 31);
}

// Both edges' dV/dy, each in its cell's unit, as an integer in the unit of the
// larger, ds orders below the field's.
__device__ __forceinline__ long long walk_pair(long long Rl, int dl, long long Rr, int dr, int &ds) {
    ds = min(dl, dr);
    return fx_sar(Rl, dl - ds) + fx_sar(Rr, dr - ds);
}

// The chunk's gradients from FP64 sums of heights, a lane an edge as in
// walk_chunk: 5 FP64 instructions a site. Out of line, as walk_edge_rare.
__device__ __noinline__ void walk_chunk_fp64(const PolyGeom &g, const double *hl, double *out, int s0,
                                             int lane, const double *hs) {
    const int n = g.n;
    auto height = [&](int j) {  // of site s0 - 1 + j
        const int i = s0 - 1 + j;
        return hs ? hs[j] : __ldg(hl + (i < 0 ? n - 1 : i < n ? i : 0));
    };
    double h = height(lane), hb = 0.0, hpb = 0.0;  // b: of the step before
    long long Rb = 0;
    int db = 0;  // -1: a NaN
    for (int k = 0; k <= kWalkSteps; ++k) {
        double hp = 0.0, hn = 0.0;
        long long R = 0;
        int d = 0;
        if (k < kWalkSteps) {
            hn = k + 1 < kWalkSteps ? height(32 * (k + 1) + lane) : height(kWalkEdges);
            hp = lane_next(h, hn, lane);
            const int e = s0 - 1 + 32 * k + lane;
            if (e >= 0 && e + 1 < n && !g.nz.dvdy_edge_store(e, hp + h, R, d)) d = -1;
        }
        if (k > 0) {  // the sites of the step before
            const int i = s0 + 32 * (k - 1) + lane;
            const double hr = lane_next(hpb, hp, lane);
            const int dr = lane_next(db, d, lane);
            int ds;
            const long long S = walk_pair(Rb, db, lane_next(Rb, R, lane), dr, ds);
            const double dv = ds < 0 ? CUDART_NAN : fx_to_double(S, -ds);
            if (i > 0 && i + 1 < n && (k < kWalkSteps || lane < 31))
                out[i - s0] = fma(g.L.c_el, fma(-2.0, hpb, hb + hr), fma(g.half_unit, dv, -g.L.fdx));
        }
        hb = h;
        hpb = hp;
        Rb = R;
        db = d;
        h = hn;
    }
}

// Gradient of site i (a wrap site) from FP64 sums and edges.
__device__ __noinline__ double walk_site_rare(const PolyGeom &g, const double *hl, int i) {
    const int n = g.n;
    const int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
    const double hm = __ldg(hl + im), h0 = __ldg(hl + i), hp = __ldg(hl + ip);
    const double dvl = walk_edge_rare(g, im, hm + h0), dvr = walk_edge_rare(g, i, h0 + hp);
    return site_gradient<NoiseBSpline64>(hm, h0, hp, dvl, dvr, 0.0, 0.0, g.L, g.lt, 0.0, false);
}

// The chunk's gradients to out[0 ..] (out: of site s0). hs: its heights from
// site s0 - 1 on in shared memory, or null.
template <bool kPow2, bool kStage>
__device__ __forceinline__ void walk_chunk(const double *__restrict__ hl, const PolyGeom &g,
                                           double *__restrict__ out, int s0, int lane,
                                           const double *hs = nullptr) {
    const int n = g.n;
    // step k's edges are s0 - 1 + 32 k + lane, each with the site at its
    // right end; the two sites of the wrap edge are done apart
    if (s0 == 0 && lane == 0) out[0] = walk_site_rare(g, hl, 0);
    if (s0 + kWalkSites >= n && lane == 1) out[n - 1 - s0] = walk_site_rare(g, hl, n - 1);
    double x[kWalkSteps];
#pragma unroll
    for (int k = 0; k < kWalkSteps; ++k) {
        const int i = s0 - 1 + 32 * k + lane;
        x[k] = kStage && hs ? hs[32 * k + lane] : __ldg(hl + (i < 0 ? n - 1 : i < n ? i : 0));
    }
    const int il = s0 - 1 + kWalkEdges;  // right end of the last edge
    const double last = kStage && hs ? hs[kWalkEdges] : __ldg(hl + (il < n ? il : 0));
    // the largest and the smallest exponent of the chunk
    unsigned mx = (unsigned)__double2hiint(last) << 1, mn = mx;
#pragma unroll
    for (int k = 0; k < kWalkSteps; ++k) {
        const unsigned b = (unsigned)__double2hiint(x[k]) << 1;
        mx = max(mx, b);
        mn = min(mn, b);
    }
    mx = __reduce_max_sync(0xffffffffu, mx) >> 21;
    mn = __reduce_min_sync(0xffffffffu, mn) >> 21;
    // midpoint in cells = a 2^-sh for a in units of 2^(mx - 1075 - guard)
    const int sh = 1075 + kWalkGuard - (int)mx - g.ky;
    bool whole = mx < 2047u && mx > 200u && sh >= 40 && sh <= 63;
    if (whole && mn + 7 < mx) {  // two neighbours that small: the integers would cut their sum
        auto large = [&](double v) {
            return __ballot_sync(0xffffffffu, (((unsigned)__double2hiint(v) << 1) >> 21) + 7 >= mx);
        };
        unsigned b = large(x[0]);
#pragma unroll
        for (int k = 0; k < kWalkSteps; ++k) {
            const unsigned nb = large(k + 1 < kWalkSteps ? x[k + 1 < kWalkSteps ? k + 1 : 0] : last);
            whole = whole && (b | __funnelshift_r(b, nb, 1)) == 0xffffffffu;
            b = nb;
        }
    }
    if (!whole) {
        walk_chunk_fp64(g, hl, out, s0, lane, kStage ? hs : nullptr);
        return;
    }
    auto fix = [&](double v) {
        const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
        const unsigned m = (hi & 0x000FFFFFu) | 0x00100000u;
        const unsigned long long w =
            ((unsigned long long)__funnelshift_l(lo, m, kWalkGuard) << 32) |
            (unsigned long long)(lo << kWalkGuard);
        const long long sg = (long long)((int)hi >> 31);
        return ((long long)fx_shr(w, (int)(mx - ((hi >> 20) & 0x7FFu))) ^ sg) - sg;
    };
    const int ek = (int)mx - 1075 - kWalkGuard;
    long long H = fix(x[0]), Rb = 0, sb = 0;  // Rb (db), sb: edge and slope of the step before
    int db = 0;
#pragma unroll
    for (int k = 0; k <= kWalkSteps; ++k) {
        long long R = 0, sl = 0;
        int d = 0;
        if (k < kWalkSteps) {
            const long long Hn = fix(k + 1 < kWalkSteps ? x[k + 1 < kWalkSteps ? k + 1 : 0] : last);
            const long long Hp = lane_next(H, Hn, lane);
            const int e = s0 - 1 + 32 * k + lane;
            R = walk_edge<kPow2>(g, e >= 0 && e + 1 < n ? e : 0, H + Hp, sh, d);
            sl = Hp - H;
            H = Hn;
        }
        if (k > 0) {  // the sites of the step before
            const int i = s0 + 32 * (k - 1) + lane;
            int ds;
            const long long S = walk_pair(Rb, db, lane_next(Rb, R, lane), lane_next(db, d, lane), ds);
            const long long D = lane_next(sb, sl, lane) - sb;
            if (i > 0 && i + 1 < n && (k < kWalkSteps || lane < 31)) {
                const double v = fma(g.L.c_el, fx_to_double(D, ek),
                                     fma(g.half_unit, fx_to_double(S, -ds), -g.L.fdx));
                if (kStage) out[i - s0] = v;
                else __stcs(out + (i - s0), v);
            }
        }
        Rb = R;
        db = d;
        sb = sl;
    }
}

template <int kMin, bool kPow2>
__global__ void __launch_bounds__(kBS, kMin)
k_gradient_poly_walk(const double *__restrict__ h, const __grid_constant__ PolyGeom g,
                     double *__restrict__ grad, int chunks, long long units) {
    const long long u = (long long)blockIdx.x * (kBS / 32) + (threadIdx.x >> 5);
    if (u >= units) return;
    const int line = (int)(u / chunks);
    const int s0 = (int)(u - (long long)line * chunks) * kWalkSites;
    const size_t off = (size_t)line * (size_t)g.n;
    walk_chunk<kPow2, false>(h + off, g, grad + off + s0, s0, threadIdx.x & 31);
}

// The same for lines in host memory (the same chunks, so the same bits): a
// persistent block takes runs of 8 chunks, whose heights come into shared
// memory in aligned 128-byte pieces while the run before is computed, and
// whose gradients leave the same way. 255-site runs of a warp touch a third
// line for every two, and the host link pays for each: 8 lines of 2^20 in
// pinned memory 14.5 G points/s with them, 19.3 so. Fewer blocks than SMs: the
// link gives less when more is in flight (two blocks an SM 17.8, one 18.0, four
// for five SMs 19.0, seven for ten 19.3, one for two 14.7; the kernel of
// 256-site tiles on FP64 sums that was here before the walk 19.65). So there are
// registers to spare, and a warp's eight gathers are in flight together.
template <bool kPow2>
__global__ void __launch_bounds__(kBS, 2)
k_gradient_poly_walk_host(const double *__restrict__ h, const __grid_constant__ PolyGeom g,
                          double *__restrict__ grad, int chunks, long long units) {
    constexpr int kWarps = kBS / 32, kRun = kWarps * kWalkSites;
    __shared__ double s_h[2][kRun + 2], s_out[kRun];
    const int n = g.n, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long runs = (units + kWarps - 1) / kWarps;
    // line and first site of a run; whole: all its chunks lie inside the line
    auto place = [&](long long r, size_t &off, int &first) {
        const long long u = r * kWarps;
        const int line = (int)(u / chunks);
        first = (int)(u - (long long)line * chunks) * kWalkSites;
        off = (size_t)line * (size_t)n;
        return r < runs && first > 0 && first < n - kRun;
    };
    auto fetch = [&](long long r, int buf) {
        size_t off;
        int first;
        if (place(r, off, first)) {
            const double *p = h + off + first - 1;
            for (int j = (int)threadIdx.x - ((int)((uintptr_t)p >> 3) & 15); j < kRun + 2; j += kBS)
                if (j >= 0) cp_async8(&s_h[buf][j], p + j);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    fetch(blockIdx.x, 0);
    int buf = 0;
    for (long long r = blockIdx.x; r < runs; r += gridDim.x, buf ^= 1) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // heights in place; the run before has left s_out and the other buffer
        fetch(r + gridDim.x, buf ^ 1);
        size_t off;
        int first;
        const bool whole = place(r, off, first);
        const long long u = r * kWarps + w;
        const int line = (int)(u / chunks);
        const int s0 = (int)(u - (long long)line * chunks) * kWalkSites;
        const size_t mine = (size_t)line * (size_t)n;
        if (u < units)
            walk_chunk<kPow2, true>(h + mine, g, s_out + w * kWalkSites, s0, lane,
                                    whole ? s_h[buf] + w * kWalkSites : nullptr);
        __syncthreads();
        if (whole) {
            double *o = grad + off + first;
            for (int j = (int)threadIdx.x - ((int)((uintptr_t)o >> 3) & 15); j < kRun; j += kBS)
                if (j >= 0) __stcs(o + j, s_out[j]);
        } else if (u < units) {
            for (int j = lane; j < min(kWalkSites, n - s0); j += 32)
                __stcs(grad + mine + s0 + j, s_out[w * kWalkSites + j]);
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// FxCubic of every (row cell j, column e) from the FP64 coefficients c
// ([ny][nx]). Each thread walks kStoreRows row cells of one column and
// filters each coefficient row along x once: cell j takes the filtered values
// of rows j-1..j+2 from a window of four. Integer arithmetic, about 120
// cycles of a warp a cell; bound by its writes (32 bytes a cell).
constexpr int kStoreRows = 32;
constexpr int kStoreBS = 256;

__global__ void __launch_bounds__(kStoreBS) k_poly_store(const double *__restrict__ c, int nx,
                                                         int ny,
                                                         const unsigned long long *max_bits,
                                                         long long *__restrict__ out) {
    const int e = blockIdx.x * kStoreBS + threadIdx.x;
    if (e >= nx) return;
    const unsigned long long mb = *max_bits;
    const int kb = qew_fix_bound(mb);
    if (kb < 0) return;  // no fixed point for this field: the store is dropped
    const int j0 = blockIdx.y * kStoreRows;
    const int j1 = min(ny, j0 + kStoreRows);
    int xs[4];
    wrap4(e, nx, xs);
    int r = (j0 == 0) ? ny - 1 : j0 - 1;  // row j0-1, periodic
    long long E[4];
    int kr[4];
    auto next_row = [&](int b) {
        const double *row = c + (size_t)r * nx;
        r = (r + 1 == ny) ? 0 : r + 1;
        const double x[4] = {__ldg(row + xs[0]), __ldg(row + xs[1]), __ldg(row + xs[2]),
                             __ldg(row + xs[3])};
        E[b] = fx_row_const(x, kb, kr[b]);
    };
    next_row(0);
    next_row(1);
    next_row(2);
    for (int j = j0; j < j1; ++j) {
        next_row(3);
        fx_store_cell(out + ((size_t)j * (size_t)nx + (size_t)e) * 4, fx_cubic(E, kr, kb));
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            E[b] = E[b + 1];
            kr[b] = kr[b + 1];
        }
    }
}

}  // namespace

qew_status qew_poly_store_build(qew_ctx *ctx, const double *c, int nx, int ny,
                                const unsigned long long *max_bits, long long *out) {
    if ((ny + kStoreRows - 1) / kStoreRows > 65535)
        return qew_fail(ctx, QEW_ERR_INVALID, "poly store: more than 2^21 field rows");
    const dim3 grid((unsigned)((nx + kStoreBS - 1) / kStoreBS),
                    (unsigned)((ny + kStoreRows - 1) / kStoreRows));
    k_poly_store<<<grid, kStoreBS, 0, ctx->stream>>>(c, nx, ny, max_bits, out);
    return qew_launch_check(ctx, "poly_store");
}

qew_status qew_gradient_poly_enqueue(qew_ctx *ctx, const qew_field *f, int count,
                                     const double *d_h, int n, const qew_params *p,
                                     double *d_grad, bool host_grad) {
    if (!f || f->kind != QEW_FIELD_BSPLINE || !f->coef64 || !f->poly) return QEW_ERR_UNSUPPORTED;
    PolyGeom g{};
    g.nz = make_bspline64(f, n, p->physical_size);
    if (!g.nz.poly || g.nz.kb < 0) return QEW_ERR_UNSUPPORTED;
    g.n = n;
    const bool pow2 = qew_is_pow2(f->dy);
    {
        // 1 / (2 dy) = m 2^ky; the double's error as a second term
        const double d = 2.0 * f->dy, q = 1.0 / d;
        int e;
        const double m = frexp(q, &e);
        const long long M = llrint(ldexp(m, 62)) + llrint(ldexp(q * fma(-q, d, 1.0), 62 - e));
        g.ky = pow2 ? e - 1 : e;
        g.recip = fx_limbs(std::min(M, (1ll << 62) - 1));
    }
    g.L = make_line_dx(p->physical_size, n, p->line_tension, p->driving_force);
    g.lt = p->line_tension;
    g.half_unit = g.L.half_dx * g.nz.fx_dv_c;
    g.inv_ny = 1.0f / (float)f->ny;
    const bool arc = (p->model == QEW_MODEL_ARCLENGTH);
    const bool walk = !arc;  // k_gradient_poly is for arclength
    // (dx / 2 times the unit leaves FP64's range: FP64 sums and combine)
    if (walk && !(g.half_unit > 0x1p-700 && g.half_unit < 0x1p+900)) return QEW_ERR_UNSUPPORTED;
    // Candidates; every one computes the same numbers (the per-site
    // arithmetic does not depend on the launch): sites per thread {1, 2, 4} x
    // resident CTAs per SM {2, 3, 4}, default 2 sites, 4 CTAs; for the walk
    // (a chunk per warp) registers for {4, 5, 6} resident CTAs per SM, default
    // 5: 92.6, 86.6 and 88.2 us on 8 lines of 2^20 points of a 1024-row field.
    static const char *const tile_names[9] = {"1 site x 2 CTA/SM", "1 site x 3 CTA/SM",
                                              "1 site x 4 CTA/SM", "2 sites x 2 CTA/SM",
                                              "2 sites x 3 CTA/SM", "2 sites x 4 CTA/SM",
                                              "4 sites x 2 CTA/SM", "4 sites x 3 CTA/SM",
                                              "4 sites x 4 CTA/SM"};
    static const char *const walk_names[3] = {"walk, 4 CTA/SM", "walk, 5 CTA/SM", "walk, 6 CTA/SM"};
    auto launch = [&](int c) -> qew_status {
        const int items = 1 << (c / 3);
        const int ctas = 2 + c % 3;
        if (walk) {
            const int chunks = (n + kWalkSites - 1) / kWalkSites;
            const long long units = (long long)chunks * count;
            const long long blocks = (units + kBS / 32 - 1) / (kBS / 32);
            if (blocks > INT_MAX)
                return qew_fail(ctx, QEW_ERR_INVALID, "gradient: more than 2^31 tiles");
            if (host_grad) {
                const int grid = (int)std::min<long long>(blocks, std::max(1, ctx->num_sms * 7 / 10));
                if (pow2)
                    k_gradient_poly_walk_host<true><<<grid, kBS, 0, ctx->stream>>>(d_h, g, d_grad, chunks, units);
                else
                    k_gradient_poly_walk_host<false><<<grid, kBS, 0, ctx->stream>>>(d_h, g, d_grad, chunks, units);
                return qew_launch_check(ctx, "gradient_poly");
            }
#define QEW_WALK_LAUNCH(M) \
    (pow2 ? k_gradient_poly_walk<M, true><<<(unsigned)blocks, kBS, 0, ctx->stream>>>(              \
                d_h, g, d_grad, chunks, units)                                                     \
          : k_gradient_poly_walk<M, false><<<(unsigned)blocks, kBS, 0, ctx->stream>>>(             \
                d_h, g, d_grad, chunks, units))
            if (c == 0) QEW_WALK_LAUNCH(4);
            else if (c == 1) QEW_WALK_LAUNCH(5);
            else QEW_WALK_LAUNCH(6);
#undef QEW_WALK_LAUNCH
            return qew_launch_check(ctx, "gradient_poly");
        }
        const long long tiles = (long long)((n + kBS * items - 1) / (kBS * items)) * count;
        if (tiles > INT_MAX)
            return qew_fail(ctx, QEW_ERR_INVALID, "gradient: more than 2^31 tiles");
        const int grid = (int)std::min<long long>(tiles, (long long)ctas * ctx->num_sms);
#define QEW_POLY_LAUNCH(I) \
    k_gradient_poly<I><<<grid, kBS, 0, ctx->stream>>>(d_h, g, d_grad, count)
        if (items == 1) QEW_POLY_LAUNCH(1);
        else if (items == 2) QEW_POLY_LAUNCH(2);
        else QEW_POLY_LAUNCH(4);
#undef QEW_POLY_LAUNCH
        return qew_launch_check(ctx, "gradient_poly");
    };
    int cand = walk ? 1 : 5;
    if (walk && host_grad) return launch(cand);  // bound by the host link
    QEW_TRY(qew_tune_pick(ctx, kTuneGradientPoly,
                          qew_tune_class((long long)n * count, (arc ? 1 : 0) + (walk ? 2 : 0) + (pow2 ? 4 : 0)),
                          walk ? 3 : 9, cand, walk ? walk_names : tile_names, launch, &cand));
    return launch(cand);
}
