// qew_internal.cuh -- shared internals of the GB300 qEW library: context and
// field handles, error plumbing, and the device-side Noise functors.
//
// Noise functors mirror the reference's `Noise` concept (qew_model.h:14-17,
// 31-48): a copyable, device-callable object with value / dV/dy / full
// sample. NoiseBSpline64 restates DeviceNoise (filtered_noise.h:67-177) on an
// x-fastest coefficient array, keeping the reference's exact coordinate
// arithmetic (x/dx, periodic fold, floor) so the cell index and fraction are
// bit-identical to the reference's; only the weight polynomials use
// multiplications by 1/6 where the reference divides (a <= 1 ulp change).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>

#include "../../include/qew_gpu.h"
#include "qew_fix.cuh"
#include "qew_nvtx.cuh"

// ---------------------------------------------------------------- handles
struct qew_ctx {
    int device = 0;
    int num_sms = 0;
    cudaStream_t stream = nullptr;
    // reduction scratch: per-block partials + a self-resetting ticket counter
    double *red_partials = nullptr;  // QEW_RED_MAX_BLOCKS * 4 doubles
    unsigned int *red_counter = nullptr;
    double *host_out = nullptr;      // 8 doubles of results: pinned, written by the kernels
    // general scratch arena (grown on demand, never shrunk)
    void *scratch = nullptr;
    size_t scratch_bytes = 0;
    uint64_t launches = 0;
    // upper bound on the warps of this context's persistent (cooperative)
    // kernels; 0 = every resident slot of the GPU. Contexts that share the GPU
    // (the server's workers) take a share each.
    int warp_cap = 0;
    // grid-barrier limits of this context's cooperative kernels: polls before
    // a wait gives up, and a CTA that skips its arrival (-1: none; a fault
    // that tests inject to make the waits run out)
    long long barrier_polls = 1LL << 26;
    int barrier_skip = -1;
    // launch-shape autotuning (qew_tune.cuh): on by default; tune_force[k]
    // >= 0 fixes kernel k's candidate (kernel ids of qew_tune.cuh)
    int autotune = 1;
    int tune_force[4] = {-1, -1, -1, -1};
    std::string last_error;
    // copy streams and slot events of the host-buffer batch pipeline
    // (created on first use)
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    cudaEvent_t ev_in[3] = {}, ev_comp[3] = {}, ev_out[3] = {}, ev_start = nullptr;
};

struct qew_field {
    int kind = QEW_FIELD_BSPLINE;
    int device = 0;
    int nx = 0, ny = 0;
    double Lx = 0, Ly = 0, dx = 1, dy = 1;
    double p0 = 0, p1 = 0, p2 = 0;
    double *coef64 = nullptr;  // [ny][nx], x fastest
    float *coef32 = nullptr;   // [ny][nx], x fastest
    float *edge32 = nullptr;   // [ny][nx]: coefficients filtered along x at e + 1/2
    long long *poly = nullptr;  // [ny][nx][4]: cell polynomials of the x-filtered field (FxCubic)
    int fixb = -1;  // biased exponent of the largest |coefficient| (qew_fix.cuh), -1: none usable
    cudaStream_t stream = nullptr;  // stream the coefficients were allocated on
};

#define QEW_RED_MAX_BLOCKS 1024

// Records the message on ctx (if any) and returns the status.
qew_status qew_fail(qew_ctx *ctx, qew_status s, const char *fmt, ...);
// Stream-ordered device allocation on ctx's stream (no device-wide sync).
qew_status qew_alloc_async(qew_ctx *ctx, void **p, size_t bytes);
void qew_free_async(void *p, cudaStream_t stream);
// Ensures ctx->scratch holds at least `bytes` (256-byte aligned base).
qew_status qew_scratch_reserve(qew_ctx *ctx, size_t bytes);
// Checks the last launch; bumps the launch counter by `k`.
qew_status qew_launch_check(qew_ctx *ctx, const char *what, int k = 1);

#define QEW_CUDA(ctx, call)                                                  \
    do {                                                                     \
        cudaError_t e__ = (call);                                            \
        if (e__ != cudaSuccess)                                              \
            return qew_fail((ctx), QEW_ERR_CUDA, "%s: %s", #call,            \
                            cudaGetErrorString(e__));                        \
    } while (0)

#define QEW_TRY(expr)                                                        \
    do {                                                                     \
        qew_status s__ = (expr);                                             \
        if (s__ != QEW_OK) return s__;                                       \
    } while (0)

// ------------------------------------------------------ bounds-check build
// Built with -DQEW_BOUNDS_CHECK (qew_gb300/build.py bounds_check=True), every
// field gather and the gradient kernels' shared-memory indices are checked:
// an index outside its array is counted in mapped host words (count, first
// index, its bound, source line; qew_bounds_check_report reads them) and
// clamped into range, so the access stays in bounds. The normal build
// compiles the bare accesses: these macros discard their check arguments.
// QEW_LDGP takes the pointer itself (the normal build's address arithmetic
// is then the unchecked code's, register for register) and the array's base.
#ifdef QEW_BOUNDS_CHECK
// Device address of the four mapped host words (allocated on first use).
unsigned long long *qew_bounds_words();
__device__ __forceinline__ long long qew_bc(long long i, long long n, unsigned long long *w,
                                            int line) {
    if (i >= 0 && i < n) return i;
    if (w && atomicAdd(w, 1ull) == 0ull) {
        w[1] = (unsigned long long)i;
        w[2] = (unsigned long long)n;
        w[3] = (unsigned long long)line;
    }
    return i < 0 ? 0 : (n > 0 ? n - 1 : 0);
}
template <class T>
__device__ __forceinline__ T qew_ldg_checked(const T *base, size_t off, size_t size,
                                             unsigned long long *w, int line) {
    return __ldg(base + (size_t)qew_bc((long long)off, (long long)size, w, line));
}
#define QEW_OOB_MEMBER unsigned long long *oob = nullptr;
#define QEW_IDX(i, n, w) ((int)qew_bc((i), (n), (w), __LINE__))
#define QEW_LDGP(ptr, base, size, w) \
    qew_ldg_checked((base), (size_t)((ptr) - (base)), (size), (w), __LINE__)
#define QEW_OOB_PARAMS , size_t oob_n, unsigned long long *oob
#define QEW_OOB_WORDS , unsigned long long *oob
#define QEW_OOB_ARGS(n, w) , (n), (w)
#else
#define QEW_OOB_MEMBER
#define QEW_IDX(i, n, w) (i)
#define QEW_LDGP(ptr, base, size, w) __ldg(ptr)
#define QEW_OOB_PARAMS
#define QEW_OOB_WORDS
#define QEW_OOB_ARGS(n, w)
#endif

// ------------------------------------------------------------ B-spline math
// Cubic B-spline weights for neighbours {i-1,i,i+1,i+2} at fraction t
// (filtered_noise.h:33-46), and their t-derivatives (filtered_noise.h:50-62).
__device__ __forceinline__ void bsw_value(double t, double w[4]) {
    const double s6 = 1.0 / 6.0;
    const double t2 = t * t, t3 = t2 * t, omt = 1.0 - t;
    w[0] = omt * omt * omt * s6;
    w[1] = (4.0 - 6.0 * t2 + 3.0 * t3) * s6;
    w[2] = (1.0 + 3.0 * t + 3.0 * t2 - 3.0 * t3) * s6;
    w[3] = t3 * s6;
}
__device__ __forceinline__ void bsw_deriv(double t, double dw[4]) {
    const double s6 = 1.0 / 6.0;
    const double t2 = t * t, omt = 1.0 - t;
    dw[0] = -omt * omt * 0.5;
    dw[1] = (-12.0 * t + 9.0 * t2) * s6;
    dw[2] = (3.0 + 6.0 * t - 9.0 * t2) * s6;
    dw[3] = 3.0 * t2 * s6;
}

// Physical -> grid coordinate along one axis with the periodic fold of
// DeviceNoise::locate (filtered_noise.h:80-92). Division by the spacing is
// replaced by a multiplication only when the spacing is a power of two
// (then both are exact); the fold is skipped when g is already in [0, n)
// (then floor(g/n) == 0 exactly, so the result is the same).
__device__ __forceinline__ void grid_locate(double x, double d, double inv_d,
                                            bool d_pow2, int n, int &ix,
                                            double &fx) {
    double g = d_pow2 ? x * inv_d : x / d;
    const double nd = (double)n;
    if (!(g >= 0.0 && g < nd)) g -= floor(g / nd) * nd;
    ix = (int)floor(g);
    if (ix >= n) {
        ix -= n;
        g -= nd;
    }
    fx = g - (double)ix;
    // Only a non-finite coordinate can leave [0, n) here; clamp so the
    // gather stays in bounds whatever the input (a no-op for finite x).
    ix = min(max(ix, 0), n - 1);
}

__device__ __forceinline__ void wrap4(int i, int n, int o[4]) {
    o[0] = (i == 0) ? n - 1 : i - 1;
    o[1] = i;
    o[2] = (i + 1 == n) ? 0 : i + 1;
    o[3] = (o[2] + 1 == n) ? 0 : o[2] + 1;
}

// True when d is a positive normal power of two: then x / d == x * (1/d)
// exactly, so a division by d may be replaced by a multiplication.
__host__ __device__ __forceinline__ bool dbl_is_pow2(double d) {
#ifdef __CUDA_ARCH__
    const long long b = __double_as_longlong(d);
#else
    long long b;
    memcpy(&b, &d, sizeof(b));
#endif
    return d > 0 && (b & 0x000FFFFFFFFFFFFFLL) == 0 && ((b >> 52) & 0x7FF) != 0;
}

// A spacing that the fixed-point locate may divide by (NoiseBSpline64::div_by):
// in [2^-500, 2^500], not the one mantissa (all ones) Markstein's theorem
// leaves out.
__host__ __device__ __forceinline__ bool qew_fixed_div_ok(double d) {
#ifdef __CUDA_ARCH__
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
#else
    unsigned long long b;
    memcpy(&b, &d, sizeof(b));
#endif
    const int ef = (int)(b >> 52);
    return ef >= 523 && ef <= 1523 && (b & 0x000FFFFFFFFFFFFFull) != 0x000FFFFFFFFFFFFFull;
}

// Line spacing dx = physical_size / n with exact shortcuts for its divisions.
// With the line's tension and force, the folded factors of the per-site
// combine as well (site_gradient, qew_model_kernels.cuh).
struct LineDx {
    double dx, inv_dx, inv_dx2;
    bool pow2, fixed;  // fixed: a spacing that slope() may divide by
    double half_dx, c_el, fdx;  // dx / 2, -Gamma / dx, dx f
    __host__ __device__ __forceinline__ double div(double v) const {
        return pow2 ? v * inv_dx : v / dx;
    }
    // v / dx to rounding, as div, for finite v of ordinary size by three FP64
    // instructions where the division takes nine (NoiseBSpline64::div_by).
    // The product with 1 / dx alone would scale every slope of a line by the
    // same rounding error.
    __device__ __forceinline__ double slope(double v) const {
        const double q = v * inv_dx;
        if (pow2) return q;
        if (!fixed || ((unsigned)__double2hiint(q) & 0x7FF00000u) > (1500u << 20)) return __ddiv_rn(v, dx);
        return fma(fma(-q, dx, v), inv_dx, q);
    }
    __host__ __device__ __forceinline__ double div2(double v) const {  // v / (dx*dx)
        return pow2 ? v * inv_dx2 : v / (dx * dx);
    }
};
__host__ __device__ __forceinline__ LineDx make_line_dx(double physical_size, int n,
                                                        double lt = 0.0, double f = 0.0) {
    LineDx L;
    L.dx = physical_size / (double)n;
    L.inv_dx = 1.0 / L.dx;
    L.inv_dx2 = 1.0 / (L.dx * L.dx);
    L.pow2 = dbl_is_pow2(L.dx);
    L.fixed = qew_fixed_div_ok(L.dx);
    L.half_dx = 0.5 * L.dx;
    L.c_el = -lt / L.dx;
    L.fdx = L.dx * f;
    return L;
}

// Physical x of the midpoint of an edge whose ends' indices add up to s:
// formed where it is used (a conversion and two products in FP64, which the
// constant-weight paths never need; as an argument they were computed for every
// edge: an FP32 Langevin step of 65536 sites 3.9 us with them, 3.05 without).
struct EdgeX {
    int s;
    double dx;
    __device__ __forceinline__ operator double() const { return (double)s * 0.5 * dx; }
};

// Marker for a spacing that is not a power of two.
constexpr int kPolyNotPow2 = 1 << 20;

struct NoiseBSpline64;
// NoiseBSpline64::dvdy (deriv) / value out of line: the FP64 16-tap sum, for
// the few edges that the fixed-point gather declines.
static __device__ __noinline__ double bspline_slow_call(const double *coef, int nx, int ny, double dx,
                                                        double dy, double inv_dx, double inv_dy,
                                                        double x, double y,
                                                        bool deriv QEW_OOB_WORDS);
__device__ __forceinline__ double bspline_slow(const NoiseBSpline64 &nz, bool deriv, double x,
                                               double y);

// DeviceNoise on x-fastest FP64 coefficients.
struct NoiseBSpline64 {
    const double *__restrict__ coef;  // [ny][nx]
    int nx, ny;
    double dx, dy, inv_dx, inv_dy;
    bool dx_pow2, dy_pow2;
    // Set when the line has n == nx points over the field's length with a
    // power-of-two spacing: every edge midpoint but the wrap edge is then at
    // grid x = e + 1/2 exactly, so its cell is e and its x weights are those
    // of t = 1/2 (bit-identical to locating it).
    bool xconst;
    // The field's cell-polynomial store (QEW_STORE_FP64_POLY) when it serves
    // this line (one point per field column), else null. ky: y * 2^ky == y / dy
    // exactly (kPolyNotPow2 when dy is not a power of two); kx the same for x.
    const long long *__restrict__ poly;
    int ky, kx;
    // The 16-tap sums in 64-bit fixed point (qew_fix.cuh): the field's bound
    // kb (-1: FP64 sums) and the units of 2 dV/dt / dy and of 6 V, for the
    // constant x weights (xconst and the store) and for general ones.
    int kb;
    double fx_dv_c, fx_v_c, fx_dv_g, fx_v_g;
    QEW_OOB_MEMBER

    // y / dy correctly rounded, from the correctly rounded 1 / dy (P.
    // Markstein, IBM J. Res. Dev. 34 (1990); C. Brisebarre, J.-M. Muller,
    // S. Raina, IEEE Trans. Comput. 53 (2004)): three FP64 instructions
    // where the division takes nine. d's exponent and y's are checked so
    // that nothing over- or underflows (fixed_div_ok, fx_locate).
    static __device__ __forceinline__ double div_by(double y, double d, double inv_d) {
        const double q = y * inv_d;
        return fma(fma(-q, d, y), inv_d, q);
    }
    // Cell and fraction of a physical coordinate, as grid_locate gives them;
    // false where the reference's fold has to decide (fx_cell).
    static __device__ __forceinline__ bool fx_locate(double x, double d, double inv_d, int kexp,
                                                     int n, int &ix, FxFrac &t) {
        if (kexp != kPolyNotPow2) return fx_cell(x, kexp, n, ix, t);
        const unsigned ef = ((unsigned)__double2hiint(x) >> 20) & 0x7FFu;
        if (ef - 523u > 1000u && x != 0.0) return false;  // |x| outside [2^-500, 2^500]
        return fx_cell(div_by(x, d, inv_d), 0, n, ix, t);
    }
    // The stencil's cubic at cell (ix, iy) from its row sums: x weights w(1/2)
    // times 48 in exact integers, E in units of 2^(K-52) / 48 ...
    __device__ __forceinline__ FxCubic fx_rows_const(int e, int iy) const {
        const bool inner = e >= 1 && e + 2 < nx && iy >= 1 && iy + 2 < ny;
        const double *p = coef + ((size_t)iy * (size_t)nx + (size_t)e);
        int xs[4], ys[4], kr[4];
        if (!inner) {
            wrap4(e, nx, xs);
            wrap4(iy, ny, ys);
        }
        long long E[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            double x[4];
            const double *row = p + (ptrdiff_t)(b - 1) * (ptrdiff_t)nx;
#pragma unroll
            for (int a = 0; a < 4; ++a)
                x[a] = inner ? QEW_LDGP(row + (a - 1), coef, (size_t)nx * (size_t)ny, oob)
                             : c(xs[a], ys[b]);
            E[b] = fx_row_const(x, kb, kr[b]);
        }
        return fx_cubic(E, kr, kb);
    }
    // ... or general x weights, E in units of 2^(K-57).
    __device__ __forceinline__ FxCubic fx_rows(int ix, FxFrac fx, int iy) const {
        const bool inner = ix >= 1 && ix + 2 < nx && iy >= 1 && iy + 2 < ny;
        const double *p = coef + ((size_t)iy * (size_t)nx + (size_t)ix);
        int xs[4], ys[4], kr[4];
        if (!inner) {
            wrap4(ix, nx, xs);
            wrap4(iy, ny, ys);
        }
        FxFrac wx[4];
        fx_weights(fx, wx);
        long long E[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            double x[4];
            const double *row = p + (ptrdiff_t)(b - 1) * (ptrdiff_t)nx;
#pragma unroll
            for (int a = 0; a < 4; ++a)
                x[a] = inner ? QEW_LDGP(row + (a - 1), coef, (size_t)nx * (size_t)ny, oob)
                             : c(xs[a], ys[b]);
            E[b] = fx_row_sum(x, wx, kb, kr[b]);
        }
        return fx_cubic(E, kr, kb);
    }

    __device__ __forceinline__ double c(int ix, int iy) const {
        ix = QEW_IDX(ix, nx, oob);
        iy = QEW_IDX(iy, ny, oob);
        return QEW_LDGP(coef + (size_t)iy * (size_t)nx + ix, coef, (size_t)nx * (size_t)ny, oob);
    }
    __device__ __forceinline__ void locate(double x, double y, int ixn[4],
                                           int iyn[4], double &fx,
                                           double &fy) const {
        int ix, iy;
        grid_locate(x, dx, inv_dx, dx_pow2, nx, ix, fx);
        grid_locate(y, dy, inv_dy, dy_pow2, ny, iy, fy);
        wrap4(ix, nx, ixn);
        wrap4(iy, ny, iyn);
    }
    // sample_value, filtered_noise.h:138-155
    __device__ __forceinline__ double value(double x, double y) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], wy[4];
        locate(x, y, ixn, iyn, fx, fy);
        bsw_value(fx, wx);
        bsw_value(fy, wy);
        double v = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) row += c(ixn[a], iyn[b]) * wy[b];
            v += wx[a] * row;
        }
        return v;
    }
    // sample_dy, filtered_noise.h:159-176
    __device__ __forceinline__ double dvdy(double x, double y) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], dwy[4];
        locate(x, y, ixn, iyn, fx, fy);
        bsw_value(fx, wx);
        bsw_deriv(fy, dwy);
        double dg = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) row += c(ixn[a], iyn[b]) * dwy[b];
            dg += wx[a] * row;
        }
        return dy_pow2 ? dg * inv_dy : dg / dy;
    }
    // Whether edge e sits at a half-integer column with the constant x
    // weights, on the store or on a grid that makes it exact; e becomes that
    // column. The wrap edge (e = nx - 1, at x = (n - 1) dx / 2) sits at one of
    // the columns when nx is even: without this its lane's general weights
    // came after the others' and a whole short line waited for it.
    __device__ __forceinline__ bool fx_const(int &e) const {
        if (!(poly || xconst)) return false;
        if (e + 1 < nx) return true;
        if (nx & 1) return false;
        e = (nx >> 1) - 1;
        return true;
    }
    // The cubic along y of edge e in row cell iy, constant x weights: one
    // 32-byte cell of the store, or the 16 taps; the same integers either way.
    __device__ __forceinline__ FxCubic fx_const_cell(int e, int iy) const {
        if (poly) {
            iy = QEW_IDX(iy, ny, oob);
            e = QEW_IDX(e, nx, oob);
            return fx_load_cell(poly + ((size_t)iy * (size_t)nx + (size_t)e) * 4);
        }
        return fx_rows_const(e, iy);
    }
    // The sums 2 dV/dt and 6 V of cell q at fraction t, in FP64 units of fx_dv_*
    // and fx_v_*.
    static __device__ __forceinline__ double fx_dv(const FxCubic &q, FxFrac t) {
        return fx_to_double(fx_dt2(q, t), -q.d);
    }
    static __device__ __forceinline__ double fx_v(const FxCubic &q, FxFrac t) {
        return fx_to_double(fx_6v(q, t), -q.d);
    }
    // Row cell and fraction of the edge midpoint at height a / 2.
    // (On the store of a spacing that is no power of two by one product, within
    // an ulp of the quotient.)
    __device__ __forceinline__ bool fx_row(double a, int &iy, FxFrac &t) const {
        if (poly && ky == kPolyNotPow2) return fx_cell(a * (0.5 * inv_dy), 0, ny, iy, t);
        return fx_locate(a, 2.0 * dy, 0.5 * inv_dy, ky == kPolyNotPow2 ? ky : ky - 1, ny, iy, t);
    }
    // dV/dy of an edge e < nx - 1 on the store as R 2^-d in units of fx_dv_c;
    // false for a NaN.
    __device__ __forceinline__ bool dvdy_edge_store(int e, double a, long long &R, int &d) const {
        int iy;
        FxFrac fy;
        if (!fx_row(a, iy, fy)) {
            double t;
            grid_locate(a * 0.5, dy, inv_dy, dy_pow2, ny, iy, t);
            if (!(t >= 0.0)) return false;
            fy = fx_frac((unsigned long long)(fmin(t, 1.0 - 0x1p-53) * 0x1p64));
        }
        const FxCubic q = fx_const_cell(e, iy);
        R = fx_dt2(q, fy);
        d = q.d;
        return true;
    }
    __device__ __forceinline__ double dvdy_edge_store(int e, double a) const {
        long long R;
        int d;
        return dvdy_edge_store(e, a, R, d) ? __dmul_rn(fx_to_double(R, -d), fx_dv_c) : a - a;
    }
    // dV/dy / V at the midpoint of edge e (xc its physical x, a the sum of its
    // two heights) in fixed point; what its locate declines (a rounded period end, huge
    // heights, non-finite ones) is summed in FP64. The last product is never
    // contracted, so every kernel gets the same bits.
    __device__ __forceinline__ double dvdy_edge_sum(int e, EdgeX xc, double a) const {
        if (kb >= 0) {
            int ix, iy;
            FxFrac fx, fy;
            if (fx_row(a, iy, fy)) {
                if (fx_const(e))
                    return __dmul_rn(fx_dv(fx_const_cell(e, iy), fy), fx_dv_c);
                if (fx_locate(xc, dx, inv_dx, kx, nx, ix, fx)) {
                    return __dmul_rn(fx_dv(fx_rows(ix, fx, iy), fy), fx_dv_g);
                }
            }
        }
        return bspline_slow(*this, true, xc, a * 0.5);
    }
    __device__ __forceinline__ double value_edge_sum(int e, EdgeX xc, double a) const {
        if (kb >= 0) {
            int ix, iy;
            FxFrac fx, fy;
            if (fx_row(a, iy, fy)) {
                if (fx_const(e))
                    return __dmul_rn(fx_v(fx_const_cell(e, iy), fy), fx_v_c);
                if (fx_locate(xc, dx, inv_dx, kx, nx, ix, fx)) {
                    return __dmul_rn(fx_v(fx_rows(ix, fx, iy), fy), fx_v_g);
                }
            }
        }
        return bspline_slow(*this, false, xc, a * 0.5);
    }
    // Both at once, from one cell: the numbers that the two give.
    __device__ __forceinline__ void both_edge_sum(int e, EdgeX xc, double a, double &v,
                                                  double &dv) const {
        if (kb >= 0) {
            int ix, iy;
            FxFrac fx, fy;
            if (fx_row(a, iy, fy)) {
                const bool cst = fx_const(e);
                if (cst || fx_locate(xc, dx, inv_dx, kx, nx, ix, fx)) {
                    const FxCubic q = cst ? fx_const_cell(e, iy) : fx_rows(ix, fx, iy);
                    v = __dmul_rn(fx_v(q, fy), cst ? fx_v_c : fx_v_g);
                    dv = __dmul_rn(fx_dv(q, fy), cst ? fx_dv_c : fx_dv_g);
                    return;
                }
            }
        }
        v = bspline_slow(*this, false, xc, a * 0.5);
        dv = bspline_slow(*this, true, xc, a * 0.5);
    }
    // sample, filtered_noise.h:103-134
    __device__ __forceinline__ void sample(double x, double y, double &v,
                                           double &dvdx_,
                                           double &dvdy_) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], dwx[4], wy[4], dwy[4];
        locate(x, y, ixn, iyn, fx, fy);
        bsw_value(fx, wx);
        bsw_deriv(fx, dwx);
        bsw_value(fy, wy);
        bsw_deriv(fy, dwy);
        double vv = 0, gx = 0, gy = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0, row_dy = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const double cc = c(ixn[a], iyn[b]);
                row += cc * wy[b];
                row_dy += cc * dwy[b];
            }
            vv += wx[a] * row;
            gx += dwx[a] * row;
            gy += wx[a] * row_dy;
        }
        v = vv;
        dvdx_ = dx_pow2 ? gx * inv_dx : gx / dx;
        dvdy_ = dy_pow2 ? gy * inv_dy : gy / dy;
    }
};

static __device__ __noinline__ double bspline_slow_call(const double *coef, int nx, int ny, double dx,
                                                        double dy, double inv_dx, double inv_dy,
                                                        double x, double y,
                                                        bool deriv QEW_OOB_WORDS) {
    NoiseBSpline64 nz;
    nz.coef = coef;
    nz.nx = nx;
    nz.ny = ny;
    nz.dx = dx;
    nz.dy = dy;
    nz.inv_dx = inv_dx;
    nz.inv_dy = inv_dy;
    nz.dx_pow2 = dbl_is_pow2(dx);
    nz.dy_pow2 = dbl_is_pow2(dy);
#ifdef QEW_BOUNDS_CHECK
    nz.oob = oob;
#endif
    return deriv ? nz.dvdy(x, y) : nz.value(x, y);
}
__device__ __forceinline__ double bspline_slow(const NoiseBSpline64 &nz, bool deriv, double x,
                                               double y) {
#ifdef QEW_BOUNDS_CHECK
    return bspline_slow_call(nz.coef, nz.nx, nz.ny, nz.dx, nz.dy, nz.inv_dx, nz.inv_dy, x, y, deriv, nz.oob);
#else
    return bspline_slow_call(nz.coef, nz.nx, nz.ny, nz.dx, nz.dy, nz.inv_dx, nz.inv_dy, x, y, deriv);
#endif
}

// ------------------------------------------- reference-exact FP64 arithmetic
// The reference is ISO C++ evaluated expression by expression: every a*b+c is
// a rounded product and a rounded sum, every weight a true division by 6
// (filtered_noise.h:33-62). The __d*_rn intrinsics are never contracted into
// FMAs, so the functions below reproduce those operations bit for bit (the
// CPU oracle is compiled with -ffp-contract=off for the same reason).
__device__ __forceinline__ void bsw_value_ref(double t, double w[4]) {
    const double t2 = __dmul_rn(t, t);
    const double t3 = __dmul_rn(t2, t);
    const double omt = __dsub_rn(1.0, t);
    w[0] = __ddiv_rn(__dmul_rn(__dmul_rn(omt, omt), omt), 6.0);
    w[1] = __ddiv_rn(__dadd_rn(__dsub_rn(4.0, __dmul_rn(6.0, t2)), __dmul_rn(3.0, t3)), 6.0);
    w[2] = __ddiv_rn(__dsub_rn(__dadd_rn(__dadd_rn(1.0, __dmul_rn(3.0, t)), __dmul_rn(3.0, t2)),
                               __dmul_rn(3.0, t3)),
                     6.0);
    w[3] = __ddiv_rn(t3, 6.0);
}
__device__ __forceinline__ void bsw_deriv_ref(double t, double dw[4]) {
    const double t2 = __dmul_rn(t, t);
    const double omt = __dsub_rn(1.0, t);
    dw[0] = __ddiv_rn(__dmul_rn(-omt, omt), 2.0);
    dw[1] = __ddiv_rn(__dadd_rn(__dmul_rn(-12.0, t), __dmul_rn(9.0, t2)), 6.0);
    dw[2] = __ddiv_rn(__dsub_rn(__dadd_rn(3.0, __dmul_rn(6.0, t)), __dmul_rn(9.0, t2)), 6.0);
    dw[3] = __ddiv_rn(__dmul_rn(3.0, t2), 6.0);
}

// DeviceNoise with the reference's arithmetic exactly (filtered_noise.h:77-176):
// the same locate, true divisions, unfused sums in the reference's order.
struct NoiseBSpline64Ref {
    NoiseBSpline64 b;  // coefficients, extents and spacings (its xconst is not used)
    __device__ __forceinline__ double c(int ix, int iy) const { return b.c(ix, iy); }
    __device__ __forceinline__ double value(double x, double y) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], wy[4];
        b.locate(x, y, ixn, iyn, fx, fy);
        bsw_value_ref(fx, wx);
        bsw_value_ref(fy, wy);
        double v = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) row = __dadd_rn(row, __dmul_rn(c(ixn[a], iyn[k]), wy[k]));
            v = __dadd_rn(v, __dmul_rn(wx[a], row));
        }
        return v;
    }
    __device__ __forceinline__ double dvdy(double x, double y) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], dwy[4];
        b.locate(x, y, ixn, iyn, fx, fy);
        bsw_value_ref(fx, wx);
        bsw_deriv_ref(fy, dwy);
        double dg = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) row = __dadd_rn(row, __dmul_rn(c(ixn[a], iyn[k]), dwy[k]));
            dg = __dadd_rn(dg, __dmul_rn(wx[a], row));
        }
        return __ddiv_rn(dg, b.dy);
    }
    __device__ __forceinline__ void sample(double x, double y, double &v, double &dvdx_,
                                           double &dvdy_) const {
        int ixn[4], iyn[4];
        double fx, fy, wx[4], dwx[4], wy[4], dwy[4];
        b.locate(x, y, ixn, iyn, fx, fy);
        bsw_value_ref(fx, wx);
        bsw_deriv_ref(fx, dwx);
        bsw_value_ref(fy, wy);
        bsw_deriv_ref(fy, dwy);
        double vv = 0, gx = 0, gy = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            double row = 0, row_dy = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double cc = c(ixn[a], iyn[k]);
                row = __dadd_rn(row, __dmul_rn(cc, wy[k]));
                row_dy = __dadd_rn(row_dy, __dmul_rn(cc, dwy[k]));
            }
            vv = __dadd_rn(vv, __dmul_rn(wx[a], row));
            gx = __dadd_rn(gx, __dmul_rn(dwx[a], row));
            gy = __dadd_rn(gy, __dmul_rn(wx[a], row_dy));
        }
        v = vv;
        dvdx_ = __ddiv_rn(gx, b.dx);
        dvdy_ = __ddiv_rn(gy, b.dy);
    }
};

// True for the functors whose callers must evaluate the rest of the model
// (elastic force, combine) with the reference's unfused arithmetic too.
template <class Noise>
struct noise_is_ref {
    static constexpr bool value = false;
};
template <>
struct noise_is_ref<NoiseBSpline64Ref> {
    static constexpr bool value = true;
};

// Analytic potentials of the reference's tests; value()/dvdy() go through
// sample() exactly like detail::noise_value/noise_dvdy (qew_model.h:31-46).
struct NoiseZero {
    __device__ __forceinline__ void sample(double, double, double &v,
                                           double &a, double &b) const {
        v = 0; a = 0; b = 0;
    }
    __device__ __forceinline__ double value(double, double) const { return 0; }
    __device__ __forceinline__ double dvdy(double, double) const { return 0; }
};
struct NoiseConst {
    double v0;
    __device__ __forceinline__ void sample(double, double, double &v,
                                           double &a, double &b) const {
        v = v0; a = 0; b = 0;
    }
    __device__ __forceinline__ double value(double, double) const { return v0; }
    __device__ __forceinline__ double dvdy(double, double) const { return 0; }
};
struct NoiseHarmonic {  // HarmonicWell{k, y0}
    double k, y0;
    __device__ __forceinline__ void sample(double, double y, double &v,
                                           double &a, double &b) const {
        const double d = y - y0;
        v = 0.5 * k * d * d; a = 0; b = k * d;
    }
    __device__ __forceinline__ double value(double, double y) const {
        const double d = y - y0;
        return 0.5 * k * d * d;
    }
    __device__ __forceinline__ double dvdy(double, double y) const {
        return k * (y - y0);
    }
};
struct NoiseWashboard {  // SinusoidNoise{A, k}: V = A cos(k y)
    double A, k;
    __device__ __forceinline__ void sample(double, double y, double &v,
                                           double &a, double &b) const {
        v = A * cos(k * y); a = 0; b = -A * k * sin(k * y);
    }
    __device__ __forceinline__ double value(double, double y) const {
        return A * cos(k * y);
    }
    __device__ __forceinline__ double dvdy(double, double y) const {
        return -A * k * sin(k * y);
    }
};
struct NoiseSinCos {  // AnalyticNoise{amp, kx, ky}
    double amp, kx, ky;
    __device__ __forceinline__ void sample(double x, double y, double &v,
                                           double &a, double &b) const {
        v = amp * sin(kx * x) * cos(ky * y);
        a = amp * kx * cos(kx * x) * cos(ky * y);
        b = -amp * ky * sin(kx * x) * sin(ky * y);
    }
    __device__ __forceinline__ double value(double x, double y) const {
        return amp * sin(kx * x) * cos(ky * y);
    }
    __device__ __forceinline__ double dvdy(double x, double y) const {
        return -amp * ky * sin(kx * x) * sin(ky * y);
    }
};

#ifdef QEW_BOUNDS_CHECK
// The error words a functor carries (none for the analytic potentials).
template <class Noise>
__device__ __forceinline__ unsigned long long *qew_noise_oob(const Noise &) { return nullptr; }
__device__ __forceinline__ unsigned long long *qew_noise_oob(const NoiseBSpline64 &nz) {
    return nz.oob;
}
__device__ __forceinline__ unsigned long long *qew_noise_oob(const NoiseBSpline64Ref &nz) {
    return nz.b.oob;
}
#endif

// Edge accessors for every functor, at the midpoint a / 2 of an edge whose
// heights add up to a: the B-spline one has its own path.
template <class Noise>
__device__ __forceinline__ double noise_dvdy_edge(const Noise &nz, int, EdgeX xc, double a) {
    return nz.dvdy(xc, a * 0.5);
}
template <class Noise>
__device__ __forceinline__ double noise_value_edge(const Noise &nz, int, EdgeX xc, double a) {
    return nz.value(xc, a * 0.5);
}
__device__ __forceinline__ double noise_dvdy_edge(const NoiseBSpline64 &nz, int e, EdgeX xc,
                                                  double a) {
    return nz.dvdy_edge_sum(e, xc, a);
}
__device__ __forceinline__ double noise_value_edge(const NoiseBSpline64 &nz, int e, EdgeX xc,
                                                   double a) {
    return nz.value_edge_sum(e, xc, a);
}

template <class Noise>
__device__ __forceinline__ void noise_both_edge(const Noise &nz, int e, EdgeX xc, double a,
                                                double &v, double &dv) {
    v = noise_value_edge(nz, e, xc, a);
    dv = noise_dvdy_edge(nz, e, xc, a);
}
__device__ __forceinline__ void noise_both_edge(const NoiseBSpline64 &nz, int e, EdgeX xc, double a,
                                                double &v, double &dv) {
    nz.both_edge_sum(e, xc, a, v, dv);
}

// Host helpers building the functors from a field handle.
static inline bool qew_is_pow2(double d) {
    int e;
    const double m = frexp(d, &e);
    return d > 0 && m == 0.5;
}
static inline NoiseBSpline64 make_bspline64(const qew_field *f, int n = 0,
                                            double physical_size = 0) {
    NoiseBSpline64 nz;
    nz.xconst = (n > 0 && n == f->nx && physical_size == f->Lx && qew_is_pow2(f->dx));
    nz.coef = f->coef64;
    nz.nx = f->nx;
    nz.ny = f->ny;
    nz.dx = f->dx;
    nz.dy = f->dy;
    nz.inv_dx = 1.0 / f->dx;
    nz.inv_dy = 1.0 / f->dy;
    nz.dx_pow2 = qew_is_pow2(f->dx);
    nz.dy_pow2 = qew_is_pow2(f->dy);
    nz.poly = (f->poly && n > 0 && n == f->nx && physical_size == f->Lx) ? f->poly : nullptr;
    {
        int e;
        const double m = frexp(f->dy, &e);  // dy = m 2^e
        nz.ky = (f->dy > 0 && m == 0.5) ? 1 - e : kPolyNotPow2;
        const double mx = frexp(f->dx, &e);
        nz.kx = (f->dx > 0 && mx == 0.5) ? 1 - e : kPolyNotPow2;
    }
    nz.kb = -1;
    nz.fx_dv_c = nz.fx_v_c = nz.fx_dv_g = nz.fx_v_g = 0.0;
    if (f->fixb >= 0 && qew_fixed_div_ok(f->dx) && qew_fixed_div_ok(f->dy)) {
        const int K = f->fixb - 1022;  // |coefficient| < 2^K
        nz.fx_dv_c = ldexp(1.0, K - 53) / (48.0 * f->dy);
        nz.fx_v_c = ldexp(1.0, K - 52) / 288.0;
        nz.fx_dv_g = ldexp(1.0, K - 58) / f->dy;
        nz.fx_v_g = ldexp(1.0, K - 57) / 6.0;
        // the units and R times them stay normal numbers, else FP64 sums
        if (fmin(nz.fx_dv_g, nz.fx_v_g) > 0x1p-700 && fmax(nz.fx_dv_c, nz.fx_v_c) < 0x1p+900)
            nz.kb = f->fixb;
    }
#ifdef QEW_BOUNDS_CHECK
    nz.oob = qew_bounds_words();
#endif
    return nz;
}

// As qew_dispatch_noise, with the B-spline kind as NoiseBSpline64Ref (the
// reference's arithmetic bit for bit).
template <class Fn>
qew_status qew_dispatch_noise_ref(qew_ctx *ctx, const qew_field *f, Fn &&fn);

// Calls `fn(noise_functor)` with the functor matching the field's kind.
// Returns QEW_ERR_INVALID for an unknown kind or a B-spline field without
// FP64 coefficients. n / physical_size describe the line (0: unknown).
template <class Fn>
qew_status qew_dispatch_noise(qew_ctx *ctx, const qew_field *f, Fn &&fn, int n = 0,
                              double physical_size = 0) {
    switch (f->kind) {
    case QEW_FIELD_BSPLINE:
        if (!f->coef64)
            return qew_fail(ctx, QEW_ERR_INVALID,
                            "field has no FP64 coefficients (created without "
                            "QEW_STORE_FP64)");
        return fn(make_bspline64(f, n, physical_size));
    case QEW_FIELD_ZERO: return fn(NoiseZero{});
    case QEW_FIELD_CONST: return fn(NoiseConst{f->p0});
    case QEW_FIELD_HARMONIC: return fn(NoiseHarmonic{f->p0, f->p1});
    case QEW_FIELD_WASHBOARD: return fn(NoiseWashboard{f->p0, f->p1});
    case QEW_FIELD_SINCOS: return fn(NoiseSinCos{f->p0, f->p1, f->p2});
    default:
        return qew_fail(ctx, QEW_ERR_INVALID, "unknown field kind %d", f->kind);
    }
}

template <class Fn>
qew_status qew_dispatch_noise_ref(qew_ctx *ctx, const qew_field *f, Fn &&fn) {
    if (f->kind == QEW_FIELD_BSPLINE) {
        if (!f->coef64)
            return qew_fail(ctx, QEW_ERR_INVALID,
                            "field has no FP64 coefficients (created without "
                            "QEW_STORE_FP64)");
        return fn(NoiseBSpline64Ref{make_bspline64(f)});
    }
    return qew_dispatch_noise(ctx, f, fn);
}

// ------------------------------------------------------ block reductions
template <int BS>
__device__ __forceinline__ double block_sum(double v, double *s_warp) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s_warp[w] = v;
    __syncthreads();
    double r = 0;
    if (w == 0) {
        r = (lane < BS / 32) ? s_warp[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;  // valid in thread 0
}
