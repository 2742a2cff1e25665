// qew_fix.cuh -- the FP64 gather on the integer pipe: 64-bit fixed point.
//
// GB300 issues one FP64 instruction of a warp every 64 cycles per scheduler
// (measured: DADD, DMUL, DFMA, compares and conversions alike, with one warp
// already saturating it), an integer instruction every 1-2. The 16-tap
// gather's sums are of the scale of their own taps -- the stencil's largest
// bounds every partial sum -- so each stencil takes its own unit, 2^-57 of that
// bound: about 2^-4 of an FP64 ulp there, where the FP64 sum rounds some twenty
// times at its terms' own ulps. (One unit for the whole field loses what a weak
// region has beside a strong one: with coefficients 4e6 apart the weak region's
// dV/dy was wrong by 5e-11 of its own scale. The stencil's unit costs some 40
// integer instructions an edge.) Measured, with
// the shorter combine of qew_model_kernels.cuh: the gradient of a
// 262144-point arclength line 45.1 -> 12.3 us, of three 100003-point lines off the
// field's grid 92.2 -> 20.5 us (in one launch), 8 lines of 2^20 points 1002 -> 218 us.
//
// Formats. A tap is an int64 X with c = X 2^(K-57), |c| < 2^K for its row of the
// stencil; the four rows' sums are then shifted to the stencil's largest K,
// which is d binary orders below the field's (taken when the field is built):
// 0 <= d <= kFxOrders, weaker stencils keep the unit of the last.
// A fraction t in [0, 1) is T = T1 2^31 + T0 in units of 2^-62, two 31-bit limbs; its product
// with an int64 w, |w| < 2^62, is three 32 x 32 + 64-bit multiply-adds
// (fx_mul, truncated below the unit of w).
#pragma once

#include <cuda_runtime.h>

#include <cstring>

// Fraction limbs: t = (t1 * 2^31 + t0) * 2^-62.
struct FxFrac {
    int t1, t0;
};

__host__ __device__ __forceinline__ FxFrac fx_frac(unsigned long long t64) {  // t = t64 * 2^-64
    return FxFrac{(int)(t64 >> 33), (int)((unsigned)(t64 >> 2) & 0x7fffffffu)};
}

// floor-like (w * t): within 2 units of w * t. |w| < 2^62.
__host__ __device__ __forceinline__ long long fx_mul(long long w, FxFrac t) {
    const int w1 = (int)(w >> 31);
    const int w0 = (int)((unsigned)w & 0x7fffffffu);
    const long long mid = (long long)w1 * t.t0 + (long long)w0 * t.t1;
    return (long long)w1 * t.t1 + (mid >> 31);
}

// u >> s for s >= 0, zero from 64 on (the PTX shift clamps its amount).
__host__ __device__ __forceinline__ unsigned long long fx_shr(unsigned long long u, int s) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(u), "r"(s));
    return r;
#else
    return s < 64 ? u >> s : 0ull;
#endif
}
__host__ __device__ __forceinline__ unsigned long long fx_shl(unsigned long long u, int s) {
#ifdef __CUDA_ARCH__
    unsigned long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(u), "r"(s));
    return r;
#else
    return s < 64 ? u << s : 0ull;
#endif
}
__host__ __device__ __forceinline__ long long fx_sar(long long u, int s) {  // s >= 0
#ifdef __CUDA_ARCH__
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(u), "r"(s));
    return r;
#else
    return u >> (s < 63 ? s : 63);
#endif
}
// Leading zeros (64 for 0).
__host__ __device__ __forceinline__ int fx_clz(unsigned long long u) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)u);
#else
    return u ? __builtin_clzll(u) : 64;
#endif
}
// The limbs of a signed number v * 2^-62, |v| < 2^62.
__host__ __device__ __forceinline__ FxFrac fx_limbs(long long v) {
    return FxFrac{(int)(v >> 31), (int)((unsigned)v & 0x7fffffffu)};
}

// Orders of magnitude below the field's largest coefficient that a stencil's
// unit follows (8 bits in the store's cells; a factor 2^255).
constexpr int kFxOrders = 255;

// The field's biased exponent from the bits of its largest |coefficient|: 1023
// for the zero field, -1 for one that fixed point does not serve (a stencil's
// unit has to stay among the normal numbers, and zero and subnormal taps below it).
__host__ __device__ __forceinline__ int qew_fix_bound(unsigned long long max_bits) {
    const int ex = (int)(max_bits >> 52);
    return max_bits == 0 ? 1023 : (ex >= kFxOrders + 65 && ex <= 1792) ? ex : -1;
}

// Biased exponent of the largest of four numbers, at least low.
__device__ __forceinline__ int fx_row_exp(double a, double b, double c, double d, int low) {
    auto ex = [](double v) { return (int)(((unsigned)__double2hiint(v) >> 20) & 0x7FFu); };
    return max(max(max(ex(a), ex(b)), max(ex(c), ex(d))), low);
}

// An FP64 number c, |c| < 2^K with K = kb - 1022, in units of
// 2^(K - 53 - kUp) (truncated towards zero; kUp <= 10). Subnormals give 0.
template <int kUp>
__device__ __forceinline__ long long fx_tap(double c, int kb) {
    const unsigned hi = (unsigned)__double2hiint(c), lo = (unsigned)__double2loint(c);
    const int s = kb - (int)((hi >> 20) & 0x7FFu);  // >= 0: the field's bound is kb
    const unsigned mh = (hi & 0x000FFFFFu) | 0x00100000u;
    const unsigned long long m =
        ((unsigned long long)__funnelshift_l(lo, mh, kUp) << 32) | (unsigned long long)(lo << kUp);
    const long long sg = (long long)((int)hi >> 31);
    return ((long long)fx_shr(m, s) ^ sg) - sg;
}

// The bits of r * 2^k as an FP64 number, rounded to nearest (ties away from
// zero), for a result in the normal range: the integer form of the
// conversion, which the FP64 unit would take 64 cycles for.
__host__ __device__ __forceinline__ unsigned long long fx_double_bits(long long r, int k) {
    const long long sg = r >> 63;
    const unsigned long long a = (unsigned long long)((r ^ sg) - sg);
    const int lz = fx_clz(a);
    const unsigned long long n = fx_shl(a, lz);  // leading bit at 63 (0 for r == 0)
    const unsigned long long m = (n >> 11) + ((n >> 10) & 1ull);
    const unsigned long long b = ((unsigned long long)(unsigned)(1085 + k - lz) << 52) + m;
    return a ? (b | ((unsigned long long)sg << 63)) : 0ull;
}
__device__ __forceinline__ double fx_to_double(long long r, int k = 0) {
    return __longlong_as_double((long long)fx_double_bits(r, k));
}

__host__ __device__ __forceinline__ unsigned long long fx_bits(double a) {
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(a);
#else
    unsigned long long b;
    memcpy(&b, &a, sizeof(b));
    return b;
#endif
}

// Row cell and fraction of g = a * 2^k in a period of n cells, from the bits
// of a: the numbers that the reference's fold gives (filtered_noise.h:80-92),
// which rounds a negative g's sum with the period to FP64. False for what the
// FP64 code has to decide: non-finite or subnormal a, |g| >= 2^50, and, outside
// the first two periods about zero, the last two FP64 numbers of a period,
// where the reference's division by the period may round up. (Declining the
// whole last cell, and |g| >= 2^30, made 8 lines of 2^20 points there 1530 us on 16
// taps where FP64 alone took 1166; now 251 and 269.)
//
// fx_fold: g outside the field's first period (b: the bits of a, e: g's binary
// exponent), out of line: with its code in every gather the Rosso-Krauth search
// outgrew the instruction cache (200 sweeps of 2048 sites 6.76 ms, 5.87 so; a
// line outside the first period pays 3 % for the call).
struct FxFold {
    unsigned long long f;
    int iy, ok;
};
static __host__ __device__ __noinline__ FxFold fx_fold(unsigned long long b, int e, int n) {
    const unsigned long long m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const int up = 12 + e;
    unsigned long long f = up >= 0 ? fx_shl(m, up) : fx_shr(m, -up);
    int iy = e >= 0 ? (int)fx_shr(m, 52 - e) : 0;
    bool later = false;  // than the two periods about zero
    if (e > 29) {        // up to 50 bits: whole periods taken out in 64-bit arithmetic
        const unsigned long long whole = fx_shr(m, 52 - e);
        later = whole >= (unsigned long long)n;
        iy = (int)(whole % (unsigned long long)n);
    } else if (iy >= n) {
        later = true;
        iy %= n;
    }
    // the fraction lies two units of a's last bit or more before the end
    const auto inside = [&]() { return f < 0ull - fx_shl(2ull, up); };
    if ((long long)b >= 0) return FxFold{f, iy, !later || iy + 1 < n || inside()};
    if (n == 1) return FxFold{f, 0, 0};
    // bits below 2^-64 leave a mark in the lowest one, for the sums with the
    // period that lie next to halfway between two numbers
    const bool cut = up < 0 && fx_shl(f, -up) != m;
    iy = (f || cut) ? n - 1 - iy : (iy ? n - iy : 0);
    f = cut ? ~f | 1ull : 0ull - f;
    const bool ok = !later || iy + 1 < n || inside();
    if (iy > 0) {  // round g + period to FP64 (to nearest even)
#ifdef __CUDA_ARCH__
        const int drop = 43 - __clz(iy);  // 12 + floor(log2(iy))
#else
        const int drop = 43 - __builtin_clz((unsigned)iy);
#endif
        const unsigned long long add = ((1ull << (drop - 1)) - 1ull) + ((f >> drop) & 1ull);
        const bool carry = f + add < f;
        f = ((f + add) >> drop) << drop;
        if (carry) {
            f = 0ull;
            iy = (iy + 1 == n) ? 0 : iy + 1;
        }
    }
    return FxFold{f, iy, ok};
}

__host__ __device__ __forceinline__ bool fx_cell64(double a, int k, int n, int &iy,
                                                   unsigned long long &f) {
    const unsigned long long b = fx_bits(a);
    const int ef = (int)(b >> 52) & 0x7FF;
    const int e = ef + k - 1023;
    if (ef == 0 || ef == 2047 || e > 49) {
        iy = 0;
        f = 0ull;
        return (b << 1) == 0ull;
    }
    const unsigned long long m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const int up = 12 + e;  // fraction bits to the top of 64 (the integer part leaves)
    f = up >= 0 ? fx_shl(m, up) : fx_shr(m, -up);
    iy = e >= 0 ? (int)fx_shr(m, 52 - e) : 0;
    bool ok = true;
    if ((long long)b < 0 || iy >= n || e > 29) {
        const FxFold r = fx_fold(b, e, n);
        iy = r.iy;
        f = r.f;
        ok = r.ok;
    }
    return ok;
}
__device__ __forceinline__ bool fx_cell(double a, int k, int n, int &iy, FxFrac &t) {
    unsigned long long f;
    const bool ok = fx_cell64(a, k, n, iy, f);
    t = fx_frac(f);
    return ok;
}
// f * 2^-64 as a float, rounded to nearest even (the conversion of the exact
// FP64 fraction; one below 2^-64 is 0 here).
__device__ __forceinline__ float fx_frac_to_float(unsigned long long f) {
    const int lz = __clzll((long long)f);
    const unsigned long long n = fx_shl(f, lz), rem = n << 24;
    unsigned m = (unsigned)(n >> 40);
    m += (rem > (1ull << 63) || (rem == (1ull << 63) && (m & 1u))) ? 1u : 0u;
    return f ? __int_as_float(((126 - lz) << 23) + (int)(m - 0x800000u)) : 0.0f;
}

// The cubic along y in one cell, from the four stencil rows' sums E
// (|E| <= 2^57.6, in some unit): with u = E0 - 2 E1 + E2 and
// w = (E3 - E0) - 3 (E2 - E1) (filtered_noise.h:33-62 expanded in t)
//   2 dV/dt = p + t (2u + t w),   6 V = v + t (3p + t (3u + t w)),
// p = E2 - E0, v = E0 + 4 E1 + E2. Every bracket is a mean of differences of
// E, so it stays below 12 max|E| < 2^62 (fx_mul's range).
struct FxCubic {
    long long v, p, u2, w;  // u2 = 2u
    int d;                  // the unit's orders below the field's
};
// Er: the rows' sums, each in the unit of its own exponent kr (K = kr - 1022);
// kb: the field's.
__device__ __forceinline__ FxCubic fx_cubic(const long long Er[4], const int kr[4], int kb) {
    const int kc = max(max(kr[0], kr[1]), max(kr[2], kr[3]));
    long long E[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) E[b] = fx_sar(Er[b], kc - kr[b]);
    const long long s = E[0] + E[2];
    return FxCubic{s + 4 * E[1], E[2] - E[0], 2 * s - 4 * E[1], (E[3] - E[0]) - 3 * (E[2] - E[1]),
                   kb - kc};
}
__device__ __forceinline__ long long fx_dt2(const FxCubic &c, FxFrac t) {
    return c.p + fx_mul(c.u2 + fx_mul(c.w, t), t);
}
__device__ __forceinline__ long long fx_6v(const FxCubic &c, FxFrac t) {
    return c.v + fx_mul(3 * c.p + fx_mul(c.u2 + (c.u2 >> 1) + fx_mul(c.w, t), t), t);
}
// One cell of the cell-polynomial store: 32 bytes, 32-byte aligned. d lies in
// the bits that the three numbers leave free: |p| <= 2 max|E| < 2^59, |u2| and
// |w| <= 8 max|E| < 2^61.
__device__ __forceinline__ long long fx_low_bits(long long v, int free) {  // sign-extended
    const int hi = (int)((unsigned)(v >> 32) << free) >> free;
    return ((long long)hi << 32) | (long long)(unsigned)v;
}
__device__ __forceinline__ FxCubic fx_load_cell(const long long *p) {
    FxCubic c;
    long long rp, ru, rw;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(c.v), "=l"(rp), "=l"(ru), "=l"(rw)
        : "l"(p));
    c.p = fx_low_bits(rp, 4);
    c.u2 = fx_low_bits(ru, 2);
    c.w = fx_low_bits(rw, 2);
    c.d = (int)((((unsigned)(rp >> 32) >> 28) << 4) | (((unsigned)(ru >> 32) >> 30) << 2) |
                ((unsigned)(rw >> 32) >> 30));
    return c;
}
__device__ __forceinline__ void fx_store_cell(long long *p, const FxCubic &c) {
    const long long m60 = (1ll << 60) - 1, m62 = (1ll << 62) - 1;
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(c.v),
                 "l"((c.p & m60) | ((long long)(c.d >> 4) << 60)),
                 "l"((c.u2 & m62) | ((long long)((c.d >> 2) & 3) << 62)),
                 "l"((c.w & m62) | ((long long)(c.d & 3) << 62))
                 : "memory");
}

// The cubic B-spline weights (filtered_noise.h:33-44) at fraction t, in units
// of 2^-62 as limbs.
__device__ __forceinline__ void fx_weights(FxFrac t, FxFrac w[4]) {
    const long long one = (1ll << 62) - 1;
    const FxFrac sixth{357913941, 715827882};  // 2^62 / 6
    const long long T = ((long long)t.t1 << 31) | (long long)t.t0;
    const long long o = one - T;
    const FxFrac fo = fx_limbs(o);
    const long long t2 = fx_mul(T, t), o3 = fx_mul(fx_mul(o, fo), fo), t3 = fx_mul(t2, t);
    const long long w0 = fx_mul(o3, sixth), w3 = fx_mul(t3, sixth);
    const long long w1 = 3074457345618258603ll - t2 + (t3 >> 1);  // 2/3 - t^2 + t^3/2
    w[0] = fx_limbs(w0);
    w[1] = fx_limbs(w1);
    w[2] = fx_limbs(one - w0 - w1 - w3);
    w[3] = fx_limbs(w3);
}

// A stencil row's sum in the unit of its own exponent kr (at least kb -
// kFxOrders, kb the field's): with the weights w(1/2) times 48, in units of
// 2^(kr - 1074) / 48; with the weights w, in units of 2^(kr - 1079).
__device__ __forceinline__ long long fx_row_const(const double x[4], int kb, int &kr) {
    kr = fx_row_exp(x[0], x[1], x[2], x[3], kb - kFxOrders);
    return ((fx_tap<4>(x[0], kr) + fx_tap<4>(x[3], kr)) +
            23 * (fx_tap<4>(x[1], kr) + fx_tap<4>(x[2], kr))) >>
           5;
}
__device__ __forceinline__ long long fx_row_sum(const double x[4], const FxFrac w[4], int kb, int &kr) {
    kr = fx_row_exp(x[0], x[1], x[2], x[3], kb - kFxOrders);
    long long s = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) s += fx_mul(fx_tap<8>(x[a], kr), w[a]);
    return s >> 4;
}

// 1 / sqrt(1 + dh^2). As FP64 instructions the root takes 7 of 64 cycles each;
// here it is in units of 2^-62 from the single precision root w0 and its
// exact error r = 1 - w0^2 - (w0 dh)^2 to second order (the third is below
// 2^-62), about 100 cycles of integer instructions, and rounds once, into the
// result: 0.29 ulp rms without bias, where the FP64 instructions round some
// four times (0.63). Below 2^-30 the root is 1 to rounding; from 2^8 on FP64's
// rsqrt takes it.
__device__ __forceinline__ double fx_invroot(double dh) {
    const unsigned hi = (unsigned)__double2hiint(dh), lo = (unsigned)__double2loint(dh);
    const int x = (int)((hi >> 20) & 0x7FFu) - 1023;  // |dh| in [2^x, 2^(x+1))
    if (x < -30) return 1.0;
    if (x > 7) return rsqrt(fma(dh, dh, 1.0));
    const unsigned mh = (hi & 0x000FFFFFu) | 0x00100000u;
    // |dh| = M 2^(x - 61), M in [2^61, 2^62)
    const unsigned long long M = ((unsigned long long)__funnelshift_l(lo, mh, 9) << 32) |
                                 (unsigned long long)(lo << 9);
    const float f = __int_as_float((int)(((x + 127) << 23) | (__funnelshift_l(lo, mh, 3) & 0x7FFFFF)));
    const float w0f = rsqrtf(fmaf(f, f, 1.0f));
    const unsigned w0 = (unsigned)(w0f * 2147483648.0f);  // 2^-31, at most 2^31
    // t = w0 |dh| in units of 2^-62 (below 2^62: w0 |dh| < 1 by more than r)
    const unsigned long long ph = (M >> 31) * w0, pl = (M & 0x7fffffffull) * w0;
    const unsigned long long t =
        x < 0 ? fx_shr(ph + (pl >> 31), -1 - x) : fx_shl(ph, x + 1) + fx_shr(pl, 30 - x);
    const long long ww = (long long)((unsigned long long)w0 * w0);  // w0^2, 2^-62
    const long long r = (1ll << 62) - ww - fx_mul((long long)t, fx_limbs((long long)t));  // |r| < 2^42
    const long long r1 = r >> 20;
    const long long c = (r >> 1) + ((3 * ((r1 * r1) >> 22)) >> 3);
    // w = w0 (1 + c) with every bit of the product, in units of 2^-62, of
    // 2^-(62 + x) where the root is that small (cut at 2^-52 it made every
    // slope too small, by 0.7 to 1 ulp)
    const int sh = max(x, 0);
    const long long cw = (c >> 20) * (long long)w0 + (((c & 0xFFFFFll) * (long long)w0) >> 20);
    const long long w = ((long long)w0 << (31 + sh)) + (cw >> (11 - sh));
    return fx_to_double(w, -62 - sh);
}
// dh / sqrt(1 + dh^2)
__device__ __forceinline__ double fx_slope(double dh) { return __dmul_rn(dh, fx_invroot(dh)); }
