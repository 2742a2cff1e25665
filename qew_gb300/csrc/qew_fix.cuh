// qew_fix.cuh -- the FP64 gather on the integer pipe: 64-bit fixed point.
//
// GB300 issues one FP64 instruction of a warp every 64 cycles per scheduler
// (measured: DADD, DMUL, DFMA, compares and conversions alike, with one warp
// already saturating it), an integer instruction every 1-2. The 16-tap
// gather's sums are all of one scale -- the field's largest coefficient
// bounds every partial sum -- so they lose nothing in fixed point with the
// unit 2^-57 of that bound: about 2^-4 of an FP64 ulp at the bound, where the
// FP64 sum rounds some twenty times at its terms' own ulps. Measured, with
// the shorter combine of qew_model_kernels.cuh: the gradient of a
// 262144-point arclength line 43.5 -> 14.0 us, of a 100003-point line off the
// field's grid 28.0 -> 11.2 us, a step of the FP64 Langevin run 22.9 -> 16.1 us.
//
// Formats. A tap is an int64 X with c = X 2^(K-57) (|c| < 2^K for the whole
// field, K from a maximum taken when the field is built). A fraction t in
// [0, 1) is T = T1 2^31 + T0 in units of 2^-62, two 31-bit limbs; its product
// with an int64 w, |w| < 2^62, is three 32 x 32 + 64-bit multiply-adds
// (fx_mul, truncated below the unit of w).
#pragma once

#include <cuda_runtime.h>

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

// floor(g) and the fraction of g = a * 2^k for a field of n cells, from the
// bits of a: false for what the reference's fold has to see (negative or
// non-finite a, g >= 2^30, a height whose cell is the last one of a period
// above the first, where the reference's division may round up).
__device__ __forceinline__ bool fx_cell(double a, int k, int n, int &iy, FxFrac &t) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(a);
    const int ef = (int)(b >> 52);  // sign bit and biased exponent
    const int e = ef + k - 1023;
    if (ef == 0 || ef >= 2047 || e > 29) {
        iy = 0;
        t = FxFrac{0, 0};
        return b == 0ull;
    }
    const unsigned long long m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
    const int up = 12 + e;  // fraction bits to the top of 64 (the integer part leaves)
    t = fx_frac(up >= 0 ? fx_shl(m, up) : fx_shr(m, -up));
    iy = e >= 0 ? (int)fx_shr(m, 52 - e) : 0;
    if (iy >= n) {
        const int q = iy / n;
        iy -= q * n;
        return iy + 1 < n;
    }
    return true;
}

// The four stencil rows' sums E (|E| <= 2^58) at fraction t, times 2:
// dV/dt = (E2 - E0)/2 + t (u + t w/2), u = E0 - 2 E1 + E2,
// w = (E3 - E0) - 3 (E2 - E1): the derivative of filtered_noise.h:33-62's
// cubic, summed in the unit of E.
__device__ __forceinline__ long long fx_cubic_dt2(const long long E[4], FxFrac t) {
    const long long u = E[0] + E[2] - 2 * E[1];
    const long long w = (E[3] - E[0]) - 3 * (E[2] - E[1]);
    return (E[2] - E[0]) + fx_mul(2 * u + fx_mul(w, t), t);
}
// The value, times 6 (|E| <= 2^57): (E0 + 4 E1 + E2) + t (3 (E2 - E0) + t (3 u + t w)).
__device__ __forceinline__ long long fx_cubic_6v(const long long E[4], FxFrac t) {
    const long long s = E[0] + E[2];
    const long long u = s - 2 * E[1];
    const long long w = (E[3] - E[0]) - 3 * (E[2] - E[1]);
    return s + 4 * E[1] + fx_mul(3 * (E[2] - E[0]) + fx_mul(3 * u + fx_mul(w, t), t), t);
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
