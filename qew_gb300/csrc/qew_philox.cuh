// qew_philox.cuh -- Philox4x32-10 counter-based generator (J. Salmon,
// M. Moraes, R. Dror, D. Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC'11) and a Box-Muller (1958) normal pair. Increment i of step s comes from
// the block of counter (i/2, 0, s_lo, s_hi) under key (seed_lo, seed_hi):
// two 53-bit uniforms u1 in (0,1], u2 in [0,1), r = sqrt(-2 ln u1),
// xi_{2j} = r cos(2 pi u2), xi_{2j+1} = r sin(2 pi u2).
#pragma once

#include <stdint.h>

#include "qew_fix.cuh"
#include "qew_normal_tables.cuh"

__host__ __device__ __forceinline__ void philox_round(uint32_t c[4], uint32_t k0, uint32_t k1) {
#ifdef __CUDA_ARCH__
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]);
    const uint32_t lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]);
    const uint32_t lo1 = 0xCD9E8D57u * c[2];
#else
    const uint64_t p0 = (uint64_t)0xD2511F53u * c[0];
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * c[2];
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
#endif
    const uint32_t n0 = hi1 ^ c[1] ^ k0;
    const uint32_t n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
}

__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint64_t seed) {
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) {
            k0 += 0x9E3779B9u;
            k1 += 0xBB67AE85u;
        }
        philox_round(c, k0, k1);
    }
}

// Box-Muller in 64-bit fixed point (qew_fix.cuh). As FP64 calls the pair's
// log, square root, sine and cosine take about 80 FP64 instructions, 64
// cycles of a scheduler's FP64 unit each; the integer form below takes about
// 370 instructions of 1-2 cycles and rounds once, into the result (absolute
// error about 2^-57: rms 5.0e-17 against the FP64 form's 2.4e-16 on 2e7 pairs).
// 2^21 pairs: 321 -> 51 us; a step of the FP64 Langevin run at L = 65536:
// 16.3 -> 12.0 us.
// Every step, with u1 = m 2^-53 (1 <= m <= 2^53) and u2 = b 2^-53:
//   -ln u1: n = m shifted to its leading bit, f = n / 2^63 in [1, 2); the
//     interval's multiplier makes r = f ic / 512 - 1 exactly, |r| <= 1/128,
//     and ln(1 + r) is its series to r^8 in units of 2^-68. The intervals at
//     f = 1 and f = 2 have the multipliers 1 and 1/2, so that near u1 = 1 the
//     logarithm keeps the relative accuracy of r;
//   sqrt(2 y): y normalised to [1/2, 2) with an even exponent, a single
//     precision reciprocal root as the first guess and the binomial series of
//     its error to second order (the third is below 2^-63);
//   cos, sin of 2 pi u2: table at the nearest 1/256 turn, the remainder's
//     series to its 6th power, and the addition theorem.
#ifdef __CUDACC__
__device__ const FxTurn g_fx_turns[256] = {QEW_FX_TURNS};
__device__ const FxLog g_fx_logs[128] = {QEW_FX_LOGS};
#endif

// (r cos, r sin) as integers in units of 2^-62 * 2^k.
__host__ __device__ __forceinline__ void fx_normal_pair(uint64_t m, uint64_t b,
                                                        const FxLog *__restrict__ logs,
                                                        const FxTurn *__restrict__ turns,
                                                        long long &z0, long long &z1, int &k) {
    // y = -ln u1 in units of 2^-57, or of 2^-68 when it is the series alone
    const int lz = fx_clz(m);
    const uint64_t n = fx_shl(m, lz);
    const FxLog lg = logs[(unsigned)(n >> 56) & 127u];
    const long long R = ((long long)((n >> 11) * (uint64_t)lg.ic) - (1ll << 61)) << 7;  // r, 2^-68
    const FxFrac r = fx_limbs(R >> 6);
    // ln(1 + r) = r - r (r q), q = 1/2 - r/3 + r^2/4 - ... + r^6/8 in units of 2^-61
    long long q = 288230376151711744ll;                  // 1/8
    q = 329406144173384850ll - fx_mul(q, r);             // 1/7
    q = 384307168202282325ll - fx_mul(q, r);             // 1/6
    q = 461168601842738790ll - fx_mul(q, r);             // 1/5
    q = 576460752303423488ll - fx_mul(q, r);             // 1/4
    q = 768614336404564651ll - fx_mul(q, r);             // 1/3
    q = 1152921504606846976ll - fx_mul(q, r);            // 1/2
    const long long big = (long long)(lz - 10) * 99893036290645747ll - lg.ln;
    const bool small = big == 0;
    // within 2^-20 of 1 (a pair in a million) the series takes r's own scale
    const uint64_t ra = (uint64_t)(R < 0 ? -R : R);
    const int up = (small && ra < (1ull << 48)) ? fx_clz(ra) - 4 : 0;
    const long long Ru = (long long)fx_shl((uint64_t)R, up);
    const long long L = Ru - fx_mul(Ru, fx_limbs(2 * fx_mul(q, r)));
    const uint64_t y = (uint64_t)(small ? -L : big - (L >> 11));
    // 2 y = N 2^e with e even, N in [2^61, 2^63)
    int s = fx_clz(y) - 1;
    int e = 1 - (small ? 68 + up : 57) - s;
    if (e & 1) {
        --s;
        ++e;
    }
    const uint64_t N = fx_shl(y, s);
    const float v = (float)(uint32_t)(N >> 32) * 9.31322574615478515625e-10f;  // 2^-30
#ifdef __CUDA_ARCH__
    const float g = rsqrtf(v);
#else
    const float g = 1.0f / sqrtf(v);
#endif
    const uint32_t Y = (uint32_t)(g * 1073741824.0f);                          // 1/sqrt, 2^-30
    auto mul31 = [](uint64_t a, uint32_t c) {                                  // a c >> 31
        return (a >> 31) * (uint64_t)c + (((a & 0x7fffffffull) * (uint64_t)c) >> 31);
    };
    const uint64_t S0 = mul31(N, Y);                                           // sqrt(N 2^-62), 2^-61
    const long long D = (1ll << 60) - (long long)mul31(S0, Y);                 // 1 - v g^2, 2^-60
    const long long D2 = ((D >> 9) * (D >> 9)) >> 42;                          // its square
    const long long C = (D >> 1) + ((3 * D2) >> 3);
    const long long S = (long long)S0 + fx_mul((long long)S0, fx_limbs(4 * C));
    // angle
    const uint64_t B = b << 11;                                                // turns, 2^-64
    const uint64_t j = (B + (1ull << 55)) >> 56;
    const long long dl = (long long)(B - (j << 56));
    const FxTurn tn = turns[(unsigned)j & 255u];
    const long long F = fx_mul(dl * 64, fx_limbs(3622009729038561421ll));      // 2 pi dl, 2^-67
    const long long P2 = fx_mul(F, fx_limbs(F >> 5));                          // its square, 2^-67
    const FxFrac w = fx_limbs(P2 >> 5);
    const FxFrac ci = fx_limbs(2305843009213693952ll -
                               fx_mul(192153584101141163ll - fx_mul(6405119470038039ll, w), w));
    const FxFrac si = fx_limbs(768614336404564651ll - fx_mul(38430716820228233ll, w));
    const long long cm = -fx_mul(P2, ci);                                      // cos - 1, 2^-67
    const long long sn = F - fx_mul(F, fx_limbs(fx_mul(P2, si) >> 5));         // sin, 2^-67
    const FxFrac tc = fx_limbs(tn.c), ts = fx_limbs(tn.s);
    const long long c = tn.c + ((fx_mul(cm, tc) - fx_mul(sn, ts)) >> 5);
    const long long d = tn.s + ((fx_mul(cm, ts) + fx_mul(sn, tc)) >> 5);
    z0 = fx_mul(S, fx_limbs(c));                                               // 2^-61
    z1 = fx_mul(S, fx_limbs(d));
    k = e / 2 - 30;  // sqrt(2 y) = S 2^-61 2^(e/2 + 31)
}

// The two N(0,1) increments of sites 2j and 2j+1 at step `step`.
__device__ __forceinline__ void philox_normal_pair(uint64_t seed, uint64_t step, uint32_t j,
                                                   double &z0, double &z1) {
    uint32_t c[4] = {j, 0u, (uint32_t)step, (uint32_t)(step >> 32)};
    philox4x32_10(c, seed);
    const uint64_t a = ((((uint64_t)c[0]) << 32) | c[1]) >> 11;
    const uint64_t b = ((((uint64_t)c[2]) << 32) | c[3]) >> 11;
    long long i0, i1;
    int k;
    fx_normal_pair(a + 1, b, g_fx_logs, g_fx_turns, i0, i1, k);
    z0 = fx_to_double(i0, k);
    z1 = fx_to_double(i1, k);
}
