// qew_field.cu -- pinning-field handles: device-side periodic cubic B-spline
// prefilter, x-fastest FP64/FP32 coefficient storage, and point sampling.
//
// The reference builds coefficients with an FFT division
// (filtered_noise.cpp:92-136): c = IFFT2(FFT2(s) / (Kx (x) Ky)) with
// K[m] = 2/3 + cos(2 pi m/N)/3, i.e. the exact solve of the circulant system
// (1/6, 2/3, 1/6) * c = s along each axis. The same exact solve is done here
// by the separable recursive filter of the cubic B-spline (pole
// z1 = sqrt(3) - 2; M. Unser, IEEE Trans. Signal Process. 41 (1993)) with the
// periodic initial conditions written in closed form, so the result equals
// the FFT division up to rounding, for any nx, ny, in O(nx*ny) work.
#include "qew_internal.cuh"
#include "qew_philox.cuh"
#include "qew_poly.cuh"

#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <random>
#include <vector>

namespace {

// Periodic cubic B-spline prefilter along one axis, in one out-of-place pass
// over chunks of kChunk samples so that every line is split over many
// threads. The filter's causal and anticausal recursions run side by side on
// the samples (its partial-fraction form): with y[k] = s[k] + z y[k-1] and
// w[k] = s[k] + z w[k+1],
//   c[k] = g (y[k] + z w[k+1]),  g = -6 z / (1 - z^2) = sqrt(3),
// which equals the cascade c = -6 z anticausal(causal(s)). A chunk starts
// each recursion kWarm samples away from zero, reading the periodic
// neighbours: the neglected tail is z^kWarm = 2.5e-37 of a sample that far away,
// so every output equals the exact periodic solve up to its own rounding, for
// any N (the warm-up wraps for short N), beside samples 1e20 times larger too. Lines are m = 0..M-1 at stride `lst`; samples
// at stride `st`; consecutive threads take consecutive lines so each step's
// accesses coalesce when lst == 1. FP64-bound: 4 instructions a sample (5
// with the gain, which the last axis applies for both, times the field's
// scale where one is given) and as much again for the warm-ups. 4096 x 1024, both
// axes: 284 -> 127 us (the cascade's four passes before; 109 with warm-ups of
// 32, whose tail of 5e-19 is no longer below rounding where a weak region lies
// beside strong samples).
constexpr double kPole = -0.26794919243112270;  // sqrt(3) - 2
constexpr int kChunk = 64;
constexpr int kWarm = 64;
constexpr int kPreBS = 128;

__device__ __forceinline__ int pmod(long k, int N) {
    long r = k % N;
    return (int)(r < 0 ? r + N : r);
}

// What the last axis's pass does besides: the gain of both axes (times
// *scale), the FP32 copy (out32, or null) and the largest |c|'s bits
// (max_bits, or null).
struct PrefilterEnd {
    double gain;
    const double *scale;
    float *out32;
    unsigned long long *max_bits;
};

template <bool kEnd>
__global__ void __launch_bounds__(kPreBS)
k_prefilter(const double *__restrict__ in, double *out, int N, long st, int M, long lst,
            PrefilterEnd end) {
    const long tid = blockIdx.x * (long)kPreBS + threadIdx.x;
    const int nchunks = (N + kChunk - 1) / kChunk;
    unsigned long long mx = 0;
    if (tid < (long)M * nchunks) {
        const int m = (int)(tid % M), c = (int)(tid / M);
        const double *a = in + (long)m * lst;
        double *b = out + (long)m * lst;
        const int k0 = c * kChunk, k1 = min(k0 + kChunk, N);
        double y = 0.0;
        int k = pmod((long)k0 - kWarm, N);
#pragma unroll 8
        for (int q = 0; q < kWarm; ++q) {
            y = fma(kPole, y, a[(long)k * st]);
            k = (k + 1 == N) ? 0 : k + 1;
        }
#pragma unroll 8
        for (k = k0; k < k1; ++k) {
            y = fma(kPole, y, a[(long)k * st]);
            b[(long)k * st] = y;
        }
        const double gain = kEnd ? (end.scale ? end.gain * *end.scale : end.gain) : 1.0;
        double w = 0.0;
        k = pmod((long)k1 - 1 + kWarm, N);
#pragma unroll 8
        for (int q = 0; q < kWarm; ++q) {
            w = fma(kPole, w, a[(long)k * st]);
            k = (k == 0) ? N - 1 : k - 1;
        }
#pragma unroll 8
        for (k = k1 - 1; k >= k0; --k) {
            double v = fma(kPole, w, b[(long)k * st]);
            w = fma(kPole, w, a[(long)k * st]);
            if (kEnd) {
                v *= gain;
                const unsigned long long vb =
                    (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
                mx = vb > mx ? vb : mx;
                if (end.out32) end.out32[(long)m * lst + (long)k * st] = (float)v;
            }
            b[(long)k * st] = v;
        }
    }
    if (kEnd && end.max_bits) {  // bit patterns of |c| are ordered like the numbers
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long q = __shfl_xor_sync(0xffffffffu, mx, o);
            mx = q > mx ? q : mx;
        }
        if ((threadIdx.x & 31) == 0) atomicMax(end.max_bits, mx);
    }
}

qew_status prefilter_axis(qew_ctx *ctx, const double *in, double *out, int N, long st, int M,
                          long lst, const PrefilterEnd *end) {
    const long threads = (long)M * ((N + kChunk - 1) / kChunk);
    const unsigned blocks = (unsigned)((threads + kPreBS - 1) / kPreBS);
    if (end)
        k_prefilter<true><<<blocks, kPreBS, 0, ctx->stream>>>(in, out, N, st, M, lst, *end);
    else
        k_prefilter<false><<<blocks, kPreBS, 0, ctx->stream>>>(in, out, N, st, M, lst,
                                                               PrefilterEnd{});
    return qew_launch_check(ctx, "prefilter");
}

// [nx][ny] -> [ny][nx] through a 32x33 shared tile.
__global__ void k_transpose(const double *__restrict__ in, double *__restrict__ out,
                            int nx, int ny) {
    __shared__ double tile[32][33];
    const int j0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int i = i0 + r, j = j0 + threadIdx.x;
        if (i < nx && j < ny) tile[r][threadIdx.x] = in[(size_t)i * ny + j];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int j = j0 + r, i = i0 + threadIdx.x;
        if (i < nx && j < ny) out[(size_t)j * nx + i] = tile[threadIdx.x][r];
    }
}

// E[j][e] = sum_a w_a(1/2) c[j][(e - 1 + a) mod nx], FP64 sum rounded once to
// FP32: the x part of the cubic B-spline sum (filtered_noise.h:33-44 at t = 1/2,
// where the weights are 1/48, 23/48, 23/48, 1/48) at the midpoint of every
// column pair; c is [ny][nx], x fastest.
__global__ void k_edge_fp32(const double *__restrict__ c, float *__restrict__ out, int nx, int ny) {
    const double w0 = 1.0 / 48.0, w1 = 23.0 / 48.0;
    for (int j = blockIdx.y; j < ny; j += gridDim.y) {
        const double *row = c + (size_t)j * (size_t)nx;
        float *o = out + (size_t)j * (size_t)nx;
        for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nx; e += gridDim.x * blockDim.x) {
            const int em = (e == 0) ? nx - 1 : e - 1;
            const int ep = (e + 1 == nx) ? 0 : e + 1;
            const int ep2 = (ep + 1 == nx) ? 0 : ep + 1;
            o[e] = (float)(w0 * row[em] + w1 * row[e] + w1 * row[ep] + w0 * row[ep2]);
        }
    }
}

template <class Noise>
__global__ void k_sample(Noise nz, const double *__restrict__ x, const double *__restrict__ y,
                         int m, double *v, double *dvdx, double *dvdy) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m) return;
    double a, b, c;
    nz.sample(x[k], y[k], a, b, c);
    if (v) v[k] = a;
    if (dvdx) dvdx[k] = b;
    if (dvdy) dvdy[k] = c;
}

// ---- synthetic field generation on the device ----
// White noise w[i][j] ~ N(0,1) from the Philox stream (seed, counter (pair of
// j, row i)), then a periodic Gaussian filter of std xi cells along each axis
// (the real-space form of exp(-(2 pi xi f)^2 / 2) in Fourier space; taps to
// |k| <= ceil(5 xi), normalised so the sum of squared taps is 1), in the
// reference's host layout [nx][ny].
// The filter runs in 64-bit fixed point (qew_fix.cuh): the noise and the filtered
// sums are bounded (ConvUnits), samples are rounded at 2^-55 and 2^-53 and the taps
// at 2^-59 of unity, so the field's error stays below 4e-16 of its deviation at
// any xi, where FP64 sums of 41000 terms (xi = 4096) come to 8e-15; a tap pair costs four 32 x 32 + 64-bit multiply-adds (about 5 cycles each) where
// FP64 takes two 64-cycle instructions: 306 -> 150 us an axis of a 4096 x 1024
// field at xi = 4 (41 taps), 115 with four outputs a thread. A sample is X = X1 2^30 + X0 in units 2^-F,
// |X| < 2^59; a tap T = T1 2^30 + T0 <= 2^58 in units 2^-q.
constexpr double kNoiseMax = 8.58;  // sqrt(2 ln 2^53) = 8.572

__global__ void k_white_noise(long long *__restrict__ w, int nx, int ny, uint64_t seed, int F) {
    const long tid = blockIdx.x * (long)blockDim.x + threadIdx.x;
    const int pairs = (ny + 1) / 2;
    if (tid >= (long)nx * pairs) return;
    const int i = (int)(tid % nx), jp = (int)(tid / nx);
    uint32_t c[4] = {(uint32_t)jp, 0u, (uint32_t)i, 0u};
    philox4x32_10(c, seed);
    const uint64_t a = ((((uint64_t)c[0]) << 32) | c[1]) >> 11;
    const uint64_t b = ((((uint64_t)c[2]) << 32) | c[3]) >> 11;
    long long z0, z1;
    int k;
    fx_normal_pair(a + 1, b, g_fx_logs, g_fx_turns, z0, z1, k);  // z 2^k, k <= -F
    const int sh = min(-k - F, 63);
    const long long half = sh > 0 ? 1ll << (sh - 1) : 0;
    w[(size_t)(2 * jp) * nx + i] = (z0 + half) >> sh;  // [ny][nx]
    if (2 * jp + 1 < ny) w[(size_t)(2 * jp + 1) * nx + i] = (z1 + half) >> sh;
}

// out[p] = sum_k tap[|k|] in[p + k] along the slow axis of in[len][width] (both
// periodic, symmetric taps, radius R), lanes along the fast one. kLast: FP64 out
// in the same layout, times 2^exp; else fixed point, shifted right by exp, as
// out[width][len], so that the other axis is the slow one next.
// The partial products of weight 2^60, 2^30 and 1 have sums of their own, the
// lower two folded, rounded to 2^44, every four pairs before they can overflow
// (2^61 a pair); the whole is in units of 2^(60 - up).
// A thread takes 4 consecutive outputs: a step in k then needs two new samples
// for the four (they slide through registers, split into their 30-bit halves
// once) where an output alone loads and splits both ends of every pair; what
// is left is 4 wide multiply-adds a pair.
template <bool kLast, int kOut>
__global__ void __launch_bounds__(256)
k_gauss_conv(const long long *__restrict__ in, void *__restrict__ out, int len, int width,
             const int2 *__restrict__ tap, int R, int exp, int up, int lsh) {
    // a block is 2^lsh lanes wide and 256 / 2^lsh threads along the slow axis,
    // whose windows overlap in L1
    const unsigned tiles = ((unsigned)width + (1u << lsh) - 1u) >> lsh;
    const unsigned row = blockIdx.x / tiles;
    const int l = (int)((blockIdx.x - row * tiles) << lsh) + (int)(threadIdx.x & ((1u << lsh) - 1u));
    const long long pl = (((long long)row << (8 - lsh)) + (threadIdx.x >> lsh)) * kOut;
    if (l >= width || pl >= len) return;
    const int p0 = (int)pl;
    constexpr int kLow = (1 << 30) - 1;
    constexpr long long kHalfM = 1ll << 13;  // of the folds' rounding
    constexpr unsigned long long kHalfL = 1ull << 43;
    int a1[kOut], a0[kOut], b1[kOut], b0[kOut];  // samples at p0 + u - k and p0 + u + k
    auto get = [&](int p, int &x1, int &x0) {
        const long long x = __ldg(in + (size_t)p * (size_t)width + l);
        x1 = (int)(x >> 30);
        x0 = (int)x & kLow;
    };
    long long P[kOut], M[kOut], A[kOut];
    unsigned long long L[kOut];
    auto add = [&](int u, int x1, int x0, int2 t) {
        P[u] += (long long)x1 * t.x;
        M[u] += (long long)x1 * t.y;
        M[u] += (long long)x0 * t.x;  // x0 < 2^31
        L[u] += (unsigned long long)(unsigned)x0 * (unsigned)t.y;
    };
    auto fold = [&]() {
#pragma unroll
        for (int u = 0; u < kOut; ++u) {
            A[u] += (M[u] >> 14) + (long long)(L[u] >> 44);
            M[u] = kHalfM;
            L[u] = kHalfL;
        }
    };
    {
        const int2 t = __ldg(tap);
        int p = p0;
#pragma unroll
        for (int u = 0; u < kOut; ++u) {
            P[u] = A[u] = 0;
            M[u] = kHalfM;
            L[u] = kHalfL;
            get(p, a1[u], a0[u]);
            b1[u] = a1[u];
            b0[u] = a0[u];
            add(u, a1[u], a0[u], t);
            p = p + 1 == len ? 0 : p + 1;
        }
    }
    int pa = p0, pb = (int)((pl + kOut - 1) % len);
    for (int k0 = 1; k0 <= R; k0 += 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (k0 + q > R) break;
            pa = pa == 0 ? len - 1 : pa - 1;
            pb = pb + 1 == len ? 0 : pb + 1;
#pragma unroll
            for (int u = kOut - 1; u > 0; --u) {
                a1[u] = a1[u - 1];
                a0[u] = a0[u - 1];
            }
#pragma unroll
            for (int u = 0; u < kOut - 1; ++u) {
                b1[u] = b1[u + 1];
                b0[u] = b0[u + 1];
            }
            get(pa, a1[0], a0[0]);
            get(pb, b1[kOut - 1], b0[kOut - 1]);
            const int2 t = __ldg(tap + k0 + q);
#pragma unroll
            for (int u = 0; u < kOut; ++u) add(u, a1[u] + b1[u], a0[u] + b0[u], t);
        }
        fold();
    }
    fold();
    long long v[kOut];
#pragma unroll
    for (int u = 0; u < kOut; ++u) v[u] = (P[u] << up) + (A[u] >> (16 - up));
    if (!kLast) {
        const long long half = (1ll << exp) >> 1;
#pragma unroll
        for (int u = 0; u < kOut; ++u) v[u] += half;
    }
    const int cnt = min(kOut, len - p0);
    if (kLast) {
        double *o = (double *)out + (size_t)p0 * (size_t)width + l;
#pragma unroll
        for (int u = 0; u < kOut; ++u)
            if (u < cnt) o[(size_t)u * (size_t)width] = fx_to_double(v[u], exp);
    } else {
        long long *o = (long long *)out + (size_t)l * (size_t)len + p0;
        if (kOut == 4 && cnt == kOut && (len & 1) == 0) {  // 16-byte aligned: p0 is a multiple of 4
            ((longlong2 *)o)[0] = make_longlong2(v[0] >> exp, v[1 % kOut] >> exp);
            ((longlong2 *)o)[1] = make_longlong2(v[2 % kOut] >> exp, v[3 % kOut] >> exp);
        } else {
#pragma unroll
            for (int u = 0; u < kOut; ++u)
                if (u < cnt) o[u] = v[u] >> exp;
        }
    }
}

// Population mean and std of n values in two passes (the second about the
// mean): per-block partial sums, the last block to arrive adds them in block
// order. stat[0] = mean after the first pass; stat[1] = amplitude / std after
// the second. One CTA read the field twice at one SM's bandwidth: 3.45 ms of
// a 4096 x 1024 field's 4.8 ms, these passes take 17 and 24 us.
constexpr int kMomBS = 256;
template <bool kCentred>
__global__ void __launch_bounds__(kMomBS)
k_moment(const double *__restrict__ a, size_t n, double amplitude, double *partials,
         unsigned int *counter, double *stat) {
    __shared__ double s_w[kMomBS / 32];
    __shared__ bool s_last;
    const double mean = kCentred ? stat[0] : 0.0;
    const size_t step = (size_t)gridDim.x * kMomBS;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    size_t k = blockIdx.x * (size_t)kMomBS + threadIdx.x;
    auto term = [&](double v, double s) { return kCentred ? fma(v - mean, v - mean, s) : s + v; };
    for (; k + 3 * step < n; k += 4 * step) {
        const double v0 = a[k], v1 = a[k + step], v2 = a[k + 2 * step], v3 = a[k + 3 * step];
        s0 = term(v0, s0);
        s1 = term(v1, s1);
        s2 = term(v2, s2);
        s3 = term(v3, s3);
    }
    for (; k < n; k += step) s0 = term(a[k], s0);
    const double bs = block_sum<kMomBS>((s0 + s1) + (s2 + s3), s_w);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = bs;
        __threadfence();
        s_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kMomBS) v += __ldcg(partials + b);
    const double tot = block_sum<kMomBS>(v, s_w);
    if (threadIdx.x == 0) {
        if (kCentred)
            stat[1] = amplitude / sqrt(tot / (double)n);
        else
            stat[0] = tot / (double)n;
        *counter = 0u;
    }
}

// stat (2 doubles on the device) of n values; scratch: the context's reduction arena.
qew_status field_moments(qew_ctx *ctx, const double *a, size_t n, double amplitude, double *stat) {
    const int blocks = (int)std::min<size_t>(
        std::min<size_t>((n + 4 * kMomBS - 1) / (4 * kMomBS), (size_t)ctx->num_sms * 6),
        QEW_RED_MAX_BLOCKS);
    k_moment<false><<<blocks, kMomBS, 0, ctx->stream>>>(a, n, amplitude, ctx->red_partials,
                                                        ctx->red_counter, stat);
    k_moment<true><<<blocks, kMomBS, 0, ctx->stream>>>(a, n, amplitude, ctx->red_partials,
                                                       ctx->red_counter, stat);
    return qew_launch_check(ctx, "field_moments", 2);
}

// Real part of the inverse transform times 1/(nx ny) (the backward
// normalisation of kokkos-fft and numpy's ifft2).
__global__ void k_real_part(const cufftDoubleComplex *__restrict__ b, size_t n, double inv_n,
                            double *__restrict__ out) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n;
         k += (size_t)gridDim.x * blockDim.x)
        out[k] = b[k].x * inv_n;
}

// numpy fftfreq(n)[k] in cycles per sample (filtered_noise.cpp:18-21).
double fft_freq(int k, int n) {
    const int ks = (k < (n + 1) / 2) ? k : k - n;
    return (double)ks / (double)n;
}

// Taps 0..R of the normalised symmetric filter; its gain (the taps' sum), and its
// norm on len periodic samples (1, more where the filter wraps onto itself).
std::vector<double> gauss_taps(double xi, int len, int &R, double &gain, double &norm) {
    R = (xi > 0) ? (int)ceil(5.0 * xi) : 0;
    std::vector<double> t(R + 1);
    double s2 = 0.0;
    for (int k = -R; k <= R; ++k) {
        const double v = (xi * xi > 0) ? exp(-0.5 * (double)k * k / (xi * xi)) : (k == 0 ? 1.0 : 0.0);
        if (k >= 0) t[k] = v;
        s2 += v * v;
    }
    gain = 0.0;
    for (int k = 0; k <= R; ++k) {
        t[k] /= sqrt(s2);
        gain += (k ? 2.0 : 1.0) * t[k];
    }
    const int period = std::min(len, 2 * R + 1);
    std::vector<double> folded(period, 0.0);
    for (int k = 0; k <= 2 * R; ++k) folded[k % period] += t[k < R ? R - k : k - R];
    norm = 0.0;
    for (double v : folded) norm += v * v;
    norm = sqrt(norm);
    return t;
}

// One filter pass's fixed point. Its sums are bounded by `bound`: |z| < 8.58 for
// the noise (53-bit uniforms) times the gain, or 40 standard deviations (a
// normal number exceeds that once in 10^350), whichever is less, as every sum of
// a part of the taps is. With b = ceil(log2 bound), samples in units 2^-F and
// taps in 2^-q, q <= 58, the sum of the upper products stays below 2^62, and the
// whole in units of 2^U, U = F + q + b - 62, as well.
struct ConvUnits {
    int q, b, up;  // up = 60 - U
    std::vector<int2> tap;
    ConvUnits(const std::vector<double> &t, int F, double bound) : b((int)ceil(log2(bound))) {
        q = std::min(58, 122 - F - b);
        up = 60 - (F + q + b - 62);
        for (double v : t) {
            const long long T = llrint(ldexp(v, q));
            tap.push_back(make_int2((int)(T >> 30), (int)(T & ((1 << 30) - 1))));
        }
    }
};

// scale (a device number, or null) multiplies the field.
qew_status field_build(qew_ctx *ctx, const double *src, bool src_on_device, int nx,
                       int ny, double Lx, double Ly, int store, qew_field **out,
                       const double *scale = nullptr) {
    if (!ctx || !out || !src || nx <= 0 || ny <= 0 || !(Lx > 0) || !(Ly > 0) ||
        (store & (QEW_STORE_FP64 | QEW_STORE_FP32)) == 0)
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create: bad arguments");
    if ((store & QEW_STORE_FP32_EDGE) && !(store & QEW_STORE_FP32))
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create: QEW_STORE_FP32_EDGE needs QEW_STORE_FP32");
    if ((store & QEW_STORE_FP64_POLY) && !(store & QEW_STORE_FP64))
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create: QEW_STORE_FP64_POLY needs QEW_STORE_FP64");
    // transposes tile 32 columns per grid row: keep both extents within the grid limit
    if (nx > 65535 * 32 || ny > 65535 * 32)
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create: nx and ny must be <= %d", 65535 * 32);
    *out = nullptr;
    QEW_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t N = (size_t)nx * ny;
    qew_field *f = new (std::nothrow) qew_field();
    if (!f) return QEW_ERR_NOMEM;
    f->kind = QEW_FIELD_BSPLINE;
    f->device = ctx->device;
    f->nx = nx;
    f->ny = ny;
    f->Lx = Lx;
    f->Ly = Ly;
    f->dx = Lx / nx;  // filtered_noise.cpp:87
    f->dy = Ly / ny;
    double *tmp = nullptr, *c64 = nullptr;
    unsigned long long *d_max = nullptr;
    f->stream = ctx->stream;
    auto cleanup = [&](qew_status s) {
        qew_free_async(tmp, ctx->stream);
        qew_free_async(c64, ctx->stream);
        qew_free_async(d_max, ctx->stream);
        qew_free_async(f->coef32, ctx->stream);
        qew_free_async(f->edge32, ctx->stream);
        qew_free_async(f->poly, ctx->stream);
        cudaStreamSynchronize(ctx->stream);
        delete f;
        return s;
    };
    if (qew_alloc_async(ctx, (void **)&tmp, N * sizeof(double)) != QEW_OK ||
        qew_alloc_async(ctx, (void **)&c64, N * sizeof(double)) != QEW_OK)
        return cleanup(QEW_ERR_NOMEM);
    cudaError_t e = cudaSuccess;
    if (!src_on_device) {
        e = cudaMemcpyAsync(c64, src, N * sizeof(double), cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess)
            return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "field upload: %s", cudaGetErrorString(e)));
        src = c64;
    }
    if (qew_alloc_async(ctx, (void **)&d_max, sizeof(*d_max)) != QEW_OK)
        return cleanup(QEW_ERR_NOMEM);
    e = cudaMemsetAsync(d_max, 0, sizeof(*d_max), ctx->stream);
    if (e != cudaSuccess) return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "%s", cudaGetErrorString(e)));
    if (store & QEW_STORE_FP32)
        if (qew_alloc_async(ctx, (void **)&f->coef32, N * sizeof(float)) != QEW_OK)
            return cleanup(QEW_ERR_NOMEM);
    // x pass in the host layout (lines j, stride ny), transpose, y pass in
    // the x-fastest layout (lines i, stride nx), each out of place; the y pass
    // applies the gain, writes the FP32 copy and takes the largest coefficient
    qew_status st = prefilter_axis(ctx, src, tmp, nx, ny, ny, 1, nullptr);
    if (st != QEW_OK) return cleanup(st);
    k_transpose<<<dim3((ny + 31) / 32, (nx + 31) / 32), dim3(32, 8), 0, ctx->stream>>>(tmp, c64, nx, ny);
    st = qew_launch_check(ctx, "transpose");
    if (st != QEW_OK) return cleanup(st);
    const PrefilterEnd end{36.0 * kPole * kPole / ((1.0 - kPole * kPole) * (1.0 - kPole * kPole)),
                           scale, f->coef32, d_max};
    st = prefilter_axis(ctx, c64, tmp, ny, nx, nx, 1, &end);
    if (st != QEW_OK) return cleanup(st);
    std::swap(tmp, c64);
    if (store & QEW_STORE_FP32_EDGE) {
        if (qew_alloc_async(ctx, (void **)&f->edge32, N * sizeof(float)) != QEW_OK)
            return cleanup(QEW_ERR_NOMEM);
        const dim3 eg((unsigned)std::min((nx + 255) / 256, 64), (unsigned)std::min(ny, 65535));
        k_edge_fp32<<<eg, 256, 0, ctx->stream>>>(c64, f->edge32, nx, ny);
        st = qew_launch_check(ctx, "edge_fp32");
        if (st != QEW_OK) return cleanup(st);
    }
    if (store & QEW_STORE_FP64_POLY) {
        if (qew_alloc_async(ctx, (void **)&f->poly, 4 * N * sizeof(long long)) != QEW_OK)
            return cleanup(QEW_ERR_NOMEM);
        st = qew_poly_store_build(ctx, c64, nx, ny, d_max, f->poly);
        if (st != QEW_OK) return cleanup(st);
    }
    // the bound of the fixed-point gather (qew_fix.cuh)
    unsigned long long max_bits = 0;
    e = cudaMemcpyAsync(&max_bits, d_max, sizeof(max_bits), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "field build: %s", cudaGetErrorString(e)));
    qew_free_async(d_max, ctx->stream);
    d_max = nullptr;
    f->fixb = qew_fix_bound(max_bits);  // < 0: no fixed point and no store
    if (f->fixb < 0 && f->poly) {
        qew_free_async(f->poly, ctx->stream);
        f->poly = nullptr;
    }
    qew_free_async(tmp, ctx->stream);
    tmp = nullptr;
    if (store & QEW_STORE_FP64) {
        f->coef64 = c64;
    } else {
        qew_free_async(c64, ctx->stream);
    }
    c64 = nullptr;
    *out = f;
    return QEW_OK;
}

}  // namespace

extern "C" {

qew_status qew_field_create_from_host(qew_ctx *ctx, const double *h_field, int nx, int ny,
                                      double Lx, double Ly, int store_flags, qew_field **out) {
    QEW_RANGE();
    return field_build(ctx, h_field, false, nx, ny, Lx, Ly, store_flags, out);
}

qew_status qew_field_create_from_device(qew_ctx *ctx, const double *d_field, int nx, int ny,
                                        double Lx, double Ly, int store_flags, qew_field **out) {
    QEW_RANGE();
    return field_build(ctx, d_field, true, nx, ny, Lx, Ly, store_flags, out);
}

qew_status qew_field_create_generated(qew_ctx *ctx, int nx, int ny, double Lx, double Ly,
                                     double amplitude, double xi_x_cells, double xi_y_cells,
                                     uint64_t seed, int store_flags, qew_field **out) {
    QEW_RANGE();
    if (!ctx || !out || nx <= 0 || ny <= 0 || !(xi_x_cells >= 0) || !(xi_y_cells >= 0) ||
        xi_x_cells > 4096 || xi_y_cells > 4096 || !(amplitude > 0))
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create_generated: bad arguments");
    QEW_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t N = (size_t)nx * ny;
    int Rx, Ry;
    double gx, gy, sx, sy;
    const std::vector<double> wx = gauss_taps(xi_x_cells, nx, Rx, gx, sx);
    const std::vector<double> wy = gauss_taps(xi_y_cells, ny, Ry, gy, sy);
    // samples in [-2^59, 2^59): 2^-F1 for the noise, 2^-F2 after the y filter
    const double by = std::min(kNoiseMax * gy, 40.0 * sy), bx = std::min(by * gx, 40.0 * sx * sy);
    const int F1 = 59 - (int)ceil(log2(kNoiseMax));
    const ConvUnits uy(wy, F1, by);
    const int F2 = 59 - uy.b;
    const ConvUnits ux(wx, F2, bx);
    const std::vector<int2> &tx = ux.tap, &ty = uy.tap;
    long long *w = nullptr, *t = nullptr;
    double *stat = nullptr;
    auto cleanup = [&](qew_status s) {
        qew_free_async(w, ctx->stream);
        qew_free_async(t, ctx->stream);
        qew_free_async(stat, ctx->stream);
        return s;
    };
    if (qew_alloc_async(ctx, (void **)&w, N * sizeof(double)) != QEW_OK ||
        qew_alloc_async(ctx, (void **)&t, N * sizeof(double)) != QEW_OK ||
        qew_alloc_async(ctx, (void **)&stat, 2 * sizeof(double) + (tx.size() + ty.size()) * sizeof(int2)) !=
            QEW_OK)
        return cleanup(QEW_ERR_NOMEM);
    int2 *tapx = (int2 *)(stat + 2), *tapy = tapx + tx.size();
    cudaError_t e = cudaMemcpyAsync(tapx, tx.data(), tx.size() * sizeof(int2),
                                    cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(tapy, ty.data(), ty.size() * sizeof(int2), cudaMemcpyHostToDevice,
                            ctx->stream);
    if (e != cudaSuccess) return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "%s", cudaGetErrorString(e)));
    const long pairs = (long)nx * ((ny + 1) / 2);
    k_white_noise<<<(unsigned)((pairs + 255) / 256), 256, 0, ctx->stream>>>(w, nx, ny, seed, F1);
    // a filtered sum is in units of 2^(U - F - q) = 2^(b - 62); the first one's
    // samples of 2^-F2 are 3 bits coarser. w [ny][nx] -> t [nx][ny] -> w [nx][ny]
    // one output a thread where four would idle threads (len < 4) or scatter
    // the lanes' loads (a field of few columns): 2^20 x 1 at xi = 3 386 us so,
    // 488 with four; 2^18 x 8 314 with four, 341 so
    auto conv = [&](auto last, auto outs, const long long *in, void *out, int len, int width,
                    const int2 *tap, int R, int exp, int up) {
        constexpr int kOut = decltype(outs)::value;
        int lsh = 0;  // 32 lanes along the fast axis, fewer only on a narrower field
        while (lsh < 5 && (1 << lsh) < width) ++lsh;
        const long long tiles = ((long long)width + (1 << lsh) - 1) >> lsh;
        const long long per = (long long)kOut << (8 - lsh);
        k_gauss_conv<decltype(last)::value, kOut>
            <<<(unsigned)(tiles * ((len + per - 1) / per)), 256, 0, ctx->stream>>>(
                in, out, len, width, tap, R, exp, up, lsh);
    };
    using One = std::integral_constant<int, 1>;
    using Four = std::integral_constant<int, 4>;
    if (ny >= 4 && nx >= 4) {
        conv(std::false_type{}, Four{}, w, t, ny, nx, tapy, Ry, 3, uy.up);
        conv(std::true_type{}, Four{}, t, w, nx, ny, tapx, Rx, ux.b - 62, ux.up);
    } else {
        conv(std::false_type{}, One{}, w, t, ny, nx, tapy, Ry, 3, uy.up);
        conv(std::true_type{}, One{}, t, w, nx, ny, tapx, Rx, ux.b - 62, ux.up);
    }
    qew_status st = qew_launch_check(ctx, "field_generate", 3);
    if (st != QEW_OK) return cleanup(st);
    st = field_moments(ctx, (const double *)w, N, amplitude, stat);
    if (st != QEW_OK) return cleanup(st);
    st = field_build(ctx, (const double *)w, true, nx, ny, Lx, Ly, store_flags, out, stat + 1);
    return cleanup(st);
}

qew_status qew_field_create_seeded(qew_ctx *ctx, int nx, int ny, double Lx, double Ly,
                                  double amplitude, double xi_x, double xi_y, uint64_t seed,
                                  int store_flags, qew_field **out) {
    QEW_RANGE();
    if (!ctx || !out || nx <= 0 || ny <= 0 || !(Lx > 0) || !(Ly > 0) ||
        !std::isfinite(amplitude) || !std::isfinite(xi_x) || !std::isfinite(xi_y))
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create_seeded: bad arguments");
    QEW_CUDA(ctx, cudaSetDevice(ctx->device));
    const size_t N = (size_t)nx * ny;
    cufftDoubleComplex *spec = nullptr, *stage = nullptr;
    double *w = nullptr;
    cufftHandle plan = 0;
    bool have_plan = false;
    const int rows = std::max(1, std::min(nx, (1 << 20) / ny));  // host rows per upload
    const size_t chunk = (size_t)rows * ny;
    cudaEvent_t done[2] = {nullptr, nullptr};
    auto cleanup = [&](qew_status s) {
        cudaStreamSynchronize(ctx->stream);
        if (have_plan) cufftDestroy(plan);
        for (cudaEvent_t &e : done)
            if (e) cudaEventDestroy(e);
        if (stage) cudaFreeHost(stage);
        qew_free_async(spec, ctx->stream);
        qew_free_async(w, ctx->stream);
        return s;
    };
    if (qew_alloc_async(ctx, (void **)&spec, N * sizeof(cufftDoubleComplex)) != QEW_OK ||
        qew_alloc_async(ctx, (void **)&w, N * sizeof(double) + 256) != QEW_OK ||
        cudaMallocHost((void **)&stage, 2 * chunk * sizeof(cufftDoubleComplex)) != cudaSuccess)
        return cleanup(qew_fail(ctx, QEW_ERR_NOMEM, "field_create_seeded: out of memory"));
    for (cudaEvent_t &e : done)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
            return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "field_create_seeded: event"));
    // Random unit phases masked to the correlation ellipse, drawn on the host in
    // the reference's order (filtered_noise.cpp:37-53: i over nx outer, j inner,
    // one draw per entry whether masked or not), uploaded in row chunks through
    // two pinned buffers so drawing overlaps the copies.
    const double two_pi = 2.0 * std::acos(-1.0);
    const double dx = Lx / nx, dy = Ly / ny;
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> phase(0.0, two_pi);
    for (int i0 = 0, b = 0; i0 < nx; i0 += rows, b ^= 1) {
        const int i1 = std::min(nx, i0 + rows);
        cufftDoubleComplex *hs = stage + (size_t)b * chunk;
        if (cudaEventSynchronize(done[b]) != cudaSuccess)
            return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "field_create_seeded: upload"));
        for (int i = i0; i < i1; ++i) {
            const double fx = fft_freq(i, nx) / dx;
            for (int j = 0; j < ny; ++j) {
                const double fy = fft_freq(j, ny) / dy;
                const double ph = phase(rng);
                cufftDoubleComplex a{0.0, 0.0};
                if (!((fx * xi_x) * (fx * xi_x) + (fy * xi_y) * (fy * xi_y) > 1.0))
                    a = cufftDoubleComplex{std::cos(ph), std::sin(ph)};
                hs[(size_t)(i - i0) * ny + j] = a;
            }
        }
        cudaError_t e = cudaMemcpyAsync(spec + (size_t)i0 * ny, hs,
                                        (size_t)(i1 - i0) * ny * sizeof(cufftDoubleComplex),
                                        cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(done[b], ctx->stream);
        if (e != cudaSuccess) return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "%s", cudaGetErrorString(e)));
    }
    if (cufftPlan2d(&plan, nx, ny, CUFFT_Z2Z) != CUFFT_SUCCESS)
        return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "cufftPlan2d Z2Z(%d, %d) failed", nx, ny));
    have_plan = true;
    if (cufftSetStream(plan, ctx->stream) != CUFFT_SUCCESS ||
        cufftExecZ2Z(plan, spec, spec, CUFFT_INVERSE) != CUFFT_SUCCESS)
        return cleanup(qew_fail(ctx, QEW_ERR_CUDA, "field_create_seeded: inverse FFT failed"));
    double *stat = w + N;
    k_real_part<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(spec, N, 1.0 / (double)N, w);
    qew_status st = qew_launch_check(ctx, "field_seeded");
    if (st == QEW_OK) st = field_moments(ctx, w, N, amplitude, stat);
    if (st != QEW_OK) return cleanup(st);
    return cleanup(field_build(ctx, w, true, nx, ny, Lx, Ly, store_flags, out, stat + 1));
}

qew_status qew_field_create_analytic(qew_ctx *ctx, int kind, double p0, double p1, double p2,
                                     qew_field **out) {
    if (!ctx || !out || kind < QEW_FIELD_ZERO || kind > QEW_FIELD_SINCOS)
        return qew_fail(ctx, QEW_ERR_INVALID, "field_create_analytic: bad kind %d", kind);
    qew_field *f = new (std::nothrow) qew_field();
    if (!f) return QEW_ERR_NOMEM;
    f->kind = kind;
    f->device = ctx->device;
    f->p0 = p0;
    f->p1 = p1;
    f->p2 = p2;
    *out = f;
    return QEW_OK;
}

qew_status qew_field_destroy(qew_field *f) {
    if (!f) return QEW_OK;
    cudaSetDevice(f->device);
    // the coefficients may be in use on any stream: wait for the device
    const bool held = f->coef64 || f->coef32 || f->edge32 || f->poly;
    if (held) cudaDeviceSynchronize();
    qew_free_async(f->coef64, f->stream);
    qew_free_async(f->coef32, f->stream);
    qew_free_async(f->edge32, f->stream);
    qew_free_async(f->poly, f->stream);
    if (held) cudaStreamSynchronize(f->stream);
    delete f;
    return QEW_OK;
}

// Release a field whose coefficients were only used on `stream`: frees in
// that stream's order, without waiting for the rest of the device.
void qew_field_release_on(qew_field *f, cudaStream_t stream) {
    if (!f) return;
    qew_free_async(f->coef64, stream);
    qew_free_async(f->coef32, stream);
    qew_free_async(f->edge32, stream);
    qew_free_async(f->poly, stream);
    delete f;
}

qew_status qew_field_get_coefficients(qew_ctx *ctx, const qew_field *f, double *h_coef) {
    if (!ctx || !f || !h_coef || f->kind != QEW_FIELD_BSPLINE || !f->coef64)
        return qew_fail(ctx, QEW_ERR_INVALID, "get_coefficients: no FP64 B-spline coefficients");
    const size_t N = (size_t)f->nx * f->ny;
    double *tmp = nullptr;
    if (cudaMalloc(&tmp, N * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        return qew_fail(ctx, QEW_ERR_NOMEM, "get_coefficients: cudaMalloc");
    }
    // [ny][nx] -> [nx][ny] is the same transpose with the roles swapped
    k_transpose<<<dim3((f->nx + 31) / 32, (f->ny + 31) / 32), dim3(32, 8), 0, ctx->stream>>>(
        f->coef64, tmp, f->ny, f->nx);
    qew_status st = qew_launch_check(ctx, "transpose");
    if (st == QEW_OK) {
        cudaError_t e = cudaMemcpyAsync(h_coef, tmp, N * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (e != cudaSuccess) st = qew_fail(ctx, QEW_ERR_CUDA, "get_coefficients: %s", cudaGetErrorString(e));
    }
    cudaFree(tmp);
    return st;
}

qew_status qew_field_sample(qew_ctx *ctx, const qew_field *f, const double *d_x, const double *d_y,
                            int m, double *d_v, double *d_dvdx, double *d_dvdy) {
    if (!ctx || !f || (m > 0 && (!d_x || !d_y)) || m < 0)
        return qew_fail(ctx, QEW_ERR_INVALID, "field_sample: bad arguments");
    if (m == 0) return QEW_OK;
    return qew_dispatch_noise(ctx, f, [&](auto nz) -> qew_status {
        k_sample<<<(m + 255) / 256, 256, 0, ctx->stream>>>(nz, d_x, d_y, m, d_v, d_dvdx, d_dvdy);
        return qew_launch_check(ctx, "sample");
    });
}

}  // extern "C"
