// film.cu -- the film output path on the device: Film::save's resolve of the
// accumulated film (core/film.cc:23-30), the reference's RGBE encoding of an HDR image
// (HDRPixel, core/image.cc:63-99) and its tone-mapping operators (GammaTmo, ReinhardTmo,
// DragoTmo, DurandTMO, core/tmo.cc:53-243, with Image::toByte, core/image.cc:476, and the
// bilateral filter of core/birateral.cc),
// plus host writers for the reference's .hdr file layout (Image::saveHdr,
// core/image.cc:390-434) and a minimal PNG.
//
// The per-pixel arithmetic is FP64, in the reference's order, so that the encoded
// bytes equal the reference's for the same float film.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_reduce.cuh>

#include "../../include/spica_gpu.h"
#include "ctx.cuh"

namespace spgpu {

namespace {

constexpr double kRefEps = 1.0e-12;   // EPS, core/common.h:55

// Film::save: pixel / (weight + EPS), per channel (core/film.cc:25-28)
__device__ __forceinline__ void resolvePixel(const float4 f, double *r, double *g, double *b) {
    const double w = static_cast<double>(f.w) + kRefEps;
    *r = static_cast<double>(f.x) / w;
    *g = static_cast<double>(f.y) / w;
    *b = static_cast<double>(f.z) / w;
}

__host__ __device__ __forceinline__ double gray(double r, double g, double b) {   // RGBSpectrum::gray
    return 0.2126 * r + 0.7152 * g + 0.0722 * b;
}

// HDRPixel(color): shared exponent of the largest channel (core/image.cc:72-88)
__host__ __device__ __forceinline__ void rgbeEncode(double r, double g, double b, uint8_t *out) {
    double d = r > g ? r : g;
    d = d > b ? d : b;
    if (d <= 1.0e-32) {
        out[0] = out[1] = out[2] = out[3] = 0;
        return;
    }
    int ie;
    const double m = frexp(d, &ie);
    d = m * 256.0 / d;
    out[0] = static_cast<uint8_t>(r * d);
    out[1] = static_cast<uint8_t>(g * d);
    out[2] = static_cast<uint8_t>(b * d);
    out[3] = static_cast<uint8_t>(ie + 128);
}

// Image::toByte (core/image.cc:476)
__device__ __forceinline__ uint8_t toByte(double d) {
    d = fmax(0.0, fmin(d, 1.0));
    return static_cast<uint8_t>(255.0 * d);
}

// The byte kernels evaluate a pixel in float32 with a bound on the error, and take the
// reference's FP64 evaluation only where the bound leaves a byte (or an exponent) open, so the
// bytes are those of the FP64 evaluation at a small part of its cost: the chip has 1/64 of its
// FP32 rate in FP64, and a pixel's divisions and powers cost some hundred FP64 operations.
// The weights for which 1 / (w + EPS) is 1 / w to float32 accuracy, and no quotient overflows:
__device__ __forceinline__ bool plainWeight(float w) { return w >= 1.0e-3f && w <= 1.0e9f; }

// float32 HDRPixel of f / w: false where a byte may differ from the FP64 encoding.  The float
// quotient is within 2^-22 of the FP64 one, so a scaled channel (below 256) is within 1e-4.
__device__ __forceinline__ bool rgbeFast(float4 f, uchar4 *out) {
    const float mx = fmaxf(f.x, fmaxf(f.y, f.z)), mn = fminf(f.x, fminf(f.y, f.z));
    if (!plainWeight(f.w) || !(mn >= 0.0f) || !(mx <= 1.0e30f)) return false;   // NaN fails too
    if (mx == 0.0f) {
        *out = make_uchar4(0, 0, 0, 0);
        return true;
    }
    const float inv = 1.0f / f.w, d = mx * inv;
    if (d < 1.0e-25f) return false;
    int ie;
    const float m = frexpf(d, &ie);
    if (m < 0.5f + 1.0e-6f || m > 1.0f - 1.0e-6f) return false;   // the exponent is open
    const float scale = ldexpf(inv, 8 - ie);
    float c[3] = {f.x * scale, f.y * scale, f.z * scale};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float b = floorf(c[k]), r = c[k] - b;
        if (c[k] != 0.0f && (r < 1.0e-4f || r > 1.0f - 1.0e-4f)) return false;
        c[k] = b;
    }
    *out = make_uchar4(static_cast<uint8_t>(c[0]), static_cast<uint8_t>(c[1]), static_cast<uint8_t>(c[2]),
                       static_cast<uint8_t>(ie + 128));
    return true;
}

// Bound by HBM (20 bytes a pixel) where the float32 encoding decides.
__global__ void k_film_rgbe(const float4 *__restrict__ film, int n, uchar4 *out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 f = film[i];
        uchar4 px;
        if (!rgbeFast(f, &px)) {
            double r, g, b;
            resolvePixel(f, &r, &g, &b);
            uint8_t e[4];
            rgbeEncode(r, g, b, e);
            px = make_uchar4(e[0], e[1], e[2], e[3]);
        }
        out[i] = px;
    }
}

// The least resolved value of each byte: byte(c) >= k where c / w >= at[k], at[k] =
// (k / 255)^gamma to FP64 accuracy.
struct GammaSteps {
    double at[257];
};

// float32 gamma byte of c / w: -1 where the FP64 evaluation may give another.  y = invG log2(c
// inv) is within invG 1e-7 + 2e-6 of the FP64 one (float quotient, log2f and exp2f, |y| <= 8
// where a byte is not 0), and 255 2^y |y| at most 255 x 0.54: the scaled value is within
// 1e-4 (1 + invG).
__device__ __forceinline__ int gammaFast(float c, float inv, float invG, float margin) {
    if (c == 0.0f) return 0;
    const float v = c * inv;
    if (!(v > 0.0f) || !(v <= 1.0e30f)) return -1;   // negative, NaN, infinite
    if (v > 1.0f + 1.0e-6f) return 255;
    const float t = 255.0f * exp2f(invG * log2f(v)), b = floorf(t);
    if (t - b < margin || t - b > 1.0f - margin) return -1;
    return static_cast<int>(b);
}

// GammaTmo::apply then Image::toByte of one channel, c the film's sum and w its weight + EPS in
// FP64: against the steps next to the float32 estimate, and by the power itself within 1e-12
// of a step (and for what the steps do not cover)
__device__ __noinline__ int gammaExact(const GammaSteps &S, float c, float wf, float invGf, double invG) {
    const double w = static_cast<double>(wf) + kRefEps, r = static_cast<double>(c);
    if (c > 0.0f && c <= 1.0e30f && plainWeight(wf) && invGf <= 32.0f) {
        const float v = c / wf;
        const int k = min(max(static_cast<int>(255.0f * exp2f(invGf * log2f(v)) + 0.5f), 0), 256);
        // the estimate is within 0.01 of the value, so the one step that it may straddle is k's
        const double t = S.at[k] * w, e = 1.0e-12 * t;
        if (r > t + e) return min(k, 255);
        if (r < t - e) return k - 1;
    }
    return toByte(fmin(fmax(pow(r / w, invG), 0.0), 1.0));
}

// GammaTmo::apply then Image::toByte, as LDRFilm::saveImage (films/ldrfilm.cc:25-31).  Bound by
// HBM (19 bytes a pixel) where the float32 bytes decide.  A block's bytes go through shared
// memory, so that a warp's byte stores are to neighbours (out has no alignment of its own).
// A 1920 x 1080 film: 1.22 ms -> 0.04 (0.026 of it this kernel, under ncu).
constexpr int kGammaBlock = 256;
__global__ void __launch_bounds__(kGammaBlock) k_film_gamma(const float4 *__restrict__ film, int n, double invG,
                                                            const __grid_constant__ GammaSteps S, uint8_t *out) {
    __shared__ uint8_t bytes[3 * kGammaBlock];
    const float invGf = static_cast<float>(invG), margin = 2.0e-4f * (1.0f + invGf);
    const bool fast = invGf <= 32.0f;
    for (int64_t base = static_cast<int64_t>(blockIdx.x) * kGammaBlock; base < n;
         base += static_cast<int64_t>(gridDim.x) * kGammaBlock) {
        const int count = static_cast<int>(min(static_cast<int64_t>(kGammaBlock), n - base));
        const int t = threadIdx.x;
        if (t < count) {
            const float4 f = film[base + t];
            int r = -1, g = -1, b = -1;
            if (fast && plainWeight(f.w)) {
                const float inv = 1.0f / f.w;
                r = gammaFast(f.x, inv, invGf, margin);
                g = gammaFast(f.y, inv, invGf, margin);
                b = gammaFast(f.z, inv, invGf, margin);
            }
            if (r < 0) r = gammaExact(S, f.x, f.w, invGf, invG);
            if (g < 0) g = gammaExact(S, f.y, f.w, invGf, invG);
            if (b < 0) b = gammaExact(S, f.z, f.w, invGf, invG);
            bytes[3 * t] = static_cast<uint8_t>(r);
            bytes[3 * t + 1] = static_cast<uint8_t>(g);
            bytes[3 * t + 2] = static_cast<uint8_t>(b);
        }
        __syncthreads();
        for (int k = t; k < 3 * count; k += kGammaBlock) out[3 * base + k] = bytes[k];
        __syncthreads();
    }
}

// The tone-mapping operators compute in FP64, which bounds them (see the Durand operator below):
// one division per pixel where the reference divides each channel several times, and one
// logarithm per thread for the log mean.  A 1920 x 1080 film: Reinhard 1.33 -> 0.60 ms, Drago
// 1.74 -> 0.88 (the scratch that calls keep counted in).

// luminance of a resolved pixel
__device__ __forceinline__ double luminance(float4 f) {
    return gray(f.x, f.y, f.z) / (static_cast<double>(f.w) + kRefEps);
}

// A sum of logarithms as a product: mantissas are multiplied, exponents added up, and one
// logarithm is taken at the end.  Values without a finite logarithm go into the sum as such.
struct LogSum {
    double mantissa = 1.0, other = 0.0;
    long long exponent = 0;
    __device__ __forceinline__ void add(double v) {
        if (!(v >= 2.2250738585072014e-308 && v <= 1.7976931348623157e308)) {
            other += log(v);
            return;
        }
        mantissa = split(mantissa * split(v));
    }
    __device__ __forceinline__ double value() const {
        return other + log(mantissa) + static_cast<double>(exponent) * 0.693147180559945309;
    }
    // v's mantissa in [1, 2), its exponent added to the sum
    __device__ __forceinline__ double split(double v) {
        const int hi = __double2hiint(v);
        exponent += (hi >> 20) - 1023;
        return __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(v));
    }
};

// luminance of each resolved pixel, and the sum of log(L + EPS) (logMean, core/tmo.cc:15)
__global__ void k_film_gray(const float4 *__restrict__ film, int n, double *grayOut, double *logSum) {
    LogSum sum;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double L = luminance(film[i]);
        grayOut[i] = L;
        sum.add(L + kRefEps);
    }
    double part = sum.value();
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(logSum, part);
}

// the film's channels times a luminance factor: the operators' r / (L + EPS) Ld, with Ld = num /
// den, over the weight
__device__ __forceinline__ void writeScaled(float4 f, double L, double num, double den, float *out) {
    const double s = num / (den * (L + kRefEps) * (static_cast<double>(f.w) + kRefEps));
    out[0] = static_cast<float>(f.x * s);
    out[1] = static_cast<float>(f.y * s);
    out[2] = static_cast<float>(f.z * s);
}

// ReinhardTmo::apply (core/tmo.cc:81-101); lw[0] = log sum, lw[1] / lw[2] = sorted
// luminances at the white point's two order statistics
__global__ void k_film_reinhard(const float4 *__restrict__ film, const double *__restrict__ lum, int n, double alpha,
                                const double *lw, const double *lmin, const double *lmax, float *out) {
    const double Lwa = exp(lw[0] / n);
    const double log2Max = log2(*lmax + kRefEps), log2Min = log2(*lmin + kRefEps);
    const double Lwhite = 1.5 * pow(2.0, log2Max - log2Min - 5);   // ReinhardTmo::whitePoint, tmo.cc:123
    const double invWhite2 = 1.0 / (Lwhite * Lwhite), scale = alpha / Lwa;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double L = lum[i], Ls = scale * L;
        writeScaled(film[i], L, Ls * (1.0 + Ls * invWhite2), 1.0 + Ls, out + 3 * static_cast<int64_t>(i));
    }
}

// DragoTmo::apply with Ldmax 100 (core/tmo.cc:135-159); lw = log sum, lmax = the largest
// luminance (lumMax, starting from 0)
__global__ void k_film_drago(const float4 *__restrict__ film, const double *__restrict__ lum, int n, double p,
                             const double *lw, const double *lmax, float *out) {
    const double Lwa = exp(lw[0] / n) / pow(1.0 + p - 0.85, 5.0);
    const double Lmax_wa = fmax(0.0, *lmax) / Lwa;
    const double c1 = log(p) / log(0.5);
    const double c2 = (100.0 / 100.0) / log10(1.0 + Lmax_wa);
    const double invLwa = 1.0 / Lwa, invMax = 1.0 / Lmax_wa;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double L = lum[i], L_wa = L * invLwa;
        const double x = L_wa * invMax;   // x^c1; pow for the bases whose power is not exp(c1 log x)
        const double bias = x > 0.0 && c1 != 0.0 ? exp(c1 * log(x)) : pow(x, c1);
        writeScaled(film[i], L, c2 * log1p(L_wa), log(2.0 + 8.0 * bias), out + 3 * static_cast<int64_t>(i));
    }
}

// DurandTMO (core/tmo.cc:171-243) with the reference's bilateral filter, the recursive
// domain-transform filter of Gastal and Oliveira (core/birateral.cc): luminances l, the
// filter's input log10(gray(l) + 1e-6), and the transformed-domain derivatives
// dctx[y][x] = 1 + (sigma_s / sigma_r) |dI/dx| (W-1 per row), dcty[y][x] likewise (H-1 rows)
//
// Everything is FP64, whose rate is what bounds these kernels (2 FMA a clock and SM), so what
// counts is FP64 operations: one division where the reference divides three channels, natural
// logarithms throughout (the filter is linear, so their scale comes out at the end) with exp for
// every power, and feedback coefficients squared from one iteration to the next.  (The gray
// value of an RGB triple of equal channels v is v up to an ulp and taken as v.)
// A 1280 x 720 film: 29.9 -> 1.04 ms, of which the 20 line passes (10 iterations) take 0.7.
__global__ void k_durand_prepare(const float4 *__restrict__ film, int n, double *lum, double *logL) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double l = luminance(film[i]);
        lum[i] = l;
        logL[i] = log(l + 1.0e-6);
    }
}
// the feedback coefficients of the first iteration, a^dct = exp(dct log a), for both directions;
// ratio is the reference's sigma_s / sigma_r of decimal logarithms over ln 10
// (the V tables of recursiveFilterHorizontal / recursiveFilterVertical)
__global__ void k_durand_feedback(const double *__restrict__ logL, int W, int H, double ratio, double logA, double *Vx,
                                  double *Vy) {
    const int n = W * H;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int y = i / W, x = i - y * W;
        const double v = logL[i];
        if (x < W - 1) Vx[static_cast<int64_t>(y) * (W - 1) + x] = exp(logA * (1.0 + ratio * fabs(logL[i + 1] - v)));
        if (y < H - 1) Vy[i] = exp(logA * (1.0 + ratio * fabs(logL[i + W] - v)));
    }
}

// One filter pass over lines (recursiveFilterHorizontal: rows, recursiveFilterVertical:
// columns): y_j = x_j + V_{j-1} (y_{j-1} - x_j) forward, then z_j = y_j + V_j (z_{j+1} - y_j)
// backward.  Each step is an affine map of its predecessor, so a line is split into kChunks
// chunks, a thread each: the chunk's composed map (A, B), a scan of the maps by one warp per
// line, and the chunk again from its incoming value.  That takes 4 instead of 3 FP64 operations
// an element, and has kChunks times the lines in flight where one thread per line ran a serial
// chain of 2 (W + H) dependent steps on a few warps.  A block holds kLines lines, up to kMaxTile
// elements of each at a time, in shared memory.  128 / 64 chunks of 2 lines: 1.35 / 1.45 ms for
// the whole operator at 1280 x 720, 4 lines 1.50 / 1.44 (1.10 for the first with the scratch
// kept between calls).
// At the end the coefficients are squared in place: the filter's width halves from one
// iteration to the next, so a_{i+1} = a_i^2 and V_{i+1} = V_i^2.
constexpr int kChunks = 128, kLines = 2, kLineThreads = kLines * kChunks;
// an odd number of elements a chunk, so that the chunks' elements lie on different banks
constexpr int kMaxTile = kChunks * 15;
// shared position of element e of line l, tile capacity cap
template <bool ROWS>
__device__ __forceinline__ int lineAt(int l, int e, int cap) {
    return ROWS ? l * cap + e : e * kLines + l;
}
// one direction over the block's tile: x[] in place; coefficient of element e: A[e + aShift];
// carry[l] comes in as the value before the tile and leaves as the tile's last one
template <bool ROWS, bool FORWARD>
__device__ __forceinline__ void filterTile(double *x, const double *A, int len, int cap, int line, int chunk, int per,
                                           double2 (*maps)[kLines], double *carry) {
    const int a = min(chunk * per, len), b = min(a + per, len);
    double ca = 1.0, cb = 0.0;
    for (int k = a; k < b; k++) {
        const int e = FORWARD ? k : len - 1 - k;
        const double v = A[lineAt<ROWS>(line, FORWARD ? e : e + 1, cap + 1)];
        double &xe = x[lineAt<ROWS>(line, e, cap)];
        const double w = fma(-v, xe, xe);   // the step is y -> v y + w
        ca *= v;
        cb = fma(v, cb, w);
        xe = w;
    }
    maps[chunk][line] = make_double2(ca, cb);
    __syncthreads();
    // a warp per line turns the chunks' maps into their incoming values
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < kLines) {
        double2 m[kChunks / 32];
        double sa = 1.0, sb = 0.0;
#pragma unroll
        for (int k = 0; k < kChunks / 32; k++) {
            m[k] = maps[kChunks / 32 * lane + k][warp];
            sb = fma(m[k].x, sb, m[k].y);
            sa *= m[k].x;
        }
        for (int off = 1; off < 32; off <<= 1) {
            const double pa = __shfl_up_sync(0xffffffffu, sa, off), pb = __shfl_up_sync(0xffffffffu, sb, off);
            if (lane >= off) {
                sb = fma(sa, pb, sb);
                sa *= pa;
            }
        }
        const double c0 = carry[warp];
        double in = __shfl_up_sync(0xffffffffu, fma(sa, c0, sb), 1);
        if (lane == 0) in = c0;
#pragma unroll
        for (int k = 0; k < kChunks / 32; k++) {
            maps[kChunks / 32 * lane + k][warp].x = in;
            in = fma(m[k].x, in, m[k].y);
        }
    }
    __syncthreads();
    double y = maps[chunk][line].x;
    for (int k = a; k < b; k++) {
        const int e = FORWARD ? k : len - 1 - k;
        double &xe = x[lineAt<ROWS>(line, e, cap)];
        y = fma(A[lineAt<ROWS>(line, FORWARD ? e : e + 1, cap + 1)], y, xe);
        xe = y;
    }
    if (b == len && a < b) carry[line] = y;
    __syncthreads();
}
template <bool ROWS>
__global__ void __launch_bounds__(kLineThreads) k_durand_lines(double *f, double *V, int W, int H, int cap) {
    extern __shared__ double tile[];
    double *x = tile, *A = tile + kLines * cap;   // A[e]: coefficient between elements e - 1 and e of the tile
    __shared__ double2 maps[kChunks][kLines];
    __shared__ double carry[kLines];
    const int n = ROWS ? W : H, lines = ROWS ? H : W;   // elements of a line, lines
    const int line0 = blockIdx.x * kLines, live = min(kLines, lines - line0);
    const int line = ROWS ? threadIdx.x / kChunks : threadIdx.x % kLines;
    const int chunk = ROWS ? threadIdx.x % kChunks : threadIdx.x / kLines;
    auto at = [&](int l, int e) {   // element e of the block's line l in f
        return ROWS ? static_cast<int64_t>(line0 + l) * W + e : static_cast<int64_t>(e) * W + line0 + l;
    };
    auto vAt = [&](int l, int e) {   // coefficient between elements e and e + 1 in V
        return ROWS ? static_cast<int64_t>(line0 + l) * (W - 1) + e : static_cast<int64_t>(e) * W + line0 + l;
    };
    const int tiles = (n + cap - 1) / cap;
    // body(line, element) over the tile's live lines and elements below len, neighbouring threads
    // on neighbouring addresses
    auto sweep = [&](int len, auto body) {
        if (ROWS) {
            for (int l = 0; l < live; l++)
#pragma unroll 4
                for (int e = threadIdx.x; e < len; e += kLineThreads) body(l, e);
        } else if (static_cast<int>(threadIdx.x) % kLines < live) {
#pragma unroll 4
            for (int e = threadIdx.x / kLines; e < len; e += kLineThreads / kLines) body(threadIdx.x % kLines, e);
        }
    };
    auto load = [&](int e0, int len) {
        sweep(len, [&](int l, int e) { x[lineAt<ROWS>(l, e, cap)] = f[at(l, e0 + e)]; });
        sweep(len + 1, [&](int l, int e) {
            const int j = e0 + e - 1;   // V_j lies between elements j and j + 1
            A[lineAt<ROWS>(l, e, cap + 1)] = j >= 0 && j < n - 1 ? V[vAt(l, j)] : 0.0;
        });
    };
    auto store = [&](int e0, int len) {
        sweep(len, [&](int l, int e) { f[at(l, e0 + e)] = x[lineAt<ROWS>(l, e, cap)]; });
    };
    if (threadIdx.x < kLines) carry[threadIdx.x] = 0.0;
    for (int t = 0; t < tiles; t++) {
        const int e0 = t * cap, len = min(cap, n - e0), per = (len + kChunks - 1) / kChunks | 1;
        load(e0, len);
        __syncthreads();
        filterTile<ROWS, true>(x, A, len, cap, line, chunk, per, maps, carry);
        if (tiles > 1) {
            store(e0, len);
            __syncthreads();
        }
    }
    if (threadIdx.x < kLines) carry[threadIdx.x] = 0.0;   // nothing beyond the last element: its coefficient is 0
    __syncthreads();
    for (int t = tiles - 1; t >= 0; t--) {
        const int e0 = t * cap, len = min(cap, n - e0), per = (len + kChunks - 1) / kChunks | 1;
        if (tiles > 1) {
            load(e0, len);
            __syncthreads();
        }
        filterTile<ROWS, false>(x, A, len, cap, line, chunk, per, maps, carry);
        store(e0, len);
        // the coefficients to the right of this tile's elements
        sweep(min(len, n - 1 - e0), [&](int l, int e) {
            const double v = A[lineAt<ROWS>(l, e + 1, cap + 1)];
            V[vAt(l, e0 + e)] = v * v;
        });
        __syncthreads();
    }
}
// elements of a line that a block holds, and the shared memory for them
int lineTile(int n) {
    const int per = (n + kChunks - 1) / kChunks | 1;
    return std::min(per * kChunks, kMaxTile);
}
size_t lineSmem(int cap) {
    return sizeof(double) * kLines * (2 * static_cast<size_t>(cap) + 1);
}
// The base layer (birateralSeparation) and its logarithm.  The detail layer is luminance over
// base, and its logarithm only ever meets an exp, so it stays a factor (k_durand_apply): a
// logarithm and a division less per pixel (a 1280 x 720 film 1.10 -> 1.04 ms).
__global__ void k_durand_base(const double *__restrict__ filt, int n, double *base, double *logBase) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double b = fmax(0.0, exp(filt[i]) - 1.0e-6) + kRefEps;
        base[i] = b;
        logBase[i] = log(b);
    }
}
// DurandTMO::apply: the compressed base times the detail, over weight and luminance
__global__ void k_durand_apply(const float4 *__restrict__ film, const double *__restrict__ lum,
                               const double *__restrict__ base, const double *__restrict__ logBase, int n,
                               double contrast, const double *maxLog, const double *minLog, float *out) {
    // the reference's compression factor is a natural logarithm over a range of decimal ones
    const double cf = log(contrast) * 2.302585092994045684 / (*maxLog - *minLog);
    const double logAbs = cf * *maxLog;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 f = film[i];
        const double l = lum[i], b = base[i];
        double d = l + kRefEps * b;   // (detail + EPS) times the base
        if (d < 0.0) d = __longlong_as_double(0x7FF8000000000000ll);   // the reference takes its logarithm
        const double s = exp(logBase[i] * cf - logAbs) * d / (b * (static_cast<double>(f.w) + kRefEps) * (l + kRefEps));
        out[3 * static_cast<int64_t>(i) + 0] = static_cast<float>(fmin(fmax(f.x * s, 0.0), 1.0));
        out[3 * static_cast<int64_t>(i) + 1] = static_cast<float>(fmin(fmax(f.y * s, 0.0), 1.0));
        out[3 * static_cast<int64_t>(i) + 2] = static_cast<float>(fmin(fmax(f.z * s, 0.0), 1.0));
    }
}

// the steps of a gamma, kept for the host thread's next call with the same one (257 host powers
// take as long as the kernel)
const GammaSteps &gammaSteps(double gamma) {
    thread_local GammaSteps S;
    thread_local double of = 0.0;
    if (of != gamma) {
        for (int k = 0; k <= 256; k++) S.at[k] = std::pow(k / 255.0, gamma);
        of = gamma;
    }
    return S;
}

// Scratch of one call: the context's kept buffer up to kKeptScratch bytes, for one call at a time
// and until its stream is done with it; the stream's pool above that, or beside another call.
// (That pool gives its memory back at every wait, which cost more than the kernels of a small
// film: 320 x 200, Reinhard 0.39 -> 0.20 ms.)
constexpr size_t kKeptScratch = size_t(128) << 20;
struct CallScratch {
    unsigned char *p = nullptr;
    cudaStream_t s;
    std::unique_lock<std::mutex> kept;
    cudaError_t status = cudaSuccess;
    CallScratch(Ctx &C, size_t bytes, cudaStream_t stream) : s(stream) {
        if (bytes <= kKeptScratch) kept = std::unique_lock<std::mutex>(C.filmScratchMu, std::try_to_lock);
        if (!kept) {
            status = cudaMallocAsync(&p, bytes, s);
            return;
        }
        if (C.filmScratchBytes < bytes) {
            cudaFree(C.filmScratch);
            C.filmScratch = nullptr;
            C.filmScratchBytes = 0;
            status = cudaMalloc(&C.filmScratch, bytes);
            if (status == cudaSuccess) C.filmScratchBytes = bytes;
        }
        p = C.filmScratch;
    }
    ~CallScratch() {
        if (kept) cudaStreamSynchronize(s);
        else if (p) cudaFreeAsync(p, s);
    }
    CallScratch(const CallScratch &) = delete;
    CallScratch &operator=(const CallScratch &) = delete;
};
size_t padded(size_t bytes) { return (bytes + 255) & ~size_t(255); }

int launchGrid(int n) { return std::max(1, std::min((n + 255) / 256, 152 * 8)); }

// ---------------------------------------------------------------- host writers
uint32_t crc32Table[256];
bool crcInit = false;
uint32_t crc32(const uint8_t *p, size_t n, uint32_t c = 0xFFFFFFFFu) {
    if (!crcInit) {   // the PNG specification's CRC-32 (polynomial 0xEDB88320)
        for (uint32_t i = 0; i < 256; i++) {
            uint32_t v = i;
            for (int k = 0; k < 8; k++) v = (v & 1u) ? 0xEDB88320u ^ (v >> 1) : v >> 1;
            crc32Table[i] = v;
        }
        crcInit = true;
    }
    for (size_t i = 0; i < n; i++) c = crc32Table[(c ^ p[i]) & 0xFFu] ^ (c >> 8);
    return c;
}
void put32(std::vector<uint8_t> &v, uint32_t x) {
    v.push_back(static_cast<uint8_t>(x >> 24));
    v.push_back(static_cast<uint8_t>(x >> 16));
    v.push_back(static_cast<uint8_t>(x >> 8));
    v.push_back(static_cast<uint8_t>(x));
}
void pngChunk(std::vector<uint8_t> &file, const char *type, const std::vector<uint8_t> &data) {
    put32(file, static_cast<uint32_t>(data.size()));
    const size_t start = file.size();
    file.insert(file.end(), type, type + 4);
    file.insert(file.end(), data.begin(), data.end());
    put32(file, crc32(file.data() + start, file.size() - start) ^ 0xFFFFFFFFu);
}

}  // namespace

int filmResolve(Ctx &C, const float *film, int W, int H, int format, double param, void *out, cudaStream_t s) {
    const int n = W * H;
    const float4 *f4 = reinterpret_cast<const float4 *>(film);
    cudaError_t e = cudaSuccess;
    if (format == SPGPU_FILM_RGBE) {
        k_film_rgbe<<<launchGrid(n), 256, 0, s>>>(f4, n, static_cast<uchar4 *>(out));
        e = cudaGetLastError();
    } else if (format == SPGPU_FILM_GAMMA_BYTES) {
        const GammaSteps &steps = gammaSteps(param);
        k_film_gamma<<<launchGrid(n), 256, 0, s>>>(f4, n, 1.0 / param, steps, static_cast<uint8_t *>(out));
        e = cudaGetLastError();
    } else if (format == SPGPU_FILM_DRAGO) {   // luminances, their log mean and maximum
        const double p = param > 0.0 ? param : 0.85;
        size_t tmpBytes = 0;
        cub::DeviceReduce::Max(nullptr, tmpBytes, static_cast<const double *>(nullptr), static_cast<double *>(nullptr),
                               n, s);
        const size_t bufBytes = padded(sizeof(double) * (static_cast<size_t>(n) + 2));
        CallScratch scratch(C, bufBytes + std::max<size_t>(tmpBytes, 16), s);
        e = scratch.status;
        double *buf = reinterpret_cast<double *>(scratch.p);
        void *tmp = scratch.p + bufBytes;
        if (e == cudaSuccess) e = cudaMemsetAsync(buf + n, 0, sizeof(double), s);
        if (e == cudaSuccess) {
            k_film_gray<<<launchGrid(n), 256, 0, s>>>(f4, n, buf, buf + n);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cub::DeviceReduce::Max(tmp, tmpBytes, buf, buf + n + 1, n, s);
        if (e == cudaSuccess) {
            k_film_drago<<<launchGrid(n), 256, 0, s>>>(f4, buf, n, p, buf + n, buf + n + 1, static_cast<float *>(out));
            e = cudaGetLastError();
        }
    } else if (format == SPGPU_FILM_DURAND) {
        const double contrast = param > 0.0 ? param : 5.0;
        const int maxiter = 20;
        const double sigmaS = std::max(W, H) * 0.02, sigmaR = 0.4;   // DurandTMO defaults, tmo.h:74
        const size_t N = static_cast<size_t>(n);
        size_t t1 = 0, t2 = 0;
        cub::DeviceReduce::Max(nullptr, t1, static_cast<const double *>(nullptr), static_cast<double *>(nullptr), n, s);
        cub::DeviceReduce::Min(nullptr, t2, static_cast<const double *>(nullptr), static_cast<double *>(nullptr), n, s);
        const size_t tmpBytes = std::max<size_t>(std::max(t1, t2), 16);
        const size_t bufBytes = padded(sizeof(double) * (6 * N + 2));
        CallScratch scratch(C, bufBytes + tmpBytes, s);
        e = scratch.status;
        double *buf = reinterpret_cast<double *>(scratch.p);   // lum | filtered | logBase | base | Vx | Vy | max | min
        void *tmp = scratch.p + bufBytes;
        double *lum = buf, *filt = buf + N, *logBase = buf + 2 * N, *base = buf + 3 * N, *Vx = buf + 4 * N,
               *Vy = buf + 5 * N, *mx = buf + 6 * N, *mn = mx + 1;
        const int capX = lineTile(W), capY = lineTile(H);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_durand_lines<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(lineSmem(kMaxTile)));
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_durand_lines<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(lineSmem(kMaxTile)));
        // log of iteration i's feedback base (domainTransformFilter, birateral.cc:118-122)
        auto logFeedback = [&](int i) {
            const double sigmaH =
                sigmaS * std::sqrt(3.0) * std::pow(2.0, maxiter - i - 1) / std::sqrt(std::pow(4.0, maxiter) - 1.0);
            return -std::sqrt(2.0) / sigmaH;
        };
        if (e == cudaSuccess) {
            k_durand_prepare<<<launchGrid(n), 256, 0, s>>>(f4, n, lum, filt);
            k_durand_feedback<<<launchGrid(n), 256, 0, s>>>(filt, W, H, sigmaS / sigmaR / std::log(10.0), logFeedback(0), Vx,
                                                            Vy);
            for (int i = 0; i < maxiter; i++) {
                // coefficients are at most the base a: below 2^-60 a pass moves no luminance
                // (log10, within 1e2) by 1e-16, and a non-finite one has spread over its line
                // and all lines in the first iteration.  10 of 20 iterations for a 720p film
                if (i > 0 && logFeedback(i) < -60.0 * std::log(2.0)) break;
                if (W > 1)
                    k_durand_lines<true><<<(H + kLines - 1) / kLines, kLineThreads, lineSmem(capX), s>>>(filt, Vx, W, H,
                                                                                                         capX);
                if (H > 1)
                    k_durand_lines<false><<<(W + kLines - 1) / kLines, kLineThreads, lineSmem(capY), s>>>(filt, Vy, W, H,
                                                                                                          capY);
            }
            k_durand_base<<<launchGrid(n), 256, 0, s>>>(filt, n, base, logBase);
            e = cudaGetLastError();
        }
        size_t tb = tmpBytes;
        if (e == cudaSuccess) e = cub::DeviceReduce::Max(tmp, tb, logBase, mx, n, s);
        tb = tmpBytes;
        if (e == cudaSuccess) e = cub::DeviceReduce::Min(tmp, tb, logBase, mn, n, s);
        if (e == cudaSuccess) {
            k_durand_apply<<<launchGrid(n), 256, 0, s>>>(f4, lum, base, logBase, n, contrast, mx, mn,
                                                          static_cast<float *>(out));
            e = cudaGetLastError();
        }
    } else {   // SPGPU_FILM_REINHARD: luminances, their log mean and two order statistics
        size_t tmpBytes = 0;
        cub::DeviceRadixSort::SortKeys(nullptr, tmpBytes, static_cast<const double *>(nullptr),
                                       static_cast<double *>(nullptr), n, 0, 64, s);
        const size_t bufBytes = padded(sizeof(double) * (2 * static_cast<size_t>(n) + 1));
        CallScratch scratch(C, bufBytes + std::max<size_t>(tmpBytes, 16), s);
        e = scratch.status;
        double *buf = reinterpret_cast<double *>(scratch.p);
        void *tmp = scratch.p + bufBytes;
        if (e == cudaSuccess) e = cudaMemsetAsync(buf + 2 * static_cast<size_t>(n), 0, sizeof(double), s);
        if (e == cudaSuccess) {
            k_film_gray<<<launchGrid(n), 256, 0, s>>>(f4, n, buf, buf + 2 * static_cast<size_t>(n));
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cub::DeviceRadixSort::SortKeys(tmp, tmpBytes, buf, buf + n, n, 0, 64, s);
        // ReinhardTmo::whitePoint's indices (tmo.cc:118-119)
        const int iMax = std::min(static_cast<int>(n * 0.99), n - 1);
        const int iMin = std::min(static_cast<int>(n * 0.01), n - 1);
        if (e == cudaSuccess) {
            k_film_reinhard<<<launchGrid(n), 256, 0, s>>>(f4, buf, n, param, buf + 2 * static_cast<size_t>(n),
                                                           buf + n + iMin, buf + n + iMax, static_cast<float *>(out));
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? 0 : cudaFail("spgpu_film_resolve", e);
}

// Image::saveHdr's header and scanlines: per row the new-style RLE marker (2, 2, width)
// and each of the four channels as literal runs of at most 127 bytes
int writeHdr(const char *path, const uint8_t *rgbe, int W, int H) {
    std::vector<uint8_t> file;
    const char nl = 0x0a;
    char buf[256];
    const std::string header = std::string("#?RADIANCE") + nl + "# Made with 100% pure HDR Shop" + nl +
                               "FORMAT=32-bit_rle_rgbe" + nl + "EXPOSURE=1.0000000000000" + nl + nl;
    file.insert(file.end(), header.begin(), header.end());
    std::snprintf(buf, sizeof(buf), "-Y %u +X %u%c", static_cast<unsigned>(H), static_cast<unsigned>(W), nl);
    file.insert(file.end(), buf, buf + std::strlen(buf));
    const unsigned w = static_cast<unsigned>(W);
    for (int y = 0; y < H; y++) {
        const uint8_t *row = rgbe + 4 * static_cast<size_t>(y) * W;
        file.push_back(0x02);
        file.push_back(0x02);
        file.push_back(static_cast<uint8_t>((w >> 8) & 0xFFu));
        file.push_back(static_cast<uint8_t>(w & 0xFFu));
        for (int c = 0; c < 4; c++) {
            for (unsigned cursor = 0; cursor < w;) {
                const unsigned run = std::min(127u, w - cursor);
                file.push_back(static_cast<uint8_t>(run));
                for (unsigned j = cursor; j < cursor + run; j++) file.push_back(row[4 * j + c]);
                cursor += run;
            }
        }
    }
    FILE *fp = std::fopen(path, "wb");
    if (!fp) {
        setError(std::string("spgpu_write_hdr: cannot open ") + path);
        return SPGPU_EINVAL;
    }
    const size_t wrote = std::fwrite(file.data(), 1, file.size(), fp);
    std::fclose(fp);
    if (wrote != file.size()) {
        setError(std::string("spgpu_write_hdr: short write to ") + path);
        return SPGPU_EINVAL;
    }
    return 0;
}

// 8-bit RGB PNG: zlib stream of stored (uncompressed) deflate blocks, filter 0 per row
int writePng(const char *path, const uint8_t *rgb, int W, int H) {
    std::vector<uint8_t> raw;
    raw.reserve(static_cast<size_t>(H) * (3 * W + 1));
    for (int y = 0; y < H; y++) {
        raw.push_back(0);
        raw.insert(raw.end(), rgb + 3 * static_cast<size_t>(y) * W, rgb + 3 * static_cast<size_t>(y + 1) * W);
    }
    std::vector<uint8_t> z = {0x78, 0x01};
    uint32_t a = 1, b = 0;   // Adler-32
    for (uint8_t v : raw) {
        a = (a + v) % 65521u;
        b = (b + a) % 65521u;
    }
    for (size_t off = 0; off < raw.size() || off == 0;) {
        const size_t len = std::min<size_t>(65535, raw.size() - off);
        const bool last = off + len >= raw.size();
        z.push_back(last ? 1 : 0);
        z.push_back(static_cast<uint8_t>(len & 0xFF));
        z.push_back(static_cast<uint8_t>(len >> 8));
        z.push_back(static_cast<uint8_t>(~len & 0xFF));
        z.push_back(static_cast<uint8_t>((~len >> 8) & 0xFF));
        z.insert(z.end(), raw.begin() + off, raw.begin() + off + len);
        off += len;
        if (last) break;
    }
    put32(z, (b << 16) | a);
    std::vector<uint8_t> file = {0x89, 'P', 'N', 'G', 0x0D, 0x0A, 0x1A, 0x0A};
    std::vector<uint8_t> ihdr;
    put32(ihdr, static_cast<uint32_t>(W));
    put32(ihdr, static_cast<uint32_t>(H));
    ihdr.insert(ihdr.end(), {8, 2, 0, 0, 0});   // 8-bit, truecolour, deflate, filter 0, no interlace
    pngChunk(file, "IHDR", ihdr);
    pngChunk(file, "IDAT", z);
    pngChunk(file, "IEND", {});
    FILE *fp = std::fopen(path, "wb");
    if (!fp) {
        setError(std::string("spgpu_write_png: cannot open ") + path);
        return SPGPU_EINVAL;
    }
    const size_t wrote = std::fwrite(file.data(), 1, file.size(), fp);
    std::fclose(fp);
    if (wrote != file.size()) {
        setError(std::string("spgpu_write_png: short write to ") + path);
        return SPGPU_EINVAL;
    }
    return 0;
}

}  // namespace spgpu
