// The two standalone post-filters of denoising/, as passes over per-pixel records.
//
// atrous_wavelet (denoising/atrous_wavelet.cpp:54-149, ping-ponged 185-197): `iterations`
// passes of the 5x5 B3-spline at step 2^i with luminance, normal-angle and albedo edge
// stopping, clamp-to-edge, centre kept when the weights vanish.
//   k_atrous_records  once per call: the unit normal (the stored normal renormalised when its
//                     squared length exceeds EPS_SMALL, atrous_wavelet.cpp:76-79), the albedo and
//                     the colour with its luminance of every pixel as float4 records;
//   k_atrous_pass     one pass. A thread owns four pixels `step` rows apart, whose 5-row windows
//                     share most of their eight rows: a tap's three records are read once for up
//                     to four pixels. The edge-stopping factors exp(a) exp(b) exp(c) and the spline
//                     weight are one base-2 exponential, the squared angle between the normals a
//                     polynomial in 1 - |cos| (angle_squared). The last pass writes the output.
//   k_atrous_pass_plain  the same pass without records, the normals renormalised at each tap
//                     (rpd_atrous_wavelet_noalloc, which has no scratch for them).
// joint_bilateral (denoising/joint_bilateral.cpp:15-132): one (2r+1)^2 window, r =
// max(1, ceil(3 sigma_p)), writing the gaussian, colour-bilateral and joint outputs at once.
//   k_bilateral_records  once per call: colour, the decoded unit normal (n * 2 - 1, then
//                     normalised, joint_bilateral.cpp:54-56,80-82) and albedo as float4 planes;
//   k_joint_bilateral a block of 32 x 8 threads, two pixels each, stages its (32 + 2r) x (16 + 2r)
//                     halo tile of the three planes in shared memory with one tensor copy
//                     (radius <= 16; larger radii read the records from global memory). Taps
//                     outside the image clamp into it, as the reference's do. A row's gaussian
//                     sums serve both pixels, whose row factors multiply them at the row's end.
// Offsets are 64-bit. Single-precision arithmetic like the reference's; the exponentials are
// CUDA's and the angle's polynomial is this file's, so outputs agree with the reference within the
// plain-form bar (1e-4 relative), not to the bit.
#include <algorithm>
#include <cmath>
#include <utility>

#include "rpd_internal.h"
#include "device_math.cuh"
#include "tma.cuh"

namespace rpd {

namespace {

// The reference's normalize(): scale by 1/sqrt(|v|^2) when |v|^2 > EPS_SMALL, operations in
// its order (the translation unit is compiled without contraction).
__device__ __forceinline__ float4 unit_or_same(float x, float y, float z) {
    const float len_sq = x * x + y * y + z * z;
    if (len_sq > 1e-8f) {
        const float inv_len = 1.0f / sqrtf(len_sq);
        x *= inv_len;
        y *= inv_len;
        z *= inv_len;
    }
    return make_float4(x, y, z, 0.0f);
}

__device__ __forceinline__ float dot_fma(float4 a, float4 b) {
    return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, a.x * b.x));
}
__device__ __forceinline__ float dist2_fma(float4 a, float4 b) {
    const float x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
    return __fmaf_rn(z, z, __fmaf_rn(y, y, x * x));
}
__device__ __forceinline__ float exp2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// to 2^-23
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// acos(clamp(d, -1, 1))^2 of N values. With t = 1 - cos a, a^2 = 4 asin^2(sqrt(t / 2)) is a power
// series in t (2t + t^2 / 3 + ...) that converges up to t = 2: for angles up to 90 degrees a polynomial
// a^2 = t p(t) of degree 7 in t, fitted to minimise the relative error over t in [0, 1] by
// iteratively reweighted least squares on Chebyshev nodes (1.7e-7 with the rounding of its
// single-precision evaluation; the square of an angle to 2 ulp is off by up to 4.8e-7). Larger angles
// through pi - acos(|d|), behind one branch for all N (normals in every direction take it at nearly every tap:
// a joint bilateral of such an image 0.87 ms with the IEEE square root, 0.63 with the approximate one). A NaN
// falls out of the saturation: the callers add 0 * d to the exponent.
template <int N>
__device__ __forceinline__ void angles_squared(const float (&d)[N], float (&a2)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float t = __saturatef(1.0f - fabsf(d[k]));
        float p = 0.00512921950f;
        p = __fmaf_rn(p, t, -0.00878358912f);
        p = __fmaf_rn(p, t, 0.01423186157f);
        p = __fmaf_rn(p, t, 0.00472163549f);
        p = __fmaf_rn(p, t, 0.03006852977f);
        p = __fmaf_rn(p, t, 0.08869015425f);
        p = __fmaf_rn(p, t, 0.33334326744f);
        p = __fmaf_rn(p, t, 1.99999988079f);
        a2[k] = p * t;
    }
    float least = d[0];
#pragma unroll
    for (int k = 1; k < N; ++k) least = fminf(least, d[k]);
    if (least < 0.0f) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float a = 3.14159265f - sqrt_approx(a2[k]);
            if (d[k] < 0.0f) a2[k] = a * a;
        }
    }
}

// w_color * w_normal * w_albedo (atrous_wavelet.cpp:122-139) times the spline weight, whose base-2
// logarithm is `spline`; d, a2: the cosine and the square of the angle between the normals. kc, kn, ka: -log2(e) / (2 sigma^2) of the colour, normal and albedo terms.
__device__ __forceinline__ float atrous_weight(float spline, float d, float a2, float li, float lj, float4 ai, float4 aj,
                                               float kc, float kn, float ka) {
    const float ld = li - lj;
    const float s = __fmaf_rn(d, 0.0f, spline);
    return exp2_approx(__fmaf_rn(ld * ld, kc, __fmaf_rn(a2, kn, __fmaf_rn(dist2_fma(ai, aj), ka, s))));
}
// log2 of the B3-spline taps 1/16, 1/4, 3/8 (atrous_wavelet.cpp:20)
__device__ __forceinline__ float b3_log2(int k) { return k == 2 ? -1.41503750f : (k & 1) ? -2.0f : -4.0f; }

__global__ void k_atrous_records(const float* __restrict__ raw, const float* __restrict__ normal,
                                 const float* __restrict__ albedo, int64_t np, float4* __restrict__ col,
                                 float4* __restrict__ nrm, float4* __restrict__ alb) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float r = raw[3 * i], g = raw[3 * i + 1], b = raw[3 * i + 2];
    col[i] = make_float4(r, g, b, luminance(r, g, b));
    nrm[i] = unit_or_same(normal[3 * i], normal[3 * i + 1], normal[3 * i + 2]);
    alb[i] = make_float4(albedo[3 * i], albedo[3 * i + 1], albedo[3 * i + 2], 0.0f);
}

constexpr int kAtrousRows = 4;

// A thread's pixels of an a-trous pass: their records and sums (rgb, weight).
struct AtrousPixels {
    float4 ni[kAtrousRows], ai[kAtrousRows];
    float li[kAtrousRows], s[kAtrousRows][4];
};

struct AtrousTap {
    float4 c, n, a;
};

// The tap in row J of the thread's eight (the first two pixels above, the last two below its own): tap
// J - k of its pixels k.
template <int J>
__device__ __forceinline__ void atrous_row(const AtrousTap& tap, float lx, float kc, float kn, float ka, AtrousPixels& p) {
    constexpr int first = J < 4 ? 0 : J - 4, last = J < kAtrousRows ? J : kAtrousRows - 1;
    constexpr int n = last - first + 1;
    const float4 c = tap.c, nj = tap.n, aj = tap.a;
    float d[n], a2[n];
#pragma unroll
    for (int i = 0; i < n; ++i) d[i] = dot_fma(p.ni[first + i], nj);
    angles_squared<n>(d, a2);
#pragma unroll
    for (int i = 0; i < n; ++i) {
        const int k = first + i;
        const float wt = atrous_weight(lx + b3_log2(J - k), d[i], a2[i], p.li[k], c.w, p.ai[k], aj, kc, kn, ka);
        p.s[k][0] = __fmaf_rn(wt, c.x, p.s[k][0]);
        p.s[k][1] = __fmaf_rn(wt, c.y, p.s[k][1]);
        p.s[k][2] = __fmaf_rn(wt, c.z, p.s[k][2]);
        p.s[k][3] += wt;
    }
}

// One a-trous pass over records (rgb, luminance), unit normals and albedo. sx, sy: the step, at most the
// image's width and height (atrous_step). rgb: the interleaved
// output of the last pass, else nullptr.
// Bound by instruction issue with the records' latency close behind (68% of the issue slots at 16
// warps per SM). One pass at 1920x1080: about 150 us with one pixel per thread, the arc cosine and the
// colour read as three components; 113-127 us with four pixels and the polynomial, 89-101 us with
// one branch per row for the angles above 90 degrees, 85-94 us with the reads a row ahead, 79-87 us
// with the approximate square root there (the IEEE one has a path of its own, which splits the code).
// Limits for three or four blocks per SM spill or lose the reads ahead: 5-7% slower.
__global__ void __launch_bounds__(256, 2) k_atrous_pass(const float4* __restrict__ in, float4* __restrict__ out,
                                                     float* __restrict__ rgb, const float4* __restrict__ nrm,
                                                     const float4* __restrict__ alb, int w, int h, int sx, int sy, float kc,
                                                     float kn, float ka) {
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int group = blockIdx.y * 8 + threadIdx.y;  // rows y0, y0 + sy, ... of one group
    const int y0 = group / sy * (kAtrousRows * sy) + group % sy;
    if (x >= w || y0 >= h) return;
    AtrousPixels p;
#pragma unroll
    for (int k = 0; k < kAtrousRows; ++k) {
        const int64_t i = int64_t(imins(y0 + k * sy, h - 1)) * w + x;
        p.ni[k] = nrm[i];
        p.ai[k] = alb[i];
        p.li[k] = in[i].w;
        p.s[k][0] = p.s[k][1] = p.s[k][2] = p.s[k][3] = 0.0f;
    }
    int64_t rows[kAtrousRows + 4];
#pragma unroll
    for (int j = 0; j < kAtrousRows + 4; ++j) rows[j] = int64_t(iclamps(y0 + (j - 2) * sy, 0, h - 1)) * w;
    auto load = [&](int j, int xx) {
        const int64_t q = rows[j] + xx;
        return AtrousTap{in[q], nrm[q], alb[q]};
    };
    int xx = iclamps(x - 2 * sx, 0, w - 1);
    AtrousTap tap[2] = {load(0, xx), {}};  // each tap is read a row ahead of its use
#pragma unroll 1
    for (int kx = 0; kx < 5; ++kx) {
        const int xn = iclamps(x + (kx - 1) * sx, 0, w - 1);
        const float lx = b3_log2(kx);
        tap[1] = load(1, xx);
        atrous_row<0>(tap[0], lx, kc, kn, ka, p);
        tap[0] = load(2, xx);
        atrous_row<1>(tap[1], lx, kc, kn, ka, p);
        tap[1] = load(3, xx);
        atrous_row<2>(tap[0], lx, kc, kn, ka, p);
        tap[0] = load(4, xx);
        atrous_row<3>(tap[1], lx, kc, kn, ka, p);
        tap[1] = load(5, xx);
        atrous_row<4>(tap[0], lx, kc, kn, ka, p);
        tap[0] = load(6, xx);
        atrous_row<5>(tap[1], lx, kc, kn, ka, p);
        tap[1] = load(7, xx);
        atrous_row<6>(tap[0], lx, kc, kn, ka, p);
        xx = xn;
        tap[0] = load(0, xx);  // the next column's first; after the last column unused
        atrous_row<7>(tap[1], lx, kc, kn, ka, p);
    }
#pragma unroll
    for (int k = 0; k < kAtrousRows; ++k) {
        const int y = y0 + k * sy;
        if (y >= h) continue;
        const int64_t i = int64_t(y) * w + x;
        float4 v;
        if (p.s[k][3] > 1e-8f) {
            const float inv = 1.0f / p.s[k][3];
            v = make_float4(p.s[k][0] * inv, p.s[k][1] * inv, p.s[k][2] * inv, 0.0f);
        } else {
            v = in[i];
        }
        if (rgb) {
            rgb[3 * i] = v.x;
            rgb[3 * i + 1] = v.y;
            rgb[3 * i + 2] = v.z;
        } else {
            v.w = luminance(v.x, v.y, v.z);
            out[i] = v;
        }
    }
}

// One a-trous pass over interleaved images: the same arithmetic in the same order, so its results are
// k_atrous_pass's.
__global__ void __launch_bounds__(256) k_atrous_pass_plain(const float* __restrict__ in, float* __restrict__ out,
                                                           const float* __restrict__ normal,
                                                           const float* __restrict__ albedo, int w, int h, int step,
                                                           float kc, float kn, float ka) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= w || y >= h) return;
    const int64_t i = int64_t(y) * w + x;
    const float cr = in[3 * i], cg = in[3 * i + 1], cb = in[3 * i + 2];
    const float li = luminance(cr, cg, cb);
    const float4 ni = unit_or_same(normal[3 * i], normal[3 * i + 1], normal[3 * i + 2]);
    const float4 ai = make_float4(albedo[3 * i], albedo[3 * i + 1], albedo[3 * i + 2], 0.0f);
    int64_t rows[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) rows[k] = int64_t(iclamps(y + (k - 2) * step, 0, h - 1)) * w;
    float sr = 0.0f, sg = 0.0f, sb = 0.0f, sw = 0.0f;
#pragma unroll 1
    for (int kx = 0; kx < 5; ++kx) {
        const int xx = iclamps(x + (kx - 2) * step, 0, w - 1);
        const float lx = b3_log2(kx);
#pragma unroll
        for (int ky = 0; ky < 5; ++ky) {
            const int64_t j = rows[ky] + xx;
            const float pr = in[3 * j], pg = in[3 * j + 1], pb = in[3 * j + 2];
            const float4 nj = unit_or_same(normal[3 * j], normal[3 * j + 1], normal[3 * j + 2]);
            const float4 aj = make_float4(albedo[3 * j], albedo[3 * j + 1], albedo[3 * j + 2], 0.0f);
            const float d[1] = {dot_fma(ni, nj)};
            float a2[1];
            angles_squared<1>(d, a2);
            const float wt = atrous_weight(lx + b3_log2(ky), d[0], a2[0], li, luminance(pr, pg, pb), ai, aj, kc, kn, ka);
            sr = __fmaf_rn(wt, pr, sr);
            sg = __fmaf_rn(wt, pg, sg);
            sb = __fmaf_rn(wt, pb, sb);
            sw += wt;
        }
    }
    if (sw > 1e-8f) {
        const float inv = 1.0f / sw;
        out[3 * i] = sr * inv;
        out[3 * i + 1] = sg * inv;
        out[3 * i + 2] = sb * inv;
    } else {
        out[3 * i] = cr;
        out[3 * i + 1] = cg;
        out[3 * i + 2] = cb;
    }
}

enum BilateralPlane { B_COL = 0, B_NRM, B_ALB, B_COUNT };

__global__ void k_bilateral_records(const float* __restrict__ raw, const float* __restrict__ normal,
                                    const float* __restrict__ albedo, int64_t np, float4* __restrict__ rec) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= np) return;
    rec[B_COL * np + i] = make_float4(raw[3 * i], raw[3 * i + 1], raw[3 * i + 2], 0.0f);
    rec[B_NRM * np + i] =
        unit_or_same(normal[3 * i] * 2.0f - 1.0f, normal[3 * i + 1] * 2.0f - 1.0f, normal[3 * i + 2] * 2.0f - 1.0f);
    rec[B_ALB * np + i] = make_float4(albedo[3 * i], albedo[3 * i + 1], albedo[3 * i + 2], 0.0f);
}

struct BilateralParams {
    int w, h, r;
    float kp, kc, kn, ka;   // -log2(e) / (2 sigma^2) of the pixel-distance, colour, normal and albedo terms
    float kp_e;             // 1 / (2 sigma_p^2)
};

constexpr int kBx = 32, kBy = 8;  // threads of a block
constexpr int kBRows = 2;         // pixels of a thread, one above the other
constexpr int kBMaxTiled = 16;    // the largest radius whose halo tile is in shared memory
constexpr size_t bilateral_tile_bytes(int r) {
    return 128 + size_t(kBx + 2 * r) * (kBy * kBRows + 2 * r) * B_COUNT * sizeof(float4) + size_t(2 * r + 1) * sizeof(float2);
}

// A thread's pixels (x, y0 .. y0 + kBRows - 1): their records and the three filters' sums (rgb, weight).
struct BilateralPixels {
    float4 ci[kBRows], ni[kBRows], ai[kBRows];
    float g[kBRows][4], c[kBRows][4], j[kBRows][4];
};

// The taps of window row cy. S: the records, row its first element at x = 0, `plane` elements between
// planes. EDGE: some tap may lie outside the image (clamped into it, joint_bilateral.cpp:60). FIRST,
// LAST: the pixels whose windows hold the row. gx[r + i]: the gaussian of the distance i in one
// direction and its log2.
template <bool EDGE, int FIRST, int LAST>
__device__ __forceinline__ void bilateral_row(const float4* __restrict__ S, int64_t row, int64_t plane,
                                              const BilateralParams& prm, const float2* __restrict__ gx,
                                              int x, int y0, int cy, BilateralPixels& p) {
    const int r = prm.r;
    constexpr int n = LAST - FIRST + 1;
    float ly[n], rg[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < n; ++k) {
        const float dd = float(y0 + FIRST + k - cy);
        ly[k] = dd * dd * prm.kp;
    }
    const float4* C = S + B_COL * plane + row;
    const float4* N = S + B_NRM * plane + row;
    const float4* A = S + B_ALB * plane + row;
    if (!EDGE) {
        C += x - r;
        N += x - r;
        A += x - r;
    }
#pragma unroll 4
    for (int i = 0; i <= 2 * r; ++i) {
        const int cx = EDGE ? iclamps(x - r + i, 0, prm.w - 1) : i;
        const float2 gl = gx[EDGE ? cx - x + r : i];
        const float4 cj = C[cx], nj = N[cx], aj = A[cx];
        rg[0] = __fmaf_rn(gl.x, cj.x, rg[0]);
        rg[1] = __fmaf_rn(gl.x, cj.y, rg[1]);
        rg[2] = __fmaf_rn(gl.x, cj.z, rg[2]);
        rg[3] += gl.x;
        float d[n], a2[n];
#pragma unroll
        for (int k = 0; k < n; ++k) d[k] = dot_fma(p.ni[FIRST + k], nj);
        angles_squared<n>(d, a2);
#pragma unroll
        for (int k = 0; k < n; ++k) {
            const int q = FIRST + k;
            // kc carries alpha = 0.5, kn beta = 2 - alpha = 1.5
            const float ec = __fmaf_rn(dist2_fma(p.ci[q], cj), prm.kc, gl.y + ly[k]);
            const float en = __fmaf_rn(a2[k], prm.kn, __fmaf_rn(d[k], 0.0f, ec));
            const float ej = __fmaf_rn(dist2_fma(p.ai[q], aj), prm.ka, en);
            const float wc = exp2_approx(ec), wj = exp2_approx(ej);
            p.c[q][0] = __fmaf_rn(wc, cj.x, p.c[q][0]);
            p.c[q][1] = __fmaf_rn(wc, cj.y, p.c[q][1]);
            p.c[q][2] = __fmaf_rn(wc, cj.z, p.c[q][2]);
            p.c[q][3] += wc;
            p.j[q][0] = __fmaf_rn(wj, cj.x, p.j[q][0]);
            p.j[q][1] = __fmaf_rn(wj, cj.y, p.j[q][1]);
            p.j[q][2] = __fmaf_rn(wj, cj.z, p.j[q][2]);
            p.j[q][3] += wj;
        }
    }
#pragma unroll
    for (int k = FIRST; k <= LAST; ++k) {
        const float wy = gx[r + cy - (y0 + k)].x;
#pragma unroll
        for (int q = 0; q < 4; ++q) p.g[k][q] = __fmaf_rn(wy, rg[q], p.g[k][q]);
    }
}

// The (2r+1)^2 taps of a thread's pixels; (ox, oy): the image position of S's first element.
template <bool EDGE>
__device__ __forceinline__ void bilateral_taps(const float4* __restrict__ S, int64_t stride, int64_t plane, int ox, int oy,
                                               const BilateralParams& prm, const float2* __restrict__ gx,
                                               int x, int y0, BilateralPixels& p) {
    static_assert(kBRows == 2, "the first and the last row belong to one pixel each");
    auto line = [&](int j) { return EDGE ? iclamps(y0 + j, 0, prm.h - 1) : y0 + j; };
    auto first = [&](int cy) { return int64_t(cy - oy) * stride - ox; };
    const int r = prm.r;
    int cy = line(-r);
    bilateral_row<EDGE, 0, 0>(S, first(cy), plane, prm, gx, x, y0, cy, p);
    for (int j = 1 - r; j <= r; ++j) {
        cy = line(j);
        bilateral_row<EDGE, 0, 1>(S, first(cy), plane, prm, gx, x, y0, cy, p);
    }
    cy = line(r + 1);
    bilateral_row<EDGE, 1, 1>(S, first(cy), plane, prm, gx, x, y0, cy, p);
}

// kTiled: the halo tile is in shared memory (one tensor copy); else the records are read from
// global memory (radius > 16).
// Bound by instruction issue (85% of the slots). At 1920x1080, r = 6: 0.94 ms with one pixel per thread,
// clamped coordinates at every tap, three separate gaussian sums and the arc cosine; 0.64 ms with two
// pixels, the row sums and the polynomial, 0.56 ms with one branch per tap for both angles and four taps
// per turn at two blocks per SM (three blocks 0.58, eight taps 0.58), 0.53 ms with the approximate square root.
template <bool kTiled>
__global__ void __launch_bounds__(kBx * kBy, 2)
    k_joint_bilateral(const float4* __restrict__ rec, BilateralParams prm, float* __restrict__ gaussian,
                      float* __restrict__ bilateral, float* __restrict__ joint, unsigned* fail,
                      const __grid_constant__ CUtensorMap tmap) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int s_fail;
    const int r = prm.r;
    constexpr int rows = kBy * kBRows;
    const int x0 = blockIdx.x * kBx, yb = blockIdx.y * rows;
    const int tid = threadIdx.y * kBx + threadIdx.x;
    const int tw = kBx + 2 * r, th = rows + 2 * r;
    const int64_t np = int64_t(prm.w) * prm.h;
    const uint32_t pad = (128u - (smem_addr(smem_raw) & 127u)) & 127u;
    float4* T = reinterpret_cast<float4*>(smem_raw + pad);
    float2* gx = reinterpret_cast<float2*>(kTiled ? T + B_COUNT * tw * th : T);  // 2r + 1 distances
    const uint32_t bar_a = smem_addr(&bar);
    if constexpr (kTiled) {
        if (tid == 0) {
            mbar_init(bar_a, 1);
            s_fail = 0;
        }
        __syncthreads();
        if (tid == 0) tile_load(T, &tmap, x0, yb, r, tw, th, B_COUNT, bar_a);
    }
    // weight_gauss = exp(-d^2 / (2 sigma_p^2)) (joint_bilateral.cpp:100) is the product of one factor
    // per direction
    for (int i = tid; i < 2 * r + 1; i += kBx * kBy) {
        const float d = float(i - r);
        gx[i] = make_float2(expf(-(d * d) * prm.kp_e), d * d * prm.kp);
    }
    if constexpr (kTiled) {
        if (!mbar_wait_bounded(bar_a, 0)) s_fail = 1;
    }
    __syncthreads();
    if constexpr (kTiled) {
        if (s_fail) {
            if (tid == 0) {
                atomicAdd(fail, 1u);
                mbar_wait_bounded(bar_a, 0);
            }
            return;
        }
    }
    const int x = x0 + threadIdx.x, y0 = yb + threadIdx.y * kBRows;
    if (x >= prm.w || y0 >= prm.h) return;
    // the tile origin, or the image itself when reading global records
    const int ox = kTiled ? x0 - r : 0, oy = kTiled ? yb - r : 0;
    const int64_t stride = kTiled ? tw : prm.w;
    const int64_t plane = kTiled ? int64_t(tw) * th : np;
    const float4* S = kTiled ? T : rec;
    BilateralPixels p;
#pragma unroll
    for (int k = 0; k < kBRows; ++k) {
        // below the image's last row: that row's pixel again, not written
        const int64_t e = int64_t(imins(y0 + k, prm.h - 1) - oy) * stride + (x - ox);
        p.ci[k] = S[B_COL * plane + e];
        p.ni[k] = S[B_NRM * plane + e];
        p.ai[k] = S[B_ALB * plane + e];
#pragma unroll
        for (int q = 0; q < 4; ++q) p.g[k][q] = p.c[k][q] = p.j[k][q] = 0.0f;
    }
    if (x0 < r || yb < r || x0 + kBx + r > prm.w || yb + rows + r > prm.h)
        bilateral_taps<true>(S, stride, plane, ox, oy, prm, gx, x, y0, p);
    else
        bilateral_taps<false>(S, stride, plane, ox, oy, prm, gx, x, y0, p);
#pragma unroll
    for (int k = 0; k < kBRows; ++k) {
        if (y0 + k >= prm.h) continue;
        const int64_t i = int64_t(y0 + k) * prm.w + x;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            gaussian[3 * i + q] = p.g[k][q] / p.g[k][3];
            bilateral[3 * i + q] = p.c[k][q] / p.c[k][3];
            joint[3 * i + q] = p.j[k][q] / p.j[k][3];
        }
    }
}

// The largest radius taken: (2 r + 1)^2 taps per pixel. (sigma_p up to 40; a call for minutes is an error,
// not a request.)
constexpr int kBMaxRadius = 120;
// Blocks of 8 rows of one pixel per thread: the tallest image that the grid's second dimension holds.
constexpr int kFilterRows = 65535 * 8;

float inv_two_sq(float sigma) { return float(1.0 / (2.0 * double(sigma) * double(sigma))); }
float neg_log2e_two_sq(float sigma, double scale = 1.0) {
    return float(-1.4426950408889634 * scale / (2.0 * double(sigma) * double(sigma)));
}

// 2^it, or the image's extent where that is less: from there on every tap but the centre's is clamped to the
// edge. (Groups of rows a step apart beyond the height would exceed the grid.)
int atrous_step(int it, int extent) { return it < 30 ? std::min(1 << it, extent) : extent; }

}  // namespace

cudaError_t filter_limits(int h, float sigma_p) {
    if (h > kFilterRows) return cudaErrorInvalidConfiguration;
    return std::ceil(3.0f * sigma_p) > float(kBMaxRadius) ? cudaErrorInvalidValue : cudaSuccess;
}

uint64_t atrous_scratch_bytes(int w, int h) { return uint64_t(w) * h * 4 * sizeof(float4); }

cudaError_t launch_atrous(const float* raw, const float* normal, const float* albedo, int w, int h, float sigma_c,
                          float sigma_n, float sigma_a, int iterations, void* scratch, float* out, cudaStream_t stream,
                          uint64_t* launches) {
    const int64_t np = int64_t(w) * h;
    if (iterations == 0) {
        if (out == raw) return cudaSuccess;
        return cudaMemcpyAsync(out, raw, size_t(np) * 12, cudaMemcpyDeviceToDevice, stream);
    }
    float4* a = static_cast<float4*>(scratch);
    float4* b = a + np;
    float4* nrm = b + np;
    float4* alb = nrm + np;
    k_atrous_records<<<grid_for(np, 256), 256, 0, stream>>>(raw, normal, albedo, np, a, nrm, alb);
    const float kc = neg_log2e_two_sq(sigma_c), kn = neg_log2e_two_sq(sigma_n), ka = neg_log2e_two_sq(sigma_a);
    for (int it = 0; it < iterations; ++it) {
        const int sx = atrous_step(it, w), sy = atrous_step(it, h);
        // groups of kAtrousRows rows sy apart: sy of them per kAtrousRows * sy rows
        const int64_t span = int64_t(kAtrousRows) * sy;
        const int64_t groups = (h + span - 1) / span * sy;
        const dim3 grid((w + 31) / 32, unsigned((groups + 7) / 8));
        k_atrous_pass<<<grid, dim3(32, 8), 0, stream>>>(a, b, it + 1 == iterations ? out : nullptr, nrm, alb, w, h, sx, sy,
                                                        kc, kn, ka);
        std::swap(a, b);
    }
    *launches += 1 + iterations;
    return cudaGetLastError();
}

cudaError_t launch_atrous_plain(const float* raw, const float* normal, const float* albedo, int w, int h, float sigma_c,
                                float sigma_n, float sigma_a, int iterations, float* buf_a, float* buf_b, float** result,
                                cudaStream_t stream) {
    const dim3 block(32, 8);
    const dim3 grid((w + 31) / 32, (h + 7) / 8);
    const float kc = neg_log2e_two_sq(sigma_c), kn = neg_log2e_two_sq(sigma_n), ka = neg_log2e_two_sq(sigma_a);
    const float* in = raw;
    float* out = buf_a;
    float* other = buf_b;
    *result = const_cast<float*>(raw);
    for (int it = 0; it < iterations; ++it) {
        k_atrous_pass_plain<<<grid, block, 0, stream>>>(in, out, normal, albedo, w, h, atrous_step(it, std::max(w, h)), kc, kn, ka);
        *result = out;
        in = out;
        float* t = out;
        out = other;
        other = t;
    }
    return cudaGetLastError();
}

uint64_t joint_bilateral_scratch_bytes(int w, int h) { return uint64_t(w) * h * B_COUNT * sizeof(float4) + 256; }

cudaError_t launch_joint_bilateral(const float* raw, const float* normal, const float* albedo, int w, int h,
                                   float sigma_c, float sigma_n, float sigma_p, float sigma_a, float* gaussian,
                                   float* bilateral, float* joint, void* scratch, cudaStream_t stream,
                                   uint64_t* launches) {
    const int64_t np = int64_t(w) * h;
    float4* rec = static_cast<float4*>(scratch);
    unsigned* fail = reinterpret_cast<unsigned*>(rec + B_COUNT * np);
    cudaError_t e = cudaMemsetAsync(fail, 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return e;
    k_bilateral_records<<<grid_for(np, 256), 256, 0, stream>>>(raw, normal, albedo, np, rec);
    BilateralParams prm{};
    prm.w = w;
    prm.h = h;
    prm.r = std::max(1, int(std::ceil(3.0f * sigma_p)));  // joint_bilateral.cpp:43
    prm.kp = neg_log2e_two_sq(sigma_p);
    prm.kc = neg_log2e_two_sq(sigma_c, 0.5);
    prm.kn = neg_log2e_two_sq(sigma_n, 1.5);
    prm.ka = neg_log2e_two_sq(sigma_a);
    prm.kp_e = inv_two_sq(sigma_p);
    const dim3 block(kBx, kBy);
    const int rows = kBy * kBRows;
    const dim3 grid((w + kBx - 1) / kBx, (h + rows - 1) / rows);
    const bool tiled = prm.r <= kBMaxTiled;
    CUtensorMap map{};
    size_t smem = 128 + size_t(2 * prm.r + 1) * sizeof(float2);  // below 48 KB up to kBMaxRadius
    if (tiled) {
        smem = bilateral_tile_bytes(prm.r);
        e = encode_record_map(&map, rec, w, h, B_COUNT, kBx + 2 * prm.r, rows + 2 * prm.r);
        if (e != cudaSuccess) return e;
    }
    // the limit belongs to the kernel, not to the call: always the largest tile's, so that no thread lowers it
    // between another one's setting and its launch
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(k_joint_bilateral<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(bilateral_tile_bytes(kBMaxTiled)));
        if (e != cudaSuccess) return e;
    }
    if (tiled)
        k_joint_bilateral<true><<<grid, block, smem, stream>>>(rec, prm, gaussian, bilateral, joint, fail, map);
    else
        k_joint_bilateral<false><<<grid, block, smem, stream>>>(rec, prm, gaussian, bilateral, joint, fail, map);
    *launches += 2;
    return cudaGetLastError();
}

}  // namespace rpd
