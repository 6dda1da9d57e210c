// Per-sample accumulation: pixel statistics, primary-hit features and the RPD grid.
//
//   k_accumulate_pixels  accumulate_sample (core/stats.h:25-41) and the feature / radiance
//                        sums of the render loops (main.cpp:572-576, 706-717), one thread
//                        per pixel walking its samples in order — bit-identical to the
//                        reference, whose pixel is also owned by a single thread.
//   k_grid_ordered       accumulate_rpf_sample_to_grid (main.cpp:329-376) regrouped by
//                        owner: one thread per (node, dependency) visits the node's support
//                        pixels in row-major order and their samples in order, which is the
//                        reference's summation order with one OpenMP thread, so the grid is
//                        bit-identical to that run. No atomics; deterministic.
//   k_merge_grid         merge_rpf_grids_into (main.cpp:378-388).
//   k_feature_cache      ensure_feature_cache (main.cpp:94-122).
//   k_finalize           FrameBuffers::finalize (core/buffers.h:152-167).
#include <cuda_fp16.h>

#include "rpd_internal.h"
#include "device_math.cuh"
#include "tma.cuh"

namespace rpd {

namespace {

constexpr int kScanBlock = 1024;

__global__ void k_offsets_uniform(int64_t* offsets, int64_t count, int32_t spp) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i <= count) offsets[i] = i * int64_t(spp);
}

// Three-phase exclusive scan of int32 counts into int64 offsets[0..count]: per-block sums, a
// scan of the block sums by one block, and the per-block scans shifted by them. Warp-shuffle
// scans, so each phase is a few steps per element.
__device__ __forceinline__ int64_t warp_incl_scan(int64_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int64_t t = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += t;
    }
    return v;
}

// inclusive scan over the block (blockDim.x == kScanBlock); `total` gets the block's sum
__device__ __forceinline__ int64_t block_incl_scan(int64_t v, int64_t* total) {
    __shared__ int64_t warp_tot[kScanBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_incl_scan(v);
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int64_t t = warp_incl_scan(warp_tot[lane]);
        warp_tot[lane] = t;
    }
    __syncthreads();
    if (warp > 0) v += warp_tot[warp - 1];
    if (total) *total = warp_tot[kScanBlock / 32 - 1];
    __syncthreads();
    return v;
}

// largest count of the block (counts are >= 0; 0 for an empty block)
__device__ __forceinline__ int32_t block_max(int32_t v) {
    __shared__ int32_t warp_max[kScanBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = __reduce_max_sync(0xffffffffu, v);
    if (lane == 0) warp_max[warp] = v;
    __syncthreads();
    if (warp == 0) v = __reduce_max_sync(0xffffffffu, warp_max[lane]);
    __syncthreads();
    return v;
}

// per block: the sum of its counts (block_sums) and their maximum (block_max)
__global__ void __launch_bounds__(kScanBlock) k_scan_block_sums(const int32_t* counts, int64_t count, int64_t* block_sums,
                                                              int64_t* block_maxima) {
    const int64_t i = int64_t(blockIdx.x) * kScanBlock + threadIdx.x;
    const int32_t c = (i < count) ? counts[i] : 0;
    int64_t total;
    block_incl_scan(int64_t(c), &total);
    const int32_t m = block_max(c < 0 ? 0 : c);
    if (threadIdx.x == 0) {
        block_sums[blockIdx.x] = total;
        block_maxima[blockIdx.x] = m;
    }
}

// one block: block_sums[0..nblocks) -> exclusive offsets, block_sums[nblocks] = the total;
// block_maxima[nblocks] = the largest count
__global__ void __launch_bounds__(kScanBlock) k_scan_block_offsets(int64_t* block_sums, int64_t* block_maxima,
                                                                 int64_t nblocks) {
    int64_t carry = 0;
    int32_t mx = 0;
    for (int64_t b0 = 0; b0 < nblocks; b0 += kScanBlock) {
        const int64_t b = b0 + threadIdx.x;
        const int64_t v = b < nblocks ? block_sums[b] : 0;
        int64_t total;
        const int64_t incl = block_incl_scan(v, &total);
        if (b < nblocks) block_sums[b] = carry + incl - v;
        carry += total;
        mx = max(mx, block_max(b < nblocks ? int32_t(block_maxima[b]) : 0));
    }
    if (threadIdx.x == 0) {
        block_sums[nblocks] = carry;
        block_maxima[nblocks] = mx;
    }
}

__global__ void __launch_bounds__(kScanBlock) k_scan_finish(const int32_t* counts, int64_t count, const int64_t* block_sums,
                                                           int64_t* offsets) {
    const int64_t i = int64_t(blockIdx.x) * kScanBlock + threadIdx.x;
    const int64_t v = (i < count) ? int64_t(counts[i]) : 0;
    const int64_t incl = block_incl_scan(v, nullptr);
    const int64_t base = block_sums[blockIdx.x];
    if (i < count) offsets[i] = base + incl - v;
    if (i == count - 1) offsets[count] = base + incl;
}

// Dependency2D::add bin (core/stats.h:166-168)
__device__ __forceinline__ int bin2d_k(float u, float v) {
    const int x = iclamps(int(u * 4.0f), 0, 3);
    const int z = iclamps(int(v * 4.0f), 0, 3);
    return z * 4 + x;
}

// TwoSum of x into the double-float (hi, lo).
__device__ __forceinline__ void df_add(float& hi, float& lo, float x) {
    const float s = hi + x;
    const float bb = s - hi;
    lo += (hi - (s - bb)) + (x - bb);
    hi = s;
}

// One traced sample as the statistics pass sees it.
struct SampleIn {
    float L[3], n[3], d, alb[3], pu[2], lu[2], bu[2], liu[2], eu[2];
    uint8_t f, cat;
    uint32_t bins;  // COMPACT_IN: the BRDF, lens, light and environment bins in the key's fields
    float root[3];  // COMPACT_IN: sqrt(max(0, L)), known exactly (L is the square of a half)
};

// x / d correctly rounded from rd = 1/d (itself correctly rounded) by Markstein's correction
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990): q = RN(x rd), the remainder x - d q is exact in a fused
// multiply-add, and RN(q + (x - d q) rd) is the correctly rounded x / d. It holds for a
// positive normal d whose mantissa is not all ones and a quotient, remainder and x in the
// normal range (or x = +0).
__device__ __forceinline__ float div_markstein(float x, float d, float rd) {
    const float q = __fmul_rn(x, rd);
    return __fmaf_rn(__fmaf_rn(-d, q, x), rd, q);
}
__device__ __forceinline__ bool markstein_ok(float x) { return x == 0.0f || fabsf(x) >= 5.42101086e-20f; }  // 2^-64

// Dependency2D::add's bin of a compact (unorm16) pair: u = q / 65536 exactly, so
// int(u * 4) = q >> 14, already within 0..3 (core/stats.h:166-168)
__device__ __forceinline__ uint32_t bin2d_q(uint16_t qu, uint16_t qv) { return uint32_t(qv >> 14) * 4u + uint32_t(qu >> 14); }

// The samples of one validity pattern (pat, 0: none yet): count, sum y and sum y^2 as double-floats.
struct PatternSums {
    uint32_t pat;
    float c, s1h, s1l, s2h, s2l;
    __device__ __forceinline__ void add(float y, float y2, float y2e) {
        c += 1.0f;
        df_add(s1h, s1l, y);
        df_add(s2h, s2l, y2);
        s2l += y2e;
    }
};

// Per-pixel running state of the statistics pass.
struct PixelAcc {
    float mean, m2;
    int n;
    float cm[3], sm[3], sq[3], rad[3], nor[3], alb[3], dep;
    int hits, nsamples;
    // pattern sums for the grid pass: the samples with the same class bits share one set of sums,
    // for the pixel's first kPatterns such patterns; samples of a further one go to per-class sums
    // and make the pixel deviant
    PatternSums pt[kPatterns];
    bool dev;
    // the per-class sums [class][count, s1 hi, s1 lo, s2 hi, s2 lo] of a deviant pixel, in the
    // thread's local memory (written only once the pixel deviates, which is rare): held in
    // registers they would cost 35 registers through the whole sample loop
    float* cs;
    uint8_t pflags;
};

// The packed random-dimension bins of a sample with (masked) flags fm (Dependency2D::add,
// core/stats.h:166-168).
template <bool COMPACT_IN>
__device__ __forceinline__ uint32_t sample_key(const SampleIn& in, uint8_t fm) {
    uint32_t key;
    if (COMPACT_IN) {
        key = (fm & RPD_SAMPLE_BRDF_VALID) ? in.bins & 0x1fu : key_absent_bit(1);
        key |= (fm & RPD_SAMPLE_LENS_VALID) ? in.bins & (0x1fu << 5) : key_absent_bit(2);
        key |= (fm & RPD_SAMPLE_LIGHT_VALID) ? in.bins & (0x1fu << 10) : key_absent_bit(3);
        key |= (fm & RPD_SAMPLE_ENV_VALID) ? in.bins & (0x1fu << 15) : key_absent_bit(4);
    } else {
        key = (fm & RPD_SAMPLE_BRDF_VALID) ? uint32_t(bin2d_k(in.bu[0], in.bu[1])) : key_absent_bit(1);
        key |= (fm & RPD_SAMPLE_LENS_VALID) ? uint32_t(bin2d_k(in.lu[0], in.lu[1])) << 5 : key_absent_bit(2);
        key |= (fm & RPD_SAMPLE_LIGHT_VALID) ? uint32_t(bin2d_k(in.liu[0], in.liu[1])) << 10 : key_absent_bit(3);
        key |= (fm & RPD_SAMPLE_ENV_VALID) ? uint32_t(bin2d_k(in.eu[0], in.eu[1])) << 15 : key_absent_bit(4);
    }
    key |= (fm & RPD_SAMPLE_LIGHT_SELECT_VALID) ? uint32_t(in.cat & RPD_CATEGORY_LIGHT_INDEX_MASK) << 20 : key_absent_bit(5);
    key |= (fm & RPD_SAMPLE_RR_VALID) ? ((in.cat & RPD_CATEGORY_RR_SURVIVED) ? 1u << 25 : 0u) : key_absent_bit(6);
    key |= (fm & RPD_SAMPLE_PIXEL_VALID) ? 0u : key_absent_bit(0);
    return key;
}

// A finite sample's luminance into its pixel's pattern sums. A tracer's pixels hold a few patterns (all
// dimensions, paths that ended before Russian roulette, paths that ended at the first hit): with
// one pattern in registers and the rest added class by class in local memory, a 1920x1080x16
// frame of such samples took 1.71 ms in this pass, with three patterns in registers 0.99 ms (0.76
// with one reciprocal per sample; 0.64 ms for a frame of a single pattern).
template <typename Acc>
__device__ __forceinline__ void class_add(Acc& a, uint8_t fm, float lum) {
    const uint32_t bits = fm & 0xfeu;
    if (bits == 0u) return;  // no validity class: nothing for the grid's totals
    const float y2 = lum * lum;
    const float y2e = __fmaf_rn(lum, lum, -y2);
    // (selects, not branches: the compiler would merge three branches into one over an array in local
    // memory)
    if (a.pt[0].pat == 0u) a.pt[0].pat = bits;
    if (a.pt[0].pat == bits) {
        a.pt[0].add(lum, y2, y2e);
        return;
    }
    if (a.pt[1].pat == 0u) a.pt[1].pat = bits;
    else if (a.pt[1].pat != bits && a.pt[2].pat == 0u) a.pt[2].pat = bits;
    const bool one = a.pt[1].pat == bits;
    if (one || a.pt[2].pat == bits) {
        PatternSums t;
        t.c = one ? a.pt[1].c : a.pt[2].c;
        t.s1h = one ? a.pt[1].s1h : a.pt[2].s1h;
        t.s1l = one ? a.pt[1].s1l : a.pt[2].s1l;
        t.s2h = one ? a.pt[1].s2h : a.pt[2].s2h;
        t.s2l = one ? a.pt[1].s2l : a.pt[2].s2l;
        t.add(lum, y2, y2e);
        a.pt[1].c = one ? t.c : a.pt[1].c;
        a.pt[1].s1h = one ? t.s1h : a.pt[1].s1h;
        a.pt[1].s1l = one ? t.s1l : a.pt[1].s1l;
        a.pt[1].s2h = one ? t.s2h : a.pt[1].s2h;
        a.pt[1].s2l = one ? t.s2l : a.pt[1].s2l;
        a.pt[2].c = one ? a.pt[2].c : t.c;
        a.pt[2].s1h = one ? a.pt[2].s1h : t.s1h;
        a.pt[2].s1l = one ? a.pt[2].s1l : t.s1l;
        a.pt[2].s2h = one ? a.pt[2].s2h : t.s2h;
        a.pt[2].s2l = one ? a.pt[2].s2l : t.s2l;
        return;
    }
    if (!a.dev) {
        a.dev = true;
        for (int q = 0; q < kClasses * 5; ++q) a.cs[q] = 0.0f;
    }
    for (int c = 0; c < kClasses; ++c) {
        if (!(bits & class_bit(c))) continue;
        float* e = a.cs + 5 * c;
        float h1 = e[1], l1 = e[2], h2 = e[3], l2 = e[4];
        df_add(h1, l1, lum);
        df_add(h2, l2, y2);
        l2 += y2e;
        e[0] += 1.0f;
        e[1] = h1;
        e[2] = l1;
        e[3] = h2;
        e[4] = l2;
    }
}

// Is a sample at offset f = fl(x + u) - x of pixel x in the pixel's own screen bin at every node? With a
// power-of-two support 4 <= S <= 2^11 the bin is floor(fl(fl(x + u) - left) / (S/4)) (the division
// and the x4 are power-of-two scalings; left is an integer): fl(X - left) is exact for left >= 0,
// and for the first node row/column (left = -S/2, X + S/2 < 2^12) it moves by at most 2^-13
// (main.cpp:352-356, core/stats.h:166-167). So it is whenever f lies in [0, 1 - 2^-12], or the
// position at least a pixel inside the bin's bin_pixels pixels.
__device__ __forceinline__ bool in_own_bin(float f, float x, int bin_pixels) {
    const float at = float(int(x) & (bin_pixels - 1)) + f;
    return (f >= 0.0f || at >= 1.0f) && (f <= kUniformMax || at <= float(bin_pixels - 1));
}

// A finite sample's screen position: does it stay in its pixel's bin, does a random dimension come
// without one.
__device__ __forceinline__ void screen_flags(const SampleIn& in, uint8_t fm, float fx, float fy, int bin_pixels,
                                             uint8_t& pflags) {
    if (fm & RPD_SAMPLE_PIXEL_VALID) {
        const float jx = (fx + in.pu[0]) - fx, jy = (fy + in.pu[1]) - fy;
        if (!(jx >= 0.0f && jx <= kUniformMax && jy >= 0.0f && jy <= kUniformMax)) {
            if (!(in_own_bin(jx, fx, bin_pixels) && in_own_bin(jy, fy, bin_pixels))) pflags &= uint8_t(~kPixUniform);
        }
    } else if (fm & (RPD_SAMPLE_LENS_VALID | RPD_SAMPLE_BRDF_VALID | RPD_SAMPLE_LIGHT_VALID | RPD_SAMPLE_ENV_VALID |
                     RPD_SAMPLE_LIGHT_SELECT_VALID | RPD_SAMPLE_RR_VALID)) {
        pflags |= kPixMixed;  // a random dimension without the screen position
    }
}

// What a thread of the statistics pass keeps of its pixel: everything, or one of two parts that share
// nothing but the radiance they read (kColour: the channels' statistics, normal and albedo sums;
// kLuminance: the luminance statistics, depth, counts, sample keys and the grid pass's sums).
enum Part { kWhole = 0, kColour = 1, kLuminance = 2 };

// COMPACT_IN: a sample decoded from the compact planes. Its radiance is the square of a
// non-negative half, so sqrt(max(0, L)) is exactly that half (in.root) and no dividend is infinite,
// and the random-dimension bins come with it (in.bins).
template <bool COMPACT_IN, Part PART>
__device__ __forceinline__ void process_sample(PixelAcc& a, const SampleIn& in, bool per_sample_albedo,
                                               const float* palb, bool prep, uint8_t plane_mask, float fx,
                                               float fy, int bin_pixels, float& lum_out, uint32_t& key_out) {
    constexpr bool colour = PART != kLuminance, lumi = PART != kColour;
    if (in.f & RPD_SAMPLE_HIT) {  // main.cpp:572-576
        if (lumi) {
            ++a.hits;
            a.dep += in.d;
        }
        if (colour) {
            for (int c = 0; c < 3; ++c) a.nor[c] += in.n[c];
            for (int c = 0; c < 3; ++c) a.alb[c] += per_sample_albedo ? in.alb[c] : palb[c];
        }
    }
    if (!finite3(in.L[0], in.L[1], in.L[2])) {  // main.cpp:707
        lum_out = __int_as_float(0x7fc00000);  // NaN: dropped by the grid pass
        key_out = kKeyNone;
        return;
    }
    // accumulate_sample (core/stats.h:25-41). The quotients by n come from one reciprocal where
    // that is exact (div_markstein): the dividends are known before any of the updates. (Of a -0
    // it makes +0, which the running means, never -0, add the same.) FP32 planes took seven
    // divisions: 1920x1080x16 of path-like samples 0.98 -> 0.76 ms, adaptive counts 541 -> 469 us.
    ++a.n;
    const float fn = float(a.n);
    float lum = 0.0f, delta = 0.0f, cd[3], root[3], sd[3];
    bool fast = a.n < (1 << 23);
    float size = 0.0f;  // FP32 radiance near the type's limits: a dividend may be infinite
    if (lumi) {
        lum = luminance(in.L[0], in.L[1], in.L[2]);
        delta = lum - a.mean;
        size += fabsf(delta);
        fast = fast && markstein_ok(delta);
    }
    if (colour) {
        for (int c = 0; c < 3; ++c) {
            root[c] = COMPACT_IN ? in.root[c] : sqrtf(fmaxs(0.0f, in.L[c]));
            cd[c] = in.L[c] - a.cm[c];
            sd[c] = root[c] - a.sm[c];
            size += fabsf(cd[c]);
            fast = fast && markstein_ok(cd[c]) && markstein_ok(sd[c]);
        }
    }
    if (!COMPACT_IN) fast = fast && size < INFINITY;
    if (fast) {
        const float rn = 1.0f / fn;
        if (lumi) a.mean += div_markstein(delta, fn, rn);
        if (colour) {
            for (int c = 0; c < 3; ++c) a.cm[c] += div_markstein(cd[c], fn, rn);
            for (int c = 0; c < 3; ++c) a.sm[c] += div_markstein(sd[c], fn, rn);
        }
    } else {
        if (lumi) a.mean += delta / fn;
        if (colour) {
            for (int c = 0; c < 3; ++c) a.cm[c] += cd[c] / fn;
            for (int c = 0; c < 3; ++c) a.sm[c] += sd[c] / fn;
        }
    }
    if (colour) {
        for (int c = 0; c < 3; ++c) a.sq[c] += sd[c] * (root[c] - a.sm[c]);
        for (int c = 0; c < 3; ++c) a.rad[c] += in.L[c];
    }
    if (!lumi) return;
    const float delta2 = lum - a.mean;
    a.m2 += delta * delta2;
    ++a.nsamples;
    lum_out = lum;
    key_out = kKeyNone;
    if (!prep) return;
    const uint8_t fm = in.f & plane_mask;
    key_out = sample_key<COMPACT_IN>(in, fm);
    class_add(a, fm, lum);
    screen_flags(in, fm, fx, fy, bin_pixels, a.pflags);
}

__device__ __forceinline__ float4 ld4(const float* p, int64_t k) { return *reinterpret_cast<const float4*>(p + k); }
__device__ __forceinline__ float lane4(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// rpd_sample_soa16 decoding (include/rpd_gb300.h)
__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ __forceinline__ float snorm16(int16_t q) { return fmaxf(float(q) * (1.0f / 32767.0f), -1.0f); }
__device__ __forceinline__ float unorm16(uint16_t q) { return float(q) * (1.0f / 65536.0f); }
__device__ __forceinline__ float sq(float v) { return v * v; }

// A pixel's running state before its first sample of the push (the class sums start empty).
__device__ __forceinline__ void acc_init(PixelAcc& a) {
    a.pflags = kPixUniform;
    a.dev = false;  // the class sums are cleared when the pixel deviates
    for (int k = 0; k < kPatterns; ++k) a.pt[k] = PatternSums{0u, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
}

// The grid-pass sums of a pixel without samples in the push.
__device__ __forceinline__ void acc_store_empty(const GridPrep& gp, int64_t idx) {
    gp.pat4[idx] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    gp.pat2[idx] = make_float2(0.0f, __uint_as_float(uint32_t(kPixUniform) << 8));
}

__device__ __forceinline__ void acc_zero(PixelAcc& a) {
    a.mean = a.m2 = 0.0f;
    a.n = 0;
    for (int c = 0; c < 3; ++c) a.cm[c] = a.sm[c] = a.sq[c] = a.rad[c] = a.nor[c] = a.alb[c] = 0.0f;
    a.dep = 0.0f;
    a.hits = a.nsamples = 0;
}

template <Part PART>
__device__ __forceinline__ void acc_load(PixelAcc& a, const PixelPlanes& p, int64_t idx) {
    a.n = p.n[idx];
    if (PART != kLuminance) {
        for (int c = 0; c < 3; ++c) {
            a.cm[c] = p.color_mean[c][idx];
            a.sm[c] = p.sqrt_mean[c][idx];
            a.sq[c] = p.sqrt_sq[c][idx];
            a.rad[c] = p.radiance[c][idx];
            a.nor[c] = p.normal[c][idx];
            a.alb[c] = p.albedo[c][idx];
        }
    }
    if (PART != kColour) {
        a.mean = p.mean[idx];
        a.m2 = p.square_diff[idx];
        a.dep = p.depth[idx];
        a.hits = p.hit_count[idx];
        a.nsamples = p.sample_count[idx];
    }
}

// The grid-pass sums of a pixel (GridPrep): its first pattern's, and either its further patterns' or, for a
// deviant pixel, the per-class sums.
template <typename Acc>
__device__ __forceinline__ void store_classes(const Acc& a, const GridPrep& gp, int64_t idx, uint8_t pflags) {
    const PatternSums& p0 = a.pt[0];
    gp.pat4[idx] = make_float4(p0.c, p0.s1h, p0.s1l, p0.s2h);
    uint32_t bits = p0.pat | (uint32_t(pflags) << 8);
    if (!a.dev) {
        for (int k = 1; k < kPatterns; ++k) bits |= a.pt[k].pat << (8 * (k + 1));
    } else {
        const uint32_t pats = p0.pat | a.pt[1].pat | a.pt[2].pat;
        const bool placed = (pats & class_bit(0)) || a.cs[0] > 0.0f;
        bits |= uint32_t(kPixDeviant | (placed ? kPixPlaced : 0)) << 8;
    }
    gp.pat2[idx] = make_float2(p0.s2l, __uint_as_float(bits));
    if (!a.dev) {
#pragma unroll
        for (int k = 1; k < kPatterns; ++k) {
            const PatternSums& t = a.pt[k];
            if (t.pat == 0u) continue;
            gp.cls[k - 1][0][idx] = t.c;
            gp.cls[k - 1][1][idx] = t.s1h;
            gp.cls[k - 1][2][idx] = t.s1l;
            gp.cls[k - 1][3][idx] = t.s2h;
            gp.cls[k - 1][4][idx] = t.s2l;
        }
        return;
    }
    // full per-class sums: the deviating samples plus the patterns'
    for (int c = 0; c < kClasses; ++c) {
        const float* e = a.cs + 5 * c;
        float h1 = e[1], l1 = e[2], h2 = e[3], l2 = e[4], cnt = e[0];
#pragma unroll
        for (int k = 0; k < kPatterns; ++k) {
            const PatternSums& t = a.pt[k];
            if (!(t.pat & class_bit(c))) continue;
            cnt += t.c;
            df_add(h1, l1, t.s1h);
            l1 += t.s1l;
            df_add(h2, l2, t.s2h);
            l2 += t.s2l;
        }
        gp.cls[c][0][idx] = cnt;
        gp.cls[c][1][idx] = h1;
        gp.cls[c][2][idx] = l1;
        gp.cls[c][3][idx] = h2;
        gp.cls[c][4][idx] = l2;
    }
}

// The pixel's statistics back to its planes, and its grid-pass sums: the pattern class's, and
// for a deviant pixel the full per-class sums.
template <Part PART>
__device__ __forceinline__ void acc_store(const PixelAcc& a, const PixelPlanes& p, const GridPrep& gp, int64_t idx,
                                          bool prep) {
    if (PART != kLuminance) {
        for (int c = 0; c < 3; ++c) {
            p.color_mean[c][idx] = a.cm[c];
            p.sqrt_mean[c][idx] = a.sm[c];
            p.sqrt_sq[c][idx] = a.sq[c];
            p.radiance[c][idx] = a.rad[c];
            p.normal[c][idx] = a.nor[c];
            p.albedo[c][idx] = a.alb[c];
        }
    }
    if (PART != kColour) {
        p.mean[idx] = a.mean;
        p.square_diff[idx] = a.m2;
        p.n[idx] = a.n;
        p.depth[idx] = a.dep;
        p.hit_count[idx] = a.hits;
        p.sample_count[idx] = a.nsamples;
        if (prep) store_classes(a, gp, idx, a.pflags);
    }
}

__device__ __forceinline__ uint8_t plane_mask_of(bool pu, bool lu, bool bu, bool li, bool eu) {
    return uint8_t(0xffu & ~((pu ? 0 : RPD_SAMPLE_PIXEL_VALID) | (lu ? 0 : RPD_SAMPLE_LENS_VALID) |
                             (bu ? 0 : RPD_SAMPLE_BRDF_VALID) | (li ? 0 : RPD_SAMPLE_LIGHT_VALID) |
                             (eu ? 0 : RPD_SAMPLE_ENV_VALID)));
}

// What the samples of a pixel share.
struct PixelIn {
    bool per_sample_albedo, prep;
    float palb[3];
    uint8_t plane_mask;  // the flags whose planes are present
    float fx, fy;
    int bin_pixels;
};

template <bool COMPACT>
__device__ __forceinline__ void load_pixel_albedo(PixelIn& px, const DeviceSamples& s, int64_t local) {
    if (COMPACT) {
        if (s.c16.pixel_albedo[0])
            for (int c = 0; c < 3; ++c) px.palb[c] = h2f(s.c16.pixel_albedo[c][local]);
    } else if (!px.per_sample_albedo && s.pixel_albedo[0]) {
        for (int c = 0; c < 3; ++c) px.palb[c] = s.pixel_albedo[c][local];
    }
}

// Four FP32 samples of a pixel, each plane's as one 16-byte load; flags and categories one byte each.
struct Quad32 {
    float4 L[3], N[3], A[3], D, PU[2], LU[2], BU[2], LI[2], EU[2];
    uint32_t F, C;
};
template <Part PART>
__device__ __forceinline__ void process_quad(PixelAcc& a, const Quad32& q, const PixelIn& px, float* lum, uint32_t* key) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        SampleIn in;
        for (int c = 0; c < 3; ++c) {
            in.L[c] = lane4(q.L[c], i);
            in.n[c] = lane4(q.N[c], i);
            in.alb[c] = lane4(q.A[c], i);
        }
        in.d = lane4(q.D, i);
        for (int c = 0; c < 2; ++c) {
            in.pu[c] = lane4(q.PU[c], i);
            in.lu[c] = lane4(q.LU[c], i);
            in.bu[c] = lane4(q.BU[c], i);
            in.liu[c] = lane4(q.LI[c], i);
            in.eu[c] = lane4(q.EU[c], i);
        }
        in.f = uint8_t(q.F >> (8 * i));
        in.cat = uint8_t(q.C >> (8 * i));
        process_sample<false, PART>(a, in, px.per_sample_albedo, px.palb, px.prep, px.plane_mask, px.fx, px.fy, px.bin_pixels, lum[i], key[i]);
    }
}

// V compact samples of a pixel (V = 4 or 8), two per 32-bit word of each plane.
template <int V>
struct Words {
    uint32_t w[V / 2];
    __device__ __forceinline__ uint16_t at(int i) const { return uint16_t(w[i >> 1] >> (16 * (i & 1))); }
};
template <int V>
struct Group16 {
    Words<V> L[3], N[3], D, PU[2], LU[2], BU[2], LI[2], EU[2];
    uint32_t F[V / 4], C[V / 4];
};
template <int V, Part PART>
__device__ __forceinline__ void process_group(PixelAcc& a, const Group16<V>& q, const PixelIn& px, float dscale, float* lum,
                                              uint32_t* key) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
        SampleIn in;
        for (int c = 0; c < 3; ++c) {
            in.root[c] = fabsf(h2f(q.L[c].at(i)));
            in.L[c] = sq(in.root[c]);
            in.n[c] = snorm16(int16_t(q.N[c].at(i)));
            in.alb[c] = 0.0f;
        }
        in.d = h2f(q.D.at(i)) * dscale;
        for (int c = 0; c < 2; ++c) in.pu[c] = unorm16(q.PU[c].at(i));
        in.bins = bin2d_q(q.BU[0].at(i), q.BU[1].at(i)) | (bin2d_q(q.LU[0].at(i), q.LU[1].at(i)) << 5) |
                  (bin2d_q(q.LI[0].at(i), q.LI[1].at(i)) << 10) | (bin2d_q(q.EU[0].at(i), q.EU[1].at(i)) << 15);
        in.f = uint8_t(q.F[i >> 2] >> (8 * (i & 3)));
        in.cat = uint8_t(q.C[i >> 2] >> (8 * (i & 3)));
        process_sample<true, PART>(a, in, false, px.palb, px.prep, px.plane_mask, px.fx, px.fy, px.bin_pixels, lum[i], key[i]);
    }
}
template <int V>
__device__ __forceinline__ void store_prep(const GridPrep& gp, int64_t k, const float* lum, const uint32_t* key) {
#pragma unroll
    for (int i = 0; i < V; i += 4) {
        *reinterpret_cast<float4*>(gp.lum + k + i) = make_float4(lum[i], lum[i + 1], lum[i + 2], lum[i + 3]);
        *reinterpret_cast<uint4*>(gp.key + k + i) = make_uint4(key[i], key[i + 1], key[i + 2], key[i + 3]);
    }
}

// VEC4: every present plane is 16-byte aligned at the pixel's first sample and the pixel's
// sample count is a multiple of 4, so each plane is read four samples per load. COMPACT: the
// planes are rpd_sample_soa16's (s.c16), decoded to float here; WIDE reads them 8 samples (16
// bytes) per load. PART: what the thread keeps of its pixel. The two parts of a split pixel both read
// its count p.n, which the luminance part writes: the block's 64 colour threads arrive at a barrier with the count in
// hand, and its 64 luminance threads wait there before they store, each thread once (local >= count: no
// pixel). The colour part, which never waits, has arrived long before. Per-pixel counts of 4 over 1280x720: 245 us; 255
// with the whole block meeting at the walk's end, 234 without any order.
template <bool VEC4, bool COMPACT, bool WIDE, Part PART>
__device__ __forceinline__ void accumulate_pixel(const PixelPlanes& p, const DeviceSamples& s, const int64_t* offsets, int spp,
                                                 int64_t local, int64_t first, int64_t count, const GridPrep& gp, int fresh) {
    constexpr bool colour = PART != kLuminance, lumi = PART != kColour, split = PART != kWhole;
    const bool mine = !split || local < count;
    const int64_t idx = first + local;
    const int64_t k0 = mine ? sample_offset(offsets, spp, local) : 0, k1 = mine ? sample_offset(offsets, spp, local + 1) : 0;
    const bool prep = gp.lum != nullptr;
    const bool has_pu = COMPACT ? s.c16.pixel_u[0] != nullptr : s.pixel_u[0] != nullptr;
    const bool has_lu = COMPACT ? s.c16.lens_u[0] != nullptr : s.lens_u[0] != nullptr;
    const bool has_bu = COMPACT ? s.c16.brdf_u[0] != nullptr : s.brdf_u[0] != nullptr;
    const bool has_li = COMPACT ? s.c16.light_u[0] != nullptr : s.light_u[0] != nullptr;
    const bool has_eu = COMPACT ? s.c16.env_u[0] != nullptr : s.env_u[0] != nullptr;
    PixelIn px{};
    px.prep = prep;
    px.plane_mask = plane_mask_of(has_pu, has_lu, has_bu, has_li, has_eu);
    px.fx = float(idx % gp.width);
    px.fy = float(idx / gp.width);
    px.bin_pixels = gp.bin_pixels;
    PixelAcc a;
    // the class sums' local array, addressed through an offset the compiler cannot fold, so that
    // it stays in local memory instead of registers
    float cls_local[kClasses * 5];
    a.cs = cls_local + (uint32_t(gp.width) >> 31);  // the width is positive: offset 0
    acc_init(a);
    if (k0 == k1) {
        if (mine && prep && lumi) acc_store_empty(gp, idx);
        if (!split) return;
    }
    const bool some = !split || k0 != k1;
    // fresh: the frame's first push over every pixel, whose statistics the frame start zeroed
    if (fresh) acc_zero(a);
    else if (some) acc_load<PART>(a, p, idx);
    // (the count is an operand: it has arrived)
    if constexpr (PART == kColour) asm volatile("barrier.cta.arrive 1, 128;" : "+r"(a.n));
    px.per_sample_albedo = !COMPACT && s.albedo[0] != nullptr;
    if (some) load_pixel_albedo<COMPACT>(px, s, local);
    const bool dims = prep && lumi;  // the random dimensions are only read for the grid pass

    if (COMPACT) {
        const DeviceSamples16& h = s.c16;
        const float dscale = h.depth_scale;
        if (VEC4) {
            // V samples per plane load: 8 (16-byte loads) when WIDE, else 4 (8-byte loads)
            constexpr int V = WIDE ? 8 : 4;
            auto ldv = [](const void* ptr, int64_t k) {
                Words<V> r;
                if constexpr (WIDE) {
                    const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(ptr) + k);
                    r.w[0] = v.x;
                    r.w[1] = v.y;
                    r.w[2] = v.z;
                    r.w[3] = v.w;
                } else {
                    const uint2 v = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(ptr) + k);
                    r.w[0] = v.x;
                    r.w[1] = v.y;
                }
                return r;
            };
            for (int64_t k = k0; k < k1; k += V) {
                Group16<V> q;
                const Words<V> z{};
                for (int c = 0; c < 3; ++c) {
                    q.L[c] = ldv(h.sqrt_radiance[c], k);
                    q.N[c] = colour ? ldv(h.normal[c], k) : z;
                }
                q.D = lumi ? ldv(h.depth, k) : z;
                for (int c = 0; c < 2; ++c) {
                    q.PU[c] = (dims && has_pu) ? ldv(h.pixel_u[c], k) : z;
                    q.LU[c] = (dims && has_lu) ? ldv(h.lens_u[c], k) : z;
                    q.BU[c] = (dims && has_bu) ? ldv(h.brdf_u[c], k) : z;
                    q.LI[c] = (dims && has_li) ? ldv(h.light_u[c], k) : z;
                    q.EU[c] = (dims && has_eu) ? ldv(h.env_u[c], k) : z;
                }
                for (int i = 0; i < V / 4; ++i) {
                    q.F[i] = *reinterpret_cast<const uint32_t*>(s.flags + k + 4 * i);
                    q.C[i] = (dims && s.category) ? *reinterpret_cast<const uint32_t*>(s.category + k + 4 * i) : 0u;
                }
                float lum[V];
                uint32_t key[V];
                process_group<V, PART>(a, q, px, dscale, lum, key);
                if (dims) store_prep<V>(gp, k, lum, key);
            }
        } else {
            for (int64_t k = k0; k < k1; ++k) {
                SampleIn in;
                for (int c = 0; c < 3; ++c) {
                    in.root[c] = fabsf(h2f(h.sqrt_radiance[c][k]));
                    in.L[c] = sq(in.root[c]);
                    in.n[c] = colour ? snorm16(h.normal[c][k]) : 0.0f;
                    in.alb[c] = 0.0f;
                }
                in.d = lumi ? h2f(h.depth[k]) * dscale : 0.0f;
                uint16_t q[4][2];
                for (int c = 0; c < 2; ++c) {
                    in.pu[c] = (dims && has_pu) ? unorm16(h.pixel_u[c][k]) : 0.0f;
                    q[0][c] = (dims && has_lu) ? h.lens_u[c][k] : uint16_t(0);
                    q[1][c] = (dims && has_bu) ? h.brdf_u[c][k] : uint16_t(0);
                    q[2][c] = (dims && has_li) ? h.light_u[c][k] : uint16_t(0);
                    q[3][c] = (dims && has_eu) ? h.env_u[c][k] : uint16_t(0);
                }
                in.bins = bin2d_q(q[1][0], q[1][1]) | (bin2d_q(q[0][0], q[0][1]) << 5) |
                          (bin2d_q(q[2][0], q[2][1]) << 10) | (bin2d_q(q[3][0], q[3][1]) << 15);
                in.f = s.flags[k];
                in.cat = (dims && s.category) ? s.category[k] : 0;
                float lum;
                uint32_t key;
                process_sample<true, PART>(a, in, false, px.palb, prep, px.plane_mask, px.fx, px.fy, px.bin_pixels, lum, key);
                if (dims) {
                    gp.lum[k] = lum;
                    gp.key[k] = key;
                    if (gp.col) gp.col[k] = uint16_t(idx % gp.width);
                }
            }
        }
    } else if (VEC4) {
        for (int64_t k = k0; k < k1; k += 4) {
            Quad32 q;
            const float4 z4 = make_float4(0, 0, 0, 0);
            for (int c = 0; c < 3; ++c) {
                q.L[c] = ld4(s.radiance[c], k);
                q.N[c] = colour ? ld4(s.normal[c], k) : z4;
                q.A[c] = colour && px.per_sample_albedo ? ld4(s.albedo[c], k) : z4;
            }
            q.D = lumi ? ld4(s.depth, k) : z4;
            for (int c = 0; c < 2; ++c) {
                q.PU[c] = (dims && s.pixel_u[0]) ? ld4(s.pixel_u[c], k) : z4;
                q.LU[c] = (dims && s.lens_u[0]) ? ld4(s.lens_u[c], k) : z4;
                q.BU[c] = (dims && s.brdf_u[0]) ? ld4(s.brdf_u[c], k) : z4;
                q.LI[c] = (dims && s.light_u[0]) ? ld4(s.light_u[c], k) : z4;
                q.EU[c] = (dims && s.env_u[0]) ? ld4(s.env_u[c], k) : z4;
            }
            q.F = *reinterpret_cast<const uint32_t*>(s.flags + k);
            q.C = (dims && s.category) ? *reinterpret_cast<const uint32_t*>(s.category + k) : 0u;
            float lum[4];
            uint32_t key[4];
            process_quad<PART>(a, q, px, lum, key);
            if (dims) store_prep<4>(gp, k, lum, key);
        }
    } else {
        for (int64_t k = k0; k < k1; ++k) {
            SampleIn in;
            for (int c = 0; c < 3; ++c) {
                in.L[c] = s.radiance[c][k];
                in.n[c] = colour ? s.normal[c][k] : 0.0f;
                in.alb[c] = colour && px.per_sample_albedo ? s.albedo[c][k] : 0.0f;
            }
            in.d = lumi ? s.depth[k] : 0.0f;
            for (int c = 0; c < 2; ++c) {
                in.pu[c] = (dims && s.pixel_u[0]) ? s.pixel_u[c][k] : 0.0f;
                in.lu[c] = (dims && s.lens_u[0]) ? s.lens_u[c][k] : 0.0f;
                in.bu[c] = (dims && s.brdf_u[0]) ? s.brdf_u[c][k] : 0.0f;
                in.liu[c] = (dims && s.light_u[0]) ? s.light_u[c][k] : 0.0f;
                in.eu[c] = (dims && s.env_u[0]) ? s.env_u[c][k] : 0.0f;
            }
            in.f = s.flags[k];
            in.cat = (dims && s.category) ? s.category[k] : 0;
            float lum;
            uint32_t key;
            process_sample<false, PART>(a, in, px.per_sample_albedo, px.palb, prep, px.plane_mask, px.fx, px.fy, px.bin_pixels, lum, key);
            if (dims) {
                gp.lum[k] = lum;
                gp.key[k] = key;
                if (gp.col) gp.col[k] = uint16_t(idx % gp.width);
            }
        }
    }

    if constexpr (PART == kLuminance) asm volatile("barrier.cta.sync 1, 128;" ::: "memory");
    if (split && !some) return;
    acc_store<PART>(a, p, gp, idx, prep);
}

// MINB: resident blocks per SM the register allocation must allow. SPLIT: two warps of a block share 32
// pixels, one part each. The general form is bound by the latency of its loads and of the chain of
// updates (40 % of the issue slots at 12 warps per SM, 156 registers a thread). Single samples per load
// leave registers to halve: 16 warps' worth of pixels in 32 warps, 1283x717x6 168 -> 134 us, compact
// 1920x1080x6 267 -> 226, adaptive counts over 1280x720 469 -> 426 us per frame. Four samples
// per load do not: 24 split warps read more lines at a time than L1 holds (1920x1080x16 0.64 -> 0.72 ms).
template <bool VEC4, bool COMPACT, bool WIDE, int MINB, bool SPLIT>
__global__ void __launch_bounds__(128, MINB) k_accumulate_pixels(PixelPlanes p, DeviceSamples s, const int64_t* offsets,
                                                                 int spp, int64_t first, int64_t count, GridPrep gp, int fresh) {
    if constexpr (SPLIT) {
        const int64_t local = int64_t(blockIdx.x) * 64 + (threadIdx.x & 63);
        if (threadIdx.x < 64) accumulate_pixel<VEC4, COMPACT, WIDE, kLuminance>(p, s, offsets, spp, local, first, count, gp, fresh);
        else accumulate_pixel<VEC4, COMPACT, WIDE, kColour>(p, s, offsets, spp, local, first, count, gp, fresh);
    } else {
        const int64_t local = int64_t(blockIdx.x) * 128 + threadIdx.x;
        if (local >= count) return;
        accumulate_pixel<VEC4, COMPACT, WIDE, kWhole>(p, s, offsets, spp, local, first, count, gp, fresh);
    }
}

// ---- the statistics pass on staged rows ------------------------------------------------------------
//
// For uniform pushes of many samples per pixel: a plane is a matrix of one row of spp samples per pixel.
// A block owns 32 pixels and fetches, into one of two buffers in turn, 32 bytes of their rows of
// every plane into shared memory, one tensor copy per plane (cp.async.bulk.tensor, completion on an mbarrier).
// Its five warps split a pixel's quantities, which are independent chains over its samples: one
// warp per colour channel (colour and square-root mean and variance, radiance, normal and albedo
// sums), one for the luminance statistics and the grid pass's class sums, one for the sample keys;
// lane i of each is pixel i, walking the samples in order with the operations of
// k_accumulate_pixels, so the results are the same bits. A thread that walks all of a pixel's planes
// has a line of each plane in flight per pixel, 61 KB a warp from 64 compact samples on: the lines
// of 12 warps on each SM do not survive in L2 until their next sectors are read (DRAM read 3.5 times the planes); with
// a pixel's work on five warps a quarter of the pixels keeps an SM busy. 2048x1152x64: 4.22 -> 2.7 ms
// compact; 1920x1080x64: 7.1 -> 2.25 ms FP32 (3.6 TB/s).
struct RowsArgs {
    CUtensorMap map[20];
    int planes;                      // present planes, in the order of the offsets below
    int albedo, pu, lu, bu, li, eu;  // a plane group's byte offset in a buffer, or -1
};
constexpr int kRowRoles = 5;
constexpr int kRowPixels = 32;
constexpr int kRowBytes = 32;  // of a pixel's row per step

// The luminance warp's state (class_add's fields).
struct LumAcc {
    float mean, m2, dep;
    int n, hits, nsamples;
    PatternSums pt[kPatterns];
    bool dev;
    float* cs;
};

// x / n and y / n, IEEE quotients (the compact pass's by one reciprocal where that is exact)
template <bool COMPACT>
__device__ __forceinline__ void quotients(float x, float y, int n, float& qx, float& qy) {
    const float fn = float(n);
    if (COMPACT && n < (1 << 23) && markstein_ok(x) && markstein_ok(y)) {
        const float rn = 1.0f / fn;
        qx = div_markstein(x, fn, rn);
        qy = div_markstein(y, fn, rn);
    } else {
        qx = x / fn;
        qy = y / fn;
    }
}

// w[i] of a small register array by selects (i is a loop counter the compiler does not unroll)
template <int N>
__device__ __forceinline__ uint32_t pick(const uint32_t (&w)[N], int i) {
    uint32_t r = w[0];
#pragma unroll
    for (int k = 1; k < N; ++k) r = i == k ? w[k] : r;
    return r;
}

template <bool COMPACT>
__global__ void __launch_bounds__(kRowRoles * 32, 4)
    k_accumulate_rows(PixelPlanes p, DeviceSamples s, int32_t spp, int64_t first, int64_t count, GridPrep gp, int fresh,
                      const __grid_constant__ RowsArgs ra) {
    constexpr int ES = COMPACT ? 2 : 4;
    constexpr int RB = kRowBytes;
    constexpr int CH = RB / ES;        // samples per step
    constexpr int V = 4;               // samples per group
    constexpr int PLANE = kRowPixels * RB;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ uint8_t s_pflags[kRowPixels];
    __shared__ int s_fail;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (a block's warps go to the SM's schedulers by index: the roles rotate over the blocks)
    const int role = (warp + int(blockIdx.x)) % kRowRoles;
    const int64_t row0 = int64_t(blockIdx.x) * kRowPixels;
    const uint32_t pad = (1024u - (smem_addr(smem_raw) & 1023u)) & 1023u;
    const int stage = (ra.planes * PLANE + 1023) & ~1023;
    unsigned char* buf = smem_raw + pad;
    const int steps = spp / CH;
    auto issue = [&](int c) {  // warp 0: lane 0 arms the barrier, lanes 0 .. planes-1 issue one plane's copy each
        const uint32_t bar = smem_addr(&bars[c & 1]);
        if (lane == 0) mbar_expect_tx(bar, uint32_t(ra.planes) * PLANE);
        __syncwarp();
        if (lane < ra.planes)
            tma_load_2d(smem_addr(buf + (c & 1) * stage + lane * PLANE), &ra.map[lane], c * CH, int(row0), bar);
    };
    if (threadIdx.x == 0) {
        mbar_init(smem_addr(&bars[0]), 1);
        mbar_init(smem_addr(&bars[1]), 1);
        s_fail = 0;
    }
    __syncthreads();
    if (warp == 0) {
        issue(0);
        if (steps > 1) issue(1);
    }
    const int64_t local = row0 + lane;
    const bool mine = local < count;
    const int64_t idx = first + local;
    const int64_t k0 = local * spp;
    const bool prep = gp.lum != nullptr;
    // step c's samples are in place; false: they did not arrive in time, the block gives up
    auto arrived = [&](int c) { return mbar_wait_bounded(smem_addr(&bars[c & 1]), (c >> 1) & 1); };
    auto done = [&](int c, bool ok) -> bool {  // step c is read: its buffer takes step c + 2
        if (!ok) s_fail = 1;
        __syncthreads();
        if (s_fail) {
            if (threadIdx.x == 0) atomicAdd(p.counters + RPD_COUNTER_DEVICE_WAIT_TIMEOUTS, 1ull);
            arrived(c);  // let the copies land (bounded) before the shared memory is released
            if (c + 1 < steps) arrived(c + 1);
            return false;
        }
        if (warp == 0 && c + 2 < steps) issue(c + 2);
        return true;
    };
    auto flag_words = [&](const uint8_t* plane, int c, uint32_t* w) {
#pragma unroll
        for (int i = 0; i < CH / 4; ++i) w[i] = mine && plane ? *reinterpret_cast<const uint32_t*>(plane + k0 + c * CH + 4 * i) : 0u;
    };
    // group q of the pixel's row in the plane at byte offset off of step c
    auto chunk = [&](int c, int off, int q) -> uint4 {
        const unsigned char* at = buf + (c & 1) * stage + off + lane * RB;
        if constexpr (COMPACT) {
            const uint2 v = *reinterpret_cast<const uint2*>(at + 16 * swizzled_chunk<RB>(q >> 1, lane) + 8 * (q & 1));
            return make_uint4(v.x, v.y, 0u, 0u);
        } else {
            return *reinterpret_cast<const uint4*>(at + 16 * swizzled_chunk<RB>(q, lane));
        }
    };
    // sample i of a chunk: its float (FP32 planes), or its 16 bits
    auto f32 = [](const uint4& v, int i) { return __uint_as_float(i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w); };
    auto u16 = [](const uint4& v, int i) {
        const uint32_t w = (i >> 1) == 0 ? v.x : (i >> 1) == 1 ? v.y : (i >> 1) == 2 ? v.z : v.w;
        return uint16_t(w >> (16 * (i & 1)));
    };
    auto finite = [&](const uint4* L, int i) {
        if constexpr (COMPACT) {
            bool ok = true;
            for (int d = 0; d < 3; ++d) ok = ok && (u16(L[d], i) & 0x7c00u) != 0x7c00u;
            return ok;
        } else {
            return finite3(f32(L[0], i), f32(L[1], i), f32(L[2], i));
        }
    };

    if (role < 3) {  // colour channel `role`
        float cm = 0.0f, sm = 0.0f, sq_ = 0.0f, rad = 0.0f, nor = 0.0f, alb = 0.0f, palb = 0.0f;
        int n = 0;
        const bool per_sample = !COMPACT && ra.albedo >= 0;
        if (mine) {
            if (!fresh) {
                n = p.n[idx];
                cm = p.color_mean[role][idx];
                sm = p.sqrt_mean[role][idx];
                sq_ = p.sqrt_sq[role][idx];
                rad = p.radiance[role][idx];
                nor = p.normal[role][idx];
                alb = p.albedo[role][idx];
            }
            if (COMPACT) {
                if (s.c16.pixel_albedo[0]) palb = h2f(s.c16.pixel_albedo[role][local]);
            } else if (!per_sample && s.pixel_albedo[0]) {
                palb = s.pixel_albedo[role][local];
            }
        }
        for (int c = 0; c < steps; ++c) {
            uint32_t F[CH / 4];
            flag_words(s.flags, c, F);
            const bool ok = arrived(c);
            if (ok && mine) {
#pragma unroll 1
                for (int q = 0; q < CH / V; ++q) {
                    uint4 L[3];
                    for (int d = 0; d < 3; ++d) L[d] = chunk(c, d * PLANE, q);
                    const uint4 N = chunk(c, (3 + role) * PLANE, q);
                    uint4 A = make_uint4(0u, 0u, 0u, 0u);
                    if (per_sample) A = chunk(c, ra.albedo + role * PLANE, q);
                    uint32_t f4[V / 4];
                    for (int i = 0; i < V / 4; ++i) f4[i] = pick(F, q * (V / 4) + i);
                    const uint4 mineL = role == 0 ? L[0] : role == 1 ? L[1] : L[2];
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        const uint32_t f = f4[i >> 2] >> (8 * (i & 3));
                        if (f & RPD_SAMPLE_HIT) {  // main.cpp:572-576
                            nor += COMPACT ? snorm16(int16_t(u16(N, i))) : f32(N, i);
                            alb += per_sample ? f32(A, i) : palb;
                        }
                        if (!finite(L, i)) continue;  // main.cpp:707
                        float v, root;
                        if constexpr (COMPACT) {
                            root = fabsf(h2f(u16(mineL, i)));
                            v = sq(root);
                        } else {
                            v = f32(mineL, i);
                            root = sqrtf(fmaxs(0.0f, v));
                        }
                        // accumulate_sample (core/stats.h:25-41), this channel
                        ++n;
                        const float cd = v - cm, sd = root - sm;
                        float qc, qs;
                        quotients<COMPACT>(cd, sd, n, qc, qs);
                        cm += qc;
                        sm += qs;
                        sq_ += sd * (root - sm);
                        rad += v;
                    }
                }
            }
            if (!done(c, ok)) return;
        }
        if (mine) {
            p.color_mean[role][idx] = cm;
            p.sqrt_mean[role][idx] = sm;
            p.sqrt_sq[role][idx] = sq_;
            p.radiance[role][idx] = rad;
            p.normal[role][idx] = nor;
            p.albedo[role][idx] = alb;
        }
        __syncthreads();
    } else if (role == 3) {  // luminance, depth, counts, class sums
        const uint8_t mask = plane_mask_of(ra.pu >= 0, ra.lu >= 0, ra.bu >= 0, ra.li >= 0, ra.eu >= 0);
        LumAcc a{};
        float cls_local[kClasses * 5];
        a.cs = cls_local + (uint32_t(gp.width) >> 31);  // in local memory (k_accumulate_pixels)
        if (mine && !fresh) {
            a.mean = p.mean[idx];
            a.m2 = p.square_diff[idx];
            a.n = p.n[idx];
            a.dep = p.depth[idx];
            a.hits = p.hit_count[idx];
            a.nsamples = p.sample_count[idx];
        }
        for (int c = 0; c < steps; ++c) {
            uint32_t F[CH / 4];
            flag_words(s.flags, c, F);
            const bool ok = arrived(c);
            if (ok && mine) {
#pragma unroll 1
                for (int q = 0; q < CH / V; ++q) {
                    uint4 L[3];
                    for (int d = 0; d < 3; ++d) L[d] = chunk(c, d * PLANE, q);
                    const uint4 D = chunk(c, 6 * PLANE, q);
                    uint32_t f4[V / 4];
                    for (int i = 0; i < V / 4; ++i) f4[i] = pick(F, q * (V / 4) + i);
                    float lum_out[V];
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        const uint32_t f = f4[i >> 2] >> (8 * (i & 3));
                        if (f & RPD_SAMPLE_HIT) {
                            ++a.hits;
                            a.dep += COMPACT ? h2f(u16(D, i)) * s.c16.depth_scale : f32(D, i);
                        }
                        lum_out[i] = __int_as_float(0x7fc00000);  // NaN: dropped by the grid pass
                        if (!finite(L, i)) continue;
                        float v[3];
                        for (int d = 0; d < 3; ++d) v[d] = COMPACT ? sq(fabsf(h2f(u16(L[d], i)))) : f32(L[d], i);
                        const float lum = luminance(v[0], v[1], v[2]);
                        const float delta = lum - a.mean;
                        ++a.n;
                        float qd, unused;
                        quotients<COMPACT>(delta, delta, a.n, qd, unused);
                        a.mean += qd;
                        a.m2 += delta * (lum - a.mean);
                        ++a.nsamples;
                        lum_out[i] = lum;
                        if (prep) class_add(a, uint8_t(f) & mask, lum);
                    }
                    if (prep) {
#pragma unroll
                        for (int i = 0; i < V; i += 4)
                            *reinterpret_cast<float4*>(gp.lum + k0 + c * CH + q * V + i) =
                                make_float4(lum_out[i], lum_out[i + 1], lum_out[i + 2], lum_out[i + 3]);
                    }
                }
            }
            if (!done(c, ok)) return;
        }
        if (mine) {
            p.mean[idx] = a.mean;
            p.square_diff[idx] = a.m2;
            p.n[idx] = a.n;
            p.depth[idx] = a.dep;
            p.hit_count[idx] = a.hits;
            p.sample_count[idx] = a.nsamples;
        }
        __syncthreads();  // the key warp's pixel flags
        if (mine && prep) store_classes(a, gp, idx, s_pflags[lane]);
    } else {  // keys and pixel flags
        const uint8_t mask = plane_mask_of(ra.pu >= 0, ra.lu >= 0, ra.bu >= 0, ra.li >= 0, ra.eu >= 0);
        uint8_t pflags = kPixUniform;
        const float fx = float(idx % gp.width), fy = float(idx / gp.width);
        for (int c = 0; c < steps; ++c) {
            uint32_t F[CH / 4], C[CH / 4];
            flag_words(s.flags, c, F);
            flag_words(s.category, c, C);
            const bool ok = arrived(c);
            if (ok && mine && prep) {
#pragma unroll 1
                for (int q = 0; q < CH / V; ++q) {
                    uint4 L[3], U[5][2];
                    const int offs[5] = {ra.pu, ra.bu, ra.lu, ra.li, ra.eu};
                    for (int d = 0; d < 3; ++d) L[d] = chunk(c, d * PLANE, q);
#pragma unroll
                    for (int g = 0; g < 5; ++g)
                        for (int d = 0; d < 2; ++d)
                            U[g][d] = offs[g] >= 0 ? chunk(c, offs[g] + d * PLANE, q) : make_uint4(0u, 0u, 0u, 0u);
                    uint32_t f4[V / 4], c4[V / 4];
                    for (int i = 0; i < V / 4; ++i) {
                        f4[i] = pick(F, q * (V / 4) + i);
                        c4[i] = pick(C, q * (V / 4) + i);
                    }
                    uint32_t key[V];
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        const uint8_t fm = uint8_t(f4[i >> 2] >> (8 * (i & 3))) & mask;
                        key[i] = kKeyNone;
                        if (!finite(L, i)) continue;
                        SampleIn in;
                        in.cat = uint8_t(c4[i >> 2] >> (8 * (i & 3)));
                        for (int d = 0; d < 2; ++d) {
                            if constexpr (COMPACT) {
                                in.pu[d] = unorm16(u16(U[0][d], i));
                            } else {
                                in.pu[d] = f32(U[0][d], i);
                                in.bu[d] = f32(U[1][d], i);
                                in.lu[d] = f32(U[2][d], i);
                                in.liu[d] = f32(U[3][d], i);
                                in.eu[d] = f32(U[4][d], i);
                            }
                        }
                        if constexpr (COMPACT) {
                            in.bins = 0u;
#pragma unroll
                            for (int g = 0; g < 4; ++g)
                                in.bins |= bin2d_q(u16(U[g + 1][0], i), u16(U[g + 1][1], i)) << (5 * g);
                        }
                        key[i] = sample_key<COMPACT>(in, fm);
                        screen_flags(in, fm, fx, fy, gp.bin_pixels, pflags);
                    }
#pragma unroll
                    for (int i = 0; i < V; i += 4)
                        *reinterpret_cast<uint4*>(gp.key + k0 + c * CH + q * V + i) =
                            make_uint4(key[i], key[i + 1], key[i + 2], key[i + 3]);
                }
            }
            if (!done(c, ok)) return;
        }
        s_pflags[lane] = pflags;
        __syncthreads();
    }
}

// Valid-flag bit each dependency needs, and whether it bins the screen position.
__device__ __forceinline__ uint8_t dep_flag(int d) {
    switch (d) {
    case D_PIXEL: return 0;
    case D_BRDF: case D_SCREEN_BRDF: return RPD_SAMPLE_BRDF_VALID;
    case D_LENS: case D_SCREEN_LENS: return RPD_SAMPLE_LENS_VALID;
    case D_LIGHT_UV: case D_SCREEN_LIGHT_UV: return RPD_SAMPLE_LIGHT_VALID;
    case D_ENV: case D_SCREEN_ENV: return RPD_SAMPLE_ENV_VALID;
    case D_LIGHT_SELECT: case D_SCREEN_LIGHT_SELECT: return RPD_SAMPLE_LIGHT_SELECT_VALID;
    default: return RPD_SAMPLE_RR_VALID;
    }
}
__device__ __forceinline__ bool dep_is_screen(int d) {
    return d == D_PIXEL || d == D_SCREEN_BRDF || d == D_SCREEN_LENS || d == D_SCREEN_LIGHT_UV ||
           d == D_SCREEN_ENV || d == D_SCREEN_LIGHT_SELECT || d == D_SCREEN_RR;
}

// Dependency2D::add bin (core/stats.h:166-168)
__device__ __forceinline__ int bin2d(float u, float v) {
    const int x = iclamps(int(u * 4.0f), 0, 3);
    const int z = iclamps(int(v * 4.0f), 0, 3);
    return z * 4 + x;
}

__global__ void __launch_bounds__(128) k_grid_ordered(Geometry g, double* pass_grid, DeviceSamples s,
                                                      const int64_t* offsets, int32_t spp, int64_t first,
                                                      int64_t count) {
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= g.nn * kDeps) return;
    const int node = int(t / kDeps);
    const int d = int(t % kDeps);
    const int nx = node % g.nodes_x, ny = node / g.nodes_x;
    const uint8_t need = dep_flag(d);
    const bool screen = dep_is_screen(d);
    const int bins = (d == D_RR) ? 2 : 16;
    // a NULL plane never validates its dependency
    const float* const* dims = nullptr;
    switch (d) {
    case D_BRDF: dims = s.brdf_u; break;
    case D_LENS: dims = s.lens_u; break;
    case D_LIGHT_UV: dims = s.light_u; break;
    case D_ENV: dims = s.env_u; break;
    default: break;
    }
    if (screen && !s.pixel_u[0]) return;
    if (dims && !dims[0]) return;
    if ((d == D_SCREEN_BRDF && !s.brdf_u[0]) || (d == D_SCREEN_LENS && !s.lens_u[0]) ||
        (d == D_SCREEN_LIGHT_UV && !s.light_u[0]) || (d == D_SCREEN_ENV && !s.env_u[0]))
        return;

    double* acc = pass_grid + int64_t(node) * kDeps * kDepStride + d * kDepStride;
    double wbin[16], ybin[16];
    for (int b = 0; b < 16; ++b) {
        wbin[b] = acc[b];
        ybin[b] = acc[16 + b];
    }
    double w_sum = acc[32], w2_sum = acc[33], y_sum = acc[34], y2_sum = acc[35];

    const float half_support = 0.5f * float(g.support);
    const float inv_dummy = 0.0f;
    (void)inv_dummy;
    // pixels whose bilinear footprint can reach this node
    const int xlo = imaxs(0, (nx - 1) * g.step - 1), xhi = imins(g.w - 1, (nx + 1) * g.step + 1);
    const int ylo = imaxs(0, (ny - 1) * g.step - 1), yhi = imins(g.h - 1, (ny + 1) * g.step + 1);
    for (int y = ylo; y <= yhi; ++y) {
        const float gy = float(y) / float(g.step);
        const int y0 = iclamps(int(floorf(gy)), 0, g.nodes_y - 1);
        const int y1 = imins(y0 + 1, g.nodes_y - 1);
        if (y0 != ny && y1 != ny) continue;
        const float ty = fclamps(gy - float(y0), 0.0f, 1.0f);
        for (int x = xlo; x <= xhi; ++x) {
            const int64_t idx = int64_t(y) * g.w + x;
            if (idx < first || idx >= first + count) continue;
            const float gx = float(x) / float(g.step);
            const int x0 = iclamps(int(floorf(gx)), 0, g.nodes_x - 1);
            const int x1 = imins(x0 + 1, g.nodes_x - 1);
            if (x0 != nx && x1 != nx) continue;
            const float tx = fclamps(gx - float(x0), 0.0f, 1.0f);
            // the four entries of main.cpp:341-346, in order; keep those naming this node
            float we[4];
            int ne = 0;
            if (x0 == nx && y0 == ny) we[ne++] = (1.0f - tx) * (1.0f - ty);
            if (x1 == nx && y0 == ny) we[ne++] = tx * (1.0f - ty);
            if (x0 == nx && y1 == ny) we[ne++] = (1.0f - tx) * ty;
            if (x1 == nx && y1 == ny) we[ne++] = tx * ty;
            bool any = false;
            for (int e = 0; e < ne; ++e) any |= we[e] > 1e-8f;
            if (!any) continue;
            const int64_t local = idx - first;
            const int64_t k0 = sample_offset(offsets, spp, local);
            const int64_t k1 = sample_offset(offsets, spp, local + 1);
            const float support_left = float(nx * g.step) - half_support;
            const float support_top = float(ny * g.step) - half_support;
            for (int64_t k = k0; k < k1; ++k) {
                uint8_t f = s.flags ? s.flags[k] : 0;
                if (!s.pixel_u[0]) f &= uint8_t(~RPD_SAMPLE_PIXEL_VALID);
                if (!s.lens_u[0]) f &= uint8_t(~RPD_SAMPLE_LENS_VALID);
                if (!s.brdf_u[0]) f &= uint8_t(~RPD_SAMPLE_BRDF_VALID);
                if (!s.light_u[0]) f &= uint8_t(~RPD_SAMPLE_LIGHT_VALID);
                if (!s.env_u[0]) f &= uint8_t(~RPD_SAMPLE_ENV_VALID);
                const bool pixel_valid = (f & RPD_SAMPLE_PIXEL_VALID) != 0;
                if (screen && !pixel_valid) continue;
                if (need && !(f & need)) continue;
                // main.cpp:330 — samples without any captured dimension are skipped
                if (!(f & (RPD_SAMPLE_PIXEL_VALID | RPD_SAMPLE_LENS_VALID | RPD_SAMPLE_LIGHT_SELECT_VALID |
                           RPD_SAMPLE_BRDF_VALID | RPD_SAMPLE_LIGHT_VALID | RPD_SAMPLE_ENV_VALID |
                           RPD_SAMPLE_RR_VALID)))
                    continue;
                const float r = s.radiance[0][k], gch = s.radiance[1][k], b = s.radiance[2][k];
                if (!finite3(r, gch, b)) continue;
                const float lum = luminance(r, gch, b);
                int bin;
                if (screen) {
                    const float su = fclamps((float(x) + s.pixel_u[0][k] - support_left) / float(g.support), 0.0f, 1.0f);
                    const float sv = fclamps((float(y) + s.pixel_u[1][k] - support_top) / float(g.support), 0.0f, 1.0f);
                    bin = bin2d(su, sv);
                } else if (d == D_LIGHT_SELECT) {
                    bin = int(s.category[k] & RPD_CATEGORY_LIGHT_INDEX_MASK);
                } else if (d == D_RR) {
                    bin = (s.category[k] & RPD_CATEGORY_RR_SURVIVED) ? 1 : 0;
                } else {
                    bin = bin2d(dims[0][k], dims[1][k]);
                }
                bin = iclamps(bin, 0, bins - 1);
                const double yd = double(lum);
                for (int e = 0; e < ne; ++e) {
                    // BinnedDependency::add (core/stats.h:102-113)
                    if (we[e] <= 1e-8f) continue;
                    const double wd = double(we[e]);
                    wbin[bin] += wd;
                    ybin[bin] += wd * yd;
                    w_sum += wd;
                    w2_sum += wd * wd;
                    y_sum += wd * yd;
                    y2_sum += wd * yd * yd;
                }
            }
        }
    }
    for (int b = 0; b < 16; ++b) {
        acc[b] = wbin[b];
        acc[16 + b] = ybin[b];
    }
    acc[32] = w_sum;
    acc[33] = w2_sum;
    acc[34] = y_sum;
    acc[35] = y2_sum;
}

// float -> double from the bits (the conversion instruction runs on the double-precision pipe,
// 2 per SM per clock); zeros keep their sign, subnormals, infinities and NaN convert as usual.
__device__ __forceinline__ double widen(float f) {
    const uint32_t b = __float_as_uint(f);
    if ((b & 0x7fffffffu) == 0u) return __longlong_as_double(static_cast<long long>(uint64_t(b) << 32));
    const uint32_t e = (b >> 23) & 0xffu;
    if (e == 0u || e == 0xffu) return double(f);
    return __longlong_as_double(static_cast<long long>((uint64_t(b >> 31) << 63) | (uint64_t(e + 896u) << 52) |
                                                       (uint64_t(b & 0x7fffffu) << 29)));
}

// grid += pass (the first pass of a frame: grid = 0 + pass), then clear the pass grid. The pass
// grid holds double-float pairs (hi, lo) in the bytes of each double in the fast grid mode, doubles
// in the exact one. The frame grid takes the first merged pass's form: in the fast mode it stays
// pairs, each merge a double-float addition (about 2^-44 relative, within the grid's 1e-9 of the
// reference) with no double-precision instruction, which GB300 issues at 2 per SM per clock; a
// frame whose passes mix the modes ends in doubles.
enum MergeMode {
    kMergePairsFresh,     // pairs -> the frame's pairs
    kMergePairsPairs,     // frame pairs + pass pairs
    kMergeDoubleFresh,    // doubles -> the frame's doubles
    kMergeDoubleDouble,   // frame doubles + pass doubles
    kMergePairsIntoDouble,  // frame doubles + pass pairs
    kMergeDoubleIntoPairs   // frame pairs + pass doubles -> frame doubles
};
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
    const float s = a.x + b.x;
    const float bb = s - a.x;
    const float e = ((a.x - (s - bb)) + (b.x - bb)) + (a.y + b.y);
    const float h = s + e;
    return make_float2(h, e - (h - s));
}

template <int MODE>
__global__ void k_merge_grid(double* grid, double* pass_grid, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2* gp = reinterpret_cast<float2*>(grid);
    const float2* pp = reinterpret_cast<const float2*>(pass_grid);
    if (MODE == kMergePairsFresh) {
        gp[i] = pp[i];
    } else if (MODE == kMergePairsPairs) {
        gp[i] = pair_add(gp[i], pp[i]);
    } else {
        double v;
        if (MODE == kMergePairsIntoDouble) v = widen(pp[i].x) + widen(pp[i].y);
        else v = pass_grid[i];
        if (MODE == kMergeDoubleFresh) {
            // 0 + v without a double-precision add: the same value, with -0 turned into +0
            const long long b = __double_as_longlong(v);
            grid[i] = __longlong_as_double(b == (long long)0x8000000000000000ull ? 0ll : b);
        } else if (MODE == kMergeDoubleIntoPairs) {
            const float2 g = gp[i];
            grid[i] = (widen(g.x) + widen(g.y)) + v;
        } else {
            grid[i] = grid[i] + v;
        }
    }
    pass_grid[i] = 0.0;
}

// The frame grid as doubles (for reads): pairs widened and added.
__global__ void k_grid_pairs_to_double(const float2* pairs, double* out, int64_t n) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 g = pairs[i];
    out[i] = widen(g.x) + widen(g.y);
}

__global__ void k_feature_cache(PixelPlanes p, int64_t np) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const int hc = p.hit_count[i];
    if (hc > 0) {
        const float h = float(hc);
        float n0 = p.normal[0][i] / h, n1 = p.normal[1][i] / h, n2 = p.normal[2][i] / h;
        const float z = dot3(n0, n1, n2, n0, n1, n2);
        if (z > 1e-8f) {
            // Eigen normalize(): divide by sqrt(squaredNorm) when positive
            const float sn = sqrtf(z);
            n0 = n0 / sn;
            n1 = n1 / sn;
            n2 = n2 / sn;
        }
        p.f_normal[0][i] = n0;
        p.f_normal[1][i] = n1;
        p.f_normal[2][i] = n2;
        p.f_depth[i] = p.depth[i] / h;
        for (int c = 0; c < 3; ++c) p.f_albedo[c][i] = p.albedo[c][i] / h;
    } else {
        for (int c = 0; c < 3; ++c) p.f_normal[c][i] = p.normal[c][i];
        p.f_depth[i] = p.depth[i];
        for (int c = 0; c < 3; ++c) p.f_albedo[c][i] = p.albedo[c][i];
    }
}

__global__ void k_finalize(PixelPlanes p, int64_t np) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const float samples = float(imaxs(1, p.sample_count[i]));
    const float hits = float(imaxs(1, p.hit_count[i]));
    for (int c = 0; c < 3; ++c) p.radiance[c][i] /= samples;
    for (int c = 0; c < 3; ++c) p.albedo[c][i] /= hits;
    float n0 = p.normal[0][i] / hits, n1 = p.normal[1][i] / hits, n2 = p.normal[2][i] / hits;
    const float z = dot3(n0, n1, n2, n0, n1, n2);
    if (z > 1e-8f) {
        const float sn = sqrtf(z);
        n0 = n0 / sn;
        n1 = n1 / sn;
        n2 = n2 / sn;
    }
    p.normal[0][i] = n0;
    p.normal[1][i] = n1;
    p.normal[2][i] = n2;
    p.depth[i] /= hits;
}

}  // namespace

cudaError_t launch_offsets_uniform(Job& j, int64_t count, int32_t spp) {
    KernelScope ks(j, RPD_KERNEL_OFFSETS);
    k_offsets_uniform<<<grid_for(count + 1, 256), 256, 0, j.stream>>>(j.offsets, count, spp);
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_offsets_scan(Job& j, const int32_t* d_counts, int64_t count) {
    KernelScope ks(j, RPD_KERNEL_OFFSETS);
    if (count <= 0) return cudaMemsetAsync(j.offsets, 0, sizeof(int64_t), j.stream);
    const int64_t nblocks = (count + kScanBlock - 1) / kScanBlock;
    // the offsets buffer reserves room for these after offsets[count]
    int64_t* block_sums = j.offsets + (count + 1);
    int64_t* block_maxima = block_sums + (nblocks + 1);
    k_scan_block_sums<<<unsigned(nblocks), kScanBlock, 0, j.stream>>>(d_counts, count, block_sums, block_maxima);
    k_scan_block_offsets<<<1, kScanBlock, 0, j.stream>>>(block_sums, block_maxima, nblocks);
    k_scan_finish<<<unsigned(nblocks), kScanBlock, 0, j.stream>>>(d_counts, count, block_sums, j.offsets);
    j.launches += 3;
    return cudaGetLastError();
}

const int64_t* offsets_count_max(const Job& j, int64_t count) {
    const int64_t nblocks = (count + kScanBlock - 1) / kScanBlock;
    return j.offsets + (count + 1) + (nblocks + 1) + nblocks;
}

// The statistics pass uses no shared memory: its launches ask for the whole unified array as L1,
// which keeps more of the sample sectors a thread reads again a step later (3 % more throughput
// on the served stream, where other requests' kernels share the SMs).
template <bool VEC4, bool COMPACT, bool WIDE, int MINB, bool SPLIT>
cudaError_t run_accumulate(Job& j, const DeviceSamples& s, int32_t spp, int64_t first, int64_t count, const GridPrep& gp, int fresh) {
    static FuncAttribute carveout;
    const cudaError_t e = carveout.at_least(reinterpret_cast<const void*>(&k_accumulate_pixels<VEC4, COMPACT, WIDE, MINB, SPLIT>),
                                            cudaFuncAttributePreferredSharedMemoryCarveout, j.ctx->device,
                                            cudaSharedmemCarveoutMaxL1);
    if (e != cudaSuccess) return e;
    k_accumulate_pixels<VEC4, COMPACT, WIDE, MINB, SPLIT><<<grid_for(count, SPLIT ? 64 : 128), 128, 0, j.stream>>>(
        j.p, s, j.offsets, spp, first, count, gp, fresh);
    return cudaSuccess;
}

// The staged form of the statistics pass, if the push allows it: uniform samples per pixel, 16-byte
// aligned planes, a pixel's row of each plane a multiple of 32 bytes, and enough samples per pixel: up to
// 16 the general form reads each line in few enough steps and executes a third fewer instructions. General / staged
// at 1920x1080: FP32 8 spp 0.33 / 0.45 ms, 16 spp 0.64 / 0.90, 32 spp 3.03 / 1.43, 64 spp 7.1 / 2.25;
// compact 16 spp 0.43 / 0.78, 32 spp 1.08 / 1.39 (1280x720 0.44 / 0.62), 48 spp 4.13 / 1.87. Compact planes without
// the random dimensions (RPD off) are half the bytes again and never take it: 32 spp 0.58 / 0.86, 64 spp 1.08 /
// 1.64, 640x360x256 0.52 / 0.78; FP32 ones are equal (64 spp 1.61 / 1.61). Below a million samples its tensor
// maps' encoding on the host would show.
constexpr int kRowMinSpp = 32, kRowMinSpp16 = 33;
template <bool COMPACT>
cudaError_t run_rows(Job& j, const DeviceSamples& s, int64_t first, int64_t count, const GridPrep& gp, int32_t spp,
                     int fresh, const void* const* planes, RowsArgs& ra) {
    constexpr int ES = COMPACT ? 2 : 4, RB = kRowBytes;
    for (int i = 0; i < ra.planes; ++i) {
        const cudaError_t e = encode_rows_map(&ra.map[i], planes[i], ES, spp, count, RB / ES, kRowPixels);
        if (e != cudaSuccess) return e;
    }
    for (int* off : {&ra.albedo, &ra.pu, &ra.lu, &ra.bu, &ra.li, &ra.eu})
        if (*off >= 0) *off *= kRowPixels * RB;
    const int smem = 1024 + 2 * ((ra.planes * kRowPixels * RB + 1023) & ~1023);
    static FuncAttribute limit;
    const cudaError_t e = limit.at_least(reinterpret_cast<const void*>(&k_accumulate_rows<COMPACT>),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, j.ctx->device, smem);
    if (e != cudaSuccess) return e;
    k_accumulate_rows<COMPACT><<<grid_for(count, kRowPixels), kRowRoles * 32, smem, j.stream>>>(j.p, s, spp, first, count, gp, fresh, ra);
    return cudaGetLastError();
}

cudaError_t launch_accumulate_rows(Job& j, const DeviceSamples& s, int64_t first, int64_t count, const GridPrep& gp,
                                   int32_t spp, int fresh, bool* taken) {
    *taken = false;
    const int es = s.compact ? 2 : 4;
    if (s.compact && !gp.lum) return cudaSuccess;
    if (spp < (s.compact ? kRowMinSpp16 : kRowMinSpp) || (int64_t(spp) * es) % kRowBytes || count * int64_t(spp) < (int64_t(1) << 20) ||
        count > INT32_MAX)
        return cudaSuccess;
    const void* planes[20];
    RowsArgs ra{};
    ra.albedo = ra.pu = ra.lu = ra.bu = ra.li = ra.eu = -1;
    bool ok = (reinterpret_cast<uintptr_t>(s.flags) & 15u) == 0 && (reinterpret_cast<uintptr_t>(s.category) & 15u) == 0 &&
              (!gp.lum || ((reinterpret_cast<uintptr_t>(gp.lum) | reinterpret_cast<uintptr_t>(gp.key)) & 15u) == 0);
    auto add = [&](const void* ptr) {
        ok = ok && ptr && (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0;
        planes[ra.planes++] = ptr;
    };
    auto group = [&](const void* a, const void* b, int* off) {
        if (!a || !gp.lum) return;
        *off = ra.planes;
        add(a);
        add(b);
    };
    if (s.compact) {
        const DeviceSamples16& h = s.c16;
        for (int c = 0; c < 3; ++c) add(h.sqrt_radiance[c]);
        for (int c = 0; c < 3; ++c) add(h.normal[c]);
        add(h.depth);
        group(h.pixel_u[0], h.pixel_u[1], &ra.pu);
        group(h.lens_u[0], h.lens_u[1], &ra.lu);
        group(h.brdf_u[0], h.brdf_u[1], &ra.bu);
        group(h.light_u[0], h.light_u[1], &ra.li);
        group(h.env_u[0], h.env_u[1], &ra.eu);
    } else {
        for (int c = 0; c < 3; ++c) add(s.radiance[c]);
        for (int c = 0; c < 3; ++c) add(s.normal[c]);
        add(s.depth);
        if (s.albedo[0]) {
            ra.albedo = ra.planes;
            for (int c = 0; c < 3; ++c) add(s.albedo[c]);
        }
        group(s.pixel_u[0], s.pixel_u[1], &ra.pu);
        group(s.lens_u[0], s.lens_u[1], &ra.lu);
        group(s.brdf_u[0], s.brdf_u[1], &ra.bu);
        group(s.light_u[0], s.light_u[1], &ra.li);
        group(s.env_u[0], s.env_u[1], &ra.eu);
    }
    if (!ok) return cudaSuccess;
    cudaError_t e = s.compact ? run_rows<true>(j, s, first, count, gp, spp, fresh, planes, ra)
                              : run_rows<false>(j, s, first, count, gp, spp, fresh, planes, ra);
    if (e == cudaErrorNotSupported || e == cudaErrorInvalidValue) {  // no tensor-map encoder: the general form runs
        cudaGetLastError();
        return cudaSuccess;
    }
    *taken = e == cudaSuccess;
    return e;
}

cudaError_t launch_accumulate_pixels(Job& j, const DeviceSamples& s, int64_t first, int64_t count,
                                     const GridPrep& gp, int32_t spp) {
    KernelScope ks(j, RPD_KERNEL_ACCUMULATE_PIXELS);
    // the frame's first push over every pixel starts from the zeros the frame start wrote
    // instead of reading them
    const int fresh = (j.acc_zero && first == 0 && count == j.g.np) ? 1 : 0;
    j.acc_zero = false;
    bool taken = false;
    if (const cudaError_t er = launch_accumulate_rows(j, s, first, count, gp, spp, fresh, &taken); er != cudaSuccess)
        return er;
    if (taken) {
        j.launches += 1;
        return cudaSuccess;
    }
    auto aligned = [](const void* ptr, uintptr_t a) { return (reinterpret_cast<uintptr_t>(ptr) & (a - 1)) == 0; };
    bool vec4 = spp > 0 && spp % 4 == 0 && aligned(s.flags, 16) && (!s.category || aligned(s.category, 16));
    if (s.compact) {
        const DeviceSamples16& h = s.c16;
        for (int c = 0; c < 3; ++c) vec4 = vec4 && aligned(h.sqrt_radiance[c], 8) && aligned(h.normal[c], 8);
        vec4 = vec4 && aligned(h.depth, 8);
        for (int c = 0; c < 2; ++c)
            vec4 = vec4 && (!h.pixel_u[0] || aligned(h.pixel_u[c], 8)) && (!h.lens_u[0] || aligned(h.lens_u[c], 8)) &&
                   (!h.brdf_u[0] || aligned(h.brdf_u[c], 8)) && (!h.light_u[0] || aligned(h.light_u[c], 8)) &&
                   (!h.env_u[0] || aligned(h.env_u[c], 8));
    } else {
        vec4 = vec4 && aligned(s.depth, 16);
        for (int c = 0; c < 3; ++c)
            vec4 = vec4 && aligned(s.radiance[c], 16) && aligned(s.normal[c], 16) && (!s.albedo[0] || aligned(s.albedo[c], 16));
        for (int c = 0; c < 2; ++c)
            vec4 = vec4 && (!s.pixel_u[0] || aligned(s.pixel_u[c], 16)) && (!s.lens_u[0] || aligned(s.lens_u[c], 16)) &&
                   (!s.brdf_u[0] || aligned(s.brdf_u[c], 16)) && (!s.light_u[0] || aligned(s.light_u[c], 16)) &&
                   (!s.env_u[0] || aligned(s.env_u[c], 16));
    }
    vec4 = vec4 && (!gp.lum || (aligned(gp.lum, 16) && aligned(gp.key, 16)));
    // Shapes measured on GB300 at 1920x1080. Up to 16 samples per pixel, more resident pixels
    // hide the per-pixel latency (four samples per load: compact planes 4 blocks per SM, FP32 planes
    // 3; single samples, the pixel split over two warps: 8). From 32 on, a thread's sample run spans more bytes per plane than L1 keeps between its
    // loads, and a block's registers are not capped; from 64 on, compact planes are read 16 bytes
    // (8 samples) per load.
    const bool many = spp > 16;
    cudaError_t e;
    if (s.compact) {
        bool wide = vec4 && spp >= 64 && spp % 8 == 0;
        const DeviceSamples16& h = s.c16;
        for (int c = 0; c < 3; ++c) wide = wide && aligned(h.sqrt_radiance[c], 16) && aligned(h.normal[c], 16);
        wide = wide && aligned(h.depth, 16);
        for (int c = 0; c < 2; ++c)
            wide = wide && (!h.pixel_u[0] || aligned(h.pixel_u[c], 16)) && (!h.lens_u[0] || aligned(h.lens_u[c], 16)) &&
                   (!h.brdf_u[0] || aligned(h.brdf_u[c], 16)) && (!h.light_u[0] || aligned(h.light_u[c], 16)) &&
                   (!h.env_u[0] || aligned(h.env_u[c], 16));
        if (wide)
            e = run_accumulate<true, true, true, 1, false>(j, s, spp, first, count, gp, fresh);
        else if (vec4 && many)
            e = run_accumulate<true, true, false, 1, false>(j, s, spp, first, count, gp, fresh);
        else if (vec4)
            e = run_accumulate<true, true, false, 4, false>(j, s, spp, first, count, gp, fresh);
        else
            e = run_accumulate<false, true, false, 8, true>(j, s, spp, first, count, gp, fresh);
    } else {
        if (vec4 && many)
            e = run_accumulate<true, false, false, 1, false>(j, s, spp, first, count, gp, fresh);
        else if (vec4)
            e = run_accumulate<true, false, false, 3, false>(j, s, spp, first, count, gp, fresh);
        else
            e = run_accumulate<false, false, false, 8, true>(j, s, spp, first, count, gp, fresh);
    }
    if (e != cudaSuccess) return e;
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_accumulate_grid(Job& j, const DeviceSamples& s, int64_t first, int64_t count, int32_t spp) {
    KernelScope ks(j, RPD_KERNEL_GRID);
    const int64_t threads = j.g.nn * kDeps;
    k_grid_ordered<<<grid_for(threads, 128), 128, 0, j.stream>>>(j.g, j.n.pass_grid, s, j.offsets, spp, first, count);
    j.pass_indirect = true;
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_merge_grid(Job& j) {
    // pushes that added straight into the frame grid leave nothing in the pass grid
    const bool any = j.pass_indirect;
    j.pass_direct = j.pass_indirect = false;
    if (!any) return cudaSuccess;
    KernelScope ks(j, RPD_KERNEL_MERGE);
    const int64_t n = j.g.nn * kDeps * kDepStride;
    const bool pass_pairs = !j.exact_grid;  // the pass grid's form (k_grid_ordered writes doubles)
    const unsigned blocks = grid_for(n, 256);
    double* g = j.n.grid;
    double* pg = j.n.pass_grid;
    if (j.grid_fresh) {
        if (pass_pairs) k_merge_grid<kMergePairsFresh><<<blocks, 256, 0, j.stream>>>(g, pg, n);
        else k_merge_grid<kMergeDoubleFresh><<<blocks, 256, 0, j.stream>>>(g, pg, n);
        j.grid_pairs = pass_pairs;
    } else if (pass_pairs && j.grid_pairs) {
        k_merge_grid<kMergePairsPairs><<<blocks, 256, 0, j.stream>>>(g, pg, n);
    } else if (!pass_pairs && !j.grid_pairs) {
        k_merge_grid<kMergeDoubleDouble><<<blocks, 256, 0, j.stream>>>(g, pg, n);
    } else if (pass_pairs) {
        k_merge_grid<kMergePairsIntoDouble><<<blocks, 256, 0, j.stream>>>(g, pg, n);
    } else {
        k_merge_grid<kMergeDoubleIntoPairs><<<blocks, 256, 0, j.stream>>>(g, pg, n);
        j.grid_pairs = false;
    }
    j.grid_fresh = false;
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_grid_to_double(Job& j, double* out) {
    const int64_t n = j.g.nn * kDeps * kDepStride;
    k_grid_pairs_to_double<<<grid_for(n, 256), 256, 0, j.stream>>>(reinterpret_cast<const float2*>(j.n.grid), out, n);
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_feature_cache(Job& j) {
    KernelScope ks(j, RPD_KERNEL_FEATURES);
    k_feature_cache<<<grid_for(j.g.np, 256), 256, 0, j.stream>>>(j.p, j.g.np);
    j.launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_finalize(Job& j) {
    KernelScope ks(j, RPD_KERNEL_OTHER);
    k_finalize<<<grid_for(j.g.np, 256), 256, 0, j.stream>>>(j.p, j.g.np);
    j.launches += 1;
    return cudaGetLastError();
}

}  // namespace rpd
