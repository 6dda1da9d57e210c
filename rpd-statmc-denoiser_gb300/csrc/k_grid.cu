// accumulate_rpf_sample_to_grid (main.cpp:329-376), fast path.
//
// One warp per (node, dimension group). Group 0 owns the `pixel` dependency; groups 1-6
// own a random dimension X (brdf, lens, light_uv, environment, light_select, rr) together
// with its screen comparator screen_X. The reference's per-sample double-precision
// accumulations are regrouped by what they depend on:
//   * the node weight w = fl(ax * ay) is a per-pixel product of an x factor and a y factor,
//     so every total of a dependency (w_sum, w2_sum, y_sum, y2_sum) is w times a per-pixel
//     class sum (count, sum y, sum y^2) that the statistics pass produced;
//   * the screen bin of a sample depends on the node and on where the sample lies in its
//     pixel; with a power-of-two support of at least 4 pixels every sample whose position
//     stays inside its pixel falls in the pixel's nominal bin, so a uniform pixel updates
//     one screen bin once (other pixels, and other supports, are binned sample by sample
//     exactly as the reference bins them);
//   * only the random-dimension bins are updated per sample, from the packed key the
//     statistics pass wrote.
// k_grid_fast walks the node's support pixels (lanes over pixels) for the totals and the
// screen bins; k_grid_random walks the support's samples (lanes over consecutive samples of
// each support row: coalesced loads) for the random-dimension bins. Each lane owns private
// accumulators, combined in a fixed order at the end: deterministic, no atomics. Sums of y are double-float (pairs of floats, exact
// products via FMA; about 2^-44 relative — GB300 executes double precision at 1/55 of its
// single-precision rate). With a power-of-two node step every weight is an exact multiple
// of 1/step^2, so the bin weights are accumulated as exact integers.
#include <cmath>
#include <type_traits>

#include "rpd_internal.h"
#include "device_math.cuh"

namespace rpd {

namespace {

constexpr int kGroups = 7;
constexpr int kStripSms = 152;  // GB300's SMs

__device__ __forceinline__ void df_add(float& hi, float& lo, float x) {
    const float s = hi + x;
    const float bb = s - hi;
    lo += (hi - (s - bb)) + (x - bb);
    hi = s;
}

// (hi, lo) += a * (bh + bl), with the product a*bh split exactly
__device__ __forceinline__ void df_add_scaled(float& hi, float& lo, float a, float bh, float bl) {
    const float p = a * bh;
    const float e = __fmaf_rn(a, bh, -p);
    df_add(hi, lo, p);
    lo += __fmaf_rn(a, bl, e);
}

struct DF {
    float h = 0.0f, l = 0.0f;
};

// The fast path's pass grid holds every entry as a double-float (hi, lo) pair in the 8 bytes
// of a double; the merge into the frame grid turns it into a double (k_merge_grid).
__device__ __forceinline__ void df_accum(float2* e, float h, float l) {
    float2 v = *e;
    df_add(v.x, v.y, h);
    v.y += l;
    *e = v;
}

// An integer bin weight (a multiple of 1/step^2, below 2^32 by the launch's bound) as a
// double-float: the float of the integer plus the float of its remainder, scaled exactly.
__device__ __forceinline__ float2 int_weight_df(uint64_t total, float inv_wscale) {
    const uint32_t t = uint32_t(total);
    const float hi = __uint2float_rz(t);          // an integer <= t
    const uint32_t rem = t - __float2uint_rz(hi);  // below 2^8, exact in float
    return make_float2(hi * inv_wscale, float(rem) * inv_wscale);
}

struct Totals {
    DF w, w2, y, y2;
};

// The screen position (pixel_u) of sample k, from either sample-plane format.
__device__ __forceinline__ float sample_pu(const DeviceSamples& s, int c, int64_t k) {
    return s.compact ? float(s.c16.pixel_u[c][k]) * (1.0f / 65536.0f) : s.pixel_u[c][k];
}

// Dependency2D::add bin (core/stats.h:166-168)
__device__ __forceinline__ int bin2d(float u, float v) {
    const int x = iclamps(int(u * 4.0f), 0, 3);
    const int z = iclamps(int(v * 4.0f), 0, 3);
    return z * 4 + x;
}

__device__ __forceinline__ void add_class(Totals& t, float w, float c, float s1h, float s1l, float s2h, float s2l) {
    df_add_scaled(t.w.h, t.w.l, w, c, 0.0f);
    const float w2 = w * w;
    const float w2e = __fmaf_rn(w, w, -w2);
    df_add_scaled(t.w2.h, t.w2.l, c, w2, w2e);
    df_add_scaled(t.y.h, t.y.l, w, s1h, s1l);
    df_add_scaled(t.y2.h, t.y2.l, w, s2h, s2l);
}

__device__ __forceinline__ void add_sample(Totals& t, float w, float y) {
    df_add(t.w.h, t.w.l, w);
    const float w2 = w * w;
    df_add(t.w2.h, t.w2.l, w2);
    t.w2.l += __fmaf_rn(w, w, -w2);
    const float wy = w * y;
    const float wye = __fmaf_rn(w, y, -wy);
    df_add(t.y.h, t.y.l, wy);
    t.y.l += wye;
    const float p = wy * y;  // (w*y)*y with w*y = wy + wye
    const float pe = __fmaf_rn(wy, y, -p);
    df_add(t.y2.h, t.y2.l, p);
    t.y2.l += __fmaf_rn(wye, y, pe);
}

// Lane-private bins in shared memory, [slot][lane] of the warp's region (conflict free).
// INT_W: slots 0-15 hold the bin weights as exact integers w * step^2, 16-31 / 32-47 the
// double-float sums of w*y. Otherwise: weights double-float in 0-15 / 16-31, sums in
// 32-47 / 48-63.
template <bool INT_W>
struct LaneBins {
    static constexpr int kSlots = INT_W ? 48 : 64;
    static constexpr int kSy = INT_W ? 16 : 32;
    float* base;
    int lane;
    float wscale;  // step^2 (INT_W)
    __device__ float& at(int slot) { return base[slot * 32 + lane]; }
    __device__ void clear() {
        for (int k = 0; k < kSlots; ++k) at(k) = 0.0f;
    }
    __device__ void add_weight(int bin, float w, float c) {  // weight += w * c
        if (INT_W) {
            uint32_t* u = reinterpret_cast<uint32_t*>(&at(bin));
            *u += uint32_t(w * wscale) * uint32_t(c);
        } else {
            float wh = at(bin), wl = at(16 + bin);
            df_add_scaled(wh, wl, w, c, 0.0f);
            at(bin) = wh;
            at(16 + bin) = wl;
        }
    }
    __device__ void add_sum(int bin, float w, float sh, float sl) {  // sum_y += w * (sh + sl)
        float yh = at(kSy + bin), yl = at(kSy + 16 + bin);
        df_add_scaled(yh, yl, w, sh, sl);
        at(kSy + bin) = yh;
        at(kSy + 16 + bin) = yl;
    }
    // Sum the 32 lanes in a fixed (rotated) order; lane v owns value v: weight[v] for v < 16,
    // sum_y[v - 16] otherwise. Returns the lane's value as a double-float.
    __device__ float2 reduce_value() {
        __syncwarp();
        const int v = lane;
        float2 out;
        if (INT_W && v < 16) {
            uint64_t total = 0;
            for (int i = 0; i < 32; ++i) total += reinterpret_cast<const uint32_t*>(base)[v * 32 + ((i + v) & 31)];
            out = int_weight_df(total, 1.0f / wscale);
        } else {
            const int hi_slot = v < 16 ? v : kSy + (v - 16);
            float h = 0.0f, l = 0.0f;
            for (int i = 0; i < 32; ++i) {
                const int src = (i + v) & 31;  // rotated: the 32 lanes read 32 different banks
                df_add(h, l, base[hi_slot * 32 + src]);
                l += base[(hi_slot + 16) * 32 + src];
            }
            out = make_float2(h, l);
        }
        __syncwarp();
        return out;
    }
    // As reduce_value, adding the result to the pass-grid entry acc[v].
    __device__ void reduce_into(float2* acc) {
        const float2 out = reduce_value();
        if (out.x != 0.0f || out.y != 0.0f) df_accum(acc + lane, out.x, out.y);
    }
};

// Warp sum of the lanes' totals (fixed shuffle tree); the result is valid in lane 0 as
// double-floats (w_sum, w2_sum, y_sum, y2_sum).
__device__ void reduce_totals(Totals t, float2* out4) {
    float v[8] = {t.w.h, t.w.l, t.w2.h, t.w2.l, t.y.h, t.y.l, t.y2.h, t.y2.l};
    for (int off = 16; off > 0; off >>= 1) {
        for (int q = 0; q < 4; ++q) {
            const float oh = __shfl_down_sync(0xffffffffu, v[2 * q], off);
            const float ol = __shfl_down_sync(0xffffffffu, v[2 * q + 1], off);
            df_add(v[2 * q], v[2 * q + 1], oh);
            v[2 * q + 1] += ol;
        }
    }
    for (int q = 0; q < 4; ++q) out4[q] = make_float2(v[2 * q], v[2 * q + 1]);
}

// v[q] for a lane-dependent q in 0-3, without indexing the registers
__device__ __forceinline__ float2 pick4(const float2* v, int q) {
    return q == 0 ? v[0] : q == 1 ? v[1] : q == 2 ? v[2] : v[3];
}

// As reduce_totals, adding the result to the pass-grid entries acc[32..35].
__device__ void reduce_totals_into(Totals t, float2* acc) {
    float2 r[4];
    reduce_totals(t, r);
    if ((threadIdx.x & 31) == 0) {
        for (int q = 0; q < 4; ++q)
            if (r[q].x != 0.0f || r[q].y != 0.0f) df_accum(acc + 32 + q, r[q].x, r[q].y);
    }
}

struct GridParams {
    Geometry g;
    int64_t first, count;
    int64_t node0;        // first node of the launch (the node rows whose supports meet the push)
    int64_t count_nodes;  // nodes of the launch
    int uniform_ok;  // power-of-two support >= 4
    int pow2_step;   // the node step is a power of two: x / step is exact
    float inv_step;
    int spp;         // samples per pixel of the push, 0 when the counts vary
    float inv_spp;
};

// x (or y) factor of the bilinear weight of node n for coordinate c (main.cpp:332-346):
// (1 - t) when floor(c / step) is n, t when it is n - 1, 0 otherwise.
__device__ __forceinline__ float axis_factor(const GridParams& gp, int c, int n, int nodes) {
    const float gc = gp.pow2_step ? float(c) * gp.inv_step : float(c) / float(gp.g.step);
    const int c0 = iclamps(int(floorf(gc)), 0, nodes - 1);
    const int c1 = imins(c0 + 1, nodes - 1);
    const float t = fclamps(gc - float(c0), 0.0f, 1.0f);
    if (c0 == n) return 1.0f - t;
    if (c1 == n) return t;
    return 0.0f;
}

// A pixel's first pattern's sums, its patterns and flags (see GridPrep).
struct PixPattern {
    float c, s1h, s1l, s2h, s2l;
    uint8_t pat, pf, more[kPatterns - 1];
};
__device__ __forceinline__ PixPattern load_pattern(const GridPrep& gp, int64_t idx) {
    const float4 a = gp.pat4[idx];
    const float2 b = gp.pat2[idx];
    const uint32_t bits = __float_as_uint(b.y);
    return PixPattern{a.x, a.y, a.z, a.w, b.x, uint8_t(bits), uint8_t(bits >> 8), {uint8_t(bits >> 16), uint8_t(bits >> 24)}};
}

// The (count, sum y hi/lo, sum y^2 hi/lo) of class c for pixel idx (see GridPrep). Both planes' sums are asked
// for before either is used: one after another, a warp whose pixels differ waits three times (the pattern
// form's totals and screen bins of a 256x256x8 frame of up to eight patterns 92 -> 188 us).
__device__ __forceinline__ void class_sums(const GridPrep& gp, int c, int64_t idx, const PixPattern& pp,
                                           float* out) {
    static_assert(kPatterns == 3, "two further patterns");
    const bool whole = (pp.pf & kPixDeviant) != 0;
    const bool in0 = !whole && (pp.pat & class_bit(c)), in1 = !whole && (pp.more[0] & class_bit(c)),
               in2 = !whole && (pp.more[1] & class_bit(c));
    float a[5], b[5];
    for (int f = 0; f < 5; ++f) {
        const float* plane = whole ? gp.cls[c][f] : gp.cls[0][f];
        a[f] = whole || in1 ? plane[idx] : 0.0f;
        b[f] = in2 ? gp.cls[1][f][idx] : 0.0f;
    }
    out[0] = in0 ? pp.c : 0.0f;
    out[1] = in0 ? pp.s1h : 0.0f;
    out[2] = in0 ? pp.s1l : 0.0f;
    out[3] = in0 ? pp.s2h : 0.0f;
    out[4] = in0 ? pp.s2l : 0.0f;
    for (const float* s : {a, b}) {
        out[0] += s[0];
        df_add(out[1], out[2], s[1]);
        out[2] += s[2];
        df_add(out[3], out[4], s[3]);
        out[4] += s[4];
    }
}

template <bool INT_W>
__global__ void __launch_bounds__(kGroups * 32) k_grid_fast(GridParams gpar, float2* pass_grid, DeviceSamples s,
                                                            const int64_t* offsets, GridPrep gp) {
    extern __shared__ float sm[];
    const int lane = threadIdx.x & 31;
    const int grp = threadIdx.x >> 5;
    const int64_t node = gpar.node0 + blockIdx.x;
    const Geometry& g = gpar.g;
    const int nx = int(node % g.nodes_x), ny = int(node / g.nodes_x);
    LaneBins<INT_W> bins{sm + grp * LaneBins<INT_W>::kSlots * 32, lane, float(g.step) * float(g.step)};
    const uint32_t absent = key_absent_bit(grp) | key_absent_bit(0);
    int dep_x = D_PIXEL, dep_s = D_PIXEL;
    switch (grp) {
    case 1: dep_x = D_BRDF; dep_s = D_SCREEN_BRDF; break;
    case 2: dep_x = D_LENS; dep_s = D_SCREEN_LENS; break;
    case 3: dep_x = D_LIGHT_UV; dep_s = D_SCREEN_LIGHT_UV; break;
    case 4: dep_x = D_ENV; dep_s = D_SCREEN_ENV; break;
    case 5: dep_x = D_LIGHT_SELECT; dep_s = D_SCREEN_LIGHT_SELECT; break;
    case 6: dep_x = D_RR; dep_s = D_SCREEN_RR; break;
    default: break;
    }
    float2* base = pass_grid + node * kDeps * kDepStride;
    const float support = float(g.support);
    const float half_support = 0.5f * support;
    const float support_left = float(nx * g.step) - half_support;
    const float support_top = float(ny * g.step) - half_support;
    const int xlo = imaxs(0, (nx - 1) * g.step - 1), xhi = imins(g.w - 1, (nx + 1) * g.step + 1);
    const int ylo = imaxs(0, (ny - 1) * g.step - 1), yhi = imins(g.h - 1, (ny + 1) * g.step + 1);
    const int cols = xhi - xlo + 1;
    const int npix = cols * (yhi - ylo + 1);

    // ---- per-pixel class sums -> totals and (uniform pixels) screen bins ------------------
    bins.clear();
    Totals tot_x, tot_s;
    for (int q0 = 0; q0 < npix; q0 += 32) {
        const int q = q0 + lane;
        bool slow = false;
        int x = 0, y = 0;
        int64_t idx = 0;
        float w = 0.0f;
        bool mixed = false;
        if (q < npix) {
            x = xlo + q % cols;
            y = ylo + q / cols;
            idx = int64_t(y) * g.w + x;
            if (idx >= gpar.first && idx < gpar.first + gpar.count) {
                w = axis_factor(gpar, x, nx, g.nodes_x) * axis_factor(gpar, y, ny, g.nodes_y);
                const PixPattern pp = load_pattern(gp, idx);
                const uint8_t pf = pp.pf;
                float cs[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
                if (w > 1e-8f) class_sums(gp, grp, idx, pp, cs);  // core/stats.h:103 skips w <= 1e-8
                const float cnt = cs[0];
                if (cnt != 0.0f) {
                    const float s1h = cs[1], s1l = cs[2], s2h = cs[3], s2l = cs[4];
                    mixed = grp > 0 && (pf & kPixMixed);
                    add_class(tot_x, w, cnt, s1h, s1l, s2h, s2l);
                    if (!mixed) add_class(tot_s, w, cnt, s1h, s1l, s2h, s2l);
                    if (gpar.uniform_ok && (pf & kPixUniform) && !mixed) {
                        const float su0 = fclamps((float(x) - support_left) / support, 0.0f, 1.0f);
                        const float sv0 = fclamps((float(y) - support_top) / support, 0.0f, 1.0f);
                        const int b = bin2d(su0, sv0);
                        bins.add_weight(b, w, cnt);
                        bins.add_sum(b, w, s1h, s1l);
                    } else {
                        slow = true;
                    }
                }
            }
        }
        // pixels binned sample by sample (and the screen_X totals of mixed pixels): the whole
        // warp walks each such pixel's samples, every lane into its own bins
        unsigned pending = __ballot_sync(0xffffffffu, slow);
        while (pending) {
            const int src = __ffs(pending) - 1;
            pending &= pending - 1;
            const int64_t pidx = __shfl_sync(0xffffffffu, idx, src);
            const float pw = __shfl_sync(0xffffffffu, w, src);
            const bool pmixed = __shfl_sync(0xffffffffu, int(mixed), src) != 0;
            const float fx = float(__shfl_sync(0xffffffffu, x, src));
            const float fy = float(__shfl_sync(0xffffffffu, y, src));
            const int64_t local = pidx - gpar.first;
            const int64_t kend = sample_offset(offsets, gpar.spp, local + 1);
            for (int64_t k = sample_offset(offsets, gpar.spp, local) + lane; k < kend; k += 32) {
                const uint32_t key = gp.key[k];
                if (key & absent) continue;
                const float yv = gp.lum[k];
                const float su = fclamps((fx + sample_pu(s, 0, k) - support_left) / support, 0.0f, 1.0f);
                const float sv = fclamps((fy + sample_pu(s, 1, k) - support_top) / support, 0.0f, 1.0f);
                const int b = bin2d(su, sv);
                bins.add_weight(b, pw, 1.0f);
                bins.add_sum(b, pw, yv, 0.0f);
                if (pmixed) add_sample(tot_s, pw, yv);
            }
        }
    }
    // screen bins and totals: `pixel` for group 0, screen_X (and X's totals) otherwise
    bins.reduce_into(base + dep_s * kDepStride);
    reduce_totals_into(tot_s, base + dep_s * kDepStride);
    if (grp == 0) return;
    reduce_totals_into(tot_x, base + dep_x * kDepStride);
}

// ---- totals and screen bins, pattern form (small images, other supports) ------------------
//
// One warp per node. Pixels of the node's pattern P0 (the pattern of its first non-deviant
// support pixel) carry the same class sums for every class in P0, so their totals are formed
// once (TP) and their screen bins once (bins A: per pixel for uniform pixels, sample by sample
// otherwise); each class then takes TP and bins A if it is in P0. Every other pixel (of
// several patterns, or of another one) goes to a list handled class by class as the per-class kernel does
// (bins B). All sums are lane-private and combined in a fixed order: deterministic.
__device__ __forceinline__ int axis_ifactor(int c, int n, int nodes, int sh) {
    // x factor * step of a power-of-two step (c < (nodes - 1) * step for every image pixel)
    const int c0 = imins(c >> sh, nodes - 1);
    const int t = c - (c0 << sh);
    return c0 == n ? (1 << sh) - t : (c0 + 1 == n ? t : 0);
}

template <bool INT_W>
__global__ void __launch_bounds__(32) k_grid_screen(GridParams gpar, float2* pass_grid, DeviceSamples s,
                                                    const int64_t* offsets, GridPrep gp) {
    extern __shared__ float sm[];
    constexpr int kS = LaneBins<INT_W>::kSlots;
    const int lane = threadIdx.x;
    const int64_t node = gpar.node0 + blockIdx.x;
    const Geometry& g = gpar.g;
    const int nx = int(node % g.nodes_x), ny = int(node / g.nodes_x);
    const float wscale = float(g.step) * float(g.step);
    LaneBins<INT_W> binsA{sm, lane, wscale};
    int* xlist = reinterpret_cast<int*>(sm + kS * 32);
    float2* base = pass_grid + node * kDeps * kDepStride;
    const float support = float(g.support);
    const float half_support = 0.5f * support;
    const float support_left = float(nx * g.step) - half_support;
    const float support_top = float(ny * g.step) - half_support;
    const int xlo = imaxs(0, (nx - 1) * g.step - 1), xhi = imins(g.w - 1, (nx + 1) * g.step + 1);
    const int ylo = imaxs(0, (ny - 1) * g.step - 1), yhi = imins(g.h - 1, (ny + 1) * g.step + 1);
    const int cols = xhi - xlo + 1;
    const int npix = cols * (yhi - ylo + 1);
    const int sh = __ffs(g.step) - 1;                 // log2(step) when the step is a power of two
    const int bsh = __ffs(g.support) - 3;             // log2(support / 4) when uniform_ok
    const int sl = nx * g.step - g.support / 2, st = ny * g.step - g.support / 2;  // integer when uniform_ok
    const float inv_wscale = 1.0f / wscale;

    auto weight = [&](int x, int y) -> float {
        if (gpar.pow2_step)
            return float(axis_ifactor(x, nx, g.nodes_x, sh) * axis_ifactor(y, ny, g.nodes_y, sh)) * inv_wscale;
        return axis_factor(gpar, x, nx, g.nodes_x) * axis_factor(gpar, y, ny, g.nodes_y);
    };
    // the pixel's nominal screen bin (every sample's, for a uniform pixel)
    auto uniform_bin = [&](int x, int y) -> int {
        const int dx = x - sl, dy = y - st;
        const int bx = dx < 0 ? 0 : imins(dx >> bsh, 3), by = dy < 0 ? 0 : imins(dy >> bsh, 3);
        return by * 4 + bx;
    };
    // samples of pixel (px, py) binned one by one by the whole warp (main.cpp:349-357): every
    // lane into its own bins; also the screen totals of a mixed pixel (samples with the
    // position and the class)
    auto bin_samples = [&](LaneBins<INT_W>& bins, int64_t pidx, float pw, int px, int py, uint32_t absent,
                           bool pmixed, Totals& ts) {
        const float fx = float(px), fy = float(py);
        const int64_t local = pidx - gpar.first;
        const int64_t kend = sample_offset(offsets, gpar.spp, local + 1);
        for (int64_t k = sample_offset(offsets, gpar.spp, local) + lane; k < kend; k += 32) {
            const uint32_t key = gp.key[k];
            if (key & absent) continue;
            const float yv = gp.lum[k];
            const float su = fclamps((fx + sample_pu(s, 0, k) - support_left) / support, 0.0f, 1.0f);
            const float sv = fclamps((fy + sample_pu(s, 1, k) - support_top) / support, 0.0f, 1.0f);
            const int b = bin2d(su, sv);
            bins.add_weight(b, pw, 1.0f);
            bins.add_sum(b, pw, yv, 0.0f);
            if (pmixed) add_sample(ts, pw, yv);
        }
    };

    // ---- P0: the pattern of the first non-deviant support pixel with a pattern ----
    uint8_t P0 = 0;
    for (int q0 = 0; q0 < npix; q0 += 32) {
        const int q = q0 + lane;
        uint8_t pat = 0;
        if (q < npix) {
            const int64_t idx = int64_t(ylo + q / cols) * g.w + xlo + q % cols;
            if (idx >= gpar.first && idx < gpar.first + gpar.count) {
                const uint32_t bits = __float_as_uint(gp.pat2[idx].y);
                if (!((bits >> 8) & kPixDeviant) && (bits >> 16) == 0u) pat = uint8_t(bits & 0xffu);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, pat != 0);
        if (m) {
            P0 = uint8_t(__shfl_sync(0xffffffffu, int(pat), __ffs(m) - 1));
            break;
        }
    }
    const bool p0pix = (P0 & RPD_SAMPLE_PIXEL_VALID) != 0;

    // ---- main pass: P0 pixels into TP / bins A, the rest into the list ----
    binsA.clear();
    Totals TP, unused;
    int nlist = 0;
    int x = xlo + lane % cols, y = ylo + lane / cols;  // position of q = q0 + lane
    // the pattern record of q, loaded one iteration ahead so the loads overlap the work
    auto fetch = [&](int q, int px, int py, PixPattern& pp, bool& in) {
        const int64_t idx = int64_t(py) * g.w + px;
        in = q < npix && idx >= gpar.first && idx < gpar.first + gpar.count;
        if (in) pp = load_pattern(gp, idx);
        else pp = PixPattern{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0, 0, {0, 0}};
    };
    PixPattern nxt;
    bool nin;
    fetch(lane, x, y, nxt, nin);
    for (int q0 = 0; q0 < npix; q0 += 32) {
        const PixPattern pp = nxt;
        const bool in = nin;
        const int cx = x, cy = y;
        x += 32;
        while (x > xhi) {
            x -= cols;
            ++y;
        }
        if (q0 + 32 < npix) fetch(q0 + 32 + lane, x, y, nxt, nin);
        bool exc = false, slow = false;
        const int64_t idx = int64_t(cy) * g.w + cx;
        float w = 0.0f;
        if (in) {
            w = weight(cx, cy);
            if (w > 1e-8f) {  // BinnedDependency::add skips w <= 1e-8 (core/stats.h:103)
                const bool dev = (pp.pf & kPixDeviant) != 0 || pp.more[0] != 0;  // several patterns
                if (!dev && pp.pat == P0 && pp.pat != 0) {
                    add_class(TP, w, pp.c, pp.s1h, pp.s1l, pp.s2h, pp.s2l);
                    if (p0pix) {
                        if (gpar.uniform_ok && (pp.pf & kPixUniform)) {
                            const int b = uniform_bin(cx, cy);
                            binsA.add_weight(b, w, pp.c);
                            binsA.add_sum(b, w, pp.s1h, pp.s1l);
                        } else {
                            slow = true;
                        }
                    }
                } else if (dev || pp.pat != 0) {
                    exc = true;
                }
            }
        }
        const int q = q0 + lane;
        const unsigned me = __ballot_sync(0xffffffffu, exc);
        if (exc) xlist[nlist + __popc(me & ((1u << lane) - 1))] = q;
        nlist += __popc(me);
        unsigned pending = __ballot_sync(0xffffffffu, slow);
        while (pending) {
            const int src = __ffs(pending) - 1;
            pending &= pending - 1;
            const int64_t pidx = __shfl_sync(0xffffffffu, idx, src);
            const float pw = __shfl_sync(0xffffffffu, w, src);
            const int px = __shfl_sync(0xffffffffu, cx, src), py = __shfl_sync(0xffffffffu, cy, src);
            bin_samples(binsA, pidx, pw, px, py, key_absent_bit(0), false, unused);
        }
    }
    __syncwarp();
    float2 tp[4];
    reduce_totals(TP, tp);
    // lane k of 0-7 adds total k & 3 of P0's pixels (the sums are lane 0's)
#pragma unroll
    for (int k = 0; k < 4; ++k) tp[k] = make_float2(__shfl_sync(0xffffffffu, tp[k].x, 0), __shfl_sync(0xffffffffu, tp[k].y, 0));
    const float2 tpq = pick4(tp, lane & 3);
    const float2 va = binsA.reduce_value();
    LaneBins<INT_W>& binsB = binsA;  // bins A are folded into va: reuse their storage

    // ---- class by class: P0's share plus the listed pixels ----
    for (int cl = 0; cl < kClasses; ++cl) {
        const bool inP0 = (P0 & class_bit(cl)) != 0;
        const bool p0screen = inP0 && p0pix;  // P0 pixels enter the screen sums of this class
        const uint32_t absent = key_absent_bit(cl) | key_absent_bit(0);
        Totals tx, ts;
        float2 vb = make_float2(0.0f, 0.0f);
        if (nlist > 0) {
            binsB.clear();
            for (int i0 = 0; i0 < nlist; i0 += 32) {
                const int i = i0 + lane;
                bool slow = false, mixed = false;
                int px = 0, py = 0;
                int64_t idx = 0;
                float w = 0.0f;
                if (i < nlist) {
                    const int q = xlist[i];
                    px = xlo + q % cols;
                    py = ylo + q / cols;
                    idx = int64_t(py) * g.w + px;
                    w = weight(px, py);
                    const PixPattern pp = load_pattern(gp, idx);
                    const uint8_t pf = pp.pf;
                    float cs[5];
                    class_sums(gp, cl, idx, pp, cs);
                    if (cs[0] != 0.0f) {
                        mixed = cl > 0 && (pf & kPixMixed);
                        add_class(tx, w, cs[0], cs[1], cs[2], cs[3], cs[4]);
                        if (!mixed) add_class(ts, w, cs[0], cs[1], cs[2], cs[3], cs[4]);
                        if (gpar.uniform_ok && (pf & kPixUniform) && !mixed) {
                            const int b = uniform_bin(px, py);
                            binsB.add_weight(b, w, cs[0]);
                            binsB.add_sum(b, w, cs[1], cs[2]);
                        } else {
                            slow = true;
                        }
                    }
                }
                unsigned pending = __ballot_sync(0xffffffffu, slow);
                while (pending) {
                    const int src = __ffs(pending) - 1;
                    pending &= pending - 1;
                    const int64_t pidx = __shfl_sync(0xffffffffu, idx, src);
                    const float pw = __shfl_sync(0xffffffffu, w, src);
                    const bool pmixed = __shfl_sync(0xffffffffu, int(mixed), src) != 0;
                    const int sx = __shfl_sync(0xffffffffu, px, src), sy = __shfl_sync(0xffffffffu, py, src);
                    bin_samples(binsB, pidx, pw, sx, sy, absent, pmixed, ts);
                }
            }
            vb = binsB.reduce_value();
        }
        int dep_x = D_PIXEL, dep_s = D_PIXEL;
        switch (cl) {
        case 1: dep_x = D_BRDF; dep_s = D_SCREEN_BRDF; break;
        case 2: dep_x = D_LENS; dep_s = D_SCREEN_LENS; break;
        case 3: dep_x = D_LIGHT_UV; dep_s = D_SCREEN_LIGHT_UV; break;
        case 4: dep_x = D_ENV; dep_s = D_SCREEN_ENV; break;
        case 5: dep_x = D_LIGHT_SELECT; dep_s = D_SCREEN_LIGHT_SELECT; break;
        case 6: dep_x = D_RR; dep_s = D_SCREEN_RR; break;
        default: break;
        }
        // screen bins (the pixel dependency for class 0): lane v owns bin value v
        float bh = vb.x, bl = vb.y;
        if (p0screen) {
            df_add(bh, bl, va.x);
            bl += va.y;
        }
        // the class's totals, one entry per lane: lanes 0-3 the screen dependency's (32-35),
        // lanes 4-7 the random dimension's (classes 1-6); with no listed pixel the list's part is
        // zero on every lane (nothing to reduce)
        float th = 0.0f, tl = 0.0f;
        float2* te = nullptr;
        {
            float2 t4s[4] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f),
                             make_float2(0.0f, 0.0f)};
            float2 t4x[4] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f),
                             make_float2(0.0f, 0.0f)};
            if (nlist > 0) {
                reduce_totals(ts, t4s);
                if (cl > 0) reduce_totals(tx, t4x);
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // the sums are lane 0's
                    t4s[k] = make_float2(__shfl_sync(0xffffffffu, t4s[k].x, 0), __shfl_sync(0xffffffffu, t4s[k].y, 0));
                    t4x[k] = make_float2(__shfl_sync(0xffffffffu, t4x[k].x, 0), __shfl_sync(0xffffffffu, t4x[k].y, 0));
                }
            }
            if (lane < 4 || (lane < 8 && cl > 0)) {
                const bool scr = lane < 4;
                const float2 ps = pick4(t4s, lane & 3), px = pick4(t4x, lane & 3);
                const float2 t = scr ? ps : px;
                th = t.x;
                tl = t.y;
                if (scr ? p0screen : inP0) {
                    df_add(th, tl, tpq.x);
                    tl += tpq.y;
                }
                te = base + (scr ? dep_s : dep_x) * kDepStride + 32 + (lane & 3);
            }
        }
        // both read-modify-writes of the lane with their loads issued first
        const bool bw = bh != 0.0f || bl != 0.0f;
        const bool tw = te != nullptr && (th != 0.0f || tl != 0.0f);
        float2* be = base + dep_s * kDepStride + lane;
        float2 bv = make_float2(0.0f, 0.0f), tv = make_float2(0.0f, 0.0f);
        if (bw) bv = *be;
        if (tw) tv = *te;
        if (bw) {
            df_add(bv.x, bv.y, bh);
            bv.y += bl;
            *be = bv;
        }
        if (tw) {
            df_add(tv.x, tv.y, th);
            tv.y += tl;
            *te = tv;
        }
    }
}

// ---- totals and screen bins, strip form ----------------------------------------------------------
//
// For power-of-two node steps from 2 to 16 (supports from 4). A pixel's samples then share the pixel's
// nominal screen bin (see uniform_ok), which is its quarter of the node's support in x and in y:
// the pixels of half a cell (step / 2 rows and columns) fall in one bin of each of the cell's four
// nodes. A lane owns a column and walks down it through the pixels' pattern sums: per half strip
// (step / 2 rows) it sums them times the row factors of the node rows above and below, and the lanes of
// a half cell add up their column-weighted sums, which are then one finished bin of four nodes. The
// totals add up over the strip's two halves and the node's two cells. Each pixel is visited once (and
// once more for the cell that neighbouring warps share) instead of once per node it supports, in
// registers instead of lane-private bins in shared memory; warps are independent of each other.
// A validity pattern at a time: its sums enter every class it holds. Then, where some pixel holds more patterns than
// the statistics pass keeps (deviant), a class at a time over the class sums of such pixels; where there are
// many patterns, a class at a time over all pixels. Samples outside
// their pixel's nominal bin, and those of deviant pixels that lack the position, are put right by
// k_grid_odd. The bound is load latency (20 warps per SM, one pass over 24 bytes a pixel): with
// k_grid_odd 0.100 ms at 1920x1080x16 against 0.213 ms for the pattern form; where a pixel's samples
// hold three patterns, 0.28 against 0.82 ms, eight patterns 0.50 against 1.01 ms (29 ms with every deviant
// pixel left to k_grid_odd, class by class and sample by sample).
struct TotalsParams {
    Geometry g;
    int64_t first, count;
    int ny0, ny1;    // node rows of the launch
    int len;         // node rows of a warp
    int col_warps;   // warps per `len` node rows
    int sh;          // log2 of the node step
    int fresh;       // the grid holds zeros (the frame's first push)
    int parts;       // warps that share a strip's classes
    int many;        // walks from which on the classes are walked instead of the patterns
    // the nodes with work for k_grid_odd: how many, and their indices
    unsigned* odd_count;
    int32_t* odd_nodes;
};

__host__ __device__ constexpr int dep_random(int c) { return c == 0 ? 0 : 2 * c - 1; }
__host__ __device__ constexpr int dep_screen(int c) { return 2 * c; }

// Of a pixel with these bits (pat2.y). Deviant: its class sums stand for the screen's too, but for samples with
// a random dimension and no position (mixed). k_grid_odd takes those out again, unless the pixel has no
// others (unplaced): then its class sums are for the random dimensions alone.
constexpr uint32_t kDeviantBit = uint32_t(kPixDeviant) << 8, kMixedBit = uint32_t(kPixMixed) << 8,
                   kPlacedBit = uint32_t(kPixPlaced) << 8;
__device__ __forceinline__ bool deviant(uint32_t bits) { return bits & kDeviantBit; }
__device__ __forceinline__ bool unplaced_pixel(uint32_t bits) {
    return (bits & (kDeviantBit | kMixedBit | kPlacedBit)) == (kDeviantBit | kMixedBit);
}
__device__ __forceinline__ bool mixed_deviant(uint32_t bits) {
    return (bits & (kDeviantBit | kMixedBit | kPlacedBit)) == (kDeviantBit | kMixedBit | kPlacedBit);
}
// Does k_grid_odd look at the pixel? (Only a sample with a position makes a pixel not uniform.)
__device__ __forceinline__ bool odd_pixel(uint32_t bits) {
    return !(bits & (uint32_t(kPixUniform) << 8)) || mixed_deviant(bits);
}

// A set of patterns, one bit each (patterns are even: bit p / 2).
struct PatternSet {
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    __device__ __forceinline__ void add(uint32_t p) {
        if (p == 0u) return;
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (int(p >> 6) == t) w[t] |= 1u << ((p >> 1) & 31u);
    }
    __device__ __forceinline__ void unite_warp() {
#pragma unroll
        for (int t = 0; t < 4; ++t) w[t] = __reduce_or_sync(0xffffffffu, w[t]);
    }
    __device__ __forceinline__ uint32_t pop() {  // the smallest, 0: empty
        uint32_t p = 0;
#pragma unroll
        for (int t = 3; t >= 0; --t)
            if (w[t]) p = uint32_t(t) * 64u + 2u * uint32_t(__ffs(w[t]) - 1);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (p && int(p >> 6) == t) w[t] &= w[t] - 1u;
        return p;
    }
};

// the sum of (h, l) over groups of `lanes` lanes (a power of two), in every lane
__device__ __forceinline__ void df_group_sum(float& h, float& l, int lanes) {
    for (int o = 1; o < lanes; o <<= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
        df_add(h, l, oh);
        l += ol;
    }
}
__device__ __forceinline__ DF df_scaled(float a, DF b) {  // a * b
    DF r;
    r.h = a * b.h;
    r.l = __fmaf_rn(a, b.l, __fmaf_rn(a, b.h, -r.h));
    return r;
}

__global__ void __launch_bounds__(128, 5) k_grid_totals(TotalsParams tp, float2* grid, GridPrep gp) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = int64_t(blockIdx.x) * 4 + (threadIdx.x >> 5), gw = warp / tp.parts;
    const int part = int(warp - gw * tp.parts);
    const Geometry& g = tp.g;
    const int sh = tp.sh, step = g.step, half = step >> 1;
    const int r0 = tp.ny0 + int(gw / tp.col_warps) * tp.len;
    if (r0 >= tp.ny1) return;  // the whole warp
    const int r1 = imins(r0 + tp.len, tp.ny1);
    const int cells = 32 >> sh;
    const int c0 = int(gw % tp.col_warps) * (cells - 1);  // its first cell, between nodes c0 and c0 + 1
    const int x = c0 * step + lane;
    const int cell = lane >> sh, col = lane & (step - 1);
    const bool xin = x < g.w;
    const bool last = (c0 + cells) * step >= g.w;
    // node c0 + j, complete in this warp: both its cells are, or lie outside the image
    auto owned = [&](int j) { return (j > 0 || c0 == 0) && (j < cells || last) && c0 + j < g.nodes_x; };
    const float inv_step = 1.0f / float(step), inv_w = inv_step * inv_step;
    auto inside = [&](int64_t p) { return p >= tp.first && p < tp.first + tp.count; };
    const int s0 = imaxs(r0 - 1, 0), s1 = r1;
    // the patterns of the warp's pixels, and the nodes (of its rows r0 .. r1 - 1) with odd pixels: the
    // lanes' strips first, then the cells'
    PatternSet set;
    bool odd_prev = false, classes = false, unplaced = false, mixed = false;
    for (int s = s0; s < s1; ++s) {
        bool odd = false;
        for (int k0 = 0; k0 < step; k0 += 4) {
            uint32_t bits[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int y = s * step + k0 + i;
                const int64_t p = int64_t(y) * g.w + x;
                bits[i] = k0 + i < step && xin && y < g.h && inside(p) ? __float_as_uint(gp.pat2[p].y) : uint32_t(kPixUniform) << 8;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                odd = odd || odd_pixel(bits[i]);
                mixed = mixed || (bits[i] & kMixedBit);
                unplaced = unplaced || unplaced_pixel(bits[i]);
                classes = classes || (deviant(bits[i]) && !unplaced_pixel(bits[i]));
                if (deviant(bits[i])) continue;
                set.add(bits[i] & 0xffu);
                set.add((bits[i] >> 16) & 0xffu);
                set.add(bits[i] >> 24);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, odd || odd_prev);  // strips s - 1 and s: node row s
        odd_prev = odd;
        if (part > 0 || s < r0 || m == 0u || lane > cells || !owned(lane)) continue;
        // node `lane`: the cells on its left and right
        const unsigned cell_lanes = cells == 1 ? 0xffffffffu : (1u << step) - 1u;
        const bool l = lane > 0 && ((m >> ((lane - 1) << sh)) & cell_lanes);
        const bool r = lane < cells && ((m >> (lane << sh)) & cell_lanes);
        if (l || r) tp.odd_nodes[atomicAdd(tp.odd_count, 1u)] = int32_t(int64_t(s) * g.nodes_x + c0 + lane);
    }
    set.unite_warp();
    classes = __any_sync(0xffffffffu, classes);
    unplaced = __any_sync(0xffffffffu, unplaced);
    mixed = __any_sync(0xffffffffu, mixed);
    // column factors (in units of 1 / step) of the cell's left and right node
    const uint32_t il = uint32_t(step - col), ir = uint32_t(col);
    const float fl = float(il) * inv_step, fr = float(ir) * inv_step;
    bool store_only = tp.fresh != 0;  // the grid is still zero: write instead of add
    // one walk over the strips for pattern P (kPattern), or for class cls (P: that class alone) of all pixels
    // (kAll) or of the deviant ones (kDeviants: unplaced ones or the others); pix: into the screen's sums, of the
    // samples that have the position; rnd: into the random dimension's
    constexpr int kPattern = 0, kDeviants = 1, kAll = 2;
    auto walk = [&](auto mode, uint32_t P, int cls, bool pix, bool rnd) {
        constexpr int kMode = decltype(mode)::value;
        constexpr int kRows = kMode == kAll ? 2 : 4;
        // the column's part of the next node row's totals: weights, squared weights, y, y^2
        uint32_t nw = 0u;
        unsigned long long nw2 = 0ull;
        DF ny, nz;
        for (int s = s0; s < s1; ++s) {
            const bool up = s >= r0, down = s + 1 < r1;
            uint32_t tw = nw;  // node row s
            unsigned long long tw2 = nw2;
            DF ty = ny, tz = nz;
            nw = 0u;
            nw2 = 0ull;
            ny = nz = DF{};
            for (int hs = 0; hs < 2; ++hs) {
                uint32_t bw[2] = {0u, 0u};  // [0] the node row above, [1] below
                DF by[2];
                // rows in fours (twos), their records loaded before any is used
                for (int k0 = hs * half; k0 < (hs + 1) * half; k0 += kRows) {
                    float4 A[kRows];
                    float2 B[kRows];
                    auto read = [&](auto load) {
#pragma unroll
                        for (int i = 0; i < kRows; ++i) {
                            const int y = s * step + k0 + i;
                            const int64_t p = int64_t(y) * g.w + x;
                            A[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            B[i] = make_float2(0.0f, 0.0f);
                            if (k0 + i < (hs + 1) * half && xin && y < g.h && inside(p)) load(i, p);
                        }
                    };
                    if constexpr (kMode == kDeviants) {
                        read([&](int i, int64_t p) {
                            A[i] = make_float4(gp.cls[cls][0][p], gp.cls[cls][1][p], gp.cls[cls][2][p], gp.cls[cls][3][p]);
                            B[i] = make_float2(gp.cls[cls][4][p], gp.pat2[p].y);
                        });
                    } else {
                        read([&](int i, int64_t p) {
                            A[i] = gp.pat4[p];
                            B[i] = gp.pat2[p];
                        });
                    }
                    if constexpr (kMode == kAll) {
                        float sums[kRows][5];
#pragma unroll
                        for (int i = 0; i < kRows; ++i) {
                            uint32_t bits = __float_as_uint(B[i].y);
                            if (pix && (bits & kMixedBit)) {  // the patterns with the position
                                if (unplaced_pixel(bits)) bits = 0u;
#pragma unroll
                                for (int q = 0; q < 32; q += q ? 8 : 16)
                                    if (!((bits >> q) & RPD_SAMPLE_PIXEL_VALID)) bits &= ~(0xffu << q);
                            }
                            const PixPattern pp{A[i].x, A[i].y, A[i].z, A[i].w, B[i].x, uint8_t(bits), uint8_t(bits >> 8),
                                                {uint8_t(bits >> 16), uint8_t(bits >> 24)}};
                            class_sums(gp, cls, int64_t(s * step + k0 + i) * g.w + x, pp, sums[i]);
                        }
#pragma unroll
                        for (int i = 0; i < kRows; ++i) {
                            A[i] = make_float4(sums[i][0], sums[i][1], sums[i][2], sums[i][3]);
                            B[i].x = sums[i][4];
                        }
                    }
#pragma unroll
                    for (int i = 0; i < kRows; ++i) {
                        const uint32_t bits = __float_as_uint(B[i].y);
                        if (kMode == kPattern && deviant(bits)) continue;
                        if (kMode == kDeviants && (!deviant(bits) || unplaced_pixel(bits) == pix)) continue;
                        float4 a = A[i];
                        float s2l = B[i].x;
                        if (kMode == kPattern && (bits & 0xffu) != P) {
                            const int more = ((bits >> 16) & 0xffu) == P ? 0 : (bits >> 24) == P ? 1 : -1;
                            if (more < 0) continue;
                            const int64_t p = int64_t(s * step + k0 + i) * g.w + x;
                            a = make_float4(gp.cls[more][0][p], gp.cls[more][1][p], gp.cls[more][2][p], gp.cls[more][3][p]);
                            s2l = gp.cls[more][4][p];
                        }
                        const int k = k0 + i;
                        const uint32_t n = uint32_t(a.x), i0 = uint32_t(step - k), i1 = uint32_t(k);
                        const float f0 = float(i0) * inv_step, f1 = float(i1) * inv_step;
                        bw[0] += i0 * n;
                        bw[1] += i1 * n;
                        tw2 += i0 * i0 * n;
                        nw2 += i1 * i1 * n;
                        df_add_scaled(by[0].h, by[0].l, f0, a.y, a.z);
                        df_add_scaled(by[1].h, by[1].l, f1, a.y, a.z);
                        df_add_scaled(tz.h, tz.l, f0, a.w, s2l);
                        df_add_scaled(nz.h, nz.l, f1, a.w, s2l);
                    }
                }
                if (!__any_sync(0xffffffffu, bw[0] != 0u)) continue;
                tw += bw[0];
                nw += bw[1];
                df_add(ty.h, ty.l, by[0].h);
                ty.l += by[0].l;
                df_add(ny.h, ny.l, by[1].h);
                ny.l += by[1].l;
                if (!pix) continue;
                // the half cell's bin of each node: quarter v * 2 + t (t: 0 left, 1 right)
                uint32_t qw[4];
                DF qy[4];
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    qw[2 * v] = bw[v] * il;
                    qw[2 * v + 1] = bw[v] * ir;
                    qy[2 * v] = df_scaled(fl, by[v]);
                    qy[2 * v + 1] = df_scaled(fr, by[v]);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    for (int o = 1; o < half; o <<= 1) qw[q] += __shfl_xor_sync(0xffffffffu, qw[q], o);
                    df_group_sum(qy[q].h, qy[q].l, half);
                }
                const int hcell = (lane >> (sh - 1)) & 1;  // left or right half of the cell
                for (int q = lane & (half - 1); q < 4; q += half) {
                    const int node = cell + (q & 1), row = s + (q >> 1);
                    if (!owned(node) || !(q < 2 ? up : down)) continue;
                    const uint32_t W = q == 0 ? qw[0] : q == 1 ? qw[1] : q == 2 ? qw[2] : qw[3];
                    DF Y;
                    Y.h = q == 0 ? qy[0].h : q == 1 ? qy[1].h : q == 2 ? qy[2].h : qy[3].h;
                    Y.l = q == 0 ? qy[0].l : q == 1 ? qy[1].l : q == 2 ? qy[2].l : qy[3].l;
                    if (W == 0u) continue;
                    const int bin = ((q < 2 ? 2 : 0) + hs) * 4 + ((q & 1) ? 0 : 2) + hcell;
                    const float2 wv = int_weight_df(W, inv_w);
                    float2* e = grid + (int64_t(row) * g.nodes_x + c0 + node) * kDeps * kDepStride + bin;
                    float2 pw[kClasses], py[kClasses];
#pragma unroll
                    for (int c = 0; c < kClasses; ++c) {
                        pw[c] = py[c] = make_float2(0.0f, 0.0f);
                        if (!(P & class_bit(c)) || store_only) continue;
                        pw[c] = e[dep_screen(c) * kDepStride];
                        py[c] = e[dep_screen(c) * kDepStride + 16];
                    }
#pragma unroll
                    for (int c = 0; c < kClasses; ++c) {
                        if (!(P & class_bit(c))) continue;
                        df_add(pw[c].x, pw[c].y, wv.x);
                        pw[c].y += wv.y;
                        df_add(py[c].x, py[c].y, Y.h);
                        py[c].y += Y.l;
                        e[dep_screen(c) * kDepStride] = pw[c];
                        e[dep_screen(c) * kDepStride + 16] = py[c];
                    }
                }
            }
            if (!up || !__any_sync(0xffffffffu, tw != 0u)) continue;
            // node row s: per cell and side, then per node (its left cell's right part and its right
            // cell's left part)
            uint32_t wl = tw * il, wr = tw * ir;
            unsigned long long w2l = tw2 * (il * il), w2r = tw2 * (ir * ir);
            DF yl = df_scaled(fl, ty), yr = df_scaled(fr, ty), zl = df_scaled(fl, tz), zr = df_scaled(fr, tz);
            for (int o = 1; o < step; o <<= 1) {
                wl += __shfl_xor_sync(0xffffffffu, wl, o);
                wr += __shfl_xor_sync(0xffffffffu, wr, o);
                w2l += __shfl_xor_sync(0xffffffffu, w2l, o);
                w2r += __shfl_xor_sync(0xffffffffu, w2r, o);
            }
            df_group_sum(yl.h, yl.l, step);
            df_group_sum(yr.h, yr.l, step);
            df_group_sum(zl.h, zl.l, step);
            df_group_sum(zr.h, zr.l, step);
            // node `cell`, on this cell's left; the lanes of the last cell also take the one on its right
            const uint32_t aw = __shfl_up_sync(0xffffffffu, wr, step);
            const unsigned long long aw2 = __shfl_up_sync(0xffffffffu, w2r, step);
            const float ayh = __shfl_up_sync(0xffffffffu, yr.h, step), ayl = __shfl_up_sync(0xffffffffu, yr.l, step);
            const float azh = __shfl_up_sync(0xffffffffu, zr.h, step), azl = __shfl_up_sync(0xffffffffu, zr.l, step);
            for (int t = 0; t < (cell == cells - 1 ? 2 : 1); ++t) {
                const int node = cell + t;
                if (!owned(node)) continue;
                uint32_t W = t ? wr : wl;
                unsigned long long W2 = t ? w2r : w2l;
                DF Y = t ? yr : yl, Z = t ? zr : zl;
                if (!t && cell > 0) {
                    W += aw;
                    W2 += aw2;
                    df_add(Y.h, Y.l, ayh);
                    Y.l += ayl;
                    df_add(Z.h, Z.l, azh);
                    Z.l += azl;
                }
                if (W == 0u) continue;
                const float w2h = __ull2float_rz(W2);
                const float w2m = float(W2 - (unsigned long long)(w2h));
                const float2 add[4] = {int_weight_df(W, inv_w),
                                       make_float2(w2h * (inv_w * inv_w), w2m * (inv_w * inv_w)),
                                       make_float2(Y.h, Y.l), make_float2(Z.h, Z.l)};
                float2* e = grid + (int64_t(s) * g.nodes_x + c0 + node) * kDeps * kDepStride + 32;
                for (int d = col; d < kDeps; d += step) {  // the cell's lanes take a dependency each
                    const int c = (d + 1) >> 1;  // its class: dep_random(c) and dep_screen(c) in order
                    if (!(P & class_bit(c)) || !((d & 1) ? rnd : pix)) continue;
                    float2* ed = e + d * kDepStride;
                    float2 o[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) o[k] = store_only ? make_float2(0.0f, 0.0f) : ed[k];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        df_add(o[k].x, o[k].y, add[k].x);
                        o[k].y += add[k].y;
                        ed[k] = o[k];
                    }
                }
            }
            __syncwarp();
        }
        store_only = false;
    };
    int patterns = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) patterns += __popc(set.w[q]);
    // (where some samples lack the position, the screen's sums and the random dimensions' are a walk each)
    if (patterns + (classes ? kClasses : 0) + (unplaced ? kClasses - 1 : 0) > (mixed ? 2 * tp.many : tp.many)) {
        // (each walk's entries are its own: the parts need no order; zero entries stay to be written)
#pragma unroll 1
        for (int q = part; q < (mixed ? 2 * kClasses - 1 : kClasses); q += tp.parts) {
            const int c = q < kClasses ? q : q - kClasses + 1;
            store_only = tp.fresh != 0;
            walk(std::integral_constant<int, kAll>{}, class_bit(c), c, q < kClasses, !mixed || q >= kClasses);
        }
        return;
    }
    if (part > 0) return;
    for (uint32_t P = set.pop(); P != 0u; P = set.pop())
        walk(std::integral_constant<int, kPattern>{}, P, 0, (P & RPD_SAMPLE_PIXEL_VALID) != 0, true);
    if (!classes && !unplaced) return;
#pragma unroll 1
    for (int c = classes ? 0 : kClasses; c < 2 * kClasses; ++c) {
        if (c == kClasses && !unplaced) return;
        if (c != kClasses)  // (class 0 is the screen)
            walk(std::integral_constant<int, kDeviants>{}, class_bit(c % kClasses), c % kClasses, c < kClasses, true);
    }
}

// What k_grid_totals leaves out, one warp per node. It takes every sample of a pixel in the pixel's
// nominal screen bin: a pixel some of whose samples may not be (a position within 2^-12 of the
// pixel's end, or outside it) is looked over sample by sample here, and a sample that the reference
// bins elsewhere is moved (very few are). A deviant pixel's samples that lack the position are taken out
// of the screen's sums. A pattern at a time, whose samples enter every class it holds. Where a node has many odd
// pixels (positions all over the place) the first pattern looked for is the first pixel's first, and the
// others turn up meanwhile; where it has a few (seven in a 1920x1080x16 frame), hardly any of their samples count, and
// a first walk notes the patterns and, up to kOddPicks of them, the samples.
// Blocks of one warp take the listed nodes in turn; each node is one warp's, in a fixed order.
constexpr int kOddPicks = 64;
struct OddPicks {
    int64_t sample[kOddPicks];
    uint16_t pixel[kOddPicks];
};
__device__ void odd_node(const GridParams& gpar, float2* grid, const DeviceSamples& s, const int64_t* offsets,
                         const GridPrep& gp, int64_t node, float* sm) {
    const int lane = threadIdx.x;
    const Geometry& g = gpar.g;
    const int nx = int(node % g.nodes_x), ny = int(node / g.nodes_x);
    const int step = g.step, sh = __ffs(step) - 1;
    const float wscale = float(step) * float(step), inv_wscale = 1.0f / wscale;
    LaneBins<false> bins{sm, lane, wscale};
    OddPicks& picks = *reinterpret_cast<OddPicks*>(sm + LaneBins<false>::kSlots * 32);
    uint16_t* list = reinterpret_cast<uint16_t*>(&picks + 1);
    float2* base = grid + node * kDeps * kDepStride;
    const float support = float(g.support);
    const float half_support = 0.5f * support;
    const float support_left = float(nx * step) - half_support;
    const float support_top = float(ny * step) - half_support;
    // the pixels the node weighs: strictly within a step of it
    const int xlo = imaxs(0, (nx - 1) * step + 1), xhi = imins(g.w - 1, (nx + 1) * step - 1);
    const int ylo = imaxs(0, (ny - 1) * step + 1), yhi = imins(g.h - 1, (ny + 1) * step - 1);
    int nodd = 0;
    // one row of 2 step - 1 pixels (or two, for steps up to 8) at a time
    const int lw = step <= 8 ? 16 : 32, rows = 32 / lw;
    const int lx = lane & (lw - 1), lr = lane / lw;
    // in batches, their loads before any is used: the scan was most of a node's time, a chain of one load
    // latency per row (the grid's totals and screen bins of 1920x1080x16, where a block takes two nodes in turn:
    // 117 -> 108 us; 98 us with the odd pixels' samples spread over the lanes below)
    constexpr int kBatch = 8;
    constexpr int kMixedEntry = 0x8000;  // a mixed_deviant
    const int x = xlo + lx;
    for (int yb = ylo; yb <= yhi; yb += rows * kBatch) {
        uint32_t bits[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const int y = yb + b * rows + lr;
            const int64_t idx = int64_t(y) * g.w + x;
            const bool in = x <= xhi && y <= yhi && idx >= gpar.first && idx < gpar.first + gpar.count;
            bits[b] = in ? __float_as_uint(gp.pat2[idx].y) : uint32_t(kPixUniform) << 8;  // not odd
        }
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            const bool odd = odd_pixel(bits[b]);
            const unsigned m = __ballot_sync(0xffffffffu, odd);
            if (odd) list[nodd + __popc(m & ((1u << lane) - 1))] = uint16_t((mixed_deviant(bits[b]) ? kMixedEntry : 0) | ((yb + b * rows + lr - ylo) * 64 + x - xlo));
            nodd += __popc(m);
        }
    }
    if (nodd == 0) return;
    __syncwarp();
    auto pixel = [&](int i, int& x, int& y, int64_t& idx) {
        x = xlo + (list[i] & 63);
        y = ylo + ((list[i] & (kMixedEntry - 1)) >> 6);
        idx = int64_t(y) * g.w + x;
    };
    auto weight = [&](int x, int y) {
        return float(axis_ifactor(x, nx, g.nodes_x, sh) * axis_ifactor(y, ny, g.nodes_y, sh)) * inv_wscale;
    };
    auto exact_bin = [&](int x, int y, int64_t k) {  // main.cpp:352-357
        const float su = fclamps((float(x) + sample_pu(s, 0, k) - support_left) / support, 0.0f, 1.0f);
        const float sv = fclamps((float(y) + sample_pu(s, 1, k) - support_top) / support, 0.0f, 1.0f);
        return bin2d(su, sv);
    };
    auto nominal_bin = [&](int x, int y) {
        return ((y - (ny - 1) * step) >> (sh - 1)) * 4 + ((x - (nx - 1) * step) >> (sh - 1));
    };
    const bool has_pu = s.compact ? s.c16.pixel_u[0] && s.c16.pixel_u[1] : s.pixel_u[0] && s.pixel_u[1];
    // f(ok, i, x, y, k) for every sample k of the odd pixels (i: the pixel's list entry), the lanes in step (ok: the
    // lane has one; else k is some sample): a uniform push's pixels and samples are one range over the lanes,
    // with per-pixel counts eight lanes take a pixel
    auto for_samples = [&](auto f) {
        int x, y;
        int64_t idx;
        if (gpar.spp > 0) {
            const int total = nodd * gpar.spp;
            for (int t0 = 0; t0 < total; t0 += 32) {
                const int t = imins(t0 + lane, total - 1), i = t / gpar.spp;
                pixel(i, x, y, idx);
                f(t0 + lane < total, i, x, y, (idx - gpar.first) * gpar.spp + (t - i * gpar.spp));
            }
            return;
        }
        for (int i0 = 0; i0 < nodd; i0 += 4) {
            const int i = imins(i0 + (lane >> 3), nodd - 1);
            pixel(i, x, y, idx);
            const int64_t kend = i0 + (lane >> 3) < nodd ? offsets[idx - gpar.first + 1] : 0;
            for (int64_t k = offsets[idx - gpar.first] + (lane & 7); __any_sync(0xffffffffu, k < kend); k += 8)
                f(k < kend, i, x, y, k < kend ? k : 0);
        }
    };
    auto pattern_of = [](uint32_t key) {
        uint32_t p = 0u;
#pragma unroll
        for (int c = 0; c < kClasses; ++c)
            if (!(key & key_absent_bit(c))) p |= class_bit(c);
        return p;
    };
    // is pixel i's sample one for the sums below? (b: its bin; without a pixel_u plane no key says that there is one)
    auto counts = [&](uint32_t key, int i, int x, int y, int b) {
        return key & key_absent_bit(0) ? key != kKeyNone && (list[i] & kMixedEntry) : b != nominal_bin(x, y);
    };
    PatternSet others;
    uint32_t P;
    int found = 0;
    const bool many = 8 * nodd > (xhi - xlo + 1) * (yhi - ylo + 1);  // more than an eighth of its pixels
    if (many) {
        int px, py;
        int64_t idx;
        pixel(0, px, py, idx);
        P = __float_as_uint(gp.pat2[idx].y) & 0xffu;
    } else {
        for_samples([&](bool ok, int i, int x, int y, int64_t k) {
            const uint32_t key = gp.key[k];
            const int b = has_pu ? exact_bin(x, y, k) : 0;
            const bool pick = ok && counts(key, i, x, y, b);
            const unsigned m = __ballot_sync(0xffffffffu, pick);
            if (m == 0u) return;
            if (pick) {
                others.add(pattern_of(key));
                const int at = found + __popc(m & ((1u << lane) - 1));
                if (at < kOddPicks) {
                    picks.sample[at] = k;
                    picks.pixel[at] = uint16_t(i);
                }
            }
            found += __popc(m);
        });
        others.unite_warp();
        P = others.pop();
        __syncwarp();
    }
    for (bool gather = many; P != 0u; gather = false) {
        Totals lost;
        bins.clear();
        __syncwarp();
        auto add = [&](bool ok, int i, int x, int y, int64_t k) {
            const uint32_t key = gp.key[k];
            const float yv = gp.lum[k];
            const int b = has_pu ? exact_bin(x, y, k) : 0;
            if (!ok || !counts(key, i, x, y, b)) return;
            const uint32_t pat = pattern_of(key);
            if (pat != P) {
                if (gather) others.add(pat);
                return;
            }
            const float w = weight(x, y);
            const int b0 = nominal_bin(x, y);
            bins.add_weight(b0, -w, 1.0f);
            bins.add_sum(b0, -w, yv, 0.0f);
            if (key & key_absent_bit(0)) {
                add_sample(lost, w, yv);
            } else {
                bins.add_weight(b, w, 1.0f);
                bins.add_sum(b, w, yv, 0.0f);
            }
        };
        if (many || found > kOddPicks) {
            for_samples(add);
        } else {
            for (int e = lane; e < found; e += 32) {
                int x, y;
                int64_t idx;
                const int i = picks.pixel[e];
                pixel(i, x, y, idx);
                add(true, i, x, y, picks.sample[e]);
            }
        }
        const float2 v = bins.reduce_value();
        float2 t[4];
        reduce_totals(lost, t);  // zeros for a pattern with the position
#pragma unroll
        for (int c = 0; c < kClasses; ++c) {
            if (!(P & class_bit(c))) continue;
            float2* e = base + dep_screen(c) * kDepStride;
            if (v.x != 0.0f || v.y != 0.0f) df_accum(e + lane, v.x, v.y);
            if (lane != 0) continue;
            for (int q = 0; q < 4; ++q)
                if (t[q].x != 0.0f || t[q].y != 0.0f) df_accum(e + 32 + q, -t[q].x, -t[q].y);
        }
        __syncwarp();
        if (gather) others.unite_warp();
        P = others.pop();
    }
}

__global__ void __launch_bounds__(32) k_grid_odd(GridParams gpar, float2* grid, DeviceSamples s, const int64_t* offsets,
                                                 GridPrep gp, const unsigned* odd_count, const int32_t* odd_nodes) {
    extern __shared__ float sm[];
    const unsigned n = *odd_count;
    for (unsigned k = blockIdx.x; k < n; k += gridDim.x) {
        odd_node(gpar, grid, s, offsets, gp, odd_nodes[k], sm);
        __syncwarp();
    }
}

// ---- random-dimension bins (Dependency2D::add / BinnedDependency::add of brdf, lens,
// light_uv, environment, light_select and rr; main.cpp:356-375) --------------------------
//
// One block per node: RW row groups x DS dimension sets of warps. A warp walks the samples of
// its row group's support rows as one flat stream (lanes over consecutive samples: coalesced,
// 16-byte loads of 4 samples when possible) and updates, for each sample, the bins of the
// dimensions of its set. Every lane owns private bins in shared memory ([slot][lane], conflict
// free; a dimension the sample does not carry updates a per-lane trash slot instead, so the
// update has no branches). The block combines row groups and lanes in a fixed order at the
// end: deterministic, no atomics.
constexpr int kRandDims = 6;
constexpr int kAllDims = 0x3f, kNoEnvDims = 0x37;  // dimension masks (bit d: dimension d)
constexpr int kRandSlots = 5 * 16 + 2;  // brdf, lens, light_uv, environment, light_select; rr has 2 bins
// d: 0 brdf, 1 lens, 2 light_uv, 3 environment, 4 light_select, 5 rr (grid group d + 1)
__host__ __device__ constexpr int rand_slot0(int d) { return d * 16; }
__host__ __device__ constexpr int rand_dep(int d) {
    return d == 0 ? D_BRDF : d == 1 ? D_LENS : d == 2 ? D_LIGHT_UV : d == 3 ? D_ENV : d == 4 ? D_LIGHT_SELECT : D_RR;
}
__host__ __device__ constexpr uint32_t rand_mask(int d) { return d == 5 ? 1u : 15u; }

// The six dimensions split into DS sets (one warp of a row group each): fewer private bins per
// warp (more resident warps) at the price of walking the samples once per set.
template <int DS>
__host__ __device__ constexpr int dim_set(int d) {
    return DS == 1 ? 0 : DS == 2 ? ((d == 0 || d == 1 || d == 5) ? 0 : 1)
                                 : ((d == 0 || d == 5) ? 0 : (d == 1 || d == 4) ? 1 : 2);
}
// first slot of dimension d within its set's region
template <int DS>
__host__ __device__ constexpr int dim_slot0(int d) {
    return DS == 1 ? d * 16 : DS == 2 ? (d == 0 ? 0 : d == 1 ? 16 : d == 5 ? 32 : d == 2 ? 0 : d == 3 ? 16 : 32)
                                      : ((d == 0 || d == 1 || d == 2) ? 0 : 16);
}
// slots of the largest set, plus the trash slot
template <int DS>
__host__ __device__ constexpr int set_slots() { return DS == 1 ? kRandSlots : DS == 2 ? 48 : 32; }

struct RandParams {
    GridParams gp;
    uint32_t spp_magic;  // floor(k / spp) == umulhi(k, magic) for every in-segment k (0: search)
    int spp_shift;       // spp is 2^shift (-1: not a power of two)
    int cols;            // support columns of a node, 2 * step + 3 (shared-memory tables)
    // a launch that runs only when the push's largest per-pixel count (*max_count, in device
    // memory) is at most (max_mode 1) or above (max_mode 2) max_limit; max_mode 0: always runs
    const int64_t* max_count;
    int64_t max_limit;
    int max_mode;
    float2* target;  // the grid the pass adds to (the pass grid or, in pairs, the frame grid)
};

template <int WB, int DS>
struct RandLayout {
    // per warp: weights [slots][32] (WB bytes each: u16 or u32 exact integers, or float2
    // double-float), then sums [slots][32] float2; slot kTrash absorbs the updates of absent
    // dimensions
    static constexpr int kTrash = set_slots<DS>();
    static constexpr int kSlots = kTrash + 1;
    static constexpr int kWeightBytes = kSlots * 32 * WB;
    static constexpr int kWarpBytes = kWeightBytes + kSlots * 32 * 8;
};

// Per-warp table of the row segments a warp walks (one chunk of up to 32 support rows).
struct RowTable {
    int64_t k0[32];    // first sample of the segment
    int base[33];      // prefix of the segment lengths (flat sample index of the segment start)
    int col0[32];      // column-factor index of the segment's first pixel
    float ay[32];      // the row's y factor
    int p0[32];        // first pixel of the segment, relative to the push (varying counts)
    int npx[32];       // pixels in the segment
    int len[32];       // samples in the segment
};

// Everything a warp's walk needs.
template <int WB, int DS>
struct WalkCtx {
    std::conditional_t<WB == 2, uint16_t, uint32_t>* wint;
    float2* wdf;
    float2* sums;
    RowTable* rt;
    const float* xf;
    int lane;
    int xlo;          // image column of xf[0]
    float wscale;
};

// One sample: add w (weights) and w*y (sums) to the bin of every dimension of set SET the
// sample carries; dimensions outside the mask DIMS are never valid in the push's keys (their
// sample planes are absent) and are skipped. Absent dimensions (and w <= 1e-8, which BinnedDependency::add skips,
// core/stats.h:103) go to the trash slot with the same arithmetic.
template <int WB, int DS, int SET, int DIMS>
__device__ __forceinline__ void rand_update(const WalkCtx<WB, DS>& c, uint32_t key, float w, uint32_t iw,
                                            float y) {
    constexpr bool INT_W = WB != 8;
    using L = RandLayout<WB, DS>;
    const bool wok = w > 1e-8f;
    const float wy = w * y;
    const float wye = __fmaf_rn(w, y, -wy);
    int slot[kRandDims];
    uint32_t wi[kRandDims];
    float2 wd[kRandDims], sy[kRandDims];
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (dim_set<DS>(d) != SET || !((DIMS >> d) & 1)) continue;
        const bool on = wok && (key & key_absent_bit(d + 1)) == 0;
        const int bin = int((key >> key_shift(d + 1)) & rand_mask(d));
        slot[d] = (on ? dim_slot0<DS>(d) + bin : L::kTrash) * 32 + c.lane;
    }
    // the dimensions own disjoint slot ranges (the trash slot is only ever a sink): load all,
    // update, store all
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (dim_set<DS>(d) != SET || !((DIMS >> d) & 1)) continue;
        if (INT_W) wi[d] = c.wint[slot[d]];
        else wd[d] = c.wdf[slot[d]];
        sy[d] = c.sums[slot[d]];
    }
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (dim_set<DS>(d) != SET || !((DIMS >> d) & 1)) continue;
        if (INT_W) wi[d] += iw;
        else df_add(wd[d].x, wd[d].y, w);
        df_add(sy[d].x, sy[d].y, wy);
        sy[d].y += wye;
    }
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (dim_set<DS>(d) != SET || !((DIMS >> d) & 1)) continue;
        if (INT_W) c.wint[slot[d]] = wi[d];
        else c.wdf[slot[d]] = wd[d];
        c.sums[slot[d]] = sy[d];
    }
}

// Walk modes: samples one by one (0); quads of 4 samples of one pixel (1, uniform counts); aligned
// quads of 4 consecutive samples of the push with each sample's column (2, per-pixel counts).
constexpr int kWalkScalar = 0, kWalkPixelQuads = 1, kWalkColumnQuads = 2;

// The flat walk of one row-segment chunk (total samples, or total quads in the quad modes) for
// dimension set SET.
template <int WB, int DS, int SET, int MODE, int DIMS>
__device__ __forceinline__ void rand_walk(const WalkCtx<WB, DS>& c, const RandParams& rp, const GridPrep& gp,
                                          const int64_t* offsets, int total) {
    constexpr bool INT_W = WB != 8;
    const RowTable* rt = c.rt;
    const int lane = c.lane;
    int r = 0;  // current segment of this lane (monotone along its walk)
    if (MODE == kWalkColumnQuads) {
        // Quads of the push's samples 4Q .. 4Q+3 (16-byte loads of keys and luminances, 8 bytes of
        // columns; the sample planes are padded to a multiple of 64 samples). A quad may start
        // before the segment or run past it: those samples weigh nothing (the trash slot). The
        // weights are formed when the quad is processed, one batch after its loads were issued.
        constexpr int U = 2;
        const int nq = total;
        auto fetchq = [&](int q, uint4& kq, float4& yq, uint2& cq, int64_t& k4, int& seg) {
            kq = make_uint4(0u, 0u, 0u, 0u);
            yq = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            cq = make_uint2(0u, 0u);
            k4 = 0;
            seg = -1;
            if (q >= nq) return;
            while (q >= rt->base[r + 1]) ++r;
            k4 = ((rt->k0[r] >> 2) + (q - rt->base[r])) << 2;
            kq = *reinterpret_cast<const uint4*>(gp.key + k4);
            yq = *reinterpret_cast<const float4*>(gp.lum + k4);
            cq = *reinterpret_cast<const uint2*>(gp.col + k4);
            seg = r;
        };
        uint4 nk[U];
        float4 nyv[U];
        uint2 ncq[U];
        int64_t nk4[U];
        int nseg[U];
#pragma unroll
        for (int u = 0; u < U; ++u) fetchq(lane + 32 * u, nk[u], nyv[u], ncq[u], nk4[u], nseg[u]);
        for (int q0 = 0; q0 < nq; q0 += 32 * U) {
            uint4 ck[U];
            float4 cy[U];
            uint2 ccq[U];
            int64_t ck4[U];
            int cseg[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ck[u] = nk[u];
                cy[u] = nyv[u];
                ccq[u] = ncq[u];
                ck4[u] = nk4[u];
                cseg[u] = nseg[u];
            }
            if (q0 + 32 * U < nq) {
#pragma unroll
                for (int u = 0; u < U; ++u) fetchq(q0 + 32 * U + lane + 32 * u, nk[u], nyv[u], ncq[u], nk4[u], nseg[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (cseg[u] >= 0) {
                    const int64_t ks = rt->k0[cseg[u]], ke = ks + rt->len[cseg[u]];
                    const float ay = rt->ay[cseg[u]];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int64_t k = ck4[u] + i;
                        const int ci = int(((i < 2 ? ccq[u].x : ccq[u].y) >> (16 * (i & 1))) & 0xffffu) - c.xlo;
                        if (k >= ks && k < ke && unsigned(ci) < unsigned(rp.cols)) w[i] = c.xf[ci] * ay;
                    }
                }
                rand_update<WB, DS, SET, DIMS>(c, ck[u].x, w[0], INT_W ? uint32_t(w[0] * c.wscale) : 0u, cy[u].x);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].y, w[1], INT_W ? uint32_t(w[1] * c.wscale) : 0u, cy[u].y);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].z, w[2], INT_W ? uint32_t(w[2] * c.wscale) : 0u, cy[u].z);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].w, w[3], INT_W ? uint32_t(w[3] * c.wscale) : 0u, cy[u].w);
            }
        }
    } else if (MODE == kWalkPixelQuads) {
        // quads of 4 consecutive samples of one pixel (the samples per pixel are a power of two
        // >= 4 and every segment starts 16-byte aligned): one 16-byte load of keys and one of
        // luminances per quad, 2 quads per lane in flight
        constexpr int U = 2;
        const int nq = total >> 2;
        auto fetchq = [&](int q, uint4& kq, float4& yq, float& w) {
            kq = make_uint4(0u, 0u, 0u, 0u);
            yq = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w = 0.0f;
            if (q >= nq) return;
            const int t = q << 2;
            while (t >= rt->base[r + 1]) ++r;
            const int kk = t - rt->base[r];
            const int64_t k = rt->k0[r] + kk;
            kq = *reinterpret_cast<const uint4*>(gp.key + k);
            yq = *reinterpret_cast<const float4*>(gp.lum + k);
            w = c.xf[rt->col0[r] + (kk >> rp.spp_shift)] * rt->ay[r];
        };
        uint4 nk[U];
        float4 nyv[U];
        float nw[U];
#pragma unroll
        for (int u = 0; u < U; ++u) fetchq(lane + 32 * u, nk[u], nyv[u], nw[u]);
        for (int q0 = 0; q0 < nq; q0 += 32 * U) {
            uint4 ck[U];
            float4 cy[U];
            float cw[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ck[u] = nk[u];
                cy[u] = nyv[u];
                cw[u] = nw[u];
            }
            if (q0 + 32 * U < nq) {
#pragma unroll
                for (int u = 0; u < U; ++u) fetchq(q0 + 32 * U + lane + 32 * u, nk[u], nyv[u], nw[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t iw = INT_W ? uint32_t(cw[u] * c.wscale) : 0u;
                rand_update<WB, DS, SET, DIMS>(c, ck[u].x, cw[u], iw, cy[u].x);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].y, cw[u], iw, cy[u].y);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].z, cw[u], iw, cy[u].z);
                rand_update<WB, DS, SET, DIMS>(c, ck[u].w, cw[u], iw, cy[u].w);
            }
        }
    } else {
        // A fetch returns the sample's column-factor index and row factor, not its weight: with
        // per-pixel counts the index comes from a load, and looking the factor up at fetch time
        // would wait for that load before the samples already fetched are processed.
        constexpr int U = 4;  // samples per lane in flight
        auto fetch = [&](int t, uint32_t& key, float& y, int& ci, float& ay) {
            key = 0u;
            y = 0.0f;
            ci = -1;
            ay = 0.0f;
            if (t >= total) return;
            while (t >= rt->base[r + 1]) ++r;
            const int kk = t - rt->base[r];
            const int64_t k = rt->k0[r] + kk;
            key = gp.key[k];
            y = gp.lum[k];
            ay = rt->ay[r];
            if (gp.col) {  // per-pixel counts: the statistics pass stored each sample's column
                ci = int(gp.col[k]) - c.xlo;
                return;
            }
            int pl;
            if (rp.spp_shift >= 0) {
                pl = kk >> rp.spp_shift;
            } else if (rp.spp_magic) {
                pl = int(__umulhi(uint32_t(kk), rp.spp_magic));
            } else {
                const int64_t* off = offsets + rt->p0[r];
                int lo = 0, hi = rt->npx[r] - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (off[mid] <= k) lo = mid; else hi = mid - 1;
                }
                pl = lo;
            }
            ci = rt->col0[r] + pl;
        };
        uint32_t nk[U];
        float nyv[U], nay[U];
        int nci[U];
#pragma unroll
        for (int u = 0; u < U; ++u) fetch(lane + 32 * u, nk[u], nyv[u], nci[u], nay[u]);
        for (int t0 = 0; t0 < total; t0 += 32 * U) {
            uint32_t ck[U];
            float cy[U], cw[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ck[u] = nk[u];
                cy[u] = nyv[u];
                cw[u] = unsigned(nci[u]) < unsigned(rp.cols) ? c.xf[nci[u]] * nay[u] : 0.0f;
            }
            if (t0 + 32 * U < total) {
#pragma unroll
                for (int u = 0; u < U; ++u) fetch(t0 + 32 * U + lane + 32 * u, nk[u], nyv[u], nci[u], nay[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                rand_update<WB, DS, SET, DIMS>(c, ck[u], cw[u], INT_W ? uint32_t(cw[u] * c.wscale) : 0u, cy[u]);
        }
    }
}

template <int WB, int RW, int DS, int MODE, int DIMS>
__global__ void __launch_bounds__(RW * DS * 32) k_grid_random(RandParams rp, float2* pass_grid,
                                                              const int64_t* offsets, GridPrep gp) {
    constexpr bool INT_W = WB != 8;
    using WT = std::conditional_t<WB == 2, uint16_t, uint32_t>;
    constexpr int NW = RW * DS;
    constexpr int VPT = (2 * kRandSlots + NW * 32 - 1) / (NW * 32);  // combined values per thread
    if (rp.max_mode != 0 && ((*rp.max_count <= rp.max_limit) != (rp.max_mode == 1))) return;  // the other form runs
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using L = RandLayout<WB, DS>;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int dset = warp % DS;     // the dimension set of this warp
    const int rgroup = warp / DS;   // its row group
    const GridParams& gpar = rp.gp;
    const Geometry& g = gpar.g;
    const int64_t node = rp.gp.node0 + blockIdx.x;
    const int nx = int(node % g.nodes_x), ny = int(node / g.nodes_x);
    unsigned char* wbase = smem_raw + warp * L::kWarpBytes;
    WalkCtx<WB, DS> c;
    c.wint = reinterpret_cast<WT*>(wbase);
    c.wdf = reinterpret_cast<float2*>(wbase);
    c.sums = reinterpret_cast<float2*>(wbase + L::kWeightBytes);
    c.rt = reinterpret_cast<RowTable*>(smem_raw + NW * L::kWarpBytes) + warp;
    float* xf = reinterpret_cast<float*>(reinterpret_cast<RowTable*>(smem_raw + NW * L::kWarpBytes) + NW);
    c.xf = xf;
    c.lane = lane;
    c.wscale = float(g.step) * float(g.step);
    RowTable* rt = c.rt;

    // the grid entries this thread adds to at the end, read now so the loads overlap the walk
    float2 prev[VPT];
    int64_t gidx[VPT];
#pragma unroll
    for (int vi = 0; vi < VPT; ++vi) {
        const int v = threadIdx.x + vi * NW * 32;
        gidx[vi] = -1;
        prev[vi] = make_float2(0.0f, 0.0f);
        if (v < 2 * kRandSlots) {
            const bool is_w = v < kRandSlots;
            const int gslot = is_w ? v : v - kRandSlots;
            int d = 0;
            while (d < kRandDims - 1 && gslot >= rand_slot0(d + 1)) ++d;
            const int bin = gslot - rand_slot0(d);
            gidx[vi] = (node * kDeps + rand_dep(d)) * kDepStride + (is_w ? bin : 16 + bin);
            prev[vi] = pass_grid[gidx[vi]];
        }
    }
    const int xlo = imaxs(0, (nx - 1) * g.step - 1), xhi = imins(g.w - 1, (nx + 1) * g.step + 1);
    const int ylo = imaxs(0, (ny - 1) * g.step - 1), yhi = imins(g.h - 1, (ny + 1) * g.step + 1);
    c.xlo = xlo;
    for (int col = threadIdx.x; col < rp.cols; col += NW * 32)
        xf[col] = (xlo + col <= xhi) ? axis_factor(gpar, xlo + col, nx, g.nodes_x) : 0.0f;
    for (int k = 0; k < L::kSlots; ++k) {
        if (INT_W) c.wint[k * 32 + lane] = 0u;
        else c.wdf[k * 32 + lane] = make_float2(0.0f, 0.0f);
        c.sums[k * 32 + lane] = make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    int xa = xhi + 1, xb = xlo - 1;  // the columns with x factor > 0
    for (int x = xlo; x <= xhi; ++x)
        if (xf[x - xlo] > 0.0f) {
            xa = imins(xa, x);
            xb = imaxs(xb, x);
        }
    const int nrows = (yhi - ylo) / RW + 1;  // rows ylo + rgroup + RW * j

    for (int c0 = 0; c0 < nrows; c0 += 32) {
        // ---- this chunk's row segments, one lane per row ----
        const int y = ylo + rgroup + RW * (c0 + lane);
        int n = 0;  // the walk's units in the segment: samples, or quads in the column-quad mode
        if (c0 + lane < nrows && y <= yhi && xa <= xb) {
            const float ay = axis_factor(gpar, y, ny, g.nodes_y);
            int64_t p0 = int64_t(y) * g.w + xa, p1 = int64_t(y) * g.w + xb + 1;
            p0 = p0 < gpar.first ? gpar.first : p0;
            p1 = p1 > gpar.first + gpar.count ? gpar.first + gpar.count : p1;
            if (ay > 0.0f && p0 < p1) {
                const int64_t k0 = sample_offset(offsets, gpar.spp, p0 - gpar.first);
                const int len = int(sample_offset(offsets, gpar.spp, p1 - gpar.first) - k0);
                n = MODE == kWalkColumnQuads ? (len > 0 ? int(((k0 + len - 1) >> 2) - (k0 >> 2) + 1) : 0) : len;
                rt->k0[lane] = k0;
                rt->len[lane] = len;
                rt->col0[lane] = int(p0 - int64_t(y) * g.w) - xlo;
                rt->ay[lane] = ay;
                rt->p0[lane] = int(p0 - gpar.first);
                rt->npx[lane] = int(p1 - p0);
            }
        }
        int incl = n;  // inclusive scan of the segment lengths
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += v;
        }
        rt->base[lane + 1] = incl;
        if (lane == 0) rt->base[0] = 0;
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();
        if (dset == 0) rand_walk<WB, DS, 0, MODE, DIMS>(c, rp, gp, offsets, total);
        if (DS > 1 && dset == 1) rand_walk<WB, DS, 1, MODE, DIMS>(c, rp, gp, offsets, total);
        if (DS > 2 && dset == 2) rand_walk<WB, DS, 2, MODE, DIMS>(c, rp, gp, offsets, total);
        __syncwarp();
    }
    __syncthreads();

    // combine: thread t owns values v = t + vi * NW*32 of [weights(kRandSlots), sums(kRandSlots)],
    // each summed over the row groups in order and over the 32 lanes in a rotated order
    // (32 different banks), two interleaved double-float chains per value
    int vslot[VPT], vset[VPT];
    bool vw[VPT];
#pragma unroll
    for (int vi = 0; vi < VPT; ++vi) {
        const int v = threadIdx.x + vi * NW * 32;
        const bool is_w = v < kRandSlots;
        const int gslot = is_w ? v : v - kRandSlots;
        int d = 0;
        while (d < kRandDims - 1 && gslot >= rand_slot0(d + 1)) ++d;
        vslot[vi] = dim_slot0<DS>(d) + (gslot - rand_slot0(d));
        vset[vi] = dim_set<DS>(d);
        vw[vi] = is_w;
    }
    uint64_t itot[VPT];
    float h[VPT][2], l[VPT][2];
#pragma unroll
    for (int vi = 0; vi < VPT; ++vi) {
        itot[vi] = 0;
        h[vi][0] = h[vi][1] = l[vi][0] = l[vi][1] = 0.0f;
    }
    for (int rg = 0; rg < RW; ++rg) {
        for (int i = 0; i < 32; i += 2) {
#pragma unroll
            for (int vi = 0; vi < VPT; ++vi) {
                if (gidx[vi] < 0) continue;
                const unsigned char* b = smem_raw + (rg * DS + vset[vi]) * L::kWarpBytes;
                const int v = threadIdx.x + vi * NW * 32;
                if (vw[vi] && INT_W) {
                    const WT* src = reinterpret_cast<const WT*>(b) + vslot[vi] * 32;
                    itot[vi] += uint64_t(src[(i + v) & 31]) + uint64_t(src[(i + 1 + v) & 31]);
                } else {
                    const float2* src =
                        reinterpret_cast<const float2*>(vw[vi] ? b : b + L::kWeightBytes) + vslot[vi] * 32;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 q = src[(i + j + v) & 31];
                        df_add(h[vi][j], l[vi][j], q.x);
                        l[vi][j] += q.y;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int vi = 0; vi < VPT; ++vi) {
        if (gidx[vi] < 0) continue;
        float oh, ol;
        if (vw[vi] && INT_W) {
            const float2 t = int_weight_df(itot[vi], 1.0f / c.wscale);
            oh = t.x;
            ol = t.y;
        } else {
            df_add(h[vi][0], l[vi][0], h[vi][1]);
            l[vi][0] += l[vi][1];
            oh = h[vi][0];
            ol = l[vi][0];
        }
        if (oh != 0.0f || ol != 0.0f) {
            float2 e = prev[vi];
            df_add(e.x, e.y, oh);
            e.y += ol;
            pass_grid[gidx[vi]] = e;
        }
    }
}


// ---- random-dimension bins, strip form -------------------------------------------------------------
//
// For uniform pushes over power-of-two node steps up to 32, where the bilinear weight of a pixel is
// the exact product of its row's and its column's multiple of 1/step. A lane owns an image column
// and walks down it: in a strip of `step` rows (between two node rows) it adds each sample to its
// private bins twice, times the row factor of the node row above and of the one below: two
// double-floats and one word of two 16-bit integer weights. At the
// strip's end the node row above is complete: its nodes' sums are the columns' bins times the
// column factors, and the node row below becomes the next strip's upper one. A sample is visited
// once instead of once per node it supports (four), and the walk needs neither row tables nor
// per-sample weights. A block's NC column warps cover NC * 32 columns and so NC * 32 / step - 1
// whole nodes of each of its `len` node rows (neighbouring blocks overlap by one cell, one strip);
// RG row groups split a strip's rows where there are too few blocks. Every sum is lane-private and
// combined in a fixed order: deterministic, no atomics.
// The bound is the shared-memory data path (for 32 samples, ten 128-byte wavefronts per dimension)
// with two warps per scheduler to hide its latency: the dimensions are split over two warps of a
// segment, whose bins share its 44 KB. At 1920x1080x16 without environment planes, one warp per
// node visiting every sample four times took 0.795 ms, this 0.387 ms (2048x1152x64: 2.75 -> 1.89 ms);
// with one warp for all dimensions and single updates 0.48 ms, with the two sets' warps on
// different schedulers 0.44 ms.
struct StripParams {
    Geometry g;
    int64_t first, count;
    int ny0, ny1;          // node rows of the launch
    int len;               // node rows of a block
    int col_blocks;        // blocks per `len` node rows
    int spp;
    int sh;                // log2 of the node step
    int fresh;             // the grid holds zeros (the frame's first push): nothing to read back
};

// slots of the dimensions in DIMS: each one's bins and a sink for samples without it
__host__ __device__ constexpr int strip_bins(int d) { return d == 5 ? 3 : 17; }
template <int DIMS>
__host__ __device__ constexpr int strip_slot0(int d) {
    int s = 0;
    for (int k = 0; k < d; ++k)
        if ((DIMS >> k) & 1) s += strip_bins(k);
    return s;
}
// the dimensions of warp set DS of two: brdf, lens and rr, or the rest
template <int DIMS>
__host__ __device__ constexpr int strip_set(int ds) { return DIMS & (ds == 0 ? 0x23 : 0x1c); }
template <int DIMS>
struct StripLayout {
    static constexpr int kSlots = strip_slot0<DIMS>(kRandDims);
    static constexpr int kHalf = kSlots * 32;                          // double-floats of one node row
    static constexpr int kSumBytes = 2 * kHalf * 8;
    static constexpr int kWarpBytes = kSumBytes + kSlots * 32 * 4;     // and two 16-bit weights
    // the segments' first and last node, shared with the next segment: (sum, weight) per slot,
    // doubled by strip parity
    static constexpr int edge_bytes(int nc) { return 2 * 2 * nc * kSlots * 12; }
};

// N (1 or 2) samples of one pixel in the dimensions of SET. Two samples' bins are all loaded before
// either is updated, and the second takes the first one's result where they meet in a bin, so that
// the two read-modify-writes overlap.
// BOTH: both node rows' sums; else only the one `sums` points at (the other's weight is 0).
template <int DIMS, int SET, int N, bool BOTH>
__device__ __forceinline__ void strip_update(uint32_t* wgt, float2* sums, const uint32_t* key, const float* y, float wa,
                                             float wb, uint32_t iw) {
    constexpr int kHalf = StripLayout<DIMS>::kHalf;
    float ya[N], yae[N], yb[N], ybe[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        ya[i] = wa * y[i];
        yae[i] = __fmaf_rn(wa, y[i], -ya[i]);
        yb[i] = wb * y[i];
        ybe[i] = __fmaf_rn(wb, y[i], -yb[i]);
    }
    uint32_t p[kRandDims][N], w[kRandDims][N];
    float2 s[kRandDims][N], r[kRandDims][N];
    // the dimensions own disjoint slots
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (!((SET >> d) & 1)) continue;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            p[d][i] = (((key[i] >> key_shift(d + 1)) & (d == 5 ? 3u : 31u)) + uint32_t(strip_slot0<DIMS>(d))) * 32u;
            w[d][i] = wgt[p[d][i]];
            s[d][i] = sums[p[d][i]];
            if (BOTH) r[d][i] = sums[p[d][i] + kHalf];
        }
    }
#pragma unroll
    for (int d = 0; d < kRandDims; ++d) {
        if (!((SET >> d) & 1)) continue;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (i > 0) {
                const bool same = p[d][i] == p[d][i - 1];
                w[d][i] = same ? w[d][i - 1] : w[d][i];
                s[d][i].x = same ? s[d][i - 1].x : s[d][i].x;
                s[d][i].y = same ? s[d][i - 1].y : s[d][i].y;
                if (BOTH) {
                    r[d][i].x = same ? r[d][i - 1].x : r[d][i].x;
                    r[d][i].y = same ? r[d][i - 1].y : r[d][i].y;
                }
            }
            w[d][i] += iw;
            df_add(s[d][i].x, s[d][i].y, ya[i]);
            s[d][i].y += yae[i];
            wgt[p[d][i]] = w[d][i];
            sums[p[d][i]] = s[d][i];
            if (BOTH) {
                df_add(r[d][i].x, r[d][i].y, yb[i]);
                r[d][i].y += ybe[i];
                sums[p[d][i] + kHalf] = r[d][i];
            }
        }
    }
}

// U samples of one pixel: keys and luminances (U = 8, 4: 16-byte loads; 1: scalar)
template <int U>
struct StripUnit {
    uint32_t key[U];
    float y[U];
};
template <int U>
__device__ __forceinline__ void strip_load(StripUnit<U>& u, const GridPrep& gp, int64_t k, bool in) {
#pragma unroll
    for (int i = 0; i < U; ++i) {
        u.key[i] = kKeyNone;
        u.y[i] = 0.0f;
    }
    if (!in) return;
    if constexpr (U == 1) {
        u.key[0] = gp.key[k];
        u.y[0] = gp.lum[k];
    } else {
#pragma unroll
        for (int i = 0; i < U; i += 4) {
            const uint4 a = *reinterpret_cast<const uint4*>(gp.key + k + i);
            const float4 b = *reinterpret_cast<const float4*>(gp.lum + k + i);
            u.key[i] = a.x, u.key[i + 1] = a.y, u.key[i + 2] = a.z, u.key[i + 3] = a.w;
            u.y[i] = b.x, u.y[i + 1] = b.y, u.y[i + 2] = b.z, u.y[i + 3] = b.w;
        }
    }
}

template <int NC, int RG, int U, int DIMS>
__global__ void __launch_bounds__(NC * RG * 64) k_grid_strips(StripParams sp, float2* grid, GridPrep gp) {
    using L = StripLayout<DIMS>;
    constexpr int NT = NC * RG * 64;  // two dimension sets
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_entry[L::kSlots];  // a slot's entry of a node's 13 x 36, -1 for a sink
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the two sets' warps of a segment are NC * RG apart, on the same one of the SM's four schedulers:
    // their unequal walks share its issue slots
    const int ds = warp / (NC * RG), rg = (warp / NC) % RG, cw = warp % NC;
    const Geometry& g = sp.g;
    const int step = g.step, sh = sp.sh;
    const int r0 = sp.ny0 + int(blockIdx.x / unsigned(sp.col_blocks)) * sp.len;  // the block's node rows
    const int r1 = imins(r0 + sp.len, sp.ny1);
    const int cells = 32 >> sh;                  // of a column warp (a segment)
    const int nb = NC * cells - 1;               // the block's nodes with both of their cells in it
    const int cb = int(blockIdx.x % unsigned(sp.col_blocks));
    const int c0 = cb * nb;                      // its first cell, between nodes c0 and c0 + 1
    const float inv_step = 1.0f / float(step);
    auto sums_of = [&](int w) { return reinterpret_cast<float2*>(smem_raw + w * L::kWarpBytes); };
    auto weights_of = [&](int w) { return reinterpret_cast<uint32_t*>(smem_raw + w * L::kWarpBytes + L::kSumBytes); };
    float2* edge_s = reinterpret_cast<float2*>(smem_raw + NC * RG * L::kWarpBytes);  // [parity][left, right][NC][slot]
    uint32_t* edge_w = reinterpret_cast<uint32_t*>(edge_s + 4 * NC * L::kSlots);
    float2* sums = sums_of(rg * NC + cw) + lane;
    uint32_t* wgt = weights_of(rg * NC + cw) + lane;
#pragma unroll 4
    for (int k = ds; k < L::kSlots; k += 2) {
        wgt[k * 32] = 0u;
        sums[k * 32] = sums[k * 32 + L::kHalf] = make_float2(0.0f, 0.0f);
    }
    for (int slot = threadIdx.x; slot < L::kSlots; slot += NT) {
        int en = -1;
#pragma unroll
        for (int d = 0; d < kRandDims; ++d) {
            if (!((DIMS >> d) & 1)) continue;
            const int bin = slot - strip_slot0<DIMS>(d);
            if (bin >= 0 && bin < strip_bins(d) - 1) en = rand_dep(d) * kDepStride + bin;
        }
        s_entry[slot] = en;
    }
    __syncthreads();

    const int x = c0 * step + cw * 32 + lane;
    const bool xin = x < g.w;
    const int upr = sp.spp / U;  // units of a pixel
    const int s0 = imaxs(r0 - 1, 0), s1 = r1;  // strips (the one below the last node row has no rows)
    const int ylast = imins(g.h, s1 * step) - 1;  // the block's last image row
    // the walk's next fetch: rows s0 * step + rg + RG j, the pixel's units of each
    int fy = s0 * step + rg, fu = 0;
    int64_t fp = int64_t(fy) * g.w + x - sp.first;
    auto fetch = [&](StripUnit<U>& u) {
        strip_load<U>(u, gp, fp * sp.spp + fu * U, xin && fy <= ylast && fp >= 0 && fp < sp.count);
        if (++fu == upr) {
            fu = 0;
            fy += RG;
            fp += int64_t(RG) * g.w;
        }
    };
    const int cell = lane >> sh, sub = lane & (step - 1);
    const int passes = (L::kSlots + step - 1) >> sh;
    auto add = [&](float2* e, float2 prev, float h, float l) {
        if (h == 0.0f && l == 0.0f) return;
        df_add(prev.x, prev.y, h);
        prev.y += l;
        *e = prev;
    };
    const float inv_w = inv_step * inv_step;

    StripUnit<U> a, b;
    fetch(a);
    fetch(b);
    for (int s = s0; s < s1; ++s) {
        // the node row above (s) uses the half s & 1 of every record, the one below the other half;
        // rows outside [r0, r1) are left out
        const int half = s & 1;
        const bool up = s >= r0, down = s + 1 < r1;
        for (int y = s * step + rg; y < imins((s + 1) * step, g.h); y += RG) {
            const int k = y - s * step;
            const uint32_t iu = up ? uint32_t(step - k) : 0u, id = down ? uint32_t(k) : 0u;
            const uint32_t iw = half ? id | (iu << 16) : iu | (id << 16);
            const float wu = float(iu) * inv_step, wd = float(id) * inv_step;
            const float wa = half ? wd : wu, wb = half ? wu : wd;
            constexpr int N = U >= 2 ? 2 : 1;
            for (int t = 0; t < upr; ++t) {
                const StripUnit<U> c = a;
                a = b;
                fetch(b);
                // a node row's own image row, and the strips at the block's ends, feed one node row
                auto go = [&](auto set, auto both, float2* to, float w0, float w1) {
#pragma unroll
                    for (int i = 0; i < U; i += N)
                        strip_update<DIMS, decltype(set)::value, N, decltype(both)::value>(wgt, to, c.key + i, c.y + i, w0,
                                                                                        w1, iw);
                };
                using Set0 = std::integral_constant<int, strip_set<DIMS>(0)>;
                using Set1 = std::integral_constant<int, strip_set<DIMS>(1)>;
                if (iu && id) {
                    if (ds == 0) go(Set0{}, std::true_type{}, sums, wa, wb);
                    else go(Set1{}, std::true_type{}, sums, wa, wb);
                } else if (iu | id) {
                    float2* to = sums + ((iu != 0) == (half == 0) ? 0 : L::kHalf);
                    const float w0 = iu ? wu : wd;
                    if (ds == 0) go(Set0{}, std::false_type{}, to, w0, 0.0f);
                    else go(Set1{}, std::false_type{}, to, w0, 0.0f);
                }
            }
        }
        if (!up) continue;  // the strip above the block's first node row: nothing complete yet
        // ---- node row s is complete. Lanes over the segment's cells and `step` slots at a time;
        // column c of a cell adds (step - c) / step of its bin to the node on the cell's left and
        // c / step to the one on its right (rotated by lane: the lanes read different banks), and
        // the bin is cleared for the node row after the next. ----
        __syncthreads();
        float2* es = edge_s + half * 2 * NC * L::kSlots;
        uint32_t* ew = edge_w + half * 2 * NC * L::kSlots;
        float2* row = grid + int64_t(s) * g.nodes_x * kDeps * kDepStride;
        const int node = c0 + cw * cells + cell;  // on the cell's left
        for (int ps = rg * 2 + ds; ps < passes; ps += RG * 2) {
            const int slot = (ps << sh) + sub;
            const int en = slot < L::kSlots ? s_entry[slot] : -1;
            const bool wr = en >= 0 && cell > 0 && node < g.nodes_x;
            float2* e = row + int64_t(node) * kDeps * kDepStride + en;
            float2 pw = make_float2(0.0f, 0.0f), py = pw;
            if (wr && !sp.fresh) {
                pw = e[0];
                py = e[16];
            }
            uint32_t wl = 0, wr_ = 0;
            float lh = 0.0f, ll = 0.0f, rh = 0.0f, rl = 0.0f;
            if (en >= 0) {
                for (int i = 0; i < step; ++i) {
                    const int c = (i + lane) & (step - 1);
                    const int at = slot * 32 + (cell << sh) + c;
                    const float fr = float(c) * inv_step, fl = float(step - c) * inv_step;
#pragma unroll
                    for (int r = 0; r < RG; ++r) {
                        float2* sv = sums_of(r * NC + cw) + half * L::kHalf + at;
                        uint16_t* wv = reinterpret_cast<uint16_t*>(weights_of(r * NC + cw)) + 2 * at + half;
                        const float2 v = *sv;
                        const uint32_t w = *wv;
                        *sv = make_float2(0.0f, 0.0f);
                        *wv = 0;
                        wl += w * uint32_t(step - c);
                        wr_ += w * uint32_t(c);
                        df_add_scaled(lh, ll, fl, v.x, v.y);
                        df_add_scaled(rh, rl, fr, v.x, v.y);
                    }
                }
            }
            if (en >= 0 && cell == 0) {
                es[cw * L::kSlots + slot] = make_float2(lh, ll);
                ew[cw * L::kSlots + slot] = wl;
            }
            if (en >= 0 && cell == cells - 1) {
                es[(NC + cw) * L::kSlots + slot] = make_float2(rh, rl);
                ew[(NC + cw) * L::kSlots + slot] = wr_;
            }
            if (cells > 1) {  // the part of the cell on the node's left
                const float ph = __shfl_up_sync(0xffffffffu, rh, step), pl = __shfl_up_sync(0xffffffffu, rl, step);
                wl += __shfl_up_sync(0xffffffffu, wr_, step);
                df_add(lh, ll, ph);
                ll += pl;
                if (wr) {
                    const float2 v = int_weight_df(wl, inv_w);
                    add(e, pw, v.x, v.y);
                    add(e + 16, py, lh, ll);
                }
            }
        }
        __syncthreads();
        // the nodes between two segments, and at the image's edges the block's first and last node
        const bool last = (c0 + nb + 1) * step >= g.w;
        for (int q = threadIdx.x; q < (NC + 1) * L::kSlots; q += NT) {
            const int seg = q / L::kSlots, slot = q % L::kSlots;
            const int en = s_entry[slot], nd = c0 + seg * cells;
            if (en < 0 || nd >= g.nodes_x || (seg == 0 && cb > 0) || (seg == NC && !last)) continue;
            float2* e = row + int64_t(nd) * kDeps * kDepStride + en;
            float2 pw = make_float2(0.0f, 0.0f), py = pw;
            if (!sp.fresh) {
                pw = e[0];
                py = e[16];
            }
            float2 v = make_float2(0.0f, 0.0f);
            uint32_t w = 0;
            if (seg > 0) {
                v = es[(NC + seg - 1) * L::kSlots + slot];
                w = ew[(NC + seg - 1) * L::kSlots + slot];
            }
            if (seg < NC) {
                const float2 l = es[seg * L::kSlots + slot];
                df_add(v.x, v.y, l.x);
                v.y += l.y;
                w += ew[seg * L::kSlots + slot];
            }
            const float2 wv = int_weight_df(w, inv_w);
            add(e, pw, wv.x, wv.y);
            add(e + 16, py, v.x, v.y);
        }
    }
}

}  // namespace

namespace {

// floor(k / spp) through a multiply-high: magic = ceil(2^32 / spp), checked for every k a
// row segment can hold (returns 0 when it does not hold, and the kernel searches instead)
uint32_t spp_magic_for(int spp, int max_k) {
    if (spp <= 0) return 0u;
    const uint64_t m = ((uint64_t(1) << 32) + uint64_t(spp) - 1) / uint64_t(spp);
    if (m > 0xffffffffull) return 0u;
    for (int k = 0; k < max_k; ++k)
        if (int((uint64_t(k) * m) >> 32) != k / spp) return 0u;
    return uint32_t(m);
}

template <int WB, int RW, int DS, int MODE, int DIMS>
cudaError_t launch_random_vec(Job& j, const RandParams& rp, const GridPrep& gp) {
    constexpr int NW = RW * DS;
    const size_t smem = size_t(NW) * RandLayout<WB, DS>::kWarpBytes + size_t(NW) * sizeof(RowTable) +
                        size_t(rp.cols) * sizeof(float);
    static FuncAttribute limit;
    const cudaError_t e = limit.at_least(reinterpret_cast<const void*>(&k_grid_random<WB, RW, DS, MODE, DIMS>),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, j.ctx->device, int64_t(smem));
    if (e != cudaSuccess) return e;
    const unsigned nblocks = unsigned(rp.gp.count_nodes);
    k_grid_random<WB, RW, DS, MODE, DIMS><<<nblocks, NW * 32, smem, j.stream>>>(rp, rp.target, j.offsets, gp);
    j.launches += 1;
    return cudaGetLastError();
}

// Pixel quads need samples per pixel a multiple of 4 (and a power of two, for the shift) with
// 16-byte aligned key and luminance planes; column quads need the per-sample columns (per-pixel
// counts) with 16-byte aligned key and luminance planes and an 8-byte aligned column plane.
template <int WB, int RW, int DS, int DIMS = kAllDims>
cudaError_t launch_random(Job& j, const RandParams& rp, const GridPrep& gp) {
    const bool aligned = (reinterpret_cast<uintptr_t>(gp.key) & 15u) == 0 && (reinterpret_cast<uintptr_t>(gp.lum) & 15u) == 0;
    if (rp.spp_shift >= 2 && aligned) return launch_random_vec<WB, RW, DS, kWalkPixelQuads, DIMS>(j, rp, gp);
    if (gp.col && aligned && (reinterpret_cast<uintptr_t>(gp.col) & 7u) == 0)
        return launch_random_vec<WB, RW, DS, kWalkColumnQuads, DIMS>(j, rp, gp);
    return launch_random_vec<WB, RW, DS, kWalkScalar, DIMS>(j, rp, gp);
}

// WB: bytes of a lane-private bin weight (8 double-float, 4 or 2 exact integers); the 2-byte
// form is built for the default shape only (the caller checks that the lane sums fit)
template <int WB>
cudaError_t launch_random_shape(Job& j, const RandParams& rp, const GridPrep& gp, int shape, bool env) {
    if constexpr (WB == 2) {
        return env ? launch_random<2, 1, 1>(j, rp, gp) : launch_random<2, 1, 1, kNoEnvDims>(j, rp, gp);
    } else {
        switch (shape) {
        case 1: return launch_random<WB, 2, 1>(j, rp, gp);
        case 2: return launch_random<WB, 2, 2>(j, rp, gp);
        case 3: return launch_random<WB, 2, 3>(j, rp, gp);
        case 4: return launch_random<WB, 1, 2>(j, rp, gp);
        case 5: return launch_random<WB, 1, 3>(j, rp, gp);
        default: return launch_random<WB, 1, 1>(j, rp, gp);
        }
    }
}

template <int NC, int RG, int U, int DIMS>
cudaError_t launch_strips_unit(Job& j, const StripParams& sp, unsigned blocks, float2* target, const GridPrep& gp) {
    constexpr int smem = NC * RG * StripLayout<DIMS>::kWarpBytes + StripLayout<DIMS>::edge_bytes(NC);
    static FuncAttribute limit;
    const cudaError_t e = limit.at_least(reinterpret_cast<const void*>(&k_grid_strips<NC, RG, U, DIMS>),
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, j.ctx->device, smem);
    if (e != cudaSuccess) return e;
    k_grid_strips<NC, RG, U, DIMS><<<blocks, NC * RG * 64, smem, j.stream>>>(sp, target, gp);
    j.launches += 1;
    return cudaGetLastError();
}

// Blocks of NC * 32 columns and `len` node rows (one more strip to walk than node rows), one block per
// SM by shared memory: the len whose waves of blocks walk the fewest strips.
template <int NC>
int64_t strip_plan(StripParams& sp) {
    const int nb = NC * 32 / sp.g.step - 1;
    if (nb < 1) return INT64_MAX;
    // blocks of nb + 1 cells, each overlapping the one before by a cell
    const int cells = (sp.g.w + sp.g.step - 1) / sp.g.step;
    sp.col_blocks = std::max(1, (cells - 1 + nb - 1) / nb);
    const int rows = sp.ny1 - sp.ny0;
    int64_t best = INT64_MAX;
    for (int len = 1; len <= rows; ++len) {
        const int64_t blocks = int64_t(sp.col_blocks) * ((rows + len - 1) / len);
        const int64_t cost = (blocks + kStripSms - 1) / kStripSms * (len + 1);
        if (cost < best) {
            best = cost;
            sp.len = len;
        }
    }
    return best;
}

// Units of 8 samples (a 32-byte sector of keys and one of luminances per lane) or 4 where the samples
// per pixel and the planes' alignment allow, else single samples.
template <int NC, int RG, int DIMS>
cudaError_t launch_strips_shape(Job& j, const StripParams& sp, float2* target, const GridPrep& gp) {
    const bool aligned = (reinterpret_cast<uintptr_t>(gp.key) & 15u) == 0 && (reinterpret_cast<uintptr_t>(gp.lum) & 15u) == 0;
    const int rows = sp.ny1 - sp.ny0;
    const unsigned blocks = unsigned(sp.col_blocks) * unsigned((rows + sp.len - 1) / sp.len);
    if (aligned && sp.spp % 8 == 0) return launch_strips_unit<NC, RG, 8, DIMS>(j, sp, blocks, target, gp);
    if (aligned && sp.spp % 4 == 0) return launch_strips_unit<NC, RG, 4, DIMS>(j, sp, blocks, target, gp);
    return launch_strips_unit<NC, RG, 1, DIMS>(j, sp, blocks, target, gp);
}

// NC column segments and RG row groups, two warps each (one per dimension set): bins of 44 KB per
// segment and group without the environment dimension, 55 KB with it, so at most four (three).
// Two row groups halve the rows a warp walks but their blocks repeat a cell in 8 (NC = 2) instead of
// 16 columns: taken where they need no more strips than the wide blocks, on images of a few
// blocks (64x48: 17 us, wide 26 us; 1080p16: 0.47 ms, wide 0.39 ms).
template <int DIMS>
cudaError_t launch_strips_dims(Job& j, const StripParams& sp, float2* target, const GridPrep& gp) {
    constexpr int NC = DIMS == kAllDims ? 3 : 4;
    StripParams wide = sp, tall = sp;
    const int64_t cw = strip_plan<NC>(wide), ct = strip_plan<2>(tall);
    const bool tall_fits = NC == 4 && sp.g.step >= 2 && ct != INT64_MAX;
    // (where a few blocks are the whole grid and a pixel's walk is long, half the rows per warp count for more than
    // the strips, up to half as many again: 256x256x32 at tile 16 85 -> 74 us, at tile 8 77 -> 62; at 4 samples
    // 18 -> 21, so from 32; 2048x1152x64, with 38 strips against 20, 1.89 -> 2.5 ms)
    const bool long_walk = tall_fits && sp.spp >= 32 && 2 * ct <= 3 * cw &&
                           int64_t(tall.col_blocks) * ((tall.ny1 - tall.ny0 + tall.len - 1) / tall.len) <= kStripSms;
    if (tall_fits && (ct <= cw || long_walk))
        return launch_strips_shape<2, NC == 4 ? 2 : 1, DIMS>(j, tall, target, gp);
    return launch_strips_shape<NC, 1, DIMS>(j, wide, target, gp);
}

}  // namespace

// Where a fast-mode push adds its bins. The reference adds each pass's grid to the frame grid at the
// end of the pass; with the frame grid in double-float pairs (or still empty) the push adds its
// pairs straight into it instead (the pairs' sums differ from pass-then-merge only in the rounding
// of the low words), and the end of the pass has nothing to merge. Otherwise the pass grid
// collects the pass as in the reference.
static cudaError_t grid_target(Job& j, float2** out) {
    const int64_t n = j.g.nn * kDeps * kDepStride;
    if (j.cfg.rpf_shrinkage_scale > 0.0f && (j.grid_fresh || j.grid_pairs)) {
        if (j.grid_fresh) {
            const cudaError_t e = cudaMemsetAsync(j.n.grid, 0, size_t(n) * sizeof(double), j.stream);
            if (e != cudaSuccess) return e;
            j.grid_fresh = false;
            j.grid_pairs = true;
        }
        j.pass_direct = true;
        *out = reinterpret_cast<float2*>(j.n.grid);
    } else {
        j.pass_indirect = true;
        *out = reinterpret_cast<float2*>(j.n.pass_grid);
    }
    return cudaSuccess;
}

cudaError_t launch_grid_fast(Job& j, const DeviceSamples& s, int64_t first, int64_t count, const GridPrep& gp,
                             int32_t spp, int32_t max_count, int64_t total_samples, const int64_t* d_max_count) {
    float2* target = nullptr;
    const bool fresh = j.cfg.rpf_shrinkage_scale > 0.0f && j.grid_fresh;  // grid_target clears the frame grid
    if (const cudaError_t e0 = grid_target(j, &target); e0 != cudaSuccess) return e0;
    const int step = j.g.step;
    const bool pow2 = (step & (step - 1)) == 0;
    GridParams gpar{j.g, first, count, 0, 0, 0, pow2 ? 1 : 0, 1.0f / float(step), spp, spp > 0 ? 1.0f / float(spp) : 0.0f};
    {
        // node rows whose support rows (ny-1)*step-1 .. (ny+1)*step+1 meet the push's rows
        const int y0 = int(first / j.g.w), y1 = int((first + count - 1) / j.g.w);
        const int ny0 = std::max(0, (y0 - 1) / step - 1), ny1 = std::min(j.g.nodes_y - 1, (y1 + 1) / step + 1);
        gpar.node0 = int64_t(ny0) * j.g.nodes_x;
        gpar.count_nodes = int64_t(ny1 - ny0 + 1) * j.g.nodes_x;
    }
    const unsigned nblocks = unsigned(gpar.count_nodes);
    const int sup = j.g.support;
    gpar.uniform_ok = (sup >= 4 && sup <= 2048 && (sup & (sup - 1)) == 0) ? 1 : 0;
    // exact integer bin weights need a power-of-two step and a per-bin total below 2^32:
    // at most support^2 pixels * max_count samples * step^2
    const double bound = double(sup + 3) * double(sup + 3) * double(std::max(max_count, 1)) * double(step) * double(step);
    // a bin's weight sum is at most the push's samples times step^2 units as well
    const double total_bound = double(std::max<int64_t>(total_samples, 1)) * double(step) * double(step);
    const bool int_w = pow2 && (bound < 4.0e9 || total_bound < 4.0e9);
    cudaError_t e;
    {
        KernelScope ks(j, RPD_KERNEL_GRID);
        int sh = 0;
        while ((1 << sh) < step) ++sh;
        // (images of a few nodes fill the GPU with neither form, and the one launch of the pattern form
        // is shorter than the two: 64x48, 63 nodes, 21 against 29 us. 256x256, 1089 nodes: one pattern 21 against 35,
        // three 75 against 48, eight 86 against 50; 640x360, 3726 nodes: 30 / 34, 134 / 79, 158 / 140; 1280x720:
        // 88 / 56, 468 / 141, 544 / 308)
        if (gpar.uniform_ok && int_w && step >= 2 && step <= 16 && gpar.count_nodes > 512) {
            const int ny0 = int(gpar.node0 / j.g.nodes_x), ny1 = ny0 + int(gpar.count_nodes / j.g.nodes_x);
            // (scratch: a node plane that recompute_sensitivity writes before it reads)
            unsigned* odd_count = reinterpret_cast<unsigned*>(j.p.counters + RPD_COUNTER_COUNT_);
            int32_t* odd_nodes = reinterpret_cast<int32_t*>(j.n.prior[0]);
            if ((e = cudaMemsetAsync(odd_count, 0, sizeof(unsigned), j.stream)) != cudaSuccess) return e;
            TotalsParams tp{j.g, first, count, ny0, ny1, 1, 1, sh, fresh ? 1 : 0, 1, 0, odd_count, odd_nodes};
            const int cells = 32 / step, image_cells = (j.g.w + step - 1) / step;
            tp.col_warps = std::max(1, (image_cells - 1 + cells - 2) / (cells - 1));
            // node rows per warp: one more strip than node rows is walked, so as many as fit in the 20
            // warps an SM holds at 90 registers, in one wave (1280x720 with an adaptive pass, grid 333 us
            // with the 16-warp quotient rounded down, two waves of single rows, and 292 us; half as many
            // warps 445)
            const int64_t resident = int64_t(kStripSms) * 20;
            const int64_t rows = (int64_t(tp.col_warps) * (ny1 - ny0) + resident - 1) / resident;
            tp.len = int(std::min<int64_t>(16, std::max<int64_t>(1, rows)));
            const int64_t warps = int64_t(tp.col_warps) * ((ny1 - ny0 + tp.len - 1) / tp.len);
            // Seven class walks stand for any number of pattern walks; each costs about 1.5 of them (up to three
            // sums per pixel), so from eleven on (totals and screen bins of up to eight patterns, 1280x720x8: 428 -> 308
            // us). Where seven times the warps fit on the GPU at once, seven share the classes, from two walks on
            // (256x256x8 of eight patterns 188 -> 50 us, of three 70 -> 48, of one 33 -> 35; 256x256x4 where some samples
            // lack the position, twice the walks, 301 -> 98); with fewer parts on
            // larger images the repeated look for patterns costs other frames on the GPU more than it gives.
            tp.parts = warps * kClasses <= resident ? kClasses : 1;
            tp.many = tp.parts > 1 ? 1 : 10;
            k_grid_totals<<<unsigned((warps * tp.parts + 3) / 4), 128, 0, j.stream>>>(tp, target, gp);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
            const size_t smem = size_t(LaneBins<false>::kSlots) * 32 * sizeof(float) + sizeof(OddPicks) + size_t(4) * step * step * sizeof(uint16_t);
            const unsigned odd_blocks = std::min<unsigned>(nblocks, unsigned(kStripSms) * 16);
            k_grid_odd<<<odd_blocks, 32, smem, j.stream>>>(gpar, target, s, j.offsets, gp, odd_count, odd_nodes);
            j.launches += 2;
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        } else {
        const int side = 2 * step + 3;
        const size_t list_bytes = size_t(side) * size_t(side) * sizeof(int);
        if (list_bytes <= size_t(64) * 1024) {
            // pattern form: one warp per node
            const size_t smem = size_t(int_w ? LaneBins<true>::kSlots : LaneBins<false>::kSlots) * 32 * sizeof(float) +
                                list_bytes;
            if (int_w) {
                static FuncAttribute limit;
                e = limit.at_least(reinterpret_cast<const void*>(&k_grid_screen<true>),
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, j.ctx->device, int64_t(smem));
                if (e != cudaSuccess) return e;
                k_grid_screen<true><<<nblocks, 32, smem, j.stream>>>(gpar, target, s, j.offsets, gp);
            } else {
                static FuncAttribute limit;
                e = limit.at_least(reinterpret_cast<const void*>(&k_grid_screen<false>),
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, j.ctx->device, int64_t(smem));
                if (e != cudaSuccess) return e;
                k_grid_screen<false><<<nblocks, 32, smem, j.stream>>>(gpar, target, s, j.offsets, gp);
            }
        } else if (int_w) {
            const size_t smem = size_t(kGroups) * LaneBins<true>::kSlots * 32 * sizeof(float);
            e = cudaFuncSetAttribute(k_grid_fast<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (e != cudaSuccess) return e;
            k_grid_fast<true><<<nblocks, kGroups * 32, smem, j.stream>>>(gpar, target, s, j.offsets, gp);
        } else {
            const size_t smem = size_t(kGroups) * LaneBins<false>::kSlots * 32 * sizeof(float);
            e = cudaFuncSetAttribute(k_grid_fast<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (e != cudaSuccess) return e;
            k_grid_fast<false><<<nblocks, kGroups * 32, smem, j.stream>>>(gpar, target, s, j.offsets, gp);
        }
        j.launches += 1;
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    }
    KernelScope ks(j, RPD_KERNEL_GRID_RANDOM);
    RandParams rp{gpar, 0u, -1, 2 * step + 3, nullptr, 0, 0, target};
    // the statistics pass clears a dimension's valid bit when the push has no plane for it: without
    // environment planes (a closed scene) the form without the environment dimension runs
    const bool env = s.compact ? s.c16.env_u[0] != nullptr : s.env_u[0] != nullptr;
    if (spp > 0) {
        if ((spp & (spp - 1)) == 0) {
            int sh = 0;
            while ((1 << sh) < spp) ++sh;
            rp.spp_shift = sh;
        } else {
            rp.spp_magic = spp_magic_for(spp, (2 * step + 3) * spp);
        }
    }
    // 16-bit lane sums (smaller bins, more resident warps) when no lane's sum can reach 2^16. Each
    // sample adds at most step^2 units. Uniform push: a lane takes at most 1/32 of a node's quads
    // (plus two partial quads per row segment). Per-pixel counts of at most M: a node's support
    // holds at most side^2 M samples, a segment of len samples spans at most len/4 + 1.5 quads, and
    // a lane takes at most 1/32 of a chunk's (up to 32 segments) quads plus one, so at most
    // side^2 M / 32 + 10 samples per chunk of 32 support rows.
    const bool default_shape = j.grid_shape == 0 || j.grid_shape == 6;
    const double units = double(step) * double(step);
    const double side = double(2 * step + 3);
    const double chunks = std::ceil(side / 32.0);
    auto counts_fit = [&](double m) { return (side * side * m / 32.0 + 10.0 * chunks) * units < 65536.0; };
    // 16-bit lane sums: a column's row factors sum to at most step^2 units per sample of a pixel
    if (int_w && default_shape && spp > 0 && step <= 32 && units * double(spp) < 65536.0 &&
        gpar.count_nodes < (int64_t(1) << 30)) {
        int sh = 0;
        while ((1 << sh) < step) ++sh;
        const int ny0 = int(gpar.node0 / j.g.nodes_x), ny1 = ny0 + int(gpar.count_nodes / j.g.nodes_x);
        const StripParams sp{j.g, first, count, ny0, ny1, 0, 0, spp, sh, fresh ? 1 : 0};
        return env ? launch_strips_dims<kAllDims>(j, sp, target, gp) : launch_strips_dims<kNoEnvDims>(j, sp, target, gp);
    }
    if (int_w && default_shape) {
        if (spp > 0) {
            if ((double(sup + 3) * double(sup + 3) * double(spp) / 32.0 + 8.0) * units < 65536.0)
                return launch_random_shape<2>(j, rp, gp, j.grid_shape, env);
        } else if (max_count != INT32_MAX) {
            if (counts_fit(double(std::max(max_count, 1)))) return launch_random_shape<2>(j, rp, gp, j.grid_shape, env);
        } else if (d_max_count) {
            // the largest count is known on the device only: launch both forms, each block of the
            // one that does not apply returns at once
            int64_t lim = int64_t(std::max(0.0, (65536.0 / units - 10.0 * chunks) * 32.0 / (side * side)));
            while (lim > 0 && !counts_fit(double(lim))) --lim;
            if (lim > 0) {
                RandParams r16 = rp;
                r16.max_count = d_max_count;
                r16.max_limit = lim;
                r16.max_mode = 1;
                if ((e = launch_random_shape<2>(j, r16, gp, j.grid_shape, env)) != cudaSuccess) return e;
                RandParams r32 = r16;
                r32.max_mode = 2;
                return launch_random_shape<4>(j, r32, gp, j.grid_shape, env);
            }
        }
    }
    return int_w ? launch_random_shape<4>(j, rp, gp, j.grid_shape, env) : launch_random_shape<8>(j, rp, gp, j.grid_shape, env);
}

}  // namespace rpd
