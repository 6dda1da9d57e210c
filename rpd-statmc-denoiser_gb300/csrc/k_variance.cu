// variance_denoise (main.cpp:1166-1268): Jacobi iterations of the gated neighbour mean
// with the upward-only update, ping-ponging two planes, the last into the denoised variance.
// Single precision throughout, in the reference's order, so the result is bit-identical.
//
// The ping-pong planes carry the hit test in their sign: a pixel with a primary hit holds its
// variance (>= EPS_SMALL), a pixel without one the negated clamped variance, which the
// iterations copy unchanged (main.cpp:1198-1201) and the last one turns back into the value
// the reference keeps. A block's halo tile is then the
// plane's box as it lies in HBM — the tensor copy's zero fill past the image edges reads as
// "no neighbour" like a pixel without a hit — so each iteration stages its tile with one
// tiled tensor copy (cp.async.bulk.tensor) instead of per-thread gathers, and the gate records
// (unit normal, depth) with a second one. Rows of the ping-pong planes are padded to 4 floats,
// the 16-byte row pitch tensor copies need.
#include <cmath>

#include "rpd_internal.h"
#include "device_math.cuh"
#include "tma.cuh"

namespace rpd {

namespace {

__device__ __forceinline__ float pixel_variance(float m2, int n) { return (n > 1) ? m2 / float(n - 1) : 0.0f; }

inline int var_pitch(int w) { return (w + 3) & ~3; }

// The clamped variance (main.cpp:1182-1186), negated for a pixel without a primary hit; the
// pixel's gate record. A pixel with a hit holds at least EPS_SMALL: the clamp's upper bound is less for
// an adaptive_sigma_max below 1e-4, but every iteration reads such a value through max(EPS_SMALL, .).
__global__ void k_var_init(PixelPlanes p, int w, int h, int pitch, float max_variance, float* curr) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= int64_t(w) * h) return;
    float v = pixel_variance(p.square_diff[i], p.n[i]);
    if (!isfinite(v)) v = 1e-8f;
    v = fclamps(v, 1e-8f, max_variance);
    const bool hit = p.hit_count[i] > 0;
    const int64_t y = i / w, x = i - y * w;
    curr[y * pitch + x] = hit ? fmaxs(1e-8f, v) : -v;
    p.var_gate[i] = make_float4(p.f_normal[0][i], p.f_normal[1][i], p.f_normal[2][i], p.f_depth[i]);
}

struct VarParams {
    int w, h, radius, pitch;
    float normal_threshold, depth_threshold, compat_sigma, shrinkage_k;
    float depth_half_ulp;  // half an ulp of the depth threshold
    // |1 - x| / sqrt(x) > compat_sigma for the ratio x of two variances: surely not for
    // lo_in <= x <= hi_in, surely for x < lo_out and x > hi_out (ratio_bounds)
    float lo_out, lo_in, hi_in, hi_out;
};

// rpf::conservative_variance_update (core/stats.h:85-91)
__device__ __forceinline__ float conservative_variance_update(float value, float neighbor, float stabilizer) {
    const float blend = fclamps(fmaxs(0.0f, neighbor - value) / fmaxs(1e-8f, value + neighbor + stabilizer), 0.0f, 1.0f);
    return lerp_std(value, neighbor, blend);
}

constexpr int kVarTx = 32, kVarTy = 16;  // a block's pixels
constexpr int kVarRows = 2;              // pixels of a thread, one above the other
constexpr float kGateBand = 1.0f / 1048576.0f;  // 2^-20
constexpr int kVarPad = 4;  // the variance box starts 4 floats left of the block (a 16-byte boundary)

// The depth gate relative_depth_delta(d_i, d_j) > threshold (main.cpp:266-268): fl(num / m)
// against the threshold, decided by the product threshold * m away from it and by the IEEE
// quotient near it.
__device__ __forceinline__ bool depth_far(float dabs_i, float di, float dj, float dthr) {
    float m = dabs_i;
    if (m < fabsf(dj)) m = fabsf(dj);
    if (m < 1e-8f) m = 1e-8f;
    const float num = fabsf(di - dj);
    const float tm = dthr * m;
    const bool d_hi = num > tm * (1.0f + kGateBand), d_lo = num < tm * (1.0f - kGateBand);
    if (tm >= 1e-30f && (d_hi || d_lo)) return d_hi;
    return num / m > dthr;
}
// The same decision by one exact fused difference (k_statmc.cu's depth_far, with its reasons), for
// thresholds of at least 1e-21. dm: max(|d_i|, EPS_SMALL).
__device__ __forceinline__ bool depth_far_fused(float di, float dm, float dj, float dthr, float half_ulp) {
    float m = dm;
    if (m < fabsf(dj)) m = fabsf(dj);
    return __fmaf_rn(-dthr, m, fabsf(di - dj)) > m * half_ulp;
}

// |var_i - var_j| / max(EPS_SMALL, sqrt(var_i * var_j)) > compat_sigma (main.cpp:1228-1232),
// by a reciprocal square root away from the threshold and the IEEE quotient near it.
__device__ __forceinline__ bool incompatible(float var_i, float var_j, float sigma) {
    const float diff = fabsf(var_i - var_j);
    const float prod = var_i * var_j;
    const float approx = diff * rsqrtf(prod);
    if (fabsf(approx - sigma) > sigma * kGateBand && prod >= 1e-16f && prod < 1e36f) return approx > sigma;
    return diff / fmaxs(1e-8f, sqrtf(prod)) > sigma;
}

// A thread's pixel: its variance, the bounds of the variances it is compatible with, its feature gate
// and the sums over its window.
template <int R>
struct VarPixel {
    static constexpr int kWords = ((2 * R + 1) * (2 * R + 1) - 1 + 31) / 32;
    float var, lo_out, lo_in, hi_in, hi_out;
    float4 g;
    float dm;                // max(|depth|, EPS_SMALL)
    uint32_t gate[kWords];   // the neighbours the hit, normal and depth gates pass, in window order
    float weighted, weight;  // over the surely compatible neighbours
    float may_weight;        // over those that may be: more than `weight` if a ratio lies between the bounds
};

// The pixel's sums again, every ratio by the reference's quotient.
template <int R>
__device__ __noinline__ float2 var_exact_sums(const float* V, int vw, float var_i, uint32_t g0, uint32_t g1, uint32_t g2,
                                            float sigma) {
    constexpr int side = 2 * R + 1, n = side * side - 1;
    float weighted = 0.0f, weight = 0.0f;
    for (int b = 0; b < n; ++b) {
        if (!(((b < 32 ? g0 : b < 64 ? g1 : g2) >> (b & 31)) & 1u)) continue;
        const int e = b < n / 2 ? b : b + 1;
        const int dy = e / side - R, dx = e % side - R;
        const float var_j = V[dy * vw + dx];
        if (incompatible(var_i, var_j, sigma)) continue;
        const float w_j = 1.0f / (1.0f + float(dx * dx + dy * dy));
        weighted += w_j * var_j;
        weight += w_j;
    }
    return make_float2(weighted, weight);
}

// One Jacobi iteration (main.cpp:1198-1249) with the radius fixed at compile time. A 32 x 16
// block's halo tile arrives by tensor copies: the variance box (the 4-float-aligned
// (32 + 8) x (16 + 2R) floats) and, unless MODE 2, the gate records' (32 + 2R) x (16 + 2R) box.
// The window is unrolled; a thread's two pixels read each of its rows once; every gate is a
// predicate (the lanes of a warp stay converged), and the accepted neighbours are added in the
// reference's order; a rejected neighbour adds nothing, as the reference's `continue` does.
//
// The hit, normal and depth gates depend on the features only, which the iterations do not
// change. MODE 0 evaluates every gate; MODE 1 also writes each pixel's geometric-gate bits (one
// per neighbour, in window order) to var_mask; MODE 2 reads them and evaluates only the
// variance-compatibility gate of the neighbours they pass.
//
// That gate compares |var_i - var_j| / max(EPS_SMALL, sqrt(var_i var_j)) with sigma, which for a given
// var_i is a test of var_j against two bounds. Within 2^-19 of a bound, where the quotient's rounding
// decides, the pixel's sums are taken again with the quotient itself (var_exact_sums). Passed neighbours are at
// least EPS_SMALL, as is every value of the planes for a pixel with a hit (k_var_init's; the update only raises
// it), so the reference's maxima with EPS_SMALL change nothing.
//
// last: the iteration's result is the denoised variance itself. The reference takes the maximum with the
// clamped raw variance (main.cpp:1252-1261), which the iterations began at or, raised to EPS_SMALL, above, and below
// which none falls; a pixel without a hit holds its negative.
//
// Bound by instruction issue. At 1920x1080, radius 3: MODE 1 184 us and MODE 2 94 us with one pixel per
// thread, an rsqrt and two guarded quotients per neighbour, 17 us for the
// final maximum; 119 and 62 us with the bounds, two pixels per thread and the fused depth gate (124 and 67 with
// an uncertainty flag per neighbour instead of a second weight sum).
template <int R, int MODE>
__global__ void __launch_bounds__(kVarTx * kVarTy / kVarRows)
    k_var_smooth_r(PixelPlanes p, VarParams prm, float* dst, int dst_pitch, bool last, unsigned long long* timeouts,
                   const __grid_constant__ CUtensorMap gmap, const __grid_constant__ CUtensorMap vmap) {
    static_assert(R <= kVarPad, "the variance box covers a halo of at most 4 columns");
    static_assert(MODE == 0 || (2 * R + 1) * (2 * R + 1) - 1 <= 64, "the gate bits fit one word");
    constexpr int gw = kVarTx + 2 * R, vw = kVarTx + 2 * kVarPad, th = kVarTy + 2 * R;
    __shared__ __align__(128) float4 G[MODE == 2 ? 1 : gw * th];  // (unit normal, depth)
    __shared__ __align__(128) float V[vw * th];                   // the source plane's box
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int s_fail;
    const int x0 = blockIdx.x * kVarTx, y0 = blockIdx.y * kVarTy;
    const int tid = threadIdx.y * kVarTx + threadIdx.x;
    const uint32_t bar_a = smem_addr(&bar);
    if (tid == 0) {
        mbar_init(bar_a, 1);
        s_fail = 0;
    }
    __syncthreads();
    if (tid == 0) {
        mbar_expect_tx(bar_a, uint32_t(vw * th * 4 + (MODE == 2 ? 0 : gw * th * 16)));
        tma_load_2d(smem_addr(V), &vmap, x0 - kVarPad, y0 - R, bar_a);
        if (MODE != 2) tma_load_3d(smem_addr(G), &gmap, 4 * (x0 - R), y0 - R, 0, bar_a);
    }
    if (!mbar_wait_bounded(bar_a, 0)) s_fail = 1;
    __syncthreads();
    if (s_fail) {  // report, and let the copies land (bounded) before the shared memory is released
        if (tid == 0) {
            atomicAdd(timeouts, 1ull);
            mbar_wait_bounded(bar_a, 0);
        }
        return;
    }
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y * kVarRows;
    if (x >= prm.w || y >= prm.h) return;
    // the first row and column of the thread's windows
    const float* Vw = V + threadIdx.y * kVarRows * vw + threadIdx.x + kVarPad - R;
    const float4* Gw = G + threadIdx.y * kVarRows * gw + threadIdx.x;
    VarPixel<R> px[kVarRows];
    float src[kVarRows];
#pragma unroll
    for (int k = 0; k < kVarRows; ++k) {
        VarPixel<R>& q = px[k];
        src[k] = Vw[(R + k) * vw + R];  // 0 below the image's last row
        q.var = src[k];
        q.lo_out = q.var * prm.lo_out;
        q.lo_in = q.var * prm.lo_in;
        q.hi_in = q.var * prm.hi_in;
        q.hi_out = q.var * prm.hi_out;
        q.weighted = q.weight = q.may_weight = 0.0f;
#pragma unroll
        for (int b = 0; b < VarPixel<R>::kWords; ++b) q.gate[b] = 0u;
        if (MODE == 2) {
            if (y + k < prm.h) {
                const uint64_t m = p.var_mask[int64_t(y + k) * prm.w + x];
                q.gate[0] = uint32_t(m);
                if (VarPixel<R>::kWords > 1) q.gate[VarPixel<R>::kWords > 1 ? 1 : 0] = uint32_t(m >> 32);
            }
        } else {
            q.g = Gw[(R + k) * gw + R];
            q.dm = fmaxs(fabsf(q.g.w), 1e-8f);
        }
    }
#pragma unroll
    for (int j = 0; j < 2 * R + kVarRows; ++j) {
#pragma unroll
        for (int i = 0; i <= 2 * R; ++i) {
            const float var_j = Vw[j * vw + i];
            float4 gj = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (MODE != 2) gj = Gw[j * gw + i];
#pragma unroll
            for (int k = 0; k < kVarRows; ++k) {
                const int dy = j - k - R, dx = i - R;
                if (dy < -R || dy > R || (dx == 0 && dy == 0)) continue;
                const int e = (dy + R) * (2 * R + 1) + i, bit = e - (e > (2 * R + 1) * R + R ? 1 : 0);
                VarPixel<R>& q = px[k];
                bool ok;
                if (MODE == 2) {
                    ok = (q.gate[bit >> 5] >> (bit & 31)) & 1u;
                } else {
                    // outside the image (zero fill) or no primary hit (negative)
                    ok = var_j > 0.0f && !(dot3(q.g.x, q.g.y, q.g.z, gj.x, gj.y, gj.z) < prm.normal_threshold);
                    ok = ok && !depth_far_fused(q.g.w, q.dm, gj.w, prm.depth_threshold, prm.depth_half_ulp);
                    if (ok) q.gate[bit >> 5] |= 1u << (bit & 31);
                }
                const float w_j = 1.0f / (1.0f + float(dx * dx + dy * dy));
                if (ok && var_j >= q.lo_out && var_j <= q.hi_out) q.may_weight += w_j;
                if (ok && var_j >= q.lo_in && var_j <= q.hi_in) {
                    q.weighted += w_j * var_j;
                    q.weight += w_j;
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kVarRows; ++k) {
        VarPixel<R>& q = px[k];
        if (y + k >= prm.h) continue;
        if (MODE == 1) {
            uint64_t m = q.gate[0];
            if (VarPixel<R>::kWords > 1) m |= uint64_t(q.gate[VarPixel<R>::kWords > 1 ? 1 : 0]) << 32;
            p.var_mask[int64_t(y + k) * prm.w + x] = m;
        }
        float out = src[k];
        if (src[k] > 0.0f) {
            if (q.may_weight != q.weight) {
                constexpr int n = VarPixel<R>::kWords;
                const float2 s = var_exact_sums<R>(Vw + (R + k) * vw + R, vw, q.var, q.gate[0], q.gate[n > 1 ? 1 : 0],
                                                   q.gate[n > 2 ? 2 : 0], prm.compat_sigma);
                q.weighted = s.x;
                q.weight = s.y;
            }
            float neighbor_mean = q.var;
            if (q.weight > 1e-8f) neighbor_mean = q.weighted / q.weight;
            out = conservative_variance_update(q.var, neighbor_mean, prm.shrinkage_k);
        } else if (last) {
            out = -src[k];  // no primary hit (hit_count == 0): its clamped raw variance
        }
        dst[int64_t(y + k) * dst_pitch + x] = out;
    }
}

// The same iteration for radii above 4 (the radius at run time) and for parameters outside the bounds'
// reasoning (launch_variance): the halo is gathered by the
// threads into dynamic shared memory, the window loops at run time.
__global__ void __launch_bounds__(kVarTx * kVarTy) k_var_smooth(PixelPlanes p, VarParams prm, const float* src,
                                                                float* dst, int dst_pitch, bool last) {
    extern __shared__ float4 vsm[];
    const int r = prm.radius;
    const int tw = kVarTx + 2 * r, th = kVarTy + 2 * r, tn = tw * th;
    const int side = 2 * r + 1;
    float4* G = vsm;                                // (normal, depth)
    float* V = reinterpret_cast<float*>(vsm + tn);  // the source plane, 0 outside the image
    float* W = V + tn;                              // 1 / (1 + d^2)
    const int x0 = blockIdx.x * kVarTx, y0 = blockIdx.y * kVarTy;
    const int tid = threadIdx.y * kVarTx + threadIdx.x;
    for (int e = tid; e < side * side; e += kVarTx * kVarTy) {
        const int dx = e % side - r, dy = e / side - r;
        W[e] = 1.0f / (1.0f + float(dx * dx + dy * dy));
    }
    for (int e = tid; e < tn; e += kVarTx * kVarTy) {
        const int gx = x0 - r + e % tw, gy = y0 - r + e / tw;
        const bool inside = gx >= 0 && gx < prm.w && gy >= 0 && gy < prm.h;
        G[e] = inside ? p.var_gate[int64_t(gy) * prm.w + gx] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        V[e] = inside ? src[int64_t(gy) * prm.pitch + gx] : 0.0f;
    }
    __syncthreads();
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
    if (x >= prm.w || y >= prm.h) return;
    const int64_t pidx = int64_t(y) * dst_pitch + x;
    const int ei = (threadIdx.y + r) * tw + threadIdx.x + r;
    const float src_i = V[ei];
    if (!(src_i > 0.0f)) {
        dst[pidx] = last ? -src_i : src_i;
        return;
    }
    const float4 gi = G[ei];
    const float var_i = fmaxs(1e-8f, src_i);
    const float dabs_i = fabsf(gi.w);
    float weight_sum = 0.0f, weighted_sum = 0.0f;
    for (int dy = -r; dy <= r; ++dy) {
        const int erow = ei + dy * tw;
        const float* wrow = W + (dy + r) * side + r;
        for (int dx = -r; dx <= r; ++dx) {
            if (dx == 0 && dy == 0) continue;
            const float src_j = V[erow + dx];
            if (!(src_j > 0.0f)) continue;  // outside the image or no primary hit
            const float4 gj = G[erow + dx];
            if (dot3(gi.x, gi.y, gi.z, gj.x, gj.y, gj.z) < prm.normal_threshold) continue;
            if (depth_far(dabs_i, gi.w, gj.w, prm.depth_threshold)) continue;
            const float var_j = fmaxs(1e-8f, src_j);
            if (incompatible(var_i, var_j, prm.compat_sigma)) continue;
            const float w_j = wrow[dx];
            weighted_sum += w_j * var_j;
            weight_sum += w_j;
        }
    }
    float neighbor_mean = var_i;
    if (weight_sum > 1e-8f) neighbor_mean = weighted_sum / weight_sum;
    dst[pidx] = conservative_variance_update(var_i, neighbor_mean, prm.shrinkage_k);
}

// Tensor maps of the gate records and the two ping-pong planes for halo radius R.
template <int R>
cudaError_t var_maps(Job& j, int pitch) {
    if (j.var_map_r == R) return cudaSuccess;
    CUtensorMap* m = reinterpret_cast<CUtensorMap*>(j.var_maps[0]);
    cudaError_t e = encode_record_map(m, j.p.var_gate, j.g.w, j.g.h, 1, kVarTx + 2 * R, kVarTy + 2 * R);
    if (e == cudaSuccess)
        e = encode_plane_map(reinterpret_cast<CUtensorMap*>(j.var_maps[1]), j.p.var_ping, j.g.w, j.g.h, pitch,
                             kVarTx + 2 * kVarPad, kVarTy + 2 * R);
    if (e == cudaSuccess)
        e = encode_plane_map(reinterpret_cast<CUtensorMap*>(j.var_maps[2]), j.p.var_pong, j.g.w, j.g.h, pitch,
                             kVarTx + 2 * kVarPad, kVarTy + 2 * R);
    if (e != cudaSuccess) return e;
    j.var_map_r = R;
    return cudaSuccess;
}

template <int R>
cudaError_t launch_smooth_r(Job& j, const VarParams& prm, float*& curr, float*& next, dim3 vgrid) {
    const cudaError_t e = var_maps<R>(j, prm.pitch);
    if (e != cudaSuccess) return e;
    CUtensorMap gmap, ping, pong;
    std::memcpy(&gmap, j.var_maps[0], sizeof(gmap));
    std::memcpy(&ping, j.var_maps[1], sizeof(ping));
    std::memcpy(&pong, j.var_maps[2], sizeof(pong));
    unsigned long long* timeouts = j.p.counters + RPD_COUNTER_DEVICE_WAIT_TIMEOUTS;
    const int iters = j.cfg.var_iterations;
    constexpr bool kMask = (2 * R + 1) * (2 * R + 1) - 1 <= 64;
    for (int it = 0; it < iters; ++it) {
        const CUtensorMap& vmap = curr == j.p.var_ping ? ping : pong;
        const bool last = it + 1 == iters;
        float* const dst = last ? j.p.variance_denoised : next;
        const int dst_pitch = last ? prm.w : prm.pitch;
        const dim3 block(kVarTx, kVarTy / kVarRows);
        if (!kMask || iters == 1)
            k_var_smooth_r<R, 0><<<vgrid, block, 0, j.stream>>>(j.p, prm, dst, dst_pitch, last, timeouts, gmap, vmap);
        else if (it == 0)
            k_var_smooth_r<R, kMask ? 1 : 0><<<vgrid, block, 0, j.stream>>>(j.p, prm, dst, dst_pitch, last, timeouts, gmap, vmap);
        else
            k_var_smooth_r<R, kMask ? 2 : 0><<<vgrid, block, 0, j.stream>>>(j.p, prm, dst, dst_pitch, last, timeouts, gmap, vmap);
        float* t = curr;
        curr = next;
        next = t;
    }
    return cudaGetLastError();
}

// The ratio bounds of VarParams. With x the ratio of two variances, |1 - x| / sqrt(x) passes sigma at
// ((sqrt(sigma^2 + 4) -+ sigma) / 2)^2, with a logarithmic slope of at least 1/2; the reference's float
// quotient is off by less than 2^-22, so its decision can differ within 2^-21 of them; 2^-19 covers the bounds'
// own roundings.
void ratio_bounds(VarParams& prm) {
    const double s = prm.compat_sigma, root = std::sqrt(s * s + 4.0), band = 1.0 / 524288.0;
    const double hi = 0.25 * (root + s) * (root + s), lo = 1.0 / hi;
    prm.lo_out = float(lo * (1.0 - band));
    prm.lo_in = float(lo * (1.0 + band));
    prm.hi_in = float(hi * (1.0 - band));
    prm.hi_out = float(hi * (1.0 + band));
}

}  // namespace

cudaError_t launch_variance(Job& j) {
    KernelScope ks(j, RPD_KERNEL_VARIANCE);
    const int64_t np = j.g.np;
    const float max_variance = j.cfg.adaptive_sigma_max * j.cfg.adaptive_sigma_max;
    const int pitch = var_pitch(j.g.w);
    float* curr = j.p.var_ping;
    float* next = j.p.var_pong;
    k_var_init<<<grid_for(np, 256), 256, 0, j.stream>>>(j.p, j.g.w, j.g.h, pitch, max_variance, curr);
    VarParams prm{j.g.w, j.g.h, j.cfg.var_window_radius, pitch, j.cfg.var_normal_threshold, j.cfg.var_depth_threshold,
                  j.cfg.var_compat_sigma, j.cfg.var_shrinkage_k};
    prm.depth_half_ulp = 0.5f * (std::nextafter(prm.depth_threshold, HUGE_VALF) - prm.depth_threshold);
    ratio_bounds(prm);
    const int r = prm.radius;
    const dim3 vgrid((j.g.w + kVarTx - 1) / kVarTx, (j.g.h + kVarTy - 1) / kVarTy);
    cudaError_t e = cudaSuccess;
    // the bounds' reasoning wants products of variances in the normal range, the fused depth gate a
    // threshold whose half ulp scales without underflow
    if (r >= 1 && r <= 4 && max_variance <= 1e18f && prm.depth_threshold >= 1e-21f && prm.depth_threshold <= 1e18f) {
        e = r == 1 ? launch_smooth_r<1>(j, prm, curr, next, vgrid)
          : r == 2 ? launch_smooth_r<2>(j, prm, curr, next, vgrid)
          : r == 3 ? launch_smooth_r<3>(j, prm, curr, next, vgrid)
                   : launch_smooth_r<4>(j, prm, curr, next, vgrid);
    } else {
        const size_t smem = size_t(kVarTx + 2 * r) * size_t(kVarTy + 2 * r) * (sizeof(float4) + sizeof(float)) +
                            size_t(2 * r + 1) * size_t(2 * r + 1) * sizeof(float);
        constexpr size_t limit = size_t(200) * 1024;
        if (smem > limit) return cudaErrorInvalidValue;  // radius beyond the shared-memory tile
        // (the kernel's limit, the same for every call: jobs on several threads may have different radii)
        e = cudaFuncSetAttribute(k_var_smooth, cudaFuncAttributeMaxDynamicSharedMemorySize, int(limit));
        for (int it = 0; it < j.cfg.var_iterations && e == cudaSuccess; ++it) {
            const bool last = it + 1 == j.cfg.var_iterations;
            k_var_smooth<<<vgrid, dim3(kVarTx, kVarTy), smem, j.stream>>>(
                j.p, prm, curr, last ? j.p.variance_denoised : next, last ? prm.w : pitch, last);
            float* t = curr;
            curr = next;
            next = t;
        }
    }
    if (e != cudaSuccess) return e;
    j.launches += 1 + j.cfg.var_iterations;
    return cudaGetLastError();
}

}  // namespace rpd
