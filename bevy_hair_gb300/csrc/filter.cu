// Reconnection filter (filter.wgsl:20-135) and the headless composite
// (composite.wgsl:162-181 + ALPHA_BLENDING + depth test, pipeline.rs:299-339).
// The filter's coverage decisions (strip test, depth rejection, "closer")
// come from float comparisons, so this file is compiled with -fmad=false like
// the raster to keep them reproducible.
#include <cuda_runtime.h>

#include "hg_device.cuh"
#include "hg_internal.h"

namespace hg {
namespace {

constexpr int kFilterRadius = 5;

// Images of at most this many pixels give a pair four threads, or two.
// Measured (us): 96 x 64: 11.0 with four, 14.8 with two, 16.9 with one;
// 400 x 300: 17.1, 23.2, 23.6; 640 x 360: 23.7, 23.8, 23.7; 512 x 512: 33.3,
// 30.5, 35.8; 800 x 600: 43.8, 35.7, 37.5; 960 x 540: 38.4, 35.5, 36.4;
// 1280 x 720: 60.6, 50.2, 47.7.  Two threads take three blocks an SM (80
// registers): at four, with spills, 700 x 400 29.8 us instead of 23.9, 800 x 600
// 40.6 instead of 35.7, though 960 x 540 31.9 instead of 35.5.
constexpr uint64_t kFilterSplit4 = 240u * 1024u, kFilterSplit2 = 512u * 1024u;

struct FilterArgs {
    hg_hair_params p;
    const unsigned long long* center;
    const unsigned long long* cons;
    const float4* shaded;
    float4* filtered;
    float* filtered_depth;
    float4* color;       // composite target (CompositeKind not kNone)
    float* depth;
    float depth_clear;   // kClear: the depth a pixel without hair gets
};

// What a pass that produces a pixel's final colour does with it.
enum CompositeKind {
    kNone,   // nothing: the composite pass follows
    kBlend,  // composite onto the target
    kClear   // composite onto a cleared target, written whole
};

// screen_tangent (filter.wgsl:9-18)
__device__ __forceinline__ float2 screen_tangent(const hg_hair_params& p, f3 world, f3 tangent) {
    Projected a = project_world(p, world);
    Projected b = project_world(p, add3(world, tangent));
    float2 d = sub2(b.screen, a.screen);
    float l = len2(d);
    if (l < 1e-3f) return make_float2(1.0f, 0.0f);
    return make_float2(__fdiv_rn(d.x, l), __fdiv_rn(d.y, l));
}

// The largest x with sqrt_rn(x) <= r (sqrt_rn is monotone), found from r*r by
// stepping one ulp at a time (a few steps at most; bounded by 8 each way).
__device__ __forceinline__ float sqrt_bound(float r) {
    float x = r * r;
    for (int k = 0; k < 8 && __fsqrt_rn(x) > r; ++k) x = nextafterf(x, 0.0f);
    for (int k = 0; k < 8; ++k) {
        const float up = nextafterf(x, __int_as_float(0x7f800000));
        if (!(__fsqrt_rn(up) <= r)) break;
        x = up;
    }
    return x;
}

// composite.wgsl:162-181 of one pixel with colour c (c.w its coverage) and
// view distance view_dist; blend src*a + dst*(1-a) (alpha: a + dst_a*(1-a)),
// depth test GreaterEqual when reverse-Z else LessEqual, depth write on.
// With KIND kClear the target holds colour 0 and depth_clear.
template <CompositeKind KIND>
__device__ __forceinline__ void composite_one(const hg_hair_params& p, float4 c, float view_dist, float4* color,
                                              float* depth_buf, float depth_clear, int32_t px, int32_t py,
                                              uint32_t pix) {
    float4 d = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float out_depth = depth_clear;
    bool pass = false;
    if (!(c.w < 0.001f)) {
        const f3 world = reconstruct_world(p, px, py, view_dist);
        const float4 clip = mat_mul(p.clip_from_world, world.x, world.y, world.z, 1.0f);
        const float depth = clampf(__fdiv_rn(clip.z, fmaxf(clip.w, 1e-5f)), 0.0f, 1.0f);
        const float dst_depth = KIND == kClear ? depth_clear : depth_buf[pix];
        pass = p.pass_mode[2] == 1u ? depth >= dst_depth : depth <= dst_depth;
        if (pass) {
            if (KIND != kClear) d = color[pix];
            const float ia = 1.0f - c.w;
            d.x = c.x * c.w + d.x * ia;
            d.y = c.y * c.w + d.y * ia;
            d.z = c.z * c.w + d.z * ia;
            d.w = c.w * 1.0f + d.w * ia;
            out_depth = depth;
        }
    }
    if (KIND == kClear || pass) {
        color[pix] = d;
        depth_buf[pix] = out_depth;
    }
}

// Taps of row dy of a pixel's window whose distance from the strand's line
// through the pixel is at most half a pixel (the strip of filter.wgsl:63), as
// bits dx + 5.  The line distance is |dx ts.y - dy ts.x|, so the taps form an
// interval of dx, found from its two ends; filter.wgsl's own float expression
// (below) lies within 1.5e-6 of that distance, and a row with an end within
// 1e-5 (in distance) of an integer dx, or one without finite ends (a
// horizontal tangent), is decided tap by tap with that expression, rounding
// for rounding.  strip2: the largest x with sqrt_rn(x) <= 1/2.
__device__ __forceinline__ uint32_t strip_row(float2 ts, float inv_ty, int dy, float strip2) {
    const float mid = (float)dy * ts.x * inv_ty, half = 0.5f * fabsf(inv_ty), slack = 1e-5f * fabsf(inv_ty);
    const float lo = mid - half, hi = mid + half;
    if (fabsf(lo - rintf(lo)) > slack && fabsf(hi - rintf(hi)) > slack) {
        const int jl = max(f2i(ceilf(lo)), -kFilterRadius), jh = min(f2i(floorf(hi)), kFilterRadius);
        return jl > jh ? 0u : (2u << (jh + kFilterRadius)) - (1u << (jl + kFilterRadius));
    }
    uint32_t m = 0;
#pragma unroll 1  // rare; unrolled it crowds the tap loop out of the instruction cache
    for (int dx = -kFilterRadius; dx <= kFilterRadius; ++dx) {
        const float fdx = (float)dx, fdy = (float)dy;
        const float d_par = fdx * ts.x + fdy * ts.y;
        const float ex = fdx - ts.x * d_par, ey = fdy - ts.y * d_par;
        // d_perp = sqrt_rn(e2); d_perp <= 0.5 exactly when e2 <= strip2
        const float e2 = ex * ex + ey * ey;
        if (e2 <= strip2) m |= 1u << (dx + kFilterRadius);
    }
    return m;
}

// 2^x, results below 2^-126 flushed to zero: a pixel's weights count only from
// a sum of 1e-5 up, where 121 such weights are below half a unit in the last
// place of it.  exp2f, which scales to keep them, gives the same outputs and
// takes 1 to 2.5 % of a frame (1920 x 1080 1,017 -> 1,026 us, 24 grooms
// 2,489 -> 2,551).
__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The spatial exponent of a tap (dx, dy), k_par d_par^2 + k_perp d_perp^2 with
// d_par and d_perp its coordinates along the strand's direction ts and across
// it, with the square in dx completed: a (dx - r dy)^2 + c dy^2.  Three
// operations a tap, and nothing cancels in them; expanded to dx^2, dx dy and
// dy^2 terms it would take one, but along the strand of a narrow filter terms
// of thousands leave a few units.  a and c are correctly rounded but for a few
// in a thousand, r is a sum rh + rl (error-free products and sums), and the
// rounded ts' distance from length 1, which leaves d_perp as it is, is taken
// out.  RMS error of a weight above 1e-5, relative, emulated over 1e5
// directions: filter_params 1, 0.2 (the default) 3.1e-7, with d_par, the vector
// across and its length formed anew for every tap 3.6e-7, expanded 5.6e-7;
// 1, 0.02: 1.3e-6, 1.8e-6 and 3.3e-5; 0.05, 1: 5.8e-7, 6.1e-7 and 6.8e-6.
struct SpatialForm {
    float a, rh, rl, c;
};
__device__ __forceinline__ SpatialForm spatial_form(float2 ts, float k_par, float k_perp) {
    const float xx = ts.x * ts.x, yy = ts.y * ts.y, xy = ts.x * ts.y;
    const float xx_low = __fmaf_rn(ts.x, ts.x, -xx), yy_low = __fmaf_rn(ts.y, ts.y, -yy);
    const float xy_low = __fmaf_rn(ts.x, ts.y, -xy);
    const bool flat = fabsf(ts.x) >= fabsf(ts.y);
    const float major = flat ? ts.x : ts.y, minor = flat ? ts.y : ts.x;
    const float excess = __fmaf_rn(minor, minor, __fmaf_rn(major, major, -1.0f));  // |ts|^2 - 1
    // a = k_par xx + k_perp yy / |ts|^2
    const float a1 = k_par * xx, a2 = k_perp * yy, a = a1 + a2, a2_in = a - a1;
    const float a_low = ((a1 - (a - a2_in)) + (a2 - a2_in)) + (__fmaf_rn(k_par, xx, -a1) + k_par * xx_low) +
                        (__fmaf_rn(k_perp, yy, -a2) + k_perp * (yy_low - yy * excess));
    // r = xy (k_perp / |ts|^2 - k_par) / a
    const float diff = k_perp - k_par, diff_in = diff - k_perp;
    const float diff_low = ((k_perp - (diff - diff_in)) - (k_par + diff_in)) - k_perp * excess;
    const float b = xy * diff, b_low = __fmaf_rn(xy, diff, -b) + __fmaf_rn(xy, diff_low, xy_low * diff);
    const float inv = 1.0f / a;
    SpatialForm f;
    f.a = a + a_low;
    f.rh = b * inv;
    f.rl = (__fmaf_rn(-f.rh, a, b) + (b_low - f.rh * a_low)) * inv;
    // c = k_par k_perp |ts|^2 / a
    const float kk = k_par * k_perp, kk_low = __fmaf_rn(k_par, k_perp, -kk) + kk * excess;
    const float c = kk * inv;
    f.c = c + (__fmaf_rn(-c, a, kk) + (kk_low - c * a_low)) * inv;
    // a vanishes where the filter has no bound along the rows: the exponent
    // is then the same for every dx.  (0, 0), the direction of a strand whose
    // screen length overflows, has all taps across it.
    if (!(a >= 1e-30f)) {
        const bool none = xx + yy == 0.0f;
        f.a = none ? k_perp : a;
        f.rh = f.rl = 0.0f;
        f.c = none ? k_perp : yy * k_par + xx * k_perp;
    }
    return f;
}

// One pixel of a thread's pair: what its taps are weighed against, and its
// sums.
struct FilterPixel {
    float2 ts;
    float inv_ty;
    float cx, cy, cz, p_norm;          // centre colour, normalised depth
    SpatialForm form;
    float ax, ay, az, weight;          // weighted colour and weight
    int h_center, h_cons;              // strip taps with a centre hit, with a conservative hit only
    bool use_color;
};

// The sums of one group of rows.
struct FilterSums {
    float x, y, z, weight;
};
__device__ __forceinline__ FilterSums operator+(FilterSums a, FilterSums b) {
    return {a.x + b.x, a.y + b.y, a.z + b.z, a.weight + b.weight};
}

// P's sums over tap's colour with weight w, where `keep`.
__device__ __forceinline__ void accumulate(bool keep, float4 tap, float w, FilterPixel& P) {
    asm("{\n.reg .pred p;\nsetp.ne.u32 p, %8, 0;\n"
        "@p fma.rn.f32 %0, %4, %7, %0;\n@p fma.rn.f32 %1, %5, %7, %1;\n@p fma.rn.f32 %2, %6, %7, %2;\n"
        "@p add.rn.f32 %3, %3, %7;\n}\n"
        : "+f"(P.ax), "+f"(P.ay), "+f"(P.az), "+f"(P.weight)
        : "f"(tap.x), "f"(tap.y), "f"(tap.z), "f"(w), "r"((uint32_t)keep));
}

// One TX x TY tile per CTA (tile (bx, by) of view a: fields p, center, cons,
// shaded, filtered, filtered_depth), TX TY S / 2 threads.  The (TX+10) x (TY+10)
// neighbourhood is staged in shared memory once: per texel the shaded colour
// and the centre word's normalised depth f32(depth)/16777214 (the exact value
// filter.wgsl:94 computes per tap; -1 marks an empty centre with a
// conservative hit, -2 both empty or off screen), and per row two bit masks of
// the texels with either kind of hit.  Pixels without hair are written at
// once; pairs of vertically adjacent pixels with hair in either are then
// listed and handed to the first threads, so the tap loop runs in full warps.
//
// The tap loop is bound by instruction issue and shared-memory bandwidth.  A
// pair shares its taps' loads (12 rows for 2 x 11); the strip counts come from
// bit masks (strip_row), row by row, instead of a distance and two tests per
// tap; the spatial exponent takes three operations a tap (spatial_form); and
// the depth test alone also rejects the texels without a centre hit.  S threads
// (1, 2 or 4) share a pair, 12 / S rows each: small images leave the chip idle
// otherwise.  However many share it, each group of three rows is summed by
// itself and the four sums are added in the order of the groups, so that an
// image's colours do not depend on S (a batch takes one thread a pair for views
// of any size).  Coverage decisions use exact arithmetic; the colour weights
// only scale colour, so they use fused operations and the fast exponential
// (ex2).  Against a thread per
// pixel with 121 tests and a distance each (us): 1920 x 1080 113 -> 94,
// 3840 x 2160 200 -> 166, 512 x 512 42 -> 32, 96 x 64 22 -> 11.
template <int TX, int TY, int S, CompositeKind KIND, class V>
__device__ __forceinline__ void filter_tile(const V& a, int32_t bx, int32_t by, float depth_clear) {
    constexpr int kHaloX = TX + 2 * kFilterRadius, kHaloY = TY + 2 * kFilterRadius;
    constexpr int kPairs = TX * TY / 2, kThreads = kPairs * S, kWarps = kThreads / 32, kPairWarps = kPairs / 32;
    constexpr int kRows = 2 * kFilterRadius + 2;  // rows a pair's two windows cover
    constexpr int kGroups = 4, kGroupRows = kRows / kGroups;
    static_assert(kPairs % 32 == 0 && kRows % kGroups == 0 && kGroups % S == 0 && kHaloX <= 64 && TX <= 32, "tile shape");
    __shared__ float4 s_tap[kHaloY][kHaloX];  // colour, normalised depth or mark
    __shared__ uint4 s_hits[kHaloY];          // bit per texel: centre hit (x, y), conservative hit only (z, w)
    __shared__ uint16_t s_list[kPairs];       // pair | hair in its upper / lower pixel << 14, 15
    __shared__ int s_warp_hair[kPairWarps];
    const hg_hair_params& p = a.p;
    const int32_t width = f2i(p.screen[0]), height = f2i(p.screen[1]);
    const int32_t x0 = bx * TX - kFilterRadius, y0 = by * TY - kFilterRadius;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int total = 0;
    {
        uint32_t entry = 0;
        if (tid < kPairs) {
            const int32_t ox = bx * TX + tid % TX;
            unsigned long long c[2] = {}, k[2] = {};
            bool inside[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int32_t oy = by * TY + 2 * (tid / TX) + q;
                inside[q] = ox < width && oy < height;
                const uint32_t own = (uint32_t)oy * (uint32_t)width + (uint32_t)ox;
                if (inside[q]) {
                    c[q] = __ldg(&a.center[own]);
                    k[q] = __ldg(&a.cons[own]);
                }
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (!inside[q]) continue;
                if (!is_empty(c[q]) || !is_empty(k[q])) {
                    entry |= 1u << (14 + q);
                } else {
                    const uint32_t own = (uint32_t)(by * TY + 2 * (tid / TX) + q) * (uint32_t)width + (uint32_t)ox;
                    a.filtered[own] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    a.filtered_depth[own] = 0.0f;
                    if (KIND == kClear) {
                        a.color[own] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        a.depth[own] = depth_clear;
                    }
                }
            }
        }
        const uint32_t ballot = __ballot_sync(0xffffffffu, entry != 0u);
        if (lane == 0 && warp < kPairWarps) s_warp_hair[warp] = __popc(ballot);
        __syncthreads();
        int base = 0;
#pragma unroll
        for (int w = 0; w < kPairWarps; ++w) {
            const int n = s_warp_hair[w];
            base += w < warp ? n : 0;
            total += n;
        }
        if (total == 0) return;  // a tile without hair needs no neighbourhood
        if (entry) s_list[base + __popc(ballot & ((1u << lane) - 1u))] = (uint16_t)(entry | (uint32_t)tid);
        // the neighbourhood, a warp per row; a warp's loads are all issued
        // before any is looked at
        constexpr int kWarpRows = (kHaloY + kWarps - 1) / kWarps, kHalves = (kHaloX + 31) / 32;
        unsigned long long word[kWarpRows][kHalves];
        float4 tap[kWarpRows][kHalves];
#pragma unroll
        for (int i = 0; i < kWarpRows; ++i)
#pragma unroll
            for (int h = 0; h < kHalves; ++h) {
                const int hy = warp + i * kWarps, hx = 32 * h + lane;
                const int32_t gx = x0 + hx, gy = y0 + hy;
                word[i][h] = kEmptyU64;
                tap[i][h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (hy < kHaloY && hx < kHaloX && gx >= 0 && gy >= 0 && gx < width && gy < height) {
                    const size_t q = (size_t)gy * width + gx;
                    word[i][h] = __ldg(&a.center[q]);
                    tap[i][h] = __ldg(&a.shaded[q]);
                }
            }
#pragma unroll
        for (int i = 0; i < kWarpRows; ++i) {
            const int hy = warp + i * kWarps;
            if (hy >= kHaloY) break;
            uint32_t hit[2] = {0u, 0u}, only[2] = {0u, 0u};
#pragma unroll
            for (int h = 0; h < kHalves; ++h) {
                const int hx = 32 * h + lane;
                const int32_t gx = x0 + hx, gy = y0 + hy;
                float4 v = tap[i][h];
                v.w = -2.0f;
                if (!is_empty(word[i][h])) {
                    v.w = __fdiv_rn(__uint2float_rn((uint32_t)(word[i][h] >> 40)), 16777214.0f);
                } else if (hx < kHaloX && gx >= 0 && gy >= 0 && gx < width && gy < height &&
                           !is_empty(__ldg(&a.cons[(size_t)gy * width + gx]))) {
                    v.w = -1.0f;
                }
                if (hx < kHaloX) s_tap[hy][hx] = v;
                hit[h] = __ballot_sync(0xffffffffu, v.w >= 0.0f);
                only[h] = __ballot_sync(0xffffffffu, v.w == -1.0f);
            }
            if (lane == 0) s_hits[hy] = make_uint4(hit[0], hit[1], only[0], only[1]);
        }
        __syncthreads();
    }
    const int slot = tid / S, sub = tid % S;
    if (S == 1 && slot >= total) return;  // no pair left for this thread
    const uint32_t entry = s_list[min(slot, total - 1)];
    const int pair = (int)(entry & 0x3fffu), sx = pair % TX, sy = 2 * (pair / TX);
    const int32_t px = bx * TX + sx;

    const float s_par = fmaxf(p.filter_params[0], 0.05f);
    const float s_perp = fmaxf(p.filter_params[1], 0.02f);
    const float sigma_par = (float)kFilterRadius * s_par;
    const float sigma_perp = (float)kFilterRadius * s_perp;
    // exp(-x) = 2^(-x log2 e): the weights' scales folded into one factor each
    const float k_par = 1.4426950408889634f / (sigma_par * sigma_par);
    const float k_perp = 1.4426950408889634f / (sigma_perp * sigma_perp);
    const float k_col = 1.4426950408889634f / (0.9f * 0.9f);
    const float depth_reject = 1.45e-3f, closer_eps = 5e-4f;
    const float strip2 = sqrt_bound(0.5f);

    FilterPixel P[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        FilterPixel& P_ = P[q];
        const bool hair = (entry >> (14 + q)) & 1u;
        const int32_t py = by * TY + sy + q;
        const uint32_t pix = (uint32_t)py * (uint32_t)width + (uint32_t)px;
        P_.ax = P_.ay = P_.az = P_.weight = 0.0f;
        P_.h_center = P_.h_cons = 0;
        P_.use_color = false;
        P_.cx = P_.cy = P_.cz = 0.0f;
        // a direction that strip_row decides at once: a pixel without hair beside
        // one with it (most pairs of sparse hair) sent its warp through the tap
        // by tap test in every row
        P_.ts = make_float2(0.0f, 1.0f);
        P_.p_norm = 1e9f;  // no tap is near it
        if (hair) {
            const unsigned long long center_word = __ldg(&a.center[pix]);
            const bool center_hit = !is_empty(center_word);
            const unsigned long long w = center_hit ? center_word : __ldg(&a.cons[pix]);
            const uint32_t high = (uint32_t)(w >> 32), low = (uint32_t)w, depth_q = high >> 8u;
            const f3 tangent = oct_decode(high & 0xffu, low >> 24u);
            const float view_dist = dequantize_depth(depth_q, p.screen[2], p.screen[3]);
            P_.ts = screen_tangent(p, reconstruct_world(p, px, py, view_dist), tangent);
            const float4 cc = __ldg(&a.shaded[pix]);
            P_.cx = cc.x;
            P_.cy = cc.y;
            P_.cz = cc.z;
            P_.p_norm = __fdiv_rn(__uint2float_rn(depth_q), 16777214.0f);
            P_.use_color = center_hit && cc.w > 0.0f;
        }
        P_.inv_ty = 1.0f / P_.ts.y;
        P_.form = spatial_form(P_.ts, k_par, k_perp);
    }

    // `done`: one thread, the sum of the groups behind it; two, their first group
    FilterSums done[2] = {};
    int left = kGroupRows;
#pragma unroll 1
    for (int r = sub * (kRows / S); r < (sub + 1) * (kRows / S); ++r) {
        const uint4 hits = s_hits[sy + r];
        const float4* row = &s_tap[sy + r][sx + kFilterRadius];
        // window rows: dy = r - 5 of the upper pixel, r - 6 of the lower
        float vertex[2], across[2], reject[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int dy = r - kFilterRadius - q;
            const bool in = dy >= -kFilterRadius && dy <= kFilterRadius;
            reject[q] = in ? depth_reject : -1.0f;
            const float fdy = (float)dy;
            vertex[q] = __fmaf_rn(P[q].form.rh, fdy, P[q].form.rl * fdy);
            across[q] = P[q].form.c * (fdy * fdy);
            if (in) {
                const uint32_t strip = strip_row(P[q].ts, P[q].inv_ty, dy, strip2);
                P[q].h_center += __popc(__funnelshift_r(hits.x, hits.y, sx) & strip);
                P[q].h_cons += __popc(__funnelshift_r(hits.z, hits.w, sx) & strip);
            }
        }
#pragma unroll
        for (int dx = -kFilterRadius; dx <= kFilterRadius; ++dx) {
            const float4 tap = row[dx];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                FilterPixel& P_ = P[q];
                // evaluated for every tap, kept for those near in depth: predicated
                // sums cost less than the branches around them
                const float u = (float)dx - vertex[q];
                float e = __fmaf_rn(u * u, P_.form.a, across[q]);
                const float cx = P_.cx - tap.x, cy = P_.cy - tap.y, cz = P_.cz - tap.z;
                const float ec = __fmaf_rn(__fmaf_rn(cz, cz, __fmaf_rn(cy, cy, cx * cx)), k_col, e);
                e = P_.use_color ? ec : e;
                accumulate(fabsf(tap.w - P_.p_norm) <= reject[q], tap, ex2(-e), P_);
            }
        }
        if (S < kGroups && --left == 0) {  // a group's end
            left = kGroupRows;
            if (S == 1 || r == sub * (kRows / S) + kGroupRows - 1) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const FilterSums own = {P[q].ax, P[q].ay, P[q].az, P[q].weight};
                    done[q] = S == 1 && r >= kGroupRows ? done[q] + own : own;
                    P[q].ax = P[q].ay = P[q].az = P[q].weight = 0.0f;
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        FilterSums sum = done[q];
        if (S > 1) {
            const FilterSums own = {P[q].ax, P[q].ay, P[q].az, P[q].weight};
            auto from = [&](const FilterSums& v, int k) {  // thread k of the pair's
                return FilterSums{__shfl_sync(0xffffffffu, v.x, k, S), __shfl_sync(0xffffffffu, v.y, k, S),
                                  __shfl_sync(0xffffffffu, v.z, k, S), __shfl_sync(0xffffffffu, v.weight, k, S)};
            };
            if (S == 2) sum = ((from(done[q], 0) + from(own, 0)) + from(done[q], 1)) + from(own, 1);
            else sum = ((from(own, 0) + from(own, 1)) + from(own, 2)) + from(own, 3);
#pragma unroll
            for (int o = 1; o < S; o <<= 1) {
                P[q].h_center += __shfl_xor_sync(0xffffffffu, P[q].h_center, o);
                P[q].h_cons += __shfl_xor_sync(0xffffffffu, P[q].h_cons, o);
            }
        }
        P[q].ax = sum.x;
        P[q].ay = sum.y;
        P[q].az = sum.z;
        P[q].weight = sum.weight;
    }
    if (S > 1 && slot >= total) return;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        // with several threads a pair, the first writes the upper pixel, the second the lower
        if (!((entry >> (14 + q)) & 1u) || (S > 1 && sub != q)) continue;
        const FilterPixel& P_ = P[q];
        const uint32_t pix = (uint32_t)(by * TY + sy + q) * (uint32_t)width + (uint32_t)px;
        const unsigned long long center_word = __ldg(&a.center[pix]), cons_word = __ldg(&a.cons[pix]);
        const bool center_hit = !is_empty(center_word), cons_hit = !is_empty(cons_word);
        const unsigned long long w = center_hit ? center_word : cons_word;
        const float view_dist = dequantize_depth((uint32_t)(w >> 40), p.screen[2], p.screen[3]);
        float cx = P_.cx, cy = P_.cy, cz = P_.cz;
        if (P_.weight > 1e-5f) {
            const float inv = 1.0f / P_.weight;
            cx = P_.ax * inv;
            cy = P_.ay * inv;
            cz = P_.az * inv;
        }
        const float h_center = (float)P_.h_center, h_cons = (float)P_.h_cons;
        const float coverage = __fdiv_rn(h_center, fmaxf(h_center + h_cons, 1.0f));
        const float cons_depth = cons_hit ? __fdiv_rn(__uint2float_rn((uint32_t)(cons_word >> 40)), 16777214.0f) : 1.0f;
        const bool closer = cons_hit && center_hit && (P_.p_norm - cons_depth) >= closer_eps;
        float alpha = closer ? 1.0f : clampf(coverage, 0.0f, 1.0f);
        if (!center_hit && P_.weight <= 1e-5f) {
            alpha = 0.0f;
            cx = cy = cz = 0.0f;
        }
        const float4 out = make_float4(cx, cy, cz, alpha);
        a.filtered[pix] = out;
        a.filtered_depth[pix] = view_dist;
        if (KIND != kNone)
            composite_one<KIND>(p, out, view_dist, a.color, a.depth, depth_clear, px, by * TY + sy + q, pix);
    }
}

template <int TX, int TY, int S, int MIN_BLOCKS, CompositeKind KIND>
__global__ void __launch_bounds__(TX* TY* S / 2, MIN_BLOCKS) filter_kernel(const FilterArgs a) {
    filter_tile<TX, TY, S, KIND>(a, blockIdx.x, blockIdx.y, a.depth_clear);
}

// Tile t of the camera views' concatenated tile space -> (view, bx, by).
__device__ __forceinline__ uint32_t tile_view(const uint32_t* __restrict__ prefix, uint32_t n, uint32_t t) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Five blocks per SM (96 registers): 744 us on 24 grooms of the batch benchmark;
// six (80) 8 us more, eight (64, spilled) 47 more.
template <int TX, int TY>
__global__ void __launch_bounds__(TX* TY / 2, 5) batch_filter_kernel(const BatchView* __restrict__ views,
                                                             const uint32_t* __restrict__ prefix, uint32_t n_cam,
                                                             float depth_clear) {
    const uint32_t v = tile_view(prefix, n_cam, blockIdx.x);
    const BatchView& a = views[v];
    const uint32_t t = blockIdx.x - prefix[v];
    const uint32_t tiles_x = (a.width + TX - 1) / TX;
    filter_tile<TX, TY, 1, kClear>(a, (int32_t)(t % tiles_x), (int32_t)(t / tiles_x), depth_clear);
}

struct CompositeArgs {
    hg_hair_params p;
    const float4* color_src;
    const float* depth_src;
    float4* color;
    float* depth;
    float depth_clear;
};

template <CompositeKind KIND, class V>
__device__ __forceinline__ void composite_pixel(const V& a, const float4* __restrict__ color_src,
                                                const float* __restrict__ depth_src, float depth_clear, int32_t px,
                                                int32_t py) {
    const hg_hair_params& p = a.p;
    const int32_t width = f2i(p.screen[0]), height = f2i(p.screen[1]);
    if (px >= width || py >= height) return;
    const uint32_t pix = (uint32_t)py * (uint32_t)width + (uint32_t)px;
    composite_one<KIND>(p, __ldg(&color_src[pix]), __ldg(&depth_src[pix]), a.color, a.depth, depth_clear, px, py, pix);
}

template <CompositeKind KIND>
__global__ void composite_kernel(const CompositeArgs a) {
    composite_pixel<KIND>(a, a.color_src, a.depth_src, a.depth_clear, blockIdx.x * blockDim.x + threadIdx.x,
                          blockIdx.y * blockDim.y + threadIdx.y);
}

// The shaded colour straight to the target (filter off).
__global__ void batch_composite_kernel(const BatchView* __restrict__ views, const uint32_t* __restrict__ prefix,
                                       uint32_t n_cam, float depth_clear) {
    const uint32_t v = tile_view(prefix, n_cam, blockIdx.x);
    const BatchView& a = views[v];
    const uint32_t t = blockIdx.x - prefix[v];
    const uint32_t tiles_x = (a.width + blockDim.x - 1) / blockDim.x;
    composite_pixel<kClear>(a, a.shaded, a.shaded_depth, depth_clear,
                            (int32_t)((t % tiles_x) * blockDim.x + threadIdx.x),
                            (int32_t)((t / tiles_x) * blockDim.y + threadIdx.y));
}

__global__ void clear_color_kernel(float4* __restrict__ color, float* __restrict__ depth, size_t pixels,
                                   float depth_clear) {
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < pixels; i += stride) {
        color[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        depth[i] = depth_clear;
    }
}

}  // namespace

namespace {

template <CompositeKind KIND>
cudaError_t launch_filter_kind(hg_ctx* ctx, const FilterArgs& a) {
    const auto tiles = [&](uint32_t tx, uint32_t ty) {
        return dim3((ctx->width + tx - 1) / tx, (ctx->height + ty - 1) / ty);
    };
    const uint64_t px = (uint64_t)ctx->width * ctx->height;
    if (px <= kFilterSplit4) filter_kernel<16, 8, 4, 3, KIND><<<tiles(16, 8), 256, 0, ctx->stream>>>(a);
    else if (px <= kFilterSplit2) filter_kernel<32, 8, 2, 3, KIND><<<tiles(32, 8), 256, 0, ctx->stream>>>(a);
    else filter_kernel<16, 16, 1, 6, KIND><<<tiles(16, 16), 128, 0, ctx->stream>>>(a);
    return cudaGetLastError();
}

FilterArgs filter_args(hg_ctx* ctx, const hg_hair_params& p) {
    FilterArgs a;
    a.p = p;
    a.center = ctx->center;
    a.cons = ctx->cons;
    a.shaded = ctx->shaded;
    a.filtered = ctx->filtered;
    a.filtered_depth = ctx->filtered_depth;
    a.color = ctx->color;
    a.depth = ctx->depth;
    a.depth_clear = 0.0f;
    return a;
}

template <CompositeKind KIND>
cudaError_t launch_composite_kind(hg_ctx* ctx, const hg_hair_params& p, uint32_t source_filtered, float depth_clear) {
    CompositeArgs a;
    a.p = p;
    a.color_src = source_filtered ? ctx->filtered : ctx->shaded;
    a.depth_src = source_filtered ? ctx->filtered_depth : ctx->shaded_depth;
    a.color = ctx->color;
    a.depth = ctx->depth;
    a.depth_clear = depth_clear;
    dim3 block(32, 8);
    dim3 grid((ctx->width + 31) / 32, (ctx->height + 7) / 8);
    composite_kernel<KIND><<<grid, block, 0, ctx->stream>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_filter(hg_ctx* ctx, const hg_hair_params& p) {
    return launch_filter_kind<kNone>(ctx, filter_args(ctx, p));
}

cudaError_t launch_composite(hg_ctx* ctx, const hg_hair_params& p, uint32_t source_filtered) {
    return launch_composite_kind<kBlend>(ctx, p, source_filtered, 0.0f);
}

// The end of a frame in one launch: filter (when on) and composite, and with
// `clear` the colour target's clear, which then is written once instead of
// cleared, read and written (20 bytes a pixel for 60 and two launches).
cudaError_t launch_filter_composite(hg_ctx* ctx, const hg_hair_params& p, bool filter, bool clear, float depth_clear) {
    if (!filter)
        return clear ? launch_composite_kind<kClear>(ctx, p, 0u, depth_clear)
                     : launch_composite_kind<kBlend>(ctx, p, 0u, depth_clear);
    FilterArgs a = filter_args(ctx, p);
    a.depth_clear = depth_clear;
    return clear ? launch_filter_kind<kClear>(ctx, a) : launch_filter_kind<kBlend>(ctx, a);
}

// Every item's filter (when on), colour clear and composite in one launch.
cudaError_t launch_batch_filter_composite(hg_ctx* ctx, const BatchDev& b) {
    if (b.filter && b.total_ftiles) {
        if (b.filter_tile == 1) batch_filter_kernel<16, 16><<<b.total_ftiles, 128, 0, ctx->stream>>>(
            b.views, b.ftile_prefix, b.n_cam, b.depth_clear);
        else batch_filter_kernel<32, 8><<<b.total_ftiles, 128, 0, ctx->stream>>>(b.views, b.ftile_prefix, b.n_cam,
                                                                                b.depth_clear);
    } else if (!b.filter && b.total_tiles) {
        batch_composite_kernel<<<b.total_tiles, dim3(b.tile_w, b.tile_h), 0, ctx->stream>>>(b.views, b.tile_prefix,
                                                                                           b.n_cam, b.depth_clear);
    }
    return cudaGetLastError();
}

cudaError_t launch_clear_color(hg_ctx* ctx, float depth_clear) {
    size_t pixels = (size_t)ctx->width * ctx->height;
    int threads = 256;
    int blocks = (int)std::min<size_t>((pixels + threads - 1) / threads, (size_t)ctx->sm_count * 8);
    if (blocks < 1) blocks = 1;
    clear_color_kernel<<<blocks, threads, 0, ctx->stream>>>(ctx->color, ctx->depth, pixels, depth_clear);
    return cudaGetLastError();
}

}  // namespace hg
