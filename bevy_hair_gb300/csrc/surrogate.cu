// Learned shading surrogate: FP64 training samples of the hair lobes, the
// FP16 tensor-core networks' inference and training kernels (forward and
// backward of a 128-sample tile per block on mma.sync; weight gradients in the
// same block for the compact 2 x 32 network, in a kernel of their own for the
// 4 x 64 one; partial gradients summed by the Adam kernel), and their C entry
// points.  The reference has no counterpart; the shading it replaces is the
// Karis fit of shade.wesl:94-190.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>

#include <cmath>
#include <cstring>
#include <mutex>
#include <new>

#include "hg_internal.h"
#include "hg_mlp.cuh"
#include "hg_mlp_small.cuh"
#include "hg_mlp_tc.cuh"
#include "hg_ring.h"

namespace hg {
namespace {

using namespace mlp;

constexpr int kGl = 64;         // quadrature order
constexpr int kPairs = kGl / 2;  // nodes with gamma_i > 0; the others mirror them
// Per positive node: gamma_i, weight (Jacobian cos(gamma_i) included), sin and cos of gamma_i.
__constant__ double c_gl_x[kPairs];
__constant__ double c_gl_w[kPairs];
__constant__ double c_gl_sin[kPairs];
__constant__ double c_gl_cos[kPairs];
constexpr double kPiD = 3.14159265358979323846;

// ------------------------------------------------------------ FP64 lobes
//
// Single scattering S_p = M_p(theta_i + theta_o - alpha_p; beta_p) N_p(phi)
// (Marschner et al. 2003; d'Eon et al. 2011; Chiang et al. 2016) with
//   N_p(phi) = 1/2 Int A_p(h) D(phi - Phi_p(h); beta_n) dh,
// integrated over gamma_i = asin h with 64-point Gauss-Legendre (smooth in
// gamma_i; ~3e-11 relative against a 20001-point Simpson rule),
//   Phi_p = 2 p gamma_t - 2 gamma_i + p pi,  A_0 = F,  A_1 = (1-F)^2 T,  A_2 = (1-F)^2 F T^2,
// and the local back-scattering of the dual-scattering model (Zinke et al.
// 2008, Eqs. 13-17) from the same lobes' exact forward/backward azimuthal
// masses.  Longitudinal shapes follow shade.wesl:124-128.
//
// The kernel is bound by the FP64 pipe (a small fraction of the FP32 rate on
// this GPU), so the work is arranged to issue as few FP64 instructions as the
// same quadrature allows:
//  - the nodes are symmetric and A_p is even in gamma_i, so F, T and gamma_t
//    are formed for 32 nodes instead of 64, from tabulated sin / cos of the
//    nodes;
//  - the backward mass of the wrapped Gaussian, the part of it in [-pi/2,
//    pi/2], is even in the exit azimuth c and has the Fourier series
//      1/2 + (2/pi) sum over odd n of (-1)^((n-1)/2) exp(-n^2 beta_n^2 / 2) / n cos(n c),
//    whose terms fall below 3e-17 after at most 22 (beta_n >= 0.2), 10 on
//    average.  One Clenshaw recurrence in cos(2c) per node and lobe (cos c
//    comes from gamma_t and gamma_i by angle sums) replaces 11 error functions;
//    the forward mass is the rest of 1;
//  - of the three images of the wrapped density, the far one is below 4e-14
//    of the central one and is scaled from it in float.
// 262,144 samples: 76.2 ms with 64 nodes and the 11 error functions a node
// and lobe, 12.9 ms so (both on 152 SMs).

constexpr int kBackTerms = 22;  // odd n up to 43: n^2 beta_n^2 / 2 > 38 beyond, for beta_n >= 0.2
constexpr double kBackCut = 38.0;

__device__ __forceinline__ double gauss_d(double b, double x) {
    const double bb = fmax(b, 1e-3);
    return exp(-0.5 * x * x / (bb * bb)) / (2.5066282746310002 * bb);
}

struct NodeTerms {
    double gt_sin, gt_cos;  // sine and cosine of gamma_t
    double f, tr[3];
};

// The terms of the quadrature nodes +-gamma_i (sin su, cos cu) that do not
// depend on the sign: gamma_t for +gamma_i, Fresnel and transmittance.
__device__ __forceinline__ NodeTerms node_terms(double su, double cu, double cos_td, double inv_eta_p,
                                                double inv_cos_tt2, double eta, double inv_eta2, const double sa[3]) {
    NodeTerms n;
    n.gt_sin = su * inv_eta_p;
    n.gt_cos = sqrt(1.0 - n.gt_sin * n.gt_sin);
    const double c = fmin(fmax(cos_td * cu, 0.0), 1.0);
    const double st2 = (1.0 - c * c) * inv_eta2;
    if (st2 >= 1.0) {
        n.f = 1.0;
    } else {
        const double ct = sqrt(1.0 - st2);
        // 1/2 (A^2 / B^2 + C^2 / D^2) over one denominator
        const double a = c - eta * ct, b = c + eta * ct, cc = eta * c - ct, d = eta * c + ct;
        const double ad = a * d, bc = b * cc, bd = b * d;
        n.f = 0.5 * (ad * ad + bc * bc) / (bd * bd);
    }
    const double path = n.gt_cos * inv_cos_tt2;
#pragma unroll
    for (int c2 = 0; c2 < 3; ++c2) n.tr[c2] = exp(-sa[c2] * path);
    return n;
}

// Unnormalised wrapped Gaussian exp(-d^2 i) over the images d, d +- 2 pi, at
// the angle x (any real).
__device__ __forceinline__ double wrapped_gauss(double x, double i) {
    const double two_pi = 2.0 * kPiD;
    const double h = fabs(x - two_pi * rint(x * (1.0 / two_pi)));
    double e = exp(-h * h * i);
    const double n = two_pi - h;  // the nearer image
    const double fall = 4.0 * kPiD * i;
    // below 4e-18 of the central term it does not change the sum
    const double near_ = fall * (kPiD - h) < 40.0 ? exp(-n * n * i) : 0.0;
    e += e * (double)__expf(-(float)(fall * (kPiD + h)));  // the farther image
    return e + near_;
}

// Sums over the L lanes that share a sample (L a power of two).
template <int L>
__device__ __forceinline__ double lane_sum(double v) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The twelve lobes of one sample on L adjacent lanes (all of the warp's lanes
// call it; every lane of a sample gets the result).  q: this thread's column
// of kBackTerms shared doubles, `stride` apart.
template <int L>
__device__ void lobes_fp64(const float* in, double tilt, double* q, int stride, double out[12]) {
    const int sub = (int)(threadIdx.x & (L - 1));
    const double sin_i = fmin(fmax((double)in[0], -1.0), 1.0), sin_o = fmin(fmax((double)in[1], -1.0), 1.0);
    const double phi = atan2((double)in[3], (double)in[2]);
    const double sa[3] = {in[4], in[5], in[6]};
    const double beta_m = in[7], beta_n = in[8], eta = in[9];
    const double th_i = asin(sin_i), th_o = asin(sin_o), th_h = th_i + th_o;
    const double alpha[3] = {tilt, -0.5 * tilt, -1.5 * tilt};
    const double beta[3] = {beta_m, 0.5 * beta_m, 2.0 * beta_m};
    const double inv_eta2 = 1.0 / (eta * eta);

    // single scattering at theta_d = (theta_o - theta_i) / 2
    {
        const double td = 0.5 * (th_o - th_i);
        const double cos_td = fmax(cos(td), 1e-3), sin_td = sin(td);
        const double inv_eta_p = cos_td / sqrt(eta * eta - sin_td * sin_td);
        const double sin_tt = sin_td / eta, inv_cos_tt2 = 2.0 / sqrt(1.0 - sin_tt * sin_tt);
        const double inv2s2 = 0.5 / (beta_n * beta_n), norm = 1.0 / (2.5066282746310002 * beta_n);
        double n0 = 0.0, n1[3] = {}, n2[3] = {};
        for (int i = sub; i < kPairs; i += L) {
            const double u = c_gl_x[i];
            const NodeTerms nt =
                node_terms(c_gl_sin[i], c_gl_cos[i], cos_td, inv_eta_p, inv_cos_tt2, eta, inv_eta2, sa);
            const double gt = asin(nt.gt_sin);
            const double w = c_gl_w[i];
            // exit azimuths p pi +- (2 p gamma_t - 2 gamma_i) of the two nodes
            double d[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const double a = 2.0 * p * gt - 2.0 * u, x = phi - p * kPiD;
                d[p] = w * (wrapped_gauss(x - a, inv2s2) + wrapped_gauss(x + a, inv2s2));
            }
            const double omf2 = (1.0 - nt.f) * (1.0 - nt.f);
            n0 += d[0] * nt.f;
            const double d1 = d[1] * omf2, d2 = d[2] * omf2 * nt.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                n1[c] += d1 * nt.tr[c];
                n2[c] += d2 * (nt.tr[c] * nt.tr[c]);
            }
        }
        n0 = lane_sum<L>(n0);
        const double m0 = norm * gauss_d(beta[0], th_h - alpha[0]), m1 = norm * gauss_d(beta[1], th_h - alpha[1]),
                     m2 = norm * gauss_d(beta[2], th_h - alpha[2]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            out[c] = m0 * 0.5 * n0;
            out[3 + c] = m1 * 0.5 * lane_sum<L>(n1[c]);
            out[6 + c] = m2 * 0.5 * lane_sum<L>(n2[c]);
        }
    }

    // dual scattering at the specular cone, theta_d = theta_o (shade.wesl:444)
    const double cos_to = fmax(sqrt(fmax(1.0 - sin_o * sin_o, 1e-6)), 1e-3);
    const double sin_to = sqrt(fmax(0.0, 1.0 - cos_to * cos_to));
    const double inv_eta_p = cos_to / sqrt(eta * eta - sin_to * sin_to);
    const double sin_tt = sin_to / eta, inv_cos_tt2 = 2.0 / sqrt(1.0 - sin_tt * sin_tt);
    // coefficients of the backward mass's odd cosine series
    const double half_b2 = 0.5 * beta_n * beta_n;
    int terms = 0;
    for (; terms < kBackTerms; ++terms) {
        const double n = 2 * terms + 1;
        if (n * n * half_b2 > kBackCut) break;
        q[terms * stride] = (terms & 1 ? -2.0 : 2.0) / (kPiD * n) * exp(-n * n * half_b2);
    }
    auto back_mass = [&](double cos_c) {
        const double x = 4.0 * cos_c * cos_c - 2.0;  // 2 cos 2c
        double b1 = 0.0, b2 = 0.0;
        for (int k = terms - 1; k >= 0; --k) {
            const double b0 = fma(x, b1, q[k * stride] - b2);
            b2 = b1;
            b1 = b0;
        }
        return fma(cos_c, b1 - b2, 0.5);
    };
    double all0 = 0.0, all1[3] = {}, all2[3] = {}, back0 = 0.0, back1[3] = {}, back2[3] = {};
    for (int i = sub; i < kPairs; i += L) {
        const double su = c_gl_sin[i], cu = c_gl_cos[i];
        const NodeTerms nt = node_terms(su, cu, cos_to, inv_eta_p, inv_cos_tt2, eta, inv_eta2, sa);
        // cosines of 2 gamma_t p - 2 gamma_i + p pi (the mirrored node's has the same)
        const double c2u = 1.0 - 2.0 * su * su, s2u = 2.0 * su * cu;
        const double c2t = 1.0 - 2.0 * nt.gt_sin * nt.gt_sin, s2t = 2.0 * nt.gt_sin * nt.gt_cos;
        const double c4t = 1.0 - 2.0 * s2t * s2t, s4t = 2.0 * s2t * c2t;
        const double mb0 = back_mass(c2u), mb1 = back_mass(-(c2t * c2u + s2t * s2u)), mb2 = back_mass(c4t * c2u + s4t * s2u);
        const double w = 2.0 * c_gl_w[i];
        const double omf2 = w * (1.0 - nt.f) * (1.0 - nt.f);
        const double wa0 = w * nt.f;
        all0 += wa0;
        back0 += wa0 * mb0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double wa1 = omf2 * nt.tr[c], wa2 = omf2 * nt.f * (nt.tr[c] * nt.tr[c]);
            all1[c] += wa1;
            all2[c] += wa2;
            back1[c] += wa1 * mb1;
            back2[c] += wa2 * mb2;
        }
    }
    all0 = lane_sum<L>(all0);
    back0 = lane_sum<L>(back0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double b[3] = {0.5 * back0, 0.5 * lane_sum<L>(back1[c]), 0.5 * lane_sum<L>(back2[c])};
        const double f[3] = {0.5 * all0 - b[0], 0.5 * lane_sum<L>(all1[c]) - b[1], 0.5 * lane_sum<L>(all2[c]) - b[2]};
        const double a_f = fmin(f[0] + f[1] + f[2], 0.95);
        const double a_b = b[0] + b[1] + b[2];
        const double b2[3] = {beta[0] * beta[0], beta[1] * beta[1], beta[2] * beta[2]};
        const double tf = fmax(a_f, 1e-5), tb = fmax(a_b, 1e-5);
        const double beta_f2 = (f[0] * b2[0] + f[1] * b2[1] + f[2] * b2[2]) / tf;
        const double alpha_b = (b[0] * alpha[0] + b[1] * alpha[1] + b[2] * alpha[2]) / tb;
        const double beta_b2 = (b[0] * b2[0] + b[1] * b2[1] + b[2] * b2[2]) / tb;
        const double af2 = a_f * a_f, rest = 1.0 - af2, ab2 = a_b * a_b, ab3 = ab2 * a_b;
        const double a_back = a_b * af2 / rest + ab3 * af2 / (rest * rest * rest);
        const double delta_b = alpha_b * (1.0 - 2.0 * ab2 / (rest * rest)) +
                               alpha_b * (2.0 * rest * rest + 4.0 * af2 * ab2) / (rest * rest * rest);
        const double beta_f = sqrt(beta_f2), beta_b = sqrt(beta_b2);
        const double sigma_b = (1.0 + 0.7 * af2) *
                               (a_b * sqrt(2.0 * beta_f2 + beta_b2) + ab3 * sqrt(2.0 * beta_f2 + 3.0 * beta_b2)) /
                               fmax(a_b + ab3 * (2.0 * beta_f + 3.0 * beta_b), 1e-5);
        out[9 + c] = 2.0 * a_back * gauss_d(sigma_b, th_h - delta_b) / kPiD;
    }
}

// SplitMix64 (Steele, Lea and Flood 2014) as a counter-based generator.
__device__ __forceinline__ uint64_t splitmix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float unit_float(uint64_t seed, uint64_t index, uint32_t dim) {
    const uint64_t h = splitmix(seed ^ splitmix(index * 16u + dim));
    return (float)(uint32_t)(h >> 40) * 0x1p-24f;
}

struct SampleArgs {
    uint64_t seed, first;
    uint32_t n;
    double tilt;
    float* inputs;   // [n][10]
    float* targets;  // [n][12] log1p(lobe / kScale), nullable
    double* lobes;   // [n][12], nullable
};

// Training distribution: sin theta_i, sin theta_o uniform in [-1, 1); phi
// uniform in [0, pi); sigma_a log-uniform in [0.02, 8]; beta_m uniform in
// [0.03, 0.3]; beta_n uniform in [0.2, 0.8]; eta = 1.55.
// L lanes share a sample's quadrature nodes; a warp whose last samples lie past
// the count evaluates the last one again and stores nothing.
constexpr int kSampleThreads = 128;
template <int L>
__global__ void __launch_bounds__(kSampleThreads) samples_kernel(const SampleArgs a) {
    __shared__ double s_q[kBackTerms][kSampleThreads];
    const uint32_t own = (blockIdx.x * kSampleThreads + threadIdx.x) / L;
    const uint32_t k = min(own, a.n - 1u);
    const uint64_t idx = a.first + k;
    float x[10];
    x[0] = 2.0f * unit_float(a.seed, idx, 0) - 1.0f;
    x[1] = 2.0f * unit_float(a.seed, idx, 1) - 1.0f;
    const double phi = kPiD * (double)unit_float(a.seed, idx, 2);
    x[2] = (float)cos(phi);
    x[3] = (float)sin(phi);
    const double l0 = log(0.02), span = log(400.0);
#pragma unroll
    for (int c = 0; c < 3; ++c) x[4 + c] = (float)exp(l0 + span * (double)unit_float(a.seed, idx, 3 + c));
    x[7] = 0.03f + 0.27f * unit_float(a.seed, idx, 6);
    x[8] = 0.2f + 0.6f * unit_float(a.seed, idx, 7);
    x[9] = 1.55f;
    double out[12];
    lobes_fp64<L>(x, a.tilt, &s_q[0][threadIdx.x], kSampleThreads, out);
    if (own >= a.n || threadIdx.x % L != 0) return;
#pragma unroll
    for (int i = 0; i < 10; ++i) a.inputs[(size_t)k * 10 + i] = x[i];
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        if (a.lobes) a.lobes[(size_t)k * 12 + i] = out[i];
        if (a.targets) a.targets[(size_t)k * 12 + i] = (float)log1p(out[i] / (double)kScale);
    }
}

// ------------------------------------------------------------ inference

constexpr int kWarps = 8;

__device__ __forceinline__ void load_raw(const float* __restrict__ inputs, uint32_t i, bool valid, float raw[10]) {
    const float dflt[10] = {0.0f, 0.0f, 1.0f, 0.0f, 0.4f, 0.4f, 0.4f, kBetaMMid, kBetaNMid, kEtaMid};
#pragma unroll
    for (int c = 0; c < 10; ++c) raw[c] = valid ? __ldg(&inputs[(size_t)i * 10 + c]) : dflt[c];
}

struct InferArgs {
    const float* inputs;
    uint32_t n;
    const __half* w16;
    const float* params;
    float* lobes;  // [n][12] decoded, nullable
    float* net;    // [n][12] network outputs, nullable
};

// A warp's rows of K outputs, one row per lane, to `rows` (at most 32)
// consecutive rows of `out`, 32 consecutive words at a time.  stage: 32 (K + 1)
// floats of the warp's own.
template <int K>
__device__ __forceinline__ void store_rows(float* stage, const float y[K], float* __restrict__ out, uint32_t rows,
                                           uint32_t lane) {
#pragma unroll
    for (int c = 0; c < K; ++c) stage[lane * (K + 1) + c] = y[c];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < K; ++c) {
        const uint32_t i = 32u * c + lane;
        if (i < rows * K) out[i] = stage[i / K * (K + 1) + i % K];
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kWarps * 32) infer_kernel(const InferArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    FwdWeights& w = *reinterpret_cast<FwdWeights*>(smem);
    WarpIo* io = reinterpret_cast<WarpIo*>(smem + sizeof(FwdWeights));
    load_fwd(w, a.w16, a.params, threadIdx.x, blockDim.x);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t base = (blockIdx.x * kWarps + warp) * 32u; base < a.n; base += gridDim.x * kWarps * 32u) {
        const uint32_t i = base + lane;
        const bool valid = i < a.n;
        float raw[10], x[10], y[12];
        load_raw(a.inputs, i, valid, raw);
        normalise(raw, x);
        forward_fast(w, io[warp], x, y);
        const uint32_t rows = min(a.n - base, 32u);
        if (a.net) store_rows<12>(&io[warp].y[0][0], y, a.net + (size_t)base * 12, rows, lane);
        if (a.lobes) {
#pragma unroll
            for (int c = 0; c < 12; ++c) y[c] = decode(y[c]);
            store_rows<12>(&io[warp].y[0][0], y, a.lobes + (size_t)base * 12, rows, lane);
        }
    }
}

// The compact network (hg_mlp_small.cuh) on mma.sync, 32 samples per warp;
// three outputs per sample (the BSDF rgb).
__global__ void __launch_bounds__(kWarps * 32) infer_small_kernel(const InferArgs a) {
    __shared__ __align__(16) mlps::Weights w;
    __shared__ __align__(16) WarpIo io[kWarps];
    mlps::load(w, a.w16, a.params, threadIdx.x, blockDim.x);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t base = (blockIdx.x * kWarps + warp) * 32u; base < a.n; base += gridDim.x * kWarps * 32u) {
        const uint32_t i = base + lane;
        const bool valid = i < a.n;
        float raw[10], x[10], y[mlp::kUsedOut];  // forward() fills 12 columns; the first kUsedOut are outputs
        load_raw(a.inputs, i, valid, raw);
        normalise(raw, x);
        mlps::forward(w, io[warp], x, y);
        constexpr int k = mlps::kUsedOut;
        const uint32_t rows = min(a.n - base, 32u);
        if (a.net) store_rows<k>(&io[warp].y[0][0], y, a.net + (size_t)base * k, rows, lane);
        if (a.lobes) {
#pragma unroll
            for (int c = 0; c < k; ++c) y[c] = decode(y[c]);
            store_rows<k>(&io[warp].y[0][0], y, a.lobes + (size_t)base * k, rows, lane);
        }
    }
}

// The same evaluation on tcgen05: four chains of 128 rows per CTA.  A chunk's
// inputs are read while the chunk before is evaluated; its outputs leave in
// rows of 32 consecutive words (store_rows): a row per thread touched 12 times
// the sectors.
__global__ void __launch_bounds__(tc::kThreads, 1) infer_tc_kernel(const InferArgs a, uint32_t* err) {
    extern __shared__ __align__(128) uint8_t smem_tc[];
    tc::Chain c = tc::setup(smem_tc, a.w16, a.params);
    const uint32_t g = threadIdx.x >> 7, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float* stage = reinterpret_cast<float*>(smem_tc + tc::kOffStage) + warp * tc::kStageFloats;
    const uint32_t chunks = a.n / tc::kM + (a.n % tc::kM != 0u);
    const uint32_t step = gridDim.x * tc::kChains;
    uint32_t ch = blockIdx.x * tc::kChains + g;
    bool failed = false;
    float raw[10];
    if (ch < chunks) load_raw(a.inputs, ch * tc::kM + c.row, ch * tc::kM + c.row < a.n, raw);
    for (; ch < chunks; ch += step) {
        float x[10], y[12];
        normalise(raw, x);
        if (ch + step < chunks) load_raw(a.inputs, (ch + step) * tc::kM + c.row, (ch + step) * tc::kM + c.row < a.n, raw);
        if (!tc::forward(c, x, y)) {
            failed = true;
            break;
        }
        const uint32_t first = ch * tc::kM + (c.row & ~31u);
        const uint32_t rows = first < a.n ? min(a.n - first, 32u) : 0u;
        if (a.net) store_rows<12>(stage, y, a.net + (size_t)first * 12, rows, lane);
        if (a.lobes) {
#pragma unroll
            for (int k = 0; k < 12; ++k) y[k] = decode(y[k]);
            store_rows<12>(stage, y, a.lobes + (size_t)first * 12, rows, lane);
        }
    }
    if (failed && c.row == 0) atomicOr(err, tc::kErrTimeout);
    tc::teardown(smem_tc, c, failed);
}

// ------------------------------------------------------------ training

// stmatrix of four 8x8 FP16 matrices, each stored transposed: lane l gives the
// address of stored row l % 8 of matrix l / 8.
__device__ __forceinline__ void stsm_x4_trans(void* p, const uint32_t r[4]) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}

__device__ __forceinline__ void ldsm_x2(uint32_t r[2], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}

__device__ __forceinline__ void ldsm_x4_trans(uint32_t r[4], const void* p) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// Asynchronous copy of a rows x cols block of halves (cols a multiple of 8)
// into padded shared rows; wait_copies() before the block's barrier.
template <int PAD>
__device__ __forceinline__ void copy_rows_async(__half (*dst)[PAD], const __half* __restrict__ src, int rows, int cols,
                                                int tid, int nthreads) {
    const int per_row = cols / 8;
    for (int i = tid; i < rows * per_row; i += nthreads) {
        const int r = i / per_row, c = (i - r * per_row) * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&dst[r][c])),
                     "l"(src + r * cols + c)
                     : "memory");
    }
}
__device__ __forceinline__ void wait_copies() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The training kernels are programmatic dependents of one another (train,
// Adam, train, ...): a kernel's blocks may be placed while the one before
// finishes, and wait here, before they touch memory, until it has completed.
__device__ __forceinline__ void wait_for_previous_kernel() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

constexpr int kTrainWarps = 8;
constexpr int kTrainThreads = 32 * kTrainWarps;
constexpr int kTrainTile = 16 * kTrainWarps;  // samples a block takes at a time, 16 (one MMA row tile) per warp
constexpr int kTilePad = kTrainTile + 8;      // halves per transposed row (conflict-free ldmatrix and stmatrix)

// acc[nt] = bias + A W^T for 16 samples, N = 8*NT outputs, K = 16*KT inputs;
// bias may be null (zero).  The products are those of layer_ldsm.
template <int NT, int KT, int PAD>
__device__ __forceinline__ void layer16(float acc[NT][4], const uint32_t a[KT][4], const __half (*w)[PAD],
                                        const float* bias, int lane) {
    const int t = lane & 3, mat = lane >> 3, r = lane & 7;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        acc[nt][0] = acc[nt][2] = bias ? bias[nt * 8 + 2 * t] : 0.0f;
        acc[nt][1] = acc[nt][3] = bias ? bias[nt * 8 + 2 * t + 1] : 0.0f;
    }
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
#pragma unroll
        for (int nt = 0; nt < NT; nt += 2) {
            uint32_t b[4];
            ldsm_x4(b, &w[(nt + (mat >> 1)) * 8 + r][kt * 16 + (mat & 1) * 8]);
            mma(acc[nt], a[kt], b[0], b[1]);
            mma(acc[nt + 1], a[kt], b[2], b[3]);
        }
    }
}

// C fragments of a 16*KT-wide layer -> A fragments of the next; RELU applies
// max(x, 0) first.
template <bool RELU, int KT>
__device__ __forceinline__ void c_to_a16(const float acc[2 * KT][4], uint32_t a[KT][4]) {
    auto v = [](float x) { return RELU ? fmaxf(x, 0.0f) : x; };
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* c = acc[2 * kt + h];
            a[kt][2 * h] = pack_h2(v(c[0]), v(c[1]));
            a[kt][2 * h + 1] = pack_h2(v(c[2]), v(c[3]));
        }
}

// The address of lane's row of the 16 x 16 block kt of [unit][sample] storage
// that fragment registers r = lane / 8 transpose to and from: units
// (r >> 1) * 8.., samples (r & 1) * 8...
__device__ __forceinline__ __half* block_row(__half (*m)[kTilePad], int kt, int col0, int lane) {
    const int r = lane >> 3, i = lane & 7;
    return &m[kt * 16 + (r >> 1) * 8 + i][col0 + (r & 1) * 8];
}

// A fragments (rows = the warp's 16 samples) into dst[unit][col0 + sample].
template <int KT>
__device__ __forceinline__ void store_t(__half (*dst)[kTilePad], const uint32_t a[KT][4], int col0, int lane) {
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) stsm_x4_trans(block_row(dst, kt, col0, lane), a[kt]);
}

// C fragments, zeroed where the ReLU output stored in h[unit][col0 + sample]
// is zero -> A fragments.  The stored values are +0 or positive, so bit 15 of
// value + 0x7fff says "not zero"; the byte permute spreads it over the half.
template <int KT>
__device__ __forceinline__ void masked_to_a16(const float acc[2 * KT][4], __half (*h)[kTilePad], uint32_t a[KT][4],
                                              int col0, int lane) {
    c_to_a16<false, KT>(acc, a);
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        uint32_t v[4];
        ldsm_x4_trans(v, block_row(h, kt, col0, lane));
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint32_t m;
            asm("prmt.b32 %0, %1, 0, 0xBB99;\n" : "=r"(m) : "r"(v[r] + 0x7fff7fffu));
            a[kt][r] &= m;
        }
    }
}

// Two adjacent partial gradients: stored by the block's first tile, added to
// by its later ones (the same thread, so in a fixed order).
__device__ __forceinline__ void put2(float* p, float x, float y, bool add) {
    float2 v = make_float2(x, y);
    if (add) {
        const float2 o = *reinterpret_cast<const float2*>(p);
        v.x += o.x;
        v.y += o.y;
    }
    *reinterpret_cast<float2*>(p) = v;
}

// Rows m0..m0+15, columns n0..n0+7 of dW = A B^T over a tile's samples (A =
// dZ^T, B = H^T, both [unit][sample] in shared memory) into the block's
// partial gradient gw (row length n_cols); with gb, also the row sums of A
// (the bias gradient), as a product with ones.  One warp.
__device__ __forceinline__ void wgrad_tile(const __half (*A)[kTilePad], const __half (*B)[kTilePad], int m0, int n0,
                                           float* gw, int n_cols, float* gb, bool add, int lane) {
    const int g = lane >> 2, t = lane & 3, mat = lane >> 3, r = lane & 7;
    float acc[4] = {}, sum[4] = {};
#pragma unroll
    for (int k = 0; k < kTrainTile; k += 16) {
        uint32_t af[4], b[2];
        ldsm_x4(af, &A[m0 + r + (mat & 1) * 8][k + (mat >> 1) * 8]);
        ldsm_x2(b, &B[n0 + r][k + (mat & 1) * 8]);
        if (gb) mma(sum, af, 0x3C003C00u, 0x3C003C00u);
        mma(acc, af, b[0], b[1]);
    }
    float* p = gw + (m0 + g) * n_cols + n0 + 2 * t;
    put2(p, acc[0], acc[1], add);
    put2(p + 8 * n_cols, acc[2], acc[3], add);
    if (gb && t == 0) {
        gb[m0 + g] = sum[0] + (add ? gb[m0 + g] : 0.0f);
        gb[m0 + g + 8] = sum[2] + (add ? gb[m0 + g + 8] : 0.0f);
    }
}

struct TileActs;

struct TrainArgs {
    const float* inputs;   // [n][10]
    const float* targets;  // [n][12] transformed
    uint32_t n;
    const __half* w16;
    const __half* wt16;    // transposed copies (4 x 64 network only)
    const float* params;
    TileActs* acts;    // 4 x 64: [tiles] activations and deltas for wgrad_kernel
    float* part;       // compact: [blocks][parameters] partial gradients, written whole
    float* loss_part;  // [blocks] partial sums of squared errors
};

// A tile's network inputs and targets, one row per sample.
struct TileRows {
    __half x[kTrainTile][kIn + 8];     // normalised inputs
    float y[kTrainTile][kUsedOut + 1]; // targets; column kUsedOut: 1 for a real sample
};

// The tile from sample `base`: the first half of the block's threads loads and
// normalises the inputs, the second the targets.  Ends with a barrier.
__device__ __forceinline__ void load_tile(TileRows& rows, const TrainArgs& a, uint32_t base) {
    const int row = threadIdx.x % kTrainTile;
    const uint32_t i = base + row;
    const bool valid = i < a.n;
    if (threadIdx.x < kTrainTile) {
        float raw[10], x[10];
        load_raw(a.inputs, i, valid, raw);
        normalise(raw, x);
#pragma unroll
        for (int k = 0; k < kIn; k += 2)
            *reinterpret_cast<uint32_t*>(&rows.x[row][k]) =
                pack_h2(k < kUsedIn ? x[k] : 0.0f, k + 1 < kUsedIn ? x[k + 1] : 0.0f);
    } else {
#pragma unroll
        for (int c = 0; c < kUsedOut; ++c) rows.y[row][c] = valid ? __ldg(&a.targets[(size_t)i * 12 + c]) : 0.0f;
        rows.y[row][kUsedOut] = valid ? 1.0f : 0.0f;
    }
    __syncthreads();
}
static_assert(kTrainThreads == 2 * kTrainTile, "half of the threads load inputs, half targets");

__device__ __forceinline__ void input_frags16(const TileRows& rows, uint32_t a0[1][4], int col0, int g, int t) {
    a0[0][0] = ld32(&rows.x[col0 + g][2 * t]);
    a0[0][1] = ld32(&rows.x[col0 + g + 8][2 * t]);
    a0[0][2] = ld32(&rows.x[col0 + g][2 * t + 8]);
    a0[0][3] = ld32(&rows.x[col0 + g + 8][2 * t + 8]);
}

// The block's sum of squared errors from its threads' shares.
__device__ __forceinline__ void put_loss(float lsum, float* s_loss, float* out) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if ((threadIdx.x & 31) == 0) s_loss[threadIdx.x >> 5] = lsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float l = 0.0f;
        for (int w = 0; w < kTrainWarps; ++w) l += s_loss[w];
        *out = l;
    }
}

// What the 4 x 64 network's weight gradients need of a tile, [unit][sample]:
// written to memory whole, padding and all, so that one bulk copy stores it
// and a row range of it loads as one.
struct TileActs {
    __half x[kIn][kTilePad];       // layer-1 inputs
    __half h[4][kHid][kTilePad];   // hidden activations h1..h4
    __half dz[4][kHid][kTilePad];  // pre-activation gradients of layers 1..4
    __half dz5[kOut][kTilePad];    // output gradients
};
constexpr uint32_t kActRowBytes = kTilePad * 2;
constexpr uint32_t kActRowH = kIn, kActRowDz = kActRowH + 4 * kHid, kActRowDz5 = kActRowDz + 4 * kHid;
static_assert(sizeof(TileActs) == (kActRowDz5 + kOut) * kActRowBytes && kActRowBytes % 16 == 0, "rows of 272 bytes");

struct TrainSmem {
    FwdWeights fw;
    BwdWeights bw;
    TileActs act;
    TileRows rows;
    float loss[kTrainWarps];
};
static_assert(sizeof(FwdWeights) % 16 == 0 && sizeof(BwdWeights) % 16 == 0 && offsetof(TrainSmem, act) % 16 == 0,
              "ldmatrix rows and bulk copies on 16-byte boundaries");
static_assert(sizeof(TrainSmem) <= 227 * 1024, "train kernel shared memory");

// Forward and backward of 128-sample tiles of a training batch, 16 samples a
// warp on mma.sync; activations and deltas are transposed in shared memory
// (stmatrix) and leave with one bulk copy per tile for wgrad_kernel.  The
// loss is the sum over samples and the 12 outputs of (y - target)^2, so dL/dy
// = 2 (y - target); the 1/(n*12) of the mean is applied by the optimiser.
//
// Bound by latency: at a batch of 16,384 an SM holds one tile, and a tile is
// ten dependent layers.  Eight warps of 16 samples (two per scheduler) hide
// more of it than four of 32, although each weight fragment then feeds half
// the products.  A step of 16,384 samples (152 SMs): 157 us with a row-per-lane
// transpose through memory and a weight-gradient kernel of 40 blocks, 22 us
// now (by ncu, cold caches: this kernel 11 us, wgrad_kernel 9.4, Adam 3.8).
__global__ void __launch_bounds__(kTrainThreads, 1) train_kernel(const TrainArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem);
    TileActs& A = S.act;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    wait_for_previous_kernel();
    copy_rows_async<kPadIn>(S.fw.w1, a.w16 + kW1, kHid, kIn, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.fw.w2, a.w16 + kW2, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.fw.w3, a.w16 + kW3, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.fw.w4, a.w16 + kW4, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.fw.w5, a.w16 + kW5, kOut, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.bw.w2t, a.wt16 + kT2, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.bw.w3t, a.wt16 + kT3, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadHid>(S.bw.w4t, a.wt16 + kT4, kHid, kHid, tid, kTrainThreads);
    copy_rows_async<kPadIn>(S.bw.w5t, a.wt16 + kT5, kHid, kOut, tid, kTrainThreads);
    for (int i = tid; i < kHid; i += kTrainThreads) {
        S.fw.b1[i] = a.params[kB1 + i];
        S.fw.b2[i] = a.params[kB2 + i];
        S.fw.b3[i] = a.params[kB3 + i];
        S.fw.b4[i] = a.params[kB4 + i];
        if (i < kOut) S.fw.b5[i] = a.params[kB5 + i];
    }
    const int col0 = 16 * warp;
    float lsum = 0.0f;
    const uint32_t tiles = a.n / kTrainTile + (a.n % kTrainTile != 0u);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        wait_copies();  // the weights, before the first tile's barrier
        // the previous tile's copy must have read the tile buffer (its issuer waits)
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
        load_tile(S.rows, a, tile * kTrainTile);
        uint32_t a0[1][4];
        input_frags16(S.rows, a0, col0, g, t);
        store_t<1>(A.x, a0, col0, lane);

        float acc[8][4];
        uint32_t h[4][4];
        layer16<8, 1, kPadIn>(acc, a0, S.fw.w1, S.fw.b1, lane);
        c_to_a16<true, 4>(acc, h);
        store_t<4>(A.h[0], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.fw.w2, S.fw.b2, lane);
        c_to_a16<true, 4>(acc, h);
        store_t<4>(A.h[1], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.fw.w3, S.fw.b3, lane);
        c_to_a16<true, 4>(acc, h);
        store_t<4>(A.h[2], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.fw.w4, S.fw.b4, lane);
        c_to_a16<true, 4>(acc, h);
        store_t<4>(A.h[3], h, col0, lane);
        float out[2][4];
        layer16<2, 4, kPadHid>(out, h, S.fw.w5, S.fw.b5, lane);

        float dy[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = col0 + g + (e >> 1) * 8, c = nt * 8 + 2 * t + (e & 1);
                float d = 0.0f;
                if (c < kUsedOut && S.rows.y[r][kUsedOut] != 0.0f) d = out[nt][e] - S.rows.y[r][c];
                lsum += d * d;
                dy[nt][e] = 2.0f * d;
            }
        uint32_t d5[1][4];
        c_to_a16<false, 1>(dy, d5);
        store_t<1>(A.dz5, d5, col0, lane);
        __syncwarp();  // the warp's stored activations, read back as masks

        layer16<8, 1, kPadIn>(acc, d5, S.bw.w5t, nullptr, lane);
        masked_to_a16<4>(acc, A.h[3], h, col0, lane);
        store_t<4>(A.dz[3], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.bw.w4t, nullptr, lane);
        masked_to_a16<4>(acc, A.h[2], h, col0, lane);
        store_t<4>(A.dz[2], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.bw.w3t, nullptr, lane);
        masked_to_a16<4>(acc, A.h[1], h, col0, lane);
        store_t<4>(A.dz[1], h, col0, lane);
        layer16<8, 4, kPadHid>(acc, h, S.bw.w2t, nullptr, lane);
        masked_to_a16<4>(acc, A.h[0], h, col0, lane);
        store_t<4>(A.dz[0], h, col0, lane);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n"
                         "cp.async.bulk.commit_group;\n" ::"l"(a.acts + tile),
                         "r"((uint32_t)__cvta_generic_to_shared(&A)), "r"((uint32_t)sizeof(TileActs))
                         : "memory");
        }
    }
    put_loss(lsum, S.loss, a.loss_part + blockIdx.x);
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
}

// Weight gradients of the 4 x 64 network, dW = dZ^T H over chunks of 2,048
// samples (16 tiles): block (c, u) computes unit u of chunk c and stores it in
// the chunk's partial gradient, which the optimiser sums.  Units: 64 rows x 32
// columns of dW2, dW3, dW4 (two each), dW1, dW5.  Four warps take 16 rows each
// (dW5: 16 columns each) and run the chunk's samples through their
// accumulators in one chain of 128 products, 16 samples at a time, with the
// next step's fragments loaded ahead; bias gradients are the row sums of the
// same dZ fragments.  A fifth warp brings the tiles' rows by bulk copies,
// kWgradStages tiles ahead.
//
// Bound by the latency of that chain: the chain's length is what rounds the
// sums, so it is not split further, and finer units only shorten each step.
// Six stages also keep a second block off the SM (two blocks of 104 KB shared
// one while others stood idle).  By ncu, a batch of
// 16,384: 192 us with 40 blocks reading global memory, 14.9 us with two
// blocks an SM and no fragments loaded ahead, 9.4 us so.  (Products over
// each 128-sample tile in train_kernel itself, summed by the optimiser, take
// 16 us a step instead of 22, but round differently: 4e-6 of the gradient,
// which a few steps at a high learning rate amplify.)
constexpr uint32_t kChunkTiles = 16;
constexpr uint32_t kWgradStages = 6;
constexpr int kWgradUnits = 8, kWgradWarps = 4, kWgradThreads = 32 * (kWgradWarps + 1);
struct WgradStage {
    __half rows[96][kTilePad];  // dZ rows, then H rows
};
struct WgradSmem {
    alignas(128) WgradStage st[kWgradStages];
    alignas(8) uint64_t full[kWgradStages];   // the stage's copies have arrived
    alignas(8) uint64_t empty[kWgradStages];  // the warps are done with it
};
constexpr size_t kWgradSmem = sizeof(WgradSmem);
static_assert(kWgradSmem <= 227 * 1024 && kWgradSmem > 114 * 1024 && sizeof(WgradStage) % 16 == 0,
              "weight-gradient stages: one block per SM");

struct WgradArgs {
    const TileActs* acts;  // [tiles]
    uint32_t tiles;
    float* part;           // [chunks][parameters]
    uint32_t* err;
};

// Rows of a tile's activations that a unit reads: dZ rows, then H rows.
struct WgradRows {
    uint32_t a, rows_a, b, rows_b;
};

__device__ __forceinline__ float h2sum(uint32_t v) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    return f.x + f.y;
}

// The copying warp (one lane): the unit's rows of every tile of the chunk, a
// stage each, as stages become free.  False when one did not in time.
__device__ __forceinline__ bool wgrad_copy(WgradSmem& S, const TileActs* acts, uint32_t tiles, WgradRows u) {
    const uint32_t full = (uint32_t)__cvta_generic_to_shared(S.full), empty = (uint32_t)__cvta_generic_to_shared(S.empty);
    auto start = [&](uint32_t s, uint32_t k) {
        const char* tile = reinterpret_cast<const char*>(acts + k);
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&S.st[s]), mbar = full + 8u * s;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mbar),
                     "r"((u.rows_a + u.rows_b) * kActRowBytes)
                     : "memory");
        auto copy = [&](uint32_t to, uint32_t row, uint32_t rows) {
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(to),
                "l"(tile + (size_t)row * kActRowBytes), "r"(rows * kActRowBytes), "r"(mbar)
                : "memory");
        };
        copy(dst, u.a, u.rows_a);
        copy(dst + u.rows_a * kActRowBytes, u.b, u.rows_b);
    };
    return feed_ring<kWgradStages>(
        tiles, [&](uint32_t s, uint32_t parity) { return tc::mbar_wait(empty + 8u * s, parity); }, start,
        [&](uint32_t s, uint32_t parity) { return tc::mbar_wait(full + 8u * s, parity); });
}

// One warp's 16 x (8 NT) products over the chunk's tiles; a_row, b_row: its
// first rows in a stage; BIAS: also the row sums of A.  False when a tile did
// not arrive in time.
template <int NT, bool BIAS>
__device__ __forceinline__ bool wgrad_chain(WgradSmem& S, uint32_t tiles, int a_row, int b_row, float acc[4][4],
                                            float& s0, float& s1, int lane) {
    const int mat = lane >> 3, r = lane & 7;
    const uint32_t full = (uint32_t)__cvta_generic_to_shared(S.full), empty = (uint32_t)__cvta_generic_to_shared(S.empty);
    for (uint32_t k = 0; k < tiles; ++k) {
        const uint32_t s = k % kWgradStages;
        if (!__all_sync(0xffffffffu, tc::mbar_wait(full + 8u * s, (k / kWgradStages) & 1u))) return false;
        const __half* pa = &S.st[s].rows[a_row + r + (mat & 1) * 8][(mat >> 1) * 8];
        const __half* pb = &S.st[s].rows[b_row + (mat >> 1) * 8 + r][(mat & 1) * 8];
        uint32_t af[2][4], b[2][NT / 2][4];
        auto load = [&](int buf, int c) {
            ldsm_x4(af[buf], pa + c);
#pragma unroll
            for (int q = 0; q < NT / 2; ++q) ldsm_x4(b[buf][q], pb + q * 16 * kTilePad + c);
        };
        load(0, 0);
#pragma unroll
        for (int i = 0; i < kTrainTile / 16; ++i) {
            const int cur = i & 1;
            if (i + 1 < kTrainTile / 16) load(cur ^ 1, 16 * (i + 1));
#pragma unroll
            for (int q = 0; q < NT / 2; ++q) {
                mma(acc[2 * q], af[cur], b[cur][q][0], b[cur][q][1]);
                mma(acc[2 * q + 1], af[cur], b[cur][q][2], b[cur][q][3]);
            }
            if (BIAS) {
                s0 += h2sum(af[cur][0]) + h2sum(af[cur][2]);
                s1 += h2sum(af[cur][1]) + h2sum(af[cur][3]);
            }
        }
        __syncwarp();
        if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(empty + 8u * s) : "memory");
    }
    return true;
}

__global__ void __launch_bounds__(kWgradThreads, 1) wgrad_kernel(const WgradArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    WgradSmem& S = *reinterpret_cast<WgradSmem*>(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t chunk = blockIdx.x, unit = blockIdx.y;
    if (threadIdx.x == 0) {
        for (uint32_t k = 0; k < kWgradStages; ++k) {
            tc::mbar_init((uint32_t)__cvta_generic_to_shared(&S.full[k]), 1);
            tc::mbar_init((uint32_t)__cvta_generic_to_shared(&S.empty[k]), kWgradWarps);
        }
        tc::fence_mbar_init();
    }
    __syncthreads();
    wait_for_previous_kernel();
    const TileActs* acts = a.acts + (size_t)chunk * kChunkTiles;
    const uint32_t tiles = min(kChunkTiles, a.tiles - chunk * kChunkTiles);
    float* part = a.part + (size_t)chunk * kParams;
    // units 0..5: dW4, dW3, dW2 = dz[l] h[l - 1]^T, 32 columns each; 6: dW1; 7: dW5
    const int l = unit < 6u ? 3 - (int)(unit >> 1) : 0, half = (int)(unit & 1u);
    const WgradRows rows = unit < 6u    ? WgradRows{kActRowDz + l * kHid, kHid, kActRowH + (l - 1) * kHid + 32 * half, 32}
                           : unit == 6u ? WgradRows{kActRowDz, kHid, 0, kIn}
                                        : WgradRows{kActRowDz5, kOut, kActRowH + 3 * kHid, kHid};
    if (warp == kWgradWarps) {
        if (lane == 0 && !wgrad_copy(S, acts, tiles, rows)) atomicOr(a.err, tc::kErrTimeout);
        return;
    }
    float acc[4][4] = {}, s0 = 0.0f, s1 = 0.0f;
    bool ok;
    float *gw, *gb = nullptr;
    int m0 = 16 * warp, n0 = 0, ncols = kHid, ntiles = 4;
    if (unit < 6u) {
        ok = half ? wgrad_chain<4, false>(S, tiles, m0, kHid, acc, s0, s1, lane)
                  : wgrad_chain<4, true>(S, tiles, m0, kHid, acc, s0, s1, lane);
        gw = part + (l == 3 ? kW4 : l == 2 ? kW3 : kW2);
        if (!half) gb = part + (l == 3 ? kB4 : l == 2 ? kB3 : kB2);
        n0 = 32 * half;
    } else if (unit == 6u) {
        ntiles = 2;
        ok = wgrad_chain<2, true>(S, tiles, m0, kHid, acc, s0, s1, lane);
        gw = part + kW1;
        gb = part + kB1;
        ncols = kIn;
    } else {  // 16 columns a warp
        ntiles = 2;
        ok = wgrad_chain<2, true>(S, tiles, 0, kOut + 16 * warp, acc, s0, s1, lane);
        gw = part + kW5;
        if (warp == 0) gb = part + kB5;
        m0 = 0;
        n0 = 16 * warp;
    }
    if (!ok) {
        if (lane == 0) atomicOr(a.err, tc::kErrTimeout);
        return;
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        if (nt >= ntiles) break;
        float* p = gw + (m0 + g) * ncols + n0 + nt * 8 + 2 * t;
        *reinterpret_cast<float2*>(p) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(p + 8 * ncols) = make_float2(acc[nt][2], acc[nt][3]);
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (gb && t == 0) {
        gb[m0 + g] = s0;
        gb[m0 + g + 8] = s1;
    }
}

// Training of the compact network on the tensor cores (mma.sync m16n8k16,
// FP16 operands, FP32 accumulation).  A warp takes 16 samples at a time:
//  forward   the inference network's products, keeping the FP16 activations
//            and the ReLU masks;
//  backward  dY = 2 (y - target) for the three BSDF channels, then
//            dZ2 = (dY W3) . [Z2 > 0] and dZ1 = (dZ2 W2) . [Z1 > 0], each a
//            product with a transposed weight matrix held in shared memory;
//  gradients dW = dZ^T A over the block's 128 samples, with the activations
//            and deltas transposed to [unit][sample] in shared memory so the
//            sample dimension is the MMAs' K and the warps share the output
//            tiles; bias gradients are products with ones.
// The deltas enter the MMAs rounded to FP16 (the usual mixed-precision
// backward).  Partial gradients go to the block's own slice with plain stores
// and the optimiser sums the slices, so nothing is zeroed, no atomics contend
// and the result does not depend on the blocks' order.  The loss is the sum over samples and the three channels of
// (y - target)^2; the targets are formed from the twelve lobes of
// hg_mlp_samples (mlps::bsdf_target).
//
// Bound by latency (a batch of 16,384 is one tile per block, on 128 blocks).
// A step of 16,384 samples: 25.5 us with shared and global atomics, a loss
// copy and a memset; 16.6 us with partial gradients and four warps of 32
// samples; 8.7 us so.
struct SmallTrainSmem {
    alignas(16) mlps::Weights w;                       // forward weights (padded rows) and biases
    alignas(16) __half w3t[mlps::kHid][mlps::kPadIn];  // W3^T: [hidden][output]
    alignas(16) __half w2t[mlps::kHid][mlps::kPadHid]; // W2^T: [hidden 1][hidden 2]
    // [unit][sample]
    alignas(16) __half x[mlps::kIn][kTilePad];
    __half a1[mlps::kHid][kTilePad];
    __half a2[mlps::kHid][kTilePad];
    __half dy[mlps::kOut][kTilePad];
    __half dz2[mlps::kHid][kTilePad];
    __half dz1[mlps::kHid][kTilePad];
    TileRows rows;
    float loss[kTrainWarps];
};
static_assert(offsetof(SmallTrainSmem, w) % 16 == 0 && offsetof(SmallTrainSmem, w3t) % 16 == 0 &&
                  offsetof(SmallTrainSmem, w2t) % 16 == 0 && offsetof(SmallTrainSmem, x) % 16 == 0,
              "ldmatrix operands on 16-byte boundaries");
static_assert(offsetof(mlps::Weights, w2) % 16 == 0 && offsetof(mlps::Weights, w3) % 16 == 0, "weight rows");
static_assert((mlps::kPadIn * 2) % 16 == 0 && (mlps::kPadHid * 2) % 16 == 0, "padded weight rows");
constexpr size_t kSmallTrainSmem = sizeof(SmallTrainSmem);

// C fragments of a 32-wide layer, zeroed where `mask` (bit nt*4 + e) is clear
// -> A fragments.
__device__ __forceinline__ void masked_to_a(const float acc[4][4], uint32_t mask, uint32_t a[2][4]) {
    float v[4][4];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[nt][e] = (mask >> (nt * 4 + e)) & 1u ? acc[nt][e] : 0.0f;
    c_to_a16<false, 2>(v, a);
}

__device__ __forceinline__ uint32_t positive_mask(const float acc[4][4]) {
    uint32_t m = 0;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) m |= (acc[nt][e] > 0.0f ? 1u : 0u) << (nt * 4 + e);
    return m;
}

// max(x, 0) fused into the FP16 conversion, as the inference path does it.
__device__ __forceinline__ void relu_to_a16(const float acc[4][4], uint32_t a[2][4]) {
#pragma unroll
    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float* c = acc[2 * kt + h];
            a[kt][2 * h] = pack_relu(c[0], c[1]);
            a[kt][2 * h + 1] = pack_relu(c[2], c[3]);
        }
}

__global__ void __launch_bounds__(kTrainThreads) small_train_kernel(const TrainArgs a) {
    extern __shared__ __align__(16) unsigned char smem_small[];
    SmallTrainSmem& S = *reinterpret_cast<SmallTrainSmem*>(smem_small);
    const int tid = threadIdx.x, nth = kTrainThreads;
    wait_for_previous_kernel();
    copy_rows_async<mlps::kPadIn>(S.w.w1, a.w16 + mlps::kW1, mlps::kHid, mlps::kIn, tid, nth);
    copy_rows_async<mlps::kPadHid>(S.w.w2, a.w16 + mlps::kW2, mlps::kHid, mlps::kHid, tid, nth);
    copy_rows_async<mlps::kPadHid>(S.w.w3, a.w16 + mlps::kW3, mlps::kOut, mlps::kHid, tid, nth);
    for (int i = tid; i < mlps::kHid; i += nth) {
        S.w.b1[i] = a.params[mlps::kB1 + i];
        S.w.b2[i] = a.params[mlps::kB2 + i];
        if (i < mlps::kOut) S.w.b3[i] = a.params[mlps::kB3 + i];
    }
    for (int i = tid; i < mlps::kHid * mlps::kOut; i += nth) {
        const int j = i / mlps::kOut, o = i % mlps::kOut;  // W3^T[j][o] = W3[o][j]
        S.w3t[j][o] = a.w16[mlps::kW3 + o * mlps::kHid + j];
    }
    for (int i = tid; i < mlps::kHid * mlps::kHid; i += nth) {
        const int j1 = i / mlps::kHid, j2 = i % mlps::kHid;  // W2^T[j1][j2] = W2[j2][j1]
        S.w2t[j1][j2] = a.w16[mlps::kW2 + j2 * mlps::kHid + j1];
    }
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int col0 = 16 * warp;
    float* part = a.part + (size_t)blockIdx.x * mlps::kParams;
    float lsum = 0.0f;
    const uint32_t tiles = a.n / kTrainTile + (a.n % kTrainTile != 0u);
    bool add = false;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        wait_copies();  // the weights, before the first tile's barrier
        load_tile(S.rows, a, tile * kTrainTile);
        // the three BSDF targets, one row per thread of the first half (read
        // behind the barrier after the forward pass)
        if (tid < kTrainTile) {
            float y[mlps::kUsedOut];
#pragma unroll
            for (int o = 0; o < mlps::kUsedOut; ++o) y[o] = mlps::bsdf_target(S.rows.y[tid], o);
#pragma unroll
            for (int o = 0; o < mlps::kUsedOut; ++o) S.rows.y[tid][o] = y[o];
        }
        // forward (the inference roundings: FP16 inputs, weights and activations)
        uint32_t a0[1][4], a1[2][4], a2[2][4];
        input_frags16(S.rows, a0, col0, g, t);
        store_t<1>(S.x, a0, col0, lane);
        float acc[4][4];
        layer16<4, 1, mlps::kPadIn>(acc, a0, S.w.w1, S.w.b1, lane);
        const uint32_t mask1 = positive_mask(acc);
        relu_to_a16(acc, a1);
        store_t<2>(S.a1, a1, col0, lane);
        layer16<4, 2, mlps::kPadHid>(acc, a1, S.w.w2, S.w.b2, lane);
        const uint32_t mask2 = positive_mask(acc);
        relu_to_a16(acc, a2);
        store_t<2>(S.a2, a2, col0, lane);
        float out[2][4];
        layer16<2, 2, mlps::kPadHid>(out, a2, S.w.w3, S.w.b3, lane);
        __syncthreads();  // the targets
        // dY as the next product's A operand
        float dy[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = col0 + g + (e >> 1) * 8, c = nt * 8 + 2 * t + (e & 1);
                float d = 0.0f;
                if (c < mlps::kUsedOut && S.rows.y[r][kUsedOut] != 0.0f) d = out[nt][e] - S.rows.y[r][c];
                lsum += d * d;
                dy[nt][e] = 2.0f * d;
            }
        uint32_t ady[1][4], dz2[2][4], dz1[2][4];
        c_to_a16<false, 1>(dy, ady);
        store_t<1>(S.dy, ady, col0, lane);
        // backward through the layers
        layer16<4, 1, mlps::kPadIn>(acc, ady, S.w3t, nullptr, lane);  // dY W3
        masked_to_a(acc, mask2, dz2);
        store_t<2>(S.dz2, dz2, col0, lane);
        layer16<4, 2, mlps::kPadHid>(acc, dz2, S.w2t, nullptr, lane);  // dZ2 W2
        masked_to_a(acc, mask1, dz1);
        store_t<2>(S.dz1, dz1, col0, lane);
        __syncthreads();
        // warp w: 8 columns of 16 rows of dW2; then dW1 (warps 0..3) and dW3 (warps 4..7)
        wgrad_tile(S.dz2, S.a1, 16 * (warp >> 2), 8 * (warp & 3), part + mlps::kW2, mlps::kHid,
                      (warp & 3) ? nullptr : part + mlps::kB2, add, lane);
        if (warp < 4)
            wgrad_tile(S.dz1, S.x, 16 * (warp >> 1), 8 * (warp & 1), part + mlps::kW1, mlps::kIn,
                          (warp & 1) ? part + mlps::kB1 : nullptr, add, lane);
        else
            wgrad_tile(S.dy, S.a2, 0, 8 * (warp - 4), part + mlps::kW3, mlps::kHid,
                          warp == 5 ? part + mlps::kB3 : nullptr, add, lane);
        add = true;
        __syncthreads();  // the next tile overwrites what the products read
    }
    put_loss(lsum, S.loss, a.loss_part + blockIdx.x);
}

struct AdamArgs {
    float* params;
    float* m;
    float* v;
    float* grad;
    __half* w16;
    __half* wt16;
    const float* part;       // [parts][parameters] partial gradients, or null (conversion only)
    const float* loss_part;  // [blocks]
    uint32_t parts, blocks;
    float* loss;             // the batch's sum of squared errors, nullable
    const uint32_t* err;     // the context's error word
    volatile uint32_t* skipped;  // hg_ctx's, in host memory
    float lr_t, beta1, beta2, eps_t, gscale;
    int update;              // 1: Adam step; 0: the summed gradient into grad, parameters as they are
};

constexpr int kAdamParams = 32, kAdamSplit = 16;  // parameters per block, threads that share one's slices

// The sum of the partial gradients, then Adam (Kingma and Ba 2015)
// with the bias corrections folded into lr_t and eps_t, then the FP16 forward
// (and, for the 4 x 64 network, transposed) copies.  Sixteen threads share a
// parameter's partials, so that each has its loads in flight at once, and add
// up in a fixed order.  While the context has a timeout to report, a partial
// gradient may be missing: nothing is summed into the parameters then, their
// moments or grad, and the host is told.
template <int N, bool TRANSPOSED>
__global__ void __launch_bounds__(kAdamParams* kAdamSplit) adam_kernel(const AdamArgs a) {
    __shared__ float s_sum[kAdamSplit][kAdamParams];
    const int q = threadIdx.x % kAdamParams, split = threadIdx.x / kAdamParams;
    const int i = blockIdx.x * kAdamParams + q;
    wait_for_previous_kernel();
    const bool own = split == 0 && i < N;
    float p = 0.0f, m = 0.0f, v = 0.0f, gr = 0.0f;
    uint32_t err = 0u;
    if (own) {
        if (a.part) err = __ldcg(a.err);
        p = a.params[i];
        if (a.update) {
            m = a.m[i];
            v = a.v[i];
        }
    }
    if (a.part && i < N) {
#pragma unroll 8
        for (uint32_t b = split; b < a.parts; b += kAdamSplit) gr += __ldcg(&a.part[(size_t)b * N + i]);
    }
    s_sum[split][q] = gr;
    if (a.loss && blockIdx.x == 0 && split == 1) {
        float l = 0.0f;
        for (uint32_t b = q; b < a.blocks; b += kAdamParams) l += __ldcg(&a.loss_part[b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (q == 0) *a.loss = l;
    }
    __syncthreads();
    if (!own) return;
    if (err & tc::kErrTimeout) {
        *a.skipped = 1u;
        return;
    }
    gr = 0.0f;
#pragma unroll
    for (int s = 0; s < kAdamSplit; ++s) gr += s_sum[s][q];
    if (a.part && !a.update) {
        a.grad[i] = gr;
        return;
    }
    if (a.update) {
        gr *= a.gscale;
        m = a.beta1 * m + (1.0f - a.beta1) * gr;
        v = a.beta2 * v + (1.0f - a.beta2) * gr * gr;
        a.m[i] = m;
        a.v[i] = v;
        p -= a.lr_t * m / (sqrtf(v) + a.eps_t);
        a.params[i] = p;
    }
    const __half hp = __float2half_rn(p);
    a.w16[i] = hp;
    if (!TRANSPOSED) return;
    int tofs = -1, rows = 0, cols = kHid, rel = 0;
    if (i >= kW2 && i < kB2) tofs = kT2, rows = kHid, rel = i - kW2;
    else if (i >= kW3 && i < kB3) tofs = kT3, rows = kHid, rel = i - kW3;
    else if (i >= kW4 && i < kB4) tofs = kT4, rows = kHid, rel = i - kW4;
    else if (i >= kW5 && i < kB5) tofs = kT5, rows = kOut, rel = i - kW5;
    if (tofs >= 0) {
        const int r = rel / cols, c = rel - r * cols;
        a.wt16[tofs + c * rows + r] = hp;
    }
}

// ------------------------------------------------------------ host side

constexpr size_t kFwdSmem = sizeof(FwdWeights) + kWarps * sizeof(WarpIo);
constexpr size_t kTrainSmem = sizeof(TrainSmem);

std::mutex g_init_mutex;
bool g_gl_ready[64] = {};
bool g_attr_ready[64] = {};
static_assert(tc::kSmemBytes <= 227 * 1024, "tcgen05 kernel shared memory");

// Gauss-Legendre nodes by Newton iteration on P_64, mapped to gamma_i in
// [-pi/2, pi/2] with the Jacobian cos(gamma_i) folded into the weights.
void gauss_legendre(double* x, double* w) {
    const int n = kGl;
    for (int i = 0; i < n; ++i) {
        double z = std::cos(kPiD * (i + 0.75) / (n + 0.5));
        double dp = 1.0;
        for (int it = 0; it < 100; ++it) {
            double p0 = 1.0, p1 = z;
            for (int k = 2; k <= n; ++k) {
                const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (z * p1 - p0) / (z * z - 1.0);
            const double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        double p0 = 1.0, p1 = z;
        for (int k = 2; k <= n; ++k) {
            const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
            p0 = p1;
            p1 = p2;
        }
        dp = n * (z * p1 - p0) / (z * z - 1.0);
        x[i] = 0.5 * kPiD * z;
        w[i] = 0.5 * kPiD * 2.0 / ((1.0 - z * z) * dp * dp) * std::cos(x[i]);
    }
}

cudaError_t ensure_device_setup(int device) {
    std::lock_guard<std::mutex> lock(g_init_mutex);
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    cudaError_t e = cudaSuccess;
    if (!g_gl_ready[device]) {
        double x[kGl], w[kGl], s[kPairs], c[kPairs];
        gauss_legendre(x, w);  // descending: the first half are the positive nodes
        for (int i = 0; i < kPairs; ++i) {
            s[i] = std::sin(x[i]);
            c[i] = std::cos(x[i]);
        }
        e = cudaMemcpyToSymbol(c_gl_x, x, sizeof(s));
        if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_gl_w, w, sizeof(s));
        if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_gl_sin, s, sizeof(s));
        if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_gl_cos, c, sizeof(c));
        if (e != cudaSuccess) return e;
        g_gl_ready[device] = true;
    }
    if (!g_attr_ready[device]) {
        e = cudaFuncSetAttribute(infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgradSmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(infer_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)tc::kSmemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(small_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kSmallTrainSmem);
        if (e != cudaSuccess) return e;
        g_attr_ready[device] = true;
    }
    return cudaSuccess;
}

hg_status fail(hg_ctx* ctx, hg_status s, const char* msg) {
    if (ctx) ctx->last_error = msg;
    return s;
}

hg_status cuda_fail(hg_ctx* ctx, cudaError_t e, const char* where) {
    if (ctx) ctx->last_error = std::string(where) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? HG_OUT_OF_MEMORY : HG_CUDA_ERROR;
}

#define MLP_CUDA(ctx, expr)                                     \
    do {                                                        \
        cudaError_t e_ = (expr);                                \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, #expr); \
    } while (0)

// For calls that have waited for the stream.  (A word in host memory that a
// kernel sets only then: a copy of the error word with each of them takes 3.5 us.)
hg_status unless_skipped(hg_ctx* ctx) {
    if (!*ctx->skipped) return HG_OK;
    return fail(ctx, HG_DEVICE_TIMEOUT, "a tensor-core wait timed out; no training step since has been taken");
}

// Most blocks a training launch uses: one (the 4 x 64 network, whose tile
// fills an SM's shared memory) or two per SM.
uint32_t max_train_blocks(const hg_mlp* m) {
    return (uint32_t)m->ctx->sm_count * (m->arch == HG_MLP_ARCH_COMPACT ? 2u : 1u);
}

uint32_t train_tiles(uint32_t n) { return n / kTrainTile + (n % kTrainTile != 0u); }

uint32_t train_blocks(const hg_mlp* m, uint32_t n) { return std::min(train_tiles(n), max_train_blocks(m)); }

// Partial gradients of a batch of n: one per chunk of tiles (4 x 64) or per block.
uint32_t train_parts(const hg_mlp* m, uint32_t n) {
    if (m->arch == HG_MLP_ARCH_COMPACT) return train_blocks(m, n);
    return (train_tiles(n) + kChunkTiles - 1) / kChunkTiles;
}

// 4 x 64: the tiles' activations and the chunks' partial gradients, grown to n
// samples (the compact network's partials are allocated with it).
cudaError_t ensure_scratch(hg_mlp* m, uint32_t n) {
    const uint32_t tiles = train_tiles(n);
    if (m->arch == HG_MLP_ARCH_COMPACT || tiles <= m->tile_capacity) return cudaSuccess;
    cudaStreamSynchronize(m->ctx->stream);
    if (m->acts) cudaFree(m->acts);
    m->acts = nullptr;
    m->part = nullptr;
    m->tile_capacity = 0;
    const size_t acts = sizeof(TileActs) * (size_t)tiles;
    cudaError_t e = cudaMalloc(&m->acts, acts + sizeof(float) * (size_t)m->n_params * train_parts(m, n));
    if (e != cudaSuccess) return e;
    m->part = reinterpret_cast<float*>(static_cast<char*>(m->acts) + acts);
    m->tile_capacity = tiles;
    return cudaSuccess;
}

// A launch that may be placed while the stream's previous kernel finishes
// (see wait_for_previous_kernel).
template <class Args>
cudaError_t launch_dependent(void (*kernel)(const Args), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                             const Args& args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

// The FP16 copies of the parameters; after a training launch of n > 0 samples,
// first the sum of its partial gradients and either an Adam step (update) or
// the sum into m->grad.
cudaError_t convert(hg_mlp* m, uint32_t n, int update, float lr_t, float eps_t, float gscale, float* loss) {
    AdamArgs a;
    a.params = m->params;
    a.m = m->adam_m;
    a.v = m->adam_v;
    a.grad = m->grad;
    a.w16 = reinterpret_cast<__half*>(m->w16);
    a.wt16 = reinterpret_cast<__half*>(m->wt16);
    a.part = n ? m->part : nullptr;
    a.loss_part = m->loss_part;
    a.parts = n ? train_parts(m, n) : 0u;
    a.blocks = n ? train_blocks(m, n) : 0u;
    a.loss = n ? loss : nullptr;
    a.err = m->ctx->err;
    a.skipped = m->ctx->skipped;
    a.lr_t = lr_t;
    a.beta1 = 0.9f;
    a.beta2 = 0.999f;
    a.eps_t = eps_t;
    a.gscale = gscale;
    a.update = update;
    const uint32_t grid = (m->n_params + kAdamParams - 1) / kAdamParams;
    const int threads = kAdamParams * kAdamSplit;
    return m->arch == HG_MLP_ARCH_COMPACT
               ? launch_dependent(adam_kernel<mlps::kParams, false>, dim3(grid), threads, 0, m->ctx->stream, a)
               : launch_dependent(adam_kernel<kParams, true>, dim3(grid), threads, 0, m->ctx->stream, a);
}

// Forward, backward and weight gradients of n samples into m->part (sized by
// ensure_scratch): train_parts(m, n) partial gradients, train_blocks(m, n)
// losses.
cudaError_t run_gradients(hg_mlp* m, const float* inputs, const float* targets, uint32_t n) {
    TrainArgs a;
    a.inputs = inputs;
    a.targets = targets;
    a.n = n;
    a.w16 = reinterpret_cast<const __half*>(m->w16);
    a.wt16 = reinterpret_cast<const __half*>(m->wt16);
    a.params = m->params;
    a.acts = static_cast<TileActs*>(m->acts);
    a.part = m->part;
    a.loss_part = m->loss_part;
    const cudaStream_t st = m->ctx->stream;
    const uint32_t blocks = train_blocks(m, n);
    if (m->arch == HG_MLP_ARCH_COMPACT)
        return launch_dependent(small_train_kernel, dim3(blocks), kTrainThreads, kSmallTrainSmem, st, a);
    cudaError_t e = launch_dependent(train_kernel, dim3(blocks), kTrainThreads, kTrainSmem, st, a);
    if (e != cudaSuccess) return e;
    WgradArgs w;
    w.acts = a.acts;
    w.tiles = train_tiles(n);
    w.part = m->part;
    w.err = m->ctx->err;
    return launch_dependent(wgrad_kernel, dim3(train_parts(m, n), kWgradUnits), kWgradThreads, kWgradSmem, st, w);
}

}  // namespace

cudaError_t launch_mlp_infer_tc(hg_mlp* m, const float* inputs, uint32_t n, float* lobes, float* net) {
    InferArgs a;
    a.inputs = inputs;
    a.n = n;
    a.w16 = reinterpret_cast<const __half*>(m->w16);
    a.params = m->params;
    a.lobes = lobes;
    a.net = net;
    const uint32_t chunks = n / tc::kM + (n % tc::kM != 0u);
    uint32_t blocks = (chunks + tc::kChains - 1) / tc::kChains;
    // one CTA per SM: it holds all 512 TMEM columns
    const uint32_t cap = (uint32_t)m->ctx->sm_count;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    infer_tc_kernel<<<blocks, tc::kThreads, tc::kSmemBytes, m->ctx->stream>>>(a, m->ctx->err);
    return cudaGetLastError();
}

cudaError_t launch_mlp_infer(hg_mlp* m, const float* inputs, uint32_t n, float* lobes, float* net) {
    InferArgs a;
    a.inputs = inputs;
    a.n = n;
    a.w16 = reinterpret_cast<const __half*>(m->w16);
    a.params = m->params;
    a.lobes = lobes;
    a.net = net;
    const uint32_t warps = (n + 31u) / 32u;
    uint32_t blocks = (warps + kWarps - 1) / kWarps;
    if (m->arch == HG_MLP_ARCH_COMPACT) {
        const uint32_t cap = (uint32_t)m->ctx->sm_count * 8u;
        if (blocks > cap) blocks = cap;
        infer_small_kernel<<<blocks, kWarps * 32, 0, m->ctx->stream>>>(a);
        return cudaGetLastError();
    }
    const uint32_t cap = (uint32_t)m->ctx->sm_count * 3u;
    if (blocks > cap) blocks = cap;
    infer_kernel<<<blocks, kWarps * 32, kFwdSmem, m->ctx->stream>>>(a);
    return cudaGetLastError();
}

}  // namespace hg

using hg::cuda_fail;
using hg::fail;

extern "C" {

hg_status hg_mlp_create(hg_ctx* ctx, hg_mlp** out) { return hg_mlp_create_arch(ctx, HG_MLP_ARCH_DEEP, out); }

hg_status hg_mlp_create_arch(hg_ctx* ctx, uint32_t arch, hg_mlp** out) {
    if (!ctx || !out) return HG_INVALID_ARG;
    *out = nullptr;
    if (arch != HG_MLP_ARCH_DEEP && arch != HG_MLP_ARCH_COMPACT)
        return fail(ctx, HG_INVALID_ARG, "unknown surrogate architecture");
    cudaSetDevice(ctx->device);
    MLP_CUDA(ctx, hg::ensure_device_setup(ctx->device));
    hg_mlp* m = new (std::nothrow) hg_mlp();
    if (!m) return fail(ctx, HG_OUT_OF_MEMORY, "allocating the surrogate");
    m->ctx = ctx;
    m->arch = arch;
    m->n_params = arch == HG_MLP_ARCH_COMPACT ? (uint32_t)hg::mlps::kParams : (uint32_t)hg::mlp::kParams;
    // one allocation, each array on a 256-byte boundary
    size_t bytes = 0;
    auto place = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255u) & ~(size_t)255u;
        return at;
    };
    const size_t pf = sizeof(float) * m->n_params;
    const size_t at_params = place(pf), at_m = place(pf), at_v = place(pf), zeroed = bytes, at_grad = place(pf),
                 at_w16 = place(sizeof(__half) * m->n_params),
                 at_wt16 = place(arch == HG_MLP_ARCH_DEEP ? sizeof(__half) * hg::mlp::kTransposed : 0),
                 at_loss = place(sizeof(float)),
                 at_loss_part = place(sizeof(float) * hg::max_train_blocks(m)),
                 at_part = place(arch == HG_MLP_ARCH_COMPACT ? pf * hg::max_train_blocks(m) : 0);
    cudaError_t e = cudaMalloc(&m->arena, bytes);
    if (e == cudaSuccess) {
        char* base = static_cast<char*>(m->arena);
        m->params = reinterpret_cast<float*>(base + at_params);
        m->adam_m = reinterpret_cast<float*>(base + at_m);
        m->adam_v = reinterpret_cast<float*>(base + at_v);
        m->grad = reinterpret_cast<float*>(base + at_grad);
        m->w16 = base + at_w16;
        m->wt16 = arch == HG_MLP_ARCH_DEEP ? base + at_wt16 : nullptr;
        m->loss = reinterpret_cast<float*>(base + at_loss);
        m->loss_part = reinterpret_cast<float*>(base + at_loss_part);
        m->part = arch == HG_MLP_ARCH_COMPACT ? reinterpret_cast<float*>(base + at_part) : nullptr;
        e = cudaMemsetAsync(m->arena, 0, zeroed, ctx->stream);
    }
    if (e == cudaSuccess) e = hg::convert(m, 0, 0, 0.0f, 0.0f, 0.0f, nullptr);
    if (e != cudaSuccess) {
        hg_mlp_destroy(m);
        return cuda_fail(ctx, e, "creating the surrogate");
    }
    *out = m;
    return HG_OK;
}

void hg_mlp_destroy(hg_mlp* m) {
    if (!m) return;
    hg_ctx* ctx = m->ctx;
    if (ctx) {
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
        if (ctx->surrogate == m) ctx->surrogate = nullptr;
    }
    if (m->arena) cudaFree(m->arena);
    if (m->acts) cudaFree(m->acts);
    delete m;
}

uint32_t hg_mlp_param_count(const hg_mlp* m) { return m ? m->n_params : 0u; }

uint32_t hg_mlp_output_count(const hg_mlp* m) {
    if (!m) return 0u;
    return m->arch == HG_MLP_ARCH_COMPACT ? (uint32_t)hg::mlps::kUsedOut : (uint32_t)hg::mlp::kUsedOut;
}

hg_status hg_mlp_set_params(hg_mlp* m, const float* params, uint32_t count) {
    if (!m || !params) return HG_INVALID_ARG;
    hg_ctx* ctx = m->ctx;
    if (count != m->n_params) return fail(ctx, HG_INVALID_ARG, "parameter count must be hg_mlp_param_count");
    for (uint32_t i = 0; i < count; ++i)
        if (!std::isfinite(params[i])) return fail(ctx, HG_INVALID_ARG, "non-finite parameter");
    const size_t pf = sizeof(float) * count;
    MLP_CUDA(ctx, cudaMemcpyAsync(m->params, params, pf, cudaMemcpyHostToDevice, ctx->stream));
    MLP_CUDA(ctx, cudaMemsetAsync(m->adam_m, 0, pf, ctx->stream));
    MLP_CUDA(ctx, cudaMemsetAsync(m->adam_v, 0, pf, ctx->stream));
    MLP_CUDA(ctx, hg::convert(m, 0, 0, 0.0f, 0.0f, 0.0f, nullptr));
    MLP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    m->step = 0;
    return HG_OK;
}

hg_status hg_mlp_get_params(hg_mlp* m, float* params, uint32_t count) {
    if (!m || !params) return HG_INVALID_ARG;
    hg_ctx* ctx = m->ctx;
    if (count != m->n_params) return fail(ctx, HG_INVALID_ARG, "parameter count must be hg_mlp_param_count");
    MLP_CUDA(ctx, cudaMemcpyAsync(params, m->params, sizeof(float) * count, cudaMemcpyDeviceToHost, ctx->stream));
    MLP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return hg::unless_skipped(ctx);
}

hg_status hg_mlp_samples(hg_ctx* ctx, uint64_t seed, uint64_t first, uint32_t count, float tilt, float* inputs,
                         float* targets, double* lobes) {
    if (!ctx) return HG_INVALID_ARG;
    if (count == 0) return HG_OK;
    if (!inputs) return fail(ctx, HG_INVALID_ARG, "null inputs buffer");
    if (!std::isfinite(tilt)) return fail(ctx, HG_INVALID_ARG, "non-finite tilt");
    cudaSetDevice(ctx->device);
    MLP_CUDA(ctx, cudaPeekAtLastError());  // an earlier error is reported, not cleared
    MLP_CUDA(ctx, hg::ensure_device_setup(ctx->device));
    hg::SampleArgs a;
    a.seed = seed;
    a.first = first;
    a.n = count;
    a.tilt = (double)tilt;
    a.inputs = inputs;
    a.targets = targets;
    a.lobes = lobes;
    // As many lanes share a sample's 32 nodes as leave at most one 128-thread
    // block per SM: the FP64 pipe is then still one warp deep everywhere.  The
    // lanes repeat the work outside the nodes, so more of them than that lose
    // (19,000 samples on 152 SMs: 0.98 ms with one lane, 1.61 ms with eight;
    // 1,000 samples: 0.98 and 0.20 ms).
    const uint64_t room = (uint64_t)ctx->sm_count * hg::kSampleThreads;
    const uint32_t lanes = (uint64_t)count * 8u <= room ? 8u : (uint64_t)count * 4u <= room ? 4u
                           : (uint64_t)count * 2u <= room ? 2u : 1u;
    const uint32_t per = hg::kSampleThreads / lanes;
    const uint32_t blocks = count / per + (count % per != 0u);
    if (lanes == 8u) hg::samples_kernel<8><<<blocks, hg::kSampleThreads, 0, ctx->stream>>>(a);
    else if (lanes == 4u) hg::samples_kernel<4><<<blocks, hg::kSampleThreads, 0, ctx->stream>>>(a);
    else if (lanes == 2u) hg::samples_kernel<2><<<blocks, hg::kSampleThreads, 0, ctx->stream>>>(a);
    else hg::samples_kernel<1><<<blocks, hg::kSampleThreads, 0, ctx->stream>>>(a);
    MLP_CUDA(ctx, cudaGetLastError());
    return HG_OK;
}

hg_status hg_mlp_infer(hg_mlp* m, const float* inputs, uint32_t count, float* lobes, float* net) {
    if (!m) return HG_INVALID_ARG;
    if (count == 0) return HG_OK;
    if (!inputs || (!lobes && !net)) return fail(m->ctx, HG_INVALID_ARG, "null buffer");
    MLP_CUDA(m->ctx, cudaPeekAtLastError());
    MLP_CUDA(m->ctx, hg::launch_mlp_infer(m, inputs, count, lobes, net));
    return HG_OK;
}

hg_status hg_mlp_infer_tc(hg_mlp* m, const float* inputs, uint32_t count, float* lobes, float* net) {
    if (!m) return HG_INVALID_ARG;
    if (m->arch != HG_MLP_ARCH_DEEP) return fail(m->ctx, HG_INVALID_ARG, "tcgen05 inference runs the 4 x 64 network");
    if (count == 0) return HG_OK;
    if (!inputs || (!lobes && !net)) return fail(m->ctx, HG_INVALID_ARG, "null buffer");
    MLP_CUDA(m->ctx, cudaPeekAtLastError());
    MLP_CUDA(m->ctx, hg::launch_mlp_infer_tc(m, inputs, count, lobes, net));
    return HG_OK;
}

hg_status hg_mlp_gradients(hg_mlp* m, const float* inputs, const float* targets, uint32_t count, float* grad,
                           float* loss) {
    if (!m) return HG_INVALID_ARG;
    hg_ctx* ctx = m->ctx;
    if (count == 0 || !inputs || !targets || !grad) return fail(ctx, HG_INVALID_ARG, "empty batch or null buffer");
    MLP_CUDA(ctx, cudaPeekAtLastError());
    const size_t pf = sizeof(float) * m->n_params;
    MLP_CUDA(ctx, hg::ensure_scratch(m, count));
    MLP_CUDA(ctx, hg::run_gradients(m, inputs, targets, count));
    MLP_CUDA(ctx, hg::convert(m, count, 0, 0.0f, 0.0f, 0.0f, m->loss));
    MLP_CUDA(ctx, cudaMemcpyAsync(grad, m->grad, pf, cudaMemcpyDeviceToHost, ctx->stream));
    float l = 0.0f;
    MLP_CUDA(ctx, cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    MLP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (loss) *loss = l;
    return hg::unless_skipped(ctx);
}

hg_status hg_mlp_train_step(hg_mlp* m, const float* inputs, const float* targets, uint32_t count, float lr,
                            float* loss_sum) {
    if (!m) return HG_INVALID_ARG;
    hg_ctx* ctx = m->ctx;
    if (count == 0 || !inputs || !targets) return fail(ctx, HG_INVALID_ARG, "empty batch or null buffer");
    if (!(lr >= 0.0f) || !std::isfinite(lr)) return fail(ctx, HG_INVALID_ARG, "learning rate must be finite, >= 0");
    MLP_CUDA(ctx, cudaPeekAtLastError());
    MLP_CUDA(ctx, hg::ensure_scratch(m, count));
    MLP_CUDA(ctx, hg::run_gradients(m, inputs, targets, count));
    m->step += 1;
    const double b1t = 1.0 - std::pow(0.9, (double)m->step), b2t = 1.0 - std::pow(0.999, (double)m->step);
    const float lr_t = (float)(lr * std::sqrt(b2t) / b1t);
    const float eps_t = (float)(1e-8 * std::sqrt(b2t));
    // the kernel stores a float; any other address takes a copy
    const bool aligned = reinterpret_cast<uintptr_t>(loss_sum) % sizeof(float) == 0;
    MLP_CUDA(ctx, hg::convert(m, count, 1, lr_t, eps_t,
                              1.0f / ((float)count * (float)hg_mlp_output_count(m)), aligned ? loss_sum : m->loss));
    if (!aligned)
        MLP_CUDA(ctx, cudaMemcpyAsync(loss_sum, m->loss, sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
    return HG_OK;
}

hg_status hg_karis_lobes(hg_ctx* ctx, const float* inputs, uint32_t count, float tilt, float* lobes) {
    if (!ctx) return HG_INVALID_ARG;
    if (count == 0) return HG_OK;
    if (!inputs || !lobes) return fail(ctx, HG_INVALID_ARG, "null buffer");
    if (!std::isfinite(tilt)) return fail(ctx, HG_INVALID_ARG, "non-finite tilt");
    cudaSetDevice(ctx->device);
    MLP_CUDA(ctx, cudaPeekAtLastError());
    MLP_CUDA(ctx, hg::launch_karis_lobes(ctx, inputs, count, tilt, lobes));
    return HG_OK;
}

hg_status hg_mlp_bind(hg_ctx* ctx, hg_mlp* m) {
    if (!ctx) return HG_INVALID_ARG;
    if (m && m->ctx != ctx) return fail(ctx, HG_INVALID_ARG, "surrogate belongs to another context");
    ctx->surrogate = m;
    return HG_OK;
}

}  // extern "C"
