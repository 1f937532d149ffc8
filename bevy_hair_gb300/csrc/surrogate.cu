// Learned shading surrogate: FP64 training samples of the hair lobes, the
// FP16 tensor-core networks' inference and training kernels (4 x 64 and compact
// 2 x 32: forward, backward and weight gradients of a 128-sample tile per
// block on mma.sync, partial gradients summed by the Adam kernel), and their
// C entry points.  The reference has no counterpart; the shading it replaces is the
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
        if (valid) {
#pragma unroll
            for (int c = 0; c < 12; ++c) {
                if (a.lobes) a.lobes[(size_t)i * 12 + c] = decode(y[c]);
                if (a.net) a.net[(size_t)i * 12 + c] = y[c];
            }
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
        if (valid) {
#pragma unroll
            for (int c = 0; c < mlps::kUsedOut; ++c) {
                if (a.lobes) a.lobes[(size_t)i * mlps::kUsedOut + c] = decode(y[c]);
                if (a.net) a.net[(size_t)i * mlps::kUsedOut + c] = y[c];
            }
        }
    }
}

// The same evaluation on tcgen05: four chains of two 128-row evaluations per CTA.
__global__ void __launch_bounds__(tc::kThreads, 1) infer_tc_kernel(const InferArgs a, uint32_t* err) {
    extern __shared__ __align__(128) uint8_t smem_tc[];
    tc::Chain c = tc::setup(smem_tc, a.w16, a.params);
    const uint32_t g = threadIdx.x >> 7;
    const uint32_t chunks = (a.n + tc::kM - 1) / tc::kM;
    const uint32_t pairs = (chunks + 1) / 2;
    bool failed = false;
    for (uint32_t pc = blockIdx.x * tc::kChains + g; pc < pairs; pc += gridDim.x * tc::kChains) {
        const bool two = 2 * pc + 1 < chunks;
        uint32_t idx[2];
        bool valid[2];
        for (uint32_t e = 0; e < 2; ++e) {
            idx[e] = (2 * pc + e) * tc::kM + c.row;
            valid[e] = idx[e] < a.n && (e == 0 || two);
            float raw[10], x[10];
            load_raw(a.inputs, idx[e], valid[e], raw);
            normalise(raw, x);
            tc::write_input_row(c, e, x);
        }
        float y[2][12];
        if (!tc::forward2(c, two, y[0], y[1])) {
            failed = true;
            break;
        }
        for (uint32_t e = 0; e < 2; ++e) {
            if (!valid[e]) continue;
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                if (a.lobes) a.lobes[(size_t)idx[e] * 12 + k] = decode(y[e][k]);
                if (a.net) a.net[(size_t)idx[e] * 12 + k] = y[e][k];
            }
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

constexpr int kTrainWarps = 4;
constexpr int kTrainTile = 32 * kTrainWarps;  // samples a block takes at a time, 32 per warp
constexpr int kTilePad = kTrainTile + 8;      // halves per transposed row (conflict-free ldmatrix and stmatrix)

// Packed A fragments (KT k-tiles of 16 units, rows = the warp's 32 samples)
// into dst[unit][col0 + sample].  Fragment register r covers units
// (r >> 1) * 8.. and samples (r & 1) * 8.., so one transposing stmatrix stores
// a 16 x 16 block.
template <int KT>
__device__ __forceinline__ void store_t(__half (*dst)[kTilePad], const uint32_t a[2][KT][4], int col0, int lane) {
    const int r = lane >> 3, i = lane & 7;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
            stsm_x4_trans(&dst[kt * 16 + (r >> 1) * 8 + i][col0 + mt * 16 + (r & 1) * 8], a[mt][kt]);
}

__device__ __forceinline__ void apply_mask(float acc[2][8][4], uint64_t m) {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (!((m >> ((mt * 8 + nt) * 4 + e)) & 1ull)) acc[mt][nt][e] = 0.0f;
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

// Rows m0..m0+15, columns n0..n0+8*NT-1 of dW = A B^T over a tile's samples
// (A = dZ^T, B = H^T, both [unit][sample] in shared memory) into the block's
// partial gradient gw (row length n_cols); with gb, also the row sums of A
// (the bias gradient), as a product with ones.  One warp.
template <int NT>
__device__ __forceinline__ void wgrad_tile(const __half (*A)[kTilePad], const __half (*B)[kTilePad], int m0, int n0,
                                           float* gw, int n_cols, float* gb, bool add, int lane) {
    const int g = lane >> 2, t = lane & 3, mat = lane >> 3, r = lane & 7;
    float acc[NT][4] = {}, sum[4] = {};
#pragma unroll
    for (int k = 0; k < kTrainTile; k += 16) {
        uint32_t af[4];
        ldsm_x4(af, &A[m0 + r + (mat & 1) * 8][k + (mat >> 1) * 8]);
        if (gb) mma(sum, af, 0x3C003C00u, 0x3C003C00u);
#pragma unroll
        for (int nt = 0; nt + 1 < NT; nt += 2) {
            uint32_t b[4];
            ldsm_x4(b, &B[n0 + (nt + (mat >> 1)) * 8 + r][k + (mat & 1) * 8]);
            mma(acc[nt], af, b[0], b[1]);
            mma(acc[nt + 1], af, b[2], b[3]);
        }
        if (NT & 1) {
            uint32_t b[2];
            ldsm_x2(b, &B[n0 + (NT - 1) * 8 + r][k + (mat & 1) * 8]);
            mma(acc[NT - 1], af, b[0], b[1]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        float* p = gw + (m0 + g) * n_cols + n0 + nt * 8 + 2 * t;
        put2(p, acc[nt][0], acc[nt][1], add);
        put2(p + 8 * n_cols, acc[nt][2], acc[nt][3], add);
    }
    if (gb && t == 0) {
        gb[m0 + g] = sum[0] + (add ? gb[m0 + g] : 0.0f);
        gb[m0 + g + 8] = sum[2] + (add ? gb[m0 + g + 8] : 0.0f);
    }
}

struct TrainArgs {
    const float* inputs;   // [n][10]
    const float* targets;  // [n][12] transformed
    uint32_t n;
    const __half* w16;
    const __half* wt16;    // transposed copies (4 x 64 network only)
    const float* params;
    float* part;  // [blocks][parameters] partial gradients, written whole
    float* loss_part;  // [blocks] partial sums of squared errors
};

struct TrainSmem {
    FwdWeights fw;
    BwdWeights bw;
    __half x[kIn][kTilePad];          // layer-1 inputs, [unit][sample]
    __half h[4][kHid][kTilePad];      // hidden activations h1..h4
    __half dz[4][kHid][kTilePad];     // pre-activation gradients of layers 1..4
    __half dz5[kOut][kTilePad];       // output gradients
    WarpIo io[kTrainWarps];
    float loss[kTrainWarps];
};
static_assert(sizeof(FwdWeights) % 16 == 0 && sizeof(BwdWeights) % 16 == 0 && (kTilePad * 2) % 16 == 0 &&
                  offsetof(TrainSmem, x) % 16 == 0 && offsetof(TrainSmem, io) % 16 == 0,
              "ldmatrix rows on 16-byte boundaries");
static_assert(sizeof(TrainSmem) <= 227 * 1024, "train kernel shared memory");

// One training batch: forward, backward and weight gradients of 128-sample
// tiles, everything between the batch's rows and the block's partial gradient
// in registers and shared memory.  Each warp runs 32 samples forward and
// backward on mma.sync and leaves its activations and deltas transposed in
// shared memory; then the block's warps share the weight-gradient products
// over the tile's 128 samples (warp w takes 16 rows of each dW).  Partial
// gradients go to the block's own slice with plain stores and the optimiser
// sums the slices, so nothing is zeroed, no atomics contend and the result
// does not depend on the blocks' order.  The loss is the sum over samples and
// the 12 outputs of (y - target)^2, so dL/dy = 2 (y - target); the 1/(n*12)
// of the mean is applied by the optimiser.
//
// Bound by latency and shared-memory traffic: at a batch of 16,384 an SM holds
// one tile.  Before, the activations went through memory (17 MB) to a second
// kernel whose 40 blocks summed dW serially: 157 us a step of 16,384 samples;
// 23.4 us now (152 SMs).
__global__ void __launch_bounds__(kTrainTile, 1) train_kernel(const TrainArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    load_fwd(S.fw, a.w16, a.params, threadIdx.x, blockDim.x);
    load_bwd(S.bw, a.wt16, threadIdx.x, blockDim.x);
    __syncthreads();
    WarpIo& w_io = S.io[warp];
    const int col0 = 32 * warp;
    float* part = a.part + (size_t)blockIdx.x * kParams;
    float lsum = 0.0f;
    bool add = false;
    for (uint32_t base = blockIdx.x * kTrainTile; base < a.n; base += gridDim.x * kTrainTile) {
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < a.n;
        // the targets are read up front: they are needed only after the forward pass
        float tgt[kUsedOut];
#pragma unroll
        for (int c = 0; c < kUsedOut; ++c) tgt[c] = valid ? __ldg(&a.targets[(size_t)i * 12 + c]) : 0.0f;
        float raw[10], x[10];
        load_raw(a.inputs, i, valid, raw);
        normalise(raw, x);
        uint32_t a0[2][1][4];
        input_frags(w_io, x, a0, lane, g, t);
        store_t<1>(S.x, a0, col0, lane);

        float acc[2][8][4];
        uint32_t h[2][4][4];
        uint64_t m1, m2, m3, m4;
        layer_ldsm<8, 1, kPadIn>(acc, a0, S.fw.w1, S.fw.b1, lane);
        c_to_a<true>(acc, h);
        m1 = relu_mask(h);
        store_t<4>(S.h[0], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.fw.w2, S.fw.b2, lane);
        c_to_a<true>(acc, h);
        m2 = relu_mask(h);
        store_t<4>(S.h[1], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.fw.w3, S.fw.b3, lane);
        c_to_a<true>(acc, h);
        m3 = relu_mask(h);
        store_t<4>(S.h[2], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.fw.w4, S.fw.b4, lane);
        c_to_a<true>(acc, h);
        m4 = relu_mask(h);
        store_t<4>(S.h[3], h, col0, lane);
        float out[2][2][4];
        layer_ldsm<2, 4, kPadHid>(out, h, S.fw.w5, S.fw.b5, lane);

        // Targets into the C layout through the warp's output stage; column 16
        // flags a real sample.
#pragma unroll
        for (int c = 0; c < kUsedOut; ++c) w_io.y[lane][c] = tgt[c];
        w_io.y[lane][16] = valid ? 1.0f : 0.0f;
        __syncwarp();
        uint32_t d5[2][1][4];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            float dy[2][4];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = mt * 16 + g + ((e >> 1) ? 8 : 0), c = nt * 8 + 2 * t + (e & 1);
                    float d = 0.0f;
                    if (c < kUsedOut && w_io.y[r][16] != 0.0f) d = out[mt][nt][e] - w_io.y[r][c];
                    lsum += d * d;
                    dy[nt][e] = 2.0f * d;
                }
            d5[mt][0][0] = pack_h2(dy[0][0], dy[0][1]);
            d5[mt][0][1] = pack_h2(dy[0][2], dy[0][3]);
            d5[mt][0][2] = pack_h2(dy[1][0], dy[1][1]);
            d5[mt][0][3] = pack_h2(dy[1][2], dy[1][3]);
        }
        __syncwarp();
        store_t<1>(S.dz5, d5, col0, lane);

        layer_ldsm<8, 1, kPadIn>(acc, d5, S.bw.w5t, nullptr, lane);
        apply_mask(acc, m4);
        c_to_a<false>(acc, h);
        store_t<4>(S.dz[3], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.bw.w4t, nullptr, lane);
        apply_mask(acc, m3);
        c_to_a<false>(acc, h);
        store_t<4>(S.dz[2], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.bw.w3t, nullptr, lane);
        apply_mask(acc, m2);
        c_to_a<false>(acc, h);
        store_t<4>(S.dz[1], h, col0, lane);
        layer_ldsm<8, 4, kPadHid>(acc, h, S.bw.w2t, nullptr, lane);
        apply_mask(acc, m1);
        c_to_a<false>(acc, h);
        store_t<4>(S.dz[0], h, col0, lane);
        __syncthreads();

        wgrad_tile<8>(S.dz[3], S.h[2], 16 * warp, 0, part + kW4, kHid, part + kB4, add, lane);
        wgrad_tile<8>(S.dz[2], S.h[1], 16 * warp, 0, part + kW3, kHid, part + kB3, add, lane);
        wgrad_tile<8>(S.dz[1], S.h[0], 16 * warp, 0, part + kW2, kHid, part + kB2, add, lane);
        wgrad_tile<2>(S.dz[0], S.x, 16 * warp, 0, part + kW1, kIn, part + kB1, add, lane);
        wgrad_tile<2>(S.dz5, S.h[3], 0, 16 * warp, part + kW5, kHid, warp == 0 ? part + kB5 : nullptr, add, lane);
        add = true;
        __syncthreads();  // the next tile overwrites what the products read
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) S.loss[warp] = lsum;
    __syncthreads();
    if (threadIdx.x == 0) a.loss_part[blockIdx.x] = (S.loss[0] + S.loss[1]) + (S.loss[2] + S.loss[3]);
}

// Training of the compact network on the tensor cores (mma.sync m16n8k16,
// FP16 operands, FP32 accumulation).  A warp takes 32 samples at a time:
//  forward   the inference network itself (mlps::forward's layers), keeping
//            the FP16 activations and the ReLU masks;
//  backward  dY = 2 (y - target) for the three BSDF channels, then
//            dZ2 = (dY W3) . [Z2 > 0] and dZ1 = (dZ2 W2) . [Z1 > 0], each a
//            product with a transposed weight matrix held in shared memory;
//  gradients dW = dZ^T A over the block's 128 samples, with the activations
//            and deltas transposed to [unit][sample] in shared memory so the
//            sample dimension is the MMAs' K and the warps share the output
//            tiles; bias gradients are products with ones.
// The deltas enter the MMAs rounded to FP16 (the usual mixed-precision
// backward).  Partial gradients go to the block's own slice, as in
// train_kernel.  The loss is the sum over samples and the three channels of
// (y - target)^2; the targets are formed from the twelve lobes of
// hg_mlp_samples (mlps::bsdf_target).
//
// Bound by latency (a batch of 16,384 is one tile per block, on 128 blocks).
// Before, each warp added its 2,128 sums to shared memory and each block to
// global memory by atomics, with a loss copy and a memset after every step:
// 25.5 us a step of 16,384 samples; SMALL_23.4 us now.
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
    alignas(16) mlp::WarpIo io[kTrainWarps];
    float loss[kTrainWarps];
};
static_assert(offsetof(SmallTrainSmem, w) % 16 == 0 && offsetof(SmallTrainSmem, w3t) % 16 == 0 &&
                  offsetof(SmallTrainSmem, w2t) % 16 == 0 && offsetof(SmallTrainSmem, x) % 16 == 0 &&
                  offsetof(SmallTrainSmem, io) % 16 == 0,
              "ldmatrix operands on 16-byte boundaries");
static_assert(offsetof(mlps::Weights, w2) % 16 == 0 && offsetof(mlps::Weights, w3) % 16 == 0, "weight rows");
static_assert((mlps::kPadIn * 2) % 16 == 0 && (mlps::kPadHid * 2) % 16 == 0, "padded weight rows");
constexpr size_t kSmallTrainSmem = sizeof(SmallTrainSmem);

// C fragments of a 32-wide layer times a 32-bit mask (bit (mt*4 + nt)*4 + e)
// -> FP16 A fragments.
__device__ __forceinline__ void masked_to_a(const float acc[2][4][4], uint32_t mask, uint32_t a[2][2][4]) {
    auto m = [&](int mt, int nt, int e) { return (mask >> ((mt * 4 + nt) * 4 + e)) & 1u ? acc[mt][nt][e] : 0.0f; };
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
            a[mt][kt][0] = mlp::pack_h2(m(mt, 2 * kt, 0), m(mt, 2 * kt, 1));
            a[mt][kt][1] = mlp::pack_h2(m(mt, 2 * kt, 2), m(mt, 2 * kt, 3));
            a[mt][kt][2] = mlp::pack_h2(m(mt, 2 * kt + 1, 0), m(mt, 2 * kt + 1, 1));
            a[mt][kt][3] = mlp::pack_h2(m(mt, 2 * kt + 1, 2), m(mt, 2 * kt + 1, 3));
        }
}

__device__ __forceinline__ uint32_t positive_mask(const float acc[2][4][4]) {
    uint32_t m = 0;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) m |= (acc[mt][nt][e] > 0.0f ? 1u : 0u) << ((mt * 4 + nt) * 4 + e);
    return m;
}

__global__ void __launch_bounds__(kTrainTile) small_train_kernel(const TrainArgs a) {
    extern __shared__ __align__(16) unsigned char smem_small[];
    SmallTrainSmem& S = *reinterpret_cast<SmallTrainSmem*>(smem_small);
    const int tid = threadIdx.x, nth = blockDim.x;
    mlps::load(S.w, a.w16, a.params, tid, nth);
    for (int i = tid; i < mlps::kHid * mlps::kOut; i += nth) {
        const int j = i / mlps::kOut, o = i % mlps::kOut;  // W3^T[j][o] = W3[o][j]
        S.w3t[j][o] = a.w16[mlps::kW3 + o * mlps::kHid + j];
    }
    for (int i = tid; i < mlps::kHid * mlps::kHid; i += nth) {
        const int j1 = i / mlps::kHid, j2 = i % mlps::kHid;  // W2^T[j1][j2] = W2[j2][j1]
        S.w2t[j1][j2] = a.w16[mlps::kW2 + j2 * mlps::kHid + j1];
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    mlp::WarpIo& io = S.io[warp];
    const int col0 = 32 * warp;
    float* part = a.part + (size_t)blockIdx.x * mlps::kParams;
    float loss = 0.0f;
    bool add = false;
    for (uint32_t base = blockIdx.x * kTrainTile; base < a.n; base += gridDim.x * kTrainTile) {
        const uint32_t k = base + tid;
        const bool valid = k < a.n;
        // the targets are read up front: they are needed only after the forward pass
        float t12[12];
#pragma unroll
        for (int c = 0; c < 12; ++c) t12[c] = valid ? __ldg(&a.targets[(size_t)k * 12 + c]) : 0.0f;
        float raw[10], xn[10];
        load_raw(a.inputs, k, valid, raw);
        normalise(raw, xn);
        // forward (the inference roundings: FP16 inputs, weights and activations)
        uint32_t a0[2][1][4];
        mlp::input_frags(io, xn, a0, lane, g, t);
        float acc[2][4][4];
        uint32_t a1[2][2][4], a2[2][2][4];
        mlp::layer_ldsm<4, 1, mlps::kPadIn>(acc, a0, S.w.w1, S.w.b1, lane);
        const uint32_t mask1 = positive_mask(acc);
        mlps::relu_to_a(acc, a1);
        mlp::layer_ldsm<4, 2, mlps::kPadHid>(acc, a1, S.w.w2, S.w.b2, lane);
        const uint32_t mask2 = positive_mask(acc);
        mlps::relu_to_a(acc, a2);
        float out[2][2][4];
        mlp::layer_ldsm<2, 2, mlps::kPadHid>(out, a2, S.w.w3, S.w.b3, lane);
        float y[mlp::kUsedOut];  // output_rows fills 12 columns; the first mlps::kUsedOut are outputs
        mlp::output_rows(io, out, y, lane, g, t);
        store_t<1>(S.x, a0, col0, lane);
        store_t<2>(S.a1, a1, col0, lane);
        store_t<2>(S.a2, a2, col0, lane);
        // dY of this lane's sample, as the next product's A operand
        float dyx[mlp::kUsedIn] = {};
#pragma unroll
        for (int o = 0; o < mlps::kUsedOut; ++o) {
            const float d = valid ? y[o] - mlps::bsdf_target(t12, o) : 0.0f;
            loss += d * d;
            dyx[o] = 2.0f * d;
        }
        uint32_t ady[2][1][4];
        mlp::input_frags(io, dyx, ady, lane, g, t);
        // backward through the layers
        mlp::layer_ldsm<4, 1, mlps::kPadIn>(acc, ady, S.w3t, nullptr, lane);  // dY W3
        uint32_t dz2[2][2][4], dz1[2][2][4];
        masked_to_a(acc, mask2, dz2);
        mlp::layer_ldsm<4, 2, mlps::kPadHid>(acc, dz2, S.w2t, nullptr, lane);  // dZ2 W2
        masked_to_a(acc, mask1, dz1);
        store_t<1>(S.dy, ady, col0, lane);
        store_t<2>(S.dz2, dz2, col0, lane);
        store_t<2>(S.dz1, dz1, col0, lane);
        __syncthreads();
        // warp w: rows 16 (w / 2).. and half the columns of dW2, dW1; 8 columns of dW3
        const int m0 = 16 * (warp >> 1), half = warp & 1;
        wgrad_tile<2>(S.dz2, S.a1, m0, 16 * half, part + mlps::kW2, mlps::kHid, half ? nullptr : part + mlps::kB2, add,
                      lane);
        wgrad_tile<1>(S.dz1, S.x, m0, 8 * half, part + mlps::kW1, mlps::kIn, half ? part + mlps::kB1 : nullptr, add,
                      lane);
        wgrad_tile<1>(S.dy, S.a2, 0, 8 * warp, part + mlps::kW3, mlps::kHid, warp == 0 ? part + mlps::kB3 : nullptr,
                      add, lane);
        add = true;
        __syncthreads();  // the next tile overwrites what the products read
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
    if (lane == 0) S.loss[warp] = loss;
    __syncthreads();
    if (tid == 0) a.loss_part[blockIdx.x] = (S.loss[0] + S.loss[1]) + (S.loss[2] + S.loss[3]);
}

struct AdamArgs {
    float* params;
    float* m;
    float* v;
    float* grad;
    __half* w16;
    __half* wt16;
    const float* part;       // [blocks][parameters] partial gradients, or null (conversion only)
    const float* loss_part;  // [blocks]
    uint32_t blocks;
    float* loss;             // the batch's sum of squared errors, nullable
    float lr_t, beta1, beta2, eps_t, gscale;
    int update;              // 1: Adam step; 0: the summed gradient into grad, parameters as they are
};

constexpr int kAdamParams = 64, kAdamSplit = 4;  // parameters per block, threads that share one's slices

// The sum over the blocks' partial gradients, then Adam (Kingma and Ba 2015)
// with the bias corrections folded into lr_t and eps_t, then the FP16 forward
// (and, for the 4 x 64 network, transposed) copies.  Four threads share a
// parameter's slices (7.5 MB for 128 blocks of the 4 x 64 network, in L2) and
// add up in a fixed order.
template <int N, bool TRANSPOSED>
__global__ void __launch_bounds__(kAdamParams* kAdamSplit) adam_kernel(const AdamArgs a) {
    __shared__ float s_sum[kAdamSplit][kAdamParams];
    const int q = threadIdx.x % kAdamParams, split = threadIdx.x / kAdamParams;
    const int i = blockIdx.x * kAdamParams + q;
    float gr = 0.0f;
    if (a.part && i < N) {
#pragma unroll 8
        for (uint32_t b = split; b < a.blocks; b += kAdamSplit) gr += __ldcg(&a.part[(size_t)b * N + i]);
    }
    s_sum[split][q] = gr;
    if (a.loss && blockIdx.x == 0 && threadIdx.x < 32) {
        float l = 0.0f;
        for (uint32_t b = threadIdx.x; b < a.blocks; b += 32) l += __ldcg(&a.loss_part[b]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (threadIdx.x == 0) *a.loss = l;
    }
    __syncthreads();
    if (split != 0 || i >= N) return;
    gr = (s_sum[0][q] + s_sum[1][q]) + (s_sum[2][q] + s_sum[3][q]);
    if (a.part && !a.update) {
        a.grad[i] = gr;
        return;
    }
    float p = a.params[i];
    if (a.update) {
        gr *= a.gscale;
        const float m = a.beta1 * a.m[i] + (1.0f - a.beta1) * gr;
        const float v = a.beta2 * a.v[i] + (1.0f - a.beta2) * gr * gr;
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

// Most blocks a training launch uses: one (the 4 x 64 network, whose tile
// fills an SM's shared memory) or two per SM; a block with several tiles adds
// them up in its slice.
uint32_t max_train_blocks(const hg_mlp* m) {
    return (uint32_t)m->ctx->sm_count * (m->arch == HG_MLP_ARCH_COMPACT ? 2u : 1u);
}

uint32_t train_blocks(const hg_mlp* m, uint32_t n) {
    return std::min(n / kTrainTile + (n % kTrainTile != 0u), max_train_blocks(m));
}

// The FP16 copies of the parameters; with `blocks` partial gradients (and
// losses) in m->part, first their sum and either an Adam step (update) or
// the summed gradient into m->grad.
cudaError_t convert(hg_mlp* m, uint32_t blocks, int update, float lr_t, float eps_t, float gscale, float* loss) {
    AdamArgs a;
    a.params = m->params;
    a.m = m->adam_m;
    a.v = m->adam_v;
    a.grad = m->grad;
    a.w16 = reinterpret_cast<__half*>(m->w16);
    a.wt16 = reinterpret_cast<__half*>(m->wt16);
    a.part = blocks ? m->part : nullptr;
    a.loss_part = m->part + (size_t)max_train_blocks(m) * m->n_params;
    a.blocks = blocks;
    a.loss = blocks ? loss : nullptr;
    a.lr_t = lr_t;
    a.beta1 = 0.9f;
    a.beta2 = 0.999f;
    a.eps_t = eps_t;
    a.gscale = gscale;
    a.update = update;
    const uint32_t grid = (m->n_params + kAdamParams - 1) / kAdamParams;
    const int threads = kAdamParams * kAdamSplit;
    if (m->arch == HG_MLP_ARCH_COMPACT)
        adam_kernel<mlps::kParams, false><<<grid, threads, 0, m->ctx->stream>>>(a);
    else
        adam_kernel<kParams, true><<<grid, threads, 0, m->ctx->stream>>>(a);
    return cudaGetLastError();
}

// Forward, backward and weight gradients of n samples into m->part:
// train_blocks(m, n) partial gradients and losses.
cudaError_t run_gradients(hg_mlp* m, const float* inputs, const float* targets, uint32_t n) {
    TrainArgs a;
    a.inputs = inputs;
    a.targets = targets;
    a.n = n;
    a.w16 = reinterpret_cast<const __half*>(m->w16);
    a.wt16 = reinterpret_cast<const __half*>(m->wt16);
    a.params = m->params;
    a.part = m->part;
    a.loss_part = m->part + (size_t)max_train_blocks(m) * m->n_params;
    const uint32_t blocks = train_blocks(m, n);
    if (m->arch == HG_MLP_ARCH_COMPACT)
        small_train_kernel<<<blocks, kTrainTile, kSmallTrainSmem, m->ctx->stream>>>(a);
    else
        train_kernel<<<blocks, kTrainTile, kTrainSmem, m->ctx->stream>>>(a);
    return cudaGetLastError();
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
    const uint32_t pairs = ((n + tc::kM - 1) / tc::kM + 1) / 2;
    uint32_t blocks = (pairs + tc::kChains - 1) / tc::kChains;
    // one CTA per SM: it holds all 512 TMEM columns and most of the shared memory
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
    const size_t pf = sizeof(float) * m->n_params;
    cudaError_t e = cudaMalloc(&m->params, pf);
    if (e == cudaSuccess) e = cudaMalloc(&m->grad, pf);
    if (e == cudaSuccess) e = cudaMalloc(&m->adam_m, pf);
    if (e == cudaSuccess) e = cudaMalloc(&m->adam_v, pf);
    if (e == cudaSuccess) e = cudaMalloc(&m->w16, sizeof(__half) * m->n_params);
    if (e == cudaSuccess && arch == HG_MLP_ARCH_DEEP)
        e = cudaMalloc(&m->wt16, sizeof(__half) * hg::mlp::kTransposed);
    if (e == cudaSuccess) e = cudaMalloc(&m->loss, sizeof(float));
    if (e == cudaSuccess)
        e = cudaMalloc(&m->part, sizeof(float) * (size_t)hg::max_train_blocks(m) * (m->n_params + 1u));
    for (void* p : {(void*)m->params, (void*)m->adam_m, (void*)m->adam_v})
        if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, pf, ctx->stream);
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
    for (void* p : {(void*)m->params, (void*)m->grad, (void*)m->adam_m, (void*)m->adam_v, (void*)m->w16,
                    (void*)m->wt16, (void*)m->loss, (void*)m->part})
        if (p) cudaFree(p);
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
    return HG_OK;
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
    // A lane per sample while that gives every SM a block; below, eight lanes
    // share a sample's 32 nodes (1,000 samples: 0.98 ms with one lane, 0.20 ms
    // with eight).
    if (count >= (uint32_t)ctx->sm_count * hg::kSampleThreads) {
        const uint32_t blocks = (count + hg::kSampleThreads - 1u) / hg::kSampleThreads;
        hg::samples_kernel<1><<<blocks, hg::kSampleThreads, 0, ctx->stream>>>(a);
    } else {
        const uint32_t per = hg::kSampleThreads / 8u;
        hg::samples_kernel<8><<<(count + per - 1u) / per, hg::kSampleThreads, 0, ctx->stream>>>(a);
    }
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
    MLP_CUDA(ctx, hg::run_gradients(m, inputs, targets, count));
    MLP_CUDA(ctx, hg::convert(m, hg::train_blocks(m, count), 0, 0.0f, 0.0f, 0.0f, m->loss));
    MLP_CUDA(ctx, cudaMemcpyAsync(grad, m->grad, pf, cudaMemcpyDeviceToHost, ctx->stream));
    float l = 0.0f;
    MLP_CUDA(ctx, cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    MLP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (loss) *loss = l;
    return HG_OK;
}

hg_status hg_mlp_train_step(hg_mlp* m, const float* inputs, const float* targets, uint32_t count, float lr,
                            float* loss_sum) {
    if (!m) return HG_INVALID_ARG;
    hg_ctx* ctx = m->ctx;
    if (count == 0 || !inputs || !targets) return fail(ctx, HG_INVALID_ARG, "empty batch or null buffer");
    if (!(lr >= 0.0f) || !std::isfinite(lr)) return fail(ctx, HG_INVALID_ARG, "learning rate must be finite, >= 0");
    MLP_CUDA(ctx, cudaPeekAtLastError());
    MLP_CUDA(ctx, hg::run_gradients(m, inputs, targets, count));
    m->step += 1;
    const double b1t = 1.0 - std::pow(0.9, (double)m->step), b2t = 1.0 - std::pow(0.999, (double)m->step);
    const float lr_t = (float)(lr * std::sqrt(b2t) / b1t);
    const float eps_t = (float)(1e-8 * std::sqrt(b2t));
    MLP_CUDA(ctx, hg::convert(m, hg::train_blocks(m, count), 1, lr_t, eps_t,
                              1.0f / ((float)count * (float)hg_mlp_output_count(m)), loss_sum));
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
