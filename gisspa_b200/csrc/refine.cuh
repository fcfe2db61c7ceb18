// Off-grid score of a pick and its gradient (adjoint), batched over picks.
//
// The objective continues the search's score off its grid of angles and
// pixels (no reference counterpart).  For pick p (window w, template J, map
// position x0, in-plane angle e, sub-pixel shift d, CTF theta = (defocus,
// dfdiff, dfang) of the template weight):
//   B   = FFT(b_J) / l^2                 b_J: padded, edge-normalised,
//                                        whitened template (main.cu:182-431);
//                                        kept as its spectrum's half plane
//   F1  = B w(k; theta)                  band-pass x |CTF| Wiener weight
//                                        (GPU_func.cu:249-290)
//   t   = Re IFFT(F1 / a), a = sqrt(sum_sel |F1|^2) / cnt  (main.cu:447-463)
//   tm  = mask . rotate_bilinear(t, e)   (GPU_func.cu:496-560, 229-247)
//   tn  = (tm - mean) / sd               full frame (main.cu:697-710)
//   F   = FFT(tn) / l^2
//   c   = Re sum_k W(k) conj(F(k)) exp(2 pi i k.(x0 + d) / l), k signed
//   sig = sqrt(sum_k |W|^2 |F|^2)        map standard deviation (Parseval)
//   s   = sgn c / sig
// The adjoint runs the same chain backwards; the forward's per-pick buffers (F1, t,
// tm and F) stay in device memory for it, tn is taken from tm again, and B is
// read from the context's half planes.
#pragma once

#include "common.cuh"
#include "kernels.cuh"

namespace gs {

// One pick: inputs of the objective.
struct RefinePickDev {
    int window, tmpl, x0, y0;  // x0, y0: unshifted map position
    float e, dx, dy;           // degrees, pixels
    float defocus, dfdiff, dfang;  // um (positive underfocus), um, degrees
};

// Per-pick accumulators (double sums) and results.
struct RefineAcc {
    double asum;        // sum_sel |F1|^2
    double m1, m2;      // sum tm, sum tm^2
    double c, sig2, cdx, cdy;
    double g1, g2;      // sum gamma, sum gamma tn
    double de;          // d s / d e
    double abar;        // -Re sum Fbar2 conj(F1)
    double dth[3];      // d s / d theta
};

struct RefineConsts {
    int l;
    long long L2;
    float apix, lambda, cs, ampconst, kk, a, b, b2, bf, bf2, bf3, hp, lp, ds;
    float d_m;
    float cnt;  // number of (r < l/2, x <= l/2) bins
};

// What the weight takes of a bin that does not depend on the pick: band-pass
// factor, s^2 and azimuth of the CTF's folded frequency, noise curve over signal
// (negative: bin not selected, the weight is the band-pass factor alone).  One
// table per call, read by every pick.
struct RefineBin {
    float band, ss, ag, ncurve;
};

__device__ __forceinline__ RefineBin refine_bin(int x, int y, const RefineConsts& rc) {
    const int l = rc.l;
    float rf;
    const int r = shell_index(x, y, l, l, &rf);
    const float band = bandpass<false>(r, rc.hp, rc.lp);
    if (!(r < l / 2 && r >= 0)) return RefineBin{band, 0.0f, 0.0f, -1.0f};
    // CTF geometry of ctf_ast(x, (y + l/2) % l)
    int x1 = x, y1 = (y + l / 2) % l;
    y1 = x1 > l / 2 ? l - y1 : y1;
    x1 = min(x1, l - x1);
    const float fx = (float)x1, fy = (float)(y1 - l / 2);
    const float ss = (fx * fx / (float)(l * l) + fy * fy / (float)(l * l)) / (rc.apix * rc.apix);
    const float ssw = rf * rc.ds;
    const float signal = expf(rc.bf * ssw * ssw + rc.bf2 * ssw + rc.bf3) / (rc.kk + 1.0f);
    const float ncurve = expf(rc.a * ssw * ssw + rc.b * ssw + rc.b2) / signal;
    return RefineBin{band, ss, atan2f(fy, fx), ncurve};
}

// Weight w(k; theta) and, with kGrad, its theta derivatives (float; the value
// path is the same arithmetic as k_weight_map).
template <bool kGrad>
__device__ __forceinline__ float refine_weight(const RefineBin& bin, const RefineConsts& rc, const RefinePickDev& pk,
                                               bool* insel, float dw[3]) {
    *insel = !(bin.ncurve < 0.0f);
    if constexpr (kGrad) dw[0] = dw[1] = dw[2] = 0.0f;
    if (!*insel) return bin.band;
    const float ss = bin.ss;
    const float D = -pk.defocus;
    const float dfu = D + pk.dfdiff, dfv = D - pk.dfdiff;
    const float ang2 = (float)(2.0 * ((double)pk.dfang * kPiRef / 180.0 - (double)bin.ag));
    const float cs2 = cosf(ang2);
    const float df_ast = 0.5f * (dfu + dfv + 2.0f * pk.dfdiff * cs2);
    const double lam = (double)rc.lambda;
    const float gamma = (float)(-2.0 * kPiRef *
                                ((double)rc.cs * 2.5e6 * lam * lam * lam * (double)ss * (double)ss +
                                 (double)df_ast * 5000.0 * lam * (double)ss));
    const float sa = sqrtf(1.0f - rc.ampconst * rc.ampconst);
    float sg, cg;
    sincosf(gamma, &sg, &cg);
    const float V = sa * sg + rc.ampconst * cg;
    const float v = fabsf(V);
    const float den = bin.ncurve + rc.kk * v * v;
    const float w = v * sqrtf(1.0f / den);
    if constexpr (kGrad) {
        // d w / d gamma = band * ncurve den^-3/2 * sign(V) (sa cos g - a sin g)
        const float dwdg = bin.band * bin.ncurve / (den * sqrtf(den)) * (V >= 0.0f ? 1.0f : -1.0f) *
                           (sa * cg - rc.ampconst * sg);
        const float dgdf = (float)(-2.0 * kPiRef * 5000.0 * lam * (double)ss);  // d gamma / d df_ast
        dw[0] = dwdg * dgdf * -1.0f;                                            // d df_ast / d defocus = -1
        dw[1] = dwdg * dgdf * cs2;                                              // d df_ast / d dfdiff
        dw[2] = dwdg * dgdf * (-2.0f * pk.dfdiff * sinf(ang2)) * (float)(kPiRef / 180.0);
    }
    return bin.band * w;
}

// Soft mask factor of apply_mask (GPU_func.cu:229-247), the arithmetic of
// k_pair_rotate, and the bins' table.
static __global__ void k_ref_maps(float* __restrict__ mask, RefineBin* __restrict__ bins, RefineConsts rc) {
    const int l = rc.l, q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= l * l) return;
    const int h = l / 2, i = q % l, j = q / l;
    const float dm = 1.5f * rc.d_m;
    const float rin = dm / 2.0f, rout = dm / 2.0f + 12.0f;
    const float r = hypotf((float)(i - h), (float)(j - h));
    float m = 1.0f;
    if (r > rout) m = 0.0f;
    else if (r >= rin) m = (float)(0.5 * (double)cosf((float)(kPiRef * (double)(r - rin) / 12.0)) + 0.5);
    mask[q] = m;
    bins[q] = refine_bin(i, j, rc);
}

// Bin (x, y) of a base spectrum from its half plane.
__device__ __forceinline__ float2 ref_base(const float2* __restrict__ H, int x, int y, int l) {
    const int hw = l / 2 + 1;
    if (x <= l / 2) return __ldg(H + y * hw + x);
    const float2 v = __ldg(H + (y ? l - y : 0) * hw + (l - x));
    return make_float2(v.x, -v.y);
}

// ---- forward ----

// F1 = B w(theta), a second copy of it (transformed in place), and sum_sel |F1|^2
// per pick.  Grid (pixel chunks, picks).
static __global__ void __launch_bounds__(256) k_ref_weight(const float2* __restrict__ base, const RefineBin* __restrict__ bins,
                                                           float2* __restrict__ F1, float2* __restrict__ copy,
                                                           const RefinePickDev* __restrict__ pks, RefineConsts rc,
                                                           RefineAcc* __restrict__ acc) {
    __shared__ double red[32];
    const int p = blockIdx.y;
    const RefinePickDev pk = pks[p];
    const int l = rc.l, npix = l * l;
    const float2* H = base + (long long)pk.tmpl * l * (l / 2 + 1);
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const int y = i / l, x = i - y * l;
        bool insel;
        const float w = refine_weight<false>(bins[i], rc, pk, &insel, nullptr);
        const float2 v = cscale(ref_base(H, x, y, l), w);
        F1[p * rc.L2 + i] = v;
        copy[p * rc.L2 + i] = v;
        if (insel && x <= l / 2) s += (double)v.x * v.x + (double)v.y * v.y;
    }
    double v1[1] = {s};
    block_sum<1>(v1, red);
    if (threadIdx.x == 0) atomicAdd(&acc[p].asum, v1[0]);
}

// Per-pick factors of the transforms: 1 / a for t = Re IFFT(F1 / a), and the pair
// coefficient (IoPairNorm) of a map that is to be taken as it is.
static __global__ void k_ref_factors(const RefineAcc* __restrict__ acc, int n, double cnt, double* __restrict__ inva,
                                     float2* __restrict__ as_is) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    inva[p] = cnt / sqrt(acc[p].asum);
    as_is[p] = make_float2(1.0f, 0.0f);
}

// Source coordinates of rotate_subIMG for output pixel (i, j) and angle e.
__device__ __forceinline__ void rot_src(int i, int j, int l, float c, float s, float* x2, float* y2) {
    const float h = (float)(l / 2);
    const float x = (float)(i - l / 2), y = (float)(j - l / 2);
    *x2 = fmaf(c, x, s * y) + h;
    *y2 = fmaf(-s, x, c * y) + h;
}

// Bilinear sample with the reference's index rules; corner indices and
// weights for the adjoint.
struct Bilin {
    int k[4];
    float w[4];
    float dt, du;  // d value / d (fractional x), d value / d (fractional y) factors
    bool inb;
};

__device__ __forceinline__ Bilin bilin(float x2, float y2, int l) {
    Bilin b;
    b.inb = !(x2 < 0.0f || x2 > (float)(l - 1) || y2 < 0.0f || y2 > (float)(l - 1));
    int ii = (int)floorf(x2), jj = (int)floorf(y2);
    ii = min(max(ii, 0), l - 1);
    jj = min(max(jj, 0), l - 1);
    const float t = x2 - (float)ii, u = y2 - (float)jj;
    int k0 = ii + jj * l, k1 = k0 + 1, k2 = k0 + l + 1, k3 = k0 + l;
    if (ii == l - 1) { k1 -= 1; k2 -= 1; }
    if (jj == l - 1) { k2 -= l; k3 -= l; }
    b.k[0] = k0; b.k[1] = k1; b.k[2] = k2; b.k[3] = k3;
    b.w[0] = (1.0f - t) * (1.0f - u);
    b.w[1] = t * (1.0f - u);
    b.w[2] = t * u;
    b.w[3] = (1.0f - t) * u;
    b.dt = t;
    b.du = u;
    return b;
}

// tm = mask . rotate(t, e) in the rows [row0, row1) that the mask's disc reaches;
// sums of tm and tm^2.
static __global__ void __launch_bounds__(256) k_ref_rotate(const float* __restrict__ T, float* __restrict__ TM,
                                                           const RefinePickDev* __restrict__ pks, RefineConsts rc,
                                                           int row0, int row1,
                                                           const float* __restrict__ mask, RefineAcc* __restrict__ acc) {
    __shared__ double red[64];
    const int p = blockIdx.y;
    const int l = rc.l;
    const double ang = (double)pks[p].e * kPiRef / 180.0;
    const float c = (float)cos(ang), s = (float)sin(ang);
    const float* src = T + p * rc.L2;
    double a2[2] = {0.0, 0.0};
    for (int i = row0 * l + blockIdx.x * blockDim.x + threadIdx.x; i < row1 * l; i += gridDim.x * blockDim.x) {
        const int y = i / l, x = i - y * l;
        const float m = mask[i];
        float v = 0.0f;
        if (m != 0.0f) {
            float x2, y2;
            rot_src(x, y, l, c, s, &x2, &y2);
            const Bilin b = bilin(x2, y2, l);
            if (b.inb) v = src[b.k[0]] * b.w[0] + src[b.k[1]] * b.w[1] + src[b.k[3]] * b.w[3] + src[b.k[2]] * b.w[2];
            v *= m;
        }
        TM[p * rc.L2 + i] = v;
        a2[0] += v;
        a2[1] += (double)v * v;
    }
    block_sum<2>(a2, red);
    if (threadIdx.x == 0) {
        atomicAdd(&acc[p].m1, a2[0]);
        atomicAdd(&acc[p].m2, a2[1]);
    }
}

__device__ __forceinline__ void ref_moments(const RefineAcc& a, double L2, double* mu, double* sd) {
    *mu = a.m1 / L2;
    const double var = a.m2 / L2 - *mu * *mu;
    *sd = sqrt(var > 0.0 ? var : 1.0);
}

// The input of FFT(tn): tm / sd in the rows [row0, row1), rounded once from double
// (the mean only reaches the zero frequency, which is 0).
static __global__ void __launch_bounds__(256) k_ref_norm(const float* __restrict__ TM, RefineConsts rc, int row0, int row1,
                                                         const RefineAcc* __restrict__ acc, float2* __restrict__ F) {
    const int p = blockIdx.y;
    double mu, sd;
    ref_moments(acc[p], (double)rc.L2, &mu, &sd);
    const double inv_sd = 1.0 / sd;
    for (int i = row0 * rc.l + blockIdx.x * blockDim.x + threadIdx.x; i < row1 * rc.l; i += gridDim.x * blockDim.x)
        F[p * rc.L2 + i] = make_float2((float)((double)TM[p * rc.L2 + i] * inv_sd), 0.0f);
}

// Phase factors exp(2 pi i kx (x0 + dx) / l), kx = 0 .. l - 1 (signed), then the
// same of ky, per pick; the integer part of the phase in integer arithmetic.
static __global__ void k_ref_phases(const RefinePickDev* __restrict__ pks, int l, double2* __restrict__ ph) {
    const int p = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * l) return;
    const int k = i < l ? i : i - l;
    const int sk = k < (l + 1) / 2 ? k : k - l;
    const RefinePickDev pk = pks[p];
    long long ip = (long long)sk * (i < l ? pk.x0 : pk.y0) % l;
    if (ip < 0) ip += l;
    const double frac = ((double)ip + (double)sk * (i < l ? pk.dx : pk.dy)) / (double)l;
    double sn, cs;
    sincospi(2.0 * (frac - floor(frac)), &sn, &cs);
    ph[(size_t)p * 2 * l + i] = make_double2(cs, sn);
}
__device__ __forceinline__ float2 ref_phase(const double2* __restrict__ ph, int kx, int ky, int l) {
    const double2 a = ph[kx], b = ph[l + ky];
    return make_float2((float)(a.x * b.x - a.y * b.y), (float)(a.x * b.y + a.y * b.x));
}

// c, sigma^2 and d c / d (dx, dy): reductions over the spectrum.
static __global__ void __launch_bounds__(256) k_ref_score(const float2* __restrict__ W, const float2* __restrict__ F,
                                                          const RefinePickDev* __restrict__ pks,
                                                          const double2* __restrict__ phases, RefineConsts rc,
                                                          RefineAcc* __restrict__ acc) {
    __shared__ double red[4 * 32];
    const int p = blockIdx.y;
    const int l = rc.l, npix = l * l;
    const float2* Wp = W + (long long)pks[p].window * rc.L2;
    const float2* Fp = F + p * rc.L2;
    const double2* ph = phases + (size_t)p * 2 * l;
    const double step = 2.0 * kPiRef / l;
    double a4[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const int ky = i / l, kx = i - ky * l;
        const int sx = kx < (l + 1) / 2 ? kx : kx - l, sy = ky < (l + 1) / 2 ? ky : ky - l;
        const float2 E = ref_phase(ph, kx, ky, l), w = Wp[i], f = Fp[i];
        const float2 GE = cmul(cmulc(w, f), E);        // W conj(F) E
        a4[0] += GE.x;
        const float w2 = w.x * w.x + w.y * w.y;
        const float f2 = f.x * f.x + f.y * f.y;
        a4[1] += (double)w2 * f2;
        // d/d dx of Re(GE) = Re(GE * 2 pi i kx / l) = -Im(GE) 2 pi kx / l
        a4[2] += -(double)GE.y * (step * sx);
        a4[3] += -(double)GE.y * (step * sy);
    }
    block_sum<4>(a4, red);
    if (threadIdx.x == 0) {
        atomicAdd(&acc[p].c, a4[0]);
        atomicAdd(&acc[p].sig2, a4[1]);
        atomicAdd(&acc[p].cdx, a4[2]);
        atomicAdd(&acc[p].cdy, a4[3]);
    }
}

// ---- backward ----

// Fbar = (sgn / sig) W E - (sgn c / sig^3) |W|^2 F, whose inverse transform is
// gamma l^2.
static __global__ void __launch_bounds__(256) k_ref_fbar(const float2* __restrict__ W, const float2* __restrict__ F,
                                                         const RefinePickDev* __restrict__ pks,
                                                         const double2* __restrict__ phases,
                                                         const RefineAcc* __restrict__ acc, int l, float sgn,
                                                         float2* __restrict__ out) {
    const int p = blockIdx.y, npix = l * l;
    const float2* Wp = W + (long long)pks[p].window * npix;
    const double2* ph = phases + (size_t)p * 2 * l;
    const double sig = sqrt(acc[p].sig2);
    const float c1 = (float)(sgn / sig);
    const float c2 = (float)(sgn * acc[p].c / (sig * sig * sig));
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const int ky = i / l, kx = i - ky * l;
        const float2 w = Wp[i], f = F[(long long)p * npix + i];
        const float w2 = w.x * w.x + w.y * w.y;
        const float2 we = cmul(w, ref_phase(ph, kx, ky, l));
        out[(long long)p * npix + i] = make_float2(c1 * we.x - c2 * w2 * f.x, c1 * we.y - c2 * w2 * f.y);
    }
}

// sums of gamma and gamma tn (tn = (tm - mu) / sd; tm is 0 outside [row0, row1)).
static __global__ void __launch_bounds__(256) k_ref_gsum(const float* __restrict__ G, const float* __restrict__ TM,
                                                         RefineConsts rc, int row0, int row1,
                                                         RefineAcc* __restrict__ acc) {
    __shared__ double red[64];
    const int p = blockIdx.y, npix = rc.l * rc.l;
    double mu, sd;
    ref_moments(acc[p], (double)rc.L2, &mu, &sd);
    double a2[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const double g = G[p * rc.L2 + i];
        const bool in = i >= row0 * rc.l && i < row1 * rc.l;
        a2[0] += g;
        a2[1] += g * ((in ? (double)TM[p * rc.L2 + i] : 0.0) - mu);
    }
    block_sum<2>(a2, red);
    if (threadIdx.x == 0) {
        atomicAdd(&acc[p].g1, a2[0]);
        atomicAdd(&acc[p].g2, a2[1] / sd);
    }
}

// Normalisation, mask and rotation adjoints: d s / d e (reduction) and
// tbar (scatter-add into the real parts of TB, zeroed beforehand in the rows
// [row0, row1), which hold all of it).
static __global__ void __launch_bounds__(256) k_ref_rot_adj(const float* __restrict__ G, const float* __restrict__ TM,
                                                            const float* __restrict__ T,
                                                            const RefinePickDev* __restrict__ pks, RefineConsts rc,
                                                            int row0, int row1, const float* __restrict__ mask,
                                                            RefineAcc* __restrict__ acc, float2* __restrict__ TB) {
    __shared__ double red[32];
    const int p = blockIdx.y;
    const int l = rc.l;
    double mu, sd;
    ref_moments(acc[p], (double)rc.L2, &mu, &sd);
    const double L2 = (double)rc.L2;
    const double mg = acc[p].g1 / L2, mgt = acc[p].g2 / L2;
    const double ang = (double)pks[p].e * kPiRef / 180.0;
    const float c = (float)cos(ang), s = (float)sin(ang);
    const float* src = T + p * rc.L2;
    float2* tb = TB + p * rc.L2;
    const double inv_sd = 1.0 / sd;
    const float dr = (float)(kPiRef / 180.0);
    double de = 0.0;
    for (int i = row0 * l + blockIdx.x * blockDim.x + threadIdx.x; i < row1 * l; i += gridDim.x * blockDim.x) {
        const float m = mask[i];
        if (m == 0.0f) continue;
        const int y = i / l, x = i - y * l;
        const double g = G[p * rc.L2 + i];
        const double tn = ((double)TM[p * rc.L2 + i] - mu) * inv_sd;
        const float gm = (float)((g - mg - tn * mgt) * inv_sd) * m;  // d s / d rotated pixel
        if (gm == 0.0f) continue;
        float x2, y2;
        rot_src(x, y, l, c, s, &x2, &y2);
        const Bilin b = bilin(x2, y2, l);
        if (!b.inb) continue;
        const float v0 = src[b.k[0]], v1 = src[b.k[1]], v2 = src[b.k[2]], v3 = src[b.k[3]];
        // value = (1-t)(1-u) v0 + t(1-u) v1 + t u v2 + (1-t) u v3
        const float dvdt = (1.0f - b.du) * (v1 - v0) + b.du * (v2 - v3);
        const float dvdu = (1.0f - b.dt) * (v3 - v0) + b.dt * (v2 - v1);
        const float xf = (float)(x - l / 2), yf = (float)(y - l / 2);
        const float dx2 = dr * (-s * xf + c * yf), dy2 = dr * (-c * xf - s * yf);
        de += (double)gm * (dvdt * dx2 + dvdu * dy2);
#pragma unroll
        for (int q = 0; q < 4; ++q) atomicAdd(&tb[b.k[q]].x, gm * b.w[q]);
    }
    double v1[1] = {de};
    block_sum<1>(v1, red);
    if (threadIdx.x == 0) atomicAdd(&acc[p].de, v1[0]);
}

// abar = -Re sum Fbar2 conj(F1) / a^2 (only the sum here).
static __global__ void __launch_bounds__(256) k_ref_abar(const float2* __restrict__ Fb2, const float2* __restrict__ F1,
                                                  RefineConsts rc, RefineAcc* __restrict__ acc) {
    __shared__ double red[32];
    const int p = blockIdx.y;
    double s = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rc.L2; i += (long long)gridDim.x * blockDim.x) {
        const float2 u = Fb2[p * rc.L2 + i], v = F1[p * rc.L2 + i];
        s += (double)u.x * v.x + (double)u.y * v.y;
    }
    double v1[1] = {s};
    block_sum<1>(v1, red);
    if (threadIdx.x == 0) atomicAdd(&acc[p].abar, v1[0]);
}

// Fbar1 = Fbar2 / a + abar_total F1 sel / (cnt^2 a); theta gradient
// reductions; with `store`, Bbar = Fbar1 w written over Fb2 (for the template
// gradient).
static __global__ void __launch_bounds__(256) k_ref_theta(float2* __restrict__ Fb2, const float2* __restrict__ F1,
                                                          const float2* __restrict__ base,
                                                          const RefineBin* __restrict__ bins,
                                                          const RefinePickDev* __restrict__ pks, RefineConsts rc,
                                                          bool store, RefineAcc* __restrict__ acc) {
    __shared__ double red[3 * 32];
    const int p = blockIdx.y;
    const RefinePickDev pk = pks[p];
    const int l = rc.l, npix = l * l;
    const float2* H = base + (long long)pk.tmpl * l * (l / 2 + 1);
    const double a = sqrt(acc[p].asum) / (double)rc.cnt;
    const double abar = -acc[p].abar / (a * a);
    const double k2 = abar / ((double)rc.cnt * (double)rc.cnt * a);
    const float inva = (float)(1.0 / a);
    double t3[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x) {
        const int y = i / l, x = i - y * l;
        bool insel;
        float dw[3];
        const float w = refine_weight<true>(bins[i], rc, pk, &insel, dw);
        if (!insel && !store) continue;
        float2 fb = cscale(Fb2[p * rc.L2 + i], inva);
        if (insel && x <= l / 2) {
            const float2 f1 = F1[p * rc.L2 + i];
            fb.x += (float)(k2 * f1.x);
            fb.y += (float)(k2 * f1.y);
        }
        const float2 bb = ref_base(H, x, y, l);
        const double re = (double)fb.x * bb.x + (double)fb.y * bb.y;  // Re(Fbar1 conj(B))
        t3[0] += re * dw[0];
        t3[1] += re * dw[1];
        t3[2] += re * dw[2];
        if (store) Fb2[p * rc.L2 + i] = cscale(fb, w);
    }
    block_sum<3>(t3, red);
    if (threadIdx.x == 0) {
        atomicAdd(&acc[p].dth[0], t3[0]);
        atomicAdd(&acc[p].dth[1], t3[1]);
        atomicAdd(&acc[p].dth[2], t3[2]);
    }
}

}  // namespace gs
