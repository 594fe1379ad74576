// Hencky-strain von Mises return mapping with hardening, tensile-energy
// history and the phase-field driving coefficient: the per-particle
// arithmetic of the reference's applyVonMises
// (ExplicitTimeIntegrator.cu:132-370, R() :64-68, computePhase_field_vol :49-62),
// and the reference's two other energy models (fixed-corotated and
// Neo-Hookean with fracture, :22-47 and :372-446).
#pragma once
#include "common.cuh"
#include "svd3.cuh"

namespace gmpm {

// The reference's FP64 build rounds these two constants through float:
// parameter1 = 2.f/3.f (ExplicitTimeIntegrator.cu:190) and sqrt(2.f/3.f) in R()
// (:67).  The same values are used here in both precisions.
template <typename R> __device__ __forceinline__ R c_p23() { return R(2.0f / 3.0f); }
template <typename R> __device__ __forceinline__ R c_sqrt_p23() { return sqrt(R(2.0f / 3.0f)); }
template <typename R> __device__ __forceinline__ R c_sqrt_p23_f() { return R(sqrtf(2.0f / 3.0f)); }

// FP32 exponentials and powers on the special-function unit (__expf, __powf:
// a few ulp for the small arguments here, the exponentials of strains and of
// softening terms and J^(-2/3) with J near 1); FP64 and the FP32 logarithms
// (Hencky strains and ln J near 1, where only a relative-accurate log keeps
// the small strains) use the accurate library functions.
__device__ __forceinline__ float exp_r(float x) { return __expf(x); }
__device__ __forceinline__ double exp_r(double x) { return exp(x); }
__device__ __forceinline__ float log_r(float x) { return logf(x); }
__device__ __forceinline__ double log_r(double x) { return log(x); }
__device__ __forceinline__ float pow_r(float x, float y) { return __powf(x, y); }
__device__ __forceinline__ double pow_r(double x, double y) { return pow(x, y); }

template <typename R, typename MR>
__device__ __forceinline__ R hardening_R(const MaterialDev<MR>& m, R alpha) {
    const R y = R(m.yield_stress);
    if (m.hardening_law == GMPM_HARDENING_LINEAR) return y + R(m.hardening) * alpha;
    const R sq = c_sqrt_p23_f<R>();
    return sq * y - div_r(sq * y - y, exp_r(R(m.hardening) * alpha));
}

template <typename R>
struct StressOut {
    R F[9];       // projected F, column-major
    R sigma[6];   // V0 * P F^T: xx yy zz xy xz yz
    R alpha, psi, FP, vol;
    R smin_over_smax;
    bool svd_ok;
};

// F column-major (r + 3c).  g_old: degradation used by the trial state (the
// reference's p_g from the previous update), c: current damage.
// SVD of F (column-major) into U, S, V (row-major), with its success and
// conditioning recorded in o.
template <typename R>
__device__ __forceinline__ void svd_of(const R* Fin, R* U, R* S, R* V, StressOut<R>& o) {
    R A[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) A[3 * r + q] = Fin[r + 3 * q];
    o.svd_ok = svd3(A, U, S, V);
    const R smax = fmax(fabs(S[0]), fmax(fabs(S[1]), fabs(S[2])));
    const R smin = fmin(fabs(S[0]), fmin(fabs(S[1]), fabs(S[2])));
    o.smin_over_smax = (smax > R(0)) ? div_r(smin, smax) : R(0);
}

template <typename R, typename MR>
__device__ __forceinline__ void von_mises_from_svd(const MaterialDev<MR>& m, R V0, const R* Fin, const R* U, R* S,
                                                   const R* V, R g, R alpha, R c, R psi, StressOut<R>& o) {
    const R lambda = R(m.lambda), mu = R(m.mu), kappa = R(m.kappa);
    const R C0 = R(2) * mu + lambda, C1 = lambda;
    R eps[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) eps[k] = (S[k] > R(0)) ? log_r(S[k]) : R(0);
    R tt[3];
    tt[0] = C0 * eps[0] + C1 * eps[1] + C1 * eps[2];
    tt[1] = C1 * eps[0] + C0 * eps[1] + C1 * eps[2];
    tt[2] = C1 * eps[0] + C1 * eps[1] + C0 * eps[2];
    const R ttF = sqrt(tt[0] * tt[0] + tt[1] * tt[1] + tt[2] * tt[2]);
    const R tsum = tt[0] + tt[1] + tt[2];
    const R divider = div_r(tsum, R(3));
    R tdev[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) tdev[k] = g * (tt[k] - divider);
    const R p23 = c_p23<R>();
    const R sp23 = c_sqrt_p23<R>();
    const R y = ttF - g * hardening_R<R>(m, alpha) * sp23;
    R alpha_out = alpha;
    R F[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) F[q] = Fin[q];
    if (y >= R(1e-12)) {
        R dl = R(0);
        const R bss = p23 * g * tsum;
        if (bss > R(0)) dl = div_r(y, bss);
        if (dl > R(m.dlambda_cap)) dl = R(m.dlambda_cap);
        if (alpha < R(m.alpha_cap)) {
            alpha += sp23 * dl;
            alpha_out = alpha;
        }
        if (alpha > R(m.alpha_cap)) alpha_out = R(m.alpha_cap);
        const R tn = sqrt(tdev[0] * tdev[0] + tdev[1] * tdev[1] + tdev[2] * tdev[2]);
        // The reference divides by |tau_dev| (ExplicitTimeIntegrator.cu:242); its
        // yield test uses the full trial stress, so a hydrostatic trial state
        // (equal singular values, exact in FP32) can yield with tau_dev = 0.
        // There is no deviator to scale then: the factor is 0 instead of NaN.
        const R taudiv = tn > R(0) ? div_r(R(1), tn) * p23 * g * tsum * dl : R(0);
        const R p2 = (R(1) / R(3)) * tsum;
        R tnn[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) tnn[k] = (tdev[k] - tdev[k] * taudiv) + p2;
        R en[3];
        en[0] = R(m.D[0]) * tnn[0] + R(m.D[1]) * tnn[1] + R(m.D[2]) * tnn[2];
        en[1] = R(m.D[3]) * tnn[0] + R(m.D[4]) * tnn[1] + R(m.D[5]) * tnn[2];
        en[2] = R(m.D[6]) * tnn[0] + R(m.D[7]) * tnn[1] + R(m.D[8]) * tnn[2];
        const R nS = sqrt(en[0] * en[0] + en[1] * en[1] + en[2] * en[2]);
        const R cap = R(m.strain_cap);
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (en[k] > cap) en[k] = en[k] * div_r(cap, nS);
#pragma unroll
        for (int k = 0; k < 3; ++k) S[k] = exp_r(en[k]);
        // F = U diag(S) V^T (column-major output)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 3; ++q)
                F[r + 3 * q] = S[0] * U[3 * r] * V[3 * q] + S[1] * U[3 * r + 1] * V[3 * q + 1] +
                               S[2] * U[3 * r + 2] * V[3 * q + 2];
    }
    const R J = S[0] * S[1] * S[2];
    const R Jbar = pow_r(J, -p23);
    R bb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) bb[k] = Jbar * S[k] * S[k];
    const R bbs = bb[0] + bb[1] + bb[2];
    const R lnJ = (J > R(0)) ? log_r(J) : R(0);
    const R psi_vol = (kappa * R(0.5)) * (((J * J - R(1)) * R(0.5)) - lnJ);
    const R psi_dev = (mu * R(0.5)) * (bbs - R(3));
    const R psi_pos = (J < R(1)) ? psi_dev : psi_dev + psi_vol;
    if (psi_pos > psi && psi_pos < R(m.psi_cap)) psi = psi_pos;
    const R p = alpha / R(2);
    R Gc;
    if (p < R(m.softening_onset))
        Gc = R(m.fracture_energy);
    else
        Gc = R(m.fracture_energy) *
             (((R(1) - R(m.residual_fracture)) * exp_r(R(m.softening_onset) - p)) + R(m.residual_fracture));
    const R theta = R(m.theta), one_minus_theta = R(m.one_minus_theta);
    o.FP = R(4) * R(m.length_scale) * one_minus_theta * psi * div_r(R(1), Gc) + R(1);
    const R tvol = (kappa * R(0.5)) * (J * J - R(1));
    const R third = (R(1) / R(3)) * bbs;
    const R gn = c * c * one_minus_theta + theta;
    R Ph[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const R td = mu * (bb[k] - third);
        Ph[k] = (J < R(1)) ? gn * td + tvol : gn * (td + tvol);
    }
    // sigma = V0 P F^T with P = U diag(Ph) V^T and F = U diag(S) V^T, i.e.
    // V0 U diag(Ph*S) U^T; evaluated as the reference does (P then P F^T) so
    // that F from the unprojected branch enters exactly.
    R P[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            P[r + 3 * q] =
                Ph[0] * U[3 * r] * V[3 * q] + Ph[1] * U[3 * r + 1] * V[3 * q + 1] + Ph[2] * U[3 * r + 2] * V[3 * q + 2];
    R sig[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            sig[r + 3 * q] = (P[r] * F[q] + P[r + 3] * F[q + 3] + P[r + 6] * F[q + 6]) * V0;
    o.sigma[0] = sig[0];
    o.sigma[1] = sig[4];
    o.sigma[2] = sig[8];
    o.sigma[3] = R(0.5) * (sig[3] + sig[1]);
    o.sigma[4] = R(0.5) * (sig[6] + sig[2]);
    o.sigma[5] = R(0.5) * (sig[7] + sig[5]);
    const R det = F[0] * F[4] * F[8] + F[3] * F[7] * F[2] + F[6] * F[1] * F[5] - F[2] * F[4] * F[6] -
                  F[1] * F[3] * F[8] - F[0] * F[5] * F[7];
#pragma unroll
    for (int q = 0; q < 9; ++q) o.F[q] = F[q];
    o.alpha = alpha_out;
    o.psi = psi;
    o.vol = V0 * det;
}

// Isotropic elastic stress from singular values: P = U diag(Ph) V^T, then
// sigma = V0 P F^T (symmetric part, xx yy zz xy xz yz), evaluated as the
// reference's contribution kernels do (P, then P F^T).  F column-major.
template <typename R>
__device__ __forceinline__ void elastic_sigma(const R* U, const R* V, const R* Ph, const R* F, R V0, R* sigma6) {
    R P[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            P[r + 3 * q] =
                Ph[0] * U[3 * r] * V[3 * q] + Ph[1] * U[3 * r + 1] * V[3 * q + 1] + Ph[2] * U[3 * r + 2] * V[3 * q + 2];
    R sig[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            sig[r + 3 * q] = (P[r] * F[q] + P[r + 3] * F[q + 3] + P[r + 6] * F[q + 6]) * V0;
    sigma6[0] = sig[0];
    sigma6[1] = sig[4];
    sigma6[2] = sig[8];
    sigma6[3] = R(0.5) * (sig[3] + sig[1]);
    sigma6[4] = R(0.5) * (sig[6] + sig[2]);
    sigma6[5] = R(0.5) * (sig[7] + sig[5]);
}

template <typename R>
__device__ __forceinline__ R det3(const R* F) {
    return F[0] * F[4] * F[8] + F[3] * F[7] * F[2] + F[6] * F[1] * F[5] - F[2] * F[4] * F[6] - F[1] * F[3] * F[8] -
           F[0] * F[5] * F[7];
}

// J^(-2/3) in single precision: the reference evaluates it with the float
// power intrinsic.  In FP64 it is taken in double and rounded to float, the
// correctly rounded single-precision value (reproducible on the host too).
__device__ __forceinline__ float jbar_r(float J) { return powf(J, -2.0f / 3.0f); }
__device__ __forceinline__ double jbar_r(double J) { return (double)(float)pow((double)(float)J, (double)(-2.0f / 3.0f)); }

// Elastic fixed-corotated energy (computeContributionFixedCorotated,
// ExplicitTimeIntegrator.cu:22-47): Ph_k = 2 mu (S_k - 1) + lambda (J - 1)
// prod_{l != k} S_l.  No plasticity and no fracture driving (FP = 1).
template <typename R, typename MR>
__device__ __forceinline__ void fixed_corotated_from_svd(const MaterialDev<MR>& m, R V0, const R* Fin, const R* U,
                                                         const R* S, const R* V, R alpha, R psi, StressOut<R>& o) {
    const R lambda = R(m.lambda), mu = R(m.mu);
    const R J = S[0] * S[1] * S[2];
    const R smu = R(2) * mu, slam = lambda * (J - R(1));
    const R Ph[3] = {smu * (S[0] - R(1)) + slam * (S[1] * S[2]), smu * (S[1] - R(1)) + slam * (S[0] * S[2]),
                     smu * (S[2] - R(1)) + slam * (S[0] * S[1])};
    elastic_sigma(U, V, Ph, Fin, V0, o.sigma);
#pragma unroll
    for (int q = 0; q < 9; ++q) o.F[q] = Fin[q];
    o.alpha = alpha;
    o.psi = psi;
    o.FP = R(1);
    o.vol = V0 * det3(Fin);
}

// Elastic Neo-Hookean energy with the tension/compression split and the
// phase-field driving (computeContributionNeoHookean,
// ExplicitTimeIntegrator.cu:372-446): psi+ history, FP = 4 L0 (1 - 0.001)
// psi+ / G_c + 1 with G_c = 3 and L0 = dx/2, degradation
// g = c^2 (1 - 1e-4) + 1e-4 on the deviatoric (compression) or whole
// (tension) Kirchhoff stress.  The reference's psi_vol uses (J - 1)/2.
template <typename R, typename MR>
__device__ __forceinline__ void neo_hookean_fracture_from_svd(const MaterialDev<MR>& m, R V0, R dx, const R* Fin,
                                                              const R* U, const R* S, const R* V, R alpha, R c,
                                                              R psi, StressOut<R>& o) {
    const R mu = R(m.mu), kappa = R(m.kappa);
    const R J = S[0] * S[1] * S[2];
    const R Jbar = jbar_r(J);
    R bb[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) bb[k] = Jbar * S[k] * S[k];
    const R bbs = bb[0] + bb[1] + bb[2];
    const R lnJ = log_r(J);
    const R psi_vol = kappa / R(2) * ((J - R(1)) / R(2) - lnJ);
    const R psi_dev = mu / R(2) * (bb[0] + bb[1] + bb[2] - R(3));
    const R psi_pos = (J < R(1)) ? psi_dev : psi_dev + psi_vol;
    if (psi_pos > psi && psi_pos < R(1e6)) psi = psi_pos;
    const R L0 = R(0.5) * dx;
    o.FP = R(4) * L0 * R(1.f - 0.001f) * psi * R(1) / R(3) + R(1);
    const R tvol = kappa / R(2) * (J * J - R(1));
    const R third = R(1.f / 3.f) * bbs;
    const R g = c * c * R(1.f - 0.0001f) + R(0.0001f);
    R Ph[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const R td = mu * (bb[k] - third);
        Ph[k] = (J < R(1)) ? g * td + tvol : g * (td + tvol);
    }
    elastic_sigma(U, V, Ph, Fin, V0, o.sigma);
#pragma unroll
    for (int q = 0; q < 9; ++q) o.F[q] = Fin[q];
    o.alpha = alpha;
    o.psi = psi;
    o.vol = V0 * det3(Fin);
}

// The least ratio of two singular values at the small strains' bound,
// |G| <= 0.1 for G = F F^T - I: eigenvalues a and b of G with a^2 + b^2 <= 0.01 give sqrt((1 + a) / (1 + b)) >= 0.9316.
constexpr float kSmallStrainRatio = 0.93f;

// FP32 von Mises update for small strains, |F F^T - I| <= 0.1 and det F > 0
// (Frobenius; false otherwise, and where the projected strain is larger).  The model is
// isotropic, so every quantity is a polynomial I, G, G^2 of G = F F^T - I, with
// coefficients from G's invariants (Cayley-Hamilton reduces the higher powers):
// the Hencky strain by the logarithm's series, the projected state by the
// exponential's.  Within the bounds the series' rest is below FP32 rounding: at
// |G| = 0.1, 7e-9 of the strain; at |2 f P| = 0.12, 5e-9; at |t| = 0.1 (the return
// map keeps the trace, which the bound on G holds below 0.09), 1.3e-8 of J^2 - 1.
// No singular vectors, and G is formed from F - I, and J^2 - 1, psi+ and the
// deviators without their leading ones, so that nothing cancels near the identity
// (a particle turned by a large angle has entries of F - I of order 1, and its G
// the rounding of F F^T).  Bound: G2P
// is bound by instruction issue, and the QR sweeps, the stress assembly from U
// and V and the logarithms were a third of its 1,900 instructions a particle.
// Measured: G2P 678 -> 567 us at 8.4M particles, 41 -> 32 us at 131k; the error
// of F against FP64 is 0.5 to 1 times the SVD's, and of velocities near rest as
// little as a thousandth.  kYield = false (the precision form, FP32 with the
// FP64 fallback) leaves yielding particles to the SVD: the return map amplifies
// a difference of rounding 1e4-fold, and that form's projected states stay as
// they were (G2P 200 -> 184 us at 1.9M particles while few yield, 1% slower
// once most warps take both paths).
template <typename MR, bool kYield>
__device__ __forceinline__ bool small_strain_update(const MaterialDev<MR>& m, float V0, const float* Fin, float g,
                                                    float alpha, float c, float psi, StressOut<float>& o) {
    float E[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) E[q] = q % 4 == 0 ? Fin[q] - 1.f : Fin[q];
    auto gram = [&](int i, int j) {
        return E[i + 3 * j] + E[j + 3 * i] + (E[i] * E[j] + E[i + 3] * E[j + 3] + E[i + 6] * E[j + 6]);
    };
    // symmetric tensors as 00 11 22 01 02 12
    const float A[6] = {gram(0, 0), gram(1, 1), gram(2, 2), gram(0, 1), gram(0, 2), gram(1, 2)};
    auto square = [](const float* T, float* Q) {
        Q[0] = T[0] * T[0] + T[3] * T[3] + T[4] * T[4];
        Q[1] = T[3] * T[3] + T[1] * T[1] + T[5] * T[5];
        Q[2] = T[4] * T[4] + T[5] * T[5] + T[2] * T[2];
        Q[3] = T[3] * (T[0] + T[1]) + T[4] * T[5];
        Q[4] = T[4] * (T[0] + T[2]) + T[3] * T[5];
        Q[5] = T[5] * (T[1] + T[2]) + T[3] * T[4];
    };
    auto det = [](const float* T) {
        return T[0] * (T[1] * T[2] - T[5] * T[5]) - T[3] * (T[3] * T[2] - T[5] * T[4]) + T[4] * (T[3] * T[5] - T[1] * T[4]);
    };
    float B[6];
    square(A, B);
    const float n2 = B[0] + B[1] + B[2];  // |G|^2
    if (!(n2 <= 0.01f)) return false;
    // F F^T does not tell a reflection from a rotation; the SVD path does, and its stress is then not a number
    float J = det3(Fin);
    if (!(J > 0.f)) return false;
    // eps = 1/2 log(I + G) = e0 I + e1 G + e2 G^2, with (p0, p1, p2) the coefficients of G^3, G^4, ...
    const float i1 = A[0] + A[1] + A[2], i2 = 0.5f * (i1 * i1 - n2), i3 = det(A);
    float e0 = 0.f, e1 = 0.5f, e2 = -0.25f;
    {
        float p0 = i3, p1 = -i2, p2 = i1;
#pragma unroll
        for (int k = 3; k <= 6; ++k) {
            const float w = (k & 1 ? 0.5f : -0.5f) / (float)k;
            e0 += w * p0;
            e1 += w * p1;
            e2 += w * p2;
            const float q0 = p2 * i3, q1 = p0 - p2 * i2, q2 = p1 + p2 * i1;
            p0 = q0;
            p1 = q1;
            p2 = q2;
        }
    }
    // trace and deviator of eps
    const float t0 = 3.f * e0 + e1 * i1 + e2 * n2;
    float P[6], Q[6];
    {
        const float sh = (e1 * i1 + e2 * n2) * (1.f / 3.f);
#pragma unroll
        for (int q = 0; q < 6; ++q) P[q] = e1 * A[q] + e2 * B[q] - (q < 3 ? sh : 0.f);
    }
    square(P, Q);
    const float PP = Q[0] + Q[1] + Q[2], dP = det(P);
    // return map (von_mises_principal, in invariants): the projected strain is f P + t / 3 I
    const float lambda = (float)m.lambda, mu = (float)m.mu, kappa = (float)m.kappa;
    const float kt = (2.f / 3.f * mu + lambda) * t0, tsum = 3.f * kt;
    const float p23 = c_p23<float>(), sp23 = c_sqrt_p23<float>();
    const float y = sqrtf(4.f * mu * mu * PP + 3.f * kt * kt) - g * hardening_R<float>(m, alpha) * sp23;
    float alpha_out = alpha, f = 1.f, t = t0;
    const bool yields = y >= 1e-12f;
    if (!kYield && yields) return false;
    if (yields) {
        float dl = 0.f;
        const float bss = p23 * g * tsum;
        if (bss > 0.f) dl = div_r(y, bss);
        if (dl > (float)m.dlambda_cap) dl = (float)m.dlambda_cap;
        if (alpha < (float)m.alpha_cap) {
            alpha += sp23 * dl;
            alpha_out = alpha;
        }
        if (alpha > (float)m.alpha_cap) alpha_out = (float)m.alpha_cap;
        const float tn = g * 2.f * mu * sqrtf(PP);
        const float taudiv = tn > 0.f ? div_r(1.f, tn) * p23 * g * tsum * dl : 0.f;
        const float d0 = (float)m.D[0] - (float)m.D[1];
        f = d0 * (1.f - taudiv) * g * 2.f * mu;
        t = 3.f * kt * (d0 + 3.f * (float)m.D[1]);
        // beyond the series (and far below any sensible strain cap, which clamps principal strains)
        if (!(f * f * PP <= 0.0036f && fabsf(t) <= 0.1f && (float)m.strain_cap >= 0.2f)) return false;
    }
    // exp(N) = a0 I + a1 N + a2 N^2 and exp(N / 2) = s0 I + s1 N + s2 N^2 for N = 2 f P
    const float q = 2.f * f * f * PP, dN = 8.f * f * f * f * dP;
    const float am = dN * (1.f / 6.f + q * (1.f / 120.f));  // a0 - 1
    const float a1 = 1.f + q * (1.f / 6.f + q * (1.f / 120.f)) + dN * (1.f / 24.f);
    const float a2 = 0.5f + q * (1.f / 24.f) + dN * (1.f / 120.f);
    const float s0 = 1.f + dN * (1.f / 48.f + q * (1.f / 3840.f));
    const float s1 = 0.5f + q * (1.f / 48.f + q * (1.f / 3840.f)) + dN * (1.f / 384.f);
    const float s2 = 0.125f + q * (1.f / 384.f) + dN * (1.f / 3840.f);
    // J^2 - 1 = x (1 + h), x = 2 t = 2 ln J
    const float x = 2.f * t;
    const float h = x * 0.5f * (1.f + x * (1.f / 3.f) * (1.f + x * 0.25f * (1.f + x * 0.2f * (1.f + x * (1.f / 6.f)))));
    const float psi_dev = (mu * 0.5f) * (3.f * am + 2.f * q * a2);
    const float psi_pos = t < 0.f ? psi_dev : psi_dev + (kappa * 0.5f) * (0.5f * x * h);
    if (psi_pos > psi && psi_pos < (float)m.psi_cap) psi = psi_pos;
    const float pl = alpha * 0.5f;
    float Gc = (float)m.fracture_energy;
    if (!(pl < (float)m.softening_onset))
        Gc *= ((1.f - (float)m.residual_fracture) * exp_r((float)m.softening_onset - pl)) + (float)m.residual_fracture;
    const float theta = (float)m.theta, one_minus_theta = (float)m.one_minus_theta;
    o.FP = 4.f * (float)m.length_scale * one_minus_theta * psi * div_r(1.f, Gc) + 1.f;
    const float tvol = (kappa * 0.5f) * (x * (1.f + h));
    const float gn = c * c * one_minus_theta + theta;
    // principal stresses w0 I + w1 N + w2 N^2, times exp(N / 2) exp(t / 3) (N^3 = q N + dN I)
    const float w1 = gn * mu * a1, w2 = gn * mu * a2;
    const float w0 = (t < 0.f ? tvol : gn * tvol) - w2 * q * (2.f / 3.f);
    const float cross = w1 * s2 + w2 * s1, u = t * (1.f / 3.f);
    const float sc = V0 * (1.f + u * (1.f + u * 0.5f * (1.f + u * (1.f / 3.f) * (1.f + u * 0.25f))));
    const float r0 = sc * (w0 * s0 + cross * dN);
    const float r1 = sc * (w0 * s1 + w1 * s0 + cross * q + w2 * s2 * dN) * (2.f * f);
    const float r2 = sc * (w0 * s2 + w1 * s1 + w2 * s0 + w2 * s2 * q) * (4.f * f * f);
#pragma unroll
    for (int k = 0; k < 6; ++k) o.sigma[k] = r1 * P[k] + r2 * Q[k] + (k < 3 ? r0 : 0.f);
#pragma unroll
    for (int k = 0; k < 9; ++k) o.F[k] = Fin[k];
    if (yields) {
        // F <- exp(h1 P + (t - t0) / 3 I) F
        const float h1 = f - 1.f, qM = 0.5f * h1 * h1 * PP, dM = h1 * h1 * h1 * dP, v = (t - t0) * (1.f / 3.f);
        const float ev = 1.f + v * (1.f + v * 0.5f * (1.f + v * (1.f / 3.f) * (1.f + v * 0.25f)));
        const float x0 = ev * (1.f + dM * (1.f / 6.f + qM * (1.f / 120.f)));
        const float x1 = ev * h1 * (1.f + qM * (1.f / 6.f + qM * (1.f / 120.f)) + dM * (1.f / 24.f));
        const float x2 = ev * h1 * h1 * (0.5f + qM * (1.f / 24.f) + dM * (1.f / 120.f));
        float X[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) X[k] = x1 * P[k] + x2 * Q[k] + (k < 3 ? x0 : 0.f);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float f0 = Fin[3 * k], f1 = Fin[3 * k + 1], f2 = Fin[3 * k + 2];
            o.F[3 * k] = X[0] * f0 + X[3] * f1 + X[4] * f2;
            o.F[3 * k + 1] = X[3] * f0 + X[1] * f1 + X[5] * f2;
            o.F[3 * k + 2] = X[4] * f0 + X[5] * f1 + X[2] * f2;
        }
        J = det3(o.F);
    }
    o.alpha = alpha_out;
    o.psi = psi;
    o.vol = V0 * J;
    o.svd_ok = true;
    o.smin_over_smax = kSmallStrainRatio;
    return true;
}

// The material's energy model, after one SVD of F.  kAnyModel = false
// compiles the von Mises model alone (scenes whose materials all use it).
// small: small strains may take the update by invariants.
template <typename R, typename MR, bool kAnyModel = true, bool kSmallYield = true>
__device__ __forceinline__ void constitutive_update(const MaterialDev<MR>& m, R V0, R dx, const R* Fin, R g_old,
                                                    R alpha, R c, R psi, StressOut<R>& o, bool small = true) {
    if constexpr (sizeof(R) == 4)
        if (small && (!kAnyModel || m.energy_model == GMPM_ENERGY_VON_MISES_FRACTURE) &&
            small_strain_update<MR, kSmallYield>(m, V0, Fin, g_old, alpha, c, psi, o))
            return;
    R U[9], V[9], S[3];
    svd_of(Fin, U, S, V, o);
    if (!kAnyModel)
        von_mises_from_svd<R, MR>(m, V0, Fin, U, S, V, g_old, alpha, c, psi, o);
    else if (m.energy_model == GMPM_ENERGY_FIXED_COROTATED)
        fixed_corotated_from_svd<R, MR>(m, V0, Fin, U, S, V, alpha, psi, o);
    else if (m.energy_model == GMPM_ENERGY_NEO_HOOKEAN_FRACTURE)
        neo_hookean_fracture_from_svd<R, MR>(m, V0, dx, Fin, U, S, V, alpha, c, psi, o);
    else
        von_mises_from_svd<R, MR>(m, V0, Fin, U, S, V, g_old, alpha, c, psi, o);
}

}  // namespace gmpm
