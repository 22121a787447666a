// lyd_physics.cuh -- device arithmetic of the Lyman-alpha M1 step, templated on the
// arithmetic type R (double for the FP64 step, float for the bulk of the mixed step).
//
// Each function restates one piece of the LYDION reference (paths inside its source tree):
// the M1 closure (src/M1Closure.jl), PLM reconstruction and the GLF/HLL fluxes
// (src/AdvectJandH.jl), and the exponentially fitted frequency leakage coefficients
// (src/FreqFactors.jl). Thresholds that depend on the storage scale of J (the floors
// Jeps, Heps^2) are passed in at run time.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace lyd {

// ---- constants (src/ConstantsAndFunctions.jl:46-170) -------------------------------------
constexpr double kC = 2.99792458e10;
constexpr double kInvC = 1.0 / kC;
constexpr double kPi = 3.14159265358979323846;
constexpr double kFourPi = 4.0 * kPi;
constexpr double kFourPiOverC = kFourPi / kC;
constexpr double kHPlanck = 6.626069573e-27;
constexpr double kKBoltz = 1.380648813e-16;
constexpr double kHOverKB = kHPlanck / kKBoltz;
constexpr double kNuLya = 2.466068e15;
constexpr double kMH = 1.0080 * 1.660539069e-24;
constexpr double kALya = 6.265e8;
constexpr double kA2g = 8.2206;
constexpr double kA2p2s = 8.78e-7;
constexpr double kA2s2p = 1.597e-9;
// src/M1Closure.jl:36-41
constexpr double kFmin = 1e-10;
constexpr double kFmax = 1.0 - 1e-10;
constexpr double kJeps = 1e-60;
constexpr double kHeps = 1e-100;
// src/FreqFactors.jl:16-18
constexpr double kPmin = 1e-3;
constexpr double kPmax = 40.0;
// src/UpdateLyaJandH.jl:43
constexpr double kEpsActive = 1e-10;

template <typename R> struct Num;
template <> struct Num<double> {
    static __device__ __forceinline__ double third() { return 1.0 / 3.0; }
    static __device__ __forceinline__ double fmin() { return kFmin; }
    static __device__ __forceinline__ double fmax() { return kFmax; }
    static __device__ __forceinline__ double tiny() { return 1e-300; }
};
template <> struct Num<float> {
    static __device__ __forceinline__ float third() { return 1.0f / 3.0f; }
    static __device__ __forceinline__ float fmin() { return 1e-10f; }
    static __device__ __forceinline__ float fmax() { return 1.0f - 1e-7f; }
    static __device__ __forceinline__ float tiny() { return 1e-37f; }
};

// Square root. FP64: the IEEE square root. FP32: the hardware's approximate square root alone
// (PTX sqrt.approx.ftz.f32, relative error within 2^-23 over the normal range); the IEEE-rounded
// FP32 root costs a refinement sequence with special-case branches on the transcendental unit,
// which the FP32 advection keeps 40 % busy (mixed advection at 256^2 x 64, 32 rows per tile:
// 0.225 -> 0.207 ms; after 2000 steps the mixed form's M_F, edge spectrum and J differ from
// FP64 by 6.1e-7, 2.6e-7 and 1.5e-6 against 5.9e-7, 2.6e-7 and 1.7e-6 with the IEEE root).
// A subnormal argument is flushed, so its root is 0: the callers that divide by a root treat
// a zero root as a zero vector (the non-flushing form, sqrt.approx.f32, costs more than the
// IEEE root here).
__device__ __forceinline__ double rsq(double x) { return sqrt(x); }
__device__ __forceinline__ float rsq(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Reciprocal 1 / y. FP64: the hardware's approximate reciprocal (PTX rcp.approx.ftz.f64)
// refined by one third-order step of the Newton-Raphson family for 1/y: with e = 1 - y x,
// 1/y = x / (1 - e) = x (1 + e + e^2 + ...), so x <- x + x (e + e^2) cubes the relative error
// (Markstein, IBM J. Res. Dev. 34 (1990) 111-119), in three fused multiply-adds where two
// quadratic steps take four. No special-case branches: the callers divide by positive normal
// numbers whose reciprocals are normal. FP32: the hardware's approximate reciprocal alone (PTX
// rcp.approx.ftz.f32, relative error within 2^-23 over the normal range, subnormals flushed),
// one instruction in place of the IEEE division's refinement sequence; the FP32 arithmetic of
// the mixed and FP32-storage forms already carries a 2^-24 rounding per operation.
template <typename R> __device__ __forceinline__ R rcp(R y);
template <> __device__ __forceinline__ double rcp<double>(double y) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(y));
    const double e = fma(-y, x, 1.0);
    return fma(x, fma(e, e, e), x);
}
template <> __device__ __forceinline__ float rcp<float>(float y) {
    float x;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(y));
    return x;
}

// Reciprocal square root 1 / sqrt(x) for FP64 arithmetic and x >= DBL_MIN: the hardware's
// approximate reciprocal square root (PTX rsqrt.approx.ftz.f64) refined by one third-order
// step: with e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2/8 + ...), so
// y <- y + y e (1/2 + 3 e / 8) cubes the relative error (Markstein, IBM J. Res. Dev. 34 (1990)
// 111-119), in two multiplies and three fused multiply-adds where two quadratic steps take
// seven operations. x * rsqrt_nr(x) is then sqrt(x) to about an ulp, and one such root gives both a
// length and its reciprocal where the IEEE root needs a root and a reciprocal.
__device__ __forceinline__ double rsqrt_nr(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}
constexpr double kDblMinNormal = 2.2250738585072014e-308;

// Reciprocal square root 1 / sqrt(x) for FP32 arithmetic: the hardware's approximation alone
// (PTX rsqrt.approx.ftz.f32, relative error within 2^-22.9 over the normal range; a subnormal
// or zero argument gives +inf, so callers check x against FLT_MIN first). One transcendental
// operation gives both a length, x * rsqf(x), and its reciprocal.
__device__ __forceinline__ float rsqf(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float kFltMinNormal = 1.17549435e-38f;

// MinMod, src/ConstantsAndFunctions.jl:1571-1582. FP64: the smaller in magnitude, or zero where the
// sign bits differ, which is the reference's a b <= 0 without its product (a b underflows to zero
// only for slopes below 1e-154, whose sum with anything is that thing).
template <typename R>
__device__ __forceinline__ R minmod(R a, R b) {
    if constexpr (sizeof(R) == 8) {
        const R m = fabs(a) < fabs(b) ? a : b;
        return (__double2hiint(a) ^ __double2hiint(b)) < 0 ? R(0) : m;
    } else {
        return (a * b <= R(0)) ? R(0) : (fabs(a) < fabs(b) ? a : b);
    }
}

// Levermore closure chi(f), src/M1Closure.jl:28-33, evaluated as (5 - 2 sqrt(4 - 3 f^2)) / 3,
// the same function (multiply numerator and denominator by 5 - 2 sqrt(4 - 3 f^2): the
// denominator becomes 3 (3 + 4 f^2)), with one square root and no reciprocal; 5 - 2 sqrt(..)
// >= 1 for f <= 1, so at most a factor 4 cancels (f = 0: 5 - 4). In FP64 the root of
// t = 4 - 3 f^2, in [1, 4], is t * rsqrt_nr(t), folded into 5 - 2 s by one fused multiply-add.
template <typename R>
__device__ __forceinline__ R chi_L84(R f) {
    R f2 = f * f;
    R t = R(4) - R(3) * f2;
    if constexpr (sizeof(R) == 4)
        return (R(5) - R(2) * rsq(t)) * R(1.0f / 3.0f);
    else
        return fma(-2.0 * t, rsqrt_nr(t), 5.0) * (1.0 / 3.0);
}

// 1 / |v| from |v|^2 for a vector whose length may vanish: the reciprocal root of s + tiny, so
// that a zero vector gets a zero direction with no test (s is far above tiny wherever a direction
// matters: |f| >= 1e-10 in the closure, and tiny is 1e-300 in FP64 and FLT_MIN in FP32).
__device__ __forceinline__ double inv_len(double s) { return rsqrt_nr(s + 1e-300); }
__device__ __forceinline__ float inv_len(float s) { return rsqf(s + kFltMinNormal); }

// The two coefficients of the Eddington tensor D = a I + b n n (src/M1Closure.jl:46-119) at reduced
// flux f <= fmax: with s = sqrt(4 - 3 f^2), chi = (5 - 2 s) / 3 and the reference's (1 - chi) / 2 and
// (3 chi - 1) / 2 are (s - 1) / 3 and 2 - s. At f below fmin (1e-10) s rounds to 2: a = 1/3, b = 0, the
// isotropic tensor the reference switches to there, so no branch is needed; and since n is a unit
// vector wherever b is not 0, D_phiphi = 1 - D_rr - D_ZZ is a.
template <typename R>
__device__ __forceinline__ void eddington_ab(R f, R &a, R &b) {
    const R t = R(4) - R(3) * (f * f);
    R s;
    if constexpr (sizeof(R) == 4) s = rsq(t);
    else s = t * rsqrt_nr(t);
    a = (s - R(1)) * Num<R>::third();
    b = R(2) - s;
}

// D : grad u (D_colon_grad_u_Cylindrical, src/ConstantsAndFunctions.jl:883-895) with the closure of
// a cell's (J, H_r, H_Z) (Compute_D_Edd, src/M1Closure.jl:46-83): a (g0 + g3 + g4) + b (n_r (n_r g0 +
// n_Z g12) + n_Z^2 g3), g0 = du_r/dr, g12 = du_r/dZ + du_Z/dr, g3 = du_Z/dZ, tr = g0 + g3 + u_r/r.
// jeps / heps2 are the floors in storage units: at or below them the tensor is isotropic.
template <typename R>
__device__ __forceinline__ R work_rate(R J, R Hr, R HZ, R jeps, R heps2, R g0, R g12, R g3, R tr) {
    const R H2 = Hr * Hr + HZ * HZ;
    bool on = J > jeps && H2 > heps2;
    // |H|^2 below the type's normal range counts as no direction
    if constexpr (sizeof(R) == 4) on = on && H2 >= kFltMinNormal;
    else on = on && H2 >= kDblMinNormal;
    R iH;
    if constexpr (sizeof(R) == 4) iH = rsqf(on ? H2 : R(1));
    else iH = rsqrt_nr(on ? H2 : R(1));
    R f = (H2 * iH) * rcp<R>(on ? J : R(1));
    f = on ? (f < Num<R>::fmax() ? f : Num<R>::fmax()) : R(0);
    R a, b;
    eddington_ab(f, a, b);
    const R nr = Hr * iH, nZ = HZ * iH;
    return a * tr + b * (nr * (nr * g0 + nZ * g12) + (nZ * nZ) * g3);
}

// Compute_D_Edd_from_f_n, src/M1Closure.jl:91-119
template <typename R>
__device__ __forceinline__ void D_from_f_n(R f, R nr, R nZ, R &Drr, R &DZZ, R &DrZ) {
    if (f > Num<R>::fmin()) {
        f = f < Num<R>::fmax() ? f : Num<R>::fmax();
        R chi = chi_L84(f);
        R a = (R(1) - chi) * R(0.5);
        R b = (R(3) * chi - R(1)) * R(0.5);
        R b_nr = b * nr;
        Drr = a + b_nr * nr;
        DZZ = a + b * nZ * nZ;
        DrZ = b_nr * nZ;
    } else {
        Drr = Num<R>::third(); DZZ = Num<R>::third(); DrZ = R(0);
    }
}

// Compute_D_Edd, src/M1Closure.jl:46-83. jeps / heps2 are the floors in storage units.
template <typename R>
__device__ __forceinline__ void D_edd(R Hr, R HZ, R J, R jeps, R heps2, R &Drr, R &DZZ, R &DrZ) {
    R H2 = Hr * Hr + HZ * HZ;
    const R fmin2 = Num<R>::fmin() * Num<R>::fmin();
    if (J <= jeps || H2 <= heps2 || H2 <= fmin2 * J * J) {
        Drr = Num<R>::third(); DZZ = Num<R>::third(); DrZ = R(0);
        return;
    }
    R Hmag, inv_H;
    // one reciprocal square root gives |H| and 1/|H|; |H|^2 below the type's normal range
    // counts as no direction
    if constexpr (sizeof(R) == 4) {
        if (!(H2 >= kFltMinNormal)) {
            Drr = Num<R>::third(); DZZ = Num<R>::third(); DrZ = R(0);
            return;
        }
        inv_H = rsqf(H2);
    } else {
        if (!(H2 >= kDblMinNormal)) {
            Drr = Num<R>::third(); DZZ = Num<R>::third(); DrZ = R(0);
            return;
        }
        inv_H = rsqrt_nr(H2);
    }
    Hmag = H2 * inv_H;
    R f = Hmag * rcp<R>(J);
    f = f < Num<R>::fmin() ? Num<R>::fmin() : (f > Num<R>::fmax() ? Num<R>::fmax() : f);
    R chi = chi_L84(f);
    R a = (R(1) - chi) * R(0.5);
    R b = (R(3) * chi - R(1)) * R(0.5);
    R nr = Hr * inv_H, nZ = HZ * inv_H;
    R b_nr = b * nr;
    Drr = a + b_nr * nr;
    DZZ = a + b * nZ * nZ;
    DrZ = b_nr * nZ;
}

// HLL_Eigenvalues, src/M1Closure.jl:273-296
template <typename R>
__device__ __forceinline__ void hll_eigen(R f, R mu, R &l1, R &l3) {
    f = f < Num<R>::fmin() ? Num<R>::fmin() : (f > Num<R>::fmax() ? Num<R>::fmax() : f);
    mu = mu < R(-1) ? R(-1) : (mu > R(1) ? R(1) : mu);
    R f2 = f * f, mu2 = mu * mu, muf = mu * f;
    R t = R(4) - R(3) * f2;
    // t >= 1 (f <= fmax < 1): one reciprocal square root gives the root and its reciprocal
    R inv_sq;
    if constexpr (sizeof(R) == 4) inv_sq = rsqf(t);
    else inv_sq = rsqrt_nr(t);
    const R sq = t * inv_sq;
    R g = R(2) / R(3) * (R(4) - R(3) * f2 - sq) + R(2) * mu2 * (R(2) - f2 - sq);
    R fac = rsq(g > R(0) ? g : R(0));
    R x1 = (muf - fac) * inv_sq, x3 = (muf + fac) * inv_sq;
    l1 = x1 < R(-1) ? R(-1) : (x1 > R(1) ? R(1) : x1);
    l3 = x3 < R(-1) ? R(-1) : (x3 > R(1) ? R(1) : x3);
}

// One cell of the reconstruction stencil.
template <typename R> struct Cell { R J, Hr, HZ; };

// ReconstructInterface output, src/AdvectJandH.jl:359-473 (the adjoint's replay keeps it whole)
template <typename R> struct Recon {
    R J_L, J_R, Hr_L, Hr_R, HZ_L, HZ_R, tau_L, tau_R, f_L, f_R, nr_L, nr_R, nZ_L, nZ_R;
};

// A stencil cell in the form ReconstructInterface works on: J and the reduced flux
// f = H / max(J, Jeps) (src/AdvectJandH.jl:373-386). Computing it once per cell lets every
// face that uses the cell share one reciprocal.
template <typename R> struct CellF { R J, fr, fZ; };

template <typename R>
__device__ __forceinline__ CellF<R> cell_f(R J, R Hr, R HZ, R jeps) {
    R iJ = rcp<R>(J > jeps ? J : jeps);
    CellF<R> c;
    c.J = J; c.fr = Hr * iJ; c.fZ = HZ * iJ;
    return c;
}

// One side of an interface: the reconstructed J (floored) and reduced flux, its flux vector after the
// causality limit |f| <= 1, and the second moments J D along the face's normal (Kn), across it (Kt)
// and along phi (kp). ZDIR: the normal is Z, else r.
template <typename R> struct Side { R J, Hr, HZ, Kn, Kt, kp, f, mu; };
template <typename R, bool ZDIR>
__device__ __forceinline__ Side<R> side_of(R J, R fr, R fZ) {
    Side<R> o;
    o.J = J;
    const R s = fr * fr + fZ * fZ;
    const R i = inv_len(s);                    // one reciprocal root gives |f| and the direction
    const R f = s * i, nr = fr * i, nZ = fZ * i;
    R a, b;
    eddington_ab(f < Num<R>::fmax() ? f : Num<R>::fmax(), a, b);
    o.f = f < R(1) ? f : R(1);
    const R fJ = o.f * J;
    o.Hr = nr * fJ;
    o.HZ = nZ * fJ;
    o.mu = ZDIR ? nZ : nr;
    o.kp = a * J;
    const R bn = (b * J) * o.mu;
    o.Kn = o.kp + bn * o.mu;
    o.Kt = bn * (ZDIR ? nr : nZ);
    return o;
}

// One interface between cells ci and cp1 (outer stencil cells cm1 and cp2): ReconstructInterface
// (src/AdvectJandH.jl:359-473), the closures of both sides, GetFluxGLF / GetFluxHLL (:81-118, 155-204)
// with the wave speeds of M1WaveSpeeds_r/Z (src/M1Closure.jl:301-326), and the advection flux of
// u*/c = uc (:276-282). iv = {dL, dR, inv_i_im1, inv_ip1_i, inv_ip2_ip1}. kL / kR: K_phiphi of the two
// sides. The diffusion-limit weight 1 - eps = tau^2 / (0.2 + tau + tau^2) is formed as that product and
// cancelled against the 1 / tau of the diffusive flux: one reciprocal, and none of the rounding of
// 1 - eps divided by a small tau. No branches (the reference's floors and limits are selects), so
// the two faces a thread computes can be scheduled together (FP64 advection at 256^2 x 64, packed
// tiles: 258 -> 205 us).
template <typename R, int FLUX, bool ZDIR>
__device__ __forceinline__ void face_flux(const CellF<R> &cm1, const CellF<R> &ci, const CellF<R> &cp1,
                                          const CellF<R> &cp2, const R iv[5], R aF_i, R aF_ip1, R uc, R jeps, R *F,
                                          R &kL, R &kR, R &JR, R &HZR) {
    const R dL = iv[0], dR = iv[1];
    const R dJc = (cp1.J - ci.J) * iv[3], dfrc = (cp1.fr - ci.fr) * iv[3], dfZc = (cp1.fZ - ci.fZ) * iv[3];
    const R J_L = ci.J + minmod((ci.J - cm1.J) * iv[2], dJc) * dL;
    const R J_R = cp1.J - minmod((cp2.J - cp1.J) * iv[4], dJc) * dR;
    const R fr_L = ci.fr + minmod((ci.fr - cm1.fr) * iv[2], dfrc) * dL;
    const R fr_R = cp1.fr - minmod((cp2.fr - cp1.fr) * iv[4], dfrc) * dR;
    const R fZ_L = ci.fZ + minmod((ci.fZ - cm1.fZ) * iv[2], dfZc) * dL;
    const R fZ_R = cp1.fZ - minmod((cp2.fZ - cp1.fZ) * iv[4], dfZc) * dR;
    const Side<R> L = side_of<R, ZDIR>(J_L > jeps ? J_L : jeps, fr_L, fZ_L);
    const Side<R> Q = side_of<R, ZDIR>(J_R > jeps ? J_R : jeps, fr_R, fZ_R);
    const R tau = aF_i * dL + aF_ip1 * dR;
    R num = R(0.2) + tau, tt = tau;
    if constexpr (sizeof(R) == 4) {
        // tau^2 leaves FP32's range (and its reciprocal is flushed from 9e18 on): beyond 1e18, where 0.2 and 1
        // are lost beside tau, both weights are 1 / (1 + tau), of terms that stay in range up to FLT_MAX
        const bool deep = tau > R(1e18);
        num = deep ? R(0.125) : num;
        tt = deep ? R(0.125) : tau;
    }
    const R r = rcp<R>(num + tt * tau);
    const R eps = num * r, te = tt * r;
    const R diff = -Num<R>::third() * (cp1.J - ci.J) * te;
    const R Kr_L = ZDIR ? L.Kt : L.Kn, Kr_R = ZDIR ? Q.Kt : Q.Kn, KZ_L = ZDIR ? L.Kn : L.Kt, KZ_R = ZDIR ? Q.Kn : Q.Kt;
    const R Hn_L = ZDIR ? L.HZ : L.Hr, Hn_R = ZDIR ? Q.HZ : Q.Hr;
    const bool up = uc < R(0);
    const R aJ = uc * (up ? Q.J : L.J), aHr = uc * (up ? Q.Hr : L.Hr), aHZ = uc * (up ? Q.HZ : L.HZ);
    if (FLUX == 0) {
        const R he = R(0.5) * eps;
        F[0] = he * ((Hn_L + Hn_R) - (Q.J - L.J)) + (diff + aJ);
        F[1] = R(0.5) * (Kr_L + Kr_R) - he * (Q.Hr - L.Hr) + aHr;
        F[2] = R(0.5) * (KZ_L + KZ_R) - he * (Q.HZ - L.HZ) + aHZ;
    } else {
        R l1L, l3L, l1R, l3R;
        hll_eigen<R>(L.f, L.mu, l1L, l3L);
        hll_eigen<R>(Q.f, Q.mu, l1R, l3R);
        R SR = l3L > l3R ? l3L : l3R, SL = l1L < l1R ? l1L : l1R;
        SR = SR > R(0) ? SR : R(0);
        SL = SL < R(0) ? SL : R(0);
        const R dS = SR - SL;
        const R w = eps * rcp<R>(dS > Num<R>::tiny() ? dS : Num<R>::tiny());
        const R SRSL = SR * SL;
        const R hom = R(0.5) * (tau * te);
        F[0] = w * (SR * Hn_L - SL * Hn_R + SRSL * (Q.J - L.J)) + (diff + aJ);
        F[1] = w * (SR * Kr_L - SL * Kr_R + SRSL * (Q.Hr - L.Hr)) + hom * (Kr_L + Kr_R) + aHr;
        F[2] = w * (SR * KZ_L - SL * KZ_R + SRSL * (Q.HZ - L.HZ)) + hom * (KZ_L + KZ_R) + aHZ;
    }
    kL = L.kp;
    kR = Q.kp;
    JR = Q.J;
    HZR = Q.HZ;
}

// Compute_K_phiphi_InnerAxis, src/AdvectJandH.jl:499-522
template <typename R>
__device__ __forceinline__ R k_phiphi_axis(R J, R HZ, R jeps) {
    J = J > jeps ? J : jeps;
    R fZ = HZ * rcp<R>(J);
    fZ = fZ < R(-1) ? R(-1) : (fZ > R(1) ? R(1) : fZ);
    R f = fabs(fZ);
    R nZ = f > R(0) ? (fZ > R(0) ? R(1) : R(-1)) : R(0);
    R Drr, DZZ, DrZ;
    D_from_f_n<R>(f, R(0), nZ, Drr, DZZ, DrZ);
    R k = R(1) - Drr - DZZ;
    k = k < R(0) ? R(0) : (k > R(1) ? R(1) : k);
    return k * J;
}

// D_colon_grad_u_Cylindrical, src/ConstantsAndFunctions.jl:883-895
template <typename R>
__device__ __forceinline__ R d_colon_grad_u(R Drr, R DrZ, R DZZ, R a, R b, R c, R d, R e) {
    R Dpp = R(1) - Drr - DZZ;
    Dpp = Dpp > R(0) ? Dpp : R(0);
    return Drr * a + DrZ * (b + c) + DZZ * d + Dpp * e;
}

// exp(x) for |x| <= 40 in FP64 by the table-driven method of P. T. P. Tang (ACM Trans. Math.
// Softw. 15 (1989) 144-157): x = (32 m + j) ln2/32 + r with |r| <= ln2/64, exp(x) = 2^m 2^(j/32)
// e^r. The 32 values 2^(j/32) are correctly rounded (generated in 80-digit decimal arithmetic),
// e^r - 1 is its Taylor polynomial to degree 6 (truncation below 4e-18 relative) and the
// result is 2^m (T + T (e^r - 1)) with one rounding: within about an ulp. round(32 x / ln2)
// comes out of one fused multiply-add with 1.5 * 2^52 (its low bits then hold the integer);
// ln2/32 is split in a 40-bit head, whose products with |32 x / ln2| < 2^13 are exact, and a
// tail. `tab` is kExp2Tab, or a copy of it in shared memory.
static __constant__ double kExp2Tab[32] = {
    0x1.0000000000000p+0, 0x1.059b0d3158574p+0, 0x1.0b5586cf9890fp+0, 0x1.11301d0125b51p+0,
    0x1.172b83c7d517bp+0, 0x1.1d4873168b9aap+0, 0x1.2387a6e756238p+0, 0x1.29e9df51fdee1p+0,
    0x1.306fe0a31b715p+0, 0x1.371a7373aa9cbp+0, 0x1.3dea64c123422p+0, 0x1.44e086061892dp+0,
    0x1.4bfdad5362a27p+0, 0x1.5342b569d4f82p+0, 0x1.5ab07dd485429p+0, 0x1.6247eb03a5585p+0,
    0x1.6a09e667f3bcdp+0, 0x1.71f75e8ec5f74p+0, 0x1.7a11473eb0187p+0, 0x1.82589994cce13p+0,
    0x1.8ace5422aa0dbp+0, 0x1.93737b0cdc5e5p+0, 0x1.9c49182a3f090p+0, 0x1.a5503b23e255dp+0,
    0x1.ae89f995ad3adp+0, 0x1.b7f76f2fb5e47p+0, 0x1.c199bdd85529cp+0, 0x1.cb720dcef9069p+0,
    0x1.d5818dcfba487p+0, 0x1.dfc97337b9b5fp+0, 0x1.ea4afa2a490dap+0, 0x1.f50765b6e4540p+0};
__device__ __forceinline__ double exp_tab(double x, const double *tab) {
    constexpr double kShift = 0x1.8p52, kInvL = 0x1.71547652b82fep+5;
    constexpr double kLhi = 0x1.62e42fefa2000p-6, kLlo = 0x1.9ef35793c7673p-46;
    const double t = fma(x, kInvL, kShift);
    const int N = __double2loint(t);
    const double Nd = t - kShift;
    double r = fma(-Nd, kLhi, x);
    r = fma(-Nd, kLlo, r);
    double q = fma(r, 1.0 / 720.0, 1.0 / 120.0);
    q = fma(q, r, 1.0 / 24.0);
    q = fma(q, r, 1.0 / 6.0);
    q = fma(q, r, 0.5);
    q = fma(q, r, 1.0);
    q *= r;
    const double T = tab[N & 31];
    // times 2^m by adding m to the exponent (|m| <= 58: no range to leave)
    const double e = fma(T, q, T);
    return __hiloint2double(__double2hiint(e) + ((N & ~31) << 15), __double2loint(e));
}

// The Peclet number clamped to [-Pmax, Pmax] (src/FreqFactors.jl:248-250) on its high word: Pmax = 40
// has a zero low word, so |P| >= 40 shows there (a NaN clamps to +-40, as through fmin/fmax).
__device__ __forceinline__ double clamp_P(double P) {
    static_assert(kPmax == 40.0, "the high word of Pmax");
    const int hi = __double2hiint(P);
    const bool big = (hi & 0x7fffffff) >= 0x40440000;
    return __hiloint2double(big ? (hi & 0x80000000) | 0x40440000 : hi, big ? 0 : __double2loint(P));
}

// OneMinusphi_L_and_chi_L / OneMinusphi_R_and_chi_R, src/FreqFactors.jl:54-133, in FP64.
// Every caller clamps P to [-Pmax, Pmax] first (src/FreqFactors.jl:248-250), so the reference's
// |P| >= Pmax branches only ever see P = +-Pmax, where they return exp(-+Pmax) and
// (1 - exp(-+Pmax)) / +-Pmax: the general expression at that P. What remains is the choice
// between the exponential and the second-order Taylor form below |P| = Pmin, taken here by a
// select on values the warp computes for every lane, so lanes of one warp never take
// different paths (at P = 0 the unused general value is not finite; the select drops it).
// The exponentials are exp_tab's (|P| <= Pmax = 40) with the table at `tab`.
__device__ __forceinline__ void omphi_L(double P, double &omp, double &chi, const double *tab) {
    const double e = exp_tab(-P, tab);
    const double x = (1.0 - e) * rcp<double>(P);
    const bool tay = fabs(P) < kPmin;
    omp = tay ? 1.0 - P + 0.5 * (P * P) : e;
    chi = tay ? 1.0 - 0.5 * P : x;
}
__device__ __forceinline__ void omphi_R(double P, double &omp, double &chi, const double *tab) {
    const double e = exp_tab(P, tab);
    const double x = (1.0 - e) * rcp<double>(P);
    const bool tay = fabs(P) < kPmin;
    omp = tay ? 1.0 + P + 0.5 * (P * P) : e;
    chi = tay ? -1.0 - 0.5 * P : x;
}
// Both of the above at once for the same P (used for P_k, which needs phi^L and phi^R):
// one exponential and one reciprocal of P serve the two.
__device__ __forceinline__ void omphi_LR(double P, double &oL, double &xL, double &oR, double &xR,
                                         const double *tab) {
    const double e = exp_tab(-P, tab);
    const double ie = rcp<double>(e);
    const double iP = rcp<double>(P);
    const bool tay = fabs(P) < kPmin;
    const double h = 0.5 * (P * P);
    oL = tay ? 1.0 - P + h : e;
    xL = tay ? 1.0 - 0.5 * P : (1.0 - e) * iP;
    oR = tay ? 1.0 + P + h : ie;
    xR = tay ? -1.0 - 0.5 * P : (1.0 - ie) * iP;
}
// Thermal velocity, Doppler width, Voigt parameter (src/ConstantsAndFunctions.jl:282-314)
__host__ __device__ __forceinline__ double compute_b(double T) { return sqrt(2.0 * kKBoltz / kMH) * sqrt(T); }
__host__ __device__ __forceinline__ double compute_dnuD(double T) { return compute_b(T) * (kNuLya / kC); }
__host__ __device__ __forceinline__ double compute_a(double T) {
    return (kALya / (kFourPi * kNuLya * 1.0 / kC)) / compute_b(T);
}

}  // namespace lyd
