// Device physics of the finite-volume path: equation of state, TVD limiters, WENO-Z reconstruction and the
// HLLC-family Riemann solvers, written for sm_100a.
//
// Every function keeps the operation order of the reference (Fenice, cpp/include/fv/Core.hpp,
// cpp/include/fv/Schemes.hpp, cpp/src/Schemes.cpp) and the library is compiled with --fmad=false, so the FP64
// instantiation gives the reference's bits: IEEE-rounded add, mul, div and sqrt, no contraction into fused
// multiply-adds. std::max / std::min are the ternaries `a < b ? b : a` / `b < a ? b : a` (fmax would pick the
// other operand for NaN and signed zeros).
//
// The functions are templates over the arithmetic type T (double: the plain form; float: the mixed form) and
// over the dimension: a planar (2-D) state has no z-momentum, and every term the reference adds for it is
// exactly +0 there, so dropping it gives the same bits.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace fvg {

constexpr int kFirstOrder = 0, kMuscl = 1, kWeno3 = 2, kWeno5 = 3;
constexpr int kMinmod = 0, kVanLeer = 1, kMC = 2, kKoren = 3;
constexpr int kHLLC = 0, kLowMach = 1;
constexpr int kIdeal = 0, kStiffened = 1;

template <typename T> struct Num;
template <> struct Num<double> {
    static constexpr double eos_eps = 1e-10;   // Core.hpp:169
    static constexpr double denom_eps = 1e-14; // Schemes.cpp:64
    static constexpr double mach_eps = 1e-12;  // Schemes.cpp:66
    static constexpr double weno_floor = 1e-300;
};
template <> struct Num<float> {
    static constexpr float eos_eps = 1e-10f;
    static constexpr float denom_eps = 1e-14f;
    static constexpr float mach_eps = 1e-12f;
    static constexpr float weno_floor = 1e-30f;  // 1e-300 is below the float range
};

template <typename T> __host__ __device__ __forceinline__ T vmax(T a, T b) { return (a < b) ? b : a; }
template <typename T> __host__ __device__ __forceinline__ T vmin(T a, T b) { return (b < a) ? b : a; }

// The equation of state (Core.hpp:173-238): ideal gas p = (gamma-1) rho e, stiffened gas p + gamma p_inf = (gamma-1) rho e.
template <typename T> struct Eos {
    int type;
    T gamma, p_inf;
    T rgm1;   // 1 / (gamma - 1), correctly rounded (0: divide); set by set_eos
};
// The gas of a run, on the host. The reciprocal is left out where Markstein's theorem does not cover it (a divisor whose
// significand is all ones).
inline void set_eos(Eos<double>& e, int type, double gamma, double p_inf) {
    e.type = type;
    e.gamma = gamma;
    e.p_inf = p_inf;
    const double d = gamma - 1.0;
    int ex = 0;
    const double m = frexp(d, &ex);
    const bool covered = d > 1e-100 && d < 1e100 && m != 1.0 - 0x1p-53;
    e.rgm1 = covered ? 1.0 / d : 0.0;
}

// State of NV components: [rho, rho u, rho v, rho E (, rho w)] or primitive [rho, u, v, p (, w)].
template <typename T, int NV> struct St {
    T v[NV];
    __device__ __forceinline__ T& operator[](int q) { return v[q]; }
    __device__ __forceinline__ const T& operator[](int q) const { return v[q]; }
};

// x / (gamma - 1), correctly rounded as the division is: the product with the rounded reciprocal, corrected twice by its
// exact residual (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990: with the
// correctly rounded reciprocal, one correction of a quotient within one unit in the last place gives the rounded quotient;
// the first correction brings the product there). Five dependent operations and no branch taken instead of a division; a
// zero, an infinity, a NaN or a quotient near the limits of the range is divided.
__device__ __forceinline__ double over_gm1(const Eos<double>& e, double x) {
    const double d = e.gamma - 1.0;
    const double q0 = __dmul_rn(x, e.rgm1);
    const unsigned ex = ((unsigned)__double2hiint(q0) >> 20) & 0x7ffu;
    if (ex - 123u > 1800u) return x / d;   // |q0| outside 2^-900 .. 2^900 (or no reciprocal: q0 = 0)
    const double q1 = __fma_rn(__fma_rn(-d, q0, x), e.rgm1, q0);
    return __fma_rn(__fma_rn(-d, q1, x), e.rgm1, q1);
}
template <typename T> __device__ __forceinline__ T over_gm1(const Eos<T>& e, T x) { return x / (e.gamma - T(1)); }

template <typename T> __device__ __forceinline__ T internal_energy(const Eos<T>& e, T p) {
    return e.type == kIdeal ? over_gm1(e, p) : over_gm1(e, p + e.gamma * e.p_inf);
}
template <typename T> __device__ __forceinline__ T pressure(const Eos<T>& e, T rho_e) {
    return e.type == kIdeal ? (e.gamma - T(1)) * rho_e : (e.gamma - T(1)) * rho_e - e.gamma * e.p_inf;
}

// prim_to_cons (Core.hpp:209-215)
template <typename T, int NV> __device__ __forceinline__ St<T, NV> p2c(const Eos<T>& e, const St<T, NV>& W) {
    St<T, NV> U;
    const T rho = W[0], u = W[1], v = W[2], p = W[3];
    T ke;
    if constexpr (NV == 5) {
        const T w = W[4];
        ke = T(0.5) * rho * (u * u + v * v + w * w);
        U[4] = rho * w;
    } else {
        ke = T(0.5) * rho * (u * u + v * v);
    }
    const T en = internal_energy(e, p);
    U[0] = rho;
    U[1] = rho * u;
    U[2] = rho * v;
    U[3] = en + ke;
    return U;
}

// cons_to_prim (Core.hpp:218-227); inv receives 1 / rho of the floored density
template <typename T, int NV> __device__ __forceinline__ St<T, NV> c2p(const Eos<T>& e, const St<T, NV>& U, T& inv) {
    St<T, NV> W;
    const T rho = vmax(U[0], Num<T>::eos_eps);
    inv = T(1) / rho;
    const T u = U[1] * inv, v = U[2] * inv;
    T e_kin;
    if constexpr (NV == 5) {
        const T w = U[4] * inv;
        e_kin = T(0.5) * rho * (u * u + v * v + w * w);
        W[4] = w;
    } else {
        e_kin = T(0.5) * rho * (u * u + v * v);
    }
    const T p = pressure(e, U[3] - e_kin);
    W[0] = rho;
    W[1] = u;
    W[2] = v;
    W[3] = vmax(p, Num<T>::eos_eps);
    return W;
}
template <typename T, int NV> __device__ __forceinline__ St<T, NV> c2p(const Eos<T>& e, const St<T, NV>& U) {
    T inv;
    return c2p(e, U, inv);
}

// sound_speed_inv (Core.hpp:234-237)
template <typename T> __device__ __forceinline__ T sound_speed_inv(const Eos<T>& e, T p, T inv_rho) {
    if (e.type == kIdeal) return sqrt(e.gamma * vmax(p, Num<T>::eos_eps) * inv_rho);
    return sqrt(e.gamma * (p + e.p_inf) * inv_rho);
}
// sound_speed (Core.hpp:229-232)
template <typename T> __device__ __forceinline__ T sound_speed(const Eos<T>& e, T p, T rho) {
    if (e.type == kIdeal) return sqrt(e.gamma * vmax(p, Num<T>::eos_eps) / vmax(rho, Num<T>::eos_eps));
    return sqrt(e.gamma * (p + e.p_inf) / vmax(rho, Num<T>::eos_eps));
}

template <typename T, int NV> __device__ __forceinline__ St<T, NV> round_trip(const Eos<T>& e, const St<T, NV>& U) {
    return p2c(e, c2p(e, U));
}

// ------------------------------------------------------------------ limiters (Schemes.hpp:93-117)
template <typename T> __device__ __forceinline__ T sgn(T x) { return (x > T(0)) ? T(1) : ((x < T(0)) ? T(-1) : T(0)); }
template <typename T> __device__ __forceinline__ T limiter(int l, T a, T b) {
    switch (l) {
    case kMinmod: return T(0.5) * (sgn(a) + sgn(b)) * vmin(fabs(a), fabs(b));
    case kVanLeer: {
        const T ab = a * b;
        return (ab > T(0)) ? T(2) * ab / (a + b) : T(0);
    }
    case kMC:
        if (!(a * b > T(0))) return T(0);
        return vmin(vmin(T(2) * fabs(a), T(0.5) * fabs(a + b)), T(2) * fabs(b)) * sgn(a);
    default:
        if (!(a * b > T(0))) return T(0);
        return fmin(fmin(T(2) * fabs(a), fabs(T(2) * a + b) / T(3)), T(2) * fabs(b)) * sgn(a);
    }
}

// ------------------------------------------------------------------ WENO-Z (Borges et al. 2008; Schemes.cpp:328-353)
// The value at the face on the right of c1 from (c0, c1, c2); eps relative to the mean square of the stencil.
template <typename T> __device__ __forceinline__ T weno3z(T c0, T c1, T c2, T eps_rel) {
    const T eps = eps_rel * (c0 * c0 + c1 * c1 + c2 * c2) * (T(1) / T(3)) + Num<T>::weno_floor;
    const T v0 = T(-0.5) * c0 + T(1.5) * c1, v1 = T(0.5) * c1 + T(0.5) * c2;
    const T b0 = (c1 - c0) * (c1 - c0), b1 = (c2 - c1) * (c2 - c1);
    const T tau = fabs(b0 - b1);
    const T a0 = (T(1) / T(3)) * (T(1) + tau / (b0 + eps)), a1 = (T(2) / T(3)) * (T(1) + tau / (b1 + eps));
    return (a0 * v0 + a1 * v1) / (a0 + a1);
}
// The value at the face on the right of c2 from (c0 .. c4).
template <typename T> __device__ __forceinline__ T weno5z(T c0, T c1, T c2, T c3, T c4, T eps_rel) {
    const T eps = eps_rel * (c0 * c0 + c1 * c1 + c2 * c2 + c3 * c3 + c4 * c4) * T(0.2) + Num<T>::weno_floor;
    const T p0 = (T(2) * c0 - T(7) * c1 + T(11) * c2) / T(6);
    const T p1 = (-c1 + T(5) * c2 + T(2) * c3) / T(6);
    const T p2 = (T(2) * c2 + T(5) * c3 - c4) / T(6);
    const T s0 = c0 - T(2) * c1 + c2, t0 = c0 - T(4) * c1 + T(3) * c2;
    const T s1 = c1 - T(2) * c2 + c3, t1 = c1 - c3;
    const T s2 = c2 - T(2) * c3 + c4, t2 = T(3) * c2 - T(4) * c3 + c4;
    const T b0 = (T(13) / T(12)) * s0 * s0 + T(0.25) * t0 * t0;
    const T b1 = (T(13) / T(12)) * s1 * s1 + T(0.25) * t1 * t1;
    const T b2 = (T(13) / T(12)) * s2 * s2 + T(0.25) * t2 * t2;
    const T tau = fabs(b0 - b2);
    const T a0 = T(0.1) * (T(1) + tau / (b0 + eps)), a1 = T(0.6) * (T(1) + tau / (b1 + eps)), a2 = T(0.3) * (T(1) + tau / (b2 + eps));
    return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2);
}
// Two FP32 values in one 64-bit register pair: sm_100a's packed add, multiply and FMA round each lane as the scalar
// operation does, at one issue slot for both.
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_get(F2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// the hardware's approximate reciprocal and square root (each within about one unit in the last place)
__device__ __forceinline__ float rcp_f(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_f(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ F2 f2_rcp(F2 v) {
    float a, b;
    f2_get(v, a, b);
    return f2(rcp_f(a), rcp_f(b));
}

// The single-precision WENO5-Z of the mixed form on packed operands (two variables, or the two values of a face): the value
// right of c from (a, b, c, d, e). Every product and sum is rounded by an explicit packed operation (FMAs placed by hand)
// and the candidates' common 1/6 folded into the last division, so that no compiler pass contracts it one way in one kernel
// and another way in the next: every kernel that solves a face gets the same bits.
__device__ __forceinline__ F2 weno5z_f2(F2 a, F2 b, F2 c, F2 d, F2 e, float eps_rel) {
    const auto k = [](float v) { return f2(v, v); };
    F2 ss = f2_mul(a, a);
    ss = f2_fma(b, b, ss);
    ss = f2_fma(c, c, ss);
    ss = f2_fma(d, d, ss);
    ss = f2_fma(e, e, ss);
    const F2 eps = f2_fma(f2_mul(k(eps_rel), ss), k(0.2f), k(Num<float>::weno_floor));
    const F2 p0 = f2_fma(k(11.0f), c, f2_fma(k(-7.0f), b, f2_mul(k(2.0f), a)));   // 6 x the three candidates
    const F2 p1 = f2_fma(k(2.0f), d, f2_fma(k(5.0f), c, f2_mul(k(-1.0f), b)));
    const F2 p2 = f2_fma(k(5.0f), d, f2_fma(k(2.0f), c, f2_mul(k(-1.0f), e)));
    const F2 s0 = f2_add(f2_fma(k(-2.0f), b, a), c), t0 = f2_fma(k(3.0f), c, f2_fma(k(-4.0f), b, a));
    const F2 s1 = f2_add(f2_fma(k(-2.0f), c, b), d), t1 = f2_fma(k(-1.0f), d, b);
    const F2 s2 = f2_add(f2_fma(k(-2.0f), d, c), e), t2 = f2_add(f2_fma(k(-4.0f), d, f2_mul(k(3.0f), c)), e);
    const F2 w = k(13.0f / 12.0f), h = k(0.25f);
    const F2 b0 = f2_fma(f2_mul(w, s0), s0, f2_mul(f2_mul(h, t0), t0));
    const F2 b1 = f2_fma(f2_mul(w, s1), s1, f2_mul(f2_mul(h, t1), t1));
    const F2 b2 = f2_fma(f2_mul(w, s2), s2, f2_mul(f2_mul(h, t2), t2));
    float dl, dr;
    f2_get(f2_fma(k(-1.0f), b2, b0), dl, dr);
    const F2 tau = f2(fabsf(dl), fabsf(dr));
    const F2 a0 = f2_mul(k(0.1f), f2_fma(tau, f2_rcp(f2_add(b0, eps)), k(1.0f)));
    const F2 a1 = f2_mul(k(0.6f), f2_fma(tau, f2_rcp(f2_add(b1, eps)), k(1.0f)));
    const F2 a2 = f2_mul(k(0.3f), f2_fma(tau, f2_rcp(f2_add(b2, eps)), k(1.0f)));
    const F2 num = f2_fma(a2, p2, f2_fma(a1, p1, f2_mul(a0, p0)));
    const F2 den = f2_mul(k(6.0f), f2_add(f2_add(a0, a1), a2));
    return f2_mul(num, f2_rcp(den));
}
// the linear fifth-order upwind value (0.1, 0.6, 0.3 of the candidates), likewise
__device__ __forceinline__ F2 lin5_f2(F2 a, F2 b, F2 c, F2 d, F2 e) {
    const auto k = [](float v) { return f2(v, v); };
    F2 s = f2_mul(k(2.0f), a);
    s = f2_fma(k(-13.0f), b, s);
    s = f2_fma(k(47.0f), c, s);
    s = f2_fma(k(27.0f), d, s);
    s = f2_fma(k(-3.0f), e, s);
    return f2_mul(s, k(1.0f / 60.0f));
}
// both values of a face of six cells: wl right of c2 from c0 .. c4, and its mirror image wr left of c3 from c5 .. c1
__device__ __forceinline__ void weno5z_pair(float c0, float c1, float c2, float c3, float c4, float c5, float eps_rel, float& wl, float& wr) {
    f2_get(weno5z_f2(f2(c0, c5), f2(c1, c4), f2(c2, c3), f2(c3, c2), f2(c4, c1), eps_rel), wl, wr);
}
__device__ __forceinline__ void lin5_pair(float c0, float c1, float c2, float c3, float c4, float c5, float& wl, float& wr) {
    f2_get(lin5_f2(f2(c0, c5), f2(c1, c4), f2(c2, c3), f2(c3, c2), f2(c4, c1)), wl, wr);
}

// ------------------------------------------------------------------ HLLC (Toro) with Einfeldt bounds (Schemes.cpp:116-200)
template <typename T> __device__ __forceinline__ T safe_denom(T x) { return copysign(vmax(fabs(x), Num<T>::denom_eps), x); }

// The velocity along `axis` of a primitive state (a choice, not an index: the axis may be a run-time value).
template <typename T, int NV> __device__ __forceinline__ T normal_velocity(const St<T, NV>& W, int axis) {
    return axis == 0 ? W[1] : (NV == 4 || axis == 1 ? W[2] : W[NV - 1]);
}
// One side's Euler flux along `axis`.
template <typename T, int NV>
__device__ __forceinline__ void hllc_side_flux(const St<T, NV>& W, T E, int axis, St<T, NV>& F) {
    constexpr int NA = NV == 5 ? 3 : 2;   // velocity components
    const T rho = W[0], p = W[3], Vn = normal_velocity(W, axis);
    F[0] = rho * Vn;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int m = a == 0 ? 1 : (a == 1 ? 2 : 4);
        const T f = rho * W[m] * Vn;
        F[m] = a == axis ? f + p : f;
    }
    F[3] = Vn * (rho * E + p);
}

// Whether the pressure jump |p_R - p_L| / min(p_L, p_R) may exceed the blend's threshold: false only where it is below it by
// more than its rounding (most faces, which are spared the division).
template <typename T> __device__ __forceinline__ bool may_blend(T p_L, T p_R, T shock_blend) {
    return !(fabs(p_R - p_L) < T(0.999) * shock_blend * vmin(p_L, p_R));
}
// F with the share phi of the upwind or HLL flux blended in.
template <typename T, int NV>
__device__ __forceinline__ void hll_blend(T S_L, T S_R, T phi, const St<T, NV>& FL, const St<T, NV>& FR, const St<T, NV>& UL, const St<T, NV>& UR,
                                          St<T, NV>& F) {
    if (S_L >= T(0)) {
#pragma unroll
        for (int q = 0; q < NV; ++q) F[q] = (T(1) - phi) * F[q] + phi * FL[q];
    } else if (S_R <= T(0)) {
#pragma unroll
        for (int q = 0; q < NV; ++q) F[q] = (T(1) - phi) * F[q] + phi * FR[q];
    } else {
        const T inv = T(1) / (S_R - S_L);
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const T fh = (S_R * FL[q] - S_L * FR[q] + S_L * S_R * (UR[q] - UL[q])) * inv;
            F[q] = (T(1) - phi) * F[q] + phi * fh;
        }
    }
}

// The flux along `axis` (0, 1, 2) from the primitive (floored) and conservative states of both sides; returns max(|S_L|, |S_R|).
// The reference forms both sides' fluxes and star states and then takes one of the four by the order of the waves; here the
// side is chosen first and only its flux and star state are formed, with the same operations (the same bits, three
// divisions instead of five).
template <typename T, int NV>
__device__ __forceinline__ T hllc_core(const St<T, NV>& WL, const St<T, NV>& WR, const St<T, NV>& UL, const St<T, NV>& UR, T inv_L,
                                       T inv_R, T c_L, T c_R, int axis, T shock_blend, St<T, NV>& F) {
    constexpr int NA = NV == 5 ? 3 : 2;   // velocity components
    const T rho_L = WL[0], p_L = WL[3];
    const T rho_R = WR[0], p_R = WR[3];
    const T Vn_L = normal_velocity(WL, axis), Vn_R = normal_velocity(WR, axis);
    const T S_L = vmin(Vn_L - c_L, Vn_R - c_R);
    const T S_R = vmax(Vn_L + c_L, Vn_R + c_R);
    const T num = rho_R * Vn_R * (S_R - Vn_R) - rho_L * Vn_L * (S_L - Vn_L) + p_L - p_R;
    const T den = rho_R * (S_R - Vn_R) - rho_L * (S_L - Vn_L);
    const T S_M = num / safe_denom(den);
    // flux selection by wave ordering: the last true one of the reference's four tests (a NaN speed leaves F = 0)
    const bool star_R = S_M < T(0) && S_R >= T(0), star_L = S_L < T(0) && S_M >= T(0);
    const bool right = S_R < T(0) || star_R;
    const bool star = !(S_R < T(0)) && (star_R || star_L);
    const bool none = !right && !star && !(S_L >= T(0));
    St<T, NV> W, U;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        W[q] = right ? WR[q] : WL[q];
        U[q] = right ? UR[q] : UL[q];
    }
    const T E = U[3] * (right ? inv_R : inv_L);
    hllc_side_flux(W, E, axis, F);
    if (star) {
        const T S = right ? S_R : S_L;
        const T rho = W[0], p = W[3], Vn = right ? Vn_R : Vn_L;
        const T den_star = safe_denom(S - S_M);
        const T den_p = safe_denom(S - Vn);
        const T f = rho * (S - Vn) / den_star;
        St<T, NV> Us;
        Us[0] = f;
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int m = a == 0 ? 1 : (a == 1 ? 2 : 4);
            Us[m] = f * (a == axis ? S_M : W[m]);
        }
        Us[3] = f * (E + (S_M - Vn) * (S_M + p / (rho * den_p)));
#pragma unroll
        for (int q = 0; q < NV; ++q) F[q] = F[q] + S * (Us[q] - U[q]);
    }
    if (none)
#pragma unroll
        for (int q = 0; q < NV; ++q) F[q] = T(0);
    if (shock_blend > T(0) && may_blend(p_L, p_R, shock_blend)) {
        const T s = fabs(p_R - p_L) / vmin(p_L, p_R);
        if (s > shock_blend) {
            const T phi = vmin((s - shock_blend) / shock_blend, T(1));
            St<T, NV> FL, FR;
            hllc_side_flux(WL, UL[3] * inv_L, axis, FL);
            hllc_side_flux(WR, UR[3] * inv_R, axis, FR);
            hll_blend(S_L, S_R, phi, FL, FR, UL, UR, F);
        }
    }
    return vmax(fabs(S_L), fabs(S_R));
}

// RiemannSolver::face_flux (Schemes.cpp:202-229): HLLC, or Thornber's low-Mach velocity-jump scaling then HLLC.
template <int RIEMANN, typename T, int NV>
__device__ __forceinline__ T face_flux(const Eos<T>& e, T shock_blend, const St<T, NV>& UL, const St<T, NV>& UR, int axis, St<T, NV>& F) {
    T inv_L, inv_R;
    St<T, NV> WL = c2p(e, UL, inv_L);
    St<T, NV> WR = c2p(e, UR, inv_R);
    const T c_L = sound_speed_inv(e, WL[3], inv_L);
    const T c_R = sound_speed_inv(e, WR[3], inv_R);
    if constexpr (RIEMANN == kHLLC) {
        return hllc_core(WL, WR, UL, UR, inv_L, inv_R, c_L, c_R, axis, shock_blend, F);
    } else {
        T mL2 = WL[1] * WL[1] + WL[2] * WL[2], mR2 = WR[1] * WR[1] + WR[2] * WR[2];
        if constexpr (NV == 5) {
            mL2 = mL2 + WL[4] * WL[4];
            mR2 = mR2 + WR[4] * WR[4];
        }
        const T M_L = sqrt(mL2) / (c_L + Num<T>::mach_eps);
        const T M_R = sqrt(mR2) / (c_R + Num<T>::mach_eps);
        const T z = vmin(vmax(vmax(M_L, M_R), T(1e-4)), T(1));
#pragma unroll
        for (int a = 0; a < (NV == 5 ? 3 : 2); ++a) {
            const int m = a == 0 ? 1 : (a == 1 ? 2 : 4);
            const T avg = T(0.5) * (WL[m] + WR[m]);
            const T half = T(0.5) * (WL[m] - WR[m]);
            WL[m] = avg + z * half;
            WR[m] = avg - z * half;
        }
        return hllc_core(WL, WR, p2c(e, WL), p2c(e, WR), inv_L, inv_R, c_L, c_R, axis, shock_blend, F);
    }
}

}   // namespace fvg
