// The mixed-precision form of the stage and viscous kernels: stencil, flux and viscous arithmetic in FP32, the
// conserved state and its Runge-Kutta accumulation in FP64.
//
// What stays FP64: the state in HBM and every stage update (a U0 + b (U + dt R), with R widened to double), and the
// pressure recovery p = (gamma - 1)(E - 1/2 rho |u|^2) of every cell (cons_to_prim in double when a cell is loaded, so a
// low-Mach cell, where E and the kinetic energy nearly cancel, loses nothing). What runs in FP32 (compiled with fast
// single-precision division and square root, and contraction into FMAs): the WENO-Z / MUSCL reconstruction of the
// primitives, the Riemann solver, the flux balance, the viscous stresses and heat flux. The linear and WENO5-Z face values,
// the balance and the FP64 update round every operation explicitly instead, so that every kernel that solves a face or
// updates a cell (the per-axis sweep, the marching kernels, the batched kernels) gives it the same bits.
//
// One algorithmic difference from the plain form: the Riemann solver takes the reconstructed primitive states directly
// (their density and pressure floored as cons_to_prim floors them) instead of converting them to conservative form and
// back, which in FP32 would recover the face pressure from a difference of nearly equal numbers. In exact arithmetic the
// two are the same; the tests state the L1 / Linf distance of this form from the FP64 oracle per field and per case.
#pragma once

#include <type_traits>

#include "grid.cuh"
#include "stage.cuh"
#include "viscous.cuh"

namespace fvg {

// The gas of the mixed form's Riemann solver: gamma, p_inf (0 for an ideal gas), 1 / (gamma - 1) and gamma p_inf.
struct GasF {
    float g, pi, g1, gpi;
};
__device__ __forceinline__ GasF gas_f(const Eos<double>& e) {
    GasF s;
    s.g = (float)e.gamma;
    s.pi = e.type == kIdeal ? 0.0f : (float)e.p_inf;
    s.g1 = __frcp_rn((float)(e.gamma - 1.0));
    s.gpi = __fmul_rn(s.g, s.pi);
    return s;
}
// maximum / minimum of two floats in one instruction, a NaN operand kept
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The Riemann solver of a face whose numbers leave the range in which riemann_f's products are finite: the formulas of the
// plain form in FP32, the wave order decided by the comparisons of vmin / vmax. A solution that blows up comes here: its
// energy flux is the difference of two overflowed terms, a NaN, which the wave-speed maxima skip. (riemann_f's one-sided
// products would give an infinity, and the run would stop as diverged where the plain formulas carry on.) Out of line, so
// that the faces that never come here pay for a comparison: states in, flux (mass, energy, momenta) and speed out.
template <int NA> struct FaceF {
    float s, m, e, v[NA];
};
template <int RIEMANN, int NA>
__device__ __noinline__ FaceF<NA> riemann_wide(GasF g, float shock_blend, float rL, float pL, FaceF<NA> L, float rR, float pR, FaceF<NA> R) {
    constexpr int NV = NA + 2;
    const Eos<float> e{g.pi == 0.0f ? kIdeal : kStiffened, g.g, g.pi, 0.0f};
    St<float, NV> WL, WR, F;
    WL[0] = vmax(rL, Num<float>::eos_eps);
    WL[3] = vmax(pL, Num<float>::eos_eps);
    WR[0] = vmax(rR, Num<float>::eos_eps);
    WR[3] = vmax(pR, Num<float>::eos_eps);
#pragma unroll
    for (int a = 0; a < NA; ++a) {   // the normal velocity in slot 1
        const int q = a < 2 ? 1 + a : 4;
        WL[q] = L.v[a];
        WR[q] = R.v[a];
    }
    const float inv_L = 1.0f / WL[0], inv_R = 1.0f / WR[0];
    const float c_L = sound_speed_inv(e, WL[3], inv_L), c_R = sound_speed_inv(e, WR[3], inv_R);
    if constexpr (RIEMANN == kLowMach) {
        float mL = 0.0f, mR = 0.0f;
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            mL += L.v[a] * L.v[a];
            mR += R.v[a] * R.v[a];
        }
        const float M_L = sqrtf(mL) / (c_L + Num<float>::mach_eps), M_R = sqrtf(mR) / (c_R + Num<float>::mach_eps);
        const float z = vmin(vmax(vmax(M_L, M_R), 1e-4f), 1.0f);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const int q = a < 2 ? 1 + a : 4;
            const float avg = 0.5f * (L.v[a] + R.v[a]), half = 0.5f * (L.v[a] - R.v[a]);
            WL[q] = avg + z * half;
            WR[q] = avg - z * half;
        }
    }
    FaceF<NA> o;
    o.s = hllc_core(WL, WR, p2c(e, WL), p2c(e, WR), inv_L, inv_R, c_L, c_R, 0, shock_blend, F);
    o.m = F[0];
    o.e = F[3];
#pragma unroll
    for (int a = 0; a < NA; ++a) o.v[a] = F[a < 2 ? 1 + a : 4];
    return o;
}
// Below this, a face's largest speed times its energies, no product of riemann_f or of the plain formulas overflows. A NaN is not
// below it.
constexpr float kFaceRange = 1e35f;

// HLLC / low-Mach HLLC of a face from its two primitive states (the Riemann solver of the mixed form): density, pressure
// and the NA velocity components of each side, the normal one first, the others in cyclic order; every operation rounded
// explicitly, so that each kernel that solves a face gets the same flux. Fm: the mass flux, Fe: the energy flux, Fv: the
// momentum fluxes in the order of the velocities; returns max(|S_L|, |S_R|). `range`: below kFaceRange no product overflowed (at
// or above it, or a NaN, the face is riemann_wide's).
//
// The star flux is written from the side the contact leaves to the other: with S the wave speed of that side, q =
// rho (S - u_n) and f = q / (S - S_M), the mass flux is f S_M, the momentum flux f S_M v (+ p* = p + q (S_M - u_n) along
// the normal) and the energy flux S_M (f E + ... + p*): the same flux as F + S (U* - U) of both sides and a choice
// between the four, in exact arithmetic, with one side's states instead of two, two reciprocals instead of five and no
// difference of nearly equal products at low Mach numbers. A supersonic face is the same formulas with S_M = u_n, f = rho,
// p* = p. The Mach number of the low-Mach scaling takes one reciprocal and one square root for both sides.
template <int RIEMANN, int NA>
__device__ __forceinline__ float riemann_f(const GasF& e, float shock_blend, float rL, float pL, float (&vL)[NA], float rR, float pR, float (&vR)[NA],
                                           float& Fm, float& Fe, float (&Fv)[NA], float& range) {
    rL = max_nan(rL, Num<float>::eos_eps);
    pL = max_nan(pL, Num<float>::eos_eps);
    rR = max_nan(rR, Num<float>::eos_eps);
    pR = max_nan(pR, Num<float>::eos_eps);
    const float iL = rcp_f(rL), iR = rcp_f(rR);
    const float aL = __fmul_rn(__fmul_rn(e.g, __fadd_rn(pL, e.pi)), iL), aR = __fmul_rn(__fmul_rn(e.g, __fadd_rn(pR, e.pi)), iR);   // c^2
    const float cL = sqrt_f(aL), cR = sqrt_f(aR);
    const auto square = [](const float (&v)[NA]) {
        float s = __fmul_rn(v[0], v[0]);
#pragma unroll
        for (int a = 1; a < NA; ++a) s = __fmaf_rn(v[a], v[a], s);
        return s;
    };
    if constexpr (RIEMANN == kLowMach) {
        const float mL = square(vL), mR = square(vR);
        const bool gl = __fmul_rn(mL, aR) > __fmul_rn(mR, aL);   // the larger Mach number's side
        const float M = sqrt_f(__fmul_rn(gl ? mL : mR, rcp_f(gl ? aL : aR)));
        const float z = min_nan(max_nan(M, 1e-4f), 1.0f);
#pragma unroll
        for (int a = 0; a < NA; ++a) {
            const float avg = __fmul_rn(0.5f, __fadd_rn(vL[a], vR[a]));
            const float half = __fmul_rn(0.5f, __fsub_rn(vL[a], vR[a]));
            vL[a] = __fmaf_rn(z, half, avg);
            vR[a] = __fmaf_rn(-z, half, avg);
        }
    }
    const float uL = vL[0], uR = vR[0];
    const float SL = min_nan(__fsub_rn(uL, cL), __fsub_rn(uR, cR)), SR = max_nan(__fadd_rn(uL, cL), __fadd_rn(uR, cR));
    const float qL = __fmul_rn(rL, __fsub_rn(SL, uL)), qR = __fmul_rn(rR, __fsub_rn(SR, uR));
    const float num = __fmaf_rn(qR, uR, __fmaf_rn(-qL, uL, __fsub_rn(pL, pR)));
    float SM = __fmul_rn(num, rcp_f(max_nan(__fsub_rn(qR, qL), Num<float>::denom_eps)));   // (qR >= 0 >= qL)
    const bool sup = SL >= 0.0f || SR < 0.0f;
    const bool left = SR >= 0.0f && (SL >= 0.0f || SM >= 0.0f);
    const float rho = left ? rL : rR, p = left ? pL : pR, q = left ? qL : qR;
    float v[NA];   // the side's velocity
#pragma unroll
    for (int a = 0; a < NA; ++a) v[a] = left ? vL[a] : vR[a];
    const float E = __fmaf_rn(0.5f, square(v), __fmul_rn(__fmul_rn(__fadd_rn(p, e.gpi), e.g1), left ? iL : iR));   // per unit mass
    const float d = __fsub_rn(SM, v[0]);
    const float w = __fsub_rn(left ? SL : SR, SM);
    const float rc = rcp_f(copysignf(max_nan(fabsf(w), Num<float>::denom_eps), w));
    float f = __fmul_rn(q, rc), ps = __fmaf_rn(q, d, p);
    float Es = __fmaf_rn(f, __fmaf_rn(d, SM, E), __fmul_rn(__fmul_rn(d, p), rc));
    const float rE = __fmul_rn(rho, E);
    if (sup) {
        SM = v[0];
        f = rho;
        ps = p;
        Es = rE;
    }
    const float s = max_nan(fabsf(SL), fabsf(SR));
    range = __fmul_rn(s, __fadd_rn(fabsf(Es), rE));
    Fm = __fmul_rn(f, SM);
    Fv[0] = __fmaf_rn(Fm, SM, ps);
#pragma unroll
    for (int a = 1; a < NA; ++a) Fv[a] = __fmul_rn(Fm, v[a]);
    Fe = __fmul_rn(SM, __fadd_rn(Es, ps));
    const float jump = fabsf(__fsub_rn(pR, pL)), pm = min_nan(pL, pR);
    if (shock_blend > 0.0f && jump > __fmul_rn(shock_blend, pm) && !sup) {
        // a strong pressure jump: the HLL flux blended in
        const float phi = min_nan(__fmul_rn(__fsub_rn(__fmul_rn(jump, rcp_f(pm)), shock_blend), rcp_f(shock_blend)), 1.0f);
        const float inv = rcp_f(__fsub_rn(SR, SL)), ss = __fmul_rn(SL, SR);
        range = max_nan(range, __fmul_rn(range, s));
        const float mL = __fmul_rn(rL, uL), mR = __fmul_rn(rR, uR);
        const float EL = __fmaf_rn(__fmul_rn(0.5f, rL), square(vL), __fmul_rn(__fadd_rn(pL, e.gpi), e.g1));
        const float ER = __fmaf_rn(__fmul_rn(0.5f, rR), square(vR), __fmul_rn(__fadd_rn(pR, e.gpi), e.g1));
        const auto blend = [&](float f0, float fl, float fr, float ul, float ur) {
            const float h = __fmul_rn(__fmaf_rn(ss, __fsub_rn(ur, ul), __fmaf_rn(SR, fl, -__fmul_rn(SL, fr))), inv);
            return __fmaf_rn(phi, h, __fmul_rn(__fsub_rn(1.0f, phi), f0));
        };
        Fm = blend(Fm, mL, mR, rL, rR);
#pragma unroll
        for (int a = 0; a < NA; ++a)
            Fv[a] = blend(Fv[a], a == 0 ? __fmaf_rn(mL, uL, pL) : __fmul_rn(mL, vL[a]), a == 0 ? __fmaf_rn(mR, uR, pR) : __fmul_rn(mR, vR[a]),
                          __fmul_rn(rL, vL[a]), __fmul_rn(rR, vR[a]));
        Fe = blend(Fe, __fmul_rn(uL, __fadd_rn(EL, pL)), __fmul_rn(uR, __fadd_rn(ER, pR)), EL, ER);
    }
    return s;
}
// riemann_f, or riemann_wide beyond its range
template <int RIEMANN, int NA>
__device__ __forceinline__ float riemann_face(const GasF& e, float shock_blend, float rL, float pL, const float (&vL)[NA], float rR, float pR,
                                              const float (&vR)[NA], float& Fm, float& Fe, float (&Fv)[NA]) {
    float l[NA], r[NA], range;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        l[a] = vL[a];
        r[a] = vR[a];
    }
    const float s = riemann_f<RIEMANN>(e, shock_blend, rL, pL, l, rR, pR, r, Fm, Fe, Fv, range);
    if (range < kFaceRange) return s;
    FaceF<NA> L, R;
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        L.v[a] = vL[a];
        R.v[a] = vR[a];
    }
    const FaceF<NA> o = riemann_wide<RIEMANN, NA>(e, shock_blend, rL, pL, L, rR, pR, R);
    Fm = o.m;
    Fe = o.e;
#pragma unroll
    for (int a = 0; a < NA; ++a) Fv[a] = o.v[a];
    return o.s;
}
// riemann_face of two primitive states in the state's order, along a compile-time axis
template <int RIEMANN, int NV>
__device__ __forceinline__ float face_flux_prim(const GasF& e, float shock_blend, const St<float, NV>& WL, const St<float, NV>& WR, int axis,
                                                St<float, NV>& F) {
    constexpr int NA = NV == 5 ? 3 : 2;   // velocity components
    float vL[NA], vR[NA], Fv[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int c = (axis + a) % NA, m = c == 0 ? 1 : (c == 1 ? 2 : 4);
        vL[a] = WL[m];
        vR[a] = WR[m];
    }
    const float s = riemann_face<RIEMANN>(e, shock_blend, WL[0], WL[3], vL, WR[0], WR[3], vR, F[0], F[3], Fv);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
        const int c = (axis + a) % NA, m = c == 0 ? 1 : (c == 1 ? 2 : 4);
        F[m] = Fv[a];
    }
    return s;
}

// The primitive state of a cell (cons_to_prim in FP64) for the mixed form, each operation rounded explicitly (the same bits
// in every kernel that rounds it to FP32); inv receives 1 / rho of the floored density: the hardware's approximate
// reciprocal and two Newton steps, within a unit in the last place of FP64.
template <int NV> __device__ __forceinline__ St<double, NV> prim_d(const Eos<double>& e, const St<double, NV>& U, double& inv) {
    St<double, NV> W;
    const double rho = vmax(U[0], Num<double>::eos_eps);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(rho));
    // (the steps take an infinite density as a finite one, whose y is 0 too: inf 0 is a NaN. A NaN is in y already.)
    const double r = __hiloint2double(min(__double2hiint(rho), 0x7fefffff), __double2loint(rho));
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    y = __fma_rn(__fma_rn(-r, y, 1.0), y, y);
    inv = y;
    const double u = __dmul_rn(U[1], inv), v = __dmul_rn(U[2], inv);
    double k = __fma_rn(v, v, __dmul_rn(u, u));
    if constexpr (NV == 5) {
        const double w = __dmul_rn(U[4], inv);
        k = __fma_rn(w, w, k);
        W[4] = w;
    }
    const double ei = __fma_rn(__dmul_rn(-0.5, rho), k, U[3]);
    const double gp = e.type == kIdeal ? 0.0 : __dmul_rn(e.gamma, e.p_inf);
    W[0] = rho;
    W[1] = u;
    W[2] = v;
    W[3] = vmax(__fma_rn(__dsub_rn(e.gamma, 1.0), ei, -gp), Num<double>::eos_eps);
    return W;
}

template <int DIM, int RECON, int TX, int TY, int TZ> struct MixedShape {
    static constexpr int NV = DIM == 3 ? 5 : 4;
    static constexpr int H = RECON == kWeno5 ? 3 : 2;
    static constexpr int NC = TX * TY * TZ;
    static constexpr int T3[3] = {TX, TY, TZ};
    static constexpr int ext(int a) { return (T3[0] + (a == 0 ? 2 * H : 0)) * (T3[1] + (a == 1 ? 2 * H : 0)) * (T3[2] + (a == 2 ? 2 * H : 0)); }
    static constexpr int nf(int a) { return (T3[0] + (a == 0)) * (T3[1] + (a == 1)) * (T3[2] + (a == 2)); }
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int EXT = cmax(cmax(ext(0), ext(1)), DIM == 3 ? ext(2) : 0);
    static constexpr int NF = cmax(cmax(nf(0), nf(1)), DIM == 3 ? nf(2) : 0);
    // floats: P [NV][EXT], WL / WR [NV][NF] (the fluxes overwrite WL), acc [NV][NC], 64 for the reduction
    static constexpr int SMEM_FLOATS = NV * EXT + 2 * NV * NF + NV * NC + 64;
    static constexpr int FLAG_BYTES = (EXT + 7) / 8 * 8;   // solidity of the extended tile (WENO5-Z beside an immersed body)
    static constexpr size_t SMEM_BYTES = sizeof(float) * SMEM_FLOATS + FLAG_BYTES;
};

// One axis of the tile sweep of mixed_stage_kernel (compile-time extents).
// GATED (WENO5-Z with the learned sensor): the tile's flag for this axis (one byte per tile and axis, from the sensor's
// last refresh) makes the reconstructions of the sweep linear (0) or WENO5-Z (1), a branch uniform over the CTA; the seam
// faces of a linear tile whose tile across stays WENO5-Z take WENO5-Z in a short pass of their own.
template <int AXIS, int DIM, int RECON, int RIEMANN, int TX, int TY, int TZ, int NT, bool GATED = false, bool FULL = true>
__device__ __forceinline__ void mixed_axis(const StageArgs& a, const GasF& ef, float sb, float weps, float* __restrict__ P,
                                           float* __restrict__ WL, float* __restrict__ WR, float* __restrict__ acc, unsigned char* __restrict__ Sf,
                                           const int o3[3], float& smax) {
    using S = MixedShape<DIM, RECON, TX, TY, TZ>;
    constexpr int NV = S::NV, H = S::H, NC = S::NC;
    constexpr int axis = AXIS;
    const Mesh& m = a.m;
    const int tid = threadIdx.x;
    const int n3[3] = {m.nx, m.ny, m.nz};
    {
        constexpr int E[3] = {TX + (AXIS == 0 ? 2 * H : 0), TY + (AXIS == 1 ? 2 * H : 0), TZ + (AXIS == 2 ? 2 * H : 0)};
        constexpr int Fd[3] = {TX + (AXIS == 0), TY + (AXIS == 1), TZ + (AXIS == 2)};
        constexpr int nE = E[0] * E[1] * E[2], nF = Fd[0] * Fd[1] * Fd[2];
        // ---- 1. load: the primitive state recovered in FP64, stored as FP32
        for (int e = tid; e < nE; e += NT) {
            int l3[3] = {e % E[0], (e / E[0]) % E[1], e / (E[0] * E[1])};
            l3[axis] -= H;
            double inv;
            const St<double, NV> w = prim_d(a.eos, stencil_cons<DIM, NV, FULL>(m, a.bc, a.eos, a.U, o3[0] + l3[0], o3[1] + l3[1], o3[2] + l3[2]), inv);
            if constexpr (RECON == kWeno5)
                if (a.bc.solid) Sf[e] = stencil_solid<DIM>(m, a.bc, o3[0] + l3[0], o3[1] + l3[1], o3[2] + l3[2]);
#pragma unroll
            for (int q = 0; q < NV; ++q) P[q * S::EXT + e] = (float)w[q];
        }
        __syncthreads();
        const int sstride = axis == 0 ? 1 : (axis == 1 ? E[0] : E[0] * E[1]);
        // GATED: whether this tile's reconstructions along the axis are linear, and whether each of its two seam faces
        // along the axis (shared with the tile before and the tile after, which solve them too) may be: only when the
        // tile across is linear as well, so both tiles compute the same flux there and the balance stays conservative.
        // A seam face is the tile's first face and its last face inside the mesh (a partial last tile included); on a
        // periodic axis the neighbour of an end tile is the other end tile; beyond any other side no tile solves the
        // face twice (and the gate keeps such tiles WENO5-Z).
        bool tile_linear = false, seam_lo = false, seam_hi = false;
        int hi_face = 0;
        if constexpr (GATED) {
            const unsigned char* fl = a.sens_flags + (long long)AXIS * a.tiles[0] * a.tiles[1] * a.tiles[2];
            const int b = blockIdx.x + a.b0;
            tile_linear = fl[b] == 0;
            if (tile_linear) {
                const int nt = a.tiles[AXIS];
                const int st = AXIS == 0 ? 1 : (AXIS == 1 ? a.tiles[0] : a.tiles[0] * a.tiles[1]);
                const int ta = AXIS == 0 ? b % a.tiles[0] : (AXIS == 1 ? (b / a.tiles[0]) % a.tiles[1] : b / (a.tiles[0] * a.tiles[1]));
                const bool wrap_lo = a.bc.halo[2 * AXIS] == kHaloWrap, wrap_hi = a.bc.halo[2 * AXIS + 1] == kHaloWrap;
                seam_lo = ta > 0 ? fl[b - st] == 0 : (wrap_lo ? fl[b + (nt - 1) * st] == 0 : true);
                seam_hi = ta < nt - 1 ? fl[b + st] == 0 : (wrap_hi ? fl[b - (nt - 1) * st] == 0 : true);
            }
            hi_face = n3[AXIS] - o3[AXIS] < Fd[AXIS] - 1 ? n3[AXIS] - o3[AXIS] : Fd[AXIS] - 1;
        }
        // ---- 2. face values
        for (int it = tid; it < nF * NV; it += NT) {
            const int f = it % nF, q = it / nF;
            const int f3[3] = {f % Fd[0], (f / Fd[0]) % Fd[1], f / (Fd[0] * Fd[1])};
            const float* c = P + q * S::EXT + (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
            float wl, wr;
            if constexpr (RECON == kMuscl) {
                const float c0 = c[0], c1 = c[sstride], c2 = c[2 * sstride], c3 = c[3 * sstride];
                const float bb = c2 - c1;
                wl = c1 + 0.5f * limiter(a.limiter, c1 - c0, bb);
                wr = c2 - 0.5f * limiter(a.limiter, c3 - c2, bb);
            } else if constexpr (RECON == kWeno3) {
                wl = weno3z(c[0], c[sstride], c[2 * sstride], weps);
                wr = weno3z(c[3 * sstride], c[2 * sstride], c[sstride], weps);
            } else {
                const float c0 = c[0], c1 = c[sstride], c2 = c[2 * sstride], c3 = c[3 * sstride], c4 = c[4 * sstride], c5 = c[5 * sstride];
                const int base = (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
                bool four = false;
                if (a.bc.solid)
#pragma unroll
                    for (int s6 = 0; s6 < 6; ++s6) four = four || Sf[base + s6 * sstride] != 0;
                if (four) {
                    wl = weno3z(c1, c2, c3, weps);
                    wr = weno3z(c4, c3, c2, weps);
                } else if (tile_linear) {
                    // a seam face whose tile across stays WENO5-Z is left to the seam pass below (so that this pass's
                    // warps all take the cheap branch)
                    if (!(f3[AXIS] == 0 ? seam_lo : (f3[AXIS] == hi_face ? seam_hi : true))) continue;
                    // linear fifth-order upwind values where the sensor passed the tile (the WENO-Z weights at their
                    // linear values 0.1, 0.6, 0.3)
                    lin5_pair(c0, c1, c2, c3, c4, c5, wl, wr);
                } else {
                    weno5z_pair(c0, c1, c2, c3, c4, c5, weps, wl, wr);
                }
            }
            WL[q * S::NF + f] = wl;
            WR[q * S::NF + f] = wr;
        }
        if constexpr (GATED) {
            // the seam pass: a linear tile's seam faces whose tile across stays WENO5-Z take WENO5-Z, as that tile does
            if (tile_linear && (!seam_lo || !seam_hi)) {
                constexpr int PL = nF / Fd[AXIS];   // faces of one layer across the axis
                const int layers = (!seam_lo ? 1 : 0) + (!seam_hi ? 1 : 0);
                for (int it = tid; it < layers * PL * NV; it += NT) {
                    const int q = it / (layers * PL), rem = it % (layers * PL), layer = rem / PL, r = rem % PL;
                    int f3[3];
                    f3[AXIS] = (layer == 0 && !seam_lo) ? 0 : hi_face;
                    constexpr int A1 = AXIS == 0 ? 1 : 0, A2 = AXIS == 2 ? 1 : 2;
                    f3[A1] = r % Fd[A1];
                    f3[A2] = r / Fd[A1];
                    const int f = (f3[2] * Fd[1] + f3[1]) * Fd[0] + f3[0];
                    const int base = (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
                    const float* c = P + q * S::EXT + base;
                    const float c0 = c[0], c1 = c[sstride], c2 = c[2 * sstride], c3 = c[3 * sstride], c4 = c[4 * sstride], c5 = c[5 * sstride];
                    bool four = false;
                    if (a.bc.solid)
#pragma unroll
                        for (int s6 = 0; s6 < 6; ++s6) four = four || Sf[base + s6 * sstride] != 0;
                    float wl, wr;
                    if (four) {
                        wl = weno3z(c1, c2, c3, weps);
                        wr = weno3z(c4, c3, c2, weps);
                    } else {
                        weno5z_pair(c0, c1, c2, c3, c4, c5, weps, wl, wr);
                    }
                    WL[q * S::NF + f] = wl;
                    WR[q * S::NF + f] = wr;
                }
            }
        }
        __syncthreads();
        // ---- 3. fluxes
        const int na = n3[axis], lo_side = 2 * axis, hi_side = 2 * axis + 1;
        for (int f = tid; f < nF; f += NT) {
            const int f3[3] = {f % Fd[0], (f / Fd[0]) % Fd[1], f / (Fd[0] * Fd[1])};
            const int g3[3] = {o3[0] + f3[0], o3[1] + f3[1], o3[2] + f3[2]};
            bool inside = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) inside = inside && (d == axis ? g3[d] <= n3[d] : g3[d] < n3[d]);
            St<float, NV> F;
#pragma unroll
            for (int q = 0; q < NV; ++q) F[q] = 0.0f;
            if (inside) {
                const int t = g3[axis];
                const bool lo_face = t == 0 && a.bc.halo[lo_side] == kHaloNone;
                const bool hi_face = t == na && a.bc.halo[hi_side] == kHaloNone;
                St<float, NV> wl, wr;
                if (lo_face || hi_face) {
                    int c3[3] = {g3[0], g3[1], g3[2]};
                    if (hi_face) c3[axis] = na - 1;
                    St<double, NV> UL, UR;
                    side_states<NV, FULL>(m, a.bc, a.eos, a.U, lo_face ? lo_side : hi_side, c3[0], c3[1], c3[2], UL, UR);
                    double inv;
                    const St<double, NV> dl = prim_d(a.eos, UL, inv), dr = prim_d(a.eos, UR, inv);
#pragma unroll
                    for (int q = 0; q < NV; ++q) {
                        wl[q] = (float)dl[q];
                        wr[q] = (float)dr[q];
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < NV; ++q) {
                        wl[q] = WL[q * S::NF + f];
                        wr[q] = WR[q * S::NF + f];
                    }
                }
                const float s = face_flux_prim<RIEMANN>(ef, sb, wl, wr, axis, F);
                if (s > smax) smax = s;
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) WL[q * S::NF + f] = F[q];
        }
        __syncthreads();
        // ---- 4. balance of this axis
        const float A = (float)m.area[axis];
        for (int c = tid; c < NC; c += NT) {
            const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
            const int fl = (c3[2] * Fd[1] + c3[1]) * Fd[0] + c3[0];
            const int fr = fl + (axis == 0 ? 1 : (axis == 1 ? Fd[0] : Fd[0] * Fd[1]));
#pragma unroll
            for (int q = 0; q < NV; ++q) {   // (explicit FMAs, never left to the compiler: every kernel of the mixed
                                               // form sums a cell's balance to the same bits)
                const float df = WL[q * S::NF + fr] - WL[q * S::NF + fl];
                acc[q * NC + c] = axis == 0 ? -__fmul_rn(df, A) : __fmaf_rn(-df, A, acc[q * NC + c]);
            }
        }
        __syncthreads();
        }
}

// The epilogue of the mixed form. A cell's global operands (U, U0, the viscous residual) are loaded first, all variables
// at once, so that their latency overlaps; then every FP64 operation is an explicit intrinsic, FMAs placed by hand
// (nothing left for a compiler pass to contract one way in one kernel and another way in the next: each kernel that
// updates a cell gives it the same bits).
template <int NV> struct CellIn {
    double u[NV], u0[NV], rv[NV];
};
template <int NV> __device__ __forceinline__ void cell_load(const StageArgs& a, long long cell, CellIn<NV>& in) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
        const long long e = q * a.m.plane + cell;
        in.u[q] = a.mode != kStoreR ? a.U[e] : 0.0;
        in.u0[q] = a.mode == kCombine ? a.U0[e] : 0.0;
        in.rv[q] = a.Rvf ? (q == 0 ? 0.0 : (double)a.Rvf[(q - 1) * a.m.plane + cell]) : (a.Rv ? a.Rv[e] : 0.0);
    }
}
// variable q's output from the tile's FP32 balance sum: the residual sum / volume plus the viscous residual (Rv, or the
// 3-D FP32 viscous balance sum of Rvf / volume; the density's viscous term is +0), then R, U + dt R, or ca U0 + cb (U + dt R)
template <int NV> __device__ __forceinline__ double cell_out(const StageArgs& a, const CellIn<NV>& in, int q, float sum, double dt) {
    double r = __dmul_rn((double)sum, a.m.inv_cell);
    if (a.Rvf)
        r = q == 0 ? __dadd_rn(r, 0.0) : __fma_rn(in.rv[q], a.m.inv_cell, r);
    else if (a.Rv)
        r = __dadd_rn(r, in.rv[q]);
    if (a.mode == kStoreR) return r;
    const double u = __fma_rn(dt, r, in.u[q]);
    if (a.mode == kAxpy) return u;
    return __fma_rn(a.ca, in.u0[q], __dmul_rn(a.cb, u));
}

// The mixed-precision stage kernel: the tile sweep of stage_kernel (same phases, same launch geometry) with FP32 stencil
// arithmetic; see the file comment for what stays FP64.
// FULL = false: a run without part interfaces or non-reflecting sides (their code compiled out of the hot loop)
// CTAs per SM, which the compiler left to itself misses by a few registers (it weighs neither the packed face values nor the
// call to riemann_wide). us per step at 128^3, two / three CTAs: WENO3-Z 877 / 748, low-Mach 900 / 767, MUSCL 833 / 701, low-Mach 854 / 721
// (before the packed operands, with 56 registers, low-Mach 816 and 766); 2-D MUSCL at 1024^2, four / five: 233 / 218.
template <int DIM, int RECON, bool FULL> constexpr int kMixedCTAs = DIM == 3 ? (FULL ? 2 : 3) : (FULL ? 3 : (RECON == kMuscl ? 5 : 4));
template <int DIM, int RECON, int RIEMANN, int TX, int TY, int TZ, int NT, bool GATED = false, bool FULL = true>
__global__ void __launch_bounds__(NT, kMixedCTAs<DIM, RECON, FULL>) mixed_stage_kernel(const StageArgs a) {
    using S = MixedShape<DIM, RECON, TX, TY, TZ>;
    constexpr int NV = S::NV, NC = S::NC;
    extern __shared__ double smem_d[];
    double* red = smem_d;                                      // [32]
    float* P = reinterpret_cast<float*>(smem_d + 32);         // [NV][EXT]
    float* WL = P + NV * S::EXT;                               // [NV][NF]
    float* WR = WL + NV * S::NF;                               // [NV][NF]
    float* acc = WR + NV * S::NF;                              // [NV][NC]
    unsigned char* Sf = reinterpret_cast<unsigned char*>(acc + NV * NC);   // [EXT]
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const GasF ef = gas_f(a.eos);
    const float sb = (float)a.shock_blend, weps = (float)a.weno_eps;
    const int tid = threadIdx.x, b = blockIdx.x + a.b0;
    const int o3[3] = {(b % a.tiles[0]) * TX, ((b / a.tiles[0]) % a.tiles[1]) * TY, (b / (a.tiles[0] * a.tiles[1])) * TZ};
    float smax = 0.0f;
    mixed_axis<0, DIM, RECON, RIEMANN, TX, TY, TZ, NT, GATED, FULL>(a, ef, sb, weps, P, WL, WR, acc, Sf, o3, smax);
    mixed_axis<1, DIM, RECON, RIEMANN, TX, TY, TZ, NT, GATED, FULL>(a, ef, sb, weps, P, WL, WR, acc, Sf, o3, smax);
    if constexpr (DIM == 3) mixed_axis<2, DIM, RECON, RIEMANN, TX, TY, TZ, NT, GATED, FULL>(a, ef, sb, weps, P, WL, WR, acc, Sf, o3, smax);
    // ---- epilogue: the residual widened to FP64 and the FP64 stage update
    const double dt = a.ctl->dt;
    for (int c = tid; c < NC; c += NT) {
        const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
        const int g3[3] = {o3[0] + c3[0], o3[1] + c3[1], o3[2] + c3[2]};
        if (g3[0] >= m.nx || g3[1] >= m.ny || g3[2] >= m.nz) continue;
        const long long cell = ((long long)g3[2] * m.ny + g3[1]) * m.nx + g3[0];
        CellIn<NV> in;
        cell_load(a, cell, in);
#pragma unroll
        for (int q = 0; q < NV; ++q) a.out[q * m.plane + cell] = cell_out(a, in, q, acc[q * NC + c], dt);
    }
    const double bm = block_max<NT>((double)smax, red);
    if (tid == 0) stage_finish(a.fin, a.blockmax, b, bm);
}

template <int TX, int TY, int TZ> struct MixedViscShape {
    static constexpr int NC = TX * TY * TZ;
    // red [32 doubles], then float4 arrays: V [NB] box (u, v, w, T), G [NE] (the sweep's four gradient entries), F [NF]
    // (the four face fluxes: rho u, rho v, rho E, rho w; the mass flux is 0), acc [NC] (the four balances); then R [NB]
    // floats (the box's rho): 4 CTAs of the 8x8x8 tile fit on an SM
    static constexpr int BX = TX + 2, BY = TY + 2, BZ = TZ + 2, NB = BX * BY * BZ;
    static constexpr int cmax(int x, int y) { return x > y ? x : y; }
    static constexpr int NE = cmax(cmax((TX + 2) * TY * TZ, TX * (TY + 2) * TZ), TX * TY * (TZ + 2));
    static constexpr int NF = cmax(cmax((TX + 1) * TY * TZ, TX * (TY + 1) * TZ), TX * TY * (TZ + 1));
    static constexpr size_t SMEM_BYTES = 256 + 16 * (NB + NE + NF + NC) + 4 * NB;
};
// component a (0 u, 1 v, 2 w, 3 T) of a box position's float4
__device__ __forceinline__ float f4c(float4 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : (a == 2 ? v.z : v.w)); }
// The mixed-precision viscous kernel: viscous_kernel's phases in FP32; the padded state is read in FP64 and each box
// position's velocity and T = p / rho come from an FP64 pressure recovery. The velocity gradients
// G[a][b] = (d(rho u_a)/dx_b - u_a d(rho)/dx_b) / rho take the box's rho and u_a: (rho+ (u_a+ - u_a) - rho- (u_a- - u_a))
// / (2 h_b rho), the same difference in exact arithmetic. A tile none of whose sides is a wall, inlet or outlet (only
// periodic sides and part interfaces around it) reads its box without the ghost rules and solves its faces without the
// wall tests; a tile wholly inside the mesh skips the test for faces beyond it. The four values a position, a face or a
// cell carries sit together in one float4 (one shared-memory access each); each axis's balance shares a phase with the
// next axis's gradients (six barriers per tile). Meshes whose every side is periodic, without an immersed body, march instead
// (march.cuh).
template <int TX, int TY, int TZ, int NT>
__global__ void __launch_bounds__(NT, 4) mixed_viscous_kernel(const ViscArgs a) {
    using S = MixedViscShape<TX, TY, TZ>;
    constexpr int NC = S::NC, BX = S::BX, BY = S::BY, NB = S::NB;
    extern __shared__ double smem_d[];
    double* red = smem_d;
    float4* V = reinterpret_cast<float4*>(smem_d + 32);   // [NB]: u, v, w, T
    float4* G = V + NB;
    float4* Fv = G + S::NE;
    float4* acc = Fv + S::NF;
    float* R = reinterpret_cast<float*>(acc + NC);         // [NB]: rho
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const int tid = threadIdx.x, b = blockIdx.x + a.b0;
    const int o3[3] = {(b % a.tiles[0]) * TX, ((b / a.tiles[0]) % a.tiles[1]) * TY, (b / (a.tiles[0] * a.tiles[1])) * TZ};
    const int n3[3] = {m.nx, m.ny, m.nz};
    const float h[3] = {(float)m.dx, (float)m.dy, (float)m.dz};
    const float mu = (float)a.mu, kc = (float)a.k_cond;
    constexpr int GA[3][4] = {{0, 1, 2, 0}, {0, 1, 2, 1}, {0, 1, 2, 2}};
    constexpr int GB[3][4] = {{1, 1, 2, 2}, {0, 0, 2, 2}, {0, 1, 0, 1}};
    auto bidx = [&](int i, int j, int k) { return ((k + 1) * BY + (j + 1)) * BX + (i + 1); };
    // whether a side of the tile lies on a side of the mesh that is neither periodic nor a part interface
    bool walls = false;
    {
#pragma unroll
        for (int x = 0; x < 3; ++x) walls = walls || (o3[x] == 0 && !a.through[2 * x]) || (o3[x] + (x == 0 ? TX : (x == 1 ? TY : TZ)) >= n3[x] && !a.through[2 * x + 1]);
    }
    const bool full = o3[0] + TX <= n3[0] && o3[1] + TY <= n3[1] && o3[2] + TZ <= n3[2];   // no cell of the tile beyond the mesh
    for (int e = tid; e < NB; e += NT) {
        int g[3] = {o3[0] + e % BX - 1, o3[1] + (e / BX) % BY - 1, o3[2] + e / (BX * BY) - 1};
#pragma unroll
        for (int x = 0; x < 3; ++x)
            if (a.periodic[x] && (g[x] < 0 || g[x] >= n3[x])) g[x] = ((g[x] % n3[x]) + n3[x]) % n3[x];
#pragma unroll
        for (int x = 0; x < 3; ++x) g[x] = box_clamp(a, x, g[x], n3[x]);
        const St<double, 5> u = walls ? padded_cons(a, g[0], g[1], g[2]) : cell_at(a, g[0], g[1], g[2]);
        double inv;
        const St<double, 5> w = prim_d(a.eos, u, inv);
        R[e] = (float)u[0];
        V[e] = make_float4((float)w[1], (float)w[2], (float)w[4], (float)(w[3] * inv));
    }
    __syncthreads();
    auto sweep = [&](auto axis_c) {
        constexpr int d = decltype(axis_c)::value;
        constexpr int E[3] = {TX + (d == 0 ? 2 : 0), TY + (d == 1 ? 2 : 0), TZ + (d == 2 ? 2 : 0)};
        constexpr int Fd[3] = {TX + (d == 0), TY + (d == 1), TZ + (d == 2)};
        constexpr int nE = E[0] * E[1] * E[2], nF = Fd[0] * Fd[1] * Fd[2];
        // the axes b of this sweep's four entries: GB[d][0..3] takes two distinct values, b0 and b1
        constexpr int b0 = GB[d][0], b1 = GB[d][1] != GB[d][0] ? GB[d][1] : GB[d][2];
        constexpr int off0 = b0 == 0 ? 1 : (b0 == 1 ? BX : BX * BY), off1 = b1 == 0 ? 1 : (b1 == 1 ? BX : BX * BY);
        for (int e = tid; e < nE; e += NT) {
            int l[3] = {e % E[0], (e / E[0]) % E[1], e / (E[0] * E[1])};
            l[d] -= 1;
            const int p = bidx(l[0], l[1], l[2]);
            const float rc = R[p];
            const float inv_rho = 1.0f / vmax(rc, Num<float>::eos_eps);
            const float rp0 = R[p + off0], rm0 = R[p - off0], rp1 = R[p + off1], rm1 = R[p - off1];
            const float4 vc = V[p], vp0 = V[p + off0], vm0 = V[p - off0], vp1 = V[p + off1], vm1 = V[p - off1];
            const float i20 = 0.5f / h[b0], i21 = 0.5f / h[b1];
            float gs[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int ga = GA[d][s];
                const bool first = GB[d][s] == b0;
                const float uc = f4c(vc, ga);
                const float up = first ? f4c(vp0, ga) : f4c(vp1, ga), um = first ? f4c(vm0, ga) : f4c(vm1, ga);
                const float rp = first ? rp0 : rp1, rm = first ? rm0 : rm1;
                gs[s] = (rp * (up - uc) - rm * (um - uc)) * (first ? i20 : i21) * inv_rho;
            }
            G[e] = make_float4(gs[0], gs[1], gs[2], gs[3]);
        }
        __syncthreads();
        const float area = (float)m.area[d];
        const float inv_h = 1.0f / h[d];
        constexpr int estride = d == 0 ? 1 : (d == 1 ? E[0] : E[0] * E[1]);
        constexpr int bstride = d == 0 ? 1 : (d == 1 ? BX : BX * BY);
        for (int f = tid; f < nF; f += NT) {
            const int f3[3] = {f % Fd[0], (f / Fd[0]) % Fd[1], f / (Fd[0] * Fd[1])};
            const int eL = (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
            const int eR = eL + estride;
            int lc[3] = {f3[0], f3[1], f3[2]};
            lc[d] -= 1;
            const int pL = bidx(lc[0], lc[1], lc[2]), pR = pL + bstride;
            float out[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            bool inside = true;
            int xL = eL, xR = eR;
            bool phys = false, lo = false;
            if (walls) {
                const int g3[3] = {o3[0] + f3[0], o3[1] + f3[1], o3[2] + f3[2]};
#pragma unroll
                for (int x = 0; x < 3; ++x) inside = inside && (x == d ? g3[x] <= n3[x] : g3[x] < n3[x]);
                const int t = g3[d];
                lo = t == 0;
                const bool hi = t == n3[d];
                const bool lo_wall = lo && !a.through[2 * d], hi_wall = hi && !a.through[2 * d + 1];
                xL = lo_wall ? eR : eL;
                xR = hi_wall ? eL : eR;
                phys = a.bface2 && (lo_wall || hi_wall);
            } else if (!full) {
                const int g3[3] = {o3[0] + f3[0], o3[1] + f3[1], o3[2] + f3[2]};
#pragma unroll
                for (int x = 0; x < 3; ++x) inside = inside && (x == d ? g3[x] <= n3[x] : g3[x] < n3[x]);
            }
            if (inside) {
                float Gc[4];
                if (phys) {
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const int ga = GA[d][s], gb = GB[d][s];
                        const int pg = lo ? pL : pR, pc = lo ? pR : pL;
                        const int off = gb == 0 ? 1 : (gb == 1 ? BX : BX * BY);
                        const float fp = 0.5f * (f4c(V[pg + off], ga) + f4c(V[pc + off], ga));
                        const float fm = 0.5f * (f4c(V[pg - off], ga) + f4c(V[pc - off], ga));
                        Gc[s] = (fp - fm) * (0.5f / h[gb]);
                    }
                } else {
                    const float4 gl = G[xL], gr = G[xR];
                    Gc[0] = 0.5f * (gl.x + gr.x);
                    Gc[1] = 0.5f * (gl.y + gr.y);
                    Gc[2] = 0.5f * (gl.z + gr.z);
                    Gc[3] = 0.5f * (gl.w + gr.w);
                }
                const float4 vl = V[pL], vr = V[pR];
                float Gn[3], vf[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    Gn[x] = (f4c(vr, x) - f4c(vl, x)) * inv_h;
                    vf[x] = 0.5f * (f4c(vl, x) + f4c(vr, x));
                }
                const float dT = (vr.w - vl.w) * inv_h;
                float tau[3];
                if (d == 0) {
                    tau[0] = mu * ((4.0f / 3.0f) * Gn[0] - (2.0f / 3.0f) * (Gc[1] + Gc[2]));
                    tau[1] = mu * (Gn[1] + Gc[0]);
                    tau[2] = mu * (Gn[2] + Gc[3]);
                } else if (d == 1) {
                    tau[0] = mu * (Gn[0] + Gc[1]);
                    tau[1] = mu * ((4.0f / 3.0f) * Gn[1] - (2.0f / 3.0f) * (Gc[0] + Gc[2]));
                    tau[2] = mu * (Gn[2] + Gc[3]);
                } else {
                    tau[0] = mu * (Gn[0] + Gc[2]);
                    tau[1] = mu * (Gn[1] + Gc[3]);
                    tau[2] = mu * ((4.0f / 3.0f) * Gn[2] - (2.0f / 3.0f) * (Gc[0] + Gc[1]));
                }
                out[0] = tau[0] * area;
                out[1] = tau[1] * area;
                out[2] = (vf[0] * tau[0] + vf[1] * tau[1] + vf[2] * tau[2] + kc * dT) * area;
                out[3] = tau[2] * area;
            }
            Fv[f] = make_float4(out[0], out[1], out[2], out[3]);
        }
        __syncthreads();
    };
    // the balance of one axis into acc: each thread its own cells (the same ones in every call and in the epilogue), so it
    // shares a phase with the next axis's gradients (disjoint arrays) and needs no barrier before the epilogue
    auto balance = [&](auto axis_c) {
        constexpr int d = decltype(axis_c)::value;
        constexpr int Fd[3] = {TX + (d == 0), TY + (d == 1), TZ + (d == 2)};
        for (int c = tid; c < NC; c += NT) {
            const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
            const int fl = (c3[2] * Fd[1] + c3[1]) * Fd[0] + c3[0];
            const int fr = fl + (d == 0 ? 1 : (d == 1 ? Fd[0] : Fd[0] * Fd[1]));
            const float4 l = Fv[fl], r = Fv[fr];
            const float4 dif = make_float4(r.x - l.x, r.y - l.y, r.z - l.z, r.w - l.w);
            if (d == 0) {
                acc[c] = dif;
            } else {
                const float4 s = acc[c];
                acc[c] = make_float4(s.x + dif.x, s.y + dif.y, s.z + dif.z, s.w + dif.w);
            }
        }
    };
    sweep(std::integral_constant<int, 0>{});
    balance(std::integral_constant<int, 0>{});
    sweep(std::integral_constant<int, 1>{});
    balance(std::integral_constant<int, 1>{});
    sweep(std::integral_constant<int, 2>{});
    balance(std::integral_constant<int, 2>{});
    double smax = 0.0;
    const float gm1 = (float)(a.eos.gamma - 1.0);
    for (int c = tid; c < NC; c += NT) {
        const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
        const int g3[3] = {o3[0] + c3[0], o3[1] + c3[1], o3[2] + c3[2]};
        if (g3[0] >= m.nx || g3[1] >= m.ny || g3[2] >= m.nz) continue;
        const long long cell = ((long long)g3[2] * m.ny + g3[1]) * m.nx + g3[0];
        const float4 s4 = acc[c];
        a.Rvf[cell] = s4.x;
        a.Rvf[m.plane + cell] = s4.y;
        a.Rvf[2 * m.plane + cell] = s4.z;
        a.Rvf[3 * m.plane + cell] = s4.w;
        const int p = bidx(c3[0], c3[1], c3[2]);
        const float rho = vmax(R[p], Num<float>::eos_eps);
        const float4 v = V[p];
        const float T = v.w;
        const float nu_eff = vmax((4.0f / 3.0f) * (mu / rho), (kc * gm1) / rho) + 1e-12f;
        const float vm = vmax(vmax(fabsf(v.x), fabsf(v.y)), fabsf(v.z));
        const float cs = sqrtf((float)a.eos.gamma * (T + (float)a.eos.p_inf / rho));
        const double s = (double)(vm + cs + 2.0f * (float)a.L * (float)a.inv_h2 * nu_eff);
        if (s > smax) smax = s;
    }
    const double bm = block_max<NT>(smax, red);
    if (tid == 0) stage_finish(a.fin, a.blockmax, b, bm);
}

}   // namespace fvg
