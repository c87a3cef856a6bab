// The fused stage kernel: reconstruction (MUSCL / WENO3-Z / WENO5-Z or first order) + Riemann solver + flux
// balance + the time-integrator update of one Runge-Kutta stage, on a tile of cells per CTA.
//
// The reference makes one pass per row (2-D) or plane (3-D) over the mesh (fused_residual_2d / 3d,
// cpp/src/Schemes.cpp:1069-1183); here a CTA owns a TX x TY x TZ tile and sweeps its axes in turn. Per axis:
//   1. load:   the primitive state of the tile extended by H cells along the axis (H = 3 for WENO5-Z, else 2)
//              into shared memory, boundary conditions applied by index mapping (stencil_cons), one
//              cons_to_prim per cell;
//   2. recon:  one thread per (face, variable) computes the left and right face values;
//   3. flux:   one thread per face converts them to conservative form and solves the Riemann problem (faces of a
//              side without a halo take the first-order side states through the round trip instead);
//   4. balance: one thread per cell adds the face-flux difference of this axis to a shared-memory accumulator,
//              in the reference's expression order ((0 - x) - y) - z, so the result has its bits.
// The faces between two tiles are solved by both (the same bits; the reference's thread blocks do the same).
// Epilogue: R = acc * (1 / volume) (+ the viscous residual of the stage, + the body force), then the stage update
//   STORE_R:  out = R
//   AXPY:     out = U + dt R                            (forward Euler, MUSCL-Hancock)
//   COMBINE:  out = a U0 + b (U + dt R)                 (SSP-RK2 / RK3 stages 2 and 3)
// with dt read from the device control block. Each CTA writes the largest face wave speed it saw.
#pragma once

#include "grid.cuh"

namespace fvg {

constexpr int kStoreR = 0, kAxpy = 1, kCombine = 2;

struct StageArgs {
    Mesh m;
    Bc bc;
    Eos<double> eos;
    double shock_blend, weno_eps;
    int limiter;
    int mode;
    double ca, cb;              // COMBINE coefficients
    const double* U;            // the state the residual is taken of (read with halos)
    // mixed_march2_kernel (march.cuh): the state is U + dt Rd, formed as it is read (null: U); then U0 is U
    const double* Rd;
    const double* U0;           // COMBINE: the state at the start of the step (read at the cell only)
    double* out;                // R or the updated state (never aliases U; may alias U0)
    const double* Rv;           // viscous residual to add (null: none)
    // the 3-D mixed form's viscous balance sums instead (FP32, the planes rho u .. rho w after the density's, whose
    // viscous term is 0): the viscous residual is each sum widened to FP64 times 1 / volume (null: none)
    const float* Rvf;
    double* blockmax;           // per-CTA largest wave speed (fin.kind == kFinNone)
    Fin fin;                    // or what is done with it
    const Ctl* ctl;             // dt
    const int* gate;            // the kernel does nothing unless *gate (the control block's `active` or `seed`)
    int tiles[3];               // tiles per axis
    int b0;                     // the tile of the launch's first CTA (a launch over a range of tiles; 0: all)
    // the learned troubled-cell sensor's tile flags (mixed-precision WENO5-Z kernels with the sensor only): one byte per
    // axis and tile (axis-major), 1 where the tile's reconstructions along the axis stay WENO5-Z, 0 where they are linear
    const unsigned char* sens_flags;
    // positivity_fallback: the cells flagged in this stage (null: none); a face next to one takes the cells' states
    const unsigned char* fb;
};

// positivity_fallback's flag of a stencil position (Schemes.cpp:548-557): the cell's; across a periodic seam the wrapped
// cell's; beyond any other side none (a ghost layer is never flagged).
template <int DIM> __device__ __forceinline__ bool fb_flagged(const Mesh& m, const Bc& bc, const unsigned char* fb, int i, int j, int k) {
    int p[3] = {i, j, k};
    const int n3[3] = {m.nx, m.ny, m.nz};
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
        if (p[a] >= 0 && p[a] < n3[a]) continue;
        if (bc.halo[2 * a + (p[a] < 0 ? 0 : 1)] != kHaloWrap) return false;
        p[a] = p[a] < 0 ? p[a] + n3[a] : p[a] - n3[a];
    }
    return fb[((long long)p[2] * m.ny + p[1]) * m.nx + p[0]] != 0;
}

template <int DIM, int RECON, int TX, int TY, int TZ> struct StageShape {
    static constexpr int NV = DIM == 3 ? 5 : 4;
    static constexpr int H = RECON == kWeno5 ? 3 : (RECON == kFirstOrder ? 1 : 2);
    static constexpr int NC = TX * TY * TZ;
    static constexpr int T3[3] = {TX, TY, TZ};
    static constexpr int ext(int a) { return (T3[0] + (a == 0 ? 2 * H : 0)) * (T3[1] + (a == 1 ? 2 * H : 0)) * (T3[2] + (a == 2 ? 2 * H : 0)); }
    static constexpr int nf(int a) { return (T3[0] + (a == 0)) * (T3[1] + (a == 1)) * (T3[2] + (a == 2)); }
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int EXT = cmax(cmax(ext(0), ext(1)), DIM == 3 ? ext(2) : 0);
    static constexpr int NF = cmax(cmax(nf(0), nf(1)), DIM == 3 ? nf(2) : 0);
    // shared memory (doubles): P [NV][EXT] primitive stencil, WL / WR [NV][NF] face values (the fluxes overwrite WL),
    // acc [NV][NC] the balance, 32 for the reduction
    static constexpr int P_SIZE = NV * EXT;
    static constexpr int SMEM_DOUBLES = P_SIZE + 2 * NV * NF + NV * NC + 32;
    static constexpr int FLAG_BYTES = (EXT + 7) / 8 * 8;   // solidity of the extended tile (WENO5-Z beside an immersed body)
    static constexpr size_t SMEM_BYTES = sizeof(double) * SMEM_DOUBLES + FLAG_BYTES;
};

// One axis of the tile sweep of stage_kernel (the axis a template parameter, so the extents of the extended tile and of
// the face grid are compile-time constants).
template <int AXIS, int DIM, int RECON, int RIEMANN, int TX, int TY, int TZ, int NT, bool FULL = true>
__device__ __forceinline__ void stage_axis(const StageArgs& a, double* __restrict__ P, double* __restrict__ WL, double* __restrict__ WR,
                                           double* __restrict__ acc, unsigned char* __restrict__ Sf, const int o3[3], double& smax) {
    using S = StageShape<DIM, RECON, TX, TY, TZ>;
    constexpr int NV = S::NV, H = S::H, NC = S::NC;
    constexpr int axis = AXIS;
    const Mesh& m = a.m;
    const int tid = threadIdx.x;
    const int n3[3] = {m.nx, m.ny, m.nz};
    {
        // extents of the extended tile and of the face grid of this axis (x fastest)
        constexpr int E[3] = {TX + (AXIS == 0 ? 2 * H : 0), TY + (AXIS == 1 ? 2 * H : 0), TZ + (AXIS == 2 ? 2 * H : 0)};
        constexpr int Fd[3] = {TX + (AXIS == 0), TY + (AXIS == 1), TZ + (AXIS == 2)};
        constexpr int nE = E[0] * E[1] * E[2], nF = Fd[0] * Fd[1] * Fd[2];
        // ---- 1. load (primitive; first order keeps the conservative state)
        for (int e = tid; e < nE; e += NT) {
            int l3[3] = {e % E[0], (e / E[0]) % E[1], e / (E[0] * E[1])};
            l3[axis] -= H;
            const St<double, NV> u = stencil_cons<DIM, NV, FULL>(m, a.bc, a.eos, a.U, o3[0] + l3[0], o3[1] + l3[1], o3[2] + l3[2]);
            if constexpr (RECON == kWeno5)
                if (a.bc.solid) Sf[e] = stencil_solid<DIM>(m, a.bc, o3[0] + l3[0], o3[1] + l3[1], o3[2] + l3[2]);
            if constexpr (RECON == kFirstOrder) {
#pragma unroll
                for (int q = 0; q < NV; ++q) P[q * S::EXT + e] = u[q];
            } else {
                const St<double, NV> w = c2p(a.eos, u);
#pragma unroll
                for (int q = 0; q < NV; ++q) P[q * S::EXT + e] = w[q];
            }
        }
        __syncthreads();
        // stride of the stencil along the axis in the extended tile, and the extended position of face f's first cell
        const int sstride = axis == 0 ? 1 : (axis == 1 ? E[0] : E[0] * E[1]);
        // ---- 2. face values
        if constexpr (RECON != kFirstOrder) {
            for (int it = tid; it < nF * NV; it += NT) {
                const int f = it % nF, q = it / nF;
                const int f3[3] = {f % Fd[0], (f / Fd[0]) % Fd[1], f / (Fd[0] * Fd[1])};
                // face t (local, between cells t-1 and t) has its stencil at extended positions t .. t + 2H - 1
                const int base = (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
                const double* c = P + q * S::EXT + base;
                double wl, wr;
                if constexpr (RECON == kMuscl) {
                    const double c0 = c[0], c1 = c[sstride], c2 = c[2 * sstride], c3 = c[3 * sstride];
                    const double bb = c2 - c1;
                    wl = c1 + 0.5 * limiter(a.limiter, c1 - c0, bb);
                    wr = c2 - 0.5 * limiter(a.limiter, c3 - c2, bb);
                } else if constexpr (RECON == kWeno3) {
                    wl = weno3z(c[0], c[sstride], c[2 * sstride], a.weno_eps);
                    wr = weno3z(c[3 * sstride], c[2 * sstride], c[sstride], a.weno_eps);
                } else {
                    const double c0 = c[0], c1 = c[sstride], c2 = c[2 * sstride], c3 = c[3 * sstride], c4 = c[4 * sstride], c5 = c[5 * sstride];
                    bool four = false;   // a solid cell among the six: the four-cell WENO3-Z stencil (weno_line_states, Schemes.cpp:815-831)
                    if (a.bc.solid)
#pragma unroll
                        for (int s6 = 0; s6 < 6; ++s6) four = four || Sf[base + s6 * sstride] != 0;
                    if (four) {
                        wl = weno3z(c1, c2, c3, a.weno_eps);
                        wr = weno3z(c4, c3, c2, a.weno_eps);
                    } else {
                        wl = weno5z(c0, c1, c2, c3, c4, a.weno_eps);
                        wr = weno5z(c5, c4, c3, c2, c1, a.weno_eps);
                    }
                }
                WL[q * S::NF + f] = wl;
                WR[q * S::NF + f] = wr;
            }
            __syncthreads();
        }
        // ---- 3. fluxes, written over the face values: slot f of WL is read and written by the thread of face f only
        const int na = n3[axis];
        const int lo_side = 2 * axis, hi_side = 2 * axis + 1;
        for (int f = tid; f < nF; f += NT) {
            const int f3[3] = {f % Fd[0], (f / Fd[0]) % Fd[1], f / (Fd[0] * Fd[1])};
            const int g3[3] = {o3[0] + f3[0], o3[1] + f3[1], o3[2] + f3[2]};
            bool inside = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) inside = inside && (d == axis ? g3[d] <= n3[d] : g3[d] < n3[d]);
            St<double, NV> F;
#pragma unroll
            for (int q = 0; q < NV; ++q) F[q] = 0.0;
            if (inside) {
                const int t = g3[axis];
                const bool lo_face = t == 0 && a.bc.halo[lo_side] == kHaloNone;
                const bool hi_face = t == na && a.bc.halo[hi_side] == kHaloNone;
                St<double, NV> UL, UR;
                if (lo_face || hi_face) {
                    int c3[3] = {g3[0], g3[1], g3[2]};
                    if (hi_face) c3[axis] = na - 1;
                    side_states<NV, FULL>(m, a.bc, a.eos, a.U, lo_face ? lo_side : hi_side, c3[0], c3[1], c3[2], UL, UR);
                    if constexpr (RECON != kFirstOrder) {
                        UL = round_trip(a.eos, UL);
                        UR = round_trip(a.eos, UR);
                    }
                } else if constexpr (RECON == kFirstOrder) {
                    // between two cells: the extended positions of the cells t-1 and t
                    const int base = (f3[2] * E[1] + f3[1]) * E[0] + f3[0];
#pragma unroll
                    for (int q = 0; q < NV; ++q) {
                        UL[q] = P[q * S::EXT + base];
                        UR[q] = P[q * S::EXT + base + sstride];
                    }
                } else {
                    int lc[3] = {g3[0], g3[1], g3[2]};
                    lc[axis] -= 1;
                    if (FULL && a.fb && (fb_flagged<DIM>(m, a.bc, a.fb, lc[0], lc[1], lc[2]) || fb_flagged<DIM>(m, a.bc, a.fb, g3[0], g3[1], g3[2]))) {
                        // next to a flagged cell: the two cells' states (the ghost of a side's halo beyond it)
                        UL = stencil_cons<DIM, NV>(m, a.bc, a.eos, a.U, lc[0], lc[1], lc[2]);
                        UR = stencil_cons<DIM, NV>(m, a.bc, a.eos, a.U, g3[0], g3[1], g3[2]);
                    } else {
                        St<double, NV> wl, wr;
#pragma unroll
                        for (int q = 0; q < NV; ++q) {
                            wl[q] = WL[q * S::NF + f];
                            wr[q] = WR[q * S::NF + f];
                        }
                        UL = p2c(a.eos, wl);
                        UR = p2c(a.eos, wr);
                    }
                }
                const double s = face_flux<RIEMANN>(a.eos, a.shock_blend, UL, UR, axis, F);
                if (s > smax) smax = s;
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) WL[q * S::NF + f] = F[q];
        }
        __syncthreads();
        // ---- 4. balance of this axis
        const double A = m.area[axis];
        const double* Ff = WL;   // [NV][NF]
        for (int c = tid; c < NC; c += NT) {
            const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
            const int fl = (c3[2] * Fd[1] + c3[1]) * Fd[0] + c3[0];
            const int fr = fl + (axis == 0 ? 1 : (axis == 1 ? Fd[0] : Fd[0] * Fd[1]));
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const double d = Ff[q * S::NF + fr] * A - Ff[q * S::NF + fl] * A;
                acc[q * NC + c] = axis == 0 ? 0.0 - d : acc[q * NC + c] - d;
            }
        }
        __syncthreads();
        }
}

// FULL = false: a run without part interfaces, non-reflecting sides, the positivity fallback or the body force (their
// code compiled out of the hot loop: a branch never taken still costs the others registers and instruction fetch).
// The epilogue's operands that no sweep reads (the tile's rows of U0 and of the viscous residual) head for L2 at the
// start of the tile, so that the epilogue's loads find them there; the arithmetic is untouched.
template <int NV, int TX, int TY, int TZ, int NT> __device__ __forceinline__ void prefetch_tile_rows(const StageArgs& a, const int o3[3]) {
    const bool u0 = a.mode == kCombine, rv = a.Rv != nullptr;
    if (!u0 && !rv) return;
    const Mesh& m = a.m;
    constexpr int R = TY * TZ;   // rows of TX cells
    for (int k = threadIdx.x; k < 2 * NV * R; k += NT) {
        const int which = k / (NV * R), q = (k / R) % NV, r = k % R;
        const int y = o3[1] + r % TY, z = o3[2] + r / TY;
        if (y >= m.ny || z >= m.nz) continue;
        const long long row = ((long long)z * m.ny + y) * m.nx + o3[0];
        if (which == 0 && u0) prefetch_l2(a.U0 + q * m.plane + row);
        if (which == 1 && rv) prefetch_l2(a.Rv + q * m.plane + row);
    }
}

template <int DIM, int RECON, int RIEMANN, int TX, int TY, int TZ, int NT, bool FULL = true, int MB = DIM == 3 ? 2 : 1>
__global__ void __launch_bounds__(NT, MB) stage_kernel(const StageArgs a) {
    using S = StageShape<DIM, RECON, TX, TY, TZ>;
    constexpr int NV = S::NV, NC = S::NC;
    extern __shared__ double smem[];
    double* P = smem;                       // [NV][EXT]
    double* WL = P + S::P_SIZE;             // [NV][NF]
    double* WR = WL + NV * S::NF;           // [NV][NF]
    double* acc = WR + NV * S::NF;          // [NV][NC]
    double* red = acc + NV * NC;            // [32]
    unsigned char* Sf = reinterpret_cast<unsigned char*>(red + 32);   // [EXT]
    if (!*a.gate) return;

    const Mesh& m = a.m;
    const int tid = threadIdx.x;
    const int b = blockIdx.x + a.b0;
    const int t0 = b % a.tiles[0], t1 = (b / a.tiles[0]) % a.tiles[1], t2 = b / (a.tiles[0] * a.tiles[1]);
    const int o3[3] = {t0 * TX, t1 * TY, t2 * TZ};
    double smax = 0.0;
    prefetch_tile_rows<NV, TX, TY, TZ, NT>(a, o3);

    stage_axis<0, DIM, RECON, RIEMANN, TX, TY, TZ, NT, FULL>(a, P, WL, WR, acc, Sf, o3, smax);
    stage_axis<1, DIM, RECON, RIEMANN, TX, TY, TZ, NT, FULL>(a, P, WL, WR, acc, Sf, o3, smax);
    if constexpr (DIM == 3) stage_axis<2, DIM, RECON, RIEMANN, TX, TY, TZ, NT, FULL>(a, P, WL, WR, acc, Sf, o3, smax);
    // ---- epilogue: the residual and the stage update
    const double dt = a.ctl->dt;
    for (int c = tid; c < NC; c += NT) {
        const int c3[3] = {c % TX, (c / TX) % TY, c / (TX * TY)};
        const int g3[3] = {o3[0] + c3[0], o3[1] + c3[1], o3[2] + c3[2]};
        if (g3[0] >= m.nx || g3[1] >= m.ny || g3[2] >= m.nz) continue;
        const long long cell = ((long long)g3[2] * m.ny + g3[1]) * m.nx + g3[0];
        St<double, NV> r;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            r[q] = acc[q * NC + c] * m.inv_cell;
            if (a.Rv) r[q] = r[q] + a.Rv[q * m.plane + cell];
        }
        // the body force, then the case's source terms, join after the viscous term (Simulation::assemble,
        // cpp/src/Simulation.cpp:1038-1049; RhsSourceTerms in the order Simulation::setup adds them, :372-412)
        if constexpr (FULL) {
            if (a.bc.grav_on) add_body_force<NV>(a.bc, read_state<NV>(a.bc, a.U, m.plane, cell), r);
            if (a.bc.src) add_source<NV>(a.bc, m.plane, cell, r);
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const long long e = q * m.plane + cell;
            double o;
            if (a.mode == kStoreR)
                o = r[q];
            else if (a.mode == kAxpy)
                o = a.U[e] + dt * r[q];
            else
                o = a.ca * a.U0[e] + a.cb * (a.U[e] + dt * r[q]);
            a.out[e] = o;
        }
    }
    const double bm = block_max<NT>(smax, red);
    if (tid == 0) stage_finish(a.fin, a.blockmax, b, bm);
}

// The FP64 stage kernel of a 2-D mesh without an immersed body, part interfaces or the other features of FULL: the tile and
// its halos along both axes are converted once (the sweep of stage_kernel converts the tile once per axis), then every face
// of both axes is solved in one pass, one thread per face with all its variables in registers (no face-value arrays), then
// each cell is balanced and updated: two barriers instead of eight, the same operations and bits. The velocity normal to
// the face is put in slot 1 (u u + v v does not depend on the order of its two terms), so one code serves both axes.
//
// A launch covers the mesh rows row0 .. row1 - 1 with tiles of TX x TY cells, TY 15 or 5: a small mesh takes the low tiles,
// whose 181 faces are one round of 192 threads, to spread over the SMs. 131 x 97 vortex (MUSCL, SSP-RK2): 32 -> 24 us per step.
template <int RECON, int TX, int TY> struct Stage2Shape {
    static constexpr int H = RECON == kWeno5 ? 3 : 2;
    static constexpr int PX = TX + 2 * H, PY = TY + 2 * H, NP = PX * PY, NROW = TY * PX, NCROSS = NROW + 2 * H * TX;
    static constexpr int NFX = (TX + 1) * TY, NFY = TX * (TY + 1), NF = NFX + NFY;
    static constexpr size_t SMEM_BYTES = sizeof(double) * (4 * NP + 4 * NF + 32);
};
template <int RECON, int RIEMANN, int TX, int TY, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) stage2d_kernel(const StageArgs a, const int row0, const int row1, const int tiles_x) {
    using S = Stage2Shape<RECON, TX, TY>;
    constexpr int NV = 4, H = S::H, PX = S::PX, NP = S::NP, NF = S::NF;
    extern __shared__ double smem[];
    double* P = smem;             // [4][NP] primitive cross
    double* Fl = P + 4 * NP;      // [4][NF] x faces, then y faces
    double* red = Fl + 4 * NF;
    after_launch_before();
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const Eos<double>& e = a.eos;
    const int tid = threadIdx.x, cta = blockIdx.x;
    const int ox = (cta % tiles_x) * TX, oy = row0 + (cta / tiles_x) * TY;
    const bool inner = ox >= H && ox + TX + H <= m.nx && oy >= H && oy + TY + H <= m.ny;   // no boundary rule (uniform over the CTA)
    for (int c = tid; c < S::NCROSS; c += NT) {
        int i, j;
        if (c < S::NROW) {
            i = c % PX - H;
            j = c / PX;
        } else {
            const int r = (c - S::NROW) / TX;
            i = (c - S::NROW) % TX;
            j = r < H ? r - H : TY + r - H;
        }
        const St<double, NV> u = inner ? read_cell<NV>(a.U, m.plane, (long long)(oy + j) * m.nx + ox + i)
                                       : stencil_cons<2, NV, false>(m, a.bc, e, a.U, ox + i, oy + j, 0);
        const St<double, NV> w = c2p(e, u);
#pragma unroll
        for (int q = 0; q < NV; ++q) P[q * NP + (j + H) * PX + i + H] = w[q];
    }
    __syncthreads();
    double smax = 0.0;
    for (int f = tid; f < NF; f += NT) {
        const int axis = f < S::NFX ? 0 : 1;
        const int r = axis == 0 ? f : f - S::NFX, FX = axis == 0 ? TX + 1 : TX;
        const int fi = r % FX, fj = r / FX, gi = ox + fi, gj = oy + fj;
        const int n_a = axis == 0 ? m.nx : m.ny, t = axis == 0 ? gi : gj;
        const bool inside = axis == 0 ? (gi <= m.nx && gj < m.ny) : (gi < m.nx && gj <= m.ny);
        St<double, NV> F;
#pragma unroll
        for (int q = 0; q < NV; ++q) F[q] = 0.0;
        if (inside) {
            const bool lo = t == 0 && a.bc.halo[2 * axis] == kHaloNone, hi = t == n_a && a.bc.halo[2 * axis + 1] == kHaloNone;
            St<double, NV> UL, UR;
            if (lo || hi) {
                side_states<NV, false>(m, a.bc, e, a.U, 2 * axis + (lo ? 0 : 1), hi && axis == 0 ? n_a - 1 : gi, hi && axis == 1 ? n_a - 1 : gj, 0, UL, UR);
                UL = round_trip(e, UL);
                UR = round_trip(e, UR);
                if (axis == 1) {
                    const double l = UL[1], r1 = UR[1];
                    UL[1] = UL[2];
                    UL[2] = l;
                    UR[1] = UR[2];
                    UR[2] = r1;
                }
            } else {
                // the face's 2 H cells along the axis, from the one H before it
                const int s = axis == 0 ? 1 : PX;
                const double* c0 = P + (fj + H) * PX + fi + H - H * s;
                St<double, NV> wl, wr;
#pragma unroll
                for (int q = 0; q < NV; ++q) {
                    const double* c = c0 + (q == 1 ? 1 + axis : (q == 2 ? 2 - axis : q)) * NP;
                    if constexpr (RECON == kMuscl) {
                        const double v0 = c[0], v1 = c[s], v2 = c[2 * s], v3 = c[3 * s], bb = v2 - v1;
                        wl[q] = v1 + 0.5 * limiter(a.limiter, v1 - v0, bb);
                        wr[q] = v2 - 0.5 * limiter(a.limiter, v3 - v2, bb);
                    } else if constexpr (RECON == kWeno3) {
                        wl[q] = weno3z(c[0], c[s], c[2 * s], a.weno_eps);
                        wr[q] = weno3z(c[3 * s], c[2 * s], c[s], a.weno_eps);
                    } else {
                        const double v0 = c[0], v1 = c[s], v2 = c[2 * s], v3 = c[3 * s], v4 = c[4 * s], v5 = c[5 * s];
                        wl[q] = weno5z(v0, v1, v2, v3, v4, a.weno_eps);
                        wr[q] = weno5z(v5, v4, v3, v2, v1, a.weno_eps);
                    }
                }
                UL = p2c(e, wl);
                UR = p2c(e, wr);
            }
            const double s = face_flux<RIEMANN>(e, a.shock_blend, UL, UR, 0, F);
            if (s > smax) smax = s;
        }
        Fl[f] = F[0];
        Fl[(1 + axis) * NF + f] = F[1];
        Fl[(2 - axis) * NF + f] = F[2];
        Fl[3 * NF + f] = F[3];
    }
    __syncthreads();
    const double dt = a.ctl->dt, Ax = m.area[0], Ay = m.area[1];
    for (int c = tid; c < TX * TY; c += NT) {
        const int ci = c % TX, cj = c / TX, gi = ox + ci, gj = oy + cj;
        if (gi >= m.nx || gj >= row1) continue;
        const long long cell = (long long)gj * m.nx + gi;
        const int fx = cj * (TX + 1) + ci, fy = S::NFX + c;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const double* Fq = Fl + q * NF;
            const double dx = Fq[fx + 1] * Ax - Fq[fx] * Ax, dy = Fq[fy + TX] * Ay - Fq[fy] * Ay;
            const long long x = q * m.plane + cell;
            double r = ((0.0 - dx) - dy) * m.inv_cell;
            if (a.Rv) r = r + a.Rv[x];
            double o;
            if (a.mode == kStoreR)
                o = r;
            else if (a.mode == kAxpy)
                o = a.U[x] + dt * r;
            else
                o = a.ca * a.U0[x] + a.cb * (a.U[x] + dt * r);
            a.out[x] = o;
        }
    }
    const double bm = block_max<NT>(smax, red);
    if (tid == 0) stage_finish(a.fin, a.blockmax, a.b0 + cta, bm);
}

// The FP64 stage kernel of a 3-D mesh: the phases of stage_kernel on an 8x8x8 tile, in a loop over the axes whose body is
// the only copy of the reconstruction and the Riemann solver (an unrolled copy per axis stalled on instruction fetch, 11 %
// of the issue slots). A position of the extended tile or of the face grid is (s, u, v): s along the axis, u and v the other
// two axes in increasing order; one slot is s * 65 + v * 8 + u (rows of 65 so that a row along s touches every bank).
//
// Bound by the latency of FP64 chains (a division is a chain of a dozen dependent operations): 512 threads, two CTAs per SM
// (32 warps; 64 registers, some spilled) beat fewer warps with more registers. ms per launch at 128^3, WENO5-Z, low-Mach HLLC /
// HLLC: the sweep with 256 threads 1.51 / 1.44, with 320 1.31 / 1.24; this loop with 256 1.52, 320 1.29 / 1.25, 384 1.30 / 1.21, 512
// 1.24 / 1.16 (kept); a pair of lanes per face, one for each side, 1.37 / 1.32. MUSCL, whose faces have no WENO divisions, is no
// faster in it (0.56 against 0.55): it keeps the sweep. Runs without the features of FULL only (an immersed body's solid cells
// are among what it serves).
template <int RECON> struct Stage3Shape {
    static_assert(RECON == kWeno3 || RECON == kWeno5, "the loop over the axes");
    static constexpr int NV = 5, H = RECON == kWeno5 ? 3 : 2;
    static constexpr int ROW = 65, NS = 8 + 2 * H, EXT = NS * ROW, NF = 9 * 64, NC = 512;
    static constexpr int FLAG_BYTES = (EXT + 7) / 8 * 8;
    static constexpr size_t SMEM_BYTES = sizeof(double) * (NV * EXT + 2 * NV * NF + NV * NC + 32) + FLAG_BYTES;
};
template <int RECON, int RIEMANN, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) stage3_kernel(const StageArgs a) {
    using S = Stage3Shape<RECON>;
    constexpr int NV = 5, H = S::H, NC = S::NC, NF = S::NF, EXT = S::EXT, ROW = S::ROW;
    extern __shared__ double smem[];
    double* P = smem;                       // [NV][EXT]
    double* WL = P + NV * EXT;              // [NV][NF]
    double* WR = WL + NV * NF;              // [NV][NF]
    double* acc = WR + NV * NF;             // [NV][NC]
    double* red = acc + NV * NC;            // [32]
    unsigned char* Sf = reinterpret_cast<unsigned char*>(red + 32);   // [EXT]
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const int tid = threadIdx.x;
    const int b = blockIdx.x + a.b0;
    const int o3[3] = {b % a.tiles[0] * 8, (b / a.tiles[0]) % a.tiles[1] * 8, b / (a.tiles[0] * a.tiles[1]) * 8};
    double smax = 0.0;
    prefetch_tile_rows<NV, 8, 8, 8, NT>(a, o3);
#pragma unroll 1
    for (int axis = 0; axis < 3; ++axis) {
        const auto place = [&](int s, int u, int v, int& i, int& j, int& k) {   // mesh position of (s, u, v)
            i = o3[0] + (axis == 0 ? s : u);
            j = o3[1] + (axis == 1 ? s : (axis == 0 ? u : v));
            k = o3[2] + (axis == 2 ? s : v);
        };
        // ---- 1. load, x fastest
        for (int e = tid; e < S::NS * 64; e += NT) {
            int s, u, v, i, j, k;
            if (axis == 0) {
                s = e % S::NS;
                u = (e / S::NS) & 7;
                v = e / (S::NS * 8);
            } else {
                u = e & 7;
                s = axis == 1 ? (e >> 3) % S::NS : e >> 6;
                v = axis == 1 ? (e >> 3) / S::NS : (e >> 3) & 7;
            }
            const int slot = s * ROW + v * 8 + u;
            place(s - H, u, v, i, j, k);
            const St<double, NV> c = stencil_cons<3, NV, false>(m, a.bc, a.eos, a.U, i, j, k);
            if constexpr (RECON == kWeno5)
                if (a.bc.solid) Sf[slot] = stencil_solid<3>(m, a.bc, i, j, k);
            const St<double, NV> w = c2p(a.eos, c);
#pragma unroll
            for (int q = 0; q < NV; ++q) P[q * EXT + slot] = w[q];
        }
        __syncthreads();
        // ---- 2. face values: face t = f / 64 has its stencil at the rows t .. t + 2H - 1
        for (int it = tid; it < NF * NV; it += NT) {
            const int q = it / NF, f = it - q * NF, slot = (f >> 6) * ROW + (f & 63);
            const double* c = P + q * EXT + slot;
            double wl, wr;
            if constexpr (RECON == kWeno3) {
                wl = weno3z(c[0], c[ROW], c[2 * ROW], a.weno_eps);
                wr = weno3z(c[3 * ROW], c[2 * ROW], c[ROW], a.weno_eps);
            } else {
                const double c0 = c[0], c1 = c[ROW], c2 = c[2 * ROW], c3 = c[3 * ROW], c4 = c[4 * ROW], c5 = c[5 * ROW];
                bool four = false;   // a solid cell among the six: the four-cell WENO3-Z stencil (weno_line_states, Schemes.cpp:815-831)
                if (a.bc.solid)
#pragma unroll
                    for (int s6 = 0; s6 < 6; ++s6) four = four || Sf[slot + s6 * ROW] != 0;
                if (four) {
                    wl = weno3z(c1, c2, c3, a.weno_eps);
                    wr = weno3z(c4, c3, c2, a.weno_eps);
                } else {
                    wl = weno5z(c0, c1, c2, c3, c4, a.weno_eps);
                    wr = weno5z(c5, c4, c3, c2, c1, a.weno_eps);
                }
            }
            WL[q * NF + f] = wl;
            WR[q * NF + f] = wr;
        }
        __syncthreads();
        // ---- 3. fluxes, written over the face values: slot f of WL is read and written by the thread of face f only
        const int na = axis == 0 ? m.nx : (axis == 1 ? m.ny : m.nz);
        const int lo_side = 2 * axis, hi_side = 2 * axis + 1;
        for (int f = tid; f < NF; f += NT) {
            int i, j, k;
            place(f >> 6, f & 7, (f >> 3) & 7, i, j, k);
            const bool inside = i < m.nx + (axis == 0) && j < m.ny + (axis == 1) && k < m.nz + (axis == 2);
            St<double, NV> F;
#pragma unroll
            for (int q = 0; q < NV; ++q) F[q] = 0.0;
            if (inside) {
                const int t = axis == 0 ? i : (axis == 1 ? j : k);
                const bool lo_face = t == 0 && a.bc.halo[lo_side] == kHaloNone;
                const bool hi_face = t == na && a.bc.halo[hi_side] == kHaloNone;
                St<double, NV> UL, UR;
                if (lo_face || hi_face) {
                    const int d = hi_face ? 1 : 0;
                    side_states<NV, false>(m, a.bc, a.eos, a.U, lo_face ? lo_side : hi_side, i - (axis == 0 ? d : 0), j - (axis == 1 ? d : 0),
                                          k - (axis == 2 ? d : 0), UL, UR);
                    UL = round_trip(a.eos, UL);
                    UR = round_trip(a.eos, UR);
                } else {
                    St<double, NV> wl, wr;
#pragma unroll
                    for (int q = 0; q < NV; ++q) {
                        wl[q] = WL[q * NF + f];
                        wr[q] = WR[q * NF + f];
                    }
                    UL = p2c(a.eos, wl);
                    UR = p2c(a.eos, wr);
                }
                const double s = face_flux<RIEMANN>(a.eos, a.shock_blend, UL, UR, axis, F);
                if (s > smax) smax = s;
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) WL[q * NF + f] = F[q];
        }
        __syncthreads();
        // ---- 4. balance of this axis
        const double A = axis == 0 ? m.area[0] : (axis == 1 ? m.area[1] : m.area[2]);
        for (int c = tid; c < NC; c += NT) {
            const int x = c & 7, y = (c >> 3) & 7, z = c >> 6;
            const int fl = axis == 0 ? x * 64 + z * 8 + y : (axis == 1 ? y * 64 + z * 8 + x : c);
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const double d = WL[q * NF + fl + 64] * A - WL[q * NF + fl] * A;
                acc[q * NC + c] = axis == 0 ? 0.0 - d : acc[q * NC + c] - d;
            }
        }
        __syncthreads();
    }
    // ---- epilogue: the residual and the stage update
    const double dt = a.ctl->dt;
    for (int c = tid; c < NC; c += NT) {
        const int g0 = o3[0] + (c & 7), g1 = o3[1] + ((c >> 3) & 7), g2 = o3[2] + (c >> 6);
        if (g0 >= m.nx || g1 >= m.ny || g2 >= m.nz) continue;
        const long long cell = ((long long)g2 * m.ny + g1) * m.nx + g0;
        St<double, NV> r;
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            r[q] = acc[q * NC + c] * m.inv_cell;
            if (a.Rv) r[q] = r[q] + a.Rv[q * m.plane + cell];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            const long long e = q * m.plane + cell;
            double o;
            if (a.mode == kStoreR)
                o = r[q];
            else if (a.mode == kAxpy)
                o = a.U[e] + dt * r[q];
            else
                o = a.ca * a.U0[e] + a.cb * (a.U[e] + dt * r[q]);
            a.out[e] = o;
        }
    }
    const double bm = block_max<NT>(smax, red);
    if (tid == 0) stage_finish(a.fin, a.blockmax, b, bm);
}

}   // namespace fvg
