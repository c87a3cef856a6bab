// The mixed-precision WENO5-Z stage kernel of a 3-D mesh: a CTA owns 32 x 8 columns of cells and marches along z.
//
// The arithmetic of mixed.cuh (the same functions, so the same bits as mixed_stage_kernel, which parts of a decomposed
// mesh and meshes with first-order sides keep), in an order that forms each thing once:
// - the primitive state of a cell is recovered once as its plane arrives and once more where the cell lies beside another
//   CTA's columns (1.9 recoveries per cell; an 8x8x8 tile with its three halos takes 3.25);
// - a thread keeps the six planes of its column around its z face in registers; the plane being solved lies in shared
//   memory with three cells around the columns, for the x and y faces (rows of 40 float4 and 40 floats: a warp
//   reads 32 neighbours of one row, no two words on a bank);
// - per plane a thread solves its low x, its low y and its high z face; the 40 faces on the high sides of the columns fall
//   to two of the warps in turn;
// - four of the five variables lie in one float4, so a stencil cell is two loads and its pairs (rho, p) and (u, v) are
//   operands of packed operations as they stand;
// - fluxes meet in shared memory, and the balance ((0 - x) - y) - z and the FP64 update finish the plane.
// All global operands of a plane (the raw state three planes ahead, the raw halo of the next plane, U, U0 and the viscous
// sums of the cell) are on their way to shared memory (cp.async, each thread its own values, so no barrier) while the plane
// before is solved. Two CTAs per SM (256 threads, at most 128 registers, 77 KB of shared memory).
//
// What bounds it: instruction issue at 16 warps per SM (DRAM 18 %). Mixed + sensor at 256^3: 7.29 ms per step in 8x8x8 tiles with
// boxes by TMA, 7.17 marching with scalar loads, a loop over the axes and a ninth warp (58 warp instructions per cell, issue
// 59 % at 192^3, where the tiles took 80), 6.28 with the viscous sweep below, 5.58 with cells as float4, 5.31 with the
// update's operands waited for where they are used. Mixed at 64^3: 225, 209, 198, 183, 182 us.
#pragma once

#include "mixed.cuh"

namespace fvg {

struct MarchShape {
    static constexpr int W = 32, H = 8, NT = 256, NCOL = W * H;
    static constexpr int PITCH = 40, PL = 14 * PITCH;             // a plane: rows y = -3 .. 10, x = -3 .. 34
    static constexpr int NHALO = 6 * W + 6 * H;                    // cells around the columns
    static constexpr int FXP = 33, NFX = H * FXP, NFY = (H + 1) * W;
    // doubles: red [32], the raw values on their way: core [5][256], halo [5][256], u [5][256], u0 [5][256]; float4 (rho, p, u,
    // v or the fluxes of rho, rho E, rho u, rho v): P [PL], FX [NFX], FY [NFY], FZ [2][256]; floats (w, or the flux of rho w):
    // the same four, and the viscous sums [4][256]
    static constexpr size_t SMEM_BYTES = 8 * (32 + 20 * NCOL) + 20 * (PL + NFX + NFY + 2 * NCOL) + 4 * 4 * NCOL;
};
// a cell's primitive state, or a face's fluxes, in the order of MarchShape
struct March5 {
    float4 a;
    float w;
};
// the face along axis A from its six cells
template <int A, int RIEMANN>
__device__ __forceinline__ float march_face(const GasF& gas, float sb, float weps, bool linear, const March5 (&c)[6], March5& F) {
    const auto lo = [&](int p) { return f2(c[p].a.x, c[p].a.y); };
    const auto hi = [&](int p) { return f2(c[p].a.z, c[p].a.w); };
    F2 l0, l1, r0, r1;
    float lw, rw;
    if (linear) {
        l0 = lin5_f2(lo(0), lo(1), lo(2), lo(3), lo(4));
        r0 = lin5_f2(lo(5), lo(4), lo(3), lo(2), lo(1));
        l1 = lin5_f2(hi(0), hi(1), hi(2), hi(3), hi(4));
        r1 = lin5_f2(hi(5), hi(4), hi(3), hi(2), hi(1));
        lin5_pair(c[0].w, c[1].w, c[2].w, c[3].w, c[4].w, c[5].w, lw, rw);
    } else {
        l0 = weno5z_f2(lo(0), lo(1), lo(2), lo(3), lo(4), weps);
        r0 = weno5z_f2(lo(5), lo(4), lo(3), lo(2), lo(1), weps);
        l1 = weno5z_f2(hi(0), hi(1), hi(2), hi(3), hi(4), weps);
        r1 = weno5z_f2(hi(5), hi(4), hi(3), hi(2), hi(1), weps);
        weno5z_pair(c[0].w, c[1].w, c[2].w, c[3].w, c[4].w, c[5].w, weps, lw, rw);
    }
    float rL, pL, rR, pR, uL, vv, uR, vR_;
    f2_get(l0, rL, pL);
    f2_get(r0, rR, pR);
    f2_get(l1, uL, vv);
    f2_get(r1, uR, vR_);
    const float L[3] = {uL, vv, lw}, R[3] = {uR, vR_, rw};
    float vL[3] = {L[A], L[(A + 1) % 3], L[(A + 2) % 3]}, vR[3] = {R[A], R[(A + 1) % 3], R[(A + 2) % 3]}, Fv[3];
    const float s = riemann_face<RIEMANN>(gas, sb, rL, pL, vL, rR, pR, vR, F.a.x, F.a.y, Fv);
    F.a.z = Fv[(3 - A) % 3];
    F.a.w = Fv[(4 - A) % 3];
    F.w = Fv[(5 - A) % 3];
    return s;
}

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// the copies since the last commit as one group; all groups but the latest one arrived
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_but_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The cell a stencil position g along an axis reads, and the side whose ghost-slab rule applies to it (-1: none); the rules
// of stencil_cons for one axis.
__device__ __forceinline__ int march_cell(const Bc& bc, int axis, int g, int n, int& side) {
    side = -1;
    if (g >= 0 && g < n) return g;
    const bool hi = g >= n;
    const int kind = bc.halo[2 * axis + (hi ? 1 : 0)];
    if (kind == kHaloWrap) return ((g % n) + n) % n;
    if (kind == kHaloSlab) {
        side = 2 * axis + (hi ? 1 : 0);
        const int l0 = hi ? g - n : -1 - g, l = l0 < n ? l0 : n - 1;
        return hi ? n - 1 - l : l;
    }
    return hi ? n - 1 : 0;
}

// z0 .. z1: the planes of the launch; lz: planes per CTA (march_launch). GATED: a face is
// linear when the tiles of both its cells are linear along its axis (inside a tile: when the tile is), which is the seam
// rule of mixed_axis face by face.
template <int RIEMANN, bool GATED, int MB = 2>
__global__ void __launch_bounds__(MarchShape::NT, MB) mixed_march_kernel(const StageArgs a, const int z0, const int z1, const int lz, const int nslots) {
    using S = MarchShape;
    constexpr int NV = 5, PL = S::PL, NCOL = S::NCOL;
    extern __shared__ double smem_d[];
    double* red = smem_d;
    double* Rc = smem_d + 32;        // raw state of the column, three planes ahead
    double* Rh = Rc + 5 * NCOL;      // raw halo of the next plane
    double* Ru = Rh + 5 * NCOL;      // U of the cell
    double* R0 = Ru + 5 * NCOL;      // U0 of the cell
    float4* P4 = reinterpret_cast<float4*>(R0 + 5 * NCOL);   // [PL] the plane being solved
    float4* FX4 = P4 + PL;                                    // [NFX]
    float4* FY4 = FX4 + S::NFX;                               // [NFY]
    float4* FZ4 = FY4 + S::NFY;                               // [2][256]: the z faces below and above the plane, by turns
    float* Pw = reinterpret_cast<float*>(FZ4 + 2 * NCOL);
    float* FXw = Pw + PL;
    float* FYw = FXw + S::NFX;
    float* FZw = FYw + S::NFY;
    float* Rv = FZw + 2 * NCOL;                               // [4][256] the viscous sums
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const GasF gas = gas_f(a.eos);
    const float sb = (float)a.shock_blend, weps = (float)a.weno_eps;
    const int tid = threadIdx.x;
    const int cx = (m.nx + S::W - 1) / S::W, cy = (m.ny + S::H - 1) / S::H;
    const int cta = blockIdx.x;
    const int x0 = (cta % cx) * S::W, y0 = ((cta / cx) % cy) * S::H, za = z0 + (cta / (cx * cy)) * lz;
    const int zb = za + lz < z1 ? za + lz : z1;
    const int tx = tid & 31, ty = tid >> 5;
    const int gx = x0 + tx, gy = y0 + ty;
    const bool cell_in = gx < m.nx && gy < m.ny;
    const long long zs = (long long)m.nx * m.ny;

    // the thread's column and its halo cell: what they read, and the side whose ghost rule they follow
    int cside, hside = -1, hslot = -1;
    long long coff, hoff = 0;
    {
        int sx, sy;
        const int ix = march_cell(a.bc, 0, gx, m.nx, sx), iy = march_cell(a.bc, 1, gy, m.ny, sy);
        coff = (long long)iy * m.nx + ix;
        cside = sx >= 0 ? sx : sy;
        if (tid < S::NHALO) {
            int hx, hy;
            if (tid < 6 * S::W) {
                const int r = tid >> 5;
                hx = tid & 31;
                hy = r < 3 ? r - 3 : S::H + r - 3;
            } else {
                const int r = tid - 6 * S::W, s = r % 6;
                hy = r / 6;
                hx = s < 3 ? s - 3 : S::W + s - 3;
            }
            const int jx = march_cell(a.bc, 0, x0 + hx, m.nx, sx), jy = march_cell(a.bc, 1, y0 + hy, m.ny, sy);
            hoff = (long long)jy * m.nx + jx;
            hside = sx >= 0 ? sx : sy;
            hslot = (hy + 3) * S::PITCH + hx + 3;
        }
    }
    const int pslot = (ty + 3) * S::PITCH + tx + 3;     // the column in a plane of P
    auto prim = [&](const double* raw, long long stride, int side) {
        St<double, NV> u;
#pragma unroll
        for (int q = 0; q < NV; ++q) u[q] = raw[q * stride];
        if (side >= 0) u = ghost_state(a.eos, a.bc, side, u);
        double inv;
        return prim_d(a.eos, u, inv);
    };
    auto fetch_core = [&](int g) {   // the column's raw state of plane g
        int sz;
        const double* src = a.U + march_cell(a.bc, 2, g, m.nz, sz) * zs + coff;
#pragma unroll
        for (int q = 0; q < NV; ++q) cp_async8(Rc + q * NCOL + tid, src + q * m.plane);
    };
    auto core_side = [&](int g) {
        int sz;
        march_cell(a.bc, 2, g, m.nz, sz);
        return sz >= 0 ? sz : cside;
    };
    auto fetch_halo = [&](int g) {
        const double* src = a.U + g * zs + hoff;
#pragma unroll
        for (int q = 0; q < NV; ++q) cp_async8(Rh + q * NCOL + tid, src + q * m.plane);
    };
    auto fetch_cell = [&](int g) {   // the operands of the cell's update
        const long long cell = g * zs + coff;
        if (a.mode != kStoreR)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Ru + q * NCOL + tid, a.U + q * m.plane + cell);
        if (a.mode == kCombine)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(R0 + q * NCOL + tid, a.U0 + q * m.plane + cell);
        if (a.Rvf)
#pragma unroll
            for (int q = 0; q < 4; ++q) cp_async4(Rv + q * NCOL + tid, a.Rvf + q * m.plane + cell);
    };
    // GATED: whether the tile of the cell at (x, y, z) is linear along an axis (a cell beyond a wrapped side: the wrapped
    // cell's; beyond another side no tile, and the tiles beside it are kept WENO5-Z by the gate)
    auto tile_linear = [&](int axis, int x, int y, int z) -> bool {
        int p[3] = {x, y, z};
        const int n3[3] = {m.nx, m.ny, m.nz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (p[d] >= 0 && p[d] < n3[d]) continue;
            if (a.bc.halo[2 * d + (p[d] < 0 ? 0 : 1)] != kHaloWrap) return true;
            p[d] = ((p[d] % n3[d]) + n3[d]) % n3[d];
        }
        const long long t = ((long long)(p[2] >> 3) * a.tiles[1] + (p[1] >> 3)) * a.tiles[0] + (p[0] >> 3);
        return a.sens_flags[(long long)axis * a.tiles[0] * a.tiles[1] * a.tiles[2] + t] == 0;
    };
    fetch_core(za + 3);
    if (hslot >= 0) fetch_halo(za);
    cp_async_commit();
    if (cell_in) fetch_cell(za);
    cp_async_commit();
    // the column's planes k - 2 .. k + 3 in registers, from k = za - 1
    const auto rounded = [](const St<double, NV>& w) {
        return March5{make_float4((float)w[0], (float)w[3], (float)w[1], (float)w[2]), (float)w[4]};
    };
    March5 r[6];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        int sz;
        const double* src = a.U + march_cell(a.bc, 2, za - 3 + p, m.nz, sz) * zs + coff;
        r[p] = rounded(prim(src, m.plane, sz >= 0 ? sz : cside));
    }
    const float Ax = (float)m.area[0], Ay = (float)m.area[1], Az = (float)m.area[2];
    const double dt = a.ctl->dt;
    float smax = 0.0f;
    int lin = 0;   // bits: the thread's low x, low y and high z faces are linear; its faces on the high sides along x and y
    const auto speed = [&](bool inside, float s) {
        if (inside && s > smax) smax = s;
    };
    // k = za - 1: only the z faces below the first plane
#pragma unroll 1
    for (int k = za - 1; k < zb; ++k) {
        const bool first = k < za;
        if (!first) {
            cp_async_wait_but_one();   // (the update's operands, issued last, are waited for where they are used)
#pragma unroll
            for (int p = 0; p < 5; ++p) r[p] = r[p + 1];
            r[5] = rounded(prim(Rc + tid, NCOL, core_side(k + 3)));
            P4[pslot] = r[2].a;
            Pw[pslot] = r[2].w;
            if (hslot >= 0) {
                const March5 h = rounded(prim(Rh + tid, NCOL, hside));
                P4[hslot] = h.a;
                Pw[hslot] = h.w;
            }
            if (k + 1 < zb) {
                fetch_core(k + 4);
                if (hslot >= 0) fetch_halo(k + 1);
            }
            cp_async_commit();
        }
        if constexpr (GATED) {
            if (k <= za || (k & 7) == 0 || (k & 7) == 7) {
                lin = (tile_linear(0, gx - 1, gy, k) && tile_linear(0, gx, gy, k) ? 1 : 0) |
                      (tile_linear(1, gx, gy - 1, k) && tile_linear(1, gx, gy, k) ? 2 : 0) |
                      (tile_linear(2, gx, gy, k) && tile_linear(2, gx, gy, k + 1) ? 4 : 0) |
                      (tx < S::H && tile_linear(0, x0 + S::W - 1, y0 + tx, k) && tile_linear(0, x0 + S::W, y0 + tx, k) ? 8 : 0) |
                      (tile_linear(1, gx, y0 + S::H - 1, k) && tile_linear(1, gx, y0 + S::H, k) ? 16 : 0);
            }
        }
        __syncthreads();
        March5 c[6], F;
        if (gy < m.ny) {   // ---- the high z face
            speed(cell_in, march_face<2, RIEMANN>(gas, sb, weps, GATED && (lin & 4), r, F));
            FZ4[(k & 1) * NCOL + tid] = F.a;
            FZw[(k & 1) * NCOL + tid] = F.w;
        }
        if (!first) {
            // ---- the low x face, and by one warp in turn the high ones of the eight rows
#pragma unroll 1
            for (int fx = tx, fy = ty;;) {
                const bool high = fx >= S::W;
                if (y0 + fy < m.ny) {
                    const float4* b4 = P4 + (fy + 3) * S::PITCH + fx;
                    const float* bw = Pw + (fy + 3) * S::PITCH + fx;
#pragma unroll
                    for (int p = 0; p < 6; ++p) c[p] = March5{b4[p], bw[p]};
                    speed(x0 + fx <= m.nx, march_face<0, RIEMANN>(gas, sb, weps, GATED && (lin & (high ? 8 : 1)), c, F));
                    FX4[fy * S::FXP + fx] = F.a;
                    FXw[fy * S::FXP + fx] = F.w;
                }
                if (high || ty != (k & 7) || tx >= S::H) break;
                fx = S::W;
                fy = tx;
            }
            // ---- the low y face, and by another warp in turn the high ones
#pragma unroll 1
            for (int fy = ty;; fy = S::H) {
                if (y0 + fy <= m.ny) {
                    const float4* b4 = P4 + fy * S::PITCH + tx + 3;
                    const float* bw = Pw + fy * S::PITCH + tx + 3;
#pragma unroll
                    for (int p = 0; p < 6; ++p) c[p] = March5{b4[p * S::PITCH], bw[p * S::PITCH]};
                    speed(gx < m.nx, march_face<1, RIEMANN>(gas, sb, weps, GATED && (lin & (fy == S::H ? 16 : 2)), c, F));
                    FY4[fy * S::W + tx] = F.a;
                    FYw[fy * S::W + tx] = F.w;
                }
                if (fy == S::H || ty != ((k + 4) & 7)) break;
            }
        }
        __syncthreads();
        // ---- the balance, the residual widened to FP64 and the FP64 update of plane k
        if (!first) cp_async_wait_but_one();
        if (!first && cell_in) {
            const long long cell = k * zs + coff;
            CellIn<NV> in;
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                in.u[q] = a.mode != kStoreR ? Ru[q * NCOL + tid] : 0.0;
                in.u0[q] = a.mode == kCombine ? R0[q * NCOL + tid] : 0.0;
                in.rv[q] = a.Rvf && q > 0 ? (double)Rv[(q - 1) * NCOL + tid] : 0.0;
            }
            const int ix = ty * S::FXP + tx, zh = (k & 1) * NCOL + tid, zl = ((k + 1) & 1) * NCOL + tid;
            const float4 xl = FX4[ix], xr = FX4[ix + 1], yl = FY4[tid], yr = FY4[tid + S::W], zd = FZ4[zl], zu = FZ4[zh];
            const auto balance = [&](float x0_, float x1, float y0_, float y1, float z0_, float z1_) {
                float acc = -__fmul_rn(x1 - x0_, Ax);
                acc = __fmaf_rn(-(y1 - y0_), Ay, acc);
                return __fmaf_rn(-(z1_ - z0_), Az, acc);
            };
            const float sum[NV] = {balance(xl.x, xr.x, yl.x, yr.x, zd.x, zu.x), balance(xl.z, xr.z, yl.z, yr.z, zd.z, zu.z),
                                   balance(xl.w, xr.w, yl.w, yr.w, zd.w, zu.w), balance(xl.y, xr.y, yl.y, yr.y, zd.y, zu.y),
                                   balance(FXw[ix], FXw[ix + 1], FYw[tid], FYw[tid + S::W], FZw[zl], FZw[zh])};
#pragma unroll
            for (int q = 0; q < NV; ++q) a.out[q * m.plane + cell] = cell_out(a, in, q, sum[q], dt);
            if (k + 1 < zb) fetch_cell(k + 1);
        }
        if (!first) cp_async_commit();
    }
    const double bm = block_max<S::NT>((double)smax, red);
    if (tid == 0) {
        if (a.fin.kind == kFinNone)   // one entry per tile of the launch is read: this CTA's, and its share of the others empty
            for (int i = cta; i < nslots; i += gridDim.x) a.blockmax[a.b0 + i] = i == cta ? bm : 0.0;
        else
            stage_finish(a.fin, nullptr, 0, bm);
    }
}

// The 2-D form: a CTA owns W columns of cells and marches along y. A thread keeps the six rows of its column around its y
// face in registers; the row being solved lies in shared memory with the halo along x; per row a thread solves its low x
// face and its high y face. A cell is one float4 (rho, p, u, v), its pairs operands of packed operations. The last column's cell belongs to the next CTA (its
// low face is this CTA's last high face), so every thread has the same work. Tiles of the gate: 16 x 15 cells. 2048^2 quadrants
// with the sensor: 342 us per launch in 16 x 15 tiles, 206 marching with scalar loads and one loop over both faces, 182 with cells
// as float4, 167 with the update's operands waited for where they are used.
template <int W_> struct March2Shape {
    static constexpr int W = W_, NT = W_, NHALO = 5, RP = W_ + 8, RAW = W_ + 8;
    // doubles: red [32], raw row [4][RAW] (the column, three rows ahead, then the halo of the next row), u [4][W], u0 [4][W],
    // viscous residual [4][W], the increments Rd of the raw row and of u; float4: P [RP], FX [W] (the fluxes of rho, rho E, rho u, rho v)
    static constexpr size_t SMEM_BYTES = 8 * (32 + 8 * RAW + 16 * W) + 16 * (RP + W);
};
// the face values along axis A from its six cells (rho, p, u, v): density, pressure and the velocities, the normal one first
template <int A>
__device__ __forceinline__ void march2_values(float weps, bool linear, const float4 (&c)[6], float& rL, float& pL, float (&vL)[2], float& rR, float& pR,
                                              float (&vR)[2]) {
    const auto lo = [&](int p) { return f2(c[p].x, c[p].y); };
    const auto hi = [&](int p) { return f2(c[p].z, c[p].w); };
    F2 l0, l1, r0, r1;
    if (linear) {
        l0 = lin5_f2(lo(0), lo(1), lo(2), lo(3), lo(4));
        r0 = lin5_f2(lo(5), lo(4), lo(3), lo(2), lo(1));
        l1 = lin5_f2(hi(0), hi(1), hi(2), hi(3), hi(4));
        r1 = lin5_f2(hi(5), hi(4), hi(3), hi(2), hi(1));
    } else {
        l0 = weno5z_f2(lo(0), lo(1), lo(2), lo(3), lo(4), weps);
        r0 = weno5z_f2(lo(5), lo(4), lo(3), lo(2), lo(1), weps);
        l1 = weno5z_f2(hi(0), hi(1), hi(2), hi(3), hi(4), weps);
        r1 = weno5z_f2(hi(5), hi(4), hi(3), hi(2), hi(1), weps);
    }
    f2_get(l0, rL, pL);
    f2_get(r0, rR, pR);
    f2_get(l1, vL[A], vL[1 - A]);
    f2_get(r1, vR[A], vR[1 - A]);
}
// the face along axis A: its flux, speed and range (riemann_f)
template <int A, int RIEMANN>
__device__ __forceinline__ float march2_face(const GasF& gas, float sb, float weps, bool linear, const float4 (&c)[6], float4& F, float& range) {
    float rL, pL, rR, pR, vL[2], vR[2], Fv[2];
    march2_values<A>(weps, linear, c, rL, pL, vL, rR, pR, vR);
    const float s = riemann_f<RIEMANN>(gas, sb, rL, pL, vL, rR, pR, vR, F.x, F.y, Fv, range);
    F.z = Fv[A];
    F.w = Fv[1 - A];
    return s;
}
// the same by riemann_wide, its face values formed once more (out of line: a row has one test for both its faces)
struct March2F {
    float4 F;
    float s;
};
template <int A, int RIEMANN>
__device__ __noinline__ March2F march2_wide(GasF gas, float sb, float weps, bool linear, float4 c0, float4 c1, float4 c2, float4 c3, float4 c4, float4 c5) {
    const float4 c[6] = {c0, c1, c2, c3, c4, c5};
    float rL, pL, rR, pR;
    FaceF<2> L, R;
    march2_values<A>(weps, linear, c, rL, pL, L.v, rR, pR, R.v);
    const FaceF<2> o = riemann_wide<RIEMANN, 2>(gas, sb, rL, pL, L, rR, pR, R);
    return March2F{make_float4(o.m, o.e, o.v[A], o.v[1 - A]), o.s};
}
template <int RIEMANN, bool GATED, int W, int MB>
__global__ void __launch_bounds__(W, MB) mixed_march2_kernel(const StageArgs a, const int z0, const int z1, const int lz, const int nslots) {
    using S = March2Shape<W>;
    constexpr int NV = 4, RAW = S::RAW;
    extern __shared__ double smem_d[];
    double* red = smem_d;
    double* Rc = smem_d + 32;
    double* Ru = Rc + 4 * RAW;
    double* R0 = Ru + 4 * W;
    double* Rv = R0 + 4 * W;
    double* Dc = Rv + 4 * W;
    double* Du = Dc + 4 * RAW;
    float4* P4 = reinterpret_cast<float4*>(Du + 4 * W);
    float4* FX4 = P4 + S::RP;
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const GasF gas = gas_f(a.eos);
    const float sb = (float)a.shock_blend, weps = (float)a.weno_eps;
    const int tid = threadIdx.x, cta = blockIdx.x;
    const int cx = (m.nx + W - 2) / (W - 1);
    const int x0 = (cta % cx) * (W - 1), za = z0 + (cta / cx) * lz;
    const int zb = za + lz < z1 ? za + lz : z1;
    const int gx = x0 + tid;
    const bool cell_in = tid < W - 1 && gx < m.nx, face_in = gx <= m.nx;
    int cside, hside = -1, coff, hoff = 0;
    coff = march_cell(a.bc, 0, gx, m.nx, cside);
    const bool halo = tid < S::NHALO;
    const int hx = tid < 3 ? tid - 3 : W + tid - 3;
    if (halo) hoff = march_cell(a.bc, 0, x0 + hx, m.nx, hside);
    const double dt = a.ctl->dt;
    auto formed = [&](double u, double d) { return __dadd_rn(u, __dmul_rn(dt, d)); };   // (rounded as k_axpy rounds it)
    auto prim = [&](const double* raw, const double* inc, long long stride, int side) {
        St<double, NV> u;
#pragma unroll
        for (int q = 0; q < NV; ++q) u[q] = a.Rd ? formed(raw[q * stride], inc[q * stride]) : raw[q * stride];
        if (side >= 0) u = ghost_state(a.eos, a.bc, side, u);
        double inv;
        return prim_d(a.eos, u, inv);
    };
    auto fetch_core = [&](int g) {
        int sy;
        const long long at = (long long)march_cell(a.bc, 1, g, m.ny, sy) * m.nx + coff;
#pragma unroll
        for (int q = 0; q < NV; ++q) cp_async8(Rc + q * RAW + tid, a.U + q * m.plane + at);
        if (a.Rd)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Dc + q * RAW + tid, a.Rd + q * m.plane + at);
    };
    auto fetch_halo = [&](int g) {
        const long long at = (long long)g * m.nx + hoff;
#pragma unroll
        for (int q = 0; q < NV; ++q) cp_async8(Rc + q * RAW + W + tid, a.U + q * m.plane + at);
        if (a.Rd)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Dc + q * RAW + W + tid, a.Rd + q * m.plane + at);
    };
    auto fetch_cell = [&](int g) {
        const long long cell = (long long)g * m.nx + coff;
        if (a.mode != kStoreR)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Ru + q * W + tid, a.U + q * m.plane + cell);
        if (a.Rd)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Du + q * W + tid, a.Rd + q * m.plane + cell);
        else if (a.mode == kCombine)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(R0 + q * W + tid, a.U0 + q * m.plane + cell);
        if (a.Rv)
#pragma unroll
            for (int q = 0; q < NV; ++q) cp_async8(Rv + q * W + tid, a.Rv + q * m.plane + cell);
    };
    auto tile_linear = [&](int axis, int x, int y) -> bool {   // (as the 3-D kernel's)
        int p[2] = {x, y};
        const int n2[2] = {m.nx, m.ny};
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            if (p[d] >= 0 && p[d] < n2[d]) continue;
            if (a.bc.halo[2 * d + (p[d] < 0 ? 0 : 1)] != kHaloWrap) return true;
            p[d] = ((p[d] % n2[d]) + n2[d]) % n2[d];
        }
        const long long t = (long long)(p[1] / 15) * a.tiles[0] + (p[0] >> 4);
        return a.sens_flags[(long long)axis * a.tiles[0] * a.tiles[1] + t] == 0;
    };
    fetch_core(za + 3);
    if (halo) fetch_halo(za);
    cp_async_commit();
    if (cell_in) fetch_cell(za);
    cp_async_commit();
    const auto rounded = [](const St<double, NV>& w) { return make_float4((float)w[0], (float)w[3], (float)w[1], (float)w[2]); };
    float4 r[6];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        int sy;
        const long long at = (long long)march_cell(a.bc, 1, za - 3 + p, m.ny, sy) * m.nx + coff;
        r[p] = rounded(prim(a.U + at, a.Rd + at, m.plane, sy >= 0 ? sy : cside));
    }
    const float Ax = (float)m.area[0], Ay = (float)m.area[1];
    float smax = 0.0f;
    float4 Fl = make_float4(0.0f, 0.0f, 0.0f, 0.0f), Fh;   // the y faces below and above the row
    int lin = 0, tile_end = za - 1;   // bit 0, 1: the thread's x and y faces are linear; the row after which to look again
#pragma unroll 1
    for (int k = za - 1; k < zb; ++k) {
        const bool first = k < za;
        if (!first) {
            cp_async_wait_but_one();   // (the update's operands, issued last, are waited for where they are used)
#pragma unroll
            for (int p = 0; p < 5; ++p) r[p] = r[p + 1];
            int sy;
            march_cell(a.bc, 1, k + 3, m.ny, sy);
            r[5] = rounded(prim(Rc + tid, Dc + tid, RAW, sy >= 0 ? sy : cside));
            P4[tid + 3] = r[2];
            if (halo) P4[hx + 3] = rounded(prim(Rc + W + tid, Dc + W + tid, RAW, hside));
            if (k + 1 < zb) {
                fetch_core(k + 4);
                if (halo) fetch_halo(k + 1);
            }
            cp_async_commit();
        }
        if constexpr (GATED) {
            if (k >= tile_end) {   // (the y face above a tile's last row looks at the next tile)
                lin = (tile_linear(0, gx - 1, k) && tile_linear(0, gx, k) ? 1 : 0) | (tile_linear(1, gx, k) && tile_linear(1, gx, k + 1) ? 2 : 0);
                const int last = k < 0 ? -1 : k / 15 * 15 + 14;
                tile_end = k < last ? last : last + 1;
            }
        }
        __syncthreads();
        float4 F = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float range, range_x = 0.0f, sx = 0.0f, sy = march2_face<1, RIEMANN>(gas, sb, weps, GATED && (lin & 2), r, Fh, range);
        const float4* c4 = P4 + tid;
        if (!first) {
            const float4 c[6] = {c4[0], c4[1], c4[2], c4[3], c4[4], c4[5]};
            sx = march2_face<0, RIEMANN>(gas, sb, weps, GATED && (lin & 1), c, F, range_x);
        }
        if (!(max_nan(range, range_x) < kFaceRange)) {
            const March2F y = march2_wide<1, RIEMANN>(gas, sb, weps, GATED && (lin & 2), r[0], r[1], r[2], r[3], r[4], r[5]);
            if (!(range < kFaceRange)) {
                Fh = y.F;
                sy = y.s;
            }
            if (!(range_x < kFaceRange)) {
                const March2F x = march2_wide<0, RIEMANN>(gas, sb, weps, GATED && (lin & 1), c4[0], c4[1], c4[2], c4[3], c4[4], c4[5]);
                F = x.F;
                sx = x.s;
            }
        }
        if (cell_in && sy > smax) smax = sy;
        if (!first) {
            if (face_in && sx > smax) smax = sx;
            FX4[tid] = F;
        }
        __syncthreads();
        if (!first) cp_async_wait_but_one();
        if (!first && cell_in) {
            const long long cell = (long long)k * m.nx + coff;
            CellIn<NV> in;
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                in.u[q] = a.mode != kStoreR ? Ru[q * W + tid] : 0.0;
                in.u0[q] = a.Rd ? in.u[q] : (a.mode == kCombine ? R0[q * W + tid] : 0.0);
                if (a.Rd) in.u[q] = formed(in.u[q], Du[q * W + tid]);
                in.rv[q] = a.Rv ? Rv[q * W + tid] : 0.0;
            }
            const float4 xl = FX4[tid], xr = FX4[tid + 1];
            const auto balance = [&](float x0_, float x1, float y0_, float y1) { return __fmaf_rn(-(y1 - y0_), Ay, -__fmul_rn(x1 - x0_, Ax)); };
            const float sum[NV] = {balance(xl.x, xr.x, Fl.x, Fh.x), balance(xl.z, xr.z, Fl.z, Fh.z), balance(xl.w, xr.w, Fl.w, Fh.w),
                                   balance(xl.y, xr.y, Fl.y, Fh.y)};
#pragma unroll
            for (int q = 0; q < NV; ++q) a.out[q * m.plane + cell] = cell_out(a, in, q, sum[q], dt);
            if (k + 1 < zb) fetch_cell(k + 1);
        }
        if (!first) cp_async_commit();
        Fl = Fh;
    }
    const double bm = block_max<W>((double)smax, red);
    if (tid == 0) {
        if (a.fin.kind == kFinNone)
            for (int i = cta; i < nslots; i += gridDim.x) a.blockmax[a.b0 + i] = i == cta ? bm : 0.0;
        else
            stage_finish(a.fin, nullptr, 0, bm);
    }
}

// Whether a launch can march: a lean WENO5-Z run without an immersed body whose every side wraps or has a ghost slab (no
// first-order boundary faces).
inline bool can_march(const StageArgs& a, int dim) {
    bool ok = !a.bc.solid && !a.bc.slot;
    for (int s = 0; s < 2 * dim; ++s) ok = ok && (a.bc.halo[s] == kHaloWrap || a.bc.halo[s] == kHaloSlab);
    return ok;
}
// The planes a CTA marches over and the launch's time: a round with c CTAs to an SM takes fill + lz (base + per c) us, `resident`
// the most that fit. Fitted to stage launches (FP32 issue grows with c, the chain of a plane does not), where it is within 10 %:
// 3-D 32^3 .. 192^3, 2-D 64^2 .. 1500^2. A plane count that is a multiple of 4 throughout, for the rounds times (lz + 3) alone, took
// 425 us a step at 80^3 (viscous; 333 now), 124 at 32^3 (62) and 45.6 at 128^2 (31.3).
struct MarchCost {
    int resident;
    double fill, base, per;
};
constexpr MarchCost kMarch3Cost = {2, 13.0, 2.4, 3.0}, kMarch2Cost = {5, 8.0, 0.9, 0.77};
struct MarchPlan {
    int lz;
    double us;
};
inline MarchPlan march_plan(const MarchCost& t, int resident, int cols, int nz, int most) {
    MarchPlan best = {0, 0.0};
    const unsigned round = 148u * resident;
    // for each count of parts along the march the fewest planes that give it (a captured launch does this once, others each time)
    for (int lz = 1, parts; lz <= nz; lz = parts > 1 ? (nz + parts - 2) / (parts - 1) : nz + 1) {
        parts = (nz + lz - 1) / lz;
        if (parts > most / cols) continue;
        const unsigned ctas = (unsigned)cols * parts, full = ctas / round, rem = ctas - full * round;
        double us = full * (t.fill + lz * (t.base + t.per * resident));
        if (rem) us += t.fill + lz * (t.base + t.per * ((rem + 147u) / 148u));
        if (!best.lz || us < best.us) best = {lz, us};
    }
    return best;
}
// The part of the mesh a launch of `nblocks` tiles from a.b0 (whole layers of 8x8x8 ones, whole rows of 16 x 15 ones) marches
// over, and how. A launch that writes its CTAs' maxima has at most as many CTAs as tiles (the array's entries).
struct MarchLaunch {
    int z0, z1, cols;
    MarchPlan plan;
    int ctas() const { return cols * ((z1 - z0 + plan.lz - 1) / plan.lz); }
};
constexpr int kMarch2W = 128;
inline int march_most(const Fin& f, int nblocks) { return f.kind == kFinNone ? nblocks : 0x7fffffff; }
inline MarchLaunch march_launch(const StageArgs& a, int dim, int nblocks) {
    const int T = dim == 3 ? 8 : 15, layer = dim == 3 ? a.tiles[0] * a.tiles[1] : a.tiles[0], n = dim == 3 ? a.m.nz : a.m.ny;
    const int end = (a.b0 + nblocks) / layer * T;
    MarchLaunch l;
    l.z0 = a.b0 / layer * T;
    l.z1 = end < n ? end : n;
    l.cols = dim == 3 ? ((a.m.nx + MarchShape::W - 1) / MarchShape::W) * ((a.m.ny + MarchShape::H - 1) / MarchShape::H) : (a.m.nx + kMarch2W - 2) / (kMarch2W - 1);
    const MarchCost& t = dim == 3 ? kMarch3Cost : kMarch2Cost;
    l.plan = march_plan(t, t.resident, l.cols, l.z1 - l.z0, march_most(a.fin, nblocks));
    return l;
}
// Whether a launch marches: where it can, and the tiles (three CTAs to an SM in 3-D, four in 2-D; there with the pass for U + dt R
// that marching spares) would take longer. Same bits either way. Meshes that leave most of their column blocks idle take the tiles:
// 72^3 without viscosity 209 us a step against 244 marching, 128 x 2048 87 against 113, 128 x 900 53 against 70; and 256^2 39 against 44, a
// round of whose tiles is short. Marching: 96^3 343 against 468, 64^3 136 against 176, 400^2 62 against 66, 2048 x 128 72 against 87.
inline bool marches(const StageArgs& a, int dim, int nblocks, MarchLaunch& l) {
    if (!can_march(a, dim)) return false;
    l = march_launch(a, dim, nblocks);
    if (a.Rd) return true;   // (only for a launch this chose)
    const int resident = dim == 3 ? 3 : 4, round = 148 * resident, rem = nblocks % round;
    double us = dim == 3 ? 0.0 : 1.0;
    us += (nblocks / round) * (dim == 3 ? 35.0 : 12.0);
    if (rem) us += (dim == 3 ? 19.0 : 8.0) + (dim == 3 ? 7.5 : 1.9) * ((rem + 147) / 148);
    return l.plan.us < us;
}
template <int RIEMANN, bool GATED> struct MarchK {
    static cudaError_t prepare() {
        return cudaFuncSetAttribute(mixed_march_kernel<RIEMANN, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MarchShape::SMEM_BYTES);
    }
    static cudaError_t launch(const StageArgs& a0, const MarchLaunch& l, int nblocks, cudaStream_t s) {
        StageArgs a = a0;
        a.fin.ctas = l.ctas();
        mixed_march_kernel<RIEMANN, GATED><<<l.ctas(), MarchShape::NT, MarchShape::SMEM_BYTES, s>>>(a, l.z0, l.z1, l.plan.lz, nblocks);
        return cudaGetLastError();
    }
};
template <int RIEMANN, bool GATED> struct March2K {
    using S = March2Shape<kMarch2W>;
    static constexpr auto kern = mixed_march2_kernel<RIEMANN, GATED, kMarch2W, kMarch2Cost.resident>;
    static cudaError_t prepare() { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM_BYTES); }
    static cudaError_t launch(const StageArgs& a0, const MarchLaunch& l, int nblocks, cudaStream_t s) {
        StageArgs a = a0;
        a.fin.ctas = l.ctas();
        kern<<<l.ctas(), S::NT, S::SMEM_BYTES, s>>>(a, l.z0, l.z1, l.plan.lz, nblocks);
        return cudaGetLastError();
    }
};

// ---------------------------------------------------------------------------------------------- viscous fluxes
// The mixed-precision viscous sweep of a mesh whose every side is periodic (parts of it included: no wall rules), marching
// along z like the stage kernel: 32 x 8 columns per CTA, three planes of the columns and one cell around them in shared
// memory (u, v, w, T in one float4, rho beside it). Per plane a thread forms the nine velocity-gradient entries of its cell
// once (the tiled sweep formed four of them for each of three axes, on a tile extended along the axis) and shares them with
// the neighbours along x and y through shared memory and along z through its own registers; then the low x, y and z faces
// of the cell; the ninth warp takes the cells and faces on the high sides. Fluxes and gradients as in mixed_viscous_kernel,
// which meshes with walls, inlets or outlets and immersed bodies keep. Bound by shared-memory
// bandwidth and issue (ncu at 192^3 before a thread kept its own column in registers: L1 77 %, issue 60 %, 20 warp instructions per
// cell; 221 -> 209 us with it). 256^3: 0.78 -> 0.48 ms per launch; the mixed + sensor step 7.17 -> 6.28 ms.
struct ViscMarchShape {
    static constexpr int W = 32, H = 8, NT = 288, BX = W + 2, BY = H + 2, NB = BX * BY, PITCH = 36, PL = BY * PITCH;
    static constexpr int NCOL = W * H, NGX = H * BX, NGY = BY * W, FXP = W + 1, NFX = H * FXP, NFY = (H + 1) * W;
    // doubles: red [32], raw [5][NB]; float4: V [3][PL], GX, GY, FX, FY; floats: R [3][PL]
    static constexpr size_t SMEM_BYTES = 8 * (32 + 5 * NB) + 16 * (3 * PL + NGX + NGY + NFX + NFY) + 4 * 3 * PL;
};

// the viscous flux through a face along axis D (rho u, rho v, rho E, rho w) times its area, from the cells before and after
// it (u, v, w, T) and their four gradient entries
template <int D>
__device__ __forceinline__ float4 visc_face(float4 vl, float4 vr, float4 gl, float4 gr, float inv_h, float mu, float kc, float area) {
    const float g0 = 0.5f * (gl.x + gr.x), g1 = 0.5f * (gl.y + gr.y), g2 = 0.5f * (gl.z + gr.z), g3 = 0.5f * (gl.w + gr.w);
    const float nu = (vr.x - vl.x) * inv_h, nv = (vr.y - vl.y) * inv_h, nw = (vr.z - vl.z) * inv_h, dT = (vr.w - vl.w) * inv_h;
    const float fu = 0.5f * (vl.x + vr.x), fv = 0.5f * (vl.y + vr.y), fw = 0.5f * (vl.z + vr.z);
    float t0, t1, t2;
    if (D == 0) {          // [du/dy, dv/dy, dw/dz, du/dz]
        t0 = mu * ((4.0f / 3.0f) * nu - (2.0f / 3.0f) * (g1 + g2));
        t1 = mu * (nv + g0);
        t2 = mu * (nw + g3);
    } else if (D == 1) {   // [du/dx, dv/dx, dw/dz, dv/dz]
        t0 = mu * (nu + g1);
        t1 = mu * ((4.0f / 3.0f) * nv - (2.0f / 3.0f) * (g0 + g2));
        t2 = mu * (nw + g3);
    } else {               // [du/dx, dv/dy, dw/dx, dw/dy]
        t0 = mu * (nu + g2);
        t1 = mu * (nv + g3);
        t2 = mu * ((4.0f / 3.0f) * nw - (2.0f / 3.0f) * (g0 + g1));
    }
    return make_float4(t0 * area, t1 * area, (fu * t0 + fv * t1 + fw * t2 + kc * dT) * area, t2 * area);
}

__global__ void __launch_bounds__(ViscMarchShape::NT, 3) mixed_viscous_march_kernel(const ViscArgs a, const int z0, const int z1, const int lz,
                                                                                    const int nslots) {
    using S = ViscMarchShape;
    constexpr int PL = S::PL, NB = S::NB;
    extern __shared__ double smem_d[];
    double* red = smem_d;
    double* raw = smem_d + 32;                                    // [5][NB]
    float4* V = reinterpret_cast<float4*>(raw + 5 * NB);          // [3][PL]
    float4* GX = V + 3 * PL;                                      // [H][BX]
    float4* GY = GX + S::NGX;                                     // [BY][W]
    float4* FX = GY + S::NGY;                                     // [H][FXP]
    float4* FY = FX + S::NFX;                                     // [H + 1][W]
    float* R = reinterpret_cast<float*>(FY + S::NFY);             // [3][PL]
    if (!*a.gate) return;
    const Mesh& m = a.m;
    const int n3[3] = {m.nx, m.ny, m.nz};
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, cta = blockIdx.x;
    const int cx = (m.nx + S::W - 1) / S::W, cy = (m.ny + S::H - 1) / S::H;
    const int x0 = (cta % cx) * S::W, y0 = ((cta / cx) % cy) * S::H, za = z0 + (cta / (cx * cy)) * lz;
    const int zb = za + lz < z1 ? za + lz : z1;
    const bool col = ty < S::H;
    const bool cell_in = col && x0 + tx < m.nx && y0 + ty < m.ny;
    const long long zs = (long long)m.nx * m.ny;
    const float mu = (float)a.mu, kc = (float)a.k_cond, gm1 = (float)(a.eos.gamma - 1.0);
    const float hx = (float)m.dx, hy = (float)m.dy, hz = (float)m.dz;
    const float ix2 = 0.5f / hx, iy2 = 0.5f / hy, iz2 = 0.5f / hz, ihx = 1.0f / hx, ihy = 1.0f / hy, ihz = 1.0f / hz;
    const float Ax = (float)m.area[0], Ay = (float)m.area[1], Az = (float)m.area[2];
    auto place = [&](int d, int g) {   // a box position onto the cells the arrays hold
        if (a.periodic[d] && (g < 0 || g >= n3[d])) g = ((g % n3[d]) + n3[d]) % n3[d];
        return box_clamp(a, d, g, n3[d]);
    };
    // the thread's one or two box cells: where they are read and where they are kept in a plane
    long long boff[2];
    int bslot[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int e = tid + j * S::NT, bx = e % S::BX, by = e / S::BX;
        bslot[j] = e < NB ? by * S::PITCH + bx : -1;
        boff[j] = e < NB ? (long long)place(1, y0 + by - 1) * m.nx + place(0, x0 + bx - 1) : 0;
    }
    auto keep = [&](int slot, int p, const St<double, 5>& u) {
        double inv;
        const St<double, 5> w = prim_d(a.eos, u, inv);
        R[p * PL + slot] = (float)u[0];
        V[p * PL + slot] = make_float4((float)w[1], (float)w[2], (float)w[4], (float)__dmul_rn(w[3], inv));
    };
    auto fetch = [&](int g) {
        const double* src = a.U + place(2, g) * zs;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (bslot[j] >= 0)
#pragma unroll
                for (int q = 0; q < 5; ++q) cp_async8(raw + q * NB + tid + j * S::NT, src + q * m.plane + boff[j]);
    };
    // planes za - 1 and za, then za + 1 on its way (plane g is kept at g mod 3, counted from za - 1)
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const double* src = a.U + place(2, za - 1 + p) * zs;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (bslot[j] >= 0) {
                St<double, 5> u;
#pragma unroll
                for (int q = 0; q < 5; ++q) u[q] = src[q * m.plane + boff[j]];
                keep(bslot[j], p, u);
            }
    }
    fetch(za + 1);
    const int own = (ty + 1) * S::PITCH + tx + 1;                                  // the column in a plane
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 gz_prev = zero, fz_prev = zero, sum_prev = zero;
    float4 cm = zero, c = zero, zp = zero;   // the column at k - 1, k, k + 1
    float rm = 0.0f, rc = 0.0f, rzp = 0.0f;
    float smax = 0.0f;
    int s0 = 0;   // the slot of plane k
#pragma unroll 1
    for (int k = za - 1; k <= zb; ++k, s0 = s0 == 2 ? 0 : s0 + 1) {
        const bool inner = k >= za && k < zb;
        const int sp = s0 == 2 ? 0 : s0 + 1, sm = s0 == 0 ? 2 : s0 - 1;   // the slots of the planes k + 1 and k - 1
        if (inner) {
            cp_async_wait();
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (bslot[j] >= 0) {
                    St<double, 5> u;
#pragma unroll
                    for (int q = 0; q < 5; ++q) u[q] = raw[q * NB + tid + j * S::NT];
                    keep(bslot[j], sp, u);
                }
            if (k + 2 <= zb) fetch(k + 2);
        }
        __syncthreads();
        const float4 *Vk = V + s0 * PL, *Vp = V + sp * PL, *Vm = V + sm * PL;
        const float *Rk = R + s0 * PL, *Rp = R + sp * PL, *Rm = R + sm * PL;
        // one gradient entry from the cells after and before along an axis
        auto entry = [](float rp, float up, float rmm, float um, float uc, float s) { return (rp * (up - uc) - rmm * (um - uc)) * s; };
        float4 gz = zero, fz = zero, gx = zero, gy = zero, xm = zero, ym = zero;
        if (col) {
            if (k < za) {
                c = Vk[own];
                rc = Rk[own];
            } else {
                cm = c;
                rm = rc;
                c = zp;
                rc = rzp;
            }
            if (k < zb) {
                zp = Vp[own];
                rzp = Rp[own];
            }
            const float4 xp = Vk[own + 1], yp = Vk[own + S::PITCH];
            xm = Vk[own - 1];
            ym = Vk[own - S::PITCH];
            const float rxp = Rk[own + 1], rxm = Rk[own - 1], ryp = Rk[own + S::PITCH], rym = Rk[own - S::PITCH];
            const float rho = vmax(rc, Num<float>::eos_eps), inv = 1.0f / rho;
            const float sx = ix2 * inv, sy = iy2 * inv, sz = iz2 * inv;
            const float ux = entry(rxp, xp.x, rxm, xm.x, c.x, sx), vy = entry(ryp, yp.y, rym, ym.y, c.y, sy);
            gz = make_float4(ux, vy, entry(rxp, xp.z, rxm, xm.z, c.z, sx), entry(ryp, yp.z, rym, ym.z, c.z, sy));
            if (inner) {
                const float wz = entry(rzp, zp.z, rm, cm.z, c.z, sz);
                gx = make_float4(entry(ryp, yp.x, rym, ym.x, c.x, sy), vy, wz, entry(rzp, zp.x, rm, cm.x, c.x, sz));
                gy = make_float4(ux, entry(rxp, xp.y, rxm, xm.y, c.y, sx), wz, entry(rzp, zp.y, rm, cm.y, c.y, sz));
                GX[ty * S::BX + tx + 1] = gx;
                GY[(ty + 1) * S::W + tx] = gy;
                if (cell_in) {   // the speed bound of the cell
                    const float nu_eff = vmax((4.0f / 3.0f) * (mu / rho), (kc * gm1) / rho) + 1e-12f;
                    const float vm = vmax(vmax(fabsf(c.x), fabsf(c.y)), fabsf(c.z));
                    const float cs = sqrtf((float)a.eos.gamma * (c.w + (float)a.eos.p_inf / rho));
                    const float s = vm + cs + 2.0f * (float)a.L * (float)a.inv_h2 * nu_eff;
                    if (s > smax) smax = s;
                }
            }
            if (k >= za) fz = visc_face<2>(cm, c, gz_prev, gz, ihz, mu, kc, Az);
        } else if (inner) {   // the ninth warp: the cells beside the columns
#pragma unroll
            for (int side = 0; side < 2; ++side) {   // below and above along y: [du/dx, dv/dx, dw/dz, dv/dz]
                const int by = side ? S::BY - 1 : 0, p = by * S::PITCH + tx + 1;
                const float4 q = Vk[p], xp = Vk[p + 1], xq = Vk[p - 1], zq = Vp[p], zm = Vm[p];
                const float rxp = Rk[p + 1], rxm = Rk[p - 1], rzq = Rp[p], rzm = Rm[p];
                const float inv = 1.0f / vmax(Rk[p], Num<float>::eos_eps), sx = ix2 * inv, sz = iz2 * inv;
                GY[by * S::W + tx] = make_float4(entry(rxp, xp.x, rxm, xq.x, q.x, sx), entry(rxp, xp.y, rxm, xq.y, q.y, sx),
                                                 entry(rzq, zq.z, rzm, zm.z, q.z, sz), entry(rzq, zq.y, rzm, zm.y, q.y, sz));
            }
            if (tx < 2 * S::H) {   // before and after along x: [du/dy, dv/dy, dw/dz, du/dz]
                const int row = tx & (S::H - 1), bx = tx < S::H ? 0 : S::BX - 1, p = (row + 1) * S::PITCH + bx;
                const float4 q = Vk[p], yp = Vk[p + S::PITCH], yq = Vk[p - S::PITCH], zq = Vp[p], zm = Vm[p];
                const float ryp = Rk[p + S::PITCH], rym = Rk[p - S::PITCH], rzq = Rp[p], rzm = Rm[p];
                const float inv = 1.0f / vmax(Rk[p], Num<float>::eos_eps), sy = iy2 * inv, sz = iz2 * inv;
                GX[row * S::BX + bx] = make_float4(entry(ryp, yp.x, rym, yq.x, q.x, sy), entry(ryp, yp.y, rym, yq.y, q.y, sy),
                                                   entry(rzq, zq.z, rzm, zm.z, q.z, sz), entry(rzq, zq.x, rzm, zm.x, q.x, sz));
            }
        }
        if (cell_in && k > za) {   // the plane below is complete: its x and y sums and its two z faces
            const long long cell = (k - 1) * zs + (long long)(y0 + ty) * m.nx + x0 + tx;
            a.Rvf[cell] = sum_prev.x + (fz.x - fz_prev.x);
            a.Rvf[m.plane + cell] = sum_prev.y + (fz.y - fz_prev.y);
            a.Rvf[2 * m.plane + cell] = sum_prev.z + (fz.z - fz_prev.z);
            a.Rvf[3 * m.plane + cell] = sum_prev.w + (fz.w - fz_prev.w);
        }
        gz_prev = gz;
        fz_prev = fz;
        if (k == zb) break;
        __syncthreads();
        float4 xl = zero, yl = zero;
        if (inner) {
            if (col) {   // the low faces of the cell: its own side's state and gradients are in registers
                xl = visc_face<0>(xm, c, GX[ty * S::BX + tx], gx, ihx, mu, kc, Ax);
                yl = visc_face<1>(ym, c, GY[tid], gy, ihy, mu, kc, Ay);
                FX[ty * S::FXP + tx] = xl;
                FY[tid] = yl;
            } else {     // the faces on the high sides of the columns
                const int p = S::H * S::PITCH + tx + 1;
                FY[S::NCOL + tx] = visc_face<1>(Vk[p], Vk[p + S::PITCH], GY[S::NCOL + tx], GY[S::NCOL + S::W + tx], ihy, mu, kc, Ay);
                if (tx < S::H) {
                    const int px = (tx + 1) * S::PITCH + S::W, g = tx * S::BX + S::W;
                    FX[tx * S::FXP + S::W] = visc_face<0>(Vk[px], Vk[px + 1], GX[g], GX[g + 1], ihx, mu, kc, Ax);
                }
            }
        }
        __syncthreads();
        if (inner && col) {
            const float4 xr = FX[ty * S::FXP + tx + 1], yr = FY[tid + S::W];
            sum_prev = make_float4((xr.x - xl.x) + (yr.x - yl.x), (xr.y - xl.y) + (yr.y - yl.y), (xr.z - xl.z) + (yr.z - yl.z),
                                   (xr.w - xl.w) + (yr.w - yl.w));
        }
    }
    const double bm = block_max<S::NT>((double)smax, red);
    if (tid == 0) {
        if (a.fin.kind == kFinNone)
            for (int i = cta; i < nslots; i += gridDim.x) a.blockmax[a.b0 + i] = i == cta ? bm : 0.0;
        else
            stage_finish(a.fin, nullptr, 0, bm);
    }
}

inline cudaError_t visc_march_launch(const ViscArgs& a0, int nblocks, cudaStream_t s) {
    ViscArgs a = a0;
    const int layer = a.tiles[0] * a.tiles[1];
    const int z0 = a.b0 / layer * 8, z_end = (a.b0 + nblocks) / layer * 8, z1 = z_end < a.m.nz ? z_end : a.m.nz;
    const int cols = ((a.m.nx + ViscMarchShape::W - 1) / ViscMarchShape::W) * ((a.m.ny + ViscMarchShape::H - 1) / ViscMarchShape::H);
    const int lz = march_plan(kMarch3Cost, 3, cols, z1 - z0, march_most(a.fin, nblocks)).lz;
    const int ctas = cols * ((z1 - z0 + lz - 1) / lz);
    mixed_viscous_march_kernel<<<ctas, ViscMarchShape::NT, ViscMarchShape::SMEM_BYTES, s>>>(a, z0, z1, lz, nblocks);
    return cudaGetLastError();
}

}   // namespace fvg
