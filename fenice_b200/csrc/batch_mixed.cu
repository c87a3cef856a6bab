// The mixed-precision batched stage kernel (the mixed form of batch_stage_kernel; see mixed.cuh for what stays FP64).
// Built with --use_fast_math, as mixed.cu.
#include "batch.cuh"
#include "batch_api.h"
#include "mixed.cuh"

namespace fvg {
namespace {

// a y face of the thin row in the mixed form: the boundary-face states in FP64 (side_states), their primitives rounded to
// FP32, the Riemann solver in FP32 (as mixed_axis does for boundary faces)
template <int RIEMANN>
__device__ __forceinline__ float thin_face_mixed(const StageArgs& a, const GasF& ef, float sb, int side, int i, St<float, 4>& F) {
    St<double, 4> UL, UR;
    side_states<4, false>(a.m, a.bc, a.eos, a.U, side, i, 0, 0, UL, UR);
    double inv;
    const St<double, 4> dl = prim_d(a.eos, UL, inv), dr = prim_d(a.eos, UR, inv);
    St<float, 4> wl, wr;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        wl[q] = (float)dl[q];
        wr[q] = (float)dr[q];
    }
    return face_flux_prim<RIEMANN>(ef, sb, wl, wr, 1, F);
}

// A work item of a one-cell-high mesh whose bottom and top have no halo (a shock tube; thin_y): a thread loads its cell
// (the first ones the halo too), solves the low x face of its cell with all variables in registers, and updates the cell
// from its own and its neighbour's flux: two barriers, where the general sweep takes four and passes every face value
// through shared memory. The y faces of a cell between copies of it cancel, where their fluxes are finite, and only their
// speed counts (riemann_f's for equal states). The bits of mixed_axis along x and of its boundary faces along y.
template <int RECON, int RIEMANN, int TX, int NT>
__device__ __forceinline__ void thin_row_mixed(const StageArgs& a, const GasF& gas, float sb, float weps, float* __restrict__ P, float* __restrict__ FX,
                                               int ox, double dt, float& smax) {
    constexpr int NV = 4, H = RECON == kWeno5 ? 3 : 2, RP = NT + 8;
    static_assert(TX == NT - 1, "one face per thread");
    const Mesh& m = a.m;
    const int tid = threadIdx.x, n = m.nx;
    for (int e = tid; e < TX + 2 * H; e += NT) {
        double inv;
        const St<double, NV> w = prim_d(a.eos, stencil_cons<2, NV, false>(m, a.bc, a.eos, a.U, ox + e - H, 0, 0), inv);
#pragma unroll
        for (int q = 0; q < NV; ++q) P[q * RP + e] = (float)w[q];
    }
    const int i = ox + tid;
    const bool cell = tid < TX && i < n;
    CellIn<NV> in;
    if (cell) cell_load(a, i, in);
    __syncthreads();
    if (i <= n) {   // the face before cell i
        St<float, NV> wl, wr, F;
        const bool lo = i == 0 && a.bc.halo[0] == kHaloNone, hi = i == n && a.bc.halo[1] == kHaloNone;
        if (lo || hi) {
            St<double, NV> UL, UR;
            double inv;
            side_states<NV, false>(m, a.bc, a.eos, a.U, lo ? 0 : 1, lo ? 0 : n - 1, 0, 0, UL, UR);
            const St<double, NV> dl = prim_d(a.eos, UL, inv), dr = prim_d(a.eos, UR, inv);
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                wl[q] = (float)dl[q];
                wr[q] = (float)dr[q];
            }
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                const float* c = P + q * RP + tid;
                if constexpr (RECON == kMuscl) {
                    const float bb = c[2] - c[1];
                    wl[q] = c[1] + 0.5f * limiter(a.limiter, c[1] - c[0], bb);
                    wr[q] = c[2] - 0.5f * limiter(a.limiter, c[3] - c[2], bb);
                } else if constexpr (RECON == kWeno3) {
                    wl[q] = weno3z(c[0], c[1], c[2], weps);
                    wr[q] = weno3z(c[3], c[2], c[1], weps);
                } else {
                    weno5z_pair(c[0], c[1], c[2], c[3], c[4], c[5], weps, wl[q], wr[q]);
                }
            }
        }
        const float s = face_flux_prim<RIEMANN>(gas, sb, wl, wr, 0, F);
        if (s > smax) smax = s;
#pragma unroll
        for (int q = 0; q < NV; ++q) FX[q * NT + tid] = F[q];
    }
    __syncthreads();
    if (!cell) return;
    const float Ax = (float)m.area[0], Ay = (float)m.area[1];
    float acc[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) acc[q] = -__fmul_rn(FX[q * NT + tid + 1] - FX[q * NT + tid], Ax);
    bool same = copy_side(a.bc.type[2]) && copy_side(a.bc.type[3]);
    if (same) {
        const float* w = P + tid + H;
        const float r = max_nan(w[0], Num<float>::eos_eps), p = max_nan(w[3 * RP], Num<float>::eos_eps), u = w[RP], v = w[2 * RP];
        const float cs = sqrt_f(__fmul_rn(__fmul_rn(gas.g, __fadd_rn(p, gas.pi)), rcp_f(r)));
        const float s = max_nan(fabsf(__fsub_rn(v, cs)), fabsf(__fadd_rn(v, cs)));
        // finite fluxes: with s = |v| + c the energy per volume is at most r (u^2 + s^2) times 1 / (gamma - 1) or a half, and s times
        // it their bound (a state beyond riemann_f's range is solved)
        same = __fmul_rn(__fmul_rn(s, r), __fmaf_rn(u, u, __fmul_rn(s, s))) < 0.01f * kFaceRange;
        if (same && s > smax) smax = s;
    }
    if (!same) {
        St<float, NV> Fb, Ft;
        const float s_b = thin_face_mixed<RIEMANN>(a, gas, sb, 2, i, Fb), s_t = thin_face_mixed<RIEMANN>(a, gas, sb, 3, i, Ft);
        if (s_b > smax) smax = s_b;
        if (s_t > smax) smax = s_t;
#pragma unroll
        for (int q = 0; q < NV; ++q) acc[q] = __fmaf_rn(-(Ft[q] - Fb[q]), Ay, acc[q]);   // (an explicit FMA, as mixed_axis's balance)
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) a.out[q * m.plane + i] = cell_out(a, in, q, acc[q], dt);
}

template <int RECON, int RIEMANN, int TX, int TY, int NT>
__global__ void __launch_bounds__(NT) batch_mixed_kernel(const BatchArgs b) {
    using S = MixedShape<2, RECON, TX, TY, 1>;
    constexpr int NV = S::NV, NC = S::NC;
    extern __shared__ double smem_d[];
    double* red = smem_d;
    float* P = reinterpret_cast<float*>(smem_d + 32);
    float* WL = P + NV * S::EXT;
    float* WR = WL + NV * S::NF;
    float* acc = WR + NV * S::NF;
    unsigned char* Sf = reinterpret_cast<unsigned char*>(acc + NV * NC);
    __shared__ StageArgs sa;
    const int tid = threadIdx.x;
    int w0, w1, cur = -1;
    batch_share(*b.nwork, w0, w1);
    float smax = 0.0f;
    for (int w = w0; w < w1; ++w) {
        const BatchWork it = b.work[w];
        if (it.prob != cur) {
            if (cur >= 0) {
                const double bm = block_max<NT>((double)smax, red);
                if (tid == 0) batch_stage_max(&b.ctl[cur], b.stage, bm);
            }
            if (tid == 0) batch_item_args(b, b.prob[it.prob], sa);
            cur = it.prob;
            smax = 0.0f;
        }
        __syncthreads();
        const Mesh& m = sa.m;
        const GasF ef = gas_f(sa.eos);
        const float sb = (float)sa.shock_blend, weps = (float)sa.weno_eps;
        const int tx = (m.nx + TX - 1) / TX;
        const int o3[3] = {(it.tile % tx) * TX, (it.tile / tx) * TY, 0};
        const double dt = b.ctl[it.prob].dt;
        bool thin = false;
        if constexpr (TY == 1) {
            thin = thin_y(m, sa.bc);
            if (thin) thin_row_mixed<RECON, RIEMANN, TX, NT>(sa, ef, sb, weps, P, P + 4 * (NT + 8), o3[0], dt, smax);
        }
        if (!thin) {
            mixed_axis<0, 2, RECON, RIEMANN, TX, TY, 1, NT, false, false>(sa, ef, sb, weps, P, WL, WR, acc, Sf, o3, smax);
            mixed_axis<1, 2, RECON, RIEMANN, TX, TY, 1, NT, false, false>(sa, ef, sb, weps, P, WL, WR, acc, Sf, o3, smax);
            for (int c = tid; c < NC; c += NT) {
                const int i = o3[0] + c % TX, j = o3[1] + c / TX;
                if (i >= m.nx || j >= m.ny) continue;
                const long long cell = (long long)j * m.nx + i;
                CellIn<NV> in;
                cell_load(sa, cell, in);
#pragma unroll
                for (int q = 0; q < NV; ++q) sa.out[q * m.plane + cell] = cell_out(sa, in, q, acc[q * NC + c], dt);
            }
        }
    }
    if (cur >= 0) {
        const double bm = block_max<NT>((double)smax, red);
        if (tid == 0) batch_stage_max(&b.ctl[cur], b.stage, bm);
    }
}

template <int SHAPE, int RECON, int RIEMANN> struct MK {
    static constexpr BatchShape sh = kBatchShape[SHAPE];
    using S = MixedShape<2, RECON, sh.tx, sh.ty, 1>;
    static constexpr auto kern = batch_mixed_kernel<RECON, RIEMANN, sh.tx, sh.ty, sh.nt>;
    static cudaError_t prepare() { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM_BYTES); }
    static cudaError_t launch(const BatchArgs& a, int grid, cudaStream_t s) {
        kern<<<grid, sh.nt, S::SMEM_BYTES, s>>>(a);
        return cudaGetLastError();
    }
    static int resident() {
        int n = 0;
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, sh.nt, S::SMEM_BYTES) == cudaSuccess ? n : 0;
    }
    static BatchStage get() { return {prepare, launch, resident}; }
};

template <int SHAPE, int RECON> BatchStage pick_r(int riemann) {
    return riemann == kLowMach ? MK<SHAPE, RECON, kLowMach>::get() : MK<SHAPE, RECON, kHLLC>::get();
}
template <int SHAPE> BatchStage pick_s(int recon, int riemann) {
    switch (recon) {
    case kMuscl: return pick_r<SHAPE, kMuscl>(riemann);
    case kWeno3: return pick_r<SHAPE, kWeno3>(riemann);
    default: return pick_r<SHAPE, kWeno5>(riemann);
    }
}

}   // namespace

BatchStage batch_mixed_stage(int shape, int recon, int riemann) {
    switch (shape) {
    case 0: return pick_s<0>(recon, riemann);
    case 1: return pick_s<1>(recon, riemann);
    case 2: return pick_s<2>(recon, riemann);
    default: return pick_s<3>(recon, riemann);
    }
}

}   // namespace fvg
