// The mixed-precision kernels' translation unit (see mixed.cuh). Built with --use_fast_math: FP32 division and square
// root are the fast approximations and multiplies and adds may contract into FMAs, except where mixed.cuh rounds each
// operation explicitly (the face values, the balance, the FP64 update); FP64 division and square root stay IEEE.
#include "mixed.cuh"
#include "march.cuh"
#include "mixed_api.h"

namespace fvg {
namespace {

template <int DIM> struct MTile;
// 3-D: 384 threads per 8x8x8 tile, three CTAs per SM (36 warps; 2.85 ms per launch at 256^3 against 3.52 with 192 threads)
template <> struct MTile<3> { static constexpr int X = 8, Y = 8, Z = 8, NT = 384; };
template <> struct MTile<2> { static constexpr int X = 16, Y = 15, Z = 1, NT = 256; };

// the marching kernels (march.cuh): the WENO5-Z lean kernels, where marches
template <int DIM, int RECON, bool FULL> constexpr bool kHasMarch = RECON == kWeno5 && !FULL;
template <int DIM, int RIEMANN, bool GATED> using MarchOf = std::conditional_t<DIM == 3, MarchK<RIEMANN, GATED>, March2K<RIEMANN, GATED>>;

template <int DIM, int RECON, int RIEMANN, bool FULL> struct MixedK {
    using T = MTile<DIM>;
    using S = MixedShape<DIM, RECON, T::X, T::Y, T::Z>;
    static cudaError_t prepare() {
        cudaError_t e = cudaFuncSetAttribute(mixed_stage_kernel<DIM, RECON, RIEMANN, T::X, T::Y, T::Z, T::NT, false, FULL>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM_BYTES);
        if constexpr (kHasMarch<DIM, RECON, FULL>)
            if (e == cudaSuccess) e = MarchOf<DIM, RIEMANN, false>::prepare();
        return e;
    }
    static cudaError_t launch(const StageArgs& a, int nblocks, cudaStream_t s) {
        if constexpr (kHasMarch<DIM, RECON, FULL>) {
            MarchLaunch l;
            if (marches(a, DIM, nblocks, l)) return MarchOf<DIM, RIEMANN, false>::launch(a, l, nblocks, s);
        }
        mixed_stage_kernel<DIM, RECON, RIEMANN, T::X, T::Y, T::Z, T::NT, false, FULL><<<nblocks, T::NT, S::SMEM_BYTES, s>>>(a);
        return cudaGetLastError();
    }
};

// the WENO5-Z kernels gated by the learned sensor
template <int DIM, int RIEMANN, bool FULL> struct GatedK {
    using T = MTile<DIM>;
    using S = MixedShape<DIM, kWeno5, T::X, T::Y, T::Z>;
    static cudaError_t prepare() {
        cudaError_t e = cudaFuncSetAttribute(mixed_stage_kernel<DIM, kWeno5, RIEMANN, T::X, T::Y, T::Z, T::NT, true, FULL>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM_BYTES);
        if constexpr (kHasMarch<DIM, kWeno5, FULL>)
            if (e == cudaSuccess) e = MarchOf<DIM, RIEMANN, true>::prepare();
        return e;
    }
    static cudaError_t launch(const StageArgs& a, int nblocks, cudaStream_t s) {
        if constexpr (kHasMarch<DIM, kWeno5, FULL>) {
            MarchLaunch l;
            if (marches(a, DIM, nblocks, l)) return MarchOf<DIM, RIEMANN, true>::launch(a, l, nblocks, s);
        }
        mixed_stage_kernel<DIM, kWeno5, RIEMANN, T::X, T::Y, T::Z, T::NT, true, FULL><<<nblocks, T::NT, S::SMEM_BYTES, s>>>(a);
        return cudaGetLastError();
    }
};

template <int DIM, int RECON, bool FULL> MixedStage pick_r(int riemann) {
    if (riemann == kLowMach) return {MixedK<DIM, RECON, kLowMach, FULL>::prepare, MixedK<DIM, RECON, kLowMach, FULL>::launch};
    return {MixedK<DIM, RECON, kHLLC, FULL>::prepare, MixedK<DIM, RECON, kHLLC, FULL>::launch};
}
template <int DIM, bool FULL> MixedStage pick(int recon, int riemann) {
    switch (recon) {
    case kMuscl: return pick_r<DIM, kMuscl, FULL>(riemann);
    case kWeno3: return pick_r<DIM, kWeno3, FULL>(riemann);
    default: return pick_r<DIM, kWeno5, FULL>(riemann);
    }
}
template <int DIM, bool FULL> MixedStage pick_gated(int riemann) {
    return riemann == kLowMach ? MixedStage{GatedK<DIM, kLowMach, FULL>::prepare, GatedK<DIM, kLowMach, FULL>::launch}
                               : MixedStage{GatedK<DIM, kHLLC, FULL>::prepare, GatedK<DIM, kHLLC, FULL>::launch};
}

}   // namespace

// full: the kernels with the code of part interfaces and non-reflecting sides; else the lean instantiation
MixedStage mixed_stage(int dim, int recon, int riemann, bool full) {
    if (dim == 3) return full ? pick<3, true>(recon, riemann) : pick<3, false>(recon, riemann);
    return full ? pick<2, true>(recon, riemann) : pick<2, false>(recon, riemann);
}

MixedStage mixed_stage_gated(int dim, int riemann, bool full) {
    if (dim == 3) return full ? pick_gated<3, true>(riemann) : pick_gated<3, false>(riemann);
    return full ? pick_gated<2, true>(riemann) : pick_gated<2, false>(riemann);
}

// the FP32 viscous sweep: the marching kernel where every side of the whole mesh is periodic and no body is immersed, else
// 8x8x8 tiles of 384 threads. (By the configuration's sides, which the parts of a decomposed mesh share: the two sweeps round
// their gradients differently, and both parts beside an interface must give its faces the same flux. An inner part of a mesh
// with walls has none itself.)
constexpr int kMixedViscNT = 384;
cudaError_t mixed_viscous_prepare() {
    cudaError_t e = cudaFuncSetAttribute(mixed_viscous_kernel<8, 8, 8, kMixedViscNT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)MixedViscShape<8, 8, 8>::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mixed_viscous_march_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ViscMarchShape::SMEM_BYTES);
    return e;
}
bool mixed_stage_marches(const StageArgs& a, int dim, int nblocks) {
    MarchLaunch l;
    return marches(a, dim, nblocks, l);
}
cudaError_t mixed_viscous_launch(const ViscArgs& a, int nblocks, cudaStream_t s) {
    if (a.all_periodic && !a.bc.slot) return visc_march_launch(a, nblocks, s);
    mixed_viscous_kernel<8, 8, 8, kMixedViscNT><<<nblocks, kMixedViscNT, MixedViscShape<8, 8, 8>::SMEM_BYTES, s>>>(a);
    return cudaGetLastError();
}

}   // namespace fvg
