// spx_k_family.cuh -- launch and occupancy entry points of the stepping kernel for one
// trajectory family, arithmetic, field-derivative method and table kind (Euler and the classic RK4
// with unrolled constants, or any Butcher table from constant memory), and for the FP32 Parker kernels
// a diffusion class and boundary layout fixed at compile time, switching over the background classes.
// Each spx_k_*.cu instantiates it once, so the kernel sets compile in parallel.
#pragma once

#include "spx_launch.hh"
#include "spx_traj.cuh"

namespace spx {

template <int TT, class R, int DM, bool GT, int DK = -1, int BL = kLayoutAny>
struct FamilyTU {
   // dynamic shared memory: a header and the boundary states of every lane of a block
   static size_t smem(int slots, int block) { return kSmemHeader + (size_t)(slots > 0 ? slots : 1) * block * sizeof(BndState<R>); }

   // the guiding-centre family runs on static backgrounds only (no kernels for the moving shocks)
   template <int BG>
   static constexpr bool kBuilt = !(TT == kGuiding && (BG == kBgShock || BG == kBgSmoothShock));

   // Lorentz, and Parker with the diffusion class fixed, have the deep FP32 build too. (The generic Parker kernel has not:
   // at three blocks the compiler fuses other products of its run-time dispatch in the solar wind, and its trajectories
   // would no longer be those of the kernels compiled for a class.)
   static constexpr int kBlocks = sizeof(R) == 4 ? kWideBlocksF32 : kBlocksF64;
   static constexpr bool kHasDeep = sizeof(R) == 4 && ((TT == kParker && DK >= 0) || TT == kLorentz);

   template <int BG, int MB>
   static cudaError_t go_build(const LaunchArgs& a)
   {
      const auto* P = static_cast<const ProblemDescT<R>*>(a.problems_r);
      step_kernel<TT, BG, R, DM, GT, DK, BL, MB><<<a.grid, a.block, smem(a.bnd_slots, a.block.x), a.stream>>>(
          P, a.problems_d, a.cfg, a.ctr, a.counts, a.sums, a.n_events, a.records, a.queue);
      return cudaGetLastError();
   }

   template <int BG>
   static cudaError_t go(const LaunchArgs& a)
   {
      if constexpr (!kBuilt<BG>) return cudaErrorInvalidValue;
      else if constexpr (kHasDeep) return a.deep ? go_build<BG, kDeepBlocksF32>(a) : go_build<BG, kBlocks>(a);
      else return go_build<BG, kBlocks>(a);
   }

   template <int BG, int MB>
   static int occ_build(int block, int slots)
   {
      int n = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, step_kernel<TT, BG, R, DM, GT, DK, BL, MB>, block, smem(slots, block)) !=
          cudaSuccess)
         n = 0;
      return n;
   }

   // deep: the deep build's occupancy, 0 where there is none
   template <int BG>
   static int occ(int block, int slots, bool deep)
   {
      if constexpr (!kBuilt<BG>) return 0;
      else if constexpr (kHasDeep) return deep ? occ_build<BG, kDeepBlocksF32>(block, slots) : occ_build<BG, kBlocks>(block, slots);
      else return deep ? 0 : occ_build<BG, kBlocks>(block, slots);
   }

   static cudaError_t launch(int bg, const LaunchArgs& a)
   {
      switch (bg) {
      case kBgUniform: return go<kBgUniform>(a);
      case kBgShock: return go<kBgShock>(a);
      case kBgSmoothShock: return go<kBgSmoothShock>(a);
      case kBgDipole: return go<kBgDipole>(a);
      case kBgSolarWind: return go<kBgSolarWind>(a);
      case kBgGrid: return go<kBgGrid>(a);
      default: return cudaErrorInvalidValue;
      }
   }

   static int occupancy(int bg, int block, int slots, bool deep)
   {
      switch (bg) {
      case kBgUniform: return occ<kBgUniform>(block, slots, deep);
      case kBgShock: return occ<kBgShock>(block, slots, deep);
      case kBgSmoothShock: return occ<kBgSmoothShock>(block, slots, deep);
      case kBgDipole: return occ<kBgDipole>(block, slots, deep);
      case kBgSolarWind: return occ<kBgSolarWind>(block, slots, deep);
      case kBgGrid: return occ<kBgGrid>(block, slots, deep);
      default: return 0;
      }
   }
};

}  // namespace spx

// One translation unit: the kernels of one family, arithmetic, derivative method (DM 1: analytic
// field derivatives; DM 0: the reference's compiled-in numerical ones, FP64 only) and table kind
// (GT 1: any Butcher table, FP64 only).
// SPX_FAMILY_TU_DK: the FP32 analytic kernels with the diffusion class fixed at compile time (DK), and
// with it the boundary layout (BL, a BndLayout).
#define SPX_FAMILY_TU_DK(fam, prec, TT, DK, BL)                                                                    \
   namespace spx {                                                                                                  \
   cudaError_t launch_##fam##_##prec(int bg, const LaunchArgs& a) { return FamilyTU<TT, float, 1, false, DK, BL>::launch(bg, a); } \
   int occupancy_##fam##_##prec(int bg, int block, int slots, bool deep) { return FamilyTU<TT, float, 1, false, DK, BL>::occupancy(bg, block, slots, deep); } \
   }

#define SPX_FAMILY_TU(fam, prec, TT, R, DM, GT)                                                                    \
   namespace spx {                                                                                                  \
   cudaError_t launch_##fam##_##prec(int bg, const LaunchArgs& a) { return FamilyTU<TT, R, DM, GT>::launch(bg, a); } \
   int occupancy_##fam##_##prec(int bg, int block, int slots, bool deep) { return FamilyTU<TT, R, DM, GT>::occupancy(bg, block, slots, deep); } \
   }
