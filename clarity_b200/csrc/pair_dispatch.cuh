// pair_dispatch.cuh -- launches of the column-pair passes (passes_pair.cuh) of a
// box that has them; each class of each functor is instantiated in a kern_pair_*.cu
// (launch.cuh).
#pragma once
#include "engine.hpp"
#include "launch.cuh"
#include "ops.cuh"
#include "passes_pair.cuh"

namespace clarity {

template <class F>
inline int pair_grid(const PairPlan& P, const F& f) {
  int nz = P.nz;
  if constexpr (requires { f.live_planes(nz); }) nz = f.live_planes(nz);
  return nz * (P.By / P.TG);
}

template <class K, class... A>
inline cudaError_t pair_launch(K k, int grid, int threads, int smem, cudaStream_t st, int family,
                               const A&... args) {
  const cudaError_t e = smem_opt_in(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess || grid <= 0) return e;
  note_launch_begin(family, st);
  CLARITY_LAUNCH_PDL(k, grid, threads, smem, st, pdl_enabled())(args...);
  note_launch_end(family, st);
  return cudaGetLastError();
}

template <class Pro, bool BIG>
cudaError_t pair_xy_forward(const PlanEntry& pe, cudaStream_t st, const Pro& pro, float2* S) {
  const PairPlan& P = pe.pair;
  return pair_launch(pr::kp_xy_forward<Pro, BIG>, pair_grid(P, pro), P.xy_threads, P.xy_smem, st,
                     KK_XY_FORWARD, P, pro, S, (const float2*)pe.pair_tw,
                     (const int*)pe.pair_slots);
}

template <class Epi, bool FUSE, bool BIG>
cudaError_t pair_xy_inverse(const PlanEntry& pe, cudaStream_t st, const Epi& epi, float2* S) {
  const PairPlan& P = pe.pair;
  constexpr int family = FUSE ? family_of<Epi, KK_XY_INV_FWD>() : (int)KK_XY_INVERSE;
  return pair_launch(pr::kp_xy_inverse<Epi, FUSE, BIG>, pair_grid(P, epi), P.xy_threads, P.xy_smem,
                     st, family, P, epi, S, (const float2*)pe.pair_tw, (const int*)pe.pair_slots);
}

template <class Mod, bool BIG>
cudaError_t pair_z(const PlanEntry& pe, cudaStream_t st, const Mod& mod, const float2* Sin,
                   float2* Sout) {
  const PairPlan& P = pe.pair;
  pr::ZSpan Z;
  Z.zn = mod.zn < P.nz ? mod.zn : P.nz;
  Z.gap = (mod.zh < P.nz ? mod.zh : P.nz) - Z.zn;
  Z.zout = mod.zout < P.nz ? mod.zout : P.nz;
  Z.dlive = fdiv_by(P.nz - Z.gap);
  Z.dout = fdiv_by(Z.zout);
  return pair_launch(pr::kp_z<Mod, BIG>, P.z_blocks, P.z_threads, P.z_smem, st, KK_Z, P, Z, mod,
                     Sin, Sout, (const float2*)pe.pair_tw);
}

#define CLARITY_PAIR_FORWARD(F, BIG) \
  template cudaError_t pair_xy_forward<F, BIG>(const PlanEntry&, cudaStream_t, const F&, float2*);
#define CLARITY_PAIR_INVERSE(F, FUSE, BIG)                                                   \
  template cudaError_t pair_xy_inverse<F, FUSE, BIG>(const PlanEntry&, cudaStream_t, const F&, \
                                                     float2*);
#define CLARITY_PAIR_Z(F, BIG)                                                    \
  template cudaError_t pair_z<F, BIG>(const PlanEntry&, cudaStream_t, const F&, \
                                      const float2*, float2*);

}  // namespace clarity
