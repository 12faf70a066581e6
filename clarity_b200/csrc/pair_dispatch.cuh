// pair_dispatch.cuh -- launches of the column-pair passes (passes_pair.cuh).
// Each returns true when the plan has them (the launch's error in *err); the
// kernels are instantiated in kern_pair_*.cu.
#pragma once
#include "engine.hpp"
#include "ops.cuh"
#include "passes_pair.cuh"

namespace clarity {

// The emulation runs one thread per block, so the register classes do not
// differ there: one instantiation halves its build.
#ifdef CLARITY_HOST_EMULATION
constexpr bool kOneClass = true;
#else
constexpr bool kOneClass = false;
#endif

template <class F>
inline int pair_grid(const PairPlan& P, const F& f) {
  int nz = P.nz;
  if constexpr (requires { f.live_planes(nz); }) nz = f.live_planes(nz);
  return nz * (P.By / P.TG);
}

template <class K, class... A>
inline void pair_launch(K k, int grid, int threads, int smem, cudaStream_t st, int family,
                        cudaError_t* err, const A&... args) {
  *err = smem_opt_in(reinterpret_cast<const void*>(k), smem);
  if (*err != cudaSuccess || grid <= 0) return;
  note_launch_begin(family, st);
  CLARITY_LAUNCH_PDL(k, grid, threads, smem, st, pdl_enabled())(args...);
  note_launch_end(family, st);
  *err = cudaGetLastError();
}

template <class Pro>
bool pair_xy_forward(const PlanEntry& pe, cudaStream_t st, const Pro& pro, float2* S,
                     cudaError_t* err) {
  if (!pe.pair.ok) return false;
  const PairPlan& P = pe.pair;
  auto k = pr::kp_xy_forward<Pro, true>;
  if constexpr (!kOneClass && sizeof(Pro) > 0)
    if (!P.big_xy) k = pr::kp_xy_forward<Pro, false>;
  pair_launch(k, pair_grid(P, pro), P.xy_threads, P.xy_smem, st, KK_XY_FORWARD, err, P, pro, S,
              (const float2*)pe.pair_tw, (const int*)pe.pair_slots);
  return true;
}

template <class Epi, bool FUSE>
bool pair_xy_inverse(const PlanEntry& pe, cudaStream_t st, const Epi& epi, float2* S,
                     cudaError_t* err) {
  if (!pe.pair.ok) return false;
  const PairPlan& P = pe.pair;
  auto k = pr::kp_xy_inverse<Epi, FUSE, true>;
  if constexpr (!kOneClass && sizeof(Epi) > 0)
    if (!P.big_xy) k = pr::kp_xy_inverse<Epi, FUSE, false>;
  constexpr int family = FUSE ? family_of<Epi, KK_XY_INV_FWD>() : (int)KK_XY_INVERSE;
  pair_launch(k, pair_grid(P, epi), P.xy_threads, P.xy_smem, st, family, err, P, epi, S,
              (const float2*)pe.pair_tw, (const int*)pe.pair_slots);
  return true;
}

template <class Mod>
bool pair_z(const PlanEntry& pe, cudaStream_t st, const Mod& mod, const float2* Sin, float2* Sout,
            cudaError_t* err) {
  if (!pe.pair.ok) return false;
  const PairPlan& P = pe.pair;
  auto k = pr::kp_z<Mod, true>;
  if constexpr (!kOneClass && sizeof(Mod) > 0)
    if (!P.big_z) k = pr::kp_z<Mod, false>;
  pr::ZSpan Z;
  Z.zn = mod.zn < P.nz ? mod.zn : P.nz;
  Z.gap = (mod.zh < P.nz ? mod.zh : P.nz) - Z.zn;
  Z.zout = mod.zout < P.nz ? mod.zout : P.nz;
  Z.dlive = fdiv_by(P.nz - Z.gap);
  Z.dout = fdiv_by(Z.zout);
  pair_launch(k, P.z_blocks, P.z_threads, P.z_smem, st, KK_Z, err, P, Z, mod, Sin, Sout,
              (const float2*)pe.pair_tw);
  return true;
}

}  // namespace clarity
