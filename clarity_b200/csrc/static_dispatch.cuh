// static_dispatch.cuh -- compile-time specialised shapes and the launch
// helpers that use them when a plan matches (else the generic kernels run).
//
// Shapes (work box x*y*z -> x radices, Ay, y0 radices, z radices, G, W),
// exactly the plans the planner produces for these boxes:
//   512x512x128   (256x256x64 image + same-size PSF): 16.16, 16, 8.4, 16.8, 2, 2
//   128x128x64    (64x64x32 image + same-size PSF):   8.8,   16, 8,   8.8,  1, 4
//   1024x1024x256 (512x512x128 image + PSF):          8.8.8, 16, 8.8, 16.16, 2, 1
//   64x64x32      (small test box):                  8.4,   16, 4,   8.4,  4, 1
#pragma once
#include "engine.hpp"
#include "ops.cuh"
#include "passes_static.cuh"
#include "passes_xy_rows.cuh"
#include "passes_xy_tma.cuh"

namespace clarity {

using ShapeW512 = st::Shape<st::Rad<16, 16>, 16, st::Rad<8, 4>, st::Rad<16, 8>, 2, 2>;
using ShapeW128 = st::Shape<st::Rad<8, 8>, 16, st::Rad<8>, st::Rad<8, 8>, 1, 4>;
// The 1024x1024x256 box's XY and z tiles (133 and 128 KB) leave room for one
// block per SM, so its XY blocks without staged rows run CLARITY_W1024_THREADS
// threads and its FP32 z blocks CLARITY_W1024_Z_THREADS (both measured against
// 256; more threads in those XY passes spill registers; the staged ones, below,
// run 1024).  The tensor-core z form keeps the XY count.
#ifndef CLARITY_W1024_THREADS
#define CLARITY_W1024_THREADS 512
#endif
#ifndef CLARITY_W1024_Z_THREADS
#define CLARITY_W1024_Z_THREADS 1024
#endif
using ShapeW1024 = st::Shape<st::Rad<8, 8, 8>, 16, st::Rad<8, 8>, st::Rad<16, 16>, 2, 1,
                             CLARITY_W1024_THREADS, CLARITY_W1024_Z_THREADS>;
using ShapeW64 = st::Shape<st::Rad<8, 4>, 16, st::Rad<4>, st::Rad<8, 4>, 4, 1>;

template <class... SHs>
struct ShapeList {};
using StaticShapes = ShapeList<ShapeW512, ShapeW128, ShapeW1024, ShapeW64>;

inline st::Tables tables_of(const PlanEntry& pe) {
  const VolPlan& P = pe.P;
  return st::Tables{pe.tw + P.ax.tw_off, pe.tw + P.ayB.tw_off, pe.tw + P.az.tw_off,
                    pe.tw + P.tw_r2c_off, pe.tw + P.tw_ny_off, pe.err};
}

// Planes a launch covers: all of them, or those a functor says can be nonzero
// (or are wanted).
template <class F>
inline int launch_planes(const F& f, int nz) {
  if constexpr (requires { f.live_planes(nz); }) return f.live_planes(nz);
  else return nz;
}

template <class K>
inline cudaError_t allow_smem_st(K kernel, int smem) {
  return smem_opt_in(reinterpret_cast<const void*>(kernel), smem);
}

// The staged XY passes (passes_xy_tma.cuh, passes_xy_rows.cuh) serve epilogues
// with a staged form unless CLARITY_XY_TMA=0.
bool xy_tma_enabled();
template <class F>
constexpr bool xy_staged() {
  if constexpr (requires { F::kStaged; }) return F::kStaged;
  else return false;
}

// Tensor map of the spectrum S as floats {2*W*BY, NZ, KG, AY} with the box of
// one XY tile.
template <class SH, class X>
inline bool encode_s_map(TensorMap* tm, const float2* S) {
  const unsigned long long row = 2ull * SH::W * SH::BY;
  const unsigned long long dim[4] = {row, (unsigned long long)SH::NZ,
                                     (unsigned long long)SH::KG, (unsigned long long)SH::AY};
  const unsigned long long stride[3] = {row * 4, row * 4 * SH::NZ,
                                        row * 4 * SH::NZ * SH::KG};
  const unsigned box[4] = {2u * X::BOXW, 1u, (unsigned)X::KGB, (unsigned)SH::AY};
  return encode_tensor_f32_4d(tm, S, dim, stride, box);
}

// Launches the TMA XY pass on tiles X; false when its rows do not fit or the
// buffer cannot be mapped.
template <class SH, class X, bool FUSE, class F>
inline bool try_xy_tma_tile(const PlanEntry& pe, cudaStream_t st, const F& fn, const float2* S,
                            int family, cudaError_t* err) {
  static_assert(X::OK, "shape not supported by the TMA XY pass");
  const int stride = X::stage_stride(fn.stage_n());
  if (X::blocks_per_sm(stride) < 1) return false;
  // the map depends only on S: encoded once per buffer
  static thread_local const float2* map_s = nullptr;
  static thread_local TensorMap tm;
  if (S != map_s) {
    if (!encode_s_map<SH, X>(&tm, S)) {
      map_s = nullptr;
      return false;
    }
    map_s = S;
  }
  auto k = st::ks_xy_tma<SH, X, F, FUSE>;
  const int smem = X::smem(stride);
  *err = allow_smem_st(k, smem);
  if (*err != cudaSuccess) return true;
  const int blocks = launch_planes(fn, SH::NZ) * (SH::BY / X::TG);
  if (blocks <= 0) return true;
  note_launch_begin(family, st);
  CLARITY_LAUNCH_PDL(k, blocks, X::THREADS, smem, st, pdl_enabled())(fn, tm, tables_of(pe), stride);
  note_launch_end(family, st);
  *err = cudaGetLastError();
  return true;
}

// Launches the pass of passes_xy_rows.cuh on tiles X; false when its rows do
// not fit.
template <class SH, class X, bool FUSE, class F>
inline bool try_xy_rows_tile(const PlanEntry& pe, cudaStream_t st, const F& fn, float2* S,
                             int family, cudaError_t* err) {
  const int stride = X::stage_stride(fn.stage_n());
  if (!X::fits(stride)) return false;
  auto k = st::ks_xy_rows<SH, X, F, FUSE>;
  const int smem = X::smem(stride);
  *err = allow_smem_st(k, smem);
  if (*err != cudaSuccess) return true;
  const int blocks = launch_planes(fn, SH::NZ) * (SH::BY / X::TG);
  if (blocks <= 0) return true;
  note_launch_begin(family, st);
  CLARITY_LAUNCH_PDL(k, blocks, X::THREADS, smem, st, pdl_enabled())(fn, S, tables_of(pe), stride);
  note_launch_end(family, st);
  *err = cudaGetLastError();
  return true;
}

// The tiles of the staged XY passes.
//   * Rows of fewer than 256 complex: passes_xy_rows.cuh, 64 threads, keeping
//     half the rows where no line has more than AY/2 live ones (the image is at
//     most half the box).
//   * Else the TMA pass.  Boxes whose spectrum rows hold two columns (16 bytes a
//     line) take two lines and 512 threads where the staged rows leave room for
//     two such blocks per SM (whole sectors: product pass 91 -> 87 us); one line
//     otherwise.  The 1024x1024x256 box's two lines of 512 columns are one block
//     of 1024 threads per SM (ratio pass 1122 -> 965 us); rows too long to stage
//     beside them (a work-box volume's) keep the passes without staging.
template <class SH, bool FUSE, class F>
inline bool try_xy_staged(const PlanEntry& pe, cudaStream_t st, const F& fn, float2* S, int family,
                          cudaError_t* err) {
  if constexpr (xy_staged<F>()) {
    if (!xy_tma_enabled()) return false;
    if constexpr (SH::M < 256) {
      constexpr int TG = SH::W >= 4 ? 1 : 2;
      if constexpr (F::has_zero_rows)
        if (fn.live_rows(0, SH::BY, SH::AY) <= SH::AY / 2)
          return try_xy_rows_tile<SH, st::XyRows<SH, TG, 64, SH::AY / 2>, FUSE>(pe, st, fn, S,
                                                                               family, err);
      return try_xy_rows_tile<SH, st::XyRows<SH, TG, 64, SH::AY>, FUSE>(pe, st, fn, S, family, err);
    } else if constexpr (SH::W == 2 && SH::M == 256) {
      using X2 = st::XyTma<SH, 2, 512>;
      if (X2::blocks_per_sm(X2::stage_stride(fn.stage_n())) >= 2 &&
          try_xy_tma_tile<SH, X2, FUSE>(pe, st, fn, S, family, err))
        return true;
      return try_xy_tma_tile<SH, st::XyTma<SH, 1, 256>, FUSE>(pe, st, fn, S, family, err);
    } else if constexpr (SH::W == 1 && SH::M == 512) {
      return try_xy_tma_tile<SH, st::XyTma<SH, 2, 1024>, FUSE>(pe, st, fn, S, family, err);
    }
  }
  return false;
}

// Kernel families that may use the specialised kernels: bit KIND of the
// CLARITY_STATIC environment variable (default: all).  Clearing bits selects
// the runtime-generic kernels, which tests use to cover both paths.
int static_family_mask();

// kind: 0 xy forward, 1 z, 2 xy inverse+forward, 3 xy inverse
template <class SH, int KIND, class F>
inline bool try_static(const PlanEntry& pe, cudaStream_t st, const F& fn, float2* Sa,
                       const float2* Sb, cudaError_t* err) {
  if (!(static_family_mask() & (1 << KIND))) return false;
  if (!st::matches<SH>(pe.P)) return false;
  const st::Tables T = tables_of(pe);
  if constexpr (KIND == 0) {
    auto k = st::ks_xy_forward<SH, F>;
    *err = allow_smem_st(k, SH::XY_SMEM);
    if (*err != cudaSuccess) return true;
    note_launch_begin(KK_XY_FORWARD, st);
    CLARITY_LAUNCH(k, launch_planes(fn, SH::NZ) * SH::NGROUPS, SH::THREADS, SH::XY_SMEM, st)
    (fn, Sa, T);
    note_launch_end(KK_XY_FORWARD, st);
  } else if constexpr (KIND == 1) {
    if constexpr (SH::Y_PER_LINE) {
      auto k = st::ks_z2<SH, F>;
      *err = allow_smem_st(k, SH::Z2_SMEM);
      if (*err != cudaSuccess) return true;
      note_launch_begin(KK_Z, st);
      CLARITY_LAUNCH_PDL(k, pe.P.z_blocks, SH::THREADS, SH::Z2_SMEM, st, pdl_enabled())(fn, Sb,
                                                                                     Sa, T);
      note_launch_end(KK_Z, st);
    } else {
      using Z3 = st::Z3<st::ZThreads<SH>>;
      static_assert(Z3::OK, "a box with BY > 32 needs the W = 1 z kernel");
      int prec = st::kDftF32;
      if constexpr (st::kTcZ<SH> && !F::forward_only) {
        // the precision form: tensor-core first z stage (the OTF stays FP32)
        prec = dft_precision();
        if (prec != st::kDftF32) {
          auto k = prec == st::kDftF16Split ? st::ks_z<SH, F, st::kDftF16Split>
                                            : st::ks_z<SH, F, st::kDftBF16Split>;
          *err = allow_smem_st(k, SH::Z_SMEM);
          if (*err != cudaSuccess) return true;
          note_launch_begin(KK_Z, st);
          CLARITY_LAUNCH(k, pe.P.z_blocks, SH::THREADS, SH::Z_SMEM, st)(fn, Sb, Sa, T);
          note_launch_end(KK_Z, st);
        }
      }
      if (prec == st::kDftF32) {
        auto k = st::ks_z3<st::ZThreads<SH>, F>;
        *err = allow_smem_st(k, Z3::SMEM);
        if (*err != cudaSuccess) return true;
        note_launch_begin(KK_Z, st);
        CLARITY_LAUNCH_PDL(k, pe.P.z_blocks, SH::Z_THREADS, Z3::SMEM, st, pdl_enabled())(fn, Sb, Sa,
                                                                                      T);
        note_launch_end(KK_Z, st);
      }
    }
  } else if constexpr (KIND == 2) {
    if (try_xy_staged<SH, true>(pe, st, fn, Sa, family_of<F, KK_XY_INV_FWD>(), err)) return true;
    auto k = st::ks_xy_inv_fwd<SH, F>;
    *err = allow_smem_st(k, SH::XY_SMEM);
    if (*err != cudaSuccess) return true;
    note_launch_begin(family_of<F, KK_XY_INV_FWD>(), st);
    CLARITY_LAUNCH(k, launch_planes(fn, SH::NZ) * SH::NGROUPS, SH::THREADS, SH::XY_SMEM, st)
    (fn, Sa, T);
    note_launch_end(family_of<F, KK_XY_INV_FWD>(), st);
  } else {
    if (try_xy_staged<SH, false>(pe, st, fn, const_cast<float2*>(Sb), KK_XY_INVERSE, err)) return true;
    auto k = st::ks_xy_inverse<SH, F>;
    *err = allow_smem_st(k, SH::XY_SMEM);
    if (*err != cudaSuccess) return true;
    note_launch_begin(KK_XY_INVERSE, st);
    CLARITY_LAUNCH(k, launch_planes(fn, SH::NZ) * SH::NGROUPS, SH::THREADS, SH::XY_SMEM, st)
    (fn, Sb, T);
    note_launch_end(KK_XY_INVERSE, st);
  }
  *err = cudaGetLastError();
  return true;
}

template <int KIND, class F, class... SHs>
inline bool try_static_all(ShapeList<SHs...>, const PlanEntry& pe, cudaStream_t st,
                           const F& fn, float2* Sa, const float2* Sb, cudaError_t* err) {
  return (try_static<SHs, KIND>(pe, st, fn, Sa, Sb, err) || ...);
}

// Entry points used by launch.cuh; each returns true when a specialised
// kernel was launched (the error, if any, in *err).
template <class F>
bool static_xy_forward(const PlanEntry& pe, cudaStream_t st, const F& f, float2* S,
                       cudaError_t* err) {
  return try_static_all<0>(StaticShapes{}, pe, st, f, S, nullptr, err);
}
template <class F>
bool static_z(const PlanEntry& pe, cudaStream_t st, const F& f, const float2* Sin,
              float2* Sout, cudaError_t* err) {
  return try_static_all<1>(StaticShapes{}, pe, st, f, Sout, Sin, err);
}
template <class F>
bool static_xy_inv_fwd(const PlanEntry& pe, cudaStream_t st, const F& f, float2* S,
                       cudaError_t* err) {
  return try_static_all<2>(StaticShapes{}, pe, st, f, S, nullptr, err);
}
template <class F>
bool static_xy_inverse(const PlanEntry& pe, cudaStream_t st, const F& f, const float2* S,
                       cudaError_t* err) {
  return try_static_all<3>(StaticShapes{}, pe, st, f, nullptr, S, err);
}

}  // namespace clarity
