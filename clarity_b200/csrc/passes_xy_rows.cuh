// passes_xy_rows.cuh -- the XY inverse (+ epilogue) (+ forward) pass of the
// small compile-time shapes, for epilogues whose real rows are staged: the pass
// of passes_xy_tma.cuh without the tensor copy.
//
// One block owns the tile (z, y0base .. y0base+TG-1): the rows y = y0 + BY*j of
// those TG y0 lines, of which only the LR first of each line can be live.
//   * Column step: one length-AY DFT per task, its AY values loaded straight
//     from the spectrum into registers.  Neighbouring lanes take the tile's
//     lines and neighbouring columns, so a warp's loads are whole sectors.  The
//     c2r pair combine of columns k and M - k exchanges values between lanes;
//     kx = 0 and kx = M share one DFT as the real and imaginary parts of one
//     complex column.
//   * The rows the epilogue reads (the RL estimate or the image) arrive in
//     shared memory meanwhile, by 16-byte asynchronous copies of all threads.
//   * x passes and epilogue as in passes_static.cuh; the epilogue's results go
//     straight to memory, and so do the forward column step's.
//
// Where a pass is one wave of short blocks, its time is a block's chain of
// latencies, and this one has no barrier and no copy through shared memory
// around the columns: RL on 64x64x32 (128x128x64 box) went from 30.7 to 27.0 us
// an iteration.  At the 512x512x128 box, with several waves to overlap, the
// tensor copy is the better one (RL product 70 us against 77, JVC 184 against
// 291).
#pragma once
#include "passes_static.cuh"
#ifdef CLARITY_HOST_EMULATION
#include <vector>
#endif

namespace clarity {
namespace st {

template <class SH, int TG_, int THR, int LR_>
struct XyRows {
  static constexpr int TG = TG_, LR = LR_, THREADS = THR;
  // the tile as a shape of its own, its lines' rows packed to LR
  struct T : Shape<typename SH::X, SH::AY, typename SH::Y, typename SH::Z, TG, SH::W, THR> {
    using B = Shape<typename SH::X, SH::AY, typename SH::Y, typename SH::Z, TG, SH::W, THR>;
    static constexpr int RAW = LR * B::ROWSTRIDE;
    static constexpr int GSTRIDE = RAW + (RAW % 16 == 0 ? 8 : 0);
  };
  static constexpr int M = SH::M, AY = SH::AY;
  static constexpr int TASKS = TG * M;  // column DFTs per tile
  static constexpr int ROWS_F2 = (TG * T::GSTRIDE + 1) / 2 * 2;
  // rows, then staged rows of `stride` floats, then the twiddles: x (M) and the
  // lines' y split (TG*AY)
  static constexpr int stage_stride(int n) { return (n + 3) / 4 * 4; }
  static constexpr int smem(int stride) {
    return ROWS_F2 * 8 + TG * LR * stride * 4 + (M + TG * AY) * 8;
  }
  static constexpr bool fits(int stride) { return smem(stride) + 2048 <= 227 * 1024; }
  static constexpr int MINB = THR >= 128 ? 1024 / THR : 12;  // 64 to 80 registers a thread
  static_assert(TASKS % THR == 0 && THR % 32 == 0 && (TG & (TG - 1)) == 0 && TG <= 16,
                "whole warps of column tasks, pair partners in one warp");
  static_assert(M % 2 == 0 && M >= 4 && AY % 2 == 0 && SH::BY % TG == 0, "shape");
};

// Column task c of the tile: line g = c % TG; within a line task 0 is the
// packed kx = 0 / kx = M pair, task 1 is kx = M/2 and tasks 2k, 2k+1 are kx = k
// and M - k for 0 < k < M/2 (lanes TG apart).
struct ColTask {
  int g, cc;
};
template <class X>
__device__ __forceinline__ ColTask col_task(int c) {
  return ColTask{c % X::TG, c / X::TG};
}
template <class X>
__device__ __forceinline__ int col_kx(int cc) {
  const int k = cc >> 1;
  return cc == 0 ? 0 : cc == 1 ? X::M / 2 : (cc & 1) ? X::M - k : k;
}

// Runs a(c, v) and b(c, v, other) for every column task c: other(j) is row j of
// the partner task (the column M - kx of the pair), by a warp shuffle; it must
// be called by every thread, in uniform control flow.  The CPU emulation, one
// thread per block, keeps every task's v in an array.
template <class X, class A, class B>
__device__ __forceinline__ void col_tasks_paired(const A& a, const B& b) {
#ifndef CLARITY_HOST_EMULATION
#pragma unroll 1
  for (int c = threadIdx.x; c < X::TASKS; c += X::THREADS) {
    float2 v[X::AY];
    a(c, v);
    auto other = [&](int j) {
      return make_float2(__shfl_xor_sync(0xffffffffu, v[j].x, X::TG),
                         __shfl_xor_sync(0xffffffffu, v[j].y, X::TG));
    };
    b(c, v, other);
  }
#else
  std::vector<float2> regs((size_t)X::TASKS * X::AY);
  for (int c = 0; c < X::TASKS; ++c) a(c, &regs[(size_t)c * X::AY]);
  for (int c = 0; c < X::TASKS; ++c) {
    const float2* o = &regs[(size_t)(c ^ X::TG) * X::AY];
    auto other = [o](int j) { return o[j]; };
    b(c, &regs[(size_t)c * X::AY], other);
  }
#endif
}

// Inverse column step: spectrum -> x rows (digit-reversed slots), rows j < L.
template <class SH, class X>
__device__ __forceinline__ void cols_inverse_rows(float2* buf, const float2* S, int z, int y0base,
                                                  const float2* __restrict__ twr,
                                                  const float2* twl, int L) {
  using T = typename X::T;
  constexpr int M = X::M, AY = X::AY, RS = T::ROWSTRIDE;
  auto load = [&](int c, float2* v) {
    const ColTask t = col_task<X>(c);
    const int y0 = y0base + t.g;
    const float2* src = S + sbase<SH>(col_kx<X>(t.cc), z, y0);
#pragma unroll
    for (int k1 = 0; k1 < AY; ++k1) v[k1] = ld_l2(src + k1 * kK1Stride<SH>);
    if (t.cc == 0) {
      // A + i B with B the kx = M column: one inverse DFT gives a + i b
      const float2* sb = S + sbase<SH>(M, z, y0);
#pragma unroll
      for (int k1 = 0; k1 < AY; ++k1) {
        const float2 b = ld_l2(sb + k1 * kK1Stride<SH>);
        v[k1] = make_float2(v[k1].x - b.y, v[k1].y + b.x);
      }
    }
    if (y0 != 0) {
#pragma unroll
      for (int k1 = 1; k1 < AY; ++k1) v[k1] = cmulc(v[k1], twl[t.g * AY + k1]);
    }
    dft<AY, +1>(v);
  };
  auto store = [&](int c, const float2* v, const auto& other) {
    const ColTask t = col_task<X>(c);
    const int cc = t.cc;
    float2* rows = buf + t.g * T::GSTRIDE;
    // pair (k, M - k), 0 < k < M/2: the even task holds X[k], the odd X[M-k]
    const bool pair = cc >= 2, odd = (cc & 1) != 0;
    const int p = xp<T>(xrev<T>(col_kx<X>(cc)));
    const float2 w = pair ? __ldg(&twr[cc >> 1]) : make_float2(1.f, 0.f);
#pragma unroll
    for (int j = 0; j < X::LR; ++j) {
      if (j >= L) continue;  // L is the same for every thread
      const float2 ov = other(j);
      if (cc == 0) {
        rows[j * RS + p] = make_float2(v[j].x + v[j].y, v[j].x - v[j].y);
      } else if (cc == 1) {
        rows[j * RS + p] = make_float2(2.f * v[j].x, -2.f * v[j].y);
      } else {
        const float2 xa = odd ? ov : v[j];
        const float2 b = conjf2(odd ? v[j] : ov);
        const float2 e = cadd(xa, b);
        const float2 o = cmulc(csub(xa, b), w);
        rows[j * RS + p] = odd ? make_float2(e.x + o.y, -e.y + o.x)
                               : make_float2(e.x - o.y, e.y + o.x);
      }
    }
  };
  col_tasks_paired<X>(load, store);
}

// Forward DFT of length AY whose inputs from LR on are zero.
template <int AY, int LR>
__device__ __forceinline__ void dft_low(float2* v) {
  if constexpr (AY == 16 && LR == 8) {
    // first radix-4 stage on two of its four inputs
    float2 u[16];
    static_for<4>([&](auto ii) {
      constexpr int i = decltype(ii)::value;
      const float2 a = v[i], b = v[i + 4];
      u[i] = cadd(a, b);
      u[i + 4] = twc<i, 16, -1>(cadd_diri<-1>(a, b));
      u[i + 8] = twc<2 * i, 16, -1>(csub(a, b));
      u[i + 12] = twc<3 * i, 16, -1>(cadd_diri<+1>(a, b));
    });
    static_for<4>([&](auto ki) {
      constexpr int k = decltype(ki)::value;
      dft<4, -1>(u + 4 * k);
      static_for<4>([&](auto ji) {
        constexpr int j = decltype(ji)::value;
        v[k + 4 * j] = u[4 * k + j];
      });
    });
  } else {
#pragma unroll
    for (int j = LR; j < AY; ++j) v[j] = make_float2(0.f, 0.f);
    dft<AY, -1>(v);
  }
}

// Forward column step: x rows (digit-reversed slots) -> spectrum.  The r2c
// split of slots k and M - k happens as the columns are read: both tasks of a
// pair read both slots and each keeps its own half.  Rows j >= L are zero.
template <class SH, class X>
__device__ __forceinline__ void cols_forward_rows(const float2* buf, float2* S, int z, int y0base,
                                                  const float2* __restrict__ twr,
                                                  const float2* twl, int L) {
  using T = typename X::T;
  constexpr int M = X::M, AY = X::AY, RS = T::ROWSTRIDE;
#pragma unroll 1
  for (int c = threadIdx.x; c < X::TASKS; c += CLARITY_BLOCK_STRIDE(X::THREADS)) {
    const ColTask t = col_task<X>(c);
    const int cc = t.cc, kx = col_kx<X>(cc), y0 = y0base + t.g;
    const float2* rows = buf + t.g * T::GSTRIDE;
    const int pa = xp<T>(xrev<T>(cc >= 2 ? cc >> 1 : kx));
    const int pb = xp<T>(xrev<T>(cc >= 2 ? M - (cc >> 1) : kx));
    const float2 w = cc >= 2 ? __ldg(&twr[cc >> 1]) : make_float2(1.f, 0.f);
    const bool odd = (cc & 1) != 0;
    float2 v[AY];
#pragma unroll
    for (int j = 0; j < X::LR; ++j) {
      if (j >= L) {
        v[j] = make_float2(0.f, 0.f);
        continue;
      }
      const float2 a = rows[j * RS + pa];
      if (cc == 0) {
        v[j] = make_float2(a.x + a.y, a.x - a.y);
      } else if (cc == 1) {
        v[j] = conjf2(a);
      } else {
        // pair (k, M - k): the even task keeps X[k], the odd X[M - k]
        const float2 b = conjf2(rows[j * RS + pb]);
        const float2 e = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
        const float2 d = csub(a, b);
        const float2 o = make_float2(0.5f * d.y, -0.5f * d.x);
        const float2 wo = cmul(w, o);
        v[j] = odd ? conjf2(csub(e, wo)) : cadd(e, wo);
      }
    }
    dft_low<AY, X::LR>(v);
    float2* dst = S + sbase<SH>(kx, z, y0);
    if (cc == 0) {
      // kx = 0 and kx = M have real columns a, b: one DFT of a + i b gives
      // P = A + i B with A[k] = (P[k] + conj P[-k]) / 2 and
      // B[k] = (P[k] - conj P[-k]) / 2i
      float2* db = S + sbase<SH>(M, z, y0);
#pragma unroll
      for (int k = 0; k < AY; ++k) {
        const float2 p = v[k], q = v[(AY - k) % AY], wl = twl[t.g * AY + k];
        dst[k * kK1Stride<SH>] =
            cmul(make_float2(0.5f * (p.x + q.x), 0.5f * (p.y - q.y)), wl);
        db[k * kK1Stride<SH>] = cmul(make_float2(0.5f * (p.y + q.y), 0.5f * (q.x - p.x)), wl);
      }
    } else {
#pragma unroll
      for (int k1 = 0; k1 < AY; ++k1) dst[k1 * kK1Stride<SH>] = cmul(v[k1], twl[t.g * AY + k1]);
    }
  }
}

// Last inverse x pass into the epilogue with the tile's real rows staged (SS
// floats apart); FUSE re-applies forward pass 0.
template <class X, class Epi, bool FUSE, class Skip, bool COMPACT>
__device__ __forceinline__ void x_last_rows(float2* sm, const float* stg, Epi& epi, int z,
                                              int y0base, const float2* tw, const Skip& skip,
                                              int L, int SS) {
  using T = typename X::T;
  using XR = typename T::X;
  constexpr int R = XR::radix(0), span = XR::span(0);
  const int total = visit_rows<T, COMPACT>(L) * span;
#pragma unroll 1
  for (int f = threadIdx.x; f < total; f += CLARITY_BLOCK_STRIDE(T::THREADS)) {
    const int rv = f / span;
    const int r = visit_row<T, COMPACT>(rv, L);
    const int i = f - rv * span;
    const int g = r / T::AY, j = r - g * T::AY;
    const int y = y0base + g + T::BY * j;
    float2* row = sm + row_off<T>(r);
    if (skip(r)) {  // known-zero row: its forward transform is zero
      if constexpr (FUSE) {
#pragma unroll
        for (int t = 0; t < R; ++t) row[xp<T>(i + t * span)] = make_float2(0.f, 0.f);
      }
      continue;
    }
    float2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = row[xp<T>(i + t * span)];
    if (i != 0) {
#pragma unroll
      for (int k = 1; k < R; ++k) v[k] = cmulc(v[k], tw[i * k]);
    }
    dft<R, +1>(v);
    const float* srow = stg + (g * X::LR + j) * SS;
    const int n = epi.in_row(y, z).nf;
#pragma unroll
    for (int t = 0; t < R; ++t) {
      // beyond the longest row, for every thread alike: zero, nothing to do
      if (2 * t * span >= epi.row_n()) v[t] = make_float2(0.f, 0.f);
      else v[t] = epi.apply_s(i + t * span, y, z, v[t], srow, n);
    }
    if constexpr (FUSE) {
      dft<R, -1>(v);
      if (i != 0) {
#pragma unroll
        for (int k = 1; k < R; ++k) v[k] = cmul(v[k], tw[i * k]);
      }
#pragma unroll
      for (int t = 0; t < R; ++t) row[xp<T>(i + t * span)] = v[t];
    }
  }
}

// The pass kernel.  FUSE = false is the final inverse (no forward transform, S
// is only read).
template <class SH, class X, class Epi, bool FUSE>
__global__ void __launch_bounds__(X::THREADS, X::MINB)
    ks_xy_rows(Epi epi, float2* S, const Tables T, const int SS) {
  using TS = typename X::T;
  CLARITY_DYN_SMEM(float2, buf);
  float* stg = reinterpret_cast<float*>(buf + X::ROWS_F2);
  float2* twx = reinterpret_cast<float2*>(stg + X::TG * X::LR * SS);
  float2* twl = twx + X::M;
  constexpr int NB = SH::BY / X::TG;
  const int z = blockIdx.x / NB;
  const int y0base = (blockIdx.x - z * NB) * X::TG;
  // twiddles into shared memory, before the previous pass has finished: the x
  // table w_M^t and the lines' y split factors w_ny^(y0*k1)
  for (int t = threadIdx.x; t < X::M; t += CLARITY_BLOCK_STRIDE(X::THREADS)) twx[t] = __ldg(&T.twx[t]);
  for (int t = threadIdx.x; t < X::TG * X::AY; t += CLARITY_BLOCK_STRIDE(X::THREADS)) {
    const int g = t / X::AY, k1 = t - g * X::AY;
    twl[t] = __ldg(&T.twny[(y0base + g) * k1]);
  }
  CLARITY_PDL_WAIT();  // the previous pass's output is complete and visible
  if constexpr (requires { epi.prepare(); }) epi.prepare();
  // rows j >= L of every line are outside the image (zero for this epilogue)
  constexpr bool CP = Epi::has_zero_rows;
  int L = X::LR;
  if constexpr (CP) {
    L = epi.live_rows(y0base, SH::BY, SH::AY);
    if (L > X::LR) L = X::LR;  // never: the launch chose LR for the most live rows
  }
  // image rows an epilogue reads in place, into L2
  if constexpr (requires { epi.prefetch_image(0, 0); })
    for (int r = threadIdx.x; r < X::TG * X::LR; r += CLARITY_BLOCK_STRIDE(X::THREADS))
      epi.prefetch_image(y0base + r / X::LR + SH::BY * (r % X::LR), z);
  // the real rows the epilogue reads, SS floats apart (SS a multiple of 4)
  for (int t = threadIdx.x; t < X::TG * X::LR * (SS / 4); t += CLARITY_BLOCK_STRIDE(X::THREADS)) {
    const int r = t / (SS / 4), x = 4 * (t - r * (SS / 4));
    const RowRef rr = epi.in_row(y0base + r / X::LR + SH::BY * (r % X::LR), z);
    if (x + 4 <= rr.nf && ((uintptr_t)(rr.p + x) & 15u) == 0) {
      cp_async16(stg + r * SS + x, rr.p + x);
    } else {  // a row that is not a 16-byte run, or its end
      for (int e = x; e < x + 4 && e < rr.nf; ++e) stg[r * SS + e] = ld_l2(rr.p + e);
    }
  }
  __syncthreads();  // the twiddles
  cols_inverse_rows<SH, X>(buf, S, z, y0base, T.twr, twl, L);
  cp_async_wait_all();
  __syncthreads();
  const RowSkip<TS, Epi> skip{epi, z, y0base};
  x_inverse_down_to<TS, 1, RowSkip<TS, Epi>, CP>(buf, twx, skip, L);
  x_last_rows<X, Epi, FUSE, RowSkip<TS, Epi>, CP>(buf, stg, epi, z, y0base, twx, skip, L, SS);
  if constexpr (FUSE) {
    __syncthreads();
    x_forward_from<TS, 1, RowSkip<TS, Epi>, CP>(buf, twx, skip, L);
    cols_forward_rows<SH, X>(buf, S, z, y0base, T.twr, twl, L);
  }
  epi.finish();
}

}  // namespace st
}  // namespace clarity
