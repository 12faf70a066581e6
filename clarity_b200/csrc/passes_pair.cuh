// passes_pair.cuh -- the fused FFT passes for work boxes without compile-time
// kernels, on pairs of columns (plan.hpp: PairPlan).
//
// What bounds these passes is issue slots and the latency of a block's chain
// of shared-memory sweeps, not memory: at the 320x320x96 box the spectrum is
// 40 MB and stays in L2.  Hence
//   * two transforms per thread in packed FP32 (dft_pair.cuh): columns kx and
//     kx+1 in the y and z passes, two row pairs in the x passes, one 16-byte
//     shared-memory access per element of both;
//   * x transforms of row pairs (row 2p + i row 2p+1): the r2c split and the
//     c2r combine are additions inside the column step, for odd nx too;
//   * columns straight between HBM/L2 and the column step's registers, and
//     only live row quads and planes transformed;
//   * the spectral operation inside the last z pass, the y0 axis in one
//     register pass where By allows;
//   * as many threads as a pass has items, several blocks per SM;
//   * programmatic dependent launch: a kernel's blocks are placed while the one
//     before drains.  What an earlier kernel may have written is read through
//     L2 (ld_l2, bulk copies), never through the read-only cache.
//
// Measured on one B200 against the runtime-planned passes (passes.cuh), which
// run 128 registers at two blocks per SM and scalar arithmetic: RL, 20
// iterations, 256x256x64 with a 64x64x32 PSF (320x320x96 box) 11.7 -> 5.3 ms;
// 140x126x36 with 31x21x13 (171x147x49) 4.3 -> 1.7 ms; 12 uneven volumes, 5
// iterations, 35.2 -> 17.7 ms.
#pragma once
#include "launch_macro.cuh"

#include "dft_pair.cuh"
#include "ops.cuh"
#include "passes.cuh"
#include "plan.hpp"
#include "tma.cuh"

namespace clarity {
namespace pr {

// Threads per block and blocks per SM the registers are sized for: radices up
// to 16 hold 64 floats of data a thread (128 registers), 17 and 19 more.
template <bool BIG>
struct Cls {
  static constexpr int MAXT = BIG ? 128 : 256;
  static constexpr int MAXR = BIG ? 19 : 16;
};

// Calls f(ic<R>{}) for the runtime radix r.
template <int MAXR, class F>
__device__ __forceinline__ void with_radix(int r, const F& f) {
  switch (r) {
#define CLARITY_RADIX_CASE(RR)                     \
  case RR:                                         \
    if constexpr (RR <= MAXR) f(ic<RR>{});         \
    break;
    CLARITY_RADIX_CASE(1)
    CLARITY_RADIX_CASE(14)
    CLARITY_RADIX_CASE(15)
    CLARITY_FOR_EACH_RADIX(CLARITY_RADIX_CASE)
#undef CLARITY_RADIX_CASE
    default:
      break;
  }
}

__device__ __forceinline__ c2 get(const float4& q) {
  return c2{make_float2(q.x, q.y), make_float2(q.z, q.w)};
}
__device__ __forceinline__ float4 put(const c2& v) {
  return make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// v[k] *= w_n^(DIR k i) (DIR = -1 forward: the table's w; +1: conjugate); W:
// float2 entries, or float4 with both parts twice
template <int R, int DIR, class W>
__device__ __forceinline__ void twiddle(c2* v, const W* tw, int i) {
  if (i == 0) return;
#pragma unroll
  for (int k = 1; k < R; ++k)
    v[k] = DIR < 0 ? pcmul(v[k], tw[i * k]) : pcmulc(v[k], tw[i * k]);
}

// ------------------------------------------------------------------ z tile
// Planes of a z pass: the live input planes z < zn and z >= zn + gap, the
// wanted output planes z < zout, and division by their numbers.
struct ZSpan {
  int zn, gap, zout;
  FDiv dlive, dout;
};

// y0 register pass s over `planes` planes (the q-th is q, or q + gap beyond
// zn): consecutive threads take consecutive planes (odd stride BS).
template <int R, int DIR>
__device__ __forceinline__ void y0_pass(float4* sm, const PairPlan& P, int s, int planes,
                                        FDiv dplanes, int zn, int gap, const float4* tw) {
  const int len = P.ayB.len[s], span = P.ayB.span[s], step = P.By / len;
  const int total = planes * (P.By / R);
  const FDiv Ds = P.ayB.dspan[s];
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int rem = quot(f, dplanes), q = f - rem * planes;
    const int z = q < zn ? q : q + gap;
    const int b = quot(rem, Ds), i = rem - b * span;
    float4* p = sm + z * P.BS + b * len + i;
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = get(p[t * span]);
    if constexpr (DIR > 0) twiddle<R, DIR>(v, tw, i * step);
    pdft<R, DIR>(v);
    if constexpr (DIR < 0) twiddle<R, DIR>(v, tw, i * step);
#pragma unroll
    for (int t = 0; t < R; ++t) p[t * span] = put(v[t]);
  }
}

// z register pass s (not the last): lines l0 = y0, adjacent in memory.
template <int R, int DIR>
__device__ __forceinline__ void z_pass(float4* sm, const PairPlan& P, int s, const float4* tw) {
  const int len = P.az.len[s], span = P.az.span[s], step = P.nz / len;
  const int total = P.By * (P.nz / R), es = span * P.BS;
  const FDiv Ds = P.az.dspan[s];
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int rem = quot(f, P.dBy), l0 = f - rem * P.By;
    const int b = quot(rem, Ds), i = rem - b * span;
    float4* p = sm + l0 + (b * len + i) * P.BS;
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = get(p[t * es]);
    if constexpr (DIR > 0) twiddle<R, DIR>(v, tw, i * step);
    pdft<R, DIR>(v);
    if constexpr (DIR < 0) twiddle<R, DIR>(v, tw, i * step);
#pragma unroll
    for (int t = 0; t < R; ++t) p[t * es] = put(v[t]);
  }
}

// Last z pass (span 1), spectral operation, first inverse pass; or (forward
// only) the spectrum's store.  gbase: the tile's offset in S.
template <int R, class Mod>
__device__ __forceinline__ void z_mod(float4* sm, const PairPlan& P, const Mod& mod,
                                      unsigned gbase, float4* CLARITY_RESTRICT out) {
  const int total = P.By * (P.nz / R);
  const Mod m = mod.resolved();
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int b = quot(f, P.dBy), l0 = f - b * P.By;
    float4* p = sm + l0 + b * R * P.BS;
    const unsigned g = gbase + (unsigned)(b * R) * P.By + l0;
    // the OTF's elements ahead of the transform (in groups beyond radix 8), so
    // their latencies overlap
    constexpr int CH = R <= 8 ? R : 4;
    float4 hv[CH];
    [[maybe_unused]] auto preload = [&](int t0) {
      if constexpr (!Mod::forward_only) {
        const float4* h = reinterpret_cast<const float4*>(m.H) + g;
#pragma unroll
        for (int t = 0; t < CH; ++t)
          if (t0 + t < R) hv[t] = ld_l2(&h[(t0 + t) * P.By]);
      }
    };
    if constexpr (CH == R) preload(0);
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = get(p[t * P.BS]);
    pdft<R, -1>(v);
    if constexpr (Mod::forward_only) {
#pragma unroll
      for (int t = 0; t < R; ++t) out[g + t * P.By] = put(v[t]);
    } else {
#pragma unroll
      for (int t0 = 0; t0 < R; t0 += CH) {
        if constexpr (CH < R) preload(t0);
#pragma unroll
        for (int t = 0; t < CH; ++t)
          if (t0 + t < R) v[t0 + t] = m.pair(hv[t], v[t0 + t]);
      }
      pdft<R, +1>(v);
#pragma unroll
      for (int t = 0; t < R; ++t) p[t * P.BS] = put(v[t]);
    }
  }
}

// One block per tile S[k1][kg]: nz rows of By slots, padded to BS in shared
// memory (dead planes zeroed there).
template <class Mod, bool BIG>
__global__ void __launch_bounds__(Cls<BIG>::MAXT, 2)
    kp_z(CLARITY_GRID_CONST PairPlan P, const ZSpan Z, Mod mod, const float2* Sin_,
         float2* Sout_, const float2* CLARITY_RESTRICT tables) {
  CLARITY_DYN_SMEM(float4, sm);
  constexpr int MAXR = Cls<BIG>::MAXR;
  const unsigned gbase = blockIdx.x * (unsigned)(P.nz * P.By);
  const float4* Sin = reinterpret_cast<const float4*>(Sin_) + gbase;
  float4* Sout = reinterpret_cast<float4*>(Sout_);
  float4* twz = sm + P.nz * P.BS;
  float4* twy = twz + P.nz;
  for (int t = threadIdx.x; t < P.nz; t += blockDim.x)
    twz[t] = twin(CLARITY_LDG(&tables[P.az.tw_off + t]));
  for (int t = threadIdx.x; t < P.By; t += blockDim.x)
    twy[t] = twin(CLARITY_LDG(&tables[P.ayB.tw_off + t]));
  CLARITY_PDL_WAIT();  // the previous kernel's output is complete and visible
  // the OTF tile this block will multiply by, into L2
  if (threadIdx.x < 4) mod.prefetch_tile(gbase * 2u, P.nz * P.By * 2, threadIdx.x, 4);
  // plain 16-byte loads: a bulk copy per plane costs more issue slots than the
  // few loads a thread has here
#pragma unroll 4
  for (int f = threadIdx.x; f < P.nz * P.By; f += blockDim.x) {
    const int z = quot(f, P.dBy);
    sm[f + z * (P.BS - P.By)] = z < Z.zn || z >= Z.zn + Z.gap ? ld_l2(&Sin[f]) : zero4();
  }
  mod.late();
  __syncthreads();
  const int nlive = P.nz - Z.gap;
  for (int s = 0; s < P.ayB.npass; ++s) {
    with_radix<MAXR>(P.ayB.radix[s], [&](auto r) {
      y0_pass<decltype(r)::value, -1>(sm, P, s, nlive, Z.dlive, Z.zn, Z.gap, twy);
    });
    __syncthreads();
  }
  const int last = P.az.npass - 1;
  for (int s = 0; s < last; ++s) {
    with_radix<MAXR>(P.az.radix[s],
                     [&](auto r) { z_pass<decltype(r)::value, -1>(sm, P, s, twz); });
    __syncthreads();
  }
  with_radix<MAXR>(P.az.radix[last],
                   [&](auto r) { z_mod<decltype(r)::value, Mod>(sm, P, mod, gbase, Sout); });
  if constexpr (!Mod::forward_only) {
    __syncthreads();
    for (int s = last - 1; s >= 0; --s) {
      with_radix<MAXR>(P.az.radix[s],
                       [&](auto r) { z_pass<decltype(r)::value, +1>(sm, P, s, twz); });
      __syncthreads();
    }
    for (int s = P.ayB.npass - 1; s >= 0; --s) {
      with_radix<MAXR>(P.ayB.radix[s], [&](auto r) {
        y0_pass<decltype(r)::value, +1>(sm, P, s, Z.zout, Z.dout, Z.zout, 0, twy);
      });
      __syncthreads();
    }
#pragma unroll 4
    for (int f = threadIdx.x; f < Z.zout * P.By; f += blockDim.x)
      Sout[gbase + f] = sm[f + quot(f, P.dBy) * (P.BS - P.By)];
  }
}

// ------------------------------------------------------------------ x rows
// Slot of the i-th element of a pass's first span.
__device__ __forceinline__ int slot_of(const PairAxis& A, int i) {
  return A.pad ? i + quot(i, A.dpad) : i;
}

struct XyCtx {
  float4* sm;
  int z, y0base, L, nql;  // rows j < L live: nql live quads per line
  FDiv dq;                // by nql
  const float2* tw;       // w_nx^t (shared memory)
};

// x register pass s over the live row quads.
template <int R, int DIR>
__device__ __forceinline__ void x_pass(const XyCtx& C, const PairPlan& P, int s) {
  const int span = P.ax.span[s], step = P.nx / P.ax.len[s];
  const int plen = P.ax.plen[s], ps = P.ax.pspan[s];
  const int per = P.nx / R, total = P.TG * C.nql * per;
  const FDiv Dper = P.ax.dper[s], Ds = P.ax.dspan[s];
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int r = quot(f, Dper), rem = f - r * per;
    const int g = quot(r, C.dq), q = r - g * C.nql;
    const int b = quot(rem, Ds), i = rem - b * span;
    float4* p = C.sm + (g * P.NQ + q) * P.rowlen + b * plen + slot_of(P.ax, i);
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = get(p[t * ps]);
    if constexpr (DIR > 0) twiddle<R, DIR>(v, C.tw, i * step);
    pdft<R, DIR>(v);
    if constexpr (DIR < 0) twiddle<R, DIR>(v, C.tw, i * step);
#pragma unroll
    for (int t = 0; t < R; ++t) p[t * ps] = put(v[t]);
  }
}

// The four rows of quad q of line y0: rows j = 4q..4q+3 (dead ones default).
// A quad's element holds (row 4q, row 4q+2, row 4q+1, row 4q+3).
template <class Fn>
struct QuadRows {
  typename Fn::Row a, b, c, d;
  __device__ __forceinline__ QuadRows(const Fn& fn, const PairPlan& P, const XyCtx& C, int g,
                                      int q) {
    const int y = C.y0base + g + 4 * q * P.By, j = 4 * q;
    if (j < C.L) a = fn.row(y, C.z);
    if (j + 1 < C.L) b = fn.row(y + P.By, C.z);
    if (j + 2 < C.L) c = fn.row(y + 2 * P.By, C.z);
    if (j + 3 < C.L) d = fn.row(y + 3 * P.By, C.z);
  }
};

// First x pass, straight from the prologue.
template <int R, class Pro>
__device__ __forceinline__ void x_first(const XyCtx& C, const PairPlan& P, const Pro& pro) {
  const int span = P.ax.span[0], ps = P.ax.pspan[0];
  const int total = P.TG * C.nql * span;
  const FDiv Ds = P.ax.dspan[0];
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int r = quot(f, Ds), i = f - r * span;
    const int g = quot(r, C.dq), q = r - g * C.nql;
    const QuadRows<Pro> w(pro, P, C, g, q);
    float4* p = C.sm + (g * P.NQ + q) * P.rowlen + slot_of(P.ax, i);
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      const int x = i + t * span;
      v[t] = c2{make_float2(w.a.load(x), w.c.load(x)), make_float2(w.b.load(x), w.d.load(x))};
    }
    pdft<R, -1>(v);
    twiddle<R, -1>(v, C.tw, i);
#pragma unroll
    for (int t = 0; t < R; ++t) p[t * ps] = put(v[t]);
  }
}

// Last inverse x pass into the epilogue; FUSE: and the first forward pass of
// what it returns.
template <int R, class Epi, bool FUSE>
__device__ __forceinline__ void x_last(const XyCtx& C, const PairPlan& P, Epi& epi) {
  const int span = P.ax.span[0], ps = P.ax.pspan[0];
  const int total = P.TG * C.nql * span, xn = epi.row_n();
  const FDiv Ds = P.ax.dspan[0];
  for (int f = threadIdx.x; f < total; f += blockDim.x) {
    const int r = quot(f, Ds), i = f - r * span;
    const int g = quot(r, C.dq), q = r - g * C.nql;
    const QuadRows<Epi> w(epi, P, C, g, q);
    float4* p = C.sm + (g * P.NQ + q) * P.rowlen + slot_of(P.ax, i);
    // what the epilogue reads is loaded in groups, and ahead of the transform
    // where the registers allow, so the loads' latencies overlap
    constexpr int CH = R <= 8 ? R : 4;
    typename Epi::Pre a[CH], b[CH], c[CH], d[CH];
    auto preload = [&](int t0) {
#pragma unroll
      for (int t = 0; t < CH; ++t) {
        const int x = i + (t0 + t) * span;
        if (t0 + t < R && (t0 + t) * span < xn) {
          a[t] = epi.pre(w.a, x);
          b[t] = epi.pre(w.b, x);
          c[t] = epi.pre(w.c, x);
          d[t] = epi.pre(w.d, x);
        }
      }
    };
    if constexpr (CH == R) preload(0);
    c2 v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = get(p[t * ps]);
    twiddle<R, +1>(v, C.tw, i);
    pdft<R, +1>(v);
#pragma unroll
    for (int t0 = 0; t0 < R; t0 += CH) {
      if constexpr (CH < R) preload(t0);
#pragma unroll
      for (int u = 0; u < CH; ++u) {
        const int t = t0 + u, x = i + t * span;
        if (t < R && t * span >= xn) {
          v[t] = get(zero4());  // beyond the longest row, for every thread alike
        } else if (t < R) {
          v[t].re.x = epi.put(w.a, x, v[t].re.x, a[u]);
          v[t].im.x = epi.put(w.b, x, v[t].im.x, b[u]);
          v[t].re.y = epi.put(w.c, x, v[t].re.y, c[u]);
          v[t].im.y = epi.put(w.d, x, v[t].im.y, d[u]);
        }
      }
    }
    if constexpr (FUSE) {
      pdft<R, -1>(v);
      twiddle<R, -1>(v, C.tw, i);
#pragma unroll
      for (int t = 0; t < R; ++t) p[t * ps] = put(v[t]);
    }
  }
}

// ---------------------------------------------------------------- columns
// Slots of one column and its mirror nx - kx in a row.
struct ColSlots {
  int s, sn;   // sn == s for kx = 0 and kx = nx/2
  bool valid;  // kx < XS
  __device__ __forceinline__ ColSlots(const PairPlan& P, const int* CLARITY_RESTRICT slots,
                                      int kx) {
    valid = kx < P.XS;
    const int k = valid ? kx : 0;
    s = CLARITY_LDG(&slots[k]);
    sn = k == 0 ? s : CLARITY_LDG(&slots[P.nx - k]);
  }
};

// S columns -> inverse Ay-DFT -> row pairs Z = row 2p + i row 2p+1 at slots kx
// and nx - kx: Z[k] = A + iB, Z[nx-k] = conj A + i conj B.  The imaginary parts
// of the self-conjugate columns are ignored (as FFTW's c2r).
template <int AY>
__device__ __forceinline__ void cols_inverse(const XyCtx& C, const PairPlan& P,
                                             const float4* CLARITY_RESTRICT S, const float4* twl,
                                             const int* CLARITY_RESTRICT slots) {
  constexpr int NQ = (AY + 3) / 4;
  const unsigned ks = (unsigned)P.KG * P.nz * P.By;
  for (int f = threadIdx.x; f < P.TG * P.KG; f += blockDim.x) {
    const int kg = quot(f, P.dTG), g = f - kg * P.TG;
    const float4* src = S + ((unsigned)kg * P.nz + C.z) * P.By + C.y0base + g;
    c2 v[NQ * 4];
#pragma unroll
    for (int k1 = 0; k1 < AY; ++k1) v[k1] = get(ld_l2(&src[k1 * ks]));
#pragma unroll
    for (int k1 = AY; k1 < NQ * 4; ++k1) v[k1] = get(zero4());
    const ColSlots c0(P, slots, 2 * kg), c1(P, slots, 2 * kg + 1);
#pragma unroll
    for (int k1 = 1; k1 < AY; ++k1) v[k1] = pcmulc(v[k1], twl[g * AY + k1]);
    pdft<AY, +1>(v);
    if (c0.s == c0.sn) {
#pragma unroll
      for (int j = 0; j < AY; ++j) v[j].im.x = 0.f;
    }
    if (c1.s == c1.sn) {
#pragma unroll
      for (int j = 0; j < AY; ++j) v[j].im.y = 0.f;
    }
    float4* row = C.sm + g * P.NQ * P.rowlen;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q >= C.nql) continue;
      const c2 A = v[4 * q], B = v[4 * q + 1], Cc = v[4 * q + 2], D = v[4 * q + 3];
      float4* rq = row + q * P.rowlen;
      rq[c0.s] = make_float4(A.re.x - B.im.x, Cc.re.x - D.im.x, A.im.x + B.re.x,
                             Cc.im.x + D.re.x);
      if (c0.sn != c0.s)
        rq[c0.sn] = make_float4(A.re.x + B.im.x, Cc.re.x + D.im.x, B.re.x - A.im.x,
                                D.re.x - Cc.im.x);
      if (c1.valid) {
        rq[c1.s] = make_float4(A.re.y - B.im.y, Cc.re.y - D.im.y, A.im.y + B.re.y,
                               Cc.im.y + D.re.y);
        if (c1.sn != c1.s)
          rq[c1.sn] = make_float4(A.re.y + B.im.y, Cc.re.y + D.im.y, B.re.y - A.im.y,
                                  D.re.y - Cc.im.y);
      }
    }
  }
}

// Row pairs -> columns A = (Z[k] + conj Z[nx-k]) / 2, B = (Z[k] - conj Z[nx-k])
// / 2i -> forward Ay-DFT -> twiddle -> S (the halves are taken at the end).
template <int AY>
__device__ __forceinline__ void cols_forward(const XyCtx& C, const PairPlan& P,
                                             float4* CLARITY_RESTRICT S, const float4* twl,
                                             const int* CLARITY_RESTRICT slots) {
  constexpr int NQ = (AY + 3) / 4;
  const unsigned ks = (unsigned)P.KG * P.nz * P.By;
  for (int f = threadIdx.x; f < P.TG * P.KG; f += blockDim.x) {
    const int kg = quot(f, P.dTG), g = f - kg * P.TG;
    const ColSlots c0(P, slots, 2 * kg), c1(P, slots, 2 * kg + 1);
    const float4* row = C.sm + g * P.NQ * P.rowlen;
    c2 v[NQ * 4];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      if (q < C.nql) {
        const float4* rq = row + q * P.rowlen;
        const float4 z0 = rq[c0.s], w0 = rq[c0.sn];
        const float4 z1 = c1.valid ? rq[c1.s] : zero4();
        const float4 w1 = c1.valid ? rq[c1.sn] : z1;
        v[4 * q] = c2{make_float2(z0.x + w0.x, z1.x + w1.x), make_float2(z0.z - w0.z, z1.z - w1.z)};
        v[4 * q + 1] = c2{make_float2(z0.z + w0.z, z1.z + w1.z),
                          make_float2(w0.x - z0.x, w1.x - z1.x)};
        v[4 * q + 2] = c2{make_float2(z0.y + w0.y, z1.y + w1.y),
                          make_float2(z0.w - w0.w, z1.w - w1.w)};
        v[4 * q + 3] = c2{make_float2(z0.w + w0.w, z1.w + w1.w),
                          make_float2(w0.y - z0.y, w1.y - z1.y)};
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) v[4 * q + t] = get(zero4());
      }
    }
    pdft<AY, -1>(v);
    float4* dst = S + ((unsigned)kg * P.nz + C.z) * P.By + C.y0base + g;
#pragma unroll
    for (int k1 = 0; k1 < AY; ++k1) {
      const c2 h{pmul(v[k1].re, both(0.5f)), pmul(v[k1].im, both(0.5f))};
      dst[k1 * ks] = put(k1 ? pcmul(h, twl[g * AY + k1]) : h);
    }
  }
}

// ----------------------------------------------------------------- kernels
// Shared memory of an XY block: TG*NQ row quads, then the lines' y split
// twiddles w_ny^(y0 k1) (TG*Ay, both parts twice) and the x twiddles (nx).
__device__ __forceinline__ const float4* stage_tables(float4* sm, const PairPlan& P, int y0base,
                                                      const float2* CLARITY_RESTRICT tables) {
  float4* twl = sm + P.TG * P.NQ * P.rowlen;
  float2* twx = reinterpret_cast<float2*>(twl + P.TG * P.Ay);
  for (int t = threadIdx.x; t < P.nx; t += blockDim.x) twx[t] = CLARITY_LDG(&tables[P.ax.tw_off + t]);
  for (int t = threadIdx.x; t < P.TG * P.Ay; t += blockDim.x) {
    const int g = t / P.Ay, k1 = t - g * P.Ay;
    twl[t] = twin(CLARITY_LDG(&tables[P.tw_ny_off + (y0base + g) * k1]));
  }
  return twl;
}
// The tile of a block: lines y0base .. y0base+TG-1 of plane z.
template <class Fn>
__device__ __forceinline__ XyCtx tile_of(float4* sm, const PairPlan& P, const Fn& fn, int z,
                                         int y0base, const float4* twl) {
  XyCtx C;
  C.sm = sm;
  C.z = z;
  C.y0base = y0base;
  C.L = fn.live_rows(y0base, P.By, P.Ay);
  C.nql = (C.L + 3) / 4;
  C.dq = fdiv_by(C.nql);
  C.tw = reinterpret_cast<const float2*>(twl + P.TG * P.Ay);
  return C;
}

template <int MAXR>
__device__ __forceinline__ void x_inverse(const XyCtx& C, const PairPlan& P) {
  for (int s = P.ax.npass - 1; s >= 1; --s) {
    with_radix<MAXR>(P.ax.radix[s], [&](auto r) { x_pass<decltype(r)::value, +1>(C, P, s); });
    __syncthreads();
  }
}
template <int MAXR>
__device__ __forceinline__ void x_forward(const XyCtx& C, const PairPlan& P) {
  for (int s = 1; s < P.ax.npass; ++s) {
    with_radix<MAXR>(P.ax.radix[s], [&](auto r) { x_pass<decltype(r)::value, -1>(C, P, s); });
    __syncthreads();
  }
}

template <class Pro, bool BIG>
__global__ void __launch_bounds__(Cls<BIG>::MAXT, 2)
    kp_xy_forward(CLARITY_GRID_CONST PairPlan P, const Pro pro, float2* S,
                  const float2* CLARITY_RESTRICT tables, const int* CLARITY_RESTRICT slots) {
  CLARITY_DYN_SMEM(float4, sm);
  constexpr int MAXR = Cls<BIG>::MAXR;
  const int groups = P.By / P.TG;
  const int pl = blockIdx.x / groups, y0base = (blockIdx.x - pl * groups) * P.TG;
  const float4* twl = stage_tables(sm, P, y0base, tables);
  __syncthreads();
  CLARITY_PDL_WAIT();
  const XyCtx C = tile_of(sm, P, pro, pro.plane(pl), y0base, twl);
  with_radix<MAXR>(P.ax.radix[0], [&](auto r) { x_first<decltype(r)::value>(C, P, pro); });
  __syncthreads();
  x_forward<MAXR>(C, P);
  with_radix<MAXR>(P.Ay, [&](auto r) {
    cols_forward<decltype(r)::value>(C, P, reinterpret_cast<float4*>(S), twl, slots);
  });
  pro.finish();
}

template <class Epi, bool FUSE, bool BIG>
__global__ void __launch_bounds__(Cls<BIG>::MAXT, 2)
    kp_xy_inverse(CLARITY_GRID_CONST PairPlan P, Epi epi, float2* S,
                  const float2* CLARITY_RESTRICT tables, const int* CLARITY_RESTRICT slots) {
  CLARITY_DYN_SMEM(float4, sm);
  constexpr int MAXR = Cls<BIG>::MAXR;
  const int groups = P.By / P.TG;
  const int z = blockIdx.x / groups, y0base = (blockIdx.x - z * groups) * P.TG;
  const float4* twl = stage_tables(sm, P, y0base, tables);
  __syncthreads();
  CLARITY_PDL_WAIT();
  const XyCtx C = tile_of(sm, P, epi, z, y0base, twl);
  with_radix<MAXR>(P.Ay, [&](auto r) {
    cols_inverse<decltype(r)::value>(C, P, reinterpret_cast<const float4*>(S), twl, slots);
  });
  __syncthreads();
  x_inverse<MAXR>(C, P);
  with_radix<MAXR>(P.ax.radix[0],
                   [&](auto r) { x_last<decltype(r)::value, Epi, FUSE>(C, P, epi); });
  if constexpr (FUSE) {
    __syncthreads();
    x_forward<MAXR>(C, P);
    with_radix<MAXR>(P.Ay, [&](auto r) {
      cols_forward<decltype(r)::value>(C, P, reinterpret_cast<float4*>(S), twl, slots);
    });
  }
  epi.finish();
}

}  // namespace pr
}  // namespace clarity
