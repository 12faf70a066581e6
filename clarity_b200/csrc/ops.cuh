// ops.cuh -- operations fused into the FFT passes.
//
// Prologues (XY forward): load_c(m, y, z) returns complex row element m of
//   row (y, z): (v[2m], v[2m+1]) for even nx, (v[m], 0) for odd nx.
//   live_planes(nz) planes can be nonzero, plane(p) is the p-th of them and
//   live_rows the leading rows of a line group inside the volume: the pass
//   transforms and writes nothing else (Mod::zn, Mod::zh say the same to the
//   z pass that reads its output).
// Epilogues (XY inverse): apply_c(m, y, z, c) receives the same pair of
//   real-space values after the inverse transform; the returned pair feeds
//   the forward transform when the epilogue is fused into k_xy_inv_fwd.
// Spectral operations (Z pass): apply(idx, v) with idx the element's offset
//   in the S layout (the OTF shares that layout).
// The column-pair passes (passes_pair.cuh) work on real rows instead: row(y, z)
// describes one (a default Row is a dead one, zero or unwanted), a prologue's
// Row::load(x) is its value at x, an epilogue's pre(row, x) loads what it needs
// there (ahead of the result) and put(row, x, v, pre) takes the result and
// returns what the forward transform sees; a spectral operation's pair(h, v)
// takes two columns at once.
#pragma once
#include "launch_macro.cuh"

#include "dft_codelets.cuh"
#include "dft_pair.cuh"
#include "plan.hpp"
#include "tma.cuh"

namespace clarity {
namespace st {
// A tile row's input for the staged pass kernels: nf floats at p
// (x = 0 .. nf-1), zero beyond; nf == 0 for a row known to be zero.
struct RowRef {
  const float* p;
  int nf;
};
}  // namespace st

// The reference divide of src/ComputePrimitives.cxx:144-148 (and
// ComputePrimitivesGPU.cu:180-184) tests fabs(b) < 1e-5 in double; for a
// float b that is exactly fabsf(b) <= 1e-5f (1e-5f is the largest float
// below 1e-5).
__device__ __forceinline__ float rl_ratio(float g, float b) {
  return (fabsf(b) <= 1e-5f) ? 0.f : g / b;
}

// The ratio inside the image, 0 outside it (where g is zero).  A zero dividend
// would send the whole warp through the division's out-of-line path -- half
// the elements of a row whose image ends at its middle -- so dead elements
// divide 1 by 1.
__device__ __forceinline__ float live_ratio(bool live, float g, float b) {
  const float q = rl_ratio(live ? g : 1.f, live ? b : 1.f);
  return live ? q : 0.f;
}

// Real volume on the padded work box, x fastest.  The planner rejects boxes
// of 2^31 voxels or more, so 32-bit offsets suffice.
struct WorkVol {
  int nx, ny, nz;
  __device__ __forceinline__ unsigned idx(int x, int y, int z) const {
    return ((unsigned)z * ny + y) * nx + x;
  }
};

// Unpadded image seen on the work box with zero shift
// (src/MaximumLikelihoodDeconvolve.cxx:278-282): the image itself inside
// [0,X)x[0,Y)x[0,Z), zero in the padding.  Only bounds checks, no modulo.
struct ImageSrc {
  const float* CLARITY_RESTRICT src;
  int X, Y, Z;
  __device__ __forceinline__ float at(int x, int y, int z) const {
    if (x < X && y < Y && z < Z) return CLARITY_LDG(&src[((unsigned)z * Y + y) * X + x]);
    return 0.f;
  }
};

// Source volume of size (X, Y, Z) seen on the work box through the
// reference's cyclic pad/shift (src/ImagePadSpatialShift.cxx:42-66):
// work coordinate d maps to s = ((d - shift) wrapped) % dim, inside when
// s < src dim, otherwise the fill value (0).
struct PaddedSrc {
  const float* CLARITY_RESTRICT src;
  int X, Y, Z;       // source dims
  int sx, sy, sz;    // shift
  int nx, ny, nz;    // work dims
  __device__ __forceinline__ static int wrap(int d, int shift, int n) {
    int s = d - shift;
    if (s < 0) s += n;
    return s % n;
  }
  __device__ __forceinline__ float at(int x, int y, int z) const {
    const int k = wrap(z, sz, nz);
    const int j = wrap(y, sy, ny);
    const int i = wrap(x, sx, nx);
    if (i >= 0 && j >= 0 && k >= 0 && i < X && j < Y && k < Z)
      return CLARITY_LDG(&src[((long long)k * Y + j) * X + i]);
    return 0.f;
  }
};

// A real row read by a prologue: n floats at p seen from x = -off on an axis
// of length `wrap` (the pad/shift map), zero elsewhere, times s.
struct SrcRow {
  const float* CLARITY_RESTRICT p = nullptr;
  int n = 0, off = 0, wrap = 1 << 30;
  float s = 1.f;
  __device__ __forceinline__ float load(int x) const {
    int i = x + off;
    if (i >= wrap) i -= wrap;
    return i < n ? s * ld_l2(p + i) : 0.f;
  }
};

// ---------------------------------------------------------------- prologues
// Plain work-box volume, optionally multiplied by a device-resident scale
// (the deferred RL flux rescale).
struct ProWork {
  const float* CLARITY_RESTRICT v;
  const float* CLARITY_RESTRICT scale;  // nullptr -> 1
  WorkVol w;
  int xmode;
  __device__ __forceinline__ float2 load_c(int m, int y, int z) const {
    const float s = scale ? *scale : 1.f;
    if (xmode == 0) {
      const float2 a = CLARITY_LDG(reinterpret_cast<const float2*>(v + w.idx(2 * m, y, z)));
      return scale ? make_float2(s * a.x, s * a.y) : a;
    }
    const float a = CLARITY_LDG(&v[w.idx(m, y, z)]);
    return make_float2(scale ? s * a : a, 0.f);
  }
  using Row = SrcRow;
  __device__ __forceinline__ Row row(int y, int z) const {
    return Row{v + w.idx(0, y, z), w.nx, 0, 1 << 30, scale ? ld_l2(scale) : 1.f};
  }
  int live_planes(int nz) const { return nz; }
  __device__ __forceinline__ int plane(int p) const { return p; }
  static constexpr bool has_zero_rows = false;
  __device__ __forceinline__ int live_rows(int, int, int ay) const { return ay; }
  __device__ __forceinline__ void finish() const {}
};

// Rows y0base + by*j of a line group that lie below Y (j < the result).
CLARITY_HD inline int rows_below(int Y, int y0base, int by, int ay) {
  const int l = (Y - y0base + by - 1) / by;
  return l < 0 ? 0 : (l > ay ? ay : l);
}

// Extrapolated estimate of accelerated RL (Biggs-Andrews): y = max(0,
// x + alpha (x - xp)), one fused multiply-add, stored to yout on the way into
// the forward transform (the product step reads it back as the estimate).
// The estimates are volumes of the image's extent (X, Y, Z): they are zero in
// the padding (see EpiRLProduct).
struct ProAccel {
  const float* CLARITY_RESTRICT x;
  const float* CLARITY_RESTRICT xp;
  const float* CLARITY_RESTRICT alpha;
  float* CLARITY_RESTRICT yout;
  int X, Y, Z;
  int xmode;
  __device__ __forceinline__ static float extrap(float a, float x, float xp) {
    return fmaxf(0.f, fmaf(a, x - xp, x));
  }
  __device__ __forceinline__ float one(float a, int i, int y, int z) const {
    if (i >= X || y >= Y || z >= Z) return 0.f;
    const unsigned o = ((unsigned)z * Y + y) * X + i;
    const float r = extrap(a, CLARITY_LDG(x + o), CLARITY_LDG(xp + o));
    yout[o] = r;
    return r;
  }
  __device__ __forceinline__ float2 load_c(int m, int y, int z) const {
    const float a = CLARITY_LDG(alpha);
    if (xmode == 0) {
      const float lo = one(a, 2 * m, y, z);
      return make_float2(lo, one(a, 2 * m + 1, y, z));
    }
    return make_float2(one(a, m, y, z), 0.f);
  }
  struct Row {
    const float *CLARITY_RESTRICT x = nullptr, *CLARITY_RESTRICT xp = nullptr;
    float* CLARITY_RESTRICT y = nullptr;
    int n = 0;
    float a = 0.f;
    __device__ __forceinline__ float load(int i) const {
      if (i >= n) return 0.f;
      const float r = extrap(a, ld_l2(x + i), ld_l2(xp + i));
      y[i] = r;
      return r;
    }
  };
  __device__ __forceinline__ Row row(int yy, int z) const {
    if (yy >= Y || z >= Z) return Row{};
    const unsigned o = ((unsigned)z * Y + yy) * X;
    return Row{x + o, xp + o, yout + o, X, ld_l2(alpha)};
  }
  int live_planes(int nz) const { return Z < nz ? Z : nz; }
  __device__ __forceinline__ int plane(int p) const { return p; }
  static constexpr bool has_zero_rows = true;
  CLARITY_HD inline int live_rows(int y0base, int by, int ay) const {
    return rows_below(Y, y0base, by, ay);
  }
  __device__ __forceinline__ void finish() const {}
};

// Unpadded source read through the pad/shift map, times an optional scale.
struct ProPadded {
  PaddedSrc p;
  const float* CLARITY_RESTRICT scale;  // nullptr -> 1
  int xmode;
  __device__ __forceinline__ float2 load_c(int m, int y, int z) const {
    const float s = scale ? *scale : 1.f;
    if (xmode == 0) {
      float a = p.at(2 * m, y, z), b = p.at(2 * m + 1, y, z);
      if (scale) { a = s * a; b = s * b; }
      return make_float2(a, b);
    }
    float a = p.at(m, y, z);
    if (scale) a = s * a;
    return make_float2(a, 0.f);
  }
  // With the shift by -Z/2 the source's planes wrap around plane 0: its upper
  // Z - Z/2 planes land on planes 0.., the others on the last Z/2.
  using Row = SrcRow;
  __device__ __forceinline__ Row row(int y, int z) const {
    const int k = PaddedSrc::wrap(z, p.sz, p.nz), j = PaddedSrc::wrap(y, p.sy, p.ny);
    if (j >= p.Y || k >= p.Z) return Row{};
    return Row{p.src + ((long long)k * p.Y + j) * p.X, p.X, -p.sx, p.nx,
               scale ? ld_l2(scale) : 1.f};
  }
  int live_planes(int) const { return p.Z; }
  __device__ __forceinline__ int plane(int q) const {
    return q < p.Z + p.sz ? q : q + (p.nz - p.Z);
  }
  static constexpr bool has_zero_rows = false;
  __device__ __forceinline__ int live_rows(int, int, int ay) const { return ay; }
  __device__ __forceinline__ void finish() const {}
};

// The padded image (zero shift) as a prologue, times an optional scale.
struct ProImage {
  ImageSrc p;
  int xmode;
  const float* CLARITY_RESTRICT scale = nullptr;
  __device__ __forceinline__ float2 load_c(int m, int y, int z) const {
    float2 v = xmode == 0 ? make_float2(p.at(2 * m, y, z), p.at(2 * m + 1, y, z))
                          : make_float2(p.at(m, y, z), 0.f);
    if (scale) {
      const float s = *scale;
      v = make_float2(s * v.x, s * v.y);
    }
    return v;
  }
  using Row = SrcRow;
  __device__ __forceinline__ Row row(int y, int z) const {
    if (y >= p.Y || z >= p.Z) return Row{};
    return Row{p.src + ((unsigned)z * p.Y + y) * p.X, p.X, 0, 1 << 30,
               scale ? ld_l2(scale) : 1.f};
  }
  int live_planes(int nz) const { return p.Z < nz ? p.Z : nz; }
  __device__ __forceinline__ int plane(int q) const { return q; }
  static constexpr bool has_zero_rows = true;
  CLARITY_HD inline int live_rows(int y0base, int by, int ay) const {
    return rows_below(p.Y, y0base, by, ay);
  }
  __device__ __forceinline__ void finish() const {}
};

// ---------------------------------------------------------------- epilogues
// Two floats at p, as one store where p allows.
__device__ __forceinline__ void store2(float* p, float a, float b) {
  if (((uintptr_t)p & 7u) == 0) {
    *reinterpret_cast<float2*>(p) = make_float2(a, b);
  } else {
    p[0] = a;
    p[1] = b;
  }
}

// Block-wide FP64 sum of per-thread partials into partial[block index]
// (fixed reduction order: deterministic).
__device__ __forceinline__ void block_sum_store(double acc, double* partial) {
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    double a = lane < nw ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) partial[CLARITY_BLOCK_ID()] = a;
  }
}

// Block-wide FP64 total of np partials (thread 0 gets it; fixed order):
// thread i sums partials i, i + blockDim.x, ..., then a tree over the block.
// The partials are read through L2 (__ldcg); they come from the previous
// kernel on the stream.
__device__ __forceinline__ double block_total(const double* partial, int np) {
  double acc = 0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) acc += __ldcg(&partial[i]);
  __shared__ double red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  double t = 0;
  if (threadIdx.x == 0) {
    for (int w = 0; w < (int)((blockDim.x + 31) >> 5); ++w) t += red[w];
  }
  return t;  // valid in thread 0
}

// Store the real-space result on the work box.
struct EpiWork {
  static constexpr bool has_zero_rows = false;
  float* CLARITY_RESTRICT out;
  WorkVol w;
  int xmode;
  __device__ __forceinline__ float2 apply_c(int m, int y, int z, float2 c) {
    if (xmode == 0)
      *reinterpret_cast<float2*>(out + w.idx(2 * m, y, z)) = c;
    else
      out[w.idx(m, y, z)] = c.x;
    return c;
  }
  struct Row {
    float* o = nullptr;
  };
  __device__ __forceinline__ Row row(int y, int z) const { return Row{out + w.idx(0, y, z)}; }
  __host__ __device__ __forceinline__ int row_n() const { return w.nx; }
  struct Pre {};
  __device__ __forceinline__ Pre pre(const Row&, int) const { return Pre{}; }
  __device__ __forceinline__ float put(const Row& r, int x, float v, Pre) {
    if (!r.o) return 0.f;
    r.o[x] = v;
    return v;
  }
  // padding rows where the result is known to be zero
  __device__ __forceinline__ bool zero_row(int, int) const { return false; }
  // rows y0base + BY*j, j < live_rows, can be nonzero (all here)
  __device__ __forceinline__ int live_rows(int, int, int ay) const { return ay; }
  __device__ __forceinline__ void prefetch_row(int, int) const {}
  __device__ __forceinline__ void finish() {}
};

// Store only the image region (crop from the origin, src/ImageClip.cxx:41-46)
// into an unpadded (X, Y, Z) volume, times an optional device scale.
struct EpiClip {
  static constexpr bool has_zero_rows = true;
  float* CLARITY_RESTRICT out;
  int X, Y, Z;
  const float* CLARITY_RESTRICT scale;
  int xmode;
  __device__ __forceinline__ void put(int x, int y, int z, float v) {
    if (x < X && y < Y && z < Z) {
      if (scale) v = *scale * v;
      out[((long long)z * Y + y) * X + x] = v;
    }
  }
  __device__ __forceinline__ float2 apply_c(int m, int y, int z, float2 c) {
    if (xmode == 0) {
      put(2 * m, y, z, c.x);
      put(2 * m + 1, y, z, c.y);
    } else {
      put(m, y, z, c.x);
    }
    return c;
  }
  struct Row {
    float* o = nullptr;
    float s = 1.f;
  };
  __device__ __forceinline__ Row row(int y, int z) const {
    if (y >= Y || z >= Z) return Row{};
    return Row{out + ((long long)z * Y + y) * X, scale ? ld_l2(scale) : 1.f};
  }
  __host__ __device__ __forceinline__ int row_n() const { return X; }
  struct Pre {};
  __device__ __forceinline__ Pre pre(const Row&, int) const { return Pre{}; }
  __device__ __forceinline__ float put(const Row& r, int x, float v, Pre) {
    if (r.o && x < X) r.o[x] = r.s * v;
    return v;
  }
  // rows and planes outside the image are not asked for: not transformed
  int live_planes(int nz) const { return Z < nz ? Z : nz; }
  CLARITY_HD inline int live_rows(int y0base, int by, int ay) const {
    return rows_below(Y, y0base, by, ay);
  }
  __device__ __forceinline__ void prefetch_row(int, int) const {}
  __device__ __forceinline__ void finish() {}
};

// RL step 4 (src/MaximumLikelihoodDeconvolve.cxx:69-70) with the flux sum of
// step 5 (:73-74): u_new = cur * c, cur = scale * u, partial sums of u_new in
// FP64.  The first estimate is zero outside its extent (X, Y, Z) -- the image's,
// or the whole work box where a caller starts from a work-box volume -- and a
// product keeps it zero there, so cur and u_new are volumes of that extent and
// the pass transforms only its rows and planes.  At the 512x512x128 box with a
// 256x256x64 image that is an eighth of the work-box volume and a quarter of
// its rows: the pass went from 176 to 112 us of device time by that, and to 71
// with its rows copied and stored by all threads (passes_xy_tma.cuh).
struct EpiRLProduct {
  static constexpr bool has_zero_rows = true;
  static constexpr int kFamily = KK_XY_PRODUCT;
  const float* CLARITY_RESTRICT cur;     // the estimate (X, Y, Z)
  int X, Y, Z;
  const float* CLARITY_RESTRICT scale;   // deferred flux scale for cur, or nullptr
  float* CLARITY_RESTRICT unew;
  double* CLARITY_RESTRICT partial;
  int xmode;
  double acc;
  int* nblocks = nullptr;  // receives the grid size (the number of partials), or nullptr
  __device__ __forceinline__ unsigned at(int x, int y, int z) const {
    return ((unsigned)z * Y + y) * X + x;
  }
  __device__ __forceinline__ float one(int x, int y, int z, float c) {
    if (x >= X || y >= Y || z >= Z) return 0.f;
    float u = CLARITY_LDG(&cur[at(x, y, z)]);
    if (scale) u = *scale * u;
    const float a = u * c;
    unew[at(x, y, z)] = a;
    acc += (double)a;
    return a;
  }
  __device__ __forceinline__ float2 apply_c(int m, int y, int z, float2 c) {
    if (xmode == 0) {
      const float a = one(2 * m, y, z, c.x);
      return make_float2(a, one(2 * m + 1, y, z, c.y));
    }
    return make_float2(one(m, y, z, c.x), 0.f);
  }
  struct Row {
    unsigned o = 0;  // offset of the row in cur and unew
    int n = 0;       // its live extent
    float s = 1.f;
  };
  __device__ __forceinline__ Row row(int y, int z) const {
    if (y >= Y || z >= Z) return Row{};
    return Row{at(0, y, z), X, scale ? ld_l2(scale) : 1.f};
  }
  using Pre = float;
  __device__ __forceinline__ Pre pre(const Row& r, int x) const {
    return x < r.n ? ld_l2(cur + (r.o + x)) : 0.f;
  }
  __device__ __forceinline__ float put(const Row& r, int x, float c, Pre u) {
    const float a = x < r.n ? (r.s * u) * c : 0.f;
    if (x < r.n) unew[r.o + x] = a;
    acc += (double)a;
    return a;
  }
  __device__ __forceinline__ bool zero_row(int y, int z) const { return y >= Y || z >= Z; }
  int live_planes(int nz) const { return Z < nz ? Z : nz; }
  CLARITY_HD inline int live_rows(int y0base, int by, int ay) const {
    return rows_below(Y, y0base, by, ay);
  }
  // the estimate row this block's epilogue will read, into L2
  __device__ __forceinline__ void prefetch_row(int y, int z) const {
    if (y < Y && z < Z) prefetch_l2_range(cur + at(0, y, z), sizeof(float) * (size_t)X);
  }
  // Staged form (passes_xy_rows.cuh): row (y, z) of cur arrives in shared memory
  // (n floats at sr).
  static constexpr bool kStaged = true;
  __device__ __forceinline__ st::RowRef in_row(int y, int z) const {
    if (y < Y && z < Z) return {cur + at(0, y, z), X};
    return {nullptr, 0};
  }
  __host__ __device__ __forceinline__ int row_n() const { return X; }
  __host__ __device__ __forceinline__ int stage_n() const { return X; }  // floats of a staged row
  float s_ = 1.f;  // the deferred scale, read once the previous pass is done
  __device__ __forceinline__ void prepare() {
    if (scale) s_ = ld_l2(scale);
  }
  __device__ __forceinline__ float2 apply_s(int m, int y, int z, float2 c, const float* sr,
                                            int n) {
    const int x = 2 * m;
    if (x >= n) return make_float2(0.f, 0.f);  // zero outside the estimate whatever c is there
    const unsigned o = at(x, y, z);
    const float a = (s_ * sr[x]) * c.x;
    acc += (double)a;
    if (x + 1 >= n) {
      unew[o] = a;
      return make_float2(a, 0.f);
    }
    const float b = (s_ * sr[x + 1]) * c.y;
    acc += (double)b;
    store2(unew + o, a, b);
    return make_float2(a, b);
  }
  __device__ __forceinline__ void finish() {
    block_sum_store(acc, partial);
    if (nblocks && CLARITY_BLOCK_ID() == 0 && threadIdx.x == 0) *nblocks = (int)CLARITY_GRID_DIM();
  }
};

// RL step 2 (src/MaximumLikelihoodDeconvolve.cxx:61-62): r = g / (h*u) with
// the 1e-5 guard, fused between the inverse and forward transforms.
struct MidRLRatio {
  static constexpr bool has_zero_rows = true;
  ImageSrc g;
  int xmode;
  // Optional trace (idiv_partial != nullptr): the I-divergence of g against
  // b = h*cur over the image, g ln(g/b) + b - g with 0 ln 0 = 0 (terms with
  // g > 0 >= b skipped), summed in FP64 per block; block 0 stores the grid
  // size in *nblocks.  Same definition as k_idiv and the oracle
  // (IDIVFunctional, src/IDivergenceDeconvolve.cxx:33-47, alpha = 0).
  double* CLARITY_RESTRICT idiv_partial = nullptr;
  int* nblocks = nullptr;
  double acc = 0.0;
  __device__ __forceinline__ void idiv_add(float a, float b) {
    if (a > 0.f) {
      if (b > 0.f) {
        const double da = a, db = b;
        acc += da * log(da / db) + db - da;
      }
    } else {
      acc += (double)b - (double)a;
    }
  }
  __device__ __forceinline__ float2 apply_c(int m, int y, int z, float2 b) {
    if (idiv_partial && y < g.Y && z < g.Z) {
      if (xmode == 0) {
        if (2 * m < g.X) idiv_add(g.at(2 * m, y, z), b.x);
        if (2 * m + 1 < g.X) idiv_add(g.at(2 * m + 1, y, z), b.y);
      } else if (m < g.X) {
        idiv_add(g.at(m, y, z), b.x);
      }
    }
    if (xmode == 0)
      return make_float2(rl_ratio(g.at(2 * m, y, z), b.x),
                         rl_ratio(g.at(2 * m + 1, y, z), b.y));
    return make_float2(rl_ratio(g.at(m, y, z), b.x), 0.f);
  }
  struct Row {
    unsigned o = 0;  // offset of the row in the image
    int n = 0;       // its live extent
  };
  __device__ __forceinline__ Row row(int y, int z) const {
    if (y >= g.Y || z >= g.Z) return Row{};
    return Row{((unsigned)z * g.Y + y) * g.X, g.X};
  }
  using Pre = float;
  __device__ __forceinline__ Pre pre(const Row& r, int x) const {
    return x < r.n ? ld_l2(g.src + (r.o + x)) : 0.f;
  }
  __device__ __forceinline__ float put(const Row& r, int x, float b, Pre a) {
    if (idiv_partial && x < r.n) idiv_add(a, b);
    return live_ratio(x < r.n, a, b);
  }
  // g is zero outside the image, so the ratio is exactly zero there
  // (0/b, or the 1e-5 guard): rows with y >= Y and planes with z >= Z need no
  // transform at all
  __device__ __forceinline__ bool zero_row(int y, int z) const { return y >= g.Y || z >= g.Z; }
  // planes a launch covers (the rest are neither read nor written: Mod::zn)
  int live_planes(int nz) const { return g.Z < nz ? g.Z : nz; }
  // rows y0base + by*j with j < live_rows lie inside the image (y < Y)
  CLARITY_HD inline int live_rows(int y0base, int by, int ay) const {
    return rows_below(g.Y, y0base, by, ay);
  }
  __device__ __forceinline__ void prefetch_row(int y, int z) const {
    if (y < g.Y && z < g.Z)
      prefetch_l2_range(g.src + ((unsigned)z * g.Y + y) * g.X, sizeof(float) * (size_t)g.X);
  }
  // Staged form: the image row arrives in shared memory.
  static constexpr bool kStaged = true;
  __device__ __forceinline__ st::RowRef in_row(int y, int z) const {
    if (y < g.Y && z < g.Z) return {g.src + ((unsigned)z * g.Y + y) * g.X, g.X};
    return {nullptr, 0};
  }
  __host__ __device__ __forceinline__ int row_n() const { return g.X; }
  __host__ __device__ __forceinline__ int stage_n() const { return g.X; }
  __device__ __forceinline__ float2 apply_s(int m, int, int, float2 b, const float* sr, int n) {
    const int x = 2 * m;
    const float a0 = x < n ? sr[x] : 0.f, a1 = x + 1 < n ? sr[x + 1] : 0.f;
    if (idiv_partial) {
      if (x < n) idiv_add(a0, b.x);
      if (x + 1 < n) idiv_add(a1, b.y);
    }
    return make_float2(live_ratio(x < n, a0, b.x), live_ratio(x + 1 < n, a1, b.y));
  }
  __device__ __forceinline__ void finish() {
    if (idiv_partial) {
      block_sum_store(acc, idiv_partial);
      if (nblocks && CLARITY_BLOCK_ID() == 0 && threadIdx.x == 0) *nblocks = (int)CLARITY_GRID_DIM();
    }
  }
};

// JVC update (src/JansenVanCittertDeconvolve.cxx:106-111,
// JansenVanCittertDeconvolveGPU.cu:43-49): i' = max(0, i + gamma(o) (g - o)),
// gamma(o) = 1 - (o - A)^2 / A^2.  cur == nullptr reads i from the padded
// image (first update).  Stores i' on the work box and returns it, so the
// fused kernel transforms it for the next iteration.
struct EpiJVC {
  static constexpr bool has_zero_rows = false;
  const float* CLARITY_RESTRICT cur;
  ImageSrc g;
  float* CLARITY_RESTRICT inext;
  float A, invASq;
  WorkVol w;
  int xmode;
  __device__ __forceinline__ float upd(float i, float gv, float o) const {
    const float diff = o - A;
    const float gamma = 1.0f - ((diff * diff) * invASq);
    const float val = i + (gamma * (gv - o));
    return val < 0.0f ? 0.0f : val;
  }
  __device__ __forceinline__ float2 apply_c(int m, int y, int z, float2 o) {
    if (xmode == 0) {
      const int x = 2 * m;
      const float g0 = g.at(x, y, z), g1 = g.at(x + 1, y, z);
      const float i0 = cur ? CLARITY_LDG(&cur[w.idx(x, y, z)]) : g0;
      const float i1 = cur ? CLARITY_LDG(&cur[w.idx(x + 1, y, z)]) : g1;
      const float2 r = make_float2(upd(i0, g0, o.x), upd(i1, g1, o.y));
      *reinterpret_cast<float2*>(inext + w.idx(x, y, z)) = r;
      return r;
    }
    const float g0 = g.at(m, y, z);
    const float i0 = cur ? CLARITY_LDG(&cur[w.idx(m, y, z)]) : g0;
    const float r = upd(i0, g0, o.x);
    inext[w.idx(m, y, z)] = r;
    return make_float2(r, 0.f);
  }
  struct Row {
    const float *CLARITY_RESTRICT i = nullptr, *CLARITY_RESTRICT g = nullptr;
    float* CLARITY_RESTRICT o = nullptr;
  };
  __device__ __forceinline__ Row row(int y, int z) const {
    const unsigned k = w.idx(0, y, z);
    const bool in = y < g.Y && z < g.Z;
    return Row{cur ? cur + k : nullptr, in ? g.src + ((unsigned)z * g.Y + y) * g.X : nullptr,
               inext + k};
  }
  using Pre = float2;  // image, estimate
  __device__ __forceinline__ Pre pre(const Row& r, int x) const {
    const float gv = r.g && x < g.X ? ld_l2(r.g + x) : 0.f;
    return make_float2(gv, r.i ? ld_l2(r.i + x) : gv);
  }
  __device__ __forceinline__ float put(const Row& r, int x, float o, Pre p) {
    if (!r.o) return 0.f;
    const float v = upd(p.y, p.x, o);
    r.o[x] = v;
    return v;
  }
  // padding rows where the result is known to be zero
  __device__ __forceinline__ bool zero_row(int, int) const { return false; }
  // rows y0base + BY*j, j < live_rows, can be nonzero (all here)
  __device__ __forceinline__ int live_rows(int, int, int ay) const { return ay; }
  __device__ __forceinline__ void prefetch_row(int y, int z) const {
    if (cur) prefetch_l2_range(cur + w.idx(0, y, z), sizeof(float) * (size_t)w.nx);
    if (y < g.Y && z < g.Z)
      prefetch_l2_range(g.src + ((unsigned)z * g.Y + y) * g.X, sizeof(float) * (size_t)g.X);
  }
  // Staged pass, reading both volumes in place: with a work-box row staged beside
  // each tile row only one-line tiles fit (512x512x128 box: 187 us staged, 172 in
  // place in two-line tiles; 292 before either).
  static constexpr bool kStaged = true;
  __device__ __forceinline__ void prefetch_image(int y, int z) const { prefetch_row(y, z); }
  __device__ __forceinline__ st::RowRef in_row(int, int) const { return {nullptr, 0}; }
  __host__ __device__ __forceinline__ int row_n() const { return w.nx; }
  __host__ __device__ __forceinline__ int stage_n() const { return 0; }
  struct InPlace {
    float2 i, g;
  };
  __device__ __forceinline__ InPlace read(int m, int y, int z) const {
    const int x = 2 * m;
    InPlace q;
    q.g = make_float2(g.at(x, y, z), g.at(x + 1, y, z));
    q.i = cur ? ld_l2(reinterpret_cast<const float2*>(cur + w.idx(x, y, z))) : q.g;
    return q;
  }
  __device__ __forceinline__ float2 apply_q(int m, int y, int z, float2 o, const InPlace& q) {
    const float2 r = make_float2(upd(q.i.x, q.g.x, o.x), upd(q.i.y, q.g.y, o.y));
    *reinterpret_cast<float2*>(inext + w.idx(2 * m, y, z)) = r;
    return r;
  }
  __device__ __forceinline__ float2 apply_s(int m, int y, int z, float2 o, const float*, int) {
    return apply_q(m, y, z, o, read(m, y, z));
  }
  __device__ __forceinline__ void finish() {}
};

// ------------------------------------------------------------ spectral ops
// src/ModulateGPU.cu:63-72 / Convolve.cxx:195-205: out = scale * (a * b),
// no conjugate, a = data, b = OTF; the arithmetic order of
// ComplexMultiplyAndScale (include/internal/Complex.h:95-102) is kept.
// scale2 (optional, device memory) multiplies the 1/N scale: the RL flux
// rescale of the transformed estimate is applied here when the estimate was
// transformed before its scale was known.
struct ModOTF {
  static constexpr bool forward_only = false;
  const float2* CLARITY_RESTRICT H;
  float scale;
  const float* CLARITY_RESTRICT scale2 = nullptr;
  // The flux rescale folded in (partial != nullptr; kernels that call late()):
  // every block forms s = energy / sum of the *np partials itself and uses it
  // in place of *scale2; block 0 stores it to scale_out and the sum to sum_out
  // for the passes that follow.
  const double* CLARITY_RESTRICT partial = nullptr;
  const int* CLARITY_RESTRICT np = nullptr;
  const double* CLARITY_RESTRICT energy = nullptr;
  double* CLARITY_RESTRICT sum_out = nullptr;
  float* CLARITY_RESTRICT scale_out = nullptr;
  // only the z planes z < zn and z >= zh of the input spectrum are nonzero
  // (the rest were never written and are read as zeros); no plane lies at or
  // beyond the default zh
  int zn = 1 << 30;
  int zh = 1 << 30;
  // only the first zout z planes of the output are read by the next pass:
  // the rest are neither inverse-transformed along y0 nor stored
  int zout = 1 << 30;
  // the OTF tile this block will multiply by, into L2 (part p of np)
  __device__ __forceinline__ void prefetch_tile(unsigned base, int tile, int p, int np) const {
    const size_t chunk = ((size_t)tile * 8 / np + 15) & ~size_t(15);
    const size_t off = chunk * p, total = (size_t)tile * 8;
    if (off < total)
      prefetch_l2_range(reinterpret_cast<const char*>(H + base) + off,
                        off + chunk <= total ? chunk : total - off);
  }
  __device__ __forceinline__ float2 apply(long long idx, float2 v) const {
    const float2 h = CLARITY_LDG(&H[idx]);
    const float f = scale2 ? scale * *scale2 : scale;
    return make_float2(f * (v.x * h.x - v.y * h.y), f * (v.x * h.y + v.y * h.x));
  }
  __device__ __forceinline__ c2 pair(float4 h, c2 v) const {
    const float2 hr = make_float2(h.x, h.y), hi = make_float2(h.z, h.w), f = both(scale);
    return c2{pmul(f, psub(pmul(v.re, hr), pmul(v.im, hi))),
              pmul(f, pfma(v.im, hr, pmul(v.re, hi)))};
  }
  // Called by every thread of a block before resolved(), with a barrier inside.
  __device__ __forceinline__ void late() {
    if (!partial) return;  // the same for every thread
    __shared__ float s_late;
    const double t = block_total(partial, *np);
    if (threadIdx.x == 0) {
      const float s = (float)energy[0] / (float)t;
      s_late = s;
      if (CLARITY_BLOCK_ID() == 0) {
        *sum_out = t;
        *scale_out = s;
      }
    }
    __syncthreads();
    scale *= s_late;
    scale2 = nullptr;
    partial = nullptr;
  }
  // the same operation with the deferred factor read once (per thread)
  __device__ __forceinline__ ModOTF resolved() const {
    ModOTF r = *this;
    if (scale2) {
      r.scale = scale * ld_l2(scale2);
      r.scale2 = nullptr;
    }
    return r;
  }
};

// src/WienerDeconvolveGPU.cu:43-49: conj(H) / (|H|^2 + eps), then
// scale * (that * G).
struct ModWiener {
  static constexpr bool forward_only = false;
  const float2* CLARITY_RESTRICT H;
  float eps, scale;
  int zn = 1 << 30;
  int zh = 1 << 30;
  int zout = 1 << 30;
  __device__ __forceinline__ void prefetch_tile(unsigned base, int tile, int p, int np) const {
    const size_t chunk = ((size_t)tile * 8 / np + 15) & ~size_t(15);
    const size_t off = chunk * p, total = (size_t)tile * 8;
    if (off < total)
      prefetch_l2_range(reinterpret_cast<const char*>(H + base) + off,
                        off + chunk <= total ? chunk : total - off);
  }
  __device__ __forceinline__ float2 apply(long long idx, float2 v) const {
    return apply_h(CLARITY_LDG(&H[idx]), v);
  }
  __device__ __forceinline__ float2 apply_h(float2 h, float2 v) const {
    const float mag = h.x * h.x + h.y * h.y;
    const float f = 1.0f / (mag + eps);
    const float a = h.x * f, b = -h.y * f;
    return make_float2(scale * (a * v.x - b * v.y), scale * (a * v.y + b * v.x));
  }
  __device__ __forceinline__ c2 pair(float4 h, c2 v) const {
    const float2 x = apply_h(make_float2(h.x, h.z), make_float2(v.re.x, v.im.x));
    const float2 y = apply_h(make_float2(h.y, h.w), make_float2(v.re.y, v.im.y));
    return c2{make_float2(x.x, y.x), make_float2(x.y, y.y)};
  }
  __device__ __forceinline__ void late() {}
  __device__ __forceinline__ ModWiener resolved() const { return *this; }
};

struct ModForward {
  static constexpr bool forward_only = true;
  int zn = 1 << 30;
  int zh = 1 << 30;
  int zout = 1 << 30;
  __device__ __forceinline__ void prefetch_tile(unsigned, int, int, int) const {}
  __device__ __forceinline__ float2 apply(long long, float2 v) const { return v; }
  __device__ __forceinline__ void late() {}
  __device__ __forceinline__ ModForward resolved() const { return *this; }
};

}  // namespace clarity
