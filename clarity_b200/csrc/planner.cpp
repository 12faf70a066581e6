// planner.cpp -- host-only planning of the fused FFT passes for one work
// box (see plan.hpp for the pass structure and the S layout).
#include <algorithm>
#include <climits>
#include <cstring>
#include <string>
#include <vector>

#include "plan.hpp"

namespace clarity {

static void search_axis(int n, int depth, int* cur, int* best, int* best_len,
                        int* best_max) {
  if (n == 1) {
    int mx = 0;
    for (int i = 0; i < depth; ++i) mx = std::max(mx, cur[i]);
    if (depth < *best_len || (depth == *best_len && mx < *best_max)) {
      *best_len = depth;
      *best_max = mx;
      for (int i = 0; i < depth; ++i) best[i] = cur[i];
    }
    return;
  }
  if (depth >= kMaxPasses || depth + 1 > *best_len) return;
  for (int r : kRadixSet) {
    if (n % r == 0) {
      // keep radices non-increasing to avoid permutations of one factor set
      if (depth > 0 && r > cur[depth - 1]) continue;
      cur[depth] = r;
      search_axis(n / r, depth + 1, cur, best, best_len, best_max);
    }
  }
}

static bool plan_axis(int n, AxisPlan* A) {
  std::memset(A, 0, sizeof(*A));
  A->n = n;
  if (n == 1) return true;
  int cur[kMaxPasses], best[kMaxPasses];
  int best_len = kMaxPasses + 1, best_max = INT_MAX;
  search_axis(n, 0, cur, best, &best_len, &best_max);
  if (best_len > kMaxPasses) return false;
  A->npass = best_len;
  int len = n;
  for (int s = 0; s < best_len; ++s) {
    A->radix[s] = best[s];
    A->len[s] = len;
    A->span[s] = len / best[s];
    len /= best[s];
  }
  return true;
}

static int ctz(int v) {
  int c = 0;
  while (v && !(v & 1)) { v >>= 1; ++c; }
  return c;
}

static constexpr int kSmemMax = 200 * 1024;
static constexpr int kSmemPerSM = 228 * 1024;

// Fills the offsets of a chosen tiling (spectrum size, twiddle layout);
// false when 32-bit offsets would not address the box.
static bool finalize_plan(VolPlan& P, std::string* why) {
  const long long spec = (long long)P.Ay * P.KG * P.nz * P.By * P.W;
  if ((long long)P.nx * P.ny * P.nz >= (1ll << 31) || spec >= (1ll << 31)) {
    if (why) *why = "work box of 2^31 voxels or more";
    return false;
  }
  P.xy_threads = 256;
  P.z_threads = 256;
  P.spec_elems = spec;
  int off = 0;
  P.ax.tw_off = off; off += std::max(P.M, 1);
  P.ayB.tw_off = off; off += std::max(P.By, 1);
  P.az.tw_off = off; off += std::max(P.nz, 1);
  P.tw_r2c_off = off; off += P.M / 2 + 1;
  P.tw_ny_off = off; off += P.ny;
  P.twiddle_count = off;
  P.xrev_off = 0;
  P.xrev_count = P.M;
  return true;
}

bool make_plan(int nx, int ny, int nz, VolPlan* out, std::string* why) {
  return make_plan_candidates(nx, ny, nz, out, 1, why) > 0;
}

int make_plan_candidates(int nx, int ny, int nz, VolPlan* out, int max_out, std::string* why) {
  VolPlan P;
  std::memset(&P, 0, sizeof(P));
  P.nx = nx; P.ny = ny; P.nz = nz;
  P.xmode = (nx % 2 == 0) ? 0 : 1;
  P.M = P.xmode == 0 ? nx / 2 : nx;
  P.XS = P.xmode == 0 ? P.M + 1 : nx;
  if (P.xmode == 0)
    P.items = (P.M % 2 == 0) ? std::max(P.M / 2, 1) : (P.M + 1) / 2;
  else
    P.items = nx;
  if (!plan_axis(P.M, &P.ax)) {
    if (why) *why = "x length " + std::to_string(nx) + " has an unsupported factor";
    return false;
  }
  if (!plan_axis(nz, &P.az)) {
    if (why) *why = "z length " + std::to_string(nz) + " has an unsupported factor";
    return false;
  }
  // x row padding in the XY shared memory
  if (P.ax.npass <= 1 || (P.ax.span[0] & 1)) P.padShift = 30;
  else P.padShift = ctz(P.ax.span[0]);
  {
    const int last = P.M - 1;
    int rs = last + (last >> P.padShift) + 1;
    if (rs % 2 == 0) rs += 1;
    P.rowStride = rs;
  }
  // the max_out best-scoring tilings, best first (insertion into a fixed
  // array: planning allocates nothing)
  constexpr int kMaxCand = 8;
  if (max_out > kMaxCand) max_out = kMaxCand;
  if (max_out < 1) max_out = 1;
  VolPlan cand[kMaxCand];
  double cscore[kMaxCand];
  int ncand = 0;
  // candidate Ay: 1 and every register radix (fixed array: planning
  // allocates nothing)
  int ays[1 + sizeof(kRadixSet) / sizeof(kRadixSet[0])];
  int nays = 0;
  ays[nays++] = 1;
  for (int r : kRadixSet) ays[nays++] = r;
  for (int ai = 0; ai < nays; ++ai) {
    const int ay = ays[ai];
    if (ny % ay) continue;
    const int by = ny / ay;
    AxisPlan ab;
    if (!plan_axis(by, &ab)) continue;
    for (int W : {1, 2, 4, 8}) {
      const long long zsm = (long long)nz * by * W * 8;
      if (zsm > kSmemMax) continue;
      for (int G = 1; G <= 16; ++G) {
        if (by % G) continue;
        const long long xysm = (long long)G * ay * P.rowStride * 8;
        if (xysm > kSmemMax) continue;
        const int KG = (P.XS + W - 1) / W;
        const long long xy_blocks = (long long)nz * (by / G);
        const long long z_blocks = (long long)ay * KG;
        const int occ_xy = std::min(8, (int)(kSmemPerSM / (xysm + 1024)));
        const int occ_z = std::min(8, (int)(kSmemPerSM / (zsm + 1024)));
        const double seg = (double)G * W * 8;
        double score = 0;
        score += 10.0 * std::min(std::min(occ_xy, occ_z), 3);
        score += seg >= 32 ? 6.0 : seg / 32.0 * 6.0;
        score += (xy_blocks >= 296 ? 3.0 : 3.0 * xy_blocks / 296.0);
        score += (z_blocks >= 296 ? 3.0 : 3.0 * z_blocks / 296.0);
        score -= 4.0 * ((double)KG * W / P.XS - 1.0);
        score -= 0.05 * std::abs(ay - 16);
        score -= 0.02 * G;  // prefer fewer rows per tile at equal merit
        int pos = ncand;
        while (pos > 0 && score > cscore[pos - 1]) --pos;
        if (pos < max_out) {
          const int last = std::min(ncand, max_out - 1);
          for (int q = last; q > pos; --q) {
            cand[q] = cand[q - 1];
            cscore[q] = cscore[q - 1];
          }
          VolPlan c = P;
          c.Ay = ay; c.By = by; c.G = G; c.W = W; c.KG = KG;
          c.ayB = ab;
          c.xy_smem = (int)xysm;
          c.z_smem = (int)zsm;
          c.xy_blocks = (int)xy_blocks;
          c.z_blocks = (int)z_blocks;
          cand[pos] = c;
          cscore[pos] = score;
          if (ncand < max_out) ++ncand;
        }
      }
    }
  }
  if (ncand == 0) {
    if (why) *why = "no tiling of y=" + std::to_string(ny) + ", z=" + std::to_string(nz) +
                    " fits in shared memory with the supported radices";
    return 0;
  }
  int nout = 0;
  for (int c = 0; c < ncand; ++c)
    if (finalize_plan(cand[c], why)) out[nout++] = cand[c];
  return nout;
}


void plan_tables(const VolPlan& P, std::vector<int>* xrev, std::vector<TwTable>* tabs) {
  xrev->assign(std::max(P.M, 1), 0);
  for (int k = 0; k < P.M; ++k) (*xrev)[k] = xrev_slot(P.ax, k);
  TwTable t[kPlanTwTables];
  plan_twiddle_tables(P, t);
  tabs->assign(t, t + kPlanTwTables);
}

// ------------------------------------------------------- column-pair passes
// Radix sequence of n with the fewest passes (then the smallest largest
// radix), non-increasing, from the radices up to 16 and, where n has those
// factors, 17 and 19.
static void search_pair(int n, int depth, int* cur, int* best, int* best_len, int* best_max) {
  if (n == 1) {
    const int mx = depth ? cur[0] : 0;
    if (depth < *best_len || (depth == *best_len && mx < *best_max)) {
      *best_len = depth;
      *best_max = mx;
      for (int i = 0; i < depth; ++i) best[i] = cur[i];
    }
    return;
  }
  if (depth >= kMaxPasses || depth + 1 > *best_len) return;
  for (int r = 19; r >= 2; --r) {
    if (r == 18 || n % r) continue;
    if (depth > 0 && r > cur[depth - 1]) continue;
    cur[depth] = r;
    search_pair(n / r, depth + 1, cur, best, best_len, best_max);
  }
}

// FDiv is exact for n d < 2^32.  What the passes divide are indices into a tile in
// shared memory, by extents of that tile: both below the 16-byte slots it has.
static_assert((kSmemMax / 16ll) * (kSmemMax / 16) < (1ll << 32), "FDiv");

static bool pair_axis(int n, bool padded, PairAxis* A) {
  std::memset(A, 0, sizeof(*A));
  A->n = n;
  if (n == 1) return true;
  int cur[kMaxPasses], best[kMaxPasses];
  int best_len = kMaxPasses + 1, best_max = INT_MAX;
  search_pair(n, 0, cur, best, &best_len, &best_max);
  if (best_len > kMaxPasses) return false;
  A->npass = best_len;
  const int rl = best[best_len - 1];
  // the last pass's consecutive threads are rl slots apart: an even rl gets
  // one empty slot per rl elements, so the stride is odd (no bank conflicts)
  A->pad = padded && best_len > 1 && rl % 2 == 0 ? rl : 0;
  int len = n;
  for (int s = 0; s < best_len; ++s) {
    A->radix[s] = best[s];
    A->len[s] = len;
    A->span[s] = len / best[s];
    A->plen[s] = len + (A->pad ? len / A->pad : 0);
    A->pspan[s] = A->span[s] + (A->pad ? A->span[s] / A->pad : 0);
    A->dspan[s] = fdiv_by(A->span[s]);
    A->dper[s] = fdiv_by(n / best[s]);
    len /= best[s];
  }
  A->dpad = fdiv_by(A->pad);
  return true;
}

static bool pair_big(const PairAxis& A) {
  for (int s = 0; s < A.npass; ++s)
    if (A.radix[s] > 16) return true;
  return false;
}

// Rough cycles of a pass kernel on the chip's 148 SMs: `n` sweeps of items[s]
// work items of radix r[s] by blocks of `threads`, as many blocks per SM as
// shared memory and registers allow.  A round of a sweep costs its latency
// (lat[s] and about 140 cycles per radix point: some 25 instructions at a
// warp's 6 cycles each) or the issue slots of all resident warps, whichever is
// more; both constants from the passes' profiles at the 320x320x96 box.
static double pair_cost(const int* items, const int* r, const int* lat, int n, int threads,
                        int smem, long long blocks, bool big) {
  const int by_regs = (big ? 256 : 512) / threads, by_smem = kSmemPerSM / (smem + 1024);
  int bps = std::min(by_regs, by_smem);
  if (bps < 1) return 1e30;
  const long long per_sm = (blocks + 147) / 148;
  const long long waves = (per_sm + bps - 1) / bps;
  bps = (int)((per_sm + waves - 1) / waves);
  double t = 1500;
  for (int s = 0; s < n; ++s) {
    const int rounds = (items[s] + threads - 1) / threads;
    t += rounds * std::max(lat[s] + 140.0 * r[s], bps * (threads / 32) * 10.0 * r[s]);
  }
  return t * (double)waves;
}

static int pair_threads(const int* items, const int* r, const int* lat, int n, int smem,
                        long long blocks, bool big, double* cost) {
  int best = 0;
  *cost = 1e30;
  for (int t = 32; t <= (big ? 128 : 256); t += 32) {
    const double c = pair_cost(items, r, lat, n, t, smem, blocks, big);
    if (c < *cost) {
      *cost = c;
      best = t;
    }
  }
  return best;
}

bool make_pair_plan(int nx, int ny, int nz, PairPlan* out) {
  PairPlan P;
  std::memset(&P, 0, sizeof(P));
  P.nx = nx;
  P.ny = ny;
  P.nz = nz;
  P.XS = nx / 2 + 1;
  P.KG = (P.XS + 1) / 2;
  out->ok = 0;
  if (nx < 2 || nz < 2 || nx > kPairMaxNx || (long long)nx * ny * nz >= (1ll << 31)) return false;
  if (!pair_axis(nx, true, &P.ax) || !pair_axis(nz, false, &P.az)) return false;
  P.rowlen = nx + (P.ax.pad ? nx / P.ax.pad : 0);
  double best = 1e30;
  for (int ay = 1; ay <= 19; ++ay) {
    if (ny % ay || ay == 18) continue;
    PairPlan c = P;
    c.Ay = ay;
    c.By = ny / ay;
    if (!pair_axis(c.By, false, &c.ayB)) continue;
    c.NQ = (ay + 3) / 4;
    c.BS = c.By | 1;
    c.spec_elems = 2ll * ay * c.KG * nz * c.By;
    if (c.spec_elems >= (1ll << 31)) continue;
    c.dBy = fdiv_by(c.By);
    const long long zsm = ((long long)nz * c.BS + nz + c.By) * 16;
    if (zsm > kSmemMax) continue;
    c.z_smem = (int)zsm;
    c.z_blocks = ay * c.KG;
    c.big_z = pair_big(c.az) || pair_big(c.ayB);
    c.big_xy = ay > 16 || pair_big(c.ax);
    // a sweep's latency: shared memory only, or through L2 or HBM
    constexpr int kSm = 500, kFar = 2000;
    int items[4 * kMaxPasses], r[4 * kMaxPasses], lat[4 * kMaxPasses], n = 0;
    for (int s = 0; s < c.ayB.npass; ++s)
      for (int d = 0; d < 2; ++d, ++n) {
        lat[n] = kSm;
        r[n] = c.ayB.radix[s];
        items[n] = nz * (c.By / r[n]);
      }
    for (int s = 0; s < c.az.npass; ++s)
      for (int d = 0; d < 2; ++d, ++n) {
        lat[n] = s == c.az.npass - 1 && d == 0 ? kFar : kSm;
        r[n] = c.az.radix[s];
        items[n] = c.By * (nz / r[n]);
      }
    double zc, xc;
    c.z_threads = pair_threads(items, r, lat, n, c.z_smem, c.z_blocks, c.big_z, &zc);
    if (!c.z_threads) continue;
    for (int tg : {1, 2, 3, 4, 8}) {
      if (c.By % tg) continue;
      const long long xsm = ((long long)tg * c.NQ * c.rowlen + tg * ay) * 16 + nx * 8;
      if (xsm > kSmemMax) continue;
      c.TG = tg;
      c.dTG = fdiv_by(tg);
      c.xy_smem = (int)xsm;
      n = 0;
      for (int d = 0; d < 2; ++d, ++n) {
        r[n] = ay + (tg == 1 ? 6 : 2);  // the column step, its global accesses wider for tg > 1
        lat[n] = d == 0 ? kFar : kSm;
        items[n] = tg * c.KG;
      }
      for (int s = 0; s < c.ax.npass; ++s)
        for (int d = 0; d < (s == 0 ? 1 : 2); ++d, ++n) {
          lat[n] = s == 0 ? kFar : kSm;
          r[n] = s == 0 ? 2 * c.ax.radix[s] : c.ax.radix[s];  // the first and last pass in one
          items[n] = tg * c.NQ * (nx / c.ax.radix[s]);
        }
      c.xy_threads = pair_threads(items, r, lat, n, c.xy_smem, (long long)nz * (c.By / tg), c.big_xy, &xc);
      if (!c.xy_threads) continue;
      // one line's columns are half sectors of the spectrum: 8% in the XY passes
      // at the 320x320x96 box
      if (tg == 1) xc *= 1.08;
      if (zc + xc < best) {
        best = zc + xc;
        *out = c;
        out->ok = 1;
      }
    }
  }
  if (!out->ok) return false;
  int off = 0;
  out->ax.tw_off = off; off += nx;
  out->ayB.tw_off = off; off += out->By;
  out->az.tw_off = off; off += nz;
  out->tw_ny_off = off; off += ny;
  out->twiddle_count = off;
  return true;
}

void pair_tables(const PairPlan& P, std::vector<int>* slots, std::vector<TwTable>* tabs) {
  slots->assign(P.nx, 0);
  for (int k = 0; k < P.nx; ++k) {
    int rem = k, e = 0;
    for (int s = 0; s < P.ax.npass; ++s) {
      e += (rem % P.ax.radix[s]) * P.ax.span[s];
      rem /= P.ax.radix[s];
    }
    (*slots)[k] = e + (P.ax.pad ? e / P.ax.pad : 0);
  }
  *tabs = {TwTable{P.ax.tw_off, P.nx, P.nx}, TwTable{P.ayB.tw_off, P.By, P.By},
           TwTable{P.az.tw_off, P.nz, P.nz}, TwTable{P.tw_ny_off, P.ny, P.ny}};
}

}  // namespace clarity
