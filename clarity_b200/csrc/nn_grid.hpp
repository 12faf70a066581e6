// nn_grid.hpp -- launch geometry of the convolution's weight gradient
// (k_conv3_wgrad, nn.cu), in plain C++ so that it can be checked without a GPU.
#pragma once
#include <algorithm>

namespace clarity {
namespace nn {

constexpr int kTZ = 2, kTY = 8, kTX = 8;  // voxel tile

// Block (x, y, z): input chunk x % (cin / 16), output channels from
// x / (cin / 16) * bm, run z * gy + y of `runs` (none beyond): tiles
// [ntiles * run / runs, ntiles * (run + 1) / runs).
struct WgradGrid {
  int bm;  // output channels a block
  int tilesx, tilesy, ntiles;
  int cols;  // blocks a run
  int runs, gy, gz;
};

// False for volumes of 2^31 voxels or more (the kernel's voxel indices are int).
inline bool wgrad_grid(int D, int H, int W, int cin, int cout, int sms, WgradGrid* g) {
  if ((long long)D * H >= (1ll << 31) || (long long)D * H * W >= (1ll << 31)) return false;
  // 32 output channels a block where they divide: twice the MMAs per input
  // fragment; more would not leave registers for three blocks per SM
  g->bm = cout % 32 == 0 ? 32 : 16;
  g->tilesx = W / kTX + (W % kTX != 0);
  g->tilesy = H / kTY + (H % kTY != 0);
  g->ntiles = g->tilesx * g->tilesy * (D / kTZ + (D % kTZ != 0));
  g->cols = (cin / 16) * (cout / g->bm);
  // runs of tiles: enough blocks for the SMs several times over, but at least
  // four tiles each (once every SM has a block) so that a block's 27 * 16 * bm
  // atomics stay a small part, and at most 12 (96 MMAs into one accumulator): the
  // tensor cores' FP32 sums lose about an ulp a step, and with 31 tiles a run dW's
  // error against 64 bits was 1.3e-6 where runs of 128 MMAs had 8e-7
  const int n = g->ntiles, cols = g->cols;
  g->runs = std::max(n / 12 + (n % 12 != 0),
                     std::min((sms * (g->bm == 16 ? 4 : 3) + cols - 1) / cols,
                              std::max(n / 4, std::min(n, sms / cols + 1))));
  // over two grid dimensions of at most 65535 (a 512x512x384 volume has 65536 runs)
  g->gz = (g->runs + 65534) / 65535;
  g->gy = (g->runs + g->gz - 1) / g->gz;
  return true;
}

}  // namespace nn
}  // namespace clarity
