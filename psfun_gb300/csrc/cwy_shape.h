// cwy_shape.h -- how the rows of a k_ar_cwy solve are laid over blocks, warps
// and lanes (host arithmetic alone, so that it can be checked without a GPU).
#pragma once

#include <cstdint>

namespace psf {

constexpr int kCwyThreads = 640;  // threads of a block, at most
// Rows of one lane in the dots, at most: the kernel has one instance of its
// loop per count.  With 16 monitor blocks on 152 SMs a block of 2^19 - 1 rows
// owns 3856 of them, seven per lane of 20 warps.
constexpr int kCwyMaxRt = 7;

struct CwyShape {
  int G = 0;  // blocks that run the steps (0: none)
  int chunk = 0, rt = 1, threads = 0;  // rows per block and per lane, threads per block
};

// n rows on at most max_blocks blocks; G = 0 where a lane would need more than
// kCwyMaxRt rows.
inline CwyShape cwy_shape(int64_t n, int max_blocks) {
  CwyShape p;
  if (n < 1 || max_blocks < 1) return p;
  const int64_t blocks = (n + 63) / 64;
  int64_t G = blocks < max_blocks ? blocks : max_blocks;
  int64_t chunk = (n + G - 1) / G;
  chunk = (chunk + 1) & ~(int64_t)1;
  G = (n + chunk - 1) / chunk;
  const int64_t rt = (chunk + kCwyThreads - 1) / kCwyThreads;
  if (rt > kCwyMaxRt) return p;
  p.G = (int)G;
  p.chunk = (int)chunk;
  p.rt = (int)rt;
  const int nrg = (p.chunk + 32 * p.rt - 1) / (32 * p.rt);
  p.threads = 32 * (nrg >= 16 ? nrg : nrg * (16 / nrg));
  return p;
}

}  // namespace psf
