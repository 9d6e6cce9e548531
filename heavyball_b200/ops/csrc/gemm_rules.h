// Which tile the split-operand GEMMs take (tf32_gemm.cu, split16_gemm.cu): 128 x 128 per CTA, two CTAs to an SM, or 256 x 256 per pair of
// CTAs.  `pairs`: pairs that can be resident at once.  Arithmetic on sizes only, also compiled by a CPU test.
#pragma once
#include <stdint.h>

namespace hb {

inline int64_t output_tiles(int64_t M, int64_t N, int64_t tile, bool symmetric) {
  const int64_t m = (M + tile - 1) / tile, n = (N + tile - 1) / tile;
  return symmetric ? n * (n + 1) / 2 : m * n;
}

enum TileChoice : int {
  kSmallTiles = 0,
  kPairTiles = 1,
  kPairTilesSmallDiagonal = 2  // symmetric: pairs, with the diagonal stored as 128 x 128 tiles store it (the bits of the small tiles)
};

// Split tf32.  Pairs once there are 96 of their tiles and K is long enough to pay for their epilogue.  (The line stands where it stood for
// the one-CTA tile of this size that the pairs replaced: whether an entry of a symmetric product near the diagonal is computed or mirrored
// depends on the tile, and with it its last bit.)
// Symmetric products that this line refuses may take pairs with the small tiles' diagonal.  130 sizes measured, 128 / pairs in us:
//   - Small tiles that do not fit at once: pairs in two waves from K = 256 on (3072 x 3072 x 2048 163 / 134, 4 of 1536 x 1536 x 1024 95 / 80,
//     x 256 48.0 / 47.2, 4 of 2048 x 2048 x 256 55.3 / 49.2).  With a shorter K the pairs' epilogue shows (4 of 1536 x 1536 x 192 44.0 / 45.1, x 64
//     35.8 / 41.0, 4 of 2048 x 2048 x 64 42.0 / 44.0).
//   - They do, but two on an SM: pairs in one wave from K = 1024 on (2 of 2048 x 2048 x 5504 251 / 204, 2 of 1536 x 1536 x 1024 45.7 / 44.5), not
//     in two (8 of 1024 x 1024 x 2048 112 / 143).
//   - One on an SM: only a long K and enough tiles (2048 x 2048 x 5504 206 / 165, 2 of 1024 x 1024 x 4096 144 / 127, 1024 x 1024 x 5504
//     142 / 158, 2048 x 2048 x 2048 62.5 / 69.3).
inline TileChoice tf32_tiles(int64_t M, int64_t N, int64_t K, int64_t batch, bool symmetric, int64_t pairs) {
  if (M < 256 || N < 256) return kSmallTiles;
  const int64_t small = output_tiles(M, N, 128, symmetric) * batch, big = output_tiles(M, N, 256, symmetric) * batch;
  if (K >= 512 && big >= 96) return kPairTiles;
  if (!symmetric) return kSmallTiles;
  bool take = false;
  if (small > 4 * pairs)
    take = K >= 256 && big <= 2 * pairs;
  else if (big <= pairs)
    take = small > 2 * pairs ? K >= 1024 : K >= 4096 && big >= 20;
  return take ? kPairTilesSmallDiagonal : kSmallTiles;
}

}  // namespace hb
