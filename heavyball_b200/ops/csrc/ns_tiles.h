// Which tile a launch of Newton-Schulz products takes (plain C++: the launcher, and a CPU test of the rule).
//
// A 256 x 256 tile on a pair of CTAs halves the operand bytes per flop but only as many pairs work as there are tiles.  Measured on
// one B200 (74 pairs, 296 one-CTA tiles resident), one product per launch, 507 sizes with all dimensions >= 512:
//   - The 128 x 128 tiles fit at once: up to 1.7 times as fast, at most 2 % slower.  Gram products, 128 / pairs:
//     8 of 512 x 512 8.5 / 12.1 us, 16 of 640 x 1920 18.4 / 31.8, 8 of 1024 x 1024 14.2 / 22.9, 2 of 2048 x 2048 22.6 / 24.7.
//   - They need more than one wave: pairs are as fast or faster, in the same number of waves or up to a third more (apply
//     products, 32 of 900 x 1300: 152.7 / 91.7 us).  All 15 products of GPT-2-small's 48 matrices: 128 / 98 us per launch, of a
//     Llama-3-8B layer 1.04 / 0.81 ms.  With half as many waves again they are not: 16 of 1024 x 1024 in two waves of small tiles
//     or three of pairs 25.7 / 30.4 us, 20 of 640 x 640 18.2 / 21.3.
//   - Rows along a long K that do not start on 128-byte lines: with two CTAs on an SM the small tile pays for its greater operand
//     traffic (6 of 900 x 1300 24.6 / 19.3 us, 3 of 1500 x 1700 34.0 / 25.1), and in every wave.  At K below 800 it still wins
//     (8 of 700 x 700 10.2 / 12.5).  Between 100 and 148 tiles it is faster by itself, but the apply product after it is then
//     already on pairs, and a chain that changes over twice a step is slower than one that does not (whole chains, small tiles /
//     pairs / both: 3 of 1000 x 1000 258 / 252 / 273 us, 4 of 1000 x 3000 566 / 404 / 474), hence the line at a third of the small
//     tiles that fit at once.
// Whole chains against "from 24 pair tiles on": 8 of 512 x 512 187 -> 133 us, 8 of 1024 x 1024 359 -> 270, 8 of 1024 x 4096
// 796 -> 651, 4 of 768 x 768 210 -> 156; the worst is 3 % slower (8 of 600 x 1800 311 -> 321).
#pragma once

namespace hb {

struct NsExtent {
  int M, N, K, batch;
  bool symmetric;
};

inline int ns_tiles(const NsExtent& p, int tile) {
  const int tm = (p.M + tile - 1) / tile, tn = (p.N + tile - 1) / tile;
  return (p.symmetric ? tm * (tm + 1) / 2 : tm * tn) * p.batch;
}

// Long enough in every dimension to fill a pair's tile and its main loop.
inline bool ns_pair_sized(const NsExtent& p) { return p.M >= 512 && p.N >= 512 && p.K >= 512; }

// Whether the products of a launch that are `ns_pair_sized` take pairs, on a device that holds `pairs` of them (and four small
// tiles in the place of one).
inline bool ns_take_pairs(const NsExtent* products, int n, int pairs) {
  long long small = 0, big = 0, unaligned = 0;
  for (int i = 0; i < n; ++i) {
    if (!ns_pair_sized(products[i])) continue;
    const int tiles = ns_tiles(products[i], 128);
    small += tiles;
    big += ns_tiles(products[i], 256);
    if (products[i].K % 64 != 0 && products[i].K >= 800) unaligned += tiles;
  }
  const long long small_waves = (small + 4 * pairs - 1) / (4 * pairs), big_waves = (big + pairs - 1) / pairs;
  if (2 * unaligned > small) return small_waves >= 2 || (3 * small > 4 * pairs && big_waves == 1);
  return small_waves >= 2 && 3 * big_waves <= 4 * small_waves;
}

}  // namespace hb
