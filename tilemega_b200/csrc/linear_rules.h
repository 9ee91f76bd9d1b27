// How a ragged step's products are cut into tiles: plain rules on sizes, apart from the kernels (linear.cu).
#pragma once
#include <algorithm>

namespace tmb {

constexpr int kRowsM = 128;                 // weight rows per tile
constexpr int kStepK = 64;                  // 16-bit elements per 128-byte swizzle row
constexpr int kWide = 256;                  // tokens of the widest tiles
constexpr int kMaxCluster = 8;

struct LinearTiling {
  int index = 0;                            // into 16, 32, 64, 128, 256 tokens a tile
  int splits = 1;                           // of K, over a cluster
  bool pair = false;                        // 256 tokens: by pairs of CTAs, 256 weight rows a tile
};

// Turns that `tiles` take, `at_once` at a time.
inline int Rounds(long long tiles, int at_once) { return int((tiles + at_once - 1) / at_once); }

// The widest tile that gives most SMs a CTA, else the narrowest that covers the tokens (at most 128), with K split over a cluster until the
// SMs are covered; further, up to two CTAs per SM, where a part keeps a long run of K. `heads`: products by heads, n rows each (0: one product).
//
// The widest by pairs of CTAs, unless 256 weight rows a tile take a round more than 128 do (49 tiles of weight rows by 3 of tokens: 147 CTAs are
// one round, 75 pairs two). At as many rounds a pair is faster: projection of 10240 rows x 4096 by 2040 tokens 105 us for 118, gated unit of 28672
// rows 297 for 318, of 16384 x 2048 by 431 35.0 for 36.5. Products by heads have 3 to 9 chunks of K and tiles end with a head's rows: 32 heads
// of 128 rows by 1000 and 2000 tokens 20.3 and 28.9 us by pairs, 18.3 and 26.5 by single CTAs; 16 heads by 1800 and 2000 19.7 and 17.5, 16.1 and
// 13.9; 32 heads of 576 rows and 3 chunks 33.4 and 55.5, 29.7 and 49.3.
inline LinearTiling ChooseLinear(int t, int n, int heads, int chunks, int sms) {
  LinearTiling c;
  const int of_head = (n + kRowsM - 1) / kRowsM, tiles = of_head * std::max(heads, 1), wide_tokens = (t + kWide - 1) / kWide;
  if (t > 128 && tiles * wide_tokens * 10 >= sms * 8) {
    c.index = 4;
    c.pair = !heads && Rounds((long long)((of_head + 1) / 2) * wide_tokens, sms / 2) <= Rounds((long long)(tiles) * wide_tokens, sms);
    return c;
  }
  while (c.index < 3 && (16 << c.index) < t) ++c.index;
  const int grid = tiles * ((t + (16 << c.index) - 1) / (16 << c.index));
  while (c.splits < kMaxCluster && grid * c.splits <= sms && chunks / (c.splits * 2) >= (grid * c.splits * 10 < sms * 8 ? 4 : 16)) c.splits *= 2;
  return c;
}

// Most tiles of `tile_rows` that a step's slots can fall into: full ones, and one more for every expert in use.
inline int MostExpertTiles(int slots, int experts, int tile_rows) { return slots / tile_rows + std::min(experts, slots); }

// Roughly what a product of n rows an expert over `chunks` of K takes in tiles of `rows` slots: rounds of tiles, a CTA an SM or two that share
// one, by the rows a tile copies. (An expert's slots end where they end: half a tile more than they fill, but no less than one.)
inline double ExpertCost(int slots, int experts, int rows, int n, int chunks, int sms) {
  const double share = double(slots) / experts, each = std::max(1.0, share / rows + 0.5);
  const double tiles = experts * each * ((n + kRowsM - 1) / kRowsM);
  return Rounds((long long)(tiles), sms) * (kRowsM + share / each) * chunks * (rows == kWide ? 1.0 : 0.9);
}

// Slots per tile: an expert's on average; most experts have no more than 4/3 of it. 256 (linear_wide) where its rounds end before those of 128
// (linear_tiles, two CTAs an SM, K split over the SMs that few tiles leave idle) for both products of an expert together: `up` rows over
// `width` columns, `width` rows over `ff`. Both by 256 and by 128, us, width 2048: 128 experts of 1152, 128 slots each 311 / 359; 32 of 768, 250 slots
// 114 / 140; 16 of 2048, 125 slots 92 / 110; but 8 of 512, 125 slots 49 / 38, 8 of 1024, 500 slots 95 / 76, 32 of 768, 125 slots 95 / 89.
inline int ExpertRows(int slots, int experts, int up, int width, int ff, int sms) {
  const int share = (slots + experts - 1) / experts;
  int rows = 16;
  while (rows < kWide && rows * 3 < share * 4) rows *= 2;
  if (rows < kWide) return rows;
  auto cost = [&](int of) {
    return ExpertCost(slots, experts, of, up, (width + kStepK - 1) / kStepK, sms) + ExpertCost(slots, experts, of, width, (ff + kStepK - 1) / kStepK, sms);
  };
  return cost(kWide) <= cost(kWide / 2) ? kWide : kWide / 2;
}

// Per expert: the tile width is that of the slot table; K splits until the tiles to be expected cover the SMs.
inline LinearTiling ChooseExpertLinear(int slots, int experts, int tile_rows, int n, int chunks, int sms) {
  LinearTiling c;
  while ((16 << c.index) < tile_rows) ++c.index;
  if (c.index == 4) return c;
  const int grid = MostExpertTiles(slots, experts, tile_rows) * ((n + kRowsM - 1) / kRowsM);
  while (c.splits < kMaxCluster && grid * c.splits <= sms && chunks / (c.splits * 2) >= 4) c.splits *= 2;
  return c;
}

}  // namespace tmb
