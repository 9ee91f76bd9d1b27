// The roles of a persistent product (linear_wide, encoder_wide): a CTA, or a pair of them, takes every `step`-th tile from `first` on. One warp fills a ring of S
// stages with the chunks of K of tile after tile, one issues the products into one of two accumulators, eight warps write the other
// one out. Everything that touches memory or a barrier is the caller's (a wait returns false once it has given up), so that
// the roles also run on the host, against waits that fail there. Below them the loader of attend_portions, for the same reason.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TMB_ROLE __device__ __forceinline__
#else
#define TMB_ROLE inline
#endif

namespace tmb {

struct Filled {
  int chunks;      // requested
  bool ok;         // and multiplied: no copy is under way any more, nor an arrival on one of this CTA's barriers
};

// tile(i): the tile from here on; weights(chunk, s), rows(chunk, s): copies of one chunk; inputs_there(): before the first rows.
// Not ok: the copies of the last S chunks may be under way still (drain_stages, drain_pair).
template <int S, class Tile, class Weights, class There, class Rows, class Empty>
TMB_ROLE Filled fill_stages(int first, int step, int tiles, int chunks, Tile tile, Weights weights, There inputs_there, Rows rows, Empty empty) {
  int c = 0;
  bool ok = true;
  for (int i = first; i < tiles && ok; i += step) {
    tile(i);
    int early = 0;
    if (i == first) {                     // weights do not depend on the kernel before this one
      for (; early < S && early < chunks; ++early) weights(early, early);
      inputs_there();
    }
    for (int chunk = 0; chunk < chunks; ++chunk, ++c) {
      const int s = c % S;
      if (c >= S) ok = empty(s, uint32_t(c / S - 1) & 1u);
      if (!ok) break;
      if (c >= early) weights(chunk, s);
      rows(chunk, s);
    }
  }
  for (int j = c > S ? c - S : 0; j < c && ok; ++j) ok = empty(j % S, uint32_t(j / S) & 1u);
  return {c, ok};
}

// Before the CTA may go: landed(s, parity) waits for a phase of full[s], for a limited time.
template <int S, class Landed> TMB_ROLE void drain_stages(int chunks, Landed landed) {
  for (int j = chunks > S ? chunks - S : 0; j < chunks; ++j) landed(j % S, uint32_t(j / S) & 1u);
}
// The same for a pair whose copies all count on the first CTA's barriers, by the first CTA, once both loaders have ended: they may have
// requested different numbers of chunks. without(s): the second CTA's share of a chunk will not come; only(s): nothing but that will.
template <int S, class Without, class Only, class Landed> TMB_ROLE void drain_pair(int mine, int peers, Without without, Only only, Landed landed) {
  const int both = mine < peers ? mine : peers, all = mine < peers ? peers : mine;
  for (int j = all > S ? all - S : 0; j < all; ++j) {
    if (j >= both) {
      if (mine > peers) without(j % S);
      else only(j % S);
    }
    landed(j % S, uint32_t(j / S) & 1u);
  }
}

// tile(i, k): the CTA's k-th tile from here on; products(chunk, s): of one chunk, behind them the stage is free;
// commit(b): sum_full[b] arrives once all products so far are done; done(b, parity): waits for that, for a limited time. The role ends behind
// the last commit's arrival, whatever the writers do: no product is under way any more when tensor memory goes.
template <int S, class Tile, class SumEmpty, class Full, class Products, class Commit, class Done>
TMB_ROLE void multiply_tiles(int first, int step, int tiles, int chunks, Tile tile, SumEmpty sum_empty, Full full, Products products, Commit commit, Done done) {
  int c = 0, k = 0, last = -1;        // last: the tile committed last
  bool ok = true;
  for (int i = first; i < tiles && ok; i += step, ++k) {
    if (k > 1) ok = sum_empty(k & 1, uint32_t((k >> 1) - 1) & 1u);
    if (!ok) break;
    tile(i, k);
    for (int chunk = 0; chunk < chunks; ++chunk, ++c) {
      const int s = c % S;
      ok = full(s, uint32_t(c / S) & 1u);
      if (!ok) break;
      products(chunk, s);
    }
    commit(k & 1);
    last = k;
  }
  if (last >= 0) done(last & 1, uint32_t(last >> 1) & 1u);
}

// begin(i, k): before the wait for the CTA's k-th tile, where the warps may meet: all of them come there for every tile, also behind a
// wait that gave up in one of them. write(i, k, last) puts the tile out; written(k & 1) gives its accumulator back.
template <class Begin, class SumFull, class Write, class Written>
TMB_ROLE void write_tiles(int first, int step, int tiles, Begin begin, SumFull sum_full, Write write, Written written) {
  bool ok = true;
  int k = 0;
  for (int i = first; i < tiles; i += step, ++k) {
    begin(i, k);
    ok = ok && sum_full(k & 1, uint32_t(k >> 1) & 1u);
    if (!ok) continue;
    write(i, k, i + step >= tiles);
    written(k & 1);
  }
}

// Blocks of keys and values for attend_portions, through rings of KS whole blocks of keys and VS half blocks of values; the keys of a
// block are requested before the values of the one before it. keys(b, s), values(b, half, s): copies; the latter is true for a half
// that is not full, whose copies count on a barrier of their own, part_landed(parity), before part(b, half, s) hands it on.
// moved(b): places of later blocks. A wait that gave up: the *_drained wait for what was requested, for a limited time.
template <int KS, int VS, class Keys, class Values, class PartLanded, class Part, class Moved, class KeyEmpty, class ValueEmpty, class KeyDrained, class ValueDrained,
          class PartDrained>
TMB_ROLE bool fill_blocks(int blocks, Keys keys, Values values, PartLanded part_landed, Part part, Moved moved, KeyEmpty key_empty, ValueEmpty value_empty,
                          KeyDrained key_drained, ValueDrained value_drained, PartDrained part_drained) {
  int k = 0, v = 0, parts = 0;
  bool ok = true, landing = false;
  for (int b = -1; b < blocks && ok; ++b) {
    if (b + 1 < blocks) {
      if (k >= KS) ok = key_empty(k % KS, uint32_t(k / KS - 1) & 1u);
      if (!ok) break;
      keys(b + 1, k % KS);
      ++k;
    }
    for (int half = 0; half < 2 && b >= 0; ++half) {
      if (v >= VS) ok = value_empty(v % VS, uint32_t(v / VS - 1) & 1u);
      if (!ok) break;
      if (values(b, half, v % VS)) {
        ok = part_landed(uint32_t(parts) & 1u);
        landing = !ok;
        if (!ok) break;
        part(b, half, v % VS);
        ++parts;
      }
      ++v;
    }
    moved(b);
  }
  for (int j = k > KS ? k - KS : 0; j < k && ok; ++j) ok = key_empty(j % KS, uint32_t(j / KS) & 1u);
  for (int j = v > VS ? v - VS : 0; j < v && ok; ++j) ok = value_empty(j % VS, uint32_t(j / VS) & 1u);
  if (ok) return true;
  for (int j = k > KS ? k - KS : 0; j < k; ++j) key_drained(j % KS, uint32_t(j / KS) & 1u);
  for (int j = v > VS ? v - VS : 0; j < v; ++j) value_drained(j % VS, uint32_t(j / VS) & 1u);
  if (landing) part_drained(uint32_t(parts) & 1u);
  return false;
}

}  // namespace tmb
