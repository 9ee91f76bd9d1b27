// Prints what the rules of tilemega_b200/csrc/linear_rules.h choose, a line per line of input:
// "linear t n heads chunks sms" -> "index splits pair"; "experts slots experts up width ff" (148 SMs) -> rows of a tile and "index splits" of
// the up product.
#include <cstdio>
#include <cstring>

#include "linear_rules.h"

int main() {
  char what[16];
  int a, b, c, d, e;
  while (std::scanf("%15s %d %d %d %d %d", what, &a, &b, &c, &d, &e) == 6) {
    if (!std::strcmp(what, "experts")) {
      const int rows = tmb::ExpertRows(a, b, c, d, e, 148);
      const tmb::LinearTiling t = tmb::ChooseExpertLinear(a, b, rows, c, (d + 63) / 64, 148);
      std::printf("%d %d %d\n", rows, t.index, t.splits);
      continue;
    }
    const tmb::LinearTiling t = tmb::ChooseLinear(a, b, c, d, e);
    std::printf("%d %d %d\n", t.index, t.splits, int(t.pair));
  }
  return 0;
}
