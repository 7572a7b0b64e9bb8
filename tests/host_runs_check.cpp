// Host-side check of htr_b200/csrc/run_arith.cuh: every quotient without a division against the division, and the runs of thread blocks against
// their definition.  Built and run by tests/test_host_logic.py; prints "ok" and exits 0 on success.
#include <cstdio>
#include <vector>

#include "../htr_b200/csrc/run_arith.cuh"

using namespace htr;

static long long bad = 0;
static void same(long long got, long long want, const char* what, long long a, long long b) {
  if (got != want && ++bad < 10) std::printf("%s(%lld, %lld): got %lld want %lld\n", what, a, b, got, want);
}

int main() {
  // one-row kernel of a chain: blocks per row block up to 128, up to 16384 row blocks
  for (int hb = 1; hb <= 128; ++hb) {
    const unsigned magic = reciprocal(hb);
    for (int rb = 0; rb <= 16384; ++rb)
      for (int d = -1; d <= 1; ++d) {
        const int u = rb * hb + d;
        if (u >= 0) same(quotient(u, magic), u / hb, "quotient", u, hb);
      }
  }
  // parts of a cluster
  for (int split = 1; split <= 16; ++split)
    for (int hb = split; hb <= 2048; ++hb)
      for (int part = 0; part <= split; ++part)
        same(part_begin(part, hb / split, hb % split, part_reciprocal(split)), (long long)part * hb / split, "part_begin", hb, split * 100 + part);
  // flat runs: units just at and above the grid, ragged, remainder 0, and beyond 2^24, where the float guess is not exact
  const int grids[] = {1, 2, 3, 7, 64, 147, 148, 296, 444, 592, 1184, 1625};
  for (int G : grids) {
    std::vector<int> units = {G, G + 1, 2 * G - 1, 2 * G, 17 * G + 5, 1187 * 64, 75968, 1 << 20, (1 << 24) + 1, (1 << 24) + 12345, 100000007, 1 << 28};
    for (int U : units) {
      if (U < G) continue;
      const FlatRuns runs(U / G, U % G, reciprocal(G), (float)G / (float)U);
      const EvenRuns even(U, G);
      for (int b = 0; b <= G; ++b) {
        const long long lo = (long long)b * U / G;
        same(runs.begin(b), lo, "FlatRuns.begin", U, b);
        same(even.begin(b), (long long)b * (U / G) + (b < U % G ? b : U % G), "EvenRuns.begin", U, b);
        for (int d = -2; d <= 2; ++d) {
          const long long x = lo + d;
          if (x < 0 || x >= U) continue;
          same(runs.owner((int)x), unit_owner(x, G, U), "FlatRuns.owner", U, x);
          const int o = runs.owner((int)x), e = even.owner((int)x);
          if (!(runs.begin(o) <= x && x < runs.begin(o + 1)) || !(even.begin(e) <= x && x < even.begin(e + 1))) ++bad;
        }
      }
    }
  }
  // row block of a unit by the float reciprocal
  for (int cg = 1; cg <= 1024; ++cg)
    for (long long rb = 0; rb < 16384; rb = rb < 64 ? rb + 1 : rb * 3 / 2)
      for (int d = -2; d <= 2; ++d) {
        const long long x = rb * cg + d;
        if (x >= 0 && x < (1ll << 31)) same(quotient((int)x, cg, 1.0f / (float)cg), x / cg, "quotient by float", x, cg);
      }
  if (bad) return 1;
  std::printf("ok\n");
  return 0;
}
