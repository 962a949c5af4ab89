// Host check of the CTA-pair tile order (gram_core.cuh: make_pair_space and
// pair_coords): every 256 x 256 tile of the full and of the upper set appears
// exactly once, for many shapes and band widths.
#include "gram_core.cuh"

#include <cstdio>
#include <vector>

using namespace gt;

static bool check(int64_t nr, int64_t nc, int symmetric, int64_t group) {
  const PairSpace ps = make_pair_space(nr, nc, symmetric, group);
  std::vector<char> seen(size_t(ps.tr * ps.tc), 0);
  int64_t expect = 0;
  for (int64_t ti = 0; ti < ps.tr; ti++)
    for (int64_t tj = 0; tj < ps.tc; tj++) expect += !symmetric || ti <= tj;
  bool ok = expect == ps.ntiles;
  for (int64_t t = 0; ok && t < ps.ntiles; t++) {
    int64_t ti = -1, tj = -1;
    pair_coords(ps, t, ti, tj);
    ok = ti >= 0 && ti < ps.tr && tj >= 0 && tj < ps.tc && (!symmetric || ti <= tj) &&
         !seen[size_t(ti * ps.tc + tj)];
    if (ok) seen[size_t(ti * ps.tc + tj)] = 1;
  }
  if (!ok)
    std::printf("FAIL nr=%lld nc=%lld symmetric=%d group=%lld\n", (long long)nr, (long long)nc,
                symmetric, (long long)group);
  return ok;
}

int main() {
  for (int64_t nr : {1, 255, 256, 257, 1000, 4096, 8193, 20000, 33000, 100001})
    for (int64_t g : {1, 2, 3, 4, 8, 12, 16}) {
      if (!check(nr, nr, 1, g)) return 1;
      for (int64_t nc : {int64_t(1), int64_t(300), int64_t(5000), nr + 77})
        if (!check(nr, nc, 0, g)) return 1;
    }
  std::printf("ok\n");
  return 0;
}
