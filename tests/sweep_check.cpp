// Checks the order of a sweep (sweep.h) on the CPU: for every (planes, slab,
// levels) each (level, plane) runs once, and what a plane's step needs, the
// previous level on the plane and its two neighbours, is ordered before it by
// stream order or an event; so is the last step of the previous sweep.
// Two launches that are not ordered may run at the same time: they must not
// be neighbours on the same level pair the wrong way round, which the first
// condition covers (a step touches only slots with its own values).
#include <cstdio>
#include <vector>

#include "../lbm-c_b200/csrc/sweep.h"

using lbmc::SweepPlan;

static int check(const SweepPlan &p, int levels) {
  const int slabs = p.slabs(levels);
  // before[a][b]: launch a is ordered before launch b
  const int n = slabs * levels;
  std::vector<std::vector<char>> before(n, std::vector<char>(n, 0));
  auto order = [&](int a, int b) {  // a before b, and all that is before a
    before[a][b] = 1;
    for (int c = 0; c < n; c++)
      if (before[c][a]) before[c][b] = 1;
  };
  int last[2] = {-1, -1};
  std::vector<int> who(levels * p.planes, -1);
  for (int k = 0; k < slabs; k++)
    for (int s = 0; s < levels; s++) {
      const int id = k * levels + s, st = k & 1;
      if (last[st] >= 0) order(last[st], id);
      if (k > 0 && s > 0) order((k - 1) * levels + s - 1, id);
      last[st] = id;
      const int b = p.begin(k, s, levels), e = p.end(k, s, levels);
      if (e <= b || e - b > p.planes || b < 0 || b >= p.planes || e > 2 * p.planes) return 1;
      for (int z = b; z < e; z++) {
        int &w = who[s * p.planes + z % p.planes];
        if (w >= 0) return 2;
        w = id;
      }
    }
  for (int s = 0; s < levels; s++)
    for (int z = 0; z < p.planes; z++) {
      const int id = who[s * p.planes + z];
      if (id < 0) return 3;
      if (s == 0) continue;
      for (int dz = -1; dz <= 1; dz++) {
        const int need = who[(s - 1) * p.planes + (z + dz + p.planes) % p.planes];
        if (need < 0 || !before[need][id]) return 4;
      }
    }
  return 0;
}

int main() {
  long long cases = 0;
  for (int planes = 3; planes <= 90; planes++)
    for (int slab = 1; slab <= 20; slab++)
      for (int levels = 2; levels <= SweepPlan::MAX_DEPTH; levels++) {
        SweepPlan p;
        p.planes = planes;
        p.slab = slab;
        p.depth = levels;
        if (planes < 2 * levels + 1) continue;
        if (const int bad = check(p, levels)) {
          printf("FAIL %d: planes %d slab %d levels %d\n", bad, planes, slab, levels);
          return 1;
        }
        cases++;
      }
  // What plan_sweep chooses is among them: room for every level, and nothing
  // for domains that stay in L2 or have too few planes.
  for (long long bytes = 1 << 12; bytes < (1ll << 33); bytes = bytes * 5 / 4 + 64)
    for (int planes = 1; planes < 5000; planes = planes * 5 / 4 + 1) {
      const SweepPlan p = lbmc::plan_sweep(planes, bytes, planes % 2 ? 2 : 4);
      if (p.depth < 1 || p.depth > SweepPlan::MAX_DEPTH) return printf("FAIL depth\n"), 1;
      if (p.depth > 1 && (planes < 2 * p.depth + 1 || p.slab < 1)) return printf("FAIL plan\n"), 1;
      if (p.depth > 1 && bytes * planes <= (126ll << 20)) return printf("FAIL in L2\n"), 1;
    }
  printf("OK %lld\n", cases);
  return 0;
}
