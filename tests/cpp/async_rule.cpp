// Host check of which kernel an asynchronous run takes (rak_internal.hpp, alt_for): the faster one for 8 slots on
// large skewed graphs only. Regions are counted from degree sequences as the plan does. Prints "ok" or the case.
#include <cmath>
#include <cstdio>
#include <vector>

#include "rak_internal.hpp"

using namespace rak;

struct Case { const char *name; int64_t n; int degree; double hub_share; int slots, gpu_rule; bool batch; int64_t lane_max; int want; };

int main() {
  const int64_t M = int64_t(1) << 22;
  // hub_share: of the edges, in vertices of 2000 neighbours; the other vertices have `degree`
  const Case cases[] = {
      {"skewed", M, 32, 0.5, 8, 0, false, 256, ALT_FAST},
      {"skewed, larger lane limit", M, 32, 0.5, 8, 0, false, 1024, ALT_FAST},
      {"skewed, a little", M, 32, 0.3, 8, 0, false, 256, ALT_FAST},
      {"skewed, hardly", M, 32, 0.05, 8, 0, false, 256, ALT_NONE},
      {"even (planted partition, lattice)", M, 16, 0, 8, 0, false, 256, ALT_NONE},
      {"even, small lane limit", M, 16, 0, 8, 0, false, 8, ALT_NONE},
      {"even, larger", 2 * M, 16, 0, 8, 0, false, 256, ALT_NONE},
      {"skewed, 2 slots", M, 32, 0.5, 2, 0, false, 256, ALT_NONE},
      {"skewed, 4 slots", M, 32, 0.5, 4, 0, false, 256, ALT_NONE},
      {"skewed, 16 slots", M, 32, 0.5, 16, 0, false, 256, ALT_NONE},
      {"skewed, 1 slot", M, 32, 0.5, 1, 0, false, 256, ALT_NONE},
      {"skewed, GPU rules", M, 32, 0.5, 8, 1, false, 256, ALT_NONE},
      {"skewed, batch", M, 32, 0.5, 8, 0, true, 256, ALT_NONE},
      {"skewed, small", M - 1, 32, 0.5, 8, 0, false, 256, ALT_NONE},
      {"skewed, sparse", M, 6, 0.5, 8, 0, false, 256, ALT_NONE},
  };
  for (const Case &c : cases) {
    const Layout ly{c.lane_max, 65536, 8192};
    const int64_t m = c.n * c.degree, hubs = int64_t(double(m) * c.hub_share) / 2000;
    Regions rg{};
    rg.vcount[key_region(plan_key(2000, ly))] += hubs;
    rg.vcount[key_region(plan_key(c.degree, ly))] += c.n - hubs;
    const int got = alt_for(c.slots, MODE_ASYNC, c.gpu_rule, c.batch, c.n, m, ly, rg);
    if (got != c.want) { std::printf("%s: %d, not %d\n", c.name, got, c.want); return 1; }
  }
  std::printf("ok\n");
  return 0;
}
