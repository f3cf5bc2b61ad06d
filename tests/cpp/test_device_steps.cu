// Steps of the device code that also compile for the host, run on the CPU:
//   carries   the hand-over of a look-back unit's carries, with every slot
//             taken again at the moment it is handed on.
// Prints one line per check and ALL PASSED when every check holds.
#include "b2p_device/pipe.cuh"

#include <cstdio>
#include <vector>

namespace {

int g_failed = 0;

void check(bool ok, const char *what) {
  printf("%s: %s\n", what, ok ? "ok" : "FAILED");
  g_failed += !ok;
}

// A carry that records what it was made of, in order.
struct TraceOps {
  using Pub = std::vector<int>;
  static Pub combine(Pub a, const Pub &b) {
    a.insert(a.end(), b.begin(), b.end());
    return a;
  }
};

// Units of 1 .. 4 tiles.  The slot of a tile may hold a later tile's aggregate
// as soon as it is handed on (here: at once), so a carry made of what the slot
// holds after that is wrong.
void carries() {
  bool ok = true;
  for (int nt = 1; nt <= 4; ++nt) {
    std::vector<std::vector<int>> agg, got;
    for (int j = 0; j < nt; ++j) agg.push_back({100 + j});
    b2p::hand_on_carries<TraceOps>(
        {7}, nt, [&](int j) { return agg[j]; },
        [&](int j, const std::vector<int> &c) {
          got.push_back(c);
          agg[j] = {-1};
        });
    ok = ok && (int)got.size() == nt;
    std::vector<int> want{7};
    for (int j = 0; j < nt && ok; ++j) {
      ok = got[j] == want;
      want.push_back(100 + j);
    }
  }
  check(ok, "carries of a unit when its slots are taken again at once");
}

}  // namespace

int main() {
  carries();
  if (g_failed == 0) printf("ALL PASSED\n");
  return g_failed != 0;
}
