// Steps of the device code that also compile for the host, run on the CPU:
//   carries   the hand-over of a look-back unit's carries, with every slot
//             taken again at the moment it is handed on;
//   windows   the windows between a merge tile's splits whose keys are in order,
//             in no order, or have NaNs among them: every read inside the tile;
//   counts    the keys that a merge tile takes of each range, for tile starts
//             in order and crossing: never more than there are.
// Prints one line per check and ALL PASSED when every check holds.
#include "b2p_device/merge.cuh"
#include "b2p_device/pipe.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
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

// A position in an array of n keys (one more readable key after them when
// `spare`): a read outside is counted, and gives the first key.
struct Checked {
  const float *base;
  int at, n;
  long long *outside;
  Checked operator+(int k) const { return {base, at + k, n, outside}; }
  Checked operator-(int k) const { return {base, at - k, n, outside}; }
  Checked &operator+=(int k) { return at += k, *this; }
  Checked &operator-=(int k) { return at -= k, *this; }
  float operator[](int k) const {
    const bool in = at + k >= 0 && at + k < n;
    *outside += !in;
    return base[in ? at + k : 0];
  }
};

// The split search of merge_keys_kernel: keys of sa[0..na) before output d.
int tile_split(Checked sa, Checked sb, int d, int na, int nb) {
  int lo = std::max(0, d - nb);
  const int hi = std::min(d, na);
  Checked pa = sa + lo, pb = sb + (d - 1 - lo);
  for (int step = 2048; step > 0; step /= 2) {
    if (lo + step <= hi && !(pb[1 - step] < pa[step - 1])) {
      lo += step;
      pa += step;
      pb -= step;
    }
  }
  return lo;
}

// One staged tile of fp32 keys: every thread's split, and its window (i < ca:
// key i of a, else key ITEMS - i of b, whose first one may be the key after b's
// last).
void tile_windows(const std::vector<float> &a, const std::vector<float> &b, long long &outside, int &crossed) {
  using Net = b2p::MergeNet<float>;
  constexpr int ITEMS = Net::kItems, NT = Net::kThreads;
  const int na = (int)a.size(), nb = (int)b.size(), cnt = na + nb;
  std::vector<float> a1(a), b1(b);
  a1.push_back(0.f);
  b1.push_back(0.f);  // (the key after b's last)
  const Checked sa{a1.data(), 0, na, &outside}, sb{b1.data(), 0, nb, &outside};
  std::vector<int> lo(NT + 1, na);
  for (int t = 0; t < NT; ++t) lo[t] = tile_split(sa, sb, std::min(t * ITEMS, cnt), na, nb);
  for (int t = 0; t < NT; ++t) {
    const int d = std::min(t * ITEMS, cnt), ca = b2p::merge_window<ITEMS>(lo[t], lo[t + 1]);
    if (d + ITEMS > cnt) continue;
    crossed += ca != lo[t + 1] - lo[t];
    const Checked wa = sa + lo[t], wb{b1.data(), d - lo[t] + ITEMS, nb + 1, &outside};
    for (int i = 0; i <= ITEMS; ++i) (void)(i < ca ? wa + i : wb - i)[0];
  }
}

void windows() {
  std::mt19937 rng(1);
  const int tile = b2p::MergeNet<float>::kTile;
  for (int kind = 0; kind < 4; ++kind) {
    long long outside = 0;
    int crossed = 0;
    for (int rep = 0; rep < 60; ++rep) {
      const int cnt = rep % 3 ? tile : 1 + (int)(rng() % tile);
      const int na = rep % 5 == 0 ? 0 : rep % 5 == 1 ? cnt : (int)(rng() % (cnt + 1));
      std::vector<float> x(cnt);
      for (float &v : x) v = (float)(int)(rng() % 20001) - 10000.f;
      std::vector<float> a(x.begin(), x.begin() + na), b(x.begin() + na, x.end());
      if (kind != 1) {
        std::sort(a.begin(), a.end());
        std::sort(b.begin(), b.end());
      }
      if (kind >= 2)  // NaNs at the end (2) or anywhere (3)
        for (std::vector<float> *s : {&a, &b}) {
          const size_t m = s->size(), from = kind == 2 ? m - m / 7 : 0;
          for (size_t i = from; i < m; ++i)
            if (kind == 2 || rng() % 9 == 0) (*s)[i] = NAN;
        }
      tile_windows(a, b, outside, crossed);
    }
    static const char *name[4] = {"windows, keys in order", "windows, keys in no order", "windows, NaNs at the end",
                                  "windows, NaNs anywhere"};
    printf("(%d splits cross) ", crossed);
    check(outside == 0 && (kind == 0) == (crossed == 0), name[kind]);
  }
}

// Tile starts of random places: each within its range (as merge_path keeps
// it), the next tile's in order or not.
void counts() {
  std::mt19937 rng(2);
  bool inside = true, same = true;
  int crossing = 0;
  for (int rep = 0; rep < 200000; ++rep) {
    const long long nA = rng() % 5000, nB = rng() % 5000;
    if (nA + nB == 0) continue;
    const long long d0 = rng() % (nA + nB);
    const int cnt = (int)std::min<long long>(1 + rng() % 4096, nA + nB - d0);
    auto start = [&](long long d) {
      const long long lo = std::max(0ll, d - nB), hi = std::min(d, nA);
      return lo + (long long)(rng() % (hi - lo + 1));
    };
    const long long i0 = start(d0), i1 = start(d0 + cnt), j0 = d0 - i0, j1 = d0 + cnt - i1;
    const int na = b2p::merge_tile_count(i0, i1, nA, j0, nB, cnt);
    inside = inside && na >= 0 && na <= cnt && i0 + na <= nA && j0 + (cnt - na) <= nB;
    if (i1 >= i0 && j1 >= j0) same = same && na == i1 - i0;
    else ++crossing;
  }
  printf("(%d starts cross) ", crossing);
  check(inside && same && crossing > 0, "keys of a merge tile");
}

}  // namespace

int main() {
  carries();
  windows();
  counts();
  if (g_failed == 0) printf("ALL PASSED\n");
  return g_failed != 0;
}
