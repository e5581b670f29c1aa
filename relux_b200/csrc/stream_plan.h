// How the persistent latent decode kernel's work is cut: the items of a sequence (host and device), and the plan of a call (host).
// Plain C++: no CUDA, so that it can be checked on its own.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define RELUX_HD __host__ __device__
#else
#define RELUX_HD
#endif

namespace relux {

// The items of a sequence of `pages` pages that begins at unit `at` of the stream: item c is its pages [begin(c), end(c)), and belongs to
// worker first + c, or (by_item) to a worker of its own.  What the host counts and the device builds from.
struct SeqCut {
  int by_item, G, at0, pages, units, first, n;
  RELUX_HD SeqCut(int by_item_, int G_, int start_units, int at, int pages_) : by_item(by_item_), G(G_), pages(pages_) {
    // with units of fixed cost, all in twos: ranges then begin on whole tiles of their sequences
    units = pages <= 0 ? 0 : by_item ? pages : start_units ? start_units + (pages + 1) / 2 * 2 : pages;
    at0 = at + (by_item ? 0 : start_units);
    first = by_item ? 0 : at0 / G;
    n = pages <= 0 ? 0 : by_item ? (pages + G - 1) / G : (at0 + pages - 1) / G - first + 1;
  }
  RELUX_HD int begin(int c) const {
    const int b = by_item ? c * G : (first + c) * G - at0;
    return b > 0 ? b : 0;
  }
  RELUX_HD int end(int c) const {
    const int e = by_item ? (c + 1) * G : (first + c + 1) * G - at0;
    return e < pages ? e : pages;
  }
  // of a range's items, is this the one with its first page?  (`at`: as above; a range that begins before the sequence holds pages of
  // the one before it)
  RELUX_HD bool leads(int c, int at) const { return (first + c) * G >= at; }
};

// What a plan costs, in tiles of two pages (about 2 us): its slowest worker's tiles and two for every item (start and write-out), 0.08 for
// every partial that a row of the merge adds up, and 0.035 for every partial of the call.  From steps of 1 to 30 short sequences with
// ranges of one and of two tiles (1 x 1300 tokens 19.9 against 21.5 us, 1 x 2600 21.5 and 21.4, 1 x 6000 26.8 and 24.0, 4 x 1200 24.0 and
// 23.3, 25 x 200 27.4 and 28.3).
inline double plan_cost(double worst, int most_items, int items) { return worst + 0.08 * most_items + 0.035 * items; }

// The cheapest plan of a call: equal ranges of the sequences laid end to end, each counted as its pages and kStartUnits, for a worker
// that starts it has a second item to start and to write out; or every sequence cut by itself into pieces of 2 t pages, a worker each.
// Measured, ranges of pages alone -> this, one build: in pieces, 1 x 1300 tokens 21.8 -> 20.2 us, 3 x <= 1500 26.9 -> 22.3, 16 x 300 28.6 ->
// 25.1, 64 x 300 41.0 -> 40.5, 40 x <= 2500 51.1 -> 45.1, 64 x 4096 93.8 -> 89.4, with 32 heads 64 x 500 42.5 -> 35.7; in ranges, 20 x 16000
// 97.3 -> 95.5, and no difference beyond the runs' own at 16 x <= 32768 (97) and 64 x 32768 (565-585).  The fit is to one query token and
// 128 heads; elsewhere: verify of 3 x <= 1500 with 4 tokens 39.1 -> 34.0, 16 x 300 with 2 43.2 -> 37.9, 32 x 1000 with 4 87.6 -> 79.3, 30 x
// <= 800 with 3 and 32 heads 52.1 -> 46.2, the other way 64 x 300 with 2 and 32 heads 48.5 -> 50.1.
constexpr int kStartUnits = 4;   // pages, two tiles: what plan_cost counts for an item
struct StreamShape {
  int G, workers, items, start_units;
  bool by_item;
  int room;   // items of the larger of the plans compared: scratch for as many serves the call on either side of their border
};
inline StreamShape cheapest_plan(const std::vector<int>& pages, int workers) {
  int longest = 0, live = 0;
  int64_t units = 0;
  for (int n : pages) {
    longest = std::max(longest, n);
    live += n > 0;
    units += SeqCut(0, 1, kStartUnits, 0, n).units;
  }
  StreamShape r{};
  r.start_units = kStartUnits;
  r.G = std::max((int)((units + workers - 1) / workers + 1) / 2 * 2, 2 * kStartUnits);
  r.workers = std::max(1, (int)((units + r.G - 1) / r.G));
  int at = 0, most = 0, of_worker = -1;
  double worst = 0, here = 0;   // of the ranges, walked as the workers walk them
  for (int n : pages) {
    const SeqCut cut(0, r.G, kStartUnits, at, n);
    for (int c = 0; c < cut.n; c++) {
      if (cut.first + c != of_worker) here = 0;
      of_worker = cut.first + c;
      here += (cut.end(c) - cut.begin(c) + 1) / 2 + 2;
      worst = std::max(worst, here);
    }
    most = std::max(most, cut.n);
    r.items += cut.n;
    at += cut.units;
  }
  r.room = r.items;
  if (live == 0 || live > workers) return r;
  double best = plan_cost(worst, most, r.items);
  auto items_of = [&](int t) {
    int items = 0;
    for (int n : pages) items += (n + 2 * t - 1) / (2 * t);
    return items;
  };
  int lo = 1, hi = (longest + 1) / 2;   // the smallest t whose pieces find a worker each: one piece a sequence does
  while (lo < hi) {
    const int t = (lo + hi) / 2;
    if (items_of(t) <= workers) hi = t;
    else lo = t + 1;
  }
  for (int t = lo; t <= lo + 1; t++) {   // one more tile each may leave fewer partials
    const int items = items_of(t);
    const double cost = plan_cost(t + 2, (longest + 2 * t - 1) / (2 * t), items);
    r.room = std::max(r.room, items);
    if (cost < best) {
      best = cost;
      r = StreamShape{2 * t, items, items, 0, true, r.room};
    }
  }
  return r;
}

}  // namespace relux
