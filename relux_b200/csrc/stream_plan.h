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

// More items than this no sequence is cut into: the projection of the partial results keeps the columns of a row together.  Only the tuning knobs
// (more workers, shorter chunks) could ask for more.
constexpr int kMaxRowItems = 240;

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

// What a plan costs, in tiles of two pages (1.1 us at 32 heads, 1.3 at 128): its slowest worker's tiles and two for every item (start and
// write-out), 0.035 for every partial of the call and 0.02 for every one of the longest row.  Fit to forced plans of 49 batches of 1 to 64
// sequences at 32, 64 and 128 heads (one query token); with 0.08 for the longest row's, from when the partials of a row were added up by loads,
// 1 x 2600 tokens took 21.3 us instead of 21.0, with 32 heads 16.4 instead of 15.3.
// A call in which every sequence has one piece is 1.4 tiles cheaper than this says (its partials are written and read as one half).  Not counted:
// P starts from one maximum then, and the sum is rounded, so that such a call is up to 2.4 % further from float64 than the same one in pieces was
// when those were merged (16 x 300 2.33e-3 -> 2.39e-3; in pieces it is 1.65e-3 now), for 4 to 9 % of a step's time.
inline double plan_cost(double worst, int most_items, int items) { return worst + 0.02 * most_items + 0.035 * items; }

// The cheapest plan of a call: equal ranges of the sequences laid end to end, each counted as its pages and kStartUnits, for a worker
// that starts it has a second item to start and to write out; or every sequence cut by itself into pieces of 2 t pages, a worker each.
// Measured, ranges forced -> this, one build: 1 x 1300 tokens 23.3 -> 20.2 us, 3 x <= 1500 24.3 -> 21.7, 16 x 300 26.3 -> 23.3, 64 x 1000 46.3
// -> 39.4, 64 x 4096 93.2 -> 84, with 32 heads 1 x 1300 18.5 -> 15.1, 64 x 1000 34.5 -> 31.7; no difference beyond the runs' own at 16 x 2000
// (30.1), 20 x 8000 (64), 16 x <= 32768 and, with 32 heads, 40 x <= 2500 (31.0).
constexpr int kStartUnits = 4;   // pages, two tiles: what plan_cost counts for an item
struct StreamShape {
  int G, workers, items, start_units;
  bool by_item;
  int room;   // scratch for as many items serves the call on either side of the plans' border, and every later length of its sequences (build_stream)
};
// Length of the equal ranges that share `units` units of sequences, each with its kStartUnits.
RELUX_HD inline int range_units(int64_t units, int workers) {
  const int G = (int)((units + workers - 1) / workers + 1) / 2 * 2;
  return G > 2 * kStartUnits ? G : 2 * kStartUnits;
}
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
  const int longest2 = (longest + 1) / 2 * 2;
  r.G = std::max(range_units(units, workers), ((longest2 + kMaxRowItems - 2) / (kMaxRowItems - 1) + 1) / 2 * 2);   // a sequence may begin and end inside ranges
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
  r.room = std::max(r.items, live + r.workers - 1);
  if (live == 0 || live > workers) return r;
  double best = plan_cost(worst, most, r.items);
  auto items_of = [&](int t) {
    int items = 0;
    for (int n : pages) items += (n + 2 * t - 1) / (2 * t);
    return items;
  };
  int lo = (longest + 2 * kMaxRowItems - 1) / (2 * kMaxRowItems), hi = (longest + 1) / 2;   // the smallest t whose pieces find a worker each: one piece a sequence does
  while (lo < hi) {
    const int t = (lo + hi) / 2;
    if (items_of(t) <= workers) hi = t;
    else lo = t + 1;
  }
  for (int t = lo; t <= lo + 1; t++) {   // one more tile each may leave fewer partials
    const int items = items_of(t);
    const double cost = plan_cost(t + 2, (longest + 2 * t - 1) / (2 * t), items);
    r.room = std::max(r.room, live + items - 1);
    if (cost < best) {
      best = cost;
      r = StreamShape{2 * t, items, items, 0, true, r.room};
    }
  }
  return r;
}

}  // namespace relux
