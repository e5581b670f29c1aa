// The plan of the persistent latent decode kernel and the items it is cut into, walked as the device builder walks them.
// With arguments (workers, then pages of every sequence): prints the plan.  Without: random calls.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "stream_plan.h"

using namespace relux;

#define CHECK(c) do { if (!(c)) { printf("line %d: %s (workers %d, %zu sequences, pieces %d, G %d)\n", __LINE__, #c, workers, pages.size(), (int)s.by_item, s.G); return false; } } while (0)

static bool check(const std::vector<int>& pages, int workers) {
  const StreamShape s = cheapest_plan(pages, workers);
  struct Item { int seq, begin, end, worker; };
  std::vector<Item> items;
  std::vector<int> worker_first(s.workers + 1, -1), chunk_off;
  int unit = 0, live = 0;
  for (int i = 0; i < (int)pages.size(); i++) {
    const SeqCut cut(s.by_item, s.G, s.start_units, unit, pages[i]);
    chunk_off.push_back((int)items.size());
    live += pages[i] > 0;
    int at = 0;
    for (int c = 0; c < cut.n; c++) {
      const int k = (int)items.size(), w = s.by_item ? k : cut.first + c;
      CHECK(cut.begin(c) == at && cut.end(c) > at);        // every page once, in order
      CHECK((cut.begin(c) & 1) == 0);                      // whole tiles
      at = cut.end(c);
      CHECK(w < s.workers);
      if (s.by_item || cut.leads(c, unit)) {
        CHECK(worker_first[w] == -1);
        worker_first[w] = k;
      }
      items.push_back({i, cut.begin(c), cut.end(c), w});
    }
    CHECK(at == pages[i]);
    unit += cut.units;
  }
  CHECK((int)items.size() == s.items);
  for (int w = s.by_item ? s.items : (unit + s.G - 1) / s.G; w <= s.workers; w++) worker_first[w] = s.items;   // as the builder pads
  CHECK(s.workers >= 1 && s.workers <= std::max(1, workers));
  CHECK(s.G > 0 && s.G % 2 == 0);
  for (int w = 0; w < s.workers; w++) {
    CHECK(worker_first[w] >= 0 && worker_first[w] <= worker_first[w + 1]);
    int units = 0;
    for (int k = worker_first[w]; k < worker_first[w + 1]; k++) {
      CHECK(items[k].worker == w);
      units += items[k].end - items[k].begin;
    }
    CHECK(units <= s.G);
    if (s.by_item) CHECK(worker_first[w + 1] == worker_first[w] + 1);
  }
  CHECK(worker_first[s.workers] == s.items && (live == 0) == (s.items == 0));
  CHECK(s.room >= s.items && s.room <= std::max(1, workers) + live);   // what scratch is sized for
  return true;
}

int main(int argc, char** argv) {
  if (argc > 1) {
    std::vector<int> pages;
    for (int i = 2; i < argc; i++) pages.push_back(atoi(argv[i]));
    const StreamShape s = cheapest_plan(pages, atoi(argv[1]));
    printf("%s %d %d %d %d\n", s.by_item ? "pieces" : "ranges", s.G, s.workers, s.items, s.room);
    return 0;
  }
  std::mt19937 rng(3);
  int pieces = 0, ranges = 0;
  const int spans[] = {2, 5, 20, 80, 513, 2000};
  for (int t = 0; t < 60000; t++) {
    const int workers = 1 + (int)(rng() % (rng() % 3 ? 74 : 9)), n = 1 + (int)(rng() % (rng() % 2 ? 8 : 130));
    const int span = spans[rng() % 6];
    std::vector<int> pages(n);
    for (int& p : pages) p = (int)(rng() % span) * (rng() % 8 != 0) + (rng() % 4 != 0);   // some of them empty
    if (!check(pages, workers)) return 1;
    (cheapest_plan(pages, workers).by_item ? pieces : ranges)++;
  }
  if (pieces < 1000 || ranges < 1000) return printf("%d pieces, %d ranges\n", pieces, ranges), 1;
  puts("ok");
  return 0;
}
