// The plan of the persistent latent decode kernel and the items it is cut into, walked as the device builder walks them.
// With arguments (workers, then pages of every sequence): prints the plan.  Without: random calls, and random lengths that a plan's launch finds
// other than those it was made for, with the up-projection's columns for both.
#include <cstdio>
#include <cstdlib>
#include <ctime>
#include <random>

#include "stream_plan.h"
#include "vup_plan.h"

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
    CHECK(cut.n <= kMaxRowItems);
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

// The pieces of every sequence as the device cuts them (build_stream) for a plan made for other lengths; empty where it has no room for them.
static std::vector<int32_t> device_first(const StreamShape& s, const std::vector<int>& pages) {
  int by_item = s.by_item, G = s.G, start_units = s.start_units;
  for (int pass = 0; pass < 2; pass++) {
    std::vector<int32_t> first(1, 0);
    int unit = 0;
    for (int n : pages) {
      const SeqCut cut(by_item, G, start_units, unit, n);
      unit += cut.units;
      first.push_back(first.back() + cut.n);
    }
    if ((by_item ? first.back() : (unit + G - 1) / G) <= s.workers && first.back() <= s.room) return first;
    int64_t units = 0;
    for (int n : pages) units += SeqCut(0, 1, kStartUnits, 0, n).units;
    by_item = 0, start_units = kStartUnits, G = range_units(units, s.workers);
  }
  return {};
}

static bool check_columns(const std::vector<int>& pages, int S, int heads, const StreamShape& s, const std::vector<int32_t>& planned, const std::vector<int32_t>& found,
                          bool loose, int halves) {
  const int workers = s.workers, rows = (int)pages.size() * S, dC = 512;
  const VupShape v = vup_shape(planned, rows, S, 148 / heads, halves, dC, loose ? workers : 0);
  CHECK(v.fits());
  const int unit = (v.blocks > 1 ? 32 : 16) / halves;
  CHECK(v.blocks >= 1 && v.n_block % unit == 0 && halves * v.n_block <= 256 && v.blocks * halves * v.n_block <= v.tmem_cols);
  CHECK(v.tmem_cols >= 32 && v.tmem_cols <= 512 && (v.tmem_cols & (v.tmem_cols - 1)) == 0);
  CHECK(v.n_stages >= 1 && v.n_stages <= kVupMaxStages && v.n_stages * v.n_kb * halves * v.n_block * 128 <= kVupRing);
  CHECK(v.groups >= 1 && (v.groups - 1) * v.rows_each < rows && v.groups * v.rows_each >= rows);
  for (int g = 0; g < v.groups; g++) {
    const int r = g * v.rows_each, end = std::min(rows, r + v.rows_each);
    CHECK(vup_col(found, S, end) - vup_col(found, S, r) <= std::min(v.most, v.blocks * v.n_block));
  }
  return true;
}

// Chunks of a graph's decode call on the CUDA-core kernel, dealt to the sequences anew: as many as were planned at most, wherever they lie.
static bool check_chunks(std::mt19937& rng, int n, int S, int heads) {
  const int span = rng() % 2 ? 6 : 40;
  std::vector<int32_t> planned(1, 0), found(1, 0);
  for (int i = 0; i < n; i++) planned.push_back(planned.back() + 1 + (int)(rng() % span));
  for (int i = 0; i < n; i++) {
    const int left = planned.back() - found.back(), most = std::min(left, kMaxRowItems);
    found.push_back(found.back() + (i == n / 2 || rng() % 8 == 0 ? most : (int)(rng() % (std::min(most, span) + 1))));
  }
  const int rows = n * S;
  const VupShape v = vup_shape(planned, rows, S, 148 / heads, 2, 512, kVupAnyChunks);
  int widest = 0;
  for (const std::vector<int32_t>* first : {&planned, &found})
    for (int r = 0; r < rows; r += v.rows_each) widest = std::max(widest, vup_col(*first, S, std::min(rows, r + v.rows_each)) - vup_col(*first, S, r));
  if (v.fits() && widest <= std::min({v.most, v.blocks * v.n_block, kVupMaxCols})) return true;
  printf("chunks: %d rows in groups of %d, %d columns of %d x %d\n", rows, v.rows_each, widest, v.blocks, v.n_block);
  return false;
}

static bool check_found(std::mt19937& rng, const std::vector<int>& pages, int S, int heads, int resident) {
  const int workers = S > 8 ? std::min(resident, std::max(1, (2 * resident + S - 1) / S)) : std::max(1, resident / S);
  const StreamShape s = cheapest_plan(pages, workers);
  const std::vector<int32_t> planned = device_first(s, pages);
  CHECK((int)planned.size() == (int)pages.size() + 1 && planned.back() == s.items);   // the host's own lengths are served as planned
  if (!check_columns(pages, S, heads, s, planned, planned, false, rng() % 2 ? 1 : 2)) return false;
  std::vector<int> now = pages;
  const int how = (int)(rng() % 4);
  for (int& n : now) n = how == 0 ? n + (int)(rng() % 2) : how == 1 ? n + (int)(rng() % 40) : how == 2 ? (int)(rng() % 400) : rng() % 5 ? 0 : (int)(rng() % 2000);
  const std::vector<int32_t> found = device_first(s, now);
  CHECK(found.size() == pages.size() + 1);
  return check_columns(pages, S, heads, s, planned, found, true, 2);
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
  for (int t = 0; t < 20000; t++) {   // of the tuning knob: more workers than a row may have pieces
    std::vector<int> pages(1 + (int)(rng() % (rng() % 2 ? 2 : 30)));
    for (int& p : pages) p = 1 + (int)(rng() % (rng() % 2 ? 16384 : 300));
    const int workers = 1 + (int)(rng() % 4096);
    if (!check(pages, workers)) return 1;
    const StreamShape s = cheapest_plan(pages, workers);
    const std::vector<int32_t> planned = device_first(s, pages);
    if (!check_columns(pages, 1, 16, s, planned, planned, t & 1, 2)) return 1;
  }
  const int heads[] = {16, 32, 40, 64, 75, 128};
  for (int t = 0; t < 60000; t++) {
    const int S = 1 + (int)(rng() % (rng() % 4 ? 4 : 40)), n = 1 + (int)(rng() % (rng() % 2 ? 8 : 160)), span = spans[rng() % 6];
    std::vector<int> pages(n);
    for (int& p : pages) p = 1 + (int)(rng() % span);
    if (!check_found(rng, pages, S, heads[rng() % 6], rng() % 4 ? 74 : 1 + (int)(rng() % 100))) return 1;
  }
  for (int t = 0; t < 20000; t++)
    if (!check_chunks(rng, 1 + (int)(rng() % (rng() % 2 ? 8 : 60)), 1 + (int)(rng() % 4), t % 3 ? 8 : 16)) return 1;
  std::vector<int32_t> first(1, 0);   // 131072 rows of one to 60 pieces: groups tried one number after another took 2.6 s
  for (int i = 0; i < 64; i++) first.push_back(first.back() + 1 + (int)(rng() % 60));
  const clock_t from = clock();
  const VupShape many = vup_shape(first, 64 * 2048, 2048, 1, 2, 512, 0);
  if (!many.fits() || clock() - from > CLOCKS_PER_SEC / 4) return printf("many rows: %d groups, %.3f s\n", many.groups, (double)(clock() - from) / CLOCKS_PER_SEC), 1;
  if (pieces < 1000 || ranges < 1000) return printf("%d pieces, %d ranges\n", pieces, ranges), 1;
  puts("ok");
  return 0;
}
