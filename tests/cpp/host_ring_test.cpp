// Replays calls of random sizes through the places of the page-locked input block: the bytes that a call writes must belong to no piece
// of a call whose kernel a wait has not covered.  A wait covers the calls before the one that waits.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "host_ring.h"

struct Piece {
  size_t lo, hi;
  int call;
};

static int replay(uint32_t seed, size_t size, const std::vector<std::pair<size_t, size_t>>& sizes, int calls) {
  std::mt19937 rng(seed);
  relux::HostRing ring{size};
  std::vector<Piece> open;   // pieces whose kernel may still be waiting to read them
  int waits = 0;
  for (int call = 0; call < calls; call++) {
    const auto& s = sizes[rng() % sizes.size()];
    const size_t bytes[2] = {s.first, s.second};
    const int n = bytes[1] ? 2 : 1;
    size_t at[2];
    auto wait = [&] {
      waits++;
      open.erase(std::remove_if(open.begin(), open.end(), [&](const Piece& o) { return o.call < call; }), open.end());
      return true;
    };
    if (!ring.take(bytes, n, at, wait)) return printf("refused\n"), -1;
    for (int i = 0; i < n; i++) {
      if (at[i] % 256 || at[i] + bytes[i] > size) return printf("call %d: place %zu + %zu\n", call, at[i], bytes[i]), -1;
      for (const Piece& o : open)
        if (at[i] < o.hi && o.lo < at[i] + bytes[i]) return printf("call %d overwrites call %d at %zu\n", call, o.call, at[i]), -1;
      open.push_back({at[i], at[i] + bytes[i], call});
    }
    if (rng() % 97 == 0) {   // a call that waits for its results
      open.clear();
      ring.restart();
    }
  }
  return waits;
}

int main() {
  const size_t K = 1024, size = 1024 * K;
  std::vector<std::vector<std::pair<size_t, size_t>>> kinds = {
      {{4 * K, 4 * K}}, {{12 * K, 12 * K}}, {{20 * K, 20 * K}}, {{16 * K, 2 * K}}, {{9 * K, 9 * 128}}, {{32 * K, 0}, {12 * K, 12 * K}}};
  std::vector<std::pair<size_t, size_t>> any;
  std::mt19937 rng(1);
  for (int i = 0; i < 200; i++) any.push_back({1 + rng() % (32 * K), rng() % (32 * K)});
  kinds.push_back(any);
  for (size_t k = 0; k < kinds.size(); k++)
    for (uint32_t seed = 0; seed < 50; seed++) {
      const int waits = replay(seed, size, kinds[k], 3000);
      if (waits < 1) return printf("sizes %zu, seed %u: %d\n", k, seed, waits), 1;
    }
  // more than the block holds is refused without a wait; a wait that fails takes nothing
  relux::HostRing ring{K};
  const size_t big[2] = {K, 1}, half[1] = {600};
  size_t at[2];
  bool waited = false;
  if (ring.take(big, 2, at, [&] { waited = true; return true; }) || waited) return 2;
  if (!ring.take(half, 1, at, [&] { return false; }) || ring.take(half, 1, at, [&] { return false; }) || ring.used != 768) return 3;
  puts("ok");
  return 0;
}
