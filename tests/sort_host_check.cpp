// Host check of the counting sort's places: the sort is followed block by block with keys that change between the blocks'
// reads (a caller's buffer that was not ordered before the call). Whenever a place stays unwritten the sum of the places'
// marks has to tell; with unchanged keys it is 0, and the result is the stable sort.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "../cheese_b200/csrc/cz_place.h"

int main() {
  std::mt19937_64 rng(5);
  int errors = 0, raised = 0, torn = 0;
  for (int it = 0; it < 4000; it++) {
    const unsigned n = 2 + rng() % 200, range = 1 + rng() % 8, changes = it % 4;
    std::vector<uint64_t> key(n);
    for (auto &k : key) k = rng() % range;
    const std::vector<uint64_t> first = key;
    std::vector<unsigned> from(n, ~0u);
    uint64_t sum = 0;
    for (unsigned i0 = 0; i0 < n; i0 += 32) {            // a block's pairs: their keys read, then all keys
      const unsigned b = std::min(32u, n - i0);
      std::vector<uint64_t> mine(key.begin() + i0, key.begin() + i0 + b);
      for (unsigned c = 0; c < changes; c++) key[rng() % n] = rng() % range;
      for (unsigned l = 0; l < b; l++) {
        unsigned pos = 0;
        for (unsigned x = 0; x < n; x++) {
          const bool before = x / 32 < i0 / 32, behind = x / 32 > i0 / 32;
          pos += before ? key[x] <= mine[l] : behind ? key[x] < mine[l] : key[x] < mine[l] || (key[x] == mine[l] && x < i0 + l);
        }
        if (pos < n) from[pos] = i0 + l;
        sum += cz::place_mark(pos) - cz::place_mark(i0 + l);
      }
    }
    bool lost = false;
    for (unsigned i = 0; i < n; i++) lost |= from[i] == ~0u;
    if (lost != (sum != 0)) errors++;
    torn += lost;
    raised += sum != 0;
    if (!changes) {
      std::vector<unsigned> order(n);
      for (unsigned i = 0; i < n; i++) order[i] = i;
      std::stable_sort(order.begin(), order.end(), [&](unsigned a, unsigned b) { return first[a] < first[b]; });
      if (sum || order != from) errors++;
    }
  }
  if (!torn || !raised) errors++;                        // the changes do tear sorts
  std::printf("errors: %d\n", errors);
  return errors != 0;
}
