// Host-side check of the look-back records of gpz_b200/csrc/gpz_kernels.cuh:
// every field lies in one 64-bit word, which one atomic OR sets and one 64-bit
// element of a load returns, so a reader that meets every word at another time
// still sees each field either unset or whole.  Records are filled in random
// order; after every pair of steps each word is read as of a random earlier
// moment.  Compiled with nvcc, runs on the CPU.
#include <cstdio>
#include <cstdint>
#include <algorithm>
#include <vector>
#include "gpz_kernels.cuh"

using namespace gpzb;

static uint64_t s = 0x2545F4914F6CDD1Dull;
static uint32_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (uint32_t)(s >> 16); }

int main() {
  long bad = 0, checks = 0;
  // fields do not overlap each other or the prefix
  unsigned long long used[4] = {0, 0, 0, kLookKnown | kLookPrefix};
  for (uint32_t i = 0; i < (uint32_t)kLookGroup; ++i) {
    const unsigned long long m = 4095ull << look_shift(i);
    bad += look_shift(i) + 12u > 64u || look_word(i) > 3u || (used[look_word(i)] & m) != 0ull;
    used[look_word(i)] |= m;
  }
  for (int it = 0; it < 20000; ++it) {
    uint32_t size[kLookGroup];
    for (auto &v : size) v = rnd() % 4 ? 1u + rnd() % 4095u : 4095u;
    const unsigned long long prefix = (((unsigned long long)rnd() << 32) | rnd()) & kLookPrefix;
    int order[kLookGroup + 1];
    for (int i = 0; i <= kLookGroup; ++i) order[i] = i;
    for (int i = kLookGroup; i > 0; --i) std::swap(order[i], order[rnd() % (uint32_t)(i + 1)]);
    std::vector<unsigned long long> hist[4];
    for (auto &h : hist) h.push_back(0ull);
    for (int k = 0; k <= kLookGroup; ++k) {
      const int i = order[k];
      for (int w = 0; w < 4; ++w) hist[w].push_back(hist[w].back());
      if (i < kLookGroup) hist[look_word(i)].back() |= (unsigned long long)size[i] << look_shift(i);
      else hist[3].back() |= kLookKnown | prefix;
      unsigned long long r[4];
      for (int w = 0; w < 4; ++w) r[w] = hist[w][rnd() % hist[w].size()];
      for (uint32_t c = 0; c < (uint32_t)kLookGroup; ++c) {
        const uint32_t v = look_size(r, c);
        bad += v != 0u && v != size[c];
      }
      bad += (r[3] & kLookKnown) != 0ull ? (r[3] & kLookPrefix) != prefix : (r[3] & kLookPrefix) != 0ull;
      ++checks;
    }
    const unsigned long long end[4] = {hist[0].back(), hist[1].back(), hist[2].back(), hist[3].back()};
    for (uint32_t c = 0; c < (uint32_t)kLookGroup; ++c) bad += look_size(end, c) != size[c];
  }
  printf("checks=%ld bad=%ld\n", checks, bad);
  return bad != 0;
}
