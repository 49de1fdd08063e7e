// Host-side check of the ranking of gpz_b200/csrc/gpz_encode.cuh: rank_buckets
// emulated thread by thread on the CPU with the kernel's own window, exchange
// steps and limits -- shared atomics in an arbitrary arrival order, starts
// relative to the quarter of the buckets a warp scans, placement, crowded
// buckets sorted on their own, four warps' windows of 288 positions, nine a
// lane -- and compared with a plain sort of (block id, rank).  That ceil(n / 2)
// rounds order every bucket of n points at every offset within a lane is shown
// over all 0-1 inputs.  The CTA's network (cta_sort) is checked position by
// position on permutations and 0-1 inputs.  Compiled with nvcc, runs on the CPU.
#include <algorithm>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <cmath>
#include <vector>
#include "gpz_encode.cuh"

using namespace gpzb;

static uint64_t s = 0x2545F4914F6CDD1Dull;
static uint32_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return (uint32_t)(s >> 11); }
static constexpr uint32_t FULL = 0xFFFFFFFFu;

// `rounds` rounds over the lanes of one window; v: 32 * kEncOrd values.
template <bool kNarrow>
static void order_window(uint32_t *v, const uint32_t *bucket, uint32_t rounds) {
  static uint32_t k[32][kEncOrd], cut[32][kEncOrd];
  for (int l = 0; l < 32; ++l)
    for (int j = 0; j < kEncOrd; ++j) {
      const int p = kEncOrd * l + j;
      k[l][j] = v[p];
      cut[l][j] = p + 1 < 32 * kEncOrd && bucket[p] == bucket[p + 1] ? 0u : FULL;
    }
  for (uint32_t it = 0; it < rounds; ++it)
    for (int h = 0; h < 2; ++h) {
      for (int l = 0; l < 32; ++l) order_pairs<kNarrow>(k[l], cut[l], h);
      uint32_t nx[32], pv[32];
      for (int l = 0; l < 32; ++l) {
        nx[l] = k[std::min(l + 1, 31)][0];
        pv[l] = k[std::max(l - 1, 0)][kEncOrd - 1];
      }
      for (int l = 0; l < 32; ++l)
        order_across<kNarrow>(k[l], cut[l], nx[l], pv[l], l == 0 ? FULL : cut[l - 1][kEncOrd - 1], l);
    }
  for (int l = 0; l < 32; ++l)
    for (int j = 0; j < kEncOrd; ++j) v[kEncOrd * l + j] = k[l][j];
}

// All 0-1 inputs of buckets of n < kEncSmall points at the nine offsets; the
// positions around belong to other buckets.
static long zero_one(long &checks) {
  long bad = 0;
  for (int n = 1; n < kEncSmall; ++n)
    for (int off = 0; off < kEncOrd; ++off)
      for (uint32_t in = 0; in < (1u << n); ++in) {
        // four lanes are enough (off + n <= 8 + 15): the other 28 rest
        static uint32_t k[4][kEncOrd], w[4][kEncOrd], cut[4][kEncOrd];
        const int first = kEncOrd + off;
        for (int p = 0; p < 4 * kEncOrd; ++p) {
          const bool inside = p >= first && p < first + n;
          k[p / kEncOrd][p % kEncOrd] = inside ? 1u + ((in >> (p - first)) & 1u) : (p < first ? 0u : 3u);
          w[p / kEncOrd][p % kEncOrd] = inside ? 1u + ((in >> (p - first)) & 1u) : (uint32_t)(p * 2654435761u);
          cut[p / kEncOrd][p % kEncOrd] = inside && p + 1 < first + n ? 0u : FULL;
        }
        for (int it = 0; it < (n + 1) / 2; ++it)
          for (int h = 0; h < 2; ++h) {
            uint32_t a[4], b[4], c[4], d[4];
            for (int l = 0; l < 4; ++l) {
              order_pairs<true>(k[l], k[l], h);
              order_pairs<false>(w[l], cut[l], h);
            }
            for (int l = 0; l < 4; ++l) {
              a[l] = k[std::min(l + 1, 3)][0]; b[l] = k[std::max(l - 1, 0)][kEncOrd - 1];
              c[l] = w[std::min(l + 1, 3)][0]; d[l] = w[std::max(l - 1, 0)][kEncOrd - 1];
            }
            for (int l = 0; l < 4; ++l) {
              order_across<true>(k[l], k[l], a[l], b[l], 0u, l == 3 ? 31 : l);
              order_across<false>(w[l], cut[l], c[l], d[l], l == 0 ? FULL : cut[l - 1][kEncOrd - 1], l == 3 ? 31 : l);
            }
          }
        const int zeros = n - __builtin_popcount(in);
        for (int p = 0; p < 4 * kEncOrd; ++p) {
          const bool inside = p >= first && p < first + n;
          const uint32_t x = k[p / kEncOrd][p % kEncOrd], y = w[p / kEncOrd][p % kEncOrd];
          const uint32_t want = 1u + (p - first >= zeros);
          bad += inside ? x != want || y != want : x != (p < first ? 0u : 3u) || y != (uint32_t)(p * 2654435761u);
        }
        ++checks;
      }
  return bad;
}

// scale of rank_buckets with the quotient off by `ulp`s
static uint32_t scale_of(uint32_t bound, int ulp) {
  float q = 4.39804e12f / ((float)bound + 1.0f);
  for (int i = 0; i < std::abs(ulp); ++i) q = std::nextafterf(q, ulp > 0 ? INFINITY : 0.0f);
  return q >= 4294967296.0f ? FULL : (uint32_t)q;
}

struct Out {
  bool declined = false;
  uint32_t id[kChunk], r[kChunk];
};

// ids by rank
static Out emulate(const std::vector<uint32_t> &ids, uint32_t bound) {
  Out o;
  const bool narrow = bound < (1u << 22);
  uint32_t low = 0;
  if (!narrow) low = 22u - (uint32_t)__builtin_clz(bound);
  const uint32_t scale = narrow ? scale_of(bound, (int)(rnd() % 5) - 2) : 0u;
  std::vector<uint32_t> b(kChunk), slot(kChunk), cnt(kEncBuckets, 0), order(kChunk);
  for (int i = 0; i < kChunk; ++i) order[i] = i;
  for (int i = kChunk - 1; i > 0; --i) std::swap(order[i], order[rnd() % (uint32_t)(i + 1)]);
  for (uint32_t r : order) {
    b[r] = narrow ? (uint32_t)(((uint64_t)ids[r] * scale) >> 32) : ids[r] >> low;
    if (b[r] >= (uint32_t)kEncBuckets) { o.declined = true; o.id[0] = FULL; return o; }  // out of range: never
    slot[r] = cnt[b[r]]++;
  }
  uint32_t biggest = 0, crowded = 0, largest = 0;
  for (uint32_t n : cnt) {
    biggest = std::max(biggest, n);
    if (n >= (uint32_t)kEncSmall) crowded += n;
    else largest = std::max(largest, n);
  }
  if (biggest > (uint32_t)kEncCrowd || crowded > (uint32_t)kEncCrowdPoints) {
    o.declined = true;
    return o;
  }
  // starts within the warp's quarter, then the quarter's own
  std::vector<uint32_t> start(kEncBuckets);
  uint32_t quarter[kEncWarps + 1] = {0};
  for (int w = 0; w < kEncWarps; ++w) {
    uint32_t sum = 0;
    for (int i = 0; i < kEncBuckets / kEncWarps; ++i) {
      start[w * (kEncBuckets / kEncWarps) + i] = sum;
      sum += cnt[w * (kEncBuckets / kEncWarps) + i];
    }
    quarter[w + 1] = quarter[w] + sum;
  }
  std::vector<uint32_t> S(kChunk, 0), B(kChunk, 0), H(kChunk, 0), R(kChunk, 0);
  for (int r = 0; r < kChunk; ++r) {
    const uint32_t pos = start[b[r]] + quarter[b[r] / (kEncBuckets / kEncWarps)] + slot[r];
    S[pos] = ((narrow ? ids[r] : ids[r] & ((1u << low) - 1u)) << 10) + (uint32_t)r;
    B[pos] = b[r];
  }
  int entries = 0;
  for (int k = 0; k < kEncBuckets; ++k)
    if (cnt[k] >= (uint32_t)kEncSmall) {
      const uint32_t p = start[k] + quarter[k / (kEncBuckets / kEncWarps)];
      std::sort(S.begin() + p, S.begin() + p + cnt[k]);
      ++entries;
    }
  if (entries > kEncCrowdPoints / kEncSmall) { o.declined = true; o.id[0] = FULL; return o; }  // list too short: never
  for (int w = 0; w < kEncWarps; ++w) {
    const uint32_t w0 = ord_window(w);
    std::vector<uint32_t> v(S.begin() + w0, S.begin() + w0 + 32 * kEncOrd), bk(B.begin() + w0, B.begin() + w0 + 32 * kEncOrd);
    if (narrow) order_window<true>(v.data(), bk.data(), (largest + 1u) >> 1);
    else order_window<false>(v.data(), bk.data(), (largest + 1u) >> 1);
    for (uint32_t i = 0; i < 32u * kEncOrd; ++i)
      if (w0 + i - 256u * w < 256u) {
        H[w0 + i] = narrow ? v[i] >> 10 : (bk[i] << low) | (v[i] >> 10);
        R[w0 + i] = v[i] & 1023u;
      }
  }
  std::copy(H.begin(), H.end(), o.id);
  std::copy(R.begin(), R.end(), o.r);
  return o;
}

// cta_sort position by position: warps sort 256, then the exchanges i with
// i ^ 511, i ^ 1023 (mirrored) and i ^ 256, each followed by i ^ j within the
// warp; the smaller value always goes to the lower position.
static void network(std::vector<uint32_t> &v) {
  auto pair = [&](uint32_t mask) {
    for (uint32_t i = 0; i < (uint32_t)kChunk; ++i)
      if (i < (i ^ mask) && v[i] > v[i ^ mask]) std::swap(v[i], v[i ^ mask]);
  };
  for (uint32_t k = 2; k <= 256; k <<= 1) {
    pair(k - 1);
    for (uint32_t j = k >> 2; j > 0; j >>= 1) pair(j);
  }
  pair(511);
  for (uint32_t j = 128; j > 0; j >>= 1) pair(j);
  pair(1023);
  pair(256);
  for (uint32_t j = 128; j > 0; j >>= 1) pair(j);
}

int main() {
  long checks = 0, declined = 0;
  long bad = zero_one(checks);
  // every bucket in range, ids in order, whatever the quotient's rounding
  for (uint32_t bound = kEncOnePass; bound < (1u << 22); bound += bound < 5000u ? 1u : 1u + rnd() % 997u)
    for (int ulp = -2; ulp <= 2; ++ulp) {
      bad += (((uint64_t)bound * scale_of(bound, ulp)) >> 32) >= (uint64_t)kEncBuckets;
      ++checks;
    }
  for (int it = 0; it < 6000; ++it) {
    std::vector<uint32_t> ids(kChunk);
    const int kind = it % 6;
    const uint32_t edges[] = {512, 513, 1022, 1023, 1024, 1025, 2047, 2048, (1u << 22) - 1, 1u << 22, (1u << 22) + 1, 0x7FFFFFFFu};
    const uint32_t bound = it % 3 ? edges[rnd() % 12] : 512u + rnd() % (1u << (10 + rnd() % 21));
    for (auto &v : ids) {
      v = (uint32_t)((((uint64_t)rnd() << 21) ^ rnd()) % ((uint64_t)bound + 1));
      if (kind == 1 && rnd() % 4 == 0) v = bound / 3 + rnd() % 5 % (bound - bound / 3);  // a crowd of about 256
      if (kind == 2 && rnd() % 3 == 0) v = (rnd() % 20) * (bound / 20);                  // twenty small ones
      if (kind == 3 && rnd() % 8 == 0) v = bound / 2;                                    // one of about 128
      if (kind == 4 && rnd() % 2 == 0) v = (rnd() % 34) * (bound / 34);                  // near the second limit
    }
    ids[rnd() % kChunk] = bound;
    const Out o = emulate(ids, bound);
    if (o.declined) {
      bad += o.id[0] == FULL;
      ++declined;
    } else {
      std::vector<uint64_t> ref(kChunk);
      for (int r = 0; r < kChunk; ++r) ref[r] = ((uint64_t)ids[r] << 10) | (uint64_t)r;
      std::sort(ref.begin(), ref.end());
      for (int p = 0; p < kChunk; ++p) bad += o.id[p] != (uint32_t)(ref[p] >> 10) || o.r[p] != (uint32_t)(ref[p] & 1023u);
    }
    ++checks;
  }
  for (int it = 0; it < 3000; ++it) {
    std::vector<uint32_t> v(kChunk);
    const int ones = (int)(rnd() % (uint32_t)(kChunk + 1));
    for (int i = 0; i < kChunk; ++i) v[i] = it % 2 ? (uint32_t)(i < ones) : rnd();
    if (it % 4 == 3)  // a rotated run
      std::rotate(v.begin(), v.begin() + (int)(rnd() % (uint32_t)kChunk), v.end());
    else
      for (int i = kChunk - 1; i > 0; --i) std::swap(v[i], v[rnd() % (uint32_t)(i + 1)]);
    std::vector<uint32_t> want = v;
    std::sort(want.begin(), want.end());
    network(v);
    bad += v != want;
    ++checks;
  }
  printf("checks=%ld declined=%ld bad=%ld\n", checks, declined, bad);
  return bad != 0 || declined == 0;
}
