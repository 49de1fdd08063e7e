// gpz_encode.cuh -- compress kernel of the B200 GPZ codec.
//
//   compress_kernel   runCompressKernel[2D] + CUB scan + header/meta assembly
//                     + runCompactKernel (reference src/cudaWarpCompress.cu:32-796,
//                     1620-1702; float64 twin src/cudaWarpCompressDouble.cu)
//                     fused into one persistent, single-pass kernel.
//
// A CTA of four warps encodes one 1024-point chunk at a time, eight points a
// thread.  The stable rank of point p among equal block ids is
// r(p) = (p % 32) * 32 + p / 32, so the composite (block id, r) is unique and
// any correct sort reproduces the reference's order.  Per chunk:
//   1. load the points, the chunk's min / max; quantize (block id in registers,
//      relative position in shared memory); place the oldest parked payload,
//      whose stream offset the last warp looks up while the first one works
//      out the chunk's scalars;
//   2. rank: 1024 buckets over the id range (shared-atomic counts, scan,
//      placement at bucket start + arrival slot, then odd-even transposition
//      between neighbouring positions); a chunk with too crowded a bucket goes
//      through a comparison network of the whole CTA (ids below 2^22) or a
//      stable radix sort (wider ids, and the few ids of one radix pass);
//   3. runs of equal ids (unique ids, deltas, counts), the payload's size,
//      which is published at once for the chunks behind;
//   4. bit planes, eight at a time per warp, into a staged payload, which
//      stays parked in shared memory until a later chunk's step 1 or 3.
//
// What bounds it: instruction issue (55 %) and shared-memory wavefronts (58 %)
// with the barriers between the steps on top; HBM needs a quarter of the time.
// One warp a chunk with 32 points a lane (128-168 registers, 12-16 warps an
// SM, payloads placed behind CTA barriers) issued 42 % and took a chunk's whole
// latency, some 50 us, on any input: this form takes 18 against 63 us on 5,003
// float 3D points, 0.75 against 1.06 ms on 50M double 3D points of a lattice,
// 1.48 against 1.55 ms on the 143.7M-point clustered snapshot, 0.36 against
// 0.42 ms on 32M uniform points.
//
// Two parked payloads a CTA: a payload can be placed once all chunks before it
// have published their sizes, and CTAs differ by tens of percent from chunk to
// chunk.  With room for one (8 CTAs an SM) nine in ten look-ups had to wait,
// with two (6 CTAs) one in twenty.
#pragma once

#include <cfloat>
#include <type_traits>
#include "gpz_kernels.cuh"

namespace gpzb {

constexpr int kEncThreads = 128;          // threads (one chunk) per CTA
constexpr int kEncWarps = kEncThreads / 32;
constexpr int kEncPer = kChunk / kEncThreads;  // points per thread
constexpr int kEncBuckets = 1024;         // ranking buckets per chunk
constexpr int kEncBucketBits = 11;        // no kernel uses it any more; a CPU check (tests/host/bucket_check.cu) does
constexpr uint32_t kEncOnePass = 512;     // ids below this: one radix pass, no buckets
constexpr int kEncSmall = 16;             // a bucket of this many points or more is sorted on its own
constexpr int kEncCrowd = 256;            // one above this size declines the chunk, and so do more than
constexpr int kEncCrowdPoints = 512;      //   this many points in all buckets of kEncSmall or more
constexpr uint32_t kEncBucketBackoff = 8; // chunks sorted directly after two declined ones in a row
constexpr int kEncSlots = 2;              // payloads a CTA can park
constexpr int kEncCtas = 6;               // resident CTAs per SM (36 KB of shared memory each)
constexpr int kEncHalo = 16;              // positions a warp orders beyond its own on either side
constexpr int kEncOrd = 9;                // positions per lane while ordering: 32 * 9 = 256 + 2 * 16
static_assert(kEncSlots >= 2, "the oldest payload is looked up while the newest is written");
static_assert(kChunk / kEncWarps + 2 * kEncHalo == 32 * kEncOrd, "ordering window");
static_assert(kEncHalo >= kEncSmall - 1, "a small bucket must fit the halo");

// Batcher's odd-even merge sort network on 32 values (191 exchanges).  No kernel
// sorts with it any more; its CPU check (tests/host/network_check.cu) stays.
__host__ __device__ __forceinline__ void oem_sort32(uint32_t (&a)[32]) {
#pragma unroll
  for (int p = 1; p < 32; p <<= 1)
#pragma unroll
    for (int k = p; k >= 1; k >>= 1)
#pragma unroll
      for (int j = k % p; j + k < 32; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < 32 && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
            const uint32_t x = a[i + j], y = a[i + j + k];
            a[i + j] = x < y ? x : y;
            a[i + j + k] = x < y ? y : x;
          }
}

// Swizzled index of element i in a 1024-word array (see swz): rows of 32
// words whose 16-byte quads are XORed by the row, so the plane jobs' row
// reads (lane l: row l) and eight consecutive words per thread are free of
// bank conflicts.
__device__ __forceinline__ uint32_t sx(uint32_t i) { return (uint32_t)swz((int)i); }

__device__ __forceinline__ float min2(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float max2(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double min2(double a, double b) { return from_ord(min(ord_of(a), ord_of(b))); }
__device__ __forceinline__ double max2(double a, double b) { return from_ord(max(ord_of(a), ord_of(b))); }

// Index of rank r in a 1024-word array that is written by points (32 ranks a
// row apart) and read in any order: the row's five bits XORed into the bank.
__device__ __forceinline__ uint32_t rx(uint32_t r) { return r ^ (r >> 5); }

// Shared memory of the ranking of a chunk.
struct RankShared {
  __align__(16) uint32_t A[2][kChunk];  // bucket counts -> sorted composites -> deltas | placed composites -> run starts
                                        // (roles alternate from chunk to chunk: clearing the counts needs no barrier)
  uint32_t R[kChunk];            // relative positions by point -> run lengths
  uint32_t Q[kChunk];            // ranks in sorted order (not of narrow chunks) -> relative positions in that order
  __align__(16) double mm[kEncWarps][8];   // warps' minima (0..2) and maxima (4..6), in the stream's type
  __align__(16) double nm[4];    // chunk: -min / (2 eb) per axis, in the stream's type
  __align__(16) uint32_t sc[4];  // chunk: id multipliers of y and z, largest id
  __align__(16) uint32_t tot[kEncWarps];   // per-warp sums of the bucket / digit scans
  __align__(16) uint32_t big[kEncWarps];   // per-warp largest bucket
  __align__(16) uint32_t cpts[kEncWarps];  // points in buckets of kEncSmall or more
  __align__(16) uint32_t small[kEncWarps]; // per-warp largest bucket below that
  uint32_t crowd[kEncCrowdPoints / kEncSmall];  // those buckets: first position << 16 | points
  uint32_t ncrowd;
};

// A compress CTA's shared memory.
struct EncShared : RankShared {
  __align__(16) uint32_t P[kEncSlots][kStageBytes / 4];  // staged payloads
  struct { unsigned long long c; uint32_t payload; } park[kEncSlots];  // their chunks and sizes
  unsigned long long goff;       // stream offset of the parked chunk (kGoffPending, kGoffNone: none)
  unsigned long long next[2];    // chunk claimed for the next iteration, by parity
  __align__(16) uint32_t relor[kEncWarps]; // OR of the relative positions
  __align__(16) uint32_t seg[8 * kEncWarps];  // run starts per 32 positions: [warp][j]
  __align__(16) uint32_t dor[kEncWarps];   // OR of the deltas
  __align__(16) uint32_t cmax[kEncWarps];  // longest run
  uint32_t first;                // smallest block id
  Control *overflowed;           // stream whose id_overflow this CTA has set last
};
constexpr unsigned long long kGoffNone = ~0ull, kGoffPending = ~0ull - 1;

__device__ __forceinline__ uint4 ld4(const uint32_t *p) { return *reinterpret_cast<const uint4 *>(p); }

// One 32-element plane word of a delta / count section: bytes 4*lane.. of the
// plane, MSB-first bit order (src/cudaWarpCompress.cu:357-408), only the
// `room` bytes the plane has there.  Reversing the word's bits reverses the
// order of its bytes too.
__device__ __forceinline__ void put_plane_bytes(uint8_t *d, int room, uint32_t word) {
  const uint32_t w = brev32(word);
  if (room > 0) d[0] = (uint8_t)(w >> 24);
  if (room > 1) d[1] = (uint8_t)(w >> 16);
  if (room > 2) d[2] = (uint8_t)(w >> 8);
  if (room > 3) d[3] = (uint8_t)w;
}

// Bit planes b0..b0+7 (those below nb; b0 a multiple of 8) of a 1024-element
// array (swizzled rows) by one warp: lane l takes elements 32l..32l+31, gathers
// the eight bits of each and turns them into plane words.
// Planes go MSB plane first to byte pos0 of the staged payload: byte planes of
// bpp bytes (bpp != 0) or planes of 32 words.
__device__ __forceinline__ void plane_job(const uint32_t *arr, uint8_t *stage, uint32_t pos0, uint32_t nb, uint32_t b0,
                                          uint32_t bpp, int lane) {
  uint32_t w[8];
  const uint32_t k = b0 >> 3;
  const uint32_t s0 = k | ((4u + k) << 4);  // byte k of both sources
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    // quads h, h+2, h+4, h+6 of the row: elements 4h.. (+0, +8, +16, +24)
    const uint4 q0 = ld4(arr + qoff(lane, h)), q1 = ld4(arr + qoff(lane, h + 2));
    const uint4 q2 = ld4(arr + qoff(lane, h + 4)), q3 = ld4(arr + qoff(lane, h + 6));
    w[4 * h + 0] = prmt(prmt(q0.x, q1.x, s0), prmt(q2.x, q3.x, s0), 0x5410);
    w[4 * h + 1] = prmt(prmt(q0.y, q1.y, s0), prmt(q2.y, q3.y, s0), 0x5410);
    w[4 * h + 2] = prmt(prmt(q0.z, q1.z, s0), prmt(q2.z, q3.z, s0), 0x5410);
    w[4 * h + 3] = prmt(prmt(q0.w, q1.w, s0), prmt(q2.w, q3.w, s0), 0x5410);
  }
  low_stages<8>(w);
  const uint32_t left = nb - b0;  // planes of this job (all 8, or the top ones)
  if (bpp) {
    const int room = (int)bpp - 4 * lane;
    uint8_t *d = stage + pos0 + (left - 1u) * bpp + 4u * lane;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if ((uint32_t)b >= left) break;
      put_plane_bytes(d, room, w[b]);
      d -= bpp;
    }
  } else {
    uint32_t *d = reinterpret_cast<uint32_t *>(stage + pos0) + 32u * (left - 1u) + lane;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      if ((uint32_t)b >= left) break;
      d[-32 * b] = w[b];
    }
  }
}

// Sum of the entries of warps before `warp`, and of all.
__device__ __forceinline__ uint32_t before4(const uint4 &t, int warp, uint32_t &all) {
  all = t.x + t.y + t.z + t.w;
  return (warp > 0 ? t.x : 0u) + (warp > 1 ? t.y : 0u) + (warp > 2 ? t.z : 0u);
}
__device__ __forceinline__ uint32_t max4(const uint4 &t) { return max(max(t.x, t.y), max(t.z, t.w)); }

// Point of rank r: r = (p % 32) * 32 + p / 32 swaps the two five-bit halves.
__device__ __forceinline__ uint32_t point_of_rank(uint32_t r) { return ((r * 1025u) >> 5) & 1023u; }

__device__ __forceinline__ uint32_t warp_inc_scan(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Stable radix sort of the chunk by block id, for chunks of up to kEncOnePass
// ids, of wide ids with too crowded a bucket, and a short last chunk: least
// significant digit first over the points in rank order, so equal ids keep
// the order of their ranks.  A warp takes 256 consecutive elements, 32 at a
// time; lanes of one digit find each other by match.any and the first of them
// advances the warp's counter of that digit, so an element's place is the
// digit's start (scan over digits, warps within a digit) plus its arrival
// number.  ceil(bits / 9) passes.
// byr: ids by rank (rx); cnt: 4 KB of counters; perm: two permutations of
// 1024 ranks.  Begins and ends with a barrier; returns the sorted ranks.
__device__ __forceinline__ const uint16_t *radix_rank(const uint32_t *byr, uint32_t *scr, uint16_t *perm,
                                                          uint32_t *tot, uint32_t idbits) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t passes = max((idbits + 8u) / 9u, 1u);
  const uint32_t dbits = max((idbits + passes - 1u) / passes, 1u), D = 1u << dbits;
  uint16_t *const cnt = reinterpret_cast<uint16_t *>(scr);  // [digit][warp]
  unsigned long long *const c8 = reinterpret_cast<unsigned long long *>(scr);
  __syncthreads();  // the ids by rank are in place, the counters' words free
#pragma unroll 1
  for (uint32_t ps = 0; ps < passes; ++ps) {
    const uint32_t shift = ps * dbits;
    for (uint32_t i = t; i < D / 2u; i += kEncThreads) reinterpret_cast<uint4 *>(scr)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const uint16_t *const from = perm + ((ps + 1u) & 1u) * kChunk;
    uint16_t *const to = perm + (ps & 1u) * kChunk;
    uint32_t dr[8], off[8];  // digit << 10 | rank; arrival number in the warp's digit
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const uint32_t i = 256u * warp + 32u * s + lane;
      const uint32_t r = ps == 0 ? i : (uint32_t)from[i] & 1023u;
      const uint32_t d = (byr[rx(r)] >> shift) & (D - 1u);
      const uint32_t peers = __match_any_sync(FULL, d);
      const uint32_t lower = __popc(peers & ((1u << lane) - 1u));
      uint16_t *const cw = cnt + 4u * d + warp;
      const uint32_t old = *cw;
      __syncwarp();
      if (lower == 0u) *cw = (uint16_t)(old + __popc(peers));
      __syncwarp();
      dr[s] = (d << 10) | r;
      off[s] = old + lower;
    }
    __syncthreads();
    // exclusive scan over (digit, warp): thread t owns digits per * t ..
    const uint32_t per = max(D / kEncThreads, 1u);
    uint32_t sum = 0;
    if (t * per < D)
      for (uint32_t i = 0; i < per; ++i) {
        const unsigned long long v = c8[t * per + i];
        const uint32_t a = (uint32_t)v, b = (uint32_t)(v >> 32);
        sum += (a & 0xFFFFu) + (a >> 16) + (b & 0xFFFFu) + (b >> 16);
      }
    const uint32_t inc = warp_inc_scan(sum, lane);
    if (lane == 31) tot[warp] = inc;
    __syncthreads();
    uint32_t all;
    uint32_t run = before4(ld4(tot), warp, all) + inc - sum;
    if (t * per < D)
      for (uint32_t i = 0; i < per; ++i) {
        const unsigned long long v = c8[t * per + i];
        const uint32_t a = (uint32_t)v, b = (uint32_t)(v >> 32);
        const uint32_t s1 = run + (a & 0xFFFFu), s2 = s1 + (a >> 16), s3 = s2 + (b & 0xFFFFu);
        c8[t * per + i] = (unsigned long long)(run | (s1 << 16)) | ((unsigned long long)(s2 | (s3 << 16)) << 32);
        run = s3 + (b >> 16);
      }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 8; ++s) to[(uint32_t)cnt[4u * (dr[s] >> 10) + warp] + off[s]] = (uint16_t)(dr[s] & 1023u);
    __syncthreads();
  }
  return perm + ((passes + 1u) & 1u) * kChunk;
}

// Compare-exchange step j of a bitonic merge of k values (lane l: positions
// K l ..): the merge's first step (j = k / 2) pairs position i with i ^ (k - 1),
// the others i with i ^ j, so the minimum always goes to the lower position.
// Partners in other lanes come by shuffles.
template <int K>
__device__ __forceinline__ void exchange(uint32_t (&v)[K], int lane, int k, int j) {
  const bool mirror = j == (k >> 1);
  if (j < K) {  // both in this lane
#pragma unroll
    for (int e = 0; e < K; ++e) {
      const int p = mirror ? e ^ (k - 1) : e ^ j;
      if (e < p) {
        const uint32_t x = v[e], y = v[p];
        v[e] = min(x, y);
        v[p] = max(x, y);
      }
    }
  } else {
    const int m = mirror ? k / K - 1 : j / K;  // partner lane ^ m
    const bool upper = (lane & (j / K)) != 0;
    uint32_t o[K];
#pragma unroll
    for (int e = 0; e < K; ++e) o[e] = __shfl_xor_sync(0xFFFFFFFFu, v[mirror ? K - 1 - e : e], m);
#pragma unroll
    for (int e = 0; e < K; ++e) v[e] = upper ? max(v[e], o[e]) : min(v[e], o[e]);
  }
}

// Ascending sort of a warp's 32 K values: about 60 / 150 / 250 / 460
// instructions for K = 1 / 2 / 4 / 8, where the same network in shared memory
// took 2,000 for 256 values.
template <int K>
__device__ __forceinline__ void warp_sort(uint32_t (&v)[K], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * K; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) exchange<K>(v, lane, k, j);
}

// The same of the n <= 32 K distinct values a[0..n), padded with the largest value.
template <int K>
__device__ __forceinline__ void warp_sort_regs(uint32_t *a, uint32_t n, int lane) {
  uint32_t v[K];
#pragma unroll
  for (int e = 0; e < K; ++e) v[e] = (uint32_t)(K * lane + e) < n ? a[K * lane + e] : 0xFFFFFFFFu;
  warp_sort<K>(v, lane);
#pragma unroll
  for (int e = 0; e < K; ++e)
    if ((uint32_t)(K * lane + e) < n) a[K * lane + e] = v[e];
}

static __device__ __noinline__ void warp_sort_small(uint32_t *a, uint32_t n, int lane) {
  if (n <= 32u) warp_sort_regs<1>(a, n, lane);
  else if (n <= 64u) warp_sort_regs<2>(a, n, lane);
  else if (n <= 128u) warp_sort_regs<4>(a, n, lane);
  else warp_sort_regs<8>(a, n, lane);
}

// Sort of a full chunk's 1024 composites id << 10 | rank (ids below 2^22) by
// the CTA, for chunks the buckets have declined: each warp sorts 256 in
// registers; the two merges above that take three exchanges between warps,
// through S and H in turn.  S: ids by rank (rx); H: the sorted composites.
// Begins and ends with a barrier.
//
// Bound by instruction issue, the same on any input, with six barriers.  The
// radix sort has five a pass, two or three passes at these ids, and its match.any
// takes the longer the more digits differ.  20M float points, half of them in one
// place: 396 -> 296 us in 2D (19-bit ids; 10.2 -> 8.8 K warp instructions and 3.1
// -> 2.4 K shared wavefronts a chunk), 419 -> 309 us in 3D (21 bits), 292 -> 280
// us with ids of two passes; 3D points on 40 sites 366 -> 296 us.
__device__ __forceinline__ void cta_sort(uint32_t *H, uint32_t *S) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  __syncthreads();  // the ids by rank are in place
  uint32_t v[kEncPer];
#pragma unroll
  for (int e = 0; e < kEncPer; ++e) v[e] = (S[rx(kEncPer * t + e)] << 10) | (uint32_t)(kEncPer * t + e);
  auto get = [](const uint32_t *buf, int from, uint32_t (&o)[kEncPer]) {
    const uint4 a = ld4(buf + 4 * from), b = ld4(buf + 4 * (kEncThreads + from));
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
    o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
  };
  // position 8t + e against thread `from`'s e (mirror: 7 - e); the upper takes the larger
  auto cross = [&](uint32_t *buf, int from, bool mirror, bool upper) {
    *reinterpret_cast<uint4 *>(buf + 4 * t) = make_uint4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint4 *>(buf + 4 * (kEncThreads + t)) = make_uint4(v[4], v[5], v[6], v[7]);
    __syncthreads();
    uint32_t o[kEncPer];
    get(buf, from, o);
#pragma unroll
    for (int e = 0; e < kEncPer; ++e) {
      const uint32_t y = o[mirror ? kEncPer - 1 - e : e];
      v[e] = upper ? max(v[e], y) : min(v[e], y);
    }
  };
  auto finish = [&]() {  // within the warp's 256 positions
#pragma unroll
    for (int j = 16 * kEncPer; j > 0; j >>= 1) exchange<kEncPer>(v, lane, 0, j);
  };
  warp_sort<kEncPer>(v, lane);
  cross(H, t ^ 63, true, (warp & 1) != 0);    // i with i ^ 511
  finish();
  cross(S, t ^ 127, true, (warp & 2) != 0);   // i with i ^ 1023
  cross(H, t ^ 32, false, (warp & 1) != 0);   // i with i ^ 256
  finish();
  __syncthreads();  // H has been read
  *reinterpret_cast<uint4 *>(H + 8 * t) = make_uint4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<uint4 *>(H + 8 * t + 4) = make_uint4(v[4], v[5], v[6], v[7]);
  __syncthreads();
}

// Ranks a chunk that the buckets do not, from the ids by rank in S: by the
// CTA's network (`network`; nullptr, the sorted composites in H) or by the radix
// sort (the sorted ranks).  One call for both: with two, the batch kernels spilt
// more (7.75 -> 7.84 ms for the bench's 256 snapshots).
static __device__ __noinline__ const uint16_t *rank_rest(uint32_t *H, uint32_t *S, uint16_t *perm, uint32_t *tot,
                                                         uint32_t idbits, bool network) {
  if (!network) return radix_rank(S, H, perm, tot, idbits);
  cta_sort(H, S);
  return nullptr;
}

// A chunk's points in registers, one 16-byte load (kVec points) at a time:
// thread t's point e = kVec h + i is point 128 kVec h + kVec t + i of the
// chunk.  Chunks of misaligned axes and a short last chunk load single points;
// the latter's slots past the end hold a copy of its first point, which leaves
// min / max, the id range and the relative positions' width unchanged.
template <typename T>
struct Points {
  static constexpr int kVec = 16 / (int)sizeof(T);
  __device__ __forceinline__ static uint32_t point(uint32_t t, int e) {
    return 128u * kVec * (e / kVec) + kVec * t + (e % kVec);
  }
  // stable rank r(p) = (p % 32) * 32 + p / 32 of point(t, e): base(t) + step(e)
  __device__ __forceinline__ static uint32_t rank_base(uint32_t t) {
    return 32u * kVec * (t % (32 / kVec)) + t / (32 / kVec);
  }
  __host__ __device__ constexpr static uint32_t rank_step(int e) { return 32u * (e % kVec) + 4u * kVec * (e / kVec); }
};

// First position that warp `warp` orders: its own 256 and kEncHalo more on
// either side (all on one side at the chunk's ends).
__host__ __device__ constexpr uint32_t ord_window(int warp) {
  return warp == 0 ? 0u : (warp == kEncWarps - 1 ? kChunk - 32u * kEncOrd : 256u * warp - kEncHalo);
}

// Odd-even transposition over a lane's kEncOrd positions: the even (h = 0) or
// odd (h = 1) pairs.  cut[j] is all ones where positions j and j + 1 are not to
// be exchanged (wide form; the narrow one's neighbours of different buckets are
// in order already).
template <bool kNarrow>
__host__ __device__ __forceinline__ void order_pairs(uint32_t (&k)[kEncOrd], const uint32_t (&cut)[kEncOrd], int h) {
#pragma unroll
  for (int j = h; j + 1 < kEncOrd; j += 2) {
    const uint32_t x = k[j], y = k[j + 1];
    k[j] = min(x, kNarrow ? y : y | cut[j]);
    k[j + 1] = max(kNarrow ? x : x & ~cut[j], y);
  }
}

// The pairs across lanes: nx is the next lane's first value, pv the previous
// lane's last, pcut the previous lane's last cut.
template <bool kNarrow>
__host__ __device__ __forceinline__ void order_across(uint32_t (&k)[kEncOrd], const uint32_t (&cut)[kEncOrd], uint32_t nx,
                                                      uint32_t pv, uint32_t pcut, int lane) {
  if (kNarrow) {
    if (lane < 31) k[kEncOrd - 1] = min(k[kEncOrd - 1], nx);
    if (lane > 0) k[0] = max(k[0], pv);
  } else {
    k[kEncOrd - 1] = min(k[kEncOrd - 1], nx | cut[kEncOrd - 1]);
    k[0] = max(k[0], pv & ~pcut);
  }
}

// Ranks a full chunk's points through buckets over their id range.
//  * kNarrow (ids below 2^22): 1024 buckets that split the range evenly
//    (id * scale >> 32; up to 1023 ids each have their own, but for the first
//    two); S holds whole composites id << 10 | r.  H receives
//    the sorted composites.
//  * wide: buckets are the id bits from `low` up; S holds the bits below with
//    r, and the bucket of every position lies beside (in Q).  H receives the
//    sorted ids and Q the sorted ranks (16 bits each).
// A few crowded buckets (kEncSmall points or more: a dense cluster) are sorted
// by one warp each; with too many points in them (kEncCrowd, kEncCrowdPoints)
// the result is false, S and H hold nothing of use and key is unchanged.  H
// and sm.ncrowd must be clear; ends with a barrier.
//
// 32M clustered points with a few percent of them in one cluster: 0.85 ms when
// any bucket of 16 points sent the chunk to the radix sort (three passes at
// these id ranges), 0.41 ms so, 0.51 ms in the one-warp form.
//
// The limits, by 20M float points of which a share lies in one place (2D, us;
// with kEncCrowd 128 / 192 / 256): 15 % 288 / 262 / 261, 20 % 282 / 310 / 263,
// 25 % 285 / 298 / 342, 30 % 289 / 297 / 307, 50 % 294 / 294 / 296.  One warp
// sorts such a bucket while three wait, so the limit's worth lies below it, and
// chunks on both sides of it in turn are the worst case.  Many crowded buckets
// (with kEncCrowdPoints 256 / 512 / 1024): an integer grid 269 / 269 / 346, 3D
// points on 40 sites 296 / 296 / 384.  kEncBucketBackoff 8 / 16: 25 % 342 / 329,
// 90 % 320 / 317, the others within 1 %.
template <typename T, bool kNarrow>
__device__ __forceinline__ bool rank_buckets(RankShared &sm, uint32_t *H, uint32_t *S, const uint32_t (&key)[kEncPer],
                                             uint32_t bound, int t, int lane, int warp) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const uint32_t rbase = Points<T>::rank_base(t);
  const uint32_t low = kNarrow ? 0u : 22u - __clz(bound);  // wide: id bits below the bucket
  // 1024 * 2^32 / (bound + 1), a little less: id * scale >> 32 <= 1023 (at
  // most 2^32 - 1, with which it is id - 1)
  const uint32_t scale = kNarrow ? __float2uint_rz(__fdividef(4.39804e12f, __uint2float_rn(bound) + 1.0f)) : 0u;
  uint32_t bs[kEncPer];  // arrival slot << 14 | bucket << 2
#pragma unroll
  for (int e = 0; e < kEncPer; ++e) {
    // in range by construction; the mask keeps the access in bounds whatever the id
    const uint32_t b = (kNarrow ? __umulhi(key[e], scale) : key[e] >> low) & (kEncBuckets - 1u);
    bs[e] = (atomicAdd(&H[b], 1u) << 14) | (b << 2);
  }
  __syncthreads();  // counts
  // exclusive scan; thread t owns buckets 8t..8t+7.  Starts are kept in bytes.
  uint32_t c8[8];
  {
    const uint4 u0 = ld4(H + 8 * t), u1 = ld4(H + 8 * t + 4);
    c8[0] = u0.x; c8[1] = u0.y; c8[2] = u0.z; c8[3] = u0.w;
    c8[4] = u1.x; c8[5] = u1.y; c8[6] = u1.z; c8[7] = u1.w;
  }
  uint32_t sum = 0, mx = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    mx = max(mx, c8[i]);
    const uint32_t n = c8[i];
    c8[i] = sum;
    sum += 4u * n;
  }
  const uint32_t inc = warp_inc_scan(sum, lane);
  mx = warp_max(mx);
  {
    const uint32_t b0 = inc - sum;
    *reinterpret_cast<uint4 *>(H + 8 * t) = make_uint4(c8[0] + b0, c8[1] + b0, c8[2] + b0, c8[3] + b0);
    *reinterpret_cast<uint4 *>(H + 8 * t + 4) = make_uint4(c8[4] + b0, c8[5] + b0, c8[6] + b0, c8[7] + b0);
  }
  uint32_t pts = 0;
  if (mx >= (uint32_t)kEncSmall) {  // the same for the whole warp
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t n = ((i < 7 ? c8[i < 7 ? i + 1 : 0] : sum) - c8[i]) >> 2;
      if (n >= (uint32_t)kEncSmall) pts += n;
    }
    pts = __reduce_add_sync(FULL, pts);
  }
  if (lane == 31) {
    sm.tot[warp] = inc;
    sm.big[warp] = mx;
    sm.cpts[warp] = pts;
  }
  __syncthreads();  // warps' totals
  const uint32_t biggest = max4(ld4(sm.big));
  // starts are relative to the quarter of the buckets a warp scanned
  const uint4 tt = ld4(sm.tot);
  const uint32_t q1 = tt.x, q2 = tt.x + tt.y, q3 = q2 + tt.z;
  if (biggest >= (uint32_t)kEncSmall) {
    const uint4 c4 = ld4(sm.cpts);
    if (biggest > (uint32_t)kEncCrowd || c4.x + c4.y + c4.z + c4.w > (uint32_t)kEncCrowdPoints) return false;
    const uint32_t b0 = inc - sum + (warp < 2 ? (warp == 0 ? 0u : q1) : (warp == 2 ? q2 : q3));
    uint32_t ms = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t n = ((i < 7 ? c8[i < 7 ? i + 1 : 0] : sum) - c8[i]) >> 2;
      if (n >= (uint32_t)kEncSmall) sm.crowd[atomicAdd(&sm.ncrowd, 1u)] = ((c8[i] + b0) << 14) | n;
      else ms = max(ms, n);
    }
    ms = warp_max(ms);
    if (lane == 0) sm.small[warp] = ms;
  }
  uint16_t *const Bk = reinterpret_cast<uint16_t *>(sm.Q);
  const uint32_t lmask = (1u << low) - 1u;
#pragma unroll
  for (int e = 0; e < kEncPer; ++e) {
    const uint32_t b4 = bs[e] & 0xFFCu;
    const uint32_t quarter = b4 < 2048u ? (b4 < 1024u ? 0u : q1) : (b4 < 3072u ? q2 : q3);
    const uint32_t pos4 = *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(H) + b4) + (bs[e] >> 12) + quarter;
    const uint32_t v = ((kNarrow ? key[e] : key[e] & lmask) << 10) + (rbase + Points<T>::rank_step(e));
    *reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(S) + pos4) = v;
    if (!kNarrow) Bk[pos4 >> 2] = (uint16_t)(b4 >> 2);
  }
  __syncthreads();  // placed
  uint32_t largest = biggest;  // of the buckets still to order
  if (biggest >= (uint32_t)kEncSmall) {
    for (uint32_t k = warp; k < sm.ncrowd; k += kEncWarps) warp_sort_small(S + (sm.crowd[k] >> 16), sm.crowd[k] & 0xFFFFu, lane);
    largest = max4(ld4(sm.small));
    __syncthreads();  // crowded buckets in order
  }
  // Order inside the buckets: every warp takes its 256 positions and 16 more
  // on either side (32 on one side at the chunk's ends), nine a lane; such a
  // bucket has at most 15 points, so each of the warp's own positions sees its
  // whole bucket.  Neighbours are compared
  // in the order even pairs, across lanes, odd pairs, across lanes: ceil(n / 2)
  // rounds order a bucket of n points wherever it lies.
  uint32_t k9[kEncOrd];
  const uint32_t p0 = ord_window(warp) + kEncOrd * lane, o0 = p0 - 256u * warp;
#pragma unroll
  for (int j = 0; j < kEncOrd; ++j) k9[j] = S[p0 + j];
  const uint32_t rounds = (largest + 1u) >> 1;
  if (kNarrow) {
#pragma unroll 1
    for (uint32_t it = 0; it < rounds; ++it) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        order_pairs<true>(k9, k9, h);
        const uint32_t nx = __shfl_down_sync(FULL, k9[0], 1), pv = __shfl_up_sync(FULL, k9[kEncOrd - 1], 1);
        order_across<true>(k9, k9, nx, pv, 0u, lane);
      }
    }
#pragma unroll
    for (int j = 0; j < kEncOrd; ++j)
      if (o0 + j < 256u) H[p0 + j] = k9[j];
  } else {
    // cut[j] = all ones where positions j and j+1 are of different buckets
    // (never exchanged), the last entry towards the next lane
    uint32_t b9[kEncOrd], cut[kEncOrd];
#pragma unroll
    for (int j = 0; j < kEncOrd; ++j)
      b9[j] = (uint32_t)Bk[p0 + j];
    const uint32_t nb = __shfl_down_sync(FULL, b9[0], 1);
#pragma unroll
    for (int j = 0; j + 1 < kEncOrd; ++j) cut[j] = b9[j] == b9[j + 1] ? 0u : FULL;
    cut[kEncOrd - 1] = lane < 31 && b9[kEncOrd - 1] == nb ? 0u : FULL;
    uint32_t pcut = __shfl_up_sync(FULL, cut[kEncOrd - 1], 1);
    if (lane == 0) pcut = FULL;
    __syncthreads();  // the buckets have been read: Q takes the ranks
#pragma unroll 1
    for (uint32_t it = 0; it < rounds; ++it) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        order_pairs<false>(k9, cut, h);
        const uint32_t nx = __shfl_down_sync(FULL, k9[0], 1), pv = __shfl_up_sync(FULL, k9[kEncOrd - 1], 1);
        order_across<false>(k9, cut, nx, pv, pcut, lane);
      }
    }
#pragma unroll
    for (int j = 0; j < kEncOrd; ++j)
      if (o0 + j < 256u) {
        H[p0 + j] = (b9[j] << low) | (k9[j] >> 10);
        Bk[p0 + j] = (uint16_t)(k9[j] & 1023u);
      }
  }
  __syncthreads();  // ranked
  return true;
}

template <typename T, int DIM>
__device__ __forceinline__ void load_points(const T *x, const T *y, const T *z, unsigned long long base,
                                            uint32_t nvalid, T (&v)[DIM][kEncPer]) {
  constexpr int V = Points<T>::kVec;
  const uint32_t t = threadIdx.x;
  const T *const X[3] = {x + base, y + base, z + base};
  uint32_t low = (uint32_t)(uintptr_t)x;
  if (DIM >= 2) low |= (uint32_t)(uintptr_t)y;
  if (DIM == 3) low |= (uint32_t)(uintptr_t)z;
  if (nvalid == (uint32_t)kChunk && (low & 15u) == 0u) {
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int h = 0; h < kEncPer / V; ++h) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(X[d]) + 128 * h + t);
        if constexpr (sizeof(T) == 4) {
          v[d][4 * h] = __uint_as_float(q.x); v[d][4 * h + 1] = __uint_as_float(q.y);
          v[d][4 * h + 2] = __uint_as_float(q.z); v[d][4 * h + 3] = __uint_as_float(q.w);
        } else {
          v[d][2 * h] = __hiloint2double((int)q.y, (int)q.x);
          v[d][2 * h + 1] = __hiloint2double((int)q.w, (int)q.z);
        }
      }
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int e = 0; e < kEncPer; ++e) {
        const uint32_t p = Points<T>::point(t, e);
        v[d][e] = __ldg(X[d] + (p < nvalid ? p : 0u));
      }
  }
}

// The warp's minima and maxima into sm.mm.
template <typename T, int DIM>
__device__ __forceinline__ void put_minmax(RankShared &sm, const T (&v)[DIM][kEncPer], int lane, int warp) {
  T mn[3], mx[3];
#pragma unroll
  for (int d = 0; d < DIM; ++d) warp_minmax(v[d], mn[d], mx[d]);
  if (lane == 0) {
    T *const m = reinterpret_cast<T *>(sm.mm[warp]);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      m[d] = mn[d];
      m[4 + d] = mx[d];
    }
  }
}

// Asks for chunk c's axes in L2 (bulk prefetches of the 16-byte aligned
// spans, one lane per axis), ahead of its load.
template <typename T, int DIM>
__device__ __forceinline__ void prefetch_points(const CArgs<T> &a, unsigned long long c, int lane) {
  if (lane < DIM && c < a.G) {
    const unsigned long long base = c * kChunk;
    const uint32_t nvalid = (uint32_t)min((unsigned long long)kChunk, a.n - base);
    const T *p = (lane == 0 ? a.x : (lane == 1 ? a.y : a.z)) + base;
    const uint32_t bytes = (nvalid * (uint32_t)sizeof(T)) & ~15u;
    if (bytes != 0u && (reinterpret_cast<uintptr_t>(p) & 15u) == 0u)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
  }
}

// Ranks a chunk's points by (block id, r): narrow buckets or the CTA's network
// (1: H holds the sorted composites), wide buckets (2: H the sorted ids, `ranks`
// the ranks) or the radix sort (0: S the ids by rank, rx, `ranks` the ranks).
// Full chunks of more than kEncOnePass ids try the buckets: spread evenly over
// 1,250 ids, 20M float 2D points took 313 us when ids below 2^11 went to two
// radix passes, 193 us so; at 441 ids one radix pass takes 276, what the buckets
// would gain there few inputs show.  No id is above
// `bound`; positions past the end of a short chunk rank last.  rank_skip counts
// the chunks still to sort without trying the buckets, declined the chunks the
// buckets have declined in a row.
template <typename T>
__device__ __forceinline__ int rank_chunk(RankShared &sm, uint32_t *H, uint32_t *S, uint32_t (&key)[kEncPer],
                                          uint32_t bound, uint32_t nvalid, uint32_t &rank_skip, uint32_t &declined,
                                          int t, int lane, int warp, const uint16_t *&ranks) {
  const bool full = nvalid == (uint32_t)kChunk, narrow = bound < (1u << 22);
  int how = 0;
  if (full && bound >= kEncOnePass && rank_skip == 0u) {
    if (narrow) how = rank_buckets<T, true>(sm, H, S, key, bound, t, lane, warp) ? 1 : 0;
    else how = rank_buckets<T, false>(sm, H, S, key, bound, t, lane, warp) ? 2 : 0;
    // one crowded chunk says little about the next (a shuffled, clustered
    // snapshot has a few); a second one in a row does (ordered points)
    if (how != 0) declined = 0u;
    else if (++declined >= 2u) rank_skip = kEncBucketBackoff;
  } else if (rank_skip != 0u) {
    --rank_skip;
  }
  ranks = reinterpret_cast<const uint16_t *>(sm.Q);
  if (how == 0) {
    const uint32_t rbase = Points<T>::rank_base(t);
    if (!full) {  // slots past the end sort last
#pragma unroll
      for (int e = 0; e < kEncPer; ++e)
        if (Points<T>::point(t, e) >= nvalid) key[e] = bound + 1u;
    }
#pragma unroll
    for (int e = 0; e < kEncPer; ++e) S[rx(rbase + Points<T>::rank_step(e))] = key[e];
    ranks = rank_rest(H, S, reinterpret_cast<uint16_t *>(sm.Q), sm.tot, bitlen(bound + (full ? 0u : 1u)),
                      full && narrow && bound >= kEncOnePass);
    if (ranks == nullptr) how = 1;
  }
  return how;
}

// The parked payloads of a CTA: `count` of them, the oldest in slot `head`.
struct Parked {
  uint32_t head, count;
};

// Header of the stream (:1674-1678; Double :1672-1680), by the first warp.
template <typename T>
__device__ __forceinline__ void put_header(const CArgs<T> &a, T eb, uint32_t seg, int lane) {
  uint32_t *h = reinterpret_cast<uint32_t *>(a.out);
  if (lane == 0) h[0] = a.dim;
  if (lane == 1) h[1] = (uint32_t)a.n;
  if (lane == 2) h[2] = (uint32_t)(a.n >> 32);
  if (lane == 3) h[3] = TT<T>::bits;
  if constexpr (sizeof(T) == 4) {
    if (lane == 4) h[4] = __float_as_uint((float)eb);
    if (lane == 5) h[5] = seg;
  } else {
    if (lane == 4) h[4] = (uint32_t)__double_as_longlong((double)eb);
    if (lane == 5) h[5] = (uint32_t)((unsigned long long)__double_as_longlong((double)eb) >> 32);
    if (lane == 6) h[6] = seg;
    if (lane == 7) h[7] = 32u;
  }
}

// Places the payload in `slot` at stream offset sm.goff, with its offset-table
// entry (:1679), and sets the stream's size after the last chunk.
template <typename T>
__device__ __forceinline__ void place_parked(const CArgs<T> &a, EncShared &sm, uint32_t slot) {
  using Tr = TT<T>;
  const unsigned long long off = sm.goff, c = sm.park[slot].c;
  const uint32_t payload = sm.park[slot].payload;
  if (off >= kGoffPending) return;  // the look-back gave up
  const uint32_t *const P = sm.P[slot];
  const unsigned long long G = a.G, pay_base = Tr::hdr + 8ull * G + (unsigned long long)Tr::meta * G;
  const int t = (int)threadIdx.x;
  constexpr int N = kEncThreads;
  if (t == 0) reinterpret_cast<unsigned long long *>(a.out + Tr::hdr)[c] = off;
  if (pay_base + off + payload > a.out_cap) {
    if (t == 0) set_status(a.ctl, kENOSPACE);
  } else {
    // four words in flight per thread: one shared-memory latency per 1.5 KB
    uint32_t *const dst = reinterpret_cast<uint32_t *>(a.out + pay_base + off);
    const uint32_t nw = payload / 4u;
    uint32_t w = t;
    for (; w + 3 * N < nw; w += 4 * N) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = P[w + i * N];
#pragma unroll
      for (int i = 0; i < 4; ++i) dst[w + i * N] = v[i];
    }
    for (; w < nw; w += N) dst[w] = P[w];
  }
  if (c == G - 1 && t == 0) a.ctl->stream_bytes = pay_base + off + payload;
}

// One warp: the stream offset of the payload in `slot` into sm.goff (kGoffPending when
// a predecessor's size is missing and `wait` is not set).
template <typename T>
__device__ __forceinline__ void look_up(const CArgs<T> &a, uint32_t slot, EncShared &sm, bool wait, int lane) {
  unsigned long long excl = 0;
  const int ok = resolve_prefix(a.ctl, a.look, sm.park[slot].c, excl, wait ? kSpinLimit : 0u, wait);
  if (lane == 0) sm.goff = ok > 0 ? excl : (ok < 0 ? kGoffPending : kGoffNone);
}

// The chunk's scalars, by one warp: per-axis values in lanes 0..2 (lane d:
// axis d).  Block counts, id multipliers, offsets -min / (2 eb) and the largest
// block id into sm.sc and sm.nm; returns the minimum (lane d) and maximum (lane
// 3 + d) of axis d, and the axis's share of the largest corner's id (term; it
// may not fit 31 bits when wide is set).
template <typename T, int DIM>
__device__ __forceinline__ T chunk_scalars(RankShared &sm, uint32_t seg, uint32_t sh, T eb, T inv, int lane,
                                           unsigned long long &term, bool &wide) {
  constexpr bool is64 = sizeof(T) == 8;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  T mmv;
  {
    const int k = lane < 6 ? (lane < 3 ? lane : lane + 1) : 0;
    T v[kEncWarps];
#pragma unroll
    for (int i = 0; i < kEncWarps; ++i) v[i] = reinterpret_cast<const T *>(sm.mm[i])[k];
    static_assert(kEncWarps == 4, "");
    const T lo = min2(min2(v[0], v[1]), min2(v[2], v[3]));
    const T hi = max2(max2(v[0], v[1]), max2(v[2], v[3]));
    mmv = lane < 3 ? lo : hi;
    if (DIM == 2 && (lane == 2 || lane == 5)) mmv = (T)0;  // 2D meta carries z = 0 (:518, :521)
  }
  const T mxv = __shfl_down_sync(FULL, mmv, 3);
  const T range = is64 ? (T)__dsub_rn((double)mxv, (double)mmv) : (T)__fsub_rn((float)mxv, (float)mmv);
  unsigned long long bn = block_num(range, seg, eb, false);
  if (is64 && DIM == 2) {
    const unsigned long long bw = block_num(range, seg, eb, true);
    bn = lane == 0 ? bw : bn;
  }
  const T nm = is64 ? (T)__dmul_rn(-(double)mmv, (double)inv) : (T)__fmul_rn(-(float)mmv, (float)inv);
  const unsigned long long qm = is64 ? __double2ull_rz(__fma_rn((double)mxv, (double)inv, (double)nm))
                                     : (unsigned long long)__float2uint_rz(__fmaf_rn((float)mxv, (float)inv, (float)nm));
  unsigned long long bnx, bny;
  if (is64) {
    bnx = __shfl_sync(FULL, bn, 0);
    bny = __shfl_sync(FULL, bn, 1);
  } else {
    bnx = __shfl_sync(FULL, (uint32_t)bn, 0);
    bny = __shfl_sync(FULL, (uint32_t)bn, 1);
  }
  const unsigned long long mult = lane == 0 ? 1ull : (lane == 1 ? bnx : bnx * bny);
  term = lane < DIM ? (qm >> sh) * mult : 0ull;
  // the chunk's largest quantized corner: every quantized value is at most its
  // axis's (the multiply-add and the truncation are monotone), so no id is
  // above the sum; ids are masked to 31 bits when it does not fit
  const float tf = lane < DIM ? __ull2float_rn(qm >> sh) * __ull2float_rn(mult) : 0.0f;
  wide = __any_sync(FULL, tf >= 7.0e8f);
  const uint32_t sum = __reduce_add_sync(FULL, (uint32_t)term);
  if (lane < 3) reinterpret_cast<T *>(sm.nm)[lane] = nm;
  if (lane == 0) *reinterpret_cast<uint4 *>(sm.sc) = make_uint4((uint32_t)bnx, (uint32_t)(bnx * bny), wide ? 0x7FFFFFFFu : sum, 0u);
  return mmv;
}

// The first warp's part of encoding chunk c between the barriers: its scalars,
// the id_overflow flag, the meta record's min / max (:332-344 / Double
// :333-345), the stream's header.
template <typename T, int DIM>
__device__ __forceinline__ void encode_scalars(const CArgs<T> &a, unsigned long long c, EncShared &sm, uint32_t seg,
                                               uint32_t sh, T eb, T inv, int lane) {
  using Tr = TT<T>;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  unsigned long long term;
  bool wide;
  const T mmv = chunk_scalars<T, DIM>(sm, seg, sh, eb, inv, lane, term, wide);
  if (wide) {
    // id_overflow: the largest corner in u64 arithmetic (terms below 7e8
    // cannot reach 2^31).  Set once per CTA and stream: the flag shares its
    // cache line with the work counter, and a store per chunk took 50M double
    // points from 1.1 to 2.3 ms.
    const unsigned long long corner = term + __shfl_down_sync(FULL, term, 1) + __shfl_down_sync(FULL, term, 2);
    if (lane == 0 && corner > 0x7FFFFFFFull && sm.overflowed != a.ctl) {
      a.ctl->id_overflow = 1u;
      sm.overflowed = a.ctl;
    }
  }
  uint8_t *meta = a.out + Tr::hdr + 8ull * a.G + (unsigned long long)Tr::meta * c;
  if (lane < 6) reinterpret_cast<T *>(meta)[lane] = mmv;
  if (c == 0) put_header<T>(a, eb, seg, lane);
}

// Encodes chunk c into a free slot of sm.P (see the top of the file) and
// returns it.  `par` is the iteration's parity, pa[slot] the arguments of a
// parked chunk; `claim` and, a phase later, `commit` run on the third warp (the
// next chunk is claimed and its points prefetched).  rank_skip counts the
// chunks still to sort without trying the buckets, declined the chunks the
// buckets have declined in a row.
template <typename T, int DIM, class PArgs, class Claim, class Commit>
__device__ __forceinline__ uint32_t encode_chunk(const CArgs<T> &a, unsigned long long c, EncShared &sm, int par,
                                                 uint32_t seg, T eb, T inv, const PArgs &pa, Parked &pk,
                                                 uint32_t &rank_skip, uint32_t &declined, Claim &&claim, Commit &&commit) {
  using Tr = TT<T>;
  constexpr bool is64 = sizeof(T) == 8;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t sh = (uint32_t)__ffs((int)seg) - 1u, msk = seg - 1u;
  const unsigned long long base = c * kChunk;
  const uint32_t nvalid = (uint32_t)min((unsigned long long)kChunk, a.n - base);
  const bool full = nvalid == (uint32_t)kChunk;
  uint32_t *const H = sm.A[par], *const S = sm.A[par ^ 1];
  bool pending;  // the oldest payload has to leave before this chunk's planes

  // ---- 1. points, min / max, quantization (:104-205) ----
  uint32_t key[kEncPer];
  uint32_t bound;  // no block id is above it
  {
    T v[DIM][kEncPer];
    load_points<T, DIM>(a.x, a.y, a.z, base, nvalid, v);
    // bucket counts (last used as run starts, done with before the last chunk's planes)
    *reinterpret_cast<uint4 *>(H + 8 * t) = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4 *>(H + 8 * t + 4) = make_uint4(0u, 0u, 0u, 0u);
    if (t == 0) sm.ncrowd = 0u;
    // NaNs are ignored and -0.0 orders below +0.0, as in the reference's warp
    // reductions (:122-139); slots past the end repeat a point
    put_minmax<T, DIM>(sm, v, lane, warp);
    __syncthreads();  // 1: minima and maxima, the oldest parked payload's offset
    pending = pk.count == (uint32_t)kEncSlots;
    if (warp == 0) encode_scalars<T, DIM>(a, c, sm, seg, sh, eb, inv, lane);
    else if (warp == kEncWarps - 1 && pending) look_up<T>(pa[pk.head], pk.head, sm, false, lane);
    __syncthreads();  // 2: the chunk's scalars

    // block id (mod 2^32, masked to 31 bits) and relative position
    const uint4 sc = ld4(sm.sc);
    bound = sc.z;
    uint32_t rel[kEncPer];
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const T nmd = reinterpret_cast<const T *>(sm.nm)[d];
      const uint32_t kmul = d == 1 ? sc.x : sc.y;
      const uint32_t rmul = d == 1 ? seg : seg * seg;
#pragma unroll
      for (int e = 0; e < kEncPer; ++e) {
        uint32_t kq, r;
        if constexpr (!is64) {
          const uint32_t q = __float2uint_rz(__fmaf_rn((float)v[d][e], (float)inv, (float)nmd));
          kq = q >> sh;
          r = q & msk;
        } else {
          const unsigned long long q = __double2ull_rz(__fma_rn((double)v[d][e], (double)inv, (double)nmd));
          kq = (uint32_t)(q >> sh);
          r = (uint32_t)q & msk;
        }
        key[e] = d == 0 ? kq : key[e] + kq * kmul;
        rel[e] = d == 0 ? r : rel[e] + r * rmul;
      }
    }
    uint32_t orv = 0;
#pragma unroll
    for (int e = 0; e < kEncPer; ++e) {
      key[e] &= 0x7FFFFFFFu;
      rel[e] &= 0x7FFFFFFFu;
      orv |= rel[e];
    }
    if constexpr (!is64) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<uint4 *>(sm.R + 512 * h + 4 * t) =
            make_uint4(rel[4 * h], rel[4 * h + 1], rel[4 * h + 2], rel[4 * h + 3]);
    } else {
#pragma unroll
      for (int h = 0; h < 4; ++h)
        *reinterpret_cast<uint2 *>(sm.R + 256 * h + 2 * t) = make_uint2(rel[2 * h], rel[2 * h + 1]);
    }
    orv = __reduce_or_sync(FULL, orv);
    if (lane == 0) sm.relor[warp] = orv;
  }
  if (pending && sm.goff != kGoffPending) {
    place_parked<T>(pa[pk.head], sm, pk.head);
    pk.head = pk.head + 1u < (uint32_t)kEncSlots ? pk.head + 1u : 0u;
    --pk.count;
    pending = false;
  }

  // ---- 2. rank the composites (block id, r) ----
  const uint16_t *ranks;
  const int how = rank_chunk<T>(sm, H, S, key, bound, nvalid, rank_skip, declined, t, lane, warp, ranks);

  // ---- 3. runs: unique ids, deltas, counts (:222-311) ----
  // thread t takes positions 128j + t, so that neighbouring lanes hold
  // neighbouring positions and write neighbouring runs
  if (warp == 2) claim();
  uint32_t U, dbits, cbits;
  {
    uint32_t id[8], rel[8], starts[8];  // id: then the delta; starts: the warp's run starts
    if (how == 1) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t k = H[128 * j + t];
        const uint32_t kp = (j == 0 && t == 0) ? k : H[128 * j + t - 1];
        rel[j] = sm.R[point_of_rank(k & 1023u)];
        if (j == 0 && t == 0) sm.first = k >> 10;
        id[j] = (k >> 10) - (kp >> 10);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t p = 128u * j + t, pp = p == 0u ? 0u : p - 1u;
        const uint32_t r = (uint32_t)ranks[p], k = how == 2 ? H[p] : S[rx(r)];
        const uint32_t kp = how == 2 ? H[pp] : S[rx((uint32_t)ranks[pp])];
        rel[j] = sm.R[point_of_rank(r)];
        if (p == 0u) sm.first = k;
        id[j] = k - kp;
        if (p >= nvalid) {  // past the end: no run; relative positions all ones (:197)
          id[j] = 0u;
          rel[j] = FULL;
        }
      }
    }
    uint32_t dor = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dor |= id[j];
      starts[j] = __ballot_sync(FULL, id[j] != 0u || (j == 0 && t == 0));
    }
    dor = __reduce_or_sync(FULL, dor);
    if (lane == 0) {
      *reinterpret_cast<uint4 *>(sm.seg + 8 * warp) =
          make_uint4(__popc(starts[0]), __popc(starts[1]), __popc(starts[2]), __popc(starts[3]));
      *reinterpret_cast<uint4 *>(sm.seg + 8 * warp + 4) =
          make_uint4(__popc(starts[4]), __popc(starts[5]), __popc(starts[6]), __popc(starts[7]));
      sm.dor[warp] = dor;
    }
    __syncthreads();  // run counts; the ranking's arrays have been read
    if (pending && warp == 3) look_up<T>(pa[pk.head], pk.head, sm, true, lane);
    // lane i: the runs that start in positions 32i..32i+31 (row i = 4j + warp)
    const uint32_t row = sm.seg[8 * (lane & 3) + (lane >> 2)];
    const uint32_t inc = warp_inc_scan(row, lane), exc = inc - row;
    U = __shfl_sync(FULL, inc, 31);
    const uint4 d4 = ld4(sm.dor);
    dbits = bitlen(d4.x | d4.y | d4.z | d4.w);
    const uint32_t below = (1u << lane) - 1u;
    // swizzled index of position 128j + t: rows 4j + warp, quads XORed by the row
    const uint32_t x0 = 32u * warp + (lane ^ (4u * warp));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      sm.Q[128 * j + (j & 1 ? x0 ^ 16u : x0)] = rel[j];
      const uint32_t u = __shfl_sync(FULL, exc, 4 * j + warp) + __popc(starts[j] & below);
      if ((starts[j] >> lane) & 1u) {
        const uint32_t i = sx(u);
        S[i] = 128u * j + t;
        H[i] = id[j];
      }
    }
    // the last, partly filled row of deltas ends in zeros
    if (warp == 1 && U + lane < (uint32_t)kChunk) H[sx(U + lane)] = 0u;
  }
  __syncthreads();  // run starts and deltas, the parked chunk's offset
  if (pending) {
    place_parked<T>(pa[pk.head], sm, pk.head);
    pk.head = pk.head + 1u < (uint32_t)kEncSlots ? pk.head + 1u : 0u;
    --pk.count;
  }
  // thread t takes runs 8t..8t+7
  {
    const uint32_t q0 = qoff(t >> 2, (2 * t) & 7), q1 = qoff(t >> 2, (2 * t + 1) & 7);
    uint32_t st[9];
    {
      const uint4 u0 = ld4(S + q0), u1 = ld4(S + q1);
      st[0] = u0.x; st[1] = u0.y; st[2] = u0.z; st[3] = u0.w;
      st[4] = u1.x; st[5] = u1.y; st[6] = u1.z; st[7] = u1.w;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) st[j] = 8u * t + j < U ? st[j] : nvalid;
    st[8] = __shfl_down_sync(FULL, st[0], 1);
    if (lane == 31) st[8] = 8u * t + 8u < U ? S[sx(8u * t + 8u)] : nvalid;
    uint32_t cm = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      st[j] = st[j + 1] - st[j];  // run length (0 past the last run)
      cm = max(cm, st[j]);
    }
    *reinterpret_cast<uint4 *>(sm.R + q0) = make_uint4(st[0], st[1], st[2], st[3]);
    *reinterpret_cast<uint4 *>(sm.R + q1) = make_uint4(st[4], st[5], st[6], st[7]);
    cm = warp_max(cm);
    if (lane == 0) sm.cmax[warp] = cm;
  }
  if (warp == 2) commit();
  __syncthreads();  // run lengths, the next chunk; the parked payload is placed
  cbits = bitlen(max4(ld4(sm.cmax)));
  const uint4 r4 = ld4(sm.relor);
  const uint32_t rbits = max(bitlen(r4.x | r4.y | r4.z | r4.w), full ? 0u : 1u);  // :200-201

  // ---- 4. bit planes -> staged payload (:313-411) ----
  const uint32_t db = section_bytes(U, dbits, Tr::pad), cb = section_bytes(U, cbits, Tr::pad);
  const uint32_t rb = rel_section_bytes(rbits, Tr::pad);
  if (t == 0) {
    sm.park[(pk.head + pk.count) % (uint32_t)kEncSlots] = {c, db + cb + rb};
    publish_size(a.ctl, a.look, c, db + cb + rb);
    uint32_t *m = reinterpret_cast<uint32_t *>(a.out + Tr::hdr + 8ull * a.G + (unsigned long long)Tr::meta * c);
    if constexpr (!is64) {
      m[6] = sm.first;
      m[7] = dbits | (cbits << 16);
      m[8] = rbits | (U << 16);
    } else {
      m[12] = sm.first;
      m[13] = 0u;
      m[14] = dbits | (cbits << 16);
      m[15] = rbits | (U << 16);
    }
  }
  const uint32_t slot = (pk.head + pk.count) % (uint32_t)kEncSlots;
  ++pk.count;
  const uint32_t bpp = (U + 7u) >> 3;
  uint8_t *const stage = reinterpret_cast<uint8_t *>(sm.P[slot]);
  {
    // jobs of eight planes, the longest first
    const uint32_t nd = (dbits + 7u) >> 3, nr = (rbits + 7u) >> 3, nc = (cbits + 7u) >> 3;
    for (uint32_t j = warp; j < nd + nr + nc; j += kEncWarps) {
      if (j - nd < nr) plane_job(sm.Q, stage, db + cb, rbits, 8u * (j - nd), 0u, lane);
      else if (j < nd) plane_job(H, stage, 0u, dbits, 8u * j, bpp, lane);
      else plane_job(sm.R, stage, db, cbits, 8u * (j - nd - nr), bpp, lane);
    }
  }
  if (warp == kEncWarps - 1) {
    // section padding is zero (the reference leaves it unwritten)
    const uint32_t a0 = dbits * bpp + lane, a1 = db + cbits * bpp + lane;
    if (a0 < db) stage[a0] = 0;
    if (a1 < db + cb) stage[a1] = 0;
  }
  return slot;
}

// Places what is parked when the work has run out.
template <typename T, class PArgs>
__device__ __forceinline__ void flush_parked(const PArgs &pa, EncShared &sm, Parked &pk, int lane, int warp) {
  for (; pk.count != 0u; --pk.count) {
    __syncthreads();
    if (warp == 0) look_up<T>(pa[pk.head], pk.head, sm, true, lane);
    __syncthreads();
    place_parked<T>(pa[pk.head], sm, pk.head);
    pk.head = pk.head + 1u < (uint32_t)kEncSlots ? pk.head + 1u : 0u;
  }
}

// The arguments of a parked chunk, when all chunks share them.
template <typename T>
struct SameArgs {
  const CArgs<T> &a;
  __device__ __forceinline__ const CArgs<T> &operator[](uint32_t) const { return a; }
};

// Persistent compress kernel: every CTA claims one chunk after another.  A
// chunk's payload size is published as soon as its runs are known and its
// payload stays parked in shared memory; the CTA looks up its stream offset
// (decoupled look-back) an iteration later without waiting, and waits for a
// predecessor only when the room is needed for the next payload.
template <typename T, int DIM>
__global__ void __launch_bounds__(kEncThreads, kEncCtas) compress_kernel(const __grid_constant__ CArgs<T> a) {
  constexpr bool is64 = sizeof(T) == 8;
  extern __shared__ __align__(16) unsigned char enc_smem[];
  EncShared &sm = *reinterpret_cast<EncShared *>(enc_smem);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  Control *ctl = a.ctl;
  const uint32_t seg = ctl->seg;
  const T eb = a.eb_dev ? (T)*a.eb_dev : a.eb;
  const T inv = is64 ? (T)__ddiv_rn(1.0, __dmul_rn(2.0, (double)eb)) : (T)__fdiv_rn(1.0f, __fmul_rn(2.0f, (float)eb));
  const unsigned long long G = a.G;
  // nothing is claimed after a failure (sampling, bound, another CTA's)
  if (t == 0) {
    sm.overflowed = nullptr;
    sm.next[0] = ld_volatile(reinterpret_cast<const uint32_t *>(&ctl->status)) != 0u
                     ? G
                     : (unsigned long long)atomicAdd(&ctl->chunk_ctr, 1u);
  }
  __syncthreads();
  Parked pk = {0u, 0u};
  uint32_t rank_skip = 0, declined = 0, claimed = 0;
  int par = 0;
  for (;;) {
    const unsigned long long c = sm.next[par];
    if (c >= G) break;
    encode_chunk<T, DIM>(
        a, c, sm, par, seg, eb, inv, SameArgs<T>{a}, pk, rank_skip, declined,
        [&]() {
          if (lane == 0) claimed = ld_volatile(&ctl->abort) ? 0xFFFFFFFFu : atomicAdd(&ctl->chunk_ctr, 1u);
        },
        [&]() {
          claimed = __shfl_sync(0xFFFFFFFFu, claimed, 0);
          if (lane == 0) sm.next[par ^ 1] = claimed;
          prefetch_points<T, DIM>(a, claimed, lane);
        });
    par ^= 1;
  }
  flush_parked<T>(SameArgs<T>{a}, sm, pk, lane, warp);
  rewind_work_counter(ctl);
}

}  // namespace gpzb
