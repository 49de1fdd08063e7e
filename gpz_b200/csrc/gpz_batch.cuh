// gpz_batch.cuh -- batched compress: many snapshots of one (float type,
// dimension) class in one persistent launch.
//
// The reference compresses one snapshot per call (CompressorManager::compressWarp,
// src/CompressorManager.cpp:12-16), so a workload of many small snapshots is
// dominated by per-call launches, syncs and an almost idle GPU.  Here every
// snapshot keeps its own stream, control block and look-back records; the
// chunks of all snapshots of a class form one global work list (snapshot
// after snapshot, so each snapshot's chunks are claimed in order), and one
// persistent kernel per class claims them.  A snapshot's stream is
// byte-identical to the one gpz_compress writes for it: the per-chunk
// encoder, the placement and the header/meta writes are the same code.
#pragma once

#include "gpz_kernels.cuh"
#include "gpz_encode.cuh"
#include "gpz_decode.cuh"

namespace gpzb {

constexpr uint32_t kBatchSegFixed = 1u;  // the segment size is given (no sampling)
constexpr uint32_t kBatchSafe31 = 2u;    // GPZ_FLAG_SAFE31 rules for the automatic segment size
constexpr uint32_t kBatchRelDev = 4u;    // absolute bound computed on the device from rel_eb
constexpr uint32_t kBatchRelMode = 8u;   // the automatic segment size follows the relative-bound rules
constexpr int kBatchLocalBits = 40;      // decompress map entry: item << 40 | chunk within the item

// One snapshot of a batch.  `a` is what the single-stream kernel gets as its
// parameter; a.eb is rewritten on the device when kBatchRelDev is set.
template <typename T>
struct BItem {
  CArgs<T> a;
  unsigned long long start;  // first chunk of the snapshot in the class's work list
  T rel_eb;
  uint32_t seg;      // segment size resolved by the sampling kernel (0: it failed)
  uint32_t seg_in;
  uint32_t flags;
};

// computeSegSize for every snapshot of the class (blockIdx.y = snapshot, 128
// blocks each), or the given segment size.
template <typename T>
__global__ void __launch_bounds__(256) batch_sample_kernel(BItem<T> *items) {
  BItem<T> &it = items[blockIdx.y];
  if (it.flags & kBatchSegFixed) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      it.a.ctl->seg = it.seg_in;
      it.a.ctl->adjusted = 0;
      it.seg = it.seg_in;
    }
    return;
  }
  seg_sample_block<T>(it.a.x, it.a.y, it.a.z, it.a.n, it.a.dim, it.seg_in, (it.flags & kBatchRelMode) ? 1 : 0, it.rel_eb, it.a.eb,
                      (it.flags & kBatchSafe31) ? 1 : 0, it.a.ctl, blockIdx.x, gridDim.x, nullptr, &it.seg);
}

// A CTA's view of the work list: the chunk of the current and of the next
// iteration (by parity), with their snapshots' arguments, and the parked
// payloads' arguments by slot.
template <typename T>
struct BatchState {
  CArgs<T> args[2];
  CArgs<T> parked[kEncSlots];
  unsigned long long chunk[2];  // chunk within the snapshot (>= G: past the list's end)
  uint32_t seg[2];
};

// One warp copies a snapshot's arguments.
template <typename T>
__device__ __forceinline__ void copy_args(CArgs<T> &dst, const CArgs<T> &src, int lane) {
  constexpr int W = (int)(sizeof(CArgs<T>) / 4);
  static_assert(sizeof(CArgs<T>) % 4 == 0 && W <= 32, "one word per lane");
  if (lane < W) reinterpret_cast<uint32_t *>(&dst)[lane] = reinterpret_cast<const uint32_t *>(&src)[lane];
}

// The last of the K snapshots whose first chunk is at or below g (a warp
// probes 32 of them per step).
template <typename T>
__device__ __forceinline__ uint32_t find_item(const BItem<T> *items, uint32_t K, unsigned long long g, int lane) {
  uint32_t lo = 0, len = K;
  while (len > 1) {
    const uint32_t step = (len + 31) / 32, i = lo + lane * step;
    const bool in = lane * step < len && items[i].start <= g;
    const int top = 31 - __clz((int)__ballot_sync(0xFFFFFFFFu, in));  // lane 0 always holds
    len = min(step, len - top * step);
    lo += top * step;
  }
  return lo;
}

// The compress loop of compress_kernel over the chunks of many snapshots.  A
// snapshot whose segment size could not be chosen (sampling error, status
// set) is skipped as a whole.
template <typename T, int DIM>
__global__ void __launch_bounds__(kEncThreads, kEncCtas)
    compress_batch_kernel(const BItem<T> *items, uint32_t K, unsigned long long total, unsigned long long *claim) {
  constexpr bool is64 = sizeof(T) == 8;
  extern __shared__ __align__(16) unsigned char enc_smem[];
  EncShared &sm = *reinterpret_cast<EncShared *>(enc_smem);
  __shared__ BatchState<T> bs;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned long long claimed = 0;
  auto claim_next = [&]() {  // one warp
    if (lane == 0) claimed = atomicAdd(claim, 1ull);
  };
  auto fetch = [&](int slot) {  // the same warp, later
    const unsigned long long g = __shfl_sync(0xFFFFFFFFu, claimed, 0);
    if (lane == 0) sm.next[slot] = g;
    if (g >= total) return;
    const BItem<T> &it = items[find_item(items, K, g, lane)];
    copy_args(bs.args[slot], it.a, lane);
    if (lane == 0) {
      bs.chunk[slot] = g - it.start;
      bs.seg[slot] = it.seg;
    }
    prefetch_points<T, DIM>(it.a, g - it.start, lane);
  };
  if (t == 0) sm.overflowed = nullptr;
  if (warp == 2) {
    claim_next();
    fetch(0);
  }
  __syncthreads();
  Parked pk = {0u, 0u};
  uint32_t rank_skip = 0, declined = 0;
  int par = 0;
  for (;;) {
    if (sm.next[par] >= total) break;
    const unsigned long long c = bs.chunk[par];
    const uint32_t seg = bs.seg[par];
    if (seg == 0u) {  // the snapshot's sampling failed
      __syncthreads();
      if (warp == 2) {
        claim_next();
        fetch(par ^ 1);
      }
      __syncthreads();
      par ^= 1;
      continue;
    }
    const CArgs<T> &a = bs.args[par];
    const T eb = a.eb;
    const T inv = is64 ? (T)__ddiv_rn(1.0, __dmul_rn(2.0, (double)eb)) : (T)__fdiv_rn(1.0f, __fmul_rn(2.0f, (float)eb));
    const uint32_t slot = encode_chunk<T, DIM>(a, c, sm, par, seg, eb, inv, bs.parked, pk, rank_skip, declined, claim_next,
                                               [&]() { fetch(par ^ 1); });
    // every look-up of this payload comes behind the next chunk's first barrier
    // or the flush's
    if (warp == 0) copy_args(bs.parked[slot], a, lane);
    par ^= 1;
  }
  flush_parked<T>(bs.parked, sm, pk, lane, warp);
}

// ---------------------------------------------------------------------------
// Batched decompress.
// ---------------------------------------------------------------------------

// One stream of a decompress batch; n is the point count the caller read
// from the stream's header (the work map is built from it); G, pay_base, eb,
// seg and ok come from the device-side header check.
template <typename T>
struct DItem {
  DArgs<T> a;
  unsigned long long n, G, pay_base;
  T eb;
  uint32_t seg;
  int32_t ok;
};

// The header checks of decompress_kernel, once per stream (one thread each).
template <typename T, int DIM>
__global__ void dbatch_header_kernel(DItem<T> *items, uint32_t K) {
  using Tr = TT<T>;
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  DItem<T> &it = items[k];
  it.ok = 0;
  Control *ctl = it.a.ctl;
  if (it.a.bytes < Tr::hdr) { set_status(ctl, kESTREAM); return; }
  const uint8_t *s = it.a.s;
  const uint32_t dim = *reinterpret_cast<const uint32_t *>(s);
  unsigned long long n;
  memcpy(&n, s + 4, 8);
  const uint32_t bits = *reinterpret_cast<const uint32_t *>(s + 12);
  T eb;
  memcpy(&eb, s + 16, sizeof(T));
  const uint32_t seg = *reinterpret_cast<const uint32_t *>(s + 16 + sizeof(T));
  const unsigned long long G = (n + kChunk - 1) / kChunk;
  if (bits != Tr::bits || dim != (uint32_t)DIM || n == 0 || n != it.n || seg == 0 ||
      G > (it.a.bytes - Tr::hdr) / (8ull + Tr::meta)) {
    set_status(ctl, kESTREAM);
    return;
  }
  if (n > it.a.cap) { set_status(ctl, kENOSPACE); return; }
  it.G = G;
  it.pay_base = Tr::hdr + 8ull * G + (unsigned long long)Tr::meta * G;
  it.eb = eb;
  it.seg = seg;
  it.ok = 1;
}

// decompress_kernel over the chunks of many streams: warps stride over the
// global chunk list, cmap[c] = stream << 40 | chunk within the stream.  The
// passes are decompress_kernel's: float64 classes run the fast pass in the
// 12 KB layout, then the general pass, which skips every stream whose fast
// pass left no chunk.
template <typename T, int DIM, class Cfg = DecCfg<T>, int PASS = kPassAll>
__global__ void __launch_bounds__(32 * Cfg::warps, Cfg::min_ctas)
    decompress_batch_kernel(const DItem<T> *__restrict__ items, const unsigned long long *__restrict__ cmap,
                            unsigned long long total) {
  constexpr int W = Cfg::warps;
  constexpr unsigned long long kLocal = (1ull << kBatchLocalBits) - 1;
  extern __shared__ __align__(16) uint32_t dec_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *const sw = dec_smem + warp * Cfg::words;
  const unsigned long long nwarps = (unsigned long long)gridDim.x * W;
  for (unsigned long long gc = (unsigned long long)blockIdx.x * W + warp; gc < total; gc += nwarps) {
    const unsigned long long m = cmap[gc];
    const DItem<T> &it = items[m >> kBatchLocalBits];
    if (!it.ok) continue;
    if (PASS == kPassGeneral && ld_volatile(&it.a.ctl->deferred) == 0u) continue;
    const DArgs<T> a = it.a;
    const unsigned long long c = m & kLocal, G = it.G;
    const uint32_t seg = it.seg;
    ChunkGeom g;
    g.seg = seg;
    g.sh = (uint32_t)__ffs((int)seg) - 1u;
    g.msk = seg - 1u;
    const uint32_t mwc = dec_meta_word<T>(a.s, G, c, lane);
    decode_chunk<T, DIM, Cfg, PASS>(a, c, it.n, G, it.pay_base, it.eb, seg, g, mwc, sw, lane);
  }
}

}  // namespace gpzb
