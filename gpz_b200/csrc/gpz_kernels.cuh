// gpz_kernels.cuh -- sm_100a kernels of the B200 GPZ codec.
//
//   seg_sample_kernel   computeSegSize (reference src/cudaWarpCompress.cu:1424-1557)
//   rel_to_abs_kernel   findMinimumValues + convertRelEb (include/utils.cuh:44-65,
//                       src/main.cpp:35-55), on the device
//   (compress_kernel: gpz_encode.cuh; decompress_kernel: gpz_decode.cuh)
//
// float64 twins: src/cudaWarpCompressDouble.cu (same line ranges +/- 3).
#pragma once

#include <cfloat>
#include "gpz_device.cuh"

namespace gpzb {

// ===========================================================================
// Automatic segment size (computeSegSize).
// ===========================================================================
// Correctly rounded scalar operations, the same on the device and on the host
// (the host build uses plain IEEE operations with contraction off).
template <typename T> struct Rn;
template <> struct Rn<float> {
  __host__ __device__ static float add(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
  }
  __host__ __device__ static float sub(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
  }
  __host__ __device__ static float mul(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
  }
  __host__ __device__ static float div(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdiv_rn(a, b);
#else
    return a / b;
#endif
  }
  __host__ __device__ static float sqrt(float a) {
#ifdef __CUDA_ARCH__
    return __fsqrt_rn(a);
#else
    return sqrtf(a);
#endif
  }
  __host__ __device__ static float from_u32(uint32_t v) {
#ifdef __CUDA_ARCH__
    return __uint2float_rn(v);
#else
    return (float)v;
#endif
  }
  // truncation with saturation (cvt.rzi.sat.u64), NaN -> 0
  __host__ __device__ static unsigned long long to_u64_rz(float v) {
#ifdef __CUDA_ARCH__
    return __float2ull_rz(v);
#else
    if (!(v > 0.0f)) return 0ull;
    if (v >= 18446744073709551616.0f) return ~0ull;
    return (unsigned long long)v;
#endif
  }
};
template <> struct Rn<double> {
  __host__ __device__ static double add(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
  }
  __host__ __device__ static double sub(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
  }
  __host__ __device__ static double mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
  }
  __host__ __device__ static double div(double a, double b) {
#ifdef __CUDA_ARCH__
    return __ddiv_rn(a, b);
#else
    return a / b;
#endif
  }
  __host__ __device__ static double sqrt(double a) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(a);
#else
    return ::sqrt(a);
#endif
  }
  __host__ __device__ static double from_u32(uint32_t v) {
#ifdef __CUDA_ARCH__
    return __uint2double_rn(v);
#else
    return (double)v;
#endif
  }
  __host__ __device__ static unsigned long long to_u64_rz(double v) {
#ifdef __CUDA_ARCH__
    return __double2ull_rz(v);
#else
    if (!(v > 0.0)) return 0ull;
    if (v >= 18446744073709551616.0) return ~0ull;
    return (unsigned long long)v;
#endif
  }
};

// Outcome of the automatic segment-size rules.
struct SegDecision {
  int status;         // kOK, kEINVAL (no segment size in abs mode) or kESEG
  uint32_t seg, adjusted;
};

// Host arithmetic of computeSegSize (src/cudaWarpCompress.cu:1488-1554; double
// twin src/cudaWarpCompressDouble.cu:1488-1553) on the sampled per-axis
// min/max mm = (x, y, z minima, x, y, z maxima).  float: the 2D variance
// divides by 2 (:1503) and seg doubles (<= 11 times) while the block count
// would exceed UINT32_MAX; double: variance divides by 3 and the reference's
// guard compares with UINT64_MAX and never fires.  With safe31 both double
// until every id fits 31 bits.  Evaluated the same on the device (sampling
// kernel) and on the host (sharded compress).
template <typename T>
__host__ __device__ SegDecision decide_seg(const T mm[6], uint32_t dim, uint32_t seg_in, int rel_mode, T rel_eb, T eb,
                                           int safe31) {
  using R = Rn<T>;
  constexpr bool is64 = sizeof(T) == 8;
  const T dx = R::sub(mm[3], mm[0]), dy = R::sub(mm[4], mm[1]), dz = R::sub(mm[5], mm[2]);
  const T mean = R::div(R::add(R::add(dx, dy), dz), (T)3);
  const T ex = R::sub(dx, mean), ey = R::sub(dy, mean), ez = R::sub(dz, mean);
  T var = R::add(R::add(R::mul(ex, ex), R::mul(ey, ey)), R::mul(ez, ez));
  var = R::div(var, (!is64 && dim == 2) ? (T)2 : (T)3);
  const T ratio = R::div(R::sqrt(var), mean);
  const T maxr3 = is64 ? (T)fmax(fmax((double)dx, (double)dy), (double)dz) : (T)fmaxf(fmaxf((float)dx, (float)dy), (float)dz);
  uint32_t seg = seg_in;
  if (seg == 0 && rel_mode) {
    if (ratio < (T)0.1f) seg = ((double)rel_eb <= 1e-4) ? 32u : 2u;
    else seg = ((double)rel_eb <= 1e-4) ? 4u : 1u;
  }
  if (seg == 0) return {kEINVAL, 0u, 0u};
  const bool guard = !is64 || safe31;
  if (!guard) return {kOK, seg, 0u};
  const unsigned long long limit = safe31 ? 0x7FFFFFFFull : 0xFFFFFFFFull;
  auto total = [&](uint32_t s) {
    const T q = R::div(maxr3, R::mul(R::from_u32(2u * s), eb));
    const T c = is64 ? (T)::ceil((double)q) : (T)::ceilf((float)q);
    const unsigned long long mb = R::to_u64_rz(c) + 1ull;
    return dim == 3 ? mb * mb * mb : mb * mb;
  };
  if (total(seg) <= limit) return {kOK, seg, 0u};
  uint32_t t = seg;
  for (int i = 0; i < 11; ++i) {
    t *= 2u;
    if (total(t) <= limit) break;
  }
  if (t > 1024u) return {kESEG, 0u, 0u};
  return {kOK, t, 1u};
}

template <typename T>
__device__ __forceinline__ void fold_minmax(T v, typename TT<T>::U &mn_inv, typename TT<T>::U &mx) {
  if (v == v) {
    const typename TT<T>::U o = ord_of(v);
    mn_inv = max(mn_inv, (typename TT<T>::U)~o);
    mx = max(mx, o);
  }
}

// Strict-bound mode (an extension; the reference holds eb only up to the
// rounding of its reconstruction, which its verifier hides with a 1.01*eb
// slack, src/utils.cu:28).  For a snapshot whose coordinates satisfy |x| <= M
// and whose per-axis ranges are at most R, every finite point reconstructs
// within eb when the stream is encoded with
//   eb' = eb - u * (3 R + 2 M + 4 eb),   u = 2^-24 (float) / 2^-53 (double),
// rounded down.  With t = (x - m) / (2 eb') (m the chunk minimum, 0 <= x - m
// <= R), inv = fl(1/(2 eb')) = (1 + d1) / (2 eb'), nmn = fl(-m inv) and
// qf = fl(x inv + nmn), |qf - t| <= u (2 t + |m| inv) + O(u^2): truncation
// leaves x within eb' + u (2R + M) of the center m + (2q+1) eb' of its bin.
// The decoder's fused multiply-add rounds the center once, by at most
// u (M + eb'), and its conversion of 2q+1 (<= R/eb' + 1) to T by at most
// u (R + eb') eb'/eb' when 2q+1 needs more than the mantissa:
//   |x - v| <= eb' + u (3R + 2M + 2 eb') + O(u^2) < eb.
// Returns 0 when no positive eb' exists.
template <typename T>
__host__ __device__ inline T strict_bound(T eb, double max_abs, double max_range) {
  const double u = sizeof(T) == 4 ? 5.9604644775390625e-08 : 1.1102230246251565e-16;
  const double e = (double)eb - u * (3.0 * max_range + 2.0 * max_abs + 4.0 * (double)eb);
  if (!(e > 0.0)) return (T)0;
  T r = (T)e;
  if ((double)r > e) r = sizeof(T) == 4 ? (T)nextafterf((float)r, 0.0f) : (T)nextafter((double)r, 0.0);
  return r;
}

// ---------------------------------------------------------------------------
// One axis of a grid-wide min / max: block `block` of `nblocks` folds its share
// of p[0..n) into the thread's accumulators (ordered values, the minimum
// inverted; NaNs ignored, -0 below +0).
//
// A pure read, bound by HBM: every thread keeps kFoldUnroll 16-byte loads in
// flight (64 bytes; 6 blocks of 256 threads per SM hold 96 KB in flight, 2.7
// times what 6.5 TB/s needs at ~800 ns), and a float axis is folded with
// three-input min / max, half an instruction per value each.  rel_to_abs on
// 143,735,721 float 3D points: 2.33 ms with one scalar load per thread, axis
// and iteration (0.74 TB/s), 0.261 ms so (6.6 TB/s); on 50M double 3D points
// 0.853 -> 0.222 ms (5.4 TB/s, 64-bit integer compares).
// ---------------------------------------------------------------------------
constexpr int kFoldUnroll = 4;

template <typename T>
__device__ __forceinline__ void fold_vec(const uint4 (&v)[kFoldUnroll], T &mnf, T &mxf, typename TT<T>::U &mn_inv,
                                         typename TT<T>::U &mx) {
#pragma unroll
  for (int u = 0; u < kFoldUnroll; ++u) {
    if constexpr (sizeof(T) == 4) {
      const float a = __uint_as_float(v[u].x), b = __uint_as_float(v[u].y), c = __uint_as_float(v[u].z),
                  d = __uint_as_float(v[u].w);
      mnf = fmin3f(fmin3f(mnf, a, b), c, d);
      mxf = fmax3f(fmax3f(mxf, a, b), c, d);
    } else {
      fold_minmax<T>((T)__hiloint2double((int)v[u].y, (int)v[u].x), mn_inv, mx);
      fold_minmax<T>((T)__hiloint2double((int)v[u].w, (int)v[u].z), mn_inv, mx);
    }
  }
}

template <typename T>
__device__ __forceinline__ void fold_axis(const T *__restrict__ p, unsigned long long n, unsigned block,
                                          unsigned nblocks, typename TT<T>::U &mn_inv, typename TT<T>::U &mx) {
  constexpr unsigned EPV = 16 / sizeof(T);  // elements per 16-byte load
  // elements before the first 16-byte boundary, and after the last whole vector
  const unsigned long long head = min(n, (unsigned long long)(((16u - ((uintptr_t)p & 15u)) & 15u) / sizeof(T)));
  const unsigned long long nv = (n - head) / EPV;
  const uint4 *pv = reinterpret_cast<const uint4 *>(p + head);
  T mnf = (T)INFINITY, mxf = (T)-INFINITY;  // float accumulators (unused for double)
  const unsigned nt = blockDim.x;
  const unsigned long long span = (unsigned long long)nt * kFoldUnroll;
  for (unsigned long long i = block * span + threadIdx.x; i < nv; i += nblocks * span) {
    uint4 v[kFoldUnroll];
    if (i + (kFoldUnroll - 1) * nt < nv) {
#pragma unroll
      for (int u = 0; u < kFoldUnroll; ++u) v[u] = __ldg(pv + i + (unsigned long long)u * nt);
    } else {
      // the ragged end: a slot past it repeats the thread's first vector
#pragma unroll
      for (int u = 0; u < kFoldUnroll; ++u) v[u] = __ldg(pv + (i + (unsigned long long)u * nt < nv ? i + (unsigned long long)u * nt : i));
    }
    fold_vec<T>(v, mnf, mxf, mn_inv, mx);
  }
  if (block == 0) {  // fewer than 2 * EPV elements
    if (threadIdx.x < head) fold_minmax<T>(p[threadIdx.x], mn_inv, mx);
    const unsigned long long tail = head + nv * EPV + threadIdx.x;
    if (threadIdx.x < EPV && tail < n) fold_minmax<T>(p[tail], mn_inv, mx);
  }
  if constexpr (sizeof(T) == 4) {
    // a thread that saw no number (all NaN, or nothing) keeps min > max
    if (mnf <= mxf) {
      mn_inv = max(mn_inv, (typename TT<T>::U)~ord_of(mnf));
      mx = max(mx, ord_of(mxf));
    }
  }
}

// The strict bound of a snapshot (strict_bound above with its largest
// coordinate magnitude and largest per-axis range, NaNs ignored), into
// ctl->strict_eb; kEINVAL in ctl->status when there is none.  Grid-stride;
// the last block decides.
template <typename T>
__global__ void __launch_bounds__(256, 6) strict_bound_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                           const T *__restrict__ z, uint64_t n, uint32_t dim, T eb,
                                                           Control *ctl) {
  using U = typename TT<T>::U;
  __shared__ U red[6][8];
  __shared__ int last;
  U acc[6] = {0, 0, 0, 0, 0, 0};  // [min_inv, max] per axis
  fold_axis<T>(x, n, blockIdx.x, gridDim.x, acc[0], acc[1]);
  fold_axis<T>(y, n, blockIdx.x, gridDim.x, acc[2], acc[3]);
  if (dim == 3) fold_axis<T>(z, n, blockIdx.x, gridDim.x, acc[4], acc[5]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const U v = warp_max(acc[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 2 * dim) {
    U v = 0;
    for (int w = 0; w < 8; ++w) v = max(v, red[threadIdx.x][w]);
    atomicMax(&ctl->mm[threadIdx.x], (unsigned long long)v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&ctl->sample_done, 1u) == gridDim.x - 1);
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    double M = 0.0, R = 0.0;
    for (uint32_t d = 0; d < dim; ++d) {
      const U mi = (U)~(U)((volatile unsigned long long *)ctl->mm)[2 * d];
      const U ma = (U)((volatile unsigned long long *)ctl->mm)[2 * d + 1];
      if (ma == 0) continue;  // no finite value on this axis
      const double lo = (double)from_ord(mi), hi = (double)from_ord(ma);
      M = fmax(M, fmax(fabs(lo), fabs(hi)));
      R = fmax(R, hi - lo);
    }
    const T e = strict_bound<T>(eb, M, R);
    if (!(e > (T)0)) set_status(ctl, kEINVAL);
    ctl->strict_eb = (double)e;
    // the sampling kernel that follows reuses these accumulators
    for (int k = 0; k < 6; ++k) ctl->mm[k] = 0;
    ctl->sample_done = 0;
  }
}

// The segment-size rules on the sampled accumulators ([min inverted, max] per
// axis) and their outcome in the control block (one thread).
template <typename T>
__device__ __forceinline__ void store_decision(const typename TT<T>::U (&acc)[6], uint32_t dim, uint32_t seg_in,
                                               int rel_mode, T rel_eb, T ebv, int safe31, Control *ctl,
                                               uint32_t *seg_out) {
  using U = typename TT<T>::U;
  T mm[6];
#pragma unroll
  for (uint32_t d = 0; d < 3; ++d) {
    mm[d] = d < dim ? from_ord((U)~acc[2 * d]) : (T)0;
    mm[3 + d] = d < dim ? from_ord(acc[2 * d + 1]) : (T)0;
  }
  const SegDecision sd = decide_seg<T>(mm, dim, seg_in, rel_mode, rel_eb, ebv, safe31);
  if (seg_out) *seg_out = sd.status == kOK ? sd.seg : 0u;
  if (sd.status != kOK) set_status(ctl, sd.status);
  else {
    ctl->seg = sd.seg;
    ctl->adjusted = sd.adjusted;
  }
}

// sampleMinMaxXYZKernel[2D] + reduceMinMax[2D] (src/cudaWarpCompress.cu:1216-1418):
// 1024 windows of 256 consecutive points at stride max((N-256)/1024, 1).
// A window that would run past N is skipped by the reference and its
// min/max slot keeps the zero-filled scratch value, so it contributes 0.0.
// Launch: 128 blocks x 256 threads, 8 windows per block.  The last block to
// finish applies the host decision rules (decide_seg).
// One block's share (8 windows) of the sampling; `block` of `nblocks`
// (128 blocks cover the 1024 windows).
template <typename T>
__device__ __forceinline__ void seg_sample_block(const T *__restrict__ x, const T *__restrict__ y,
                                                 const T *__restrict__ z, uint64_t n, uint32_t dim, uint32_t seg_in,
                                                 int rel_mode, T rel_eb, T eb, int safe31, Control *ctl,
                                                 unsigned block, unsigned nblocks, const double *eb_dev = nullptr,
                                                 uint32_t *seg_out = nullptr) {
  using U = typename TT<T>::U;
  __shared__ U red[6][8];
  __shared__ int last;
  const unsigned long long L = 256, B = 1024;
  const unsigned long long stride = max((n - L) / B, 1ull);
  U acc[6] = {0, 0, 0, 0, 0, 0};  // [min_inv, max] per axis
  // the thread's point of all 8 windows on all axes is in flight at once: the
  // kernel is one load latency long, not eight (18.7 -> 6.2 us on the
  // 143.7M-point snapshot, 8.5 -> 4.3 us on 5,003 points); a window past the
  // end gives 0
  const T *X[3] = {x, y, z};
  T v[3][8];
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const unsigned long long st = ((unsigned long long)block * 8 + w) * stride;
    const bool in = st + L <= n;
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d][w] = in && d < (int)dim ? X[d][st + threadIdx.x] : (T)0;
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
    if (d < (int)dim) {
#pragma unroll
      for (int w = 0; w < 8; ++w) fold_minmax<T>(v[d][w], acc[2 * d], acc[2 * d + 1]);
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const U v = warp_max(acc[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 2 * dim) {
    U v = 0;
    for (int w = 0; w < 8; ++w) v = max(v, red[threadIdx.x][w]);
    atomicMax(&ctl->mm[threadIdx.x], (unsigned long long)v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&ctl->sample_done, 1u) == nblocks - 1);
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    U all[6];
    for (uint32_t k = 0; k < 6; ++k) all[k] = (U)((volatile unsigned long long *)ctl->mm)[k];
    const T ebv = eb_dev ? (T)*(const volatile double *)eb_dev : eb;
    store_decision<T>(all, dim, seg_in, rel_mode, rel_eb, ebv, safe31, ctl, seg_out);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) seg_sample_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                         const T *__restrict__ z, uint64_t n, uint32_t dim,
                                                         uint32_t seg_in, int rel_mode, T rel_eb, T eb,
                                                         int safe31, Control *ctl, const double *eb_dev) {
  if (eb_dev && ld_volatile(reinterpret_cast<const uint32_t *>(&ctl->status)) != 0) return;
  seg_sample_block<T>(x, y, z, n, dim, seg_in, rel_mode, rel_eb, eb, safe31, ctl, blockIdx.x, gridDim.x, eb_dev);
}

// Per-axis accumulators of a 1024-thread block's values, in every thread of the
// first warp (lane k: accumulator k).
template <typename U>
__device__ __forceinline__ U block_max6(const U (&acc)[6], U (*red)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const U v = warp_max(acc[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  U mine = 0;
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const U v = warp_max(red[k][lane]);
      if (lane == k) mine = v;
    }
  }
  return mine;
}

// Snapshots of up to this many points take one block for what surrounds the
// compress kernel (their look-back records all lie in the control block): the
// clearing memset, the cross-block atomics and the last-block election go.
constexpr uint64_t kSmallPoints = 16384;

// seg_sample_kernel of a small snapshot, in one block that clears the control
// block first.  Its windows overlap (stride <= 15), so they are one span of
// the array, read once.  5,003 float points: 81 -> 77 us for the whole call
// (with rel_to_abs_small_kernel) against a memset and 128 blocks.
template <typename T>
__global__ void __launch_bounds__(1024) seg_small_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                         const T *__restrict__ z, uint64_t n, uint32_t dim,
                                                         uint32_t seg_in, int rel_mode, T rel_eb, T eb, int safe31,
                                                         Control *ctl) {
  using U = typename TT<T>::U;
  __shared__ U red[6][32];
  if (threadIdx.x < kCtlBytes / 4) reinterpret_cast<uint32_t *>(ctl)[threadIdx.x] = 0u;
  const uint64_t L = 256, B = 1024;
  // windows inside the array, and the end of the last of them
  const uint64_t stride = n >= L ? max((n - L) / B, (uint64_t)1) : 1, inside = n >= L ? min(B, (n - L) / stride + 1) : 0;
  const uint64_t end = inside ? (inside - 1) * stride + L : 0;
  U acc[6] = {0, 0, 0, 0, 0, 0};
  if (inside < B) {  // the others contribute 0
#pragma unroll
    for (int d = 0; d < 3; ++d) fold_minmax<T>((T)0, acc[2 * d], acc[2 * d + 1]);
  }
  fold_axis<T>(x, end, 0, 1, acc[0], acc[1]);
  fold_axis<T>(y, end, 0, 1, acc[2], acc[3]);
  if (dim == 3) fold_axis<T>(z, end, 0, 1, acc[4], acc[5]);
  const U mine = block_max6(acc, red);  // its barrier also orders the clearing before the result
  if (threadIdx.x < 32) {
    U all[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) all[k] = __shfl_sync(0xFFFFFFFFu, mine, k);
    if (threadIdx.x == 0) store_decision<T>(all, dim, seg_in, rel_mode, rel_eb, eb, safe31, ctl, nullptr);
  }
}

// The sampling windows of computeSegSize restricted to one shard
// [begin, begin + count) of a larger array (pointers start at `begin`): folds
// the shard's share of every window into ctl->mm (windows past n contribute
// 0.0, as in seg_sample_kernel).  Combining the shards' accumulators with an
// unsigned max gives exactly the whole array's.
template <typename T>
__global__ void __launch_bounds__(256) seg_sample_shard_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                               const T *__restrict__ z, uint64_t n, uint64_t begin,
                                                               uint64_t count, uint32_t dim, Control *ctl) {
  using U = typename TT<T>::U;
  __shared__ U red[6][8];
  const unsigned long long L = 256, B = 1024;
  const unsigned long long stride = max((n - L) / B, 1ull);
  U acc[6] = {0, 0, 0, 0, 0, 0};
  const T *X[3] = {x, y, z};
  for (int w = 0; w < 8; ++w) {
    const unsigned long long win = (unsigned long long)blockIdx.x * 8 + w;
    const unsigned long long st = win * stride;
    if (st + L > n) {
      for (uint32_t d = 0; d < dim; ++d) fold_minmax<T>((T)0, acc[2 * d], acc[2 * d + 1]);
      continue;
    }
    const unsigned long long p = st + threadIdx.x;
    if (p >= begin && p - begin < count)
      for (uint32_t d = 0; d < dim; ++d) fold_minmax<T>(X[d][p - begin], acc[2 * d], acc[2 * d + 1]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const U v = warp_max(acc[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 2 * dim) {
    U v = 0;
    for (int w = 0; w < 8; ++w) v = max(v, red[threadIdx.x][w]);
    atomicMax(&ctl->mm[threadIdx.x], (unsigned long long)v);
  }
}

// The segment size chosen by the caller is used as is (sharded compress).
static __global__ void set_seg_kernel(Control *ctl, uint32_t seg) {
  ctl->seg = seg;
  ctl->adjusted = 0;
}

// The bound and the min / max from the accumulators ([min inverted, max] per
// axis), one thread.
template <typename T>
__device__ __forceinline__ void store_rel_bound(const typename TT<T>::U (&acc)[6], T rel, Control *ctl, T *eb_out) {
  using U = typename TT<T>::U;
  T mn[3], mx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    mn[d] = from_ord((U)~acc[2 * d]);
    mx[d] = from_ord(acc[2 * d + 1]);
    ctl->out_mm[d] = (double)mn[d];
    ctl->out_mm[3 + d] = (double)mx[d];
  }
  T r;
  if (sizeof(T) == 4) {
    const float xr = __fsub_rn((float)mx[0], (float)mn[0]), yr = __fsub_rn((float)mx[1], (float)mn[1]);
    const float zr = __fsub_rn((float)mx[2], (float)mn[2]);
    r = (T)__fmul_rn(fmaxf(fmaxf(xr, yr), zr), (float)rel);
  } else {
    const double xr = __dsub_rn((double)mx[0], (double)mn[0]), yr = __dsub_rn((double)mx[1], (double)mn[1]);
    const double zr = __dsub_rn((double)mx[2], (double)mn[2]);
    r = (T)__dmul_rn(fmax(fmax(xr, yr), zr), (double)rel);
  }
  ctl->out_eb = (double)r;
  if (eb_out) *eb_out = r;
}

// findMinimumValues<T> + convertRelEb<T> on the device.  The host scan starts
// from float limits (include/utils.cuh:48-53) and ignores NaNs; 2D data has
// z == 0 (utils.cuh:141).
// One block (`block` of `nblocks`) of the grid-stride min/max; the last block
// to finish converts, stores the bound in ctl->out_eb and, when eb_out is
// given, in *eb_out.
template <typename T>
__device__ __forceinline__ void rel_to_abs_block(const T *__restrict__ x, const T *__restrict__ y,
                                                 const T *__restrict__ z, uint64_t n, uint32_t dim, T rel,
                                                 Control *ctl, T *eb_out, unsigned block, unsigned nblocks) {
  using U = typename TT<T>::U;
  __shared__ U red[6][8];
  __shared__ int last;
  U acc[6];
  // min starts at FLT_MAX and max at -FLT_MAX, as on the host
  for (int d = 0; d < 3; ++d) {
    acc[2 * d] = (U)~ord_of((T)FLT_MAX);
    acc[2 * d + 1] = ord_of((T)(-FLT_MAX));
  }
  fold_axis<T>(x, n, block, nblocks, acc[0], acc[1]);
  fold_axis<T>(y, n, block, nblocks, acc[2], acc[3]);
  if (dim == 3) fold_axis<T>(z, n, block, nblocks, acc[4], acc[5]);
  else fold_minmax<T>((T)0, acc[4], acc[5]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const U v = warp_max(acc[k]);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    U v = 0;
    for (int w = 0; w < 8; ++w) v = max(v, red[threadIdx.x][w]);
    atomicMax(&ctl->mm[threadIdx.x], (unsigned long long)v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(&ctl->sample_done, 1u) == nblocks - 1);
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    U all[6];
    for (int k = 0; k < 6; ++k) all[k] = (U)((volatile unsigned long long *)ctl->mm)[k];
    store_rel_bound<T>(all, rel, ctl, eb_out);
  }
}

template <typename T>
__global__ void __launch_bounds__(256, 6) rel_to_abs_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                         const T *__restrict__ z, uint64_t n, uint32_t dim,
                                                         T rel, Control *ctl) {
  rel_to_abs_block<T>(x, y, z, n, dim, rel, ctl, nullptr, blockIdx.x, gridDim.x);
}

// The same for a small snapshot (kSmallPoints), in one block, without a cleared
// control block.
template <typename T>
__global__ void __launch_bounds__(1024) rel_to_abs_small_kernel(const T *__restrict__ x, const T *__restrict__ y,
                                                                const T *__restrict__ z, uint64_t n, uint32_t dim,
                                                                T rel, Control *ctl) {
  using U = typename TT<T>::U;
  __shared__ U red[6][32];
  U acc[6];
  for (int d = 0; d < 3; ++d) {
    acc[2 * d] = (U)~ord_of((T)FLT_MAX);
    acc[2 * d + 1] = ord_of((T)(-FLT_MAX));
  }
  fold_axis<T>(x, n, 0, 1, acc[0], acc[1]);
  fold_axis<T>(y, n, 0, 1, acc[2], acc[3]);
  if (dim == 3) fold_axis<T>(z, n, 0, 1, acc[4], acc[5]);
  else fold_minmax<T>((T)0, acc[4], acc[5]);
  const U mine = block_max6(acc, red);
  if (threadIdx.x < 32) {
    U all[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) all[k] = __shfl_sync(0xFFFFFFFFu, mine, k);
    if (threadIdx.x == 0) store_rel_bound<T>(all, rel, ctl, nullptr);
  }
}

// ===========================================================================
// Compress.
// ===========================================================================
template <typename T>
struct CArgs {
  const T *x, *y, *z;
  uint8_t *out;
  unsigned long long out_cap;
  Control *ctl;
  unsigned long long *look;  // look-back records (16-byte aligned)
  unsigned long long n, G;
  T eb;
  const double *eb_dev;  // when set, the bound is read here on the device (strict-bound mode)
  uint32_t dim;
};

// ---------------------------------------------------------------------------
// Decoupled look-back over the chunk sizes.  One 32-byte record (four 64-bit
// words) serves 16 chunks: their payload sizes in 4-byte units, 12 bits each
// (five to a word, the sixteenth on top of the last word; zero until it is
// known), and below that the group's prefix -- the stream offset of its first
// chunk in 4-byte units -- with kLookKnown once somebody has it.  Every field
// lies in one word, is set by one relaxed atomic OR of that word and read with
// the whole word, so it is valid by itself and neither side needs a fence (an
// offset kept beside its flag cost two per chunk, 4-5 thousand cycles under
// load).  The two 16-byte loads a record takes have 64-bit elements: with
// 32-bit ones the sizes of every third chunk and the prefix span two elements,
// which nothing orders.
//
// A chunk's offset is the nearest known prefix at or below its own group plus
// the sizes from there on; a step reads 512 predecessors, one record a lane,
// since with over a thousand chunks in flight the nearest prefix is a few
// hundred chunks back.  Record 0 stands in the control block's last 32 bytes,
// the others follow at `look` + 4 words a record.
// ---------------------------------------------------------------------------
constexpr int kLookGroup = 16;
constexpr unsigned long long kLookKnown = 1ull << 51, kLookPrefix = kLookKnown - 1;
constexpr int kLookTail = kCtlBytes - 32;  // record 0 in the control block
static_assert(sizeof(Control) <= kLookTail, "record 0 must not touch the control fields");
static_assert(kStageBytes / 4 < 4096, "payload size in 12 bits");

// Bytes of the records after the first, for G chunks.
__host__ __device__ inline unsigned long long look_bytes(unsigned long long G) {
  return 32ull * ((G + kLookGroup - 1) / kLookGroup - 1);
}

__device__ __forceinline__ unsigned long long *look_record(Control *ctl, unsigned long long *look,
                                                           unsigned long long g) {
  return g == 0 ? reinterpret_cast<unsigned long long *>(reinterpret_cast<uint8_t *>(ctl) + kLookTail) : look + 4 * g;
}

// The word and the lowest bit of the size of a record's chunk i.
__host__ __device__ constexpr uint32_t look_word(uint32_t i) { return i == 15u ? 3u : i / 5u; }
__host__ __device__ constexpr uint32_t look_shift(uint32_t i) { return i == 15u ? 52u : 12u * (i % 5u); }

// Size of a record's chunk i (4-byte units; 0: not known yet) in its words.
__host__ __device__ __forceinline__ uint32_t look_size(const unsigned long long (&w)[4], uint32_t i) {
  return (uint32_t)(w[look_word(i)] >> look_shift(i)) & 4095u;
}

// One thread: the payload size of chunk c (bytes, a multiple of 4, not 0).
__device__ __forceinline__ void publish_size(Control *ctl, unsigned long long *look, unsigned long long c,
                                             uint32_t bytes) {
  const uint32_t i = (uint32_t)c & (kLookGroup - 1u);
  red_or_relaxed(look_record(ctl, look, c / kLookGroup) + look_word(i), (unsigned long long)(bytes >> 2) << look_shift(i));
}

// Warp-collective: the stream offset of chunk c, and its group's prefix for
// those behind.  Returns 1; while a predecessor has published nothing: -1
// without `wait`; with it, polls up to `limit` times and returns 0 when that
// or another CTA gave up (the kernel then stops taking chunks and reports
// GPZ_ETIMEOUT).
static __device__ int resolve_prefix(Control *ctl, unsigned long long *look, unsigned long long c,
                                     unsigned long long &excl_out, uint32_t limit = kSpinLimit, bool wait = true) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  const uint32_t own = (uint32_t)c & (kLookGroup - 1u);  // predecessors in the chunk's own group
  long long top = (long long)(c / kLookGroup);           // group of lane 31
  uint32_t in_group = 0;                                 // their sizes
  unsigned long long excl = 0;                           // units
  uint32_t spins = 0, backoff = 32;
  for (;;) {
    const long long g = top - 31 + lane;
    ulonglong2 q0 = make_ulonglong2(0ull, 0ull), q1 = q0;
    if (g >= 0) {
      const unsigned long long *const rec = look_record(ctl, look, (unsigned long long)g);
      q0 = ld_relaxed2(rec);
      q1 = ld_relaxed2(rec + 2);
    }
    const unsigned long long w[4] = {q0.x, q0.y, q1.x, q1.y};
    const bool known = g <= 0 || (w[3] & kLookKnown) != 0ull;
    const int near = 31 - __clz((int)__ballot_sync(FULL, known));  // -1: none in the window
    // sizes of this lane's chunks before c
    const uint32_t cnt = g == (long long)(c / kLookGroup) ? own : (uint32_t)kLookGroup;
    uint32_t sum = 0;
    bool missing = false;
#pragma unroll
    for (uint32_t i = 0; i < (uint32_t)kLookGroup; ++i) {
      const uint32_t v = look_size(w, i);
      if (i < cnt) {
        sum += v;
        missing |= v == 0u;
      }
    }
    const bool counts = g >= 0 && lane >= near;
    if (__any_sync(FULL, counts && missing)) {
      if (!wait) return -1;
      if (++spins > limit || ld_volatile(&ctl->abort)) {
        if (lane == 0) {
          atomicExch(&ctl->abort, 1u);
          set_status(ctl, kETIMEOUT);
        }
        return 0;
      }
      __nanosleep(backoff);
      backoff = min(backoff * 2, 256u);
      continue;
    }
    excl += __reduce_add_sync(FULL, counts ? sum : 0u);
    if (top == (long long)(c / kLookGroup)) in_group = __shfl_sync(FULL, sum, 31);
    if (near >= 0) {
      const unsigned long long pre = g <= 0 ? 0ull : (w[3] & kLookPrefix);
      excl += __shfl_sync(FULL, pre, near);
      // the group's prefix, unless it is there (setting it again changes nothing)
      if (lane == 31 && !(top == (long long)(c / kLookGroup) && near == 31))
        red_or_relaxed(look_record(ctl, look, c / kLookGroup) + 3, kLookKnown | (excl - in_group));
      break;
    }
    top -= 32;
  }
  excl_out = 4ull * excl;
  return 1;
}

}  // namespace gpzb
