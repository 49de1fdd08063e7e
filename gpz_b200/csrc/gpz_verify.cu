// gpz_verify.cu -- per-point verification of a reconstruction against the
// original points (gpz_verify of include/gpz_b200.h).
//
// The reference verifier (src/utils.cu:17-217) sorts every axis of both
// arrays and compares the sorted sequences: it never pairs a reconstructed
// point with its original, because the decoder emits points in the stream's
// order (sorted by block within each chunk).  Here the pairing is recovered
// exactly: for each 1024-point chunk the kernel recomputes what the encoder
// sorted -- the composite (block id - min block id) << 10 | r, r being the
// point's rank in the encoder's input order -- and ranks it, so sorted
// position s of the chunk names the point the decoder wrote at s.  Every point is then checked against the bound, and per axis the
// maximum error and the squared-error sum (for MSE / PSNR) are accumulated.
// The quantization arithmetic is the compress kernel's (gpz_encode.cuh step
// 1) so the block ids are the encoder's bit for bit.

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "gpz_b200.h"
#include "gpz_encode.cuh"
#include "gpz_launch.h"

using namespace gpzb;

namespace {

struct VerifyAcc {
  unsigned long long over;      // points with some axis off by more than eb
  unsigned long long over_tol;  // ... by more than 1.01 * eb (the reference verifier's tolerance)
  unsigned long long max_err[3];  // ordered keys of the largest |error| per axis (non-negative floats)
  double sq[3];                 // squared-error sums
  unsigned long long mm[6];     // ordered min (inverted) / max of the originals, per axis
};

// Shared memory of a verify CTA: the ranking's, and the CTA's sums.
struct VerifyShared : RankShared {
  double sq[3][kEncWarps];
  uint32_t over[kEncWarps], over_tol[kEncWarps];
  unsigned long long emax[3][kEncWarps];
  unsigned long long mn[3], mx[3];  // ordered minimum (inverted) / maximum of the chunks so far
};
constexpr int kVerifyCtas = 6;  // resident CTAs per SM the registers are sized for

// A CTA of four warps takes one chunk after another: it repeats the encoder's
// block ids and ranking (the same code: gpz_encode.cuh), which says which point
// the decoder wrote at each position, and compares axis by axis, the originals
// taken from shared memory in ranked order.
//
// Bound by instruction issue like the encoder (the 24 bytes a point would take
// a tenth of the time).  A warp per chunk with a bitonic network of 64-bit
// composites in shared memory (55 steps of 16 exchanges a lane) took 238 us on
// 4M float 3D points; this form 43 us.
template <typename T, int DIM>
__global__ void __launch_bounds__(kEncThreads, kVerifyCtas)
    verify_kernel(const T *__restrict__ x, const T *__restrict__ y, const T *__restrict__ z, const T *__restrict__ rx,
                  const T *__restrict__ ry, const T *__restrict__ rz, unsigned long long n, T eb, uint32_t seg, T bound,
                  VerifyAcc *acc) {
  using UO = typename TT<T>::U;
  constexpr bool is64 = sizeof(T) == 8;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(16) unsigned char verify_smem[];
  VerifyShared &sm = *reinterpret_cast<VerifyShared *>(verify_smem);
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const T *const X[3] = {x, y, z};
  const T *const Y[3] = {rx, ry, rz};
  const uint32_t sh = (uint32_t)__ffs((int)seg) - 1u;
  const T inv = is64 ? (T)__ddiv_rn(1.0, __dmul_rn(2.0, (double)eb)) : (T)__fdiv_rn(1.0f, __fmul_rn(2.0f, (float)eb));
  const unsigned long long G = (n + kChunk - 1) / kChunk;
  const T tol = (T)1.01f * bound;
  uint32_t over = 0, over_tol = 0, rank_skip = 0, declined = 0;
  T emax[3] = {0, 0, 0};
  double sq[3] = {0.0, 0.0, 0.0};
  if (t < 3) sm.mn[t] = sm.mx[t] = 0ull;
  for (unsigned long long c = blockIdx.x; c < G; c += gridDim.x) {
    const unsigned long long base = c * kChunk;
    const uint32_t nvalid = (uint32_t)min((unsigned long long)kChunk, n - base);
    const bool full = nvalid == (uint32_t)kChunk;
    uint32_t *const H = sm.A[0], *const S = sm.A[1];
    // ---- block ids exactly as the encoder computes them ----
    uint32_t key[kEncPer], bnd;
    {
      T v[DIM][kEncPer];
      load_points<T, DIM>(x, y, z, base, nvalid, v);
      __syncthreads();  // the previous chunk's arrays have been read
      *reinterpret_cast<uint4 *>(H + 8 * t) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4 *>(H + 8 * t + 4) = make_uint4(0u, 0u, 0u, 0u);
      if (t == 0) sm.ncrowd = 0u;
      put_minmax<T, DIM>(sm, v, lane, warp);
      __syncthreads();
      if (warp == 0) {
        unsigned long long term;
        bool wide;
        const T mmv = chunk_scalars<T, DIM>(sm, seg, sh, eb, inv, lane, term, wide);
        if (lane < DIM) sm.mn[lane] = max(sm.mn[lane], (unsigned long long)(UO)~ord_of(mmv));
        if (lane >= 3 && lane < 3 + DIM) sm.mx[lane - 3] = max(sm.mx[lane - 3], (unsigned long long)ord_of(mmv));
      }
      __syncthreads();
      const uint4 sc = ld4(sm.sc);
      bnd = sc.z;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const T nmd = reinterpret_cast<const T *>(sm.nm)[d];
        const uint32_t kmul = d == 1 ? sc.x : sc.y;
#pragma unroll
        for (int e = 0; e < kEncPer; ++e) {
          uint32_t kq;
          if constexpr (!is64) kq = __float2uint_rz(__fmaf_rn((float)v[d][e], (float)inv, (float)nmd)) >> sh;
          else kq = (uint32_t)(__double2ull_rz(__fma_rn((double)v[d][e], (double)inv, (double)nmd)) >> sh);
          key[e] = d == 0 ? kq : key[e] + kq * kmul;
        }
      }
#pragma unroll
      for (int e = 0; e < kEncPer; ++e) key[e] &= 0x7FFFFFFFu;
    }
    // ---- the order the encoder gave them ----
    const uint16_t *ranks;
    const int how = rank_chunk<T>(sm, H, S, key, bnd, nvalid, rank_skip, declined, t, lane, warp, ranks);
    uint32_t r[8];  // point at position 128j + t
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = point_of_rank(how == 1 ? H[128 * j + t] & 1023u : (uint32_t)ranks[128 * j + t]);
    __syncthreads();  // the ranking's arrays are free
    // ---- position s holds the point the decoder wrote at s ----
    uint32_t off = 0, off_tol = 0;  // bit j: position 128j + t is off on some axis
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      // the axis by point, in one of two 8 KB halves in turn
      T *const O = reinterpret_cast<T *>(d & 1 ? sm.R : sm.A[0]);
      {
        T v[1][kEncPer];
        load_points<T, 1>(X[d], X[d], X[d], base, nvalid, v);
#pragma unroll
        for (int e = 0; e < kEncPer; ++e) O[Points<T>::point(t, e)] = v[0][e];
      }
      T rec[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) rec[j] = full || 128u * j + t < nvalid ? Y[d][base + 128u * j + t] : (T)0;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (!full && 128u * j + t >= nvalid) continue;
        const T o = O[r[j]];
        const T e = o > rec[j] ? o - rec[j] : rec[j] - o;
        if (!(e <= bound)) off |= 1u << j;
        if (!(e <= tol)) off_tol |= 1u << j;
        emax[d] = fmax(emax[d], e);
        sq[d] += (double)e * (double)e;
      }
    }
    over += __popc(off);
    over_tol += __popc(off_tol);
  }
  // ---- CTA sums, then one atomic per value and CTA ----
  over = __reduce_add_sync(FULL, over);
  over_tol = __reduce_add_sync(FULL, over_tol);
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const UO em = warp_max(ord_of(emax[d]));
    double s = sq[d];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (lane == 0) {
      sm.emax[d][warp] = (unsigned long long)em;
      sm.sq[d][warp] = s;
    }
  }
  if (lane == 0) {
    sm.over[warp] = over;
    sm.over_tol[warp] = over_tol;
  }
  __syncthreads();
  if (t < DIM) {
    unsigned long long em = 0;
    double s = 0.0;
    for (int w = 0; w < kEncWarps; ++w) {
      em = max(em, sm.emax[t][w]);
      s += sm.sq[t][w];
    }
    atomicMax(&acc->max_err[t], em);
    atomicAdd(&acc->sq[t], s);
    atomicMax(&acc->mm[2 * t], sm.mn[t]);
    atomicMax(&acc->mm[2 * t + 1], sm.mx[t]);
  }
  if (t == 32) atomicAdd(&acc->over, (unsigned long long)sm.over[0] + sm.over[1] + sm.over[2] + sm.over[3]);
  if (t == 33) atomicAdd(&acc->over_tol, (unsigned long long)sm.over_tol[0] + sm.over_tol[1] + sm.over_tol[2] + sm.over_tol[3]);
}

template <typename T>
double unord(unsigned long long o) {
  if constexpr (sizeof(T) == 4) return (double)from_ord((uint32_t)o);
  else return from_ord(o);
}

template <typename T>
int verify_t(uint32_t dim, uint64_t n, const void *dx, const void *dy, const void *dz, const void *rx, const void *ry,
             const void *rz, double eb, uint32_t seg, double bound, void *d_scratch, gpz_verify_result *out,
             cudaStream_t st) {
  VerifyAcc *acc = static_cast<VerifyAcc *>(d_scratch);
  if (cudaMemsetAsync(acc, 0, sizeof(VerifyAcc), st) != cudaSuccess) return GPZ_ECUDA;
  const size_t smem = sizeof(VerifyShared);
  const T *x = (const T *)dx, *y = (const T *)dy, *z = (const T *)(dim == 3 ? dz : dy);
  const T *a = (const T *)rx, *b = (const T *)ry, *c = (const T *)(dim == 3 ? rz : ry);
  const int sms = current_sms();
  const uint64_t G = (n + kChunk - 1) / kChunk;
  auto launch = [&](auto kernel) -> bool {
    const int occ = resident_ctas(kernel, kEncThreads, smem);
    if (occ == 0) return false;
    const uint64_t grid = std::min<uint64_t>(G, (uint64_t)sms * occ);
    kernel<<<(unsigned)grid, kEncThreads, smem, st>>>(x, y, z, a, b, c, n, (T)eb, seg, (T)bound, acc);
    return true;
  };
  if (!(dim == 3 ? launch(verify_kernel<T, 3>) : launch(verify_kernel<T, 2>))) return GPZ_ECUDA;
  if (cudaGetLastError() != cudaSuccess) return GPZ_ECUDA;
  VerifyAcc h;
  if (cudaMemcpyAsync(&h, acc, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess) return GPZ_ECUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return GPZ_ECUDA;
  memset(out, 0, sizeof(*out));
  out->points = n;
  out->over_bound = h.over;
  out->over_bound_tol = h.over_tol;
  double nrm = 0.0;
  for (uint32_t d = 0; d < dim; ++d) {
    using UO = typename TT<T>::U;
    out->max_abs_err[d] = unord<T>(h.max_err[d]);
    out->mse[d] = h.sq[d] / (double)n;
    const double mn = unord<T>((UO) ~(UO)h.mm[2 * d]), mx = unord<T>(h.mm[2 * d + 1]);
    out->value_range[d] = mx - mn;
    out->psnr[d] = 20.0 * log10(mx - mn) - 10.0 * log10(out->mse[d]);
    const double r = pow(10.0, out->psnr[d] / -20.0);
    nrm += r * r;
  }
  const double rms = sqrt(nrm / dim);
  out->psnr_combined = rms > 0.0 ? -20.0 * log10(rms) : INFINITY;
  return GPZ_OK;
}

}  // namespace

extern "C" {

uint64_t gpz_verify_scratch_bytes(void) { return 256; }

int gpz_verify_bound(uint32_t float_bits, uint32_t dim, uint64_t n, const void *d_x, const void *d_y, const void *d_z,
                     const void *d_rx, const void *d_ry, const void *d_rz, double eb, uint32_t seg_size, double bound,
                     void *d_scratch, uint64_t scratch_bytes, gpz_verify_result *result, void *stream) {
  if ((float_bits != 32 && float_bits != 64) || (dim != 2 && dim != 3) || n == 0 || !d_x || !d_y ||
      (dim == 3 && !d_z) || !d_rx || !d_ry || (dim == 3 && !d_rz) || seg_size == 0 || !(eb > 0.0) ||
      !(bound > 0.0) || !d_scratch || !result)
    return GPZ_EINVAL;
  if (scratch_bytes < sizeof(VerifyAcc)) return GPZ_ENOSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return float_bits == 32
             ? verify_t<float>(dim, n, d_x, d_y, d_z, d_rx, d_ry, d_rz, eb, seg_size, bound, d_scratch, result, st)
             : verify_t<double>(dim, n, d_x, d_y, d_z, d_rx, d_ry, d_rz, eb, seg_size, bound, d_scratch, result, st);
}

int gpz_verify(uint32_t float_bits, uint32_t dim, uint64_t n, const void *d_x, const void *d_y, const void *d_z,
               const void *d_rx, const void *d_ry, const void *d_rz, double eb, uint32_t seg_size, void *d_scratch,
               uint64_t scratch_bytes, gpz_verify_result *result, void *stream) {
  return gpz_verify_bound(float_bits, dim, n, d_x, d_y, d_z, d_rx, d_ry, d_rz, eb, seg_size, eb, d_scratch,
                          scratch_bytes, result, stream);
}

}  // extern "C"
