// gpz_batchapi.cu -- batched compress / decompress: workspace layout, table
// building and kernel launches (gpz_batch_host.h), and the plan API of
// include/gpz_b200.h (gpz_batch_*, gpz_dbatch_*), which puts them in a CUDA
// graph.
//
// Classes are (float, 2D), (float, 3D), (double, 2D), (double, 3D): (compress)
// rel->abs when any of its snapshots asks for it, sampling, one persistent
// compress kernel; (decompress) a header check per stream, one persistent
// decompress kernel.  A plan's graph runs its classes as parallel branches, so
// that a class's launches and last chunks overlap the others' work: 368 -> 290
// us for 48 mixed snapshots of 10,000 to 1.2M points, 137 -> 57 us for 16 of
// 1,600 to 200,000.  The server's batches run them one after another on the
// slot's stream.

#include <algorithm>
#include <cstring>
#include <new>
#include <tuple>
#include <vector>

#include "gpz_b200.h"
#include "gpz_batch.cuh"
#include "gpz_batch_host.h"
#include "gpz_launch.h"

using namespace gpzb;

namespace {

constexpr uint64_t kRelPointsPerBlock = 1u << 13;  // points per rel->abs block of a snapshot
constexpr uint64_t kRelMaxBlocks = 1024;

inline uint64_t align256(uint64_t v) { return (v + 255u) & ~255ull; }
inline uint64_t chunks_of(uint64_t n) { return (n + kChunk - 1) / kChunk; }
inline uint64_t rel_blocks_of(uint64_t n) { return std::min(kRelMaxBlocks, std::max<uint64_t>(1, n / kRelPointsPerBlock)); }
int class_of(uint32_t bits, uint32_t dim) { return (bits == 64 ? 2 : 0) + (dim == 3 ? 1 : 0); }
template <typename T>
void fill_item(BItem<T> &bi, const gpz_batch_item &it, uint8_t *dev, uint64_t ctl_off, uint64_t look_off,
               uint64_t start) {
  memset(&bi, 0, sizeof(bi));
  bi.a.x = static_cast<const T *>(it.d_x);
  bi.a.y = static_cast<const T *>(it.d_y);
  bi.a.z = static_cast<const T *>(it.dim == 3 ? it.d_z : it.d_y);
  bi.a.out = static_cast<uint8_t *>(it.d_out);
  bi.a.out_cap = it.out_capacity;
  bi.a.ctl = reinterpret_cast<Control *>(dev + ctl_off);
  bi.a.look = reinterpret_cast<unsigned long long *>(dev + look_off - 32)  /* record 1 lies at look + 32 */;
  bi.a.n = it.n;
  bi.a.G = chunks_of(it.n);
  bi.a.eb = (T)it.eb;
  bi.a.eb_dev = nullptr;
  bi.a.dim = it.dim;
  bi.start = start;
  bi.rel_eb = (T)it.rel_eb;
  bi.seg_in = it.seg_size;
  bi.flags = ((it.flags & GPZ_FLAG_SEG_FIXED) ? kBatchSegFixed : 0u) | ((it.flags & GPZ_FLAG_SAFE31) ? kBatchSafe31 : 0u) |
             ((it.flags & GPZ_FLAG_REL_ON_DEVICE) ? kBatchRelDev : 0u) | (it.rel_mode ? kBatchRelMode : 0u);
}

template <typename T>
void fill_ditem(DItem<T> &d, const gpz_dbatch_item &it, Control *ctl) {
  memset(&d, 0, sizeof(d));
  d.a.s = static_cast<const uint8_t *>(it.d_stream);
  d.a.bytes = it.stream_bytes;
  d.a.x = static_cast<T *>(it.d_x);
  d.a.y = static_cast<T *>(it.d_y);
  d.a.z = static_cast<T *>(it.dim == 3 ? it.d_z : it.d_y);
  d.a.cap = it.out_capacity;
  d.a.ctl = ctl;
  auto al = [](const void *p) { return ((uintptr_t)p & 15u) == 0; };
  d.a.vec_ok = al(it.d_x) && al(it.d_y) && (it.dim == 2 || al(it.d_z));
  d.n = it.n;
}

// findMinimumValues + convertRelEb for the GPZ_FLAG_REL_ON_DEVICE snapshots
// of a class, sized to each snapshot: rmap[block] = snapshot << 40 |
// blocks of the snapshot << 20 | block within the snapshot.  The result is
// exactly gpz_rel_to_abs's (min and max do not depend on the partition) and
// goes to the snapshot's descriptor, where sampling and compress read it.
template <typename T>
__global__ void __launch_bounds__(256, 6) batch_rel_mapped_kernel(BItem<T> *items, const unsigned long long *rmap,
                                                                 uint32_t count) {
  const unsigned long long e = rmap[blockIdx.x];
  BItem<T> &it = items[e >> 40];
  // the snapshot's second control block, `count` blocks behind its first
  Control *rctl = reinterpret_cast<Control *>(reinterpret_cast<uint8_t *>(it.a.ctl) + (size_t)count * kCtlBytes);
  const unsigned nb = (unsigned)((e >> 20) & 0xFFFFFu), b = (unsigned)(e & 0xFFFFFu);
  rel_to_abs_block<T>(it.a.x, it.a.y, it.a.z, it.a.n, it.a.dim, it.rel_eb, rctl, &it.a.eb, b, nb);
}

// Grids of the batched persistent kernels on the current device (-1 when the
// kernel's shared-memory attribute cannot be raised there).
template <typename T, int DIM>
int compress_grid(uint64_t chunks) {
  const int o = resident_ctas(compress_batch_kernel<T, DIM>, kEncThreads, sizeof(EncShared));
  return o ? (int)std::min<uint64_t>(chunks, (uint64_t)current_sms() * o) : -1;
}

template <typename T, int DIM, class Cfg = DecCfg<T>, int PASS = kPassAll>
int dec_grid(uint64_t chunks) {
  constexpr int W = Cfg::warps;
  const int o = resident_ctas(decompress_batch_kernel<T, DIM, Cfg, PASS>, 32 * W, dec_smem_bytes_of<Cfg>());
  return o ? (int)std::min<uint64_t>((chunks + W - 1) / W, (uint64_t)current_sms() * o) : -1;
}

// Where a batch's work goes: a stream (one class after another), or a graph,
// whose classes become parallel branches behind the clearing of the control
// range.  Each branch beyond the first costs a plan some 45 us when the graph
// is instantiated and 48 us when it is destroyed, on the host; the graph is
// built node by node because capturing a stream took another 97 us for that
// stream's creation and destruction.  A decompress plan of 16 mixed streams
// that is created, launched once and destroyed: 1,122 us with one branch from
// a capture and a result copy per stream, 1,237 with branches from a capture,
// 1,101 so (single-class plans 990 / 847 / 751).
class Sink {
 public:
  explicit Sink(cudaStream_t st) : st_(st) {}
  explicit Sink(cudaGraph_t graph) : graph_(graph) {}

  // Clears `bytes` (a multiple of 4) at dev; the graph's first node.
  void clear(uint8_t *dev, uint64_t bytes) {
    if (!graph_) {
      cudaMemsetAsync(dev, 0, bytes, st_);
      return;
    }
    cudaMemsetParams m = {};
    m.dst = dev;
    m.elementSize = 4;
    m.width = bytes / 4;
    m.height = 1;
    ok_ = ok_ && cudaGraphAddMemsetNode(&root_, graph_, nullptr, 0, &m) == cudaSuccess;
  }
  // What follows waits for the clearing alone.
  void branch() { last_ = root_; }

  template <class... P, class... A>
  void launch(void (*kernel)(P...), dim3 grid, int threads, size_t smem, A... args) {
    if (!graph_) {
      kernel<<<grid, threads, smem, st_>>>(args...);
      return;
    }
    std::tuple<P...> values(args...);
    std::apply(
        [&](P &...v) {
          void *ptrs[] = {const_cast<void *>(static_cast<const volatile void *>(&v))...};
          cudaKernelNodeParams k = {};
          k.func = reinterpret_cast<void *>(kernel);
          k.gridDim = grid;
          k.blockDim = dim3((unsigned)threads);
          k.sharedMemBytes = (unsigned)smem;
          k.kernelParams = ptrs;  // copied by the call
          cudaGraphNode_t node = nullptr;
          ok_ = ok_ && cudaGraphAddKernelNode(&node, graph_, &last_, 1, &k) == cudaSuccess;
          last_ = node;
        },
        values);
  }
  bool ok() const { return ok_; }  // graph: every node was added

 private:
  cudaStream_t st_ = nullptr;
  cudaGraph_t graph_ = nullptr;
  cudaGraphNode_t root_ = nullptr, last_ = nullptr;
  bool ok_ = true;
};

template <typename T, int DIM>
void put_class(const gpzb_host::ClassPlan &cp, uint32_t count, uint8_t *dev, uint64_t claim_off, Sink &to) {
  BItem<T> *tab = reinterpret_cast<BItem<T> *>(dev + cp.table_off);
  to.branch();
  if (cp.rel_blocks)
    to.launch(batch_rel_mapped_kernel<T>, (unsigned)cp.rel_blocks, 256, 0, tab,
              reinterpret_cast<const unsigned long long *>(dev + cp.rmap_off), count);
  to.launch(batch_sample_kernel<T>, dim3(128, (unsigned)cp.items.size()), 256, 0, tab);
  to.launch(compress_batch_kernel<T, DIM>, (unsigned)cp.grid, kEncThreads, sizeof(EncShared), tab,
            (uint32_t)cp.items.size(), cp.work, reinterpret_cast<unsigned long long *>(dev + claim_off));
}

template <typename T, int DIM>
void put_dclass(const gpzb_host::ClassPlan &cp, uint8_t *dev, Sink &to) {
  DItem<T> *tab = reinterpret_cast<DItem<T> *>(dev + cp.table_off);
  const uint32_t K = (uint32_t)cp.items.size();
  to.branch();
  to.launch(dbatch_header_kernel<T, DIM>, (K + 127) / 128, 128, 0, tab, K);
  const auto *map = reinterpret_cast<const unsigned long long *>(dev + cp.map_off);
  if constexpr (sizeof(T) == 4) {
    to.launch(decompress_batch_kernel<T, DIM>, (unsigned)cp.grid, 32 * DecCfg<T>::warps, dec_smem_bytes<T>(), tab, map,
              cp.work);
  } else {
    to.launch(decompress_batch_kernel<T, DIM, DecCfgF64Fast, kPassFast>, (unsigned)cp.grid, 32 * DecCfgF64Fast::warps,
              dec_smem_bytes_of<DecCfgF64Fast>(), tab, map, cp.work);
    to.launch(decompress_batch_kernel<T, DIM, DecCfg<T>, kPassGeneral>, (unsigned)cp.grid2, 32 * DecCfg<T>::warps,
              dec_smem_bytes<T>(), tab, map, cp.work);
  }
}

void put_compress(const gpzb_host::Layout &L, uint8_t *dev, Sink &to) {
  to.clear(dev, L.zero_bytes);
  for (int c = 0; c < 4; ++c) {
    if (L.cls[c].items.empty()) continue;
    const uint64_t claim = L.claim_off + 8ull * c;
    switch (c) {
      case 0: put_class<float, 2>(L.cls[c], L.count, dev, claim, to); break;
      case 1: put_class<float, 3>(L.cls[c], L.count, dev, claim, to); break;
      case 2: put_class<double, 2>(L.cls[c], L.count, dev, claim, to); break;
      default: put_class<double, 3>(L.cls[c], L.count, dev, claim, to); break;
    }
  }
}

void put_decompress(const gpzb_host::Layout &L, uint8_t *dev, Sink &to) {
  to.clear(dev, L.zero_bytes);
  for (int c = 0; c < 4; ++c) {
    if (L.cls[c].items.empty()) continue;
    switch (c) {
      case 0: put_dclass<float, 2>(L.cls[c], dev, to); break;
      case 1: put_dclass<float, 3>(L.cls[c], dev, to); break;
      case 2: put_dclass<double, 2>(L.cls[c], dev, to); break;
      default: put_dclass<double, 3>(L.cls[c], dev, to); break;
    }
  }
}

}  // namespace

// ===========================================================================
// Workspace layout, tables, launches.
// ===========================================================================
namespace gpzb_host {

bool compress_item_ok(const gpz_batch_item &it) {
  const uint64_t hdr = it.float_bits == 64 ? 32 : 24, meta = it.float_bits == 64 ? 64 : 36;
  return (it.float_bits == 32 || it.float_bits == 64) && (it.dim == 2 || it.dim == 3) && it.n >= 1 && it.d_x &&
         it.d_y && (it.dim == 2 || it.d_z) && it.d_out && it.out_capacity >= hdr + chunks_of(it.n) * (8 + meta) &&
         !((it.flags & GPZ_FLAG_SEG_FIXED) && it.seg_size == 0) &&
         (it.flags & ~(GPZ_FLAG_SAFE31 | GPZ_FLAG_SEG_FIXED | GPZ_FLAG_REL_ON_DEVICE)) == 0;
}

bool decompress_item_ok(const gpz_dbatch_item &it) {
  return (it.float_bits == 32 || it.float_bits == 64) && (it.dim == 2 || it.dim == 3) && it.n >= 1 && it.d_stream &&
         ((uintptr_t)it.d_stream & 7u) == 0 && it.d_x && it.d_y && (it.dim == 2 || it.d_z) && it.out_capacity >= it.n;
}

bool compress_layout(const gpz_batch_item *items, uint32_t count, Layout &L) {
  L = Layout();
  L.count = count;
  L.look_off.resize(count);
  uint64_t off = 2ull * count * kCtlBytes;
  for (uint32_t i = 0; i < count; ++i) {
    L.look_off[i] = off;
    const int c = class_of(items[i].float_bits, items[i].dim);
    off += look_bytes(chunks_of(items[i].n));
    ClassPlan &cp = L.cls[c];
    cp.items.push_back(i);
    cp.work += chunks_of(items[i].n);
    if (items[i].flags & GPZ_FLAG_REL_ON_DEVICE) cp.rel_blocks += rel_blocks_of(items[i].n);
  }
  L.claim_off = align256(off);
  L.zero_bytes = L.claim_off + 4 * 8;
  off = align256(L.zero_bytes);
  for (int c = 0; c < 4; ++c) {
    ClassPlan &cp = L.cls[c];
    if (cp.items.empty()) continue;
    cp.table_off = off;
    off = align256(off + (c < 2 ? sizeof(BItem<float>) : sizeof(BItem<double>)) * cp.items.size());
    cp.rmap_off = off;
    off = align256(off + 8 * cp.rel_blocks);
    switch (c) {
      case 0: cp.grid = compress_grid<float, 2>(cp.work); break;
      case 1: cp.grid = compress_grid<float, 3>(cp.work); break;
      case 2: cp.grid = compress_grid<double, 2>(cp.work); break;
      default: cp.grid = compress_grid<double, 3>(cp.work); break;
    }
    if (cp.grid < 1) return false;
  }
  L.bytes = off;
  return true;
}

bool decompress_layout(const gpz_dbatch_item *items, uint32_t count, Layout &L) {
  L = Layout();
  L.count = count;
  for (uint32_t i = 0; i < count; ++i) {
    ClassPlan &cp = L.cls[class_of(items[i].float_bits, items[i].dim)];
    cp.items.push_back(i);
    cp.work += chunks_of(items[i].n);
  }
  L.zero_bytes = (uint64_t)count * kCtlBytes;
  uint64_t off = align256(L.zero_bytes);
  for (int c = 0; c < 4; ++c) {
    ClassPlan &cp = L.cls[c];
    if (cp.items.empty()) continue;
    cp.table_off = off;
    off = align256(off + (c < 2 ? sizeof(DItem<float>) : sizeof(DItem<double>)) * cp.items.size());
    cp.map_off = off;
    off = align256(off + 8 * cp.work);
    switch (c) {
      case 0: cp.grid = dec_grid<float, 2>(cp.work); break;
      case 1: cp.grid = dec_grid<float, 3>(cp.work); break;
      case 2:
        cp.grid = dec_grid<double, 2, DecCfgF64Fast, kPassFast>(cp.work);
        cp.grid2 = dec_grid<double, 2, DecCfg<double>, kPassGeneral>(cp.work);
        break;
      default:
        cp.grid = dec_grid<double, 3, DecCfgF64Fast, kPassFast>(cp.work);
        cp.grid2 = dec_grid<double, 3, DecCfg<double>, kPassGeneral>(cp.work);
        break;
    }
    if (cp.grid < 1 || (c >= 2 && cp.grid2 < 1)) return false;
  }
  L.bytes = off;
  return true;
}

void compress_tables(const gpz_batch_item *items, const Layout &L, uint8_t *dev, uint8_t *image) {
  auto H = [&](uint64_t dev_off) { return image + (dev_off - L.zero_bytes); };
  for (int c = 0; c < 4; ++c) {
    const ClassPlan &cp = L.cls[c];
    if (cp.items.empty()) continue;
    uint64_t start = 0, rb = 0;
    unsigned long long *rmap = reinterpret_cast<unsigned long long *>(H(cp.rmap_off));
    for (size_t k = 0; k < cp.items.size(); ++k) {
      const uint32_t i = cp.items[k];
      const gpz_batch_item &it = items[i];
      if (c < 2) fill_item<float>(reinterpret_cast<BItem<float> *>(H(cp.table_off))[k], it, dev, ctl_off(i),
                                  L.look_off[i], start);
      else fill_item<double>(reinterpret_cast<BItem<double> *>(H(cp.table_off))[k], it, dev, ctl_off(i),
                             L.look_off[i], start);
      start += chunks_of(it.n);
      if (it.flags & GPZ_FLAG_REL_ON_DEVICE) {
        const uint64_t nb = rel_blocks_of(it.n);
        for (uint64_t q = 0; q < nb; ++q) rmap[rb++] = ((unsigned long long)k << 40) | (nb << 20) | q;
      }
    }
  }
}

void decompress_tables(const gpz_dbatch_item *items, const Layout &L, uint8_t *dev, uint8_t *image) {
  auto H = [&](uint64_t dev_off) { return image + (dev_off - L.zero_bytes); };
  for (int c = 0; c < 4; ++c) {
    const ClassPlan &cp = L.cls[c];
    if (cp.items.empty()) continue;
    uint64_t q = 0;
    unsigned long long *map = reinterpret_cast<unsigned long long *>(H(cp.map_off));
    for (size_t k = 0; k < cp.items.size(); ++k) {
      const uint32_t i = cp.items[k];
      Control *ctl = reinterpret_cast<Control *>(dev + ctl_off(i));
      if (c < 2) fill_ditem<float>(reinterpret_cast<DItem<float> *>(H(cp.table_off))[k], items[i], ctl);
      else fill_ditem<double>(reinterpret_cast<DItem<double> *>(H(cp.table_off))[k], items[i], ctl);
      const uint64_t G = chunks_of(items[i].n);
      for (uint64_t ch = 0; ch < G; ++ch) map[q++] = ((unsigned long long)k << kBatchLocalBits) | ch;
    }
  }
}

void compress_enqueue(const Layout &L, uint8_t *dev, cudaStream_t st) {
  Sink to(st);
  put_compress(L, dev, to);
}

void decompress_enqueue(const Layout &L, uint8_t *dev, cudaStream_t st) {
  Sink to(st);
  put_decompress(L, dev, to);
}

}  // namespace gpzb_host

// ===========================================================================
// Plans: the workspace allocated once, the launches as a graph.
// ===========================================================================
namespace {

struct Plan {
  uint32_t count = 0;
  uint8_t *mem = nullptr;
  uint64_t bytes = 0;
  cudaGraphExec_t exec = nullptr;
  ~Plan() {
    if (exec) cudaGraphExecDestroy(exec);
    if (mem) cudaFree(mem);
  }
};

// Allocates the workspace, uploads the table image built by `tables` and
// builds the plan's graph from what `put` launches.
template <typename Tables, typename Put>
int make_plan(Plan &p, const gpzb_host::Layout &L, Tables tables, Put put) {
  p.count = L.count;
  p.bytes = L.bytes;
  if (cudaMalloc(&p.mem, p.bytes) != cudaSuccess) {
    p.mem = nullptr;
    return GPZ_ECUDA;
  }
  std::vector<uint8_t> image(L.bytes - L.zero_bytes);
  tables(p.mem, image.data());
  if (cudaMemcpy(p.mem + L.zero_bytes, image.data(), image.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    return GPZ_ECUDA;
  cudaGraph_t graph = nullptr;
  bool ok = cudaGraphCreate(&graph, 0) == cudaSuccess;
  if (ok) {
    Sink to(graph);
    put(L, p.mem, to);
    ok = to.ok() && cudaGraphInstantiate(&p.exec, graph, 0) == cudaSuccess;
    cudaGraphDestroy(graph);
  }
  if (!ok) cudaGetLastError();
  return ok ? GPZ_OK : GPZ_ECUDA;
}

// The plan's control blocks lie one behind the other at the head of its
// workspace and come back in one copy: a copy per block cost 8-10 us of host
// time each (1.44 -> 0.40 ms for a launch of 48 snapshots with its results).
int read_controls(const uint8_t *dev, uint32_t blocks, std::vector<uint8_t> &h, cudaStream_t st) {
  static_assert(kCtlBytes == 256, "gpzb_host::ctl_off");
  h.resize((size_t)blocks * kCtlBytes);
  if (cudaMemcpyAsync(h.data(), dev, h.size(), cudaMemcpyDeviceToHost, st) != cudaSuccess) return GPZ_ECUDA;
  return cudaStreamSynchronize(st) == cudaSuccess ? GPZ_OK : GPZ_ECUDA;
}

const Control &control(const std::vector<uint8_t> &h, uint32_t i) {
  return *reinterpret_cast<const Control *>(h.data() + gpzb_host::ctl_off(i));
}

}  // namespace

struct gpz_batch {
  Plan plan;
  std::vector<gpz_batch_item> items;
};

struct gpz_dbatch {
  Plan plan;
};

extern "C" {

int gpz_batch_create(const gpz_batch_item *items, uint32_t count, gpz_batch **batch, uint32_t *bad_item) {
  if (!batch || !items || count == 0) return GPZ_EINVAL;
  *batch = nullptr;
  for (uint32_t i = 0; i < count; ++i)
    if (!gpzb_host::compress_item_ok(items[i])) {
      if (bad_item) *bad_item = i;
      return GPZ_EINVAL;
    }
  gpzb_host::Layout L;
  if (!gpzb_host::compress_layout(items, count, L)) return GPZ_ECUDA;
  gpz_batch *b = new (std::nothrow) gpz_batch;
  if (!b) return GPZ_ECUDA;
  b->items.assign(items, items + count);
  const int rc = make_plan(
      b->plan, L, [&](uint8_t *dev, uint8_t *image) { gpzb_host::compress_tables(items, L, dev, image); }, put_compress);
  if (rc != GPZ_OK) {
    delete b;
    return rc;
  }
  *batch = b;
  return GPZ_OK;
}

int gpz_batch_launch(gpz_batch *b, void *stream) {
  if (!b || !b->plan.exec) return GPZ_EINVAL;
  return cudaGraphLaunch(b->plan.exec, static_cast<cudaStream_t>(stream)) == cudaSuccess ? GPZ_OK : GPZ_ECUDA;
}

int gpz_batch_results(gpz_batch *b, gpz_result *results, double *h_eb, void *stream) {
  if (!b || !results) return GPZ_EINVAL;
  const uint32_t n = b->plan.count;
  std::vector<uint8_t> h;
  const int rc = read_controls(b->plan.mem, 2 * n, h, static_cast<cudaStream_t>(stream));
  if (rc != GPZ_OK) return rc;
  for (uint32_t i = 0; i < n; ++i) {
    const Control &c = control(h, i);
    results[i].stream_bytes = c.stream_bytes;
    results[i].seg_size = c.seg;
    results[i].adjusted = c.adjusted;
    results[i].status = c.status;
    results[i].id_overflow = c.id_overflow;
    if (h_eb) {
      const gpz_batch_item &it = b->items[i];
      if (it.flags & GPZ_FLAG_REL_ON_DEVICE) h_eb[i] = control(h, n + i).out_eb;
      else h_eb[i] = it.float_bits == 32 ? (double)(float)it.eb : it.eb;
    }
  }
  return GPZ_OK;
}

uint64_t gpz_batch_device_bytes(const gpz_batch *b) { return b ? b->plan.bytes : 0; }

int gpz_batch_destroy(gpz_batch *b) {
  if (!b) return GPZ_EINVAL;
  delete b;
  return GPZ_OK;
}

int gpz_dbatch_create(const gpz_dbatch_item *items, uint32_t count, gpz_dbatch **batch, uint32_t *bad_item) {
  if (!batch || !items || count == 0) return GPZ_EINVAL;
  *batch = nullptr;
  for (uint32_t i = 0; i < count; ++i)
    if (!gpzb_host::decompress_item_ok(items[i])) {
      if (bad_item) *bad_item = i;
      return GPZ_EINVAL;
    }
  gpzb_host::Layout L;
  if (!gpzb_host::decompress_layout(items, count, L)) return GPZ_ECUDA;
  gpz_dbatch *b = new (std::nothrow) gpz_dbatch;
  if (!b) return GPZ_ECUDA;
  const int rc = make_plan(
      b->plan, L, [&](uint8_t *dev, uint8_t *image) { gpzb_host::decompress_tables(items, L, dev, image); }, put_decompress);
  if (rc != GPZ_OK) {
    delete b;
    return rc;
  }
  *batch = b;
  return GPZ_OK;
}

int gpz_dbatch_launch(gpz_dbatch *b, void *stream) {
  if (!b || !b->plan.exec) return GPZ_EINVAL;
  return cudaGraphLaunch(b->plan.exec, static_cast<cudaStream_t>(stream)) == cudaSuccess ? GPZ_OK : GPZ_ECUDA;
}

int gpz_dbatch_results(gpz_dbatch *b, gpz_result *results, void *stream) {
  if (!b || !results) return GPZ_EINVAL;
  std::vector<uint8_t> h;
  const int rc = read_controls(b->plan.mem, b->plan.count, h, static_cast<cudaStream_t>(stream));
  if (rc != GPZ_OK) return rc;
  for (uint32_t i = 0; i < b->plan.count; ++i) {
    memset(&results[i], 0, sizeof(gpz_result));
    results[i].status = control(h, i).status;
  }
  return GPZ_OK;
}

int gpz_dbatch_destroy(gpz_dbatch *b) {
  if (!b) return GPZ_EINVAL;
  delete b;
  return GPZ_OK;
}

}  // extern "C"
