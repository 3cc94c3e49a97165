// ccdgpu — C ABI implementation (include/ccdgpu.h).
//
// A handle holds the whole CCD state of one system in device memory, laid out for the
// kernels in ccd_kernels.cuh:
//   * amplitudes packed, one in four (a < b, i < j; two buffers, ping-pong by a device-side parity
//     bit), and in the reference's layouts for the table path, the stage calls and the readers;
//   * V_pppp as the pp ladder's chunks in their shared-memory image (of a symmetric channel one
//     triangle of blocks), for mixed handles also as bf16 terms in the tensor core's layout;
//   * V_hhpp packed like the amplitudes, and transposed to pp x hh;
//   * the ring's operands of each pair of transposed modified channels in fragment order;
//   * the loadMaps tables as int32 flat offsets into the target slabs, validated at create;
//   * a Control block with the solve loop's state (energy history, stop rule, parity), so a
//     captured iteration graph can be replayed without host synchronisation.
#include <cuda_runtime.h>
#include <omp.h>

#include <algorithm>
#include <atomic>
#include <queue>
#include <chrono>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "ccd_channels.cuh"
#include "ccd_device.cuh"
#include "ccd_general.cuh"
#include "ccd_kernels.cuh"
#include "ccd_setup.cuh"
#include "ccd_tc.cuh"
#include "ccdgpu.h"
#include "host/channel_order.h"

using namespace ccd;

namespace {

struct DevBuf {
  void *p = nullptr;
  size_t bytes = 0;
};

}  // namespace

// A handle's streams and events (see the pool below).
constexpr int kStreams = 5, kEvents = 17;
struct StreamSet {
  int dev = -1;
  cudaStream_t s[kStreams] = {};
  cudaEvent_t ev[kEvents] = {};
};

struct ccdgpu_handle {
  ccdgpu_options opt{};
  StreamSet sset;  // the streams and events below, from the process-wide pool
  cudaStream_t s0 = nullptr, s1 = nullptr, s2 = nullptr, s3 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_fork2 = nullptr, ev_fork3 = nullptr;
  cudaEvent_t ev_join = nullptr, ev_join2 = nullptr, ev_join3 = nullptr;
  cudaEvent_t ev[10] = {};
  uint64_t nch = 0, nsp = 0, np = 0, npart = 0;
  int64_t n_t = 0, n_m = 0, n_h = 0, n_p = 0;
  int n_hh_cta = 0, n_hh_warp = 0;  // hh-ladder units: one per CTA (hk > 8) first, then per warp
  int n_hh_out = 0;    // hh-ladder reduction outputs
  int n_row_tiles = 0;  // row tiles of all channels
  int n_act = 0, n_mod = 0, n_mod_small = 0, n_tiles = 0;
  int n_ranges = 0;
  int n_asm_blocks = 0;  // fused assembly CTAs (persistent, striding over quad_items)
  int n_cls[3] = {0, 0, 0};  // FP64 pp-ladder tiles per column class (thin, mid, wide)
  int n_mod_pad[4] = {0, 0, 0, 0};  // ring channels by padded size 32, 48, 64, 80 (after small)
  bool have_3body = false;
  std::vector<DevBuf> allocs;

  ChanInfo *chans = nullptr;
  ModInfo *mods = nullptr;        // small (n_mod_small), then by padded size 32 .. 80
  LadderTile *tiles = nullptr;
  HHTile *hh_tiles = nullptr;
  HHOut *hh_out = nullptr;
  TXTile *tx_tiles = nullptr;
  int n_tx = 0;
  int32_t *prow = nullptr, *hcol = nullptr;  // pp / hh pair -> 2 u (+ 1 when a > b), -1
  double *part = nullptr;
  ElemRange *ranges = nullptr;
  QuadItem *quad_items = nullptr;  // fused assembly: work items of quads (u, w)
  QuadRow *quad_rows = nullptr;    // fused assembly: per strict packed row / hole pair tables
  int64_t n_quad_rows = 0;
  QuadCol *quad_cols = nullptr;
  int n_quad_items = 0;
  int2 *pp_pairs = nullptr, *hh_pairs = nullptr;
  int32_t *pp_swap = nullptr, *hh_swap = nullptr;
  int64_t *list_off = nullptr;
  int32_t *list = nullptr;
  double *eps = nullptr, *v_pphh = nullptr, *v_hhhh = nullptr, *v_t = nullptr;
  // Packed layout (quads): amplitudes (ping-pong by the control block's parity), V_hhpp, and
  // the two ring sums of each quad.
  double *tq[2] = {nullptr, nullptr}, *vq = nullptr, *r_quad = nullptr;
  int64_t n_q = 0;
  double *v_hpph = nullptr, *v_hphp = nullptr;
  double *t[2] = {nullptr, nullptr}, *dmat = nullptr, *old_phhp = nullptr, *r_phhp = nullptr;
  // t[0] of the fused path holds the amplitudes in the reference order only while slab_current
  // (it is expanded when they are read); dmat likewise holds t2Diff_pphh unless d_from names
  // the iteration kind (1 FP64, 2 mixed) whose ladder planes it is expanded from when read.
  bool slab_current = true;
  // Fused path, for the stage calls: whether old_phhp and the three-body chains hold the current
  // amplitudes too, and whether t[1] holds the T2 that ccdgpu_map_to_distributed scatters (the
  // last one loaded or assembled by a stage; else it is the current amplitudes).
  bool chains_current = true, t2_staged = false;
  int d_from = 0;
  double *x = nullptr, *tx = nullptr;  // hh-ladder X; 0.5 T X in the packed layout
  double *v_x = nullptr;               // V_hhhh in the layout of X
  double *s = nullptr, *r = nullptr, *xh = nullptr, *yp = nullptr, *epart = nullptr;
  int32_t *flat = nullptr;
  uint32_t *ring_quads = nullptr;  // phhp position -> 4 x packed position + term (kNoQuad: none)
  // Fused-path ring: units by group size (4, 2, 1 warps), operand images, destinations, and the
  // T' images with where their elements come from.
  RingUnit *ring_units = nullptr;
  double *ring_img = nullptr, *ring_tp = nullptr;
  int32_t *ring_to = nullptr, *ring_src = nullptr;
  int n_ring[3] = {0, 0, 0};
  int64_t n_tp = 0;
  bool ring_cols = false;               // the four-warp units hold only their columns of T'
  size_t ring_smem[3] = {0, 0, 0};  // dynamic shared memory of the groups' kernels
  double ring_flops[3] = {}, ring_bytes[3] = {};  // of the small, mid and large groups
  bool ring_paired = false;  // else the fused ring runs channel by channel
  double create_ms[5] = {};   // ccdgpu_profile::ms_create
  double loop_graph_ms = 0;   // ccdgpu_profile::ms_loop_graph
  int64_t *o_h = nullptr, *o_p = nullptr;
  double *v_h_hpp = nullptr, *v_phh_p = nullptr;
  double *old_h1pp_h2 = nullptr, *old_h2pp_h1 = nullptr, *diff_h2pp_h1 = nullptr;
  double *old_p1_p2hh = nullptr, *old_p2_p1hh = nullptr, *diff_p2_p1hh = nullptr;
  double *gath = nullptr;
  Control *ctl = nullptr;
  Control *h_ctl = nullptr;  // pinned mirror
  bool ctl_current = false;  // the mirror is what the device holds (but for err and the trace)
  int32_t *ticket = nullptr;  // assembly's last-CTA ticket
  double *e_out = nullptr;
  int32_t *err = nullptr;
  // The interaction model on the device (present when the problem carries one), and the
  // buffer of ccdgpu_reference_energy: n_sp bare energies in, n_sp normal-ordered + E_ref out.
  ModelDev md{};
  bool has_model = false;
  double *eps_io = nullptr;
  // Inputs that lack the antisymmetry in (a, b) or (i, j) that the packed kernels rely on: host V
  // blocks or tables, and the amplitudes last loaded.  The table path and the stage calls then form
  // t2Diff_pphh element by element (ccd_general.cuh); dmat_full: it has elements outside the quads.
  unsigned long long *irr = nullptr;  // largest element, and the check's mark
  bool irregular = false, irregular_t = false, dmat_full = false, v_generated = false;
  int64_t n_vhh = 0;         // hh x hh elements of all channels
  double *x_full = nullptr;  // X, hh x hh (allocated when first needed)

  cudaGraphExec_t graph = nullptr;
  int64_t kernels_per_graph = 0;
  bool profiling = false;
  bool inject_next_step = false;  // ccdgpu_inject_wait_timeout armed for the next step
  ccdgpu_profile prof{};
  double flops = 0, ladder_flops = 0, ladder_bytes = 0;
  int64_t launches = 0;

  // pp-ladder work lists (make_ladder_tiles), in their own allocation so the autotuner can
  // rebuild them.
  std::vector<ChanInfo> host_chans;
  int64_t n_list = 0;  // entries of the one-body segment lists
  ccdgpu_schedule schedule{};
  void *tile_mem = nullptr;
  size_t tile_bytes = 0;
  LadderRows *lrows = nullptr, *tc_lrows = nullptr;  // D planes per row tile
  double *d_planes = nullptr, *tc_planes = nullptr;
  // Tile counter and exit ticket of the FP64 ladder, then of the tensor-core ladder (zero
  // between launches).
  int32_t *sched = nullptr;

  // Mixed precision (nt bf16 terms per operand; 0 for an FP64 handle).
  int nt = 0;
  int n_tc_tiles = 0;
  LadderTile *tc_tiles = nullptr;
  int32_t *kcol = nullptr;  // pp index of the w-th c<d pair of each channel (pk_off + w)
  __nv_bfloat16 *v_tc = nullptr, *tkt_tc = nullptr;
  bool tc_tx = false;     // the tensor-core ladder does T X too
  double *tx_zero = nullptr;  // ... and the assembly then adds this in place of tx
  bool tc_stale = false;  // tkt_tc is not the image of the current amplitudes
  // Electron gas with V generated on the device: the tensor-core ladder generates its V
  // planes itself (no v_tc images) from these per-row / per-K-column codes and the q^2 table.
  bool tc_gen = false;
  VGenRow *vg_rows = nullptr;
  uint32_t *vg_cols = nullptr;
  double *vg_tab = nullptr;
  int64_t n_vtc = 0, n_tkttc = 0;  // plane strides (elements)
  size_t tc_smem = 0;
  double ladder_bytes_tc = 0;
  cudaGraphExec_t graph_tc = nullptr;
  int64_t kernels_per_graph_tc = 0;

  // Device solve loop: graphs of WHILE conditional nodes whose bodies are one iteration each
  // (loop64: FP64 iterations; loop_tc: mixed iterations, then FP64 ones).  loop_state: 0 not
  // built yet, 1 built, -1 unavailable (the batched graph replay is used instead).  A mixed
  // handle builds loop_tc first and loop64 only when a launch needs it (a solve still in FP64
  // iterations after a whole loop chunk); loop_pdl: the capture that worked used PDL launches.
  cudaGraphExec_t loop64 = nullptr, loop_tc = nullptr;
  int loop_state = 0;
  bool loop_pdl = true;
  int loop_capture = 0;  // while capturing a loop body: 1 FP64 body, 2 mixed body
  cudaGraphConditionalHandle loop_cond = 0;
  int64_t kernels_per_body64 = 0, kernels_per_body_tc = 0;
};

namespace {

int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return CCDGPU_OK;
  if (e == cudaErrorMemoryAllocation) return CCDGPU_ERR_OUT_OF_MEMORY;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return CCDGPU_ERR_NO_DEVICE;
  return CCDGPU_ERR_CUDA;
}

#define CK(call)                              \
  do {                                        \
    cudaError_t e_ = (call);                  \
    if (e_ != cudaSuccess) {                  \
      (void)cudaGetLastError();               \
      return cuda_status(e_);                 \
    }                                         \
  } while (0)

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

int find_pair(const ccdgpu_pair *list, int64_t n, uint64_t p, uint64_t q) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) / 2;
    if (list[mid].p < p || (list[mid].p == p && list[mid].q < q)) lo = mid + 1;
    else hi = mid;
  }
  if (lo < n && list[lo].p == p && list[lo].q == q) return (int)lo;
  return -1;
}

// Swap partner of every pair of a channel map sorted by (p, q): sw[k] = index of (q_k, p_k),
// -1 if absent.  One pass records where each first index's run starts (row[p], stamped with
// the channel so that the array is never cleared), then each partner is found by a scan of
// its run (a channel holds few pairs per first index), O(n) instead of n binary searches
// whose unpredictable branches dominated create on the largest bases.
struct SwapIndex {
  std::vector<int32_t> row;
  std::vector<uint32_t> stamp;
  uint32_t cur = 0;
  explicit SwapIndex(size_t nsp) : row(nsp, 0), stamp(nsp, 0) {}
  bool build(const ccdgpu_pair *m, int64_t n, int32_t *sw) {
    ++cur;
    for (int64_t k = 0; k < n; k++)
      if (k == 0 || m[k].p != m[k - 1].p) {
        if (m[k].p >= row.size()) return false;
        row[m[k].p] = (int32_t)k;
        stamp[m[k].p] = cur;
      }
    for (int64_t k = 0; k < n; k++) {
      const uint64_t a = m[k].p, b = m[k].q;
      sw[k] = -1;
      if (b >= row.size() || stamp[b] != cur) continue;
      for (int64_t j = row[b]; j < n && m[j].p == b && m[j].q <= a; j++)
        if (m[j].q == a) { sw[k] = (int32_t)j; break; }
    }
    return true;
  }
};

// Process-wide cache of device blocks given back by destroyed handles, by create's scratch
// and by schedule changes, reused by later allocations on the same device instead of
// cudaMalloc / cudaFree (hundreds of microseconds each; cudaFree also waits for the whole
// device).  Holds at most kCacheMax bytes; ccdgpu_release_cached_memory returns them.
constexpr size_t kCacheMax = size_t(16) << 30;

struct CachedBlock {
  int dev;
  void *p;
  size_t bytes;
};

struct BlockCache {
  std::mutex mu;
  std::vector<CachedBlock> blocks;
  size_t total = 0;
};

BlockCache &block_cache() {
  static BlockCache c;
  return c;
}

// Frees the cached blocks of device `dev` (all devices for dev < 0).
void release_cache(int dev) {
  BlockCache &C = block_cache();
  std::vector<CachedBlock> drop;
  {
    std::lock_guard<std::mutex> lock(C.mu);
    std::vector<CachedBlock> keep;
    for (const CachedBlock &b : C.blocks) (dev < 0 || b.dev == dev ? drop : keep).push_back(b);
    C.blocks.swap(keep);
    for (const CachedBlock &b : drop) C.total -= b.bytes;
  }
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess) cur = -1;
  for (const CachedBlock &b : drop) {
    cudaSetDevice(b.dev);
    cudaFree(b.p);
  }
  if (cur >= 0) cudaSetDevice(cur);
  (void)cudaGetLastError();
}

// A block of at least `bytes` on the current device: the smallest cached one that is at most
// twice as large (plus 64 MiB), else a new allocation, retried once after this device's cache
// has been freed.  *got receives the block's size.
cudaError_t dev_alloc(size_t bytes, void **p, size_t *got) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  BlockCache &C = block_cache();
  {
    std::lock_guard<std::mutex> lock(C.mu);
    int best = -1;
    for (int i = 0; i < (int)C.blocks.size(); i++) {
      const CachedBlock &b = C.blocks[i];
      if (b.dev == dev && b.bytes >= bytes && b.bytes <= 2 * bytes + (size_t(64) << 20) &&
          (best < 0 || b.bytes < C.blocks[best].bytes))
        best = i;
    }
    if (best >= 0) {
      *p = C.blocks[best].p;
      *got = C.blocks[best].bytes;
      C.total -= *got;
      C.blocks.erase(C.blocks.begin() + best);
      return cudaSuccess;
    }
  }
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    (void)cudaGetLastError();
    release_cache(dev);
    e = cudaMalloc(p, bytes);
  }
  *got = bytes;
  return e;
}

// Gives a block back (to the cache while it has room).  The caller has waited for every use.
void dev_free(void *p, size_t bytes) {
  if (!p) return;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) {
    BlockCache &C = block_cache();
    std::lock_guard<std::mutex> lock(C.mu);
    if (C.total + bytes <= kCacheMax) {
      C.blocks.push_back({dev, p, bytes});
      C.total += bytes;
      return;
    }
  }
  cudaFree(p);
}

// Page-locked Control mirrors, handed out from slabs of 64 that live for the process:
// cudaMallocHost / cudaFreeHost per handle cost more than a small create's own work.
struct CtlPool {
  std::mutex mu;
  std::vector<Control *> free;
};

CtlPool &ctl_pool() {
  static CtlPool p;
  return p;
}

Control *ctl_acquire() {
  CtlPool &pool = ctl_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  if (pool.free.empty()) {
    Control *slab = nullptr;
    if (cudaMallocHost(reinterpret_cast<void **>(&slab), 64 * sizeof(Control)) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    for (int i = 63; i >= 0; i--) pool.free.push_back(slab + i);
  }
  Control *c = pool.free.back();
  pool.free.pop_back();
  std::memset(c, 0, sizeof(Control));
  return c;
}

void ctl_release(Control *c) {
  CtlPool &pool = ctl_pool();
  std::lock_guard<std::mutex> lock(pool.mu);
  pool.free.push_back(c);
}

// Process-wide pool of the streams and events a handle uses (kStreams streams, kEvents events a
// set), by device: a create takes a set that a destroyed handle gave back instead of creating
// twenty objects, and a destroy returns its set (after its streams are idle) instead of
// destroying them.  Emptied by ccdgpu_release_cached_memory.
struct StreamPool {
  std::mutex mu;
  std::vector<StreamSet> sets;
};
StreamPool &stream_pool() {
  static StreamPool p;
  return p;
}
void destroy_set(StreamSet &ss) {
  for (cudaEvent_t &e : ss.ev)
    if (e) cudaEventDestroy(e);
  for (cudaStream_t &st : ss.s)
    if (st) cudaStreamDestroy(st);
}
// A set for the current device: from the pool, else new (events 0-9 time, the rest only order).
cudaError_t acquire_set(StreamSet &ss) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  {
    StreamPool &P = stream_pool();
    std::lock_guard<std::mutex> lock(P.mu);
    for (size_t i = 0; i < P.sets.size(); i++)
      if (P.sets[i].dev == dev) {
        ss = P.sets[i];
        P.sets.erase(P.sets.begin() + i);
        return cudaSuccess;
      }
  }
  ss.dev = dev;
  for (int k = 0; k < kStreams && e == cudaSuccess; k++)
    e = cudaStreamCreateWithFlags(&ss.s[k], cudaStreamNonBlocking);
  for (int k = 0; k < kEvents && e == cudaSuccess; k++)
    e = k < 10 ? cudaEventCreate(&ss.ev[k]) : cudaEventCreateWithFlags(&ss.ev[k], cudaEventDisableTiming);
  if (e != cudaSuccess) {
    destroy_set(ss);
    ss = StreamSet{};
  }
  return e;
}
void release_set(StreamSet &ss) {
  if (ss.dev < 0) return;
  StreamPool &P = stream_pool();
  std::lock_guard<std::mutex> lock(P.mu);
  P.sets.push_back(ss);
  ss = StreamSet{};
}
void release_stream_pool() {
  std::vector<StreamSet> drop;
  {
    StreamPool &P = stream_pool();
    std::lock_guard<std::mutex> lock(P.mu);
    drop.swap(P.sets);
  }
  int cur = 0;
  if (cudaGetDevice(&cur) != cudaSuccess) cur = -1;
  for (StreamSet &ss : drop) {
    cudaSetDevice(ss.dev);
    destroy_set(ss);
  }
  if (cur >= 0) cudaSetDevice(cur);
  (void)cudaGetLastError();
}

void release(ccdgpu_handle *h) {
  if (!h) return;
  // Cached blocks are handed to other handles: nothing of this one may still run on them.
  for (cudaStream_t st : h->sset.s)
    if (st) cudaStreamSynchronize(st);
  for (cudaGraphExec_t g : {h->graph, h->graph_tc, h->loop64, h->loop_tc})
    if (g) cudaGraphExecDestroy(g);
  h->graph = h->graph_tc = h->loop64 = h->loop_tc = nullptr;
  for (auto &b : h->allocs) dev_free(b.p, b.bytes);
  h->allocs.clear();
  dev_free(h->tile_mem, h->tile_bytes);
  h->tile_mem = nullptr;
  if (h->h_ctl) ctl_release(h->h_ctl);
  h->h_ctl = nullptr;
  // The streams are idle (synchronised above): their set goes back to the pool.
  if (cudaGetLastError() == cudaSuccess) release_set(h->sset);
  else destroy_set(h->sset);
}

// Bump allocator over one device allocation (256-byte aligned pieces), zero-filled on s0 at
// commit, except the pieces added with add_unset, which follow the others and which the
// caller writes in full before anything reads them.
struct Arena {
  size_t used = 0, unset = 0;
  std::vector<std::pair<void **, size_t>> reqs, unset_reqs;
  static size_t piece(size_t bytes) { return (std::max<size_t>(bytes, 1) + 255) & ~size_t(255); }
  template <typename T>
  void add(T **p, size_t count) {
    reqs.push_back({reinterpret_cast<void **>(p), used});
    used += piece(count * sizeof(T));
  }
  template <typename T>
  void add_unset(T **p, size_t count) {
    unset_reqs.push_back({reinterpret_cast<void **>(p), unset});
    unset += piece(count * sizeof(T));
  }
  int commit(ccdgpu_handle *h) {
    void *base = nullptr;
    size_t got = 0;
    CK(dev_alloc(used + unset, &base, &got));
    h->allocs.push_back({base, got});
    CK(cudaMemsetAsync(base, 0, used, h->s0));
    for (auto &r : reqs) *r.first = static_cast<char *>(base) + r.second;
    for (auto &r : unset_reqs) *r.first = static_cast<char *>(base) + used + r.second;
    return CCDGPU_OK;
  }
};

// Process-wide pinned staging for large host -> device uploads: two page-locked buffers of
// kStageChunk bytes, allocated on first use and kept until the process exits.  A copy from
// pageable memory is bounced by the driver through small internal buffers at a fraction of
// the link bandwidth; here host threads fill one pinned buffer while the copy engine drains
// the other.  Creates on other threads that find the buffers busy copy directly.
constexpr size_t kStageChunk = size_t(16) << 20;
constexpr size_t kStageMin = size_t(1) << 20;  // smaller copies go direct

struct Staging {
  std::mutex mu;
  char *buf = nullptr;  // 2 * kStageChunk, cudaHostAllocPortable
  bool failed = false;
};

Staging &staging() {
  static Staging s;
  return s;
}

// Host runs (src[i], bytes[i]) to consecutive device bytes from dst.  Large totals go through
// the staging buffers: each chunk is filled by host threads from pieces of the runs (a run may
// span chunks, a chunk may hold many runs) and moved by one device copy.
int copy_runs_to_device(ccdgpu_handle *h, char *dst, const std::vector<const char *> &src,
                        const std::vector<size_t> &bytes) {
  size_t total = 0;
  std::vector<size_t> at(src.size());
  for (size_t i = 0; i < src.size(); i++) {
    at[i] = total;
    total += bytes[i];
  }
  if (!total) return CCDGPU_OK;
  Staging &S = staging();
  std::unique_lock<std::mutex> lock(S.mu, std::defer_lock);
  if (total >= kStageMin && lock.try_lock()) {
    if (!S.buf && !S.failed &&
        cudaHostAlloc(reinterpret_cast<void **>(&S.buf), 2 * kStageChunk,
                      cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      S.buf = nullptr;
      S.failed = true;
    }
    if (S.buf) {
      cudaEvent_t ev[2] = {nullptr, nullptr};
      bool pending[2] = {false, false};
      cudaError_t e = cudaSuccess;
      for (int k = 0; k < 2 && e == cudaSuccess; k++)
        e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
      const int threads = std::max(1, std::min(omp_get_max_threads(), 16));
      size_t r0 = 0;  // first run that reaches into the current chunk
      struct Piece {
        size_t to;
        const char *from;
        size_t n;
      };
      std::vector<Piece> pieces;
      for (size_t off = 0, k = 0; off < total && e == cudaSuccess; off += kStageChunk, k ^= 1) {
        const size_t n = std::min(kStageChunk, total - off), end = off + n;
        char *stage = S.buf + k * kStageChunk;
        if (pending[k] && (e = cudaEventSynchronize(ev[k])) != cudaSuccess) break;
        // Pieces of at most n / threads bytes, so that one large run is copied in parallel too.
        const size_t piece = std::max<size_t>(size_t(64) << 10, (n + threads - 1) / threads);
        pieces.clear();
        while (at[r0] + bytes[r0] <= off) r0++;
        for (size_t i = r0; i < src.size() && at[i] < end; i++) {
          const size_t lo = std::max(at[i], off), hi = std::min(at[i] + bytes[i], end);
          for (size_t x = lo; x < hi; x += piece)
            pieces.push_back(Piece{x - off, src[i] + (x - at[i]), std::min(piece, hi - x)});
        }
#pragma omp parallel for num_threads(threads) schedule(dynamic, 8)
        for (int64_t j = 0; j < (int64_t)pieces.size(); j++)
          std::memcpy(stage + pieces[j].to, pieces[j].from, pieces[j].n);
        e = cudaMemcpyAsync(dst + off, stage, n, cudaMemcpyHostToDevice, h->s0);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k], h->s0);
        pending[k] = e == cudaSuccess;
      }
      // The buffers are free for the next upload only once their copies have completed.
      for (int k = 0; k < 2; k++) {
        if (pending[k]) {
          const cudaError_t w = cudaEventSynchronize(ev[k]);
          if (e == cudaSuccess) e = w;
        }
        if (ev[k]) cudaEventDestroy(ev[k]);
      }
      if (e != cudaSuccess) {
        (void)cudaStreamSynchronize(h->s0);
        (void)cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? CCDGPU_ERR_OUT_OF_MEMORY : CCDGPU_ERR_CUDA;
      }
      return CCDGPU_OK;
    }
  }
  for (size_t i = 0; i < src.size(); i++)
    if (bytes[i]) CK(cudaMemcpyAsync(dst + at[i], src[i], bytes[i], cudaMemcpyHostToDevice, h->s0));
  return CCDGPU_OK;
}

// Device bytes [src, src + total) to host memory dst, through the staging buffers for large
// totals, in slots of kD2HSlot bytes: the copy engine fills up to kD2HSlots slots ahead while
// host threads move each landed slot into dst, so only the last slot's host copy trails the
// transfer (a pageable device-to-host copy runs at about half of that).  Returns after every
// byte has arrived.
constexpr size_t kD2HSlot = size_t(4) << 20;
constexpr int kD2HSlots = (int)(2 * kStageChunk / kD2HSlot);

int copy_from_device(ccdgpu_handle *h, char *dst, const char *src, size_t total) {
  if (!total) return CCDGPU_OK;
  Staging &S = staging();
  std::unique_lock<std::mutex> lock(S.mu, std::defer_lock);
  if (total >= kStageMin && lock.try_lock()) {
    if (!S.buf && !S.failed &&
        cudaHostAlloc(reinterpret_cast<void **>(&S.buf), 2 * kStageChunk,
                      cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      S.buf = nullptr;
      S.failed = true;
    }
    if (S.buf) {
      cudaEvent_t ev[kD2HSlots] = {};
      cudaError_t e = cudaSuccess;
      for (int k = 0; k < kD2HSlots && e == cudaSuccess; k++)
        e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
      const int threads = std::max(1, std::min(omp_get_max_threads(), 16));
      const size_t nchunks = (total + kD2HSlot - 1) / kD2HSlot;
      auto issue = [&](size_t c) {
        const size_t off = c * kD2HSlot, n = std::min(kD2HSlot, total - off);
        const int k = (int)(c % kD2HSlots);
        cudaError_t r = cudaMemcpyAsync(S.buf + k * kD2HSlot, src + off, n,
                                        cudaMemcpyDeviceToHost, h->s0);
        if (r == cudaSuccess) r = cudaEventRecord(ev[k], h->s0);
        return r;
      };
      size_t issued = 0;
      for (; e == cudaSuccess && issued < std::min<size_t>(nchunks, kD2HSlots); issued++)
        e = issue(issued);
      for (size_t c = 0; c < nchunks && e == cudaSuccess; c++) {
        const int k = (int)(c % kD2HSlots);
        if ((e = cudaEventSynchronize(ev[k])) != cudaSuccess) break;
        const size_t off = c * kD2HSlot, n = std::min(kD2HSlot, total - off);
        const char *stage = S.buf + k * kD2HSlot;
        const size_t piece = std::max<size_t>(size_t(64) << 10, (n + threads - 1) / threads);
#pragma omp parallel for num_threads(threads) schedule(static)
        for (int64_t x = 0; x < (int64_t)((n + piece - 1) / piece); x++) {
          const size_t lo = (size_t)x * piece;
          std::memcpy(dst + off + lo, stage + lo, std::min(piece, n - lo));
        }
        if (issued < nchunks) e = issue(issued++);  // into the slot just emptied
      }
      (void)cudaStreamSynchronize(h->s0);
      for (int k = 0; k < kD2HSlots; k++)
        if (ev[k]) cudaEventDestroy(ev[k]);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return CCDGPU_ERR_CUDA;
      }
      return CCDGPU_OK;
    }
  }
  CK(cudaMemcpyAsync(dst, src, total, cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}

// One host array bound for its own device destination.
struct UploadPiece {
  char *dst;
  const char *src;
  size_t n;
};

// Many host arrays to their device destinations in one pass.  Large batches go through the
// staging buffers: host threads pack the next pieces into one buffer (16-byte aligned), then
// every piece is one asynchronous copy out of page-locked memory, so the copy engine runs
// them back to back while the host packs the other buffer.  Small batches are pageable copies.
// Returns after every byte has arrived, except with `hold` when the batch fit one buffer: the
// copies are then left in flight on s0 and the staging lock moves to *hold, which the caller
// keeps until s0 has passed them (no staging use by this thread meanwhile).
int copy_pieces_to_device(ccdgpu_handle *h, const std::vector<UploadPiece> &pcs,
                          std::unique_lock<std::mutex> *hold = nullptr) {
  size_t total = 0;
  for (const UploadPiece &p : pcs) total += p.n;
  if (!total) return CCDGPU_OK;
  Staging &S = staging();
  std::unique_lock<std::mutex> lock(S.mu, std::defer_lock);
  if (total >= kStageMin && lock.try_lock()) {
    if (!S.buf && !S.failed &&
        cudaHostAlloc(reinterpret_cast<void **>(&S.buf), 2 * kStageChunk,
                      cudaHostAllocPortable) != cudaSuccess) {
      (void)cudaGetLastError();
      S.buf = nullptr;
      S.failed = true;
    }
    if (S.buf) {
      cudaEvent_t ev[2] = {nullptr, nullptr};
      bool pending[2] = {false, false};
      cudaError_t e = cudaSuccess;
      for (int k = 0; k < 2 && e == cudaSuccess; k++)
        e = cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming);
      const int threads = std::max(1, std::min(omp_get_max_threads(), 16));
      struct Part {
        size_t off;  // in the staging buffer
        const char *src;
        char *dst;
        size_t n;
      };
      std::vector<Part> parts, work;
      size_t i = 0, done = 0;  // current piece, and its bytes already placed
      for (int k = 0; i < pcs.size() && e == cudaSuccess; k ^= 1) {
        char *stage = S.buf + k * kStageChunk;
        if (pending[k] && (e = cudaEventSynchronize(ev[k])) != cudaSuccess) break;
        parts.clear();
        size_t used = 0;
        while (i < pcs.size() && used < kStageChunk) {
          const size_t n = std::min(pcs[i].n - done, kStageChunk - used);
          if (n) parts.push_back(Part{used, pcs[i].src + done, pcs[i].dst + done, n});
          used = std::min(kStageChunk, used + ((n + 15) & ~size_t(15)));
          done += n;
          if (done == pcs[i].n) {
            i++;
            done = 0;
          }
        }
        // Host threads fill the buffer in slices of at most used / threads bytes.
        const size_t slice = std::max<size_t>(size_t(64) << 10, (used + threads - 1) / threads);
        work.clear();
        for (const Part &p : parts)
          for (size_t x = 0; x < p.n; x += slice)
            work.push_back(Part{p.off + x, p.src + x, nullptr, std::min(slice, p.n - x)});
#pragma omp parallel for num_threads(threads) schedule(dynamic, 4)
        for (int64_t j = 0; j < (int64_t)work.size(); j++)
          std::memcpy(stage + work[j].off, work[j].src, work[j].n);
        for (size_t j = 0; j < parts.size() && e == cudaSuccess; j++)
          e = cudaMemcpyAsync(parts[j].dst, stage + parts[j].off, parts[j].n,
                              cudaMemcpyHostToDevice, h->s0);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k], h->s0);
        pending[k] = e == cudaSuccess;
      }
      if (hold && e == cudaSuccess && total <= kStageChunk) {
        for (int k = 0; k < 2; k++)
          if (ev[k]) cudaEventDestroy(ev[k]);
        *hold = std::move(lock);
        return CCDGPU_OK;
      }
      for (int k = 0; k < 2; k++) {
        if (pending[k]) {
          const cudaError_t w = cudaEventSynchronize(ev[k]);
          if (e == cudaSuccess) e = w;
        }
        if (ev[k]) cudaEventDestroy(ev[k]);
      }
      if (e != cudaSuccess) {
        (void)cudaStreamSynchronize(h->s0);
        (void)cudaGetLastError();
        return CCDGPU_ERR_CUDA;
      }
      return CCDGPU_OK;
    }
  }
  for (const UploadPiece &p : pcs)
    if (p.n) CK(cudaMemcpyAsync(p.dst, p.src, p.n, cudaMemcpyHostToDevice, h->s0));
  return CCDGPU_OK;
}

// Copies per-channel host blocks (block k of `count[k]` elements at src[k]) to consecutive
// device positions; blocks adjacent in host memory form one run.
template <typename T>
int upload_runs(ccdgpu_handle *h, T *dst, const std::vector<const T *> &src,
                const std::vector<int64_t> &count) {
  std::vector<const char *> rs;
  std::vector<size_t> rl;
  for (size_t k = 0; k < src.size(); k++) {
    if (!count[k]) continue;
    const char *p = reinterpret_cast<const char *>(src[k]);
    const size_t n = (size_t)count[k] * sizeof(T);
    if (!rs.empty() && rs.back() + rl.back() == p) {
      rl.back() += n;
    } else {
      rs.push_back(p);
      rl.push_back(n);
    }
  }
  return copy_runs_to_device(h, reinterpret_cast<char *>(dst), rs, rl);
}

constexpr int kSched = 4;
int materialize_d(ccdgpu_handle *h);

// pp-ladder work tiles for a schedule (split factors of K per column class), in their own
// device allocation with the D planes they write; drops captured graphs, which hold the old
// lists.  An FP64 class is cut into K segments of at most 1 / (148 mul) of all the classes' chunks
// (mul: its split factor, three times that for the wide class, whose chunks take three times as
// long): longer tiles would leave SMs idle at the end, shorter ones cost planes (EG N=54
// |n|^2 <= 36: 171 us an iteration at mul = 1 to 4, 175 at 8, 180 at 16).  The tensor-core
// ladder's row tiles are cut into about tc_split_mul tiles per SM of at least four chunks.  Each
// segment writes its own plane, which the assembly adds in segment order (deterministic).
// The persistent CTAs claim tiles in list order from a launch-wide counter: FP64 tiles by class,
// wide first (the longest work per byte), then by decreasing cost, the tensor-core tiles by
// decreasing cost.  Cost = bytes streamed per K chunk x chunks, plus two chunks' worth for the
// pipeline fill and the epilogue.
int make_ladder_tiles(ccdgpu_handle *h, const ccdgpu_schedule &sch) {
  if (int rc = materialize_d(h)) return rc;  // it reads the planes that go away here
  const std::vector<ChanInfo> &chans = h->host_chans;
  const int mid_mul = sch.mid_split_mul > 0 ? sch.mid_split_mul : sch.wide_split_mul;
  int64_t chunks = 0, tc_blocks = 0;
  for (const ChanInfo &a : chans) {
    for (int mt = 0; mt < a.nmt; mt++) chunks += a.nkc - ladder_kc0(a.sym, mt);
    tc_blocks += a.nmt;
  }
  auto want_of = [&](int64_t mul, int64_t b, int64_t most) {
    return (int)std::min<int64_t>(most, std::max<int64_t>(1, ceil_div(mul * kSMs, std::max<int64_t>(b, 1))));
  };
  // Longest K segment of a class, in chunks.
  auto longest_of = [&](int64_t mul) { return (int)std::max<int64_t>(4, ceil_div(chunks, mul * kSMs)); };
  const int longest[3] = {longest_of(sch.thin_split_mul), longest_of(mid_mul),
                          longest_of(3 * sch.wide_split_mul)};
  const int want_tc = want_of(sch.tc_split_mul, tc_blocks, 32);
  struct Key {
    int64_t cost;
    int32_t cls, pos;
  };
  auto make = [&](bool tc, std::vector<LadderTile> &out, std::vector<LadderRows> &lrows,
                  int64_t &planes) {
    std::vector<LadderTile> tiles;
    std::vector<Key> keys;
    lrows.assign(h->n_row_tiles, LadderRows{0, 1, 0});
    planes = 0;
    for (int ai = 0; ai < h->n_act; ai++) {
      const ChanInfo &a = chans[ai];
      if (!a.nmt) continue;
      const int nk = tc ? a.nkct : a.nkc;
      auto segs = [&](int len) {
        return tc ? std::max(1, std::min(want_tc, len / 4))
                  : (int)ceil_div(len, longest[ladder_class(a.hs)]);
      };
      const int room = segs(nk);  // segments of the longest row tile
      const bool sym = !tc && a.sym;
      const int64_t plane = (int64_t)kMaxBM * a.hs;
      for (int mt = 0; mt < a.nmt; mt++) {
        const int rows = std::min(kMaxBM, a.pk - mt * kMaxBM), first = ladder_kc0(sym, mt);
        const int len = nk - first, nseg = segs(len);
        const int64_t base = planes + ladder_plane(sym, room, mt) * plane;
        const int direct = sym ? mt : 0;  // planes of the transposed blocks come first
        lrows[a.rt_off + mt] = LadderRows{base, direct + nseg, (int32_t)plane};
        for (int sg = 0; sg < nseg; sg++) {
          LadderTile t{};
          t.ch = ai; t.mt = mt; t.rows = rows;
          // Whole stages of two chunks.
          auto cut = [&](int k) { return k == nseg ? nk : first + 2 * (int)((int64_t)(len / 2) * k / nseg); };
          t.kc0 = cut(sg);
          t.nks = cut(sg + 1) - t.kc0;
          t.hk = a.hk; t.hs = a.hs; t.nb = a.nbt;
          t.sym = sym; t.nseg = room; t.pk = a.pk;
          t.out = base + (direct + sg) * plane;
          t.planes = planes;
          int64_t cost;
          if (tc) {
            const int rg = (rows + 7) / 8, ng = a.nbt / 8;
            t.a_base = a.vtc_base + (int64_t)mt * kTcBM * nk * kTcKC + (int64_t)t.kc0 * rg * kTcGroup;
            t.b_base = a.tkt_tc_base + (int64_t)t.kc0 * ng * kTcGroup;
            t.nkx = a.nkx; t.tmt_base = a.tmt_base; t.xt_base = a.xt_base;
            cost = (int64_t)(t.nks + 2) * (8 * rg + a.nbt);
          } else {
            t.a_base = a.vkt_base + ladder_chunk(sym, nk, mt, t.kc0, rows);
            t.b_base = a.q_off + (int64_t)t.kc0 * kBK * a.hs;
            t.ti_base = a.q_off + (int64_t)mt * kMaxBM * a.hs;
            cost = (int64_t)(t.nks + 2) * (ladder_as(rows) + a.hs);
          }
          keys.push_back(Key{cost, tc ? 0 : 2 - ladder_class(a.hs), (int32_t)tiles.size()});
          tiles.push_back(t);
        }
      }
      planes += ladder_plane(sym, room, a.nmt) * plane;
    }
    std::sort(keys.begin(), keys.end(), [](const Key &x, const Key &y) {
      return x.cls != y.cls ? x.cls < y.cls : x.cost != y.cost ? x.cost > y.cost : x.pos < y.pos;
    });
    out.resize(tiles.size());
    for (size_t i = 0; i < keys.size(); i++) out[i] = tiles[keys[i].pos];
  };
  std::vector<LadderTile> tiles, tc_tiles;
  std::vector<LadderRows> lrows, tc_lrows;
  int64_t planes = 0, tc_planes = 0;
  make(false, tiles, lrows, planes);
  if (h->nt) make(true, tc_tiles, tc_lrows, tc_planes);
  // Device copies: one allocation, written on s3, which s0 then waits for.  A schedule that
  // replaces another first waits for the handle's work in flight (the old lists may be in use);
  // the first one, made in create while the set-up kernels run on s0, has nothing to wait for,
  // so create's host work goes on beside them.
  const bool first = h->tile_mem == nullptr;
  if (!first) {
    CK(cudaStreamSynchronize(h->s0));
    CK(cudaStreamSynchronize(h->s2));
    CK(cudaStreamSynchronize(h->s3));
  }
  // Captured graphs hold the previous lists; they go before the block they point into.
  for (cudaGraphExec_t *g : {&h->graph, &h->graph_tc, &h->loop64, &h->loop_tc})
    if (*g) { cudaGraphExecDestroy(*g); *g = nullptr; }
  h->loop_state = 0;
  dev_free(h->tile_mem, h->tile_bytes);
  h->tile_mem = nullptr;
  h->tile_bytes = 0;
  h->tiles = h->tc_tiles = nullptr;
  h->lrows = h->tc_lrows = nullptr;
  h->d_planes = h->tc_planes = nullptr;
  h->sched = nullptr;
  h->n_tiles = h->n_tc_tiles = 0;
  Arena ar;
  ar.add(&h->tiles, tiles.size()); ar.add(&h->tc_tiles, tc_tiles.size());
  ar.add(&h->lrows, lrows.size()); ar.add(&h->tc_lrows, tc_lrows.size());
  ar.add(&h->sched, kSched);
  ar.add(&h->d_planes, planes); ar.add(&h->tc_planes, tc_planes);
  CK(dev_alloc(ar.used, &h->tile_mem, &h->tile_bytes));
  for (auto &r : ar.reqs) *r.first = static_cast<char *>(h->tile_mem) + r.second;
  // The planes are written in full (where the assembly reads them) by every ladder.
  CK(cudaMemsetAsync(h->sched, 0, kSched * sizeof(int32_t), h->s3));
  auto up = [&](auto *dst, const auto &v) -> int {
    if (v.empty()) return CCDGPU_OK;
    return cuda_status(cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(v[0]),
                                       cudaMemcpyHostToDevice, h->s3));
  };
  if (int rc = up(h->tiles, tiles)) return rc;
  if (int rc = up(h->tc_tiles, tc_tiles)) return rc;
  if (int rc = up(h->lrows, lrows)) return rc;
  if (int rc = up(h->tc_lrows, tc_lrows)) return rc;
  CK(cudaEventRecord(h->ev_fork2, h->s3));
  CK(cudaStreamWaitEvent(h->s0, h->ev_fork2, 0));
  if (!first) CK(cudaStreamSynchronize(h->s0));
  h->n_tiles = (int)tiles.size();
  h->n_cls[0] = h->n_cls[1] = h->n_cls[2] = 0;
  for (const LadderTile &t : tiles) h->n_cls[ladder_class(t.hs)]++;
  h->n_tc_tiles = (int)tc_tiles.size();
  h->schedule = sch;
  return CCDGPU_OK;
}

using TcKernel = void (*)(const LadderTile *, int, int32_t *, const __nv_bfloat16 *, int64_t,
                         const __nv_bfloat16 *, int64_t, double *, const Control *, int32_t *,
                         const ChanInfo *, const VGenRow *, const uint32_t *, const double *);
TcKernel tc_kernel_of(int nt, bool gen) {
  if (nt == 2) return gen ? pp_ladder_tc_kernel<2, true> : pp_ladder_tc_kernel<2, false>;
  return gen ? pp_ladder_tc_kernel<3, true> : pp_ladder_tc_kernel<3, false>;
}

// Host work lists of build(), kept per thread between creates: their pages are touched once
// (first-touch page faults of ~20 MB of fresh vectors were most of a warm create's host time
// on the largest bases), later creates only clear them.
struct BuildScratch {
  std::vector<int32_t> rowmap, kcol, pp_swap, hh_swap, prow, hcol, qrow, list;
  std::vector<int2> pp_pairs, hh_pairs, mod_ph, mod_hp, mod_dims;
  std::vector<RingPair> pairs;
  std::vector<RingUnit> units;
  std::vector<int32_t> mod_owner;
  std::vector<int2> mod_least, mod_named;
  std::vector<int4> vrows;
  std::vector<QuadCol> quad_cols;
  std::vector<QuadItem> quad_items;
  std::vector<ElemRange> ranges;
  std::vector<int64_t> o_t, o_m, o_m_scratch, list_cnt;
  std::vector<int4> gv_items, gvt_items;
  std::vector<int32_t> mod_gen_chan;
};
thread_local BuildScratch t_build_scratch;

double ms_since(std::chrono::steady_clock::time_point t0) {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

void ready_loop_graphs(ccdgpu_handle *h);
int launch_antisymmetry(ccdgpu_handle *h, const double *src);

int build(ccdgpu_handle *h, const ccdgpu_problem *P) {
  const auto t_build = std::chrono::steady_clock::now();
  const uint64_t nch = P->n_channels, nsp = P->n_sp, np = P->n_particles;
  h->nch = nch; h->nsp = nsp; h->np = np; h->npart = nsp - np;
  const ccdgpu_channel_dims *D = P->chan_dims, *MD = P->chan_mod_dims;
  // V_ON_THE_FLY: V_pppp is generated on the device from the model, P->v_pppp is not read.
  const bool on_the_fly =
      h->opt.v_mode == CCDGPU_V_ON_THE_FLY || h->opt.v_mode == CCDGPU_V_IN_LADDER;
  const ccdgpu_model *M = P->model;
  const bool model_ok = M && M->qn && M->kind >= CCDGPU_MODEL_PAIRING &&
                        M->kind <= CCDGPU_MODEL_ELECTRON_GAS &&
                        M->qn_stride >= (M->kind == CCDGPU_MODEL_PAIRING ? 2 : 5);
  if (on_the_fly && !model_ok) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (!on_the_fly && !P->v_pppp) return CCDGPU_ERR_INVALID_ARGUMENT;
  // No V_hhhh, V_hhpp and modified-channel V at all (all four NULL): generated on the device
  // from the model, like V_pppp in the on-the-fly mode.
  const int n_vblocks = (P->v_hhhh ? 1 : 0) + (P->v_hhpp ? 1 : 0) + (P->v_hpph_mod ? 1 : 0) +
                        (P->v_hphp_mod ? 1 : 0);
  if (n_vblocks != 0 && n_vblocks != 4) return CCDGPU_ERR_INVALID_ARGUMENT;
  const bool gen_v = n_vblocks == 0;
  if (gen_v && !model_ok) return CCDGPU_ERR_INVALID_ARGUMENT;
  // No loadMaps tables at all: the library derives them on the device from the channel maps.
  int n_maps = 0;
  for (int k = 0; k < 8; k++) n_maps += P->maps[k] ? 1 : 0;
  if (n_maps != 0 && n_maps != 8) return CCDGPU_ERR_INVALID_ARGUMENT;
  const bool derive_tables = n_maps == 0;

  BuildScratch &bs = t_build_scratch;
  std::vector<int64_t> &o_t = bs.o_t, &o_m = bs.o_m;
  o_t.assign(nch + 1, 0);
  o_m.assign(nch + 1, 0);
  for (uint64_t c = 0; c < nch; c++) {
    o_t[c + 1] = o_t[c] + (int64_t)(D[c].pp * D[c].hh);
    o_m[c + 1] = o_m[c] + (int64_t)(MD[c].ph * MD[c].hp);
  }
  h->n_t = o_t[nch];
  h->n_m = o_m[nch];
  if (h->n_t != h->n_m) return CCDGPU_ERR_BAD_TABLE;  // pphh <-> phhp must be a bijection
  if (h->n_t >= (int64_t)INT32_MAX / 2) return CCDGPU_ERR_UNSUPPORTED;
  const int64_t n_t = h->n_t;

  // ---- per-channel metadata (O(sum pp) host work) ----
  // Active channels (pp, hh > 0) and their pair offsets; then two passes over the channels,
  // run in parallel (each writes its own ranges): pairs, swap partners and validation, then the
  // packed-row and K index lists, whose offsets need every channel's counts from the first.
  std::vector<ChanInfo> chans;
  std::vector<uint64_t> act_chan;  // reference channel of each active channel
  std::vector<int64_t> a_pp_off(1, 0), a_hh_off(1, 0);
  for (uint64_t c = 0; c < nch; c++) {
    const int64_t pp = D[c].pp, hh = D[c].hh;
    if (!pp || !hh) continue;
    if (hh > kMaxHH || pp > (1 << 20)) return CCDGPU_ERR_UNSUPPORTED;
    if (!P->chan_maps[c].pp || !P->chan_maps[c].hh) return CCDGPU_ERR_INVALID_ARGUMENT;
    act_chan.push_back(c);
    a_pp_off.push_back(a_pp_off.back() + pp);
    a_hh_off.push_back(a_hh_off.back() + hh);
  }
  const int n_act = (int)act_chan.size();
  std::vector<int32_t> &rowmap = bs.rowmap, &kcol = bs.kcol;
  std::vector<int2> &pp_pairs = bs.pp_pairs, &hh_pairs = bs.hh_pairs;
  std::vector<int4> &vrows = bs.vrows;
  std::vector<int32_t> &pp_swap = bs.pp_swap, &hh_swap = bs.hh_swap, &prow = bs.prow,
                       &hcol = bs.hcol, &qrow = bs.qrow;
  pp_pairs.resize(a_pp_off[n_act]);
  pp_swap.resize(a_pp_off[n_act]);
  prow.resize(a_pp_off[n_act]);
  qrow.resize(a_pp_off[n_act]);
  hh_pairs.resize(a_hh_off[n_act]);
  hh_swap.resize(a_hh_off[n_act]);
  hcol.resize(a_hh_off[n_act]);
  std::vector<int32_t> a_pr(n_act), a_pk(n_act), a_hk(n_act);
  std::atomic<int> bad{0};
  const int host_threads = std::max(1, std::min(omp_get_max_threads(), 16));
#pragma omp parallel num_threads(host_threads)
  {
    SwapIndex swap_index(nsp);
#pragma omp for schedule(dynamic, 4)
    for (int ai = 0; ai < n_act; ai++) {
      const uint64_t c = act_chan[ai];
      const ccdgpu_pair *pm = P->chan_maps[c].pp, *hm = P->chan_maps[c].hh;
      const int64_t pp = D[c].pp, hh = D[c].hh, off = a_pp_off[ai], hoff = a_hh_off[ai];
      if (!swap_index.build(pm, pp, pp_swap.data() + off)) {
        bad = CCDGPU_ERR_BAD_TABLE;
        continue;
      }
      int pr = 0, pk = 0;
      for (int64_t k = 0; k < pp; k++) {
        const uint64_t a = pm[k].p, b = pm[k].q;
        if (a < np || b < np || a >= nsp || b >= nsp || pp_swap[off + k] < 0) {
          bad = CCDGPU_ERR_BAD_TABLE;
          break;
        }
        pp_pairs[off + k] = make_int2((int)a, (int)b);
        pk += a < b;
        pr += a <= b;
      }
      a_pr[ai] = pr;
      a_pk[ai] = pk;
      int hk = 0;
      for (int64_t k = 0; k < hh; k++) {
        const uint64_t i = hm[k].p, j = hm[k].q;
        const int sw = (i < np && j < np) ? find_pair(hm, hh, j, i) : -1;
        if (sw < 0) {
          bad = CCDGPU_ERR_BAD_TABLE;
          break;
        }
        hh_pairs[hoff + k] = make_int2((int)i, (int)j);
        hh_swap[hoff + k] = sw;
        hcol[hoff + k] = i < j ? 2 * hk++ : -1;  // the mirrors in the second pass
      }
      a_hk[ai] = hk;
    }
  }
  if (bad) return bad;
  std::vector<int64_t> a_row_off(n_act + 1, 0), a_pk_off(n_act + 1, 0), a_vrow_off(n_act + 1, 0);
  for (int ai = 0; ai < n_act; ai++) {
    a_row_off[ai + 1] = a_row_off[ai] + a_pr[ai];
    a_pk_off[ai + 1] = a_pk_off[ai] + a_pk[ai];
    a_vrow_off[ai + 1] = a_vrow_off[ai] + a_pk[ai];
  }
  rowmap.resize(on_the_fly ? 0 : a_row_off[n_act]);  // rows a <= b, as V_pppp is uploaded
  // Row items of the stored-V tiling kernels (not needed when V_pppp is generated).
  vrows.resize(on_the_fly ? 0 : a_vrow_off[n_act]);
  kcol.resize(a_pk_off[n_act]);
#pragma omp parallel for num_threads(host_threads) schedule(dynamic, 4)
  for (int ai = 0; ai < n_act; ai++) {
    const int64_t pp = D[act_chan[ai]].pp, off = a_pp_off[ai];
    const int64_t hh = D[act_chan[ai]].hh, hoff = a_hh_off[ai];
    int32_t *rm = on_the_fly ? nullptr : rowmap.data() + a_row_off[ai];
    int4 *vr = on_the_fly ? nullptr : vrows.data() + a_vrow_off[ai];
    int32_t *kc = kcol.data() + a_pk_off[ai];
    int pr = 0, pk = 0;
    for (int64_t k = 0; k < pp; k++) {
      const int a = pp_pairs[off + k].x, b = pp_pairs[off + k].y;
      prow[off + k] = qrow[off + k] = -1;
      if (a < b) {
        if (vr) vr[pk] = make_int4(ai, pk, pr, 0);
        prow[off + k] = 2 * pk;
        qrow[off + k] = (int32_t)(a_pk_off[ai] + pk);
        kc[pk++] = (int32_t)k;
      }
      if (rm && a <= b) rm[pr] = (int32_t)k;
      pr += a <= b;
    }
    for (int64_t k = 0; k < pp; k++)
      if (pp_pairs[off + k].x > pp_pairs[off + k].y) {
        prow[off + k] = prow[off + pp_swap[off + k]] + 1;
        qrow[off + k] = qrow[off + pp_swap[off + k]];
      }
    for (int64_t k = 0; k < hh; k++)
      if (hh_pairs[hoff + k].x > hh_pairs[hoff + k].y)
        hcol[hoff + k] = hcol[hoff + hh_swap[hoff + k]] + 1;
  }
  // Small systems: every channel one row tile of the tensor-core ladder.
  h->tc_tx = h->nt > 0;
  for (int ai = 0; ai < n_act; ai++)
    if (a_hk[ai] && a_pk[ai] > kTcBM) h->tc_tx = false;
  int64_t vhh_tot = 0, x_tot = 0, q_tot = 0, vt = 0, part_tot = 0, qcol_tot = 0;
  int64_t vraw_tot = 0;
  int64_t vtc = 0, tkttc = 0;
  std::vector<int64_t> vraw_off;
  for (int ai = 0; ai < n_act; ai++) {
    const uint64_t c = act_chan[ai];
    const int64_t pp = D[c].pp, hh = D[c].hh;
    const int pk = a_pk[ai], hk = a_hk[ai];
    ChanInfo ci{};
    ci.pp = (int)pp; ci.hh = (int)hh;
    ci.pk = pk; ci.hk = hk;
    ci.hs = quad_hs(hk);
    ci.pk_off = a_pk_off[ai];
    ci.pp_off = a_pp_off[ai]; ci.hh_off = a_hh_off[ai];
    ci.t_off = o_t[c];
    ci.vhh_off = vhh_tot; ci.x_off = x_tot; ci.q_off = q_tot; ci.vkt_base = vt;
    ci.qcol_off = qcol_tot;
    ci.vtc_base = vtc; ci.tkt_tc_base = tkttc;
    ci.part_off = part_tot;
    vhh_tot += hh * hh;
    qcol_tot += hk;
    if (pk && hk) {
      ci.nkc = (int)ceil_div(pk, kBK);
      ci.nmt = (int)ceil_div(pk, kMaxBM);
      ci.sym = hk <= kSymHK;  // stored V: unless it turns out not to be symmetric
      ci.rt_off = h->n_row_tiles;
      h->n_row_tiles += ci.nmt;
      ci.nhht = (int)ceil_div(pk, kHHRows);
      ci.nbt = tc_nb(hk);
      ci.nkct = (int)ceil_div(pk, kTcKC);
      vtc += (int64_t)ci.nkct * kTcGroup * ceil_div(pk, 8);
      tkttc += (int64_t)ci.nkct * (ci.nbt / 8) * kTcGroup;
      if (h->tc_tx) {
        ci.nkx = (int)ceil_div(hh, kTcKC);
        ci.tmt_base = tkttc;
        tkttc += (int64_t)ci.nkx * ceil_div(pk, 8) * kTcGroup;
        ci.xt_base = tkttc;
        tkttc += (int64_t)ci.nkx * (ci.nbt / 8) * kTcGroup;
      }
      x_tot += hk * ci.hs;
      q_tot += (int64_t)ci.nkc * kBK * ci.hs;
      // Stored V: room for the whole of it, should it not be symmetric.
      vt += ladder_chunk(on_the_fly && ci.sym, ci.nkc, ci.nmt - 1, ci.nkc, pk - (ci.nmt - 1) * kMaxBM);
      part_tot += (int64_t)ci.nhht * hk * hk;
    } else if (!on_the_fly) {
      vt += (int64_t)pk * pk;  // row-major, for ccd_general.cuh alone
    }
    vraw_off.push_back(vraw_tot);
    if (!on_the_fly) vraw_tot += (int64_t)a_pr[ai] * pp;  // rows a <= b only
    chans.push_back(ci);
  }
  // 2 x a packed position is 31-bit, 4 x one 32-bit (the ring's tables).  Amplitudes below the limit
  // above reach this only if their padding (rows to 16, 5 hole pairs to 12) quadruples them.
  if (q_tot * 2 >= INT32_MAX) return CCDGPU_ERR_UNSUPPORTED;
  // Records that the device fills in (hh_records_kernel): where each channel's start.
  // hh-ladder units: one per CTA (hk > 8) first, then one per warp; within each the largest
  // (rows x hk^2) first, so that the short ones fill in behind them: a channel's full slices and
  // its last, shorter one are sorted as runs, by class and cost.
  {
    struct Run {
      int32_t ai, n;
      bool warp, full;
      int64_t cost;
    };
    std::vector<Run> runs;
    runs.reserve(2 * n_act);
    for (int ai = 0; ai < n_act; ai++) {
      const ChanInfo &a = chans[ai];
      const int full = a.nmt ? a.pk / kHHRows : 0, rest = a.nmt ? a.pk % kHHRows : 0;
      const int64_t hk2 = (int64_t)a.hk * a.hk;
      if (full) runs.push_back(Run{ai, full, a.hk <= 8, true, kHHRows * hk2});
      if (rest) runs.push_back(Run{ai, 1, a.hk <= 8, false, rest * hk2});
      (a.hk > 8 ? h->n_hh_cta : h->n_hh_warp) += full + (rest ? 1 : 0);
    }
    std::stable_sort(runs.begin(), runs.end(), [](const Run &x, const Run &y) {
      if (x.warp != y.warp) return y.warp;
      return x.cost > y.cost;
    });
    int32_t at = 0;
    for (const Run &r : runs) {
      (r.full ? chans[r.ai].hht_first : chans[r.ai].hht_last) = at;
      at += r.n;
    }
  }
  // T X: the widest channels first, the short units fill in behind them.
  for (ChanInfo &a : chans) {
    a.hh_first = h->n_hh_out;
    if (a.nmt) h->n_hh_out += a.hk * a.hk;
  }
  for (const int rows : {16, 64, 128})
    for (ChanInfo &a : chans)
      if (a.nmt && tx_rows(a.hk) == rows) {
        a.tx_first = h->n_tx;
        h->n_tx += (int)(ceil_div(a.pk, rows) * ceil_div(a.hk, 16));
      }
  h->n_q = q_tot;
  h->n_act = n_act;
  h->n_vhh = vhh_tot;
  h->v_generated = on_the_fly;
  const int64_t pp_tot = a_pp_off[n_act], hh_tot = a_hh_off[n_act];
  // Per orbital w, the strict pairs that hold w, in the order of the ordered pairs whose first
  // index is w (particles: rows of r, holes: entries of s): a counting sort.  The pp elements (first index a particle)
  // are split into one contiguous range per host thread: per-thread bucket counts, then each
  // thread places its range from its own start in every bucket, so a bucket keeps ascending
  // element order.  The hh elements (first index a hole, buckets of their own) follow serially.
  std::vector<int64_t> list_off(nsp + 1, 0);
  std::vector<int32_t> &list = bs.list;
  {
    std::vector<int64_t> &cnt = bs.list_cnt;  // [thread][orbital]: counts, then start offsets
    cnt.assign((size_t)host_threads * nsp, 0);
    int team = 1;
#pragma omp parallel num_threads(host_threads)
    {
#pragma omp single
      team = omp_get_num_threads();
      const int t = omp_get_thread_num();
      const int64_t lo = pp_tot * t / team, hi = pp_tot * (t + 1) / team;
      int64_t *c = cnt.data() + (size_t)t * nsp;
      for (int64_t e = lo; e < hi; e++) c[pp_pairs[e].x] += qrow[e] >= 0;
#pragma omp barrier
#pragma omp single
      {
        for (int64_t e = 0; e < hh_tot; e++) list_off[hh_pairs[e].x + 1] += hcol[e] >= 0;
        for (uint64_t w = 0; w < nsp; w++) {
          int64_t s = 0;
          for (int u = 0; u < team; u++) s += cnt[(size_t)u * nsp + w];
          list_off[w + 1] += s;
        }
        for (uint64_t w = 0; w < nsp; w++) list_off[w + 1] += list_off[w];
        list.resize(list_off[nsp]);
        for (uint64_t w = 0; w < nsp; w++) {
          int64_t at = list_off[w];
          for (int u = 0; u < team; u++) {
            const int64_t n = cnt[(size_t)u * nsp + w];
            cnt[(size_t)u * nsp + w] = at;
            at += n;
          }
        }
      }
      for (int64_t e = lo; e < hi; e++)
        if (qrow[e] >= 0) list[c[pp_pairs[e].x]++] = qrow[e];
    }
    std::vector<int64_t> &cur = bs.o_m_scratch;
    cur.assign(list_off.begin(), list_off.end() - 1);
    for (const ChanInfo &a : chans)
      for (int64_t e = a.hh_off; e < a.hh_off + a.hh; e++)
        if (hcol[e] >= 0) list[cur[hh_pairs[e].x]++] = (int32_t)(a.qcol_off + (hcol[e] >> 1));
  }
  h->n_list = list_off[nsp];

  // Modified channels: small ones (one warp each) first, then one group per padded size
  // (32, 48, 64, 80; one CTA per channel).
  std::vector<ModInfo> mods, mods_pad[4];
  std::vector<int2> &mod_dims = bs.mod_dims;
  mod_dims.resize(nch);
  int64_t y_tot = 0;
  std::vector<const double *> src_hpph, src_hphp;
  std::vector<int64_t> cnt_hpph, cnt_hphp;
  std::vector<ModGen> mod_gen;        // modified channels in channel order
  std::vector<int32_t> &mod_gen_chan = bs.mod_gen_chan;  // ... and their channel slots
  mod_gen_chan.clear();
  std::vector<int2> &mod_ph = bs.mod_ph, &mod_hp = bs.mod_hp;  // ... their ph' (b, j), hp' (i, a) pairs
  std::vector<int2> &mod_least = bs.mod_least;
  const bool fused = h->opt.path == CCDGPU_PATH_FUSED;
  bool mod_maps = true;  // the problem carries the ph' and hp' pair lists
  const bool lists_needed = derive_tables || gen_v;
  for (uint64_t c = 0; c < nch; c++) {
    const int64_t ph = MD[c].ph, hp = MD[c].hp;
    mod_dims[c] = make_int2((int)ph, (int)hp);
    if (!ph || !hp) continue;
    if (ph > kRingMax || hp > kRingMax) return CCDGPU_ERR_UNSUPPORTED;  // ring tiles
    ModInfo m{};
    m.ph = (int)ph; m.hp = (int)hp; m.m_off = o_m[c]; m.y_off = y_tot;
    // The pairs themselves are copied in parallel after this loop.
    if (!P->chan_mod_maps || !P->chan_mod_maps[c].ph || !P->chan_mod_maps[c].hp) {
      if (lists_needed) return CCDGPU_ERR_INVALID_ARGUMENT;
      mod_maps = false;
    }
    const int64_t ph0 = mod_gen.empty() ? 0 : mod_gen.back().ph_off + mod_gen.back().ph;
    const int64_t hp0 = mod_gen.empty() ? 0 : mod_gen.back().hp_off + mod_gen.back().hp;
    mod_gen.push_back(ModGen{(int)ph, (int)hp, m.m_off, m.y_off, ph0, hp0});
    mod_gen_chan.push_back((int32_t)c);
    if (!gen_v) {
      if (!P->v_hpph_mod[c] || !P->v_hphp_mod[c]) return CCDGPU_ERR_INVALID_ARGUMENT;
      src_hpph.push_back(P->v_hpph_mod[c]); cnt_hpph.push_back(ph * hp);
      src_hphp.push_back(P->v_hphp_mod[c]); cnt_hphp.push_back(hp * hp);
    }
    y_tot += hp * hp;
    const int64_t w = std::max(ph, hp);
    if (w <= kRingSmall) mods.push_back(m);
    else mods_pad[w <= 32 ? 0 : w <= 48 ? 1 : w <= 64 ? 2 : 3].push_back(m);
  }
  const bool lists_used = !mod_gen.empty() && (fused || lists_needed);
  mod_ph.resize(lists_used ? mod_gen.back().ph_off + mod_gen.back().ph : 0);
  mod_hp.resize(lists_used ? mod_gen.back().hp_off + mod_gen.back().hp : 0);
  if (lists_used) {
    const std::vector<int32_t> &mod_chan = mod_gen_chan;
    std::atomic<int> bad_mod{0};
    // Slots (a - np) * np + i of the smallest ph' and hp' pair; -1: an entry is missing.
    auto find_least = [&](int64_t g) {
      const ModGen &m = mod_gen[g];
      int32_t p = INT32_MAX, q = INT32_MAX;
      for (int k = 0; k < m.ph; k++) {
        const int2 ai = mod_ph[m.ph_off + k];
        p = std::min(p, ai.x < 0 ? -1 : (ai.x - (int)np) * (int)np + ai.y);
      }
      for (int k = 0; k < m.hp; k++) {
        const int2 ia = mod_hp[m.hp_off + k];
        q = std::min(q, ia.x < 0 ? -1 : (ia.y - (int)np) * (int)np + ia.x);
      }
      mod_least[g] = make_int2(p, q);
    };
    mod_least.resize(mod_gen.size());
    if (mod_maps) {
#pragma omp parallel for num_threads(host_threads) schedule(dynamic, 16)
      for (int64_t g = 0; g < (int64_t)mod_gen.size(); g++) {
        const ModGen &mg = mod_gen[g];
        const ccdgpu_pair *phm = P->chan_mod_maps[mod_chan[g]].ph, *hpm = P->chan_mod_maps[mod_chan[g]].hp;
        for (int64_t k = 0; k < mg.ph; k++) {
          if (phm[k].p < np || phm[k].p >= nsp || phm[k].q >= np) bad_mod = 1;
          mod_ph[mg.ph_off + k] = make_int2((int)phm[k].p, (int)phm[k].q);
        }
        for (int64_t k = 0; k < mg.hp; k++) {
          if (hpm[k].p >= np || hpm[k].q < np || hpm[k].q >= nsp) bad_mod = 1;
          mod_hp[mg.hp_off + k] = make_int2((int)hpm[k].p, (int)hpm[k].q);
        }
        find_least(g);
      }
      if (bad_mod && lists_needed) return CCDGPU_ERR_BAD_TABLE;
    }
    if (fused && (!mod_maps || bad_mod)) {
      // A problem with tables and V blocks but without usable pair lists: the ai_jb table names the
      // (a, i) of every ph' row and the (j, b) of every hp' column.
      std::fill(mod_ph.begin(), mod_ph.end(), make_int2(-1, -1));
      std::fill(mod_hp.begin(), mod_hp.end(), make_int2(-1, -1));
      std::vector<int64_t> gen_of(nch, -1);
      for (size_t g = 0; g < mod_gen.size(); g++) gen_of[mod_chan[g]] = (int64_t)g;
      auto put = [](int2 &at, int x, int y) {  // rows and columns recur in other channels
        const int2 v = make_int2(x, y);
        int64_t bits;
        std::memcpy(&bits, &v, sizeof(bits));
        __atomic_store_n(reinterpret_cast<int64_t *>(&at), bits, __ATOMIC_RELAXED);
      };
      std::atomic<int> rc_maps{0};
#pragma omp parallel for num_threads(host_threads) schedule(dynamic, 4)
      for (int ai = 0; ai < n_act; ai++) {
        const ccdgpu_chain_index *mp = P->maps[CCDGPU_MAP_AI_JB][act_chan[ai]];
        const ChanInfo &a = chans[ai];
        if (!mp) rc_maps = CCDGPU_ERR_INVALID_ARGUMENT;
        for (int64_t e = 0; mp && e < (int64_t)a.pp * a.hh; e++) {
          const int2 ab = pp_pairs[a.pp_off + e / a.hh], ij = hh_pairs[a.hh_off + e % a.hh];
          const int64_t g = mp[e].channel < nch ? gen_of[mp[e].channel] : -1;
          if (g < 0 || mp[e].row >= (uint64_t)mod_gen[g].ph ||
              mp[e].column >= (uint64_t)mod_gen[g].hp) {
            rc_maps = CCDGPU_ERR_BAD_TABLE;
            break;
          }
          put(mod_ph[mod_gen[g].ph_off + mp[e].row], ab.x, ij.x);
          put(mod_hp[mod_gen[g].hp_off + mp[e].column], ij.y, ab.y);
        }
      }
      if (rc_maps) return rc_maps;
      for (size_t g = 0; g < mod_gen.size(); g++) find_least(g);
    }
  }
  // Fused-path ring: each channel with its transpose, the channel whose ph' pairs are this one's
  // hp' pairs exchanged (the first of the two in channel order names the pair).
  // Named by the smallest pair of each list; that the lists agree in full is checked on the device
  // (ring_image_kernel).  Tables from the host may describe blocks that do not pair up; then (and if
  // their rows and columns turn out not to be those of the lists) the ring runs channel by channel,
  // as on the table path.
  std::vector<RingPair> &pairs = bs.pairs;
  std::vector<RingUnit> &units = bs.units;
  pairs.clear();
  units.clear();
  int64_t img_tot = 0, tp_tot = 0, to_tot = 0;
  auto pair_up = [&]() {
    const int n = (int)mod_gen.size();
    // The channel whose hp' list has a slot as its smallest; entries of earlier creates are told by
    // their channel's list.
    std::vector<int32_t> &owner = bs.mod_owner;
    std::vector<int2> &named = bs.mod_named;  // channels that name their pair, their transposes
    owner.resize(np * h->npart);
    named.clear();
    for (int g = 0; g < n; g++)
      if (mod_least[g].y >= 0) owner[mod_least[g].y] = g;
    auto partner = [&](int g) {
      const int slot = mod_least[g].x, o = slot >= 0 ? owner[slot] : -1;
      return o >= 0 && o < n && mod_least[o].y == slot ? o : -1;
    };
    // The largest first, so that the short ones fill in behind them: counted by tiles of 16 x 16.
    constexpr int kMaxTiles = (kRingMax / 16) * (kRingMax / 16);
    auto tiles_of = [](const ModGen &m) { return pad16(m.ph) / 16 * (pad16(m.hp) / 16); };
    int at[kMaxTiles + 1] = {};
    for (int g = 0; g < n; g++) {
      const int other = partner(g);
      if (other < 0 || partner(other) != g) return false;
      const ModGen &m = mod_gen[g], &o = mod_gen[other];
      if (o.hp != m.ph || o.ph != m.hp) return false;
      if (other < g) continue;  // named by its transpose
      named.push_back(make_int2(g, other));
      at[tiles_of(m)]++;
    }
    for (int t = kMaxTiles, sum = 0; t >= 0; t--) {
      const int c = at[t];
      at[t] = sum;
      sum += c;
    }
    pairs.resize(named.size());
    for (const int2 &go : named) {
      const ModGen &m = mod_gen[go.x], &o = mod_gen[go.y];
      RingPair &r = pairs[at[tiles_of(m)]++];
      r = RingPair{};
      r.ph = m.ph; r.hp = m.hp;
      r.ph_off = (int)m.ph_off; r.hp_off = (int)m.hp_off;
      r.other = mod_gen_chan[go.y];
      r.self = go.x == go.y;
      r.m_off = m.m_off; r.a_off = m.y_off; r.b_src = o.y_off;
      r.c_src = gen_v ? -1 : o.m_off;
      r.g = ring_group(r.ph, r.hp);
    }
    return true;
  };
  h->ring_paired = fused && pair_up();
  if (!h->ring_paired) {
    pairs.clear();
    if (fused && derive_tables) return CCDGPU_ERR_BAD_TABLE;  // no tables could fit such lists
  } else {
    // Warps of a pair's units by its width; a group that does not fill the SMs joins the next wider
    // one: a launch and a graph branch less (pairing: 0.1 ms less in create, mixed 0.2 ms).
    auto units_of = [](const RingPair &r) { return ceil_div((r.hp + 7) / 8, kPairNC); };
    int64_t group_units[5] = {};
    for (const RingPair &r : pairs) group_units[r.g] += units_of(r);
    for (int g : {1, 2}) {
      const int to = group_units[2 * g] ? 2 * g : 4;
      if (group_units[g] >= kSMs || !group_units[to]) continue;
      for (RingPair &r : pairs)
        if (r.g == g) r.g = to;
      group_units[to] += group_units[g];
      group_units[g] = 0;
    }
    for (RingPair &r : pairs) {
      const int64_t p = pad16(r.ph), q = pad16(r.hp), n8 = (r.hp + 7) / 8;
      r.tp = tp_tot;
      tp_tot += p * (q + 4);
      r.b_img = img_tot;
      r.c_img = r.b_img + p * p;
      r.a_img = r.c_img + q * p;
      img_tot = r.a_img + q * 8 * n8;
      r.to_img = to_tot;
      to_tot += p * 8 * n8;
    }
    // Units: the pair's column tiles in blocks of at most kPairNC, as equal as they come.
    for (int k = 0; k < 3; k++) {
      const size_t first = units.size();
      for (const RingPair &r : pairs) {
        if (r.g != 4 >> k) continue;
        const int n8 = (r.hp + 7) / 8, blocks = (n8 + kPairNC - 1) / kPairNC;
        for (int q = 0; q < blocks; q++)
          units.push_back({r.ph, r.hp, n8 * q / blocks, n8 * (q + 1) / blocks - n8 * q / blocks,
                           r.tp, r.a_img, r.b_img, r.c_img, r.to_img});
      }
      h->n_ring[k] = (int)(units.size() - first);
    }
    h->ring_cols = ring_cols(h->n_ring[0]);
    for (const RingPair &r : pairs) {
      const int n8 = (r.hp + 7) / 8, nt = (int)ceil_div(n8, units_of(r));  // of the widest unit
      size_t &smem = h->ring_smem[r.g == 4 ? 0 : r.g == 2 ? 1 : 2];
      smem = std::max(smem, (r.g == 1 ? 4 : 1) * sizeof(double) *
                                ring_unit_smem(r.g, r.g == 4 && h->ring_cols, pad16(r.ph),
                                               pad16(r.hp), nt));
      const int k = r.g == 1 ? 0 : r.g == 2 ? 1 : 2;
      const double e = (double)r.ph * r.hp;
      h->ring_flops[k] += 2.0 * e * (2.0 * r.hp + r.ph);
      h->ring_bytes[k] += 28.0 * e + 8.0 * ((double)r.hp * r.hp + (double)r.ph * r.ph);
    }
  }
  h->n_tp = tp_tot;
  // Largest channels first within a group, so that the short ones fill in behind them.
  auto by_work = [](const ModInfo &x, const ModInfo &y) {
    return (int64_t)x.ph * x.hp * x.hp > (int64_t)y.ph * y.hp * y.hp;
  };
  h->n_mod_small = (int)mods.size();
  for (int k = 0; k < 4; k++) {
    std::stable_sort(mods_pad[k].begin(), mods_pad[k].end(), by_work);
    h->n_mod_pad[k] = (int)mods_pad[k].size();
    mods.insert(mods.end(), mods_pad[k].begin(), mods_pad[k].end());
  }
  h->n_mod = (int)mods.size();

  std::vector<int64_t> o_h(np + 1, 0), o_p(h->npart + 1, 0);
  for (uint64_t k = 0; k < np; k++) o_h[k + 1] = o_h[k] + (int64_t)P->three_body_dims[k].hpp;
  for (uint64_t a = 0; a < h->npart; a++)
    o_p[a + 1] = o_p[a] + (int64_t)P->three_body_dims[np + a].phh;
  h->n_h = o_h[np];
  h->n_p = o_p[h->npart];
  if (h->n_h != n_t || h->n_p != n_t) return CCDGPU_ERR_BAD_TABLE;
  // Three-body V of the table path: from the host, or generated with the other V blocks when
  // the problem carries none of them and the handle runs the table path (the fused path reads
  // none: its one-body sums come from the hh ladder's row dots).
  const bool gen_v3 = gen_v && !P->v_h_hpp && !P->v_phh_p && h->opt.path == CCDGPU_PATH_TABLES;
  h->have_3body = (P->v_h_hpp && P->v_phh_p) || gen_v3;

  h->host_chans = chans;

  std::vector<ElemRange> &ranges = bs.ranges;
  ranges.clear();
  const int64_t per = (int64_t)kAsmThreads * kAsmPerThread;
  for (int ai = 0; ai < h->n_act; ai++) {
    const ChanInfo &a = chans[ai];
    const int64_t n = (int64_t)a.pp * a.hh;
    for (int64_t e = 0; e < n; e += per) ranges.push_back({ai, 0, a.t_off + e, a.t_off + std::min(n, e + per)});
  }
  h->n_ranges = (int)ranges.size();
  // Fused assembly: quads (strict packed row a < b, strict hole pair i < j) per channel, their
  // static tables, and work items of up to kQuadPerItem quads of one channel.
  std::vector<QuadCol> &quad_cols = bs.quad_cols;
  std::vector<QuadItem> &quad_items = bs.quad_items;
  quad_cols.clear();
  quad_items.clear();
  // Rows: the packed rows with a < b (pk of them per channel), filled in parallel below;
  // columns (i < j) and work items here.
  for (int ai = 0; ai < h->n_act; ai++) {
    const ChanInfo &a = chans[ai];
    for (int j = 0; j < a.hh; j++) {
      const int2 pij = hh_pairs[a.hh_off + j];
      if (pij.x >= pij.y) continue;  // i = j: zero column; i > j: the mirror of (j, i)
      QuadCol c{};
      c.c_ij = j; c.c_ji = hh_swap[a.hh_off + j]; c.i = pij.x; c.j = pij.y;
      c.eij = P->sp_energy[pij.x] + P->sp_energy[pij.y];
      quad_cols.push_back(c);
    }
    const int64_t nq = (int64_t)a.pk * a.hk;
    if (nq >= ((int64_t)1 << 31) / 2) return CCDGPU_ERR_UNSUPPORTED;
    for (int64_t q = 0; q < nq; q += kQuadPerItem)
      quad_items.push_back({ai, (int32_t)q, (int32_t)std::min<int64_t>(nq, q + kQuadPerItem),
                            a.hk, a.hs, a.rt_off, a.q_off, a.pk_off, a.qcol_off});
  }
  h->n_quad_rows = a_pk_off[n_act];  // built on the device (quad_rows_kernel)

  h->host_chans = chans;
  h->n_quad_items = (int)quad_items.size();
  // Persistent assembly grid: kAsmCTAsPerSM resident CTAs per SM at most (one CTA if there is no quad,
  // for the energy and the stop rule).
  h->n_asm_blocks = h->n_act ? std::max(1, std::min(h->n_quad_items, kAsmCTAsPerSM * kSMs)) : 0;

  // Work estimate (reference GEMM flops) for roofline reporting.
  double fl = 0, lf = 0, vbp = 0;
  for (const ChanInfo &a : chans) {
    lf += 2.0 * a.pp * a.pp * a.hh;
    fl += 2.0 * a.pp * a.pp * a.hh + 4.0 * a.pp * a.hh * (double)a.hh;
    if (a.hk) vbp += 8.0 * a.pk * (double)a.pk;
  }
  for (const ModInfo &m : mods) fl += 4.0 * m.ph * (double)m.hp * m.hp;
  h->flops = fl; h->ladder_flops = lf;
  // Bytes one pp-ladder launch must move: packed V (of a symmetric channel one triangle), the
  // packed amplitudes in and D out.
  double lb = vbp;
  for (const ChanInfo &a : chans)
    lb += 16.0 * (double)a.pk * a.hk - (a.sym ? 4.0 * a.pk * (a.pk - 1.0) : 0.0);
  h->ladder_bytes = lb;
  double lbt = 0;
  for (const ChanInfo &a : chans)
    if (a.hk)
      lbt += 2.0 * h->nt * ((double)a.pk * a.pk + (double)a.pk * a.hk) + 8.0 * a.pk * (double)a.hk;
  h->ladder_bytes_tc = lbt;

  // Tensor-core ladder with V generated in the kernel (electron gas, on-the-fly V, momenta
  // |n_i| <= 6 so that q^2 <= 432): per packed row u the codes of a and b, per K
  // index w the code of c (momentum bytes biased by 64, spin in byte 3), and the
  // direct term by q^2.
  std::vector<VGenRow> vg_rows;
  std::vector<uint32_t> vg_cols;
  std::vector<double> vg_tab;
  if (h->opt.v_mode == CCDGPU_V_IN_LADDER && h->nt && model_ok &&
      M->kind == CCDGPU_MODEL_ELECTRON_GAS) {
    int nmax = 0;
    for (uint64_t o = 0; o < nsp; o++)
      for (int i = 0; i < 3; i++) nmax = std::max(nmax, std::abs(M->qn[o * M->qn_stride + i]));
    if (nmax <= 6) {
      h->tc_gen = true;
      auto code = [&](int o) {
        const int32_t *q = M->qn + (int64_t)o * M->qn_stride;
        return (uint32_t)(q[0] + 64) | ((uint32_t)(q[1] + 64) << 8) |
               ((uint32_t)(q[2] + 64) << 16) | ((uint32_t)(q[3] > 0 ? kVGenSpin : 0) << 24);
      };
      vg_rows.resize(kcol.size());
      vg_cols.resize(kcol.size());
      for (const ChanInfo &a : chans)
        for (int u = 0; u < a.pk; u++) {
          const int2 ab = pp_pairs[a.pp_off + kcol[a.pk_off + u]];
          vg_rows[a.pk_off + u] = VGenRow{code(ab.x), code(ab.y)};
          vg_cols[a.pk_off + u] = code(ab.x);
        }
      // w(q^2) = e^2 / L^3 * 4 pi / (2 pi / L)^2 q^2, zero for q = 0 (ElectronGasSPBasis.cpp:
      // 453-466 as a function of q^2).
      const double L = M->params[0], e_sq = M->params[1];
      vg_tab.assign(kTcGenTab, 0.0);
      for (int q2 = 1; q2 <= 3 * 12 * 12; q2++) {  // beyond: spins differ, zero
        const double rel = (2 * M_PI / L) * (2 * M_PI / L) * q2;
        vg_tab[q2] = e_sq / (L * L * L) * 4 * M_PI / rel;
      }
      // The ladder then moves no V bytes: the T operand image and D.
      double lbg = 0;
      for (const ChanInfo &a : chans) lbg += (2.0 * h->nt + 8.0) * a.pk * (double)a.hk;
      h->ladder_bytes_tc = lbg;
    }
  }

  // ---- one device allocation ----
  h->create_ms[0] = ms_since(t_build);
  Arena ar;
  ar.add(&h->chans, chans.size()); ar.add(&h->mods, mods.size());
  ar.add(&h->hh_tiles, h->n_hh_cta + h->n_hh_warp); ar.add(&h->hh_out, h->n_hh_out);
  ar.add(&h->tx_tiles, h->n_tx);
  ar.add(&h->ranges, ranges.size());
  ar.add(&h->pp_pairs, pp_pairs.size()); ar.add(&h->hh_pairs, hh_pairs.size());
  ar.add(&h->pp_swap, pp_swap.size()); ar.add(&h->hh_swap, hh_swap.size());
  ar.add(&h->list_off, list_off.size()); ar.add(&h->list, list.size());
  ar.add(&h->prow, prow.size()); ar.add(&h->hcol, hcol.size());
  ar.add(&h->part, part_tot);
  ar.add(&h->tq[0], q_tot); ar.add(&h->tq[1], q_tot); ar.add(&h->vq, q_tot);

  ar.add(&h->eps, nsp);
  // Generated V images are written in full (padding included) by the V generators.
  ar.add(&h->v_pphh, n_t); ar.add(&h->v_hhhh, vhh_tot);
  if (on_the_fly) ar.add_unset(&h->v_t, vt);
  else ar.add(&h->v_t, vt);
  ar.add(&h->v_hpph, h->n_m); ar.add(&h->v_hphp, y_tot);
  ar.add(&h->flat, (size_t)8 * n_t); ar.add(&h->ring_quads, n_t); ar.add(&h->r_quad, fused ? 2 * q_tot : 0);
  ar.add(&h->ring_units, units.size()); ar.add(&h->ring_img, img_tot);
  ar.add(&h->ring_tp, tp_tot); ar.add(&h->ring_src, tp_tot); ar.add(&h->ring_to, to_tot);
  ar.add(&h->o_h, o_h.size()); ar.add(&h->o_p, o_p.size());
  ar.add(&h->t[0], n_t); ar.add(&h->t[1], n_t); ar.add(&h->dmat, n_t);
  ar.add(&h->old_phhp, h->n_m); ar.add(&h->r_phhp, h->n_m);
  ar.add(&h->x, x_tot); ar.add(&h->v_x, x_tot); ar.add(&h->tx, q_tot); ar.add(&h->tx_zero, h->tc_tx ? q_tot : 0);
  ar.add(&h->s, quad_cols.size()); ar.add(&h->r, h->n_quad_rows); ar.add(&h->xh, np); ar.add(&h->yp, h->npart);
  ar.add(&h->quad_items, quad_items.size());
  ar.add(&h->quad_rows, h->n_quad_rows); ar.add(&h->quad_cols, quad_cols.size());
  ar.add(&h->kcol, kcol.size());  // V tiling at create
  ar.add(&h->epart, std::max(h->n_ranges, h->n_asm_blocks)); ar.add(&h->ctl, 1); ar.add(&h->e_out, 1);
  ar.add(&h->ticket, 1); ar.add(&h->irr, 2);
  if (h->nt) {
    auto round_up = [](int64_t n) { return std::max<int64_t>(256, (n + 255) / 256 * 256); };
    h->n_vtc = round_up(vtc); h->n_tkttc = round_up(tkttc);
    if (h->tc_gen) {
      h->n_vtc = 0;  // V planes generated in the ladder
      ar.add(&h->vg_rows, vg_rows.size()); ar.add(&h->vg_cols, vg_cols.size());
      ar.add(&h->vg_tab, vg_tab.size());
    } else if (on_the_fly) {
      ar.add_unset(&h->v_tc, (size_t)h->nt * h->n_vtc);
    } else {
      ar.add(&h->v_tc, (size_t)h->nt * h->n_vtc);
    }
    ar.add(&h->tkt_tc, (size_t)h->nt * h->n_tkttc);
  }
  if (h->have_3body) {
    ar.add(&h->v_h_hpp, h->n_h); ar.add(&h->v_phh_p, h->n_p);
    ar.add(&h->old_h1pp_h2, h->n_h); ar.add(&h->old_h2pp_h1, h->n_h); ar.add(&h->diff_h2pp_h1, h->n_h);
    ar.add(&h->old_p1_p2hh, h->n_p); ar.add(&h->old_p2_p1hh, h->n_p); ar.add(&h->diff_p2_p1hh, h->n_p);
    ar.add(&h->gath, (size_t)8 * n_t);
  }
  int rc;
#define TRY(x) do { rc = (x); if (rc) return rc; } while (0)
  TRY(ar.commit(h));
  h->err = &h->ctl->err;
  // Scratch for the raw inputs, released at the end of create.
  Arena sc;
  double *vraw = nullptr, *hhpp_raw = nullptr, *hpph_raw = nullptr;
  RawIndex *raw_idx = nullptr;
  int32_t *counts = nullptr;
  int2 *d_mod_dims = nullptr;
  int4 *d_vrows = nullptr;
  int32_t *d_prow_raw = nullptr, *d_asym = nullptr;
  int4 *d_gv_items = nullptr, *d_gvt_items = nullptr;
  // Generated V_pppp: one item per operand-image chunk (channel, row tile, K chunk).
  // Counted per channel, then filled in parallel, each channel at its offset.
  std::vector<int4> &gv_items = bs.gv_items, &gvt_items = bs.gvt_items;
  gv_items.clear();
  gvt_items.clear();
  if (on_the_fly) {
    // With bf16 images both images come from the tensor-core chunks (gen_v_both_chunks_kernel).
    const bool tc_images = h->nt && !h->tc_gen;
    std::vector<int64_t> go(h->n_act + 1, 0), gto(h->n_act + 1, 0);
    for (int ai = 0; ai < h->n_act; ai++) {
      const ChanInfo &a = chans[ai];
      int64_t chunks = 0;
      for (int mt = 0; mt < a.nmt; mt++) chunks += a.nkc - ladder_kc0(a.sym, mt);
      go[ai + 1] = go[ai] + (tc_images ? 0 : chunks);
      gto[ai + 1] = gto[ai] + (tc_images ? (int64_t)a.nmt * a.nkct : 0);
    }
    gv_items.resize(go[h->n_act]);
    gvt_items.resize(gto[h->n_act]);
#pragma omp parallel for num_threads(host_threads) schedule(dynamic, 4)
    for (int ai = 0; ai < h->n_act; ai++) {
      const ChanInfo &a = chans[ai];
      int4 *g = gv_items.data() + go[ai];
      if (!tc_images)
        for (int mt = 0; mt < a.nmt; mt++)
          for (int kc = ladder_kc0(a.sym, mt); kc < a.nkc; kc++) *g++ = make_int4(ai, mt, kc, 0);
      int4 *gt = gvt_items.data() + gto[ai];
      if (tc_images)
        for (int mt = 0; mt < a.nmt; mt++)
          for (int kc = 0; kc < a.nkct; kc++) *gt++ = make_int4(ai, mt, kc, 0);
    }
  }
  int64_t *d_vraw_off = nullptr, *d_o_m = nullptr;
  // Derived tables: per-pair block offsets; and (fused path: for the ring's pairs too) the
  // modified-channel lookup of (particle, hole) pairs, built on the device from the pair lists.
  int32_t *d_hblk = nullptr, *d_pblk = nullptr;
  int4 *d_mlook = nullptr;
  const uint64_t n_mlook = derive_tables || h->ring_paired ? (nsp - np) * np : 0;
  sc.add(&d_mlook, n_mlook);
  if (!derive_tables) sc.add(&raw_idx, (size_t)8 * n_t);
  if (derive_tables || gen_v3) {  // block offsets inside hpp(k) and phh(a)
    sc.add(&d_hblk, np * np);
    sc.add(&d_pblk, (nsp - np) * (nsp - np));
  }
  RingPair *d_pairs = nullptr;
  sc.add(&d_pairs, pairs.size());
  ModGen *d_mod_gen = nullptr;
  int2 *d_mod_ph = nullptr, *d_mod_hp = nullptr;
  int32_t *d_mod_chan = nullptr;
  // With tables from the host, the lists that the ring's pairs rest on are checked against them.
  const bool check_lists = h->ring_paired && !derive_tables;
  const bool lists_on_device = gen_v || n_mlook;
  std::vector<int2> mod_at(check_lists ? nch : 0, make_int2(0, 0));
  for (size_t g = 0; g < mod_gen.size() && check_lists; g++)
    mod_at[mod_gen_chan[g]] = make_int2((int)mod_gen[g].ph_off, (int)mod_gen[g].hp_off);
  int2 *d_mod_at = nullptr;
  sc.add(&d_mod_at, mod_at.size());
  if (lists_on_device) {
    sc.add(&d_mod_ph, mod_ph.size()); sc.add(&d_mod_hp, mod_hp.size());
    sc.add(&d_mod_gen, mod_gen.size()); sc.add(&d_mod_chan, mod_gen_chan.size());
  }
  sc.add(&vraw, vraw_tot); sc.add(&hhpp_raw, gen_v ? 0 : n_t);
  sc.add(&hpph_raw, gen_v ? 0 : h->n_m);
  sc.add(&counts, (size_t)5 * n_t); sc.add(&d_vrows, vrows.size());
  // Row of V_pppp's uploaded rows (a <= b) of each packed row, and a mark per channel.
  std::vector<int32_t> prow_raw(on_the_fly ? 0 : kcol.size());
  for (const int4 &v : vrows) prow_raw[chans[v.x].pk_off + v.y] = v.z;
  sc.add(&d_prow_raw, prow_raw.size()); sc.add(&d_asym, n_act);
  sc.add(&d_gv_items, gv_items.size()); sc.add(&d_gvt_items, gvt_items.size());
  sc.add(&d_vraw_off, vraw_off.size()); sc.add(&d_mod_dims, mod_dims.size()); sc.add(&d_o_m, o_m.size());
  // The model on the device (on-the-fly V, E_ref and normal ordering): quantum numbers and
  // (electron gas) the direct Coulomb term by momentum transfer, computed here with the
  // reference's expression (ElectronGasSPBasis.cpp:424-448).  Kept for the handle's lifetime.
  ModelDev md{};
  std::vector<UploadPiece> batch;  // host -> device copies made together, after the lists
  std::unique_lock<std::mutex> staging_hold;  // staging buffers with copies still in flight
  std::vector<double> vq;
  std::vector<uint32_t> ocode;
  int32_t *d_qn = nullptr;
  double *d_vq = nullptr;
  uint32_t *d_ocode = nullptr;
  if (model_ok) {
    md.kind = M->kind;
    md.stride = M->qn_stride;
    md.g = M->params[0];
    md.Lb = M->params[0];
    if (M->kind == CCDGPU_MODEL_ELECTRON_GAS) {
      int nmax = 0;
      for (uint64_t o = 0; o < nsp; o++)
        for (int i = 0; i < 3; i++) nmax = std::max(nmax, std::abs(M->qn[o * M->qn_stride + i]));
      md.R = 2 * nmax;
      md.W = md.R + 1;  // components of the transfer by magnitude (see ModelDev)
      const double L = M->params[0], e_sq = M->params[1];
      vq.assign((size_t)md.W * md.W * md.W, 0.0);
      for (int dx = 0; dx <= md.R; dx++)
        for (int dy = 0; dy <= md.R; dy++)
          for (int dz = 0; dz <= md.R; dz++) {
            const int d[3] = {dx, dy, dz};
            const double prefactor = e_sq / (L * L * L);
            double rel = 0.0, mu = 0.0;
            for (int i = 0; i < 3; i++) {
              const double term = 2 * M_PI * d[i] / L;
              rel += term * term;
            }
            const double v = rel < 1.e-5 ? 0.0 : prefactor * 4 * M_PI / (rel + mu * mu);
            vq[((size_t)dx * md.W + dy) * md.W + dz] = v;
          }
      if (nmax <= 63) {
        ocode.resize(nsp);
        for (uint64_t o = 0; o < nsp; o++) {
          const int32_t *q = M->qn + o * M->qn_stride;
          ocode[o] = (uint32_t)(q[0] + 64) | ((uint32_t)(q[1] + 64) << 8) |
                     ((uint32_t)(q[2] + 64) << 16) | ((uint32_t)(q[3] & 0xff) << 24);
        }
      }
    }
    Arena mr;
    mr.add(&d_qn, (size_t)nsp * M->qn_stride);
    mr.add(&d_vq, vq.size());
    mr.add(&d_ocode, ocode.size());
    mr.add(&h->eps_io, 2 * nsp + 1);
    TRY(mr.commit(h));
    batch.push_back(UploadPiece{reinterpret_cast<char *>(d_qn),
                                reinterpret_cast<const char *>(M->qn),
                                (size_t)nsp * M->qn_stride * sizeof(int32_t)});
    batch.push_back(UploadPiece{reinterpret_cast<char *>(d_vq),
                                reinterpret_cast<const char *>(vq.data()), vq.size() * 8});
    batch.push_back(UploadPiece{reinterpret_cast<char *>(d_ocode),
                                reinterpret_cast<const char *>(ocode.data()), ocode.size() * 4});
    md.qn = d_qn;
    md.vq = d_vq;
    md.ocode = ocode.empty() ? nullptr : d_ocode;
    h->md = md;
    h->has_model = true;
  }
  const size_t n_allocs = h->allocs.size();
  TRY(sc.commit(h));

  // The host lists go up together with the model's (copy_pieces_to_device below); they stay
  // alive until then.
  auto put = [&](auto *dst, const auto &v) -> int {
    if (!v.empty())
      batch.push_back(UploadPiece{reinterpret_cast<char *>(dst),
                                  reinterpret_cast<const char *>(v.data()),
                                  v.size() * sizeof(v[0])});
    return CCDGPU_OK;
  };
  TRY(put(h->chans, chans)); TRY(put(h->mods, mods));
  TRY(put(d_pairs, pairs)); TRY(put(h->ring_units, units));
  TRY(put(h->ranges, ranges)); TRY(put(h->quad_items, quad_items));
  TRY(put(h->quad_cols, quad_cols));

  TRY(put(h->kcol, kcol));
  if (h->tc_gen) {
    TRY(put(h->vg_rows, vg_rows)); TRY(put(h->vg_cols, vg_cols)); TRY(put(h->vg_tab, vg_tab));
  }
  TRY(put(h->pp_pairs, pp_pairs)); TRY(put(h->hh_pairs, hh_pairs));
  TRY(put(h->pp_swap, pp_swap)); TRY(put(h->hh_swap, hh_swap));
  TRY(put(h->list_off, list_off)); TRY(put(h->list, list));
  TRY(put(h->prow, prow)); TRY(put(h->hcol, hcol));
  TRY(put(h->o_h, o_h)); TRY(put(h->o_p, o_p));
  TRY(put(d_vrows, vrows)); TRY(put(d_vraw_off, vraw_off)); TRY(put(d_prow_raw, prow_raw));
  TRY(put(d_gv_items, gv_items)); TRY(put(d_gvt_items, gvt_items));
  TRY(put(d_mod_dims, mod_dims)); TRY(put(d_o_m, o_m));
  batch.push_back(UploadPiece{reinterpret_cast<char *>(h->eps),
                              reinterpret_cast<const char *>(P->sp_energy), nsp * 8});

  // V blocks and tables, uploaded in their reference layouts (runs of adjacent blocks).
  {
    std::vector<const double *> sp, sx, sh;
    std::vector<int64_t> np2, nx, nh;
    std::vector<const ccdgpu_chain_index *> sm[8];
    std::vector<int64_t> nm;
    for (size_t ai = 0; ai < chans.size(); ai++) {
      const uint64_t c = act_chan[ai];
      const ChanInfo &a = chans[ai];
      if ((!on_the_fly && !P->v_pppp[c]) || (!gen_v && (!P->v_hhpp[c] || !P->v_hhhh[c])))
        return CCDGPU_ERR_INVALID_ARGUMENT;
      if (!on_the_fly)  // the rows a <= b of V_pppp (the ladder reads those with a < b)
        for (int u = 0; u < a_pr[ai]; u++) {
          sp.push_back(P->v_pppp[c] + (int64_t)rowmap[a_row_off[ai] + u] * a.pp);
          np2.push_back(a.pp);
        }
      if (!gen_v) {
        sx.push_back(P->v_hhpp[c]); nx.push_back((int64_t)a.pp * a.hh);
        sh.push_back(P->v_hhhh[c]); nh.push_back((int64_t)a.hh * a.hh);
      }
      for (int k = 0; k < 8 && !derive_tables; k++) {
        if (!P->maps[k][c]) return CCDGPU_ERR_INVALID_ARGUMENT;
        sm[k].push_back(P->maps[k][c]);
      }
      nm.push_back((int64_t)a.pp * a.hh);
    }
    TRY(upload_runs(h, vraw, sp, np2));
    TRY(upload_runs(h, hhpp_raw, sx, nx));
    TRY(upload_runs(h, h->v_hhhh, sh, nh));
    static_assert(sizeof(RawIndex) == sizeof(ccdgpu_chain_index), "ChainIndex layout");
    for (int k = 0; k < 8 && !derive_tables; k++)
      TRY(upload_runs(h, reinterpret_cast<ccdgpu_chain_index *>(raw_idx) + (size_t)k * n_t, sm[k], nm));
    TRY(put(d_mod_at, mod_at));
    if (lists_on_device) {
      TRY(put(d_mod_ph, mod_ph));
      TRY(put(d_mod_hp, mod_hp));
      TRY(put(d_mod_gen, mod_gen));
      TRY(put(d_mod_chan, mod_gen_chan));
    }
    TRY(upload_runs(h, hpph_raw, src_hpph, cnt_hpph));
    TRY(upload_runs(h, h->v_hphp, src_hphp, cnt_hphp));
    if (h->have_3body && !gen_v3) {
      std::vector<const double *> s5, s6;
      std::vector<int64_t> n5, n6;
      for (uint64_t k = 0; k < np; k++) {
        const int64_t n = o_h[k + 1] - o_h[k];
        if (n && !P->v_h_hpp[k]) return CCDGPU_ERR_INVALID_ARGUMENT;
        s5.push_back(P->v_h_hpp[k]); n5.push_back(n);
      }
      for (uint64_t a = 0; a < h->npart; a++) {
        const int64_t n = o_p[a + 1] - o_p[a];
        if (n && !P->v_phh_p[a]) return CCDGPU_ERR_INVALID_ARGUMENT;
        s6.push_back(P->v_phh_p[a]); n6.push_back(n);
      }
      TRY(upload_runs(h, h->v_h_hpp, s5, n5));
      TRY(upload_runs(h, h->v_phh_p, s6, n6));
    }
    // The last use of the staging buffers in create: the lists' copies stay in flight (the
    // staging lock is held until the set-up's final synchronisation).
    TRY(copy_pieces_to_device(h, batch, &staging_hold));
  }
  // Device layout transforms.
  h->create_ms[1] = ms_since(t_build) - h->create_ms[0];
  if (h->n_quad_rows) {
    quad_rows_kernel<<<(unsigned)h->n_act, 256, 0, h->s0>>>(
        h->chans, h->kcol, h->pp_swap, h->pp_pairs, h->eps, (int)np, h->quad_rows);
    CK(cudaGetLastError());
  }
  if (gen_v && !mod_gen.empty()) {
    gen_v_mod_kernel<<<(unsigned)mod_gen.size(), 256, 0, h->s0>>>(d_mod_gen, d_mod_ph, d_mod_hp,
                                                                 md, h->v_hpph, h->v_hphp);
    CK(cudaGetLastError());
  } else if (h->n_mod) {
    transpose_hpph_kernel<<<h->n_mod, 256, 0, h->s0>>>(h->mods, hpph_raw, h->v_hpph);
    CK(cudaGetLastError());
  }
  if (h->n_ranges) {
    if (gen_v) {
      gen_v_pphh_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->pp_pairs,
                                                        h->hh_pairs, md, h->v_pphh);
      CK(cudaGetLastError());
      gen_v_hhhh_kernel<<<(unsigned)chans.size(), 256, 0, h->s0>>>(h->chans, h->hh_pairs, md,
                                                                   h->v_hhhh);
    } else {
      transpose_hhpp_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, hhpp_raw,
                                                            h->v_pphh);
    }
    CK(cudaGetLastError());
    if (h->n_quad_items) {
      pack_quads_kernel<<<h->n_quad_items, kAsmThreads, 0, h->s0>>>(
          h->quad_items, h->chans, h->quad_rows, h->quad_cols, h->v_pphh, h->vq);
      CK(cudaGetLastError());
      hh_records_kernel<<<(unsigned)h->n_act, 256, 0, h->s0>>>(
          h->chans, h->quad_cols, h->v_hhhh, h->v_x, h->hh_tiles, h->hh_out, h->tx_tiles);
      CK(cudaGetLastError());
    }
    if (derive_tables || gen_v3) {
      pair_sizes_kernel<<<(unsigned)chans.size(), 256, 0, h->s0>>>(
          h->chans, h->pp_pairs, h->hh_pairs, (int)np, (int)h->npart, d_hblk, d_pblk);
      CK(cudaGetLastError());
      row_scan_kernel<<<(unsigned)np, 256, 0, h->s0>>>(d_hblk, (int)np);
      CK(cudaGetLastError());
      row_scan_kernel<<<(unsigned)h->npart, 256, 0, h->s0>>>(d_pblk, (int)h->npart);
      CK(cudaGetLastError());
    }
    if (gen_v3) {
      gen_v3_kernel<<<(unsigned)chans.size(), 256, 0, h->s0>>>(
          h->chans, h->pp_pairs, h->hh_pairs, md, h->o_h, h->o_p, d_hblk, d_pblk, (int)np,
          (int)h->npart, h->v_h_hpp, h->v_phh_p, h->err);
      CK(cudaGetLastError());
    }
    // Lists that contradict each other: bad where the tables come from them, else not to be paired.
    const int32_t list_err = derive_tables ? kErrBadIndex : kErrRingLists;
    if (n_mlook) {
      CK(cudaMemsetAsync(d_mlook, 0xff, n_mlook * sizeof(int4), h->s0));  // every field -1
      if (!mod_gen.empty()) {
        mod_lookup_kernel<<<(unsigned)mod_gen.size(), 128, 0, h->s0>>>(
            d_mod_gen, d_mod_chan, d_mod_ph, d_mod_hp, (int)np, d_mlook, list_err, h->err);
        CK(cudaGetLastError());
      }
    }
    if (derive_tables) {
      DeriveGeometry dg{h->o_h, h->o_p, d_o_m, d_mod_dims, d_hblk, d_pblk, d_mlook,
                        (int32_t)np, (int32_t)h->npart};
      derive_tables_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->pp_pairs,
                                                           h->hh_pairs, dg, n_t, h->flat, counts,
                                                           h->err);
    } else {
      TableGeometry geo{h->o_h, h->o_p, d_o_m, d_mod_dims, nch, np, h->npart};
      convert_tables_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, raw_idx, n_t, geo,
                                                            h->flat, counts, h->err);
      CK(cudaGetLastError());
      if (check_lists)
        check_lists_kernel<<<h->n_ranges, 256, 0, h->s0>>>(
            h->ranges, h->chans, h->pp_pairs, h->hh_pairs, raw_idx + CCDGPU_MAP_AI_JB * n_t, nch,
            d_mod_dims, d_mod_at, d_mod_ph, d_mod_hp, h->err);
    }
    CK(cudaGetLastError());
    const int nb = (int)std::min<int64_t>(ceil_div(5 * n_t, 256), kSMs * 32);
    check_counts_kernel<<<std::max(nb, 1), 256, 0, h->s0>>>(counts, 5 * n_t, h->err);
    CK(cudaGetLastError());
    ring_maps_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->pp_swap, h->hh_swap,
                                                     h->prow, h->hcol, h->flat, n_t,
                                                     h->ring_quads,
                                                     derive_tables ? nullptr : h->irr + 1, h->err);
    CK(cudaGetLastError());
    if (!gen_v) {
      TRY(launch_antisymmetry(h, h->v_pphh));
      antisymmetry_hhhh_kernel<<<(unsigned)h->n_act, 256, 0, h->s0>>>(h->chans, h->hh_swap,
                                                                      h->v_hhhh, h->irr + 1);
      CK(cudaGetLastError());
    }
    if (!pairs.empty()) {
      ring_image_kernel<<<(unsigned)pairs.size(), 256, 0, h->s0>>>(
          d_pairs, d_mod_ph, d_mod_hp, d_mlook, (int)np, h->v_hpph, h->v_hphp, h->ring_quads,
          h->ring_img, h->ring_src, h->ring_to, list_err, h->err);
      CK(cudaGetLastError());
    }
  }
  if (a_vrow_off[n_act] > 0) {
    if (on_the_fly) {
      // FP64 tiles, and the bf16 images unless the tensor-core ladder generates its own V: one
      // CTA per image chunk; with bf16 images, one CTA per tensor-core chunk writes both.
      if (!gv_items.empty()) {
        auto kern64 = md.ocode ? gen_v_chunks_kernel<true> : gen_v_chunks_kernel<false>;
        kern64<<<(unsigned)gv_items.size(), 256, 0, h->s0>>>(
            h->chans, d_gv_items, h->kcol, h->pp_pairs, md, h->v_t);
        CK(cudaGetLastError());
      }
      if (h->nt && !h->tc_gen && !gvt_items.empty()) {
        auto kern = md.ocode ? (h->nt == 3 ? gen_v_both_chunks_kernel<3, true>
                                           : gen_v_both_chunks_kernel<2, true>)
                             : (h->nt == 3 ? gen_v_both_chunks_kernel<3, false>
                                           : gen_v_both_chunks_kernel<2, false>);
        kern<<<(unsigned)gvt_items.size(), 256, 0, h->s0>>>(h->chans, d_gvt_items, h->kcol,
                                                           h->pp_pairs, md, h->v_t, h->v_tc,
                                                           h->n_vtc);
      }
    } else {
      // Laid out as symmetric; where it is not, again below, once the error word is read.
      v_symmetry_kernel<<<(unsigned)vrows.size(), 128, 0, h->s0>>>(
          h->chans, d_vrows, h->kcol, d_prow_raw, d_vraw_off, vraw, d_asym, h->err);
      CK(cudaGetLastError());
      tile_v_kernel<<<(unsigned)vrows.size(), 128, 0, h->s0>>>(h->chans, d_vrows, h->kcol,
                                                               d_vraw_off, vraw, h->v_t);
    }
    CK(cudaGetLastError());
    if (h->nt && !on_the_fly) {
      tile_v_tc_kernel<<<(unsigned)vrows.size(), 128, 0, h->s0>>>(
          h->chans, d_vrows, h->kcol, d_vraw_off, vraw, h->v_tc, h->n_vtc, h->nt);
      CK(cudaGetLastError());
    }
  }
  // Host work that needs no result of the set-up kernels runs while they do: kernel
  // attributes, the ladder schedules and, for device-loop handles, the loop graph's capture
  // (nothing of it executes until a solve launches it).  Then the set-up's error word is read.
  const auto t_sched = std::chrono::steady_clock::now();
#undef TRY
  h->h_ctl = ctl_acquire();
  if (!h->h_ctl) return CCDGPU_ERR_OUT_OF_MEMORY;

  // The attribute belongs to the kernel, not to this handle: set the device's opt-in maximum
  // (the same value for every handle), so that handles of different channel sizes coexist.
  int smem_optin = 0;
  CK(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->opt.device));
  if (ring16_smem(80) > (size_t)smem_optin) return CCDGPU_ERR_UNSUPPORTED;
  CK(cudaFuncSetAttribute(ring_pair_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          ring_unit_smem(4, false, kRingMax, kRingMax, kPairNC) * (int)sizeof(double)));
  CK(cudaFuncSetAttribute(ring_pair_kernel<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          ring_unit_smem(4, true, kRingMax, kRingMax, kPairNC) * (int)sizeof(double)));
  CK(cudaFuncSetAttribute(pp_ladder_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)kLadderSmem));
  CK(cudaFuncSetAttribute(pp_ladder_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  CK(cudaFuncSetAttribute(ring16_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)ring16_smem(32)));
  CK(cudaFuncSetAttribute(ring16_kernel<48>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)ring16_smem(48)));
  CK(cudaFuncSetAttribute(ring16_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)ring16_smem(64)));
  CK(cudaFuncSetAttribute(ring16_kernel<80>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)ring16_smem(80)));
  ccdgpu_schedule sch{};
  sch.thin_split_mul = 1;
  sch.wide_split_mul = 3;
  sch.tc_split_mul = 2;
  if (int rc2 = make_ladder_tiles(h, sch)) return rc2;
  if (h->nt) {
    h->tc_smem = tc_smem_bytes(h->nt);
    CK(cudaFuncSetAttribute(tc_kernel_of(h->nt, h->tc_gen),
                            cudaFuncAttributeMaxDynamicSharedMemorySize, (int)h->tc_smem));
  }
  if (h->opt.path == CCDGPU_PATH_FUSED && h->opt.use_graph && h->opt.device_loop) {
    ready_loop_graphs(h);
    if (h->loop_state != 1) h->loop_state = 0;  // retried by the first solve, on an idle stream
  }
  h->create_ms[3] = ms_since(t_sched);
  int32_t e = 0;
  unsigned long long irr = 0;
  CK(cudaMemcpyAsync(&e, h->err, sizeof(e), cudaMemcpyDeviceToHost, h->s0));
  CK(cudaMemcpyAsync(&irr, h->irr + 1, sizeof(irr), cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  h->create_ms[2] = ms_since(t_build) - h->create_ms[0] - h->create_ms[1];
  h->irregular = irr != 0 || (e & kErrRingMaps);
  if (e & kErrAsym) {  // those channels are stored and streamed in full
    e &= ~kErrAsym;
    std::vector<int32_t> asym(n_act);
    CK(cudaMemcpyAsync(asym.data(), d_asym, n_act * sizeof(int32_t), cudaMemcpyDeviceToHost, h->s0));
    CK(cudaStreamSynchronize(h->s0));
    for (int ai = 0; ai < n_act; ai++)
      if (asym[ai]) {
        ChanInfo &a = h->host_chans[ai];
        a.sym = 0;
        h->ladder_bytes += 4.0 * a.pk * (a.pk - 1.0);
      }
    CK(cudaMemcpyAsync(h->chans, h->host_chans.data(), n_act * sizeof(ChanInfo),
                       cudaMemcpyHostToDevice, h->s0));
    CK(cudaMemsetAsync(h->v_t, 0, vt * sizeof(double), h->s0));
    tile_v_kernel<<<(unsigned)vrows.size(), 128, 0, h->s0>>>(h->chans, d_vrows, h->kcol,
                                                             d_vraw_off, vraw, h->v_t);
    CK(cudaGetLastError());
    CK(cudaMemsetAsync(h->err, 0, sizeof(int32_t), h->s0));
    if (int rc2 = make_ladder_tiles(h, sch)) return rc2;
    CK(cudaStreamSynchronize(h->s0));
  }
  if (e & kErrRingLists) {  // the tables' blocks are not those that the lists name
    e &= ~kErrRingLists;
    h->ring_paired = false;
    for (int k = 0; k < 3; k++) h->ring_flops[k] = h->ring_bytes[k] = 0.0;
    h->n_tp = h->n_ring[0] = h->n_ring[1] = h->n_ring[2] = 0;
    if (h->loop64) cudaGraphExecDestroy(h->loop64);
    if (h->loop_tc) cudaGraphExecDestroy(h->loop_tc);
    h->loop64 = h->loop_tc = nullptr;
    h->loop_state = 0;
    CK(cudaMemsetAsync(h->err, 0, sizeof(int32_t), h->s0));
  }
  // Release the scratch allocation.
  for (size_t i = n_allocs; i < h->allocs.size(); i++) dev_free(h->allocs[i].p, h->allocs[i].bytes);
  h->allocs.resize(n_allocs);
  if (e & kErrBadIndex) return CCDGPU_ERR_BAD_TABLE;
  // The fused path relies on the structure of the ring tables; the table path does not.
  if ((e & kErrRingMaps) && h->opt.path == CCDGPU_PATH_FUSED) return CCDGPU_ERR_BAD_TABLE;
  if (e & ~kErrRingMaps) return CCDGPU_ERR_CUDA;
  if (e) CK(cudaMemsetAsync(h->err, 0, sizeof(int32_t), h->s0));
  return CCDGPU_OK;
}

// ---- launches -------------------------------------------------------------------------

// Launch with the programmatic-stream-serialization attribute (PDL): the kernel may begin
// launching while its stream predecessor drains; it waits in griddepcontrol.wait before
// touching the predecessor's results (skip_iteration / pdl_enter in every kernel).
thread_local bool t_pdl = true;  // cleared while retrying a loop-graph capture without PDL

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem,
                       cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = t_pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// gate: 0 = kernel of an FP64 iteration, 1 = of a mixed-precision iteration.
// only: -1 everything, 0 units of hk <= 8, 1 the other units, 2 the reduction.
int launch_hh_ladder(ccdgpu_handle *h, cudaStream_t st, int gate, int only = -1) {
  const int n_cta = (only < 0 || only == 1) ? h->n_hh_cta : 0;
  const int n_warp = only <= 0 ? h->n_hh_warp : 0;
  if (n_cta + n_warp) {
    h->launches++;
    CK(launch_pdl(hh_slice_kernel, n_cta + (int)ceil_div(n_warp, kHHThreads / 32), kHHThreads,
                  n_cta ? kHHSmem : 0, st,
                  (const HHTile *)(h->hh_tiles + (n_cta ? 0 : h->n_hh_cta)), n_cta, n_warp,
                  (const double *)h->vq, (const double *)h->tq[0], (const double *)h->tq[1], h->part, h->r,
                  (const Control *)h->ctl, gate));
  }
  if (h->n_hh_out && (only < 0 || only == 2)) {
    h->launches++;
    const int nt = h->tc_tx && gate ? h->nt : 0;
    CK(launch_pdl(nt == 3 ? hh_reduce_kernel<3> : nt ? hh_reduce_kernel<2> : hh_reduce_kernel<0>,
                  (int)ceil_div((int64_t)h->n_hh_out * kHHLanes, 128), 128, 0, st,
                  (const HHOut *)h->hh_out, h->n_hh_out, (const double *)h->v_x,
                  (const double *)h->part, h->x, h->s, h->tkt_tc, h->n_tkttc,
                  (const Control *)h->ctl, gate));
  }
  return CCDGPU_OK;
}
int launch_pp_ladder_tc(ccdgpu_handle *h, cudaStream_t st) {
  if (!h->n_tc_tiles) return CCDGPU_OK;
  h->launches++;
  return cuda_status(launch_pdl(
      tc_kernel_of(h->nt, h->tc_gen), std::min(h->n_tc_tiles, kTcGrid), tc_threads(h->tc_gen),
      h->tc_smem, st, (const LadderTile *)h->tc_tiles, h->n_tc_tiles, h->sched + 2,
      (const __nv_bfloat16 *)h->v_tc, h->n_vtc, (const __nv_bfloat16 *)h->tkt_tc, h->n_tkttc,
      h->tc_planes, (const Control *)h->ctl, h->err, (const ChanInfo *)h->chans,
      (const VGenRow *)h->vg_rows, (const uint32_t *)h->vg_cols, (const double *)h->vg_tab));
}
// FP64 ladder; cls >= 0: the tiles of one column class alone (wide, mid, thin in list order).
int launch_pp_ladder(ccdgpu_handle *h, cudaStream_t st, int cls = -1) {
  const int first = cls < 0 || cls == 2 ? 0 : h->n_cls[2] + (cls == 0 ? h->n_cls[1] : 0);
  const int n = cls < 0 ? h->n_tiles : h->n_cls[cls];
  if (!n) return CCDGPU_OK;
  h->launches++;
  return cuda_status(launch_pdl(
      pp_ladder_kernel, std::min(n, kSMs), kLadderThreads, kLadderSmem, st,
      (const LadderTile *)(h->tiles + first), n, h->sched, (const double *)h->v_t,
      (const double *)h->tq[0], (const double *)h->tq[1], h->d_planes, (const Control *)h->ctl,
      h->err, 0));
}
// t2Diff_pphh from the ladder's planes (tc: the tensor-core ladder's) and T X.
int launch_expand_d(ccdgpu_handle *h, bool tc) {
  if (h->dmat_full) CK(cudaMemsetAsync(h->dmat, 0, h->n_t * sizeof(double), h->s0));
  h->dmat_full = false;
  if (!h->n_quad_items) return CCDGPU_OK;
  expand_d_kernel<<<h->n_quad_items, kAsmThreads, 0, h->s0>>>(
      h->quad_items, h->chans, tc ? h->tc_lrows : h->lrows, h->quad_rows, h->quad_cols,
      tc ? h->tc_planes : h->d_planes, tc && h->tc_tx ? h->tx_zero : h->tx, h->dmat);
  h->launches++;
  return cuda_status(cudaGetLastError());
}
// t2Diff_pphh of the last fused iteration into dmat, if that has not been done.
int materialize_d(ccdgpu_handle *h) {
  if (!h->d_from) return CCDGPU_OK;
  const bool tc = h->d_from == 2;
  h->d_from = 0;
  return launch_expand_d(h, tc);
}
// t[0] of the fused path: the current amplitudes in the reference order.
int materialize_t(ccdgpu_handle *h) {
  if (h->slab_current || h->opt.path != CCDGPU_PATH_FUSED) return CCDGPU_OK;
  h->slab_current = true;
  if (!h->n_ranges) return CCDGPU_OK;
  expand_t_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->prow, h->hcol, h->tq[0],
                                                  h->tq[1], h->ctl, h->t[0]);
  h->launches++;
  return cuda_status(cudaGetLastError());
}
// Marks in h->irr whether src (t2_pphh layout) lacks the antisymmetry of the packed layout.
int launch_antisymmetry(ccdgpu_handle *h, const double *src) {
  if (!h->n_ranges) return CCDGPU_OK;
  CK(cudaMemsetAsync(h->irr, 0, sizeof(*h->irr), h->s0));
  max_abs_kernel<<<(unsigned)std::min<int64_t>(ceil_div(h->n_t, 1024), kSMs * 8), 256, 0, h->s0>>>(
      src, h->n_t, h->irr);
  CK(cudaGetLastError());
  antisymmetry_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->pp_swap, h->hh_swap,
                                                      src, h->irr, h->irr + 1);
  h->launches += 2;
  return cuda_status(cudaGetLastError());
}
// The state that the stage calls read, on a handle of the fused path, whose iterations keep the
// packed amplitudes alone: t2Old_pphh, t2Old_phhp and the three-body chains.
int launch_map_to(ccdgpu_handle *h, cudaStream_t st, const double *src, double *dst, int mark = 0);
int ready_slabs(ccdgpu_handle *h) {
  if (h->opt.path != CCDGPU_PATH_FUSED) return CCDGPU_OK;
  if (int rc = materialize_t(h)) return rc;
  if (h->chains_current) return CCDGPU_OK;
  h->chains_current = true;
  return launch_map_to(h, h->s0, h->t[0], h->t[0]);
}
// A fused iteration leaves the packed amplitudes ahead of everything in the reference's layouts.
void slabs_behind(ccdgpu_handle *h) {
  h->slab_current = h->chains_current = h->t2_staged = h->irregular_t = false;
}
// The amplitudes in t[1] have been scattered: everything but the bf16 image is current.
void slabs_loaded(ccdgpu_handle *h) {
  h->slab_current = h->chains_current = h->t2_staged = h->tc_stale = true;
}
// The bf16 image of the current amplitudes, before a mixed iteration that does not follow a
// mixed iteration.
int refresh_tc_image(ccdgpu_handle *h) {
  if (!h->nt || !h->tc_stale) return CCDGPU_OK;
  h->tc_stale = false;
  if (!h->n_quad_items) return CCDGPU_OK;
  t_image_kernel<<<h->n_quad_items, kAsmThreads, 0, h->s0>>>(
      h->quad_items, h->chans, h->quad_cols, h->tq[0], h->tq[1], h->ctl, h->tkt_tc, h->n_tkttc, h->nt);
  h->launches++;
  return cuda_status(cudaGetLastError());
}

// t2Old_phhp of a fused handle from its current amplitudes.
int launch_phhp_gather(ccdgpu_handle *h, cudaStream_t st) {
  if (!h->n_m) return CCDGPU_OK;
  h->launches++;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(h->n_m, 256), kSMs * 16);
  phhp_gather_kernel<<<blocks, 256, 0, st>>>(h->ring_quads, h->n_m, h->tq[0], h->tq[1],
                                             h->old_phhp, h->ctl);
  return cuda_status(cudaGetLastError());
}
// Table path: T' from the phhp slab, R to t2Diff_phhp.
int launch_ring(ccdgpu_handle *h, cudaStream_t st, int gate) {
  if (h->n_mod_small) {
    CK(launch_pdl(ring_small_kernel, (int)ceil_div(h->n_mod_small, kRingSmallWarps),
                  kRingSmallWarps * 32, 0, st, (const ModInfo *)h->mods, h->n_mod_small,
                  (const double *)h->v_hpph, (const double *)h->v_hphp,
                  (const double *)h->old_phhp, h->r_phhp, (const Control *)h->ctl, gate));
    h->launches++;
  }
  const ModInfo *mp = h->mods + h->n_mod_small;  // groups by padded size
  for (int k = 0; k < 4; k++) {
    const int n = h->n_mod_pad[k];
    if (n) {
      auto go = [&](auto kern, int pad) {
        return launch_pdl(kern, n, 32 * ring16_warps(pad), ring16_smem(pad), st, mp,
                          (const double *)h->v_hpph, (const double *)h->v_hphp,
                          (const double *)h->old_phhp, h->r_phhp, (const Control *)h->ctl, gate);
      };
      switch (k) {
        case 0: CK(go(ring16_kernel<32>, 32)); break;
        case 1: CK(go(ring16_kernel<48>, 48)); break;
        case 2: CK(go(ring16_kernel<64>, 64)); break;
        default: CK(go(ring16_kernel<80>, 80)); break;
      }
      h->launches++;
    }
    mp += n;
  }
  return CCDGPU_OK;
}
// Fused-path ring: the T' images, and the units of group k (0: 4 warps, 1: 2, 2: 1).  Without pairs
// the whole of it: the phhp slab, the table path's kernels, the quads' two sums.
int launch_tp_gather(ccdgpu_handle *h, cudaStream_t st, int gate) {
  if (!h->ring_paired) {
    if (!h->n_quad_items) return CCDGPU_OK;
    int rc;
    if ((rc = launch_phhp_gather(h, st)) || (rc = launch_ring(h, st, gate))) return rc;
    ring_sums_kernel<<<h->n_quad_items, kAsmThreads, 0, st>>>(
        h->quad_items, h->chans, h->quad_rows, h->quad_cols, h->flat + CCDGPU_MAP_AI_JB * h->n_t,
        h->r_phhp, h->r_quad);
    h->launches++;
    return cuda_status(cudaGetLastError());
  }
  if (!h->n_tp) return CCDGPU_OK;
  h->launches++;
  return cuda_status(launch_pdl(
      tp_gather_kernel, (unsigned)ceil_div(h->n_tp, (int64_t)kGatherThreads * kGatherPer),
      kGatherThreads, 0, st, (const int32_t *)h->ring_src, h->n_tp, (const double *)h->tq[0],
      (const double *)h->tq[1], h->ring_tp, (const Control *)h->ctl, gate));
}
int launch_ring_units(ccdgpu_handle *h, cudaStream_t st, int gate, int k) {
  const int n = h->n_ring[k];
  if (!n) return CCDGPU_OK;
  const RingUnit *units = h->ring_units;
  for (int j = 0; j < k; j++) units += h->n_ring[j];
  auto kern = k == 0 ? (h->ring_cols ? ring_pair_kernel<4, true> : ring_pair_kernel<4>) : k == 1 ? ring_pair_kernel<2> : ring_pair_kernel<1>;
  h->launches++;
  return cuda_status(launch_pdl(kern, k == 2 ? (int)ceil_div(n, 4) : n, k == 1 ? 64 : 128,
                                h->ring_smem[k], st, units, n, (const double *)h->ring_img,
                                (const int32_t *)h->ring_to, (const double *)h->ring_tp,
                                h->r_quad, (const Control *)h->ctl, h->err, gate));
}
// One-body sums and T X.  only: -1 both, 0 the sums, 1 T X.
int launch_hh_post(ccdgpu_handle *h, cudaStream_t st, int gate, int only = -1) {
  const int n_ob = only != 1 ? (int)ceil_div((int64_t)h->nsp, kPostThreads / 32) : 0;
  const int n_tx = only != 0 ? (int)ceil_div(h->n_tx, kPostThreads / 32) : 0;
  if (!(n_ob + n_tx)) return CCDGPU_OK;
  h->launches++;
  return cuda_status(launch_pdl(
      hh_post_kernel, n_ob + n_tx, kPostThreads, 0, st, n_ob, (int)h->np, (int)h->nsp, h->list_off,
      h->list, h->s, h->r, h->xh, h->yp, (const TXTile *)h->tx_tiles, h->n_tx, (const double *)h->x,
      (const double *)h->tq[0], (const double *)h->tq[1], h->tx, (const Control *)h->ctl, gate));
}
int launch_assemble_fused(ccdgpu_handle *h, cudaStream_t st, int gate) {
  h->ctl_current = false;
  if (!h->n_asm_blocks) return CCDGPU_OK;
  h->launches++;
  return cuda_status(launch_pdl(
      h->loop_capture ? assemble_fused_kernel<true> : assemble_fused_kernel<false>,
      h->n_asm_blocks, kAsmThreads, 0, st, (const QuadItem *)h->quad_items, h->n_quad_items,
      (const ChanInfo *)h->chans, (const LadderRows *)(gate ? h->tc_lrows : h->lrows),
      (const QuadRow *)h->quad_rows, (const QuadCol *)h->quad_cols, (const double *)h->vq,
      (const double *)(gate ? h->tc_planes : h->d_planes),
      (const double *)(gate && h->tc_tx ? h->tx_zero : h->tx),
      (const double *)h->r_quad, (const double *)h->xh, (const double *)h->yp, h->tq[0], h->tq[1],
      h->epart, h->ticket, h->ctl, h->tkt_tc, h->n_tkttc, gate ? h->nt : 0,
      (cudaGraphConditionalHandle)(h->loop_capture ? h->loop_cond : 0), h->loop_capture, gate));
}
int launch_energy(ccdgpu_handle *h, cudaStream_t st, int flags) {
  if (flags) h->ctl_current = false;
  energy_kernel<<<1, kEnergyThreads, 0, st>>>(h->epart, h->n_ranges, h->ctl, flags, h->e_out, 0);
  h->launches++;
  return cuda_status(cudaGetLastError());
}
// mark: the pass over non-finite elements (map_to_kernel) instead of the scatters.
int launch_map_to(ccdgpu_handle *h, cudaStream_t st, const double *src, double *dst, int mark) {
  if (!h->n_ranges) return CCDGPU_OK;
  map_to_kernel<<<h->n_ranges, 256, 0, st>>>(h->ranges, h->chans, h->prow, h->hcol, h->flat,
                                             h->n_t, src, dst, h->old_h2pp_h1, h->old_h1pp_h2,
                                             h->old_p1_p2hh, h->old_p2_p1hh, h->old_phhp,
                                             h->tq[0], h->tq[1], h->have_3body ? 1 : 0, h->ctl,
                                             mark);
  h->launches++;
  return cuda_status(cudaGetLastError());
}

// t2Diff_pphh of the table path and the stage calls into dmat, from t2Old_pphh (t[0]).
int launch_pphh(ccdgpu_handle *h) {
  int rc;
  if (!h->irregular && !h->irregular_t) {
    if ((rc = launch_hh_ladder(h, h->s0, 0)) || (rc = launch_hh_post(h, h->s0, 0, 1)) ||
        (rc = launch_pp_ladder(h, h->s0)))
      return rc;
    return launch_expand_d(h, false);
  }
  if (!h->n_ranges) return CCDGPU_OK;
  if (!h->x_full) {
    void *p = nullptr;
    size_t got = 0;
    CK(cudaSetDevice(h->opt.device));
    CK(dev_alloc(std::max<int64_t>(h->n_vhh, 1) * sizeof(double), &p, &got));
    h->allocs.push_back({p, got});
    h->x_full = static_cast<double *>(p);
  }
  h->dmat_full = true;
  general_x_kernel<<<dim3((unsigned)h->n_act, 8), 256, 0, h->s0>>>(h->chans, h->v_pphh, h->v_hhhh,
                                                                   h->t[0], h->x_full);
  CK(cudaGetLastError());
  general_d_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->prow, h->kcol, h->pp_swap,
                                                   h->pp_pairs, h->v_t, h->md, h->v_generated,
                                                   h->x_full, h->t[0], h->dmat);
  h->launches += 2;
  return cuda_status(cudaGetLastError());
}

// One fused iteration: the pp ladder on s0, the ring on s1, s3 and the fifth stream, and the hh
// ladder with the one-body sums and T X on s2 side by side (each needs only the amplitudes), then
// the assembly on s0.  The ladder is bound by HBM on one CTA per SM, the others by latency and the
// L2.
// mixed: the pp ladder runs on the tensor cores (split bf16) instead of the FP64 pipe.
int enqueue_fused_iteration(ccdgpu_handle *h, bool mixed) {
  int rc;
  const int gate = mixed ? 1 : 0;
  auto ladder = [&](cudaStream_t st) {
    return mixed ? launch_pp_ladder_tc(h, st) : launch_pp_ladder(h, st);
  };
  if (h->profiling) {
    // One family after another: ev 0 start, 1 after hh ladder, 2 after one-body, 3 after pp
    // ladder, 4/5 ring, 8 before and 6, 7 after the assembly.
    CK(cudaEventRecord(h->ev[0], h->s0));
    if ((rc = launch_hh_ladder(h, h->s0, gate))) return rc;
    CK(cudaEventRecord(h->ev[1], h->s0));
    if ((rc = launch_hh_post(h, h->s0, gate, mixed && h->tc_tx ? 0 : -1))) return rc;
    CK(cudaEventRecord(h->ev[2], h->s0));
    if ((rc = ladder(h->s0))) return rc;
    CK(cudaEventRecord(h->ev[3], h->s0));
    CK(cudaEventRecord(h->ev[4], h->s0));
    if ((rc = launch_tp_gather(h, h->s0, gate))) return rc;
    for (int k = 0; k < 3; k++)
      if ((rc = launch_ring_units(h, h->s0, gate, k))) return rc;
    CK(cudaEventRecord(h->ev[5], h->s0));
    CK(cudaEventRecord(h->ev[8], h->s0));
    if ((rc = launch_assemble_fused(h, h->s0, gate))) return rc;
    CK(cudaEventRecord(h->ev[6], h->s0));
    CK(cudaEventRecord(h->ev[7], h->s0));
    return CCDGPU_OK;
  }
  // Kernels reach the GPU in the order in which they become ready, and the CTAs of one wait behind
  // all CTAs of those before it; of branches that become ready together the one captured last comes
  // first.  So: the ladder (it needs an SM's registers before smaller CTAs take them), the hh
  // slices and the gather, then the short kernels that follow the hh slices, then the ring.
  // In a mixed iteration, whose ladder is short, a large ring waits for X as well as for the
  // gather, which end together: ahead of T X it would hold that back to the end of the iteration.
  // By its units of four and two warps, not waiting and waiting, us an iteration: EG N=54 752
  // 55.5, 57.1; 828 67.8, 67.4; 1134 95.2, 92.2; 1632 136.0, 135.0; PNM N=66 680 55.6, 58.8; 1014
  // 82.2, 80.5; 1416 123.5, 120.6.  In FP64 the ladder covers both, and waiting only starts the
  // ring later: EG N=54 578 47.2, 50.4; 1632 150.2, 151.0; PNM N=66 2136 206.1, 207.6.
  CK(cudaEventRecord(h->ev_fork, h->s0));
  CK(cudaStreamWaitEvent(h->s1, h->ev_fork, 0));
  CK(cudaStreamWaitEvent(h->s2, h->ev_fork, 0));
  if ((rc = launch_tp_gather(h, h->s1, gate))) return rc;
  if ((rc = launch_hh_ladder(h, h->s2, gate))) return rc;
  if (mixed && h->n_ring[0] + h->n_ring[1] > 800) {
    CK(cudaEventRecord(h->ev_join2, h->s2));
    CK(cudaStreamWaitEvent(h->s1, h->ev_join2, 0));
  }
  // The groups of units side by side; the first that the system has stays on s1.  (The one-warp units
  // behind the widest ones, a branch less, build and tear the loop graph down 0.1 ms faster each, but
  // EG N=54 |n|^2 <= 36 took 0.3 to 0.6 % longer to solve, and |n|^2 <= 21 8 % an iteration.)
  CK(cudaEventRecord(h->ev_fork3, h->s1));
  const struct { cudaStream_t st; cudaEvent_t ev; } branch[3] = {
      {h->s1, h->ev_join}, {h->s3, h->ev_join3}, {h->sset.s[4], h->sset.ev[16]}};
  int used = 0;
  for (int k = 0; k < 3; k++) {
    if (!h->n_ring[k]) continue;
    if (used) CK(cudaStreamWaitEvent(branch[used].st, h->ev_fork3, 0));
    if ((rc = launch_ring_units(h, branch[used++].st, gate, k))) return rc;
  }
  for (int k = 0; k < std::max(used, 1); k++) CK(cudaEventRecord(branch[k].ev, branch[k].st));
  if (mixed && h->tc_tx) {  // the ladder reads X
    CK(cudaEventRecord(h->ev_fork2, h->s2));
    CK(cudaStreamWaitEvent(h->s0, h->ev_fork2, 0));
  }
  if ((rc = launch_hh_post(h, h->s2, gate, mixed && h->tc_tx ? 0 : -1))) return rc;
  CK(cudaEventRecord(h->ev_join2, h->s2));
  if ((rc = ladder(h->s0))) return rc;
  for (int k = 0; k < std::max(used, 1); k++) CK(cudaStreamWaitEvent(h->s0, branch[k].ev, 0));
  CK(cudaStreamWaitEvent(h->s0, h->ev_join2, 0));
  if ((rc = launch_assemble_fused(h, h->s0, gate))) return rc;  // + energy and stop rule
  if (h->loop_capture && !h->n_asm_blocks) {  // else the assembly set the loop condition
    h->launches++;
    CK(launch_pdl(loop_ctl_kernel, 1, 32, 0, h->s0, (const Control *)h->ctl, h->loop_cond,
                  h->loop_capture == 2 ? 1 : 0));
  }
  return CCDGPU_OK;
}

// Table path stages (mirrors main.cpp:591-665).
int stage_onebody_tables(ccdgpu_handle *h, int holes, int particles) {
  if (!h->have_3body) return CCDGPU_ERR_UNSUPPORTED;
  if (holes) {
    onebody_tables_kernel<kOBHoles><<<(unsigned)h->np, kOBHoles, 0, h->s0>>>(
        h->o_h, h->v_h_hpp, h->old_h2pp_h1, h->old_h1pp_h2, h->diff_h2pp_h1, 0.5);
    h->launches++;
  }
  if (particles) {
    onebody_tables_kernel<kOBParticles><<<(unsigned)h->npart, kOBParticles, 0, h->s0>>>(
        h->o_p, h->old_p1_p2hh, h->v_phh_p, h->old_p2_p1hh, h->diff_p2_p1hh, -0.5);
    h->launches++;
  }
  return cuda_status(cudaGetLastError());
}
int stage_gather(ccdgpu_handle *h) {
  if (!h->have_3body) return CCDGPU_ERR_UNSUPPORTED;
  const int blocks = (int)std::min<int64_t>(ceil_div(h->n_t, 256), kSMs * 16);
  gather8_kernel<<<std::max(blocks, 1), 256, 0, h->s0>>>(h->n_t, h->flat, h->diff_h2pp_h1,
                                                         h->diff_p2_p1hh, h->r_phhp, h->gath);
  h->launches++;
  return cuda_status(cudaGetLastError());
}
int stage_assemble_tables(ccdgpu_handle *h, double mixing) {
  if (!h->have_3body) return CCDGPU_ERR_UNSUPPORTED;
  if (h->n_ranges) {
    assemble_tables_kernel<<<h->n_ranges, kAsmThreads, 0, h->s0>>>(
        h->ranges, h->chans, h->pp_pairs, h->hh_pairs, h->v_pphh, h->dmat, h->gath, h->n_t, h->eps,
        h->t[0], h->t[1], h->epart, mixing);
    h->launches++;
    CK(cudaGetLastError());
  }
  return CCDGPU_OK;
}

constexpr size_t kCtlUpload = offsetof(Control, err);  // what the host writes of it

int sync_ctl(ccdgpu_handle *h) {
  CK(cudaMemcpyAsync(h->h_ctl, h->ctl, sizeof(Control), cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  h->ctl_current = true;
  return CCDGPU_OK;
}
// The same where no kernel that writes the block has been launched since: nothing to read (a call
// that only launches one stage spent 20 of its 20 to 50 us on reading and writing it).
int fresh_ctl(ccdgpu_handle *h) {
  return h->ctl_current && h->h_ctl->trace_iter < 0 ? CCDGPU_OK : sync_ctl(h);
}

// read: fetch the error word first (otherwise sync_ctl just has).
int check_errors(ccdgpu_handle *h, bool read = true) {
  if (read) {
    CK(cudaMemcpyAsync(&h->h_ctl->err, h->err, sizeof(int32_t), cudaMemcpyDeviceToHost, h->s0));
    CK(cudaStreamSynchronize(h->s0));
  }
  if (h->h_ctl->err & kErrTimeout) {
    // Reported once: the handle stays usable (the timed-out iteration's amplitudes are
    // incomplete; ccdgpu_reset or ccdgpu_set_t2 starts over).  A ladder CTA that gave up may
    // have left its tile counter and exit ticket behind: zero them for the next launch.
    CK(cudaMemsetAsync(h->err, 0, sizeof(int32_t), h->s0));
    h->h_ctl->err = 0;
    if (h->sched) CK(cudaMemsetAsync(h->sched, 0, kSched * sizeof(int32_t), h->s0));
    return CCDGPU_ERR_TIMEOUT;
  }
  if (h->h_ctl->error & kErrNonFinite) return CCDGPU_ERR_NONFINITE;
  return CCDGPU_OK;
}

int set_ctl(ccdgpu_handle *h, int active, double tol, int64_t max_iters, double mixing,
            bool reset_loop, int parity = -1, int phase = 0) {
  int rc = fresh_ctl(h);
  if (rc) return rc;
  Control &c = *h->h_ctl;
  unsigned char was[kCtlUpload];
  std::memcpy(was, &c, kCtlUpload);
  if (parity >= 0) c.parity = parity;
  if (reset_loop) {
    c.e_prev = 100.0;
    c.e_diff = 1.0;
    c.iterations = 0;
    c.done = 0;
    c.error = 0;
    c.polish_iters = 0;
    std::memset(c.energies, 0, sizeof(c.energies));
  }
  c.phase = phase;
  c.polish_rel = h->opt.polish_threshold;
  c.active = active;
  c.tol = tol;
  c.max_iters = max_iters;
  c.mixing = mixing;
  // In stream order before what is launched next; the next host change of the mirror is either
  // after a synchronisation or followed by its own upload.
  if (std::memcmp(was, &c, kCtlUpload) != 0)
    CK(cudaMemcpyAsync(h->ctl, h->h_ctl, kCtlUpload, cudaMemcpyHostToDevice, h->s0));
  return CCDGPU_OK;
}

// The Control block of a new handle in one upload: what set_ctl(h, 0, 0.0, 100, 0.5, true)
// and ccdgpu_trace_arm(h, -1) would write over the zeroed device copy.
int init_ctl(ccdgpu_handle *h) {
  Control &c = *h->h_ctl;
  std::memset(&c, 0, sizeof(Control));
  c.e_prev = 100.0;
  c.e_diff = 1.0;
  c.polish_rel = h->opt.polish_threshold;
  c.max_iters = 100;
  c.mixing = 0.5;
  c.trace_iter = -1;
  for (int k = 0; k < kTraceKernels; k++) c.trace_first[k] = ~0ull;
  CK(cudaMemcpyAsync(h->ctl, h->h_ctl, kCtlUpload, cudaMemcpyHostToDevice, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  h->ctl_current = true;
  return CCDGPU_OK;
}

int fused_ready_graph(ccdgpu_handle *h, bool mixed) {
  cudaGraphExec_t &exec = mixed ? h->graph_tc : h->graph;
  if (exec) return CCDGPU_OK;
  cudaGraph_t g = nullptr;
  const int64_t before = h->launches;
  CK(cudaStreamBeginCapture(h->s0, cudaStreamCaptureModeThreadLocal));
  int rc = enqueue_fused_iteration(h, mixed);
  (mixed ? h->kernels_per_graph_tc : h->kernels_per_graph) = h->launches - before;
  h->launches = before;
  cudaError_t e = cudaStreamEndCapture(h->s0, &g);
  if (rc) { if (g) cudaGraphDestroy(g); return rc; }
  CK(e);
  e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  CK(e);
  return CCDGPU_OK;
}

// The device solve loop.  Graph: [WHILE c_mix { mixed iteration }] -> WHILE c64 { FP64
// iteration }; each body ends with the fused assembly, whose stop-rule CTA sets the body's
// condition (loop_ctl_kernel when a system has no assembly blocks).  Both
// conditions default to 1 at every launch; one launch runs until the stop rule fires or
// ctl->stop_at is reached.
int capture_loop_graph(ccdgpu_handle *h, bool mixed, cudaGraphExec_t *exec) {
  cudaGraph_t g = nullptr;
  CK(cudaGraphCreate(&g, 0));
  cudaGraphNode_t prev = nullptr;
  int rc = CCDGPU_OK;
  const int64_t before = h->launches;
  for (int pass = mixed ? 0 : 1; pass < 2 && !rc; pass++) {
    const bool body_mixed = pass == 0;
    cudaGraphConditionalHandle cond = 0;
    cudaError_t e = cudaGraphConditionalHandleCreate(&cond, g, 1, cudaGraphCondAssignDefault);
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = cond;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    cudaGraphNode_t node = nullptr;
    if (e == cudaSuccess) e = cudaGraphAddNode(&node, g, prev ? &prev : nullptr, prev ? 1 : 0, &p);
    if (e == cudaSuccess)
      e = cudaStreamBeginCaptureToGraph(h->s0, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      rc = cuda_status(e);
      break;
    }
    h->loop_capture = body_mixed ? 2 : 1;
    h->loop_cond = cond;
    const int64_t b0 = h->launches;
    rc = enqueue_fused_iteration(h, body_mixed);
    (body_mixed ? h->kernels_per_body_tc : h->kernels_per_body64) = h->launches - b0;
    h->loop_capture = 0;
    cudaGraph_t body = nullptr;
    e = cudaStreamEndCapture(h->s0, &body);
    if (!rc && e != cudaSuccess) rc = cuda_status(e);
    (void)cudaGetLastError();
    prev = node;
  }
  h->launches = before;
  if (!rc) {
    cudaError_t e = cudaGraphInstantiate(exec, g, 0);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      *exec = nullptr;
      rc = cuda_status(e);
    }
  }
  cudaGraphDestroy(g);
  return rc;
}

// Builds the loop graph a solve starts with (loop_tc for mixed handles, loop64 otherwise)
// once; any failure (for example a driver without conditional nodes, or without programmatic
// launches inside them, retried without) leaves the batched replay.
void ready_loop_graphs(ccdgpu_handle *h) {
  if (h->loop_state) return;
  const auto t0 = std::chrono::steady_clock::now();
  for (int attempt = 0; attempt < 2 && h->loop_state == 0; attempt++) {
    t_pdl = attempt == 0;
    const int rc = h->nt ? capture_loop_graph(h, true, &h->loop_tc)
                         : capture_loop_graph(h, false, &h->loop64);
    if (!rc) {
      h->loop_state = 1;
      h->loop_pdl = t_pdl;
    } else {
      if (h->loop64) cudaGraphExecDestroy(h->loop64);
      if (h->loop_tc) cudaGraphExecDestroy(h->loop_tc);
      h->loop64 = h->loop_tc = nullptr;
    }
  }
  t_pdl = true;
  if (h->loop_state == 0) h->loop_state = -1;
  h->loop_graph_ms = ms_since(t0);
}

// One table-path iteration: exactly the reference loop body.
int tables_iteration(ccdgpu_handle *h, double mixing, double *corr) {
  int rc;
  if ((rc = stage_onebody_tables(h, 0, 1))) return rc;     // calcT2Diff_p2_p1hh
  if ((rc = stage_onebody_tables(h, 1, 0))) return rc;     // calcT2Diff_h2pp_h1
  if ((rc = launch_ring(h, h->s0, 0))) return rc;   // calcT2Diff_phhp
  if ((rc = launch_pphh(h))) return rc;                    // calcT2Diff_pphh
  if ((rc = stage_gather(h))) return rc;                   // 8 x mapFromDistributed
  if ((rc = stage_assemble_tables(h, mixing))) return rc;  // calcT2_pphh
  if ((rc = launch_energy(h, h->s0, 2))) return rc;
  if ((rc = launch_map_to(h, h->s0, h->t[1], h->t[0]))) return rc;  // set + 5 x mapToDistributed
  (void)corr;
  return CCDGPU_OK;
}

}  // namespace

extern "C" {

void ccdgpu_default_options(ccdgpu_options *opt) {
  if (!opt) return;
  std::memset(opt, 0, sizeof(*opt));
  opt->device = 0;
  opt->precision = CCDGPU_PREC_FP64;
  opt->v_mode = CCDGPU_V_STORED;
  opt->path = CCDGPU_PATH_FUSED;
  opt->polish_threshold = 1e-6;
  opt->use_graph = 1;
  opt->device_loop = 1;
}

const char *ccdgpu_strerror(int status) {
  switch (status) {
    case CCDGPU_OK: return "ok";
    case CCDGPU_ERR_INVALID_ARGUMENT: return "invalid argument";
    case CCDGPU_ERR_CUDA: return "CUDA error";
    case CCDGPU_ERR_OUT_OF_MEMORY: return "out of device memory";
    case CCDGPU_ERR_BAD_TABLE: return "remap table out of range or not a bijection";
    case CCDGPU_ERR_NONFINITE: return "non-finite amplitudes or energy";
    case CCDGPU_ERR_NO_DEVICE: return "no CUDA device";
    case CCDGPU_ERR_UNSUPPORTED: return "unsupported problem or option";
    case CCDGPU_ERR_NOT_CONVERGED: return "not converged within the iteration cap";
    case CCDGPU_ERR_TIMEOUT: return "device wait timed out";
    default: return "unknown status";
  }
}

int ccdgpu_create(const ccdgpu_problem *prob, const ccdgpu_options *opt, ccdgpu_handle **out) {
  if (!prob || !out) return CCDGPU_ERR_INVALID_ARGUMENT;
  const auto t_create = std::chrono::steady_clock::now();
  *out = nullptr;
  if (!prob->sp_energy || !prob->chan_dims || !prob->chan_mod_dims || !prob->chan_maps ||
      !prob->three_body_dims || prob->n_particles == 0 || prob->n_particles >= prob->n_sp)
    return CCDGPU_ERR_INVALID_ARGUMENT;
  ccdgpu_handle *h = new (std::nothrow) ccdgpu_handle();
  if (!h) return CCDGPU_ERR_OUT_OF_MEMORY;
  if (opt) h->opt = *opt;
  else ccdgpu_default_options(&h->opt);
  switch (h->opt.precision) {
    case CCDGPU_PREC_FP64: h->nt = 0; break;
    case CCDGPU_PREC_MIXED_BF16: h->nt = 2; break;
    case CCDGPU_PREC_MIXED_BF16X3: h->nt = 3; break;
    default: delete h; return CCDGPU_ERR_UNSUPPORTED;
  }
  if (h->nt && h->opt.path != CCDGPU_PATH_FUSED) { delete h; return CCDGPU_ERR_UNSUPPORTED; }
  if (h->nt && !(h->opt.polish_threshold >= 0)) { delete h; return CCDGPU_ERR_INVALID_ARGUMENT; }
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0) { (void)cudaGetLastError(); delete h; return CCDGPU_ERR_NO_DEVICE; }
  if (h->opt.device < 0 || h->opt.device >= ndev) { delete h; return CCDGPU_ERR_INVALID_ARGUMENT; }
  int rc = cuda_status(cudaSetDevice(h->opt.device));
  if (!rc) rc = cuda_status(acquire_set(h->sset));
  if (!rc) {
    h->s0 = h->sset.s[0]; h->s1 = h->sset.s[1]; h->s2 = h->sset.s[2]; h->s3 = h->sset.s[3];
    for (int i = 0; i < 10; i++) h->ev[i] = h->sset.ev[i];
    h->ev_fork = h->sset.ev[10]; h->ev_fork2 = h->sset.ev[11]; h->ev_fork3 = h->sset.ev[12];
    h->ev_join = h->sset.ev[13]; h->ev_join2 = h->sset.ev[14]; h->ev_join3 = h->sset.ev[15];
  }
  if (!rc) rc = build(h, prob);
  if (!rc) rc = init_ctl(h);
  if (rc) { release(h); delete h; return rc; }
  h->create_ms[4] = ms_since(t_create);
  *out = h;
  return CCDGPU_OK;
}

void ccdgpu_release_cached_memory(void) {
  release_cache(-1);
  release_stream_pool();
}

void ccdgpu_destroy(ccdgpu_handle *h) {
  if (!h) return;
  cudaSetDevice(h->opt.device);
  if (h->s0) cudaStreamSynchronize(h->s0);
  release(h);
  delete h;
}

uint64_t ccdgpu_t2_size(const ccdgpu_handle *h) { return h ? (uint64_t)h->n_t : 0; }

int ccdgpu_reset(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  if (int rc = fresh_ctl(h)) return rc;
  // The fused path iterates on the packed amplitudes alone; its slabs follow when they are read.
  const bool fused = h->opt.path == CCDGPU_PATH_FUSED;
  const std::pair<double *, int64_t> z[] = {
      {h->tq[h->h_ctl->parity], h->n_q}, {h->old_phhp, h->n_m},
      {fused ? nullptr : h->t[0], h->n_t}, {fused ? nullptr : h->t[1], h->n_t},
      {h->old_h1pp_h2, h->n_h}, {h->old_h2pp_h1, h->n_h},
      {h->old_p1_p2hh, h->n_p}, {h->old_p2_p1hh, h->n_p}};
  for (const auto &b : z)
    if (b.first && b.second) CK(cudaMemsetAsync(b.first, 0, b.second * 8, h->s0));
  if (h->nt) CK(cudaMemsetAsync(h->tkt_tc, 0, (size_t)h->nt * h->n_tkttc * 2, h->s0));
  slabs_behind(h);
  h->chains_current = true;  // zeroed above
  h->tc_stale = false;
  if (int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, true)) return rc;
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}

int ccdgpu_set_t2(ccdgpu_handle *h, const double *t2, uint64_t n) {
  if (!h || !t2 || n != (uint64_t)h->n_t) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc;
  CK(cudaMemcpyAsync(h->t[1], t2, n * 8, cudaMemcpyHostToDevice, h->s0));
  if ((rc = launch_map_to(h, h->s0, h->t[1], h->t[0]))) return rc;
  if ((rc = launch_map_to(h, h->s0, h->t[1], h->t[0], 1))) return rc;
  slabs_loaded(h);
  unsigned long long irr = 0;
  CK(cudaMemsetAsync(h->irr + 1, 0, sizeof(irr), h->s0));
  if ((rc = launch_antisymmetry(h, h->t[1]))) return rc;
  CK(cudaMemcpyAsync(&irr, h->irr + 1, sizeof(irr), cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  h->irregular_t = irr != 0;
  return CCDGPU_OK;
}

int ccdgpu_mbpt2(ccdgpu_handle *h, int32_t init_t2, double *e_mbpt2) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc) return rc;
  if (h->n_ranges) {
    mbpt2_kernel<<<h->n_ranges, 256, 0, h->s0>>>(h->ranges, h->chans, h->pp_pairs, h->hh_pairs,
                                                  h->v_pphh, h->eps, init_t2 ? h->t[1] : nullptr,
                                                  h->epart);
    CK(cudaGetLastError());
  }
  if ((rc = launch_energy(h, h->s0, 0))) return rc;
  if (init_t2) {  // the amplitudes become the current ones, as after ccdgpu_set_t2
    if ((rc = launch_map_to(h, h->s0, h->t[1], h->t[0]))) return rc;
    slabs_loaded(h);
    h->irregular_t = false;  // V / D: as V_hhpp
  }
  double e = 0.0;
  CK(cudaMemcpyAsync(&e, h->e_out, 8, cudaMemcpyDeviceToHost, h->s0));
  rc = check_errors(h);
  if (e_mbpt2) *e_mbpt2 = h->n_ranges ? e : 0.0;
  return rc;
}

int ccdgpu_reference_energy(ccdgpu_handle *h, const double *sp_energy_bare, double *e_ref,
                            double *sp_energy_normal) {
  if (!h || !sp_energy_bare || !e_ref) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (!h->has_model) return CCDGPU_ERR_UNSUPPORTED;
  CK(cudaSetDevice(h->opt.device));
  const int nsp = (int)h->nsp;
  std::vector<double> out((size_t)nsp + 1);
  CK(cudaMemcpyAsync(h->eps_io, sp_energy_bare, (size_t)nsp * 8, cudaMemcpyHostToDevice, h->s0));
  normal_order_kernel<<<(nsp + 128) / 128, 128, 0, h->s0>>>(h->md, h->eps_io, nsp, (int)h->np,
                                                            h->eps_io + nsp);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(out.data(), h->eps_io + nsp, out.size() * 8, cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  *e_ref = out[nsp];
  if (sp_energy_normal) std::copy(out.begin(), out.begin() + nsp, sp_energy_normal);
  return CCDGPU_OK;
}

int ccdgpu_build_channels(const ccdgpu_channel_rule *rule, ccdgpu_channel_dims *dims,
                          ccdgpu_channel_dims *mod_dims, ccdgpu_pair *const lists[4],
                          ccdgpu_pair *const mod_lists[4], uint32_t *chan, uint32_t *mod_chan,
                          uint32_t *pos, uint32_t *mod_pos) {
  if (!rule || !rule->qn || !dims || !mod_dims || !lists || !mod_lists) return CCDGPU_ERR_INVALID_ARGUMENT;
  const uint64_t nsp = rule->n_sp, np = rule->n_particles, nch = rule->n_channels;
  if (np == 0 || np >= nsp || nch == 0 || rule->kind < CCDGPU_MODEL_PAIRING ||
      rule->kind > CCDGPU_MODEL_ELECTRON_GAS ||
      rule->qn_stride < (rule->kind == CCDGPU_MODEL_PAIRING ? 2 : 5) || rule->nmax < 0)
    return CCDGPU_ERR_INVALID_ARGUMENT;
  if (nsp > 65535 || nch * 4 >= (uint64_t(1) << 31)) return CCDGPU_ERR_UNSUPPORTED;
  const uint64_t npart = nsp - np, n = nsp * nsp;
  const uint64_t tot[4] = {npart * npart, np * np, np * npart, npart * np};  // pp, hh, hp, ph
  for (int k = 0; k < 4; k++)
    if (!lists[k] || !mod_lists[k]) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (rule->device >= 0) CK(cudaSetDevice(rule->device));
  cudaStream_t st = nullptr;
  CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  // One device block: qn, the per-pair arrays and the per-(channel, kind) arrays.
  size_t used = 0;
  auto take = [&](size_t bytes) {
    const size_t o = used;
    used += (bytes + 255) & ~size_t(255);
    return o;
  };
  const size_t o_qn = take(nsp * rule->qn_stride * 4), o_c0 = take(n * 4), o_mc0 = take(n * 4),
               o_codes = take(n * 4), o_mcodes = take(n * 4), o_chan = take(n * 4),
               o_mchan = take(n * 4), o_pos = take(n * 4), o_mpos = take(n * 4),
               o_cnt = take(nch * 16), o_mcnt = take(nch * 16), o_fill = take(nch * 16),
               o_mfill = take(nch * 16), o_err = take(4), o_zero_end = used,
               o_inv = take(nch * 4), o_seg = take(nch * 16), o_mseg = take(nch * 16),
               o_segs = take(nch * 8 * sizeof(PairSegment));
  void *base = nullptr;
  size_t got = 0;
  int rc = CCDGPU_OK;
  std::vector<uint32_t> cnt(nch * 4), mcnt(nch * 4);
  std::vector<uint32_t> inv(nch), seg(nch * 4), mseg(nch * 4), codes(n), mcodes(n);
  std::vector<PairSegment> segs;
  int32_t err = 0;
  auto at = [&](size_t o) { return static_cast<char *>(base) + o; };
  auto run = [&]() -> int {
    CK(dev_alloc(used, &base, &got));
    CK(cudaMemsetAsync(at(o_cnt), 0, o_zero_end - o_cnt, st));
    CK(cudaMemcpyAsync(at(o_qn), rule->qn, nsp * rule->qn_stride * 4, cudaMemcpyHostToDevice, st));
    ChannelRuleDev r{reinterpret_cast<const int32_t *>(at(o_qn)), rule->kind, rule->qn_stride,
                     rule->nmax, rule->chan_tz_max, rule->mod_chan_tz_max, nsp, np, nch};
    const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, kSMs * 16);
    uint32_t *c0 = reinterpret_cast<uint32_t *>(at(o_c0)), *mc0 = reinterpret_cast<uint32_t *>(at(o_mc0));
    pair_channel_kernel<<<grid, 256, 0, st>>>(r, c0, mc0, reinterpret_cast<uint32_t *>(at(o_cnt)),
                                               reinterpret_cast<uint32_t *>(at(o_mcnt)),
                                               reinterpret_cast<int32_t *>(at(o_err)));
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(cnt.data(), at(o_cnt), nch * 16, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(mcnt.data(), at(o_mcnt), nch * 16, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&err, at(o_err), 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (err) return CCDGPU_ERR_INVALID_ARGUMENT;  // a pair outside the channel slots
    // Channel order, dimensions and segment starts (kinds one after another).
    std::vector<ccdgpu_channel_dims> d0(nch), md0(nch);
    for (uint64_t c = 0; c < nch; c++) {
      d0[c] = {cnt[c * 4 + 0], cnt[c * 4 + 1], cnt[c * 4 + 2], cnt[c * 4 + 3]};
      md0[c] = {mcnt[c * 4 + 0], mcnt[c * 4 + 1], mcnt[c * 4 + 2], mcnt[c * 4 + 3]};
    }
    const std::vector<uint64_t> order = ffd_channel_order(d0);
    for (uint64_t i = 0; i < nch; i++) {
      inv[order[i]] = (uint32_t)i;
      dims[i] = d0[order[i]];
      mod_dims[i] = md0[order[i]];
    }
    uint64_t base_k = 0;
    for (int k = 0; k < 4; k++) {
      uint64_t o = base_k, mo = base_k;
      for (uint64_t i = 0; i < nch; i++) {
        const uint64_t len = (&dims[i].pp)[k], mlen = (&mod_dims[i].pp)[k];
        if (len > (uint64_t)kMaxSegment || mlen > (uint64_t)kMaxSegment) return CCDGPU_ERR_UNSUPPORTED;
        seg[i * 4 + k] = (uint32_t)o;
        mseg[i * 4 + k] = (uint32_t)mo;
        if (len) segs.push_back(PairSegment{(uint32_t)o, (uint32_t)len, 0, 0});
        if (mlen) segs.push_back(PairSegment{(uint32_t)mo, (uint32_t)mlen, 1, 0});
        o += len;
        mo += mlen;
      }
      if (o - base_k != tot[k] || mo - base_k != tot[k]) return CCDGPU_ERR_INVALID_ARGUMENT;
      base_k += tot[k];
    }
    if (segs.size() > nch * 8) return CCDGPU_ERR_INVALID_ARGUMENT;
    CK(cudaMemcpyAsync(at(o_inv), inv.data(), nch * 4, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(at(o_seg), seg.data(), nch * 16, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(at(o_mseg), mseg.data(), nch * 16, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(at(o_segs), segs.data(), segs.size() * sizeof(PairSegment),
                       cudaMemcpyHostToDevice, st));
    uint32_t *codes_d = reinterpret_cast<uint32_t *>(at(o_codes));
    uint32_t *mcodes_d = reinterpret_cast<uint32_t *>(at(o_mcodes));
    place_pairs_kernel<<<grid, 256, 0, st>>>(
        nsp, np, c0, mc0, reinterpret_cast<const uint32_t *>(at(o_inv)),
        reinterpret_cast<const uint32_t *>(at(o_seg)), reinterpret_cast<const uint32_t *>(at(o_mseg)),
        reinterpret_cast<uint32_t *>(at(o_fill)), reinterpret_cast<uint32_t *>(at(o_mfill)),
        codes_d, mcodes_d, reinterpret_cast<uint32_t *>(at(o_chan)),
        reinterpret_cast<uint32_t *>(at(o_mchan)));
    CK(cudaGetLastError());
    if (!segs.empty()) {
      sort_segments_kernel<<<(unsigned)segs.size(), 512, 0, st>>>(
          reinterpret_cast<const PairSegment *>(at(o_segs)), codes_d, mcodes_d,
          reinterpret_cast<uint32_t *>(at(o_pos)), reinterpret_cast<uint32_t *>(at(o_mpos)));
      CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(codes.data(), codes_d, n * 4, cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(mcodes.data(), mcodes_d, n * 4, cudaMemcpyDeviceToHost, st));
    if (chan) CK(cudaMemcpyAsync(chan, at(o_chan), n * 4, cudaMemcpyDeviceToHost, st));
    if (mod_chan) CK(cudaMemcpyAsync(mod_chan, at(o_mchan), n * 4, cudaMemcpyDeviceToHost, st));
    if (pos) CK(cudaMemcpyAsync(pos, at(o_pos), n * 4, cudaMemcpyDeviceToHost, st));
    if (mod_pos) CK(cudaMemcpyAsync(mod_pos, at(o_mpos), n * 4, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    // Codes -> pairs.
    uint64_t kb[4] = {0, tot[0], tot[0] + tot[1], tot[0] + tot[1] + tot[2]};
    for (int k = 0; k < 4; k++) {
#pragma omp parallel for schedule(static)
      for (int64_t j = 0; j < (int64_t)tot[k]; j++) {
        const uint32_t x = codes[kb[k] + j], y = mcodes[kb[k] + j];
        lists[k][j] = ccdgpu_pair{x / nsp, x % nsp};
        mod_lists[k][j] = ccdgpu_pair{y / nsp, y % nsp};
      }
    }
    return CCDGPU_OK;
  };
  rc = run();
  (void)cudaStreamSynchronize(st);
  if (base) dev_free(base, got);
  cudaStreamDestroy(st);
  if (rc) (void)cudaGetLastError();
  return rc;
}

int ccdgpu_get_t2(ccdgpu_handle *h, double *t2, uint64_t n) {
  if (!h || !t2 || n != (uint64_t)h->n_t) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = fresh_ctl(h);
  if (rc) return rc;
  if ((rc = materialize_t(h))) return rc;
  const double *src = h->opt.path == CCDGPU_PATH_TABLES ? h->t[1] : h->t[0];
  return copy_from_device(h, reinterpret_cast<char *>(t2), reinterpret_cast<const char *>(src),
                          n * 8);
}

int ccdgpu_step(ccdgpu_handle *h, double mixing, double *e_corr) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  const bool inject = h->inject_next_step;
  h->inject_next_step = false;
  int rc = set_ctl(h, 0, h->h_ctl->tol, INT64_MAX / 2, mixing, false);
  if (rc) return rc;
  if (inject) {
    const int32_t one = 1;
    CK(cudaMemcpyAsync(&h->ctl->inject, &one, sizeof(one), cudaMemcpyHostToDevice, h->s0));
  }
  if (h->opt.path == CCDGPU_PATH_TABLES) {
    rc = tables_iteration(h, mixing, nullptr);
  } else if (!(rc = refresh_tc_image(h))) {
    rc = enqueue_fused_iteration(h, h->nt > 0);
    slabs_behind(h);
    h->d_from = h->nt ? 2 : 1;
  }
  if (inject) {  // the fault applies to this iteration only
    const int32_t zero = 0;
    CK(cudaMemcpyAsync(&h->ctl->inject, &zero, sizeof(zero), cudaMemcpyHostToDevice, h->s0));
  }
  if (rc) return rc;
  if ((rc = sync_ctl(h))) return rc;
  if ((rc = check_errors(h, false))) return rc;
  if (e_corr) *e_corr = h->h_ctl->e_corr;
  return std::isfinite(h->h_ctl->e_corr) ? CCDGPU_OK : CCDGPU_ERR_NONFINITE;
}

}  // extern "C"

namespace {

// A solve in two halves, so that a batch can put every handle's device loop in flight before
// waiting for any of them.
struct SolveState {
  bool fused = false, mixed = false, graph = false, device_loop = false;
  double tol = 0;
  int64_t cap = 0, it0 = 0, pol0 = 0;
  std::chrono::steady_clock::time_point t0;
};
constexpr int64_t kLoopChunk = 128;  // iterations one device-loop launch may run

// Device loop: launch up to kLoopChunk iterations without the host (no synchronisation).
int loop_launch(ccdgpu_handle *h, SolveState &st) {
  Control &c = *h->h_ctl;
  st.it0 = c.iterations;
  st.pol0 = c.polish_iters;
  c.stop_at = c.iterations + kLoopChunk;
  CK(cudaMemcpyAsync(&h->ctl->stop_at, &c.stop_at, sizeof(int64_t), cudaMemcpyHostToDevice,
                     h->s0));
  cudaGraphExec_t &g = st.mixed && c.phase == 1 ? h->loop_tc : h->loop64;
  if (!g) {  // a mixed handle's FP64 loop, first needed now (the stream is idle here)
    t_pdl = h->loop_pdl;
    const int rc = capture_loop_graph(h, false, &g);
    t_pdl = true;
    if (rc) return rc;
  }
  h->ctl_current = false;
  CK(cudaGraphLaunch(g, h->s0));
  return CCDGPU_OK;
}

int solve_begin(ccdgpu_handle *h, double tol, int64_t max_iters, double mixing, SolveState &st) {
  if (!h || max_iters < 0 || !(tol >= 0)) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  st.fused = h->opt.path == CCDGPU_PATH_FUSED;
  st.mixed = st.fused && h->nt > 0;
  st.tol = tol;
  st.cap = max_iters + 1;
  // A mixed solve starts in phase 1 (tensor-core ladder) and finishes in phase 2 (FP64).
  int rc = set_ctl(h, 1, tol, max_iters, mixing, true, -1, st.mixed ? 1 : 0);
  if (rc) return rc;
  st.graph = st.fused && h->opt.use_graph && !h->profiling;
  if (st.graph && h->opt.device_loop) ready_loop_graphs(h);
  st.device_loop = st.graph && h->opt.device_loop && h->loop_state == 1;
  if (st.graph && !st.device_loop && (rc = fused_ready_graph(h, false))) return rc;
  if (st.graph && !st.device_loop && st.mixed && (rc = fused_ready_graph(h, true))) return rc;
  if (st.fused) {
    if ((rc = refresh_tc_image(h))) return rc;
    slabs_behind(h);
    h->d_from = 0;  // until solve_finish
  }
  st.t0 = std::chrono::steady_clock::now();
  if (st.device_loop) return loop_launch(h, st);
  return CCDGPU_OK;
}

int solve_finish(ccdgpu_handle *h, SolveState &st, double mixing, ccdgpu_result *res) {
  CK(cudaSetDevice(h->opt.device));
  int rc;
  int64_t launched = 0;
  while (st.device_loop) {
    if ((rc = sync_ctl(h))) return rc;
    Control &c = *h->h_ctl;
    const int64_t fp = (c.polish_iters - st.pol0) + (st.mixed ? 0 : c.iterations - st.it0);
    h->launches += (c.iterations - st.it0 - fp) * h->kernels_per_body_tc + fp * h->kernels_per_body64;
    if (c.done || c.iterations >= st.cap || c.iterations == st.it0) break;
    if ((rc = loop_launch(h, st))) return rc;
  }
  while (!st.device_loop) {
    // Iterations are launched in batches; once the device-side stop rule fires the remaining
    // launches of the batch return immediately.
    const int64_t batch = (st.fused && !h->profiling)
                              ? std::min<int64_t>(launched < 8 ? 4 : 8, st.cap - launched)
                              : 1;
    // The phase can only change inside a batch from 1 to 2; mixed iterations that follow
    // the switch in the same batch are no-ops on the device.
    const bool mphase = st.mixed && h->h_ctl->phase == 1;
    for (int64_t b = 0; b < batch; b++) {
      if (st.graph) CK(cudaGraphLaunch(mphase ? h->graph_tc : h->graph, h->s0));
      else if (st.fused) { if ((rc = enqueue_fused_iteration(h, mphase))) return rc; }
      else {
        if ((rc = tables_iteration(h, mixing, nullptr))) return rc;
      }
    }
    launched += batch;
    h->ctl_current = false;
    if (st.graph)
      h->launches += batch * (mphase ? h->kernels_per_graph_tc : h->kernels_per_graph);
    if ((rc = sync_ctl(h))) return rc;
    if (h->profiling && st.fused && !st.graph) {
      float a = 0, b = 0, c = 0, d = 0, e = 0, f = 0;
      cudaEventElapsedTime(&a, h->ev[0], h->ev[1]);
      cudaEventElapsedTime(&b, h->ev[1], h->ev[2]);
      cudaEventElapsedTime(&c, h->ev[2], h->ev[3]);
      cudaEventElapsedTime(&d, h->ev[4], h->ev[5]);
      cudaEventElapsedTime(&e, h->ev[8], h->ev[7]);
      cudaEventElapsedTime(&f, h->ev[0], h->ev[7]);
      h->prof.ms_hh_ladder += a;
      h->prof.ms_onebody += b;
      h->prof.ms_ladder += c;
      h->prof.ms_ring += d;
      h->prof.ms_assemble += e;
      h->prof.ms_total += f;
      h->prof.iterations += 1;
    }
    if (h->h_ctl->done || launched >= st.cap) break;
  }
  auto t1 = std::chrono::steady_clock::now();
  if (st.fused) {
    // The last iteration was an FP64 one unless a mixed solve never left its mixed phase.
    const bool last64 = !st.mixed || h->h_ctl->polish_iters > 0;
    h->d_from = last64 ? 1 : 2;
    if (st.mixed && last64) h->tc_stale = true;
  }
  // The result reflects the control block also when the solve failed (for example non-finite
  // amplitudes of a diverging iteration); the status says so.
  const Control &c = *h->h_ctl;
  if (res) {
    res->e_corr = c.e_corr;
    res->e_diff = c.e_diff;
    res->iterations = c.iterations;
    res->converged = std::fabs(c.e_diff) <= st.tol ? 1 : 0;
    res->polish_iterations = (int32_t)c.polish_iters;
    res->seconds = std::chrono::duration<double>(t1 - st.t0).count();
  }
  return check_errors(h, false);
}

}  // namespace

extern "C" {

int ccdgpu_solve(ccdgpu_handle *h, double tol, int64_t max_iters, double mixing, ccdgpu_result *res) {
  SolveState st;
  int rc = solve_begin(h, tol, max_iters, mixing, st);
  if (rc) return rc;
  return solve_finish(h, st, mixing, res);
}

int ccdgpu_solve_batch(ccdgpu_handle *const *hs, int32_t n, double tol, int64_t max_iters,
                       double mixing, ccdgpu_result *res) {
  if (!hs || n < 0) return CCDGPU_ERR_INVALID_ARGUMENT;
  for (int32_t i = 0; i < n; i++)
    for (int32_t j = 0; j < i; j++)
      if (!hs[i] || hs[i] == hs[j]) return CCDGPU_ERR_INVALID_ARGUMENT;
  std::vector<SolveState> st(n);
  int first_rc = CCDGPU_OK;
  std::vector<int> begun(n, 0);
  // Every handle's device loop goes in flight on its own streams before any is waited for.
  for (int32_t i = 0; i < n; i++) {
    const int rc = solve_begin(hs[i], tol, max_iters, mixing, st[i]);
    if (rc && !first_rc) first_rc = rc;
    begun[i] = rc == CCDGPU_OK;
  }
  for (int32_t i = 0; i < n; i++) {
    if (!begun[i]) continue;
    const int rc = solve_finish(hs[i], st[i], mixing, res ? &res[i] : nullptr);
    if (rc && !first_rc) first_rc = rc;
  }
  return first_rc;
}

int ccdgpu_energy_history(ccdgpu_handle *h, double *out, int64_t cap, int64_t *n_out) {
  if (!h || cap < 0) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = fresh_ctl(h);
  if (rc) return rc;
  const int64_t n = std::min<int64_t>(h->h_ctl->iterations, 128);
  if (n_out) *n_out = n;
  if (out) std::memcpy(out, h->h_ctl->energies, sizeof(double) * std::min(n, cap));
  return CCDGPU_OK;
}

int ccdgpu_calc_t2diff_p2_p1hh(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc || (rc = ready_slabs(h)) || (rc = stage_onebody_tables(h, 0, 1))) return rc;
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}
int ccdgpu_calc_t2diff_h2pp_h1(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc || (rc = ready_slabs(h)) || (rc = stage_onebody_tables(h, 1, 0))) return rc;
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}
int ccdgpu_calc_t2diff_phhp(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc || (rc = ready_slabs(h)) || (rc = launch_ring(h, h->s0, 0))) return rc;
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}
int ccdgpu_calc_t2diff_pphh(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc || (rc = ready_slabs(h)) || (rc = launch_pphh(h))) return rc;
  h->d_from = 0;
  return check_errors(h);
}
int ccdgpu_map_from_distributed(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = stage_gather(h);
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}
int ccdgpu_calc_t2_pphh(ccdgpu_handle *h, double mixing, double *corr) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = ready_slabs(h);
  if (rc || (rc = stage_assemble_tables(h, mixing)) || (rc = launch_energy(h, h->s0, 0))) return rc;
  h->t2_staged = true;
  double e = 0;
  CK(cudaMemcpyAsync(&e, h->e_out, 8, cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  if (corr) *corr = e;
  return CCDGPU_OK;
}
int ccdgpu_map_to_distributed(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  int rc = ready_slabs(h);
  const bool staged = h->t2_staged || h->opt.path == CCDGPU_PATH_TABLES;
  if (rc || (rc = launch_map_to(h, h->s0, h->t[staged ? 1 : 0], h->t[0]))) return rc;
  slabs_loaded(h);
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}

int ccdgpu_read_chain(ccdgpu_handle *h, int32_t chain, double *out, uint64_t n, uint64_t *n_out) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = fresh_ctl(h);
  if (rc) return rc;
  const double *src = nullptr;
  uint64_t len = 0;
  const bool tables = h->opt.path == CCDGPU_PATH_TABLES;
  switch (chain) {
    case CCDGPU_CHAIN_T2: src = h->t[tables ? 1 : 0]; len = h->n_t; break;
    case CCDGPU_CHAIN_T2_OLD: src = h->t[0]; len = h->n_t; break;
    case CCDGPU_CHAIN_DIFF_PPHH: src = h->dmat; len = h->n_t; break;
    case CCDGPU_CHAIN_DIFF_PHHP: src = h->r_phhp; len = h->n_m; break;
    case CCDGPU_CHAIN_OLD_PHHP: src = h->old_phhp; len = h->n_m; break;
    case CCDGPU_CHAIN_DIFF_H2PP_H1: src = h->diff_h2pp_h1; len = h->n_h; break;
    case CCDGPU_CHAIN_DIFF_P2_P1HH: src = h->diff_p2_p1hh; len = h->n_p; break;
    default:
      if (chain >= CCDGPU_CHAIN_GATHERED0 && chain < CCDGPU_CHAIN_GATHERED0 + 8 && h->gath) {
        src = h->gath + (int64_t)(chain - CCDGPU_CHAIN_GATHERED0) * h->n_t;
        len = h->n_t;
      }
  }
  if (!src && !(chain >= 0 && chain <= 7)) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (n_out) *n_out = len;
  if (!out) return CCDGPU_OK;
  if (!src) return CCDGPU_ERR_UNSUPPORTED;
  if (n < len) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (chain == CCDGPU_CHAIN_OLD_PHHP && !h->chains_current) {
    // The fused path's iterations do not keep this slab.
    if ((rc = launch_phhp_gather(h, h->s0))) return rc;
    CK(cudaStreamSynchronize(h->s0));
  }
  if (chain == CCDGPU_CHAIN_DIFF_PPHH && (rc = materialize_d(h))) return rc;
  if ((chain == CCDGPU_CHAIN_T2 || chain == CCDGPU_CHAIN_T2_OLD) && (rc = materialize_t(h)))
    return rc;
  CK(cudaMemcpyAsync(out, src, len * 8, cudaMemcpyDeviceToHost, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}

int ccdgpu_get_profile(ccdgpu_handle *h, ccdgpu_profile *prof) {
  if (!h || !prof) return CCDGPU_ERR_INVALID_ARGUMENT;
  *prof = h->prof;
  prof->launches = h->launches;
  for (int k = 0; k < 5; k++) prof->ms_create[k] = h->create_ms[k];
  prof->ms_loop_graph = h->loop_graph_ms;
  return CCDGPU_OK;
}
int ccdgpu_enable_profiling(ccdgpu_handle *h, int32_t on) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  h->profiling = on != 0;
  h->prof = ccdgpu_profile{};
  return CCDGPU_OK;
}
void *ccdgpu_stream(ccdgpu_handle *h) { return h ? (void *)h->s0 : nullptr; }

int ccdgpu_inject_wait_timeout(ccdgpu_handle *h) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  h->inject_next_step = true;
  return CCDGPU_OK;
}

// Each class of the other kernels launched alone, `reps` times between CUDA events on the handle's
// stream; with the executed flops and the algorithmic bytes of each class.
int ccdgpu_kernel_profile(ccdgpu_handle *h, int32_t reps, double *ms, double *flops,
                          double *bytes) {
  if (!h || reps < 1 || !ms || !flops || !bytes) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc) return rc;
  if ((rc = materialize_d(h))) return rc;  // the kernels overwrite what it is expanded from
  for (int k = 0; k < 7; k++) ms[k] = flops[k] = bytes[k] = 0;
  // Ring (fused path): S = T' (A + C T') + B T' per pair of channels; reads A, B, C, T' and the
  // destinations, writes S.  The small class is launched with the gather of the T' images.
  for (int k = 0; k < 3; k++) {
    flops[k] = h->ring_flops[k];
    bytes[k] = h->ring_bytes[k];
  }
  // hh ladder: P = V_hhpp T over the packed rows and r = row dots; reads packed V and T, writes
  // the slice partials of P and r.  Reduction: reads the partials and V_hhhh, writes X and s.
  for (const ChanInfo &a : h->host_chans) {
    const int k = a.hk <= 8 ? 3 : 4;
    const double hk2 = (double)a.hk * a.hk;
    flops[k] += 2.0 * a.pk * a.hk * (a.hk + 1.0);
    bytes[k] += a.hk ? 16.0 * a.pk * a.hk + 8.0 * a.nhht * hk2 + 8.0 * a.pk : 0.0;
    flops[6] += (double)a.nhht * hk2;
    bytes[6] += 8.0 * a.nhht * hk2 + 16.0 * hk2 + 8.0 * a.hk;
  }
  // One-body: segmented sums of s and r (one value per pair) into x_k and y_a; and T X (reads T and
  // X, writes 0.5 T X) where the handle's iterations have it here.
  bytes[5] = 16.0 * (double)(h->nsp) + 12.0 * (double)h->n_list;
  for (const ChanInfo &a : h->host_chans) {
    if (!a.nmt || h->tc_tx) continue;
    flops[5] += 2.0 * a.pk * a.hk * (double)a.hk;
    bytes[5] += 16.0 * a.pk * a.hk + 8.0 * a.hk * (double)a.hk;
  }
  for (int k = 0; k < 7; k++) {
    auto launch = [&]() -> int {
      if (k == 0)
        if (const int r = launch_tp_gather(h, h->s0, 0)) return r;
      if (k <= 2) return launch_ring_units(h, h->s0, 0, 2 - k);
      if (k <= 4) return launch_hh_ladder(h, h->s0, 0, k - 3);
      if (k == 6) return launch_hh_ladder(h, h->s0, 0, 2);
      return launch_hh_post(h, h->s0, 0, h->tc_tx ? 0 : -1);
    };
    if ((rc = launch())) return rc;  // warm-up
    CK(cudaEventRecord(h->ev[0], h->s0));
    for (int i = 0; i < reps && !rc; i++) rc = launch();
    if (rc) return rc;
    CK(cudaEventRecord(h->ev[1], h->s0));
    CK(cudaEventSynchronize(h->ev[1]));
    float t = 0;
    CK(cudaEventElapsedTime(&t, h->ev[0], h->ev[1]));
    ms[k] = t / reps;
  }
  return check_errors(h);
}

// Each pp-ladder class launched alone (FP64 thin, mid, wide; tensor-core ladder), likewise; flops
// packed: rows a<b, columns i<j, K over c<d.
int ccdgpu_ladder_profile(ccdgpu_handle *h, int32_t reps, double *ms, double *flops,
                          double *bytes) {
  if (!h || reps < 1 || !ms || !flops || !bytes) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc) return rc;
  if ((rc = materialize_d(h))) return rc;  // the kernels overwrite what it is expanded from
  for (int k = 0; k < 4; k++) ms[k] = flops[k] = bytes[k] = 0;
  for (const ChanInfo &a : h->host_chans) {
    if (!a.nmt) continue;
    const int k = ladder_class(a.hs);
    // Algorithmic traffic: a symmetric channel's V once on and above the diagonal.
    const double v = (double)a.pk * a.pk, q = (double)a.pk * a.hk;
    flops[k] += 2.0 * v * a.hk;
    bytes[k] += 8.0 * ((a.sym ? 0.5 * (v + a.pk) : v) + 2.0 * q);
    if (h->nt) {
      flops[3] += 2.0 * v * a.hk;
      bytes[3] += 2.0 * h->nt * ((h->tc_gen ? 0.0 : v) + q) + 8.0 * q;
    }
  }
  for (int k = 0; k < 4; k++) {
    if (k < 3 && !h->n_cls[k]) continue;
    if (k == 3 && !h->n_tc_tiles) continue;
    auto launch = [&]() -> int {
      return k == 3 ? launch_pp_ladder_tc(h, h->s0) : launch_pp_ladder(h, h->s0, k);
    };
    if ((rc = launch())) return rc;  // warm-up
    CK(cudaEventRecord(h->ev[0], h->s0));
    for (int i = 0; i < reps && !rc; i++) rc = launch();
    if (rc) return rc;
    CK(cudaEventRecord(h->ev[1], h->s0));
    CK(cudaEventSynchronize(h->ev[1]));
    float t = 0;
    CK(cudaEventElapsedTime(&t, h->ev[0], h->ev[1]));
    ms[k] = t / reps;
  }
  return check_errors(h);
}

int ccdgpu_set_schedule(ccdgpu_handle *h, const ccdgpu_schedule *sch) {
  if (!h || !sch || sch->thin_split_mul < 1 || sch->wide_split_mul < 1 || sch->tc_split_mul < 1 ||
      sch->mid_split_mul < 0)
    return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  return make_ladder_tiles(h, *sch);
}

int ccdgpu_get_schedule(const ccdgpu_handle *h, ccdgpu_schedule *sch) {
  if (!h || !sch) return CCDGPU_ERR_INVALID_ARGUMENT;
  *sch = h->schedule;
  return CCDGPU_OK;
}

// Times `reps` launches of the handle's pp ladders for each candidate schedule (CUDA events on
// the handle's stream; the ladders only overwrite the iteration's D) and keeps the fastest.
int ccdgpu_autotune(ccdgpu_handle *h, int32_t reps, ccdgpu_schedule *chosen, double *ms_fp64,
                    double *ms_tc) {
  if (!h || reps < 1) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = set_ctl(h, 0, h->h_ctl->tol, h->h_ctl->max_iters, h->h_ctl->mixing, false);
  if (rc) return rc;
  auto time_ladder = [&](bool tc, double *ms) -> int {
    int r = tc ? launch_pp_ladder_tc(h, h->s0) : launch_pp_ladder(h, h->s0);  // warm-up
    if (r) return r;
    CK(cudaEventRecord(h->ev[0], h->s0));
    for (int i = 0; i < reps && !r; i++) r = tc ? launch_pp_ladder_tc(h, h->s0) : launch_pp_ladder(h, h->s0);
    if (r) return r;
    CK(cudaEventRecord(h->ev[1], h->s0));
    CK(cudaEventSynchronize(h->ev[1]));
    float t = 0;
    CK(cudaEventElapsedTime(&t, h->ev[0], h->ev[1]));
    *ms = t / reps;
    return check_errors(h);
  };
  ccdgpu_schedule best = h->schedule;
  double best64 = 0, besttc = 0;
  // FP64 ladder: split factors of the thin and the mid/wide classes (mid as wide), then the
  // mid class's own.
  const int thin_c[] = {1, 2, 4}, wide_c[] = {1, 2, 3, 6, 12, 24, 48};
  bool first = true;
  best.mid_split_mul = 0;
  for (int tm : thin_c)
    for (int wm : wide_c) {
      ccdgpu_schedule c = best;
      c.thin_split_mul = tm;
      c.wide_split_mul = wm;
      if ((rc = make_ladder_tiles(h, c))) return rc;
      double ms = 0;
      if ((rc = time_ladder(false, &ms))) return rc;
      if (first || ms < best64) { best64 = ms; best.thin_split_mul = tm; best.wide_split_mul = wm; }
      first = false;
    }
  for (int mm : wide_c) {
    ccdgpu_schedule c = best;
    c.mid_split_mul = mm;
    if ((rc = make_ladder_tiles(h, c))) return rc;
    double ms = 0;
    if ((rc = time_ladder(false, &ms))) return rc;
    if (ms < best64) { best64 = ms; best.mid_split_mul = mm; }
  }
  // Tensor-core ladder: split factor.
  if (h->nt) {
    first = true;
    const int tc_c[] = {1, 2, 4, 8, 16};
    for (int tm : tc_c) {
      ccdgpu_schedule c = best;
      c.tc_split_mul = tm;
      if ((rc = make_ladder_tiles(h, c))) return rc;
      double ms = 0;
      if ((rc = time_ladder(true, &ms))) return rc;
      if (first || ms < besttc) { besttc = ms; best.tc_split_mul = tm; }
      first = false;
    }
  }
  if ((rc = make_ladder_tiles(h, best))) return rc;
  if (chosen) *chosen = best;
  if (ms_fp64) *ms_fp64 = best64;
  if (ms_tc) *ms_tc = besttc;
  return CCDGPU_OK;
}

int ccdgpu_trace_arm(ccdgpu_handle *h, int64_t iteration) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = sync_ctl(h);
  if (rc) return rc;
  Control &c = *h->h_ctl;
  c.trace_iter = iteration;
  for (int k = 0; k < kTraceKernels; k++) {
    c.trace_first[k] = ~0ull;
    c.trace_last[k] = 0;
    c.trace_end[k] = 0;
  }
  CK(cudaMemcpyAsync(h->ctl, h->h_ctl, kCtlUpload, cudaMemcpyHostToDevice, h->s0));
  CK(cudaStreamSynchronize(h->s0));
  return CCDGPU_OK;
}

int ccdgpu_trace_read(ccdgpu_handle *h, uint64_t *first, uint64_t *last, int32_t n) {
  if (!h || !first || !last || n < 0) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = sync_ctl(h);
  if (rc) return rc;
  for (int k = 0; k < n && k < kTraceKernels; k++) {
    first[k] = h->h_ctl->trace_first[k];
    last[k] = h->h_ctl->trace_last[k];
  }
  return CCDGPU_OK;
}
int ccdgpu_trace_read_end(ccdgpu_handle *h, uint64_t *end, int32_t n) {
  if (!h || !end || n < 0) return CCDGPU_ERR_INVALID_ARGUMENT;
  CK(cudaSetDevice(h->opt.device));
  int rc = sync_ctl(h);
  if (rc) return rc;
  for (int k = 0; k < n && k < kTraceKernels; k++) end[k] = h->h_ctl->trace_end[k];
  return CCDGPU_OK;
}
int ccdgpu_work_per_iteration(const ccdgpu_handle *h, double *flops, double *v_pppp_bytes,
                              double *ladder_flops) {
  if (!h) return CCDGPU_ERR_INVALID_ARGUMENT;
  if (flops) *flops = h->flops;
  if (v_pppp_bytes) *v_pppp_bytes = h->nt ? h->ladder_bytes_tc : h->ladder_bytes;
  if (ladder_flops) *ladder_flops = h->ladder_flops;
  return CCDGPU_OK;
}

}  // extern "C"
