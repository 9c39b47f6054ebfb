// C-ABI layer of libb2fil.so: error convention, forest lifetime, prediction entry points.
// Declarations and the reference interfaces they replace are in include/b2fil.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "forest.hpp"
#include "host_pool.hpp"
#include "kernels.hpp"
#include "kernels_q.hpp"

using namespace b2fil;

namespace {

thread_local std::string g_last_error;
std::atomic<int64_t> g_launches{0};

int set_error(int code, const std::string& msg)
{
  g_last_error = msg;
  return code;
}
int cuda_error(const char* what, cudaError_t e)
{
  return set_error(B2FIL_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define B2FIL_CUDA(call)                                  \
  do {                                                    \
    const cudaError_t e_ = (call);                        \
    if (e_ != cudaSuccess) return cuda_error(#call, e_);  \
  } while (0)

// Makes a device current for the lifetime of the guard and restores the previous one.
struct DeviceGuard {
  int prev = -1;
  bool ok  = false;
  explicit DeviceGuard(int dev)
  {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    ok = cudaSetDevice(dev) == cudaSuccess;
  }
  ~DeviceGuard()
  {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// Peer access is a per-process setting of a device pair.  It is switched on the first time a pair
// is used (forest replication, output gather) and remembered: 1 = `dev` maps `peer`'s memory
// directly (copies between them do not pass through host memory), 0 = it cannot.
std::mutex g_peer_mu;
std::map<std::pair<int, int>, int> g_peer;

int enable_peer_one_way(int dev, int peer)
{
  if (dev == peer) return 1;
  std::lock_guard<std::mutex> lock(g_peer_mu);
  const auto key = std::make_pair(dev, peer);
  const auto it  = g_peer.find(key);
  if (it != g_peer.end()) return it->second;
  int can = 0;
  if (cudaDeviceCanAccessPeer(&can, dev, peer) != cudaSuccess) {
    cudaGetLastError();
    can = 0;
  }
  if (can) {
    DeviceGuard guard(dev);
    const cudaError_t e = cudaDeviceEnablePeerAccess(peer, 0);
    if (e == cudaErrorPeerAccessAlreadyEnabled) {
      cudaGetLastError();  // somebody else in the process (e.g. the array library) did it already
    } else if (e != cudaSuccess) {
      cudaGetLastError();
      can = 0;
    }
  }
  g_peer[key] = can;
  return can;
}

// Both directions: a peer copy is direct when either side can issue it, the library enables both.
int enable_peer_pair(int a, int b)
{
  const int ab = enable_peer_one_way(a, b);
  const int ba = enable_peer_one_way(b, a);
  return (ab && ba) ? 1 : 0;
}

// Device times of the calling thread's last b2fil_predict_sharded call.
struct ShardTiming {
  double compute_ms = 0, gather_ms = 0, wall_ms = 0;
  int direct = 0, valid = 0;
};
thread_local ShardTiming g_shard_timing;

// Pipeline shape of b2fil_predict_host (tuning aids B2FIL_HOST_BLOCK_MB / B2FIL_HOST_SLOTS /
// B2FIL_HOST_STAGED_BLOCK_MB / B2FIL_HOST_COPY_THREADS, read from the environment once).
constexpr int kMaxHostSlots = 4;
struct HostPipeCfg {
  // rows predicted by one launch: pinned arrays, and pageable arrays, which are staged
  size_t block_bytes        = size_t(256) << 20;
  size_t staged_block_bytes = size_t(64) << 20;
  int slots                 = 4;  // such blocks in flight
  int copy_threads          = 0;
  HostPipeCfg()
  {
    const unsigned hw = std::thread::hardware_concurrency();
    copy_threads      = static_cast<int>(std::max(1u, std::min(6u, hw / 2)));
    auto number = [](const char* name, long lo, long hi, auto set) {
      const char* e = getenv(name);
      if (!e) return;
      const long v = atol(e);
      if (v >= lo && v <= hi) set(v);
    };
    number("B2FIL_HOST_COPY_THREADS", 1, 64, [&](long v) { copy_threads = static_cast<int>(v); });
    number("B2FIL_HOST_STAGED_BLOCK_MB", 1, 1024,
           [&](long v) { staged_block_bytes = static_cast<size_t>(v) << 20; });
    number("B2FIL_HOST_BLOCK_MB", 1, 4096, [&](long v) { block_bytes = static_cast<size_t>(v) << 20; });
    number("B2FIL_HOST_SLOTS", 1, kMaxHostSlots, [&](long v) { slots = static_cast<int>(v); });
  }
};
const HostPipeCfg& host_pipe_cfg()
{
  static const HostPipeCfg cfg;
  return cfg;
}

}  // namespace

namespace {
// Scratch of predictions comes from one stream-ordered memory pool per device, shared by the
// forests on it: creating and first growing a pool costs milliseconds, which every newly loaded
// model would otherwise pay.  It keeps what was freed for the next call (a pool of its own leaves
// the settings of the device's default pool alone) and is destroyed with the last forest.
// What a freed forest needed beyond the others' largest prediction goes back to the device.
struct ScratchPool {
  cudaMemPool_t pool = nullptr;
  std::vector<const std::atomic<int64_t>*> users;  // most scratch that a prediction of each has taken
};
std::mutex g_pool_mu;
std::map<int, ScratchPool> g_pools;

cudaError_t acquire_scratch_pool(int device, const std::atomic<int64_t>* peak, cudaMemPool_t* out)
{
  std::lock_guard<std::mutex> lock(g_pool_mu);
  ScratchPool& s = g_pools[device];
  if (!s.pool) {
    cudaMemPoolProps props{};
    props.allocType     = cudaMemAllocationTypePinned;
    props.handleTypes   = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id   = device;
    cudaError_t e       = cudaMemPoolCreate(&s.pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = ~uint64_t(0);
    e = cudaMemPoolSetAttribute(s.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(s.pool);
      s.pool = nullptr;
      return e;
    }
  }
  s.users.push_back(peak);
  *out = s.pool;
  return cudaSuccess;
}
void release_scratch_pool(int device, const std::atomic<int64_t>* peak)
{
  std::lock_guard<std::mutex> lock(g_pool_mu);
  ScratchPool& s = g_pools[device];
  s.users.erase(std::remove(s.users.begin(), s.users.end(), peak), s.users.end());
  if (s.users.empty()) {
    cudaMemPoolDestroy(s.pool);
    s.pool = nullptr;
    return;
  }
  // (up to 64 MiB are not worth the milliseconds of taking them again)
  int64_t most = int64_t(64) << 20;
  for (const auto* u : s.users) most = std::max(most, u->load());
  cudaMemPoolTrimTo(s.pool, static_cast<size_t>(most));
}

// Pinned host memory through which predictions on host arrays pass.  It belongs to the process, and a
// call takes what it needs and gives it back when its work is done: pinning takes a millisecond and
// more, which the first call of every model paid when each had its own.  Kept for later calls: 64 MiB,
// or more if that much was in use at one time; every forest that is freed brings it back to 64 MiB, the
// last one to nothing.  Sizes are rounded up, so that batches that grow a little find their buffer.
struct PinnedBuf {
  void* ptr    = nullptr;
  size_t bytes = 0;
};
class PinnedPool {
 public:
  static PinnedPool& get()
  {
    static PinnedPool* pool = new PinnedPool;
    return *pool;
  }
  // A buffer of at least `bytes`, in place of the one in `b`.
  cudaError_t take(size_t bytes, PinnedBuf& b)
  {
    if (b.bytes >= bytes) return cudaSuccess;
    give(b);
    {
      std::lock_guard<std::mutex> lock(mu_);
      size_t best = free_.size();
      for (size_t i = 0; i < free_.size(); ++i)
        if (free_[i].bytes >= bytes && (best == free_.size() || free_[i].bytes < free_[best].bytes)) best = i;
      if (best < free_.size()) {
        b            = free_[best];
        free_[best]  = free_.back();
        free_.pop_back();
        kept_ -= b.bytes;
        used_ += b.bytes;
        most_used_ = std::max(most_used_, used_);
        return cudaSuccess;
      }
    }
    const size_t size   = pinned_size(bytes);
    void* ptr           = nullptr;
    const cudaError_t e = cudaHostAlloc(&ptr, size, cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) return e;
    b = PinnedBuf{ptr, size};
    std::lock_guard<std::mutex> lock(mu_);
    used_ += size;
    most_used_ = std::max(most_used_, used_);
    return cudaSuccess;
  }
  // Nothing on the GPU uses the buffer any more.
  void give(PinnedBuf& b)
  {
    if (!b.ptr) return;
    {
      std::lock_guard<std::mutex> lock(mu_);
      used_ -= b.bytes;
      if (users_ > 0 && kept_ + b.bytes <= std::max(kKeep, most_used_)) {
        free_.push_back(b);
        kept_ += b.bytes;
        b = PinnedBuf{};
      }
    }
    if (b.ptr) cudaFreeHost(b.ptr);
    b = PinnedBuf{};
  }
  void add_user()
  {
    std::lock_guard<std::mutex> lock(mu_);
    ++users_;
  }
  void drop_user()
  {
    std::vector<PinnedBuf> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      --users_;
      most_used_         = used_;
      const size_t limit = users_ > 0 ? kKeep : 0;
      // the largest first: what is left serves most calls
      std::sort(free_.begin(), free_.end(), [](const PinnedBuf& x, const PinnedBuf& y) { return x.bytes < y.bytes; });
      while (kept_ > limit && !free_.empty()) {
        kept_ -= free_.back().bytes;
        gone.push_back(free_.back());
        free_.pop_back();
      }
    }
    for (PinnedBuf& b : gone) cudaFreeHost(b.ptr);
  }

 private:
  static constexpr size_t kKeep = size_t(64) << 20;
  std::mutex mu_;
  std::vector<PinnedBuf> free_;
  size_t kept_ = 0, used_ = 0, most_used_ = 0;
  int users_ = 0;
};

// Status words live in pinned host memory, so that the host reads one without a copy (12 us per
// call).  A page of them serves a thousand forests; pages are kept.
std::mutex g_status_mu;
std::vector<int32_t*> g_status_free;
cudaError_t acquire_status_word(int32_t** out)
{
  std::lock_guard<std::mutex> lock(g_status_mu);
  if (g_status_free.empty()) {
    void* page          = nullptr;
    const size_t bytes  = 4096;
    const cudaError_t e = cudaHostAlloc(&page, bytes, cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) return e;
    for (size_t i = bytes / 4; i-- > 0;) g_status_free.push_back(static_cast<int32_t*>(page) + i);
  }
  *out = g_status_free.back();
  g_status_free.pop_back();
  **out = 0;
  return cudaSuccess;
}
void release_status_word(int32_t* word)
{
  std::lock_guard<std::mutex> lock(g_status_mu);
  g_status_free.push_back(word);
}
}  // namespace

// One slot of the host-buffer pipeline: device staging buffers and the stream that orders them.
struct HostSlot {
  cudaStream_t stream = nullptr;
  void* x             = nullptr;  // rows and results on the device, from the scratch pool
  void* out           = nullptr;
  size_t x_bytes      = 0;
  size_t out_bytes    = 0;
  // sharded prediction: results on their way to the first device (memory of its own, which peers may
  // read), and the events begin, kernels done, gathered
  void* shard_out        = nullptr;
  size_t shard_out_bytes = 0;
  cudaEvent_t ev[3]      = {nullptr, nullptr, nullptr};
};

constexpr int kStageChunks = 4;  // pieces of pinned memory through which pageable inputs pass

struct b2fil_forest {
  ForestView view{};
  int32_t precision = B2FIL_F32, storage = 0, layout = 0, align_bytes = 0, node_bytes = 0;
  int32_t device = 0, sm_count = 0, default_chunk = 0;
  int64_t n_nodes_in = 0, n_nodes_packed = 0, device_bytes = 0;
  int32_t* status = nullptr;     // pinned host word that kernels set when a bounded wait runs out
  cudaMemPool_t pool = nullptr;  // the device's scratch pool (shared, see acquire_scratch_pool)
  mutable std::atomic<int64_t> scratch_peak{0};  // most scratch one prediction took from it
  void* arena = nullptr;         // device memory of all blocks
  size_t arena_bytes = 0;
  std::vector<uint32_t> q_top;   // host copy of the three top nodes per tree (may be empty)
  struct Block {
    size_t at;           // offset in the arena
    size_t view_offset;  // offset of the pointer member inside ForestView
  };
  void place_blocks()
  {
    for (const Block& b : blocks) {
      void* d = static_cast<char*>(arena) + b.at;
      std::memcpy(reinterpret_cast<char*>(&view) + b.view_offset, &d, sizeof(void*));
    }
  }
  std::vector<Block> blocks;
  int32_t clone_src_device = -1;  // device this forest was replicated from, or -1
  int32_t clone_direct     = -1;  // 1: that replication went over a direct peer path
  std::mutex host_mu;  // serialises the calls that use the slots below
  HostSlot slots[kMaxHostSlots];
  cudaEvent_t chunk_free[kStageChunks] = {};  // the last copy from that piece of pinned memory is done
  ~b2fil_forest()
  {
    DeviceGuard g(device);
    for (auto& s : slots) {
      if (s.x) cudaFreeAsync(s.x, s.stream);
      if (s.out) cudaFreeAsync(s.out, s.stream);
      if (s.shard_out) cudaFree(s.shard_out);
      if (s.stream) {
        cudaStreamSynchronize(s.stream);
        cudaStreamDestroy(s.stream);
      }
      for (auto& e : s.ev)
        if (e) cudaEventDestroy(e);
    }
    for (auto& e : chunk_free)
      if (e) cudaEventDestroy(e);
    if (arena) cudaFree(arena);
    if (status) release_status_word(status);
    if (pool) {
      release_scratch_pool(device, &scratch_peak);
      PinnedPool::get().drop_user();
    }
  }
};

namespace {

// Device memory of a forest: its arrays, one after the other in a single allocation (fifteen
// allocations and frees of their own took most of the time of loading a small model).
struct Upload {
  const void* data;
  size_t bytes, view_offset;
};
template <typename V>
void add_upload(std::vector<Upload>& list, const V& host, size_t view_offset)
{
  if (!host.empty())
    list.push_back({host.data(), host.size() * sizeof(typename V::value_type), view_offset});
}

int allocate_arena(b2fil_forest* f, size_t bytes)
{
  const cudaError_t e = cudaMalloc(&f->arena, std::max<size_t>(bytes, 256));
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return set_error(B2FIL_ERR_NO_MEMORY, "device allocation of " + std::to_string(bytes) +
                                            " bytes for the forest failed");
  }
  if (e != cudaSuccess) return cuda_error("cudaMalloc", e);
  f->arena_bytes = bytes;
  return B2FIL_OK;
}

int upload_all(b2fil_forest* f, const std::vector<Upload>& list)
{
  size_t total = 0;
  for (const Upload& u : list) {
    f->blocks.push_back({total, u.view_offset});
    f->device_bytes += static_cast<int64_t>(u.bytes);
    total += (u.bytes + 255) / 256 * 256;
  }
  const int rc = allocate_arena(f, total);
  if (rc != B2FIL_OK) return rc;
  for (size_t i = 0; i < list.size(); ++i)
    B2FIL_CUDA(cudaMemcpy(static_cast<char*>(f->arena) + f->blocks[i].at, list[i].data,
                          list[i].bytes, cudaMemcpyHostToDevice));
  f->place_blocks();
  return B2FIL_OK;
}

int init_device_state(b2fil_forest* f)
{
  int sms = 0;
  B2FIL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, f->device));
  f->sm_count = sms;
  B2FIL_CUDA(acquire_status_word(&f->status));
  B2FIL_CUDA(acquire_scratch_pool(f->device, &f->scratch_peak, &f->pool));
  PinnedPool::get().add_user();
  return B2FIL_OK;
}

size_t elem_bytes(const b2fil_forest* f) { return f->precision == B2FIL_F32 ? 4 : 8; }

int64_t out_elems(const b2fil_forest* f, int kind)
{
  switch (kind) {
    case B2FIL_INFER_DEFAULT: return f->view.n_outputs;
    case B2FIL_INFER_PER_TREE:
      return static_cast<int64_t>(f->view.n_trees) *
             (f->view.leaf_vector_len > 1 ? f->view.n_outputs : 1);
    case B2FIL_INFER_LEAF_ID: return f->view.n_trees;
    case B2FIL_INFER_CLASS: return 1;
    case B2FIL_INFER_PROBA2: return 2;
    default: return 0;
  }
}
size_t out_elem_bytes(const b2fil_forest* f, int kind)
{
  if (kind == B2FIL_INFER_LEAF_ID || kind == B2FIL_INFER_CLASS) return 4;
  return elem_bytes(f);
}

int check_predict_args(const b2fil_forest* f, int kind, const void* X, int64_t n_rows,
                       int64_t row_stride, const void* out)
{
  if (!f) return set_error(B2FIL_ERR_INVALID_ARG, "forest is NULL");
  if (out_elems(f, kind) == 0) return set_error(B2FIL_ERR_INVALID_ARG, "unknown infer_kind");
  if (n_rows < 0) return set_error(B2FIL_ERR_INVALID_ARG, "n_rows is negative");
  if (n_rows > 0 && (!X || !out)) return set_error(B2FIL_ERR_INVALID_ARG, "NULL buffer");
  if (row_stride < f->view.n_features)
    return set_error(B2FIL_ERR_INVALID_ARG, "row_stride is smaller than n_features");
  if (kind == B2FIL_INFER_PROBA2 && f->view.n_outputs != 1)
    return set_error(B2FIL_ERR_INVALID_ARG, "B2FIL_INFER_PROBA2 needs a forest with one output");
  return B2FIL_OK;
}

int enqueue(const b2fil_forest* f, int kind, const void* X, int64_t n_rows, int64_t row_stride,
            void* out, int chunk_size, double threshold, cudaStream_t stream)
{
  PredictParams p{};
  p.f          = f->view;
  p.X          = X;
  p.n_rows     = n_rows;
  p.row_stride = row_stride;
  p.out        = out;
  p.kind       = kind;
  p.threshold  = threshold;
  p.status     = f->status;
  p.q_top      = f->q_top.empty() ? nullptr : f->q_top.data();
  std::string err;
  int64_t n = 0;
  const Scratch scratch{f->pool, &f->scratch_peak};
  const int rc = launch_predict(p, chunk_size > 0 ? chunk_size : f->default_chunk, f->sm_count,
                                stream, &scratch, err, &n);
  g_launches += n;
  if (rc != B2FIL_OK) return set_error(rc, err);
  return B2FIL_OK;
}

// Make a slot's device buffer hold `want` bytes.  Stream-ordered: batches that grow do not stall the
// device, and grow the buffer by half at least.
int grow_buffer(const b2fil_forest* f, HostSlot& s, void** buf, size_t* have, size_t want)
{
  if (*have >= want) return B2FIL_OK;
  size_t size = std::max(want, *have + *have / 2);
  if (*buf) B2FIL_CUDA(cudaFreeAsync(*buf, s.stream));
  *buf          = nullptr;
  *have         = 0;
  cudaError_t e = cudaMallocFromPoolAsync(buf, size, f->pool, s.stream);
  if (e == cudaErrorMemoryAllocation && size > want) {
    cudaGetLastError();
    size = want;
    e    = cudaMallocFromPoolAsync(buf, size, f->pool, s.stream);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *buf = nullptr;
    return set_error(e == cudaErrorMemoryAllocation ? B2FIL_ERR_NO_MEMORY : B2FIL_ERR_CUDA,
                     std::string("device staging buffer: ") + cudaGetErrorString(e));
  }
  *have = size;
  return B2FIL_OK;
}
int ensure_stream(HostSlot& s)
{
  if (!s.stream) B2FIL_CUDA(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
  return B2FIL_OK;
}
int ensure_slot(const b2fil_forest* f, HostSlot& s, size_t x_bytes, size_t out_bytes)
{
  int rc = ensure_stream(s);
  if (rc == B2FIL_OK) rc = grow_buffer(f, s, &s.x, &s.x_bytes, x_bytes);
  if (rc == B2FIL_OK) rc = grow_buffer(f, s, &s.out, &s.out_bytes, out_bytes);
  return rc;
}

// Read and clear the status word.  The caller has already waited for the work it cares about.
int read_status_word(const b2fil_forest* f, int32_t* status)
{
  volatile int32_t* word = f->status;
  *status                = *word;
  if (*status != 0) {
    *word = 0;  // reported once: the next prediction starts from a clean word
    static const char* const where[] = {"", "tree ring (producer)", "tree ring (consumer)",
                                        "row-tile buffer", "rank tables", "self test"};
    const char* w = (*status >= 1 && *status <= 5) ? where[*status] : "unknown";
    return set_error(B2FIL_ERR_TIMEOUT, std::string("a bounded wait inside a kernel ran out: ") +
                                          w + " (status " + std::to_string(*status) + ")");
  }
  return B2FIL_OK;
}

// True when the CUDA runtime does not know the host pointer: ordinary (pageable) memory.  Copies
// from such memory are staged by the driver through a small internal buffer and run at a
// fraction of the link; the library stages them itself instead.
// `mapped`: the address kernels reach it at, or null.
bool is_pageable(const void* p, void** mapped)
{
  cudaPointerAttributes a{};
  *mapped = nullptr;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  if (a.type == cudaMemoryTypeHost) *mapped = a.devicePointer;
  return a.type == cudaMemoryTypeUnregistered;
}

int ensure_pinned(PinnedBuf& b, size_t want)
{
  const cudaError_t e = PinnedPool::get().take(want, b);
  if (e == cudaSuccess) return B2FIL_OK;
  cudaGetLastError();
  return set_error(B2FIL_ERR_NO_MEMORY, std::string("pinned staging buffer: ") + cudaGetErrorString(e));
}

// Copy `n_rows` rows of `row_bytes` bytes (source rows `src_stride` bytes apart) into a dense
// buffer, in pieces that the copy threads share.
void copy_rows(char* dst, const char* src, int64_t n_rows, size_t row_bytes, size_t src_stride)
{
  const size_t total  = static_cast<size_t>(n_rows) * row_bytes;
  const size_t piece  = std::min(size_t(128) << 10, std::max(size_t(16) << 10, total / 16));
  const int64_t step  = std::max<int64_t>(1, static_cast<int64_t>(piece / std::max<size_t>(1, row_bytes)));
  const size_t pieces = static_cast<size_t>((n_rows + step - 1) / step);
  CopyPool::get(host_pipe_cfg().copy_threads).run(pieces, [&](size_t i) {
    const int64_t b = static_cast<int64_t>(i) * step, e = std::min(n_rows, b + step);
    if (src_stride == row_bytes) {
      std::memcpy(dst + static_cast<size_t>(b) * row_bytes, src + static_cast<size_t>(b) * src_stride,
                  static_cast<size_t>(e - b) * row_bytes);
    } else {
      for (int64_t r = b; r < e; ++r)
        std::memcpy(dst + static_cast<size_t>(r) * row_bytes, src + static_cast<size_t>(r) * src_stride,
                    row_bytes);
    }
  });
}

// Host-array prediction, in one of three ways by the size of the input:
//  in_place (up to 16 KiB): the kernel reads its rows over the link and writes its results back over
//    it; pinned host memory is mapped, and no copy starts as fast as that.
//  short_call (up to 16 MiB): a kernel fetches the rows from pinned memory, piece by piece while the
//    copy threads fill the next one.  Between kernels of a stream there is about a microsecond; a
//    copy-engine transfer costs 5 us to start and again to hand over (1,000 rows of 50 features:
//    46 -> 30 us).
//  blocks: row blocks are copied to the device, predicted and copied back on a few streams, so that
//    the copies of one block overlap the kernels of another; about eight blocks per call keep the
//    last block's kernels, which nothing overlaps, short.  Pinned inputs are copied from where they
//    are.  Pageable ones pass through four pinned chunks of at most 4 MiB: the copy threads fill one
//    (they stay in the host's cache, 100 GB/s) while another is on the link (large enough for 52 of
//    its 55 GB/s); the driver's own staging of pageable memory reaches 12 to 19 GB/s.
// The caller holds the forest's host mutex and has made its device current.
class HostPrediction {
 public:
  HostPrediction(b2fil_forest* f, int kind, const void* X, int64_t n_rows, int64_t row_stride,
                 void* out, int chunk_size, double threshold)
      : f_(f), kind_(kind), x_(static_cast<const char*>(X)), out_(static_cast<char*>(out)),
        n_rows_(n_rows), chunk_size_(chunk_size), threshold_(threshold)
  {
    in_row_b_   = static_cast<size_t>(f->view.n_features) * elem_bytes(f);
    in_stride_  = static_cast<size_t>(row_stride) * elem_bytes(f);
    out_row_b_  = static_cast<size_t>(out_elems(f, kind)) * out_elem_bytes(f, kind);
    in_bytes_   = static_cast<size_t>(n_rows) * in_row_b_;
    out_bytes_  = static_cast<size_t>(n_rows) * out_row_b_;
    in_pinned_  = !is_pageable(X, &in_mapped_);
    out_pinned_ = !is_pageable(out, &out_mapped_);
  }
  HostPrediction(const HostPrediction&) = delete;
  ~HostPrediction()
  {
    // also after an error: work already enqueued still uses the caller's arrays and the staging
    if (!drained_)
      for (HostSlot& s : f_->slots)
        if (s.stream) cudaStreamSynchronize(s.stream);
    for (PinnedBuf& b : chunk_) PinnedPool::get().give(b);
    for (Result& r : result_) PinnedPool::get().give(r.pinned);
  }

  int run()
  {
    int rc;
    if (in_bytes_ <= kInPlaceIn && out_bytes_ <= (per_tree() ? kPerTreeOut : kInPlaceOut)) {
      rc = in_place();
    } else if (in_bytes_ <= kShortIn && out_bytes_ <= kShortIn) {
      rc = short_call();
    } else {
      rc = blocks();
    }
    for (int i = 0; i < kMaxHostSlots && rc == B2FIL_OK; ++i) rc = flush(i);
    if (rc != B2FIL_OK) return rc;
    drained_       = true;
    int32_t status = 0;
    return read_status_word(f_, &status);
  }

 private:
  static constexpr size_t kInPlaceIn  = size_t(16) << 10;
  static constexpr size_t kInPlaceOut = size_t(64) << 10;
  static constexpr size_t kShortIn    = size_t(16) << 20;
  static constexpr size_t kShortOut   = size_t(256) << 10;  // results that the kernel writes to the host itself
  static constexpr size_t kPerTreeOut = size_t(2) << 10;
  static constexpr size_t kChunkMax   = size_t(4) << 20;
  bool per_tree() const { return kind_ == B2FIL_INFER_LEAF_ID || kind_ == B2FIL_INFER_PER_TREE; }

  int in_place()
  {
    HostSlot& s  = f_->slots[0];
    PinnedBuf& c = chunk_[0];
    Result& r    = result_[0];
    int rc       = ensure_stream(s);
    if (rc == B2FIL_OK) rc = ensure_pinned(c, kInPlaceIn);
    if (rc == B2FIL_OK) rc = ensure_pinned(r.pinned, kInPlaceOut);
    if (rc != B2FIL_OK) return rc;
    copy_rows(static_cast<char*>(c.ptr), x_, n_rows_, in_row_b_, in_stride_);
    rc = enqueue(f_, kind_, c.ptr, n_rows_, f_->view.n_features, r.pinned.ptr, chunk_size_, threshold_,
                 s.stream);
    r.row0 = 0;
    r.rows = n_rows_;
    return rc;
  }

  int short_call()
  {
    HostSlot& s       = f_->slots[0];
    PinnedBuf& c      = chunk_[0];
    Result& r         = result_[0];
    const bool direct = in_mapped_ != nullptr && in_stride_ == in_row_b_ &&
                        reinterpret_cast<uintptr_t>(in_mapped_) % 16 == 0;
    // results without a copy: consecutive ones, not a store of its own per row and tree
    const bool write  = out_bytes_ <= (per_tree() ? kPerTreeOut : kShortOut);
    int rc            = ensure_slot(f_, s, in_bytes_, write ? 0 : out_bytes_);
    if (rc == B2FIL_OK && !direct) rc = ensure_pinned(c, in_bytes_);
    const bool to_pin = write ? out_mapped_ == nullptr : !out_pinned_;
    if (rc == B2FIL_OK && to_pin) rc = ensure_pinned(r.pinned, out_bytes_);
    if (rc != B2FIL_OK) return rc;
    std::string err;
    if (direct) {
      rc = launch_fetch(s.x, in_mapped_, in_bytes_, f_->sm_count, s.stream, err);
    } else {
      rc = stage_and_fetch(static_cast<char*>(c.ptr), static_cast<char*>(s.x), s.stream, err);
    }
    if (rc != B2FIL_OK) return set_error(rc, err);
    void* to = to_pin ? r.pinned.ptr : (write ? out_mapped_ : static_cast<void*>(out_));
    rc = enqueue(f_, kind_, s.x, n_rows_, f_->view.n_features, write ? to : s.out, chunk_size_,
                 threshold_, s.stream);
    if (rc != B2FIL_OK) return rc;
    if (!write) B2FIL_CUDA(cudaMemcpyAsync(to, s.out, out_bytes_, cudaMemcpyDeviceToHost, s.stream));
    r.row0 = 0;
    r.rows = to_pin ? n_rows_ : 0;
    return B2FIL_OK;
  }

  // All rows to pinned memory and, part by part as the copy threads get on, to the device.
  int stage_and_fetch(char* pinned, char* device, cudaStream_t stream, std::string& err)
  {
    // items of whole rows, and parts of whole items, that start on 16-byte boundaries
    const int64_t unit  = in_row_b_ % 16 == 0 ? 1 : 4;
    auto rows_of = [&](size_t bytes) {
      return std::max(unit, static_cast<int64_t>(bytes / in_row_b_) / unit * unit);
    };
    const int64_t item_rows = rows_of(std::min(size_t(64) << 10, std::max(size_t(16) << 10, in_bytes_ / 32)));
    const size_t n_items    = static_cast<size_t>((n_rows_ + item_rows - 1) / item_rows);
    // Few parts, each twice the one before: every transfer kernel adds the link's latency, and the
    // copy threads are faster than the link, so a larger part is ready when a smaller one is over.
    constexpr size_t kMost = 4;
    size_t part_end[kMost], n_parts = 0;
    for (size_t end = 0, size = std::max(size_t(256) << 10, in_bytes_ / 7); end < n_items; size *= 2) {
      end += std::max<size_t>(1, static_cast<size_t>(rows_of(size) / item_rows));
      if (n_parts == kMost - 1 || end + end / 2 > n_items) end = n_items;
      part_end[n_parts++] = end;
    }
    std::atomic<size_t> done[kMost] = {};
    size_t sent = 0;
    int rc      = B2FIL_OK;
    auto copy = [&](size_t i) {
      const int64_t b = static_cast<int64_t>(i) * item_rows, e = std::min(n_rows_, b + item_rows);
      if (in_stride_ == in_row_b_) {
        std::memcpy(pinned + static_cast<size_t>(b) * in_row_b_, x_ + static_cast<size_t>(b) * in_row_b_,
                    static_cast<size_t>(e - b) * in_row_b_);
      } else {
        for (int64_t r = b; r < e; ++r)
          std::memcpy(pinned + static_cast<size_t>(r) * in_row_b_,
                      x_ + static_cast<size_t>(r) * in_stride_, in_row_b_);
      }
      size_t part = 0;
      while (i >= part_end[part]) ++part;
      done[part].fetch_add(1);
    };
    auto send = [&] {
      for (; sent < n_parts; ++sent) {
        const size_t first = sent > 0 ? part_end[sent - 1] : 0, last = part_end[sent];
        if (done[sent].load() < last - first) return false;
        const size_t at  = first * static_cast<size_t>(item_rows) * in_row_b_;
        const size_t end = std::min(in_bytes_, last * static_cast<size_t>(item_rows) * in_row_b_);
        if (rc == B2FIL_OK)
          rc = launch_fetch(device + at, pinned + at, end - at, f_->sm_count, stream, err);
      }
      return true;
    };
    CopyPool::get(host_pipe_cfg().copy_threads).run(n_items, copy, send);
    return rc;
  }

  int blocks()
  {
    const HostPipeCfg& pipe = host_pipe_cfg();
    const size_t row_b      = std::max(in_row_b_, out_row_b_);
    const size_t most       = in_pinned_ ? pipe.block_bytes : pipe.staged_block_bytes;
    const size_t want       = std::max<size_t>(static_cast<size_t>(n_rows_) * row_b / 8, size_t(8) << 20);
    int64_t block_rows      = static_cast<int64_t>(std::max<size_t>(1, std::min(most, want) / row_b));
    block_rows              = std::max<int64_t>(block_rows / 256 * 256, 256);
    block_rows              = std::min(block_rows, n_rows_);
    const int n_slots       = static_cast<int>(std::min<int64_t>(pipe.slots, (n_rows_ + block_rows - 1) / block_rows));
    for (int i = 0; i < n_slots; ++i) {
      int rc = ensure_slot(f_, f_->slots[i], static_cast<size_t>(block_rows) * in_row_b_,
                           static_cast<size_t>(block_rows) * out_row_b_);
      if (rc == B2FIL_OK && !out_pinned_)
        rc = ensure_pinned(result_[i].pinned, static_cast<size_t>(block_rows) * out_row_b_);
      if (rc != B2FIL_OK) return rc;
    }
    int which = 0;
    for (int64_t r0 = 0; r0 < n_rows_; r0 += block_rows, which = (which + 1) % n_slots) {
      HostSlot& s     = f_->slots[which];
      Result& r       = result_[which];
      const int64_t n = std::min(block_rows, n_rows_ - r0);
      // stream order makes the slot's previous block finish before its device buffers are reused
      int rc = flush(which);
      if (rc == B2FIL_OK) rc = in_pinned_ ? send(s, r0, n) : send_staged(s, r0, n);
      if (rc == B2FIL_OK)
        rc = enqueue(f_, kind_, s.x, n, f_->view.n_features, s.out, chunk_size_, threshold_, s.stream);
      if (rc != B2FIL_OK) return rc;
      void* to = out_pinned_ ? out_ + static_cast<size_t>(r0) * out_row_b_ : static_cast<char*>(r.pinned.ptr);
      B2FIL_CUDA(cudaMemcpyAsync(to, s.out, static_cast<size_t>(n) * out_row_b_,
                                 cudaMemcpyDeviceToHost, s.stream));
      r.row0 = r0;
      r.rows = out_pinned_ ? 0 : n;
    }
    return B2FIL_OK;
  }

  // Rows [r0, r0 + n) of a pinned array to the slot's device buffer.
  int send(HostSlot& s, int64_t r0, int64_t n)
  {
    const char* from = x_ + static_cast<size_t>(r0) * in_stride_;
    if (in_stride_ == in_row_b_) {
      B2FIL_CUDA(cudaMemcpyAsync(s.x, from, static_cast<size_t>(n) * in_row_b_,
                                 cudaMemcpyHostToDevice, s.stream));
    } else {
      B2FIL_CUDA(cudaMemcpy2DAsync(s.x, in_row_b_, from, in_stride_, in_row_b_,
                                   static_cast<size_t>(n), cudaMemcpyHostToDevice, s.stream));
    }
    return B2FIL_OK;
  }
  // The same through pinned chunks.
  int send_staged(HostSlot& s, int64_t r0, int64_t n)
  {
    for (int64_t b = 0, m; b < n; b += m) {
      // the first chunks of a call are smaller: the link waits for the first one to be filled
      const size_t size = std::min(kChunkMax, next_size_);
      next_size_        = size * 2;
      m = std::min(std::max<int64_t>(1, static_cast<int64_t>(size / in_row_b_)), n - b);
      const size_t bytes = static_cast<size_t>(m) * in_row_b_;
      PinnedBuf& c       = chunk_[next_chunk_];
      cudaEvent_t& free  = f_->chunk_free[next_chunk_];
      next_chunk_        = (next_chunk_ + 1) % kStageChunks;
      if (!free) B2FIL_CUDA(cudaEventCreateWithFlags(&free, cudaEventDisableTiming));
      B2FIL_CUDA(cudaEventSynchronize(free));  // its last copy, in this call or one before
      const int rc = ensure_pinned(c, std::max(bytes, kChunkMax));
      if (rc != B2FIL_OK) return rc;
      copy_rows(static_cast<char*>(c.ptr), x_ + static_cast<size_t>(r0 + b) * in_stride_, m,
                in_row_b_, in_stride_);
      B2FIL_CUDA(cudaMemcpyAsync(static_cast<char*>(s.x) + static_cast<size_t>(b) * in_row_b_, c.ptr,
                                 bytes, cudaMemcpyHostToDevice, s.stream));
      B2FIL_CUDA(cudaEventRecord(free, s.stream));
    }
    return B2FIL_OK;
  }
  // Wait for a slot and hand its results to the caller.
  int flush(int slot)
  {
    Result& r = result_[slot];
    if (r.row0 < 0) return B2FIL_OK;
    B2FIL_CUDA(cudaStreamSynchronize(f_->slots[slot].stream));
    if (r.rows > 0)
      copy_rows(out_ + static_cast<size_t>(r.row0) * out_row_b_, static_cast<const char*>(r.pinned.ptr),
                r.rows, out_row_b_, out_row_b_);
    r.row0 = -1;
    return B2FIL_OK;
  }

  // Results of a slot's block that are still on their way to the caller; those for pageable arrays pass
  // through pinned memory.
  struct Result {
    PinnedBuf pinned;
    int64_t row0 = -1, rows = 0;
  };

  b2fil_forest* f_;
  int kind_;
  const char* x_;
  char* out_;
  int64_t n_rows_;
  int chunk_size_;
  double threshold_;
  size_t in_row_b_, in_stride_, out_row_b_, in_bytes_, out_bytes_;
  bool in_pinned_, out_pinned_;
  void *in_mapped_ = nullptr, *out_mapped_ = nullptr;
  PinnedBuf chunk_[kStageChunks];
  Result result_[kMaxHostSlots];
  bool drained_   = false;
  int next_chunk_ = 0;
  size_t next_size_ = size_t(1) << 20;  // bytes of the next staged chunk
};

}  // namespace

extern "C" {

const char* b2fil_last_error(void) { return g_last_error.c_str(); }

int b2fil_version(void) { return 100; }

int64_t b2fil_kernel_launches(void) { return g_launches.load(); }

int b2fil_forest_create(const b2fil_forest_desc* desc, const b2fil_create_opts* opts,
                        b2fil_forest** out)
{
  if (!desc || !opts || !out) return set_error(B2FIL_ERR_INVALID_ARG, "NULL argument");
  *out = nullptr;
  try {
    int n_dev = 0;
    cudaError_t e = cudaGetDeviceCount(&n_dev);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return set_error(B2FIL_ERR_CUDA, std::string("no usable CUDA device: ") +
                                         cudaGetErrorString(e));
    }
    if (opts->device_id < 0 || opts->device_id >= n_dev)
      return set_error(B2FIL_ERR_INVALID_ARG, "device_id " + std::to_string(opts->device_id) +
                                                " out of range (" + std::to_string(n_dev) +
                                                " devices)");
    PackedForest pf;
    std::string err;
    int rc = pack_forest(*desc, *opts, dense_ok, pf, err);
    if (rc != B2FIL_OK) return set_error(rc, err);

    if (pf.view.c_enabled && !build_blocks(pf)) pf.view.c_enabled = 0;
    if (pf.view.q_enabled) {
      for (auto* image : {&pf.q_nodes, &pf.q_nodes_ids, &pf.q_nodes_nan}) split_category_sets(pf.view, *image);
      walk_order(pf);
    }

    std::unique_ptr<b2fil_forest> f(new b2fil_forest());
    f->device = opts->device_id;
    DeviceGuard guard(f->device);
    if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
    f->view           = pf.view;
    f->precision      = pf.precision;
    f->storage        = pf.storage;
    f->layout         = opts->layout;
    f->align_bytes    = pf.align_bytes;
    f->node_bytes     = pf.node_bytes;
    f->n_nodes_in     = pf.n_nodes_in;
    f->n_nodes_packed = pf.n_nodes_packed;
    f->default_chunk  = std::max(0, opts->default_chunk_size);
    if ((rc = init_device_state(f.get())) != B2FIL_OK) return rc;
    std::vector<Upload> list;
    add_upload(list, pf.nodes, offsetof(ForestView, nodes));
    add_upload(list, pf.roots, offsetof(ForestView, roots));
    add_upload(list, pf.leaf_ids, offsetof(ForestView, leaf_ids));
    add_upload(list, pf.cat_pool, offsetof(ForestView, cat_pool));
    add_upload(list, pf.tree_class, offsetof(ForestView, tree_class));
    add_upload(list, pf.tree_orig, offsetof(ForestView, tree_orig));
    add_upload(list, pf.leaf_vectors, offsetof(ForestView, leaf_vectors));
    add_upload(list, pf.out_scale, offsetof(ForestView, out_scale));
    add_upload(list, pf.out_bias, offsetof(ForestView, out_bias));
    if (f->view.c_enabled) {
      add_upload(list, pf.b_blocks, offsetof(ForestView, c_blocks));
      add_upload(list, pf.b_exact, offsetof(ForestView, c_exact));
      add_upload(list, pf.b_leaf_payload, offsetof(ForestView, c_leaf_payload));
      add_upload(list, pf.b_leaf_ids, offsetof(ForestView, c_leaf_ids));
      add_upload(list, pf.b_top, offsetof(ForestView, c_top));
      add_upload(list, pf.b_top_exact, offsetof(ForestView, c_top_exact));
    }
    if (pf.view.q_enabled) {
      add_upload(list, pf.q_nodes, offsetof(ForestView, q_nodes));
      add_upload(list, pf.q_nodes_ids, offsetof(ForestView, q_nodes_ids));
      add_upload(list, pf.q_nodes_nan, offsetof(ForestView, q_nodes_nan));
      add_upload(list, pf.q_blob, offsetof(ForestView, q_blob));
      add_upload(list, pf.q_groups, offsetof(ForestView, q_groups));
      add_upload(list, pf.q_bundles, offsetof(ForestView, q_bundles));
      f->q_top = std::move(pf.q_top);
    }
    if ((rc = upload_all(f.get(), list)) != B2FIL_OK) return rc;
    *out = f.release();
    return B2FIL_OK;
  } catch (const std::bad_alloc&) {
    return set_error(B2FIL_ERR_NO_MEMORY, "host allocation failed while packing the forest");
  } catch (const std::exception& ex) {
    return set_error(B2FIL_ERR_INVALID_ARG, std::string("unexpected failure: ") + ex.what());
  }
}

int b2fil_forest_clone_to_device(const b2fil_forest* src, int device_id, b2fil_forest** out)
{
  if (!src || !out) return set_error(B2FIL_ERR_INVALID_ARG, "NULL argument");
  *out = nullptr;
  try {
    int n_dev = 0;
    B2FIL_CUDA(cudaGetDeviceCount(&n_dev));
    if (device_id < 0 || device_id >= n_dev)
      return set_error(B2FIL_ERR_INVALID_ARG, "device_id out of range");
    std::unique_ptr<b2fil_forest> f(new b2fil_forest());
    f->view           = src->view;
    f->precision      = src->precision;
    f->storage        = src->storage;
    f->layout         = src->layout;
    f->align_bytes    = src->align_bytes;
    f->node_bytes     = src->node_bytes;
    f->n_nodes_in     = src->n_nodes_in;
    f->n_nodes_packed = src->n_nodes_packed;
    f->default_chunk  = src->default_chunk;
    f->q_top          = src->q_top;
    f->device         = device_id;
    DeviceGuard guard(device_id);
    if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
    int rc;
    if ((rc = init_device_state(f.get())) != B2FIL_OK) return rc;
    f->clone_src_device = src->device;
    f->clone_direct     = enable_peer_pair(device_id, src->device);
    if ((rc = allocate_arena(f.get(), src->arena_bytes)) != B2FIL_OK) return rc;
    f->blocks       = src->blocks;
    f->device_bytes = src->device_bytes;
    // direct over the peer path when it could be enabled above, staged through the host otherwise
    B2FIL_CUDA(cudaMemcpyPeer(f->arena, device_id, src->arena, src->device, src->arena_bytes));
    f->place_blocks();
    *out = f.release();
    return B2FIL_OK;
  } catch (const std::bad_alloc&) {
    return set_error(B2FIL_ERR_NO_MEMORY, "host allocation failed");
  }
}

int b2fil_forest_free(b2fil_forest* f)
{
  delete f;
  return B2FIL_OK;
}

int b2fil_forest_info(const b2fil_forest* f, b2fil_info* info)
{
  if (!f || !info) return set_error(B2FIL_ERR_INVALID_ARG, "NULL argument");
  std::memset(info, 0, sizeof(*info));
  info->precision          = f->precision;
  info->layout             = f->layout;
  info->storage            = f->storage;
  info->device_id          = f->device;
  info->n_trees            = f->view.n_trees;
  info->n_features         = f->view.n_features;
  info->n_outputs          = f->view.n_outputs;
  info->leaf_vector_len    = f->view.leaf_vector_len;
  info->max_depth          = f->view.max_depth;
  info->dense_depth        = f->view.dense_depth;
  info->node_bytes         = f->node_bytes;
  info->has_categorical    = f->view.has_categorical;
  info->n_nodes_in         = f->n_nodes_in;
  info->n_nodes_packed     = f->n_nodes_packed;
  info->device_bytes       = f->device_bytes;
  info->default_chunk_size = f->default_chunk;
  info->row_quantization   = f->view.q_enabled;
  info->compact_image      = f->view.c_enabled;
  info->top_levels         = f->view.c_enabled ? f->view.c_top_levels : 0;
  info->peer_direct        = f->clone_direct;
  info->clone_src_device   = f->clone_src_device;
  info->scratch_pool_bytes = f->scratch_peak.load();
  return B2FIL_OK;
}

int64_t b2fil_output_elems_per_row(const b2fil_forest* f, int infer_kind)
{
  if (!f) {
    set_error(B2FIL_ERR_INVALID_ARG, "forest is NULL");
    return 0;
  }
  const int64_t n = out_elems(f, infer_kind);
  if (n == 0) set_error(B2FIL_ERR_INVALID_ARG, "unknown infer_kind");
  return n;
}


int b2fil_forest_status(const b2fil_forest* f, int32_t* status)
{
  if (!f || !status) return set_error(B2FIL_ERR_INVALID_ARG, "NULL argument");
  DeviceGuard guard(f->device);
  if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
  // every stream of the device, the non-blocking ones included: a plain copy on the default
  // stream would not wait for them
  B2FIL_CUDA(cudaDeviceSynchronize());
  return read_status_word(f, status);
}

int b2fil_forest_selftest_timeout(b2fil_forest* f, int tries, void* cuda_stream)
{
  if (!f) return set_error(B2FIL_ERR_INVALID_ARG, "forest is NULL");
  if (tries < 1 || tries > 4096)
    return set_error(B2FIL_ERR_INVALID_ARG, "tries must be between 1 and 4096");
  DeviceGuard guard(f->device);
  if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
  std::string err;
  const int rc = launch_bounded_wait_selftest(f->status, static_cast<uint32_t>(tries),
                                              static_cast<cudaStream_t>(cuda_stream), err);
  if (rc != B2FIL_OK) return set_error(rc, err);
  return B2FIL_OK;
}

int b2fil_enable_peer_access(int device_a, int device_b)
{
  int n_dev = 0;
  B2FIL_CUDA(cudaGetDeviceCount(&n_dev));
  if (device_a < 0 || device_b < 0 || device_a >= n_dev || device_b >= n_dev)
    return set_error(B2FIL_ERR_INVALID_ARG, "device ordinal out of range");
  return enable_peer_pair(device_a, device_b);
}

int b2fil_set_tuning(const char* key, int value)
{
  if (!key) return set_error(B2FIL_ERR_INVALID_ARG, "key is NULL");
  set_tuning_value(key, value);
  return B2FIL_OK;
}

int b2fil_last_variant(char* buf, size_t buf_bytes)
{
  if (!buf || buf_bytes == 0) return set_error(B2FIL_ERR_INVALID_ARG, "NULL or empty buffer");
  const std::string v = last_launch_variant();
  const size_t n      = std::min(v.size(), buf_bytes - 1);
  std::memcpy(buf, v.data(), n);
  buf[n] = 0;
  return static_cast<int>(v.size());
}

int b2fil_last_sharded_timing(double* compute_ms, double* gather_ms, double* wall_ms,
                              int* gather_direct)
{
  const ShardTiming& t = g_shard_timing;
  if (!t.valid) return set_error(B2FIL_ERR_INVALID_ARG, "no sharded prediction on this thread yet");
  if (compute_ms) *compute_ms = t.compute_ms;
  if (gather_ms) *gather_ms = t.gather_ms;
  if (wall_ms) *wall_ms = t.wall_ms;
  if (gather_direct) *gather_direct = t.direct;
  return B2FIL_OK;
}

int b2fil_predict(const b2fil_forest* f, int infer_kind, const void* X_dev, int64_t n_rows,
                  int64_t row_stride, void* out_dev, int chunk_size, double threshold,
                  void* cuda_stream)
{
  int rc = check_predict_args(f, infer_kind, X_dev, n_rows, row_stride, out_dev);
  if (rc != B2FIL_OK) return rc;
  DeviceGuard guard(f->device);
  if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
  return enqueue(f, infer_kind, X_dev, n_rows, row_stride, out_dev, chunk_size, threshold,
                 static_cast<cudaStream_t>(cuda_stream));
}

int b2fil_predict_fixed_scratch(const b2fil_forest* f, int infer_kind, const void* X_dev,
                                int64_t n_rows, int64_t row_stride, void* out_dev, int chunk_size,
                                double threshold, void* cuda_stream)
{
  int rc = check_predict_args(f, infer_kind, X_dev, n_rows, row_stride, out_dev);
  if (rc != B2FIL_OK) return rc;
  DeviceGuard guard(f->device);
  if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
  PredictParams p{};
  p.f          = f->view;
  p.X          = X_dev;
  p.n_rows     = n_rows;
  p.row_stride = row_stride;
  p.out        = out_dev;
  p.kind       = infer_kind;
  p.threshold  = threshold;
  p.status     = f->status;
  p.q_top      = f->q_top.empty() ? nullptr : f->q_top.data();
  std::string err;
  int64_t n = 0;
  rc = launch_predict_fixed_scratch(p, chunk_size > 0 ? chunk_size : f->default_chunk,
                                    f->sm_count, f->device,
                                    static_cast<cudaStream_t>(cuda_stream), err, &n);
  g_launches += n;
  if (rc != B2FIL_OK) return set_error(rc, err);
  return B2FIL_OK;
}

int b2fil_predict_host(b2fil_forest* f, int infer_kind, const void* X_host, int64_t n_rows,
                       int64_t row_stride, void* out_host, int chunk_size, double threshold)
{
  int rc = check_predict_args(f, infer_kind, X_host, n_rows, row_stride, out_host);
  if (rc != B2FIL_OK) return rc;
  if (n_rows == 0) return B2FIL_OK;
  std::lock_guard<std::mutex> lock(f->host_mu);
  DeviceGuard guard(f->device);
  if (!guard.ok) return set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
  try {
    return HostPrediction(f, infer_kind, X_host, n_rows, row_stride, out_host, chunk_size, threshold)
      .run();
  } catch (const std::exception& ex) {
    return set_error(B2FIL_ERR_NO_MEMORY, std::string("host-array prediction: ") + ex.what());
  }
}

int b2fil_predict_sharded(b2fil_forest* const* forests, int n_devices, int infer_kind,
                          const void* const* X_shards, const int64_t* shard_rows,
                          int64_t row_stride, void* out_dev0, int chunk_size, double threshold)
{
  if (!forests || !X_shards || !shard_rows || n_devices <= 0)
    return set_error(B2FIL_ERR_INVALID_ARG, "NULL argument or no devices");
  for (int i = 0; i < n_devices; ++i) {
    if (!forests[i]) return set_error(B2FIL_ERR_INVALID_ARG, "forest is NULL");
    const int rc = check_predict_args(forests[i], infer_kind, X_shards[i], shard_rows[i],
                                      row_stride, out_dev0);
    if (rc != B2FIL_OK) return rc;
  }
  for (int i = 0; i < n_devices; ++i) {
    for (int j = 0; j < i; ++j) {
      if (forests[i] == forests[j] || forests[i]->device == forests[j]->device)
        return set_error(B2FIL_ERR_INVALID_ARG, "every shard needs its own forest on its own device");
    }
  }
  b2fil_forest* f0       = forests[0];
  const size_t out_row_b = static_cast<size_t>(out_elems(f0, infer_kind)) * out_elem_bytes(f0, infer_kind);
  // every device predicts its shard on its own stream; shards of devices other than the first
  // land in a staging buffer on their device and are pushed to device 0 by a peer copy.
  // The forests' locks are taken in address order, so two callers that pass the same forests in
  // different orders cannot wait for each other.
  std::vector<b2fil_forest*> by_address(forests, forests + n_devices);
  std::sort(by_address.begin(), by_address.end(), std::less<b2fil_forest*>());
  std::vector<std::unique_lock<std::mutex>> locks;
  for (b2fil_forest* f : by_address) locks.emplace_back(f->host_mu);
  int direct = 1;
  for (int i = 1; i < n_devices; ++i)
    direct &= enable_peer_pair(forests[i]->device, f0->device);

  const auto t0  = std::chrono::steady_clock::now();
  int rc_final   = B2FIL_OK;
  int64_t row_off = 0;
  std::vector<int> fed;  // devices that have work enqueued
  for (int i = 0; i < n_devices && rc_final == B2FIL_OK; ++i) {
    b2fil_forest* f = forests[i];
    DeviceGuard guard(f->device);
    if (!guard.ok) {
      rc_final = set_error(B2FIL_ERR_CUDA, "cudaSetDevice failed");
      break;
    }
    HostSlot& s     = f->slots[0];
    const int64_t n = shard_rows[i];
    char* dst0      = static_cast<char*>(out_dev0) + static_cast<size_t>(row_off) * out_row_b;
    row_off += n;
    if (n == 0) continue;
    const bool local = f->device == f0->device;
    int rc = ensure_stream(s);
    if (const size_t want = static_cast<size_t>(n) * out_row_b; rc == B2FIL_OK && !local && s.shard_out_bytes < want) {
      if (s.shard_out) cudaFree(s.shard_out);
      s.shard_out       = nullptr;
      s.shard_out_bytes = 0;
      const cudaError_t e = cudaMalloc(&s.shard_out, want);
      if (e != cudaSuccess) {
        rc = cuda_error("cudaMalloc", e);
      } else {
        s.shard_out_bytes = want;
      }
    }
    for (auto& ev : s.ev) {
      if (rc == B2FIL_OK && !ev && cudaEventCreate(&ev) != cudaSuccess)
        rc = set_error(B2FIL_ERR_CUDA, "cudaEventCreate failed");
    }
    if (rc != B2FIL_OK) {
      rc_final = rc;
      break;
    }
    fed.push_back(i);
    cudaEventRecord(s.ev[0], s.stream);
    rc = enqueue(f, infer_kind, X_shards[i], n, row_stride, local ? static_cast<void*>(dst0) : s.shard_out,
                 chunk_size, threshold, s.stream);
    cudaEventRecord(s.ev[1], s.stream);
    if (rc == B2FIL_OK && !local) {
      const cudaError_t e = cudaMemcpyPeerAsync(dst0, f0->device, s.shard_out, f->device,
                                                static_cast<size_t>(n) * out_row_b, s.stream);
      if (e != cudaSuccess) rc = cuda_error("cudaMemcpyPeerAsync", e);
    }
    cudaEventRecord(s.ev[2], s.stream);
    if (rc != B2FIL_OK) rc_final = rc;
  }
  // Wait for every device that was fed, also after an error on a later device: their kernels and
  // copies still write into the caller's output.
  ShardTiming timing;
  for (int i : fed) {
    b2fil_forest* f = forests[i];
    DeviceGuard guard(f->device);
    HostSlot& s         = f->slots[0];
    const cudaError_t e = cudaStreamSynchronize(s.stream);
    if (e != cudaSuccess) {
      if (rc_final == B2FIL_OK) rc_final = cuda_error("cudaStreamSynchronize", e);
      continue;
    }
    float ms = 0;
    if (cudaEventElapsedTime(&ms, s.ev[0], s.ev[1]) == cudaSuccess)
      timing.compute_ms = std::max(timing.compute_ms, static_cast<double>(ms));
    if (cudaEventElapsedTime(&ms, s.ev[1], s.ev[2]) == cudaSuccess)
      timing.gather_ms = std::max(timing.gather_ms, static_cast<double>(ms));
    int32_t status = 0;
    const int rc   = read_status_word(f, &status);
    if (rc != B2FIL_OK && rc_final == B2FIL_OK) rc_final = rc;
  }
  timing.wall_ms =
    std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  timing.direct  = direct;
  timing.valid   = 1;
  g_shard_timing = timing;
  return rc_final;
}

}  // extern "C"
