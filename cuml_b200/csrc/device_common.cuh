// Device-side building blocks shared by every kernel translation unit: shared-memory and
// mbarrier primitives (inline PTX), per-precision traits, the node test, row staging, the CTA
// epilogue (reduction over tree groups, averaging, base score, postprocessor, output
// conversion) and the leaf bookkeeping.  Everything lives in an unnamed namespace: each
// translation unit that includes this file gets its own copy.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <type_traits>
#include <utility>

#include "kernels.hpp"

namespace b2fil {
namespace {


#ifndef B2FIL_SPIN_NS
#define B2FIL_SPIN_NS 256  // sleep between two tries of a bounded mbarrier wait
#endif
constexpr uint32_t kSpinLimit = 1u << 22;  // tries of a bounded mbarrier wait
constexpr int kBarBytes       = 256;       // room for the mbarriers at the start of shared memory
constexpr int kQBarBytes      = 192;       // the same in the traversal over ranks, to which the last bytes matter
constexpr int kMaxStages      = 8;

// ---------------------------------------------------------------------------------------------
// shared-memory and mbarrier primitives (inline PTX)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init()
{
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
    "{\n"
    ".reg .pred p;\n"
    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
    "selp.u32 %0, 1, 0, p;\n"
    "}\n"
    : "=r"(ok)
    : "r"(bar), "r"(parity)
    : "memory");
  return ok != 0;
}
// Bounded wait: false when the barrier did not complete within `limit` tries (each try blocks
// for a hardware-defined short time, then the warp sleeps briefly).
__device__ __forceinline__ bool mbar_wait_limited(uint32_t bar, uint32_t parity, uint32_t limit)
{
  for (uint32_t i = 0; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    // a waiting warp must not compete for issue slots with the warps that are walking trees
#if B2FIL_SPIN_NS > 0
    __nanosleep(B2FIL_SPIN_NS);
#endif
  }
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity)
{
  return mbar_wait_limited(bar, parity, kSpinLimit);
}
// Set the forest's status word (pinned host memory) after a wait that ran out.
__device__ __forceinline__ void report_status(int32_t* status, int32_t code)
{
  *reinterpret_cast<volatile int32_t*>(status) = code;
}
// A warp gives a stage of the ring back to the producer.  The arrival does not wait for shared-memory
// loads that the warp has issued, and the bulk copy that refills the stage does not queue behind
// them as another warp's store would: a load that is held up (the walk of deep forests fills the
// load pipe with fetches from HBM) then reads the next batch.  200 trees of depth 20 in fp64, 200,000
// rows: one prediction in twelve had a few leaves of the wrong tree.  So the arrival depends on what was
// read: `read` is any condition on the last values that this lane has loaded from the stage (all
// loads before them fed their addresses), the vote needs it from every lane, and the arrival's
// address needs the vote, by way of a zero that only the host knows to be one.  The vote is the
// warp's meeting as well; a __syncwarp() beside it is not needed, nothing being written to the stage
// (1.5 M rows of the headline forest: 3.99 ms without the dependency, 4.00 with it, 4.02 with both).
__device__ __forceinline__ void release_stage(uint32_t bar, int lane, bool read, uint32_t zero)
{
  const uint32_t all = __ballot_sync(0xffffffffu, read);
  if (lane == 0) mbar_arrive(bar + (all & zero));
}
// The same where everything that was read has been stored to global memory (one output per row and tree):
// a store leaves the warp with its data, and __syncwarp() keeps the stores before the arrival.  (The
// vote costs leaf ids of 300 trees x 100,003 rows about half a percent.)
__device__ __forceinline__ void release_stored_stage(uint32_t bar, int lane)
{
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}
// Position in a ring of S stages: the stage index and the parity of its current use, advanced
// without a division.
struct RingPos {
  uint32_t stage = 0, phase = 0;
  __device__ __forceinline__ void advance(int S)
  {
    if (++stage == static_cast<uint32_t>(S)) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

// Bulk asynchronous copy global -> shared memory of this CTA, completing `bytes` on `bar`.
// Both addresses are 16-byte aligned and `bytes` is a multiple of 16.
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dst, const void* src, uint32_t bytes,
                                              uint32_t bar)
{
  asm volatile(
    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
      dst),
    "l"(src), "r"(bytes), "r"(bar)
    : "memory");
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a)
{
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t a)
{
  uint32_t v;  // a 16-bit load into a 32-bit register zero-extends
  asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
template <uint32_t OFF>
__device__ __forceinline__ uint32_t lds_u32_at(uint32_t a)  // [a + OFF], OFF an immediate
{
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF));
  return v;
}
// Calls f(std::integral_constant<int, K>) for K = 0, 1, ...: a loop whose counter is a constant
// expression inside the body.
template <typename F, int... Ks>
__device__ __forceinline__ void for_each_constant(F&& f, std::integer_sequence<int, Ks...>)
{
  (f(std::integral_constant<int, Ks>{}), ...);
}
// Barrier among the consumer threads only (the producer warp never joins it).
__device__ __forceinline__ void consumer_sync(int n_threads)
{
  asm volatile("bar.sync 1, %0;" ::"r"(n_threads) : "memory");
}

// Thread-block clusters: barrier over the live threads of all CTAs, and a read of another CTA's
// shared memory (`a`: the address the datum has in this CTA).
__device__ __forceinline__ void cluster_arrive()
{
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t a, uint32_t cta_rank)
{
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta_rank));
  return r;
}
__device__ __forceinline__ float cluster_ld(uint32_t a, float)
{
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double cluster_ld(uint32_t a, double)
{
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
// Programmatic dependent launch.  A kernel enqueued with pdl_attribute() may start while the
// kernel before it in the stream is still running; it reads and writes nothing but the (constant)
// forest before grid_wait(), which returns once that kernel is complete.  grid_release() lets
// the kernel behind this one start in the same way.  Both do nothing in ordinary launches.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------
// per-precision traits
// ---------------------------------------------------------------------------------------------
template <typename T>
struct Traits;

template <>
struct Traits<float> {
  using Val                    = uint32_t;
  static constexpr uint32_t NB = 8;  // dense node bytes
  static constexpr uint32_t ES = 4;  // element bytes (rows, leaves, outputs)
  static __device__ __forceinline__ void ld_node(uint32_t a, Val& v, uint32_t& m)
  {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v), "=r"(m) : "r"(a));
  }
  static __device__ __forceinline__ float ld_real(uint32_t a)
  {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
  }
  // read-only global load that stays where it is written (the compiler may not sink it)
  static __device__ __forceinline__ float ldg_here(const float* ptr)
  {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(ptr));
    return v;
  }
  template <uint32_t OFF>
  static __device__ __forceinline__ float ld_real_at(uint32_t a)  // [a + OFF], OFF an immediate
  {
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
  }
  // a += inc when t <= x (false for NaN), as one predicated add
  static __device__ __forceinline__ void add_if_le(uint32_t& a, float t, float x, uint32_t inc)
  {
    asm("{\n.reg .pred p;\nsetp.le.f32 p, %1, %2;\n@p add.u32 %0, %0, %3;\n}"
        : "+r"(a)
        : "f"(t), "f"(x), "r"(inc));
  }
  static __device__ __forceinline__ void st_real(uint32_t a, float v)
  {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
  }
  static __device__ __forceinline__ Val ld_val(uint32_t a)
  {
    Val v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ float as_real(Val v) { return __uint_as_float(v); }
  static __device__ __forceinline__ uint32_t low32(Val v) { return v; }
  static __device__ __forceinline__ float exp_(float x) { return expf(x); }
  static __device__ __forceinline__ float exp2_(float x) { return exp2f(x); }
  static __device__ __forceinline__ float log1p_(float x) { return log1pf(x); }
};

template <>
struct Traits<double> {
  using Val                    = uint64_t;
  static constexpr uint32_t NB = 16;
  static constexpr uint32_t ES = 8;
  static __device__ __forceinline__ void ld_node(uint32_t a, Val& v, uint32_t& m)
  {
    uint64_t second;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v), "=l"(second) : "r"(a));
    m = static_cast<uint32_t>(second);
  }
  static __device__ __forceinline__ double ld_real(uint32_t a)
  {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ double ldg_here(const double* ptr)
  {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(ptr));
    return v;
  }
  template <uint32_t OFF>
  static __device__ __forceinline__ double ld_real_at(uint32_t a)
  {
    double v;
    asm volatile("ld.shared.f64 %0, [%1+%2];" : "=d"(v) : "r"(a), "n"(OFF));
    return v;
  }
  static __device__ __forceinline__ void add_if_le(uint32_t& a, double t, double x, uint32_t inc)
  {
    asm("{\n.reg .pred p;\nsetp.le.f64 p, %1, %2;\n@p add.u32 %0, %0, %3;\n}"
        : "+r"(a)
        : "d"(t), "d"(x), "r"(inc));
  }
  static __device__ __forceinline__ void st_real(uint32_t a, double v)
  {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
  }
  static __device__ __forceinline__ Val ld_val(uint32_t a)
  {
    Val v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
    return v;
  }
  static __device__ __forceinline__ double as_real(Val v) { return __longlong_as_double(v); }
  static __device__ __forceinline__ uint32_t low32(Val v) { return static_cast<uint32_t>(v); }
  static __device__ __forceinline__ double exp_(double x) { return exp(x); }
  static __device__ __forceinline__ double exp2_(double x) { return exp2(x); }
  static __device__ __forceinline__ double log1p_(double x) { return log1p(x); }
};

// ---------------------------------------------------------------------------------------------
// one test: does the row go to the right child?
//   numerical: x < threshold goes left; categorical: a listed category goes right;
//   a missing value (NaN) follows the node's default direction.
// ---------------------------------------------------------------------------------------------
template <typename T, bool CAT, bool NANS>
__device__ __forceinline__ bool goes_right(typename Traits<T>::Val v, uint32_t meta, T x,
                                           const ForestView& f)
{
  bool left = x < Traits<T>::as_real(v);
  if (CAT) {
    if (meta & META_CATEGORICAL) {
      // category = truncated value; negative and huge values match nothing
      const bool in_range = (x >= T(0)) && (x < T(16777216));
      const uint32_t c    = in_range ? static_cast<uint32_t>(x) : 0u;
      bool matched;
      if (f.cat_inline) {
        const uint32_t bits = Traits<T>::low32(v);
        matched             = in_range && (c < 32u) && (((bits >> (c & 31u)) & 1u) != 0u);
      } else {
        const uint32_t off     = Traits<T>::low32(v);
        const uint32_t n_words = __ldg(f.cat_pool + off);
        const uint32_t w       = c >> 5;
        matched                = false;
        if (in_range && w < n_words) {
          matched = ((__ldg(f.cat_pool + off + 1 + w) >> (c & 31u)) & 1u) != 0u;
        }
      }
      left = !matched;
    }
  }
  if (CAT || NANS) {
    if (x != x) left = (meta & META_DEFAULT_LEFT) != 0u;
  }
  return !left;
}

// ---------------------------------------------------------------------------------------------
// shared pieces of both kernels: row-tile staging, accumulation of a leaf, epilogue
// ---------------------------------------------------------------------------------------------

// The tile of stage_rows, V neighbouring values of one row per lane and item, U items in flight.  No
// branch per load: dead lanes and items past the end read the tile's first row (one address for all of
// them), and only the stores look at them (with a branch around every load the smallest predictions took 0.3 to
// 0.8 us longer, up to a tenth).
template <typename T, typename OUT, bool WIDE>
__device__ __forceinline__ bool stage_items(const PredictParams& p, uint32_t tile, int R, int64_t row0,
                                            int warp, int lane, int n_warps)
{
  constexpr int V       = 16 / sizeof(T);
  constexpr int U       = 4;
  constexpr uint32_t ES = sizeof(OUT);
  const int F           = p.f.n_features;
  const int rw          = R >> 5;
  const int wshift      = 31 - __clz(rw);
  const int items       = (F + V - 1) / V * rw;
  const T* X            = static_cast<const T*>(p.X) + row0 * p.row_stride;
  const int n_live      = static_cast<int>(min(static_cast<int64_t>(R), p.n_rows - row0));
  bool saw_nan          = false;
  for (int item = warp; item < items; item += U * n_warps) {
    T v[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int it    = item + u * n_warps;
      const int r     = (it & (rw - 1)) * 32 + lane;
      const int c     = (min(it, items - 1) >> wshift) * V;
      const bool live = it < items && r < n_live;
      const T* at     = X + static_cast<int64_t>(live ? r : 0) * p.row_stride;
      if constexpr (WIDE) {
        const uint4 raw = __ldg(reinterpret_cast<const uint4*>(at + c));
        memcpy(v[u], &raw, 16);
      } else {
#pragma unroll
        for (int k = 0; k < V; ++k) v[u][k] = __ldg(at + min(c + k, F - 1));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int it = item + u * n_warps;
      const int r  = (it & (rw - 1)) * 32 + lane;
      const int c  = (it >> wshift) * V;
      if (it >= items) break;
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const T x = r < n_live ? v[u][k] : T(0);
        saw_nan |= x != x;
        OUT y;
        if constexpr (sizeof(T) > sizeof(OUT)) {
          y = __double2float_rd(x);
        } else {
          y = x;
        }
        if (WIDE || c + k < F) Traits<OUT>::st_real(tile + ((c + k) * R + r) * ES, y);
      }
    }
  }
  return saw_nan;
}

// Stage rows [row0, row0 + R) feature-major, R elements per feature, so that the 32 rows of a warp are
// 32 banks whatever feature each lane asks for.  (With a padded stride the lanes' different features
// shifted them over each other: three wavefronts per test operand, more than half of the
// shared-memory traffic of the sparse walk; dense fp32 walk, 500 trees of depth 8 x 200,000 rows
// without ranks: 652 -> 523 us.)  For stores without conflicts the lanes of a warp take 32 rows and 16
// bytes of each, in one load where rows start on 16-byte boundaries.  OUT is T, or float for doubles
// that are rounded down.  Rows past the end of the batch become zeros.  Returns true when this thread
// saw a NaN.
template <typename T, typename OUT>
__device__ __forceinline__ bool stage_rows(const PredictParams& p, uint32_t tile, int R,
                                           int64_t row0, int warp, int lane, int n_warps)
{
  const bool wide = ((reinterpret_cast<uintptr_t>(p.X) | (p.row_stride * sizeof(T)) |
                      (p.f.n_features * sizeof(T))) & 15u) == 0;
  return wide ? stage_items<T, OUT, true>(p, tile, R, row0, warp, lane, n_warps)
              : stage_items<T, OUT, false>(p, tile, R, row0, warp, lane, n_warps);
}

template <typename T>
__device__ __forceinline__ T postprocess_one(T s, int postproc, T alpha, T ratio_c)
{
  switch (postproc) {
    case B2FIL_POST_SIGMOID:
    case B2FIL_POST_MULTICLASS_OVA: return T(1) / (T(1) + Traits<T>::exp_(-alpha * s));
    case B2FIL_POST_EXPONENTIAL: return Traits<T>::exp_(s);
    case B2FIL_POST_LOG1PEXP: return Traits<T>::log1p_(Traits<T>::exp_(s));
    case B2FIL_POST_SIGNED_SQUARE: return (s < T(0) ? T(-1) : T(1)) * s * s;
    case B2FIL_POST_HINGE: return s > T(0) ? T(1) : T(0);
    case B2FIL_POST_EXP_STD_RATIO: return Traits<T>::exp2_(-s / ratio_c);
    default: return s;
  }
}

// Epilogue of a row tile, one thread per row: fixed-order sum over the G tree groups, average and
// base score, postprocessor, then the output the caller asked for.  `acc` is laid out
// [group][output][row]; results overwrite group 0.
template <typename T>
__device__ __forceinline__ void finish_row(const PredictParams& p, T* acc, int R, int G, int j,
                                           int64_t row)
{
  const ForestView& f = p.f;
  const int NC        = f.n_outputs;
  const T* scale      = static_cast<const T*>(f.out_scale);
  const T* bias       = static_cast<const T*>(f.out_bias);
  const T alpha       = static_cast<T>(f.sigmoid_alpha);
  const T ratio_c     = static_cast<T>(f.ratio_c);
  T mx                = T(0);
  for (int c = 0; c < NC; ++c) {
    T s = acc[c * R + j];
    for (int g = 1; g < G; ++g) s += acc[(g * NC + c) * R + j];
    s = s * __ldg(scale + c) + __ldg(bias + c);
    if (f.postproc != B2FIL_POST_SOFTMAX) s = postprocess_one(s, f.postproc, alpha, ratio_c);
    acc[c * R + j] = s;
    mx             = (c == 0 || s > mx) ? s : mx;
  }
  if (f.postproc == B2FIL_POST_SOFTMAX) {
    T z = T(0);
    for (int c = 0; c < NC; ++c) {
      const T e      = Traits<T>::exp_(acc[c * R + j] - mx);
      acc[c * R + j] = e;
      z += e;
    }
    for (int c = 0; c < NC; ++c) acc[c * R + j] = acc[c * R + j] / z;
  }
  if (row >= p.n_rows) return;
  if (p.kind == B2FIL_INFER_DEFAULT) {
    T* out = static_cast<T*>(p.out) + row * NC;
    for (int c = 0; c < NC; ++c) out[c] = acc[c * R + j];
  } else if (p.kind == B2FIL_INFER_PROBA2) {
    T* out       = static_cast<T*>(p.out) + row * 2;
    const T prob = acc[j];
    out[0]       = T(1) - prob;
    out[1]       = prob;
  } else {  // B2FIL_INFER_CLASS
    int best = 0;
    if (NC == 1) {
      best = acc[j] > static_cast<T>(p.threshold) ? 1 : 0;
    } else {
      T bv = acc[j];
      for (int c = 1; c < NC; ++c) {
        const T s = acc[c * R + j];
        if (s > bv) {  // first maximum wins
          bv   = s;
          best = c;
        }
      }
    }
    static_cast<int32_t*>(p.out)[row] = best;
  }
}

// Epilogue of a row tile whose trees were split over the CTAs of a cluster.  `acc` [group][output]
// [row] holds this CTA's sums; they are added over its groups, then every CTA takes its share of the
// rows and adds the CTAs' sums in rank order from their shared memory: no scratch in global
// memory, no second kernel.  Called by the consumer threads of every CTA (consumer_sync before);
// ends in a cluster_arrive() that the caller has to match with cluster_wait() before it exits.
template <typename T>
__device__ __forceinline__ void finish_cluster_rows(const PredictParams& p, T* acc, int R, int G,
                                                    int64_t row0, int n_ct, int n_splits, int rank)
{
  const int NC = p.f.n_outputs;
  for (int i = threadIdx.x; i < NC * R; i += n_ct) {
    T s = acc[i];
    for (int g = 1; g < G; ++g) s += acc[g * NC * R + i];
    acc[i] = s;
  }
  cluster_arrive();
  cluster_wait();
  // rows [begin, end) of the tile are this CTA's to finish; nobody else reads their sums here
  const int begin = R * rank / n_splits, n_mine = R * (rank + 1) / n_splits - begin;
  for (int i = threadIdx.x; i < NC * n_mine; i += n_ct) {
    T* at            = acc + i / n_mine * R + begin + i % n_mine;
    const uint32_t a = smem_addr(at);
    T part[8];  // loads in flight together (a cluster has at most eight CTAs)
#pragma unroll
    for (int k = 0; k < 8; ++k) part[k] = k < n_splits ? cluster_ld(cluster_map(a, k), T(0)) : T(0);
    T s = part[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) s += part[k];
    *at = s;
  }
  consumer_sync(n_ct);
  if (threadIdx.x < n_mine)
    finish_row<T>(p, acc, R, 1, begin + threadIdx.x, row0 + begin + threadIdx.x);
  cluster_arrive();
}

// Kernel modes.
constexpr int MODE_SCALAR  = 0;  // scalar leaves, reduced outputs
constexpr int MODE_VECTOR  = 1;  // vector leaves, reduced outputs
constexpr int MODE_PERTREE = 2;  // raw per-tree outputs
constexpr int MODE_LEAFID  = 3;  // id of the leaf reached

// Per-thread running state of the reduced modes: the sum of the class that scalar leaves are
// currently feeding, or, for vector leaves of up to kRegClasses outputs, one sum per output
// (forests with more outputs add every leaf vector to shared memory directly).
constexpr int kRegClasses = kQInlineClasses;
template <typename T>
struct Running {
  T sum;
  int cls;
  T v[kRegClasses];
};

// Consume one leaf.  `payload` is the leaf's scalar (as bits) or the index of its vector;
// `leaf_id_index` is the index of the leaf in `leaf_ids`.
template <typename T, int MODE>
__device__ __forceinline__ void take_leaf(const PredictParams& p, int tree,
                                          typename Traits<T>::Val payload, uint32_t leaf_id_index,
                                          T* acc_group, int R, int r, int64_t row, Running<T>& run)
{
  const ForestView& f = p.f;
  const int NC        = f.n_outputs;
  if (MODE == MODE_SCALAR) {
    if (NC > 1) {
      const int cls = __ldg(f.tree_class + tree);  // same for the whole warp
      if (cls != run.cls) {
        acc_group[run.cls * R + r] += run.sum;
        run.sum = T(0);
        run.cls = cls;
      }
    }
    run.sum += Traits<T>::as_real(payload);
  } else if (MODE == MODE_VECTOR) {
    const T* lv = static_cast<const T*>(f.leaf_vectors) +
                  static_cast<size_t>(Traits<T>::low32(payload)) * NC;
    if (NC <= kRegClasses) {
      // few outputs (binary and small multi-class forests of vector leaves, i.e. every
      // scikit-learn style random-forest classifier): sums stay in registers until the tile ends
#pragma unroll
      for (int c = 0; c < kRegClasses; ++c) {
        if (c < NC) run.v[c] += __ldg(lv + c);
      }
    } else {
      // four outputs at a time: the loads of a chunk are in flight together (one after the other
      // they cost a load latency per output)
      int c = 0;
      // (vectors of a multiple of four floats start on 16-byte boundaries: one load per chunk)
      const bool wide = sizeof(T) == 4 && (NC & 3) == 0;
      for (; c + 4 <= NC; c += 4) {
        T v[4], a[4];
        if (wide) {
          const float4 q = __ldg(reinterpret_cast<const float4*>(lv + c));
          v[0] = static_cast<T>(q.x);
          v[1] = static_cast<T>(q.y);
          v[2] = static_cast<T>(q.z);
          v[3] = static_cast<T>(q.w);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) v[u] = __ldg(lv + c + u);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = acc_group[(c + u) * R + r];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc_group[(c + u) * R + r] = a[u] + v[u];
      }
      for (; c < NC; ++c) acc_group[c * R + r] += __ldg(lv + c);
    }
  } else if (MODE == MODE_PERTREE) {
    if (row < p.n_rows) {
      const int orig = __ldg(f.tree_orig + tree);
      if (f.leaf_vector_len > 1) {
        const T* lv = static_cast<const T*>(f.leaf_vectors) +
                      static_cast<size_t>(Traits<T>::low32(payload)) * NC;
        T* out = static_cast<T*>(p.out) + (row * f.n_trees + orig) * NC;
        for (int c = 0; c < NC; ++c) out[c] = __ldg(lv + c);
      } else {
        static_cast<T*>(p.out)[row * f.n_trees + orig] = Traits<T>::as_real(payload);
      }
    }
  } else {
    if (row < p.n_rows) {
      const int orig = __ldg(f.tree_orig + tree);
      static_cast<uint32_t*>(p.out)[row * f.n_trees + orig] = __ldg(f.leaf_ids + leaf_id_index);
    }
  }
}

// Four consecutive outputs of every lane's row (outputs c..c+3 of a row-major array with `width` outputs
// per row) where a row does not start on a 16-byte boundary.  The 4 x 4 values of four lanes are
// transposed with shuffles, then a store covers eight rows x four neighbouring outputs: 11 sectors on
// average instead of the 32 of a store of one output per row.  Called by whole warps; `row` is the
// lane's row and `n_rows` the end of the batch.
template <typename V>
__device__ __forceinline__ void store_quads(V* out, int64_t width, int64_t row, int64_t n_rows, int c,
                                            V v0, V v1, V v2, V v3)
{
  const int lane = threadIdx.x & 31;
  auto swap = [&](bool upper, int mask, V& a, V& b) {
    const V got = __shfl_xor_sync(0xffffffffu, upper ? a : b, mask);
    (upper ? a : b) = got;
  };
  swap(lane & 1, 1, v0, v1);
  swap(lane & 1, 1, v2, v3);
  swap(lane & 2, 2, v0, v2);
  swap(lane & 2, 2, v1, v3);
  // v<j> is now output c + (lane & 3) of the j-th row of the four lanes
  const int64_t first = row - (lane & 3);
  V* at               = out + first * width + c + (lane & 3);
  if (first < n_rows) at[0] = v0;
  if (first + 1 < n_rows) at[width] = v1;
  if (first + 2 < n_rows) at[2 * width] = v2;
  if (first + 3 < n_rows) at[3 * width] = v3;
}

// A condition on the running sums for release_stage(): a reduced walk adds every leaf it reads to them.
template <typename T, int MODE>
__device__ __forceinline__ bool sums_known(const Running<T>& run)
{
  if (MODE == MODE_SCALAR) return run.sum == run.sum;
  bool b = true;
#pragma unroll
  for (int c = 0; c < kRegClasses; ++c) b = b && run.v[c] == run.v[c];
  return b;
}

// Add a thread's running sums to its accumulators in shared memory (end of a row tile), or store
// them where nothing else was added to the tile's accumulators.
template <typename T, int MODE>
__device__ __forceinline__ void flush_running(const ForestView& f, const Running<T>& run,
                                              T* acc_group, int R, int r, bool store = false)
{
  if (MODE == MODE_SCALAR) {
    T* at = acc_group + run.cls * R + r;
    *at   = store ? run.sum : *at + run.sum;
  }
  if (MODE == MODE_VECTOR && f.n_outputs <= kRegClasses) {
#pragma unroll
    for (int c = 0; c < kRegClasses; ++c) {
      if (c < f.n_outputs) {
        T* at = acc_group + c * R + r;
        *at   = store ? run.v[c] : *at + run.v[c];
      }
    }
  }
}

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) / 16 * 16; }

// Position of row r among the R uint16 entries of one feature in a rank tile.  Rows r and r + 32
// share a 32-bit word, so the 32 consecutive rows of a warp sit in 32 different banks whatever
// feature each lane reads (with the plain order two neighbouring rows share a bank and collide
// as soon as they read different features).  Tiles of 32 rows keep the plain order.
__device__ __forceinline__ uint32_t q_slot(uint32_t r, int R)
{
  return R >= 64 ? (((r & 31u) << 1) | ((r >> 5) & 1u) | ((r >> 6) << 6)) : r;
}
// The row that sits in slot s (inverse of q_slot).
__device__ __forceinline__ uint32_t q_row_of_slot(uint32_t s, int R)
{
  return R >= 64 ? (((s >> 6) << 6) | ((s & 63u) >> 1) | ((s & 1u) << 5)) : s;
}

}  // namespace
}  // namespace b2fil
