// Prediction kernels for sm_100a.
//
// Work decomposition (both storages): a CTA owns a tile of R consecutive rows, staged once in
// shared memory feature-major (`tile[f][r]`) so that the 32 lanes of a
// warp - 32 different rows - always read 32 different banks whatever feature each lane needs.
// Warps are organised as (R/32 row sets) x (G tree groups): every warp walks its 32 rows through
// the trees of its group, NT trees at a time for instruction-level parallelism, and keeps its
// partial sums private; a fixed-order reduction over the G groups, averaging, base score and the
// postprocessor run in the CTA's epilogue, so one launch reads every row once and writes every
// result once.
//
// DENSE storage: trees are complete and heap ordered, so a step is "load node, load feature,
// compare, index = 2*index + went_right" with no child pointer.  A producer warp streams batches
// of G*NT whole trees from global memory (L2 resident) into a ring of shared-memory stages with
// bulk asynchronous copies (cp.async.bulk, completion on an mbarrier); consumer warps release a
// stage through a second mbarrier.  CTAs are persistent (one per SM) and loop over row tiles.
//
// SPARSE storage: nodes are fetched from global memory through the read-only path; each thread
// keeps NT independent traversals in flight to cover the latency of the dependent loads.
//
// Every wait on an mbarrier is bounded: when the bound is hit the kernel sets the status word,
// stops working and returns.
#include <map>
#include <mutex>

#include "device_common.cuh"
#include "kernels_q.hpp"

namespace b2fil {
namespace {
// What the calling thread launched last (see last_launch_variant()).  Plain data: filling it costs
// a few stores per call, the text is only formatted when somebody asks.
struct LaunchRecord {
  const char* prepass = nullptr;  // kernel that ran before the traversal, or null
  const char* kernel  = nullptr;  // traversal kernel family
  const char* real    = "";       // float / double
  int mode = 0, nt = 0, depth = -1, cat = -1, fmt = -1, top = -1;
  int R = 0, G = 0, S = 0, K = 0, splits = 1, tiles = 1, nan_columns = 0;
  int ranks = 0;  // per thread and store of the pre-pass
};
thread_local LaunchRecord g_last_launch;

const char* mode_name(int mode)
{
  switch (mode) {
    case 0: return "scalar";
    case 1: return "vector";
    case 2: return "per_tree";
    default: return "leaf_id";
  }
}

// ---------------------------------------------------------------------------------------------
// bounded-wait self test
// ---------------------------------------------------------------------------------------------
__global__ void bounded_wait_selftest_kernel(int32_t* status, const uint32_t tries)
{
  __shared__ __align__(8) unsigned long long bar_word;
  const uint32_t bar = smem_addr(&bar_word);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);  // one arrival expected; nothing ever arrives
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0 && !mbar_wait_limited(bar, 0, tries)) report_status(status, 5);
}

// ---------------------------------------------------------------------------------------------
// rows from mapped host memory
// ---------------------------------------------------------------------------------------------
// Bound by the link (45 of its 55 GB/s from 4 MB on): four 16-byte loads in flight per thread and a
// thread for every 64 bytes, as long as the SMs hold them, cover its 1.5 us.
__global__ void __launch_bounds__(256)
fetch_kernel(uint4* __restrict__ dst, const uint4* __restrict__ src, const uint32_t n,
             const uint32_t tail_words)
{
  grid_release();
  grid_wait();  // the kernel before this one may still be reading what dst held
  // (the source may be the caller's own array: not a word behind its end is read)
  if (blockIdx.x == 0 && threadIdx.x < tail_words)
    reinterpret_cast<uint32_t*>(dst + n)[threadIdx.x] =
      __ldcs(reinterpret_cast<const uint32_t*>(src + n) + threadIdx.x);
  const uint32_t step = gridDim.x * 256u;
  for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += 4u * step) {
    uint4 v[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (i + k * step < n) v[k] = __ldcs(src + i + k * step);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
      if (i + k * step < n) dst[i + k * step] = v[k];
  }
}

// ---------------------------------------------------------------------------------------------
// DENSE kernel
// ---------------------------------------------------------------------------------------------
// Shared memory: [mbarriers 256 B][row tile][accumulators][flags 16 B][S tree stages].
template <typename T, bool CAT, int MODE, int NT>
struct DenseWalker {
  using TR = Traits<T>;

  // Walk the warp's rows through all trees of the CTA's current tile.
  template <bool NANS>
  static __device__ __forceinline__ bool walk(const PredictParams& p, int G, int S, int g, int r,
                                              int64_t row, int lane, uint32_t bars,
                                              uint32_t stages, uint32_t stage_bytes,
                                              uint32_t row_addr, uint32_t stride_b, T* acc_group,
                                              int R, RingPos& pos, Running<T>& run, int t_begin,
                                              int t_end)
  {
    const ForestView& f    = p.f;
    const int D            = f.dense_depth;
    const uint32_t tstride = static_cast<uint32_t>(f.tree_stride);
    const uint32_t width_b = (1u << D) * TR::NB;  // bytes of the node array of one tree
    const int per_batch    = G * NT;
    bool ok                = true;
    uint32_t seen          = 0u;  // the payloads read, folded
    for (int batch = t_begin; batch < t_end; batch += per_batch) {
      const uint32_t s = pos.stage;
      if (ok) ok = mbar_wait(bars + 8u * s, pos.phase);
      if (ok) {
        const int first = batch + g * NT;
        const int n_act = min(NT, t_end - first);
        if (n_act > 0) {
          uint32_t base[NT], a[NT];
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            // slots past the end of the forest repeat the last live tree; results are dropped
            const int slot = g * NT + min(k, n_act - 1);
            base[k]        = stages + s * stage_bytes + slot * tstride;
            a[k]           = base[k] + TR::NB;  // heap index 1
          }
          for (int lvl = 0; lvl < D; ++lvl) {
#pragma unroll
            for (int k = 0; k < NT; ++k) {
              typename TR::Val v;
              uint32_t meta;
              TR::ld_node(a[k], v, meta);
              // flag bits 30/31 of meta leave the 32-bit product: stride_b is a multiple of 4
              const T x        = TR::ld_real(meta * stride_b + row_addr);
              const bool right = goes_right<T, CAT, NANS>(v, meta, x, f);
              // address of heap node 2i+right from the address of node i
              a[k] = 2u * a[k] - base[k] + (right ? TR::NB : 0u);
            }
          }
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            if (k < n_act) {
              const uint32_t slot = (a[k] - base[k]) / TR::NB - (1u << D);
              const typename TR::Val payload = TR::ld_val(base[k] + width_b + slot * TR::ES);
              if (MODE == MODE_VECTOR) seen ^= TR::low32(payload);
              take_leaf<T, MODE>(p, first + k, payload,
                                 (static_cast<uint32_t>(first + k) << D) + slot, acc_group, R, r,
                                 row, run);
            }
          }
        }
      }
      const uint32_t empty = bars + 8u * (kMaxStages + s);
      if (MODE >= MODE_PERTREE) {
        release_stored_stage(empty, lane);
      } else {
        // (scalar leaves: their sum will do; the indices of vector leaves are folded on the way)
        release_stage(empty, lane, MODE == MODE_SCALAR ? sums_known<T, MODE>(run) : seen != 0xffffffffu,
                      p.zero);
      }
      pos.advance(S);
    }
    return ok;
  }
};

// With n_splits > 1 (small batches) the trees of a row tile are split over n_splits CTAs, each of
// which streams and walks only its share.  Reduced outputs launch those CTAs as a cluster and meet
// in its distributed shared memory (finish_cluster_rows); per-tree outputs need no meeting.
// What bounds such a launch is latency: launch, tile, trees, walk, sum, one after the other.  So
// the barriers are set up and the trees requested before grid_wait(), while the kernel before
// this one may still be running.
template <typename T, bool CAT, int MODE, int NT>
__global__ void __launch_bounds__(544, 1)
dense_kernel(const __grid_constant__ PredictParams p, const int R, const int G, const int S,
             const int n_splits)
{
  using TR = Traits<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  const ForestView& f = p.f;
  const int F         = f.n_features;
  const int NC        = f.n_outputs;
  const int rw        = R >> 5;
  const int n_cw      = rw * G;        // consumer warps
  const int n_ct      = n_cw * 32;     // consumer threads
  const int warp      = threadIdx.x >> 5;
  const int lane      = threadIdx.x & 31;

  const uint32_t stride_b   = R * TR::ES;
  const size_t tile_bytes   = align16(static_cast<size_t>(F) * stride_b);
  const size_t acc_bytes    = (MODE <= MODE_VECTOR) ? align16(static_cast<size_t>(G) * NC * R * TR::ES) : 0;
  unsigned char* tile_ptr   = smem + kBarBytes;
  T* acc                    = reinterpret_cast<T*>(tile_ptr + tile_bytes);
  volatile int* flags       = reinterpret_cast<volatile int*>(tile_ptr + tile_bytes + acc_bytes);
  unsigned char* stage_ptr  = tile_ptr + tile_bytes + acc_bytes + 16;
  const uint32_t bars       = smem_addr(smem);
  const uint32_t tile       = smem_addr(tile_ptr);
  const uint32_t stages     = smem_addr(stage_ptr);
  const uint32_t tstride    = static_cast<uint32_t>(f.tree_stride);
  const int per_batch       = G * NT;
  const uint32_t stage_bytes = per_batch * tstride;
  const int split           = static_cast<int>(blockIdx.x) % n_splits;
  const int t_begin         = static_cast<int>(static_cast<int64_t>(f.n_trees) * split / n_splits);
  const int t_end           = static_cast<int>(static_cast<int64_t>(f.n_trees) * (split + 1) / n_splits);
  const int64_t n_tiles     = (p.n_rows + R - 1) / R;
  const int64_t tile_step   = gridDim.x / n_splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bars + 8u * s, 1);                    // full: the producer's expect_tx arrival
      mbar_init(bars + 8u * (kMaxStages + s), n_cw);  // empty: one arrival per consumer warp
    }
    flags[0] = 0;
    flags[1] = 0;
    mbar_fence_init();
  }
  __syncthreads();
  grid_release();

  if (warp == n_cw) {
    // ---- producer: one thread streams tree batches into the stage ring ----------------------
    if (lane == 0) {
      const unsigned char* src = static_cast<const unsigned char*>(f.nodes);
      RingPos pos;
      bool primed = false;  // every stage has been filled once
      for (int64_t t = blockIdx.x / n_splits; t < n_tiles; t += tile_step) {
        for (int first = t_begin; first < t_end; first += per_batch) {
          const uint32_t s = pos.stage;
          if (primed && !mbar_wait(bars + 8u * (kMaxStages + s), pos.phase ^ 1u)) {
            report_status(p.status, 1);
            return;
          }
          const int count      = min(per_batch, t_end - first);
          const uint32_t bytes = count * tstride;
          mbar_expect_tx(bars + 8u * s, bytes);
          bulk_copy_g2s(stages + s * stage_bytes, src + static_cast<size_t>(first) * tstride,
                        bytes, bars + 8u * s);
          pos.advance(S);
          if (pos.stage == 0) primed = true;
        }
      }
    }
    return;
  }

  // ---- consumers ------------------------------------------------------------------------------
  const int g           = warp / rw;
  const int r           = (warp % rw) * 32 + lane;
  T* acc_group          = acc + static_cast<size_t>(g) * NC * R;
  const uint32_t row_addr = tile + r * TR::ES;
  RingPos pos;
  bool ok               = true;
  grid_wait();
  for (int64_t t = blockIdx.x / n_splits; t < n_tiles; t += tile_step) {
    const int64_t row0 = t * R;
    const bool saw_nan = stage_rows<T, T>(p, tile, R, row0, warp, lane, n_cw);
    if (MODE <= MODE_VECTOR) {
      for (int i = threadIdx.x; i < G * NC * R; i += n_ct) acc[i] = T(0);
    }
    if (__any_sync(0xffffffffu, saw_nan) && lane == 0) flags[0] = 1;
    consumer_sync(n_ct);
    const bool nans = flags[0] != 0;
    Running<T> run{T(0), 0, {}};
    if (ok) {
      if (CAT || nans) {
        ok = DenseWalker<T, CAT, MODE, NT>::template walk<true>(
          p, G, S, g, r, row0 + r, lane, bars, stages, stage_bytes, row_addr, stride_b, acc_group,
          R, pos, run, t_begin, t_end);
      } else {
        ok = DenseWalker<T, CAT, MODE, NT>::template walk<false>(
          p, G, S, g, r, row0 + r, lane, bars, stages, stage_bytes, row_addr, stride_b, acc_group,
          R, pos, run, t_begin, t_end);
      }
      if (!ok) report_status(p.status, 2);
    }
    flush_running<T, MODE>(f, run, acc_group, R, r);
    consumer_sync(n_ct);
    if (MODE <= MODE_VECTOR) {
      if (n_splits > 1) {
        finish_cluster_rows<T>(p, acc, R, G, row0, n_ct, n_splits, split);
        cluster_wait();
      } else if (threadIdx.x < R) {
        finish_row<T>(p, acc, R, G, threadIdx.x, row0 + threadIdx.x);
      }
    }
    if (threadIdx.x == 0) flags[0] = 0;
    consumer_sync(n_ct);
  }
}

// ---------------------------------------------------------------------------------------------
// RANK QUANTISATION of rows (pre-pass of the quantised dense kernel)
// ---------------------------------------------------------------------------------------------
// One CTA owns a bundle of feature groups (usually one group of 32 features; a narrow tail is several
// groups, dealt to its warps): the groups' blobs (feature records, bucket tables, sorted thresholds,
// both tables interleaved across the group's features) arrive in shared memory with one bulk copy,
// then the CTA loops over row tiles.  The group size GF is a power of two, so a thread keeps one
// feature for good (its record sits in registers) and with 32-feature groups a warp reads 128
// contiguous bytes of one row per load and its 32 table lookups never share a bank.  A thread owns NU
// consecutive slots of the rank tile (slot = q_slot(row)), packs their ranks two per word and writes
// its piece of Q[tile][feature][slot] (uint16) with one vector store, the layout the traversal kernel
// pulls into shared memory with a single bulk copy.  Groups or tiles too small to occupy the CTA's
// threads that way are ranked several tiles at a time.  Nothing is exchanged between threads, so the
// tile loop has no barrier.
// The stores of a warp go to 32 different lines, one wavefront of the L1's data pipe each, whatever their
// width: with 16 bytes per lane and store (NU = 8) they were 4 of the 14 wavefronts that 32 values cost, and that
// pipe was busy 80 % of the time.  Sixteen ranks leave as one 32-byte store, a whole sector (NU = 16).  With
// that and one halving less (better bucket grids) 1.5 M rows of 256 features are ranked in 590 us instead of
// 750, 200,000 rows of 512 features in 330 instead of 380.
// Next come the issue slots: 46 instructions per 32 values in the first version, of which the search
// (table entry, four halvings) was 17.  So values are ranked where they were loaded (the next tile's
// load follows in the same registers), the conversion to a bucket saturates instead of clamping,
// ranks are made relative two at a time, and NaN and categories are fixed up off the common path.
// Shared memory: [mbarrier 16 B][blobs].

// Where the pre-pass reports NaN and what it clears for the traversal.
struct QFlags {
  // [tile][n_features, rounded up to a multiple of 4]: a group reports in the bytes of its features;
  // every byte is written, nothing has to be zeroed beforehand; or
  uint8_t* bytes;
  int32_t* words;     // one word per tile, zeroed by the caller
  int32_t* arrived;   // counters of shared row tiles to zero, one per tile, or null
};

// Bucket of a value, the same as q_bucket_host: fma, truncation that saturates at zero (also for NaN),
// clamp to the last bucket.
__device__ __forceinline__ uint32_t q_bucket(float x, float scale, float offset, uint32_t last)
{
  return min(__float2uint_rz(fmaf(x, scale, offset)), last);
}
__device__ __forceinline__ uint32_t q_bucket(double x, double scale, double offset, uint32_t last)
{
  // (a double NaN would not convert to zero)
  return min(__double2uint_rz(fmax(fma(x, scale, offset), 0.0)), last);
}

// GFC > 0 fixes the group size at compile time (table strides become immediates), GFC == 0 reads it
// from the group.  `tid`: the thread's number among those of its group; `tiles_par`: tiles that the
// CTA ranks at a time; it takes batch `first` of them and every `step`-th one after.
template <typename T, int STEPS, int NU, int GFC>
__device__ __forceinline__ void quantise_tiles(const PredictParams& p, const QGroup& grp,
                                               uint16_t* __restrict__ Q, const QFlags& flags, int R,
                                               uint32_t blob_a, const QFeatRec* rec, int tid,
                                               int first, int step, int tiles_par)
{
  using TR               = Traits<T>;
  constexpr int CH       = 4;  // values ranked side by side
  const int GF           = GFC > 0 ? GFC : static_cast<int>(grp.f_end - grp.f_begin);
  const int gshift       = 31 - __clz(GF);
  const int i            = tid & (GF - 1);
  const int per_tile     = R * GF / NU;  // threads of a tile, a power of two
  const int sub          = tid >> (31 - __clz(per_tile));
  const int in_tile      = tid & (per_tile - 1);
  const uint32_t s0      = static_cast<uint32_t>(in_tile >> gshift) * NU;  // first slot of the thread
  const QFeatRec mine    = rec[i];
  const T scale          = static_cast<T>(mine.scale);
  const T offset         = static_cast<T>(mine.offset);
  const uint32_t last    = mine.nbm1;
  const uint32_t lut_row = static_cast<uint32_t>(GF) * 2u;      // bytes between table entries
  const uint32_t thr_row = static_cast<uint32_t>(GF) * TR::ES;  // bytes between thresholds
  const int eshift       = gshift + (TR::ES == 4 ? 2 : 3);      // log2(thr_row)
  const uint32_t lut     = blob_a + mine.lut_off;
  const uint32_t thr_m1  = blob_a + mine.thr_off - thr_row;
  const uint32_t zero2   = (thr_m1 >> eshift) * 0x10001u;  // two ranks of 0, before they are made relative
  const bool any_cat     = __any_sync(0xffffffffu, mine.is_cat != 0);
  const uint32_t tile_elems = static_cast<uint32_t>(p.f.n_features) * R;  // ranks per tile
  const int n_rows       = static_cast<int>(p.n_rows);  // a chunk of the batch
  const int rshift       = 31 - __clz(R);  // R is a power of two
  const int n_tiles      = (n_rows + R - 1) >> rshift;
  const int n_full       = n_rows >> rshift;  // without the partial one at the end
  const int stride       = step * tiles_par;  // tiles between two rounds of the CTA
  // slots s0 + j, j = 0..NU-1, hold rows b + (j >> 1) * pair + (j & 1) * odd (see q_slot)
  const int b            = static_cast<int>(q_row_of_slot(s0, R));
  const int pair         = R >= 64 ? 1 : 2;
  const int odd          = R >= 64 ? 32 : 1;
  int base               = first * tiles_par;  // first tile of the round
  const T* src  = static_cast<const T*>(p.X) +
                 (static_cast<int64_t>(base + sub) * R + b) * p.row_stride + grp.f_begin + i;
  uint16_t* dst = Q + static_cast<int64_t>(base + sub) * tile_elems + (grp.f_begin + i) * R + s0;
  const uint32_t rs      = static_cast<uint32_t>(p.row_stride);  // below 2^22: offsets inside a tile fit 32 bits
  const int64_t advance  = static_cast<int64_t>(stride) * R * p.row_stride;

  // Up to eight values per thread are in flight (more did not fit the registers: 16 spilled).
  constexpr int CHUNKS = NU / CH, AHEAD = CHUNKS < 2 ? CHUNKS : 2;
  T xs[AHEAD * CH];
  // loads chunk c (slots s0 + c * CH ...) of the round that starts at `tile`
  auto fetch = [&](const T* at, int tile, int c) {
    T* to = xs + c % AHEAD * CH;
    if (tile + tiles_par <= n_full) {
#pragma unroll
      for (int j = c * CH; j < c * CH + CH; ++j)
        to[j - c * CH] = TR::ldg_here(at + static_cast<uint32_t>((j >> 1) * pair + (j & 1) * odd) * rs);
    } else {
      const int row = (tile + sub) * R + b;
#pragma unroll
      for (int j = c * CH; j < c * CH + CH; ++j) {
        const int off  = (j >> 1) * pair + (j & 1) * odd;
        to[j - c * CH] = row + off < n_rows ? TR::ldg_here(at + static_cast<uint32_t>(off) * rs) : T(0);
      }
    }
  };
  if (base < n_tiles) {
#pragma unroll
    for (int c = 0; c < AHEAD; ++c) fetch(src, base, c);
  }
  for (; base < n_tiles; base += stride) {
    uint32_t packed[NU / 2];
    bool saw_nan = false;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const T* cur = xs + c % AHEAD * CH;
      // rank of the CH values, step by step across all of them so that the dependent
      // shared-memory lookups of different values overlap.  A NaN walks the same code (bucket 0,
      // every comparison false) and is replaced by Q_NAN_CODE at the end; so does a categorical
      // value (its feature has empty tables), replaced by its category.
      uint32_t a[CH];  // address of the threshold below the current window
#pragma unroll
      for (int u = 0; u < CH; ++u)
        a[u] = (lds_u16(lut + q_bucket(cur[u], scale, offset, last) * lut_row) << eshift) + thr_m1;
      if (STEPS > 0 && GFC > 0) {
        // group size and step count known: the probe offsets are immediates of the loads
        for_each_constant(
          [&](auto kc) {
            constexpr int k        = (STEPS > 0 ? STEPS : 1) - 1 - decltype(kc)::value;
            constexpr uint32_t S_B = (static_cast<uint32_t>(GFC > 0 ? GFC : 1) * TR::ES) << k;
            T thr[CH];
#pragma unroll
            for (int u = 0; u < CH; ++u) thr[u] = TR::template ld_real_at<S_B>(a[u]);
#pragma unroll
            for (int u = 0; u < CH; ++u) TR::add_if_le(a[u], thr[u], cur[u], S_B);
          },
          std::make_integer_sequence<int, (STEPS > 0 ? STEPS : 0)>{});
      } else if (STEPS >= 0) {
#pragma unroll
        for (int k = STEPS - 1; k >= 0; --k) {
          const uint32_t s_b = thr_row << k;
          T thr[CH];
#pragma unroll
          for (int u = 0; u < CH; ++u) thr[u] = TR::ld_real(a[u] + s_b);
#pragma unroll
          for (int u = 0; u < CH; ++u) TR::add_if_le(a[u], thr[u], cur[u], s_b);
        }
      } else {  // very full buckets: the number of halvings is only known at run time
        for (int k = static_cast<int>(grp.steps) - 1; k >= 0; --k) {
          const uint32_t s_b = thr_row << k;
#pragma unroll
          for (int u = 0; u < CH; ++u) TR::add_if_le(a[u], TR::ld_real(a[u] + s_b), cur[u], s_b);
        }
      }
      uint32_t* two = packed + c * (CH / 2);
      bool special  = any_cat;
#pragma unroll
      for (int u = 0; u < CH; u += 2) {
        two[u >> 1] = ((a[u + 1] >> eshift) << 16) + (a[u] >> eshift) - zero2;
        special     = special || cur[u] != cur[u] || cur[u + 1] != cur[u + 1];
      }
      if (__any_sync(0xffffffffu, special)) {
        if (any_cat) {
          // the code of a categorical value is the category itself (truncated value); negative and
          // huge values match no listed category
#pragma unroll
          for (int u = 0; u < CH; ++u) {
            const T x           = cur[u];
            const uint32_t code = (x >= T(0)) && (x < T(Q_NO_CATEGORY)) ? static_cast<uint32_t>(x) : Q_NO_CATEGORY;
            const uint32_t keep = (u & 1) ? 0xffffu : 0xffff0000u;
            if (mine.is_cat) two[u >> 1] = (two[u >> 1] & keep) | (code << (16 * (u & 1)));
          }
        }
#pragma unroll
        for (int u = 0; u < CH; u += 2) {
          const uint32_t nan = (cur[u] != cur[u] ? 0xffffu : 0u) | (cur[u + 1] != cur[u + 1] ? 0xffff0000u : 0u);
          two[u >> 1] = (two[u >> 1] & ~nan) | (Q_NAN_CODE * 0x10001u & nan);
          saw_nan |= nan != 0u;
        }
      }
      // the chunk after next, of this round or the CTA's next one, goes into the registers just read
      // (an additional L2 prefetch further ahead measured slower)
      if (c + AHEAD < CHUNKS) {
        fetch(src, base, c + AHEAD);
      } else if (base + stride < n_tiles) {
        if (c + AHEAD == CHUNKS) src += advance;
        fetch(src, base + stride, c + AHEAD - CHUNKS);
      }
    }
    const bool live = base + sub < n_tiles;
    // Q[tile][feature][slot]: the thread's NU consecutive slots of its feature in one store
    if (live) {
      if constexpr (NU == 16) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(packed[0]),
                     "r"(packed[1]), "r"(packed[2]), "r"(packed[3]), "r"(packed[NU > 8 ? 4 : 0]),
                     "r"(packed[NU > 8 ? 5 : 0]), "r"(packed[NU > 8 ? 6 : 0]), "r"(packed[NU > 8 ? 7 : 0])
                     : "memory");
      } else if constexpr (NU == 8) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0], packed[1], packed[NU > 4 ? 2 : 0], packed[NU > 4 ? 3 : 0]);
      } else {
        *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
      }
    }
    dst += static_cast<int64_t>(stride) * tile_elems;
    // NaN flags.  The lanes of a warp rank one tile, or (groups of few features) several
    const uint32_t nan_lanes = __ballot_sync(0xffffffffu, saw_nan);
    if (flags.bytes != nullptr) {
      const int lanes = min(32, per_tile);
      if ((in_tile & (lanes - 1)) == 0 && live) {
        const uint32_t mask = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1u) << (tid & 31);
        // bytes: the lanes' share of the group's, lanes * GF / per_tile = lanes * NU / R
        const int n = per_tile < 32 ? GF : (32 * NU) >> rshift;
        uint8_t* at = flags.bytes + static_cast<int64_t>(base + sub) * ((p.f.n_features + 3) & ~3) +
                      grp.f_begin + (in_tile >> 5) * n;
        for (int k = 0; k < n; ++k) at[k] = (nan_lanes & mask) != 0u ? 1 : 0;
        if (grp.f_end == static_cast<uint32_t>(p.f.n_features) && in_tile == 0)
          for (uint32_t k = grp.f_end; k & 3u; ++k) at[k - grp.f_begin] = 0;  // the padding
      }
    } else if (saw_nan) {
      flags.words[base + sub] = 1;
    }
  }
}

template <typename T, int STEPS>
__device__ __forceinline__ void quantise_rows(const PredictParams& p, const QGroup& grp,
                                              uint16_t* __restrict__ Q, const QFlags& flags, int R,
                                              uint32_t blob_a, const QFeatRec* rec, int tid, int first,
                                              int step, int slots, int tiles_par)
{
  if constexpr (sizeof(T) == 4) {
    if (slots == 16) {
      if (grp.f_end - grp.f_begin == 32 && STEPS >= 2) {
        quantise_tiles<T, STEPS, 16, 32>(p, grp, Q, flags, R, blob_a, rec, tid, first, step, tiles_par);
      } else {
        quantise_tiles<T, STEPS, 16, 0>(p, grp, Q, flags, R, blob_a, rec, tid, first, step, tiles_par);
      }
      return;
    }
  }
  // full-width groups on large tiles, the shape of big batches, get the group size baked in
  if (grp.f_end - grp.f_begin == 32 && STEPS >= 2 && slots == 8) {
    quantise_tiles<T, STEPS, 8, 32>(p, grp, Q, flags, R, blob_a, rec, tid, first, step, tiles_par);
  } else if (slots == 8) {
    quantise_tiles<T, STEPS, 8, 0>(p, grp, Q, flags, R, blob_a, rec, tid, first, step, tiles_par);
  } else {
    quantise_tiles<T, STEPS, 4, 0>(p, grp, Q, flags, R, blob_a, rec, tid, first, step, tiles_par);
  }
}

template <typename T>
__global__ void __launch_bounds__(1024, 1)
quantise_kernel(const __grid_constant__ PredictParams p, uint16_t* __restrict__ Q, const QFlags flags,
                const int R, const int slots, const int ctas)
{
  extern __shared__ __align__(128) unsigned char smem[];
  const ForestView& f   = p.f;
  const uint32_t bar    = smem_addr(smem);
  unsigned char* blob   = smem + 16;
  const uint32_t blob_a = smem_addr(blob);
  // `ctas` CTAs per bundle; the last one may have fewer features, and then takes what is left
  const int which       = min(static_cast<int>(blockIdx.x) / ctas, f.q_n_bundles - 1);
  const int first       = static_cast<int>(blockIdx.x) - which * ctas;
  const int step        = which + 1 == f.q_n_bundles ? static_cast<int>(gridDim.x) - which * ctas : ctas;
  const QBundle bundle  = f.q_bundles[which];
  const int64_t n_tiles = (p.n_rows + R - 1) / R;
  // every feature has 1024 / width threads and every thread `slots` slots of a tile
  const int threads_per_feature = 1024 / static_cast<int>(bundle.width);
  const int tiles_par           = threads_per_feature * slots / R;
  if (static_cast<int64_t>(first) * tiles_par >= n_tiles) return;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    mbar_expect_tx(bar, bundle.blob_bytes);
    bulk_copy_g2s(blob_a, f.q_blob + bundle.blob_off, bundle.blob_bytes, bar);
  }
  // which of the bundle's groups is the thread's?
  int tid       = threadIdx.x;  // the thread's number among those of its group
  QGroup grp    = f.q_groups[bundle.first_group];
  int n_threads = static_cast<int>(grp.f_end - grp.f_begin) * threads_per_feature;
  bool idle     = false;
  for (uint32_t i = 1; tid >= n_threads; ++i) {
    if (i == bundle.n_groups) {
      idle = true;  // the width is rounded up to a power of two
      break;
    }
    tid -= n_threads;
    grp       = f.q_groups[bundle.first_group + i];
    n_threads = static_cast<int>(grp.f_end - grp.f_begin) * threads_per_feature;
  }
  const uint32_t group_at = grp.blob_off - bundle.blob_off;
  const QFeatRec* rec     = reinterpret_cast<const QFeatRec*>(blob + group_at);
  __syncthreads();
  grid_release();
  grid_wait();  // the tables are part of the forest; rows and scratch may still be in use
  // while the tables arrive, ask the L2 for the rows of the CTA's first tile
  if (threadIdx.x < R) {
    const int64_t row = static_cast<int64_t>(first) * tiles_par * R + threadIdx.x;
    if (row < p.n_rows)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const T*>(p.X) + row * p.row_stride + grp.f_begin));
  }
  if (flags.arrived != nullptr && which == 0) {
    for (int64_t t = first * 1024ll + threadIdx.x; t < n_tiles; t += step * 1024ll)
      flags.arrived[t] = 0;
  }
  if (idle) return;
  if (!mbar_wait(bar, 0)) {
    if (threadIdx.x == 0) report_status(p.status, 4);
    return;
  }
  // the number of halvings is fixed per group: pick the unrolled body once
  const uint32_t tables = blob_a + group_at;
  switch (grp.steps) {
    case 0: quantise_rows<T, 0>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    case 1: quantise_rows<T, 1>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    case 2: quantise_rows<T, 2>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    case 3: quantise_rows<T, 3>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    case 4: quantise_rows<T, 4>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    case 5: quantise_rows<T, 5>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
    default: quantise_rows<T, -1>(p, grp, Q, flags, R, tables, rec, tid, first, step, slots, tiles_par); break;
  }
}

// ---------------------------------------------------------------------------------------------
// SPARSE kernel
// ---------------------------------------------------------------------------------------------
template <int FMT>
struct SparseFmt;
template <>
struct SparseFmt<FMT_SPARSE_8> {
  using T = float;
  struct Node {
    uint32_t value, meta, offset;
  };
  static __device__ __forceinline__ Node load(const void* nodes, uint32_t i, int feat_bits)
  {
    const uint2 raw = __ldg(static_cast<const uint2*>(nodes) + i);
    Node n;
    n.value  = raw.x;
    n.meta   = raw.y;
    n.offset = (raw.y & META_LOW29) >> feat_bits;
    return n;
  }
  static __device__ __forceinline__ uint32_t feature(const Node& n, int feat_bits)
  {
    return n.meta & ((1u << feat_bits) - 1u);
  }
};
template <>
struct SparseFmt<FMT_SPARSE_16F> {
  using T = float;
  struct Node {
    uint32_t value, meta, offset;
  };
  static __device__ __forceinline__ Node load(const void* nodes, uint32_t i, int)
  {
    const uint4 raw = __ldg(static_cast<const uint4*>(nodes) + i);
    return Node{raw.x, raw.y, raw.z};
  }
  static __device__ __forceinline__ uint32_t feature(const Node& n, int)
  {
    return n.meta & META_LOW29;
  }
};
template <>
struct SparseFmt<FMT_SPARSE_16D> {
  using T = double;
  struct Node {
    uint64_t value;
    uint32_t meta, offset;
  };
  static __device__ __forceinline__ Node load(const void* nodes, uint32_t i, int)
  {
    const uint4 raw = __ldg(static_cast<const uint4*>(nodes) + i);
    return Node{static_cast<uint64_t>(raw.x) | (static_cast<uint64_t>(raw.y) << 32), raw.z, raw.w};
  }
  static __device__ __forceinline__ uint32_t feature(const Node& n, int)
  {
    return n.meta & META_LOW29;
  }
};

// Shared memory: [row tile (when rows_in_smem)][accumulators].
template <int FMT, int MODE, int NT>
__global__ void __launch_bounds__(1024, 1)
sparse_kernel(const PredictParams p, const int R, const int G, const int rows_in_smem)
{
  using SF = SparseFmt<FMT>;
  using T  = typename SF::T;
  using TR = Traits<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  const ForestView& f = p.f;
  const int F         = f.n_features;
  const int NC        = f.n_outputs;
  const int rw        = R >> 5;
  const int n_warps   = rw * G;
  const int warp      = threadIdx.x >> 5;
  const int lane      = threadIdx.x & 31;
  const int g         = warp / rw;
  const int r         = (warp % rw) * 32 + lane;
  const bool dfs      = f.layout == B2FIL_LAYOUT_DEPTH_FIRST;
  const int fb        = f.feat_bits;

  const uint32_t stride_b = R * TR::ES;
  const size_t tile_bytes = rows_in_smem ? align16(static_cast<size_t>(F) * stride_b) : 0;
  T* acc                  = reinterpret_cast<T*>(smem + tile_bytes);
  T* acc_group            = acc + static_cast<size_t>(g) * NC * R;
  const uint32_t tile     = smem_addr(smem);
  const uint32_t row_addr = tile + r * TR::ES;
  const int64_t n_tiles   = (p.n_rows + R - 1) / R;
  const int per_batch     = G * NT;
  const T* X              = static_cast<const T*>(p.X);

  for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const int64_t row0 = t * R;
    const int64_t row  = row0 + r;
    if (rows_in_smem) stage_rows<T, T>(p, tile, R, row0, warp, lane, n_warps);
    if (MODE <= MODE_VECTOR) {
      for (int i = threadIdx.x; i < G * NC * R; i += n_warps * 32) acc[i] = T(0);
    }
    __syncthreads();
    // rows past the end of the batch read row 0 of the tile's global memory when not staged
    const T* xrow = X + (row < p.n_rows ? row : row0) * p.row_stride;
    Running<T> run{T(0), 0, {}};
    for (int first = g * NT; first < f.n_trees; first += per_batch) {
      const int n_act = min(NT, f.n_trees - first);
      uint32_t idx[NT];
      typename SF::Node node[NT];
#pragma unroll
      for (int k = 0; k < NT; ++k) idx[k] = __ldg(f.roots + first + min(k, n_act - 1));
      // max_depth + 1 nodes lie on the longest path: the loop cannot run away on a bad forest.
      // Every step first issues the node fetches of all NT walks (a walk that has reached its
      // leaf fetches the leaf again, a cache hit), then advances them without branches, so a
      // thread really has NT independent fetches in flight; the warp leaves the loop together.
      for (int step = 0; step <= f.max_depth; ++step) {
#pragma unroll
        for (int k = 0; k < NT; ++k) node[k] = SF::load(f.nodes, idx[k], fb);
        bool walking = false;
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          const bool leaf     = (node[k].meta & META_LEAF) != 0;
          const uint32_t feat = leaf ? 0u : SF::feature(node[k], fb);
          const T x = rows_in_smem ? TR::ld_real(feat * stride_b + row_addr) : __ldg(xrow + feat);
          typename TR::Val v  = node[k].value;
          const bool right    = f.has_categorical
                                  ? goes_right<T, true, true>(v, node[k].meta, x, f)
                                  : goes_right<T, false, true>(v, node[k].meta, x, f);
          // depth-first: left child follows its parent, `offset` reaches the right child;
          // otherwise the children are adjacent and `offset` reaches the left one
          const uint32_t hop =
            dfs ? (right ? node[k].offset : 1u) : (node[k].offset + (right ? 1u : 0u));
          idx[k] += leaf ? 0u : hop;
          walking |= !leaf;
        }
        if (!__any_sync(0xffffffffu, walking)) break;
      }
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        if (k < n_act && (node[k].meta & META_LEAF) != 0) {
          take_leaf<T, MODE>(p, first + k, node[k].value, idx[k], acc_group, R, r, row, run);
        }
      }
    }
    flush_running<T, MODE>(f, run, acc_group, R, r);
    __syncthreads();
    if (MODE <= MODE_VECTOR) {
      if (threadIdx.x < R) finish_row<T>(p, acc, R, G, threadIdx.x, row0 + threadIdx.x);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// host side: launch shapes and dispatch
// ---------------------------------------------------------------------------------------------
size_t dense_tree_stride(int depth, int precision)
{
  const size_t nb = precision == B2FIL_F32 ? 8 : 16;
  const size_t lb = precision == B2FIL_F32 ? 4 : 8;
  return align16((size_t(1) << depth) * (nb + lb));
}

size_t dense_smem(int depth, int precision, int F, int NC, bool reduce, int R, int G, int NT, int S)
{
  const size_t es = precision == B2FIL_F32 ? 4 : 8;
  size_t b        = kBarBytes;
  b += align16(static_cast<size_t>(F) * R * es);
  if (reduce) b += align16(static_cast<size_t>(G) * NC * R * es);
  b += 16;
  b += static_cast<size_t>(S) * G * NT * dense_tree_stride(depth, precision);
  return b;
}

// Raise a kernel's dynamic shared-memory limit to `bytes`.  The limit is a per-device attribute
// of the kernel: it is set once per (device, kernel) and only raised afterwards, so the steady
// state of a serving loop pays a table lookup instead of a driver call.
template <typename K>
int set_smem(K kernel, size_t bytes, std::string& err)
{
  return set_smem_bytes(reinterpret_cast<const void*>(kernel), bytes, err);
}

template <typename T, bool CAT, int MODE>
int launch_dense_mode(const PredictParams& p, const DenseCfg& c, const SplitLaunch& l, int n_splits,
                      std::string& err)
{
  auto k = c.trees_in_flight == 2 ? dense_kernel<T, CAT, MODE, 2> : dense_kernel<T, CAT, MODE, 1>;
  return launch_split(l, err, k, p, c.rows_per_tile, c.tree_groups, c.stages, n_splits);
}

template <typename T, bool CAT>
int launch_dense_cat(const PredictParams& p, int mode, const DenseCfg& c, const SplitLaunch& l,
                     int n_splits, std::string& err)
{
  switch (mode) {
    case MODE_SCALAR: return launch_dense_mode<T, CAT, MODE_SCALAR>(p, c, l, n_splits, err);
    case MODE_VECTOR: return launch_dense_mode<T, CAT, MODE_VECTOR>(p, c, l, n_splits, err);
    case MODE_PERTREE: return launch_dense_mode<T, CAT, MODE_PERTREE>(p, c, l, n_splits, err);
    default: return launch_dense_mode<T, CAT, MODE_LEAFID>(p, c, l, n_splits, err);
  }
}

template <int FMT>
int launch_sparse_fmt(const PredictParams& p, int mode, int R, int G, int rows_in_smem, int grid,
                      size_t smem, cudaStream_t stream, std::string& err)
{
  constexpr int NT = 4;
  const int threads = (R / 32) * G * 32;
  int rc;
#define B2FIL_SPARSE_CASE(M)                                                       \
  {                                                                                \
    auto k = sparse_kernel<FMT, M, NT>;                                            \
    if ((rc = set_smem(k, smem, err)) != B2FIL_OK) return rc;                      \
    k<<<grid, threads, smem, stream>>>(p, R, G, rows_in_smem);                     \
  }
  switch (mode) {
    case MODE_SCALAR: B2FIL_SPARSE_CASE(MODE_SCALAR) break;
    case MODE_VECTOR: B2FIL_SPARSE_CASE(MODE_VECTOR) break;
    case MODE_PERTREE: B2FIL_SPARSE_CASE(MODE_PERTREE) break;
    default: B2FIL_SPARSE_CASE(MODE_LEAFID) break;
  }
#undef B2FIL_SPARSE_CASE
  return B2FIL_OK;
}

size_t dense_q_smem(size_t qstride, int precision, int F, int NC, bool reduce, int R, int G, int NT,
                    int S, int K, int tile_bufs = 1, int acc_bufs = 1, int columns = 1)
{
  const size_t es = precision == B2FIL_F32 ? 4 : 8;
  size_t b        = kQBarBytes;
  b += static_cast<size_t>(tile_bufs) * columns * F * R * 2;
  if (reduce) b += acc_bufs * align16(static_cast<size_t>(G) * NC * R * es);
  b += 16;
  b += static_cast<size_t>(S) * G * NT * K * qstride;
  return b;
}

// Bytes of a tree's test nodes when kernels exist that keep only those in the stages
// (dense_q_leafg_kernel: fp32 scalar leaves, no categorical tests, depth 9 or 10), else 0.
size_t q_node_only_stride(const ForestView& f, int mode)
{
  const bool ok = mode == MODE_SCALAR && q_far(f);
  return ok ? walk_nodes_stride(f.dense_depth) : 0;
}

// Most trees a warp of the quantised kernel may walk side by side: the kernels that exist.
int q_max_trees_in_flight(const ForestView& f, int mode, bool has_top)
{
  if (f.q_has_cat) {
    return f.format == FMT_DENSE_F && mode == MODE_SCALAR && f.dense_depth >= 4 && f.dense_depth <= 8 ? 6 : 4;
  }
  if (!q_walk_order(f)) return 4;
  return mode <= MODE_VECTOR ? 6 : (has_top ? 8 : 4);
}

// Can tiles with missing values be walked with doubled columns?
bool has_nan_image(const ForestView& f, int mode)
{
  return f.q_nodes_nan != nullptr && mode != MODE_LEAFID;
}
// Words of NaN flags per row tile that the traversal has to look at: none when every test sends
// missing values to the right, where the NaN code compares to by itself.
int nan_flag_words(const ForestView& f, int words)
{
  return (f.q_any_default_left || f.q_has_cat) ? words : 0;
}

// Launch shape of the quantised dense kernel: the largest row tile that fits, then as many warps
// as fit (31 consumer warps at most), then as many trees in flight per warp as there is a kernel
// for, then the deepest tree ring that still fits.
// `node_stride` > 0 says that kernels exist which keep only a tree's test nodes (that many bytes)
// in the stages and fetch leaf payloads from global memory; the shape with them is taken when it
// puts at least a third more walks in flight.
bool dense_q_config(size_t qstride, int max_nt, int precision, int F, int NC, bool reduce,
                    int64_t n_rows, int chunk_size, int sm_count, DenseCfg& cfg,
                    size_t node_stride, int64_t visits_per_row, bool nan_image)
{
  int want = 256;
  if (chunk_size > 0) {
    want = chunk_rows(chunk_size, 256);
  } else {
    // tiles are cut between CTAs, so their number need not fill the SMs; larger ones stream the
    // forest less often.  Smaller ones serve forests with few visits per row, which have too few
    // tree batches to cut, and small batches with many outputs, where the sums of a cut tile
    // are the larger part.
    if (n_rows < static_cast<int64_t>(256) * sm_count &&
        (visits_per_row < 1000 || (NC > 4 && n_rows < static_cast<int64_t>(32) * sm_count)))
      want = 128;
  }
  // tuning aid "R,G,NT,S,K": from the environment (read once per process) or, taking
  // precedence, from the knobs q_R, q_G, q_NT, q_S, q_K of b2fil_set_tuning
  static const struct ForcedShape {
    bool set = false;
    int R = 0, G = 0, NT = 0, S = 0, K = 0;
    ForcedShape()
    {
      const char* e = getenv("B2FIL_Q_SHAPE");
      set = e && sscanf(e, "%d,%d,%d,%d,%d", &R, &G, &NT, &S, &K) == 5;
    }
  } from_env;
  ForcedShape forced = from_env;
  if (const int R = tuning_value("q_R", 0); R > 0) {
    forced.set = true;
    forced.R   = R;
    forced.G   = tuning_value("q_G", 1);
    forced.NT  = tuning_value("q_NT", 1);
    forced.S   = tuning_value("q_S", 2);
    forced.K   = tuning_value("q_K", 1);
  }
  if (forced.set) {
    const int R = forced.R, G = forced.G, NT = forced.NT, S = forced.S, K = forced.K;
    const bool leafg = node_stride > 0 && tuning_value("q_leafg", 0) == 1 && NT >= 2 && NT <= 4;
    if (R >= 32 && R % 32 == 0 &&
        R <= 256 && (R & (R - 1)) == 0 && G >= 1 && (R / 32) * G <= 31 &&
        (NT == 1 || NT == 2 || NT == 4 || (NT > 4 && NT == max_nt && (R / 32) * G <= 24) || (NT == 3 && leafg)) &&
        S >= 2 && S <= kMaxStages && K >= 1) {
      const size_t b = dense_q_smem(leafg ? node_stride : qstride, precision, F, NC, reduce, R, G, NT, S, K);
      if (b <= kMaxSmemBytes) {
        cfg = DenseCfg{R, G, NT, S, b, ((R / 32) * G + 1) * 32, K, leafg ? 1 : 0};
        return true;
      }
    }
  }
  const int leafg_knob = tuning_value("q_leafg", -1);  // -1 automatic, 0 never, 1 whenever possible
  for (int R = want; R >= 32; R /= 2) {
    const int rw = R / 32;
    // Among the (tree groups, trees in flight) pairs that fit with a two-stage ring, take the one
    // with the most walks in flight per CTA (row warps x groups x trees): that is what hides the
    // latency of a step, and shapes that shared memory keeps small are bound by exactly it
    // (measured on 2000 depth-10 trees over 512 features, where only 12 trees fit: 3 groups x 2
    // trees 7.2e7 rows/s, 5 groups x 1 tree 6.3e7).  Ties go to more warps.
    int best_g = 0, best_nt = 0, two_g = 0, two_nt = 0;
    // a CTA holds at most 32 warps and one of them is the producer
    // (eight trees: from a tile per SM and 1000 visits per row on; below, 100 trees of depth 8 x 150,000 rows took
    // 66 us instead of 59, 300 of depth 6 x 20,000 25.4 instead of 24.2)
    const bool eight = n_rows >= static_cast<int64_t>(256) * sm_count && visits_per_row >= 1000;
    for (int G = std::min(8, 31 / rw); G >= 1; --G) {
      for (int NT = max_nt == 8 && !eight ? 4 : max_nt; NT >= 1; NT = NT == 6 ? 4 : NT / 2) {
        // the kernels for six and eight trees are built for at most 24 consumer warps (80 registers a thread)
        if (NT > 4 && rw * G > 24) continue;
        auto fits = [&](int tiles) {
          return dense_q_smem(qstride, precision, F, NC, reduce, R, G, NT, 2, 1, tiles) <= kMaxSmemBytes;
        };
        if (G * NT > best_g * best_nt && fits(1)) {
          best_g  = G;
          best_nt = NT;
        }
        if (G * NT > two_g * two_nt && fits(2)) {
          two_g  = G;
          two_nt = NT;
        }
      }
    }
    // (small tiles of forests with few visits: with room for a second one, where that costs little)
    if (R < 256 && visits_per_row < 1000 && two_g * two_nt * 4 >= best_g * best_nt * 3) {
      best_g  = two_g;
      best_nt = two_nt;
    }
    size_t stride = qstride;
    int leafg     = 0;
    if (node_stride > 0 && leafg_knob != 0) {
      // the same search with node-only trees (kernels for two to four trees in flight)
      auto search = [&](int R, int& lg, int& lnt) {
        for (int G = std::min(8, 31 / (R / 32)); G >= 1; --G) {
          for (int NT = 4; NT >= 2; --NT) {
            if (dense_q_smem(node_stride, precision, F, NC, reduce, R, G, NT, 2, 1) > kMaxSmemBytes) continue;
            if (G * NT > lg * lnt) {
              lg  = G;
              lnt = NT;
            }
            break;
          }
        }
      };
      int lg = 0, lnt = 0, half_g = 0, half_nt = 0;
      search(R, lg, lnt);
      // A tile that leaves room for so few trees that half of it would put twice as many walks in flight: such
      // shapes wait for their loads, in walking order, where a test takes longer, more than in heap order (500
      // trees of depth 10, 400 features, 150,000 rows: 734 us in heap order, 767 in walking order, 480 with tiles
      // of 128 rows; 430 features, depth 9: 918 -> 438; 1.3 times as many walks: 689 -> 725).
      if (chunk_size <= 0 && R > 32 && lg > 0) search(R / 2, half_g, half_nt);
      if (half_g * half_nt >= 4 * lg * lnt && lg > 0) continue;
      if (lg > 0 && (leafg_knob == 1 || lg * lnt * 3 >= best_g * best_nt * 4)) {
        best_g  = lg;
        best_nt = lnt;
        stride  = node_stride;
        leafg   = 1;
      }
    }
    if (best_g == 0) continue;
    // a stage holds K sub-batches so that a warp waits and signals once per K * NT trees.
    // Two stages already hide the bulk copies (measured: S = 2 and S = 3 run alike), so a second
    // row tile and room for doubled columns come first - the tile where the trees of a row last only
    // a few microseconds -, and a second set of accumulators takes what is left.
    // One output per row and tree, eight trees at a time: the stores need the L1, and what shared memory leaves
    // of it is more use than a second row tile or longer stages (leaf ids of 300 depth-6 trees, 100,003 rows:
    // 109 us with both, 101 without).
    const bool lean       = best_nt == 8;
    const bool tile_first = visits_per_row < 4000;
    for (int pass = 0; pass < 4; ++pass) {
      const int tiles   = (pass == 0 || pass == (tile_first ? 1 : 2)) ? 2 : 1;
      const int columns = (pass == 0 || pass == (tile_first ? 2 : 1)) ? 2 : 1;
      if ((columns == 2 && !nan_image) || (tiles == 2 && lean)) continue;
      for (int K = lean ? 1 : 2; K >= 1; K /= 2) {
        for (int S = lean ? 2 : 3; S >= 2; --S) {
          for (int accs = reduce ? 2 : 1; accs >= 1; --accs) {
            const size_t b = dense_q_smem(stride, precision, F, NC, reduce, R, best_g, best_nt, S,
                                          K, tiles, accs, columns);
            if (b <= kMaxSmemBytes) {
              cfg = DenseCfg{R, best_g, best_nt, S, b, (rw * best_g + 1) * 32, K, leafg, tiles, accs,
                             columns - 1};
              return true;
            }
          }
        }
      }
    }
  }
  return false;
}

// Launch shapes with at most this many walks in flight per CTA take the child-pair walk.
constexpr int kPairWalkLimit = 0;  // 0: never automatically (set from measurements)

// Pick the kernel family for a launch of the quantised traversal; the families are instantiated
// in the kernels_q_*.cu translation units.
int launch_dense_q_kernel(const QLaunch& L, int mode, bool f64, std::string& err)
{
  const ForestView& f = L.p.f;
  LaunchRecord& rec   = g_last_launch;
  const int ranks     = rec.ranks;  // of the pre-pass, which was launched before
  rec                 = LaunchRecord{};
  rec.ranks           = ranks;
  rec.prepass         = "quantise_kernel";
  rec.kernel          = "dense_q_kernel";
  rec.real            = f64 ? "double" : "float";
  rec.mode            = mode;
  rec.nt              = L.c.trees_in_flight;
  rec.tiles           = L.c.tile_bufs;
  rec.nan_columns     = L.c.nan_columns;
  rec.depth           = 0;  // read at run time unless a specialised body is picked below
  rec.cat             = f.q_has_cat ? 1 : 0;
  rec.R               = L.c.rows_per_tile;
  rec.G               = L.c.tree_groups;
  rec.S               = L.c.stages;
  rec.K               = L.c.sub_batches;
  if (f.q_has_cat) {
    // kernels_q_cat.cu: fp32 scalar leaves of depth 4..8 with four trees in flight are specialised
    if (!f64 && mode == MODE_SCALAR && L.c.trees_in_flight >= 4 && f.dense_depth >= 4 &&
        f.dense_depth <= 8)
      rec.depth = f.dense_depth;
    return launch_q_cat(L, mode, f64, err);
  }
  // Few walks in flight (shapes that shared memory keeps small): the latency of a step is the
  // limit, and the walk that fetches both children ahead of the test halves it.
  const int walks  = (L.c.rows_per_tile / 32) * L.c.tree_groups * L.c.trees_in_flight;
  const int pair   = tuning_value("q_pair", -1);
  const bool can_pair = !f64 && mode == MODE_SCALAR && L.c.trees_in_flight <= 4 && f.dense_depth >= 1;
  if (can_pair && (pair == 1 || (pair < 0 && walks <= kPairWalkLimit))) {
    rec.kernel = "dense_q_pair_kernel";
    return launch_q_pair(L, err);
  }
  if (L.c.leaves_global) {
    rec.kernel = "dense_q_leafg_kernel";
    rec.depth  = f.dense_depth;
    return launch_q_leafg(L, err);
  }
  const bool unrolled = q_walk_order(f);  // the depth is a constant in every kernel from here on, but for the generic one
  const bool has_top  = L.p.q_top != nullptr && f.n_trees <= kQTopTrees;
  if (unrolled && mode >= MODE_PERTREE && (L.c.trees_in_flight == 4 || L.c.trees_in_flight == 8)) {
    rec.depth = f.dense_depth;
    if (has_top) {
      rec.kernel = "dense_q_top_kernel";
      return launch_q_top_out(L, mode, err);
    }
    return launch_q_out4(L, mode, err);
  }
  if (unrolled && mode == MODE_VECTOR && (L.c.trees_in_flight == 6 || L.c.trees_in_flight == 4)) {
    rec.depth = f.dense_depth;
    if (has_top && L.c.trees_in_flight == 6) {
      rec.kernel = "dense_q_top_kernel";
      return launch_q_top_vec(L, err);
    }
    return launch_q_vec(L, err);
  }
  const bool specialised = unrolled && mode == MODE_SCALAR;
  if (specialised && L.c.trees_in_flight == 6) {
    // the common boosted-tree shapes: depth-specialised bodies with six trees in flight
    // (q_max_trees_in_flight offers six only for them)
    rec.depth = f.dense_depth;
    if (has_top) {
      rec.kernel = "dense_q_top_kernel";
      return launch_q_top6(L, err);
    }
    return launch_q_plain6(L, err);
  }
  if (specialised && L.c.trees_in_flight == 4) {
    rec.depth = f.dense_depth;
    return launch_q_plain4(L, err);
  }
  if (unrolled) {  // one or two
    rec.depth = f.dense_depth;
    return launch_q_narrow(L, mode, err);
  }
  return launch_q_generic(L, mode, f64, err);
}

// CTAs per bundle of the rank pre-pass.  Every CTA loads the tables of one bundle of feature groups
// (about 200 KB of an SM's 48 bytes per cycle from L2) and then ranks its share of the row tiles; the
// SMs take the grid in waves of one CTA each.  Taken is the count with the least estimated time,
//   waves x (start and tables + rounds of a CTA x time per round),
// a warp ranking 32 values in kRankCycles SM cycles (measured on 1 M rows of 256 features).  With large
// batches many short CTAs fill the last wave (64 bundles on 148 SMs: 37 CTAs each), with 20,000 rows
// loading the tables twice on an SM costs more than it evens out.
constexpr double kRankCycles = 14.0, kRankCycles16 = 11.0;  // (sixteen ranks per thread and store)
int quantise_ctas_per_bundle(const ForestView& f, int R, int slots, int sm_count, int64_t n_tiles)
{
  const double bundles = f.q_n_bundles - 1 + static_cast<double>(f.q_last_features) / f.q_bundle_features;
  const double tables  = 3000.0 + static_cast<double>(f.q_max_blob_bytes) / 48.0;
  int width = 1;
  while (width < f.q_bundle_features) width *= 2;
  const int par          = 1024 / width * slots / R;  // tiles that a CTA ranks at a time
  const int64_t n_rounds = (n_tiles + par - 1) / par;
  const double per_round = (slots == 16 ? kRankCycles16 : kRankCycles) * R * par * f.q_bundle_features / 32.0 + 100.0;
  int best = 1;
  double best_cost = 1e300;
  const int most = static_cast<int>(std::min<double>(n_rounds, std::max(48.0, sm_count / bundles)));
  for (int gx = 1; gx <= most; ++gx) {
    const int waves   = (static_cast<int>(std::ceil(gx * bundles)) + sm_count - 1) / sm_count;
    const double cost = waves * (tables + static_cast<double>((n_rounds + gx - 1) / gx) * per_round);
    if (cost < best_cost * 0.995) {  // ties and near ties: fewer CTAs
      best_cost = cost;
      best      = gx;
    }
  }
  return best;
}

// Enqueue the rank pre-pass of p's rows.
int launch_quantise(const PredictParams& p, uint16_t* Q, const QFlags& flags, int R, bool f64,
                    int sm_count, cudaStream_t stream, std::string& err)
{
  const ForestView& f = p.f;
  // shared memory: mbarrier and the largest bundle of tables
  const size_t smem = 16 + static_cast<size_t>(f.q_max_blob_bytes);
  // Eight ranks per thread and store; four where tiles are small and so few that the CTAs have one
  // round of them each: there the time of one thread counts.  Sixteen where a CTA has some rounds of so many
  // (from 256 rows and 32 features per SM on) and all features are in groups of 32: whole calls of 13 forests
  // with 32 to 512 features took 0.87 to 0.99 of the time with eight from there on, 1.0 to 1.1 below, and with a
  // narrow group at the end (its CTAs rank 8 or 16 tiles at a time) 0.93 to 1.08.
  const int64_t n_tiles = (p.n_rows + R - 1) / R;
  const bool sixteen    = !f64 && f.n_features % 32 == 0 && f.q_bundle_features == 32 &&
                       f.q_last_features == 32 && p.n_rows * f.q_n_bundles >= int64_t(256) * sm_count;
  const int slots       = R <= 128 && n_tiles * f.q_n_bundles <= sm_count ? 4 : (sixteen ? 16 : 8);
  g_last_launch.ranks   = slots;
  const int gx          = quantise_ctas_per_bundle(f, R, slots, sm_count, n_tiles);
  const int last        = (gx * f.q_last_features + f.q_bundle_features - 1) / f.q_bundle_features;
  // A kernel that overlaps the one before it inherits how that one divided the SM's memory, and the
  // traversal leaves little of it to the L1.  Rows that do not start on 128-byte lines occupy two
  // lines per load in flight, which then no longer fit once they come from HBM (400,000 rows of 100
  // features: 139 us on a fresh division, 236 us on the inherited one); other loads do, and win 5 us
  // of start-up.
  const size_t row_b = static_cast<size_t>(p.row_stride) * (f64 ? 8 : 4);
  const bool overlap = f.q_n_bundles == 1 || row_b % 128 == 0 ||
                       static_cast<size_t>(p.n_rows) * row_b <= size_t(64) << 20;
  const SplitLaunch l{dim3(gx * (f.q_n_bundles - 1) + last), 1024, smem, stream, 1, overlap};
  return f64 ? launch_split(l, err, quantise_kernel<double>, p, Q, flags, R, slots, gx)
             : launch_split(l, err, quantise_kernel<float>, p, Q, flags, R, slots, gx);
}

// Rank-quantised prediction: rows are processed in chunks of whole waves of tiles; for each
// chunk the pre-pass writes the ranks into stream-ordered scratch and the traversal kernel reads
// them back.
int launch_dense_q(const PredictParams& p, int mode, int chunk_size, int sm_count,
                   cudaStream_t stream, const Scratch& pool, std::string& err,
                   int64_t* launches)
{
  const ForestView& f = p.f;
  const int precision = f.format == FMT_DENSE_F ? B2FIL_F32 : B2FIL_F64;
  const bool reduce   = mode <= MODE_VECTOR;
  DenseCfg c;
  if (!dense_q_config(static_cast<size_t>(f.q_tree_stride), q_max_trees_in_flight(f, mode, p.q_top != nullptr), precision,
                      f.n_features, f.n_outputs, reduce, p.n_rows, chunk_size, sm_count, c,
                      q_node_only_stride(f, mode),
                      static_cast<int64_t>(f.n_trees) * f.dense_depth, has_nan_image(f, mode))) {
    err = "no quantised launch shape fits shared memory";
    return B2FIL_ERR_UNSUPPORTED;
  }
  const int R            = c.rows_per_tile;
  const size_t es        = precision == B2FIL_F32 ? 4 : 8;
  const size_t tile_b    = static_cast<size_t>(f.n_features) * R * 2;
  const int64_t wave     = static_cast<int64_t>(R) * sm_count;
  // measured on the 1000-tree depth-8 forest: 64 MB chunks (rank image resident in L2) 2.51e8
  // rows/s, 512 MB chunks 2.62e8: fewer, longer launches beat L2 residency because HBM has
  // plenty of headroom on this path
  // (B2FIL_Q_CHUNK_MB, a tuning aid, overrides the size; the environment is read once)
  static const size_t target = [] {
    size_t t = size_t(512) << 20;
    if (const char* e = getenv("B2FIL_Q_CHUNK_MB")) {
      const long mb = atol(e);
      if (mb >= 1 && mb <= 16384) t = static_cast<size_t>(mb) << 20;
    }
    return t;
  }();
  const int64_t waves    = std::max<int64_t>(1, static_cast<int64_t>(target / (tile_b * sm_count)));
  const int64_t chunk    = std::min<int64_t>(wave * waves, (p.n_rows + R - 1) / R * R);
  const int64_t ch_tiles = (chunk + R - 1) / R;
  // scratch: ranks, sums of shared tiles, NaN flags and arrival counters (zeroed together)
  const int per_batch    = c.tree_groups * c.trees_in_flight * c.sub_batches;
  const int64_t batches  = (f.n_trees + per_batch - 1) / per_batch;
  const size_t q_bytes   = static_cast<size_t>(ch_tiles) * tile_b;
  const size_t sum_bytes =
    reduce ? align16(static_cast<size_t>(2 * sm_count) * f.n_outputs * R * es) : 0;
  const int flag_words   = (f.n_features + 3) / 4;  // a byte per feature
  const size_t fl_bytes  = static_cast<size_t>(ch_tiles) * flag_words * 4;
  const size_t arr_bytes = reduce ? static_cast<size_t>(ch_tiles) * 4 : 0;
  const size_t need      = q_bytes + sum_bytes + fl_bytes + arr_bytes;
  unsigned char* scratch = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&scratch),
                                          need, pool.pool, stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    err = std::string("scratch allocation for quantised rows failed: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? B2FIL_ERR_NO_MEMORY : B2FIL_ERR_CUDA;
  }
  for (int64_t seen = pool.peak->load(); seen < static_cast<int64_t>(need) &&
                                         !pool.peak->compare_exchange_weak(seen, need);) {
  }
  uint16_t* Q     = reinterpret_cast<uint16_t*>(scratch);
  uint8_t* flags  = scratch + q_bytes + sum_bytes;
  int32_t* arrive = reduce ? reinterpret_cast<int32_t*>(flags + fl_bytes) : nullptr;
  int rc          = B2FIL_OK;
  const size_t out_row_b =
    (p.kind == B2FIL_INFER_LEAF_ID ? size_t(4) * f.n_trees
     : p.kind == B2FIL_INFER_CLASS ? size_t(4)
     : p.kind == B2FIL_INFER_PROBA2 ? 2 * es
     : p.kind == B2FIL_INFER_PER_TREE
       ? es * f.n_trees * (f.leaf_vector_len > 1 ? f.n_outputs : 1)
       : es * f.n_outputs);
  for (int64_t r0 = 0; r0 < p.n_rows && rc == B2FIL_OK; r0 += chunk) {
    PredictParams pc = p;
    pc.n_rows        = std::min<int64_t>(chunk, p.n_rows - r0);
    pc.X             = static_cast<const unsigned char*>(p.X) + static_cast<size_t>(r0) * p.row_stride * es;
    pc.out           = static_cast<unsigned char*>(p.out) + static_cast<size_t>(r0) * out_row_b;
    const int64_t n_tiles = (pc.n_rows + R - 1) / R;
    rc = launch_quantise(pc, Q, QFlags{flags, nullptr, arrive}, R, precision != B2FIL_F32,
                         sm_count, stream, err);
    if (rc != B2FIL_OK) break;
    const int grid = static_cast<int>(std::min<int64_t>(n_tiles * batches, sm_count));
    const QArgs qa{Q, reinterpret_cast<const uint32_t*>(flags), nan_flag_words(f, flag_words),
                   reduce ? scratch + q_bytes : nullptr, arrive, R, c.tree_groups, c.stages,
                   c.sub_batches, c.tile_bufs, c.nan_columns, c.acc_bufs};
    rc = launch_dense_q_kernel(QLaunch{pc, qa, c, grid, stream}, mode, precision != B2FIL_F32, err);
    if (launches) *launches += 2;
  }
  cudaFreeAsync(scratch, stream);
  return rc;
}

// ---------------------------------------------------------------------------------------------
// prediction on rank-quantised rows with a fixed, preallocated scratch array
// ---------------------------------------------------------------------------------------------
// The rank image of a batch normally lives in stream-ordered scratch taken from a memory pool.
// This array replaces it for callers that must not allocate while they predict.  It is part of
// the library image: every GPU that loads the library holds it until the process exits.
constexpr size_t kFixedScratchBytes = B2FIL_FIXED_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_fixed_scratch[kFixedScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_fixed_mu;
void* g_fixed_ptr[kMaxDevices] = {};

// Device address of g_fixed_scratch on the current device (`device` is its ordinal).  In host
// code the array's name is only a handle for the runtime, not an address a kernel can use, so the
// address is asked for once per device and cached.
int fixed_scratch_address(int device, void** out, std::string& err)
{
  if (device < 0 || device >= kMaxDevices) {
    err = "device ordinal beyond the fixed-scratch table";
    return B2FIL_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_fixed_mu);
  if (!g_fixed_ptr[device]) {
    void* ptr           = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_fixed_scratch);
    if (e != cudaSuccess || !ptr) {
      err = std::string("cudaGetSymbolAddress(fixed scratch): ") + cudaGetErrorString(e);
      return B2FIL_ERR_CUDA;
    }
    g_fixed_ptr[device] = ptr;
  }
  *out = g_fixed_ptr[device];
  return B2FIL_OK;
}

int pick_rows_per_tile(int64_t n_rows, int chunk_size, int sm_count)
{
  if (chunk_size > 0) return chunk_rows(chunk_size, 128);
  // keep every SM busy before growing the tile
  if (n_rows >= static_cast<int64_t>(128) * sm_count) return 128;
  if (n_rows >= static_cast<int64_t>(64) * sm_count) return 64;
  return 32;
}

std::mutex g_smem_mu;
std::map<std::pair<int, const void*>, size_t> g_smem_set;
std::mutex g_tuning_mu;
std::map<std::string, int> g_tuning;
}  // namespace

int tuning_value(const char* key, int fallback)
{
  std::lock_guard<std::mutex> lock(g_tuning_mu);
  if (g_tuning.empty()) return fallback;
  const auto it = g_tuning.find(key);
  return it == g_tuning.end() ? fallback : it->second;
}
void set_tuning_value(const char* key, int value)
{
  std::lock_guard<std::mutex> lock(g_tuning_mu);
  g_tuning[key] = value;
}

int set_smem_bytes(const void* kernel, size_t bytes, std::string& err)
{
  int device = 0;
  cudaGetDevice(&device);
  const auto key = std::make_pair(device, kernel);
  {
    std::lock_guard<std::mutex> lock(g_smem_mu);
    const auto it = g_smem_set.find(key);
    if (it != g_smem_set.end() && it->second >= bytes) return B2FIL_OK;
  }
  const cudaError_t e = cudaFuncSetAttribute(
    kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) {
    err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_smem_mu);
  size_t& have = g_smem_set[key];
  have         = std::max(have, bytes);
  return B2FIL_OK;
}

bool dense_config(int depth, int precision, int n_features, int n_outputs, bool reduce_kind,
                  int64_t n_rows, int chunk_size, int sm_count, DenseCfg& cfg)
{
  int want = pick_rows_per_tile(n_rows, chunk_size, sm_count);
  for (int R = want; R >= 32; R /= 2) {
    const int rw = R / 32;
    for (int G = 16 / rw; G >= 1; G /= 2) {
      for (int NT = 2; NT >= 1; --NT) {
        for (int S = 3; S >= 2; --S) {
          const size_t b =
            dense_smem(depth, precision, n_features, n_outputs, reduce_kind, R, G, NT, S);
          if (b <= kMaxSmemBytes) {
            cfg = DenseCfg{R, G, NT, S, b, (rw * G + 1) * 32, 1, 0};
            return true;
          }
        }
      }
    }
  }
  return false;
}

// Small batches: at most one round of 128-row tiles.
bool n_rows_small(int64_t n_rows, int sm_count) { return n_rows <= int64_t(128) * sm_count; }

// Measured time of small batches per estimated SM cycle (1000 depth-8 trees x 4,000 rows: 36 us
// for 51,000 cycles).
constexpr double kDenseUsPerCycle = 0.0007;

// Estimated time of the same batch on the rank path: two kernels with their start-up, the ranks of
// every value, the node visits at the pace of large batches.
double rank_path_us(const ForestView& f, int mode, int64_t n_rows, int sm_count)
{
  const bool plain    = f.format == FMT_DENSE_F && !f.q_has_cat && mode == MODE_SCALAR;
  const double visits = static_cast<double>(n_rows) * f.n_trees * std::max(1, f.dense_depth);
  const double values = static_cast<double>(n_rows) * f.n_features;
  const double sms    = sm_count / 148.0;  // the rates are those of 148 SMs
  const double fixed  = mode <= MODE_VECTOR ? 13.0 : 7.5;  // per-tree outputs: no sums to meet
  return fixed + (visits / (plain ? 3.0e6 : 2.0e6) + values / 5.2e5) / sms;
}

// Launch shape of a small batch: row tiles of R rows, each shared by n_splits CTAs that walk their
// part of the forest.  Takes the shape with the least estimated time (in SM cycles):
//   waves x (fixed + rows + max(walk, trees))
// `fixed` is what every CTA spends on starting, meeting and finishing, `rows` and `trees` the time
// to bring the row tile and the CTA's trees in at the 48 bytes per cycle an SM gets from L2, `walk`
// the steps of its tree batches, each bound by the latency of two dependent shared-memory loads
// or by the wavefronts of all its warps (4 per warp and step in fp32, 7 in fp64: a little above the
// 3.7 and 6.1 of large batches, at which fp64 took shapes a quarter slower).  Of 13 forests from 1 to
// 18,000 rows, 5.6 sent 300 depth-6 trees x 5,000 rows to the rank path (17.7 us, now 14.6) and
// 400 depth-9 trees x 2,500 rows (20.6, now 18.4).
struct SplitShape {
  DenseCfg c;
  int n_splits;
  double us;  // estimated time
};
// `rows_per_tile` > 0 asks for that R (the caller's chunk_size).
bool pick_split_shape(const ForestView& f, int mode, int precision, int64_t n_rows,
                      int rows_per_tile, int sm_count, SplitShape& best)
{
  const bool reduce   = mode <= MODE_VECTOR;
  const double es     = precision == B2FIL_F32 ? 4 : 8;
  const double stride = static_cast<double>(dense_tree_stride(f.dense_depth, precision));
  const double wave_w = (precision == B2FIL_F32 ? 4.0 : 7.0) * (f.has_categorical ? 2.0 : 1.0);
  const double leaf_w = mode == MODE_SCALAR ? 4.0 : (mode == MODE_VECTOR ? 32.0 : 64.0);
  const int depth     = std::max(1, f.dense_depth);
  double best_cost    = 1e300;
  for (int R = 32; R <= 128; R *= 2) {
    if (rows_per_tile > 0 ? R != rows_per_tile : (R > 32 && n_rows <= R / 2)) continue;
    const int rw          = R / 32;
    const int64_t n_tiles = (n_rows + R - 1) / R;
    for (int G = 16 / rw; G >= 1; G /= 2) {
      for (int NT = 2; NT >= 1; --NT) {
        int S    = 3;
        size_t b = dense_smem(f.dense_depth, precision, f.n_features, f.n_outputs, reduce, R, G, NT, S);
        if (b > kMaxSmemBytes)
          b = dense_smem(f.dense_depth, precision, f.n_features, f.n_outputs, reduce, R, G, NT, S = 2);
        if (b > kMaxSmemBytes) continue;
        for (int C = 1; C <= (reduce ? kMaxCluster : 64) && C <= f.n_trees; C *= 2) {
          // one CTA per SM and wave: a second one shares the SM's bandwidth, and clusters of eight
          // that overlap the previous launch (half the SMs taken) wait for a whole free GPC slice
          const double waves = std::ceil(static_cast<double>(n_tiles) * C /
                                         cluster_ctas(sm_count, reduce ? C : 1));
          const int trees    = (f.n_trees + C - 1) / C;
          const int batches  = (trees + G * NT - 1) / (G * NT);
          const double walk  = std::max(batches * (150.0 + depth * 120.0),
                                        rw * trees * (depth * wave_w + leaf_w));
          const double rows  = static_cast<double>(R) * f.n_features * es / 48.0;
          const double load  = trees * stride / 48.0;
          const double cost  = waves * (4000.0 + rows + std::max(walk, load));
          if (cost < best_cost) {
            best_cost     = cost;
            best.us       = cost * kDenseUsPerCycle;
            best.c        = DenseCfg{R, G, NT, S, b, (rw * G + 1) * 32, 1, 0};
            best.n_splits = C;
          }
        }
      }
    }
  }
  return best_cost < 1e300;
}

// The same from a small per-thread table of recent answers: the search takes a few microseconds,
// and a serving loop asks for the same few shapes again and again.  The key is all that
// pick_split_shape() looks at.
bool split_shape(const ForestView& f, int mode, int precision, int64_t n_rows, int rows_per_tile,
                 int sm_count, SplitShape& out)
{
  struct Entry {
    int32_t depth, precision, mode, n_features, n_outputs, n_trees, has_categorical, rows_per_tile, sm_count;
    int64_t n_rows;
    bool found;
    SplitShape shape;
  };
  static thread_local Entry table[8] = {};
  static thread_local int next       = 0;
  for (const Entry& e : table) {
    if (e.n_rows == n_rows && e.depth == f.dense_depth && e.precision == precision &&
        e.mode == mode && e.n_features == f.n_features && e.n_outputs == f.n_outputs &&
        e.n_trees == f.n_trees && e.has_categorical == f.has_categorical &&
        e.rows_per_tile == rows_per_tile && e.sm_count == sm_count) {
      out = e.shape;
      return e.found;
    }
  }
  Entry& e = table[next];
  next     = (next + 1) % 8;
  e        = Entry{f.dense_depth, precision, mode, f.n_features, f.n_outputs, f.n_trees,
                   f.has_categorical, rows_per_tile, sm_count, n_rows, false, {}};
  e.found  = pick_split_shape(f, mode, precision, n_rows, rows_per_tile, sm_count, e.shape);
  out      = e.shape;
  return e.found;
}

int dense_ok(int depth, int precision, int n_features, int n_outputs)
{
  // usable when at least 64 rows and two tree groups fit next to a two-stage ring
  if (dense_smem(depth, precision, n_features, n_outputs, true, 64, 2, 1, 2) <= kMaxSmemBytes) return 1;
  // else the traversal over rank-quantised rows alone, if a 32-row tile of ranks and two stages
  // of one tree fit (a tree counted at its largest: 8-byte test nodes, four inline outputs)
  const size_t es      = precision == B2FIL_F32 ? 4 : 8;
  // (without categories the nodes have four bytes, and the holes of the walking order fit into that, too)
  const size_t qstride = (size_t(8) + 4 * es) << depth;
  if (dense_q_smem(qstride, precision, n_features, n_outputs, true, 32, 1, 1, 2, 1) <= kMaxSmemBytes &&
      n_features < (1 << 14))
    return 2;
  return 0;
}

int launch_predict(const PredictParams& p, int chunk_size, int sm_count, cudaStream_t stream,
                   const Scratch* scratch, std::string& err, int64_t* launches)
{
  const ForestView& f = p.f;
  if (p.n_rows == 0) return B2FIL_OK;
  int mode;
  switch (p.kind) {
    case B2FIL_INFER_DEFAULT:
    case B2FIL_INFER_CLASS: mode = f.leaf_vector_len > 1 ? MODE_VECTOR : MODE_SCALAR; break;
    case B2FIL_INFER_PROBA2:
      if (f.n_outputs != 1) {
        err = "B2FIL_INFER_PROBA2 needs a forest with one output";
        return B2FIL_ERR_INVALID_ARG;
      }
      mode = MODE_SCALAR;
      break;
    case B2FIL_INFER_PER_TREE: mode = MODE_PERTREE; break;
    case B2FIL_INFER_LEAF_ID: mode = MODE_LEAFID; break;
    default: err = "unknown infer_kind"; return B2FIL_ERR_INVALID_ARG;
  }
  const bool reduce = mode <= MODE_VECTOR;
  int rc            = B2FIL_OK;
  // the pre-pass indexes a row tile with 32-bit element offsets
  // (small batches skip the pre-pass: with fewer 128-row tiles than half the SMs the forest is
  // split across CTAs of the plain dense kernel instead, which is what bounds their latency)
  // (forests whose row tile only fits as ranks - a thousand features and more - have no other
  // dense kernel and take this path at every batch size)
  const bool dense_fmt = f.format == FMT_DENSE_F || f.format == FMT_DENSE_D;
  const bool ranks_only =
    dense_fmt && dense_ok(f.dense_depth, f.format == FMT_DENSE_F ? B2FIL_F32 : B2FIL_F64,
                          f.n_features, f.n_outputs) != 1;
  // (other small batches take whichever of the two kernels is estimated to be faster)
  const int prec = f.format == FMT_DENSE_F ? B2FIL_F32 : B2FIL_F64;
  SplitShape split;
  bool have_split =
    dense_fmt && !ranks_only && n_rows_small(p.n_rows, sm_count) &&
    split_shape(f, mode, prec, p.n_rows,
                chunk_size > 0 ? pick_rows_per_tile(p.n_rows, chunk_size, sm_count) : 0, sm_count, split);
  if (dense_fmt && f.q_enabled && p.row_stride < (int64_t(1) << 22) && scratch != nullptr &&
      (chunk_size > 0 || !have_split || split.us > rank_path_us(f, mode, p.n_rows, sm_count))) {
    rc = launch_dense_q(p, mode, chunk_size, sm_count, stream, *scratch, err, launches);
    if (rc != B2FIL_OK) return rc;
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      err = std::string("kernel launch: ") + cudaGetErrorString(e);
      return B2FIL_ERR_CUDA;
    }
    return B2FIL_OK;
  }
  if (f.format == FMT_DENSE_F || f.format == FMT_DENSE_D) {
    const int precision = f.format == FMT_DENSE_F ? B2FIL_F32 : B2FIL_F64;
    DenseCfg c;
    int n_splits = 1;
    // small batches split the forest over CTAs: a CTA then streams only its share of the trees
    const bool small = have_split;
    if (have_split) {
      c        = split.c;
      n_splits = split.n_splits;
    } else if (!dense_config(f.dense_depth, precision, f.n_features, f.n_outputs, reduce, p.n_rows,
                             chunk_size, sm_count, c)) {
      err = "no dense launch shape fits shared memory";
      return B2FIL_ERR_UNSUPPORTED;
    }
    const int64_t n_tiles = (p.n_rows + c.rows_per_tile - 1) / c.rows_per_tile;
    const int64_t ctas    = small ? n_tiles * n_splits : std::min<int64_t>(n_tiles, sm_count);
    const SplitLaunch l{dim3(static_cast<unsigned>(ctas)), c.threads, c.smem_bytes, stream,
                        reduce ? n_splits : 1, small};
    {
      LaunchRecord& rec = g_last_launch;
      rec               = LaunchRecord{};
      rec.kernel        = "dense_kernel";
      rec.real          = precision == B2FIL_F32 ? "float" : "double";
      rec.mode          = mode;
      rec.nt            = c.trees_in_flight == 2 ? 2 : 1;
      rec.cat           = f.has_categorical ? 1 : 0;
      rec.R             = c.rows_per_tile;
      rec.G             = c.tree_groups;
      rec.S             = c.stages;
      rec.splits        = n_splits;
    }
    if (precision == B2FIL_F32) {
      rc = f.has_categorical ? launch_dense_cat<float, true>(p, mode, c, l, n_splits, err)
                             : launch_dense_cat<float, false>(p, mode, c, l, n_splits, err);
    } else {
      rc = f.has_categorical ? launch_dense_cat<double, true>(p, mode, c, l, n_splits, err)
                             : launch_dense_cat<double, false>(p, mode, c, l, n_splits, err);
    }
  } else if (CompactCfg cc; compact_config(f, reduce, pick_rows_per_tile(p.n_rows, chunk_size, sm_count),
                                          p.n_rows, sm_count, chunk_size <= 0, cc)) {
    // deep / ragged forests with a compact image: heaps of the top levels through shared memory,
    // blocks of four nodes below
    LaunchRecord& rec = g_last_launch;
    rec               = LaunchRecord{};
    rec.kernel        = "sparse_compact_kernel";
    rec.real          = f.format == FMT_SPARSE_16D ? "double" : "float";
    rec.mode          = mode;
    rec.nt            = kCompactTreesInFlight;
    rec.cat           = f.has_categorical ? 1 : 0;
    rec.top           = f.c_top_levels;
    rec.R             = cc.rows_per_tile;
    rec.G             = cc.tree_groups;
    rec.S             = cc.stages;
    rec.splits        = cc.splits;
    rc = launch_sparse_compact(p, mode, cc, stream, err);
  } else {
    const size_t es = f.format == FMT_SPARSE_16D ? 8 : 4;
    int R           = pick_rows_per_tile(p.n_rows, chunk_size, sm_count);
    int G           = std::min(8, 32 / (R / 32));
    G               = std::max(1, std::min(G, (f.n_trees + 3) / 4));
    // two CTAs per SM when the tile is small enough, else one; rows stay in global memory when
    // even a 32-row tile does not fit
    size_t acc_b = 0, tile_b = 0;
    int rows_in_smem = 1;
    for (;;) {
      acc_b  = reduce ? align16(static_cast<size_t>(G) * f.n_outputs * R * es) : 0;
      tile_b = align16(static_cast<size_t>(f.n_features) * R * es);
      if (acc_b + tile_b <= kMaxSmemBytes) break;
      if (R > 32) {
        R /= 2;
        continue;
      }
      rows_in_smem = 0;
      tile_b       = 0;
      if (acc_b > kMaxSmemBytes) {
        if (G > 1) {
          G /= 2;
          continue;
        }
        err = "too many outputs for the accumulators to fit shared memory";
        return B2FIL_ERR_UNSUPPORTED;
      }
      break;
    }
    const size_t smem     = acc_b + tile_b;
    const int64_t n_tiles = (p.n_rows + R - 1) / R;
    const int grid        = static_cast<int>(std::min<int64_t>(n_tiles, int64_t(sm_count) * 8));
    {
      LaunchRecord& rec = g_last_launch;
      rec               = LaunchRecord{};
      rec.kernel        = "sparse_kernel";
      rec.real          = f.format == FMT_SPARSE_16D ? "double" : "float";
      rec.mode          = mode;
      rec.nt            = 4;
      rec.fmt           = f.format;
      rec.R             = R;
      rec.G             = G;
    }
    switch (f.format) {
      case FMT_SPARSE_8:
        rc = launch_sparse_fmt<FMT_SPARSE_8>(p, mode, R, G, rows_in_smem, grid, smem, stream, err);
        break;
      case FMT_SPARSE_16F:
        rc = launch_sparse_fmt<FMT_SPARSE_16F>(p, mode, R, G, rows_in_smem, grid, smem, stream, err);
        break;
      default:
        rc = launch_sparse_fmt<FMT_SPARSE_16D>(p, mode, R, G, rows_in_smem, grid, smem, stream, err);
        break;
    }
  }
  if (rc != B2FIL_OK) return rc;
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("kernel launch: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  if (launches) ++*launches;
  return B2FIL_OK;
}


int launch_predict_fixed_scratch(const PredictParams& p, int chunk_size, int sm_count, int device,
                                 cudaStream_t stream, std::string& err, int64_t* launches)
{
  const ForestView& f = p.f;
  if (p.n_rows == 0) return B2FIL_OK;
  const bool quantised = (f.format == FMT_DENSE_F || f.format == FMT_DENSE_D) && f.q_enabled &&
                         p.row_stride < (int64_t(1) << 22);
  // forests that predict without scratch take the ordinary path, which allocates nothing for them
  if (!quantised) return launch_predict(p, chunk_size, sm_count, stream, nullptr, err, launches);
  int mode;
  switch (p.kind) {
    case B2FIL_INFER_DEFAULT:
    case B2FIL_INFER_CLASS: mode = f.leaf_vector_len > 1 ? MODE_VECTOR : MODE_SCALAR; break;
    case B2FIL_INFER_PROBA2:
      if (f.n_outputs != 1) {
        err = "B2FIL_INFER_PROBA2 needs a forest with one output";
        return B2FIL_ERR_INVALID_ARG;
      }
      mode = MODE_SCALAR;
      break;
    case B2FIL_INFER_PER_TREE: mode = MODE_PERTREE; break;
    case B2FIL_INFER_LEAF_ID: mode = MODE_LEAFID; break;
    default: err = "unknown infer_kind"; return B2FIL_ERR_INVALID_ARG;
  }
  const int precision = f.format == FMT_DENSE_F ? B2FIL_F32 : B2FIL_F64;
  DenseCfg c;
  int R           = 0;
  int64_t n_tiles = 0;
  size_t q_bytes = 0, fl_bytes = 0;
  auto fits = [&] { return q_bytes + fl_bytes <= kFixedScratchBytes; };
  // (a batch may fit with the largest tiles alone: their flags are the fewest)
  for (const int chunk : {chunk_size, chunk_size > 0 ? chunk_size : 256 / 32}) {
    if (!dense_q_config(static_cast<size_t>(f.q_tree_stride), q_max_trees_in_flight(f, mode, p.q_top != nullptr), precision,
                        f.n_features, f.n_outputs, mode <= MODE_VECTOR, p.n_rows, chunk,
                        sm_count, c, q_node_only_stride(f, mode),
                        static_cast<int64_t>(f.n_trees) * f.dense_depth, has_nan_image(f, mode))) {
      err = "no quantised launch shape fits shared memory";
      return B2FIL_ERR_UNSUPPORTED;
    }
    R        = c.rows_per_tile;
    n_tiles  = (p.n_rows + R - 1) / R;
    q_bytes  = static_cast<size_t>(n_tiles) * f.n_features * R * 2;
    fl_bytes = (static_cast<size_t>(n_tiles) * 4 + 255) / 256 * 256;
    if (fits()) break;
  }
  if (!fits()) {
    const size_t per_row = static_cast<size_t>(f.n_features) * 2 + 1;
    err = "batch too large for the fixed scratch array: " + std::to_string(p.n_rows) +
          " rows of " + std::to_string(f.n_features) + " features need " +
          std::to_string(q_bytes + fl_bytes) + " bytes, the array holds " +
          std::to_string(kFixedScratchBytes) + " (about " +
          std::to_string(kFixedScratchBytes / per_row / 256 * 256) + " rows per call)";
    return B2FIL_ERR_TOO_LARGE;
  }
  void* base = nullptr;
  int rc     = fixed_scratch_address(device, &base, err);
  if (rc != B2FIL_OK) return rc;
  uint16_t* Q    = reinterpret_cast<uint16_t*>(base);
  int32_t* flags = reinterpret_cast<int32_t*>(static_cast<unsigned char*>(base) + q_bytes);
  // the array keeps what the previous call left in it: the NaN flags of the tiles are only ever set
  // and must start at zero (the ranks themselves are fully rewritten)
  cudaError_t e = cudaMemsetAsync(flags, 0, static_cast<size_t>(n_tiles) * 4, stream);
  if (e != cudaSuccess) {
    err = std::string("cudaMemsetAsync: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  rc = launch_quantise(p, Q, QFlags{nullptr, flags, nullptr}, R, precision != B2FIL_F32, sm_count,
                       stream, err);
  if (rc != B2FIL_OK) return rc;
  const int grid = static_cast<int>(std::min<int64_t>(n_tiles, sm_count));
  // (the array holds nothing but ranks and flags: row tiles are not shared by CTAs)
  const QArgs qa{Q, reinterpret_cast<const uint32_t*>(flags), nan_flag_words(f, 1), nullptr,
                 nullptr, R, c.tree_groups, c.stages, c.sub_batches, c.tile_bufs, c.nan_columns,
                 c.acc_bufs};
  rc = launch_dense_q_kernel(QLaunch{p, qa, c, grid, stream}, mode, precision != B2FIL_F32, err);
  if (rc != B2FIL_OK) return rc;
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("kernel launch: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  if (launches) *launches += 2;
  return B2FIL_OK;
}

int launch_fetch(void* dst, const void* src_mapped, size_t bytes, int sm_count, cudaStream_t stream,
                 std::string& err)
{
  const uint32_t n   = static_cast<uint32_t>(bytes / 16);
  const int blocks   = static_cast<int>(std::min<uint32_t>((n + 1023) / 1024, sm_count * 8u));
  const SplitLaunch l{dim3(std::max(1, blocks)), 256, 0, stream, 1, true};
  return launch_split(l, err, fetch_kernel, static_cast<uint4*>(dst),
                      static_cast<const uint4*>(src_mapped), n, static_cast<uint32_t>(bytes % 16 / 4));
}

std::string last_launch_variant()
{
  const LaunchRecord& r = g_last_launch;
  if (!r.kernel) return std::string();
  std::string s;
  if (r.prepass) s += std::string(r.prepass) + "<" + r.real + "> + ";
  s += std::string(r.kernel) + "<" + r.real;
  if (r.fmt >= 0) {
    s += r.fmt == FMT_SPARSE_8 ? ",node8" : (r.fmt == FMT_SPARSE_16F ? ",node16f" : ",node16d");
  }
  s += std::string(",") + mode_name(r.mode) + ",NT=" + std::to_string(r.nt);
  if (r.depth >= 0) s += ",DEPTH=" + (r.depth ? std::to_string(r.depth) : std::string("runtime"));
  if (r.cat >= 0) s += r.cat ? ",CAT" : "";
  if (r.top >= 0) s += ",TOP=" + std::to_string(r.top);
  s += "> R=" + std::to_string(r.R) + " G=" + std::to_string(r.G);
  if (r.S) s += " S=" + std::to_string(r.S);
  if (r.K) s += " K=" + std::to_string(r.K);
  if (r.tiles > 1) s += " tiles=" + std::to_string(r.tiles);
  if (r.nan_columns) s += " nan_columns";
  if (r.splits > 1) s += " forest_splits=" + std::to_string(r.splits);
  if (r.prepass) s += " ranks=" + std::to_string(r.ranks);
  return s;
}

int launch_bounded_wait_selftest(int32_t* status, uint32_t tries, cudaStream_t stream,
                                 std::string& err)
{
  bounded_wait_selftest_kernel<<<1, 32, 0, stream>>>(status, tries);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    err = std::string("kernel launch: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  return B2FIL_OK;
}

}  // namespace b2fil
