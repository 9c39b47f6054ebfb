// Kernel for sparse forests that carry the compact image (forest.hpp): deep, ragged trees whose
// prediction is a chain of dependent node fetches.
//
// A CTA owns a tile of R rows staged feature-major in shared memory, like the other kernels, and
// its warps form (R/32 row sets) x (G tree groups); a warp walks its 32 rows through NT trees at
// a time.  Every walk has two parts:
//   1. the top T levels of the tree are a complete heap that a producer warp streams through a
//      ring of shared-memory stages (bulk copies from the L2-resident heap array; one stage =
//      the heaps of G * NT trees): T steps without a global fetch, then one exit that names the
//      block to continue at or the leaf reached;
//   2. below the heap the walk goes from block to block in global memory: 32 bytes, one sector, with
//      a node, its two children and one grandchild (forest.hpp).  The tests of a block are
//      straight-line code and end in the predicated fetch of the next one; only a test that the
//      float compare leaves open (missing value, fp64 tie) takes a branch.
// A stage is released as soon as the warp has left the heaps, before it starts on part 2, so the
// next batch of heaps arrives while the warps wait for their node fetches.
// The row tile holds floats also for fp64 forests: every value is rounded DOWN to float when the
// tile is staged.  With lo = the largest float <= threshold (what an fp64 forest's 8-byte node
// stores) and xl = the largest float <= x:  xl < lo proves x < threshold, xl > lo proves
// x > threshold, and only xl == lo leaves the answer open; then, and only then (once in 2^24
// visits on continuous data), the walk reads the row's double from global memory and the exact
// threshold from a side array.  So fp64 forests run on 4-byte tiles and float compares and still
// decide every test exactly.  (fp32 forests: xl = x, lo = threshold, only a missing value is open.)
// Categories survive the rounding too: integers below 2^24 are floats, so trunc(xl) = trunc(x).
// Small batches split the tree batches of a row tile over the CTAs of a cluster, like the dense
// kernel does.
#include "device_common.cuh"
#include "kernels_q.hpp"

namespace b2fil {
namespace {

// 23 consumer warps and a producer: 80 registers a thread.  A walk holds a block (8 registers) and four
// of them are in flight; with the 64 registers that 31 consumer warps leave, the blocks spill (200
// trees of depth 20, 300,000 fp64 rows: 28 warps 2100 us, 20 warps 1694 us, 16 warps 1864 us).  At 80
// some words still spill: 60 bytes in fp64 and 24 in fp32 for sums of scalar leaves, 8 and none for leaf
// ids; sums of leaf vectors and categorical tests more.
constexpr int kCompactWarps   = 23;
constexpr int kCompactThreads = (kCompactWarps + 1) * 32;

__device__ __forceinline__ void lds_node(uint32_t a, uint32_t& value, uint32_t& meta)
{
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(value), "=r"(meta) : "r"(a));
}

// One block, issued only where `wanted`; the registers keep their contents otherwise.  A predicated
// instruction rather than a branch: the walks of a warp want their fetches at different steps, and a
// branch per fetch costs more issue slots than the fetch.  L2-only (.cg): the fetches of a warp go to
// 32 unrelated lines and nothing is reused, so the L1 should only track the misses in flight (measured
// 4 to 8 % faster than the read-only path; L2 eviction hints measured slower).
__device__ __forceinline__ void ld_block_if(bool wanted, const uint32_t* ptr, uint32_t (&w)[8])
{
  asm volatile(
    "{\n\t"
    ".reg .pred want;\n\t"
    "setp.ne.u32 want, %9, 0;\n\t"
    "@want ld.global.cg.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
    "}"
    : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7])
    : "l"(ptr), "r"(static_cast<uint32_t>(wanted)));
}

// A test is the float compare xl < lo, where xl is the row's value rounded down to float and lo
// the node's float (fp64 forests: the largest float <= threshold).  It is OPEN when that compare
// does not settle it: the value is missing, or, in an fp64 forest, xl == lo (lo <= x < next float:
// only the doubles know).  One compare instruction (equal-or-unordered) finds both.
template <typename T>
__device__ __forceinline__ bool test_is_open(float xl, float lo)
{
  if constexpr (sizeof(T) == 8) return !(xl < lo || xl > lo);
  return xl != xl;
}

// Exact form of an fp64 test that the floats left open; `exact` points to its threshold.
__device__ __forceinline__ bool compact_exact_left(const double* row_values, const double* exact, uint32_t feat)
{
  // rows past the end of the batch (no values) were staged as zeros
  const double x = row_values != nullptr ? __ldg(row_values + feat) : 0.0;
  return x < __ldg(exact);
}

// Settle an open test off the common path and rewrite (xl, lo) so that the plain compare
// xl < lo gives the answer.
template <typename T, typename Exact>
__device__ __forceinline__ void settle_open_test(float& xl, float& lo, bool default_left, uint32_t feat,
                                                 const double* row_values, Exact exact)
{
  if (!test_is_open<T>(xl, lo)) return;
  bool left = false;  // fp32 forests: xl == lo is x == threshold, which goes right
  if (xl != xl) {
    left = default_left;
  } else if constexpr (sizeof(T) == 8) {
    left = compact_exact_left(row_values, exact(), feat);
  }
  lo = 0.f;
  xl = left ? -1.f : 1.f;
}

// A categorical test, also rewritten into (xl, lo).
__device__ __forceinline__ void settle_categorical_test(float& xl, float& lo, uint32_t value,
                                                        uint32_t meta, const ForestView& f)
{
  const bool right = goes_right<float, true, true>(value, meta, xl, f);
  lo               = 0.f;
  xl               = right ? 1.f : -1.f;
}

// Shared memory: [mbarriers 256 B][row tile][accumulators][16 B][S stages of G * NT heaps].
template <typename T, bool CAT, int MODE, int NT>
__global__ void __launch_bounds__(kCompactThreads, 1)
sparse_compact_kernel(const __grid_constant__ PredictParams p, const int R, const int G, const int S,
                      const int n_splits)
{
  using TR  = Traits<T>;
  using Val = typename TR::Val;
  extern __shared__ __align__(128) unsigned char smem[];
  const ForestView& f = p.f;
  const int F         = f.n_features;
  const int NC        = f.n_outputs;
  const int rw        = R >> 5;
  const int n_cw      = rw * G;
  const int n_ct      = n_cw * 32;
  const int warp      = threadIdx.x >> 5;
  const int lane      = threadIdx.x & 31;
  const int TL        = f.c_top_levels;
  const uint32_t heap_n     = 1u << TL;
  const uint32_t top_stride = static_cast<uint32_t>(f.c_top_stride);

  const uint32_t stride_b    = R * 4u;  // the tile holds floats whatever the forest precision
  const size_t tile_bytes    = align16(static_cast<size_t>(F) * stride_b);
  const size_t acc_bytes     = (MODE <= MODE_VECTOR) ? align16(static_cast<size_t>(G) * NC * R * TR::ES) : 0;
  unsigned char* tile_ptr    = smem + kBarBytes;
  T* acc                     = reinterpret_cast<T*>(tile_ptr + tile_bytes);
  unsigned char* stage_ptr   = tile_ptr + tile_bytes + acc_bytes + 16;
  const uint32_t bars        = smem_addr(smem);
  const uint32_t tile        = smem_addr(tile_ptr);
  const uint32_t stages      = smem_addr(stage_ptr);
  const int per_batch        = G * NT;
  const uint32_t stage_bytes = per_batch * top_stride;
  const int n_batches        = (f.n_trees + per_batch - 1) / per_batch;
  // small batches: the tree batches of a row tile are split over n_splits CTAs, like in
  // dense_kernel (reduced outputs: a cluster)
  const int split   = static_cast<int>(blockIdx.x) % n_splits;
  const int b_begin = static_cast<int>(static_cast<int64_t>(n_batches) * split / n_splits);
  const int b_end   = static_cast<int>(static_cast<int64_t>(n_batches) * (split + 1) / n_splits);
  const int64_t n_tiles   = (p.n_rows + R - 1) / R;
  const int64_t tile0     = blockIdx.x / n_splits;
  const int64_t tile_step = gridDim.x / n_splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bars + 8u * s, 1);                    // full: the producer's expect_tx arrival
      mbar_init(bars + 8u * (kMaxStages + s), n_cw);  // empty: one arrival per consumer warp
    }
    mbar_fence_init();
  }
  __syncthreads();
  grid_release();

  if (warp == n_cw) {
    // ---- producer: one thread streams the heaps of tree batches into the stage ring ------------
    if (lane == 0) {
      const unsigned char* src = f.c_top;
      RingPos pos;
      bool primed = false;  // every stage has been filled once
      for (int64_t t = tile0; t < n_tiles; t += tile_step) {
        for (int b = b_begin; b < b_end; ++b) {
          const uint32_t s = pos.stage;
          if (primed && !mbar_wait(bars + 8u * (kMaxStages + s), pos.phase ^ 1u)) {
            report_status(p.status, 1);
            return;
          }
          const int first      = b * per_batch;
          const int count      = min(per_batch, f.n_trees - first);
          const uint32_t bytes = count * top_stride;
          mbar_expect_tx(bars + 8u * s, bytes);
          bulk_copy_g2s(stages + s * stage_bytes, src + static_cast<size_t>(first) * top_stride,
                        bytes, bars + 8u * s);
          pos.advance(S);
          if (pos.stage == 0) primed = true;
        }
      }
    }
    return;
  }
  if (warp > n_cw) return;

  // ---- consumers --------------------------------------------------------------------------------
  const int g             = warp / rw;
  const int r             = (warp % rw) * 32 + lane;
  T* acc_group            = acc + static_cast<size_t>(g) * NC * R;
  const uint32_t row_addr = tile + r * 4u;
  RingPos pos;
  bool ok = true;
  grid_wait();
  for (int64_t t = tile0; t < n_tiles; t += tile_step) {
    const int64_t row0 = t * R;
    const int64_t row  = row0 + r;
    stage_rows<T, float>(p, tile, R, row0, warp, lane, n_cw);
    if (MODE <= MODE_VECTOR) {
      for (int i = threadIdx.x; i < G * NC * R; i += n_ct) acc[i] = T(0);
    }
    consumer_sync(n_ct);
    {
      // ask the L2 for the rows of this CTA's next tile, so that staging them does not wait on HBM
      const int64_t next0 = row0 + tile_step * R;
      const int row_bytes = F * static_cast<int>(sizeof(T));
      const int lines     = (row_bytes + 127) >> 7;
      for (int i = threadIdx.x; i < R * lines; i += n_ct) {
        const int64_t nrow = next0 + i / lines;
        if (nrow < p.n_rows) {
          const char* at = reinterpret_cast<const char*>(static_cast<const T*>(p.X) + nrow * p.row_stride) +
                           min((i % lines) << 7, row_bytes - 1);
          asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
        }
      }
    }
    Running<T> run{T(0), 0, {}};
    // the row's doubles, for the tests that the float tile leaves open
    auto row_values = [&]() -> const double* {
      return row < p.n_rows ? static_cast<const double*>(p.X) + row * p.row_stride : nullptr;
    };
    for (int b = b_begin; b < b_end; ++b) {
      const uint32_t s = pos.stage;
      if (ok) ok = mbar_wait(bars + 8u * s, pos.phase);
      const int first = b * per_batch + g * NT;
      const int n_act = ok ? min(NT, f.n_trees - first) : 0;
      uint32_t k[NT];  // the block a walk is on, or, with bit 31, the leaf it has reached
      if (n_act > 0) {
        // part 1: the heaps in shared memory
        uint32_t base[NT], h[NT];
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) {
          // slots past the end of the forest repeat the last live tree; results are dropped
          base[kk] = stages + s * stage_bytes +
                     static_cast<uint32_t>(g * NT + min(kk, n_act - 1)) * top_stride;
          h[kk] = 1u;
        }
        for (int lvl = 0; lvl < TL; ++lvl) {
          uint32_t value[NT], meta[NT];
          float xl[NT], lo[NT];
          bool any_open = false;
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) lds_node(base[kk] + h[kk] * 8u, value[kk], meta[kk]);
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            xl[kk] = Traits<float>::ld_real((meta[kk] & CMETA_LOW27) * stride_b + row_addr);
            lo[kk] = __uint_as_float(value[kk]);
            if (CAT && (meta[kk] & META_CATEGORICAL))
              settle_categorical_test(xl[kk], lo[kk], value[kk], meta[kk], f);
            any_open |= test_is_open<T>(xl[kk], lo[kk]);
          }
          if (any_open) {
#pragma unroll
            for (int kk = 0; kk < NT; ++kk) {
              settle_open_test<T>(xl[kk], lo[kk], (meta[kk] & META_DEFAULT_LEFT) != 0u,
                                  meta[kk] & CMETA_LOW27, row_values(), [&]() {
                                    const size_t tree = static_cast<size_t>(first + min(kk, n_act - 1));
                                    return f.c_top_exact + tree * heap_n + h[kk];
                                  });
            }
          }
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) h[kk] = 2u * h[kk] + (xl[kk] < lo[kk] ? 0u : 1u);
        }
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) {
          // the exits follow the 2^T node slots: exit e sits at 8 * (2^T + e) = 8 * h
          k[kk] = lds_u32(base[kk] + h[kk] * 8u);
        }
      }
      // the heaps of this batch are no longer needed: let the producer refill the stage
      uint32_t exits = 0u;
      if (n_act > 0) {
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) exits ^= k[kk];
      }
      release_stage(bars + 8u * (kMaxStages + s), lane, exits != 0xffffffffu, p.zero);
      pos.advance(S);
      if (n_act > 0) {
        // part 2: blocks in global memory.  All lanes of the warp do the three tests of the block
        // they are on, without a branch: root, the child it leads to, and the grandchild (whose
        // operands do not depend on the others) where the walk comes past it.
        uint32_t w[NT][8];
        const uint32_t* blocks = f.c_blocks;
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) {
          // a walk that ended in the heap keeps a block whose tests no value leaves open
          w[kk][0] = w[kk][1] = w[kk][2] = w[kk][3] = 0x00800001u;
          w[kk][4] = w[kk][5] = w[kk][6] = w[kk][7] = 0u;
          ld_block_if(static_cast<int32_t>(k[kk]) >= 0, blocks + static_cast<size_t>(k[kk] & ~C_EXIT_LEAF) * 8,
                      w[kk]);
        }
        // the row's value and the node's for test number `slot(kk)` = test word `half(kk)`
        auto run_tests = [&](auto value, auto half, auto slot, bool (&right)[NT]) {
          float xl[NT], lo[NT];
          bool any_open = false;
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            xl[kk] = Traits<float>::ld_real((half(kk) & BLK_FEATURE) * stride_b + row_addr);
            lo[kk] = __uint_as_float(value(kk));
          }
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            if (CAT && (half(kk) & BLK_CATEGORICAL))
              settle_categorical_test(xl[kk], lo[kk], value(kk),
                                      META_CATEGORICAL | ((half(kk) & BLK_DEFAULT_LEFT) ? META_DEFAULT_LEFT : 0u), f);
            any_open |= test_is_open<T>(xl[kk], lo[kk]);
          }
          if (any_open) {
#pragma unroll
            for (int kk = 0; kk < NT; ++kk) {
              // (a finished walk repeats its last tests: nothing to settle)
              if (static_cast<int32_t>(k[kk]) >= 0)
                settle_open_test<T>(xl[kk], lo[kk], (half(kk) & BLK_DEFAULT_LEFT) != 0u,
                                    half(kk) & BLK_FEATURE, row_values(),
                                    [&]() { return f.c_exact + static_cast<size_t>(k[kk]) * 4 + slot(kk); });
            }
          }
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) right[kk] = !(xl[kk] < lo[kk]);
        };
        for (int step = 0; step < f.c_block_steps; ++step) {
          bool right[NT];
          // edges to leaves (5 bits), place of the grandchild << 8, its answer << 12, root's << 13
          uint32_t facts[NT], value[NT], half[NT];
          run_tests([&](int kk) { return w[kk][3]; }, [&](int kk) { return w[kk][5] >> 16; },
                    [](int) { return 3; }, right);
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            facts[kk] = (w[kk][4] >> 29) | ((w[kk][5] >> 10) & 0x18u) | (right[kk] ? 0x1000u : 0u) |
                        ((w[kk][4] & BLK_HAS_FOURTH) ? (w[kk][4] >> (BLK_FOURTH_SHIFT - 8)) & 0x300u : 0x400u);
          }
          run_tests([&](int kk) { return w[kk][0]; }, [&](int kk) { return w[kk][4]; },
                    [](int) { return 0; }, right);
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            value[kk] = right[kk] ? w[kk][2] : w[kk][1];
            half[kk]  = right[kk] ? w[kk][5] : w[kk][4] >> 16;
            facts[kk] |= right[kk] ? 0x2000u : 0u;
          }
          run_tests([&](int kk) { return value[kk]; }, [&](int kk) { return half[kk]; },
                    [&](int kk) { return (facts[kk] & 0x2000u) ? 2 : 1; }, right);
          bool walking = false;
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            const uint32_t pos    = ((facts[kk] >> 12) & 2u) + (right[kk] ? 1u : 0u);
            const uint32_t fourth = (facts[kk] >> 8) & 7u;
            // past the grandchild's place, or at it and to its right
            const uint32_t edge   = pos + ((2u * pos + ((facts[kk] >> 12) & 1u) > 2u * fourth) ? 1u : 0u);
            const uint32_t before = __popc(facts[kk] & 0x1fu & ~(0xffffffffu << edge));
            const bool leaf       = ((facts[kk] >> edge) & 1u) != 0u;
            const uint32_t next   = leaf ? (w[kk][7] + before) | C_EXIT_LEAF : w[kk][6] + edge - before;
            const bool live       = static_cast<int32_t>(k[kk]) >= 0;
            if (live) k[kk] = next;
            const bool go = live && !leaf;
            ld_block_if(go, blocks + static_cast<size_t>(next & ~C_EXIT_LEAF) * 8, w[kk]);
            walking |= go;
          }
          if (!__any_sync(0xffffffffu, walking)) break;
        }
        uint32_t L[NT];
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) L[kk] = k[kk] & ~C_EXIT_LEAF;
        // the leaves: payload (or id) from the leaf arrays
        if (MODE == MODE_LEAFID) {
          uint32_t id[NT];
#pragma unroll
          for (int kk = 0; kk < NT; ++kk)
            id[kk] = __ldg(f.c_leaf_ids + L[kk]);
          // four live trees that are also the caller's trees o, o + 1, o + 2, o + 3 with o a
          // multiple of four: the row's four ids are contiguous and leave as one 16-byte store
          // (scalar 4-byte stores at a stride of a whole output row cost a sector request each)
          int orig[NT];
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) orig[kk] = __ldg(f.tree_orig + first + min(kk, n_act - 1));
          bool quad = NT == 4 && n_act == NT;
#pragma unroll
          for (int kk = 1; kk < NT; ++kk) quad = quad && orig[kk] == orig[0] + kk;
          const bool wide = quad && (orig[0] & 3) == 0 && (f.n_trees & 3) == 0 &&
                            (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
          if (wide) {
            if (row < p.n_rows) {
              uint32_t* dst = static_cast<uint32_t*>(p.out) + row * f.n_trees + orig[0];
              *reinterpret_cast<uint4*>(dst) =
                make_uint4(id[0], id[NT > 1 ? 1 : 0], id[NT > 2 ? 2 : 0], id[NT > 3 ? 3 : 0]);
            }
          } else if (quad) {
            store_quads<uint32_t>(static_cast<uint32_t*>(p.out), f.n_trees, row, p.n_rows, orig[0], id[0],
                                  id[NT > 1 ? 1 : 0], id[NT > 2 ? 2 : 0], id[NT > 3 ? 3 : 0]);
          } else {
#pragma unroll
            for (int kk = 0; kk < NT; ++kk) {
              if (kk < n_act && row < p.n_rows)
                static_cast<uint32_t*>(p.out)[row * f.n_trees + orig[kk]] = id[kk];
            }
          }
        } else {
          Val pay[NT];
#pragma unroll
          for (int kk = 0; kk < NT; ++kk) {
            pay[kk] = __ldg(static_cast<const Val*>(f.c_leaf_payload) + L[kk]);
          }
          bool quad = false, wide = false;
          int first_orig = 0;
          if (MODE == MODE_PERTREE) {
            // per-tree scalar outputs: the same stores as for leaf ids
            first_orig = __ldg(f.tree_orig + first);
            quad       = NT == 4 && n_act == NT && f.leaf_vector_len <= 1;
#pragma unroll
            for (int kk = 1; kk < NT; ++kk)
              quad = quad && __ldg(f.tree_orig + first + min(kk, n_act - 1)) == first_orig + kk;
            wide = quad && (first_orig & 3) == 0 && (f.n_trees & 3) == 0 &&
                   (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
          }
          if (MODE == MODE_PERTREE && wide) {
            if (row < p.n_rows) {
              Val* dst = static_cast<Val*>(p.out) + row * f.n_trees + first_orig;
              if constexpr (sizeof(Val) == 4) {
                *reinterpret_cast<uint4*>(dst) = make_uint4(pay[0], pay[NT > 1 ? 1 : 0],
                                                            pay[NT > 2 ? 2 : 0], pay[NT > 3 ? 3 : 0]);
              } else {
                *reinterpret_cast<ulonglong2*>(dst)     = make_ulonglong2(pay[0], pay[NT > 1 ? 1 : 0]);
                *reinterpret_cast<ulonglong2*>(dst + 2) = make_ulonglong2(pay[NT > 2 ? 2 : 0],
                                                                          pay[NT > 3 ? 3 : 0]);
              }
            }
          } else if (MODE == MODE_PERTREE && quad) {
            store_quads<Val>(static_cast<Val*>(p.out), f.n_trees, row, p.n_rows, first_orig, pay[0],
                             pay[NT > 1 ? 1 : 0], pay[NT > 2 ? 2 : 0], pay[NT > 3 ? 3 : 0]);
          } else {
#pragma unroll
            for (int kk = 0; kk < NT; ++kk) {
              if (kk < n_act) take_leaf<T, MODE>(p, first + kk, pay[kk], 0u, acc_group, R, r, row, run);
            }
          }
        }
      }
    }
    if (!ok) report_status(p.status, 2);
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
    consumer_sync(n_ct);
  }
}

size_t compact_smem(const ForestView& f, size_t es, bool reduce, int R, int G, int NT, int S)
{
  size_t b = kBarBytes;
  b += align16(static_cast<size_t>(f.n_features) * R * 4);  // the row tile holds floats
  if (reduce) b += align16(static_cast<size_t>(G) * f.n_outputs * R * es);
  b += 16;
  b += static_cast<size_t>(S) * G * NT * static_cast<size_t>(f.c_top_stride);
  return b;
}

template <typename T, bool CAT, int MODE>
int launch_mode(const PredictParams& p, const CompactCfg& c, cudaStream_t stream, std::string& err)
{
  auto k = sparse_compact_kernel<T, CAT, MODE, kCompactTreesInFlight>;
  const SplitLaunch l{dim3(c.grid * c.splits), c.threads, c.smem_bytes, stream,
                      MODE <= MODE_VECTOR ? c.splits : 1, c.splits > 1};
  return launch_split(l, err, k, p, c.rows_per_tile, c.tree_groups, c.stages, c.splits);
}

template <typename T, bool CAT>
int launch_cat(const PredictParams& p, int mode, const CompactCfg& c, cudaStream_t stream,
               std::string& err)
{
  switch (mode) {
    case MODE_SCALAR: return launch_mode<T, CAT, MODE_SCALAR>(p, c, stream, err);
    case MODE_VECTOR: return launch_mode<T, CAT, MODE_VECTOR>(p, c, stream, err);
    case MODE_PERTREE: return launch_mode<T, CAT, MODE_PERTREE>(p, c, stream, err);
    default: return launch_mode<T, CAT, MODE_LEAFID>(p, c, stream, err);
  }
}

}  // namespace

bool compact_config(const ForestView& f, bool reduce, int rows_per_tile, int64_t n_rows,
                    int sm_count, bool may_split, CompactCfg& cfg)
{
  if (!f.c_enabled) return false;
  const size_t es = f.format == FMT_SPARSE_16D ? 8 : 4;
  // Batches of up to two rounds of 128-row tiles: what counts is how many tree batches an SM walks one
  // after the other.  The tree batches of a tile are split over CTAs (reduced outputs: a cluster) where
  // SMs would stay idle, and tile and groups are taken with the least estimated time,
  //   rounds of CTAs x (3 us + tree batches of a CTA x (6 us + 0.15 us per warp)),
  // a tree batch being a chain of dependent fetches whose length hardly depends on its width (100
  // trees of depth 18 on 10,000 rows: 128-row tiles of five groups 51 us, 64-row tiles, which take two
  // rounds, 59 us).  More than 160 KiB of shared memory cost a quarter (the L1 keeps the fetches in
  // flight), and large clusters that need most of the chip wait for the launch before them.
  if (may_split && n_rows <= static_cast<int64_t>(256) * sm_count && tuning_value("compact_R", 0) == 0) {
    const int n_quads = (f.n_trees + kCompactTreesInFlight - 1) / kCompactTreesInFlight;
    double best       = 1e300;
    for (int R = 32; R <= 128; R *= 2) {
      const int rw        = R / 32;
      const int64_t tiles = (n_rows + R - 1) / R;
      int most            = std::min(kCompactWarps / rw, n_quads);
      for (const size_t limit : {kMaxSmemBytes, size_t(160) * 1024}) {
        while (most > 0 && compact_smem(f, es, reduce, R, most, kCompactTreesInFlight, 1) > limit) --most;
        if (most == 0) break;
        for (int C = 1; C <= (reduce ? kMaxCluster : 32); ++C) {
          const int G         = std::min(most, (n_quads + C - 1) / C);
          const int n_batches = (n_quads + G - 1) / G;
          if (C > n_batches) break;
          const double rounds = std::ceil(static_cast<double>(tiles * C) / cluster_ctas(sm_count, reduce ? C : 1));
          const size_t smem   = compact_smem(f, es, reduce, R, G, kCompactTreesInFlight, 1);
          const double walk   = (6.0 + 0.15 * rw * G) * (smem > size_t(160) * 1024 ? 1.25 : 1.0);
          const double wait   = reduce && C > 4 && tiles * C > sm_count / 2 ? 2.0 : 0.0;
          const double cost   = rounds * (3.0 + wait + (n_batches + C - 1) / C * walk);
          if (cost < best) {
            best = cost;
            cfg  = CompactCfg{R, G, 1, smem, (rw * G + 1) * 32, static_cast<int>(tiles), C};
          }
        }
      }
    }
    if (best < 1e300) return true;
  }
  if (const int R = tuning_value("compact_R", 0), G = tuning_value("compact_G", 0),
      S = tuning_value("compact_S", 0);
      R >= 32 && (R & (R - 1)) == 0 && R <= 128 && G >= 1 && (R / 32) * G <= kCompactWarps && S >= 1 &&
      S <= kMaxStages) {  // tuning aid: forced shape
    const size_t b = compact_smem(f, es, reduce, R, G, kCompactTreesInFlight, S);
    if (b <= kMaxSmemBytes) {
      const int64_t n_tiles = (n_rows + R - 1) / R;
      cfg = CompactCfg{R, G, S, b, ((R / 32) * G + 1) * 32,
                       static_cast<int>(std::min<int64_t>(n_tiles, sm_count)), 1};
      return true;
    }
  }
  // Shared memory left unused becomes L1, which is what keeps the node fetches in flight: shapes
  // that stay under 160 KiB are preferred (measured: the same kernel runs twice as fast at
  // 110 KiB as at 216 KiB).  Within a limit: as many warps as there are registers for, then a second
  // stage.
  for (const size_t limit : {size_t(160) * 1024, kMaxSmemBytes}) {
    for (int R = rows_per_tile; R >= 32; R /= 2) {
      const int rw = R / 32;
      for (int G = std::min(kCompactWarps / rw, std::max(1, (f.n_trees + kCompactTreesInFlight - 1) /
                                                    kCompactTreesInFlight));
           G >= 1; --G) {
        for (int S = 2; S >= 1; --S) {
          const size_t b = compact_smem(f, es, reduce, R, G, kCompactTreesInFlight, S);
          if (b <= limit) {
            const int64_t n_tiles = (n_rows + R - 1) / R;
            cfg = CompactCfg{R, G, S, b, (rw * G + 1) * 32,
                             static_cast<int>(std::min<int64_t>(n_tiles, sm_count)), 1};
            return true;
          }
        }
      }
    }
  }
  return false;
}

int launch_sparse_compact(const PredictParams& p, int mode, const CompactCfg& c,
                          cudaStream_t stream, std::string& err)
{
  const ForestView& f = p.f;
  if (f.format == FMT_SPARSE_16D)
    return f.has_categorical ? launch_cat<double, true>(p, mode, c, stream, err)
                             : launch_cat<double, false>(p, mode, c, stream, err);
  return f.has_categorical ? launch_cat<float, true>(p, mode, c, stream, err)
                           : launch_cat<float, false>(p, mode, c, stream, err);
}

}  // namespace b2fil
