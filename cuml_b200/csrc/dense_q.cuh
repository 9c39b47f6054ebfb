// Traversal kernels over rank-quantised rows (templates) and the helper that launches one
// instantiation.  Included by the kernels_q_*.cu translation units, each of which instantiates
// one family of these kernels, so that the families compile in parallel.
#pragma once

#include "device_common.cuh"
#include "kernels_q.hpp"

namespace b2fil {
namespace {

// ---------------------------------------------------------------------------------------------
// DENSE kernel on rank-quantised rows
// ---------------------------------------------------------------------------------------------
// Shared memory: [mbarriers][1 or 2 row tiles F x R uint16][1 or 2 sets of accumulators][16 B]
// [S tree stages].
// The row tile arrives with one bulk copy per tile (the pre-pass already stored it feature-major),
// where there is room for two while the tile before it is being walked (forests whose trees last
// only a few microseconds per tile spend a fifth of them waiting for it otherwise);
// tree batches stream through the stage ring exactly as in dense_kernel.  A node is 4 bytes, a test one
// half-precision compare and a step one predicated addition (forest.hpp), or, in heap order, one signed
// subtraction and a funnel shift.
constexpr int NAN_NONE = 0, NAN_TESTED = 1, NAN_COLUMNS = 2;

constexpr int kBarTileFull  = 2 * kMaxStages;      // mbarrier slots after the stage ring: two each
constexpr int kBarTileEmpty = 2 * kMaxStages + 2;

// node - (q << 17) in one multiply-add: the sign of (j - rank) lands in bit 31.
__device__ __forceinline__ uint32_t rank_diff(uint32_t node, uint32_t q)
{
  static_assert(Q_RANK_SHIFT == 17, "the multiplier below is -(1 << Q_RANK_SHIFT)");
  uint32_t d;
  asm("mad.lo.u32 %0, %1, 0xFFFE0000, %2;" : "=r"(d) : "r"(q), "r"(node));
  return d;
}

// A test and the step behind it: the walk at `a` goes on to the right, `inc` bytes further in its level, when
// the row's rank q is above the node's threshold.  NANS: the tile may hold missing values and its columns
// are not doubled.  A visit is five instructions (node, address of the rank, rank, compare, addition)
// instead of six in heap order with signed subtractions (multiply-add, funnel shift, address): the
// headline forest executes 1.76e9 warp instructions per million rows instead of 2.14e9 at the same 5.9e8
// shared-memory wavefronts, and the traversal takes 2.17 ms instead of 2.24.
template <bool NANS>
__device__ __forceinline__ void walk_step(uint32_t& a, uint32_t node, uint32_t q, uint32_t inc)
{
  static_assert(Q_NAN_CODE == 0x3FFFu, "the constant below");
  if constexpr (!NANS) {
    asm("{\n.reg .pred p;\n.reg .b16 l, h, j, r, z;\n"
        "mov.b32 {l, h}, %1;\nabs.f16 j, h;\nmov.b32 {r, z}, %2;\n"
        "setp.gt.f16 p, r, j;\n@p add.u32 %0, %0, %3;\n}"
        : "+r"(a)
        : "r"(node), "r"(q), "r"(inc));
  } else {
    asm("{\n.reg .pred p, m;\n.reg .b16 l, h, j, r, z;\n"
        "mov.b32 {l, h}, %1;\nabs.f16 j, h;\nmov.b32 {r, z}, %2;\n"
        "setp.lt.s32 m, %1, 0;\nsetp.eq.and.u32 m, %2, 0x3FFF, m;\n"
        "setp.gt.and.f16 p, r, j, !m;\n@p add.u32 %0, %0, %3;\n}"
        : "+r"(a)
        : "r"(node), "r"(q), "r"(inc));
  }
}
// The same at the root, where both children are at hand: returns the one that the row goes to.
template <bool NANS>
__device__ __forceinline__ uint32_t root_step(uint32_t& a, uint32_t node, uint32_t q, uint32_t left, uint32_t right)
{
  uint32_t next;
  if constexpr (!NANS) {
    asm("{\n.reg .pred p;\n.reg .b16 l, h, j, r, z;\n"
        "mov.b32 {l, h}, %2;\nabs.f16 j, h;\nmov.b32 {r, z}, %3;\n"
        "setp.gt.f16 p, r, j;\nselp.b32 %1, %5, %4, p;\n@p add.u32 %0, %0, 4;\n}"
        : "+r"(a), "=r"(next)
        : "r"(node), "r"(q), "r"(left), "r"(right));
  } else {
    asm("{\n.reg .pred p, m;\n.reg .b16 l, h, j, r, z;\n"
        "mov.b32 {l, h}, %2;\nabs.f16 j, h;\nmov.b32 {r, z}, %3;\n"
        "setp.lt.s32 m, %2, 0;\nsetp.eq.and.u32 m, %3, 0x3FFF, m;\n"
        "setp.gt.and.f16 p, r, j, !m;\nselp.b32 %1, %5, %4, p;\n@p add.u32 %0, %0, 4;\n}"
        : "+r"(a), "=r"(next)
        : "r"(node), "r"(q), "r"(left), "r"(right));
  }
  return next;
}

// The three top nodes (words 1..3) of every tree, passed to the kernel by value: kernel
// parameters live in the constant bank, so the first two levels of every walk read their nodes
// through the constant cache and spend no shared-memory bandwidth, the resource that bounds the
// traversal (a warp reads the same tree in all lanes, so each lookup is one constant access).
// In two sizes: 24 KB of parameters make a launch 1 to 2 us longer than four.
template <int TREES>
struct QTop {
  uint32_t w[3 * TREES];
};
constexpr int kQTopFew = 320;
static_assert(kQTopFew < kQTopTrees, "two sizes");

__device__ __forceinline__ uint2 lds_u32x2(uint32_t a)
{
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}

// A categorical node is recognisable by its rank field, the largest there is (0x3FFF, or 0x3FFE in the
// image for doubled columns).  Only such nodes have a category set, in an array of its own behind the
// nodes, and only lanes on such a node fetch it: in a forest with one categorical test in sixteen
// that is less than half a shared-memory wavefront per visit, against one and more for nodes that
// carry their set along (5000 depth-6 trees, 8 of 128 features categorical).
template <uint32_t OFF>
__device__ __forceinline__ uint32_t lds_if_categorical(uint32_t node, uint32_t a)
{
  // (the address register takes the set, so that a lane without one needs no other value for it)
  asm volatile(
    "{\n.reg .pred p;\nsetp.ge.s32 p, %1, 0x7FFC0000;\n@p ld.shared.u32 %0, [%0+%2];\n}"
    : "+r"(a)
    : "r"(node), "n"(OFF));
  return a;
}
__device__ __forceinline__ uint32_t shift_if_categorical(uint32_t node, uint32_t d, uint32_t set, uint32_t code)
{
  static_assert(((Q_MAX_RANK_FIELD - 1u) << Q_RANK_SHIFT) == 0x7FFC0000u, "the constant below");
  asm("{\n.reg .pred p;\nsetp.ge.s32 p, %1, 0x7FFC0000;\n@p shf.l.clamp.b32 %0, %0, %2, %3;\n}"
      : "+r"(d)
      : "r"(node), "r"(set), "r"(code));
  return d;
}

// DEPTH > 0 fixes the tree depth at compile time (the level loop is fully unrolled); DEPTH == 0
// reads it from the forest.
// HEAP: the image is in heap order (words 2i and 2i + 1 of a tree's block are the children of word i); a
// test is one signed subtraction whose sign goes into the heap index with one funnel shift.  Otherwise it is
// in walking order, which pays where levels are constants (q_walk_order()): with the depth read at run time two
// places have to be worked out per level, and the same kernels took 1.15 to 1.4 of the time in heap order (300
// depth-6 trees x 50 features, fp64, 150,000 rows: 181 us against 141; 100 depth-11 trees, fp32: 161 against 119).
// CAT (heap order): forests with categorical tests.  A category set takes part in the subtraction by a shift;
// with compares and predicates it took as many instructions in walking order, and a longer way from the
// rank to the next node (5000 depth-6 trees, 150,000 rows: 1894 us against 1871).
// TOPC: the first two levels take their nodes from `top`.
// PAIR: the walk for launch shapes that shared memory keeps small (few warps, few trees in
// flight), where the latency of one step, not the shared-memory pipe, is the limit: both children
// of the current node are requested together
// with the row's rank, before the test is decided, so the next node is already there when the
// test is known; a step costs one shared-memory latency instead of two, and one more wavefront.
// LEAFG: the stages hold only the test nodes of the trees and a walk fetches its leaf payload from
// the forest image in global memory (L2).  Deep trees are half payloads (4 KB of 8 KB at depth
// 10); where shared memory next to the row tile holds only a dozen whole trees, leaving the
// payloads out doubles the walks in flight, which is what such shapes are bound by.  The payload
// fetch of a sub-batch is consumed one sub-batch later, behind the next walk.  Nodes and payloads are
// arrays of their own: a stage is one copy (a copy per tree was 20 us slower with 2000 trees of depth 10 on
// 200,000 rows), and the payloads of ways that part late are neighbours (180 us: in the order of the
// walk, whose last steps are the longest, every row fetched another sector).
template <typename T, int MODE, int NT, int DEPTH, bool CAT, bool HEAP, bool TOPC, bool PAIR, bool LEAFG>
struct DenseQWalker {
  using TR = Traits<T>;
  // Walk the warp's 32 rows through all trees.  A stage of the ring holds K sub-batches of G * NT
  // trees; the warp waits once per stage and walks its NT trees of every sub-batch.
  // MISSING says what a missing value costs: nothing (NAN_NONE: there is none, or NAN_COLUMNS: the
  // doubled columns of the tile take care of it; only the top nodes, which exist once, pick the
  // column by their direction) or a comparison per test (NAN_TESTED).
  template <int MISSING>
  static __device__ __forceinline__ bool walk(const PredictParams& p, int G, int S, int K, int g,
                                              int r, int64_t row, int lane, uint32_t bars,
                                              uint32_t stages, uint32_t stage_bytes,
                                              uint32_t row_addr, uint32_t stride_b, T* acc_group,
                                              int R, RingPos& pos, Running<T>& run,
                                              const uint32_t* top, int b_begin, int b_end,
                                              uint32_t copy_off)
  {
    constexpr bool NANS = MISSING == NAN_TESTED;
    static_assert(HEAP || (!CAT && sizeof(T) == 4 && (DEPTH >= 4 || PAIR)), "forests in walking order");
    static_assert(!TOPC || (DEPTH >= 2 && !HEAP), "top nodes need two levels, and are in walking order");
    static_assert(!PAIR || (!CAT && !TOPC && MODE == MODE_SCALAR && sizeof(T) == 4),
                  "the child-pair walk exists for fp32 scalar leaves without categorical tests");
    static_assert(!LEAFG || (!HEAP && !PAIR && MODE == MODE_SCALAR && sizeof(T) == 4),
                  "payloads outside the stages exist for fp32 scalar leaves without categorical tests");
    const ForestView& f    = p.f;
    const int D            = DEPTH > 0 ? DEPTH : f.dense_depth;
    // HEAP: from a node to its category set
    const uint32_t sets_at = 4u << D;
    // bytes between two trees of a stage
    constexpr uint32_t kStride = LEAFG ? walk_nodes_stride(DEPTH)
                                       : static_cast<uint32_t>(walk_tree_stride(DEPTH, TR::ES));
    constexpr bool known_stride = MODE == MODE_SCALAR && DEPTH > 0 && !HEAP;
    const uint32_t tstride      = known_stride ? kStride : static_cast<uint32_t>(f.q_tree_stride);
    // bytes per leaf payload: the element size, except where vector leaves sit in the tree block
    const uint32_t lbytes  = MODE == MODE_SCALAR ? TR::ES : static_cast<uint32_t>(f.q_leaf_bytes);
    const bool inline_vec  = MODE != MODE_SCALAR && lbytes > TR::ES;
    // from the start of a tree to its payloads
    const uint32_t leaves_at = HEAP ? (CAT ? 8u : 4u) << D : 4u * walk_leaves_at(D, lbytes);
    // walking order: words from one block of a tree to the next, where it has blocks
    const uint32_t pitch = HEAP ? 0u : walk_pitch(D, !LEAFG && lbytes == 4u);
    const uint32_t fstride = stride_b >> Q_FEATURE_SHIFT;  // R / 2 <= 128: fits a byte
    const int per_sub      = G * NT;
    const int per_batch    = per_sub * K;
    const uint32_t mine    = static_cast<uint32_t>(g * NT) * tstride;  // this warp's trees in a sub-batch
    const uint32_t sub_b   = static_cast<uint32_t>(per_sub) * tstride;
    bool ok                = true;
    uint32_t seen          = 0u;  // what release_stage() cannot tell from the sums, folded

    // LEAFG: payloads requested by the previous sub-batch, not yet added
    uint32_t pend[NT] = {};
    int pend_first = 0, pend_n = 0;
    auto take_pending = [&]() {
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        if (k < pend_n) take_leaf<T, MODE>(p, pend_first + k, pend[k], 0u, acc_group, R, r, row, run);
      }
      pend_n = 0;
    };
    // One sub-batch: NT trees side by side.  FULL means all NT slots hold live trees, which lets
    // the compiler drop every per-slot guard.
    auto sub_batch = [&](auto full_tag, uint32_t base0, int first, int n_act) {
      constexpr bool FULL = decltype(full_tag)::value;
      // Where the size of a tree is a constant its slot is part of the loads' immediate offsets (headline
      // forest, 1.5 M rows: 3980 -> 3945 us in heap order).
      constexpr uint32_t TS = FULL && known_stride ? kStride : 0u;
      using Each = std::make_integer_sequence<int, NT>;
      // slots past the end of the forest repeat the last live tree; results are dropped
      auto slot = [&](int k) { return static_cast<uint32_t>(FULL ? k : min(k, n_act - 1)) * tstride; };
      auto start = [&](int k) { return TS ? base0 : base0 + slot(k); };
      // walking order: start of the tree's block (the first one's, TS > 0) + 4 * place in the level;
      // heap order: address of the node, its heap index, and start of the block
      uint32_t a[NT], idx[NT], base[NT];
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        a[k] = start(k);
        if (HEAP) {
          base[k] = a[k];
          idx[k]  = 1u;
          a[k] += 4u;
        }
      }
      // the NT walks are independent: all node loads are issued first, then all rank loads,
      // so that their shared-memory latencies overlap inside one warp.
      // heap_level(): a level in heap order.  The sign bit of d[k] is the step to the right.
      auto heap_test = [&](const uint32_t(&node)[NT], uint32_t(&d)[NT]) {
        uint32_t q[NT], bits[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          // (see step())
          q[k] = lds_u16(__dp2a_lo(node[k], fstride, row_addr));
        }
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (CAT) bits[k] = lds_if_categorical<DEPTH ? 4u << DEPTH : 0u>(node[k], a[k] + (DEPTH ? 0u : sets_at));
        }
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          // rank j in the high half: x < T[j] <=> rank(x) <= j, so right <=> j - rank < 0
          d[k] = rank_diff(node[k], q[k]);
          // the code of a categorical value is its category and the node's set is stored
          // bit-reversed: the clamped funnel shift by the code moves the category's bit to the sign
          // position, and leaves d for every code of 32 and above (no category, NaN), which the
          // large rank of a categorical node has made non-negative, or right for a missing value
          // of a doubled column.  Predicated: the walk has no data-dependent branch.
          if (CAT) d[k] = shift_if_categorical(node[k], d[k], bits[k], q[k]);
          // the missing-goes-right flag sits 15 bits below the sign.  (Both forms compute the same; each
          // kernel family keeps the one it was measured fastest with: the two walks of a kernel share
          // its register allocation.)
          if (NANS && CAT && q[k] == Q_NAN_CODE) d[k] = node[k] << 15;
          if (NANS && !CAT && q[k] == Q_NAN_CODE) d[k] = (node[k] & Q_DEFAULT_RIGHT) ? 0x80000000u : 0u;
        }
      };
      auto heap_level = [&]() {
        uint32_t node[NT], d[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) node[k] = lds_u32(a[k]);
        heap_test(node, d);
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          // heap index 2i + right in one funnel shift: (i << 1) | (d >> 31)
          idx[k] = __funnelshift_l(d[k], idx[k], 1);
          a[k]   = idx[k] * 4u + base[k];
        }
      };
      // step(): the rows' ranks against NT nodes in walking order.
      auto step = [&](const uint32_t(&node)[NT], auto from_param, auto&& move) {
        constexpr bool PARAM = decltype(from_param)::value;
        uint32_t q[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          uint32_t from = row_addr;
          // (top nodes from the parameter block exist once and pick the column by their direction)
          if (PARAM && MISSING == NAN_COLUMNS && static_cast<int32_t>(node[k]) < 0) from += copy_off;
          // the low half of a node is feature * 4: one dot-product instruction (low half x byte 0
          // of fstride, high half x byte 1 = 0) turns it into the address of the row's rank of
          // that feature
          q[k] = lds_u16(__dp2a_lo(node[k], fstride, from));
        }
#pragma unroll
        for (int k = 0; k < NT; ++k) move(k, node[k], q[k]);
      };
      // `lvl`: a constant
      auto level = [&](auto lvl) {
        constexpr int LVL = decltype(lvl)::value;
        uint32_t node[NT];
        for_each_constant(
          [&](auto kc) {
            constexpr int k = decltype(kc)::value;
            node[k] = lds_u32_at<k * TS + 4u * walk_level_at(DEPTH, LVL)>(a[k]);
          },
          Each{});
        step(node, std::false_type{}, [&](int k, uint32_t n, uint32_t q) {
          walk_step<NANS>(a[k], n, q, 4u * walk_step_words(DEPTH, LVL));
        });
      };
      if constexpr (PAIR) {
        uint32_t node[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) node[k] = lds_u32(HEAP ? a[k] : a[k] + 4u);  // the root
#pragma unroll 2
        for (int lvl = 0; lvl < D; ++lvl) {
          // both children; below the last level these are the two leaf payloads (4-byte payloads go on
          // behind the nodes)
          uint32_t left[NT], right[NT];
          if constexpr (HEAP) {
            uint32_t d[NT];
#pragma unroll
            for (int k = 0; k < NT; ++k) {
              const uint2 pair = lds_u32x2(base[k] + idx[k] * 8u);
              left[k]          = pair.x;
              right[k]         = pair.y;
            }
            heap_test(node, d);
#pragma unroll
            for (int k = 0; k < NT; ++k) {
              idx[k]  = __funnelshift_l(d[k], idx[k], 1);
              node[k] = static_cast<int32_t>(d[k]) < 0 ? right[k] : left[k];
            }
          } else {
            uint32_t inc      = 4u * walk_step_words(D, lvl);
            const uint32_t at = lvl + 1 < D ? 4u * walk_level_at(D, lvl + 1) : leaves_at;
            if (walk_blocks(D) && lvl == 4) {
              inc *= pitch;
#pragma unroll
              for (int k = 0; k < NT; ++k) a[k] = a[k] * pitch + start(k) * (1u - pitch);
            }
#pragma unroll
            for (int k = 0; k < NT; ++k) {
              left[k]  = lds_u32(a[k] + at);
              right[k] = lds_u32(a[k] + at + inc);
            }
            step(node, std::false_type{}, [&](int k, uint32_t n, uint32_t q) {
              const uint32_t before = a[k];
              walk_step<NANS>(a[k], n, q, inc);
              node[k] = a[k] != before ? right[k] : left[k];
            });
          }
        }
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (FULL || k < n_act)
            take_leaf<T, MODE>(p, first + k, node[k], 0u, acc_group, R, r, row, run);
        }
        return;
      }
      if constexpr (TOPC) {
        // root and children from the constant bank: the same words in every lane
        uint32_t n1[NT], n2[NT], n3[NT], node[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          const int t = 3 * (first + (FULL ? k : min(k, n_act - 1)));
          n1[k]       = top[t];
          n2[k]       = top[t + 1];
          n3[k]       = top[t + 2];
        }
        step(n1, std::true_type{},
             [&](int k, uint32_t n, uint32_t q) { node[k] = root_step<NANS>(a[k], n, q, n2[k], n3[k]); });
        step(node, std::true_type{}, [&](int k, uint32_t n, uint32_t q) { walk_step<NANS>(a[k], n, q, 8u); });
      }
      [[maybe_unused]] uint32_t from[NT];  // blocks: where the walks were before they went into them
      if constexpr (HEAP) {
        if (DEPTH > 0) {
#pragma unroll
          for (int lvl = 0; lvl < DEPTH; ++lvl) heap_level();
        } else {
#pragma unroll 4
          for (int lvl = 0; lvl < D; ++lvl) heap_level();
        }
        // fp64: the payload's address instead of the places it follows from (registers are short)
        if (TR::ES == 8) {
#pragma unroll
          for (int k = 0; k < NT; ++k) a[k] = base[k] + leaves_at + (idx[k] - (1u << D)) * lbytes;
        }
      } else {
        constexpr int SKIP = TOPC ? 2 : 0;
        for_each_constant(
          [&](auto lc) {
            constexpr int L = decltype(lc)::value + SKIP;
            if constexpr (walk_blocks(DEPTH) && L == 5) {
#pragma unroll
              for (int k = 0; k < NT; ++k) {
                from[k] = a[k];
                a[k]    = a[k] * pitch + start(k) * (1u - pitch);
              }
            }
            level(std::integral_constant<int, L>{});
          },
          std::make_integer_sequence<int, DEPTH - SKIP>{});
        if constexpr (walk_blocks(DEPTH) && MODE != MODE_SCALAR) {
          // from the last place to the payload (walk_payload_number(): a block has a word less than payloads); at
          // once, so that `from` is not needed any longer (with vector leaves registers were spilled)
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            a[k] = lbytes == 4u ? a[k] + leaves_at
                                : start(k) + leaves_at + (a[k] + from[k] - 2u * start(k)) * (lbytes >> 2);
          }
        }
      }
      // address of the payload, of `bytes` bytes, that walk k ended on
      auto payload_at = [&](int k, uint32_t bytes) {
        // (4-byte payloads go on behind the nodes in heap order, too)
        if constexpr (HEAP && (TR::ES == 8 || (MODE == MODE_SCALAR && !CAT))) return a[k];
        if constexpr (HEAP) return base[k] + leaves_at + (idx[k] - (1u << D)) * bytes;
        if constexpr (walk_blocks(DEPTH) && MODE != MODE_SCALAR) return a[k];
        return bytes == 4u ? a[k] + k * TS + leaves_at : start(k) + leaves_at + (a[k] - start(k)) * (bytes >> 2);
      };
      auto leaf_at = [&](int k) { return payload_at(k, lbytes); };
      // scalar leaves of a multi-class forest: trees are stored class by class, so when the
      // first and the last tree of the sub-batch feed the class of the running sum, all do
      bool same_class = false;
      if (MODE == MODE_SCALAR && CAT) {
        same_class = f.n_outputs == 1 ||
                     (__ldg(f.tree_class + first) == run.cls &&
                      __ldg(f.tree_class + first + n_act - 1) == run.cls);
      }
      if constexpr (LEAFG) {
        // add the payloads that the previous sub-batch requested (they arrived during this
        // walk), then request this sub-batch's; nothing touches them until the next one is done
        take_pending();
        const unsigned char* far = static_cast<const unsigned char*>(f.q_nodes) +
                                   static_cast<size_t>(f.n_trees) * walk_tree_stride(DEPTH, TR::ES);
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          // walk_far_number() of block and place in it
          const uint32_t block = from[k] - start(k), place = a[k] - start(k) - block * pitch;
          const uint32_t at    = (block << (DEPTH - 5)) + ((place >> (DEPTH - 8) | place << 3) & ((4u << (DEPTH - 5)) - 4u));
          const int tree       = first + (FULL ? k : min(k, n_act - 1));
          seen ^= at;
          pend[k] = __ldg(reinterpret_cast<const uint32_t*>(
            far + (static_cast<size_t>(tree) << (DEPTH + 2)) + at));
        }
        pend_first = first;
        pend_n     = FULL ? NT : n_act;
        return;
      }
      if (MODE >= MODE_PERTREE) {
        // One output per (row, tree).  The payload slot holds what is reported: the leaf value,
        // or the leaf id when the CTA streams the image made for that (MODE_LEAFID).  With four
        // live trees that are also the caller's trees first..first+3, a row's four outputs are
        // contiguous and leave as 16-byte stores, or, where the rows are not aligned for that,
        // four lanes at a time (store_quads): scalar 4-byte stores at a stride of a whole output
        // row cost one sector request each and bound these predictions otherwise.
        typename TR::Val val[NT];
#pragma unroll
        for (int k = 0; k < NT; ++k) val[k] = TR::ld_val(leaf_at(k));
        const bool scalar_out = MODE == MODE_LEAFID || f.leaf_vector_len <= 1;
        const bool quad = FULL && NT % 4 == 0 && scalar_out && f.q_trees_in_order != 0;
        using Out = std::conditional_t<MODE == MODE_LEAFID, uint32_t, typename TR::Val>;
        Out* out  = static_cast<Out*>(p.out);
        if (quad && (f.n_trees & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0) {
          if (row < p.n_rows) {
            Out* dst = out + row * f.n_trees + first;
#pragma unroll
            for (int k = 0; k + 3 < NT; k += 4) {
              if constexpr (sizeof(Out) == 4) {
                *reinterpret_cast<uint4*>(dst + k) = make_uint4(TR::low32(val[k]), TR::low32(val[k + 1]),
                                                                TR::low32(val[k + 2]), TR::low32(val[k + 3]));
              } else {
                *reinterpret_cast<ulonglong2*>(dst + k)     = make_ulonglong2(val[k], val[k + 1]);
                *reinterpret_cast<ulonglong2*>(dst + k + 2) = make_ulonglong2(val[k + 2], val[k + 3]);
              }
            }
          }
        } else if (quad) {
#pragma unroll
          for (int k = 0; k + 3 < NT; k += 4)
            store_quads<Out>(out, f.n_trees, row, p.n_rows, first + k, static_cast<Out>(val[k]),
                             static_cast<Out>(val[k + 1]), static_cast<Out>(val[k + 2]),
                             static_cast<Out>(val[k + 3]));
        } else {
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            if (FULL || k < n_act) {
              if (MODE == MODE_LEAFID) {
                if (row < p.n_rows) {
                  const int orig = __ldg(f.tree_orig + first + k);
                  static_cast<uint32_t*>(p.out)[row * f.n_trees + orig] = TR::low32(val[k]);
                }
              } else if (inline_vec) {
                // per-tree outputs of vector leaves that sit in the tree block
                if (row < p.n_rows) {
                  const int orig = __ldg(f.tree_orig + first + k);
                  T* out = static_cast<T*>(p.out) + (row * f.n_trees + orig) * f.n_outputs;
                  for (int c = 0; c < f.n_outputs; ++c) out[c] = TR::ld_real(leaf_at(k) + c * TR::ES);
                }
              } else {
                take_leaf<T, MODE>(p, first + k, val[k], 0u, acc_group, R, r, row, run);
              }
            }
          }
        }
      } else if (MODE == MODE_VECTOR && inline_vec && f.n_outputs == 2 && sizeof(T) == 4) {
        // two classes, the common random-forest classifier: one 8-byte load per leaf
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (FULL || k < n_act) {
            const uint2 v = lds_u32x2(payload_at(k, 8u));
            run.v[0] += static_cast<T>(__uint_as_float(v.x));
            run.v[1] += static_cast<T>(__uint_as_float(v.y));
          }
        }
      } else if (TR::ES == 8 && MODE == MODE_VECTOR && inline_vec) {
        // (the same as below: fp64 kernels spill less this way, fp32 ones the other way)
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (FULL || k < n_act) {
            const uint32_t leaf_a = leaf_at(k);
#pragma unroll
            for (int c = 0; c < kRegClasses; ++c) {
              if (c < f.n_outputs) run.v[c] += TR::ld_real(leaf_a + c * TR::ES);
            }
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          if (FULL || k < n_act) {
            const uint32_t leaf_a = leaf_at(k);
            if (TR::ES == 4 && MODE == MODE_VECTOR && inline_vec) {
              // the leaf's vector sits in the tree block: one sum per output, in registers
#pragma unroll
              for (int c = 0; c < kRegClasses; ++c) {
                if (c < f.n_outputs) run.v[c] += TR::ld_real(leaf_a + c * TR::ES);
              }
              continue;
            }
            const typename TR::Val payload = TR::ld_val(leaf_a);
            if (MODE == MODE_VECTOR) seen ^= TR::low32(payload);
            if (MODE == MODE_SCALAR && same_class) {
              run.sum += TR::as_real(payload);
            } else {
              take_leaf<T, MODE>(p, first + k, payload, 0u, acc_group, R, r, row, run);
            }
          }
        }
      }
    };

    for (int b = b_begin; b < b_end; ++b) {
      const uint32_t s = pos.stage;
      if (ok) ok = mbar_wait(bars + 8u * s, pos.phase);
      if (ok) {
        uint32_t base0 = stages + s * stage_bytes + mine;
        int first      = b * per_batch + g * NT;  // first tree of this warp inside the stage
        for (int kk = 0; kk < K; ++kk, base0 += sub_b, first += per_sub) {
          const int n_act = f.n_trees - first;
          if (n_act >= NT) {
            sub_batch(std::true_type{}, base0, first, NT);
          } else if (n_act > 0) {
            sub_batch(std::false_type{}, base0, first, n_act);
          } else {
            break;
          }
        }
      }
      const uint32_t empty = bars + 8u * (kMaxStages + s);
      if (MODE >= MODE_PERTREE) {
        release_stored_stage(empty, lane);
      } else {
        bool read = seen != 0xffffffffu;
        if ((MODE == MODE_SCALAR && !LEAFG) || (MODE == MODE_VECTOR && inline_vec))
          read = sums_known<T, MODE>(run);
        release_stage(empty, lane, read, p.zero);
      }
      pos.advance(S);
    }
    if constexpr (LEAFG) take_pending();
    return ok;
  }
};

// Which (row tile, tree batches) a CTA walks.  The row tiles of a launch, each with all its tree
// batches, form one line of units that is cut into equal parts, one per CTA: a CTA walks the end
// of one tile, some whole tiles, and the beginning of another, so that a launch takes the time of
// its average CTA however few tiles there are (157 tiles on 148 SMs used to take two rounds, the
// second almost empty).  Tiles that are cut leave partial sums (finish_shared_tile).  When sums
// cannot be exchanged (QArgs::partial is null and outputs are reduced) only whole tiles are dealt.
struct QSegments {
  int32_t tile, begin;           // current tile, and the first tree batch of the segment
  int32_t last_tile, last_end;   // the CTA's part ends before batch last_end of tile last_tile
  int32_t n_batches;
  __device__ __forceinline__ QSegments(int64_t n_tiles, int nb, bool cut) : n_batches(nb)
  {
    int64_t u0 = n_tiles * blockIdx.x / gridDim.x, u1 = n_tiles * (blockIdx.x + 1) / gridDim.x;
    if (cut) {
      const int64_t units = n_tiles * nb;
      u0        = units * blockIdx.x / gridDim.x;
      u1        = units * (blockIdx.x + 1) / gridDim.x;
      tile      = static_cast<int32_t>(u0 / nb);
      begin     = static_cast<int32_t>(u0 - static_cast<int64_t>(tile) * nb);
      last_tile = static_cast<int32_t>(u1 / nb);
      last_end  = static_cast<int32_t>(u1 - static_cast<int64_t>(last_tile) * nb);
    } else {
      tile      = static_cast<int32_t>(u0);
      last_tile = static_cast<int32_t>(u1);
      begin = last_end = 0;
    }
  }
  __device__ __forceinline__ int32_t end() const { return tile < last_tile ? n_batches : last_end; }
  __device__ __forceinline__ bool live() const
  {
    return tile < last_tile || (tile == last_tile && begin < last_end);
  }
  // does another segment follow this one?
  __device__ __forceinline__ bool more() const
  {
    return tile + 1 < last_tile || (tile + 1 == last_tile && last_end > 0);
  }
  __device__ __forceinline__ bool whole() const { return begin == 0 && tile < last_tile; }
  __device__ __forceinline__ void next()
  {
    ++tile;
    begin = 0;
  }
};

// A tile that several CTAs share.  The CTA leaves its sums in global memory; the one that arrives
// last adds all of them in CTA order (a fixed order whoever is last) and finishes the rows.
// Called by the consumer threads, `sums` = the CTA's accumulators [group][output][row].
template <typename T>
__device__ __forceinline__ void finish_shared_tile(const PredictParams& p, const QArgs& q,
                                                   const QSegments& seg, bool first_segment,
                                                   T* sums, volatile int* last_flag, int n_ct,
                                                   int64_t n_tiles)
{
  const int NC    = p.f.n_outputs;
  const int R     = q.R;
  T* partial      = static_cast<T*>(q.partial);
  T* mine         = partial + static_cast<int64_t>(2 * blockIdx.x + (first_segment ? 0 : 1)) * NC * R;
  for (int i = threadIdx.x; i < NC * R; i += n_ct) {
    T s = sums[i];
    for (int g = 1; g < q.G; ++g) s += sums[g * NC * R + i];
    __stcg(mine + i, s);
  }
  __threadfence();
  consumer_sync(n_ct);
  if (threadIdx.x == 0) {
    const int n    = seg.end() - seg.begin;
    const int seen = atomicAdd(q.arrived + seg.tile, n);
    __threadfence();
    *last_flag = seen + n == seg.n_batches;
  }
  consumer_sync(n_ct);
  if (*last_flag == 0) return;
  // CTAs that share the tile: those whose units overlap [tile * n_batches, (tile + 1) * n_batches)
  const int64_t units = n_tiles * seg.n_batches;
  const int64_t u     = static_cast<int64_t>(seg.tile) * seg.n_batches;
  const int lo        = static_cast<int>(((u + 1) * gridDim.x - 1) / units);
  const int hi        = static_cast<int>(((u + seg.n_batches) * gridDim.x - 1) / units);
  // the tile is the first segment of every one of them but, perhaps, the first
  const int lo_slot = units * lo / gridDim.x >= u ? 2 * lo : 2 * lo + 1;
  const int64_t stride = static_cast<int64_t>(2) * NC * R;  // between the first segments of two CTAs
  for (int i = threadIdx.x; i < NC * R; i += n_ct) {
    T s           = __ldcg(partial + static_cast<int64_t>(lo_slot) * NC * R + i);
    const T* from = partial + stride * (lo + 1) + i;
    for (int k0 = lo + 1; k0 <= hi; k0 += 8, from += 8 * stride) {
      T part[8];  // loads in flight together
#pragma unroll
      for (int k = 0; k < 8; ++k) part[k] = k0 + k <= hi ? __ldcg(from + k * stride) : T(0);
#pragma unroll
      for (int k = 0; k < 8; ++k) s += part[k];
    }
    sums[i] = s;
  }
  consumer_sync(n_ct);
  if (threadIdx.x < R)
    finish_row<T>(p, sums, R, 1, threadIdx.x, static_cast<int64_t>(seg.tile) * R + threadIdx.x);
}

template <typename T, int MODE, int NT, int DEPTH, bool CAT, bool HEAP, bool TOPC, bool PAIR = false,
          bool LEAFG = false>
__device__ __forceinline__ void dense_q_body(const PredictParams& p, const QArgs& q,
                                             const uint32_t* top)
{
  using TR = Traits<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  const ForestView& f = p.f;
  const int R         = q.R;
  const int G         = q.G;
  const int S         = q.S;
  const int K         = q.K;
  const int F         = f.n_features;
  const int NC        = f.n_outputs;
  const int rw        = R >> 5;
  const int n_cw      = rw * G;
  const int n_ct      = n_cw * 32;
  const int warp      = threadIdx.x >> 5;
  const int lane      = threadIdx.x & 31;
  constexpr bool REDUCE = MODE <= MODE_VECTOR;

  const uint32_t stride_b    = R * 2u;  // bytes between features in the tile
  const uint32_t tile_bytes  = static_cast<uint32_t>(F) * stride_b;  // multiple of 64
  const uint32_t acc_bytes   = REDUCE ? static_cast<uint32_t>(align16(static_cast<size_t>(G) * NC * R * TR::ES)) : 0u;
  unsigned char* tile_ptr    = smem + kQBarBytes;
  const uint32_t tile_room   = tile_bytes * (q.nan_columns ? 2u : 1u);  // per buffer
  unsigned char* acc_ptr     = tile_ptr + q.tile_bufs * tile_room;
  volatile int* last_flag    = reinterpret_cast<volatile int*>(acc_ptr + q.acc_bufs * acc_bytes);
  unsigned char* stage_ptr   = acc_ptr + q.acc_bufs * acc_bytes + 16;
  const uint32_t bars        = smem_addr(smem);
  const uint32_t tile        = smem_addr(tile_ptr);
  const uint32_t stages      = smem_addr(stage_ptr);
  // trees in the image and in a stage: whole, or (LEAFG) only their test nodes
  const uint32_t tstride     = LEAFG ? walk_nodes_stride(DEPTH) : static_cast<uint32_t>(f.q_tree_stride);
  const int per_batch        = G * NT * K;
  const uint32_t stage_bytes = per_batch * tstride;
  const int n_batches        = (f.n_trees + per_batch - 1) / per_batch;
  const int64_t n_tiles      = (p.n_rows + R - 1) / R;
  const uint32_t bar_tfull   = bars + 8u * kBarTileFull;
  const uint32_t bar_tempty  = bars + 8u * kBarTileEmpty;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bars + 8u * s, 1);
      mbar_init(bars + 8u * (kMaxStages + s), n_cw);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_tfull + 8u * i, 1);
      mbar_init(bar_tempty + 8u * i, n_cw);
    }
    mbar_fence_init();
  }
  __syncthreads();
  grid_release();
  QSegments seg(n_tiles, n_batches, !REDUCE || q.partial != nullptr);

  // Does the tile hold a missing value?  (asked by whole warps)  Read past the L1: the pre-pass may have
  // written the flags while this kernel was already on the SM, next to the traversal of the call
  // before it, which read the flags of its own rows at the same addresses.
  auto has_nan = [&](int t) {
    uint32_t bits = 0;
    for (int i = lane; i < q.flag_words; i += 32)
      bits |= __ldcg(q.flags + static_cast<int64_t>(t) * q.flag_words + i);
    return __any_sync(0xffffffffu, bits != 0u);
  };

  if (warp == n_cw) {
    // ---- producer: row tiles, and the tree batches of each of them -----------------------------
    // predictions that report leaves stream the image whose payload slots hold the leaf ids
    const unsigned char* image = static_cast<const unsigned char*>(MODE == MODE_LEAFID ? f.q_nodes_ids : f.q_nodes);
    const unsigned char* image_nan = static_cast<const unsigned char*>(f.q_nodes_nan);
    if (LEAFG) {  // the nodes without payloads
      const size_t trees = static_cast<size_t>(f.n_trees) * walk_tree_stride(DEPTH, 4);
      image += trees + (static_cast<size_t>(f.n_trees) << (DEPTH + 2));
      image_nan += trees;
    }
    const unsigned char* qsrc = reinterpret_cast<const unsigned char*>(q.Q);
    RingPos pos;
    bool primed = false;  // every stage has been filled once
    RingPos tpos;         // buffer of the next tile to request, and the parity of its use
    bool tprimed = false;
    auto request_tile = [&](int t) {
      // a buffer is free once every consumer warp has left the trees of the tile it held
      if (tprimed && !mbar_wait(bar_tempty + 8u * tpos.stage, tpos.phase ^ 1u)) {
        report_status(p.status, 3);
        return false;
      }
      const uint32_t bar = bar_tfull + 8u * tpos.stage;
      mbar_expect_tx(bar, tile_bytes);
      bulk_copy_g2s(tile + tpos.stage * tile_room, qsrc + static_cast<size_t>(t) * tile_bytes,
                    tile_bytes, bar);
      tpos.advance(q.tile_bufs);
      if (tpos.stage == 0) tprimed = true;
      return true;
    };
    grid_wait();
    bool going = seg.live();
    if (lane == 0 && going) going = request_tile(seg.tile);
    for (; seg.live(); seg.next()) {
      const bool nan_image = q.nan_columns && has_nan(seg.tile);
      if (lane != 0 || !going) continue;
      const unsigned char* src = nan_image ? image_nan : image;
      const bool more = seg.more();
      const int end   = seg.end();
      // with two buffers the next tile is requested once the ring is full of this tile's trees
      const int ask_at = q.tile_bufs == 2 ? min(end, seg.begin + S) - 1 : end - 1;
      for (int b = seg.begin; b < end && going; ++b) {
        const uint32_t s = pos.stage;
        if (primed && !mbar_wait(bars + 8u * (kMaxStages + s), pos.phase ^ 1u)) {
          report_status(p.status, 1);
          going = false;
          break;
        }
        const int first      = b * per_batch;
        const uint32_t bytes = min(per_batch, f.n_trees - first) * tstride;
        mbar_expect_tx(bars + 8u * s, bytes);
        bulk_copy_g2s(stages + s * stage_bytes, src + static_cast<size_t>(first) * tstride, bytes, bars + 8u * s);
        pos.advance(S);
        if (pos.stage == 0) primed = true;
        if (more && b == ask_at) going = request_tile(seg.tile + 1);
      }
    }
    return;
  }

  // ---- consumers ------------------------------------------------------------------------------
  const int g             = warp / rw;
  const int r             = (warp % rw) * 32 + lane;
  const uint32_t row_slot = tile + q_slot(r, R) * 2u;
  // sums that the walk keeps in registers to its end are stored, others are added to zeroed ones
  const bool stored       = MODE == MODE_SCALAR ? NC == 1 : NC <= kRegClasses;
  RingPos pos, tpos;
  int acc_set             = 0;
  int finisher            = 0;     // the tree group that finishes the rows of the tile
  bool first_segment      = true;
  bool ok                 = true;
  grid_wait();
  for (; seg.live(); seg.next()) {
    const int64_t row0 = static_cast<int64_t>(seg.tile) * R;
    T* acc             = reinterpret_cast<T*>(acc_ptr + acc_set * acc_bytes);
    T* acc_group       = acc + static_cast<size_t>(g) * NC * R;
    if (REDUCE && !stored) {
      for (int c = 0; c < NC; ++c) acc_group[c * R + r] = T(0);  // nobody else's
    }
    const bool nans = has_nan(seg.tile);
    if (ok) ok = mbar_wait(bar_tfull + 8u * tpos.stage, tpos.phase);
    Running<T> run{T(0), 0, {}};
    const uint32_t at_tile = tpos.stage * tile_room;
    if (nans && q.nan_columns) {
      // the second set of columns: missing values move from "right" to "left"
      for (uint32_t i = threadIdx.x * 16u; i < tile_bytes; i += n_ct * 16u) {
        uint4* from = reinterpret_cast<uint4*>(tile_ptr + at_tile + i);
        uint4 v     = *from;
        uint32_t* w = &v.x;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          w[k] |= __vcmpeq2(w[k], Q_NAN_CODE * 0x10001u) & Q_NAN_LEFT_BIT * 0x10001u;
        *reinterpret_cast<uint4*>(tile_ptr + at_tile + tile_bytes + i) = v;
      }
      consumer_sync(n_ct);
    }
    if (ok) {
      const uint32_t row_addr = row_slot + at_tile;
      auto go = [&](auto missing) {
        return DenseQWalker<T, MODE, NT, DEPTH, CAT, HEAP, TOPC, PAIR, LEAFG>::template walk<decltype(missing)::value>(
          p, G, S, K, g, r, row0 + r, lane, bars, stages, stage_bytes, row_addr, stride_b, acc_group, R,
          pos, run, top, seg.begin, seg.end(), tile_bytes);
      };
      if (nans && !q.nan_columns) {
        ok = go(std::integral_constant<int, NAN_TESTED>{});
      } else if (TOPC && nans) {
        ok = go(std::integral_constant<int, TOPC ? NAN_COLUMNS : NAN_NONE>{});
      } else {
        // (without top nodes in the parameter block the walk over doubled columns is the same one)
        ok = go(std::integral_constant<int, NAN_NONE>{});
      }
      if (!ok) report_status(p.status, 2);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_tempty + 8u * tpos.stage);
    tpos.advance(q.tile_bufs);
    if (REDUCE) {
      flush_running<T, MODE>(f, run, acc_group, R, r, stored);
      consumer_sync(n_ct);
      if (seg.whole()) {
        if (g == finisher) finish_row<T>(p, acc, R, G, r, row0 + r);
        if (++finisher == G) finisher = 0;
      } else {
        finish_shared_tile<T>(p, q, seg, first_segment, acc, last_flag, n_ct, n_tiles);
      }
      first_segment = false;
      // with two sets of accumulators the next meeting is early enough: by then the finishers
      // have read this set
      if (q.acc_bufs == 2) {
        acc_set ^= 1;
      } else {
        consumer_sync(n_ct);
      }
    }
  }
}


template <typename T, int MODE, int NT, int DEPTH, bool CAT>
__global__ void __launch_bounds__(NT > 4 ? 800 : 1024, 1)
dense_q_kernel(const __grid_constant__ PredictParams p, const __grid_constant__ QArgs q)
{
  dense_q_body<T, MODE, NT, DEPTH, CAT, CAT || DEPTH == 0, false>(p, q, nullptr);
}

// Same kernel with the child-pair walk (see DenseQWalker).
template <int NT, bool HEAP>
__global__ void __launch_bounds__(1024, 1)
dense_q_pair_kernel(const __grid_constant__ PredictParams p, const __grid_constant__ QArgs q)
{
  dense_q_body<float, MODE_SCALAR, NT, 0, false, HEAP, false, true>(p, q, nullptr);
}

// Same kernel with the leaf payloads left in global memory (see DenseQWalker), and the same with the top nodes
// in the parameter block.
template <int NT, int DEPTH>
__global__ void __launch_bounds__(1024, 1)
dense_q_leafg_kernel(const __grid_constant__ PredictParams p, const __grid_constant__ QArgs q)
{
  dense_q_body<float, MODE_SCALAR, NT, DEPTH, false, false, false, false, true>(p, q, nullptr);
}
template <int NT, int DEPTH, int TREES>
__global__ void __launch_bounds__(1024, 1)
dense_q_leafg_kernel(const __grid_constant__ PredictParams p, const __grid_constant__ QArgs q,
                     const __grid_constant__ QTop<TREES> top)
{
  dense_q_body<float, MODE_SCALAR, NT, DEPTH, false, false, true, false, true>(p, q, top.w);
}

// Same kernel with the top nodes of every tree in the parameter block.
template <typename T, int MODE, int NT, int DEPTH, int TREES>
__global__ void __launch_bounds__(NT > 4 ? 800 : 1024, 1)
dense_q_top_kernel(const __grid_constant__ PredictParams p, const __grid_constant__ QArgs q,
                   const __grid_constant__ QTop<TREES> top)
{
  dense_q_body<T, MODE, NT, DEPTH, false, false, true>(p, q, top.w);
}

// The three top nodes of every tree, which travel in the parameter block.
template <int TREES>
const QTop<TREES>& top_nodes(const QLaunch& L)
{
  static thread_local QTop<TREES> top;
  std::memcpy(top.w, L.p.q_top, static_cast<size_t>(L.p.f.n_trees) * 3 * sizeof(uint32_t));
  return top;
}

// Launch one instantiation of dense_q_top_kernel.
template <typename T, int MODE, int NT, int DEPTH>
int launch_q_top(const QLaunch& L, std::string& err)
{
  if (L.p.f.n_trees <= kQTopFew)
    return launch_split(L.shape(), err, dense_q_top_kernel<T, MODE, NT, DEPTH, kQTopFew>, L.p, L.q,
                        top_nodes<kQTopFew>(L));
  return launch_split(L.shape(), err, dense_q_top_kernel<T, MODE, NT, DEPTH, kQTopTrees>, L.p, L.q,
                      top_nodes<kQTopTrees>(L));
}
template <typename T, int MODE, int NT>
int launch_q_top_depth(const QLaunch& L, std::string& err)
{
  switch (L.p.f.dense_depth) {
    case 4: return launch_q_top<T, MODE, NT, 4>(L, err);
    case 5: return launch_q_top<T, MODE, NT, 5>(L, err);
    case 6: return launch_q_top<T, MODE, NT, 6>(L, err);
    case 7: return launch_q_top<T, MODE, NT, 7>(L, err);
    case 8: return launch_q_top<T, MODE, NT, 8>(L, err);
    case 9: return launch_q_top<T, MODE, NT, 9>(L, err);
    default: return launch_q_top<T, MODE, NT, 10>(L, err);
  }
}

// Launch one instantiation of dense_q_kernel.
template <typename T, int MODE, int NT, int DEPTH, bool CAT>
int launch_q(const QLaunch& L, std::string& err)
{
  auto k = dense_q_kernel<T, MODE, NT, DEPTH, CAT>;
  return launch_split(L.shape(), err, k, L.p, L.q);
}

// One case per output mode of the generic-depth kernels.
template <typename T, int NT, bool CAT>
int launch_q_modes(const QLaunch& L, int mode, std::string& err)
{
  switch (mode) {
    case MODE_SCALAR: return launch_q<T, MODE_SCALAR, NT, 0, CAT>(L, err);
    case MODE_VECTOR: return launch_q<T, MODE_VECTOR, NT, 0, CAT>(L, err);
    case MODE_PERTREE: return launch_q<T, MODE_PERTREE, NT, 0, CAT>(L, err);
    default: return launch_q<T, MODE_LEAFID, NT, 0, CAT>(L, err);
  }
}

}  // namespace
}  // namespace b2fil
