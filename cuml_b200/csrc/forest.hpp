// Packed-forest types shared by the host packer, the kernels and the C-ABI layer.
//
// Two device storages exist.
//
// DENSE: every tree is padded to a complete binary tree of depth D (the forest's maximum depth)
// and stored in heap order with 1-based indices: the root is node 1, the children of node i are
// 2i and 2i+1, level d is [2^d, 2^(d+1)), leaf slot j is heap index 2^D + j.  One tree is one
// contiguous block
//     [ 2^D test nodes (entry 0 unused) ][ 2^D leaf payloads ]
// so that a whole tree moves to shared memory with one bulk copy and no child index is stored.
//
// SPARSE: nodes keep an offset to their children and honour the requested node order
// (depth-first: left child adjacent, offset to the right child; breadth-first / layered:
// children adjacent to each other, offset to the left child).
//
// In both storages every numerical test is normalised at import to "x < threshold goes left" and
// every categorical test to "listed category goes right", by swapping children and moving
// thresholds to the next representable value where needed, so the kernels evaluate one operator.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <limits>
#include <string>
#include <vector>

#include "../../include/b2fil.h"

#ifdef __CUDACC__
#define B2FIL_HD __host__ __device__
#else
#define B2FIL_HD
#endif

namespace b2fil {

// ---- meta word of a test node -----------------------------------------------------------------
// bit 31: a missing value goes left; bit 30: categorical test; bit 29: leaf (sparse only).
// Dense nodes keep the feature index in bits 0..29.  The two top bits fall off the end of the
// 32-bit shared-memory address when the meta word is multiplied by a row stride that is a
// multiple of four bytes, so the hot loop never masks them.
constexpr uint32_t META_DEFAULT_LEFT = 0x80000000u;
constexpr uint32_t META_CATEGORICAL  = 0x40000000u;
constexpr uint32_t META_LEAF         = 0x20000000u;
constexpr uint32_t META_LOW29        = 0x1FFFFFFFu;

// ---- node records -----------------------------------------------------------------------------
struct DenseNodeF {  // 8 bytes
  uint32_t value;    // float threshold bits | inline category bitset | category pool offset
  uint32_t meta;     // flags | feature
};
struct DenseNodeD {  // 16 bytes
  uint64_t value;    // double threshold bits | bitset / pool offset in the low word
  uint32_t meta;
  uint32_t pad;
};
struct SparseNode8 {  // fp32, compact: feature and child offset share the low 29 meta bits
  uint32_t value;     // threshold | bitset | pool offset | leaf scalar | leaf-vector index
  uint32_t meta;      // flags | offset << feat_bits | feature
};
struct SparseNode16F {  // fp32, wide
  uint32_t value;
  uint32_t meta;  // flags | feature
  uint32_t offset;
  uint32_t pad;
};
struct SparseNode16D {  // fp64
  uint64_t value;
  uint32_t meta;  // flags | feature
  uint32_t offset;
};

// ---- rank quantisation of rows (dense storage without categorical tests) -----------------------
// For every feature the distinct thresholds of the forest are sorted: T[0] < T[1] < ...  The rank
// of a value, r(x) = #{i : T[i] <= x}, decides every test on that feature exactly:
//     x < T[j]  <=>  r(x) <= j.
// A pre-pass kernel turns each row into 16-bit ranks (NaN becomes 0x3FFF); the traversal kernel
// then reads 2-byte values and 4-byte nodes
//     bits 31..17: j (0x7FFF = never left)   bit 16: missing goes right
//     bits 15..2: feature                    bits 1..0: zero
// so a test is one signed subtraction: right <=> int(node) - (rank << 17) < 0 (the flag in bit 16
// is below the weight of one rank and cannot change the sign), and the low half is the feature
// times four: one 16-bit x 8-bit dot-product instruction scales it by a quarter of the byte
// stride between features and adds the row's address.
// Categorical features (every test on them is categorical, every listed category below 32) keep
// their place in the same scheme: the "rank" of a value is its category (Q_NO_CATEGORY when it is
// negative, fractional-truncated out of range or too large), and in such forests every node has
// a 32-bit category set (8 bytes {node, set} in the packed host image; before the upload
// split_category_sets moves the sets of a tree behind its nodes); a set bit sends the row right.  A
// categorical node is recognisable by j = Q_MAX_RANK_FIELD, and the walk loads the set only there;
// the low half of every node stays a clean feature * 4 for the address arithmetic.  The sets are stored bit-reversed (category c in bit 31 - c) and a categorical node
// carries the largest rank, so its rank comparison always says "left" and the walk can simply OR
// the two answers: sign(node - (code << 17)) | sign(set << code).
// Row tiles that hold missing values are walked with a second image of the nodes where room allows
// (q_nodes_nan).  Beside the tile's columns there is then a copy of each in which the NaN code has
// bit 14 set: 0x3FFF in the first set is a rank above every j (the test says "right"), 0x7FFF in
// the copy is -1 in the 15 bits of the subtraction (the test says "left"), and a node reads its
// feature from the set of its own missing direction (copies are numbered n_features and up).  So
// missing values cost no instruction in the walk.  Categorical nodes carry j = 0x3FFE there, below
// the NaN code and not below any other code.
// The rank is found through a per-feature bucket table: bucket(x) = clamp(int(fma(x, scale,
// offset)), 0, n_buckets-1) is monotone in x, lut[b] is the number of thresholds in buckets below
// b (all of them are <= x), thresholds of higher buckets are all > x, so the rank is lut[b] plus
// the number of thresholds <= x in a window of 2^steps - 1 entries starting at lut[b], found with
// `steps` branch-free halvings (2^steps exceeds the fullest bucket; the array ends with NaN
// padding, for which `T <= x` is false).
struct QFeature {      // host-side table of one feature
  uint32_t t_off;      // first threshold of the feature in PackedForest::q_thresholds
  uint32_t lut_off;    // first entry of the feature's bucket table in PackedForest::q_lut
  uint32_t m;          // number of distinct thresholds
  uint32_t n_buckets;
  uint32_t max_occupancy;  // thresholds in the fullest bucket
  uint32_t is_cat;         // categorical feature: no tables
  double scale;        // bucket(x) = fma(x, scale, offset) evaluated in the forest precision
  double offset;
};
// Device tables are grouped: a power-of-two run of GF consecutive features whose tables fit one
// CTA's shared memory forms a group, stored as one contiguous blob that the pre-pass pulls in with
// a single bulk copy:
//   [kQMaxGroupFeatures x QFeatRec][bucket tables (uint16)][thresholds + NaN padding]
// Both tables are interleaved across the group: entry k of the group's i-th feature sits at
// element k * GF + i, and every feature's columns are padded to the longest table of the group
// (zeros / NaN).  The lanes of a warp hold one feature each, so whatever entries they probe they
// read different shared-memory banks.
struct QFeatRec {      // 32 bytes
  uint32_t lut_off;    // byte offset of entry 0 from the start of the blob; entry k: + k * GF * 2
  uint32_t thr_off;    // same for the thresholds; entry k: + k * GF * sizeof(T)
  uint32_t nbm1;       // n_buckets - 1
  uint32_t is_cat;     // 1: the value's code is its category, no table lookup
  double scale, offset;
};
struct QGroup {        // 32 bytes
  uint32_t f_begin, f_end;
  uint32_t blob_off;   // byte offset of the group's blob in ForestView::q_blob (16-byte multiple)
  uint32_t blob_bytes; // 16-byte multiple
  uint32_t steps;      // halvings of the window search, shared by the group's features
  uint32_t pad[3];
};
// What one CTA of the pre-pass ranks: consecutive groups with at most kQMaxGroupFeatures features and
// one CTA's shared memory in all (a tail of 28 features is groups of 16, 8 and 4).  The CTA's threads
// are dealt evenly to `width` features (a power of two, the last few may be missing), its tables come
// with one bulk copy.
struct QBundle {        // 32 bytes
  uint32_t first_group, n_groups;
  uint32_t blob_off, blob_bytes;
  uint32_t width, n_features;
  uint32_t pad[2];
};
constexpr uint32_t Q_NAN_CODE      = 0x3FFFu;
constexpr uint32_t Q_NAN_LEFT_BIT  = 0x4000u;  // set in the NaN codes of the second set of columns
constexpr uint32_t Q_MAX_RANK      = 0x3FFEu;
constexpr uint32_t Q_NO_CATEGORY   = 0x3FFEu;
constexpr uint32_t Q_MAX_FEATURES  = 0x4000u;
constexpr uint32_t Q_FEATURE_FIELD = 0xFFFCu;  // feature << 2
constexpr uint32_t Q_FEATURE_SHIFT = 2;
constexpr uint32_t Q_DEFAULT_RIGHT = 0x10000u;  // missing values go right (stored in this sense: << 15 makes it the sign)
constexpr uint32_t Q_RANK_SHIFT    = 17;
constexpr uint32_t Q_NEVER_LEFT    = 0x7FFFu;  // j of a test that no value passes
constexpr uint32_t Q_MAX_RANK_FIELD = 0x3FFFu;  // j of a test that every code passes (categorical nodes)
// Kernels that have the depth as a constant (q_walk_order()) read this image in walking order (walk_order()
// before the upload):
//     bits 31..16: a half-precision float, the bits of j, whose sign says that missing values go left
//     bits 15..2: feature                    bits 1..0: zero
// Ranks below 0x4000 are the bits of small positive floats in the same order, so one half-precision compare
// takes both operands from the halves of the words they were loaded in: right <=> rank > |j|.  A missing
// value, 0x3FFF, is above every j, and in the copies of columns 0x7FFF, not a number, above none.
// The nodes of a level are together, and their places in it grow with the way: a step to the right on level l
// adds walk_step_words() to the place and a step to the left nothing, one predicated addition, and the
// level itself is the constant offset of the load.  (In heap order, 2 i + right, a step took two more
// instructions.)  The steps are 1, 2, 4, 8, 16 words, then 33, 66, ...: with powers of two all nodes below one of
// level 5 would be in one bank of shared memory, and rows that are together there are many (headline
// forest: 21 wavefronts per 32 rows and tree against 18 in heap order and this way).  So there is a hole
// behind every 32 words.
// Trees of depth 9 and 10, of which a stage holds few, have no room for holes.  Below level 5 they are 32 blocks, one
// per node of that level: a subtree in the same order without holes, at a distance that is odd, so that one place of
// different blocks is in different banks.  Going down to level 5 the place is multiplied by the distance, one
// more instruction per tree.  (Counted over random trees of depth 10 and rows, wavefronts per 32 rows and tree with
// the payload: 18.1 in heap order and with blocks, 19.5 with fewer holes, steps of 32, 65, 129, 258, ...)
// Payloads are in the same order.  In the blocks they are the last level where they have four bytes and are
// staged with the nodes; other payloads follow behind all nodes, numbered by block and place in the block.
B2FIL_HD inline constexpr bool walk_blocks(int depth) { return depth >= 9; }
B2FIL_HD inline constexpr uint32_t walk_step_words(int depth, int level)
{
  return level < 5 ? 1u << level : (walk_blocks(depth) ? 1u : 33u) << (level - 5);
}
// First word of a level, counted from the start of the tree (of its first block); word 0 is unused.
B2FIL_HD inline constexpr uint32_t walk_level_at(int depth, int level)
{
  if (walk_blocks(depth)) return level < 5 ? 1u << level : 31u + (1u << (level - 5));
  return level < 6 ? 1u << level : (33u << (level - 5)) - 2u;
}
// Words from one block to the next, with or without payloads as the last level.
B2FIL_HD inline constexpr uint32_t walk_pitch(int depth, bool payloads)
{
  return ((payloads ? 2u : 1u) << (depth - 5)) - 1u;
}
// First word of the payloads (8-byte ones are loaded at once).
B2FIL_HD inline constexpr uint32_t walk_leaves_at(int depth, size_t leaf_bytes)
{
  if (walk_blocks(depth)) return leaf_bytes == 4 ? walk_level_at(depth, depth) : 1u << depth;
  return (walk_level_at(depth, depth) + 1u) & ~1u;
}
// Bytes from one tree to the next.
B2FIL_HD inline constexpr size_t walk_tree_stride(int depth, size_t leaf_bytes)
{
  if (walk_blocks(depth)) return (4 + leaf_bytes) << depth;
  const size_t places = depth < 6 ? size_t(1) << depth : size_t(33) << (depth - 5);  // of the payloads
  return (4u * walk_leaves_at(depth, leaf_bytes) + places * leaf_bytes + 15) / 16 * 16;
}
// Where level `level` is reached by `way` (bit l: to the right on level l): a word of the tree ...
inline uint32_t walk_word(int depth, uint32_t pitch, int level, uint32_t way)
{
  uint32_t place = 0;
  for (int l = 0; l < level; ++l) {
    if (walk_blocks(depth) && l == 5) place *= pitch;
    if (way >> l & 1u) place += walk_step_words(depth, l);
  }
  if (walk_blocks(depth) && level == 5) place *= pitch;
  return walk_level_at(depth, level) + place;
}
// ... and the number of a payload that is not a level of the blocks.
inline uint32_t walk_payload_number(int depth, uint32_t way)
{
  return (way & 31u) << (depth - 5) | way >> 5;
}
// Payloads that stay in global memory (depth 9 and 10, four bytes each) are numbered so that the ways that part on one
// of the last three levels end next to each other: rows that are together deep in a tree then fetch the same sector.
inline uint32_t walk_far_number(int depth, uint32_t way)
{
  const uint32_t place = way >> 5;
  const int rest       = depth - 8;
  return (way & 31u) << (depth - 5) | place >> rest | (place & ((1u << rest) - 1u)) << 3;
}
// Bytes of such a tree's nodes alone.
B2FIL_HD inline constexpr uint32_t walk_nodes_stride(int depth) { return 4u << depth; }
// Forests of at most this many trees, at least two levels deep and without categorical tests also
// keep the three top nodes of every tree on the host: the traversal kernel takes them as a launch
// parameter and reads them through the constant cache instead of shared memory.
constexpr int kQTopTrees = 2048;
// Vector leaves of forests with at most this many outputs are stored in the tree blocks of the
// rank-quantised image (and summed in registers): the walk then never leaves shared memory.
constexpr int kQInlineClasses = 4;

// ---- compact image of a sparse forest -----------------------------------------------------------
// Deep, ragged forests are bound by the chain of dependent node fetches from L2 / HBM.  Sparse
// forests whose fields fit therefore carry a second image built for exactly that.  The packer writes
// it node by node; what the kernel reads below the heaps are blocks made from it (further down).
//  * internal nodes only, 8 bytes each {value, meta}, in depth-first order per tree, the child
//    with the larger subtree first (rows are more likely to go where the training data went);
//    the first child of node k is node k + 1;
//  * leaves live in their own arrays (payload, id), numbered in the same depth-first order.  A
//    walk carries the pair (k, L) = (internal node, number of leaves that precede it); with
//    `off` = 1 + internal nodes of the first child's subtree,
//        first child : k + 1,   L          second child : k + off, L + off
//    (a subtree with m internal nodes has m + 1 leaves), and two flags in the node say when the
//    child reached is a leaf, whose number is then L (first) or L + off (second);
//  * meta = default-left << 31 | categorical << 30 | first-is-leaf << 29 | second-is-leaf << 28 |
//    first-child-is-the-right-child << 27 | off << feat_bits | feature;
//  * fp64 forests keep `value` = the largest float <= threshold, and the kernel stages rows as
//    floats rounded down: xl < value proves x < threshold, xl > value proves x > threshold, and
//    only when xl == value the row's double and the exact threshold (`c_exact`) are read (one in
//    2^24 visits on continuous data), so 4-byte values decide every fp64 test exactly;
//  * the top `c_top_levels` levels of every tree are also stored as a complete heap
//    [2^T nodes {value, feature | flags}][2^T exits], which the kernel streams through
//    shared memory: a walk starts with T steps that cost no global fetch and leaves the heap
//    through an exit: the node to continue at (in the uploaded heaps its block), or the leaf reached
//    (bit 31).
constexpr uint32_t CMETA_FIRST_LEAF  = 0x20000000u;
constexpr uint32_t CMETA_SECOND_LEAF = 0x10000000u;
constexpr uint32_t CMETA_SWAPPED     = 0x08000000u;  // the first (adjacent) child is the right child
constexpr uint32_t CMETA_LOW27       = 0x07FFFFFFu;
constexpr uint32_t C_EXIT_LEAF      = 0x80000000u;
constexpr uint32_t C_NO_NODE        = 0xFFFFFFFFu;
constexpr int kCMaxTopLevels        = 10;
// What the kernel walks below the heaps is made from these arrays at upload (blocks.cpp): blocks of
// 32 bytes, one sector, that hold a node, its two children and the heaviest of its grandchildren, so
// that a fetch is good for two tests always and for a third one more often than not (the pairs of
// depth-first neighbours that the 8-byte nodes allow were good for 1.35 on average, and the sectors
// between L1 and L2 are what bounds the walk):
//   words 0..3: values of root, left child, right child, grandchild
//   words 4, 5: a 16-bit test each: feature | missing-goes-left | categorical, and three more bits
//     root: is there a grandchild (else the fourth test is a filler), whose place it has: 0..3
//     left and right child: which of the edges out of the block lead to a leaf (3 + 2 bits)
//   word 6: first child block, word 7: first leaf.
// The edges are numbered left to right, five with the grandchild and four without; the blocks that
// the edges lead to are consecutive, and so are the leaves.  A leaf in a child's place stands on both
// sides of a filler test, twice in the leaf arrays.  Exits of the heaps name a block or a leaf.
constexpr uint32_t BLK_FEATURE      = 0x7FFu;
constexpr uint32_t BLK_DEFAULT_LEFT = 0x800u;
constexpr uint32_t BLK_CATEGORICAL  = 0x1000u;
constexpr uint32_t BLK_FOURTH_SHIFT = 13;
constexpr uint32_t BLK_HAS_FOURTH   = 0x8000u;
struct CompactNode {  // 8 bytes
  uint32_t value;     // float threshold bits (fp64 forests: rounded down) | bitset | pool offset
  uint32_t meta;
};
// Levels of every tree that go into the heap (0: no compact image).  Measured on a 200-tree
// depth-20 forest: the walk below the heap is bound by how many dependent fetches an SM keeps in
// flight (warps x walks per warp, and the L1 that tracks the misses: it shrinks as shared memory
// grows), so heap levels are only worth their shared memory while they do not cost warps.  Eight
// levels (4 KB per tree) on 128-row tiles were the best trade when 8-byte nodes were walked by 28
// warps (9.5e7 rows/s; six levels 8.9e7, nine levels - room for 12 warps only - 5.8e7); the walk over
// blocks, with 20 warps, kept them.
constexpr int kCDefaultTopLevels = 8;
// With many features the row tile leaves little room: the heaps then get fewer levels, so that
// 24 warps would still fit under the 160 KiB that the launch code prefers (one warp per CTA next to
// eight-level heaps ran a 1024-feature forest at 3.7e7 rows/s).  On the safe side of what is launched:
// 20 warps on 128-row tiles, 23 at most, and a tile without the padding word per feature.
inline int compact_pick_top_levels(int elem_bytes, int n_features, int n_outputs, int max_depth)
{
  const size_t hard = 218 * 1024, soft = 160 * 1024;
  constexpr int kWalks = 4;  // trees a warp walks at once (kCompactTreesInFlight)
  int fallback = 0;
  for (int T = kCDefaultTopLevels; T >= 1; --T) {
    const size_t heap = static_cast<size_t>(16) << T;
    for (int R = 128; R >= 32; R /= 2) {
      const size_t tile = static_cast<size_t>(n_features) * (R + 1) * 4;  // rows are staged as floats
      const int G       = (24 + R / 32 - 1) / (R / 32);
      const size_t acc  = static_cast<size_t>(G) * n_outputs * R * elem_bytes;
      if (tile + acc + heap * G * kWalks <= soft) return std::max(1, std::min(T, max_depth));
      if (fallback == 0 && tile + static_cast<size_t>(8) * n_outputs * R * elem_bytes + heap * 8 <= hard)
        fallback = T;
    }
  }
  return fallback == 0 ? 0 : std::max(1, std::min(fallback, max_depth));
}

enum NodeFormat : int32_t {
  FMT_DENSE_F   = 0,
  FMT_DENSE_D   = 1,
  FMT_SPARSE_8  = 2,
  FMT_SPARSE_16F = 3,
  FMT_SPARSE_16D = 4,
};

// Device view handed to kernels by value.  Pointers are device pointers on the forest's device.
struct ForestView {
  int32_t format;
  int32_t n_trees;
  int32_t n_features;
  int32_t n_outputs;
  int32_t leaf_vector_len;
  int32_t postproc;
  int32_t has_categorical;
  int32_t cat_inline;       // 1: every category list fits a 32-bit inline bitset
  int32_t max_depth;        // loop bound of sparse traversal
  int32_t dense_depth;      // D
  int32_t feat_bits;        // SparseNode8: width of the feature field
  int32_t layout;
  int64_t tree_stride;      // dense: bytes between trees
  const void* nodes;        // dense: tree blocks; sparse: node array
  const uint32_t* roots;    // sparse: index of every tree's root in `nodes`
  const uint32_t* leaf_ids; // dense: [n_trees << D] id per leaf slot; sparse: [n_nodes] id per node
  const uint32_t* cat_pool; // [n_words, words...] records of large category lists
  const int32_t* tree_class;// [n_trees] output a scalar leaf adds to (packed tree order)
  const int32_t* tree_orig; // [n_trees] index of the packed tree in the description
  const void* leaf_vectors; // [n_vectors * n_outputs] of the forest precision
  const void* out_scale;    // [n_outputs] 1/divisor of average_tree_output (or 1)
  const void* out_bias;     // [n_outputs] base scores
  double sigmoid_alpha;
  double ratio_c;
  // rank-quantised copy of a dense forest (q_enabled != 0)
  int32_t q_enabled;
  int32_t q_n_bundles;
  int32_t q_has_cat;            // 1: tree blocks carry a third array of 32-bit category sets
  int32_t q_trees_in_order;     // 1: packed tree t is the caller's tree t (tree_orig is the identity)
  int32_t q_leaf_bytes;         // bytes per leaf payload: the element size (scalar, or index of the
                                // leaf's vector), or n_outputs elements when the vectors of a
                                // forest with few outputs sit in the tree blocks themselves
  int32_t q_any_default_left;   // 0: missing values go right in every test, also in walking order
  int64_t q_tree_stride;        // bytes between trees, 16-byte multiple: 2^D * (node bytes + leaf bytes), or, in
                                // walking order, walk_tree_stride()
  const void* q_nodes;          // [n_trees] blocks of [2^D nodes][2^D leaf payloads] of uint32 nodes,
                                // with [2^D category sets] in between when q_has_cat; in walking order with
                                // the places of walk_level_at(), and behind the blocks of all trees, where
                                // payloads may stay in global memory (q_far()), [n_trees][2^D] payloads by
                                // walk_far_number() and [n_trees] nodes without payloads, walk_nodes_stride() bytes
                                // (no pointers of their own: with three more the parameters of every kernel were
                                // 408 bytes instead of 384, and one row of 1000 depth-8 trees took 8.57 us, not 8.45)
  const void* q_nodes_ids;      // same blocks with the leaf id (uint32) in every leaf payload slot:
                                // what the traversal streams when it reports leaf ids
  const void* q_nodes_nan;      // q_nodes for tiles with missing values and doubled columns (see
                                // above), or null; the nodes without payloads follow at once
  int64_t q_max_blob_bytes;     // largest bundle of group blobs
  int32_t q_bundle_features;    // features of the widest bundle
  int32_t q_last_features;      // features of the last one
  const unsigned char* q_blob;  // group blobs
  const QGroup* q_groups;
  const QBundle* q_bundles;     // [q_n_bundles]
  // compact image of a sparse forest (c_enabled != 0), see above
  int32_t c_enabled;
  int32_t c_top_levels;         // T
  int32_t c_feat_bits;
  int32_t c_block_steps;        // most blocks on a walk
  int64_t c_top_stride;         // bytes between the heaps of two trees: 2^T * 16
  const uint32_t* c_blocks;     // [n_blocks * 8]
  const double* c_exact;        // [n_blocks * 4] exact thresholds (fp64 forests), else null
  const void* c_leaf_payload;   // [n_leaves] scalar in the forest precision or vector index
  const uint32_t* c_leaf_ids;   // [n_leaves] id of the leaf in the imported model
  const unsigned char* c_top;   // [n_trees] heaps
  const double* c_top_exact;    // [n_trees << T] exact thresholds of the heap nodes (fp64), -inf = padding
};

// Host-side result of packing, before upload.
struct PackedForest {
  ForestView view{};  // pointer members unset
  int32_t precision = B2FIL_F32;
  int32_t storage   = B2FIL_STORAGE_SPARSE;
  int32_t align_bytes = 0;
  int32_t node_bytes = 0;
  int64_t n_nodes_in = 0;
  int64_t n_nodes_packed = 0;
  std::vector<uint8_t> nodes;
  std::vector<uint32_t> roots;
  std::vector<uint32_t> leaf_ids;
  std::vector<uint32_t> cat_pool;
  std::vector<int32_t> tree_class;
  std::vector<int32_t> tree_orig;
  std::vector<uint8_t> leaf_vectors;
  std::vector<uint8_t> out_scale;
  std::vector<uint8_t> out_bias;
  std::vector<uint8_t> q_nodes;
  std::vector<uint8_t> q_nodes_ids;  // q_nodes with leaf ids in the payload slots
  std::vector<uint8_t> q_nodes_nan;  // q_nodes for doubled columns, or empty
  std::vector<uint32_t> q_top;  // root and its two children of every tree (3 words per tree), or empty
  std::vector<uint8_t> q_thresholds;
  std::vector<uint16_t> q_lut;
  std::vector<QFeature> q_feats;
  std::vector<QGroup> q_groups;
  std::vector<QBundle> q_bundles;
  std::vector<uint8_t> q_blob;
  std::vector<uint32_t> c_nodes;          // two words per internal node
  std::vector<uint32_t> c_leaves_before;  // L of every internal node (host only: the exits carry it)
  std::vector<double> c_exact;
  std::vector<uint8_t> c_leaf_payload;
  std::vector<uint32_t> c_leaf_ids;
  std::vector<uint8_t> c_top;
  std::vector<uint32_t> c_top_src;
  // blocks of the compact image, filled by build_blocks()
  std::vector<uint32_t> b_blocks;
  std::vector<double> b_exact;
  std::vector<uint8_t> b_leaf_payload;
  std::vector<uint32_t> b_leaf_ids;
  std::vector<uint8_t> b_top;
  std::vector<double> b_top_exact;
};

// Bucket of a value in a feature's table; the same expression runs on the device
// (fma and float->int truncation are exactly specified, so host and device agree bit for bit).
template <typename T>
inline uint32_t q_bucket_host(T x, T scale, T offset, uint32_t n_buckets)
{
  T v = std::fma(x, scale, offset);
  v   = std::fmax(v, T(0));  // also turns NaN (inf * 0) into 0
  v   = std::fmin(v, static_cast<T>(n_buckets - 1));
  return static_cast<uint32_t>(v);
}

// Shared memory the quantisation kernel may spend on the tables of one feature group.
constexpr uint32_t kQGroupSmemBudget = 208 * 1024;
constexpr uint32_t kQMaxGroupFeatures = 32;

// Rows of a tile for a caller's chunk_size > 0 (units of 32 rows): rounded down to a power of two, which
// is what every kernel's tile arithmetic needs, and at most `most`, itself a power of two.
inline int chunk_rows(int chunk_size, int most)
{
  int rows = 32;
  while (rows < most && rows / 16 <= chunk_size) rows *= 2;
  return rows;
}

// Before the upload: the blocks of a forest with a compact image.  False when a field does not fit.
bool build_blocks(PackedForest& pf);

// Before the upload: the tree blocks of a rank-quantised image with categorical tests change from
// [2^D {node, category set}] to [2^D nodes][2^D category sets], which is what the kernels read.
void split_category_sets(const ForestView& view, std::vector<uint8_t>& image);

// Is the image uploaded in walking order?  Only where every kernel that may walk it knows the depth at compile
// time: fp32, depth 4 to 10, no categorical tests.
inline bool q_walk_order(int format, int depth, bool has_cat)
{
  return format == FMT_DENSE_F && depth >= 4 && depth <= 10 && !has_cat;
}
inline bool q_walk_order(const ForestView& v) { return q_walk_order(v.format, v.dense_depth, v.q_has_cat != 0); }
// May the payloads stay in global memory (depth 9 and 10, scalar leaves)?  A quarter more device memory.
inline bool q_far(const ForestView& v) { return q_walk_order(v) && walk_blocks(v.dense_depth) && v.leaf_vector_len <= 1; }
// Before the upload of such images (others stay as they are): heap order and ranks << 17 become what the kernels walk
// (see above), trees of walk_tree_stride() bytes, and the arrays for payloads in global memory are made.
void walk_order(PackedForest& pf);

// Validate `desc`, normalise its tests and lay its nodes out.  Returns B2FIL_OK or an error code
// with `err` set.  `dense_ok(depth, precision, n_features, n_outputs)` tells whether the dense
// kernels can run a forest of that shape (shared-memory fit): 0 no, 1 yes, 2 only the traversal
// over rank-quantised rows (its 2-byte row tile fits where a tile of reals does not: forests with
// a thousand features and more); AUTO storage asks it.
int pack_forest(const b2fil_forest_desc& desc, const b2fil_create_opts& opts,
                int (*dense_ok)(int depth, int precision, int n_features, int n_outputs),
                PackedForest& out,
                std::string& err);

}  // namespace b2fil
