// Test-only: the rank-quantised images in heap order against the same images as walk_order() leaves them for
// the kernels.  Both are walked over random codes per feature, the first with signed subtractions and heap
// indices, the second with half-precision compares and places in a level; the payloads must agree.
#include <cmath>
#include <cstring>
#include <random>
#include <string>

#include "../../cuml_b200/csrc/forest.hpp"

using namespace b2fil;

namespace {
int yes(int, int, int, int) { return 1; }
// value of a half-precision float
double half_value(uint32_t h)
{
  const int e = (h >> 10) & 31, m = h & 1023;
  double v;
  if (e == 31) {
    v = m ? NAN : INFINITY;
  } else {
    v = e ? std::ldexp(1024 + m, e - 25) : std::ldexp(m, -24);
  }
  return (h & 0x8000u) ? -v : v;
}
}  // namespace

// Number of (row of codes, tree) pairs that differ; -1 when the forest has no ranks.
extern "C" int64_t walk_check(const b2fil_forest_desc* desc, const b2fil_create_opts* opts, int n, int seed)
{
  PackedForest pf;
  std::string err;
  if (pack_forest(*desc, *opts, yes, pf, err) != B2FIL_OK || !pf.view.q_enabled || pf.view.q_has_cat) return -1;
  const ForestView& v = pf.view;
  PackedForest walked = pf;
  walk_order(walked);
  if (!q_walk_order(v))  // stays in heap order
    return walked.q_nodes == pf.q_nodes && walked.q_nodes_ids == pf.q_nodes_ids &&
               walked.q_nodes_nan == pf.q_nodes_nan && walked.q_top == pf.q_top
             ? 0 : 1;
  const int D = v.dense_depth, F = v.n_features;
  const size_t width = size_t(1) << D, leaves = width * 4;
  const size_t lbytes = static_cast<size_t>(v.q_leaf_bytes);
  const size_t to     = size_t(4) * walk_leaves_at(D, lbytes);
  const size_t stride = walk_tree_stride(D, static_cast<size_t>(v.q_leaf_bytes));
  std::mt19937 rng(seed);
  int64_t bad = 0;
  for (int image = 0; image < 3; ++image) {
    const std::vector<uint8_t>& heap = image == 0 ? pf.q_nodes : (image == 1 ? pf.q_nodes_ids : pf.q_nodes_nan);
    const std::vector<uint8_t>& walk =
      image == 0 ? walked.q_nodes : (image == 1 ? walked.q_nodes_ids : walked.q_nodes_nan);
    const size_t nodes_alone = q_far(v) ? walk_nodes_stride(D) : 0, payloads_alone = q_far(v) ? 4 * width : 0;
    const size_t tree_bytes = stride + (image == 1 ? 0 : nodes_alone) + (image == 0 ? payloads_alone : 0);
    if (walk.size() != (heap.empty() ? 0 : tree_bytes * v.n_trees)) return -2;
    if (heap.empty()) continue;
    const bool doubled = image == 2;
    for (int r = 0; r < n; ++r) {
      std::vector<uint32_t> a(2 * F);  // codes of the columns and of their copies
      std::vector<bool> missing(F);
      for (int f = 0; f < F; ++f) {
        missing[f]     = rng() % 8 == 0;
        const uint32_t code = rng() % 9 == 0 ? Q_MAX_RANK : rng() % (pf.q_feats[f].m + 1);
        a[f]     = missing[f] ? Q_NAN_CODE : code;
        a[F + f] = missing[f] ? Q_NAN_CODE | Q_NAN_LEFT_BIT : code;
      }
      for (int t = 0; t < v.n_trees; ++t) {
        const uint8_t* hb = heap.data() + static_cast<size_t>(v.q_tree_stride) * t;
        const uint8_t* wb = walk.data() + stride * t;
        uint32_t i = 1, place = 0, block = 0;
        const uint32_t pitch = walk_blocks(D) ? walk_pitch(D, lbytes == 4) : 1u;
        for (int l = 0; l < D; ++l) {
          uint32_t node;
          if (walk_blocks(D) && l == 5) {
            block = place;
            place *= pitch;
          }
          std::memcpy(&node, hb + i * 4, 4);
          const uint32_t f = (node & Q_FEATURE_FIELD) >> Q_FEATURE_SHIFT;
          bool right       = static_cast<int32_t>(node - (a[f] << Q_RANK_SHIFT)) < 0;
          if (!doubled && missing[f]) right = (node & Q_DEFAULT_RIGHT) != 0;
          i = 2 * i + (right ? 1 : 0);

          const size_t at = (walk_level_at(D, l) + place) * 4;
          std::memcpy(&node, wb + at, 4);
          const uint32_t g   = (node & Q_FEATURE_FIELD) >> Q_FEATURE_SHIFT;
          const uint32_t hi  = node >> 16;
          const uint32_t code = a[g];
          right = half_value(code) > std::fabs(half_value(hi));
          // (the kernels look at the direction of missing values only in forests that are marked for it)
          if (!doubled && code == Q_NAN_CODE && v.q_any_default_left) right = (hi & 0x8000) == 0;
          if (right) place += walk_step_words(D, l);
        }
        if (walk_blocks(D) && lbytes != 4) place += block;
        if (to + (place + 1) * lbytes > stride ||
            std::memcmp(hb + leaves + (i - width) * lbytes, wb + to + place * lbytes, lbytes) != 0)
          ++bad;
      }
    }
  }
  for (size_t t = 0; 3 * t < walked.q_top.size(); ++t)
    if (std::memcmp(&walked.q_top[3 * t], walked.q_nodes.data() + stride * t + 4, 12) != 0) ++bad;
  if (q_far(v)) {
    // nodes alone and payloads for global memory: the walk over the former ends, by the kernels' arithmetic, on
    // the payload that the walk over both ends on
    for (int image = 0; image < 2; ++image) {
      const std::vector<uint8_t>& walk = image == 0 ? walked.q_nodes : walked.q_nodes_nan;
      if (walk.empty()) continue;
      const uint8_t* far   = walked.q_nodes.data() + stride * v.n_trees;
      const uint8_t* nodes = walk.data() + stride * v.n_trees + (image == 0 ? size_t(4) * width * v.n_trees : 0);
      const uint32_t with = walk_pitch(D, true), without = walk_pitch(D, false);
      for (int i = 0; i < 4 * n; ++i) {
        const size_t t = rng() % v.n_trees;
        uint32_t a = 0, b = 0, block = 0;
        for (int l = 0; l < D; ++l) {
          if (l == 5) {
            block = a;
            a *= with;
            b *= without;
          }
          if (std::memcmp(walk.data() + stride * t + 4u * (walk_level_at(D, l) + a),
                          nodes + size_t(walk_nodes_stride(D)) * t + 4u * (walk_level_at(D, l) + b), 4) != 0)
            ++bad;
          if (rng() & 1u) {
            a += walk_step_words(D, l);
            b += walk_step_words(D, l);
          }
        }
        const uint32_t place = 4u * (b - block * without);
        const uint32_t at = ((4u * block) << (D - 5)) + ((place >> (D - 8) | place << 3) & ((4u << (D - 5)) - 4u));
        if (at / 4 >= width || std::memcmp(far + 4 * width * t + at, walk.data() + stride * t + to + 4u * a, 4) != 0) ++bad;
      }
    }
  }
  return bad;
}
