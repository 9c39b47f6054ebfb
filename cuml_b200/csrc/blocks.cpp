// The image of a sparse forest that the compact kernel walks (layout in forest.hpp), made from the
// compact image of the packer.
#include <algorithm>
#include <cstring>

#include "each_tree.hpp"
#include "forest.hpp"

namespace b2fil {
namespace {

// A child in the compact image: internal node or leaf.
struct Child {
  bool leaf;
  uint32_t index;
};

// Blocks and leaves of one tree, numbered from 0; place() puts them behind those of the trees before.
struct TreeBlocks {
  const PackedForest& pf;
  const ForestView& v;
  const std::vector<uint32_t>& size;  // internal nodes in the subtree of every node of the forest
  std::vector<uint32_t> roots;        // root node of every block
  std::vector<int32_t> level;         // blocks above every block, from its heap exit
  std::vector<uint32_t> words;        // eight per block
  std::vector<uint32_t> exits;        // {block | leaf and flag} per exit of the heap
  std::vector<uint32_t> leaves;       // by their number in the forest

  TreeBlocks(const PackedForest& p, const std::vector<uint32_t>& s) : pf(p), v(p.view), size(s) {}

  static uint32_t meta(const PackedForest& pf, uint32_t k) { return pf.c_nodes[size_t(k) * 2 + 1]; }
  static uint32_t offset(const PackedForest& pf, uint32_t k)
  {
    return (meta(pf, k) & CMETA_LOW27) >> pf.view.c_feat_bits;
  }
  static Child first(const PackedForest& pf, uint32_t k)
  {
    if (meta(pf, k) & CMETA_FIRST_LEAF) return {true, pf.c_leaves_before[k]};
    return {false, k + 1};
  }
  static Child second(const PackedForest& pf, uint32_t k)
  {
    if (meta(pf, k) & CMETA_SECOND_LEAF) return {true, pf.c_leaves_before[k] + offset(pf, k)};
    return {false, k + offset(pf, k)};
  }
  Child left(uint32_t k) const { return meta(pf, k) & CMETA_SWAPPED ? second(pf, k) : first(pf, k); }
  Child right(uint32_t k) const { return meta(pf, k) & CMETA_SWAPPED ? first(pf, k) : second(pf, k); }
  uint32_t weight(Child c) const { return c.leaf ? 0u : size[c.index]; }

  uint32_t add_root(uint32_t node, int32_t lvl)
  {
    roots.push_back(node);
    level.push_back(lvl);
    return static_cast<uint32_t>(roots.size() - 1);
  }

  // Test word of a node: feature, missing-goes-left, categorical.
  uint32_t half(uint32_t k) const
  {
    const uint32_t m = meta(pf, k);
    return (m & ((1u << v.c_feat_bits) - 1u)) | ((m & META_DEFAULT_LEFT) ? BLK_DEFAULT_LEFT : 0u) |
           ((m & META_CATEGORICAL) ? BLK_CATEGORICAL : 0u);
  }

  // Nodes of a block (C_NO_NODE: filler), the place of the fourth or -1, and the edges out of it, left
  // to right.
  struct Shape {
    uint32_t node[4];
    int fourth, n_edges;
    Child edges[5];
  };
  Shape shape(uint32_t root) const
  {
    Shape s{{root, C_NO_NODE, C_NO_NODE, C_NO_NODE}, -1, 0, {}};
    const Child kids[2] = {left(root), right(root)};
    Child grand[4];
    for (int i = 0; i < 2; ++i) {
      if (kids[i].leaf) {
        grand[2 * i] = grand[2 * i + 1] = kids[i];
      } else {
        s.node[1 + i]    = kids[i].index;
        grand[2 * i]     = left(kids[i].index);
        grand[2 * i + 1] = right(kids[i].index);
      }
    }
    // the grandchild with the largest subtree joins the block
    int heavy = 0;
    for (int i = 1; i < 4; ++i)
      if (weight(grand[i]) > weight(grand[heavy])) heavy = i;
    for (int i = 0; i < 4; ++i) {
      if (i == heavy && !grand[i].leaf) {
        s.fourth             = i;
        s.node[3]            = grand[i].index;
        s.edges[s.n_edges++] = left(grand[i].index);
        s.edges[s.n_edges++] = right(grand[i].index);
      } else {
        s.edges[s.n_edges++] = grand[i];
      }
    }
    return s;
  }

  void block(uint32_t b)
  {
    const Shape s = shape(roots[b]);
    // filler tests: both sides lead to the same leaf, or nobody asks
    uint32_t value[4] = {0x7F800000u, 0x7F800000u, 0x7F800000u, 0x7F800000u}, test[4] = {0, 0, 0, 0};
    for (int i = 0; i < 4; ++i) {
      if (s.node[i] == C_NO_NODE) continue;
      value[i] = pf.c_nodes[size_t(s.node[i]) * 2];
      test[i]  = half(s.node[i]);
    }
    uint32_t leaf_mask        = 0;
    const uint32_t child_base = static_cast<uint32_t>(roots.size());
    const uint32_t leaf_base  = static_cast<uint32_t>(leaves.size());
    for (int e = 0; e < s.n_edges; ++e) {
      if (s.edges[e].leaf) {
        leaf_mask |= 1u << e;
        leaves.push_back(s.edges[e].index);
      } else {
        add_root(s.edges[e].index, level[b] + 1);
      }
    }
    if (s.fourth >= 0) test[0] |= BLK_HAS_FOURTH | static_cast<uint32_t>(s.fourth) << BLK_FOURTH_SHIFT;
    test[1] |= (leaf_mask & 7u) << 13;
    test[2] |= (leaf_mask >> 3) << 13;
    const uint32_t w[8] = {value[0], value[1], value[2], value[3], test[0] | test[1] << 16,
                           test[2] | test[3] << 16, child_base, leaf_base};
    words.insert(words.end(), w, w + 8);
  }

  void build(int t)
  {
    const size_t heap_n = size_t(1) << v.c_top_levels;
    const uint8_t* from = pf.c_top.data() + static_cast<size_t>(v.c_top_stride) * t + heap_n * 8;
    Child last{false, C_NO_NODE};
    for (size_t e = 0; e < heap_n; ++e) {
      // neighbours may be the same leaf
      uint32_t to;
      std::memcpy(&to, from + e * 8, 4);
      const Child c{(to & C_EXIT_LEAF) != 0u, to & ~C_EXIT_LEAF};
      if (c.leaf && last.leaf && c.index == last.index) {
        exits.push_back(exits.back());
      } else if (c.leaf) {
        leaves.push_back(c.index);
        exits.push_back(static_cast<uint32_t>(leaves.size() - 1) | C_EXIT_LEAF);
      } else {
        exits.push_back(add_root(c.index, 1));
      }
      last = c;
    }
    // children are appended behind all blocks known so far: a block's children are contiguous
    for (size_t b = 0; b < roots.size(); ++b) block(static_cast<uint32_t>(b));
  }

  void place(PackedForest& out, int t, uint32_t block0, uint32_t leaf0) const
  {
    for (size_t b = 0; b < roots.size(); ++b) {
      uint32_t* w = out.b_blocks.data() + (size_t(block0) + b) * 8;
      std::memcpy(w, words.data() + b * 8, 32);
      w[6] += block0;
      w[7] += leaf0;
      if (!out.c_exact.empty()) {
        const Shape s = shape(roots[b]);
        for (int i = 0; i < 4; ++i)
          out.b_exact[(size_t(block0) + b) * 4 + i] =
            s.node[i] == C_NO_NODE ? std::numeric_limits<double>::infinity() : out.c_exact[s.node[i]];
      }
    }
    const size_t bytes = out.precision == B2FIL_F32 ? 4 : 8;
    for (size_t i = 0; i < leaves.size(); ++i) {
      std::memcpy(out.b_leaf_payload.data() + (size_t(leaf0) + i) * bytes,
                  out.c_leaf_payload.data() + size_t(leaves[i]) * bytes, bytes);
      out.b_leaf_ids[size_t(leaf0) + i] = out.c_leaf_ids[leaves[i]];
    }
    uint8_t* to = out.b_top.data() + static_cast<size_t>(v.c_top_stride) * t + (size_t(8) << v.c_top_levels);
    for (size_t e = 0; e < exits.size(); ++e) {
      const uint32_t exit[2] = {exits[e] + ((exits[e] & C_EXIT_LEAF) ? leaf0 : block0), 0u};
      std::memcpy(to + e * 8, exit, 8);
    }
  }
};

}  // namespace

bool build_blocks(PackedForest& pf)
{
  ForestView& v = pf.view;
  if (v.n_features > static_cast<int32_t>(BLK_FEATURE) + 1) return false;
  const int n_trees      = v.n_trees;
  const uint32_t n_nodes = static_cast<uint32_t>(pf.c_leaf_ids.size()) - static_cast<uint32_t>(n_trees);
  // children follow their parents in the node order
  std::vector<uint32_t> size(n_nodes, 1);
  for (uint32_t k = n_nodes; k-- > 0;) {
    for (const Child c : {TreeBlocks::first(pf, k), TreeBlocks::second(pf, k)})
      if (!c.leaf) size[k] += size[c.index];
  }
  // Large forests are cut on several threads; the result does not depend on how many.  On one thread the
  // blocks took a third of the time of the rest of the packer (200 trees, 1.2e7 nodes: 700 ms in fp64 and
  // 515 in fp32 beside 2300 and 1900; on eight cores 330 and 205).
  const int threads = pack_threads(n_nodes, n_trees);
  std::vector<TreeBlocks> trees(n_trees, TreeBlocks(pf, size));
  for_each_tree(n_trees, threads, [&](int t) { trees[t].build(t); });
  std::vector<uint64_t> block0(n_trees + 1, 0), leaf0(n_trees + 1, 0);
  int32_t steps = 0;
  for (int t = 0; t < n_trees; ++t) {
    block0[t + 1] = block0[t] + trees[t].roots.size();
    leaf0[t + 1]  = leaf0[t] + trees[t].leaves.size();
    for (int32_t l : trees[t].level) steps = std::max(steps, l);
  }
  if (block0[n_trees] >= (uint64_t(1) << 31) || leaf0[n_trees] >= (uint64_t(1) << 31)) return false;
  // (never an empty array)
  pf.b_blocks.resize(std::max<uint64_t>(1, block0[n_trees]) * 8, 0u);
  if (!pf.c_exact.empty()) pf.b_exact.resize(std::max<uint64_t>(1, block0[n_trees]) * 4, 0.0);
  pf.b_leaf_payload.resize(leaf0[n_trees] * (pf.precision == B2FIL_F32 ? 4 : 8));
  pf.b_leaf_ids.resize(leaf0[n_trees]);
  pf.b_top = pf.c_top;
  for_each_tree(n_trees, threads, [&](int t) {
    trees[t].place(pf, t, static_cast<uint32_t>(block0[t]), static_cast<uint32_t>(leaf0[t]));
  });
  v.c_block_steps = steps;
  if (!pf.c_top_src.empty()) {
    pf.b_top_exact.assign(pf.c_top_src.size(), -std::numeric_limits<double>::infinity());
    for (size_t i = 0; i < pf.c_top_src.size(); ++i)
      if (pf.c_top_src[i] != C_NO_NODE) pf.b_top_exact[i] = pf.c_exact[pf.c_top_src[i]];
  }
  return true;
}

}  // namespace b2fil
