// The image of a sparse forest that the compact kernel walks (layout in forest.hpp), made from the
// compact image of the packer.
#include <algorithm>
#include <cstring>

#include "forest.hpp"

namespace b2fil {
namespace {

// A child in the compact image: internal node or leaf.
struct Child {
  bool leaf;
  uint32_t index;
};

struct BlockBuilder {
  PackedForest& pf;
  const ForestView& v;
  const uint32_t n_nodes;
  const size_t payload_bytes;
  std::vector<uint32_t> size;      // internal nodes in the subtree of every node
  std::vector<uint32_t> roots;     // root node of every block
  std::vector<int32_t> level;      // blocks above every block, from its heap exit
  uint32_t n_leaves = 0;

  explicit BlockBuilder(PackedForest& p)
      : pf(p), v(p.view), n_nodes(static_cast<uint32_t>(p.c_leaf_ids.size()) - static_cast<uint32_t>(p.view.n_trees)),
        payload_bytes(p.precision == B2FIL_F32 ? 4 : 8)
  {
  }

  uint32_t meta(uint32_t k) const { return pf.c_nodes[size_t(k) * 2 + 1]; }
  uint32_t offset(uint32_t k) const { return (meta(k) & CMETA_LOW27) >> v.c_feat_bits; }
  Child first(uint32_t k) const
  {
    if (meta(k) & CMETA_FIRST_LEAF) return {true, pf.c_leaves_before[k]};
    return {false, k + 1};
  }
  Child second(uint32_t k) const
  {
    if (meta(k) & CMETA_SECOND_LEAF) return {true, pf.c_leaves_before[k] + offset(k)};
    return {false, k + offset(k)};
  }
  Child left(uint32_t k) const { return meta(k) & CMETA_SWAPPED ? second(k) : first(k); }
  Child right(uint32_t k) const { return meta(k) & CMETA_SWAPPED ? first(k) : second(k); }
  uint32_t weight(Child c) const { return c.leaf ? 0u : size[c.index]; }

  void measure()
  {
    // children follow their parents in the node order
    size.assign(n_nodes, 1);
    for (uint32_t k = n_nodes; k-- > 0;) size[k] = 1 + weight(first(k)) + weight(second(k));
  }

  uint32_t add_root(uint32_t node, int32_t lvl)
  {
    roots.push_back(node);
    level.push_back(lvl);
    return static_cast<uint32_t>(roots.size() - 1);
  }
  void add_leaf(uint32_t leaf)
  {
    const size_t at = pf.b_leaf_payload.size();
    pf.b_leaf_payload.resize(at + payload_bytes);
    std::memcpy(pf.b_leaf_payload.data() + at, pf.c_leaf_payload.data() + size_t(leaf) * payload_bytes,
                payload_bytes);
    pf.b_leaf_ids.push_back(pf.c_leaf_ids[leaf]);
    ++n_leaves;
  }

  // Test word of a node: feature, missing-goes-left, categorical.
  uint32_t half(uint32_t k) const
  {
    const uint32_t m = meta(k);
    return (m & ((1u << v.c_feat_bits) - 1u)) | ((m & META_DEFAULT_LEFT) ? BLK_DEFAULT_LEFT : 0u) |
           ((m & META_CATEGORICAL) ? BLK_CATEGORICAL : 0u);
  }

  void block(uint32_t b)
  {
    const uint32_t root = roots[b];
    uint32_t value[4], test[4] = {0, 0, 0, 0};
    double exact[4];
    for (int i = 0; i < 4; ++i) {  // filler tests: both sides lead to the same leaf, or nobody asks
      value[i] = 0x7F800000u;
      exact[i] = std::numeric_limits<double>::infinity();
    }
    auto put = [&](int i, uint32_t k) {
      value[i] = pf.c_nodes[size_t(k) * 2];
      test[i]  = half(k);
      if (!pf.c_exact.empty()) exact[i] = pf.c_exact[k];
    };
    put(0, root);
    Child edges[5];
    const Child kids[2] = {left(root), right(root)};
    Child grand[4];
    for (int i = 0; i < 2; ++i) {
      if (kids[i].leaf) {
        grand[2 * i] = grand[2 * i + 1] = kids[i];
      } else {
        put(1 + i, kids[i].index);
        grand[2 * i]     = left(kids[i].index);
        grand[2 * i + 1] = right(kids[i].index);
      }
    }
    // the grandchild with the largest subtree joins the block
    int heavy = 0;
    for (int i = 1; i < 4; ++i)
      if (weight(grand[i]) > weight(grand[heavy])) heavy = i;
    const bool has = !grand[heavy].leaf;
    int n_edges    = 0;
    for (int i = 0; i < 4; ++i) {
      if (has && i == heavy) {
        put(3, grand[i].index);
        edges[n_edges++] = left(grand[i].index);
        edges[n_edges++] = right(grand[i].index);
      } else {
        edges[n_edges++] = grand[i];
      }
    }
    uint32_t leaf_mask        = 0;
    const uint32_t child_base = static_cast<uint32_t>(roots.size());
    const uint32_t leaf_base  = n_leaves;
    for (int e = 0; e < n_edges; ++e) {
      if (edges[e].leaf) {
        leaf_mask |= 1u << e;
        add_leaf(edges[e].index);
      } else {
        add_root(edges[e].index, level[b] + 1);
      }
    }
    if (has) test[0] |= BLK_HAS_FOURTH | static_cast<uint32_t>(heavy) << BLK_FOURTH_SHIFT;
    test[1] |= (leaf_mask & 7u) << 13;
    test[2] |= (leaf_mask >> 3) << 13;
    const uint32_t words[8] = {value[0], value[1], value[2], value[3], test[0] | test[1] << 16,
                               test[2] | test[3] << 16, child_base, leaf_base};
    pf.b_blocks.insert(pf.b_blocks.end(), words, words + 8);
    if (!pf.c_exact.empty()) pf.b_exact.insert(pf.b_exact.end(), exact, exact + 4);
  }

  bool build()
  {
    if (v.n_features > static_cast<int32_t>(BLK_FEATURE) + 1) return false;
    measure();
    const size_t heap_n = size_t(1) << v.c_top_levels;
    const size_t bytes  = static_cast<size_t>(v.c_top_stride);
    pf.b_blocks.reserve(size_t(n_nodes) * 3 + 64);
    pf.b_leaf_payload.reserve(pf.c_leaf_payload.size() + pf.c_leaf_payload.size() / 8);
    pf.b_leaf_ids.reserve(pf.c_leaf_ids.size() + pf.c_leaf_ids.size() / 8);
    if (!pf.c_exact.empty()) pf.b_exact.reserve(size_t(n_nodes) * 2);
    pf.b_top = pf.c_top;
    size_t done = 0;  // blocks written
    for (int t = 0; t < v.n_trees; ++t) {
      uint8_t* exits = pf.b_top.data() + bytes * t + heap_n * 8;
      Child last{false, C_NO_NODE};
      uint32_t last_to = 0;
      for (size_t e = 0; e < heap_n; ++e) {
        // {block to continue at, 0} or {leaf | flag, 0}; neighbours may be the same leaf
        uint32_t to;
        std::memcpy(&to, exits + e * 8, 4);
        const Child c{(to & C_EXIT_LEAF) != 0u, to & ~C_EXIT_LEAF};
        if (!(c.leaf && last.leaf && c.index == last.index)) {
          if (c.leaf) {
            add_leaf(c.index);
            last_to = (n_leaves - 1) | C_EXIT_LEAF;
          } else {
            last_to = add_root(c.index, 1);
          }
          last = c;
        }
        const uint32_t exit[2] = {last_to, 0u};
        std::memcpy(exits + e * 8, exit, 8);
      }
      // children are appended behind all blocks known so far: a block's children are contiguous
      for (; done < roots.size(); ++done) block(static_cast<uint32_t>(done));
    }
    if (roots.size() >= (size_t(1) << 31) || n_leaves >= (1u << 31)) return false;
    if (pf.b_blocks.empty()) pf.b_blocks.assign(8, 0u);
    int32_t steps = 0;
    for (int32_t l : level) steps = std::max(steps, l);
    pf.view.c_block_steps = steps;
    if (!pf.c_top_src.empty()) {
      pf.b_top_exact.assign(pf.c_top_src.size(), -std::numeric_limits<double>::infinity());
      for (size_t i = 0; i < pf.c_top_src.size(); ++i)
        if (pf.c_top_src[i] != C_NO_NODE) pf.b_top_exact[i] = pf.c_exact[pf.c_top_src[i]];
      if (pf.b_exact.empty()) pf.b_exact.assign(4, 0.0);
    }
    return true;
  }
};

}  // namespace

bool build_blocks(PackedForest& pf)
{
  return BlockBuilder(pf).build();
}

}  // namespace b2fil
