// Host-side interface between the launch code (kernels.cu) and the translation units that
// instantiate the traversal kernels over rank-quantised rows.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "kernels.hpp"

namespace b2fil {

// Raise the dynamic shared memory limit of `kernel` on the current device to `bytes` (cached per
// device and kernel).
int set_smem_bytes(const void* kernel, size_t bytes, std::string& err);

// A launch that may be split over clusters and may overlap the tail of the kernel before it.
struct SplitLaunch {
  dim3 grid;            // CTAs; grid.x is a multiple of `cluster`
  int threads;
  size_t smem_bytes;
  cudaStream_t stream;
  int cluster;          // CTAs per cluster (1: none)
  bool overlap;         // programmatic dependent launch: the kernel calls grid_wait()
};
template <typename... Params, typename... Args>
int launch_split(const SplitLaunch& l, std::string& err, void (*kernel)(Params...),
                 const Args&... args)
{
  const int rc = set_smem_bytes(reinterpret_cast<const void*>(kernel), l.smem_bytes, err);
  if (rc != B2FIL_OK) return rc;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg{};
  cfg.gridDim          = l.grid;
  cfg.blockDim         = dim3(l.threads);
  cfg.dynamicSmemBytes = l.smem_bytes;
  cfg.stream           = l.stream;
  cfg.attrs            = attr;
  if (l.cluster > 1) {
    attr[cfg.numAttrs].id             = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim = {static_cast<unsigned>(l.cluster), 1, 1};
    ++cfg.numAttrs;
  }
  if (l.overlap) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
    ++cfg.numAttrs;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  if (e != cudaSuccess) {
    cudaGetLastError();
    err = std::string("kernel launch: ") + cudaGetErrorString(e);
    return B2FIL_ERR_CUDA;
  }
  return B2FIL_OK;
}
// What the quantised traversal kernels take beside the prediction itself; passed by value.
struct QArgs {
  const uint16_t* Q;      // rank image of the chunk
  // which tiles hold a NaN: flag_words 32-bit words per tile, any of them non-zero
  const uint32_t* flags;
  int32_t flag_words;
  // Reduced outputs of a balanced launch (see dense_q_body): sums of row tiles that several CTAs
  // share, [2 per CTA][output][row] of the forest precision, and per tile the tree batches that
  // have arrived (zeroed by the pre-pass).  Null: every row tile belongs to one CTA.
  void* partial;
  int32_t* arrived;
  int32_t R, G, S, K;
  int32_t tile_bufs;      // row-tile buffers: 2 bring the next tile in during the walk of this one
  int32_t nan_columns;    // 1: tiles with missing values are walked with doubled columns (room for them)
  int32_t acc_bufs;       // sets of accumulators: with 2 the CTA meets once per tile, not twice
};

// One launch of a quantised traversal kernel.
struct QLaunch {
  PredictParams p;
  QArgs q;
  DenseCfg c;
  int grid;
  cudaStream_t stream;
  SplitLaunch shape() const
  {
    return SplitLaunch{dim3(grid), c.threads, c.smem_bytes, stream, 1, true};
  }
};

// CTAs of a launch in clusters of `cluster` that run at the same time, one per SM.  Clusters live
// inside one GPC, so the larger they are the more SMs stay idle: measured on 148 SMs, 148 CTAs in
// pairs, 132 in fours, 120 in eights.
inline int cluster_ctas(int sm_count, int cluster)
{
  const double usable = cluster <= 2 ? 1.0 : (cluster <= 4 ? 0.893 : 0.811);
  return static_cast<int>(sm_count * usable) / cluster * cluster;
}
constexpr int kMaxCluster = 8;  // largest portable cluster

// fp32, scalar leaves, no categorical tests, depth 4..10, six trees in flight; `top6` takes the
// top nodes of every tree from p.q_top (at most kQTopTrees trees).
int launch_q_top6(const QLaunch& L, std::string& err);
int launch_q_plain6(const QLaunch& L, std::string& err);
// The same with vector leaves, and (four trees in flight) with one output per row and tree.
int launch_q_top_vec(const QLaunch& L, std::string& err);
int launch_q_top_out(const QLaunch& L, int mode, std::string& err);
// One output per row and tree, four trees in flight, top nodes in the stages (more than kQTopTrees trees).
int launch_q_out4(const QLaunch& L, int mode, std::string& err);
// fp32, scalar leaves, no categorical tests, depth 4..10, four trees in flight.
int launch_q_plain4(const QLaunch& L, std::string& err);
// fp32, no categorical tests, depth 4..10, one or two trees in flight, every output mode.
int launch_q_narrow(const QLaunch& L, int mode, std::string& err);
// fp32, vector leaves, no categorical tests, depth 4..10, six or four trees in flight.
int launch_q_vec(const QLaunch& L, std::string& err);
// fp32, scalar leaves, no categorical tests, any depth, 1, 2 or 4 trees in flight: the walk that
// fetches both children of a node ahead of the test (for launch shapes with few walks in flight).
int launch_q_pair(const QLaunch& L, std::string& err);
// fp32 scalar leaves of depth 9 and 10, two to four trees in flight, payloads left in global memory.
int launch_q_leafg(const QLaunch& L, std::string& err);
// Forests with categorical tests: every precision, output mode and depth; 1, 2 or 4 trees in
// flight (depth-specialised bodies for fp32 scalar leaves of depth 4..8 with four and six trees).
int launch_q_cat(const QLaunch& L, int mode, bool f64, std::string& err);
// Forests that q_walk_order() leaves in heap order, without categorical tests: depth read at run time, every
// precision and output mode; 1, 2 or 4 trees in flight.
int launch_q_generic(const QLaunch& L, int mode, bool f64, std::string& err);

// Sparse forests with a compact image (kernels_sparse_c.cu).
constexpr int kCompactTreesInFlight = 4;
struct CompactCfg {
  int rows_per_tile;  // R
  int tree_groups;    // G
  int stages;         // S: depth of the ring of heap batches
  size_t smem_bytes;
  int threads;
  int grid;
  int splits;         // CTAs that share the tree batches of a row tile (small batches), else 1
};
// Value of a named tuning knob (b2fil_set_tuning), or `fallback` when it was never set.
int tuning_value(const char* key, int fallback);
void set_tuning_value(const char* key, int value);
// Launch shape for `n_rows` rows starting from tiles of `rows_per_tile`; false when the forest has
// no compact image or no shape fits shared memory (the plain sparse kernel runs then).
// `may_split`: small batches may split the forest over CTAs.
bool compact_config(const ForestView& f, bool reduce, int rows_per_tile, int64_t n_rows,
                    int sm_count, bool may_split, CompactCfg& cfg);
int launch_sparse_compact(const PredictParams& p, int mode, const CompactCfg& c,
                          cudaStream_t stream, std::string& err);

}  // namespace b2fil
