// dense_q_top_kernel<float, vector leaves, 6 trees in flight, depth 4..10>: random-forest classifiers.
// The shared-memory pipe bounds the walk; the top nodes in the parameter block take two of its
// wavefronts per (warp, tree) away, like for scalar leaves, and the two classes of a binary leaf come
// with one load (100 depth-8 trees, 2 classes, 1 M rows, traversal: 377 -> 308 us).
#include "dense_q.cuh"

namespace b2fil {
int launch_q_top_vec(const QLaunch& L, std::string& err)
{
  return launch_q_top_depth<float, MODE_VECTOR, 6>(L, err);
}
}  // namespace b2fil
