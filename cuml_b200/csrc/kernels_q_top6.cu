// dense_q_top_kernel<float, scalar leaves, 6 trees in flight, depth 4..10>.
#include "dense_q.cuh"

namespace b2fil {
int launch_q_top6(const QLaunch& L, std::string& err)
{
  return launch_q_top_depth<float, MODE_SCALAR, 6>(L, err);
}
}  // namespace b2fil
