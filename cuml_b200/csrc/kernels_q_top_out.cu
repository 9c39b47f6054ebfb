// dense_q_top_kernel<float, leaf ids or per-tree outputs, 4 trees in flight, depth 4..10>: unrolled
// walks with the top nodes in the parameter block, one output per (row, tree).  Four trees because
// a row's four outputs leave together.
#include "dense_q.cuh"

namespace b2fil {
int launch_q_top_out(const QLaunch& L, int mode, std::string& err)
{
  return mode == MODE_LEAFID ? launch_q_top_depth<float, MODE_LEAFID, 4>(L, err)
                             : launch_q_top_depth<float, MODE_PERTREE, 4>(L, err);
}
}  // namespace b2fil
