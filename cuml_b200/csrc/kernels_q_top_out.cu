// dense_q_top_kernel<float, leaf ids or per-tree outputs, 8 or 4 trees in flight, depth 4..10>: unrolled walks with
// the top nodes in the parameter block, one output per (row, tree).  Multiples of four trees because a row's
// four outputs leave together.
#include "dense_q.cuh"

namespace b2fil {
int launch_q_top_out(const QLaunch& L, int mode, std::string& err)
{
  if (L.c.trees_in_flight == 8)
    return mode == MODE_LEAFID ? launch_q_top_depth<float, MODE_LEAFID, 8>(L, err)
                               : launch_q_top_depth<float, MODE_PERTREE, 8>(L, err);
  return mode == MODE_LEAFID ? launch_q_top_depth<float, MODE_LEAFID, 4>(L, err)
                             : launch_q_top_depth<float, MODE_PERTREE, 4>(L, err);
}
}  // namespace b2fil
