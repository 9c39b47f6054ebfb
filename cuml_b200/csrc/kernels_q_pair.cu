// dense_q_pair_kernel: fp32 scalar leaves without categorical tests, generic depth, 1, 2 or 4
// trees in flight, both children of a node fetched ahead of the test.
#include "dense_q.cuh"

namespace b2fil {
namespace {
template <int NT>
int launch_pair(const QLaunch& L, std::string& err)
{
  auto k = q_walk_order(L.p.f) ? dense_q_pair_kernel<NT, false> : dense_q_pair_kernel<NT, true>;
  return launch_split(L.shape(), err, k, L.p, L.q);
}
}  // namespace

int launch_q_pair(const QLaunch& L, std::string& err)
{
  switch (L.c.trees_in_flight) {
    case 4: return launch_pair<4>(L, err);
    case 2: return launch_pair<2>(L, err);
    default: return launch_pair<1>(L, err);
  }
}
}  // namespace b2fil
