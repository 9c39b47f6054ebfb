// dense_q_leafg_kernel: fp32 scalar leaves without categorical tests, depth 9 and 10, two to four
// trees in flight, leaf payloads fetched from global memory instead of riding in the stages.
#include "dense_q.cuh"

namespace b2fil {
namespace {
template <int NT, int DEPTH>
int launch_leafg(const QLaunch& L, std::string& err)
{
  // (the parameter block costs a launch 2.5 us)
  if (L.p.q_top != nullptr && L.p.n_rows * L.p.f.n_trees * DEPTH > int64_t(200) << 20) {
    void (*k)(const PredictParams, const QArgs, const QTop) = dense_q_leafg_kernel<NT, DEPTH>;
    return launch_split(L.shape(), err, k, L.p, L.q, top_nodes(L));
  }
  void (*k)(const PredictParams, const QArgs) = dense_q_leafg_kernel<NT, DEPTH>;
  return launch_split(L.shape(), err, k, L.p, L.q);
}

template <int DEPTH>
int launch_leafg_depth(const QLaunch& L, std::string& err)
{
  switch (L.c.trees_in_flight) {
    case 4: return launch_leafg<4, DEPTH>(L, err);
    case 3: return launch_leafg<3, DEPTH>(L, err);
    default: return launch_leafg<2, DEPTH>(L, err);
  }
}
}  // namespace

int launch_q_leafg(const QLaunch& L, std::string& err)
{
  return L.p.f.dense_depth == 9 ? launch_leafg_depth<9>(L, err) : launch_leafg_depth<10>(L, err);
}
}  // namespace b2fil
