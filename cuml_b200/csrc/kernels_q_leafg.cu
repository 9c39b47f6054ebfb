// dense_q_leafg_kernel: fp32 scalar leaves without categorical tests, depth 9 and 10, two to four
// trees in flight, leaf payloads fetched from global memory instead of riding in the stages.
#include "dense_q.cuh"

namespace b2fil {
namespace {
template <int NT, int DEPTH>
int launch_leafg(const QLaunch& L, std::string& err)
{
  if (L.p.q_top != nullptr && L.p.f.n_trees <= kQTopFew)
    return launch_split(L.shape(), err, dense_q_leafg_kernel<NT, DEPTH, kQTopFew>, L.p, L.q, top_nodes<kQTopFew>(L));
  // (the launch of the large parameter block takes what it saves in calls of less than about 100 us)
  if (L.p.q_top != nullptr && L.p.n_rows * L.p.f.n_trees * DEPTH > int64_t(200) << 20)
    return launch_split(L.shape(), err, dense_q_leafg_kernel<NT, DEPTH, kQTopTrees>, L.p, L.q,
                        top_nodes<kQTopTrees>(L));
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
