// dense_q_kernel<float, every output mode, depth 4..10, no categorical tests> with one or two trees in flight: shapes
// of which shared memory holds few trees next to the row tile.  And four trees in flight with one output per row
// and tree, for forests of more than kQTopTrees trees.
#include "dense_q.cuh"

namespace b2fil {
namespace {
template <int MODE, int NT>
int launch_depth(const QLaunch& L, std::string& err)
{
  switch (L.p.f.dense_depth) {
    case 4: return launch_q<float, MODE, NT, 4, false>(L, err);
    case 5: return launch_q<float, MODE, NT, 5, false>(L, err);
    case 6: return launch_q<float, MODE, NT, 6, false>(L, err);
    case 7: return launch_q<float, MODE, NT, 7, false>(L, err);
    case 8: return launch_q<float, MODE, NT, 8, false>(L, err);
    case 9: return launch_q<float, MODE, NT, 9, false>(L, err);
    default: return launch_q<float, MODE, NT, 10, false>(L, err);
  }
}
template <int NT>
int launch_mode(const QLaunch& L, int mode, std::string& err)
{
  switch (mode) {
    case MODE_SCALAR: return launch_depth<MODE_SCALAR, NT>(L, err);
    case MODE_VECTOR: return launch_depth<MODE_VECTOR, NT>(L, err);
    case MODE_PERTREE: return launch_depth<MODE_PERTREE, NT>(L, err);
    default: return launch_depth<MODE_LEAFID, NT>(L, err);
  }
}
}  // namespace

int launch_q_out4(const QLaunch& L, int mode, std::string& err)
{
  return mode == MODE_LEAFID ? launch_depth<MODE_LEAFID, 4>(L, err) : launch_depth<MODE_PERTREE, 4>(L, err);
}
int launch_q_narrow(const QLaunch& L, int mode, std::string& err)
{
  return L.c.trees_in_flight == 2 ? launch_mode<2>(L, mode, err) : launch_mode<1>(L, mode, err);
}
}  // namespace b2fil
