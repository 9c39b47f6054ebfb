// dense_q_kernel for forests with categorical tests.  Three shared-memory instructions per visit (node,
// rank, predicated category set) bound the walk; with six trees in flight the pipe is busy 90 % of the
// time instead of 84 % (150,000 rows of 5000 depth-6 trees, 5 % NaN: 2022 -> 1890 us).
#include "dense_q.cuh"

namespace b2fil {
namespace {
template <typename T>
int launch_cat(const QLaunch& L, int mode, std::string& err)
{
  switch (L.c.trees_in_flight) {
    case 4: return launch_q_modes<T, 4, true>(L, mode, err);
    case 2: return launch_q_modes<T, 2, true>(L, mode, err);
    default: return launch_q_modes<T, 1, true>(L, mode, err);
  }
}
template <int NT>
int launch_cat_depth(const QLaunch& L, std::string& err)
{
  switch (L.p.f.dense_depth) {
    case 4: return launch_q<float, MODE_SCALAR, NT, 4, true>(L, err);
    case 5: return launch_q<float, MODE_SCALAR, NT, 5, true>(L, err);
    case 6: return launch_q<float, MODE_SCALAR, NT, 6, true>(L, err);
    case 7: return launch_q<float, MODE_SCALAR, NT, 7, true>(L, err);
    default: return launch_q<float, MODE_SCALAR, NT, 8, true>(L, err);
  }
}
}  // namespace

int launch_q_cat(const QLaunch& L, int mode, bool f64, std::string& err)
{
  // fp32 scalar leaves: depth-specialised bodies
  if (!f64 && mode == MODE_SCALAR && L.c.trees_in_flight == 6) return launch_cat_depth<6>(L, err);
  if (!f64 && mode == MODE_SCALAR && L.c.trees_in_flight == 4 && L.p.f.dense_depth >= 4 &&
      L.p.f.dense_depth <= 8)
    return launch_cat_depth<4>(L, err);
  return f64 ? launch_cat<double>(L, mode, err) : launch_cat<float>(L, mode, err);
}
}  // namespace b2fil
