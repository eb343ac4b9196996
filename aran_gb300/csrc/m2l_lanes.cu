// m2l_lanes.cu -- dispatch of the lane-parallel M2L (m2l_lanes.cuh) and its
// instances at the orders 4, 8 and 12; the other even orders compile beside
// it in m2l_lanes_b.cu and m2l_lanes_c.cu.
#include "m2l_lanes.cuh"

namespace aran {

// Runs the M2L pass with the lane-parallel kernel when the order has one;
// false leaves it to m2l.cu.
bool launch_m2l_lanes(AranGpuSolver3d *s, OpTables<float> &tb, const int *parents, int count,
                      const cplx<float> *mult, cplx<float> *loc, cudaStream_t st) {
  const int p = s->cfg.order;
  if (!m2l_hk_order(p) || tb.dir_lanes.ptr == nullptr || count <= 0) return false;
  switch (p) {
    case 4: return launch_p<4>(s, tb, parents, count, mult, loc, st);
    case 8: return launch_p<8>(s, tb, parents, count, mult, loc, st);
    case 12: return launch_p<12>(s, tb, parents, count, mult, loc, st);
    case 16: return launch_m2l_lanes_c(s, tb, parents, count, mult, loc, st);
    default: return launch_m2l_lanes_b(s, tb, parents, count, mult, loc, st);
  }
}

}  // namespace aran
