// m2l_lanes_b.cu -- the lane-parallel M2L at the orders 6, 10 and 14.
#include "m2l_lanes.cuh"

namespace aran {

bool launch_m2l_lanes_b(AranGpuSolver3d *s, OpTables<float> &tb, const int *parents, int count,
                        const cplx<float> *mult, cplx<float> *loc, cudaStream_t st) {
  switch (s->cfg.order) {
    case 6: return launch_p<6>(s, tb, parents, count, mult, loc, st);
    case 10: return launch_p<10>(s, tb, parents, count, mult, loc, st);
    case 14: return launch_p<14>(s, tb, parents, count, mult, loc, st);
    default: return false;
  }
}

}  // namespace aran
