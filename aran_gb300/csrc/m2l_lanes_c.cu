// m2l_lanes_c.cu -- the lane-parallel M2L at order 16.
#include "m2l_lanes.cuh"

namespace aran {

bool launch_m2l_lanes_c(AranGpuSolver3d *s, OpTables<float> &tb, const int *parents, int count,
                        const cplx<float> *mult, cplx<float> *loc, cudaStream_t st) {
  return launch_p<16>(s, tb, parents, count, mult, loc, st);
}

}  // namespace aran
