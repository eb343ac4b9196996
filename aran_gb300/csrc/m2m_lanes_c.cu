// m2m_lanes_c.cu -- the lane-parallel M2M and L2L at order 16.
#include "m2m_lanes.cuh"

namespace aran {

void launch_oct_lanes_c(AranGpuSolver3d *s, bool down, const float *tab, cplx<float> *ser, int d0,
                        int d1, cudaStream_t st) {
  if (down) launch_levels<16, true>(s, tab, ser, d0, d1, st);
  else launch_levels<16, false>(s, tab, ser, d0, d1, st);
}

}  // namespace aran
