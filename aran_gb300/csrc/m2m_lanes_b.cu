// m2m_lanes_b.cu -- the lane-parallel M2M and L2L at the orders 10 and 14, and
// the M2M at order 6.
#include "m2m_lanes.cuh"

namespace aran {

void launch_oct_lanes_b(AranGpuSolver3d *s, bool down, const float *tab, cplx<float> *ser, int d0,
                        int d1, cudaStream_t st) {
  switch (s->cfg.order) {
    case 6:
      if (!down) launch_levels<6, false>(s, tab, ser, d0, d1, st);
      break;
    case 10:
      down ? launch_levels<10, true>(s, tab, ser, d0, d1, st)
           : launch_levels<10, false>(s, tab, ser, d0, d1, st);
      break;
    default:
      down ? launch_levels<14, true>(s, tab, ser, d0, d1, st)
           : launch_levels<14, false>(s, tab, ser, d0, d1, st);
  }
}

}  // namespace aran
