// leaf_ops_c.cu -- the FP32 P2M and L2P at order 16.
#include "leaf_ops.cuh"

namespace aran {

bool launch_leaf_p2m_c(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 16: leaf_p2m<16>(s, st); return true;
    default: return false;
  }
}

bool launch_leaf_l2p_c(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 16: leaf_l2p<16>(s, st); return true;
    default: return false;
  }
}

}  // namespace aran
