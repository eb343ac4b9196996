// leaf_ops_b.cu -- the FP32 P2M and L2P at the orders 6, 10 and 14.
#include "leaf_ops.cuh"

namespace aran {

bool launch_leaf_p2m_b(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 6: leaf_p2m<6>(s, st); return true;
    case 10: leaf_p2m<10>(s, st); return true;
    case 14: leaf_p2m<14>(s, st); return true;
    default: return false;
  }
}

bool launch_leaf_l2p_b(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 6: leaf_l2p<6>(s, st); return true;
    case 10: leaf_l2p<10>(s, st); return true;
    case 14: leaf_l2p<14>(s, st); return true;
    default: return false;
  }
}

}  // namespace aran
