// leaf_ops.cu -- dispatch of the FP32 P2M and L2P (leaf_ops.cuh) and their instances
// at the orders 4, 8 and 12.
#include "leaf_ops.cuh"

namespace aran {

bool launch_leaf_p2m(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 4: leaf_p2m<4>(s, st); return true;
    case 8: leaf_p2m<8>(s, st); return true;
    case 12: leaf_p2m<12>(s, st); return true;
    case 6:
    case 10:
    case 14: return launch_leaf_p2m_b(s, st);
    case 16: return launch_leaf_p2m_c(s, st);
    default: return false;
  }
}

bool launch_leaf_l2p(AranGpuSolver3d *s, cudaStream_t st) {
  switch (s->cfg.order) {
    case 4: leaf_l2p<4>(s, st); return true;
    case 8: leaf_l2p<8>(s, st); return true;
    case 12: leaf_l2p<12>(s, st); return true;
    case 6:
    case 10:
    case 14: return launch_leaf_l2p_b(s, st);
    case 16: return launch_leaf_l2p_c(s, st);
    default: return false;
  }
}

}  // namespace aran
