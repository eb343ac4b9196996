// m2m_lanes.cu -- tables and dispatch of the lane-parallel M2M and L2L
// (m2m_lanes.cuh) and their instances at the orders 4, 8 and 12; the other
// even orders compile beside it in m2m_lanes_b.cu and m2m_lanes_c.cu.
#include "m2m_lanes.cuh"

namespace aran {

namespace {

// the stream table of one kind from octant 0's FP32 direction table (layout
// of tables.cu, kind 1 or 2) and the vertical factors (vm or vl)
__global__ void k_oct_lane_tables(int p, int down, const float *__restrict__ dir, int ef, int of,
                                  int ei, int oi, int ph, int rp, const float *__restrict__ vert,
                                  float *__restrict__ dst) {
  const int LD = down ? p + 1 : p;
  const int NR = oct_sq(LD), NV = oct_tet(LD);
  const int FW = (2 * (p + 1) + 3) & ~3;
  const int VT = FW + 8 * ((NR + 3) / 4), BW = VT + 4 * ((NV + 3) / 4);
  const int stride = BW + 8 * ((NR + 3) / 4);
  for (int e = threadIdx.x; e < stride; e += blockDim.x) {
    float v = 0.f;
    if (e < FW) {
      if (e < 2 * (p + 1)) v = dir[ph + e];
    } else if (e < VT || e >= BW) {
      const int q = e < VT ? e - FW : e - BW;
      const int t = 4 * (q >> 3) + (q & 3), part = (q >> 2) & 1;
      // term t of the (l, m', m) order sits at sq_off(l) + m' (l+1) + m = t
      if (t < NR) v = dir[(e < VT ? (part ? of : ef) : (part ? oi : ei)) + t];
    } else if (e - VT < NV) {
      const int t = e - VT;
      for (int m = 0; m < LD; ++m)
        for (int l = m; l < LD; ++l) {
          const int n0 = down ? l : m, n1 = down ? LD - 1 : l;
          for (int n = n0; n <= n1; ++n)
            if (oct_vidx(LD, down != 0, m, l, n) == t)
              v = down ? vert[oct_tri(l) * (p + 1) + m * (p + 1) + n] * dir[rp + n - l]
                       : vert[(oct_tri(l) + m) * p + n] * dir[rp + l - n];
        }
    }
    dst[e] = v;
  }
}

}  // namespace

void build_oct_lane_tables(OpTables<float> &tb, cudaStream_t st) {
  const int p = tb.p;
  if (!m2l_hk_order(p)) return;
  for (int down = 0; down < 2; ++down) {
    const int LD = down ? p + 1 : p;
    const int NR = oct_sq(LD), NV = oct_tet(LD);
    const int FW = (2 * (p + 1) + 3) & ~3;
    const int stride = FW + 8 * ((NR + 3) / 4) + 4 * ((NV + 3) / 4) + 8 * ((NR + 3) / 4);
    const int kind = down ? 2 : 1;
    DBuf<float> &dst = tb.oct_lanes[down];
    dst.reserve(stride);
    k_oct_lane_tables<<<1, 256, 0, st>>>(
        p, down, down ? tb.dir_l2l.ptr : tb.dir_m2m.ptr, dir_offset(p, kind, 0),
        dir_offset(p, kind, 1), dir_offset(p, kind, 2), dir_offset(p, kind, 3),
        dir_offset(p, kind, 4), dir_offset(p, kind, 5), down ? tb.vl.ptr : tb.vm.ptr, dst.ptr);
    ACHECK(cudaGetLastError());
  }
}

bool launch_m2m_lanes(AranGpuSolver3d *s, OpTables<float> &tb, cplx<float> *mult, int dhi,
                      int dlo, cudaStream_t st) {
  if (!m2l_hk_order(tb.p) || tb.oct_lanes[0].ptr == nullptr) return false;
  const float *tab = tb.oct_lanes[0].ptr;
  switch (tb.p) {
    case 4: launch_levels<4, false>(s, tab, mult, dhi, dlo, st); return true;
    case 8: launch_levels<8, false>(s, tab, mult, dhi, dlo, st); return true;
    case 12: launch_levels<12, false>(s, tab, mult, dhi, dlo, st); return true;
    case 16: launch_oct_lanes_c(s, false, tab, mult, dhi, dlo, st); return true;
    default: launch_oct_lanes_b(s, false, tab, mult, dhi, dlo, st); return true;
  }
}

// child depths dlo (at least 3) up to dhi
bool launch_l2l_lanes(AranGpuSolver3d *s, OpTables<float> &tb, cplx<float> *loc, int dlo,
                      int dhi, cudaStream_t st) {
  // order 6 stays with passes.cu's kernel: the same time on 4M particles (0.20
  // ms), 0.023 against 0.039 ms on 200k
  if (!m2l_hk_order(tb.p) || tb.p == 6 || tb.oct_lanes[1].ptr == nullptr) return false;
  const int d0 = (dlo < 3 ? 3 : dlo) - 1, d1 = dhi - 1;
  const float *tab = tb.oct_lanes[1].ptr;
  switch (tb.p) {
    case 4: launch_levels<4, true>(s, tab, loc, d0, d1, st); return true;
    case 8: launch_levels<8, true>(s, tab, loc, d0, d1, st); return true;
    case 12: launch_levels<12, true>(s, tab, loc, d0, d1, st); return true;
    case 16: launch_oct_lanes_c(s, true, tab, loc, d0, d1, st); return true;
    default: launch_oct_lanes_b(s, true, tab, loc, d0, d1, st); return true;
  }
}

}  // namespace aran
