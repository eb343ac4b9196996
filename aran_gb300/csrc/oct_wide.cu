// oct_wide.cu -- M2M and L2L with a thread per part of a coefficient, for
// levels of few nodes and for FP64 (operators as in m2m_lanes.cuh and passes.cu:
// aran_development3d_m2m_rotate, arandevelopment3d.c:402-409, and
// aran_development3d_l2l_rotate, :444-451).
//
// A level of few nodes is bound by the latency of one translation: the
// lane-parallel kernels run it in one warp, thousands of unrolled instructions
// that are fetched once (42 us a level at order 16, 20 at order 12).  Here a CTA
// takes one (parent, octant): thread 2c + h makes part h (real, imaginary) of
// coefficient c through z-phase, rotation, translation along z, rotation back
// and conjugate phase, each a sum of at most p + 1 products over shared memory
// with its factors' loads in flight together.  M2M's eight octants are
// threads of one CTA where it holds them (up to order 10: order 8 7.5 us a level,
// 10 with the lane-parallel kernel or a cluster), else the CTAs of a cluster,
// which sum their parts in octant order from each other's shared memory.
//
// In FP32 every sum runs over the same tables (octant 0's stream table, the
// octant's mirror applied on the way in and out) with the same operations in
// the same order as k_oct_lanes, so both give the same bits and the number of
// nodes in a level, which depends on what else is solved, picks the kernel.
// In FP64 (the octant's own table) it serves every level: half as many lanes
// idle on the FP64 pipe as with a warp per child (200k Plummer particles at
// order 12: M2M 0.63 -> 0.49 ms, L2L 1.4 ms either way).
#include <cooperative_groups.h>

#include "internal.cuh"

namespace cg = cooperative_groups;

namespace aran {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ constexpr int w_tet(int k) { return k * (k + 1) * (k + 2) / 6; }
__host__ __device__ constexpr int w_sq(int l) { return l * (l + 1) * (2 * l + 1) / 6; }

// factors of a translation: a stream table of octant 0 (FP32, the layout of
// m2m_lanes.cuh) or an octant's direction table (FP64, the layout of tables.cu)
struct WideTab {
  const void *base;             // stream table / direction tables
  int fw, vt, bw;               // stream: sections
  int ef, of, ei, oi, ph, rp, stride;   // direction table
  const void *vert;             // direction: vertical factors (vm or vl)
};

// ONE: M2M with the eight octants' threads in one CTA (tpo threads each)
template <typename T, bool DOWN, bool ONE>
__global__ void k_oct_wide(int off, const int *__restrict__ list, const int *__restrict__ child,
                           const int *__restrict__ begin, const int *__restrict__ end, int p,
                           WideTab tb, int tpo, const uint8_t *__restrict__ lm,
                           cplx<T> *__restrict__ ser) {
  extern __shared__ unsigned char smem_raw[];
  constexpr bool STREAM = sizeof(T) == 4;
  const int LD = DOWN ? p + 1 : p, NC = tri(LD);
  const int o = ONE ? threadIdx.x / tpo : blockIdx.x;
  const int i = ONE ? threadIdx.x - o * tpo : threadIdx.x, c = i >> 1, h = i & 1;
  T *x = reinterpret_cast<T *>(smem_raw) + (ONE ? 4 * NC * o : 0), *y = x + 2 * NC;
  const int par = list ? list[blockIdx.y] : off + (int)blockIdx.y;
  const int c0 = child[par];
  if (c0 < 0) return;                       // the whole cluster
  const int ch = c0 + o;
  const bool live = end[ch] > begin[ch];
  const bool mine = c < NC;
  const int l = mine ? lm[2 * c] : 0, m = mine ? lm[2 * c + 1] : 0;
  // octant 0's table serves the others through the mirror images
  const int bx = STREAM ? o & 1 : 0, by = STREAM ? (o >> 1) & 1 : 0, bz = STREAM ? o >> 2 : 0;
  const T *t0 = static_cast<const T *>(tb.base) + (STREAM ? 0 : (size_t)o * tb.stride);
  const T ec = t0[(STREAM ? 0 : tb.ph) + 2 * m], es = t0[(STREAM ? 0 : tb.ph) + 2 * m + 1];
  // rotation terms (l, m', m) t = w_sq(l) + m' (l + 1) + m
  auto rotate = [&](const T *in, bool back) -> T {
    const int tt = w_sq(l) + m * (l + 1);
    const T *f = STREAM ? t0 + (back ? tb.bw : tb.fw) + 4 * h
                        : t0 + (back ? (h ? tb.oi : tb.ei) : (h ? tb.of : tb.ef)) + tt;
    const T *s = in + 2 * tri(l) + h;
    T acc = 0;
#pragma unroll 6
    for (int k = 0; k <= l; ++k) {
      const int t = tt + k;
      acc = fma(STREAM ? f[8 * (t >> 2) + (t & 3)] : f[k], s[2 * k], acc);
    }
    return acc;
  };
  const bool work = live && mine;
  if (work) {
    const cplx<T> v = ser[(size_t)(DOWN ? par : ch) * NC + c];
    const T g = ((bx ^ bz) & m & 1) ? (T)-1 : (T)1;
    const T cj = (bx ^ by) ? -g : g;
    const T pa = g * (h ? es : ec), pb = cj * (h ? ec : -es);
    const T sn = (bz && (l & 1)) ? (T)-1 : (T)1;
    x[i] = sn * fma(v.re, pa, v.im * pb);
  }
  __syncthreads();
  if (work) y[i] = rotate(x, false);
  __syncthreads();
  T z = 0;
  if (work) {
    // translation along z: order m, output degree l, source degrees n
    const int n0 = DOWN ? l : m, n1 = DOWN ? LD - 1 : l;
    const T *vf = nullptr, *rp = t0 + tb.rp;
    if (STREAM)
      vf = t0 + tb.vt + w_tet(LD) - w_tet(LD - m) +
           (DOWN ? tri(LD - m) - tri(LD - l) - l : tri(l - m) - m);
    else
      vf = static_cast<const T *>(tb.vert) + (size_t)c * (DOWN ? p + 1 : p);
#pragma unroll 6
    for (int n = n0; n <= n1; ++n)
      z = fma(STREAM ? vf[n] : vf[n] * rp[DOWN ? n - l : l - n], y[2 * tri(n, m) + h], z);
  }
  __syncthreads();
  if (work) x[i] = z;
  __syncthreads();
  const T a = work ? rotate(x, true) : (T)0;
  // conjugate z-phase, mirror on the way out
  const T b = __shfl_xor_sync(kFull, a, 1);
  T v = fma(a, ec, b * (h ? -es : es));
  if (((bz & (l + m)) ^ (bx & m) ^ (h & (bx ^ by))) & 1) v = -v;
  if (DOWN) {
    if (work) reinterpret_cast<T *>(ser)[(size_t)ch * 2 * NC + i] += v;
  } else if (ONE) {
    // the eight octants' parts in order
    if (mine) y[i] = live ? v : (T)0;
    __syncthreads();
    const T *all = reinterpret_cast<const T *>(smem_raw) + 2 * NC;
    for (int k = threadIdx.x; k < 2 * NC; k += blockDim.x) {
      T sum = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) sum += all[4 * NC * q + k];
      reinterpret_cast<T *>(ser)[(size_t)par * 2 * NC + k] = sum;
    }
  } else {
    // the eight octants' parts in order, each CTA an eighth of the values
    if (mine) y[i] = live ? v : (T)0;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    const int n = 2 * NC, per = (n + 7) / 8;
    for (int k = o * per + i; k < min(n, (o + 1) * per); k += blockDim.x) {
      T sum = 0;
#pragma unroll
      for (int r = 0; r < 8; ++r) sum += *cl.map_shared_rank(y + k, r);
      reinterpret_cast<T *>(ser)[(size_t)par * n + k] = sum;
    }
    cl.sync();                              // nobody leaves while its parts are read
  }
}

template <typename T, bool DOWN>
void launch(AranGpuSolver3d *s, const WideTab &tb, const uint8_t *lm, cplx<T> *ser, int cnt,
            int off, const int *list, cudaStream_t st) {
  DevTree &t = s->tree;
  const int p = s->cfg.order, NC = tri(DOWN ? p + 1 : p);
  // M2M: one CTA for a parent's octants where its threads hold them (order 10)
  const int tpo = (2 * NC + 31) & ~31;
  const bool one = !DOWN && 8 * tpo <= 1024;
  const size_t sm = (size_t)4 * NC * sizeof(T) * (one ? 8 : 1);
  auto kern = one ? k_oct_wide<T, DOWN, !DOWN> : k_oct_wide<T, DOWN, false>;
  // grid.y holds 65,535 nodes at most
  for (int b = 0; b < cnt; b += 65535) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(one ? 1 : 8, cnt - b < 65535 ? cnt - b : 65535);
    cfg.blockDim = dim3(one ? 8 * tpo : tpo);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = DOWN || one ? 1 : 8;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    ACHECK(cudaLaunchKernelEx(&cfg, kern, off + (list ? 0 : b),
                              (const int *)(list ? list + b : nullptr),
                              (const int *)t.child.ptr, (const int *)t.begin.ptr,
                              (const int *)t.end.ptr, p, tb, tpo, lm, ser));
    s->launches++;
  }
}

}  // namespace

void launch_oct_wide(AranGpuSolver3d *s, bool down, const float *stream, cplx<float> *ser,
                     int cnt, int off, const int *list, cudaStream_t st) {
  const int p = s->cfg.order, LD = down ? p + 1 : p;
  WideTab tb = {};
  tb.base = stream;
  tb.fw = (2 * (p + 1) + 3) & ~3;
  tb.vt = tb.fw + 8 * ((w_sq(LD) + 3) / 4);
  tb.bw = tb.vt + 4 * ((w_tet(LD) + 3) / 4);
  const uint8_t *lm = s->t32.lm.ptr;
  if (down) launch<float, true>(s, tb, lm, ser, cnt, off, list, st);
  else launch<float, false>(s, tb, lm, ser, cnt, off, list, st);
}

void launch_oct_wide64(AranGpuSolver3d *s, bool down, cplx<double> *ser, int cnt, int off,
                       const int *list, cudaStream_t st) {
  const int p = s->cfg.order, kind = down ? 2 : 1;
  OpTables<double> &t = s->t64;
  WideTab tb = {};
  tb.base = down ? t.dir_l2l.ptr : t.dir_m2m.ptr;
  tb.ef = dir_offset(p, kind, 0);
  tb.of = dir_offset(p, kind, 1);
  tb.ei = dir_offset(p, kind, 2);
  tb.oi = dir_offset(p, kind, 3);
  tb.ph = dir_offset(p, kind, 4);
  tb.rp = dir_offset(p, kind, 5);
  tb.stride = dir_offset(p, kind, 6);
  tb.vert = down ? t.vl.ptr : t.vm.ptr;
  if (down) launch<double, true>(s, tb, t.lm.ptr, ser, cnt, off, list, st);
  else launch<double, false>(s, tb, t.lm.ptr, ser, cnt, off, list, st);
}

}  // namespace aran
