// m2l_lanes.cuh -- lane-parallel M2L for the FP32 path at the orders
// m2l_hk_order(p) accepts (even orders 4 to 16; one translation unit per
// group of orders instantiates it).  Same operator as m2l.cu (the "point and
// shoot" translation of aran_spherical_seriesd_to_local_rotate,
// aran/aransphericalseriesd-rotate.c:165-207, applied by far_func,
// aran/aransolver3d.c:333-354) with the work laid out the other way round:
//
//  * after the z-phase, the rotation, the translation along z and the
//    rotation back never mix real and imaginary parts (the even/odd Wigner
//    blocks act on the real/imaginary parts, the vertical factors are real),
//    so one lane carries the real part and its neighbour the imaginary part
//    of one (target, source) translation;
//  * a CTA takes the children of 16 to 32 parents, child by child, a lane
//    pair each, and all its lane pairs apply the same offset's table at a
//    time: every table read is a broadcast of 16 bytes (four factors) from
//    shared memory, and a lane's whole series stays in registers, the order
//    being a compile-time constant;
//  * child w = (bx, by, bz) reaches its sources through the offsets with
//    d_x in [bx-3, bx+2] (same for y, z); the mirror image sigma_w (x -> -x
//    where bx = 1, likewise y, z) maps them onto child 0's 189 offsets, and
//    the translation obeys T_d = S T_{sigma d} S, with S the action of the
//    mirror on series: (l, m) -> (-1)^{l+m} on a z flip, conjugation on a y
//    flip, (-1)^m conjugation on an x flip.  So all warps walk child 0's
//    offsets together, each lane pair applying its child's S to its sources
//    on the way in and once to its accumulated locals on the way out: every
//    table in the ring serves the whole CTA;
//  * the translation along z runs in the scaled frame of m2l_hk_* (fmm_math
//    .cuh), where its factor depends on j + n alone and is a constant of the
//    code: no table is read for it, and the orders m, m + 1 go through
//    packed FP32 pairs (fma.rn.f32x2), one instruction for two products;
//  * the two lanes of a pair exchange their rotated-back parts with one
//    shuffle to apply the conjugate z-phase, in the same offset order for
//    every run.  The sums over the offsets live in registers up to order 6
//    and in tensor memory above (a warp's lanes are 32 rows of its quarter,
//    one column per coefficient): the registers they would take hold more
//    warps instead, sums in shared memory would take the bandwidth that the
//    table broadcasts need and, from order 14, more room than there is.
//
// What bounds it: latency and issue, with two to four warps per scheduler (at
// order 12 the FMA pipes are active 54 % of the cycles, 63 % of the issue
// slots are used, shared memory moves data in 49 %).  Measured on GB300, M2L
// of a 4 M-particle Plummer set (leaf 64, 38.9 M translations): order 12
// 11.6 ms (14.3 with the vertical factors in the table stream, the sums in
// shared memory and 8 warps a CTA; with 8 warps and the rest as now 0.4 more;
// with neighbouring degrees packed through the rotations too 0.5 more, the
// packing's moves costing what the products saved), order 8 5.0 ms (6.5),
// order 16 25.8 ms, order 10 7.9 ms and order 6 3.2 ms (about 118, 42 and 20
// with the kernel of m2l.cu, whose lanes run over one translation's
// coefficients).
//
// The offset tables stream through a three-slot ring of TMA bulk copies;
// the next offset's source multipoles are brought into shared memory by one
// bulk copy each while the current one is translated.  Every mbarrier
// wait is bounded; a wait that gives up sets the error word and the CTA
// stops.
//
// A target's sum is the sum of 8 or 16 segments of the offset list, each summed
// on its own: a pass with few parents, which would leave most SMs idle (one
// CTA takes its parents through up to 189 offsets in turn), gives the
// segments to several CTAs, which leave their sums in a workspace for
// k_m2l_lanes_sum to add (10k uniform particles, order 8, leaf 20: 0.11 ms,
// 0.55 in one part); a pass with many parents adds them up as it goes.  So
// the result does not depend on how many CTAs share a target's offsets: a
// system solved alone, in a forest or beside others gets the same bits.
#pragma once

#include "internal.cuh"
#include "async.cuh"
#include "f32x2.cuh"
#include "tcgen05.cuh"

namespace aran {

namespace {

constexpr int kLaneNst = 3;      // table ring slots
constexpr unsigned kFull = 0xffffffffu;

// first packed pair of degree l: pairs (l, 2k), (l, 2k + 1), k = 0..l/2
__host__ __device__ constexpr int lane_pair(int l) {
  return ((l + 1) / 2) * ((l + 1) / 2 + 1) - ((l & 1) ? (l + 1) / 2 : 0);
}

// column of (l, m) among a target's sums
__host__ __device__ constexpr int lane_col(int l, int m) { return 2 * lane_pair(l) + m; }

template <int P>
struct LaneDims {
  static constexpr int NM = P * (P + 1) / 2;        // multipole coefficients
  static constexpr int NL = (P + 1) * (P + 2) / 2;  // local coefficients
  // the source rows are copied whole 16-byte units at a time: an odd NM
  // takes one coefficient more and starts 8 bytes early at odd nodes; rows
  // are an odd number of 16-byte units apart, so the 16 lane pairs' reads
  // spread over the banks
  static constexpr bool ODD = (NM & 1) != 0;
  static constexpr int NMC = NM + (ODD ? 1 : 0);
  static constexpr int NMP = ((NMC / 2) | 1) * 2;
  static constexpr int STRIDE = m2l_hk_stride(P);
  static constexpr int NP = lane_pair(P + 1);       // packed pairs of a local
  // warps per CTA (each 16 lane pairs, so 2 W parents and their children)
  // and CTAs per SM: as many warps as the registers of the order allow (80
  // a thread at order 4, 128 up to order 8, 168 up to 12, 255 above).  With
  // 8 warps a CTA of order 12 kept 0.59 of its issue slots busy.
  static constexpr int W = P <= 4 ? 8 : (P <= 8 ? 16 : (P <= 12 ? 12 : 8));
  static constexpr int PAR = 2 * W;                 // parents per CTA
  static constexpr int CTAS = P <= 4 ? 3 : 1;
  static constexpr bool TM = P >= 8;                // sums in tensor memory
  static constexpr int NCH = (2 * NP + 15) / 16;    // 16-column pieces of a warp's sums
  // segments of the 189 offsets: more of them spread a small pass over more
  // CTAs, each costs a large one a pass of its sums through the L2 (0.1 ms of
  // 11.3 at order 12, 0.15 ms of 27.3 at order 16, 4 M particles)
  static constexpr int SEGS = P <= 12 ? 16 : 8;
  static constexpr int COLS = 16 * NCH;             // columns of a warp in the workspace
  // columns of a CTA: W / 4 warps share each quarter of the rows
  static constexpr int TCOLS = NCH * 16 * (W / 4) <= 256 ? 256 : 512;
  static_assert(NCH * 16 * (W / 4) <= 512, "sums exceed the tensor memory");
};

template <int P>
constexpr size_t lanes_smem() {
  using D = LaneDims<P>;
  size_t off = (size_t)kLaneNst * D::STRIDE * sizeof(float);
  off += 2 * kLaneNst * sizeof(uint64_t) + D::W * sizeof(uint64_t);
  off += (size_t)D::W * 16 * D::NMP * sizeof(cplx<float>);
  off += (size_t)D::PAR * 216 * sizeof(int);
  off += 16 * sizeof(unsigned) + 192 * sizeof(unsigned) + 2 * 192 * sizeof(uint16_t);
  return off + 64;
}

__device__ __forceinline__ float sel4(const float4 &v, int k) {
  return k == 0 ? v.x : (k == 1 ? v.y : (k == 2 ? v.z : v.w));
}

// 16 columns of this warp's tensor-memory rows, read and written without
// waiting; the wait names the registers so no use moves ahead of it
__device__ __forceinline__ void tm_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tm_wait_ld(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ void tm_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// constants of the scaled frame: 1 / A(l, m) by coefficient and the packed
// pairs (H(k), H(k))
constexpr double lane_sqrt(double v) {
  double x = v > 1. ? v : 1.;
  for (int i = 0; i < 200; ++i) {
    const double y = 0.5 * (x + v / x);
    if (y >= x) break;
    x = y;
  }
  return x;
}
template <int P>
struct LaneConst {
  float inva[(P + 1) * (P + 2) / 2];
  float h[2 * P];
  constexpr LaneConst() : inva(), h() {
    for (int l = 0; l <= P; ++l)
      for (int m = 0; m <= l; ++m) {
        double f = 1., q = 1.;
        for (int k = 2; k <= l - m; ++k) f *= k;
        for (int k = 2; k <= l + m; ++k) f *= k;
        for (int k = 0; k < l; ++k) q *= 4.;
        inva[l * (l + 1) / 2 + m] = (float)(lane_sqrt(f) / q);
      }
    double v = 1.;
    for (int k = 0; k < 2 * P; ++k) {
      if (k > 0) v *= k / 4.;
      h[k] = (float)v;
    }
  }
};

template <int P>
__device__ constexpr LaneConst<P> kLaneConst{};

struct LaneArgs {
  int nparents, nsplit;
  const int *parents, *child, *begin, *end, *col, *ncol, *ijk;
  const uint8_t *depth;
  const float *dirs;
  double scale_e;
  const cplx<float> *mult;
  cplx<float> *loc;
  float *part;      // sums [segment][group][warp][column / 4][lane][column % 4]; one CTA
                    // per group (nsplit = 1): the running sum in segment 0's place
  int *err;
  int polls;
};

// four sums of a lane to the workspace: stored, or added to what it holds
__device__ __forceinline__ void part_put(float4 *dst, bool add, float x, float y, float z,
                                         float w) {
  if (add)
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(x),
                 "f"(y), "f"(z), "f"(w)
                 : "memory");
  else
    *dst = make_float4(x, y, z, w);
}
// the reductions' sum: denormals are flushed
__device__ __forceinline__ float add_ftz(float a, float b) {
  float r;
  asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int P>
__device__ __forceinline__ void m2l_lanes_body(const LaneArgs &a) {
  using D = LaneDims<P>;
  constexpr int NM = D::NM, NL = D::NL, NMP = D::NMP, STRIDE = D::STRIDE, NP = D::NP;
  constexpr int W = D::W, PAR = D::PAR, NCH = D::NCH;
  constexpr bool TM = D::TM;
  const LaneConst<P> &K = kLaneConst<P>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // shared layout: ring tables | full[NST] | empty[NST] | per-warp source
  // barriers | staged multipoles [warp][pair][NMP] | PAR 6x6x6 source grids |
  // offset mask | cells of the offsets | active offsets | offset codes
  size_t off = 0;
  float *tab = reinterpret_cast<float *>(smem_raw);
  off += (size_t)kLaneNst * STRIDE * sizeof(float);
  uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw + off);
  uint64_t *empty = full + kLaneNst;
  uint64_t *sbar = empty + kLaneNst;    // per warp: its staged sources have landed
  off += 2 * kLaneNst * sizeof(uint64_t) + W * sizeof(uint64_t);
  off = (off + 15) & ~(size_t)15;
  cplx<float> *stg = reinterpret_cast<cplx<float> *>(smem_raw + off);
  off += (size_t)W * 16 * NMP * sizeof(cplx<float>);
  int *grid = reinterpret_cast<int *>(smem_raw + off);
  off += (size_t)PAR * 216 * sizeof(int);
  unsigned *mask = reinterpret_cast<unsigned *>(smem_raw + off);
  off += 16 * sizeof(unsigned);
  unsigned *dcell = reinterpret_cast<unsigned *>(smem_raw + off);   // 189 of them
  off += 192 * sizeof(unsigned);
  uint16_t *active = reinterpret_cast<uint16_t *>(smem_raw + off);
  off += 192 * sizeof(uint16_t);
  uint16_t *dcode = reinterpret_cast<uint16_t *>(smem_raw + off);   // 189 of them
  __shared__ uint32_t s_tmem;

  for (int i = threadIdx.x; i < PAR * 216; i += blockDim.x) grid[i] = -1;
  if (threadIdx.x < 16) mask[threadIdx.x] = 0u;
  // child 0's offsets (dx, dy, dz) in [-3,2]^3 minus [-1,1]^3, dz slowest:
  // index = L - (near cells below L), L = (dx+3) + 6 (dy+3) + 36 (dz+3); table
  // code (dx+3) + 7 (dy+3) + 49 (dz+3); grid cell parts dx+3, 6 (dy+3),
  // 36 (dz+3) in bytes
  for (int L = threadIdx.x; L < 216; L += blockDim.x) {
    const int a0 = L % 6, b0 = (L / 6) % 6, c0 = L / 36;
    auto in = [](int v) { return v >= 2 && v <= 4; };
    auto below = [](int v) { return v < 2 ? 0 : (v > 4 ? 3 : v - 2); };
    if (in(a0) && in(b0) && in(c0)) continue;
    const int nb = 9 * below(c0) + (in(c0) ? 3 * below(b0) + (in(b0) ? below(a0) : 0) : 0);
    const int di = L - nb;
    dcode[di] = (uint16_t)(a0 + 7 * b0 + 49 * c0);
    dcell[di] = (unsigned)(a0 | (6 * b0) << 8 | (36 * c0) << 16);
  }
  if (threadIdx.x == 0) {
    for (int b = 0; b < kLaneNst; ++b) {
      mbar_init(&full[b], 1);
      mbar_init(&empty[b], W);
    }
    for (int k = 0; k < W; ++k) mbar_init(&sbar[k], 1);
    fence_mbar_init();
  }
  if (TM && w == 0) tmem_alloc(&s_tmem, D::TCOLS);
  if (TM) tc_fence_before();
  __syncthreads();
  if (TM) tc_fence_after();
  const uint32_t tm =
      TM ? s_tmem + ((uint32_t)((w & 3) * 32) << 16) + (uint32_t)((w >> 2) * NCH * 16)
         : 0u;
  if (TM) {
    uint32_t zero[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) zero[i] = 0u;
    for (int c = 0; c < NCH; ++c) tm_st16(tm + 16 * c, zero);
    tm_wait_st();
  }
  // the parents of this CTA: their colleagues' children fill the grids (a
  // warp takes two parents, so their chains of loads run side by side)
  for (int g = w; g < PAR; g += W) {
    const int pidx = blockIdx.x * PAR + g;
    if (pidx >= a.nparents) break;
    const int Pn = a.parents[pidx];
    const int pi = a.ijk[3 * Pn], pj = a.ijk[3 * Pn + 1], pk = a.ijk[3 * Pn + 2];
    const int nc = a.ncol[Pn];
    for (int e = lane; e < nc * 8; e += 32) {
      const int q = a.col[27 * Pn + e / 8];
      const int qc = a.child[q];
      if (qc < 0) continue;
      const int o = e & 7;
      const int s = qc + o;
      if (a.end[s] == a.begin[s]) continue;
      const int gx = 2 * (a.ijk[3 * q] - pi + 1) + (o & 1);
      const int gy = 2 * (a.ijk[3 * q + 1] - pj + 1) + ((o >> 1) & 1);
      const int gz = 2 * (a.ijk[3 * q + 2] - pk + 1) + ((o >> 2) & 1);
      grid[g * 216 + gx + 6 * (gy + 6 * gz)] = s;
    }
  }
  __syncthreads();
  // lane pair 16 w + i / 2 of the CTA takes child cw of parent gp, child by
  // child; h = 0 real part, 1 imaginary part
  const int pi_ = lane >> 1, h = lane & 1;
  const int cw = (16 * w + pi_) / PAR, gp = (16 * w + pi_) % PAR;
  int tgt = -1;
  {
    const int pidx = blockIdx.x * PAR + gp;
    if (pidx < a.nparents) {
      const int t = a.child[a.parents[pidx]] + cw;
      if (a.end[t] > a.begin[t]) tgt = t;
    }
  }
  // child cw = (bx, by, bz) at cell (2+bx, 2+by, 2+bz) of the grid; its
  // offset for child 0's offset d is sigma_cw d, so its source is at cell
  // 2 - dx = 5 - (dx+3) along an axis it does not flip, 3 + dx along one it
  // does
  const int bx = cw & 1, by = (cw >> 1) & 1, bz = (cw >> 2) & 1;
  const int *my_grid = grid + gp * 216 + (bx ? 0 : 5) + (by ? 0 : 30) + (bz ? 0 : 180);
  auto source_of = [&](int di) -> int {
    if (tgt < 0) return -1;
    const unsigned c = dcell[di];
    const int cx = c & 255u, cy = (c >> 8) & 255u, cz = c >> 16;
    return my_grid[(bx ? cx : -cx) + (by ? cy : -cy) + (bz ? cz : -cz)];
  };
  for (int di = 0; di < 189; ++di) {
    const unsigned any = __ballot_sync(kFull, source_of(di) >= 0);
    if (lane == 0 && any) atomicOr(&mask[di >> 5], 1u << (di & 31));
  }
  __syncthreads();
  for (int di = threadIdx.x; di < 189; di += blockDim.x) {
    const unsigned m = mask[di >> 5];
    if ((m >> (di & 31)) & 1u) {
      int pos = __popc(m & ((1u << (di & 31)) - 1u));
      for (int k = 0; k < (di >> 5); ++k) pos += __popc(mask[k]);
      active[pos] = (uint16_t)di;
    }
  }
  __syncthreads();
  // this CTA's segments of the offset list; offset di belongs to segment
  // di D::SEGS / 189
  const int seg0 = D::SEGS * (int)blockIdx.y / a.nsplit;
  const int seg1 = D::SEGS * ((int)blockIdx.y + 1) / a.nsplit;
  auto active_below = [&](int seg) -> int {
    const int d = (189 * seg + D::SEGS - 1) / D::SEGS;   // offsets below it
    int n = 0;
    for (int k = 0; k < 6; ++k) {
      const int left = d - 32 * k;
      if (left > 0) n += __popc(mask[k] & (left >= 32 ? kFull : (1u << left) - 1u));
    }
    return n;
  };
  const int a0 = active_below(seg0);
  const int nact = active_below(seg1) - a0;
  active += a0;

  // the ring: thread 0 fills the first slots; afterwards warp 0 refills
  // slot b with offset it + NST once all warps have released it (no
  // separate producer warp, so two warps share each scheduler's registers)
  constexpr uint32_t kTabBytes = STRIDE * (uint32_t)sizeof(float);
  static_assert(kTabBytes % 16 == 0, "bulk copies of whole 16-byte rows");
  auto issue = [&](int i) {
    const int b = i % kLaneNst;
    mbar_expect_tx(&full[b], kTabBytes);
    bulk_g2s(tab + (size_t)b * STRIDE, a.dirs + (size_t)dcode[active[i]] * STRIDE, kTabBytes,
             &full[b]);
  };
  int issued = 0;   // table copies issued (thread 0)
  if (threadIdx.x == 0)
    for (; issued < kLaneNst && issued < nact; ++issued) issue(issued);

  cplx<float> *my_stg = stg + (size_t)(w * 16 + pi_) * NMP;
  uint64_t racc[TM ? 1 : NP];   // the sums over the offsets, packed pairs
#pragma unroll
  for (int c = 0; c < (TM ? 1 : NP); ++c) racc[c] = 0ull;
  int next_i = 0, next_s = -1;
  auto find_next = [&](int from) {
    for (next_i = from; next_i < nact; ++next_i) {
      next_s = source_of(active[next_i]);
      if (__any_sync(kFull, next_s >= 0)) break;
    }
  };
  // one bulk copy per source (issued by the pair's first lane) completing
  // on the warp's barrier; pairs without a source zero their slot.  At odd
  // NM the rows of odd nodes start 8 bytes into a 16-byte unit: the copy
  // begins there and the pair reads from the second coefficient
  constexpr uint32_t kSrcBytes = D::NMC * (uint32_t)sizeof(cplx<float>);
  static_assert(kSrcBytes % 16 == 0, "bulk copies of whole 16-byte rows");
  bool pending = false;
  uint32_t sph = 0;
  int shift = 0;
  auto prefetch = [&]() {
    if (next_i >= nact) return;
    const unsigned cp = __ballot_sync(kFull, h == 0 && next_s >= 0);
    if (lane == 0) mbar_expect_tx(&sbar[w], (uint32_t)__popc(cp) * kSrcBytes);
    __syncwarp();
    if (D::ODD) shift = next_s >= 0 ? next_s & 1 : 0;
    if (next_s >= 0) {
      if (h == 0) bulk_g2s(my_stg, a.mult + (size_t)next_s * NM - shift, kSrcBytes, &sbar[w]);
    } else {
      for (int c = h; c < D::NMC; c += 2) my_stg[c] = cmake<float>(0.f, 0.f);
    }
    pending = true;
  };
  find_next(0);
  prefetch();

  // the segments' sums: stored (split pass) or added to the running sum
  const bool whole = a.nsplit == 1;
  const size_t seg_step = (size_t)gridDim.x * W * D::COLS * 8;
  float4 *my_part = reinterpret_cast<float4 *>(a.part) +
                    ((size_t)blockIdx.x * W + w) * D::COLS * 8 + lane;
  bool started = false;    // the running sum holds a segment
  int it = 0;
  bool stop = false;
  for (int seg = seg0; seg < seg1 && !stop; ++seg) {
  bool any_src = false;    // this warp met a source in the segment
  for (; it < nact && active[it] * D::SEGS / 189 == seg; ++it) {
    const int b = it % kLaneNst;
    const bool ok =
        __all_sync(kFull, mbar_wait_or_flag(&full[b], (it / kLaneNst) & 1, a.err, a.polls));
    if (!ok) {
      if (lane == 0) atomicOr(a.err, kErrTimeout);
      stop = true;
      break;
    }
    if (it == next_i) {
      const float *tb = tab + (size_t)b * STRIDE;
      if (!__all_sync(kFull, mbar_wait(&sbar[w], sph))) {
        if (lane == 0) atomicOr(a.err, kErrTimeout);
        stop = true;
        break;
      }
      any_src = true;
      sph ^= 1u;
      pending = false;
      __syncwarp();
      // mirror S, z-phase and rotation to the z axis (degrees < p): this
      // lane's part of the phased mirrored source (l, m), in the scaled
      // frame, is sn (x.re pa[m] + x.im pb[m]) / A(l, m), sn = -1 for odd l
      // under a z flip
      float y[NM];
      {
        float pa[P], pb[P];
        {
          const float4 *PA = reinterpret_cast<const float4 *>(tb + (h ? m2l_hk_cp(P) : 0));
          const float4 *PB = reinterpret_cast<const float4 *>(tb + (h ? 0 : m2l_hk_cp(P)));
          const float g = (bx ^ bz) ? -1.f : 1.f;                 // (-1)^m of x and z flips
          const float c0 = ((bx ^ by) != h) ? 1.f : -1.f;          // conjugation
          float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), qb = qa;
#pragma unroll
          for (int m = 0; m < P; ++m) {
            if ((m & 3) == 0) {
              qa = PA[m >> 2];
              qb = PB[m >> 2];
            }
            pa[m] = (m & 1) ? g * sel4(qa, m & 3) : sel4(qa, m & 3);
            pb[m] = ((m & 1) ? g * c0 : c0) * sel4(qb, m & 3);
          }
        }
        const float4 *X4 = reinterpret_cast<const float4 *>(my_stg);
        const float2 *X2 = reinterpret_cast<const float2 *>(my_stg) + (D::ODD ? shift : 0);
        const float4 *F4 = reinterpret_cast<const float4 *>(tb + m2l_hk_f(P)) + h;
        const float f0 = h ? 0.f : 2.f;
        const float sn = bz ? -1.f : 1.f;
        float4 xq = make_float4(0.f, 0.f, 0.f, 0.f), fq = xq;
#pragma unroll
        for (int l = 0; l < P; ++l) {
          float xp[P], yl[P];
#pragma unroll
          for (int m = 0; m <= l; ++m) {
            const int c = l * (l + 1) / 2 + m;
            float xr, xi;
            if (D::ODD) {
              const float2 v = X2[c];
              xr = v.x;
              xi = v.y;
            } else {
              if ((c & 1) == 0) xq = X4[c >> 1];
              xr = (c & 1) ? xq.z : xq.x;
              xi = (c & 1) ? xq.w : xq.y;
            }
            float v = fmaf(xr, pa[m], xi * pb[m]) * K.inva[c];
            if (l & 1) v *= sn;
            xp[m] = v;
            yl[m] = 0.f;
          }
          // lower triangle (m <= m') direct, upper triangle by symmetry; the
          // first row's upper part is summed apart (its factor is f0)
          float y0 = 0.f;
#pragma unroll
          for (int mp = 0; mp <= l; ++mp)
#pragma unroll
            for (int m = 0; m <= mp; ++m) {
              const int t = m2l_lane_tet(l) + mp * (mp + 1) / 2 + m;
              if ((t & 3) == 0) fq = F4[2 * (t >> 2)];
              const float v = sel4(fq, t & 3);
              yl[mp] = fmaf(v, xp[m], yl[mp]);
              if (m < mp) {
                const float xs = ((m + mp) & 1) ? -xp[mp] : xp[mp];
                if (m == 0) y0 = fmaf(v, xs, y0);
                else yl[m] = fmaf(v, xs, yl[m]);
              }
            }
          yl[0] = fmaf(f0, y0, yl[0]);
#pragma unroll
          for (int m = 0; m <= l; ++m) y[l * (l + 1) / 2 + m] = yl[m];
        }
      }
      find_next(it + 1);
      __syncwarp();           // both lanes of every pair are done with the staged source
      prefetch();
      // translation along z in the scaled frame: z(j, m) = sum_n H(j + n)
      // y(n, m), the orders m, m + 1 in packed pairs
      float z[NL];
      static_for<P / 2>([&](auto mc) {
        constexpr int m = 2 * decltype(mc)::value;
        uint64_t y2[P - m], z2[P - m + 1];
#pragma unroll
        for (int n = m; n < P; ++n)
          y2[n - m] =
              pack2(y[n * (n + 1) / 2 + m], n > m ? y[n * (n + 1) / 2 + m + (n > m)] : 0.f);
#pragma unroll
        for (int n = m; n < P; ++n)
#pragma unroll
          for (int j = m; j <= P; ++j) {
            const uint64_t hk = pack2(K.h[j + n], K.h[j + n]);
            z2[j - m] = n == m ? mul2(hk, y2[0]) : fma2(hk, y2[n - m], z2[j - m]);
          }
#pragma unroll
        for (int j = m; j <= P; ++j) {
          float lo, hi;
          unpack2(z2[j - m], lo, hi);
          z[j * (j + 1) / 2 + m] = lo;
          if (j > m) z[j * (j + 1) / 2 + m + (j > m)] = hi;
        }
      });
      z[NL - 1] = 0.f;   // no source term has order p
      // rotation back (degrees <= p), conjugate z-phase and sum: real part
      // += a cos + b sin, imaginary part += a cos - b sin, with a this
      // lane's part and b the partner's
      {
        const float4 *B4 = reinterpret_cast<const float4 *>(tb + m2l_hk_b(P)) + h;
        const float f0 = h ? 0.f : 2.f;
        const uint64_t *C2 = reinterpret_cast<const uint64_t *>(tb);
        const uint64_t *S2 = reinterpret_cast<const uint64_t *>(tb + m2l_hk_cp(P));
        const uint64_t hs = h ? pack2(-1.f, -1.f) : pack2(1.f, 1.f);
        float4 bq = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int l = 0; l <= P; ++l) {
          float zi[P + 1], ol[P + 1];
#pragma unroll
          for (int m = 0; m <= l; ++m) {
            zi[m] = z[l * (l + 1) / 2 + m];
            ol[m] = 0.f;
          }
          float o0 = 0.f;
#pragma unroll
          for (int mp = 0; mp <= l; ++mp)
#pragma unroll
            for (int m = 0; m <= mp; ++m) {
              const int t = m2l_lane_tet(l) + mp * (mp + 1) / 2 + m;
              if ((t & 3) == 0) bq = B4[2 * (t >> 2)];
              const float v = sel4(bq, t & 3);
              ol[mp] = fmaf(v, zi[m], ol[mp]);
              if (m < mp) {
                if (m == 0) o0 = fmaf(v, zi[mp], o0);
                else ol[m] = fmaf(v, zi[mp], ol[m]);
              }
            }
          ol[0] = fmaf(f0, o0, ol[0]);
#pragma unroll
          for (int m = 0; m <= l; ++m) z[l * (l + 1) / 2 + m] = ol[m];
        }
        uint64_t cph[P / 2 + 1], sphs[P / 2 + 1];
#pragma unroll
        for (int k = 0; k <= P / 2; ++k) {
          cph[k] = C2[k];
          sphs[k] = mul2(hs, S2[k]);
        }
        uint32_t r[2][16];
        if (TM) {
          tm_wait_st();        // the last offset's sums have been written
          tm_ld16(tm, r[0]);
        }
#pragma unroll
        for (int l = 0; l <= P; ++l)
#pragma unroll
          for (int k = 0; k <= l / 2; ++k) {
            const int q = lane_pair(l) + k, c = l * (l + 1) / 2 + 2 * k;
            const float a0_ = z[c], a1_ = 2 * k + 1 <= l ? z[c + (2 * k + 1 <= l)] : 0.f;
            const float b0_ = __shfl_xor_sync(kFull, a0_, 1);
            const float b1_ = 2 * k + 1 <= l ? __shfl_xor_sync(kFull, a1_, 1) : 0.f;
            const uint64_t av = pack2(a0_, a1_), bv = pack2(b0_, b1_);
            if (TM) {
              const int ch = q >> 3, e = 2 * (q & 7);
              uint32_t (&rc)[16] = r[ch & 1];
              if ((q & 7) == 0) {
                tm_wait_ld(rc);
                if (ch + 1 < NCH) tm_ld16(tm + 16 * (ch + 1), r[(ch + 1) & 1]);
              }
              float lo, hi;
              const uint64_t sum = fma2(
                  bv, sphs[k],
                  fma2(av, cph[k], pack2(__uint_as_float(rc[e]), __uint_as_float(rc[e + 1]))));
              unpack2(sum, lo, hi);
              rc[e] = __float_as_uint(lo);
              rc[e + 1] = __float_as_uint(hi);
              if ((q & 7) == 7 || q == NP - 1) tm_st16(tm + 16 * ch, rc);
            } else {
              racc[TM ? 0 : q] = fma2(bv, sphs[k], fma2(av, cph[k], racc[TM ? 0 : q]));
            }
          }
      }
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(&empty[b]);
      if (w == 0 && it + kLaneNst < nact) {
        if (!mbar_wait_or_flag(&empty[b], (it / kLaneNst) & 1, a.err)) {
          atomicOr(a.err, kErrTimeout);
        } else {
          issue(it + kLaneNst);
          ++issued;
        }
      }
    }
    __syncwarp();
  }
  // the segment's sum to the workspace, four columns at a time, and back to
  // zero; added with reductions, which the L2 carries out while the next
  // segment runs (loading, adding and storing the running sum here took 15 %
  // longer at order 16)
  if (stop || (whole && !any_src)) continue;
  float4 *dst = whole ? my_part : my_part + seg * seg_step;
  const bool add = whole && started;
  started = true;
  if constexpr (TM) {
    uint32_t zero[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) zero[i] = 0u;
    tm_wait_st();
#pragma unroll 1
    for (int ch = 0; ch < NCH; ++ch) {
      uint32_t r[16];
      tm_ld16(tm + 16 * ch, r);
      tm_wait_ld(r);
      tm_st16(tm + 16 * ch, zero);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        part_put(dst + 32 * (4 * ch + i), add, __uint_as_float(r[4 * i]),
                 __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                 __uint_as_float(r[4 * i + 3]));
    }
  } else {
#pragma unroll
    for (int q = 0; q < NP; q += 2) {
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      unpack2(racc[q], v[0], v[1]);
      racc[q] = 0ull;
      if (q + 1 < NP) {
        unpack2(racc[q + 1 < NP ? q + 1 : 0], v[2], v[3]);
        racc[q + 1 < NP ? q + 1 : 0] = 0ull;
      }
      part_put(dst + 16 * q, add, v[0], v[1], v[2], v[3]);
    }
  }
  }
  // copies still in flight after an early exit land before the CTA leaves
  if (pending) mbar_wait(&sbar[w], sph);
  if (threadIdx.x == 0)
    for (int i = it; i < issued; ++i) mbar_wait(&full[i % kLaneNst], (i / kLaneNst) & 1);
  __syncwarp();
  // back from the mirror frame and the scaled frame into the target's local
  if (whole && started && tgt >= 0) {
    const float ih = (float)((double)(1ull << a.depth[tgt]) / a.scale_e);   // 2^depth / scale
    float *lo = reinterpret_cast<float *>(a.loc) + (size_t)tgt * NL * 2 + h;
    int c = 0;
    for (int l = 0; l <= P; ++l)
#pragma unroll 4
      for (int m = 0; m <= l; ++m, ++c) {
        const bool neg = ((bz & (l + m)) ^ (bx & m) ^ (h & (bx ^ by))) & 1;
        const int col = lane_col(l, m);
        const float v = __ldcg(reinterpret_cast<const float *>(my_part + 32 * (col >> 2)) +
                               (col & 3));
        lo[2 * c] = v * K.inva[c] * (neg ? -ih : ih);
      }
  }
  if (TM) tm_wait_st();
  if (TM) {
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (w == 0) tmem_dealloc(s_tmem, D::TCOLS);
  }
}

// the kernel at the orders of the benchmark, and at the other even orders
template <int P>
__global__ void __launch_bounds__(32 * LaneDims<P>::W, LaneDims<P>::CTAS) k_m2l_lanes(LaneArgs a) {
  m2l_lanes_body<P>(a);
}
template <int P>
__global__ void __launch_bounds__(32 * LaneDims<P>::W, LaneDims<P>::CTAS)
    k_m2l_sibling_lanes(LaneArgs a) {
  m2l_lanes_body<P>(a);
}

// the segments of a split pass added in order: block (group, warp), one
// thread per lane and every eighth coefficient
template <int P>
__global__ void __launch_bounds__(256) k_m2l_lanes_sum(LaneArgs a) {
  constexpr int NL = LaneDims<P>::NL;
  constexpr int W = LaneDims<P>::W, PAR = LaneDims<P>::PAR;
  const int lane = threadIdx.x & 31, w = blockIdx.y, h = lane & 1;
  const int cw = (16 * w + (lane >> 1)) / PAR, gp = (16 * w + (lane >> 1)) % PAR;
  const int pidx = blockIdx.x * PAR + gp;
  if (pidx >= a.nparents) return;
  const int t = a.child[a.parents[pidx]] + cw;
  if (a.end[t] <= a.begin[t]) return;
  const int bx = cw & 1, by = (cw >> 1) & 1, bz = (cw >> 2) & 1;
  const float ih = (float)((double)(1ull << a.depth[t]) / a.scale_e);
  constexpr int COLS = LaneDims<P>::COLS;
  const size_t step = (size_t)gridDim.x * W * COLS * 32;
  for (int c = threadIdx.x >> 5; c < NL; c += 8) {
    int l = 0;
    while ((l + 1) * (l + 2) / 2 <= c) ++l;
    const int m = c - l * (l + 1) / 2;
    const int col = lane_col(l, m);
    const float *p = a.part + ((size_t)blockIdx.x * W + w) * COLS * 32 +
                     (32 * (col >> 2) + lane) * 4 + (col & 3);
    float v = p[0];
#pragma unroll
    for (int k = 1; k < LaneDims<P>::SEGS; ++k) v = add_ftz(v, p[k * step]);
    const bool neg = ((bz & (l + m)) ^ (bx & m) ^ (h & (bx ^ by))) & 1;
    reinterpret_cast<float *>(a.loc)[((size_t)t * NL + c) * 2 + h] =
        v * kLaneConst<P>.inva[c] * (neg ? -ih : ih);
  }
}

// CTAs that share a group's segments: the least number of waves of CTAs
// times the work of each (1 / K of the segments and the set-up, about 1/40 of
// a whole list); none where the workspace of all segments would be large
inline int lane_split(int groups, int resident, int segs) {
  int best = 1;
  double cost = 1e30;
  for (int k = 1; k <= (groups <= 2 * resident ? segs : 1); k *= 2) {
    const double c = (double)(((int64_t)groups * k + resident - 1) / resident) * (1. / k + 0.025);
    if (c < 0.97 * cost) {
      cost = c;
      best = k;
    }
  }
  return best;
}

template <int P>
bool launch_p(AranGpuSolver3d *s, OpTables<float> &tb, const int *parents, int count,
              const cplx<float> *mult, cplx<float> *loc, cudaStream_t st) {
  using D = LaneDims<P>;
  DevTree &t = s->tree;
  const size_t sm = lanes_smem<P>();
  int dev_smem = 0, nsm = 0;
  ACHECK(cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device));
  ACHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, s->device));
  if ((int)sm > dev_smem) return false;
  void (*kern)(LaneArgs);
  if constexpr (m2l_lane_order(P)) kern = k_m2l_lanes<P>;
  else kern = k_m2l_sibling_lanes<P>;
  smem_opt_in(kern, sm);
  LaneArgs a;
  a.nparents = count;
  a.parents = parents;
  a.child = t.child.ptr;
  a.begin = t.begin.ptr;
  a.end = t.end.ptr;
  a.col = t.col.ptr;
  a.ncol = t.ncol.ptr;
  a.ijk = t.ijk.ptr;
  a.depth = t.depth.ptr;
  a.dirs = tb.dir_lanes.ptr;
  a.scale_e = s->scale_e;
  a.mult = mult;
  a.loc = loc;
  a.err = s->err_dev.ptr;
  a.polls = consumer_wait_polls();
  const int groups = ceil_div(count, D::PAR);
  a.nsplit = lane_split(groups, nsm * D::CTAS, D::SEGS);
  s->m2l_part.reserve((size_t)(a.nsplit > 1 ? D::SEGS : 1) * groups * D::W * D::COLS * 32);
  a.part = s->m2l_part.ptr;
  kern<<<dim3(groups, a.nsplit), 32 * D::W, sm, st>>>(a);
  ACHECK(cudaGetLastError());
  s->launches++;
  if (a.nsplit > 1) {
    k_m2l_lanes_sum<P><<<dim3(groups, D::W), 256, 0, st>>>(a);
    ACHECK(cudaGetLastError());
    s->launches++;
  }
  return true;
}

}  // namespace

}  // namespace aran
