// p2p.cu -- the near field (P2P) on the device.
//
// LibAran calls the user p2p callback for every pair of points of every near
// leaf pair (near_func, aran/aransolver3d.c:254-324) with the Newton kernels
// of tests/newtonpot3.c:61-78 (potential) and tests/newtonfield3.c:91-119
// (field, |r| > 1e-5 guard).  Here every target particle sums its near
// sources directly (both sides of a pair are evaluated by their own targets
// instead of the symmetric update).
//
// Work decomposition: a block per target leaf (k_p2p_tile in mixed precision,
// k_p2p64 in FP64), several for a leaf above the capacity.  Near ranges of more than
// kBigRange points (a coarse leaf next to a deep subtree, common in clustered
// sets) are cut into leaf-aligned chunks processed by extra blocks that accumulate
// atomically.
//
// Mixed precision: a source's offset from the target leaf's centre comes from
// FP32 hi + lo positions in the box, short runs of FP32 terms go into Kahan sums
// and those into the FP64 accumulators, and pairs closer than 1/8 of the target
// leaf size (where FP32 cancellation would show) are made from the FP64
// positions.
#include <cub/cub.cuh>

#include <algorithm>

#include "internal.cuh"
#include "f32x2.cuh"

namespace aran {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// 1/sqrt(x) on the MUFU unit with denormals flushed: without the flush the
// FP32 rsqrt carries a denormal rescaling path; the near-field distances
// here are at least 1e-10 squared box units, far from denormal
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__global__ void k_leaf_info(int nleaves, const int *__restrict__ leaf_node,
                            const int *__restrict__ begin, const int *__restrict__ end,
                            const uint8_t *__restrict__ depth, const double *__restrict__ center,
                            const int *__restrict__ sys, const double *__restrict__ sys_box,
                            double ex, double ey, double ez, int2 *__restrict__ be,
                            float4 *__restrict__ chi, float4 *__restrict__ clo) {
  int L = blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= nleaves) return;
  int node = leaf_node[L];
  be[L] = make_int2(begin[node], end[node]);
  const double *b = sys_box + 9 * sys[node];   // from the box's corner, as the positions
  double cx = center[3 * node] - b[0], cy = center[3 * node + 1] - b[1],
         cz = center[3 * node + 2] - b[2];
  float hx = (float)cx, hy = (float)cy, hz = (float)cz;
  double h = fmin(ex, fmin(ey, ez)) / ldexp(1.0, depth[node]);
  float thr = (float)(h * 0.125);
  chi[L] = make_float4(hx, hy, hz, thr * thr);
  clo[L] = make_float4((float)(cx - (double)hx), (float)(cy - (double)hy), (float)(cz - (double)hz), 0.f);
}

__device__ __forceinline__ int rng_count(const int2 *be, int la, int lb) {
  return be[lb - 1].y - be[la].x;
}

// heavy ranges -> leaf-aligned chunks of about kBigRange points: one block
// per heavy range (listed by k_near with the offset of its first chunk), one
// thread per chunk, whose ends are the first leaves whose points start at or
// beyond p0 + i kBigRange (binary searches, independent per chunk)
__global__ void k_big_items(const int *__restrict__ heavy, int nleaves,
                            const int *__restrict__ near_off, const int *__restrict__ near_rng,
                            const int2 *__restrict__ be, int4 *__restrict__ items) {
  const int r = heavy[2 * blockIdx.x], coff = heavy[2 * blockIdx.x + 1];
  const int la = near_rng[2 * r], lb = near_rng[2 * r + 1];
  const int c = rng_count(be, la, lb);
  const int nch = (c + kBigRange - 1) / kBigRange;
  int lo = 0, hi = nleaves;                   // target leaf: last L with near_off[L] <= r
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (near_off[mid] <= r) lo = mid; else hi = mid;
  }
  const int L = lo;
  const int p0 = be[la].x;
  auto boundary = [&](int i) -> int {          // first leaf of chunk i
    if (i <= 0) return la;
    if (i >= nch) return lb;
    int l2 = la, h2 = lb;
    const int target = p0 + i * kBigRange;
    while (l2 < h2) {
      const int mid = (l2 + h2) >> 1;
      if (be[mid].x < target) l2 = mid + 1; else h2 = mid;
    }
    return l2;
  };
  for (int i = threadIdx.x; i < nch; i += blockDim.x)
    items[coff + i] = make_int4(L, boundary(i), boundary(i + 1), 0);
}

// 1/sqrt(x) in FP64 from the hardware approximation's upper word y0 (20
// significant bits, so y0^2 is exact) by one third-order Householder step,
// y0 + y0 e (1/2 + 3/8 e) with e = 1 - x y0^2 rounded once: five FP64
// operations, within an ulp of the correctly rounded value.  Outside the
// normal range's middle the library function takes over.
__device__ __forceinline__ double rsqrt_h3(double x) {
  double a;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(a) : "d"(x));
  const double y0 = __hiloint2double(__double2hiint(a), 0);
  const double e = fma(-x, y0 * y0, 1.0);
  return fma(y0, e * fma(e, 0.375, 0.5), y0);
}

// FP64 near field, a block of 128 threads per target leaf (BIG: per chunk of
// a heavy range).  The FP64 pipe takes half a lane per cycle and scheduler,
// so its instructions times idle lanes are the whole cost and index
// arithmetic is free: a leaf of n targets gets floor(128 / n) threads per
// target, which stride over the concatenation of the leaf's near ranges (the
// sorted particles of a range lie side by side), so all lanes but a few are
// busy to the last source; the field takes 18 FP64 operations a pair.
// Measured on GB300, 200k Plummer particles (leaf 64, 5.9e8 directed pairs):
// 16.3 ms and 8.0 ms for the chunks, the FP64 pipe active 88 % of the SMs'
// active cycles; the whole FP64 solve of order 12 went from 69.5 to 54.8 ms
// against 16, 8, 4, .. threads per target by powers of two (56 % of the
// lanes at 18 points a leaf) and the library's reciprocal square root.
template <bool FIELD, bool BIG>
__global__ void __launch_bounds__(128, 8) k_p2p64(
    const int4 *__restrict__ items, const int *__restrict__ near_off,
    const int *__restrict__ near_rng, const int2 *__restrict__ be,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, double *__restrict__ acc_pot, double *__restrict__ acc_fld) {
  constexpr int NV = FIELD ? 4 : 1;
  __shared__ double red[NV][128];
  int L = blockIdx.x, ia = 0, ib = 0;
  if (BIG) {
    const int4 it = items[blockIdx.x];
    L = it.x;
    ia = it.y;
    ib = it.z;
  }
  const int2 tbe = be[L];
  const int nt = tbe.y - tbe.x;
  const int r0 = BIG ? 0 : near_off[L], r1 = BIG ? 1 : near_off[L + 1];
  const long long guard = __double_as_longlong(FIELD ? 1e-10 : 0.);
  for (int tb = blockIdx.y * 128; tb < nt; tb += 128 * gridDim.y) {
    const int rem = min(nt - tb, 128);
    const int s = 128 / rem;                  // threads per target
    const int ti = threadIdx.x / s, sub = threadIdx.x - ti * s;
    const bool active = ti < rem;
    const int t = tbe.x + tb + (active ? ti : 0);
    double v[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) v[c] = 0.;
    if (active) {
      const double tx = sx[t], ty = sy[t], tz = sz[t];
      // source j of the concatenated ranges; je the end of its range
      int rr = r0 - 1, je = 0, j = sub;
      auto advance = [&]() -> bool {   // j counts past je: into the next ranges
        while (j >= je) {
          if (++rr >= r1) return false;
          int la, lb;
          if (BIG) {
            la = ia;
            lb = ib;
          } else {
            la = near_rng[2 * rr];
            lb = near_rng[2 * rr + 1];
          }
          if (lb <= la) continue;
          const int b0 = be[la].x, e0 = be[lb - 1].y;
          if (!BIG && e0 - b0 > kBigRange) continue;   // chunked by the BIG pass
          j += b0 - je;
          je = e0;
        }
        return true;
      };
      while (advance()) {
        const double dx = tx - sx[j], dy = ty - sy[j], dz = tz - sz[j];
        const double r2 = dx * dx + dy * dy + dz * dz;
        // the point itself and coincident points: r2 == 0, skipped (r2 >= 0:
        // its bits order like its value)
        const long long bits = __double_as_longlong(r2);
        if (bits > guard) {
          const unsigned ex = (unsigned)(bits >> 52);
          double inv = rsqrt_h3(r2);
          if (ex - 23u > 2000u) inv = rsqrt(r2);
          const double qi = sq[j] * inv;
          v[0] += qi;
          if (FIELD) {
            const double q3 = qi * (inv * inv);
            v[NV > 1 ? 1 : 0] -= q3 * dx;
            v[NV > 1 ? 2 : 0] -= q3 * dy;
            v[NV > 1 ? 3 : 0] -= q3 * dz;
          }
        }
        j += s;
      }
    }
    // the s sums of a target, halving
#pragma unroll
    for (int c = 0; c < NV; ++c) red[c][threadIdx.x] = v[c];
    __syncthreads();
    int o = 1;
    while (2 * o < s) o *= 2;
    for (; o > 0 && s > 1; o >>= 1) {
      if (active && sub < o && sub + o < s)
#pragma unroll
        for (int c = 0; c < NV; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + o];
      __syncthreads();
    }
    if (active && sub == 0) {
#pragma unroll
      for (int c = 0; c < NV; ++c) {
        double *dst = c == 0 ? &acc_pot[t] : &acc_fld[3 * (size_t)t + (c - 1)];
        if (BIG) atomicAdd(dst, red[c][threadIdx.x]);
        else *dst = red[c][threadIdx.x];
      }
    }
    __syncthreads();
  }
}

// Mixed near field, a block of T threads per target leaf.  The sources of a
// leaf are the concatenation of its near ranges (the sorted particles of a
// range lie side by side): the block stages up to 2 T of them at a time in
// shared memory, as offsets from the target leaf's centre made from FP32
// hi + lo positions, and the threads sum them two at a time in packed FP32
// pairs: a leaf of n targets gets floor(T / n) threads per target, so the
// lanes are busy whatever n is.  The pair loop has no branch: pairs closer
// than h/8 (and the point itself) are left out, and a thread whose part held
// one adds those pairs from the FP64 positions afterwards.  Up to 22 pairs are
// summed plainly, the runs in Kahan sums (one run a tile, 128 pairs, was 6 to 10 %
// faster on leaves of 40 points and more, with three times the rounding error
// of a warp per leaf's runs of up to 32 sources; shorter runs where leaves, and with
// them those runs, are short), and the parts of a target are added with
// compensation.  Rms error of one-sign potentials in one box of 8 leaves of 16, 60
// and 120 points: 1.9e-8, 2.1e-8, 1.6e-8; one run a tile 1.9e-8, 4.6e-8, 6.5e-8; a
// warp per leaf 2.0e-8, 2.7e-8, 2.0e-8.
// Ranges of more than kBigRange points are left to the chunked pass.
// Bound by issue and the FP32 pipes: 13 operations a pair with the field (3
// subtractions, 3 for r^2, 4 for q/r and q/r^3, 3 sums), 23 instructions for
// two pairs; about two thirds of the instructions are the pair loop's.
// Measured on GB300 against a warp per leaf with 1 to 32 lanes per target (in
// powers of two), sources staged leaf by leaf and pairs taken singly: 300k
// blobs (leaf 64) 0.48 ms, 1.08 before; 4M Plummer 3.7 ms, 5.2; 10k uniform
// (leaf 20, potential) 0.02 ms, 0.09.  With one run a tile T = 64, 96 and 256 took
// 0.68, 0.70 and 0.66 ms on the blobs where 128 took 0.61; tiles of twice and four
// times the sources changed nothing; 10 blocks an SM with 48 registers a thread beat
// 8, 6 and 12.
constexpr int kP2pRanges = 32;   // near ranges taken together

template <bool FIELD, bool BIG, int T>
__global__ void __launch_bounds__(T, 1280 / T) k_p2p_tile(
    const int4 *__restrict__ items, const int *__restrict__ near_off,
    const int *__restrict__ near_rng,
    const int2 *__restrict__ be, const float4 *__restrict__ chi, const float4 *__restrict__ clo,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const real4<float> *__restrict__ rel32, const float4 *__restrict__ phi,
    const float4 *__restrict__ plo, double *__restrict__ acc_pot, double *__restrict__ acc_fld) {
  constexpr int NV = FIELD ? 4 : 1;
  // pair p of the tile: (-x0, -x1, -y0, -y1) and (-z0, -z1, q0, q1)
  __shared__ ulonglong2 tA[T], tB[T];
  __shared__ int tj[2 * T];                       // their particles
  __shared__ int rs[kP2pRanges], rp[kP2pRanges];  // ranges: first particle, place
  __shared__ int s_tot;
  __shared__ float red[2 * NV][T];
  int L = blockIdx.x, ia = 0, ib = 0;
  if (BIG) {
    const int4 it = items[blockIdx.x];
    L = it.x;
    ia = it.y;
    ib = it.z;
  }
  const int2 tbe = be[L];
  const int nt = tbe.y - tbe.x;
  const float4 tch = chi[L], tcl = clo[L];
  const float thr2 = FIELD ? fmaxf(tch.w, 1e-10f) : tch.w;
  const int r0 = BIG ? 0 : near_off[L], r1 = BIG ? 1 : near_off[L + 1];
  for (int tb = blockIdx.y * T; tb < nt; tb += T * gridDim.y) {
    const int rem = min(nt - tb, T);
    const int S = T / rem;                        // threads per target
    const int run = T == 64 && rem <= 24 ? 8 : 22;   // pairs summed plainly
    // target by target within a part, so that a warp reads few pairs at a time
    const int sub = threadIdx.x / rem, ti = threadIdx.x - sub * rem;
    const bool active = sub < S;
    const int t = tbe.x + tb + ti;
    const real4<float> q0 = rel32[t];
    const uint64_t tx2 = pack2(q0.x, q0.x), ty2 = pack2(q0.y, q0.y), tz2 = pack2(q0.z, q0.z);
    float ks[NV] = {}, kc[NV] = {};
    for (int rb = r0; rb < r1; rb += kP2pRanges) {
      // places of the ranges in their concatenation (heavy ones empty)
      if (threadIdx.x < kP2pRanges) {
        const int rr = rb + threadIdx.x;
        int first = 0, len = 0;
        if (rr < r1) {
          const int la = BIG ? ia : near_rng[2 * rr], lb = BIG ? ib : near_rng[2 * rr + 1];
          if (lb > la) {
            first = be[la].x;
            len = be[lb - 1].y - first;
            if (!BIG && len > kBigRange) len = 0;   // chunked by the BIG pass
          }
        }
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(kFull, incl, o);
          if (threadIdx.x >= o) incl += v;
        }
        rs[threadIdx.x] = first;
        rp[threadIdx.x] = incl - len;
        if (threadIdx.x == kP2pRanges - 1) s_tot = incl;
      }
      __syncthreads();
      const int tot = s_tot;
      // no tile and none of its barriers (every range heavy): the next ranges
      // wait until all threads have read this total
      if (tot == 0) __syncthreads();
      for (int k0 = 0; k0 < tot; k0 += 2 * T) {
        const int np = min(T, (tot - k0 + 1) / 2);   // pairs of this tile
        if (threadIdx.x < np) {
          const int k = k0 + 2 * threadIdx.x;
          int g = 0;                                 // last range that starts at or before k
#pragma unroll
          for (int o = kP2pRanges / 2; o > 0; o >>= 1)
            if (rp[g + o] <= k) g += o;
          float x[2], y[2], z[2], q[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            if (e == 1)
              while (g < kP2pRanges - 1 && rp[g + 1] <= k + 1) ++g;
            const bool in = k + e < tot;
            const int j = in ? rs[g] + (k + e - rp[g]) : -1;
            tj[2 * threadIdx.x + e] = j;
            if (in) {
              const float4 hi = phi[j], lo = plo[j];
              x[e] = (tch.x - hi.x) + (tcl.x - lo.x);
              y[e] = (tch.y - hi.y) + (tcl.y - lo.y);
              z[e] = (tch.z - hi.z) + (tcl.z - lo.z);
              q[e] = hi.w;
            } else {                                 // no source: no charge, far away
              x[e] = 1e18f;
              y[e] = z[e] = q[e] = 0.f;
            }
          }
          tA[threadIdx.x] = make_ulonglong2(pack2(x[0], x[1]), pack2(y[0], y[1]));
          tB[threadIdx.x] = make_ulonglong2(pack2(z[0], z[1]), pack2(q[0], q[1]));
        }
        __syncthreads();
        if (active) {
          unsigned close = 0;   // 1 + pair of the last close pair, above it the one before
          for (int p0 = sub; p0 < np; p0 += run * S) {
            const int p1 = min(np, p0 + run * S);
            uint64_t p2[NV];
#pragma unroll
            for (int c = 0; c < NV; ++c) p2[c] = 0ull;
#pragma unroll 2
            for (int p = p0; p < p1; p += S) {
              const ulonglong2 A = tA[p], B = tB[p];
              const uint64_t dx = add2(tx2, A.x), dy = add2(ty2, A.y), dz = add2(tz2, B.x);
              const uint64_t r2 = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
              float ra, rb2;
              unpack2(r2, ra, rb2);
              const bool ca = ra < thr2, cb = rb2 < thr2;
              if (ca || cb) close = (close << 16) + (unsigned)(p + 1);
              const uint64_t inv = pack2(ca ? 0.f : rsqrt_ftz(ra), cb ? 0.f : rsqrt_ftz(rb2));
              const uint64_t qi = mul2(B.y, inv);
              p2[0] = add2(p2[0], qi);
              if (FIELD) {
                const uint64_t q3 = mul2(qi, mul2(inv, inv));
                p2[NV > 1 ? 1 : 0] = fma2(q3, dx, p2[NV > 1 ? 1 : 0]);
                p2[NV > 1 ? 2 : 0] = fma2(q3, dy, p2[NV > 1 ? 2 : 0]);
                p2[NV > 1 ? 3 : 0] = fma2(q3, dz, p2[NV > 1 ? 3 : 0]);
              }
            }
#pragma unroll
            for (int c = 0; c < NV; ++c) {
              float lo, hi;
              unpack2(p2[c], lo, hi);
              kahan(ks[c], kc[c], lo + hi);
            }
          }
          if (close) {
            // close pairs, left out above, from the FP64 positions (nothing
            // for the point itself or inside the field guard).  Mostly the
            // point itself alone, whose place is known; else the part is
            // searched
            const bool one = close < 65536u;
            for (int p = one ? (int)close - 1 : sub; p < np; p += one ? T : S) {
              const float4 fa = reinterpret_cast<const float4 *>(tA)[p],
                           fb = reinterpret_cast<const float4 *>(tB)[p];
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const float dx = q0.x + (e ? fa.y : fa.x), dy = q0.y + (e ? fa.w : fa.z),
                            dz = q0.z + (e ? fb.y : fb.x);
                const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                if (!(r2 < thr2)) continue;
                const int j = tj[2 * p + e];
                if (j < 0) continue;
                if (j == t) continue;
                const float sq = e ? fb.w : fb.z;
                const float ex = (float)(sx[t] - sx[j]), ey = (float)(sy[t] - sy[j]),
                            ez = (float)(sz[t] - sz[j]);
                const float e2 = ex * ex + ey * ey + ez * ez;
                if (!(FIELD ? (e2 > 1e-10f) : (e2 > 0.f))) continue;
                const float inv = rsqrt_ftz(e2);
                const float qi = sq * inv;
                kahan(ks[0], kc[0], qi);
                if (FIELD) {
                  const float q3 = qi * (inv * inv);
                  kahan(ks[NV > 1 ? 1 : 0], kc[NV > 1 ? 1 : 0], q3 * ex);
                  kahan(ks[NV > 1 ? 2 : 0], kc[NV > 1 ? 2 : 0], q3 * ey);
                  kahan(ks[NV > 1 ? 3 : 0], kc[NV > 1 ? 3 : 0], q3 * ez);
                }
              }
            }
          }
        }
        __syncthreads();
      }
    }
    // a target's parts added by one thread per value, compensated, and
    // stored (the field is minus the gradient's sum)
#pragma unroll
    for (int c = 0; c < NV; ++c) {
      red[c][threadIdx.x] = ks[c];
      red[NV + c][threadIdx.x] = kc[c];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < rem * NV; i += T) {
      const int tt = i / NV, c = i - tt * NV;
      float s = red[c][tt], e = -red[NV + c][tt];
      for (int k = 1; k < S; ++k) {
        const float v = red[c][tt + k * rem];
        const float n = s + v, bb = n - s;
        e += ((s - (n - bb)) + (v - bb)) - red[NV + c][tt + k * rem];
        s = n;
      }
      const double v = (double)s + (double)e;
      const int64_t o = tbe.x + tb + tt;
      double *dst = c == 0 ? acc_pot + o : acc_fld + 3 * o + (c - 1);
      const double w = c == 0 ? v : -v;
      if (BIG) atomicAdd(dst, w);
      else *dst = w;
    }
    __syncthreads();
  }
}

// A leaf above the capacity (depth limit, leaf predicate) goes to several blocks, T
// targets at a time; not too many, as most leaves have none for them.  6,000
// coincident points in one leaf at capacity 16: mixed 7.3 ms, 208 with one block of
// 64 threads (104 with a warp per leaf and chunks of 128 threads), FP64 11 ms, 83.
int leaf_tiles(const DevTree &t, int T) {
  return std::min({ceil_div(t.max_leaf, T), 2048 / T, 1 + 100000 / t.nleaves});
}

template <bool FIELD>
void launch_mixed(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  // 64 threads per leaf at leaf capacities up to 24, 128 above (1M Plummer,
  // 400k uniform, 300k blobs: 0.77, 0.18, 0.27 ms at capacity 20 with 64, 0.92,
  // 0.20, 0.31 with 128; 2.08, 0.17, 0.63 and 1.27, 0.19, 0.57 at 64).  (The
  // capacity and not the mean occupancy: a system's bits do not depend on
  // its company in a forest.)
  const bool small = s->cfg.maxbox <= 24;
  const int T = small ? 64 : 128;
  const int tiles = leaf_tiles(t, T);
  auto run = [&](auto kern, int grid) {
    kern<<<dim3(grid, tiles), T, 0, st>>>(
        t.big_items.ptr, t.near_off.ptr, t.near_rng.ptr, t.leaf_be.ptr, t.leaf_chi.ptr,
        t.leaf_clo.ptr, s->sx.ptr, s->sy.ptr, s->sz.ptr, s->rel32.ptr, s->abs_hi.ptr,
        s->abs_lo.ptr, s->acc_pot.ptr, s->acc_fld.ptr);
    ACHECK(cudaGetLastError());
    s->launches++;
  };
  run(small ? k_p2p_tile<FIELD, false, 64> : k_p2p_tile<FIELD, false, 128>, t.nleaves);
  if (t.n_big) run(small ? k_p2p_tile<FIELD, true, 64> : k_p2p_tile<FIELD, true, 128>, t.n_big);
}

template <bool FIELD, bool BIG>
void launch_fp64(AranGpuSolver3d *s, int grid, cudaStream_t st) {
  DevTree &t = s->tree;
  k_p2p64<FIELD, BIG><<<dim3(grid, leaf_tiles(t, 128)), 128, 0, st>>>(
      t.big_items.ptr, t.near_off.ptr, t.near_rng.ptr, t.leaf_be.ptr, s->sx.ptr, s->sy.ptr,
      s->sz.ptr, s->sq.ptr, s->acc_pot.ptr, s->acc_fld.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
}

}  // namespace

void build_p2p_work(AranGpuSolver3d *s) {
  cudaStream_t st = s->s0;
  DevTree &t = s->tree;
  const int TB = 256;
  int nl = t.nleaves;
  t.leaf_be.reserve(nl);
  t.leaf_chi.reserve(nl);
  t.leaf_clo.reserve(nl);
  double ex = s->cfg.ub[0] - s->cfg.lb[0], ey = s->cfg.ub[1] - s->cfg.lb[1],
         ez = s->cfg.ub[2] - s->cfg.lb[2];
  k_leaf_info<<<ceil_div(nl, TB), TB, 0, st>>>(nl, t.leaf_node.ptr, t.begin.ptr, t.end.ptr,
                                               t.depth.ptr, t.center.ptr, t.sys.ptr,
                                               s->sys_box.ptr, ex, ey, ez,
                                               t.leaf_be.ptr, t.leaf_chi.ptr, t.leaf_clo.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  if (t.n_big) {
    t.big_items.reserve(t.n_big);
    k_big_items<<<t.n_heavy, 64, 0, st>>>(t.big_rng.ptr + 2, nl, t.near_off.ptr, t.near_rng.ptr,
                                       t.leaf_be.ptr, t.big_items.ptr);
    ACHECK(cudaGetLastError());
    s->launches++;
  }
}

void launch_p2p(AranGpuSolver3d *s, cudaStream_t st) {
  const bool mixed = s->cfg.precision == ARAN_PRECISION_MIXED;
  const bool field = s->cfg.field != 0;
  if (mixed) {
    if (field) launch_mixed<true>(s, st);
    else launch_mixed<false>(s, st);
  } else {
    const int nb = s->tree.n_big;
    if (field) {
      launch_fp64<true, false>(s, s->tree.nleaves, st);
      if (nb) launch_fp64<true, true>(s, nb, st);
    } else {
      launch_fp64<false, false>(s, s->tree.nleaves, st);
      if (nb) launch_fp64<false, true>(s, nb, st);
    }
  }
}

}  // namespace aran
