// p2p.cu -- the near field (P2P) on the device.
//
// LibAran calls the user p2p callback for every pair of points of every near
// leaf pair (near_func, aran/aransolver3d.c:254-324) with the Newton kernels
// of tests/newtonpot3.c:61-78 (potential) and tests/newtonfield3.c:91-119
// (field, |r| > 1e-5 guard).  Here every target particle sums its near
// sources directly (both sides of a pair are evaluated by their own targets
// instead of the symmetric update).
//
// Work decomposition: mixed precision takes a warp per target leaf
// (k_p2p_warp), FP64 a block (k_p2p64).  Near ranges of more than kBigRange
// points (a coarse leaf next to a deep subtree, common in clustered sets) are
// cut into leaf-aligned chunks processed by extra blocks that accumulate
// atomically.
//
// Mixed precision: positions are FP32 relative to their leaf centre, the
// centre difference comes from FP32 hi+lo centre pairs, per-source-leaf FP32
// partial sums go into FP64 accumulators, and pairs closer than 1/8 of the
// target leaf size (where FP32 cancellation would show) are recomputed from
// the FP64 positions.
#include <cub/cub.cuh>

#include <type_traits>

#include "internal.cuh"

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
                            double ex, double ey, double ez, int2 *__restrict__ be,
                            float4 *__restrict__ chi, float4 *__restrict__ clo) {
  int L = blockIdx.x * blockDim.x + threadIdx.x;
  if (L >= nleaves) return;
  int node = leaf_node[L];
  be[L] = make_int2(begin[node], end[node]);
  double cx = center[3 * node], cy = center[3 * node + 1], cz = center[3 * node + 2];
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

// one chunk of a heavy near range of a mixed solve: threads-per-target (tpt)
// grows as the leaf shrinks (n <= 8: 16, <= 16: 8, <= 32: 4, <= 64: 2, else
// 1), and a target's tpt threads take the chunk's leaves round-robin (tiny
// target leaves) or split every source leaf's points
template <bool FIELD>
__global__ void __launch_bounds__(128, 10) k_p2p_chunk(
    const int4 *__restrict__ items, const int2 *__restrict__ be, const float4 *__restrict__ chi,
    const float4 *__restrict__ clo, const double *__restrict__ sx, const double *__restrict__ sy,
    const double *__restrict__ sz, const real4<float> *__restrict__ rel32,
    double *__restrict__ acc_pot, double *__restrict__ acc_fld) {
  const int4 it = items[blockIdx.x];
  const int L = it.x, ia = it.y, ib = it.z;
  const int2 tbe = be[L];
  const int b = tbe.x, nt = tbe.y - tbe.x;
  const int tpt = nt <= 8 ? 16 : (nt <= 16 ? 8 : (nt <= 32 ? 4 : (nt <= 64 ? 2 : 1)));
  const int gsz = blockDim.x / tpt;
  const int sub = threadIdx.x % tpt;
  const bool leaf_strided = nt <= 8;
  const float4 tch = chi[L], tcl = clo[L];
  for (int tb = 0; tb < nt; tb += gsz) {
    const int ti = tb + threadIdx.x / tpt;
    const bool active = ti < nt;
    if (!__any_sync(kFull, active)) continue;   // a warp with no target of this pass
    const int t = b + (active ? ti : 0);
    // per-source-leaf FP32 sums are added with Kahan compensation in FP32
    // (FP64 adds per leaf would occupy the FP64 pipe, 1/64 of FP32)
    float ks0 = 0.f, ks1 = 0.f, ks2 = 0.f, ks3 = 0.f;
    float kc0 = 0.f, kc1 = 0.f, kc2 = 0.f, kc3 = 0.f;
    auto kahan = [](float &sum, float &comp, float v) {
      const float y = v - comp;
      const float t2 = sum + y;
      comp = (t2 - sum) - y;
      sum = t2;
    };
    const double tx64 = sx[t], ty64 = sy[t], tz64 = sz[t];
    const real4<float> r = rel32[t];
    auto do_leaf = [&](int lf, int j0, int js) {
      const int2 sbe = be[lf];
      const float4 sh = chi[lf], sl = clo[lf];
      // target position relative to the source leaf centre
      const float ox = r.x - ((sh.x - tch.x) + (sl.x - tcl.x));
      const float oy = r.y - ((sh.y - tch.y) + (sl.y - tcl.y));
      const float oz = r.z - ((sh.z - tch.z) + (sl.z - tcl.z));
      const float thr2 = tch.w;
      float p0 = 0.f, f0 = 0.f, f1 = 0.f, f2 = 0.f;
#pragma unroll 4
      for (int j = sbe.x + j0; j < sbe.y; j += js) {
        const real4<float> sj = rel32[j];
        float dx = ox - sj.x, dy = oy - sj.y, dz = oz - sj.z;
        float r2 = dx * dx + dy * dy + dz * dz;
        if (__builtin_expect(r2 < thr2, 0)) {
          if (j == t) {
            r2 = 0.f;
          } else {
            // close pair: difference from the FP64 positions
            dx = (float)(tx64 - sx[j]);
            dy = (float)(ty64 - sy[j]);
            dz = (float)(tz64 - sz[j]);
            r2 = dx * dx + dy * dy + dz * dz;
          }
        }
        const bool ok = FIELD ? (r2 > 1e-10f) : (r2 > 0.f);
        const float inv = ok ? rsqrt_ftz(r2) : 0.f;
        const float qi = sj.q * inv;
        p0 += qi;
        if (FIELD) {
          const float q3 = qi * inv * inv;
          f0 -= q3 * dx;
          f1 -= q3 * dy;
          f2 -= q3 * dz;
        }
      }
      kahan(ks0, kc0, p0);
      if (FIELD) {
        kahan(ks1, kc1, f0);
        kahan(ks2, kc2, f1);
        kahan(ks3, kc3, f2);
      }
    };
    if (leaf_strided)
      for (int lf = ia + sub; lf < ib; lf += tpt) do_leaf(lf, 0, 1);
    else
      for (int lf = ia; lf < ib; ++lf) do_leaf(lf, sub, tpt);
    double v[4] = {(double)ks0 - (double)kc0, (double)ks1 - (double)kc1,
                   (double)ks2 - (double)kc2, (double)ks3 - (double)kc3};
    for (int o = 1; o < tpt; o <<= 1)
#pragma unroll
      for (int c = 0; c < (FIELD ? 4 : 1); ++c) v[c] += __shfl_xor_sync(kFull, v[c], o);
    if (active && sub == 0) {
      atomicAdd(&acc_pot[t], v[0]);
      if (FIELD)
        for (int c = 0; c < 3; ++c) atomicAdd(&acc_fld[3 * (size_t)t + c], v[1 + c]);
    }
  }
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
  for (int tb = 0; tb < nt; tb += 128) {
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

// Mixed near field, one warp per target leaf (four per block).  The warp
// walks the leaf's near source leaves; for each it stages up to 32 source
// points in shared memory, shifted to the target leaf's frame by the lane
// that loads them, and every lane sums them against its own targets from
// broadcast reads: lanes per target S = 32 / (n rounded up to a power of
// two) for n <= 16, else 1 (32 targets per pass), so the per-leaf set-up (centres, Kahan adds of the
// leaf partials) is paid once per lane per source leaf.  The pair loop has no
// branch: the distance is clamped below at h/8, and a lane whose chunk held a
// closer pair (or the point itself) takes the stand-ins back and adds those
// pairs from the FP64 positions afterwards.
// Ranges of more than kBigRange points are left to the chunked pass.
template <bool FIELD>
__global__ void __launch_bounds__(128, 8) k_p2p_warp(
    int nleaves, const int *__restrict__ near_off, const int *__restrict__ near_rng,
    const int2 *__restrict__ be, const float4 *__restrict__ chi, const float4 *__restrict__ clo,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const real4<float> *__restrict__ rel32, double *__restrict__ acc_pot,
    double *__restrict__ acc_fld) {
  __shared__ float4 sbuf[4][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int L = blockIdx.x * 4 + w;
  if (L >= nleaves) return;
  const int2 tbe = be[L];
  const int b = tbe.x, nt = tbe.y - tbe.x;
  // lanes per target as a compile-time constant: one body per S
  const int Sd = nt <= 1 ? 32 : (nt <= 2 ? 16 : (nt <= 4 ? 8 : (nt <= 8 ? 4 : (nt <= 16 ? 2 : 1))));
  auto body = [&](auto sc) {
  constexpr int S = decltype(sc)::value;
  const int sub = lane & (S - 1);
  const float4 tch = chi[L], tcl = clo[L];
  const float thr2 = FIELD ? fmaxf(tch.w, 1e-10f) : tch.w;
  const int r0 = near_off[L], r1 = near_off[L + 1];
  float4 *buf = sbuf[w];
  const int step = 32 / S;
  for (int tb = 0; tb < nt; tb += step) {
    const int ti0 = tb + lane / S;
    const bool act0 = ti0 < nt;
    const int t0 = b + (act0 ? ti0 : 0);
    const real4<float> q0 = rel32[t0];
    float ks[4] = {}, kc[4] = {};
    auto kahan = [](float &sum, float &comp, float v) {
      const float y = v - comp;
      const float t2 = sum + y;
      comp = (t2 - sum) - y;
      sum = t2;
    };
    // one target against a staged source, r2 clamped below at thr2 (h/8
    // squared, at least the field guard 1e-10): close pairs and the point
    // itself add a bounded stand-in that close_fix takes back
    auto pair = [&](const real4<float> &q, const float4 &sv, float *p, float &rmin) {
      const float dx = q.x - sv.x, dy = q.y - sv.y, dz = q.z - sv.z;
      const float r2 = dx * dx + dy * dy + dz * dz;
      rmin = fminf(rmin, r2);
      const float inv = rsqrt_ftz(fmaxf(r2, thr2));
      const float qi = sv.w * inv;
      p[0] += qi;
      if (FIELD) {
        const float q3 = qi * inv * inv;
        p[1] -= q3 * dx;
        p[2] -= q3 * dy;
        p[3] -= q3 * dz;
      }
    };
    // for a close pair: remove the stand-in (the same FP32 expressions) and
    // add the pair from the FP64 positions (nothing for the point itself or
    // inside the field guard)
    auto close_fix = [&](const real4<float> &q, int t, const float4 &sv, int j, float *p) {
      const float dx = q.x - sv.x, dy = q.y - sv.y, dz = q.z - sv.z;
      const float r2 = dx * dx + dy * dy + dz * dz;
      if (!(r2 < thr2)) return;
      {
        const float inv = rsqrt_ftz(fmaxf(r2, thr2));
        const float qi = sv.w * inv;
        p[0] -= qi;
        if (FIELD) {
          const float q3 = qi * inv * inv;
          p[1] += q3 * dx;
          p[2] += q3 * dy;
          p[3] += q3 * dz;
        }
      }
      if (j == t) return;
      const float ex = (float)(sx[t] - sx[j]), ey = (float)(sy[t] - sy[j]),
                  ez = (float)(sz[t] - sz[j]);
      const float e2 = ex * ex + ey * ey + ez * ez;
      if (!(FIELD ? (e2 > 1e-10f) : (e2 > 0.f))) return;
      const float inv = rsqrt_ftz(e2);
      const float qi = sv.w * inv;
      p[0] += qi;
      if (FIELD) {
        const float q3 = qi * inv * inv;
        p[1] -= q3 * ex;
        p[2] -= q3 * ey;
        p[3] -= q3 * ez;
      }
    };
    for (int rr = r0; rr < r1; ++rr) {
      const int la = near_rng[2 * rr], lb = near_rng[2 * rr + 1];
      if (lb <= la) continue;
      if (rng_count(be, la, lb) > kBigRange) continue;  // chunked by the BIG pass
      for (int lf = la; lf < lb; ++lf) {
        const int2 sbe = be[lf];
        const float4 sh = chi[lf], sl = clo[lf];
        // source leaf centre relative to the target leaf centre
        const float cx = (sh.x - tch.x) + (sl.x - tcl.x);
        const float cy = (sh.y - tch.y) + (sl.y - tcl.y);
        const float cz = (sh.z - tch.z) + (sl.z - tcl.z);
        for (int j0 = sbe.x; j0 < sbe.y; j0 += 32) {
          const int cnt = min(32, sbe.y - j0);
          __syncwarp();
          if (lane < cnt) {
            const real4<float> r = rel32[j0 + lane];
            buf[lane] = make_float4(cx + r.x, cy + r.y, cz + r.z, r.q);
          }
          __syncwarp();
          float p0[4] = {0.f, 0.f, 0.f, 0.f};
          float rmin = 3.0e38f;
#pragma unroll 4
          for (int k = sub; k < cnt; k += S) pair(q0, buf[k], p0, rmin);
          const bool flag = rmin < thr2;
          if (__any_sync(kFull, flag) && flag)
            for (int k = sub; k < cnt; k += S) close_fix(q0, t0, buf[k], j0 + k, p0);
#pragma unroll
          for (int c = 0; c < (FIELD ? 4 : 1); ++c) kahan(ks[c], kc[c], p0[c]);
        }
      }
    }
    double v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (double)ks[c] - (double)kc[c];
    for (int o = 1; o < S; o <<= 1)
#pragma unroll
      for (int c = 0; c < (FIELD ? 4 : 1); ++c) v[c] += __shfl_xor_sync(kFull, v[c], o);
    if (act0 && sub == 0) {
      acc_pot[t0] = v[0];
      if (FIELD) {
        acc_fld[3 * (size_t)t0] = v[1];
        acc_fld[3 * (size_t)t0 + 1] = v[2];
        acc_fld[3 * (size_t)t0 + 2] = v[3];
      }
    }
  }
  };
  if (Sd == 32) body(std::integral_constant<int, 32>{});
  else if (Sd == 16) body(std::integral_constant<int, 16>{});
  else if (Sd == 8) body(std::integral_constant<int, 8>{});
  else if (Sd == 4) body(std::integral_constant<int, 4>{});
  else if (Sd == 2) body(std::integral_constant<int, 2>{});
  else body(std::integral_constant<int, 1>{});
}

template <bool FIELD>
void launch_mixed(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  k_p2p_warp<FIELD><<<ceil_div(t.nleaves, 4), 128, 0, st>>>(
      t.nleaves, t.near_off.ptr, t.near_rng.ptr, t.leaf_be.ptr, t.leaf_chi.ptr, t.leaf_clo.ptr,
      s->sx.ptr, s->sy.ptr, s->sz.ptr, s->rel32.ptr, s->acc_pot.ptr, s->acc_fld.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  if (!t.n_big) return;
  k_p2p_chunk<FIELD><<<t.n_big, 128, 0, st>>>(
      t.big_items.ptr, t.leaf_be.ptr, t.leaf_chi.ptr, t.leaf_clo.ptr, s->sx.ptr, s->sy.ptr,
      s->sz.ptr, s->rel32.ptr, s->acc_pot.ptr, s->acc_fld.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
}

template <bool FIELD, bool BIG>
void launch_fp64(AranGpuSolver3d *s, int grid, cudaStream_t st) {
  DevTree &t = s->tree;
  k_p2p64<FIELD, BIG><<<grid, 128, 0, st>>>(
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
                                               t.depth.ptr, t.center.ptr, ex, ey, ez,
                                               t.leaf_be.ptr, t.leaf_chi.ptr, t.leaf_clo.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
  // chunk total and heavy-range count, as k_near listed them
  int *hb = s->h_small + 8;   // pinned
  hb[0] = hb[1] = 0;
  if (t.n_near_rng > 0) {
    ACHECK(cudaMemcpyAsync(hb, t.big_rng.ptr, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    ACHECK(cudaStreamSynchronize(st));
  }
  const int nbig = hb[0], nheavy = hb[1];
  t.n_big = nbig;
  if (nbig) {
    t.big_items.reserve(nbig);
    k_big_items<<<nheavy, 64, 0, st>>>(t.big_rng.ptr + 2, nl, t.near_off.ptr, t.near_rng.ptr,
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
