// leaf_ops.cuh -- FP32 P2M and L2P with the order a compile-time constant (the
// even orders 4 to 16, one translation unit per group of orders); passes.cu
// holds the kernels of FP64 and the other orders.  4M Plummer particles (leaf
// 64, field) on GB300, P2M + L2P: order 16 0.88 + 1.51 ms (2.04 + 2.16 with
// passes.cu's), order 10 0.40 + 0.40 (0.88 + 0.94), order 12 P2M 0.47 (0.97 with
// the same butterflies, their buffer in local memory), order 8 P2M 0.38 (0.60).
#pragma once

#include "internal.cuh"
#include "f32x2.cuh"

namespace aran {

namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float leaf_inv_scale(int depth, double scale_e) {
  // 1/h_d = 2^d / 2^E (exact power of two)
  return (float)(ldexp(1.0, depth) / scale_e);
}

// P2M (passes.cu k_p2m's sums, one warp per leaf) with the sum over a leaf's
// particles done by butterflies: the terms of each particle (lane) are made
// in m-major order (the recurrence's natural order) into a 32-value buffer;
// each full buffer is summed over the warp by one butterfly of 31 shuffles
// (afterwards lane k holds value k of the batch) instead of a 5-shuffle tree
// per value, and the lanes' batch sums add up over the leaf's chunks.
template <int P>
__global__ void __launch_bounds__(128) k_p2m_bfly(int nleaves, const int *__restrict__ leaf_node,
                                               const int *__restrict__ begin,
                                               const int *__restrict__ end,
                                               const uint8_t *__restrict__ depth,
                                               const real4<float> *__restrict__ rel,
                                               const float *__restrict__ rec_g,
                                               const float *__restrict__ p2mf_g, double scale_e,
                                               float *__restrict__ mult) {
  constexpr int NM = P * (P + 1) / 2, NV = 2 * NM, NB = (NV + 31) / 32;
  __shared__ float rec[(P + 1) * (P + 2)];
  __shared__ float p2mf[P + 1];
  for (int i = threadIdx.x; i < (P + 1) * (P + 2); i += blockDim.x) rec[i] = rec_g[i];
  for (int i = threadIdx.x; i <= P; i += blockDim.x) p2mf[i] = p2mf_g[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int L = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (L >= nleaves) return;
  const int node = leaf_node[L];
  const int b = begin[node], e = end[node];
  const float ih = leaf_inv_scale(depth[node], scale_e);
  float acc[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) acc[k] = 0.f;
  for (int base = b; base < e; base += 32) {
    const int i = base + lane;
    float x = 0.f, y = 0.f, z = 0.f, q = 0.f;
    if (i < e) {
      const real4<float> r = rel[i];
      x = r.x * ih;
      y = r.y * ih;
      z = r.z * ih;
      q = r.q;
    }
    const float r2 = x * x + y * y + z * z;
    float u[32];
    float dre = rec[0], dim = 0.f;
    static_for<P>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      if (m > 0) {
        const float a = rec[2 * tri(m, m)];
        const float nre = a * (x * dre - y * dim), nim = a * (x * dim + y * dre);
        dre = nre;
        dim = nim;
      }
      float s1re = dre, s1im = dim, s2re = 0.f, s2im = 0.f;
#pragma unroll
      for (int l = m; l < P; ++l) {
        float sre = dre, sim = dim;
        if (l > m) {
          const float c0 = rec[2 * tri(l, m)], c1 = rec[2 * tri(l, m) + 1];
          sre = c0 * z * s1re - c1 * r2 * s2re;
          sim = c0 * z * s1im - c1 * r2 * s2im;
          s2re = s1re;
          s2im = s1im;
          s1re = sre;
          s1im = sim;
        }
        const float f = q * p2mf[l];
        // value index 2 slot + part, slot the m-major place of (l, m)
        const int kr = 2 * (m * P - m * (m - 1) / 2 + (l - m));
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const int k = kr + part;
          u[k & 31] = part ? -f * sim : f * sre;
          if ((k & 31) == 31 || k == NV - 1) {
            if (k == NV - 1)            // last, partial batch: zero its tail
#pragma unroll
              for (int t = 0; t < 32; ++t)
                if (t > (k & 31)) u[t] = 0.f;
            // butterfly: the lane keeps the half whose index bit o matches
            // its lane bit and adds the partner's half; lane j ends with
            // value j of the batch summed over the warp
#pragma unroll
            for (int st = 0; st < 5; ++st) {
              const int o = 16 >> st, n = 32 >> st;
              const bool upper = (lane & o) != 0;
#pragma unroll
              for (int t = 0; t < n / 2; ++t) {
                const float send = upper ? u[t] : u[t + n / 2];
                const float keep = upper ? u[t + n / 2] : u[t];
                u[t] = keep + __shfl_xor_sync(kFull, send, o);
              }
            }
            acc[k >> 5] += u[0];
          }
        }
      }
    });
  }
  // lane k of batch bt holds m-major value 32 bt + k: slot (l, m), part
#pragma unroll
  for (int bt = 0; bt < NB; ++bt) {
    const int kv = 32 * bt + lane;
    if (kv >= NV) continue;
    int slot = kv >> 1, m = 0;
    while (slot > P - 1 - m) {
      slot -= P - m;
      ++m;
    }
    const int l = m + slot;
    mult[(size_t)node * NV + 2 * tri(l, m) + (kv & 1)] = acc[bt];
  }
}

// ---------------------------------------------------------------------------
// FP32 L2P (+ gradient) over windows of 32 consecutive particles (leaf
// order), the order P a compile-time constant: the same evaluation as k_l2p,
// with every lane busy whatever the leaves' sizes.  Warp w takes particles
// 32 w .. 32 w + 31, which belong to leaves win_leaf[w] onwards (at most
// 32 of them); each lane evaluates with its own leaf's coefficients, staged
// four leaves at a time in shared memory: the local with the m-weight
// (2 for m > 0) folded in and, for the gradient, the d/dz local and the
// (d/dx - i d/dy) local's m' = m and m' = -m parts combined per (l, m) into
// the two real vectors that multiply (Re S, Im S) for its real and
// imaginary parts (S^{-m} = (-1)^m conj(S^m)).  Each term is formed, then
// added to its sum once.  The solid harmonics run by degree (outer,
// unrolled) and order (inner), so every table offset is a constant.
// ---------------------------------------------------------------------------
// leaves staged at a time per warp
template <int P>
constexpr int kWinSlots = P <= 12 ? 4 : 2;
constexpr int kWinWarps = 4;     // warps per block

template <int P, bool FIELD>
__host__ __device__ constexpr int win_slot() {   // float2 per staged leaf
  return (P + 1) * (P + 2) / 2 + (FIELD ? 3 * (P * (P + 1) / 2) : 0);
}

template <int P, bool FIELD>
__global__ void __launch_bounds__(32 * kWinWarps)
    k_l2p_win(int64_t n, int nleaves, const int *__restrict__ win_leaf,
              const int *__restrict__ leaf_node, const int *__restrict__ begin,
              const uint8_t *__restrict__ depth, const real4<float> *__restrict__ rel,
              const float *__restrict__ rec_g, const float *__restrict__ gz_g,
              const float *__restrict__ gm_g, double scale_e, const cplx<float> *__restrict__ loc,
              double *__restrict__ acc_pot, double *__restrict__ acc_fld) {
  constexpr int NL = (P + 1) * (P + 2) / 2, NM = P * (P + 1) / 2;
  constexpr int SLOT = win_slot<P, FIELD>();
  __shared__ __align__(8) float rec[2 * NL];
  __shared__ uint8_t lmt[2 * NL];
  __shared__ float2 coef[kWinWarps][kWinSlots<P>][SLOT];
  for (int i = threadIdx.x; i < 2 * NL; i += blockDim.x) rec[i] = rec_g[i];
  for (int c = threadIdx.x; c < NL; c += blockDim.x) {
    int l = 0;
    while ((l + 1) * (l + 2) / 2 <= c) ++l;
    lmt[2 * c] = (uint8_t)l;
    lmt[2 * c + 1] = (uint8_t)(c - l * (l + 1) / 2);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t wid = (int64_t)blockIdx.x * kWinWarps + w;
  const int64_t j0 = wid * 32;
  if (j0 >= n) return;
  // the window's leaves: lane k holds leaf win_leaf + k (node, first particle)
  const int L0 = win_leaf[wid];
  int nd_k = -1;
  int64_t b_k = INT64_MAX;
  if (L0 + lane < nleaves) {
    nd_k = leaf_node[L0 + lane];
    b_k = begin[nd_k];
  }
  // bit i: particle j0 + i starts a leaf after the window's first
  const unsigned bit = (lane >= 1 && b_k > j0 && b_k < j0 + 32) ? 1u << (int)(b_k - j0) : 0u;
  const unsigned M = __reduce_or_sync(kFull, bit);
  const int nslots = __popc(M) + 1;
  const int64_t j = j0 + lane;
  const bool act = j < n;
  const int slot = __popc(M & ((2u << lane) - 1u));
  const int nd = __shfl_sync(kFull, nd_k, slot);
  const float ih = leaf_inv_scale(act ? depth[nd] : 0, scale_e);
  const real4<float> r = act ? rel[j] : real4<float>{0.f, 0.f, 0.f, 0.f};
  const float x = r.x * ih, y = r.y * ih, z = r.z * ih;
  const float r2 = x * x + y * y + z * z;
  float phi = 0.f, dz = 0.f, gre = 0.f, gim = 0.f;
  for (int g0 = 0; g0 < nslots; g0 += kWinSlots<P>) {
    // stage leaves g0 .. g0 + 3 of the window
    __syncwarp();
    for (int sidx = 0; sidx < kWinSlots<P> && g0 + sidx < nslots; ++sidx) {
      const int node = __shfl_sync(kFull, nd_k, g0 + sidx);
      const cplx<float> *Lg = loc + (size_t)node * NL;
      float2 *cf = coef[w][sidx];
      for (int c = lane; c < NL; c += 32) {
        const cplx<float> v = Lg[c];
        const float wm = lmt[2 * c + 1] ? 2.f : 1.f;
        cf[c] = make_float2(wm * v.re, wm * v.im);
      }
      if (FIELD)
        for (int c = lane; c < NM; c += 32) {
          const int l = lmt[2 * c], m = lmt[2 * c + 1];
          const float wm = m ? 2.f : 1.f;
          // d/dz: L(l+1, m) gz
          const cplx<float> a = Lg[(l + 1) * (l + 2) / 2 + m];
          const float gz = gz_g[c];
          cf[NL + c] = make_float2(wm * gz * a.re, wm * gz * a.im);
          // (d/dx - i d/dy), m' = m: bp = L(l+1, m+1) gm[l^2 + l + m]
          const cplx<float> vp = Lg[(l + 1) * (l + 2) / 2 + m + 1];
          const float gp = gm_g[l * l + l + m];
          const float bpr = gp * vp.re, bpi = gp * vp.im;
          // m' = -m (m > 0): source order 1 - m, times (-1)^m for S^{-m}
          float bnr = 0.f, bni = 0.f;
          if (m > 0) {
            const float gn = gm_g[l * l + l - m];
            cplx<float> u;
            if (m == 1) u = Lg[(l + 1) * (l + 2) / 2];
            else {
              const cplx<float> v = Lg[(l + 1) * (l + 2) / 2 + m - 1];
              u = ((m - 1) & 1) ? cmake<float>(-v.re, v.im) : cmake<float>(v.re, -v.im);
            }
            const float sg = (m & 1) ? -gn : gn;
            bnr = sg * u.re;
            bni = sg * u.im;
          }
          // real part bp S + bn conj(S): (bpr + bnr) Re S + (bni - bpi) Im S;
          // imaginary part: (bpi + bni) Re S + (bpr - bnr) Im S
          cf[NL + NM + c] = make_float2(bpr + bnr, bni - bpi);
          cf[NL + 2 * NM + c] = make_float2(bpi + bni, bpr - bnr);
        }
    }
    __syncwarp();
    if (act && slot >= g0 && slot < g0 + kWinSlots<P>) {
      const float2 *cf = coef[w][slot - g0];
      // s1[m] = S_{l-1}^m, s2[m] = S_{l-2}^m
      float s1r[P + 1], s1i[P + 1], s2r[P + 1], s2i[P + 1];
#pragma unroll
      for (int l = 0; l <= P; ++l) {
        // the diagonal term first: S_l^l = a_l (x + i y) S_{l-1}^{l-1}
        float Sr, Si;
        if (l == 0) {
          Sr = rec[0];
          Si = 0.f;
        } else {
          const float a = rec[2 * (l * (l + 1) / 2 + l)];
          Sr = a * (x * s1r[l - 1] - y * s1i[l - 1]);
          Si = a * (x * s1i[l - 1] + y * s1r[l - 1]);
        }
        float dr[P + 1], di[P + 1];
        dr[l] = Sr;
        di[l] = Si;
#pragma unroll
        for (int m = 0; m < l; ++m) {
          const float2 cc = *reinterpret_cast<const float2 *>(&rec[2 * (l * (l + 1) / 2 + m)]);
          const float t0 = cc.x * z, t1 = cc.y * r2;
          const float pr = m + 1 < l ? s2r[m] : 0.f, pi = m + 1 < l ? s2i[m] : 0.f;
          dr[m] = t0 * s1r[m] - t1 * pr;
          di[m] = t0 * s1i[m] - t1 * pi;
        }
#pragma unroll
        for (int m = 0; m <= l; ++m) {
          const int c = l * (l + 1) / 2 + m;
          const float Sr_ = dr[m], Si_ = di[m];
          const float2 Lv = cf[c];
          phi += fmaf(Lv.x, Sr_, -Lv.y * Si_);
          if (FIELD && l < P) {
            const float2 a = cf[NL + c];
            dz += fmaf(a.x, Sr_, -a.y * Si_);
            const float2 gr = cf[NL + NM + c], gi = cf[NL + 2 * NM + c];
            gre += fmaf(gr.x, Sr_, gr.y * Si_);
            gim += fmaf(gi.x, Sr_, gi.y * Si_);
          }
          if (m < l) {
            s2r[m] = s1r[m];
            s2i[m] = s1i[m];
          }
          s1r[m] = Sr_;
          s1i[m] = Si_;
        }
      }
    }
  }
  if (act) {
    acc_pot[j] += (double)phi;
    if (FIELD) {
      acc_fld[3 * j] += (double)(gre * ih);
      acc_fld[3 * j + 1] += (double)(-gim * ih);
      acc_fld[3 * j + 2] += (double)(dz * ih);
    }
  }
}

template <int P>
void leaf_p2m(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  constexpr int WPB = 4;
  k_p2m_bfly<P><<<ceil_div(t.nleaves, WPB), WPB * 32, 0, st>>>(
      t.nleaves, t.leaf_node.ptr, t.begin.ptr, t.end.ptr, t.depth.ptr, s->rel32.ptr,
      s->t32.rec.ptr, s->t32.p2mf.ptr, s->scale_e, s->mult32.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
}

template <int P>
void leaf_l2p(AranGpuSolver3d *s, cudaStream_t st) {
  DevTree &t = s->tree;
  const int nb = ceil_div((t.n + 31) / 32, kWinWarps);
  if (nb == 0) return;
  auto kern = s->cfg.field ? k_l2p_win<P, true> : k_l2p_win<P, false>;
  kern<<<nb, 32 * kWinWarps, 0, st>>>(
      t.n, t.nleaves, t.win_leaf.ptr, t.leaf_node.ptr, t.begin.ptr, t.depth.ptr, s->rel32.ptr,
      s->t32.rec.ptr, s->t32.gz.ptr, s->t32.gm.ptr, s->scale_e,
      reinterpret_cast<const cplx<float> *>(s->loc32.ptr), s->acc_pot.ptr, s->acc_fld.ptr);
  ACHECK(cudaGetLastError());
  s->launches++;
}

}  // namespace

}  // namespace aran
