// Block eigensolver for 64 < T <= 128: one CTA of TMAX threads (TMAX = 96 or 128;
// 64 when asked for) per matrix, thread i owning row i.
//
// The algorithm is eigh_reg_kernel's (eigh_reg.cuh): Householder
// tridiagonalisation, Sturm counts, the MP rank test, twisted eigenvectors,
// back-transform, modified Gram-Schmidt - with a row per thread instead of rows
// per lane:
//
//  * Householder: row i of the working matrix in thread i's registers (every
//    column index compile-time). Two barriers a step: one after column k is in
//    shared memory, one after p. The norm and p.v are summed by every warp for
//    itself, the matrix-vector product runs on the unscaled column (p_r = tau (sc
//    sum_j a_rj x_j + a_r,k+1)), so the reflector needs no barrier of its own, and
//    A -= v p^T + (p + 2 kc v) v^T needs no second vector. Column k + 1 of the own
//    row is picked once a step and carried through the update. Four loops, one per
//    quarter of the columns, without the column groups that are dead by then.
//  * Eigenvalues: thread j cuts eigenvalue j's interval at two points a round (the
//    eigenvalues that share one cut it into 2 m + 1 parts).
//  * MP rank, twisted vectors and Gram-Schmidt on the first warp, the
//    back-transform with the vectors dealt to the warps.
//
// Measured on B200, eigensolve kernel, against the version with eight barriers a
// step, bisection by the quotient recurrence and LU inverse iteration: 100800
// matrices at T = 96 41.0 -> 24 ms, 5054 2.17 -> 1.3, 10752 at T = 65 3.05 -> 2.0, 4536 at T =
// 127 6.35 -> 3.1. Cycles at T = 96 with 4 CTAs per SM: reduction 171 K (303 K
// before, at 5), eigenvalues 40 K (118 K), vectors 33 K (46 K), back-transform 41 K
// (79 K). Latency bounds it: 15 warps per SM at the 128 registers of 5 CTAs (4 CTAs
// without spills 26.5 ms).
//
// The results agree with the one-warp routines to float32 round-off, and the
// same tests queue patches for the float64 pass.
#pragma once

#include "eigh.cuh"
#include "eigh_reg.cuh"

namespace lrd {

// Start of quarter q's reflectors in HV: the rows of a quarter are stored from its
// first column group on (TMAX - q TMAX / 4 floats each).
template <int TMAX>
__host__ __device__ constexpr int eigh_cta_hv_at(int q) {
  return TMAX / 4 * (q * TMAX - TMAX / 4 * (q * (q - 1) / 2));
}

// Shared-memory floats: HV, d, e, tau, lam, and the
// column, reflector and p of a step (7 TMAX), the work area W (the vectors' factors,
// 2 TMAX kInvGroup; before them the Sturm coefficients, points and counts, or the
// MP scratch), 8 scalars.
template <int TMAX>
__host__ __device__ constexpr size_t eigh_cta_smem_floats() {
  return eigh_cta_hv_at<TMAX>(4) + 7 * (size_t)TMAX + (size_t)2 * TMAX * kInvGroup + 8;
}

// One CTA of TMAX threads per patch: the body solves the launch's patch ``b``
// (patch index patch0 + b), n <= TMAX. ``gram`` (read) and ``vecs`` (written) may
// alias: the CTA reads its whole matrix before writing.
template <int TMAX>
__device__ __forceinline__ void eigh_cta_body(const float* gram, float* vecs, float* __restrict__ lam_out,
                                              int32_t* __restrict__ ranks, float* __restrict__ wgt,
                                              float* __restrict__ sig2, int n, int nvox, long long patch0,
                                              int* __restrict__ refine_count, int* __restrict__ refine_ids,
                                              long long b) {
  constexpr int NW = TMAX / 32, NG = TMAX / 4, R = TMAX / 32;
  extern __shared__ __align__(16) float sc_[];
  float* HV = sc_;
  float* d = HV + eigh_cta_hv_at<TMAX>(4);
  float* e = d + TMAX;
  float* tau = e + TMAX;
  float* lam = tau + TMAX;
  float* xb = lam + TMAX;
  float* vb = xb + TMAX;
  float* pb = vb + TMAX;
  float* W = pb + TMAX;
  float* scal = W + 2 * TMAX * kInvGroup;  // alpha; the rank
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* G = gram + b * (long long)n * n;
  const bool rv = tid < n;
  LRD_STAMP(0);

  // ---- own row, exact power-of-two scaling ------------------------------------
  float2 a[TMAX / 2];
  {
    const float* row = G + (long long)tid * n;
    const bool vec = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(gram) & 15) == 0;
#pragma unroll
    for (int J = 0; J < NG; ++J) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (vec) {
        if (rv && 4 * J < n) v = reinterpret_cast<const float4*>(row)[J];
      } else if (rv) {
        if (4 * J + 0 < n) v.x = row[4 * J + 0];
        if (4 * J + 1 < n) v.y = row[4 * J + 1];
        if (4 * J + 2 < n) v.z = row[4 * J + 2];
        if (4 * J + 3 < n) v.w = row[4 * J + 3];
      }
      a[2 * J] = make_float2(v.x, v.y);
      a[2 * J + 1] = make_float2(v.z, v.w);
    }
  }
  float dmax = 0.f;  // every warp over the whole diagonal
  for (int i = lane; i < n; i += 32) dmax = fmaxf(dmax, fabsf(G[(long long)i * n + i]));
  dmax = warp_max(dmax);
  int ex = 0;
  if (dmax > 0.f && isfinite(dmax)) frexpf(dmax, &ex);
  const float scale = ldexpf(1.f, -ex), unscale = ldexpf(1.f, ex);
#pragma unroll
  for (int j = 0; j < TMAX / 2; ++j) {
    a[j].x *= scale;
    a[j].y *= scale;
  }
  LRD_STAMP(1);

  // ---- Householder tridiagonalisation -------------------------------------------
  auto column = [&](int k) {  // a[k] of the own row
    float x = 0.f;
#define LRD_CCOL(J)                                                 \
  case J:                                                           \
    if constexpr (J < NG) {                                         \
      const float2 pr = (k & 2) ? a[2 * J + 1] : a[2 * J];          \
      x = (k & 1) ? pr.y : pr.x;                                    \
    }                                                               \
    break;
    switch (k >> 2) {
      LRD_CCOL(0) LRD_CCOL(1) LRD_CCOL(2) LRD_CCOL(3) LRD_CCOL(4) LRD_CCOL(5) LRD_CCOL(6) LRD_CCOL(7)
      LRD_CCOL(8) LRD_CCOL(9) LRD_CCOL(10) LRD_CCOL(11) LRD_CCOL(12) LRD_CCOL(13) LRD_CCOL(14) LRD_CCOL(15)
      LRD_CCOL(16) LRD_CCOL(17) LRD_CCOL(18) LRD_CCOL(19) LRD_CCOL(20) LRD_CCOL(21) LRD_CCOL(22) LRD_CCOL(23)
      LRD_CCOL(24) LRD_CCOL(25) LRD_CCOL(26) LRD_CCOL(27) LRD_CCOL(28) LRD_CCOL(29) LRD_CCOL(30) LRD_CCOL(31)
      default: break;
    }
#undef LRD_CCOL
    return x;
  };
  float x = a[0].x;  // column k of the own row
  auto quarter = [&](auto qtag) {
    constexpr int Q = decltype(qtag)::value, J0 = Q * NG / 4;
    float* hv = HV + eigh_cta_hv_at<TMAX>(Q) - 4 * J0;  // hv[c] = column c of the step's reflector
#pragma unroll 1
    for (int k = 4 * J0; k < min(n - 2, 4 * J0 + TMAX / 4); ++k, hv += TMAX - 4 * J0) {
      xb[tid] = tid >= k + 2 ? x : 0.f;
      if (tid == k + 1) scal[0] = x;
      if (tid == k) d[k] = x;
      __syncthreads();
      float part = 0.f;
#pragma unroll
      for (int i = 0; i < R; ++i) part = fmaf(xb[lane + 32 * i], xb[lane + 32 * i], part);
      const float xnorm2 = warp_sum(part);
      // sum over the unscaled column, while the reflector's scalars are formed
      const float4* xb4 = reinterpret_cast<const float4*>(xb);
      float2 s01 = make_float2(0.f, 0.f), s23 = make_float2(0.f, 0.f);
#pragma unroll
      for (int J = J0; J < NG; ++J) {
        const float4 x4 = xb4[J];
        fma2(s01, a[2 * J], make_float2(x4.x, x4.y));
        fma2(s23, a[2 * J + 1], make_float2(x4.z, x4.w));
      }
      const float c1 = column(k + 1);
      const float alpha = scal[0];
      float taui = 0.f, beta = alpha, sc = 0.f, one = 0.f;
      {
        const float nrm2 = fmaf(alpha, alpha, xnorm2);
        float rs = rsqrtf(nrm2);
        rs = fmaf(0.5f * rs, fmaf(-nrm2 * rs, rs, 1.f), rs);
        const float nrm = nrm2 * rs, den = fabsf(alpha) + nrm;
        float rd = __fdividef(1.f, den);
        rd = fmaf(rd, fmaf(-den, rd, 1.f), rd);
        if (xnorm2 > 0.f) {
          beta = -copysignf(nrm, alpha);
          taui = fmaf(fabsf(alpha), rs, 1.f);
          sc = copysignf(rd, alpha);
          one = 1.f;
        }
      }
      if (tid == 0) {
        e[k] = beta;
        tau[k] = taui;
      }
      const float v = tid == k + 1 ? one : (tid >= k + 2 ? x * sc : 0.f);
      const float p = tid >= k + 1 ? taui * fmaf(sc, (s01.x + s01.y) + (s23.x + s23.y), one * c1) : 0.f;
      vb[tid] = v;
      pb[tid] = p;
      if (tid >= 4 * J0) hv[tid] = v;
      __syncthreads();
      float part2 = 0.f;
#pragma unroll
      for (int i = 0; i < R; ++i) part2 = fmaf(pb[lane + 32 * i], vb[lane + 32 * i], part2);
      const float c = fmaf(-taui * warp_sum(part2), v, p);  // p + 2 kc v
      const float2 mv = make_float2(-v, -v), mc = make_float2(-c, -c);
      const float4* vb4 = reinterpret_cast<const float4*>(vb);
      const float4* pb4 = reinterpret_cast<const float4*>(pb);
#pragma unroll
      for (int J = J0; J < NG; ++J) {
        const float4 v4 = vb4[J];
        const float4 p4 = pb4[J];
        fma2(a[2 * J], mv, make_float2(p4.x, p4.y));
        fma2(a[2 * J + 1], mv, make_float2(p4.z, p4.w));
        fma2(a[2 * J], mc, make_float2(v4.x, v4.y));
        fma2(a[2 * J + 1], mc, make_float2(v4.z, v4.w));
      }
      x = fmaf(-c, vb[k + 1], fmaf(-v, pb[k + 1], c1));  // the same update of column k + 1
      // (xb and alpha are rewritten before, vb and pb after the next barrier)
    }
  };
  quarter(IntTag<0>{});
  quarter(IntTag<1>{});
  quarter(IntTag<2>{});
  quarter(IntTag<3>{});
  {
    const float y = column(n - 1);
    if (tid == n - 2) d[n - 2] = x;
    if (tid == n - 1) {
      e[n - 2] = x;
      d[n - 1] = y;
      e[n - 1] = 0.f;
    }
  }
  __syncthreads();
  LRD_STAMP(2);

  // ---- eigenvalues: thread j = eigenvalue j (see bisect_reg) ---------------------
  const float eps = Num<float>::eps();
  float glo = FLT_MAX, ghi = -FLT_MAX;
  for (int i = lane; i < n; i += 32) {
    const float r = (i > 0 ? fabsf(e[i - 1]) : 0.f) + (i < n - 1 ? fabsf(e[i]) : 0.f);
    glo = fminf(glo, d[i] - r);
    ghi = fmaxf(ghi, d[i] + r);
  }
  glo = warp_min(glo);
  ghi = warp_max(ghi);
  const float tnorm = fmaxf(fmaxf(fabsf(glo), fabsf(ghi)), FLT_MIN);
  {
    glo -= 4.f * eps * tnorm * n;
    ghi += 4.f * eps * tnorm * n;
    int et = 0;
    if (isfinite(tnorm)) frexpf(tnorm, &et);
    const float ts = ldexpf(1.f, -et), tu = ldexpf(1.f, et);
    const float abstol = eps * tnorm * ts;
    float4* co = reinterpret_cast<float4*>(W);
    float2* px = reinterpret_cast<float2*>(W + 4 * TMAX);  // two points per eigenvalue, their counts
    int2* cnt = reinterpret_cast<int2*>(W + 6 * TMAX);
    const int n16 = (n + 15) & ~15;
    if (tid < n16) {
      const float di = rv ? d[tid] * ts : 2.f;
      const float ei = (tid > 0 && rv) ? e[tid - 1] * ts : 0.f;
      const float e2 = (tid > 0 && rv) ? fmaxf(ei * ei, 0x1p-60f) : 0.f;
      co[tid] = make_float4(di, di, -e2, -e2);
    }
    float lo = glo * ts, hi = ghi * ts;
    int clo = 0, chi = n;  // the eigenvalues in (lo, hi]
    for (int it = 0; it < 200; ++it) {
      const float tol = fmaxf(abstol, 2.f * eps * fmaxf(fabsf(lo), fabsf(hi)));
      const float mid = 0.5f * (lo + hi);
      const bool run = rv && hi - lo > tol && mid > lo && mid < hi;
      if (!__syncthreads_or(run)) break;  // (also: co is written, the last round's points are read)
      const int m = chi - clo;
      const float w = __fdividef(hi - lo, (float)(2 * m + 1));
      const float r = (float)(2 * (tid - clo) + 1);
      const float xs[2] = {fmaf(r, w, lo), fmaf(r + 1.f, w, lo)};
      int c[2];
      sturm_counts<2>(co, n16, xs, c);
      const bool several = __syncthreads_or(rv && m > 1);
      if (several) {
        px[tid] = make_float2(xs[0], xs[1]);
        cnt[tid] = make_int2(c[0], c[1]);
        __syncthreads();
      }
      if (rv && m > 1) {
        // first point of the interval with more than j eigenvalues below it
        const float* ps = reinterpret_cast<const float*>(px);
        const int* cs = reinterpret_cast<const int*>(cnt);
        const int p0 = 2 * clo, p1 = 2 * chi;
        int s = p0, t = p1;
        while (s < t) {
          const int h = (s + t) >> 1;
          if (cs[h] > tid) t = h; else s = h + 1;
        }
        if (s > p0) {
          lo = ps[s - 1];
          clo = max(clo, cs[s - 1]);
        }
        if (s < p1) {
          hi = ps[s];
          chi = min(chi, cs[s]);
        }
      } else if (c[0] > tid) {
        hi = xs[0];
      } else if (c[1] > tid) {
        lo = xs[0];
        hi = xs[1];
      } else {
        lo = xs[1];
      }
    }
    if (rv) lam[tid] = 0.5f * (lo + hi) * tu;
  }
  __syncthreads();
  LRD_STAMP(3);

  // ---- MP rank (first warp) -------------------------------------------------------
  int* pshare = reinterpret_cast<int*>(scal + 1);
  bool queue = false;  // (first warp; as in eigh_reg_body)
  if (warp == 0) {
    int p;
    queue = mp_rank_sub<32>(lam, unscale, n, nvox, W, p, sig2 ? sig2 + b : nullptr) < kRefineTol;
    if (lane == 0) {
      ranks[b] = p;
      wgt[b] = (float)(1.0 / (2.0 + (double)p));
      *pshare = p;
    }
  }
  if (lam_out != nullptr && rv) lam_out[b * n + tid] = lam[tid] * unscale;
  __syncthreads();
  const int p = *pshare;
  LRD_STAMP(4);

  // ---- top-p eigenvectors, in chunks of kInvGroup ---------------------------------
  float* V = vecs + b * (long long)n * n;
  float* Z = W;
  float* U = W + TMAX * kInvGroup;
#pragma unroll 1
  for (int j0 = 0; j0 < p; j0 += kInvGroup) {
    const int g = min(kInvGroup, p - j0);
    if (warp == 0) twisted_vectors<32>(d, e, lam, Z, U, n, j0, g, tnorm);
    __syncthreads();
    LRD_STAMP(5);
    // back-transform x = H(0) ... H(n-3) z: warp w's vectors w, w + NW, ..., row
    // lane + 32 ri in a lane
    constexpr int GW = (kInvGroup + NW - 1) / NW;
    float y[R][GW];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int r = lane + 32 * ri;
#pragma unroll
      for (int u = 0; u < GW; ++u) y[ri][u] = (r < n && warp + NW * u < g) ? Z[r * kInvGroup + warp + NW * u] : 0.f;
    }
    if (warp < g) {
      float h[R], hn[R];
      auto reflector = [&](int k, float (&out)[R]) {
        const int qk = k / (TMAX / 4), c0 = qk * (TMAX / 4);  // its quarter and first stored column
        const float* hrow = HV + eigh_cta_hv_at<TMAX>(qk) + (k - c0) * (TMAX - c0) - c0;
#pragma unroll
        for (int ri = 0; ri < R; ++ri) out[ri] = lane + 32 * ri >= c0 ? hrow[lane + 32 * ri] : 0.f;
      };
      if (n > 2) reflector(n - 3, hn);
#pragma unroll 1
      for (int k = n - 3; k >= 0; --k) {
#pragma unroll
        for (int ri = 0; ri < R; ++ri) h[ri] = hn[ri];
        reflector(max(k - 1, 0), hn);  // in flight during this one's sums
        const float tk = tau[k];
        float dq[GW];
#pragma unroll
        for (int u = 0; u < GW; ++u) {
          dq[u] = 0.f;
#pragma unroll
          for (int ri = 0; ri < R; ++ri) dq[u] = fmaf(h[ri], y[ri][u], dq[u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int u = 0; u < GW; ++u)
            dq[u] += __shfl_xor_sync(0xffffffffu, dq[u], o);
#pragma unroll
        for (int u = 0; u < GW; ++u) {
          const float f = -tk * dq[u];
#pragma unroll
          for (int ri = 0; ri < R; ++ri) y[ri][u] = fmaf(f, h[ri], y[ri][u]);
        }
      }
#pragma unroll
      for (int ri = 0; ri < R; ++ri) {
        const int r = lane + 32 * ri;
#pragma unroll
        for (int u = 0; u < GW; ++u)
          if (r < n && warp + NW * u < g) Z[r * kInvGroup + warp + NW * u] = y[ri][u];
      }
    }
    __syncthreads();
    LRD_STAMP(6);
    if (warp == 0) {
      float2 z[R][kInvGroup / 2];
#pragma unroll
      for (int ri = 0; ri < R; ++ri) {
        const int r = lane + 32 * ri;
#pragma unroll
        for (int q = 0; q < kInvGroup; q += 2) {
          const float2 zz = *reinterpret_cast<const float2*>(Z + r * kInvGroup + q);
          z[ri][q / 2] = make_float2(r < n && q < g ? zz.x : 0.f, r < n && q + 1 < g ? zz.y : 0.f);
        }
      }
      queue |= gram_schmidt<32, R>(z, V, lam, tnorm, n, j0, g, g, true);
    }
    __syncthreads();
  }
  if (tid == 0 && refine_count != nullptr && queue) refine_ids[atomicAdd(refine_count, 1)] = (int)(patch0 + b);
  LRD_STAMP(7);
}

// CTAs per SM by the registers a row needs.
template <int TMAX>
__host__ __device__ constexpr int eigh_cta_min_blocks() {
  return TMAX <= 64 ? 8 : (TMAX <= 96 ? 5 : 3);
}

template <int TMAX>
__global__ void __launch_bounds__(TMAX, eigh_cta_min_blocks<TMAX>())
    eigh_cta_kernel(const float* gram, float* vecs, float* __restrict__ lam_out, int32_t* __restrict__ ranks,
                    float* __restrict__ wgt, float* __restrict__ sig2, int n, int nvox, long long patch0,
                    int* __restrict__ refine_count, int* __restrict__ refine_ids) {
  eigh_cta_body<TMAX>(gram, vecs, lam_out, ranks, wgt, sig2, n, nvox, patch0, refine_count, refine_ids,
                      (long long)blockIdx.x);
}

}  // namespace lrd
