// Register-resident float32 eigensolver for T <= TMAX (TMAX in {32, 48, 64}).
//
// Householder tridiagonalisation, eigenvalues by Sturm counts, MP rank, the top-p
// eigenvectors of the tridiagonal by twisted factorisations, back-transform,
// Gram-Schmidt. L lanes hold one matrix in registers, rows l, l + L, ... of lane
// l (every column index compile-time): L = 8 for TMAX = 32, so a warp solves four
// matrices side by side, L = 16 for 48 (two), L = 32 for 64.
//
// A reduction step is a chain of a dozen dependent stages (norm, reflector,
// matrix-vector product, dot product, update), and only a quarter of its
// instructions are the products: with one matrix per warp the instruction issue
// was 60% busy at 16 warps per SM and the FMA pipe 23%. Two matrices per warp share
// every instruction of that chain, 48 rows fill 16 lanes x 3 without padding, and
// the packed FMA halves the products' issue slots.
//
//  * Step k: every lane picks column k of its own rows (a switch on k / 4: the
//    register indices stay compile-time); the reflector goes to shared memory (HV,
//    row k stored from its first live 4-column group on) and is read back as
//    float4 for p = tau A v. With kc = -tau/2 p.v the update is A -= v p^T + (p + 2
//    kc v) v^T, so p goes to shared memory before p.v is summed. Dead column groups
//    are skipped by a switch that enters the unrolled groups at the first live one.
//  * Eigenvalues: Sturm counts by the division-free recurrence p_i = (d_i - x)
//    p_{i-1} - e_{i-1}^2 p_{i-2} (an eigenvalue below x per sign change), rescaled
//    every four steps, C chains per lane. Chains whose eigenvalues still share an
//    interval evaluate different points of it: 44 noise eigenvalues in one interval
//    cut it into 45 a round, and bisection only starts where they part.
//  * Vectors: for the shift lambda one lane factors T - lambda from the top, another
//    from the bottom; the row r where the two meet with the smallest |gamma_r| starts
//    the vector (z_r = 1, one multiplication per entry to either side). gamma_r /
//    |z|^2 is the Rayleigh correction of lambda; a second pass with it gives the
//    vector.
//
// Measured on B200 (kernel time, against one matrix per warp with bisection by the
// quotient recurrence and inverse iteration by partial-pivoting LU): 12600 matrices
// at T = 48 0.885 -> 0.52 ms, 372416 at T = 32 11.5 -> 5.2 (16 lanes per matrix 5.5),
// 37392 at T = 64 4.55 -> 2.9 (phase 3.07, with the reflector read ahead 2.89), one
// matrix 105 -> 85 us (eigh_reg_wide_kernel). Cycles per warp at T = 48, 12 warps per SM (two matrices):
// load 9 K, reduction 128 K, eigenvalues 67 K, rank 5 K, vectors 18 K, back-transform
// 15 K, Gram-Schmidt 4 K (one matrix per warp at 16 warps: 12 / 147 / 93 / 6 / 29 / 22 /
// 4 K). Instruction issue 46%, three warps per scheduler: latency bounds it, the
// 168 registers of 12 warps and the shared memory bound the warps. Measured slower:
// the reduction as four straight-line loops without the dead column groups of each
// quarter (T = 48 alone 107 -> 71 K cycles, but 11 warps: 0.74 -> 0.77 ms; T = 64 3.10 ->
// 3.39), the update as two rank-1 passes with the reflector read two groups ahead
// (T = 48 0.75, T = 32 no change), points shared out among the intervals (12 rounds instead of 20, twice the
// instructions around them: 0.80), two points per eigenvalue (0.83).
//
// The near-tie test (mp_rank's margin) and vectors that coincide queue patches for the
// float64 pass.
#pragma once

#include "eigh.cuh"

namespace lrd {

#ifdef LRD_PHASE_CLOCKS
__device__ long long* g_phase_clocks;  // 8 stamps per block, set by a probe build
#define LRD_STAMP(i) \
  do { __syncwarp(); if ((threadIdx.x & 31) == 0) g_phase_clocks[(long long)blockIdx.x * 8 + (i)] = clock64(); } while (0)
#else
#define LRD_STAMP(i) \
  do { } while (0)
#endif

// Lanes per matrix and matrices per warp (= per block).
template <int TMAX>
__host__ __device__ constexpr int eigh_reg_lanes() {
  return TMAX <= 32 ? 8 : (TMAX <= 48 ? 16 : 32);
}
template <int TMAX>
__host__ __device__ constexpr int eigh_reg_mats() {
  return 32 / eigh_reg_lanes<TMAX>();
}
// Eigenvectors formed at once: two lanes each.
template <int TMAX>
__host__ __device__ constexpr int eigh_reg_group() {
  return eigh_reg_lanes<TMAX>() >= 2 * kInvGroup ? kInvGroup : eigh_reg_lanes<TMAX>() / 2;
}

// Shared-memory floats per matrix: packed HV, d, e, tau, lam, p (5 TMAX), the work
// area W (the vectors' factors, 2 TMAX kInvGroup; before them the Sturm
// sequence's coefficients and the points and counts of a round, or the MP
// scratch); an odd multiple of 16, so two matrices' equal offsets lie in
// different banks.
template <int TMAX>
__host__ __device__ constexpr size_t eigh_reg_mat_floats() {
  const size_t f = eigh_hv_floats<TMAX>() + 5 * TMAX + (size_t)2 * TMAX * eigh_reg_group<TMAX>();
  return ((f + 31) & ~size_t(31)) + (eigh_reg_mats<TMAX>() == 4 ? 8 : 16);
}
template <int TMAX>
__host__ __device__ constexpr size_t eigh_reg_smem_floats() {
  return eigh_reg_mats<TMAX>() * eigh_reg_mat_floats<TMAX>();
}

// Sum, minimum and maximum over the L lanes of a matrix.
template <int L>
__device__ __forceinline__ float sub_sum(float v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int L, typename Real>
__device__ __forceinline__ Real sub_max(Real v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int L, typename Real>
__device__ __forceinline__ Real sub_min(Real v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sums of 2 G values (G pairs) over the L lanes of a matrix, every lane getting
// all of them: halving exchanges until a lane holds one value, the remaining xor
// steps, then a broadcast per value (16 shuffles for 8 values over 16 lanes; 32
// for a butterfly each).
template <int L, int G>
__device__ __forceinline__ void sub_allsum(float2 (&v)[G]) {
  static_assert(G == 2 || G == 4, "4 or 8 values");
  constexpr int N = 2 * G;
  const int lane = threadIdx.x & 31;
  float f[N];
#pragma unroll
  for (int i = 0; i < G; ++i) {
    f[2 * i] = v[i].x;
    f[2 * i + 1] = v[i].y;
  }
  int o = L / 2;
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float keep = up ? f[i + half] : f[i], send = up ? f[i] : f[i + half];
      f[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) f[0] += __shfl_xor_sync(0xffffffffu, f[0], o);
  // value q sits in the lanes whose top log2(N) bits (of log2(L)) spell q
#pragma unroll
  for (int i = 0; i < G; ++i) {
    v[i].x = __shfl_sync(0xffffffffu, f[0], (2 * i) * (L / N), L);
    v[i].y = __shfl_sync(0xffffffffu, f[0], (2 * i + 1) * (L / N), L);
  }
}

// Sturm counts: c[j] = sign changes of the sequence at x[j] = eigenvalues below
// x[j]. co[i] = (d_i, d_i, -e_{i-1}^2, -e_{i-1}^2) of a tridiagonal scaled to a norm
// below 1, e^2 >= 2^-60 (four steps shrink the sequence by 2^-120 at most before
// it is rescaled); entries past the matrix are d = 2, e = 0, which changes no sign.
// n16 = rows rounded up to 16. Chains go in pairs through the packed FMA, an odd
// one alone.
template <int C>
__device__ __forceinline__ void sturm_counts(const float4* __restrict__ co, int n16, const float (&x)[C], int (&c)[C]) {
  constexpr int C2 = C / 2, C1 = C & 1;
  float2 p1[C2], p2[C2], xs[C2];
  float r1 = 1.f, r2 = 0.f;
  unsigned last[C];
#pragma unroll
  for (int j = 0; j < C2; ++j) {
    p1[j] = make_float2(1.f, 1.f);
    p2[j] = make_float2(0.f, 0.f);
    xs[j] = make_float2(-x[2 * j], -x[2 * j + 1]);
  }
#pragma unroll
  for (int j = 0; j < C; ++j) last[j] = c[j] = 0;
#pragma unroll 1
  for (int i0 = 0; i0 < n16; i0 += 16) {
    unsigned m[C];
#pragma unroll
    for (int j = 0; j < C; ++j) m[j] = last[j];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const float4 k = co[i0 + u];
#pragma unroll
      for (int j = 0; j < C2; ++j) {
        const float2 t = add2(make_float2(k.x, k.y), xs[j]);
        float2 w = mul2(make_float2(k.z, k.w), p2[j]);
        fma2(w, t, p1[j]);
        p2[j] = p1[j];
        p1[j] = w;
        m[2 * j] = __funnelshift_l(__float_as_uint(w.x), m[2 * j], 1);
        m[2 * j + 1] = __funnelshift_l(__float_as_uint(w.y), m[2 * j + 1], 1);
      }
      if (C1) {
        const float w = fmaf(k.x - x[C - 1], r1, k.z * r2);
        r2 = r1;
        r1 = w;
        m[C - 1] = __funnelshift_l(__float_as_uint(w), m[C - 1], 1);
      }
      if ((u & 3) == 3) {
        // rescale by a power of two to about 1: the complement of the (even part of
        // the) exponent is the scale's exponent
#pragma unroll
        for (int j = 0; j < C2; ++j) {
          const unsigned ex = ~__float_as_uint(fabsf(p1[j].x) + fabsf(p2[j].x)) & 0x7f000000u;
          const unsigned ey = ~__float_as_uint(fabsf(p1[j].y) + fabsf(p2[j].y)) & 0x7f000000u;
          const float2 sc = make_float2(__uint_as_float(ex), __uint_as_float(ey));
          p1[j] = mul2(p1[j], sc);
          p2[j] = mul2(p2[j], sc);
        }
        if (C1) {
          const float sc = __uint_as_float(~__float_as_uint(fabsf(r1) + fabsf(r2)) & 0x7f000000u);
          r1 *= sc;
          r2 *= sc;
        }
      }
    }
    // bits 15..0: this block's signs in order, bit 16: the sign before it
#pragma unroll
    for (int j = 0; j < C; ++j) {
      c[j] += __popc((m[j] ^ (m[j] >> 1)) & 0xffffu);
      last[j] = m[j] & 1u;
    }
  }
}

// All eigenvalues of the tridiagonal (d, e in shared memory) ascending into lam;
// tnorm = Gerschgorin bound. An interval [lo, hi] with count(lo) <= j < count(hi)
// per eigenvalue j = l + L c, cut until max(eps tnorm, 2 eps |lambda|): the absolute
// part is LAPACK's default tolerance (eps times the norm of the tridiagonal),
// below the float32 reduction's own error in the eigenvalues. In a round the m
// eigenvalues that share an interval evaluate m evenly spaced points of it. W:
// 6 TMAX floats.
template <int TMAX>
__device__ __forceinline__ void bisect_reg(const float* d, const float* e, float* lam, float* W, int n,
                                           float& tnorm_out) {
  constexpr int L = eigh_reg_lanes<TMAX>(), C = (TMAX + L - 1) / L;
  const int lane = threadIdx.x & 31, l = lane & (L - 1), sh = lane & ~(L - 1);
  const float eps = Num<float>::eps();
  float glo = FLT_MAX, ghi = -FLT_MAX;
  for (int i = l; i < n; i += L) {
    const float r = (i > 0 ? fabsf(e[i - 1]) : 0.f) + (i < n - 1 ? fabsf(e[i]) : 0.f);
    glo = fminf(glo, d[i] - r);
    ghi = fmaxf(ghi, d[i] + r);
  }
  glo = sub_min<L>(glo);
  ghi = sub_max<L>(ghi);
  const float tnorm = fmaxf(fmaxf(fabsf(glo), fabsf(ghi)), FLT_MIN);
  tnorm_out = tnorm;
  glo -= 4.f * eps * tnorm * n;
  ghi += 4.f * eps * tnorm * n;
  // scaled by a power of two to a norm in [0.5, 1); an off-diagonal below 2^-30
  // of it is raised to that (an eigenvalue moves by 1/32 of the tolerance)
  int ex = 0;
  if (isfinite(tnorm)) frexpf(tnorm, &ex);
  const float ts = ldexpf(1.f, -ex), tu = ldexpf(1.f, ex);
  glo *= ts;
  ghi *= ts;
  const float abstol = eps * tnorm * ts;
  float4* co = reinterpret_cast<float4*>(W);
  float* px = W + 4 * TMAX;
  int* cnt = reinterpret_cast<int*>(W + 5 * TMAX);
  const int n16 = (n + 15) & ~15;
  for (int i = l; i < n16; i += L) {
    const float di = i < n ? d[i] * ts : 2.f;
    const float ei = (i > 0 && i < n) ? e[i - 1] * ts : 0.f;
    const float e2 = (i > 0 && i < n) ? fmaxf(ei * ei, 0x1p-60f) : 0.f;
    co[i] = make_float4(di, di, -e2, -e2);
  }
  __syncwarp();
  // [clo, chi): the eigenvalues between the ends, j among them; they all have this
  // interval
  float lo[C], hi[C], x[C];
  int clo[C], chi[C], c[C];
#pragma unroll
  for (int k = 0; k < C; ++k) {
    lo[k] = glo;
    hi[k] = ghi;
    clo[k] = 0;
    chi[k] = n;
  }
  // The matrices of a warp go through the rounds together; what happens to one
  // depends on itself alone (one that is done keeps its intervals).
  constexpr unsigned field = L == 32 ? 0xffffffffu : (1u << (L & 31)) - 1u;
  for (int it = 0; it < 200; ++it) {
    bool run = false, several = false;
#pragma unroll
    for (int k = 0; k < C; ++k) {
      const int j = l + L * k;
      const float tol = fmaxf(abstol, 2.f * eps * fmaxf(fabsf(lo[k]), fabsf(hi[k])));
      const float mid = 0.5f * (lo[k] + hi[k]);
      run |= j < n && hi[k] - lo[k] > tol && mid > lo[k] && mid < hi[k];
      several |= j < n && chi[k] - clo[k] > 1;
      x[k] = mid;
    }
    const unsigned running = __ballot_sync(0xffffffffu, run);
    if (running == 0) break;
    const bool on = (running >> (sh & 31)) & field;
    const bool any_several = __any_sync(0xffffffffu, several && on);
    if (any_several) {
#pragma unroll
      for (int k = 0; k < C; ++k) {
        const int m = chi[k] - clo[k];
        if (m > 1)
          x[k] = fmaf(hi[k] - lo[k], __fdividef((float)(l + L * k - clo[k] + 1), (float)(m + 1)), lo[k]);
      }
    }
    sturm_counts<C>(co, n16, x, c);
    if (any_several) {
#pragma unroll
      for (int k = 0; k < C; ++k) {
        px[l + L * k] = x[k];
        cnt[l + L * k] = c[k];
      }
      __syncwarp();
    }
    if (on) {
#pragma unroll
      for (int k = 0; k < C; ++k) {
        const int j = l + L * k;
        if (chi[k] - clo[k] > 1 && j < n) {
          // first point of the interval with more than j eigenvalues below it
          const int p0 = clo[k], p1 = chi[k];
          int a = p0, b = p1;
          while (a < b) {
            const int mid = (a + b) >> 1;
            if (cnt[mid] > j) b = mid; else a = mid + 1;
          }
          if (a > p0) {
            lo[k] = px[a - 1];
            clo[k] = max(clo[k], cnt[a - 1]);
          }
          if (a < p1) {
            hi[k] = px[a];
            chi[k] = min(chi[k], cnt[a]);
          }
        } else if (c[k] > j) {
          hi[k] = x[k];
        } else {
          lo[k] = x[k];
        }
      }
    }
    if (any_several) __syncwarp();  // the next round's points go to the same place
  }
#pragma unroll
  for (int k = 0; k < C; ++k)
    if (l + L * k < n) lam[l + L * k] = 0.5f * (lo[k] + hi[k]) * tu;
  __syncwarp();
}

// mp_rank (eigh.cuh) in float32 for the L lanes of a matrix; W: 2 n floats.
template <int L>
__device__ __forceinline__ double mp_rank_sub(const float* lam, float unscale, int n, int nvox, float* W, int& p_out,
                                              float* sig2_out) {
  const int lane = threadIdx.x & 31, l = lane & (L - 1), sh = lane & ~(L - 1);
  const int t = n - 1;
  float* eg = W;      // descending eigs, t entries
  float* rc = W + n;  // float32 suffix sums
  for (int i = l; i < t; i += L) eg[i] = __fdiv_rn(fmaxf(lam[n - 1 - i] * unscale, 0.f), (float)nvox);
  __syncwarp();
  if (l == 0) {
    float acc = 0.f;  // (0 + the first term is that term)
    int i = t - 1;
    for (; i >= 7; i -= 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = eg[i - u];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        acc = __fadd_rn(acc, v[u]);
        rc[i - u] = acc;
      }
    }
    for (; i >= 0; --i) {
      acc = __fadd_rn(acc, eg[i]);
      rc[i] = acc;
    }
  }
  __syncwarp();
  int p = 0;
  double margin = DBL_MAX;
  const double sq = sqrt((double)((long long)t * (long long)nvox));
  const float elast = eg[t - 1];
  for (int i0 = 0; i0 < t; i0 += L) {
    const int i = i0 + l;
    bool sig = false;
    if (i < t) {
      const double lhs = (double)__fsub_rn(eg[i], elast) * (double)(t - i) * (double)(nvox - i);
      const double rhs = (double)__fmul_rn(4.f, rc[i]) * sq;
      sig = lhs > rhs;
      if (rhs > 0.0) margin = fmin(margin, fabs(lhs - rhs) / rhs);
    }
    const unsigned b = __ballot_sync(0xffffffffu, sig);
    p += __popc(L == 32 ? b : (b >> sh) & ((1u << (L & 31)) - 1u));
  }
  margin = sub_min<L>(margin);
  p_out = p;
  if (sig2_out != nullptr && l == 0) *sig2_out = (p < t) ? __fdiv_rn(rc[p], (float)(t - p)) : 0.f;
  return margin;
}

// Eigenvectors of the tridiagonal for the eigenvalues lam[n - 1 - j0 - q], q < g <=
// IG, unnormalised, entry i at Z[i * IG + q], by the L lanes of a
// matrix, two per vector. Z and U: n x IG each.
template <int L, int IG = kInvGroup>
__device__ __forceinline__ void twisted_vectors(const float* d, const float* e, const float* lam, float* Z, float* U,
                                                int n, int j0, int g, float tnorm) {
  const int l = threadIdx.x & (L - 1);
  const int q = l & (IG - 1), down = (l / IG) & 1;  // down 0: from the top, 1: from the bottom
  const bool on = l < 2 * IG && q < g;
  const float pivtol = Num<float>::eps() * tnorm;
  float sig = on ? lam[n - 1 - j0 - q] : 0.f;
  float* F = (down ? U : Z) + q;  // e_i / pivot of this direction
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    __syncwarp();
    if (on) {
      float D = d[down ? n - 1 : 0] - sig;
#pragma unroll 4
      for (int s = 0; s < n - 1; ++s) {
        const int i = down ? n - 2 - s : s;
        const float ei = e[i], dn = d[down ? i : i + 1] - sig;
        if (fabsf(D) < pivtol) D = D < 0.f ? -pivtol : pivtol;
        const float r = __fdividef(ei, D);
        F[i * IG] = r;
        D = fmaf(-ei, r, dn);
      }
    }
    __syncwarp();
    // gamma_r = (d_r - lambda) - e_{r-1} Z_{r-1} - e_r U_r: every other row each
    float best = FLT_MAX, gam = 0.f;
    int at = 0;
    if (on) {
#pragma unroll 4
      for (int r = down; r < n; r += 2) {
        float gr = d[r] - sig;
        if (r > 0) gr = fmaf(-e[r - 1], Z[(r - 1) * IG + q], gr);
        if (r < n - 1) gr = fmaf(-e[r], U[r * IG + q], gr);
        if (fabsf(gr) < best) {
          best = fabsf(gr);
          gam = gr;
          at = r;
        }
      }
    }
    {
      const float ob = __shfl_xor_sync(0xffffffffu, best, IG), og = __shfl_xor_sync(0xffffffffu, gam, IG);
      const int oa = __shfl_xor_sync(0xffffffffu, at, IG);
      if (ob < best || (ob == best && oa < at)) {
        best = ob;
        gam = og;
        at = oa;
      }
    }
    float z = 1.f, s2 = 0.f;
    if (on) {
      if (down == 0) {
        if (pass == 1) Z[at * IG + q] = 1.f;  // (the bottom lane writes below this row)
#pragma unroll 4
        for (int i = at - 1; i >= 0; --i) {
          z = -Z[i * IG + q] * z;
          s2 = fmaf(z, z, s2);
          if (pass == 1) Z[i * IG + q] = z;
        }
      } else {
#pragma unroll 4
        for (int i = at; i < n - 1; ++i) {
          z = -U[i * IG + q] * z;
          s2 = fmaf(z, z, s2);
          if (pass == 1) Z[(i + 1) * IG + q] = z;
        }
      }
    }
    if (pass == 0) {
      s2 = 1.f + s2 + __shfl_xor_sync(0xffffffffu, s2, IG);
      // the correction stays within the eigenvalue's own tolerance
      const float cor = __fdividef(gam, s2), lim = 2.f * pivtol;
      sig += fminf(fmaxf(cor, -lim), lim);
    }
  }
  __syncwarp();
}

// Modified Gram-Schmidt in descending eigenvalue order of the chunk's g vectors
// (y[ri][q / 2] = vectors q, q + 1, row l + L ri), against each other and the j0
// vectors before them, which are read from the output ``V``; then written there.
// gmax >= g: vectors of the fullest matrix of the warp (one with fewer works on
// zeros).
// Returns whether the float32 vectors could not tell a kept eigenvalue from an earlier
// one: what the projections leave of its vector is below a tenth in length. Two
// eigenvalues that agree to the shifts' errors can start both vectors from the same
// row, and the rest would be round-off. An eigenvalue below kRoundOff of the norm is
// round-off itself, and any orthonormal vector does: of a rank-deficient matrix the
// tail of the tridiagonal is round-off, its vectors are unit vectors that coincide,
// and nothing is left of one after two rounds; it goes on from vectors of signs.
constexpr float kParallel = 1e-2f;
constexpr float kRoundOff = 0x1p-21f;
constexpr int kGsRounds = 10;
template <int L, int R, int IG = kInvGroup>
__device__ __forceinline__ bool gram_schmidt(float2 (&y)[R][IG / 2], float* V, const float* lam, float tnorm, int n,
                                             int j0, int g, int gmax, bool mine) {
  bool lost = false;
  const int l = threadIdx.x & (L - 1);
  auto vq = [&](int ri, int q) -> float& { return (q & 1) ? y[ri][q / 2].y : y[ri][q / 2].x; };
#pragma unroll
  for (int q = 0; q < IG; ++q) {
    if (q >= gmax) continue;
    auto norm2 = [&]() {
      float s_ = 0.f;
#pragma unroll
      for (int ri = 0; ri < R; ++ri) s_ = fmaf(vq(ri, q), vq(ri, q), s_);
      return sub_sum<L>(s_);
    };
    auto project = [&](const float (&w)[R], bool on) {  // takes the part along w out
      float s_ = 0.f;
#pragma unroll
      for (int ri = 0; ri < R; ++ri) s_ = fmaf(w[ri], vq(ri, q), s_);
      const float sum = sub_sum<L>(s_), dot = on ? sum : 0.f;  // (the shuffles by the whole warp)
#pragma unroll
      for (int ri = 0; ri < R; ++ri) vq(ri, q) = fmaf(-dot, w[ri], vq(ri, q));
    };
    float before = norm2();
    bool on = q < g;  // this matrix takes part
#pragma unroll 1
    for (int round = 0; round < kGsRounds; ++round) {
      if (round >= 2) {  // nothing but round-off was left: another start
#pragma unroll
        for (int ri = 0; ri < R; ++ri) {
          const unsigned r = l + L * ri;
          unsigned h = (r + 1u) * 0x9E3779B1u ^ (unsigned)(j0 + q + 128 * round) * 0x85EBCA6Bu;
          h = (h ^ (h >> 15)) * 0xC2B2AE35u;
          const float s_ = (h >> 16) & 1u ? 1.f : -1.f;
          if (on) vq(ri, q) = (int)r < n && q < g ? s_ : 0.f;
        }
        before = on ? (float)n : before;
      }
      for (int i = 0; i < j0; ++i) {  // earlier chunks, from the output
        float w[R];
#pragma unroll
        for (int ri = 0; ri < R; ++ri) w[ri] = (l + L * ri < n && q < g) ? V[(long long)i * n + l + L * ri] : 0.f;
        project(w, on);
      }
#pragma unroll
      for (int i = 0; i < q; ++i) {
        float w[R];
#pragma unroll
        for (int ri = 0; ri < R; ++ri) w[ri] = vq(ri, i);
        project(w, on);
      }
      const float after = norm2();
      const float inv = on ? rsqrtf(fmaxf(after, FLT_MIN)) : 1.f;
#pragma unroll
      for (int ri = 0; ri < R; ++ri) vq(ri, q) *= inv;
      // little left of it (nearly parallel to the earlier ones): once more, from
      // the normalised rest
      if (round == 0 && on && after < kParallel * before) lost |= lam[n - 1 - j0 - q] > kRoundOff * tnorm;
      on &= after < 1e-3f * before;
      before = 1.f;
      if (!__any_sync(0xffffffffu, on)) break;
    }
  }
  if (mine) {
#pragma unroll
    for (int q = 0; q < IG; ++q)
      if (q < g)
#pragma unroll
        for (int ri = 0; ri < R; ++ri) {
          const int r = l + L * ri;
          if (r < n) V[(long long)(j0 + q) * n + r] = vq(ri, q);
        }
  }
  return lost;
}

// Body of one warp's matrices ``b0``, b0 + 1, ... (the launch's patch index, below nmat;
// patch patch0 + b), shared by the single-volume kernels and the packed launch.
// PF: whether the reflector's next column groups are read two groups ahead: a switch's
// labels keep the compiler from moving a load up. Eigensolve phase off / on: 37392
// matrices at T = 64 3.07 / 2.91 ms, 12600 at T = 48 0.731 / 0.745 (out of registers;
// eigh_reg_wide_kernel has them), 372416 at T = 32 5.21 / 5.21.
template <int TMAX, bool PF = (TMAX > 48)>
__device__ __forceinline__ void eigh_reg_body(const float* gram, float* vecs, float* __restrict__ lam_out,
                                              int32_t* __restrict__ ranks, float* __restrict__ wgt,
                                              float* __restrict__ sig2, int n, int nvox, long long patch0,
                                              int* __restrict__ refine_count, int* __restrict__ refine_ids,
                                              long long b0, long long nmat) {
  constexpr int L = eigh_reg_lanes<TMAX>(), R = TMAX / L, NG = TMAX / 4, IG = eigh_reg_group<TMAX>();
  extern __shared__ __align__(16) float sr[];
  const int lane = threadIdx.x & 31, l = lane & (L - 1);
  const bool mine = b0 + lane / L < nmat;  // the last warp's second half may have no matrix of its own
  const long long b = mine ? b0 + lane / L : nmat - 1;
  float* HV = sr + (lane / L) * eigh_reg_mat_floats<TMAX>();
  float* d = HV + eigh_hv_floats<TMAX>();
  float* e = d + TMAX;
  float* tau = e + TMAX;
  float* lam = tau + TMAX;
  float* ps = lam + TMAX;  // tridiagonalisation: p = tau A v
  float* W = ps + TMAX;
  const float* G = gram + b * (long long)n * n;
  LRD_STAMP(0);

  // ---- own rows, exact power-of-two scaling ------------------------------------
  float2 a[R][TMAX / 2];
  const bool vec = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(gram) & 15) == 0;
#pragma unroll
  for (int ri = 0; ri < R; ++ri) {
    const int r = l + L * ri;
    const float* row = G + (long long)r * n;
#pragma unroll
    for (int J = 0; J < NG; ++J) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (vec) {
        if (r < n && 4 * J < n) v = reinterpret_cast<const float4*>(row)[J];
      } else if (r < n) {
        if (4 * J + 0 < n) v.x = row[4 * J + 0];
        if (4 * J + 1 < n) v.y = row[4 * J + 1];
        if (4 * J + 2 < n) v.z = row[4 * J + 2];
        if (4 * J + 3 < n) v.w = row[4 * J + 3];
      }
      a[ri][2 * J] = make_float2(v.x, v.y);
      a[ri][2 * J + 1] = make_float2(v.z, v.w);
    }
  }
  float dmax = 0.f;
#pragma unroll
  for (int ri = 0; ri < R; ++ri) {
    const int r = l + L * ri;
    if (r < n) dmax = fmaxf(dmax, fabsf(G[(long long)r * n + r]));
  }
  dmax = sub_max<L>(dmax);
  int ex = 0;
  if (dmax > 0.f && isfinite(dmax)) frexpf(dmax, &ex);
  const float scale = ldexpf(1.f, -ex), unscale = ldexpf(1.f, ex);
#pragma unroll
  for (int ri = 0; ri < R; ++ri)
#pragma unroll
    for (int j = 0; j < TMAX / 2; ++j) {
      a[ri][j].x *= scale;
      a[ri][j].y *= scale;
    }
  LRD_STAMP(1);

  // ---- Householder tridiagonalisation ------------------------------------------
  int hbase = 0;  // packed offset of row k of HV
  float x[R];     // column k of the own rows
  auto column = [&](int k) {
#define LRD_COL(J)                                                        \
  case J:                                                                 \
    if constexpr (J < NG) {                                               \
      _Pragma("unroll") for (int ri = 0; ri < R; ++ri) {                  \
        const float2 pr = (k & 2) ? a[ri][2 * J + 1] : a[ri][2 * J];      \
        x[ri] = (k & 1) ? pr.y : pr.x;                                    \
      }                                                                   \
    }                                                                     \
    break;
    switch (k >> 2) {
      LRD_COL(0) LRD_COL(1) LRD_COL(2) LRD_COL(3) LRD_COL(4) LRD_COL(5) LRD_COL(6) LRD_COL(7)
      LRD_COL(8) LRD_COL(9) LRD_COL(10) LRD_COL(11) LRD_COL(12) LRD_COL(13) LRD_COL(14) LRD_COL(15)
      default: break;
    }
#undef LRD_COL
  };
  auto at_row = [&](int r) {  // x of row r (the same r in every lane), from its lane
    float v = x[0];
#pragma unroll
    for (int ri = 1; ri < R; ++ri)
      if (r / L == ri) v = x[ri];
    return __shfl_sync(0xffffffffu, v, r & (L - 1), L);
  };
#pragma unroll 1
  for (int k = 0; k < n - 2; ++k) {
    column(k);
    float part = 0.f;
#pragma unroll
    for (int ri = 0; ri < R; ++ri) part = (l + L * ri >= k + 2) ? fmaf(x[ri], x[ri], part) : part;
    const float alpha = at_row(k + 1);
    const float dk = at_row(k);
    const float xnorm2 = sub_sum<L>(part);
    // beta = -sign(alpha) |x|, tau = (beta - alpha) / beta, sc = 1 / (alpha - beta);
    // the approximate reciprocal (root) and a Newton step
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
    if (l == 0) {
      d[k] = dk;
      e[k] = beta;
      tau[k] = taui;
    }
    // row k of HV from its first live column group j4lo on; hv[c] = column c (all
    // zero where there is nothing to reflect)
    const int j4lo = (k + 1) >> 2;
    float* hv = HV + hbase - 4 * j4lo;
    hbase += TMAX - 4 * j4lo;
    float v[R];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int r = l + L * ri;
      v[ri] = (r == k + 1) ? one : ((r >= k + 2) ? x[ri] * sc : 0.f);
      if (r >= 4 * j4lo) hv[r] = v[ri];
    }
    __syncwarp();
    // p = tau A v over the live column groups (hv is 0 below column k + 1)
    const float4* hv4 = reinterpret_cast<const float4*>(hv);
    float2 s01[R], s23[R];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) s01[ri] = s23[ri] = make_float2(0.f, 0.f);
    float4 ve, vo;
    if constexpr (PF) ve = hv4[(j4lo + 1) & ~1], vo = hv4[j4lo | 1];
#define LRD_MV(J)                                                    \
  case J:                                                            \
    if constexpr (J < NG) {                                          \
      float4& v4 = (J & 1) ? vo : ve;                                \
      if constexpr (!PF) v4 = hv4[J];                                \
      _Pragma("unroll") for (int ri = 0; ri < R; ++ri) {             \
        fma2(s01[ri], a[ri][2 * J], make_float2(v4.x, v4.y));        \
        fma2(s23[ri], a[ri][2 * J + 1], make_float2(v4.z, v4.w));    \
      }                                                              \
      if constexpr (PF && J + 2 < NG) v4 = hv4[J + 2];               \
    }
    switch (j4lo) {
      LRD_MV(0) LRD_MV(1) LRD_MV(2) LRD_MV(3) LRD_MV(4) LRD_MV(5) LRD_MV(6) LRD_MV(7)
      LRD_MV(8) LRD_MV(9) LRD_MV(10) LRD_MV(11) LRD_MV(12) LRD_MV(13) LRD_MV(14) LRD_MV(15)
      default: break;
    }
#undef LRD_MV
    float p[R], part2 = 0.f;
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int r = l + L * ri;
      p[ri] = r >= k + 1 ? taui * ((s01[ri].x + s01[ri].y) + (s23[ri].x + s23[ri].y)) : 0.f;
      ps[r] = p[ri];
      part2 = fmaf(p[ri], v[ri], part2);
    }
    const float kc2 = -taui * sub_sum<L>(part2);  // 2 kc
    __syncwarp();
    // A -= v p^T + (p + 2 kc v) v^T over the live column groups
    const float4* ps4 = reinterpret_cast<const float4*>(ps);
    float2 mv[R], mc[R];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const float c = fmaf(kc2, v[ri], p[ri]);
      mv[ri] = make_float2(-v[ri], -v[ri]);
      mc[ri] = make_float2(-c, -c);
    }
    float4 pe, po;
    if constexpr (PF) {
      ve = hv4[(j4lo + 1) & ~1], vo = hv4[j4lo | 1];
      pe = ps4[(j4lo + 1) & ~1], po = ps4[j4lo | 1];
    }
#define LRD_UPD(J)                                                   \
  case J:                                                            \
    if constexpr (J < NG) {                                          \
      float4 &v4 = (J & 1) ? vo : ve, &p4 = (J & 1) ? po : pe;       \
      if constexpr (!PF) v4 = hv4[J], p4 = ps4[J];                   \
      _Pragma("unroll") for (int ri = 0; ri < R; ++ri) {             \
        fma2(a[ri][2 * J], mc[ri], make_float2(v4.x, v4.y));         \
        fma2(a[ri][2 * J + 1], mc[ri], make_float2(v4.z, v4.w));     \
        fma2(a[ri][2 * J], mv[ri], make_float2(p4.x, p4.y));         \
        fma2(a[ri][2 * J + 1], mv[ri], make_float2(p4.z, p4.w));     \
      }                                                              \
      if constexpr (PF && J + 2 < NG) {                              \
        v4 = hv4[J + 2];                                             \
        p4 = ps4[J + 2];                                             \
      }                                                              \
    }
    switch (j4lo) {
      LRD_UPD(0) LRD_UPD(1) LRD_UPD(2) LRD_UPD(3) LRD_UPD(4) LRD_UPD(5) LRD_UPD(6) LRD_UPD(7)
      LRD_UPD(8) LRD_UPD(9) LRD_UPD(10) LRD_UPD(11) LRD_UPD(12) LRD_UPD(13) LRD_UPD(14) LRD_UPD(15)
      default: break;
    }
#undef LRD_UPD
    // (ps is rewritten only after the next step's first __syncwarp)
  }
  {
    column(n - 2);
    const float d2 = at_row(n - 2), e2 = at_row(n - 1);
    column(n - 1);
    const float d1 = at_row(n - 1);
    if (l == 0) {
      d[n - 2] = d2;
      e[n - 2] = e2;
      d[n - 1] = d1;
      e[n - 1] = 0.f;
    }
  }
  __syncwarp();
  LRD_STAMP(2);

  // ---- eigenvalues, MP rank ------------------------------------------------------
  float tnorm;
  bisect_reg<TMAX>(d, e, lam, W, n, tnorm);
  LRD_STAMP(3);
  int p;
  const double margin = mp_rank_sub<L>(lam, unscale, n, nvox, W, p, (sig2 && mine) ? sig2 + b : nullptr);
  // queued for float64: a near-tie, or a vector that Gram-Schmidt finds lost
  bool queue = margin < kRefineTol;
  if (l == 0 && mine) {
    ranks[b] = p;
    wgt[b] = (float)(1.0 / (2.0 + (double)p));
  }
  if (lam_out != nullptr && mine)
    for (int i = l; i < n; i += L) lam_out[b * n + i] = lam[i] * unscale;
  LRD_STAMP(4);
  const int pmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)p);

  // ---- top-p eigenvectors, IG at a time -------------------------------------------
  float* V = vecs + b * (long long)n * n;
  float* Z = W;
  float* U = W + TMAX * IG;
#pragma unroll 1
  for (int j0 = 0; j0 < pmax; j0 += IG) {
    const int g = min(IG, p - j0);  // <= 0: this matrix has no more
    __syncwarp();
    twisted_vectors<L, IG>(d, e, lam, Z, U, n, j0, g, tnorm);
    LRD_STAMP(5);
    // row-distributed: y[ri][q / 2] = vectors q, q + 1, row l + L ri
    float2 y[R][IG / 2];
#pragma unroll
    for (int ri = 0; ri < R; ++ri) {
      const int r = l + L * ri;
#pragma unroll
      for (int q = 0; q < IG; q += 2) {
        const float2 z = *reinterpret_cast<const float2*>(Z + r * IG + q);
        y[ri][q / 2] = make_float2(r < n && q < g ? z.x : 0.f, r < n && q + 1 < g ? z.y : 0.f);
      }
    }
    // back-transform x = H(0) ... H(n-3) y, on the first 2 GP vectors of the chunk
    auto back_transform = [&](auto gtag) {
      constexpr int GP = decltype(gtag)::value;
      int hb = hbase;  // end of the packed rows
#pragma unroll 1
      for (int k = n - 3; k >= 0; --k) {
        const int j4lo = (k + 1) >> 2;
        hb -= TMAX - 4 * j4lo;
        const float* hrow = HV + hb - 4 * j4lo;
        const float tk = tau[k];
        float h[R];
        float2 dq[GP];
#pragma unroll
        for (int ri = 0; ri < R; ++ri) {
          const int r = l + L * ri;
          h[ri] = r >= 4 * j4lo ? hrow[r] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < GP; ++q) {
          dq[q] = make_float2(0.f, 0.f);
#pragma unroll
          for (int ri = 0; ri < R; ++ri) fma2(dq[q], make_float2(h[ri], h[ri]), y[ri][q]);
        }
        sub_allsum<L, GP>(dq);
#pragma unroll
        for (int q = 0; q < GP; ++q) {
          const float2 f = make_float2(-tk * dq[q].x, -tk * dq[q].y);
#pragma unroll
          for (int ri = 0; ri < R; ++ri) fma2(y[ri][q], make_float2(h[ri], h[ri]), f);
        }
      }
    };
    if (IG == 4 || pmax - j0 <= 4)
      back_transform(IntTag<2>{});
    else
      back_transform(IntTag<IG / 2>{});
    LRD_STAMP(6);
    queue |= gram_schmidt<L, R, IG>(y, V, lam, tnorm, n, j0, g, min(IG, pmax - j0), mine);
    __syncwarp();
  }
  if (l == 0 && mine && refine_count != nullptr && queue) refine_ids[atomicAdd(refine_count, 1)] = (int)(patch0 + b);
  LRD_STAMP(7);
}

// Warps per SM: 168 registers, what 32 x 4, 48 x 3 and 64 x 2 row entries and the
// rest leave with few spills (bytes stored / loaded, alone and in the packed launch:
// T = 32 20 / 44 and 24 / 24, T = 48 208 / 240 and 324 / 244, T = 64 88 / 52 and 8 / 8).
template <int TMAX>
__host__ __device__ constexpr int eigh_reg_min_blocks() {
  return 12;
}

template <int TMAX>
__global__ void __launch_bounds__(32, eigh_reg_min_blocks<TMAX>())
    eigh_reg_kernel(const float* gram, float* vecs, float* __restrict__ lam_out, int32_t* __restrict__ ranks,
                    float* __restrict__ wgt, float* __restrict__ sig2, int n, int nvox, long long patch0,
                    int* __restrict__ refine_count, int* __restrict__ refine_ids, long long nmat) {
  eigh_reg_body<TMAX>(gram, vecs, lam_out, ranks, wgt, sig2, n, nvox, patch0, refine_count, refine_ids,
                      (long long)blockIdx.x * eigh_reg_mats<TMAX>(), nmat);
}

// The same with eight warps per SM and the registers that gives: for launches that
// fit the device at once, where a matrix's latency is all that counts (bit-identical
// results; the same operations in the same order). Fewer matrices a warp while they fit
// measured slower (600 matrices at T = 48 0.089 -> 0.105 ms, 2000 at T = 32 0.084 -> 0.092).
constexpr int kEighWideBlocks = 8;
template <int TMAX>
__global__ void __launch_bounds__(32, kEighWideBlocks)
    eigh_reg_wide_kernel(const float* gram, float* vecs, float* __restrict__ lam_out, int32_t* __restrict__ ranks,
                         float* __restrict__ wgt, float* __restrict__ sig2, int n, int nvox, long long patch0,
                         int* __restrict__ refine_count, int* __restrict__ refine_ids, long long nmat) {
  eigh_reg_body<TMAX, true>(gram, vecs, lam_out, ranks, wgt, sig2, n, nvox, patch0, refine_count, refine_ids,
                            (long long)blockIdx.x * eigh_reg_mats<TMAX>(), nmat);
}

}  // namespace lrd
