// Batched T x T symmetric eigensolver + Marchenko-Pastur rank + weight.
//
// Replaces the ladder's ``torch.linalg.eigh`` (step8_tuned.py:134; cuSOLVER),
// ``mp_keep`` (step8_tuned.py:96-113), the projector bmm (step8:136) and the
// weight (step8:137). For each patch's Gram matrix:
//
//  1. exact power-of-two scaling so the largest diagonal entry is in [0.5, 1);
//  2. Householder reduction to tridiagonal form, one reflector per column;
//  3. every eigenvalue from Sturm counts, its interval cut at one or several
//     points a round;
//  4. the MP rank from the full spectrum, evaluated like step0_numpy_loop.py:
//     18-24: eigs = float32(max(lambda, 0) / N) in descending order with the
//     smallest (null) eigenvalue dropped (step4_gram_eigh.py:49), float32
//     suffix sums rcum, and the test
//       float64(float32(eigs_i - eigs_last)) * (t - i) * (N - i)
//         > float64(float32(4 * rcum_i)) * sqrt(float64(t * N))
//     counted over all i (NumPy promotes the ladder's test to float64);
//  5. the top-p eigenvectors, a few at a time: those of the tridiagonal matrix,
//     the Householder back-transform, then modified Gram-Schmidt in descending
//     eigenvalue order;
//  6. w = float32(1 / (2 + p)) (step0:36).
//
// The main pass runs these steps in float32 on the float32 Gram, the matrix in the
// registers of a warp's lanes or of a CTA's threads, its vectors by twisted
// factorisations (eigh_reg.cuh, eigh_cta.cuh). A patch whose MP test has an index
// with |lhs/rhs - 1| below kRefineTol (a near-tie that float32 round-off could
// decide either way), or one of whose kept vectors float32 could not tell from an
// earlier one, is queued, and eigh_refine_kernel (eigh_refine.cuh) redoes it in
// float64: each voxel's time course centred in float64 from the input volume (the
// float64 mean of its float32 values), the Gram from float64 products with a
// float64 sum, then the same steps in float64, the vectors by inverse iteration
// (partial-pivoting LU) from pseudo-random starts - so near-ties are decided as
// the float64 evaluation of the algorithm decides them, down to margins far
// below the float32 centred data's own rounding.
//
// Output per patch: the p eigenvectors (descending eigenvalue order) as the
// rows of a compact p x T block at the start of the patch's T x T slot (the
// projector of step8:136 is V_p V_p^T; the reconstruction applies it as
// (x V_p) V_p^T), the rank, the weight, optionally the ascending eigenvalues.
#pragma once

#include <float.h>

#include "lrd_common.cuh"

namespace lrd {

template <typename Real>
struct Num;
template <>
struct Num<float> {
  static __device__ __forceinline__ float eps() { return FLT_EPSILON * 0.5f; }
  static __device__ __forceinline__ float tiny() { return FLT_MIN; }
  static __device__ __forceinline__ float huge() { return FLT_MAX; }
  static __device__ __forceinline__ float rsq(float a) { return rsqrtf(a); }
};
template <>
struct Num<double> {
  static __device__ __forceinline__ double eps() { return DBL_EPSILON * 0.5; }
  static __device__ __forceinline__ double tiny() { return DBL_MIN; }
  static __device__ __forceinline__ double huge() { return DBL_MAX; }
  static __device__ __forceinline__ double rsq(double a) { return rsqrt(a); }
};

template <typename Real>
__device__ __forceinline__ Real warp_sum(Real v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename Real>
__device__ __forceinline__ Real warp_max(Real v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <typename Real>
__device__ __forceinline__ Real warp_min(Real v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Deterministic start vector entry in [-1, 1) for inverse iteration.
__device__ __forceinline__ float start_entry(int i, int j) {
  unsigned h = (unsigned)i * 0x9E3779B1u ^ ((unsigned)j + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return (float)(h >> 8) * (2.0f / 16777216.0f) - 1.0f;
}

constexpr int kInvGroup = 8;  // eigenvectors formed at once, at most
constexpr int kInvSolves = 2;  // float64 pass: inverse-iteration solves per eigenvector

// Floats of the packed Householder reflector rows of the float32 solvers: row
// k (k < n - 2 <= TMAX - 2) is stored from its first live 4-column group on,
// columns [4 * ((k + 1) >> 2), TMAX), about half of TMAX x TMAX.
template <int TMAX>
__host__ __device__ constexpr size_t eigh_hv_floats() {
  size_t f = 0;
  for (int k = 0; k < TMAX - 2; ++k) f += (size_t)(TMAX - 4 * ((k + 1) >> 2));
  return f;
}
constexpr int kLdy = kInvGroup + 1;  // eigenvector chunk row stride
constexpr double kRefineTol = 1e-4;  // MP-test margin below which float64 redoes the patch
// Margin of the float64 pass's step-0 emulation below which its decision is
// taken from the test in float64 throughout (within float32 resolution of the
// data, step 0's float32 arithmetic could decide either way).
constexpr double kTieFloor = 1e-6;

// MP rank from the ascending eigenvalues lam * unscale, evaluated like
// step0_numpy_loop.py:18-24 (float32 eigs and suffix sums, float64 test,
// a count over all indices); W holds 2n floats of scratch (4n + 2 in the
// float64 instantiation, whose W is 8-byte aligned). Returns the
// smallest |lhs/rhs - 1| over the indices. With ``sig2_out`` lane 0 also
// writes the patch's noise variance estimate, the mean of the t - p noise
// eigenvalues: rcum_p / (t - p) in float32 (0 when p = t). One warp.
template <typename Real>
__device__ double mp_rank(const Real* lam, Real unscale, int n, int nvox, float* W, int& p_out,
                          float* sig2_out = nullptr) {
  const int lane = threadIdx.x & 31;
  // eigs = float32(max(lambda, 0) / N), as step 0's float32 s**2 / n.
  const int t = n - 1;
  float* eg = W;                             // descending eigs, t entries
  float* rc = eg + n;                        // float32 suffix sums
  for (int i = lane; i < t; i += 32) {
    const Real l = fmax(lam[n - 1 - i] * unscale, Real(0));
    eg[i] = (sizeof(Real) == 4) ? __fdiv_rn((float)l, (float)nvox) : (float)(l / (Real)nvox);
  }
  __syncwarp();
  if (lane == 0) {
    float acc = eg[t - 1];
    rc[t - 1] = acc;
    for (int i = t - 2; i >= 0; --i) {
      acc = __fadd_rn(acc, eg[i]);
      rc[i] = acc;
    }
  }
  __syncwarp();
  int p = 0;
  double margin = DBL_MAX;
  {
    const double sq = sqrt((double)((long long)t * (long long)nvox));
    const float elast = eg[t - 1];
    for (int i0 = 0; i0 < t; i0 += 32) {
      const int i = i0 + lane;
      bool sig = false;
      if (i < t) {
        const double lhs = (double)__fsub_rn(eg[i], elast) * (double)(t - i) * (double)(nvox - i);
        const double rhs = (double)__fmul_rn(4.f, rc[i]) * sq;
        sig = lhs > rhs;
        if (rhs > 0.0) margin = fmin(margin, fabs(lhs - rhs) / rhs);
      }
      p += __popc(__ballot_sync(0xffffffffu, sig));
    }
    margin = warp_min(margin);
  }
  if constexpr (sizeof(Real) == 8) {
    // The float64 near-tie pass. Below a margin of kTieFloor the step-0
    // emulation (float32 eigs and sums) decides within float32 resolution of
    // the data - step 0's own float32 SVD could land either way - so the
    // count is taken from the test in float64 throughout (eigs, suffix sums
    // and products), the decision of the float64 run of the algorithm.
    if (margin < kTieFloor) {
      double* e64 = reinterpret_cast<double*>(rc + n);  // past the float32 arrays (float offset 2n: 8-byte aligned)
      for (int i = lane; i < t; i += 32) e64[i] = fmax((double)lam[n - 1 - i] * (double)unscale, 0.0) / nvox;
      __syncwarp();
      double r64 = 0.0, tail = 0.0;
      const double sq = sqrt((double)((long long)t * (long long)nvox));
      int p64 = 0;
      // suffix sums in double by lane 0 (t <= 127 terms), then the count
      if (lane == 0) {
        for (int i = t - 1; i >= 0; --i) {
          r64 += e64[i];
          const double lhs = (e64[i] - e64[t - 1]) * (double)(t - i) * (double)(nvox - i);
          p64 += lhs > 4.0 * r64 * sq;
        }
        tail = (double)p64;
      }
      p = (int)__shfl_sync(0xffffffffu, tail, 0);
      __syncwarp();
    }
  }
  p_out = p;
  if (sig2_out != nullptr && lane == 0) *sig2_out = (p < t) ? __fdiv_rn(rc[p], (float)(t - p)) : 0.f;
  return margin;
}

}  // namespace lrd
