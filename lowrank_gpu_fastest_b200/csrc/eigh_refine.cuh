// Float64 pass over the near-tie patches: Gram matrix from the input volume,
// eigenvalues, MP rank and the top-p eigenvectors of one patch per CTA.
//
// A queue holds a handful of patches per volume (0..2 of the headline's
// 12600), so this kernel is one patch's latency added to every call that has
// a near-tie, and everything in it is laid out for that: 16 warps on one
// patch, few barriers, no serial chain that can be spread.
//
//  * Gram: chunks of voxel rows, the next chunk's loads in flight while this
//    one is used, centred in float64 by eight lanes per row as they are
//    staged. Threads own 4 x 4 blocks of the upper block triangle, several
//    threads per block splitting the chunk's rows (1.66 M DFMA per patch at
//    T = 48, N = 1331: 26 K cycles of the SM's 64 DFMA a clock; 8 shared
//    doubles feed 16 DFMA). Block b holds frames 2b, 2b + 1 and those nb pairs
//    further on, so neighbouring threads read neighbouring 16 bytes.
//  * Householder: the full symmetric matrix in shared memory, TPR threads per
//    row; three barriers a step. Both dot products are formed by every warp
//    for itself, and with p = tau A v, kc = -tau/2 p.v the update is
//    A -= v p^T + (p + 2 kc v) v^T, which needs no second vector.
//  * Eigenvalues: 512 / n threads share an eigenvalue and cut its interval
//    into that many + 1 parts a round (11 rounds at T = 48 instead of 38
//    bisections), counting with the division-free Sturm recurrence
//    p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (a sign change per eigenvalue
//    below x), rescaled every eight steps.
//  * Inverse iteration (a lane per vector), back-transform (a warp per
//    vector), modified Gram-Schmidt.
//
// Measured on B200, one queued patch of 1331 voxels, against the 128-thread
// kernel this replaces (kernel time): T = 48 990 -> 215 us, T = 96 2926 -> 490
// us; 254 patches of 125 voxels at T = 32: 287 -> 200 us. Cycles at T = 48: Gram
// 140 K, Householder 148 K (3200 a step, a chain of rsqrt, reciprocal, two
// shuffle sums and three barriers), eigenvalues 58 K, inverse iteration 32 K,
// back-transform 15 K. IEEE float64 division (410 cycles) and shuffles with a
// mask per row (which serialise over the masks of a warp) are kept out of it.
#pragma once

#include "eigh.cuh"

namespace lrd {

constexpr int kRefineThreads = 512;
constexpr int kRefineRows = 64;  // voxel rows per staged chunk: four per warp, eight lanes each

// Threads per matrix row (a power of two) and the row stride that keeps a
// half-warp's (16 / TPR rows) x TPR doubles on distinct banks.
__host__ __device__ inline int refine_tpr(int n) {
  int t = 1;
  while (t < 32 && 2 * t * n <= (n <= 64 ? 256 : kRefineThreads)) t *= 2;
  return t;
}
__host__ __device__ inline int refine_lda(int n) {
  const int want = refine_tpr(n) & 15;
  int lda = n;
  while ((lda & 15) != want) ++lda;
  return lda;
}
// Doubles of the work area W: LU of kInvGroup shifted tridiagonals, or two
// buffers of Sturm counts and the scaled tridiagonal.
__host__ __device__ inline int refine_work_elems(int n) {
  const int lu = 4 * n * kInvGroup, cnt = kRefineThreads + 2 * n;
  return lu > cnt ? lu : cnt;
}
__host__ __device__ inline size_t refine_elems(int n) {
  return (size_t)n * refine_lda(n) + (size_t)n * kLdy + 5 * (size_t)n + refine_work_elems(n) + 8;
}
// Staged voxel rows: two chunks, over the memory the solver uses later. Above
// 124 frames the blocks outnumber the threads, the patch is walked twice, and
// the chunks (16 rows) follow that memory instead.
__host__ __device__ inline bool refine_two_pass(int n) { return n > 124; }
__host__ __device__ inline int refine_rows(int n) { return refine_two_pass(n) ? 16 : kRefineRows; }
__host__ __device__ inline size_t refine_stage_at(int n) {
  return refine_two_pass(n) ? (refine_elems(n) + 1) & ~size_t(1) : 0;
}
__host__ __device__ inline size_t eigh_refine_smem_bytes(int n) {
  const size_t end = refine_stage_at(n) + 2 * (size_t)refine_rows(n) * ((n + 3) & ~3);
  return sizeof(double) * (end > refine_elems(n) ? end : refine_elems(n));
}

// 1 / a for a normal, nonzero a, to an ulp or so: the square of rsqrt and one
// Newton step (110 cycles of latency; the IEEE division measured 410).
__device__ __forceinline__ double recip(double a) {
  const double r = rsqrt(fabs(a)), y = copysign(r * r, a);
  return fma(y, fma(-a, y, 1.0), y);
}

// Sign changes of the Sturm sequence of the n x n tridiagonal (d, e2 > 0; both
// scaled so that the norm is below 1): the number of eigenvalues below x.
// Entries shrink by at most 2^-116 in two steps (e2 is at least that), so
// eight steps between rescalings stay far from underflow.
__device__ __forceinline__ int sturm_changes(const double* d, const double* e2, int n, double x) {
  double p2 = 1.0, p1 = d[0] - x;
  int c = (int)((unsigned)__double2hiint(p1) >> 31);
  auto step = [&](double di, double ei) {
    const double p = fma(di - x, p1, -(ei * p2));
    c += (int)((unsigned)(__double2hiint(p) ^ __double2hiint(p1)) >> 31);
    p2 = p1;
    p1 = p;
  };
  int i = 1;
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) step(d[i + u], e2[i + u - 1]);
    const int h = max(__double2hiint(p1) & 0x7fffffff, __double2hiint(p2) & 0x7fffffff) >> 20;
    const double s = __hiloint2double((2046 - min(max(h, 1), 2045)) << 20, 0);
    p1 *= s;
    p2 *= s;
  }
  for (; i < n; ++i) step(d[i], e2[i - 1]);
  return c;
}

// Eigen-decomposition of the n x n matrix in ``A`` (row stride lda, full), MP
// rank and weight, top-p eigenvectors as the rows of the compact p x n block
// ``V``, optionally the ascending eigenvalues.
__device__ __forceinline__ void refine_solve(double* A, int n, int nvox, float* V, float* lam_out, int32_t* rank_out,
                                             float* w_out, float* s2_out) {
  constexpr int NT = kRefineThreads, NWARP = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lda = refine_lda(n), tpr = refine_tpr(n);
  double* Y = A + (size_t)n * lda;
  double* d = Y + n * kLdy;
  double* e = d + n;
  double* e2 = e + n;
  double* tau = e2 + n;
  double* lam = tau + n;
  double* W = lam + n;
  int* pshare = reinterpret_cast<int*>(W + refine_work_elems(n));
  const double eps = Num<double>::eps();

  // exact power-of-two scaling: the largest diagonal entry into [0.5, 1)
  double dm = 0.0;
  for (int i = lane; i < n; i += 32) dm = fmax(dm, fabs(A[i * lda + i]));
  dm = warp_max(dm);
  int ex = 0;
  if (dm > 0.0 && isfinite(dm)) frexp(dm, &ex);
  const double scale = ldexp(1.0, -ex), unscale = ldexp(1.0, ex);
  __syncthreads();
  const int row = tid / tpr, sub = tid - row * tpr;  // this thread's row and share of its columns
  if (row < n)
    for (int j = sub; j < n; j += tpr) A[row * lda + j] *= scale;
  __syncthreads();

  // ---- Householder tridiagonalisation ----------------------------------------
  double* vv = W;
  double* pp = W + n;
  double* xn = W + 2 * n;
  double xnorm2 = 0.0;
  const int wlast = ((n - 1) * tpr) >> 5;  // the warp of row n - 1 is at work in every step
  const int row_hi = (warp * 32 + 31) / tpr;  // the last row of this warp's threads
  for (int k = 0; k < n - 2; ++k) {
    // (a warp none of whose rows is left only joins the barriers)
    const bool at_work = warp <= wlast && row_hi > k;
    const bool live = row > k && row < n;
    double taui = 0.0;
    if (at_work) {
      // row k (= column k): its norm was left by the threads that updated it
      const double* xrow = A + k * lda;
      if (k == 0) {
        double part = 0.0;
        for (int j = 2 + lane; j < n; j += 32) part = fma(xrow[j], xrow[j], part);
        xnorm2 = warp_sum(part);
      } else {
        xnorm2 = *xn;
      }
      const double alpha = xrow[k + 1];
      double beta = alpha, scv = 0.0;
      if (xnorm2 > 0.0) {
        // beta = -sign(alpha) |x|, tau = (beta - alpha) / beta, scv = 1 / (alpha - beta)
        const double nrm2 = fma(alpha, alpha, xnorm2), rs = rsqrt(nrm2), nrm = nrm2 * rs;
        beta = -copysign(nrm, alpha);
        taui = fma(fabs(alpha), rs, 1.0);
        scv = copysign(recip(fabs(alpha) + nrm), alpha);
      }
      if (warp == wlast) {
        for (int j = k + 1 + lane; j < n; j += 32) vv[j] = j == k + 1 ? 1.0 : xrow[j] * scv;
        if (lane == 0) {
          d[k] = xrow[k];
          e[k] = beta;
          tau[k] = taui;
        }
      }
    }
    __syncthreads();
    // columns of this thread: j = sub (mod tpr), j > k
    const int j0 = k + 1 + ((sub - (k + 1)) & (tpr - 1));
    if (at_work && taui != 0.0) {
      // (shuffles by whole warps: with a mask per row they took most of the step)
      double s0 = 0.0, s1 = 0.0;
      if (live) {
        const double* ar = A + row * lda;
        for (int j = j0; j < n; j += 4 * tpr) {
          double av[4], xv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = j + u * tpr < n;
            av[u] = in ? ar[j + u * tpr] : 0.0;
            xv[u] = in ? vv[j + u * tpr] : 0.0;
          }
          s0 = fma(av[2], xv[2], fma(av[0], xv[0], s0));
          s1 = fma(av[3], xv[3], fma(av[1], xv[1], s1));
        }
      }
      s0 += s1;
      for (int o = tpr >> 1; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      if (live && sub == 0) pp[row] = taui * s0;
    }
    __syncthreads();
    if (at_work && taui != 0.0) {
      double dots[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = k + 1 + lane + 32 * u;
        dots[u] = j < n ? pp[j] * vv[j] : 0.0;
      }
      const double kc = -0.5 * taui * warp_sum((dots[0] + dots[1]) + (dots[2] + dots[3]));
      double sq = 0.0;
      if (live) {
        const double vi = vv[row], ci = fma(2.0 * kc, vi, pp[row]);
        double* ar = A + row * lda;
        for (int j = j0; j < n; j += 4 * tpr) {
          double av[4], xv[4], pv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const bool in = j + u * tpr < n;
            av[u] = in ? ar[j + u * tpr] : 0.0;
            xv[u] = in ? vv[j + u * tpr] : 0.0;
            pv[u] = in ? pp[j + u * tpr] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double v = fma(-vi, pv[u], fma(-ci, xv[u], av[u]));
            if (j + u * tpr < n) ar[j + u * tpr] = v;
            if (j + u * tpr >= k + 3) sq = fma(v, v, sq);
          }
        }
      }
      if (warp == wlast)  // the reflector, for the back-transform
        for (int j = k + 1 + lane; j < n; j += 32) A[k * lda + j] = vv[j];
      if (warp == ((k + 1) * tpr) >> 5) {  // the next step's norm, from the threads of row k + 1
        for (int o = tpr >> 1; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (row == k + 1 && sub == 0) *xn = sq;
      }
    } else if (warp == wlast) {  // nothing to reflect: the next row is as it was
      const double* xnext = A + (k + 1) * lda;
      double part = 0.0;
      for (int j = k + 3 + lane; j < n; j += 32) part = fma(xnext[j], xnext[j], part);
      part = warp_sum(part);
      if (lane == 0) *xn = part;
    }
    __syncthreads();
  }
  if (tid == 0) {
    d[n - 2] = A[(n - 2) * lda + (n - 2)];
    e[n - 2] = A[(n - 1) * lda + (n - 2)];
    tau[n - 2] = 0.0;
    d[n - 1] = A[(n - 1) * lda + (n - 1)];
    e[n - 1] = 0.0;
    tau[n - 1] = 0.0;
  }
  __syncthreads();

  // ---- eigenvalues -------------------------------------------------------------
  // intervals end at 100 eps of the norm bound (1e-14): this pass settles the
  // MP test and the top eigenvectors
  double glo = Num<double>::huge(), ghi = -Num<double>::huge();
  for (int i = lane; i < n; i += 32) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    glo = fmin(glo, d[i] - r);
    ghi = fmax(ghi, d[i] + r);
  }
  glo = warp_min(glo);
  ghi = warp_max(ghi);
  const double tnorm = fmax(fmax(fabs(glo), fabs(ghi)), Num<double>::tiny());
  glo -= 4.0 * eps * tnorm * n;
  ghi += 4.0 * eps * tnorm * n;
  {
    // the tridiagonal scaled by a power of two to a norm in [0.5, 1); an
    // off-diagonal below 2^-58 of the norm is raised to it (an eigenvalue moves
    // by no more than that), so the Sturm sequence cannot die out
    int ext = 0;
    if (isfinite(tnorm)) frexp(tnorm, &ext);
    const double ts = ldexp(1.0, -ext), tu = ldexp(1.0, ext);
    int* cnt = reinterpret_cast<int*>(W);  // two buffers of NT counts
    double* ds = W + NT;
    double* es = ds + n;
    for (int i = tid; i < n; i += NT) {
      ds[i] = d[i] * ts;
      const double ei = i < n - 1 ? e[i] * ts : 0.0;
      es[i] = fmax(ei * ei, 0x1p-116);
    }
    glo *= ts;
    ghi *= ts;
    __syncthreads();
    const double h0 = (ghi - glo) / (NT + 1);
    cnt[tid] = sturm_changes(ds, es, n, glo + (tid + 1) * h0);
    __syncthreads();
    const int m = NT / n;  // threads per eigenvalue (>= 4)
    const int j = tid / m, q = tid - j * m;
    double lo = glo, hi = ghi;
    if (j < n) {
      int lo_m = -1, hi_m = NT;  // cnt[lo_m] <= j < cnt[hi_m] holds along the search
      while (hi_m - lo_m > 1) {
        const int mid = (lo_m + hi_m) >> 1;
        if (cnt[mid] <= j) lo_m = mid; else hi_m = mid;
      }
      if (lo_m >= 0) lo = glo + (lo_m + 1) * h0;
      if (hi_m < NT) hi = glo + (hi_m + 1) * h0;
    }
    // (ghi - glo) / (NT + 1) < 2.1 / NT of the norm: rounds until 1e-14 of it
    int rounds = 0;
    for (double w = 2.1 / NT; w > 100.0 * eps && rounds < 40; w /= m + 1) ++rounds;
    for (int r = 0; r < rounds; ++r) {
      int* buf = cnt + ((r & 1) ? 0 : NT);  // the other buffer is still being read
      const double h = (hi - lo) / (m + 1);
      if (j < n) buf[tid] = sturm_changes(ds, es, n, lo + (q + 1) * h);
      __syncthreads();
      if (j < n) {
        int c = 0;
        while (c < m && buf[j * m + c] <= j) ++c;
        const double base = lo;
        if (c < m) hi = base + (c + 1) * h;
        if (c > 0) lo = base + c * h;
      }
    }
    if (j < n && q == 0) lam[j] = 0.5 * (lo + hi) * tu;
  }
  __syncthreads();

  if (warp == 0) {
    int p;
    mp_rank<double>(lam, unscale, n, nvox, reinterpret_cast<float*>(W), p, s2_out);
    if (lane == 0) {
      *rank_out = p;
      *w_out = (float)(1.0 / (2.0 + (double)p));
      *pshare = p;
    }
  }
  if (lam_out != nullptr)
    for (int i = tid; i < n; i += NT) lam_out[i] = (float)(lam[i] * unscale);
  __syncthreads();
  const int p = *pshare;

  // ---- top-p eigenvectors, kInvGroup at a time ---------------------------------
  const double pivtol = eps * tnorm;
  double* RU0 = W;
  double* U1 = RU0 + n * kInvGroup;
  double* ML = U1 + n * kInvGroup;
  double* SW = ML + n * kInvGroup;
  for (int j0 = 0; j0 < p; j0 += kInvGroup) {
    const int g = min(kInvGroup, p - j0);
    __syncthreads();
    if (warp == 0 && lane < g) {
      const int q = lane;
      const int j = j0 + q;
      const double sig = lam[n - 1 - j];
      double c = d[0] - sig, s = e[0];
      for (int i = 0; i < n - 1; ++i) {
        const double ei = e[i];
        const double an = d[i + 1] - sig;
        const double en = (i + 1 < n - 1) ? e[i + 1] : 0.0;
        const bool keep = fabs(c) >= fabs(ei);
        double piv = keep ? c : ei;
        if (fabs(piv) < pivtol) piv = (piv < 0.0) ? -pivtol : pivtol;
        const double rp = recip(piv);
        const double m = (keep ? ei : c) * rp;
        U1[i * kInvGroup + q] = keep ? s : an;
        ML[i * kInvGroup + q] = m;
        SW[i * kInvGroup + q] = keep ? 0.0 : 1.0;
        RU0[i * kInvGroup + q] = rp;
        const double cn = keep ? fma(-m, s, an) : fma(-m, an, s);
        s = keep ? en : -m * en;
        c = cn;
      }
      if (fabs(c) < pivtol) c = (c < 0.0) ? -pivtol : pivtol;
      RU0[(n - 1) * kInvGroup + q] = recip(c);
      for (int i = 0; i < n; ++i) Y[i * kLdy + q] = start_entry(i, j);
      for (int iter = 0; iter < kInvSolves; ++iter) {
        double y = Y[q];
        for (int i = 0; i < n - 1; ++i) {
          const double yn = Y[(i + 1) * kLdy + q];
          const double m = ML[i * kInvGroup + q];
          const bool sw = SW[i * kInvGroup + q] != 0.0;
          Y[i * kLdy + q] = sw ? yn : y;
          y = sw ? fma(-m, yn, y) : fma(-m, y, yn);
        }
        double x2 = y * RU0[(n - 1) * kInvGroup + q];
        Y[(n - 1) * kLdy + q] = x2;
        double x1 = (Y[(n - 2) * kLdy + q] - U1[(n - 2) * kInvGroup + q] * x2) * RU0[(n - 2) * kInvGroup + q];
        Y[(n - 2) * kLdy + q] = x1;
        double amax = fmax(fabs(x2), fabs(x1));
        for (int i = n - 3; i >= 0; --i) {
          const double u2 = (SW[i * kInvGroup + q] != 0.0) ? e[i + 1] : 0.0;
          const double xi = (Y[i * kLdy + q] - U1[i * kInvGroup + q] * x1 - u2 * x2) * RU0[i * kInvGroup + q];
          Y[i * kLdy + q] = xi;
          amax = fmax(amax, fabs(xi));
          x2 = x1;
          x1 = xi;
        }
        if (!(amax > 0.0) || !isfinite(amax)) {
          for (int i = 0; i < n; ++i) Y[i * kLdy + q] = start_entry(i, j + 977 * (iter + 1));
          continue;
        }
        const double sa = 1.0 / amax;
        double n0 = 0.0, n1 = 0.0;
        for (int i = 0; i + 1 < n; i += 2) {
          const double v0 = Y[i * kLdy + q] * sa, v1 = Y[(i + 1) * kLdy + q] * sa;
          n0 = fma(v0, v0, n0);
          n1 = fma(v1, v1, n1);
        }
        if (n & 1) {
          const double v = Y[(n - 1) * kLdy + q] * sa;
          n0 = fma(v, v, n0);
        }
        const double inv = sa * Num<double>::rsq(n0 + n1);
        for (int i = 0; i < n; ++i) Y[i * kLdy + q] *= inv;
      }
    }
    __syncthreads();
    for (int q = warp; q < g; q += NWARP) {  // back-transform, rows lane + 32 u in registers
      double y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) y[u] = lane + 32 * u < n ? Y[(lane + 32 * u) * kLdy + q] : 0.0;
      for (int k = n - 3; k >= 0; --k) {
        const double tk = tau[k];
        double vr[4], part = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = lane + 32 * u;
          vr[u] = (i > k && i < n) ? A[k * lda + i] : 0.0;
          part = fma(vr[u], y[u], part);
        }
        if (tk == 0.0) continue;
        const double f = tk * warp_sum(part);
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = fma(-f, vr[u], y[u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (lane + 32 * u < n) Y[(lane + 32 * u) * kLdy + q] = y[u];
    }
    __syncthreads();
    if (warp == 0) {  // modified Gram-Schmidt in descending eigenvalue order
      for (int q = 0; q < g; ++q) {
        double y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = lane + 32 * u < n ? Y[(lane + 32 * u) * kLdy + q] : 0.0;
        for (int i = 0; i <= j0 + q; ++i) {  // i = j0 + q: the vector's own norm
          double z[4], part = 0.0;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int r = lane + 32 * u;
            z[u] = i == j0 + q ? y[u]
                   : r >= n    ? 0.0
                   : i < j0    ? (double)V[i * n + r]
                               : Y[r * kLdy + (i - j0)];
            part = fma(z[u], y[u], part);
          }
          const double dot = warp_sum(part);
          if (i < j0 + q) {
#pragma unroll
            for (int u = 0; u < 4; ++u) y[u] = fma(-dot, z[u], y[u]);
          } else {
            const double inv = Num<double>::rsq(fmax(dot, Num<double>::tiny()));
#pragma unroll
            for (int u = 0; u < 4; ++u) y[u] *= inv;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (lane + 32 * u < n) Y[(lane + 32 * u) * kLdy + q] = y[u];
        __syncwarp();
      }
    }
    __syncthreads();
    for (int idx = tid; idx < n * g; idx += NT) {
      const int c = idx / n, r = idx - c * n;
      V[(j0 + c) * n + r] = (float)Y[r * kLdy + c];
    }
  }
  __syncthreads();
}

// Body: this block is block ``bid`` of ``nblocks`` working on one volume's queue
// (refine_count[0] entries). ``vol`` (nullable): the input volume - its voxel
// rows are centred here in float64; without it the float32 centred rows ``xc``
// are used as they are.
__device__ __forceinline__ void eigh_refine_body(const float* __restrict__ vol, const float* __restrict__ xc,
                                                 float* vecs, float* __restrict__ lam_out,
                                                 int32_t* __restrict__ ranks, float* __restrict__ wgt,
                                                 float* __restrict__ sig2, const Geom& g, const AxisTables& tab,
                                                 const int* __restrict__ refine_count,
                                                 const int* __restrict__ refine_ids, int bid, int nblocks) {
  extern __shared__ __align__(16) double sm_ref[];
  constexpr int NT = kRefineThreads;
  const int n = g.nt;
  const int lda = refine_lda(n);
  const int nb = (n + 3) >> 2, ld = 4 * nb;  // 4 x 4 blocks; staged row length
  const int nblk = nb * (nb + 1) / 2;
  const int tid = threadIdx.x;
  const int count = refine_count[0];
  const int rows = refine_rows(n);
  const int nvox = g.nvox_patch;
  const int nchunk = (nvox + rows - 1) / rows;
  const int ks = max(1, NT / nblk);  // threads per 4 x 4 block, splitting the rows
  const float* src = vol != nullptr ? vol : xc;
  const int lds = vol != nullptr ? n : g.ldx;
  const double rn = vol != nullptr ? 1.0 / n : 0.0;  // 0: rows used as they are
  double* A = sm_ref;
  double* stage = sm_ref + refine_stage_at(n);
  for (int w = bid; w < count; w += nblocks) {
    const long long pid = refine_ids[w];
    int ci, cj, ck;
    patch_axes(g, pid, ci, cj, ck);
    const int cx = tab.corners[0][ci], cy = tab.corners[1][cj], cz = tab.corners[2][ck];
    // eight lanes per voxel row of a chunk: row sr, frames l8, l8 + 8, ...
    const int sr = tid >> 3, l8 = tid & 7;
    float pre[16];
    auto fetch = [&](int c) {
      const int v = c * rows + sr;
      const bool ok = sr < rows && v < nvox;
      const int x = v / (g.py * g.pz), yz = v - x * (g.py * g.pz), y = yz / g.pz;
      const float* p = src + (ok ? voxel_row(g, cx + x, cy + y, cz + (yz - y * g.pz)) * lds : 0);
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (8 * t < n) pre[t] = (ok && l8 + 8 * t < n) ? p[l8 + 8 * t] : 0.f;
    };
    // centred in float64 (the float32 input is exact in it); the padding
    // frames of a row and the rows past the patch are zero
    auto store = [&](double* buf) {
      double m = 0.0;
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (8 * t < n) m += (double)pre[t];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      m *= rn;
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        const int f = l8 + 8 * t;
        if (8 * t < ld && sr < rows && f < ld) buf[sr * ld + f] = f < n ? (double)pre[t] - m : 0.0;
      }
    };
    for (int blk0 = 0; blk0 < nblk; blk0 += NT) {
      const int kq = tid / nblk, blk = ks > 1 ? tid - kq * nblk : blk0 + tid;
      const bool owner = ks > 1 ? kq < ks : blk < nblk;
      int bi = 0, bj = 0;
      if (owner) {
        int rem = blk;
        while (rem >= nb - bi) {
          rem -= nb - bi;
          ++bi;
        }
        bj = bi + rem;
      }
      double acc[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) acc[u] = 0.0;
      __syncthreads();  // the area is free
      fetch(0);
      store(stage);
      __syncthreads();
      for (int c = 0; c < nchunk; ++c) {
        const double* cur = stage + (size_t)(c & 1) * rows * ld;
        if (c + 1 < nchunk) fetch(c + 1);
        if (owner) {
          const int left = min(rows, nvox - c * rows);
#pragma unroll 2
          for (int r = ks > 1 ? kq : 0; r < left; r += ks) {
            const double2* rp = reinterpret_cast<const double2*>(cur + r * ld);
            const double2 a0 = rp[bi], a1 = rp[nb + bi], b0 = rp[bj], b1 = rp[nb + bj];
            const double av[4] = {a0.x, a0.y, a1.x, a1.y}, bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
              for (int v = 0; v < 4; ++v) acc[u * 4 + v] = fma(av[u], bv[v], acc[u * 4 + v]);
          }
        }
        if (c + 1 < nchunk) store(stage + (size_t)((c + 1) & 1) * rows * ld);
        __syncthreads();
      }
      // the row split's partial sums added in order
      for (int s = 0; s < ks; ++s) {
        if (owner && (ks > 1 ? kq : 0) == s) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int r = (u < 2 ? 2 * bi : 2 * nb + 2 * bi - 2) + u, cc = (v < 2 ? 2 * bj : 2 * nb + 2 * bj - 2) + v;
              if (r < n && cc < n) {
                const double val = (s > 0 ? A[r * lda + cc] : 0.0) + acc[u * 4 + v];
                A[r * lda + cc] = val;
                if (bi != bj) A[cc * lda + r] = val;
              }
            }
        }
        __syncthreads();
      }
    }
    refine_solve(A, n, nvox, vecs + pid * (long long)n * n, lam_out ? lam_out + pid * n : nullptr, ranks + pid,
                 wgt + pid, sig2 ? sig2 + pid : nullptr);
  }
}

__global__ void __launch_bounds__(kRefineThreads)
    eigh_refine_kernel(const float* __restrict__ vol, const float* __restrict__ xc, float* vecs,
                       float* __restrict__ lam_out, int32_t* __restrict__ ranks, float* __restrict__ wgt,
                       float* __restrict__ sig2, Geom g, AxisTables tab, const int* __restrict__ refine_count,
                       const int* __restrict__ refine_ids) {
  eigh_refine_body(vol, xc, vecs, lam_out, ranks, wgt, sig2, g, tab, refine_count, refine_ids, (int)blockIdx.x,
                   (int)gridDim.x);
}

}  // namespace lrd
