// Reconstruction + weighted overlap accumulation + normalisation by warps that own
// blocks of voxels, with no block-level synchronisation.
//
// Same role and the same per-voxel arithmetic as recon_kernel (recon.cuh):
// the ladder's recon_scatter_kernel (step8_tuned.py:59-86) and final division
// (step8:144-145) with the step-0 loop's rounding (step0_numpy_loop.py:25,
// 36-39):
//
//   y_k  = (x - m) . v_k             four frame chunks, ((c0 + c1) + (c2 + c3)),
//                                    a chunk's even and odd frames summed apart
//   xd   = float32(sum_k y_k v_k) + m
//   out += float32(w) * xd,  wsum += float32(w)   (float32, x-major patch order)
//   out  = out / max(wsum, 1e-12)
//
// so its output is bit-identical to recon_kernel's for every form. What
// changes is the work decomposition, for T in {32, 48, 64, 96}:
//
//  * LPV lanes per voxel (4; 8 at T = 96), group s of lanes owning frames [sQ, sQ +
//    Q), so a voxel's y_k is its lanes' sums combined by shuffles in the chunk
//    tree's order;
//  * a lane carries two voxels (A and B, two planes apart along z; adjacent planes
//    at LPV = 8): a warp owns 2 x 2 x 4 (2 x 2 x 2) voxels. A patch that ends between
//    a lane's two voxels takes a path with one of them (at 11^3 / stride 3 a third of
//    the patches of a block);
//  * a CTA is two warps along z and walks the patches of its brick in x-major order
//    in chunks: consecutive patches along z whose rows of v_k fit a shared-memory
//    buffer, brought there by one bulk copy per patch (the p x T block is
//    contiguous) while the chunk before is used; one barrier per chunk (four warps
//    a CTA waited 17% of the time at it, 7% slower at the headline; one warp
//    6%). Ranks and weights of a chunk are loaded one per lane, a chunk ahead.
//    Read straight from global memory, a row costs a warp four clocks of the SM's
//    data path per 16 bytes a lane, whatever the lanes share, and an L1 or L2
//    latency per patch (half of all stall cycles); neighbouring lanes here belong
//    to different voxels and read the same 16 bytes, which takes two clocks;
//  * frames go through the packed FMA, add and multiply in pairs (IEEE rounding
//    each); everything that depends on T is compile-time.
//
// The float64 sums of ACCURATE take one voxel per lane (LPV = 4): 16 frames of two
// voxels would need 64 registers for the sums alone.
//
// Reconstruction phase on B200, one voxel per lane from global memory -> here: headline
// 1.10 -> 0.83 ms (accurate 1.365 -> 1.08), dense 5^3 at T = 32 1.92 -> 1.65, 7^3 at T =
// 64 2.14 -> 1.31, T = 96 1.11 -> 0.76, 128x128x64x96 / 11^3 / stride 2 17.0 -> 11.5. Per
// patch of rank 4 a warp issues about 220 instructions for two 16-voxel
// contractions of 96 packed FMAs; the FMA pipe is 44% busy, issue 52%.
//
// The brick a CTA covers is recon_warp_brick()'s in the plan's brick grid, so the
// host pipeline and slab sharding address it exactly like recon_kernel's bricks.
// Waits for the copies are bounded as in gram_z.cuh; a warp whose wait gave up also
// writes NaN.
#pragma once

#include "copy_phases.h"
#include "gram_z.cuh"  // mbarrier waits
#include "lrd_common.cuh"
#include "recon.cuh"

namespace lrd {

constexpr int kReconWarps = 2;

// Frame counts the warp kernel is built for, its lanes per voxel, voxels per lane
// and z-planes per warp.
__host__ __device__ inline bool recon_warp_supported(int T) { return T == 32 || T == 48 || T == 64 || T == 96; }
template <int T, bool ACCURATE>
__host__ __device__ constexpr int recon_warp_lanes() {
  return T == 96 && !ACCURATE ? 8 : 4;
}
template <bool ACCURATE>
__host__ __device__ constexpr int recon_warp_nv() {
  return ACCURATE ? 1 : 2;
}
template <int T, bool ACCURATE>
__host__ __device__ constexpr int recon_warp_bz() {  // 32 / LPV voxels, four per plane
  return 8 / recon_warp_lanes<T, ACCURATE>() * recon_warp_nv<ACCURATE>();
}
// The brick of a CTA.
inline void recon_warp_brick(int T, bool accurate, int b[3]) {
  b[0] = 2;
  b[1] = 2;
  b[2] = kReconWarps * (accurate ? recon_warp_bz<48, true>() : T == 96 ? recon_warp_bz<96, false>() : recon_warp_bz<48, false>());
}

// Rows of v_k a buffer holds: any patch's (p < T), except that at T = 96 a patch of
// more than 40 components is read from global memory (96 rows would leave three
// CTAs per SM instead of six). Dynamic shared memory: two buffers and their
// barriers.
template <int T>
__host__ __device__ constexpr int recon_warp_rows() {
  return T == 96 ? 40 : T < 48 ? 48 : T;
}
template <int T>
__host__ __device__ constexpr size_t recon_warp_smem_of() {
  return sizeof(float) * 2 * (size_t)recon_warp_rows<T>() * T + 2 * sizeof(uint64_t);
}
inline size_t recon_warp_smem_bytes(int T) {
  return T == 32   ? recon_warp_smem_of<32>()
         : T == 48 ? recon_warp_smem_of<48>()
         : T == 64 ? recon_warp_smem_of<64>()
                   : recon_warp_smem_of<96>();
}

// A chunk of the walk: patches (i, j, kb .. kb + cnt - 1) of the corner grid; lane q
// holds the rank and weight of patch kb + q and the rows before it in the buffer.
struct ReconChunk {
  int i, j, kb, cnt, rows;  // rows 0: nothing to copy, -1: one patch beyond the buffer
  int p, off;
  float w;
};

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// One patch (p rows of v_k at vb, this lane's frames; weight w) on the lane's voxels
// V0 .. V1; cov: it covers voxel v.
template <int T, bool ACCURATE, int V0, int V1, int NV, int Q2, int QA, int QD>
__device__ __forceinline__ void recon_patch(const float4* vb, int p, float w, const bool (&cov)[NV],
                                            const float2 (&xr)[NV][Q2], const float (&m)[NV], float2 (&acc)[NV][QA],
                                            double (&acc64)[NV][QD], float (&wacc)[NV], double (&wacc64)[NV]) {
  constexpr int LPV = recon_warp_lanes<T, ACCURATE>(), Q4 = Q2 / 2;
  // a chunk of 24 frames (T = 96) is summed in halves: at LPV = 8 they are two lanes'
  constexpr int H = Q2 == 12 ? 2 : 1;
  const float2 nz = neg_zero();
  float2 xd[NV][Q2];
  auto row = [&](int k, auto first) {  // v_k's share; the first row starts the sums
    float2 q[Q2];
#pragma unroll
    for (int u = 0; u < Q4; ++u) {
      const float4 f = vb[k * (T / 4) + u];
      q[2 * u] = make_float2(f.x, f.y);
      q[2 * u + 1] = make_float2(f.z, f.w);
    }
#pragma unroll
    for (int v = V0; v <= V1; ++v) {
      float part = 0.f;  // this lane's frames of y_k, even and odd ones in order
#pragma unroll
      for (int h = 0; h < H; ++h) {
        float2 eo = mul2(xr[v][h * (Q2 / H)], q[h * (Q2 / H)]);
#pragma unroll
        for (int u = h * (Q2 / H) + 1; u < (h + 1) * (Q2 / H); ++u) fma2(eo, xr[v][u], q[u]);
        const float hs = __fadd_rn(eo.x, eo.y);
        part = h == 0 ? hs : __fadd_rn(part, hs);
      }
#pragma unroll
      for (int o = 32 / LPV; o < 32; o <<= 1) part = __fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, o));
      const float2 pp = make_float2(part, part);
#pragma unroll
      for (int u = 0; u < Q2; ++u) {
        if (decltype(first)::value)
          xd[v][u] = mul2_rn(pp, q[u], nz);
        else
          fma2(xd[v][u], pp, q[u]);
      }
    }
  };
  if (p > 0) {
    row(0, IntTag<1>{});
#pragma unroll 2
    for (int k = 1; k < p; ++k) row(k, IntTag<0>{});
  } else {
#pragma unroll
    for (int v = V0; v <= V1; ++v)
#pragma unroll
      for (int u = 0; u < Q2; ++u) xd[v][u] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int v = V0; v <= V1; ++v)
    if (cov[v]) {
      if constexpr (ACCURATE) {
        const double wd = (double)w;
#pragma unroll
        for (int u = 0; u < Q2; ++u) {
          acc64[v][2 * u] = fma(wd, (double)xd[v][u].x, acc64[v][2 * u]);
          acc64[v][2 * u + 1] = fma(wd, (double)xd[v][u].y, acc64[v][2 * u + 1]);
        }
        wacc64[v] += wd;
      } else {
        const float2 mm = make_float2(m[v], m[v]), ww = make_float2(w, w);
#pragma unroll
        for (int u = 0; u < Q2; ++u) acc[v][u] = add2(acc[v][u], mul2_rn(ww, add2(xd[v][u], mm), nz));
        wacc[v] = __fadd_rn(wacc[v], w);
      }
    }
}

// Body of one CTA: brick brick0 + bid of the plan's brick grid.
template <int T, bool ACCURATE>
__device__ __forceinline__ void recon_warp_body(const float* __restrict__ xc, const float* __restrict__ mean,
                                                const float* __restrict__ vecs, const int32_t* __restrict__ ranks,
                                                const float* __restrict__ wgt, float* __restrict__ out,
                                                const Geom& g, const AxisTables& tab, int brick0, const SlabIO& io,
                                                int* status, int bid) {
  constexpr int LPV = recon_warp_lanes<T, ACCURATE>(), NV = recon_warp_nv<ACCURATE>();
  constexpr int Q = T / LPV, Q2 = Q / 2, Q4 = Q / 4;
  constexpr int ZS = recon_warp_bz<T, ACCURATE>() / NV;  // planes between a lane's voxels
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int s = lane / (32 / LPV);         // frames [sQ, sQ + Q)
  const int vl = lane & (32 / LPV - 1);    // voxel of the warp: z fastest, then y, x

  int brick = brick0 + bid;
  const int bzi = brick % g.nbz;
  brick /= g.nbz;
  const int byi = brick % g.nby;
  const int bxi = brick / g.nby;
  const int x = bxi * 2 + vl / (2 * ZS), y = byi * 2 + (vl / ZS) % 2;
  const int z0 = bzi * (kReconWarps * NV * ZS) + warp * (NV * ZS) + vl % ZS;
  const bool vxy = x < g.nx && y < g.ny && x >= io.x_lo && x < io.x_hi;

  // the voxels' covering corner ranges, and the warp's along z; the brick's walk
  int cxlo = 1 << 30, cxhi = -1, cylo = 1 << 30, cyhi = -1, czlo[NV], czhi[NV];
  bool valid[NV];
  if (vxy) {
    cxlo = tab.cover[0][2 * x];
    cxhi = tab.cover[0][2 * x + 1];
    cylo = tab.cover[1][2 * y];
    cyhi = tab.cover[1][2 * y + 1];
  }
  int jlo = cylo, jhi = cyhi, klo[NV], khi[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int z = z0 + v * ZS;
    valid[v] = vxy && z < g.nz;
    czlo[v] = valid[v] ? tab.cover[2][2 * z] : 1 << 30;
    czhi[v] = valid[v] ? tab.cover[2][2 * z + 1] : -1;
    klo[v] = czlo[v];
    khi[v] = czhi[v];
  }
#pragma unroll
  for (int o = 1; o < 32 / LPV; o <<= 1) {  // lanes of one voxel hold the same ranges
    jlo = min(jlo, __shfl_xor_sync(0xffffffffu, jlo, o));
    jhi = max(jhi, __shfl_xor_sync(0xffffffffu, jhi, o));
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      klo[v] = min(klo[v], __shfl_xor_sync(0xffffffffu, klo[v], o));
      khi[v] = max(khi[v], __shfl_xor_sync(0xffffffffu, khi[v], o));
    }
  }
  const int bilo = tab.brick[0][2 * bxi], bihi = tab.brick[0][2 * bxi + 1];
  const int bjlo = tab.brick[1][2 * byi], bjhi = tab.brick[1][2 * byi + 1];
  const int bklo = tab.brick[2][2 * bzi], bkhi = tab.brick[2][2 * bzi + 1];

  // centred frames of this lane, temporal mean, running sums
  const long long row0 = vxy ? voxel_row(g, x, y, z0) : 0;
  float2 xr[NV][Q2];
  float2 acc[NV][ACCURATE ? 1 : Q2];
  double acc64[NV][ACCURATE ? Q : 1];
  float m[NV], wacc[NV];
  double wacc64[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const long long row = row0 + v * ZS;
    const float4* xp = reinterpret_cast<const float4*>(xc + row * T + s * Q);
#pragma unroll
    for (int u = 0; u < Q4; ++u) {
      const float4 f = valid[v] ? xp[u] : make_float4(0.f, 0.f, 0.f, 0.f);
      xr[v][2 * u] = make_float2(f.x, f.y);
      xr[v][2 * u + 1] = make_float2(f.z, f.w);
    }
    m[v] = valid[v] ? mean[row] : 0.f;
    wacc[v] = 0.f;
    wacc64[v] = 0.0;
    const bool cont = valid[v] && x < io.hin && io.halo_in != nullptr;  // continue a lower slab's sums
    const double* hp = cont ? io.halo_in + row * (T + 1) : nullptr;
#pragma unroll
    for (int u = 0; u < Q2; ++u) {
      const double h0 = cont ? hp[s * Q + 2 * u] : 0.0, h1 = cont ? hp[s * Q + 2 * u + 1] : 0.0;
      if constexpr (ACCURATE) {
        acc64[v][2 * u] = h0;
        acc64[v][2 * u + 1] = h1;
      } else {
        acc[v][u] = make_float2((float)h0, (float)h1);
      }
    }
    if (cont) {
      wacc64[v] = hp[T];
      wacc[v] = (float)hp[T];
    }
  }

  // ---- the walk ----------------------------------------------------------------
  extern __shared__ __align__(128) float sm_rw[];
  constexpr int ROWS = recon_warp_rows<T>();
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm_rw + 2 * (size_t)ROWS * T);
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars), buf0 = (uint32_t)__cvta_generic_to_shared(sm_rw);
  if (threadIdx.x == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar0 + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  auto fetch = [&](ReconChunk& c) {  // its ranks and weights, as far as the z-run and the lanes go
    const bool in = c.i <= bihi && c.kb + lane <= bkhi;
    const long long pid = ((long long)c.i * g.ncy + c.j) * g.ncz + c.kb + lane;
    c.p = in ? __ldg(ranks + pid) : 0;
    c.w = in ? __ldg(wgt + pid) : 0.f;
  };
  auto size = [&](ReconChunk& c) {  // how many of them fit the buffer, and where
    int inc = c.p;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    c.off = inc - c.p;
    c.cnt = c.i <= bihi ? __popc(__ballot_sync(0xffffffffu, inc <= ROWS && c.kb + lane <= bkhi)) : 0;
    c.rows = c.cnt > 0 ? __shfl_sync(0xffffffffu, inc, c.cnt - 1) : 0;
    if (c.cnt == 0 && c.i <= bihi) {
      c.cnt = 1;
      c.rows = -1;
    }
  };
  auto after = [&](const ReconChunk& c) {  // where the next chunk starts
    ReconChunk n = c;
    n.kb = c.kb + c.cnt;
    if (n.kb > bkhi) {
      n.kb = bklo;
      if (++n.j > bjhi) {
        n.j = bjlo;
        ++n.i;
      }
    }
    return n;
  };
  CopyPhases ph;
  auto copy = [&](const ReconChunk& c, int b) {  // warp 0: the chunk's rows into buffer b
    if (c.rows <= 0 || !ph.ok) return;
    if (lane == 0) {
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      mbar_expect_tx(bar0 + 8 * b, (uint32_t)(c.rows * T * sizeof(float)));
    }
    __syncwarp();
    if (lane < c.cnt && c.p > 0) {
      const long long pid = ((long long)c.i * g.ncy + c.j) * g.ncz + c.kb + lane;
      bulk_copy(buf0 + (uint32_t)((b * ROWS + c.off) * T * sizeof(float)), vecs + pid * (T * T),
                (uint32_t)(c.p * T * sizeof(float)), bar0 + 8 * b);
    }
    ph.issued(b);
  };
  const bool none = bihi < bilo || bjhi < bjlo || bkhi < bklo;  // a brick no patch touches
  ReconChunk cur{none ? bihi + 1 : bilo, bjlo, bklo, 0, 0, 0, 0, 0.f}, nxt;
  fetch(cur);
  size(cur);
  __syncthreads();  // the barriers are initialised
  if (warp == 0) copy(cur, 0);
  nxt = after(cur);
  fetch(nxt);
  for (int b = 0; cur.cnt > 0; b ^= 1) {
    size(nxt);
    __syncthreads();  // every warp is done with the other buffer
    if (warp == 0) copy(nxt, b ^ 1);
    ReconChunk then = after(nxt);
    fetch(then);
    if (cur.rows > 0 && ph.ok)
      ph.waited(b, __all_sync(0xffffffffu, mbar_wait_bounded(bar0 + 8 * b, ph.parity(b), status)));
    if (cur.j >= jlo && cur.j <= jhi) {  // (a warp's two x are the brick's)
      const bool cxy = cur.i >= cxlo && cur.i <= cxhi && cur.j >= cylo && cur.j <= cyhi;
      if (cur.rows < 0) {  // its rows straight from global memory
        const long long pid = ((long long)cur.i * g.ncy + cur.j) * g.ncz + cur.kb;
        bool cov[NV], any = false;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          cov[v] = cxy && cur.kb >= czlo[v] && cur.kb <= czhi[v];
          any |= cov[v];
        }
        if (__any_sync(0xffffffffu, any))
          recon_patch<T, ACCURATE, 0, NV - 1>(reinterpret_cast<const float4*>(vecs + pid * (T * T)) + s * Q4,
                                              __shfl_sync(0xffffffffu, cur.p, 0), __shfl_sync(0xffffffffu, cur.w, 0),
                                              cov, xr, m, acc, acc64, wacc, wacc64);
        cur = nxt;
        nxt = then;
        continue;
      }
      const float4* vs = reinterpret_cast<const float4*>(sm_rw + (size_t)b * ROWS * T) + s * Q4;
      // along z first the patches that reach voxel A's planes only, then both
      // voxels', then voxel B's only (the corners of a run increase)
      auto segment = [&](auto v0, auto v1, int from, int to) {
        for (int k = max(from, cur.kb); k <= min(to, cur.kb + cur.cnt - 1); ++k) {
          const int q = k - cur.kb;
          const int p = __shfl_sync(0xffffffffu, cur.p, q), off = __shfl_sync(0xffffffffu, cur.off, q);
          const float w = __shfl_sync(0xffffffffu, cur.w, q);
          bool cov[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) cov[v] = cxy && k >= czlo[v] && k <= czhi[v];
          recon_patch<T, ACCURATE, decltype(v0)::value, decltype(v1)::value>(vs + off * (T / 4), p, w, cov, xr, m, acc,
                                                                             acc64, wacc, wacc64);
        }
      };
      if (NV == 1) {
        segment(IntTag<0>{}, IntTag<0>{}, klo[0], khi[0]);
      } else {
        segment(IntTag<0>{}, IntTag<0>{}, klo[0], min(khi[0], klo[NV - 1] - 1));
        segment(IntTag<0>{}, IntTag<NV - 1>{}, klo[NV - 1], khi[0]);
        segment(IntTag<NV - 1>{}, IntTag<NV - 1>{}, max(klo[NV - 1], khi[0] + 1), khi[NV - 1]);
      }
    }
    cur = nxt;
    nxt = then;
  }
  // a wait of warp 0 gave up: its copies still in flight land (or time out) before
  // the CTA's shared memory is freed
  if (warp == 0 && lane == 0 && !ph.ok)
    for (int b = 0; b < 2; ++b)
      if (ph.in_flight(b)) mbar_wait_bounded(bar0 + 8 * b, ph.parity(b), status);

#pragma unroll
  for (int v = 0; v < NV; ++v) {
    if (!valid[v]) continue;
    if (!ph.ok) {  // rows that never came: no caller can take the result for one
      m[v] = wacc[v] = __int_as_float(0x7fffffff);
      wacc64[v] = (double)m[v];
    }
    const long long row = row0 + v * ZS;
    if (x >= io.own_hi) {  // the next slab's halo: unnormalised sums in patch order
      double* hp = io.halo_out + (row - (long long)io.own_hi * g.ny * g.nz) * (T + 1);
#pragma unroll
      for (int u = 0; u < Q; ++u) {
        if constexpr (ACCURATE)
          hp[s * Q + u] = acc64[v][u];
        else
          hp[s * Q + u] = (double)((u & 1) ? acc[v][u / 2].y : acc[v][u / 2].x);
      }
      if (s == 0) hp[T] = ACCURATE ? wacc64[v] : (double)wacc[v];
      continue;
    }
    float4* op = reinterpret_cast<float4*>(out + row * T + s * Q);
    if constexpr (ACCURATE) {
      // a voxel no patch covers (stride > patch side) gets 0, as 0 / max(0, 1e-12)
      // does in the ladder
      const double inv = wacc64[v] == 0.0 ? 0.0 : 1.0 / wacc64[v];
      const double mm = wacc64[v] == 0.0 ? 0.0 : (double)m[v];
#pragma unroll
      for (int u = 0; u < Q4; ++u)
        op[u] = make_float4((float)(mm + acc64[v][4 * u + 0] * inv), (float)(mm + acc64[v][4 * u + 1] * inv),
                            (float)(mm + acc64[v][4 * u + 2] * inv), (float)(mm + acc64[v][4 * u + 3] * inv));
    } else {
      const float den = ph.ok ? fmaxf(wacc[v], 1e-12f) : wacc[v];
#pragma unroll
      for (int u = 0; u < Q4; ++u)
        op[u] = make_float4(__fdiv_rn(acc[v][2 * u].x, den), __fdiv_rn(acc[v][2 * u].y, den),
                            __fdiv_rn(acc[v][2 * u + 1].x, den), __fdiv_rn(acc[v][2 * u + 1].y, den));
    }
  }
}

// CTAs per SM, which cap the registers. Reconstruction phase on B200, ms with 6 / 8 /
// 10, at 96x96x48xT / 11^3 / stride 3 and 64x64x32xT / 5^3 / stride 1:
//   T = 32  plain 0.735 / 0.651 / 0.670, 0.781 / 0.705 / 0.733 (372416 patches of 5^3 1.94 / 1.68 / 1.65)
//           accurate 0.904 / 0.930 / 0.858, 0.840 / 0.865 / 0.815
//   T = 48  plain 0.867 / 0.835 / 1.30, 0.924 / 0.890 / 1.32; accurate 1.23 / 1.08 / 1.14, 1.14 / 1.02 / 1.03
//   T = 64  plain 1.07 / 2.57 / 3.05 (spills), 1.11 / 2.49 / 3.08; accurate 1.45 / 1.47 / 3.58, 1.35 / 1.37 / 3.05
//   T = 96  plain 1.65 / 1.92 / 3.64, 1.47 / 1.65 / 3.13; accurate 1.85 / 3.67 / 4.24, 1.73 / 3.34 / 3.96
// and at 80x70x40xT / 7^3 / 2 and 64x64x40xT / 11^3 / 2 alike.
template <int T, bool ACCURATE>
__host__ __device__ constexpr int recon_warp_ctas() {
  return T == 32 ? 10 : T == 48 ? 8 : 6;
}

template <int T, bool ACCURATE>
__global__ void __launch_bounds__(32 * kReconWarps, recon_warp_ctas<T, ACCURATE>())
    recon_warp_kernel(const float* __restrict__ xc, const float* __restrict__ mean, const float* __restrict__ vecs,
                      const int32_t* __restrict__ ranks, const float* __restrict__ wgt, float* __restrict__ out,
                      Geom g, AxisTables tab, int brick0, SlabIO io, int* status) {
  recon_warp_body<T, ACCURATE>(xc, mean, vecs, ranks, wgt, out, g, tab, brick0, io, status, (int)blockIdx.x);
}

}  // namespace lrd
