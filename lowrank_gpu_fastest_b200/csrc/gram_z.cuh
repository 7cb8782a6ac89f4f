// Per-patch Gram matrices with the z-planes of a patch column shared.
//
// All patches with the same (x, y) corners form a column along z. Their Gram
// matrices G(cz) = sum_{z = cz}^{cz + pz - 1} H(z) are sums of the same
// per-plane Grams H(z) = sum over the px*py voxels of plane z of xc xc^T.
// gram_kernel recomputes every H(z) for each of the ~pz/stride windows that
// contain z; this kernel computes each H(z) once and adds it into every active
// window, which cuts the FFMA work by that factor (3.2x at 11^3 / stride 3).
//
// Layout: one CTA per (x-corner, y-corner) column; KS lanes of a warp share an
// 8 x 8 block of the upper block triangle, each summing every KS-th voxel row.
// The column's planes are streamed into a two-slot shared-memory ring by TMA (one
// 4D box (T, 1, py, px) of the centred volume per plane, completion on an
// mbarrier); the window accumulators of the active windows live in shared memory
// (a ring of ``ring`` slots, slot = window index mod ring).
//
// A 4 x 4 block reads 2 bytes of shared memory per FMA, and LDS.128 returns 128
// bytes a clock to an SM's 128 FMA lanes: that bound the kernel (77% of the shared
// data pipe, 38% of the FMA pipe). An 8 x 8 block reads 1 byte per FMA. The packed
// FMA (two IEEE FMAs) halves the issue slots: 107 instead of 94 FMA a clock at 12
// warps per SM in a loop of nothing else. What bounds it now is 9 to 12 warps per
// SM that stop at the plane barrier and at the flush below. Gram phase on B200:
// 96x96x48x48 / 11^3 / stride 3 0.61 -> 0.53 ms, 96x96x48x32 / 5^3 / stride 1 1.58
// -> 1.43, 101x87x43x64 / 7^3 / stride 2 1.21 -> 1.00, 64x64x48x96 / 11^3 / stride 3
// 0.99 -> 0.70; 128x128x64x96 / 11^3 / stride 2, whose ring of six windows (208 KB) passed
// the kernel's former limit of 200 KB and which ran a CTA per patch, 68.1 -> 10.4.
//
// Planes that lie in the same windows (two of three at 11^3 / stride 3) are summed
// in registers, at most gramz_group() of them; at the last the KS lanes' partial sums are
// combined by halving exchanges and added to the windows in float32, and a window is
// written out (and its slot cleared) after its last plane. The K = px*py*pz sum
// therefore rounds as a blocked sum: rows of a plane group, lanes, window.
// A frame count that is not a multiple of 4 has the rows of its centred volume padded
// to one with zeros (TMA strides are multiples of 16 bytes), and its windows add
// without rounding (gramz_exact): with a CTA per patch 61x53x37x65 / 7^3 / stride 2
// 1.49 ms, 0.61 here (0.39 with windows rounded at each plane, but 4% further from
// the float64 Gram at T = 17 and 31); 40x40x32x127 2.15 and 0.71.
// Tried and dropped (headline ms): a producer warp with chunks of x-rows and no
// CTA barrier 0.59 (its warp leaves one of the SM's four schedulers idle), the
// same with thread 0 of the first warp as producer 0.63, the next row's loads
// moved ahead of this row's products by hand 0.81.
//
// Every mbarrier wait is bounded by a %globaltimer deadline. On expiry the
// kernel records LRD_STATUS_TMA_TIMEOUT in the status word (the result is
// then invalid and the host reports it), issues no further copy, and the
// issuing thread waits - with the same bound - for the copies it still has in
// flight into the CTA's shared memory before the CTA exits.
#pragma once

#include <cuda.h>

#include "lrd_common.cuh"

namespace lrd {

constexpr int kStatusTmaTimeout = 1;
constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s per wait

__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}

// Bounded wait for the phase with parity ``parity`` to complete; after
// ``limit_ns`` ``code`` is or-ed into the status word and the wait gives up.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, int* status,
                                                  int code = kStatusTmaTimeout,
                                                  unsigned long long limit_ns = kWaitNs) {
  unsigned long long t0 = 0;  // the clock is read only once the first try has failed
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (t0 == 0) {
      t0 = globaltimer_ns();
    } else if (globaltimer_ns() - t0 > limit_ns) {
      atomicOr(status, code);
      return false;
    }
  }
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];\n" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}

__host__ __device__ inline size_t gramz_plane_floats(int rows, int T) {
  return ((size_t)rows * T + 31) & ~size_t(31);  // 128-byte multiple
}

// 8 x 8 blocks of the upper block triangle: block b of nb = ceil(T / 8) owns the
// 4-frame quads b and b + nb (the second one absent at the end of an odd count).
__host__ __device__ inline int gramz_nb(int T) { return (((T + 3) >> 2) + 1) >> 1; }
__host__ __device__ inline int gramz_nblk(int T) {
  const int nb = gramz_nb(T);
  return nb * (nb + 1) / 2;
}

// Whether the windows add their planes without rounding (a high and a low word): the
// frame counts that are not a multiple of 4, which a CTA per patch summed over planes
// in float64 before their rows were padded for this kernel.
__host__ __device__ inline bool gramz_exact(int T) { return (T & 3) != 0; }

// CTAs that share a column's blocks: two for the 136 blocks of T > 120, which four
// lanes each would make 17 warps of 128 registers (two lanes each sum 61 rows of an
// 11 x 11 plane one after the other: 11^3 / stride 2 / T = 128 6.2e-8 of the Gram
// off against 5.5e-8).
__host__ __device__ inline int gramz_shares(int T, int ks) { return ks >= 4 && gramz_nblk(T) > 128 ? 2 : 1; }
__host__ __device__ inline int gramz_cta_blocks(int T, int ks) {
  return gramz_nblk(T) / gramz_shares(T, ks);  // (136 or a share of one)
}

// Threads of a column CTA for T frames and K-split ks: its blocks, 32 / ks to a
// warp, times ks.
__host__ __device__ inline int gramz_threads(int T, int ks) {
  const int per_warp = 32 / ks;
  return 32 * ((gramz_cta_blocks(T, ks) + per_warp - 1) / per_warp);
}

// Planes of a group, so that a lane's chain of additions has an end: without a limit a
// patch that no window cuts (stride at or beyond its side, a volume one patch deep) was
// one chain, and the Gram twice as far from float64. Relative error of the Gram (random
// centred rows, rms, over that of planes summed one by one with half as many lanes a
// block; windows in float64 where they carry two words here) without a limit and with 2
// / 3 / 4 planes: stride = side, 11^3 at T = 48 1.26, 0.78 / 0.76 / 0.69, T = 64 2.04, 0.75 / 0.79 /
// 0.80, T = 96 2.03, 0.73 / 0.79 / 0.80, T = 65 2.65, 0.69 / 0.86 / 1.06; 7^3 at T = 64 1.23, 0.79 /
// 0.88 / 0.84, T = 31 1.75, 0.80 / 0.98 / 1.15; 15^3 at T = 96 2.72, 0.69 / 0.79 / 0.82; two lanes a
// block, 11^3 at T = 64 3.76, 0.89 / 1.15 / 1.25. A flush has its price (Gram ms without a
// limit, and with 2 / 3 / 4): 96x96x48x48 / 11^3 / stride 3 0.528, 0.553 / 0.530 / 0.530 (groups
// of one and two planes, three at the volume's ends), stride 11 0.072, 0.083 / 0.078 / 0.076.
template <int KS, bool EXACT>
__host__ __device__ constexpr int gramz_group() {
  return EXACT || KS == 2 ? 2 : 3;
}

// Dynamic shared memory: two plane slots, ``ring`` window accumulators (64 floats
// per block, twice that where they carry their rounding errors), two mbarriers.
__host__ __device__ inline size_t gramz_smem_bytes(int px, int py, int T, int ks, int ring) {
  return sizeof(float) * (2 * gramz_plane_floats(px * py, (T + 3) & ~3) +
                          (size_t)ring * (gramz_exact(T) ? 128 : 64) * gramz_cta_blocks(T, ks)) +
         2 * sizeof(uint64_t);
}

// (hi, lo) += x: Knuth's two-sum, its error into lo.
__device__ __forceinline__ void add_exact(float& hi, float& lo, float x) {
  const float s = __fadd_rn(hi, x), b = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
  hi = s;
}

// (an overflowed sum's error term is a NaN)
__device__ __forceinline__ float joined(float hi, float lo) { return lo == lo ? __fadd_rn(hi, lo) : hi; }

// grid: gramz_shares(T, KS) CTAs, neighbours, for each of nfull + (columns - nfull) *
// nsplit units; block: gramz_threads(T, KS)
// (KS in {2, 4, 8}; voxel rows of ldx = 4 ceil(T / 4) floats). Unit b < nfull computes every window of column
// col0 + b; the columns after the first nfull are each cut into nsplit units
// of consecutive windows (a unit reads only the planes of its windows; it needs
// min(windows active at a plane, windows of the unit) <= ring), so a launch
// whose last wave would hold a few whole columns spreads that tail over many
// SMs, and a ring that does not fit shared memory is cut to one that does. The
// planes are grouped by the column's windows, not the unit's, and a unit starts and
// ends with a group, so the result does not depend on the cut. ``col0`` = first column (x-major index
// ci * ncy + cj); ``gram`` points at the Gram block of the launch's first
// patch (patch index col0 * ncz).
// Body of one CTA (index ``cta``); ``xmap`` points at the tensor map (a kernel
// parameter, or a 64-byte aligned copy in global memory for the packed
// multi-volume launch).
template <int KS, bool EXACT>
__device__ __forceinline__ void gram_z_body(const CUtensorMap* xmap, float* __restrict__ gram, const Geom& g,
                                            const AxisTables& tab, long long col0, int ring, int nfull, int nsplit,
                                            int* status, int cta) {
  static_assert(KS == 2 || KS == 4 || KS == 8, "threads per block");
  constexpr int BW = 32 / KS;  // blocks per warp: lane = kq * BW + block
  constexpr int NR = 8 / KS;   // rows of its block a thread ends up with: kq * NR ...
  extern __shared__ __align__(128) float smz[];
  const int T = g.nt, ldx = EXACT ? (T + 3) & ~3 : T;  // (g.ldx)
  const int rows = g.px * g.py;
  const size_t pf = gramz_plane_floats(rows, ldx);
  const int nq = ldx >> 2, nb = gramz_nb(T);
  // this CTA's blocks (of two, 68 each)
  const int shares = gramz_shares(T, KS), nblk = gramz_nblk(T) / shares;
  const int bid = shares == 2 ? cta >> 1 : cta, blk0 = shares == 2 ? (cta & 1) * nblk : 0;
  const int nthreads = blockDim.x;
  const int nown = nblk * KS;                             // threads that own a share of a block
  constexpr int SLOT = EXACT ? 32 : 16;  // float4s of a window per block
  float4* win = reinterpret_cast<float4*>(smz + 2 * pf);  // [ring][high(, low)][2 NR][nown]
  uint64_t* bars = reinterpret_cast<uint64_t*>(win + (size_t)ring * SLOT * nblk);
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(bars);

  // this CTA's column and windows [wlo, whi]
  const bool cut = bid >= nfull;
  const int u0 = cut ? bid - nfull : 0, nparts = cut ? nsplit : 1, part = u0 % nparts;
  const long long col = col0 + (cut ? nfull + u0 / nparts : bid);
  const int wlo = part * g.ncz / nparts, whi = (part + 1) * g.ncz / nparts - 1;
  const int zlo = tab.corners[2][wlo], zhi = tab.corners[2][whi] + g.pz - 1;  // its planes
  const int ci = (int)(col / g.ncy), cj = (int)(col % g.ncy);
  const int cx = tab.corners[0][ci], cy = tab.corners[1][cj];
  const int tid = threadIdx.x, lane = tid & 31;
  const int kq = lane / BW, blk = (tid >> 5) * BW + (lane & (BW - 1));
  const bool owner = blk < nblk;
  int bi = 0, bj = 0;
  if (owner) {
    int rem = blk0 + blk;
    while (rem >= nb - bi) {
      rem -= nb - bi;
      ++bi;
    }
    bj = bi + rem;
  }
  // quads of the block's rows and columns (an absent one reads the last quad;
  // what comes of it is not stored)
  const int qa0 = bi, qa1 = min(bi + nb, nq - 1), qb0 = bj, qb1 = min(bj + nb, nq - 1);
  const uint32_t plane_bytes = (uint32_t)(rows * ldx * sizeof(float));
  auto fetch = [&](int z, int slot) {  // plane z into a slot that nothing reads or fills
    mbar_expect_tx(bar0 + 8 * slot, plane_bytes);
    tma_load_4d((uint32_t)__cvta_generic_to_shared(smz + slot * pf), xmap, bar0 + 8 * slot, 0, z, cy, cx);
  };

  for (int e = tid; e < ring * SLOT * nblk; e += nthreads) win[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tid == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar0 + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (tid == 0 && zlo <= zhi) fetch(zlo, 0);
  float* G0 = gram + (size_t)((col - col0) * g.ncz) * T * T;
  // rows of G take float4 (a caller's block may not be aligned)
  const bool aligned = !EXACT && (reinterpret_cast<uintptr_t>(gram) & 15) == 0;
  float2 acc[8][4];  // row u of the block, column pairs
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = make_float2(0.f, 0.f);
  int nlo = tab.cover[2][2 * zlo], nhi = tab.cover[2][2 * zlo + 1];
  int held = 0;  // planes summed in acc
  for (int z = zlo; z <= zhi; ++z) {
    const int slot = (z - zlo) & 1;
    // Each slot's barrier has at most one phase pending: plane z + 1 goes into
    // the slot whose previous plane (z - 1) every thread waited for in full.
    if (tid == 0 && z < zhi) {
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      fetch(z + 1, slot ^ 1);
    }
    // the column's windows holding plane z, and this unit's among them; the next
    // plane's are fetched here
    const int clo = nlo, chi = nhi;
    if (z < zhi) {
      nlo = tab.cover[2][2 * z + 2];
      nhi = tab.cover[2][2 * z + 3];
    }
    const int klo = max(clo, wlo), khi = min(chi, whi);
    const uint32_t parity = ((z - zlo) >> 1) & 1;
    const bool ok = mbar_wait_bounded(bar0 + 8 * slot, parity, status);
    if (klo <= khi) {
      const float4* row = reinterpret_cast<const float4*>(smz + slot * pf) + kq * nq;
      auto add_row = [&]() {
        const float4 a0 = row[qa0], a1 = row[qa1], b0 = row[qb0], b1 = row[qb1];
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const float2 bv[4] = {{b0.x, b0.y}, {b0.z, b0.w}, {b1.x, b1.y}, {b1.z, b1.w}};
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) fma2(acc[u][v], make_float2(av[u], av[u]), bv[v]);
        row += KS * nq;
      };
      // (the same number of rows for every lane, then the remainder)
#pragma unroll 2
      for (int i = rows / KS; i > 0; --i) add_row();
      if (kq < rows % KS) add_row();
    }
    // this slot is refilled by the copy issued at the start of the next iteration
    if (__syncthreads_or(!ok)) {
      // A wait gave up: nothing more is issued; thread 0 waits (bounded) for the
      // copies still in flight - this plane if its own wait gave up, and the next -
      // so that none lands after the CTA's shared memory is freed.
      if (tid == 0) {
        if (!ok) mbar_wait_bounded(bar0 + 8 * slot, parity, status);
        if (z < zhi) mbar_wait_bounded(bar0 + 8 * (slot ^ 1), ((z + 1 - zlo) >> 1) & 1, status);
      }
      return;
    }
    if (klo > khi) continue;
    // Planes in the same windows are summed together, up to gramz_group(); the sum goes
    // to the windows at the last of them (a window starts and ends at such a break).
    if (++held < gramz_group<KS, EXACT>() && z < zhi && nlo == clo && nhi == chi) continue;
    held = 0;
    // halving exchanges over the KS lanes of a block: each step a lane keeps half
    // of its rows and adds its partner's copies of them
    float2 mine[NR][4];
    {
      float2 h4[4][4], h2[2][4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const bool hi = kq >= KS / 2;
          const float2 keep = hi ? acc[u + 4][v] : acc[u][v], send = hi ? acc[u][v] : acc[u + 4][v];
          h4[u][v].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 16);
          h4[u][v].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 16);
        }
      if constexpr (KS == 2) {
#pragma unroll
        for (int u = 0; u < NR; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) mine[u][v] = h4[u][v];
      } else {
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const bool hi = (lane >> 3) & 1;
            const float2 keep = hi ? h4[u + 2][v] : h4[u][v], send = hi ? h4[u][v] : h4[u + 2][v];
            h2[u][v].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 8);
            h2[u][v].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 8);
          }
        if constexpr (KS == 4) {
#pragma unroll
          for (int u = 0; u < NR; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) mine[u][v] = h2[u][v];
        } else {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const bool hi = (lane >> 2) & 1;
            const float2 keep = hi ? h2[1][v] : h2[0][v], send = hi ? h2[0][v] : h2[1][v];
            mine[0][v].x = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 4);
            mine[0][v].y = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 4);
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = make_float2(0.f, 0.f);
    if (!owner) continue;
    // Windows are consecutive and their corners increase, so only the lowest
    // window holding plane z (klo) can end at z.
    const bool klo_ends = z == tab.corners[2][klo] + g.pz - 1;
    int wslot = klo % ring;
    for (int k = klo; k <= khi; ++k) {
      float4* w = win + (size_t)wslot * SLOT * nblk + kq * nblk + blk;
      const bool ends = k == klo && klo_ends;
      float* G = G0 + (size_t)k * T * T;
#pragma unroll
      for (int u = 0; u < NR; ++u)
#pragma unroll
        for (int cq = 0; cq < 2; ++cq) {  // the row's two column quads
          float4 v = w[(2 * u + cq) * nown];
          if constexpr (EXACT) {
            float4& low = w[(2 * (NR + u) + cq) * nown];
            float4 l = low;
            add_exact(v.x, l.x, mine[u][2 * cq].x);
            add_exact(v.y, l.y, mine[u][2 * cq].y);
            add_exact(v.z, l.z, mine[u][2 * cq + 1].x);
            add_exact(v.w, l.w, mine[u][2 * cq + 1].y);
            low = ends ? make_float4(0.f, 0.f, 0.f, 0.f) : l;
            w[(2 * u + cq) * nown] = ends ? make_float4(0.f, 0.f, 0.f, 0.f) : v;
            v = make_float4(joined(v.x, l.x), joined(v.y, l.y), joined(v.z, l.z), joined(v.w, l.w));
          } else {
            v.x += mine[u][2 * cq].x;
            v.y += mine[u][2 * cq].y;
            v.z += mine[u][2 * cq + 1].x;
            v.w += mine[u][2 * cq + 1].y;
            w[(2 * u + cq) * nown] = ends ? make_float4(0.f, 0.f, 0.f, 0.f) : v;
          }
          const int ub = kq * NR + u;  // row of the block
          const int fr = ub < 4 ? 4 * bi + ub : 4 * (bi + nb) + ub - 4, qc = cq ? bj + nb : bj;
          if (ends && fr < T && qc < nq) {
            float* gr = G + (size_t)fr * T + 4 * qc;
            if (aligned) {
              *reinterpret_cast<float4*>(gr) = v;
            } else {
              const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (!EXACT || 4 * qc + i < T) gr[i] = vs[i];
            }
            if (bi != bj) {
              float* gc = G + (size_t)(4 * qc) * T + fr;
              const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int i = 0; i < 4; ++i)
                if (!EXACT || 4 * qc + i < T) gc[i * (size_t)T] = vs[i];
            }
          }
        }
      if (++wslot == ring) wslot = 0;
    }
  }
}

// (KS = 4 needs at most 480 threads, KS = 2 288; KS = 8 runs up to T = 80)
constexpr int kGramzMaxThreads = 512;

template <int KS, bool EXACT>
__global__ void __maxnreg__(128)
    gram_z_kernel(const __grid_constant__ CUtensorMap xmap, float* __restrict__ gram, Geom g, AxisTables tab,
                  long long col0, int ring, int nfull, int nsplit, int* status) {
  gram_z_body<KS, EXACT>(&xmap, gram, g, tab, col0, ring, nfull, nsplit, status, (int)blockIdx.x);
}

// Self-test of the bounded wait: one thread waits on a freshly initialised
// mbarrier that nothing arrives at, gives up after ``limit_ns`` and records
// ``code`` in ``status``; no copy or MMA is in flight, so the kernel simply
// returns. grid 1, block 32.
__global__ void wait_timeout_selftest_kernel(int* status, unsigned long long limit_ns, int code) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    const uint32_t b = (uint32_t)__cvta_generic_to_shared(&bar);
    mbar_init(b, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    mbar_wait_bounded(b, 0, status, code, limit_ns);
  }
}

}  // namespace lrd
