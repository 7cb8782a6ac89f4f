// Temporal mean and centring of every voxel's time course.
//
// The ladder centres each patch's Casorati matrix with NumPy's float32 mean
// (step0_numpy_loop.py:11, ``x.mean(axis=1)``); the mean depends on the voxel
// only, so it is computed once per voxel here (step8_tuned.py:50-52 recompute
// it per patch). The sum follows NumPy's pairwise float32 summation for a
// contiguous row of n <= 128 values (8 interleaved partial sums over the
// largest multiple of 8, combined as ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)), the
// tail added in order; n < 8 summed in order from 0), added to the reduction's
// identity 0, then divided by n in float32 - bit-identical to ``x.mean``.
// The centred value is the float32 difference ``x - m`` (step0:12).
//
// Eight lanes per voxel row: lane q sums elements q, q + 8, ... in order, which is
// NumPy's partial sum r_q, and three shuffles form its combination; the tail is
// added by every lane in order. A warp's load covers a 32-byte sector of each of
// its four rows, the values stay in registers until they are centred, and nothing
// is staged. Memory bounds it: 96x96x48x48 (85 MB read, 85 MB written) 0.048 ms with
// rows staged in shared memory and a row per lane, 0.035 here; 64x64x48x96 0.062 and
// 0.032, 101x87x43x64 0.062 and 0.037.
#pragma once

#include "lrd_common.cuh"

namespace lrd {

constexpr int kCenterRows = 2;  // groups of four rows a warp has in flight
constexpr int kCenterWarps = 8;

// Rows one block of kCenterWarps warps centres.
__host__ __device__ constexpr int center_block_rows() { return 4 * kCenterRows * kCenterWarps; }

// Body of one block (index ``bid``); shared by the single-volume kernel below
// and the packed multi-volume launch (batch.cuh). The centred rows are ldx >= T
// floats apart, zero past T. N8 = ceil(T / 8).
template <int N8>
__device__ __forceinline__ void center_rows(const float* __restrict__ vol, float* __restrict__ xc,
                                            float* __restrict__ mean, long long nvox, int T, int ldx, long long bid) {
  const int lane = threadIdx.x & 31, q = lane & 7;
  const long long v0 = bid * center_block_rows() + (threadIdx.x >> 5) * (4 * kCenterRows) + (lane >> 3);
  float x[kCenterRows][N8];
#pragma unroll
  for (int u = 0; u < kCenterRows; ++u) {
    const long long v = v0 + 4 * u;
#pragma unroll
    for (int i = 0; i < N8; ++i) x[u][i] = (v < nvox && 8 * i + q < T) ? vol[v * T + 8 * i + q] : 0.f;
  }
  const int full = T >> 3, rem = T & 7;
#pragma unroll
  for (int u = 0; u < kCenterRows; ++u) {
    float r = x[u][0], tail = x[u][0];
#pragma unroll
    for (int i = 1; i < N8; ++i) {
      if (i < full) r = __fadd_rn(r, x[u][i]);
      if (i == full) tail = x[u][i];
    }
    r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));
    r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));
    r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 4));
    if (full == 0) r = 0.f;  // fewer than eight values: summed in order from 0
    for (int i = 0; i < rem; ++i) r = __fadd_rn(r, __shfl_sync(0xffffffffu, tail, i, 8));
    const float m = __fdiv_rn(__fadd_rn(0.f, r), (float)T);
    const long long v = v0 + 4 * u;
    if (v < nvox) {
      if (q == 0) mean[v] = m;
#pragma unroll
      for (int i = 0; i < N8; ++i) {
        const int t = 8 * i + q;
        if (t < ldx) xc[v * ldx + t] = t < T ? __fsub_rn(x[u][i], m) : 0.f;
      }
    }
  }
}

__device__ __forceinline__ void center_body(const float* __restrict__ vol, float* __restrict__ xc,
                                            float* __restrict__ mean, long long nvox, int T, int ldx,
                                            long long bid) {
  if (T <= 32)
    center_rows<4>(vol, xc, mean, nvox, T, ldx, bid);
  else if (T <= 48)
    center_rows<6>(vol, xc, mean, nvox, T, ldx, bid);
  else if (T <= 64)
    center_rows<8>(vol, xc, mean, nvox, T, ldx, bid);
  else if (T <= 96)
    center_rows<12>(vol, xc, mean, nvox, T, ldx, bid);
  else
    center_rows<16>(vol, xc, mean, nvox, T, ldx, bid);
}

// grid: ceil(nvox / center_block_rows()) blocks of 32 * kCenterWarps threads
__global__ void __launch_bounds__(32 * kCenterWarps)
    center_kernel(const float* __restrict__ vol, float* __restrict__ xc, float* __restrict__ mean, long long nvox,
                  int T, int ldx) {
  center_body(vol, xc, mean, nvox, T, ldx, blockIdx.x);
}

}  // namespace lrd
