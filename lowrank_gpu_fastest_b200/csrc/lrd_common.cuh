// Shared device-side types of the MP-PCA denoiser kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace lrd {

// Largest frame count the compiled kernels take (register/shared tiles are
// sized from it). The problem family spans T in 32..96.
constexpr int kMaxT = 128;

// Per-axis patch-index tables, device pointers (built by the plan).
//  corners[a][i]          corner position of axis-a index i (sorted, common.py:40-43)
//  cover[a][2*x+{0,1}]    inclusive corner-index range [lo, hi] covering voxel x
//  brick[a][2*b+{0,1}]    inclusive corner-index range touching recon brick b
struct AxisTables {
  const int32_t* corners[3];
  const int32_t* cover[3];
  const int32_t* brick[3];
};

struct Geom {
  int nx, ny, nz, nt;      // volume
  int ldx;                 // floats per voxel row of the centred volume: nt, or nt rounded up to 4 (zeros)
  int px, py, pz;          // patch
  int ncx, ncy, ncz;       // corners per axis
  long long npatch;        // ncx*ncy*ncz
  int nvox_patch;          // px*py*pz
  int bx, by, bz;          // recon brick (voxels per axis)
  int nbx, nby, nbz;       // bricks per axis
};

// Patch linear index (x-major, common.py:37-44 itertools.product order) ->
// axis corner indices.
__device__ __forceinline__ void patch_axes(const Geom& g, long long p, int& i, int& j, int& k) {
  k = (int)(p % g.ncz);
  long long r = p / g.ncz;
  j = (int)(r % g.ncy);
  i = (int)(r / g.ncy);
}

__device__ __forceinline__ long long voxel_row(const Geom& g, int x, int y, int z) {
  return ((long long)x * g.ny + y) * g.nz + z;
}

// Packed float32 arithmetic: two IEEE operations in one instruction. c += a b. (A
// mul2 may be contracted with an add2 of its result: see mul2_rn.)
__device__ __forceinline__ void fma2(float2& c, float2 a, float2 b) {
  unsigned long long ra, rb, rc;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(rc) : "l"(ra), "l"(rb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(rc));
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long ra, rb, rc;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rc) : "l"(ra), "l"(rb));
  float2 c;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(rc));
  return c;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long ra, rb, rc;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(rc) : "l"(ra), "l"(rb));
  float2 c;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(rc));
  return c;
}

// a b rounded, as a packed FMA onto -0. The assembler contracts a packed multiply and
// a packed add that follows it into one FMA, the .rn of both notwithstanding (every
// one of 13157 sampled differences to the two roundings was the fused result), so
// where both roundings count the product is formed here; ``nz`` is neg_zero(), a
// value it cannot know.
__device__ __forceinline__ float2 mul2_rn(float2 a, float2 b, float2 nz) {
  unsigned long long ra, rb, rz, rc;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rz) : "f"(nz.x), "f"(nz.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rc) : "l"(ra), "l"(rb), "l"(rz));
  float2 c;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(rc));
  return c;
}
// (the launches here are one-dimensional)
__device__ __forceinline__ float2 neg_zero() {
  const float z = __uint_as_float(0x80000000u ^ (gridDim.y - 1u));
  return make_float2(z, z);
}

// A compile-time index as an argument.
template <int V>
struct IntTag {
  static constexpr int value = V;
};

}  // namespace lrd
