// Insertion of slice values into the interleaved (model, weight) accumulators,
// shared by the compress kernels.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "fixed.cuh"
#include "tc.cuh"
#include "voxel.h"

namespace emc {

namespace {

// (model, weight) += (x, y) at one voxel as a single vector reduction.
__device__ __forceinline__ void red_add_v2(float2* p, float x, float y) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}
// The same at two neighbouring voxels; p is 16-byte aligned.
__device__ __forceinline__ void red_add_v4(float2* p, float x0, float y0, float x1, float y1) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x0), "f"(y0), "f"(x1),
               "f"(y1)
               : "memory");
}

// The copy that rotation r adds to.
__device__ __forceinline__ InsertAcc acc_copy(const InsertAcc& a, int64_t r) {
  const int64_t o = (r & (a.copies - 1)) * a.stride;
  return InsertAcc{a.acc + o, a.odd ? a.odd + o : nullptr, a.acc64, a.stride, a.copies};
}

__device__ __forceinline__ void insert_add(const InsertAcc& a, int vox, float x, float y) {
  if (a.acc64) {
    add_fixed(a.acc64 + 8 * (int64_t)vox, x);
    add_fixed(a.acc64 + 8 * (int64_t)vox + 4, y);
  } else {
    red_add_v2(a.acc + vox, x, y);
  }
}

__device__ __forceinline__ void insert_nearest(const InsertAcc& a, const float* u, int side,
                                               float val, float wT) {
  int vox;
  if (emc_voxel::nearest32(u, side, 0, &vox)) insert_add(a, vox, val, wT);
}

// The eight corners of u with their weights (those of trilinear_corner, the
// same products in the same order).  The two corners along x are neighbours in
// memory, so a pair is one 16-byte reduction: the L2 takes reductions by the
// request, and this halves them (the list compress of 11,000 patterns x 36,540
// rotations at 96^3: 9.4 -> 5.5 ms).
__device__ __forceinline__ void insert_trilinear(const InsertAcc& a, const float* u, int side,
                                                 float val, float wT) {
  const float fx = floorf(u[0]), fy = floorf(u[1]), fz = floorf(u[2]);
  const int x0 = (int)fx, y0 = (int)fy, z0 = (int)fz;
  const float ax = u[0] - fx, ay = u[1] - fy, az = u[2] - fz;
  const bool lo = x0 >= 0 && x0 < side, hi = x0 >= -1 && x0 < side - 1;
  if (!(lo || hi)) return;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int by = c & 1, bz = c >> 1, ky = y0 + by, kz = z0 + bz;
    if (ky < 0 || ky >= side || kz < 0 || kz >= side) continue;
    const float wy = by ? ay : 1.0f - ay, wz = bz ? az : 1.0f - az;
    const float w0 = (1.0f - ax) * wy * wz, w1 = ax * wy * wz;
    const int v = (kz * side + ky) * side + x0;
    if (lo && hi && a.odd && w0 != 0.0f && w1 != 0.0f) {
      red_add_v4((v & 1) ? a.odd + v + 1 : a.acc + v, w0 * val, w0 * wT, w1 * val, w1 * wT);
    } else {
      if (lo && w0 != 0.0f) insert_add(a, v, w0 * val, w0 * wT);
      if (hi && w1 != 0.0f) insert_add(a, v + 1, w1 * val, w1 * wT);
    }
  }
}

}  // namespace
}  // namespace emc
