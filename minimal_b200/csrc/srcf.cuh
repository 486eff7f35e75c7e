// FP32 sources of the mixed form (leaf-relative bodies).
#pragma once
#include <cuda_runtime.h>

namespace fmm {

// The near field's copy: the bodies of a leaf in pairs, {x0, x1, y0, y1},
// {z0, z1, q0, q1} at pairs[2 (b + k)] for pair k of the leaf whose first body
// is b (so a leaf starts at twice its body index and fills half the room); the
// last pair of an odd leaf is filled with a zero charge at the leaf's centre.
// Body r of nb, v = (x, y, z, q):
__device__ __forceinline__ void put_pair(float4 *pairs, int b, int r, int nb, float4 v) {
  float *p = (float *)(pairs + 2 * ((long)b + (r >> 1)));
  const int o = r & 1;
  p[o] = v.x;
  p[2 + o] = v.y;
  p[4 + o] = v.z;
  p[6 + o] = v.w;
  if (r == nb - 1 && o == 0) p[1] = p[3] = p[5] = p[7] = 0.f;
}

}  // namespace fmm
