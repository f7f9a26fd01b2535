// mxsum.cuh - sums of an MXFP4 row that the tensor-core products cannot make, once more in f32.
// An activation that is no finite number has no pieces (its block's are NaN), scale byte 255 is no number, weights of 2^128
// and more (scale bytes from 253 on) are no bf16, and a sum may leave a float's range piece by piece where the f32 sum
// does not. Such a sum comes out as an infinity or a NaN: it is made again from the weights and rows as stored, with the
// operations of the row kernels (kernels_basic.cu, rows_mx_f32). Rare: a thread's own loop over K; where every sum is
// finite it costs an fma an output.
#pragma once

#include "tcgen.cuh"

// blocks b0 .. b1 of a row of codes (16 bytes a block) and scale bytes against x
__device__ __forceinline__ float mx_sum_f32(const uint8_t *codes, const uint8_t *scales, const float *x, int b0, int b1) {
  float a = 0.0f;
#pragma unroll 1
  for (int b = b0; b < b1; b++) {
    float t = 0.0f;
    const uint4 q = __ldg((const uint4 *)(codes + (size_t)b * 16));
#pragma unroll 1
    for (int j = 0; j < 4; j++) {  // values 4 j .. and 16 + 4 j ..
      const uint32_t c = j < 2 ? (j == 0 ? q.x : q.y) : (j == 2 ? q.z : q.w);
      const float4 lo = *(const float4 *)(x + 32 * b + 4 * j), hi = *(const float4 *)(x + 32 * b + 16 + 4 * j);
      const float xl[4] = {lo.x, lo.y, lo.z, lo.w}, xh[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        t = __fmaf_rn(pm_e2m1((c >> (8 * k)) & 15u), xl[k], t);
        t = __fmaf_rn(pm_e2m1((c >> (8 * k + 4)) & 15u), xh[k], t);
      }
    }
    a = __fmaf_rn(pm_e8(__ldg(scales + b)), t, a);
  }
  return a;
}
// N sums of a thread: those that are not finite are replaced by sum(i), unless i is no place of its own (valid(i))
template <int N, class Valid, class Sum> __device__ __forceinline__ void mx_repair(float (&v)[N], Valid valid, Sum sum) {
  float poison = 0.0f;
#pragma unroll
  for (int i = 0; i < N; i++) poison = __fmaf_rn(v[i], 0.0f, poison);
  if (poison == 0.0f) return;
#pragma unroll 1
  for (int u = 0; u < N; u++) {
    float a = 0.0f;
#pragma unroll
    for (int i = 0; i < N; i++) a = i == u ? v[i] : a;
    if (fabsf(a) <= 3.4028234e38f || !valid(u)) continue;
    a = sum(u);
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = i == u ? a : v[i];
  }
}
