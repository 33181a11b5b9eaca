// RMSNorm of rows of up to 1024 floats (a multiple of 128), a warp per row (reference src/ops.rs:8-56): the row lives in registers, the
// reductions are warp shuffles.  For ops.cu, and rmsnorm_lr.cu with the low-rank product of the result.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace rt {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// A warp's row: lane l holds float4 l, l + 32, ..
template <int NV>  // float4s per lane: d = 128 * NV
__device__ __forceinline__ void rms_load_row(const float* row, int lane, float4* v) {
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = ((const float4*)row)[lane + 32 * k];
}
__device__ __forceinline__ uint2 half4(float4 v) {
  __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  return make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
}
// The four products of a lane's float4, and a x - b y: fused by name, so that a row gets the same bits in every kernel it may run
// through (a block's second forward takes the one without a product, and the backward's form goes by the number of rows).
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.x, b.x, a.y * b.y))); }
__device__ __forceinline__ float ax_by(float a, float x, float b, float y) { return fmaf(a, x, -(b * y)); }
// put(k, four f16): what lane + 32 k of the result is
template <int NV, class Put>
__device__ __forceinline__ void rms_fwd_row(const float4* v, const float* __restrict__ w, float eps, int lane, Put put) {
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) ss += dot4(v[k], v[k]);
  ss = warp_sum(ss);
  const float ir = 1.0f / sqrtf(ss / (float)(128 * NV) + eps);
  const float4* w4 = (const float4*)w;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const float4 g = w4[lane + 32 * k];
    put(k, half4(make_float4(v[k].x * ir * g.x, v[k].y * ir * g.y, v[k].z * ir * g.z, v[k].w * ir * g.w)));
  }
}
// v becomes the row of `out`, its largest magnitude is returned (of the warp's row); g: the row of dn, r: of dres or zeros
template <int NV>
__device__ __forceinline__ float rms_bwd_row(const float4* xv, float4* gv, const float4* rv, const float* __restrict__ w, float eps, int lane) {
  float ss = 0.f, gx = 0.f;
  const float4* w4 = (const float4*)w;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const float4 wv = w4[lane + 32 * k];
    gv[k] = make_float4(gv[k].x * wv.x, gv[k].y * wv.y, gv[k].z * wv.z, gv[k].w * wv.w);
    ss += dot4(xv[k], xv[k]);
    gx += dot4(gv[k], xv[k]);
  }
  ss = warp_sum(ss);
  gx = warp_sum(gx);
  const float ir = 1.0f / sqrtf(ss / (float)(128 * NV) + eps);
  const float c = gx * ir * ir * ir / (float)(128 * NV);
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    float4 v = make_float4(ax_by(gv[k].x, ir, xv[k].x, c), ax_by(gv[k].y, ir, xv[k].y, c), ax_by(gv[k].z, ir, xv[k].z, c),
                           ax_by(gv[k].w, ir, xv[k].w, c));
    v.x += rv[k].x; v.y += rv[k].y; v.z += rv[k].z; v.w += rv[k].w;
    gv[k] = v;
    m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
  return m;
}

}  // namespace rt
