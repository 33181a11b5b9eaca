// Memory-bound device ops around the frozen matmuls: RMSNorm, QK-norm + RoPE, SwiGLU,
// cross-entropy, row gathers, LoRA gradient reductions, AdamW.  One CTA per token row unless
// noted.  Every kernel that produces the 16-bit input of a backward matmul writes the row
// divided by its largest magnitude plus that magnitude as a per-row scale: f16 then keeps 11
// significant bits whatever the size of the gradients, and the matmul's epilogue multiplies
// the scale back in (the matmul is linear in each token row).
#include "ctx.h"
#include "lowrank_rows.cuh"
#include "ops.h"
#include "pdl.cuh"
#include "rmsnorm_row.cuh"
#include <algorithm>

namespace rt {

// ------------------------------------------------------------------ reductions
__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Block-wide reductions (blockDim.x <= 1024); result broadcast to every thread.
__device__ float block_sum(float v) {
  __shared__ float sh[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < (int)((blockDim.x + 31) >> 5) ? sh[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) sh[32] = t;
  }
  __syncthreads();
  return sh[32];
}
__device__ float block_max(float v) {
  __shared__ float sh[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < (int)((blockDim.x + 31) >> 5) ? sh[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) sh[32] = t;
  }
  __syncthreads();
  return sh[32];
}
__device__ double block_sum_d(double v) {
  __shared__ double sh[33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum_d(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    double t = lane < (int)((blockDim.x + 31) >> 5) ? sh[lane] : 0.0;
    t = warp_sum_d(t);
    if (lane == 0) sh[32] = t;
  }
  __syncthreads();
  return sh[32];
}

// ------------------------------------------------------------------ conversions
template <bool F16>
__global__ void f32_to_16_kernel(const float* __restrict__ in, uint16_t* __restrict__ out, size_t n) {
  size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i + 3 < n) {
    float4 v = *(const float4*)(in + i);
    uint32_t a, b;
    if (F16) {
      __half2 x = __floats2half2_rn(v.x, v.y), y = __floats2half2_rn(v.z, v.w);
      a = *(uint32_t*)&x; b = *(uint32_t*)&y;
    } else {
      __nv_bfloat162 x = __floats2bfloat162_rn(v.x, v.y), y = __floats2bfloat162_rn(v.z, v.w);
      a = *(uint32_t*)&x; b = *(uint32_t*)&y;
    }
    *(uint2*)(out + i) = make_uint2(a, b);
  } else {
    for (; i < n; ++i) {
      if (F16) { __half h = __float2half_rn(in[i]); out[i] = *(uint16_t*)&h; }
      else { __nv_bfloat16 h = __float2bfloat16_rn(in[i]); out[i] = *(uint16_t*)&h; }
    }
  }
}
void launch_f32_to_16(const float* in, void* out, size_t n, bool to_f16, cudaStream_t st) {
  if (n == 0) return;
  size_t threads = (n + 3) / 4;
  unsigned blocks = (unsigned)((threads + 255) / 256);
  if (to_f16) { f32_to_16_kernel<true><<<blocks, 256, 0, st>>>(in, (uint16_t*)out, n); RT_COUNT_LAUNCH(1); }
  else { f32_to_16_kernel<false><<<blocks, 256, 0, st>>>(in, (uint16_t*)out, n); RT_COUNT_LAUNCH(1); }
}

__global__ void split_f32_hi_lo_kernel(const float* __restrict__ w, size_t n, __half* __restrict__ hi, __half* __restrict__ lo) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float v = w[i];
  const __half h = __float2half_rn(v);
  hi[i] = h;
  lo[i] = __float2half_rn(v - __half2float(h));
}
void launch_split_f32_hi_lo(const float* w, size_t n, __half* hi, __half* lo, cudaStream_t st) {
  if (n == 0) return;
  split_f32_hi_lo_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w, n, hi, lo);
  RT_COUNT_LAUNCH(1);
}

// Row-normalised f16 copy: y16[r,:] = x[r,:] / amax_r, scale[r] = amax_r (1 if the row is zero).
__global__ void normalize_rows_kernel(const float* x, int d, __half* __restrict__ y16,
                                      float* __restrict__ scale) {
  pdl_entry();
  const size_t r = blockIdx.x;
  const float* xr = x + r * d;
  float m = 0.f;
  for (int i = threadIdx.x; i < d; i += blockDim.x) m = fmaxf(m, fabsf(xr[i]));
  m = block_max(m);
  const float s = m > 0.f ? m : 1.f, inv = 1.f / s;
  for (int i = threadIdx.x; i < d; i += blockDim.x) y16[r * d + i] = __float2half_rn(xr[i] * inv);
  // an all-zero row reports the factor 0, not 1: consumers that weigh rows by factor / largest
  // factor (attention backward, the token contractions) must not see a 1 that towers over the
  // real rows' small factors and pushes their f16 products into the subnormals
  if (threadIdx.x == 0) scale[r] = m;
}
void launch_normalize_rows(const float* x, int rows, int d, __half* y16, float* scale, cudaStream_t st) {
  if (rows > 0) { pdl(normalize_rows_kernel, rows, 256, 0, st)(x, d, y16, scale); RT_COUNT_LAUNCH(1); }
}

// ------------------------------------------------------------------ RMSNorm (reference src/ops.rs:8-56)
// y16 = x * ir * w  with ir = 1/sqrt(mean(x^2) + eps)
__global__ void rmsnorm_fwd_kernel(const float* __restrict__ x, const float* __restrict__ w, int d, float eps,
                                   __half* __restrict__ y16) {
  const size_t r = blockIdx.x;
  const float* xr = x + r * d;
  float ss = 0.f;
  for (int i = threadIdx.x; i < d; i += blockDim.x) ss += xr[i] * xr[i];
  ss = block_sum(ss);
  const float ir = 1.0f / sqrtf(ss / (float)d + eps);
  for (int i = threadIdx.x; i < d; i += blockDim.x) y16[r * d + i] = __float2half_rn(xr[i] * ir * w[i]);
}
// Longer rows (d % 4 == 0, up to 12288): a block per row, three float4 per thread, the row in registers: one
// round of memory latency and one barrier.  (Looping over the row twice: 3072 columns, 8192 rows 39 us
// forward, 77-87 backward; floors 23 and 70.)
constexpr int RMS_NV = 3;
inline int rms_row_threads(int d) { return ((d / 4 + RMS_NV - 1) / RMS_NV + 31) & ~31; }
// two block-wide sums through one barrier
__device__ __forceinline__ void block_sum2(float& a, float& b) {
  __shared__ float sa[32], sb[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
  a = warp_sum(a);
  b = warp_sum(b);
  if (lane == 0) { sa[w] = a; sb[w] = b; }
  __syncthreads();
  a = b = 0.f;
  for (int k = 0; k < nw; ++k) { a += sa[k]; b += sb[k]; }
}
__global__ void __launch_bounds__(1024) rmsnorm_fwd_row_kernel(const float* x, const float* __restrict__ w, int d, float eps,
                                                               __half* __restrict__ y16) {
  pdl_entry();
  const size_t r = blockIdx.x;
  const float4* x4 = (const float4*)(x + r * d);
  float4 v[RMS_NV];
  float ss = 0.f, unused = 0.f;
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    v[k] = i < d / 4 ? x4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
  block_sum2(ss, unused);
  const float ir = 1.0f / sqrtf(ss / (float)d + eps);
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    if (i >= d / 4) break;
    const float4 g = ((const float4*)w)[i];
    __half2 a = __floats2half2_rn(v[k].x * ir * g.x, v[k].y * ir * g.y), b = __floats2half2_rn(v[k].z * ir * g.z, v[k].w * ir * g.w);
    *(uint2*)(y16 + r * d + 4 * i) = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
  }
}
// Warp-per-row versions for rows of up to 1024 floats (rmsnorm_row.cuh): eight rows per CTA keep far more bytes in
// flight per SM than one small CTA per row.
template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_warp_kernel(const float* x, const float* __restrict__ w, int rows, float eps,
                        __half* __restrict__ y16) {
  pdl_entry();
  constexpr int D = 128 * NV;
  const int lane = threadIdx.x & 31;
  const size_t r = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= (size_t)rows) return;
  float4 v[NV];
  rms_load_row<NV>(x + r * D, lane, v);
  rms_fwd_row<NV>(v, w, eps, lane, [&](int k, uint2 o) { *(uint2*)(y16 + r * D + 4 * (lane + 32 * k)) = o; });
}
template <int NV>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_warp_kernel(const float* x, const float* __restrict__ w, const float* dn,
                        const float* dres, int rows, float eps, float* out, __half* __restrict__ out16,
                        float* __restrict__ scale) {
  pdl_entry();
  constexpr int D = 128 * NV;
  const int lane = threadIdx.x & 31;
  const size_t r = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= (size_t)rows) return;
  float4 xv[NV], gv[NV], rv[NV];
  // every load of the row is issued before the first reduction: one round of memory latency, not two
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    xv[k] = ((const float4*)(x + r * D))[lane + 32 * k];
    gv[k] = ((const float4*)(dn + r * D))[lane + 32 * k];
    rv[k] = dres ? ((const float4*)(dres + r * D))[lane + 32 * k] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float m = rms_bwd_row<NV>(xv, gv, rv, w, eps, lane);
#pragma unroll
  for (int k = 0; k < NV; ++k) ((float4*)(out + r * D))[lane + 32 * k] = gv[k];
  if (out16) {
    m = warp_max(m);
    const float sc = m > 0.f ? m : 1.f, inv = 1.f / sc;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      *(uint2*)(out16 + r * D + 4 * (lane + 32 * k)) = half4(make_float4(gv[k].x * inv, gv[k].y * inv, gv[k].z * inv, gv[k].w * inv));
    if (lane == 0) scale[r] = m;
  }
}

void launch_rmsnorm_fwd(const float* x, const float* w, int rows, int d, float eps, __half* y16, cudaStream_t st) {
  if (rows <= 0) return;
  const int nv = d / 128, grid = (rows + 7) / 8;
  const bool warp_ok = d % 128 == 0 && nv >= 1 && nv <= 8 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0;
  if (warp_ok) {
    switch (nv) {
      case 1: pdl(rmsnorm_fwd_warp_kernel<1>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 2: pdl(rmsnorm_fwd_warp_kernel<2>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 3: pdl(rmsnorm_fwd_warp_kernel<3>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 4: pdl(rmsnorm_fwd_warp_kernel<4>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 5: pdl(rmsnorm_fwd_warp_kernel<5>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 6: pdl(rmsnorm_fwd_warp_kernel<6>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      case 7: pdl(rmsnorm_fwd_warp_kernel<7>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
      default: pdl(rmsnorm_fwd_warp_kernel<8>, grid, 256, 0, st)(x, w, rows, eps, y16); break;
    }
  } else if (d % 4 == 0 && rms_row_threads(d) <= 1024 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
    pdl(rmsnorm_fwd_row_kernel, rows, rms_row_threads(d), 0, st)(x, w, d, eps, y16);
  } else {
    rmsnorm_fwd_kernel<<<rows, 256, 0, st>>>(x, w, d, eps, y16);
  }
  RT_COUNT_LAUNCH(1);
}

// dx = g*ir - x*c, g = dn*w, c = dot(g,x)*ir^3/d;  out = (dres ? dres : 0) + dx.
// Optionally also the row-normalised f16 copy of `out` and its scale.
__global__ void rmsnorm_bwd_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                   const float* __restrict__ dn, const float* dres, int d, float eps, float* out,
                                   __half* __restrict__ out16, float* __restrict__ scale) {
  const size_t r = blockIdx.x;
  const float* xr = x + r * d;
  const float* dnr = dn + r * d;
  float ss = 0.f, gx = 0.f, m = 0.f;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float xv = xr[i];
    ss += xv * xv;
    gx += dnr[i] * w[i] * xv;
  }
  ss = block_sum(ss);
  gx = block_sum(gx);
  const float ir = 1.0f / sqrtf(ss / (float)d + eps);
  const float c = gx * ir * ir * ir / (float)d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float v = dnr[i] * w[i] * ir - xr[i] * c;
    if (dres) v += dres[r * d + i];
    out[r * d + i] = v;
    m = fmaxf(m, fabsf(v));
  }
  if (out16) {
    m = block_max(m);  // includes a __syncthreads: this thread's stores above are its own re-reads below
    const float sc = m > 0.f ? m : 1.f, inv = 1.f / sc;
    for (int i = threadIdx.x; i < d; i += blockDim.x) out16[r * d + i] = __float2half_rn(out[r * d + i] * inv);
    if (threadIdx.x == 0) scale[r] = m;
  }
}
__global__ void __launch_bounds__(1024) rmsnorm_bwd_row_kernel(const float* x, const float* __restrict__ w,
                                                               const float* dn, const float* dres, int d, float eps,
                                                               float* out, __half* __restrict__ out16, float* __restrict__ scale) {
  pdl_entry();
  const size_t r = blockIdx.x;
  const float4 *x4 = (const float4*)(x + r * d), *d4 = (const float4*)(dn + r * d);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 xv[RMS_NV], gv[RMS_NV], rv[RMS_NV];
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    const bool in = i < d / 4;
    xv[k] = in ? x4[i] : zero;
    gv[k] = in ? d4[i] : zero;
    rv[k] = in && dres ? ((const float4*)(dres + r * d))[i] : zero;
  }
  float ss = 0.f, gx = 0.f;
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    const float4 wv = i < d / 4 ? ((const float4*)w)[i] : zero;
    gv[k] = make_float4(gv[k].x * wv.x, gv[k].y * wv.y, gv[k].z * wv.z, gv[k].w * wv.w);
    ss += xv[k].x * xv[k].x + xv[k].y * xv[k].y + xv[k].z * xv[k].z + xv[k].w * xv[k].w;
    gx += gv[k].x * xv[k].x + gv[k].y * xv[k].y + gv[k].z * xv[k].z + gv[k].w * xv[k].w;
  }
  block_sum2(ss, gx);
  const float ir = 1.0f / sqrtf(ss / (float)d + eps);
  const float c = gx * ir * ir * ir / (float)d;
  float m = 0.f;
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    float4 v = make_float4(gv[k].x * ir - xv[k].x * c, gv[k].y * ir - xv[k].y * c, gv[k].z * ir - xv[k].z * c, gv[k].w * ir - xv[k].w * c);
    v.x += rv[k].x; v.y += rv[k].y; v.z += rv[k].z; v.w += rv[k].w;
    if (i < d / 4) ((float4*)(out + r * d))[i] = v;
    gv[k] = v;  // zero past the row's end
    m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
  }
  if (!out16) return;
  m = block_max(m);
  const float sc = m > 0.f ? m : 1.f, inv = 1.f / sc;
#pragma unroll
  for (int k = 0; k < RMS_NV; ++k) {
    const int i = k * blockDim.x + threadIdx.x;
    if (i >= d / 4) break;
    __half2 a = __floats2half2_rn(gv[k].x * inv, gv[k].y * inv), b = __floats2half2_rn(gv[k].z * inv, gv[k].w * inv);
    *(uint2*)(out16 + r * d + 4 * i) = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
  }
  if (threadIdx.x == 0) scale[r] = m;
}
void launch_rmsnorm_bwd(const float* x, const float* w, const float* dn, const float* dres, int rows, int d, float eps,
                        float* out, __half* out16, float* scale, cudaStream_t st) {
  if (rows <= 0) return;
  const int nv = d / 128, grid = (rows + 7) / 8;
  const bool warp_ok = d % 128 == 0 && nv >= 1 && nv <= 8 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0 &&
                       ((uintptr_t)dn & 15) == 0 && ((uintptr_t)out & 15) == 0 && (!dres || ((uintptr_t)dres & 15) == 0);
  if (warp_ok) {
#define RT_RMSB(N) pdl(rmsnorm_bwd_warp_kernel<N>, grid, 256, 0, st)(x, w, dn, dres, rows, eps, out, out16, scale)
    switch (nv) {
      case 1: RT_RMSB(1); break;
      case 2: RT_RMSB(2); break;
      case 3: RT_RMSB(3); break;
      case 4: RT_RMSB(4); break;
      case 5: RT_RMSB(5); break;
      case 6: RT_RMSB(6); break;
      case 7: RT_RMSB(7); break;
      default: RT_RMSB(8); break;
    }
#undef RT_RMSB
  } else if (d % 4 == 0 && rms_row_threads(d) <= 1024 &&
             (((uintptr_t)x | (uintptr_t)w | (uintptr_t)dn | (uintptr_t)out | (uintptr_t)dres) & 15) == 0) {
    pdl(rmsnorm_bwd_row_kernel, rows, rms_row_threads(d), 0, st)(x, w, dn, dres, d, eps, out, out16, scale);
  } else {
    rmsnorm_bwd_kernel<<<rows, 256, 0, st>>>(x, w, dn, dres, d, eps, out, out16, scale);
  }
  RT_COUNT_LAUNCH(1);
}

// ------------------------------------------------------------------ RoPE tables (reference src/ops.rs:118-154)
__global__ void rope_table_kernel(const float* __restrict__ inv_freq, int half, int max_pos, float* __restrict__ cs,
                                  float* __restrict__ sn) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= max_pos * half) return;
  int p = i / half, f = i % half;
  float a = (float)p * inv_freq[f];
  cs[i] = cosf(a);
  sn[i] = sinf(a);
}
void launch_rope_table(const float* inv_freq, int half, int max_pos, float* cs, float* sn, cudaStream_t st) {
  int n = max_pos * half;
  if (n > 0) { rope_table_kernel<<<(n + 255) / 256, 256, 0, st>>>(inv_freq, half, max_pos, cs, sn); RT_COUNT_LAUNCH(1); }
}

// ------------------------------------------------------------------ QK-norm + RoPE + f16 rounding
// (reference src/attention.rs:170-185).  One CTA per token, one warp per head in turn.
// Heads 0..nh-1 are q, nh..nh+nkv-1 are k, then nkv heads of v (copied and rounded only).
__global__ void qk_rope_fwd_kernel(const float* __restrict__ q_raw, const float* __restrict__ k_raw,
                                   const float* __restrict__ v_raw, const float* __restrict__ qw,
                                   const float* __restrict__ kw, const int* __restrict__ pos,
                                   const float* __restrict__ cs, const float* __restrict__ sn, int nh, int nkv, int hd,
                                   int rot, int neox, float eps, __half* __restrict__ q16, __half* __restrict__ k16,
                                   __half* __restrict__ v16) {
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int half = rot / 2;
  const int p = pos[m];
  const float* csr = cs + (size_t)p * half;
  const float* snr = sn + (size_t)p * half;
  for (int h = warp; h < nh + 2 * nkv; h += nwarps) {
    if (h >= nh + nkv) {
      const int hv = h - nh - nkv;
      const float* src = v_raw + (m * nkv + hv) * hd;
      __half* dst = v16 + (m * nkv + hv) * hd;
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 v = *(const float4*)(src + i);
        __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
        *(uint2*)(dst + i) = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
      }
      continue;
    }
    const bool is_q = h < nh;
    const float* src = is_q ? q_raw + (m * nh + h) * hd : k_raw + (m * nkv + (h - nh)) * hd;
    const float* nw = is_q ? qw : kw;
    __half* dst = is_q ? q16 + (m * nh + h) * hd : k16 + (m * nkv + (h - nh)) * hd;
    float ir = 1.f;
    if (nw) {
      float ss = 0.f;
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 v = *(const float4*)(src + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
      }
      ss = warp_sum(ss);
      ir = 1.0f / sqrtf(ss / (float)hd + eps);
    }
    // two rotation pairs per lane and round; elements beyond rot pass through
    for (int i = lane * 2; i < half; i += 64) {
      const float2 c = *(const float2*)(csr + i), s = *(const float2*)(snr + i);
      if (neox) {
        float2 x1 = *(const float2*)(src + i), x2 = *(const float2*)(src + i + half);
        if (nw) {
          const float2 w1 = *(const float2*)(nw + i), w2 = *(const float2*)(nw + i + half);
          x1.x *= ir * w1.x; x1.y *= ir * w1.y; x2.x *= ir * w2.x; x2.y *= ir * w2.y;
        }
        *(__half2*)(dst + i) = __floats2half2_rn(x1.x * c.x - x2.x * s.x, x1.y * c.y - x2.y * s.y);
        *(__half2*)(dst + i + half) = __floats2half2_rn(x2.x * c.x + x1.x * s.x, x2.y * c.y + x1.y * s.y);
      } else {
        float4 x = *(const float4*)(src + 2 * i);  // pairs (2i, 2i+1), (2i+2, 2i+3)
        if (nw) {
          const float4 w4 = *(const float4*)(nw + 2 * i);
          x.x *= ir * w4.x; x.y *= ir * w4.y; x.z *= ir * w4.z; x.w *= ir * w4.w;
        }
        __half2 a = __floats2half2_rn(x.x * c.x - x.y * s.x, x.y * c.x + x.x * s.x);
        __half2 b = __floats2half2_rn(x.z * c.y - x.w * s.y, x.w * c.y + x.z * s.y);
        *(uint2*)(dst + 2 * i) = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
      }
    }
    for (int i = rot + lane; i < hd; i += 32) {
      float x = src[i];
      if (nw) x = x * (ir * nw[i]);
      dst[i] = __float2half_rn(x);
    }
  }
}

// Register-resident versions of the two kernels above for the usual shapes (head size 64 or
// 128, at most 8 heads per warp): a warp holds a whole head, EPL consecutive elements per lane,
// so every global load of a token's heads is issued before any of them is used, the rotation
// partner comes from a lane shuffle, and nothing is staged in shared memory.
template <int EPL>
struct RopeLane {
  // what lane `lane` needs to rotate its EPL elements of one head
  float c[EPL], s[EPL];  // cos, and sin signed for the FORWARD rotation (0 / 1 beyond rot)
  int src_lane;          // neox: the lane holding the partner elements; interleaved: unused
  bool rotates;
};
template <int EPL>
__device__ __forceinline__ RopeLane<EPL> rope_lane(int lane, const float* csr, const float* snr, int half, int rot, int neox) {
  RopeLane<EPL> r;
  const int e0 = lane * EPL;
  r.rotates = e0 < rot;
  r.src_lane = lane;
#pragma unroll
  for (int k = 0; k < EPL; ++k) { r.c[k] = 1.f; r.s[k] = 0.f; }
  if (!r.rotates) return r;
  if (neox) {
    const bool first = e0 < half;
    r.src_lane = first ? lane + half / EPL : lane - half / EPL;
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      const int i = first ? e0 + k : e0 + k - half;
      r.c[k] = csr[i];
      r.s[k] = first ? -snr[i] : snr[i];
    }
  } else {
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      const int i = (e0 + k) >> 1;
      r.c[k] = csr[i];
      r.s[k] = (k & 1) ? snr[i] : -snr[i];
    }
  }
  return r;
}
// out = own*c + partner*s*dir  (dir = +1 forward, -1 inverse)
template <int EPL>
__device__ __forceinline__ void rope_apply(const RopeLane<EPL>& r, int neox, float dir, const float* x, float* out) {
  float partner[EPL];
  if (neox) {
#pragma unroll
    for (int k = 0; k < EPL; ++k) partner[k] = __shfl_sync(0xffffffffu, x[k], r.src_lane);
  } else {
#pragma unroll
    for (int k = 0; k < EPL; ++k) partner[k] = x[k ^ 1];
  }
#pragma unroll
  for (int k = 0; k < EPL; ++k) out[k] = x[k] * r.c[k] + partner[k] * (r.s[k] * dir);
}
template <int EPL>
__device__ __forceinline__ void load_epl(const float* p, float* v) {
  if (EPL == 4) { const float4 t = *(const float4*)p; v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w; }
  else { const float2 t = *(const float2*)p; v[0] = t.x; v[1] = t.y; }
}
// What is read once and not again, past L1.  (Volatile: it stays behind a wait, through whatever pointer.)
template <int EPL>
__device__ __forceinline__ void load_epl_once(const float* p, float* v) {
  if constexpr (EPL == 4) asm volatile("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "l"(p));
  else asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p));
}
template <int EPL>
__device__ __forceinline__ void store_epl_h(__half* p, const float* v) {
  if (EPL == 4) {
    __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
    *(uint2*)p = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
  } else {
    *(__half2*)p = __floats2half2_rn(v[0], v[1]);
  }
}

template <int EPL, int HPW>
__global__ void __launch_bounds__(256)
qk_rope_fwd_reg_kernel(const float* q_raw, const float* k_raw, const float* v_raw,
                       size_t pq, size_t pk, size_t pv,  // row pitches of the three inputs, in elements
                       const float* __restrict__ qw, const float* __restrict__ kw, const int* __restrict__ pos,
                       const float* __restrict__ cs, const float* __restrict__ sn, int nh, int nkv, int rot, int neox,
                       float eps, __half* __restrict__ q16, __half* __restrict__ k16, __half* __restrict__ v16) {
  pdl_entry();
  constexpr int HD = 32 * EPL;
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = rot / 2, nheads = nh + 2 * nkv;
  // the rows first: the position -> cos/sin table chain is two dependent loads, which then run under them
  float x[HPW][EPL];
#pragma unroll
  for (int t = 0; t < HPW; ++t) {
    const int h = warp + t * 8;
    if (h < nheads) {
      const float* src = h < nh ? q_raw + m * pq + h * HD : (h < nh + nkv ? k_raw + m * pk + (h - nh) * HD
                                                                         : v_raw + m * pv + (h - nh - nkv) * HD);
      load_epl<EPL>(src + lane * EPL, x[t]);
    }
  }
  const int p = pos[m];
  const RopeLane<EPL> rl = rope_lane<EPL>(lane, cs + (size_t)p * half, sn + (size_t)p * half, half, rot, neox);
#pragma unroll
  for (int t = 0; t < HPW; ++t) {
    const int h = warp + t * 8;
    if (h >= nheads) continue;  // uniform in the warp
    if (h >= nh + nkv) {
      store_epl_h<EPL>(v16 + (m * nkv + (h - nh - nkv)) * HD + lane * EPL, x[t]);
      continue;
    }
    const bool is_q = h < nh;
    const float* nw = is_q ? qw : kw;
    if (nw) {
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < EPL; ++k) ss += x[t][k] * x[t][k];
      ss = warp_sum(ss);
      const float ir = 1.0f / sqrtf(ss / (float)HD + eps);
      float w[EPL];
      load_epl<EPL>(nw + lane * EPL, w);
#pragma unroll
      for (int k = 0; k < EPL; ++k) x[t][k] *= ir * w[k];
    }
    float o[EPL];
    rope_apply<EPL>(rl, neox, 1.f, x[t], o);
    __half* dst = is_q ? q16 + (m * nh + h) * HD : k16 + (m * nkv + (h - nh)) * HD;
    store_epl_h<EPL>(dst + lane * EPL, o);
  }
}

// The same for the common geometry with nothing left to decide per head: full rotation
// (rot == head_dim), query and KV head counts that are multiples of the CTA's eight warps (warp w
// owns query heads w, w + 8, .. and KV heads w, w + 8, ..), both norms present or both absent.  The
// general kernel above spends more issue slots on choosing pointers and on uniform branches than on
// arithmetic; it is bound by instruction issue, not by bytes.
template <int EPL, int QPW, int KPW, bool NEOX, bool NORM>
__global__ void __launch_bounds__(256)
qk_rope_fwd_fast_kernel(const float* q_raw, const float* k_raw, const float* v_raw,
                        size_t pq, size_t pk, size_t pv, const float* __restrict__ qw, const float* __restrict__ kw,
                        const int* __restrict__ pos, const float* __restrict__ cs, const float* __restrict__ sn, float eps,
                        __half* __restrict__ q16, __half* __restrict__ k16, __half* __restrict__ v16) {
  pdl_launch_dependents();
  const int p = pos[blockIdx.x];  // the batch's: the tables' rows are read with the wait over, not behind this too
  pdl_wait();
  constexpr int HD = 32 * EPL, HALF = HD / 2, NH = 8 * QPW, NKV = 8 * KPW;
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = lane * EPL;
  const float* qs = q_raw + m * pq + warp * HD + e0;
  const float* ks = k_raw + m * pk + warp * HD + e0;
  const float* vs = v_raw + m * pv + warp * HD + e0;
  float xq[QPW][EPL], xk[KPW][EPL], xv[KPW][EPL];
#pragma unroll
  for (int t = 0; t < QPW; ++t) load_epl_once<EPL>(qs + t * 8 * HD, xq[t]);
#pragma unroll
  for (int t = 0; t < KPW; ++t) load_epl_once<EPL>(ks + t * 8 * HD, xk[t]);
#pragma unroll
  for (int t = 0; t < KPW; ++t) load_epl_once<EPL>(vs + t * 8 * HD, xv[t]);
  float wq[EPL], wk[EPL];
  if (NORM) {
    load_epl<EPL>(qw + e0, wq);
    load_epl<EPL>(kw + e0, wk);
  }
  const float* csr = cs + (size_t)p * HALF;
  const float* snr = sn + (size_t)p * HALF;
  float c[EPL], sg[EPL];
  if (NEOX) {
    const bool first = e0 < HALF;
    float sv_[EPL];
    load_epl<EPL>(csr + (first ? e0 : e0 - HALF), c);
    load_epl<EPL>(snr + (first ? e0 : e0 - HALF), sv_);
#pragma unroll
    for (int k = 0; k < EPL; ++k) sg[k] = first ? -sv_[k] : sv_[k];
  } else {
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      c[k] = csr[(e0 + k) >> 1];
      const float t = snr[(e0 + k) >> 1];
      sg[k] = (k & 1) ? t : -t;
    }
  }
  auto finish = [&](float* x, const float* w, __half* dst) {
    if (NORM) {
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < EPL; ++k) ss += x[k] * x[k];
      ss = warp_sum(ss);
      const float ir = 1.0f / sqrtf(ss / (float)HD + eps);
#pragma unroll
      for (int k = 0; k < EPL; ++k) x[k] *= ir * w[k];
    }
    float o[EPL];
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      const float partner = NEOX ? __shfl_xor_sync(0xffffffffu, x[k], 16) : x[k ^ 1];
      o[k] = x[k] * c[k] + partner * sg[k];
    }
    store_epl_h<EPL>(dst, o);
  };
#pragma unroll
  for (int t = 0; t < QPW; ++t) finish(xq[t], wq, q16 + (m * NH + warp + 8 * t) * HD + e0);
#pragma unroll
  for (int t = 0; t < KPW; ++t) finish(xk[t], wk, k16 + (m * NKV + warp + 8 * t) * HD + e0);
#pragma unroll
  for (int t = 0; t < KPW; ++t) store_epl_h<EPL>(v16 + (m * NKV + warp + 8 * t) * HD + e0, xv[t]);
}

template <int EPL, int HPW>
__global__ void __launch_bounds__(256, 4)
qk_rope_bwd_reg_kernel(const float* dq, const float* dk, const float* dv,
                       const float* q_raw, const float* k_raw, size_t pq, size_t pk,
                       size_t oq, size_t ok, size_t ov, int common,  // output row pitches; one scale for all three
                       const float* __restrict__ qw,
                       const float* __restrict__ kw, const int* __restrict__ pos, const float* __restrict__ cs,
                       const float* __restrict__ sn, int nh, int nkv, int rot, int neox, float eps,
                       __half* __restrict__ dq16, __half* __restrict__ dk16, __half* __restrict__ dv16,
                       float* __restrict__ sq, float* __restrict__ sk, float* __restrict__ sv) {
  pdl_entry();
  constexpr int HD = 32 * EPL;
  __shared__ float wmax[3][8];
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = rot / 2, nheads = nh + 2 * nkv;
  float g[HPW][EPL], xr[HPW][EPL];
#pragma unroll
  for (int t = 0; t < HPW; ++t) {
    const int h = warp + t * 8;
    if (h < nheads) {
      const float* src = h < nh ? dq + (m * nh + h) * HD : (h < nh + nkv ? dk + (m * nkv + (h - nh)) * HD
                                                                        : dv + (m * nkv + (h - nh - nkv)) * HD);
      load_epl<EPL>(src + lane * EPL, g[t]);
      const float* nw = h < nh ? qw : (h < nh + nkv ? kw : nullptr);
      if (nw) load_epl<EPL>((h < nh ? q_raw + m * pq + h * HD : k_raw + m * pk + (h - nh) * HD) + lane * EPL, xr[t]);
    }
  }
  // after the rows: the position -> cos/sin table chain (two dependent loads) runs under them
  const int p = pos[m];
  const RopeLane<EPL> rl = rope_lane<EPL>(lane, cs + (size_t)p * half, sn + (size_t)p * half, half, rot, neox);
  float mx[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int t = 0; t < HPW; ++t) {
    const int h = warp + t * 8;
    if (h >= nheads) continue;
    const int kind = h < nh ? 0 : (h < nh + nkv ? 1 : 2);
    if (kind < 2) {
      float o[EPL];
      rope_apply<EPL>(rl, neox, -1.f, g[t], o);  // inverse rotation
      const float* nw = kind == 0 ? qw : kw;
      if (nw) {
        float w[EPL];
        load_epl<EPL>(nw + lane * EPL, w);
        float ss = 0.f, gx = 0.f;
#pragma unroll
        for (int k = 0; k < EPL; ++k) { ss += xr[t][k] * xr[t][k]; gx += o[k] * w[k] * xr[t][k]; }
        ss = warp_sum(ss);
        gx = warp_sum(gx);
        const float ir = 1.0f / sqrtf(ss / (float)HD + eps);
        const float c = gx * ir * ir * ir / (float)HD;
#pragma unroll
        for (int k = 0; k < EPL; ++k) o[k] = o[k] * w[k] * ir - xr[t][k] * c;
      }
#pragma unroll
      for (int k = 0; k < EPL; ++k) g[t][k] = o[k];
    }
#pragma unroll
    for (int k = 0; k < EPL; ++k) mx[kind] = fmaxf(mx[kind], fabsf(g[t][k]));
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float v = warp_max(mx[k]);
    if (lane == 0) wmax[k][warp] = v;
  }
  __syncthreads();
  float s3[3], inv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v = fmaxf(v, wmax[k][w]);
    s3[k] = v;
  }
  if (common) s3[0] = s3[1] = s3[2] = fmaxf(s3[0], fmaxf(s3[1], s3[2]));
#pragma unroll
  if (threadIdx.x == 0) { sq[m] = s3[0]; sk[m] = s3[1]; sv[m] = s3[2]; }  // 0 for an all-zero row
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s3[k] = s3[k] > 0.f ? s3[k] : 1.f;
    inv[k] = 1.f / s3[k];
  }
#pragma unroll
  for (int t = 0; t < HPW; ++t) {
    const int h = warp + t * 8;
    if (h >= nheads) continue;
    const int kind = h < nh ? 0 : (h < nh + nkv ? 1 : 2);
    float o[EPL];
#pragma unroll
    for (int k = 0; k < EPL; ++k) o[k] = g[t][k] * inv[kind];
    __half* dst = kind == 0 ? dq16 + m * oq + h * HD : (kind == 1 ? dk16 + m * ok + (h - nh) * HD
                                                                   : dv16 + m * ov + (h - nh - nkv) * HD);
    store_epl_h<EPL>(dst + lane * EPL, o);
  }
}

// Backward for the same common geometry as qk_rope_fwd_fast_kernel (full rotation, head counts
// that are multiples of eight, both norms or none): no per-head decisions left.
template <int EPL, int QPW, int KPW, bool NEOX, bool NORM>
__global__ void __launch_bounds__(256, (QPW + 2 * KPW <= 4) ? 4 : ((QPW + 2 * KPW <= 6) ? 3 : 2))
qk_rope_bwd_fast_kernel(const float* dq, const float* dk, const float* dv,
                        const float* q_raw, const float* k_raw, size_t pq, size_t pk, size_t oq,
                        size_t ok, size_t ov, int common, const float* __restrict__ qw, const float* __restrict__ kw,
                        const int* __restrict__ pos, const float* __restrict__ cs, const float* __restrict__ sn, float eps,
                        __half* __restrict__ dq16, __half* __restrict__ dk16, __half* __restrict__ dv16,
                        float* __restrict__ sq, float* __restrict__ sk, float* __restrict__ sv) {
  pdl_launch_dependents();
  const int p = pos[blockIdx.x];  // the batch's: the tables' rows are read with the wait over, not behind this too
  pdl_wait();
  constexpr int HD = 32 * EPL, HALF = HD / 2, NH = 8 * QPW, NKV = 8 * KPW;
  __shared__ float wmax[3][8];
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = lane * EPL;
  float gq[QPW][EPL], gk[KPW][EPL], gv[KPW][EPL], xq[QPW][EPL], xk[KPW][EPL];
#pragma unroll
  for (int t = 0; t < QPW; ++t) {
    load_epl<EPL>(dq + (m * NH + warp + 8 * t) * HD + e0, gq[t]);
    if (NORM) load_epl<EPL>(q_raw + m * pq + (warp + 8 * t) * HD + e0, xq[t]);
  }
#pragma unroll
  for (int t = 0; t < KPW; ++t) {
    load_epl<EPL>(dk + (m * NKV + warp + 8 * t) * HD + e0, gk[t]);
    load_epl<EPL>(dv + (m * NKV + warp + 8 * t) * HD + e0, gv[t]);
    if (NORM) load_epl<EPL>(k_raw + m * pk + (warp + 8 * t) * HD + e0, xk[t]);
  }
  float wq[EPL], wk[EPL];
  if (NORM) {
    load_epl<EPL>(qw + e0, wq);
    load_epl<EPL>(kw + e0, wk);
  }
  const float* csr = cs + (size_t)p * HALF;
  const float* snr = sn + (size_t)p * HALF;
  float c[EPL], sg[EPL];  // sin signed for the FORWARD rotation; the inverse subtracts
  if (NEOX) {
    const bool first = e0 < HALF;
    float sv_[EPL];
    load_epl<EPL>(csr + (first ? e0 : e0 - HALF), c);
    load_epl<EPL>(snr + (first ? e0 : e0 - HALF), sv_);
#pragma unroll
    for (int k = 0; k < EPL; ++k) sg[k] = first ? -sv_[k] : sv_[k];
  } else {
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      c[k] = csr[(e0 + k) >> 1];
      const float t = snr[(e0 + k) >> 1];
      sg[k] = (k & 1) ? t : -t;
    }
  }
  auto back = [&](float* g, const float* xr, const float* w) -> float {
    float o[EPL];
#pragma unroll
    for (int k = 0; k < EPL; ++k) {
      const float partner = NEOX ? __shfl_xor_sync(0xffffffffu, g[k], 16) : g[k ^ 1];
      o[k] = g[k] * c[k] + partner * (sg[k] * -1.f);
    }
    if (NORM) {
      float ss = 0.f, gx = 0.f;
#pragma unroll
      for (int k = 0; k < EPL; ++k) { ss += xr[k] * xr[k]; gx += o[k] * w[k] * xr[k]; }
      ss = warp_sum(ss);
      gx = warp_sum(gx);
      const float ir = 1.0f / sqrtf(ss / (float)HD + eps);
      const float cc = gx * ir * ir * ir / (float)HD;
#pragma unroll
      for (int k = 0; k < EPL; ++k) o[k] = o[k] * w[k] * ir - xr[k] * cc;
    }
    float mx = 0.f;
#pragma unroll
    for (int k = 0; k < EPL; ++k) { g[k] = o[k]; mx = fmaxf(mx, fabsf(o[k])); }
    return mx;
  };
  float mx[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int t = 0; t < QPW; ++t) mx[0] = fmaxf(mx[0], back(gq[t], xq[t], wq));
#pragma unroll
  for (int t = 0; t < KPW; ++t) mx[1] = fmaxf(mx[1], back(gk[t], xk[t], wk));
#pragma unroll
  for (int t = 0; t < KPW; ++t)
#pragma unroll
    for (int k = 0; k < EPL; ++k) mx[2] = fmaxf(mx[2], fabsf(gv[t][k]));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float v = warp_max(mx[k]);
    if (lane == 0) wmax[k][warp] = v;
  }
  __syncthreads();
  float s3[3], inv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v = fmaxf(v, wmax[k][w]);
    s3[k] = v;
  }
  if (common) s3[0] = s3[1] = s3[2] = fmaxf(s3[0], fmaxf(s3[1], s3[2]));
  if (threadIdx.x == 0) { sq[m] = s3[0]; sk[m] = s3[1]; sv[m] = s3[2]; }  // 0 for an all-zero row
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s3[k] = s3[k] > 0.f ? s3[k] : 1.f;
    inv[k] = 1.f / s3[k];
  }
  float o[EPL];
#pragma unroll
  for (int t = 0; t < QPW; ++t) {
#pragma unroll
    for (int k = 0; k < EPL; ++k) o[k] = gq[t][k] * inv[0];
    store_epl_h<EPL>(dq16 + m * oq + (warp + 8 * t) * HD + e0, o);
  }
#pragma unroll
  for (int t = 0; t < KPW; ++t) {
#pragma unroll
    for (int k = 0; k < EPL; ++k) o[k] = gk[t][k] * inv[1];
    store_epl_h<EPL>(dk16 + m * ok + (warp + 8 * t) * HD + e0, o);
#pragma unroll
    for (int k = 0; k < EPL; ++k) o[k] = gv[t][k] * inv[2];
    store_epl_h<EPL>(dv16 + m * ov + (warp + 8 * t) * HD + e0, o);
  }
}

// the shapes the register-resident kernels cover
static bool rope_reg_ok(int nh, int nkv, int hd, int rot, int neox, int* epl, int* hpw) {
  if (hd != 64 && hd != 128) return false;
  const int e = hd / 32, half = rot / 2;
  if (rot <= 0 || rot > hd || (rot & 1) || rot % e != 0) return false;
  if (neox && half % e != 0) return false;
  const int heads = nh + 2 * nkv;
  const int per = (heads + 7) / 8;
  if (per > 8) return false;
  *epl = e;
  *hpw = per <= 4 ? 4 : (per <= 6 ? 6 : 8);
  return true;
}
bool qk_rope_takes_pitches(int nh, int nkv, int hd, int rot, int neox) {
  int e, h;
  return rope_reg_ok(nh, nkv, hd, rot, neox, &e, &h);
}
void launch_qk_rope_fwd(const float* q_raw, const float* k_raw, const float* v_raw, size_t raw_pitch, const float* qw,
                        const float* kw, const int* pos, const float* cs, const float* sn, int M, int nh, int nkv, int hd,
                        int rot, int neox, float eps, __half* q16, __half* k16, __half* v16, cudaStream_t st) {
  if (M <= 0) return;
  int epl = 0, hpw = 0;
  // raw_pitch = 0: three separate row-major matrices; else one row pitch for all three (slices of one matrix)
  const size_t pq = raw_pitch ? raw_pitch : (size_t)nh * hd, pk = raw_pitch ? raw_pitch : (size_t)nkv * hd, pv = pk;
  if (hd == 128 && rot == hd && (qw != nullptr) == (kw != nullptr) && nh % 8 == 0 && nkv % 8 == 0) {
    const int qpw = nh / 8, kpw = nkv / 8;
#define RT_ROPE_FAST(Q, K)                                                                                                        \
  if (qpw == Q && kpw == K) {                                                                                                     \
    if (neox) {                                                                                                                   \
      if (qw) pdl(qk_rope_fwd_fast_kernel<4, Q, K, true, true>, M, 256, 0, st)(q_raw, k_raw, v_raw, pq, pk, pv, qw, kw, pos, cs, sn, eps, q16, k16, v16);   \
      else pdl(qk_rope_fwd_fast_kernel<4, Q, K, true, false>, M, 256, 0, st)(q_raw, k_raw, v_raw, pq, pk, pv, qw, kw, pos, cs, sn, eps, q16, k16, v16);     \
    } else {                                                                                                                      \
      if (qw) pdl(qk_rope_fwd_fast_kernel<4, Q, K, false, true>, M, 256, 0, st)(q_raw, k_raw, v_raw, pq, pk, pv, qw, kw, pos, cs, sn, eps, q16, k16, v16);  \
      else pdl(qk_rope_fwd_fast_kernel<4, Q, K, false, false>, M, 256, 0, st)(q_raw, k_raw, v_raw, pq, pk, pv, qw, kw, pos, cs, sn, eps, q16, k16, v16);    \
    }                                                                                                                             \
    RT_COUNT_LAUNCH(1);                                                                                                           \
    return;                                                                                                                       \
  }
    RT_ROPE_FAST(2, 1)
    RT_ROPE_FAST(3, 1)
    RT_ROPE_FAST(4, 1)
    RT_ROPE_FAST(4, 2)
    RT_ROPE_FAST(1, 1)
#undef RT_ROPE_FAST
  }
  if (rope_reg_ok(nh, nkv, hd, rot, neox, &epl, &hpw)) {
#define RT_ROPE_FWD(E, H) pdl(qk_rope_fwd_reg_kernel<E, H>, M, 256, 0, st)(q_raw, k_raw, v_raw, pq, pk, pv, qw, kw, pos, cs, sn, nh, nkv, rot, neox, eps, q16, k16, v16)
    if (epl == 4) { if (hpw == 4) RT_ROPE_FWD(4, 4); else if (hpw == 6) RT_ROPE_FWD(4, 6); else RT_ROPE_FWD(4, 8); }
    else { if (hpw == 4) RT_ROPE_FWD(2, 4); else if (hpw == 6) RT_ROPE_FWD(2, 6); else RT_ROPE_FWD(2, 8); }
#undef RT_ROPE_FWD
  } else {
    qk_rope_fwd_kernel<<<M, 256, 0, st>>>(q_raw, k_raw, v_raw, qw, kw, pos, cs, sn, nh, nkv, hd, rot, neox, eps, q16, k16, v16);
  }
  RT_COUNT_LAUNCH(1);
}

// Backward of the above (reference src/attention.rs:331-341): inverse rotation, then the
// QK-norm backward with the norm's input recomputed from q_raw/k_raw; dv passes through.
// Outputs are the three row-normalised f16 matrices (+ per-token scales) the q/k/v
// backward matmuls consume.  Dynamic shared memory: (nh + 2*nkv) * hd floats.
__global__ void qk_rope_bwd_kernel(const float* __restrict__ dq, const float* __restrict__ dk,
                                   const float* __restrict__ dv, const float* __restrict__ q_raw,
                                   const float* __restrict__ k_raw, const float* __restrict__ qw,
                                   const float* __restrict__ kw, const int* __restrict__ pos,
                                   const float* __restrict__ cs, const float* __restrict__ sn, int nh, int nkv, int hd,
                                   int rot, int neox, float eps, __half* __restrict__ dq16, __half* __restrict__ dk16,
                                   __half* __restrict__ dv16, float* __restrict__ sq, float* __restrict__ sk,
                                   float* __restrict__ sv) {
  extern __shared__ __align__(16) float buf[];  // [q heads | k heads | v heads] of this token, f32 results
  __shared__ float wmax[3][32];
  const size_t m = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int half = rot / 2;
  const int p = pos[m];
  const float* csr = cs + (size_t)p * half;
  const float* snr = sn + (size_t)p * half;
  float mx[3] = {0.f, 0.f, 0.f};
  for (int h = warp; h < nh + 2 * nkv; h += nwarps) {
    float* out = buf + (size_t)h * hd;
    if (h >= nh + nkv) {
      const float* src = dv + (m * nkv + (h - nh - nkv)) * hd;
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 v = *(const float4*)(src + i);
        *(float4*)(out + i) = v;
        mx[2] = fmaxf(mx[2], fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      }
      continue;
    }
    const bool is_q = h < nh;
    const float* g = is_q ? dq + (m * nh + h) * hd : dk + (m * nkv + (h - nh)) * hd;
    const float* xr = is_q ? q_raw + (m * nh + h) * hd : k_raw + (m * nkv + (h - nh)) * hd;
    const float* nw = is_q ? qw : kw;
    // inverse rotation (sin negated) into shared memory
    for (int i = lane * 2; i < half; i += 64) {
      const float2 c = *(const float2*)(csr + i), s = *(const float2*)(snr + i);
      if (neox) {
        const float2 x1 = *(const float2*)(g + i), x2 = *(const float2*)(g + i + half);
        *(float2*)(out + i) = make_float2(x1.x * c.x + x2.x * s.x, x1.y * c.y + x2.y * s.y);
        *(float2*)(out + i + half) = make_float2(x2.x * c.x - x1.x * s.x, x2.y * c.y - x1.y * s.y);
      } else {
        const float4 x = *(const float4*)(g + 2 * i);
        *(float4*)(out + 2 * i) = make_float4(x.x * c.x + x.y * s.x, x.y * c.x - x.x * s.x, x.z * c.y + x.w * s.y,
                                              x.w * c.y - x.z * s.y);
      }
    }
    for (int i = rot + lane; i < hd; i += 32) out[i] = g[i];
    __syncwarp();
    float mm = 0.f;
    if (nw) {
      float ss = 0.f, gx = 0.f;
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 xv = *(const float4*)(xr + i), ov = *(const float4*)(out + i), wv = *(const float4*)(nw + i);
        ss += xv.x * xv.x + xv.y * xv.y + xv.z * xv.z + xv.w * xv.w;
        gx += ov.x * wv.x * xv.x + ov.y * wv.y * xv.y + ov.z * wv.z * xv.z + ov.w * wv.w * xv.w;
      }
      ss = warp_sum(ss);
      gx = warp_sum(gx);
      const float ir = 1.0f / sqrtf(ss / (float)hd + eps);
      const float c = gx * ir * ir * ir / (float)hd;
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 xv = *(const float4*)(xr + i), ov = *(const float4*)(out + i), wv = *(const float4*)(nw + i);
        const float4 v = make_float4(ov.x * wv.x * ir - xv.x * c, ov.y * wv.y * ir - xv.y * c, ov.z * wv.z * ir - xv.z * c,
                                     ov.w * wv.w * ir - xv.w * c);
        *(float4*)(out + i) = v;
        mm = fmaxf(mm, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      }
    } else {
      for (int i = lane * 4; i < hd; i += 128) {
        const float4 v = *(const float4*)(out + i);
        mm = fmaxf(mm, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      }
    }
    mx[is_q ? 0 : 1] = fmaxf(mx[is_q ? 0 : 1], mm);
  }
  for (int k = 0; k < 3; ++k) {
    float v = warp_max(mx[k]);
    if (lane == 0) wmax[k][warp] = v;
  }
  __syncthreads();
  float s3[3];
  for (int k = 0; k < 3; ++k) {
    float v = 0.f;
    for (int w = 0; w < nwarps; ++w) v = fmaxf(v, wmax[k][w]);
    s3[k] = v;
  }
  if (threadIdx.x == 0) { sq[m] = s3[0]; sk[m] = s3[1]; sv[m] = s3[2]; }  // 0 for an all-zero row
  for (int k = 0; k < 3; ++k) s3[k] = s3[k] > 0.f ? s3[k] : 1.f;
  const int nq = nh * hd, nk = nkv * hd;
  const float i0 = 1.f / s3[0], i1 = 1.f / s3[1], i2 = 1.f / s3[2];
  for (int i = threadIdx.x * 4; i < nq + 2 * nk; i += blockDim.x * 4) {  // nq, nk are multiples of 4
    const float4 v = *(const float4*)(buf + i);
    const float inv = i < nq ? i0 : (i < nq + nk ? i1 : i2);
    __half* dst = i < nq ? dq16 + m * nq + i : (i < nq + nk ? dk16 + m * nk + (i - nq) : dv16 + m * nk + (i - nq - nk));
    __half2 a = __floats2half2_rn(v.x * inv, v.y * inv), b = __floats2half2_rn(v.z * inv, v.w * inv);
    *(uint2*)dst = make_uint2(*(uint32_t*)&a, *(uint32_t*)&b);
  }
}
void launch_qk_rope_bwd(const float* dq, const float* dk, const float* dv, const float* q_raw, const float* k_raw,
                        size_t raw_pitch, const float* qw, const float* kw, const int* pos, const float* cs, const float* sn,
                        int M, int nh, int nkv, int hd, int rot, int neox, float eps, __half* dq16, __half* dk16,
                        __half* dv16, size_t out_pitch, float* sq, float* sk, float* sv, cudaStream_t st) {
  if (M <= 0) return;
  int epl = 0, hpw = 0;
  // out_pitch != 0: the three outputs are slices of one matrix and share ONE scale per token
  const size_t pq = raw_pitch ? raw_pitch : (size_t)nh * hd, pk = raw_pitch ? raw_pitch : (size_t)nkv * hd;
  const size_t oq = out_pitch ? out_pitch : (size_t)nh * hd, ok = out_pitch ? out_pitch : (size_t)nkv * hd, ov = ok;
  const int common = out_pitch ? 1 : 0;
  if (hd == 128 && rot == hd && (qw != nullptr) == (kw != nullptr) && nh % 8 == 0 && nkv % 8 == 0) {
    const int qpw = nh / 8, kpw = nkv / 8;
#define RT_ROPE_BFAST_ARGS (dq, dk, dv, q_raw, k_raw, pq, pk, oq, ok, ov, common, qw, kw, pos, cs, sn, eps, dq16, dk16, dv16, sq, sk, sv)
#define RT_ROPE_BFAST(Q, K)                                                                            \
  if (qpw == Q && kpw == K) {                                                                          \
    if (neox) {                                                                                        \
      if (qw) pdl(qk_rope_bwd_fast_kernel<4, Q, K, true, true>, M, 256, 0, st) RT_ROPE_BFAST_ARGS;     \
      else pdl(qk_rope_bwd_fast_kernel<4, Q, K, true, false>, M, 256, 0, st) RT_ROPE_BFAST_ARGS;       \
    } else {                                                                                           \
      if (qw) pdl(qk_rope_bwd_fast_kernel<4, Q, K, false, true>, M, 256, 0, st) RT_ROPE_BFAST_ARGS;    \
      else pdl(qk_rope_bwd_fast_kernel<4, Q, K, false, false>, M, 256, 0, st) RT_ROPE_BFAST_ARGS;      \
    }                                                                                                  \
    RT_COUNT_LAUNCH(1);                                                                                \
    return;                                                                                            \
  }
    RT_ROPE_BFAST(2, 1)
    RT_ROPE_BFAST(3, 1)
    RT_ROPE_BFAST(4, 1)
    RT_ROPE_BFAST(4, 2)
    RT_ROPE_BFAST(1, 1)
#undef RT_ROPE_BFAST
#undef RT_ROPE_BFAST_ARGS
  }
  if (rope_reg_ok(nh, nkv, hd, rot, neox, &epl, &hpw)) {
#define RT_ROPE_BWD(E, H) pdl(qk_rope_bwd_reg_kernel<E, H>, M, 256, 0, st)(dq, dk, dv, q_raw, k_raw, pq, pk, oq, ok, ov, common, qw, kw, pos, cs, sn, nh, nkv, rot, neox, eps, dq16, dk16, dv16, sq, sk, sv)
    if (epl == 4) { if (hpw == 4) RT_ROPE_BWD(4, 4); else if (hpw == 6) RT_ROPE_BWD(4, 6); else RT_ROPE_BWD(4, 8); }
    else { if (hpw == 4) RT_ROPE_BWD(2, 4); else if (hpw == 6) RT_ROPE_BWD(2, 6); else RT_ROPE_BWD(2, 8); }
#undef RT_ROPE_BWD
  } else {
    size_t smem = (size_t)(nh + 2 * nkv) * hd * sizeof(float);
    qk_rope_bwd_kernel<<<M, 256, smem, st>>>(dq, dk, dv, q_raw, k_raw, qw, kw, pos, cs, sn, nh, nkv, hd, rot, neox, eps,
                                             dq16, dk16, dv16, sq, sk, sv);
  }
  RT_COUNT_LAUNCH(1);
}

// ------------------------------------------------------------------ SwiGLU (reference src/model.rs:113-134, src/tensor.rs:122-143)
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) {
  if (x >= 0.f) return 1.0f / (1.0f + expf(-x));
  float e = expf(x);
  return e / (1.0f + e);
}
// true when one of the eight f16 values is inf or NaN: the product left f16's range (the reference
// computes it in f32); the host gets RT_ERR_NONFINITE instead of a NaN loss
__device__ __forceinline__ bool any_nonfinite_f16x8(const uint4& o) {
  const uint32_t w[4] = {o.x, o.y, o.z, o.w};
  bool bad = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) bad |= ((w[k] & 0x7C00u) == 0x7C00u) | ((w[k] & 0x7C000000u) == 0x7C000000u);
  return bad;
}
__device__ __forceinline__ uint4 swiglu8(const uint4& gv, const uint4& uv) {
  const __half2* g2 = (const __half2*)&gv;
  const __half2* u2 = (const __half2*)&uv;
  uint4 o;
  __half2* o2 = (__half2*)&o;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 a = __half22float2(g2[k]), b = __half22float2(u2[k]);
    o2[k] = __floats2half2_rn(__fdividef(a.x, 1.0f + __expf(-a.x)) * b.x, __fdividef(a.y, 1.0f + __expf(-a.y)) * b.y);
  }
  return o;
}
__global__ void swiglu_fwd_kernel(const __half* g, const __half* u, __half* __restrict__ h,
                                  size_t n, int* status) {
  pdl_entry();
  size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i + 7 < n) {
    const uint4 o = swiglu8(*(const uint4*)(g + i), *(const uint4*)(u + i));
    *(uint4*)(h + i) = o;
    if (status && any_nonfinite_f16x8(o)) report_status(status, RT_ERR_NONFINITE);
  } else {
    for (; i < n; ++i) {
      const __half v = __float2half_rn(silu_f(__half2float(g[i])) * __half2float(u[i]));
      h[i] = v;
      if (status && (__hisinf(v) || __hisnan(v))) report_status(status, RT_ERR_NONFINITE);
    }
  }
}
// gate and up as column slices of one [rows x pitch] matrix (ff a multiple of 8)
__global__ void swiglu_fwd_pitched_kernel(const __half* g, const __half* u, size_t pitch, int ff,
                                          size_t n, __half* __restrict__ h, int* status) {
  pdl_entry();
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i >= n) return;
  const size_t r = i / ff, c = i % ff;
  const uint4 o = swiglu8(*(const uint4*)(g + r * pitch + c), *(const uint4*)(u + r * pitch + c));
  *(uint4*)(h + i) = o;
  if (status && any_nonfinite_f16x8(o)) report_status(status, RT_ERR_NONFINITE);
}
void launch_swiglu_fwd(const __half* g, const __half* u, size_t in_pitch, int rows, int ff, __half* h, int* status,
                       cudaStream_t st) {
  const size_t n = (size_t)rows * ff;
  if (n == 0) return;
  size_t threads = (n + 7) / 8;
  if (in_pitch && in_pitch != (size_t)ff && (ff & 7) == 0)
    pdl(swiglu_fwd_pitched_kernel, (unsigned)((threads + 255) / 256), 256, 0, st)(g, u, in_pitch, ff, n, h, status);
  else
    pdl(swiglu_fwd_kernel, (unsigned)((threads + 255) / 256), 256, 0, st)(g, u, h, n, status);
  RT_COUNT_LAUNCH(1);
}
// The product alone, of rows that are in memory, NT groups of LR_TOKENS of them per CTA; up to 16 rank indices and 2048 columns:
// every CTA reads all the weights, so that the tcgen05 stream, which reads them once for 64 or 128 tokens, is the better one where they
// are larger (4096 columns with 48 indices in a step of 1024 tokens 14 us against 5.8, 3072 with 16 at 8192 tokens 17.8 against
// 16.3).  2048 columns, 16 indices, in a step of 1024 tokens 5.8 -> 3.6 us, of 8192 as fast.
constexpr int LR_WARPS = 16, LR_MANY_K = 1024, LR_MANY_GROUPS = 2;
template <int NT>
__global__ void __launch_bounds__(32 * LR_WARPS) lowrank_rows_kernel(const __half* x, int K, int rows, const LowRank lr) {
  __shared__ __align__(16) float sums[lr_sum_floats(LR_WARPS, 1)];
  lr_prefetch(lr.w, lr.r, K);
  pdl_wait();
  pdl_launch_dependents();  // only now: QGemmArgs::late_wait
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m0 = (int)blockIdx.x * (LR_TOKENS * NT);
  const int r = m0 + (lane >> 2);
  const __half* xr = x + (size_t)r * K + (lane & 3) * 8;
  LrAcc<1> acc[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n].clear();
  LrWeights<1> w;
#pragma unroll 4
  for (int k = warp * 32; k < K; k += LR_WARPS * 32) {
    uint4 v[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) v[n] = r + n * LR_TOKENS < rows ? *(const uint4*)(xr + (size_t)(n * LR_TOKENS) * K + k) : make_uint4(0, 0, 0, 0);
    w.load(lr.w, lr.r, K, k, lane);
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n].add(w, v[n]);
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    if (n) __syncthreads();
    lr_finish<1, 1, LR_WARPS>(acc[n], sums, 0, warp, lane, m0 + n * LR_TOKENS, rows, lr.out);
  }
}
// The same sums for rows of up to 1024 columns and more tokens than the GPU holds at a time: two CTAs an SM that keep their warps' two
// blocks of the weights in registers and fetch the next tokens under the sums of these.  Bound: DRAM (1024 columns, 16 indices, 16384 tokens
// before a product of 1024 features: 43.3 us with a CTA for every 16 tokens, which all wait for their weights; 40.9 behind the
// tcgen05 stream; 39.4 so).
__global__ void __launch_bounds__(32 * LR_WARPS, 2) lowrank_rows_many_kernel(const __half* x, int K, int rows, const LowRank lr) {
  constexpr int NT = LR_MANY_GROUPS, NB = LR_MANY_K / 32 / LR_WARPS;
  __shared__ __align__(16) float sums[2][NT * lr_sum_floats(LR_WARPS, 1)];  // in turn: one barrier for each group
  lr_prefetch(lr.w, lr.r, K);
  pdl_wait();
  pdl_launch_dependents();  // only now: QGemmArgs::late_wait
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, step = (int)gridDim.x * (LR_TOKENS * NT);
  const __half* xr = x + (size_t)(lane >> 2) * K + warp * 32 + (lane & 3) * 8;
  int m0 = (int)blockIdx.x * (LR_TOKENS * NT);
  uint4 v[NB][NT];
  auto fetch = [&](int m) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int k = b * (LR_WARPS * 32), t = m + n * LR_TOKENS;
        v[b][n] = warp * 32 + k < K && t + (lane >> 2) < rows ? *(const uint4*)(xr + (size_t)t * K + k) : make_uint4(0, 0, 0, 0);
      }
  };
  fetch(m0);
  LrWeights<1> w[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int k = warp * 32 + b * (LR_WARPS * 32);
    w[b] = {};
    if (k < K) w[b].load(lr.w, lr.r, K, k, lane);
  }
  for (int buf = 0; m0 < rows; m0 += step, buf ^= 1) {
    LrAcc<1> acc[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      acc[n].clear();
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[n].add(w[b], v[b][n]);
    }
    fetch(m0 + step);
#pragma unroll
    for (int n = 0; n < NT; ++n) lr_put<1, LR_WARPS>(acc[n], sums[buf], n, warp, lane);
    __syncthreads();
    lr_sum<1, NT, LR_WARPS>(sums[buf], (int)threadIdx.x, m0, rows, lr.out);
  }
}
bool lowrank_rows_takes(int K, int r) { return K % 32 == 0 && K <= 2048 && r >= 1 && r <= 16; }
void launch_lowrank_rows(rt_ctx* c, const __half* x, int rows, int K, const LowRank& lr) {
  if (rows <= 0) return;
  constexpr int CTA = 2 * LR_TOKENS;  // tokens of a CTA beyond 2048 of them
  static_assert(CTA == LR_MANY_GROUPS * LR_TOKENS);
  const int at_a_time = 2 * c->num_sms;  // CTAs; from 6000 tokens on the persistent ones are faster (9000 of 1024: 25.7 -> 23.9 us), at 4096 as fast
  if (rows <= 2048) pdl(lowrank_rows_kernel<1>, (rows + LR_TOKENS - 1) / LR_TOKENS, 32 * LR_WARPS, 0, c->stream)(x, K, rows, lr);
  else if (K > LR_MANY_K || rows <= at_a_time * CTA) pdl(lowrank_rows_kernel<2>, (rows + CTA - 1) / CTA, 32 * LR_WARPS, 0, c->stream)(x, K, rows, lr);
  else pdl(lowrank_rows_many_kernel, at_a_time, 32 * LR_WARPS, 0, c->stream)(x, K, rows, lr);
  RT_COUNT_LAUNCH(1);
}
// dg = dh*u*silu'(g), du = dh*silu(g); both written row-normalised in f16 with per-row scales.
// The kernel is bound by the exp/divide per element, so sigma is computed once per element with
// the fast intrinsics (2 ulp, far inside the f16 rounding that follows) and the products are
// kept in registers between the max pass and the write pass.
__device__ __forceinline__ float ld1f(const float* p) { return *p; }
__device__ __forceinline__ float ld1f(const __half* p) { return __half2float(*p); }

template <typename DT>
struct Raw8;  // eight elements as loaded
template <>
struct Raw8<__half> {
  uint4 v;
  __device__ __forceinline__ void load(const __half* p) { v = *(const uint4*)p; }
  __device__ __forceinline__ float2 pair(int k) const { return __half22float2(((const __half2*)&v)[k]); }
};
template <>
struct Raw8<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) { a = *(const float4*)p; b = *(const float4*)(p + 4); }
  __device__ __forceinline__ float2 pair(int k) const {
    return k == 0 ? make_float2(a.x, a.y) : k == 1 ? make_float2(a.z, a.w) : k == 2 ? make_float2(b.x, b.y) : make_float2(b.z, b.w);
  }
};
template <typename DT>
__device__ __forceinline__ void swiglu_grad8(const Raw8<DT>& dh, const Raw8<__half>& g, const Raw8<__half>& u, float* dg, float* du) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 d = dh.pair(k), a = g.pair(k), b = u.pair(k);
    const float s0 = __fdividef(1.0f, 1.0f + __expf(-a.x)), s1 = __fdividef(1.0f, 1.0f + __expf(-a.y));
    dg[2 * k] = d.x * b.x * (s0 * (1.0f + a.x * (1.0f - s0)));
    dg[2 * k + 1] = d.y * b.y * (s1 * (1.0f + a.y * (1.0f - s1)));
    du[2 * k] = d.x * (a.x * s0);
    du[2 * k + 1] = d.y * (a.y * s1);
  }
}
// dh is f32, or f16 rows that still lack their per-row factor in_scale[r] (which then only
// multiplies the two output scales).
template <typename DT>  // NCH 8-element chunks per thread, kept in registers: ff <= NCH * 8 * blockDim.x, ff % 8 == 0
__global__ void __launch_bounds__(512) swiglu_bwd_cached_kernel(const DT* dh, const float* in_scale,
                                         const __half* g,
                                         const __half* u, size_t gp, int ff, __half* __restrict__ dg16,
                                         __half* __restrict__ du16, size_t op, int common, float* __restrict__ sg,
                                         float* __restrict__ su) {
  pdl_entry();
  const size_t r = blockIdx.x;
  constexpr int NCH = 3;
  Raw8<DT> rd[NCH];
  Raw8<__half> rg[NCH], ru[NCH];
#pragma unroll
  for (int c = 0; c < NCH; ++c) {  // every load before the first use
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    if (i < ff) {
      rd[c].load(dh + r * ff + i);
      rg[c].load(g + r * gp + i);
      ru[c].load(u + r * gp + i);
    }
  }
  float a[NCH][8], b[NCH][8];
  float mg = 0.f, mu = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    if (i < ff) {
      swiglu_grad8(rd[c], rg[c], ru[c], a[c], b[c]);
#pragma unroll
      for (int k = 0; k < 8; ++k) { mg = fmaxf(mg, fabsf(a[c][k])); mu = fmaxf(mu, fabsf(b[c][k])); }
    }
  }
  {  // both row maxima through one barrier (magnitudes: 0 is the identity)
    __shared__ float shg[32], shu[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    mg = warp_max(mg);
    mu = warp_max(mu);
    if (lane == 0) { shg[w] = mg; shu[w] = mu; }
    __syncthreads();
    mg = mu = 0.f;
    for (int k = 0; k < nw; ++k) { mg = fmaxf(mg, shg[k]); mu = fmaxf(mu, shu[k]); }
  }
  if (common) mg = mu = fmaxf(mg, mu);  // gate and up gradients form ONE matrix with one scale per row
  const float s_g = mg > 0.f ? mg : 1.f, s_u = mu > 0.f ? mu : 1.f;
  const float ig = 1.f / s_g, iu = 1.f / s_u;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int i = (c * blockDim.x + threadIdx.x) * 8;
    if (i < ff) {
      uint4 oa, ob;
      __half2* pa = (__half2*)&oa;
      __half2* pb = (__half2*)&ob;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        pa[k] = __floats2half2_rn(a[c][2 * k] * ig, a[c][2 * k + 1] * ig);
        pb[k] = __floats2half2_rn(b[c][2 * k] * iu, b[c][2 * k + 1] * iu);
      }
      *(uint4*)(dg16 + r * op + i) = oa;
      *(uint4*)(du16 + r * op + i) = ob;
    }
  }
  if (threadIdx.x == 0) {
    const float f = in_scale ? in_scale[r] : 1.0f;
    sg[r] = mg * f;  // 0 for an all-zero row
    su[r] = mu * f;
  }
}
// general row length: scalar, recomputed in the second pass
template <typename DT>
__global__ void swiglu_bwd_kernel(const DT* __restrict__ dh, const float* __restrict__ in_scale, const __half* __restrict__ g,
                                  const __half* __restrict__ u, size_t gp, int ff, __half* __restrict__ dg16,
                                  __half* __restrict__ du16, size_t op, int common, float* __restrict__ sg,
                                  float* __restrict__ su) {
  const size_t r = blockIdx.x;
  const DT* dhr = dh + r * ff;
  const __half* gr = g + r * gp;
  const __half* ur = u + r * gp;
  float mg = 0.f, mu = 0.f;
  for (int i = threadIdx.x; i < ff; i += blockDim.x) {
    const float gv = __half2float(gr[i]), uv = __half2float(ur[i]), d = ld1f(dhr + i);
    const float s = sigmoid_f(gv);
    mg = fmaxf(mg, fabsf(d * uv * (s * (1.0f + gv * (1.0f - s)))));
    mu = fmaxf(mu, fabsf(d * silu_f(gv)));
  }
  mg = block_max(mg);
  mu = block_max(mu);
  if (common) mg = mu = fmaxf(mg, mu);
  const float s_g = mg > 0.f ? mg : 1.f, s_u = mu > 0.f ? mu : 1.f;
  const float ig = 1.f / s_g, iu = 1.f / s_u;
  for (int i = threadIdx.x; i < ff; i += blockDim.x) {
    const float gv = __half2float(gr[i]), uv = __half2float(ur[i]), d = ld1f(dhr + i);
    const float s = sigmoid_f(gv);
    dg16[r * op + i] = __float2half_rn(d * uv * (s * (1.0f + gv * (1.0f - s))) * ig);
    du16[r * op + i] = __float2half_rn(d * silu_f(gv) * iu);
  }
  if (threadIdx.x == 0) {
    const float f = in_scale ? in_scale[r] : 1.0f;
    sg[r] = mg * f;  // 0 for an all-zero row
    su[r] = mu * f;
  }
}
template <typename DT>
static void launch_swiglu_bwd_t(const DT* dh, const float* in_scale, const __half* g, const __half* u, size_t gp, int rows,
                                int ff, __half* dg16, __half* du16, size_t op, int common, float* sg, float* su,
                                cudaStream_t st) {
  // Three chunks of eight elements per thread and as many threads as that takes: no idle threads, and
  // several rows per SM at any width.  (512 threads for every row above 4096 left two thirds of them
  // idle on 4864 columns and one row per SM: 8192 rows 181 us, 8192 columns 269 us; floor 62 and 104.)
  const int threads = (((ff >> 3) + 2) / 3 + 31) & ~31;
  if ((ff & 7) == 0 && threads <= 512) pdl(swiglu_bwd_cached_kernel<DT>, rows, threads, 0, st)(dh, in_scale, g, u, gp, ff, dg16, du16, op, common, sg, su);
  else swiglu_bwd_kernel<DT><<<rows, 256, 0, st>>>(dh, in_scale, g, u, gp, ff, dg16, du16, op, common, sg, su);
  RT_COUNT_LAUNCH(1);
}
void launch_swiglu_bwd(const void* dh, int dh_f16, const float* in_scale, const __half* g, const __half* u, size_t in_pitch,
                       int rows, int ff, __half* dg16, __half* du16, size_t out_pitch, float* sg, float* su, cudaStream_t st) {
  if (rows <= 0) return;
  // in_pitch / out_pitch = 0: separate row-major matrices; else gate|up (dg|du) are slices of one
  // matrix with that row pitch, and with out_pitch the two outputs share one scale per row
  const size_t gp = in_pitch ? in_pitch : (size_t)ff, op = out_pitch ? out_pitch : (size_t)ff;
  const int common = out_pitch ? 1 : 0;
  if (dh_f16) launch_swiglu_bwd_t((const __half*)dh, in_scale, g, u, gp, rows, ff, dg16, du16, op, common, sg, su, st);
  else launch_swiglu_bwd_t((const float*)dh, in_scale, g, u, gp, rows, ff, dg16, du16, op, common, sg, su, st);
}

// ------------------------------------------------------------------ row gather / scatter
__global__ void gather_f32_rows_kernel(const float* x, const int* __restrict__ idx, int d,
                                       float* __restrict__ out) {
  pdl_entry();
  const size_t r = blockIdx.x;
  const float* src = x + (size_t)idx[r] * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) out[r * d + i] = src[i];
}
void launch_gather_f32_rows(const float* x, const int* idx, int rows, int d, float* out, cudaStream_t st) {
  if (rows > 0) { pdl(gather_f32_rows_kernel, rows, 256, 0, st)(x, idx, d, out); RT_COUNT_LAUNCH(1); }
}
// dx[idx[r], :] += src[r, :]   (atomic: two targets may name the same position)
__global__ void scatter_add_rows_kernel(const float* src, const int* __restrict__ idx, int d,
                                        float* dx) {
  pdl_entry();
  const size_t r = blockIdx.x;
  float* dst = dx + (size_t)idx[r] * d;
  for (int i = threadIdx.x; i < d; i += blockDim.x) atomicAdd(dst + i, src[r * d + i]);
}
void launch_scatter_add_rows(const float* src, const int* idx, int rows, int d, float* dx, cudaStream_t st) {
  if (rows > 0) { pdl(scatter_add_rows_kernel, rows, 256, 0, st)(src, idx, d, dx); RT_COUNT_LAUNCH(1); }
}

// ------------------------------------------------------------------ cross-entropy over one row of logits
// (reference src/model.rs:579-596, src/ops.rs:238-247): lse with an f64 normaliser, logp of
// the target, hit = no logit above the target's, and d16 = p - onehot in f16 with the row scale
// w (so dlogits = w*(p - onehot) exactly as the reference forms it).
// The greedy token of a row: the LAST index holding the maximum, which is what the reference's
// Iterator::max_by(total_cmp) returns on ties (src/eval.rs:167).  One more read of the row.
__device__ void ce_row_argmax(const float* row, int v, float m, int* __restrict__ out) {
  __shared__ int s_arg[32];
  int best = -1;
  for (int i = threadIdx.x; i < v; i += blockDim.x)
    if (row[i] == m) best = i;  // i grows: the thread keeps its last
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_arg[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = threadIdx.x < (blockDim.x + 31) / 32 ? s_arg[threadIdx.x] : -1;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, off));
    if (threadIdx.x == 0) *out = best;
  }
}

__global__ void ce_row_kernel(const float* logits, int v, const int* __restrict__ target,
                              const float* __restrict__ weight, float* __restrict__ logp, int* hits,
                              __half* __restrict__ d16, float* __restrict__ scale, int* __restrict__ argmax, int* status) {
  pdl_entry();
  const size_t r = blockIdx.x;
  const float* row = logits + r * v;
  const int tgt = target[r];
  if (tgt < 0 || tgt >= v) {
    if (threadIdx.x == 0) report_status(status, RT_ERR_BAD_INDEX);
    return;
  }
  float m = -INFINITY;
  for (int i = threadIdx.x; i < v; i += blockDim.x) m = fmaxf(m, row[i]);
  m = block_max(m);
  double s = 0.0;
  for (int i = threadIdx.x; i < v; i += blockDim.x) s += (double)expf(row[i] - m);
  s = block_sum_d(s);
  const float tl = row[tgt];
  if (threadIdx.x == 0) {
    logp[r] = tl - (m + (float)log(s));
    if (tl >= m) atomicAdd(hits, 1);
    if (scale) scale[r] = weight[r];
  }
  if (argmax) ce_row_argmax(row, v, m, argmax + r);
  if (d16) {
    const float inv = (float)(1.0 / s);
    for (int i = threadIdx.x; i < v; i += blockDim.x) {
      float p = expf(row[i] - m) * inv;
      if (i == tgt) p -= 1.0f;
      d16[r * v + i] = __float2half_rn(p);
    }
  }
}
// The same for rows whose length is a multiple of 4: 128-bit loads, the maximum and the sum found in ONE
// pass (each thread keeps a running maximum and rescales its partial sum when the maximum moves; the partial
// sums meet in f64).  What the chip can hold of the row's exponentials stays there for the second pass: five
// float4 per thread in registers and twelve in shared memory, each chunk of them relative to the running
// maximum it met (one factor per chunk brings them to the row's); the rest, half of 151936 columns, is
// still in L2, with one block per SM, and is read and exponentiated again.  What bounds it: the stream of
// logits in and gradients out, 0.93 GB for 1024 rows of 151936 columns (141 us at the copy rate), and
// the exponentials.  1024 rows: 262 us with everything read twice by two blocks per SM, 201 so, 246 keeping the
// logits instead of the exponentials, 247 as two blocks of 512 threads, 274 as a cluster of eight
// blocks that reads each logit once into registers (nothing runs under its reductions).
constexpr int CE_THREADS = 1024, CE_REG4 = 5, CE_CHUNK_BYTES = 4 * CE_THREADS * 16;
__global__ void __launch_bounds__(CE_THREADS, 1)
ce_row_vec_kernel(const float* logits, int v, const int* __restrict__ target,
                  const float* __restrict__ weight, float* __restrict__ logp, int* hits,
                  __half* __restrict__ d16, float* __restrict__ scale, int* __restrict__ argmax, int* status, int n_chunks) {
  extern __shared__ float4 s_row[];  // [n_chunks <= 3][4][CE_THREADS]
  pdl_entry();
  const size_t r = blockIdx.x;
  const float4* row4 = (const float4*)(logits + r * v);
  const int n4 = v >> 2, tid = threadIdx.x;
  const int tgt = target[r];
  if (tgt < 0 || tgt >= v) {
    if (tid == 0) report_status(status, RT_ERR_BAD_INDEX);
    return;
  }
  const float4 none = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
  float mt = -INFINITY, st = 0.f;
  auto max4 = [](const float4& x) { return fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)); };
  auto take = [&](float cm) {  // a chunk's maximum joins the running one
    if (cm > mt) { st *= expf(mt - cm); mt = cm; }  // expf(-inf) = 0 on the first chunk
    return mt > -INFINITY ? mt : 0.f;
  };
  auto exp4 = [](const float4& x, float ref) { return make_float4(expf(x.x - ref), expf(x.y - ref), expf(x.z - ref), expf(x.w - ref)); };
  auto add4 = [&](const float4& e) { st += (e.x + e.y) + (e.z + e.w); };
  float4 keep[CE_REG4];
#pragma unroll
  for (int k = 0; k < CE_REG4; ++k) {
    const int i = tid + k * CE_THREADS;
    keep[k] = i < n4 ? __ldcs(row4 + i) : none;
  }
  float cm = -INFINITY;
#pragma unroll
  for (int k = 0; k < CE_REG4; ++k) cm = fmaxf(cm, max4(keep[k]));
  const float ref0 = take(cm);
#pragma unroll
  for (int k = 0; k < CE_REG4; ++k) {
    keep[k] = exp4(keep[k], ref0);
    add4(keep[k]);
  }
  float ref[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    ref[c] = 0.f;
    if (c >= n_chunks) continue;
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = (CE_REG4 + c * 4 + k) * CE_THREADS + tid;
      x[k] = i < n4 ? __ldcs(row4 + i) : none;
    }
    ref[c] = take(fmaxf(fmaxf(max4(x[0]), max4(x[1])), fmaxf(max4(x[2]), max4(x[3]))));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 e = exp4(x[k], ref[c]);
      add4(e);
      s_row[(c * 4 + k) * CE_THREADS + tid] = e;
    }
  }
  const int i_rest = (CE_REG4 + n_chunks * 4) * CE_THREADS + tid;
  for (int i0 = i_rest; i0 < n4; i0 += 4 * CE_THREADS) {
    float4 x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k] = i0 + k * CE_THREADS < n4 ? row4[i0 + k * CE_THREADS] : none;
    const float rf = take(fmaxf(fmaxf(max4(x[0]), max4(x[1])), fmaxf(max4(x[2]), max4(x[3]))));
#pragma unroll
    for (int k = 0; k < 4; ++k) add4(exp4(x[k], rf));
  }
  const float m = block_max(mt);
  const double s = block_sum_d(mt > -INFINITY ? (double)st * (double)expf(mt - m) : 0.0);
  const float tl = logits[r * v + tgt];
  if (tid == 0) {
    logp[r] = tl - (m + (float)log(s));
    if (tl >= m) atomicAdd(hits, 1);
    if (scale) scale[r] = weight[r];
  }
  if (argmax) ce_row_argmax(logits + r * v, v, m, argmax + r);
  if (d16) {
    const float inv = (float)(1.0 / s);
    uint2* out = (uint2*)(d16 + r * v);
    const int t4 = tgt >> 2, tk = tgt & 3;
    auto put = [&](int i, const float4& e, float f) {
      float p0 = e.x * f, p1 = e.y * f, p2 = e.z * f, p3 = e.w * f;
      if (i == t4) {
        if (tk == 0) p0 -= 1.0f; else if (tk == 1) p1 -= 1.0f; else if (tk == 2) p2 -= 1.0f; else p3 -= 1.0f;
      }
      const __half2 a = __floats2half2_rn(p0, p1), b = __floats2half2_rn(p2, p3);
      __stcs(out + i, make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b));
    };
    for (int i0 = i_rest; i0 < n4; i0 += 4 * CE_THREADS) {
      float4 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i0 + k * CE_THREADS < n4) x[k] = __ldcs(row4 + i0 + k * CE_THREADS);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i0 + k * CE_THREADS < n4) put(i0 + k * CE_THREADS, exp4(x[k], m), inv);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (c >= n_chunks) continue;
      const float f = expf(ref[c] - m) * inv;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = (CE_REG4 + c * 4 + k) * CE_THREADS + tid;
        if (i < n4) put(i, s_row[(c * 4 + k) * CE_THREADS + tid], f);
      }
    }
    const float f0 = expf(ref0 - m) * inv;
#pragma unroll
    for (int k = 0; k < CE_REG4; ++k)
      if (tid + k * CE_THREADS < n4) put(tid + k * CE_THREADS, keep[k], f0);
  }
}
int launch_ce_rows(rt_ctx* c, const float* logits, int rows, int v, const int* target, const float* weight, float* logp, int* hits,
                   __half* d16, float* scale, int* argmax) {
  if (rows <= 0) return 0;
  cudaError_t e;
  if ((v & 3) == 0 && ((uintptr_t)logits & 15) == 0 && (d16 == nullptr || ((uintptr_t)d16 & 7) == 0)) {
    const int left = v / 4 - CE_REG4 * CE_THREADS;  // float4s beyond the registers; a row without gradient is read once and needs no place
    const int n_chunks = d16 && left > 0 ? std::min(3, (left + 4 * CE_THREADS - 1) / (4 * CE_THREADS)) : 0;
    if (n_chunks > 0 && !c->raise_smem(ce_row_vec_kernel, 3 * CE_CHUNK_BYTES)) return 3;
    e = pdl(ce_row_vec_kernel, rows, CE_THREADS, n_chunks * CE_CHUNK_BYTES, c->stream)(logits, v, target, weight, logp, hits, d16, scale, argmax,
                                                                                     c->status_dev, n_chunks);
  } else {
    e = pdl(ce_row_kernel, rows, 1024, 0, c->stream)(logits, v, target, weight, logp, hits, d16, scale, argmax, c->status_dev);
  }
  RT_COUNT_LAUNCH(1);
  return e == cudaSuccess ? 0 : 3;
}

// ------------------------------------------------------------------ LoRA shadows and gradients
// 16-bit operand copies of one adapter, rebuilt after every parameter update:
//   a_s  [r x K]  f16 = s*A      (weight of Hs = X.(sA)^T)
//   a_h  [r x K]  f16 = A        (extra rows of the backward matmul: dX += Gs.A)
//   bp   [N x 64] f16 = B, zero padded (extra columns of the forward matmul: Y += Hs.B^T)
//   bt_s [r x N]  f16 = s*B^T    (weight of Gs = dY.(sB))
__global__ void lora_refresh_kernel(const float* __restrict__ a, const float* __restrict__ b, int r, int K, int N,
                                    float s, __half* a_s, __half* a_h, __half* bp, __half* bt_s) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t na = (size_t)r * K, nb = (size_t)N * 64;
  if (i < na) {
    a_s[i] = __float2half_rn(a[i] * s);
    a_h[i] = __float2half_rn(a[i]);
  }
  if (i < nb) {
    const int n = (int)(i / 64), j = (int)(i % 64);
    const float v = j < r ? b[(size_t)n * r + j] : 0.f;
    bp[i] = __float2half_rn(v);
    if (j < r) bt_s[(size_t)j * N + n] = __float2half_rn(v * s);
  }
}
// The same copies of one adapter written into the stacked operands of a group of linears that
// share their input (q|k|v, gate|up): a_s / a_h are this adapter's rows of [R x K]; bp points at
// (this linear's first row, this adapter's first column) of [N_total x 64]; bt_s at (this
// adapter's first row, this linear's first column) of [R x N_total], row pitch ldb.
__global__ void lora_refresh_group_kernel(const float* __restrict__ a, const float* __restrict__ b, int r, int K, int N,
                                          float s, __half* a_s, __half* a_h, __half* bp, __half* bt_s, size_t ldb) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t na = (size_t)r * K, nb = (size_t)N * r;
  if (i < na) {
    a_s[i] = __float2half_rn(a[i] * s);
    a_h[i] = __float2half_rn(a[i]);
  }
  if (i < nb) {
    const int n = (int)(i / r), j = (int)(i % r);
    const float v = b[i];
    bp[(size_t)n * 64 + j] = __float2half_rn(v);
    bt_s[(size_t)j * ldb + n] = __float2half_rn(v * s);
  }
}
// Every stale adapter of a model in one launch: a block finds its row of the table by counting the rows that start no later, then
// does what the two kernels above do for one adapter, eight elements a thread with their loads in flight together.  What goes down
// bt_s is turned round in shared memory, so that a warp writes neighbours of a row of it.  (Two bytes into each of 16 rows at a
// time: 55 us for the 196 adapters of the 0.6B shape at rank 16, 115 MB; now 46.)
__global__ void __launch_bounds__(256) lora_refresh_table_kernel(const LoraRefreshJob* __restrict__ jobs, int n_jobs) {
  // [rank index][rows of b], rows an odd number of words apart where a block's rows are a power of two
  __shared__ __half turned[LORA_REFRESH_PER_BLOCK + 5 * 64];
  int row = -1;
  for (int t = 0; t < n_jobs; t += 256)
    row += __syncthreads_count(t + (int)threadIdx.x < n_jobs && jobs[t + threadIdx.x].first_block <= blockIdx.x);
  const LoraRefreshJob j = jobs[row];
  constexpr int PT = LORA_REFRESH_PER_BLOCK / 256;
  const size_t first = (size_t)(blockIdx.x - j.first_block) * LORA_REFRESH_PER_BLOCK, i0 = first + threadIdx.x;
  const unsigned width = j.pad64 ? 64u : (unsigned)j.r;  // elements of a row of b as they are counted
  const size_t na = (size_t)j.r * j.K, nb = (size_t)j.N * width;
  float va[PT], vb[PT];
  unsigned n[PT], c[PT];
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const size_t i = i0 + k * 256;
    va[k] = i < na ? j.a[i] : 0.f;
    n[k] = j.pad64 ? (unsigned)(i >> 6) : (unsigned)i / (unsigned)j.r;
    c[k] = (unsigned)i - n[k] * width;
    vb[k] = i < nb && c[k] < (unsigned)j.r ? j.b[(size_t)n[k] * j.r + c[k]] : 0.f;
  }
  const unsigned n0 = (unsigned)first / width, rows = ((unsigned)first + LORA_REFRESH_PER_BLOCK - 1) / width - n0 + 1, pitch = (rows + 1) / 2 * 2 + 2;
#pragma unroll
  for (int k = 0; k < PT; ++k) {
    const size_t i = i0 + k * 256;
    if (i < na) {
      j.a_s[i] = __float2half_rn(va[k] * j.s);
      j.a_h[i] = __float2half_rn(va[k]);
    }
    if (i < nb) {
      j.bp[(size_t)n[k] * 64 + c[k]] = __float2half_rn(vb[k]);
      if (c[k] < (unsigned)j.r) turned[c[k] * pitch + (n[k] - n0)] = __float2half_rn(vb[k] * j.s);
    }
  }
  __syncthreads();
  for (unsigned e = threadIdx.x; e < (unsigned)j.r * rows; e += 256) {
    const unsigned cc = e / rows, m = e - cc * rows;
    const size_t i = (size_t)(n0 + m) * width + cc;  // (a row that two blocks share: each writes its own part)
    if (i >= first && i < first + LORA_REFRESH_PER_BLOCK && i < nb) j.bt_s[(size_t)cc * j.ldb + n0 + m] = turned[cc * pitch + m];
  }
}
void launch_lora_refresh_table(const LoraRefreshJob* jobs_dev, int n_jobs, unsigned total_blocks, cudaStream_t st) {
  if (n_jobs <= 0 || total_blocks == 0) return;
  { lora_refresh_table_kernel<<<total_blocks, 256, 0, st>>>(jobs_dev, n_jobs); RT_COUNT_LAUNCH(1); }
}
void launch_lora_refresh_group(const float* a, const float* b, int r, int K, int N, float s, __half* a_s, __half* a_h,
                               __half* bp, __half* bt_s, size_t ldb, cudaStream_t st) {
  size_t n = (size_t)r * K > (size_t)N * r ? (size_t)r * K : (size_t)N * r;
  { lora_refresh_group_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, b, r, K, N, s, a_s, a_h, bp, bt_s, ldb); RT_COUNT_LAUNCH(1); }
}
void launch_lora_refresh(const float* a, const float* b, int r, int K, int N, float s, __half* a_s, __half* a_h,
                         __half* bp, __half* bt_s, cudaStream_t st) {
  size_t n = (size_t)r * K > (size_t)N * 64 ? (size_t)r * K : (size_t)N * 64;
  { lora_refresh_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(a, b, r, K, N, s, a_s, a_h, bp, bt_s); RT_COUNT_LAUNCH(1); }
}

// ------------------------------------------------------------------ optimiser (reference src/optim.rs:48-90)
// Sum of squares in f64: fixed-size blocks write partials, one block adds them in order.
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const float* __restrict__ g, size_t n, double* __restrict__ part) {
  const size_t at = (size_t)blockIdx.x * blockDim.x + threadIdx.x, step = (size_t)gridDim.x * blockDim.x, n4 = n / 4;
  double s = 0.0;
  for (size_t i = at; i < n4; i += 4 * step) {
    float4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k * step < n4 ? ((const float4*)g)[i + k * step] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double x = v[k].x, y = v[k].y, z = v[k].z, w = v[k].w;
      s += x * x + y * y + (z * z + w * w);
    }
  }
  if (at < n % 4) s += (double)g[4 * n4 + at] * (double)g[4 * n4 + at];
  s = block_sum_d(s);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}
__global__ void sumsq_final_kernel(const double* __restrict__ part, int n, double* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  s = block_sum_d(s);
  if (threadIdx.x == 0) out[0] = s;
}
void launch_sumsq(const float* g, size_t n, double* part /* >= 1024 */, double* out, cudaStream_t st) {
  // sixteen values a thread, at most what is on the GPU at a time and `part` has room for
  const int blocks = (int)std::min<size_t>(1024, std::max<size_t>(1, (n + 4095) / 4096));
  { sumsq_partial_kernel<<<blocks, 256, 0, st>>>(g, n, part); RT_COUNT_LAUNCH(1); }
  { sumsq_final_kernel<<<1, 256, 0, st>>>(part, blocks, out); RT_COUNT_LAUNCH(1); }
}
// clip (scale read from the device-side norm) fused with the AdamW update.  Bound: DRAM, four arrays read and three or, where the norm
// clips, four written; four parameters a thread (10 million: one a thread 81 us, now 41; the copy rate would take 49 with the gradients' write).
__device__ __forceinline__ void adamw_one(float& p, float& g, float& m, float& v, float clip, float lr, float beta1, float beta2, float eps, float wd,
                                          float bc1, float bc2) {
  if (clip != 1.0f) g *= clip;
  m = beta1 * m + (1.0f - beta1) * g;
  v = beta2 * v + (1.0f - beta2) * g * g;
  const float mh = m / bc1, vh = v / bc2;
  p -= lr * (mh / (sqrtf(vh) + eps) + wd * p);
}
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                                                    size_t n, const double* __restrict__ sumsq, float max_norm, float lr, float beta1,
                                                    float beta2, float eps, float wd, float bc1, float bc2, float* __restrict__ norm_out) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, i = 4 * t;
  const bool whole = i + 3 < n;
  float4 pv, gv, mv, vv;
  if (whole) {  // before the norm, a load that these do not depend on
    pv = *(const float4*)(p + i); gv = *(const float4*)(g + i); mv = *(const float4*)(m + i); vv = *(const float4*)(v + i);
  }
  const float norm = (float)sqrt(sumsq[0]);
  float clip = 1.0f;
  if (max_norm > 0.f && norm > max_norm) clip = max_norm / (norm + 1e-6f);
  if (t == 0 && norm_out) norm_out[0] = norm;
  if (whole) {
    adamw_one(pv.x, gv.x, mv.x, vv.x, clip, lr, beta1, beta2, eps, wd, bc1, bc2);
    adamw_one(pv.y, gv.y, mv.y, vv.y, clip, lr, beta1, beta2, eps, wd, bc1, bc2);
    adamw_one(pv.z, gv.z, mv.z, vv.z, clip, lr, beta1, beta2, eps, wd, bc1, bc2);
    adamw_one(pv.w, gv.w, mv.w, vv.w, clip, lr, beta1, beta2, eps, wd, bc1, bc2);
    *(float4*)(p + i) = pv;
    if (clip != 1.0f) *(float4*)(g + i) = gv;
    *(float4*)(m + i) = mv;
    *(float4*)(v + i) = vv;
  } else {
    for (size_t k = i; k < n; ++k) adamw_one(p[k], g[k], m[k], v[k], clip, lr, beta1, beta2, eps, wd, bc1, bc2);
  }
}
void launch_adamw(float* p, float* g, float* m, float* v, size_t n, const double* sumsq, float max_norm, float lr,
                  float beta1, float beta2, float eps, float wd, float bc1, float bc2, float* norm_out,
                  cudaStream_t st) {
  if (n == 0) return;
  { adamw_kernel<<<(unsigned)((n + 1023) / 1024), 256, 0, st>>>(p, g, m, v, n, sumsq, max_norm, lr, beta1, beta2, eps, wd,
                                                               bc1, bc2, norm_out); RT_COUNT_LAUNCH(1); }
}

}  // namespace rt
