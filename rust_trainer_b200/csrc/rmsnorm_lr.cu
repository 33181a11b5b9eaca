// RMSNorm forward and backward with the low-rank product of their 16-bit rows (lowrank_rows.cuh): persistent CTAs of NT groups of eight warps that
// keep the product's weights in shared memory, a warp per row; the rows' f16 copies go into shared memory as well as to where they belong.
// Bound: the chain of launches at 1024 rows (forward 3.8 us + 5 for a low-rank launch of its own -> 4.3; backward 6.2 + 4.8 ->
// 5.1, and the matmul behind it finds all SMs free), DRAM at 8192 (forward with 48 rank indices 17.2 -> 15.3 us, backward 29.1 -> 28.1;
// with the weights read from L2 by every eight rows 21.5 and 33).
//
// A file of its own: CUDA loads a file's kernels with the first of them.  These are eight widths by four rank groups by four forms, and among
// the other row kernels they made a process's first linear call 17 ms instead of 7, its first pass over a small model 18 instead of 12.
#include "ctx.h"
#include "lowrank_rows.cuh"
#include "ops.h"
#include "pdl.cuh"
#include "rmsnorm_row.cuh"
#include <algorithm>

namespace rt {

template <int NV, int MT, int NT>
struct RmsLr {
  static constexpr int D = 128 * NV, PITCH = lr_row_pitch(D);  // of weights and rows
  static constexpr int TILE = NT * LR_TOKENS * PITCH, SUMS = NT * lr_sum_floats(LR_SLICES, MT) * 4;
  static constexpr int bytes(int r) { return TILE + SUMS + r * PITCH; }
  static constexpr int ctas(int most) {  // of an SM
    const int fit = SMEM_PER_SM / (bytes(16 * MT) + 1024);
    return fit < most ? fit : most;
  }
  static constexpr int FWD_CTAS = ctas(4 / NT), BWD_CTAS = ctas(2);
};
template <int NV, int MT, int NT>
__global__ void __launch_bounds__(256 * NT, (RmsLr<NV, MT, NT>::FWD_CTAS))
rmsnorm_fwd_lr_kernel(const float* x, const float* __restrict__ w, int rows, float eps, __half* __restrict__ y16,
                      const LowRank lr) {
  using C = RmsLr<NV, MT, NT>;
  extern __shared__ __align__(16) uint8_t lr_smem[];
  uint8_t* tile = lr_smem;
  float* sums = (float*)(lr_smem + C::TILE);
  uint8_t* weights = lr_smem + C::TILE + C::SUMS;
  pdl_launch_dependents();
  lr_prefetch(lr.w, lr.r, C::D);
  pdl_wait();
  lr_fetch_weights(lr.w, lr.r, C::D, weights, C::PITCH);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int step = (int)gridDim.x * 8 * NT;
  float4 v[NV];
  int r = (int)blockIdx.x * 8 * NT + warp;
  if (r < rows) rms_load_row<NV>(x + (size_t)r * C::D, lane, v);
  for (; r - warp < rows; r += step) {
    uint8_t* t = tile + warp * C::PITCH + 8 * lane;
    if (r < rows)
      rms_fwd_row<NV>(v, w, eps, lane, [&](int k, uint2 o) {
        *(uint2*)(y16 + (size_t)r * C::D + 4 * (lane + 32 * k)) = o;
        *(uint2*)(t + 256 * k) = o;
      });
    if (r + step < rows) rms_load_row<NV>(x + (size_t)(r + step) * C::D, lane, v);  // the next rows, under this one's product
    cp_async_wait<0>();
    __syncthreads();
    lr_of_rows<MT, NT, C::D, true>(lr, tile, weights, {}, C::PITCH, sums, warp, lane, r - warp, rows);
  }
}
template <int NV, int MT, bool SHARED>
__global__ void __launch_bounds__(256, (SHARED ? RmsLr<NV, MT, 1>::BWD_CTAS : 1))
rmsnorm_bwd_lr_kernel(const float* x, const float* __restrict__ w, const float* dn, const float* dres, int rows,
                      float eps, float* out, __half* __restrict__ out16, float* __restrict__ scale, const LowRank lr) {
  using C = RmsLr<NV, MT, 1>;
  extern __shared__ __align__(16) uint8_t lr_smem[];
  uint8_t* tile = lr_smem;
  float* sums = (float*)(lr_smem + C::TILE);
  uint8_t* weights = lr_smem + C::TILE + C::SUMS;
  pdl_launch_dependents();
  lr_prefetch(lr.w, lr.r, C::D);
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  LrWeights<MT> first = {};
  if (SHARED) lr_fetch_weights(lr.w, lr.r, C::D, weights, C::PITCH);
  else if (warp * 32 < C::D) first.load(lr.w, lr.r, C::D, warp * 32, lane);
  const int step = (int)gridDim.x * 8;
  for (int r = (int)blockIdx.x * 8 + warp; r - warp < rows; r += step) {
    uint8_t* t = tile + warp * C::PITCH + 8 * lane;
    if (r < rows) {
      const size_t at = (size_t)r * C::D;
      float4 xv[NV], gv[NV], rv[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        xv[k] = ((const float4*)(x + at))[lane + 32 * k];
        gv[k] = ((const float4*)(dn + at))[lane + 32 * k];
        rv[k] = dres ? ((const float4*)(dres + at))[lane + 32 * k] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      float m = rms_bwd_row<NV>(xv, gv, rv, w, eps, lane);
#pragma unroll
      for (int k = 0; k < NV; ++k) ((float4*)(out + at))[lane + 32 * k] = gv[k];
      m = warp_max(m);
      const float sc = m > 0.f ? m : 1.f, inv = 1.f / sc;
#pragma unroll
      for (int k = 0; k < NV; ++k) {
        const uint2 o = half4(make_float4(gv[k].x * inv, gv[k].y * inv, gv[k].z * inv, gv[k].w * inv));
        *(uint2*)(out16 + at + 4 * (lane + 32 * k)) = o;
        *(uint2*)(t + 256 * k) = o;
      }
      if (lane == 0) scale[r] = m;
    }
    if (SHARED) cp_async_wait<0>();
    __syncthreads();
    lr_of_rows<MT, 1, C::D, SHARED>(lr, tile, weights, first, C::PITCH, sums, warp, lane, r - warp, rows);
    if (!SHARED) break;  // a CTA for every eight rows
  }
}

// Up to so many rows: forward eight rows of a CTA at a time, beyond sixteen, which read the weights half as often (as many CTAs as
// fit in either case, which loop where there are more groups: 1024 columns with 48 rank indices from 1185 rows on); backward a CTA
// for every eight rows with the weights from L2 (1024 rows of 1024, 16 rank indices, in a step 5.1 us; persistent 7.6, its row's registers
// no longer fit), beyond persistent ones (8192 rows 28 us, 33 the other way).
constexpr int RMS_LR_WIDE = 2048;
// The two with the product, for rows of 128..1024 floats and all that its 64 columns hold.  A 0.6B layer's forward and backward against
// products of their own: 32 rank indices (stacks of 64) 349 us at 1024 tokens (351 with the forward's apart, 359 with the backward's), 459
// (463, 466) at 2048, 644 (644, 651) at 4096, 1087 (1086, 1089) at 8192; 64 indices, which only the backward takes, 392 (403), 514 (520),
// 700 (705), 1136 (1135); at 16384 tokens and with 256 or 512 columns the same picture.
bool rmsnorm_takes_lowrank(int d, int r) { return d % 128 == 0 && d <= 1024 && r >= 1 && r <= 64; }
template <class Kernel, class... A>
static int launch_rms_lr(rt_ctx* c, Kernel* kernel, int rows, int nt, int ctas, int most_smem, int smem, A... a) {
  if (!c->raise_smem(kernel, most_smem)) return 3;
  const int groups = (rows + 8 * nt - 1) / (8 * nt);
  if (pdl(kernel, ctas ? std::min(groups, ctas * c->num_sms) : groups, 256 * nt, smem, c->stream)(a...) != cudaSuccess) return 3;
  RT_COUNT_LAUNCH(1);
  return 0;
}
template <int NV, int MT>
static int rmsnorm_fwd_lr(rt_ctx* c, const float* x, const float* w, int rows, float eps, __half* y16, const LowRank& lr) {
  using A = RmsLr<NV, MT, 1>;
  using B = RmsLr<NV, MT, 2>;
  if (rows <= RMS_LR_WIDE) return launch_rms_lr(c, rmsnorm_fwd_lr_kernel<NV, MT, 1>, rows, 1, A::FWD_CTAS, A::bytes(16 * MT), A::bytes(lr.r), x, w, rows, eps, y16, lr);
  return launch_rms_lr(c, rmsnorm_fwd_lr_kernel<NV, MT, 2>, rows, 2, B::FWD_CTAS, B::bytes(16 * MT), B::bytes(lr.r), x, w, rows, eps, y16, lr);
}
#define RT_LR_MT(F, NV, ...)                          \
  switch ((lr.r + 15) / 16) {                         \
    case 1: return F<NV, 1>(__VA_ARGS__);             \
    case 2: return F<NV, 2>(__VA_ARGS__);             \
    case 3: return F<NV, 3>(__VA_ARGS__);             \
    default: return F<NV, 4>(__VA_ARGS__);            \
  }
#define RT_LR_NV(F, ...)                              \
  switch (d / 128) {                                  \
    case 1: RT_LR_MT(F, 1, __VA_ARGS__)               \
    case 2: RT_LR_MT(F, 2, __VA_ARGS__)               \
    case 3: RT_LR_MT(F, 3, __VA_ARGS__)               \
    case 4: RT_LR_MT(F, 4, __VA_ARGS__)               \
    case 5: RT_LR_MT(F, 5, __VA_ARGS__)               \
    case 6: RT_LR_MT(F, 6, __VA_ARGS__)               \
    case 7: RT_LR_MT(F, 7, __VA_ARGS__)               \
    default: RT_LR_MT(F, 8, __VA_ARGS__)              \
  }
int launch_rmsnorm_fwd_lr(rt_ctx* c, const float* x, const float* w, int rows, int d, float eps, __half* y16, const LowRank& lr) {
  if (rows <= 0) return 0;
  if (!rmsnorm_takes_lowrank(d, lr.r)) return 3;
  RT_LR_NV(rmsnorm_fwd_lr, c, x, w, rows, eps, y16, lr)
}
template <int NV, int MT>
static int rmsnorm_bwd_lr(rt_ctx* c, const float* x, const float* w, const float* dn, const float* dres, int rows, float eps, float* out,
                          __half* out16, float* scale, const LowRank& lr) {
  using C = RmsLr<NV, MT, 1>;
  if (rows <= RMS_LR_WIDE) return launch_rms_lr(c, rmsnorm_bwd_lr_kernel<NV, MT, false>, rows, 1, 0, C::bytes(0), C::bytes(0), x, w, dn, dres, rows, eps, out, out16, scale, lr);
  return launch_rms_lr(c, rmsnorm_bwd_lr_kernel<NV, MT, true>, rows, 1, C::BWD_CTAS, C::bytes(16 * MT), C::bytes(lr.r), x, w, dn, dres, rows, eps, out, out16, scale, lr);
}
int launch_rmsnorm_bwd_lr(rt_ctx* c, const float* x, const float* w, const float* dn, const float* dres, int rows, int d, float eps,
                          float* out, __half* out16, float* scale, const LowRank& lr) {
  if (rows <= 0) return 0;
  if (!rmsnorm_takes_lowrank(d, lr.r)) return 3;
  RT_LR_NV(rmsnorm_bwd_lr, c, x, w, dn, dres, rows, eps, out, out16, scale, lr)
}

}  // namespace rt
