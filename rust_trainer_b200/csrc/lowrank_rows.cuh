// The low-rank products Hs = X.(sA)^T and Gs = dY.(sB) of a LoRA linear (reference src/linear.rs:84-91,105-117) inside the kernel
// that makes X (or over rows in memory): out[M x 64] (f16) = X[M x K] . Wt[r x K]^T, r <= 64, K a multiple of 32.
//
// A CTA has LR_TOKENS tokens and all of K; its warps take the 32-wide blocks of K in turn (block b is warp b % warps'), each
// adding its own into registers, and the warps' sums are added in warp order.  So what a token gets depends on K and
// the number of warps alone, in any batch.
// The tokens are the N = 8 of mma.m16n8k16, the rank indices its M: a warp's whole state is four registers for each 16 rank
// indices, no shared memory, TMEM or barrier has to be set up, and the product costs the kernel it stands in the time of its
// weights' way from L2.  (A tcgen05 product wants 128 rank rows and its operands in shared memory: as a launch of its own
// the stream of lowrank_tc.cu is 5 to 6 us of a chain of dependent launches, on SMs that the matmul behind it waits for.)
// 28-layer 0.6B shape: step of 1024 tokens 7.87 -> 7.30 ms, scoring 157 tokens 1.98 -> 1.86 ms, of a step of 8192 tokens no change.
#pragma once
#include "ptx.cuh"
#include <cuda_fp16.h>
#include <stdint.h>

namespace rt {

// Where a row kernel leaves the low-rank product of the rows it writes; w null: nowhere.
struct LowRank {
  const __half* w = nullptr;  // [r x K], 16-byte aligned
  int r = 0;
  __half* out = nullptr;  // [M x 64], zero from column r up
};

constexpr int LR_TOKENS = 8;
constexpr int LR_SLICES = 8;  // warps that share K where rows and weights are in shared memory

// A lane's part of the product's operands in block b of K.  Lane 4 g + q holds eight consecutive elements, k = 32 b + 8 q.., of
// row g: token g for X, rank indices g and g + 8 of a group of 16 for the weights.  The MMA's own order of k within a block
// is another one, but the same one for both operands.
__device__ __forceinline__ void lr_mma(float* d, const uint4& lo, const uint4& hi, const uint4& x) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(lo.x), "r"(hi.x), "r"(lo.y), "r"(hi.y), "r"(x.x), "r"(x.y));
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(lo.z), "r"(hi.z), "r"(lo.w), "r"(hi.w), "r"(x.z), "r"(x.w));
}

template <int MT>  // groups of 16 rank indices
struct LrWeights {
  uint4 lo[MT], hi[MT];
  __device__ __forceinline__ void load(const __half* w, int r, int K, int k, int lane) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const __half* p = w + (size_t)(16 * m + g) * K + k + 8 * q;
      lo[m] = 16 * m + g < r ? *(const uint4*)p : make_uint4(0, 0, 0, 0);
      hi[m] = 16 * m + g + 8 < r ? *(const uint4*)(p + (size_t)8 * K) : make_uint4(0, 0, 0, 0);
    }
  }
};
template <int MT>
struct LrAcc {
  float d[MT][4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int m = 0; m < MT; ++m) d[m][0] = d[m][1] = d[m][2] = d[m][3] = 0.f;
  }
  __device__ __forceinline__ void add(const LrWeights<MT>& w, const uint4& x) {
#pragma unroll
    for (int m = 0; m < MT; ++m) lr_mma(d[m], w.lo[m], w.hi[m], x);
  }
};

// floats of shared memory for the warps' sums
__host__ __device__ constexpr int lr_pitch(int mt) { return 16 * mt + 4; }  // keeps a warp's stores in different banks
__host__ __device__ constexpr int lr_sum_floats(int warps, int mt) { return warps * LR_TOKENS * lr_pitch(mt); }

// A warp's sum of a group, where lr_sum finds it.
template <int MT, int WARPS>
__device__ __forceinline__ void lr_put(const LrAcc<MT>& acc, float* sums, int group, int slice, int lane) {
  constexpr int P = lr_pitch(MT);
  float* s = sums + (group * WARPS + slice) * (LR_TOKENS * P) + 2 * (lane & 3) * P + (lane >> 2);
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    s[16 * m] = acc.d[m][0];
    s[16 * m + P] = acc.d[m][1];
    s[16 * m + 8] = acc.d[m][2];
    s[16 * m + 8 + P] = acc.d[m][3];
  }
}
// Adds the warps' sums up and writes tokens m0.. (those below M) of NT groups; thread: of the CTA.
template <int MT, int NT, int WARPS>
__device__ __forceinline__ void lr_sum(const float* sums, int thread, int m0, int M, __half* __restrict__ out) {
  constexpr int P = lr_pitch(MT);
  const int t = thread >> 4, c = (thread & 15) * 4;
  if (t < NT * LR_TOKENS && m0 + t < M) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < 16 * MT) {
      const float* s = sums + (t / LR_TOKENS * WARPS * LR_TOKENS + t % LR_TOKENS) * P + c;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float4 p = *(const float4*)(s + w * (LR_TOKENS * P));
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
      }
    }
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    *(uint2*)(out + (size_t)(m0 + t) * 64 + c) = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
  }
}
// Both, called by the whole CTA, WARPS warps for each group; nobody reads `sums` any more.
template <int MT, int NT, int WARPS>
__device__ __forceinline__ void lr_finish(const LrAcc<MT>& acc, float* sums, int group, int slice, int lane, int m0, int M, __half* __restrict__ out) {
  lr_put<MT, WARPS>(acc, sums, group, slice, lane);
  __syncthreads();
  lr_sum<MT, NT, WARPS>(sums, (group * WARPS + slice) * 32 + lane, m0, M, out);
}

// The CTAs' shares of the weights on their way to L2 while the kernel in front still runs (nothing is read).
__device__ __forceinline__ void lr_prefetch(const __half* w, int r, int K) {
  const size_t bytes = (size_t)r * K * 2, step = (size_t)gridDim.x * blockDim.x * 128;
  for (size_t at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 128; at < bytes; at += step)
    asm volatile("prefetch.global.L2 [%0];" ::"l"((const uint8_t*)w + at));
}

// Rows that lie in shared memory: `lr_row_pitch` bytes apart, which puts the two rows that a quarter warp reads into different banks.
__host__ __device__ constexpr int lr_row_pitch(int k) { return 2 * k + 64; }
__device__ __forceinline__ void lr_fetch_weights(const __half* w, int r, int K, uint8_t* dst, int pitch) {
  const int per_row = K / 8;
  for (int i = (int)threadIdx.x; i < r * per_row; i += (int)blockDim.x) {
    const int row = i / per_row, c = i - row * per_row;
    cp_async_16(smem_u32(dst + row * pitch + c * 16), w + (size_t)row * K + c * 8);
  }
  cp_async_commit();
}
// The product of NT groups of LR_TOKENS rows that lie in shared memory, by LR_SLICES warps for each group.  The weights lie there
// too (`weights`), or come from L2, those of the warp's first block, `first`, before the rows are ready.
template <int MT, int NT, int K, bool SHARED>
__device__ __forceinline__ void lr_of_rows(const LowRank& lr, const uint8_t* rows, const uint8_t* weights, const LrWeights<MT>& first,
                                           int pitch, float* sums, int warp, int lane, int m0, int M) {
  const int group = NT == 1 ? 0 : warp / LR_SLICES, slice = NT == 1 ? warp : warp % LR_SLICES, g = lane >> 2, q = lane & 3;
  LrAcc<MT> acc;
  acc.clear();
  const uint8_t* x = rows + (group * LR_TOKENS + g) * pitch + q * 16;
  const uint8_t* a = weights + g * pitch + q * 16;
#pragma unroll
  for (int b = 0; b < (K / 32 + LR_SLICES - 1) / LR_SLICES; ++b) {
    const int k = (b * LR_SLICES + slice) * 32;
    if (K / 32 % LR_SLICES != 0 && k >= K) break;
    LrWeights<MT> w;
    if (SHARED) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        w.lo[m] = 16 * m + g < lr.r ? *(const uint4*)(a + 16 * m * pitch + 2 * k) : make_uint4(0, 0, 0, 0);
        w.hi[m] = 16 * m + g + 8 < lr.r ? *(const uint4*)(a + (16 * m + 8) * pitch + 2 * k) : make_uint4(0, 0, 0, 0);
      }
    } else if (b > 0) {
      w.load(lr.w, lr.r, K, k, lane);
    } else {
      w = first;
    }
    acc.add(w, *(const uint4*)(x + 2 * k));
  }
  lr_finish<MT, NT, LR_SLICES>(acc, sums, group, slice, lane, m0, M, lr.out);
}

}  // namespace rt
