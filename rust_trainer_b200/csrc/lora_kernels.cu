// The LoRA gradients' second stage for batches whose token splits do not fit one cluster
// (lora_grads_tc.cu): partial sums in memory, added in split order.
#include "ops.h"
#include "pdl.cuh"
#include "rt_internal.h"

namespace rt {

namespace {

// One linear, or a group that shares X: partB is [splits][R x N_total] with the members'
// diagonal blocks wanted (member j: rows rank_off..+r of the rank axis, columns row_off..+rows),
// partA is [splits][R x K] with member j owning rows rank_off..+r.
__global__ void lora_grads_group_reduce_kernel(const float* __restrict__ partB, const float* __restrict__ partA, int splits,
                                               int NT, int K, int R, const LoraGroupTable t) {
  pdl_entry();
  size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nB = (size_t)R * NT, nA = (size_t)R * K;
  for (int j = 0; j < t.n; ++j) {
    const LoraGroupMember& mb = t.m[j];
    const size_t cb = (size_t)mb.r * mb.rows, ca = (size_t)mb.r * K;
    if (e < cb) {
      const int i = (int)(e / mb.rows), n = (int)(e % mb.rows);
      const size_t src = (size_t)(mb.rank_off + i) * NT + mb.row_off + n;
      float s = 0.f;
      for (int k = 0; k < splits; ++k) s += partB[(size_t)k * nB + src];
      mb.gb[(size_t)n * mb.r + i] += s;
      return;
    }
    e -= cb;
    if (e < ca) {
      const size_t src = (size_t)mb.rank_off * K + e;
      float s = 0.f;
      for (int k = 0; k < splits; ++k) s += partA[(size_t)k * nA + src];
      mb.ga[e] += s;
      return;
    }
    e -= ca;
  }
}

}  // namespace

void launch_lora_grads_group_reduce(const float* partB, const float* partA, int splits, int N, int K, int r, const LoraGroupTable& t,
                                    cudaStream_t st) {
  size_t total = 0;
  for (int j = 0; j < t.n; ++j) total += (size_t)t.m[j].r * ((size_t)t.m[j].rows + (size_t)K);
  pdl(lora_grads_group_reduce_kernel, (unsigned)((total + 255) / 256), 256, 0, st)(partB, partA, splits, N, K, r, t);
  RT_COUNT_LAUNCH(1);
}

}  // namespace rt
