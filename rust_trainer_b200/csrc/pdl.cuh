// Programmatic dependent launch: a kernel launched through pdl(...) may be scheduled while the
// kernel before it on the stream is still running; it must not touch global memory before
// pdl_wait(), which returns once that kernel has completed and its writes are visible.  What runs
// before the wait (barrier init, TMEM allocation, tensor-map prefetch, block scheduling itself)
// overlaps the predecessor's tail.  Rules of the kernels launched this way:
//   - every CTA executes pdl_wait() before its first access to anything the pass computes and before any
//     early return (a grid that is complete has then waited, so ordering stays transitive).  What a batch
//     brings along and no kernel writes (tile lists, where sequences start) may be read before it;
//   - what the pass computes is read through plain pointers.  __restrict__ promises the compiler that nobody else writes there while the
//     kernel runs, which the kernel in front of it still does: a conditional load may then move in front of the wait (a kernel that
//     was not kept read its input too early), or go through a cache that neither the wait nor pdl_unwaited's fence refreshes;
//   - pdl_launch_dependents() is called at entry: the next kernel may be scheduled as soon as
//     every CTA of this one has started.  A CTA that has not got its TMEM yet must then find it: a CTA of a later kernel that took the
//     columns on the same SM waits for this kernel, which would wait for them.  So a kernel with TMEM lets the next one start once it
//     holds its columns; or no block of a kernel that could take them fits beside its blocks: none at all beside a
//     matmul's, no low-rank one beside two of the attention's forward or dQ (256 columns each; behind them the low-rank
//     kernel is the first with TMEM, and it lets nothing start before they are complete).  The constants below say so.  (Later, once
//     it holds its columns, in the matmul too: scoring 157 tokens 2.00 -> 2.02 ms.)
// Three pairs of kernels depart from both.  (1) A matmul behind a low-rank stream (QGemmArgs::late_wait) reads
// weights, activations and residual without waiting and waits only where it loads the stream's result.  That
// is sound because of what lowrank_tc_kernel and the matmul keep between them:
//   - lowrank_tc_kernel (and the lowrank_rows kernels in its place) triggers only after its own wait, so that everything older than it is complete and
//     visible once the matmul runs.  Moved to the kernel's entry, the trigger would make a race of this;
//   - it writes nothing the matmul reads but that result, and the matmul writes nothing it reads;
//   - at least one CTA of the matmul waits (the last piece of a contraction always ends in the low-rank
//     step), so that whoever waits for the matmul has waited for the stream.
// (2) The attention's dQ kernel behind its dK/dV kernel, which it needs nothing from (attention_tc.cu): dK/dV triggers only
// after its own wait, so that what both read is complete and visible; neither writes what the other reads or writes;
// and every CTA of dQ waits before it ends, so that whoever waits for dQ has waited for both.
// (3) A matmul behind the adapter gradients of its block (QGemmArgs::end_wait), under the same conditions: the gradients read
// what the matmul reads and write what nothing in the block reads; they trigger after their wait; every CTA of the matmul
// waits before it ends.
// Complete means that the writes are in L2.  A line that the SM's L1 holds from before them is only sure to be gone after the wait,
// so a CTA of the three that reads by ordinary loads what the pass computes executes pdl_unwaited() first, in one warp in front of
// the barrier at the end of its set-up.  (TMA and cp.async.cg read L2.)
// Inside stream capture these launches become programmatic edges of the graph.
// Used for passes of up to PDL_MAX_TOKENS tokens, whose kernels leave SMs free for the next one's CTAs to
// start on: the 28-layer 0.6B step 10.67 -> 10.14 ms at 1024 tokens, scoring 157 tokens 3.01 -> 2.84 ms.  At
// 8192 tokens the kernels fill every SM and a waiting successor only takes room from them: 46.2 -> 46.9
// ms, and the 3B step 153.7 -> 155.5.  RT_B200_PDL=0 or 1 in the environment decides for every size.
// (The kernels carry the wait either way; without the launch attribute it returns at once.)
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <utility>

namespace rt {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// In place of the wait, where a kernel reads what was complete before it could start: an acquire fence, so that its loads do not
// take from L1 what an earlier kernel left there.  (Loads past L1 instead, in the epilogues: scoring 157 tokens 1.98 -> 2.04 ms.)
__device__ __forceinline__ void pdl_unwaited() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
// the usual entry sequence of a kernel that has no prologue worth overlapping
__device__ __forceinline__ void pdl_entry() {
  pdl_launch_dependents();
  pdl_wait();
}

// Shared memory of an SM, 1 KB of each block's being the system's; the least a block of the low-rank kernel takes, and of any kernel
// with TMEM but the matmul; what a block takes so that two of it and one of the first do not fit, and so that it and one of the
// second do not.
constexpr int SMEM_PER_SM = 228 * 1024, LOWRANK_KERNEL_SMEM = 97 * 1024, TMEM_KERNEL_SMEM = 64 * 1024;
constexpr int TWO_BLOCKS_SMEM = 65 * 1024, ALONE_SMEM = 163 * 1024;
static_assert(2 * (TWO_BLOCKS_SMEM + 1024) + LOWRANK_KERNEL_SMEM + 1024 > SMEM_PER_SM && TWO_BLOCKS_SMEM >= TMEM_KERNEL_SMEM &&
              ALONE_SMEM + TMEM_KERNEL_SMEM + 2 * 1024 > SMEM_PER_SM);

constexpr int PDL_MAX_TOKENS = 4096;
inline thread_local int g_pdl_tokens = 0;  // tokens of the pass this thread is launching, see PdlScope
struct PdlScope {
  int before;
  explicit PdlScope(size_t tokens) : before(g_pdl_tokens) { g_pdl_tokens = tokens > (1u << 30) ? 1 << 30 : (int)tokens; }
  ~PdlScope() { g_pdl_tokens = before; }
};
inline int pdl_forced() {  // 1 always, 0 never, -1 by the pass's size
  static const int forced = [] {
    const char* e = getenv("RT_B200_PDL");
    return e ? (atoi(e) ? 1 : 0) : -1;
  }();
  return forced;
}
inline bool pdl_enabled() {
  return pdl_forced() >= 0 ? pdl_forced() != 0 : g_pdl_tokens > 0 && g_pdl_tokens <= PDL_MAX_TOKENS;
}
inline bool pdl_any_size() { return pdl_forced() != 0; }  // for a kernel that runs beside the one in front of it

template <typename... KArgs>
struct PdlLaunch {
  void (*kernel)(KArgs...);
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
  bool programmatic = pdl_enabled();
  template <typename... A>
  cudaError_t operator()(A&&... a) const {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = programmatic ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(std::forward<A>(a))...);
  }
};

// kernel<<<grid, block, smem, st>>>(args...)  becomes  pdl(kernel, grid, block, smem, st)(args...)
template <typename... KArgs>
inline PdlLaunch<KArgs...> pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
  return PdlLaunch<KArgs...>{kernel, grid, block, smem, st};
}

}  // namespace rt
