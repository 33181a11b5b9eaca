// The low-rank side products of a LoRA linear, Hs = X.(sA)^T and Gs = dY.(sB) (reference
// src/linear.rs:84-91,105-117), on tcgen05: out[M x 64] (f16) = X[M x K] . Wt[r x K]^T, r <= 64.
//
// The product is a pure stream over X (2 K bytes per token against 2 r K flops): what matters is how
// many bytes are in flight.  The contraction is cut into up to eight pieces, each with a TMEM
// accumulator of its own; a cluster of CTAs shares a tile of TN tokens, each taking PPC of the pieces
// through its own ring of stages, and the CTAs' sums meet in shared memory, each CTA finishing its
// share of the tile.  (One CTA per 64 tokens walking the whole contraction, the form before, left most
// of the GPU idle below 8192 tokens: 6.2 us for 1024 columns and 2.5 more per further 1024 at 1024 tokens,
// 27 us for 6144 columns at 8192.)
//
// How the contraction is cut depends on K only (lr_piece_steps) and the pieces are added as the leaves
// of one fixed binary tree however many of them a CTA holds, so a token's result is the same in any
// batch.  The TOKENS are the MMA's N dimension (M = 128 rank lanes, N = TN tokens, K = 16).  Only r of
// the MMA's 128 A rows are loaded: the other rows of the operand are whatever follows in shared
// memory, and row i only reaches accumulator lane i.  Columns from r up to 63 of the result are exact
// zeros, which is what the big matmul's low-rank chunk expects to find there.
#include "ctx.h"
#include "pdl.cuh"
#include "ptx.cuh"
#include <cuda_fp16.h>
#include <stdint.h>

namespace rt {

namespace {

// contraction steps (64 columns) of one piece, and how many pieces a contraction of nk steps has: at most
// eight (the portable cluster size), none shorter than four steps unless the whole is
constexpr int LR_MAX_PIECES = 8;
inline int lr_piece_steps(int nk) {
  const int base = (nk + LR_MAX_PIECES - 1) / LR_MAX_PIECES;
  return base < 4 ? 4 : base;
}

template <int TN, int NS>
struct LrCfg {
  static constexpr uint32_t W_BYTES = 64 * 128, X_BYTES = TN * 128, STAGE = W_BYTES + X_BYTES;
  // the MMA's A descriptor spans 128 rows = 16 KB from a stage's start: the last stage needs that much behind it
  static constexpr uint32_t OFF_BAR = NS * STAGE + (STAGE < 16384 ? 16384 - STAGE : 0);
  static constexpr uint32_t TOTAL = OFF_BAR + 256 + 1024;
  // the CTA's sums, [TN tokens][64 + 4] f32 (a cluster) or [TN][64] f16 (a CTA alone), take the place of the
  // operand stages once those are used up
  static constexpr int PITCH = 68;
  static_assert(TOTAL >= LOWRANK_KERNEL_SMEM, "blocks of kernels with TMEM in front of it could share its SM (pdl.cuh)");
  static_assert(STAGE % 1024 == 0, "stages start on a swizzle atom");
  static_assert(TN * PITCH * 4 <= NS * STAGE, "the sums fit over the stages");
};
enum { SITE_LR_FREE = 491, SITE_LR_FULL, SITE_LR_DONE };

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ void add32(uint32_t* a, const uint32_t* b) {
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) + __uint_as_float(b[i]));
}

template <int TN, int NS, int PPC>
__global__ void __launch_bounds__(128)
lowrank_tc_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, int M, int nk, int piece,
                  int n_ctas, int r, __half* __restrict__ out, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  using Cfg = LrCfg<TN, NS>;
  uint8_t* sm = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* bars = (uint64_t*)(sm + Cfg::OFF_BAR);
  uint64_t* full = bars;         // [NS]
  uint64_t* empty = bars + NS;   // [NS]
  uint64_t* done = bars + 2 * NS;
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * NS + 2);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = n_ctas > 1 ? (int)cluster_ctarank() : 0;
  const int m0 = (int)(blockIdx.x / n_ctas) * TN;
  const int k0 = rank * PPC * piece, n_steps = min(nk - k0, PPC * piece);

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    mbar_fence_init();
    prefetch_tmap(&tm_x);
    prefetch_tmap(&tm_w);
  }
  if (warp == 3) {
    tmem_alloc(tmem_slot, TN * PPC);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  pdl_wait();
  // Only now: the matmul that follows (QGemmArgs::late_wait) takes everything older than this kernel as
  // complete once it runs, and waits for this kernel alone, before the last step of its contraction.
  pdl_launch_dependents();

  bool ok = true;
  if (warp == 2) {
    if (elect_one()) {
      const uint32_t bytes = Cfg::X_BYTES + (uint32_t)((r + 7) & ~7) * 128u;
      int s = 0;
      uint32_t ph = 0;
      for (int kc = 0; kc < n_steps; ++kc) {
        if (!mbar_wait(&empty[s], ph ^ 1, status, SITE_LR_FREE)) break;
        mbar_expect_tx(&full[s], bytes);
        tma_load_2d(sm + s * Cfg::STAGE + Cfg::W_BYTES, &tm_x, (k0 + kc) * 64, m0, &full[s]);
        tma_load_2d(sm + s * Cfg::STAGE, &tm_w, (k0 + kc) * 64, 0, &full[s]);
        if (++s == NS) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 3) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc(0, 0, 0, 0, 128, TN);
      const uint64_t a0 = umma_desc_sw128(smem_u32(sm), 16, 1024), b0 = umma_desc_sw128(smem_u32(sm) + Cfg::W_BYTES, 16, 1024);
      int s = 0, in_piece = 0;
      uint32_t ph = 0, d = tmem_base;
      for (int kc = 0; kc < n_steps; ++kc) {
        if (!mbar_wait(&full[s], ph, status, SITE_LR_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t off = (uint32_t)s * (Cfg::STAGE >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16_split<false>(d, (uint32_t)a0 + off + kk * 2, (uint32_t)(a0 >> 32), (uint32_t)b0 + off + kk * 2,
                                (uint32_t)(b0 >> 32), idesc, (uint32_t)((in_piece | kk) != 0));
        umma_commit(&empty[s]);
        if (++s == NS) { s = 0; ph ^= 1; }
        if (++in_piece == piece) { in_piece = 0; d += TN; }
      }
      if (ok) umma_commit(done);
    }
  } else if (mbar_wait(done, 0, status, SITE_LR_DONE)) {
    // thread = rank index = TMEM lane; a piece's TN columns are the tile's tokens
    tc_fence_after();
    const int held = (n_steps + piece - 1) / piece;
    const bool keep = warp * 32 + lane < r;  // lanes from r up hold products with whatever follows the factor tile
    float* part = (float*)sm + warp * 32 + lane;
    __half* alone = (__half*)sm + warp * 32 + lane;
#pragma unroll
    for (int c = 0; c < TN; c += 32) {
      const uint32_t a = tmem_base + ((uint32_t)(warp * 32) << 16) + c;
      uint32_t v[32], w[32];
      tmem_ld32(a, v);
      if (PPC > 1 && held > 1) {
        tmem_ld32(a + TN, w);
        tmem_ld_wait();
        add32(v, w);
      }
      if (PPC > 2 && held > 2) {
        tmem_ld32(a + 2 * TN, w);
        tmem_ld_wait();
        if (held > 3) {
          uint32_t u[32];
          tmem_ld32(a + 3 * TN, u);
          tmem_ld_wait();
          add32(w, u);
        }
        add32(v, w);
      }
      tmem_ld_wait();
#pragma unroll
      for (int t = 0; t < 32; ++t) {
        const float x = keep ? __uint_as_float(v[t]) : 0.f;
        if (n_ctas > 1) part[(c + t) * Cfg::PITCH] = x;
        else alone[(c + t) * 64] = __float2half_rn(x);
      }
    }
  }
  if (*(volatile int*)status != 0) {
    for (int k = 0; k < 1000; ++k) __nanosleep(1000);
    ok = false;
  }
  tc_fence_before();
  __syncwarp();
  if (n_ctas > 1) {
    cluster_sync_all();  // every CTA's sums are in its shared memory
    // this CTA's share of the tile's (token, four rank indices) items, added up along the tree
    const int items = TN * 16, per = (items + n_ctas - 1) / n_ctas, end = min(items, (rank + 1) * per);
    constexpr int LEAVES = LR_MAX_PIECES / PPC;
    if (ok)
      for (int e = rank * per + threadIdx.x; e < end; e += 128) {
        const int t = e >> 4, c = (e & 15) * 4;
        const uint32_t a = smem_u32(sm) + (uint32_t)(t * Cfg::PITCH + c) * 4u;
        float4 x[LEAVES];
#pragma unroll
        for (int i = 0; i < LEAVES; ++i) x[i] = i < n_ctas ? ld_cluster_f4(mapa_u32(a, (uint32_t)i)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 1; w < LEAVES; w *= 2)
#pragma unroll
          for (int i = 0; i < LEAVES; i += 2 * w) x[i] = x[i] + x[i + w];
        if (m0 + t < M) {
          __half2* o = (__half2*)(out + (size_t)(m0 + t) * 64 + c);
          o[0] = __floats2half2_rn(x[0].x, x[0].y);
          o[1] = __floats2half2_rn(x[0].z, x[0].w);
        }
      }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while its shared memory may still be read
  } else {
    __syncthreads();
    const int rows = min(M - m0, TN);  // [TN tokens][64] f16 is one contiguous block of the output
    const uint4* src = (const uint4*)sm;
    uint4* dst = (uint4*)(out + (size_t)m0 * 64);
    if (ok)
      for (int e = threadIdx.x; e < rows * 8; e += 128) dst[e] = src[e];
  }
  if (warp == 3) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TN * PPC);
  }
}

template <int TN, int NS, int PPC>
int lowrank_launch(rt_ctx* c, const __half* X, const __half* Wt, int M, int K, int r, __half* out64) {
  using Cfg = LrCfg<TN, NS>;
  if (!c->raise_smem(lowrank_tc_kernel<TN, NS, PPC>, Cfg::TOTAL)) return 3;
  CUtensorMap tx, tw;
  if (tensor_map_f16_2d(c, &tx, X, (uint64_t)M, (uint64_t)K, 64, TN)) return 3;
  if (tensor_map_f16_2d(c, &tw, Wt, (uint64_t)r, (uint64_t)K, 64, (uint32_t)((r + 7) & ~7))) return 3;
  const int nk = (K + 63) / 64, piece = lr_piece_steps(nk), n_ctas = (nk + piece * PPC - 1) / (piece * PPC);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)n_ctas;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)((M + TN - 1) / TN * n_ctas));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = Cfg::TOTAL;
  cfg.stream = c->stream;
  cfg.attrs = at;
  cfg.numAttrs = n_ctas > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, lowrank_tc_kernel<TN, NS, PPC>, tx, tw, M, nk, piece, n_ctas, r, out64, c->status_dev) != cudaSuccess) return 3;
  RT_COUNT_LAUNCH(1);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace

// 0: launched; 1: shape not supported (the caller has other routes); 3: launch failure
int launch_lowrank_tc(rt_ctx* c, const __half* X, const __half* Wt, int M, int K, int r, __half* out64) {
  if (M <= 0) return 0;
  if (r <= 0 || r > 64 || K % 8 != 0 || ((uintptr_t)X & 15) || ((uintptr_t)Wt & 15) || ((uintptr_t)out64 & 15)) return 1;
  // How many CTAs share a tile, from a sweep over 64..16384 tokens and 128..9728 columns (r = 48; us at 1024 |
  // 3072 | 6144 columns): eight while that leaves SMs idle (1024 tokens: 5.8 | 6.9 | 8.1), four up to twice
  // that (4096 tokens: 6.6 | 9.2 | 12.1), then two (8192 tokens: 6.8 | 12.5 | 20.0), long contractions with
  // tokens twice as wide, which halves the factor's share of the traffic (8192: 8.7 | 12.2 | 18.5).
  if (M <= 2048) return lowrank_launch<64, 6, 1>(c, X, Wt, M, K, r, out64);
  if (M <= 4096) return lowrank_launch<64, 6, 2>(c, X, Wt, M, K, r, out64);
  if (K < 3072) return lowrank_launch<64, 6, 4>(c, X, Wt, M, K, r, out64);
  return lowrank_launch<128, 4, 2>(c, X, Wt, M, K, r, out64);
}

}  // namespace rt
