// LoRA gradients of one linear (or of a stacked group) as token contractions on tcgen05
// (reference src/linear.rs:105-117):
//
//   dB[n, i] = sum_m dY[m, n] * Hs[m, i]      dA[i, k] = sum_m Gs[m, i] * X[m, k]
//
// Both are sums over tokens of Small[m, i] * Big[m, c] with Big = dY or X ([M x C], read ONCE: the
// kernel is a stream over Big) and Small = Hs or Gs ([M x 64]).  One CTA takes 128 columns of Big and a
// range of tokens; the tokens are the MMA's K dimension, so both operands are read MN-major straight from
// their row-major tiles:
//   A = Big tile   [64 tokens][128 columns]  (two swizzled panels of 64 columns, TMA)
//   B = Small tile [64 tokens][64]           (TMA)
//   D[column (lane), i] in 64 TMEM columns, two of them in turn.
// Warps: 0-3 the epilogue, 4 the TMA producer, 5 issues the MMAs.
// The range is a row of splits of at most 1024 tokens (the tensor core's accumulator error grows with a
// chain's length); a split's sums are drained into registers under the next split's products.
// dY arrives row-normalised with one factor per token.  The factors go onto the Small rows
// relative to the split's largest factor (rounded up to a power of two, so what a row rounds to
// does not depend on its split mates), and the largest factor multiplies the split's sums.  A launch of its
// own does that for all the jobs (scaling each tile in place between its landing and its MMAs, in each
// of the 40-odd column tiles, was the pipeline's longest link: 100 us for the four jobs of a block at 8192
// tokens, 320 MB to read).
// A column tile is one cluster of up to eight CTAs: each leaves its sums in shared memory, and the CTAs add
// them in token order straight into the gradient buffers, each its share of the tile.  Deterministic, no
// atomics.  As many CTAs per cluster as fit the GPU at once, so that the launch is one wave: with a CTA for
// every 1024 tokens the clusters of eight (which leave 28 SMs without one) took 3.4 waves, 84 us
// for the four jobs of a block at 8192 tokens and 19456 columns in all, at 49 % of the DRAM rate; now 71 (floor 48),
// 45056 columns 200 -> 154 (floor 112).
#include "ctx.h"
#include "ops.h"
#include "pdl.cuh"
#include "ptx.cuh"
#include "rt_internal.h"
#include <cuda_fp16.h>
#include <stdint.h>
#include <algorithm>

namespace rt {

namespace {

constexpr int LG_NS = 3, LG_THREADS = 192, LG_CTAS_PER_SM = 3;
constexpr uint32_t LG_Q_BYTES = 2 * 64 * 128, LG_P_BYTES = 64 * 128, LG_STAGE = LG_Q_BYTES + LG_P_BYTES;
constexpr uint32_t LG_OFF_BAR = LG_NS * LG_STAGE;
constexpr uint32_t LG_TOTAL = LG_OFF_BAR + 256 + 1024;
static_assert(LG_TOTAL >= TMEM_KERNEL_SMEM, "a matmul's block could share its SM (pdl.cuh)");
enum { SITE_LG_FREE = 495, SITE_LG_FULL, SITE_LG_DONE, SITE_LG_DRAINED };

struct LgMaps {
  CUtensorMap pb, qb, pa, qa;
};
struct LgJob {
  const float* top;  // [splits] largest factor, or null: the rows carry none
  int N, K, r;
  int first, nbB;    // the job's first column tile in the grid, and how many of its tiles are dB's
  LoraGroupTable t;  // of one linear (offsets 0) or of a stacked group
};
struct LgArgs {
  LgMaps maps[LORA_GRAD_JOBS];
  LgJob job[LORA_GRAD_JOBS];
  int n_jobs, M, tps, per_cta;  // tokens per split, splits per CTA
};
// sums of a CTA, [rank index][128 columns + 1] f32, over the operand stages once those are used up
constexpr int LG_PITCH = 129;
static_assert(64 * LG_PITCH * 4 <= (int)(LG_NS * LG_STAGE), "the sums fit over the stages");

__global__ void __launch_bounds__(LG_THREADS, LG_CTAS_PER_SM)
lora_grads_tc_kernel(const __grid_constant__ LgArgs ga, int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* bars = (uint64_t*)(sm + LG_OFF_BAR);
  uint64_t* full = bars;           // [NS] TMA landed
  uint64_t* empty = bars + LG_NS;  // [NS] MMAs retired
  uint64_t* done = bars + 2 * LG_NS;         // [2] a split's products have completed
  uint64_t* drained = bars + 2 * LG_NS + 2;  // [2] ... and been read
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * LG_NS + 4);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  int jx = 0;
  while (jx + 1 < ga.n_jobs && (int)blockIdx.x >= ga.job[jx + 1].first) ++jx;
  const LgJob& g = ga.job[jx];
  const LgMaps& maps = ga.maps[jx];
  const int bx = (int)blockIdx.x - g.first;
  const bool isB = bx < g.nbB;
  const CUtensorMap* tm_p = isB ? &maps.pb : &maps.pa;
  const CUtensorMap* tm_q = isB ? &maps.qb : &maps.qa;
  const int C = isB ? g.N : g.K;
  const int j0 = (isB ? bx : bx - g.nbB) * 128;
  const int m_begin = blockIdx.y * ga.per_cta * ga.tps, m_end = min(ga.M, m_begin + ga.per_cta * ga.tps);
  const int nchunks = (m_end - m_begin + 63) / 64, split_chunks = ga.tps / 64, n_splits = (nchunks + split_chunks - 1) / split_chunks;

  if (threadIdx.x == 0) {
    for (int i = 0; i < LG_NS; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&done[i], 1);
      mbar_init(&drained[i], 4);
    }
    mbar_fence_init();
    prefetch_tmap(tm_p);
    prefetch_tmap(tm_q);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  pdl_wait();
  pdl_launch_dependents();  // only now: a matmul behind this kernel takes everything older as complete (QGemmArgs::end_wait)

  if (warp == 4) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      for (int ch = 0; ch < nchunks; ++ch) {
        if (!mbar_wait(&empty[s], ph ^ 1, status, SITE_LG_FREE)) break;
        const int mrow = m_begin + ch * 64;
        uint8_t* dst = sm + s * LG_STAGE;
        mbar_expect_tx(&full[s], LG_STAGE);
        tma_load_2d(dst, tm_q, j0, mrow, &full[s]);
        tma_load_2d(dst + 8192, tm_q, j0 + 64, mrow, &full[s]);
        tma_load_2d(dst + LG_Q_BYTES, tm_p, 0, mrow, &full[s]);
        if (++s == LG_NS) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc(0, 0, 1, 1, 128, 64);
      const uint64_t a0 = umma_desc_sw128(smem_u32(sm), 8192, 1024), b0 = umma_desc_sw128(smem_u32(sm) + LG_Q_BYTES, 8192, 1024);
      int s = 0;
      uint32_t ph = 0;
      int in_split = 0, sp = 0;
      for (int ch = 0; ch < nchunks; ++ch) {
        if (in_split == 0 && sp >= 2 && !mbar_wait(&drained[sp & 1], ((uint32_t)(sp >> 1) & 1) ^ 1, status, SITE_LG_DRAINED)) break;
        if (!mbar_wait(&full[s], ph, status, SITE_LG_FULL)) break;
        tc_fence_after();
        const uint32_t off = (uint32_t)s * (LG_STAGE >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_f16_split<false>(tmem_base + (sp & 1) * 64, (uint32_t)a0 + off + kk * (2048 >> 4), (uint32_t)(a0 >> 32), (uint32_t)b0 + off + kk * (2048 >> 4),
                                (uint32_t)(b0 >> 32), idesc, (uint32_t)((in_split | kk) != 0));
        umma_commit(&empty[s]);
        if (++s == LG_NS) { s = 0; ph ^= 1; }
        if (++in_split == split_chunks || ch + 1 == nchunks) {
          umma_commit(&done[sp & 1]);
          in_split = 0;
          ++sp;
        }
      }
    }
  } else {
    // ---- 128 threads: a column each, its sums over the CTA's splits in registers
    const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    bool ok = true;
    for (int sp = 0; sp < n_splits && ok; ++sp) {
      const float mul = g.top ? g.top[blockIdx.y * ga.per_cta + sp] : 1.0f;  // what the split's sums are multiplied by
      ok = mbar_wait(&done[sp & 1], (uint32_t)(sp >> 1) & 1, status, SITE_LG_DONE);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q * 16 >= g.r) break;
        uint32_t v[16];
        tmem_ld16(lane_addr + (sp & 1) * 64 + q * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[q * 16 + i] += __uint_as_float(v[i]) * mul;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&drained[sp & 1]);
    }
    if (ok) {  // every product has completed: the stages are free
      float* mine = (float*)sm + warp * 32 + lane;
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (i < g.r) mine[i * LG_PITCH] = acc[i];
    }
  }
  if (*(volatile int*)status != 0) {
    for (int k = 0; k < 1000; ++k) __nanosleep(1000);
  }
  tc_fence_before();
  __syncwarp();
  if (gridDim.y > 1) cluster_sync_all();  // every CTA's sums are in its shared memory
  else __syncthreads();
  if (*(volatile int*)status == 0) {
    const int n_cta = (int)gridDim.y, ncol = min(128, C - j0);
    // A thread's gradients go six at a time: reading the buffer, reading the CTAs' parts and writing back is a chain of
    // about 1000 cycles, which one at a time made 18 in a row of the q|k|v adapters' dA (the launch at 1024 tokens 20.9 -> 14.6 us).
    constexpr int U = 6;
    for (int q = 0; q < g.t.n; ++q) {
      const LoraGroupMember& mb = g.t.m[q];
      // a member owns whole column tiles of dB (its rows start on a multiple of 128) and r rows of dA
      if (isB && (j0 < mb.row_off || j0 >= mb.row_off + mb.rows)) continue;
      const int items = ncol * mb.r, per = (items + n_cta - 1) / n_cta, end = min(items, ((int)blockIdx.y + 1) * per);
      for (int e0 = (int)blockIdx.y * per + threadIdx.x; e0 < end; e0 += U * LG_THREADS) {
        float *dst[U], old[U], sum[U];
        uint32_t part[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int e = min(e0 + u * LG_THREADS, end - 1);  // (past the end: read again, not written)
          const int outer = e / (isB ? mb.r : ncol), inner = e - outer * (isB ? mb.r : ncol);
          const int i = mb.rank_off + (isB ? inner : outer), col = isB ? outer : inner;
          dst[u] = isB ? mb.gb + (size_t)(j0 - mb.row_off) * mb.r + e : mb.ga + (size_t)outer * g.K + j0 + inner;
          old[u] = *dst[u];
          part[u] = smem_u32(sm) + (uint32_t)(i * LG_PITCH + col) * 4u;
        }
#pragma unroll 1
        for (int k = 0; k < n_cta; ++k)
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float x = n_cta > 1 ? ld_cluster_f32(mapa_u32(part[u], (uint32_t)k)) : ld_shared_f32(part[u]);
            sum[u] = k == 0 ? x : sum[u] + x;
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (e0 + u * LG_THREADS < end) *dst[u] = old[u] + sum[u];  // nobody else adds to it
      }
    }
  }
  __syncwarp();
  if (gridDim.y > 1) cluster_sync_all();  // nobody leaves while its shared memory may still be read
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 128);
  }
}

// What the main kernel reads instead of Hs and Gs: row m times factor_m / (its split's largest factor).
struct LgScaleJob {
  const __half *hs, *gs;
  const float* pscale;
  __half *hs_out, *gs_out;
  float* top;  // [splits]
};
struct LgScaleArgs {
  LgScaleJob job[LORA_GRAD_JOBS];
  int M, tps;
};
// one block per (64 tokens, job); a split is a multiple of 64 tokens
__global__ void __launch_bounds__(256) lora_scale_small_kernel(const LgScaleArgs a) {
  pdl_entry();
  __shared__ float s_red[8];
  const LgScaleJob& g = a.job[blockIdx.y];
  const int m0 = blockIdx.x * 64, split = m0 / a.tps, m_begin = split * a.tps, m_end = min(a.M, m_begin + a.tps);
  const int rows = min(64, a.M - m0), tid = threadIdx.x;
  uint4 v[2][2];  // this thread's 16-byte units tid and tid + 256 of the 64 x 64 tile, of Hs and of Gs
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int e = tid + k * 256;
    if ((e >> 3) < rows) {
      v[0][k] = ((const uint4*)(g.hs + (size_t)m0 * 64))[e];
      v[1][k] = ((const uint4*)(g.gs + (size_t)m0 * 64))[e];
    }
  }
  // largest factor of the split (factors are >= 0), rounded up to a power of two so that dividing by it
  // changes no mantissa
  float mx = 0.f;
  for (int m = m_begin + tid; m < m_end; m += 256) mx = fmaxf(mx, g.pscale[m]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((tid & 31) == 0) s_red[tid >> 5] = mx;
  __syncthreads();
  mx = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) mx = fmaxf(mx, s_red[k]);
  mx = __int_as_float((__float_as_int(mx) + 0x007FFFFF) & 0x7F800000);
  const float inv = mx > 0.f ? 1.0f / mx : 0.f;
  if (m0 == m_begin && tid == 0) g.top[split] = mx;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int e = tid + k * 256;
    if ((e >> 3) >= rows) continue;
    const float f = g.pscale[m0 + (e >> 3)] * inv;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      __half2* h2 = (__half2*)&v[q][k];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 x = __half22float2(h2[i]);
        h2[i] = __floats2half2_rn(x.x * f, x.y * f);
      }
      ((uint4*)((q == 0 ? g.hs_out : g.gs_out) + (size_t)m0 * 64))[e] = v[q][k];
    }
  }
}

}  // namespace

struct LgPlan {
  int tps, splits, per_cta, n_ctas;  // tokens per split, splits, splits per CTA, CTAs per column tile
};
static LgPlan lora_grads_plan(const LoraGradJob* jobs, int n, int M, int num_sms) {
  int tiles = 0;
  for (int j = 0; j < n; ++j) tiles += (jobs[j].N + 127) / 128 + (jobs[j].K + 127) / 128;
  LgPlan p;
  // a power of two up to the portable cluster size, while all of the launch's CTAs fit the GPU at once and have 64 tokens
  p.n_ctas = 1;
  while (p.n_ctas < 8 && tiles * p.n_ctas * 2 <= LG_CTAS_PER_SM * num_sms && p.n_ctas * 64 < M) p.n_ctas *= 2;
  const int per = (M + p.n_ctas - 1) / p.n_ctas;  // tokens of a CTA
  p.per_cta = (per + 1023) / 1024;
  p.tps = ((per + p.per_cta - 1) / p.per_cta + 63) / 64 * 64;
  p.splits = (M + p.tps - 1) / p.tps;
  p.n_ctas = (p.splits + p.per_cta - 1) / p.per_cta;
  return p;
}
bool lora_grads_tc_takes(const LoraGradJob& j) {
  return j.r > 0 && j.r <= 64 && j.N % 8 == 0 && j.K % 8 == 0 && j.ld_dy % 8 == 0 && j.t.n >= 1 && j.t.n <= 3 &&
         (((uintptr_t)j.hs | (uintptr_t)j.dy | (uintptr_t)j.gs | (uintptr_t)j.x) & 15) == 0;
}
// per job: the scaled Hs and Gs, and the splits' largest factors
size_t lora_grads_tc_workspace_floats(rt_ctx* c, const LoraGradJob* jobs, int n, int M) {
  const LgPlan p = lora_grads_plan(jobs, n, M, c->num_sms);
  return (size_t)n * ((size_t)M * 64 + ((size_t)p.splits + 63) / 64 * 64);
}

// One launch for all the jobs (a block's linears): a launch per linear left half of the GPU idle at 1024
// tokens (152 CTAs of 296 places, 10.6 us each) and ended in a nearly empty wave at 8192.
int launch_lora_grads_tc(rt_ctx* c, const LoraGradJob* jobs, int n, int M, float* ws) {
  if (M <= 0 || n <= 0) return 0;
  if (n > LORA_GRAD_JOBS) return 3;
  if (!c->raise_smem(lora_grads_tc_kernel, LG_TOTAL)) return 3;
  LgArgs g;
  g.n_jobs = n;
  g.M = M;
  const LgPlan plan = lora_grads_plan(jobs, n, M, c->num_sms);
  const int splits = plan.splits;
  g.tps = plan.tps;
  g.per_cta = plan.per_cta;
  LgScaleArgs sa;
  sa.M = M;
  sa.tps = g.tps;
  int tiles = 0, n_scaled = 0;
  for (int j = 0; j < n; ++j) {
    const LoraGradJob& q = jobs[j];
    const __half *hs = q.hs, *gs = q.gs;
    LgJob& t = g.job[j];
    t.top = nullptr;
    if (q.dscale) {
      LgScaleJob& w = sa.job[n_scaled++];
      w = LgScaleJob{q.hs, q.gs, q.dscale, (__half*)ws, (__half*)ws + (size_t)M * 64, ws + (size_t)M * 64};
      hs = w.hs_out;
      gs = w.gs_out;
      t.top = w.top;
    }
    ws += (size_t)M * 64 + ((size_t)splits + 63) / 64 * 64;
    LgMaps& m = g.maps[j];
    if (tensor_map_f16_2d_ld(c, &m.pb, hs, (uint64_t)M, 64, 64, 64, 64)) return 3;
    if (tensor_map_f16_2d_ld(c, &m.qb, q.dy, (uint64_t)M, (uint64_t)q.N, (uint64_t)q.ld_dy, 64, 64)) return 3;
    if (tensor_map_f16_2d_ld(c, &m.pa, gs, (uint64_t)M, 64, 64, 64, 64)) return 3;
    if (tensor_map_f16_2d_ld(c, &m.qa, q.x, (uint64_t)M, (uint64_t)q.K, (uint64_t)q.K, 64, 64)) return 3;
    t.N = q.N;
    t.K = q.K;
    t.r = q.r;
    t.first = tiles;
    t.nbB = (q.N + 127) / 128;
    t.t = q.t;
    tiles += t.nbB + (q.K + 127) / 128;
  }
  if (n_scaled > 0) {
    pdl(lora_scale_small_kernel, dim3((M + 63) / 64, n_scaled), 256, 0, c->stream)(sa);
    RT_COUNT_LAUNCH(1);
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1;
  at[1].val.clusterDim.y = (unsigned)plan.n_ctas;
  at[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)plan.n_ctas);
  cfg.blockDim = dim3(LG_THREADS);
  cfg.dynamicSmemBytes = LG_TOTAL;
  cfg.stream = c->stream;
  cfg.attrs = at;
  cfg.numAttrs = plan.n_ctas > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, lora_grads_tc_kernel, g, c->status_dev) != cudaSuccess) return 3;
  RT_COUNT_LAUNCH(1);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace rt
