// Causal grouped-query attention on the fifth-generation tensor cores (tcgen05 + TMEM + TMA).
//
//   forward  (reference src/attention.rs:187-230): P = softmax(mask(q.k^T / sqrt(hd))), O = P.V
//
// One CTA owns 128 query rows of one head; a thread of the four softmax warps owns ONE row, which
// is one TMEM lane, so the row maximum and the row sum need no shuffles.  Per key tile of 64:
//   S = Q.K^T   tcgen05.mma, A = Q [128 x hd] and B = K [64 x hd] both K-major in shared memory
//               (TMA, 128-byte swizzle), D = S in TMEM (two buffers of 64 columns)
//   softmax     tcgen05.ld of the thread's row, mask, running maximum, p = 2^(s - m), P back into S's
//               TMEM columns in f16 as the next product's A operand
//   O += P.V    tcgen05.mma, B = V [64 x hd] read MN-major from the tile TMA brought, D = O in TMEM
// The running maximum moves only when a row's new maximum exceeds it by more than 2^8 (p stays
// below 256, exact in f16's range); only then is O rescaled in TMEM (tcgen05.ld / st), which after
// the first tiles of a row almost never happens.  K and V tiles are double buffered; QK(n+1) is
// issued before the softmax of tile n, so the tensor core works under the exponentials.  Two CTAs
// fit an SM (96 KB of shared memory, 256 TMEM columns each) and cover each other's prologue.
//
// A batch is a concatenation of independent sequences: row i sees keys j with
// seq_start[i] <= j <= i and, when a gap array is given, j outside [gap[i].x, gap[i].y) (the
// reference's `allowed` rule for packed shared-prompt groups, src/ops.rs:156-164).
// Every wait is bounded and reports through the ctx status word.
#include "ctx.h"
#include "ops.h"
#include "pdl.cuh"
#include "ptx.cuh"
#include <cuda_fp16.h>
#include <stdint.h>
#include <algorithm>
#include <utility>
#include <vector>

namespace rt {

namespace {

constexpr int BM = 128;  // query rows per CTA (TMEM lanes)
constexpr int BN = 64;   // keys per tile
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_THRESHOLD = 8.0f;  // log2 units the stale maximum may lag behind

// wait sites reported with RT_ERR_DEVICE_WAIT_TIMEOUT
enum { SITE_Q = 401, SITE_KFREE, SITE_VFREE, SITE_KFULL, SITE_SFREE, SITE_PFULL, SITE_VFULL, SITE_SFULL, SITE_PVDONE, SITE_ODONE };

template <int HD>
struct FwdLayout {
  static constexpr int PAN = HD / 64;                    // 64-column panels per row
  static constexpr uint32_t Q_PANEL = BM * 128;          // bytes: [128 rows][64 f16]
  static constexpr uint32_t KV_PANEL = BN * 128;         // bytes: [64 rows][64 f16]
  static constexpr uint32_t Q_BYTES = PAN * Q_PANEL, KV_BYTES = PAN * KV_PANEL;
  static constexpr uint32_t OFF_Q = 0, OFF_K = Q_BYTES, OFF_V = OFF_K + 2 * KV_BYTES;
  static constexpr uint32_t OFF_BAR = OFF_V + 2 * KV_BYTES;
  // Two CTAs must fit an SM's 228 KB (each also pays 1 KB of system shared memory), so the slack for
  // rounding the base up to a 1 KB boundary is 768 bytes: enough for any base that is 256-byte
  // aligned (the kernel checks, and reports a status instead of running, if it ever is not).
  static constexpr uint32_t USED = OFF_BAR + 256;
  // No less than what keeps a low-rank block away from two of these (64-wide heads): the kernel lets the next one start before
  // its blocks hold their TMEM (pdl.cuh).
  static constexpr uint32_t TOTAL = USED + 768 > TWO_BLOCKS_SMEM ? USED + 768 : TWO_BLOCKS_SMEM;
  static constexpr uint32_t TMEM_COLS = 256;               // S[2] (64 each) + O (hd <= 128)
  static constexpr uint32_t COL_S = 0, COL_O = 2 * BN;
};

__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *(uint32_t*)&h;
}

template <int HD>
__global__ void __launch_bounds__(192, 2)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                   const int* __restrict__ seq_start, const int2* __restrict__ gap, const int* __restrict__ tiles, int M, int nh,
                   int nkv, float scale, float* __restrict__ lse, int* status) {
  using L = FwdLayout<HD>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;  // 128-byte-swizzled tiles start on 1 KB boundaries
  pdl_launch_dependents();
  if (pad + L::USED > L::TOTAL) {
    pdl_wait();
    if (threadIdx.x == 0) report_status(status, RT_ERR_CUDA);
    return;
  }
  uint8_t* sm = smem_raw + pad;
  uint64_t* bars = (uint64_t*)(sm + L::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;   // [2]
  uint64_t* v_full = bars + 3;   // [2]
  uint64_t* k_free = bars + 5;   // [2]
  uint64_t* v_free = bars + 7;   // [2]
  uint64_t* s_full = bars + 9;   // [2]
  uint64_t* p_full = bars + 11;  // [2]
  uint64_t* o_done = bars + 13;  // the last product has completed: one phase, so its parity says which
  uint32_t* tmem_slot = (uint32_t*)(bars + 14);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // the tiles that see the most keys start first, every head of one before the next
  const int m0 = tiles[blockIdx.x / nh] * BM, h = (int)blockIdx.x % nh, g = h / (nh / nkv);
  const int kbeg = seq_start[m0];
  const int kend = min(m0 + BM, M);
  const int ntiles = (kend - kbeg + BN - 1) / BN;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&k_free[i], 1);
      mbar_init(&v_free[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);   // one arrival per softmax warp
    }
    mbar_init(o_done, 1);
    mbar_fence_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_o);
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  pdl_wait();  // seq_start, read above, is an input of the whole pass, not a predecessor's output

  if (warp == 4) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(q_full, L::Q_BYTES);
      for (int p = 0; p < L::PAN; ++p) tma_load_2d(sm + L::OFF_Q + p * L::Q_PANEL, &tm_q, h * HD + p * 64, m0, q_full);
      for (int n = 0; n < ntiles; ++n) {
        const int b = n & 1;
        const uint32_t free_parity = ((n >> 1) & 1) ^ 1;  // the first use of a buffer finds it free
        const int n0 = kbeg + n * BN;
        if (!mbar_wait(&k_free[b], free_parity, status, SITE_KFREE)) break;
        mbar_expect_tx(&k_full[b], L::KV_BYTES);
        for (int p = 0; p < L::PAN; ++p)
          tma_load_2d(sm + L::OFF_K + b * L::KV_BYTES + p * L::KV_PANEL, &tm_k, g * HD + p * 64, n0, &k_full[b]);
        if (!mbar_wait(&v_free[b], free_parity, status, SITE_VFREE)) break;
        mbar_expect_tx(&v_full[b], L::KV_BYTES);
        for (int p = 0; p < L::PAN; ++p)
          tma_load_2d(sm + L::OFF_V + b * L::KV_BYTES + p * L::KV_PANEL, &tm_v, g * HD + p * 64, n0, &v_full[b]);
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------ MMA issue (one thread)
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(0, 0, 0, 0, BM, BN);   // S: A, B K-major, N = 64 keys
      const uint32_t idesc_o = umma_idesc(0, 0, 0, 1, BM, HD);   // O: A K-major (P), B MN-major (V), N = hd
      const uint32_t sQ = smem_u32(sm + L::OFF_Q), sK = smem_u32(sm + L::OFF_K), sV = smem_u32(sm + L::OFF_V);
      bool ok = mbar_wait(q_full, 0, status, SITE_Q);
      auto issue_qk = [&](int n) -> bool {
        const int b = n & 1;
        const uint32_t u = (uint32_t)(n >> 1) & 1;
        if (!mbar_wait(&k_full[b], u, status, SITE_KFULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ad = umma_desc_sw128(sQ + (kk >> 2) * L::Q_PANEL + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = umma_desc_sw128(sK + b * L::KV_BYTES + (kk >> 2) * L::KV_PANEL + (kk & 3) * 32, 16, 1024);
          umma_f16(tmem_base + L::COL_S + b * BN, ad, bd, idesc_s, kk != 0);
        }
        umma_commit(&s_full[b]);
        umma_commit(&k_free[b]);
        return true;
      };
      // S's two buffers: QK(n + 2) overwrites the P that PV(n) reads, and is issued after it (the tensor
      // core works through one thread's products in order)
      if (ok) ok = issue_qk(0) && (ntiles < 2 || issue_qk(1));
      for (int n = 0; n < ntiles && ok; ++n) {
        const int b = n & 1;
        const uint32_t u = (uint32_t)(n >> 1) & 1;
        if (!mbar_wait(&p_full[b], u, status, SITE_PFULL) || !mbar_wait(&v_full[b], u, status, SITE_VFULL)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          // V tile: rows are keys (the contraction), 64-column panels L::KV_PANEL bytes apart are hd (N)
          const uint64_t bd = umma_desc_sw128(sV + b * L::KV_BYTES + kk * 2048, L::KV_PANEL, 1024);
          umma_f16_ta(tmem_base + L::COL_O, tmem_base + L::COL_S + b * BN + kk * 8, bd, idesc_o, (n | kk) != 0);
        }
        umma_commit(&v_free[b]);
        if (n + 2 < ntiles && !issue_qk(n + 2)) { ok = false; break; }
      }
      // the last arrivals of the tensor core on this CTA's barriers land before the CTA leaves
      if (ok) {
        umma_commit(o_done);
        mbar_wait(o_done, 0, status, SITE_ODONE);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax: thread = query row = TMEM lane
    const int r = warp * 32 + lane;
    const int i = m0 + r;
    const int ss_i = i < M ? seq_start[i] : 0x7fffffff;
    const int2 gp = (gap && i < M) ? gap[i] : make_int2(0, 0);
    const int ss_last = seq_start[kend - 1];  // the largest first-key index among the tile's rows
    const float sl2 = scale * LOG2E;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(warp * 32) << 16);
    float m_used = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int n = 0; n < ntiles; ++n) {
      const int b = n & 1;
      const int n0 = kbeg + n * BN;
      if (!mbar_wait(&s_full[b], (uint32_t)(n >> 1) & 1, status, SITE_SFULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t v[BN];
      tmem_ld32(lane_addr + L::COL_S + b * BN, v);
      tmem_ld32(lane_addr + L::COL_S + b * BN + 32, v + 32);
      tmem_ld_wait();
      // a tile wholly below the diagonal of every row, inside every row's sequence, needs no mask
      const bool need_mask = (n0 + BN - 1 > m0) || (n0 < ss_last);
      if (need_mask || gap != nullptr) {
        // valid keys of this row inside the tile: columns [c_lo, c_hi], minus the hidden range
        const int c_lo = ss_i - n0, c_hi = i - n0;
        const int g_lo = gp.x - n0, g_hi = gp.y - n0;
#pragma unroll
        for (int c = 0; c < BN; ++c) {
          const bool valid = c >= c_lo && c <= c_hi && (c < g_lo || c >= g_hi);
          if (!valid) v[c] = 0xff800000u;  // -inf
        }
      }
      // four interleaved chains for the maximum and for the sum: a thread is alone on its row, so the
      // instruction-level parallelism has to come from inside the row.  The scale and the running
      // maximum go into one packed fma per two scores.
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < BN; c += 2) mx4[(c >> 1) & 3] = fmaxf(fmaxf(mx4[(c >> 1) & 3], __uint_as_float(v[c])), __uint_as_float(v[c + 1]));
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;
      const bool grow = mx > m_used + RESCALE_THRESHOLD;  // also the first tile that shows the row a key
      const float m_new = grow ? mx : m_used;
      const float corr = grow ? ex2_approx(m_used - m_new) : 1.0f;  // 0 when the row had seen nothing
      const float mref = m_new == -INFINITY ? 0.f : m_new;
      l_run *= corr;
      uint32_t ph[BN / 2];
      const uint64_t sl2v = f32x2(sl2, sl2), mv = f32x2(-mref, -mref);
      uint64_t sum4[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
      for (int c = 0; c < BN; c += 2) {
        const float2 x = unpack_f32x2(fma_f32x2(f32x2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), sl2v, mv));
        const float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
        sum4[(c >> 1) & 3] = add_f32x2(sum4[(c >> 1) & 3], f32x2(p0, p1));
        ph[c >> 1] = pack_h2(p0, p1);
      }
      const float2 sum = unpack_f32x2(add_f32x2(add_f32x2(sum4[0], sum4[1]), add_f32x2(sum4[2], sum4[3])));
      l_run += sum.x + sum.y;
      m_used = m_new;
      if (n > 0 && __any_sync(0xffffffffu, grow && corr != 1.0f)) {
        // O is at rest once the previous tile's P.V has completed.  (Its phase of v_free cannot be taken for
        // another: the one before, of P.V(n - 3), was over before K(n) was loaded, and P.V(n + 1) waits for this warp.)
        if (!mbar_wait(&v_free[(n - 1) & 1], (uint32_t)((n - 1) >> 1) & 1, status, SITE_PVDONE)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t t[32];
          tmem_ld32(lane_addr + L::COL_O + c * 32, t);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 32; ++k) t[k] = __float_as_uint(__uint_as_float(t[k]) * corr);
          tmem_st32(lane_addr + L::COL_O + c * 32, t);
        }
      }
      tmem_st32(lane_addr + L::COL_S + b * BN, ph);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[b]);
    }
    // A barrier of its own: between this warp's last P and here none, one or two of the last products may have
    // completed, and the parity of a barrier that counts them all tells two of these states apart, not three.
    ok = ok && mbar_wait(o_done, 0, status, SITE_ODONE);
    if (ok) {
      // O / l as f16 into Q's shared memory (every product that read Q has completed), in the
      // layout of a swizzled TMA box, then one bulk store per 64-column panel: rows past the end of
      // the batch are clipped by the tensor map
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t t[32];
        tmem_ld32(lane_addr + L::COL_O + c * 32, t);
        tmem_ld_wait();
        uint8_t* orow = sm + L::OFF_Q + (c >> 1) * L::Q_PANEL + r * 128;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint4 w;
          w.x = pack_h2(__uint_as_float(t[8 * k]) * inv, __uint_as_float(t[8 * k + 1]) * inv);
          w.y = pack_h2(__uint_as_float(t[8 * k + 2]) * inv, __uint_as_float(t[8 * k + 3]) * inv);
          w.z = pack_h2(__uint_as_float(t[8 * k + 4]) * inv, __uint_as_float(t[8 * k + 5]) * inv);
          w.w = pack_h2(__uint_as_float(t[8 * k + 6]) * inv, __uint_as_float(t[8 * k + 7]) * inv);
          const int chunk = (c & 1) * 4 + k;
          *(uint4*)(orow + ((chunk ^ (r & 7)) << 4)) = w;
        }
      }
      if (i < M) lse[(size_t)h * M + i] = m_used / LOG2E + logf(l_run);
      fence_proxy_async_smem();
    }
    __syncwarp();
    named_barrier_sync(1, 128);  // the four softmax warps only, also after a wait that gave up
    if (ok && threadIdx.x == 0) {
      for (int p = 0; p < L::PAN; ++p) tma_store_2d(&tm_o, h * HD + p * 64, m0, sm + L::OFF_Q + p * L::Q_PANEL);
      bulk_commit_group();
      bulk_wait_group_read<0>();  // shared memory may go once the store has read it
    }
  }

  // ---------------------------------------------------------------- teardown
  if (*(volatile int*)status != 0) {
    // a wait gave up somewhere: give copies already in flight time to land before shared memory goes away
    for (int k = 0; k < 1000; ++k) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

template <int HD>
int fwd_tc_impl(rt_ctx* c, const __half* q, const __half* k, const __half* v, const AttnBatch& b, int nh, int nkv, __half* o, float* lse) {
  const int M = b.M;
  using L = FwdLayout<HD>;
  if (!c->raise_smem(attn_fwd_tc_kernel<HD>, L::TOTAL)) return 3;
  CUtensorMap tq, tk, tv, to;
  if (tensor_map_f16_2d(c, &tq, q, (uint64_t)M, (uint64_t)nh * HD, 64, BM)) return 3;
  if (tensor_map_f16_2d(c, &to, o, (uint64_t)M, (uint64_t)nh * HD, 64, BM)) return 3;
  if (tensor_map_f16_2d(c, &tk, k, (uint64_t)M, (uint64_t)nkv * HD, 64, BN)) return 3;
  if (tensor_map_f16_2d(c, &tv, v, (uint64_t)M, (uint64_t)nkv * HD, 64, BN)) return 3;
  const unsigned grid = (unsigned)nh * ((M + BM - 1) / BM);
  pdl(attn_fwd_tc_kernel<HD>, grid, 192, L::TOTAL, c->stream)(tq, tk, tv, to, b.seq_start, (const int2*)b.gap, b.tiles_q, M, nh, nkv,
                                                            1.0f / sqrtf((float)HD), lse, c->status_dev);
  RT_COUNT_LAUNCH(1);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}


// ==================================================================== backward
//   (reference src/attention.rs:272-328)  dV = P^T.dO, dP = dO.V^T, dS = P*(dP - rowsum(P*dP))/sqrt(hd),
//   dQ = dS.K, dK = dS^T.Q, the K/V gradients summed over the query heads that share a KV head.
// Two kernels, so that every output element has exactly one writer (no float atomics: the same
// bits every run).  P is recomputed from the forward's log-sum-exp.  dO arrives as f16 rows
// divided by a per-row factor; a query row enters the sums over queries with weight
// factor / top (top = a power of two >= the largest factor, so the weights change no mantissa),
// and dQ rows get their own factor back.
//
// Both kernels keep sixteen compute warps on an SM in two groups, so one group's exponentials run
// under the other's products and four warps per scheduler cover each other's latencies: in one CTA that
// takes alternate work items (dK/dV), or as two CTAs (dQ).  In a group, warps w and w + 4 share TMEM lane quarter w and take 32 of an item's 64
// columns each.  P and dS go back into the TMEM columns that S and dP came in, as the A operands of
// the next products: no shared-memory round trip, no proxy fence, and no wait for a buffer, because
// an item's scores are issued after the products that read the P of the item two before, and the
// tensor core works through one thread's products in order.  (One group of eight warps, P and dS
// through shared memory, took about 3400 cycles per item of 128 x 64 against 1150 of products.)

// ------------------------------------------------------------------ dK, dV: per (128 keys, KV head)
// Thread = key row = TMEM lane.  K and V stay in shared memory; the query tiles of 64 rows that can see
// these keys stream through a ring.  Per item: S^T = K.Q^T and dP^T = V.dO^T into TMEM, the threads
// turn them into P^T and dS^T, then dV += P^T.dO and dK += dS^T.Q with Q and dO read MN-major from the
// same tiles.  A CTA takes four of the query heads that share a KV head; more go to the CTAs of one cluster
// (up to eight), whose sums meet in shared memory at the end and are added in head order.  (14 heads over
// two KV heads, 8 x 1024 tokens: one CTA for the seven heads 105 us, four and three 74, clusters of four 95, of
// seven 142; 24 heads over 8, 4 x 2048: three heads in one CTA 289 us, clusters of two 371.)  The line
// depends on the model only, so a sequence's sums do not depend on its batch.  TMEM: 2 x 64 + 2 x 64 + hd + hd columns (512 for hd = 128).
// P (<= 1, times a row weight <= 1) and dS are handed to the tensor cores in f16, whose normal
// range ends at 6e-5: attention probabilities of long rows and the gradients of lightly weighted
// rows live below that.  They are therefore stored times a power of two (exact), which the f32
// results are divided by again: 2^14 keeps P.w <= 16384, 2^10 keeps dS inside f16 for |dP - delta|
// up to ~700.
constexpr float P_BOOST = 16384.0f, P_BOOST_LOG2 = 14.0f, DS_BOOST = 1024.0f;
constexpr int BQ = 64;  // query rows per work item
constexpr int BWD_THREADS = 576, BWD_TMA_WARP = 16, BWD_MMA_WARP = 17;  // warps 0-15 compute
constexpr int MAX_HEAD_CTAS = 8;  // portable cluster size
enum { SITE_B_KV = 451, SITE_B_QFREE, SITE_B_QFULL, SITE_B_PFULL, SITE_B_SFULL, SITE_B_PDDONE, SITE_B_END };

// What dK/dV needs per (head, query row), prepared by the delta kernel as [nh][query_pitch(M)] f32 (whole
// tiles, so that a tile's 64 values are one aligned bulk copy): the exponent offset
// log2(weight * 2^14) - lse * log2(e), so that P.w.2^14 = 2^(s.scale.log2(e) + offset), -inf for rows past the
// batch and rows of weight 0; and -delta * scale * 2^10 / 2^14.  (Gathered per item by the producer warp, their
// latency, not the products, set the pace: 3400 cycles per item.)
__host__ __device__ inline size_t query_pitch(int M) { return ((size_t)M + 63) / 64 * 64; }

template <int HD>
struct DkvLayout {
  static constexpr int PAN = HD / 64;
  static constexpr uint32_t KV_PANEL = 128 * 128, Q_PANEL = BQ * 128;
  static constexpr uint32_t KV_BYTES = PAN * KV_PANEL, Q_BYTES = PAN * Q_PANEL;
  static constexpr int NS = 4;  // ring of items: Q, dO and the per-query vectors; a slot is released by the item's last product
  static constexpr uint32_t OFF_K = 0, OFF_V = KV_BYTES, OFF_Q = 2 * KV_BYTES, OFF_DO = OFF_Q + NS * Q_BYTES;
  static constexpr uint32_t OFF_AUX = OFF_DO + NS * Q_BYTES;
  static constexpr uint32_t AUX_BYTES = 2 * BQ * 4;  // exponent offset and scaled -delta per query row
  static constexpr uint32_t OFF_BAR = OFF_AUX + NS * AUX_BYTES;
  static constexpr uint32_t USED = OFF_BAR + 256, TOTAL = USED + 1024;
  static_assert(TOTAL >= TMEM_KERNEL_SMEM, "a matmul's block could share its SM (pdl.cuh)");
  static constexpr uint32_t COL_ST = 0, COL_DPT = 2 * BQ, COL_DV = 4 * BQ, COL_DK = 4 * BQ + HD;
  static constexpr uint32_t TMEM_COLS = 512;
  // the CTA's sums for its cluster, [2][128 keys][hd + 4] f32, over the operands once those are used up
  static constexpr int PITCH = HD + 4;
  static_assert(2 * 128 * PITCH * 4 <= (int)OFF_AUX, "the sums fit over the operands");
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}

template <int HD>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkdv_tc_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                        const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                        const float* tops, const float* query_vecs, const int* __restrict__ seq_start,
                        const int2* __restrict__ gap, const int2* __restrict__ tiles, int M, int nh, int nkv, int heads_per_cta,
                        int n_ctas, float scale, float* __restrict__ dk, float* __restrict__ dv, int* status) {
  using L = DkvLayout<HD>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint64_t* bars = (uint64_t*)(sm + L::OFF_BAR);
  constexpr int NS = L::NS;
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;         // [NS] Q, dO and the per-query vectors of an item
  uint64_t* q_free = bars + 1 + NS;    // [NS]
  uint64_t* s_full = bars + 1 + 2 * NS;   // [2]  S^T and dP^T of an item are in TMEM
  uint64_t* p_full = bars + 3 + 2 * NS;   // [2]  ... and have become P^T and dS^T
  uint64_t* pd_done = bars + 5 + 2 * NS;  //      every dV, dK product has completed
  uint32_t* tmem_slot = (uint32_t*)(bars + 6 + 2 * NS);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int per_tile = nkv * n_ctas, g = (int)blockIdx.x % per_tile / n_ctas, rank = n_ctas > 1 ? (int)cluster_ctarank() : 0, group = nh / nkv;
  const int2 tile = tiles[blockIdx.x / per_tile];
  const int n0 = tile.x * 128;
  const int h0 = g * group + rank * heads_per_cta, n_heads = min(heads_per_cta, group - rank * heads_per_cta);
  // queries that can see these keys: [n0, end of the sequence holding the tile's last key)
  const int nqt = (tile.y - n0 + BQ - 1) / BQ;
  const int n_items = n_heads * nqt;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < NS; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_free[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);  // one arrival per warp of the group
    }
    mbar_init(pd_done, 1);
    mbar_fence_init();
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_do);
  }
  if (warp == BWD_MMA_WARP) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  pdl_wait();
  // Only now: the dQ kernel behind this one runs beside it without a wait, and takes everything older as complete (pdl.cuh).
  pdl_launch_dependents();

  bool ok = true;
  if (warp == BWD_TMA_WARP) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * L::KV_BYTES);
      for (int p = 0; p < L::PAN; ++p) {
        tma_load_2d(sm + L::OFF_K + p * L::KV_PANEL, &tm_k, g * HD + p * 64, n0, kv_full);
        tma_load_2d(sm + L::OFF_V + p * L::KV_PANEL, &tm_v, g * HD + p * 64, n0, kv_full);
      }
      const size_t pitch = query_pitch(M);
      int rb = 0, qt = 0, h = h0;
      uint32_t ph = 0;
      for (int it = 0; it < n_items; ++it) {
        const int m0 = n0 + qt * BQ;
        if (!mbar_wait(&q_free[rb], ph ^ 1, status, SITE_B_QFREE)) break;
        mbar_expect_tx(&q_full[rb], 2 * L::Q_BYTES + L::AUX_BYTES);
        for (int p = 0; p < L::PAN; ++p) {
          tma_load_2d(sm + L::OFF_Q + rb * L::Q_BYTES + p * L::Q_PANEL, &tm_q, h * HD + p * 64, m0, &q_full[rb]);
          tma_load_2d(sm + L::OFF_DO + rb * L::Q_BYTES + p * L::Q_PANEL, &tm_do, h * HD + p * 64, m0, &q_full[rb]);
        }
        const float* vec = query_vecs + (size_t)h * pitch + m0;
        uint8_t* aux = sm + L::OFF_AUX + rb * L::AUX_BYTES;
        bulk_load_1d(aux, vec, BQ * 4, &q_full[rb]);
        bulk_load_1d(aux + BQ * 4, vec + (size_t)nh * pitch, BQ * 4, &q_full[rb]);
        if (++rb == NS) { rb = 0; ph ^= 1; }
        if (++qt == nqt) { qt = 0; ++h; }
      }
    }
  } else if (warp == BWD_MMA_WARP) {
    // ------------------------------------------------------------ MMA issue (one thread)
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(0, 0, 0, 0, 128, BQ);
      const uint32_t idesc_g = umma_idesc(0, 0, 0, 1, 128, HD);
      const uint32_t sK = smem_u32(sm + L::OFF_K), sV = smem_u32(sm + L::OFF_V), sQ = smem_u32(sm + L::OFF_Q);
      const uint32_t sDO = smem_u32(sm + L::OFF_DO);
      ok = mbar_wait(kv_full, 0, status, SITE_B_KV);
      auto issue_s = [&](int it) -> bool {
        const int b = it & 1, rb = it % NS;  // TMEM buffer, ring slot
        if (!mbar_wait(&q_full[rb], (uint32_t)(it / NS) & 1, status, SITE_B_QFULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ad = umma_desc_sw128(sK + (kk >> 2) * L::KV_PANEL + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = umma_desc_sw128(sQ + rb * L::Q_BYTES + (kk >> 2) * L::Q_PANEL + (kk & 3) * 32, 16, 1024);
          umma_f16(tmem_base + L::COL_ST + b * BQ, ad, bd, idesc_s, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ad = umma_desc_sw128(sV + (kk >> 2) * L::KV_PANEL + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = umma_desc_sw128(sDO + rb * L::Q_BYTES + (kk >> 2) * L::Q_PANEL + (kk & 3) * 32, 16, 1024);
          umma_f16(tmem_base + L::COL_DPT + b * BQ, ad, bd, idesc_s, kk != 0);
        }
        umma_commit(&s_full[b]);
        return true;
      };
      if (ok) ok = issue_s(0) && (n_items < 2 || issue_s(1));
      for (int it = 0; it < n_items && ok; ++it) {
        const int b = it & 1, rb = it % NS;
        if (!mbar_wait(&p_full[b], ((uint32_t)it >> 1) & 1, status, SITE_B_PFULL)) { ok = false; break; }
        tc_fence_after();
        // A operands in TMEM: 16 queries are 8 columns; queries 32.. of an item start 32 columns on (each half where its threads read S)
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk) {
          // dO / Q tiles: rows are queries (the contraction), 64-column panels Q_PANEL bytes apart are hd (N)
          const uint64_t bo = umma_desc_sw128(sDO + rb * L::Q_BYTES + kk * 2048, L::Q_PANEL, 1024);
          umma_f16_ta(tmem_base + L::COL_DV, tmem_base + L::COL_ST + b * BQ + (kk >> 1) * 32 + (kk & 1) * 8, bo, idesc_g, (it | kk) != 0);
        }
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk) {
          const uint64_t bq = umma_desc_sw128(sQ + rb * L::Q_BYTES + kk * 2048, L::Q_PANEL, 1024);
          umma_f16_ta(tmem_base + L::COL_DK, tmem_base + L::COL_DPT + b * BQ + (kk >> 1) * 32 + (kk & 1) * 8, bq, idesc_g, (it | kk) != 0);
        }
        umma_commit(&q_free[rb]);
        if (it + 2 < n_items && !issue_s(it + 2)) { ok = false; break; }
      }
      if (ok) {
        umma_commit(pd_done);
        mbar_wait(pd_done, 0, status, SITE_B_END);
      }
    }
  } else {
    // ------------------------------------------------------------ compute: key row = TMEM lane
    const int grp = warp >> 3, quarter = warp & 3, hf = (warp >> 2) & 1;
    const int r = quarter * 32 + lane;
    const int j = n0 + r;
    const float sl2 = scale * LOG2E, dsc = scale * (DS_BOOST / P_BOOST);
    const uint64_t sl2v = f32x2(sl2, sl2), dscv = f32x2(dsc, dsc);
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t st_col = lane_addr + L::COL_ST + grp * BQ + hf * 32, dp_col = lane_addr + L::COL_DPT + grp * BQ + hf * 32;
    const int ss_last = seq_start[min(n0 + 128, M) - 1];  // where the sequence of the tile's last key starts
    int qt = grp < nqt ? grp : grp % nqt;  // query tile of the item, advanced by two
    for (int it = grp; it < n_items; it += 2) {
      const int rb = it % NS;
      const int m0 = n0 + qt * BQ;
      qt += 2;
      while (qt >= nqt) qt -= nqt;
      if (!mbar_wait(&s_full[grp], ((uint32_t)it >> 1) & 1, status, SITE_B_SFULL)) { ok = false; break; }
      // (completed long ago; passing it makes the copied per-query vectors visible here)
      if (!mbar_wait(&q_full[rb], (uint32_t)(it / NS) & 1, status, SITE_B_QFULL)) { ok = false; break; }
      tc_fence_after();
      const float* aux = (const float*)(sm + L::OFF_AUX + rb * L::AUX_BYTES);
      // A tile whose queries all lie past these keys, inside the sequence of all of them, without hidden
      // ranges, needs no mask.  (Past the last key every query up to tile.y is of that key's sequence.)
      const bool need_mask = m0 < n0 + 127 || ss_last > n0 || m0 + BQ > tile.y;
#pragma unroll
      for (int h2 = 0; h2 < 2; ++h2) {  // 16 of this thread's 32 query columns at a time: what the registers have room for
        uint32_t st[16], dp[16], ph[8], dh[8];
        tmem_ld16(st_col + h2 * 16, st);
        tmem_ld16(dp_col + h2 * 16, dp);
        tmem_ld_wait();
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
          // element (key row j, query column i): P^T (weighted) and dS^T, two columns per packed operation, the
          // per-query vectors fetched four at a time
          const int il0 = hf * 32 + h2 * 16 + c4 * 4;
          const float4 ea = *(const float4*)(aux + il0), de = *(const float4*)(aux + BQ + il0);
          const float2 x0 = unpack_f32x2(fma_f32x2(f32x2(__uint_as_float(st[c4 * 4]), __uint_as_float(st[c4 * 4 + 1])), sl2v, f32x2(ea.x, ea.y)));
          const float2 x1 = unpack_f32x2(fma_f32x2(f32x2(__uint_as_float(st[c4 * 4 + 2]), __uint_as_float(st[c4 * 4 + 3])), sl2v, f32x2(ea.z, ea.w)));
          float pv[4] = {ex2_approx(x0.x), ex2_approx(x0.y), ex2_approx(x1.x), ex2_approx(x1.y)};
          if (need_mask) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int m = m0 + il0 + e;
              pv[e] = (j <= m && j >= seq_start[min(m, M - 1)]) ? pv[e] : 0.f;  // (rows past the batch: p is 0 already)
            }
          }
          if (gap != nullptr) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int2 gm = gap[min(m0 + il0 + e, M - 1)];
              pv[e] = (j < gm.x || j >= gm.y) ? pv[e] : 0.f;
            }
          }
          const uint64_t d0 = fma_f32x2(f32x2(__uint_as_float(dp[c4 * 4]), __uint_as_float(dp[c4 * 4 + 1])), dscv, f32x2(de.x, de.y));
          const uint64_t d1 = fma_f32x2(f32x2(__uint_as_float(dp[c4 * 4 + 2]), __uint_as_float(dp[c4 * 4 + 3])), dscv, f32x2(de.z, de.w));
          const float2 s0 = unpack_f32x2(mul_f32x2(f32x2(pv[0], pv[1]), d0)), s1 = unpack_f32x2(mul_f32x2(f32x2(pv[2], pv[3]), d1));
          ph[2 * c4] = pack_h2(pv[0], pv[1]);
          ph[2 * c4 + 1] = pack_h2(pv[2], pv[3]);
          dh[2 * c4] = pack_h2(s0.x, s0.y);
          dh[2 * c4 + 1] = pack_h2(s1.x, s1.y);
        }
        tmem_st8(st_col + h2 * 8, ph);
        tmem_st8(dp_col + h2 * 8, dh);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[grp]);
    }
    // group 0 hands out dK, group 1 dV; each of a row's two threads half of its columns, into shared memory, from
    // where a row leaves as one bulk copy (a thread per row storing 16 bytes at a time touched 32 sectors per
    // instruction, 8000 cycles of a CTA's 17000 outside its items: 16 x 512 tokens, 16 heads on 8, 91 -> 77 us, dQ 73 -> 60)
    if (ok) ok = mbar_wait(pd_done, 0, status, SITE_B_PDDONE);
    if (ok) {
      tc_fence_after();
      // a key row only ever meets queries of its own sequence, so its sums are in units of that sequence's largest factor
      const float top_j = tops[min(j, M - 1)];
      const float sc = n_ctas > 1 ? 1.0f : top_j * (grp == 0 ? 1.0f / DS_BOOST : 1.0f / P_BOOST);
      float* row = (float*)sm + (grp * 128 + r) * L::PITCH;
#pragma unroll
      for (int cc = 0; cc < HD / 64; ++cc) {
        const int c = hf * (HD / 64) + cc;
        uint32_t a[32];
        tmem_ld32(lane_addr + (grp == 0 ? L::COL_DK : L::COL_DV) + c * 32, a);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          *(float4*)(row + c * 32 + 4 * k) = make_float4(__uint_as_float(a[4 * k]) * sc, __uint_as_float(a[4 * k + 1]) * sc,
                                                         __uint_as_float(a[4 * k + 2]) * sc, __uint_as_float(a[4 * k + 3]) * sc);
      }
      fence_proxy_async_smem();
    }
    if (n_ctas == 1) {
      __syncwarp();
      named_barrier_sync(1 + grp, 256);  // also after a wait that gave up: nobody is left waiting here
      if (ok && hf == 0 && j < M) {
        bulk_store_1d((grp == 0 ? dk : dv) + ((size_t)j * nkv + g) * HD, (float*)sm + (grp * 128 + r) * L::PITCH, HD * 4);
        bulk_commit_group();
        bulk_wait_group_read<0>();
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
    cluster_sync_all();  // every head's sums are in its CTA's shared memory
    // this CTA's share of the (dK | dV, key, four columns) items, added up in head order
    constexpr int ITEMS = 2 * 128 * (HD / 4);
    const int per = (ITEMS + n_ctas - 1) / n_ctas, end = min(ITEMS, (rank + 1) * per);
    if (ok)
      for (int e = rank * per + threadIdx.x; e < end; e += BWD_THREADS) {
        const int c = (e % (HD / 4)) * 4, kr = (e / (HD / 4)) & 127, which = e / (HD / 4 * 128), j = n0 + kr;
        if (j >= M) continue;
        const uint32_t a = smem_u32(sm) + (uint32_t)((which * 128 + kr) * L::PITCH + c) * 4u;
        float4 x[MAX_HEAD_CTAS];
#pragma unroll
        for (int k = 0; k < MAX_HEAD_CTAS; ++k)
          if (k < n_ctas) x[k] = ld_cluster_f4(mapa_u32(a, (uint32_t)k));
        float4 s = x[0];
#pragma unroll
        for (int k = 1; k < MAX_HEAD_CTAS; ++k)
          if (k < n_ctas) { s.x += x[k].x; s.y += x[k].y; s.z += x[k].z; s.w += x[k].w; }
        const float sc = tops[j] * (which == 0 ? 1.0f / DS_BOOST : 1.0f / P_BOOST);
        *(float4*)((which == 0 ? dk : dv) + ((size_t)j * nkv + g) * HD + c) = make_float4(s.x * sc, s.y * sc, s.z * sc, s.w * sc);
      }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while its shared memory may still be read
  } else {
    __syncthreads();
  }
  if (warp == BWD_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

// ------------------------------------------------------------------ dQ: one CTA per (128 query rows, head)
// Thread = query row = TMEM lane.  Q and dO stay in shared memory; per key tile of 64:
// S = Q.K^T and dP = dO.V^T into TMEM, dS = P*(dP - delta)*scale back into S's columns in f16, then
// dQ += dS.K with K read MN-major from the tile that just served Q.K^T.  Two CTAs fit an SM (112 KB of
// shared memory, 256 TMEM columns, eight compute warps each): they are each other's second group, and
// one's prologue and output run under the other's tiles, which is most of the time at 512 tokens a
// sequence.
enum { SITE_Q_QDO = 471, SITE_Q_KFREE, SITE_Q_VFREE, SITE_Q_KFULL, SITE_Q_VFULL, SITE_Q_DSFULL, SITE_Q_SFULL, SITE_Q_DQDONE, SITE_Q_END };

template <int HD>
struct DqLayout {
  static constexpr int PAN = HD / 64;
  static constexpr uint32_t Q_PANEL = BM * 128, KV_PANEL = BN * 128;
  static constexpr uint32_t Q_BYTES = PAN * Q_PANEL, KV_BYTES = PAN * KV_PANEL;
  static constexpr int NK = 2;  // K slots (a slot is released by its tile's dQ product; V's one slot by the dP product)
  static constexpr uint32_t OFF_Q = 0, OFF_DO = Q_BYTES, OFF_K = 2 * Q_BYTES, OFF_V = OFF_K + NK * KV_BYTES;
  static constexpr uint32_t OFF_BAR = OFF_V + KV_BYTES;
  static constexpr uint32_t USED = OFF_BAR + 256;
  static constexpr uint32_t TOTAL = USED + 768 > TWO_BLOCKS_SMEM ? USED + 768 : TWO_BLOCKS_SMEM;  // slack and least as in the forward's layout
  static constexpr uint32_t COL_S = 0, COL_DP = BN, COL_DQ = 2 * BN, TMEM_COLS = 256;
  static constexpr int PITCH = HD + 4;  // dQ as f32 over the operands once those are used up
  static_assert(BM * PITCH * 4 <= (int)OFF_BAR, "dQ fits over the operands");
};

constexpr int DQ_THREADS = 320, DQ_TMA_WARP = 8, DQ_MMA_WARP = 9;  // warps 0-7 compute

template <int HD>
__global__ void __launch_bounds__(DQ_THREADS, 2)
attn_bwd_dq_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                      const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                      const float* row_scale, const float* lse,
                      const float* query_vecs, const int* __restrict__ seq_start, const int2* __restrict__ gap,
                      const int* __restrict__ tiles, int M, int nh, int nkv, float scale, float* __restrict__ dq, int* status) {
  using L = DqLayout<HD>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
  pdl_launch_dependents();
  if (pad + L::USED > L::TOTAL) {
    pdl_wait();
    if (threadIdx.x == 0) report_status(status, RT_ERR_CUDA);
    return;
  }
  uint8_t* sm = smem_raw + pad;
  uint64_t* bars = (uint64_t*)(sm + L::OFF_BAR);
  constexpr int NK = L::NK;
  uint64_t* qdo_full = bars + 0;
  uint64_t* k_full = bars + 1;            // [NK]
  uint64_t* k_free = bars + 1 + NK;       // [NK]
  uint64_t* v_full = bars + 1 + 2 * NK;
  uint64_t* v_free = bars + 2 + 2 * NK;
  uint64_t* s_full = bars + 3 + 2 * NK;
  uint64_t* ds_full = bars + 4 + 2 * NK;
  uint64_t* dq_done = bars + 5 + 2 * NK;
  uint32_t* tmem_slot = (uint32_t*)(bars + 6 + 2 * NK);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // the tiles that see the most keys start first, every head of one before the next
  const int m0 = tiles[blockIdx.x / nh] * BM, h = (int)blockIdx.x % nh, g = h / (nh / nkv);
  const int kbeg = seq_start[m0];
  const int kend = min(m0 + BM, M);
  const int ntiles = (kend - kbeg + BN - 1) / BN;

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int i = 0; i < NK; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_free[i], 1);
    }
    mbar_init(v_full, 1);
    mbar_init(v_free, 1);
    mbar_init(s_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(dq_done, 1);
    mbar_fence_init();
    prefetch_tmap(&tm_q);
    prefetch_tmap(&tm_do);
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
  }
  if (warp == DQ_MMA_WARP) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == 0) pdl_unwaited();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  // no wait here: what this kernel reads was complete before the dK/dV kernel, in front of it, let it start

  if (warp == DQ_TMA_WARP) {
    if (elect_one()) {
      mbar_expect_tx(qdo_full, 2 * L::Q_BYTES);
      for (int p = 0; p < L::PAN; ++p) {
        tma_load_2d(sm + L::OFF_Q + p * L::Q_PANEL, &tm_q, h * HD + p * 64, m0, qdo_full);
        tma_load_2d(sm + L::OFF_DO + p * L::Q_PANEL, &tm_do, h * HD + p * 64, m0, qdo_full);
      }
      for (int n = 0; n < ntiles; ++n) {
        const int rb = n % NK, n0 = kbeg + n * BN;
        if (!mbar_wait(&k_free[rb], ((uint32_t)(n / NK) & 1) ^ 1, status, SITE_Q_KFREE)) break;
        mbar_expect_tx(&k_full[rb], L::KV_BYTES);
        for (int p = 0; p < L::PAN; ++p)
          tma_load_2d(sm + L::OFF_K + rb * L::KV_BYTES + p * L::KV_PANEL, &tm_k, g * HD + p * 64, n0, &k_full[rb]);
        if (!mbar_wait(v_free, ((uint32_t)n & 1) ^ 1, status, SITE_Q_VFREE)) break;
        mbar_expect_tx(v_full, L::KV_BYTES);
        for (int p = 0; p < L::PAN; ++p) tma_load_2d(sm + L::OFF_V + p * L::KV_PANEL, &tm_v, g * HD + p * 64, n0, v_full);
      }
    }
  } else if (warp == DQ_MMA_WARP) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc(0, 0, 0, 0, BM, BN);
      const uint32_t idesc_g = umma_idesc(0, 0, 0, 1, BM, HD);
      const uint32_t sQ = smem_u32(sm + L::OFF_Q), sDO = smem_u32(sm + L::OFF_DO), sK = smem_u32(sm + L::OFF_K);
      const uint32_t sV = smem_u32(sm + L::OFF_V);
      bool ok = mbar_wait(qdo_full, 0, status, SITE_Q_QDO);
      // S and dP have one buffer each: a tile's are issued after the product that reads the dS before them
      auto issue_s = [&](int n) -> bool {
        const int rb = n % NK;
        if (!mbar_wait(&k_full[rb], (uint32_t)(n / NK) & 1, status, SITE_Q_KFULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ad = umma_desc_sw128(sQ + (kk >> 2) * L::Q_PANEL + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = umma_desc_sw128(sK + rb * L::KV_BYTES + (kk >> 2) * L::KV_PANEL + (kk & 3) * 32, 16, 1024);
          umma_f16(tmem_base + L::COL_S, ad, bd, idesc_s, kk != 0);
        }
        if (!mbar_wait(v_full, (uint32_t)n & 1, status, SITE_Q_VFULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t ad = umma_desc_sw128(sDO + (kk >> 2) * L::Q_PANEL + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = umma_desc_sw128(sV + (kk >> 2) * L::KV_PANEL + (kk & 3) * 32, 16, 1024);
          umma_f16(tmem_base + L::COL_DP, ad, bd, idesc_s, kk != 0);
        }
        umma_commit(s_full);
        umma_commit(v_free);
        return true;
      };
      if (ok) ok = issue_s(0);
      for (int n = 0; n < ntiles && ok; ++n) {
        const int rb = n % NK;
        if (!mbar_wait(ds_full, (uint32_t)n & 1, status, SITE_Q_DSFULL)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          const uint64_t bd = umma_desc_sw128(sK + rb * L::KV_BYTES + kk * 2048, L::KV_PANEL, 1024);  // K tile read MN-major: rows are keys
          umma_f16_ta(tmem_base + L::COL_DQ, tmem_base + L::COL_S + (kk >> 1) * 32 + (kk & 1) * 8, bd, idesc_g, (n | kk) != 0);
        }
        umma_commit(&k_free[rb]);
        if (n + 1 < ntiles && !issue_s(n + 1)) { ok = false; break; }
      }
      if (ok) {
        umma_commit(dq_done);
        mbar_wait(dq_done, 0, status, SITE_Q_END);
      }
    }
  } else {
    // ------------------------------------------------------------ compute: query row = TMEM lane
    const int quarter = warp & 3, hf = warp >> 2;
    const int r = quarter * 32 + lane;
    const int i = m0 + r;
    const int ss_i = i < M ? seq_start[i] : 0x7fffffff;
    const int2 gp = (gap && i < M) ? gap[i] : make_int2(0, 0);
    const int ss_last = seq_start[kend - 1];
    const float sl2 = scale * LOG2E, dsc = scale * DS_BOOST;
    const float l2 = i < M ? -lse[(size_t)h * M + i] * LOG2E : 0.f;
    const float dl = i < M ? query_vecs[(nh + h) * query_pitch(M) + i] * P_BOOST : 0.f;  // -delta * scale * 2^10
    const uint64_t sl2v = f32x2(sl2, sl2), l2v = f32x2(l2, l2), dscv = f32x2(dsc, dsc), dlv = f32x2(dl, dl);
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_col = lane_addr + L::COL_S + hf * 32, dp_col = lane_addr + L::COL_DP + hf * 32;
    bool ok = true;
    for (int n = 0; n < ntiles; ++n) {
      const int n0 = kbeg + n * BN;
      if (!mbar_wait(s_full, (uint32_t)n & 1, status, SITE_Q_SFULL)) { ok = false; break; }
      tc_fence_after();
      const bool need_mask = (n0 + BN - 1 > m0) || (n0 < ss_last);
      const int c_lo = ss_i - n0, c_hi = i - n0, g_lo = gp.x - n0, g_hi = gp.y - n0;
#pragma unroll
      for (int h2 = 0; h2 < 2; ++h2) {
        uint32_t sv[16], dp[16], dh[8];
        tmem_ld16(s_col + h2 * 16, sv);
        tmem_ld16(dp_col + h2 * 16, dp);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
          const int cc = hf * 32 + h2 * 16 + c;
          const float2 x = unpack_f32x2(fma_f32x2(f32x2(__uint_as_float(sv[c]), __uint_as_float(sv[c + 1])), sl2v, l2v));
          float p0 = ex2_approx(x.x), p1 = ex2_approx(x.y);
          if (need_mask) {
            p0 = (cc >= c_lo && cc <= c_hi) ? p0 : 0.f;
            p1 = (cc + 1 >= c_lo && cc + 1 <= c_hi) ? p1 : 0.f;
          }
          if (gap != nullptr) {
            p0 = (cc < g_lo || cc >= g_hi) ? p0 : 0.f;
            p1 = (cc + 1 < g_lo || cc + 1 >= g_hi) ? p1 : 0.f;
          }
          const float2 ds = unpack_f32x2(mul_f32x2(f32x2(p0, p1), fma_f32x2(f32x2(__uint_as_float(dp[c]), __uint_as_float(dp[c + 1])), dscv, dlv)));
          dh[c >> 1] = pack_h2(ds.x, ds.y);
        }
        tmem_st8(s_col + h2 * 8, dh);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    // each of a row's two threads hands out half of its columns
    if (ok) ok = mbar_wait(dq_done, 0, status, SITE_Q_DQDONE);
    if (ok) {
      tc_fence_after();
      // a query row's gradient carries only that row's factor
      const float sc = (i < M ? row_scale[i] : 0.f) * (1.0f / DS_BOOST);
      constexpr int NC = HD / 2;
      const int c0 = hf * NC;
      float* qrow = (float*)sm + r * L::PITCH + c0;  // a row leaves shared memory as one bulk copy, as in dK/dV
#pragma unroll
      for (int c = 0; c < NC; c += 16) {
        uint32_t a[16];
        tmem_ld16(lane_addr + L::COL_DQ + c0 + c, a);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          *(float4*)(qrow + c + 4 * k) = make_float4(__uint_as_float(a[4 * k]) * sc, __uint_as_float(a[4 * k + 1]) * sc,
                                                     __uint_as_float(a[4 * k + 2]) * sc, __uint_as_float(a[4 * k + 3]) * sc);
      }
      fence_proxy_async_smem();
    }
    __syncwarp();
    named_barrier_sync(1 + quarter, 64);  // the row's two warps; also after a wait that gave up
    if (ok && hf == 0 && i < M) {
      bulk_store_1d(dq + ((size_t)i * nh + h) * HD, (float*)sm + r * L::PITCH, HD * 4);
      bulk_commit_group();
      bulk_wait_group_read<0>();
    }
  }

  pdl_wait();  // for dK/dV: whoever waits for this kernel has waited for both
  if (*(volatile int*)status != 0) {
    for (int k = 0; k < 1000; ++k) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == DQ_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

// delta[h, m] = sum_d O * dO (the row sum of P * dP, src/attention.rs:282-287), handed on as the two
// per-query vectors of dK/dV (see query_pitch), and the row weights: tops[m] is a power of two >= the
// largest factor among the rows of m's own sequence (nothing a sequence's backward sees may depend on its
// batch mates; 1 for an all-zero sequence), a row's weight its factor / tops[m].  A pure stream over O and
// dO, one block per (128 tokens, head): HD / 8 lanes share a row with one 16-byte load of each operand per
// lane, all of the block's loads in flight before the first use; the scan of the sequence's factors (a
// launch of its own before, one block for the whole batch: 12 us at 8192 tokens) runs under them.
template <int HD>
__global__ void __launch_bounds__(256)
attn_delta_tc_kernel(const __half* o, const __half* dO, const float* lse,
                     const float* row_scale, const int* __restrict__ seq_start, const int2* __restrict__ tiles, int M, int nh,
                     float scale, float* __restrict__ query_vecs, float* __restrict__ tops) {
  constexpr int LPR = HD / 8, RPW = 32 / LPR, UN = 16 / RPW;
  __shared__ int s_max[129];     // by where the sequence starts: its first token in this tile, 128: before the tile
  __shared__ float s_delta[128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPR, grp = lane / LPR;
  // Before the wait what the batch brings along, behind it all that the rest needs, so that loads do not follow one another
  // (16 heads in a step, 8192 tokens 16.8 -> 14.9 us; 1024 tokens 7.1 as before, whose blocks find no room before the wait is over).
  pdl_launch_dependents();
  const int2 tile = tiles[blockIdx.x];
  const int h = blockIdx.y, t0 = tile.x * 128, m = t0 + (int)threadIdx.x;
  const int seq_first = seq_start[t0], my_seq = threadIdx.x < 128 && m < M ? seq_start[m] : 0;
  // the scan of the factors, from the start of the tile's first sequence to the end of its last
  auto scan_at = [&](int i0) { return min(i0 + (int)threadIdx.x, tile.y - 1); };
  int scan_seq = seq_start[scan_at(seq_first)];
  pdl_wait();
  float scan_scale = row_scale[scan_at(seq_first)], my_scale = 0.f, my_lse = 0.f;
  if (threadIdx.x < 128 && m < M) {
    my_scale = row_scale[m];
    my_lse = lse[(size_t)h * M + m];
  }
  uint4 av[UN], bv[UN];
#pragma unroll
  for (int u = 0; u < UN; ++u) {
    const int q = t0 + warp * 16 + u * RPW + grp;
    const size_t at = ((size_t)q * nh + h) * HD + sub * 8;
    av[u] = q < M ? *(const uint4*)(o + at) : make_uint4(0u, 0u, 0u, 0u);
    bv[u] = q < M ? *(const uint4*)(dO + at) : make_uint4(0u, 0u, 0u, 0u);
  }
  if (threadIdx.x < 129) s_max[threadIdx.x] = 0;
  __syncthreads();
  for (int i0 = seq_first; i0 < tile.y; i0 += 256) {
    const int slot = scan_seq < t0 ? 128 : scan_seq - t0;
    const int v = __float_as_int(fmaxf(scan_scale, 0.f));  // (of values >= 0 the bits order as the values do)
    if (i0 + 256 < tile.y) {
      scan_seq = seq_start[scan_at(i0 + 256)];
      scan_scale = row_scale[scan_at(i0 + 256)];
    }
    int same;
    __match_all_sync(0xffffffffu, slot, &same);
    if (same) {
      const int w = __reduce_max_sync(0xffffffffu, v);
      if (lane == 0) atomicMax(&s_max[slot], w);
    } else {
      atomicMax(&s_max[slot], v);
    }
  }
#pragma unroll
  for (int u = 0; u < UN; ++u) {
    const __half2* a2 = (const __half2*)&av[u];
    const __half2* b2 = (const __half2*)&bv[u];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 x = __half22float2(a2[k]), y = __half22float2(b2[k]);
      s += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (sub == 0) s_delta[warp * 16 + u * RPW + grp] = s;
  }
  __syncthreads();
  const size_t pitch = query_pitch(M);
  if (threadIdx.x >= 128 || (size_t)m >= pitch) return;
  float off = -INFINITY, delta = 0.f;
  if (m < M) {
    const int mx = s_max[my_seq < t0 ? 128 : my_seq - t0];
    const float top = mx > 0 ? __int_as_float((mx + 0x007FFFFF) & 0x7F800000) : 1.f;
    const float w = fmaxf(my_scale, 0.f) / top;
    if (h == 0) tops[m] = top;
    // (fused by name: whether the compiler fuses it depends on where the load stands)
    if (w > 0.f) off = fmaf(-my_lse, LOG2E, log2f(w) + P_BOOST_LOG2);
    delta = s_delta[threadIdx.x];
  }
  query_vecs[(size_t)h * pitch + m] = off;
  query_vecs[(size_t)(nh + h) * pitch + m] = -delta * (scale * (DS_BOOST / P_BOOST));
}

template <int HD>
int bwd_tc_impl(rt_ctx* c, const __half* q, const __half* k, const __half* v, const __half* o, const __half* dO,
                const float* row_scale, const float* lse, const AttnBatch& b, int nh, int nkv, float* work, float* dq, float* dk,
                float* dv) {
  const int M = b.M;
  const int2* gap = (const int2*)b.gap;
  using LK = DkvLayout<HD>;
  using LQ = DqLayout<HD>;
  if (!c->raise_smem(attn_bwd_dkdv_tc_kernel<HD>, LK::TOTAL) || !c->raise_smem(attn_bwd_dq_tc_kernel<HD>, LQ::TOTAL)) return 3;
  CUtensorMap tq128, tdo128, tk64, tv64, tk128, tv128, tq64, tdo64;
  if (tensor_map_f16_2d(c, &tq128, q, (uint64_t)M, (uint64_t)nh * HD, 64, 128)) return 3;
  if (tensor_map_f16_2d(c, &tdo128, dO, (uint64_t)M, (uint64_t)nh * HD, 64, 128)) return 3;
  if (tensor_map_f16_2d(c, &tq64, q, (uint64_t)M, (uint64_t)nh * HD, 64, 64)) return 3;
  if (tensor_map_f16_2d(c, &tdo64, dO, (uint64_t)M, (uint64_t)nh * HD, 64, 64)) return 3;
  if (tensor_map_f16_2d(c, &tk128, k, (uint64_t)M, (uint64_t)nkv * HD, 64, 128)) return 3;
  if (tensor_map_f16_2d(c, &tv128, v, (uint64_t)M, (uint64_t)nkv * HD, 64, 128)) return 3;
  if (tensor_map_f16_2d(c, &tk64, k, (uint64_t)M, (uint64_t)nkv * HD, 64, 64)) return 3;
  if (tensor_map_f16_2d(c, &tv64, v, (uint64_t)M, (uint64_t)nkv * HD, 64, 64)) return 3;
  const float scale = 1.0f / sqrtf((float)HD);
  cudaStream_t st = c->stream;
  float *query_vecs = work, *tops = work + 2 * (size_t)nh * query_pitch(M);
  pdl(attn_delta_tc_kernel<HD>, dim3((M + 127) / 128, nh), 256, 0, st)(o, dO, lse, row_scale, b.seq_start, (const int2*)b.tiles_k, M, nh, scale,
                                                                      query_vecs, tops);
  const int group = nh / nkv, hpc = std::min(group, std::max(4, (group + MAX_HEAD_CTAS - 1) / MAX_HEAD_CTAS)), n_ctas = (group + hpc - 1) / hpc, n_tiles = (M + 127) / 128;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)n_ctas;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(nkv * n_ctas) * n_tiles);
  cfg.blockDim = dim3(BWD_THREADS);
  cfg.dynamicSmemBytes = LK::TOTAL;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = n_ctas > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, attn_bwd_dkdv_tc_kernel<HD>, tk128, tv128, tq64, tdo64, (const float*)tops, (const float*)query_vecs,
                         b.seq_start, gap, (const int2*)b.tiles_k, M, nh, nkv, hpc, n_ctas, scale, dk, dv, c->status_dev) != cudaSuccess)
    return 3;
  // dQ reads nothing of dK/dV's: it starts as soon as that kernel's last CTAs have, in passes of every size.
  PdlLaunch dq_launch = pdl(attn_bwd_dq_tc_kernel<HD>, (unsigned)nh * n_tiles, DQ_THREADS, LQ::TOTAL, st);
  dq_launch.programmatic = pdl_any_size();
  if (dq_launch(tq128, tdo128, tk64, tv64, row_scale, lse, query_vecs, b.seq_start, gap, b.tiles_q, M, nh, nkv, scale, dq, c->status_dev) != cudaSuccess)
    return 3;
  RT_COUNT_LAUNCH(3);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace

size_t attn_bwd_work_floats(int M, int nh) { return 2 * (size_t)nh * query_pitch(M) + (size_t)M; }

void attn_plan_tiles(const int* seq_start, int M, int* tiles_q, int* tiles_k) {
  const int n = (M + 127) / 128;
  std::vector<std::pair<int, int>> wq(n), wk(n);  // (minus the loop's length, tile)
  std::vector<int> end(n);
  for (int t = n - 1, e = M, at = M; t >= 0; --t) {
    const int t0 = t * 128, t1 = std::min(M, t0 + 128);
    // e: end of the sequence that holds row t1 - 1; `at` walks down from the row that fixed it
    for (int i = at - 1; i >= t1 - 1; --i)
      if (i + 1 < M && seq_start[i + 1] != seq_start[i]) e = i + 1;
    at = t1 - 1;
    end[t] = e;
    wq[t] = {seq_start[t0] - t1, t};
    wk[t] = {t0 - e, t};
  }
  std::stable_sort(wq.begin(), wq.end(), [](auto& a, auto& b) { return a.first < b.first; });
  std::stable_sort(wk.begin(), wk.end(), [](auto& a, auto& b) { return a.first < b.first; });
  for (int t = 0; t < n; ++t) {
    tiles_q[t] = wq[t].second;
    tiles_k[2 * t] = wk[t].second;
    tiles_k[2 * t + 1] = end[wk[t].second];
  }
}

int launch_attn_fwd_tc(rt_ctx* c, const __half* q, const __half* k, const __half* v, const AttnBatch& b, int nh, int nkv, int hd,
                       __half* o, float* lse) {
  if (b.M <= 0) return 0;
  if (hd == 128) return fwd_tc_impl<128>(c, q, k, v, b, nh, nkv, o, lse);
  if (hd == 64) return fwd_tc_impl<64>(c, q, k, v, b, nh, nkv, o, lse);
  return 1;
}

int launch_attn_bwd_tc(rt_ctx* c, const __half* q, const __half* k, const __half* v, const __half* o, const __half* dO16,
                       const float* row_scale, const float* lse, const AttnBatch& b, int nh, int nkv, int hd, float* work, float* dq,
                       float* dk, float* dv) {
  if (b.M <= 0) return 0;
  if (hd == 128) return bwd_tc_impl<128>(c, q, k, v, o, dO16, row_scale, lse, b, nh, nkv, work, dq, dk, dv);
  if (hd == 64) return bwd_tc_impl<64>(c, q, k, v, o, dO16, row_scale, lse, b, nh, nkv, work, dq, dk, dv);
  return 1;
}

}  // namespace rt
