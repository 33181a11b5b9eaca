// Frozen quantised matmul on tcgen05 tensor cores (sm_100a).
//
//   forward  (reference src/rie.rs:74-82,  RieFrozen::forward)        Y[M x N]  = X[M x K] . W^T
//   backward (reference src/rie.rs:84-120, RieFrozen::backward_input) dX[M x K] = dY[M x N] . W
//
// both read the SAME packed weight bytes (64x64 bricks of ggml codes, see qformat.cuh); no
// dequantised copy of W exists in global memory.  The weight is the UMMA "A" operand (128
// weight rows or columns per CTA, 64 in half tiles and slim pairs), the activations are the "B" operand (up
// to 256 tokens per tile), so the TMEM accumulator is the transposed output tile [rows x tokens].
//
// One persistent CTA per SM, warp-specialised (23 warps, 15 without unpacking; roles by warp id, see the kernel):
//   producer : one thread issues the TMA tiles of activations (and of 16-bit weights), 128B swizzle
//   bricks   : one thread issues the bulk copies of packed bricks, running ahead in its own ring
//   MMA      : one thread issues tcgen05.mma (kind::f16, fp32 accumulate in TMEM)
//   unpack   : sixteen warps turn packed bricks into the f16 tile in the UMMA shared-memory layout
//              (forward reads it K-major, backward reads the same bytes MN-major)
//   epilogue : four warps tcgen05.ld the accumulator (double buffered: 2 x 256 TMEM columns),
//              add bias / per-token factors; 16-bit results are staged and TMA-stored, f32 ones
//              go straight from registers to memory
// The LoRA low-rank term is one more contraction chunk fed through the same accumulator.
#include "pdl.cuh"
#include "ptx.cuh"
#include "qformat.cuh"
#include "ctx.h"

namespace rt {


// The kernel is compiled per launch kind and weight format (one switch on the host instead of one
// per unpacked unit on the device).
enum QKind : int {
  QK_PAIR = 0,    // a CTA pair per tile of 256 weight rows x up to 256 tokens
  QK_WIDE = 1,    // one CTA per tile of 128 weight rows x up to 256 tokens: converted 16-bit weights, and all
                  // formats where CTA pairs cannot run or are switched off
  QK_NARROW = 2,  // one CTA per tile of 128 weight rows x up to 64 tokens
  QK_HALF = 3,    // one CTA per tile of 64 weight rows x up to 64 tokens
  // Narrow tiles of packed weights in the forward direction, with the unpacked weights in TMEM: a thread that owns a
  // weight row is the TMEM lane the MMA reads it from, and the weight tile no longer passes through shared
  // memory twice.  4096x1024 in Q8_0 at 157 tokens 7.0 us, on slim pairs 8.3.  (Backward reads the
  // bricks down their columns: only the shared-memory operand can be read transposed.  Half tiles leave half of the
  // lanes, and so of the unpack warps, without a row.)
  QK_NARROW_T = 4,
  // A CTA pair per tile of 128 weight rows x up to 128 tokens: 64 rows of weights and half of the tokens in each CTA, so that a CTA
  // unpacks, writes and hands to the tensor core half the weights of a narrow tile for the same number of results.
  // What bounds a narrow tile is shared memory: 128 rows written and read, 64 tokens written and read, the codes in and out, by
  // its 128 bytes a cycle 420 cycles for each 64 contraction elements (Q4_0) against 290 here.  6144x1024 Q4_0 backward at 1024
  // tokens, one round of 96 such steps: 25.6 us on narrow tiles, 18.4 on slim pairs.
  QK_SLIM = 5,
};
// How the results leave: a kernel holds the code of one way only (all of them in one kernel cost the small
// launches 0.4 us each in instruction fetches and the f16 epilogue of a pair registers, 5 % of the
// 6144x1024 product at 8192 tokens).
enum QOut : int {
  QO_TMA16 = 0,   // 16-bit, staged in shared memory and stored by TMA
  QO_DIRECT = 1,  // from registers: f32, partial sums, 16-bit that TMA cannot address
  QO_RES = 2,     // f32 with a residual that comes by asynchronous copies (CTA pairs only: in the few blocks of a
                  // smaller tile the pipeline gains nothing)
};
// Weight formats as the kernel sees them: ggml's ids for packed weights, and two 16-bit cases.
constexpr int QF_16 = 0;       // 16-bit weights of the activations' type, straight from TMA
constexpr int QF_16CONV = 1;   // 16-bit weights of the other 16-bit type, converted in place

// Shared-memory plan of one CTA.
template <int KIND, int FMT, int OUT>
struct QCfg {
  static constexpr bool SLIM = KIND == QK_SLIM, PAIR = KIND == QK_PAIR || SLIM, HALF = KIND == QK_HALF, NARROW = KIND == QK_NARROW || KIND == QK_NARROW_T;
  static constexpr bool TM = KIND == QK_NARROW_T;  // unpacked weights in TMEM
  // Weight rows of the CTA's tile, as many as its MMA takes (a slim pair's takes both CTAs').  A half tile whose results are staged
  // takes 128 all the same, because a quarter of the accumulator then has the 32 rows of a staged block: the upper 64 are
  // whatever follows the tile in shared memory, and their lanes are not read.  (Without staging 6144x1024 Q4_0 at 157 tokens to f16 13.8 us, 9.6
  // so; f32 results of 3072x8192 at 157 tokens 25.6 us with 128 rows, 24.5 with 64.)
  static constexpr bool M64 = HALF && OUT == QO_DIRECT;
  static constexpr int ROWS = HALF || SLIM ? 64 : 128, BRICKS = ROWS / 64;
  static constexpr int W_SUB = ROWS * 128;  // bytes of a [ROWS x 64] 16-bit weight tile
  static constexpr bool PACKED = FMT > QF_16CONV;
  static constexpr bool WIDE = KIND == QK_WIDE;
  // Unpack warps.  Sixteen for packed weights: one unpack pass is a chain of dependent operations
  // (codes -> convert -> swizzled store -> fence -> arrive), so what counts is how many passes are
  // in flight per scheduler.  (Eight warps of twice the work each: 8192x3072 Q6_K at 8192 tokens
  // 406 us against 363.)  Without unpacking eight warps stay, to help with the last tile's epilogue.
  static constexpr int NUW = PACKED ? 16 : 8;
  // + activation / brick producers, MMA, 4 epilogue warps, and one idle where four unpack warps of each residue are needed
  static constexpr int THREADS = 32 * (7 + NUW + (TM ? 1 : 0));
  // 64-element contraction steps per stage.  Two for narrow and half tiles and slim pairs: their MMAs are short, and one
  // hand-off between the roles costs about 500 cycles whatever it hands over.
  static constexpr int KS = NARROW || HALF || SLIM ? 2 : 1;
  // Activation / unpacked-weight stages, and packed-brick stages in the room that is left beside them and
  // the epilogue staging.
  static constexpr int NS = PAIR ? (PACKED ? 5 : 6) : WIDE ? 3 : HALF || TM ? 4 : PACKED ? 3 : 4;
  static constexpr int RAW_STAGE = PACKED ? KS * BRICKS * fmt_brick_bytes(FMT) : 0;
  static constexpr int ACT_SUB = KIND == QK_PAIR ? 16384 : WIDE ? 32768 : 8192;  // tokens of the CTA's tile x 64 x 16-bit
  static constexpr int ACT_STAGE = KS * ACT_SUB;
  static constexpr int W_BYTES = (TM ? 1 : KS) * W_SUB;    // weights of a stage (in TMEM: the low-rank step's only)
  // TMEM columns of a stage's unpacked weights, beside the two accumulators of up to 64 columns at 0 and 256
  __device__ static constexpr uint32_t a_col(int st) { return 128u + (uint32_t)(st & 1) * 64u + (uint32_t)(st >> 1) * 256u; }
  static_assert(!TM || (PACKED && NS <= 4), "four stages fit TMEM");
  // Epilogue staging per warp of 16-bit outputs and of residuals: three blocks of [32 tokens x 32 features], 2 KB each.  What leaves
  // straight from registers has none, and its room goes to the brick ring: Q8_0 on pairs and slim pairs has seven slots so, four with
  // it (8192x3072 at 24 tokens backward on slim pairs 29.5 -> 25.5 us, at 157 forward on pairs 21.1 -> 18.4, 3072x8192 at 1024 forward 53.2 -> 49.1).
  static constexpr int OUT_BUFS = 3, OUT_WARP = OUT == QO_DIRECT ? 0 : OUT_BUFS * 2048;
  static constexpr int SMEM_MAX = 232448, SMEM_REST = 4 * OUT_WARP + 512 + 2 * 1024;  // staging, barriers, alignment
  static constexpr int NR_FIT = PACKED ? (SMEM_MAX - SMEM_REST - NS * (ACT_STAGE + W_BYTES)) / (RAW_STAGE ? RAW_STAGE : 1) : 0;
  static constexpr int NR = NR_FIT > 8 ? 8 : NR_FIT;
  // The unpack warps work as UG groups on alternate stages.  Waits are by phase parity,
  // which is only sound while a waiter cannot run two phases ahead of its barrier: UG <= NS keeps a
  // group from reaching a stage before the use two back has been released, and NS <= NR + 1 keeps a
  // group from reaching a brick slot's next use (NR stages later, NR + 1 across a low-rank step,
  // which takes a stage but no bricks) before the MMAs of its previous use are done, so that a copy
  // that lands late cannot be taken for the one after it.
  static constexpr int UG = PAIR ? 4 : 2;                  // a power of two
  static constexpr int UTG = NUW * 32 / UG;                // threads per group
  static_assert(UG <= NS && (!PACKED || (NS <= NR + 1 && UG <= NR)), "unpack groups would alias barrier phases");
  // A thread of a group owns one unit of each half of a weight tile; with a group of twice the threads (wide tiles) of one half.
  static constexpr int HALVES = WIDE ? 1 : BRICKS;
  // A group of fewer threads than that goes over the stage's 64-element tiles one after the other.
  static constexpr int PASSES = KS * 128 * (BRICKS / HALVES) / UTG;
  static_assert(!PACKED || PASSES * UTG == KS * 128 * (BRICKS / HALVES), "the group's threads cover a stage's units");
  static constexpr int OFF_W = NS * ACT_STAGE;
  static constexpr int OFF_RAW = OFF_W + NS * W_BYTES;
  static constexpr int OFF_OUT = (OFF_RAW + NR * RAW_STAGE + 1023) / 1024 * 1024;  // (a swizzled store's source starts on its pattern)
  static constexpr int OFF_BAR = OFF_OUT + 4 * OUT_WARP;
  static constexpr int N_BARS = 3 * NS + 2 * NR + 5;
  // At least so much that no other kernel with TMEM fits beside it: it lets the next one start before it holds its columns (pdl.cuh).
  static constexpr int SMEM_USED = OFF_BAR + N_BARS * 8 + 16 + 1024;
  static constexpr int SMEM_BYTES = SMEM_USED > ALONE_SMEM ? SMEM_USED : ALONE_SMEM;
  static_assert(SMEM_BYTES <= SMEM_MAX && N_BARS * 8 + 16 <= 512, "shared memory plan exceeds one SM");
  static_assert(OUT == QO_DIRECT || OFF_RAW >= 11 * 8192, "the last tile's helpers stage in the operand stages");
};

struct KParams {
  const uint8_t* bricks;
  int nb, nbk;   // bricks along the output rows of this direction, bricks per brick row
  int act_f16;   // activations (and therefore the unpacked weight tile) are f16, else bf16
  int conv16;    // QF_16CONV only: 1 = f16 -> bf16, 2 = bf16 -> f16
  int dir, out_rows, M, TN;
  int n_main, lora_mmas;
  int n_splits, steps_per_split;  // work item = (tile, piece of the contraction); partial results go to `part`
  float* part;                    // [n_splits][M][out_rows] f32 partials when n_splits > 1
  int n_row_tiles, n_tok_tiles;   // a row tile is 128 weight rows, 256 for a pair, 64 for a half tile
  int tok_first;                  // a row tile's token tiles are neighbours, instead of a token tile's row tiles
  int inner;                      // tiles of a run of neighbours
  void* out;
  int out_dtype, accumulate, ld_out;
  const float* row_scale;  // optional per-token factor applied to the result
  const float* residual;   // optional f32 matrix laid out as `out` that the result is added to
  const float* bias;
  uint32_t idesc;
  int* status;
  int late_wait, end_wait;  // see QGemmArgs
};

// ------------------------------------------------------------------ unpackers
// One thread turns one unit (32 codes of one brick row) into 64 bytes of the 16-bit weight tile:
// four 16-byte chunks at tile_base + off[j].  The swizzled offsets depend on the thread only and
// are computed once per kernel.
//
// Codes become f16 through the magic number 0x6400 (1024 + code in the mantissa).  The integer
// pipe has half the rate of the f16 one and was the unpackers' limit (ncu: 57 % of its peak over
// all four schedulers, 76 % on the three that had unpack warps), so a 4-bit field is extracted
// where it stands: field 0 as 1024 + v, field 1 as 1024 + 16 v, which one exact fma scales back,
// and a single shift by 8 brings fields 2 and 3 into their places.
struct UnitDst {
  uint32_t off[4];
  __device__ __forceinline__ explicit UnitDst(int t) {
    const int r = t >> 1, cb = (t & 1) * 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) off[j] = (uint32_t)(r * 128 + (((cb + j) ^ (r & 7)) << 4));
  }
};
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
template <bool WBF16>
__device__ __forceinline__ uint32_t fin(__half2 h) {
  if (WBF16) {
    __nv_bfloat162 b = __float22bfloat162_rn(__half22float2(h));
    return *(uint32_t*)&b;
  }
  return *(uint32_t*)&h;
}
__device__ __forceinline__ __half2 u32_as_h2(uint32_t x) { return *(__half2*)&x; }
__device__ __forceinline__ __half2 h2c(float x) { return __floats2half2_rn(x, x); }
// pair p (0..3) of a word of eight 4-bit fields, OR-ed with `more` (bits 4-5 of an even pair's halves, 8-9 of
// an odd pair's), minus `bias`: exact for codes below 64
__device__ __forceinline__ __half2 code_pair(uint32_t w, uint32_t w8, int p, uint32_t more, float bias) {
  const uint32_t src = p < 2 ? w : w8;
  if (p & 1) return __hfma2(u32_as_h2((src & 0x00F000F0u) | 0x64006400u | more), h2c(0.0625f), h2c(-64.f - bias));
  return __hsub2(u32_as_h2((src & 0x000F000Fu) | 0x64006400u | more), h2c(1024.f + bias));
}

// REGS: the unit's sixteen registers are left in `regs` instead of being stored
template <int FMT, bool WBF16, bool REGS>
__device__ __forceinline__ void unpack_unit(const uint8_t* brick, int t, uint32_t tile, const UnitDst& ud, uint32_t* regs) {
  auto put = [&](int j, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    if (REGS) { regs[4 * j] = a; regs[4 * j + 1] = b; regs[4 * j + 2] = c; regs[4 * j + 3] = d; }
    else st_shared_v4(tile + ud.off[j], a, b, c, d);
  };
  if (FMT == GGML_Q4_0) {
    const uint4 q = *(const uint4*)(brick + t * 16);
    const __half2 d2 = __half2half2(((const __half*)(brick + 2048))[t]);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w8 = w[j] >> 8;
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) o[p] = fin<WBF16>(__hmul2(code_pair(w[j], w8, p, 0u, 8.f), d2));
      put(j, o[0], o[1], o[2], o[3]);
    }
  } else if (FMT == GGML_Q8_0) {
    const uint4 qa = *(const uint4*)(brick + t * 16);
    const uint4 qb = *(const uint4*)(brick + 2048 + t * 16);
    const __half2 d2 = __half2half2(((const __half*)(brick + 4096))[t]);
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const uint32_t x = __byte_perm(w[2 * j + (p >> 1)], 0x64646464u, (p & 1) ? 0x4342 : 0x4140);
        o[p] = fin<WBF16>(__hmul2(__hsub2(u32_as_h2(x), h2c(1152.f)), d2));  // 1024 (magic) + 128 (stored offset)
      }
      put(j, o[0], o[1], o[2], o[3]);
    }
  } else if (FMT == GGML_Q4_K) {
    const uint4 q = *(const uint4*)(brick + t * 16);
    const float2 ddf = __half22float2(((const __half2*)(brick + 2048))[t >> 1]);
    const uchar2 sm = ((const uchar2*)(brick + 2304))[t];
    // value = (d*sc)*q - dmin*m is a difference of like-sized terms: each factor is carried as an
    // f16 pair (hi + lo) so the only rounding that matters is the final one, relative to the value
    const float dscf = ddf.x * (float)sm.x, ndmf = -ddf.y * (float)sm.y;
    const __half dsc_h = __float2half_rn(dscf), ndm_h = __float2half_rn(ndmf);
    const __half2 dsc = __half2half2(dsc_h), ndm = __half2half2(ndm_h);
    const __half2 dsc_lo = __half2half2(__float2half_rn(dscf - __half2float(dsc_h)));
    const __half2 ndm_lo = __half2half2(__float2half_rn(ndmf - __half2float(ndm_h)));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w8 = w[j] >> 8;
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const __half2 qv = code_pair(w[j], w8, p, 0u, 0.f);
        o[p] = fin<WBF16>(__hadd2(__hfma2(qv, dsc, ndm), __hfma2(qv, dsc_lo, ndm_lo)));
      }
      put(j, o[0], o[1], o[2], o[3]);
    }
  } else if (FMT == GGML_Q6_K) {
    const uint4 lo = *(const uint4*)(brick + t * 16);
    const uint2 hi = *(const uint2*)(brick + 2048 + t * 8);
    const char2 sc = ((const char2*)(brick + 3072))[t];
    const float d = __half2float(((const __half*)(brick + 3328))[t >> 1]);
    const __half2 ds0 = __half2half2(__float2half_rn(d * (float)sc.x));
    const __half2 ds1 = __half2half2(__float2half_rn(d * (float)sc.y));
    const uint32_t w[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t h = j < 2 ? hi.x : hi.y, w8 = w[j] >> 8;
      const __half2 ds = j < 2 ? ds0 : ds1;
      // pairs 0, 1 | 2, 3 of an even word under rotations 0 | 8, of an odd word under 2 | 10 (q6k_hi_pos)
      const uint32_t h01 = (j & 1) ? __funnelshift_r(h, h, 2) : h;
      const uint32_t h23 = __funnelshift_r(h, h, (j & 1) ? 10 : 8);
      uint32_t o[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const uint32_t more = (p < 2 ? h01 : h23) & ((p & 1) ? 0x03000300u : 0x00300030u);
        o[p] = fin<WBF16>(__hmul2(code_pair(w[j], w8, p, more, 32.f), ds));
      }
      put(j, o[0], o[1], o[2], o[3]);
    }
  }
}

// ------------------------------------------------------------------ kernel
// PAIR: a cluster of two CTAs shares a tile of 256 weight rows x TN tokens.  Each CTA holds its own
//   128 weight rows (unpacked by its own warps) and HALF of the token tile; the leader CTA (cluster
//   rank 0) issues tcgen05.mma.cta_group::2, which reads both CTAs' shared memory and writes 128
//   accumulator rows into each CTA's TMEM.  Per CTA and per MMA cycle this halves the activation
//   bytes that TMA writes and the tensor core reads.  Barriers that gate the MMA (full, acc_empty)
//   live in the leader and are arrived on from both CTAs; barriers the MMA releases (stage_empty,
//   acc_full) exist in both CTAs and are signalled by one multicast commit.
// SLIM: a pair that shares a tile of 128 weight rows: each CTA holds 64 of them and half of the tokens, and the MMA (M = 128
//   over the pair) writes, in each CTA's TMEM, its 64 rows to lanes 0..63 for the first half of the tokens and to lanes 64..127
//   for the second, in half as many columns.  All the rest is as for PAIR, which is set for both.
template <int KIND, int FMT, int OUT>
__global__ void __launch_bounds__((QCfg<KIND, FMT, OUT>::THREADS), 1)
qgemm_kernel(const __grid_constant__ CUtensorMap tm_act, const __grid_constant__ CUtensorMap tm_w16,
             const __grid_constant__ CUtensorMap tm_lact, const __grid_constant__ CUtensorMap tm_lw,
             const __grid_constant__ CUtensorMap tm_out, const KParams p) {
  using C = QCfg<KIND, FMT, OUT>;
  constexpr bool PAIR = C::PAIR, SLIM = C::SLIM, TM = C::TM, PACKED = C::PACKED, CONV = FMT == QF_16CONV, IS16 = !PACKED;
  constexpr int NS = C::NS, NR = C::NR, UG = C::UG, UTG = C::UTG, KS = C::KS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sAct = smem;
  uint8_t* sW = smem + C::OFF_W;
  uint8_t* sRaw = smem + C::OFF_RAW;
  uint8_t* sOut = smem + C::OFF_OUT;
  uint64_t* bars = (uint64_t*)(smem + C::OFF_BAR);
  uint64_t* full = bars;                   // [NS] activations (+ weight tile) in place           (leader's is used)
  uint64_t* w_ready = bars + NS;           // [NS] in-place conversion done (QF_16CONV)
  uint64_t* stage_empty = bars + 2 * NS;   // [NS] MMAs reading the stage have completed          (every CTA)
  uint64_t* raw_full = bars + 3 * NS;      // [NR]                                                (every CTA)
  uint64_t* raw_empty = raw_full + NR;     // [NR]
  uint64_t* acc_full = raw_empty + NR;     // [2]                                                 (every CTA)
  uint64_t* acc_empty = acc_full + 2;      // [2]                                                 (leader's is used)
  uint64_t* last_full = acc_empty + 2;     // the last tile's accumulator is complete: what its helpers wait for (they
                                           // have not followed acc_full's phases)                (every CTA)
  uint32_t* tmem_slot = (uint32_t*)(bars + C::N_BARS);
  pdl_launch_dependents();

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // Roles by warp.  A warp runs on scheduler (warp % 4).  The MMA-issuing thread's instruction
  // latency sets the pace of the whole pipeline (every tcgen05.mma and commit goes through it), so
  // its scheduler (1) hosts fewer unpack warps than the others; the epilogue needs one warp per
  // residue (a warp reads TMEM lanes 32 * (warp % 4) ..).
  //   warp 1 MMA | 5 activation producer | 9 packed-brick producer | 0, 2, 3, 13 epilogue | rest unpack
  constexpr int R_PROD = 0, R_MMA = 1, R_UNPACK = 2, R_EPI = 3, R_RAW = 4;
  // A warp writes TMEM lanes by its residue too, so unpacking into TMEM takes four warps of each:
  //   warp 1 MMA | 23 activation producer | 22 brick producer | 0, 2, 3, 13 epilogue | 20 idle | rest unpack
  constexpr int R_IDLE = 5;
  int role = R_UNPACK, uidx = 0;  // uidx: position among the unpack warps, neighbours on different schedulers
  if (TM) switch (warp) {
    case 1: role = R_MMA; break;
    case 23: role = R_PROD; break;
    case 22: role = R_RAW; break;
    case 0: case 2: case 3: case 13: role = R_EPI; break;
    case 20: role = R_IDLE; break;
    default: uidx = (warp >> 2) - 1 - ((warp & 3) == 1 && warp > 13 ? 1 : 0); break;  // 0..3 within the residue
  }
  else switch (warp) {
    case 1: role = R_MMA; break;
    case 5: role = R_PROD; break;
    case 9: role = R_RAW; break;
    case 0: case 2: case 3: case 13: role = R_EPI; break;
    case 4: uidx = 0; break;
    case 6: uidx = 1; break;
    case 7: uidx = 2; break;
    case 8: uidx = 3; break;
    case 10: uidx = 4; break;
    case 11: uidx = 5; break;
    case 12: uidx = 6; break;
    case 14: uidx = 7; break;
    default: uidx = warp - 7; break;  // warps 15..22
  }
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;  // 0 = leader
  constexpr int n_cta = PAIR ? 2 : 1;
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int tn_cta = PAIR ? p.TN >> 1 : p.TN;  // token rows of the tile this CTA loads
  const int n_tiles = p.n_row_tiles * p.n_tok_tiles;
  const int n_items = n_tiles * p.n_splits;
// work item -> tile, its range of contraction steps, and whether the LoRA chunk is appended
#define QG_ITEM_DECODE(item)                                                                  \
  const int tile = (item) % n_tiles, split = (item) / n_tiles;                                \
  const int s_begin = split * p.steps_per_split;                                              \
  const int s_main = min(p.n_main, s_begin + p.steps_per_split) - s_begin;                    \
  const int n_main_st = (s_main + KS - 1) / KS;  /* stages of the weight's own contraction */  \
  const int n_steps = n_main_st + ((p.lora_mmas > 0 && split == p.n_splits - 1) ? 1 : 0);     \
  (void)split; (void)n_main_st
// first weight row (output feature) of this CTA's half of the tile, first token of the tile
#define QG_TILE_ORIGIN()                                                                      \
  const int t_in = tile % p.inner, t_out = tile / p.inner;                                     \
  const int r0 = (PAIR && p.tok_first ? t_out : t_in) * (C::ROWS * n_cta) + (int)rank * C::ROWS;   \
  const int m0 = (PAIR && p.tok_first ? t_in : t_out) * p.TN

  if (threadIdx.x == 0) {
    for (int i = 0; i < NS; ++i) {
      // One barrier gates a step's MMAs: the producer's expect-tx arrival (with the bytes TMA brings)
      // plus, for packed weights, one arrival per warp of the unpack group that owns the step, from
      // every CTA of the pair.  Only the in-place 16-bit conversion needs the landing and the
      // conversion told apart: then the warps wait on `full` themselves and report on `w_ready`.
      mbar_init(&full[i], PACKED ? 1 + (UTG / 32) * n_cta : 1);
      mbar_init(&w_ready[i], UTG / 32);
      mbar_init(&stage_empty[i], 1);
    }
    for (int i = 0; i < NR; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], UTG / 32); }  // per warp
    for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4 * n_cta); }  // per epilogue warp
    mbar_init(last_full, 1);
    mbar_fence_init();
    prefetch_tmap(&tm_act);
    if (IS16) prefetch_tmap(&tm_w16);
    if (p.lora_mmas > 0) { prefetch_tmap(&tm_lact); prefetch_tmap(&tm_lw); }
    if (OUT == QO_TMA16) prefetch_tmap(&tm_out);
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(tmem_slot, 512); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  }
  if (warp == 2 && (p.late_wait || p.end_wait) && (p.row_scale || (p.residual && OUT != QO_RES))) pdl_unwaited();
  tc_fence_before();
  __syncwarp();
  if (PAIR) cluster_sync_all();  // both CTAs' barriers are initialised and both hold their TMEM columns
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  // barriers, TMEM and descriptors are set up; from here on the kernel reads what its predecessor wrote.  Packed weights
  // no kernel of a pass writes: their bricks are fetched and unpacked under the predecessor's end.
  const bool weights_only = PACKED && (role == R_RAW || role == R_UNPACK);
  if (!p.late_wait && !p.end_wait && !weights_only) pdl_wait();

  // Where the 32 accumulator lanes of quarter wq belong.  A slim pair's accumulator has 64 rows in each CTA: lanes 0..63 hold
  // them for the tile's first half of the tokens, lanes 64..127 for the second, in half as many columns.
  const int tn_q = SLIM ? p.TN >> 1 : p.TN;  // tokens (columns) of a quarter
  // An accumulator of 64 rows in one CTA has them in the first sixteen lanes of each quarter.
  auto q_row = [&](int wq) { return SLIM ? (wq & 1) * 32 : C::M64 ? wq * 16 : wq * 32; };
  auto q_tok = [&](int wq) { return SLIM ? (wq >> 1) * tn_q : 0; };

  // One [32 tokens x 32 features] block of a 16-bit output -> staging -> TMA store.  `stage_base` is
  // private to the calling warp; a block of it is reused only after the store that read it is done.
  auto tma_chunk = [&](int acc, int wq, int c, int r0, int m0, uint8_t* stage_base, uint32_t& cnt) {
    const int buf = (int)(cnt % C::OUT_BUFS);
    ++cnt;
    uint8_t* stage = stage_base + buf * 2048;
    const uint32_t tcol = tmem_base + acc * 256 + ((uint32_t)(wq * 32) << 16) + c * 32;
    // The accumulator block arrives in mma-fragment layout (a thread holds two neighbouring tokens
    // of one feature), is rounded to pairs and written with transposing matrix stores into a
    // [32 tokens][32 features] block of 64-byte rows, 16-byte units XOR-swizzled by (token / 2) % 4
    // as the output map's 64-byte swizzle expects.
    uint32_t v[2][16];
    tmem_ld_16x256b_x4(tcol, v[0]);
    tmem_ld_16x256b_x4(tcol + (16u << 16), v[1]);
    float2 rs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int tok = m0 + q_tok(wq) + c * 32 + 8 * k + 2 * (lane & 3);
      rs[k] = make_float2(1.f, 1.f);
      if (p.row_scale) {
        rs[k].x = tok < p.M ? p.row_scale[tok] : 0.f;
        rs[k].y = tok + 1 < p.M ? p.row_scale[tok + 1] : 0.f;
      }
    }
    float bv[4] = {0.f, 0.f, 0.f, 0.f};  // features 16h + lane/4 + 8e -> bv[2h + e]
    if (p.bias) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = r0 + q_row(wq) + 8 * e + (lane >> 2);
        bv[e] = row < p.out_rows ? p.bias[row] : 0.f;
      }
    }
    if (lane == 0) bulk_wait_group_read<C::OUT_BUFS - 1>();
    tmem_ld_wait();
    __syncwarp();
    // matrix mi = lane / 8 of a store: tokens 8(2kp + mi/2).., feature unit 2h + (mi & 1); this lane addresses row lane % 8
    const uint32_t sbase = smem_u32(stage);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int kp = 0; kp < 2; ++kp) {
        uint32_t pk[4];  // tokens 16kp + 8(i / 2).., features 16h + 8(i & 1)..
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int k = 2 * kp + (i >> 1), e = i & 1;
          const float lo = __uint_as_float(v[h][4 * k + 2 * e]) * rs[k].x + bv[2 * h + e];
          const float hi = __uint_as_float(v[h][4 * k + 2 * e + 1]) * rs[k].y + bv[2 * h + e];
          if (p.out_dtype == OUT_BF16) { __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi); pk[i] = *(uint32_t*)&b; }
          else { __half2 b = __floats2half2_rn(lo, hi); pk[i] = *(uint32_t*)&b; }
        }
        const int mi = lane >> 3;
        const int tok = 8 * (2 * kp + (mi >> 1)) + (lane & 7);
        const int unit = 2 * h + (mi & 1);
        stmatrix_x4_trans(sbase + tok * 64 + ((unit ^ ((tok >> 1) & 3)) << 4), pk[0], pk[1], pk[2], pk[3]);
      }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(&tm_out, r0 + q_row(wq), m0 + q_tok(wq) + c * 32, stage);
      bulk_commit_group();
    }
  };
  // The same block straight from registers to memory (lane = output feature, register j = token): f32
  // results, partial sums, and 16-bit outputs TMA cannot address.  A warp writes 128 contiguous
  // bytes per token, of a half tile's 64 rows 64.  (f32 blocks used to go through two 4 KB staging buffers and TMA: the store of
  // the block before last had to be read out first, and the 4096x1024 product at 8192 tokens
  // waited for its epilogue, 73 us; its stores knocked out it ran in 61.)
  // The epilogue warps share their schedulers with the unpack warps, so what counts is the number of
  // instructions per value: whole blocks take straight-line code without a test per value (with one,
  // the same product took 135 us).
  // A residual is added before anything is stored, eight loads in flight, in whole and ragged blocks alike: a load behind a store
  // that it might alias waits for it, in a last block of 1 to 31 tokens a chain of as many round trips to L2.  Value by value there
  // scoring 157 tokens took 1780 us instead of 1724, accumulating over ragged batches 32.7 ms instead of 31.4, and, with a test per value
  // for whether there is a residual, 24 tokens through a frozen [8192 x 3072] 47.4 us instead of 45.9 (one call after the other, with their host work).
  // A loop of their own for whole blocks: 4 x 256 tokens 7.11 ms against 7.07-7.16; four values at a time, or all 32 left to the compiler, 7.20 and 7.16.
  auto direct_chunk = [&](int acc, int wq, int c, int r0, int m0, int split) {
    const int tok0 = m0 + q_tok(wq) + c * 32, row = r0 + q_row(wq) + lane;
    if (tok0 >= p.M) return;
    uint32_t v[32];
    tmem_ld32(tmem_base + acc * 256 + ((uint32_t)(wq * 32) << 16) + c * 32, v);
    const bool row_ok = row < p.out_rows && (!C::M64 || lane < 16);
    const int nvalid = min(min(32, tn_q - c * 32), p.M - tok0);
    const bool fin_out = p.part == nullptr;  // partial sums are scaled, biased and added up by the reduce kernel
    float rs_lane = 1.0f;
    if (fin_out && p.row_scale) rs_lane = lane < nvalid ? p.row_scale[tok0 + lane] : 0.f;
    const float bias_v = (fin_out && p.bias != nullptr && row_ok) ? p.bias[row] : 0.f;
    tmem_ld_wait();
    if (fin_out && p.row_scale) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j));
    }
    if (!row_ok) return;
    const size_t ld = fin_out ? (size_t)p.ld_out : (size_t)p.out_rows;
    const size_t base = fin_out ? (size_t)tok0 * ld + row : ((size_t)split * p.M + tok0) * ld + row;
    float* o = (fin_out ? (float*)p.out : p.part) + base;
    if (!fin_out || p.out_dtype == OUT_F32) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + bias_v);
      if (fin_out && p.residual) {
        const float* res = p.residual + base;
#pragma unroll
        for (int q = 0; q < 32; q += 8) {  // what the registers have room for
          float old[8];
#pragma unroll
          for (int j = 0; j < 8; ++j, res += ld) old[j] = q + j < nvalid ? *res : 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) v[q + j] = __float_as_uint(__uint_as_float(v[q + j]) + old[j]);
        }
      }
      if (nvalid == 32) {
        if (fin_out && p.accumulate) {  // each element receives exactly one addition per launch
#pragma unroll
          for (int j = 0; j < 32; ++j, o += ld) atomicAdd(o, __uint_as_float(v[j]));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j, o += ld) *o = __uint_as_float(v[j]);
        }
        return;
      }
      const bool add = fin_out && p.accumulate;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < nvalid) {
          if (add) atomicAdd(o + (size_t)j * ld, __uint_as_float(v[j]));
          else o[(size_t)j * ld] = __uint_as_float(v[j]);
        }
      return;
    }
    // 16-bit outputs TMA cannot address
    __half* o16 = (__half*)p.out + base;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < nvalid) {
        const float val = __uint_as_float(v[j]) + bias_v;
        if (p.out_dtype == OUT_BF16) ((__nv_bfloat16*)o16)[(size_t)j * ld] = __float2bfloat16_rn(val);
        else o16[(size_t)j * ld] = __float2half_rn(val);
      }
  };
  // A tile's f32 result with a residual added: the residual's blocks come as asynchronous copies of [16 tokens x
  // 32 features] into the warp's three staging buffers, three ahead of their use.  (Loaded by the thread
  // that adds, eight values at a time, their latency made the epilogue longer than the next tile's contraction:
  // 1024x2048 at 8192 tokens 55.6 us against 32.8 without a residual, 37.3 so.)
  auto res_issue = [&](int k, int wq, int turn, int turns, int r0, int m0, uint32_t stage) {  // the k-th half block of this warp
    const int c = turn + (k >> 1) * turns, col = r0 + wq * 32 + (lane & 7) * 4;
    if (c < p.TN / 32 && col < p.out_rows) {
      const int tok = m0 + c * 32 + (k & 1) * 16 + (lane >> 3);
      const float* src = p.residual + (size_t)tok * p.ld_out + col;
      const uint32_t dst = stage + (uint32_t)(k % 3) * 2048u + (uint32_t)lane * 16u;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (tok + i * 4 < p.M) cp_async_16(dst + i * 512, src + (size_t)(i * 4) * p.ld_out);
    }
    cp_async_commit();
  };
  auto residual_start = [&](int wq, int turn, int turns, int r0, int m0, uint32_t stage) {
#pragma unroll
    for (int k = 0; k < 3; ++k) res_issue(k, wq, turn, turns, r0, m0, stage);
  };
  auto residual_tile = [&](int acc, int wq, int turn, int turns, int r0, int m0, uint32_t stage) {
    const int row = r0 + wq * 32 + lane;
    const bool row_ok = row < p.out_rows;
    const float bias_v = (p.bias != nullptr && row_ok) ? p.bias[row] : 0.f;
    int k = 0;
    for (int c = turn; c < p.TN / 32; c += turns) {
      const int tok0 = m0 + c * 32, nvalid = min(32, p.M - tok0);
      uint32_t v[32];
      tmem_ld32(tmem_base + acc * 256 + ((uint32_t)(wq * 32) << 16) + c * 32, v);
      const float rs_lane = p.row_scale && lane < nvalid ? p.row_scale[tok0 + lane] : 1.f;
      tmem_ld_wait();
      if (p.row_scale) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * __shfl_sync(0xffffffffu, rs_lane, j));
      }
      float* o = (float*)p.out + (size_t)tok0 * p.ld_out + row;
#pragma unroll
      for (int h = 0; h < 2; ++h, ++k) {
        cp_async_wait<2>();
        __syncwarp();
        const uint32_t buf = stage + (uint32_t)(k % 3) * 2048u + (uint32_t)lane * 4u;
#pragma unroll
        for (int q = 0; q < 16; q += 8) {
          float old[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) old[j] = ld_shared_f32(buf + (q + j) * 128);
          if (!row_ok) continue;
#pragma unroll
          for (int j = 0; j < 8; ++j, o += p.ld_out)
            if (nvalid == 32 || h * 16 + q + j < nvalid) *o = __uint_as_float(v[h * 16 + q + j]) + bias_v + old[j];
        }
        __syncwarp();
        res_issue(k + 3, wq, turn, turns, r0, m0, stage);
      }
    }
    cp_async_wait<0>();
  };
  const int n_my = worker < n_items ? (n_items - worker + n_workers - 1) / n_workers : 0;
  uint32_t out_chunk = 0;  // of an epilogue warp, staged so far

  if (role == R_PROD) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      int st = 0;        // stage ring position and its phase
      uint32_t ph = 0;
      bool ok = true;
      for (int item = worker; item < n_items && ok; item += n_workers) {
        QG_ITEM_DECODE(item);
        QG_TILE_ORIGIN();
        const int m_cta = m0 + (int)rank * tn_cta;  // this CTA's half of the tokens
        for (int si = 0; si < n_steps; ++si) {
          if (!mbar_wait(&stage_empty[st], ph ^ 1, p.status, 101)) { ok = false; break; }
          const bool lora = si >= n_main_st;
          const int subs = KS == 1 || lora ? 1 : min(KS, s_main - si * KS);
          uint8_t* a_dst = sAct + st * C::ACT_STAGE;
          uint8_t* w_dst = sW + st * C::W_BYTES;
          // the leader's barrier counts the bytes both CTAs will bring
          if (rank == 0)
            mbar_expect_tx(&full[st], (uint32_t)subs * ((uint32_t)p.TN * 128u + ((IS16 || lora) ? (uint32_t)(C::W_SUB * n_cta) : 0u)));
          const uint32_t fbar = PAIR ? mapa_u32(smem_u32(&full[st]), 0) : 0u;
          auto load2d = [&](void* dst, const CUtensorMap* map, int x, int y) {
            if (PAIR) tma_load_2d_pair(dst, map, x, y, fbar);
            else tma_load_2d(dst, map, x, y, &full[st]);
          };
          if (!lora) {
#pragma unroll
            for (int u = 0; u < KS; ++u) {
              if (u >= subs) break;
              const int s = s_begin + si * KS + u;
              load2d(a_dst + u * C::ACT_SUB, &tm_act, s * 64, m_cta);
              if (IS16) {
#pragma unroll
                for (int b = 0; b < C::BRICKS; ++b) {
                  uint8_t* w = w_dst + u * C::W_SUB + b * 8192;
                  if (p.dir == QG_FWD) load2d(w, &tm_w16, s * 64, r0 + b * 64);
                  else load2d(w, &tm_w16, r0 + b * 64, s * 64);
                }
              }
            }
          } else {
            if (p.late_wait) pdl_wait();
            load2d(a_dst, &tm_lact, 0, m_cta);
#pragma unroll
            for (int b = 0; b < C::BRICKS; ++b) {
              if (p.dir == QG_FWD) load2d(w_dst + b * 8192, &tm_lw, 0, r0 + b * 64);
              else load2d(w_dst + b * 8192, &tm_lw, r0 + b * 64, 0);
            }
          }
          if (++st == NS) { st = 0; ph ^= 1; }
        }
      }
    }
  } else if (role == R_MMA) {
    // ------------------------------------------------------------ MMA issue (the leader's thread only)
    if (rank == 0 && elect_one()) {
      uint32_t tcount = 0;
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      // Descriptors: the high words are fixed for the launch, the low words are address >> 4 plus
      // the leading-dimension field; a stage or a K step of 16 only adds a constant to them.
      const uint64_t a_d0 = (p.dir == QG_FWD) ? umma_desc_sw128(smem_u32(sW), 16, 1024) : umma_desc_sw128(smem_u32(sW), 8192, 1024);
      const uint64_t b_d0 = umma_desc_sw128(smem_u32(sAct), 16, 1024);
      const uint32_t a_hi = (uint32_t)(a_d0 >> 32), b_hi = (uint32_t)(b_d0 >> 32);
      const uint32_t a_k = (p.dir == QG_FWD) ? (32u >> 4) : (2048u >> 4);  // low-word step per K = 16
      constexpr uint32_t b_k = 32u >> 4;
      const uint32_t idesc = p.idesc;
      for (int item = worker; item < n_items && ok; item += n_workers, ++tcount) {
        QG_ITEM_DECODE(item);
        (void)tile; (void)s_begin;
        const int acc = tcount & 1;
        const uint32_t aph = (tcount >> 1) & 1;
        if (!mbar_wait(&acc_empty[acc], aph ^ 1, p.status, 301)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        auto step_ready = [&]() {
          if (!mbar_wait(&full[st], ph, p.status, 302)) return false;
          if (CONV && !mbar_wait(&w_ready[st], ph, p.status, 303)) return false;
          tc_fence_after();
          return true;
        };
        auto step_done = [&]() {
          if (PAIR) umma_commit_pair(&stage_empty[st], 3);
          else umma_commit(&stage_empty[st]);
          const bool wrap = st == NS - 1;
          st = wrap ? 0 : st + 1;
          ph ^= (uint32_t)wrap;
        };
#pragma unroll 1
        for (int s = 0; s < n_main_st; ++s) {
          if (!step_ready()) { ok = false; break; }
          const uint32_t a_lo = (uint32_t)a_d0 + (uint32_t)st * (C::W_BYTES >> 4);
          const uint32_t b_lo = (uint32_t)b_d0 + (uint32_t)st * (C::ACT_STAGE >> 4);
#pragma unroll
          for (int u = 0; u < KS; ++u) {
            if (u > 0 && s * KS + u >= s_main) break;
            const uint32_t au = a_lo + u * (C::W_SUB >> 4), bu = b_lo + u * (C::ACT_SUB >> 4);
            if (TM) {
              const uint32_t at = tmem_base + C::a_col(st) + u * 32;
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                umma_f16_ta(d_tmem, at + kk * 8, ((uint64_t)b_hi << 32) | (bu + kk * b_k), idesc, (uint32_t)((u | s | kk) != 0));
              continue;
            }
            umma_f16_split<PAIR>(d_tmem, au, a_hi, bu, b_hi, idesc, (uint32_t)(u != 0 || s != 0));
            umma_f16_split<PAIR>(d_tmem, au + a_k, a_hi, bu + b_k, b_hi, idesc, 1u);
            umma_f16_split<PAIR>(d_tmem, au + 2 * a_k, a_hi, bu + 2 * b_k, b_hi, idesc, 1u);
            umma_f16_split<PAIR>(d_tmem, au + 3 * a_k, a_hi, bu + 3 * b_k, b_hi, idesc, 1u);
          }
          step_done();
        }
        if (ok && n_steps > n_main_st) {
          if (!step_ready()) { ok = false; break; }
          const uint32_t a_lo = (uint32_t)a_d0 + (uint32_t)st * (C::W_BYTES >> 4);
          const uint32_t b_lo = (uint32_t)b_d0 + (uint32_t)st * (C::ACT_STAGE >> 4);
#pragma unroll 1
          for (int kk = 0; kk < p.lora_mmas; ++kk)
            umma_f16_split<PAIR>(d_tmem, a_lo + kk * a_k, a_hi, b_lo + kk * b_k, b_hi, idesc, (uint32_t)((s_main | kk) != 0));
          step_done();
        }
        if (ok) {
          if (PAIR) umma_commit_pair(&acc_full[acc], 3);
          else umma_commit(&acc_full[acc]);
          if (item + n_workers >= n_items) {
            if (PAIR) umma_commit_pair(last_full, 3);
            else umma_commit(last_full);
          }
        }
      }
    }
  } else if (role == R_UNPACK) {
    // ------------------------------------------------------------ unpack
    // One pass over a weight tile (load codes, convert, store, fence, arrive) is a chain of
    // dependent shared-memory operations: its latency, not its instruction count, sets the pace.
    // The warps therefore work as UG groups on alternate contraction steps, so UG passes are in
    // flight at a time.
    if (PACKED || CONV) {
      const int t = uidx * 32 + lane;
      const int grp = TM ? uidx >> 1 : t / UTG, tg = TM ? 0 : t % UTG;
      const UnitDst ud(tg & 127);
      const uint32_t w_base = smem_u32(sW);
      constexpr int BB = PACKED ? C::RAW_STAGE / (C::BRICKS * KS) : 0;  // bytes of a brick
      // A group goes straight from one of its steps to the next, UG further on in the rings: counting through the other
      // groups' steps took a third of its time (6144x1024 Q4_0 backward at 1024 tokens on narrow tiles 31 -> 26 us).
      int st = grp, rs = grp, s = grp;  // ring positions of the group's step, and its number within the item
      uint32_t ph = 0, rph = 0;
      bool ok = true;
      for (int item = worker; item < n_items && ok; item += n_workers) {
        QG_ITEM_DECODE(item);
        (void)tile; (void)s_begin;
        for (; s < n_steps; s += UG) {
          const bool main_step = s < n_main_st;
          const int subs = KS == 1 ? 1 : min(KS, s_main - s * KS);
          if (!mbar_wait(&stage_empty[st], ph ^ 1, p.status, 201)) { ok = false; break; }
          if (CONV && main_step) {
            // the TMA'd 16-bit weight tile has the other 16-bit type: convert it in place
            // (element-wise, so the swizzled placement is untouched)
            if (!mbar_wait(&full[st], ph, p.status, 203)) { ok = false; break; }
            uint4* tile16 = (uint4*)(sW + st * C::W_BYTES);
            for (int i = 0; i < subs * (C::W_SUB / 16) / UTG; ++i) {
              uint4 v = tile16[tg + i * UTG];
              uint32_t* w = (uint32_t*)&v;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (p.conv16 == 1) {
                  __nv_bfloat162 b = __float22bfloat162_rn(__half22float2(*(__half2*)&w[j]));
                  w[j] = *(uint32_t*)&b;
                } else {
                  __half2 h = __float22half2_rn(__bfloat1622float2(*(__nv_bfloat162*)&w[j]));
                  w[j] = *(uint32_t*)&h;
                }
              }
              tile16[tg + i * UTG] = v;
            }
            fence_proxy_async_smem();
          }
          if (TM && main_step) {
            // one of the group's two warps per lane quarter takes each of the stage's two steps; a thread unpacks the
            // 64 codes of its weight row, which it is the TMEM lane of
            if (!mbar_wait(&raw_full[rs], rph, p.status, 202)) { ok = false; break; }
            tc_fence_after();
            const int row = (warp & 3) * 32 + lane, u = uidx & 1;
            if (u < subs) {
              const uint8_t* raw = sRaw + rs * C::RAW_STAGE + u * BB + (row >> 6) * (KS * BB);
              const uint32_t dst = tmem_base + C::a_col(st) + ((uint32_t)((warp & 3) * 32) << 16) + u * 32;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint32_t o[16];
                if (p.act_f16) unpack_unit<FMT, false, true>(raw, 2 * (row & 63) + h, 0, ud, o);
                else unpack_unit<FMT, true, true>(raw, 2 * (row & 63) + h, 0, ud, o);
                tmem_st16(dst + h * 16, o);
              }
              tmem_st_wait();
            }
            tc_fence_before();
          } else if (PACKED && main_step) {
            if (!mbar_wait(&raw_full[rs], rph, p.status, 202)) { ok = false; break; }
            // two bricks per 64-element tile: brick b fills the 8 KB half b.  A stage of two tiles goes to the
            // two halves of the group.
#pragma unroll
            for (int pass = 0; pass < C::PASSES; ++pass) {
              const int u = C::WIDE ? 0 : (tg >> 7) + pass, half = C::WIDE ? tg >> 7 : 0;
              if (u >= subs) break;
              const int next = p.dir == QG_FWD ? KS * BB : BB;
              const uint8_t* raw = sRaw + rs * C::RAW_STAGE + (p.dir == QG_FWD ? u * BB : C::BRICKS * u * BB) + half * next;
              const uint32_t dst = w_base + (uint32_t)st * C::W_BYTES + (uint32_t)u * C::W_SUB + (uint32_t)half * 8192;
              if (p.act_f16) {
#pragma unroll
                for (int b = 0; b < C::HALVES; ++b) unpack_unit<FMT, false, false>(raw + b * next, tg & 127, dst + b * 8192, ud, nullptr);
              } else {
#pragma unroll 1
                for (int b = 0; b < C::HALVES; ++b) unpack_unit<FMT, true, false>(raw + b * next, tg & 127, dst + b * 8192, ud, nullptr);
              }
            }
            fence_proxy_async_smem();
          }
          // one arrival per warp, after every lane's writes are fenced towards the tensor core's
          // reads; then the brick slot, which every lane has read, goes back to its producer
          __syncwarp();
          if (lane == 0) {
            if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&full[st]), 0));
            else if (PACKED) mbar_arrive(&full[st]);
            else mbar_arrive(&w_ready[st]);
            if (PACKED && main_step) mbar_arrive(&raw_empty[rs]);
          }
          st += UG;
          if (st >= NS) { st -= NS; ph ^= 1; }
          if (PACKED) {
            rs += UG;
            if (rs >= NR) { rs -= NR; rph ^= 1; }
          }
        }
        s -= n_steps;  // the next item's
        if (PACKED && n_steps > n_main_st && --rs < 0) { rs += NR; rph ^= 1; }  // a low-rank step takes a stage but no bricks
      }
    }
  } else if (role == R_RAW) {
    // ------------------------------------------------------------ packed-brick producer
    // Runs ahead of the stage ring: a brick pair is fetched as soon as its slot in the raw ring
    // is free, so its latency is not added to the time a weight stage is held.
    if (PACKED && elect_one()) {
      int rs = 0;
      uint32_t rph = 0;
      bool ok = true;
      constexpr uint32_t bb = (uint32_t)C::RAW_STAGE / (C::BRICKS * KS);
      for (int item = worker; item < n_items && ok; item += n_workers) {
        QG_ITEM_DECODE(item);
        (void)n_steps;
        QG_TILE_ORIGIN();
        (void)m0;
        // a pair's second half may lie past the last brick row: it then works on the last one again
        // (its results are not stored)
        const int br = min(r0 >> 6, p.nb - C::BRICKS);
        const uint8_t* b0 = p.bricks + (p.dir == QG_FWD ? ((size_t)br * p.nbk + s_begin) * bb : ((size_t)s_begin * p.nbk + br) * bb);
        const size_t b1 = p.dir == QG_FWD ? (size_t)p.nbk * bb : (size_t)bb;    // the tile's second brick
        const size_t step = p.dir == QG_FWD ? (size_t)bb : (size_t)p.nbk * bb;  // the next contraction step
        for (int si = 0; si < n_main_st; ++si, b0 += KS * step) {
          if (!mbar_wait(&raw_empty[rs], rph ^ 1, p.status, 102)) { ok = false; break; }
          const uint32_t subs = KS == 1 ? 1u : (uint32_t)min(KS, s_main - si * KS);
          uint8_t* dst = sRaw + rs * C::RAW_STAGE;
          mbar_expect_tx(&raw_full[rs], subs * C::BRICKS * bb);
          if (p.dir == QG_FWD) {  // a brick row's steps are adjacent
            bulk_load_1d(dst, b0, subs * bb, &raw_full[rs]);
            if (C::BRICKS > 1) bulk_load_1d(dst + KS * bb, b0 + b1, subs * bb, &raw_full[rs]);
          } else {  // column neighbours are adjacent
            bulk_load_1d(dst, b0, C::BRICKS * bb, &raw_full[rs]);
            if (KS > 1 && subs > 1) bulk_load_1d(dst + C::BRICKS * bb, b0 + step, C::BRICKS * bb, &raw_full[rs]);
          }
          if (++rs == NR) { rs = 0; rph ^= 1; }
        }
      }
    }
  } else if (role == R_EPI) {
    // ------------------------------------------------------------ epilogue of all tiles but the last
    const int wq = warp & 3;  // TMEM lane quarter this warp may read
    uint32_t tcount = 0;
    for (int item = worker; item + n_workers < n_items; item += n_workers, ++tcount) {
      QG_ITEM_DECODE(item);
      (void)s_begin; (void)n_steps; (void)s_main;
      QG_TILE_ORIGIN();
      const int acc = tcount & 1;
      const uint32_t aph = (tcount >> 1) & 1;
      const bool mine = SLIM || C::M64 || wq * 32 < C::ROWS;
      const uint32_t stage = smem_u32(sOut + wq * C::OUT_WARP);
      if (OUT == QO_RES && mine) residual_start(wq, 0, 1, r0, m0, stage);
      if (!mbar_wait(&acc_full[acc], aph, p.status, 401)) break;
      tc_fence_after();
      if (OUT == QO_RES) {
        if (mine) residual_tile(acc, wq, 0, 1, r0, m0, stage);
      } else for (int c = mine ? 0 : p.TN; c * 32 < tn_q; ++c) {
        if (OUT == QO_TMA16) tma_chunk(acc, wq, c, r0, m0, sOut + wq * C::OUT_WARP, out_chunk);
        else direct_chunk(acc, wq, c, r0, m0, split);
      }
      // the accumulator buffer is free once every epilogue warp of every CTA has read its lanes
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[acc]), 0));
        else mbar_arrive(&acc_empty[acc]);
      }
    }
  }
  // The epilogue of a CTA's LAST tile has nothing to hide behind, so the warps whose own work
  // is over by then help: every warp with residue q (mod 4) may read TMEM lane quarter q.
  // Quarter q's blocks go round-robin over its epilogue warp (turn 0) and its helpers (turns
  // 1..) among warps 0..14: residues 0 and 2 have three unpack warps each, residue 3 two, residue
  // 1 the two producer warps.  Helpers stage in the operand stages, which are idle once the last
  // accumulator is complete.  All of them run the same instructions: in a launch of one tile they are cold, and a copy of them in
  // each role was fetched by each role (from the complete accumulator to the end of the launch 2.3 us of 10.2, 1024x2048 Q4_0 at 1024 tokens).
  __syncwarp();
  const int q_res = warp & 3;
  const bool epi = role == R_EPI;
  if (n_my > 0 && (epi || (warp < 15 && role != R_MMA)) && (SLIM || C::M64 || q_res * 32 < C::ROWS)) {
    if (!p.late_wait && !p.end_wait && weights_only) pdl_wait();
    const int turn = epi ? 0 : warp >> 2, q_turns = (q_res == 0 || q_res == 2) ? 4 : 3;  // epilogue warp + helpers of this residue
    uint8_t* stage = epi ? sOut + q_res * C::OUT_WARP : smem + (warp - 4) * 8192;
    const int tc_last = n_my - 1, item = worker + tc_last * n_workers;
    QG_ITEM_DECODE(item);
    (void)s_begin; (void)n_steps; (void)s_main;
    QG_TILE_ORIGIN();
    const int acc = tc_last & 1;
    if (OUT == QO_RES && epi) residual_start(q_res, turn, q_turns, r0, m0, smem_u32(stage));
    if (mbar_wait(last_full, 0, p.status, 402)) {
      tc_fence_after();
      if (OUT == QO_RES) {
        if (!epi) residual_start(q_res, turn, q_turns, r0, m0, smem_u32(stage));  // (only now: over the operand stages)
        residual_tile(acc, q_res, turn, q_turns, r0, m0, smem_u32(stage));
      } else for (int c = turn; c * 32 < tn_q; c += q_turns) {
        if (OUT == QO_TMA16) tma_chunk(acc, q_res, c, r0, m0, stage, out_chunk);
        else direct_chunk(acc, q_res, c, r0, m0, split);
      }
    }
    if (lane == 0) bulk_wait_group_read<0>();  // staging may go once read; the writes land by the end of the grid
  }

  // ---------------------------------------------------------------- teardown
  if (p.end_wait) pdl_wait();
  if (*(volatile int*)p.status != 0) {
    // A wait gave up somewhere: give copies already in flight time to land before smem goes away.
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncwarp();
  // a CTA of a pair must not leave while its partner may still signal its barriers or read its memory
  if (PAIR) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

// Sums the pieces' partials in order (deterministic) and applies the epilogue the fused path would have
// applied: per-token scale, bias, accumulate or residual.  Output is f32 with row pitch ld.
__global__ void splitk_reduce_kernel(const float* part, int splits, int M, int R, float* out, size_t ld,
                                     const float* row_scale, const float* __restrict__ bias, int accumulate,
                                     const float* residual) {
  pdl_entry();
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t n = (size_t)M * R;
  if (e >= n) return;
  const int tok = (int)(e / R), row = (int)(e % R);
  float v = 0.f;
  for (int k = 0; k < splits; ++k) v += part[(size_t)k * n + e];
  if (row_scale) v *= row_scale[tok];
  if (bias) v += bias[row];
  const size_t at = tok * ld + row;
  if (accumulate) v += out[at];
  if (residual) v += residual[at];
  out[at] = v;
}

// ------------------------------------------------------------------ host side
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static PFN_encodeTiled g_encode = nullptr;

// Every (kind, format) the dispatch can ask for, with its launch shape.
struct QKernel {
  const void* fn;
  int threads, smem;
};
template <int KIND, int FMT, int OUT>
static QKernel qkernel() {
  return {(const void*)qgemm_kernel<KIND, FMT, OUT>, QCfg<KIND, FMT, OUT>::THREADS, QCfg<KIND, FMT, OUT>::SMEM_BYTES};
}
// fmt: a packed ggml format, QF_16 or QF_16CONV
template <int KIND, int OUT>
static QKernel qkernel_fmt(int fmt) {
  constexpr bool TM = KIND == QK_NARROW_T;
  if constexpr (KIND != QK_PAIR && KIND != QK_SLIM && !TM) {
    if (fmt == QF_16CONV) return qkernel<KIND, QF_16CONV, OUT>();
  }
  if constexpr (!TM) {
    if (fmt == QF_16) return qkernel<KIND, QF_16, OUT>();
  }
  switch (fmt) {
    case GGML_Q4_0: return qkernel<KIND, GGML_Q4_0, OUT>();
    case GGML_Q8_0: return qkernel<KIND, GGML_Q8_0, OUT>();
    case GGML_Q4_K: return qkernel<KIND, GGML_Q4_K, OUT>();
    case GGML_Q6_K: return qkernel<KIND, GGML_Q6_K, OUT>();
  }
  return {nullptr, 0, 0};
}
static QKernel qkernel_for(int kind, int fmt, int out) {
  const bool t = out == QO_TMA16;
  switch (kind) {
    case QK_PAIR: return t ? qkernel_fmt<QK_PAIR, QO_TMA16>(fmt) : out == QO_RES ? qkernel_fmt<QK_PAIR, QO_RES>(fmt) : qkernel_fmt<QK_PAIR, QO_DIRECT>(fmt);
    case QK_WIDE: return t ? qkernel_fmt<QK_WIDE, QO_TMA16>(fmt) : qkernel_fmt<QK_WIDE, QO_DIRECT>(fmt);
    case QK_NARROW: return t ? qkernel_fmt<QK_NARROW, QO_TMA16>(fmt) : qkernel_fmt<QK_NARROW, QO_DIRECT>(fmt);
    case QK_NARROW_T: return t ? qkernel_fmt<QK_NARROW_T, QO_TMA16>(fmt) : qkernel_fmt<QK_NARROW_T, QO_DIRECT>(fmt);
    case QK_HALF: return t ? qkernel_fmt<QK_HALF, QO_TMA16>(fmt) : qkernel_fmt<QK_HALF, QO_DIRECT>(fmt);
    case QK_SLIM: return t ? qkernel_fmt<QK_SLIM, QO_TMA16>(fmt) : qkernel_fmt<QK_SLIM, QO_DIRECT>(fmt);
  }
  return {nullptr, 0, 0};
}

// how many CTA pairs the device runs at once (0: the pair kernel is not used)
static int g_pair_workers = -1;

int qgemm_init() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || !fn)
      return RT_ERR_CUDA;
    g_encode = (PFN_encodeTiled)fn;
  }
  auto raise_smem = [](bool wide) {  // wide tiles of weights that are not converted: only where there are no pairs
    for (int kind : {(int)QK_PAIR, (int)QK_WIDE, (int)QK_NARROW, (int)QK_HALF, (int)QK_NARROW_T, (int)QK_SLIM})
      for (int fmt : {QF_16, QF_16CONV, (int)GGML_Q4_0, (int)GGML_Q8_0, (int)GGML_Q4_K, (int)GGML_Q6_K})
        for (int out : {(int)QO_TMA16, (int)QO_DIRECT, (int)QO_RES}) {
          if ((kind == QK_WIDE && fmt != QF_16CONV) != wide) continue;
          const QKernel k = qkernel_for(kind, fmt, out);
          if (k.fn && cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem) != cudaSuccess) return false;
        }
    return true;
  };
  if (!raise_smem(false)) return RT_ERR_CUDA;
  if (g_pair_workers < 0) {
    int dev = 0, sms = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const QKernel k = qkernel_for(QK_PAIR, GGML_Q8_0, QO_TMA16);  // one CTA per SM in every format
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(sms & ~1));
    cfg.blockDim = dim3((unsigned)k.threads);
    cfg.dynamicSmemBytes = (size_t)k.smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, k.fn, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    const char* e = getenv("RT_B200_NO_PAIR");
    g_pair_workers = (e && atoi(e)) ? 0 : n;
  }
  if (g_pair_workers == 0 && !raise_smem(true)) return RT_ERR_CUDA;
  return RT_OK;
}

// 2-D row-major 16-bit matrix [rows x cols]; box = box_cols x box_rows, 128-byte swizzle.
static int encode_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_cols,
                      uint32_t box_rows, bool is_bf16, uint64_t ld = 0) {
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {(ld ? ld : cols) * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(m, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                        const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? RT_OK : RT_ERR_CUDA;
}

std::atomic<unsigned long long> g_launch_count{0};

static int make_map_cached(rt_ctx* ctx, CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_cols,
                           uint32_t box_rows, bool is_bf16, uint64_t ld = 0) {
  if (ld == cols) ld = 0;
  if (!ctx) return encode_map(m, base, rows, cols, box_cols, box_rows, is_bf16, ld);  // no cache: nothing is allocated
  auto key = std::make_tuple(base, rows, cols | (ld << 32), box_cols, box_rows, is_bf16);
  auto it = ctx->tmap_cache.find(key);
  if (it != ctx->tmap_cache.end()) {
    *m = it->second;
    return RT_OK;
  }
  int rc = encode_map(m, base, rows, cols, box_cols, box_rows, is_bf16, ld);
  if (rc) return rc;
  if (ctx->tmap_cache.size() > 8192) ctx->tmap_cache.clear();
  ctx->tmap_cache.emplace(key, *m);
  return RT_OK;
}
#define make_map(m, ...) make_map_cached(a.fixed_part ? nullptr : ctx, m, __VA_ARGS__)

int tensor_map_f16_2d(rt_ctx* ctx, CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_cols,
                      uint32_t box_rows) {
  if (!g_encode) {
    int rc = qgemm_init();
    if (rc) return rc;
  }
  return make_map_cached(ctx, m, base, rows, cols, box_cols, box_rows, false);
}

int tensor_map_f16_2d_ld(rt_ctx* ctx, CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                         uint32_t box_cols, uint32_t box_rows) {
  if (!g_encode) {
    int rc = qgemm_init();
    if (rc) return rc;
  }
  return make_map_cached(ctx, m, base, rows, cols, box_cols, box_rows, false, ld);
}

// Output matrix [rows x cols] of bf16 / f16 with a row pitch of `ld` elements; box = 32 columns x 32 rows
// (one epilogue warp's block) of 64-byte rows, 64-byte swizzle.
static int make_out_map(rt_ctx* ctx, CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, int dtype) {
  auto key = std::make_tuple(base, rows, cols | (ld << 32), 32u, 32u | ((uint32_t)dtype << 8), true);
  if (ctx) {
    auto it = ctx->tmap_cache.find(key);
    if (it != ctx->tmap_cache.end()) {
      *m = it->second;
      return RT_OK;
    }
  }
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = dtype == OUT_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = g_encode(m, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return RT_ERR_CUDA;
  if (!ctx) return RT_OK;
  if (ctx->tmap_cache.size() > 8192) ctx->tmap_cache.clear();
  ctx->tmap_cache.emplace(key, *m);
  return RT_OK;
}

// Which kernel and token-tile width a product gets: the one whose persistent grid is estimated to finish
// first: the launch + rounds of tiles x (contraction steps x the step's time + a tile's own time), in us, 64 contraction
// elements a step.  The constants are fitted so that the choice is right, not each time: to every kind and width of 2880 products
// (21 shapes of 128..16384 rows and columns, both directions, 1..8192 tokens, five formats, weights from memory), each
// behind itself, where launches overlap, and behind a kernel that lets nothing start under it.  Against the best kind and
// width of each, the choice is 0.9 % off on average (0.84 and 0.92 on the two halves of the products); 3 % of the products are off by
// more than 10 % in one of the two, nearly all of them launches below 10 us, the worst by 26 % (4096x1024 Q8_0 at 100 tokens, 8.0
// us on half tiles, 6.4 on narrow ones).  (Before, with 0.5 to 1 us more for the launch of pairs and slim pairs and a fourth more
// for their steps, 3.0 % off, a tenth of the times by more than 10 %: 3072x1024 Q4_0 at 400 tokens on narrow tiles 10.4 us, and 14.7
// behind a kernel that lets nothing start, on pairs 9.3 and 12.9.)
// (On 1400 products of twelve shapes, in graphs, since f32 results gave their staging's room to the brick ring: 2.4 % off behind itself,
// 1.0 % behind such a kernel; the constants fitted anew would be 2.2 and 0.9 % off, and stand.)
// What a step's time stands for: a pair's for its MMAs from about 96 tokens of width on and for the hand-offs between the
// roles below; a slim pair's for shared memory; half and narrow tiles' for one round of unpacking, which is
// shortest for Q8_0's codes.
// Slim pairs against narrow tiles at 1024 tokens, Q4_0 | Q6_K: 6144x1024 backward 25.6 -> 18.4 | 30.1 -> 20.5 us, 4096x1024 backward
// 18.6 -> 14.1 | 21.4 -> 15.3, 1024x3072 forward 13.4 -> 11.9 | 15.2 -> 12.8; against half tiles, 8192x3072 Q6_K backward at 24
// tokens 26.7 -> 24.2.
// The choice changes no result: an output element's contraction is one chain in any tile.
struct QPlan {
  int kind, TN;
};
static QPlan qgemm_plan(int kfmt, int dir, int M, int out_rows, int n_splits, int steps, int num_sms, bool out16) {
  QPlan best = {QK_NARROW, 64};
  double best_cost = -1;
  auto consider = [&](int kind, int tn, double step_us, double tile_us, double launch_us) {
    const int rows = kind == QK_PAIR ? 256 : kind == QK_HALF ? 64 : 128;
    const long tiles = (long)((out_rows + rows - 1) / rows) * ((M + tn - 1) / tn) * n_splits;
    const long workers = kind == QK_PAIR || kind == QK_SLIM ? g_pair_workers : num_sms;
    const double cost = launch_us + (double)((tiles + workers - 1) / workers) * (steps * step_us + tile_us);
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = {kind, tn}; }
  };
  const bool packed = kfmt > QF_16CONV;
  if (kfmt == QF_16CONV) {  // single CTAs only: their warps convert what TMA brought
    for (int tn = M > 32 ? 64 : 32; tn >= 32; tn -= 32) {
      consider(QK_NARROW, tn, 0.25, 0.5, 0);
      consider(QK_HALF, tn, tn == 64 ? 0.16 : 0.155, 0.5, 0);
    }
    for (int tn = 256; tn >= 128; tn -= 32) consider(QK_WIDE, tn, 0.25 + 0.0012 * tn, 0.5, 0);
    return best;
  }
  const bool q8 = kfmt == GGML_Q8_0;
  for (int tn = M > 32 ? 64 : 32; tn >= 32; tn -= 32) {
    if (packed && dir == QG_FWD) consider(QK_NARROW_T, tn, q8 ? 0.17 : 0.195, 0.4, 2.5);
    else consider(QK_NARROW, tn, 0.23, 0.45, 2.7);
    consider(QK_HALF, tn, (q8 ? 0.14 : packed ? 0.215 : 0.23) - (tn == 32 ? 0.01 : 0.0), 0.6, 2.1);
  }
  if (g_pair_workers > 0) {
    for (int tn = M > 64 ? 128 : M > 32 || out16 ? 64 : 32; tn >= (out16 ? 64 : 32); tn /= 2) consider(QK_SLIM, tn, packed ? 0.14 : 0.128, 0.87, packed ? 3.6 : 4.2);
    for (int tn = 256; tn >= 64 && M > 64; tn -= 32) consider(QK_PAIR, tn, 0.146 + 0.0008 * tn > 0.218 ? 0.146 + 0.0008 * tn : 0.218, 0.4, 5.0);
  } else if (M > 64) {  // without pairs: 8192x3072 Q8_0 at 4096 tokens 171-181 us, 279-341 on 64-token tiles
    for (int tn = 256; tn >= 96; tn -= 32) consider(QK_WIDE, tn, 0.15 + 0.0012 * tn > 0.35 ? 0.15 + 0.0012 * tn : 0.35, 0.5, 2.4);
  }
  return best;
}

// How a product runs: the weight as the kernel sees it, where the contraction is cut, and the tiles.
struct QSetup {
  int kfmt, conv16, contract, out_rows, n_main, steps_per_split, n_splits;
  QPlan plan;
};
static QSetup qgemm_setup(const rt_ctx* ctx, const QWeight& w, int dir, bool act_f16, int M, int out_dtype) {
  QSetup q;
  q.conv16 = (w.fmt == GGML_F16 && !act_f16) ? 1 : (w.fmt == GGML_BF16 && act_f16) ? 2 : 0;
  q.kfmt = !fmt_is_16bit(w.fmt) ? w.fmt : q.conv16 ? QF_16CONV : QF_16;
  q.contract = dir == QG_FWD ? w.cols : w.rows;
  q.out_rows = dir == QG_FWD ? w.rows : w.cols;
  q.n_main = (q.contract + 63) / 64;
  // How the contraction is cut into accumulation chains depends on the weight's shape ONLY, never
  // on the number of tokens: the tensor core's accumulator does not round to nearest, so two
  // partitions of one sum differ by a few 1e-6 relative, which the next 16-bit rounding of the
  // activations amplifies a hundredfold.  With a token-dependent split-K a sequence's result
  // depended on its batch mates (a shard of one or two sequences against the whole batch: 7e-4
  // on the gradients); with a fixed partition it is bit-identical in any batch.
  // A very long contraction (the head's backward runs over the whole vocabulary) is accumulated
  // in pieces of a FIXED 8192 elements whose f32 partial sums are added afterwards: the error of
  // one chain grows with its length (about 3e-4 relative over 150 000 elements).
  q.steps_per_split = q.n_main;
  if (out_dtype == OUT_F32 && q.n_main > 256) q.steps_per_split = 128;
  q.n_splits = (q.n_main + q.steps_per_split - 1) / q.steps_per_split;
  q.plan = qgemm_plan(q.kfmt, dir, M, q.out_rows, q.n_splits, q.steps_per_split, ctx->num_sms, out_dtype != OUT_F32);
  return q;
}

int qgemm_launch(rt_ctx* ctx, const QWeight& w, const QGemmArgs& a) {
  const int num_sms = ctx->num_sms;
  cudaStream_t st = ctx->stream;
  if (!g_encode) {
    int rc = qgemm_init();
    if (rc) return rc;
  }
  if (a.M <= 0) return RT_OK;
  const bool is16 = fmt_is_16bit(w.fmt);
  const QSetup setup = qgemm_setup(ctx, w, a.dir, a.act_f16 != 0, a.M, a.out_dtype);
  const QPlan plan = setup.plan;
  const int kfmt = setup.kfmt, contract = setup.contract, out_rows = setup.out_rows;
  if (contract % 8 != 0 || (is16 && w.cols % 8 != 0)) return RT_ERR_BAD_SHAPE;
  if ((a.accumulate || a.residual) && a.out_dtype != OUT_F32) return RT_ERR_BAD_ARG;
  if (a.lora.rank > 64 || (a.lora.rank > 0 && (!a.lora.act || !a.lora.w))) return RT_ERR_BAD_ARG;

  KParams p;
  p.bricks = w.bricks;
  p.nb = a.dir == QG_FWD ? w.nbr : w.nbk;
  p.nbk = w.nbk;
  p.act_f16 = a.act_f16 ? 1 : 0;
  p.conv16 = setup.conv16;
  p.row_scale = a.row_scale;
  p.residual = a.residual;
  p.late_wait = a.late_wait && a.lora.rank > 0 ? 1 : 0;
  p.end_wait = a.end_wait;
  p.dir = a.dir;
  p.out_rows = out_rows;
  p.M = a.M;
  p.n_main = setup.n_main;
  p.lora_mmas = a.lora.rank > 0 ? (a.lora.rank + 15) / 16 : 0;
  p.out = a.out;
  p.out_dtype = a.out_dtype;
  p.accumulate = a.accumulate;
  p.ld_out = a.ld_out > 0 ? a.ld_out : out_rows;
  p.bias = a.dir == QG_FWD ? a.bias : nullptr;
  p.status = ctx->status_dev;
  p.steps_per_split = setup.steps_per_split;
  p.n_splits = setup.n_splits;
  const bool pair = plan.kind == QK_PAIR || plan.kind == QK_SLIM;
  p.TN = plan.TN;
  const int tile_rows = plan.kind == QK_PAIR ? 256 : plan.kind == QK_HALF ? 64 : 128;
  p.n_row_tiles = (out_rows + tile_rows - 1) / tile_rows;
  p.n_tok_tiles = (a.M + p.TN - 1) / p.TN;
  // Tiles that run together share a token tile's activations; but weights that do not fit beside them in L2 (126 MB)
  // come from memory again for every token tile (the head's 151936x1024 in Q8_0 at 1024 tokens: 664 MB read for
  // 165), so then the token tiles of the same weights run together, while the activations do fit.  128256x3072 in Q6_K at
  // 1024 tokens 631 -> 609 us; at 87 MB of weights, which stay in L2, the other order is the better one by a little.
  p.tok_first = p.n_tok_tiles > 1 && w.dev_nbytes > ((size_t)96 << 20) && (size_t)a.M * contract * 2 <= ((size_t)32 << 20) && plan.kind == QK_PAIR;
  p.inner = p.tok_first ? p.n_tok_tiles : p.n_row_tiles;
  const int tn_cta = pair ? p.TN / 2 : p.TN;  // each CTA of a pair fetches its half of the token tile
  // tcgen05.mma kind::f16 needs A and B of ONE 16-bit type (f16 x bf16 is an illegal instruction).
  const int ab_fmt = a.act_f16 ? 0 : 1;

  CUtensorMap tm_act, tm_w16, tm_lact, tm_lw;
  int rc = make_map(&tm_act, a.act, (uint64_t)a.M, (uint64_t)contract, 64, (uint32_t)tn_cta, !a.act_f16);
  if (rc) return rc;
  tm_w16 = tm_act;
  tm_lact = tm_act;
  tm_lw = tm_act;
  if (is16) {
    rc = make_map(&tm_w16, w.dense16, (uint64_t)w.rows, (uint64_t)w.cols, 64, 64, w.fmt == GGML_BF16);
    if (rc) return rc;
  }
  if (a.lora.rank > 0) {
    rc = make_map(&tm_lact, a.lora.act, (uint64_t)a.M, 64, 64, (uint32_t)tn_cta, !a.act_f16);
    if (rc) return rc;
    if (a.dir == QG_FWD) rc = make_map(&tm_lw, a.lora.w, (uint64_t)w.rows, 64, 64, 64, !a.act_f16);
    else rc = make_map(&tm_lw, a.lora.w, (uint64_t)a.lora.rank, (uint64_t)w.cols, 64, 64, !a.act_f16);
    if (rc) return rc;
  }
  p.part = nullptr;
  if (p.n_splits > 1) {
    const size_t need = (size_t)p.n_splits * a.M * out_rows;
    if (a.fixed_part) {
      if (need > a.fixed_part_floats) return RT_ERR_TOO_LARGE;
      p.part = a.fixed_part;
    } else {
      p.part = (float*)ctx->get_scratch(3, need * sizeof(float));
      if (!p.part) return RT_ERR_CUDA;
    }
  }
  int out_kind = QO_DIRECT;
  if (plan.kind == QK_PAIR && !p.part && a.residual && (uintptr_t)a.residual % 16 == 0 && p.ld_out % 4 == 0 && out_rows % 4 == 0) out_kind = QO_RES;
  // 16-bit outputs leave through TMA whenever it can address them (16-byte aligned base and row pitch)
  CUtensorMap tm_out = tm_act;
  const bool out_blocks = plan.kind != QK_SLIM || p.TN >= 64;  // a quarter of the accumulator is whole blocks of 32 tokens
  if (!p.part && out_blocks && a.out_dtype != OUT_F32 && (uintptr_t)a.out % 16 == 0 && (uint64_t)p.ld_out % 8 == 0) {
    rc = make_out_map(a.fixed_part ? nullptr : ctx, &tm_out, a.out, (uint64_t)a.M, (uint64_t)out_rows, (uint64_t)p.ld_out, a.out_dtype);
    if (rc) return rc;
    out_kind = QO_TMA16;
  }
  p.idesc = umma_idesc(ab_fmt, ab_fmt, a.dir == QG_BWD ? 1 : 0, 0, plan.kind == QK_PAIR ? 256 : plan.kind == QK_HALF && out_kind == QO_DIRECT ? 64 : 128, p.TN);
  const int n_items = p.n_row_tiles * p.n_tok_tiles * p.n_splits;
  const int workers = pair ? g_pair_workers : num_sms;
  const int grid = (n_items < workers ? n_items : workers) * (pair ? 2 : 1);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ctx->profiling && !a.fixed_part) {
    if (ctx->prof_used + 2 > ctx->prof_events.size()) {
      for (int i = 0; i < 256; ++i) {
        cudaEvent_t e;
        if (cudaEventCreate(&e) != cudaSuccess) return RT_ERR_CUDA;
        ctx->prof_events.push_back(e);
      }
    }
    e0 = ctx->prof_events[ctx->prof_used++];
    e1 = ctx->prof_events[ctx->prof_used++];
    cudaEventRecord(e0, st);
  }
  {
    const QKernel k = qkernel_for(plan.kind, kfmt, out_kind);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() || (a.end_wait && pdl_any_size()) ? 1 : 0;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 2;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)k.threads);
    cfg.dynamicSmemBytes = (size_t)k.smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = pair ? 2 : 1;
    void* args[] = {&tm_act, &tm_w16, &tm_lact, &tm_lw, &tm_out, &p};
    if (cudaLaunchKernelExC(&cfg, k.fn, args) != cudaSuccess) return RT_ERR_CUDA;
  }
  RT_COUNT_LAUNCH(1);
  if (p.part) {
    const size_t n = (size_t)a.M * out_rows;
    pdl(splitk_reduce_kernel, (unsigned)((n + 255) / 256), 256, 0, st)(p.part, p.n_splits, a.M, out_rows, (float*)a.out, (size_t)p.ld_out,
                                                                    a.row_scale, p.bias, a.accumulate, a.residual);
    RT_COUNT_LAUNCH(1);
  }
  if (e1) {
    cudaEventRecord(e1, st);
    const double out_bytes = a.out_dtype == OUT_F32 ? 4.0 : 2.0;
    ctx->prof_flops += 2.0 * (double)a.M * (double)w.rows * (double)w.cols;
    ctx->prof_recs.push_back({a.dir, a.M, out_rows, contract});
    ctx->prof_bytes += (double)w.dev_nbytes + 2.0 * (double)a.M * contract + out_bytes * (double)a.M * out_rows * (a.accumulate || a.residual ? 2.0 : 1.0);
  }
  return cudaGetLastError() == cudaSuccess ? RT_OK : RT_ERR_CUDA;
}


// ------------------------------------------------------------------ the bounded wait, exercised on its own
// One warp waits on a barrier nobody arrives on, with a short limit: the wait gives up, records
// its site code and the kernel returns normally, which is what every wait of the matmul kernel
// does when a peer never shows up.  The context stays usable.
__global__ void wait_selftest_kernel(int* status, long long limit_cycles) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(&bar, 0, status, 999, limit_cycles);
}

// ------------------------------------------------------------------ allocation-free entry point
// The partial sums of a contraction that is accumulated in pieces (more than 16384 weight rows)
// live here for rt_frozen_backward_input_dev_noalloc instead of in memory from cudaMalloc.  Every GPU that loads the library holds these 8 MiB until the process exits.
constexpr size_t NOALLOC_SCRATCH_FLOATS = (size_t)2 << 20;
static __device__ __align__(256) float g_noalloc_scratch[NOALLOC_SCRATCH_FLOATS];
static float* g_noalloc_scratch_addr[64] = {nullptr};  // device address of the array, per device ordinal

// In host code `g_noalloc_scratch` is only a stand-in for the symbol, not a device address: the
// address a kernel can use comes from cudaGetSymbolAddress, asked once per device with that
// device current.
static int noalloc_scratch_for(int device, float** out) {
  if (device < 0 || device >= 64) return RT_ERR_BAD_ARG;
  if (!g_noalloc_scratch_addr[device]) {
    void* p = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return RT_ERR_CUDA;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return RT_ERR_CUDA;
    g_noalloc_scratch_addr[device] = (float*)p;
  }
  *out = g_noalloc_scratch_addr[device];
  return RT_OK;
}

}  // namespace rt

extern "C" rt_status rt_ctx_selftest_wait_timeout(rt_ctx* c, uint64_t limit_cycles) {
  if (!c) return RT_ERR_BAD_ARG;
  if (limit_cycles == 0 || limit_cycles > 2000000000ull) return c->fail(RT_ERR_BAD_ARG, "limit must be 1..2e9 cycles");
  if (cudaSetDevice(c->device) != cudaSuccess) return RT_ERR_CUDA;
  rt::wait_selftest_kernel<<<1, 32, 0, c->stream>>>(c->status_dev, (long long)limit_cycles);
  if (cudaGetLastError() != cudaSuccess) return c->fail(RT_ERR_CUDA, "self-test launch failed");
  return c->check_device_status("rt_ctx_selftest_wait_timeout");  // expected: RT_ERR_DEVICE_WAIT_TIMEOUT, site 999
}

extern "C" rt_status rt_frozen_tile(const rt_frozen* f, int backward, size_t t, int in_dtype, int out_dtype, int* kind, int* tokens) {
  static_assert(RT_TILE_PAIR == rt::QK_PAIR && RT_TILE_WIDE == rt::QK_WIDE && RT_TILE_NARROW == rt::QK_NARROW && RT_TILE_HALF == rt::QK_HALF &&
                    RT_TILE_NARROW_TMEM == rt::QK_NARROW_T && RT_TILE_SLIM == rt::QK_SLIM,
                "the header's kinds are the kernel's");
  if (!f || !kind || !tokens || t == 0 || t > (1u << 24)) return RT_ERR_BAD_ARG;
  if ((in_dtype != RT_DT_F16 && in_dtype != RT_DT_BF16) || out_dtype < 0 || out_dtype > 2) return RT_ERR_BAD_ARG;
  const rt::QPlan plan =
      rt::qgemm_setup(f->ctx, f->w, backward ? rt::QG_BWD : rt::QG_FWD, in_dtype == RT_DT_F16, (int)t, out_dtype).plan;
  *kind = plan.kind;
  *tokens = plan.TN;
  return RT_OK;
}

extern "C" rt_status rt_frozen_backward_input_dev_noalloc(rt_frozen* f, const void* dy_dev, int in_dtype, size_t t,
                                                          void* dx_dev, int out_dtype, int accumulate) {
  if (!f || !dy_dev || !dx_dev) return RT_ERR_BAD_ARG;
  rt_ctx* c = f->ctx;
  if (t == 0) return RT_OK;
  if (t > (1u << 24)) return RT_ERR_BAD_SHAPE;
  if (in_dtype != RT_DT_F16 && in_dtype != RT_DT_BF16) return RT_ERR_BAD_ARG;
  if (out_dtype < 0 || out_dtype > 2 || (accumulate && out_dtype != RT_DT_F32)) return RT_ERR_BAD_ARG;
  if (cudaSetDevice(c->device) != cudaSuccess) return RT_ERR_CUDA;
  float* scratch = nullptr;
  int rc = rt::noalloc_scratch_for(c->device, &scratch);  // first call on a device: looks the array up
  if (rc) return rc;
  rt::QGemmArgs a;
  a.dir = rt::QG_BWD;
  a.act = dy_dev;
  a.act_f16 = in_dtype == RT_DT_F16;
  a.M = (int)t;
  a.out = dx_dev;
  a.out_dtype = out_dtype;
  a.accumulate = accumulate ? 1 : 0;
  a.fixed_part = scratch;
  a.fixed_part_floats = rt::NOALLOC_SCRATCH_FLOATS;
  return rt::qgemm_launch(c, f->w, a);
}
