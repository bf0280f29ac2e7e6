// Backward dynamic-mask attention for sm_100a, head dims up to 128, masks and biases that are broadcast over the queries (or
// absent) and packed sequences: dQ, dK, dV and dBias from dO, O, LSE. Per-query masks and biases: fdma_bwd_sm100.cu.
//
// Math of the reference's compute_dq_dk_dv_1colblock (csrc/flash_sparse_attn/src/flash_bwd_kernel.h:79-1142):
//   P = exp(S - LSE), dP = dO V^T, dS = P o (dP - D), D = rowsum(dO o O),
//   dV = P^T dO, dK = scale dS^T Q, dQ = scale dS K, dBias = dS.
// Two passes over the scores, whose CTAs share one launch, both a stationary tile of 128 rows and tiles of 64 rows that stream by:
//                stationary      streamed            products per step
//     key pass   K, V (a tile)   Q, dO (each head)   St = K Q^T, dPt = V dO^T, dV += P^T dO, dK += dS^T Q
//     row pass   Q, dO (a tile)  K, V                S = Q K^T,  dP = dO V^T,  dQ += dS K
// A stationary operand lives in TENSOR MEMORY, as the A operand of its products (copied there once per tile), and so do P and dS,
// written back over the scores in 16 bit; the tensor core reads little but the 64 streamed rows from shared memory (a 128 x 64 x 16
// product takes 33 cycles with A in tensor memory and 54 with A in shared memory). The single pass this replaces formed five products
// instead of seven, but moved 48 + 48 KB per step through shared memory for the scores, 48 KB for dQ^T = K^T dS^T, 16 KB of dS and twice
// 32 KB of fp32 dQ on its way to a buffer in global memory, which also had to be zeroed, added to and converted. Here dQ stays in the
// CTA: the tensor core sums up 128 keys at a time (it truncates its sums: over 2048 keys dQ lost 1.1e-5 of its size), and the softmax
// threads add those sums up in registers, rounding to nearest. It is the same bits every time: nothing changes for `deterministic`.
// Whole backward in us, single pass (with the slower issue it had) -> this: plain causal 4096 x 32 heads 580 -> 464, 8192 packed tokens
// 583 -> 364, 32768 queries over 2048 kept keys 2246 -> 2059, deterministic, 8192 queries over 2048 kept keys 1020 -> 609.
//
// Tensor memory, columns: scores[2] 2 x 64 | dP 64 (key pass at D = 128) or 2 x 64 | accumulators | stationary operands.
// Only V in the key pass at D = 128 finds no room there (scores 128, dP 64, K 64, dV 128, dK 128) and stays in shared memory.
//
// Warps: 0 TMA producer | 1 MMA issuer | 2 row pass: addend and position of the step's 64 keys | 3 row pass: which key tiles the
// next item works on | 4-7 and 8-11 two softmax teams (thread = stationary row = TMEM lane), 32 of a step's 64 columns each. Scores
// have two buffers: the products of step i+1 run under the softmax of step i, behind the gradient products of step i-1. (With the
// teams on alternate steps, a team's 64 columns and the products that wait for them made one chain: 531 against 488 us, plain 4096.)
// What bounds it: the softmax warps, two per scheduler, some 1000 cycles for a step of 64 columns against 512 of exp2. Every mbarrier
// wait is bounded.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>

#include "fdma_internal.h"
#include "fdma_packed.cuh"
#include "fdma_ptx.cuh"

namespace fdma {
namespace {

constexpr int kBN = 128;      // stationary rows per tile
constexpr int kBM = 64;       // streamed rows per step
constexpr int kThreads = 384;
constexpr int kStages = 4;    // ring of streamed tiles
constexpr int kVecSlots = 4;  // ring of key addends and positions (row pass)
// 64-key steps whose dQ the tensor core sums up (128 keys, as a key tile's dQ was added to a buffer in memory before). Taking the sums out
// at the start of a step, with no wait of their own, against at the end of it: plain causal 8192 x 16 heads 850 against 883 us, 32768
// queries over 2048 gathered keys 1988 against 2020 (1936 with sums over all 2048 keys).
constexpr int kFlush = 2;
// 64-query steps whose dK and dV the tensor core sums up: 192 additions, no more than one CTA of the single pass made (that took up to a
// whole group's queries, or 80 steps and more of them). Moving them out costs some 1700 cycles (0.9 us), the time of 128 KB on their way to L2.
constexpr int kKeyFlush = 48;
constexpr int kMaxBits = 4096;   // 64-key tiles the activity bits of a row-pass item can hold
constexpr int kMaxHeads = 4096;  // query heads of a group whose activity differs from head to head
constexpr int kDbHeads = 16;    // query heads of a group whose dBias sums have room in shared memory
constexpr float kLog2e = 1.4426950408889634f;

enum DbiasMode { kDbNone = 0, kDbColsum = 1, kDbAtomic = 3 };
enum WaitCode {
  kWaitX = 401, kWaitXEmpty = 402, kWaitReady = 403, kWaitStFull = 404, kWaitStEmpty = 405, kWaitS = 406, kWaitDpFree = 407,
  kWaitPds = 408, kWaitVecFull = 409, kWaitVecEmpty = 410, kWaitFinal = 411, kWaitAccFree = 412, kWaitItemFull = 413,
  kWaitItemEmpty = 414
};

struct BwdRowsParams {
  CUtensorMap tm_q, tm_do, tm_k, tm_v;  // boxes of 64 rows x 64 elements
  const uint8_t* mask;
  const void* bias;
  const float* lse2;   // (B,H,Sq_r) LSE * log2(e); +inf for empty and padded rows
  const float* dsum;   // (B,H,Sq_r) D = rowsum(dO o O)
  void* dq;
  void* dk;
  void* dv;
  void* dbias;         // column-sum mode: the output tensor
  float* dbias_acc;    // atomic mode: fp32 buffer (dbias_b, dbias_h, dbias_keys), zeroed
  float* dq_part;      // more than one key range: fp32 partials [ranges][B][H][Sq][D] instead of dq
  float* dkv_sums;     // more than kKeyFlush steps: fp32 [2: dV, dK][nsplit][B][h_k][NT*128 * D], a CTA's rows as [D / 4][rows][4]
  float* dkv_part;     // null, or fp32 partials [2: dV, dK][nsplit][B][h_k][NT*128][D] instead of dk / dv
  float* dbias_part;   // with dkv_part, column-sum mode: fp32 partials [nsplit][B][h_k][NT*128]
  int* status;
  int64_t mask_batch_stride, mask_head_stride, bias_batch_stride, bias_head_stride;
  int64_t dq_batch_stride, dq_row_stride, dq_head_stride;
  int64_t dk_batch_stride, dk_row_stride, dk_head_stride;
  int64_t dv_batch_stride, dv_row_stride, dv_head_stride;
  int64_t dbias_batch_stride, dbias_head_stride;
  int b, seqlen_q, seqlen_k, sq_r, h, h_k, h_mask, h_bias, d;
  int dbias_b, dbias_h, dbias_keys, dbias_mode;
  int is_causal;
  const int32_t* key_pos;  // ascending positions of compacted keys, or null
  int64_t pos_batch_stride, pos_head_stride;
  int h_pos, causal_shift;
  PackedSeqs seqs;   // packed sequences, each with tiles of its own; streamed query tiles are cut at fixed rows
  int n_tiles;       // key tiles (packed: places for them)
  int q_tiles;       // row-pass tiles (packed: places for them)
  int nsplit;        // query-range splits per key tile
  int n_key_ctas;    // CTAs of the key pass
  int heads_per_cta; // query heads a row-pass CTA works on, one after the other
  int ranges;        // key ranges a row-pass tile is cut into, a CTA each
  float scale_log2, scale;
};

template <int D>
struct SmemR {
  static constexpr int kTile = kBN * D * 2;                 // a stationary tile: D / 64 blocks of [128 rows][64]
  static constexpr int kStep = kBM * D * 2;                 // a streamed tile: D / 64 blocks of [64 rows][64]
  static constexpr int kXOff = 0;                           // K or Q, on its way to tensor memory
  static constexpr int kX2Off = kTile;                      // V or dO
  static constexpr int kStOff = 2 * kTile;                  // stages: Q then dO, or K then V
  static constexpr int kLdOff = kStOff + kStages * 2 * kStep;        // key pass, per stage: 64 x LSE*log2e, 64 x D
  static constexpr int kVecOff = kLdOff + kStages * 2 * kBM * 4;     // row pass, per slot: 64 addends, 64 positions
  static constexpr int kBitsOff = kVecOff + kVecSlots * 2 * kBM * 4; // row pass: two tables of activity bits
  static constexpr int kHeadsOff = kBitsOff;                         // key pass: list of the group's active heads (16 bit)
  static constexpr int kRedOff = kBitsOff + kMaxHeads * 2;
  static constexpr int kDbOff = kRedOff + kBN * 4;                   // key pass: dBias sums, [2 teams][kDbHeads][kBN]
  static constexpr int kBarOff = kDbOff + 2 * kDbHeads * kBN * 4;
  static constexpr int kNumBars = 3 + 2 * kStages + 2 + 2 + 2 + 2 * kVecSlots + 2 + 4;
  static constexpr int kMiscOff = kBarOff + kNumBars * 8;
  static constexpr int kTotal = kMiscOff + 64;
  static constexpr int kAlloc = kTotal + 1024;  // slack to align the base to 1024 B
  static_assert(2 * (kMaxBits / 8) <= kMaxHeads * 2, "the bit tables lie in the head list's place");
  static_assert(kAlloc <= 232448, "shared memory budget of one CTA");
};

template <bool kBf16>
__device__ __forceinline__ float raw16_to_f(uint16_t u) {
  if (kBf16) return __uint_as_float(static_cast<uint32_t>(u) << 16);
  return __half2float(__ushort_as_half(u));
}
template <bool kBf16>
__device__ __forceinline__ uint16_t f_to_raw16(float x) {
  return static_cast<uint16_t>(pack_16x2<kBf16>(x, 0.f) & 0xFFFFu);
}

// 64512 registers (384 threads x 168 at launch) = 128 x 64 (warps 0-3) + 256 x 216 (softmax teams) + 1024. The instruction stands at the
// top of each role's branch, where the compiler takes it for the limit of that branch.
#define FDMA_LIGHT_REGS() asm volatile("setmaxnreg.dec.sync.aligned.u32 64;")
#define FDMA_TEAM_REGS() asm volatile("setmaxnreg.inc.sync.aligned.u32 216;")

// s_full, dp_free and pds come in pairs, by step parity: the softmax warps may be done with two steps before the MMA warp, held up by
// another wait, looks for the first of them, and would then have moved one barrier on by two phases, which reads as none.
struct Bars {
  uint64_t *x_full, *x_empty, *ready, *st_full, *st_empty, *s_full, *dp_free, *pds, *vec_full, *vec_empty, *final_, *acc_free,
      *item_full, *item_empty;
  __device__ explicit Bars(uint64_t* p)
      : x_full(p), x_empty(p + 1), ready(p + 2), st_full(p + 3), st_empty(st_full + kStages), s_full(st_empty + kStages),
        dp_free(s_full + 2), pds(dp_free + 2), vec_full(pds + 2), vec_empty(vec_full + kVecSlots), final_(vec_empty + kVecSlots),
        acc_free(final_ + 1), item_full(acc_free + 1), item_empty(item_full + 2) {}
};

template <int D, bool kKeys>
struct Cols {
  static constexpr uint32_t kS = 0, kDp = 128;
  static constexpr uint32_t kAcc = 256;  // dV, then dK; or dQ
  static constexpr uint32_t kX = kKeys ? (D == 128 ? 192 : 384) : 384;
  static constexpr uint32_t kX2 = kX + D / 2;
};

// This thread's row of a stationary tile from shared memory (128-byte swizzle) into tensor memory, as an A operand.
template <int D>
__device__ __forceinline__ void tile_row_to_tmem(const unsigned char* tile, int row, uint32_t taddr) {
#pragma unroll
  for (int kb = 0; kb < D / 64; ++kb) {
    uint32_t v[32];
    const unsigned char* src = tile + kb * (kBN * 128) + row * 128;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint4 x = *reinterpret_cast<const uint4*>(src + ((c ^ (row & 7)) << 4));
      v[c * 4] = x.x; v[c * 4 + 1] = x.y; v[c * 4 + 2] = x.z; v[c * 4 + 3] = x.w;
    }
    tmem_st_x32(taddr + kb * 32, v);
  }
}

// [128 x 64] = stationary (tensor memory) x streamed^T
template <int D, bool kBf16>
__device__ __forceinline__ void product_ts(uint32_t lead, uint32_t dst, uint32_t a_tmem, uint32_t b_smem) {
  constexpr uint32_t idesc = umma_idesc(kBN, kBM, kBf16, false, false);
  const uint64_t b = umma_desc_sw128(b_smem, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
    umma_ts(lead, dst, a_tmem + kk * 8, umma_desc_at(b, (kk >> 2) * (kBM * 128) + (kk & 3) * 32), idesc, kk > 0 ? 1u : 0u);
}
template <int D, bool kBf16>
__device__ __forceinline__ void product_ss(uint32_t lead, uint32_t dst, uint32_t a_smem, uint32_t b_smem) {
  constexpr uint32_t idesc = umma_idesc(kBN, kBM, kBf16, false, false);
  const uint64_t a = umma_desc_sw128(a_smem, 16, 1024), b = umma_desc_sw128(b_smem, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk)
    umma_ss(lead, dst, umma_desc_at(a, (kk >> 2) * (kBN * 128) + (kk & 3) * 32),
            umma_desc_at(b, (kk >> 2) * (kBM * 128) + (kk & 3) * 32), idesc, kk > 0 ? 1u : 0u);
}
// [128 x D] += (16-bit probabilities or dS of the step) x streamed tile. Each team writes back into the 32 score columns it has read:
// columns 0-31 of the step sit in [0,16) of the score block, 32-63 in [32,48).
template <int D, bool kBf16>
__device__ __forceinline__ void gradient(uint32_t lead, uint32_t acc, uint32_t a_tmem, uint32_t b_smem, bool fresh) {
  constexpr uint32_t idesc = umma_idesc(kBN, D, kBf16, false, true);  // B MN-major
  const uint64_t b = umma_desc_sw128(b_smem, kBM * 128, 1024);
#pragma unroll
  for (int s = 0; s < 4; ++s)
    umma_ts(lead, acc, a_tmem + (s < 2 ? s * 8 : 16 + s * 8), umma_desc_at(b, s * 2048), idesc, (fresh && s == 0) ? 0u : 1u);
}

// 32 (row, column) elements of a thread: x = scores, y = dP in, P and dS out, 16 bit. add(j): pair of addends, in log2 units;
// dsub(j): pair of D. Returns the sum of dS. Packed fp32x2 arithmetic, two columns per instruction.
template <bool kBf16, bool kP, class Add, class Sub>
__device__ __forceinline__ float softmax_step(const uint32_t (&x)[32], const uint32_t (&y)[32], float scale_log2, Add add, Sub dsub,
                                              uint32_t (&p16)[16], uint32_t (&ds16)[16]) {
  const float2 sc2 = make_float2(scale_log2, scale_log2), neg1 = make_float2(-1.f, -1.f);
  float2 part[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float2 e = __ffma2_rn(make_float2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])), sc2, add(j));
    const float2 pj = make_float2(fast_exp2(e.x), fast_exp2(e.y));
    const float2 ds = __fmul2_rn(pj, __ffma2_rn(dsub(j), neg1, make_float2(__uint_as_float(y[2 * j]), __uint_as_float(y[2 * j + 1]))));
    if (kP) {
      p16[j] = pack_16x2<kBf16>(pj.x, pj.y);
      part[j & 1] = __fadd2_rn(part[j & 1], ds);
    }
    ds16[j] = pack_16x2<kBf16>(ds.x, ds.y);
  }
  return (part[0].x + part[0].y) + (part[1].x + part[1].y);
}

// ---------------------------------------------------------------------------------------------------------------------
// Key pass: one tile of 128 keys of one (batch, kv head), every 64-row query tile of its range x every query head of the
// group, so that dK, dV and dBias leave the CTA already summed over the group (the reference writes per-query-head temporaries
// and reduces them on the host with at::sum_out, flash_api.cpp:970-983, :1027-1047).
// ---------------------------------------------------------------------------------------------------------------------
template <int D, bool kBf16, bool packed>
__device__ __forceinline__ void key_pass(const BwdRowsParams& p, unsigned char* smem, uint32_t tmem_base, const Bars& bar,
                                         const WaitCtl& ctl) {
  using L = SmemR<D>;
  using C = Cols<D, true>;
  constexpr uint32_t kAcc2 = C::kAcc + D;
  constexpr int kDpBufs = D == 128 ? 1 : 2;
  constexpr bool kX2Tmem = D == 64;  // V in tensor memory as well
  float* s_ld = reinterpret_cast<float*>(smem + L::kLdOff);
  uint16_t* s_heads = reinterpret_cast<uint16_t*>(smem + L::kHeadsOff);
  float* s_red = reinterpret_cast<float*>(smem + L::kRedOff);
  int* s_count = reinterpret_cast<int*>(smem + L::kMiscOff + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.h / p.h_k;
  const int Sq = p.seqlen_q, Sk = p.seqlen_k, NT = (Sk + kBN - 1) / kBN;
  const bool causal = p.is_causal != 0;
  // (query-range split, key tile), then kv head, then batch element. With more than one split the CTA covers the query tiles
  // [m_lo, M64) and leaves fp32 partials. The last query ranges, which causal masking never empties, run first.
  const int per = p.n_tiles * p.nsplit;
  const int item = blockIdx.x % per, n = item % p.n_tiles, split = p.nsplit - 1 - item / p.n_tiles;
  const int hk = blockIdx.x / per % p.h_k, b = blockIdx.x / per / p.h_k;
  const int M64_all = (Sq + kBM - 1) / kBM;
  const int m_chunk = (M64_all + p.nsplit - 1) / p.nsplit;
  const int m_lo = split * m_chunk;
  int M64 = min(M64_all, m_lo + m_chunk);
  // Compacted keys carry their original positions (ascending); the causal test then runs on positions.
  const int32_t* pos_row = nullptr;
  if (causal && p.key_pos) pos_row = p.key_pos + b * p.pos_batch_stride + (p.h_pos == p.h_k ? hk : 0) * p.pos_head_stride;
  int coff = pos_row ? p.causal_shift : Sk - Sq;
  // Packed sequences: the tile covers the keys [key0, key_end) of one of them, whose queries are [q_lo, q_hi).
  int key0 = n * kBN, key_end = Sk, q_lo = 0, q_hi = Sq, m_start = 0;
  if (pos_row) {
    const int64_t first = (static_cast<int64_t>(pos_row[n * kBN]) - coff) / kBM;
    m_start = static_cast<int>(max(static_cast<int64_t>(0), min(first, static_cast<int64_t>(M64))));
  } else if (causal) {
    m_start = max(0, (n * kBN - coff) / kBM);  // first query tile with a row that sees key n*128
  }
  if (packed) {
    const PackedTile t = packed_tile(p.seqs.cu_k, p.seqs.n, Sk, kBN, n);
    const int2 q = packed_range(p.seqs.cu_q, p.seqs.n, Sq, t.seq);
    key0 = t.begin + t.tile * kBN;
    key_end = t.end;
    q_lo = q.x;
    q_hi = key0 < key_end ? q.y : q.x;  // (an empty place has no queries)
    coff = key_end - q_hi;              // the last query sees the last key
    m_start = (causal ? max(q_lo, key0 - coff) : q_lo) / kBM;
    M64 = warp_uniform(q_lo < q_hi ? min(M64, (q_hi + kBM - 1) / kBM) : 0);
  }
  m_start = warp_uniform(max(m_start, m_lo));
  // The query heads for which the tile holds a kept key: all, none, or (a mask per query head) those in the list s_heads.
  const bool list = p.mask && p.h_mask == p.h && G > 1;
  if (warp == 2) {
    int cnt = 0;
    for (int g = 0; g < (list ? G : 1); ++g) {
      bool any = !p.mask;
      if (p.mask) {
        const int hm = p.h_mask == p.h ? hk * G + g : (p.h_mask == p.h_k ? hk : 0);
        const uint8_t* mrow = p.mask + b * p.mask_batch_stride + hm * p.mask_head_stride + n * kBN;
        for (int i = lane; i < kBN; i += 32) any = any || (n * kBN + i < Sk && mrow[i] != 0);
      }
      any = __any_sync(0xffffffffu, any);
      if (any) {
        if (list && lane == 0) s_heads[cnt] = static_cast<uint16_t>(g);
        ++cnt;
      }
    }
    if (lane == 0) *s_count = list ? cnt : (cnt ? G : 0);
  }
  __syncthreads();
  const int GA = warp_uniform(*s_count);
  const int n_steps = GA > 0 && M64 > m_start ? (M64 - m_start) * GA : 0;

  if (warp < 4) {
    FDMA_LIGHT_REGS();
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      if (lane == 0 && n_steps > 0) {
        mbar_arrive_expect_tx(bar.x_full, 2 * L::kTile);
#pragma unroll
        for (int kb = 0; kb < D / 64; ++kb)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int dst = kb * (kBN * 128) + r * (kBM * 128);
            tma_load_4d(smem + L::kXOff + dst, &p.tm_k, bar.x_full, kb * 64, hk, key0 + r * kBM, b);
            tma_load_4d(smem + L::kX2Off + dst, &p.tm_v, bar.x_full, kb * 64, hk, key0 + r * kBM, b);
          }
        int i = 0;
        bool ok = true;
        for (int m = m_start; m < M64 && ok; ++m) {
          for (int a = 0; a < GA; ++a, ++i) {
            const int stage = i % kStages;
            ok = mbar_wait(bar.st_empty + stage, ((i / kStages) & 1) ^ 1, ctl, kWaitStEmpty);
            if (!ok) break;
            mbar_arrive_expect_tx(bar.st_full + stage, 2 * L::kStep + 2 * kBM * 4);
            unsigned char* dst = smem + L::kStOff + stage * 2 * L::kStep;
            const int h = hk * G + (list ? s_heads[a] : a);
            const int64_t row0 = (static_cast<int64_t>(b) * p.h + h) * p.sq_r + m * kBM;
            bulk_load_1d(s_ld + stage * (2 * kBM), p.lse2 + row0, kBM * 4, bar.st_full + stage);
            bulk_load_1d(s_ld + stage * (2 * kBM) + kBM, p.dsum + row0, kBM * 4, bar.st_full + stage);
#pragma unroll
            for (int kb = 0; kb < D / 64; ++kb) {
              tma_load_4d(dst + kb * (kBM * 128), &p.tm_q, bar.st_full + stage, kb * 64, h, m * kBM, b);
              tma_load_4d(dst + L::kStep + kb * (kBM * 128), &p.tm_do, bar.st_full + stage, kb * 64, h, m * kBM, b);
            }
          }
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer (whole warp, uniform control flow; the issue wrappers are predicated on one lane) ----------------
      if (n_steps > 0) {
        const uint32_t lead = umma_leader(), st_addr = smem_u32(smem + L::kStOff);
        auto wait = [&](uint64_t* b_, int phase, int code) {
          const bool r = __all_sync(0xffffffffu, mbar_wait(b_, phase & 1, ctl, code));
          tc_fence_after_sync();
          return r;
        };
        // Packed sequences: rows of other sequences that came along in a query tile become zeros (LSE = +inf, D = 0), as TMA fills
        // them in at the end of a tensor; the sums over queries take them in. Only the first and the last query tile can hold such
        // rows: steps below `head_steps` and from `tail` on. (Foreign keys of the stationary tile only reach rows that are not stored.)
        const int head_steps = packed && m_start * kBM < q_lo ? GA : 0;
        const int tail = packed && M64 * kBM > q_hi ? n_steps - GA : n_steps;
        auto stage_ready = [&](int step) {
          const int stage = step % kStages;
          if (!wait(bar.st_full + stage, step / kStages, kWaitStFull)) return false;
          if (packed && (step < head_steps || step >= tail)) {
            const int q0 = (step < head_steps ? m_start : M64 - 1) * kBM;
            const int from = max(q_lo - q0, 0), to = min(q_hi - q0, kBM);
            unsigned char* st = smem + L::kStOff + stage * 2 * L::kStep;
            for (int t = 0; t < 2; ++t) {
              zero_tile_rows(st + t * L::kStep, D / 64, kBM * 128, 0, from);
              zero_tile_rows(st + t * L::kStep, D / 64, kBM * 128, to, kBM);
            }
            float* ld = s_ld + stage * (2 * kBM);
            for (int r = lane; r < kBM; r += 32)
              if (r < from || r >= to) {
                ld[r] = CUDART_INF_F;
                ld[kBM + r] = 0.f;
              }
            fence_proxy_async_smem();
            __threadfence_block();
            __syncwarp();
          }
          return true;
        };
        auto scores = [&](int step) {
          product_ts<D, kBf16>(lead, tmem_base + C::kS + (step & 1) * kBM, tmem_base + C::kX, st_addr + (step % kStages) * 2 * L::kStep);
        };
        auto dp = [&](int step) {
          const uint32_t dst = tmem_base + C::kDp + (kDpBufs == 2 ? (step & 1) * kBM : 0);
          const uint32_t g = st_addr + (step % kStages) * 2 * L::kStep + L::kStep;
          if constexpr (kX2Tmem) product_ts<D, kBf16>(lead, dst, tmem_base + C::kX2, g);
          else product_ss<D, kBf16>(lead, dst, smem_u32(smem + L::kX2Off), g);
        };
        int summed = 0, acc = 0;  // steps in the sums so far, sums before these
        auto gradients = [&](int step) {
          const bool fresh = summed == 0;
          if (!wait(bar.pds + (step & 1), step >> 1, kWaitPds)) return false;
          if (fresh && acc > 0 && !wait(bar.acc_free, acc - 1, kWaitAccFree)) return false;  // the sums before have been read
          const uint32_t st = st_addr + (step % kStages) * 2 * L::kStep, pc = tmem_base + C::kS + (step & 1) * kBM;
          gradient<D, kBf16>(lead, tmem_base + C::kAcc, pc, st + L::kStep, fresh);
          gradient<D, kBf16>(lead, tmem_base + kAcc2, pc + 16, st, fresh);
          umma_commit(lead, bar.st_empty + (step % kStages));
          if (++summed == kKeyFlush || step == n_steps - 1) {
            umma_commit(lead, bar.final_);
            summed = 0;
            ++acc;
          }
          return true;
        };
        bool ok = wait(bar.x_full, 0, kWaitX) && wait(bar.ready, 0, kWaitReady) && stage_ready(0);
        if (ok) {
          dp(0);
          scores(0);
          umma_commit(lead, bar.s_full + 0);
        }
        for (int i = 0; i < n_steps && ok; ++i) {
          // Scores of step i+1 take the place of P and dS of step i-1, behind its gradient products. dP: with two blocks as soon as
          // the teams have read that of step i-1, with one as soon as they have read that of step i.
          const bool more = i + 1 < n_steps;
          if (more) {
            ok = stage_ready(i + 1);
            if (ok && kDpBufs == 2) {
              if (i > 0) ok = wait(bar.dp_free + ((i - 1) & 1), (i - 1) >> 1, kWaitDpFree);
              if (ok) dp(i + 1);
            }
          }
          if (ok && i > 0) ok = gradients(i - 1);
          if (!ok) break;
          if (more) {
            scores(i + 1);
            if (kDpBufs == 1) {
              ok = wait(bar.dp_free + (i & 1), i >> 1, kWaitDpFree);
              if (!ok) break;
              dp(i + 1);
            }
            umma_commit(lead, bar.s_full + ((i + 1) & 1));
          }
        }
        if (ok) gradients(n_steps - 1);
      }
    }
  } else {
    FDMA_TEAM_REGS();
    // ---------------- softmax teams: thread = key ----------------
    const int half = (warp - 4) >> 2;
    const int krow = (warp & 3) * 32 + lane;  // key inside the tile == TMEM lane
    const int key = key0 + krow;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool key_ok = key < key_end;
    bool ok = true;
    if (n_steps > 0) {  // K (and V) into tensor memory
      ok = __all_sync(0xffffffffu, mbar_wait(bar.x_full, 0, ctl, kWaitX));
      if (ok) {
        if (half == 0) tile_row_to_tmem<D>(smem + L::kXOff, krow, tmem_base + lane_addr + C::kX);
        else if (kX2Tmem) tile_row_to_tmem<D>(smem + L::kX2Off, krow, tmem_base + lane_addr + C::kX2);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.ready);
      }
    }
    // value compared with q + coff in the causal test: the key's position
    // (clamped so that ckey - coff cannot overflow; padding slots hold INT_MAX and are masked out anyway)
    const int ckey = pos_row ? (key_ok ? min(pos_row[key], 0x3FFFFFFF) : 0x3FFFFFFF) : key;
    const int ckey_wmax = pos_row ? __shfl_sync(0xffffffffu, ckey, 31) : key0 + (warp & 3) * 32 + 31;
    // query rows [qlo, qhi) see this key, those of [qlo_max, qhi_min) all keys of the warp
    int qlo = causal ? ckey - coff : -0x7FFFFFFF, qhi = 0x7FFFFFFF;
    int qlo_max = causal ? ckey_wmax - coff : -0x7FFFFFFF, qhi_min = 0x7FFFFFFF;
    if (packed) {
      qlo = max(qlo, q_lo);
      qlo_max = max(qlo_max, q_lo);
      qhi = qhi_min = q_hi;
    }
    // addend of this key for query head h: bias in log2 units, -inf when the key is masked out (P = exp2(-inf) = 0 without any
    // per-element select). One value per thread for the whole CTA unless mask or bias differ between the heads of the group.
    auto addend = [&](int h) {
      const int hm = p.h_mask == p.h ? h : (p.h_mask == p.h_k ? hk : 0), hb = p.h_bias == p.h ? h : (p.h_bias == p.h_k ? hk : 0);
      if (!key_ok || (p.mask && p.mask[b * p.mask_batch_stride + hm * p.mask_head_stride + key] == 0)) return -CUDART_INF_F;
      if (!p.bias) return 0.f;
      return raw16_to_f<kBf16>(reinterpret_cast<const uint16_t*>(p.bias)[b * p.bias_batch_stride + hb * p.bias_head_stride + key]) * kLog2e;
    };
    // dV (team 0) and dK (team 1) out of tensor memory: 128 columns of this thread's key, in pieces that a warp stores in one go
    const uint32_t acc_addr = tmem_base + lane_addr + (half == 0 ? C::kAcc : kAcc2);
    const int rows = min(kBN, key_end - key0);
    float4* const sums = reinterpret_cast<float4*>(p.dkv_sums) +
                         ((((static_cast<int64_t>(half) * p.nsplit + split) * p.b + b) * p.h_k + hk) * (NT * kBN) + key0) * (D / 4) + krow;
    int moved = 0;  // how often
    auto move_sums = [&]() {
#pragma unroll 1  // (little code: it lies in the loop over the steps)
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        tmem_ld_x32(acc_addr + c * 32, r);
        tmem_wait_ld();
        if (c == D / 32 - 1) {  // the next sums may take their place
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar.acc_free);
        }
        if (key_ok) {
#pragma unroll
          for (int v4 = 0; v4 < 8; ++v4) {
            float4* dst = sums + (c * 8 + v4) * rows;
            const float4 x = make_float4(__uint_as_float(r[v4 * 4]), __uint_as_float(r[v4 * 4 + 1]), __uint_as_float(r[v4 * 4 + 2]),
                                         __uint_as_float(r[v4 * 4 + 3]));
            if (moved) red_add_f32x4(dst, x);
            else *dst = x;
          }
        }
        __syncwarp();
      }
      ++moved;
    };
    const bool hoist = G == 1 || ((!p.bias || p.h_bias != p.h) && (!p.mask || p.h_mask != p.h));
    float bv = addend(hk * G);
    float colsum = 0.f;  // dBias: sum of dS over the CTA's queries and heads
    // A dBias per query head of the group: one sum each, of this thread's own. (Both teams added to memory in every step, as they still do
    // for larger groups: 4 x 2048, 16 heads over 4, 565 -> 536 us; a bias shared by the batch, which takes one sum, 531 -> 511.)
    const bool per_head = p.dbias_mode == kDbAtomic && p.dbias_h == p.h && G > 1, db_smem = per_head && G <= kDbHeads;
    float* const s_db = reinterpret_cast<float*>(smem + L::kDbOff) + half * (kDbHeads * kBN) + krow;
    if (db_smem)
      for (int g = 0; g < G; ++g) s_db[g * kBN] = 0.f;
    const int db_b = p.dbias_b == 1 ? 0 : b;
    auto dbias_acc = [&](int h) { return p.dbias_acc + (static_cast<int64_t>(db_b) * p.dbias_h + h / (p.h / p.dbias_h)) * p.dbias_keys + key; };
    int m = m_start, a = 0;  // the step's query tile and place in the list of heads
    auto sums_ready = [&]() {
      ok = __all_sync(0xffffffffu, mbar_wait(bar.final_, moved & 1, ctl, kWaitFinal));
      tc_fence_after_sync();
      return ok;
    };
    int i = 0;
    while (true) {
      const int end = min(n_steps, (moved + 1) * kKeyFlush + 1);
      for (; i < end && ok; ++i) {
        const int h = hk * G + (list ? s_heads[a] : a);
        if (!hoist) bv = addend(h);
        ok = __all_sync(0xffffffffu, mbar_wait(bar.s_full + (i & 1), (i >> 1) & 1, ctl, kWaitS));
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t rs[32], rp[32], pk[16], dsk[16];
        const uint32_t s_col = tmem_base + lane_addr + C::kS + (i & 1) * kBM + half * 32;
        tmem_ld_x32(s_col, rs);
        tmem_ld_x32(tmem_base + lane_addr + C::kDp + (kDpBufs == 2 ? (i & 1) * kBM : 0) + half * 32, rp);
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.dp_free + (i & 1));  // the dP block may be overwritten from here on
        // LSE and D of the step's queries: bulk-copied under the stage barrier, which the MMA warp observed before it issued the
        // products this team has just waited for
        const float4* l4 = reinterpret_cast<const float4*>(s_ld + (i % kStages) * (2 * kBM) + half * 32);
        const float4* d4 = l4 + kBM / 4;
        const int q0 = m * kBM + half * 32;
        auto pair = [](const float4* v, int j) {
          const float4 x = v[j >> 1];
          return (j & 1) ? make_float2(x.z, x.w) : make_float2(x.x, x.y);
        };
        const float2 neg1 = make_float2(-1.f, -1.f);
        float sum;
        if (qlo_max > q0 || qhi_min < q0 + 32) {  // warp-uniform: some (query, key) of the warp is out of sight
          sum = softmax_step<kBf16, true>(rs, rp, p.scale_log2, [&](int j) {
            const int q = q0 + 2 * j;
            return __ffma2_rn(pair(l4, j), neg1, make_float2(q < qlo || q >= qhi ? -CUDART_INF_F : bv, q + 1 < qlo || q + 1 >= qhi ? -CUDART_INF_F : bv));
          }, [&](int j) { return pair(d4, j); }, pk, dsk);
        } else {
          const float2 bv2 = make_float2(bv, bv);
          sum = softmax_step<kBf16, true>(rs, rp, p.scale_log2, [&](int j) { return __ffma2_rn(pair(l4, j), neg1, bv2); },
                                          [&](int j) { return pair(d4, j); }, pk, dsk);
        }
        // back into the 32 columns just read: P^T pairs in the first 16, dS^T pairs in the last 16
        tmem_st_x16(s_col, pk);
        tmem_st_x16(s_col + 16, dsk);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.pds + (i & 1));
        if (!per_head) colsum += sum;
        else if (db_smem) s_db[(h - hk * G) * kBN] += sum;
        else if (key_ok) atomicAdd(dbias_acc(h), sum);
        if (++a == GA) {
          a = 0;
          ++m;
        }
      }
      if (!ok || n_steps <= (moved + 1) * kKeyFlush || !sums_ready()) break;
      move_sums();  // one step behind: the first product of the next sums follows that step
    }
    // ---------------- epilogue: dV (team 0) and dK (team 1), column-sum dBias ----------------
    if (p.dbias_mode != kDbNone) {
      if (half == 1) s_red[krow] = colsum;
      named_bar_sync(1, 256);
      if (p.dbias_mode == kDbAtomic) {
        if (half == 0 && key_ok && n_steps > 0) {
          if (!per_head) atomicAdd(dbias_acc(hk * G), colsum + s_red[krow]);
          if (db_smem)
            for (int g = 0; g < G; ++g) atomicAdd(dbias_acc(hk * G + g), s_db[g * kBN] + s_db[(kDbHeads + g) * kBN]);
        }
      } else if (half == 0 && key < p.dbias_keys) {
        // dbias_h == h_k: this CTA saw every query head of the group. dbias_h == h with a group of one: same.
        const float tot = colsum + s_red[krow];
        if (p.dkv_part)
          p.dbias_part[((static_cast<int64_t>(split) * p.b + b) * p.h_k + hk) * (NT * kBN) + key] = key_ok ? tot : 0.f;
        else
          reinterpret_cast<uint16_t*>(p.dbias)[b * p.dbias_batch_stride + hk * p.dbias_head_stride + key] = f_to_raw16<kBf16>(key_ok ? tot : 0.f);
      }
    }
    if (ok && n_steps > 0) sums_ready();
    if (ok) {
      const float mul = half == 0 ? 1.f : p.scale;
      uint16_t* dst = half == 0 ? reinterpret_cast<uint16_t*>(p.dv) + b * p.dv_batch_stride + hk * p.dv_head_stride +
                                      static_cast<int64_t>(min(key, Sk - 1)) * p.dv_row_stride
                                : reinterpret_cast<uint16_t*>(p.dk) + b * p.dk_batch_stride + hk * p.dk_head_stride +
                                      static_cast<int64_t>(min(key, Sk - 1)) * p.dk_row_stride;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        if (n_steps > 0) {
          tmem_ld_x32(acc_addr + c * 32, r);
          tmem_wait_ld();
          if (moved && key_ok) {
#pragma unroll
            for (int v4 = 0; v4 < 8; ++v4) {
              const float4 x = __ldcg(sums + (c * 8 + v4) * rows);  // (from L2, where they were added up)
              r[v4 * 4] = __float_as_uint(__uint_as_float(r[v4 * 4]) + x.x);
              r[v4 * 4 + 1] = __float_as_uint(__uint_as_float(r[v4 * 4 + 1]) + x.y);
              r[v4 * 4 + 2] = __float_as_uint(__uint_as_float(r[v4 * 4 + 2]) + x.z);
              r[v4 * 4 + 3] = __float_as_uint(__uint_as_float(r[v4 * 4 + 3]) + x.w);
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        if (p.dkv_part) {
          // fp32 partial: part[dv|dk][split][b][hk][key][d]
          if (packed && !key_ok) continue;  // (after the warp-wide load)
          float* part = p.dkv_part + ((((static_cast<int64_t>(half) * p.nsplit + split) * p.b + b) * p.h_k + hk) * (NT * kBN) + key) * D + c * 32;
#pragma unroll
          for (int v4 = 0; v4 < 8; ++v4)
            *reinterpret_cast<float4*>(part + v4 * 4) =
                make_float4(__uint_as_float(r[v4 * 4 + 0]) * mul, __uint_as_float(r[v4 * 4 + 1]) * mul,
                            __uint_as_float(r[v4 * 4 + 2]) * mul, __uint_as_float(r[v4 * 4 + 3]) * mul);
        } else if (key_ok) {
#pragma unroll
          for (int v4 = 0; v4 < 4; ++v4) {
            if (c * 32 + v4 * 8 >= p.d) break;
            uint4 o;
            o.x = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 0]) * mul, __uint_as_float(r[v4 * 8 + 1]) * mul);
            o.y = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 2]) * mul, __uint_as_float(r[v4 * 8 + 3]) * mul);
            o.z = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 4]) * mul, __uint_as_float(r[v4 * 8 + 5]) * mul);
            o.w = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 6]) * mul, __uint_as_float(r[v4 * 8 + 7]) * mul);
            *reinterpret_cast<uint4*>(dst + c * 32 + v4 * 8) = o;
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// Row pass: one tile of 128 query rows, `heads_per_cta` query heads one after the other (an item each). Barrier phases and ring
// positions carry over; the next item's Q and dO wait in shared memory when an item ends, its first score products are issued
// before the softmax teams store the item's dQ.
// ---------------------------------------------------------------------------------------------------------------------
template <int D, bool kBf16, bool packed>
__device__ __forceinline__ void row_pass(const BwdRowsParams& p, unsigned char* smem, uint32_t tmem_base, const Bars& bar,
                                         const WaitCtl& ctl) {
  using L = SmemR<D>;
  using C = Cols<D, false>;
  float* s_vec = reinterpret_cast<float*>(smem + L::kVecOff);
  uint32_t* s_bits_all = reinterpret_cast<uint32_t*>(smem + L::kBitsOff);
  volatile int* s_item = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 16);  // [2][4]: first 64-key tile, end of them, steps
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.h / p.h_k;
  const bool causal = p.is_causal != 0;
  const int hgroups = (p.h + p.heads_per_cta - 1) / p.heads_per_cta;
  const int idx = blockIdx.x - p.n_key_ctas;
  // the last query tiles, which see most keys, run first; heads that share K and V meet in L2
  const int per_tile = hgroups * p.b * p.ranges;
  int n = p.q_tiles - 1 - idx / per_tile;
  const int range = idx % per_tile / (hgroups * p.b);
  const int b = idx % (hgroups * p.b) / hgroups;
  const int h0 = idx % hgroups * p.heads_per_cta, h1 = min(p.h, h0 + p.heads_per_cta);
  int q0 = 0, sq = p.seqlen_q, k0 = 0, sk = p.seqlen_k;  // rows of the tile's sequence: first query and their number, keys
  if (packed) {
    const PackedTile t = packed_tile(p.seqs.cu_q, p.seqs.n, p.seqlen_q, kBN, n);
    const int2 keys = packed_range(p.seqs.cu_k, p.seqs.n, p.seqlen_k, t.seq);
    n = t.tile;
    q0 = t.begin;
    sq = t.end - t.begin;
    k0 = keys.x;
    sk = keys.y - keys.x;
    if (n * kBN >= sq) return;  // an empty place (the whole CTA agrees)
  }
  const int q_last = min(n * kBN + kBN, sq) - 1;  // last query row of the tile
  const bool use_pos = causal && p.key_pos;
  const int coff = use_pos ? p.causal_shift : sk - sq;
  auto pos_of = [&](int h) {
    return use_pos ? p.key_pos + b * p.pos_batch_stride + (p.h_pos == p.h_k ? h / G : 0) * p.pos_head_stride : nullptr;
  };
  auto mask_of = [&](int h) {
    return p.mask ? p.mask + b * p.mask_batch_stride + (p.h_mask == p.h ? h : (p.h_mask == p.h_k ? h / G : 0)) * p.mask_head_stride : nullptr;
  };
  const bool use_bits = p.mask != nullptr;
  // Steps of an item: the 64-key tiles [first, end) that hold a kept key
  auto next = [&](int m, int first, int end, const uint32_t* bits) {
    do ++m;
    while (use_bits && m < end && !((bits[(m - first) >> 5] >> ((m - first) & 31)) & 1u));
    return m;
  };

  if (warp < 4) {
    FDMA_LIGHT_REGS();
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      if (lane == 0) {
        int it = 0, xc = 0;
        bool ok = true;
        for (int ic = 0; h0 + ic < h1 && ok; ++ic) {
          const int h = h0 + ic, buf = ic & 1;
          ok = mbar_wait(bar.item_full + buf, (ic >> 1) & 1, ctl, kWaitItemFull);
          if (!ok) break;
          const int first = s_item[buf * 4], end = s_item[buf * 4 + 1], n_steps = s_item[buf * 4 + 2];
          const uint32_t* bits = s_bits_all + buf * (kMaxBits / 32);
          if (n_steps > 0) {
            ok = mbar_wait(bar.x_empty, (xc & 1) ^ 1, ctl, kWaitXEmpty);
            if (!ok) break;
            ++xc;
            mbar_arrive_expect_tx(bar.x_full, 2 * L::kTile);
#pragma unroll
            for (int kb = 0; kb < D / 64; ++kb)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const int dst = kb * (kBN * 128) + r * (kBM * 128), row = q0 + n * kBN + r * kBM;
                tma_load_4d(smem + L::kXOff + dst, &p.tm_q, bar.x_full, kb * 64, h, row, b);
                tma_load_4d(smem + L::kX2Off + dst, &p.tm_do, bar.x_full, kb * 64, h, row, b);
              }
          }
          for (int i = 0, m = next(first - 1, first, end, bits); i < n_steps; ++i, m = next(m, first, end, bits), ++it) {
            const int stage = it % kStages;
            ok = mbar_wait(bar.st_empty + stage, ((it / kStages) & 1) ^ 1, ctl, kWaitStEmpty);
            if (!ok) break;
            mbar_arrive_expect_tx(bar.st_full + stage, 2 * L::kStep);
            unsigned char* dst = smem + L::kStOff + stage * 2 * L::kStep;
#pragma unroll
            for (int kb = 0; kb < D / 64; ++kb) {
              tma_load_4d(dst + kb * (kBM * 128), &p.tm_k, bar.st_full + stage, kb * 64, h / G, k0 + m * kBM, b);
              tma_load_4d(dst + L::kStep + kb * (kBM * 128), &p.tm_v, bar.st_full + stage, kb * 64, h / G, k0 + m * kBM, b);
            }
          }
          mbar_arrive(bar.item_empty + buf);
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer ----------------
      const uint32_t lead = umma_leader(), st_addr = smem_u32(smem + L::kStOff);
      auto wait = [&](uint64_t* b_, int phase, int code) {
        const bool r = __all_sync(0xffffffffu, mbar_wait(b_, phase & 1, ctl, code));
        tc_fence_after_sync();
        return r;
      };
      auto scores = [&](int g) {
        product_ts<D, kBf16>(lead, tmem_base + C::kS + (g & 1) * kBM, tmem_base + C::kX, st_addr + (g % kStages) * 2 * L::kStep);
        umma_commit(lead, bar.s_full + (g & 1));  // covers dP of the step, issued before
      };
      auto dp = [&](int g) {
        product_ts<D, kBf16>(lead, tmem_base + C::kDp + (g & 1) * kBM, tmem_base + C::kX2, st_addr + (g % kStages) * 2 * L::kStep + L::kStep);
      };
      int g0 = 0, rc = 0, acc = 0;  // steps, items with steps, sums handed to the softmax teams so far
      bool ok = true;
      for (int ic = 0; h0 + ic < h1 && ok; ++ic) {
        const int buf = ic & 1;
        ok = wait(bar.item_full + buf, ic >> 1, kWaitItemFull);
        if (!ok) break;
        const int end = warp_uniform(s_item[buf * 4 + 1]), n_steps = warp_uniform(s_item[buf * 4 + 2]);
        // Packed sequences: K and V rows beyond the sequence, in its last tile, become zeros, as TMA fills them in at the end of a
        // tensor (zero probabilities alone would pass a NaN on).
        auto stage_ready = [&](int i) {
          const int stage = (g0 + i) % kStages;
          if (!wait(bar.st_full + stage, (g0 + i) / kStages, kWaitStFull)) return false;
          if (packed && i == n_steps - 1 && sk - (end - 1) * kBM < kBM) {
            unsigned char* st = smem + L::kStOff + stage * 2 * L::kStep;
            for (int t = 0; t < 2; ++t) zero_tile_rows(st + t * L::kStep, D / 64, kBM * 128, sk - (end - 1) * kBM, kBM);
            fence_proxy_async_smem();
            __syncwarp();
          }
          return true;
        };
        auto dq = [&](int i) {  // dQ += dS K of the item's step i
          const int g = g0 + i;
          const bool fresh = i % kFlush == 0;
          if (!wait(bar.pds + (g & 1), g >> 1, kWaitPds)) return false;
          if (fresh && acc > 0 && !wait(bar.acc_free, acc - 1, kWaitAccFree)) return false;  // the sums before have been read
          gradient<D, kBf16>(lead, tmem_base + C::kAcc, tmem_base + C::kS + (g & 1) * kBM, st_addr + (g % kStages) * 2 * L::kStep, fresh);
          umma_commit(lead, bar.st_empty + (g % kStages));
          if (i % kFlush == kFlush - 1 || i == n_steps - 1) {
            umma_commit(lead, bar.final_);
            ++acc;
          }
          return true;
        };
        if (n_steps > 0) {
          ok = wait(bar.ready, rc++, kWaitReady) && stage_ready(0);
          if (!ok) break;
          dp(g0);  // (every step of the item before has been handed over: its dP has been read)
          scores(g0);
        }
        for (int i = 0; i < n_steps && ok; ++i) {
          const int g = g0 + i;
          if (i + 1 < n_steps) {  // dP of the next step as soon as that of the step before has been read
            ok = stage_ready(i + 1);
            if (ok && i > 0) ok = wait(bar.dp_free + ((g - 1) & 1), (g - 1) >> 1, kWaitDpFree);
            if (!ok) break;
            dp(g + 1);
          }
          if (i > 0) ok = dq(i - 1);
          if (!ok) break;
          if (i + 1 < n_steps) scores(g + 1);  // in the place of dS of the step before
        }
        if (ok && n_steps > 0) ok = dq(n_steps - 1);
        if (!ok) break;
        g0 += n_steps;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.item_empty + buf);
      }
    } else if (warp == 2) {
      // addend (bias in log2 units, or -inf where masked out) and position of the step's 64 keys, two per lane
      int vi = 0;
      bool ok = true;
      for (int ic = 0; h0 + ic < h1 && ok; ++ic) {
        const int h = h0 + ic, buf = ic & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar.item_full + buf, (ic >> 1) & 1, ctl, kWaitItemFull));
        if (!ok) break;
        const int first = s_item[buf * 4], end = s_item[buf * 4 + 1], n_steps = s_item[buf * 4 + 2];
        const uint32_t* bits = s_bits_all + buf * (kMaxBits / 32);
        const uint8_t* mrow = mask_of(h);
        const uint16_t* brow = p.bias ? reinterpret_cast<const uint16_t*>(p.bias) + b * p.bias_batch_stride +
                                            (p.h_bias == p.h ? h : (p.h_bias == p.h_k ? h / G : 0)) * p.bias_head_stride : nullptr;
        const int32_t* pos_row = pos_of(h);
        for (int i = 0, m = next(first - 1, first, end, bits); i < n_steps; ++i, m = next(m, first, end, bits), ++vi) {
          const int k = m * kBM + lane * 2;
          const uint32_t mb = mrow ? *reinterpret_cast<const uint16_t*>(mrow + k) : 0x0101u;
          const uint32_t bb = brow ? *reinterpret_cast<const uint32_t*>(brow + k) : 0u;
          const float2 add = make_float2(k < sk && (mb & 0xFFu) ? raw16_to_f<kBf16>(static_cast<uint16_t>(bb & 0xFFFFu)) * kLog2e : -CUDART_INF_F,
                                         k + 1 < sk && (mb >> 8) ? raw16_to_f<kBf16>(static_cast<uint16_t>(bb >> 16)) * kLog2e : -CUDART_INF_F);
          int2 pos = make_int2(k, k + 1);
          if (pos_row) pos = make_int2(k < sk ? pos_row[k] : 0x7FFFFFFF, k + 1 < sk ? pos_row[k + 1] : 0x7FFFFFFF);
          const int slot = vi % kVecSlots;
          ok = __all_sync(0xffffffffu, mbar_wait(bar.vec_empty + slot, ((vi / kVecSlots) & 1) ^ 1, ctl, kWaitVecEmpty));
          if (!ok) break;
          float* dst = s_vec + slot * (2 * kBM);
          reinterpret_cast<float2*>(dst)[lane] = add;
          reinterpret_cast<int2*>(dst + kBM)[lane] = pos;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar.vec_full + slot);
        }
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(bar.item_empty + buf);
      }
    } else {
      // which 64-key tiles each item works on, one item ahead of the other roles
      bool ok = true;
      for (int ic = 0; h0 + ic < h1 && ok; ++ic) {
        const int h = h0 + ic, buf = ic & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(bar.item_empty + buf, ((ic >> 1) & 1) ^ 1, ctl, kWaitItemEmpty));
        if (!ok) break;
        int vis = sk;  // keys in sight of the tile's last row
        if (use_pos) {
          // 32-way search in the ascending positions for the first one beyond the limit
          const int32_t* pos_row = pos_of(h);
          const int64_t lim = static_cast<int64_t>(q_last) + coff;
          int lo = 0, len = sk;  // the answer lies in [lo, lo + len]
          while (len > 0) {
            const int step = (len + 31) / 32;
            const int i = min(lo + (lane + 1) * step - 1, lo + len - 1);
            const int cnt = __popc(__ballot_sync(0xffffffffu, static_cast<int64_t>(pos_row[i]) <= lim));  // a prefix of the lanes
            const int new_lo = min(lo + cnt * step, lo + len);
            len = cnt == 32 ? 0 : min(step - 1, lo + len - new_lo);
            lo = new_lo;
          }
          vis = lo;
        } else if (causal) {
          vis = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(sk), static_cast<int64_t>(q_last) + coff + 1)));
        }
        const int n_sub = (vis + kBM - 1) / kBM, chunk = (n_sub + p.ranges - 1) / p.ranges;
        const int first = min(range * chunk, n_sub), end = min(first + chunk, n_sub);
        int n_steps = end - first;
        if (use_bits) {
          const uint8_t* mrow = mask_of(h);
          uint32_t* bits = s_bits_all + buf * (kMaxBits / 32);
          n_steps = 0;
          for (int w = 0; first + w * 32 < end; ++w) {  // a lane per tile
            const int m = first + w * 32 + lane;
            uint32_t any = 0;
            if (m < end) {
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const uint4 v = *reinterpret_cast<const uint4*>(mrow + m * kBM + c * 16);
                uint32_t x[4] = {v.x, v.y, v.z, v.w};
                if (m * kBM + c * 16 + 16 > sk) {  // ragged end: drop keys beyond the last
#pragma unroll
                  for (int e = 0; e < 16; ++e)
                    if (m * kBM + c * 16 + e >= sk) x[e >> 2] &= ~(0xFFu << ((e & 3) * 8));
                }
                any |= x[0] | x[1] | x[2] | x[3];
              }
            }
            const uint32_t word = __ballot_sync(0xffffffffu, any != 0);
            if (lane == 0) bits[w] = word;
            n_steps += __popc(word);
          }
        }
        if (lane == 0) {
          s_item[buf * 4] = first;
          s_item[buf * 4 + 1] = end;
          s_item[buf * 4 + 2] = n_steps;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.item_full + buf);
      }
    }
  } else {
    FDMA_TEAM_REGS();
    // ---------------- softmax teams: thread = query row ----------------
    const int half = (warp - 4) >> 2;
    const int trow = (warp & 3) * 32 + lane;  // row inside the tile == TMEM lane
    const int row = n * kBN + trow, warp_row = n * kBN + (warp & 3) * 32;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool row_ok = row < sq;
    // last position this row (and the warp's first row) sees
    auto clamp = [](int64_t x) { return static_cast<int>(max(static_cast<int64_t>(-1), min(x, static_cast<int64_t>(0x7FFFFFFE)))); };
    const int qlim = causal ? clamp(static_cast<int64_t>(row) + coff) : 0x7FFFFFFE;
    const int qlim_wmin = causal ? clamp(static_cast<int64_t>(warp_row) + coff) : 0x7FFFFFFE;
    const int row_g = q0 + min(row, sq - 1);  // row in the tensors
    constexpr int kHalfCols = D / 2;          // columns of dQ each team takes out
    int g0 = 0, xc = 0, sums = 0;  // steps, items with steps, sums received so far
    int todo = -1, todo_steps = 0;  // head whose dQ is to be stored
    bool ok = true;
    float2 acc[kHalfCols / 2];  // dQ of this thread's row and team
#pragma unroll
    for (int j = 0; j < kHalfCols / 2; ++j) acc[j] = make_float2(0.f, 0.f);
    auto load_sums = [&](uint32_t (&r)[kHalfCols / 32][32]) {
#pragma unroll
      for (int c = 0; c < kHalfCols / 32; ++c) tmem_ld_x32(tmem_base + lane_addr + C::kAcc + half * kHalfCols + c * 32, r[c]);
    };
    auto add_sums = [&](const uint32_t (&r)[kHalfCols / 32][32]) {
      ++sums;
#pragma unroll
      for (int c = 0; c < kHalfCols / 32; ++c)
#pragma unroll
        for (int j = 0; j < 16; ++j)
          acc[c * 16 + j] = __fadd2_rn(acc[c * 16 + j], make_float2(__uint_as_float(r[c][2 * j]), __uint_as_float(r[c][2 * j + 1])));
    };
    auto sums_taken = [&]() {  // after tmem_wait_ld: the accumulator may be overwritten from here on
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar.acc_free);
    };
    auto collect = [&]() {  // the oldest sums not yet taken
      ok = __all_sync(0xffffffffu, mbar_wait(bar.final_, sums & 1, ctl, kWaitFinal));
      if (!ok) return;
      tc_fence_after_sync();
      uint32_t r[kHalfCols / 32][32];
      load_sums(r);
      tmem_wait_ld();
      sums_taken();
      add_sums(r);
    };
    auto store = [&](int h, int n_steps) {  // dQ of a finished item
      if (n_steps > 0) collect();
      if (!ok) return;
      if (p.ranges > 1) {  // a partial sum
        float4* part = reinterpret_cast<float4*>(
            p.dq_part + (((static_cast<int64_t>(range) * p.b + b) * p.h + h) * p.seqlen_q + row_g) * D + half * kHalfCols);
#pragma unroll
        for (int v = 0; v < kHalfCols / 4; ++v)
          if (row_ok) part[v] = make_float4(acc[v * 2].x, acc[v * 2].y, acc[v * 2 + 1].x, acc[v * 2 + 1].y);
      }
      uint16_t* dst = reinterpret_cast<uint16_t*>(p.dq) + b * p.dq_batch_stride + h * p.dq_head_stride +
                      static_cast<int64_t>(row_g) * p.dq_row_stride + half * kHalfCols;
#pragma unroll
      for (int v = 0; v < kHalfCols / 8; ++v) {
        if (p.ranges > 1 || !row_ok || half * kHalfCols + v * 8 >= p.d) break;
        uint4 o;
        o.x = pack_16x2<kBf16>(acc[v * 4].x * p.scale, acc[v * 4].y * p.scale);
        o.y = pack_16x2<kBf16>(acc[v * 4 + 1].x * p.scale, acc[v * 4 + 1].y * p.scale);
        o.z = pack_16x2<kBf16>(acc[v * 4 + 2].x * p.scale, acc[v * 4 + 2].y * p.scale);
        o.w = pack_16x2<kBf16>(acc[v * 4 + 3].x * p.scale, acc[v * 4 + 3].y * p.scale);
        *reinterpret_cast<uint4*>(dst + v * 8) = o;
      }
#pragma unroll
      for (int j = 0; j < kHalfCols / 2; ++j) acc[j] = make_float2(0.f, 0.f);
    };
    for (int ic = 0; ok; ++ic) {
      const int h = h0 + ic, buf = ic & 1;
      int n_steps = 0;
      float lse = CUDART_INF_F, dsum = 0.f;
      if (h < h1) {
        if (row_ok) {
          const int64_t idx2 = (static_cast<int64_t>(b) * p.h + h) * p.sq_r + row_g;
          lse = p.lse2[idx2];
          dsum = p.dsum[idx2];
        }
        ok = __all_sync(0xffffffffu, mbar_wait(bar.item_full + buf, (ic >> 1) & 1, ctl, kWaitItemFull));
        if (!ok) break;
        n_steps = s_item[buf * 4 + 2];
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.item_empty + buf);
        if (n_steps > 0) {
          // Q (team 0) and dO (team 1) into tensor memory; the last products that read what is there were those of the last step,
          // which every warp has waited for
          ok = __all_sync(0xffffffffu, mbar_wait(bar.x_full, xc & 1, ctl, kWaitX));
          if (!ok) break;
          ++xc;
          tc_fence_after_sync();
          if (half == 0) tile_row_to_tmem<D>(smem + L::kXOff, trow, tmem_base + lane_addr + C::kX);
          else tile_row_to_tmem<D>(smem + L::kX2Off, trow, tmem_base + lane_addr + C::kX2);
          tmem_wait_st();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(bar.ready);
            mbar_arrive(bar.x_empty);
          }
        }
      }
      if (todo >= 0) store(todo, todo_steps);
      if (h >= h1 || !ok) break;
      todo = h;
      todo_steps = n_steps;
      const float2 nlse2 = make_float2(-lse, -lse), dsum2 = make_float2(dsum, dsum);
      for (int i = 0; i < n_steps && ok; ++i) {
        const int g = g0 + i, slot = g % kVecSlots;
        ok = __all_sync(0xffffffffu, mbar_wait(bar.vec_full + slot, (g / kVecSlots) & 1, ctl, kWaitVecFull));
        if (!ok) break;
        ok = __all_sync(0xffffffffu, mbar_wait(bar.s_full + (g & 1), (g >> 1) & 1, ctl, kWaitS));
        if (!ok) break;
        tc_fence_after_sync();
        uint32_t rs[32], rp[32], dsk[16];
        const uint32_t s_col = tmem_base + lane_addr + C::kS + (g & 1) * kBM + half * 32;
        // Sums that ended two steps ago: their product was issued before the scores just waited for, so it is complete; the next
        // one, which starts new sums, waits for this.
        if (i > kFlush && i % kFlush == 1 % kFlush) {
          uint32_t r[kHalfCols / 32][32];
          load_sums(r);
          tmem_wait_ld();
          sums_taken();
          add_sums(r);
        }
        tmem_ld_x32(s_col, rs);
        tmem_ld_x32(tmem_base + lane_addr + C::kDp + (g & 1) * kBM + half * 32, rp);
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar.dp_free + (g & 1));
        const float4* v4 = reinterpret_cast<const float4*>(s_vec + slot * (2 * kBM) + half * 32);
        const int* pos = reinterpret_cast<const int*>(v4 + kBM / 4);
        auto pair = [&](int j) {
          const float4 x = v4[j >> 1];
          return __fadd2_rn((j & 1) ? make_float2(x.z, x.w) : make_float2(x.x, x.y), nlse2);
        };
        auto d2 = [&](int) { return dsum2; };
        if (causal && pos[31] > qlim_wmin) {  // warp-uniform: some (row, key) of the warp is out of sight
          softmax_step<kBf16, false>(rs, rp, p.scale_log2, [&](int j) {
            float2 add = pair(j);
            if (pos[2 * j] > qlim) add.x = -CUDART_INF_F;
            if (pos[2 * j + 1] > qlim) add.y = -CUDART_INF_F;
            return add;
          }, d2, dsk, dsk);
        } else {
          softmax_step<kBf16, false>(rs, rp, p.scale_log2, pair, d2, dsk, dsk);
        }
        tmem_st_x16(s_col, dsk);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar.pds + (g & 1));
          mbar_arrive(bar.vec_empty + slot);
        }
      }
      if (ok && n_steps > 1 && (n_steps - 1) % kFlush == 0) collect();  // (those of the step before the last)
      g0 += n_steps;
    }
  }
}

template <int D, bool kBf16, bool packed>
__global__ void __launch_bounds__(kThreads, 1) bwd_rows_kernel(const __grid_constant__ BwdRowsParams p) {
  using L = SmemR<D>;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = align_smem_1024(smem_dyn);
  const Bars bar(reinterpret_cast<uint64_t*>(smem + L::kBarOff));
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + L::kMiscOff);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const WaitCtl ctl{s_abort, p.status};
  if (tid == 0) {
    *s_abort = 0;
    mbar_init(bar.x_full, 1);
    mbar_init(bar.x_empty, 8);
    mbar_init(bar.ready, 8);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bar.st_full + i, 1);
      mbar_init(bar.st_empty + i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar.s_full + i, 1);
      mbar_init(bar.dp_free + i, 8);  // one arrival per softmax warp
      mbar_init(bar.pds + i, 8);
      mbar_init(bar.item_full + i, 1);
      mbar_init(bar.item_empty + i, 11);  // producer, MMA issuer, vector warp, softmax warps
    }
    for (int i = 0; i < kVecSlots; ++i) {
      mbar_init(bar.vec_full + i, 1);
      mbar_init(bar.vec_empty + i, 8);
    }
    mbar_init(bar.final_, 1);
    mbar_init(bar.acc_free, 8);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(s_tmem, 512);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&p.tm_q);
    prefetch_tmap(&p.tm_do);
    prefetch_tmap(&p.tm_k);
    prefetch_tmap(&p.tm_v);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*s_tmem);
  if (blockIdx.x < static_cast<unsigned>(p.n_key_ctas)) key_pass<D, kBf16, packed>(p, smem, tmem_base, bar, ctl);
  else row_pass<D, kBf16, packed>(p, smem, tmem_base, bar, ctl);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// (row tile, head, batch element) of a call: the CTAs of the row pass at one range and head each
int64_t row_tiles(const fdma_fwd_params& p) { return static_cast<int64_t>((p.seqlen_q + kBN - 1) / kBN) * p.h * p.b; }

struct RowsPlan {
  int D, sq_r, nsplit, dbias_mode;
  int ranges;  // key ranges per row-pass tile
  bool part;  // dK, dV (and column sums) leave the kernel as fp32 partials
  size_t lse2_off, dsum_off, dq_off, dbias_off, sums_off, part_off, dbpart_off, total;
};

// Query-range splits per key tile: one CTA per SM, as long as a split keeps 32 steps, and on to two per SM while it keeps 160. The row pass,
// whose many short CTAs run last, evens out what unequal key CTAs leave; every split writes and reads fp32 partials of its key tile. (What
// the tensor core sums up has its own bound, kKeyFlush.) Backward in us, at least one / two CTAs per SM: 8192 x 16 heads over 4, causal
// 847 / 880, plain 4096 x 32 over 8 465 / 507, 8192 packed tokens 365 / 409, 4 x 2048, 512 gathered keys, d = 64 251 / 267; but 32768 over 2048
// gathered keys (splits of 1024 / 683 steps) 2100 / 2063, 8192 over 2048 (256 / 171 steps) 613 / 598.
int pick_nsplit(const fdma_fwd_params& p) {
  const int64_t ctas = static_cast<int64_t>((p.seqlen_k + kBN - 1) / kBN) * p.h_k * p.b;
  const int64_t steps = static_cast<int64_t>((p.seqlen_q + kBM - 1) / kBM) * (p.h / p.h_k);
  if (ctas >= sm_count()) return 1;
  const int64_t one = std::min((sm_count() + ctas - 1) / ctas, steps / 32), two = std::min((2 * sm_count() + ctas - 1) / ctas, steps / 160);
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(std::max(one, two), 64)));
}

// Key ranges per row-pass tile, where there are few rows and at least four times as many keys: else a few CTAs walk all keys one tile after
// the other. Of the calls this file takes (see bwd_rows_taken) half a CTA per SM, so that both passes fit in one wave, with eight steps
// each: 128 queries over 4096 keys, 8 heads over 2 61 -> 28 us (29 in a single pass), over 2048 34 -> 27 (29), over 1024 (not cut) 25.
// The fp32 partials are added up in one order by bwd_finish_kernel.
int pick_ranges(const fdma_fwd_params& p) {
  const int64_t ctas = row_tiles(p), steps = (p.seqlen_k + kBM - 1) / kBM;
  if (p.seqlen_k < 4ll * p.seqlen_q || steps < 32 || ctas > sm_count() / 8) return 1;
  return static_cast<int>(std::min<int64_t>(sm_count() / 2 / ctas, steps / 8));
}

// Query heads a row-pass CTA works on, one after the other: as many as leave six CTAs per SM, so that set-up and the first loads
// of a CTA are paid once for several items and the last ones still even out. 32768 queries, 32 heads, backward in us with one head / 12 / 6 / 3
// CTAs per SM: 2048 gathered keys 2265 / 2077 / 2057 / 2058, 128 keys 808 / 654 / 651 / 656; three per SM also 4 x 2048 at head dim 64 265 -> 251,
// but 16384 x 8 heads at head dim 64 2523 -> 2690.
int pick_heads_per_cta(int64_t tiles, int h) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(std::min(h, 16), tiles * h / (6 * sm_count()))));
}

// Keys of the fp32 buffer of the atomic dBias mode: those of the tensor, or with gathered keys the gathered ones.
int atomic_keys(const fdma_bwd_params& bp) { return bp.scatter_pos ? bp.f.seqlen_k : bp.dbias_keys; }

RowsPlan plan(const fdma_bwd_params& bp) {
  const fdma_fwd_params& p = bp.f;
  RowsPlan pl;
  pl.D = tile_head_dim(p.d);
  pl.sq_r = static_cast<int>(round_up(p.seqlen_q, kBM));
  if (!bp.dbias) pl.dbias_mode = kDbNone;
  else if (bp.dbias_b == p.b && (bp.dbias_h == p.h_k || (bp.dbias_h == p.h && p.h == p.h_k))) pl.dbias_mode = kDbColsum;
  else pl.dbias_mode = kDbAtomic;
  size_t o = 0;
  const size_t rows = static_cast<size_t>(p.b) * p.h * pl.sq_r;
  pl.lse2_off = o; o += align256(rows * 4);
  pl.dsum_off = o; o += align256(rows * 4);
  pl.ranges = pick_ranges(p);
  pl.dq_off = o;
  if (pl.ranges > 1) o += align256(static_cast<size_t>(pl.ranges) * p.b * p.h * p.seqlen_q * pl.D * 4);
  pl.dbias_off = o;
  if (pl.dbias_mode == kDbAtomic) o += align256(static_cast<size_t>(bp.dbias_b) * bp.dbias_h * atomic_keys(bp) * 4);
  pl.nsplit = pick_nsplit(p);
  pl.sums_off = o;
  const int64_t m_tiles = (p.seqlen_q + kBM - 1) / kBM;
  if ((m_tiles + pl.nsplit - 1) / pl.nsplit * (p.h / p.h_k) > kKeyFlush)
    o += align256(static_cast<size_t>(2) * pl.nsplit * p.b * p.h_k * round_up(p.seqlen_k, kBN) * pl.D * 4);
  pl.part = pl.nsplit > 1 || bp.scatter_pos != nullptr;
  pl.part_off = pl.dbpart_off = o;
  if (pl.part) {
    const size_t keys_r = round_up(p.seqlen_k, kBN);
    o += align256(static_cast<size_t>(2) * pl.nsplit * p.b * p.h_k * keys_r * pl.D * 4);
    pl.dbpart_off = o;
    if (pl.dbias_mode == kDbColsum) o += align256(static_cast<size_t>(pl.nsplit) * p.b * p.h_k * keys_r * 4);
  }
  pl.total = o;
  return pl;
}

template <int D, bool kBf16>
int launch(const fdma_bwd_params& bp, const RowsPlan& pl, const PackedSeqs& seqs, cudaStream_t stream) {
  using L = SmemR<D>;
  const fdma_fwd_params& p = bp.f;
  if (!p.workspace || p.workspace_bytes < pl.total) return FDMA_ERR_WORKSPACE;
  char* ws = static_cast<char*>(p.workspace);
  BwdRowsParams kp;
  auto encode = [&](CUtensorMap* tm, const void* base, int heads, int rows, int64_t sb, int64_t sr, int64_t sh) {
    if (heads == 1) sh = p.d;
    if (rows == 1) sr = static_cast<int64_t>(heads) * p.d;
    if (p.b == 1) sb = static_cast<int64_t>(rows) * heads * p.d;
    const uint64_t dims[4] = {static_cast<uint64_t>(p.d), static_cast<uint64_t>(heads), static_cast<uint64_t>(rows),
                              static_cast<uint64_t>(p.b)};
    const uint64_t str[3] = {static_cast<uint64_t>(sh) * 2, static_cast<uint64_t>(sr) * 2,
                             static_cast<uint64_t>(sb) * 2};
    const uint32_t box[4] = {64, 1, static_cast<uint32_t>(kBM), 1};
    return encode_tmap_4d(tm, base, 2, dims, str, box);
  };
  int st = encode(&kp.tm_q, p.q, p.h, p.seqlen_q, p.q_batch_stride, p.q_row_stride, p.q_head_stride);
  if (st) return st;
  st = encode(&kp.tm_do, bp.dout, p.h, p.seqlen_q, bp.do_batch_stride, bp.do_row_stride, bp.do_head_stride);
  if (st) return st;
  st = encode(&kp.tm_k, p.k, p.h_k, p.seqlen_k, p.k_batch_stride, p.k_row_stride, p.k_head_stride);
  if (st) return st;
  st = encode(&kp.tm_v, p.v, p.h_k, p.seqlen_k, p.v_batch_stride, p.v_row_stride, p.v_head_stride);
  if (st) return st;

  float* lse2 = reinterpret_cast<float*>(ws + pl.lse2_off);
  float* dsum = reinterpret_cast<float*>(ws + pl.dsum_off);
  {
    BwdPrepArgs a;
    a.out = p.out; a.dout = bp.dout; a.lse = p.lse; a.lse2 = lse2; a.dsum = dsum; a.dq_acc = nullptr;
    a.b = p.b; a.h = p.h; a.sq = p.seqlen_q; a.sq_r = pl.sq_r; a.d = p.d; a.acc_bytes = 0;
    a.o_sb = p.o_batch_stride; a.o_sr = p.o_row_stride; a.o_sh = p.o_head_stride;
    a.do_sb = bp.do_batch_stride; a.do_sr = bp.do_row_stride; a.do_sh = bp.do_head_stride;
    st = launch_bwd_prep(a, D, kBf16, stream);
    if (st) return st;
    st = export_softmax_d(bp, dsum, pl.sq_r, stream);
    if (st) return st;
  }
  cudaError_t e = cudaSuccess;
  kp.dbias_acc = nullptr;
  if (pl.dbias_mode == kDbAtomic) {
    kp.dbias_acc = reinterpret_cast<float*>(ws + pl.dbias_off);
    e = cudaMemsetAsync(kp.dbias_acc, 0, static_cast<size_t>(bp.dbias_b) * bp.dbias_h * atomic_keys(bp) * 4, stream);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  kp.mask = static_cast<const uint8_t*>(p.mask);
  kp.bias = p.bias;
  kp.lse2 = lse2;
  kp.dsum = dsum;
  kp.dq = bp.dq;
  kp.dk = bp.dk;
  kp.dv = bp.dv;
  kp.dbias = bp.dbias;
  kp.dq_part = reinterpret_cast<float*>(ws + pl.dq_off);
  kp.dkv_sums = reinterpret_cast<float*>(ws + pl.sums_off);
  kp.dkv_part = pl.part ? reinterpret_cast<float*>(ws + pl.part_off) : nullptr;
  kp.dbias_part = reinterpret_cast<float*>(ws + pl.dbpart_off);
  kp.status = kernel_status_ptr();
  if (!kp.status) return FDMA_ERR_DRIVER;
  kp.mask_batch_stride = p.mask_batch_stride; kp.mask_head_stride = p.mask_head_stride;
  kp.bias_batch_stride = p.bias_batch_stride; kp.bias_head_stride = p.bias_head_stride;
  kp.dq_batch_stride = bp.dq_batch_stride; kp.dq_row_stride = bp.dq_row_stride; kp.dq_head_stride = bp.dq_head_stride;
  kp.dk_batch_stride = bp.dk_batch_stride; kp.dk_row_stride = bp.dk_row_stride; kp.dk_head_stride = bp.dk_head_stride;
  kp.dv_batch_stride = bp.dv_batch_stride; kp.dv_row_stride = bp.dv_row_stride; kp.dv_head_stride = bp.dv_head_stride;
  kp.dbias_batch_stride = bp.dbias_batch_stride; kp.dbias_head_stride = bp.dbias_head_stride;
  kp.b = p.b; kp.seqlen_q = p.seqlen_q; kp.seqlen_k = p.seqlen_k; kp.sq_r = pl.sq_r; kp.h = p.h; kp.h_k = p.h_k; kp.d = p.d;
  kp.h_mask = p.h_mask; kp.h_bias = p.h_bias;
  kp.dbias_b = bp.dbias_b; kp.dbias_h = bp.dbias_h;
  kp.dbias_keys = bp.scatter_pos ? p.seqlen_k : bp.dbias_keys;
  kp.dbias_mode = pl.dbias_mode;
  kp.is_causal = p.is_causal;
  kp.key_pos = p.key_pos;
  kp.pos_batch_stride = p.key_pos_batch_stride; kp.pos_head_stride = p.key_pos_head_stride;
  kp.h_pos = p.h_pos; kp.causal_shift = p.causal_shift;
  kp.seqs = seqs;
  kp.n_tiles = seqs.cu_q ? packed_slots(p.seqlen_k, seqs.n, kBN) : (p.seqlen_k + kBN - 1) / kBN;
  kp.q_tiles = seqs.cu_q ? packed_slots(p.seqlen_q, seqs.n, kBN) : (p.seqlen_q + kBN - 1) / kBN;
  kp.nsplit = pl.nsplit;
  kp.ranges = seqs.cu_q ? 1 : pl.ranges;
  kp.heads_per_cta = pick_heads_per_cta(static_cast<int64_t>(kp.q_tiles) * p.b * kp.ranges, p.h);
  kp.scale_log2 = p.softmax_scale * kLog2e;
  kp.scale = p.softmax_scale;

  auto kern = seqs.cu_q ? bwd_rows_kernel<D, kBf16, true> : bwd_rows_kernel<D, kBf16, false>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kAlloc);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int64_t key_ctas = static_cast<int64_t>(kp.n_tiles) * pl.nsplit * p.h_k * p.b;
  const int64_t ctas = key_ctas + static_cast<int64_t>(kp.q_tiles) * p.b * kp.ranges * ((p.h + kp.heads_per_cta - 1) / kp.heads_per_cta);
  if (ctas > 0x7FFFFFFF) return FDMA_ERR_TOO_LARGE;
  kp.n_key_ctas = static_cast<int>(key_ctas);
  cudaEvent_t ev0, ev1;
  take_timing_events(&ev0, &ev1);
  if (ev0) cudaEventRecord(ev0, stream);
  kern<<<static_cast<unsigned>(ctas), kThreads, L::kAlloc, stream>>>(kp);
  if (ev1) cudaEventRecord(ev1, stream);
  e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);

  BwdFinishArgs f = {};
  f.b = p.b; f.h = p.h; f.sq = p.seqlen_q; f.sq_r = pl.sq_r; f.d = p.d; f.D = D;
  f.h_k = p.h_k; f.keys_r = static_cast<int>(round_up(p.seqlen_k, kBN));
  f.rows_out = bp.scatter_pos ? bp.scatter_rows : p.seqlen_k;
  f.scale = p.softmax_scale;
  if (kp.ranges > 1) {
    f.dq_acc = kp.dq_part; f.dq_nsplit = kp.ranges;
    f.dq_split_stride = static_cast<int64_t>(p.b) * p.h * p.seqlen_q * D;
    f.dq = bp.dq; f.dq_sb = bp.dq_batch_stride; f.dq_sr = bp.dq_row_stride; f.dq_sh = bp.dq_head_stride;
  }
  f.pos = bp.scatter_pos; f.pos_sb = bp.scatter_batch_stride; f.pos_sh = bp.scatter_head_stride;
  f.h_pos = bp.scatter_h; f.cap = p.seqlen_k;
  if (pl.part) {
    f.part = kp.dkv_part; f.nsplit = pl.nsplit;
    f.split_stride = static_cast<int64_t>(p.b) * p.h_k * f.keys_r * D;
    f.dk = bp.dk; f.dk_sb = bp.dk_batch_stride; f.dk_sr = bp.dk_row_stride; f.dk_sh = bp.dk_head_stride;
    f.dv = bp.dv; f.dv_sb = bp.dv_batch_stride; f.dv_sr = bp.dv_row_stride; f.dv_sh = bp.dv_head_stride;
  }
  if (pl.dbias_mode == kDbAtomic || (pl.dbias_mode == kDbColsum && pl.part)) {
    const bool atomic = pl.dbias_mode == kDbAtomic;
    f.db_part = atomic ? kp.dbias_acc : kp.dbias_part;
    f.db_nsplit = atomic ? 1 : pl.nsplit;
    f.db_pitch = atomic ? atomic_keys(bp) : f.keys_r;
    f.db_split_stride = static_cast<int64_t>(p.b) * p.h_k * f.keys_r;
    f.db_b = bp.dbias_b; f.db_h = bp.dbias_h; f.db_keys = bp.dbias_keys;
    f.dbias = bp.dbias; f.db_sb = bp.dbias_batch_stride; f.db_sh = bp.dbias_head_stride;
  }
  return launch_bwd_finish(f, kBf16, false, stream);
}

}  // namespace

// Calls of tc_bwd (head dims up to 128) that this file takes: mask and bias broadcast over the queries, or absent, and a dBias,
// if asked for, that is summed over them; but not those of few queries over many keys, beyond what fits in one wave of CTAs. There the row
// pass is a few long chains of key tiles, while the single pass of fdma_bwd_sm100.cu spreads dQ over all key tiles. Backward in us, here
// without ranges / single pass, head dim 128 (queries x keys, heads): 128 x 65536, 8 over 2 962 / 150, 32 over 8 1286 / 540; 1024 x 16384,
// 32 over 8 856 / 682; 512 x 4096, 16 over 4 98 / 65; 1024 x 4096 gathered, 8 over 2 138 / 94; 256 x 2048, 32 over 8 56 / 42; but 512 x 2048,
// 8 over 2 39 / 63, 1024 x 512, 16 over 4 64 / 77.
// Per tile the single pass is the slower one at head dim 64 (4096 x 8192, 16 over 4 686 / 830), with less than three query heads to share
// what a query tile needs (8192 x 1024 gathered, MHA 491 / 684), with addends per query head and with fixed-point sums (2048 x 8192
// 502 / 729). Such calls go there only while row tiles x heads leave half the SMs idle, three quarters in fixed point (256 x 8192, 32 heads,
// 64 row tiles: d = 64 152 / 120, MHA 280 / 224, per head 230 / 176, fixed point 183 / 180).
bool bwd_rows_taken(const fdma_bwd_params& bp) {
  const fdma_fwd_params& p = bp.f;
  const bool mask_b = !p.mask || p.mask_row_stride == 0 || p.seqlen_q == 1;
  const bool bias_b = !p.bias || p.bias_row_stride == 0 || p.seqlen_q == 1;
  if (!mask_b || !bias_b || (bp.dbias && bp.dbias_rows != 1)) return false;
  // Masks with more tiles than the activity bits hold: 1024 queries, 8 heads over 2, d = 64, 300000 keys, every tile worked on here / single
  // pass: 11 kept keys 3367 / 641 us, half of them 4811 / 3299.
  if (p.mask && p.seqlen_k > kMaxBits * kBM) return false;
  if (p.seqlen_k < 2048 || p.seqlen_k < (p.seqlen_k < 4096 ? 8ll : 4ll) * p.seqlen_q) return true;
  const int half_sms = sm_count() / 2;
  const int64_t key_tiles = static_cast<int64_t>((p.seqlen_k + kBN - 1) / kBN) * p.h_k * p.b;
  if (key_tiles <= half_sms && row_tiles(p) <= half_sms / 4) return true;
  const bool per_head = (p.mask && p.h_mask == p.h) || (p.bias && p.h_bias == p.h);
  if (tile_head_dim(p.d) == 128 && p.h >= 3 * p.h_k && !per_head && !bp.deterministic) return false;
  return row_tiles(p) > (bp.deterministic ? half_sms / 2 : half_sms);
}

// Packed sequences, whose lengths only the device knows: by all their queries and keys. Here / single pass, us, 8 heads over 2: 2 x 64 queries
// over 2 x 16384 keys 244 / 70, one query over 65536 keys beside 127 over 64 919 / 169, 2 x 128 over 2 x 1024 25 / 31; 16 over 4: 2 x 1024 over 2 x
// 16384 875 / 706, 4 x 512 over 4 x 2048 170 / 163, 4 x 256 over 4 x 1024 71 / 72; MHA at head dim 64, 2 x 256 over 2 x 4096 182 / 195.
bool bwd_rows_taken_packed(const fdma_bwd_params& bp) { return bp.f.seqlen_k < 4096 || bp.f.seqlen_k < 4ll * bp.f.seqlen_q; }

size_t bwd_rows_workspace_bytes(const fdma_bwd_params& bp) { return plan(bp).total; }

int bwd_rows(const fdma_bwd_params& bp, cudaStream_t stream, const PackedSeqs& seqs) {
  const RowsPlan pl = plan(bp);
  const bool bf16 = bp.f.dtype == FDMA_BF16;
  if (pl.D == 64) return bf16 ? launch<64, true>(bp, pl, seqs, stream) : launch<64, false>(bp, pl, seqs, stream);
  return bf16 ? launch<128, true>(bp, pl, seqs, stream) : launch<128, false>(bp, pl, seqs, stream);
}

}  // namespace fdma
