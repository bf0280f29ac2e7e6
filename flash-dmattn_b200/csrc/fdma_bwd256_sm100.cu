// Dynamic-mask attention backward for head dims 136 to 256 on Blackwell tensor cores (tcgen05 + TMEM + TMA), for
// row-broadcast masks and biases (the shape create_mask produces from a (B, Hk, 1, Sk) bias).
//
// Same mathematics as the head-dim-128 kernel next door (fdma_bwd_sm100.cu; the reference kernel is
// csrc/flash_sparse_attn/src/flash_bwd_kernel.h:79-1142). What differs is the budget: at d = 256 the accumulator of ONE
// gradient of a 128-row tile takes 256 of the 512 TMEM columns and a 128-row operand 64 KB of shared memory. So every
// gradient has its own pass, and all three are the same pipeline over a stationary 128-row tile and 64-row tiles that
// stream by:
//              stationary        streamed, 64 rows    scores          gradient product
//     kDk      K, V (128 keys)   Q, dO (each head)    St, dPt         dK += dS^T Q
//     kDv      K    (128 keys)   Q, dO (each head)    St              dV += P^T dO
//     kDq      Q, dO (128 rows)  K, V                 S, dP           dQ += dS K
// with scores[row, column] = (stationary row) . (streamed row), the probabilities or dS written back in 16 bit over the
// scores as the A operand (from TMEM), and the B operand read MN-major from the streamed tile. dK's pass also sums dS over its queries
// for dBias. dQ is complete in TMEM up to kFlush key tiles: no accumulator in memory, nothing to zero, add to or convert, and the
// same bits every time. Beyond, the CTA adds what it has to an fp32 tile of its own in memory every kFlush steps: the tensor
// core truncates its sums, which over 65536 keys made dQ in fp16 3 % less exact (2.95e-4 -> 3.05e-4).
//
// TMEM: scores[2] 2 x 64 | dP[2] 2 x 64 | accumulator 256. The products of step i+1 are issued before the gradient
// product of step i, so the softmax of a step runs under 1536 cycles of tensor work of the next (d = 256, N = 64 products are bound by the
// shared-memory reads of their operands: 48 cycles per 16 columns of d against 32 of arithmetic). Shared memory: the operand of the
// gradient product must stay until that product is done and has two slots, the other streamed operand one (two for kDv).
// 8 products of 128 x 64 x 256 per tile pair instead of the 7 of a two-pass form (dV and dQ in one pass, dK in the other) that had
// one slot for everything, no overlap between steps and an fp32 dQ buffer in memory. 65536 queries, 16 heads over one kv head,
// 2048 kept keys: kernel 8.3 -> 5.5 ms, with the kernels around it 8.95 -> 5.8 ms.
// One launch: the CTAs of the three passes are mixed, dK first.
//
// Warps: 0 TMA producer | 1 MMA issuer | 2 row vectors (LSE and D of 64 queries, or addend and position of 64 keys) |
// 4-7, 8-11 softmax and epilogue (thread = stationary row; score columns 0-31 / 32-63). Every mbarrier wait is bounded.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>

#include "fdma_internal.h"
#include "fdma_ptx.cuh"

namespace fdma {
namespace {

constexpr int kD = 256;
constexpr int kBN = 128;  // stationary rows per CTA
constexpr int kBM = 64;   // streamed rows per step
constexpr int kThreads = 384;
constexpr int kFlush = 64;  // 64-key steps whose dQ the tensor core sums up (4096 keys)
constexpr int kMaxBits = 4096;  // 64-key tiles the activity bits of a dQ pass can hold; beyond, every tile is worked on
constexpr float kLog2e = 1.4426950408889634f;

enum Pass { kDk = 0, kDv = 1, kDq = 2 };
enum WaitCode256 {
  kW256X = 301, kW256AEmpty = 302, kW256AFull = 303, kW256SFull = 304, kW256Pds = 305, kW256BEmpty = 306,
  kW256BFull = 307, kW256VecEmpty = 308, kW256VecFull = 309, kW256Final = 310
};

struct Bwd256Params {
  CUtensorMap tm_q, tm_do, tm_k, tm_v;  // boxes of 64 rows x 64 elements
  const uint8_t* mask;
  const void* bias;
  const float* lse2;   // (B,H,Sq_r) LSE * log2(e); +inf for empty and padded rows
  const float* dsum;   // (B,H,Sq_r) D = rowsum(dO o O)
  void* dq;
  void* dk;
  void* dv;
  void* dbias;
  float* dq_acc;       // more than kFlush key tiles: fp32 (B,H,Sq,256), each row the running sum of one dQ CTA
  float* dkv_part;     // null, or fp32 partials [2: dV, dK][nsplit][B][h_k][NT*128][256] instead of dk / dv
  float* dbias_part;   // with dkv_part: fp32 partials [nsplit][B][h_k][NT*128]
  int* status;
  int64_t mask_batch_stride, mask_head_stride, bias_batch_stride, bias_head_stride;
  int64_t dq_batch_stride, dq_row_stride, dq_head_stride;
  int64_t dk_batch_stride, dk_row_stride, dk_head_stride;
  int64_t dv_batch_stride, dv_row_stride, dv_head_stride;
  int64_t dbias_batch_stride, dbias_head_stride;
  int b, seqlen_q, seqlen_k, sq_r, h, h_k, h_mask, h_bias, d;
  int dbias_keys, want_dbias, nsplit, is_causal;
  int n_kv_ctas;       // CTAs of the dK pass, and of the dV pass
  const int32_t* key_pos;
  int64_t pos_batch_stride, pos_head_stride;
  int h_pos, causal_shift;
  float scale_log2, scale;
};

struct Smem256 {
  static constexpr int kTile = kBN * kD * 2;                // 64 KB: 4 blocks of [128 rows][64 d]
  static constexpr int kStep = kBM * kD * 2;                // 32 KB: 4 blocks of [64 rows][64 d]
  static constexpr int kXOff = 0;                           // stationary operand of the scores
  static constexpr int kX2Off = kTile;                      // ... of dP; kDv: second slot of the other streamed operand
  static constexpr int kAOff = 2 * kTile;                   // two slots: streamed operand of the gradient product
  static constexpr int kBOff = kAOff + 2 * kStep;           // one slot: the other streamed operand
  static constexpr int kVecOff = kBOff + kStep;             // [2][128] 32-bit values of the step's 64 columns
  static constexpr int kBitsOff = kVecOff + 2 * 128 * 4;
  static constexpr int kBarOff = kBitsOff + kMaxBits / 8;
  static constexpr int kNumBars = 18;
  static constexpr int kMiscOff = kBarOff + kNumBars * 8;
  static constexpr int kTotal = kMiscOff + 32;
  static constexpr int kAlloc = kTotal + 1024;  // slack to align the base to 1024 B
};
static_assert(Smem256::kAlloc <= 232448, "shared memory budget of one CTA");

template <bool kBf16>
__device__ __forceinline__ float raw16_to_f(uint16_t u) {
  if (kBf16) return __uint_as_float(static_cast<uint32_t>(u) << 16);
  return __half2float(__ushort_as_half(u));
}
template <bool kBf16>
__device__ __forceinline__ uint16_t f_to_raw16(float x) {
  return static_cast<uint16_t>(pack_16x2<kBf16>(x, 0.f) & 0xFFFFu);
}

template <bool kBf16, int kPass>
__device__ __forceinline__ void pass256(const Bwd256Params& p, unsigned char* smem, int item) {
  using L = Smem256;
  constexpr bool kKeys = kPass != kDq;     // stationary rows are keys
  constexpr bool kDp = kPass != kDv;       // the pass needs dP
  constexpr int kBSlots = kDp ? 1 : 2;
  float* s_vec = reinterpret_cast<float*>(smem + L::kVecOff);
  uint32_t* s_bits = reinterpret_cast<uint32_t*>(smem + L::kBitsOff);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* bar_x = bars;
  uint64_t* bar_a_full = bars + 1;       // [2]
  uint64_t* bar_a_empty = bars + 3;      // [2]
  uint64_t* bar_b_full = bars + 5;       // [2], kDk and kDq use the first
  uint64_t* bar_b_empty = bars + 7;      // [2]
  uint64_t* bar_s_full = bars + 9;       // [2]
  uint64_t* bar_pds = bars + 11;         // [2]
  uint64_t* bar_vec_full = bars + 13;    // [2]
  uint64_t* bar_vec_empty = bars + 15;   // [2]
  uint64_t* bar_final = bars + 17;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + L::kMiscOff);
  volatile int* s_abort = reinterpret_cast<volatile int*>(smem + L::kMiscOff + 4);
  int* s_count = reinterpret_cast<int*>(smem + L::kMiscOff + 8);   // [0] active 64-key tiles, [1] visible kept keys

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = p.h / p.h_k;
  const int Sq = p.seqlen_q, Sk = p.seqlen_k;
  const int NT = (Sk + kBN - 1) / kBN;
  const bool causal = p.is_causal != 0;
  // the CTA's stationary tile n, its (kv) head and batch element; key passes: its range of 64-row query tiles
  int n, hk, b, h = 0, split = 0;
  if (kKeys) {
    // (query-range split, key tile): with more than one split the CTA covers the query tiles [m_start, M64) of its key tile
    // and leaves fp32 partials. The last ranges, never emptied by causal masking, run first.
    const int per = NT * p.nsplit;
    n = item % per % NT;
    split = p.nsplit - 1 - item % per / NT;
    hk = item / per % p.h_k;
    b = item / per / p.h_k;
  } else {
    const int per = p.h * p.b;  // the last query tiles, which see most keys, run first; heads of a group meet in L2
    n = (Sq + kBN - 1) / kBN - 1 - item / per;
    h = item % per % p.h;
    b = item % per / p.h;
    hk = h / G;
  }
  const int32_t* pos_row = nullptr;  // compacted keys: the causal test runs on their original positions
  if (causal && p.key_pos)
    pos_row = p.key_pos + b * p.pos_batch_stride + (p.h_pos == p.h_k ? hk : 0) * p.pos_head_stride;
  const int coff = pos_row ? p.causal_shift : Sk - Sq;
  const int hm = p.h_mask == p.h_k ? hk : 0;  // heads of mask / bias are 1 or h_k here (or h == h_k)
  const int hb = p.h_bias == p.h_k ? hk : 0;
  const uint8_t* mrow = p.mask ? p.mask + b * p.mask_batch_stride + hm * p.mask_head_stride : nullptr;
  const uint16_t* brow = p.bias ? reinterpret_cast<const uint16_t*>(p.bias) + b * p.bias_batch_stride + hb * p.bias_head_stride
                                : nullptr;
  int m_start = 0, M64 = 0;
  if (kKeys) {
    const int M64_all = (Sq + kBM - 1) / kBM;
    const int m_chunk = (M64_all + p.nsplit - 1) / p.nsplit;
    M64 = min(M64_all, (split + 1) * m_chunk);
    if (pos_row) {
      const int64_t first = (static_cast<int64_t>(pos_row[n * kBN]) - coff) / kBM;
      m_start = static_cast<int>(max(static_cast<int64_t>(0), min(first, static_cast<int64_t>(M64))));
    } else if (causal) {
      m_start = max(0, (n * kBN - coff) / kBM);
    }
    m_start = max(m_start, split * m_chunk);
  }
  const WaitCtl ctl{s_abort, p.status};

  // ---------------- set-up ----------------
  if (tid == 0) {
    *s_abort = 0;
    s_count[0] = s_count[1] = 0;
    mbar_init(bar_x, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_a_full + i, 1);
      mbar_init(bar_a_empty + i, 1);
      mbar_init(bar_b_full + i, 1);
      mbar_init(bar_b_empty + i, 1);
      mbar_init(bar_s_full + i, 1);
      mbar_init(bar_pds + i, 8);  // one arrival per softmax warp
      mbar_init(bar_vec_full + i, 1);
      mbar_init(bar_vec_empty + i, 8);
    }
    mbar_init(bar_final, 1);
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
  // dQ pass: one activity bit per 64-key tile, where there is a mask and the table is large enough
  const bool use_bits = !kKeys && mrow && (Sk + kBM - 1) / kBM <= kMaxBits;
  if (use_bits)
    for (int i = tid; i < kMaxBits / 32; i += kThreads) s_bits[i] = 0;
  __syncthreads();
  const int q_last = min(n * kBN + kBN, Sq) - 1;  // dQ pass: last query row of the tile
  if (kKeys) {
    if (warp == 2) {  // does this key tile hold a kept key at all?
      bool any = !mrow;
      if (mrow)
        for (int i = lane; i < kBN; i += 32) any = any || (n * kBN + i < Sk && mrow[n * kBN + i] != 0);
      any = __any_sync(0xffffffffu, any);
      if (lane == 0) s_count[0] = any ? 1 : 0;
    }
  } else {
    if (use_bits) {
      for (int c = tid; c < (Sk + 15) / 16; c += kThreads) {
        const uint4 v = *reinterpret_cast<const uint4*>(mrow + c * 16);
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
        if (c * 16 + 16 > Sk) {
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (c * 16 + e >= Sk) w[e >> 2] &= ~(0xFFu << ((e & 3) * 8));
        }
        if (w[0] | w[1] | w[2] | w[3]) atomicOr(&s_bits[c >> 7], 1u << ((c >> 2) & 31));
      }
    }
    if (pos_row) {  // keys the last query row sees: a prefix of the ascending positions
      int cnt = 0;
      for (int k = tid; k < Sk; k += kThreads) cnt += static_cast<int64_t>(pos_row[k]) <= static_cast<int64_t>(q_last) + coff ? 1 : 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, s);
      if (lane == 0) atomicAdd(&s_count[1], cnt);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*s_tmem);
  int n_steps, n_sub = 0;
  if (kKeys) {
    n_steps = (s_count[0] && M64 > m_start) ? (M64 - m_start) * G : 0;
  } else {
    int vis = Sk;
    if (pos_row) vis = s_count[1];
    else if (causal) vis = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(Sk), static_cast<int64_t>(q_last) + coff + 1)));
    n_sub = (vis + kBM - 1) / kBM;
    n_steps = n_sub;
    if (use_bits) {
      n_steps = 0;
      for (int w = 0; w * 32 < n_sub; ++w)
        n_steps += __popc(s_bits[w] & (n_sub - w * 32 >= 32 ? 0xFFFFFFFFu : (1u << (n_sub - w * 32)) - 1u));
    }
  }
  n_steps = warp_uniform(n_steps);
  // Steps: (query tile m, head g of the group), or key tile m
  int m = kKeys ? m_start : -1, g = 0;
  auto next = [&]() {
    if (kKeys) {
      if (++g == G) {
        g = 0;
        ++m;
      }
    } else {
      do ++m;
      while (use_bits && m < n_sub && !((s_bits[m >> 5] >> (m & 31)) & 1u));
    }
  };
  if (!kKeys) next();  // to the first active tile
  constexpr uint32_t kColS = 0, kColDp = 128, kColAcc = 256;
  auto b_slot = [&](int i) { return smem + ((kBSlots == 2 && (i & 1)) ? L::kX2Off : L::kBOff); };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0 && n_steps > 0) {
      const int hx = kKeys ? hk : h;
      mbar_arrive_expect_tx(bar_x, (kDp ? 2 : 1) * L::kTile);
#pragma unroll
      for (int kb = 0; kb < kD / 64; ++kb)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int dst = kb * (kBN * 128) + r * (kBM * 128), row = n * kBN + r * kBM;
          tma_load_4d(smem + L::kXOff + dst, kKeys ? &p.tm_k : &p.tm_q, bar_x, kb * 64, hx, row, b);
          if (kDp) tma_load_4d(smem + L::kX2Off + dst, kKeys ? &p.tm_v : &p.tm_do, bar_x, kb * 64, hx, row, b);
        }
      const CUtensorMap* tm_a = kPass == kDk ? &p.tm_q : kPass == kDv ? &p.tm_do : &p.tm_k;
      const CUtensorMap* tm_b = kPass == kDk ? &p.tm_do : kPass == kDv ? &p.tm_q : &p.tm_v;
      bool ok = true;
      for (int i = 0; i < n_steps && ok; ++i, next()) {
        const int head = kKeys ? hk * G + g : hk, row = m * kBM;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          // in the order the products want them: kDv computes its scores from the other operand
          if ((k == 0) == kDp) {
            ok = mbar_wait(bar_a_empty + (i & 1), ((i >> 1) & 1) ^ 1, ctl, kW256AEmpty);
            if (!ok) break;
            mbar_arrive_expect_tx(bar_a_full + (i & 1), L::kStep);
#pragma unroll
            for (int kb = 0; kb < kD / 64; ++kb)
              tma_load_4d(smem + L::kAOff + (i & 1) * L::kStep + kb * (kBM * 128), tm_a, bar_a_full + (i & 1), kb * 64, head, row, b);
          } else {
            const int slot = i % kBSlots;
            ok = mbar_wait(bar_b_empty + slot, ((i / kBSlots) & 1) ^ 1, ctl, kW256BEmpty);
            if (!ok) break;
            mbar_arrive_expect_tx(bar_b_full + slot, L::kStep);
#pragma unroll
            for (int kb = 0; kb < kD / 64; ++kb)
              tma_load_4d(b_slot(i) + kb * (kBM * 128), tm_b, bar_b_full + slot, kb * 64, head, row, b);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (whole warp, uniform control flow; the issue wrappers are predicated on one lane) -------
    if (n_steps > 0) {
      const uint32_t lead = umma_leader();
      constexpr uint32_t idesc_s = umma_idesc(kBN, kBM, kBf16, false, false);  // scores, dP: 128 x 64, K-major
      constexpr uint32_t idesc_g = umma_idesc(kBN, kD, kBf16, false, true);    // gradient: A from TMEM, B MN-major
      const uint32_t x_addr = smem_u32(smem + L::kXOff), x2_addr = smem_u32(smem + L::kX2Off);
      auto product = [&](uint32_t col, uint32_t x, uint32_t y) {  // [128 x 64] = x y^T
        const uint64_t xd = umma_desc_sw128(x, 16, 1024), yd = umma_desc_sw128(y, 16, 1024);
#pragma unroll
        for (int kk = 0; kk < kD / 16; ++kk)
          umma_ss(lead, tmem_base + col, umma_desc_at(xd, (kk >> 2) * (kBN * 128) + (kk & 3) * 32),
                  umma_desc_at(yd, (kk >> 2) * (kBM * 128) + (kk & 3) * 32), idesc_s, kk > 0 ? 1u : 0u);
      };
      auto wait = [&](uint64_t* bar, int phase, int code) {
        const bool r = __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, ctl, code));
        tc_fence_after_sync();
        return r;
      };
      auto scores = [&](int i) {
        const uint32_t a_addr = smem_u32(smem + L::kAOff + (i & 1) * L::kStep), b_addr = smem_u32(b_slot(i));
        if (kDp) {
          if (!wait(bar_a_full + (i & 1), i >> 1, kW256AFull)) return false;
          product(kColS + (i & 1) * kBM, x_addr, a_addr);
          if (!wait(bar_b_full, i, kW256BFull)) return false;
          product(kColDp + (i & 1) * kBM, x2_addr, b_addr);
        } else {
          if (!wait(bar_b_full + (i & 1), i >> 1, kW256BFull)) return false;
          product(kColS + (i & 1) * kBM, x_addr, b_addr);
        }
        umma_commit(lead, bar_s_full + (i & 1));
        umma_commit(lead, bar_b_empty + i % kBSlots);
        return true;
      };
      bool ok = wait(bar_x, 0, kW256X) && scores(0);
      for (int i = 0; i < n_steps && ok; ++i) {
        // The buffers of step i+1 were last used by step i-1: its scores by the gradient product issued before, its dP by
        // softmax warps that have handed step i-1 over.
        if (i + 1 < n_steps) ok = scores(i + 1);
        if (ok) ok = wait(bar_pds + (i & 1), i >> 1, kW256Pds);
        if (ok && !kDp) ok = wait(bar_a_full + (i & 1), i >> 1, kW256AFull);
        if (!ok) break;
        const uint64_t ad = umma_desc_sw128(smem_u32(smem + L::kAOff + (i & 1) * L::kStep), kBM * 128, 1024);
        const bool fresh = kPass == kDq ? i % kFlush == 0 : i == 0;
#pragma unroll
        for (int s = 0; s < 4; ++s)  // columns 0-31 of the step sit in [0,16) of the score block, 32-63 in [32,48)
          umma_ts(lead, tmem_base + kColAcc, tmem_base + kColS + (i & 1) * kBM + (s < 2 ? s * 8 : 32 + (s - 2) * 8),
                  umma_desc_at(ad, s * 2048), idesc_g, (fresh && s == 0) ? 0u : 1u);
        umma_commit(lead, bar_a_empty + (i & 1));
        // (the next product waits for softmax warps that have read the sums by then)
        if (kPass == kDq && i % kFlush == kFlush - 1 && i + 1 < n_steps) umma_commit(lead, bar_final);
      }
      if (ok) umma_commit(lead, bar_final);
    }
  } else if (warp == 2) {
    // ---------------- vectors of the step's 64 columns ----------------
    bool ok = true;
    for (int i = 0; i < n_steps && ok; ++i, next()) {
      uint4 v;
      int2 pos = make_int2(0, 0);
      if (kKeys) {  // LSE (lanes 0-15) and D (16-31) of 64 queries
        const int64_t row0 = (static_cast<int64_t>(b) * p.h + hk * G + g) * p.sq_r + m * kBM;
        v = *reinterpret_cast<const uint4*>((lane < 16 ? p.lse2 : p.dsum) + row0 + (lane & 15) * 4);
      } else {  // addend (bias in log2 units, or -inf where masked out) and position of two keys per lane
        const int k = m * kBM + lane * 2;
        const uint32_t mb = mrow ? *reinterpret_cast<const uint16_t*>(mrow + k) : 0x0101u;
        const uint32_t bb = brow ? *reinterpret_cast<const uint32_t*>(brow + k) : 0u;
        v.x = __float_as_uint(k < Sk && (mb & 0xFFu) ? raw16_to_f<kBf16>(static_cast<uint16_t>(bb & 0xFFFFu)) * kLog2e : -CUDART_INF_F);
        v.y = __float_as_uint(k + 1 < Sk && (mb >> 8) ? raw16_to_f<kBf16>(static_cast<uint16_t>(bb >> 16)) * kLog2e : -CUDART_INF_F);
        pos = make_int2(k, k + 1);
        if (pos_row) pos = make_int2(k < Sk ? pos_row[k] : 0x7FFFFFFF, k + 1 < Sk ? pos_row[k + 1] : 0x7FFFFFFF);
      }
      ok = __all_sync(0xffffffffu, mbar_wait(bar_vec_empty + (i & 1), ((i >> 1) & 1) ^ 1, ctl, kW256VecEmpty));
      if (!ok) break;
      float* dst = s_vec + (i & 1) * 128;
      if (kKeys) {
        reinterpret_cast<uint4*>(dst)[lane] = v;
      } else {
        reinterpret_cast<uint2*>(dst)[lane] = make_uint2(v.x, v.y);
        reinterpret_cast<int2*>(dst + 64)[lane] = pos;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_vec_full + (i & 1));
    }
  } else if (warp >= 4) {
    // ---------------- softmax warpgroups: thread = stationary row = TMEM lane; `half` takes 32 of the 64 columns ----
    const int half = (warp - 4) >> 2;
    const int row = n * kBN + (warp & 3) * 32 + lane;
    const int warp_row = n * kBN + (warp & 3) * 32;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool row_ok = row < (kKeys ? Sk : Sq);
    // key passes: addend of this key, and the value compared with q + coff in the causal test, its position
    // (clamped so that ckey - coff cannot overflow; padding slots hold INT_MAX and are masked out anyway)
    float bv = -CUDART_INF_F;
    int ckey = 0, ckey_wmax = 0;
    // dQ pass: LSE and D of this query, and the last position it (and the warp's first query) sees
    float lse = CUDART_INF_F, dsum = 0.f;
    int qlim = 0x7FFFFFFE, qlim_wmin = 0x7FFFFFFE;
    if (kKeys) {
      ckey = pos_row ? (row_ok ? min(pos_row[row], 0x3FFFFFFF) : 0x3FFFFFFF) : row;
      ckey_wmax = pos_row ? __shfl_sync(0xffffffffu, ckey, 31) : warp_row + 31;
      if (row_ok && (!mrow || mrow[row])) bv = brow ? raw16_to_f<kBf16>(brow[row]) * kLog2e : 0.f;
    } else {
      if (row_ok) {
        const int64_t idx = (static_cast<int64_t>(b) * p.h + h) * p.sq_r + row;
        lse = p.lse2[idx];
        dsum = p.dsum[idx];
      }
      if (causal) {
        auto clamp = [](int64_t x) { return static_cast<int>(max(static_cast<int64_t>(-1), min(x, static_cast<int64_t>(0x7FFFFFFE)))); };
        qlim = clamp(static_cast<int64_t>(row) + coff);
        qlim_wmin = clamp(static_cast<int64_t>(warp_row) + coff);
      }
    }
    float colsum = 0.f;
    bool ok = true;
    int flushed = 0;  // dQ pass: sums moved to memory so far
    float* acc_row = kKeys ? nullptr : p.dq_acc + ((static_cast<int64_t>(b) * p.h + h) * Sq + min(row, Sq - 1)) * kD + half * 128;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    const float2 neg1 = make_float2(-1.f, -1.f);
    for (int i = 0; i < n_steps && ok; ++i, next()) {
      const float* vec = s_vec + (i & 1) * 128 + half * 32;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_vec_full + (i & 1), (i >> 1) & 1, ctl, kW256VecFull));
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait(bar_s_full + (i & 1), (i >> 1) & 1, ctl, kW256SFull));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t rs[32], rp[32], pk[16];
      tmem_ld_x32(tmem_base + lane_addr + kColS + (i & 1) * kBM + half * 32, rs);
      if (kDp) tmem_ld_x32(tmem_base + lane_addr + kColDp + (i & 1) * kBM + half * 32, rp);
      tmem_wait_ld();
      const int* pos = reinterpret_cast<const int*>(vec + 64);
      const int q0 = m * kBM + half * 32;
      const bool diag = causal && (kKeys ? static_cast<int64_t>(ckey_wmax) > static_cast<int64_t>(q0) + coff
                                         : pos[31] > qlim_wmin);  // warp-uniform
      float2 part[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int j4 = 0; j4 < 8; ++j4) {
        const float4 v4 = reinterpret_cast<const float4*>(vec)[j4];
        float4 d4 = make_float4(dsum, dsum, dsum, dsum);
        if (kKeys && kDp) d4 = reinterpret_cast<const float4*>(vec + 64)[j4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = j4 * 2 + e;  // pair of columns
          const float2 vv = e == 0 ? make_float2(v4.x, v4.y) : make_float2(v4.z, v4.w);
          const float2 dv = e == 0 ? make_float2(d4.x, d4.y) : make_float2(d4.z, d4.w);
          float2 add;  // bias - LSE, or -inf
          if (kKeys) {
            float2 b2 = make_float2(bv, bv);
            if (diag) {
              if (ckey - coff > q0 + 2 * j) b2.x = -CUDART_INF_F;
              if (ckey - coff > q0 + 2 * j + 1) b2.y = -CUDART_INF_F;
            }
            add = __ffma2_rn(vv, neg1, b2);
          } else {
            add = __fadd2_rn(vv, make_float2(-lse, -lse));
            if (diag) {
              if (pos[2 * j] > qlim) add.x = -CUDART_INF_F;
              if (pos[2 * j + 1] > qlim) add.y = -CUDART_INF_F;
            }
          }
          const float2 x = __ffma2_rn(make_float2(__uint_as_float(rs[2 * j]), __uint_as_float(rs[2 * j + 1])), sc2, add);
          const float2 pj = make_float2(fast_exp2(x.x), fast_exp2(x.y));
          if (kDp) {
            const float2 dpd = __ffma2_rn(dv, neg1, make_float2(__uint_as_float(rp[2 * j]), __uint_as_float(rp[2 * j + 1])));
            const float2 ds = __fmul2_rn(pj, dpd);
            if (kPass == kDk) part[e] = __fadd2_rn(part[e], ds);
            pk[j] = pack_16x2<kBf16>(ds.x, ds.y);
          } else {
            pk[j] = pack_16x2<kBf16>(pj.x, pj.y);
          }
        }
      }
      if (kPass == kDk) colsum += (part[0].x + part[0].y) + (part[1].x + part[1].y);
      tmem_st_x16(tmem_base + lane_addr + kColS + (i & 1) * kBM + half * 32, pk);
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bar_vec_empty + (i & 1));
        mbar_arrive(bar_pds + (i & 1));
      }
      if (kPass == kDq && i % kFlush == kFlush - 1 && i + 1 < n_steps) {
        ok = __all_sync(0xffffffffu, mbar_wait(bar_final, flushed & 1, ctl, kW256Final));
        if (!ok) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld_x32(tmem_base + lane_addr + kColAcc + half * 128 + c * 32, r);
          tmem_wait_ld();
          if (row_ok) {
#pragma unroll
            for (int v4 = 0; v4 < 8; ++v4) {
              float4* dst = reinterpret_cast<float4*>(acc_row + c * 32 + v4 * 4);
              float4 x = make_float4(__uint_as_float(r[v4 * 4]), __uint_as_float(r[v4 * 4 + 1]), __uint_as_float(r[v4 * 4 + 2]),
                                     __uint_as_float(r[v4 * 4 + 3]));
              if (flushed) {
                const float4 y = *dst;
                x = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
              }
              *dst = x;
            }
          }
        }
        ++flushed;
      }
    }
    // ---------------- the gradient tile; dBias sums of the dK pass ----------------
    if (kPass == kDk && p.want_dbias) {
      named_bar_sync(1, 256);  // the step vectors have been read: their place takes the sums of the second half
      if (half == 1) s_vec[row - n * kBN] = colsum;
      named_bar_sync(1, 256);
      if (half == 0 && row < p.dbias_keys) {
        const float tot = row_ok ? colsum + s_vec[row - n * kBN] : 0.f;
        if (p.dkv_part)
          p.dbias_part[((static_cast<int64_t>(split) * p.b + b) * p.h_k + hk) * (NT * kBN) + row] = tot;
        else
          reinterpret_cast<uint16_t*>(p.dbias)[b * p.dbias_batch_stride + hk * p.dbias_head_stride + row] = f_to_raw16<kBf16>(tot);
      }
    }
    if (ok && n_steps > 0) ok = __all_sync(0xffffffffu, mbar_wait(bar_final, flushed & 1, ctl, kW256Final));
    tc_fence_after_sync();
    if (ok) {
      const float mul = kPass == kDv ? 1.f : p.scale;
      const int64_t row_g = min(row, (kKeys ? Sk : Sq) - 1);
      uint16_t* dst = kPass == kDv   ? reinterpret_cast<uint16_t*>(p.dv) + b * p.dv_batch_stride + hk * p.dv_head_stride + row_g * p.dv_row_stride
                      : kPass == kDk ? reinterpret_cast<uint16_t*>(p.dk) + b * p.dk_batch_stride + hk * p.dk_head_stride + row_g * p.dk_row_stride
                                     : reinterpret_cast<uint16_t*>(p.dq) + b * p.dq_batch_stride + h * p.dq_head_stride + row_g * p.dq_row_stride;
      // partial: part[dv|dk][split][b][hk][key][256]
      float* part = p.dkv_part + ((((static_cast<int64_t>(kPass == kDk ? 1 : 0) * p.nsplit + split) * p.b + b) * p.h_k + hk) *
                                      (NT * kBN) + row) * kD;
#pragma unroll
      for (int c = 0; c < 4; ++c) {  // this warpgroup's 128 of the 256 columns
        const int col = half * 128 + c * 32;
        uint32_t r[32];
        if (n_steps > 0) {
          tmem_ld_x32(tmem_base + lane_addr + kColAcc + col, r);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        if (kPass == kDq && flushed && row_ok) {
#pragma unroll
          for (int v4 = 0; v4 < 8; ++v4) {
            const float4 y = *reinterpret_cast<const float4*>(acc_row + c * 32 + v4 * 4);
            r[v4 * 4] = __float_as_uint(__uint_as_float(r[v4 * 4]) + y.x);
            r[v4 * 4 + 1] = __float_as_uint(__uint_as_float(r[v4 * 4 + 1]) + y.y);
            r[v4 * 4 + 2] = __float_as_uint(__uint_as_float(r[v4 * 4 + 2]) + y.z);
            r[v4 * 4 + 3] = __float_as_uint(__uint_as_float(r[v4 * 4 + 3]) + y.w);
          }
        }
        if (kKeys && p.dkv_part) {
#pragma unroll
          for (int v4 = 0; v4 < 8; ++v4)
            *reinterpret_cast<float4*>(part + col + v4 * 4) =
                make_float4(__uint_as_float(r[v4 * 4 + 0]) * mul, __uint_as_float(r[v4 * 4 + 1]) * mul,
                            __uint_as_float(r[v4 * 4 + 2]) * mul, __uint_as_float(r[v4 * 4 + 3]) * mul);
        } else if (row_ok) {
#pragma unroll
          for (int v4 = 0; v4 < 4; ++v4) {
            if (col + v4 * 8 >= p.d) break;
            uint4 o;
            o.x = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 0]) * mul, __uint_as_float(r[v4 * 8 + 1]) * mul);
            o.y = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 2]) * mul, __uint_as_float(r[v4 * 8 + 3]) * mul);
            o.z = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 4]) * mul, __uint_as_float(r[v4 * 8 + 5]) * mul);
            o.w = pack_16x2<kBf16>(__uint_as_float(r[v4 * 8 + 6]) * mul, __uint_as_float(r[v4 * 8 + 7]) * mul);
            *reinterpret_cast<uint4*>(dst + col + v4 * 8) = o;
          }
        }
      }
    }
  }

  // ---------------- tear-down ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <bool kBf16>
__global__ void __launch_bounds__(kThreads, 1) bwd256_kernel(const __grid_constant__ Bwd256Params p) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = align_smem_1024(smem_dyn);
  const int item = blockIdx.x;
  if (item < p.n_kv_ctas) pass256<kBf16, kDk>(p, smem, item);
  else if (item < 2 * p.n_kv_ctas) pass256<kBf16, kDv>(p, smem, item - p.n_kv_ctas);
  else pass256<kBf16, kDq>(p, smem, item - 2 * p.n_kv_ctas);
}

struct Plan256 {
  int sq_r, nsplit;
  bool want_dbias;
  bool part;  // dK, dV and column sums leave the main kernel as fp32 partials
  size_t lse2_off, dsum_off, dq_off, part_off, dbpart_off, total;
};

// Query-range splits per key tile: a grid that cannot fill the GPU twice is cut along the query dimension until each of the
// two key passes has about two CTAs per SM (the many short CTAs of the dQ pass, last in the launch, even out what is left);
// every split keeps at least 32 steps. More splits only add partials: 37 instead of 19 at 2048 kept keys write and read 80 MB more.
int pick_nsplit256(const fdma_fwd_params& p) {
  const int64_t ctas = static_cast<int64_t>((p.seqlen_k + kBN - 1) / kBN) * p.h_k * p.b;
  if (ctas >= 2 * sm_count()) return 1;
  const int64_t steps = static_cast<int64_t>((p.seqlen_q + kBM - 1) / kBM) * (p.h / p.h_k);
  const int64_t want = (2 * sm_count() + ctas - 1) / ctas;
  const int64_t cap = std::max<int64_t>(1, steps / 32);
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(std::min(want, cap), 64)));
}

Plan256 plan256(const fdma_bwd_params& bp) {
  const fdma_fwd_params& p = bp.f;
  Plan256 pl;
  pl.sq_r = static_cast<int>(round_up(p.seqlen_q, kBM));
  pl.nsplit = pick_nsplit256(p);
  pl.want_dbias = bp.dbias != nullptr;
  size_t o = 0;
  const size_t rows = static_cast<size_t>(p.b) * p.h * pl.sq_r;
  pl.lse2_off = o; o += align256(rows * 4);
  pl.dsum_off = o; o += align256(rows * 4);
  pl.dq_off = o;
  if (p.seqlen_k > kFlush * kBM) o += align256(static_cast<size_t>(p.b) * p.h * p.seqlen_q * kD * 4);
  pl.part_off = pl.dbpart_off = o;
  pl.part = pl.nsplit > 1 || bp.scatter_pos != nullptr;
  if (pl.part) {
    const size_t keys_r = round_up(p.seqlen_k, kBN);
    o += align256(static_cast<size_t>(2) * pl.nsplit * p.b * p.h_k * keys_r * kD * 4);
    pl.dbpart_off = o;
    if (pl.want_dbias) o += align256(static_cast<size_t>(pl.nsplit) * p.b * p.h_k * keys_r * 4);
  }
  pl.total = o;
  return pl;
}

bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

template <bool kBf16>
int launch256(const fdma_bwd_params& bp, const Plan256& pl, cudaStream_t stream) {
  const fdma_fwd_params& p = bp.f;
  if (!p.workspace || p.workspace_bytes < pl.total) return FDMA_ERR_WORKSPACE;
  char* ws = static_cast<char*>(p.workspace);
  Bwd256Params kp;
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
    st = launch_bwd_prep(a, kD, kBf16, stream);
    if (st) return st;
    st = export_softmax_d(bp, dsum, pl.sq_r, stream);
    if (st) return st;
  }
  kp.mask = static_cast<const uint8_t*>(p.mask);
  kp.bias = p.bias;
  kp.lse2 = lse2;
  kp.dsum = dsum;
  kp.dq = bp.dq;
  kp.dk = bp.dk;
  kp.dv = bp.dv;
  kp.dbias = bp.dbias;
  kp.dq_acc = reinterpret_cast<float*>(ws + pl.dq_off);
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
  // head extents equal to h only occur here with h == h_k (see tc_bwd256_supported): fold them onto h_k
  kp.h_mask = p.h_mask == p.h ? p.h_k : p.h_mask;
  kp.h_bias = p.h_bias == p.h ? p.h_k : p.h_bias;
  kp.dbias_keys = !bp.dbias ? 0 : bp.scatter_pos ? p.seqlen_k : bp.dbias_keys;
  kp.want_dbias = pl.want_dbias ? 1 : 0;
  kp.nsplit = pl.nsplit;
  kp.is_causal = p.is_causal;
  kp.key_pos = p.key_pos;
  kp.pos_batch_stride = p.key_pos_batch_stride; kp.pos_head_stride = p.key_pos_head_stride;
  kp.h_pos = p.h_pos == p.h ? p.h_k : p.h_pos;
  kp.causal_shift = p.causal_shift;
  kp.scale_log2 = p.softmax_scale * kLog2e;
  kp.scale = p.softmax_scale;

  auto kern = bwd256_kernel<kBf16>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem256::kAlloc);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int64_t kv = static_cast<int64_t>((p.seqlen_k + kBN - 1) / kBN) * pl.nsplit * p.h_k * p.b;
  const int64_t ctas = 2 * kv + static_cast<int64_t>((p.seqlen_q + kBN - 1) / kBN) * p.h * p.b;
  if (ctas > 0x7FFFFFFF) return FDMA_ERR_TOO_LARGE;
  kp.n_kv_ctas = static_cast<int>(kv);
  const dim3 grid(static_cast<unsigned>(ctas));
  cudaEvent_t ev0, ev1;
  take_timing_events(&ev0, &ev1);
  if (ev0) cudaEventRecord(ev0, stream);
  kern<<<grid, kThreads, Smem256::kAlloc, stream>>>(kp);
  if (ev1) cudaEventRecord(ev1, stream);
  e = cudaGetLastError();
  if (e != cudaSuccess) return static_cast<int>(e);

  BwdFinishArgs f = {};
  f.b = p.b; f.h = p.h; f.sq = p.seqlen_q; f.sq_r = pl.sq_r; f.d = p.d; f.D = kD;
  f.h_k = p.h_k; f.keys_r = static_cast<int>(round_up(p.seqlen_k, kBN));
  f.rows_out = bp.scatter_pos ? bp.scatter_rows : p.seqlen_k;
  f.pos = bp.scatter_pos; f.pos_sb = bp.scatter_batch_stride; f.pos_sh = bp.scatter_head_stride;
  f.h_pos = bp.scatter_h; f.cap = p.seqlen_k;
  if (pl.part) {
    f.part = kp.dkv_part; f.nsplit = pl.nsplit;
    f.split_stride = static_cast<int64_t>(p.b) * p.h_k * f.keys_r * kD;
    f.dk = bp.dk; f.dk_sb = bp.dk_batch_stride; f.dk_sr = bp.dk_row_stride; f.dk_sh = bp.dk_head_stride;
    f.dv = bp.dv; f.dv_sb = bp.dv_batch_stride; f.dv_sr = bp.dv_row_stride; f.dv_sh = bp.dv_head_stride;
    if (pl.want_dbias) {
      f.db_part = kp.dbias_part; f.db_nsplit = pl.nsplit; f.db_pitch = f.keys_r;
      f.db_split_stride = static_cast<int64_t>(p.b) * p.h_k * f.keys_r;
      f.db_b = bp.dbias_b; f.db_h = bp.dbias_h; f.db_keys = bp.dbias_keys;
      f.dbias = bp.dbias; f.db_sb = bp.dbias_batch_stride; f.db_sh = bp.dbias_head_stride;
    }
  }
  return launch_bwd_finish(f, kBf16, false, stream);
}

}  // namespace

// Head dims above 128 on the tensor-core backward: row-broadcast mask and bias with one row per kv head at most, dBias (if
// asked for) of shape (B, h_k, 1, keys); everything else at this head dim stays on the CUDA-core kernels.
bool tc_bwd256_supported(const fdma_bwd_params& bp) {
  const fdma_fwd_params& p = bp.f;
  if (tile_head_dim(p.d) != kD || !tc_fwd_supported(p)) return false;
  if (p.h_k > 65535 || p.b > 65535) return false;
  const int G = p.h / p.h_k;
  const bool mask_b = !p.mask || p.mask_row_stride == 0 || p.seqlen_q == 1;
  const bool bias_b = !p.bias || p.bias_row_stride == 0 || p.seqlen_q == 1;
  if (!mask_b || !bias_b) return false;
  if (G > 1 && ((p.mask && p.h_mask == p.h) || (p.bias && p.h_bias == p.h))) return false;
  if (p.key_pos && p.is_causal && p.h_pos == p.h && G > 1) return false;
  if (bp.dbias) {
    if (!p.bias) return false;
    const bool colsum = bp.dbias_b == p.b && bp.dbias_rows == 1 && (bp.dbias_h == p.h_k || (bp.dbias_h == p.h && G == 1));
    if (!colsum) return false;
  }
  const void* ptrs[4] = {bp.dout, bp.dq, bp.dk, bp.dv};
  for (const void* x : ptrs)
    if (!aligned16(x)) return false;
  const int64_t strides[12] = {bp.do_batch_stride, bp.do_row_stride, bp.do_head_stride, bp.dq_batch_stride,
                               bp.dq_row_stride,   bp.dq_head_stride, bp.dk_batch_stride, bp.dk_row_stride,
                               bp.dk_head_stride,  bp.dv_batch_stride, bp.dv_row_stride,  bp.dv_head_stride};
  for (int64_t s : strides)
    if (s % 8) return false;
  return true;
}

size_t tc_bwd256_workspace_bytes(const fdma_bwd_params& bp) { return plan256(bp).total; }

int tc_bwd256(const fdma_bwd_params& bp, cudaStream_t stream) {
  const Plan256 pl = plan256(bp);
  return bp.f.dtype == FDMA_BF16 ? launch256<true>(bp, pl, stream) : launch256<false>(bp, pl, stream);
}

}  // namespace fdma
