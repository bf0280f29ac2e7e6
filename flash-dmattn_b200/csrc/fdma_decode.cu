// Single-query (decode) forward: HBM-bound, so the unit of work is the KEPT KEY ROW.
//
// The reference runs decode through its split-KV kernel (csrc/flash_sparse_attn/src/flash_fwd_kernel.h:808-1587,
// merge :1618-1813) and, at 64- or 128-key tiles, streams every K/V row because a top-w mask leaves some kept key
// in nearly every tile. Here the kernel walks the ascending list of kept positions -- the one the selection kernel wrote
// (fdma_decode_kept), one derived from a bool mask first (fdma_fwd with a mask), or the identity (no mask) -- and reads
// only those rows of K and V, once per kv head: the query heads that share a kv head (up to 16) are the M rows of
// mma.sync.m16n8k16.
//
// What bounds it is DRAM: scattered 256-byte rows can be read at 6.2 TB/s on a B200 (95 % of a copy) as long as each SM has
// some 50 KB of whole-row requests in flight all the time, which decides the design:
//  * K and V rows travel to shared memory with cp.async, a row per 16 lanes at d = 128 (register loads in the fragments'
//    own 64-byte pieces reached only half the bandwidth), in a ring of two 16-key stages per warp: 12 warps per SM at
//    d = 128, each with one stage (8 KB) in flight while it works on the other. ldmatrix (transposed for V) forms the
//    fragments. 16 keys fill the k = 16 of P V; with 8-key stages the instructions per key doubled and bound the kernel.
//  * the list, not the key range, is divided: every warp gets the same number of kept rows.
//  * the warps' partial results are combined in shared memory and over the CTAs of a cluster through distributed shared
//    memory; only lists too long for one cluster per (batch, kv head) go through scratch and a second kernel.
// B = 32, 65536 keys, 4096 kept, 8 kv heads x 4, d = 128 (0.537 GB of rows): 206 us with the mask-scanning predecessor and
// its merge kernel, 121 us (4.4 TB/s) now; one sequence of 4097 keys, 1024 kept: 33 -> 7.6 us. Left: the scattered biases
// (16 us) and the products between two stages (15 us).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>

#include "fdma_internal.h"

namespace fdma {
namespace {

namespace cg = cooperative_groups;

constexpr int kChunk = 16;        // kept rows per warp and stage
constexpr int kStages = 2;        // ring depth
constexpr int kWarps = 4;         // per CTA
constexpr int kThreads = kWarps * 32;
constexpr int kMaxCluster = 8;
constexpr float kLog2e = 1.4426950408889634f;

// NJ: 32-wide blocks of the head dim
template <int NJ>
struct Ring {
  static constexpr int kRowBytes = NJ * 64 + 16;  // +16: the eight rows of an ldmatrix tile fall into different banks
  static constexpr int kStageBytes = 2 * kChunk * kRowBytes;  // K rows, then V rows
  static constexpr int kWarpBytes = kStages * kStageBytes;
  static constexpr int kLanesPerRow = NJ <= 2 ? 8 : NJ <= 4 ? 16 : 32;  // 16-byte pieces of a row
};

struct DecodeParams {
  const uint16_t *q, *k, *v, *bias;
  const int32_t* pos;    // kept positions, ascending, or null: slot i is key i
  const int32_t* count;  // kept keys per list, or null: all `slots`
  uint16_t* out;
  float* lse;
  float* partial;        // nsplit > 1: (B, H, nsplit, D + 2) fp32: acc[D], max (log2 units), sum
  int64_t q_sb, q_sh, k_sb, k_sh, v_sb, v_sh, o_sb, o_sh;
  int k_sr, v_sr;        // row strides in elements, below 2^31: one widening multiply per address
  int64_t pos_sb, pos_sh, count_sb, count_sh, bias_sb, bias_sh;
  int h, h_k, h_pos, h_bias, d, seqlen_k, slots, nsplit;
  int row_align;         // kPieces: bytes K and V rows are aligned to
  int heads;             // query heads per CTA
  int head_blocks;       // CTA rows per (batch, split)
  float scale_log2;
};

__device__ __forceinline__ uint32_t smem_addr(const void* x) { return static_cast<uint32_t>(__cvta_generic_to_shared(x)); }
// K / V rows are read once: they leave L2 first, so that the biases (and the lists) stay there
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t x;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(x));
  return x;
}
__device__ __forceinline__ void cp_async16(uint32_t smem, const void* gmem, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(smem), "l"(gmem), "l"(policy) : "memory");
}
// 16 bytes of a row whose pieces are aligned to `align` (4 or 8) bytes only
__device__ __forceinline__ void cp_async16_in_pieces(uint32_t smem, const void* gmem, int align) {
  const char* g = static_cast<const char*>(gmem);
  if (align == 8) {
#pragma unroll
    for (int o = 0; o < 16; o += 8)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem + o), "l"(g + o) : "memory");
  } else {
#pragma unroll
    for (int o = 0; o < 16; o += 4)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem + o), "l"(g + o) : "memory");
  }
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool kBf16>
__device__ __forceinline__ void mma_16816(float (&c)[2], float (&c8)[2], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  if (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c8[0]), "+f"(c8[1]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c8[0]), "+f"(c8[1]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if (kBf16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <bool kBf16>
__device__ __forceinline__ float raw_to_f(uint16_t u) {
  if (kBf16) return __uint_as_float(static_cast<uint32_t>(u) << 16);
  return __half2float(__ushort_as_half(u));
}
template <bool kBf16>
__device__ __forceinline__ uint16_t f_to_raw(float x) {
  if (kBf16) return __bfloat16_as_ushort(__float2bfloat16_rn(x));
  return __half_as_ushort(__float2half_rn(x));
}
// (lo, hi) as 16-bit values, and what that leaves of them: three in a row add up to all 24 significant bits of a number (bf16:
// 3 x 8; fp16: 3 x 11, cut at 2^-24).
template <bool kBf16>
__device__ __forceinline__ uint32_t split_off2(float& lo, float& hi) {
  const uint32_t u = pack2<kBf16>(lo, hi);
  lo -= raw_to_f<kBf16>(static_cast<uint16_t>(u & 0xFFFFu));
  hi -= raw_to_f<kBf16>(static_cast<uint16_t>(u >> 16));
  return u;
}
__device__ __forceinline__ float exp2_or_zero(float x) { return x == -CUDART_INF_F ? 0.f : exp2f(x); }

// kM16: 9 to 16 query heads (both halves of the M rows of the products), else up to 8. Fragments of mma.m16n8k16
// (g = lane / 4, c = lane % 4): A row g (+ 8), k = 2c, 2c+1 (+ 8); B k = 2c, 2c+1 (+ 8), n = g; C row g (+ 8), n = 2c, 2c+1.
// kPieces: K / V rows that are aligned to 4 or 8 bytes only.
template <int NJ, bool kBf16, bool kM16, bool kPieces>
__global__ void __launch_bounds__(kThreads, NJ <= 4 && !kPieces ? 3 : 1) decode_rows_kernel(const DecodeParams p) {
  using L = Ring<NJ>;
  constexpr int D = NJ * 32;
  constexpr int kHalves = kM16 ? 2 : 1;
  constexpr int kHeads = 8 * kHalves;
  // Head dims above 128, and rows in pieces: the probabilities keep their 32 bits, as sums of three 16-bit values with a product
  // each. fp16 holds them times 2^14, away from its smallest numbers. (8 x 65536 keys, 4096 kept, 32 heads over 8, d = 256: 104 us with 16-bit
  // probabilities, which are 15 % further from the exact result, 113 us so.)
  constexpr int kTerms = D > 128 || kPieces ? 3 : 1;
  constexpr float kPScale = kTerms > 1 && !kBf16 ? 16384.f : 1.f;
  extern __shared__ __align__(16) unsigned char s_dyn[];  // the warps' rings; afterwards [kWarps][kHeads][D] fp32 partials
  __shared__ uint32_t s_q[kHalves][2 * NJ][2][32];        // A fragments of Q, one word per lane
  __shared__ float s_m[kWarps][kHeads], s_l[kWarps][kHeads];
  __shared__ float s_cm[kHeads], s_cl[kHeads];            // this CTA's max and sum
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = cluster.block_rank(), nrank = cluster.num_blocks();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const int b = blockIdx.z, hb = blockIdx.y % p.head_blocks, split = blockIdx.y / p.head_blocks;
  const int group = p.h / p.h_k;
  // a CTA's heads all belong to one kv head
  const int blocks_per_kv = p.head_blocks / p.h_k;
  const int hk = hb / blocks_per_kv;
  const int h0 = hk * group + (hb - hk * blocks_per_kv) * p.heads;
  const int nh = min(p.heads, (hk + 1) * group - h0);
  const int hp = p.h_pos == p.h ? h0 : (p.h_pos == p.h_k ? hk : 0);
  const int32_t* pos_row = p.pos ? p.pos + b * p.pos_sb + hp * p.pos_sh : nullptr;
  const int n_keys = p.count ? min(p.count[b * p.count_sb + hp * p.count_sh], p.slots) : p.slots;
  const int sub = lane / L::kLanesPerRow, piece = lane % L::kLanesPerRow;
  const bool in = piece * 8 < p.d;
  const uint16_t* krow = p.k + b * p.k_sb + hk * p.k_sh + piece * 8;
  const uint16_t* vrow = p.v + b * p.v_sb + hk * p.v_sh + piece * 8;
  const int64_t k_sr = p.k_sr, v_sr = p.v_sr;
  const uint32_t ring = smem_addr(s_dyn) + warp * L::kWarpBytes;

  // Q fragments, the same for every warp
  for (int i = warp; i < kHalves * 2 * NJ; i += kWarps) {
    const int t = i / (2 * NJ), ks = i - t * 2 * NJ, head = g + 8 * t;
    const uint16_t* qp = p.q + b * p.q_sb + (h0 + min(head, nh - 1)) * p.q_sh;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int dd = ks * 16 + e * 8 + c * 2;
      s_q[t][ks][e][lane] = head < nh && dd < p.d ? *reinterpret_cast<const uint32_t*>(qp + dd) : 0u;
    }
  }
  // columns beyond the head dim stay zero in every stage
  if (p.d < L::kLanesPerRow * 8)
    for (int i = lane; i < L::kWarpBytes / 16; i += 32)
      reinterpret_cast<uint4*>(s_dyn + warp * L::kWarpBytes)[i] = make_uint4(0, 0, 0, 0);
  const uint16_t* bias_row[kHalves];
#pragma unroll
  for (int t = 0; t < kHalves; ++t) {
    const int head = h0 + min(g + 8 * t, nh - 1);
    bias_row[t] = p.bias ? p.bias + b * p.bias_sb + (p.h_bias == p.h ? head : (p.h_bias == p.h_k ? hk : 0)) * p.bias_sh : nullptr;
  }
  float o[kHalves][4 * NJ][2];  // O[head g + 8 t][8 nt + 2c + {0, 1}]
  float m[kHalves], l[kHalves];  // running max of the head; this LANE's share of the sum
#pragma unroll
  for (int t = 0; t < kHalves; ++t) {
    m[t] = -CUDART_INF_F;
    l[t] = 0.f;
#pragma unroll
    for (int nt = 0; nt < 4 * NJ; ++nt) o[t][nt][0] = o[t][nt][1] = 0.f;
  }
  float zero[2] = {0.f, 0.f};  // rows 8-15 of the accumulators when they are not heads: always zero, one shared pair
  __syncthreads();

  // chunks of 16 slots, contiguous per warp
  const int n_chunks = (n_keys + kChunk - 1) / kChunk;
  const int n_warps = p.nsplit * nrank * kWarps;
  const int per_warp = (n_chunks + n_warps - 1) / n_warps;
  const int first = ((split * nrank + rank) * kWarps + warp) * per_warp;
  const int n = max(0, min(per_warp, n_chunks - first));
  // Positions of the 32 slots from chunk i of this warp on. Nothing here or in `issue` touches a loaded value before the
  // stage that needs it: a comparison beside the load made every stage wait for it.
  auto load_pos = [&](int i) {
    const int slot = (first + i) * kChunk + lane;
    return slot < n_keys && i < n ? (pos_row ? __ldg(pos_row + slot) : slot) : -1;
  };
  int my_pos = -1, next_pos = load_pos(0);
  const uint64_t policy = evict_first_policy();
  // Per stage and lane (key lane & 15): position and 16-bit bias, the latter -inf where there is no key. One load per lane
  // here and four shuffles where the scores are formed; with every lane loading the biases of its own four scores the
  // kernel took a fifth longer.
  int key_pos[kStages];
  uint16_t key_bias[kStages];
  constexpr uint16_t kNegInf = kBf16 ? 0xFF80u : 0xFC00u;
  const bool head_bias = p.bias && p.h_bias == p.h && group > 1;  // a bias row per query head
  auto issue = [&](int i, int st, int& kp, uint16_t& kb) {
    if ((i & 1) == 0) {
      my_pos = next_pos >= p.seqlen_k ? -1 : next_pos;
      next_pos = load_pos(i + 2);
    }
    const uint32_t dst = ring + st * L::kStageBytes + piece * 16;
    constexpr int kRowsPerCopy = 32 / L::kLanesPerRow;
#pragma unroll
    for (int r0 = 0; r0 < kChunk; r0 += kRowsPerCopy) {
      const int r = r0 + sub;
      const int pos = __shfl_sync(0xffffffffu, my_pos, (i & 1) * kChunk + r);
      if (in) {
        const uint32_t kd = dst + r * L::kRowBytes, vd = kd + kChunk * L::kRowBytes;
        if (pos >= 0) {
          const uint16_t *ks = krow + static_cast<int64_t>(pos) * k_sr, *vs = vrow + static_cast<int64_t>(pos) * v_sr;
          if (kPieces) {
            cp_async16_in_pieces(kd, ks, p.row_align);
            cp_async16_in_pieces(vd, vs, p.row_align);
          } else {
            cp_async16(kd, ks, policy);
            cp_async16(vd, vs, policy);
          }
        } else {
          asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(kd), "r"(0) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(vd), "r"(0) : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    kp = __shfl_sync(0xffffffffu, my_pos, (i & 1) * kChunk + (lane & 15));
    kb = kp < 0 ? kNegInf : p.bias && !head_bias ? __ldg(bias_row[0] + kp) : static_cast<uint16_t>(0);
  };
  auto consume = [&](int st, int kp, uint16_t kb) {
    const uint32_t kst = ring + st * L::kStageBytes, vst = kst + kChunk * L::kRowBytes;
    // K: matrices (rows 0-7 | 8-15) x (two 8-wide pieces); V, transposed: two pieces x (rows 0-7 | 8-15)
    const uint32_t kaddr = kst + ((lane & 7) + (lane & 16 ? 8 : 0)) * L::kRowBytes + (lane & 8 ? 16 : 0);
    const uint32_t vaddr = vst + ((lane & 7) + (lane & 8 ? 8 : 0)) * L::kRowBytes + (lane & 16 ? 16 : 0);
    float s0[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, s8[2][2] = {{0.f, 0.f}, {0.f, 0.f}};  // [keys 0-7 | 8-15]
#pragma unroll
    for (int ks = 0; ks < 2 * NJ; ++ks) {
      uint32_t f[4];
      ldmatrix_x4(f, kaddr + ks * 32);
      const uint32_t q0 = s_q[0][ks][0][lane], q2 = s_q[0][ks][1][lane];
      const uint32_t q1 = kM16 ? s_q[kHalves - 1][ks][0][lane] : 0u, q3 = kM16 ? s_q[kHalves - 1][ks][1][lane] : 0u;
#pragma unroll
      for (int u = 0; u < 2; ++u)
        mma_16816<kBf16>(s0[u], kM16 ? s8[u] : zero, q0, q1, q2, q3, f[2 * u], f[2 * u + 1]);
    }
    const float kbf = raw_to_f<kBf16>(kb) * kLog2e;
    uint32_t pa[kTerms][kHalves][2];
#pragma unroll
    for (int t = 0; t < kHalves; ++t) {
      float x[2][2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int src = u * 8 + 2 * c + e;
          float add = __shfl_sync(0xffffffffu, kbf, src);
          if (head_bias) {
            const int pk = __shfl_sync(0xffffffffu, kp, src);
            if (pk >= 0) add = raw_to_f<kBf16>(__ldg(bias_row[t] + pk)) * kLog2e;
          }
          x[u][e] = fmaf(t == 0 ? s0[u][e] : s8[u][e], p.scale_log2, add);
        }
      float mx = fmaxf(fmaxf(x[0][0], x[0][1]), fmaxf(x[1][0], x[1][1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      if (__any_sync(0xffffffffu, mx > m[t])) {
        const float m_new = fmaxf(m[t], mx);
        const float corr = exp2_or_zero(m[t] - (m_new == -CUDART_INF_F ? 0.f : m_new));
        m[t] = m_new;
        l[t] *= corr;
#pragma unroll
        for (int nt = 0; nt < 4 * NJ; ++nt) {
          o[t][nt][0] *= corr;
          o[t][nt][1] *= corr;
        }
      }
      const float base = m[t] == -CUDART_INF_F ? 0.f : m[t];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float p0 = exp2f(x[u][0] - base), p1 = exp2f(x[u][1] - base);
        l[t] += p0 + p1;
        p0 *= kPScale;
        p1 *= kPScale;
#pragma unroll
        for (int term = 0; term < kTerms; ++term) pa[term][t][u] = split_off2<kBf16>(p0, p1);
      }
    }
#pragma unroll
    for (int j = 0; j < 2 * NJ; ++j) {
      uint32_t f[4];
      ldmatrix_x4_trans(f, vaddr + j * 32);
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int term = kTerms - 1; term >= 0; --term)
          mma_16816<kBf16>(o[0][2 * j + r], kM16 ? o[kHalves - 1][2 * j + r] : zero, pa[term][0][0],
                           kM16 ? pa[term][kHalves - 1][0] : 0u, pa[term][0][1], kM16 ? pa[term][kHalves - 1][1] : 0u, f[2 * r],
                           f[2 * r + 1]);
    }
    __syncwarp();  // every lane has read the stage before it is overwritten
  };
  auto step = [&](int i, int st, int& kp, uint16_t& kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");  // all but the newest stages have landed
    __syncwarp();
    consume(st, kp, kb);
    if (i + kStages < n) issue(i + kStages, st, kp, kb);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int st = 0; st < kStages; ++st) {
    if (st < n) issue(st, st, key_pos[st], key_bias[st]);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int i = 0; i < n; i += kStages) {
#pragma unroll
    for (int st = 0; st < kStages; ++st)
      if (i + st < n) step(i + st, st, key_pos[st], key_bias[st]);
  }

  // ---- warps of the CTA: maxima first, then every warp leaves its rescaled O ----
  float* s_part = reinterpret_cast<float*>(s_dyn);
#pragma unroll
  for (int t = 0; t < kHalves; ++t) {
    l[t] += __shfl_xor_sync(0xffffffffu, l[t], 1);
    l[t] += __shfl_xor_sync(0xffffffffu, l[t], 2);
    if (c == 0) {
      s_m[warp][g + 8 * t] = m[t];
      s_l[warp][g + 8 * t] = l[t];
    }
  }
  __syncthreads();  // (also: the rings are not needed any more)
#pragma unroll
  for (int t = 0; t < kHalves; ++t) {
    const int head = g + 8 * t;
    float cm = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) cm = fmaxf(cm, s_m[w][head]);
    const float base = cm == -CUDART_INF_F ? 0.f : cm;
    const float f = exp2_or_zero(m[t] - base) * (1.f / kPScale);
    if (warp == 0 && c == 0) {
      float cl = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) cl += s_l[w][head] * exp2_or_zero(s_m[w][head] - base);
      s_cm[head] = cm;
      s_cl[head] = cl;
    }
    if (head < nh) {
      float* dst = s_part + (warp * kHeads + head) * D + c * 2;
#pragma unroll
      for (int nt = 0; nt < 4 * NJ; ++nt)
        *reinterpret_cast<float2*>(dst + nt * 8) = make_float2(o[t][nt][0] * f, o[t][nt][1] * f);
    }
  }
  __syncthreads();
  for (int i = tid; i < nh * D; i += kThreads) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) a += s_part[w * kHeads * D + i];
    s_part[i] = a;
  }
  cluster.sync();  // (also orders the CTA's own sums before they are read below)

  // ---- CTAs of the cluster: each takes its share of the head's elements ----
  const int total = nh * D, share = (total + nrank - 1) / nrank;
  for (int i = rank * share + tid; i < min(total, (rank + 1) * share); i += kThreads) {
    const int head = i / D, dd = i - head * D;
    float M = -CUDART_INF_F;
    for (int r = 0; r < nrank; ++r) M = fmaxf(M, *cluster.map_shared_rank(&s_cm[head], r));
    const float base = M == -CUDART_INF_F ? 0.f : M;
    float acc = 0.f, sum = 0.f;
    for (int r = 0; r < nrank; ++r) {
      const float f = exp2_or_zero(*cluster.map_shared_rank(&s_cm[head], r) - base);
      sum += f * *cluster.map_shared_rank(&s_cl[head], r);
      acc += f * *cluster.map_shared_rank(&s_part[i], r);
    }
    const int h = h0 + head;
    if (p.nsplit > 1) {
      float* dst = p.partial + ((static_cast<int64_t>(b) * p.h + h) * p.nsplit + split) * (D + 2);
      dst[dd] = acc;
      if (dd == 0) {
        dst[D] = M;
        dst[D + 1] = sum;
      }
    } else {
      if (dd < p.d) p.out[b * p.o_sb + h * p.o_sh + dd] = f_to_raw<kBf16>(sum > 0.f ? acc / sum : 0.f);
      if (dd == 0) p.lse[static_cast<int64_t>(b) * p.h + h] = sum > 0.f ? (M + log2f(sum)) * 0.6931471805599453f : CUDART_INF_F;
    }
  }
  cluster.sync();  // nobody leaves while its shared memory may still be read
}

// O = sum_i 2^(m_i - M) acc_i / sum_i 2^(m_i - M) l_i, LSE = (M + log2(sum)) * ln2 over the P <= 32 splits; one CTA of D
// threads per (b, h).
template <bool kBf16>
__global__ void decode_merge_kernel(const float* __restrict__ partial, uint16_t* __restrict__ out, float* __restrict__ lse,
                                    int H, int P, int D, int d, int64_t ob, int64_t oh) {
  const int w = blockIdx.x, h = w % H, b = w / H, dd = threadIdx.x;
  const float* base = partial + static_cast<int64_t>(w) * P * (D + 2);
  float M = -CUDART_INF_F;
  for (int i = 0; i < P; ++i) M = fmaxf(M, base[i * (D + 2) + D]);
  float L = 0.f, a = 0.f;
  for (int i = 0; i < P; ++i) {
    const float f = exp2_or_zero(base[i * (D + 2) + D] - (M == -CUDART_INF_F ? 0.f : M));
    L += f * base[i * (D + 2) + D + 1];
    a = fmaf(f, base[i * (D + 2) + dd], a);
  }
  if (dd < d) out[b * ob + h * oh + dd] = f_to_raw<kBf16>(L > 0.f ? a / L : 0.f);
  if (dd == 0) lse[w] = L > 0.f ? (M + log2f(L)) * 0.6931471805599453f : CUDART_INF_F;
}

int blocks_of(int d) { return d <= 64 ? 2 : d <= 96 ? 3 : d <= 128 ? 4 : 8; }  // instantiated NJ

struct DecodePlan {
  int heads, head_blocks;  // query heads per CTA, CTA rows per (batch, split)
  int cluster, nsplit;
  int list_h;              // bool mask: heads of the position list derived from it
  size_t pos_off, count_off, part_off, total;
};

// `slots`: length of the list (an upper bound for one derived from a bool mask).
DecodePlan plan(const fdma_fwd_params& p, int slots, int h_pos, bool index) {
  DecodePlan pl;
  const int group = p.h / p.h_k;
  // heads share a pass over the rows unless every query head has a list of its own
  // (at d > 128 the accumulators of 16 heads would not fit the registers: at most 8 there)
  pl.heads = h_pos == p.h && group > 1 ? 1 : std::min(group, p.d > 128 ? 8 : 16);
  pl.head_blocks = p.h_k * ((group + pl.heads - 1) / pl.heads);
  const int64_t units = static_cast<int64_t>(p.b) * pl.head_blocks;
  // CTAs per list: a launch lasts about (waves of resident CTAs) x (rows per warp + 48), where 48 rows stand for a CTA's
  // set-up and combination; every warp keeps at least one stage of rows. Beyond one cluster per list the partials go
  // through scratch and a merge kernel (3 us, about 300 rows).
  const int resident = (p.d <= 128 ? 3 : 1) * sm_count();
  double best = 1e30;
  pl.cluster = pl.nsplit = 1;
  for (int ns = 1; ns <= 32; ns *= 2)
    for (int c = ns == 1 ? 1 : kMaxCluster; c <= kMaxCluster; c *= 2) {
      const int64_t ctas = units * c * ns;
      const int rows = (slots + c * ns * kWarps - 1) / (c * ns * kWarps);
      if (rows < kChunk && ns * c > 1) continue;
      const double waves = std::max(1.0, static_cast<double>(ctas) / resident);
      // a partly filled last wave counts in full while it is one of few, less as CTAs spread out over many
      const double cost = (waves + (std::ceil(waves) - waves) * 0.5) * (rows + 48) + (ns > 1 ? 300 : 0);
      if (cost < best) {
        best = cost;
        pl.cluster = c;
        pl.nsplit = ns;
      }
    }
  size_t o = 0;
  pl.list_h = p.h_mask;
  pl.pos_off = o;
  if (index) o += align256(static_cast<size_t>(p.b) * p.h_mask * round_up(p.seqlen_k, kKeyPad) * 4);
  pl.count_off = o;
  if (index) o += align256(static_cast<size_t>(p.b) * p.h_mask * 4);
  pl.part_off = o;
  if (pl.nsplit > 1) o += align256(static_cast<size_t>(p.b) * p.h * pl.nsplit * (blocks_of(p.d) * 32 + 2) * sizeof(float));
  pl.total = o;
  return pl;
}

template <int NJ, bool kBf16, bool kM16, bool kPieces>
int launch(const DecodeParams& dp, const DecodePlan& pl, int batch, cudaStream_t stream) {
  auto kern = decode_rows_kernel<NJ, kBf16, kM16, kPieces>;
  constexpr int parts = kWarps * (kM16 ? 16 : 8) * NJ * 32 * static_cast<int>(sizeof(float));
  constexpr int smem = std::max(parts, kWarps * Ring<NJ>::kWarpBytes);
  if (smem > 40 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pl.cluster, pl.head_blocks * pl.nsplit, batch);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pl.cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, kern, dp));
}
template <int NJ, bool kPieces>
int launch_nj(const DecodeParams& dp, const DecodePlan& pl, int batch, bool bf16, cudaStream_t stream) {
  constexpr bool kM16 = NJ <= 4;
  if (kM16 && pl.heads > 8)
    return bf16 ? launch<NJ, true, kM16, kPieces>(dp, pl, batch, stream) : launch<NJ, false, kM16, kPieces>(dp, pl, batch, stream);
  return bf16 ? launch<NJ, true, false, kPieces>(dp, pl, batch, stream) : launch<NJ, false, false, kPieces>(dp, pl, batch, stream);
}

// Bytes that every row of K and V is aligned to: 16, 8, 4 or 2.
int row_align(const fdma_fwd_params& p) {
  uint64_t x = reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v);
  if (p.seqlen_k > 1) x |= static_cast<uint64_t>(p.k_row_stride | p.v_row_stride) * 2;
  if (p.h_k > 1) x |= static_cast<uint64_t>(p.k_head_stride | p.v_head_stride) * 2;
  if (p.b > 1) x |= static_cast<uint64_t>(p.k_batch_stride | p.v_batch_stride) * 2;
  return x % 16 == 0 ? 16 : x % 8 == 0 ? 8 : x % 4 == 0 ? 4 : 2;
}

int run(const fdma_fwd_params& p, const DecodePlan& pl, const int32_t* pos, int64_t pos_sb, int64_t pos_sh, int h_pos,
        const int32_t* count, int64_t count_sb, int64_t count_sh, int slots, cudaStream_t stream) {
  DecodeParams dp = {};
  dp.q = static_cast<const uint16_t*>(p.q); dp.k = static_cast<const uint16_t*>(p.k);
  dp.v = static_cast<const uint16_t*>(p.v); dp.bias = static_cast<const uint16_t*>(p.bias);
  dp.out = static_cast<uint16_t*>(p.out); dp.lse = p.lse;
  dp.partial = pl.nsplit > 1 ? reinterpret_cast<float*>(static_cast<char*>(p.workspace) + pl.part_off) : nullptr;
  dp.pos = pos; dp.pos_sb = pos_sb; dp.pos_sh = pos_sh; dp.h_pos = h_pos;
  dp.count = count; dp.count_sb = count_sb; dp.count_sh = count_sh;
  dp.q_sb = p.q_batch_stride; dp.q_sh = p.q_head_stride;
  dp.k_sb = p.k_batch_stride; dp.k_sr = static_cast<int>(p.k_row_stride); dp.k_sh = p.k_head_stride;
  dp.v_sb = p.v_batch_stride; dp.v_sr = static_cast<int>(p.v_row_stride); dp.v_sh = p.v_head_stride;
  dp.o_sb = p.o_batch_stride; dp.o_sh = p.o_head_stride;
  dp.bias_sb = p.bias_batch_stride; dp.bias_sh = p.bias_head_stride;
  dp.h = p.h; dp.h_k = p.h_k; dp.h_bias = p.h_bias; dp.d = p.d; dp.seqlen_k = p.seqlen_k;
  dp.slots = slots; dp.nsplit = pl.nsplit; dp.heads = pl.heads; dp.head_blocks = pl.head_blocks;
  dp.scale_log2 = p.softmax_scale * kLog2e;
  dp.row_align = row_align(p);
  const bool pieces = dp.row_align < 16;
  const bool bf16 = p.dtype == FDMA_BF16;
  cudaEvent_t ev0, ev1;
  take_timing_events(&ev0, &ev1);
  if (ev0) cudaEventRecord(ev0, stream);
  int st;
  switch (blocks_of(p.d)) {
    case 2: st = pieces ? launch_nj<2, true>(dp, pl, p.b, bf16, stream) : launch_nj<2, false>(dp, pl, p.b, bf16, stream); break;
    case 3: st = launch_nj<3, false>(dp, pl, p.b, bf16, stream); break;
    case 4: st = pieces ? launch_nj<4, true>(dp, pl, p.b, bf16, stream) : launch_nj<4, false>(dp, pl, p.b, bf16, stream); break;
    default: st = launch_nj<8, false>(dp, pl, p.b, bf16, stream); break;
  }
  if (ev1) cudaEventRecord(ev1, stream);
  if (st || pl.nsplit == 1) return st;
  const int D = blocks_of(p.d) * 32;
  if (bf16) decode_merge_kernel<true><<<p.b * p.h, D, 0, stream>>>(dp.partial, dp.out, dp.lse, p.h, pl.nsplit, D, p.d, dp.o_sb, dp.o_sh);
  else decode_merge_kernel<false><<<p.b * p.h, D, 0, stream>>>(dp.partial, dp.out, dp.lse, p.h, pl.nsplit, D, p.d, dp.o_sb, dp.o_sh);
  return static_cast<int>(cudaGetLastError());
}

// heads of the lists: per query head only where the mask is
int mask_list_heads(const fdma_fwd_params& p) { return p.mask ? p.h_mask : 1; }

}  // namespace

bool decode_supported(const fdma_fwd_params& p) {
  if (p.seqlen_q != 1 || p.seqlen_k <= 0 || p.d % 8 || p.d > 256) return false;
  if (p.mask && p.mask_bits) return false;
  // K and V rows are read in 16-byte pieces, at head dims 64 and 128 also in 4- and 8-byte ones; Q in 4-byte words
  const int align = row_align(p);
  if (align < 16 && !((p.d == 64 || p.d == 128) && align >= 4)) return false;
  if ((reinterpret_cast<uintptr_t>(p.q) & 3u) || p.q_batch_stride % 2 || p.q_head_stride % 2) return false;
  if (p.k_row_stride < 0 || p.k_row_stride > 0x7FFFFFFF || p.v_row_stride < 0 || p.v_row_stride > 0x7FFFFFFF) return false;
  return p.b <= 65535 && p.h <= 2047;  // grid limits: head rows x up to 32 splits in y
}

size_t decode_workspace_bytes(const fdma_fwd_params& p) {
  return plan(p, p.seqlen_k, mask_list_heads(p), p.mask != nullptr).total;
}

int decode_fwd(const fdma_fwd_params& p, cudaStream_t stream) {
  const DecodePlan pl = plan(p, p.seqlen_k, mask_list_heads(p), p.mask != nullptr);
  if (pl.total && (!p.workspace || p.workspace_bytes < pl.total)) return FDMA_ERR_WORKSPACE;
  if (!p.mask) return run(p, pl, nullptr, 0, 0, 1, nullptr, 0, 0, p.seqlen_k, stream);
  // a bool mask from elsewhere: its position lists first (rows of a broadcast batch are indexed once per batch element)
  char* ws = static_cast<char*>(p.workspace);
  int32_t* pos = reinterpret_cast<int32_t*>(ws + pl.pos_off);
  int32_t* count = reinterpret_cast<int32_t*>(ws + pl.count_off);
  const int cap = static_cast<int>(round_up(p.seqlen_k, kKeyPad));
  fdma_compact_params cp = {};
  cp.mask = p.mask;
  cp.mask_batch_stride = p.mask_batch_stride; cp.mask_head_stride = p.mask_head_stride;
  cp.b_mask = p.b; cp.h_mask = p.h_mask; cp.seqlen_k = p.seqlen_k; cp.capacity = cap;
  cp.key_pos = pos; cp.count = count;
  const int st = fdma_compact_index(&cp, stream);
  if (st) return st;
  return run(p, pl, pos, static_cast<int64_t>(p.h_mask) * cap, cap, p.h_mask, count, p.h_mask, p.h_mask == 1 ? 0 : 1,
             p.seqlen_k, stream);
}

// The same for a bool mask in less scratch than the position lists of all rows take: one batch element and as many mask heads
// at a time as fit, one after the other. FDMA_ERR_WORKSPACE when a single row's list does not fit.
int decode_fwd_sliced(const fdma_fwd_params& p, cudaStream_t stream) {
  const int group = p.h / p.h_k, per_mask = p.h / p.h_mask;  // query heads per kv head, per mask head
  auto slice = [&](int b, int m0, int m) {  // mask heads [m0, m0 + m): whole kv heads, or part of one
    const int h0 = m0 * per_mask, hk0 = h0 / group;
    fdma_fwd_params s = p;
    s.b = 1;
    s.h = m * per_mask;
    s.h_k = std::max(1, s.h / group);
    s.h_mask = m;
    s.q = static_cast<const uint16_t*>(p.q) + b * p.q_batch_stride + h0 * p.q_head_stride;
    s.k = static_cast<const uint16_t*>(p.k) + b * p.k_batch_stride + hk0 * p.k_head_stride;
    s.v = static_cast<const uint16_t*>(p.v) + b * p.v_batch_stride + hk0 * p.v_head_stride;
    s.out = static_cast<uint16_t*>(p.out) + b * p.o_batch_stride + h0 * p.o_head_stride;
    s.lse = p.lse + static_cast<int64_t>(b) * p.h + h0;
    s.mask = static_cast<const uint8_t*>(p.mask) + b * p.mask_batch_stride + m0 * p.mask_head_stride;
    if (p.bias) {
      const int bias_head = p.h_bias == p.h ? h0 : p.h_bias == p.h_k ? hk0 : 0;
      s.bias = static_cast<const uint16_t*>(p.bias) + b * p.bias_batch_stride + bias_head * p.bias_head_stride;
      s.h_bias = p.h_bias == p.h ? s.h : p.h_bias == p.h_k ? s.h_k : 1;
    }
    return s;
  };
  const int lists_per_kv = std::max(1, p.h_mask / p.h_k);  // mask heads that make up a kv head
  int m = p.h_mask;
  while (decode_workspace_bytes(slice(0, 0, m)) > p.workspace_bytes) {
    if (m == 1) return FDMA_ERR_WORKSPACE;
    if (m > lists_per_kv) {
      m = std::max(lists_per_kv, m / 2 / lists_per_kv * lists_per_kv);
    } else {
      do --m;
      while (lists_per_kv % m);
    }
  }
  for (int b = 0; b < p.b; ++b)
    for (int m0 = 0; m0 < p.h_mask; m0 += m) {
      const int st = decode_fwd(slice(b, m0, std::min(m, p.h_mask - m0)), stream);
      if (st) return st;
    }
  return 0;
}

}  // namespace fdma

using namespace fdma;

extern "C" size_t fdma_decode_kept_workspace_bytes(const fdma_decode_params* p) {
  if (!p || p->f.b <= 0 || p->f.h <= 0 || p->f.h_k <= 0 || p->f.d <= 0 || p->kept_capacity <= 0) return 0;
  return plan(p->f, p->kept_capacity, p->kept_h, false).total;
}

extern "C" int fdma_decode_kept(const fdma_decode_params* p, void* stream) {
  if (!p) return FDMA_ERR_BAD_ARG;
  fdma_fwd_params f = p->f;
  if (!f.q || !f.k || !f.v || !f.out || !f.lse || !p->kept_pos || p->kept_capacity <= 0) return FDMA_ERR_BAD_ARG;
  if (f.b <= 0 || f.seqlen_k <= 0 || f.h <= 0 || f.h_k <= 0 || f.d <= 0 || f.h % f.h_k) return FDMA_ERR_BAD_ARG;
  if (p->kept_h != 1 && p->kept_h != f.h_k && p->kept_h != f.h) return FDMA_ERR_BAD_ARG;
  if (f.bias && f.h_bias != 1 && f.h_bias != f.h_k && f.h_bias != f.h) return FDMA_ERR_BAD_ARG;
  if (f.dtype != FDMA_BF16 && f.dtype != FDMA_FP16) return FDMA_ERR_UNSUPPORTED;
  f.mask = nullptr;
  if (!f.bias) f.h_bias = 1;
  if (!decode_supported(f)) return FDMA_ERR_UNSUPPORTED;
  const DecodePlan pl = plan(f, p->kept_capacity, p->kept_h, false);
  if (pl.total && (!f.workspace || f.workspace_bytes < pl.total)) return FDMA_ERR_WORKSPACE;
  return run(f, pl, p->kept_pos, p->kept_batch_stride, p->kept_head_stride, p->kept_h, p->kept_count, p->count_batch_stride,
             p->count_head_stride, p->kept_capacity, static_cast<cudaStream_t>(stream));
}
