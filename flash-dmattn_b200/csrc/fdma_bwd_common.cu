// The two small kernels on either side of every tensor-core backward kernel (head dims 64, 128, 256):
//   bwd_prep_kernel    D = rowsum(dO o O), LSE in log2 units, and the zero fill of the fp32 dQ accumulator (head dims up to 128)
//   bwd_finish_kernel  dQ accumulator -> 16-bit dQ; sum of the query-range partials -> 16-bit dK, dV; fp32 column sums
//                      -> 16-bit dBias; for gathered keys every gradient row goes straight to its key's position and all
//                      other rows are written as zeros
// Both are bound by HBM. Each does in ONE launch what used to take several (a memset node and a kernel before; three
// reductions, a conversion, three memsets and three scatters after): for small calls the launches were the time, for
// large ones the gathered gradients made one more trip through memory. Measured on a B200: training step at S = 256
// (2 heads) 27 launches -> 8; zero fill + scatter of dK / dV / dBias at S = 32768 (8 kv heads) 58 us -> 32 us.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>

#include "fdma_internal.h"
#include "fdma_ptx.cuh"

namespace fdma {
namespace {

constexpr int kThreads = 256;
// Gradient rows (key positions) per CTA of the finish kernel. Gathered keys: most rows are zeros, and a larger CTA makes
// fewer searches in the position list (193 us against 204 at 8 x 32768 rows). All rows summed from partials: 32 leave too
// few CTAs in flight to cover the latency of the sums (95 us against 48 at 8 x 4096 keys, 5 splits).
constexpr int kRowsGathered = 32, kRowsAll = 8;
constexpr int kHeads = 16;  // kv heads per CTA of the finish kernel
constexpr float kLog2e = 1.4426950408889634f;

template <bool kBf16>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if (kBf16) return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
  const __half2 h = *reinterpret_cast<const __half2*>(&u);
  return make_float2(__low2float(h), __high2float(h));
}

// One warp per eight consecutive query rows of one (b, h); D / 8 lanes hold a row (16 B each), all loads issued up
// front. Rows [Sq, Sq_r) are padding (LSE = +inf, D = 0). The dQ accumulator rows of the warp are zeroed on the way.
template <int D, bool kBf16>
__global__ void __launch_bounds__(kThreads) bwd_prep_kernel(const BwdPrepArgs a) {
  constexpr int kLanes = D / 8, kPerPass = 32 / kLanes, kPasses = 8 / kPerPass;
  const int lane = threadIdx.x & 31, sub = lane / kLanes, l = lane % kLanes;
  const uint32_t w = (blockIdx.x * kThreads + threadIdx.x) >> 5;
  const uint32_t groups = a.sq_r / 8;
  if (w >= groups * a.h * a.b) return;
  const uint32_t bh = w / groups;
  const int q0 = static_cast<int>(w - bh * groups) * 8;
  const int h = bh % a.h, b = bh / a.h;
  const uint16_t* o = static_cast<const uint16_t*>(a.out) + b * a.o_sb + h * a.o_sh + l * 8;
  const uint16_t* g = static_cast<const uint16_t*>(a.dout) + b * a.do_sb + h * a.do_sh + l * 8;
  uint4 x[kPasses], y[kPasses];
#pragma unroll
  for (int u = 0; u < kPasses; ++u) {
    const int q = q0 + u * kPerPass + sub;
    x[u] = y[u] = make_uint4(0, 0, 0, 0);
    if (q < a.sq && l * 8 < a.d) {
      x[u] = *reinterpret_cast<const uint4*>(o + static_cast<int64_t>(q) * a.o_sr);
      y[u] = *reinterpret_cast<const uint4*>(g + static_cast<int64_t>(q) * a.do_sr);
    }
  }
  if (D <= 128 && a.dq_acc) {  // accumulator rows of this warp: (B,H,Sq,D) elements of acc_bytes each
    char* base = static_cast<char*>(a.dq_acc) + (static_cast<int64_t>(bh) * a.sq + q0) * D * a.acc_bytes;
    const int n16 = min(8, a.sq - q0) * D * a.acc_bytes / 16;
    for (int i = lane; i < n16; i += 32) reinterpret_cast<uint4*>(base)[i] = make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int u = 0; u < kPasses; ++u) {
    const uint32_t xw[4] = {x[u].x, x[u].y, x[u].z, x[u].w}, yw[4] = {y[u].x, y[u].y, y[u].z, y[u].w};
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 p = unpack2<kBf16>(xw[j]), r = unpack2<kBf16>(yw[j]);
      acc = fmaf(p.x, r.x, acc);
      acc = fmaf(p.y, r.y, acc);
    }
#pragma unroll
    for (int s = kLanes / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    const int q = q0 + u * kPerPass + sub;
    if (l == 0) {
      const int64_t idx = static_cast<int64_t>(bh) * a.sq_r + q;
      const bool in = q < a.sq;
      a.lse2[idx] = in ? a.lse[static_cast<int64_t>(bh) * a.sq + q] * kLog2e : CUDART_INF_F;
      a.dsum[idx] = in ? acc : 0.f;
    }
  }
}

// The CTAs of one launch take three roles by block index: dK / dV rows, dBias, dQ.
template <bool kBf16, bool kDet>
__global__ void __launch_bounds__(kThreads) bwd_finish_kernel(const BwdFinishArgs a) {
  __shared__ int s_slot[kHeads][kRowsGathered];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t blk = blockIdx.x;
  if (blk < static_cast<uint32_t>(a.kv_blocks)) {
    const int kRows = a.pos ? kRowsGathered : kRowsAll;
    // ---- dK, dV: kRows consecutive key positions x up to kHeads kv heads of one batch element ----
    const uint32_t hgroups = (a.h_k + kHeads - 1) / kHeads, chunks = (a.rows_out + kRows - 1) / kRows;
    const int hg = blk % hgroups;
    const uint32_t rest = blk / hgroups;
    const int r0 = static_cast<int>(rest % chunks) * kRows, b = rest / chunks;
    const int h0 = hg * kHeads, nh = min(kHeads, a.h_k - h0);
    for (int h = warp; h < nh; h += kThreads / 32) {
      if (a.pos) {
        // 32-way search for the first slot whose position is >= r0 (positions ascend, unused slots hold INT32_MAX);
        // at most kRows slots from there on fall into this CTA's rows
        const int32_t* prow = a.pos + b * a.pos_sb + (a.h_pos == 1 ? 0 : h0 + h) * a.pos_sh;
        int lo = 0, len = a.cap;  // the answer lies in [lo, lo + len]
        while (len > 0) {
          const int step = (len + 31) / 32;
          const int i = min(lo + (lane + 1) * step - 1, lo + len - 1);
          const uint32_t below = __ballot_sync(0xffffffffu, prow[i] < r0);  // a prefix of the lanes
          const int cnt = __popc(below);
          const int new_lo = min(lo + cnt * step, lo + len);
          len = cnt == 32 ? 0 : min(step - 1, lo + len - new_lo);
          lo = new_lo;
        }
        if (lane < kRows) s_slot[h][lane] = -1;
        __syncwarp();
        const int i = lo + min(lane, kRows - 1);
        const int pos = i < a.cap ? prow[i] : 0x7FFFFFFF;
        if (pos < r0 + kRows && pos < a.rows_out) s_slot[h][pos - r0] = i;
      } else if (lane < kRows) {
        s_slot[h][lane] = r0 + lane;
      }
    }
    __syncthreads();
    const int vecs = a.d / 8;
    const int per_row = nh * vecs;
    const int rows = min(kRows, a.rows_out - r0);
    for (int i = tid; i < rows * per_row; i += kThreads) {
      const int r = i / per_row, hv = i - r * per_row, h = hv / vecs, c = hv - h * vecs;
      const int slot = s_slot[h][r];
      const int64_t src = ((static_cast<int64_t>(b) * a.h_k + h0 + h) * a.keys_r + slot) * a.D + c * 8;
#pragma unroll
      for (int which = 0; which < 2; ++which) {  // 0: dV, 1: dK
        uint4 o = make_uint4(0, 0, 0, 0);
        if (slot >= 0) {
          const float* p = a.part + which * a.nsplit * a.split_stride + src;
          float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
          for (int s = 0; s < a.nsplit; ++s) {
            const float4 x = *reinterpret_cast<const float4*>(p + s * a.split_stride);
            const float4 y = *reinterpret_cast<const float4*>(p + s * a.split_stride + 4);
            acc[0] += x.x; acc[1] += x.y; acc[2] += x.z; acc[3] += x.w;
            acc[4] += y.x; acc[5] += y.y; acc[6] += y.z; acc[7] += y.w;
          }
          o.x = pack_16x2<kBf16>(acc[0], acc[1]);
          o.y = pack_16x2<kBf16>(acc[2], acc[3]);
          o.z = pack_16x2<kBf16>(acc[4], acc[5]);
          o.w = pack_16x2<kBf16>(acc[6], acc[7]);
        }
        uint16_t* dst = which == 0 ? static_cast<uint16_t*>(a.dv) + b * a.dv_sb + static_cast<int64_t>(r0 + r) * a.dv_sr +
                                         (h0 + h) * a.dv_sh
                                   : static_cast<uint16_t*>(a.dk) + b * a.dk_sb + static_cast<int64_t>(r0 + r) * a.dk_sr +
                                         (h0 + h) * a.dk_sh;
        *reinterpret_cast<uint4*>(dst + c * 8) = o;
      }
    }
    return;
  }
  blk -= a.kv_blocks;
  if (blk < static_cast<uint32_t>(a.db_blocks)) {
    // ---- row-broadcast dBias: one warp per 32 consecutive keys of one (batch, head) ----
    const uint32_t chunks = (a.db_keys + 31) / 32;
    const uint32_t w = blk * (kThreads / 32) + warp;
    if (w >= chunks * a.db_b * a.db_h) return;
    const uint32_t bh = w / chunks;
    const int r0 = static_cast<int>(w - bh * chunks) * 32;
    const int h = bh % a.db_h, b = bh / a.db_h;
    int slot = r0 + lane;
    if (slot >= a.rows_out) slot = -1;  // padding keys beyond the last row
    if (a.pos) {
      const int hp = a.h_pos == 1 ? 0 : h / (a.db_h / a.h_pos);
      const int32_t* prow = a.pos + b * a.pos_sb + hp * a.pos_sh;
      // every lane searches its own position
      int lo = 0, hi = a.cap;
      const int want = r0 + lane;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (prow[mid] < want) lo = mid + 1;
        else hi = mid;
      }
      slot = lo < a.cap && want < a.rows_out && prow[lo] == want ? lo : -1;
    }
    float acc = 0.f;
    if (slot >= 0)
      for (int s = 0; s < a.db_nsplit; ++s) acc += a.db_part[s * a.db_split_stride + static_cast<int64_t>(bh) * a.db_pitch + slot];
    if (r0 + lane < a.db_keys)
      static_cast<uint16_t*>(a.dbias)[b * a.db_sb + h * a.db_sh + r0 + lane] =
          static_cast<uint16_t>(pack_16x2<kBf16>(acc, 0.f) & 0xFFFFu);
    return;
  }
  blk -= a.db_blocks;
  // ---- dQ: accumulator (B,H,Sq,D), D = 64 or 128, * scale -> (B,Sq,H,d) 16-bit ----
  const uint32_t dq_blocks = gridDim.x - a.kv_blocks - a.db_blocks;
  const uint32_t vec_log2 = a.D == 128 ? 4 : 3;
  const int64_t n_vec = (static_cast<int64_t>(a.b) * a.h * a.sq) << vec_log2;
  for (int64_t i = blk * static_cast<int64_t>(kThreads) + tid; i < n_vec; i += static_cast<int64_t>(dq_blocks) * kThreads) {
    const uint32_t row = static_cast<uint32_t>(i >> vec_log2);
    const uint32_t bh = row / a.sq, q = row - bh * a.sq;
    const int dd = (static_cast<int>(i) & ((1 << vec_log2) - 1)) * 8;
    if (dd >= a.d) continue;
    const uint32_t b = bh / a.h, h = bh - b * a.h;
    float x[8];
    if (kDet) {
      // 64-bit fixed point. It cannot carry NaN / Inf: a non-finite dO or O element makes D = rowsum(dO o O) of its row
      // non-finite, and with it every dS of the row; such rows come out as NaN, as the fp32 accumulator would give.
      const float unit = a.scale * (1.0f / static_cast<float>(1ll << kDetFracBits));
      const longlong2* p = reinterpret_cast<const longlong2*>(static_cast<const long long*>(a.dq_acc) + i * 8);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const longlong2 v = p[j];
        x[2 * j] = __ll2float_rn(v.x) * unit;
        x[2 * j + 1] = __ll2float_rn(v.y) * unit;
      }
      if (!isfinite(a.dsum[static_cast<int64_t>(bh) * a.sq_r + q])) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __int_as_float(0x7FC00000);
      }
    } else {
      const float* p = static_cast<const float*>(a.dq_acc) + i * 8;
      float4 u = *reinterpret_cast<const float4*>(p), v = *reinterpret_cast<const float4*>(p + 4);
#pragma unroll 4
      for (int s = 1; s < a.dq_nsplit; ++s) {
        const float4 y = *reinterpret_cast<const float4*>(p + s * a.dq_split_stride);
        const float4 z = *reinterpret_cast<const float4*>(p + s * a.dq_split_stride + 4);
        u.x += y.x; u.y += y.y; u.z += y.z; u.w += y.w;
        v.x += z.x; v.y += z.y; v.z += z.z; v.w += z.w;
      }
      x[0] = u.x * a.scale; x[1] = u.y * a.scale; x[2] = u.z * a.scale; x[3] = u.w * a.scale;
      x[4] = v.x * a.scale; x[5] = v.y * a.scale; x[6] = v.z * a.scale; x[7] = v.w * a.scale;
    }
    uint4 o;
    o.x = pack_16x2<kBf16>(x[0], x[1]);
    o.y = pack_16x2<kBf16>(x[2], x[3]);
    o.z = pack_16x2<kBf16>(x[4], x[5]);
    o.w = pack_16x2<kBf16>(x[6], x[7]);
    *reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.dq) + b * a.dq_sb + static_cast<int64_t>(q) * a.dq_sr +
                              h * a.dq_sh + dd) = o;
  }
}

template <bool kBf16>
void launch_prep(const BwdPrepArgs& a, int D, unsigned blocks, cudaStream_t stream) {
  if (D == 64) bwd_prep_kernel<64, kBf16><<<blocks, kThreads, 0, stream>>>(a);
  else if (D == 128) bwd_prep_kernel<128, kBf16><<<blocks, kThreads, 0, stream>>>(a);
  else bwd_prep_kernel<256, kBf16><<<blocks, kThreads, 0, stream>>>(a);
}

}  // namespace

int launch_bwd_prep(const BwdPrepArgs& a, int D, bool bf16, cudaStream_t stream) {
  const int64_t warps = static_cast<int64_t>(a.b) * a.h * (a.sq_r / 8);
  if (warps > 0x7FFFFFFF / 32) return FDMA_ERR_TOO_LARGE;
  const unsigned blocks = static_cast<unsigned>((warps * 32 + kThreads - 1) / kThreads);
  if (bf16) launch_prep<true>(a, D, blocks, stream);
  else launch_prep<false>(a, D, blocks, stream);
  return static_cast<int>(cudaGetLastError());
}

int launch_bwd_finish(BwdFinishArgs a, bool bf16, bool deterministic, cudaStream_t stream) {
  int64_t kv = 0, db = 0;
  const int kRows = a.pos ? kRowsGathered : kRowsAll;
  if (a.part)
    kv = static_cast<int64_t>(a.b) * ((a.rows_out + kRows - 1) / kRows) * ((a.h_k + kHeads - 1) / kHeads);
  if (a.db_part) {
    const int64_t warps = static_cast<int64_t>(a.db_b) * a.db_h * ((a.db_keys + 31) / 32);
    db = (warps + kThreads / 32 - 1) / (kThreads / 32);
  }
  // dQ rows: a grid-stride loop of at least four 32-byte pieces per thread on large tensors
  const int64_t n_vec = static_cast<int64_t>(a.b) * a.h * a.sq * (a.D / 8);
  const int64_t dq = a.dq_acc ? std::max<int64_t>(1, std::min<int64_t>((n_vec + kThreads - 1) / kThreads, sm_count() * 32)) : 0;
  if (kv + db + dq == 0) return 0;
  if (kv + db + dq > 0x7FFFFFFF) return FDMA_ERR_TOO_LARGE;
  a.kv_blocks = static_cast<int>(kv);
  a.db_blocks = static_cast<int>(db);
  const unsigned blocks = static_cast<unsigned>(kv + db + dq);
  if (bf16) {
    if (deterministic) bwd_finish_kernel<true, true><<<blocks, kThreads, 0, stream>>>(a);
    else bwd_finish_kernel<true, false><<<blocks, kThreads, 0, stream>>>(a);
  } else {
    if (deterministic) bwd_finish_kernel<false, true><<<blocks, kThreads, 0, stream>>>(a);
    else bwd_finish_kernel<false, false><<<blocks, kThreads, 0, stream>>>(a);
  }
  return static_cast<int>(cudaGetLastError());
}

}  // namespace fdma
