// Internal declarations shared by the translation units of libfdma_sm100.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/fdma.h"

namespace fdma {

constexpr int kKeyPad = 128;  // mask/bias rows are readable up to round_up(Sk, kKeyPad) keys

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
inline size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

// ---- CUDA-core ("SIMT") kernels: any head dim <= 256 that is a multiple of 8 -------------------
size_t simt_bwd_workspace_bytes(const fdma_bwd_params& p);
int simt_fwd(const fdma_fwd_params& p, cudaStream_t stream);
int simt_bwd(const fdma_bwd_params& p, cudaStream_t stream);

// ---- tcgen05 / TMA kernels ---------------------------------------------------------------------
// Packed sequences: cumulative lengths on the device, n + 1 entries each, ascending; null: an ordinary call.
struct PackedSeqs {
  const int32_t *cu_q = nullptr, *cu_k = nullptr;
  int n = 0;
};
bool tc_fwd_supported(const fdma_fwd_params& p);
size_t tc_fwd_workspace_bytes(const fdma_fwd_params& p);
// seqs: packed sequences, see fdma_fwd_varlen
int tc_fwd(const fdma_fwd_params& p, cudaStream_t stream, const PackedSeqs& seqs = {});

// Per-tile mask activity map for per-query masks: act[b][h_mask][ceil(Sq/128)][ceil(Sk/128)] bytes.
int launch_tile_activity(const fdma_fwd_params& p, uint8_t* act, cudaStream_t stream);

// head dim 256, row-broadcast mask / bias (fdma_bwd256_sm100.cu); reached through the three tc_bwd entry points
bool tc_bwd256_supported(const fdma_bwd_params& p);
size_t tc_bwd256_workspace_bytes(const fdma_bwd_params& p);
int tc_bwd256(const fdma_bwd_params& p, cudaStream_t stream);

// head dims up to 128, row-broadcast mask / bias, packed sequences (fdma_bwd_rows_sm100.cu); also reached through tc_bwd
bool bwd_rows_taken(const fdma_bwd_params& p);
bool bwd_rows_taken_packed(const fdma_bwd_params& p);  // the same call, about packed sequences
size_t bwd_rows_workspace_bytes(const fdma_bwd_params& p);
int bwd_rows(const fdma_bwd_params& p, cudaStream_t stream, const PackedSeqs& seqs);

bool tc_bwd_supported(const fdma_bwd_params& p);
size_t tc_bwd_workspace_bytes(const fdma_bwd_params& p);
int tc_bwd(const fdma_bwd_params& p, cudaStream_t stream, const PackedSeqs& seqs = {});  // seqs: head dims up to 128

// ---- the kernels before and after every tensor-core backward (fdma_bwd_common.cu) ---------------
constexpr int kDetFracBits = 40;  // deterministic dQ accumulator: fixed point, |dQ / scale| < 2^23, resolution 2^-40

// Head dim the tensor-core kernels run a call at: tiles are 64, 128 or 256 wide; the columns beyond d are zeros that
// the TMA loads fill in, so no tensor is ever padded in memory.
inline int tile_head_dim(int d) { return d <= 64 ? 64 : d <= 128 ? 128 : 256; }

struct BwdPrepArgs {
  const void *out, *dout;
  const float* lse;
  float *lse2, *dsum;  // (B,H,sq_r)
  void* dq_acc;        // null, or (D <= 128) zeroed: (B,H,Sq,D) elements of acc_bytes
  int b, h, sq, sq_r, d, acc_bytes;
  int64_t o_sb, o_sr, o_sh, do_sb, do_sr, do_sh;
};
int launch_bwd_prep(const BwdPrepArgs& a, int D, bool bf16, cudaStream_t stream);

struct BwdFinishArgs {
  // dQ, or dq_acc = null (already written by the main kernel); fp32: the sum of dq_nsplit partials (0: of one)
  const void* dq_acc;
  int dq_nsplit;
  int64_t dq_split_stride;
  void* dq;
  const float* dsum;  // deterministic mode: rows with a non-finite D become NaN
  int64_t dq_sb, dq_sr, dq_sh;
  float scale;
  int b, h, sq, sq_r, d, D;
  // dK, dV: fp32 partials [2: dV, dK][nsplit][B][h_k][keys_r][D], or part = null (already written by the main kernel)
  const float* part;
  int64_t split_stride;
  int nsplit, h_k, keys_r;
  void *dk, *dv;
  int64_t dk_sb, dk_sr, dk_sh, dv_sb, dv_sr, dv_sh;
  int rows_out;  // key rows of dk / dv
  // gathered keys: ascending positions ({B|1}, {h_k|1}, cap) of the partials' rows; null: row = key
  const int32_t* pos;
  int64_t pos_sb, pos_sh;
  int h_pos, cap;
  // row-broadcast dBias: fp32 sums [db_nsplit][db_b * db_h][db_pitch], or db_part = null
  const float* db_part;
  int64_t db_split_stride;
  int db_nsplit, db_pitch, db_b, db_h, db_keys;
  void* dbias;
  int64_t db_sb, db_sh;
  int kv_blocks, db_blocks;  // set by the launcher
};
int launch_bwd_finish(BwdFinishArgs a, bool bf16, bool deterministic, cudaStream_t stream);

// ---- single-query (decode) forward: row-granular skipping, split over keys + merge -------------
bool decode_supported(const fdma_fwd_params& p);
size_t decode_workspace_bytes(const fdma_fwd_params& p);
int decode_fwd(const fdma_fwd_params& p, cudaStream_t stream);
int decode_fwd_sliced(const fdma_fwd_params& p, cudaStream_t stream);
// fdma_fwd for a single query with a bool mask in whatever workspace there is: position lists a few rows at a time, or where
// not even one list fits, the kernels that need none. FDMA_ERR_TOO_LARGE for other calls.
int single_query_fwd_in(const fdma_fwd_params& p, cudaStream_t stream);

// ---- create_mask -------------------------------------------------------------------------------
int create_mask(const fdma_mask_params& p, cudaStream_t stream);

// ---- helpers -----------------------------------------------------------------------------------
// Device address of the current device's kernel status word (written by bounded waits that give up).
int* kernel_status_ptr();

// Copies D = rowsum(dO o O) from a kernel's scratch layout (B*H rows of `sq_r` floats, zeros beyond Sq) into the
// caller's optional fdma_bwd_params::softmax_d (B, H, round_up(Sq,128)); no-op when that pointer is null.
int export_softmax_d(const fdma_bwd_params& bp, const float* dsum, int sq_r, cudaStream_t stream);

// Number of SMs of the current device (cudaDevAttrMultiProcessorCount, cached per device).
int sm_count();

// Events registered by fdma_time_next_kernel for this host thread (both null when none); take_* clears them.
void take_timing_events(cudaEvent_t* start, cudaEvent_t* stop);

// Encodes a 4-D tiled tensor map (dims innermost first) with 128-byte swizzle; returns 0 or a status.
int encode_tmap_4d(void* out_map, const void* base, int elem_bytes, const uint64_t dims[4],
                   const uint64_t strides_bytes[3], const uint32_t box[4]);

}  // namespace fdma
