// Native host path of the operator layer: what flash_sparse_attn_func and create_mask do between the Python call and the
// kernel launches -- checks, route choice, allocation, the autograd node -- in C++ on top of the C ABI of
// libfdma_sm100.so (include/fdma.h), which is opened at run time.
//
// Why: a training call at S = 256 spends 0.05 ms on the GPU and spent 0.6 ms in Python (custom-op dispatch, ctypes
// structures field by field, one allocation call per tensor). Every function here returns an empty result for inputs it
// does not handle (wrong types, odd layouts, tracing); the Python layer then runs its own path, which also raises the
// argument errors.
#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/dynamo/compiled_autograd.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <array>
#include <mutex>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/fdma.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

struct Api {
  decltype(&fdma_fwd_workspace_bytes) fwd_workspace_bytes;
  decltype(&fdma_fwd) fwd;
  decltype(&fdma_bwd_workspace_bytes) bwd_workspace_bytes;
  decltype(&fdma_bwd) bwd;
  decltype(&fdma_fwd_varlen) fwd_varlen;
  decltype(&fdma_bwd_varlen) bwd_varlen;
  decltype(&fdma_create_mask) create_mask;
  decltype(&fdma_gather_kept) gather_kept;
  decltype(&fdma_decode_kept) decode_kept;
  decltype(&fdma_decode_kept_workspace_bytes) decode_kept_workspace_bytes;
  decltype(&fdma_strerror) strerror;
  decltype(&fdma_poll_kernel_status) poll_kernel_status;
  decltype(&fdma_last_kernel_status) last_kernel_status;
} api;

void init(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("cannot open ") + path + ": " + dlerror());
  auto get = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(dlsym(h, name));
    if (!fn) throw std::runtime_error(path + " does not export " + name);
  };
  get(api.fwd_workspace_bytes, "fdma_fwd_workspace_bytes");
  get(api.fwd, "fdma_fwd");
  get(api.bwd_workspace_bytes, "fdma_bwd_workspace_bytes");
  get(api.bwd, "fdma_bwd");
  get(api.fwd_varlen, "fdma_fwd_varlen");
  get(api.bwd_varlen, "fdma_bwd_varlen");
  get(api.create_mask, "fdma_create_mask");
  get(api.gather_kept, "fdma_gather_kept");
  get(api.decode_kept, "fdma_decode_kept");
  get(api.decode_kept_workspace_bytes, "fdma_decode_kept_workspace_bytes");
  get(api.strerror, "fdma_strerror");
  get(api.poll_kernel_status, "fdma_poll_kernel_status");
  get(api.last_kernel_status, "fdma_last_kernel_status");
}

constexpr int64_t kTile = 128;
// What the tile tables of the tensor-core kernels hold. The gradients of gathered keys and bit masks have no other kernels.
constexpr int64_t kMaxKeys = 1 << 20, kMaxQueries = 1 << 19;
int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

void check(int status, const char* what) {
  if (status != 0)
    throw std::runtime_error(std::string(what) + " failed: " + api.strerror(status) + " (status " + std::to_string(status) + ")");
}

cudaStream_t stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// A kernel whose bounded wait gave up surfaces at the next operator call (one host load, no GPU work).
void raise_if_timed_out(cudaStream_t stream) {
  if (api.poll_kernel_status(nullptr) == 0) return;
  int32_t detail = 0;
  api.last_kernel_status(stream, &detail);
  throw std::runtime_error("an earlier attention kernel on this device gave up a bounded wait (code " + std::to_string(detail) +
                           "): " + api.strerror(FDMA_ERR_TIMEOUT) + "; results of calls since then are not valid");
}

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
Tensor empty_as(const Tensor& t) {
  return t.is_contiguous() ? empty(t.sizes(), t.scalar_type(), t) : at::empty_like(t);
}
Tensor inner_contiguous(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
// A (.., rows, heads, d) tensor as the tensor-core kernels load it: 16-byte aligned base and strides, nothing expanded. Calls
// that only those kernels serve (gathered keys, bit masks, packed sequences) get a dense copy of anything else: an output
// gradient that `sum` expanded or that was cut out of wider rows, a query slice with an odd stride.
Tensor kernel_layout(const Tensor& t) {
  bool ok = t.stride(-1) == 1 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  for (int64_t i = 0; i + 1 < t.dim(); ++i) ok = ok && t.stride(i) > 0 && t.stride(i) % 8 == 0;
  return ok ? t : t.clone(at::MemoryFormat::Contiguous);
}
const Tensor& get(const OptTensor& t) {
  static const Tensor none;
  return t.has_value() ? *t : none;
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return FDMA_BF16;
    case at::kHalf: return FDMA_FP16;
    case at::kFloat: return FDMA_FP32;
    default: return -1;
  }
}

struct Bsh {
  int64_t b, r, h;
};
// (batch, row, head) element strides of a (B, S, H, d) tensor; dimensions of extent 1 get a dense stride
Bsh bsh(const Tensor& t) {
  Bsh s{t.stride(0), t.stride(1), t.stride(2)};
  if (t.size(2) == 1) s.h = t.size(3);
  if (t.size(1) == 1 && s.h == t.size(3)) s.r = t.size(2) * t.size(3);
  if (t.size(0) == 1) s.b = std::max<int64_t>(s.b, 1);
  return s;
}
int64_t bcast_stride(const Tensor& t, int dim) { return t.size(dim) == 1 ? 0 : t.stride(dim); }

// Everything one attention call needs besides q, k, v: the same struct serves the forward call and the autograd node.
struct Call {
  float scale = 0.f;
  bool causal = false, deterministic = false, bits = false, gathered = false, packed = false;
  int path = FDMA_PATH_AUTO;
  int64_t seqlen_k = 0;      // keys of the caller's K
  int64_t bias_keys = 0;     // key extent of the caller's bias
  std::vector<int64_t> bias_c;  // gathered: shape of the gathered bias (empty: no bias)
};

// Gathered K, V and bias live in one buffer: [K_c | V_c | bias_c], each 256-byte aligned.
struct KvB {
  void *k, *v, *bias;
};
KvB split_kvb(const Tensor& buf, int64_t kv_elems, bool has_bias) {
  char* p = static_cast<char*>(buf.data_ptr());
  const int64_t step = round_up(kv_elems * 2, 256);
  return {p, p + step, has_bias ? p + 2 * step : nullptr};
}

void fill_geometry(fdma_fwd_params& p, const Tensor& q, int64_t seqlen_k, int64_t h_k, const Call& c) {
  p.q = q.data_ptr();
  const Bsh sq = bsh(q);
  p.q_batch_stride = sq.b; p.q_row_stride = sq.r; p.q_head_stride = sq.h;
  p.b = static_cast<int32_t>(q.size(0));
  p.seqlen_q = static_cast<int32_t>(q.size(1));
  p.seqlen_k = static_cast<int32_t>(seqlen_k);
  p.h = static_cast<int32_t>(q.size(2));
  p.h_k = static_cast<int32_t>(h_k);
  p.h_mask = p.h_bias = 1;
  p.d = static_cast<int32_t>(q.size(3));
  p.dtype = dtype_code(q);
  p.is_causal = c.causal ? 1 : 0;
  p.softmax_scale = c.scale;
  p.path = c.path;
}
void fill_kv(fdma_fwd_params& p, const Tensor& k, const Tensor& v) {
  const Bsh sk = bsh(k), sv = bsh(v);
  p.k = k.data_ptr(); p.v = v.data_ptr();
  p.k_batch_stride = sk.b; p.k_row_stride = sk.r; p.k_head_stride = sk.h;
  p.v_batch_stride = sv.b; p.v_row_stride = sv.r; p.v_head_stride = sv.h;
}
void fill_out(fdma_fwd_params& p, const Tensor& out, const Tensor& lse) {
  const Bsh so = bsh(out);
  p.out = out.data_ptr(); p.lse = lse.data_ptr<float>();
  p.o_batch_stride = so.b; p.o_row_stride = so.r; p.o_head_stride = so.h;
}
void fill_mask_bias(fdma_fwd_params& p, const Tensor& mask, const Tensor& bias, const Tensor& activity, const Call& c) {
  if (mask.defined()) {
    p.mask = mask.data_ptr();
    p.h_mask = static_cast<int32_t>(mask.size(1));
    if (c.bits) {
      p.mask_bits = 1;
      p.mask_batch_stride = mask.stride(0);
      p.mask_head_stride = bcast_stride(mask, 1);
      p.mask_row_stride = mask.stride(2);
      p.tile_activity = static_cast<const uint8_t*>(activity.data_ptr());
    } else {
      p.mask_batch_stride = bcast_stride(mask, 0);
      p.mask_head_stride = bcast_stride(mask, 1);
      p.mask_row_stride = bcast_stride(mask, 2);
    }
  }
  if (bias.defined()) {
    p.bias = bias.data_ptr();
    p.h_bias = static_cast<int32_t>(bias.size(1));
    p.bias_batch_stride = bcast_stride(bias, 0);
    p.bias_head_stride = bcast_stride(bias, 1);
    p.bias_row_stride = bcast_stride(bias, 2);
  }
}
// gathered keys: dense (B, cap, Hk, d) rows and their positions
void fill_gathered(fdma_fwd_params& p, const KvB& kv, const Tensor& key_pos, const Tensor& slot_mask, const Call& c) {
  const int64_t cap = key_pos.size(2), hk = p.h_k, d = p.d;
  p.k = kv.k; p.v = kv.v;
  p.k_batch_stride = p.v_batch_stride = cap * hk * d;
  p.k_row_stride = p.v_row_stride = hk * d;
  p.k_head_stride = p.v_head_stride = d;
  p.mask = slot_mask.data_ptr();
  p.h_mask = static_cast<int32_t>(slot_mask.size(1));
  p.mask_batch_stride = bcast_stride(slot_mask, 0);
  p.mask_head_stride = bcast_stride(slot_mask, 1);
  p.mask_row_stride = 0;
  if (!c.bias_c.empty()) {
    p.bias = kv.bias;
    p.h_bias = static_cast<int32_t>(c.bias_c[1]);
    p.bias_batch_stride = c.bias_c[0] == 1 ? 0 : c.bias_c[1] * cap;
    p.bias_head_stride = c.bias_c[1] == 1 ? 0 : cap;
    p.bias_row_stride = 0;
  }
  p.key_pos = key_pos.data_ptr<int32_t>();
  p.key_pos_batch_stride = bcast_stride(key_pos, 0);
  p.key_pos_head_stride = key_pos.stride(1);
  p.h_pos = static_cast<int32_t>(key_pos.size(1));
  p.causal_shift = static_cast<int32_t>(c.seqlen_k - p.seqlen_q);
}

// ---- backward --------------------------------------------------------------------------------------------------
// One node for the four routes. Saved: dense   q, k, v, mask, bias, out, lse
//                                       bits    q, k, v, bits, bias, out, lse, activity
//                                       gathered q, kvb, -, slot_mask, -, out, lse, key_pos
//                                       packed  q, k, v, -, -, out, lse, cu (2, n + 1): the sequences' boundaries
enum { kQ, kK, kV, kMask, kBias, kOut, kLse, kExtra, kNumSaved };
using SavedTensors = std::array<Tensor, kNumSaved>;

// What the node knows besides tensors, and the same as plain values for compiled autograd.
struct Meta {
  Call c;
  std::vector<int64_t> k_sizes, bias_sizes;  // of the caller's tensors
  bool want_bias = false;

  std::vector<int64_t> pack() const {
    std::vector<int64_t> x = {c.causal, c.deterministic, c.bits, c.gathered, c.packed, c.path, c.seqlen_k, c.bias_keys, want_bias};
    for (const auto* v : {&c.bias_c, &k_sizes, &bias_sizes}) {
      x.push_back(static_cast<int64_t>(v->size()));
      x.insert(x.end(), v->begin(), v->end());
    }
    return x;
  }
  static Meta unpack(const std::vector<int64_t>& x, double scale) {
    Meta m;
    size_t i = 0;
    auto next = [&] { return x.at(i++); };
    m.c.scale = static_cast<float>(scale);
    m.c.causal = next(); m.c.deterministic = next(); m.c.bits = next(); m.c.gathered = next(); m.c.packed = next();
    m.c.path = static_cast<int>(next());
    m.c.seqlen_k = next(); m.c.bias_keys = next(); m.want_bias = next();
    for (auto* v : {&m.c.bias_c, &m.k_sizes, &m.bias_sizes}) {
      v->resize(next());
      for (int64_t& e : *v) e = next();
    }
    return m;
  }
};

variable_list backward(const Tensor& grad, const SavedTensors& t, const Meta& meta);

struct AttnBackward : public torch::autograd::Node {
  Meta meta;
  std::array<SavedVariable, kNumSaved> saved;

  std::string name() const override { return "FlashSparseAttnBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);  // another thread may run this node
    for (SavedVariable& s : saved) s.reset_data();
  }
  SavedTensors unpack() {
    SavedTensors t;
    for (int i = 0; i < kNumSaved; ++i) t[i] = saved[i].unpack(i == kOut ? getptr() : nullptr);
    return t;
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    // Unpacked before anything is switched off: a hook may recompute the region the call belongs to (checkpointing),
    // which has to record a graph of its own while it does.
    variable_list res = backward(grads[0], unpack(), meta);
    if (!at::GradMode::is_enabled()) return res;
    // create_graph: the gradients come from kernels without a derivative. They carry a node that says so when it is
    // reached; without one a gradient penalty would silently leave the attention out.
    for (Tensor& t : res)
      if (t.defined()) t.set_requires_grad(true);
    auto error = std::make_shared<torch::autograd::DelayedError>(
        "trying to differentiate twice through flash_sparse_attn, whose backward has no derivative", static_cast<int64_t>(res.size()));
    return error->apply(std::move(res));
  }

  // Compiled autograd: the node is one opaque call in the graph it captures.
  void compiled_args(torch::dynamo::autograd::CompiledNodeArgs& args) const override {
    for (int i = 0; i < kNumSaved; ++i) args.collect(saved[i], /*is_output=*/i == kOut);
    args.collect(static_cast<double>(meta.c.scale));
    args.collect(meta.pack());
  }
  variable_list apply_with_saved(const variable_list& grads, torch::dynamo::autograd::SwapSavedVariables& swap) override {
    namespace ca = torch::dynamo::autograd;
    for (SavedVariable& s : saved) swap.before(s);
    ca::PackedArgs packed;
    for (const Tensor& t : unpack()) packed.pack(t);
    packed.pack(static_cast<double>(meta.c.scale));
    packed.pack(meta.pack());
    const std::vector<at::IValue> args = packed.vec();
    std::vector<at::TypePtr> schema;
    for (const at::IValue& x : args) schema.push_back(x.isTensor() ? at::TypePtr(at::TensorType::get()) : x.type());
    const auto outputs = ca::IValuePacker<std::vector<std::optional<torch::autograd::InputMetadata>>>::pack(ca::get_input_metadata(next_edges()));
    const auto& compiler = ca::getPyCompilerInterface();
    const std::string fn = compiler->bind_function(swap.get_py_compiler(), name(), &functional, schema, /*is_custom_function=*/true,
                                                   /*is_traceable=*/false);
    variable_list res = compiler->call_function(swap.get_py_compiler(), "apply_functional", fn, grads, args, outputs);
    for (SavedVariable& s : saved) swap.after(s);
    return res;
  }
  static variable_list functional(const variable_list& grads, const std::vector<at::IValue>& args) {
    torch::dynamo::autograd::PackedArgs packed(args);
    SavedTensors t;
    for (Tensor& x : t) x = packed.unpack<Tensor>();
    const double scale = packed.unpack<double>();
    return backward(grads[0], t, Meta::unpack(packed.unpack<std::vector<int64_t>>(), scale));
  }
};

// Gradients of packed sequences: (tokens, heads, d) tensors, one row of tokens for the kernels.
variable_list packed_backward(const SavedTensors& t, const Call& c, const Tensor& dout, cudaStream_t stream) {
  const Tensor &tq = t[kQ], &tk = t[kK], &tv = t[kV], &tout = t[kOut], &tlse = t[kLse], &cu = t[kExtra];
  variable_list res(3);
  Tensor dq = empty(tq.sizes(), tq.scalar_type(), tq), dk = empty(tk.sizes(), tk.scalar_type(), tk), dv = empty(tv.sizes(), tv.scalar_type(), tv);
  fdma_bwd_params bp = {};
  const Tensor q4 = tq.unsqueeze(0), k4 = tk.unsqueeze(0);
  fill_geometry(bp.f, q4, tk.size(0), tk.size(1), c);
  fill_kv(bp.f, k4, tv.unsqueeze(0));
  fill_out(bp.f, tout.unsqueeze(0), tlse);
  const Bsh so = bsh(dout.unsqueeze(0)), sq = bsh(dq.unsqueeze(0)), sk = bsh(dk.unsqueeze(0));
  bp.dout = dout.data_ptr();
  bp.do_batch_stride = so.b; bp.do_row_stride = so.r; bp.do_head_stride = so.h;
  bp.dq = dq.data_ptr(); bp.dk = dk.data_ptr(); bp.dv = dv.data_ptr();
  bp.dq_batch_stride = sq.b; bp.dq_row_stride = sq.r; bp.dq_head_stride = sq.h;
  bp.dk_batch_stride = bp.dv_batch_stride = sk.b;
  bp.dk_row_stride = bp.dv_row_stride = sk.r;
  bp.dk_head_stride = bp.dv_head_stride = sk.h;
  bp.deterministic = c.deterministic ? 1 : 0;
  const size_t bytes = api.bwd_workspace_bytes(&bp);
  Tensor ws;
  if (bytes) {
    ws = empty({static_cast<int64_t>(bytes)}, at::kByte, tq);
    bp.f.workspace = ws.data_ptr();
    bp.f.workspace_bytes = bytes;
  }
  const int32_t* cu_q = cu.data_ptr<int32_t>();
  check(api.bwd_varlen(&bp, cu_q, cu_q + cu.stride(0), static_cast<int32_t>(cu.size(1) - 1), stream), "fdma_bwd_varlen");
  res[0] = dq; res[1] = dk; res[2] = dv;
  return res;
}

variable_list backward(const Tensor& grad, const SavedTensors& t, const Meta& meta) {
  const Call& c = meta.c;
  variable_list res(c.packed ? 3 : 4);
  if (!grad.defined()) return res;
  const Tensor &tq = t[kQ], &tk = t[kK], &tv = t[kV], &tmask = t[kMask], &tbias = t[kBias], &tlse = t[kLse], &textra = t[kExtra], &tout = t[kOut];
  at::AutoDispatchBelowADInplaceOrView guard;
  const c10::cuda::CUDAGuard device(tq.device());
  const cudaStream_t stream = stream_of(tq);
  raise_if_timed_out(stream);
  if (c.packed) return packed_backward(t, c, kernel_layout(grad), stream);
  const Tensor dout = c.gathered || c.bits ? kernel_layout(grad) : inner_contiguous(grad);

  fdma_bwd_params bp = {};
  Tensor dq = empty_as(tq), dk, dv, dbias;
  if (c.gathered) {
    dk = empty(meta.k_sizes, tq.scalar_type(), tq);
    dv = empty(meta.k_sizes, tq.scalar_type(), tq);
    const int64_t cap = textra.size(2), hk = meta.k_sizes[2], d = tq.size(3);
    fill_geometry(bp.f, tq, cap, hk, c);
    fill_gathered(bp.f, split_kvb(tk, tq.size(0) * cap * hk * d, !c.bias_c.empty()), textra, tmask, c);
    bp.scatter_pos = textra.data_ptr<int32_t>();
    bp.scatter_batch_stride = bp.f.key_pos_batch_stride;
    bp.scatter_head_stride = bp.f.key_pos_head_stride;
    bp.scatter_h = bp.f.h_pos;
    bp.scatter_rows = static_cast<int32_t>(c.seqlen_k);
    if (meta.want_bias) dbias = empty(meta.bias_sizes, tq.scalar_type(), tq);
  } else {
    dk = empty_as(tk);
    dv = empty_as(tv);
    fill_geometry(bp.f, tq, tk.size(1), tk.size(2), c);
    fill_kv(bp.f, tk, tv);
    fill_mask_bias(bp.f, tmask, tbias, textra, c);
    if (meta.want_bias) dbias = empty(tbias.sizes(), tbias.scalar_type(), tbias);
  }
  fill_out(bp.f, tout, tlse);
  const Bsh so = bsh(dout), sq = bsh(dq), sk = bsh(dk), sv = bsh(dv);
  bp.dout = dout.data_ptr();
  bp.do_batch_stride = so.b; bp.do_row_stride = so.r; bp.do_head_stride = so.h;
  bp.dq = dq.data_ptr(); bp.dk = dk.data_ptr(); bp.dv = dv.data_ptr();
  bp.dq_batch_stride = sq.b; bp.dq_row_stride = sq.r; bp.dq_head_stride = sq.h;
  bp.dk_batch_stride = sk.b; bp.dk_row_stride = sk.r; bp.dk_head_stride = sk.h;
  bp.dv_batch_stride = sv.b; bp.dv_row_stride = sv.r; bp.dv_head_stride = sv.h;
  if (dbias.defined()) {
    bp.dbias = dbias.data_ptr();
    bp.dbias_batch_stride = dbias.stride(0); bp.dbias_head_stride = dbias.stride(1); bp.dbias_row_stride = dbias.stride(2);
    bp.dbias_b = static_cast<int32_t>(dbias.size(0));
    bp.dbias_h = static_cast<int32_t>(dbias.size(1));
    bp.dbias_rows = static_cast<int32_t>(dbias.size(2));
    bp.dbias_keys = static_cast<int32_t>(dbias.size(3));
  }
  bp.deterministic = c.deterministic ? 1 : 0;
  const size_t bytes = api.bwd_workspace_bytes(&bp);
  Tensor ws;
  if (bytes) {
    ws = empty({static_cast<int64_t>(bytes)}, at::kByte, tq);
    bp.f.workspace = ws.data_ptr();
    bp.f.workspace_bytes = bytes;
  }
  check(api.bwd(&bp, stream), "fdma_bwd");
  if (dbias.defined() && !c.gathered && c.bias_keys != dbias.size(3)) {
    dbias = dbias.narrow(3, 0, c.seqlen_k);
    if (c.bias_keys == 1) dbias = dbias.sum({3}, /*keepdim=*/true);
  }
  res[0] = dq; res[1] = dk; res[2] = dv; res[3] = dbias;
  return res;
}

// ---- forward ---------------------------------------------------------------------------------------------------
bool plain(const Tensor& t) { return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.dim() == 4; }

bool needs_grad(const Tensor& t) { return t.defined() && t.requires_grad(); }

Tensor fit_keys(const Tensor& t, int64_t keys_r) {
  if (t.size(3) == keys_r) return t;
  if (t.size(3) == 1) return t.expand({t.size(0), t.size(1), t.size(2), keys_r});
  return at::constant_pad_nd(t, {0, keys_r - t.size(3)}, 0);
}

// mask / bias extents the kernels take; anything else goes to the Python path, which raises the right error
bool broadcastable(const Tensor& t, int64_t B, int64_t H, int64_t Hk, int64_t Sq) {
  return (t.size(0) == 1 || t.size(0) == B) && (t.size(1) == 1 || t.size(1) == Hk || t.size(1) == H) &&
         (t.size(2) == 1 || t.size(2) == Sq);
}

// A single query over the kept keys of the list; nullopt for layouts the decode kernel does not take.
std::optional<Tensor> decode(const Tensor& q0, const Tensor& k, const Tensor& v, const Tensor& bias0, const Tensor& key_pos, const Call& c) {
  const int64_t B = q0.size(0), H = q0.size(2), Hk = k.size(2), Sk = k.size(1);
  if (k.stride(3) != 1 || v.stride(3) != 1 || q0.stride(3) != 1 || !key_pos.is_contiguous()) return std::nullopt;
  if ((key_pos.size(0) != 1 && key_pos.size(0) != B) || (key_pos.size(1) != 1 && key_pos.size(1) != Hk && key_pos.size(1) != H))
    return std::nullopt;
  if (bias0.defined() && (bias0.size(2) != 1 || bias0.size(3) < Sk || bias0.stride(3) != 1)) return std::nullopt;
  at::AutoDispatchBelowADInplaceOrView guard;
  const c10::cuda::CUDAGuard device(q0.device());
  const cudaStream_t stream = stream_of(q0);
  raise_if_timed_out(stream);
  Tensor out = empty_as(q0), lse = empty({B, H, 1}, at::kFloat, q0);
  fdma_decode_params p = {};
  fill_geometry(p.f, q0, Sk, Hk, c);
  fill_kv(p.f, k, v);
  fill_mask_bias(p.f, Tensor(), bias0, Tensor(), c);
  fill_out(p.f, out, lse);
  p.kept_pos = key_pos.data_ptr<int32_t>();
  p.kept_batch_stride = bcast_stride(key_pos, 0);
  p.kept_head_stride = bcast_stride(key_pos, 1);
  p.kept_h = static_cast<int32_t>(key_pos.size(1));
  p.kept_capacity = static_cast<int32_t>(key_pos.size(2));
  const size_t bytes = api.decode_kept_workspace_bytes(&p);
  Tensor ws;
  if (bytes) {
    ws = empty({static_cast<int64_t>(bytes)}, at::kByte, q0);
    p.f.workspace = ws.data_ptr();
    p.f.workspace_bytes = bytes;
  }
  const int st = api.decode_kept(&p, stream);
  if (st == FDMA_ERR_UNSUPPORTED) return std::nullopt;
  check(st, "fdma_decode_kept");
  return out;
}

// Runs one attention call; nullopt for inputs this path does not take. Exactly one form of mask is given: a bool tensor,
// the position list of the kept keys (key_pos, slot_mask), bits with their tile activity, or none.
std::optional<Tensor> attention(const Tensor& q0, const Tensor& k0, const Tensor& v0, const OptTensor& mask_, const OptTensor& bias_,
                                const OptTensor& key_pos_, const OptTensor& slot_mask_, const OptTensor& bits_,
                                const OptTensor& activity_, double scale, bool causal, bool deterministic, int path) {
  const Tensor &mask0 = get(mask_), &bias0 = get(bias_), &key_pos = get(key_pos_), &slot_mask = get(slot_mask_),
               &bits = get(bits_), &activity = get(activity_);
  if (!plain(q0) || !plain(k0) || !plain(v0)) return std::nullopt;
  const auto type = q0.scalar_type();
  if ((type != at::kBFloat16 && type != at::kHalf) || k0.scalar_type() != type || v0.scalar_type() != type) return std::nullopt;
  const int64_t B = q0.size(0), Sq = q0.size(1), H = q0.size(2), d = q0.size(3), Sk = k0.size(1), Hk = k0.size(2);
  if (B <= 0 || Sq <= 0 || Sk <= 0 || H <= 0 || Hk <= 0 || H % Hk || d % 8 || d <= 0 || d > 256) return std::nullopt;
  if (k0.size(0) != B || k0.size(3) != d || v0.sizes() != k0.sizes()) return std::nullopt;
  if (k0.device() != q0.device() || v0.device() != q0.device()) return std::nullopt;
  if (bias0.defined() && (!plain(bias0) || bias0.scalar_type() != type || bias0.device() != q0.device() ||
                          !broadcastable(bias0, B, H, Hk, Sq)))
    return std::nullopt;
  const int64_t Sk_r = round_up(Sk, kTile);
  const bool grad = at::GradMode::is_enabled() && (needs_grad(q0) || needs_grad(k0) || needs_grad(v0) || needs_grad(bias0));

  Call c;
  c.scale = static_cast<float>(scale);
  c.causal = causal;
  c.deterministic = deterministic;
  c.path = path;
  c.seqlen_k = Sk;
  c.bias_keys = bias0.defined() ? bias0.size(3) : 0;
  if (key_pos.defined() && Sq == 1) {
    if (grad) return std::nullopt;
    return decode(q0, k0, v0, bias0, key_pos, c);
  }
  if (key_pos.defined()) {
    c.gathered = true;
    const int64_t Bm = key_pos.size(0), Hm = key_pos.size(1), cap = key_pos.size(2);
    if (Sq <= 1 || (Bm != 1 && Bm != B) || (Hm != 1 && Hm != Hk) || cap % kTile || !key_pos.is_contiguous() ||
        !slot_mask.is_contiguous() || slot_mask.numel() != key_pos.numel())
      return std::nullopt;
    if (k0.stride(3) != 1 || v0.stride(3) != 1) return std::nullopt;
    for (int i = 0; i < 3; ++i)
      if (k0.stride(i) % 8 || v0.stride(i) % 8) return std::nullopt;
    if ((reinterpret_cast<uintptr_t>(k0.data_ptr()) | reinterpret_cast<uintptr_t>(v0.data_ptr())) & 15) return std::nullopt;
    if (cap > kMaxKeys || (d <= 128 && Sq > kMaxQueries) || H > 65535 || B > 65535) return std::nullopt;
    if (bias0.defined()) {
      // the gathered bias has the bias' own extents: the list must not vary along a dimension the bias is shared over
      if (bias0.size(2) != 1 || bias0.size(3) < Sk || bias0.size(3) == 1) return std::nullopt;
      if ((Bm > 1 && bias0.size(0) != B) || bias0.size(1) % Hm) return std::nullopt;
      if (d > 128 && H != Hk && bias0.size(1) == H) return std::nullopt;  // gradients of such a bias: CUDA-core kernels
      if (d > 128 && (bias0.size(0) != B || bias0.size(1) != Hk)) return std::nullopt;
      c.bias_c = {bias0.size(0), bias0.size(1), 1, cap};
    }
  } else if (bits.defined()) {
    c.bits = true;
    if (d > 128 || Sq == 1 || bits.size(0) != B || bits.size(2) != Sq || bits.size(3) != Sk_r / 32) return std::nullopt;
    if (bits.size(1) != 1 && bits.size(1) != Hk && bits.size(1) != H) return std::nullopt;
    if (!bits.is_contiguous() || !activity.is_contiguous() || (reinterpret_cast<uintptr_t>(bits.data_ptr()) & 15)) return std::nullopt;
    // (the tile table of the backward holds one row of tiles per query head whose mask differs)
    if (Sk > kMaxKeys || round_up(Sq, kTile) * (bits.size(1) == H ? H / Hk : 1) > kMaxQueries || H > 65535 || B > 65535) return std::nullopt;
  } else if (mask0.defined()) {
    if (!plain(mask0) || mask0.scalar_type() != at::kBool || mask0.device() != q0.device() ||
        !broadcastable(mask0, B, H, Hk, Sq) || (mask0.size(3) != 1 && mask0.size(3) != Sk && mask0.size(3) != Sk_r))
      return std::nullopt;
  }
  if (!c.gathered && bias0.defined() && bias0.size(3) != 1 && bias0.size(3) != Sk && bias0.size(3) != Sk_r) return std::nullopt;

  Tensor out, lse, q, k, v, mask, bias, kvb;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    const c10::cuda::CUDAGuard device(q0.device());
    const cudaStream_t stream = stream_of(q0);
    raise_if_timed_out(stream);
    const auto layout = c.gathered || c.bits ? kernel_layout : inner_contiguous;
    q = layout(q0);
    out = empty_as(q);
    lse = empty({B, H, Sq}, at::kFloat, q);
    fdma_fwd_params p = {};
    if (c.gathered) {
      const int64_t cap = key_pos.size(2), kv_elems = B * cap * Hk * d;
      const bool has_bias = bias0.defined();
      const int64_t bytes = 2 * round_up(kv_elems * 2, 256) + (has_bias ? c.bias_c[0] * c.bias_c[1] * cap * 2 : 0);
      kvb = empty({bytes}, at::kByte, q);
      const KvB kv = split_kvb(kvb, kv_elems, has_bias);
      fdma_kept_params g = {};
      const Bsh sk = bsh(k0), sv = bsh(v0);
      g.k = k0.data_ptr(); g.v = v0.data_ptr();
      g.k_c = kv.k; g.v_c = kv.v;
      g.k_batch_stride = sk.b; g.k_row_stride = sk.r; g.k_head_stride = sk.h;
      g.v_batch_stride = sv.b; g.v_row_stride = sv.r; g.v_head_stride = sv.h;
      if (B == 1) g.k_batch_stride = g.v_batch_stride = 0;
      g.key_pos = key_pos.data_ptr<int32_t>();
      g.key_pos_batch_stride = bcast_stride(key_pos, 0);
      g.key_pos_head_stride = key_pos.stride(1);
      g.b = static_cast<int32_t>(B); g.h_k = static_cast<int32_t>(Hk); g.h_pos = static_cast<int32_t>(key_pos.size(1));
      g.seqlen_k = static_cast<int32_t>(Sk); g.capacity = static_cast<int32_t>(cap); g.d = static_cast<int32_t>(d);
      g.dtype = dtype_code(q);
      if (has_bias) {
        g.bias = bias0.data_ptr(); g.bias_c = kv.bias;
        g.bias_batch_stride = bcast_stride(bias0, 0); g.bias_head_stride = bcast_stride(bias0, 1);
        g.bias_key_stride = bias0.stride(3);
        g.bias_b = static_cast<int32_t>(c.bias_c[0]); g.bias_h = static_cast<int32_t>(c.bias_c[1]);
      }
      check(api.gather_kept(&g, stream), "fdma_gather_kept");
      fill_geometry(p, q, cap, Hk, c);
      fill_gathered(p, kv, key_pos, slot_mask, c);
    } else {
      k = layout(k0);
      v = layout(v0);
      if (c.bits) mask = bits;
      else if (mask0.defined()) mask = inner_contiguous(fit_keys(mask0, Sk_r));
      if (bias0.defined()) bias = inner_contiguous(fit_keys(bias0, Sk_r));
      if (c.bits && bias0.defined()) {  // 16-byte loads; expanded dimensions are fine
        bool ok = (reinterpret_cast<uintptr_t>(bias.data_ptr()) & 15) == 0;
        for (int i = 0; i < 3; ++i) ok = ok && bcast_stride(bias, i) % 8 == 0;
        if (!ok) bias = bias.clone(at::MemoryFormat::Contiguous);
      }
      fill_geometry(p, q, Sk, Hk, c);
      fill_kv(p, k, v);
      fill_mask_bias(p, mask, bias, activity, c);
    }
    fill_out(p, out, lse);
    const size_t bytes = api.fwd_workspace_bytes(&p);
    Tensor ws;
    if (bytes) {
      ws = empty({static_cast<int64_t>(bytes)}, at::kByte, q);
      p.workspace = ws.data_ptr();
      p.workspace_bytes = bytes;
    }
    check(api.fwd(&p, stream), "fdma_fwd");
  }
  if (grad) {
    auto node = std::shared_ptr<AttnBackward>(new AttnBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q0, k0, v0, bias0));
    torch::autograd::set_history(out, node);
    node->meta.want_bias = bias0.defined() && (needs_grad(bias0));
    node->meta.k_sizes = k0.sizes().vec();
    if (bias0.defined()) node->meta.bias_sizes = bias0.sizes().vec();
    // tensors made here are saved as they are; the caller's own go in with their version, so in-place edits are noticed
    node->saved[kQ] = SavedVariable(q.is_same(q0) ? q0 : q, false);
    if (c.gathered) {
      node->saved[kK] = SavedVariable(kvb, false);
      node->saved[kMask] = SavedVariable(slot_mask, false);
      node->saved[kExtra] = SavedVariable(key_pos, false);
    } else {
      node->saved[kK] = SavedVariable(k, false);
      node->saved[kV] = SavedVariable(v, false);
      if (mask.defined()) node->saved[kMask] = SavedVariable(mask, false);
      if (bias.defined()) node->saved[kBias] = SavedVariable(bias, false);
      if (activity.defined()) node->saved[kExtra] = SavedVariable(activity, false);
    }
    node->saved[kOut] = SavedVariable(out, /*is_output=*/true);
    node->saved[kLse] = SavedVariable(lse, false);
    node->meta.c = std::move(c);
  }
  return out;
}

// Packed sequences in one launch: q (Tq, H, d), k and v (Tk, Hk, d), cu_q / cu_k (n + 1) int32 on the device, ascending from 0
// to Tq / Tk (the caller has looked). Returns (out, lse (1, H, Tq)); empty for inputs this path does not take.
std::vector<Tensor> packed_attention(const Tensor& q0, const Tensor& k0, const Tensor& v0, const Tensor& cu_q, const Tensor& cu_k,
                                     double scale, bool causal, bool deterministic) {
  for (const Tensor* t : {&q0, &k0, &v0})
    if (!t->defined() || !t->is_cuda() || t->layout() != at::kStrided || t->dim() != 3 || t->device() != q0.device()) return {};
  const auto type = q0.scalar_type();
  if ((type != at::kBFloat16 && type != at::kHalf) || k0.scalar_type() != type || v0.scalar_type() != type) return {};
  const int64_t Tq = q0.size(0), H = q0.size(1), d = q0.size(2), Tk = k0.size(0), Hk = k0.size(1);
  if (Tq <= 0 || Tk <= 0 || H <= 0 || Hk <= 0 || H % Hk || d <= 0 || d % 8 || d > 128 || k0.size(2) != d || v0.sizes() != k0.sizes()) return {};
  if (Hk > 65535 || H > 65535 || Tq > kMaxQueries || Tk > kMaxKeys) return {};
  for (const Tensor* t : {&cu_q, &cu_k})
    if (!t->is_cuda() || t->device() != q0.device() || t->scalar_type() != at::kInt || t->dim() != 1 || !t->is_contiguous() || t->size(0) < 2) return {};
  if (cu_q.size(0) != cu_k.size(0)) return {};
  // what the kernels' TMA loads ask of the tensors; anything else goes sequence by sequence
  for (const Tensor* t : {&q0, &k0, &v0}) {
    if (t->stride(2) != 1 || (reinterpret_cast<uintptr_t>(t->data_ptr()) & 15)) return {};
    for (int i = 0; i < 2; ++i)
      if (t->size(i) > 1 && (t->stride(i) <= 0 || t->stride(i) % 8)) return {};
  }
  const bool grad = at::GradMode::is_enabled() && (needs_grad(q0) || needs_grad(k0) || needs_grad(v0));
  Call c;
  c.scale = static_cast<float>(scale);
  c.causal = causal;
  c.deterministic = deterministic;
  c.packed = true;
  c.seqlen_k = Tk;
  Tensor out, lse, cu;
  {
    at::AutoDispatchBelowADInplaceOrView guard;
    const c10::cuda::CUDAGuard device(q0.device());
    const cudaStream_t stream = stream_of(q0);
    raise_if_timed_out(stream);
    out = empty(q0.sizes(), type, q0);
    lse = empty({1, H, Tq}, at::kFloat, q0);
    const int32_t *pq = cu_q.data_ptr<int32_t>(), *pk = cu_k.data_ptr<int32_t>();
    if (grad) {  // the backward keeps boundaries of its own: the caller may fill its buffers for the next call before
      cu = cu_q.is_same(cu_k) ? cu_q.clone().unsqueeze(0).expand({2, cu_q.size(0)}) : at::stack({cu_q, cu_k});
    }
    fdma_fwd_params p = {};
    const Tensor q4 = q0.unsqueeze(0), k4 = k0.unsqueeze(0);
    fill_geometry(p, q4, Tk, Hk, c);
    fill_kv(p, k4, v0.unsqueeze(0));
    fill_out(p, out.unsqueeze(0), lse);
    check(api.fwd_varlen(&p, pq, pk, static_cast<int32_t>(cu_q.size(0) - 1), stream), "fdma_fwd_varlen");
  }
  if (grad) {
    auto node = std::shared_ptr<AttnBackward>(new AttnBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q0, k0, v0));
    torch::autograd::set_history(out, node);
    node->saved[kQ] = SavedVariable(q0, false);
    node->saved[kK] = SavedVariable(k0, false);
    node->saved[kV] = SavedVariable(v0, false);
    node->saved[kOut] = SavedVariable(out, /*is_output=*/true);
    node->saved[kLse] = SavedVariable(lse, false);
    node->saved[kExtra] = SavedVariable(cu, false);
    node->meta.c = std::move(c);
  }
  return {out, lse};
}

// ---- create_mask -------------------------------------------------------------------------------------------------
// Top-k selection: (mask, key_pos, count, slot_mask) for a row-broadcast bias, (mask, bits, activity) for a per-query one
// where the kernel writes bits, (mask) otherwise. Empty for inputs this path does not take.
std::vector<Tensor> topk_mask(const Tensor& bias, const OptTensor& premask_, int64_t window, double min_value) {
  const Tensor& pm = get(premask_);
  std::vector<Tensor> res;
  if (!plain(bias) || bias.stride(3) != 1 || dtype_code(bias) < 0) return res;
  const int64_t keys = bias.size(3);
  if (window <= 0 || window > keys) return res;
  int64_t shape[3];
  for (int i = 0; i < 3; ++i) shape[i] = bias.size(i);
  if (pm.defined()) {
    if (!plain(pm) || pm.scalar_type() != at::kBool || pm.device() != bias.device() || pm.stride(3) != 1 || pm.size(3) != keys)
      return res;
    for (int i = 0; i < 3; ++i) {
      if (pm.size(i) != shape[i] && pm.size(i) != 1 && shape[i] != 1) return res;
      if (pm.size(i) != 1) shape[i] = pm.size(i);
    }
  }
  const int64_t B = shape[0], Hm = shape[1], rows = shape[2];
  if (B * Hm * rows * keys == 0) return res;
  at::AutoDispatchBelowADInplaceOrView guard;
  const c10::cuda::CUDAGuard device(bias.device());
  const cudaStream_t stream = stream_of(bias);
  fdma_mask_params p = {};
  p.bias = bias.data_ptr();
  p.bias_batch_stride = bcast_stride(bias, 0); p.bias_head_stride = bcast_stride(bias, 1); p.bias_row_stride = bcast_stride(bias, 2);
  if (pm.defined()) {
    p.premask = pm.data_ptr();
    p.pm_batch_stride = bcast_stride(pm, 0); p.pm_head_stride = bcast_stride(pm, 1); p.pm_row_stride = bcast_stride(pm, 2);
  }
  p.out_b = static_cast<int32_t>(B); p.out_h = static_cast<int32_t>(Hm); p.out_rows = static_cast<int32_t>(rows);
  p.keys = static_cast<int32_t>(keys);
  p.window = static_cast<int32_t>(window);
  p.dtype = dtype_code(bias);
  p.kind = FDMA_MASK_TOPK;
  p.min_value = static_cast<float>(min_value);
  Tensor mask = empty({B, Hm, rows, keys}, at::kBool, bias);
  p.out = mask.data_ptr();
  res.push_back(mask);
  if (rows == 1) {
    const int64_t cap = std::max(kTile, round_up(std::min(window, keys), kTile));
    Tensor key_pos = empty({B, Hm, cap}, at::kInt, bias), count = empty({B, Hm}, at::kInt, bias),
           slot_mask = empty({B, Hm, 1, cap}, at::kBool, bias);
    p.key_pos = key_pos.data_ptr<int32_t>();
    p.count = count.data_ptr<int32_t>();
    p.slot_mask = slot_mask.data_ptr();
    p.capacity = static_cast<int32_t>(cap);
    res.insert(res.end(), {key_pos, count, slot_mask});
    check(api.create_mask(&p, stream), "fdma_create_mask");
    return res;
  }
  const int64_t keys_r = round_up(keys, kTile);
  Tensor bits = empty({B, Hm, rows, keys_r / 32}, at::kInt, bias);
  if (keys != keys_r) bits.zero_();  // the kernel writes the bits of keys [0, keys)
  Tensor act = empty({B, Hm, (rows + 127) / 128, keys_r / kTile}, at::kByte, bias);
  p.bits = reinterpret_cast<uint32_t*>(bits.data_ptr<int32_t>());
  p.activity = static_cast<uint8_t*>(act.data_ptr());
  int st = api.create_mask(&p, stream);
  if (st == FDMA_ERR_UNSUPPORTED) {  // rows the bit-writing kernel does not serve: bool mask alone
    p.bits = nullptr;
    p.activity = nullptr;
    st = api.create_mask(&p, stream);
  } else {
    res.push_back(bits);
    res.push_back(act);
  }
  check(st, "fdma_create_mask");
  return res;
}

// ---- Python -----------------------------------------------------------------------------------------------------
// Only exact torch.Tensor / Parameter objects, no active dispatch mode (fake tensors, make_fx) and no torch.jit.trace, which
// records dispatched operators only: everything else is the Python path's.
bool eager() { return !c10::impl::TorchDispatchModeTLS::any_modes_set() && !at::tracer::impl::is_dispatch_enabled(); }
bool exact(PyObject* o) { return THPVariable_CheckExact(o); }
// Tensors that stand for something else (vmap and grad transforms, functionalisation, lazy conjugation) or carry a
// forward-mode tangent are the Python path's as well: the node below has neither batching rules nor a jvp.
bool ordinary(const Tensor& t) {
  constexpr c10::DispatchKeySet kWrapped({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                          c10::DispatchKey::Functionalize, c10::DispatchKey::Python, c10::DispatchKey::Conjugate,
                                          c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  return !t.key_set().has_any(kWrapped) && !t._fw_grad(0).defined();
}
bool as_tensor(const py::handle& o, OptTensor& t) {
  if (o.is_none()) return true;
  if (!exact(o.ptr())) return false;
  t = THPVariable_Unpack(o.ptr());
  return ordinary(*t);
}

py::object py_attention(py::handle q, py::handle k, py::handle v, py::handle mask, py::handle bias, py::handle key_pos,
                        py::handle slot_mask, py::handle bits, py::handle activity, py::handle scale, bool causal,
                        bool deterministic, int path) {
  OptTensor t[9];
  const py::handle in[9] = {q, k, v, mask, bias, key_pos, slot_mask, bits, activity};
  for (int i = 0; i < 9; ++i)
    if (!as_tensor(in[i], t[i])) return py::none();
  if (!t[0] || !t[1] || !t[2] || !eager()) return py::none();
  double s;
  if (scale.is_none()) {
    if (t[0]->dim() != 4) return py::none();
    s = 1.0 / std::sqrt(static_cast<double>(t[0]->size(3)));
  } else {
    s = py::cast<double>(scale);
  }
  std::optional<Tensor> out;
  {
    py::gil_scoped_release release;
    out = attention(*t[0], *t[1], *t[2], t[3], t[4], t[5], t[6], t[7], t[8], s, causal, deterministic, path);
  }
  if (!out) return py::none();
  return py::reinterpret_steal<py::object>(THPVariable_Wrap(*out));
}

py::object py_packed_attention(py::handle q, py::handle k, py::handle v, py::handle cu_q, py::handle cu_k, double scale, bool causal,
                               bool deterministic) {
  OptTensor t[5];
  const py::handle in[5] = {q, k, v, cu_q, cu_k};
  for (int i = 0; i < 5; ++i)
    if (!as_tensor(in[i], t[i]) || !t[i]) return py::none();
  if (!eager()) return py::none();
  std::vector<Tensor> res;
  {
    py::gil_scoped_release release;
    res = packed_attention(*t[0], *t[1], *t[2], *t[3], *t[4], scale, causal, deterministic);
  }
  if (res.empty()) return py::none();
  py::tuple out(res.size());
  for (size_t i = 0; i < res.size(); ++i) out[i] = py::reinterpret_steal<py::object>(THPVariable_Wrap(res[i]));
  return out;
}

py::object py_topk_mask(py::handle bias, py::handle premask, int64_t window, double min_value) {
  OptTensor b, pm;
  if (!as_tensor(bias, b) || !as_tensor(premask, pm) || !b || !eager()) return py::none();
  std::vector<Tensor> res;
  {
    py::gil_scoped_release release;
    res = topk_mask(*b, pm, window, min_value);
  }
  if (res.empty()) return py::none();
  py::tuple out(res.size());
  for (size_t i = 0; i < res.size(); ++i) out[i] = py::reinterpret_steal<py::object>(THPVariable_Wrap(res[i]));
  return out;
}

}  // namespace

PYBIND11_MODULE(_fdma_torch, m) {
  m.def("init", &init);
  m.def("attention", &py_attention);
  m.def("packed_attention", &py_packed_attention);
  m.def("topk_mask", &py_topk_mask);
}
