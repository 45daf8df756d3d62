// Host path of the Python entry points: argument checks, output and scratch tensors, argument structures and the
// sequence of C-ABI calls of one op call, in C++.
//
// The calls these wrap take the GPU a few microseconds when there are few sequences (one decode step: 4 us); a Python
// host path of tensor attribute accesses and ctypes structures took 19 us for one decode call, 60 us for a plain
// forward and 135 to 240 us for a context-parallel one, and that was the time of the call.  Exceptions (types and
// messages) are those of the Python functions that call this module.
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>
#include <torch/version.h>

#include <algorithm>
#include <array>
#include <atomic>

#include "../../include/flashqla_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// The entry points release the GIL (py::gil_scoped_release): torch's allocator and launches may block, and a host callback
// or another Python thread may be what they wait for.  What needs the interpreter takes it back: exceptions, the first look
// at a device's status word, and the result tuple.
[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(type, msg.c_str());
  throw py::error_already_set();
}
[[noreturn]] void value_error(const std::string& msg) { raise(PyExc_ValueError, msg); }
void require(bool ok, const char* msg) {
  if (!ok) raise(PyExc_AssertionError, msg);
}

std::string shape_str(const Tensor& t) {  // as a Python tuple prints
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + (t.dim() == 1 ? ",)" : ")");
}

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return QLA_DT_F32;
    case at::kBFloat16: return QLA_DT_BF16;
    case at::kHalf: return QLA_DT_F16;
    default: value_error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
  }
}
template <typename T = void>
T* ptr(const OptTensor& t) {
  return t.has_value() ? static_cast<T*>(t->data_ptr()) : nullptr;
}
template <typename T = void>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}
Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
Tensor aligned(const Tensor& t, unsigned bytes) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & (bytes - 1)) == 0 ? t : t.clone(); }
Tensor as(const Tensor& t, const at::Device& dev, at::ScalarType dtype) {
  if (t.scalar_type() == dtype && t.device() == dev) return contiguous(t);
  return t.to(dev, dtype).contiguous();
}
Tensor as_i32(const OptTensor& t, const at::Device& dev) { return t.has_value() ? as(*t, dev, at::kInt) : Tensor(); }
Tensor new_tensor(at::IntArrayRef size, at::ScalarType dtype, const at::Device& dev) {
  return at::empty(size, at::TensorOptions().dtype(dtype).device(dev));
}

// The int32 word the kernels of a device report faults to.  It belongs to flashqla_b200.utils, which also reads it;
// the reference kept here is never dropped, so that nothing touches the device when the process ends.
int32_t* status_word(const at::Device& dev) {
  static std::atomic<int32_t*> words[64];
  const int i = dev.index();
  TORCH_CHECK(i >= 0 && i < 64, "device index out of range");
  int32_t* word = words[i].load();
  if (word == nullptr) {
    py::gil_scoped_acquire gil;
    word = (new Tensor(py::module_::import("flashqla_b200.utils").attr("device_status")(py::cast(dev)).cast<Tensor>()))->data_ptr<int32_t>();
    words[i].store(word);
  }
  return word;
}

void check(int code, const char* what) {
  if (code == QLA_OK) return;
  const std::string msg = std::string(what) + ": " + qla_status_string(code) + ": " + qla_last_error();
  if (code == QLA_ERR_INVALID_ARG) value_error(msg);
  if (code == QLA_ERR_UNSUPPORTED) raise(PyExc_NotImplementedError, msg);
  py::gil_scoped_acquire gil;
  raise(py::module_::import("flashqla_b200._cabi").attr("QlaError").ptr(), msg);
}
void* current_stream(const at::Device& dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }
// A tensor of this package that is kept between calls (start order, plan) was allocated on the stream of the call that made
// it: its memory must not go back to that stream while a kernel of this one may still read it.
void used_here(const Tensor& t) {
  c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), c10::cuda::getCurrentCUDAStream(t.get_device()));
}

// ------------------------------------------------------------------------------------------------ recurrent op
Tensor recurrent_update(const OptTensor& A_log_, const Tensor& a_, const OptTensor& dt_bias_, const Tensor& q_, const Tensor& k_,
                        const Tensor& v_, const Tensor& b_, const Tensor& state, const OptTensor& state_indices,
                        std::optional<double> scale, double softplus_beta, double softplus_threshold, bool l2norm,
                        const OptTensor& cu_seqlens, bool disable_state_update, const OptTensor& inter,
                        const OptTensor& inter_indices, std::optional<int64_t> cache_steps, const OptTensor& parent_token,
                        std::optional<int64_t> block_dv, bool assume_regular, bool b_is_beta, bool a_is_log_decay) {
  py::gil_scoped_release nogil;
  if (q_.dim() != 4 || k_.dim() != 4 || v_.dim() != 4) value_error("q, k and v must be [1, total_tokens, heads, 128]");
  if (k_.size(1) < q_.size(1) || k_.size(2) != q_.size(2) || k_.size(3) != q_.size(3) || v_.size(1) < q_.size(1))
    value_error("k must have the shape of q, and v as many tokens");
  const Tensor q = aligned(contiguous(q_), 8), k = aligned(contiguous(k_), 8), v = contiguous(v_), a = contiguous(a_);
  Tensor b = contiguous(b_);
  const int64_t NT = q.size(1), Hk = q.size(2), K = q.size(3), Hv = v.size(2), V = v.size(3);
  if (Hk == 0 || Hv % Hk != 0) value_error("num_value_heads must be divisible by num_key_heads");
  if (K != 128 || V != 128) value_error("FlashQLA recurrent GDN kernel currently specializes Qwen GDN K=V=128");
  if (a.sizes() != at::IntArrayRef({1, NT, Hv})) value_error("a shape " + shape_str(a) + " does not match [1, total_tokens, HV]");
  if (b.sizes() != at::IntArrayRef({1, NT, Hv})) value_error("b shape " + shape_str(b) + " does not match [1, total_tokens, HV]");
  if (a.scalar_type() != b.scalar_type()) b = b.to(a.scalar_type());
  Tensor A_log, dt_bias;
  if (!a_is_log_decay) {
    if (!A_log_.has_value() || A_log_->sizes() != at::IntArrayRef({Hv})) value_error("A_log must have shape [HV]");
    if (!dt_bias_.has_value() || dt_bias_->sizes() != at::IntArrayRef({Hv})) value_error("dt_bias must have shape [HV]");
    A_log = contiguous(*A_log_);
    dt_bias = contiguous(*dt_bias_);
  }
  // The pool is updated in place, so a non-contiguous one (which the reference would silently copy, losing the
  // update: recurrent_fused.py:6270-6284) is rejected.
  if (state.dim() != 4) value_error("initial_state_source must be a 4-D tensor");
  if (state.size(1) != Hv)
    value_error("initial_state_source head dim " + std::to_string(state.size(1)) + " != num_value_heads " + std::to_string(Hv));
  if (state.size(2) != V || state.size(3) != K)
    value_error("initial_state_source must have trailing shape [V, K] for recurrent GDN layout "
                "or [K, V] when K == V-compatible contiguous storage is intended");
  if (!state.is_contiguous()) value_error("initial_state_source must be contiguous: it is updated in place");
  if (state.scalar_type() != at::kFloat && state.scalar_type() != at::kBFloat16)
    raise(PyExc_NotImplementedError, "initial_state_source must be float32 or bfloat16");
  const at::Device dev = q.device();
  Tensor cu = as_i32(cu_seqlens, dev);
  const Tensor sidx = as_i32(state_indices, dev);
  const int64_t N = cu.defined() ? cu.numel() - 1 : sidx.defined() ? sidx.numel() : state.size(0);
  if (sidx.defined() && sidx.numel() != N) value_error("initial_state_indices length must equal num_sequences");
  if (!sidx.defined() && N > state.size(0)) value_error("cu_seqlens length must equal num_sequences + 1");
  int64_t tokens_per_seq = 0;
  if (!cu.defined() || assume_regular) {
    if (N == 0 || NT % N != 0)
      value_error(assume_regular ? "assume_regular=True requires total_tokens divisible by num_sequences"
                                 : "total_tokens must be divisible by num_sequences when cu_seqlens is omitted");
    tokens_per_seq = NT / N;
    cu = Tensor();
  }
  Tensor cidx;
  int64_t inter_steps = 0;
  if (inter.has_value()) {
    if (inter->dim() != 5 || inter->size(2) != Hv || inter->size(3) != V || inter->size(4) != K)
      value_error("intermediate_states_buffer must be [slots, steps, HV, V, K]");
    if (!inter->is_contiguous()) value_error("intermediate_states_buffer must be contiguous: it is written in place");
    if (inter->scalar_type() != at::kFloat && inter->scalar_type() != at::kBFloat16)
      raise(PyExc_NotImplementedError, "intermediate_states_buffer must be float32 or bfloat16");
    inter_steps = inter->size(1);
    if (inter_steps < cache_steps.value_or(inter_steps))
      value_error("intermediate_states_buffer cache dimension is smaller than cache_steps");
    cidx = as_i32(inter_indices, dev);
    if (!cidx.defined() && inter->size(0) < N) value_error("intermediate_states_buffer must have at least num_sequences slots");
    if (tokens_per_seq > inter_steps)
      value_error("intermediate_states_buffer cache dimension is smaller than tokens per sequence");
  }
  const Tensor parents = as_i32(parent_token, dev);
  if (parents.defined()) {
    if (!inter.has_value()) value_error("retrieve_parent_token requires intermediate_states_buffer");
    if (parents.dim() != 2 || parents.size(0) != N) value_error("retrieve_parent_token first dimension must equal num_sequences");
    if (tokens_per_seq > parents.size(1)) value_error("retrieve_parent_token has fewer columns than tokens per sequence");
  }

  c10::cuda::OptionalCUDAGuard guard(dev);
  const Tensor o = at::empty_like(v);
  QlaRecurrentArgs r{};
  r.num_seqs = N; r.total_tokens = NT; r.tokens_per_seq = tokens_per_seq; r.num_k_heads = Hk; r.num_v_heads = Hv;
  r.qkv_dtype = dtype_code(q); r.a_dtype = dtype_code(a);
  r.a_log_dtype = a_is_log_decay ? 0 : dtype_code(A_log);
  r.dt_bias_dtype = a_is_log_decay ? 0 : dtype_code(dt_bias);
  r.inter_dtype = inter.has_value() ? dtype_code(*inter) : 0;
  r.inter_steps = inter_steps; r.parents_stride = parents.defined() ? parents.stride(0) : 0;
  r.flags = (l2norm ? QLA_REC_QK_L2NORM : 0) | (disable_state_update ? QLA_REC_DISABLE_STATE_UPDATE : 0) |
            (a_is_log_decay ? QLA_REC_A_IS_LOG_DECAY : 0) | (b_is_beta ? QLA_REC_B_IS_BETA : 0);
  r.rows_per_cta = !block_dv.has_value() ? 0 : (*block_dv <= 16 ? 16 : 32);
  r.state_slots = state.size(0); r.inter_slots = inter.has_value() ? inter->size(0) : 0;
  r.scale = scale.has_value() ? *scale : 1.0 / std::sqrt(static_cast<double>(K));
  r.softplus_beta = softplus_beta; r.softplus_threshold = softplus_threshold;
  r.A_log = ptr(A_log); r.a = ptr(a); r.dt_bias = ptr(dt_bias); r.q = ptr(q); r.k = ptr(k); r.v = ptr(v); r.b = ptr(b);
  r.state = ptr(state); r.state_indices = ptr<int32_t>(sidx); r.cu_seqlens = ptr<int32_t>(cu); r.inter = ptr(inter);
  r.inter_indices = ptr<int32_t>(cidx); r.parents = ptr<int32_t>(parents); r.o = ptr(o); r.status = status_word(dev);
  r.state_dtype = dtype_code(state); r.parents_steps = parents.defined() ? parents.size(1) : 0;
  check(qla_recurrent_update(&r, current_stream(dev)), "qla_recurrent_update");
  return o;
}

void state_commit(const Tensor& state, const Tensor& inter, const Tensor& num_accepted, const OptTensor& state_indices,
                  const OptTensor& inter_indices) {
  py::gil_scoped_release nogil;
  if (inter.dim() != 5 || inter.size(3) != 128 || inter.size(4) != 128)
    value_error("intermediate_states_buffer must be [slots, steps, HV, 128, 128]");
  const int64_t Hv = inter.size(2), elems = Hv * 128 * 128;
  if (Hv == 0) value_error("intermediate_states_buffer has no heads");
  if (!state.is_contiguous() || !inter.is_contiguous())
    value_error("the state pool and intermediate_states_buffer must be contiguous");
  if ((state.scalar_type() != at::kFloat && state.scalar_type() != at::kBFloat16) || state.numel() % elems != 0)
    value_error("initial_state_source must be a float32 or bfloat16 pool of [HV, 128, 128] states");
  if (inter.scalar_type() != at::kFloat && inter.scalar_type() != at::kBFloat16)
    raise(PyExc_NotImplementedError, "intermediate_states_buffer must be float32 or bfloat16");
  const at::Device dev = state.device();
  const Tensor acc = as(num_accepted, dev, at::kInt), sidx = as_i32(state_indices, dev), cidx = as_i32(inter_indices, dev);
  c10::cuda::OptionalCUDAGuard guard(dev);
  QlaStateCommitArgs c{};
  c.num_seqs = acc.numel(); c.num_v_heads = Hv; c.inter_dtype = dtype_code(inter); c.inter_steps = inter.size(1);
  c.inter_slots = inter.size(0); c.state_slots = state.numel() / elems; c.inter = ptr(inter); c.accepted = ptr<int32_t>(acc);
  c.state_indices = ptr<int32_t>(sidx); c.inter_indices = ptr<int32_t>(cidx); c.state = ptr(state); c.status = status_word(dev);
  c.state_dtype = dtype_code(state);
  check(qla_state_commit(&c, current_stream(dev)), "qla_state_commit");
}

// ------------------------------------------------------------------------------------------------ chunked op
// Context-parallel plan of one list of sequence lengths (flashqla_b200/cp.py): device tables, made once per plan.
struct Plan {
  Tensor cu, seg_next, seg_raw, raw_first, identity, seg_start_of, seg_prev, tables;
  int64_t num_segments, num_raw;
};

struct Sizes {
  int64_t B, T, Hk, Hv, N;
};
Sizes chunk_check(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                  const OptTensor& initial_state, const OptTensor& cu_seqlens, bool transpose_state_layout) {
  require(q.scalar_type() == k.scalar_type() && k.scalar_type() == v.scalar_type(), "q, k, v must share a dtype");
  require(q.scalar_type() != at::kFloat, "ChunkGatedDeltaRuleFunction does not support float32. Please use bfloat16.");
  require(q.dim() == 4 && k.sizes() == q.sizes() && v.dim() == 4, "q,k [B,T,Hk,K]; v [B,T,Hv,V]");
  Sizes s{q.size(0), q.size(1), q.size(2), v.size(2), q.size(0)};
  require(v.size(0) == s.B && v.size(1) >= s.T, "q,k [B,T,Hk,K]; v [B,T,Hv,V]");
  require(q.size(3) == 128 && v.size(3) == 128, "K = V = 128 only");
  require(s.Hk > 0 && s.Hv % s.Hk == 0, "the number of v heads must be a multiple of the number of q/k heads");
  const std::array<int64_t, 3> gates{s.B, s.T, s.Hv};
  require(g.sizes() == at::IntArrayRef(gates) && beta.sizes() == at::IntArrayRef(gates), "g, beta must be [B,T,Hv]");
  if (cu_seqlens.has_value()) {
    if (s.B != 1)
      value_error("The batch size is expected to be 1 rather than " + std::to_string(s.B) + " when using `cu_seqlens`."
                  "Please flatten variable-length inputs before processing.");
    s.N = cu_seqlens->numel() - 1;
  }
  if (initial_state.has_value()) {
    if (initial_state->dim() == 0 || initial_state->size(0) != s.N)
      value_error("The number of initial states is expected to be equal to the number of input sequences, i.e., " +
                  std::to_string(s.N) + " rather than " + std::to_string(initial_state->dim() ? initial_state->size(0) : 0) + ".");
    if (initial_state->sizes() != at::IntArrayRef({s.N, s.Hv, 128, 128}))
      value_error("initial_state must have shape (" + std::to_string(s.N) + ", " + std::to_string(s.Hv) +
                  ", 128, 128), got " + shape_str(*initial_state));
  }
  (void)transpose_state_layout;  // K = V: both layouts have the same shape
  return s;
}
py::tuple chunk_check_py(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta,
                         const OptTensor& initial_state, const OptTensor& cu_seqlens, bool transpose_state_layout) {
  const Sizes s = chunk_check(q, k, v, g, beta, initial_state, cu_seqlens, transpose_state_layout);
  return py::make_tuple(s.B, s.T, s.Hk, s.Hv, s.N);
}

int64_t chunks_of(int64_t tokens) { return (tokens + 63) / 64; }
// Chunk states of a packed batch.  The storage has room for as many chunks as any `seqs` intervals of `tokens` can have:
// the scan numbers chunks by what cu_seqlens holds when it runs, `n_chunks` is what it held when its lengths were read.
Tensor new_h(int64_t n_chunks, int64_t tokens, int64_t seqs, int64_t heads, at::ScalarType dtype, const at::Device& dev) {
  return new_tensor({std::max(n_chunks, tokens / 64 + seqs), heads, 128, 128}, dtype, dev).narrow(0, 0, n_chunks);
}

// Plan (+ start states) -> warm-up and transition passes (one launch) -> chaining, on the segments of `plan`; `a` is
// filled for the main scan.  The scratch holds, per segment and head, the two limits and the warm-up lengths, the
// state a segment starts from (fp32 [K][V]) and the transition matrices.
struct SegmentScratch {
  Tensor ints, h0, M;
  int32_t *warm_limit, *m_limit, *lead;
};
SegmentScratch segment_scratch(const Plan& p, int64_t Hv, const at::Device& dev, bool inline_warmup) {
  SegmentScratch s;
  const int64_t n = p.num_segments * Hv;
  s.ints = new_tensor({3, n}, at::kInt, dev);
  s.warm_limit = s.ints.data_ptr<int32_t>();
  s.m_limit = s.warm_limit + n;
  s.lead = inline_warmup ? s.warm_limit + 2 * n : nullptr;
  s.h0 = new_tensor({p.num_segments, Hv, 128, 128}, at::kFloat, dev);
  s.M = new_tensor({p.num_segments, Hv, 128, 128}, at::kFloat, dev);
  return s;
}
void segment_plan(const Plan& p, double threshold, const SegmentScratch& s, int64_t Hv, const float* g_cumsum, const OptTensor& h0,
                  const int32_t* h0_map, bool h0_transposed, bool reverse, void* stream) {
  QlaCpPlanArgs a{};
  a.num_segments = p.num_segments; a.num_v_heads = Hv; a.threshold = threshold; a.g_cumsum = g_cumsum;
  a.cu_seqlens = ptr<int32_t>(p.cu); a.seg_next = ptr<int32_t>(reverse ? p.seg_prev : p.seg_next);
  a.warm_limit = s.warm_limit; a.m_limit = s.m_limit; a.cp_h0 = s.h0.data_ptr<float>();
  a.seg_start_of = ptr<int32_t>(reverse ? p.seg_raw : p.seg_start_of); a.h0 = ptr(h0); a.h0_map = h0_map;
  a.h0_dtype = h0.has_value() ? dtype_code(*h0) : QLA_DT_F32; a.h0_transposed = h0_transposed; a.reverse = reverse;
  a.num_raw_seqs = p.num_raw; a.lead = s.lead; a.raw_first_seg = ptr<int32_t>(p.raw_first);
  check(qla_cp_plan(&a, stream), "qla_cp_plan");
}
void segment_chain(const Plan& p, const SegmentScratch& s, int64_t Hv, bool reverse, void* stream) {
  QlaCpChainArgs a{};
  a.num_raw_seqs = p.num_raw; a.num_v_heads = Hv; a.h0 = s.h0.data_ptr<float>(); a.M = s.M.data_ptr<float>();
  a.m_limit = s.m_limit; a.raw_first_seg = ptr<int32_t>(p.raw_first); a.reverse = reverse;
  a.has_status = 1; a.status = status_word(s.h0.device());
  check(qla_cp_chain(&a, stream), "qla_cp_chain");
}
void use_tables(QlaChunkFwdArgs& a, const Tensor& tables) {
  a.workspace = tables.data_ptr();
  a.workspace_bytes = tables.nbytes();
  a.flags |= QLA_CHUNK_TABLES_READY;
}
// Workspace for the chunk tables of the caller's cu_seqlens, which a launch of the call derives from what the tensor holds
// then: a table kept from an earlier call would be stale after a write that no version counter sees (a graph replay, a raw
// kernel).  The returned tensor keeps the workspace alive.
Tensor table_workspace(QlaChunkFwdArgs& a, const at::Device& dev) {
  if (a.cu_seqlens == nullptr) return Tensor();
  Tensor ws = new_tensor({static_cast<int64_t>(qla_chunk_fwd_workspace_bytes(&a))}, at::kByte, dev);
  a.workspace = ws.data_ptr();
  a.workspace_bytes = ws.nbytes();
  return ws;
}

// The raw forward (chunk.chunk_gated_delta_rule_fwd says what the arguments mean).  `order` is the order in which the
// sequences of cu_seqlens are started, `plan` the context-parallel plan or None.  Without `keep` (and h, v_new) A and w are not
// wanted either.
py::tuple chunk_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_,
                    std::optional<double> scale, const OptTensor& initial_state, const OptTensor& initial_state_indices,
                    const OptTensor& cu_seqlens, const OptTensor& order, int64_t n_chunks,
                    bool output_final_state, bool output_h, bool output_v_new, bool transposed, bool l2norm,
                    const OptTensor& A_log_, const OptTensor& dt_bias_, bool beta_is_logit, const OptTensor& final_state_out,
                    const OptTensor& final_state_indices, const OptTensor& norm_gate, const OptTensor& norm_weight,
                    double norm_eps, const Plan* plan, bool inline_warmup, double threshold, bool keep) {
  py::gil_scoped_release nogil;
  const Sizes s = chunk_check(q_, k_, v_, g_, beta_, initial_state_indices.has_value() ? OptTensor() : initial_state, cu_seqlens,
                              transposed);
  if (A_log_.has_value() != dt_bias_.has_value()) value_error("A_log and dt_bias go together");
  if (!q_.is_cuda()) value_error("flashqla_b200 requires CUDA tensors");
  const at::Device dev = q_.device();
  const auto dtype = q_.scalar_type();
  const Tensor q = contiguous(q_), k = contiguous(k_), v = contiguous(v_), g = contiguous(g_);
  Tensor beta = contiguous(beta_);
  const bool pooled = initial_state_indices.has_value() || final_state_out.has_value();
  const int64_t B = s.B, T = s.T, Hk = s.Hk, Hv = s.Hv, N = s.N;
  auto is_pool = [&](const Tensor& t) { return t.dim() == 4 && t.size(1) == Hv && t.size(2) == 128 && t.size(3) == 128; };
  auto pool_type = [](const Tensor& t) {
    return (t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16) && t.is_contiguous();
  };
  OptTensor h0;
  Tensor h0_map, fs_map;
  if (initial_state.has_value()) {
    if (initial_state_indices.has_value()) {
      if (!is_pool(*initial_state))
        value_error("a state pool must be [slots, " + std::to_string(Hv) + ", 128, 128], got " + shape_str(*initial_state));
      if (!pool_type(*initial_state)) value_error("a state pool must be a contiguous float32 or bfloat16 tensor");
      if (initial_state_indices->numel() != N)
        value_error("initial_state_indices must have one entry per sequence (" + std::to_string(N) + ")");
      h0 = *initial_state;
      h0_map = as_i32(initial_state_indices, dev);
    } else {
      const bool keep = pooled && initial_state->scalar_type() == at::kBFloat16;
      h0 = keep ? contiguous(*initial_state) : as(*initial_state, initial_state->device(), at::kFloat);
    }
  }
  if (final_state_out.has_value()) {
    if (!is_pool(*final_state_out))
      value_error("final_state_out must be [rows, " + std::to_string(Hv) + ", 128, 128], got " + shape_str(*final_state_out));
    if (!pool_type(*final_state_out)) value_error("final_state_out must be a contiguous float32 or bfloat16 tensor");
    if (h0.has_value() && h0->scalar_type() != final_state_out->scalar_type())
      value_error("initial states and final_state_out must share a dtype");
    if (final_state_indices.has_value()) {
      if (final_state_indices->numel() != N)
        value_error("final_state_indices must have one entry per sequence (" + std::to_string(N) + ")");
      fs_map = as_i32(final_state_indices, dev);
    } else if (final_state_out->size(0) < N) {
      value_error("final_state_out needs one row per sequence");
    }
  } else if (final_state_indices.has_value()) {
    value_error("final_state_indices needs final_state_out");
  }
  Tensor gate, weight;
  if (norm_gate.has_value()) {
    if (!norm_weight.has_value() || norm_weight->numel() < 128 || norm_gate->sizes() != v.sizes() || norm_gate->scalar_type() != v.scalar_type())
      value_error("out_norm_gate must have v's shape and dtype and needs out_norm_weight [128]");
    if (output_h || output_v_new) value_error("the output norm is an inference epilogue: not with output_h / output_v_new");
    gate = aligned(contiguous(*norm_gate), 16);
    weight = aligned(as(*norm_weight, dev, at::kFloat), 16);
  }

  c10::cuda::OptionalCUDAGuard guard(dev);
  void* stream = current_stream(dev);
  const Tensor cu = as_i32(cu_seqlens, dev);
  const Tensor g_cumsum = new_tensor({B, T, Hv}, at::kFloat, dev), A = new_tensor({B, T, Hv, 64}, dtype, dev);
  // A call that keeps neither A nor w: the scan forms w itself, and A is scratch in its own form.  The results are the same bits, and
  // no size was found where it is slower (whole calls, us, with w / without: 1 x 64 tokens of 16 / 32 heads 14.6 / 12.8, 1 x 777 34.0 /
  // 33.7, 8 x 500 of 8 / 8 heads 28.0 / 27.0; preparation + scan: 64 chains of 32 chunks 68 / 59, 512 of 32 431 / 382, 512 of 4 85 / 74,
  // 8000 of 1 498 / 480).
  const bool w_in_scan = !keep && !output_h && !output_v_new;
  const Tensor w = new_tensor({B, T, Hv, w_in_scan ? 64 : 128}, dtype, dev), o = at::empty_like(v);
  Tensor h, v_new, rnorm, beta_act, final_state, A_log, dt_bias;
  if (output_h)
    h = cu.defined() ? new_h(n_chunks, T, N, Hv, dtype, dev).unsqueeze(0) : new_tensor({B, chunks_of(T), Hv, 128, 128}, dtype, dev);
  if (output_v_new) v_new = at::empty_like(v);
  if (l2norm) rnorm = new_tensor({B, T, Hk, 2}, at::kFloat, dev);
  if (final_state_out.has_value()) final_state = *final_state_out;
  else if (output_final_state)
    final_state = new_tensor({N, Hv, 128, 128}, (h0.has_value() && pooled) ? h0->scalar_type() : at::kFloat, dev);
  if (A_log_.has_value()) {
    A_log = as(*A_log_, dev, at::kFloat);
    dt_bias = as(*dt_bias_, dev, at::kFloat);
  }
  if (beta_is_logit) beta_act = new_tensor({B, T, Hv}, at::kFloat, dev);

  QlaChunkFwdArgs a{};
  a.batch = B; a.seq_len = T; a.num_seqs = N; a.num_k_heads = Hk; a.num_v_heads = Hv;
  a.qkv_dtype = dtype_code(q); a.gate_dtype = dtype_code(g); a.beta_dtype = dtype_code(beta);
  a.scale = scale.has_value() ? *scale : 1.0 / std::sqrt(128.0);
  a.q = ptr(q); a.k = ptr(k); a.v = ptr(v); a.g = ptr(g); a.beta = ptr(beta);
  a.g_cumsum = ptr<float>(g_cumsum); a.A = ptr(A); a.w = ptr(w); a.qk_rnorm = ptr<float>(rnorm);
  a.A_log = ptr<float>(A_log); a.dt_bias = ptr<float>(dt_bias); a.beta_out = ptr<float>(beta_act);
  a.status = status_word(dev); a.cu_seqlens = ptr<int32_t>(cu);
  const int norm_flag = (l2norm ? QLA_CHUNK_QK_L2NORM : 0) | (w_in_scan ? QLA_CHUNK_W_IN_SCAN : 0);
  const int act_flags = (A_log.defined() ? QLA_CHUNK_GATE_ACT : 0) | (beta_is_logit ? QLA_CHUNK_BETA_LOGIT : 0);
  const int out_flag = gate.defined() ? QLA_CHUNK_OUT_GATED_RMSNORM : 0, layout = transposed ? QLA_CHUNK_TRANSPOSE_STATE : 0;
  if (final_state.defined() || h0.has_value()) a.state_dtype = dtype_code(final_state.defined() ? final_state : *h0);

  if (plan != nullptr) {
    used_here(plan->cu);  // (every table of a plan lies in one allocation)
    // g_cumsum, A and w on the original sequences, then per-segment initial states, then the scan over segments
    // (segments are whole chunks, so chunk numbering is unchanged)
    a.flags = QLA_CHUNK_PREPARE_ONLY | norm_flag | act_flags;
    const Tensor ws = table_workspace(a, dev);
    check(qla_chunk_fwd(&a, stream), "qla_chunk_fwd");
    if (beta_is_logit) {  // every later stage reads the activated values
      a.beta = a.beta_out;
      a.beta_dtype = QLA_DT_F32;
    }
    const SegmentScratch sc = segment_scratch(*plan, Hv, dev, inline_warmup);
    segment_plan(*plan, threshold, sc, Hv, a.g_cumsum, h0, ptr<int32_t>(h0_map), transposed, false, stream);
    // One launch, two passes: segment-end states from the trailing `warm_limit` chunks, written straight into the
    // successor's row, and the transition matrices of the (segment, head) pairs that never decayed below the threshold.
    QlaChunkFwdArgs b = a;
    b.batch = 1; b.seq_len = B * T; b.num_seqs = plan->num_segments; b.cu_seqlens = ptr<int32_t>(plan->cu);
    b.g = nullptr; b.A_log = nullptr; b.dt_bias = nullptr; b.beta_out = nullptr;
    use_tables(b, plan->tables);
    const int state_dtype = b.state_dtype;
    b.flags = QLA_CHUNK_STATE_ONLY | QLA_CHUNK_SKIP_PREPARE | QLA_CHUNK_DUAL_TRANSITION | QLA_CHUNK_TABLES_READY | norm_flag;
    b.state_dtype = QLA_DT_F32; b.final_state = ptr(sc.h0); b.seq_map = ptr<int32_t>(plan->seg_next);
    b.chunk_limit = sc.warm_limit; b.chunk_limit_b = sc.m_limit; b.seq_map_b = ptr<int32_t>(plan->identity);
    b.final_state_b = ptr<float>(sc.M);
    check(qla_chunk_fwd(&b, stream), "qla_chunk_fwd");
    segment_chain(*plan, sc, Hv, false, stream);
    b.flags = QLA_CHUNK_SKIP_PREPARE | QLA_CHUNK_H0_KV_F32 | QLA_CHUNK_TABLES_READY | layout | norm_flag | out_flag;
    b.state_dtype = state_dtype; b.chunk_limit = b.chunk_limit_b = b.seq_map_b = nullptr; b.final_state_b = nullptr;
    b.h0 = ptr(sc.h0); b.lead = sc.lead; b.seq_map = ptr<int32_t>(plan->seg_raw); b.final_map = ptr<int32_t>(fs_map);
    b.o = ptr(o); b.h = ptr(h); b.v_new = ptr(v_new); b.final_state = ptr(final_state);
    b.norm_gate = ptr(gate); b.norm_weight = ptr<float>(weight); b.norm_eps = norm_eps;
    check(qla_chunk_fwd(&b, stream), "qla_chunk_fwd");
  } else {
    a.flags = layout | norm_flag | act_flags | out_flag;
    const Tensor ws = table_workspace(a, dev);
    if (order.has_value()) used_here(*order);
    a.seq_order = ptr<int32_t>(order);  // packed batches of unequal lengths: the longest sequences start first
    a.h0 = ptr(h0); a.h0_map = ptr<int32_t>(h0_map); a.seq_map = ptr<int32_t>(fs_map);
    a.o = ptr(o); a.h = ptr(h); a.v_new = ptr(v_new); a.final_state = ptr(final_state);
    a.norm_gate = ptr(gate); a.norm_weight = ptr<float>(weight); a.norm_eps = norm_eps;
    check(qla_chunk_fwd(&a, stream), "qla_chunk_fwd");
  }
  py::gil_scoped_acquire gil;
  auto opt = [](const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); };
  return py::make_tuple(g_cumsum, w_in_scan ? py::none() : py::cast(A), o, opt(h), opt(final_state), opt(v_new),
                        w_in_scan ? py::none() : py::cast(w), opt(rnorm), opt(beta_act));
}

// The raw backward (chunk.chunk_gated_delta_rule_bwd): `g_` is the cumulative gate of the forward, `order` the order in which the
// sequences of cu_seqlens are started.
py::tuple chunk_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, const Tensor& A_,
                    const Tensor& do_, const OptTensor& dht_, std::optional<double> scale_, const OptTensor& initial_state,
                    const OptTensor& cu_seqlens, const OptTensor& order, int64_t n_chunks, const OptTensor& h_,
                    const OptTensor& v_new_, bool transposed, const OptTensor& w_, const Plan* plan, bool inline_warmup,
                    double threshold) {
  py::gil_scoped_release nogil;
  const Sizes s = chunk_check(q_, k_, v_, g_, beta_, initial_state, cu_seqlens, transposed);
  if (!q_.is_cuda()) value_error("flashqla_b200 requires CUDA tensors");
  const at::Device dev = q_.device();
  const auto dtype = q_.scalar_type();
  const Tensor q = contiguous(q_), k = contiguous(k_), v = contiguous(v_), beta = contiguous(beta_), A = contiguous(A_);
  const Tensor d_o = contiguous(do_.scalar_type() == dtype ? do_ : do_.to(dtype)), g_cumsum = contiguous(g_.to(at::kFloat));
  const int64_t B = s.B, T = s.T, Hk = s.Hk, Hv = s.Hv;
  const float scale = scale_.has_value() ? *scale_ : 1.0 / std::sqrt(128.0);
  OptTensor h0, dht;
  if (initial_state.has_value()) h0 = contiguous(initial_state->to(at::kFloat));
  if (dht_.has_value()) dht = contiguous(dht_->to(at::kFloat));

  c10::cuda::OptionalCUDAGuard guard(dev);
  void* stream = current_stream(dev);
  const Tensor cu = as_i32(cu_seqlens, dev);
  const int layout = transposed ? QLA_CHUNK_TRANSPOSE_STATE : 0;
  Tensor h = h_.value_or(Tensor()), v_new = v_new_.value_or(Tensor()), w = w_.value_or(Tensor());
  if (!h.defined() || !v_new.defined() || !w.defined()) {
    // what the forward did not keep is recomputed: h and v_new by a state-only scan, w on its way (or alone)
    QlaChunkFwdArgs a{};
    const bool scan = !h.defined() || !v_new.defined(), have_w = w.defined();
    if (scan) {
      h = cu.defined() ? new_h(n_chunks, T, s.N, Hv, dtype, dev) : new_tensor({n_chunks, Hv, 128, 128}, dtype, dev);
      v_new = at::empty_like(v);
    }
    if (!have_w) w = new_tensor({B, T, Hv, 128}, dtype, dev);
    w = contiguous(w);
    a.batch = B; a.seq_len = T; a.num_seqs = s.N; a.num_k_heads = Hk; a.num_v_heads = Hv; a.qkv_dtype = dtype_code(q);
    a.gate_dtype = QLA_DT_F32; a.beta_dtype = dtype_code(beta); a.scale = scale;
    a.k = ptr(k); a.v = ptr(v); a.beta = ptr(beta); a.cu_seqlens = ptr<int32_t>(cu); a.g_cumsum = ptr<float>(g_cumsum);
    a.A = ptr(A); a.w = ptr(w); a.status = status_word(dev); a.state_dtype = QLA_DT_F32;
    a.flags = have_w ? QLA_CHUNK_SKIP_PREPARE : QLA_CHUNK_A_GIVEN;
    if (scan) {
      a.flags |= layout | QLA_CHUNK_STATE_ONLY;
      a.h0 = ptr(h0); a.h = ptr(h); a.v_new = ptr(v_new);
    } else {
      a.flags |= QLA_CHUNK_PREPARE_ONLY;
    }
    const Tensor ws = table_workspace(a, dev);
    check(qla_chunk_fwd(&a, stream), "qla_chunk_fwd");
  }
  w = contiguous(w); h = contiguous(h); v_new = contiguous(v_new);

  const Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  const Tensor db = new_tensor({B, T, Hv}, at::kFloat, dev), dg = new_tensor({B, T, Hv}, at::kFloat, dev);
  Tensor dh0;
  if (h0.has_value()) dh0 = new_tensor({s.N, Hv, 128, 128}, at::kFloat, dev);
  QlaChunkBwdArgs a{};
  a.batch = B; a.seq_len = T; a.num_seqs = s.N; a.num_k_heads = Hk; a.num_v_heads = Hv; a.qkv_dtype = dtype_code(q);
  a.beta_dtype = dtype_code(beta); a.flags = layout; a.scale = scale;
  a.q = ptr(q); a.k = ptr(k); a.v = ptr(v); a.g_cumsum = ptr<float>(g_cumsum); a.beta = ptr(beta); a.A = ptr(A); a.h = ptr(h);
  a.v_new = ptr(v_new); a.w = ptr(w); a.d_o = ptr(d_o); a.dht = ptr<float>(dht); a.cu_seqlens = ptr<int32_t>(cu);
  a.dq = ptr(dq); a.dk = ptr(dk); a.dv = ptr(dv); a.dbeta = ptr<float>(db); a.dg = ptr<float>(dg); a.dh0 = ptr<float>(dh0);
  a.status = status_word(dev);
  SegmentScratch sc;
  if (plan != nullptr) {
    // Long sequences on few heads: the reverse scan runs over the same segments as the forward's.  Plan (reverse:
    // decay accumulated from a segment's START; rows of the last segments take the caller's dht) -> one launch of
    // the scan in state-only mode over the leading chunks of every segment together with the transition matrices
    // -> reverse chaining.
    used_here(plan->cu);
    sc = segment_scratch(*plan, Hv, dev, inline_warmup);
    segment_plan(*plan, threshold, sc, Hv, a.g_cumsum, dht, nullptr, transposed, true, stream);
    QlaChunkBwdArgs b{};
    b.batch = 1; b.seq_len = B * T; b.num_seqs = plan->num_segments; b.num_k_heads = Hk; b.num_v_heads = Hv;
    b.qkv_dtype = a.qkv_dtype; b.beta_dtype = QLA_DT_F32; b.flags = QLA_CHUNK_STATE_ONLY | QLA_CHUNK_DUAL_TRANSITION;
    b.scale = scale; b.q = a.q; b.k = a.k; b.g_cumsum = a.g_cumsum; b.w = a.w; b.d_o = a.d_o; b.status = a.status;
    b.cu_seqlens = ptr<int32_t>(plan->cu); b.dh0 = ptr<float>(sc.h0); b.chunk_limit = sc.warm_limit;
    b.out_map = ptr<int32_t>(plan->seg_prev); b.chunk_limit_b = sc.m_limit; b.out_map_b = ptr<int32_t>(plan->identity);
    b.out_b = ptr<float>(sc.M);
    check(qla_chunk_bwd(&b, stream), "qla_chunk_bwd (state-only)");
    segment_chain(*plan, sc, Hv, true, stream);
    a.num_segments = plan->num_segments; a.seg_cu = ptr<int32_t>(plan->cu); a.seg_dht = ptr<float>(sc.h0);
    a.seg_dh0_map = ptr<int32_t>(plan->seg_start_of); a.seg_lead = sc.lead; a.seg_tables = ptr<int32_t>(plan->tables);
  } else if (order.has_value()) {
    used_here(*order);
    a.seq_order = ptr<int32_t>(order);
  }
  const size_t bytes = qla_chunk_bwd_workspace_bytes(&a);
  const Tensor ws = new_tensor({static_cast<int64_t>(bytes)}, at::kByte, dev);
  a.workspace = ws.data_ptr();
  a.workspace_bytes = bytes;
  check(qla_chunk_bwd(&a, stream), "qla_chunk_bwd");
  py::gil_scoped_acquire gil;
  return py::make_tuple(dq, dk, dv, db, dg, dh0.defined() ? py::cast(dh0) : py::none());
}

// ------------------------------------------------------------------------------------------------ layer prologue, backward
// Normalised q and k (16-bit, as l2norm gives them) for the backward of a forward that folded the norm in.
py::tuple l2norm_pair(const Tensor& q_, const Tensor& k_) {
  py::gil_scoped_release nogil;
  const Tensor q = contiguous(q_), k = contiguous(k_);
  c10::cuda::OptionalCUDAGuard guard(q.device());
  const Tensor qn = at::empty_like(q), kn = at::empty_like(k);
  QlaLayerBwdArgs a{};
  a.rows = q.numel() / 128; a.qkv_dtype = dtype_code(q); a.eps = 1e-6f;
  a.q = ptr(q); a.k = ptr(k); a.qn = ptr(qn); a.kn = ptr(kn);
  check(qla_layer_bwd(&a, current_stream(q.device())), "qla_layer_bwd");
  py::gil_scoped_acquire gil;
  return py::make_tuple(qn, kn);
}

// Chain rule of the prologue: in place on dq / dk (gradients of the normalised rows), and from dg / db (gradients of
// the activated gate and beta) to those of the raw inputs and of A_log / dt_bias.  None where a map was not applied.
py::tuple layer_bwd(const OptTensor& q_, const OptTensor& k_, const OptTensor& dq, const OptTensor& dk, const OptTensor& a_in_,
                    const OptTensor& A_log_, const OptTensor& dt_bias_, const Tensor& dg, const OptTensor& b_in,
                    const OptTensor& beta_act, const Tensor& db) {
  py::gil_scoped_release nogil;
  const at::Device dev = dg.device();
  c10::cuda::OptionalCUDAGuard guard(dev);
  QlaLayerBwdArgs a{};
  a.eps = 1e-6f;
  Tensor q, k, a_in, A_log, dt_bias, da, dA, ddt, dbr, partial;
  if (q_.has_value()) {
    q = contiguous(*q_);
    k = contiguous(*k_);
    a.rows = q.numel() / 128; a.qkv_dtype = dtype_code(q); a.q = ptr(q); a.k = ptr(k); a.dq = ptr(dq); a.dk = ptr(dk);
  }
  const int64_t Hv = dg.size(2);
  a.num_v_heads = Hv;
  a.tokens = dg.size(0) * dg.size(1);
  if (a_in_.has_value()) {
    a_in = contiguous(*a_in_);
    A_log = as(*A_log_, dev, at::kFloat);
    dt_bias = as(*dt_bias_, dev, at::kFloat);
    da = at::empty_like(a_in);
    Tensor sums = new_tensor({2, Hv}, at::kFloat, dev);
    dA = sums.select(0, 0);
    ddt = sums.select(0, 1);
    a.gate_dtype = dtype_code(a_in); a.a = ptr(a_in); a.A_log = ptr<float>(A_log); a.dt_bias = ptr<float>(dt_bias);
    a.dg = ptr<float>(dg); a.da = ptr(da); a.dsums = ptr<float>(sums);
    partial = new_tensor({static_cast<int64_t>(qla_layer_bwd_workspace_bytes(&a))}, at::kByte, dev);
    a.workspace = partial.data_ptr();
  }
  if (b_in.has_value()) {
    dbr = new_tensor(db.sizes(), b_in->scalar_type(), dev);
    a.beta_dtype = dtype_code(dbr); a.beta = ptr<float>(beta_act); a.db = ptr<float>(db); a.db_raw = ptr(dbr);
  }
  check(qla_layer_bwd(&a, current_stream(dev)), "qla_layer_bwd");
  py::gil_scoped_acquire gil;
  auto opt = [](const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); };
  return py::make_tuple(opt(da), opt(dA), opt(ddt), opt(dbr));
}

}  // namespace

PYBIND11_MODULE(_fq_host, m) {
  m.attr("torch_version") = TORCH_VERSION;  // (flashqla_b200._cabi.host compares it with the torch that is running)
  py::class_<Plan>(m, "Plan")
      .def(py::init([](Tensor cu, Tensor seg_next, Tensor seg_raw, Tensor raw_first, Tensor identity, Tensor seg_start_of,
                       Tensor seg_prev, Tensor tables) {
        const int64_t n_seg = seg_next.numel(), n_raw = raw_first.numel() - 1;
        return Plan{cu, seg_next, seg_raw, raw_first, identity, seg_start_of, seg_prev, tables, n_seg, n_raw};
      }));
  m.def("recurrent_update", &recurrent_update);
  m.def("state_commit", &state_commit);
  m.def("chunk_check", &chunk_check_py);
  m.def("chunk_fwd", &chunk_fwd);
  m.def("chunk_bwd", &chunk_bwd);
  m.def("l2norm_pair", &l2norm_pair);
  m.def("layer_bwd", &layer_bwd);
}
