// Host path of the layers in native code: one call per layer that checks the tensors, takes outputs and workspaces from
// PyTorch's allocator and enqueues the layer's kernels through the C ABI (include/b200ta.h).
//
// At small token counts a block's kernels take some 100 us of GPU time, and the same steps written with ctypes and
// torch functions in Python took several times that on the host (about 40 us per launch: argument conversion of 20 to
// 30 values, tensor attributes, empty(), the stream object, a getattr per parameter for the weight check); from here a
// layer call costs its launches and a few microseconds.
//
// The kernels' library is not linked: bind() takes its entry points from the file that the ctypes binding loaded.
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <cstring>
#include <string>

#include "../../include/b200ta.h"

namespace py = pybind11;

namespace {

struct Library {
#define B200TA_ENTRY(name) decltype(&b200ta_##name) name = nullptr;
#define B200TA_ENTRIES(X)                                                                                            \
  X(last_error) X(node_workspace_bytes) X(node_forward) X(transition) X(transition_relu) X(trimul_project)           \
  X(trimul_contract) X(trimul_output) X(trimul_output_f32) X(pair_bias) X(row_stats) X(linear) X(attention)            \
  X(attention_masked) X(prologue) X(epilogue) X(mask_lengths) X(mask_bits)
  B200TA_ENTRIES(B200TA_ENTRY)
#undef B200TA_ENTRY
} lib;

py::object error_type;  // _lib.B200TAError

void bind(const std::string& path, py::object error) {
  void* handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (handle == nullptr) throw py::import_error("cannot open " + path + ": " + dlerror());
#define B200TA_LOAD(name)                                                                                    \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(handle, "b200ta_" #name));                           \
  if (lib.name == nullptr) throw py::import_error("b200ta_" #name " is not exported by " + path);
  B200TA_ENTRIES(B200TA_LOAD)
#undef B200TA_LOAD
  error_type = std::move(error);
}

// Raises what _lib.call raises for a non-zero status.
void check(int code, const char* fn) {
  if (code == B200TA_OK) return;
  const std::string reason = lib.last_error();
  if (code == B200TA_ERR_INVALID) throw py::value_error(std::string(fn) + ": " + reason);
  PyErr_SetObject(error_type.ptr(), error_type(fn, code, reason).ptr());
  throw py::error_already_set();
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

std::string shape_of(const at::Tensor& t) {
  std::string s = "(";
  for (int64_t d : t.sizes()) s += std::to_string(d) + ", ";
  return s + ")";
}

void require_bf16(const char* name, const at::Tensor& t) {
  if (!t.is_cuda()) throw py::value_error(std::string(name) + " must be a CUDA tensor (this package has no CPU path)");
  if (t.scalar_type() != at::kBFloat16) throw py::value_error(std::string(name) + " must be bfloat16");
}

// A pair tensor [B, N, N, 128] as the kernels see it; `swap` exchanges the two pair axes.
struct Pair {
  int B, N;
  int64_t sb, sr, ss;
};
Pair pair_of(const char* name, const at::Tensor& z, bool swap) {
  require_bf16(name, z);
  if (z.dim() != 4 || z.size(1) != z.size(2) || z.size(3) != B200TA_C || z.stride(3) != 1)
    throw py::value_error(std::string(name) + ": expected a square pair tensor [B, N, N, 128] with unit channel stride, got " +
                          shape_of(z));
  return {int(z.size(0)), int(z.size(1)), z.stride(0), z.stride(swap ? 2 : 1), z.stride(swap ? 1 : 2)};
}

at::Tensor new_bf16(const at::Tensor& like, at::IntArrayRef shape) {
  return at::empty(shape, like.options().dtype(at::kBFloat16).memory_format(c10::MemoryFormat::Contiguous));
}

// The buffer kept in `buffers` (a dict or None) under `key`, replaced when it is not a contiguous tensor of this shape, dtype
// and device (callers put their own in as well); a fresh tensor when there is no dict.
at::Tensor buffer(const py::object& buffers, const char* key, at::IntArrayRef shape, at::ScalarType dtype,
                  const at::Tensor& like) {
  if (!buffers.is_none()) {
    if (PyObject* held = PyDict_GetItemString(buffers.ptr(), key); held != nullptr && THPVariable_Check(held)) {
      const at::Tensor& t = THPVariable_Unpack(held);
      if (t.sizes() == shape && t.scalar_type() == dtype && t.device() == like.device() && t.is_contiguous()) return t;
    }
  }
  at::Tensor t = at::empty(shape, like.options().dtype(dtype));
  if (!buffers.is_none()) buffers[key] = py::cast(t);
  return t;
}

struct Lengths {
  const int32_t* ptr = nullptr;
  int64_t sb = 0, sr = 0;
  at::Tensor held;  // as [B, R]; a copy if the values do not lie like that, so held until the launch
};
Lengths lengths_of(const c10::optional<at::Tensor>& lengths, int64_t B, int64_t R) {
  if (!lengths) return {};
  const at::Tensor& t = *lengths;
  if (t.scalar_type() != at::kInt || !t.is_cuda() || t.numel() != B * R)
    throw py::value_error("lengths must be a CUDA int32 tensor with B*N=" + std::to_string(B * R) + " values");
  const at::Tensor v = t.reshape({B, R});
  return {v.data_ptr<int32_t>(), v.stride(0), v.stride(1), v};
}

struct Mask {
  const float* ptr = nullptr;
  int64_t sb = 0, si = 0, sj = 0;
};
Mask mask_of(const c10::optional<at::Tensor>& mask, int64_t B, int64_t N, bool swap) {
  if (!mask) return {};
  const at::Tensor& t = *mask;
  if (t.scalar_type() != at::kFloat || !t.is_cuda() || t.dim() != 3 || t.size(0) != B || t.size(1) != N || t.size(2) != N)
    throw py::value_error("mask must be a CUDA float32 tensor of shape [B, N, N], got " + shape_of(t));
  return {t.data_ptr<float>(), t.stride(0), t.stride(swap ? 2 : 1), t.stride(swap ? 1 : 2)};
}

// ---- layers ------------------------------------------------------------------------------------------------------

at::Tensor node_workspace(const py::object& buffers, const at::Tensor& z) {
  return buffer(buffers, "tri_attn_workspace", {int64_t(lib.node_workspace_bytes(int(z.size(0)), int(z.size(1))))}, at::kByte, z);
}

void node_into(const at::Tensor& z, const at::Tensor& packed, const c10::optional<at::Tensor>& lengths, double eps, bool ending,
               bool residual, const at::Tensor& out, const at::Tensor& ws, int empty_row_mode) {
  const Pair p = pair_of("z", z, ending);
  const Pair o = pair_of("out", out, ending);
  const Lengths l = lengths_of(lengths, p.B, p.N);
  check(lib.node_forward(z.data_ptr(), p.sb, p.sr, p.ss, packed.data_ptr(), float(eps), l.ptr, l.sb, l.sr, empty_row_mode,
                         residual, out.data_ptr(), o.sb, o.sr, o.ss, ws.data_ptr(), size_t(ws.numel()), p.B, p.N, stream()),
        "b200ta_node_forward");
}

at::Tensor node(const at::Tensor& z, const at::Tensor& packed, const c10::optional<at::Tensor>& lengths, double eps,
                bool ending, bool residual, bool inplace, const py::object& buffers, int empty_row_mode) {
  pair_of("z", z, ending);
  const at::Tensor out = inplace ? z : new_bf16(z, z.sizes());
  node_into(z, packed, lengths, eps, ending, residual, out, node_workspace(buffers, z), empty_row_mode);
  return out;
}

// The node with one bit per key beside the row lengths (masks that are not left-aligned), from prologue to epilogue.
at::Tensor node_masked(const at::Tensor& z, const at::Tensor& packed, const at::Tensor& lengths, const at::Tensor& bits,
                       double eps, bool ending, bool residual, bool inplace, const py::object& buffers, int empty_row_mode) {
  const Pair p = pair_of("z", z, ending);
  const int64_t B = p.B, N = p.N, dim = B200TA_HEAD_DIM, heads = B200TA_HEADS, pad = (N + 7) / 8 * 8, words = (N + 31) / 32;
  if (bits.scalar_type() != at::kInt || !bits.is_cuda() || !bits.is_contiguous() || bits.numel() != B * N * words)
    throw py::value_error("key bits must be a contiguous CUDA int32 tensor [B, N, ceil(N / 32)]");
  const at::Tensor out = inplace ? z : new_bf16(z, z.sizes());
  const Pair o = pair_of("out", out, ending);
  const Lengths l = lengths_of(lengths, B, N);
  const at::Tensor bias = buffer(buffers, "tri_attn_bias", {B, heads, N, pad}, at::kBFloat16, z);
  const at::Tensor qkvg = buffer(buffers, "tri_attn_qkvg", {4, B * N, heads, N, dim}, at::kBFloat16, z);
  const at::Tensor og = buffer(buffers, "tri_attn_output", {B * N, N, heads, dim}, at::kBFloat16, z);
  void* s = stream();
  const int64_t head = N * dim, row = heads * head, plane = B * N * row;
  check(lib.prologue(z.data_ptr(), p.sb, p.sr, p.ss, packed.data_ptr(), float(eps), qkvg.data_ptr(), plane, row, head, dim, 1,
                     bias.data_ptr(), heads * N * pad, N * pad, pad, 1, p.B, p.N, p.N, int(pad), s),
        "b200ta_prologue");
  char* q = static_cast<char*>(qkvg.data_ptr());
  check(lib.attention_masked(q, q + 2 * plane, q + 4 * plane, q + 6 * plane, row, head, dim, bias.data_ptr(), heads * N * pad,
                             N * pad, pad, l.ptr, l.sb, l.sr, reinterpret_cast<const uint32_t*>(bits.data_ptr<int32_t>()),
                             N * words, words, og.data_ptr(), N * B200TA_C, B200TA_C, dim, nullptr, 0.17677669529663687f,
                             empty_row_mode, p.B, p.N, p.N, int(pad), s),
        "b200ta_attention_masked");
  check(lib.epilogue(og.data_ptr(), N * N * B200TA_C, N * B200TA_C, B200TA_C, packed.data_ptr(),
                     residual ? z.data_ptr() : nullptr, p.sb, p.sr, p.ss, out.data_ptr(), o.sb, o.sr, o.ss, p.B, p.N, p.N, s),
        "b200ta_epilogue");
  return out;
}

void trimul_into(const at::Tensor& z, const c10::optional<at::Tensor>& mask, const at::Tensor& packed, double eps, bool incoming,
                 const c10::optional<at::Tensor>& b_scale, const at::Tensor& ab, const at::Tensor& x, const at::Tensor& out,
                 bool residual, bool mask_output) {
  const Pair p = pair_of("z", z, false);
  const int64_t pitch = ab.size(3);
  const bool f32 = out.scalar_type() == at::kFloat;
  void* s = stream();
  const Mask m = mask_of(mask, p.B, p.N, incoming);
  check(lib.trimul_project(z.data_ptr(), p.sb, incoming ? p.ss : p.sr, incoming ? p.sr : p.ss, m.ptr, m.sb, m.si, m.sj,
                           b_scale ? b_scale->data_ptr<float>() : nullptr, packed.data_ptr(), float(eps), ab.data_ptr(), pitch,
                           p.B, p.N, p.N, s),
        "b200ta_trimul_project");
  check(lib.trimul_contract(ab.data_ptr(), x.data_ptr(), p.B, p.N, pitch, s), "b200ta_trimul_contract");
  const Mask om = mask_output ? mask_of(mask, p.B, p.N, false) : Mask{};
  check((f32 ? lib.trimul_output_f32 : lib.trimul_output)(z.data_ptr(), p.sb, p.sr, p.ss, x.data_ptr(), pitch, om.ptr, om.sb,
                                                          om.si, om.sj, packed.data_ptr(), float(eps), residual,
                                                          out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), p.B,
                                                          p.N, s),
        "b200ta_trimul_output");
}

struct TrimulBuffers {
  at::Tensor ab, x;
};
TrimulBuffers trimul_buffers(const py::object& buffers, const at::Tensor& z) {
  const int64_t B = z.size(0), N = z.size(1), pitch = (N + 15) / 16 * 16;
  return {buffer(buffers, "trimul_ab", {B, 2 * B200TA_C, N, pitch}, at::kBFloat16, z),
          buffer(buffers, "trimul_contracted", {B, B200TA_C, N, pitch}, at::kBFloat16, z)};
}

at::Tensor trimul(const at::Tensor& z, const c10::optional<at::Tensor>& mask, const at::Tensor& packed, double eps,
                  bool incoming, const c10::optional<at::Tensor>& b_scale, const py::object& buffers, bool residual,
                  bool mask_output, bool f32) {
  pair_of("z", z, false);
  const TrimulBuffers t = trimul_buffers(buffers, z);
  const at::Tensor out = at::empty(z.sizes(), z.options().dtype(f32 ? at::kFloat : at::kBFloat16)
                                                  .memory_format(c10::MemoryFormat::Contiguous));
  trimul_into(z, mask, packed, eps, incoming, b_scale, t.ab, t.x, out, residual, mask_output);
  return out;
}

at::Tensor transition(const at::Tensor& x, const at::Tensor& packed, const c10::optional<at::Tensor>& mask, double eps,
                      bool residual, bool inplace, bool relu) {
  require_bf16("x", x);
  if (x.dim() < 1 || x.size(-1) != B200TA_C) throw py::value_error("last dimension must be 128");
  if (!x.is_contiguous()) throw py::value_error("transition needs a contiguous input");
  const at::Tensor out = inplace ? x : at::empty_like(x);
  const int64_t rows = x.numel() / B200TA_C;
  at::Tensor m;
  if (mask) {
    m = mask->to(at::kBFloat16).expand(x.sizes().slice(0, x.dim() - 1)).contiguous();
    if (!m.is_cuda()) throw py::value_error("mask must be a CUDA tensor");
  }
  check((relu ? lib.transition_relu : lib.transition)(x.data_ptr(), B200TA_C, mask ? m.data_ptr() : nullptr, packed.data_ptr(),
                                                      float(eps), out.data_ptr(), B200TA_C, rows, residual, stream()),
        relu ? "b200ta_transition_relu" : "b200ta_transition");
  return out;
}

// A transition of other widths: (row statistics,) two GEMMs.  w1 / w2 bf16, sc1 / sc2 {rowsum, const} per output column.
at::Tensor transition_gemms(const at::Tensor& x, const at::Tensor& w1, const at::Tensor& sc1, const at::Tensor& w2,
                            const at::Tensor& sc2, bool normalize, double eps, bool residual, bool inplace) {
  require_bf16("x", x);
  if (!x.is_contiguous()) throw py::value_error("transition needs a contiguous input");
  const int64_t K = x.size(-1), rows = x.numel() / K, hidden = w2.size(1);
  if (K != w1.size(1)) throw py::value_error("last dimension must be " + std::to_string(w1.size(1)));
  void* s = stream();
  at::Tensor stats;
  if (normalize) {
    stats = at::empty({rows, 2}, x.options().dtype(at::kFloat));
    check(lib.row_stats(x.data_ptr(), K, rows, int(K), float(eps), stats.data_ptr(), s), "b200ta_row_stats");
  }
  const at::Tensor h = new_bf16(x, {rows, hidden});
  check(lib.linear(x.data_ptr(), rows * K, K, 128, w1.data_ptr(), sc1.data_ptr(), normalize ? stats.data_ptr() : nullptr,
                   nullptr, 0, h.data_ptr(), hidden, 0, 2, 1, int(rows), int(K), int(2 * hidden), s),
        "b200ta_linear");
  const at::Tensor out = inplace ? x : at::empty_like(x);
  check(lib.linear(h.data_ptr(), rows * hidden, hidden, 128, w2.data_ptr(), sc2.data_ptr(), nullptr,
                   residual ? x.data_ptr() : nullptr, residual ? K : 0, out.data_ptr(), K, 0, 1, 1, int(rows), int(hidden),
                   int(K), s),
        "b200ta_linear");
  return out;
}

// bias[b, h, q, k] of the single-track attention, [B, 16, N, ceil8(N)], kept in `buffers` under `key`.
at::Tensor pair_bias(const at::Tensor& z, const at::Tensor& packed_z, double eps_z, const py::object& buffers,
                     const char* key) {
  const Pair p = pair_of("z", z, false);
  const int64_t heads = 16, pad = (p.N + 7) / 8 * 8;
  const at::Tensor bias = buffer(buffers, key, {p.B, heads, p.N, pad}, at::kBFloat16, z);
  check(lib.pair_bias(z.data_ptr(), p.sb, p.sr, p.ss, packed_z.data_ptr(), float(eps_z), bias.data_ptr(), bias.stride(0),
                      bias.stride(1), bias.stride(2), 1, int(heads), p.B, p.N, p.N, int(pad), stream()),
        "b200ta_pair_bias");
  return bias;
}

// `s` has to have the width that the in-projection's weights were folded for, and a residual the shape of `s`: the kernels
// take both as given.
void check_single(const at::Tensor& s, int64_t B, int64_t N, const at::Tensor& w_in) {
  require_bf16("s", s);
  if (!s.is_contiguous() || s.dim() != 3 || s.size(0) != B || s.size(1) != N || s.size(2) != w_in.size(1))
    throw py::value_error("s must be a contiguous [" + std::to_string(B) + ", " + std::to_string(N) + ", " +
                          std::to_string(w_in.size(1)) + "] tensor that matches z and the weights, got " + shape_of(s));
}

// The single-track attention with the bias that pair_bias() wrote.  `lengths` int32 [4 B]: the key count of a batch entry
// four times (the attention kernel sees its 16 heads as four items of four).
at::Tensor pair_bias_attention(const at::Tensor& s16, const at::Tensor& bias, const c10::optional<at::Tensor>& lengths,
                               const at::Tensor& w_in, const at::Tensor& sc_in, const at::Tensor& w_o, const at::Tensor& sc_o,
                               bool normalize, double eps_s, double scale, const c10::optional<at::Tensor>& residual,
                               const py::object& buffers) {
  const int64_t B = bias.size(0), N = bias.size(2), heads = 16, dim = B200TA_HEAD_DIM, pad = bias.size(3);
  check_single(s16, B, N, w_in);
  const int64_t c_s = s16.size(2);
  if (residual) {
    require_bf16("residual", *residual);
    if (!residual->is_contiguous() || residual->sizes() != s16.sizes())
      throw py::value_error("residual must be a contiguous tensor of the shape of s, got " + shape_of(*residual));
  }
  void* st = stream();
  at::Tensor stats;
  if (normalize) {
    stats = at::empty({B * N, 2}, s16.options().dtype(at::kFloat));
    check(lib.row_stats(s16.data_ptr(), c_s, B * N, int(c_s), float(eps_s), stats.data_ptr(), st), "b200ta_row_stats");
  }
  const at::Tensor planes = buffer(buffers, "pw_qkvg", {4, B, heads, N, dim}, at::kBFloat16, s16);
  check(lib.linear(s16.data_ptr(), N * c_s, c_s, 128, w_in.data_ptr(), sc_in.data_ptr(), normalize ? stats.data_ptr() : nullptr,
                   nullptr, 0, planes.data_ptr(), 0, planes.stride(0), 0, int(B), int(N), int(c_s), int(4 * heads * dim), st),
        "b200ta_linear");
  const at::Tensor attn = buffer(buffers, "pw_attn_output", {4 * B, 1, N, B200TA_C}, at::kBFloat16, s16);
  const Lengths l = lengths_of(lengths, 4 * B, 1);
  char* q = static_cast<char*>(planes.data_ptr());
  const int64_t plane = planes.stride(0) * 2, head = N * dim;
  check(lib.attention(q, q + plane, q + 2 * plane, q + 3 * plane, 4 * head, head, dim, bias.data_ptr(), 4 * N * pad, N * pad,
                      pad, l.ptr, l.sb, l.sr, attn.data_ptr(), N * B200TA_C, B200TA_C, dim, nullptr, float(scale),
                      B200TA_EMPTY_ROW_UNIFORM, int(4 * B), 1, int(N), int(pad), st),
        "b200ta_attention");
  const at::Tensor out = at::empty_like(s16);
  check(lib.linear(attn.data_ptr(), 4 * N * B200TA_C, B200TA_C, N * B200TA_C, w_o.data_ptr(), sc_o.data_ptr(), nullptr,
                   residual ? residual->data_ptr() : nullptr, residual ? c_s : 0, out.data_ptr(), c_s, 0, 1, int(B), int(N),
                   int(heads * dim), int(c_s), st),
        "b200ta_linear");
  return out;
}

// ---- a second stream for the single track -------------------------------------------------------------------------

// In a block the single track needs the pair tensor's bias, but nothing of the next block's pair track needs the single
// track: a stack enqueues it on a stream of its own.  Its kernels have one row per token (a few to 144 blocks, 2-13 us
// each, bound by latency), and run beside the pair track's instead of between them.
// The stream is of high priority, so that the few blocks start at the next kernel boundary of the pair track.
class SideTrack {
 public:
  SideTrack() : side_(c10::cuda::getStreamFromPool(/*isHighPriority=*/true)), main_(c10::cuda::getCurrentCUDAStream()) {
    for (cudaEvent_t* e : {&ready_, &done_[0], &done_[1]}) cuda(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  SideTrack(const SideTrack&) = delete;
  ~SideTrack() {
    for (cudaEvent_t e : {ready_, done_[0], done_[1]}) cudaEventDestroy(e);
  }
  // `slot` (0 or 1): what the side stream has been given so far is the last use of the slot's bias buffer ...
  void done(int slot) { cuda(cudaEventRecord(done_[slot & 1], side_.stream())); }
  // ... which the main stream may overwrite after this.
  void wait(int slot) { cuda(cudaStreamWaitEvent(main_.stream(), done_[slot & 1], 0)); }
  // `result` was allocated on the side stream and goes to a user of the main stream.
  void hand_over(const at::Tensor& result) {
    c10::cuda::CUDACachingAllocator::recordStream(result.storage().data_ptr(), main_);
  }

  // The side stream is the current one while this lives.
  class Inside {
   public:
    explicit Inside(SideTrack& track) : main_(track.main_) { c10::cuda::setCurrentCUDAStream(track.side_); }
    Inside(const Inside&) = delete;
    ~Inside() { c10::cuda::setCurrentCUDAStream(main_); }

   private:
    c10::cuda::CUDAStream main_;
  };

  // A call's use of the side stream, which the main stream joins on every way out of the call: what was enqueued there
  // works on tensors of the main stream's pool, which the end of the call, or an exception, hands back.
  class Use {
   public:
    explicit Use(SideTrack* track) : track_(track) {}
    Use(const Use&) = delete;
    ~Use() {
      if (forked_ && cudaEventRecord(track_->ready_, track_->side_.stream()) == cudaSuccess)
        cudaStreamWaitEvent(track_->main_.stream(), track_->ready_, 0);
    }
    // The side stream continues from what the main stream has been given so far.
    void fork() {
      forked_ = true;
      cuda(cudaEventRecord(track_->ready_, track_->main_.stream()));
      cuda(cudaStreamWaitEvent(track_->side_.stream(), track_->ready_, 0));
    }
    void join() {
      cuda(cudaEventRecord(track_->ready_, track_->side_.stream()));
      cuda(cudaStreamWaitEvent(track_->main_.stream(), track_->ready_, 0));
      forked_ = false;
    }

   private:
    SideTrack* track_;
    bool forked_ = false;
  };

 private:
  static void cuda(cudaError_t e) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA: ") + cudaGetErrorString(e));
  }
  c10::cuda::CUDAStream side_, main_;
  cudaEvent_t ready_ = nullptr, done_[2] = {nullptr, nullptr};
};

// ---- a whole stack ---------------------------------------------------------------------------------------------------

// The blocks of a pairformer stack with their packed weights, enqueued by one call: the Python of seven layers per block
// took some 100 us of host time, as much as a block's kernels need at 120 tokens.  The pair tensor alternates between two
// buffers (the attention nodes and the transition work in place); the single track runs on the side stream.
class Stack {
 public:
  struct Weights {
    at::Tensor packed;
    double eps;
  };
  struct Node {
    at::Tensor packed;
    double eps;
    int empty_row_mode;
  };
  struct Single {
    at::Tensor w_in, sc_in, w_o, sc_o, packed_z, w1, sc1, w2, sc2;
    bool norm, norm_t;
    double eps, eps_z, scale, eps_t;
  };
  void add(const at::Tensor& tri_out, double eps_out, const at::Tensor& tri_in, double eps_in, const at::Tensor& start,
           double eps_start, int mode_start, const at::Tensor& end, double eps_end, int mode_end, const at::Tensor& transition,
           double eps_transition) {
    blocks_.push_back({{tri_out, eps_out}, {tri_in, eps_in}, {start, eps_start, mode_start}, {end, eps_end, mode_end},
                       {transition, eps_transition}});
  }
  void add_single(const at::Tensor& w_in, const at::Tensor& sc_in, const at::Tensor& w_o, const at::Tensor& sc_o,
                  const at::Tensor& packed_z, bool norm, double eps, double eps_z, double scale, const at::Tensor& w1,
                  const at::Tensor& sc1, const at::Tensor& w2, const at::Tensor& sc2, bool norm_t, double eps_t) {
    singles_.push_back({w_in, sc_in, w_o, sc_o, packed_z, w1, sc1, w2, sc2, norm, norm_t, eps, eps_z, scale, eps_t});
  }

  // z bf16 [B, N, N, 128] (left as it is), mask fp32 [B, N, N] or None, row lengths of the mask and of its transpose.
  at::Tensor run_pair(const at::Tensor& z, const c10::optional<at::Tensor>& mask, const c10::optional<at::Tensor>& lengths,
                      const c10::optional<at::Tensor>& lengths_t, bool mask_output, const py::object& buffers) {
    return run(c10::nullopt, z, mask, lengths, lengths_t, mask_output, c10::nullopt, buffers, nullptr).second;
  }
  std::pair<at::Tensor, at::Tensor> run_both(const at::Tensor& s, const at::Tensor& z, const c10::optional<at::Tensor>& mask,
                                             const c10::optional<at::Tensor>& lengths,
                                             const c10::optional<at::Tensor>& lengths_t, bool mask_output,
                                             const at::Tensor& key_counts, const py::object& buffers, SideTrack& track) {
    return run(s, z, mask, lengths, lengths_t, mask_output, key_counts, buffers, &track);
  }

 private:
  struct Block {
    Weights tri_out, tri_in;
    Node start, end;
    Weights transition;
  };
  std::pair<at::Tensor, at::Tensor> run(c10::optional<at::Tensor> s, at::Tensor z, const c10::optional<at::Tensor>& mask,
                                        const c10::optional<at::Tensor>& lengths, const c10::optional<at::Tensor>& lengths_t,
                                        bool mask_output, const c10::optional<at::Tensor>& key_counts,
                                        const py::object& given_buffers, SideTrack* track) {
    pair_of("z", z, false);
    if (s && singles_.size() != blocks_.size()) throw py::value_error("every block needs the weights of its single track");
    if (s && !singles_.empty()) check_single(*s, z.size(0), z.size(1), singles_[0].w_in);  // before anything is enqueued
    const py::object buffers = given_buffers.is_none() ? py::object(py::dict()) : given_buffers;  // held until the join
    const at::Tensor ws = node_workspace(buffers, z);
    const TrimulBuffers t = trimul_buffers(buffers, z);
    const at::Tensor a = new_bf16(z, z.sizes()), out = new_bf16(z, z.sizes());
    at::Tensor s16;
    if (s) {
      s16 = *s;
      const int64_t B = z.size(0), N = z.size(1);
      // used on the side stream, but allocated on the caller's, which has joined it when they are freed
      buffer(buffers, "pw_qkvg", {4, B, 16, N, B200TA_HEAD_DIM}, at::kBFloat16, z);
      buffer(buffers, "pw_attn_output", {4 * B, 1, N, B200TA_C}, at::kBFloat16, z);
    }
    SideTrack::Use use(track);  // after the tensors, so that it ends before them
    for (size_t i = 0; i < blocks_.size(); ++i) {
      const Block& b = blocks_[i];
      trimul_into(z, mask, b.tri_out.packed, b.tri_out.eps, false, c10::nullopt, t.ab, t.x, a, true, mask_output);
      trimul_into(a, mask, b.tri_in.packed, b.tri_in.eps, true, c10::nullopt, t.ab, t.x, out, true, mask_output);
      z = out;
      node_into(z, b.start.packed, lengths, b.start.eps, false, true, z, ws, b.start.empty_row_mode);
      node_into(z, b.end.packed, lengths_t, b.end.eps, true, true, z, ws, b.end.empty_row_mode);
      transition(z, b.transition.packed, c10::nullopt, b.transition.eps, true, true, false);
      if (!s) continue;
      const Single& w = singles_[i];
      if (i >= 2) track->wait(int(i));
      const at::Tensor bias = pair_bias(z, w.packed_z, w.eps_z, buffers, (i & 1) ? "pw_pair_bias_1" : "pw_pair_bias_0");
      use.fork();
      const SideTrack::Inside inside(*track);
      s16 = pair_bias_attention(s16, bias, key_counts, w.w_in, w.sc_in, w.w_o, w.sc_o, w.norm, w.eps, w.scale, s16, buffers);
      transition_gemms(s16, w.w1, w.sc1, w.w2, w.sc2, w.norm_t, w.eps_t, true, true);
      track->done(int(i));
    }
    if (s) {
      use.join();
      track->hand_over(s16);
    }
    return {s16, z};
  }
  std::vector<Block> blocks_;
  std::vector<Single> singles_;
};

int64_t current_stream() { return reinterpret_cast<int64_t>(stream()); }

// ---- masks -----------------------------------------------------------------------------------------------------------

at::Tensor new_int32(const at::Tensor& like, at::IntArrayRef shape) { return at::empty(shape, like.options().dtype(at::kInt)); }

// Masks are reduced on their own device, which need not be the current one (they may be made before a model's device is
// entered).
// Keys with mask > 0.5 per row of a float [B, I, J] mask and per row of its transpose.
std::pair<at::Tensor, at::Tensor> mask_lengths(const at::Tensor& mask) {
  const c10::cuda::CUDAGuard guard(mask.device());
  const int B = int(mask.size(0)), I = int(mask.size(1)), J = int(mask.size(2));
  const at::Tensor rows = new_int32(mask, {B, I}), cols = new_int32(mask, {B, J});
  check(lib.mask_lengths(mask.data_ptr<float>(), mask.stride(0), mask.stride(1), mask.stride(2), rows.data_ptr<int32_t>(),
                         cols.data_ptr<int32_t>(), B, I, J, stream()),
        "b200ta_mask_lengths");
  return {rows, cols};
}

// Row lengths (last valid key + 1) and key bits of a float [B, R, S] mask; valid: > 0.5, or >= 0 in the additive form.
std::pair<at::Tensor, at::Tensor> mask_bits(const at::Tensor& mask, bool additive) {
  const c10::cuda::CUDAGuard guard(mask.device());
  const int B = int(mask.size(0)), R = int(mask.size(1)), S = int(mask.size(2));
  const at::Tensor lengths = new_int32(mask, {B, R}), bits = new_int32(mask, {B, R, (S + 31) / 32});
  check(lib.mask_bits(mask.data_ptr<float>(), mask.stride(0), mask.stride(1), mask.stride(2), additive,
                      lengths.data_ptr<int32_t>(), reinterpret_cast<uint32_t*>(bits.data_ptr<int32_t>()), B, R, S, stream()),
        "b200ta_mask_bits");
  return {lengths, bits};
}

// ---- state of modules ------------------------------------------------------------------------------------------------

// What a visit of modules looks at, in an order that depends on the modules alone.  A visitor has object(PyObject*) and
// tensor(const at::Tensor&), which return false to end the visit.
struct Names {
  PyObject* const parameters = PyUnicode_InternFromString("_parameters");
  PyObject* const buffers = PyUnicode_InternFromString("_buffers");
  PyObject* const weight = PyUnicode_InternFromString("weight");
  PyObject* const bias = PyUnicode_InternFromString("bias");
  PyObject* const modules = PyUnicode_InternFromString("_modules");
  PyObject* const hooks = PyUnicode_InternFromString("_forward_hooks");
  PyObject* const pre_hooks = PyUnicode_InternFromString("_forward_pre_hooks");
  PyObject* const compiled = PyUnicode_InternFromString("_compiled_call_impl");
};
const Names& names() {
  static const Names n;
  return n;
}

template <typename Visitor>
bool visit_tensors(PyObject* tensors, Visitor& v) {
  PyObject *key, *value;
  Py_ssize_t pos = 0;
  if (tensors != nullptr && PyDict_Check(tensors))
    while (PyDict_Next(tensors, &pos, &key, &value))
      if (THPVariable_Check(value) && !v.tensor(THPVariable_Unpack(value))) return false;
  return true;
}

// The tensors that a layer's weights are made from, in the module with this dict: its parameters and buffers, and a weight or
// bias that is a plain attribute (replicas of a module and pruned or re-parameterised ones have such).
template <typename Visitor>
bool visit_own_weights(PyObject* dict, Visitor& v) {
  const Names& n = names();
  if (!visit_tensors(PyDict_GetItemWithError(dict, n.parameters), v) || !visit_tensors(PyDict_GetItemWithError(dict, n.buffers), v)) return false;
  for (PyObject* k : {n.weight, n.bias})
    if (PyObject* t = PyDict_GetItemWithError(dict, k); t != nullptr && THPVariable_Check(t) && !v.tensor(THPVariable_Unpack(t))) return false;
  return true;
}

// The weights of `module` and of every module under it.
template <typename Visitor>
bool visit_weights(PyObject* module, Visitor& v) {
  PyObject** dict = _PyObject_GetDictPtr(module);
  if (dict == nullptr || *dict == nullptr) return true;
  if (!visit_own_weights(*dict, v)) return false;
  PyObject *key, *value;
  Py_ssize_t pos = 0;
  if (PyObject* modules = PyDict_GetItemWithError(*dict, names().modules); modules != nullptr && PyDict_Check(modules))
    while (PyDict_Next(modules, &pos, &key, &value))
      if (value != Py_None && !visit_weights(value, v)) return false;
  return true;
}

// `module`, the names and values of its attributes (options, packed weights, ...), its forward hooks and its weights, and
// the same of every module under it.
template <typename Visitor>
bool visit_all(PyObject* module, Visitor& v) {
  if (!v.object(module)) return false;
  PyObject** dict = _PyObject_GetDictPtr(module);
  if (dict == nullptr || *dict == nullptr) return true;
  const Names& n = names();
  PyObject *modules = nullptr, *hooks[2] = {nullptr, nullptr}, *key, *value;
  Py_ssize_t pos = 0;
  while (PyDict_Next(*dict, &pos, &key, &value)) {
    if (!v.object(key) || !v.object(value)) return false;
    if (key == n.modules) modules = value;
    if (key == n.hooks) hooks[0] = value;
    if (key == n.pre_hooks) hooks[1] = value;
  }
  for (PyObject* h : hooks) {
    pos = 0;
    if (h != nullptr && PyDict_Check(h))
      while (PyDict_Next(h, &pos, &key, &value))
        if (!v.object(value)) return false;
  }
  if (!visit_own_weights(*dict, v)) return false;
  pos = 0;
  if (modules != nullptr && PyDict_Check(modules))
    while (PyDict_Next(modules, &pos, &key, &value))
      if (value != Py_None && !visit_all(value, v)) return false;
  return true;
}

// Weights as they were seen: storage, address, in-place write count, device.  The storages are held weakly: their
// memory is free to go, but another storage cannot come to be at the address of one that was seen, so that a weight
// replaced twice does not look unchanged when its memory is given out again.  Not copied or pickled with the layers that
// keep one.
class WeightState {
 public:
  void add(const at::Tensor& t) { seen_.push_back({t.storage().getWeakStorageImpl(), t.data_ptr(), version(t), t.device()}); }
  bool same(size_t i, const at::Tensor& t) const {
    return i < seen_.size() && seen_[i].storage._unsafe_get_target() == t.storage().unsafeGetStorageImpl() &&
           seen_[i].data == t.data_ptr() && seen_[i].version == version(t) && seen_[i].device == t.device();
  }
  size_t size() const { return seen_.size(); }

 private:
  struct Seen {
    c10::weak_intrusive_ptr<c10::StorageImpl> storage;
    const void* data;
    int64_t version;
    c10::Device device;
  };
  static int64_t version(const at::Tensor& t) { return t.is_inference() ? -1 : int64_t(t._version()); }  // inference tensors have none
  std::vector<Seen> seen_;
};

struct RecordAll {
  WeightState weights;
  std::vector<PyObject*> objects;
  bool object(PyObject* o) { return objects.push_back(o), true; }
  bool tensor(const at::Tensor& t) { return weights.add(t), true; }
};
struct CompareAll {
  const WeightState* weights;
  PyObject* const* objects = nullptr;
  size_t num_objects = 0, i = 0, k = 0;
  bool object(PyObject* o) { return i < num_objects && objects[i++] == o; }
  bool tensor(const at::Tensor& t) { return weights->same(k++, t); }
  bool complete() const { return i == num_objects && k == weights->size(); }
};

// The weights under the modules, and whether they are still what `state` (None: nothing) saw: loading, editing or replacing
// one changes that.
WeightState weight_state(const py::args& modules) {
  RecordAll r;
  for (const py::handle& m : modules) visit_weights(m.ptr(), r);
  return std::move(r.weights);
}
bool same_weights(const WeightState* state, const py::args& modules) {
  if (state == nullptr) return false;
  CompareAll c{state};
  for (const py::handle& m : modules)
    if (!visit_weights(m.ptr(), c)) return false;
  return c.complete();
}

// All that visit_all() sees of `module`: the objects in a tuple, which holds them (an object in it cannot make room for
// another one at its address), and the weights.
std::pair<py::tuple, WeightState> module_state(const py::handle& module) {
  RecordAll r;
  visit_all(module.ptr(), r);
  py::tuple objects(r.objects.size());
  for (size_t i = 0; i < r.objects.size(); ++i) {
    Py_INCREF(r.objects[i]);
    PyTuple_SET_ITEM(objects.ptr(), i, r.objects[i]);
  }
  return {std::move(objects), std::move(r.weights)};
}
bool same_state(const py::tuple& objects, const WeightState& weights, const py::handle& module) {
  CompareAll c{&weights, PySequence_Fast_ITEMS(objects.ptr()), objects.size()};
  return visit_all(module.ptr(), c) && c.complete();
}

// Whether a call of `module`, or of a module under it, may do something else than its class's forward: it is hooked or
// compiled, or one of the class's functions is replaced in the instance.
bool more_than_its_class(PyObject* module) {
  PyObject** dict = _PyObject_GetDictPtr(module);
  if (dict == nullptr || *dict == nullptr) return true;
  const Names& n = names();
  PyObject *modules = nullptr, *key, *value;
  Py_ssize_t pos = 0;
  while (PyDict_Next(*dict, &pos, &key, &value)) {
    if (key == n.modules) modules = value;
    if ((key == n.hooks || key == n.pre_hooks) && PyDict_Check(value) && PyDict_Size(value) > 0) return true;
    if (key == n.compiled && value != Py_None) return true;
    if (!PyCallable_Check(value)) continue;
    PyObject* of_class = PyObject_GetAttr(reinterpret_cast<PyObject*>(Py_TYPE(module)), key);
    const bool replaced = of_class != nullptr && PyCallable_Check(of_class);
    Py_XDECREF(of_class);
    PyErr_Clear();
    if (replaced) return true;
  }
  pos = 0;
  if (modules != nullptr && PyDict_Check(modules))
    while (PyDict_Next(modules, &pos, &key, &value))
      if (value != Py_None && more_than_its_class(value)) return true;
  return false;
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.doc() = "Native host path of the layers (see csrc/torch_host.cpp).";
  m.def("bind", &bind);
  m.def("node", &node);
  m.def("node_masked", &node_masked);
  m.def("trimul", &trimul);
  m.def("transition", &transition);
  m.def("transition_gemms", &transition_gemms);
  m.def("pair_bias", &pair_bias);
  m.def("pair_bias_attention", &pair_bias_attention);
  m.def("current_stream", &current_stream);
  py::class_<SideTrack>(m, "SideTrack").def(py::init<>());
  py::class_<Stack>(m, "Stack")
      .def(py::init<>())
      .def("add", &Stack::add)
      .def("add_single", &Stack::add_single)
      .def("run_pair", &Stack::run_pair)
      .def("run_both", &Stack::run_both);
  m.def("more_than_its_class", [](const py::handle& module) { return more_than_its_class(module.ptr()); });
  m.def("module_state", &module_state);
  m.def("same_state", &same_state);
  m.def("mask_lengths", &mask_lengths);
  m.def("mask_bits", &mask_bits);
  py::class_<WeightState>(m, "WeightState")
      .def("__deepcopy__", [](const WeightState&, const py::object&) { return py::none(); })
      .def("__reduce__", [](const WeightState&) { return py::make_tuple(py::type::of(py::none()), py::tuple()); });
  m.def("same_weights", &same_weights);
  m.def("weight_state", &weight_state);
}
