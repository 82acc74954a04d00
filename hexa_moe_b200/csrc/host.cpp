// Native side of the operator wrappers in ops.py: output and scratch allocation, pointer / stride / dtype plumbing, the
// current stream, error translation - everything between a Python call and the C ABI of include/hexa_moe_b200.h.
//
// Why: a layer step is ~20 launches of a few microseconds each at small sizes, and a wrapper that collects two dozen
// pointers, strides and sizes in Python and hands them to ctypes cost ~20 us per operator.  Here it is one call:
// 16 tokens forward 370 -> 204 us, the README layer's step 941 -> 593 us, 4608 tokens x 32 experts 1037 -> 709 us when it came
// (82, 279 and 574 us with fewer launches, the nodes below and early starts since).
// The C ABI is bound at run time from the library that _lib.py has loaded (bind()), so this module links against torch only.
// The interpreter lock is released around every library call: a launch can block on a full queue, and the thread that
// would resolve the stall may need the lock.
//
// The second half of the file is the training layer itself: the autograd nodes of the gate projection, of softmax + top-k + loss
// and of the MoE layer on one GPU.  A node's forward and backward are one call each into the functions above, the backward
// without the interpreter (the engine's thread takes its lock once, to set config.stage).
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <stdlib.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/hexa_moe_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

struct Api {
#define HEXA_API(X)                                                                                                            \
  X(hexa_last_error_string) X(hexa_pending_device_status) X(hexa_route_row_capacity) X(hexa_route_workspace_bytes)             \
  X(hexa_route_pair_capacity) X(hexa_route) X(hexa_gather_rows) X(hexa_gather_rows_ess)                 \
  X(hexa_combine_rows) X(hexa_esmm_experts) X(hexa_esmm_f32_workspace_bytes) X(hexa_esmm_f32) X(hexa_esmm_ess) X(hexa_estmm_workspace_bytes) X(hexa_estmm)                       \
  X(hexa_ess_workspace_bytes) X(hexa_ess) X(hexa_gate_workspace_bytes) X(hexa_gate_topk) X(hexa_gate_loss_grad)                \
  X(hexa_gate_split_terms) X(hexa_gate_sum_terms) X(hexa_ids_from_lists) X(hexa_ids_from_lists_i64)                          \
  X(hexa_gate_project) X(hexa_gate_project_grad)
#define HEXA_FIELD(name) decltype(&::name) name = nullptr;
  HEXA_API(HEXA_FIELD)
} api;

struct Bound {      // what _lib.py hands over; lives as long as the process (nothing to release after the interpreter)
  py::object error, ensure_status_word, status_text;
};
Bound* bound = nullptr;
bool status_installed[64] = {false};

// (may run on the autograd engine's thread, which holds no lock)
[[noreturn]] void fail(const std::string& message) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(bound->error.ptr(), message.c_str());
  throw py::error_already_set();
}

// Raise on a non-zero return code, and on a code that a kernel launched earlier left in the device's status word.
void check(int rc, const char* what) {
  if (rc != 0) fail(std::string(what) + " failed (" + std::to_string(rc) + "): " + api.hexa_last_error_string());
  const int code = api.hexa_pending_device_status();
  if (code != 0) {
    py::gil_scoped_acquire gil;
    fail(std::string(what) + ": " + bound->status_text(code).cast<std::string>());
  }
}

// Lets other Python threads run while it lives, on a thread that holds the interpreter's lock; elsewhere it does nothing.
struct Unlocked {
  std::optional<py::gil_scoped_release> release;
  Unlocked() {
    if (PyGILState_Check()) release.emplace();
  }
};

template <typename F> void call(const char* what, F&& f) {
  int rc;
  {
    Unlocked unlocked;
    rc = f();
  }
  check(rc, what);
}

void* stream_of(const Tensor& t) {
  if (!t.is_cuda()) fail("hexa_moe_b200 operators run on CUDA tensors only (no CPU path)");
  const int dev = t.get_device();
  if (dev < 0 || dev >= 64 || !status_installed[dev]) {
    py::gil_scoped_acquire gil;
    bound->ensure_status_word(dev);
    if (dev >= 0 && dev < 64) status_installed[dev] = true;
  }
  return c10::cuda::getCurrentCUDAStream(dev).stream();
}

// Kernels take raw pointers: an operand on another device, or on the host, has to be refused here.
void same_device(const Tensor& anchor, const Tensor& t) {
  if (t.device() != anchor.device()) fail("operands are on different devices: " + anchor.device().str() + " and " + t.device().str());
}
void same_device(const Tensor& anchor, const OptTensor& t) {
  if (t) same_device(anchor, *t);
}
template <typename... Ts> void on_device_of(const Tensor& anchor, const Ts&... others) { (same_device(anchor, others), ...); }

int dt(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return HEXA_F32;
    case at::kHalf: return HEXA_F16;
    case at::kBFloat16: return HEXA_BF16;
    default: fail(std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
  }
}

// A bias or sum operand is fp32 or of the data's own 16-bit type, which a flag on the dtype says.
bool same16(const Tensor& t, const Tensor& data) { return t.scalar_type() == data.scalar_type() && data.scalar_type() != at::kFloat; }

int64_t ld(const Tensor& t) {
  if (t.dim() != 2 || t.stride(1) != 1) fail("expected a 2-D tensor with unit inner stride");
  return t.stride(0);
}

void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
const int32_t* i32(const Tensor& t) { return static_cast<const int32_t*>(t.data_ptr()); }
const int32_t* i32(const OptTensor& t) { return t.has_value() ? i32(*t) : nullptr; }

Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device()));
}
Tensor scratch(size_t bytes, const Tensor& like) { return empty({(int64_t)(bytes < 4 ? 4 : bytes)}, at::kByte, like); }
// Scratch that an operator can do without: none when the device has not that much left.
OptTensor scratch_if_free(size_t bytes, const Tensor& like) {
  try {
    return scratch(bytes, like);
  } catch (const c10::OutOfMemoryError&) {
    return std::nullopt;
  }
}

// [rows, cols] whose row pitch is a multiple of 8 elements (16 bytes of 16-bit data), as the TMA-fed GEMMs need
Tensor sorted_buffer(int64_t rows, int64_t cols, at::ScalarType type, const Tensor& like) {
  const int64_t pitch = (cols + 7) / 8 * 8;
  Tensor t = empty({rows, pitch}, type, like);
  return pitch == cols ? t : t.narrow(1, 0, cols);
}

// (counts, seg_offsets, pad_offsets, row_token, token_row, tile_expert, pair_block | None, T, k, row_capacity)
py::tuple route(const Tensor& ids, int E, int align, bool route_major) {
  if (ids.scalar_type() != at::kInt) fail("route: ids must be int32");
  if (ids.dim() != 2) fail("route: ids must be 2-D");
  const int dt_ = route_major ? 1 : 0;
  const int64_t T = ids.size(dt_), k = ids.size(1 - dt_), st = ids.stride(dt_), sk = ids.stride(1 - dt_);
  void* s = stream_of(ids);
  const int64_t cap = api.hexa_route_row_capacity(T, (int)k, E, align);
  if (cap < 0) fail("route: bad sizes");
  auto ints = [&](int64_t n) { return empty({n < 1 ? 1 : n}, at::kInt, ids); };
  OptTensor pairs;
  if (align == 128) pairs = ints(api.hexa_route_pair_capacity(T, (int)k, E));
  Tensor counts = ints(E), seg = ints(E + 1), pad = ints(E + 1), row_token = ints(cap), token_row = ints(T * k), tiles = ints(cap / align);
  Tensor ws = scratch(api.hexa_route_workspace_bytes(T, (int)k, E), ids);
  auto out = [](const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); };
  call("hexa_route", [&] {
    return api.hexa_route(i32(ids), T, (int)k, st, sk, E, align, out(counts), out(seg), out(pad), out(row_token), out(token_row),
                          out(tiles), pairs ? out(*pairs) : nullptr, ptr(ws), (size_t)ws.numel(), s);
  });
  return py::make_tuple(counts, seg, pad, row_token, token_row, tiles, pairs, T, k, cap);
}

Tensor ids_from_lists(int64_t num_toks, const Tensor& tok_ids_, const Tensor& exp_ids_, int chunk) {
  void* s = stream_of(tok_ids_);
  on_device_of(tok_ids_, exp_ids_);
  const bool narrow = tok_ids_.scalar_type() == at::kInt;      // anything else is read as 64 bits: an id must not wrap
  const Tensor tok_ids = tok_ids_.to(narrow ? at::kInt : at::kLong).contiguous(), exp_ids = exp_ids_.to(at::kInt).contiguous();
  if (chunk < 1 || tok_ids.numel() > (int64_t)chunk * exp_ids.numel()) fail("ids_from_lists: more token ids than the expert ids cover");
  Tensor ids = empty({num_toks}, at::kInt, tok_ids);
  call("hexa_ids_from_lists", [&] {
    return narrow ? api.hexa_ids_from_lists(i32(tok_ids), i32(exp_ids), tok_ids.numel(), chunk, num_toks, static_cast<int32_t*>(ptr(ids)), s)
                  : api.hexa_ids_from_lists_i64(static_cast<const int64_t*>(ptr(tok_ids)), i32(exp_ids), tok_ids.numel(), chunk, num_toks,
                                                static_cast<int32_t*>(ptr(ids)), s);
  });
  return ids;
}

Tensor gather_at(const Tensor& src, const int32_t* row_token, const int32_t* pad_offsets, int E, int64_t cap, const OptTensor& out_) {
  const int64_t cols = src.size(1);
  void* s = stream_of(src);
  on_device_of(src, out_);
  Tensor out = out_ ? *out_ : sorted_buffer(cap, cols, src.scalar_type(), src);
  const int type = dt(src);
  const int64_t lds = ld(src), ldo = ld(out);
  call("hexa_gather_rows", [&] { return api.hexa_gather_rows(ptr(src), lds, row_token, pad_offsets, E, cap, cols, ptr(out), ldo, type, s); });
  return out;
}
Tensor gather_rows(const Tensor& src, const Tensor& row_token, const Tensor& pad_offsets, int E, int64_t cap, const OptTensor& out_) {
  stream_of(src);
  on_device_of(src, row_token, pad_offsets);
  return gather_at(src, i32(row_token), i32(pad_offsets), E, cap, out_);
}

std::tuple<Tensor, Tensor> gather_ess_at(const Tensor& src, const int32_t* row_token, const int32_t* pad_offsets, int E, int64_t cap, at::ScalarType sums_type) {
  const int64_t cols = src.size(1);
  void* s = stream_of(src);
  Tensor out = sorted_buffer(cap, cols, src.scalar_type(), src), sums = empty({E, cols}, sums_type, src);
  if (sums_type != at::kFloat && !same16(sums, src)) fail("gather_rows_ess: sums are float32 or of the data's 16-bit type");
  Tensor ws = scratch(api.hexa_ess_workspace_bytes(cap, cols), src);
  const int type = dt(src) | (sums_type != at::kFloat ? HEXA_SUMS_16 : 0);
  const int64_t lds = ld(src), ldo = ld(out);
  call("hexa_gather_rows_ess", [&] {
    return api.hexa_gather_rows_ess(ptr(src), lds, row_token, pad_offsets, E, cap, cols, ptr(out), ldo,
                                    static_cast<float*>(ptr(sums)), cols, type, ptr(ws), (size_t)ws.numel(), s);
  });
  return {out, sums};
}
std::tuple<Tensor, Tensor> gather_rows_ess(const Tensor& src, const Tensor& row_token, const Tensor& pad_offsets, int E, int64_t cap, at::ScalarType sums_type) {
  stream_of(src);
  on_device_of(src, row_token, pad_offsets);
  return gather_ess_at(src, i32(row_token), i32(pad_offsets), E, cap, sums_type);
}

Tensor combine_at(const Tensor& src, const int32_t* token_row, int64_t T, int top_k, const OptTensor& out_) {
  const int64_t cols = src.size(1);
  void* s = stream_of(src);
  on_device_of(src, out_);
  Tensor out = out_ ? *out_ : empty({T, cols}, src.scalar_type(), src);
  const int type = dt(src);
  const int64_t lds = ld(src), ldo = ld(out);
  call("hexa_combine_rows", [&] { return api.hexa_combine_rows(ptr(src), lds, token_row, T, top_k, cols, ptr(out), ldo, type, s); });
  return out;
}
Tensor combine_rows(const Tensor& src, const Tensor& token_row, int64_t T, int top_k, const OptTensor& out_) {
  stream_of(src);
  on_device_of(src, token_row);
  return combine_at(src, i32(token_row), T, top_k, out_);
}

Tensor ess_at(const Tensor& src, const int32_t* pad_offsets, int E, int64_t cap, const OptTensor& out_, at::ScalarType out_type) {
  const int64_t cols = src.size(1);
  void* s = stream_of(src);
  on_device_of(src, out_);
  Tensor out = out_ ? *out_ : empty({E, cols}, out_type, src);
  if (out.scalar_type() != at::kFloat && !same16(out, src)) fail("ess: the result is float32 or of the data's 16-bit type");
  Tensor ws = scratch(api.hexa_ess_workspace_bytes(cap, cols), src);
  const int type = dt(src) | (out.scalar_type() != at::kFloat ? HEXA_SUMS_16 : 0);
  const int64_t lds = ld(src), ldo = ld(out);
  call("hexa_ess", [&] {
    return api.hexa_ess(ptr(src), lds, pad_offsets, E, cap, cols, static_cast<float*>(ptr(out)), ldo, type, ptr(ws), (size_t)ws.numel(), s);
  });
  return out;
}
Tensor ess(const Tensor& src, const Tensor& pad_offsets, int E, int64_t cap, const OptTensor& out_, at::ScalarType out_type) {
  stream_of(src);
  on_device_of(src, pad_offsets);
  return ess_at(src, i32(pad_offsets), E, cap, out_, out_type);
}

// The tables of a routing that the kernels read.
struct Tables {
  const int32_t *tile_expert, *pad_offsets, *row_token, *pair_block;
  int E;
  int64_t cap;
};

Tensor esmm_on(const Tensor& a, const Tensor& b, int b_layout, const Tables& r, const OptTensor& bias, int epilogue, int act, const OptTensor& aux,
               const OptTensor& out_, int engine, int64_t n_out, int64_t k, int e0, int e1, const OptTensor& sums) {
  const int E = r.E;
  const int64_t cap = r.cap;
  if (a.scalar_type() != b.scalar_type())
    fail(std::string("esmm: a is ") + c10::toString(a.scalar_type()) + " but b is " + c10::toString(b.scalar_type()));
  if (bias && bias->scalar_type() != at::kFloat && !same16(*bias, a)) fail("esmm: bias must be float32 or of the data's 16-bit type");
  if (sums && (e0 != 0 || e1 != E || (sums->scalar_type() != at::kFloat && !same16(*sums, a)) || sums->dim() != 2 || sums->size(0) != E || sums->size(1) != n_out ||
               sums->stride(1) != 1))
    fail("esmm: sums must be [E, n_out], float32 or of the data's 16-bit type, and needs the full expert range");
  void* s = stream_of(a);
  on_device_of(a, b, bias, aux, out_, sums);
  const int type = dt(a) | (bias && bias->scalar_type() != at::kFloat ? HEXA_BIAS_16 : 0);
  Tensor out = out_ ? *out_ : sorted_buffer(cap, n_out, a.scalar_type(), a);
  const int64_t lda = ld(a), ldo = ld(out), ldbias = bias ? ld(*bias) : 0, ldaux = aux ? ld(*aux) : 0;
  const float* bp = static_cast<const float*>(ptr(bias));
  const bool relu = epilogue == HEXA_EPI_ACT && act == HEXA_ACT_RELU;      // stays with the FMA chain, see hexa_esmm_f32
  const size_t planes = type == HEXA_F32 && engine == HEXA_ENGINE_AUTO && r.pair_block && e0 == 0 && e1 == E && !relu
                            ? api.hexa_esmm_f32_workspace_bytes(E, cap, n_out, k) : 0;
  if (OptTensor ws = planes ? scratch_if_free(planes, a) : std::nullopt) {
    auto f = [](void* v) { return static_cast<float*>(v); };
    call("hexa_esmm_f32", [&] {
      return api.hexa_esmm_f32(f(ptr(a)), lda, f(ptr(b)), b_layout, b.stride(1), b.stride(0), bp, ldbias, f(ptr(aux)), ldaux, f(ptr(out)),
                               ldo, r.tile_expert, r.pad_offsets, r.row_token, r.pair_block, E, cap, n_out, k, epilogue,
                               act, ptr(ws), (size_t)ws->numel(), s);
    });
    ws.reset();
    if (sums) ess_at(out, r.pad_offsets, E, cap, sums, at::kFloat);
    return out;
  }
  if (sums) {
    const int sums_flag = sums->scalar_type() != at::kFloat ? HEXA_SUMS_16 : 0;
    Tensor ws = scratch(api.hexa_ess_workspace_bytes(cap, n_out), a);
    call("hexa_esmm_ess", [&] {
      return api.hexa_esmm_ess(ptr(a), lda, ptr(b), b_layout, b.stride(1), b.stride(0), bp, ldbias, ptr(aux), ldaux, ptr(out), ldo,
                               r.tile_expert, r.pad_offsets, r.row_token, r.pair_block, E, cap, n_out, k, type | sums_flag, epilogue, act,
                               engine, static_cast<float*>(ptr(sums)), sums->stride(0), ptr(ws), (size_t)ws.numel(), s);
    });
    return out;
  }
  call("hexa_esmm", [&] {
    return api.hexa_esmm_experts(ptr(a), lda, ptr(b), b_layout, b.stride(1), b.stride(0), bp, ldbias, ptr(aux), ldaux, ptr(out), ldo,
                                 r.tile_expert, r.pad_offsets, r.row_token, r.pair_block, E, cap, n_out, k, type, epilogue,
                                 act, engine, e0, e1, s);
  });
  return out;
}
Tensor esmm(const Tensor& a, const Tensor& b, int b_layout, const Tensor& tile_expert, const Tensor& pad_offsets, const Tensor& row_token,
            const OptTensor& pair_block, int E, int64_t cap, const OptTensor& bias, int epilogue, int act, const OptTensor& aux,
            const OptTensor& out_, int engine, int64_t n_out, int64_t k, int e0, int e1, const OptTensor& sums) {
  stream_of(a);
  on_device_of(a, tile_expert, pad_offsets, row_token, pair_block);
  return esmm_on(a, b, b_layout, {i32(tile_expert), i32(pad_offsets), i32(row_token), i32(pair_block), E, cap}, bias, epilogue, act, aux,
                 out_, engine, n_out, k, e0, e1, sums);
}

// out given: its strides say where results go ([E, m, n], or [ranks, E, m / ranks, n] with ranks > 1)
Tensor estmm_at(const Tensor& p, const Tensor& q, const int32_t* pad_offsets, int E, int64_t cap, const OptTensor& out_,
                std::optional<at::ScalarType> out_dtype, int beta, int engine, int64_t ranks) {
  const int64_t m = p.size(1), n = q.size(1);
  if (p.scalar_type() != q.scalar_type()) fail("estmm: p and q dtypes differ");
  const at::ScalarType type = out_dtype.value_or(p.scalar_type());
  Tensor out;
  int64_t ldo, estride, m_split = 0, split_stride = 0;
  if (ranks > 1) {
    if (m % ranks) fail("estmm: the row count must be divisible by ranks");
    out = out_ ? *out_ : empty({ranks, E, m / ranks, n}, type, p);
    ldo = out.stride(2); estride = out.stride(1); m_split = m / ranks; split_stride = out.stride(0);
  } else {
    if (!out_ && beta) fail("estmm: beta=1 needs an existing out");
    out = out_ ? *out_ : empty({E, m, n}, type, p);
    ldo = out.stride(1); estride = out.stride(0);
  }
  if (out.stride(-1) != 1) fail("estmm: out must have unit inner stride");
  void* s = stream_of(p);
  on_device_of(p, q, out);
  const int in_type = dt(p), o_type = dt(out);
  const int64_t ldp = ld(p), ldq = ld(q);
  size_t bytes = engine != HEXA_ENGINE_SIMT ? api.hexa_estmm_workspace_bytes(E, cap, m, n, in_type) : 0;
  OptTensor ws;
  if (bytes && in_type == HEXA_F32) ws = scratch_if_free(bytes, p);
  else if (bytes) ws = scratch(bytes, p);      // the chunks of a 16-bit weight gradient bound its error
  if (!ws) bytes = 0;
  call("hexa_estmm", [&] {
    return api.hexa_estmm(ptr(p), ldp, ptr(q), ldq, pad_offsets, E, cap, m, n, ptr(out), ldo, estride, m_split, split_stride, in_type,
                          o_type, beta, engine, ptr(ws), bytes, s);
  });
  return out;
}
Tensor estmm(const Tensor& p, const Tensor& q, const Tensor& pad_offsets, int E, int64_t cap, const OptTensor& out_,
             std::optional<at::ScalarType> out_dtype, int beta, int engine, int64_t ranks) {
  on_device_of(p, q, pad_offsets);
  return estmm_at(p, q, i32(pad_offsets), E, cap, out_, out_dtype, beta, engine, ranks);
}

// ---- the step before routing ---------------------------------------------------------------------------------------------
std::tuple<Tensor, Tensor, Tensor, Tensor> gate_topk(const Tensor& logits, int top_k) {
  if (logits.scalar_type() != at::kFloat || logits.dim() != 2 || logits.stride(1) != 1)
    fail("gate_topk: logits must be float32 [T,E] with unit inner stride");
  const int64_t T = logits.size(0), E = logits.size(1);
  void* s = stream_of(logits);
  Tensor ids = empty({top_k, T}, at::kInt, logits), mass = empty({E}, at::kFloat, logits), cnt = empty({E}, at::kInt, logits);
  Tensor loss = empty({}, at::kFloat, logits), ws = scratch(api.hexa_gate_workspace_bytes(), logits);
  call("hexa_gate_topk", [&] {
    return api.hexa_gate_topk(static_cast<const float*>(ptr(logits)), logits.stride(0), T, (int)E, top_k, static_cast<int32_t*>(ptr(ids)),
                              static_cast<float*>(ptr(mass)), static_cast<int32_t*>(ptr(cnt)), static_cast<float*>(ptr(loss)), ptr(ws),
                              (size_t)ws.numel(), s);
  });
  return {ids, loss, cnt, mass};
}

Tensor gate_loss_grad(const Tensor& logits, const Tensor& first_count, const Tensor& dloss_) {
  const int64_t T = logits.size(0), E = logits.size(1);
  void* s = stream_of(logits);
  on_device_of(logits, first_count, dloss_);
  Tensor out = empty({T, E}, at::kFloat, logits);
  const Tensor dloss = dloss_.detach().to(at::kFloat).reshape({1}).contiguous();
  const int64_t ldl = ld(logits);
  call("hexa_gate_loss_grad", [&] {
    return api.hexa_gate_loss_grad(static_cast<const float*>(ptr(logits)), ldl, T, (int)E, i32(first_count),
                                   static_cast<const float*>(ptr(dloss)), static_cast<float*>(ptr(out)), E, s);
  });
  return out;
}

Tensor gate_split_terms(const Tensor& src, bool by_rows) {
  if (src.scalar_type() != at::kFloat || src.dim() != 2 || !src.is_contiguous()) fail("gate_split_terms: src must be contiguous float32");
  const int64_t rows = src.size(0), cols = src.size(1);
  void* s = stream_of(src);
  Tensor out = by_rows ? empty({4 * rows, cols}, at::kBFloat16, src) : empty({rows, 4 * cols}, at::kBFloat16, src);
  call("hexa_gate_split_terms", [&] { return api.hexa_gate_split_terms(static_cast<const float*>(ptr(src)), cols, rows, cols, by_rows, ptr(out), s); });
  return out;
}

Tensor gate_sum_terms(const Tensor& part, int64_t rows, int64_t cols, bool lo_first) {
  if (part.scalar_type() != at::kFloat || !part.is_contiguous() || part.numel() != 3 * rows * cols)
    fail("gate_sum_terms: part must be contiguous float32 of 3 * rows * cols elements");
  void* s = stream_of(part);
  Tensor out = empty({rows, cols}, at::kFloat, part);
  call("hexa_gate_sum_terms", [&] {
    return api.hexa_gate_sum_terms(static_cast<const float*>(ptr(part)), rows, cols, lo_first, static_cast<float*>(ptr(out)), s);
  });
  return out;
}

Tensor gate_project(const Tensor& x, const Tensor& w) {
  if (w.scalar_type() != at::kFloat || w.dim() != 2 || !w.is_contiguous() || x.dim() != 2 || x.size(1) != w.size(1))
    fail("gate_project: w must be contiguous float32 [E, d] and x [T, d]");
  void* s = stream_of(x);
  on_device_of(x, w);
  const int type = dt(x);
  const int64_t ldx = ld(x), T = x.size(0), E = w.size(0);
  Tensor out = empty({T, E}, at::kFloat, x);
  call("hexa_gate_project", [&] {
    return api.hexa_gate_project(ptr(x), ldx, static_cast<const float*>(ptr(w)), T, (int)E, x.size(1), type, static_cast<float*>(ptr(out)), s);
  });
  return out;
}

std::tuple<OptTensor, OptTensor> gate_project_grad(const Tensor& g, const Tensor& x, const Tensor& w, bool want_dx, bool want_dw) {
  if (g.scalar_type() != at::kFloat || g.dim() != 2 || !g.is_contiguous() || g.size(0) != x.size(0) || g.size(1) != w.size(0) || !w.is_contiguous())
    fail("gate_project_grad: g must be contiguous float32 [T, E]");
  void* s = stream_of(g);
  on_device_of(g, x, w);
  const int type = dt(x);
  const int64_t ldx = ld(x);
  OptTensor dx, dw;
  if (want_dx) dx = empty({x.size(0), x.size(1)}, x.scalar_type(), x);
  if (want_dw) dw = empty({w.size(0), w.size(1)}, at::kFloat, x);
  call("hexa_gate_project_grad", [&] {
    return api.hexa_gate_project_grad(static_cast<const float*>(ptr(g)), ptr(x), ldx, static_cast<const float*>(ptr(w)), x.size(0), (int)w.size(0),
                                      x.size(1), type, ptr(dx), static_cast<float*>(ptr(dw)), s);
  });
  return {dx, dw};
}

// ---- the layer as autograd nodes --------------------------------------------------------------------------------------------
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

bool wants_grad(std::initializer_list<const Tensor*> inputs) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : inputs)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// Whether something follows the operations of a backward pass one by one (create_graph, batches of gradients, dispatch modes,
// tracing): kernels that take raw pointers would escape it.
bool followed(const Tensor& grad) {
  constexpr c10::DispatchKeySet wrapped({c10::DispatchKey::Batched, c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                         c10::DispatchKey::Python, c10::DispatchKey::Functionalize});
  return at::GradMode::is_enabled() || grad.key_set().has_any(wrapped) || c10::impl::dispatch_mode_enabled() ||
         c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) || torch::jit::tracer::isTracing() ||
         grad._fw_grad(0).defined();
}

template <typename N, typename... Args> std::shared_ptr<N> make_node(torch::autograd::edge_list&& edges, Args&&... args) {
  std::shared_ptr<N> node(new N(std::forward<Args>(args)...), torch::autograd::deleteNode);
  node->set_next_edges(std::move(edges));
  return node;
}

// 2-D with rows of whole, aligned 16-byte groups that do not overlap, as the projection kernels read them
bool whole_groups(const Tensor& t) {
  return t.is_cuda() && t.dim() == 2 && t.size(1) % 8 == 0 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && t.stride(0) >= t.size(1) &&
         reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// logits = x W^T of few tokens (hexa_gate_project)
struct GateLinearBackward : Node {
  SavedVariable x_, w_;
  GateLinearBackward(const Tensor& x, const Tensor& w) : x_(x, false), w_(w, false) {}
  std::string name() const override { return "HexaGateLinearBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    x_.reset_data();
    w_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(2);
    if (!grads[0].defined()) return out;
    const Tensor x = x_.unpack(), w = w_.unpack();
    const bool dx = should_compute_output(0), dw = should_compute_output(1);
    const Tensor g = grads[0].to(at::kFloat);
    if (followed(grads[0]) || !(whole_groups(x) && whole_groups(w) && w.is_contiguous())) {
      // create_graph, batched gradients, or saved tensors that a hook gave back otherwise: the same products in operations
      // that autograd and vmap can follow and that take any layout
      if (dx) out[0] = g.matmul(w).to(x.scalar_type());
      if (dw) out[1] = g.t().matmul(x.to(at::kFloat));
      return out;
    }
    auto [gx, gw] = gate_project_grad(g.contiguous(), x, w, dx, dw);
    if (gx) out[0] = *gx;
    if (gw) out[1] = *gw;
    return out;
  }
};

Tensor gate_linear(const Tensor& x, const Tensor& w) {
  Tensor logits;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    logits = gate_project(x, w);
  }
  if (wants_grad({&x, &w}))
    torch::autograd::set_history(logits, make_node<GateLinearBackward>(torch::autograd::collect_next_edges(x, w), x, w));
  return logits;
}

// softmax + top-k + GShard loss (hexa_gate_topk / hexa_gate_loss_grad)
struct TopKBackward : Node {
  SavedVariable logits_, first_count_;
  TopKBackward(const Tensor& logits, const Tensor& first) : logits_(logits, false), first_count_(first, false) {}
  std::string name() const override { return "HexaTopKGShardBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    logits_.reset_data();
    first_count_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(1);
    if (grads[0].defined()) out[0] = gate_loss_grad(logits_.unpack(), first_count_.unpack(), grads[0]);
    return out;
  }
};

std::tuple<Tensor, Tensor> topk_gshard(const Tensor& logits, int top_k) {
  Tensor ids, loss, first, mass;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    std::tie(ids, loss, first, mass) = gate_topk(logits, top_k);
  }
  if (wants_grad({&logits}))
    torch::autograd::set_history(loss, make_node<TopKBackward>(torch::autograd::collect_next_edges(logits), logits, first));
  return {ids, loss};
}

// What the backward of a layer needs, all in sorted-row layout.
struct LayerState {
  Tensor ints;                  // every table of the routing
  Tables r;
  const int32_t* token_row;     // in `ints`, as the pointers of `r`
  int64_t T;
  int k;
  Tensor xs, y1, h, w1, w2;
  bool has_b1, has_b2;
  int act;
};

bool sums_with_gemm() {      // HEXA_FUSED_ESS=0: db1 by the separate pass
  const char* v = getenv("HEXA_FUSED_ESS");
  return !v || std::string(v) != "0";
}

Tensor layer_forward(const Tensor& x, const Tensor& ids, const Tensor& w1, const Tensor& w2, const OptTensor& b1, const OptTensor& b2, int act,
                     LayerState& st, bool keep) {
  const int E = (int)w1.size(0), k = (int)ids.size(0);
  const int64_t T = x.size(0), H = w1.size(1), d = w1.size(2), d_out = w2.size(2);
  void* s = stream_of(x);
  const int64_t cap = api.hexa_route_row_capacity(T, k, E, 128), pairs = api.hexa_route_pair_capacity(T, k, E);
  if (cap < 0 || pairs < 0) fail("route: bad sizes");
  // one allocation for the routing's tables and its workspace, each on a 256-byte boundary
  const size_t ws_bytes = api.hexa_route_workspace_bytes(T, k, E);
  int64_t words = 0;
  auto take = [&](int64_t n) {
    const int64_t at = words;
    words += (n + 63) / 64 * 64;
    return at;
  };
  const int64_t o_counts = take(E), o_seg = take(E + 1), o_pad = take(E + 1), o_row = take(cap), o_token = take(T * k), o_tile = take(cap / 128),
                o_pair = take(pairs), o_ws = take((int64_t)(ws_bytes + 3) / 4);
  st.ints = empty({words}, at::kInt, x);
  int32_t* base = static_cast<int32_t*>(ptr(st.ints));
  call("hexa_route", [&] {
    return api.hexa_route(i32(ids), T, k, ids.stride(1), ids.stride(0), E, 128, base + o_counts, base + o_seg, base + o_pad, base + o_row,
                          base + o_token, base + o_tile, base + o_pair, base + o_ws, ws_bytes, s);
  });
  st.r = {base + o_tile, base + o_pad, base + o_row, base + o_pair, E, cap};
  st.token_row = base + o_token;
  st.T = T;
  st.k = k;
  st.xs = gather_at(x, st.r.row_token, st.r.pad_offsets, E, cap, std::nullopt);
  st.h = sorted_buffer(cap, H, x.scalar_type(), x);
  OptTensor y1;      // only a backward pass reads the pre-activation
  if (keep) y1 = st.y1 = sorted_buffer(cap, H, x.scalar_type(), x);
  esmm_on(st.xs, w1, HEXA_B_NK, st.r, b1, HEXA_EPI_ACT, act, y1, st.h, HEXA_ENGINE_AUTO, H, d, 0, E, std::nullopt);
  if (!keep) st.xs.reset();
  const Tensor ys = esmm_on(st.h, w2, HEXA_B_KN, st.r, b2, HEXA_EPI_LINEAR, HEXA_ACT_NONE, std::nullopt, std::nullopt, HEXA_ENGINE_AUTO, d_out, H,
                            0, E, std::nullopt);
  return combine_at(ys, st.token_row, T, k, std::nullopt);
}

struct MoELayerBackward : Node {
  std::unique_ptr<LayerState> st;
  std::shared_ptr<PyObject> config;
  int64_t stage;
  MoELayerBackward(std::unique_ptr<LayerState> state, std::shared_ptr<PyObject> cfg, int64_t stage_)
      : st(std::move(state)), config(std::move(cfg)), stage(stage_) {}
  std::string name() const override { return "HexaMoELayerBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    st.reset();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(5);
    if (!st) throw std::runtime_error("Trying to backward through an MoE layer a second time: it keeps what its backward pass needs for one pass");
    if (!grads[0].defined()) return out;
    {
      at::AutoGradMode no_grad(false);
      const std::unique_ptr<LayerState> s = std::move(st);
      const Tensor dy = grads[0].contiguous();
      const Tables& r = s->r;
      const int E = r.E;
      const int64_t H = s->w1.size(1), d = s->w1.size(2), d_out = s->w2.size(2);
      const at::ScalarType type = dy.scalar_type();
      Tensor dys;
      if (s->has_b2) std::tie(dys, out[4]) = gather_ess_at(dy, r.row_token, r.pad_offsets, E, r.cap, type);
      else dys = gather_at(dy, r.row_token, r.pad_offsets, E, r.cap, std::nullopt);
      out[2] = estmm_at(s->h, dys, r.pad_offsets, E, r.cap, std::nullopt, type, 0, HEXA_ENGINE_AUTO, 1);
      const bool with_gemm = s->has_b1 && sums_with_gemm();
      if (with_gemm) out[3] = empty({E, H}, type, dy);
      const Tensor dh = esmm_on(dys, s->w2, HEXA_B_NK, r, std::nullopt, HEXA_EPI_DACT, s->act, s->y1, std::nullopt, HEXA_ENGINE_AUTO, H, d_out, 0, E,
                                with_gemm ? OptTensor(out[3]) : std::nullopt);
      dys.reset();
      if (s->has_b1 && !with_gemm) out[3] = ess_at(dh, r.pad_offsets, E, r.cap, std::nullopt, type);
      out[1] = estmm_at(dh, s->xs, r.pad_offsets, E, r.cap, std::nullopt, type, 0, HEXA_ENGINE_AUTO, 1);
      const Tensor dxs = esmm_on(dh, s->w1, HEXA_B_KN, r, std::nullopt, HEXA_EPI_LINEAR, HEXA_ACT_NONE, std::nullopt, std::nullopt, HEXA_ENGINE_AUTO, d,
                                 H, 0, E, std::nullopt);
      out[0] = combine_at(dxs, s->token_row, s->T, s->k, std::nullopt);
    }
    py::gil_scoped_acquire gil;
    py::reinterpret_borrow<py::object>(config.get())["stage"] = py::int_(stage - 1);
    return out;
  }
};

// The layer on one GPU, or None where a call needs more than this does (the caller then takes the general path): weights,
// biases and tokens of one type, biases that the kernels read as they are.
py::object moe_layer(const py::object& config, int64_t stage, int act, const Tensor& x, const Tensor& ids, const Tensor& w1, const Tensor& w2,
                     const OptTensor& b1, const OptTensor& b2) {
  const at::ScalarType type = x.scalar_type();
  auto weight = [&](const Tensor& w) { return w.scalar_type() == type && w.dim() == 3 && w.stride(2) == 1 && w.device() == x.device(); };
  auto bias = [&](const OptTensor& b, int64_t n) {
    if (!b) return true;
    return b->scalar_type() == type && b->device() == x.device() && b->dim() == 2 && b->size(0) == w1.size(0) && b->size(1) == n &&
           b->stride(1) == 1 && b->stride(0) >= n && (type != at::kFloat || (n % 4 == 0 && b->is_contiguous()));
  };
  if ((type != at::kFloat && type != at::kHalf && type != at::kBFloat16) || !x.is_cuda() || x.dim() != 2 || !x.is_contiguous() || x.size(0) == 0 ||
      !weight(w1) || !weight(w2) || w1.size(0) != w2.size(0) || w1.size(1) != w2.size(1) || w1.size(2) != x.size(1) || !bias(b1, w1.size(1)) ||
      !bias(b2, w2.size(2)) || ids.scalar_type() != at::kInt || ids.dim() != 2 || ids.size(1) != x.size(0) || ids.device() != x.device())
    return py::none();
  const Tensor none, &c1 = b1 ? *b1 : none, &c2 = b2 ? *b2 : none;
  const bool grad = wants_grad({&x, &w1, &w2, &c1, &c2});
  auto st = std::make_unique<LayerState>();
  Tensor y;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    y = layer_forward(x, ids, w1, w2, b1, b2, act, *st, grad);
  }
  if (grad) {
    st->w1 = w1.detach();
    st->w2 = w2.detach();
    st->has_b1 = b1.has_value();
    st->has_b2 = b2.has_value();
    st->act = act;
    Py_INCREF(config.ptr());
    std::shared_ptr<PyObject> held(config.ptr(), [](PyObject* p) {
      if (!Py_IsInitialized()) return;      // the interpreter is gone, and the object with it
      py::gil_scoped_acquire gil;
      Py_DECREF(p);
    });
    torch::autograd::set_history(y, make_node<MoELayerBackward>(torch::autograd::collect_next_edges(x, w1, w2, c1, c2), std::move(st), std::move(held), stage));
  }
  return py::cast(y);
}

void bind(const std::string& path, py::object error, py::object ensure, py::object text) {
  void* handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!handle) throw std::runtime_error(dlerror());
#define HEXA_BIND(name)                                                  \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(handle, #name)); \
  if (!api.name) throw std::runtime_error(path + " does not export " #name);
  HEXA_API(HEXA_BIND)
  bound = new Bound{std::move(error), std::move(ensure), std::move(text)};
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("bind", &bind);
  m.def("route", &route);
  m.def("ids_from_lists", &ids_from_lists);
  m.def("gather_rows", &gather_rows);
  m.def("gather_rows_ess", &gather_rows_ess);
  m.def("combine_rows", &combine_rows);
  m.def("esmm", &esmm);
  m.def("estmm", &estmm);
  m.def("ess", &ess);
  m.def("gate_topk", &gate_topk);
  m.def("gate_loss_grad", &gate_loss_grad);
  m.def("gate_project", &gate_project);
  m.def("gate_project_grad", &gate_project_grad);
  m.def("gate_split_terms", &gate_split_terms);
  m.def("gate_sum_terms", &gate_sum_terms);
  // (wrapped: what a saved-tensor hook raises comes out as it was raised)
  m.def("gate_linear", torch::wrap_pybind_function(&gate_linear));
  m.def("topk_gshard", torch::wrap_pybind_function(&topk_gshard));
  m.def("moe_layer", torch::wrap_pybind_function(&moe_layer));
}
