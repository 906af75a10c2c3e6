// The host side of a call in native code: a CPython module (built as _host_path.so, linked against
// libbnb_trunk.so) that gathers a trunk's parameters, fills the C structs, takes outputs from torch's
// allocator and launches, without an interpreter in between.
//
// Why it exists: the same work as Python over ctypes took 230-250 us per trunk call (64 parameters
// x several attribute look-ups and checks, then the operator dispatcher), against 140 us of kernels
// at the small end.  Here it is a few microseconds beside the launches themselves.
//
// The Python side (yemong/_ops.py, yemong/_end_ops.py) keeps what is policy: which buffer is the
// scratch of a stream, the warning about slow engine choices, the autograd formulas.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstdlib>
#include <cstring>
#include <memory>
#include <vector>

#include "bnb_trunk.h"
#include "host_calls.h"
#include "mlp_kernels.h"
#include "policy_tail.h"
#include "split_kernels.h"
#include "tensor_kernels.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = c10::optional<Tensor>;

namespace {

// ------------------------------------------------------------------ parameters of a trunk

// Names interned once; a module's children and parameters are read from its own dictionaries, so a
// replaced sub-module or parameter is seen at the next call.
struct Names {
  PyObject *modules, *parameters, *spatial, *temporal, *field_sub, *norm1, *qkv, *out_proj, *norm2, *ffn, *gate_proj, *up_proj,
      *down_proj, *norm_bullet, *kv_bullet, *weight, *bias, *linear1, *conv, *rg_lru, *log_lambda, *linear_a, *linear_x, *linear2,
      *linear_out, *gated_mlp;
};
const Names& names() {
  static const Names* n = [] {
    auto s = [](const char* t) { return PyUnicode_InternFromString(t); };
    return new Names{s("_modules"), s("_parameters"), s("spatial"), s("temporal"), s("field_sub"), s("norm1"), s("qkv"), s("out_proj"),
                     s("norm2"), s("ffn"), s("gate_proj"), s("up_proj"), s("down_proj"), s("norm_bullet"), s("kv_bullet"), s("weight"),
                     s("bias"), s("linear1"), s("conv"), s("rg_lru"), s("log_lambda"), s("linear_a"), s("linear_x"), s("linear2"),
                     s("linear_out"), s("gated_mlp")};
  }();
  return *n;
}

// Borrowed reference to module.<dict>[key], or nullptr without an exception set.
PyObject* member(PyObject* module, PyObject* dict_name, PyObject* key) {
  if (!module) return nullptr;
  PyObject* d = PyObject_GetAttr(module, dict_name);
  if (!d) { PyErr_Clear(); return nullptr; }
  PyObject* v = PyDict_Check(d) ? PyDict_GetItemWithError(d, key) : nullptr;
  Py_DECREF(d);   // the module keeps it
  return v;
}
struct Gather {
  std::vector<Tensor> out;
  bool ok = true;
  PyObject* child(PyObject* m, PyObject* key) { return member(m, names().modules, key); }
  void param(PyObject* m, PyObject* key) {
    PyObject* p = member(m, names().parameters, key);
    if (!p || !THPVariable_Check(p)) { ok = false; return; }
    out.push_back(THPVariable_Unpack(p));
  }
  void weight(PyObject* m, PyObject* name) { param(child(m, name), names().weight); }
  void mlp(PyObject* m) {
    const Names& n = names();
    weight(m, n.gate_proj);
    weight(m, n.up_proj);
    weight(m, n.down_proj);
  }
  std::vector<PyObject*> items(PyObject* list) {   // children of a ModuleList, in order
    std::vector<PyObject*> v;
    if (!list) { ok = false; return v; }
    PyObject* d = PyObject_GetAttr(list, names().modules);
    if (!d) { PyErr_Clear(); ok = false; return v; }
    PyObject *k, *m;
    Py_ssize_t pos = 0;
    if (PyDict_Check(d)) while (PyDict_Next(d, &pos, &k, &m)) v.push_back(m);
    Py_DECREF(d);
    return v;
  }
};

// Parameters of `blocks` (YemongBlock modules) in the order of yemong/_weights.py, block-major, with
// the field substitutes where the call has field tokens; None when a module does not hold its
// parameters in the ordinary place (a parametrisation), and the caller gathers them by attribute.
py::object trunk_params(const py::sequence& blocks, bool has_fields) {
  const Names& n = names();
  Gather g;
  g.out.reserve(80);
  for (const auto& b : blocks) {
    PyObject* block = b.ptr();
    for (PyObject* sp : g.items(g.child(block, n.spatial))) {
      g.weight(sp, n.norm1);
      g.weight(sp, n.qkv);
      g.weight(sp, n.out_proj);
      g.weight(sp, n.norm2);
      g.mlp(g.child(sp, n.ffn));
      if (g.child(sp, n.kv_bullet)) {
        g.weight(sp, n.norm_bullet);
        g.weight(sp, n.kv_bullet);
      }
    }
    const auto subs = g.items(g.child(block, n.field_sub));
    size_t j = 0;
    for (PyObject* tp : g.items(g.child(block, n.temporal))) {
      PyObject* lru = g.child(tp, n.rg_lru);
      PyObject* conv = g.child(tp, n.conv);
      g.weight(tp, n.norm1);
      g.weight(tp, n.linear1);
      g.param(conv, n.weight);
      g.param(conv, n.bias);
      g.param(lru, n.log_lambda);
      PyObject* la = g.child(lru, n.linear_a);
      PyObject* lx = g.child(lru, n.linear_x);
      g.param(la, n.weight);
      g.param(la, n.bias);
      g.param(lx, n.weight);
      g.param(lx, n.bias);
      g.weight(tp, n.linear2);
      g.weight(tp, n.linear_out);
      g.weight(tp, n.norm2);
      g.mlp(g.child(tp, n.gated_mlp));
      if (has_fields) {
        if (j >= subs.size()) { g.ok = false; break; }
        g.param(subs[j], n.weight);
      }
      ++j;
    }
    if (!g.ok) return py::none();
  }
  return py::cast(g.out);
}

// ------------------------------------------------------------------ small helpers

constexpr int kEngineSimt = BNB_ENGINE_SIMT;

const void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }

Tensor f32c(const Tensor& t) {
  if (t.scalar_type() == at::kBFloat16 && t.is_cuda() && t.is_contiguous() && t.numel() % 8 == 0 &&
      reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0) {
    const c10::cuda::CUDAGuard guard(t.device());
    const Tensor f = at::empty(t.sizes(), t.options().dtype(at::kFloat));
    if (bnb::host::widen(t.data_ptr(), static_cast<float*>(f.data_ptr()), (size_t)t.numel(), at::cuda::getCurrentCUDAStream(t.device().index()).stream()) != BNB_OK)
      throw std::runtime_error("the bfloat16 conversion could not be launched");
    return f;
  }
  const Tensor f = t.scalar_type() == at::kFloat ? t : t.to(at::kFloat);
  return f.is_contiguous() ? f : f.contiguous();
}
Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
// One byte per element: a bool tensor as it is, anything else compared with zero.
OptTensor bytes_of(const OptTensor& t) {
  if (!t.has_value()) return c10::nullopt;
  return t->scalar_type() == at::kBool ? contiguous(*t) : contiguous(t->ne(0));
}
const float* parameter(const Tensor& t, const c10::Device& dev, const char* what) {
  if (t.device() != dev)
    throw std::runtime_error(std::string(what) + " parameter is on " + t.device().str() + ", input on " + dev.str());
  if (t.scalar_type() != at::kFloat || !t.is_contiguous())
    throw std::runtime_error(std::string(what) + " parameter must be contiguous float32 (got " + c10::toString(t.scalar_type()) + ")");
  return static_cast<const float*>(t.data_ptr());
}
void check(const char* fn, int status) {
  if (status == BNB_OK) return;
  const std::string text = std::string(fn) + ": " + bnb_status_string(status);
  if (status == BNB_ERR_UNSUPPORTED_DIMS) throw py::value_error(text);
  throw std::runtime_error(text + " (status " + std::to_string(status) + ")");
}
// A bounded wait of an earlier call on this device ran out (its kernels drained and its outputs were
// garbage): say so once, at the next call, without synchronising.
void raise_pending_status(const c10::Device& dev) {
  const int st = bnb_last_status();
  if (!st) return;
  bnb_clear_status();
  throw std::runtime_error("an earlier tensor-core call on " + dev.str() + " gave up a bounded wait: " + bnb_status_string(st) +
                           " (status " + std::to_string(st) + "); its outputs, and any state carried from them, are invalid");
}

constexpr int N_SPATIAL = 7, N_TEMPORAL = 15;   // parameters of a sublayer, + bullets / field substitute

// The integers of a call (yemong/_ops.py names the entries).
struct Geometry {
  int blocks, spatial, temporal, heads, bullet_cross, field_sub, envs, tokens_per_env, ships_per_env, max_tokens, total_tokens,
      total_ships, tiles, timesteps, engine, precision;
  explicit Geometry(const std::vector<int64_t>& g) {
    if (g.size() != 16) throw std::runtime_error("geom must hold 16 integers");
    int* f[] = {&blocks, &spatial, &temporal, &heads, &bullet_cross, &field_sub, &envs, &tokens_per_env, &ships_per_env, &max_tokens,
                &total_tokens, &total_ships, &tiles, &timesteps, &engine, &precision};
    for (int i = 0; i < 16; ++i) *f[i] = (int)g[i];
  }
  BnbBatch batch(const std::vector<Tensor>& offsets) const {
    BnbBatch b{};
    b.n_envs = envs;
    b.tokens_per_env = offsets.empty() ? tokens_per_env : 0;
    b.ships_per_env = offsets.empty() ? ships_per_env : 0;
    b.max_tokens_per_env = max_tokens;
    b.total_tokens = total_tokens;
    b.total_ships = total_ships;
    if (!offsets.empty()) {
      b.tok_off = static_cast<const int32_t*>(offsets[0].data_ptr());
      b.ship_off = static_cast<const int32_t*>(offsets[1].data_ptr());
      if (offsets.size() > 2) b.tile_env_begin = static_cast<const int32_t*>(offsets[2].data_ptr());
      if (offsets.size() > 3) b.tile_env_ids = static_cast<const int32_t*>(offsets[3].data_ptr());
      b.n_tiles = tiles;
    }
    return b;
  }
};

struct Weights {
  std::vector<BnbSpatialWeights> spatial;
  std::vector<BnbTemporalWeights> temporal;
};
Weights weight_structs(const Geometry& g, const std::vector<Tensor>& ts, const c10::Device& dev) {
  Weights w;
  w.spatial.resize((size_t)g.blocks * g.spatial);
  w.temporal.resize((size_t)g.blocks * g.temporal);
  size_t want = 0, pos = 0;
  for (int j = 0; j < g.spatial; ++j) want += N_SPATIAL + (j < g.bullet_cross ? 2 : 0);
  want += (size_t)g.temporal * (N_TEMPORAL + (g.field_sub ? 1 : 0));
  want *= g.blocks;
  if (want != ts.size())
    throw std::runtime_error("expected " + std::to_string(want) + " parameter tensors for this trunk structure, got " + std::to_string(ts.size()));
  for (int i = 0; i < g.blocks; ++i) {
    for (int j = 0; j < g.spatial; ++j) {
      BnbSpatialWeights& s = w.spatial[(size_t)i * g.spatial + j];
      s = BnbSpatialWeights{};
      const float** f[] = {&s.norm1_w, &s.qkv_w, &s.out_w, &s.norm2_w, &s.gate_w, &s.up_w, &s.down_w, &s.norm_bullet_w, &s.kv_bullet_w};
      const int n = N_SPATIAL + (j < g.bullet_cross ? 2 : 0);
      for (int k = 0; k < n; ++k) *f[k] = parameter(ts[pos++], dev, "spatial");
    }
    for (int j = 0; j < g.temporal; ++j) {
      BnbTemporalWeights& s = w.temporal[(size_t)i * g.temporal + j];
      s = BnbTemporalWeights{};
      const float** f[] = {&s.norm1_w, &s.linear1_w, &s.conv_w, &s.conv_b, &s.log_lambda, &s.a_w, &s.a_b, &s.x_w, &s.x_b, &s.linear2_w,
                           &s.out_w, &s.norm2_w, &s.gate_w, &s.up_w, &s.down_w, &s.field_sub_w};
      const int n = N_TEMPORAL + (g.field_sub ? 1 : 0);
      for (int k = 0; k < n; ++k) *f[k] = parameter(ts[pos++], dev, "temporal");
    }
  }
  return w;
}

// The bullet tokens of a call in the form the C ABI takes; holds what it converted.
struct Bullets {
  Tensor tokens;
  OptTensor active;
  BnbBullets arg{};
  bool present = false;
  Bullets(const OptTensor& bullets, const OptTensor& mask, int64_t n_envs, int64_t d_model, bool keep_bf16) {
    if (!bullets.has_value()) return;
    const Tensor& b = *bullets;
    if (b.dim() != 3 || b.size(0) != n_envs || b.size(2) != d_model || b.size(1) < 1) {
      std::ostringstream s;
      s << "bullets must have shape (" << n_envs << ", NB >= 1, " << d_model << "), got " << b.sizes();
      throw std::runtime_error(s.str());
    }
    if (!b.is_cuda())
      throw std::runtime_error("bullets is on " + b.device().str() + "; the trunk kernels run on CUDA only (sm_100a) and have no CPU path");
    if (mask.has_value() && (mask->dim() != 2 || mask->size(0) != b.size(0) || mask->size(1) != b.size(1))) {
      std::ostringstream s;
      s << "bullet_mask must have shape (" << b.size(0) << ", " << b.size(1) << "), got " << mask->sizes();
      throw std::runtime_error(s.str());
    }
    const bool is_bf16 = keep_bf16 && b.scalar_type() == at::kBFloat16;
    tokens = is_bf16 ? contiguous(b) : f32c(b);
    active = bytes_of(mask);
    arg.tokens = static_cast<const float*>(tokens.data_ptr());
    arg.active = static_cast<const uint8_t*>(ptr(active));
    arg.per_env = (int)b.size(1);
    arg.tokens_bf16 = is_bf16 ? 1 : 0;
    present = true;
  }
  const BnbBullets* get() const { return present ? &arg : nullptr; }
};

size_t round256(size_t v) { return (v + 255) / 256 * 256; }

// ------------------------------------------------------------------ the trunk

// What bnb_b200::trunk_forward does (yemong/_ops.py).  scratch_for(device, bytes) returns the byte
// buffer of the current stream.
std::tuple<Tensor, Tensor> trunk_forward(const Tensor& x, const OptTensor& alive, const Tensor& hidden, const OptTensor& done,
                                         const OptTensor& reset_env, const OptTensor& bullets, const OptTensor& bullet_mask,
                                         const std::vector<Tensor>& weights, const std::vector<Tensor>& offsets,
                                         const std::vector<int64_t>& geom, const py::object& scratch_for) {
  const Geometry g(geom);
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int64_t D = x.size(-1);
  const int T = g.timesteps > 1 ? g.timesteps : 1;
  const BnbBatch batch = g.batch(offsets);
  const bool bf16 = g.precision == BNB_BF16, tensor_engine = bf16 && g.engine != kEngineSimt;
  const bool built = tensor_engine && g.max_tokens > 0 && bnb_supported((int)D, g.heads, g.max_tokens, BNB_BF16, BNB_ENGINE_TENSOR);
  // bfloat16 tokens stay bfloat16 on the way in and out where the fused kernels serve the call;
  // anything else is converted to float32 here
  const bool io16 = built && x.scalar_type() == at::kBFloat16 && (offsets.empty() || offsets.size() > 2);
  // a float32 step runs from weight images too, unless the caller named the exact engine
  const bool split = !bf16 && g.engine != kEngineSimt && g.timesteps == 0 && bnb::split::supported((int)D, g.heads);
  const bool images = split || (tensor_engine && bnb_supported((int)D, g.heads, 1, BNB_BF16, BNB_ENGINE_TENSOR));

  Weights w = weight_structs(g, weights, dev);
  const Tensor hin = f32c(hidden);
  const OptTensor alive_u8 = bytes_of(alive), done_u8 = bytes_of(done), reset_u8 = bytes_of(reset_env);
  Tensor hout = at::empty_like(hin);
  raise_pending_status(dev);
  const auto stream = at::cuda::getCurrentCUDAStream(dev.index());

  auto run = [&](bool tokens16, bool bullets16, Tensor* y, bool* used_bullets16) {
    const Tensor xin = tokens16 ? contiguous(x) : f32c(x);
    *y = at::empty_like(xin);
    const Bullets b(g.bullet_cross > 0 ? bullets : c10::nullopt, bullet_mask, (int64_t)T * batch.n_envs, D, bullets16);
    *used_bullets16 = b.present && b.arg.tokens_bf16;
    const size_t need = round256(bnb_scratch_bytes((int)D, &batch, T, b.arg.per_env));
    const size_t sp = round256(split ? bnb::split::spatial_image_bytes() : bnb_packed_spatial_bytes((int)D));
    const size_t tp = round256(split ? bnb::split::temporal_image_bytes() : bnb_packed_temporal_bytes((int)D));
    const size_t image_bytes = images ? sp * w.spatial.size() + tp * w.temporal.size() : 0;
    const Tensor scratch = scratch_for(dev, need + image_bytes).cast<Tensor>();
    uint8_t* base = static_cast<uint8_t*>(scratch.data_ptr());
    // The weight images live behind the call's scratch and are rewritten from the parameters by every
    // call, so they cannot go stale: not after an optimizer step, not after p.data.copy_() (which bumps
    // no version counter; the reference's running-average policy is updated that way,
    // train/rl/opponents.py:112), and not in a replayed CUDA graph.
    uint8_t* image = base + need;
    for (auto& s : w.spatial) { s.packed = images ? image : nullptr; image += sp; }
    for (auto& s : w.temporal) { s.packed = images ? image : nullptr; image += tp; }
    return bnb::host::trunk_call(w.spatial.data(), w.temporal.data(), g.blocks, g.spatial, g.temporal, (int)D, g.heads, xin.data_ptr(),
                                 static_cast<const uint8_t*>(ptr(alive_u8)), b.get(), y->data_ptr(),
                                 static_cast<const float*>(hin.data_ptr()), static_cast<float*>(hout.data_ptr()),
                                 static_cast<const uint8_t*>(ptr(done_u8)), static_cast<const uint8_t*>(ptr(reset_u8)), &batch, T,
                                 tokens16 ? BNB_BF16_IO : g.precision, g.engine, base, (size_t)scratch.numel(), stream.stream(),
                                 g.timesteps != 0, images);
  };
  Tensor y;
  bool used16 = false;
  int st = run(io16, built, &y, &used16);
  // a shape the tensor-core kernels do not serve (say, more bullet slots than their attention stages;
  // nothing was launched): once more with float32 copies for the kernels that read float32
  if (st == BNB_ERR_UNSUPPORTED_DIMS && (io16 || used16)) st = run(false, false, &y, &used16);
  check(g.timesteps == 0 ? "bnb_trunk_step" : "bnb_trunk_sequence", st);
  if (x.scalar_type() == at::kBFloat16 && y.scalar_type() != at::kBFloat16) y = y.to(at::kBFloat16);
  return {y, hout};
}

// ------------------------------------------------------------------ the trunk under autograd

int grad_precision(const Geometry& g) { return g.precision == BNB_BF16 ? BNB_BF16 : BNB_FP32; }

// Whether a differentiated call keeps its activations (faster) or lets the backward recompute them:
// BNB_GRAD_MODE=keep | recompute decides; otherwise keep when the kept buffer plus the backward's scratch
// fit in 70 % of the memory that is free or cached.  What torch's allocator holds unused is looked at
// first: the driver's own answer takes 0.1 ms.
bool keep_activations(const c10::Device& dev, const Geometry& g, int64_t D, int64_t n_bullets) {
  const char* env = std::getenv("BNB_GRAD_MODE");
  const std::string mode = env ? env : "";
  if (mode == "recompute") return false;
  const c10::cuda::CUDAGuard guard(dev);
  const BnbBatch b = g.batch({});
  const int T = g.timesteps > 1 ? g.timesteps : 1;
  size_t need = bnb_trunk_kept_bytes(g.blocks, g.spatial, g.temporal, (int)D, g.heads, &b, T, (int)n_bullets, grad_precision(g));
  if (need == 0) return false;
  if (mode == "keep") return true;
  need += bnb_trunk_bwd_scratch_bytes(g.blocks, g.spatial, g.temporal, (int)D, &b, T, (int)n_bullets, grad_precision(g));
  const auto stats = c10::cuda::CUDACachingAllocator::getDeviceStats(dev.index());
  const double cached = (double)(stats.reserved_bytes[0].current - stats.allocated_bytes[0].current);
  if ((double)need <= 0.7 * cached) return true;
  size_t free_bytes = 0, total = 0;
  if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) return false;
  return (double)need <= 0.7 * ((double)free_bytes + cached);
}

template <class S>
void fill_grads(S& out, const float* flat, const std::vector<Tensor>& ts, size_t& pos, int n, size_t& off) {
  float** f = reinterpret_cast<float**>(&out);   // the struct is a row of float*
  for (int k = 0; k < n; ++k) {
    f[k] = const_cast<float*>(flat) + off;
    off += ((size_t)ts[pos++].numel() + 3) / 4 * 4;   // 16-byte granules
  }
}

struct BackwardResult { Tensor dx, dh, dbul, flat; };
// bnb_b200::trunk_backward (yemong/_ops.py).
BackwardResult run_backward(const Tensor& dy, const OptTensor& dhidden, const OptTensor& kept, const Tensor& x, const OptTensor& alive,
                            const Tensor& hidden, const OptTensor& done, const OptTensor& bullets, const OptTensor& mask,
                            const std::vector<Tensor>& weights, const std::vector<int64_t>& geom) {
  const Geometry g(geom);
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int D = (int)x.size(-1), T = g.timesteps > 1 ? g.timesteps : 1;
  const BnbBatch batch = g.batch({});
  const Tensor xin = f32c(x), hin = f32c(hidden), dyin = f32c(dy);
  OptTensor arena;   // may have been somewhere else since the forward wrote it
  if (kept.has_value()) {
    if (kept->device() != dev || kept->scalar_type() != at::kByte || kept->dim() != 1)
      throw std::runtime_error("the kept activations came back as another tensor: saved-tensor hooks have to return device, type and shape as they were");
    arena = contiguous(*kept);
    if (reinterpret_cast<uintptr_t>(arena->data_ptr()) % 256) arena = arena->clone();   // its layout counts from a 256-byte boundary
  }
  OptTensor dho;
  if (dhidden.has_value() && dhidden->defined()) dho = f32c(*dhidden);
  const OptTensor alive_u8 = bytes_of(alive), done_u8 = bytes_of(done);
  const Weights w = weight_structs(g, weights, dev);
  size_t total = 0;
  for (const Tensor& t : weights) total += ((size_t)t.numel() + 3) / 4 * 4;
  BackwardResult r;
  // one zeroed buffer for every parameter gradient: the kernels accumulate into it
  r.flat = at::zeros({(int64_t)total}, xin.options());
  std::vector<BnbSpatialGrads> sg(w.spatial.size());
  std::vector<BnbTemporalGrads> tg(w.temporal.size());
  size_t pos = 0, off = 0;
  const float* flat = static_cast<const float*>(r.flat.data_ptr());
  for (int i = 0; i < g.blocks; ++i) {
    for (int j = 0; j < g.spatial; ++j) {
      BnbSpatialGrads& s = sg[(size_t)i * g.spatial + j];
      s = BnbSpatialGrads{};
      fill_grads(s, flat, weights, pos, N_SPATIAL + (j < g.bullet_cross ? 2 : 0), off);
    }
    for (int j = 0; j < g.temporal; ++j) {
      BnbTemporalGrads& t = tg[(size_t)i * g.temporal + j];
      t = BnbTemporalGrads{};
      fill_grads(t, flat, weights, pos, N_TEMPORAL + (g.field_sub ? 1 : 0), off);
    }
  }
  const Bullets b(g.bullet_cross > 0 ? bullets : c10::nullopt, mask, (int64_t)T * batch.n_envs, D, false);
  r.dx = at::empty_like(xin);
  r.dh = at::zeros_like(hin);
  r.dbul = b.present ? at::empty_like(b.tokens) : at::empty({0}, xin.options());   // zeroed by the library
  const size_t bytes = bnb_trunk_bwd_scratch_bytes(g.blocks, g.spatial, g.temporal, D, &batch, T, b.arg.per_env, grad_precision(g));
  const Tensor scratch = at::empty({(int64_t)std::max<size_t>(bytes, 256)}, xin.options().dtype(at::kByte));   // released after the call's stream work
  check("bnb_trunk_sequence_bwd",
        bnb_trunk_sequence_bwd(w.spatial.data(), w.temporal.data(), sg.data(), tg.data(), g.blocks, g.spatial, g.temporal, D, g.heads,
                               static_cast<const float*>(xin.data_ptr()), static_cast<const uint8_t*>(ptr(alive_u8)), b.get(),
                               static_cast<const float*>(hin.data_ptr()), static_cast<const uint8_t*>(ptr(done_u8)), &batch, T, grad_precision(g),
                               static_cast<const float*>(dyin.data_ptr()), static_cast<const float*>(ptr(dho)), static_cast<float*>(r.dx.data_ptr()),
                               static_cast<float*>(r.dh.data_ptr()), b.present ? static_cast<float*>(r.dbul.data_ptr()) : nullptr,
                               arena.has_value() ? arena->data_ptr() : nullptr, arena.has_value() ? (size_t)arena->numel() : 0, scratch.data_ptr(),
                               (size_t)scratch.numel(), at::cuda::getCurrentCUDAStream(dev.index()).stream()));
  return r;
}
std::vector<Tensor> trunk_backward(const Tensor& dy, const OptTensor& dhidden, const OptTensor& kept, const Tensor& x, const OptTensor& alive,
                                   const Tensor& hidden, const OptTensor& done, const OptTensor& bullets, const OptTensor& mask,
                                   const std::vector<Tensor>& weights, const std::vector<int64_t>& geom) {
  const BackwardResult r = run_backward(dy, dhidden, kept, x, alive, hidden, done, bullets, mask, weights, geom);
  return {r.dx, r.dh, r.dbul, r.flat};
}

// bnb_b200::trunk_forward_train (yemong/_ops.py): (y, new hidden, kept activations).
std::tuple<Tensor, Tensor, Tensor> trunk_forward_train(const Tensor& x, const OptTensor& alive, const Tensor& hidden, const OptTensor& done,
                                                       const OptTensor& bullets, const OptTensor& mask, const std::vector<Tensor>& weights,
                                                       const std::vector<int64_t>& geom) {
  const Geometry g(geom);
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard guard(dev);
  const int D = (int)x.size(-1), T = g.timesteps > 1 ? g.timesteps : 1;
  const BnbBatch batch = g.batch({});
  const Tensor xin = f32c(x), hin = f32c(hidden);
  const OptTensor alive_u8 = bytes_of(alive), done_u8 = bytes_of(done);
  const Weights w = weight_structs(g, weights, dev);
  raise_pending_status(dev);
  const Bullets b(g.bullet_cross > 0 ? bullets : c10::nullopt, mask, (int64_t)T * batch.n_envs, D, false);
  Tensor y = at::empty_like(xin), hout = at::empty_like(hin);
  const auto bytes = xin.options().dtype(at::kByte);
  Tensor kept = at::empty({(int64_t)std::max<size_t>(256, bnb_trunk_kept_bytes(g.blocks, g.spatial, g.temporal, D, g.heads, &batch, T, b.arg.per_env, grad_precision(g)))}, bytes);
  const size_t need = bnb_trunk_bwd_scratch_bytes(g.blocks, g.spatial, g.temporal, D, &batch, T, b.arg.per_env, grad_precision(g));
  const Tensor scratch = at::empty({(int64_t)std::max<size_t>(need, 256)}, bytes);
  check("bnb_trunk_sequence_fwd_train",
        bnb_trunk_sequence_fwd_train(w.spatial.data(), w.temporal.data(), g.blocks, g.spatial, g.temporal, D, g.heads,
                                     static_cast<const float*>(xin.data_ptr()), static_cast<const uint8_t*>(ptr(alive_u8)), b.get(),
                                     static_cast<float*>(y.data_ptr()), static_cast<const float*>(hin.data_ptr()), static_cast<float*>(hout.data_ptr()),
                                     static_cast<const uint8_t*>(ptr(done_u8)), &batch, T, grad_precision(g), kept.data_ptr(), (size_t)kept.numel(),
                                     scratch.data_ptr(), (size_t)scratch.numel(), at::cuda::getCurrentCUDAStream(dev.index()).stream()));
  if (x.scalar_type() == at::kBFloat16) y = y.to(at::kBFloat16);
  return {y, hout, kept};
}

// Behind the gradients of a backward pass that is itself recorded (create_graph=True): the trunk has no second-order
// gradient, and whoever asks for one is told so, as by an operator without an autograd formula.
struct NoSecondOrder : public torch::autograd::Node {
  torch::autograd::variable_list apply(torch::autograd::variable_list&&) override {
    throw std::runtime_error("the gradients of the CUDA trunk cannot be differentiated again (a second-order gradient through it was asked for)");
  }
};

// The autograd node of an eager differentiated call: what the operators' formulas do, without Python in
// the backward pass.
struct TrunkNode : public torch::autograd::Node {
  // saved as autograd saves them, the kept activations among them: saved-tensor hooks (torch.utils.checkpoint,
  // save_on_cpu) move or recompute what they are given, and nothing else here holds on to it
  torch::autograd::SavedVariable x, alive, hidden, done, bullets, mask, kept;
  std::vector<torch::autograd::SavedVariable> weights;
  std::vector<int64_t> geom;
  bool consumed = false;

  static OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : c10::nullopt; }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (consumed)
      throw std::runtime_error("the kept activations of this trunk call were consumed by an earlier backward; for a second backward "
                               "through the same graph set BNB_GRAD_MODE=recompute");
    consumed = true;
    const bool recorded = at::GradMode::is_enabled();
    const at::NoGradGuard no_grad;
    const Tensor xv = x.unpack(), av = alive.unpack(), hv = hidden.unpack(), ov = done.unpack(), bv = bullets.unpack(), mv = mask.unpack();
    const Tensor kv = kept.unpack();
    kept.reset_data();
    std::vector<Tensor> ws;
    ws.reserve(weights.size());
    for (auto& w : weights) ws.push_back(w.unpack());
    const Tensor dy = grads[0].defined() ? grads[0] : at::zeros_like(xv, xv.options().dtype(at::kFloat));
    const BackwardResult r = run_backward(dy, opt(grads[1]), kv, xv, opt(av), hv, opt(ov), opt(bv), opt(mv), ws, geom);
    torch::autograd::variable_list out;
    out.reserve(3 + ws.size());
    out.push_back(task_should_compute_output(0) ? r.dx.reshape(xv.sizes()).to(xv.scalar_type()) : Tensor());
    out.push_back(task_should_compute_output(1) ? r.dh.reshape(hv.sizes()).to(hv.scalar_type()) : Tensor());
    out.push_back(bv.defined() && r.dbul.numel() && task_should_compute_output(2) ? r.dbul.reshape(bv.sizes()).to(bv.scalar_type()) : Tensor());
    int64_t off = 0;
    for (size_t i = 0; i < ws.size(); ++i) {
      const int64_t n = ws[i].numel();
      out.push_back(task_should_compute_output(3 + i) ? r.flat.narrow(0, off, n).view(ws[i].sizes()) : Tensor());
      off += (n + 3) / 4 * 4;
    }
    if (recorded) {
      torch::autograd::variable_list from{xv, hv, bv, grads[0], grads[1]};
      from.insert(from.end(), ws.begin(), ws.end());
      auto again = std::make_shared<NoSecondOrder>();
      again->set_next_edges(torch::autograd::collect_next_edges(from));
      for (Tensor& t : out)
        if (t.defined()) {
          t = t.detach();   // a tensor of its own, not a view of the flat buffer
          torch::autograd::create_gradient_edge(t, again);
        }
    }
    return out;
  }
  void release_variables() override {
    for (auto* v : {&x, &alive, &hidden, &done, &bullets, &mask, &kept}) v->reset_data();
    weights.clear();
  }
};

// A differentiated call with its activations kept: (y, new hidden) with the node above behind them.
std::tuple<Tensor, Tensor> trunk_train(const Tensor& x, const OptTensor& alive, const Tensor& hidden, const OptTensor& done,
                                       const OptTensor& bullets, const OptTensor& mask, const std::vector<Tensor>& weights,
                                       const std::vector<int64_t>& geom) {
  auto node = std::make_shared<TrunkNode>();
  torch::autograd::variable_list inputs{x, hidden, bullets.has_value() ? *bullets : Tensor()};
  inputs.insert(inputs.end(), weights.begin(), weights.end());
  node->set_next_edges(torch::autograd::collect_next_edges(inputs));
  Tensor y, hout, kept;
  {
    const at::NoGradGuard no_grad;
    std::tie(y, hout, kept) = trunk_forward_train(x, alive, hidden, done, bullets, mask, weights, geom);
  }
  using torch::autograd::SavedVariable;
  auto save = [](const OptTensor& t) { return SavedVariable(t.has_value() ? *t : Tensor(), false); };
  node->x = SavedVariable(x, false);
  node->alive = save(alive);
  node->hidden = SavedVariable(hidden, false);
  node->done = save(done);
  node->bullets = save(bullets);
  node->mask = save(mask);
  node->kept = SavedVariable(kept, false);
  node->weights.reserve(weights.size());
  for (const Tensor& w : weights) node->weights.emplace_back(w, false);
  node->geom = geom;
  torch::autograd::create_gradient_edge(y, node);
  torch::autograd::create_gradient_edge(hout, node);
  return {y, hout};
}

// ------------------------------------------------------------------ ragged batches

// RaggedBatch.build (yemong/trunk.py): the batch integers of a call, the device arrays [tok_off,
// ship_off(, tile_env_begin, tile_env_ids)] and the share of tile rows in use.  Everything is laid out in
// one pinned buffer and uploaded with one asynchronous copy: from pageable memory the copies waited for
// the kernels of the previous step, and the planning then ran with the device idle.
std::tuple<std::vector<int64_t>, std::vector<Tensor>, double> ragged_build(const Tensor& n_tokens, const Tensor& n_ships, const c10::Device& dev) {
  const Tensor nt = n_tokens.to(at::kCPU, at::kLong).contiguous(), ns = n_ships.to(at::kCPU, at::kLong).contiguous();
  if (nt.dim() != 1 || nt.sizes() != ns.sizes()) throw std::runtime_error("n_tokens and n_ships must be 1-D tensors of equal length");
  const int64_t B = nt.numel();
  const int64_t *t = nt.data_ptr<int64_t>(), *s = ns.data_ptr<int64_t>();
  const c10::cuda::OptionalCUDAGuard guard(dev.is_cuda() ? c10::optional<c10::Device>(dev) : c10::nullopt);
  const int64_t stride = (B + 1 + 3) / 4 * 4;   // 16-byte pieces
  Tensor host = at::empty({4 * stride}, at::TensorOptions().dtype(at::kInt).pinned_memory(dev.is_cuda()));
  int32_t* tok = host.data_ptr<int32_t>();
  int32_t *ship = tok + stride, *tiles = tok + 2 * stride, *ids = tok + 3 * stride;
  int64_t most = 0, least = INT64_MAX;
  tok[0] = ship[0] = 0;
  for (int64_t e = 0; e < B; ++e) {
    if (s[e] > t[e] || s[e] < 0) throw std::runtime_error("each environment needs 0 <= n_ships <= n_tokens");
    most = std::max(most, t[e]);
    least = std::min(least, t[e]);
    tok[e + 1] = tok[e] + (int32_t)t[e];
    ship[e + 1] = ship[e] + (int32_t)s[e];
  }
  int n_tiles = 0;
  const bool planned = B > 0 && most <= 128 && least >= 1;   // the tensor-core engine's ragged tiles
  if (planned) check("bnb_plan_tiles", bnb_plan_tiles(tok, (int)B, tiles, ids, (int)B + 1, &n_tiles));
  const Tensor device = host.slice(0, 0, planned ? 4 * stride : 2 * stride).to(at::TensorOptions().device(dev), /*non_blocking=*/true);
  std::vector<Tensor> offsets{device.slice(0, 0, B + 1), device.slice(0, stride, stride + B + 1)};
  if (planned) {
    offsets.push_back(device.slice(0, 2 * stride, 2 * stride + n_tiles + 1));
    offsets.push_back(device.slice(0, 3 * stride, 3 * stride + B));
  }
  return {{B, 0, 0, most, tok[B], ship[B], n_tiles}, offsets, n_tiles ? tok[B] / (128.0 * n_tiles) : 0.0};
}

// ------------------------------------------------------------------ the ends of the policy step

int pad32(int64_t n) { return (int)((n + 31) / 32 * 32); }

// The first Linear's input rows and one chain's parameters, where the tiled kernel serves the widths.
bool chain_supported(int64_t in_dim, int64_t hidden, int64_t out_dim) {
  return in_dim <= 128 && hidden <= 256 && out_dim <= 128 && bnb::mlp::supported(pad32(in_dim), (int)hidden, pad32(out_dim));
}
bool on16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }
const float* held_parameter(const Tensor& copy, const c10::Device& dev, const char* what, std::vector<Tensor>& held) {
  held.push_back(copy);
  return parameter(copy, dev, what);
}
// A parameter that its kernel reads in pieces of 16 bytes and that may start anywhere: a view into a flat buffer that
// does not is copied, and the copy lives in `held` until the call is queued.
const float* aligned_parameter(const Tensor& t, const c10::Device& dev, const char* what, std::vector<Tensor>& held) {
  const float* p = parameter(t, dev, what);
  return on16(p) ? p : held_parameter(t.detach().clone(), dev, what, held);
}
// One that may be strided (a transposed view).
const float* strided_parameter(const Tensor& t, const c10::Device& dev, const char* what, std::vector<Tensor>& held) {
  return t.is_contiguous() ? parameter(t, dev, what) : held_parameter(t.detach().contiguous(), dev, what, held);
}
// An encoder's first layer and a head's second one may be strided, the latter may start anywhere too.  Kernels read first
// weights of whole 32-column pieces, and an encoder's second one, in 16-byte pieces and refuse them elsewhere; first
// weights of other widths are read element by element.
bnb::mlp::MlpChain chain_of(const std::vector<Tensor>& ps, const c10::Device& dev, const char* what, void* y, int out, int y_ld,
                            std::vector<Tensor>& held) {
  bnb::mlp::MlpChain c{};
  const bool encoder = ps.size() > 5;
  c.w1 = encoder ? strided_parameter(ps[0], dev, what, held) : parameter(ps[0], dev, what);
  c.b1 = parameter(ps[1], dev, what);
  c.g1 = parameter(ps[2], dev, what);
  c.w2 = encoder ? parameter(ps[3], dev, what) : ps[3].is_contiguous() ? aligned_parameter(ps[3], dev, what, held) : strided_parameter(ps[3], dev, what, held);
  c.b2 = encoder ? parameter(ps[4], dev, what) : strided_parameter(ps[4], dev, what, held);
  c.g2 = encoder ? parameter(ps[5], dev, what) : nullptr;
  if ((ps[0].size(1) % 32 == 0 && !on16(c.w1)) || !on16(c.w2))
    throw std::runtime_error(std::string(what) + " parameter is not 16-byte aligned");
  c.y = static_cast<__nv_bfloat16*>(y);
  c.out_store = out;
  c.y_ld = y_ld;
  return c;
}

// bnb_b200::mlp_chain (yemong/_end_ops.py): params = w1, b1, g1, w2, b2[, g2].  active (rows,): only
// those rows are computed, the others are left unwritten.
Tensor mlp_chain(const Tensor& x, const std::vector<Tensor>& params, int precision, const OptTensor& active) {
  const c10::Device dev = x.device();
  if (active.has_value() && (active->numel() != x.size(0) || active->device() != dev))
    throw std::runtime_error("active must hold one element per row, on the rows' device");
  const c10::cuda::CUDAGuard guard(dev);
  const bool bf16 = precision == BNB_BF16, encoder = params.size() > 5;
  const char* what = encoder ? "encoder" : "head";
  const int64_t in_dim = params[0].size(1), hidden = params[0].size(0), out_dim = params[3].size(0);
  const auto stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
  Tensor y = at::empty({x.size(0), out_dim}, x.options().dtype(bf16 ? at::kBFloat16 : at::kFloat));
  if (bf16 && chain_supported(in_dim, hidden, out_dim)) {
    // a head fed bfloat16 tokens reads them as they are
    const bool x16 = x.scalar_type() == at::kBFloat16 && in_dim % 32 == 0;
    Tensor rows = x16 ? contiguous(x) : f32c(x);
    if (x16 && (reinterpret_cast<uintptr_t>(rows.data_ptr()) & 15)) rows = rows.clone();
    const OptTensor on = bytes_of(active);
    bnb::mlp::MlpCall call{};
    call.x = rows.data_ptr();
    call.x_bf16 = x16 ? 1 : 0;
    call.n_rows = (int)rows.size(0);
    call.in_dim = call.w1_ld = (int)in_dim;
    call.active = static_cast<const uint8_t*>(ptr(on));
    std::vector<Tensor> held;
    call.chain[0] = chain_of(params, dev, what, y.data_ptr(), (int)out_dim, (int)out_dim, held);
    check(encoder ? "bnb_encoder_mlp_fwd" : "bnb_head_mlp_fwd", bnb::mlp::run(call, 1, pad32(in_dim), (int)hidden, pad32(out_dim), stream));
    return y;
  }
  // the CUDA-core kernels take weights padded with zeros to multiples of 32
  const Tensor rows = f32c(x);
  const int n = (int)rows.size(0);
  const float *b1 = parameter(params[1], dev, what), *g1 = parameter(params[2], dev, what);
  if (encoder) {
    const int in_pad = pad32(in_dim);
    const Tensor w1 = in_pad == in_dim ? contiguous(params[0].detach()) : at::constant_pad_nd(params[0].detach(), {0, in_pad - in_dim});
    check("bnb_encoder_mlp_fwd",
          bnb_encoder_mlp_fwd(parameter(w1, dev, what), b1, g1, parameter(params[3], dev, what), parameter(params[4], dev, what),
                              parameter(params[5], dev, what), (int)in_dim, in_pad, (int)hidden, (int)out_dim,
                              static_cast<const float*>(rows.data_ptr()), y.data_ptr(), n, precision, stream));
  } else {
    const int out_pad = pad32(out_dim);
    const Tensor w2 = at::constant_pad_nd(params[3].detach(), {0, 0, 0, out_pad - out_dim});
    const Tensor b2 = at::constant_pad_nd(params[4].detach(), {0, out_pad - out_dim});
    check("bnb_head_mlp_fwd",
          bnb_head_mlp_fwd(parameter(params[0], dev, what), b1, g1, parameter(w2, dev, what), parameter(b2, dev, what), (int)in_dim,
                           (int)hidden, (int)out_dim, out_pad, static_cast<const float*>(rows.data_ptr()), y.data_ptr(), n, precision,
                           stream));
  }
  return y;
}

// Whether policy_tail below serves a step of these sizes.
bool tail_supported(int64_t d_model, int64_t n_heads, int64_t ships, const std::vector<int64_t>& heads) {
  if (d_model != 128 || n_heads != 4 || ships < 1 || ships > bnb::tail::MAX_SHIPS) return false;
  for (size_t i = 0; i + 2 < heads.size(); i += 3)   // input, hidden and output width
    if (heads[i] != d_model || heads[i + 1] != 2 * d_model || heads[i + 2] < 1 || heads[i + 2] > 32) return false;
  return heads.size() >= 3 && heads[2] == 12 && chain_supported(d_model, 2 * d_model, 32);
}

// Whether a bfloat16 trunk call with these environments reads the tokens of active bullet slots only
// (the tensor-core kernels compact them; the exact kernels multiply masked values by zero).
bool bullets_compacted(int64_t d_model, int64_t n_heads, int64_t tokens, int64_t slots) {
  BnbBatch b{};
  b.n_envs = 1;
  b.tokens_per_env = b.max_tokens_per_env = b.total_tokens = (int)tokens;
  return slots > 0 && bnb::tensor::supported_batch((int)d_model, (int)n_heads, b) && bnb::tensor::supported_bullets(b, (int)slots);
}

// The value columns that the win head's outputs go to, as indexing a tensor takes them: from the end when negative,
// refused outside, and each an output that the win head has.
std::vector<uint8_t> value_columns(const std::vector<int64_t>& win_cols, int64_t value_width, int64_t win_width) {
  auto refuse = [](int64_t i, int64_t size) {
    throw py::index_error("index " + std::to_string(i) + " is out of bounds for a last dimension of size " + std::to_string(size));
  };
  std::vector<uint8_t> cols;
  for (int64_t k : win_cols) {
    if (k < -value_width || k >= value_width) refuse(k, value_width);
    if ((int64_t)cols.size() >= win_width) refuse((int64_t)cols.size(), win_width);
    cols.push_back((uint8_t)(k < 0 ? k + value_width : k));
  }
  return cols;
}

void expect_shape(const Tensor& t, c10::IntArrayRef want, const char* what) {
  if (t.defined() && t.sizes() == want) return;
  std::ostringstream s;
  s << what << " must have shape " << want << ", got ";
  if (t.defined()) s << t.sizes();
  else s << "nothing";
  throw std::runtime_error(s.str());
}
// What the kernels of policy_tail take on trust: the sizes of everything they read.
void check_tail(const Tensor& x, const Tensor& alive, const Tensor& team, const Tensor& uniforms, const std::vector<Tensor>& heads,
                const std::vector<Tensor>& pma, int64_t N) {
  if (x.dim() != 3 || x.size(2) != 128 || x.scalar_type() != at::kBFloat16) throw std::runtime_error("expected bfloat16 tokens of shape (B, N+M, 128)");
  const int64_t B = x.size(0), NM = x.size(1), D = x.size(2);
  if (N < 1 || N > NM || N > bnb::tail::MAX_SHIPS)
    throw std::runtime_error(std::to_string(N) + " ships of " + std::to_string(NM) + " tokens are not served by the native end of the policy step");
  expect_shape(uniforms, {B * N, 3}, "uniforms");
  if (uniforms.scalar_type() != at::kFloat || !uniforms.is_contiguous()) throw std::runtime_error("uniforms must be contiguous float32");
  if (heads.size() != (pma.empty() ? 15u : 20u) || (!pma.empty() && pma.size() != 4)) throw std::runtime_error("expected five parameters per head and four of TeamPMA");
  for (size_t h = 0; h < heads.size(); h += 5) {
    const int64_t out = heads[h + 3].dim() == 2 ? heads[h + 3].size(0) : 0;
    if (out < 1 || out > 32 || (h == 0 && out != 12)) throw std::runtime_error("a head of this width is not served by the native end of the policy step");
    expect_shape(heads[h], {2 * D, D}, "a head's first weight");
    expect_shape(heads[h + 1], {2 * D}, "a head's first bias");
    expect_shape(heads[h + 2], {2 * D}, "a head's norm");
    expect_shape(heads[h + 3], {out, 2 * D}, "a head's second weight");
    expect_shape(heads[h + 4], {out}, "a head's second bias");
  }
  if (!pma.empty()) {
    expect_shape(pma[0], {2, D}, "TeamPMA's seeds");
    expect_shape(pma[1], {3 * D, D}, "TeamPMA's in_proj");
    expect_shape(pma[2], {D, D}, "TeamPMA's out_proj");
    expect_shape(pma[3], {D}, "TeamPMA's norm");
    expect_shape(alive, {B, NM}, "alive");
    if (!team.defined() || team.dim() != 2 || team.size(0) != B || team.size(1) < N) {
      std::ostringstream s;
      s << "team_id must have shape (" << B << ", " << N << ") or more columns";
      throw std::runtime_error(s.str());
    }
  }
}
void check_tail_devices(const Tensor& x, std::initializer_list<const Tensor*> others) {
  if (!x.is_cuda()) throw std::runtime_error("x is on " + x.device().str() + "; the policy's kernels run on CUDA only (sm_100a)");
  for (const Tensor* t : others)
    if (t->defined() && t->device() != x.device())
      throw std::runtime_error("an input of the policy step is on " + t->device().str() + ", the tokens on " + x.device().str());
}

// bnb_b200::policy_tail (yemong/_end_ops.py): everything of the rollout step behind the trunk.  x
// (B, N+M, 128) bfloat16, alive (B, N+M) and team_id (B, N or more columns) only read with pma, heads = five parameters each of the action, next-state and value head [and the
// win head], pma = seeds, in_proj, out_proj, norm (empty: no team value), win_cols the value columns the
// win head fills.
std::tuple<Tensor, Tensor, Tensor, Tensor> policy_tail(const Tensor& x_in, const OptTensor& alive_in, const OptTensor& team_in,
                                                       const Tensor& uniforms, const std::vector<Tensor>& heads,
                                                       const std::vector<Tensor>& pma, const std::vector<int64_t>& win_cols, int64_t N) {
  Tensor team = team_in.has_value() ? *team_in : Tensor();
  Tensor flags = alive_in.has_value() ? *alive_in : Tensor();
  check_tail(x_in, flags, team, uniforms, heads, pma, N);
  const int64_t K = heads[13].size(0), P = heads[8].size(0), W = pma.empty() ? 0 : (int64_t)win_cols.size();
  const std::vector<uint8_t> cols = W > 0 ? value_columns(win_cols, K, heads[18].size(0)) : std::vector<uint8_t>();
  if (W == 0) team = flags = Tensor();   // only read with a win head
  check_tail_devices(x_in, {&uniforms, &flags, &team});
  const c10::Device dev = x_in.device();
  const c10::cuda::CUDAGuard guard(dev);
  const auto stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
  const Tensor x = contiguous(x_in);
  const OptTensor alive = W > 0 ? bytes_of(flags) : OptTensor();
  if (team.defined()) {
    if (team.scalar_type() != at::kLong && team.scalar_type() != at::kInt) team = team.to(at::kInt);
    if (team.stride(1) != 1 || team.stride(0) > INT32_MAX) team = team.contiguous();
  }
  const int64_t B = x.size(0), NM = x.size(1), D = x.size(2);
  bnb::tail::Ships s{};
  s.x = static_cast<const __nv_bfloat16*>(x.data_ptr());
  s.alive = static_cast<const uint8_t*>(ptr(alive));
  if (team.defined()) {
    s.team_id = team.data_ptr();
    s.team_is_64 = team.scalar_type() == at::kLong ? 1 : 0;
    s.team_ld = (int)team.stride(0);
  }
  s.n_envs = (int)B;
  s.ships = (int)N;
  s.tokens = (int)NM;

  const auto bf = x.options();
  Tensor logits = at::empty({B, N, 12}, bf), pred = at::empty({B, N, P}, bf), value = at::empty({B, N, K}, bf);
  Tensor action = at::empty({B, N, 3}, bf.dtype(at::kLong)), logprob = at::empty({B, N}, bf);

  std::vector<Tensor> held;
  auto five = [&](int i) { return std::vector<Tensor>(heads.begin() + 5 * i, heads.begin() + 5 * i + 5); };
  bnb::mlp::MlpCall call{};
  call.x = x.data_ptr();
  call.x_bf16 = 1;
  call.n_rows = (int)(B * N);
  call.in_dim = call.w1_ld = (int)D;
  call.group_rows = (int)N;
  call.group_stride = (int)NM;
  call.chain[0] = chain_of(five(0), dev, "head", logits.data_ptr(), 12, 12, held);
  call.chain[1] = chain_of(five(1), dev, "head", pred.data_ptr(), (int)P, (int)P, held);
  call.chain[2] = chain_of(five(2), dev, "head", value.data_ptr(), (int)K, (int)K, held);
  Tensor win, rows, fold;
  bnb::mlp::MlpCall wc{};   // the win head over the teams' rows, in the heads' launch
  if (W > 0) {
    rows = at::empty({B * 2, D}, bf);
    win = at::empty({B * 2, W}, bf);
    fold = at::empty({(int64_t)bnb::tail::scratch_bytes()}, bf.dtype(at::kByte));
    const float *in_proj = parameter(pma[1], dev, "TeamPMA"), *out_proj = parameter(pma[2], dev, "TeamPMA");
    if (!on16(in_proj) || !on16(out_proj)) check("bnb_team_pma_fwd", BNB_ERR_MISALIGNED);
    check("bnb_team_pma_fwd", bnb::tail::team_rows(s, aligned_parameter(pma[0], dev, "TeamPMA", held), in_proj, out_proj,
                                                   aligned_parameter(pma[3], dev, "TeamPMA", held), fold.data_ptr(),
                                                   static_cast<__nv_bfloat16*>(rows.data_ptr()), stream));
    wc.x = rows.data_ptr();
    wc.x_bf16 = 1;
    wc.n_rows = (int)(B * 2);
    wc.in_dim = wc.w1_ld = (int)D;
    wc.chain[0] = chain_of(five(3), dev, "head", win.data_ptr(), (int)W, (int)W, held);
  }
  check("bnb_head_mlp_fwd", bnb::mlp::run(call, 3, (int)D, (int)(2 * D), 32, stream, W > 0 ? &wc : nullptr, 1));
  check("bnb_action_dist_fwd", bnb::tail::finish(s, static_cast<const __nv_bfloat16*>(logits.data_ptr()), static_cast<const float*>(uniforms.data_ptr()),
                                                 static_cast<int64_t*>(action.data_ptr()), static_cast<__nv_bfloat16*>(logprob.data_ptr()),
                                                 W > 0 ? static_cast<const __nv_bfloat16*>(win.data_ptr()) : nullptr, (int)W, cols.data(),
                                                 static_cast<__nv_bfloat16*>(value.data_ptr()), (int)K, stream));
  return {action, logprob, value, pred};
}

}  // namespace

PYBIND11_MODULE(_host_path, m) {
  m.def("trunk_params", &trunk_params);
  m.def("keep_activations", [](const c10::Device& dev, const std::vector<int64_t>& geom, int64_t d_model, int64_t n_bullets) {
    return keep_activations(dev, Geometry(geom), d_model, n_bullets);
  });
  m.def("trunk_backward", &trunk_backward);
  m.def("trunk_forward_train", &trunk_forward_train);
  m.def("trunk_train", torch::wrap_pybind_function(trunk_train));   // saved-tensor hooks may raise
  m.def("ragged_build", &ragged_build);
  m.def("mlp_chain", &mlp_chain);
  m.def("policy_tail", &policy_tail);
  m.def("tail_supported", &tail_supported);
  m.def("bullets_compacted", &bullets_compacted);
  m.def("trunk_forward", &trunk_forward);
}
