// PyTorch binding: one C call per operator.
//
// The operators are small (a few microseconds of GPU work for a short cache), so what the host does around a launch is
// part of their time: through ctypes an operator spent 10-20 us in Python on argument conversion, device guards, stream
// look-ups and one torch.empty per output (96 us per layer pair of a streamed frame, against about 100 us of kernels at the
// start of a sequence).  These functions are plain CPython vector-call functions over at::Tensor: they check, allocate
// from PyTorch's caching allocator, take the current stream and launch.  The computing stays behind the C ABI of
// libgct_b200.so, which this module is linked against; nothing here includes a kernel.
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <mutex>

#include "gct_common.h"

namespace {

using at::Tensor;
using gct::kHeadDim;

__attribute__((used)) const char kBuiltFor[] = "binding built for " GCT_BUILT_FOR ";";      // looked for by build.py

PyObject* g_error_class = nullptr;      // _lib.GctError(code, message)

// An exception of the given Python type, thrown through C++ frames and set at the boundary.
struct Raise {
  PyObject* type;
  std::string msg;
};
[[noreturn]] void value_error(const std::string& m) { throw Raise{PyExc_ValueError, m}; }
[[noreturn]] void type_error(const std::string& m) { throw Raise{PyExc_TypeError, m}; }
[[noreturn]] void runtime_error(const std::string& m) { throw Raise{PyExc_RuntimeError, m}; }
struct Failed {                          // a C ABI status code other than GCT_OK
  int code;
};
void check(int rc) {
  if (rc != GCT_OK) throw Failed{rc};
}

// What may wait runs without the interpreter lock, as the ctypes calls and PyTorch's own operators do: a launch while the
// stream's queue is full, a plan behind an upload eight plans back, a cudaMalloc.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};
template <typename F>
auto unlocked(F&& f) {
  WithoutGil free_others;
  return f();
}

template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const Raise& r) {
    PyErr_SetString(r.type, r.msg.c_str());
  } catch (const Failed& e) {
    const char* text = gct_last_error();
    if (e.code == GCT_ERR_POOL_EXHAUSTED || e.code == GCT_ERR_UNDERFLOW) {
      PyErr_SetString(PyExc_AssertionError, text);      // the reference signals these with `assert`
    } else if (g_error_class != nullptr) {
      PyObject* exc = PyObject_CallFunction(g_error_class, "is", e.code, text);
      if (exc != nullptr) {
        PyErr_SetObject(g_error_class, exc);
        Py_DECREF(exc);
      }
    } else {
      PyErr_SetString(PyExc_RuntimeError, text);
    }
  } catch (python_error& e) {
    e.restore();
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());      // what PyTorch makes of its own: OutOfMemoryError among them
  }
  return nullptr;
}

void need(Py_ssize_t got, Py_ssize_t want, const char* who) {
  if (got != want) type_error(std::string(who) + ": wrong number of arguments");
}
const Tensor& tensor(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) type_error(std::string(name) + " must be a tensor");
  return THPVariable_Unpack(o);
}
const Tensor* optional_tensor(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor(o, name); }
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
gct_mgr_t* manager(PyObject* o) { return reinterpret_cast<gct_mgr_t*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLong(o))); }

void need_cuda(const Tensor& t, const char* name) {
  if (!t.is_cuda()) runtime_error(std::string(name) + " must be a CUDA tensor: the B200 backend has no CPU path");
}
void need_beside(const Tensor& t, const char* name, const Tensor& rows) {
  need_cuda(t, name);
  if (t.device() != rows.device()) value_error(std::string(name) + " lives on " + t.device().str() + ", the rows on " + rows.device().str());
}
int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return GCT_F32;
  if (t.scalar_type() == at::kBFloat16) return GCT_BF16;
  type_error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + ": the B200 backend takes float32 or bfloat16");
}
Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const Tensor& like) {
  return at::detail::empty_cuda(size, dtype, like.device(), c10::nullopt);
}
cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
const __nv_bfloat16* bf16(const Tensor& t) { return static_cast<const __nv_bfloat16*>(t.data_ptr()); }

// Status word of the operators that have no manager, one per device for the life of the process.
int* status_of(const Tensor& like) {
  static std::atomic<int*> words[64];
  static std::mutex mu;
  const int dev = like.device().index();
  if (dev < 0 || dev >= 64) value_error("device ordinal out of range");
  int* p = words[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    std::lock_guard<std::mutex> lock(mu);
    p = words[dev].load(std::memory_order_relaxed);
    if (p == nullptr) {
      Tensor* word = new Tensor(at::zeros({64}, at::TensorOptions().dtype(at::kInt).device(like.device())));
      p = word->data_ptr<int>();
      words[dev].store(p, std::memory_order_release);
    }
  }
  return p;
}

// The four q/k norm parameters (null: none), from Python's arguments.
struct Norm {
  const Tensor* t[4];
  explicit Norm(PyObject* const* o) {
    for (int i = 0; i < 4; ++i) t[i] = optional_tensor(o[i], "a norm parameter");
  }
};

// LayerNorm parameters and rotation table as the prologue kernel takes them.  `keep` holds tensors that had to be
// converted (a norm parameter that is neither fp32 nor bf16, or not of the dtype of the others) until the launch is queued.
struct NormRope {
  Tensor keep[5];
  // Everything has to lie on the device of the rows: the kernel gets addresses.
  void fill(gct::PrepLaunch* p, const Norm& norm, const Tensor* c, int64_t mode, const Tensor& rows) {
    const Tensor* const* t = norm.t;
    static const char* names[4] = {"q_norm_w", "q_norm_b", "k_norm_w", "k_norm_b"};
    bool all_bf16 = true;
    for (int i = 0; i < 4; ++i) {
      if (t[i] != nullptr) {
        need_beside(*t[i], names[i], rows);
        if (t[i]->numel() != kHeadDim) value_error(std::string(names[i]) + " must have 64 elements");
        all_bf16 &= t[i]->scalar_type() == at::kBFloat16;
      }
    }
    if ((t[0] == nullptr) != (t[1] == nullptr) || (t[2] == nullptr) != (t[3] == nullptr)) {
      gct::set_error("norm weight and bias must come together");
      throw Failed{GCT_ERR_INVALID};
    }
    const void* ptr[4] = {nullptr, nullptr, nullptr, nullptr};
    for (int i = 0; i < 4; ++i) {
      if (t[i] == nullptr) continue;
      const at::ScalarType want = all_bf16 ? at::kBFloat16 : at::kFloat;
      // the launcher takes 16-byte aligned parameters only: a bf16 one at another address (a slice of a flat buffer) is copied,
      // as the conversion to fp32 once did; an fp32 one there was always refused and is
      const bool in_place = t[i]->is_contiguous() && (want == at::kFloat || (reinterpret_cast<uintptr_t>(t[i]->data_ptr()) & 15) == 0);
      if (t[i]->scalar_type() == want && in_place) {
        ptr[i] = t[i]->data_ptr();
      } else {
        keep[i] = t[i]->detach().to(want).clone(at::MemoryFormat::Contiguous);
        ptr[i] = keep[i].data_ptr();
      }
    }
    p->qn_w = ptr[0];
    p->qn_b = ptr[1];
    p->kn_w = ptr[2];
    p->kn_b = ptr[3];
    p->norm_dtype = all_bf16 ? GCT_BF16 : GCT_F32;
    p->rope_mode = static_cast<int>(mode);
    if (c == nullptr || mode == GCT_ROPE_NONE) return;
    need_beside(*c, "rope_cs", rows);
    const bool is_complex = c->scalar_type() == at::kComplexFloat || c->scalar_type() == at::kComplexDouble;
    if (c->numel() < static_cast<int64_t>(p->tokens_per_frame) * (is_complex ? 32 : 64)) value_error("rope_cs holds too few rows");
    Tensor table = c->is_conj() ? c->resolve_conj() : *c;
    if (mode == GCT_ROPE_2D || !(is_complex || c->scalar_type() == at::kFloat)) {
      if (c->scalar_type() != at::kFloat) table = is_complex ? at::view_as_real(c->to(at::kComplexFloat)) : c->to(at::kFloat);
    }
    if (!table.is_contiguous()) table = table.contiguous();
    p->rope_f64 = table.scalar_type() == at::kComplexDouble;
    p->rope_cs = table.data_ptr();
    keep[4] = std::move(table);
  }
};

void fill_qkv(gct::PrepLaunch* p, const Tensor& qkv, int64_t heads) {
  const size_t esz = qkv.element_size();
  const int64_t C = heads * kHeadDim;
  if (qkv.stride(0) < 3 * C) {
    gct::set_error("qkv: row stride smaller than 3*H*64");
    throw Failed{GCT_ERR_INVALID};
  }
  const uint8_t* base = static_cast<const uint8_t*>(qkv.data_ptr());
  p->q_src = base;
  p->k_src = base + C * esz;
  p->v_src = base + 2 * C * esz;
  p->src_dtype_qk = p->src_dtype_v = dtype_code(qkv);
  p->src_token_stride = qkv.stride(0);
  p->src_head_stride = kHeadDim;
}

struct Qkv {
  Tensor q, k, v;
};
Qkv prep(Tensor qkv, int64_t heads, int64_t tokens_per_frame, const Norm& norm, const Tensor* cs, int64_t mode) {
  need_cuda(qkv, "qkv");
  if (qkv.dim() != 2 || qkv.size(1) != 3 * heads * kHeadDim) value_error("qkv must be [tokens, 3*H*64]");
  if (qkv.stride(1) != 1) qkv = qkv.contiguous();
  c10::cuda::CUDAGuard guard(qkv.device());
  gct::PrepLaunch p;
  fill_qkv(&p, qkv, heads);
  p.tokens = static_cast<int>(qkv.size(0));
  p.tokens_per_frame = static_cast<int>(tokens_per_frame);
  p.heads = static_cast<int>(heads);
  NormRope nr;
  nr.fill(&p, norm, cs, mode, qkv);
  Qkv r{empty({qkv.size(0), heads, kHeadDim}, at::kBFloat16, qkv), empty({qkv.size(0), heads, kHeadDim}, at::kBFloat16, qkv),
        empty({qkv.size(0), heads, kHeadDim}, at::kBFloat16, qkv)};
  p.q_out = const_cast<__nv_bfloat16*>(bf16(r.q));
  p.k_out = const_cast<__nv_bfloat16*>(bf16(r.k));
  p.v_out = const_cast<__nv_bfloat16*>(bf16(r.v));
  check(gct::launch_prep(p, stream_of(qkv)));
  return r;
}

// prep_qkv(qkv, heads, tokens_per_frame, qw, qb, kw, kb, rope_cs, rope_mode) -> (q, k, v)
PyObject* py_prep_qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 9, "prep_qkv");
    const Tensor &qkv = tensor(a[0], "qkv"), *cs = optional_tensor(a[7], "rope_cs");
    const int64_t heads = integer(a[1]), tokens_per_frame = integer(a[2]), mode = integer(a[8]);
    const Norm norm(a + 3);
    Qkv r = unlocked([&] { return prep(qkv, heads, tokens_per_frame, norm, cs, mode); });
    PyObject* out = PyTuple_New(3);
    if (out == nullptr) throw python_error();
    PyTuple_SET_ITEM(out, 0, wrap(std::move(r.q)));
    PyTuple_SET_ITEM(out, 1, wrap(std::move(r.k)));
    PyTuple_SET_ITEM(out, 2, wrap(std::move(r.v)));
    return out;
  });
}

// Split-KV partials come from the caching allocator, and only when a call splits: calls on several streams or threads
// do not share them, and the allocator takes them back when the call returns.
constexpr int kDenseMaxSplits = 8;
Tensor dense(const Tensor& q, const Tensor& k, const Tensor& v, Tensor out) {
  const Tensor* t[3] = {&q, &k, &v};
  static const char* names[3] = {"q", "k", "v"};
  for (int i = 0; i < 3; ++i) {
    need_beside(*t[i], names[i], q);
    if (t[i]->scalar_type() != at::kBFloat16 || t[i]->dim() != 4 || t[i]->size(3) != kHeadDim || t[i]->stride(3) != 1)
      value_error(std::string(names[i]) + " must be bf16 [B, N, H, 64] with contiguous head_dim");
  }
  const int64_t B = q.size(0), Nq = q.size(1), H = q.size(2), Nkv = k.size(1);
  if (k.sizes() != v.sizes() || k.size(0) != B || k.size(2) != H) value_error("k/v shape mismatch");
  c10::cuda::CUDAGuard guard(q.device());
  if (!out.defined()) out = empty({B, Nq, H, kHeadDim}, at::kBFloat16, q);
  gct::DensePlan plan;
  check(gct::dense_attention_plan(static_cast<int>(B), static_cast<int>(Nq), static_cast<int>(Nkv), static_cast<int>(H), kDenseMaxSplits, &plan));
  const int64_t rows = B * Nq * H;
  Tensor scratch;
  float* part = nullptr;
  if (plan.splits > 1) {
    scratch = empty({plan.splits * rows * (kHeadDim + 1)}, at::kFloat, q);
    part = scratch.data_ptr<float>();
  }
  const int64_t qs[3] = {q.stride(0), q.stride(1), q.stride(2)}, ks[3] = {k.stride(0), k.stride(1), k.stride(2)},
                vs[3] = {v.stride(0), v.stride(1), v.stride(2)};
  check(gct::dense_attention_run(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), static_cast<int>(B), static_cast<int>(Nq),
                                 static_cast<int>(Nkv), static_cast<int>(H), qs, ks, vs, plan, part,
                                 part == nullptr ? nullptr : part + plan.splits * rows * kHeadDim, status_of(q), stream_of(q)));
  return out;
}

// dense_attention(q, k, v, out | None) -> out
PyObject* py_dense_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 4, "dense_attention");
    const Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k"), &v = tensor(a[2], "v"), *out = optional_tensor(a[3], "out");
    return wrap(unlocked([&] { return dense(q, k, v, out == nullptr ? Tensor() : *out); }));
  });
}

// operator_status(device_index) -> value of the status word; waits for the device
PyObject* py_operator_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 1, "operator_status");
    const c10::Device dev(c10::kCUDA, static_cast<c10::DeviceIndex>(integer(a[0])));
    c10::cuda::CUDAGuard guard(dev);
    const Tensor like = at::detail::empty_cuda({0}, at::kInt, dev, c10::nullopt);
    int* word = status_of(like);
    return PyLong_FromLong(at::from_blob(word, {1}, at::TensorOptions().dtype(at::kInt).device(dev)).item<int>());
  });
}

// ---- cache manager ----------------------------------------------------------------------------

// [tokens, H, 64] rows of one frame, contiguous
Tensor frame_rows(const Tensor& t, const char* name, const gct_mgr_config_t& cfg, int64_t device) {
  if (!t.is_cuda() || t.device().index() != device)
    value_error(std::string(name) + " lives on " + t.device().str() + ", the cache on cuda:" + std::to_string(device));
  if (t.dim() != 3 || t.size(1) != cfg.num_heads || t.size(2) != kHeadDim)
    value_error(std::string(name) + " must be [tokens, " + std::to_string(cfg.num_heads) + ", 64]");
  return t.is_contiguous() ? t : t.contiguous();
}

// append(manager, device, block, k, v)
PyObject* py_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "append");
    gct_mgr_t* m = manager(a[0]);
    const int64_t dev = integer(a[1]);
    const Tensor k = frame_rows(tensor(a[3], "k"), "k", gct::mgr_config(m), dev), v = frame_rows(tensor(a[4], "v"), "v", gct::mgr_config(m), dev);
    if (k.size(0) != gct::mgr_config(m).tokens_per_frame || v.size(0) != k.size(0)) value_error("k and v must hold the tokens of one frame");
    c10::cuda::CUDAGuard guard(k.device());
    const int block = static_cast<int>(integer(a[2]));
    check(unlocked([&] { return gct_mgr_append(m, block, k.data_ptr(), dtype_code(k), v.data_ptr(), dtype_code(v), stream_of(k)); }));
    Py_RETURN_NONE;
  });
}

Tensor append_fused(gct_mgr_t* m, int64_t device, int64_t block, Tensor qkv, const Norm& norm, const Tensor* cs, int64_t mode, Tensor q_out) {
  const gct_mgr_config_t& cfg = gct::mgr_config(m);
  const int64_t T = cfg.tokens_per_frame, H = cfg.num_heads;
  if (qkv.dim() != 2 || qkv.size(0) != T || qkv.size(1) != 3 * H * kHeadDim)
    value_error("qkv must be [" + std::to_string(T) + ", " + std::to_string(3 * H * kHeadDim) + "]");
  if (!qkv.is_cuda() || qkv.device().index() != device) value_error("qkv lives on " + qkv.device().str() + ", the cache on cuda:" + std::to_string(device));
  if (qkv.stride(1) != 1) qkv = qkv.contiguous();
  c10::cuda::CUDAGuard guard(qkv.device());
  gct::PrepLaunch p;
  fill_qkv(&p, qkv, H);
  p.tokens_per_frame = static_cast<int>(T);
  NormRope nr;
  nr.fill(&p, norm, cs, mode, qkv);
  if (!q_out.defined()) q_out = empty({T, H, kHeadDim}, at::kBFloat16, qkv);
  p.q_out = static_cast<__nv_bfloat16*>(q_out.data_ptr());
  check(gct::mgr_append(m, static_cast<int>(block), p, stream_of(qkv)));
  return q_out;
}

// append_fused(manager, device, block, qkv, qw, qb, kw, kb, rope_cs, rope_mode, q_out | None) -> q
PyObject* py_append_fused(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 11, "append_fused");
    const Tensor &qkv = tensor(a[3], "qkv"), *cs = optional_tensor(a[8], "rope_cs"), *q_out = optional_tensor(a[10], "q_out");
    const int64_t device = integer(a[1]), block = integer(a[2]), mode = integer(a[9]);
    gct_mgr_t* m = manager(a[0]);
    const Norm norm(a + 4);
    return wrap(unlocked([&] { return append_fused(m, device, block, qkv, norm, cs, mode, q_out == nullptr ? Tensor() : *q_out); }));
  });
}

struct Attended {
  Tensor out, lse;
};
// The page table is planned at block 0 and reused by the other blocks of the frame; `planned`: the caller has done it.
Attended attend(gct_mgr_t* m, int64_t device, int64_t block, const Tensor& q_in, bool want_lse, bool planned = false) {
  const gct_mgr_config_t& cfg = gct::mgr_config(m);
  const Tensor q = frame_rows(q_in, "q", cfg, device);
  c10::cuda::CUDAGuard guard(q.device());
  cudaStream_t s = stream_of(q);
  if (block == 0 && !planned) check(gct_mgr_plan(m, 0, -1, s));
  Attended r;
  r.out = empty(q.sizes(), at::kBFloat16, q);
  if (want_lse) r.lse = empty({q.size(0), q.size(1)}, at::kFloat, q);
  check(gct_mgr_attention(m, static_cast<int>(block), q.data_ptr(), dtype_code(q), static_cast<int>(q.size(0)), r.out.data_ptr(),
                          want_lse ? r.lse.data_ptr<float>() : nullptr, s));
  return r;
}

// attention(manager, device, block, q, want_lse, plan | None) -> out | (out, lse) | None (nothing cached yet)
// plan: called at block 0 in place of the plan over all visible pages.
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 6, "attention");
    gct_mgr_t* m = manager(a[0]);
    int64_t stats[6];
    check(gct_mgr_stats(m, static_cast<int>(integer(a[2])), stats));
    if (stats[0] == 0) Py_RETURN_NONE;
    const bool want_lse = PyObject_IsTrue(a[4]) == 1;
    const Tensor& q = tensor(a[3], "q");
    const int64_t device = integer(a[1]), block = integer(a[2]);
    const bool planned = a[5] != Py_None;
    if (planned && block == 0) {
      frame_rows(q, "q", gct::mgr_config(m), device);      // a tensor that is refused is refused before the plan changes
      PyObject* done = PyObject_CallNoArgs(a[5]);
      if (done == nullptr) throw python_error();
      Py_DECREF(done);
    }
    Attended r = unlocked([&] { return attend(m, device, block, q, want_lse, planned); });
    if (!want_lse) return wrap(std::move(r.out));
    PyObject* out = PyTuple_New(2);
    if (out == nullptr) throw python_error();
    PyTuple_SET_ITEM(out, 0, wrap(std::move(r.out)));
    PyTuple_SET_ITEM(out, 1, wrap(std::move(r.lse)));
    return out;
  });
}

// The bookkeeping calls of every layer of every frame.
PyObject* py_append_bookkeeping(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "append_bookkeeping");
    check(gct_mgr_append_bookkeeping(manager(a[0]), static_cast<int>(integer(a[1]))));
    Py_RETURN_NONE;
  });
}
PyObject* py_evict(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "evict");
    check(gct_mgr_evict(manager(a[0]), static_cast<int>(integer(a[1])), static_cast<int>(integer(a[2]))));
    Py_RETURN_NONE;
  });
}
PyObject* py_rollback(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "rollback");
    check(gct_mgr_rollback(manager(a[0]), static_cast<int>(integer(a[1]))));
    Py_RETURN_NONE;
  });
}

// ---- whole layers -------------------------------------------------------------------------------
//
// The streaming forward of the frame attention layer and of the global block in one call each: this library's kernels
// around the library GEMMs of the Linear layers.  As modules, a layer pair was some fifty launches and as many Python
// round trips (0.8 ms of host time for 0.2-0.6 ms of GPU work): casts of activations and norm parameters for autocast, the
// rotation tables element by element, norms, scales and sums one operation each.  The caller (block.py) makes sure that the
// modules are the stock ones; what is left to check here returns NotImplemented, and the module code runs instead.

PyObject* g_parameter_class = nullptr;

struct NotStock {};
// A plain tensor or parameter, or nothing.  Not plain: tensor subclasses, lazily conjugated or negated views (their memory holds
// other values), and tensors that carry a forward-mode tangent (the modules propagate it through the residual sums).
const Tensor* stock(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (!THPVariable_CheckExact(o) && reinterpret_cast<PyObject*>(Py_TYPE(o)) != g_parameter_class) throw NotStock{};
  const Tensor& t = THPVariable_Unpack(o);
  if (t.is_conj() || t.is_neg() || t._fw_grad(0).defined()) throw NotStock{};
  return &t;
}
bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// bf16 is what the Linear layers compute in: under autocast whatever the parameters are, else only if all of it is bf16.
// A parameter on another device than x is the modules' to refuse.
struct Precision {
  bool autocast;
  c10::Device device;
  Precision(const Tensor& x) : device(x.device()) {
    autocast = at::autocast::is_autocast_enabled(at::kCUDA);
    const bool known = x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16;
    if (!known || (autocast ? at::autocast::get_autocast_dtype(at::kCUDA) != at::kBFloat16 : x.scalar_type() != at::kBFloat16)) throw NotStock{};
  }
  // a Linear parameter in bf16, from autocast's own cache where it keeps one
  Tensor linear(PyObject* o) const {
    const Tensor* t = stock(o);
    if (t == nullptr) return Tensor();
    if (t->device() != device) throw NotStock{};
    if (t->scalar_type() == at::kBFloat16) return *t;
    if (!autocast || t->scalar_type() != at::kFloat) throw NotStock{};
    return at::autocast::cached_cast(at::kBFloat16, *t, c10::kCUDA);
  }
  // a norm or scale parameter of `n` values as it is
  const Tensor* row(PyObject* o, int64_t n) const {
    const Tensor* t = stock(o);
    if (t == nullptr) return nullptr;
    const bool bf = t->scalar_type() == at::kBFloat16;
    if (t->device() != device || t->numel() != n || !t->is_contiguous() || !(bf || (autocast && t->scalar_type() == at::kFloat)) || !aligned16(*t)) throw NotStock{};
    return t;
  }
};

Tensor linear(const Tensor& rows, const Tensor& w, const Tensor& b) {
  return b.defined() ? at::addmm(b, rows, w.t()) : at::mm(rows, w.t());
}

// Norm of the rows of x as bf16; with y, of the sum x + gamma * y, which is returned in *sum.  The kernel takes dense rows.
Tensor residual_norm(const Tensor& x, const Tensor* y, const Tensor* gamma, Tensor* sum, const Tensor* w, const Tensor* b, double eps) {
  if (!x.is_contiguous() || (y != nullptr && (!y->is_contiguous() || y->sizes() != x.sizes()))) runtime_error("residual norm: rows must be contiguous");
  gct::RowLaunch p;
  p.rows = x.size(0);
  p.cols = static_cast<int>(x.size(1));
  p.x = x.data_ptr();
  p.x_dtype = dtype_code(x);
  if (y != nullptr) {
    p.y = bf16(*y);
    if (gamma != nullptr) {
      p.gamma = gamma->data_ptr();
      p.gamma_dtype = dtype_code(*gamma);
    }
    const bool f32 = p.x_dtype == GCT_F32 || (gamma != nullptr && p.gamma_dtype == GCT_F32);
    *sum = empty(x.sizes(), f32 ? at::kFloat : at::kBFloat16, x);
    p.sum_out = sum->data_ptr();
    p.sum_dtype = f32 ? GCT_F32 : GCT_BF16;
  }
  Tensor out;
  if (w != nullptr) {
    out = empty(x.sizes(), at::kBFloat16, x);
    p.norm_w = w->data_ptr();
    p.norm_b = b->data_ptr();
    p.norm_dtype = dtype_code(*w);
    p.eps = static_cast<float>(eps);
    p.norm_out = static_cast<__nv_bfloat16*>(out.data_ptr());
  }
  check(gct::launch_residual_norm(p, stream_of(x)));
  return out;
}

// Rotation table for the `tokens` tokens of x from what the modules pass as positions.
Tensor rotation(const Tensor* p, int64_t mode, double base, int64_t tokens, const Tensor& x) {
  if (mode == GCT_ROPE_NONE || p == nullptr) return Tensor();
  if (p->device() != x.device()) throw NotStock{};
  if (mode == GCT_ROPE_3D) {
    if ((p->scalar_type() != at::kComplexFloat && p->scalar_type() != at::kComplexDouble) || p->numel() != tokens * 32) throw NotStock{};
    return *p;
  }
  if (p->scalar_type() != at::kLong || p->dim() != 3 || p->size(0) < 1 || p->size(1) != tokens || p->size(2) != 2) throw NotStock{};
  Tensor cs = empty({tokens, 32, 2}, at::kFloat, *p);
  check(gct::launch_rope2d_positions(p->data_ptr<int64_t>(), p->stride(1), p->stride(2), static_cast<int>(tokens), static_cast<float>(base),
                                     cs.data_ptr<float>(), stream_of(*p)));
  return cs;
}

template <typename F>
PyObject* layer(F&& f) {
  return guarded([&]() -> PyObject* {
    try {
      return f();
    } catch (const NotStock&) {
      Py_RETURN_NOTIMPLEMENTED;
    }
  });
}

// frame_layer(x, (qkv_w, qkv_b, qn_w, qn_b, kn_w, kn_b, proj_w, proj_b), heads, pos, rope_mode, rope_base) -> y
PyObject* py_frame_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return layer([&]() -> PyObject* {
    need(n, 6, "frame_layer");
    const Tensor* px = stock(a[0]);
    if (px == nullptr || !px->is_cuda() || px->dim() != 3 || PyTuple_GET_SIZE(a[1]) != 8) throw NotStock{};
    const Precision prec(*px);
    PyObject* const* w = &PyTuple_GET_ITEM(a[1], 0);
    const int64_t B = px->size(0), N = px->size(1), C = px->size(2), heads = integer(a[2]), mode = integer(a[4]);
    if (B < 1 || N < 1 || C != heads * kHeadDim) throw NotStock{};
    const Tensor qkv_w = prec.linear(w[0]), qkv_b = prec.linear(w[1]), proj_w = prec.linear(w[6]), proj_b = prec.linear(w[7]);
    for (int i = 2; i < 6; ++i) prec.row(w[i], kHeadDim);
    const Norm norm(w + 2);
    const Tensor* pos = stock(a[3]);
    const double base = real(a[5]);
    return wrap(unlocked([&]() -> Tensor {
      c10::cuda::CUDAGuard guard(px->device());
      at::AutoDispatchBelowADInplaceOrView below;
      c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
      const Tensor cs = rotation(pos, mode, base, N, *px);
      Tensor rows = px->reshape({B * N, C});
      if (rows.scalar_type() != at::kBFloat16) rows = rows.to(at::kBFloat16);
      Qkv r = prep(linear(rows, qkv_w, qkv_b), heads, N, norm, cs.defined() ? &cs : nullptr, cs.defined() ? mode : GCT_ROPE_NONE);
      const Tensor o = dense(r.q.view({B, N, heads, kHeadDim}), r.k.view({B, N, heads, kHeadDim}), r.v.view({B, N, heads, kHeadDim}), Tensor());
      return linear(o.view({B * N, C}), proj_w, proj_b).view({B, N, proj_w.size(0)});
    }));
  });
}

// block_layer(x, (n1_w, n1_b, qkv_w, qkv_b, qn_w, qn_b, kn_w, kn_b, proj_w, proj_b, gamma1, n2_w, n2_b, fc1_w, fc1_b, fc2_w, fc2_b,
//             gamma2), eps1, eps2, heads, with_ffn, pos, rope_mode, rope_base, manager | 0, device, block, window, frames, skip_append) -> y
// manager and frames <= 1: one streamed frame on the paged cache.  manager and frames > 1: the scale pass, all tokens attend to
// each other, then every frame is appended.  No manager: dense attention per batch entry.
PyObject* py_block_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return layer([&]() -> PyObject* {
    need(n, 15, "block_layer");
    const Tensor* px = stock(a[0]);
    if (px == nullptr || !px->is_cuda() || px->dim() != 3 || PyTuple_GET_SIZE(a[1]) != 18) throw NotStock{};
    const Precision prec(*px);
    PyObject* const* w = &PyTuple_GET_ITEM(a[1], 0);
    const int64_t B = px->size(0), N = px->size(1), C = px->size(2), heads = integer(a[4]), mode = integer(a[7]);
    const bool with_ffn = PyObject_IsTrue(a[5]) == 1, skip = PyObject_IsTrue(a[14]) == 1;
    gct_mgr_t* m = manager(a[9]);
    const int64_t device = integer(a[10]), block = integer(a[11]), window = integer(a[12]), frames = integer(a[13]);
    if (B < 1 || N < 1 || C != heads * kHeadDim || C > gct::kRowMaxCols) throw NotStock{};
    if (m != nullptr) {
      const gct_mgr_config_t& cfg = gct::mgr_config(m);
      if (B != 1 || N != std::max<int64_t>(frames, 1) * cfg.tokens_per_frame || heads != cfg.num_heads || device != px->device().index() ||
          (frames > 1 && skip))
        throw NotStock{};
    }
    const Tensor qkv_w = prec.linear(w[2]), qkv_b = prec.linear(w[3]), proj_w = prec.linear(w[8]), proj_b = prec.linear(w[9]);
    for (int i = 4; i < 8; ++i) prec.row(w[i], kHeadDim);
    const Tensor *n1w = prec.row(w[0], C), *n1b = prec.row(w[1], C), *g1 = prec.row(w[10], C);
    const Tensor *n2w = nullptr, *n2b = nullptr, *g2 = nullptr;
    Tensor fc1_w, fc1_b, fc2_w, fc2_b;
    if (n1w == nullptr || n1b == nullptr || n1w->scalar_type() != n1b->scalar_type() || proj_w.dim() != 2 || proj_w.size(0) != C) throw NotStock{};
    if (with_ffn) {
      n2w = prec.row(w[11], C);
      n2b = prec.row(w[12], C);
      g2 = prec.row(w[17], C);
      fc1_w = prec.linear(w[13]);
      fc1_b = prec.linear(w[14]);
      fc2_w = prec.linear(w[15]);
      fc2_b = prec.linear(w[16]);
      if (n2w == nullptr || n2b == nullptr || n2w->scalar_type() != n2b->scalar_type() || !fc1_w.defined() || !fc2_w.defined() ||
          fc2_w.dim() != 2 || fc2_w.size(0) != C)
        throw NotStock{};
    }
    const Norm norm(w + 4);
    const Tensor* pos = stock(a[6]);
    const double eps1 = real(a[2]), eps2 = real(a[3]), base = real(a[8]);
    return wrap(unlocked([&]() -> Tensor {
      c10::cuda::CUDAGuard guard(px->device());
      at::AutoDispatchBelowADInplaceOrView below;
      c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
      const Tensor table = rotation(pos, mode, base, N, *px);
      const Tensor* cs = table.defined() ? &table : nullptr;
      const int64_t rope = table.defined() ? mode : GCT_ROPE_NONE;
      Tensor x = px->reshape({B * N, C});
      // reshape hands back a view wherever strides allow (a column slice, every other token, a transposed or expanded input)
      if (!x.is_contiguous() || !aligned16(x)) x = x.clone(at::MemoryFormat::Contiguous);
      const Tensor normed = residual_norm(x, nullptr, nullptr, nullptr, n1w, n1b, eps1);
      const Tensor qkv = linear(normed, qkv_w, qkv_b);
      const int blk = static_cast<int>(block);
      Tensor o;
      if (m != nullptr && frames <= 1) {
        int deferred = 0;
        if (skip) {
          check(gct_mgr_get_defer(m, &deferred));
          check(gct_mgr_set_defer(m, 1));
        }
        const Tensor q = append_fused(m, device, block, qkv, norm, cs, rope, Tensor());
        if (!skip) check(gct_mgr_evict(m, blk, static_cast<int>(window)));
        o = attend(m, device, block, q, false).out;
        if (skip) {
          check(gct_mgr_rollback(m, blk));
          check(gct_mgr_set_defer(m, deferred));
        }
      } else {
        Qkv r = prep(qkv, heads, N, norm, cs, rope);
        o = dense(r.q.view({B, N, heads, kHeadDim}), r.k.view({B, N, heads, kHeadDim}), r.v.view({B, N, heads, kHeadDim}), Tensor());
        if (m != nullptr)
          check(gct::mgr_append_frames(m, blk, bf16(r.k), bf16(r.v), static_cast<int>(frames), static_cast<int>(window), stream_of(x)));
      }
      const Tensor attn = linear(o.view({B * N, C}), proj_w, proj_b);
      Tensor sum;
      const Tensor normed2 = residual_norm(x, &attn, g1, &sum, n2w, n2b, eps2);
      if (with_ffn) {
        const Tensor h = linear(normed2, fc1_w, fc1_b);
        check(gct::launch_gelu(static_cast<__nv_bfloat16*>(h.data_ptr()), h.numel(), stream_of(h)));
        const Tensor f = linear(h, fc2_w, fc2_b);
        Tensor out;
        residual_norm(sum, &f, g2, &out, nullptr, nullptr, 0.0);
        sum = out;
      }
      return sum.view({B, N, C});
    }));
  });
}

// ---- camera head, rotation tables ---------------------------------------------------------------

// decode_attention(q, k_new, v_new, cache_k, cache_v, cached, store, workspace) -> out
PyObject* py_decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 8, "decode_attention");
    const Tensor &ck = tensor(a[3], "cache_k"), &cv = tensor(a[4], "cache_v"), &ws = tensor(a[7], "workspace");
    auto rows = [&](PyObject* o, const char* name) {
      const Tensor& t = tensor(o, name);
      return t.is_contiguous() ? t : t.contiguous();
    };
    const Tensor q = rows(a[0], "q"), k = rows(a[1], "k_new"), v = rows(a[2], "v_new");
    const Tensor* all[5] = {&q, &k, &v, &ck, &cv};
    for (const Tensor* t : all) {
      need_cuda(*t, "decode attention: every tensor");
      if (t->scalar_type() != at::kFloat || t->dim() != 3 || !t->is_contiguous() || t->size(1) != ck.size(1) || t->size(2) != ck.size(2) ||
          t->device() != ck.device())
        value_error("decode attention: tensors must be contiguous float32 [rows, H, D] on one device");
    }
    if (k.size(0) != q.size(0) || v.size(0) != q.size(0)) value_error("decode attention: q, k and v must have the same number of rows");
    c10::cuda::CUDAGuard guard(q.device());
    Tensor out = empty(q.sizes(), at::kFloat, q);
    const int cached = static_cast<int>(integer(a[5])), store = PyObject_IsTrue(a[6]) == 1;
    check(unlocked([&] { return gct_decode_attention(q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), static_cast<int>(q.size(0)), ck.data_ptr<float>(),
                               cv.data_ptr<float>(), cached, static_cast<int>(ck.size(0)), store,
                               static_cast<int>(ck.size(1)), static_cast<int>(ck.size(2)), out.data_ptr<float>(), ws.data_ptr(), ws.nbytes(),
                               stream_of(q)); }));
    return wrap(std::move(out));
  });
}

// rope3d_table(frame_index, pph, ppw, num_special, out)
PyObject* py_rope3d_table(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 5, "rope3d_table");
    const Tensor& out = tensor(a[4], "out");
    need_cuda(out, "out");
    const int64_t pph = integer(a[1]), ppw = integer(a[2]), ns = integer(a[3]);
    // (cos, sin) pairs: as complex64 [tokens, 32] the same bytes
    const int64_t floats = out.scalar_type() == at::kFloat ? out.numel() : out.scalar_type() == at::kComplexFloat ? 2 * out.numel() : 0;
    if (!out.is_contiguous() || out.is_conj() || floats < (ns + pph * ppw) * 64) value_error("out must be contiguous float32 [tokens, 32, 2]");
    c10::cuda::CUDAGuard guard(out.device());
    check(gct_rope3d_table(static_cast<int>(integer(a[0])), static_cast<int>(pph), static_cast<int>(ppw), static_cast<int>(ns),
                           static_cast<float*>(out.data_ptr()), stream_of(out)));
    Py_RETURN_NONE;
  });
}

// ---- point clouds -------------------------------------------------------------------------------

Tensor float_rows(const Tensor& t, const char* name) {
  need_cuda(t, name);
  Tensor r = t.is_contiguous() ? t : t.contiguous();
  return r.scalar_type() == at::kFloat ? r : r.to(at::kFloat);
}

// frustum_cull(pts, R_cw, t_cw, fx, fy, cx, cy, W, H, near, far) -> bool mask
PyObject* py_frustum_cull(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 11, "frustum_cull");
    const Tensor pts = float_rows(tensor(a[0], "pts"), "pts");
    Tensor R = tensor(a[1], "R_cw").detach(), t = tensor(a[2], "t_cw").detach();
    if (R.numel() != 9 || t.numel() != 3) value_error("R_cw must hold 9 values, t_cw 3");
    c10::cuda::CUDAGuard guard(pts.device());
    const bool on_device = R.is_cuda() || t.is_cuda();
    // a camera of which one half is on the device goes there whole: a copy to the device does not wait, one back does
    auto place = [&](Tensor x) {
      if (x.scalar_type() != at::kFloat) x = x.to(at::kFloat);
      if (on_device && x.device() != pts.device()) x = x.to(pts.device());
      return on_device || x.is_contiguous() ? x : x.contiguous();
    };
    R = place(R);
    t = place(t);
    // the kernel steps through R by row and column strides: nine values of any other shape ([1, 9], a flat [9]) are taken in order
    if (R.sizes() != at::IntArrayRef({3, 3})) R = R.reshape({3, 3});
    if (t.dim() != 1) t = t.reshape({3});
    // their owner may free them on another stream as soon as this returns, as it could when the call waited for a copy
    for (const Tensor* c : {&R, &t})
      if (c->is_cuda()) c10::cuda::CUDACachingAllocator::recordStream(c->storage().data_ptr(), c10::cuda::getCurrentCUDAStream(pts.device().index()));
    const int strides[3] = {static_cast<int>(R.stride(0)), static_cast<int>(R.stride(1)), static_cast<int>(t.stride(0))};
    const int64_t count = pts.size(0);
    Tensor visible = empty({count}, at::kBool, pts);
    if (count > 0)
      check(gct::frustum_cull(pts.data_ptr<float>(), count, R.data_ptr<float>(), t.data_ptr<float>(), on_device ? strides : nullptr, static_cast<float>(real(a[3])),
                              static_cast<float>(real(a[4])), static_cast<float>(real(a[5])), static_cast<float>(real(a[6])),
                              static_cast<int>(integer(a[7])), static_cast<int>(integer(a[8])), static_cast<float>(real(a[9])),
                              static_cast<float>(real(a[10])), static_cast<uint8_t*>(visible.data_ptr()), stream_of(pts)));
    return wrap(std::move(visible));
  });
}

// voxelize_frame(xyz, rgb, voxel_size) -> (centers, colors, codes) | None (more points than the sort takes)
PyObject* py_voxelize_frame(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 3, "voxelize_frame");
    const Tensor &in_xyz = tensor(a[0], "pts_xyz"), &in_rgb = tensor(a[1], "pts_rgb");
    need_cuda(in_xyz, "pts_xyz");
    const int64_t count = in_xyz.size(0);
    if (count < 1 || count > gct::kVoxelMaxPoints) Py_RETURN_NONE;
    const Tensor xyz = float_rows(in_xyz, "pts_xyz"), rgb = float_rows(in_rgb, "pts_rgb");
    need_beside(rgb, "pts_rgb", xyz);
    if (xyz.numel() < 3 * count || rgb.numel() < 3 * count) value_error("pts_xyz and pts_rgb must be [N, 3]");
    const float voxel = static_cast<float>(real(a[2]));
    c10::cuda::CUDAGuard guard(xyz.device());
    cudaStream_t s = stream_of(xyz);
    size_t bytes = 0;
    int tiles = 0;
    check(gct::voxel_sort_layout(count, &bytes, &tiles));
    Tensor scratch = empty({static_cast<int64_t>(bytes)}, at::kByte, xyz);
    Tensor report = at::empty({tiles}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    int64_t voxels = 0;
    int rc;
    {
      WithoutGil free_others;      // waits: the outputs are sized by the number of voxels
      rc = gct::voxel_sort(xyz.data_ptr<float>(), voxel, count, scratch.data_ptr(), report.data_ptr<int32_t>(), &voxels, s);
    }
    check(rc);
    Tensor centers = empty({voxels, 3}, at::kFloat, xyz), colors = empty({voxels, 3}, at::kFloat, xyz), codes = empty({voxels}, at::kLong, xyz);
    check(gct::voxel_gather(xyz.data_ptr<float>(), rgb.data_ptr<float>(), voxel, count, scratch.data_ptr(), centers.data_ptr<float>(),
                            colors.data_ptr<float>(), codes.data_ptr<int64_t>(), s));
    PyObject* out = PyTuple_New(3);
    if (out == nullptr) throw python_error();
    PyTuple_SET_ITEM(out, 0, wrap(std::move(centers)));
    PyTuple_SET_ITEM(out, 1, wrap(std::move(colors)));
    PyTuple_SET_ITEM(out, 2, wrap(std::move(codes)));
    return out;
  });
}

// set_classes(GctError, torch.nn.Parameter)
PyObject* py_set_classes(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need(n, 2, "set_classes");
    Py_XSETREF(g_error_class, Py_NewRef(a[0]));
    Py_XSETREF(g_parameter_class, Py_NewRef(a[1]));
    Py_RETURN_NONE;
  });
}

#define FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(prep_qkv),
                           FAST(dense_attention),
                           FAST(operator_status),
                           FAST(append),
                           FAST(append_fused),
                           FAST(attention),
                           FAST(append_bookkeeping),
                           FAST(evict),
                           FAST(rollback),
                           FAST(decode_attention),
                           FAST(rope3d_table),
                           FAST(frustum_cull),
                           FAST(voxelize_frame),
                           FAST(frame_layer),
                           FAST(block_layer),
                           FAST(set_classes),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_gct_torch", "PyTorch binding of libgct_b200.so", -1, g_methods,
                        nullptr,               nullptr,      nullptr,                             nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__gct_torch() { return PyModule_Create(&g_module); }
