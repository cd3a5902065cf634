// Host side of the calls that a program makes per layer and per token: allocate the outputs, fill in the job
// descriptions of the C ABI, launch.  In Python the same work took 80 to 160 us for one layer's compress_kv and
// decompress_kv and 330 us for a generation step of 32 layers, several times what the GPU needs for them.
//
// Every function takes the plain case only -- ordinary strided CUDA tensors on the current device, of the expected types
// and shapes -- and returns None for anything else; the caller then runs its general Python path, which also raises the
// errors.  Nothing is kept between calls except the step plan, which belongs to the cache that made it.

#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "../../include/turboquant_b200.h"

namespace {

struct Api {
  decltype(&tq_quantize) quantize = nullptr;
  decltype(&tq_dequantize) dequantize = nullptr;
  decltype(&tq_copy_rows) copy_rows = nullptr;
  decltype(&tq_qjl_compress) qjl_compress = nullptr;
  decltype(&tq_qjl_compress_workspace_bytes) qjl_compress_ws = nullptr;
  decltype(&tq_prod_inner_product) prod_inner = nullptr;
  decltype(&tq_score_packed) score_packed = nullptr;
  decltype(&tq_score_workspace_bytes) score_ws = nullptr;
  decltype(&tq_decode_attention) decode_attention = nullptr;
  decltype(&tq_decode_attention_workspace_bytes) decode_attention_ws = nullptr;
  decltype(&tq_qjl_scores_packed) qjl_scores_packed = nullptr;
  decltype(&tq_qjl_scores_packed_workspace_bytes) qjl_scores_packed_ws = nullptr;
  PyObject* check = nullptr;               // Python: check(rc, what) raises for rc != 0
  // the classes' own job methods, as functions: MSECompressor.compress_job, decompress_job, TurboQuantV3.compress_jobs, decompress_jobs
  PyObject* jobs = nullptr;
} api;

// ---------------------------------------------------------------- small helpers
// A reference that this scope owns.
struct Ref {
  PyObject* p;
  explicit Ref(PyObject* q = nullptr) : p(q) {}
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  PyObject* release() { PyObject* q = p; p = nullptr; return q; }
  explicit operator bool() const { return p != nullptr; }
};

PyObject* none() { Py_RETURN_NONE; }

PyObject* intern(const char* s) { return PyUnicode_InternFromString(s); }

#define TQ_NAME(var, text) static PyObject* const var = intern(text)

int dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return TQ_F32;
    case at::kHalf: return TQ_F16;
    case at::kBFloat16: return TQ_BF16;
    default: return -1;
  }
}

// an ordinary strided tensor on CUDA device `dev`
bool plain(PyObject* o, int dev) {
  if (!THPVariable_CheckExact(o)) return false;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.get_device() == dev && !t.is_conj() && !t.is_neg();
}
bool float_plain(PyObject* o, int dev) { return plain(o, dev) && dtype_of(THPVariable_Unpack(o)) >= 0; }

// 1 found (tensor), 0 None, -1 neither
int attr_ptr(PyObject* o, PyObject* name, int dev, void** out) {
  Ref a(PyObject_GetAttr(o, name));
  if (!a) { PyErr_Clear(); return -1; }
  if (a.p == Py_None) { *out = nullptr; return 0; }
  if (!plain(a.p, dev)) return -1;
  *out = THPVariable_Unpack(a.p).data_ptr();
  return 1;
}
bool attr_int(PyObject* o, PyObject* name, int64_t* out) {
  Ref a(PyObject_GetAttr(o, name));
  if (!a || !PyLong_Check(a.p)) { PyErr_Clear(); return false; }
  *out = PyLong_AsLongLong(a.p);
  return true;
}

// the constants of one MSECompressor (or an object with the same attributes)
struct Codec {
  void *pi = nullptr, *pi_t = nullptr, *cb = nullptr, *img_q = nullptr, *img_d = nullptr;
  int64_t bits = 0, dim = 0;
};
bool read_codec(PyObject* o, int dev, Codec* c) {
  TQ_NAME(n_pi, "Pi"); TQ_NAME(n_pit, "_pi_t"); TQ_NAME(n_cb, "_cb"); TQ_NAME(n_iq, "_img_q"); TQ_NAME(n_id, "_img_d");
  TQ_NAME(n_bits, "bits"); TQ_NAME(n_dim, "head_dim");
  return attr_int(o, n_bits, &c->bits) && c->bits >= 1 && c->bits <= 8 && attr_int(o, n_dim, &c->dim) && c->dim >= 1 && c->dim <= 256 &&
         attr_ptr(o, n_pi, dev, &c->pi) == 1 && attr_ptr(o, n_pit, dev, &c->pi_t) == 1 && attr_ptr(o, n_cb, dev, &c->cb) == 1 &&
         attr_ptr(o, n_iq, dev, &c->img_q) >= 0 && attr_ptr(o, n_id, dev, &c->img_d) >= 0;
}
// `method` is number `i` of the classes' own job methods, bound.  What this file does stands in for them; a method that a
// subclass, an object or a patch has put in their place is asked instead.
bool own_method(PyObject* method, int i) { return PyMethod_Check(method) && PyMethod_GET_FUNCTION(method) == PyTuple_GET_ITEM(api.jobs, i); }
bool own_codec(PyObject* codec, bool compress) {
  TQ_NAME(n_c, "compress_job"); TQ_NAME(n_d, "decompress_job");
  Ref m(PyObject_GetAttr(codec, compress ? n_c : n_d));
  if (!m) { PyErr_Clear(); return false; }
  return own_method(m.p, compress ? 0 : 1);
}
int64_t row_bytes(int64_t dim, int64_t bits) { const int64_t ipb = 8 / bits; return (dim + ipb - 1) / ipb; }

at::Tensor make(at::IntArrayRef sizes, at::ScalarType type, int dev) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(at::Device(at::kCUDA, (c10::DeviceIndex)dev)));
}

void* stream_of(int dev) { return (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }

// tokens [start, start + length) of a (B, H, S, D) tensor: what narrow(2, ...) gives, for half its host time (1.4 -> 0.76 us; a
// generation step of 32 layers hands out 64 of them)
at::Tensor tokens(const at::Tensor& t, int64_t start, int64_t length) {
  const int64_t sizes[4] = {t.size(0), t.size(1), length, t.size(3)};
  return at::as_strided(t, sizes, t.strides(), t.storage_offset() + start * t.stride(2));
}

// runs a call of the C ABI without the interpreter lock; false with a Python exception set when it fails
template <typename F>
bool call(const char* what, F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = f();
  Py_END_ALLOW_THREADS
  if (rc == 0) return true;
  Ref r(PyObject_CallFunction(api.check, "is", rc, what));
  if (r) PyErr_Format(PyExc_RuntimeError, "%s failed with code %d", what, rc);
  return false;
}

PyObject* shape_tuple(int64_t b, int64_t h, int64_t s, int64_t d) { return Py_BuildValue("(LLLL)", (long long)b, (long long)h, (long long)s, (long long)d); }

bool set_item(PyObject* dict, PyObject* key, PyObject* value) {      // takes over `value`
  if (value == nullptr) return false;
  const int rc = PyDict_SetItem(dict, key, value);
  Py_DECREF(value);
  return rc == 0;
}

// quantise job for tokens [0, s) of a (B, H, S, D) tensor; allocates the packed rows and norms
TqQuantizeJob quantize_job(const at::Tensor& x, int64_t s, const Codec& c, int dev, at::Tensor* idx, at::Tensor* norms) {
  const int64_t b = x.size(0), h = x.size(1), d = x.size(3);
  *idx = make({b, h, s, row_bytes(d, c.bits)}, at::kByte, dev);
  *norms = make({b, h, s}, at::kHalf, dev);
  TqQuantizeJob j{};
  j.x = x.data_ptr(); j.x_dtype = dtype_of(x); j.D = (int32_t)d; j.bits = (int32_t)c.bits; j.normalize = 1;
  j.B = b; j.H = h; j.S = s;
  j.stride_b = x.stride(0); j.stride_h = x.stride(1); j.stride_s = x.stride(2);
  j.rotation_t = (const float*)c.pi_t; j.codebook = (const float*)c.cb; j.idx_mode = TQ_IDX_PACKED;
  j.idx_out = idx->data_ptr(); j.norms_out = (uint16_t*)norms->data_ptr(); j.rotation_image = c.img_q;
  return j;
}
bool quantisable(const at::Tensor& x, const Codec& c) {
  return x.dim() == 4 && x.size(3) == c.dim && (x.stride(3) == 1 || x.size(3) == 1);
}

PyObject* packed_dict(const at::Tensor& idx, const at::Tensor& norms, int64_t b, int64_t h, int64_t s, int64_t d, int64_t bits) {
  TQ_NAME(k_idx, "idx_bytes"); TQ_NAME(k_norms, "vec_norms"); TQ_NAME(k_shape, "shape"); TQ_NAME(k_pad, "idx_pad");
  const int64_t ipb = 8 / bits;
  Ref dict(PyDict_New());
  if (!dict || !set_item(dict.p, k_idx, THPVariable_Wrap(idx)) || !set_item(dict.p, k_norms, THPVariable_Wrap(norms)) ||
      !set_item(dict.p, k_shape, shape_tuple(b, h, s, d)) || !set_item(dict.p, k_pad, PyLong_FromLongLong((ipb - d % ipb) % ipb)))
    return nullptr;
  return dict.release();
}

// four integers of dict["shape"]
bool read_shape(PyObject* dict, int64_t (&v)[4]) {
  TQ_NAME(k_shape, "shape");
  PyObject* t = PyDict_GetItem(dict, k_shape);
  if (t == nullptr || !PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 4) return false;
  for (int i = 0; i < 4; ++i) {
    PyObject* e = PyTuple_GET_ITEM(t, i);
    if (!PyLong_Check(e)) return false;
    v[i] = PyLong_AsLongLong(e);
  }
  return true;
}

// dequantise job of a packed dict into the tokens [0, s) of `out`; false when the dict is not in the plain form
// (`keep` holds its tensors until the launch is out: the interpreter lock is given up for that)
bool dequantize_job(PyObject* dict, const Codec& c, int dev, const int64_t (&shape)[4], const at::Tensor& out, TqDequantizeJob* j,
                    at::Tensor (&keep)[2]) {
  TQ_NAME(k_idx, "idx_bytes"); TQ_NAME(k_norms, "vec_norms");
  PyObject *io = PyDict_GetItem(dict, k_idx), *no = PyDict_GetItem(dict, k_norms);
  if (io == nullptr || no == nullptr || !plain(io, dev) || !plain(no, dev)) return false;
  const at::Tensor &idx = THPVariable_Unpack(io), &norms = THPVariable_Unpack(no);
  const int64_t n = shape[0] * shape[1] * shape[2];
  if (idx.scalar_type() != at::kByte || norms.scalar_type() != at::kHalf || !idx.is_contiguous() || !norms.is_contiguous() ||
      idx.numel() != n * row_bytes(shape[3], c.bits) || norms.numel() != n || shape[3] != c.dim)
    return false;
  keep[0] = idx;
  keep[1] = norms;
  *j = TqDequantizeJob{};
  j->idx = idx.data_ptr(); j->norms = (const uint16_t*)norms.data_ptr(); j->idx_mode = TQ_IDX_PACKED;
  j->D = (int32_t)shape[3]; j->bits = (int32_t)c.bits; j->out_dtype = dtype_of(out);
  j->B = shape[0]; j->H = shape[1]; j->S = shape[2];
  j->out = out.data_ptr();
  j->ostride_b = out.stride(0); j->ostride_h = out.stride(1); j->ostride_s = out.stride(2);
  j->rotation = (const float*)c.pi; j->codebook = (const float*)c.cb; j->rotation_image = c.img_d;
  return true;
}

// ---------------------------------------------------------------- one layer's K and V
// compress_kv(key_codec, value_codec, keys, values, window, the layer's compress_jobs) -> (dict, dict) | None
PyObject* compress_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  if (n != 6 || !float_plain(a[2], dev) || !float_plain(a[3], dev) || !PyLong_Check(a[4]) || !own_method(a[5], 2) || !own_codec(a[0], true) ||
      !own_codec(a[1], true))
    return none();
  const at::Tensor &k = THPVariable_Unpack(a[2]), &v = THPVariable_Unpack(a[3]);
  const int64_t window = PyLong_AsLongLong(a[4]);
  Codec ck, cv;
  if (window < 0 || !read_codec(a[0], dev, &ck) || !read_codec(a[1], dev, &cv) || !quantisable(k, ck) || !quantisable(v, cv) ||
      k.sizes() != v.sizes() || k.size(2) <= window)
    return none();
  c10::AutoGradMode no_grad(false);
  const int64_t b = k.size(0), h = k.size(1), s = k.size(2), d = k.size(3), cut = s - window;
  TqQuantizeJob jobs[2];
  at::Tensor idx[2], norms[2];
  jobs[0] = quantize_job(k, cut, ck, dev, &idx[0], &norms[0]);
  jobs[1] = quantize_job(v, cut, cv, dev, &idx[1], &norms[1]);
  void* st = stream_of(dev);
  if (!call("tq_quantize", [&] { return api.quantize(jobs, 2, st); })) return nullptr;
  TQ_NAME(k_comp, "compressed"); TQ_NAME(k_fp16, "fp16"); TQ_NAME(k_shape, "shape"); TQ_NAME(k_split, "split_at");
  Ref out(PyTuple_New(2));
  if (!out) return nullptr;
  for (int i = 0; i < 2; ++i) {
    const at::Tensor& x = i ? v : k;
    Ref dict(PyDict_New());
    if (!dict || !set_item(dict.p, k_comp, packed_dict(idx[i], norms[i], b, h, cut, d, i ? cv.bits : ck.bits)) ||
        !set_item(dict.p, k_fp16, THPVariable_Wrap(tokens(x, cut, window))) || !set_item(dict.p, k_shape, shape_tuple(b, h, s, d)) ||
        !set_item(dict.p, k_split, PyLong_FromLongLong(cut)))
      return nullptr;
    PyTuple_SET_ITEM(out.p, i, dict.release());
  }
  return out.release();
  END_HANDLE_TH_ERRORS
}

bool copy_fits(const at::Tensor& t, int64_t eb) {
  if ((uintptr_t)t.data_ptr() & 15u) return false;
  for (int i = 0; i < 3; ++i)
    if (t.size(i) > 1 && (t.stride(i) < 0 || t.stride(i) * eb % 16 != 0)) return false;
  return t.stride(3) == 1 && t.size(3) * eb % 16 == 0;
}

// decompress_kv(key_codec, value_codec, compressed_k, compressed_v, the layer's decompress_jobs) -> (keys, values) | None
PyObject* decompress_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TQ_NAME(k_comp, "compressed"); TQ_NAME(k_fp16, "fp16"); TQ_NAME(k_split, "split_at");
  const int dev = c10::cuda::current_device();
  if (n != 5 || !own_method(a[4], 3) || !own_codec(a[0], false) || !own_codec(a[1], false)) return none();
  c10::AutoGradMode no_grad(false);
  TqDequantizeJob jobs[2];
  TqCopyJob copies[2];
  at::Tensor full[2];
  PyObject* comps[2];
  Codec codec[2];
  int64_t inner[2][4], outer[2][4];
  at::Tensor windows[2], keep[2][2];
  for (int i = 0; i < 2; ++i) {                       // look everything over before anything is allocated or launched
    PyObject* side = a[2 + i];
    if (!PyDict_CheckExact(side) || !read_codec(a[i], dev, &codec[i])) return none();
    PyObject *comp = PyDict_GetItem(side, k_comp), *win = PyDict_GetItem(side, k_fp16), *split = PyDict_GetItem(side, k_split);
    if (comp == nullptr || !PyDict_CheckExact(comp) || win == nullptr || !float_plain(win, dev) || split == nullptr || !PyLong_Check(split))
      return none();
    if (!read_shape(side, outer[i]) || !read_shape(comp, inner[i])) return none();
    const int64_t cut = PyLong_AsLongLong(split);
    windows[i] = THPVariable_Unpack(win);
    const int64_t kept = outer[i][2] - cut;
    if (kept < 0 || cut < 0 || inner[i][0] != outer[i][0] || inner[i][1] != outer[i][1] || inner[i][2] != cut || inner[i][3] != outer[i][3] ||
        windows[i].sizes() != at::IntArrayRef({outer[i][0], outer[i][1], kept, outer[i][3]}))
      return none();
    comps[i] = comp;
  }
  if (windows[0].scalar_type() != windows[1].scalar_type()) return none();
  for (int i = 0; i < 2; ++i) {
    full[i] = make({outer[i][0], outer[i][1], outer[i][2], outer[i][3]}, windows[i].scalar_type(), dev);
    if (!dequantize_job(comps[i], codec[i], dev, inner[i], full[i], &jobs[i], keep[i])) return none();
  }
  int n_copies = 0;
  for (int i = 0; i < 2; ++i) {
    if (windows[i].numel() == 0) continue;
    const at::Tensor dst = tokens(full[i], inner[i][2], windows[i].size(2));
    const int64_t eb = dst.element_size();
    if (!copy_fits(windows[i], eb) || !copy_fits(dst, eb)) { const_cast<at::Tensor&>(dst).copy_(windows[i]); continue; }
    TqCopyJob& c = copies[n_copies++];
    c = TqCopyJob{};
    c.src = windows[i].data_ptr(); c.dst = dst.data_ptr(); c.elem_bytes = (int32_t)eb; c.D = (int32_t)dst.size(3);
    c.B = dst.size(0); c.H = dst.size(1); c.S = dst.size(2);
    c.sstride_b = windows[i].stride(0); c.sstride_h = windows[i].stride(1); c.sstride_s = windows[i].stride(2);
    c.dstride_b = dst.stride(0); c.dstride_h = dst.stride(1); c.dstride_s = dst.stride(2);
  }
  void* st = stream_of(dev);
  if (n_copies > 0 && !call("tq_copy_rows", [&] { return api.copy_rows(copies, n_copies, st); })) return nullptr;
  if (!call("tq_dequantize", [&] { return api.dequantize(jobs, 2, st); })) return nullptr;
  Ref k(THPVariable_Wrap(full[0])), v(THPVariable_Wrap(full[1]));
  if (!k || !v) return nullptr;
  return PyTuple_Pack(2, k.p, v.p);
  END_HANDLE_TH_ERRORS
}

// compress(codec, states) -> dict | None
PyObject* compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  Codec c;
  if (n != 2 || !float_plain(a[1], dev) || !own_codec(a[0], true) || !read_codec(a[0], dev, &c)) return none();
  const at::Tensor& x = THPVariable_Unpack(a[1]);
  if (!quantisable(x, c)) return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor idx, norms;
  TqQuantizeJob job = quantize_job(x, x.size(2), c, dev, &idx, &norms);
  void* st = stream_of(dev);
  if (!call("tq_quantize", [&] { return api.quantize(&job, 1, st); })) return nullptr;
  return packed_dict(idx, norms, x.size(0), x.size(1), x.size(2), x.size(3), c.bits);
  END_HANDLE_TH_ERRORS
}

// decompress(codec, dict) -> fp32 tensor | None
PyObject* decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  Codec c;
  int64_t shape[4];
  if (n != 2 || !PyDict_CheckExact(a[1]) || !own_codec(a[0], false) || !read_codec(a[0], dev, &c) || !read_shape(a[1], shape)) return none();
  for (int64_t s : shape)
    if (s < 0) return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor out = make({shape[0], shape[1], shape[2], shape[3]}, at::kFloat, dev);
  TqDequantizeJob job;
  at::Tensor keep[2];
  if (!dequantize_job(a[1], c, dev, shape, out, &job, keep)) return none();
  void* st = stream_of(dev);
  if (!call("tq_dequantize", [&] { return api.dequantize(&job, 1, st); })) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- first-generation classes: rows of d values
// quantize_rows(x, pi_t, codebook, bits, d) -> int64 indices of x's shape | None
PyObject* quantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  if (n != 5 || !float_plain(a[0], dev) || !plain(a[1], dev) || !plain(a[2], dev)) return none();
  const at::Tensor& x = THPVariable_Unpack(a[0]);
  const int64_t bits = PyLong_AsLongLong(a[3]), d = PyLong_AsLongLong(a[4]);
  if (bits < 1 || bits > 8 || d < 1 || d > 256 || x.dim() < 1 || x.size(-1) != d || !x.is_contiguous()) return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor idx = make(x.sizes(), at::kLong, dev);
  TqQuantizeJob j{};
  j.x = x.data_ptr(); j.x_dtype = dtype_of(x); j.D = (int32_t)d; j.bits = (int32_t)bits;
  j.B = 1; j.H = 1; j.S = x.numel() / d; j.stride_b = x.numel(); j.stride_h = x.numel(); j.stride_s = d;
  j.rotation_t = (const float*)THPVariable_Unpack(a[1]).data_ptr(); j.codebook = (const float*)THPVariable_Unpack(a[2]).data_ptr();
  j.idx_mode = TQ_IDX_I64; j.idx_out = idx.data_ptr();
  void* st = stream_of(dev);
  if (!call("tq_quantize", [&] { return api.quantize(&j, 1, st); })) return nullptr;
  return THPVariable_Wrap(idx);
  END_HANDLE_TH_ERRORS
}

// dequantize_rows(indices, pi, codebook, bits, d) -> fp32 of the indices' shape | None
PyObject* dequantize_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  if (n != 5 || !plain(a[0], dev) || !plain(a[1], dev) || !plain(a[2], dev)) return none();
  const at::Tensor& idx = THPVariable_Unpack(a[0]);
  const int64_t bits = PyLong_AsLongLong(a[3]), d = PyLong_AsLongLong(a[4]);
  if (bits < 1 || bits > 8 || d < 1 || d > 256 || idx.scalar_type() != at::kLong || idx.dim() < 1 || idx.size(-1) != d || !idx.is_contiguous())
    return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor out = make(idx.sizes(), at::kFloat, dev);
  TqDequantizeJob j{};
  j.idx = idx.data_ptr(); j.idx_mode = TQ_IDX_I64; j.D = (int32_t)d; j.bits = (int32_t)bits; j.out_dtype = TQ_F32;
  j.B = 1; j.H = 1; j.S = idx.numel() / d; j.out = out.data_ptr(); j.ostride_b = idx.numel(); j.ostride_h = idx.numel(); j.ostride_s = d;
  j.rotation = (const float*)THPVariable_Unpack(a[1]).data_ptr(); j.codebook = (const float*)THPVariable_Unpack(a[2]).data_ptr();
  void* st = stream_of(dev);
  if (!call("tq_dequantize", [&] { return api.dequantize(&j, 1, st); })) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// prod_inner(y (1 or n, d), idx (n, d), signs (n, m), rnorm (n,), pi, codebook, qjl_t) -> (n,) | None
PyObject* prod_inner(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  if (n != 7) return none();
  for (int i = 0; i < 7; ++i)
    if (!plain(a[i], dev) || !THPVariable_Unpack(a[i]).is_contiguous()) return none();
  const at::Tensor &y = THPVariable_Unpack(a[0]), &idx = THPVariable_Unpack(a[1]), &signs = THPVariable_Unpack(a[2]), &rn = THPVariable_Unpack(a[3]);
  if (y.scalar_type() != at::kFloat || idx.scalar_type() != at::kLong || signs.scalar_type() != at::kFloat || rn.scalar_type() != at::kFloat ||
      y.dim() != 2 || idx.dim() != 2 || signs.dim() != 2 || rn.dim() != 1)
    return none();
  const int64_t rows = idx.size(0), d = idx.size(1), m = signs.size(1);
  if (rows < 1 || y.size(1) != d || (y.size(0) != rows && y.size(0) != 1) || signs.size(0) != rows || rn.size(0) != rows) return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor out = make({rows}, at::kFloat, dev);
  at::Tensor ws = make({(y.size(0) == 1 ? 2 : rows + y.size(0)) * 256 * 4}, at::kByte, dev);
  void* st = stream_of(dev);
  const float *pi = (const float*)THPVariable_Unpack(a[4]).data_ptr(), *cb = (const float*)THPVariable_Unpack(a[5]).data_ptr(),
              *qt = (const float*)THPVariable_Unpack(a[6]).data_ptr();
  const bool ok = call("tq_prod_inner_product", [&] {
    return api.prod_inner((const float*)y.data_ptr(), y.size(0), (const int64_t*)idx.data_ptr(), (const float*)signs.data_ptr(),
                          (const float*)rn.data_ptr(), rows, (int)d, (int)m, pi, cb, qt, (float*)out.data_ptr(), ws.data_ptr(),
                          (size_t)ws.numel(), st);
  });
  if (!ok) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- MSE + QJL
// qjl_compress(x (B,H,S,D), pi, pi_t, codebook, qjl_t, bits, form) -> tuple | None.  form 0: the V2 dict's tensors
// (k_mse, signs, rnorm); 1: packed (rows, sign bits, rnorm, norms), only where the tensor-core path takes it; 2: the
// first generation's (indices, signs, rnorm) in int64 and fp32, vectors taken as they are; 3 and 4: forms 0 and 1 with the
// vectors' own leading dimensions instead of rows
PyObject* qjl_compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  if (n != 7 || !float_plain(a[0], dev)) return none();
  for (int i = 1; i < 5; ++i)
    if (!plain(a[i], dev)) return none();
  const at::Tensor &x = THPVariable_Unpack(a[0]), &qt = THPVariable_Unpack(a[4]);
  const int64_t bits = PyLong_AsLongLong(a[5]), asked = PyLong_AsLongLong(a[6]), form = asked >= 3 ? asked - 3 : asked;
  if (x.dim() != 4 || x.numel() == 0 || x.stride(3) != 1 || bits < 1 || bits > 8 || qt.dim() != 2) return none();
  const int64_t b = x.size(0), h = x.size(1), s = x.size(2), d = x.size(3), m = qt.size(1), rows = b * h * s;
  if (d > 256 || m > 256 || qt.size(0) != d || THPVariable_Unpack(a[1]).size(0) != d) return none();
  c10::AutoGradMode no_grad(false);
  TqQjlCompressJob j{};
  j.x = x.data_ptr(); j.x_dtype = dtype_of(x); j.D = (int32_t)d; j.bits = (int32_t)bits; j.normalize = form != 2;
  j.B = b; j.H = h; j.S = s; j.stride_b = x.stride(0); j.stride_h = x.stride(1); j.stride_s = x.stride(2);
  j.rotation = (const float*)THPVariable_Unpack(a[1]).data_ptr(); j.rotation_t = (const float*)THPVariable_Unpack(a[2]).data_ptr();
  j.codebook = (const float*)THPVariable_Unpack(a[3]).data_ptr(); j.qjl_t = (const float*)qt.data_ptr(); j.M = (int32_t)m;
  at::Tensor ws;
  if (form != 2 && x.scalar_type() == at::kHalf) {
    const size_t bytes = api.qjl_compress_ws(rows, (int)d);
    if (bytes) { ws = make({(int64_t)bytes}, at::kByte, dev); j.workspace = ws.data_ptr(); j.workspace_bytes = bytes; }
  }
  at::Tensor first, signs, rnorm, norms;
  const bool shaped = asked >= 3;
  auto rows_of = [&](int64_t width, at::ScalarType type) { return shaped ? make({b, h, s, width}, type, dev) : make({rows, width}, type, dev); };
  auto one_of = [&](at::ScalarType type) { return shaped ? make({b, h, s}, type, dev) : make({rows}, type, dev); };
  if (form == 0) {
    first = rows_of(d, at::kHalf); signs = rows_of(m, at::kChar); rnorm = one_of(at::kHalf);
    j.k_mse_out = (uint16_t*)first.data_ptr(); j.idx_mode = TQ_IDX_U8; j.rnorm_dtype = TQ_F16;
  } else if (form == 1) {
    if (!ws.defined() || !x.is_contiguous() || m != d || (d != 128 && d != 256) || ((uintptr_t)x.data_ptr() & 15u)) return none();
    first = rows_of(row_bytes(d, bits), at::kByte); signs = rows_of(d / 8, at::kByte);
    rnorm = one_of(at::kHalf); norms = one_of(at::kFloat);
    j.idx_out = first.data_ptr(); j.idx_mode = TQ_IDX_PACKED; j.signs_dtype = 2; j.rnorm_dtype = TQ_F16; j.vec_norms_out = (float*)norms.data_ptr();
  } else {
    first = make({rows, d}, at::kLong, dev); signs = make({rows, m}, at::kFloat, dev); rnorm = make({rows}, at::kFloat, dev);
    j.idx_out = first.data_ptr(); j.idx_mode = TQ_IDX_I64; j.signs_dtype = 1; j.rnorm_dtype = TQ_F32;
  }
  j.signs_out = signs.data_ptr(); j.rnorm_out = rnorm.data_ptr();
  void* st = stream_of(dev);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = api.qjl_compress(&j, st);
  Py_END_ALLOW_THREADS
  if (rc == TQ_EINVAL && form == 1) return none();       // not for the tensor-core path: the caller goes through the unpacked form
  if (rc != 0 && !call("tq_qjl_compress", [&] { return rc; })) return nullptr;
  Ref r0(THPVariable_Wrap(first)), r1(THPVariable_Wrap(signs)), r2(THPVariable_Wrap(rnorm));
  if (!r0 || !r1 || !r2) return nullptr;
  if (form != 1) return PyTuple_Pack(3, r0.p, r1.p, r2.p);
  Ref r3(THPVariable_Wrap(norms));
  if (!r3) return nullptr;
  return PyTuple_Pack(4, r0.p, r1.p, r2.p, r3.p);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- attention from packed keys
bool is(const at::Tensor& t, at::ScalarType type, at::IntArrayRef sizes) { return t.scalar_type() == type && t.sizes() == sizes && t.is_contiguous(); }
bool bit_width(PyObject* o, int64_t* bits) {
  if (!PyLong_Check(o)) return false;
  *bits = PyLong_AsLongLong(o);
  if (*bits == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  return *bits >= 1 && *bits <= 8;
}
// a float argument; false for anything that is not a plain number
bool number(PyObject* o, float* v) {
  if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
  const double d = PyFloat_AsDouble(o);
  if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  *v = (float)d;
  return true;
}
at::Tensor scratch(size_t bytes, int dev) { return make({(int64_t)(bytes > 256 ? bytes : 256)}, at::kByte, dev); }

// score_packed(q, idx_bytes, norms, pi_t, codebook, bits, scale, softmax) -> logits | (logits, probs) | None
PyObject* score_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  int64_t bits;
  float scale;
  if (n != 8 || !float_plain(a[0], dev) || !bit_width(a[5], &bits) || !number(a[6], &scale) || !PyBool_Check(a[7])) return none();
  for (int i = 1; i < 5; ++i)
    if (!plain(a[i], dev)) return none();
  const at::Tensor &q = THPVariable_Unpack(a[0]), &idx = THPVariable_Unpack(a[1]), &norms = THPVariable_Unpack(a[2]),
                   &pi_t = THPVariable_Unpack(a[3]), &cb = THPVariable_Unpack(a[4]);
  if (q.dim() != 4 || idx.dim() != 4 || !q.is_contiguous()) return none();
  const int64_t b = q.size(0), hq = q.size(1), sq = q.size(2), d = q.size(3), hkv = idx.size(1), sk = idx.size(2);
  if (d < 1 || d > 256 || hkv < 1 || hq % hkv != 0 || !is(idx, at::kByte, {b, hkv, sk, row_bytes(d, bits)}) || !is(norms, at::kHalf, {b, hkv, sk}) ||
      !is(pi_t, at::kFloat, {d, d}) || cb.scalar_type() != at::kFloat || cb.numel() != TQ_CODEBOOK_FLOATS || !cb.is_contiguous())
    return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor logits = make({b, hq, sq, sk}, at::kFloat, dev), probs;
  if (a[7] == Py_True) probs = make({b, hq, sq, sk}, at::kFloat, dev);
  at::Tensor ws = scratch(api.score_ws(b, hq, sq, sk, (int)d), dev);
  TqScoreJob j{};
  j.q = q.data_ptr(); j.q_dtype = dtype_of(q); j.D = (int32_t)d; j.bits = (int32_t)bits;
  j.B = b; j.Hq = hq; j.Sq = sq; j.Hkv = hkv; j.Sk = sk;
  j.idx_bytes = (const uint8_t*)idx.data_ptr(); j.norms = (const uint16_t*)norms.data_ptr();
  j.rotation_t = (const float*)pi_t.data_ptr(); j.codebook = (const float*)cb.data_ptr(); j.scale = scale;
  j.logits = (float*)logits.data_ptr(); j.probs = probs.defined() ? (float*)probs.data_ptr() : nullptr;
  j.workspace = ws.data_ptr(); j.workspace_bytes = (size_t)ws.numel();
  void* st = stream_of(dev);
  if (!call("tq_score_packed", [&] { return api.score_packed(&j, st); })) return nullptr;
  Ref l(THPVariable_Wrap(logits));
  if (!l || !probs.defined()) return l.release();
  Ref p(THPVariable_Wrap(probs));
  return p ? PyTuple_Pack(2, l.p, p.p) : nullptr;
  END_HANDLE_TH_ERRORS
}

// decode_attention(q, k dict, v dict, key_codec, value_codec, k_window, v_window, scale) -> fp32 of q's shape | None
PyObject* decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TQ_NAME(k_idx, "idx_bytes"); TQ_NAME(k_norms, "vec_norms");
  const int dev = c10::cuda::current_device();
  float scale;
  if (n != 8 || !float_plain(a[0], dev) || !PyDict_CheckExact(a[1]) || !PyDict_CheckExact(a[2]) || !float_plain(a[5], dev) ||
      !float_plain(a[6], dev) || !number(a[7], &scale))
    return none();
  const at::Tensor &q = THPVariable_Unpack(a[0]), &kw = THPVariable_Unpack(a[5]), &vw = THPVariable_Unpack(a[6]);
  if (q.dim() != 4 || q.size(3) != 128 || !q.is_contiguous()) return none();
  const int64_t b = q.size(0), hq = q.size(1), sq = q.size(2);
  Codec codec[2];
  at::Tensor idx[2], norms[2];                        // held until the launch is out
  for (int i = 0; i < 2; ++i) {
    PyObject *io = PyDict_GetItem(a[1 + i], k_idx), *no = PyDict_GetItem(a[1 + i], k_norms);
    if (io == nullptr || no == nullptr || !plain(io, dev) || !plain(no, dev) || !read_codec(a[3 + i], dev, &codec[i]) || codec[i].dim != 128) return none();
    idx[i] = THPVariable_Unpack(io);
    norms[i] = THPVariable_Unpack(no);
    if (idx[i].dim() != 4 || norms[i].dim() != 3) return none();
  }
  const int64_t hkv = idx[0].size(1), sk = idx[0].size(2);
  if (hkv < 1 || hq % hkv != 0) return none();
  for (int i = 0; i < 2; ++i)
    if (!is(idx[i], at::kByte, {b, hkv, sk, row_bytes(128, codec[i].bits)}) || !is(norms[i], at::kHalf, {b, hkv, sk})) return none();
  if (kw.dim() != 4 || kw.sizes() != vw.sizes() || kw.scalar_type() != vw.scalar_type() || kw.strides() != vw.strides()) return none();
  const int64_t w = kw.size(2);
  if (w > 0 && (kw.size(0) != b || kw.size(1) != hkv || kw.size(3) != 128 || kw.stride(3) != 1)) return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor out = make({b, hq, sq, 128}, at::kFloat, dev);
  at::Tensor ws = scratch(api.decode_attention_ws(b, hq, sq, sk), dev);
  TqDecodeAttnJob j{};
  j.q = q.data_ptr(); j.q_dtype = dtype_of(q); j.D = 128; j.key_bits = (int32_t)codec[0].bits; j.value_bits = (int32_t)codec[1].bits;
  j.B = b; j.Hq = hq; j.Sq = sq; j.Hkv = hkv; j.Sk = sk;
  j.k_idx = (const uint8_t*)idx[0].data_ptr(); j.k_norms = (const uint16_t*)norms[0].data_ptr();
  j.v_idx = (const uint8_t*)idx[1].data_ptr(); j.v_norms = (const uint16_t*)norms[1].data_ptr();
  j.k_rotation_t = (const float*)codec[0].pi_t; j.v_rotation = (const float*)codec[1].pi;
  j.k_codebook = (const float*)codec[0].cb; j.v_codebook = (const float*)codec[1].cb;
  j.window_dtype = w > 0 ? dtype_of(kw) : TQ_F16;
  if (w > 0) {
    j.k_window = kw.data_ptr(); j.v_window = vw.data_ptr(); j.W = w;
    j.wstride_b = kw.stride(0); j.wstride_h = kw.stride(1); j.wstride_s = kw.stride(2);
  }
  j.scale = scale;
  j.out = (float*)out.data_ptr(); j.workspace = ws.data_ptr(); j.workspace_bytes = (size_t)ws.numel();
  void* st = stream_of(dev);
  if (!call("tq_decode_attention", [&] { return api.decode_attention(&j, st); })) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// qjl_scores_packed(q, rows, sign_bits, vec_norms, rnorm, pi_t, qjl_t, codebook, bits) -> fp32 (B, H, Sq, Sk) | None
PyObject* qjl_scores_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const int dev = c10::cuda::current_device();
  int64_t bits;
  if (n != 9 || !float_plain(a[0], dev) || !bit_width(a[8], &bits)) return none();
  for (int i = 1; i < 8; ++i)
    if (!plain(a[i], dev)) return none();
  const at::Tensor &q = THPVariable_Unpack(a[0]), &rows = THPVariable_Unpack(a[1]), &sb = THPVariable_Unpack(a[2]), &vn = THPVariable_Unpack(a[3]),
                   &rn = THPVariable_Unpack(a[4]), &pi_t = THPVariable_Unpack(a[5]), &qt = THPVariable_Unpack(a[6]), &cb = THPVariable_Unpack(a[7]);
  if (q.dim() != 4 || rows.dim() != 4 || !q.is_contiguous()) return none();
  const int64_t b = q.size(0), h = q.size(1), sq = q.size(2), d = q.size(3), sk = rows.size(2);
  if ((d != 128 && d != 256) || !is(rows, at::kByte, {b, h, sk, row_bytes(d, bits)}) || !is(sb, at::kByte, {b, h, sk, d / 8}) ||
      !is(vn, at::kFloat, {b, h, sk}) || !is(rn, at::kHalf, {b, h, sk}) || !is(pi_t, at::kFloat, {d, d}) || !is(qt, at::kFloat, {d, d}) ||
      cb.scalar_type() != at::kFloat || cb.numel() != TQ_CODEBOOK_FLOATS || !cb.is_contiguous())
    return none();
  c10::AutoGradMode no_grad(false);
  at::Tensor out = make({b, h, sq, sk}, at::kFloat, dev);
  at::Tensor ws = scratch(api.qjl_scores_packed_ws(b * h, sq, (int)d), dev);
  TqQjlPackedScoreJob j{};
  j.q = q.data_ptr(); j.q_dtype = dtype_of(q); j.D = (int32_t)d; j.bits = (int32_t)bits; j.BH = b * h; j.Sq = sq; j.Sk = sk;
  j.idx_packed = (const uint8_t*)rows.data_ptr(); j.sign_bits = (const uint8_t*)sb.data_ptr(); j.vec_norms = (const float*)vn.data_ptr();
  j.rnorm = (const uint16_t*)rn.data_ptr(); j.rotation_t = (const float*)pi_t.data_ptr(); j.qjl_t = (const float*)qt.data_ptr();
  j.codebook = (const float*)cb.data_ptr(); j.scores = (float*)out.data_ptr(); j.workspace = ws.data_ptr(); j.workspace_bytes = (size_t)ws.numel();
  void* st = stream_of(dev);
  if (!call("tq_qjl_scores_packed", [&] { return api.qjl_scores_packed(&j, st); })) return nullptr;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------- one token for every layer (V3Cache.step)
struct StepPlan {
  std::vector<TqQuantizeJob> q;
  std::vector<TqDequantizeJob> d;
  std::vector<TqCopyJob> c;
  std::vector<int64_t> row, base, size_a, size_b;
  int64_t L = 0, B = 0, H = 0, D = 0, cap = 0, window = 0, tok_bytes = 0;
  int dtype = 0, dev = 0;
};
const char* const kPlanName = "turboquant.step_plan";
void free_plan(PyObject* cap) { delete static_cast<StepPlan*>(PyCapsule_GetPointer(cap, kPlanName)); }

// step_plan(layer states, window) -> capsule | None.  Fills in what does not change from step to step: the layers'
// buffers (equal shape, strides of their own, capacity the least of all), codecs and constants.
PyObject* step_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TQ_NAME(n_k, "k"); TQ_NAME(n_v, "v"); TQ_NAME(n_codec, "codec"); TQ_NAME(n_kc, "key_compressor"); TQ_NAME(n_vc, "val_compressor");
  if (n != 2 || !PyList_CheckExact(a[0]) || PyList_GET_SIZE(a[0]) < 1 || !PyLong_Check(a[1])) return none();
  const int dev = c10::cuda::current_device();
  auto* p = new StepPlan;
  Ref cap(PyCapsule_New(p, kPlanName, free_plan));
  if (!cap) { delete p; return nullptr; }
  p->L = PyList_GET_SIZE(a[0]);
  p->window = PyLong_AsLongLong(a[1]);
  p->dev = dev;
  const size_t jobs = (size_t)(2 * p->L);
  p->q.assign(jobs, TqQuantizeJob{}); p->d.assign(jobs, TqDequantizeJob{}); p->c.assign(jobs, TqCopyJob{});
  p->row.resize(jobs); p->base.resize(jobs); p->size_a.resize(jobs); p->size_b.resize(jobs);
  for (size_t i = 0; i < jobs; ++i) {
    PyObject* st = PyList_GET_ITEM(a[0], (Py_ssize_t)(i / 2));
    Ref buf(PyObject_GetAttr(st, (i & 1) ? n_v : n_k)), codec(PyObject_GetAttr(st, n_codec));
    Ref comp(codec ? PyObject_GetAttr(codec.p, (i & 1) ? n_vc : n_kc) : nullptr);
    Codec c;
    if (!buf || !comp) { PyErr_Clear(); return none(); }
    if (!float_plain(buf.p, dev) || !read_codec(comp.p, dev, &c)) return none();
    const at::Tensor& t = THPVariable_Unpack(buf.p);
    if (t.dim() != 4 || t.stride(3) != 1 || t.size(3) != c.dim) return none();
    if (i == 0) {
      p->B = t.size(0); p->H = t.size(1); p->D = t.size(3); p->cap = t.size(2);
      p->dtype = dtype_of(t);
      p->tok_bytes = p->D * (int64_t)t.element_size();
    }
    if (t.size(0) != p->B || t.size(1) != p->H || t.size(3) != p->D || dtype_of(t) != p->dtype || t.stride(2) != p->D) return none();
    if (t.size(2) < p->cap) p->cap = t.size(2);
    p->row[i] = row_bytes(p->D, c.bits);
    p->base[i] = (int64_t)(uintptr_t)t.data_ptr();
    TqQuantizeJob& q = p->q[i];
    q.x_dtype = p->dtype; q.D = (int32_t)p->D; q.bits = (int32_t)c.bits; q.normalize = 1;
    q.B = p->B; q.H = p->H; q.stride_b = t.stride(0); q.stride_h = t.stride(1); q.stride_s = t.stride(2);
    q.rotation_t = (const float*)c.pi_t; q.codebook = (const float*)c.cb; q.idx_mode = TQ_IDX_PACKED; q.rotation_image = c.img_q;
    TqDequantizeJob& d = p->d[i];
    d.idx_mode = TQ_IDX_PACKED; d.D = (int32_t)p->D; d.bits = (int32_t)c.bits; d.out_dtype = p->dtype;
    d.B = p->B; d.H = p->H; d.ostride_b = t.stride(0); d.ostride_h = t.stride(1); d.ostride_s = t.stride(2);
    d.rotation = (const float*)c.pi; d.codebook = (const float*)c.cb; d.rotation_image = c.img_d;
    TqCopyJob& k = p->c[i];
    k.elem_bytes = (int32_t)t.element_size(); k.D = (int32_t)p->D; k.B = p->B; k.H = p->H;
    k.dstride_b = t.stride(0); k.dstride_h = t.stride(1); k.dstride_s = t.stride(2);
  }
  return cap.release();
  END_HANDLE_TH_ERRORS
}

// step(plan, layer states, keys, values, return_views, log) -> list of views | False (no views wanted) | None.  What left the
// window goes into `log` as ONE entry (store, bytes of int64: first token, tokens, four offsets of every layer): an
// entry per layer would be 64 more objects a step for the garbage collector to walk, for ever (118 -> 140 to 410 us).
PyObject* step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TQ_NAME(n_total, "total"); TQ_NAME(n_comp, "compressed"); TQ_NAME(n_k, "k"); TQ_NAME(n_v, "v");
  if (n != 6 || !PyList_CheckExact(a[5]) || !PyCapsule_IsValid(a[0], kPlanName)) return none();
  StepPlan& p = *static_cast<StepPlan*>(PyCapsule_GetPointer(a[0], kPlanName));
  const int dev = c10::cuda::current_device();
  if (dev != p.dev || !PyList_CheckExact(a[1]) || PyList_GET_SIZE(a[1]) != p.L) return none();
  Ref ks(PySequence_Fast(a[2], "keys")), vs(PySequence_Fast(a[3], "values"));
  if (!ks || !vs || PySequence_Fast_GET_SIZE(ks.p) != p.L || PySequence_Fast_GET_SIZE(vs.p) != p.L) { PyErr_Clear(); return none(); }
  const bool views = PyObject_IsTrue(a[4]) == 1;
  // look every layer over first: nothing has changed yet when the general path has to take the call
  int64_t s_new = -1;
  std::vector<int64_t> total((size_t)p.L), comp((size_t)p.L), leave((size_t)p.L);
  for (int64_t l = 0; l < p.L; ++l) {
    PyObject* st = PyList_GET_ITEM(a[1], l);
    if (!attr_int(st, n_total, &total[l]) || !attr_int(st, n_comp, &comp[l])) return none();
    for (int j = 0; j < 2; ++j) {
      PyObject* o = PySequence_Fast_GET_ITEM(j ? vs.p : ks.p, l);
      if (!float_plain(o, dev)) return none();
      const at::Tensor& x = THPVariable_Unpack(o);
      if (x.dim() != 4 || dtype_of(x) != p.dtype || x.size(0) != p.B || x.size(1) != p.H || x.size(3) != p.D || x.stride(3) != 1) return none();
      if (s_new < 0) s_new = x.size(2);
      if (x.size(2) != s_new) return none();
    }
    if (total[l] + s_new > p.cap) return none();
    const int64_t recent = total[l] + s_new - comp[l];
    leave[l] = p.window == 0 ? recent : (recent > p.window ? recent - p.window : 0);
  }
  if (s_new < 1 || p.D * (p.dtype == TQ_F32 ? 4 : 2) % 16 != 0) return none();
  c10::AutoGradMode no_grad(false);
  const int64_t slabs = p.B * p.H;
  int64_t bytes = 0;
  for (int64_t i = 0; i < 2 * p.L; ++i) {
    const int64_t rows = slabs * leave[i / 2];
    p.size_a[i] = (rows * p.row[i] + 15) / 16 * 16;
    p.size_b[i] = (2 * rows + 15) / 16 * 16;
    bytes += p.size_a[i] + p.size_b[i];
  }
  at::Tensor store;                                   // this step's packed rows and norms of every layer
  uint8_t* sp = nullptr;
  Ref store_obj;
  if (bytes > 0) {
    store = make({bytes < 16 ? 16 : bytes}, at::kByte, dev);
    sp = (uint8_t*)store.data_ptr();
    store_obj.p = THPVariable_Wrap(store);
    if (!store_obj) return nullptr;
  }
  int64_t off = 0;
  std::vector<int64_t> offs((size_t)(4 * p.L));
  for (int64_t i = 0; i < 2 * p.L; ++i) {
    const int64_t l = i / 2;
    const at::Tensor& x = THPVariable_Unpack(PySequence_Fast_GET_ITEM((i & 1) ? vs.p : ks.p, l));
    TqCopyJob& c = p.c[i];
    c.src = x.data_ptr(); c.S = s_new;
    c.sstride_b = x.stride(0); c.sstride_h = x.stride(1); c.sstride_s = x.stride(2);
    c.dst = (void*)(p.base[i] + total[l] * p.tok_bytes);
    void* slot = (void*)(p.base[i] + comp[l] * p.tok_bytes);
    p.q[i].S = p.d[i].S = leave[l];
    p.q[i].x = slot; p.d[i].out = slot;
    p.q[i].idx_out = sp + off; p.d[i].idx = sp + off;
    offs[2 * i] = off;
    off += p.size_a[i];
    p.q[i].norms_out = (uint16_t*)(sp + off); p.d[i].norms = (const uint16_t*)(sp + off);
    offs[2 * i + 1] = off;
    off += p.size_b[i];
  }
  void* st = stream_of(dev);
  const int jobs = (int)(2 * p.L);
  if (!call("tq_copy_rows", [&] { return api.copy_rows(p.c.data(), jobs, st); })) return nullptr;
  if (bytes > 0) {
    if (!call("tq_quantize", [&] { return api.quantize(p.q.data(), jobs, st); })) return nullptr;
    if (!call("tq_dequantize", [&] { return api.dequantize(p.d.data(), jobs, st); })) return nullptr;
  }
  Ref out(views ? PyList_New(p.L) : PyBool_FromLong(0));
  if (!out) return nullptr;
  if (bytes > 0) {
    std::vector<int64_t> record;
    record.reserve((size_t)(6 * p.L));
    record.insert(record.end(), comp.begin(), comp.end());
    record.insert(record.end(), leave.begin(), leave.end());
    record.insert(record.end(), offs.begin(), offs.end());
    Ref blob(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(record.data()), (Py_ssize_t)(record.size() * sizeof(int64_t))));
    Ref entry(blob ? PyTuple_Pack(2, store_obj.p, blob.p) : nullptr);
    if (!entry || PyList_Append(a[5], entry.p) != 0) return nullptr;
  }
  for (int64_t l = 0; l < p.L; ++l) {
    PyObject* lay = PyList_GET_ITEM(a[1], l);
    Ref t(PyLong_FromLongLong(total[l] + s_new)), c(PyLong_FromLongLong(comp[l] + leave[l]));
    if (!t || !c || PyObject_SetAttr(lay, n_total, t.p) != 0 || PyObject_SetAttr(lay, n_comp, c.p) != 0) return nullptr;
    if (views) {
      Ref k(PyObject_GetAttr(lay, n_k)), v(PyObject_GetAttr(lay, n_v));
      if (!k || !v) return nullptr;
      Ref kv(THPVariable_Wrap(tokens(THPVariable_Unpack(k.p), 0, total[l] + s_new)));
      Ref vv(THPVariable_Wrap(tokens(THPVariable_Unpack(v.p), 0, total[l] + s_new)));
      if (!kv || !vv) return nullptr;
      PyObject* pair = PyTuple_Pack(2, kv.p, vv.p);
      if (pair == nullptr) return nullptr;
      PyList_SET_ITEM(out.p, l, pair);
    }
  }
  return out.release();
  END_HANDLE_TH_ERRORS
}

// bind(addresses of the C functions in the order of Api, check, the four job methods)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  constexpr int kFns = 12;
  void* p[kFns];
  if (n != kFns + 2 || !PyTuple_Check(a[kFns + 1]) || PyTuple_GET_SIZE(a[kFns + 1]) != 4) {
    PyErr_SetString(PyExc_TypeError, "bind takes twelve addresses, a function and a tuple of four");
    return nullptr;
  }
  for (int i = 0; i < kFns; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (p[i] == nullptr) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address"); return nullptr; }
  }
  api.quantize = (decltype(api.quantize))p[0]; api.dequantize = (decltype(api.dequantize))p[1];
  api.copy_rows = (decltype(api.copy_rows))p[2]; api.qjl_compress = (decltype(api.qjl_compress))p[3];
  api.qjl_compress_ws = (decltype(api.qjl_compress_ws))p[4]; api.prod_inner = (decltype(api.prod_inner))p[5];
  api.score_packed = (decltype(api.score_packed))p[6]; api.score_ws = (decltype(api.score_ws))p[7];
  api.decode_attention = (decltype(api.decode_attention))p[8]; api.decode_attention_ws = (decltype(api.decode_attention_ws))p[9];
  api.qjl_scores_packed = (decltype(api.qjl_scores_packed))p[10]; api.qjl_scores_packed_ws = (decltype(api.qjl_scores_packed_ws))p[11];
  Py_INCREF(a[kFns]);
  Py_XDECREF(api.check);
  api.check = a[kFns];
  Py_INCREF(a[kFns + 1]);
  Py_XDECREF(api.jobs);
  api.jobs = a[kFns + 1];
  Py_RETURN_NONE;
}

#define TQ_FN(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {TQ_FN(bind), TQ_FN(compress_kv), TQ_FN(decompress_kv), TQ_FN(compress), TQ_FN(decompress),
                         TQ_FN(quantize_rows), TQ_FN(dequantize_rows), TQ_FN(prod_inner), TQ_FN(qjl_compress), TQ_FN(score_packed),
                         TQ_FN(decode_attention), TQ_FN(qjl_scores_packed),
                         TQ_FN(step_plan), TQ_FN(step), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_tq_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__tq_host(void) { return PyModule_Create(&module); }
