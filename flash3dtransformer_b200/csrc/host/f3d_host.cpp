// Operator calls without Python in between: the argument checks, the pointers, the stream and the call of the C entry point for
// the operators whose own work on the device is shorter than the interpreter's on the host.  A call through ctypes costs 8 to 12
// us of host time before the first launch (checks on every tensor, conversion of ten to twenty arguments); here it is below one.
//
// Every function either makes the call and returns its status, or returns None when an argument is not what the operator takes:
// the caller's own checks then find the reason and raise it, so messages and exceptions live in one place.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/f3d_b200.h"

namespace {

// entry points of libf3d_b200.so, handed over by bind()
struct Entry {
  decltype(&f3d_linear_dtype) linear = nullptr;
  decltype(&f3d_buck_swin_fwd_dtype) swin_fwd = nullptr;
  decltype(&f3d_batch_psh_scatter_pad_hash) scatter = nullptr;
  decltype(&f3d_scatter_index) index = nullptr;
  decltype(&f3d_bbox_f16) bbox = nullptr;
} g_entry;

struct Bad {};                                        // not a call that is made here

const at::Tensor &tensor(PyObject *o) {
  if (!THPVariable_Check(o)) throw Bad{};
  return THPVariable_Unpack(o);
}
// contiguous, on CUDA device `dev` (set by the first tensor), of the type asked for
const at::Tensor &checked(PyObject *o, int &dev, at::ScalarType type) {
  const at::Tensor &t = tensor(o);
  if (!t.is_cuda() || !t.is_contiguous() || t.scalar_type() != type) throw Bad{};
  if (dev < 0) dev = t.get_device();
  else if (t.get_device() != dev) throw Bad{};
  return t;
}
long long integer(PyObject *o) {
  if (!PyLong_CheckExact(o)) throw Bad{};
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); throw Bad{}; }
  return v;
}
uint32_t u32(PyObject *o) {
  const long long v = integer(o);
  if (v < 0 || v > 0xFFFFFFFFll) throw Bad{};
  return (uint32_t)v;
}
int i32(int64_t v) {
  if (v < 0 || v > 0x7FFFFFFF) throw Bad{};
  return (int)v;
}
void want(bool ok) { if (!ok) throw Bad{}; }
void *stream(int dev) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }

template <class F> PyObject *call(F &&f) {
  try {
    return PyLong_FromLong(f());
  } catch (const Bad &) {
  } catch (const std::exception &) {
  }
  Py_RETURN_NONE;
}
template <class F> int without_gil(F &&f) {
  PyThreadState *const s = PyEval_SaveThread();
  const int st = f();
  PyEval_RestoreThread(s);
  return st;
}
int float_code(at::ScalarType t) { return t == at::kBFloat16 ? 0 : 1; }

// (x, weight, bias or None, out, residual or None, nsplit, epilogue)
PyObject *linear(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return call([&] {
    want(n == 7 && g_entry.linear);
    int dev = -1;
    const at::ScalarType type = tensor(a[0]).scalar_type();
    want(type == at::kBFloat16 || type == at::kHalf);
    const at::Tensor &x = checked(a[0], dev, type), &w = checked(a[1], dev, type), &out = checked(a[3], dev, type);
    const long long nsplit = integer(a[5]), epilogue = integer(a[6]);
    want(x.dim() == 2 && w.dim() == 2 && w.size(1) == x.size(1) && nsplit > 0 && nsplit < 1024 && epilogue >= 0 && epilogue < 1024);
    const int64_t m = x.size(0), k = x.size(1), cols = w.size(0), out_n = epilogue == 2 ? cols / 2 : cols;
    want(out.numel() == m * out_n);
    const void *bias = nullptr, *res = nullptr;
    if (a[2] != Py_None) {
      const at::Tensor &b = checked(a[2], dev, at::kFloat);
      want(b.numel() == cols);
      bias = b.data_ptr();
    }
    if (a[4] != Py_None) {
      const at::Tensor &r = checked(a[4], dev, type);
      want(r.dim() == 2 && r.size(0) == m && r.size(1) == out_n);
      res = r.data_ptr();
    }
    const int M = i32(m), N = i32(cols), K = i32(k);
    const void *xp = x.data_ptr(), *wp = w.data_ptr();
    void *op = out.data_ptr(), *st = stream(dev);
    return without_gil([&] { return g_entry.linear(xp, wp, bias, res, op, M, N, K, (int)nsplit, (int)epilogue, float_code(type), dev, st); });
  });
}

// (Q, K, V, O, L, Scope_buckets, bucket_size)
PyObject *swin_fwd(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return call([&] {
    want(n == 7 && g_entry.swin_fwd);
    int dev = -1;
    const at::ScalarType type = tensor(a[0]).scalar_type();
    want(type == at::kBFloat16 || type == at::kHalf);
    const at::Tensor &q = checked(a[0], dev, type), &k = checked(a[1], dev, type), &v = checked(a[2], dev, type), &o = checked(a[3], dev, type),
                     &l = checked(a[4], dev, at::kFloat), &s = checked(a[5], dev, at::kUInt32);
    const uint32_t bucket = u32(a[6]);
    want(q.dim() == 4 && k.sizes() == q.sizes() && v.sizes() == q.sizes() && o.sizes() == q.sizes() && s.dim() == 2);
    want(l.dim() == 3 && l.size(0) == q.size(0) && l.size(1) == q.size(1) && l.size(2) == q.size(2));
    const int B = i32(q.size(0)), L = i32(q.size(1)), H = i32(q.size(2)), D = i32(q.size(3)), scopes = i32(s.size(0)), size = i32(s.size(1));
    const void *qp = q.data_ptr(), *kp = k.data_ptr(), *vp = v.data_ptr(), *sp = s.data_ptr();
    void *op = o.data_ptr(), *lp = l.data_ptr(), *st = stream(dev);
    return without_gil([&] { return g_entry.swin_fwd(qp, kp, vp, op, lp, sp, B, L, H, D, scopes, size, bucket, float_code(type), dev, st); });
  });
}

// (coord, bucket_id, bucket_counter, bucket_offset, batch_sep, instance_max_N, num_bucket, bucket_divisor, bucket_size, num_vox,
//  bbox_min, bbox_max, probe_offsets, cumsum_counter, scatter_coord, pad_num, hash_type)
PyObject *scatter(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return call([&] {
    want(n == 17 && g_entry.scatter);
    int dev = -1;
    const at::Tensor &c = checked(a[0], dev, at::kHalf), &id = checked(a[1], dev, at::kUInt16), &cnt = checked(a[2], dev, at::kUInt32),
                     &off = checked(a[3], dev, at::kUInt32), &sep = checked(a[4], dev, at::kUInt32), &lo = checked(a[10], dev, at::kHalf),
                     &hi = checked(a[11], dev, at::kHalf), &probe = checked(a[12], dev, at::kShort), &sum = checked(a[13], dev, at::kUInt32),
                     &out = checked(a[14], dev, at::kHalf);
    const uint32_t max_n = u32(a[5]), nb = u32(a[6]), divisor = u32(a[7]), cap = u32(a[8]), vox = u32(a[9]), hash = u32(a[16]);
    want(PyFloat_CheckExact(a[15]));
    const float pad = (float)PyFloat_AS_DOUBLE(a[15]);
    want(c.dim() == 2 && c.size(1) == 3 && out.dim() == 2 && out.size(1) == 3 && sep.dim() >= 1);
    const int64_t total = c.size(0), batch = sep.size(0);
    want(id.numel() >= total && off.numel() >= total && cnt.numel() == batch * (int64_t)nb && sum.numel() == batch * (int64_t)nb &&
         probe.numel() == 128 * 3 && lo.numel() == 3 && hi.numel() == 3 && total <= 0x7FFFFFFF && batch <= 0x7FFFFFFF && out.size(0) <= 0x7FFFFFFF);
    void *idp = id.data_ptr(), *cp = cnt.data_ptr(), *fp = off.data_ptr(), *up = sum.data_ptr(), *op = out.data_ptr(), *st = stream(dev);
    const void *xp = c.data_ptr(), *sp = sep.data_ptr(), *lp = lo.data_ptr(), *hp = hi.data_ptr(), *pp = probe.data_ptr();
    const uint32_t pad_to = (uint32_t)out.size(0);
    return without_gil([&] {
      return g_entry.scatter(xp, idp, cp, fp, sp, (uint32_t)total, (uint32_t)batch, max_n, nb, divisor, cap, vox, lp, hp, pp, up, op, pad_to, pad,
                             hash, dev, st);
    });
  });
}

// (bucket_id, bucket_offset, cumsum_counter, batch_sep, out2in, in2out or None)
PyObject *index(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return call([&] {
    want(n == 6 && g_entry.index);
    int dev = -1;
    const at::Tensor &id = checked(a[0], dev, at::kUInt16), &off = checked(a[1], dev, at::kUInt32), &sum = checked(a[2], dev, at::kUInt32),
                     &sep = checked(a[3], dev, at::kUInt32), &o2i = checked(a[4], dev, at::kUInt32);
    const int64_t pts = id.numel();
    want(off.numel() == pts && sum.dim() == 2 && sum.size(0) == sep.numel() && o2i.numel() >= pts && o2i.numel() <= 0x7FFFFFFF);
    void *i2o = nullptr;
    if (a[5] != Py_None) {
      const at::Tensor &t = checked(a[5], dev, at::kUInt32);
      want(t.numel() == pts);
      i2o = t.data_ptr();
    }
    const void *ip = id.data_ptr(), *fp = off.data_ptr(), *up = sum.data_ptr(), *sp = sep.data_ptr();
    void *op = o2i.data_ptr(), *st = stream(dev);
    const uint32_t batch = (uint32_t)sep.numel(), nb = (uint32_t)sum.size(1), rows = (uint32_t)o2i.numel();
    return without_gil([&] { return g_entry.index(ip, fp, up, sp, op, i2o, (uint32_t)pts, batch, nb, rows, dev, st); });
  });
}

// (coords, bbox_min, bbox_max)
PyObject *bbox(PyObject *, PyObject *const *a, Py_ssize_t n) {
  return call([&] {
    want(n == 3 && g_entry.bbox);
    int dev = -1;
    const at::Tensor &c = checked(a[0], dev, at::kHalf), &lo = checked(a[1], dev, at::kHalf), &hi = checked(a[2], dev, at::kHalf);
    want(c.dim() == 2 && c.size(1) == 3 && lo.numel() == 3 && hi.numel() == 3 && c.size(0) <= 0x7FFFFFFF);
    const void *cp = c.data_ptr();
    void *lp = lo.data_ptr(), *hp = hi.data_ptr(), *st = stream(dev);
    const uint32_t rows = (uint32_t)c.size(0);
    return without_gil([&] { return g_entry.bbox(cp, lp, hp, rows, dev, st); });
  });
}

// empties(device, code, rows, cols, code, rows, cols, ...): uninitialised tensors [rows, cols], or [rows] where cols is 0; code 0
// uint16, 1 uint32, 2 float16.  None where a tensor cannot be made here.
PyObject *empties(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n < 4 || n % 3 != 1 || n > 31) Py_RETURN_NONE;
  at::Tensor out[10];
  const Py_ssize_t count = n / 3;
  try {
    const at::Device dev(at::kCUDA, (c10::DeviceIndex)u32(a[0]));
    for (Py_ssize_t i = 0; i < count; ++i) {
      const long long code = integer(a[3 * i + 1]), rows = integer(a[3 * i + 2]), cols = integer(a[3 * i + 3]);
      want(code >= 0 && code < 3 && rows >= 0 && cols >= 0);
      const at::TensorOptions opt = at::TensorOptions().device(dev).dtype(code == 0 ? at::kUInt16 : code == 1 ? at::kUInt32 : at::kHalf);
      const int64_t size[2] = {rows, cols};
      out[i] = at::empty(at::IntArrayRef(size, cols ? 2 : 1), opt);
    }
  } catch (const Bad &) {
    Py_RETURN_NONE;
  } catch (const std::exception &) {           // the caller's own allocation raises it
    Py_RETURN_NONE;
  }
  PyObject *const t = PyTuple_New(count);
  if (!t) return nullptr;
  for (Py_ssize_t i = 0; i < count; ++i) PyTuple_SET_ITEM(t, i, THPVariable_Wrap(std::move(out[i])));
  return t;
}

// bind(linear, swin_fwd, scatter, index, bbox): addresses of the C entry points
PyObject *bind(PyObject *, PyObject *const *a, Py_ssize_t n) {
  void *p[5];
  if (n != 5) { PyErr_SetString(PyExc_TypeError, "five addresses"); return nullptr; }
  for (int i = 0; i < 5; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (!p[i] && PyErr_Occurred()) return nullptr;
  }
  g_entry.linear = reinterpret_cast<decltype(g_entry.linear)>(p[0]);
  g_entry.swin_fwd = reinterpret_cast<decltype(g_entry.swin_fwd)>(p[1]);
  g_entry.scatter = reinterpret_cast<decltype(g_entry.scatter)>(p[2]);
  g_entry.index = reinterpret_cast<decltype(g_entry.index)>(p[3]);
  g_entry.bbox = reinterpret_cast<decltype(g_entry.bbox)>(p[4]);
  Py_RETURN_NONE;
}

#define F3D_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {F3D_METHOD(linear), F3D_METHOD(swin_fwd), F3D_METHOD(scatter), F3D_METHOD(index),
                           F3D_METHOD(bbox), F3D_METHOD(empties), F3D_METHOD(bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_f3d_host", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__f3d_host(void) { return PyModule_Create(&g_module); }
