// Native host path of the module forwards: one call from Python per layer call.
//
// A layer call launches two to four kernels that take 20 to 100 us together; prepared in Python
// (attribute walks, argument checks, thirty ctypes conversions: 55 to 60 us) every call below about
// 10k tokens would be bound by the host.  Here the facts that do not change between
// calls (weight addresses, shapes, packed copies) are kept in a plan, and a call only checks that
// the plan still describes the module, allocates the outputs and enters the C ABI.
//
// The plan never serves stale weights: each of its links names the dictionary slot a parameter, a
// sub-module or a packed image sits in, and a call compares what is in the slot now (object, storage
// address, version counter) with what the plan was made from.  A mismatch returns None and the caller
// makes a new plan.  (Writes past the version counter are announced by emptying the image's slot.)
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/core/CachingHostAllocator.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <memory>
#include <vector>

#include "../../include/d2dmoe.h"

namespace {

struct Link {
  PyObject* dict;      // slot holder; null: roots[root]
  int root;
  PyObject* key;
  PyObject* obj;       // what the slot held when the plan was made
  const void* data;    // tensors: storage address and version counter
  int64_t version;
  bool tensor;
};

struct Plan {
  std::vector<Link> links;
  at::Tensor hold[2];                  // packed router / experts images
  PyObject* marks[2] = {};             // behind the kernels that wrote them (capsules of a Mark), or null
  std::vector<cudaStream_t> users;     // other streams that have waited for those
  const void *wa = nullptr, *wb = nullptr, *rp = nullptr;
  const void *w1 = nullptr, *b1 = nullptr, *wup = nullptr, *w2 = nullptr, *ep = nullptr;
  const void* last_bias = nullptr;
  int64_t d = 0, R = 0, E = 0, H = 0, act = 0;
  at::ScalarType dtype = at::kFloat;
  c10::Device device = c10::Device(c10::kCUDA, 0);
  ~Plan() {
    for (PyObject* m : marks) Py_XDECREF(m);
    for (Link& l : links) {
      Py_XDECREF(l.dict);
      Py_XDECREF(l.key);
      Py_XDECREF(l.obj);
    }
  }
};

constexpr const char* kPlan = "d2dmoe_b200.plan";

void plan_free(PyObject* cap) { delete static_cast<Plan*>(PyCapsule_GetPointer(cap, kPlan)); }

const at::Tensor* tensor_of(PyObject* o) {
  return o != nullptr && THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr;
}

const void* ptr_of(PyObject* o) {
  const at::Tensor* t = tensor_of(o);
  return t ? t->data_ptr() : nullptr;
}

bool still_valid(const Plan& p, PyObject* const* roots) {
  for (const Link& l : p.links) {
    PyObject* now = PyDict_GetItemWithError(l.dict ? l.dict : roots[l.root], l.key);   // borrowed
    if (now != l.obj) return false;
    if (l.tensor) {
      const at::Tensor& t = THPVariable_Unpack(now);
      if (t.data_ptr() != l.data || t._version() != l.version) return false;
    }
  }
  return !PyErr_Occurred();
}

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing(s, &st));
  return st != cudaStreamCaptureStatusNone;
}

// The point of a stream behind the kernels that wrote a packed image.
struct Mark {
  cudaEvent_t event = nullptr;
  cudaStream_t stream = nullptr;
};
constexpr const char* kMark = "d2dmoe_b200.mark";
void mark_free(PyObject* cap) {
  Mark* m = static_cast<Mark*>(PyCapsule_GetPointer(cap, kMark));
  cudaEventDestroy(m->event);
  delete m;
}

// mark(device index) -> Mark of the current stream, or None while it captures (a graph's event means
// nothing outside it)
PyObject* mark(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 1, "mark(device index)");
  const auto dev = (c10::DeviceIndex)PyLong_AsLong(a[0]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::CUDAGuard guard(dev);
  auto m = std::make_unique<Mark>();
  m->stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  if (capturing(m->stream)) Py_RETURN_NONE;
  C10_CUDA_CHECK(cudaEventCreateWithFlags(&m->event, cudaEventDisableTiming));
  const cudaError_t err = cudaEventRecord(m->event, m->stream);
  if (err != cudaSuccess) cudaEventDestroy(m->event);
  C10_CUDA_CHECK(err);
  return PyCapsule_New(m.release(), kMark, mark_free);
  END_HANDLE_TH_ERRORS
}

// Before `s` reads the image: it comes behind the kernels that wrote it, and the allocator learns that
// `s` uses it.  (A capture cannot depend on work outside it; it starts behind that.)
void wait_for(const Mark* m, const at::Tensor& image, c10::cuda::CUDAStream s) {
  if (s.stream() == m->stream) return;
  C10_CUDA_CHECK(cudaStreamWaitEvent(s.stream(), m->event, 0));
  c10::cuda::CUDACachingAllocator::recordStream(image.storage().data_ptr(), s);
}

// wait_mark(mark, image): the current stream may read the image
PyObject* wait_mark(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  const at::Tensor* t = n == 2 ? tensor_of(a[1]) : nullptr;
  TORCH_CHECK(t, "wait_mark(mark, image)");
  const Mark* m = static_cast<const Mark*>(PyCapsule_GetPointer(a[0], kMark));
  if (!m) return nullptr;
  c10::cuda::CUDAGuard guard(t->device());
  const auto s = c10::cuda::getCurrentCUDAStream(t->device().index());
  if (s.stream() != m->stream && !capturing(s.stream())) wait_for(m, *t, s);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

void use_on(Plan& p, c10::cuda::CUDAStream s) {
  const Mark* m[2];
  bool other = false;
  for (int i = 0; i < 2; ++i) {
    m[i] = p.marks[i] ? static_cast<const Mark*>(PyCapsule_GetPointer(p.marks[i], kMark)) : nullptr;
    other |= m[i] && m[i]->stream != s.stream();
  }
  if (!other) return;
  for (cudaStream_t u : p.users)
    if (u == s.stream()) return;
  if (capturing(s.stream())) return;
  for (int i = 0; i < 2; ++i)
    if (m[i]) wait_for(m[i], p.hold[i], s);
  if (p.users.size() >= 16) p.users.clear();
  p.users.push_back(s.stream());
}

// make_plan(links, (wa, wb, router_packed, mark), (w1, b1, w_up, w2, experts_packed, mark), last_bias,
//           act, modules, parameters, attributes)
//   links: sequence of (holder, key); holder = a dict, or 0 / 1 / 2 for the module's own _modules /
//   _parameters / __dict__, which run_layer receives with every call (the plan does not refer to its
//   module)
PyObject* make_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "make_plan takes 8 arguments");
    return nullptr;
  }
  auto p = std::make_unique<Plan>();
  PyObject* const roots[3] = {a[5], a[6], a[7]};
  PyObject* seq = PySequence_Fast(a[0], "links");
  if (!seq) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) {
    PyObject* it = PySequence_Fast_GET_ITEM(seq, i);
    PyObject* holder = PyTuple_GetItem(it, 0);
    PyObject* key = PyTuple_GetItem(it, 1);
    if (!holder || !key) {
      Py_DECREF(seq);
      return nullptr;
    }
    Link l = {};
    if (PyLong_Check(holder)) {
      l.root = (int)PyLong_AsLong(holder);
      TORCH_CHECK(l.root >= 0 && l.root < 3, "link holder");
    } else {
      Py_INCREF(holder);
      l.dict = holder;
    }
    Py_INCREF(key);
    l.key = key;
    PyObject* now = PyDict_GetItemWithError(l.dict ? l.dict : roots[l.root], key);
    Py_XINCREF(now);
    l.obj = now;
    if (const at::Tensor* t = tensor_of(now)) {
      l.tensor = true;
      l.data = t->data_ptr();
      l.version = t->_version();
    }
    p->links.push_back(l);
  }
  Py_DECREF(seq);
  PyObject *r = a[1], *e = a[2];
  if (r != Py_None) {
    const at::Tensor* wa = tensor_of(PyTuple_GetItem(r, 0));
    TORCH_CHECK(wa, "router weight");
    p->wa = wa->data_ptr();
    p->wb = ptr_of(PyTuple_GetItem(r, 1));
    p->R = wa->size(0);
    if (const at::Tensor* t = tensor_of(PyTuple_GetItem(r, 2))) {
      p->hold[0] = *t;
      p->rp = t->data_ptr();
      if (PyObject* m = PyTuple_GetItem(r, 3); m && m != Py_None) p->marks[0] = Py_NewRef(m);
    }
  }
  const at::Tensor* w1 = tensor_of(PyTuple_GetItem(e, 0));
  TORCH_CHECK(w1 && w1->dim() == 3 && w1->is_cuda(), "expert weights");
  p->w1 = w1->data_ptr();
  p->b1 = ptr_of(PyTuple_GetItem(e, 1));
  p->wup = ptr_of(PyTuple_GetItem(e, 2));
  p->w2 = ptr_of(PyTuple_GetItem(e, 3));
  if (const at::Tensor* t = tensor_of(PyTuple_GetItem(e, 4))) {
    p->hold[1] = *t;
    p->ep = t->data_ptr();
    if (PyObject* m = PyTuple_GetItem(e, 5); m && m != Py_None) p->marks[1] = Py_NewRef(m);
  }
  p->E = w1->size(0);
  p->d = w1->size(1);
  p->H = w1->size(2);
  p->dtype = w1->scalar_type();
  p->device = w1->device();
  p->last_bias = ptr_of(a[3]);
  p->act = PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  return PyCapsule_New(p.release(), kPlan, plan_free);
  END_HANDLE_TH_ERRORS
}

// buffers of one call: ops.Workspace of (tokens, experts, device), from a cache of the module's
struct Buffers {
  void *mask, *idx, *off, *ws, *status;
  size_t ws_bytes;
};

PyObject* s_get;      // "raw"

// keep: a list that holds on to it, or null
bool buffers_of(PyObject* cache, const Plan& p, int64_t N, Buffers* b, PyObject* keep = nullptr) {
  // the cache is a dictionary (tokens, experts, device index) -> Workspace with a miss handler, which
  // allocates on the current stream
  PyObject* key = Py_BuildValue("(LLi)", (long long)N, (long long)p.E, (int)p.device.index());
  if (!key) return false;
  PyObject* w = PyDict_GetItemWithError(cache, key);       // borrowed
  PyObject* made = nullptr;
  if (!w && !PyErr_Occurred()) w = made = PyObject_GetItem(cache, key);   // __missing__ allocates
  Py_DECREF(key);
  if (!w) return false;
  PyObject* raw = keep && PyList_Append(keep, w) != 0
                      ? nullptr
                      : PyObject_GetAttr(w, s_get);         // bytes: five addresses and a size
  Py_XDECREF(made);                                         // the cache keeps it
  if (!raw) return false;
  const bool ok = PyBytes_Check(raw) && PyBytes_GET_SIZE(raw) == 48;
  if (ok) {
    uint64_t v[6];
    memcpy(v, PyBytes_AS_STRING(raw), 48);
    *b = {(void*)v[0], (void*)v[1], (void*)v[2], (void*)v[3], (void*)v[4], (size_t)v[5]};
  } else {
    PyErr_SetString(PyExc_TypeError, "workspace addresses");
  }
  Py_DECREF(raw);
  return ok;
}

// run_layer(plan, modules, parameters, attributes, workspaces, x, rule, k, tau, residual, scores, norm,
//           capture)
//   -> (out, routing[, norms]) | status code (int) | None: the plan is stale | False: it is as the module
//   is, but this call takes the general path
// rule: D2D_RULE_*; k / tau as that rule reads them (MAX: threshold 1 - tau).
// scores: None or [.., E] of x's dtype.  norm: None or (kind, gamma, beta|None, eps, gamma_offset):
// x + layer(norm(x)).  capture: None or (norm layer, ord), with D2D_RULE_ALL.
PyObject* run_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 13) {
    PyErr_SetString(PyExc_TypeError, "run_layer takes 13 arguments");
    return nullptr;
  }
  Plan* p = static_cast<Plan*>(PyCapsule_GetPointer(a[0], kPlan));
  if (!p) return nullptr;
  if (!still_valid(*p, a + 1)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const at::Tensor* xp = tensor_of(a[5]);
  if (!xp || !xp->is_cuda() || xp->scalar_type() != p->dtype || xp->device() != p->device ||
      xp->dim() < 1 || xp->size(-1) != p->d || xp->numel() == 0)
    Py_RETURN_FALSE;
  const at::Tensor x = xp->contiguous();
  const int64_t N = x.numel() / p->d;
  const int rule = (int)PyLong_AsLong(a[6]);
  const int k = (int)PyLong_AsLong(a[7]);
  const bool reads_tau = rule == D2D_RULE_MAX || rule == D2D_RULE_DYNK;
  const double tau = reads_tau ? PyFloat_AsDouble(a[8]) : 0.0;
  const int residual = PyObject_IsTrue(a[9]);
  if (PyErr_Occurred()) return nullptr;
  const float mult = (float)(1.0 - tau);
  const bool ranked = rule == D2D_RULE_TOPK || rule == D2D_RULE_DYNK;
  at::Tensor scores, scratch;
  const bool given = a[10] != Py_None;
  if (given) {
    const at::Tensor* sp = tensor_of(a[10]);
    if (!sp || !sp->is_cuda() || sp->scalar_type() != p->dtype || sp->device() != p->device ||
        sp->numel() != N * p->E)
      Py_RETURN_FALSE;
    scores = sp->contiguous();
  } else if (!p->wa && rule != D2D_RULE_ALL) {
    Py_RETURN_FALSE;
  }
  c10::cuda::CUDAGuard guard(p->device);
  const auto cur = c10::cuda::getCurrentCUDAStream(p->device.index());
  const auto stream = (d2d_stream_t)cur.stream();
  Buffers b;
  if (!buffers_of(a[4], *p, N, &b)) return nullptr;
  use_on(*p, cur);
  const int dt = p->dtype == at::kBFloat16 ? D2D_BF16 : D2D_F32;
  const auto opts = x.options();
  at::Tensor out = at::detail::empty_cuda(x.sizes(), opts);
  c10::SmallVector<int64_t, 5> rs(x.sizes().begin(), x.sizes().end());
  rs.back() = p->E;
  at::Tensor rt = at::detail::empty_cuda(rs, opts);
  if (ranked && !given) scratch = at::detail::empty_cuda({N, p->E}, opts);
  const void* xin = x.data_ptr();
  const void* lb = p->last_bias;
  int res = residual ? 1 : 0, rc = D2D_OK;
  at::Tensor xn, norms;
  int norm_layer = 0, norm_ord = 0;
  if (a[12] != Py_None) {
    norm_layer = (int)PyLong_AsLong(PyTuple_GetItem(a[12], 0));
    norm_ord = (int)PyLong_AsLong(PyTuple_GetItem(a[12], 1));
    if (PyErr_Occurred()) return nullptr;
    norms = at::detail::empty_cuda({p->E, N}, opts);
  }
  if (a[11] != Py_None) {
    PyObject* nm = a[11];
    xn = at::detail::empty_cuda(x.sizes(), opts);
    const long kind = PyLong_AsLong(PyTuple_GetItem(nm, 0));
    const double eps = PyFloat_AsDouble(PyTuple_GetItem(nm, 3));
    const double goff = PyFloat_AsDouble(PyTuple_GetItem(nm, 4));
    if (PyErr_Occurred()) return nullptr;
    const at::Tensor* gt = tensor_of(PyTuple_GetItem(nm, 1));
    const at::Tensor* bt = tensor_of(PyTuple_GetItem(nm, 2));
    const auto fits = [&](const at::Tensor* t) {
      return t->numel() == p->d && t->scalar_type() == p->dtype && t->device() == p->device;
    };
    TORCH_CHECK(gt && fits(gt) && (!bt || fits(bt)), "norm parameters: ", p->d,
                " values of x's dtype, on its device");
    const at::Tensor g = gt->contiguous(), bb = bt ? bt->contiguous() : at::Tensor();
    rc = d2d_prenorm_init(xin, g.data_ptr(), bt ? bb.data_ptr() : nullptr, (float)eps, (int)kind,
                          (float)goff, lb, xn.data_ptr(), out.data_ptr(), N, (int)p->d, dt, stream);
    xin = xn.data_ptr();
    lb = nullptr;
    res = D2D_OUT_PREINITIALISED;
  }
  if (rc == D2D_OK)
    rc = d2d_moe_forward_rule(
        xin, given ? nullptr : p->wa, given ? nullptr : p->wb, given ? nullptr : p->rp,
        given ? scores.data_ptr() : nullptr, scratch.defined() ? scratch.data_ptr() : nullptr, rule,
        k, (float)tau, mult, p->w1, p->b1, p->wup, p->w2, p->ep, lb, res, out.data_ptr(),
        (uint32_t*)b.mask, (int32_t*)b.idx, (int32_t*)b.off, N, (int)p->d, (int)p->R, (int)p->E,
        (int)p->H, (int)p->act, dt, b.ws, b.ws_bytes, (int*)b.status, rt.data_ptr(),
        norms.defined() ? norms.data_ptr() : nullptr, norm_layer, norm_ord, stream);
  if (rc != D2D_OK) return PyLong_FromLong(rc);
  const bool has_norms = norms.defined();
  PyObject* res_t = PyTuple_New(has_norms ? 3 : 2);
  if (!res_t) return nullptr;
  PyTuple_SET_ITEM(res_t, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(res_t, 1, THPVariable_Wrap(std::move(rt)));
  if (has_norms) PyTuple_SET_ITEM(res_t, 2, THPVariable_Wrap(std::move(norms)));
  return res_t;
  END_HANDLE_TH_ERRORS
}

// ---- host-buffer pipeline -------------------------------------------------------
// Two staging buffers for slices of x, three for slices of the output; the events say when the
// stream that last used one is done with it (never recorded: at once).
constexpr int kIn = 2, kOut = 3;
struct HostPipe {
  int device = 0;
  cudaEvent_t in_full[kIn] = {}, in_free[kIn] = {}, out_full[kOut] = {}, out_free[kOut] = {},
              caller = nullptr;
  unsigned long long n = 0;            // slices so far, over all calls
  std::vector<cudaEvent_t*> all() {
    std::vector<cudaEvent_t*> v = {&caller};
    for (auto& e : in_full) v.push_back(&e);
    for (auto& e : in_free) v.push_back(&e);
    for (auto& e : out_full) v.push_back(&e);
    for (auto& e : out_free) v.push_back(&e);
    return v;
  }
};
constexpr const char* kPipe = "d2dmoe_b200.host_pipe";
void pipe_free(PyObject* cap) {
  auto* h = static_cast<HostPipe*>(PyCapsule_GetPointer(cap, kPipe));
  for (cudaEvent_t* e : h->all())
    if (*e) cudaEventDestroy(*e);
  delete h;
}

PyObject* make_pipe(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 1, "make_pipe(device index)");
  auto h = std::make_unique<HostPipe>();
  h->device = (int)PyLong_AsLong(a[0]);
  if (PyErr_Occurred()) return nullptr;
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)h->device);
  for (cudaEvent_t* e : h->all())
    C10_CUDA_CHECK(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  return PyCapsule_New(h.release(), kPipe, pipe_free);
  END_HANDLE_TH_ERRORS
}

// run_host(plan, modules, parameters, attributes, workspaces, pipe, x_host, out_host,
//          staging (kIn + kOut tensors), (stream in, stream run, stream out), slices, rule, k, tau,
//          residual, sync)
//   -> True | status code (int) | None / False as run_layer
// Slice i's copy in, the kernels of slice i - 1 and the copy out of slice i - 2 overlap.  (Issued from
// Python it takes 70 us of host time per slice, more than a slice's copies.)
PyObject* run_host(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 16, "run_host takes 16 arguments");
  Plan* p = static_cast<Plan*>(PyCapsule_GetPointer(a[0], kPlan));
  HostPipe* h = static_cast<HostPipe*>(PyCapsule_GetPointer(a[5], kPipe));
  if (!p || !h) return nullptr;
  if (!still_valid(*p, a + 1)) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const at::Tensor *xh = tensor_of(a[6]), *oh = tensor_of(a[7]);
  if (!xh || !oh || xh->scalar_type() != p->dtype || oh->scalar_type() != p->dtype ||
      !xh->is_contiguous() || !oh->is_contiguous() || !oh->is_cpu() || xh->sizes() != oh->sizes() ||
      xh->dim() < 2 || xh->size(-1) != p->d || xh->numel() == 0 || h->device != p->device.index())
    Py_RETURN_FALSE;
  void* stage[kIn + kOut];
  for (int i = 0; i < kIn + kOut; ++i) stage[i] = const_cast<void*>(ptr_of(PyTuple_GetItem(a[8], i)));
  cudaStream_t st[3];
  for (int i = 0; i < 3; ++i) st[i] = (cudaStream_t)PyLong_AsVoidPtr(PyTuple_GetItem(a[9], i));
  const int64_t slices = PyLong_AsLongLong(a[10]);
  const int rule = (int)PyLong_AsLong(a[11]), k = (int)PyLong_AsLong(a[12]);
  const bool reads_tau = rule == D2D_RULE_MAX || rule == D2D_RULE_DYNK;
  const double tau = reads_tau ? PyFloat_AsDouble(a[13]) : 0.0;
  const int residual = PyObject_IsTrue(a[14]), sync = PyObject_IsTrue(a[15]);
  if (PyErr_Occurred()) return nullptr;
  if ((rule != D2D_RULE_ALL && !p->wa) || (rule != D2D_RULE_ALL && rule != D2D_RULE_MAX))
    Py_RETURN_FALSE;
  c10::cuda::CUDAGuard guard(p->device);
  const cudaStream_t cur = c10::cuda::getCurrentCUDAStream(p->device.index()).stream();
  if (sync) {                          // what the caller's stream has queued comes first
    C10_CUDA_CHECK(cudaEventRecord(h->caller, cur));
    for (cudaStream_t s : st) C10_CUDA_CHECK(cudaStreamWaitEvent(s, h->caller, 0));
  }
  const int dt = p->dtype == at::kBFloat16 ? D2D_BF16 : D2D_F32;
  const int64_t B = xh->size(0), per = xh->numel() / B;      // values of one batch entry
  // `workspaces` is the pipeline's own: allocated and used on the stream of the kernels alone, whatever
  // the caller's stream is doing, so that one that leaves the cache is reused in stream order
  const auto run = c10::cuda::getStreamFromExternal(st[1], p->device.index());
  std::vector<Buffers> bufs((size_t)slices);
  THPObjectPtr keep(PyList_New(0));
  if (!keep) return nullptr;
  {
    c10::cuda::CUDAStreamGuard on_run(run);
    for (int64_t i = 0; i < slices; ++i)
      if (!buffers_of(a[4], *p, (B * (i + 1) / slices - B * i / slices) * per / p->d, &bufs[i],
                      keep))
        return nullptr;
  }
  use_on(*p, run);
  // pinned blocks that their owner drops are not handed out again before these copies are done (memory
  // of another origin is none of the allocator's)
  const std::pair<const at::Tensor*, cudaStream_t> used[2] = {{xh, st[0]}, {oh, st[2]}};
  for (const auto& u : used)
    at::getHostAllocator(at::kCUDA)->record_event(
        u.first->data_ptr(), u.first->storage().data_ptr().get_context(),
        c10::cuda::getStreamFromExternal(u.second, p->device.index()).unwrap());
  const size_t es = xh->element_size();
  const char* src = static_cast<const char*>(xh->data_ptr());
  char* dst = static_cast<char*>(oh->data_ptr());
  int rc = D2D_OK;
  for (int64_t i = 0; i < slices && rc == D2D_OK; ++i, ++h->n) {
    const int64_t lo = B * i / slices, hi = B * (i + 1) / slices, N = (hi - lo) * per / p->d;
    const int b = (int)(h->n % kIn), o = (int)(h->n % kOut);
    const size_t bytes = (size_t)((hi - lo) * per) * es, at = (size_t)(lo * per) * es;
    const Buffers& buf = bufs[i];
    C10_CUDA_CHECK(cudaStreamWaitEvent(st[0], h->in_free[b], 0));
    C10_CUDA_CHECK(cudaMemcpyAsync(stage[b], src + at, bytes, cudaMemcpyHostToDevice, st[0]));
    C10_CUDA_CHECK(cudaEventRecord(h->in_full[b], st[0]));
    C10_CUDA_CHECK(cudaStreamWaitEvent(st[1], h->in_full[b], 0));
    C10_CUDA_CHECK(cudaStreamWaitEvent(st[1], h->out_free[o], 0));
    rc = d2d_moe_forward_rule(stage[b], p->wa, p->wb, p->rp, nullptr, nullptr, rule, k, (float)tau,
                              (float)(1.0 - tau), p->w1, p->b1, p->wup, p->w2, p->ep, p->last_bias,
                              residual ? 1 : 0, stage[kIn + o], (uint32_t*)buf.mask,
                              (int32_t*)buf.idx, (int32_t*)buf.off, N, (int)p->d, (int)p->R,
                              (int)p->E, (int)p->H, (int)p->act, dt, buf.ws, buf.ws_bytes,
                              (int*)buf.status, nullptr, nullptr, 0, 0, (d2d_stream_t)st[1]);
    C10_CUDA_CHECK(cudaEventRecord(h->in_free[b], st[1]));
    C10_CUDA_CHECK(cudaEventRecord(h->out_full[o], st[1]));
    C10_CUDA_CHECK(cudaStreamWaitEvent(st[2], h->out_full[o], 0));
    C10_CUDA_CHECK(cudaMemcpyAsync(dst + at, stage[kIn + o], bytes, cudaMemcpyDeviceToHost, st[2]));
    C10_CUDA_CHECK(cudaEventRecord(h->out_free[o], st[2]));
  }
  if (sync) {                          // the last copy out is behind everything else
    cudaError_t err;
    Py_BEGIN_ALLOW_THREADS
    err = cudaStreamSynchronize(st[2]);
    Py_END_ALLOW_THREADS
    C10_CUDA_CHECK(err);
  }
  if (rc != D2D_OK) return PyLong_FromLong(rc);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"mark", (PyCFunction)(void (*)(void))mark, METH_FASTCALL, nullptr},
    {"wait_mark", (PyCFunction)(void (*)(void))wait_mark, METH_FASTCALL, nullptr},
    {"make_pipe", (PyCFunction)(void (*)(void))make_pipe, METH_FASTCALL, nullptr},
    {"run_host", (PyCFunction)(void (*)(void))run_host, METH_FASTCALL, nullptr},
    {"make_plan", (PyCFunction)(void (*)(void))make_plan, METH_FASTCALL, nullptr},
    {"run_layer", (PyCFunction)(void (*)(void))run_layer, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_d2d_torch", nullptr, -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__d2d_torch(void) {
  s_get = PyUnicode_InternFromString("raw");
  return PyModule_Create(&kModule);
}
