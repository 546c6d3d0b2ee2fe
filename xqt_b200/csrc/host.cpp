// Native call path of the bound layers: a `Bound` object holds everything one layer call needs -- the checks of its
// input, the shape of its output, its scratch, and the library calls to make with their resolved arguments -- and a
// call goes from the Python argument to the kernel launches without running Python code.  A layer that takes any number of
// rows is one object too: row counts enter the resolved arguments as factors, so a prompt length that was never seen costs
// what a repeated one does.
//
// What bounds it: a decode projection's kernel runs 4 us, and the same call made by a Python closure (attribute checks,
// torch.empty, a 19-argument ctypes call) cost 12-17 us of host time, so every small call ran at the host's pace.
//
// The object checks what it must in order to pass a raw pointer on (dtype, device, shape, contiguity, current device).
// Whatever it does not take on itself -- keyword arguments, a failed check, an output or residual that does not fit --
// goes to the Python callable it was built with, which raises the layer's own error or serves the call.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <structmember.h>

#include <cstring>
#include <memory>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/xqt_b200.h"

namespace {

// An integer argument that may depend on the number of rows.
struct Number {
  int value, per_row;
  int at(int m) const { return value + per_row * m; }
};

// Where a pointer argument comes from; `value` is an address or a byte offset, to which `per_row` bytes are added per row.
enum Source : int { kConst = 0, kInput = 1, kOutput = 2, kResidual = 3, kScratch = 4, kWorkspace = 5 };
struct Pointer {
  int source;
  intptr_t value, per_row;
};

// The library entry of a step.  Its arguments are its pointers, then its integers, in the order of the C prototype;
// workspace address and size (where the entry takes them) and the stream come last.
enum Op : int { kDecodeLanes, kW4A16Run, kSwiglu, kRotateQuantize, kW8A8Gemm, kLowrankDown, kW4A4Gemm, kActPrologue, kW8A8LowrankGemm, kSwigluMlp, kOpCount };
constexpr int kPointerCount[kOpCount] = {8, 7, 2, 5, 7, 4, 8, 6, 8, 8};
constexpr int kIntCount[kOpCount] = {9, 11, 3, 7, 4, 3, 5, 8, 4, 10};
constexpr int kMaxPointers = 8;
struct Step {
  int op;
  void* fn;
  std::vector<Pointer> ptrs;
  std::vector<Number> ints;
  Pointer ws;
  size_t ws_bytes;                       // or, for the rows m of a call:
  size_t (*ws_need)(int m, int, int);
  int ws_args[2];
};

// The calls of one range of row counts.  A layer that takes any number of rows has several; the first one whose range and
// guards (library functions that say whether an entry serves a size) hold is taken.
constexpr int kMaxInts = 11, kMaxSteps = 4;
struct Guard {
  void* fn;
  Number rows;
  std::vector<int> args;
  bool holds(int m) const {
    if (args.size() == 3) return reinterpret_cast<int (*)(int, int, int, int)>(fn)(rows.at(m), args[0], args[1], args[2]) != 0;
    return reinterpret_cast<int (*)(int, int, int, int, int)>(fn)(rows.at(m), args[0], args[1], args[2], args[3]) != 0;
  }
};
struct Plan {
  int lo, hi;
  std::vector<Guard> guards;
  std::vector<Step> steps;
  int64_t scratch_bytes, scratch_per_row;
};
// What a row count resolves to; the last one is kept, so a repeated count asks the library nothing.
struct Resolved {
  int m;
  const Plan* plan;
  size_t ws_bytes[kMaxSteps], ws_most;
};

// The workspaces of native.py's pool, mirrored here so that a call finds the current one without running Python code: per
// device, stream and tag the buffer in use (guarded by the GIL).  A call holds a reference while it launches; a bound layer
// keeps none, so a buffer that the pool has replaced is released, and status words are read where the kernels write them.
struct SpaceKey {
  int device;
  uintptr_t stream;
  int tag;
  bool operator==(const SpaceKey& o) const { return device == o.device && stream == o.stream && tag == o.tag; }
};
struct SpaceHash {
  size_t operator()(const SpaceKey& k) const { return std::hash<uintptr_t>()(k.stream * 31 + (uintptr_t)k.tag * 7 + (uintptr_t)k.device); }
};
struct Space {
  PyObject* tensor;
  char* data;
  size_t bytes;
  bool captured;         // a graph capture has recorded its address
};
std::unordered_map<SpaceKey, Space, SpaceHash>& spaces() {
  static auto* map = new std::unordered_map<SpaceKey, Space, SpaceHash>();
  return *map;
}
int tag_id(const char* tag) {
  static auto* tags = new std::vector<std::string>();
  for (size_t i = 0; i < tags->size(); ++i)
    if ((*tags)[i] == tag) return (int)i;
  tags->push_back(tag);
  return (int)tags->size() - 1;
}

struct Bound {
  PyObject_HEAD
  vectorcallfunc vectorcall;
  PyObject* slow;        // the Python callable with the same signature
  PyObject* on_error;    // called with (code, step) when a library call fails: raises
  PyObject* workspace;   // None, or called with a size: the pool's workspace for the current stream, at least that large
  PyObject* keep;
  at::ScalarType dtype, out_dtype;
  int device;
  int64_t rows, k, n;    // rows < 0: any number that one of the plans takes
  bool any_rank;         // the input may have any leading dimensions that multiply to `rows`
  bool takes_residual;   // a third positional argument, [rows, n] in the input dtype
  int tag;               // the workspace's
  std::vector<Plan>* plans;
  Resolved last;
  PyObject *dict, *weakrefs;      // like the closures it stands for, it takes attributes and weak references
};

const Resolved* resolve(Bound* b, int m) {
  Resolved& r = b->last;
  if (r.m == m) return &r;
  for (const Plan& plan : *b->plans) {
    if (m < plan.lo || m > plan.hi) continue;
    bool holds = true;
    for (const Guard& g : plan.guards) holds = holds && g.holds(m);
    if (!holds) continue;
    r.plan = &plan;
    r.ws_most = 0;
    for (size_t i = 0; i < plan.steps.size(); ++i) {
      const Step& s = plan.steps[i];
      r.ws_bytes[i] = s.ws_need != nullptr ? s.ws_need(m, s.ws_args[0], s.ws_args[1]) : s.ws_bytes;
      if (s.ws.source == kWorkspace && r.ws_bytes[i] > r.ws_most) r.ws_most = r.ws_bytes[i];
    }
    r.m = m;
    return &r;
  }
  return nullptr;
}

int run_step(const Step& s, void* const* p, const int* i, void* ws, size_t ws_bytes, cudaStream_t stream) {
  xqt_b200_stream_t st = (xqt_b200_stream_t)stream;
  switch (s.op) {
    case kDecodeLanes:
      return reinterpret_cast<decltype(&xqt_b200_w4a16_decode_lanes)>(s.fn)(
          p[0], p[1], p[2], p[3], (const float*)p[4], p[5], p[6], i[0], i[1], i[2], i[3], i[4], i[5], i[6], i[7], i[8],
          (unsigned int*)p[7], st);
    case kW4A16Run:
      return reinterpret_cast<decltype(&xqt_b200_w4a16_run)>(s.fn)(
          p[0], p[1], p[2], p[3], (const float*)p[4], p[5], p[6], i[0], i[1], i[2], i[3], i[4], i[5], i[6], i[7], i[8], i[9], ws,
          ws_bytes, i[10], st);
    case kSwiglu:
      return reinterpret_cast<decltype(&xqt_b200_swiglu)>(s.fn)(p[0], p[1], i[0], i[1], i[2], st);
    case kRotateQuantize:
      return reinterpret_cast<decltype(&xqt_b200_rotate_quantize)>(s.fn)(p[0], (const float*)p[1], p[2], (float*)p[3], p[4], i[0],
                                                                         i[1], i[2], i[3], i[4], i[5], i[6], st);
    case kW8A8Gemm:
      return reinterpret_cast<decltype(&xqt_b200_w8a8_gemm_addend)>(s.fn)(p[0], p[1], (const float*)p[2], (const float*)p[3],
                                                                          (const float*)p[4], (const float*)p[5], p[6], i[0], i[1],
                                                                          i[2], i[3], ws, ws_bytes, st);
    case kLowrankDown:
      return reinterpret_cast<decltype(&xqt_b200_lowrank_down)>(s.fn)(p[0], p[1], (float*)p[2], p[3], i[0], i[1], i[2], st);
    case kW4A4Gemm:
      return reinterpret_cast<decltype(&xqt_b200_w4a4_gemm)>(s.fn)(p[0], (const float*)p[1], p[2], p[3], p[4], (const float*)p[5],
                                                                   (const float*)p[6], p[7], i[0], i[1], i[2], i[3], i[4], ws,
                                                                   ws_bytes, st);
    case kW8A8LowrankGemm:
      return reinterpret_cast<decltype(&xqt_b200_w8a8_gemm_lowrank)>(s.fn)(p[0], p[1], (const float*)p[2], (const float*)p[3],
                                                                           (const float*)p[4], p[5], p[6], p[7], i[0], i[1], i[2], i[3],
                                                                           ws, ws_bytes, st);
    case kSwigluMlp:
      return reinterpret_cast<decltype(&xqt_b200_w4a16_swiglu_mlp)>(s.fn)(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], i[0], i[1], i[2], i[3],
                                                                          i[4], i[5], i[6], i[7], i[8], i[9], ws, ws_bytes, st);
    case kActPrologue: {
      float scale;                     // the first integer is the bit pattern of lora_scale
      memcpy(&scale, &i[0], sizeof(scale));
      return reinterpret_cast<decltype(&xqt_b200_act_prologue)>(s.fn)(p[0], (const float*)p[1], p[2], (float*)p[3], p[4], p[5], scale,
                                                                      i[1], i[2], i[3], i[4], i[5], i[6], i[7], st);
    }
  }
  return (int)cudaErrorInvalidValue;
}

char* stream_space(Bound* b, cudaStream_t stream, size_t bytes, THPObjectPtr& held) {
  const SpaceKey key{b->device, (uintptr_t)stream, b->tag};
  auto it = spaces().find(key);
  if (it == spaces().end() || it->second.bytes < bytes) {
    held = PyObject_CallFunction(b->workspace, "n", (Py_ssize_t)bytes);
    if (!held) return nullptr;
    it = spaces().find(key);
    if (it == spaces().end() || it->second.bytes < bytes) {
      PyErr_SetString(PyExc_RuntimeError, "Bound: the workspace pool has no buffer of the size asked for");
      return nullptr;
    }
  }
  Space& space = it->second;
  if (!space.captured && c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) space.captured = true;
  char* data = space.data;
  Py_INCREF(space.tensor);
  held = space.tensor;
  return data;
}

bool plain(const at::Tensor& t, at::ScalarType dtype, int device) {
  return t.scalar_type() == dtype && t.is_cuda() && t.device().index() == device && t.layout() == at::kStrided && t.is_contiguous();
}

struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// Any of the queries below may throw (a fake or functorch tensor has no data, symbolic sizes are no integers, an allocation
// fails): `bound_call` turns that into the Python exception torch would raise.
PyObject* call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Bound* b = reinterpret_cast<Bound*>(self);
  const Py_ssize_t nargs = PyVectorcall_NARGS(nargsf);
  auto slow = [&]() {
    Py_INCREF(b->slow);                          // it may be replaced while it runs
    THPObjectPtr held(b->slow);
    return PyObject_Vectorcall(held.get(), args, nargsf, kwnames);
  };
  if (kwnames != nullptr || nargs < 1 || nargs > 3 || !THPVariable_Check(args[0])) return slow();
  const at::Tensor& x = THPVariable_Unpack(args[0]);
  if (!plain(x, b->dtype, b->device) || c10::cuda::current_device() != b->device) return slow();
  const auto shape = x.sizes();
  const int64_t dim = (int64_t)shape.size();
  if (dim < 1 || shape[dim - 1] != b->k || b->k < 1 || (!b->any_rank && dim != 2)) return slow();
  const int64_t rows = x.numel() / b->k;
  if (b->rows >= 0 ? rows != b->rows : rows < 1 || rows > INT32_MAX) return slow();
  if ((reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) != 0) return slow();      // the entries' loads are 16 bytes wide
  const Resolved* found = resolve(b, (int)rows);
  if (found == nullptr) return slow();
  const Resolved how = *found;                   // another thread may resolve another count while this one launches
  const int m = how.m;

  const bool has_out = nargs >= 2 && args[1] != Py_None;
  if (has_out) {
    if (!THPVariable_Check(args[1])) return slow();
    const at::Tensor& o = THPVariable_Unpack(args[1]);
    if (b->any_rank || !plain(o, b->out_dtype, b->device) || o.dim() != 2 || o.size(0) != rows || o.size(1) != b->n) return slow();
  }
  void* residual = nullptr;
  if (nargs == 3 && args[2] != Py_None) {
    if (!b->takes_residual || !THPVariable_Check(args[2])) return slow();
    const at::Tensor& r = THPVariable_Unpack(args[2]);
    if (!plain(r, b->dtype, b->device) || r.dim() != 2 || r.size(0) != rows || r.size(1) != b->n) return slow();
    residual = r.data_ptr();
  }
  const c10::Device device(c10::kCUDA, (c10::DeviceIndex)b->device);
  at::Tensor out, scratch;
  if (has_out) {
    out = THPVariable_Unpack(args[1]);
  } else if (dim == 2) {
    out = at::detail::empty_cuda({rows, b->n}, b->out_dtype, device, c10::nullopt);
  } else {
    std::vector<int64_t> oshape(shape.begin(), shape.end());
    oshape.back() = b->n;
    out = at::detail::empty_cuda(oshape, b->out_dtype, device, c10::nullopt);
  }
  const int64_t scratch_bytes = how.plan->scratch_bytes + how.plan->scratch_per_row * rows;
  if (scratch_bytes > 0) scratch = at::detail::empty_cuda({scratch_bytes}, at::kByte, device, c10::nullopt);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)b->device).stream();
  char* base[6] = {nullptr, static_cast<char*>(x.data_ptr()), static_cast<char*>(out.data_ptr()), static_cast<char*>(residual),
                   scratch.defined() ? static_cast<char*>(scratch.data_ptr()) : nullptr, nullptr};
  THPObjectPtr held;
  if (how.ws_most > 0) {
    base[kWorkspace] = stream_space(b, stream, how.ws_most, held);
    if (base[kWorkspace] == nullptr) return nullptr;
  }
  int code = 0;
  size_t at_step = 0;
  {
    const WithoutGil released;
    const std::vector<Step>& steps = how.plan->steps;
    for (; at_step < steps.size(); ++at_step) {
      const Step& s = steps[at_step];
      void* p[kMaxPointers];
      int ints[kMaxInts];
      for (size_t i = 0; i < s.ptrs.size(); ++i) {
        char* from = base[s.ptrs[i].source];
        p[i] = s.ptrs[i].source == kResidual && from == nullptr ? nullptr : from + (s.ptrs[i].value + s.ptrs[i].per_row * m);
      }
      for (size_t i = 0; i < s.ints.size(); ++i) ints[i] = s.ints[i].at(m);
      code = run_step(s, p, ints, base[s.ws.source] + s.ws.value, how.ws_bytes[at_step], stream);
      if (code != 0) break;
    }
  }
  if (code != 0) {
    THPObjectPtr r(PyObject_CallFunction(b->on_error, "in", code, (Py_ssize_t)at_step));
    if (r) PyErr_SetString(PyExc_RuntimeError, "Bound: library call failed");
    return nullptr;
  }
  if (has_out) {
    Py_INCREF(args[1]);
    return args[1];
  }
  return THPVariable_Wrap(std::move(out));
}

PyObject* bound_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  try {
    return call(self, args, nargsf, kwnames);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

bool parse_pointer(PyObject* o, Pointer* p) {
  long long value = 0, per_row = 0;
  int source = 0;
  if (PyTuple_Check(o)) {
    if (!PyArg_ParseTuple(o, "iL|L", &source, &value, &per_row)) return false;
  } else {
    value = PyLong_AsLongLong(o);
    if (value == -1 && PyErr_Occurred()) return false;
  }
  if (source < kConst || source > kWorkspace) {
    PyErr_SetString(PyExc_ValueError, "Bound: unknown pointer source");
    return false;
  }
  *p = Pointer{source, (intptr_t)value, (intptr_t)per_row};
  return true;
}

bool parse_number(PyObject* o, Number* n) {
  n->per_row = 0;
  if (PyTuple_Check(o)) return PyArg_ParseTuple(o, "ii", &n->value, &n->per_row) != 0;
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) return false;
  n->value = (int)v;
  return true;
}

bool parse_step(PyObject* o, Step* s) {
  PyObject *ptrs, *ints, *ws, *ws_bytes;
  unsigned long long fn;
  if (!PyArg_ParseTuple(o, "iKO!O!OO", &s->op, &fn, &PyTuple_Type, &ptrs, &PyTuple_Type, &ints, &ws, &ws_bytes)) return false;
  if (s->op < 0 || s->op >= kOpCount || fn == 0 || PyTuple_GET_SIZE(ptrs) != kPointerCount[s->op] || PyTuple_GET_SIZE(ints) != kIntCount[s->op]) {
    PyErr_SetString(PyExc_ValueError, "Bound: a step does not have the arguments of its library entry");
    return false;
  }
  s->fn = reinterpret_cast<void*>(fn);
  s->ws_bytes = 0;
  s->ws_need = nullptr;
  if (PyTuple_Check(ws_bytes)) {
    unsigned long long need;
    if (!PyArg_ParseTuple(ws_bytes, "Kii", &need, &s->ws_args[0], &s->ws_args[1])) return false;
    s->ws_need = reinterpret_cast<size_t (*)(int, int, int)>(need);
  } else {
    s->ws_bytes = PyLong_AsSize_t(ws_bytes);
    if (PyErr_Occurred()) return false;
  }
  s->ptrs.resize((size_t)PyTuple_GET_SIZE(ptrs));
  for (size_t i = 0; i < s->ptrs.size(); ++i)
    if (!parse_pointer(PyTuple_GET_ITEM(ptrs, (Py_ssize_t)i), &s->ptrs[i])) return false;
  s->ints.resize((size_t)PyTuple_GET_SIZE(ints));
  for (size_t i = 0; i < s->ints.size(); ++i)
    if (!parse_number(PyTuple_GET_ITEM(ints, (Py_ssize_t)i), &s->ints[i])) return false;
  return parse_pointer(ws, &s->ws);
}

// (function, rows, (3 or 4 integers))
bool parse_guard(PyObject* o, Guard* g) {
  unsigned long long fn;
  PyObject *rows, *args;
  if (!PyArg_ParseTuple(o, "KOO!", &fn, &rows, &PyTuple_Type, &args) || !parse_number(rows, &g->rows)) return false;
  if (fn == 0 || PyTuple_GET_SIZE(args) < 3 || PyTuple_GET_SIZE(args) > 4) {
    PyErr_SetString(PyExc_ValueError, "Bound: a guard takes a function of the row count and three or four integers");
    return false;
  }
  g->fn = reinterpret_cast<void*>(fn);
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args); ++i) {
    Number n;
    if (!parse_number(PyTuple_GET_ITEM(args, i), &n)) return false;
    g->args.push_back(n.value);
  }
  return true;
}

// (first row count, last row count, guards, steps, scratch bytes, scratch bytes per row)
bool parse_plan(PyObject* o, Plan* p) {
  PyObject *guards, *steps;
  long long bytes, per_row;
  if (!PyArg_ParseTuple(o, "iiO!O!LL", &p->lo, &p->hi, &PyTuple_Type, &guards, &PyTuple_Type, &steps, &bytes, &per_row)) return false;
  if (PyTuple_GET_SIZE(steps) > kMaxSteps) {
    PyErr_SetString(PyExc_ValueError, "Bound: too many steps");
    return false;
  }
  p->scratch_bytes = bytes;
  p->scratch_per_row = per_row;
  p->guards.resize((size_t)PyTuple_GET_SIZE(guards));
  for (size_t i = 0; i < p->guards.size(); ++i)
    if (!parse_guard(PyTuple_GET_ITEM(guards, (Py_ssize_t)i), &p->guards[i])) return false;
  p->steps.resize((size_t)PyTuple_GET_SIZE(steps));
  for (size_t i = 0; i < p->steps.size(); ++i)
    if (!parse_step(PyTuple_GET_ITEM(steps, (Py_ssize_t)i), &p->steps[i])) return false;
  return true;
}

int bound_traverse(PyObject* self, visitproc visit, void* arg) {
  Bound* b = reinterpret_cast<Bound*>(self);
  Py_VISIT(b->slow);
  Py_VISIT(b->on_error);
  Py_VISIT(b->workspace);
  Py_VISIT(b->keep);
  Py_VISIT(b->dict);
  return 0;
}
int bound_clear(PyObject* self) {
  Bound* b = reinterpret_cast<Bound*>(self);
  Py_CLEAR(b->slow);
  Py_CLEAR(b->on_error);
  Py_CLEAR(b->workspace);
  Py_CLEAR(b->keep);
  Py_CLEAR(b->dict);
  return 0;
}
void bound_dealloc(PyObject* self) {
  Bound* b = reinterpret_cast<Bound*>(self);
  PyObject_GC_UnTrack(self);
  if (b->weakrefs != nullptr) PyObject_ClearWeakRefs(self);
  bound_clear(self);
  delete b->plans;
  Py_TYPE(self)->tp_free(self);
}

PyObject* make(PyTypeObject* type, PyObject* args, PyObject* kwargs) {
  static const char* names[] = {"plans", "slow", "on_error", "dtype", "out_dtype", "device", "rows", "k", "n", "any_rank",
                                "takes_residual", "workspace", "tag", "keep", nullptr};
  PyObject *plans, *slow, *on_error, *dtype, *out_dtype, *workspace = Py_None, *keep = Py_None;
  const char* tag = "run";
  int device, any_rank = 0, takes_residual = 0;
  long long rows, k, n;
  if (!PyArg_ParseTupleAndKeywords(args, kwargs, "O!OOOOiLLL|ppOsO", const_cast<char**>(names), &PyTuple_Type, &plans, &slow, &on_error,
                                   &dtype, &out_dtype, &device, &rows, &k, &n, &any_rank, &takes_residual, &workspace,
                                   &tag, &keep))
    return nullptr;
  if (!THPDtype_Check(dtype) || !THPDtype_Check(out_dtype)) {
    PyErr_SetString(PyExc_TypeError, "Bound: dtype and out_dtype must be torch dtypes");
    return nullptr;
  }
  auto parsed = std::make_unique<std::vector<Plan>>((size_t)PyTuple_GET_SIZE(plans));
  for (size_t i = 0; i < parsed->size(); ++i) {
    Plan& plan = (*parsed)[i];
    if (!parse_plan(PyTuple_GET_ITEM(plans, (Py_ssize_t)i), &plan)) return nullptr;
    for (const Step& s : plan.steps)
      if (s.ws.source == kWorkspace && workspace == Py_None) {
        PyErr_SetString(PyExc_ValueError, "Bound: a step needs a workspace");
        return nullptr;
      }
  }
  Bound* b = reinterpret_cast<Bound*>(type->tp_alloc(type, 0));
  if (b == nullptr) return nullptr;
  b->vectorcall = bound_call;
  b->plans = parsed.release();
  b->last = Resolved{};
  b->last.m = -1;
  b->tag = tag_id(tag);
  Py_INCREF(slow); b->slow = slow;
  Py_INCREF(on_error); b->on_error = on_error;
  Py_INCREF(workspace); b->workspace = workspace;
  Py_INCREF(keep); b->keep = keep;
  b->dtype = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
  b->out_dtype = reinterpret_cast<THPDtype*>(out_dtype)->scalar_type;
  b->device = device;
  b->rows = rows; b->k = k; b->n = n;
  b->any_rank = any_rank != 0;
  b->takes_residual = takes_residual != 0;
  return reinterpret_cast<PyObject*>(b);
}

PyObject* bound_new(PyTypeObject* type, PyObject* args, PyObject* kwargs) {
  try {
    return make(type, args, kwargs);
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
}

PyMemberDef bound_members[] = {{"keep", T_OBJECT, offsetof(Bound, keep), READONLY, "the objects whose memory the calls use"},
                               {nullptr, 0, 0, 0, nullptr}};

PyObject* get_slow(PyObject* self, void*) {
  PyObject* slow = reinterpret_cast<Bound*>(self)->slow;
  if (slow == nullptr) slow = Py_None;
  Py_INCREF(slow);
  return slow;
}
int set_slow(PyObject* self, PyObject* value, void*) {
  if (value == nullptr || !PyCallable_Check(value)) {
    PyErr_SetString(PyExc_TypeError, "Bound.slow must be callable");
    return -1;
  }
  Py_INCREF(value);
  PyObject* before = reinterpret_cast<Bound*>(self)->slow;
  reinterpret_cast<Bound*>(self)->slow = value;
  Py_XDECREF(before);
  return 0;
}
PyGetSetDef bound_getset[] = {{"slow", get_slow, set_slow, "the callable that gets what the native path does not take", nullptr},
                              {"__dict__", PyObject_GenericGetDict, PyObject_GenericSetDict, nullptr, nullptr},
                              {nullptr, nullptr, nullptr, nullptr, nullptr}};

// As for a closure, a copy is the object itself (the addresses it holds are those of tensors that `keep` shares).
PyObject* copy_self(PyObject* self, PyObject*) {
  Py_INCREF(self);
  return self;
}
PyMethodDef bound_methods[] = {{"__copy__", copy_self, METH_NOARGS, nullptr}, {"__deepcopy__", copy_self, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyTypeObject bound_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// set_workspace(device, stream, tag, tensor): the pool's buffer from now on; the one before it is released
PyObject* set_workspace(PyObject*, PyObject* args) {
  int device;
  unsigned long long stream;
  const char* tag;
  PyObject* tensor;
  if (!PyArg_ParseTuple(args, "iKsO", &device, &stream, &tag, &tensor)) return nullptr;
  if (!THPVariable_Check(tensor)) {
    PyErr_SetString(PyExc_TypeError, "set_workspace: a tensor is needed");
    return nullptr;
  }
  try {
    const at::Tensor& t = THPVariable_Unpack(tensor);
    Space fresh{tensor, static_cast<char*>(t.data_ptr()), (size_t)t.nbytes(), false};
    Space& space = spaces()[SpaceKey{device, (uintptr_t)stream, tag_id(tag)}];
    THPObjectPtr before(space.tensor);       // value-initialised when new
    Py_INCREF(tensor);
    space = fresh;
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
  Py_RETURN_NONE;
}

// workspace_captured(device, stream, tag[, mark]): whether a graph capture has recorded the buffer's address; `mark` says so
PyObject* workspace_captured(PyObject*, PyObject* args) {
  int device, mark = 0;
  unsigned long long stream;
  const char* tag;
  if (!PyArg_ParseTuple(args, "iKs|p", &device, &stream, &tag, &mark)) return nullptr;
  bool captured = false;
  try {
    auto it = spaces().find(SpaceKey{device, (uintptr_t)stream, tag_id(tag)});
    if (it != spaces().end()) {
      it->second.captured |= mark != 0;
      captured = it->second.captured;
    }
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());
    return nullptr;
  }
  return PyBool_FromLong(captured);
}

PyMethodDef host_methods[] = {{"set_workspace", set_workspace, METH_VARARGS, "Mirror a buffer of the workspace pool."},
                              {"workspace_captured", workspace_captured, METH_VARARGS, "Whether a graph capture uses a buffer of the pool."},
                              {nullptr, nullptr, 0, nullptr}};
PyModuleDef host_module = {PyModuleDef_HEAD_INIT, "_host", "Native call path of the bound layers.", -1, host_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  bound_type.tp_name = "xqt_b200._host.Bound";
  bound_type.tp_basicsize = sizeof(Bound);
  bound_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
  bound_type.tp_new = bound_new;
  bound_type.tp_dealloc = bound_dealloc;
  bound_type.tp_traverse = bound_traverse;
  bound_type.tp_clear = bound_clear;
  bound_type.tp_call = PyVectorcall_Call;
  bound_type.tp_vectorcall_offset = offsetof(Bound, vectorcall);
  bound_type.tp_members = bound_members;
  bound_type.tp_getset = bound_getset;
  bound_type.tp_methods = bound_methods;
  bound_type.tp_dictoffset = offsetof(Bound, dict);
  bound_type.tp_weaklistoffset = offsetof(Bound, weakrefs);
  if (PyType_Ready(&bound_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&host_module);
  if (m == nullptr) return nullptr;
  Py_INCREF(&bound_type);
  if (PyModule_AddObject(m, "Bound", reinterpret_cast<PyObject*>(&bound_type)) < 0) {
    Py_DECREF(&bound_type);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
