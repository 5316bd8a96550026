// The host side of a pass in native code: the operator constructors' accepted cases and the
// eval driver's loop over a graph of operators, as a CPython extension (_host).
//
// Why: a pass of seven operators spent 59 us in Python and 29 in the C calls that launch
// (415 rows of a speech encoder layer, 27 us of kernels), a decoder's token 110 us in Python.
//
// Python stays the definition of both.  Everything here either does exactly what the Python
// code beside it does (ops.py, executor.py), on the same Value / PendingOp / DeviceBuffer
// objects, or leaves the whole call to it: a constructor that meets anything but the plain
// accepted case (other types, options it does not know, an argument to refuse) returns None
// before it has made anything, and evaluate() returns False before its first side effect.
// A single operator it cannot place goes to the executor's own dispatch().
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <initializer_list>
#include <new>
#include <unordered_map>
#include <vector>

#include "rt_attn.h"

namespace {

// ---- what bind() is given: classes, constants, the library's entry points ---------------

PyTypeObject *gValue, *gMeta, *gPending, *gBuffer, *gExecutor;
Py_ssize_t gShapeAt, gBufferAt, gPendingAt, gReleasedAt;   // slots of a Value
Py_ssize_t gPtrAt, gOwnedAt;                               // slots of a DeviceBuffer
PyObject *gRecycled;          // the reason evalValues marks a recycled value with
PyObject *gLib, *gCheck, *gNoArgs;
PyObject *gActCode;           // name -> code
long long gWindowInf, gMaxHeadDim, gMaxDecodeHeadDim;

constexpr int kMethods = 5;
const char* const kMethodNames[kMethods] = {"dispatch", "acquireOutput", "releaseOutput", "submit", "_alloc"};
PyObject *gMethodName[kMethods], *gMethod[kMethods];   // the executor's own, to tell an override

#define RT_STRINGS(X)                                                                              \
  X(attn) X(matmul) X(rope) X(softmax) X(writeRows) X(sliceRows) X(sliceCols) X(argmaxDot)         \
  X(f16) X(f32) X(qHeads) X(kvHeads) X(headDim) X(windowLeft) X(windowRight)     \
  X(qPosOffset) X(sinks) X(segments) X(maxSegment) X(keyBias) X(srcStart) X(width) X(baseRow)      \
  X(bias) X(addend) X(activation) X(scales) X(bits) X(groupSize) X(value)                          \
  X(dispatches) X(_pool) X(_live) X(_ctx) X(_lib) X(_disposed) X(ctx)
#define X(n) PyObject* s_##n;
RT_STRINGS(X)
#undef X
PyObject *s_decodeAppend, *s_decodeRopeAppend;

struct Entry {
  decltype(&rt_matmul) matmul;
  decltype(&rt_rope) rope;
  decltype(&rt_slice) slice;
  decltype(&rt_attn) attn;
  decltype(&rt_attn_route) route;
  decltype(&rt_attn_decode) decode;
  decltype(&rt_argmax_dot) argmaxDot;
  decltype(&rt_kv_append) kvAppend;
  decltype(&rt_softmax) softmax;
  decltype(&rt_windows) windows;
} gEntry;

// ---- small pieces ------------------------------------------------------------------------

struct Ref {   // an owned reference
  PyObject* p;
  explicit Ref(PyObject* o = nullptr) : p(o) {}
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  PyObject* take() {
    PyObject* o = p;
    p = nullptr;
    return o;
  }
  explicit operator bool() const { return p != nullptr; }
};

PyObject*& slot(PyObject* o, Py_ssize_t at) { return *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o) + at); }
void set_slot(PyObject* o, Py_ssize_t at, PyObject* v) {
  PyObject*& s = slot(o, at);
  PyObject* old = s;
  Py_INCREF(v);
  s = v;
  Py_XDECREF(old);
}

bool is_str(PyObject* o, PyObject* interned) {
  if (o == interned) return true;
  return o && PyUnicode_CheckExact(o) && PyUnicode_Compare(o, interned) == 0;
}

// A plain int that fits; other types (bool, float, numpy's) are left to Python.
bool as_int(PyObject* o, long long& v) {
  if (!o || !PyLong_CheckExact(o)) return false;
  int overflow = 0;
  v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

constexpr long long kMost = 1ll << 31;   // sizes above are left to Python

// dtype code of a name, -1 for others
int dtype_code(PyObject* o) {
  if (is_str(o, s_f16)) return RT_F16;
  if (is_str(o, s_f32)) return RT_F32;
  return -1;
}

struct Meta {
  long long elems, rows, cols;
  int dtype;
  bool matrix;   // two dims
};
bool read_meta(PyObject* value, Meta& m) {
  if (Py_TYPE(value) != gValue) return false;
  PyObject* s = slot(value, gShapeAt);
  if (!s || Py_TYPE(s) != gMeta || PyTuple_GET_SIZE(s) != 3) return false;
  m.dtype = dtype_code(PyTuple_GET_ITEM(s, 1));
  if (m.dtype < 0 || !as_int(PyTuple_GET_ITEM(s, 0), m.elems) || m.elems < 0) return false;
  PyObject* d = PyTuple_GET_ITEM(s, 2);
  m.matrix = PyTuple_CheckExact(d) && PyTuple_GET_SIZE(d) == 2 && as_int(PyTuple_GET_ITEM(d, 0), m.rows) &&
             as_int(PyTuple_GET_ITEM(d, 1), m.cols) && m.rows > 0 && m.cols > 0 && m.rows < kMost && m.cols < kMost;
  return true;
}
bool read_matrix(PyObject* value, Meta& m) { return read_meta(value, m) && m.matrix; }

PyObject* dtype_name(int code) { return code == RT_F16 ? s_f16 : s_f32; }

// Device pointer of a buffer; false leaves the operator to Python.
bool buffer_ptr(PyObject* b, char*& p) {
  if (!b || Py_TYPE(b) != gBuffer) return false;
  PyObject* o = slot(b, gPtrAt);
  if (!o || !PyLong_CheckExact(o)) return false;
  p = static_cast<char*>(PyLong_AsVoidPtr(o));
  if (!p && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}

// ---- making a pending node ---------------------------------------------------------------

PyObject* tuple_of(PyTypeObject* type, std::initializer_list<PyObject*> items) {   // steals the items
  bool ok = true;
  for (PyObject* i : items) ok = ok && i;
  PyObject* t = ok ? type->tp_alloc(type, (Py_ssize_t)items.size()) : nullptr;
  Py_ssize_t n = 0;
  for (PyObject* i : items) {
    if (t) PyTuple_SET_ITEM(t, n++, i);
    else Py_XDECREF(i);
  }
  return t;
}
PyObject* ints(std::initializer_list<long long> v) {
  Ref t(PyTuple_New((Py_ssize_t)v.size()));
  Py_ssize_t n = 0;
  for (long long x : v) {
    PyObject* o = t ? PyLong_FromLongLong(x) : nullptr;
    if (!o) return nullptr;
    PyTuple_SET_ITEM(t.p, n++, o);
  }
  return t.take();
}
PyObject* refs(std::initializer_list<PyObject*> v) {   // those that are there
  Py_ssize_t n = 0;
  for (PyObject* x : v) n += x != nullptr;
  PyObject* t = PyTuple_New(n);
  if (!t) return nullptr;
  n = 0;
  for (PyObject* x : v)
    if (x) PyTuple_SET_ITEM(t, n++, Py_NewRef(x));
  return t;
}

// Value(ValueMeta(rows * cols, dtype, (rows, cols)), None, PendingOp(op, inputs, None, attrs));
// steals inputs and attrs.
PyObject* node(long long rows, long long cols, int dtype, PyObject* op, PyObject* inputs, PyObject* attrs) {
  Ref meta(tuple_of(gMeta, {PyLong_FromLongLong(rows * cols), Py_NewRef(dtype_name(dtype)), ints({rows, cols})}));
  Ref pend(tuple_of(gPending, {Py_NewRef(op), inputs, Py_NewRef(Py_None), attrs}));
  if (!meta || !pend) return nullptr;
  PyObject* v = gValue->tp_new(gValue, gNoArgs, nullptr);   // (its __init__ sets these four)
  if (!v) return nullptr;
  set_slot(v, gShapeAt, meta.p);
  set_slot(v, gBufferAt, Py_None);
  set_slot(v, gPendingAt, pend.p);
  set_slot(v, gReleasedAt, Py_None);
  return v;
}

#define DEFER Py_RETURN_NONE   // left to the Python constructor

// An option: borrowed, nullptr where it is missing or None.
PyObject* option(PyObject* opts, PyObject* key) {
  PyObject* v = PyDict_GetItemWithError(opts, key);   // (string keys: no error to meet)
  return v == Py_None ? nullptr : v;
}
bool int_option(PyObject* opts, PyObject* key, long long fallback, long long& v) {
  PyObject* o = option(opts, key);
  if (!o) {
    v = fallback;
    return true;
  }
  return as_int(o, v);
}
// A window: a non-negative int or infinity.
bool window_option(PyObject* opts, PyObject* key, long long& v) {
  PyObject* o = option(opts, key);
  if (!o) return false;
  if (PyFloat_CheckExact(o)) {
    v = gWindowInf;
    return PyFloat_AS_DOUBLE(o) == HUGE_VAL;
  }
  if (!as_int(o, v) || v < 0) return false;
  if (v > gWindowInf) v = gWindowInf;
  return true;
}

// ---- constructors: the accepted cases of ops.py -----------------------------------------

PyObject* op_matmul(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) DEFER;
  PyObject *a = args[0], *b = args[1], *opts = args[2];
  PyObject *bias = nullptr, *addend = nullptr;
  long long act = 0, base = 0;
  bool hasBase = false;
  Meta ma, mb, m;
  if (!read_matrix(a, ma) || !read_matrix(b, mb) || ma.dtype != mb.dtype) DEFER;
  if (opts != Py_None) {
    if (!PyDict_CheckExact(opts)) DEFER;
    if (option(opts, s_scales) || option(opts, s_bits) || option(opts, s_groupSize)) DEFER;
    hasBase = option(opts, s_baseRow) != nullptr;
    if (!int_option(opts, s_baseRow, 0, base) || base < 0) DEFER;
    bias = option(opts, s_bias);
    addend = option(opts, s_addend);
    if (PyObject* name = option(opts, s_activation)) {
      PyObject* code = PyUnicode_CheckExact(name) ? PyDict_GetItemWithError(gActCode, name) : nullptr;
      if (!code || !as_int(code, act)) DEFER;
    }
  }
  if (base > mb.rows || ma.cols > mb.rows - base || (!hasBase && ma.cols != mb.rows)) DEFER;
  if (bias && (!read_meta(bias, m) || m.dtype != ma.dtype || m.elems != mb.cols)) DEFER;
  if (addend && (!read_meta(addend, m) || m.dtype != ma.dtype || m.elems != ma.rows * mb.cols)) DEFER;
  return node(ma.rows, mb.cols, ma.dtype, s_matmul, refs({a, b, bias, addend}),
              ints({bias != nullptr, addend != nullptr, act, base, hasBase}));
}

PyObject* op_rope(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4 || !PyDict_CheckExact(args[3])) DEFER;
  PyObject* opts = args[3];
  Meta x, t;
  long long hd, start, w;
  if (!read_matrix(args[0], x) || !as_int(PyDict_GetItemWithError(opts, s_headDim), hd)) DEFER;
  if (!int_option(opts, s_srcStart, 0, start) || !int_option(opts, s_width, x.cols, w)) DEFER;
  if (hd <= 0 || hd % 2 || start < 0 || start % 2 || w <= 0 || start > x.cols || w > x.cols - start || w % hd) DEFER;
  for (int i = 1; i < 3; i++)
    if (!read_meta(args[i], t) || t.dtype != RT_F32 || t.elems != x.rows * hd) DEFER;
  return node(x.rows, w, x.dtype, s_rope, refs({args[0], args[1], args[2]}), ints({hd, start, w}));
}

PyObject* op_slice(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) DEFER;
  Meta x;
  long long dim, start, end;
  if (!read_matrix(args[0], x) || !as_int(args[1], dim) || !as_int(args[2], start) || !as_int(args[3], end)) DEFER;
  if (dim < 0) dim += 2;
  if (dim < 0 || dim > 1 || start < 0 || start >= end || end > (dim == 0 ? x.rows : x.cols)) DEFER;
  const long long len = end - start;
  return node(dim == 0 ? len : x.rows, dim == 0 ? x.cols : len, x.dtype, dim == 0 ? s_sliceRows : s_sliceCols,
              refs({args[0]}), ints({start, end}));
}

// The options sdpa and sdpaPacked share; segments need more than one row.
struct AttnOpts {
  long long qHeads, kvHeads, hd, wl, wr, pos, maxSegment;
  PyObject *sinks, *segments;
};
bool attn_options(PyObject* opts, long long rows, AttnOpts& o) {
  if (!PyDict_CheckExact(opts) || !as_int(PyDict_GetItemWithError(opts, s_qHeads), o.qHeads) ||
      !as_int(PyDict_GetItemWithError(opts, s_kvHeads), o.kvHeads) ||
      !as_int(PyDict_GetItemWithError(opts, s_headDim), o.hd))
    return false;
  if (o.qHeads <= 0 || o.kvHeads <= 0 || o.hd <= 0 || o.qHeads >= kMost || o.hd >= kMost || o.qHeads % o.kvHeads)
    return false;
  if (!window_option(opts, s_windowLeft, o.wl) || !window_option(opts, s_windowRight, o.wr)) return false;
  if (!int_option(opts, s_qPosOffset, 0, o.pos) || o.pos < 0 || o.pos >= kMost) return false;
  Meta m;
  o.sinks = option(opts, s_sinks);
  if (o.sinks && (!read_meta(o.sinks, m) || m.dtype != RT_F32 || m.elems != o.qHeads)) return false;
  o.segments = option(opts, s_segments);
  if (o.segments && (!read_meta(o.segments, m) || m.dtype != RT_F32 || m.elems != 2 * rows || rows == 1))
    return false;
  if (!int_option(opts, s_maxSegment, 0, o.maxSegment) || o.maxSegment < 0 || (o.maxSegment && !o.segments))
    return false;
  return true;
}

PyObject* op_sdpa(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) DEFER;
  Meta q, k, v;
  AttnOpts o;
  if (!read_matrix(args[0], q) || !read_matrix(args[1], k) || !read_matrix(args[2], v)) DEFER;
  if (!attn_options(args[3], q.rows, o) || option(args[3], s_keyBias)) DEFER;
  const long long kvw = o.kvHeads * o.hd;
  if (q.cols != o.qHeads * o.hd || k.cols != kvw || v.cols != kvw || v.rows != k.rows) DEFER;
  if (k.dtype != q.dtype || v.dtype != q.dtype || o.hd > (q.rows == 1 ? gMaxDecodeHeadDim : gMaxHeadDim)) DEFER;
  if (o.wr != gWindowInf && o.pos + q.rows > k.rows) DEFER;
  return node(q.rows, q.cols, q.dtype, s_attn, refs({args[0], args[1], args[2], o.sinks, o.segments}),
              ints({o.qHeads, o.kvHeads, o.hd, o.wl, o.wr, o.pos, o.sinks != nullptr, o.segments != nullptr,
                    o.maxSegment, 0}));
}

PyObject* op_sdpa_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) DEFER;
  Meta x;
  AttnOpts o;
  if (!read_matrix(args[0], x) || x.rows == 1 || !attn_options(args[1], x.rows, o)) DEFER;
  if (x.cols != (o.qHeads + 2 * o.kvHeads) * o.hd || o.hd > 128 || (o.wr != gWindowInf && o.pos > 0)) DEFER;
  return node(x.rows, o.qHeads * o.hd, x.dtype, s_attn, refs({args[0], o.sinks, o.segments}),
              ints({o.qHeads, o.kvHeads, o.hd, o.wl, o.wr, o.pos, o.sinks != nullptr, o.segments != nullptr,
                    o.maxSegment, 1}));
}

PyObject* op_write_rows(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) DEFER;
  Meta d, s;
  long long start;
  if (!read_matrix(args[0], d) || !read_matrix(args[1], s) || !as_int(args[2], start)) DEFER;
  if (slot(args[0], gReleasedAt) != Py_None || slot(args[0], gBufferAt) == Py_None) DEFER;
  if (s.dtype != d.dtype || s.cols != d.cols || start < 0 || start > d.rows || s.rows > d.rows - start) DEFER;
  return node(start + s.rows, d.cols, d.dtype, s_writeRows, refs({args[0], args[1]}), ints({start}));
}

PyObject* op_argmax_dot(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 2) DEFER;
  Meta w, x;
  if (!read_matrix(args[0], w) || !read_matrix(args[1], x) || x.rows != 1 || x.cols != w.cols || x.dtype != w.dtype)
    DEFER;
  return node(1, 1, RT_F32, s_argmaxDot, refs({args[0], args[1]}), Py_NewRef(Py_None));
}

// ---- the eval driver ---------------------------------------------------------------------

enum Op { kOther, kMatmul, kAttn, kWriteRows, kRope, kSliceRows, kSliceCols, kSoftmax, kArgmaxDot };

struct Fused {   // what executor.py's _fusable_appends plans for an attn node
  int k = -1, v = -1, ropeQ = -1, ropeK = -1, vSlice = -1;
  bool on = false;
};

struct Node {
  PyObject *v, *inputs, *attrs;   // v owned; the others belong to it
  Op op;
  int uses = 0, left = 0;
  bool target = false, skipped = false, elided = false, aliased = false;
  Fused fused;
};

struct Evaluation {
  std::vector<Node> order;
  std::unordered_map<PyObject*, int> at;
  ~Evaluation() {
    for (Node& n : order) Py_DECREF(n.v);
  }
  int find(PyObject* v) const {
    auto i = at.find(v);
    return i == at.end() ? -1 : i->second;
  }
};

Op op_of(PyObject* name) {
  if (is_str(name, s_matmul)) return kMatmul;
  if (is_str(name, s_attn)) return kAttn;
  if (is_str(name, s_rope)) return kRope;
  if (is_str(name, s_sliceCols)) return kSliceCols;
  if (is_str(name, s_writeRows)) return kWriteRows;
  if (is_str(name, s_argmaxDot)) return kArgmaxDot;
  if (is_str(name, s_softmax)) return kSoftmax;
  if (is_str(name, s_sliceRows)) return kSliceRows;
  return kOther;
}

// Pending values in dependency order.  False: leave the evaluation to Python (a released value,
// whose error Python words; a type of another make; a graph as deep as Python's stack).
bool collect(Evaluation& e, PyObject* v, int depth) {
  if (Py_TYPE(v) != gValue || depth > 400) return false;
  PyObject *released = slot(v, gReleasedAt), *buffer = slot(v, gBufferAt), *pend = slot(v, gPendingAt);
  if (released != Py_None || !buffer) return false;
  if (buffer != Py_None || e.at.count(v)) return true;
  if (!pend || Py_TYPE(pend) != gPending || PyTuple_GET_SIZE(pend) != 4) return false;
  PyObject *inputs = PyTuple_GET_ITEM(pend, 1), *attrs = PyTuple_GET_ITEM(pend, 3);
  if (!PyTuple_CheckExact(inputs)) return false;
  e.at.emplace(v, -1);   // (seen; its place is known once its inputs have theirs)
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(inputs); i++) {
    PyObject* in = PyTuple_GET_ITEM(inputs, i);
    if (Py_TYPE(in) != gValue) return false;
    if (slot(in, gBufferAt) == Py_None || slot(in, gReleasedAt) != Py_None)
      if (!collect(e, in, depth + 1)) return false;
  }
  e.at[v] = (int)e.order.size();
  Node n;
  n.v = Py_NewRef(v);
  n.inputs = inputs;
  n.attrs = attrs;
  n.op = op_of(PyTuple_GET_ITEM(pend, 0));
  e.order.push_back(n);
  return true;
}

bool attr(const Node& n, int i, long long& v) {
  return n.attrs && PyTuple_CheckExact(n.attrs) && i < PyTuple_GET_SIZE(n.attrs) && as_int(PyTuple_GET_ITEM(n.attrs, i), v);
}
PyObject* input(const Node& n, int i) { return PyTuple_GET_ITEM(n.inputs, i); }
Py_ssize_t inputs_of(const Node& n) { return PyTuple_GET_SIZE(n.inputs); }

// executor.py's _fusable_appends.  False: an attribute that Python should look at.
bool plan_appends(Evaluation& e) {
  bool any = false;
  for (const Node& n : e.order) any |= n.op == kWriteRows;
  if (!any) return true;
  for (const Node& n : e.order)
    for (Py_ssize_t i = 0; i < inputs_of(n); i++) {
      const int at = e.find(input(n, (int)i));
      if (at >= 0) e.order[at].uses++;
    }
  auto priv = [&](PyObject* v, Op op) {   // pending, of that op, read once and by no caller
    const int at = e.find(v);
    return at >= 0 && e.order[at].op == op && e.order[at].uses == 1 && !e.order[at].target ? at : -1;
  };
  for (Node& n : e.order) {
    if (n.op != kAttn) continue;
    long long packed, wr, pos, hd, x;
    if (!attr(n, 9, packed) || !attr(n, 4, wr) || !attr(n, 5, pos) || !attr(n, 2, hd)) return false;
    Meta q, m;
    if (packed || inputs_of(n) < 3 || wr != 0) continue;
    if (!read_matrix(input(n, 0), q)) return false;
    if (q.rows != 1) continue;
    PyObject *kv[2] = {input(n, 1), input(n, 2)}, *fresh[2] = {nullptr, nullptr};
    int write[2];
    bool ok = kv[0] != kv[1];
    for (int i = 0; i < 2 && ok; i++) {
      write[i] = priv(kv[i], kWriteRows);
      if (write[i] < 0) {
        ok = false;
        break;
      }
      const Node& w = e.order[write[i]];
      if (inputs_of(w) != 2 || !attr(w, 0, x) || !read_matrix(input(w, 1), m)) return false;
      ok = m.rows == 1 && x == pos;
      if (!read_matrix(kv[i], m)) return false;
      ok = ok && m.rows == pos + 1;
      fresh[i] = input(w, 1);
    }
    if (!ok) continue;
    Fused f;
    f.on = true;
    f.k = write[0];
    f.v = write[1];
    const int rq = priv(input(n, 0), kRope), rk = priv(fresh[0], kRope);
    if (rq >= 0 && rk >= 0) {
      const Node &a = e.order[rq], &b = e.order[rk];
      long long ha, hb;
      Meta ra, rb;
      if (inputs_of(a) != 3 || inputs_of(b) != 3 || !attr(a, 0, ha) || !attr(b, 0, hb) ||
          !read_matrix(input(a, 0), ra) || !read_matrix(input(b, 0), rb))
        return false;
      if (input(a, 1) == input(b, 1) && input(a, 2) == input(b, 2) && ha == hd && hb == hd && ra.rows == 1 &&
          rb.rows == 1)
        f.ropeQ = rq, f.ropeK = rk;
    }
    const int vs = priv(fresh[1], kSliceCols);
    if (vs >= 0) {
      if (!read_matrix(input(e.order[vs], 0), m)) return false;
      if (m.rows == 1) f.vSlice = vs;
    }
    n.fused = f;
  }
  for (const Node& n : e.order) {
    if (!n.fused.on) continue;
    e.order[n.fused.k].skipped = e.order[n.fused.v].skipped = true;
    for (int i : {n.fused.ropeQ, n.fused.ropeK, n.fused.vSlice})
      if (i >= 0) e.order[i].elided = true;
  }
  return true;
}

// The executor while its loop runs: references of its own, since other threads run during calls.
struct Exec {
  PyObject* self;
  Ref pool, live, names, ctxObject;
  rt_ctx* ctx = nullptr;
};

bool exec_attr(PyObject* ex, PyObject* name, Ref& out) {
  out.p = PyObject_GetAttr(ex, name);
  return out.p != nullptr;
}

PyObject* acquire(Exec& x, PyObject* meta) {
  Ref key(PyTuple_Pack(2, PyTuple_GET_ITEM(meta, 1), PyTuple_GET_ITEM(meta, 0)));
  if (!key) return nullptr;
  PyObject* bucket = PyDict_GetItemWithError(x.pool.p, key.p);
  if (!bucket && PyErr_Occurred()) return nullptr;
  if (!bucket || !PyList_CheckExact(bucket) || PyList_GET_SIZE(bucket) == 0)
    return PyObject_CallMethodOneArg(x.self, gMethodName[1], meta);
  const Py_ssize_t last = PyList_GET_SIZE(bucket) - 1;
  PyObject* b = Py_NewRef(PyList_GET_ITEM(bucket, last));
  if (PyList_SetSlice(bucket, last, last + 1, nullptr) < 0 || PySet_Add(x.live.p, b) < 0) {
    Py_DECREF(b);
    return nullptr;
  }
  return b;
}

bool give_back(Exec& x, PyObject* buffer, PyObject* meta) {
  if (Py_TYPE(buffer) != gBuffer) {
    Ref r(PyObject_CallMethodObjArgs(x.self, gMethodName[2], buffer, meta, nullptr));
    return bool(r);
  }
  if (slot(buffer, gOwnedAt) != Py_True) return true;
  Ref key(PyTuple_Pack(2, PyTuple_GET_ITEM(meta, 1), PyTuple_GET_ITEM(meta, 0)));
  if (!key || PySet_Discard(x.live.p, buffer) < 0) return false;
  PyObject* bucket = PyDict_GetItemWithError(x.pool.p, key.p);
  if (bucket) return PyList_Append(bucket, buffer) == 0;
  if (PyErr_Occurred()) return false;
  Ref fresh(PyList_New(1));
  if (!fresh) return false;
  PyList_SET_ITEM(fresh.p, 0, Py_NewRef(buffer));
  return PyDict_SetItem(x.pool.p, key.p, fresh.p) == 0;
}

// One reader less of each of a node's inputs; those that nobody reads any more go back.
bool release(Evaluation& e, Exec& x, PyObject* inputs) {
  const Py_ssize_t n = PyTuple_GET_SIZE(inputs);
  for (Py_ssize_t i = 0; i < n; i++) {
    PyObject* in = PyTuple_GET_ITEM(inputs, i);
    bool again = false;
    for (Py_ssize_t k = 0; k < i; k++) again |= PyTuple_GET_ITEM(inputs, k) == in;
    const int at = again ? -1 : e.find(in);
    if (at < 0) continue;
    Node& m = e.order[at];
    if (--m.left == 0 && !m.aliased && !m.elided) {
      PyObject *buffer = slot(in, gBufferAt), *meta = slot(in, gShapeAt);
      if (!buffer || buffer == Py_None || !meta) continue;
      if (!give_back(x, buffer, meta)) return false;
      set_slot(in, gReleasedAt, gRecycled);
    }
  }
  return true;
}

// Raises what check() makes of a status that is not RT_OK.
bool report(Exec& x, int status) {
  if (status == 0) return true;
  Ref code(PyLong_FromLong(status));
  Ref r(code ? PyObject_CallFunctionObjArgs(gCheck, code.p, x.ctxObject.p, nullptr) : nullptr);
  if (r) PyErr_SetString(PyExc_SystemError, "a failed call was not reported");
  return false;
}

// -1: an exception is set; 0: left to the executor's dispatch(); 1: done.
int dispatch(Evaluation& e, Exec& x, const Node& n, PyObject* out) {
  char *o = nullptr, *in[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  Meta m, self;
  const Py_ssize_t count = inputs_of(n);
  if (count > 5 || !read_matrix(n.v, self) || (out && !buffer_ptr(out, o))) return 0;
  for (Py_ssize_t i = 0; i < count; i++) {
    PyObject* v = input(n, (int)i);
    const int at = e.find(v);
    if (at >= 0 && e.order[at].elided) continue;   // computed inside the fused kernel
    if (Py_TYPE(v) != gValue || slot(v, gReleasedAt) != Py_None || !buffer_ptr(slot(v, gBufferAt), in[i])) return 0;
  }
  // (a context that another thread has disposed of meanwhile: Python's property says so)
  Ref disposed(PyObject_GetAttr(x.self, s__disposed));
  if (!disposed) return -1;
  if (disposed.p != Py_False) return 0;

  int status = 0;
  PyObject* name = nullptr;
  const char* route = nullptr;
  long long a[10];
  switch (n.op) {
    case kMatmul: {
      Meta b;
      if (count < 2 || !read_matrix(input(n, 0), m) || !read_matrix(input(n, 1), b)) return 0;
      for (int i = 0; i < 4; i++)
        if (!attr(n, i, a[i])) return 0;
      if (count != 2 + (a[0] != 0) + (a[1] != 0)) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.matmul(x.ctx, in[0], in[1], a[0] ? in[2] : nullptr, a[1] ? in[2 + (a[0] != 0)] : nullptr, o,
                             m.rows, m.cols, b.cols, b.rows, a[3], (int32_t)a[2], self.dtype);
      Py_END_ALLOW_THREADS;
      name = s_matmul;
      break;
    }
    case kRope:
      if (count != 3 || !read_matrix(input(n, 0), m)) return 0;
      for (int i = 0; i < 3; i++)
        if (!attr(n, i, a[i])) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.rope(x.ctx, in[0], reinterpret_cast<float*>(in[1]), reinterpret_cast<float*>(in[2]), o, m.rows,
                           m.cols, (int32_t)a[0], a[1], a[2], m.dtype);
      Py_END_ALLOW_THREADS;
      name = s_rope;
      break;
    case kSliceRows:
    case kSliceCols:
      if (count != 1 || !read_matrix(input(n, 0), m) || !attr(n, 0, a[0]) || !attr(n, 1, a[1])) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = n.op == kSliceRows
                   ? gEntry.slice(x.ctx, in[0], o, m.rows, m.cols, a[0], a[1], 0, m.cols, m.dtype)
                   : gEntry.slice(x.ctx, in[0], o, m.rows, m.cols, 0, m.rows, a[0], a[1], m.dtype);
      Py_END_ALLOW_THREADS;
      name = n.op == kSliceRows ? s_sliceRows : s_sliceCols;
      break;
    case kArgmaxDot:
      if (count != 2 || !read_matrix(input(n, 0), m)) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.argmaxDot(x.ctx, in[0], in[1], reinterpret_cast<float*>(o), m.rows, m.cols, m.dtype);
      Py_END_ALLOW_THREADS;
      name = s_argmaxDot;
      break;
    case kSoftmax:
      for (int i = 0; i < 3; i++)
        if (!attr(n, i, a[i])) return 0;
      if (count != 1 + (a[0] != 0)) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.softmax(x.ctx, in[0], o, a[0] ? reinterpret_cast<float*>(in[1]) : nullptr, self.rows, self.cols,
                              (int32_t)a[1], (int32_t)a[2], self.dtype);
      Py_END_ALLOW_THREADS;
      name = s_softmax;
      break;
    case kWriteRows: {
      Meta s;
      if (count != 2 || !read_matrix(input(n, 0), m) || !read_matrix(input(n, 1), s) || !attr(n, 0, a[0])) return 0;
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.kvAppend(x.ctx, in[0], in[1], a[0], s.rows, s.cols, m.rows, m.dtype);
      Py_END_ALLOW_THREADS;
      name = s_writeRows;
      break;
    }
    case kAttn: {
      if (!n.attrs || !PyTuple_CheckExact(n.attrs) || PyTuple_GET_SIZE(n.attrs) != 10) return 0;   // key bias: Python's
      for (int i = 0; i < 10; i++)
        if (!attr(n, i, a[i])) return 0;
      const int base = a[9] ? 1 : 3;
      if (count != base + (a[6] != 0) + (a[7] != 0)) return 0;
      Meta k;
      if (!read_matrix(input(n, 0), m) || !read_matrix(input(n, a[9] ? 0 : 1), k)) return 0;
      const float* sinks = a[6] ? reinterpret_cast<float*>(in[base]) : nullptr;
      const float* segs = a[7] ? reinterpret_cast<float*>(in[base + (a[6] != 0)]) : nullptr;
      if (n.fused.on) {
        // every window of a row is read where the row lies
        auto window = [&](int at, int attrAt, char*& p) {
          const Node& w = e.order[at];
          PyObject* v = input(w, 0);
          Meta row;
          long long col;
          if (!read_matrix(v, row) || !attr(w, attrAt, col) || slot(v, gReleasedAt) != Py_None ||
              !buffer_ptr(slot(v, gBufferAt), p))
            return false;
          p += col * (row.dtype == RT_F16 ? 2 : 4);
          return true;
        };
        auto plain = [&](PyObject* v, char*& p) {
          return slot(v, gReleasedAt) == Py_None && buffer_ptr(slot(v, gBufferAt), p);
        };
        const Fused& f = n.fused;
        const Node &wk = e.order[f.k], &wv = e.order[f.v];
        char *kc, *vc, *kn, *vn, *q = in[0], *cs = nullptr, *sn = nullptr;
        Meta cache;
        if (!plain(input(wk, 0), kc) || !plain(input(wv, 0), vc) || !read_matrix(input(wk, 0), cache)) return 0;
        if (f.ropeQ >= 0) {
          const Node& r = e.order[f.ropeQ];
          if (!window(f.ropeQ, 1, q) || !window(f.ropeK, 1, kn) || !plain(input(r, 1), cs) || !plain(input(r, 2), sn))
            return 0;
        } else if (!plain(input(wk, 1), kn)) {
          return 0;
        }
        if (f.vSlice >= 0 ? !window(f.vSlice, 0, vn) : !plain(input(wv, 1), vn)) return 0;
        rt_decode_args d{};
        d.q = q;
        d.out = o;
        d.kCache = kc;
        d.vCache = vc;
        d.kNew = kn;
        d.vNew = vn;
        d.ropeCos = reinterpret_cast<float*>(cs);
        d.ropeSin = reinterpret_cast<float*>(sn);
        d.sinks = sinks;
        d.dtype = self.dtype;
        d.batch = 1;
        d.cacheRows = (int32_t)cache.rows;
        d.kvLen = (int32_t)k.rows;
        d.qHeads = (int32_t)a[0];
        d.kvHeads = (int32_t)a[1];
        d.headDim = (int32_t)a[2];
        d.windowLeft = (int32_t)a[3];
        Py_BEGIN_ALLOW_THREADS;
        status = gEntry.decode(x.ctx, &d);
        Py_END_ALLOW_THREADS;
        name = f.ropeQ >= 0 ? s_decodeRopeAppend : s_decodeAppend;
        break;
      }
      rt_attn_args t{};
      t.q = in[0];
      t.k = a[9] ? in[0] : in[1];
      t.v = a[9] ? in[0] : in[2];
      t.out = o;
      t.sinks = sinks;
      t.segments = segs;
      t.dtype = self.dtype;
      t.qkvPacked = (int32_t)a[9];
      t.qLen = m.rows;
      t.kvLen = k.rows;
      t.qHeads = (int32_t)a[0];
      t.kvHeads = (int32_t)a[1];
      t.headDim = (int32_t)a[2];
      t.windowLeft = (int32_t)a[3];
      t.windowRight = (int32_t)a[4];
      t.maxSegment = (int32_t)a[8];
      t.qPosOffset = a[5];
      Py_BEGIN_ALLOW_THREADS;
      status = gEntry.route(x.ctx, &t, &route);
      if (status == 0) status = gEntry.attn(x.ctx, &t);
      Py_END_ALLOW_THREADS;
      break;
    }
    default:
      return 0;
  }
  if (!report(x, status)) return -1;
  Ref text(route ? PyUnicode_FromString(route) : Py_NewRef(name));
  if (!text || PyList_Append(x.names.p, text.p) < 0) return -1;
  return 1;
}

// Ropes and column slices that follow one another over the same tensor (q and k rotated, v cut out
// of a fused qkv projection) from place `i` of the order on: one call for up to four of them, whose
// outputs come from acquire().  -1: an exception is set; 0: not here; else how many were run.
int dispatch_windows(Evaluation& e, Exec& x, size_t i) {
  rt_window w[RT_MAX_WINDOWS] = {};
  PyObject* source = input(e.order[i], 0);
  Meta m;
  int n = 0;
  for (; n < RT_MAX_WINDOWS && i + n < e.order.size(); n++) {
    const Node& d = e.order[i + n];
    const bool rope = d.op == kRope;
    if (d.elided || !(rope || d.op == kSliceCols) || inputs_of(d) != (rope ? 3 : 1) || input(d, 0) != source) break;
    long long a[3];
    char *p, *cs = nullptr, *sn = nullptr;
    if (!read_matrix(source, m) || slot(source, gReleasedAt) != Py_None || !buffer_ptr(slot(source, gBufferAt), p) ||
        !attr(d, 0, a[0]) || !attr(d, 1, a[1]) || (rope && !attr(d, 2, a[2])))
      break;
    if (rope) {
      PyObject *c = input(d, 1), *s = input(d, 2);
      if (Py_TYPE(c) != gValue || Py_TYPE(s) != gValue || slot(c, gReleasedAt) != Py_None ||
          slot(s, gReleasedAt) != Py_None || !buffer_ptr(slot(c, gBufferAt), cs) || !buffer_ptr(slot(s, gBufferAt), sn))
        break;
    }
    w[n].x = p;
    w[n].cosT = reinterpret_cast<float*>(cs);
    w[n].sinT = reinterpret_cast<float*>(sn);
    w[n].rows = m.rows;
    w[n].cols = m.cols;
    w[n].start = rope ? a[1] : a[0];
    w[n].width = rope ? a[2] : a[1] - a[0];
    w[n].headDim = rope ? (int32_t)a[0] : 0;
  }
  if (n < 2) return 0;
  Ref disposed(PyObject_GetAttr(x.self, s__disposed));
  if (!disposed) return -1;
  if (disposed.p != Py_False) return 0;
  Ref out[RT_MAX_WINDOWS];
  for (int k = 0; k < n; k++) {
    char* o;
    out[k].p = acquire(x, slot(e.order[i + k].v, gShapeAt));
    if (!out[k]) return -1;
    if (!buffer_ptr(out[k].p, o)) {
      PyErr_SetString(PyExc_TypeError, "acquireOutput gave no DeviceBuffer");
      return -1;
    }
    w[k].out = o;
  }
  int status;
  Py_BEGIN_ALLOW_THREADS;
  status = gEntry.windows(x.ctx, w, n, m.dtype);
  Py_END_ALLOW_THREADS;
  if (!report(x, status)) return -1;
  for (int k = 0; k < n; k++) {
    Node& d = e.order[i + k];
    if (PyList_Append(x.names.p, d.op == kRope ? s_rope : s_sliceCols) < 0) return -1;
    set_slot(d.v, gBufferAt, out[k].p);
  }
  for (int k = 0; k < n; k++)
    if (!release(e, x, e.order[i + k].inputs)) return -1;
  return n;
}

// dispatch() of the executor, with the arguments the Python loop gives it.
bool dispatch_python(Evaluation& e, Exec& x, const Node& n, PyObject* out, PyObject* extrasOf) {
  Ref list(PyList_New(inputs_of(n)));
  if (!list) return false;
  for (Py_ssize_t i = 0; i < inputs_of(n); i++) {
    PyObject* v = input(n, (int)i);
    const int at = e.find(v);
    PyObject* b = at >= 0 && e.order[at].elided ? Py_None : slot(v, gBufferAt);
    PyList_SET_ITEM(list.p, i, Py_NewRef(b));
  }
  Ref extras(Py_NewRef(Py_None));
  if (n.fused.on) {
    // {"fusedAppend": _fused_extras(plan)}, from the plan's nodes
    const Fused& f = n.fused;
    auto v = [&](int at) { return at >= 0 ? e.order[at].v : Py_None; };
    Py_DECREF(extras.p);
    extras.p = PyObject_CallFunctionObjArgs(extrasOf, v(f.k), v(f.v), v(f.ropeQ), v(f.vSlice), nullptr);
    if (!extras) return false;
  }
  Ref r(PyObject_CallMethodObjArgs(x.self, gMethodName[0], n.v, list.p, out, extras.p, nullptr));
  return bool(r);
}

// evaluate(targets, executor, extrasOf) -> True, or False if Python has to do it.
PyObject* evaluate_graph(PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3 || !gExecutor) Py_RETURN_FALSE;
  PyObject *targets = args[0], *ex = args[1];
  if (Py_TYPE(ex) != gExecutor || !(PyList_CheckExact(targets) || PyTuple_CheckExact(targets))) Py_RETURN_FALSE;
  // An executor whose methods were replaced, on the class or on the object, runs in Python.
  Ref own(PyObject_GenericGetDict(ex, nullptr));
  if (!own) return nullptr;
  for (int i = 0; i < kMethods; i++) {
    Ref method(PyObject_GetAttr(reinterpret_cast<PyObject*>(gExecutor), gMethodName[i]));
    if (!method) return nullptr;
    if (method.p != gMethod[i] || PyDict_GetItemWithError(own.p, gMethodName[i]) != nullptr) Py_RETURN_FALSE;
  }
  if (PyDict_GetItemWithError(own.p, s__lib) != gLib) Py_RETURN_FALSE;

  Evaluation e;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(targets);
  for (Py_ssize_t i = 0; i < n; i++)
    if (!collect(e, PySequence_Fast_GET_ITEM(targets, i), 0)) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < n; i++) {
    const int at = e.find(PySequence_Fast_GET_ITEM(targets, i));
    if (at >= 0) e.order[at].target = true, e.order[at].left = 1;   // (a reader that never reads)
  }
  if (e.order.empty()) Py_RETURN_TRUE;
  if (!plan_appends(e)) Py_RETURN_FALSE;
  for (const Node& m : e.order)
    for (Py_ssize_t i = 0; i < inputs_of(m); i++) {
      bool again = false;
      for (Py_ssize_t k = 0; k < i; k++) again |= input(m, (int)k) == input(m, (int)i);
      const int at = again ? -1 : e.find(input(m, (int)i));
      if (at >= 0) e.order[at].left++;
    }

  Exec x;
  x.self = ex;
  if (!exec_attr(ex, s_ctx, x.ctxObject)) return nullptr;   // (raises for a disposed executor)
  Ref handle(PyObject_GetAttr(x.ctxObject.p, s_value));
  if (!handle) return nullptr;
  if (!PyLong_CheckExact(handle.p)) Py_RETURN_FALSE;
  x.ctx = static_cast<rt_ctx*>(PyLong_AsVoidPtr(handle.p));
  if (!exec_attr(ex, s__pool, x.pool) || !exec_attr(ex, s__live, x.live) || !exec_attr(ex, s_dispatches, x.names))
    return nullptr;
  if (!PyDict_CheckExact(x.pool.p) || !PySet_CheckExact(x.live.p) || !PyList_CheckExact(x.names.p)) Py_RETURN_FALSE;

  for (size_t i = 0; i < e.order.size(); i++) {
    Node& m = e.order[i];
    if (m.elided) continue;
    if (m.op == kRope || m.op == kSliceCols) {
      const int ran = dispatch_windows(e, x, i);
      if (ran < 0) return nullptr;
      if (ran > 0) {
        i += ran - 1;
        continue;
      }
    }
    if (m.op == kWriteRows) {
      PyObject* out = slot(input(m, 0), gBufferAt);
      Ref keep(Py_NewRef(out));
      m.aliased = true;
      if (!m.skipped) {
        const int done = dispatch(e, x, m, out);
        if (done < 0 || (done == 0 && !dispatch_python(e, x, m, out, args[2]))) return nullptr;
      }
      set_slot(m.v, gBufferAt, out);
      if (!m.skipped && !release(e, x, m.inputs)) return nullptr;
      continue;   // (a skipped one's inputs are read by the fused kernel: released after that)
    }
    Ref out(acquire(x, slot(m.v, gShapeAt)));
    if (!out) return nullptr;
    const int done = dispatch(e, x, m, out.p);
    if (done < 0 || (done == 0 && !dispatch_python(e, x, m, out.p, args[2]))) return nullptr;
    set_slot(m.v, gBufferAt, out.p);
    if (!release(e, x, m.inputs)) return nullptr;
    if (m.fused.on) {
      if (!release(e, x, e.order[m.fused.k].inputs) || !release(e, x, e.order[m.fused.v].inputs)) return nullptr;
      for (int k : {m.fused.ropeQ, m.fused.ropeK, m.fused.vSlice})
        if (k >= 0 && !release(e, x, e.order[k].inputs)) return nullptr;
    }
  }
  Py_RETURN_TRUE;
}

PyObject* evaluate(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  try {
    return evaluate_graph(args, nargs);
  } catch (const std::bad_alloc&) {
    return PyErr_NoMemory();
  }
}

// ---- bind --------------------------------------------------------------------------------

bool slot_offset(PyTypeObject* type, const char* name, Py_ssize_t& at) {
  Ref d(PyObject_GetAttrString(reinterpret_cast<PyObject*>(type), name));
  if (!d || Py_TYPE(d.p) != &PyMemberDescr_Type) {
    if (!PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "%s.%s is not a slot", type->tp_name, name);
    return false;
  }
  at = reinterpret_cast<PyMemberDescrObject*>(d.p)->d_member->offset;
  return true;
}

// bind_ops(Value, ValueMeta, PendingOp, DeviceBuffer, ACT_CODE, WINDOW_INF, MAX_HEAD_DIM,
// MAX_DECODE_HEAD_DIM): from then on the constructors answer.
PyObject* bind_ops(PyObject*, PyObject* args) {
  PyObject *v, *m, *p, *b, *act;
  if (!PyArg_ParseTuple(args, "OOOOOLLL", &v, &m, &p, &b, &act, &gWindowInf, &gMaxHeadDim, &gMaxDecodeHeadDim))
    return nullptr;
  gValue = reinterpret_cast<PyTypeObject*>(Py_NewRef(v));
  gMeta = reinterpret_cast<PyTypeObject*>(Py_NewRef(m));
  gPending = reinterpret_cast<PyTypeObject*>(Py_NewRef(p));
  gBuffer = reinterpret_cast<PyTypeObject*>(Py_NewRef(b));
  gActCode = Py_NewRef(act);
  if (!slot_offset(gValue, "shape", gShapeAt) || !slot_offset(gValue, "_buffer", gBufferAt) ||
      !slot_offset(gValue, "pending", gPendingAt) || !slot_offset(gValue, "_released", gReleasedAt) ||
      !slot_offset(gBuffer, "ptr", gPtrAt) || !slot_offset(gBuffer, "owned", gOwnedAt))
    return nullptr;
  Py_RETURN_NONE;
}

// bind_executor(CudaExecutor, recycled reason, check)
PyObject* bind_executor(PyObject*, PyObject* args) {
  PyObject *ex, *reason, *check;
  if (!PyArg_ParseTuple(args, "OOO", &ex, &reason, &check)) return nullptr;
  for (int i = 0; i < kMethods; i++) {
    gMethodName[i] = PyUnicode_InternFromString(kMethodNames[i]);
    if (!gMethodName[i] || !(gMethod[i] = PyObject_GetAttr(ex, gMethodName[i]))) return nullptr;
  }
  gRecycled = Py_NewRef(reason);
  gCheck = Py_NewRef(check);
  gExecutor = reinterpret_cast<PyTypeObject*>(Py_NewRef(ex));
  Py_RETURN_NONE;
}

// bind_library(lib, addresses in the order of Entry): the library the executors hold.
PyObject* bind_library(PyObject*, PyObject* args) {
  PyObject *lib, *list;
  if (!PyArg_ParseTuple(args, "OO!", &lib, &PyTuple_Type, &list)) return nullptr;
  constexpr Py_ssize_t kCount = sizeof(Entry) / sizeof(void*);
  if (PyTuple_GET_SIZE(list) != kCount) return PyErr_Format(PyExc_ValueError, "%zd addresses expected", kCount);
  void* at[kCount];
  for (Py_ssize_t i = 0; i < kCount; i++) {
    at[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(list, i));
    if (!at[i]) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "a NULL address");
  }
  memcpy(&gEntry, at, sizeof gEntry);
  PyObject* old = gLib;
  gLib = Py_NewRef(lib);
  Py_XDECREF(old);
  Py_RETURN_NONE;
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f))
PyMethodDef kFunctions[] = {
    {"matmul", FAST(op_matmul), METH_FASTCALL, nullptr},
    {"rope", FAST(op_rope), METH_FASTCALL, nullptr},
    {"slice", FAST(op_slice), METH_FASTCALL, nullptr},
    {"sdpa", FAST(op_sdpa), METH_FASTCALL, nullptr},
    {"sdpaPacked", FAST(op_sdpa_packed), METH_FASTCALL, nullptr},
    {"writeRows", FAST(op_write_rows), METH_FASTCALL, nullptr},
    {"argmaxDot", FAST(op_argmax_dot), METH_FASTCALL, nullptr},
    {"evaluate", FAST(evaluate), METH_FASTCALL, nullptr},
    {"bind_ops", bind_ops, METH_VARARGS, nullptr},
    {"bind_executor", bind_executor, METH_VARARGS, nullptr},
    {"bind_library", bind_library, METH_VARARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Native operator constructors and eval driver.", -1, kFunctions,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
#define X(n) \
  if (!(s_##n = PyUnicode_InternFromString(#n))) return nullptr;
  RT_STRINGS(X)
#undef X
  s_decodeAppend = PyUnicode_InternFromString("decode+append");
  s_decodeRopeAppend = PyUnicode_InternFromString("decode+rope+append");
  gNoArgs = PyTuple_New(0);
  if (!s_decodeAppend || !s_decodeRopeAppend || !gNoArgs) return nullptr;
  return PyModule_Create(&kModule);
}
