"""The constructors and the eval loop in native code (csrc/host.cpp) against the Python they
stand for: the same nodes, the same refusals, the same calls of the C ABI in the same order, the
same buffers in the pool.  The library is a stub that writes its calls down (no GPU)."""
import contextlib
import ctypes as C
import importlib.util
import math
import os
import shutil
import subprocess

import pytest

import runntime_b200 as rt
from runntime_b200 import _lib as L, build as B, executor as X, ops
from runntime_b200.value import DeviceBuffer, ValueMeta, materialized

INF = math.inf
pytestmark = pytest.mark.skipif(L.host is None, reason="_host.so is not built")

STUB = r"""
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include "rt_attn.h"
static char text[1 << 20];
static int used, fail_at = -1, calls;
static char* at = (char*)0x10000;
const char* stub_log(void) { return text; }
void stub_reset(int failAt) { used = 0; text[0] = 0; fail_at = failAt; calls = 0; at = (char*)0x10000; }
static int line(const char* f, const void* a, size_t n, const char* fmt, ...) {
  (void)fmt;
  used += sprintf(text + used, "%s", f);
  const unsigned char* b = (const unsigned char*)a;
  for (size_t i = 0; i < n; i++) used += sprintf(text + used, "%02x", b[i]);
  used += sprintf(text + used, "\n");
  return calls++ == fail_at ? RT_INVALID_ARGUMENT : RT_OK;
}
#define W(...) int64_t w[] = {__VA_ARGS__}
#define I(x) (int64_t)(intptr_t)(x)
int rt_ctx_create(int d, rt_ctx** o) { *o = (rt_ctx*)0x1234; return 0; }
int rt_ctx_destroy(rt_ctx* c) { return 0; }
int rt_buf_free(rt_ctx* c, void* p) { return 0; }
int rt_buf_alloc(rt_ctx* c, size_t n, void** p) { *p = at; at += 4096; W((int64_t)n); return line("alloc ", w, sizeof w, 0); }
const char* rt_last_error(const rt_ctx* c) { return "stub"; }
int rt_attn_route(rt_ctx* c, const rt_attn_args* a, const char** r) { *r = a->qLen == 1 ? "decode" : "prefill"; return line("route ", a, sizeof *a, 0); }
int rt_attn(rt_ctx* c, const rt_attn_args* a) { return line("attn ", a, sizeof *a, 0); }
int rt_attn_decode(rt_ctx* c, const rt_decode_args* a) { return line("decode ", a, sizeof *a, 0); }
int rt_matmul(rt_ctx* c, const void* a, const void* b, const void* bias, const void* addend, void* out, int64_t m,
              int64_t k, int64_t n, int64_t bRows, int64_t baseRow, int32_t act, int32_t dtype) {
  W(I(c), I(a), I(b), I(bias), I(addend), I(out), m, k, n, bRows, baseRow, act, dtype);
  return line("matmul ", w, sizeof w, 0); }
int rt_rope(rt_ctx* c, const void* x, const float* cs, const float* sn, void* out, int64_t rows, int64_t cols,
            int32_t hd, int64_t start, int64_t width, int32_t dtype) {
  W(I(c), I(x), I(cs), I(sn), I(out), rows, cols, hd, start, width, dtype); return line("rope ", w, sizeof w, 0); }
int rt_slice(rt_ctx* c, const void* x, void* out, int64_t rows, int64_t cols, int64_t r0, int64_t r1, int64_t c0,
             int64_t c1, int32_t dtype) {
  W(I(c), I(x), I(out), rows, cols, r0, r1, c0, c1, dtype); return line("slice ", w, sizeof w, 0); }
int rt_windows(rt_ctx* c, const rt_window* w, int32_t n, int32_t dtype) {
  int s = 0;
  for (int i = 0; i < n && !s; i++)
    s = w[i].cosT ? rt_rope(c, w[i].x, w[i].cosT, w[i].sinT, w[i].out, w[i].rows, w[i].cols, w[i].headDim, w[i].start, w[i].width, dtype)
                  : rt_slice(c, w[i].x, w[i].out, w[i].rows, w[i].cols, 0, w[i].rows, w[i].start, w[i].start + w[i].width, dtype);
  return s; }
int rt_argmax_dot(rt_ctx* c, const void* a, const void* x, float* out, int64_t rows, int64_t cols, int32_t dtype) {
  W(I(c), I(a), I(x), I(out), rows, cols, dtype); return line("argmax ", w, sizeof w, 0); }
int rt_kv_append(rt_ctx* c, void* d, const void* s, int64_t start, int64_t rows, int64_t cols, int64_t dstRows, int32_t dtype) {
  W(I(c), I(d), I(s), start, rows, cols, dstRows, dtype); return line("append ", w, sizeof w, 0); }
int rt_softmax(rt_ctx* c, const void* x, void* out, const float* segs, int64_t rows, int64_t cols, int32_t wl, int32_t wr, int32_t dtype) {
  W(I(c), I(x), I(out), I(segs), rows, cols, wl, wr, dtype); return line("softmax ", w, sizeof w, 0); }
int rt_local_attention(rt_ctx* c, const void* x, const float* rel, const float* qs, void* out, int64_t rows,
                       int32_t heads, int32_t hd, int32_t window, float ks, float cap, int32_t dtype) {
  W(I(c), I(x), I(rel), I(qs), I(out), rows, heads, hd, window, (int64_t)(ks * 64), (int64_t)(cap * 64), dtype);
  return line("local ", w, sizeof w, 0); }
"""


@pytest.fixture(scope="module")
def stub(tmp_path_factory):
    if shutil.which("gcc") is None:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("stub")
    names = [n for n in L.SYMBOLS if f" {n}(" not in STUB]
    (d / "stub.c").write_text(STUB.replace('#include "rt_attn.h"', f'#include "{L._HERE}/../include/rt_attn.h"'))
    (d / "rest.c").write_text("".join(f"int {n}() {{ return 0; }}\n" for n in names))
    subprocess.check_call(["gcc", "-w", "-shared", "-fPIC", str(d / "stub.c"), str(d / "rest.c"), "-o",
                           str(d / "stub.so")])
    return str(d / "stub.so")


@contextlib.contextmanager
def stubbed(stub, monkeypatch):
    """The stub in the library's place; afterwards the native code calls the one that was there again."""
    before = L._lib
    monkeypatch.setattr(L, "LIB_PATH", stub)
    monkeypatch.setattr(L, "_lib", None)
    lib = L.load()
    lib.stub_log.restype, lib.stub_reset.argtypes = C.c_char_p, [C.c_int]
    try:
        yield lib
    finally:
        if before is not None:
            L.bind_host(before)


@pytest.fixture
def lib(stub, monkeypatch):
    with stubbed(stub, monkeypatch) as lib:
        yield lib


def python_only(monkeypatch):
    monkeypatch.setattr(ops, "_native", ops._Deferring())
    monkeypatch.setattr(X, "host", None)
    # (a node's inputs go back to the pool in the order of a set of objects: here in their own)
    monkeypatch.setattr(X, "set", lambda *a: list(dict.fromkeys(a[0])) if a else set(), raising=False)


def val(rows, cols, dtype="f16", ptr=0x1000, dims=None):
    m = ValueMeta(rows * cols, dtype, (rows, cols) if dims is None else dims)
    return materialized(m, DeviceBuffer(ptr, m.elems * 4, owned=False))


def made(fn):
    """What a constructor answers: a node in plain terms, or the error it raises."""
    try:
        v = fn()
    except Exception as e:  # noqa: BLE001
        return type(e).__name__, str(e)
    assert type(v) is rt.Value and v.state == "pending" and type(v.shape) is ValueMeta
    assert type(v.pending).__name__ == "PendingOp" and v.pending.scalar is None
    attrs = v.pending.attrs
    return (tuple(v.shape), v.pending.op, tuple((tuple(i.shape), i.state) for i in v.pending.inputs),
            None if attrs is None else tuple((type(a), a) for a in attrs))


def constructor_calls():
    x, w, wide = val(3, 16), val(16, 48), val(40, 48)
    one, f32 = val(1, 16), val(3, 16, "f32")
    flat, bias, add = val(3, 16, dims=(48,)), val(1, 48), val(3, 48)
    released = val(4, 16)
    released.markReleased("gone")
    for opts in (None, {}, {"bias": bias}, {"addend": add}, {"bias": bias, "addend": add, "activation": "gelu"},
                 {"bias": add}, {"addend": bias}, {"activation": "none"}, {"activation": "bad"}, {"activation": ""},
                 {"baseRow": 3}, {"baseRow": 0}, {"baseRow": 3.0}, {"baseRow": -1}, {"baseRow": 25},
                 {"baseRow": True}, {"baseRow": 1 << 70}, {"baseRow": (1 << 63) - 1}, {"scales": bias},
                 {"bits": 0}, {"bits": 4}, {"unknown": 1}):
        for a, b in ((x, w), (x, wide), (f32, w), (flat, w), (one, w), (w, x)):
            yield lambda a=a, b=b, o=opts: rt.matmul(a, b, o) if o is not None else rt.matmul(a, b)
    cos = val(3, 4, "f32")
    for opts in ({"headDim": 4}, {"headDim": 4, "srcStart": 8, "width": 8}, {"headDim": 4.0}, {"headDim": 3}, {},
                 {"headDim": 4, "srcStart": 3}, {"headDim": 4, "srcStart": 16, "width": 4}, {"headDim": 0},
                 {"headDim": 4, "width": 6}, {"headDim": 4, "width": None}, {"headDim": 4, "srcStart": -2},
                 {"headDim": True}):
        for a, c in ((x, cos), (f32, cos), (x, val(3, 4)), (x, val(2, 4, "f32")), (flat, cos)):
            yield lambda a=a, c=c, o=opts: rt.rope(a, c, c, o)
    for dim in (0, 1, -1, -2, 2, 1.0, "a"):
        for lo, hi in ((0, 1), (0, 3), (1, 16), (2, 2), (-1, 2), (0, 17), (0.0, 2.0), (0, True)):
            yield lambda d=dim, lo=lo, hi=hi: rt.slice(x, d, lo, hi)
    yield lambda: rt.slice(flat, 0, 0, 1)
    base = dict(qHeads=4, kvHeads=2, headDim=4, windowLeft=INF, windowRight=0)
    sinks, segs = val(1, 4, "f32"), val(3, 2, "f32")
    for extra in ({}, {"windowRight": INF}, {"windowLeft": 3}, {"windowLeft": -1}, {"windowLeft": 2.0},
                  {"windowLeft": 1 << 40}, {"windowLeft": None}, {"windowRight": -INF}, {"windowRight": math.nan},
                  {"qPosOffset": 1}, {"qPosOffset": 2}, {"qPosOffset": -1}, {"qPosOffset": 1.0}, {"sinks": sinks},
                  {"sinks": segs}, {"segments": segs}, {"segments": sinks}, {"segments": segs, "maxSegment": 3},
                  {"maxSegment": 3}, {"segments": segs, "maxSegment": 0}, {"segments": segs, "maxSegment": 2.0},
                  {"segments": segs, "sinks": sinks}, {"kvHeads": 3}, {"kvHeads": 0}, {"qHeads": 8}, {"headDim": 8},
                  {"keyBias": {}}, {"keyBias": {"start": 0, "end": 2, "value": 1.5}}, {"qHeads": 4.0},
                  {"qHeads": -4, "headDim": -4}):
        o = {**base, **extra}
        for q, k, v in ((x, val(4, 8), val(4, 8)), (one, val(4, 8), val(4, 8)), (x, val(2, 8), val(2, 8)),
                        (x, val(4, 8), val(5, 8)), (f32, val(4, 8), val(4, 8)), (x, val(4, 16), val(4, 16)),
                        (flat, val(4, 8), val(4, 8))):
            yield lambda q=q, k=k, v=v, o=o: rt.sdpa(q, k, v, o)
        for qkv in (val(3, 32), val(1, 32), val(3, 32, "f32"), val(3, 48)):
            yield lambda x=qkv, o=o: rt.sdpaPacked(x, o)
    big = {**base, "qHeads": 1, "kvHeads": 1}
    for hd in (64, 128, 129, 512, 513):
        for rows in (1, 3):
            yield lambda hd=hd, n=rows: rt.sdpa(val(n, hd), val(4, hd), val(4, hd), {**big, "headDim": hd})
            yield lambda hd=hd, n=rows: rt.sdpaPacked(val(n, 3 * hd), {**big, "headDim": hd})
    pend = rt.matmul(x, val(16, 16))
    for dst, src in ((val(8, 16), x), (released, x), (pend, x), (val(8, 16), f32), (val(2, 16), x), (val(8, 8), x),
                     (val(8, 16), pend), (flat, x)):
        for start in (0, 5, 6, -1, 2.0, 1 << 70, None):
            yield lambda d=dst, s=src, n=start: rt.writeRows(d, s, n)
    for wv, xv in ((val(9, 16), one), (val(9, 16), x), (val(9, 8), one), (val(9, 16, "f32"), one), (flat, one)):
        yield lambda a=wv, b=xv: rt.argmaxDot(a, b)


def test_constructors_answer_as_the_python_does(monkeypatch):
    calls = list(constructor_calls())
    native = [made(c) for c in calls]
    python_only(monkeypatch)
    for i, c in enumerate(calls):
        assert made(c) == native[i], i
    assert sum(isinstance(n[0], tuple) for n in native) > 100


def graph(name, ex):
    """Targets of a small graph over wrapped tensors, and all of its nodes."""
    n = [0]

    def t(rows, cols, dtype="f16"):
        n[0] += 1
        return ex.wrap(0x900000 + 0x1000 * n[0], (rows, cols), dtype)

    w, hd = 16, 4
    o = dict(qHeads=4, kvHeads=4, headDim=hd, windowLeft=INF)
    if name in ("encoder", "twice"):
        x, rows = t(5, w), 5
        qkv = rt.matmul(x, t(w, 3 * w), dict(bias=t(1, 3 * w)))
        cos, sin = t(rows, hd, "f32"), t(rows, hd, "f32")
        q = rt.rope(qkv, cos, sin, dict(headDim=hd, srcStart=0, width=w))
        k = rt.rope(qkv, cos, sin, dict(headDim=hd, srcStart=w, width=w))
        v = rt.slice(qkv, 1, 2 * w, 3 * w)
        att = rt.sdpa(q, k, v, dict(o, windowRight=INF, sinks=t(1, 4, "f32")))
        y = rt.matmul(att, t(w, w), dict(addend=x, activation="silu"))
        z = rt.matmul(rt.slice(y, 0, 1, 4), t(w, w))
        nodes = [qkv, q, k, v, att, y, z]
        return ([y, z, y] if name == "twice" else [z]), nodes
    if name == "packed":
        qkv = rt.matmul(t(6, w), t(w, 3 * w), dict(baseRow=0))
        a = rt.sdpaPacked(qkv, dict(o, windowRight=INF, segments=t(6, 2, "f32"), maxSegment=4))
        b = rt.sdpa(a, a, a, dict(o, windowRight=INF, keyBias=dict(start=0, end=2, value=0.5)))
        s = rt.softmax(rt.matmul(b, t(w, 6)), dict(segments=t(6, 2, "f32"), windowLeft=2))
        u = rt.softmax(s)
        loc = rt.localAttention(qkv, t(3, w, "f32"), t(1, hd, "f32"),
                                dict(heads=4, headDim=hd, window=3, kScale=1.0, softcap=50.0))
        return [u, loc], [qkv, a, b, s, u, loc]
    # a decoder's step, in the forms the append can take
    p, x, kc, vc = 3, t(1, w), t(8, w), t(8, w)
    qkv = rt.matmul(x, t(w, 3 * w))
    cos, sin = t(1, hd, "f32"), t(1, hd, "f32")
    q = rt.rope(qkv, cos, sin, dict(headDim=hd, srcStart=0, width=w))
    kn = rt.rope(qkv, t(1, hd, "f32") if name == "tables" else cos, sin, dict(headDim=hd, srcStart=w, width=w))
    vn = t(1, w) if name == "ownv" else rt.slice(qkv, 1, 2 * w, 3 * w)
    k, v = rt.writeRows(kc, kn, p), rt.writeRows(vc, vn, p + 1 if name == "elsewhere" else p)
    if name == "elsewhere":
        v = rt.writeRows(vc, rt.slice(v, 0, p, p + 1), p)
    att = rt.sdpa(q, k, v, dict(o, windowRight=INF if name == "cross" else 0,
                                qPosOffset=0 if name == "cross" else p))
    y = rt.matmul(att, t(w, w), dict(addend=x))
    att2 = rt.sdpa(rt.matmul(y, t(w, w)), t(9, w), t(9, w), dict(o, windowRight=INF))
    z = rt.matmul(att2, t(w, w), dict(addend=y))
    token = rt.argmaxDot(t(30, w), z)
    targets = [z, token] + ([k] if name == "keep" else []) + ([q] if name == "keepq" else [])
    return targets, [qkv, q, kn, k, v, att, y, att2, z, token]


GRAPHS = ["encoder", "twice", "packed", "step", "tables", "ownv", "elsewhere", "cross", "keep", "keepq"]


def settled(log):
    """The calls without the allocations: windows of one tensor take their outputs together."""
    return [line for line in log.split(b"\n") if not line.startswith(b"alloc")]


def run(lib, name, failAt=-1):
    lib.stub_reset(failAt)
    ex = rt.CudaExecutor(0)
    out = []
    for _ in range(2):   # the second pass meets a filled pool
        targets, nodes = graph(name, ex)
        error = None
        try:
            rt.evalValues(targets, ex)
        except Exception as e:  # noqa: BLE001
            error = type(e).__name__, str(e)
        out.append((error, list(ex.dispatches),
                    [(v.state, v.releasedReason, v._buffer and (v._buffer.ptr, v._buffer.nbytes, v._buffer.owned))
                     for v in nodes],
                    sorted((k, [b.ptr for b in bs]) for k, bs in ex._pool.items() if bs),
                    sorted(b.ptr for b in ex._live)))
        ex.releaseValues(targets)
    return out, settled(lib.stub_log())


@pytest.mark.parametrize("name", GRAPHS)
def test_evaluation_makes_the_same_calls(lib, monkeypatch, name):
    native = run(lib, name)
    failures = (1, 3, 20)   # (an allocation, the first product, a second pass's call)
    failed = [run(lib, name, at) for at in failures]
    taken = []
    real = L.host.evaluate
    monkeypatch.setattr(X, "host", type("Spy", (), {"evaluate": staticmethod(
        lambda *a: taken.append(real(*a)) or taken[-1])}))
    run(lib, name)
    assert taken == [True, True]   # it was the native loop that ran
    python_only(monkeypatch)
    assert run(lib, name) == native
    for at, native in zip(failures, failed):
        python = run(lib, name, at)
        assert [p[0] for p in python[0]] == [n[0] for n in native[0]], at
    assert any(b"matmul" in line for line in native[1])


def test_overridden_executors_and_released_values_stay_with_python(lib):
    ex = rt.CudaExecutor(0)
    seen = []
    ex.dispatch = lambda node, *a: seen.append(node.pending.op)
    (y,), _ = graph("encoder", ex)
    rt.evalValues([y], ex)
    assert seen.count("matmul") == 3

    class Mine(rt.CudaExecutor):
        def acquireOutput(self, shape):
            seen.append("acquired")
            return super().acquireOutput(shape)

    (y,), nodes = graph("encoder", Mine(0))
    rt.evalValues((y,), Mine(0))
    assert seen.count("acquired") == 8
    with pytest.raises(RuntimeError, match="buffer was recycled by eval"):
        rt.evalValues([rt.matmul(nodes[0], val(48, 4))], rt.CudaExecutor(0))
    ex = rt.CudaExecutor(0)
    (y,), _ = graph("encoder", ex)
    ex.dispose()
    with pytest.raises(rt.RunntimeError, match="executor was disposed"):
        rt.evalValues([y], ex)
    rt.evalValues([val(2, 2)], ex)   # nothing to do


def test_the_real_library_is_bound_again_after_the_stub(stub):
    if not os.path.exists(L.LIB_PATH):
        pytest.skip("librt_attn.so is not built")
    real = L.load()
    ex = X.CudaExecutor.__new__(X.CudaExecutor)
    ex._lib = real
    with pytest.MonkeyPatch.context() as m:
        with stubbed(stub, m):
            assert L.host.evaluate([val(2, 2)], ex, None) is False     # (left to Python: another library)
    assert L.load() is real and L.host.evaluate([val(2, 2)], ex, None) is True


def test_an_extension_that_does_not_compile_leaves_none_behind(tmp_path, monkeypatch):
    """A stale one goes, the rest is built all the same."""
    (tmp_path / "host.cpp").write_text("#error\n")
    stale = tmp_path / "_host.so"
    stale.write_bytes(b"old")
    os.utime(stale, (0, 0))
    monkeypatch.setattr(B, "CSRC", str(tmp_path))
    monkeypatch.setattr(B, "HOST", str(stale))
    monkeypatch.setattr(B, "_stale", lambda: False)
    with pytest.warns(UserWarning, match="host.cpp was not built"):
        assert B.build() == B.LIB
    assert sorted(p.name for p in tmp_path.iterdir()) == ["host.cpp"]


def test_the_extension_is_named_after_the_interpreter(tmp_path, monkeypatch):
    assert L.host.__file__ == B.HOST
    monkeypatch.setattr(B, "HOST", str(tmp_path / os.path.basename(B.HOST)))
    assert B.build_host() and [p.name for p in tmp_path.iterdir()] == [os.path.basename(B.HOST)]
    spec = importlib.util.spec_from_file_location("_host", B.HOST)
    assert hasattr(importlib.util.module_from_spec(spec), "evaluate")


@pytest.mark.gpu
def test_graphs_run_in_native_code_on_the_gpu(monkeypatch):
    """An evaluation of plain operators is the native code's, not the Python that stands in for it."""
    import numpy as np
    ex, said = rt.CudaExecutor(0), []

    class Watched:
        @staticmethod
        def evaluate(*a):
            said.append(L.host.evaluate(*a))
            return said[-1]

    try:
        monkeypatch.setattr(X, "host", Watched)
        x, w = ex.upload(np.eye(4, 8), [4, 8], "f16"), ex.upload(np.ones((8, 6)), [8, 6], "f16")
        got = rt.toArray(rt.slice(rt.matmul(x, w), 1, 1, 3), ex)
        assert said == [True] and (got == 1).all()
    finally:
        ex.dispose()
