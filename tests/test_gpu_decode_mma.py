"""Decode of f16 caches on the tensor cores (csrc/decode.cu, decode_mma_kernel): several query heads
per kv head, and many wide heads over short caches."""
import math

import numpy as np
import pytest

import oracle
from gpu_harness import ex  # noqa: F401
from oracle import sdpa_ref

pytestmark = pytest.mark.gpu

# (query heads, kv heads, head size): one warp per kv head, two, four and eight; head blocks;
# the largest group; one query head each
SHAPES = [(16, 8, 36), (8, 4, 52), (6, 2, 64), (8, 1, 128), (64, 8, 128), (32, 16, 128), (32, 32, 128), (24, 24, 128)]
LENS = [1, 2, 15, 16, 17, 31, 33, 64, 65, 127, 130, 300]


def _state(heads, kv, hd, rows, batch, seed=0, scale=1.0):
    import torch
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    rnd = lambda *s, f=1.0: (torch.randn(*s, generator=g, device=dev) * f).half()  # noqa: E731
    return dict(q=rnd(batch, heads * hd, f=scale * hd ** -0.5), k=rnd(batch, rows, kv * hd), v=rnd(batch, rows, kv * hd),
                kn=rnd(batch, kv * hd), vn=rnd(batch, kv * hd),
                sinks=torch.randn(heads, generator=g, device=dev))


def _decode(ex, s, heads, kv, hd, lens, **opts):
    import torch
    from runntime_b200.engine import decode_batched
    out = torch.empty_like(s["q"])
    dl = torch.tensor(lens, dtype=torch.int32, device=out.device)
    ex.setStream(torch.cuda.current_stream().cuda_stream)
    try:
        decode_batched(ex, s["q"], out, s["k"], s["v"], dtype="f16", batch=len(lens), cacheRows=s["k"].shape[1],
                       qHeads=heads, kvHeads=kv, headDim=hd, kvLen=max(lens), kvLens=dl, **opts)
        ex.sync()
    finally:
        ex.setStream(None)
    return out.float().cpu().numpy()


@pytest.mark.parametrize("heads,kv,hd", SHAPES)
@pytest.mark.parametrize("splits", [0, 1, 3])
@pytest.mark.parametrize("append,sinks,window", [(True, False, None), (False, True, None), (True, True, 40)])
def test_against_oracle(ex, heads, kv, hd, splits, append, sinks, window):
    s = _state(heads, kv, hd, 320, len(LENS), seed=hd + heads)
    old = s["k"].clone(), s["v"].clone()
    opts = dict(splits=splits, windowLeft=window)
    if append:
        opts.update(kNew=s["kn"], vNew=s["vn"])
    if sinks:
        opts.update(sinks=s["sinks"])
    got = _decode(ex, s, heads, kv, hd, LENS, **opts)
    for b, n in enumerate(LENS):
        k, v = old[0][b].clone(), old[1][b].clone()
        if append:
            k[n - 1], v[n - 1] = s["kn"][b], s["vn"][b]
        assert (s["k"][b] == k).all() and (s["v"][b] == v).all()   # the appended row, and nothing else
        want = sdpa_ref(s["q"][b:b + 1].float().cpu().numpy(), k[:n].float().cpu().numpy(), v[:n].float().cpu().numpy(),
                        qHeads=heads, kvHeads=kv, headDim=hd, qPosOffset=n - 1,
                        windowLeft=math.inf if window is None else window, windowRight=0,
                        sinks=s["sinks"].cpu().numpy() if sinks else None)
        oracle.assert_close(got[b], want.reshape(-1), "f16", f"length {n}")


@pytest.mark.parametrize("heads,kv,hd", [(16, 8, 36), (8, 2, 64), (32, 8, 128), (32, 32, 128)])
@pytest.mark.parametrize("splits", [1, 2])
def test_infinities_and_nan_stay_where_they_are(ex, heads, kv, hd, splits):
    """Infinite values give infinite columns of their own head, whatever half of a probability they
    meet; a NaN key makes its head NaN.  Everything else keeps its value."""
    lens = [40, 40, 40, 40]
    s = _state(heads, kv, hd, 64, 4, seed=5)
    group = heads // kv
    clean = _decode(ex, s, heads, kv, hd, lens, splits=splits).reshape(4, heads, hd)
    s["v"].view(4, 64, kv, hd)[0, 7, kv - 1, 3] = math.inf
    s["v"].view(4, 64, kv, hd)[1, 39, 0, hd - 1] = -math.inf     # the last key
    s["v"].view(4, 64, kv, hd)[2, 45, 0, 1] = math.inf           # past the length: not read
    s["k"].view(4, 64, kv, hd)[3, 21, 0, 2] = math.nan
    got = _decode(ex, s, heads, kv, hd, lens, splits=splits).reshape(4, heads, hd)
    want = clean.copy()
    want[0, (kv - 1) * group:, 3] = math.inf
    want[1, :group, hd - 1] = -math.inf
    want[3, :group] = math.nan
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert (np.sign(got[np.isinf(want)]) == np.sign(want[np.isinf(want)])).all()
    # (heads computed again key by key round their sums in another order: one ulp of f16)
    assert (np.abs(got[ok] - want[ok]) <= 2.0 ** -10 * np.abs(want[ok]) + 2.0 ** -14).all()


def test_no_less_precise_than_f32_sums(ex):
    """Long caches and steep scores: the error against 64 bits is that of rounding the result."""
    heads, kv, hd, n = 16, 4, 128, 3000
    s = _state(heads, kv, hd, n, 2, seed=9, scale=4.0)
    got = _decode(ex, s, heads, kv, hd, [n, n]).astype(np.float64)
    for b in range(2):
        q, k, v = (s[x][b].double().cpu().numpy() for x in ("q", "k", "v"))
        k, v = (np.repeat(t.reshape(n, kv, hd), heads // kv, 1) for t in (k, v))
        w = np.einsum("hd,nhd->hn", q.reshape(heads, hd), k)
        w = np.exp(w - w.max(1, keepdims=True))
        want = np.einsum("hn,nhd->hd", w / w.sum(1, keepdims=True), v).reshape(-1)
        nearest = want.astype(np.float16).astype(np.float64)
        # (a handful of results lie so near the middle of two halves that 24 bits decide either way)
        assert (got[b] != nearest).mean() < 0.01
        assert np.linalg.norm(got[b] - want) <= np.linalg.norm(nearest - want) * 1.01


@pytest.mark.parametrize("heads,kv,hd,batch,rows,runs", [
    (64, 32, 36, 275, 2048, True),    # the FP32 kernel would not split it, the tensor cores would: they take it whole
    (16, 8, 128, 300, 1000, False),   # both would split it
    (8, 1, 128, 1024, 8192, False),   # only the FP32 kernel would
])
def test_where_the_fixed_scratch_holds_no_splits(heads, kv, hd, batch, rows, runs):
    import ctypes as C
    import torch
    import runntime_b200._lib as L
    lib = L.load()
    s = _state(heads, kv, hd, rows, 1)
    g = torch.Generator(device=s["q"].device).manual_seed(3)
    q = (torch.randn(batch, heads * hd, generator=g, device=s["q"].device) * hd ** -0.5).half()
    out = torch.full_like(q, 9.0)
    k, v = (torch.full((batch,), s[x].data_ptr(), dtype=torch.int64, device=q.device) for x in "kv")   # one cache for all
    a = L.DecodeArgs()
    a.q, a.out, a.kCachePtrs, a.vCachePtrs = q.data_ptr(), out.data_ptr(), k.data_ptr(), v.data_ptr()
    a.dtype, a.batch, a.cacheRows, a.kvLen = L.DTYPE_CODE["f16"], batch, rows, rows
    a.qHeads, a.kvHeads, a.headDim, a.windowLeft = heads, kv, hd, L.WINDOW_INF
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.rt_attn_decode_noalloc(C.byref(a), stream) == (0 if runs else 6)   # 6: INVALID_ARGUMENT
    assert lib.rt_attn_decode_noalloc_status(stream) == 0
    if not runs:
        assert (out == 9.0).all()
        return
    for b in (0, batch - 1):
        want = sdpa_ref(q[b:b + 1].float().cpu().numpy(), s["k"][0].float().cpu().numpy(), s["v"][0].float().cpu().numpy(),
                        qHeads=heads, kvHeads=kv, headDim=hd, qPosOffset=rows - 1, windowRight=0)
        oracle.assert_close(out[b].float().cpu().numpy(), want.reshape(-1), "f16", f"sequence {b}")


def test_given_splits_under_capture_with_the_other_kernels_counters():
    """32 heads of 128 are one block of the FP32 kernel and four of this one: a context warmed by the
    former has counters for too few of the latter, and none can be made under a capture."""
    import torch
    import runntime_b200 as rt
    heads, hd, rows, batch = 32, 128, 200, 4
    s = _state(heads, heads, hd, rows, batch)
    ex = rt.CudaExecutor(0)
    lens = torch.tensor([200, 1, 130, 64], dtype=torch.int32, device=s["q"].device)
    out = torch.empty_like(s["q"])
    from runntime_b200.engine import decode_batched
    kw = dict(batch=batch, cacheRows=rows, qHeads=heads, kvHeads=heads, headDim=hd, kvLen=rows, kvLens=lens, splits=3)
    stream = torch.cuda.Stream()
    try:
        ex.setStream(stream.cuda_stream)
        f = {x: s[x].float() for x in ("q", "k", "v")}
        torch.cuda.synchronize()
        decode_batched(ex, f["q"], torch.empty_like(f["q"]), f["k"], f["v"], dtype="f32", **kw)
        ex.sync()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            decode_batched(ex, s["q"], out, s["k"], s["v"], dtype="f16", **kw)
        graph.replay()
        torch.cuda.synchronize()
        for b, n in enumerate(lens.tolist()):
            want = sdpa_ref(s["q"][b:b + 1].float().cpu().numpy(), s["k"][b, :n].float().cpu().numpy(),
                            s["v"][b, :n].float().cpu().numpy(), qHeads=heads, kvHeads=heads, headDim=hd,
                            qPosOffset=n - 1, windowRight=0)
            oracle.assert_close(out[b].float().cpu().numpy(), want.reshape(-1), "f16", f"length {n}")
        del graph
    finally:
        ex.dispose()
