"""Decode of f16 caches on the tensor cores (csrc/decode.cu, decode_mma_kernel): several query heads
per kv head, and many wide heads over short caches."""
import math

import numpy as np
import pytest

import oracle
from gpu_harness import capture, ex  # noqa: F401
from oracle import sdpa_ref

pytestmark = pytest.mark.gpu

# (query heads, kv heads, head size): one warp per kv head, two, four and eight; head blocks;
# the largest group; one query head each
SHAPES = [(16, 8, 36), (8, 4, 52), (6, 2, 64), (8, 1, 128), (64, 8, 128), (32, 16, 128), (32, 32, 128), (24, 24, 128),
          (32, 8, 36), (16, 2, 36), (64, 8, 52), (5, 1, 52), (56, 8, 64)]
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


@pytest.mark.parametrize("heads,kv,hd", [(16, 8, 36), (8, 2, 64), (32, 8, 128), (32, 32, 128), (8, 2, 36), (32, 4, 52)])
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


@pytest.mark.parametrize("heads,kv,hd", [(16, 2, 36), (8, 2, 64), (32, 8, 128)])
@pytest.mark.parametrize("splits", [1, 2])
def test_a_key_of_minus_infinity_weighs_nothing(ex, heads, kv, hd, splits):
    """Its score is -inf for a query that is positive there, also for one whose lower bits are zeros (the
    part of it that the tensor core multiplies the infinity with)."""
    lens, at = [40, 40], (7, 33)
    s = _state(heads, kv, hd, 64, 2, seed=11)
    q, k = s["q"].view(2, heads, hd), s["k"].view(2, 64, kv, hd)
    q[0, :, 2], q[1, :, 2] = 0.5, 0.3337
    for b in range(2):
        k[b, at[b], :, 2] = -math.inf
    got = _decode(ex, s, heads, kv, hd, lens, splits=splits)
    for b, n in enumerate(lens):
        left = [i for i in range(n) if i != at[b]]
        want = sdpa_ref(s["q"][b:b + 1].float().cpu().numpy(), s["k"][b, left].float().cpu().numpy(),
                        s["v"][b, left].float().cpu().numpy(), qHeads=heads, kvHeads=kv, headDim=hd, qPosOffset=n - 2,
                        windowRight=0)
        oracle.assert_close(got[b], want.reshape(-1), "f16", f"sequence {b}")


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


def _partials(ex, q, k, v, kv, group, hd, sinks, **opts):
    import torch
    from runntime_b200.engine import decode_batched
    batch, rows = k.shape[:2]
    part = torch.empty(batch, kv * group, 2 + hd, device=k.device)
    ex.setStream(torch.cuda.current_stream().cuda_stream)
    try:
        decode_batched(ex, q.reshape(batch, -1).contiguous(), None, k.reshape(batch, rows, -1).contiguous(),
                       v.reshape(batch, rows, -1).contiguous(), dtype="f16", batch=batch, cacheRows=rows,
                       qHeads=kv * group, kvHeads=kv, headDim=hd, kvLen=rows, partialsOut=part,
                       sinks=None if sinks is None else sinks.reshape(-1).contiguous(), **opts)
        ex.sync()
    finally:
        ex.setStream(None)
    return part


@pytest.mark.parametrize("kv,group,hd", [(8, 8, 36), (2, 4, 36), (2, 4, 52), (8, 8, 52), (8, 4, 64), (2, 4, 64),
                                         (8, 2, 128), (8, 4, 128), (8, 8, 128)])
@pytest.mark.parametrize("rows", [50, 487, 3000])
@pytest.mark.parametrize("kind,scale", [("flat", .1), ("plain", 1), ("steep", 4), ("steeper", 16), ("sink", 1),
                                        ("top", 1)])
def test_partials_no_less_precise_than_the_f32_kernels(ex, kv, group, hd, rows, kind, scale):
    """The f32 rows that leave the kernel against 64 bits.  The yardstick is the FP32 kernel on the same
    heads: it takes the call with 3 or 9 kv heads, these among them.  sink: e^20 times what the keys come to;
    top: a key that outweighs the others by about 2^40 and whose values are zeros, so that the
    output is what the others come to."""
    import torch
    dev, batch, more = torch.device("cuda", 0), 16, 9 if kv == 8 else 3
    g = torch.Generator(device=dev).manual_seed(hd + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)  # noqa: E731
    q = (rnd(batch, more, group, hd) * hd ** -0.5 * scale).half()
    k, v, sinks = rnd(batch, rows, more, hd).half(), rnd(batch, rows, more, hd).half(), None
    if kind == "sink":
        sinks = rnd(more, group) * 2 + 30
    if kind == "top":     # one query head of a group, in turn, along the key
        at = torch.arange(batch, device=dev)
        qt = q[at, :, at % group].float()
        k[at, at * 3] = (qt * (28 / qt.square().sum(-1, keepdim=True))).half()
        v[at, at * 3] = 0
    own = lambda t, d: t.narrow(d, 0, kv)  # noqa: E731
    s = torch.einsum("bkgd,bnkd->bkgn", own(q, 1).double(), own(k, 2).double())
    m = s.amax(-1, keepdim=True)
    if sinks is not None:
        sk = (own(sinks, 0).double() * math.log(2)).view(1, kv, group, 1)
        m = torch.maximum(m, sk)
    w = torch.exp(s - m)
    total = w.sum(-1, keepdim=True) + (0 if sinks is None else torch.exp(sk - m))
    want = (torch.einsum("bkgn,bnkd->bkgd", w, own(v, 2).double()) / total).reshape(batch, kv * group, hd)
    wantLog = (m + torch.log(total)).reshape(batch, kv * group)

    def errors(part):
        part = part.double()
        e = (part[..., 2:] / part[..., 1:2] - want).norm(dim=-1) / want.norm(dim=-1)
        z = part[..., 0] + torch.log(part[..., 1]) - wantLog
        return e.square().mean().sqrt().item(), z.square().mean().sqrt().item()

    for splits in (1, 3):
        mine = errors(_partials(ex, own(q, 1), own(k, 2), own(v, 2), kv, group, hd,
                                None if sinks is None else own(sinks, 0), splits=splits))
        f32 = _partials(ex, q, k, v, more, group, hd, sinks, splits=splits)
        f32 = errors(f32.view(batch, more, group, -1)[:, :kv].reshape(batch, kv * group, -1))
        # (both are sums of independent roundings: in another order, the FP32 kernel's own differ by up to
        # 1.3; half an ulp of the numbers compared.  Under one key the output is divided by that key's
        # weight, and so carries its score's last rounding: half an ulp of 28)
        assert mine[0] <= 1.3 * f32[0] + 2.0 ** -24 * (28 if kind == "top" else 1), (splits, mine, f32)
        assert mine[1] <= 1.3 * f32[1] + 2.0 ** -24 * max(1.0, wantLog.abs().max().item()), (splits, mine, f32)


@pytest.mark.parametrize("heads,kv,hd", [(32, 8, 128), (8, 1, 128), (8, 2, 52), (64, 8, 36), (32, 32, 128)])
@pytest.mark.parametrize("splits", [0, 2])
def test_shards_with_append_merge_to_the_whole(ex, heads, kv, hd, splits):
    """Caches cut into shards of 96 rows, rope and the appended row included: each shard's partials,
    merged, are the attention over the whole sequence; the row goes to one shard."""
    import torch
    from runntime_b200.engine import decode_batched, merge_partials
    lens, per, parts = [250, 1, 96, 97, 192, 193], 96, 3
    batch, rows = len(lens), per * parts
    s = _state(heads, kv, hd, rows, batch, seed=heads + hd)
    dev = s["q"].device
    g = torch.Generator(device=dev).manual_seed(1)
    angle = torch.rand(rows, hd // 2, generator=g, device=dev).repeat_interleave(2, 1) * 6
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    dl = torch.tensor(lens, dtype=torch.int32, device=dev)
    kw = dict(dtype="f16", batch=batch, qHeads=heads, kvHeads=kv, headDim=hd, kvLen=max(lens), kvLens=dl, kNew=s["kn"],
              vNew=s["vn"], ropeCos=cos, ropeSin=sin, ropeByPosition=True)
    shards = [(s["k"][:, r * per:(r + 1) * per].contiguous(), s["v"][:, r * per:(r + 1) * per].contiguous())
              for r in range(parts)]
    parted = torch.empty(parts, batch, heads, 2 + hd, device=dev)
    whole, out = torch.empty_like(s["q"]), torch.empty_like(s["q"])
    ex.setStream(torch.cuda.current_stream().cuda_stream)
    try:
        for r, (k, v) in enumerate(shards):
            decode_batched(ex, s["q"], None, k, v, cacheRows=per, kvSharded=True, shardStart=r * per,
                           partialsOut=parted[r], splits=splits, **kw)
        merge_partials(ex, parted, parts, batch * heads, hd, out, "f16")
        decode_batched(ex, s["q"], whole, s["k"], s["v"], cacheRows=rows, splits=splits, **kw)
        ex.sync()
    finally:
        ex.setStream(None)
    assert torch.equal(torch.cat([k for k, _ in shards], 1), s["k"])
    assert torch.equal(torch.cat([v for _, v in shards], 1), s["v"])
    for b, n in enumerate(lens):
        assert (parted[(n - 1) // per + 1:, b, :, 1] == 0).all()      # shards past the sequence's end
    # (two orders of f32 sums, each rounded to f16 once: an ulp)
    assert ((out.float() - whole.float()).abs() <= 2.0 ** -10 * whole.float().abs() + 2.0 ** -14).all()


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


@pytest.mark.parametrize("splits", [3, 0])
def test_splits_under_capture_with_the_other_kernels_counters(splits):
    """32 heads of 128 are one block of the FP32 kernel and four of this one: a context warmed by the
    former has counters for too few of the latter, and none can be made under a capture.  The FP32 kernel
    then takes the call, and splits it."""
    import torch
    import runntime_b200 as rt
    heads, hd, rows, batch = 32, 128, 200, 4
    s = _state(heads, heads, hd, rows, batch)
    ex = rt.CudaExecutor(0)
    lens = torch.tensor([200, 1, 130, 64], dtype=torch.int32, device=s["q"].device)
    out = torch.empty_like(s["q"])
    from runntime_b200.engine import decode_batched
    kw = dict(batch=batch, cacheRows=rows, qHeads=heads, kvHeads=heads, headDim=hd, kvLen=rows, kvLens=lens)
    stream = torch.cuda.Stream()
    try:
        ex.setStream(stream.cuda_stream)
        f = {x: s[x].float() for x in ("q", "k", "v")}
        torch.cuda.synchronize()
        decode_batched(ex, f["q"], torch.empty_like(f["q"]), f["k"], f["v"], dtype="f32", splits=3, **kw)
        ex.sync()
        graph, grids = capture(lambda: decode_batched(ex, s["q"], out, s["k"], s["v"], dtype="f16", splits=splits, **kw),
                               stream)
        assert grids[0][1:] == (batch, 1)      # all heads in a block: the FP32 kernel
        assert grids[0][0] == splits if splits else grids[0][0] > 1
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


def test_splits_under_capture_without_scratch_for_the_other_kernel():
    """Too few counters, and no scratch for two splits of either kernel: the tensor cores take the call whole."""
    import torch
    import runntime_b200 as rt
    from runntime_b200.engine import decode_batched
    heads, hd, rows, batch = 32, 128, 200, 4
    s = _state(heads, heads, hd, rows, batch)
    out, stream, ex = torch.empty_like(s["q"]), torch.cuda.Stream(), rt.CudaExecutor(0)
    torch.cuda.synchronize()
    try:
        ex.setStream(stream.cuda_stream)
        graph, grids = capture(lambda: decode_batched(
            ex, s["q"], out, s["k"], s["v"], dtype="f16", batch=batch, cacheRows=rows, qHeads=heads, kvHeads=heads,
            headDim=hd, kvLen=rows), stream)
        assert grids == [(1, batch, 4)]
        graph.replay()
        torch.cuda.synchronize()
        for b in range(batch):
            want = sdpa_ref(s["q"][b:b + 1].float().cpu().numpy(), s["k"][b].float().cpu().numpy(),
                            s["v"][b].float().cpu().numpy(), qHeads=heads, kvHeads=heads, headDim=hd, windowRight=0,
                            qPosOffset=rows - 1)
            oracle.assert_close(out[b].float().cpu().numpy(), want.reshape(-1), "f16", f"sequence {b}")
        del graph
    finally:
        ex.dispose()
