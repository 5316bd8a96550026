"""The merge of a decode launch's key splits: more splits than lanes, more (head, split) weights
than fit at once, odd head sizes (single columns), splits that see no key, partials out."""
import numpy as np
import pytest

import oracle
from gpu_harness import ex  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("splits", [2, 17, 33, 64])
@pytest.mark.parametrize("heads,kvHeads,hd", [(8, 8, 36), (3, 1, 37), (64, 1, 128), (200, 1, 8), (5, 5, 1)])
def test_against_the_oracle(ex, dtype, splits, heads, kvHeads, hd):
    import torch
    from runntime_b200.engine import decode_batched
    batch, rows = 3, 150
    lens = [150, 1, 70]          # with 64 splits most hold no key of a short sequence
    td = torch.float16 if dtype == "f16" else torch.float32
    g = torch.Generator().manual_seed(splits * hd)
    q, k, v = (torch.randn(*s, generator=g).to(td) for s in
               ((batch, heads * hd), (batch, rows, kvHeads * hd), (batch, rows, kvHeads * hd)))
    q = (q * hd ** -0.5).to(td)
    dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
    out = torch.empty_like(dq)
    part = torch.empty(batch, heads, 2 + hd, device="cuda")
    dl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    kw = dict(dtype=dtype, batch=batch, cacheRows=rows, qHeads=heads, kvHeads=kvHeads, headDim=hd,
              kvLen=rows, kvLens=dl, splits=splits)
    decode_batched(ex, dq, out, dk, dv, **kw)
    decode_batched(ex, dq, out, dk, dv, partialsOut=part, **kw)
    ex.sync()
    for b, n in enumerate(lens):
        want = oracle.sdpa_ref(q[b:b + 1].float().numpy(), k[b, :n].float().numpy(), v[b, :n].float().numpy(),
                               qHeads=heads, kvHeads=kvHeads, headDim=hd)
        oracle.assert_close(out[b].float().cpu().numpy(), np.asarray(want).reshape(-1), dtype, f"out {b}")
        p = part[b].cpu().numpy()
        assert (p[:, 1] > 0).all()
        oracle.assert_close((p[:, 2:] / p[:, 1:2]).reshape(-1), np.asarray(want).reshape(-1), dtype, f"partials {b}")


@pytest.mark.parametrize("batch,heads,hd,rows", [(1, 8, 36, 100), (1, 8, 52, 415), (4, 32, 128, 700)])
def test_a_first_call_under_capture_needs_no_allocation(batch, heads, hd, rows):
    """A graph is captured before the context has any scratch for splits, and once more with
    too little of it."""
    import torch
    import runntime_b200 as rt
    from runntime_b200.engine import decode_batched
    w = heads * hd
    g = torch.Generator().manual_seed(rows)
    q, k, v = (torch.randn(*s, generator=g).half() for s in ((batch, w), (batch, rows, w), (batch, rows, w)))
    q = (q * hd ** -0.5).half()
    dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
    out = torch.empty_like(dq)
    e = rt.CudaExecutor(0)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        e.setStream(stream.cuda_stream)
        call = lambda n: decode_batched(e, dq, out, dk, dv, dtype="f16", batch=batch, cacheRows=rows,  # noqa: E731
                                        qHeads=heads, kvHeads=heads, headDim=hd, kvLen=n)
        for warm in (None, 1):
            if warm:    # scratch for a shorter call than the one captured
                decode_batched(e, dq, out, dk, dv, dtype="f16", batch=1, cacheRows=rows, qHeads=heads,
                               kvHeads=heads, headDim=hd, kvLen=rows, splits=2)
                e.sync()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                call(rows)
            out.fill_(7)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            got = out.float().cpu().numpy()
            for b in range(batch):
                want = oracle.sdpa_ref(q[b:b + 1].float().numpy(), k[b].float().numpy(), v[b].float().numpy(),
                                       qHeads=heads, kvHeads=heads, headDim=hd)
                oracle.assert_close(got[b], np.asarray(want).reshape(-1), "f16", f"warm {warm} {b}")
            del graph
    finally:
        e.dispose()


def test_a_graph_keeps_its_scratch_when_a_larger_call_needs_more():
    import torch
    import runntime_b200 as rt
    from runntime_b200.engine import decode_batched
    heads, hd, rows, w = 8, 36, 415, 288
    g = torch.Generator().manual_seed(9)
    q, k, v = (torch.randn(*s, generator=g).half() for s in ((1, w), (rows, w), (rows, w)))
    q = (q * hd ** -0.5).half()
    dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
    out = torch.empty_like(dq)
    e = rt.CudaExecutor(0)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        e.setStream(stream.cuda_stream)
        kw = dict(dtype="f16", cacheRows=rows, qHeads=heads, kvHeads=heads, headDim=hd, kvLen=rows)
        decode_batched(e, dq, out, dk, dv, batch=1, splits=13, **kw)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            decode_batched(e, dq, out, dk, dv, batch=1, splits=13, **kw)
        n = 64
        many = [x.expand(n, *x.shape).contiguous() for x in (dq.view(-1), dk, dv)]
        torch.cuda.synchronize()
        for splits in (13, 60):     # two larger scratches
            decode_batched(e, many[0], torch.empty_like(many[0]), many[1], many[2], batch=n, splits=splits, **kw)
        e.sync()
        taken = [torch.full((1 << 18,), 7.0, device="cuda") for _ in range(8)]   # freed memory would be theirs
        out.fill_(7)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        want = oracle.sdpa_ref(*(x.float().numpy() for x in (q, k, v)), qHeads=heads, kvHeads=heads, headDim=hd)
        oracle.assert_close(out.float().cpu().numpy().reshape(-1), np.asarray(want).reshape(-1), "f16", "replayed")
        assert all(bool((t == 7).all()) for t in taken)
        del graph
    finally:
        e.dispose()
