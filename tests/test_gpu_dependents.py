"""Kernels launched as programmatic dependents, in chains where each reads what the one before
wrote and overwrites what that one read: back to back and as a captured graph they leave the same
bits as one by one with a wait for the GPU between them."""
import ctypes as C

import pytest

from gpu_harness import capture

pytestmark = pytest.mark.gpu


class Chain:
    """Two buffers of the same memory for all steps, weights and tables beside them."""

    def __init__(self, dtype, elems):
        import torch
        import runntime_b200 as rt
        from runntime_b200 import _lib as L
        self.torch, self.L, self.ex, self.code = torch, L, rt.CudaExecutor(0), L.DTYPE_CODE[dtype]
        self.size, self.td = (2, torch.float16) if dtype == "f16" else (4, torch.float32)
        self.g = torch.Generator(device="cuda").manual_seed(7)
        self.start = (torch.randn(elems, generator=self.g, device="cuda") * .5).to(self.td)
        self.a, self.b = self.start.clone(), torch.zeros_like(self.start)
        self.steps, self.keep, self.stream = [], [], torch.cuda.Stream()

    def tensor(self, *shape, scale=1.0, td=None):
        t = (self.torch.randn(*shape, generator=self.g, device="cuda") * scale).to(td or self.td)
        self.keep.append(t)
        return t

    def segments(self, rows, longest):
        ends = list(range(longest, rows, longest)) + [rows]
        t = self.torch.zeros(rows, 2)
        for lo, hi in zip([0] + ends, ends):
            t[lo:hi, 0], t[lo:hi, 1] = lo, hi
        t = t.cuda()
        self.keep.append(t)
        return t

    def add(self, call, *args):
        """A call of the C ABI whose pointers are tensors."""
        lib, ex = self.L.load(), self.ex
        args = [a.data_ptr() if hasattr(a, "data_ptr") else a for a in args]
        self.steps.append(lambda: self.L.check(getattr(lib, call)(ex.ctx, *args), ex.ctx))

    def attend(self, q, k, v, out, route, rows, heads, hd, **more):
        p = lambda t: t if isinstance(t, int) else t.data_ptr()  # noqa: E731
        a = self.L.AttnArgs()
        a.q, a.k, a.v, a.out, a.dtype, a.qLen, a.kvLen = p(q), p(k), p(v), p(out), self.code, rows, rows
        a.qHeads = a.kvHeads = heads
        a.headDim, a.windowLeft, a.windowRight = hd, self.L.WINDOW_INF, self.L.WINDOW_INF
        for key, value in more.items():
            setattr(a, key, value)
        name = C.c_char_p()
        self.L.check(self.L.load().rt_attn_route(self.ex.ctx, C.byref(a), C.byref(name)), self.ex.ctx)
        assert name.value.decode() == route
        self.steps.append(lambda: self.L.check(self.L.load().rt_attn(self.ex.ctx, C.byref(a)), self.ex.ctx))

    def at(self, buffer, elems):
        return buffer.data_ptr() + elems * self.size

    def run(self, wait):
        for s in self.steps:
            s()
            if wait:
                self.ex.sync()

    def check(self):
        """Twice in a row each way, from the same start."""
        torch, bits = self.torch, self.torch.int16 if self.size == 2 else self.torch.int32
        state = [t for t in self.keep if getattr(t, "changes", False)]
        first = [t.clone() for t in state]
        ways = {}
        self.ex.setStream(self.stream.cuda_stream)
        try:
            for way in ("one by one", "back to back", "graph"):
                self.a.copy_(self.start)
                self.b.zero_()
                for t, old in zip(state, first):
                    t.copy_(old)
                torch.cuda.synchronize()
                if way == "graph":
                    graph, grids = capture(lambda: self.run(False), self.stream)
                    assert len(grids) >= len(self.steps)
                    graph.replay()
                    graph.replay()
                else:
                    for _ in range(2):
                        self.run(way == "one by one")
                torch.cuda.synchronize()
                ways[way] = [t.view(bits).clone() for t in (self.a, self.b, *state)]
                if way == "graph":
                    del graph
            self.ex.sync()
        finally:
            self.ex.dispose()
        assert not torch.isnan(self.a.float()).any() and not torch.isnan(self.b.float()).any()
        for way in ("back to back", "graph"):
            for got, want in zip(ways[way], ways["one by one"]):
                assert torch.equal(got, want), way


def _layer(dtype):
    import torch
    t, heads, hd = 640, 4, 64
    w, f32 = heads * hd, torch.float32
    c = Chain(dtype, 1 << 20)
    a, b, A = c.a, c.b, c.at
    tile = c.tensor(w, 3 * w, scale=w ** -.5)
    c.add("rt_matmul", a, tile, None, None, b, t, w, 3 * w, w, 0, 0, c.code)
    angle = c.tensor(t, hd // 2, td=f32).repeat_interleave(2, 1)
    cos, sin = angle.cos().contiguous(), angle.sin().contiguous()
    c.keep += [cos, sin]
    wins = (c.L.Window * 3)()
    for i in range(3):
        o = wins[i]
        o.x, o.out, o.rows, o.cols, o.start, o.width = b.data_ptr(), A(a, i * t * w), t, 3 * w, i * w, w
        if i < 2:
            o.cosT, o.sinT, o.headDim = cos.data_ptr(), sin.data_ptr(), hd
    c.steps.append(lambda: c.L.check(c.L.load().rt_windows(c.ex.ctx, wins, 3, c.code), c.ex.ctx))
    c.attend(A(a, 0), A(a, t * w), A(a, 2 * t * w), b, "prefill_tc3" if dtype == "f16" else "prefill_f32_tc", t, heads, hd)
    rows = t // 3
    c.add("rt_local_attention", b, c.tensor(12, w, td=f32, scale=.1), c.tensor(hd, td=f32, scale=hd ** -.5), a, rows, heads,
          hd, 12, 1.0, 50.0, c.code)
    packed = rows * w // 192          # rows of two heads of 32
    segs = c.segments(packed, 40)
    c.attend(a, a, a, b, "prefill_mma" if dtype == "f16" else "prefill_f32_tc", packed, 2, 32, qkvPacked=1,
             segments=segs.data_ptr(), maxSegment=40)
    c.add("rt_softmax", b, a, c.segments(132, 30), 132, 132, c.L.WINDOW_INF, c.L.WINDOW_INF, c.code)
    c.add("rt_softmax", a, b, None, 131, 131, 0, 0, c.code)
    # (in f32 one slice of the contraction: the sums of more meet in atomics, in any order)
    deep = w if dtype == "f16" else 32
    c.add("rt_matmul", b, c.tensor(deep, 512, scale=4.), c.tensor(512), None, a, 8, deep, 512, deep, 0, 0, c.code)
    batch, kv, cache = 2, 2, 70       # two steps appended to caches of 70 rows
    d = c.L.DecodeArgs()
    k, v = c.tensor(batch, cache, kv * 64), c.tensor(batch, cache, kv * 64)
    k.changes = v.changes = True
    d.q, d.kNew, d.vNew, d.out = A(a, 0), A(a, 1024), A(a, 1536), b.data_ptr()
    d.kCache, d.vCache, d.cacheSeqStride = k.data_ptr(), v.data_ptr(), cache * kv * 64
    d.dtype, d.batch, d.cacheRows, d.kvLen = c.code, batch, cache, cache
    d.qHeads, d.kvHeads, d.headDim, d.windowLeft, d.splits = 8, kv, 64, c.L.WINDOW_INF, 2
    c.steps.append(lambda: c.L.check(c.L.load().rt_attn_decode(c.ex.ctx, C.byref(d)), c.ex.ctx))
    c.add("rt_argmax_dot", A(b, 0), A(b, 512), a, 32, 16, c.code)
    return c


@pytest.mark.parametrize("dtype", ["f16", "f32"])
def test_a_chain_of_all_kernels(dtype):
    _layer(dtype).check()


@pytest.mark.parametrize("dtype", ["f16", "f32"])
def test_a_chain_of_softmax_kernels(dtype):
    """Quads by warp and by block, chunks by warp, by block and four rows to a block, element by element."""
    c = Chain(dtype, 5003 * 5003)
    x, y, inf = c.a, c.b, c.L.WINDOW_INF
    for n, longest in ((5003, 200), (2560, 300), (5003, 1800), (1601, 100), (2053, 2053), (515, 60), (1200, 70)):
        c.add("rt_softmax", x, y, c.segments(n, longest), n, n, inf, inf, c.code)
        x, y = y, x
    c.add("rt_softmax", x, y, None, 3001, 515, 0, 0, c.code)
    c.check()
