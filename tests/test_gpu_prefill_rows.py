"""Prefill in 16-row pieces: padded batches and packed segments of short sequences on either side of the
lengths at which the tile kernels take over, rows off four-element boundaries, and values that are not
finite beside rows that do not see them.  Against attention in f64 at the suite's tolerance."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_harness import ex  # noqa: F401

pytestmark = pytest.mark.gpu


def run(ex, dtype, hd, lens, stride, heads, kvHeads, wl=None, packed=False, odd=None):
    """Sequences of `lens` rows, `stride` rows apart with NaN between them (padded batch), or
    back to back (packed segments); the route and the largest sequence's rows are checked."""
    import torch
    from runntime_b200._lib import AttnArgs, DTYPE_CODE, WINDOW_INF, check
    td = torch.float16 if dtype == "f16" else torch.float32
    g = torch.Generator().manual_seed(hd * 1000 + stride)
    t = sum(lens) if packed else len(lens) * stride
    starts = [sum(lens[:b]) if packed else b * stride for b in range(len(lens))]
    q, k, v = (torch.randn(t, n * hd, generator=g).mul(s).to(td) for n, s in
               ((heads, hd ** -0.5), (kvHeads, 1.0), (kvHeads, 1.0)))
    if odd is not None:
        v[starts[0] + lens[0] - 1, 1] = odd      # seen by the first sequence only
    want = torch.zeros(t, heads * hd, dtype=torch.float64)
    live = torch.zeros(t, dtype=torch.bool)
    for b, n in enumerate(lens):
        r = slice(starts[b], starts[b] + n)
        live[r] = True
        d = torch.arange(n)[None] - torch.arange(n)[:, None]
        mask = d < -wl if wl is not None else torch.zeros(n, n, dtype=torch.bool)
        for h in range(heads):
            y = h // (heads // kvHeads)
            c, ck = slice(h * hd, h * hd + hd), slice(y * hd, y * hd + hd)
            p = torch.softmax((q[r, c].double() @ k[r, ck].double().T).masked_fill(mask, -torch.inf), -1)
            want[r, c] = p @ v[r, ck].double()
    for x in (q, k, v):
        x[~live] = float("nan")
    dq, dk, dv = (torch.cat([q, k, v], 1).cuda(),) * 3 if packed else (q.cuda(), k.cuda(), v.cuda())
    out = torch.full((t, heads * hd), 7.0, dtype=td, device="cuda")
    a = AttnArgs()
    a.q, a.k, a.v, a.out = dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), out.data_ptr()
    a.dtype, a.qLen, a.kvLen, a.qHeads, a.kvHeads, a.headDim = DTYPE_CODE[dtype], t, t, heads, kvHeads, hd
    a.windowLeft, a.windowRight = WINDOW_INF if wl is None else wl, WINDOW_INF
    if packed:
        segs = torch.tensor([[s, s + n] for s, n in zip(starts, lens) for _ in range(n)], dtype=torch.float32).cuda()
        a.qkvPacked, a.segments, a.maxSegment = 1, segs.data_ptr(), max(lens)
    else:
        dl = torch.tensor(lens, dtype=torch.int32, device="cuda")
        a.seqStride, a.seqLens = stride, dl.data_ptr()
    route = C.c_char_p()
    check(ex._lib.rt_attn_route(ex.ctx, C.byref(a), C.byref(route)), ex.ctx)
    torch.cuda.synchronize()
    check(ex._lib.rt_attn(ex.ctx, C.byref(a)), ex.ctx)
    ex.sync()
    return out.float().cpu().numpy(), want.numpy(), route.value.decode()


# heads of every column block, strides of one and of several sequences to 16 rows, few blocks and many
@pytest.mark.parametrize("hd", [4, 32, 36, 64, 100, 128, 256])
@pytest.mark.parametrize("stride,batch,heads,kvHeads", [(2, 700, 2, 1), (3, 5, 2, 2), (16, 40, 8, 8), (17, 330, 1, 1),
                                                        (33, 100, 4, 2), (64, 80, 2, 1), (113, 40, 2, 2)])
def test_short_padded_batches(ex, hd, stride, batch, heads, kvHeads):
    lens = [max(1, stride - (5 * b) % (stride // 2 + 1)) for b in range(batch)]
    got, want, route = run(ex, "f32", hd, lens, stride, heads, kvHeads)
    oracle.assert_close(got.reshape(-1), want.reshape(-1), "f32", f"{hd} {stride}")
    if stride == 2:
        assert route == "prefill_simt"
    if stride > 64 and hd > 64:
        assert route == "prefill_f32_tc"


@pytest.mark.parametrize("hd,stride,batch,heads", [(80, 2, 300, 2), (80, 30, 4, 2), (100, 64, 40, 8), (512, 3, 60, 2),
                                                   (20, 24, 9, 1), (36, 16, 9, 1)])
def test_short_padded_batches_in_halves(ex, hd, stride, batch, heads):
    lens = [max(1, stride - b % 3) for b in range(batch)]
    got, want, _ = run(ex, "f16", hd, lens, stride, heads, 1)
    oracle.assert_close(got.reshape(-1), want.reshape(-1), "f16", f"{hd} {stride}")


@pytest.mark.parametrize("hd", [8, 32, 64, 128])
@pytest.mark.parametrize("n,count", [(5, 300), (16, 9), (40, 70), (97, 60)])
def test_short_segments(ex, hd, n, count):
    got, want, _ = run(ex, "f32", hd, [max(1, n - b % 4) for b in range(count)], n, 4, 4, wl=20, packed=True)
    oracle.assert_close(got.reshape(-1), want.reshape(-1), "f32", f"{hd} {n}")


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("hd", [1, 5, 33, 63, 97, 129, 255, 511])
def test_rows_off_four_elements(ex, dtype, hd):
    got, want, route = run(ex, dtype, hd, [70, 1, 45], 70, 3, 1)
    assert route == "prefill_simt"
    oracle.assert_close(got.reshape(-1), want.reshape(-1), dtype, f"{hd}")


@pytest.mark.parametrize("hd", [33, 64])
@pytest.mark.parametrize("odd", [np.inf, -np.inf, np.nan])
def test_an_odd_value_stays_with_its_sequence(ex, hd, odd):
    lens = [5] * 400
    got, want, _ = run(ex, "f32", hd, lens, 7, 1, 1, odd=odd)
    assert np.isfinite(got[7:]).all() and not np.isfinite(got[:5, 1]).any()
    oracle.assert_close(got[7:].reshape(-1), want[7:].reshape(-1), "f32", f"{odd}")
    oracle.assert_close(got[:5, 2:].reshape(-1), want[:5, 2:].reshape(-1), "f32", f"{odd}")
