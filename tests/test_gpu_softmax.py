"""Row softmax on the GPU against the f64 oracle: the reference suite's shapes,
known answers and masks
(packages/runntime/test/core/kernels/reduce/softmax.gpu.test.ts:57-170)."""
import math

import numpy as np
import pytest

import oracle
from gpu_harness import ex  # noqa: F401

pytestmark = pytest.mark.gpu
INF = math.inf

# f32: exp and the division are a few ulp each; f16 output adds 2^-11 relative.
TOLERANCE = {"f32": dict(atol=1e-7, rtol=1e-5), "f16": dict(atol=1e-5, rtol=2e-3)}


def close(got, want, dtype):
    t = TOLERANCE[dtype]
    want = np.asarray(want, np.float64).reshape(-1)
    bad = np.abs(got - want) > t["atol"] + t["rtol"] * np.abs(want)
    assert not bad.any(), f"{bad.sum()} of {bad.size} off, worst {np.abs(got - want).max()}"


SHAPES = [(3, 4), (5, 128), (2, 260), (1, 32768), (70000, 4), (1, 1), (3, 7), (4, 65),
          (37, 1001), (70000, 3), (9, 2048), (3, 2052), (2, 4099)]


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_softmax_shapes(ex, dtype, rows, cols):
    import runntime_b200 as rt
    # Scaled so a row spans e^+-8 and the running max has to rescale the sum.
    x = 8 * oracle.random_f32(rows * cols, 1)
    x = (oracle.round_f16(x) if dtype == "f16" else x).reshape(rows, cols)
    got = rt.toArray(rt.softmax(ex.upload(x, [rows, cols], dtype)), ex)
    close(got, oracle.softmax_ref(x), dtype)


@pytest.mark.parametrize("x,want", [
    ([1, 2, 3], [0.09003057, 0.24472847, 0.66524096]),
    ([1001, 1002, 1003, -1000], [0.09003057, 0.24472847, 0.66524096, 0]),
])
def test_softmax_matches_torch_known_answers(ex, x, want):
    import runntime_b200 as rt
    got = rt.toArray(rt.softmax(ex.upload(np.array(x, np.float32), [1, len(x)])), ex)
    assert np.all(np.abs(got - want) <= 1e-7 + 1e-6 * np.abs(want))


MASKS = [(INF, INF), (INF, 0), (2, 1), (0, 0)]


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("n", [12, 9, 136, 1000])
@pytest.mark.parametrize("wl,wr", MASKS)
def test_masked_softmax(ex, dtype, n, wl, wr):
    import runntime_b200 as rt
    half = n // 2
    x = 8 * oracle.random_f32(n * n, 2)
    x = (oracle.round_f16(x) if dtype == "f16" else x).reshape(n, n)
    segs = np.array([[0, half] if r < half else [half, n] for r in range(n)], np.float32)
    got = rt.toArray(rt.softmax(ex.upload(x, [n, n], dtype),
                                dict(segments=ex.upload(segs, [n, 2]), windowLeft=wl,
                                     windowRight=wr)), ex)
    close(got, oracle.softmax_ref(x, segs, wl, wr), dtype)


def test_a_row_that_keeps_nothing_is_zero(ex):
    import runntime_b200 as rt
    n = 8
    x = oracle.random_f32(n * n, 3).reshape(n, n)
    segs = np.array([[0, n]] * n, np.float32)
    segs[3] = (5, 5)       # empty range
    segs[6] = (0, 2)       # range that the causal window never reaches... it does: keeps 0, 1
    got = rt.toArray(rt.softmax(ex.upload(x, [n, n]), dict(segments=ex.upload(segs, [n, 2]),
                                                          windowLeft=1, windowRight=0)), ex)
    got = got.reshape(n, n)
    assert (got[3] == 0).all() and (got[6] == 0).all()   # row 6 sees keys 5..6, range is [0, 2)
    assert abs(got[2].sum() - 1) < 1e-6


def test_softmax_runs_past_2p24_elements(ex):
    import runntime_b200 as rt
    rows, cols = 4100, 4096
    x = oracle.random_f32(rows * cols, 3).reshape(rows, cols)
    got = rt.toArray(rt.softmax(ex.upload(x, [rows, cols])), ex)
    close(got, oracle.softmax_ref(x), "f32")


def test_matmul_attention_path_agrees_with_the_fused_op(ex):
    """softmax(q k^T) v with the masked softmax equals sdpaPacked's answer: the
    equivalence the reference keeps both paths for
    (packages/runntime/src/core/kernels/reduce/softmax.ts:128-133)."""
    import runntime_b200 as rt
    t, heads, hd = 96, 1, 32
    q = oracle.random_f32(t * hd, 1).reshape(t, hd) * hd ** -0.5 * 2
    k = oracle.random_f32(t * hd, 2).reshape(t, hd)
    v = oracle.random_f32(t * hd, 3).reshape(t, hd)
    segs = np.array([[0, 40]] * 40 + [[40, 96]] * 56, np.float32)
    scores = (q.astype(np.float64) @ k.astype(np.float64).T).astype(np.float32)
    S = ex.upload(segs, [t, 2])
    probs = rt.toArray(rt.softmax(ex.upload(scores, [t, t]),
                                  dict(segments=S, windowLeft=8, windowRight=8)), ex).reshape(t, t)
    viaMatmul = probs.astype(np.float64) @ v.astype(np.float64)
    fused = rt.toArray(rt.sdpa(ex.upload(q, [t, hd]), ex.upload(k, [t, hd]), ex.upload(v, [t, hd]),
                               dict(qHeads=heads, kvHeads=heads, headDim=hd, windowLeft=8,
                                    windowRight=8, segments=S)), ex).reshape(t, hd)
    assert np.all(np.abs(fused - viaMatmul) <= 2e-5 + 1e-4 * np.abs(viaMatmul))


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("shift,outShift", [(0, 0), (3, 3), (1, 5), (4, 0), (2, 1)])
@pytest.mark.parametrize("rows,cols", [(2, 5), (5, 33), (3, 2051), (2050, 67), (2049, 2307)])
def test_rows_that_start_anywhere(ex, dtype, shift, outShift, rows, cols):
    """x and out `shift` elements into an allocation: chunks of 16 bytes, 8 bytes or one
    element, ragged ends on either side; nothing outside the rows is written."""
    import ctypes as C
    import torch
    from runntime_b200._lib import DTYPE_CODE, check
    td = torch.float16 if dtype == "f16" else torch.float32
    x = 8 * oracle.random_f32(rows * cols, 4)
    x = oracle.round_f16(x) if dtype == "f16" else x
    src = torch.zeros(rows * cols + 16, dtype=td, device="cuda")
    src[shift:shift + rows * cols] = torch.from_numpy(x).to("cuda", td)
    out = torch.full((rows * cols + 16,), 7.0, dtype=td, device="cuda")
    torch.cuda.synchronize()
    es = src.element_size()
    check(ex._lib.rt_softmax(ex.ctx, C.c_void_p(src.data_ptr() + shift * es),
                             C.c_void_p(out.data_ptr() + outShift * es), None, rows, cols, 0, 0,
                             DTYPE_CODE[dtype]), ex.ctx)
    ex.sync()
    got = out.float().cpu().numpy()
    close(got[outShift:outShift + rows * cols], oracle.softmax_ref(x.reshape(rows, cols)), dtype)
    assert (got[:outShift] == 7).all() and (got[outShift + rows * cols:] == 7).all()


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("wl,wr", [(INF, INF), (1100, 3), (0, 0)])
@pytest.mark.parametrize("n,shift,outShift", [(2049, 0, 0), (2051, 3, 3), (2051, 4, 0), (2051, 2, 1), (2052, 0, 0)])
def test_masked_rows_of_a_block(ex, dtype, n, shift, outShift, wl, wr):
    """Rows of more than 2048 columns: kept ranges of up to 1024 columns belong to one warp of the
    block, longer ones to all of it, and all of it stores the zeros.  Ranges of no, one, 1024 and
    1025 columns that begin or end in the row's first or last 16 bytes or beside them; nothing of
    what the output held is left, and nothing around it is written."""
    import ctypes as C
    import torch
    from runntime_b200._lib import DTYPE_CODE, WINDOW_INF, check
    ends = [(0, 0), (5, 5), (n, n), (0, 1), (n - 1, n), (n // 2, n // 2 + 1)]
    for kept in (1023, 1024, 1025, n - 1, n):
        ends += [(at, at + kept) for at in (0, 1, 3, 7, 8, n - kept - 9, n - kept - 8, n - kept - 1, n - kept)
                 if at >= 0 and at + kept <= n]
    segs = np.array([ends[r % len(ends)] for r in range(n)], np.float32)
    td = torch.float16 if dtype == "f16" else torch.float32
    x = 8 * oracle.random_f32(n * n, 7)
    x = oracle.round_f16(x) if dtype == "f16" else x
    src = torch.zeros(n * n + 16, dtype=td, device="cuda")
    src[shift:shift + n * n] = torch.from_numpy(x).to("cuda", td)
    out = torch.full((n * n + 16,), 7.0, dtype=td, device="cuda")
    dev = torch.from_numpy(segs).cuda()
    torch.cuda.synchronize()
    es = src.element_size()
    check(ex._lib.rt_softmax(ex.ctx, C.c_void_p(src.data_ptr() + shift * es),
                             C.c_void_p(out.data_ptr() + outShift * es), C.c_void_p(dev.data_ptr()), n, n,
                             *(WINDOW_INF if w == INF else w for w in (wl, wr)), DTYPE_CODE[dtype]), ex.ctx)
    ex.sync()
    got = out.float().cpu().numpy()
    close(got[outShift:outShift + n * n], oracle.softmax_ref(x.reshape(n, n), segs, wl, wr), dtype)
    assert (got[:outShift] == 7).all() and (got[outShift + n * n:] == 7).all()


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("n", [511, 767, 769, 2047])
@pytest.mark.parametrize("parts", [1, 2, 3])
def test_masked_rows_of_a_warp(ex, dtype, n, parts):
    """Rows that start anywhere, on either side of the width up to which they go element by element."""
    import runntime_b200 as rt
    x = 8 * oracle.random_f32(n * n, 5)
    x = (oracle.round_f16(x) if dtype == "f16" else x).reshape(n, n)
    at = [n * p // parts for p in range(parts + 1)]
    segs = np.array([[at[r * parts // n], at[r * parts // n + 1]] for r in range(n)], np.float32)
    segs[3], segs[4], segs[5] = (0, n // 2), (n // 2 - 1, n), (n, n)
    got = rt.toArray(rt.softmax(ex.upload(x, [n, n], dtype), dict(segments=ex.upload(segs, [n, 2]))), ex)
    close(got, oracle.softmax_ref(x, segs), dtype)


@pytest.mark.parametrize("n,shift", [(5001, 0), (5003, 3), (5002, 4)])
def test_long_half_precision_rows_in_groups(ex, n, shift):
    """Four rows to a block: all narrow (a warp each), all wide, one wide among narrow ones, rows
    that keep nothing, ranges at either end; the rows that have a block of their own; what the
    output held is overwritten and nothing around it."""
    import ctypes as C
    import torch
    from runntime_b200._lib import WINDOW_INF, check
    g = torch.Generator(device="cuda").manual_seed(n)
    src = torch.empty(n * n + 16, device="cuda").normal_(0, 3, generator=g).half()
    out = torch.full((n * n + 16,), 7.0, device="cuda", dtype=torch.float16)
    x = src[shift:shift + n * n].view(n, n)
    kinds = [[(0, 40), (9, 1033), (n - 1024, n), (n - 1, n)], [(0, n), (1, n), (0, n - 1), (3, 1028)],
             [(5, 60), (0, 1025), (7, 7), (0, 0)], [(n, n), (0, 0), (4, 4), (1, 1)],
             [(8, 1032), (n - 1033, n - 9), (0, 1024), (2, 3)]]
    segs = [kinds[(r // 4) % len(kinds)][r % 4] for r in range(n)]
    dev = torch.tensor(segs, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    check(ex._lib.rt_softmax(ex.ctx, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr() + 2 * shift),
                             C.c_void_p(dev.data_ptr()), n, n, WINDOW_INF, WINDOW_INF, 1), ex.ctx)
    ex.sync()
    at = torch.arange(n, device="cuda")
    lo, hi = dev[:, :1].long(), dev[:, 1:].long()
    keep = (at[None] >= lo) & (at[None] < hi)
    want = torch.softmax(x.double().masked_fill(~keep, -math.inf), 1).nan_to_num(0.0) if n else None
    got = out[shift:shift + n * n].view(n, n).double()
    # one rounding to f16, and exponentials of approximate scores (2^-21 of the value)
    assert ((got - want).abs() <= want * 2.0 ** -10 + 2.0 ** -24).all()
    assert (got[~keep] == 0).all()
    assert (out[:shift] == 7).all() and (out[shift + n * n:] == 7).all()
