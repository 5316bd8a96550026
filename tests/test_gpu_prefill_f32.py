"""f32 prefill on the tensor cores and on the FP32 pipes: edges of the 16-row, 16-key, 32-row
and 64-key tiles, head sizes around the 16- and 32-column blocks, padded batches whose
sequences do not end on a tile, against the f64 oracle at the suite's f32 tolerance; and
inputs that are not finite."""
import numpy as np
import pytest

import cases
import oracle
from gpu_harness import check_sdpa, ex, run_sdpa  # noqa: F401
from oracle import SdpaCase, make_inputs

pytestmark = pytest.mark.gpu
OPT_PREFILL_TC = 1
ROUTES = [(1, "prefill_f32_tc"), (0, "prefill_simt")]


@pytest.fixture(params=ROUTES, ids=[r for _, r in ROUTES])
def route(request, ex):
    ex.setOption(OPT_PREFILL_TC, request.param[0])
    yield request.param[1]
    ex.setOption(OPT_PREFILL_TC, 1)


@pytest.mark.parametrize("hd", [4, 16, 20, 32, 36, 52, 64, 100, 128, 132, 200, 256])
@pytest.mark.parametrize("t", [2, 15, 33, 63, 65, 130, 257])
def test_head_sizes_and_tile_edges(ex, route, hd, t):
    check_sdpa(ex, SdpaCase(qLen=t, kvLen=t, qHeads=2, kvHeads=1, headDim=hd, windowRight=0), "f32", route)
    check_sdpa(ex, SdpaCase(qLen=t, kvLen=t, qHeads=2, kvHeads=2, headDim=hd, windowLeft=20, windowRight=3),
               "f32", route)


@pytest.mark.parametrize("hd", [32, 52, 128, 256])
def test_every_option(ex, route, hd):
    for name, c in cases.option_cases(150, hd):
        if not (c.packed and hd > 128):
            check_sdpa(ex, c, "f32", route)


@pytest.mark.parametrize("seq", [17, 40, 64, 100])
@pytest.mark.parametrize("hd", [52, 256])
def test_padded_batches(ex, route, hd, seq):
    """Rows past a sequence's length hold NaN: nothing may read them into a live row."""
    import torch
    from runntime_b200.engine import prefill_batched
    lens = [seq, 1, seq // 2, seq - 1]
    g = torch.Generator().manual_seed(seq * hd)
    q, k, v = (torch.randn(len(lens) * seq, hd, generator=g) * s for s in (hd ** -0.5, 1.0, 1.0))
    want = torch.zeros(len(lens) * seq, hd, dtype=torch.float64)
    for b, n in enumerate(lens):
        r = slice(b * seq, b * seq + n)
        want[r] = torch.softmax(q[r].double() @ k[r].double().T, -1) @ v[r].double()
        for x in (q, k, v):
            x[b * seq + n:(b + 1) * seq] = float("nan")
    dev = [x.cuda() for x in (q, k, v)]
    out = torch.empty_like(dev[0])
    torch.cuda.synchronize()
    prefill_batched(ex, *dev, out, dtype="f32", batch=len(lens), seqStride=seq,
                    seqLens=torch.tensor(lens, dtype=torch.int32, device="cuda"), qHeads=1, kvHeads=1,
                    headDim=hd)
    ex.sync()
    oracle.assert_close(out.cpu().numpy().reshape(-1), want.numpy().reshape(-1), "f32", f"batch {seq} {hd}")


@pytest.mark.parametrize("value", [np.inf, -np.inf, 3.4e38])
def test_values_past_the_split(ex, route, value):
    """A value the 11-bit parts cannot hold: rows that see its key get what f32 products give
    (the value itself carries into the sum), rows before it are untouched."""
    c = SdpaCase(qLen=90, kvLen=90, qHeads=1, kvHeads=1, headDim=32, windowRight=0)
    x = make_inputs(c, "f32")
    x.v.reshape(90, 32)[40, 5] = value
    got = run_sdpa(ex, x).reshape(90, 32)
    assert ex.dispatches[-1] == route
    with np.errstate(all="ignore"):
        want = oracle.sdpa_ref_inputs(x).reshape(90, 32)
    finite = np.isfinite(want) & (np.abs(want) < 1e30)
    assert np.isfinite(got[finite]).all()
    oracle.assert_close(got[finite], want[finite], "f32", "finite part")
    seen = got[40:, 5]
    assert (np.sign(seen) == np.sign(value)).all() and (np.abs(seen) > 1e30).all()


def scores_ref(q, k, v):
    """Causal attention of one head in f64: a score of -inf weighs nothing, a row with one of
    +inf or NaN is NaN."""
    import torch
    q, k, v = (torch.from_numpy(x).double() for x in (q, k, v))
    return torch.stack([torch.softmax(k[:i + 1] @ q[i], 0) @ v[:i + 1] for i in range(len(q))]).numpy()


def check_marked(ex, route, hd, where, value):
    """Column 5 of row 40 of q, k or v is `value`: the rows that see it are what the op's
    definition gives, NaN where it is NaN; the others have nothing to do with it."""
    import runntime_b200 as rt
    rng = np.random.default_rng(hd)
    x = {c: rng.standard_normal((90, hd)).astype(np.float32) * s for c, s in zip("qkv", (0.3, 0.3, 1))}
    x[where][40, 5] = value
    with np.errstate(all="ignore"):
        want = scores_ref(x["q"], x["k"], x["v"])
    got = rt.toArray(rt.sdpa(*(ex.upload(x[c], [90, hd]) for c in "qkv"),
                             dict(qHeads=1, kvHeads=1, headDim=hd, windowLeft=np.inf, windowRight=0)), ex)
    assert ex.dispatches[-1] == route
    got = got.reshape(90, hd)
    assert (np.isnan(got) == np.isnan(want)).all()
    finite = np.isfinite(want)
    assert not finite.all() or (where == "k" and value == -np.inf)
    oracle.assert_close(got[finite], want[finite], "f32", f"{where} {value}")


@pytest.mark.parametrize("hd", [32, 52, 128, 256])
@pytest.mark.parametrize("where", ["q", "k"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_scores_that_are_not_finite(ex, route, hd, where, value):
    check_marked(ex, route, hd, where, value)


@pytest.mark.parametrize("hd", [32, 256])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("bits", [0x7fffffff, 0xffffffff, 0x7f800001])
def test_every_nan_stays_one(ex, route, hd, where, bits):
    """0x7fffffff is the NaN that GPU arithmetic makes."""
    check_marked(ex, route, hd, where, np.uint32(bits).view(np.float32))
