"""The tiled tensor-core matmul where its tiles can go wrong: several tiles per block in each
tile width, ragged last rows, columns and K, a single partial tile, an addend that no TMA load
can take.  Against f64 sums of the same halves; the result is rounded to f16 (2^-11 of it) after
f32 accumulation (K 2^-24 of the absolute sum, far below)."""
import pytest

from gpu_harness import ex  # noqa: F401

pytestmark = pytest.mark.gpu

# (m, k, n): many 64-column tiles per block; 128-column; 256-column; one partial tile; the
# smallest; more tiles than blocks by one
SHAPES = [(8300, 64, 1000), (4100, 200, 1000), (4700, 1100, 4000), (17, 72, 64), (130, 64, 136),
          (149 * 128, 64, 64)]


def run(ex, m, k, n, act, bias, addend, shift=0):
    import torch
    import runntime_b200 as rt
    g = torch.Generator(device="cuda").manual_seed(m + k + n)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    a, b = rand(m, k).half(), (rand(k, n) * k ** -0.5).half()
    bv, flat = rand(n).half(), rand(m * n + shift).half()
    av = flat[shift:].view(m, n)
    torch.cuda.synchronize()
    wrap = lambda t, *s: ex.wrap(t.data_ptr(), s, "f16", keepalive=t)  # noqa: E731
    opts = {}
    want = a.double() @ b.double()
    if bias:
        opts["bias"] = wrap(bv, n)
        want = want + bv.double()
    if act == "gelu":
        opts["activation"] = "gelu"
        want = torch.nn.functional.gelu(want)
    if addend:
        opts["addend"] = wrap(av, m, n)
        want = want + av.double()
    y = rt.matmul(wrap(a, m, k), wrap(b, k, n), opts)
    got = torch.from_numpy(rt.toArray(y, ex)).cuda().double().view(m, n)
    ex.releaseValues([y])
    # one rounding of the result to f16, half an ulp; f32 accumulation of sums of magnitude
    # sqrt(K) <= 33: 33 * 2^-24 = 2e-6, four times that for the order and truncation of the adds
    bad = (got - want).abs() > 2.0 ** -11 * want.abs() + 8e-6
    assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} off by up to {float((got - want).abs().max())}"


@pytest.mark.parametrize("m,k,n", SHAPES)
@pytest.mark.parametrize("act,bias,addend", [(None, False, False), (None, True, True), ("gelu", True, False)])
def test_tiles(ex, m, k, n, act, bias, addend):
    run(ex, m, k, n, act, bias, addend)


@pytest.mark.parametrize("m,k,n", [(8300, 64, 1000), (130, 64, 136)])
def test_addend_off_a_16_byte_boundary(ex, m, k, n):
    run(ex, m, k, n, None, True, True, shift=1)


@pytest.mark.parametrize("act", [None, "tanh", "gelu", "silu", "relu", "geluTanh", "elu"])
def test_activations_do_not_depend_on_the_row_count(ex, act):
    """Sums at the ends of the range, infinite ones and NaN: 17 rows (this kernel) answer as 16 do
    (the cluster kernel, whole divisions).  Finite results may differ by one rounding to f16."""
    import numpy as np
    import runntime_b200 as rt
    ends = [np.inf, -np.inf, np.nan, 65504, -65504, 1e4, -1e4, 90, -90, 88, -88, 44, -44, 9, -9, 1, -1, 0, -0.0, 1e-7]
    bias = np.zeros(128, np.float32)
    bias[:len(ends)] = ends
    rows = []
    for m in (16, 17):
        opts = dict(bias=ex.upload(bias, [128], "f16"))
        if act:
            opts["activation"] = act
        y = rt.matmul(ex.upload(np.zeros((m, 64)), [m, 64], "f16"), ex.upload(np.zeros((64, 128)), [64, 128], "f16"),
                      opts)
        rows.append(rt.toArray(y, ex).reshape(m, 128))
    few, many = rows[0][0], rows[1][-1]
    assert (np.isnan(few) == np.isnan(many)).all(), (few, many)
    assert (few[np.isinf(few) | np.isinf(many)] == many[np.isinf(few) | np.isinf(many)]).all(), (few, many)
    assert act not in ("gelu", "geluTanh", "silu") or many[0] == np.inf
    finite = np.isfinite(few)
    # (below 2^-14 halves are 2^-24 apart)
    few, many = few[finite], many[finite]
    assert (np.abs(few - many) <= 2.0 ** -10 * np.abs(few) + 2.0 ** -24).all(), (few, many)
