"""The tensor-core form of localAttention (f16, heads of 64 and 128) at the edges of its tiles:
64 rows per block, 16 per warp, 16 or 32 rows of halo.  Against the op in f64."""
import pytest

from gpu_harness import ex  # noqa: F401

pytestmark = pytest.mark.gpu


def want_of(qkv, rel, qScale, heads, hd, window, kScale, softcap):
    import torch
    n = qkv.shape[0]
    x = qkv.double().view(n, 3, heads, hd)
    q, k, v = x[:, 0] * qScale.double(), x[:, 1] * kScale, x[:, 2]
    r = rel.double().view(window, heads, hd)
    s = torch.full((n, heads, window), -torch.inf, dtype=torch.float64, device=qkv.device)
    for j in range(min(window, n)):
        s[j:, :, j] = softcap * torch.tanh((q[j:] * (k[:n - j] + r[j])).sum(-1) / softcap)
    p = torch.softmax(s, -1)
    out = torch.zeros(n, heads, hd, dtype=torch.float64, device=qkv.device)
    for j in range(min(window, n)):
        out[j:] += p[j:, :, j, None] * v[:n - j]
    return out.reshape(n, heads * hd)


def check(ex, rows, heads, hd, window, *, kScale=1.0, softcap=50.0, qs=None, rs=1.0):
    import torch
    import runntime_b200 as rt
    g = torch.Generator(device="cuda").manual_seed(rows * 64 + window)
    w = heads * hd
    qkv = torch.randn(rows, 3 * w, generator=g, device="cuda").half()
    rel = torch.randn(window, w, generator=g, device="cuda") * rs
    qScale = (torch.rand(hd, generator=g, device="cuda") + 0.1) * (hd ** -0.5 if qs is None else qs)
    torch.cuda.synchronize()
    wrap = lambda t, d: ex.wrap(t.data_ptr(), t.shape, d, keepalive=t)  # noqa: E731
    y = rt.localAttention(wrap(qkv, "f16"), wrap(rel, "f32"), wrap(qScale, "f32"),
                          dict(heads=heads, headDim=hd, window=window, kScale=kScale, softcap=softcap))
    got = torch.from_numpy(rt.toArray(y, ex)).cuda().double().view(rows, w)
    ex.releaseValues([y])
    want = want_of(qkv, rel, qScale, heads, hd, window, kScale, softcap)
    # the rounding to f16, half an ulp; scores in f32 products (22 bits, sums of hd of them) move
    # the probabilities by less than 1e-5, and so a sum of values of order one
    bad = (got - want).abs() > 2.0 ** -11 * want.abs() + 2e-5
    assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} off by up to {float((got - want).abs().max())}"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [1, 9, 12, 16, 17, 24, 32])
@pytest.mark.parametrize("rows", [1, 15, 64, 65, 333])
def test_edges(ex, rows, window, hd):
    check(ex, rows, 3, hd, window)


@pytest.mark.parametrize("window", [12, 32])
def test_operands_past_the_range_of_a_half(ex, window):
    """q * qScale near 2^20 and bias rows near 2^-20 and 2^20: neither fits a half as it is.
    A score is 2^20 times a key; its f32 product is off by 2^-22 of that, a score of order
    one when the soft cap of 2^24 leaves it as it is — so a cap that decides by sign instead."""
    check(ex, 200, 2, 128, window, softcap=4.0, qs=2.0 ** -20, rs=2.0 ** 20)
    check(ex, 200, 2, 128, window, softcap=4.0, qs=2.0 ** 16, rs=2.0 ** -20, kScale=2.0 ** -16)


@pytest.mark.parametrize("hd,window", [(64, 12), (128, 32)])
@pytest.mark.parametrize("apart", [6, 9, 12, 14])
def test_a_key_that_weighs_little(ex, hd, window, apart):
    """The row's own key outweighs the others by e^apart and has a value of zero: what is left is the
    others' weight times values near the top of the range."""
    import torch
    import runntime_b200 as rt
    rows, softcap = 100, 1e4
    g = torch.Generator(device="cuda").manual_seed(apart)
    qkv = torch.zeros(rows, 3 * hd, device="cuda")
    qkv[:, 0] = 1
    qkv[::2, 2 * hd:] = (torch.rand(rows // 2, hd, generator=g, device="cuda") + 0.5) * 3e4
    qkv = qkv.half()
    rel = torch.zeros(window, hd, device="cuda")
    rel[0, 0] = apart
    rel[2::2, 0] = torch.rand(window // 2 - 1, generator=g, device="cuda")
    qScale = torch.ones(hd, device="cuda")
    torch.cuda.synchronize()
    wrap = lambda t, d: ex.wrap(t.data_ptr(), t.shape, d, keepalive=t)  # noqa: E731
    y = rt.localAttention(wrap(qkv, "f16"), wrap(rel, "f32"), wrap(qScale, "f32"),
                          dict(heads=1, headDim=hd, window=window, kScale=1.0, softcap=softcap))
    got = torch.from_numpy(rt.toArray(y, ex)).cuda().double().view(rows, hd)[1::2]
    ex.releaseValues([y])
    want = want_of(qkv, rel, qScale, 1, hd, window, 1.0, softcap)[1::2]
    # half an ulp of the result, and 2^-17 of it: scores up to 14 in f32 are off by 2^-20, tanhf and
    # the exponential by a few 2^-24 of theirs (tanhf's argument times the cap: 2 ulp of the score)
    bad = (got - want).abs() > (2.0 ** -11 + 2.0 ** -17) * want.abs() + 2.0 ** -25
    assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} off, by up to {float(((got - want) / want).abs().max()):.2g} of the result"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("rows", [2, 8, 9])
def test_a_few_rows(ex, rows, hd):
    """Either side of the count from which the tensor cores take the call."""
    check(ex, rows, 5, hd, 12)
    check(ex, rows, 5, hd, 32)
