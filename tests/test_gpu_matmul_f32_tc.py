"""f32 matmul of more than 16 rows: edges of the 64 x 64 x 32 tiles, every epilogue at a ragged
shape, a weight that starts inside a taller one, shapes that stay on the FP32 pipes, and inputs that are
not finite."""
import numpy as np
import pytest

from gpu_harness import ex  # noqa: F401
from test_gpu_matmul import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [17, 63, 64, 65, 200])
@pytest.mark.parametrize("n", [4, 60, 64, 68, 132])
@pytest.mark.parametrize("k", [4, 28, 32, 36, 96, 388])
def test_tile_edges(ex, m, k, n):
    check(ex, m, k, n, "f32")
    check(ex, m, k, n, "f32", bias=True, addend=True, act="gelu")


@pytest.mark.parametrize("act", [None, "tanh", "gelu", "silu", "relu", "geluTanh", "elu"])
def test_epilogues(ex, act):
    check(ex, 77, 100, 92, "f32", bias=True, addend=True, act=act)
    check(ex, 77, 100, 92, "f32", act=act, baseRow=3, extra=8)


@pytest.mark.parametrize("k,n", [(33, 64), (64, 33), (7, 5)])
def test_shapes_of_the_fp32_pipes(ex, k, n):
    check(ex, 70, k, n, "f32", bias=True)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
def test_values_past_the_split(ex, value):
    """One element of a that the parts cannot hold: its row is what f32 products give, the
    other rows are untouched."""
    import runntime_b200 as rt
    rng = np.random.default_rng(5)
    a = rng.standard_normal((40, 64)).astype(np.float32)
    b = rng.standard_normal((64, 48)).astype(np.float32)
    b[7, :4] = 0.5
    a[9, 7] = value
    got = rt.toArray(rt.matmul(ex.upload(a, [40, 64]), ex.upload(b, [64, 48])), ex).reshape(40, 48)
    with np.errstate(all="ignore"):
        want = a.astype(np.float64) @ b.astype(np.float64)
    rest = np.arange(40) != 9
    assert np.allclose(got[rest], want[rest], rtol=1e-5, atol=1e-5)
    if np.isnan(value):
        assert np.isnan(got[9]).all()
    else:
        # the element times b decides: infinite, or 1.7e38 where b is a half
        with np.errstate(all="ignore"):
            w32 = want[9].astype(np.float32)
        big = np.abs(w32) > 1e30
        assert big.any() and (np.sign(got[9][big]) == np.sign(w32[big])).all()
        assert np.allclose(got[9][:4], w32[:4], rtol=1e-5)


@pytest.mark.parametrize("where", ["a", "b"])
@pytest.mark.parametrize("bits", [0x7fffffff, 0xffffffff, 0x7fc00000, 0x7f800001])
def test_every_nan_stays_one(ex, where, bits):
    """0x7fffffff is the NaN that GPU arithmetic makes: an earlier operator's NaN is the next
    projection's too."""
    import runntime_b200 as rt
    rng = np.random.default_rng(6)
    x = dict(a=rng.standard_normal((40, 64)).astype(np.float32), b=rng.standard_normal((64, 48)).astype(np.float32))
    want = x["a"].astype(np.float64) @ x["b"].astype(np.float64)
    x[where][9, 7] = np.uint32(bits).view(np.float32)
    got = rt.toArray(rt.matmul(ex.upload(x["a"], [40, 64]), ex.upload(x["b"], [64, 48])), ex).reshape(40, 48)
    hit = np.zeros((40, 48), bool)
    if where == "a":
        hit[9] = True
    else:
        hit[:, 7] = True
    assert np.isnan(got[hit]).all()
    assert np.allclose(got[~hit], want[~hit], rtol=1e-5, atol=1e-5)
