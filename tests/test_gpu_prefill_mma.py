"""Packed short segments with narrow heads (f16): edges of the 64-row and 64-key tiles and of a
warp's 16 rows, segments that straddle tiles, rows that see nothing, every mask, 16- and 8-byte
rows, against the f64 oracle at the suite's f16 tolerance."""
import numpy as np
import pytest

import oracle
from gpu_harness import ex, run_sdpa  # noqa: F401
from oracle import SdpaCase, make_inputs

pytestmark = pytest.mark.gpu
LENS = [37, 200, 5, 130, 1, 64, 63, 65, 16, 128]


def check(ex, lens, route="prefill_mma", pad=0, **kw):
    T = sum(lens) + pad
    c = SdpaCase(qLen=T, kvLen=T, segments=True, maxSegment=max(lens), **kw)
    x = make_inputs(c, "f16")
    segs = np.zeros((T, 2), np.float32)      # (the padding rows keep nothing)
    at = 0
    for n in lens:
        segs[at:at + n] = (at, at + n)
        at += n
    x.segs = segs
    got = run_sdpa(ex, x)
    assert ex.dispatches[-1] == route
    oracle.assert_close(got, oracle.sdpa_ref_inputs(x), "f16", str(c))


@pytest.mark.parametrize("hd", [4, 8, 16, 20, 28, 32])
@pytest.mark.parametrize("packed", [False, True])
def test_head_sizes(ex, hd, packed):
    check(ex, LENS, pad=70, qHeads=4, kvHeads=2, headDim=hd, packed=packed)


@pytest.mark.parametrize("opts", [dict(windowRight=0), dict(windowLeft=3, windowRight=0),
                                  dict(windowLeft=40, windowRight=7), dict(sinks=True), dict(keyBias=True),
                                  dict(sinks=True, keyBias=True, windowRight=0), dict(windowLeft=0, windowRight=0)])
def test_masks(ex, opts):
    check(ex, LENS, qHeads=3, kvHeads=1, headDim=32, **opts)


@pytest.mark.parametrize("lens", [[2], [15, 1], [17], [64], [65], [256], [512] * 10 + [1], [1] * 130])
def test_tile_edges(ex, lens):
    check(ex, lens, qHeads=3, kvHeads=3, headDim=32)


def test_other_calls_stay_where_they_were(ex):
    check(ex, [513, 20], "prefill_tc3", qHeads=2, kvHeads=2, headDim=32)
    check(ex, [300, 20], "prefill_tc3", qHeads=2, kvHeads=2, headDim=32)    # too few blocks for 300 keys
    check(ex, [100, 20], "prefill_tc3", qHeads=2, kvHeads=2, headDim=36)
    check(ex, [100, 20], "prefill_simt", qHeads=2, kvHeads=2, headDim=30)
