"""fconvsMT with one buffer of taps under several filter sizes: transposed dims, a prefix of a
larger filter, the same filter twice.  Against a copy of each filter on its own and against the
oracle, bit for bit in FP32."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _views(buf, dims):
    """Filters [31][b1][b0] that start at the same address."""
    return [buf[:31 * b1 * b0].reshape(31, b1, b0) for b1, b0 in dims]


# (b1, b0) of the filters: transposed dims, the later bank shorter and longer, a prefix, four groups of one buffer
@pytest.mark.parametrize("dims", [[(8, 3), (3, 8)], [(9, 4), (4, 9)], [(6, 6), (5, 3)], [(6, 6), (6, 6)],
                                  [(12, 3), (3, 12), (4, 9), (9, 4)]])
@pytest.mark.parametrize("conv", ["fp32", "bf16", "fp8"])
def test_one_buffer_under_several_sizes(dims, conv):
    import geye_gb300 as g
    rng = np.random.default_rng(len(dims))
    feat = rng.random((31, 37, 29), np.float32)
    buf = rng.normal(0.0, 0.05, 31 * max(a * b for a, b in dims)).astype(np.float32)
    views = _views(buf, dims)
    assert len({v.ctypes.data for v in views}) == 1
    with g.Context(0, conv={"fp32": g.CONV_FP32, "bf16": g.CONV_BF16, "fp8": g.CONV_FP8}[conv]) as c:
        got = c.fconvsMT(feat, views)
        want = c.fconvsMT(feat, [v.copy() for v in views])
    for k, v in enumerate(views):
        assert np.array_equal(got[k].view(np.int32), want[k].view(np.int32)), k
        if conv == "fp32":
            assert np.array_equal(got[k].view(np.int32), O.fconv(feat, v).view(np.int32)), k
