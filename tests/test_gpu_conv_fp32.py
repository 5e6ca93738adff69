"""FP32 convolution at the edges of its tiles and groups, bit for bit against the oracle:
groups of one to four filters, every unrolled column length and the general one, filters
wider than a stage, maps of one position up to several tiles, and a call with so many
tiles that the warps take whole ones."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import geye_gb300 as g
    with g.Context(0) as c:
        yield c


def _check(ctx, rng, a0, a1, shapes):
    feat = (rng.random((31, a1, a0)) * 0.4).astype(np.float32)
    filters = [rng.normal(0, 0.02, size=(31, b1, b0)).astype(np.float32) for b0, b1 in shapes]
    for got, f in zip(ctx.fconvsMT(feat, filters), filters):
        assert np.array_equal(got.view(np.int32), O.fconv(feat, f).view(np.int32)), f.shape


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("b0", [1, 3, 4, 5, 6, 7, 8, 9, 10, 11, 14])
def test_groups_and_column_lengths(ctx, n, b0):
    _check(ctx, np.random.default_rng(100 * n + b0), b0 + 33, 21, [(b0, 4)] * n)


@pytest.mark.parametrize("a0,a1,b0,b1", [(6, 6, 6, 6), (7, 6, 6, 6), (5, 40, 5, 17), (9, 70, 3, 33), (65, 9, 2, 1),
                                         (130, 19, 6, 6), (260, 8, 100, 3), (47, 66, 13, 40), (64, 64, 40, 40)])
def test_map_and_filter_edges(ctx, a0, a1, b0, b1):
    rng = np.random.default_rng(a0 * 1000 + a1)
    _check(ctx, rng, a0, a1, [(b0, b1)] * 3 + [(max(b0 // 2, 1), b1)])


def test_many_tiles(ctx):
    _check(ctx, np.random.default_rng(5), 181, 243, [(4, 3)] * 60 + [(6, 4)] * 43 + [(9, 2)] * 3 + [(5, 5)] * 2)
