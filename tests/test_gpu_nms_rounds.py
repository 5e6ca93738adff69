"""Pipeline NMS where its chunks, batches and pick groups end: thresholds that let from a few
boxes to all of them through, overlaps on both sides of a half (few and thousands of kept
boxes), frames whose equal scores run longer than a batch and than a chunk.  The kept
records against the oracle's, bit for bit."""
import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def paths(tmp_path_factory):
    return synth.write_model_csv(synth.CAR_SPEC, str(tmp_path_factory.mktemp("nms_rounds")))


@pytest.fixture(scope="module")
def ctx():
    import geye_gb300 as g
    with g.Context(0) as c:
        yield c


def _check(ctx, paths, frame, thresh, overlap):
    import geye_gb300 as g
    gm = g.Model(ctx, *paths)
    for _ in range(2):   # (the second one through the captured graph again)
        got = ctx.car_detection(frame, gm, thresh, None, overlap)
    gm.close()
    want = O.car_detection(O.Model(*paths), frame, thresh, overlap)
    assert got["num"] == want["K"]
    for k in ("point", "or_point", "type"):
        assert np.array_equal(got[k], want[k]), k
    assert np.array_equal(got["score"].view(np.int32), want["score"].view(np.int32))
    return got["num"]


@pytest.mark.parametrize("overlap", [0.05, 0.3, 0.4999, 0.5, 0.7, 0.9])
@pytest.mark.parametrize("thresh", [0.62, 0.5, 0.3, -0.5])
def test_overlaps_and_counts(ctx, paths, overlap, thresh):
    _check(ctx, paths, synth.make_frame(331, 253, seed=5), thresh, overlap)


def test_thousands_kept(ctx, paths):
    assert _check(ctx, paths, synth.make_frame(400, 300, seed=2), -0.5, 0.97) > 1024


@pytest.mark.parametrize("overlap", [0.3, 0.5])
def test_runs_of_equal_scores(ctx, paths, overlap):
    frame = np.full((240, 320, 3), 90, np.uint8)
    _check(ctx, paths, frame, -0.5, overlap)   # every level one run
    frame[:, 160:] = synth.make_frame(160, 240, seed=1)
    _check(ctx, paths, frame, -0.5, overlap)
