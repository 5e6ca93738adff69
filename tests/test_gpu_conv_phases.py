"""Tensor-core convolution in column phases: every tile shape of the autotuner on frames
whose slabs need none, some and every filter column a phase, part filters of one size and
of many.  Every tile's products are added in the same order, so all shapes that fit
give the same detections, bit for bit."""
import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [0, 7] + list(range(11, 15))   # the stage ring as a reference, then the phased shapes


@pytest.mark.parametrize("mode", ["bf16", "fp8"])
@pytest.mark.parametrize("specs", [(synth.CAR_SPEC, synth.PERSON_SPEC), (synth.CAR_TRAINED_LIKE, synth.PERSON_TRAINED_LIKE)])
@pytest.mark.parametrize("w,h", [(240, 180), (641, 479), (1280, 720)])
def test_shapes_agree(tmp_path, monkeypatch, mode, specs, w, h):
    import geye_gb300 as g
    conv = {"bf16": g.CONV_BF16, "fp8": g.CONV_FP8}[mode]
    thresh = -0.5 if specs[0] is synth.CAR_SPEC else -2.9
    paths = [synth.write_model_csv(s, str(tmp_path)) for s in specs]
    frame = synth.make_frame(w, h, seed=w)
    first = None
    for shape in SHAPES:
        monkeypatch.setenv("GEYE_TC_SHAPE", str(shape))
        with g.Context(0, conv=conv) as c:
            ms = [g.Model(c, *p) for p in paths]
            got = c.detect_multi(frame, ms, thresh, 0.5)
            for m in ms:
                m.close()
        first = first or got
        for a, b in zip(first, got):
            assert a["num"] == b["num"], shape
            for k in ("point", "or_point", "type"):
                assert np.array_equal(a[k], b[k]), (shape, k)
            for k in ("score", "scale"):
                assert np.array_equal(a[k].view(np.int32), b[k].view(np.int32)), (shape, k)
