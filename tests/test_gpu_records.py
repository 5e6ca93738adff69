"""Records of the kept boxes formed at the end: models of one to thirty-two parts, two
models of different part counts in one call, few and thousands of kept boxes.  Against the
oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

from geye_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [(1, 8), (5, 3), (13, 1), (32, 7)])
@pytest.mark.parametrize("overlap", [0.5, 0.96])
def test_part_counts(tmp_path, parts, overlap):
    import geye_gb300 as g
    specs = [dataclasses.replace(s, name=f"{s.name}{n}", parts_per_component=n)
             for s, n in zip((synth.CAR_SPEC, synth.PERSON_SPEC), parts)]
    paths = [synth.write_model_csv(s, str(tmp_path)) for s in specs]
    frame = synth.make_frame(331, 253, seed=sum(parts))
    with g.Context(0) as c:
        ms = [g.Model(c, *p) for p in paths]
        runs = [c.detect_multi(frame, ms, -0.5, overlap) for _ in range(2)]
        for m in ms:
            m.close()
    for k, p in enumerate(paths):
        want = O.car_detection(O.Model(*p), frame, -0.5, overlap)
        for got in (r[k] for r in runs):
            assert got["num"] == want["K"] > 0
            for f in ("point", "or_point", "type"):
                assert np.array_equal(got[f], want[f]), f
            for f in ("score",):
                assert np.array_equal(got[f].view(np.int32), want[f].view(np.int32)), f
