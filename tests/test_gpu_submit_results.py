"""A submitted frame's results belong to it: other frames that run on the same context, of the same
size and models, before it is collected do not change them; more kept boxes than the pinned block
holds included."""
import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu

W, H = 560, 420


def _same(a, b):
    assert a["num"] == b["num"]
    for k in ("point", "or_point", "type", "scale", "score"):
        assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("overlap", [0.5, 0.99])   # (0.99: more than 2048 kept boxes)
@pytest.mark.parametrize("conv", ["fp32", "bf16"])
def test_frames_between_submit_and_collect(tmp_path, conv, overlap):
    import geye_gb300 as g
    import torch
    frames = [synth.make_frame(W, H, seed=s) for s in range(3)]
    with g.Context(0, conv={"fp32": g.CONV_FP32, "bf16": g.CONV_BF16}[conv]) as c:
        ms = [g.Model(c, *synth.write_model_csv(s, str(tmp_path))) for s in (synth.CAR_SPEC, synth.PERSON_SPEC)]
        want = [c.detect_multi(f, ms, -0.5, overlap) for f in frames]
        if overlap > 0.9:
            assert max(r["num"] for r in want[0]) > 2048
        dev = torch.from_numpy(frames[1]).cuda()
        torch.cuda.synchronize()
        for between in ("device", "multi", "both"):
            c.detect_submit(frames[0], ms, -0.5, overlap)
            if between != "multi":
                c.detect_device(dev.data_ptr(), W, H, ms, -0.5, overlap)
                for k in range(2):
                    _same(c.fetch_result(k), want[1][k])
            if between != "device":
                for got, w in zip(c.detect_multi(frames[2], ms, -0.5, overlap), want[2]):
                    _same(got, w)
            for got, w in zip(c.detect_collect(), want[0]):
                _same(got, w)
            # and the next frame of the context is its own again
            c.detect_submit(frames[1], ms, -0.5, overlap)
            for got, w in zip(c.detect_collect(), want[1]):
                _same(got, w)
        for m in ms:
            m.close()
