"""detect_submit on a caller's stream returns while the caller's earlier work on that stream is still
running, and leaves the caller's frame buffer free."""
import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu


def test_submit_does_not_wait_for_the_callers_work(tmp_path):
    import geye_gb300 as g
    import torch
    frames = [synth.make_frame(320, 240, seed=s) for s in (1, 2)]
    s = torch.cuda.Stream()
    with g.Context(0, stream=s.cuda_stream) as c:
        m = g.Model(c, *synth.write_model_csv(synth.CAR_SPEC, str(tmp_path)))
        want = [c.detect_multi(f, [m], -0.5, 0.5)[0] for f in frames]
        for pinned in (False, True):
            buf = torch.from_numpy(frames[0].copy())
            if pinned:
                buf = buf.pin_memory()
            with torch.cuda.stream(s):
                torch.cuda._sleep(1 << 30)   # about half a second of the caller's own work
                busy = torch.cuda.Event()
                busy.record()
            c.detect_submit(buf.numpy(), [m], -0.5, 0.5)
            assert not busy.query()          # it is still running
            buf.numpy()[:] = frames[1]       # the buffer is the caller's again
            got = c.detect_collect()[0]
            assert got["num"] == want[0]["num"] != 0
            assert np.array_equal(got["point"], want[0]["point"]) and np.array_equal(got["score"], want[0]["score"])
        m.close()
