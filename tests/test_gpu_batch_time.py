"""A batch's last_ms holds the frames' uploads: what a call takes beyond it is less than the uploads alone."""
import time

import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu


def test_last_ms_holds_the_uploads(tmp_path):
    import geye_gb300 as g
    import torch
    frames = [synth.make_frame(1920, 1080, seed=s) for s in range(2)] * 4
    dev = [torch.empty(f.shape, dtype=torch.uint8, device="cuda") for f in frames]

    def upload():
        torch.cuda.synchronize()
        t = time.perf_counter()
        for d, f in zip(dev, frames):
            d.copy_(torch.from_numpy(f))
        torch.cuda.synchronize()
        return 1000.0 * (time.perf_counter() - t)

    with g.Context(0, conv=g.CONV_BF16) as c:
        m = g.Model(c, *synth.write_model_csv(synth.CAR_SPEC, str(tmp_path)))
        b = g.Batch([m], conv=g.CONV_BF16, max_frames=len(frames))

        def beyond():
            t = time.perf_counter()
            b.run(frames, 5.0, 0.5)   # (nothing detected: next to nothing to read back)
            return 1000.0 * (time.perf_counter() - t) - b.stats()["last_ms"]

        for _ in range(3):
            upload()
            beyond()
        up, rest = (np.median([f() for _ in range(9)]) for f in (upload, beyond))
        b.close()
        m.close()
    assert rest < up, (rest, up)
