"""A server's submit that returns an error of a frame before it has queued its own frame: the ticket it
handed out is of a frame that waits."""
import ctypes as C

import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu


def test_the_frame_of_a_failed_submit_waits_in_the_queue(tmp_path):
    import geye_gb300 as g
    wide = np.zeros((96, 4608, 3), np.uint8)   # part maps of more columns than the DT takes: its plan fails at every attempt
    frame = synth.make_frame(320, 240, seed=1)
    with g.Context(0) as c:
        m = g.Model(c, *synth.write_model_csv(synth.CAR_SPEC, str(tmp_path)))
        with g.Server([m], conv=g.CONV_FP32, max_slots=2) as srv:
            tickets = []
            for k, f in enumerate((wide, frame, frame)):
                t = C.c_longlong(-1)
                h, w, _ = f.shape
                assert g.lib().geye_server_submit(srv.h, 0, f.ctypes.data, w, h, 3 * w, C.byref(t)) != 0
                tickets.append(t.value)
                assert srv.stats()["queued"] == k + 1
            # the head's age lets it go, and the frames behind it with it, each once
            srv.set_admission(0, 1e-6)
            done = srv.poll(16)
            assert [d["ticket"] for d in done] == tickets and all(d["dropped"] for d in done)
            srv.set_admission(0, 0.0)
            srv.submit(0, frame)
            srv.drain()
            assert srv.poll(4)[0]["results"][0]["num"] > 0
        m.close()
