"""Every ticket of a server comes back once: frames dropped on their age at submit."""
import numpy as np
import pytest

from geye_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(tmp_path_factory):
    import geye_gb300 as g
    c = g.Context(0)
    m = g.Model(c, *synth.write_model_csv(synth.CAR_SPEC, str(tmp_path_factory.mktemp("admission"))))
    yield g, m
    m.close()
    c.close()


@pytest.mark.parametrize("max_queued", [0, 1])
def test_a_frame_dropped_on_its_age_is_reported_once(setup, max_queued):
    g, m = setup
    frame = synth.make_frame(320, 240, seed=1)
    with g.Server([m], conv=g.CONV_FP32, max_slots=2) as srv:
        first = srv.submit(0, frame)
        srv.drain()
        srv.set_admission(max_queued, 1e-6)   # a nanosecond: every frame is too old when its turn comes
        tickets = [srv.submit(k % 2, frame) for k in range(4)]
        srv.drain()
        done = srv.poll(64)
        assert sorted(d["ticket"] for d in done) == [first] + tickets
        assert [d["dropped"] for d in sorted(done, key=lambda d: d["ticket"])] == [False] + [True] * 4
        st = srv.stats()
        assert st["dropped"] == 4 and st["completed"] == 1 and st["queued"] == 0
        srv.set_admission(0, 0.0)             # without limits it serves again
        last = srv.submit(0, frame)
        srv.drain()
        done = srv.poll(8)
        assert [(d["ticket"], d["dropped"]) for d in done] == [(last, False)]
        assert done[0]["results"][0]["num"] > 0
