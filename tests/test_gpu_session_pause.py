"""A session that is resumed and paused again at once ends up paused, each time."""

import time

import pytest

from minirender_b200 import scene as sc

pytestmark = pytest.mark.gpu


def test_resume_then_pause_at_once_pauses():
    from minirender_b200 import api
    scene = api.Scene(sc.cornell_box().snapshot())
    session = api.RenderSession()
    session.start(scene, api.RenderSettings(64, 64, 1_000_000, 3), api.IntegratorSettings(),
                  api.SessionSettings(0, 16, 1))

    def wait_for(state):
        deadline = time.time() + 5
        while session.progress()["state"] != state and time.time() < deadline:
            time.sleep(0.001)
        assert session.progress()["state"] == state

    wait_for("running")
    assert session.pause()
    wait_for("paused")
    for _ in range(200):
        assert session.resume()
        assert session.pause()
        wait_for("paused")
    session.cancel()
    session.wait()
    assert session.progress()["state"] == "cancelled"
    session.close()
