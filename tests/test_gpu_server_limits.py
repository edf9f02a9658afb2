"""What a scene server takes of the GPU: its scenes are launched plainly from their
first update on.
"""
import pytest

pytestmark = pytest.mark.gpu


def test_scenes_are_launched_plainly_from_the_first_update(monkeypatch):
    # the launches are those of a system with dependent launches (and with them the
    # solve in one launch) off
    from sphgpu import scenes
    from sphgpu.server import SceneServer
    sc = scenes.serving_dam_break(8000, "IISPH", seed=2)
    steps, chunk = 20, 5
    with SceneServer(chunk_steps=chunk) as srv:
        r = srv.wait(srv.submit(sc, steps), 300)
    assert r["steps"] == steps and r["graph_replays"] == 0
    monkeypatch.setenv("SPHGPU_DEPENDENT_LAUNCH", "0")
    with scenes.build_system(sc) as g:
        g.set_step_graphs(chunk)
        g.step_forward_in_time(steps)
        g.take_measurement()
        assert g.launch_count() == r["kernel_launches"]
