"""What a scene server takes of the GPU: its scenes are launched plainly from their
first update on, and the memory of its scenes together with what is kept of earlier
ones stays within its budget.
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


def test_memory_kept_of_earlier_scenes_counts_against_the_budget():
    # eight scenes one after the other, no two with a buffer of one size; 32 MB for what
    # the driver allocates beside the buffers (graphs, local memory)
    import torch
    from sphgpu import scenes
    from sphgpu.server import SceneServer
    sizes = [60000 + 20000 * k for k in range(8)]
    scs = [scenes.serving_dam_break(n, "IISPH", seed=n) for n in sizes]
    scenes.build_system(scs[-1]).close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    budget = 300 << 20
    with SceneServer(memory_budget_bytes=budget, max_active=1, chunk_steps=5) as srv:
        for sc in scs:
            r = srv.wait(srv.submit(sc, 5), 300)
            assert r["steps"] == 5 and r["device_bytes_reserved"] <= budget
            assert before - torch.cuda.mem_get_info()[0] <= budget + (32 << 20), sc.position.shape


@pytest.mark.parametrize("solver,precision", [("SESPH", "f32"), ("SESPHwSplitting", "f32"), ("SESPHwSplitting", "f64"),
                                              ("IISPH", "f32"), ("IISPH", "f64")])
def test_the_reservation_covers_a_scene(solver, precision):
    from sphgpu import scenes
    from sphgpu.server import SceneServer
    sc = scenes.serving_dam_break(40000, "IISPH" if solver == "IISPH" else "SESPH", seed=1)
    sc.procedures = dict(sc.procedures, pressure_solver=solver)
    with SceneServer(chunk_steps=5) as srv:
        r = srv.wait(srv.submit(sc, 5, precision=precision), 300)
    with scenes.build_system(sc, precision=precision) as g:
        g.set_step_graphs(5)
        g.step_forward_in_time(5)
        assert g.device_bytes() * 1.125 <= r["device_bytes_reserved"]  # (rounded up to the pool's size classes)
