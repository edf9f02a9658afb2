"""The cooperative solve at its limits: which launches a step makes, a launch that
ends before the solve does, a barrier whose wait runs out, and two solves at once
whose blocks each fill the GPU.

SPHGPU_BARRIER_POLLS and SPHGPU_SOLVE_SWEEPS lower the looks of a waiting block and
the sweeps of one launch; they are read once a system is initialized and again when
it restarts from a checkpoint.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(n, cap, tde):
    from sphgpu import scenes
    sc = scenes.serving_dam_break(n, solver="IISPH")
    sc.parameters = dict(sc.parameters, max_solver_iterations=cap, target_density_error=tde)
    return sc


def _state(g):
    from sphgpu import _capi as A
    return [g.download(f) for f in (A.FIELD_POSITION, A.FIELD_VELOCITY, A.FIELD_PRESSURE, A.FIELD_ACCELERATION)]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _step(g):
    """Launches and sweeps of one step."""
    before = g.launch_count()
    g.step_forward_in_time(1)
    return g.launch_count() - before, g.step_stats()["solver_iterations"]


@pytest.mark.parametrize("n,at_once", [(5000, True), (130000, True), (160000, False)])
def test_launches_of_a_step(n, at_once):
    # a solve in one launch takes the same launches whatever its sweeps, a launch per pass two per sweep
    from sphgpu import scenes
    steps = []
    for cap in (3, 9):
        with scenes.build_system(_scene(n, cap, 1e-9)) as g:
            steps.append(_step(g))
    assert [s[1] for s in steps] == [3, 9]
    assert (steps[0][0] == steps[1][0]) == at_once


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_a_solve_goes_on_in_further_launches(monkeypatch, precision):
    from sphgpu import scenes
    sc = _scene(5000, 0, 50.0)  # (an error that three sweeps reach)
    with scenes.build_system(sc, precision=precision) as g:
        want = [(_step(g), _state(g)) for _ in range(3)]
    monkeypatch.setenv("SPHGPU_SOLVE_SWEEPS", "1")
    with scenes.build_system(sc, precision=precision) as g:
        for (launches, sweeps), state in want:
            got = _step(g)
            assert got == (launches + sweeps - 1, sweeps) and sweeps > 2
            assert _same(_state(g), state)


@pytest.mark.parametrize("captured", [0, 2])
def test_a_wait_that_runs_out_is_an_error_and_the_handle_restarts(monkeypatch, captured):
    from sphgpu import _capi as A, scenes
    sc = _scene(8000, 30, 0.1)
    with scenes.build_system(sc) as ref:
        ref.step_forward_in_time(2)
        ck = ref.get_fluid_checkpoint()
        ref.continue_from_checkpoint(ck)
        first = _state(ref)
        ref.step_forward_in_time(2)
        second = _state(ref)
    monkeypatch.setenv("SPHGPU_BARRIER_POLLS", "1")
    with scenes.build_system(sc) as g:
        g.set_step_graphs(captured)
        for _ in range(2):
            with pytest.raises(A.SPHError) as e:
                g.step_forward_in_time(2)
            assert e.value.code == A.SPH_ERR_CUDA
        with pytest.raises(A.SPHError):  # the limit still holds
            g.continue_from_checkpoint(ck)
        monkeypatch.delenv("SPHGPU_BARRIER_POLLS")
        g.continue_from_checkpoint(ck)
        assert _same(_state(g), first)
        g.step_forward_in_time(2)
        assert _same(_state(g), second)


def test_two_solves_at_once_that_each_fill_the_gpu():
    from sphgpu import scenes
    sc = _scene(130000, 6, 1e-9)

    def run(out, k):
        with scenes.build_system(sc) as g:
            g.step_forward_in_time(4)
            out[k] = _state(g)
    states = {}
    run(states, "alone")
    threads = [threading.Thread(target=run, args=(states, k)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert _same(states[0], states["alone"]) and _same(states[1], states["alone"])
