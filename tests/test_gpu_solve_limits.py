"""The cooperative solve at its limits: which launches a step makes, a launch that
ends before the solve does, a barrier whose wait runs out, two solves at once whose
blocks each fill the GPU, and the sweeps that a launch per pass makes in vain.

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


@pytest.mark.parametrize("cap", [4, 10, 40, 100])
def test_no_sweep_is_launched_beyond_the_cap(monkeypatch, cap):
    # an error that is never reached: two launches per sweep of the cap, no more
    from sphgpu import scenes
    monkeypatch.setenv("SPHGPU_DEPENDENT_LAUNCH", "0")
    launches = []
    for c in (3, cap):
        with scenes.build_system(_scene(8000, c, 1e-9)) as g:
            launches.append([_step(g) for _ in range(3)])
    for (base, three), (got, sweeps) in zip(*launches):
        assert (three, sweeps) == (3, cap)
        assert got - base == 2 * (cap - 3)


@pytest.mark.parametrize("n", [8000, 160000])
def test_the_launches_of_a_solve_do_not_depend_on_earlier_ones(monkeypatch, n):
    # the same state after other flows; a converging solve has sweeps in vain, but no
    # more than twice those that it took
    from sphgpu import scenes
    monkeypatch.setenv("SPHGPU_DEPENDENT_LAUNCH", "0")
    sc = _scene(n, 100, 0.1)
    ck = None
    out = []
    for history in range(3):
        with scenes.build_system(sc) as g:
            if ck is None:
                ck = g.get_fluid_checkpoint()
                x = ck["position"]
                ck["velocity"] = -8.0 * (x - x.mean(0))
            if history == 1:
                g.step_forward_in_time(8)
            if history == 2:
                g.continue_from_checkpoint(dict(ck, velocity=0.25 * ck["velocity"]))
                g.step_forward_in_time(2)
            before = g.launch_count()
            g.continue_from_checkpoint(ck)
            got = [(g.launch_count() - before, g.step_stats()["solver_iterations"])]
            out.append(got + [_step(g) for _ in range(3)])
    assert out[1] == out[0] and out[2] == out[0]
    assert max(s for _, s in out[0]) > 6, out[0]
    with scenes.build_system(_scene(n, 3, 0.1)) as g:
        base = _step(g)[0]
    for launches, sweeps in out[0][1:]:
        assert launches - base <= 2 * (sweeps - 3) + 2 * max(8, 2 * sweeps), out[0]
