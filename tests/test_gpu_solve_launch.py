"""A solve in one cooperative launch takes the same operations in the same order
as its passes launched one by one (what a system with profiling on does), so the
states and the sweep counts are equal bit for bit: one block with a remainder,
many blocks, as many as the GPU holds and more, halos staged and not, capped
and uncapped solves, stepping by calls and by a captured graph.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(n, solver, precision, cap, profiling, captured, steps):
    from sphgpu import _capi as A, scenes
    sc = scenes.serving_dam_break(n, solver=solver)
    if solver == "IISPHwOST":
        sc.procedures = dict(sc.procedures, integration_scheme="TakePredicted")
    # (without a cap: an error that three sweeps reach)
    sc.parameters = dict(sc.parameters, max_solver_iterations=cap, target_density_error=0.1 if cap else 50.0)
    with scenes.build_system(sc, precision=precision) as g:
        g.set_profiling(profiling)
        if captured:
            g.set_step_graphs(steps)
            g.step_forward_in_time(steps)
        else:
            for _ in range(steps):
                g.step_forward_in_time(1)
        return [g.download(f) for f in (A.FIELD_POSITION, A.FIELD_VELOCITY, A.FIELD_PRESSURE)] + \
            [np.array(g.step_stats()["solver_iterations"])]


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n,solver,precision,cap,stage", [
    (200, "IISPH", "f32", 30, None),
    (700, "IISPH", "f64", 30, None),
    (5000, "IISPHwOST", "f32", 30, None),
    (5000, "IISPH", "f32", 0, None),
    (30000, "IISPH", "f32", 30, "300"),
    (30000, "IISPH", "f64", 30, "300"),
    (150000, "IISPH", "f32", 30, None),
    (160000, "IISPH", "f32", 30, None),
])
def test_one_launch_equals_the_passes(monkeypatch, n, solver, precision, cap, stage, captured):
    if stage:
        monkeypatch.setenv("SPHGPU_HALO_STAGE", stage)
    want = _run(n, solver, precision, cap, True, captured, 3)
    got = _run(n, solver, precision, cap, False, captured, 3)
    assert got[-1] > 0 and np.isfinite(got[0]).all()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
