"""Neighbor passes stage no halo records while most blocks' halos are larger than the
staging capacity (a compressed scene), and stage them again once the halos fit: the
steps are those of one fixed setting, bit for bit, called one by one and captured, while
a scene goes from one side of the rule to the other.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _flow(n, seed):
    """A lattice pressed together that flies apart."""
    from sphgpu import scenes
    sc = scenes.serving_dam_break(n, "SESPH", stiffness=3000.0, seed=seed)
    x = 0.45 * (sc.position - sc.position.mean(0))
    sc.position = x.astype(np.float32).astype(np.float64)
    sc.velocity = (40.0 * x).astype(np.float32).astype(np.float64)
    sc.sample_boundaries = []
    sc.parameters = dict(sc.parameters, time_increment=5e-4)
    return sc


@pytest.mark.parametrize("solver", ["SESPH", "SESPHwSplitting"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("chunk", [0, 4])
def test_the_rule_changes_no_result(monkeypatch, solver, precision, chunk):
    from sphgpu import _capi as A, scenes
    sc = _flow(12000, 3)
    sc.procedures = dict(sc.procedures, pressure_solver=solver)

    def run(stage):
        if stage is not None:
            monkeypatch.setenv("SPHGPU_HALO_STAGE", stage)
        else:
            monkeypatch.delenv("SPHGPU_HALO_STAGE", raising=False)
        out, most = [], []
        with scenes.build_system(sc, precision=precision) as g:
            g.set_step_graphs(chunk)
            for _ in range(24):
                g.step_forward_in_time(4)
                most.append(g.step_stats()["max_neighbors"])
                out.append([g.download(f) for f in (A.FIELD_POSITION, A.FIELD_VELOCITY, A.FIELD_PRESSURE)])
        return out, most
    want, most = run("0")
    assert most[0] > 200 and most[-1] < 100, most
    got, _ = run(None)
    for a, b in zip(got, want):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
