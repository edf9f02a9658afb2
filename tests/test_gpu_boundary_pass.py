"""The pass over the boundary samples: buckets with more samples than a warp
stages at a time, cells of one and of many particles, corners of three walls,
a dynamic body next to the fluid. Volumes, accelerations and the body's force
and torque are compared with the oracle after the first update.

Bounds: f64 1e-9 relative to the largest value (other summation orders of some
hundred terms). f32: sums of up to a few hundred terms of single precision,
2^-23 each, times the condition of the sums (terms of both signs), below 1e-4
of the largest value.
"""
import numpy as np
import pytest

from conftest import build_oracle

pytestmark = pytest.mark.gpu


def _scene(samples, spread, solver, body):
    from sphgpu import scenes
    from sphgpu.system import RigidInit
    h = 0.02
    sc = scenes.dam_break_sesph_8k(n_side=6)
    lo = sc.position.min(axis=0)
    x = lo + (sc.position - lo) * spread
    sc.position = x.astype(np.float32).astype(np.float64)
    sc.velocity = np.random.default_rng(2).uniform(-0.3, 0.3, x.shape).astype(np.float32).astype(np.float64)
    verts = scenes.transform_mesh(scenes.CUBE_VERTICES, scale=(0.3,) * 3)
    walls = scenes.sample_triangle_mesh_surface(verts, scenes.CUBE_FACES_INWARD, samples * h)
    walls = walls[(walls < lo.max() + 0.2).all(axis=1)].astype(np.float32).astype(np.float64)
    sc.sample_boundaries = [(walls, None)]
    if body:
        side = 0.08
        bv = scenes.transform_mesh(scenes.CUBE_VERTICES, scale=(side / 2,) * 3)
        pts = scenes.sample_triangle_mesh_surface(bv, scenes.CUBE_FACES_OUTWARD, samples * h)
        top = sc.position[:, 2].max()
        sc.sample_boundaries.append((pts.astype(np.float32).astype(np.float64), RigidInit(
            mass=0.4, inertia_body=scenes.box_inertia(0.4, side),
            center_of_mass=(float(np.float32(lo[0] + 0.06)), float(np.float32(lo[1] + 0.06)),
                            float(np.float32(top + side / 2 + 0.015))), angular_velocity=(0.0, 0.5, 0.0))))
    sc.procedures = dict(sc.procedures, pressure_solver=solver)
    sc.parameters = dict(sc.parameters, max_solver_iterations=4, target_density_error=0.1, relaxation_factor=0.5,
                         min_diagonal_element=1e-10)
    return sc


@pytest.mark.parametrize("samples,spread", [(0.7, 1.0), (0.25, 1.0), (0.4, 2.2)])
@pytest.mark.parametrize("solver", ["SESPH", "SESPHwSplitting", "IISPH"])
@pytest.mark.parametrize("body", [False, True])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_first_update_matches_the_oracle(samples, spread, solver, body, precision):
    import oracle as O
    from sphgpu import capi, scenes
    sc = _scene(samples, spread, solver, body)
    tol = 1e-4 if precision == "f32" else 1e-9
    o = build_oracle(sc)
    with scenes.build_system(sc, precision=precision) as g:
        for field, ofield in ((capi.FIELD_VOLUME, O.F_VOLUME), (capi.FIELD_ACCELERATION, O.F_ACCELERATION)):
            want = o.download(ofield)
            assert np.abs(g.download(field) - want).max() <= tol * np.abs(want).max()
        if body:
            want = np.asarray(o.rigid_state(1))[13:]
            assert np.abs(g.rigid_state(1)[13:] - want).max() <= tol * np.abs(want).max()
