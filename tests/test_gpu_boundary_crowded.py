"""The pass over the boundary samples where a block holds fewer cells than warps
(compressed fluid): cells of up to a block's particles, with remainders of the groups
of eight that its warps take, against the oracle like the ordinary forms
(test_gpu_boundary_pass, whose bounds hold here too).
"""
import numpy as np
import pytest

from conftest import build_oracle
from test_gpu_boundary_pass import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [0.2, 0.35, 0.5, 0.7])
@pytest.mark.parametrize("solver,body", [("SESPH", True), ("SESPHwSplitting", False), ("IISPH", True)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_first_update_of_a_compressed_fluid(spread, solver, body, precision):
    import oracle as O
    from sphgpu import capi, scenes
    sc = _scene(0.5, spread, solver, body)
    tol = 1e-4 if precision == "f32" else 1e-9
    o = build_oracle(sc)
    with scenes.build_system(sc, precision=precision) as g:
        for field, ofield in ((capi.FIELD_VOLUME, O.F_VOLUME), (capi.FIELD_ACCELERATION, O.F_ACCELERATION)):
            want = o.download(ofield)
            assert np.abs(g.download(field) - want).max() <= tol * np.abs(want).max()
        if body:
            want = np.asarray(o.rigid_state(1))[13:]
            assert np.abs(g.rigid_state(1)[13:] - want).max() <= tol * np.abs(want).max()
