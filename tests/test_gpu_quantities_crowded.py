"""Quantities at positions in a compressed fluid, where a position has far more
particles in reach than the candidate list holds, for calls of whole and of partial
warps whose positions lie in one cell or in many, some of them with nothing in reach.

The density, sum_j m_j W(r), is summed in f64 from f32 positions and rounded to f32 once:
2^-24 of the value, and as much again for the sum's own rounding.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, SPACING = 0.04, 0.02


@pytest.fixture(scope="module", params=["f32", "f64"])
def fluid(request):
    from sphgpu import GpuSystem, make_config
    x = np.random.default_rng(4).uniform(0, 5 * H, (7500, 3)).astype(np.float32).astype(np.float64)
    m = 1000.0 * SPACING ** 3
    p = dict(rest_density_grid_spacing=SPACING, kernel_support_radius=H, disable_particles_below=-1e6,
             time_increment=1e-4, stiffness=10.0)
    g = GpuSystem(make_config({"pressure_solver": "SESPH", "integration_scheme": "EulerCromer"}, p,
                              precision=request.param))
    g.upload_fluid(x, None, np.full(len(x), m))
    g.initialize()
    yield g, x, float(np.float32(m)) if request.param == "f32" else m
    g.close()


@pytest.mark.parametrize("count", [1, 31, 32, 33, 257, 1000])
@pytest.mark.parametrize("where", ["one cell", "the fluid", "in and out"])
def test_density(fluid, count, where):
    from sphgpu import capi
    g, x, m = fluid
    lo, hi = {"one cell": (2.1, 2.9), "the fluid": (0.0, 5.0), "in and out": (-3.0, 8.0)}[where]
    p = np.random.default_rng(count).uniform(lo * H, hi * H, (count, 3)).astype(np.float32)
    got = g.get_quantity_at_positions(capi.Q_DENSITY, p)
    for i in range(count):
        d = p[i].astype(np.float64) - x
        r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        q = r[r < H] / H
        w = 16.0 / np.pi / H ** 3 * (np.maximum(1 - q, 0) ** 3 - 4 * np.maximum(0.5 - q, 0) ** 3)
        assert abs(got[i] - m * w.sum()) <= 2.0 ** -23 * m * w.sum(), i
