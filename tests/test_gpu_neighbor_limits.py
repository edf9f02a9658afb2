"""The fluid neighbor search at its limits: candidates in the guard band of a list
that is longer than its capacity, positions that are not finite, halos that fill the
staged positions or go through them in pieces, a halo as large as 16-bit positions allow.

Lists are compared, as sets per particle, with a brute-force f64 search (the
reference's predicate, sqrt((dx^2 + dy^2) + dz^2) < h).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(x, h, spacing, solver="SESPH", precision="f32", **parameters):
    from sphgpu import GpuSystem, make_config
    params = dict(rest_density_grid_spacing=spacing, kernel_support_radius=h, disable_particles_below=-1e6,
                  time_increment=1e-4, stiffness=10.0, max_solver_iterations=3, **parameters)
    g = GpuSystem(make_config({"pressure_solver": solver, "integration_scheme": "EulerCromer",
                               "boundary_handling": "StaticSampleBoundary"}, params, precision=precision))
    g.upload_fluid(x, None, np.full(len(x), 1000.0 * spacing ** 3))
    g.initialize()
    return g


def _near(x, i, h):
    d = x[i] - x
    return np.nonzero(np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) < h)[0]


# A lattice has whole shells of neighbors at the support radius: 24 at sqrt(6)
# and sqrt(10) spacings, 56 and 122 nearer ones. In a ball of that radius the
# center's list is longer than the capacity with the shell and shorter without it;
# every other list is shorter.
@pytest.mark.parametrize("shell,capacity", [(6, 72), (10, 132)])
@pytest.mark.parametrize("solver", ["SESPH", "IISPH"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_shell_at_the_support_radius_beyond_the_capacity(shell, capacity, solver, precision):
    spacing = 1.0 / 64
    h = np.sqrt(shell) * spacing
    c = np.arange(-4, 5)
    x = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    x = x[(x * x).sum(1) <= shell] * spacing + 0.25
    with _system(x, h, spacing, solver, precision, neighbor_capacity=capacity) as g:
        off, idx = g.fluid_neighbors()
    for i in range(len(x)):
        assert np.array_equal(np.sort(idx[off[i]:off[i + 1]]), _near(x, i, h)), i


# Not a number and infinite positions are nobody's neighbors and have none (every
# comparison with such a distance is false), whatever the sign of the NaN.
@pytest.mark.parametrize("value", [0x7FF8 << 48, 0xFFF8 << 48, 0x7FF0 << 48, 0xFFF0 << 48])
@pytest.mark.parametrize("count", [1, 3])
@pytest.mark.parametrize("solver", ["SESPH", "IISPH"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_positions_that_are_not_finite_have_no_neighbors(value, count, solver, precision):
    h = 0.04
    c = (np.arange(5) + 0.5) * 0.5 * h
    x = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3).astype(np.float32).astype(np.float64)
    x[10:10 + count, 1] = np.array([value], np.uint64).view(np.float64)[0]
    with _system(x, h, 0.5 * h, solver, precision) as g:
        off, idx = g.fluid_neighbors()
    for i in range(len(x)):
        got = np.sort(idx[off[i]:off[i + 1]])
        if 10 <= i < 10 + count:
            got = got[got != i]  # (the row of a particle holds the particle itself)
            assert len(got) == 0, i
        else:
            with np.errstate(invalid="ignore"):
                assert np.array_equal(got, _near(x, i, h)), i


# Blocks on both sides of a corner see the same eight cells from either side: 34000
# particles, 68000 halo positions with the second copies. Alone, the particles have a
# bucket grid of eight cells per axis, on whose edge the corner lies; with one far away,
# the grid is larger and the Morton curve jumps there. 16 ulp as in the search's own test.
@pytest.mark.parametrize("far", [0, 1])
def test_halo_beyond_16_bit_positions_only_with_second_copies(far):
    from sphgpu import capi
    h, n = 0.04, 34000
    rng = np.random.default_rng(1)
    x = np.column_stack([rng.uniform(0.01, 1.99, n), rng.uniform(0.01, 1.99, n), rng.uniform(15.01, 16.99, n)]) * h
    x = np.concatenate([x, np.full((far, 3), 40.0 * h)]).astype(np.float32).astype(np.float64)
    with _system(x, h, 0.5 * h) as g:
        vol = g.download(capi.FIELD_VOLUME)
    for i in rng.integers(0, n, 200):
        d = x[i] - x[_near(x, i, h)]
        q = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) / h
        w = 16.0 / np.pi / h ** 3 * (np.maximum(1 - q, 0) ** 3 - 4 * np.maximum(0.5 - q, 0) ** 3)
        assert abs(vol[i] * w.sum() - 1.0) < 16 * 2.0 ** -23, i


def _check_lists(x, h, spacing, solver, precision):
    from sphgpu import capi
    with _system(x, h, spacing, solver, precision) as g:
        off, idx = g.fluid_neighbors()
        vol = g.download(capi.FIELD_VOLUME)
    tol = 16 * 2.0 ** -23 if precision == "f32" else 1e-13  # (as in the search's own test)
    for i in range(len(x)):
        near = _near(x, i, h)
        assert np.array_equal(np.sort(idx[off[i]:off[i + 1]]), near), i
        d = x[i] - x[near]
        q = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]) / h
        w = 16.0 / np.pi / h ** 3 * (np.maximum(1 - q, 0) ** 3 - 4 * np.maximum(0.5 - q, 0) ** 3)
        assert abs(vol[i] * w.sum() - 1.0) < tol, i


# All particles of a scene in 2 x 2 x 2 cells are every block's halo: around one, two and
# four pieces of 1024 (f64) and 2048 (f32) staged positions.
@pytest.mark.parametrize("n", [1023, 1024, 1025, 2047, 2048, 2049, 4096, 4099])
@pytest.mark.parametrize("solver,precision", [("SESPH", "f32"), ("IISPH", "f32"), ("SESPH", "f64")])
def test_halo_in_pieces(n, solver, precision):
    h = 0.04
    x = np.random.default_rng(n).uniform(0.01, 1.99, (n, 3)) * h
    _check_lists(x.astype(np.float32).astype(np.float64), h, 0.5 * h, solver, precision)


# 72 pairs of a particle at the support radius, in a halo of some pieces
@pytest.mark.parametrize("solver", ["SESPH", "IISPH"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_shell_at_the_support_radius_in_pieces(solver, precision):
    spacing = 1.0 / 64
    c = np.arange(14) * spacing
    x = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    _check_lists(x, np.sqrt(26.0) * spacing, spacing, solver, precision)
