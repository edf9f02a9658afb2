"""The fluid neighbor search on the shapes that take its different routes.

Lists are compared, as sets per particle, with a brute-force f64 search (the
reference's predicate, sqrt((dx^2 + dy^2) + dz^2) < h), volumes with the f64
sum. The f32 volume's bound: each kernel value and each step of the
compensated sum carries a few ulp (2^-23), the last division and product one
each, so 16 ulp hold whatever the number of neighbors (all terms are
positive).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 0.04
SPACING = 0.5 * H


def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _clouds():
    rng = np.random.default_rng(3)
    g = np.arange(13) * SPACING
    lattice = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)
    jittered = lattice + rng.uniform(-0.2 * SPACING, 0.2 * SPACING, lattice.shape)
    out = {f"first_{n}": jittered[:n] for n in (1, 2, 31, 255, 256, 257)}
    out["lattice"] = lattice                                     # pairs at the support radius: the exact predicate
    out["lattice_negative"] = lattice - 0.11                     # cells on both sides of the origin
    out["long_lists"] = rng.uniform(0, 3 * H, (1900, 3))         # hundreds of neighbors, halo staged
    out["large_halo"] = rng.uniform(0, 3 * H, (4200, 3))         # halo beyond the staged positions
    out["sparse"] = rng.uniform(-30 * H, 30 * H, (700, 3))       # a cell per particle
    out["far_clusters"] = np.concatenate([jittered[:300], jittered[:300] + 700 * H])
    out["coincident"] = np.repeat(jittered[:150], 2, axis=0)
    thin = np.stack(np.meshgrid(np.arange(90) * SPACING, np.arange(90) * SPACING, [0.0], indexing="ij"), -1)
    out["layer"] = thin.reshape(-1, 3) + rng.uniform(0, 0.3 * SPACING, (8100, 3))
    return {k: _f32(v) for k, v in out.items()}


CLOUDS = _clouds()


def _brute(x):
    rows, vol = [], np.empty(len(x))
    alpha, V0 = 16.0 / np.pi, SPACING ** 3
    for i in range(len(x)):
        d = x[i] - x
        r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        near = np.nonzero(r < H)[0]
        rows.append(near)
        q = r[near] / H
        w = alpha / H ** 3 * (np.maximum(1 - q, 0) ** 3 - 4 * np.maximum(0.5 - q, 0) ** 3)
        vol[i] = V0 / (V0 * w.sum())
    return rows, vol


@pytest.mark.parametrize("cloud", list(CLOUDS))
@pytest.mark.parametrize("solver", ["SESPH", "IISPH"])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_lists_and_volumes(cloud, solver, precision):
    from sphgpu import GpuSystem, capi, make_config
    x = CLOUDS[cloud]
    rows, vol = _brute(x)
    params = dict(rest_density_grid_spacing=SPACING, kernel_support_radius=H, disable_particles_below=-1e6,
                  time_increment=1e-4, stiffness=10.0, max_solver_iterations=3)
    cfg = make_config({"pressure_solver": solver, "integration_scheme": "EulerCromer",
                       "boundary_handling": "StaticSampleBoundary"}, params, precision=precision)
    with GpuSystem(cfg) as g:
        g.upload_fluid(x, None, np.full(len(x), 1000.0 * SPACING ** 3))
        g.initialize()
        off, idx = g.fluid_neighbors()
        for i, near in enumerate(rows):
            assert np.array_equal(idx[off[i]:off[i + 1]], near), (cloud, i)
        got = g.download(capi.FIELD_VOLUME)
        tol = 16 * 2.0 ** -23 if precision == "f32" else 1e-13
        assert np.max(np.abs(got - vol) / vol) < tol
