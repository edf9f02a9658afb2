"""A fluid uploaded again before initialize: what the first upload still does to its
buffers is over before they go back to the pool (the order is read from the source,
since a block in use by two systems need not show), and the result is the last
upload's.
"""
import os
import re
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_an_upload_waits_for_all_it_has_launched():
    with open(os.path.join(ROOT, "fluid-simulation_b200", "csrc", "sph_system.cu")) as f:
        text = f.read()
    body = re.search(r"void upload_fluid\(.*?\n  }\n", text, re.S).group(0)
    load = re.search(r"void load_state\(.*?\n  }\n", text, re.S).group(0)
    assert load.rstrip().endswith("sync();\n  }")
    assert "stream_" not in body[body.index("load_state("):]


@pytest.mark.gpu
def test_the_last_upload_counts():
    from sphgpu import GpuSystem, capi, make_config
    h, sp = 0.04, 0.02

    def system():
        return GpuSystem(make_config({"pressure_solver": "SESPH", "integration_scheme": "EulerCromer"},
                                     dict(rest_density_grid_spacing=sp, kernel_support_radius=h, time_increment=1e-4,
                                          stiffness=10.0, disable_particles_below=-1e6)))

    def block(n, seed):
        rng = np.random.default_rng(seed)
        c = np.arange(n) * sp
        return np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(0, 0.2 * sp, (n ** 3, 3))

    def run(sizes, seed):
        with system() as g:
            for k, n in enumerate(sizes):
                x = block(n, seed + k)
                g.upload_fluid(x, None, np.full(len(x), 1000.0 * sp ** 3))
            g.initialize()
            g.step_forward_in_time(2)
            return g.download(capi.FIELD_POSITION), g.download(capi.FIELD_ACCELERATION)
    keep = system()  # from here on freed blocks are kept
    want = [run([17], 3), run([24], 9)]
    got = {}
    threads = [threading.Thread(target=lambda k=k: got.update({k: run([30, 9, [17, 24][k]], [1, 7][k])}))
               for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert all(np.array_equal(a, b) for a, b in zip(got[k], want[k])), k
    keep.close()
