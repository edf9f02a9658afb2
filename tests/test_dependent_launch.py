"""Kernels that may start while the one before them still writes (programmatic
dependent launch) promise nothing about their buffers that does not hold then, and
wait before they use them. Read from the source: such an overlap cannot be forced
from outside, and a wrong order need not show.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-simulation_b200", "csrc")


def _read(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _close(text, i):
    """The index behind the parenthesis that closes the one before index i."""
    depth = 1
    while depth:
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        i += 1
    return i


def _functions(text):
    """name -> (parameters, body) of the functions at top level that have one."""
    while "__launch_bounds__(" in text:
        i = text.index("__launch_bounds__(")
        text = text[:i] + text[_close(text, i + len("__launch_bounds__(")):]
    out = {}
    for m in re.finditer(r"^(?:__global__|__device__)[^;{(]*?\b(\w+)\(", text, re.M):
        i = _close(text, m.end())
        if text[i:i + 60].lstrip().startswith("{"):
            out[m.group(1)] = (text[m.end():i - 1], text[i:text.index("\n}", i)])
    return out


KERNELS = _functions(_read("sph_kernels.cuh"))
SYSTEM = _read("sph_system.cu")
DEPENDENT = sorted(set(re.findall(r"launch_dep\([^;]*?\b(k_\w+)", SYSTEM)) |
                   set(re.findall(r"launch_impl\([^;]*?\b(k_\w+)", SYSTEM)))


def test_the_launches_are_found():
    assert {"k_scan_tiles", "k_scatter", "k_gather_particles", "k_neighbors_density", "k_volume", "k_accel",
            "k_sweep_accel", "k_sweep_jacobi", "k_sample_boundary", "k_vm_sample"} <= set(DEPENDENT)


@pytest.mark.parametrize("kernel", DEPENDENT)
def test_dependent_kernel(kernel):
    parameters, body = KERNELS[kernel]
    assert "grid_dep_begin();" in body or "grid_dep_wait();" in body
    assert "__restrict__" not in parameters


def test_helpers_on_overlapped_buffers_promise_nothing():
    for name in ("scan_load8", "ranked_place"):
        assert "__restrict__" not in KERNELS[name][0]


def test_non_coherent_loads_are_of_settled_data():
    loads = re.findall(r"__ldg\(([^)]*)\)", _read("sph_kernels.cuh").split("grid_dep_begin()", 1)[1])
    assert loads and all(re.match(r"H\.idx \+ l$|base \+ offset\(k$", x) for x in loads), loads
