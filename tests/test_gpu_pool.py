"""Systems built from memory that earlier systems left: the results are those of
fresh memory, bit for bit, whatever ran in between (other sizes, solvers and
precisions, several threads), and memory goes back once no system is alive.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(solver, n, precision="f32", graph=0, steps=3, seed=1):
    from sphgpu import capi, scenes
    sc = scenes.serving_dam_break(n, "IISPH" if solver == "IISPH" else "SESPH", seed=seed)
    sc.procedures["pressure_solver"] = solver
    with scenes.build_system(sc, precision=precision) as g:
        g.set_step_graphs(graph)
        g.step_forward_in_time(steps)
        return [g.download(f) for f in (capi.FIELD_POSITION, capi.FIELD_VELOCITY, capi.FIELD_VOLUME,
                                        capi.FIELD_PRESSURE, capi.FIELD_ACCELERATION)]


CASES = [("IISPH", 4000, "f32", 0), ("SESPH", 9000, "f32", 3), ("SESPHwSplitting", 2500, "f64", 0),
         ("IISPH", 6000, "f64", 2), ("SESPHwSplitting", 5000, "f32", 0)]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_reused_memory_changes_no_result():
    from sphgpu import scenes
    fresh = [_run(*c) for c in CASES]  # nothing is alive between these: fresh memory each
    keep = scenes.build_system(scenes.dam_break_sesph_8k(n_side=6))  # from here on freed blocks are kept
    for order in (range(len(CASES)), reversed(range(len(CASES)))):
        for k in order:
            assert _same(_run(*CASES[k]), fresh[k]), CASES[k]
    results = {}

    def work(k):
        for _ in range(3):
            results[k] = _run(*CASES[k])
            assert _same(results[k], fresh[k])
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(CASES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert sorted(results) == list(range(len(CASES))) and all(_same(results[k], fresh[k]) for k in results)
    keep.close()


def test_memory_goes_back_with_the_last_system():
    import torch
    from sphgpu import scenes
    torch.cuda.synchronize()
    sc = scenes.serving_dam_break(60000, "IISPH", seed=2)
    scenes.build_system(sc).close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        scenes.build_system(sc).close()
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 4 << 20
