"""apbf_set_scene between substeps: the next substep uses the new acceleration, range and
resolution also where substeps are replayed from a captured graph (mode 2, batches)."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def _run(how):
    from apbf_gb300.api import Batch, Context

    spec = scenes.dam_break(n_side=10)
    ctx = Context(particle_capacity=1200, max_neighbors=128, max_log2res=max(spec.log2res, 3))
    ctx.set_settings(basic_pbf=1, solver_iterations=4)
    ctx.load_scene(spec)
    batch = None
    if how == "batch":
        batch = Batch([ctx])
    else:
        ctx.set_solve_graph(how)
    step = (lambda: batch.substep(spec.dt)) if batch else (lambda: ctx.substep(spec.dt))
    for k in range(12):
        if k == 6:
            ctx.set_scene(spec.grid_min, spec.grid_max, spec.log2res, (150.0, -300.0, 40.0))
        if k == 9:
            ctx.set_scene(spec.grid_min, spec.grid_max, spec.log2res - 1, (0.0, -392.4, 0.0))
        step()
    ctx.check_status()
    out = ctx.download()[0]
    if batch:
        batch.close()
    ctx.close()
    return out


@pytest.mark.parametrize("how", [1, 2, "batch"])
def test_scene_changes_reach_captured_substeps(how):
    want, got = _run(0), _run(how)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
