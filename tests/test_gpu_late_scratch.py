"""Scratch that only some uses need is made when the first of them is set up: a context for
sorts or short solves holds none of the tile plans, one that never runs the binary search none
of its cell table.  A search captured before the table exists gives the same rows."""
import numpy as np
import pytest
import torch

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu

CAP = 1 << 20


def _bytes_used(f):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    f()
    torch.cuda.synchronize()
    return (before - torch.cuda.mem_get_info()[0]) / CAP  # per particle


def test_scratch_is_made_when_needed():
    from apbf_gb300.api import Context

    ctx = Context(particle_capacity=CAP, max_neighbors=4, max_log2res=3)
    plan = 4 * 640 / 128 + 4 + 16 * 8 + 4  # halo, lane, rows, tail
    assert _bytes_used(lambda: ctx.set_settings(basic_pbf=1, solver_iterations=3)) < 8
    assert 0.95 * plan < _bytes_used(lambda: ctx.set_settings(solver_iterations=8)) < plan + 12
    assert _bytes_used(lambda: ctx.set_settings(solver_iterations=9)) < 8
    assert 0.95 * plan < _bytes_used(lambda: ctx.set_settings(basic_pbf=0, base_kernel_width_on_boundary_distance=0)) < plan + 12
    assert 30 < _bytes_used(lambda: ctx.set_neighborhood_search("binary_search")) < 70
    assert _bytes_used(lambda: ctx.set_neighborhood_search("green")) < 8
    assert _bytes_used(lambda: ctx.set_neighborhood_search("binary_search")) < 8
    ctx.close()


@pytest.mark.parametrize("equal", [True, False])
def test_binary_search_captured_before_its_table(equal):
    from apbf_gb300.api import Context, neighborhood_binary_search

    rng = np.random.default_rng(6)
    st = scenes.make_state(rng.uniform(0.0, 20.0, size=(3000, 3)))
    if not equal:
        st["kernel_width"] = (st["kernel_width"] * rng.uniform(0.5, 1.2, size=3000)).astype(np.float32)

    def context():
        ctx = Context(particle_capacity=4000, max_neighbors=256, max_log2res=3)
        ctx.upload(st)
        return ctx, neighborhood_binary_search().set_data(ctx).set_range_scale(1.0)

    ref, search = context()
    search.apply()
    ctx, search = context()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        search.apply()
    graph.replay()
    torch.cuda.synchronize()
    ctx.check_status()
    want, got = ref.download_rows(), ctx.download_rows()
    assert len(want) == len(got) == 3000
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    ref.close()
    ctx.close()
