"""The tiled solve of apbf_substep against the direct passes of the stage objects, bit for
bit, on the forms of rows that differ: transposed rows (spread kernel widths, the binary
search with radii that differ) and their boundariness filter, the filter asked in the density
pass, kernel widths several times narrower than their neighbours' (exponents below -126),
rows of more than 64 entries whose rest comes from the pool, from the list by threads, and
from the list when the pool is full; per-kernel launches, the solve loop's graph and the whole
substep as a graph."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 240.0
SPREAD = dict(basic_pbf=0, base_kernel_width_on_boundary_distance=0)
CASES = {
    # settings, share of particles with another width and its factor, width factor of the others, binary search
    "plain": ({}, 0.0, 1.0, 1.0, False),
    "uneven": ({}, 1.0, (0.7, 1.3), 1.0, False),
    "bs_equal": ({}, 0.0, 1.0, 1.0, True),
    "bs_uneven": ({}, 1.0, (0.7, 1.3), 1.0, True),
    "spread": (SPREAD, 1.0, (0.8, 1.2), 1.0, False),
    "spread_drop": (dict(SPREAD, kernel_width_adaption_speed=0.95), 0.04, 4.0, 1.0, False),
    "narrow": ({}, 0.05, 0.25, 1.0, False),
    "rests_pool": ({}, 0.03, 2.4, 1.0, False),
    "rests_full": ({}, 0.15, 2.6, 1.0, False),
    "rests_lanes": ({}, 0.0, 1.0, 1.6, False),
    "rests_lanes_bs": ({}, 1.0, (0.9, 1.1), 1.6, True),
}


def _state(case, n=1500):
    settings, share, factor, others, _ = CASES[case]
    rng = np.random.default_rng(len(case))
    side = int(np.ceil(n ** (1.0 / 3.0)))
    st = scenes.make_state(scenes.lattice([20.0, 6.0, 20.0], [side] * 3, 1.9, 0.3, rng)[:n])
    f = np.full(n, others)
    pick = rng.uniform(size=n) < share
    f[pick] *= rng.uniform(*factor, size=int(pick.sum())) if isinstance(factor, tuple) else factor
    st["kernel_width"] = (st["kernel_width"] * f).astype(np.float32)
    if not settings.get("basic_pbf", 1):
        st["target_radius"] = rng.uniform(1.0, 1.6, size=n).astype(np.float32)
    return st


def _ctx(case, st, capacity, filter_in_density):
    from apbf_gb300.api import Context

    ctx = Context(particle_capacity=capacity, max_neighbors=1500, max_log2res=4)
    ctx.set_settings(**{"basic_pbf": 1, "solver_iterations": 6, **CASES[case][0]})
    ctx.set_scene((-4.0, -4.0, -4.0), (60.0, 60.0, 60.0), 4, (0.0, -392.4, 0.0))
    ctx.set_boxes(np.array([[-2.0, -2.0, -2.0, 0.0]], np.float32), np.array([[60.0, 7.0, 60.0, 0.0]], np.float32))
    if CASES[case][4]:
        ctx.set_neighborhood_search("binary_search")
    if filter_in_density:
        ctx.set_tuning(filter_in_density=1)
    ctx.upload(st)
    return ctx


class _BinarySearch:
    """neighborhood_binary_search in the place of the Green search of SubstepStages."""

    def __init__(self, ctx):
        from apbf_gb300.api import neighborhood_binary_search

        self.stage = neighborhood_binary_search().set_data(ctx)

    def set_range_scale(self, scale):
        self.stage.set_range_scale(scale)
        return self

    def set_position_range(self, *_):
        return self

    def apply(self, stream=None):
        self.stage.apply(stream)


def _staged(case, st, capacity, filter_in_density, substeps):
    from apbf_gb300.api import SubstepStages

    ctx = _ctx(case, st, capacity, filter_in_density)
    stages = SubstepStages(ctx)
    if CASES[case][4]:
        stages.neighborhood = _BinarySearch(ctx)
    for _ in range(substeps):
        stages.update(DT)
    out = ctx.download()[0]
    rows = [len(r) for r in ctx.download_rows()]
    ctx.close()
    return out, np.array(rows)


@pytest.mark.parametrize("capacity", [2000, 30_000])  # the 64 x 2 and the 128 x 1 tiles
@pytest.mark.parametrize("case,filter_in_density", [(c, 0) for c in CASES] + [("plain", 1), ("uneven", 1), ("rests_pool", 1),
                                                                          ("rests_lanes", 1)])
def test_tiles_equal_direct_passes(capacity, case, filter_in_density):
    st = _state(case)
    want, rows = _staged(case, st, capacity, filter_in_density, 3)
    if case.startswith("rests"):
        assert np.any(rows > 64)
    for mode in ("profiled", 0, 1, 2):
        ctx = _ctx(case, st, capacity, filter_in_density)
        if mode == "profiled":
            ctx.profile_enable(True)
        else:
            ctx.set_solve_graph(mode)
        for _ in range(3):
            ctx.substep(DT)
        if mode == "profiled":
            names, _ = ctx.profile_read()
            assert "k_density_tiles" in names and "k_delta_tiles" in names and "k_density_lambda" not in names
            assert names["k_tile_rows"][0] == (6 if CASES[case][4] or not CASES[case][0].get("basic_pbf", 1) else 3)
        got = ctx.download()[0]
        ctx.check_status()
        for k in want:
            assert got[k].tobytes() == want[k].tobytes(), (mode, k)
        ctx.close()


def test_blocks_that_take_a_second_tile():
    """More tiles than the passes have blocks (152 x 64): each block goes on to another tile."""
    from apbf_gb300.api import Context, SubstepStages

    side = 110
    n = side ** 3
    rng = np.random.default_rng(1)
    st = scenes.make_state(scenes.lattice([4.0, 4.0, 4.0], [side] * 3, 1.9, 0.3, rng))
    st["kernel_width"] = (st["kernel_width"] * rng.uniform(0.9, 1.1, size=n)).astype(np.float32)
    out = []
    for fused in (True, False):
        ctx = Context(particle_capacity=n, max_neighbors=96, max_log2res=6)
        ctx.set_settings(basic_pbf=1, solver_iterations=4)
        ctx.set_scene((-4.0,) * 3, (252.0,) * 3, 6, (0.0, -392.4, 0.0))
        ctx.set_boxes(np.array([[-2.0, -2.0, -2.0, 0.0]], np.float32), np.array([[250.0, 5.0, 250.0, 0.0]], np.float32))
        ctx.upload(st)
        if fused:
            ctx.substep(DT)
        else:
            SubstepStages(ctx).update(DT)
        ctx.check_status()
        out.append(ctx.download()[0])
        ctx.close()
    for k in out[0]:
        assert out[0][k].tobytes() == out[1][k].tobytes(), k
