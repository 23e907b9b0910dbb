"""The tiled solve of apbf_substep against the direct passes of the stage objects, bit for
bit: lists that end at the edges of a tile (64 and 128 particles), rows of more than 64
entries, tiles with more outside neighbours than fit, rows cut at their capacity, equal and
differing kernel widths, in both tile shapes."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def _ctx(state, capacity, maxn, iterations):
    from apbf_gb300.api import Context

    ctx = Context(particle_capacity=capacity, max_neighbors=maxn, max_log2res=4)
    ctx.set_settings(basic_pbf=1, solver_iterations=iterations)
    ctx.set_scene((-4.0, -4.0, -4.0), (60.0, 60.0, 60.0), 4, (0.0, -392.4, 0.0))
    ctx.set_boxes(np.array([[-2.0, -2.0, -2.0, 0.0]], np.float32), np.array([[60.0, 9.0, 60.0, 0.0]], np.float32))
    ctx.upload(state)
    return ctx


def _state(n, dense, widths):
    rng = np.random.default_rng(n + int(7 * dense))
    if dense == 0:
        side = int(np.ceil(n ** (1.0 / 3.0)))
        pos = scenes.lattice([20.0, 8.0, 20.0], [side] * 3, 1.9, 0.3, rng)[:n]
    else:  # everyone within reach of (almost) everyone: long rows, large halos
        pos = rng.uniform(0.0, dense, size=(n, 3)) + 20.0
    st = scenes.make_state(pos)
    if widths:
        st["kernel_width"] = (st["kernel_width"] * rng.uniform(0.7, 1.3, size=n)).astype(np.float32)
    return st


@pytest.mark.parametrize("capacity", [4096, 30_000])  # the 64 x 2 and the 128 x 1 tiles
@pytest.mark.parametrize("n,dense,maxn,widths", [
    (1, 0, 64, False), (63, 0, 64, False), (64, 0, 64, True), (129, 0, 96, False), (1000, 0, 128, True),
    (300, 2.0, 320, False),    # rows of about 300 entries: the pool
    (1500, 3.0, 1600, True),   # halos of more than 640 particles
    (500, 2.0, 70, False),     # rows cut at their capacity, six entries past the rewritten ones
])
def test_tiles_equal_direct_passes(capacity, n, dense, maxn, widths):
    from apbf_gb300.api import SubstepStages

    st = _state(n, dense, widths)
    fused, staged = (_ctx(st, capacity, maxn, 6) for _ in range(2))
    stages = SubstepStages(staged)
    fused.profile_enable(True)  # per-kernel launches, named
    for _ in range(2):
        fused.substep(1.0 / 240.0)
        stages.update(1.0 / 240.0)
    names, _ = fused.profile_read()
    assert "k_density_tiles" in names and "k_delta_tiles" in names
    a, _ = fused.download()
    b, _ = staged.download()
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
    assert fused.status().density_passes == staged.status().density_passes
    fused.close()
    staged.close()


def test_tiles_equal_direct_passes_empty_list():
    ctx = _ctx(_state(8, 0, False), 4096, 64, 6)
    ctx.set_lengths(0, 0)
    ctx.substep(1.0 / 240.0)
    assert ctx.check_status().density_passes == 6
    assert ctx.lengths()[0] == 0
    ctx.close()
