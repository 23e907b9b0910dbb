"""The adaptive stages on rows of more than 64 entries, against the oracle: a few of them
among short ones (walked by whole warps), most of them long (each thread its own), and
mixtures; lists that end inside a warp."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def _state(n, kind):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    st = scenes.make_state(scenes.lattice([20.0] * 3, [side] * 3, 1.9, 0.4, rng)[:n])
    share = {"few": 0.02, "some": 0.15, "most": 0.9, "all": 1.0}[kind]
    wide = rng.uniform(size=n) < share
    factor = np.where(wide, rng.uniform(1.5, 2.6, size=n), rng.uniform(0.6, 0.9, size=n))
    st["kernel_width"] = (st["kernel_width"] * factor).astype(np.float32)
    st["target_radius"] = rng.uniform(1.0, 2.0, size=n).astype(np.float32)
    st["boundary_distance"] = rng.integers(0, 40 << 18, size=n).astype(np.uint32)
    st["boundariness"] = rng.uniform(0.0, 1.2, size=n).astype(np.float32)
    return st


def _searched(st, **settings):
    from apbf_gb300.api import Context, neighborhood_green

    n = st["radius"].size
    ctx = Context(particle_capacity=n + 64, max_neighbors=1100, max_log2res=4)
    ctx.set_settings(**settings)
    ctx.upload(st)
    neighborhood_green().set_data(ctx).set_range_scale(1.0).set_position_range((0.0,) * 3, (80.0,) * 3, 4).apply()
    before, _ = ctx.download()
    return ctx, before, ctx.download_rows()


@pytest.mark.parametrize("n", [33, 700, 1000])
@pytest.mark.parametrize("kind", ["few", "some", "most", "all"])
def test_spread_and_update_on_long_rows(orc, n, kind):
    from apbf_gb300.api import spread_kernel_width, update_transfers

    st = _state(n, kind)
    ctx, before, rows = _searched(st, base_kernel_width_on_boundary_distance=0)
    long_rows = sum(len(r) > 64 for r in rows)
    assert n < 100 or 0 < long_rows and (kind in ("most", "all")) == (2 * long_rows > n)
    spread_kernel_width().set_data(ctx).apply()
    ctx.check_status()
    g, _ = ctx.download()
    g_rows = ctx.download_rows()
    fs = orc.FluidState(before)
    orc.set_rows(fs, rows)
    orc.spread_kernel_width(fs, orc.settings_from(ctx.settings))
    assert np.array_equal(g["kernel_width"], fs.state()["kernel_width"])
    for full, got, want in zip(rows, g_rows, fs.rows()):
        assert np.array_equal(got, full[np.isin(full, want)])  # pruned, the order kept
    ctx.close()

    ctx, before, rows = _searched(st, merge=0, split=0)
    update_transfers().set_data(ctx).apply()
    ctx.check_status()
    g, _ = ctx.download()
    fs = orc.FluidState(before)
    orc.set_rows(fs, rows)
    orc.update_transfers(fs, orc.settings_from(ctx.settings))
    o = fs.state()
    for k in ("boundary_distance", "boundariness", "target_radius"):
        assert np.array_equal(g[k], o[k]), k
    ctx.close()
