"""The neighbour rows where a particle's box spans from one cell of the grid to more than the
walk's table of cells holds, both in one warp, inside the grid and across its faces: against
brute force, entry by entry."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu

LO, HI = -4.0, 60.0


@pytest.mark.parametrize("capacity", [4096, 40_000, 120_000])  # 32, 16 and 8 threads per particle
@pytest.mark.parametrize("L,widths", [(6, (0.05, 0.6)), (6, (1.0, 2.2)), (6, (0.1, 7.0)), (7, (0.3, 3.0)), (3, (0.2, 9.0))])
@pytest.mark.parametrize("origin", [20.0, -9.0])
def test_rows_over_small_cells(capacity, L, widths, origin):
    from apbf_gb300.api import Context, neighborhood_green

    rng = np.random.default_rng(L)
    n = 500
    st = scenes.make_state(rng.uniform(0.0, 18.0, size=(n, 3)) + origin)
    st["kernel_width"] = (st["kernel_width"] * rng.uniform(*widths, size=n)).astype(np.float32)
    ctx = Context(particle_capacity=capacity, max_neighbors=n, max_log2res=L)
    ctx.upload(st)
    neighborhood_green().set_data(ctx).set_range_scale(1.0).set_position_range((LO,) * 3, (HI,) * 3, L).apply()
    ctx.check_status()
    g, _ = ctx.download()
    v = ctx.neighbors_view()
    cnt, idx = v["count"][:n].cpu().numpy(), v["index"][:, :n].cpu().numpy()
    p = g["position"][:, :3].astype(np.int64)
    lo, hi = round(LO * 2**18), round(HI * 2**18)
    cell = np.clip(((p - lo) << L) // (hi - lo), 0, (1 << L) - 1)
    R = np.floor(g["kernel_width"].astype(np.float64) * 2.0**18).astype(np.int64)
    d2 = ((p[:, None, :] - p[None, :, :]) ** 2).sum(2)
    for i in range(n):
        js = np.nonzero((d2[i] <= R[i] * R[i]) & (np.arange(n) != i))[0]
        js = js[np.lexsort((js, cell[js, 0], cell[js, 1], cell[js, 2]))]
        assert cnt[i] == len(js)
        assert np.array_equal(idx[:cnt[i], i], js), i
    ctx.close()
