"""The neighbour rows entry by entry: every neighbour within the search radius, cells in z,
y, x order and particles in list order within a cell, for each number of threads the walk
gives a particle (chosen by the list's capacity); rows longer than the walk stages, rows
cut at their capacity, particles outside the grid."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu

LO, HI, L = -4.0, 60.0, 4


@pytest.mark.parametrize("capacity", [4096, 40_000, 120_000])  # 32, 16 and 8 threads per particle
@pytest.mark.parametrize("n,spread,maxn", [(1, 10.0, 32), (33, 6.0, 64), (700, 14.0, 256), (260, 2.0, 300),
                                           (200, 2.0, 40), (500, 70.0, 64)])
def test_rows_in_walk_order(capacity, n, spread, maxn):
    from apbf_gb300.api import Context, neighborhood_green

    rng = np.random.default_rng(n)
    st = scenes.make_state(rng.uniform(0.0, spread, size=(n, 3)) + (-6.0 if spread > 60.0 else 20.0))
    st["kernel_width"] = (st["kernel_width"] * rng.uniform(0.8, 1.2, size=n)).astype(np.float32)
    ctx = Context(particle_capacity=capacity, max_neighbors=maxn, max_log2res=L)
    ctx.upload(st)
    neighborhood_green().set_data(ctx).set_range_scale(1.0).set_position_range((LO,) * 3, (HI,) * 3, L).apply()
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
        assert cnt[i] == min(len(js), maxn)
        assert np.array_equal(idx[:cnt[i], i], js[:maxn]), i
    ctx.close()
