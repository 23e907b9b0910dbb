"""The binary-search rows against brute force where the cells come from the table (all
radii of one level) and where they are searched (several levels, radii below the table's
levels, an invalid width), for each number of threads per particle; cells that wrap around
the ends of the 32-bit range."""
import numpy as np
import pytest

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", [4096, 30_000, 60_000])  # 32, 16 and 8 threads per particle
@pytest.mark.parametrize("kind", ["equal", "one_level", "levels", "tiny", "nan", "wrap", "dense"])
def test_bs_rows_against_brute_force(capacity, kind):
    from apbf_gb300.api import Context, neighborhood_binary_search

    rng = np.random.default_rng(5)
    n = 600
    side = 2.0 if kind == "dense" else 14.0
    st = scenes.make_state(rng.uniform(0.0, side, size=(n, 3)) + 20.0)
    w = st["kernel_width"].astype(np.float64)
    if kind == "one_level":
        w *= rng.uniform(0.76, 0.99, size=n)
    elif kind == "levels":
        w *= rng.uniform(0.2, 2.5, size=n)
    elif kind == "tiny":  # radii of at most 900 units
        st["position"][:, :3] = (rng.integers(0, 6000, size=(n, 3)) + 5_000_000).astype(np.int32)
        w[:] = 900.0 / 2**18
    elif kind == "nan":
        w[7] = np.nan
    elif kind == "wrap":
        st["position"][:, 0] = (rng.integers(-(1 << 21), 1 << 21, size=n) + (1 << 31)).astype(np.uint32).view(np.int32)
    st["kernel_width"] = w.astype(np.float32)
    ctx = Context(particle_capacity=capacity, max_neighbors=640, max_log2res=3)
    ctx.upload(st)
    neighborhood_binary_search().set_data(ctx).set_range_scale(1.0).apply()
    g, _ = ctx.download()
    rows = ctx.download_rows()
    p = g["position"][:, :3].astype(np.int64)
    kw = g["kernel_width"].astype(np.float64)
    R = np.where(np.isnan(kw), -1, np.floor(np.nan_to_num(kw) * 2.0**18)).astype(np.int64)
    d = np.minimum(np.abs(p[:, None, :] - p[None, :, :]), 1 << 30)  # (radii are below 2^30: no overflow)
    d2 = (d ** 2).sum(2)
    for i in range(n):
        js = np.nonzero((d2[i] <= R[i] * R[i]) & (R[i] >= 0) & (np.arange(n) != i))[0]
        assert np.array_equal(rows[i], js), i
    ctx.close()
