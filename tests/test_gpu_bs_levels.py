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


@pytest.mark.parametrize("capacity", [4096, 30_000, 300_000])  # the three forms of the sort
@pytest.mark.parametrize("low,high", [(0, 1 << 18), (-(1 << 20), 1 << 20), (-(1 << 31), (1 << 31) - 1),
                                      (1 << 24, (1 << 24) + 9), (77, 77)])
def test_bs_order_of_the_codes(capacity, low, high):
    """Stable order of the 96-bit codes: digits that all particles share, signs mixed, many
    equal codes, all equal; three searches of one context."""
    from apbf_gb300.api import Context, neighborhood_binary_search

    rng = np.random.default_rng(11)
    n = 3000
    st = scenes.make_state(rng.uniform(0.0, 14.0, size=(n, 3)))
    ctx = Context(particle_capacity=capacity, max_neighbors=128, max_log2res=3)
    for lo, hi in ((low, high), (-5, 1 << 22), (low, high)):
        p = rng.integers(lo, hi + 1, size=(n, 3))
        p[n // 2:] = p[rng.integers(0, n // 2, size=n - n // 2)]
        st["position"][:, :3] = p.astype(np.uint32).view(np.int32)
        st["kernel_width"] = np.full(n, -1.0, np.float32)  # no neighbours
        st["velocity"][:, 0] = np.arange(n, dtype=np.float32)  # the list order
        ctx.upload(st)
        neighborhood_binary_search().set_data(ctx).set_range_scale(1.0).apply()
        g, _ = ctx.download()
        u = p.astype(np.uint32)
        code = [sum(((int(v[a]) >> b) & 1) << (3 * b + a) for b in range(32) for a in range(3)) for v in u]
        want = sorted(range(n), key=lambda i: code[i])  # (stable)
        assert np.array_equal(g["velocity"][:, 0].astype(np.int64), np.array(want))
    ctx.close()
