"""The stable sort at the sizes where its form changes (one block for 4 096 and 16 384
pairs, tiles with a look-back up to 2^18, counted tiles above) and at the edges of its
tiles, against numpy's stable order; a device count below the capacity; sorting in place."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bits", [(1, 32), (31, 8), (4095, 21), (4096, 32), (4097, 13), (16_384, 30), (16_385, 32),
                                    (18_432, 24), ((1 << 18), 32), ((1 << 18) + 1, 32), (300_001, 5), (65_536 * 5, 21)])
@pytest.mark.parametrize("in_place", [False, True])
def test_sort_forms(n, bits, in_place):
    from apbf_gb300.api import Context, algorithms

    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, size=n, dtype=np.uint64).astype(np.uint32)
    k[: n // 3] = np.sort(k[: n // 3])
    ctx = Context(particle_capacity=n, max_neighbors=8, max_log2res=3)
    keys = torch.from_numpy(k.view(np.int32)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda") * 3
    m = n - n // 7  # the device's count
    cnt = torch.tensor([m], dtype=torch.int32, device="cuda")
    ok, ov = (keys, vals) if in_place else (torch.full_like(keys, -1), torch.full_like(vals, -1))
    tail = (ok[m:].clone(), ov[m:].clone())
    algorithms.sort(ctx, keys, vals, cnt, n, ok, ov, (1 << bits) - 1)
    torch.cuda.synchronize()
    ctx.check_status()
    order = np.argsort(k[:m], kind="stable")
    assert np.array_equal(ov[:m].cpu().numpy(), order * 3)
    assert np.array_equal(ok[:m].cpu().numpy().view(np.uint32), k[:m][order])
    assert torch.equal(ok[m:], tail[0]) and torch.equal(ov[m:], tail[1])  # nothing past the count
    ctx.close()


@pytest.mark.parametrize("n", [1, 16_384, 16_385, 20_481, 1 << 18, (1 << 18) + 1])
@pytest.mark.parametrize("spread", [0x00000000, 0x000000ff, 0x00ff0000, 0xff0000ff, 0x80000000, 0x00ffff00])
def test_sort_of_shared_digits(n, spread):
    """Keys that differ in some of their digits only; the others are the same in all keys."""
    from apbf_gb300.api import Context, algorithms

    rng = np.random.default_rng(n)
    k = (rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32) & np.uint32(spread)) | np.uint32(
        0x5a3c96e1 & ~spread)
    ctx = Context(particle_capacity=n, max_neighbors=8, max_log2res=3)
    keys = torch.from_numpy(k.view(np.int32)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    m = n - n // 9
    cnt = torch.tensor([m], dtype=torch.int32, device="cuda")
    ok, ov = torch.full_like(keys, -1), torch.full_like(vals, -1)
    algorithms.sort(ctx, keys, vals, cnt, n, ok, ov, (1 << 32) - 1)
    torch.cuda.synchronize()
    ctx.check_status()
    order = np.argsort(k[:m], kind="stable")
    assert np.array_equal(ov[:m].cpu().numpy(), order)
    assert np.array_equal(ok[:m].cpu().numpy().view(np.uint32), k[:m][order])
    assert bool((ok[m:] == -1).all()) and bool((ov[m:] == -1).all())
    ctx.close()
