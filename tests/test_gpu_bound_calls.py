"""Calls on lists bound by the caller go by the caller's length words, which it may have set
since the last call: the binary search, the collision and glue stages, the position codes, the
host-list copies, batches and the particle-info files, against a context with lists of its own."""
import numpy as np
import pytest
import torch

from apbf_gb300 import scenes

pytestmark = pytest.mark.gpu


def _pair(n_side=10):
    """A context with its own lists and one on the caller's, the same state in both; the
    caller's length words are written after the bind."""
    from apbf_gb300.api import FLUID_FIELDS, CallerLists, Context

    spec = scenes.dam_break(n_side=n_side)
    n = spec.n
    own, bound = (Context(particle_capacity=n + 300, max_neighbors=128, max_log2res=max(spec.log2res, 3))
                  for _ in range(2))
    for ctx in (own, bound):
        ctx.set_settings(basic_pbf=1, solver_iterations=4)
        ctx.set_scene(spec.grid_min, spec.grid_max, spec.log2res, spec.acceleration)
        ctx.set_boxes(spec.box_min, spec.box_max)
    own.upload(spec.state)
    lists = CallerLists.for_context(bound)
    bound.bind_lists(lists)
    for name, (dt, comps) in FLUID_FIELDS.items():
        a = np.ascontiguousarray(spec.state[name]).view(np.int32 if dt == torch.int32 else np.float32)
        lists.fluid[0][name][:n].copy_(torch.from_numpy(a.reshape((n, comps) if comps > 1 else (n,))))
    lists.len_particles.fill_(n)
    torch.cuda.synchronize()
    return spec, own, bound, lists


def _same(own, bound, lists):
    torch.cuda.synchronize()
    assert own.lengths() == bound.lengths()
    assert int(lists.len_particles.item()) == own.lengths()[0]
    a, b = own.download()[0], bound.download()[0]
    for k in a:
        assert np.array_equal(a[k], b[k]), k


def test_binary_search_and_collisions():
    from apbf_gb300.api import inter_particle_collision, neighborhood_binary_search, sphere_collision

    spec, own, bound, lists = _pair()
    for ctx in (own, bound):
        neighborhood_binary_search().set_data(ctx).set_range_scale(1.0).apply()
    _same(own, bound, lists)
    rows = own.download_rows()
    assert sum(len(r) for r in rows) > 0
    for a, b in zip(rows, bound.download_rows()):
        assert np.array_equal(a, b)
    for ctx in (own, bound):
        sphere_collision().set_data(ctx).set_sphere((20.0, 5.0, 20.0), 9.0, False).apply()
        inter_particle_collision().set_data(ctx).apply()
    _same(own, bound, lists)
    assert torch.equal(own.position_codes(), bound.position_codes())


def test_sphere_collision_first():
    from apbf_gb300.api import sphere_collision

    spec, own, bound, lists = _pair()
    for ctx in (own, bound):
        sphere_collision().set_data(ctx).set_sphere((10.0, 10.0, 10.0), 9.0, False).apply()
    _same(own, bound, lists)
    assert not np.array_equal(own.download()[0]["position"][:, :3], spec.state["position"][:, :3])


def test_host_lists():
    from apbf_gb300.api import FLUID_FIELDS

    spec, own, bound, lists = _pair()
    n = spec.n

    def host():
        return {k: torch.zeros((n, c) if c > 1 else (n,), dtype=d).pin_memory() for k, (d, c) in FLUID_FIELDS.items()}

    got, count = host(), torch.zeros(1, dtype=torch.int32).pin_memory()
    bound.fluid_read(got, n, count)
    torch.cuda.synchronize()
    assert int(count[0]) == n
    for pinned in (True, False):
        part = n - (100 if pinned else 57)
        src = {k: (v if pinned else v.clone()) for k, v in got.items()}
        for ctx in (own, bound):
            ctx.fluid_write(src, part)
            ctx.substep(spec.dt)
        _same(own, bound, lists)
        assert own.lengths()[0] == part


def test_batch():
    from apbf_gb300.api import Batch

    spec, own, bound, lists = _pair()
    batch = Batch([bound])
    for k in range(6):
        if k == 3:  # the caller takes particles off its list's end
            torch.cuda.synchronize()
            lists.len_particles.fill_(spec.n - 120)
            own.fluid_write({}, spec.n - 120)
        own.substep(spec.dt)
        batch.substep(spec.dt)
    _same(own, bound, lists)
    batch.close()


def test_particle_info_files(tmp_path):
    spec, own, bound, lists = _pair()
    from apbf_gb300.api import neighborhood_green

    for name, ctx in (("own", own), ("bound", bound)):
        neighborhood_green().set_data(ctx).set_range_scale(1.0).set_position_range(
            spec.grid_min, spec.grid_max, spec.log2res).apply()
    torch.cuda.synchronize()
    lists.len_particles.fill_(spec.n - 30)
    own.fluid_write({}, spec.n - 30)
    for name, ctx in (("own", own), ("bound", bound)):
        (tmp_path / name).mkdir()
        ctx.save_particle_info(str(tmp_path / name))
    files = sorted(p.name for p in (tmp_path / "own").iterdir())
    assert files and files == sorted(p.name for p in (tmp_path / "bound").iterdir())
    for f in files:
        assert (tmp_path / "own" / f).read_bytes() == (tmp_path / "bound" / f).read_bytes(), f
