"""What a user of this framework has it do, as cases that can be timed and compared.

Most cases are frames of a scene: the program writes its particle state from pinned host
memory into the lists (apbf_fluid_write), advances them by one or more substeps and takes
the resulting lists.  Every pass starts from the same state, so that a pass does the same
work however often it is repeated.  The states are taken from running scenes (after the
dam has broken, the drop has hit the pool, the stream has reached the slope), not from
their lattices.  Besides frames: the stage objects called one by one, batches of scenes,
the sort primitive and a training step of the warm-start network.
"""
from types import SimpleNamespace

import numpy as np
import torch

from apbf_gb300 import _native as N
from apbf_gb300 import scenes
from apbf_gb300.api import FLUID_FIELDS, Batch, Context, SubstepStages, algorithms
from apbf_gb300.warmstart import PARAMS, WarmStartNet

TARGET = 0.001      # mean density error a solve is run to
MAX_PASSES = 100    # passes a solve may take to it


def listed():
    return [
        # the smallest scene: a few thousand particles and the reference's four iterations;
        # launches and latency are all there is
        {"name": "dam_2k", "kind": "dam", "side": 13, "iterations": 4, "graph": 1, "presteps": 60, "substeps": 1},
        # the 32 768-particle dam break of the benchmark, solved to the error target
        {"name": "dam_32k", "kind": "dam", "side": 32, "iterations": 0, "graph": 2, "presteps": 35, "substeps": 2},
        # a port of the reference's scene code: the stage objects called one by one
        {"name": "stages_20k", "kind": "stages", "side": 27, "iterations": 4, "graph": 1, "presteps": 60,
         "substeps": 1},
        # the reference's default neighbour search (binary search) in the substep
        {"name": "binary_64k", "kind": "drop", "total": 64_019, "iterations": 4, "graph": 2, "search": "binary_search",
         "presteps": 60, "substeps": 1},
        # the learned warm start with projected passes, to the error target
        {"name": "learned_120k", "kind": "learned", "total": 119_771, "iterations": 0, "graph": 2, "presteps": 90,
         "substeps": 2},
        # the benchmark's water drop as a plain fluid at the scene's own six iterations
        {"name": "drop_250k", "kind": "drop", "total": 250_000, "iterations": 6, "graph": 1, "search": "green",
         "presteps": 110, "substeps": 2},
        # the same drop with split/merge and kernel widths spread across neighbours
        {"name": "spread_250k", "kind": "spread", "total": 250_000, "iterations": 0, "graph": 2, "presteps": 110,
         "substeps": 2},
        # the benchmark's headline scene: adaptive waterfall at about one million particles
        {"name": "waterfall_1m", "kind": "waterfall", "scale": 1.0, "iterations": 0, "graph": 2, "presteps": 300,
         "substeps": 2},
        # independent scenes of uneven sizes advanced together by one graph launch
        {"name": "batch_16", "kind": "batch", "scenes": 16, "lo": 4_000, "hi": 60_000, "iterations": 0, "presteps": 30,
         "substeps": 1},
        # the sort primitive on its own: a million 30-bit keys with their ids, an odd count
        {"name": "sort_1m", "kind": "sort", "count": 1_000_003, "bits": 30},
        # one minibatch of the warm start's training, at fit()'s batch size
        {"name": "train_32k", "kind": "train", "rows": 32_768},
    ]


def _log(rng, lo, hi):
    return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))


def draw(rng):
    kind = rng.choice(["dam", "dam", "stages", "drop", "drop", "learned", "spread", "waterfall", "waterfall", "batch",
                       "sort", "train"])
    c = {"kind": kind}
    if kind in ("dam", "stages"):
        c["side"] = int(round(_log(rng, 10.0, 60.0 if kind == "dam" else 48.0)))
        c["iterations"] = rng.choice([0, 2, 4, 5, 8]) if kind == "dam" else rng.choice([1, 3, 4, 6])
        c["graph"] = rng.choice([1, 2]) if kind == "dam" else 1
        c["presteps"] = rng.randint(20, 90)
        c["substeps"] = rng.randint(1, 3)
    elif kind in ("drop", "learned", "spread"):
        c["total"] = int(_log(rng, 8_000, 250_000 if kind == "spread" else 420_000))
        c["iterations"] = rng.choice([0, 4, 6, 7]) if kind == "drop" else 0
        c["graph"] = rng.choice([1, 2])
        if kind == "drop":
            c["search"] = rng.choice(["green", "green", "binary_search"])
        c["presteps"] = rng.randint(40, 110)
        c["substeps"] = rng.randint(1, 2)
    elif kind == "waterfall":
        c.update(scale=round(rng.uniform(0.3, 0.95), 3), iterations=0, graph=2, presteps=rng.randint(200, 300),
                 substeps=rng.randint(1, 2))
    elif kind == "batch":
        lo = int(_log(rng, 2_000, 8_000))
        c.update(scenes=rng.randint(4, 20), lo=lo, hi=int(lo * rng.uniform(3.0, 12.0)), iterations=rng.choice([0, 4]),
                 presteps=rng.randint(10, 40), substeps=1)
    elif kind == "sort":
        c.update(count=int(_log(rng, 1_000, 4_000_000)), bits=rng.randint(5, 32))
    else:
        c.update(rows=int(_log(rng, 500, 260_000)))
    return c


# ---------------------------------------------------------------------------- scenes


def _waterfall(scale, seed):
    """The benchmark's waterfall: at scale 1, a million particles after 300 substeps."""
    return scenes.waterfall(initial=int(384_000 * scale ** 3), seed=seed, scale=scale,
                            per_substep=max(50, int(round(2000 * scale ** 2))))


def _net_params(seed):
    """Parameters of a warm-start network as a program loads them: hidden layers at their
    usual scale around a path that carries the plain lambda, an over-relaxation bound
    of 3 and the plain lambda below 16 neighbours."""
    g = np.random.default_rng(1000 + seed)
    p = np.zeros(PARAMS, np.float32)
    p[8:15] = (0.05, 2.0, 0.5, 1.0, 0.05, 0.2, 0.2)  # 1 / sigma of the seven features
    w1 = (g.standard_normal((64, 8)) * 0.3).astype(np.float32)
    w1[:, 7] = 0.0
    w1[0] = 0.0
    w1[0, 3] = -1.0  # relu(-lambda)
    w2 = (g.standard_normal((64, 64)) * 0.05).astype(np.float32)
    w2[0] = 0.0
    w2[0, 0] = 1.0
    w3 = (g.standard_normal(64) * 0.01).astype(np.float32)
    w3[0] = -1.6
    p[16:528] = w1.ravel()
    p[592:4688] = w2.ravel()
    p[4752:4816] = w3
    p[4817] = 1.0   # y_scale
    p[4819] = 3.0   # omega_max
    p[4820] = 16.0  # min_neighbors
    return torch.from_numpy(p).cuda()


def _context(spec, case, max_neighbors, settings=None, warm=0, capacity=None, seed=0):
    ctx = Context(particle_capacity=capacity or int(spec.n * 1.25) + 1024, max_neighbors=max_neighbors,
                  max_log2res=max(spec.log2res, 3))
    it = case["iterations"]
    ctx.set_settings(basic_pbf=1 if spec.basic_pbf else 0, solver_iterations=it or MAX_PASSES,
                     density_error_target=0.0 if it else TARGET, **(settings or {}))
    ctx.load_scene(spec)
    ctx.set_solve_graph(case.get("graph", 2))
    if warm & N.WARM_LEARNED:
        ctx.mlp_load(_net_params(seed))
    if warm:
        ctx.set_warm_start(warm)
    return ctx


def _host_lists(rows):
    """Pinned host arrays of the particle lists, as fluid_write and fluid_read take them."""
    return {k: torch.zeros((rows, c) if c > 1 else (rows,), dtype=d).pin_memory() for k, (d, c) in FLUID_FIELDS.items()}


def _frame_state(spec, ctx, presteps, stages=None):
    """The scene after `presteps` substeps: its lists in pinned host memory, its transfers on
    the device."""
    for _ in range(presteps):
        ctx.substep(spec.dt)
    ctx.check_status()
    n, nt = ctx.lengths()
    host, count = _host_lists(n), torch.zeros(1, dtype=torch.int32).pin_memory()
    host["lambda_prev"] = torch.zeros(n, dtype=torch.float32).pin_memory()
    ctx.fluid_read(host, n, count)
    tv = ctx.transfers_view()
    transfers = {k: tv[k][:nt].clone() for k in ("source", "target", "time_left")}
    transfers["length"] = tv["length"].clone()
    torch.cuda.synchronize()
    adaptive = not spec.basic_pbf
    return SimpleNamespace(ctx=ctx, host=host, n=n, transfers=transfers, dt=spec.dt, adaptive=adaptive, stages=stages,
                           count=count, rows=0, result=_host_lists(ctx.capacity) if adaptive else None)


def _scene(case, seed):
    kind, warm = case["kind"], 0
    if kind in ("dam", "stages"):
        spec = scenes.dam_break(n_side=case["side"], seed=seed)
        ctx = _context(spec, case, 160)
    elif kind in ("drop", "learned"):
        spec = scenes.water_drop(total=case["total"], seed=seed, basic_pbf=True)
        warm = N.WARM_LEARNED | N.WARM_PROJECTED if kind == "learned" else 0
        ctx = _context(spec, case, 192, warm=warm, seed=seed)
        if case.get("search") == "binary_search":
            ctx.set_neighborhood_search("binary_search")
    elif kind == "spread":
        spec = scenes.water_drop(total=case["total"], seed=seed, basic_pbf=False)
        ctx = _context(spec, case, 2048, {"base_kernel_width_on_boundary_distance": 0,
                                          "target_radius_scale_factor": 0.025})
    else:
        spec = _waterfall(case["scale"], seed)
        ctx = _context(spec, case, 256, warm=N.WARM_PROJECTED, capacity=int(spec.meta["capacity"] * 1.15))
    return spec, ctx


def _batch_specs(case, seed):
    """A table of seeded scenes, as the benchmark's batch: sizes log-uniform, every other
    scene a dam break, the rest water drops, half of them adaptive."""
    rng = np.random.default_rng(7)
    counts = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), size=case["scenes"])).astype(int)
    out = []
    for k, c in enumerate(counts):
        if k % 2 == 0:
            out.append(scenes.dam_break(n_side=max(8, int(round(c ** (1.0 / 3.0)))), seed=seed * 64 + k))
        else:
            out.append(scenes.water_drop(total=int(c), seed=seed * 64 + k, basic_pbf=k % 4 == 1))
    return out


# ---------------------------------------------------------------------------- training


def _train_data(rows, seed):
    """A minibatch as the recorded samples look: counts, density ratios, widths, lambdas,
    and normalised targets that follow the plain lambda."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.randn((rows, 8), device="cuda", generator=g)
    x = torch.zeros_like(r)
    x[:, 0] = (28.0 + 9.0 * r[:, 0]).clamp_(0.0, 120.0).round_()
    x[:, 1] = 0.08 * r[:, 1]
    x[:, 2] = 4.0 + 0.5 * r[:, 2]
    x[:, 3] = -0.4 * x[:, 1] / 0.08 + 0.1 * r[:, 3]
    x[:, 4] = 8.0 * r[:, 4]
    x[:, 5] = -r[:, 5].abs()
    x[:, 6] = 0.5 * x[:, 5] + 0.1 * r[:, 6]
    t = 1.5 * x[:, 3].clamp(max=0.0) + 0.4 * x[:, 5]
    return x.contiguous(), t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        n, bits = case["count"], case["bits"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        keys = torch.randint(0, 1 << bits, (n,), device="cuda", generator=g).to(torch.int32)
        return SimpleNamespace(case=case, ctx=Context(particle_capacity=n, max_neighbors=8, max_log2res=3), keys=keys,
                               ids=torch.arange(n, dtype=torch.int32, device="cuda"),
                               count=torch.tensor([n], dtype=torch.int32, device="cuda"),
                               out_keys=torch.empty_like(keys), out_ids=torch.empty_like(keys),
                               bound=(1 << bits) - 1)
    if kind == "train":
        net = WarmStartNet(seed=seed)
        x, t = _train_data(case["rows"], seed)
        net.set_normalization(x, t)
        return SimpleNamespace(case=case, net=net, x=x, t=net.normalise_targets(t))
    if kind == "batch":
        parts = []
        for spec in _batch_specs(case, seed):
            ctx = _context(spec, case, (160 if spec.name == "dam_break" else 192) if spec.basic_pbf else 256)
            parts.append(_frame_state(spec, ctx, case["presteps"]))
        return SimpleNamespace(case=case, parts=parts, batch=Batch([p.ctx for p in parts]), dt=1.0 / 240.0)
    spec, ctx = _scene(case, seed)
    st = _frame_state(spec, ctx, case["presteps"])
    if kind == "stages":
        st.stages = SubstepStages(ctx)
    st.case = case
    return st


# ---------------------------------------------------------------------------- passes


def _write(p):
    p.ctx.fluid_write(p.host, p.n)
    if p.adaptive:  # split/merge transfers under way
        tv = p.ctx.transfers_view()
        nt = p.transfers["source"].numel()
        for k in ("source", "target", "time_left"):
            if nt:
                tv[k][:nt].copy_(p.transfers[k])
        tv["length"].copy_(p.transfers["length"])


def _xyz(lists):
    """position's and pos_backup's fourth words are the library's."""
    return {k: v[:, :3] if k in ("position", "pos_backup") else v for k, v in lists.items()}


def _lists(p):
    """The lists after a frame.  Of a scene whose count stays: the device lists (they alias
    the context's memory, so each holds on to it).  Of an adaptive scene: its count, then
    that many particles read back into host arrays of the lists' capacity."""
    if not p.adaptive:
        v = p.ctx.fluid_view()
        out = _xyz({k: v[k][:p.n] for k in FLUID_FIELDS})
        for t in out.values():
            t.context = p.ctx
        return out
    n, nt = p.ctx.lengths()
    p.ctx.fluid_read(p.result, n, p.count)
    for a in p.result.values():
        a[n:p.rows].zero_()  # slots a longer list left
    p.rows = n
    torch.cuda.current_stream().synchronize()
    return {**_xyz(p.result), "particles": n, "transfers": nt}


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "sort":
        algorithms.sort(state.ctx, state.keys, state.ids, state.count, state.keys.numel(), state.out_keys,
                        state.out_ids, state.bound)
        return {"keys": state.out_keys, "ids": state.out_ids}
    if kind == "train":
        net = state.net
        net.train_step(state.x, state.t, 2e-3, over_weight=8.0)
        return {"params": net.params, "m": net.m, "v": net.v, "loss": net.loss}
    if kind == "batch":
        for p in state.parts:
            _write(p)
        for _ in range(case["substeps"]):
            state.batch.substep(state.dt)
        out = []
        for p in state.parts:
            r = _lists(p)
            out.append([r["position"], r["velocity"], r["boundariness"]])
        return out
    _write(state)
    for _ in range(case["substeps"]):
        if state.stages is not None:
            state.stages.update(state.dt)
        else:
            state.ctx.substep(state.dt)
    return _lists(state)


# ---------------------------------------------------------------------------- work, exact values

# directed pairs per particle and passes a substep of these scenes needs to the target
_PAIRS = {"dam": 30, "stages": 30, "drop": 30, "learned": 30, "spread": 30, "waterfall": 20, "batch": 30}
_PASSES = {"dam": 20, "drop": 20, "learned": 14, "spread": 30, "waterfall": 20, "batch": 20}
_PAIR_FLOPS = 22 + 14  # kernel, gradient and sums of a pair; its position term


def work(case):
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 16 * case["count"], "flops": 0}
    if kind == "train":
        # forward, both backward products; features, targets and the optimiser's state
        return {"bytes": 36 * case["rows"] + 24 * PARAMS, "flops": 3 * 2 * case["rows"] * (7 * 64 + 64 * 64 + 64)}
    if kind in ("dam", "stages"):
        n = case["side"] ** 3
    elif kind == "batch":
        n = case["scenes"] * int((case["hi"] - case["lo"]) / np.log(case["hi"] / case["lo"]))
    elif kind == "waterfall":
        n = int(384_000 * case["scale"] ** 3 + 2000 * case["scale"] ** 2 * case["presteps"])
    else:
        n = case["total"]
    passes = case["iterations"] or _PASSES[kind]
    return {"bytes": 2 * 84 * n * case["substeps"],
            "flops": _PAIR_FLOPS * _PAIRS[kind] * n * passes * case["substeps"]}


def _exact_train(case, seed):
    """One Adam step of the network in 64 bits."""
    x, t = _train_data(case["rows"], seed)
    xu = x[:, :7].double()
    mu, sd = xu.mean(0), xu.std(0)
    ys, ym = t.double().std(), t.double().mean()
    rng = np.random.default_rng(seed)  # WarmStartNet's initial weights
    w1 = (rng.standard_normal((64, 8)) * np.sqrt(2.0 / 7)).astype(np.float32)
    w1[:, 7] = 0.0
    w2 = (rng.standard_normal((64, 64)) * np.sqrt(2.0 / 64)).astype(np.float32)
    w3 = (rng.standard_normal(64) * np.sqrt(1.0 / 64) * 0.1).astype(np.float32)
    p = torch.zeros(PARAMS, dtype=torch.float64)
    p[0:7], p[8:15] = mu.float().double().cpu(), (1.0 / sd).float().double().cpu()
    p[16:528], p[592:4688] = torch.from_numpy(w1.ravel()).double(), torch.from_numpy(w2.ravel()).double()
    p[4752:4816] = torch.from_numpy(w3).double()
    p[4817], p[4818] = ys.float().double().cpu(), ym.float().double().cpu()
    p = p.cuda()
    tn = (t.double() - p[4818]) / p[4817]
    q = p.clone().requires_grad_(True)
    xn = (x.double() - q[0:8].detach()) * q[8:16].detach()
    h1 = torch.relu(xn @ q[16:528].view(64, 8).T + q[528:592])
    h2 = torch.relu(h1 @ q[592:4688].view(64, 64).T + q[4688:4752])
    e = h2 @ q[4752:4816] + q[4816] - tn
    loss = (torch.where(e < 0, 8.0, 1.0) * e * e).mean()
    (g,) = torch.autograd.grad(loss, q)
    g[:16], g[4817:] = 0.0, 0.0
    m, v = 0.1 * g, 0.001 * g * g
    params = p - 2e-3 * g / (g.abs() + 1e-8)
    params[:16], params[4817:] = p[:16], p[4817:]
    return {"params": params, "m": m, "v": v, "loss": loss.detach().reshape(1)}


def exact(case, seed):
    """The simulation's state is whole numbers and what follows from them; the training
    step is the one with a value in 64 bits."""
    return _exact_train(case, seed) if case["kind"] == "train" else None
