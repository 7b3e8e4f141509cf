"""What a user of this library has it do, as cases that can be timed and compared.

  listed()             the cases, plain dicts
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  the state a program holds before the call, on the GPU
  run(state)           one pass through the public entry points, and its outputs
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    the outputs in 64 bits, in plain torch, without the library

Positions are returned in 64 bits.  A run in the single-precision mode keeps
its other fields as float32, which is what its sums carry (the learned stepper
keeps its velocities that way too); a run in double precision keeps all in 64
bits.
"""
import math

import numpy as np
import torch

from sources_b200 import Solver, ensemble, learn, scenes
from sources_b200.abi import SPHG_FP32, SPHG_FP64

DEV = "cuda"
FULL = ("x", "vx", "dvx", "av", "rho", "drho", "p", "c", "vof", "dvof", "vof2", "sxx", "sxy", "syy", "dsxx", "dsxy",
        "dsyy", "dp", "vcc")


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # The reference's own program on the small water configuration (0.2 x 0.4 m column, dx 5 mm): state in, one
        # call and one statistics read a step, state out.  Launches and latency are all there is.
        dict(name="dam_break_4k_host_loop", do="host", kind="dam_break", col_w=40, col_h=80, box_w=160, dx=0.005,
             fp=64, skf=1, steps=20, per_call=1),
        # The small soil configuration (0.2 x 0.1 m column, dx 2 mm), a stretch between two saves in one call.
        dict(name="granular_7k_run", do="host", kind="granular", col_w=100, col_h=50, box_w=500, dx=0.002, fp=32,
             skf=1, steps=60, per_call=60),
        # A host that keeps its own integrator and asks for the right-hand side only, every array handed over.
        dict(name="two_phase_58k_rhs", do="rhs", kind="two_phase", col_w=103, col_h=51, box_w=521, water_h=97,
             dx=0.004, fp=64, skf=1),
        # An ordinary submerged collapse of odd sizes with the reference's default kernel function (Wendland) and
        # the quadratic drag.
        dict(name="two_phase_150k_steps", do="steps", kind="two_phase", col_w=331, col_h=87, box_w=827, water_h=153,
             dx=0.003, fp=32, skf=4, drag=4.0e4, steps=10),
        # The full-size two-phase workload in its benchmark precision, and in the parity precision.
        dict(name="two_phase_912k_steps", do="steps", kind="two_phase", col_w=500, col_h=200, box_w=2000, water_h=400,
             dx=0.002, fp=32, skf=1, drag=0.0, steps=10),
        dict(name="two_phase_912k_fp64_steps", do="steps", kind="two_phase", col_w=500, col_h=200, box_w=2000,
             water_h=400, dx=0.002, fp=64, skf=1, drag=0.0, steps=10),
        # A large water-only dam-break and a large dry column: the single-phase steps.
        dict(name="dam_break_330k_steps", do="steps", kind="dam_break", col_w=523, col_h=617, box_w=1301, dx=0.002,
             fp=32, skf=1, steps=10),
        dict(name="granular_190k_steps", do="steps", kind="granular", col_w=613, col_h=307, box_w=1207, dx=0.002,
             fp=32, skf=1, steps=10),
        # The batched ensemble: many uneven scenes of the three kinds, one graph a step.
        dict(name="ensemble_40_steps", do="ensemble", scenes=40, steps=10),
        # The learned stepper: its edge layer alone at a held-out group's size, the whole network with its graph
        # search (inference), and one training iteration (graph, forward, loss, backward, Adam).
        dict(name="edge_layer_1m7", do="edge", kind="two_phase", nodes=91000),
        dict(name="learned_forward_92k", do="forward", kind="two_phase", nodes=92000),
        dict(name="learned_train_24k", do="train", kind="dam_break", nodes=24000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(("host", "host", "rhs", "steps", "steps", "steps", "ensemble", "edge", "forward", "train"))
    if do == "ensemble":
        return dict(do=do, scenes=rng.randint(3, 40), steps=10, first=rng.randint(0, 200))
    if do in ("edge", "forward", "train"):
        return dict(do=do, kind=rng.choice(("dam_break", "granular", "two_phase")),
                    nodes=_log(rng, 2000, 24000 if do == "train" else 90000))
    kind = rng.choice(("dam_break", "granular", "two_phase"))
    n = _log(rng, 2000, 60000 if do != "steps" else 600000)
    aspect = rng.uniform(0.5, 2.0)
    c = dict(do=do, kind=kind, dx=rng.choice((0.002, 0.003, 0.004, 0.005)), fp=rng.choice((32, 64)),
             skf=rng.choice((1, 4)))
    if do == "rhs":
        c["fp"] = 64
    if kind == "two_phase":
        n = max(n // 2, 1000)
        high = max(8, int(math.sqrt(n * 0.3)))
        c["water_h"], c["box_w"] = high, max(12, n // high)
        c["col_w"], c["col_h"] = max(4, int(c["box_w"] * rng.uniform(0.2, 0.5))), max(4, int(high * rng.uniform(0.3, 0.7)))
        c["drag"] = rng.choice((0.0, 4.0e4))
    else:
        c["col_w"] = max(6, int(math.sqrt(n / aspect)))
        c["col_h"] = max(6, n // c["col_w"])
        c["box_w"] = int(c["col_w"] * rng.uniform(1.5, 3.0))
    if do == "host":
        c["steps"] = rng.randint(5, 30)
        c["per_call"] = rng.choice((1, c["steps"]))
    elif do == "steps":
        c["steps"] = 10
    return c


# ------------------------------------------------------------------ inputs

def _rng(seed):
    return np.random.default_rng(int(seed))


def _scene(c, seed):
    """The scene's lattice as a collapse has it under way: every real particle displaced a little, in a smooth swirl
    of a few tenths of a metre a second with a little noise on it."""
    dx, fp = c["dx"], SPHG_FP32 if c["fp"] == 32 else SPHG_FP64
    if c["kind"] == "dam_break":
        s = scenes.dam_break(width=c["col_w"] * dx, height=c["col_h"] * dx, tank_w=c["box_w"] * dx,
                             tank_h=1.5 * c["col_h"] * dx, dx=dx, skf=c["skf"], precision=fp)
    elif c["kind"] == "granular":
        s = scenes.granular_column(width=c["col_w"] * dx, height=c["col_h"] * dx, box_w=c["box_w"] * dx,
                                   box_h=2 * c["col_h"] * dx, dx=dx, skf=c["skf"], precision=fp)
    else:
        s = scenes.two_phase(width=c["box_w"] * dx, height=1.25 * c["water_h"] * dx, block_w=c["col_w"] * dx,
                             block_h=c["col_h"] * dx, water_h=c["water_h"] * dx, dx=dx, skf=c["skf"], precision=fp,
                             forchheimer_b=c.get("drag", 0.0))
    wide, high = (c["box_w"], c["water_h"]) if c["kind"] == "two_phase" else (c["col_w"], c["col_h"])
    _set_moving(s.phases, _rng(seed), wide * dx, high * dx)
    return s


def _set_moving(phases, g, wide, high, base=None):
    """base: where each particle's own scene begins (0 when None)."""
    speed = g.choice((-1.0, 1.0)) * g.uniform(0.2, 0.4)
    for k, P in enumerate(phases):
        real = (P.itype > 0)[:, None]
        x = P.x - (base[k] if base is not None else 0.0)
        ax, ay = np.pi * x[:, 0] / wide, np.pi * x[:, 1] / high
        swirl = speed * np.stack([np.sin(ax) * np.cos(ay), -high / wide * np.cos(ax) * np.sin(ay)], 1)
        P.vx[...] = real * (swirl + g.uniform(-0.02, 0.02, size=P.x.shape))
        P.x += real * g.uniform(-0.02, 0.02, size=P.x.shape) * P.dspp


def _cloud(c, seed):
    """Positions, stride velocities, node constants and grid of a settled scene of about c["nodes"] particles."""
    n, dx = c["nodes"], 0.004
    if c["kind"] == "two_phase":
        high = max(10, int(math.sqrt(n / 1.3 * 0.3)))
        wide = max(14, int(n / 1.3 / high))
        s = scenes.two_phase(width=wide * dx, height=1.2 * high * dx, block_w=wide // 3 * dx, block_h=high // 2 * dx,
                             water_h=high * dx, dx=dx)
        kind = "submerged"
    else:
        side = max(12, int(math.sqrt(n / 1.1)))
        make = scenes.dam_break if c["kind"] == "dam_break" else scenes.granular_column
        box = dict(tank_w=2 * side * dx, tank_h=1.2 * side * dx) if c["kind"] == "dam_break" else \
            dict(box_w=2 * side * dx, box_h=1.2 * side * dx)
        s = make(width=side * dx, height=side * dx, dx=dx, **box)
        kind = "dam_break" if c["kind"] == "dam_break" else "dry"
    g = _rng(seed)
    x0 = np.concatenate([P.x for P in s.phases])
    real = np.concatenate([P.itype > 0 for P in s.phases])[:, None]
    x = x0 + real * g.uniform(-0.15 * dx, 0.15 * dx, size=x0.shape)
    v = real * g.normal(0.0, 0.2, size=(learn.HIST,) + x0.shape)
    h = float(s.phases[0].hsml[0])
    r, p = 2.0 * h, s.params
    xmin, ymin = p.x_min - 4 * r, p.y_min - 4 * r
    grid = learn.Grid(xmin, ymin, r, int(math.ceil((p.x_max + 4 * r - xmin) / r)) + 1,
                      int(math.ceil((p.y_max + 4 * r - ymin) / r)) + 1)
    nodes = learn.node_table(s, 0.0, learn.K_STRIDE * p.dt, kind)
    return dict(x=torch.from_numpy(x).to(DEV), x0=torch.from_numpy(x0).to(DEV),
                v=torch.from_numpy(v.astype(np.float32)).to(DEV),
                nodes=torch.from_numpy(nodes.view(np.uint8).reshape(-1, 32).copy()).to(DEV), table=nodes, grid=grid,
                inv2h=1.0 / r, target=torch.from_numpy(g.normal(0.0, 1.0, size=x0.shape).astype(np.float32)).to(DEV))


def _weights():
    return dict(np.load(learn.DEFAULT_WEIGHTS))


def _edge_inputs(c, seed):
    """Latents (from the seed), receiver rows and the radius graph (the case's own) of one message-passing layer."""
    k = _cloud(c, 0)
    net = learn.MPNet.from_state(_weights())
    n = k["x"].shape[0]
    off, src, dst, ne = net.graph.build(k["x"], n, k["grid"], net.stream)
    m, rows = learn.pad128(ne), learn.pad128(n)
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    e = torch.randn((m, 128), device=DEV, generator=g).to(torch.bfloat16)
    h = torch.randn((rows, 128), device=DEV, generator=g).to(torch.bfloat16)
    pd = (h.float() @ net.W["p1.wsd"]["wb"][128:].float().t()).contiguous()
    return dict(net=net, src=src, dst=dst, ne=ne, e=e, h=h, pd=pd)


def prepare(case, seed):
    do = case["do"]
    if do == "ensemble":
        ens = ensemble.Ensemble(ensemble.specs(case["scenes"], case.get("first", 0)), tune=False)
        _moving(ens, seed)
        stream = torch.cuda.Stream()
        ens.set_stream(stream.cuda_stream)
        return dict(case=case, ens=ens, stream=stream, out=[_buffers(g.scene) for g in ens.groups])
    if do == "edge":
        s = _edge_inputs(case, seed)
        return dict(case=case, out=torch.empty_like(s["e"]), **s)
    if do in ("forward", "train"):
        return dict(case=case, net=learn.MPNet.from_state(_weights()), **_cloud(case, seed))
    s = _scene(case, seed)
    sv = Solver(s)
    state = dict(case=case, scene=s, sv=sv)
    if do == "steps":
        state["stream"] = torch.cuda.Stream()   # one for the solver's work and what reads its results
        sv.set_stream(state["stream"].cuda_stream)
        state["out"] = _buffers(s)
    return state


def _moving(ens, seed):
    g = _rng(seed)
    for grp, sv in zip(ens.groups, ens.solvers):
        base = [np.stack([np.asarray(grp.offsets)[ids], np.zeros(len(ids))], 1) for ids in grp.sids]
        _set_moving(grp.scene.phases, g, 1.0, 1.0, base)
        for k, P in enumerate(grp.scene.phases):
            sv.upload(k + 1, P)
            sv.upload_scene_ids(k + 1, grp.sids[k])


def _buffers(scene):
    return [(torch.empty((P.n, 2), dtype=torch.float64, device=DEV), torch.empty((P.n, 2), dtype=torch.float64, device=DEV))
            for P in scene.phases]


def _read(sv, bufs, fp):
    """Positions and velocities of every phase, on the device."""
    out = []
    for k, (x, v) in enumerate(bufs):
        sv.export_xv(k + 1, x.data_ptr(), v.data_ptr())
        out.append(dict(x=x, v=v if fp == 64 else v.float()))
    return out


def run(state):
    c = state["case"]
    do = c["do"]
    if do == "steps":
        with torch.cuda.stream(state["stream"]):
            state["sv"].time_integration(c["steps"])
            return _read(state["sv"], state["out"], c["fp"])
    if do == "ensemble":
        with torch.cuda.stream(state["stream"]):
            state["ens"].time_integration(c["steps"])
            return [_read(sv, b, 32) for sv, b in zip(state["ens"].solvers, state["out"])]
    if do == "edge":
        net, W, B = state["net"], state["net"].W, state["net"].B
        wsd = W["p1.wsd"]["wb"]
        learn._call(net.L.sphg_gnn_edge_layer_nodes(
            state["e"].data_ptr(), state["out"].data_ptr(), state["h"].data_ptr(), state["pd"].data_ptr(),
            state["h"].shape[0], state["src"].data_ptr(), state["dst"].data_ptr(), state["ne"], state["e"].shape[0],
            W["p1.we"]["wb"].data_ptr(), wsd.data_ptr(), B["p1.be"]["w"].data_ptr(), W["p1.w2"]["wb"].data_ptr(),
            B["p1.b2"]["w"].data_ptr(), net.err.data_ptr(), net.stream), "sphg_gnn_edge_layer_nodes")
        return state["out"]
    if do == "forward":
        net = state["net"]
        b = net.make_batch(state["x"], state["nodes"], state["v"], 0, state["grid"], state["inv2h"], x0=state["x0"])
        return net.forward(b, keep=False)
    if do == "train":
        net = state["net"]
        b = net.make_batch(state["x"], state["nodes"], state["v"], 0, state["grid"], state["inv2h"],
                           target=state["target"], x0=state["x0"])
        loss = net.train_step(b, 1.0e-5, learn.HUBER_DELTA)
        return dict(loss=loss, **{k: d["g"] for k, d in list(net.W.items()) + list(net.B.items())})
    # host arrays in, host arrays out
    sv, s = state["sv"], state["scene"]
    for k, P in enumerate(s.phases):
        sv.upload(k + 1, P)
    if do == "rhs":
        sv.single_step(1)
    else:
        sv.itimestep, sv.time = 0, 0.0
        for _ in range(c["steps"] // c["per_call"]):
            sv.time_integration(c["per_call"])
            sv.stats()
    got = [sv.download(k + 1) for k in range(sv.nphase)]
    if c["fp"] == 32:
        return [dict(x=P.x, **{f: getattr(P, f).astype(np.float32) for f in ("vx", "rho", "p", "sxx", "sxy", "syy")})
                for P in got]
    return [{f: getattr(P, f) for f in FULL} for P in got]


# ------------------------------------------------------------------ work

def _counts(c):
    """(water, soil) particles, walls included."""
    walls = 2 * (c["box_w"] + 4) + 4 * int(round((1.25 * c["water_h"] if c["kind"] == "two_phase" else
                                                 (1.5 if c["kind"] == "dam_break" else 2.0) * c["col_h"])))
    if c["kind"] == "two_phase":
        return c["box_w"] * c["water_h"] + walls, c["col_w"] * c["col_h"] + walls
    n = c["col_w"] * c["col_h"] + walls
    return (n, 0) if c["kind"] == "dam_break" else (0, n)


def work(case):
    do = case["do"]
    if do in ("edge", "forward", "train"):
        n, e = case["nodes"], 19 * case["nodes"]
        layer = (128 * 128 * 2 * 3) * e                 # edge MLP, sender term included
        if do == "edge":
            return dict(bytes=e * (2 * 256 + 8) + n * (256 + 512), flops=layer)
        node = (128 * 128 * 2 * 4) * n
        fwd = 4 * (layer + node) + e * 2 * (64 + 128) * 128 + n * 2 * (64 + 3 * 128) * 128
        if do == "forward":                              # edge rows of every layer in and out, and the encoder's
            return dict(bytes=e * (4 * 2 * 256 + 256) + n * 4 * 1024, flops=fwd)
        return dict(bytes=e * (4 * 6 * 256), flops=3 * fwd)
    if do == "ensemble":
        wet = dry = 0
        for s in ensemble.specs(case["scenes"], case.get("first", 0)):
            wet += 0 if s.kind == "dry" else s.n_target
            dry += 0 if s.kind == "dam_break" else s.n_target // (3 if s.kind == "submerged" else 1)
        fp, steps, host = 32, case["steps"], 0
    else:
        wet, dry = _counts(case)
        fp, steps, host = case["fp"], case.get("steps", 1), do in ("host", "rhs")
    # a step reads and writes each particle's state once: x, v, rho, rates, mass, type, cell key, volume fraction (water)
    # or stresses and their rates (soil); 20 neighbours a particle, two sums over them for water, one for soil
    a, b = (112, 168) if fp == 32 else (180, 268)
    return dict(bytes=steps * (a * wet + b * dry) + host * 37 * 8 * 2 * (wet + dry),
                flops=steps * 20 * (110 * wet + 75 * dry))


# ------------------------------------------------------------------ 64 bits

PI = float(np.float32(3.14159265359))


def _pairs(xa, xb, radius, same):
    """Every ordered pair (i of a, j of b) closer than radius, by cells of that side."""
    lo = torch.minimum(xa.min(0).values, xb.min(0).values)
    ca, cb = (((x - lo) / radius).floor().long() + 1 for x in (xa, xb))
    nx = int(max(ca[:, 0].max(), cb[:, 0].max())) + 2
    kb, order = torch.sort(cb[:, 1] * nx + cb[:, 0], stable=True)
    I, J = [], []
    for dy in (-1, 0, 1):
        mid = (ca[:, 1] + dy) * nx + ca[:, 0]
        b = torch.searchsorted(kb, mid - 1)
        cnt = torch.searchsorted(kb, mid + 1, right=True) - b
        i = torch.repeat_interleave(torch.arange(len(xa), device=xa.device), cnt)
        start = torch.cumsum(cnt, 0) - cnt
        j = order[torch.arange(len(i), device=xa.device) - start[i] + b[i]]
        d = xa[i] - xb[j]
        keep = (d * d).sum(1).sqrt() < radius
        if same:
            keep &= i != j
        I.append(i[keep])
        J.append(j[keep])
    return torch.cat(I), torch.cat(J)


def _kernel(skf, r, h):
    """W and the factor s with grad W = s dx."""
    q = r / h
    if skf == 1:
        f = 15.0 / (7.0 * PI * h * h)
        near = q <= 1.0
        w = torch.where(near, f * (float(np.float32(2.0 / 3.0)) - q * q + q ** 3 / 2), f / 6 * (2 - q) ** 3)
        s = torch.where(near, f * (-2 + 1.5 * q) / (h * h), -f / 2 * (2 - q) ** 2 / (h * torch.clamp(r, min=1e-300)))
        return w, s
    f = 7.0 / (4.0 * PI * h * h)
    u = 1 - q / 2
    return f * u ** 4 * (1 + 2 * q), f * (-5 + 7.5 * q - 3.75 * q * q + 0.625 * q ** 3) / (h * h)


class _Sums:
    """The ordered pairs of one list with their kernel values; sum() adds a pair quantity up per particle of a."""

    def __init__(self, A, B, skf, scale, same):
        self.i, self.j = _pairs(A["x"], B["x"], scale * A["h"], same)
        self.n = len(A["x"])
        d = A["x"][self.i] - B["x"][self.j]
        self.dx, self.dy = d[:, 0], d[:, 1]
        self.rr = self.dx ** 2 + self.dy ** 2
        self.w, self.s = _kernel(skf, self.rr.sqrt(), A["h"])
        self.gx, self.gy = self.s * self.dx, self.s * self.dy

    def sum(self, v):
        return torch.zeros(self.n, dtype=torch.float64, device=v.device).index_add_(0, self.i, v)


def _momentum(p, k, P, rho, ci, cj):
    """Artificial viscosity, XSPH and (two-phase) the wall force, which every step shares."""
    v, m, h = P["v"], P["m"], P["h"]
    du, dv = v[k.i, 0] - v[k.j, 0], v[k.i, 1] - v[k.j, 1]
    mr, mb = 0.5 * (rho[k.i] + rho[k.j]), m[k.j]
    vr = du * k.dx + dv * k.dy
    muv = h * vr / (k.rr + h * h * p.etq * p.etq)
    piv = torch.where(vr < 0, (p.beta * muv - p.alpha * 0.5 * (ci + cj)) * muv / mr, torch.zeros_like(vr))
    ax, ay = -k.sum(mb * piv * k.gx), -k.sum(mb * piv * k.gy)
    q = mb * k.w / mr
    av = torch.stack([-k.sum(q * du), -k.sum(q * dv)], 1)
    av = torch.where(P["real"][:, None], p.epsilon * av, av)
    if not p.single_phase:
        r = k.rr.sqrt()
        on = P["real"][k.i] & ~P["real"][k.j] & (r <= P["dspp"])
        z = P["dspp"] / torch.where(on, r, torch.ones_like(r))
        f = torch.where(on, p.dd * (z ** p.p1 - z ** p.p2) / k.rr, torch.zeros_like(r))
        ax, ay = ax + k.sum(f * k.dx), ay + k.sum(f * k.dy)
    return ax, ay + p.gravity, av


C23 = float(np.float32(2.0 / 3.0))


def _strain(k, vol, du, dv):
    vb = vol[k.j]
    return (k.sum(vb * C23 * (2 * du * k.gx - dv * k.gy)), k.sum(vb * (du * k.gy + dv * k.gx)),
            k.sum(vb * C23 * (2 * dv * k.gy - du * k.gx)))


def _water(p, W, scale):
    """Sums of the water phase; returns what the cross pairs need."""
    m, v, h = W["m"], W["v"], W["h"]
    k = _Sums(W, W, p.skf, scale, True)
    vb = (m / W["rho"])[k.j]
    du, dv = v[k.j, 0] - v[k.i, 0], v[k.j, 1] - v[k.i, 1]
    if p.single_phase:
        w0 = _kernel(p.skf, torch.zeros(1, dtype=torch.float64, device=m.device), h)[0]
        rho = (w0 * m + k.sum(m[k.j] * k.w)) / (w0 * m / W["rho"] + k.sum(vb * k.w))
        con = -k.sum(m[k.j] * (du * k.gx + dv * k.gy))
        W["rho"] = rho
    else:
        rho = W["rho"]
        con = -k.sum(m[k.j] * (du * k.gx + dv * k.gy))
    vol = m / rho
    vb = vol[k.j]
    pref = p.delta * h * W["c"]
    W["drho"] = con + pref * k.sum(vb * (rho[k.i] - rho[k.j]) * 2 * k.s)
    if p.single_phase:
        su, sv = v[k.i, 0] + v[k.j, 0], v[k.i, 1] + v[k.j, 1]
        t = [k.sum(vb * a) for a in (su * k.gx, sv * k.gy, su * k.gy, sv * k.gx)]
        txx, txy, tyy = C23 * (2 * t[0] - t[1]), t[2] + t[3], C23 * (2 * t[1] - t[0])
        W["p"] = p.water.b * ((rho / p.water.rho0) ** p.water.gamma - 1)
        phi = torch.ones_like(rho)
    else:
        txx, txy, tyy = _strain(k, vol, du, dv)
        phi = W["vof"]
        ratio = rho / (p.water.rho0 * phi)
        W["p"] = p.water.b * (ratio ** p.water.gamma - 1)
        W["c"] = p.water.c * ratio ** 3
    W["sxx"], W["sxy"], W["syy"] = (p.water.viscosity * t for t in (txx, txy, tyy))
    pr, sx = W["p"], {f: phi * W[f] for f in ("sxx", "sxy", "syy")}
    pp = pr[k.i] + pr[k.j]
    st = {f: a[k.i] + a[k.j] for f, a in sx.items()}
    ax, ay, W["av"] = _momentum(p, k, W, rho, W["c"][k.i], W["c"][k.j])
    ax = ax + (-phi * k.sum(vb * pp * k.gx) + k.sum(vb * (st["sxx"] * k.gx + st["sxy"] * k.gy))) / rho
    ay = ay + (-phi * k.sum(vb * pp * k.gy) + k.sum(vb * (st["sxy"] * k.gx + st["syy"] * k.gy))) / rho
    W["dv"] = torch.stack([ax, ay], 1)
    W["dvof"] = torch.zeros_like(rho)
    if not p.single_phase:
        W["dvof"] = p.delta * h * W["c"] * k.sum(vb * (phi[k.i] - phi[k.j]) * 2 * k.s)


def _soil(p, S, scale):
    m, v, h, rho = S["m"], S["v"], S["h"], S["rho"]
    k = _Sums(S, S, p.skf, scale, True)
    vol = m / rho
    vb, mb, e = vol[k.j], m[k.j], 2 * k.s
    du, dv = v[k.j, 0] - v[k.i, 0], v[k.j, 1] - v[k.i, 1]
    S["drho"] = -k.sum(mb * (du * k.gx + dv * k.gy)) + p.delta * h * S["c"] * k.sum(vb * (rho[k.i] - rho[k.j]) * e)
    txx, txy, tyy = _strain(k, vol, du, dv)
    vcc = k.sum(vb * (du * k.gx + dv * k.gy))
    wxy = k.sum(vb * 0.5 * (du * k.gy - dv * k.gx))
    f = {}
    for q in ("p", "sxx", "sxy", "syy"):
        a = S[q] if p.single_phase else S["vof"] * S[q] / rho ** 2
        f[q] = (a[k.i] + a[k.j]) * (vb if p.single_phase else mb)
    one = 1.0 / rho if p.single_phase else 1.0
    cs = torch.full_like(k.rr, p.soil.c)
    ax, ay, S["av"] = _momentum(p, k, S, rho, cs, cs)
    S["ax"] = ax + one * k.sum((f["sxx"] - f["p"]) * k.gx + f["sxy"] * k.gy)
    S["ay"] = ay + one * k.sum(f["sxy"] * k.gx + (f["syy"] - f["p"]) * k.gy)
    G, K, al = p.soil.E / (2 * (1 + p.soil.niu)), p.soil.k, _alpha1(p)
    sxx, sxy, syy, pr = S["sxx"], S["sxy"], S["syy"], S["p"]
    J = (sxx ** 2 + 2 * sxy ** 2 + syy ** 2 + (sxx + syy) ** 2) / 2
    on = (J.sqrt() + 1e-6 - al * 3 * pr).abs() < float(np.float32(1e-5))
    sde = sxx * (txx / 2 + vcc / 3) + sxy * txy + syy * (tyy / 2 + vcc / 3)
    rJ = (J + 1e-10).sqrt()
    lam = (3 * al * K * vcc + G / rJ * sde) / (9 * al * al * K + G)
    lam = torch.where(on & ~(lam < 0), lam, torch.zeros_like(lam))
    d = {q: p.delta * h * p.soil.c * k.sum(vb * e * (S[q][k.i] - S[q][k.j])) for q in ("p", "sxx", "sxy", "syy")}
    S["dsxx"] = G * txx - lam * G / rJ * sxx + 2 * sxy * wxy + d["sxx"]
    S["dsxy"] = G * txy - lam * G / rJ * sxy - (sxx - syy) * wxy + d["sxy"]
    S["dsyy"] = G * tyy - lam * G / rJ * syy - 2 * sxy * wxy + d["syy"]
    S["dp"] = -K * vcc + 3 * K * al * lam + d["p"]
    S["vcc"] = vcc
    S["txx"], S["tyy"], S["wxy"] = txx, tyy, wxy
    S["c"] = torch.full_like(S["c"], p.soil.c)
    S["dv"] = torch.stack([S["ax"], S["ay"]], 1)


def _cross(p, W, S, scale):
    phis, drag, kb = S["vof"], -p.numeric_gravity / p.soil.permeability, p.soil.permeability * p.forchheimer_b
    for A, B, water in ((W, S, True), (S, W, False)):
        k = _Sums(A, B, p.skf, scale, False)
        u = A["v"][k.i] - B["v"][k.j]
        q = (B["m"] / B["rho"])[k.j] * k.w * (1 + kb * (u * u).sum(1).sqrt())
        if water:
            q = q * phis[k.j]
            fac = A["vof"] * drag
            mb = B["m"][k.j]
            A["dvof"] = A["dvof"] - k.sum(mb * (u[:, 0] * k.gx + u[:, 1] * k.gy)) / p.soil.rho0
            A["vof2"] = 1 - k.sum(mb * k.w) / p.soil.rho0
        else:
            q = q * B["rho"][k.j] * B["vof"][k.j]
            fac = phis * drag / A["rho"]
            mp = (B["m"] / B["rho"] * B["p"])[k.j]
            A["dv"] = A["dv"] - (phis / A["rho"])[:, None] * torch.stack([k.sum(mp * k.gx), k.sum(mp * k.gy)], 1)
        A["dv"] = A["dv"] - fac[:, None] * torch.stack([k.sum(q * u[:, 0]), k.sum(q * u[:, 1])], 1)
    S["vof"] = S["rho"] / p.soil.rho0


def _alpha1(p):
    t = math.tan(p.soil.phi)
    return t / math.sqrt(9.0 + 12.0 * t * t)


def _return(p, S):
    """Drucker-Prager return of the stress."""
    S["p"] = torch.clamp(S["p"], min=0.0)
    J = ((S["sxx"] ** 2 + 2 * S["sxy"] ** 2 + S["syy"] ** 2 + (S["sxx"] + S["syy"]) ** 2) / 2).sqrt() + 1e-6
    lim = _alpha1(p) * 3 * S["p"]
    f = torch.where(J > lim, lim / J, torch.ones_like(J))
    for q in ("sxx", "sxy", "syy"):
        S[q] = f * S[q]


def _rhs(p, ph):
    scale = {1: 2, 2: 3, 3: 3, 4: 2}[p.skf]
    for P in ph:
        if P["soil"]:
            _return(p, P)
    for P in ph:
        (_soil if P["soil"] else _water)(p, P, scale)
    if len(ph) == 2:
        _cross(p, ph[0], ph[1], scale)


def _leapfrog(p, ph, steps):
    dt = p.dt
    for it in range(1, steps + 1):
        first = it == 1
        for P in ph:
            if first:
                continue
            P["rho0"], P["v0"], P["vof0"] = P["rho"], P["v"], P["vof"]
            P["rho"] = P["rho"] + dt / 2 * P["drho"]
            if not P["soil"] and len(ph) == 2:
                P["vof"] = P["vof"] + dt / 2 * P["dvof"]
            P["v"] = torch.where(P["real"][:, None], P["v"] + dt / 2 * P["dv"], P["v"])
            if P["soil"]:
                _return(p, P)
        _rhs(p, ph)
        for P in ph:
            half = dt / 2 if first else dt
            P["rho"] = (P["rho"] if first else P["rho0"]) + half * P["drho"]
            if not P["soil"] and len(ph) == 2:
                P["vof"] = (P["vof"] if first else P["vof0"]) + half * P["dvof"]
            if P["soil"]:
                for q in ("p", "sxx", "sxy", "syy"):
                    P[q] = P[q] + dt * P["d" + q]
                _return(p, P)
            v = (P["v"] if first else P["v0"]) + half * P["dv"] + P["av"]
            P["v"] = torch.where(P["real"][:, None], v, P["v"])
            P["x"] = torch.where(P["real"][:, None], P["x"] + dt * v, P["x"])


def _phases(s):
    out = []
    for P in s.phases:
        t = {k: torch.from_numpy(getattr(P, f).copy()).to(DEV) for k, f in
             (("x", "x"), ("v", "vx"), ("rho", "rho"), ("p", "p"), ("c", "c"), ("m", "mass"), ("vof", "vof"),
              ("sxx", "sxx"), ("sxy", "sxy"), ("syy", "syy"))}
        t.update(h=float(P.hsml[0]), real=torch.from_numpy(P.itype > 0).to(DEV), soil=P.material == 2, dspp=P.dspp)
        out.append(t)
    return out


def _mlp(x, w1, b1, w2, b2):
    return torch.relu(x @ w1.t() + b1) @ w2.t() + b2


def _network(w, k, vscale):
    """The message-passing network over the radius graph of k, in 64 bits: (output, real rows)."""
    x, x0, inv = k["x"], k["x0"], k["inv2h"]
    n = x.shape[0]
    dst, src = _pairs(x, x, 1.0 / inv, True)
    tab = k["table"]
    col = {f: torch.from_numpy(tab[f].astype(np.float64)).to(DEV) for f in ("xl", "xr", "yf", "dts", "porosity", "phi")}
    typ = torch.from_numpy(tab["type"].copy()).to(DEV)
    vel = (k["v"].double() / vscale).permute(1, 0, 2).reshape(n, 10)
    wall = (torch.stack([x[:, 0] - col["xl"], col["xr"] - x[:, 0], x[:, 1] - col["yf"]], 1) * inv).clamp(0, 1)
    fn = torch.zeros((n, 64), dtype=torch.float64, device=DEV)
    fn[:, :21] = torch.cat([vel, torch.nn.functional.one_hot(typ.long(), 3).double(), wall,
                            torch.stack([col["porosity"], col["phi"], col["dts"] * 1e3], 1),
                            ((x - x0) * inv).clamp(-16, 16)], 1)
    d, d0 = (x[dst] - x[src]) * inv, (x0[dst] - x0[src]) * inv
    fe = torch.zeros((len(dst), 64), dtype=torch.float64, device=DEV)
    fe[:, :6] = torch.cat([d, (d * d).sum(1, keepdim=True).sqrt(), (typ[dst] == typ[src]).double()[:, None],
                           (d - d0).clamp(-4, 4)], 1)
    h = _mlp(fn, w["enc_n.w1"], w["enc_n.b1"], w["enc_n.w2"], w["enc_n.b2"])
    e = _mlp(fe, w["enc_e.w1"], w["enc_e.b1"], w["enc_e.w2"], w["enc_e.b2"])
    for l in range(learn.LAYERS):
        p = "p%d." % l
        P = h @ w[p + "wsd"].t()
        z = e @ w[p + "we"].t() + P[src, :128] + P[dst, 128:] + w[p + "be"]
        e = e + torch.relu(z) @ w[p + "w2"].t() + w[p + "b2"]
        agg = torch.zeros_like(h).index_add(0, dst, e) * learn.AGG_SCALE
        h = h + _mlp(torch.cat([h, agg], 1), w[p + "v1"], w[p + "c1"], w[p + "v2"], w[p + "c2"])
    return _mlp(h, w["dec.w1"], w["dec.b1"], w["dec.w2"], w["dec.b2"]), typ != learn.GNN_BOUNDARY


def _weights64(grad):
    d = _weights()
    w = {k: torch.from_numpy(v.astype(np.float64)).to(DEV).requires_grad_(grad) for k, v in d.items()
         if not k.startswith("_")}
    return w, float(d["_vscale"][0])


def exact(case, seed):
    do = case["do"]
    if do == "ensemble":
        return None           # scenes of several time steps in one context; the single scenes' cases have values
    if do == "edge":
        s = _edge_inputs(case, seed)
        w, _ = _weights64(False)
        ne, e, h = s["ne"], s["e"].double(), s["h"].double()
        z = e @ w["p1.we"].to(torch.bfloat16).double().t() + w["p1.be"]
        ws = (h @ w["p1.wsd"][:128].to(torch.bfloat16).double().t())
        z[:ne] += ws[s["src"].long()] + s["pd"].double()[s["dst"].long()]
        return e + torch.relu(z) @ w["p1.w2"].to(torch.bfloat16).double().t() + w["p1.b2"]
    if do == "forward":
        k = _cloud(case, seed)
        w, vs = _weights64(False)
        out, _ = _network(w, k, vs)
        full = torch.zeros((learn.pad128(len(out)), 128), dtype=torch.float64, device=DEV)
        full[:len(out)] = out
        zero = torch.zeros((1, 64), dtype=torch.float64, device=DEV)    # padding rows: no inputs, no edges
        h = _mlp(zero, w["enc_n.w1"], w["enc_n.b1"], w["enc_n.w2"], w["enc_n.b2"])
        for l in range(learn.LAYERS):
            p = "p%d." % l
            h = h + _mlp(torch.cat([h, torch.zeros_like(h)], 1), w[p + "v1"], w[p + "c1"], w[p + "v2"], w[p + "c2"])
        full[len(out):] = _mlp(h, w["dec.w1"], w["dec.b1"], w["dec.w2"], w["dec.b2"])
        return full
    if do == "train":
        k = _cloud(case, seed)
        w, vs = _weights64(True)
        out, real = _network(w, k, vs)
        d = (out[:, :2] - k["target"].double())[real]
        a, lim = d.abs(), learn.HUBER_DELTA
        loss = torch.where(a <= lim, d * d, lim * (2 * a - lim)).sum() / d.numel()
        loss.backward()
        return dict(loss=float(loss), **{n: t.grad for n, t in w.items()})
    s = _scene(case, seed)
    ph = _phases(s)
    if do == "rhs":
        for P in ph:
            P["av"] = P["dvof"] = None
        _rhs(s.params, ph)
    else:
        _leapfrog(s.params, ph, case["steps"])
    if do == "steps":
        return [dict(x=P["x"], v=P["v"]) for P in ph]
    names = {"vx": "v", "dvx": "dv"}
    keep = ("x", "vx", "rho", "p") if case["fp"] == 32 else \
        ("x", "vx", "dvx", "av", "rho", "drho", "p", "c", "dvof")
    out = []
    for P in ph:
        fields = keep + (("sxx", "sxy", "syy") if P["soil"] else ())
        o = {f: P[names.get(f, f)] for f in fields if P.get(names.get(f, f)) is not None}
        out.append({f: o.get(f) for f in (FULL if case["fp"] == 64 else ("x", "vx", "rho", "p", "sxx", "sxy", "syy"))})
    return out
