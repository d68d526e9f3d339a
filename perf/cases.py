"""The work a user of this engine has it do, as cases that can be timed.

Every case goes through the package's public entry points: whole runs of steps
to the next snapshot in each force form, the step of a host-held state, the
reference-shaped stage calls, the locally essential tree exchange's local part,
and the training of the acceptance network.  Inputs are seeded synthetic solar
systems (the Sun, eight planets, asteroids from Keplerian element
distributions: an inner belt, an outer belt, Jupiter's trojan clouds).
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

bh = importlib.import_module("barnes-hut_gb300")

G = 1.48812e-34       # AU^3 kg^-1 day^-2
DT = 1.0 / 24.0       # one hour, the step of every configuration
MU_SUN = G * 1.989e30
MODES = {"plain": bh.MODE_PLAIN_FP64, "list": bh.MODE_FP64_LIST, "fp32": bh.MODE_FP32_FAR,
         "learned": bh.MODE_LEARNED, "group": bh.MODE_FP32_GROUP}
# Body-steps of one pass in each form, at most: no drawn case costs more than
# the largest listed one.
MOST_BODY_STEPS = {"plain": 460_000, "list": 1_200_000, "fp32": 4_000_000, "learned": 2_000_000,
                   "group": 16_000_000}


def listed():
    return [
        # A toy system a day (24 hourly steps) at a time, as the tests and
        # smoke run it: every kernel is a few blocks, launches and latency count.
        dict(name="plain_1k_day", kind="steps", mode="plain", n=1000, theta=1.05, nsteps=24, outer=0.0, trojan=0.0),
        # The CPU-runnable configuration (19,054 bodies, bit-exact form), a day
        # between two snapshots.
        dict(name="plain_19k_day", kind="steps", mode="plain", n=19_054, theta=1.05, nsteps=24, outer=0.0,
             trojan=0.0),
        # The reference's own call sequence on host arrays (bounding box, keys,
        # sort, octree, accelerations): the drop-in boundary, default form.
        dict(name="plain_100k_stages", kind="stages", mode="plain", n=100_003, theta=1.05, outer=0.1, trojan=0.0),
        # The headline workload: 300,149 bodies in the FP64 list form.
        dict(name="list_300k_steps", kind="steps", mode="list", n=300_149, theta=1.05, nsteps=4, outer=0.1,
             trojan=0.0),
        # A driver that holds its bodies in host memory and hands them over for
        # each step.
        dict(name="list_65k_host", kind="host", mode="list", n=65_537, theta=1.05, nsteps=1, outer=0.1, trojan=0.0),
        # A small system in the precision form: a day between two snapshots.
        dict(name="fp32_19k_day", kind="steps", mode="fp32", n=19_054, theta=1.05, nsteps=24, outer=0.0, trojan=0.0),
        # The precision form's configuration at its middle angle.
        dict(name="fp32_1m_steps", kind="steps", mode="fp32", n=1_000_000, theta=0.8, nsteps=4, outer=0.1,
             trojan=0.0),
        # The learned criterion at its tightest evaluated budget.
        dict(name="learned_1m_steps", kind="steps", mode="learned", n=1_000_000, theta=1.05, nsteps=2, outer=0.1,
             trojan=0.0, budget=1e-6),
        # The combined scale run's system in the fastest form at its angle.
        dict(name="group_4m_steps", kind="steps", mode="group", n=4_000_000, theta=1.05, nsteps=4, outer=0.1,
             trojan=0.05),
        # One rank's share of a distributed step: the export to a neighbour and
        # the forces with the records received from the others.
        dict(name="let_250k", kind="let", n=250_007, ranks=4, theta=1.05, outer=0.1, trojan=0.0),
        # An epoch of the acceptance network's training, default batch.
        dict(name="train_128k", kind="train", n=131_072, epochs=1, batch=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["host", "stages", "let", "train"])
    if kind == "train":
        return dict(kind="train", n=_log_int(rng, 20_000, 131_072), epochs=1, batch=rng.choice([1000, 2048, 4096]))
    mix = dict(outer=rng.choice([0.0, 0.1, 0.1]), trojan=rng.choice([0.0, 0.0, 0.05]))
    theta = round(rng.uniform(0.5, 1.3), 3)
    if kind == "let":
        return dict(kind="let", n=_log_int(rng, 10_000, 250_000), ranks=rng.choice([2, 4, 8]),
                    theta=round(rng.uniform(0.8, 1.3), 3), **mix)
    if kind == "stages":
        return dict(kind="stages", mode=rng.choice(["plain", "plain", "list", "fp32", "group"]),
                    n=_log_int(rng, 1000, 100_000), theta=theta, **mix)
    mode = rng.choice(["plain", "list", "list", "fp32", "group", "learned"])
    if kind == "host":
        mode = rng.choice(["plain", "list", "fp32", "group"])
        most = 0.25 * MOST_BODY_STEPS[mode] * min(1.0, theta * theta)
        return dict(kind="host", mode=mode, n=_log_int(rng, 1000, most), theta=theta, nsteps=1, **mix)
    most = MOST_BODY_STEPS[mode] * min(1.0, theta * theta)
    n = _log_int(rng, 1000, min(most, 4_000_000))
    case = dict(kind="steps", mode=mode, n=n, theta=theta, nsteps=max(1, min(24, int(most / n))), **mix)
    if mode == "learned":
        case["budget"] = rng.choice([1e-6, 3e-6, 1e-5])
    return case


# ------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _system(seed, n, outer, trojan):
    """(pos, vel, mass, ids) of a seeded synthetic solar system, as host arrays."""
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(int(seed))

    def uni(k, lo, hi):
        return lo + (hi - lo) * torch.rand(k, generator=g, device=dev, dtype=torch.float64)

    k = n - 9
    kind = torch.rand(k, generator=g, device=dev, dtype=torch.float64)
    out, tro = kind < outer, (kind >= outer) & (kind < outer + trojan)
    deg = math.pi / 180.0
    a = torch.where(out, uni(k, 30.0, 50.0), uni(k, 2.1, 3.3))
    e = torch.where(out, uni(k, 0.0, 0.2), torch.where(tro, uni(k, 0.0, 0.1), uni(k, 0.0, 0.3)))
    inc = torch.where(out, uni(k, 0.0, 30.0 * deg), uni(k, 0.0, 20.0 * deg))
    a = torch.where(tro, torch.full_like(a, 5.2), a)
    node, peri, anom = (uni(k, 0.0, 2 * math.pi) for _ in range(3))
    planet_a = torch.tensor([0.387, 0.723, 1.0, 1.524, 5.203, 9.537, 19.19, 30.07], device=dev, dtype=torch.float64)
    planet_m = torch.tensor([3.301e23, 4.867e24, 5.972e24, 6.417e23, 1.898e27, 5.683e26, 8.681e25, 1.024e26],
                            device=dev, dtype=torch.float64)
    phase = uni(8, 0.0, 2 * math.pi)
    # A trojan's mean longitude lies within 30 degrees of Jupiter's L4 or L5.
    lon = phase[4] + torch.where(uni(k, 0.0, 1.0) < 0.5, 60.0, -60.0) * deg + uni(k, -30.0 * deg, 30.0 * deg)
    anom = torch.where(tro, lon - node - peri, anom)
    a, e = torch.cat([planet_a, a]), torch.cat([torch.zeros_like(planet_a), e])
    zero = torch.zeros_like(planet_a)
    inc, node, peri = torch.cat([zero, inc]), torch.cat([zero, node]), torch.cat([zero, peri])
    anom = torch.remainder(torch.cat([phase, anom]), 2 * math.pi)
    ecc = anom.clone()
    for _ in range(12):
        ecc = ecc - (ecc - e * torch.sin(ecc) - anom) / (1.0 - e * torch.cos(ecc))
    ce, se = torch.cos(ecc), torch.sin(ecc)
    b = torch.sqrt(1.0 - e * e)
    speed = torch.sqrt(MU_SUN / a) / (1.0 - e * ce)
    x, y, u, v = a * (ce - e), a * b * se, -speed * se, speed * b * ce
    cn, sn, cw, sw, ci, si = (f(q) for q in (node, peri, inc) for f in (torch.cos, torch.sin))
    px, py, pz = cn * cw - sn * sw * ci, sn * cw + cn * sw * ci, sw * si
    qx, qy, qz = -cn * sw - sn * cw * ci, -sn * sw + cn * cw * ci, cw * si
    pos = torch.zeros(n, 3, device=dev, dtype=torch.float64)
    vel = torch.zeros_like(pos)
    pos[1:] = torch.stack([x * px + y * qx, x * py + y * qy, x * pz + y * qz], 1)
    vel[1:] = torch.stack([u * px + v * qx, u * py + v * qy, u * pz + v * qz], 1)
    mass = torch.cat([torch.tensor([1.989e30], device=dev, dtype=torch.float64), planet_m,
                      10.0 ** uni(k, 12.0, 20.0)])
    return pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy(), np.arange(n, dtype=np.uint64)


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available()).numpy()


def _model(seed):
    """A deterministic acceptance network on raw features: the quadrupole
    estimate f3 + 2 f1 of the log10 error less 0.3 (what training arrives at on
    average), with the other units small and seeded."""
    r = np.random.default_rng(seed)
    w1, b1 = r.normal(0.0, 0.1, (64, 8)), np.zeros(64)
    w2, b2, w3 = r.normal(0.0, 0.02, (64, 64)), np.zeros(64), r.normal(0.0, 0.02, 64)
    w1[:2] = 0.0
    w1[0, 1], w1[0, 3], w1[1, 1], w1[1, 3] = 2.0, 1.0, -2.0, -1.0
    w2[:2] = 0.0
    w2[0, 0], w2[1, 1] = 1.0, 1.0
    w3[:2] = 1.0, -1.0
    params = np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [-0.3]]).astype(np.float32)
    scale = np.concatenate([np.zeros(8), np.ones(8), np.full(8, -1e3), np.full(8, 1e3), [0.0, 1.0]]).astype(np.float32)
    return params, scale


def _keys(pos, lo, hi):
    """63-bit Morton keys (21 bits per axis) of torch positions in a box."""
    span = hi - lo
    span = torch.where(span == 0, torch.ones_like(span), span)
    t = ((pos - lo) / span).clamp(0.0, 1.0 - 2.0 ** -53)
    q = (t * 2097152.0).to(torch.int64)
    key = torch.zeros(pos.shape[0], dtype=torch.int64, device=pos.device)
    for bit in range(21):
        for ax in range(3):
            key |= ((q[:, ax] >> bit) & 1) << (3 * bit + ax)
    return key


def _shares(pos, ranks):
    """Morton keys, the box, and the key-order share of rank 0 and of rank 1."""
    p = torch.from_numpy(pos).to(_device())
    lo, hi = p.min(0).values, p.max(0).values
    key = _keys(p, lo, hi)
    order = torch.sort(key, stable=True).indices
    return p, key, lo, hi, order


def _let_inputs(case, seed):
    """Rank 0's bodies, the global box, a neighbour's domain boxes and the
    records received from the other ranks (their cells 7 levels down)."""
    n, ranks = case["n"], case["ranks"]
    pos, vel, mass, ids = _system(seed, n * ranks, case["outer"], case["trojan"])
    p, key, lo, hi, order = _shares(pos, ranks)
    mine = np.sort(order[:n].cpu().numpy())
    bbox = torch.cat([lo, hi]).cpu().numpy()
    theirs = order[n:]
    depth = 7
    mask = ~((1 << (63 - 3 * depth)) - 1)
    cell, inv = torch.unique(key[theirs] & mask, return_inverse=True)
    m = torch.from_numpy(mass).to(p.device)[theirs]
    cm = torch.zeros(len(cell), dtype=torch.float64, device=p.device).index_add_(0, inv, m)
    cw = torch.zeros(len(cell), 3, dtype=torch.float64, device=p.device).index_add_(0, inv, m[:, None] * p[theirs])
    # Sums in 64 bits by index_add_ vary in their last bits from run to run:
    # rounded to 32 bits they are the same inputs for everybody.
    cm = cm.to(torch.float32).to(torch.float64)
    com = (cw / cm[:, None]).to(torch.float32).to(torch.float64)
    bucket = torch.unique(key[order[n:2 * n]] & ~((1 << (63 - 18)) - 1)).cpu().numpy().astype(np.uint64)
    return dict(pos=pos[mine], vel=vel[mine], mass=mass[mine], ids=ids[mine], bbox=bbox, buckets=bucket,
                rec=(cell.cpu().numpy().astype(np.uint64), np.full(len(cell), depth, np.uint8), cm.cpu().numpy(),
                     com.cpu().numpy()))


def _pairs(case, seed):
    r = np.random.default_rng(seed)
    f = r.normal(0.0, 1.0, (case["n"], 8)).astype(np.float32) * np.float32(0.7) - np.float32(0.4)
    label = f[:, 3] + 2.0 * f[:, 1] + 0.3 * f[:, 0] * f[:, 4] + r.normal(0.0, 0.25, case["n"])
    return f, label.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        f, label = _pairs(case, seed)
        return dict(case=case, features=f, labels=label, seed=int(seed) & 0xFFFF)
    if kind == "let":
        s = _let_inputs(case, seed)
        ctx = bh.Context(case["n"])
        ctx.set_bodies(s["pos"], s["vel"], s["mass"], s["ids"])
        ctx.set_bbox(s["bbox"])
        ctx.compute_keys()
        ctx.sort_bodies()
        # The send buffer the exported records are packed into (the tree keeps
        # at most 2 n nodes).
        send = tuple(np.zeros((2 * case["n"],) + tail, dt)
                     for tail, dt in (((), np.uint64), ((), np.uint8), ((), np.float64), ((3,), np.float64)))
        return dict(case=case, ctx=ctx, boxes=bh.let_bucket_boxes(s["buckets"], 18, s["bbox"]), send=send, **s)
    pos, vel, mass, ids = _system(seed, case["n"], case["outer"], case["trojan"])
    ctx = bh.Context(case["n"])
    state = dict(case=case, ctx=ctx, t=0.0)
    if kind == "stages":
        return dict(state, pos=pos, vel=vel, mass=mass, ids=ids)
    n = case["n"]
    state["out"] = out = (_pinned((n, 3)), _pinned((n, 3)), _pinned((n,)), _pinned((n,), torch.int64).view(np.uint64),
                          _pinned((n, 3)))
    if kind == "host":
        for dst, src in zip(out, (pos, vel, mass, ids, np.zeros((n, 3)))):
            dst[...] = src
        return state
    ctx.set_bodies(pos, vel, mass, ids)
    if case["mode"] == "learned":
        ctx.learned_set_model(*_model(seed), case["budget"], 3.0)
    return state


# ---------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        params, scale, losses = bh.mlp_train(state["features"], state["labels"], epochs=case["epochs"],
                                             batch=case["batch"], seed=state["seed"])
        return {"params": params, "scale": scale, "losses": losses}
    ctx = state["ctx"]
    if kind == "let":
        ctx.build_tree(merge=False)
        records = ctx.let_export(state["boxes"], state["bbox"], case["theta"] ** 2)
        for dst, src in zip(state["send"], records):
            dst[:len(src)] = src
        acc = ctx.let_accelerations(*state["rec"], theta=case["theta"], G=G)
        prefix, depth, mass, com = state["send"]
        return {"count": len(records[0]), "prefix": prefix.view(np.int64), "depth": depth, "mass": mass, "com": com,
                "acc": acc}
    mode, theta = MODES[case["mode"]], case["theta"]
    if kind == "stages":
        ctx.set_bodies(state["pos"], state["vel"], state["mass"], state["ids"])
        box = ctx.compute_bbox()
        keys = ctx.compute_keys()
        perm = ctx.sort_bodies()
        ctx.build_tree()
        return {"bbox": box, "keys": keys.view(np.int64), "perm": perm,
                "acc": bh.computeAccelerations(ctx, theta, G, 0.0, mode)}
    pos, vel, mass, ids, acc = state["out"]
    if kind == "host":
        state["t"] = ctx.step_host(pos, vel, mass, ids, acc, DT, theta, G, case["nsteps"], mode, state["t"])
    else:
        state["t"] = ctx.step(DT, theta, G, case["nsteps"], mode, state["t"])
        ctx.get_bodies(out=state["out"])
    return {"pos": pos, "vel": vel, "mass": mass, "ids": ids.view(np.int64), "acc": acc}


# --------------------------------------------------------------------- work
def work(case):
    n = case["n"]
    if case["kind"] == "train":
        # Forward and backward: 2 flops per weight and pass, three passes (the
        # first layer needs no input gradient).
        return {"bytes": 36.0 * n + 4.0 * 4801, "flops": case["epochs"] * n * (6.0 * (4096 + 64) + 4.0 * 512)}
    # Interactions per body of the opening test at theta, as measured from 19k
    # to 4M bodies (per-body forms); 20 flops each.
    inter = 24.0 * math.log2(n * case.get("ranks", 1)) / max(case["theta"], 0.3) ** 2
    steps = case.get("nsteps", 1)
    # A step reads position, velocity, acceleration, mass and id, and writes
    # them: 2 x 88 bytes; what goes over the host boundary comes on top.
    host = {"steps": 88.0, "host": 176.0, "stages": 64.0 + 40.0, "let": 24.0}[case["kind"]]
    return {"bytes": n * (176.0 * steps + host), "flops": 20.0 * inter * n * steps}


# -------------------------------------------------------------------- exact
def _direct(xt, xs, ms):
    """Direct-sum accelerations of xt from the masses ms at xs, in 64 bits."""
    out = torch.empty_like(xt)
    rows = max(1, min(len(xt), (1 << 27) // max(1, len(xs))))
    for k in range(0, len(xt), rows):
        d = [xs[None, :, a] - xt[k:k + rows, None, a] for a in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        w = torch.where(r2 > 0, G * ms[None] / (r2 * torch.sqrt(r2)), torch.zeros_like(r2))
        for a in range(3):
            out[k:k + rows, a] = (w * d[a]).sum(1)
    return out


def exact(case, seed):
    """The same step by direct summation in 64 bits (the tree's own
    approximation is part of every side's distance from it)."""
    kind, n = case["kind"], case["n"]
    if kind == "train" or case.get("nsteps", 1) * float(n) ** 2 > 4e11:
        return None
    dev = _device()
    if kind == "let":
        s = _let_inputs(case, seed)
        pos = torch.from_numpy(s["pos"]).to(dev)
        box = torch.from_numpy(s["bbox"]).to(dev)
        order = torch.sort(_keys(pos, box[:3], box[3:]), stable=True).indices
        x, m = pos[order], torch.from_numpy(s["mass"]).to(dev)[order]
        acc = _direct(x, x, m) + _direct(x, torch.from_numpy(s["rec"][3]).to(dev),
                                         torch.from_numpy(s["rec"][2]).to(dev))
        return {"count": None, "prefix": None, "depth": None, "mass": None, "com": None, "acc": acc}
    x, v, m, ids = (torch.from_numpy(a.view(np.int64) if a.dtype == np.uint64 else a).to(dev)
                    for a in _system(seed, n, case["outer"], case["trojan"]))
    if kind == "stages":
        lo, hi = x.min(0).values, x.max(0).values
        key = _keys(x, lo, hi)
        order = torch.sort(key, stable=True).indices
        acc = _direct(x[order], x[order], m[order])
        return {"bbox": torch.cat([lo, hi]), "keys": key, "perm": order, "acc": acc}
    a, t = torch.zeros_like(x), 0.0
    for _ in range(case["nsteps"]):
        if t > 0:
            v = v + 0.5 * DT * a
        x = x + DT * v
        order = torch.sort(_keys(x, x.min(0).values, x.max(0).values), stable=True).indices
        x, v, m, ids = x[order], v[order], m[order], ids[order]
        a = _direct(x, x, m)
        v = v + 0.5 * DT * a
        t += DT
    return {"pos": x, "vel": v, "mass": m, "ids": ids, "acc": a}
