"""The work a user of this framework has it do, as timed cases.

Every case goes through the package's public entry points the way a program calls them:
a plan, network, ensemble or store is made once (`prepare`), and `run` is one pass on it:
some steps of a simulation, one training epoch, one prediction, one sample of observables,
one grid build with its broad phase. Passes continue where the last one stopped.

Kinds and their ranges (`draw` takes one of them):
  network   one dense contractile network of the benchmark's composition at its density,
            500 to 500,000 rods, 1 to 20 steps a call, FP32 or FP64 rod centres
  sweep     networks of a parameter sweep packed into one batch, 2 to 16 of them
  turnover  one network with actin turnover, 2,000 to 40,000 rods, across a biochem cadence
  free      free Brownian rods, 256 to 250,000, all three noise sources
  fit       one epoch of the surrogate ensemble's training
  predict   the trained ensemble on 500 to 150,000 points
  observe   contraction, stress and cluster observables of a packed batch
  pairs     body cells, grid build and broad phase over one network's body view
"""
import functools
import math

import numpy as np
import torch

from softbox_b200 import ensemble, scenes
from softbox_b200.batch import BatchedNetworks
from softbox_b200.engine import DenseNetwork, FreeRods, TurnoverNetwork
from softbox_b200.observables import Observables
from softbox_b200.surrogate import MLPEnsemble
from softbox_b200.systems import SpatialGrid


def listed():
    return [
        # an interactive program that steps a small network and looks at it each time: the
        # smallest call there is
        {"name": "network of 1,000 rods, one step", "kind": "network", "rods": 1000, "steps": 1, "fp64": False},
        # the benchmark network, as in the contractile runs: many steps between looks
        {"name": "network of 20,000 rods", "kind": "network", "rods": 20000, "steps": 20, "fp64": True},
        # the scale sweep's middle sizes
        {"name": "network of 99,370 rods", "kind": "network", "rods": 99370, "steps": 8, "fp64": True},
        {"name": "network of 500,000 rods", "kind": "network", "rods": 500000, "steps": 2, "fp64": True},
        # a parameter sweep: networks of uneven size advanced together
        {"name": "sweep of 12 networks", "kind": "sweep", "nets": 12, "points": 3, "steps": 4},
        # a run with growth, severing and births: one cadence of 100 steps
        {"name": "turnover, 20,000 rods", "kind": "turnover", "rods": 20000, "steps": 100},
        # the free-diffusion check of the method: few rods, many steps, counter-based noise
        {"name": "1,024 free rods", "kind": "free", "rods": 1024, "steps": 1000, "noise": "philox", "fp64": False},
        # the same at ensemble size, with the reference's draws
        {"name": "150,001 free rods", "kind": "free", "rods": 150001, "steps": 20, "noise": "wang", "fp64": True},
        # the surrogate of the sweep: one epoch on 4,096 runs, and 100,000 fresh points
        {"name": "surrogate epoch", "kind": "fit", "points": 4096, "nets": 5, "batch": 256},
        {"name": "surrogate on 100,000 points", "kind": "predict", "points": 100000, "nets": 5},
        # what a sweep reads between its runs of steps
        {"name": "observables of 12 networks", "kind": "observe", "nets": 12, "points": 3},
        # candidate pairs of one body view, by the grid
        {"name": "pairs of 132,000 bodies", "kind": "pairs", "rods": 100000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["network", "network", "network", "sweep", "turnover", "free", "free", "fit", "predict",
                       "observe", "pairs"])
    if kind == "network":
        rods = _log(rng, 500, 400000)
        most = max(1, min(20, 900000 // rods))
        return {"kind": kind, "rods": rods, "steps": rng.randint(1, most), "fp64": rng.random() < 0.7}
    if kind == "sweep":
        return {"kind": kind, "nets": rng.randint(2, 12), "points": rng.randrange(1000), "steps": rng.randint(1, 4)}
    if kind == "turnover":
        return {"kind": kind, "rods": _log(rng, 2000, 40000), "steps": rng.randint(20, 100)}
    if kind == "free":
        rods = _log(rng, 256, 250000)
        return {"kind": kind, "rods": rods, "steps": rng.randint(10, max(11, min(1000, 3000000 // rods))),
                "noise": rng.choice(["wang", "philox", "supplied"]), "fp64": rng.random() < 0.5}
    if kind == "fit":
        return {"kind": kind, "points": _log(rng, 512, 4096), "nets": rng.randint(3, 8),
                "batch": rng.choice([64, 128, 256])}
    if kind == "predict":
        return {"kind": kind, "points": _log(rng, 500, 150000), "nets": rng.randint(3, 8)}
    if kind == "observe":
        return {"kind": kind, "nets": rng.randint(2, 16), "points": rng.randrange(1000)}
    return {"kind": kind, "rods": _log(rng, 1000, 200000)}


# ---------------------------------------------------------------- inputs
# Building a large network on the host takes seconds, so one network of each size is kept
# and a state is a replicate of it: the same geometry with random draws of its own seed,
# advanced until heads have bound.
@functools.lru_cache(maxsize=4)
def _network(rods):
    return scenes.dense_contractile(scenes.dense_scaled(rods))


@functools.lru_cache(maxsize=4)
def _packed(nets, points):
    return ensemble.build_batch(ensemble.sample_points(nets, points))


def _seeds(seed, n):
    return np.random.default_rng(seed).integers(1, 2**31 - 1, n)


def _replicate(rods, seed):
    base = _network(rods)
    s = [int(x) for x in _seeds(seed, 3)]
    fil = dict(base["fil"], counts=base["fil"]["counts"].copy())
    fil["counts"][2] = s[2]
    return dict(base, fil=fil, seed=s[0], seedBb=s[1])


def _batch(case, seed):
    packed, info = _packed(case["nets"], case["points"])
    seeds = _seeds(seed, 3 * case["nets"]).astype(np.int32)
    return BatchedNetworks(dict(packed, batch=dict(packed["batch"], seeds=seeds)), info, fp64_coords=True)


def _surrogate_points(n, seed):
    """Sweep parameters scaled to [0, 1] and smooth observables of them with noise."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(size=(n, 6))
    y = np.stack([np.sin(3 * x[:, 0]) + x[:, 1] * x[:, 2], 1 + 2 * np.exp(-x[:, 3]),
                  2 + x[:, 4] - x[:, 5] ** 2], axis=1)
    return x, y + 0.05 * rng.standard_normal(y.shape)


def _warm_steps(rods):
    return max(20, min(400, 4000000 // rods))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "network":
        net = DenseNetwork(_replicate(case["rods"], seed), fp64_coords=case["fp64"])
        t = _warm_steps(case["rods"])
        net.run(0, t)
        return {"case": case, "net": net, "t": t}
    if kind == "sweep":
        net = _batch(case, seed)
        net.run(0, 20)
        return {"case": case, "net": net, "t": 20}
    if kind == "turnover":
        s = [int(x) for x in _seeds(seed, 4)]
        cfg = scenes.dense_scaled(case["rods"], seed=s[0], seed_bb=s[1], seed_fil=s[2])
        net = TurnoverNetwork(scenes.dense_turnover(cfg, turnover_seed=s[3]), fp64_coords=True)
        net.run(0, 250)
        return {"case": case, "net": net, "t": 250}
    if kind == "free":
        rods = FreeRods(scenes.free_rods_box(n=case["rods"], box_um=10.0 * (case["rods"] / 1024) ** (1 / 3), seed=seed),
                        fp64_coords=case["fp64"])
        state = {"case": case, "rods": rods, "t": 0, "philox": int(_seeds(seed, 1)[0]), "noise": None}
        if case["noise"] == "supplied":
            g = torch.Generator(device="cuda").manual_seed(seed)
            state["noise"] = torch.randn((case["steps"], 6, case["rods"]), device="cuda", generator=g)
        return state
    if kind == "fit":
        x, y = _surrogate_points(case["points"], seed)
        ens = MLPEnsemble(n_nets=case["nets"], batch=case["batch"], seed=seed)
        ens.set_normalisation(x, y)
        return {"case": case, "ens": ens, "x": x, "y": y, "seed": seed}
    if kind == "predict":
        x, y = _surrogate_points(2048, seed)
        ens = MLPEnsemble(n_nets=case["nets"], seed=seed)
        ens.set_normalisation(x, y)
        return {"case": case, "ens": ens, "x": _surrogate_points(case["points"], seed + 1)[0]}
    if kind == "observe":
        net = _batch(case, seed)
        net.run(0, 20)
        return {"case": case, "net": net, "obs": Observables(net)}
    # a body view of the network whose bodies have moved by up to half a rod
    dev = _body_view(case, seed)
    cap = dev["center"].numel() // 3
    dev["candPartner"] = torch.full((cap * SpatialGrid.MAX_CAND,), -1, dtype=torch.int32, device="cuda")
    dev["candCount"] = torch.zeros(cap, dtype=torch.int32, device="cuda")
    return {"case": case, "view": dev}


def _body_view(case, seed):
    sc = _network(case["rods"])
    g, n, nm = sc["grid"], sc["fil"]["body"]["n"], sc["mot"]["nMotors"]
    mb = sc["mot"]["body"]
    rng = np.random.default_rng(seed)
    heads = mb["coord"].reshape(3, -1)[:, 2::3]
    c = np.concatenate([sc["fil"]["body"]["coord"].reshape(3, n), heads], axis=1)
    c = (c + rng.uniform(-0.05, 0.05, c.shape)).astype(np.float32)
    r = np.concatenate([0.5 * sc["fil"]["body"]["segLength"] + np.float32(scenes.ACTIN_RADIUS), sc["mot"]["reach"]])
    host = {"center": c.reshape(-1), "boundingRadius": r.astype(np.float32)}
    for k in ("gridParams", "gridDims", "gridCounts", "bodyCell", "cellCount", "chunkSum", "gridCellOffsets",
              "gridCellContents"):
        host[k] = g[k].copy()
    host["gridCounts"][1] = n + nm
    return {k: torch.from_numpy(v).cuda() for k, v in host.items()}


# ---------------------------------------------------------------- a pass
_BODY = ("coord", "uVec", "yVec", "zVec", "end1", "end2", "forceSum", "torqueSum", "randForce", "randTorque")


def _network_state(d):
    """The stores a program reads back: poses and forces, binding, links, the step's grid."""
    out = {"fil." + k: d["fil"]["body"][k] for k in _BODY}
    out.update({"mot." + k: d["mot"]["body"][k] for k in _BODY})
    out.update({"bb." + k: d["mini"]["backbone"][k] for k in ("coord", "uVec", "forceSum", "torqueSum")})
    out.update({"mot." + k: d["mot"][k] for k in ("boundSeg", "bindArc", "nucleotideState", "forceDotFil", "forceMag",
                                                  "cooldown", "stats")})
    out.update({"xl." + k: d["xl"][k] for k in ("linkState", "xlinkData", "strainHist", "torqueMagHist",
                                                "activeLinkCount", "segOffsetsA", "segIdxA")})
    out.update({"grid." + k: d["grid"][k] for k in ("bodyCell", "gridCellOffsets", "gridCellContents", "reachCount")})
    out.update({k: d[k] for k in ("bondData", "segMotorOffsets", "segMotorCount")})
    for name, b in (("fil", d["fil"]["body"]), ("mot", d["mot"]["body"])):
        if b.get("coord64") is not None:
            out[name + ".coord64"] = b["coord64"]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("network", "sweep", "turnover"):
        net = state["net"]
        net.run(state["t"], case["steps"])
        state["t"] += case["steps"]
        out = _network_state(net.dev)
        if kind == "turnover":
            d = net.dev
            out.update({"fil." + k: d["fil"][k] for k in ("monomerCount", "filState", "end1NbrSlot", "end2NbrSlot")})
            out["pool"] = d["turnover"]["pool"]
        return out
    if kind == "free":
        rods = state["rods"]
        rods.run(state["t"], case["steps"], noise=case["noise"], philox_seed=state["philox"], supplied=state["noise"])
        state["t"] += case["steps"]
        b = rods.dev["body"]
        keys = ("coord", "uVec", "yVec", "zVec", "end1", "end2", "randForce", "randTorque")
        return {k: b[k] for k in keys + (("coord64",) if case["fp64"] else ())}
    if kind == "fit":
        ens = state["ens"]
        loss = ens.fit(state["x"], state["y"], epochs=1, seed=state["seed"])
        return {"loss": loss, "W": ens.W, "b": ens.b, "mW": ens.mW, "mb": ens.mb, "vW": ens.vW, "vb": ens.vb}
    if kind == "predict":
        mean, std, y = state["ens"].predict(state["x"])
        return {"mean": mean, "std": std, "y": y}
    if kind == "observe":
        obs = state["obs"]
        out = obs.sample()
        return dict(out, label=obs.label, size=obs.size)
    v = state["view"]
    SpatialGrid.bodyCell(v["center"], v["gridParams"], v["gridDims"], v["gridCounts"], v["bodyCell"])
    SpatialGrid.build(v["bodyCell"], v["gridCounts"], v["gridDims"], v["cellCount"], v["chunkSum"],
                      v["gridCellOffsets"], v["gridCellContents"])
    SpatialGrid.broadPhase(v["center"], v["boundingRadius"], v["bodyCell"], v["gridCellOffsets"],
                           v["gridCellContents"], v["gridDims"], v["gridParams"], v["gridCounts"], v["candPartner"],
                           v["candCount"])
    return {k: v[k] for k in ("bodyCell", "cellCount", "gridCellOffsets", "gridCellContents", "candPartner",
                              "candCount")}


# ---------------------------------------------------------------- work of a pass
def _net_size(case):
    """(rods, heads, links, backbones) of a network or of a packed batch."""
    if "rods" in case:
        cfg = scenes.dense_scaled(case["rods"])
        return cfg.n_seg, cfg.n_mini * 4 * cfg.dimers_per_end, cfg.n_links, cfg.n_mini
    cfgs = [ensemble.point_config(p) for p in ensemble.sample_points(case["nets"], case["points"])]
    return (sum(c.n_seg for c in cfgs), sum(c.n_mini * 4 * c.dimers_per_end for c in cfgs),
            sum(c.n_links for c in cfgs), sum(c.n_mini for c in cfgs))


def _step_work(case, fp64):
    """One step: poses, drag, scales and topology read once, poses, geometry and forces
    written once; the binding state, the link state and the grid read and written once. Per
    body the draws and the Langevin update take about 400 operations, a chain joint, bond or
    link about 600."""
    n, heads, links, bb = _net_size(case)
    bodies = n + 3 * heads + bb
    body = 4 * (9 + 6 + 3) + 4 * 30 + (48 if fp64 else 0)
    b = bodies * body + n * (16 + 24) + (n + heads) * 4 * 7 + heads * (2 * 4 * 22 + 104 + 48) + links * (2 * 4 * 30 + 20)
    return b, bodies * 400 + (n + 4 * heads + links) * 600


def work(case):
    kind = case["kind"]
    if kind in ("network", "sweep", "turnover"):
        b, f = _step_work(case, case.get("fp64", True))
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "free":
        n, s = case["rods"], case["steps"]
        b = n * 4 * (9 + 6 + 6 + 3 + 24) + (n * 48 if case["fp64"] else 0)
        if case["noise"] == "supplied":
            b += 24 * n * s
        return {"bytes": b, "flops": n * s * (130 if case["noise"] == "supplied" else 430)}
    params = 6 * 256 + 3 * 256 * 256 + 256 * 3
    if kind == "fit":
        steps = case["points"] // case["batch"]
        rows = steps * case["batch"]
        return {"bytes": case["nets"] * (steps * params * 28 + rows * 36), "flops": 6.0 * params * rows * case["nets"]}
    if kind == "predict":
        n, z = case["points"], case["nets"]
        return {"bytes": n * (48 + 24 * (2 + z)) + z * params * 2, "flops": 2.0 * params * n * z}
    if kind == "observe":
        n, heads, links, bb = _net_size(case)
        return {"bytes": n * (24 + 4 + 4 + 8) + links * (12 + 8 + 8 + 48) + heads * (8 + 8) + 8 * (n + bb),
                "flops": 10.0 * n + 20.0 * links}
    n, heads, _, _ = _net_size(case)
    cap = n + heads
    return {"bytes": cap * (16 + 8 + 8 + 4 + 4 * 12), "flops": cap * 36 * 10.0}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    """What `run` returns for these inputs, in 64-bit arithmetic. A network's step is left
    out: its dozen force laws, each with thresholds that decide binding and release, have no
    short plain form. The outputs of `pairs` are whole numbers."""
    kind = case["kind"]
    if kind == "free":
        return _exact_free(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "predict":
        s = prepare(case, seed)
        ens = s["ens"]
        x = torch.from_numpy((s["x"] - ens.x_mean) / ens.x_std).cuda()
        y = torch.stack([_mlp([w[z].double() for w in ens.W], [b[z].double() for b in ens.b], x)
                         for z in range(case["nets"])])[:, :, :3].cpu().numpy() * ens.y_std + ens.y_mean
        return {"mean": y.mean(axis=0), "std": y.std(axis=0), "y": y}
    if kind == "observe":
        return _exact_observe(case, seed)
    return None


def _mlp(W, b, x):
    a = x
    for l, (w, c) in enumerate(zip(W, b)):
        k = a.shape[1]
        a = a @ w[:, :k].T + c
        if l < len(W) - 1:
            a = torch.nn.functional.gelu(a)
    return a


def _exact_fit(case, seed):
    s = prepare(case, seed)
    ens = s["ens"]
    x = torch.from_numpy((s["x"] - ens.x_mean) / ens.x_std).cuda()
    y = torch.from_numpy((s["y"] - ens.y_mean) / ens.y_std).cuda()
    n, B, nz = case["points"], case["batch"], case["nets"]
    g = torch.Generator(device="cpu").manual_seed(seed)
    perms = [torch.randperm(n, generator=g).cuda() for _ in range(nz)]
    par = [[w[z].double().clone().requires_grad_() for w in ens.W] + [c[z].double().clone().requires_grad_()
                                                                      for c in ens.b] for z in range(nz)]
    m = [[torch.zeros_like(p) for p in q] for q in par]
    v = [[torch.zeros_like(p) for p in q] for q in par]
    L = len(ens.W)
    loss = 0.0
    for k in range(max(1, n // B)):
        loss = 0.0
        for z in range(nz):
            idx = perms[z][k * B:(k + 1) * B]
            e = (_mlp(par[z][:L], par[z][L:], x[idx])[:, :3] - y[idx]).square().mean()
            loss += float(e) / nz
            for p, q, r, gr in zip(par[z], m[z], v[z], torch.autograd.grad(e, par[z])):
                q.mul_(0.9).add_(0.1 * gr)
                r.mul_(0.999).add_(0.001 * gr * gr)
                with torch.no_grad():
                    p -= ens.lr * (q / (1 - 0.9 ** (k + 1))) / ((r / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)

    def layers(lists, first):
        return [torch.stack([q[first + l].detach() for q in lists]) for l in range(L)]

    return {"loss": [loss], "W": layers(par, 0), "b": layers(par, L), "mW": layers(m, 0), "mb": layers(m, L),
            "vW": layers(v, 0), "vb": layers(v, L)}


def _exact_observe(case, seed):
    s = prepare(case, seed)
    d, info = s["net"].dev, s["net"].info
    seg, nets = info["seg"], case["nets"]
    c = d["fil"]["body"]["coord64"].cpu().numpy().reshape(3, -1)
    rms = np.array([np.sqrt(((c[:, a:b] - c[:, a:b].mean(axis=1, keepdims=True)) ** 2).sum(axis=0).mean())
                    for a, b in zip(seg[:-1], seg[1:])])
    f64 = lambda x: x.cpu().numpy().astype(np.float64)  # noqa: E731
    fb, xl, mot = d["fil"]["body"], d["xl"], d["mot"]
    fc, fu, e1 = (f64(fb[k]).reshape(3, -1) for k in ("coord", "uVec", "end1"))
    A, B, on = xl["linkFilA"].cpu().numpy(), xl["linkFilB"].cpu().numpy(), xl["linkState"].cpu().numpy() >= 0
    pay = f64(xl["xlinkData"]).reshape(-1, 12)
    r = (e1[:, A] + f64(xl["loc1"]) * fu[:, A]) - (e1[:, B] + f64(xl["loc2"]) * fu[:, B])
    wl = np.where(on, 1e-6 * (r[0] * pay[:, 0] + r[1] * pay[:, 1]), 0.0)
    bs = mot["boundSeg"].cpu().numpy()
    hc, hu = (f64(mot["body"][k]).reshape(3, -1)[:, 2::3] for k in ("coord", "uVec"))
    bd = f64(d["bondData"]).reshape(-1, 13)
    at = fc[:, bs] + (f64(mot["bindArc"]) - 0.5 * f64(fb["segLength"])[bs]) * fu[:, bs]
    q = hc + 0.01 * hu - at
    wm = np.where(bs >= 0, 1e-6 * (q[0] * bd[:, 0] + q[1] * bd[:, 1]), 0.0)
    box = d["batch"]["boxParams"].cpu().numpy().astype(np.float64).reshape(-1, 8)
    lk, mt = info["link"], info["mot"]
    stress = np.array([-(wl[lk[k]:lk[k + 1]].sum() + wm[mt[k]:mt[k + 1]].sum()) /
                       (2e-18 * box[k, 1] * box[k, 2] * box[k, 3]) for k in range(nets)])
    rods = np.diff(seg).astype(np.float64)
    return {"rms_um": rms, "rods": rods, "largest": None, "active": None, "largest_fraction": None,
            "stress_pa": stress, "label": None, "size": None}


def _wang(s):
    s = (s ^ np.uint32(61)) ^ (s >> np.uint32(16))
    s = s * np.uint32(9)
    s = s ^ (s >> np.uint32(4))
    s = s * np.uint32(0x27D4EB2D)
    return s ^ (s >> np.uint32(15))


def _philox(i, step, word, seed):
    c = [i.astype(np.uint64), np.full(i.size, step, np.uint64), np.full(i.size, word, np.uint64),
         np.full(i.size, 0x53425830, np.uint64)]
    k0, k1, low = seed & 0xFFFFFFFF, seed >> 32, np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [x.astype(np.uint32) for x in c]


def _gaussians(case, state, i, t, seed):
    """The step's six Gaussians of every rod: Box-Muller on six uniforms of the counter."""
    if case["noise"] == "supplied":
        return state["noise"][t].double().cpu().numpy()
    if case["noise"] == "wang":
        base = (i * np.uint32(1000003)) ^ np.uint32(t * 999983 & 0xFFFFFFFF) ^ np.uint32(seed * 7919 & 0xFFFFFFFF)
        h = [_wang(base ^ np.uint32(k)) for k in (0, 0x9E3779B9, 0x85EBCA6B, 0xC2B2AE35, 0x517CC1B7, 0x1F0A7ED5)]
    else:
        a, b = (_philox(i, t, w, state["philox"]) for w in (0, 1))
        h = [a[0], a[1], a[2], a[3], b[0], b[1]]
    # the uniforms are single-precision values by definition
    u = [((x >> np.uint32(1)).astype(np.int32).astype(np.float32) / np.float32(2147483648.0)).astype(np.float64) for x in h]
    out = [None] * 6
    for k in range(3):
        r = np.sqrt(-2 * np.log(np.maximum(np.float64(np.float32(1e-7)), u[2 * k])))
        out[k], out[3 + k] = r * np.cos(2 * np.pi * u[2 * k + 1]), r * np.sin(2 * np.pi * u[2 * k + 1])
    return np.stack(out)


def _cross(a, b):
    return np.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _exact_free(case, seed):
    state = prepare(case, seed)
    d = state["rods"].dev
    b = {k: v.double().cpu().numpy() for k, v in d["body"].items() if torch.is_tensor(v)}
    n = case["rods"]
    c, u, y = (b[k].reshape(3, n).copy() for k in ("coord", "uVec", "yVec"))
    gT, gR = b["bTransGam"].reshape(3, n), b["bRotGam"].reshape(3, n)
    dt, mag = (float(v) for v in d["params"])
    i = np.arange(n, dtype=np.uint32)
    key = int(d["counts"][2])
    unit = lambda v: v / np.sqrt((v * v).sum(axis=0))  # noqa: E731
    z = rf = rt = None
    for t in range(case["steps"]):
        g = _gaussians(case, state, i, t, key)
        rf, rt = b["brownTransScale"] * mag * np.sqrt(gT) * g[:3], b["brownRotScale"] * mag * np.sqrt(gR) * g[3:]
        z = unit(_cross(u, y))
        vel, w = 1e6 * rf / gT, rt / gR
        c += dt * (u * vel[0] + y * vel[1] + z * vel[2])
        nu = unit(u + y * (w[2] * dt) - z * (w[1] * dt))
        ny = unit(-u * (w[2] * dt) + y + z * (w[0] * dt))
        u, z = nu, unit(_cross(nu, ny))
        y = _cross(z, u)
    half = 0.5 * b["segLength"]
    flat = lambda v: v.reshape(-1)  # noqa: E731
    out = {"coord": flat(c), "uVec": flat(u), "yVec": flat(y), "zVec": flat(z), "end1": flat(c - half * u),
           "end2": flat(c + half * u), "randForce": flat(rf), "randTorque": flat(rt)}
    if case["fp64"]:
        out["coord64"] = flat(c)
    return out
