"""The workloads whose speed this framework answers for.

Each case is one call, or the few calls in a row, that a program using the
library makes: the drop-in pair make_tree + biot_tree_batch on host arrays, a
device-resident solve in the plain, mixed or learned form, a batch of
independent sets, a time step, the FP64 direct sum, and the training of the
order selector.  Blob sets are the benchmark's distributions
(2dfmm_gb300/workloads.py), drawn on the GPU from a seed.
"""
import importlib
import math

import numpy as np
import torch

P = importlib.import_module("2dfmm_gb300")
LEARN = importlib.import_module("2dfmm_gb300.learn")

MODES = {"plain": P.MODE_PLAIN, "mixed": P.MODE_MIXED, "learned": P.MODE_LEARNED}

# Most target-source pairs of the 64-bit yardstick (a few seconds on the GPU).
EXACT_PAIRS = 4.5e10


def _tree(name, call, mode, dist, n, nterms=13, num_p=65, theta=0.5, points=0, pinned=False):
    c = dict(call=call, mode=mode, dist=dist, n=n, nterms=nterms, num_p=num_p, theta=theta, points=points, pinned=pinned)
    return dict(c, name=name) if name else c


def listed():
    return [
        # An embedding without an allocator of its own solves a young wake: a
        # few thousand blobs, where only latency counts.
        _tree("static_plain_4k", "static", "plain", "uniform", 4096, 11, 33),
        # The vortex solver's call, unchanged: make_tree on its host arrays,
        # then the velocity at every blob (the 20,000-blob benchmark set).
        _tree("dropin_plain_20k", "host", "plain", "uniform", 20_000, 11, 33),
        # The same solver with the parameters it ships (15 terms, 250 blobs a
        # leaf) at its snapshot's size, asking for its body panels too: points
        # off the blobs.
        _tree("dropin_plain_27743_panels", "host", "plain", "lamb_oseen", 27_743, 15, 250, points=2001),
        # A large run of the reference's method, device-resident.
        _tree("plain_lamb_oseen_1m", "device", "plain", "lamb_oseen", 1_048_576),
        # A mid-size run in the mixed form, at an odd size.
        _tree("mixed_uniform_50k", "device", "mixed", "uniform", 50_021, 11, 33),
        # A mixed run that also samples the flow field around the blobs (a
        # plot's grid or a body's surface): points off the blobs.
        _tree("mixed_262k_field_points", "host", "mixed", "two_patch_sheet", 262_144, points=65_537),
        # The headline set: two patches and a sheet, 4 Mi blobs.
        _tree("mixed_two_patch_4m", "device", "mixed", "two_patch_sheet", 4_194_304),
        # The headline set end to end in the learned form, from page-locked
        # host buffers and back.
        _tree("dropin_learned_4m", "host", "learned", "two_patch_sheet", 4_194_304, pinned=True),
        # The first half of a two-stage time step in the learned form: the
        # velocities, then the positions half a step on.
        _tree("learned_stage_1m", "stage", "learned", "lamb_oseen", 1_048_576),
        # An ensemble in one call: 512 sets of 2,048 to 200,000 blobs.
        dict(name="sets_512", call="sets", mode="mixed", nsets=512, lo=2048, hi=200_000, nterms=11, num_p=33, theta=0.5),
        # The yardstick: the FP64 direct sum at sampled targets.
        dict(name="direct_16k_of_262k", call="direct", dist="two_patch_sheet", ntgt=16_384, nsrc=262_144),
        # Training the order selector, as a loop does that looks at its loss
        # every 20 steps: 200,000 samples, mini-batches of 4,096.
        dict(name="train_20_steps", call="train", samples=200_000, steps=20, batch=4096),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "host", "host", "points", "device", "device", "mixed", "mixed", "learned", "stage", "sets",
                       "direct", "train"])
    dist = rng.choice(["uniform", "lamb_oseen", "two_patch_sheet"])
    theta = rng.choice([0.4, 0.5, 0.5, 0.6, 0.7])
    nterms = rng.choice([5, 9, 11, 13, 13, 15, 17, 21])
    num_p = rng.choice([17, 33, 65, 65, 129, 251])
    if kind == "static":
        return _tree(None, "static", "plain", dist, _logint(rng, 500, 65_536), nterms, num_p, max(theta, 0.5))
    if kind == "host":
        return _tree(None, "host", "plain", dist, _logint(rng, 1000, 200_000), nterms, num_p, theta)
    if kind == "points":
        return _tree(None, "host", rng.choice(["plain", "mixed", "learned"]), dist, _logint(rng, 2000, 200_000), nterms,
                     num_p, theta, _logint(rng, 100, 50_000))
    if kind == "device":
        return _tree(None, "device", "plain", dist, _logint(rng, 1000, 300_000), nterms, num_p, theta)
    if kind in ("mixed", "learned"):
        return _tree(None, "device", kind, dist, _logint(rng, 2000, 4_000_000))
    if kind == "stage":
        return _tree(None, "stage", rng.choice(["mixed", "learned", "learned"]), dist, _logint(rng, 20_000, 1_000_000))
    if kind == "sets":
        nsets = _logint(rng, 3, 300)
        return dict(call="sets", mode="mixed", nsets=nsets, lo=_logint(rng, 500, 4000), hi=_logint(rng, 8000, 100_000),
                    nterms=11, num_p=33, theta=0.5)
    if kind == "direct":
        return dict(call="direct", dist=dist, ntgt=_logint(rng, 500, 16_384), nsrc=_logint(rng, 2000, 260_000))
    return dict(call="train", samples=_logint(rng, 5000, 200_000), steps=rng.randint(4, 20), batch=_logint(rng, 256, 4096))


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _blobs(dist, n, g):
    """(xy, cir, cor) on the GPU, float64: the distributions of workloads.py."""
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)    # noqa: E731
    randn = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    if dist == "uniform":
        xy, cir, sigma = rand(n, 2), randn(n) / n, 0.005
    elif dist == "lamb_oseen":
        r = 0.1 * torch.sqrt(-2.0 * torch.log1p(-rand(n)))
        a = rand(n) * (2.0 * math.pi)
        xy = torch.stack([0.5 + r * torch.cos(a), 0.5 + r * torch.sin(a)], dim=1)
        cir = torch.exp(-r * r / 0.02)
        cir, sigma = cir / cir.sum(), 0.002
    else:
        n1 = int(round(0.45 * n))
        ns = n - 2 * n1
        sx = rand(ns)
        patches = 0.05 * randn(2 * n1, 2) + 0.5
        patches[:n1, 0] -= 0.1
        patches[n1:, 0] += 0.1
        xy = torch.cat([patches, torch.stack([sx, 0.2 + 0.01 * torch.sin(8.0 * math.pi * sx)], dim=1)])
        cir = torch.cat([randn(2 * n1).abs(), torch.full((ns,), -1.0 / ns, device="cuda", dtype=torch.float64)])
        xy, cir, sigma = xy.float().double(), cir.float().double(), float(np.float32(0.001))
    return xy.contiguous(), cir.contiguous(), torch.full((n,), sigma, device="cuda", dtype=torch.float64)


def _points(m, g):
    """Query points off the blobs: the unit square and a little around it."""
    return torch.rand(m, 2, generator=g, device="cuda", dtype=torch.float64) * 1.1 - 0.05


def _sizes(case):
    k = (np.arange(case["nsets"]) + 0.5) / case["nsets"]
    return (case["lo"] * (case["hi"] / case["lo"]) ** k).astype(np.int64)


def _make(case, seed):
    """The case's arrays on the GPU."""
    g = _generator(seed)
    if case["call"] == "sets":
        sizes = _sizes(case)
        sizes = sizes[torch.randperm(len(sizes), generator=g, device="cuda").cpu().numpy()]
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
        per = torch.repeat_interleave(torch.from_numpy(sizes).cuda().double(), torch.from_numpy(sizes).cuda())
        n = int(off[-1])
        xy = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
        cir = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) / per
        return dict(xy=xy, cir=cir, cor=0.5 / torch.sqrt(per), off=off)
    if case["call"] == "train":
        # the features' ranges, and labels that depend on them
        X = torch.randn(case["samples"], 16, generator=g, device="cuda")
        X[:, 12:] = 0.0
        y = torch.clamp((X[:, 0] * 3 + X[:, 1] * 2 + 2).round(), 0, 13).int()
        y = torch.where(torch.rand(len(y), generator=g, device="cuda") < 0.7, torch.zeros_like(y), y)
        theta = torch.zeros(P.learn_param_count(), device="cuda")
        at = 0
        for rows, cols in ((64, 16), (64, 64), (64, 64), (16, 64)):
            w = torch.randn(rows * cols, generator=g, device="cuda") * math.sqrt(2.0 / cols)
            theta[at:at + rows * cols] = w
            at += rows * cols + rows
        return dict(X=X.cpu().numpy(), y=y.cpu().numpy(), theta=theta.cpu().numpy())
    n = case["nsrc"] if case["call"] == "direct" else case["n"]
    xy, cir, cor = _blobs(case["dist"], n, g)
    d = dict(xy=xy, cir=cir, cor=cor)
    if case["call"] == "direct":
        d["txy"] = xy[torch.randperm(n, generator=g, device="cuda")[: min(n, case["ntgt"])]].contiguous()
    elif case["points"]:
        d["points"] = _points(case["points"], g)
    return d


def _host(t, pinned):
    return t.cpu().pin_memory().numpy() if pinned else t.cpu().numpy()


def prepare(case, seed):
    s = dict(_make(case, seed), case=case)
    call = case["call"]
    if call == "train":
        return s
    if call == "direct":
        s["uv"] = torch.empty_like(s["txy"])
        return s
    # what the program sets once, at its start
    P.set_params(case["nterms"], case["num_p"], case["theta"])
    P.set_mode(MODES[case["mode"]])
    if case["mode"] == "learned":
        P.learn_set_weights(LEARN.load_weights())
        P.learn_set_envelope(*LEARN.load_envelope())
    if call == "host":
        for k in ("xy", "cir", "cor", "points"):
            if k in s:
                s[k] = _host(s[k], case["pinned"])
        if case["pinned"]:
            s["uv"] = torch.empty(case["n"], 2, dtype=torch.float64).pin_memory().numpy()
    else:
        s["uv"] = torch.empty_like(s["xy"])
        if call == "stage":
            s["stage"] = torch.empty_like(s["xy"])
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run

def run(s):
    case = s["case"]
    call = case["call"]
    if call == "train":
        P.learn_set_weights(s["theta"])
        loss = P.learn_train(s["X"], s["y"], steps=case["steps"], batch=case["batch"], lr=2e-3, seed=1)
        return {"theta": P.learn_get_weights(), "loss": np.array([loss], np.float32)}
    if call == "host":
        P.make_tree(s["xy"], s["cir"], s["cor"])
        r = {"uv": P.biot_tree_batch(s["xy"], out=s.get("uv"))}
        if "points" in s:
            r["points"] = P.biot_tree_batch(s["points"])
        return r
    stream = torch.cuda.current_stream().cuda_stream
    a = [s[k].data_ptr() for k in ("xy", "cir", "cor")]
    if call == "direct":
        P.direct_device(s["txy"].data_ptr(), len(s["txy"]), a[0], a[1], a[2], len(s["cir"]), s["uv"].data_ptr(), stream)
        return s["uv"]
    if call == "sets":
        P.solve_sets(a[0], a[1], a[2], s["uv"].data_ptr(), s["off"], stream)
        return s["uv"]
    n = case["n"]
    if call == "static":
        rc = P.solve_device_static(a[0], a[1], a[2], s["uv"].data_ptr(), n, stream)
        if rc != P.OK:
            raise P.Tree2DError(rc, "solve_device_static")
        return s["uv"]
    P.solve_device(a[0], a[1], a[2], s["uv"].data_ptr(), n, stream)
    if call == "stage":
        s["stage"].copy_(s["xy"])
        P.advect_device(s["stage"].data_ptr(), s["uv"].data_ptr(), n, 0.5e-3, stream)
        return {"uv": s["uv"], "stage": s["stage"]}
    return s["uv"]


# -------------------------------------------------------------------- work

def work(case):
    """Bytes of the inputs and outputs, and the method's arithmetic: for the
    plain treecode about 3 pi / theta^2 accepted cells per level and
    pi / theta^2 leaves per target; for the mixed form nine leaves of pairs
    and the expansions."""
    call = case["call"]
    if call == "train":
        rows = case["steps"] * case["batch"]
        weights = 16 * 64 + 2 * 64 * 64 + 64 * 16
        return {"bytes": 68 * case["samples"] + 8 * 10448, "flops": 6 * weights * rows}
    if call == "direct":
        t = min(case["ntgt"], case["nsrc"])
        return {"bytes": 32 * case["nsrc"] + 32 * t, "flops": 20.0 * t * case["nsrc"]}
    n = int(_sizes(case).sum()) if call == "sets" else case["n"]
    m = 0 if call == "sets" else case["points"]
    bytes_ = 48 * n + 32 * m
    if call == "host":
        bytes_ += 16 * n  # the positions again, as query points
    if call == "stage":
        bytes_ += 16 * n
    if case["mode"] == "plain":
        leaf = max(1.0, 0.5 * case["num_p"])
        levels = max(1.0, math.log(max(4.0, n / leaf), 4.0))
        cells = 3.0 * math.pi / case["theta"] ** 2 * max(0.0, levels - 1.0)
        pairs = min(float(n), math.pi / case["theta"] ** 2 * leaf)
        per = cells * (8 * (case["nterms"] - 1) + 10) + 20 * pairs
    else:
        per = 20.0 * 9 * 64 + 8 * 16 * 4
    return {"bytes": bytes_, "flops": per * (n + m)}


# ------------------------------------------------------------------- exact

def _direct64(t, xy, cir, cor):
    """The sum that every form of the library approximates, in float64: blobs
    closer than 1e-10 left out."""
    out = torch.empty_like(t)
    step = max(1, (1 << 25) // len(xy))
    for b in range(0, len(t), step):
        rx = t[b:b + step, 0:1] - xy[:, 0]
        ry = t[b:b + step, 1:2] - xy[:, 1]
        r2 = rx * rx + ry * ry
        f = -torch.expm1(-r2 / (cor * cor)) / r2 * cir
        f = torch.where(r2 > 1e-20, f, torch.zeros_like(f))
        out[b:b + step, 0] = -(f * ry).sum(1) * (0.5 / math.pi)
        out[b:b + step, 1] = (f * rx).sum(1) * (0.5 / math.pi)
    return out


def exact(case, seed):
    call = case["call"]
    if call == "train":
        return None  # a chain of Adam steps has no value of its own in other bits
    if call == "direct":
        pairs = min(case["ntgt"], case["nsrc"]) * case["nsrc"]
    elif call == "sets":
        pairs = float((_sizes(case).astype(np.float64) ** 2).sum())
    else:
        pairs = float(case["n"] + case["points"]) * case["n"]
    if pairs > EXACT_PAIRS:
        return None
    d = _make(case, seed)
    if call == "direct":
        return _direct64(d["txy"], d["xy"], d["cir"], d["cor"])
    if call == "sets":
        o = d["off"]
        return torch.cat([_direct64(d["xy"][b:e], d["xy"][b:e], d["cir"][b:e], d["cor"][b:e]) for b, e in zip(o[:-1], o[1:])])
    uv = _direct64(d["xy"], d["xy"], d["cir"], d["cor"])
    if call == "stage":
        return {"uv": uv, "stage": d["xy"] + 0.5e-3 * uv}
    if call == "host":
        r = {"uv": uv}
        if "points" in d:
            r["points"] = _direct64(d["points"], d["xy"], d["cir"], d["cor"])
        return r
    return uv
