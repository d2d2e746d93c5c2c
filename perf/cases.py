"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values; ``listed()`` names the ones that are always
measured, ``draw(rng)`` makes others over the same ranges, ``prepare`` builds
what a program holds before the call (sampler, scene, buffers, points, keys),
``run`` is one pass through the public entry points, ``work`` counts what the
path cannot do without and ``exact`` gives the outputs in 64 bits where they
have such a value.

The ``path`` of a case:

* ``frame``   one frame by the device-side loop (``render_graph``);
* ``app``     one frame by the calls a sample application makes itself:
              InitialSampling, the integrand, SamplingPass until the budget is
              reached, Integrate, ConvertToBytes;
* ``batch``   many images of uneven size, budget and dimension in one render;
* ``locate``  hierarchy over a frame's leaves, then the leaves of query points;
* ``sort``    (key, value) pairs by radix sort;
* ``train``   one training step of the leaf-priority network;
* ``targets`` features and true errors of a frame's leaves (training data);
* ``truth``   the reference image that a frame's quality is measured against.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import pmdas_gb300 as P
from pmdas_gb300 import kdgrid as K
from pmdas_gb300._native import MLP_PARAMS
from pmdas_gb300.workloads import batch_image

MB, DOF, MBDOF, LIGHT = P.SCENE_DISCS_MB, P.SCENE_DISCS_DOF, P.SCENE_DISCS_MBDOF, P.SCENE_DIRECT_LIGHT
SCENES = {"mb": (MB, 3), "dof": (DOF, 4), "mbdof": (MBDOF, 5), "light": (LIGHT, 4)}


def _frame(path, scene, width, height, spp, prims, **kw):
    c = dict(path=path, scene=scene, dim=SCENES[scene][1], width=width, height=height, spp=spp, prims=prims,
             bitsPerDim=1, extraImgBits=8, alpha=0.25, candidates=4, ieee=False, learned=False)
    c.update(kw)
    return c


def listed():
    named = {
        # an interactive preview: 3-D motion blur, 256x256 at 8 spp, passes of a few
        # thousand leaves, where launches and latency count
        "preview_mb256": _frame("frame", "mb", 256, 256, 8, 64, extraImgBits=6),
        # the benchmark's headline frame: 4-D depth of field, 1024x1024 at 16 spp
        "frame_dof1024": _frame("frame", "dof", 1024, 1024, 16, 256),
        # 5-D motion blur and depth of field, 1920x1080 at 32 spp
        "frame_mbdof1080": _frame("frame", "mbdof", 1920, 1080, 32, 256),
        # the same scene kind with the learned leaf priority at half the budget
        "learned_mbdof1080": _frame("frame", "mbdof", 1920, 1080, 16, 256, learned=True),
        # a sample application's own loop over the drop-in calls: 4-D direct lighting in 4K
        "app_light4k": _frame("app", "light", 3840, 2160, 16, 4),
        # the same loop in the reproducible (strict IEEE) arithmetic, an odd resolution and a
        # dimension that the integrand does not read
        "app_ieee_odd": _frame("app", "mbdof", 853, 479, 12, 128, dim=6, extraImgBits=5, candidates=5, ieee=True),
        # a batch of twelve images of the batched workload
        "batch_12": dict(path="batch", first=200, count=12),
        # point queries on the final leaves of the headline frame
        "locate_dof1024": _frame("locate", "dof", 1024, 1024, 16, 256, points=1_000_003),
        # as many 64-bit keys as the headline frame has leaves
        "sort_6m": dict(path="sort", count=5_944_990, beginBit=0, endBit=64, values=False),
        # a training step at the trainer's batch size
        "train_65536": dict(path="train", rows=65_536),
        # the trainer's data collection at one pass of a frame: all leaves' features, of which
        # 16,384 are taken with their true errors
        "targets_mbdof1080": _frame("targets", "mbdof", 1920, 1080, 4, 256, extraImgBits=7, leaves=16_384,
                                    samples=64),
        # a reference image: 1024 spp, a preview's size
        "truth_dof256": _frame("truth", "dof", 256, 256, 1024, 256),
    }
    return [dict(c, name=n) for n, c in named.items()]


MOST_SAMPLES = 133_000_000  # of the largest listed frame (app_light4k)
MOST_BATCH = 200_000_000    # of the listed batch


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _draw_frame(rng, path, most=MOST_SAMPLES):
    scene = rng.choice(sorted(SCENES))
    dim = SCENES[scene][1]
    if rng.random() < 0.15:
        dim = min(6, dim + 1)  # one dimension more than the integrand reads
    width = int(_log(rng, 160, 3840))
    height = max(90, int(width * rng.choice((1.0, 0.75, 0.5625, 0.4167))))
    cells = width * height
    bpd = 1 if rng.random() < 0.8 else 0
    # an initial grid of at most one sample per pixel, so that passes follow
    eib = max(0, int(math.floor(math.log(max(1.0, cells / (4 << (bpd * dim))), 4))))
    eib = min(eib, (28 - bpd * dim) // 2)
    spp = round(_log(rng, 2, 48), 2)
    spp = min(spp, most / cells)
    ieee = rng.random() < 0.15
    if ieee:
        spp = min(spp, 40_000_000 / cells)
    return _frame(path, scene, width, height, spp, 4 if scene == "light" else int(_log(rng, 16, 512)), dim=dim,
                  bitsPerDim=bpd, extraImgBits=eib, alpha=rng.choice((0.015625, 0.0625, 0.25, 0.25)),
                  candidates=rng.choice((2, 4, 4, 5, 8)), ieee=ieee)


def draw(rng):
    path = rng.choice(("frame", "frame", "frame", "app", "app", "batch", "locate", "sort", "train", "targets", "truth"))
    if path == "frame":
        c = _draw_frame(rng, path)
        c["learned"] = rng.random() < 0.3
        return c
    if path == "app":
        return _draw_frame(rng, path)
    if path == "batch":
        first, count = rng.randrange(1000), int(_log(rng, 2, 17))
        while count > 2 and sum(batch_image(first + k).budget for k in range(count)) > MOST_BATCH:
            count -= 1
        return dict(path="batch", first=first, count=count)
    if path == "locate":
        return dict(_draw_frame(rng, path, 20_000_000), ieee=False, points=int(_log(rng, 100, 2_000_000)))
    if path == "sort":
        count = int(_log(rng, 1000, 12_000_000))
        end = rng.randint(20, 64)
        return dict(path="sort", count=count, beginBit=rng.choice((0, 0, 3)), endBit=end, values=rng.random() < 0.5)
    if path == "train":
        return dict(path="train", rows=int(_log(rng, 200, 200_000)))
    if path == "targets":
        return dict(_draw_frame(rng, path, 20_000_000), ieee=False, leaves=int(_log(rng, 500, 50_000)),
                    samples=rng.choice((16, 64, 64, 100)))
    c = _draw_frame(rng, path, 1e9)
    c["width"], c["height"] = int(_log(rng, 60, 512)), int(_log(rng, 60, 512))
    strata = int(_log(rng, 8, 65))
    strata = max(4, min(strata, int(math.sqrt(67_000_000 / (c["width"] * c["height"])))))
    return dict(c, dim=SCENES[c["scene"]][1], ieee=False, spp=strata * strata, prims=min(c["prims"], 256))


# ---- what a program holds before the call

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(P.__file__)), "weights", "priority_mbdof1080.f32")


def _budget(c):
    return int(c["spp"] * c["width"] * c["height"])


def _initial_samples(c):
    return 4 * ((1 << (c["bitsPerDim"] * c["dim"])) << (2 * c["extraImgBits"]))


def _sampler(c, seed):
    need = max(_budget(c), _initial_samples(c))
    grid = P.KDGrid(c["dim"], (3 * need + 1) // 2, c["candidates"], c["bitsPerDim"], c["extraImgBits"], c["alpha"],
                    c["width"], c["height"], arith=P.ARITH_IEEE if c["ieee"] else P.ARITH_REFERENCE)
    if c["learned"]:
        grid.LearnedEnable(params=np.fromfile(WEIGHTS, "<f4"))
    return dict(grid=grid, scene=_scene(c, seed))


def _scene(c, seed):
    return P.Scene(SCENES[c["scene"]][0], seed, c["prims"], c["width"], c["height"], c["width"], c["height"])


def _pixels(w, h):
    return torch.zeros(h, w, 4, device="cuda")


class _Buffer:
    """A sampler's own device buffer as an array; holds the sampler, so a view outlives other references to it."""

    def __init__(self, grid, address, columns):
        self.grid = grid
        self.__cuda_array_interface__ = dict(data=(address, False), shape=(grid.GetMaxSamples(), columns),
                                             typestr="<f4", version=3, strides=None)


def _buffers(grid):
    """The sample buffers, whole, as the program that evaluates them holds them; zero where no sample lies."""
    return (torch.as_tensor(_Buffer(grid, grid.GetSampleCoordinatesPtr(), grid.dim), device="cuda").zero_(),
            torch.as_tensor(_Buffer(grid, grid.GetSampleValuesPtr(), 3), device="cuda").zero_())


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _train_inputs(c, seed):
    """Features and targets as the trainer's: features within about a unit, targets within 8 bits / 32."""
    gen = _generator(seed)
    p = torch.cat([(torch.rand(n, device="cuda", generator=gen) * 2 - 1) / math.sqrt(fan)
                   for n, fan in ((64 * 16, 16), (64, 16), (64 * 64, 64), (64, 64), (64, 64), (1, 64))])
    x = torch.randn(c["rows"], 16, device="cuda", generator=gen) * 0.5
    y = (torch.randn(c["rows"], device="cuda", generator=gen) * 0.1).clamp(-0.25, 0.25)
    return p, x, y


def prepare(case, seed):
    c = case
    s = dict(case=c)
    if c["path"] == "sort":
        gen = _generator(seed)
        s["keys"] = torch.randint(-(1 << 63), (1 << 63) - 1, (c["count"],), dtype=torch.int64, device="cuda",
                                  generator=gen)
        s["values"] = (torch.randint(0, 1 << 31, (c["count"],), dtype=torch.int32, device="cuda", generator=gen)
                       if c["values"] else None)
    elif c["path"] == "train":
        s["params"], s["features"], s["targets"] = _train_inputs(c, seed)
        s["m1"], s["m2"], s["step"] = torch.zeros_like(s["params"]), torch.zeros_like(s["params"]), 0
    elif c["path"] == "truth":
        s["scene"] = _scene(c, seed)
    elif c["path"] == "batch":
        images = [batch_image(c["first"] + k) for k in range(c["count"])]
        s["grids"] = [P.KDGrid(w.dim, w.maxSamples, w.candidatesNum, w.bitsPerDim, w.extraImgBits, w.alpha, w.scaleX,
                               w.scaleY) for w in images]
        s["scenes"] = [P.Scene(w.scene_kind, seed + k, w.scene_count, w.scaleX, w.scaleY, w.width, w.height)
                       for k, w in enumerate(images)]
        s["pixels"] = [_pixels(w.width, w.height) for w in images]
        s["batch"] = P.Batch(s["grids"], s["scenes"], [w.budget for w in images], s["pixels"],
                             [w.width for w in images], [w.height for w in images])
        s["buffers"] = [_buffers(g) for g in s["grids"]]
    else:
        s.update(_sampler(c, seed))
        w, h = c["width"], c["height"]
        s["pixels"] = _pixels(w, h)
        s["coords"], s["values"] = _buffers(s["grid"])
        if c["path"] == "app":
            s["bytes"] = torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")
        if c["path"] in ("locate", "targets"):
            P.render_graph(s["grid"], s["scene"], _budget(c), s["pixels"], w, h)
        if c["path"] == "locate":
            scale = torch.tensor([w, h] + [1] * (c["dim"] - 2), dtype=torch.float32, device="cuda")
            s["points"] = torch.rand(c["points"], c["dim"], device="cuda", generator=_generator(seed)) * scale
        if c["path"] == "targets":
            s["grid"].ComputeErrors()  # the features read current leaf errors
            s["leaves"] = torch.randint(0, s["grid"].GetNumberOfNodes(), (c["leaves"],), dtype=torch.int32,
                                        device="cuda", generator=_generator(seed))
            s["seed"] = seed
    return s


# ---- one pass

def run(state):
    return {"frame": _run_frame, "app": _run_app, "batch": _run_batch, "locate": _run_locate, "sort": _run_sort,
            "train": _run_train, "targets": _run_targets, "truth": _run_truth}[state["case"]["path"]](state)


def _run_frame(s):
    c = s["case"]
    st = P.render_graph(s["grid"], s["scene"], _budget(c), s["pixels"], c["width"], c["height"])
    return dict(image=s["pixels"], coords=s["coords"], values=s["values"], samples=st.numberOfSamples,
                leaves=st.numberOfNodes, passes=st.passes)


def _run_app(s):
    c, grid, scene = s["case"], s["grid"], s["scene"]
    budget, most = _budget(c), grid.GetMaxSamples()
    grid.InitialSampling()
    n = grid.GetNumberOfSamples()
    scene.evaluate(grid, 0, n)
    while n < budget and n + grid.GetNumberOfNodes() <= most:
        grid.SamplingPass()
        n, new = grid.GetNumberOfSamples(), grid.GetNewSamples()
        scene.evaluate(grid, n - new, new)
    grid.Integrate(s["pixels"], c["width"], c["height"])
    grid.ConvertToBytes(s["pixels"], s["bytes"], c["width"], c["height"])
    # (the bytes round an image whose float sums may differ by the order of their
    # additions, so the image itself stands for both)
    return dict(image=s["pixels"], coords=s["coords"], values=s["values"], samples=n,
                leaves=grid.GetNumberOfNodes())


def _run_batch(s):
    stats = s["batch"].render()
    return [dict(image=px, coords=b[0], values=b[1], samples=st.numberOfSamples,
                 leaves=st.numberOfNodes) for px, b, st in zip(s["pixels"], s["buffers"], stats)]


def _run_locate(s):
    s["grid"].BuildHierarchy()
    return s["grid"].Locate(s["points"])


def _run_sort(s):
    c = s["case"]
    return P.radix_sort_pairs(s["keys"], s["values"], c["beginBit"], c["endBit"])


def _run_train(s):
    s["step"] += 1
    g, loss = K.mlp_gradients(s["params"], s["features"], s["targets"])
    K.mlp_adam(s["params"], s["m1"], s["m2"], g, s["step"], 1e-3)
    return dict(loss=loss, m1=s["m1"], m2=s["m2"], params=s["params"])


def _run_targets(s):
    c = s["case"]
    features = s["grid"].LeafFeatures()[s["leaves"].long()]
    return features, s["grid"].LeafTrueErrors(s["scene"], samples=c["samples"], seed=s["seed"], leaves=s["leaves"])


def _run_truth(s):
    c = s["case"]
    return s["scene"].reference_image(c["width"], c["height"], spp=c["spp"], seed=12345)


# ---- what a pass cannot do without

def _frame_bytes(samples, dim, pixels):
    """Every sample's coordinates and value, the leaves (about 0.35 per sample: node, box, error, seed), the image."""
    return samples * (4 * dim + 12) + 0.35 * samples * (24 + 8 * dim) + 16 * pixels


def work(case):
    c = case
    if c["path"] == "sort":
        return dict(bytes=(8 + 8 + 4 + (4 if c["values"] else 0)) * c["count"], flops=0)
    if c["path"] == "train":
        # forward 2 * (16 * 64 + 64 * 64 + 64) per row, backward twice that
        return dict(bytes=c["rows"] * 68 + 7 * 4 * MLP_PARAMS, flops=c["rows"] * 6 * 5184)
    if c["path"] == "truth":
        # one distance test per sample at least
        return dict(bytes=24 * c["width"] * c["height"], flops=20.0 * c["spp"] * c["width"] * c["height"])
    if c["path"] == "batch":
        images = [batch_image(c["first"] + k) for k in range(c["count"])]
        return dict(bytes=sum(_frame_bytes(w.budget, w.dim, w.width * w.height) for w in images), flops=0)
    samples = max(_budget(c), _initial_samples(c))
    if c["path"] == "locate":
        # node, box of every leaf; key, order, children, parents, box of the tree; the points and answers
        return dict(bytes=0.35 * samples * (44 + 16 * c["dim"]) + c["points"] * (4 * c["dim"] + 4), flops=0)
    if c["path"] == "targets":
        # every leaf's record, values, error and features; a distance test per target sample at least
        return dict(bytes=0.35 * samples * (16 + 8 * c["dim"] + 36 + 4 + 64) + c["leaves"] * 8,
                    flops=20.0 * c["leaves"] * c["samples"])
    extra = 4 * c["width"] * c["height"] if c["path"] == "app" else 0
    return dict(bytes=_frame_bytes(samples, c["dim"], c["width"] * c["height"]) + extra, flops=0)


# ---- the outputs in 64 bits

def exact(case, seed):
    # A frame has no such value: which leaves a pass refines follows from the
    # 32-bit errors of the passes before, so other roundings give another,
    # equally good set of samples.  The same goes for what is read off a frame
    # (its leaves' features and errors).  Sorted pairs and leaf indices are whole.
    if case["path"] == "train":
        return _exact_train(case, seed)
    if case["path"] == "truth" and case["scene"] != "light":
        return _exact_truth(case, seed)
    return None


def _exact_train(c, seed):
    p32, x, y = _train_inputs(c, seed)
    p = p32.double().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, (64 * 16, 64, 64 * 64, 64, 64, 1))
    h = torch.relu(x.double() @ w1.view(64, 16).T + b1)
    h = torch.relu(h @ w2.view(64, 64).T + b2)
    loss = ((h @ w3 + b3 - y.double()) ** 2).mean()
    (g,) = torch.autograd.grad(loss, p)
    m1, m2 = 0.1 * g, 0.001 * g * g
    step = 1e-3 * (m1 / 0.1) / (torch.sqrt(m2 / 0.001) + 1e-8)
    return dict(loss=float(loss), m1=m1, m2=m2, params=(p - step).detach())


def _splitmix(seed):
    """Uniforms of the seeded scenes: 24 bits of splitmix64."""
    mask, s = (1 << 64) - 1, seed & ((1 << 64) - 1)
    while True:
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        yield ((z ^ (z >> 31)) >> 40) / 16777216.0


def _exact_discs(c, seed):
    """The disc scene as 32-bit numbers in the order they are drawn: x, y, depth, radius, velocity, colour."""
    f, u = np.float32, _splitmix(seed)
    between = lambda a, b: f(a) + (f(b) - f(a)) * f(next(u))  # noqa: E731
    half = f(math.sqrt(2.0) - 1.0)
    half_w = half * (f(c["width"]) / f(c["height"]))
    discs = []
    for _ in range(c["prims"]):
        if c["scene"] == "mb":
            x, y = f(next(u)), f(next(u))
            r = between(0.02, 0.08)
            rgb = [f(next(u)) for _ in range(3)]
            discs.append([x, y, f(0), r, between(-0.1, 0.1), between(-0.1, 0.1)] + rgb)
        else:
            z, r = between(1, 10), between(0.05, 0.3)
            rgb = [f(next(u)) for _ in range(3)]
            x = (f(2) * f(next(u)) - f(1)) * (z * half_w)
            y = (f(2) * f(next(u)) - f(1)) * (z * half)
            discs.append([x, y, z, r, f(0), f(0)] + rgb)
    if c["scene"] == "mb":
        discs.reverse()  # the last listed disc is in front
    else:
        discs.sort(key=lambda d: d[2])  # the nearest is in front
        if c["scene"] == "mbdof":
            for d in discs:
                d[4], d[5] = between(-0.1, 0.1), between(-0.1, 0.1)
    return torch.tensor(np.array(discs), dtype=torch.float64, device="cuda"), float(half_w), float(half)


def _exact_truth(c, seed):
    discs, half_w, half_h = _exact_discs(c, seed)
    w, h, strata, dims = c["width"], c["height"], math.isqrt(c["spp"]), SCENES[c["scene"]][1]
    wrap = lambda v: (v + (1 << 63)) % (1 << 64) - (1 << 63)  # noqa: E731
    pixel = torch.arange(w * h, dtype=torch.int64, device="cuda")
    lcg = (pixel + 1) * wrap(0x9E3779B97F4A7C15) ^ 12345

    def uniform():
        nonlocal lcg
        lcg = lcg * wrap(6364136223846793005) + wrap(1442695040888963407)
        return ((lcg >> 40) & 0xFFFFFF).double() / 16777216.0

    px, py = (pixel % w).double(), (pixel // w).double()
    colours = torch.cat([discs[:, 6:9], torch.full((1, 3), float(np.float32(0.1)), dtype=torch.float64, device="cuda")])
    total = torch.zeros(w * h, 3, dtype=torch.float64, device="cuda")
    columns = [v[:, None] for v in discs.T]
    for i in range(strata):
        for j in range(strata):
            x = (px + (i + uniform()) / strata) / w
            y = (py + (j + uniform()) / strata) / h
            rest = [uniform() for _ in range(dims - 2)]
            t = rest[0] if c["scene"] != "dof" else torch.zeros_like(x)
            cx, cy = columns[0] + columns[4] * t, columns[1] + columns[5] * t
            if c["scene"] == "mb":
                dx, dy = x - cx, y - cy
            else:
                ax, ay = 2 * rest[-2] - 1, 2 * rest[-1] - 1
                wide = ax.abs() > ay.abs()
                r = torch.where(wide, ax, ay)
                phi = math.pi / 4 * torch.where(wide, ay, ax) / torch.where(r == 0, torch.ones_like(r), r)
                co, si = torch.cos(phi), torch.sin(phi)
                lx, ly = 0.1 * r * torch.where(wide, co, si), 0.1 * r * torch.where(wide, si, co)
                s = columns[2] / 4
                dx = lx + s * (4 * (2 * x - 1) * half_w - lx) - cx
                dy = ly + s * (4 * (2 * y - 1) * half_h - ly) - cy
            inside = dx * dx + dy * dy <= columns[3] ** 2
            first = torch.where(inside.any(0), inside.to(torch.uint8).argmax(0), len(discs))
            total += colours[first]
    return (total / (strata * strata)).view(h, w, 3)
