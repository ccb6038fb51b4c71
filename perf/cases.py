"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case goes through a public entry point on the arrays that such a program holds: the bundle
adjustment of a packed scene (``solve_packed``), chained adjustments of a scene kept on the device
(``ResidentScene``), a batch of local windows (``batch_adjust``), the adjoint of a solve
(``bundle_vjp``), the evaluation of a scene's observations (``tba_evaluate_observations``) and the
inverse-depth linearisation (``linearize_rows``).  These entry points take host arrays by their
nature, so a case's inputs are page-locked host arrays and its pass is the whole call, the copies
included.  Scenes are drawn on the GPU from the seed; their geometry is that of the benchmark's
configurations (a ring, a helix, a sphere, arcs), with pixel noise, outliers and a perturbed start.
"""
import ctypes
import math

import numpy as np
import torch

import typecv_b200 as tb
from typecv_b200 import _lib
from typecv_b200 import adjoint, batch, inverse_depth
from typecv_b200.resident import ResidentScene

F64 = torch.float64


def listed():
    return [
        # One local window as the mapper adjusts it after each new view: the smallest call.
        {"name": "window", "op": "solve", "kind": "arc", "C": 7, "P": 611, "fixed": 0, "shared": False,
         "precision": "fp64", "iterations": 6},
        # A small turntable scene with its focal length refined (the benchmark's configuration 0).
        {"name": "ring", "op": "solve", "kind": "ring", "C": 10, "P": 2000, "fixed": 1, "shared": True,
         "precision": "fp64", "iterations": 20},
        # A sequence of a few dozen views.
        {"name": "sequence", "op": "solve", "kind": "sphere", "C": 61, "P": 12345, "fixed": 1, "shared": False,
         "precision": "fp64", "iterations": 10},
        # A medium map, 200 views and 100k points (configuration 1), badly conditioned.
        {"name": "helix", "op": "solve", "kind": "helix", "C": 200, "P": 100000, "fixed": 1, "shared": False,
         "precision": "fp64", "iterations": 6},
        # A map kept on the device, adjusted twice as it grows, with bearings and several fixed views.
        {"name": "resident", "op": "resident", "kind": "sphere", "C": 317, "P": 41003, "fixed": 3, "bearings": 64,
         "shared": False, "precision": "fp64", "iterations": 6},
        # The global adjustment of a large map (configuration 2): with the focal length, and in the mixed form.
        {"name": "global fp64", "op": "solve", "kind": "sphere", "C": 1500, "P": 1000000, "fixed": 1, "shared": True,
         "precision": "fp64", "iterations": 10},
        {"name": "global mixed", "op": "solve", "kind": "sphere", "C": 1500, "P": 1000000, "fixed": 1, "shared": False,
         "precision": "mixed", "iterations": 10},
        # A few local windows at once, with the focal length; and a whole map's windows (configuration 3).
        {"name": "windows 24", "op": "batch", "count": 24, "shared": True, "precision": "fp64", "iterations": 4},
        {"name": "windows 512", "op": "batch", "count": 512, "shared": False, "precision": "fp64", "iterations": 6},
        # The gradient of a solution by its pixels, at configuration 4's size.
        {"name": "adjoint", "op": "vjp", "kind": "sphere", "C": 200, "P": 50000, "newton": 0},
        # The evaluation and depth filter of all observations after a global adjustment.
        {"name": "observations", "op": "observations", "kind": "sphere", "C": 1500, "P": 1000000, "bound": 0.05},
        # The linearisation of an inverse-depth adjustment's measurements.
        {"name": "inverse depth", "op": "rows", "rows": 262147},
    ]


def draw(rng):
    """One more case of the listed ranges: sizes over their logarithm, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["solve", "solve", "solve", "resident", "batch", "vjp", "observations", "rows"])
    if op == "batch":
        shared = rng.random() < 0.5
        return {"op": op, "count": size(3, 300), "shared": shared, "precision": "fp64",
                "iterations": 4 if shared else rng.randint(4, 6)}
    if op == "vjp":
        C = size(8, 200)
        return {"op": op, "kind": "sphere", "C": C, "P": C * rng.randint(50, 250) + rng.randint(0, 31),
                "newton": rng.choice([0, 0, 2])}
    if op == "rows":
        return {"op": op, "rows": size(100, 1000000)}
    if op == "observations":
        C = size(10, 1500)
        return {"op": op, "kind": "sphere", "C": C, "P": C * rng.randint(40, 600) + rng.randint(0, 31),
                "bound": rng.choice([0.0, 0.05])}
    C = size(5, 1500)
    kind = "arc" if C <= 12 else ("ring" if C <= 24 else rng.choice(["sphere", "sphere", "helix"]))
    fixed = rng.choice([1, 1, 3])
    case = {"op": op, "kind": kind, "C": C, "P": C * rng.randint(60, 500) + rng.randint(0, 31), "fixed": fixed,
            "shared": rng.random() < 0.5, "precision": "fp64", "iterations": rng.randint(4, 10)}
    if C > 800 and rng.random() < 0.5:  # the mixed form is for large maps
        case.update(shared=False, precision="mixed")
    if kind == "helix":
        case.update(shared=False, iterations=min(case["iterations"], 6))
    if kind == "arc":
        case.update(fixed=0, iterations=min(case["iterations"], 6))
    if kind == "sphere" and rng.random() < 0.3:
        case["bearings"] = rng.randint(3, 64)
    return case


# ---- scenes ------------------------------------------------------------------------------------------

WIDTH, HEIGHT = 1024.0, 768.0
C_SEED = 20260


class Draws:
    """The random numbers of one scene, on the GPU, from its seed alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(int(seed) % (1 << 62))

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda", dtype=F64)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return lo + (hi - lo) * torch.rand(*shape, generator=self.g, device="cuda", dtype=F64)

    def below(self, n, *shape):
        return torch.randint(0, n, shape, generator=self.g, device="cuda")


def look_at(centers, targets):
    """World-to-camera poses (C x 12) of cameras at `centers` looking at `targets`, image y down."""
    z = torch.nn.functional.normalize(targets - centers, dim=1)
    up = torch.zeros_like(z)
    polar = z[:, 2].abs() > 0.99
    up[:, 2] = (~polar).double()
    up[:, 1] = polar.double()
    x = torch.nn.functional.normalize(torch.linalg.cross(z, up), dim=1)
    R = torch.stack([x, torch.linalg.cross(z, x), z], dim=1)
    t = -(R @ centers[:, :, None])[:, :, 0]
    return torch.cat([R.reshape(-1, 9), t], dim=1)


def camera_frame(poses, c, X, bearing=False):
    q = (poses[c, :9].reshape(-1, 3, 3) @ X[:, :, None])[:, :, 0]
    return q if bearing else q + poses[c, 9:]


def pixels_of(cams, q):
    xy = q[:, :2] / q[:, 2:]
    r2 = (xy * xy).sum(1)
    d = 1 + cams[:, 4] * r2 + cams[:, 5] * r2 * r2
    return cams[:, :2] * xy * d[:, None] + cams[:, 2:4], r2


def visible(poses, cams, c, X, bearing=False):
    q = camera_frame(poses, c, X, bearing)
    front = q[:, 2] > 0.1
    px, r2 = pixels_of(cams[c], torch.where(front[:, None], q, torch.ones_like(q)))
    return front & (px[:, 0] > 2) & (px[:, 0] < WIDTH - 2) & (px[:, 1] > 2) & (px[:, 1] < HEIGHT - 2) & (r2 < 3.3)


def tracks(rnd, poses, cams, X, lo, hi, mean=None, bearing=False, candidates=48):
    """Each point's cameras: one that sees it and the nearest to that one that see it too, up to the
    track's length (geometric with `mean`, or uniform in lo..hi).  (cameras, points), point-major."""
    C, P = len(poses), len(X)
    centers = -(poses[:, :9].reshape(-1, 3, 3).transpose(1, 2) @ poses[:, 9:, None])[:, :, 0]
    near = torch.cdist(centers, centers).argsort(dim=1, stable=True)[:, :min(candidates, C)]
    if mean:
        want = torch.ceil(torch.log(rnd.uniform(P, lo=1e-12)) / math.log(1 - 1 / mean)).clamp(lo, hi)
    else:
        want = lo + rnd.below(hi + 1 - lo, P)
    home = rnd.below(C, P)
    if bearing:  # a bearing is seen by the cameras that face it
        home = (poses[:, 6:9] @ X.T).argmax(dim=0)
    else:
        for _ in range(12):
            bad = ~visible(poses, cams, home, X)
            home = torch.where(bad, rnd.below(C, P), home)
    cs, ps = [], []
    for s in range(0, P, 100000):
        e = min(P, s + 100000)
        cand = near[home[s:e]]
        K = cand.shape[1]
        vis = visible(poses, cams, cand.reshape(-1), X[s:e].repeat_interleave(K, dim=0), bearing).reshape(-1, K)
        take = vis & (vis.cumsum(dim=1) <= want[s:e, None])
        take &= take.sum(dim=1, keepdim=True) >= max(2, lo if lo <= 2 else 2)
        rows, cols = take.nonzero(as_tuple=True)
        cs.append(cand[rows, cols])
        ps.append(rows + s)
    c, p = torch.cat(cs), torch.cat(ps)
    order = (p * C + c).argsort()
    return c[order], p[order]


def scene(case, seed):
    """A scene of the case: its true and its perturbed state, and its observations (CUDA tensors).  Where
    the outputs follow the observations, the tracks are the case's and the pixels the seed's."""
    rnd = Draws(C_SEED + case["C"] + case["P"] if case["op"] in ("vjp", "observations") else seed)
    kind, C, P = case["kind"], case["C"], case["P"]
    D = case.get("bearings", 0)
    k = torch.arange(C, device="cuda", dtype=F64)
    zero = torch.zeros(C, device="cuda", dtype=F64)
    f = torch.full((C,), 800.0, device="cuda", dtype=F64)
    if kind == "ring":
        a = 2 * math.pi * k / C
        centers = torch.stack([5 * a.cos(), 5 * a.sin(), zero], dim=1)
        targets = torch.zeros_like(centers)
        X = rnd.uniform(P, 3, lo=-1.0)
        track = (2, C, None)
    elif kind == "arc":
        a = math.pi / 24 * (k - (C - 1) / 2)
        centers = torch.stack([5 * a.cos(), 5 * a.sin(), zero], dim=1)
        targets = torch.zeros_like(centers)
        X = rnd.uniform(P, 3, lo=-1.0)
        track = (3, 10, None)
    elif kind == "helix":
        a = 2 * math.pi * 3 * k / C
        h = a / (2 * math.pi) - 1.5
        centers = torch.stack([8 * a.cos(), 8 * a.sin(), h], dim=1)
        targets = torch.stack([zero, zero, h], dim=1)
        X = rnd.uniform(P, 3, lo=-2.0, hi=2.0)
        f = rnd.uniform(C, lo=700.0, hi=900.0)
        track = (3, 12, None)
    else:
        phi = torch.arccos(1 - 2 * (k + 0.5) / C)
        th = math.pi * (1 + 5 ** 0.5) * (k + 0.5)
        dirs = torch.stack([th.cos() * phi.sin(), th.sin() * phi.sin(), phi.cos()], dim=1)
        centers = 20 * torch.nn.functional.normalize(dirs + 0.02 * rnd.normal(C, 3), dim=1)
        targets = torch.zeros_like(centers)
        mu = torch.nn.functional.normalize(rnd.normal(64, 3), dim=1) * 8.5 * rnd.uniform(64, 1) ** (1 / 3)
        X = mu[rnd.below(64, P)] + 0.5 * rnd.normal(P, 3)
        X = X * (10 / X.norm(dim=1, keepdim=True)).clamp(max=1.0)
        f = rnd.uniform(C, lo=700.0, hi=900.0)
        track = (2, 40, 6.0)
    poses = look_at(centers, targets)
    cams = torch.stack([f, f, zero + WIDTH / 2, zero + HEIGHT / 2, zero - 0.05, zero], dim=1)
    if kind == "ring":
        c, p = torch.arange(C, device="cuda").repeat(P), torch.arange(P, device="cuda").repeat_interleave(C)
        keep = visible(poses, cams, c, X[p])
        c, p = c[keep], p[keep]
    else:
        c, p = tracks(rnd, poses, cams, X, *track)
    if D:
        B = torch.nn.functional.normalize(-centers[rnd.below(C, D)] / 20 + 0.05 * rnd.normal(D, 3), dim=1)
        bc, bp = tracks(rnd, poses, cams, B, 2, 8, bearing=True)
        X, c, p = torch.cat([X, B]), torch.cat([c, bc]), torch.cat([p, bp + P])
    # Points with fewer than two observations leave the scene.
    keep = torch.bincount(p, minlength=len(X)) >= 2
    number = keep.cumsum(0) - 1
    on = keep[p]
    c, p, bearing = c[on], number[p[on]], (p[on] >= P)
    D = int(keep[P:].sum())
    X = X[keep]
    rnd = Draws(65537 * int(seed) + 11)
    q = camera_frame(poses, c, X[p])
    q = torch.where(bearing[:, None], camera_frame(poses, c, X[p], True), q)
    px = pixels_of(cams[c], q)[0] + 0.5 * rnd.normal(len(c), 2)
    wild = rnd.uniform(len(c)) < case.get("outliers", 0.03)
    px = torch.where(wild[:, None], rnd.uniform(len(c), 2) * torch.tensor([WIDTH, HEIGHT], device="cuda"), px)
    # The start: rotations 0.01 rad off, translations 1% off, points 1 cm off, the focal length 3%.
    w = 0.01 * torch.nn.functional.normalize(rnd.normal(C, 3), dim=1)
    K = torch.zeros(C, 3, 3, device="cuda", dtype=F64)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 0] = -w[:, 2], w[:, 1], w[:, 2]
    K[:, 1, 2], K[:, 2, 0], K[:, 2, 1] = -w[:, 0], -w[:, 1], w[:, 0]
    R0 = torch.matrix_exp(K) @ poses[:, :9].reshape(-1, 3, 3)
    t = poses[:, 9:]
    t0 = t + 0.01 * t.norm(dim=1, keepdim=True) * torch.nn.functional.normalize(rnd.normal(C, 3), dim=1)
    poses0 = torch.cat([R0.reshape(-1, 9), t0], dim=1)
    active = torch.ones(C, device="cuda", dtype=torch.int64)
    fixed = case.get("fixed", 1)  # the first two views, then the last ones; 0: every fourth view
    fixed = list(range(min(fixed, 2))) + [C - 1 - j for j in range(fixed - 2)] or [1] + list(range(0, C, 4))
    poses0[fixed], active[fixed] = poses[fixed], 0
    X0 = X + 0.01 * rnd.normal(len(X), 3)
    if D:
        X0[-D:] = torch.nn.functional.normalize(X[-D:] + 0.002 * rnd.normal(D, 3), dim=1)
    cams0 = cams.clone()
    cams0[:, :2] *= 1.03 if case.get("shared") else 1.0
    return {"poses": poses, "points": X, "cams": cams, "poses0": poses0, "points0": X0, "cams0": cams0,
            "c": c, "p": p, "px": px, "active": active, "C": C, "P": len(X), "M": len(c), "D": D}


def pinned(x, dtype):
    out = torch.empty(x.numel(), dtype=dtype, pin_memory=True)
    out.copy_(x.reshape(-1))
    a = out.numpy()
    return a.view(np.uint32) if dtype == torch.int32 else a


def packed(s, poses, points, cams):
    """The packed scene and index arrays of tba_bundle_adjust, page-locked."""
    values = torch.cat([v.reshape(-1) for v in (poses, points, cams, s["px"])])
    ends = [torch.cat([torch.zeros(1, device="cuda", dtype=torch.int64), torch.bincount(x, minlength=n).cumsum(0)])
            for x, n in ((s["p"], s["P"]), (s["c"], s["C"]))]
    index = torch.cat([s["c"], s["p"], ends[0], ends[1], s["c"].argsort(stable=True), s["active"]])
    return pinned(values, F64), pinned(index.to(torch.int32), torch.int32)


# ---- the cases' states ---------------------------------------------------------------------------------

_device = None


def device():
    """The program's one device handle."""
    global _device
    if _device is None:
        _device = tb.ShadeDevice.open(0)
    return _device


class Resident:
    """A scene on the device, given back with its state."""

    def __init__(self, control, values, index):
        self.scene = ResidentScene(device(), control, values, index)

    def __del__(self):
        self.scene.close()


def control_of(case, s):
    precision = _lib.TBA_PRECISION_MIXED if case["precision"] == "mixed" else _lib.TBA_PRECISION_FP64
    return tb.make_control(s["C"], s["P"], s["M"], anchor=0, scale_view=1, iterations=case["iterations"],
                           shared_focal=case["shared"], precision=precision, directional=s["D"])


def window_sizes(case):
    """The windows of a batch: 5 to 40 views (every fourth of them fixed, as the views around a window are), 500 to 20,000 points over their logarithm."""
    r = np.random.default_rng(case["count"])
    C = r.integers(5, 41, size=case["count"])
    P = np.rint(np.exp(r.uniform(math.log(500), math.log(20000), size=case["count"]))).astype(int)
    return [(int(a), int(b)) for a, b in zip(C, P)]


def windows(case, seed):
    return [scene({"op": "batch", "kind": "arc", "C": C, "P": P, "shared": case["shared"], "fixed": 0}, 1000003 * int(seed) + k)
            for k, (C, P) in enumerate(window_sizes(case))]


def depth_rows(case, seed):
    """Inverse-depth measurements (34 words each): points anchored in a ring camera, seen by a next one."""
    rnd, n = Draws(seed), case["rows"]
    k = torch.arange(512, device="cuda", dtype=F64)
    a = 2 * math.pi * k / 512
    centers = torch.stack([5 * a.cos(), 5 * a.sin(), 0.3 * (3 * a).sin()], dim=1)
    poses = look_at(centers, torch.zeros_like(centers))
    ref = rnd.below(512, n)
    obs = (ref + 1 + rnd.below(8, n)) % 512
    q = camera_frame(poses, ref, rnd.uniform(n, 3, lo=-1.0))
    K = torch.tensor([800.0, 800.0, 512.0, 384.0, -0.05, 0.0, 1 / 0.15], device="cuda", dtype=F64)
    return torch.cat([q[:, :2] / q[:, 2:], 1 / q[:, 2:], poses[ref], poses[obs], K.expand(n, 7)], dim=1)


def cotangent(s, seed):
    g = Draws(7919 * int(seed) + 1).normal(12 * s["C"] + 3 * s["P"])
    return g / g.norm()


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        problems = []
        for s in windows(case, seed):
            problems.append(batch.PackedProblem(s["C"], s["P"], s["M"], *packed(s, s["poses0"], s["points0"], s["cams0"])))
        n = [sum(getattr(q, k).size for q in problems) for k in ("scene", "index")]
        values = torch.empty(n[0], dtype=F64, pin_memory=True).numpy()
        index = torch.empty(n[1], dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        whole = batch.pack_batch(problems, case["shared"], scene=values, index=index)
        out = torch.empty(whole.output_len, dtype=F64, pin_memory=True).numpy()
        return {"case": case, "batch": whole, "out": out}
    if op == "rows":
        return {"case": case, "rows": pinned(depth_rows(case, seed), F64).reshape(-1, 34)}
    s = scene(case if op != "vjp" else dict(case, outliers=0.0), seed)
    state = {"case": case, "C": s["C"], "P": s["P"], "M": s["M"], "D": s["D"]}
    if op == "observations":
        state["cameras"] = pinned(torch.cat([s["poses"], s["cams"]], dim=1), F64)
        state["points"], state["pixels"] = pinned(s["points"], F64), pinned(s["px"], F64)
        state["indices"] = pinned(torch.stack([s["c"], s["p"]], dim=1).to(torch.int32), torch.int32)
        ends = torch.bincount(s["p"], minlength=s["P"]).cumsum(0)
        state["offsets"] = pinned(torch.cat([ends.new_zeros(1), ends]).to(torch.int32), torch.int32)
        n = s["M"] + (s["P"] if case["bound"] > 0 else 0)
        state["flags"] = torch.zeros(n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
        state["summary"] = np.zeros(2)
        return state
    if op == "vjp":  # at the true state of a scene without outliers: next to its solution
        state["scene"], state["index"] = packed(s, s["poses"], s["points"], s["cams"])
        state["cotangent"] = pinned(cotangent(s, seed), F64)
        return state
    values, index = packed(s, s["poses0"], s["points0"], s["cams0"])
    state["control"] = control_of(case, s)
    if op == "resident":
        state["scene"] = Resident(state["control"], values, index)
        state["poses"], state["points"] = pinned(s["poses0"], F64), pinned(s["points0"], F64)
        return state
    state["scene"], state["index"] = values, index
    n = 12 * s["C"] + 3 * s["P"] + 27
    state["out"] = torch.empty(n, dtype=F64, pin_memory=True).numpy()
    return state


def record(out, C, P, shared):
    """The parts of a result record that describe the solution: the poses, the points, the final and
    initial cost and squared error, and the refined log focal scale."""
    n = 12 * C + 3 * P
    parts = {"poses": out[:12 * C], "points": out[12 * C:n], "cost": out[n + 6:n + 10]}
    if shared:
        parts["focal"] = out[n + 26:n + 27]
    return parts


def run(state):
    case = state["case"]
    op = case["op"]
    dev = device()
    if op == "solve":
        out, _ = tb.solve_packed(dev, state["control"], state["scene"], state["index"], state["out"])
        return record(out, state["C"], state["P"], case["shared"])
    if op == "resident":
        r = state["scene"].scene
        r.write(state["poses"], state["points"])
        _, first, _ = r.adjust()
        _, last, _ = r.adjust()
        poses, points = r.read()
        return {"poses": poses, "points": points, "first": first[6:10], "last": last[6:10]}
    if op == "batch":
        records, _ = batch.batch_adjust(dev, state["batch"], iterations=case["iterations"], shared_focal=case["shared"],
                                        precision=case["precision"], max_cg=256, output=state["out"])
        each = [record(r, C, P, case["shared"]) for r, (C, P) in zip(records, state["batch"].sizes)]
        return {k: np.concatenate([e[k] for e in each]) for k in each[0]}
    if op == "vjp":
        ybar, kbar, solution, _ = adjoint.bundle_vjp(dev, state["C"], state["P"], state["M"], state["scene"],
                                                     state["index"], state["cotangent"], newton_steps=case["newton"],
                                                     want_solution=True)
        return {"pixels": ybar, "intrinsics": kbar, "solution": solution}
    if op == "rows":
        return inverse_depth.linearize_rows(dev, state["rows"])["out"]
    lib = _lib.load()
    ctl = _lib.ObservationControl(state["C"], state["P"], state["M"], 0, 3.0, case["bound"], 1.0)
    d, u = _lib.dptr, _lib.uptr
    status = lib.tba_evaluate_observations(
        dev.handle, ctypes.byref(ctl), d(state["cameras"]), state["cameras"].size, d(state["points"]),
        state["points"].size, d(state["pixels"]), state["pixels"].size, u(state["indices"]), state["indices"].size,
        u(state["offsets"]), state["offsets"].size, u(state["flags"]), state["flags"].size, d(state["summary"]), None)
    if status != _lib.TBA_OK:
        raise RuntimeError(lib.tba_last_error(dev.handle).decode())
    return {"flags": state["flags"], "summary": state["summary"]}


def expected(case):
    """About how many observations a scene of the case has (views x points seen)."""
    mean = {"ring": case["C"], "arc": min(6.5, (3 + case["C"]) / 2), "helix": 7.5, "sphere": 6.1}[case["kind"]]
    return case["P"] * mean


def work(case):
    """Each input read once and each output written once; the operations of the linearisations, the
    point and camera blocks and the candidate's cost, about 600 an observation and iteration (the
    linear solve's share depends on its method and is left out)."""
    op = case["op"]
    if op == "rows":
        return {"bytes": 456.0 * case["rows"], "flops": 250.0 * case["rows"]}
    if op == "batch":
        cases = [{"op": "solve", "kind": "arc", "C": C, "P": P, "iterations": case["iterations"]}
                 for C, P in window_sizes(case)]
        each = [work(c) for c in cases]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    C, P, M = case["C"], case["P"], expected(case)
    if op == "observations":
        return {"bytes": 144.0 * C + 24 * P + 28 * M + (8.0 * P if case["bound"] else 0.0), "flops": 120.0 * M}
    scene_bytes = 144.0 * C + 24 * P + 28 * M + 4 * P + 8 * C
    solution = 96.0 * C + 24 * P
    if op == "vjp":
        return {"bytes": scene_bytes + 2 * solution + 16 * M, "flops": 2500.0 * M * (1 + case["newton"])}
    if op == "resident":
        return {"bytes": scene_bytes + 2 * solution, "flops": 2 * 600.0 * M * case["iterations"]}
    return {"bytes": scene_bytes + solution, "flops": 600.0 * M * case["iterations"]}


# ---- the same results from plain torch in 64 bits -----------------------------------------------------

def project_rows(q, cams):
    """Pixel offsets from the principal point and their derivative by the camera-frame point."""
    iz = 1 / q[:, 2]
    x, y = q[:, 0] * iz, q[:, 1] * iz
    r2 = x * x + y * y
    d = 1 + cams[:, 4] * r2 + cams[:, 5] * r2 * r2
    g = 2 * (cams[:, 4] + 2 * cams[:, 5] * r2)
    xx, xy, yy = d + g * x * x, g * x * y, d + g * y * y
    off = torch.stack([cams[:, 0] * x * d, cams[:, 1] * y * d], dim=1)
    du = (cams[:, 0] * iz)[:, None] * torch.stack([xx, xy, -(xx * x + xy * y)], dim=1)
    dv = (cams[:, 1] * iz)[:, None] * torch.stack([xy, yy, -(xy * x + yy * y)], dim=1)
    return off, torch.stack([du, dv], dim=1)


def exp_so3(w):
    K = torch.zeros(len(w), 3, 3, device=w.device, dtype=F64)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 0] = -w[:, 2], w[:, 1], w[:, 2]
    K[:, 1, 2], K[:, 2, 0], K[:, 2, 1] = -w[:, 0], -w[:, 1], w[:, 0]
    th = w.norm(dim=1)
    tiny = th < 1e-7
    s = torch.where(tiny, torch.ones_like(th), th)
    a = torch.where(tiny, 1 - th * th / 6, s.sin() / s)[:, None, None]
    b = torch.where(tiny, 0.5 - th * th / 24, (1 - s.cos()) / (s * s))[:, None, None]
    return torch.eye(3, device=w.device, dtype=F64) + a * K + b * (K @ K)


class Solve:
    """The bundle adjustment in plain torch: Levenberg-Marquardt steps, each by conjugate gradients on
    the point-eliminated system, with the entry point's damping, stopping and acceptance rules."""

    def __init__(self, s, case, max_cg, huber=2.0, tol=1e-6):
        self.s, self.shared, self.max_cg, self.huber, self.tol = s, case["shared"], max_cg, huber, tol
        self.poses, self.points = s["poses0"].clone(), s["points0"].clone()
        self.log_focal = 0.0
        self.free = s["active"].double()
        self.dir = (s["p"] >= s["P"] - s["D"])

    def sum_by(self, index, n, v):
        return torch.zeros(n, *v.shape[1:], device="cuda", dtype=F64).index_add_(0, index, v)

    def cameras(self, log_focal):
        cams = self.s["cams0"].clone()
        cams[:, :2] *= math.exp(log_focal)
        return cams

    def frame(self, poses, points):
        s = self.s
        X = points[s["p"]]
        q = (poses[s["c"], :9].reshape(-1, 3, 3) @ X[:, :, None])[:, :, 0]
        return q + torch.where(self.dir[:, None], 0.0, 1.0) * poses[s["c"], 9:]

    def cost(self, poses, points, log_focal):
        cams = self.cameras(log_focal)[self.s["c"]]
        q = self.frame(poses, points)
        r = project_rows(q, cams)[0] + cams[:, 2:4] - self.s["px"]
        sq = (r * r).sum(1)
        e = sq.sqrt()
        cost = torch.where(e <= self.huber, sq, 2 * self.huber * e - self.huber ** 2)
        # Outside the lens model's domain (behind the camera, beyond the radial fold) a candidate costs 1e30.
        r2 = (q[:, :2] ** 2).sum(1) / q[:, 2] ** 2
        bad = ~((q[:, 2] > 1e-12) & (r2 < -1 / (3 * cams[:, 4])))
        return float(torch.where(bad, 1e30, cost).sum()), float(torch.where(bad, 1e30, sq).sum())

    def adjust(self, iterations, stall):
        s, h = self.s, self.huber
        self.log_focal = 0.0  # the scene's cameras keep their focal lengths between adjustments
        c, p, C, P = s["c"], s["p"], s["C"], s["P"]
        lam = 1e-3
        R0 = self.poses[0, :9].reshape(3, 3)
        origin = -R0.T @ self.poses[0, 9:]

        def baseline(poses):
            return float((-poses[1, :9].reshape(3, 3).T @ poses[1, 9:] - origin).norm())

        base = baseline(self.poses)
        first = cost, sse = self.cost(self.poses, self.points, self.log_focal)
        for _ in range(iterations):
            cams = self.cameras(self.log_focal)[c]
            q = self.frame(self.poses, self.points)
            jf, D = project_rows(q, cams)
            r = jf + cams[:, 2:4] - s["px"]
            sq = (r * r).sum(1)
            w = torch.where(sq > h * h, h / sq.sqrt().clamp(min=1e-300), 1.0)
            Jp = D @ self.poses[c, :9].reshape(-1, 3, 3)
            Jc = torch.cat([torch.linalg.cross(q[:, None, :].expand_as(D), D),
                            D * torch.where(self.dir[:, None, None], 0.0, 1.0)], dim=2)
            Jc = Jc * self.free[c][:, None, None]
            W = (w[:, None, None] * Jc).transpose(1, 2) @ Jp
            V = self.sum_by(p, P, (w[:, None, None] * Jp).transpose(1, 2) @ Jp)
            bp = -self.sum_by(p, P, ((w[:, None] * r)[:, None, :] @ Jp)[:, 0])
            diag = torch.diagonal(V, dim1=1, dim2=2)
            V = V + torch.diag_embed(lam * diag.clamp(min=1e-10))
            Vi = torch.linalg.inv(V)
            Vi = (Vi + Vi.transpose(1, 2)) / 2
            U = self.sum_by(c, C, (w[:, None, None] * Jc).transpose(1, 2) @ Jc)
            bc = -self.sum_by(c, C, ((w[:, None] * r)[:, None, :] @ Jc)[:, 0])
            diag = torch.diagonal(U, dim1=1, dim2=2)
            U = U + torch.diag_embed(lam * diag.clamp(min=1e-10))
            on = self.free[:, None, None]
            U = U * on + torch.eye(6, device="cuda", dtype=F64) * (1 - on)
            WV = W @ Vi[p]
            Sd = U - self.sum_by(c, C, WV @ W.transpose(1, 2))
            Mi = torch.linalg.inv(Sd)
            rhs = (bc - self.sum_by(c, C, (WV @ bp[p][:, :, None])[:, :, 0])) * self.free[:, None]
            ff = bf = 0.0
            if self.shared:
                gp = self.sum_by(p, P, ((w[:, None] * jf)[:, None, :] @ Jp)[:, 0])
                hcf = self.sum_by(c, C, ((w[:, None] * jf)[:, None, :] @ Jc)[:, 0])
                hff = float((w * (jf * jf).sum(1)).sum())
                hff += lam * max(hff, 1e-10)
                Vg = (Vi @ gp[:, :, None])[:, :, 0]
                scf = hcf - self.sum_by(c, C, (W @ Vg[p][:, :, None])[:, :, 0])
                ff = hff - float((Vg * gp).sum())
                bf = -float((w * (jf * r).sum(1)).sum()) - float((Vg * bp).sum())

            def product(x, xf):
                t = self.sum_by(p, P, (W.transpose(1, 2) @ x[c][:, :, None])[:, :, 0])
                y = (Vi @ t[:, :, None])[:, :, 0]
                out = (U @ x[:, :, None])[:, :, 0] - self.sum_by(c, C, (W @ y[p][:, :, None])[:, :, 0])
                return (out + scf * xf, float((scf * x).sum()) + ff * xf) if self.shared else (out, 0.0)

            x, xf = torch.zeros_like(rhs), 0.0
            res, resf = rhs, bf
            z, zf = (Mi @ res[:, :, None])[:, :, 0], (resf / ff if self.shared else 0.0)
            d, df = z, zf
            rho = float((res * z).sum()) + resf * zf
            r0 = r2 = float((res * res).sum()) + resf * resf
            for _ in range(self.max_cg):
                if not r0 > 0:
                    break
                Sd_, Sf = product(d, df)
                alpha = rho / (float((d * Sd_).sum()) + df * Sf)
                x, xf = x + alpha * d, xf + alpha * df
                res, resf = res - alpha * Sd_, resf - alpha * Sf
                z, zf = (Mi @ res[:, :, None])[:, :, 0], (resf / ff if self.shared else 0.0)
                r2 = float((res * res).sum()) + resf * resf
                if r2 <= self.tol ** 2 * r0:
                    break
                new = float((res * z).sum()) + resf * zf
                beta, rho = new / rho, new
                d, df = z + beta * d, zf + beta * df
            taken = False
            if r2 <= self.tol ** 2 * r0:
                dR = exp_so3(x[:, :3])
                R = dR @ self.poses[:, :9].reshape(-1, 3, 3)
                t = (dR @ self.poses[:, 9:, None])[:, :, 0] + x[:, 3:]
                trial = torch.where(self.free[:, None] > 0, torch.cat([R.reshape(-1, 9), t], dim=1), self.poses)
                Wx = (W.transpose(1, 2) @ x[c][:, :, None])[:, :, 0]
                if self.shared:
                    Wx = Wx + ((w[:, None] * jf)[:, None, :] @ Jp)[:, 0] * xf
                X = self.points + (Vi @ (bp - self.sum_by(p, P, Wx))[:, :, None])[:, :, 0]
                if int((self.free == 0).sum()) == 1:
                    k = base / baseline(trial)
                    Ro = (trial[:, :9].reshape(-1, 3, 3) @ origin)
                    moved = trial.clone()
                    moved[:, 9:] = k * trial[:, 9:] + (k - 1) * Ro
                    moved[0] = trial[0]
                    trial = moved
                    scaled = origin + k * (X - origin)
                else:
                    scaled = X
                if s["D"]:
                    scaled = scaled.clone()
                    scaled[-s["D"]:] = torch.nn.functional.normalize(X[-s["D"]:], dim=1)
                lf = self.log_focal + xf
                new_cost, new_sse = self.cost(trial, scaled, lf)
                taken = new_cost < cost
            if taken:
                change = cost - new_cost
                self.poses, self.points, self.log_focal, cost, sse = trial, scaled, lf, new_cost, new_sse
                lam = max(1e-10, lam / 3)
                if change < max(stall, 1e-9) * max(1.0, cost):
                    break
            else:
                lam *= 10
                if lam > 1e12:
                    break
        return torch.tensor([cost, sse, *first], dtype=F64)


def exact_rows(m):
    R, S = m[:, 3:12].reshape(-1, 3, 3), m[:, 15:24].reshape(-1, 3, 3)
    centre = -(R.transpose(1, 2) @ m[:, 12:15, None])
    A = S @ R.transpose(1, 2)
    T = (S @ centre)[:, :, 0] + m[:, 24:27]
    q = m[:, 0:1] * A[:, :, 0] + m[:, 1:2] * A[:, :, 1] + A[:, :, 2] + m[:, 2:3] * T
    off, J = project_rows(q, m[:, 27:33])
    point = J @ torch.stack([A[:, :, 0], A[:, :, 1], T], dim=2)
    turn = torch.linalg.cross(q[:, None, :].expand_as(J), J)
    pose = torch.cat([turn, m[:, 2, None, None] * J], dim=2)
    n = len(m)
    out = torch.cat([torch.ones(n, 1, device="cuda", dtype=F64), off + m[:, 29:31], point.reshape(n, 6),
                     pose.reshape(n, 12), off], dim=1)
    return out


def exact_observations(case, s):
    c, p, X = s["c"], s["p"], s["points"]
    q = camera_frame(s["poses"], c, X[p])
    off, J = project_rows(q, s["cams"][c])
    e = (off + s["cams"][c, 2:4] - s["px"]).norm(dim=1)
    inlier = (e <= 3.0)
    flags = inlier.to(torch.int64)
    if case["bound"] > 0:
        R = s["poses"][c, :9].reshape(-1, 3, 3)
        Jp = J @ R
        info = torch.zeros(s["P"], 3, 3, device="cuda", dtype=F64).index_add_(
            0, p, inlier.double()[:, None, None] * (Jp.transpose(1, 2) @ Jp))
        count = torch.zeros(s["P"], device="cuda", dtype=F64).index_add_(0, p, inlier.double())
        checked = inlier & (count[p] >= 2)
        axis = R[:, 2]
        var = torch.zeros(s["M"], device="cuda", dtype=F64)
        some = torch.linalg.solve(info[p[checked]], axis[checked])
        var[checked] = (axis[checked] * some).sum(1)
        bad = checked & ~(var.sqrt() / q[:, 2] <= case["bound"])
        rejected = torch.zeros(s["P"], device="cuda", dtype=F64).index_add_(0, p, bad.double()) > 0
        inlier &= ~rejected[p]
        flags = torch.cat([inlier.to(torch.int64), rejected.to(torch.int64)])
    total = torch.stack([(e * inlier).sum(), inlier.double().sum()])
    return {"flags": flags, "summary": total}


def exact_adjoint(case, s, seed):
    """The vector-Jacobian product at the scene's state: the exact Hessian of the robust cost by
    automatic differentiation, and a dense solve of its point-eliminated system."""
    c, p, C, P, M, h = s["c"], s["p"], s["C"], s["P"], s["M"], 2.0
    poses, X = s["poses"], s["points"]
    R, t = poses[:, :9].reshape(-1, 3, 3), poses[:, 9:]
    free = s["active"].double()
    q0, Ro = camera_frame(poses, c, X[p]), R[c]

    def cost(step, y, focal, k1):
        step = torch.cat([step[:, :6] * free[c][:, None], step[:, 6:]], dim=1)
        w, v = step[:, :3], step[:, 3:6]
        q = q0 + (Ro @ step[:, 6:, None])[:, :, 0]
        wq = torch.linalg.cross(w, q)
        q = q + wq + torch.linalg.cross(w, wq) / 2 + v
        cams = torch.cat([s["cams"][c, :2] * torch.exp(focal), s["cams"][c, 2:4], s["cams"][c, 4:5] + k1,
                          s["cams"][c, 5:]], dim=1)
        sq = ((pixels_of(cams, q)[0] - y) ** 2).sum(1)
        e = sq.sqrt()
        return torch.where(e <= h, sq, 2 * h * e - h * h) / 2

    step = torch.zeros(M, 9, device="cuda", dtype=F64, requires_grad=True)
    y = s["px"].clone().requires_grad_()
    focal, k1 = (torch.zeros(1, device="cuda", dtype=F64, requires_grad=True) for _ in range(2))
    grad = torch.autograd.grad(cost(step, y, focal, k1).sum(), step, create_graph=True)[0]
    H = torch.stack([torch.autograd.grad(grad[:, a].sum(), step, retain_graph=True)[0] for a in range(9)], dim=1)
    H = H.detach()
    V = torch.zeros(P, 3, 3, device="cuda", dtype=F64).index_add_(0, p, H[:, 6:, 6:])
    # A block that is not definite is shifted by the smallest power of ten of its mean diagonal that makes it so.
    I3, scale = torch.eye(3, device="cuda", dtype=F64), (torch.diagonal(V, dim1=1, dim2=2).sum(1).abs() / 3).clamp(min=1e-12)
    shifted = V
    for k in range(-8, 3):
        bad = torch.linalg.cholesky_ex(shifted)[1] > 0
        shifted = torch.where(bad[:, None, None], V + 10.0 ** k * scale[:, None, None] * I3, shifted)
    L = torch.linalg.cholesky(torch.linalg.inv(shifted))
    A = torch.zeros(P * C, 6, 3, device="cuda", dtype=F64).index_add_(0, p * C + c, H[:, :6, 6:] @ L[p])
    A = A.reshape(P, C, 6, 3).permute(0, 3, 1, 2).reshape(3 * P, 6 * C)
    U = torch.zeros(C, 6, 6, device="cuda", dtype=F64).index_add_(0, c, H[:, :6, :6])
    # The gauge: the cotangent projected along the scale, and the baseline's gradient made definite.
    origin = -R[0].T @ t[0]
    e = -R[1].T @ t[1] - origin
    n = -(R[1] @ e) / e.norm()
    mu = torch.diagonal(U[1])[3:].mean().clamp(min=1e-12)
    U[1, 3:, 3:] += mu * torch.outer(n, n)
    U = torch.where(free[:, None, None] > 0, U, torch.eye(6, device="cuda", dtype=F64))
    g = cotangent(s, seed)
    gR, gt = g[:12 * C].reshape(C, 12)[:, :9].reshape(C, 3, 3), g[:12 * C].reshape(C, 12)[:, 9:]
    gX = g[12 * C:].reshape(P, 3)
    B = gR @ R.transpose(1, 2)
    turn = torch.stack([B[:, 2, 1] - B[:, 1, 2], B[:, 0, 2] - B[:, 2, 0], B[:, 1, 0] - B[:, 0, 1]], dim=1)
    gc = torch.cat([turn + torch.linalg.cross(t, gt), gt], dim=1) * free[:, None]
    dot = ((t + R @ origin) * gt * free[:, None]).sum() + ((X - origin) * gX).sum()
    gc[1, 3:] -= n * dot / e.norm()
    S = torch.block_diag(*U) - A.T @ A
    rhs = gc.reshape(-1) - A.T @ (L.transpose(1, 2) @ gX[:, :, None]).reshape(-1)
    x = torch.linalg.solve(S, rhs)
    lp = (L @ (L.transpose(1, 2) @ gX[:, :, None] - (A @ x).reshape(P, 3, 1)))[:, :, 0]
    lam = torch.cat([x.reshape(C, 6)[c] * free[c][:, None], lp[p]], dim=1)
    bars = torch.autograd.grad((grad * lam).sum(), [y, focal, k1])
    return {"pixels": -bars[0].cpu(), "intrinsics": -torch.cat(bars[1:]).cpu(),
            "solution": torch.cat([poses.reshape(-1), X.reshape(-1)]).cpu()}


def max_cg_of(case):
    C = case["C"]
    return min(256, max(32, 12 * C + 1)) if case["shared"] else min(96, max(24, 12 * C))


def exact(case, seed):
    op = case["op"]
    if op == "rows":
        return exact_rows(depth_rows(case, seed)).cpu()
    if op == "batch":
        if case["count"] > 24:
            return None
        parts = {"poses": [], "points": [], "cost": [], "focal": []}
        for s in windows(case, seed):
            S = Solve(s, case, 256)
            parts["cost"].append(S.adjust(case["iterations"], 1e-9))
            parts["poses"].append(S.poses.reshape(-1).cpu())
            parts["points"].append(S.points.reshape(-1).cpu())
            parts["focal"].append(torch.tensor([S.log_focal], dtype=F64))
        if not case["shared"]:
            del parts["focal"]
        return {k: torch.cat(v) for k, v in parts.items()}
    if op == "vjp":  # after Newton steps the point is the solver's own
        return None if case["newton"] else exact_adjoint(case, scene(dict(case, outliers=0.0), seed), seed)
    s = scene(case, seed)
    if op == "observations":
        return {k: v.cpu() for k, v in exact_observations(case, s).items()}
    S = Solve(s, case, max_cg_of(case))
    cost = S.adjust(case["iterations"], 1e-9)
    if op == "resident":
        first, cost = cost, S.adjust(case["iterations"], 1e-9)
        return {"poses": S.poses.reshape(-1).cpu(), "points": S.points.reshape(-1).cpu(), "first": first, "last": cost}
    parts = {"poses": S.poses.reshape(-1).cpu(), "points": S.points.reshape(-1).cpu(), "cost": cost}
    if case["shared"]:
        parts["focal"] = torch.tensor([S.log_focal], dtype=F64)
    return parts
