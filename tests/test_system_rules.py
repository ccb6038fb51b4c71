"""Which form a call solves on, and what the explicit reduced system may cost a call that gains nothing by
it: the rule's two sides, a call without iterations, and a device whose memory is taken."""
import numpy as np
import pytest

import typecv_b200 as tb
from oracle.adjoint_dense import Problem
from typecv_b200 import _lib
from typecv_b200 import adjoint as AD
from typecv_b200 import batch as B
from typecv_b200 import synthetic as S
from typecv_b200.bundle import pack_arrays
from typecv_b200.resident import ResidentScene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


def solve(device, sc, packed=None, flags=0, **kw):
    s, i = packed or sc.packed()
    return tb.solve_packed(device, tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, flags=flags, **kw), s, i)


@pytest.mark.parametrize("shared", [False, True])
def test_a_call_without_iterations_forms_no_system(device, shared):
    sc = S.ring_scene(seed=1, cameras=7, points=301)
    out, rep = solve(device, sc, iterations=0, shared_focal=shared)
    # The set-up (2), the cost (2) and the result (1), with the checks of the arrays uncounted.
    assert rep["engine"] == 0 and rep["lm_iterations"] == 0 and rep["kernel_launches"] <= 5
    after, more = solve(device, sc, iterations=1, shared_focal=shared)
    base = 12 * sc.C + 3 * sc.P
    assert more["engine"] == 2 and out[base + 6] == out[base + 8] == after[base + 8]


class Taken:
    """Device memory taken until at most `left` bytes are free."""

    def __init__(self, left):
        import torch
        self.torch, self.parts = torch, []
        while torch.cuda.mem_get_info()[0] - left > 4 << 20:
            size = torch.cuda.mem_get_info()[0] - left
            self.parts.append(torch.empty(size // (2 << 20) * (2 << 20), dtype=torch.uint8, device="cuda"))

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.parts.clear()
        self.torch.cuda.empty_cache()


def test_a_resident_scene_takes_the_room_of_the_last_solves_system():
    kept = S.sphere_scene(seed=14, cameras=801, points=30_001)  # over 180 MB of S beside a small scene
    large = S.helix_scene(seed=15, cameras=60, points=60_001)   # 14 MB
    with tb.ShadeDevice.open(0) as dev:
        out, rep = solve(dev, kept, iterations=2)
        assert rep["engine"] == 2
        ctl = tb.make_control(large.C, large.P, large.M, anchor=0, scale_view=1, iterations=2)
        s, i = large.packed()
        with Taken(6 << 20), ResidentScene(dev, ctl, s, i) as scene:
            poses, points = scene.read()
            assert np.array_equal(poses, s[:12 * large.C]) and np.array_equal(points, s[12 * large.C:][:3 * large.P])
        again, rep = solve(dev, kept, iterations=2)
        base = 12 * kept.C + 3 * kept.P
        assert rep["engine"] == 2 and abs(again[base + 6] - out[base + 6]) <= 1e-9 * out[base + 6]


@pytest.fixture(scope="module")
def dense_ring():
    # Every one of 26 cameras sees every point, 12.5 pairs an observation: on the edge of the rule.
    sc = S.ring_scene(seed=1, cameras=26, points=80_000)
    assert sc.M == 26 * 80_000
    return sc, sc.packed()


@pytest.mark.parametrize("precision,options,engine", [
    (0, dict(), 2), (1, dict(), 2),                                          # 22 steps an iteration
    (0, dict(tolerance=1e-3), 2), (1, dict(tolerance=1e-3), 0),              # 14: the FP32 product's are cheaper
    (0, dict(tolerance=1e-2), 0), (1, dict(tolerance=1e-2), 0),              # 10
    (0, dict(max_cg=16), 0), (1, dict(max_cg=16), 2),                        # 14 and, with restarts, 32
    (0, dict(max_cg=24), 2), (0, dict(max_cg=1), 0), (1, dict(max_cg=1), 0)])
def test_short_solves_of_long_tracks_keep_the_product(device, dense_ring, precision, options, engine):
    sc, packed = dense_ring
    out, rep = solve(device, sc, packed, iterations=1, precision=precision, **options)
    assert rep["engine"] == engine
    base = 12 * sc.C + 3 * sc.P
    assert out[base + 6] <= out[base + 8]


@pytest.mark.parametrize("cameras,points,engine", [(300, 50, 2), (400, 30, 2), (600, 30, 0), (600, 10, 0)])
def test_a_full_system_beyond_the_caches_is_not_formed(device, cameras, points, engine):
    # Every camera sees every point: S is full, 26, 46 and 104 MB.
    sc = S.ring_scene(seed=3, cameras=cameras, points=points)
    _, rep = solve(device, sc, iterations=1)
    assert sc.M == cameras * points and rep["engine"] == engine


def scattered(cameras, points, track, seed=1):
    """Points near the origin, each seen by cameras picked at random from a sphere around it: any two cameras
    share points."""
    rng = np.random.default_rng(seed)
    like = S.sphere_scene(seed=seed, cameras=cameras, points=64, track_mean=20.0)
    pick = np.sort(np.argsort(rng.random((points, cameras)), axis=1)[:, :track], axis=1)
    return S.finish("scattered", rng, like.truth_poses, like.truth_cameras, rng.normal(size=(points, 3)), pick.ravel(),
                    np.repeat(np.arange(points), track), width=1024, height=768)


@pytest.mark.parametrize("kind,cameras,points,engine", [
    ("scattered", 400, 12_000, 2), ("scattered", 900, 30_000, 0), ("scattered", 1500, 30_000, 0), ("sphere", 900, 30_000, 2),
    ("sphere", 1500, 60_000, 2), ("helix", 1000, 30_000, 2)])
def test_cameras_that_all_share_points_form_no_large_system(kind, cameras, points, engine):
    # The same sizes, and systems of 30 to 500 MB where neighbours alone would make 4 to 52.
    sc = scattered(cameras, points, 5) if kind == "scattered" else \
        (S.sphere_scene if kind == "sphere" else S.helix_scene)(seed=3, cameras=cameras, points=points)
    packed = sc.packed()
    with tb.ShadeDevice.open(0) as dev:
        out, rep = solve(dev, sc, packed, iterations=2, tolerance=1e-9, max_cg=200)
        assert rep["engine"] == engine
        # A resident scene, and the adjoint, take the same side.
        ctl = tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=2, tolerance=1e-9, max_cg=200)
        with ResidentScene(dev, ctl, *packed) as scene:
            kept, _, rep = scene.adjust(output=True)
        base = 12 * sc.C + 3 * sc.P
        assert rep["engine"] == engine and abs(kept[base + 6] - out[base + 6]) <= 1e-9 * out[base + 6]
        _, _, _, rep = AD.bundle_vjp(dev, sc.C, sc.P, sc.M, *packed, np.zeros(base), max_cg=200, tolerance=1e-6)
        assert (rep["product_blocks"] == 0) == (engine == 2)


@pytest.mark.parametrize("shared", [False, True])
def test_the_product_error_of_a_mixed_request_is_the_fp32_products(device, shared):
    # FP32 rounds the factors at 6e-8; averaged over a camera's thousands of observations that leaves more than
    # 1e-11 of S p (FP64's product leaves less than 1e-12 there).
    sc = S.ring_scene(seed=11)
    kw = dict(iterations=2, shared_focal=shared, tolerance=1e-8, max_cg=200)
    _, fp64 = solve(device, sc, flags=_lib.TBA_FLAG_PRODUCT_ERROR, precision=0, **kw)
    out, mixed = solve(device, sc, flags=_lib.TBA_FLAG_PRODUCT_ERROR, precision=1, **kw)
    assert fp64["engine"] == 2 and fp64["product_error_norm"] < 1e-12
    assert mixed["engine"] == 0 and 1e-11 < mixed["product_error_norm"] < 1e-5
    plain, rep = solve(device, sc, precision=1, **kw)
    base = 12 * sc.C + 3 * sc.P
    assert rep["engine"] == 2 and abs(out[base + 6] - plain[base + 6]) <= 1e-6 * plain[base + 6]


def test_a_system_that_does_not_fit_leaves_the_product():
    # 801 cameras: over 180 MB of S beside a workspace of 40 MB, the adjoint's of 100.
    sc = S.sphere_scene(seed=14, cameras=801, points=30_001, outlier_rate=0.0)
    s, i = sc.packed()
    kw = dict(iterations=3, tolerance=1e-9, max_cg=200)
    n = 12 * sc.C + 3 * sc.P
    g = np.random.default_rng(3).normal(size=n)
    g /= np.linalg.norm(g)
    with tb.ShadeDevice.open(0) as dev:
        want, rep = solve(dev, sc, (s, i), **kw)
        assert rep["engine"] == 2
        at, _ = solve(dev, sc, (s, i), iterations=20, tolerance=1e-10, max_cg=256)
        there = np.concatenate([at[:n], s[n:]])
        ybar, kbar, _, rep = AD.bundle_vjp(dev, sc.C, sc.P, sc.M, there, i, g)
        assert rep["failed"] == 0 and rep["product_blocks"] == 0
    with tb.ShadeDevice.open(0) as dev, Taken(150 << 20):
        got, rep = solve(dev, sc, (s, i), **kw)
        assert rep["engine"] == 0 and abs(got[n + 6] - want[n + 6]) <= 1e-9 * want[n + 6]
        assert np.max(np.abs(got[:12 * sc.C] - want[:12 * sc.C])) < 1e-7
        y2, k2, _, rep = AD.bundle_vjp(dev, sc.C, sc.P, sc.M, there, i, g)
        assert rep["failed"] == 0 and rep["product_blocks"] > 0
        assert np.linalg.norm(y2 - ybar) <= 1e-8 * np.linalg.norm(ybar)
        assert np.all(np.abs(k2 - kbar) <= 1e-8 * np.abs(kbar) + 1e-12)
    with tb.ShadeDevice.open(0) as dev:  # with the memory back, so is the system
        _, rep = solve(dev, sc, (s, i), **kw)
        assert rep["engine"] == 2


def test_windows_whose_systems_do_not_fit_run_on_the_persistent_launch():
    # 64 MB with their systems, 30 without.
    scenes = [S.arc_scene(seed=100 + k, cameras=40, points=4000 + k, track=(8, 10)) for k in range(6)]
    probs = [B.PackedProblem(sc.C, sc.P, sc.M, *sc.packed(), sc.anchor, sc.scale_view) for sc in scenes]
    kw = dict(iterations=4, precision="fp64", max_cg=200)
    with tb.ShadeDevice.open(0) as dev:
        want, rep = B.batch_adjust(dev, probs, **kw)
        want = [r.copy() for r in want]
        assert rep["schedule"] == 4
        for schedule in (1, 2, 3, 4):  # (the kernels' stacks are allocated once a process)
            B.batch_adjust(dev, probs, schedule=schedule, **kw)
    with tb.ShadeDevice.open(0) as dev, Taken(48 << 20):
        with pytest.raises(tb.RangeError, match="budget"):
            B.batch_adjust(dev, probs, schedule=5, **kw)
        got, rep = B.batch_adjust(dev, probs, **kw)
        assert rep["schedule"] < 4 and rep["tune_ms"] > 0
        for sc, a, b in zip(scenes, got, want):
            base = 12 * sc.C + 3 * sc.P
            assert abs(a[base + 6] - b[base + 6]) <= 1e-9 * b[base + 6]
            assert np.max(np.abs(a[:12 * sc.C] - b[:12 * sc.C])) < 1e-7


@pytest.mark.parametrize("shared", [False, True])
def test_a_mixed_request_keeps_the_budgets_of_its_runs(device, shared):
    # The mixed form's PCG takes up to four runs of the budget (two in a batch); on the explicit system its one run
    # takes as many steps.  An FP64 request's solve ends, and fails, with its budget.
    sc = S.ring_scene(seed=1, cameras=7, points=301)
    packed = sc.packed()
    base = 12 * sc.C + 3 * sc.P
    kw = dict(iterations=1, shared_focal=shared, tolerance=1e-6)
    free, rep = solve(device, sc, packed, max_cg=200, **kw)
    steps = rep["cg_iterations"]
    assert rep["engine"] == 2 and steps >= 10 and free[base + 10] == 1
    few = steps // 2 + 1
    out, _ = solve(device, sc, packed, max_cg=few, **kw)
    assert out[base + 10] == 0 and out[base + 17] == 1
    for flags in (0, _lib.TBA_FLAG_HOST_PCG_LOOP):
        out, rep = solve(device, sc, packed, max_cg=few, precision=1, flags=flags, **kw)
        assert rep["engine"] == 2 and abs(rep["cg_iterations"] - steps) <= 1
        assert out[base + 10] == 1 and out[base + 17] == 0
        assert abs(out[base + 6] - free[base + 6]) <= 1e-9 * free[base + 6]
    out, rep = solve(device, sc, packed, max_cg=steps // 5, precision=1, **kw)
    assert rep["cg_iterations"] == 4 * (steps // 5) and out[base + 10] == 0 and out[base + 17] == 1
    window = B.PackedProblem(sc.C, sc.P, sc.M, *packed, sc.anchor, sc.scale_view)
    for precision, accepted in (("fp64", 0), ("mixed", 1)):
        recs, _ = B.batch_adjust(device, [window] * 2, max_cg=few, precision=precision, **kw)
        assert [r[base + 10] for r in recs] == [accepted] * 2 and recs[1][base + 17] == 1 - accepted


@pytest.mark.parametrize("fixed,system", [((0,), True), ((0, 1, 3, 4, 5), False), ((0, 1, 2, 3, 4, 5), False)])
def test_an_adjoint_of_one_variable_camera_forms_no_system(device, fixed, system):
    sc = S.arc_scene(seed=5, cameras=6, points=203, outlier_rate=0.0)
    active = np.ones(sc.C, np.uint32)
    active[list(fixed)] = 0
    s, i = pack_arrays(sc.truth_poses, sc.points, sc.truth_cameras, sc.obs_camera, sc.obs_point, sc.pixels, active)
    out, _ = solve(device, sc, (s, i), iterations=20, tolerance=1e-10)
    n = 12 * sc.C + 3 * sc.P
    s[:n] = out[:n]
    g = np.random.default_rng(6).normal(size=n)
    g /= np.linalg.norm(g)
    ybar, kbar, sol, rep = AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, g, newton_steps=2, want_solution=True)
    assert rep["failed"] == 0 and (rep["product_blocks"] == 0) == system
    s[:n] = sol
    # (differences of 1e-7: the residuals' distances to the Huber threshold are larger)
    want, _ = Problem(sc.C, sc.P, sc.M, s, i).vjp(g, h=1e-7)
    assert np.linalg.norm(ybar - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("kind,count,cameras,points,track,grid", [
    ("scattered", 2, 60, 400, 5, True), ("scattered", 2, 144, 250, 12, False), ("scattered", 2, 144, 4000, 5, True),
    ("scattered", 150, 144, 300, 5, False), ("arc", 2, 144, 600, 5, True)])
def test_windows_of_large_systems_run_on_the_persistent_launch(device, kind, count, cameras, points, track, grid):
    base = [scattered(cameras, points, track, seed=k) if kind == "scattered" else
            S.arc_scene(seed=k, cameras=cameras, points=points, track=(track - 1, track + 1)) for k in range(2)]
    probs = [B.PackedProblem(sc.C, sc.P, sc.M, *sc.packed(), sc.anchor, sc.scale_view) for sc in base] * (count // 2)
    kw = dict(iterations=3, max_cg=256, tolerance=1e-9)
    recs, rep = B.batch_adjust(device, probs, precision="fp64", **kw)
    assert (rep["schedule"] == 4) == grid
    for sc, rec in zip(base, recs):
        out, _ = solve(device, sc, **kw)
        n = 12 * sc.C + 3 * sc.P
        assert abs(rec[n + 6] - out[n + 6]) <= 1e-9 * out[n + 6]
