"""The forms that solve without the explicit reduced system, on problems that its rule leaves to them: the
product over stored factors in FP64 and in the mixed form (FP32 staged, FP64 staged and not), its restarts and its
FP64 finish, the adjoint's one-pass and two-pass products, and the persistent launches of a batch with their
tuner.  Against the oracle's operator, the dense adjoint, the other form or one call a problem."""
import numpy as np
import pytest

import typecv_b200 as tb
from oracle import bundle_adjust as ob
from oracle.adjoint_dense import Problem
from typecv_b200 import _lib
from typecv_b200 import adjoint as AD
from typecv_b200 import batch as B
from typecv_b200 import synthetic as S
from typecv_b200.bundle import pack_arrays

pytestmark = pytest.mark.gpu

COST_REL, MIXED_REL = 1e-9, 1e-6
POSE_ABS, MIXED_POSE_ABS = 1e-7, 1e-5


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


# Every one of 160 cameras sees every point (79.5 pairs an observation); and 3,000 cameras, whose camera sums and
# direction do not both fit a block's shared memory in FP64.
@pytest.fixture(scope="module", params=["dense", "many"])
def scene(request):
    sc = S.ring_scene(seed=3, cameras=160, points=800) if request.param == "dense" else \
        S.sphere_scene(seed=33, cameras=3000, points=5000, track=(40, 48), track_mean=44.0)
    return sc, sc.packed()


def solve(device, scene, flags=0, **kw):
    sc, (s, i) = scene
    out, rep = tb.solve_packed(device, tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, flags=flags, **kw), s, i)
    assert rep["engine"] == 0 and rep["product_blocks"] > 0
    return out, rep


def cost(scene, out):
    return out[12 * scene[0].C + 3 * scene[0].P + 6]


@pytest.mark.parametrize("shared", [False, True])
def test_both_forms_match_the_oracle(device, scene, shared):
    sc, (s, i) = scene
    kw = dict(iterations=3, shared_focal=shared, tolerance=1e-9, max_cg=200)
    fp64, r64 = solve(device, scene, precision=0, **kw)
    mixed, r32 = solve(device, scene, precision=1, **kw)
    ref = ob.gpu_operator_packed({"C": sc.C, "P": sc.P, "M": sc.M, "scene": s, "index": i}, 0, 1, iterations=3, huber=2.0,
                                 max_cg=200, shared=shared, tolerance=1e-9)
    want, base = cost(scene, ref), 12 * sc.C + 3 * sc.P
    assert abs(cost(scene, fp64) - want) <= COST_REL * want and abs(cost(scene, mixed) - want) <= MIXED_REL * want
    for out in (fp64, mixed):
        assert out[base + 10] == ref[base + 10] and out[base + 11] == ref[base + 11]
    assert np.max(np.abs(fp64[:12 * sc.C] - ref[:12 * sc.C])) < POSE_ABS
    assert np.max(np.abs(mixed[:12 * sc.C] - ref[:12 * sc.C])) < MIXED_POSE_ABS
    # A run on the FP32 product stops at 1e-6 at best: every solve to 1e-9 needs restarts.
    assert r64["refinements"] == 0 and r32["refinements"] > 0
    assert r32["cg_iterations"] > r64["cg_iterations"] > 0


@pytest.mark.parametrize("precision,low,high", [(0, 0.0, 1e-12), (1, 1e-11, 1e-5)])
@pytest.mark.parametrize("shared", [False, True])
def test_a_products_error_against_the_two_pass_product(device, scene, shared, precision, low, high):
    _, rep = solve(device, scene, flags=_lib.TBA_FLAG_PRODUCT_ERROR, iterations=1, shared_focal=shared, tolerance=1e-8,
                   max_cg=200, precision=precision)
    assert low <= rep["product_error_norm"] < high and rep["product_error_max"] < 10 * high


@pytest.mark.parametrize("precision", [0, 1])
def test_the_device_loop_matches_the_host_loop(device, scene, precision):
    # One graph of a while node a PCG run, against the same kernels launched in chunks from the host; the sums in
    # shared memory are atomic, so the two agree to the rounding that a PCG to 1e-8 carries on.
    sc, _ = scene
    rel, pose = (1e-12, 1e-6) if precision == 0 else (MIXED_REL, MIXED_POSE_ABS)
    for shared in (False, True):
        kw = dict(iterations=4, shared_focal=shared, tolerance=1e-8, max_cg=200, precision=precision)
        chunked, rc = solve(device, scene, flags=_lib.TBA_FLAG_HOST_PCG_LOOP, **kw)
        timed, rt = solve(device, scene, flags=_lib.TBA_FLAG_TIME_PRODUCTS, **kw)
        assert rc["product_launches"] == 0 < rt["product_launches"]
        for _ in range(2):  # the second call launches the first one's graph
            graph, rg = solve(device, scene, **kw)
            for out in (graph, timed):
                assert abs(cost(scene, out) - cost(scene, chunked)) <= rel * cost(scene, chunked)
                assert np.max(np.abs(out[:12 * sc.C] - chunked[:12 * sc.C])) < pose
            assert rg["lm_iterations"] == rc["lm_iterations"] and rg["product_launches"] == 0
    budget = dict(iterations=2, tolerance=1e-8, max_cg=3, precision=precision)
    _, rg = solve(device, scene, **budget)
    _, rc = solve(device, scene, flags=_lib.TBA_FLAG_HOST_PCG_LOOP, **budget)
    assert rg["lm_iterations"] == rc["lm_iterations"] > 0
    if precision == 0:
        assert 0 < rg["cg_iterations"] == rc["cg_iterations"] <= 3 * rg["lm_iterations"]


def test_the_mixed_form_finishes_on_the_fp64_product(device):
    # Two restarts on the FP32 product do not reach 1e-12 in every solve of these.
    finished = 0
    for shared in (False, True):
        for seed in (3, 4):
            sc = S.ring_scene(seed=seed, cameras=160, points=800)
            scene = sc, sc.packed()
            kw = dict(iterations=6, shared_focal=shared, tolerance=1e-12, max_cg=256)
            fp64, _ = solve(device, scene, precision=0, **kw)
            mixed, rep = solve(device, scene, precision=1, **kw)
            finished += rep["fp64_iterations"]
            assert rep["refinements"] > 0 and abs(cost(scene, mixed) - cost(scene, fp64)) <= COST_REL * cost(scene, fp64)
            assert np.max(np.abs(mixed[:12 * sc.C] - fp64[:12 * sc.C])) < POSE_ABS
    assert finished > 0


# ---- the adjoint ----------------------------------------------------------------------------------


def stationary(device, sc, active):
    """The scene packed at its own solution for fixed intrinsics, from the true cameras, with these variable."""
    s, i = pack_arrays(sc.truth_poses, sc.points, sc.truth_cameras, sc.obs_camera, sc.obs_point, sc.pixels, active)
    out, _ = tb.solve_packed(device, tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=20, max_cg=256,
                                                     tolerance=1e-10), s, i)
    n = 12 * sc.C + 3 * sc.P
    s[:n] = out[:n]
    return s, i


def with_idle_cameras(C, P, M, s, i, total):
    """The same problem after `total` - C fixed cameras that see nothing."""
    extra = total - C
    pose = np.concatenate([np.eye(3).ravel(), np.zeros(3)])
    scene = np.concatenate([s[:12 * C], np.tile(pose, extra), s[12 * C:12 * C + 3 * P], s[12 * C + 3 * P:18 * C + 3 * P],
                            np.tile([800.0, 800, 512, 384, 0, 0], extra), s[18 * C + 3 * P:]])
    ends = 2 * M + P + 1 + C + 1
    index = np.concatenate([i[:ends], np.full(extra, M, np.uint32), i[ends:ends + M + C], np.zeros(extra, np.uint32)])
    return scene, index.astype(np.uint32)


MANY = 5000  # cameras whose sums do not fit a block's shared memory: the two-pass product


def vjp(device, C, P, M, s, i, g, total, **kw):
    n = 12 * C
    scene, index = with_idle_cameras(C, P, M, s, i, total) if total > C else (s, i)
    cot = np.concatenate([g[:n], np.zeros(12 * (total - C)), g[n:]])
    ybar, kbar, sol, rep = AD.bundle_vjp(device, total, P, M, scene, index, cot, want_solution=True, **kw)
    assert rep["failed"] == 0 and rep["adjoint_residual"] < 1e-10
    return ybar, kbar, np.concatenate([sol[:n], sol[12 * total:]]), rep


def test_the_adjoints_two_pass_product_matches_the_dense_reference(device):
    sc = S.sphere_scene(seed=12, cameras=29, points=203, outlier_rate=0.0)
    active = np.ones(sc.C, np.uint32)
    active[:2] = 0  # with more than one camera fixed, the scale's camera is
    s, i = stationary(device, sc, active)
    g = np.random.default_rng(13).normal(size=12 * sc.C + 3 * sc.P)
    g /= np.linalg.norm(g)
    ybar, kbar, sol, rep = vjp(device, sc.C, sc.P, sc.M, s, i, g, MANY, newton_steps=3)
    assert rep["product_blocks"] == 0 and rep["newton_steps"] > 0
    s[:sol.size] = sol
    ybar_d, kbar_d = Problem(sc.C, sc.P, sc.M, s, i).vjp(g)
    assert np.linalg.norm(ybar - ybar_d) <= 1e-6 * np.linalg.norm(ybar_d)
    assert np.all(np.abs(kbar - kbar_d) <= 1e-6 * np.abs(kbar_d) + 1e-12)


def test_the_adjoints_one_pass_product_matches_its_two_pass_product(device):
    # Every one of 400 cameras sees every point: 199.5 pairs an observation, beyond the rule for the system.
    sc = S.ring_scene(seed=3, cameras=400, points=500, outlier_rate=0.0)
    active = np.ones(sc.C, np.uint32)
    active[:2] = 0
    s, i = stationary(device, sc, active)
    g = np.random.default_rng(5).normal(size=12 * sc.C + 3 * sc.P)
    g /= np.linalg.norm(g)
    one, k1, sol1, r1 = vjp(device, sc.C, sc.P, sc.M, s, i, g, sc.C, newton_steps=2)
    two, k2, sol2, r2 = vjp(device, sc.C, sc.P, sc.M, s, i, g, MANY, newton_steps=2)
    assert r1["product_blocks"] > 0 and r2["product_blocks"] == 0
    assert np.max(np.abs(sol1 - sol2)) < 1e-9
    assert np.linalg.norm(one - two) <= 1e-8 * np.linalg.norm(two)
    assert np.all(np.abs(k1 - k2) <= 1e-8 * np.abs(k2) + 1e-12)
    timed, _, _, rt = vjp(device, sc.C, sc.P, sc.M, s, i, g, sc.C, newton_steps=2, time_products=True)
    assert rt["product_launches"] > 0 and np.linalg.norm(timed - one) <= 1e-8 * np.linalg.norm(one)


# ---- the batch ------------------------------------------------------------------------------------


@pytest.fixture(scope="module")
def long_track_windows():
    # Every camera sees every point, 34.5 to 47 pairs an observation: beyond the grid kernels' rule.
    scenes = [S.ring_scene(seed=70 + k, cameras=c, points=p) for k, (c, p) in enumerate([(70, 201), (95, 150), (80, 77)])]
    return scenes, [B.PackedProblem(sc.C, sc.P, sc.M, *sc.packed(), sc.anchor, sc.scale_view) for sc in scenes]


def against_single_calls(device, scenes, probs, recs, shared, rel, pose):
    for sc, p, rec in zip(scenes, probs, recs):
        want, _ = tb.solve_packed(device, tb.make_control(sc.C, sc.P, sc.M, anchor=sc.anchor, scale_view=sc.scale_view,
                                                          iterations=5, shared_focal=shared, max_cg=200), p.scene, p.index)
        base = 12 * sc.C + 3 * sc.P
        assert abs(rec[base + 6] - want[base + 6]) <= rel * want[base + 6] and rec[base + 17] == 0
        assert np.max(np.abs(rec[:12 * sc.C] - want[:12 * sc.C])) < pose


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_the_tuner_of_long_track_windows(long_track_windows, precision):
    scenes, probs = long_track_windows
    with tb.ShadeDevice.open(0) as device:
        packed = B.pack_batch(probs, True)
        kw = dict(iterations=5, shared_focal=True, precision=precision, max_cg=200)
        recs, first = B.batch_adjust(device, packed, **kw)
        recs = [r.copy() for r in recs]
        again, second = B.batch_adjust(device, packed, **kw)
        assert first["tune_ms"] > 0 and second["tune_ms"] == 0 and second["graph_replayed"] == 1
        assert first["schedule"] == second["schedule"] < 4 and first["form"] == second["form"]
        rel, pose = (COST_REL, POSE_ABS) if precision == "fp64" else (MIXED_REL, MIXED_POSE_ABS)
        against_single_calls(device, scenes, probs, recs, True, rel, pose)
        against_single_calls(device, scenes, probs, again, True, rel, pose)


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("schedule", [1, 2, 3, 4])
def test_the_mixed_form_at_every_persistent_shape(device, long_track_windows, schedule, shared):
    short = [S.arc_scene(seed=60 + k, cameras=c, points=p, track=(2, min(c, 10))) for k, (c, p) in enumerate([(5, 301), (31, 1203)])]
    scenes = long_track_windows[0] + short
    probs = long_track_windows[1] + [B.PackedProblem(sc.C, sc.P, sc.M, *sc.packed(), sc.anchor, sc.scale_view) for sc in short]
    recs, rep = B.batch_adjust(device, probs, iterations=5, shared_focal=shared, precision="mixed", max_cg=200,
                               schedule=schedule)
    assert rep["schedule"] == schedule - 1 and rep["form"] == _lib.TBA_PRECISION_MIXED
    against_single_calls(device, scenes, probs, recs, shared, MIXED_REL, MIXED_POSE_ABS)
