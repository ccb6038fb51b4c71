"""The explicit reduced camera system (tba_schur.cu, tba_pcg.cu) where it can go wrong: systems that just
fit one block and just do not, tracks longer than a warp, a camera that sees a point twice, a rule that
keeps the product over stored factors, batched windows at odd places, and the adjoint's persistent PCG;
each against the oracle's operator, the one-call solve or the dense adjoint, at the parity bars of those
comparisons elsewhere in the tests."""
import numpy as np
import pytest

import typecv_b200 as tb
from typecv_b200 import _lib
from typecv_b200 import adjoint as AD
from typecv_b200 import batch as B
from typecv_b200 import synthetic as S
from typecv_b200.bundle import pack_arrays
from oracle import bundle_adjust as ob
from oracle.adjoint_dense import Problem

pytestmark = pytest.mark.gpu

COST_REL = 1e-9
POSE_ABS = 1e-7


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


def solve(device, C, P, M, s, i, flags=0, **kw):
    return tb.solve_packed(device, tb.make_control(C, P, M, anchor=0, scale_view=1, flags=flags, **kw), s, i)


def against_oracle(device, C, P, M, s, i, shared, iterations, engine, tolerance=1e-6):
    kw = dict(iterations=iterations, shared_focal=shared, max_cg=200, tolerance=tolerance)
    out, rep = solve(device, C, P, M, s, i, **kw)
    assert rep["engine"] == engine
    ref = ob.gpu_operator_packed({"C": C, "P": P, "M": M, "scene": s, "index": i}, 0, 1, iterations=iterations,
                                 huber=2.0, max_cg=200, shared=shared, tolerance=tolerance)
    b = 12 * C + 3 * P
    assert out[b + 10] == ref[b + 10] and out[b + 11] == ref[b + 11]
    assert abs(out[b + 6] - ref[b + 6]) <= COST_REL * ref[b + 6]
    assert np.max(np.abs(out[:12 * C] - ref[:12 * C])) < POSE_ABS
    # Steps launched one by one (the same system, its product as a kernel of its own).
    host, _ = solve(device, C, P, M, s, i, flags=_lib.TBA_FLAG_HOST_PCG_LOOP, **kw)
    assert abs(host[b + 6] - out[b + 6]) <= COST_REL * out[b + 6]
    return out


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("scene", [
    lambda: S.arc_scene(seed=3, cameras=2, points=41, track=(2, 2)),
    lambda: S.ring_scene(seed=4, cameras=25, points=333),   # the largest dense system of one block
    lambda: S.ring_scene(seed=5, cameras=27, points=301),   # the smallest of two
    lambda: S.helix_scene(seed=6, cameras=97, points=4003),
    lambda: S.sphere_scene(seed=7, cameras=331, points=9001),
    lambda: S.sphere_scene(seed=8, cameras=48, points=601, track=(30, 40), track_mean=36.0),  # beyond a warp
], ids=["pair", "one-block", "two-blocks", "helix", "sphere", "long-tracks"])
def test_explicit_system_matches_the_oracle(device, scene, shared):
    sc = scene()
    s, i = sc.packed()
    against_oracle(device, sc.C, sc.P, sc.M, s, i, shared, 5, engine=2)


@pytest.mark.parametrize("shared", [False, True])
def test_a_system_read_from_global_memory(device, shared):
    # Over 36 MB of S, 240 KB a block: the PCG's blocks cannot hold their shares, and read them 16 bytes at a
    # time.  (Fewer points would not be worth the system's steps.)
    sc = S.sphere_scene(seed=12, cameras=1301, points=180001)
    s, i = sc.packed()
    against_oracle(device, sc.C, sc.P, sc.M, s, i, shared, 4, engine=2, tolerance=1e-9)


def test_a_camera_that_sees_a_point_twice(device):
    sc = S.arc_scene(seed=9, cameras=9, points=257)
    rng = np.random.default_rng(1)
    twice = np.flatnonzero(rng.random(sc.M) < 0.2)
    at = np.sort(np.concatenate([np.arange(sc.M), twice]))
    pixels = sc.pixels[at] + rng.normal(scale=0.3, size=(at.size, 2))
    active = np.ones(sc.C, dtype=np.uint32)
    active[0] = 0
    s, i = pack_arrays(sc.poses, sc.points, sc.cameras, sc.obs_camera[at], sc.obs_point[at], pixels, active)
    against_oracle(device, sc.C, sc.P, at.size, s, i, True, 5, engine=2)


def test_every_camera_fixed_but_one(device):
    sc = S.arc_scene(seed=10, cameras=8, points=203)
    active = np.zeros(sc.C, dtype=np.uint32)
    active[5] = 1
    s, i = sc.packed(active)
    against_oracle(device, sc.C, sc.P, sc.M, s, i, False, 4, engine=2)


def test_dense_covisibility_keeps_the_product_over_factors(device):
    # Every one of 120 cameras sees every point: 59 pairs an observation.  (At the default PCG tolerance two
    # solves of this scene that differ in rounding alone stop 1e-7 apart, on the bar itself.)
    sc = S.ring_scene(seed=11, cameras=120, points=1500)
    s, i = sc.packed()
    against_oracle(device, sc.C, sc.P, sc.M, s, i, True, 2, engine=0, tolerance=1e-9)


@pytest.mark.parametrize("shared", [False, True])
def test_windows_at_odd_places(device, shared):
    # Scene lengths 18C + 3P + 2M with odd P put every later window at an odd 8-byte place.
    sizes = [(5, 301), (13, 777), (40, 1501), (2, 33), (27, 999), (31, 1203)]
    scenes = [S.arc_scene(seed=60 + k, cameras=c, points=p, track=(2, min(c, 10))) for k, (c, p) in enumerate(sizes)]
    probs = [B.PackedProblem(sc.C, sc.P, sc.M, *sc.packed(), sc.anchor, sc.scale_view) for sc in scenes]
    assert any(p.scene.size % 2 for p in probs)
    kw = dict(iterations=5, shared_focal=shared, max_cg=200)
    for schedule in (0, 5):
        recs, rep = B.batch_adjust(device, probs, precision="fp64", schedule=schedule, **kw)
        assert rep["schedule"] == 4 and rep["tune_ms"] == 0
        for sc, p, rec in zip(scenes, probs, recs):
            want, _ = solve(device, sc.C, sc.P, sc.M, p.scene, p.index, **kw)
            b = 12 * sc.C + 3 * sc.P
            assert rec[b + 10] == want[b + 10] and rec[b + 11] == want[b + 11]
            assert rec[b + 12] == want[b + 12] and rec[b + 15] == want[b + 15]  # of the last iteration that ran
            assert abs(rec[b + 6] - want[b + 6]) <= COST_REL * want[b + 6]
            assert np.max(np.abs(rec[:12 * sc.C] - want[:12 * sc.C])) < POSE_ABS


def test_adjoint_on_a_system_of_several_blocks(device):
    sc = S.sphere_scene(seed=12, cameras=29, points=203, outlier_rate=0.0)
    s, i = sc.packed()
    out, _ = solve(device, sc.C, sc.P, sc.M, s, i, iterations=20, max_cg=200, tolerance=1e-10)
    n = 12 * sc.C + 3 * sc.P
    s[:n] = out[:n]
    g = np.random.default_rng(13).normal(size=n)
    g /= np.linalg.norm(g)
    ybar, kbar, sol, rep = AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, g, newton_steps=3, want_solution=True)
    assert rep["failed"] == 0 and rep["adjoint_residual"] < 1e-10
    s[:n] = sol
    ybar_d, kbar_d = Problem(sc.C, sc.P, sc.M, s, i).vjp(g)
    assert np.linalg.norm(ybar - ybar_d) <= 1e-6 * np.linalg.norm(ybar_d)
    assert np.all(np.abs(kbar - kbar_d) <= 1e-6 * np.abs(kbar_d) + 1e-12)
