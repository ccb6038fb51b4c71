"""The O(M) checks of the batch on the grid kernels, the adjoint and the observation evaluation, which run
on the device from 8,192 observations: every corruption gets the message of the host's checks, the first of
several failures included, and the handle stays usable."""
import ctypes

import numpy as np
import pytest

import typecv_b200 as tb
from test_device_checks import KINDS, corrupt
from typecv_b200 import _lib
from typecv_b200 import adjoint as AD
from typecv_b200 import batch as B
from typecv_b200 import synthetic as S
from typecv_b200.resident import ResidentScene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


@pytest.fixture(scope="module")
def problem():
    sc = S.ring_scene(cameras=6, points=2000)
    assert sc.M >= 8192
    s, i = sc.packed()
    return sc, s, i


@pytest.mark.parametrize("kind", KINDS)
def test_the_host_checks_message(device, problem, kind):
    sc, s0, i0 = problem
    s, i = corrupt(sc, s0, i0, kind)
    with pytest.raises(tb.RangeError) as want:
        ResidentScene(device, tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=3), s, i)
    with pytest.raises(tb.RangeError) as got:
        AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, np.zeros(12 * sc.C + 3 * sc.P), tolerance=1e-6)
    assert str(got.value) == str(want.value)
    good = B.PackedProblem(sc.C, sc.P, sc.M, s0, i0, 0, 1)
    bad = B.PackedProblem(sc.C, sc.P, sc.M, s, i, 0, 1)
    later = B.PackedProblem(sc.C, sc.P, sc.M, *corrupt(sc, s0, i0, "scene_nan" if kind != "scene_nan" else "activity"), 0, 1)
    for schedule in (0, 5):
        with pytest.raises(tb.RangeError) as got:
            B.batch_adjust(device, [good, bad, later], iterations=2, schedule=schedule)
        assert str(got.value) == str(want.value)
        recs, _ = B.batch_adjust(device, [good, good], iterations=2, schedule=schedule)
        assert np.all(np.isfinite(recs[1]))


def evaluate(device, C, P, M, cameras, points, pixels, indices, offsets):
    lib = _lib.load()
    ctl = _lib.ObservationControl(C, P, M, 0, 3.0, 0.2, 1.0)
    flags, summary = np.zeros(M + P, np.uint32), np.zeros(2)
    status = lib.tba_evaluate_observations(device.handle, ctypes.byref(ctl), _lib.dptr(cameras), cameras.size,
                                           _lib.dptr(points), points.size, _lib.dptr(pixels), pixels.size,
                                           _lib.uptr(indices), indices.size, _lib.uptr(offsets), offsets.size,
                                           _lib.uptr(flags), flags.size, _lib.dptr(summary), None)
    return status, lib.tba_last_error(device.handle).decode(), summary


INDICES = "Invalid GPU observation indices: a camera or point out of range"
OFFSETS = "Invalid GPU observation arrays: track offsets"
BOUNDS = "Invalid GPU scene coordinate bounds"


@pytest.mark.parametrize("where,value,message", [
    ("indices", (8000, 6), INDICES), ("indices", (8001, 2000), INDICES), ("indices", (8001, 5), OFFSETS),
    ("offsets", (0, 1), OFFSETS), ("offsets", (2000, 5), OFFSETS), ("offsets", (77, 1 << 31), OFFSETS),
    ("offsets", (77, 0), OFFSETS), ("cameras", (107, np.nan), BOUNDS), ("points", (5999, 1e10), BOUNDS),
    ("pixels", (1, 1e-31), BOUNDS)])
def test_an_evaluation_out_of_order(device, problem, where, value, message):
    sc, _, _ = problem
    C, P, M = sc.C, sc.P, sc.M
    arrays = {"cameras": np.concatenate([np.asarray(sc.poses).reshape(C, 12), np.asarray(sc.cameras).reshape(C, 6)], 1).ravel(),
              "points": np.array(sc.points, dtype=np.float64).ravel(),
              "pixels": np.array(sc.pixels, dtype=np.float64).ravel(),
              "indices": np.stack([sc.obs_camera, sc.obs_point], 1).astype(np.uint32).ravel(),
              "offsets": np.concatenate([[0], np.cumsum(np.bincount(sc.obs_point, minlength=P))]).astype(np.uint32)}
    assert (C, P) == (6, 2000) and 2 * M > 8001
    status, _, first = evaluate(device, C, P, M, **arrays)
    assert status == _lib.TBA_OK
    bad = {k: v.copy() for k, v in arrays.items()}
    bad[where][value[0]] = value[1]
    status, said, _ = evaluate(device, C, P, M, **bad)
    assert status == _lib.TBA_ERROR_ARGUMENT and said == message
    status, _, again = evaluate(device, C, P, M, **arrays)
    assert status == _lib.TBA_OK and np.array_equal(first, again)
