"""Guarded observation evaluations whose tracks are empty, as long as a warp, longer, or very long: the flags and
the error sum against the oracle's evaluation, and the structural checks of the tracks."""
import ctypes

import numpy as np
import pytest

import typecv_b200 as tb
from oracle import observations as OO
from typecv_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


def evaluation(C, tracks, seed=0):
    """A request of tracks of these lengths: cameras side by side, about one observation in five an outlier."""
    rng = np.random.default_rng(seed)
    P, M = len(tracks), int(sum(tracks))
    t = np.stack([np.linspace(-1, 1, C), 0.1 * rng.normal(size=C), np.zeros(C)], 1)
    X = np.stack([rng.normal(size=P), rng.normal(size=P), 8 + 4 * rng.random(P)], 1)
    camera, point = rng.integers(0, C, M), np.repeat(np.arange(P), tracks)
    q = X[point] + t[camera]
    pixels = 800 * q[:, :2] / q[:, 2:] + (512, 384) + rng.normal(scale=0.5, size=(M, 2)) + 40 * (rng.random((M, 1)) < 0.2)
    return dict(C=C, P=P, count=M, guarded=True, max_error=3.0, noise=1.0, limit=0.02,
                cameras=np.concatenate([np.tile(np.eye(3).ravel(), (C, 1)), t,
                                        np.tile([800.0, 800, 512, 384, 0, 0], (C, 1))], 1).ravel(),
                points=X.ravel(), pixels=pixels.ravel(), indices=np.stack([camera, point], 1).astype(np.uint32).ravel(),
                offsets=np.concatenate([[0], np.cumsum(tracks)]).astype(np.uint32))


def evaluate(device, q):
    lib = _lib.load()
    C, P, M = q["C"], q["P"], q["count"]
    ctl = _lib.ObservationControl(C, P, M, 0, q["max_error"], q["limit"], q["noise"])
    flags, summary, report = np.full(M + P, 7, np.uint32), np.zeros(2), _lib.ObservationReport()
    arrays = [q[k] for k in ("cameras", "points", "pixels")]
    words = [q[k] for k in ("indices", "offsets")]
    status = lib.tba_evaluate_observations(
        device.handle, ctypes.byref(ctl), *[x for a in arrays for x in (_lib.dptr(a), a.size)],
        *[x for a in words for x in (_lib.uptr(a), a.size)], _lib.uptr(flags), flags.size, _lib.dptr(summary),
        ctypes.byref(report))
    return status, lib.tba_last_error(device.handle).decode(), flags, summary, report


# A run of empty tracks of its own lies behind a track longer than a warp: in front, inside, at the end (behind
# the last observation), longer than a warp; others share a run with short tracks.
@pytest.mark.parametrize("tracks", [[2, 40, 0], [33, 0, 0, 0], [0, 0, 40, 0, 34, 5], [0, 3, 0, 4, 0], [40] + 70 * [0],
                                    [32, 0, 32, 0]])
def test_empty_tracks_take_no_part(device, tracks):
    q = evaluation(9, tracks)
    status, said, flags, summary, _ = evaluate(device, q)
    assert status == _lib.TBA_OK, said
    want = OO.evaluate_cpp(q)
    assert np.array_equal(flags, want["flags"]) and np.all(flags[q["count"]:][np.array(tracks) == 0] == 0)
    assert summary[1] == want["summary"][1] > 0 and abs(summary[0] - want["summary"][0]) <= 1e-12 * want["summary"][0]


def test_the_checks_of_a_long_track_cost_less_than_its_evaluation(device):
    q = evaluation(50, [200_000, 200_000])
    spent = []
    for _ in range(5):
        status, said, _, _, rep = evaluate(device, q)
        assert status == _lib.TBA_OK, said
        spent.append((rep.wall_ms - rep.evaluate_ms, rep.evaluate_ms))
    copies_and_checks, kernels = min(spent)
    assert copies_and_checks < 0.5 * kernels, spent


# Empty tracks, tracks of one, of a warp and of more, and long ones: a foreign observation at either end of a
# track or inside it, offsets that move a track's end, and indices just out of range.
@pytest.mark.parametrize("where,at,value,message", [
    (None, 0, 0, ""), ("indices", 1, 2, "offsets"), ("indices", 2 * 8000 + 1, 3, "offsets"),
    ("indices", 2 * 8999 + 1, 4, "offsets"), ("indices", -1, 3, "offsets"), ("indices", 1, 0, "offsets"),
    ("offsets", 6, 8999, "offsets"), ("offsets", 6, 9001, "offsets"), ("offsets", 3, 0, "offsets"),
    ("offsets", 4, 10_290, "offsets"), ("indices", 2 * 8000, 50, "out of range"), ("indices", -1, 8, "out of range")])
def test_track_checks_at_the_edges(device, where, at, value, message):
    q = evaluation(50, [0, 1, 0, 33, 257, 8709, 1289, 0])
    assert (q["count"], q["P"]) == (10_289, 8) and q["offsets"][6] == 9000
    if where:
        q[where][at] = value
        status, said, _, _, _ = evaluate(device, q)
        assert status == _lib.TBA_ERROR_ARGUMENT and message in said
        return
    status, said, flags, _, _ = evaluate(device, q)
    assert status == _lib.TBA_OK, said
    assert np.array_equal(flags, OO.evaluate_cpp(q)["flags"])
