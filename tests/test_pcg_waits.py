"""The bounded waits between the blocks of a PCG on the explicit reduced system: with no polls left they run
out in every block, the call ends with an error, and the handle's next call is correct."""
import numpy as np
import pytest

import typecv_b200 as tb
from typecv_b200 import _lib
from typecv_b200 import adjoint as AD
from typecv_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def device():
    dev = tb.ShadeDevice.open(0)
    yield dev
    dev.close()


class NoPolls:
    def __init__(self, device):
        self.device = device

    def __enter__(self):
        assert _lib.load().tba_device_set_wait_limit(self.device.handle, 0) == _lib.TBA_OK

    def __exit__(self, *exc):
        assert _lib.load().tba_device_set_wait_limit(self.device.handle, _lib.TBA_WAIT_LIMIT_DEFAULT) == _lib.TBA_OK


# Over two blocks, and over as many as the device has, each with iterations issued ahead of the failing one.
@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("cameras,points", [(29, 401), (200, 9001)])
def test_a_solve_whose_waits_run_out(device, cameras, points, shared):
    sc = S.sphere_scene(seed=21, cameras=cameras, points=points)
    s, i = sc.packed()
    ctl = tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=6, shared_focal=shared)
    want, rep = tb.solve_packed(device, ctl, s, i)
    assert rep["engine"] == 2
    with NoPolls(device):
        with pytest.raises(tb.DeviceError, match="a wait between the PCG's blocks ran out"):
            tb.solve_packed(device, ctl, s, i)
    got, _ = tb.solve_packed(device, ctl, s, i)
    base = 12 * sc.C + 3 * sc.P
    assert abs(got[base + 6] - want[base + 6]) <= 1e-9 * want[base + 6] and got[base + 17] == want[base + 17]


def test_a_system_in_one_block_waits_for_nothing(device):
    sc = S.ring_scene(seed=4, cameras=25, points=333)
    s, i = sc.packed()
    ctl = tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=4)
    with NoPolls(device):
        out, rep = tb.solve_packed(device, ctl, s, i)
    assert rep["engine"] == 2 and out[12 * sc.C + 3 * sc.P + 10] > 0


def test_an_adjoint_whose_waits_run_out(device):
    sc = S.sphere_scene(seed=12, cameras=29, points=203, outlier_rate=0.0)
    s, i = sc.packed()
    out, _ = tb.solve_packed(device, tb.make_control(sc.C, sc.P, sc.M, anchor=0, scale_view=1, iterations=20,
                                                     max_cg=200, tolerance=1e-10), s, i)
    n = 12 * sc.C + 3 * sc.P
    s[:n] = out[:n]
    g = np.random.default_rng(13).normal(size=n)
    want, _, _, rep = AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, g)
    assert rep["failed"] == 0 and rep["product_blocks"] == 0
    with NoPolls(device):
        with pytest.raises(tb.DeviceError, match="a wait between the PCG's blocks ran out"):
            AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, g)
    got, _, _, rep = AD.bundle_vjp(device, sc.C, sc.P, sc.M, s, i, g)
    assert rep["failed"] == 0 and np.linalg.norm(got - want) <= 1e-8 * np.linalg.norm(want)
