"""Which form a call solves on, and what the explicit reduced system may cost a call that gains nothing by
it: the rule's two sides, a call without iterations, long tracks under the device's checks, and a device
whose memory is taken."""
import numpy as np
import pytest

import typecv_b200 as tb
from typecv_b200 import _lib
from typecv_b200 import synthetic as S

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
