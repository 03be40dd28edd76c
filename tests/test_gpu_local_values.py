"""Plan.local_values gives the last execute's values and writes no more of them
than its field count has, also where an earlier execute had more fields; what an
execute left behind ends with the target lists it was made for."""
import ctypes

import numpy as np
import pytest

import pacman_b200 as pacman

pytestmark = pytest.mark.gpu


def test_fewer_fields_than_before():
    rng = np.random.default_rng(0)
    S, T = rng.random((2000, 3)), rng.random((1500, 3))
    v = np.sin(S @ rng.random((3, 8)))
    plan, fresh = pacman.rbf.Plan(3, S, T), pacman.rbf.Plan(3, S, T)
    plan.execute(0x11, v)
    plan.execute(0x11, v[:, :2])
    fresh.execute(0x11, v[:, :2])
    want = fresh.local_values()
    buf = np.full(4 * want.size, 7.0)  # what the first execute's eight fields take
    assert plan._lib.pacman_b200_plan_local_values(
        plan._h, buf.ctypes.data_as(ctypes.c_void_p)) == 0
    assert np.array_equal(buf[:want.size], want.ravel())
    assert np.all(buf[want.size:] == 7.0)
    assert np.array_equal(plan.local_values(), want)


def test_nothing_is_left_of_an_execute_before_the_shard():
    rng = np.random.default_rng(1)
    S, T = rng.random((2000, 3)), rng.random((1500, 3))
    v = np.sin(S @ [3.0, 2.0, 1.0])
    plan = pacman.rbf.Plan(3, S, T)
    plan.execute(0x11, v, save_for_adjoint=True)
    plan.shard(0, 2)
    with pytest.raises((RuntimeError, ValueError)):
        plan.local_values()
    with pytest.raises((RuntimeError, ValueError)):
        plan.adjoint(np.ones(len(T)))
    out = plan.execute(0x11, v, save_for_adjoint=True)
    plan.local_values()
    gv, _ = plan.adjoint(out)
    assert np.isfinite(gv).all()
