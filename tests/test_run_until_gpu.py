"""GPU: what run_until costs once the end time is reached."""
import numpy as np
import pytest

import tsuner_b200 as T
from tsuner_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_run_until_enqueues_no_more_steps_than_dt_needs(precision):
    """Every step of a grid loads its tiles before it can know that the end
    time has passed, so the last batch of a run holds the steps that the
    current dt needs and one more, and a run that is at its end already one."""
    w = W.hump(96, 64, 10.0, sigma=80.0)
    w.sw.precision = precision
    s = T.solver_for(w)
    try:
        s.step(40)
        t, dt, _ = s.time()
        n = s.run_until(t + 20.5 * dt)
        t1, _, steps = s.time()
        assert steps == 40 + n and t1 >= t + 20.5 * dt
        assert 20 <= n <= 23  # dt moves by a few per cent over 20 steps
        # at most 22 steps, then one or two more if dt fell
        assert s.last_launches() <= 2 * 22
        V = s.state()
        assert s.run_until(t1) == 0
        assert s.last_launches() == 2
        assert np.array_equal(V, s.state())
        assert s.run_until(t1 + 1e9, 5) == 5 and s.last_launches() == 10
    finally:
        s.close()


def members(dxs, n=256):
    """One hump per member; the coarser the grid, the larger its steps."""
    ws = []
    for k, dx in enumerate(dxs):
        w = W.hump(n, n, dx, sigma=20.0 * dx, seed=k)
        w.sw.precision = 1
        ws.append(w)
    return ws


def ensemble(ws):
    e = T.Ensemble([w.p for w in ws], [w.sw for w in ws])
    e.load(ws)
    e.reset()
    return e


def test_finished_members_leave_the_tile_list():
    """Steps of tsu_ens_run_until cost what the members that have not reached
    the end time cost: nothing when all have (the steps still count), and as
    much as an ensemble of the others when some have."""
    coarse, fine = [80.0] * 6, [10.0] * 2
    e, alone = ensemble(members(coarse + fine)), ensemble(members(fine))
    try:
        t_end = 64 * e.members[0].time()[1]  # the coarse ones end after about 64 steps, the fine ones after 500
        e.run_until(t_end, 128)
        assert all(m.time()[0] >= t_end for m in e.members[:6])
        assert all(m.time()[0] < 0.5 * t_end for m in e.members[6:])
        before = [m.state() for m in e.members]
        both, one = [], []
        for _ in range(5):
            assert e.run_until(t_end, 16) == 16
            both.append(e.last_ms())
            alone.step(16)
            one.append(alone.last_ms())
        assert min(both) < 1.3 * min(one), (both, one)
        for k, m in enumerate(e.members):
            assert np.array_equal(before[k], m.state()) == (k < 6)
        t = [m.time() for m in e.members]
        assert e.run_until(0.0, 100) == 64 and e.last_launches() == 0  # all have passed 0
        assert [m.time() for m in e.members] == t
    finally:
        e.close()
        alone.close()


@pytest.mark.parametrize("config", [None, (0, 0, 0), (8, 1, 0)])  # default, static stride, dynamic
def test_members_that_end_at_different_times_equal_members_alone(config):
    ws = members([10.0, 45.0, 20.0, 80.0, 30.0], n=96)
    e = ensemble(ws)
    try:
        if config:
            e.set_config(*config)
        t_end = 150 * e.members[3].time()[1]
        n = e.run_until(t_end)
        assert n % 64 == 0
        for w, m in zip(ws, e.members):
            s = T.solver_for(w)
            try:
                s.run_until(t_end)
                assert s.time() == m.time() and np.array_equal(s.state(), m.state())
            finally:
                s.close()
        e.step(1)  # the open end time and the whole list are back
        assert all(m.time()[0] > t_end for m in e.members)
    finally:
        e.close()
