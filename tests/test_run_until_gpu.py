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


def test_finished_members_skip_their_tiles():
    """A finished member is left before anything of its tiles is loaded.  Of a
    live step it keeps the launches and two dependent reads per tile: well
    below a quarter (24 members of 128^2 .. 1024^2: 158 of 750 us; loading the
    tiles first takes 278)."""
    ws = W.ensemble(nmembers=16, lo=256, hi=768, seed=5, t_series=200.0)
    e = T.Ensemble([w.p for w in ws], [w.sw for w in ws])
    try:
        e.load(ws)
        e.reset()
        e.step(32)
        live, past = [], []
        for _ in range(5):
            e.step(32)
            live.append(e.last_ms() / 32)
            e.run_until(0.0, 64)
            past.append(e.last_ms() / 64)
        assert min(past) < 0.25 * min(live), (past, live)
        before = [m.state() for m in e.members]
        e.run_until(0.0, 64)
        for V, m in zip(before, e.members):
            assert np.array_equal(V, m.state())
    finally:
        e.close()
