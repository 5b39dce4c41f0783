"""GPU: both forms of the FP64 stage arithmetic (the branch-free one and the
general one it falls back to) and both tile shapes, against the oracle value
for value.  The states mix what separates them in one grid: dry land, films
around the velocity cutoff of 1e-6 m, speeds on both sides of the 7 m/s test
and of the 10 m/s clamp, still water, and momentum and load down to 1e-300."""
import numpy as np
import pytest

import oracle
import tsuner_b200 as T
from tsuner_b200 import workloads as W
from tsuner_b200.abi import make_switches

pytestmark = pytest.mark.gpu


def mixed_state(nx, ny, seed):
    """Patches of a few cells of each kind over a rough sloping bed."""
    r = np.random.default_rng(seed)
    w = W.hump(nx, ny, 10.0, seed=seed, sigma=0.2 * nx * 10.0)
    H = r.uniform(-1.0, 3.0, (ny, nx))
    kind = np.repeat(np.repeat(r.integers(0, 7, (ny // 3 + 1, nx // 3 + 1)), 3, 0), 3, 1)[:ny, :nx]
    h = np.maximum(H + r.uniform(-0.2, 0.4, (ny, nx)), 0.0)
    h = np.where(kind == 0, 0.0, h)
    h = np.where(kind == 1, 10.0 ** r.uniform(-7.5, -4.5, (ny, nx)), h)
    speed = np.where(kind == 2, r.uniform(6.0, 12.0, (ny, nx)), r.uniform(0.0, 1.0, (ny, nx)))
    speed = np.where(kind == 3, 0.0, speed)
    speed = np.where(kind == 4, 10.0 ** r.uniform(-300.0, -230.0, (ny, nx)), speed)
    th = r.uniform(0.0, 2.0 * np.pi, (ny, nx))
    load = np.where(kind == 5, 10.0 ** r.uniform(-300.0, -230.0, (ny, nx)), r.choice([0.0, 1e-3], (ny, nx)))
    w.V[0], w.V[3] = h, H
    w.V[1], w.V[2], w.V[4] = h * speed * np.cos(th), h * speed * np.sin(th), h * load
    w.mask = (r.uniform(size=(ny, nx)) > 0.2).astype(np.int32)
    return w


# sides around the 16 x 4 tile, the 32 x 8 tile and its halo; 545 x 171 is the
# smallest of these above the small-grid rule (18 x 22 = 396 tiles)
@pytest.mark.parametrize("nx,ny", [(1, 1), (15, 3), (16, 4), (17, 5), (20, 9), (36, 12), (37, 13), (97, 51), (545, 171)])
@pytest.mark.parametrize("wbc,order", [(1, 2), (2, 2), (0, 1)])
def test_mixed_states_equal_the_oracle(nx, ny, wbc, order):
    w = mixed_state(nx, ny, 100 * nx + ny)
    sw = make_switches(order=order, wbc=wbc, read_files=0)
    s = T.Solver(w.p, sw)
    try:
        s.set_state(w.V)
        s.set_mask(w.mask)
        s.reset()
        k = s.consts()
        s.step(4)
        V, (t, dt, _), ext = s.state(), s.time(), s.extrema()
    finally:
        s.close()
    o = oracle.OracleRun(w.p, sw, w.V, w.mask, None, None, kconsts=k)
    o.run(4)
    assert np.isfinite(V).all()
    for f in range(5):
        assert np.array_equal(V[f], o.V[f]), (f, np.abs(V[f] - o.V[f]).max())
    assert t == o.t.value and dt == o.dt.value
    for a, b in zip(ext, (o.hmax, o.bmin, o.eta_max)):
        assert np.array_equal(a.reshape(-1), np.asarray(b).reshape(-1))


@pytest.mark.parametrize("rk", [1, 0])
def test_periodic_seam_with_an_expired_series(rk):
    """The seam then mirrors the low side's discharge into the high side's
    face, with that face's depth and transverse discharge."""
    w = mixed_state(61, 29, 5)
    CC, tCC = W.expired_series(61, 29)
    sw = make_switches(order=2, wbc=2, read_files=1, rk=rk)
    s = T.Solver(w.p, sw)
    try:
        s.set_state(w.V)
        s.set_mask(w.mask)
        s.set_boundary_series(CC, tCC)
        s.reset()
        k = s.consts()
        s.step(3)
        V = s.state()
    finally:
        s.close()
    o = oracle.OracleRun(w.p, sw, w.V, w.mask, CC, tCC, kconsts=k)
    o.run(3)
    for f in range(5):
        assert np.array_equal(V[f], o.V[f]), (f, np.abs(V[f] - o.V[f]).max())


@pytest.mark.parametrize("nx,ny", [(37, 13), (545, 171)])
@pytest.mark.parametrize("order", [2, 1])
def test_grass_law_at_fronts_equals_the_oracle(nx, ny, order):
    """Grass's bed flux has no depth in it: water that moves below the bed of
    the dry cell beside it moves sediment, where every other flux is a zero."""
    w = mixed_state(nx, ny, nx + 7)
    w.mask = np.ones((ny, nx), dtype=np.int32)
    sw = make_switches(order=order, wbc=1, read_files=0, bedload_law=1, grass_ag=1e-3)
    s = T.Solver(w.p, sw)
    try:
        s.set_state(w.V)
        s.set_mask(w.mask)
        s.reset()
        k = s.consts()
        s.step(4)
        V = s.state()
    finally:
        s.close()
    o = oracle.OracleRun(w.p, sw, w.V, w.mask, None, None, kconsts=k)
    o.run(4)
    for f in range(5):
        assert np.array_equal(V[f], o.V[f]), (f, np.abs(V[f] - o.V[f]).max())
