"""GPU: a tile that holds a cell out of the range of the branch-free slope
limiter (2^100 and beyond) is reconstructed by the general form, so that what
overflows there spreads as in the oracle: the new state is equal value for
value, NaN for NaN."""
import numpy as np
import pytest

import oracle
import tsuner_b200 as T
from tsuner_b200 import workloads as W
from tsuner_b200.abi import make_switches

pytestmark = pytest.mark.gpu


# (plane, value) of the odd cell: a depth whose slopes overflow in the limiter,
# one that does not, the first beyond the range and the last inside it; a load
# and a discharge of the same kind
CELLS = [(0, 1e308), (0, 1e200), (0, 2.0 ** 100), (0, np.nextafter(2.0 ** 100, 0.0)), (4, 1e308), (4, -1e308),
         (4, 2.0 ** 103), (1, 1e308)]


# 48 x 40: 16 x 4 tiles; 640 x 200: 32 x 8 tiles (500 of them)
@pytest.mark.parametrize("nx,ny", [(48, 40), (640, 200)])
@pytest.mark.parametrize("plane,value", CELLS)
def test_overflowing_slopes_equal_the_oracle(nx, ny, plane, value):
    w = W.hump(nx, ny, 10.0, sigma=100.0)
    x = np.arange(nx)[None, :]
    w.V[0] = 40.0 - 3.0 * np.abs((x % 12) - 6.0) + 0.01 * np.arange(ny)[:, None]  # slopes of both signs
    w.V[3] = w.V[0]
    w.V[1] = 0.3 * w.V[0]
    w.V[4] = 1e-4 * w.V[0] * (1 + x % 5)
    for i, j in ((9, 7), (nx - 11, ny - 9), (nx // 2, ny // 2)):  # on a falling, a rising and any side
        w.V[plane, j, i] = value
    sw = make_switches(order=2, wbc=1, read_files=0)
    s = T.Solver(w.p, sw)
    try:
        s.set_state(w.V)
        s.set_mask(w.mask)
        s.reset()
        k = s.consts()
        s.step(1)
        V = s.state()  # the step itself; the status word is not looked at
    finally:
        s.close()
    o = oracle.OracleRun(w.p, sw, w.V, w.mask, None, None, kconsts=k)
    o.run(1)
    assert np.array_equal(V, o.V, equal_nan=True), np.argwhere(~((V == o.V) | (np.isnan(V) & np.isnan(o.V))))[:10]
