"""GPU: the FP32 form's tiles that load their cells with ordinary instructions
(boundary tiles, every tile of a periodic or a small grid, all with
TSU_STAGE_TMA=0): the tile shapes, whose threads load one to three cells each,
give the same values."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import sys, numpy as np
import tsuner_b200 as T
from tsuner_b200 import workloads as W
w = W.hump(%d, %d, 10.0, sigma=80.0)
w.sw.precision, w.sw.wbc, w.sw.order = 1, %d, %d
s = T.solver_for(w)
s.step(20)
np.savez(sys.argv[1], V=s.state(), t=np.array(s.time()))
s.close()
"""


@pytest.mark.parametrize("nx,ny,wbc,order", [(70, 45, 2, 2), (131, 67, 1, 1)])
def test_every_tile_shape_loads_the_same_cells(nx, ny, wbc, order, tmp_path):
    out = []
    for tile in (None, 1, 3, 7):  # 32 x 8, 16 x 16, 64 x 4, 32 x 16
        for tma in ("1", "0") if tile is None else ("1",):
            env = dict(os.environ, TSU_STAGE_TMA=tma)
            env.pop("TSU_TILE32", None)
            if tile is not None:
                env["TSU_TILE32"] = str(tile)
            path = str(tmp_path / ("%s_%s.npz" % (tile, tma)))
            r = subprocess.run([sys.executable, "-c", RUN % (nx, ny, wbc, order), path], env=env, capture_output=True,
                               text=True, timeout=120, cwd=ROOT)
            assert r.returncode == 0, r.stderr[-2000:]
            out.append((tile, tma, np.load(path)))
    for tile, tma, r in out[1:]:
        assert np.array_equal(r["V"], out[0][2]["V"]) and np.array_equal(r["t"], out[0][2]["t"]), (tile, tma)
