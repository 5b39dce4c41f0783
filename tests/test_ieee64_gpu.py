"""GPU: the branch-free quotients and roots of csrc/ieee64.h with the device's
own seeds (tests/ieee64_device_check.cu), and the source terms' divisors
outside of the range that the branch-free form takes, against the oracle."""
import os
import subprocess

import numpy as np
import pytest

import oracle
import tsuner_b200 as T
from tsuner_b200 import build as B
from tsuner_b200 import workloads as W
from tsuner_b200.abi import make_switches

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_device_quotients_and_roots_are_correctly_rounded(tmp_path):
    exe = str(tmp_path / "ieee64_device_check")
    subprocess.run([B.NVCC] + B.ARCH + ["-O2", "-std=c++17", "-fmad=false", "-I" + B.CSRC,
                                        os.path.join(HERE, "ieee64_device_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("nx,ny", [(48, 40), (640, 200)])  # both tiles
@pytest.mark.parametrize("eps_h", [0.0, -0.5, -1e300, 1e300, np.inf])
def test_any_wet_threshold_equals_the_oracle(nx, ny, eps_h):
    w = W.hump(nx, ny, 10.0, sigma=100.0)
    w.p.epsilon_h = eps_h
    x = np.arange(nx)[None, :]
    w.V[0] = 0.5 + 0.25 * (x % 3) + 0.0 * w.V[0]  # a third of the cells: h + eps_h = 0 for -0.5
    w.V[1] = 0.4 * w.V[0]
    w.V[4] = 1e-3 * w.V[0]
    sw = make_switches(order=2, wbc=1, read_files=0)
    s = T.Solver(w.p, sw)
    try:
        s.set_state(w.V)
        s.set_mask(w.mask)
        s.reset()
        k = s.consts()
        s.step(2)
        V = s.state()
    finally:
        s.close()
    o = oracle.OracleRun(w.p, sw, w.V, w.mask, None, None, kconsts=k)
    o.run(2)
    assert np.array_equal(V, o.V, equal_nan=True)
