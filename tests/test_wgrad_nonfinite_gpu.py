"""GPU: the weight gradient of operands that hold infinities and NaN, against
its definition in 64 bits: sum over the pixels p of dZ[p] X[p + off], zeros
around X.  The zeros around dZ, which the kernel's tiles also hold, must not
meet an infinity in X."""
import ctypes as C

import pytest

import tsuner_b200 as T

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
F = torch.nn.functional


def gradient(X, dZ):
    dW = torch.zeros(32, 9, 32, device="cuda:0")
    db = torch.zeros(32, device="cuda:0")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    n, h, w, _ = X.shape
    assert T.lib().tsu_corr_conv3x3_wgrad(p(X), p(dZ), n, h, w, p(dW), p(db), None) == 0
    assert T.lib().tsu_corr_status() == 0
    return dW.cpu().double(), db.cpu().double()


def definition(X, dZ):
    n, h, w, _ = X.shape
    Xp = F.pad(X.cpu().double(), (0, 0, 1, 1, 1, 1))
    Z = dZ.cpu().double()
    out = torch.zeros(32, 9, 32, dtype=torch.float64)
    for tap in range(9):
        dy, dx = tap // 3, tap % 3
        V = Xp[:, dy:dy + h, dx:dx + w]
        for co in range(32):  # no product left out: inf * 0 is a NaN
            out[co, tap] = (Z[..., co, None] * V).sum((0, 1, 2))
    return out, Z.sum((0, 1, 2))


INF, NAN = float("inf"), float("nan")


# 16 x 32: whole tiles (8 columns x 16 rows); 17 x 13: cut by both borders
@pytest.mark.parametrize("n,h,w", [(2, 16, 32), (1, 17, 13), (3, 40, 24)])
@pytest.mark.parametrize("which", ["X", "dZ", "both"])
@pytest.mark.parametrize("value", [INF, -INF, NAN])
@pytest.mark.parametrize("at", ["west", "east", "north", "south", "corner", "inside", "none"])
def test_nonfinite_operands(n, h, w, which, value, at):
    g = torch.Generator(device="cuda:0").manual_seed(h * 100 + w)
    X = torch.randn(n, h, w, 32, generator=g, device="cuda:0").to(torch.bfloat16)
    dZ = torch.randn(n, h, w, 32, generator=g, device="cuda:0").to(torch.bfloat16)
    y, x = {"west": (h // 2, 0), "east": (h // 2, w - 1), "north": (h - 1, w // 2), "south": (0, w // 2),
            "corner": (0, w - 1), "inside": (h // 2, w // 2), "none": (0, 0)}[at]
    if at != "none":
        if which != "dZ":
            X[n - 1, y, x, 5] = value
        if which != "X":
            dZ[0, y, x, 7] = value
    dW, db = gradient(X, dZ)
    rW, rb = definition(X, dZ)
    for a, r in ((dW, rW), (db, rb)):
        assert torch.equal(torch.isnan(a), torch.isnan(r))
        assert torch.equal(torch.isinf(a), torch.isinf(r)) and torch.equal(a[torch.isinf(a)], r[torch.isinf(r)])
        ok = torch.isfinite(r)
        # products of 8-bit significands are exact in FP32, a sum of N of them
        # is off by at most N rounding errors of the running sum, here < 2^8 ulp
        assert (a[ok] - r[ok]).abs().max() < 1e-4 * (n * h * w) ** 0.5
