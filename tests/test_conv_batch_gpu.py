"""GPU: the forward convolution of several images in one call equals the same
images one by one, value for value.  The split of the work differs (sets of 16
column groups across images, segments of rows per CTA, wraps of the accumulator
ring), the order in which an output adds its taps does not."""
import ctypes as C

import pytest

import tsuner_b200 as T

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def conv(X, Wk, b, gate, fp32):
    n, h, w, _ = X.shape
    Y = torch.empty(X.shape, device=X.device, dtype=torch.float32 if fp32 else torch.bfloat16)
    assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 0 if fp32 else 1, ptr(gate),
                                    None if fp32 else ptr(Y), ptr(Y) if fp32 else None, None) == 0
    assert T.lib().tsu_corr_status() == 0
    return Y


@pytest.mark.parametrize("n,h,w", [(2, 1, 9), (5, 37, 121), (3, 150, 129), (8, 64, 40), (4, 299, 8)])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("gated", [False, True])
def test_one_call_equals_image_by_image(n, h, w, fp32, gated):
    g = torch.Generator(device="cuda:0").manual_seed(100 * h + w)
    X = torch.randn(n, h, w, 32, generator=g, device="cuda:0").to(torch.bfloat16)
    Wk = (0.1 * torch.randn(32, 9, 32, generator=g, device="cuda:0")).to(torch.bfloat16)
    b = 0.1 * torch.randn(32, generator=g, device="cuda:0")
    gate = torch.randn(X.shape, generator=g, device="cuda:0").to(torch.bfloat16) if gated else None
    Y = conv(X, Wk, b, gate, fp32)
    assert Y.abs().max() > 0
    for k in range(n):
        assert torch.equal(Y[k:k + 1], conv(X[k:k + 1], Wk, b, None if gate is None else gate[k:k + 1], fp32)), k
