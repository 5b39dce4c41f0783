"""GPU: the corrector's convolution kernels at the sizes where their work
split can go wrong, against plain PyTorch FP32 convolutions of the same BF16
operands.  Forward: the last group of 8 columns not full, the last set of 16
groups not full, sets of several images, CTAs whose rows cross from one set to
the next, one to three output rows per CTA.  Weight gradient: one tile, tiles
cut by both borders, and more tiles per CTA than one, two and three batches of
accumulators hold."""
import ctypes as C

import pytest

import tsuner_b200 as T

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
F = torch.nn.functional


def ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def case(n, h, w, seed):
    g = torch.Generator(device="cuda:0").manual_seed(seed)
    X = torch.randn(n, h, w, 32, generator=g, device="cuda:0").to(torch.bfloat16)
    Wt = (0.1 * torch.randn(32, 32, 3, 3, generator=g, device="cuda:0")).to(torch.bfloat16)
    b = 0.1 * torch.randn(32, generator=g, device="cuda:0")
    return X, Wt, b


@pytest.fixture
def no_tf32():
    was = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = False
    yield
    torch.backends.cudnn.allow_tf32 = was


@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 2, 9), (3, 5, 7), (2, 3, 128), (5, 4, 121), (1, 700, 8), (7, 37, 40),
                                   (2, 149, 147), (1, 299, 129)])
def test_forward_work_split(n, h, w, no_tf32):
    X, Wt, b = case(n, h, w, 1000 * h + w)
    Wk = Wt.permute(0, 2, 3, 1).reshape(32, 9, 32).contiguous()
    ref = F.conv2d(X.float().permute(0, 3, 1, 2), Wt.float(), b, padding=1).permute(0, 2, 3, 1)
    # a guard band after the output must stay untouched
    buf = torch.full((n * h * w * 32 + 4096,), 7.0, device="cuda:0")
    Y = buf[: n * h * w * 32].view(n, h, w, 32)
    assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 0, None, None, ptr(Y), None) == 0
    assert T.lib().tsu_corr_status() == 0
    assert torch.allclose(Y, ref, rtol=1e-4, atol=1e-4 * float(ref.abs().max()))
    assert bool((buf[n * h * w * 32:] == 7.0).all())
    Yb = torch.empty(n, h, w, 32, device="cuda:0", dtype=torch.bfloat16)
    gate = torch.roll(X, 1, 3).contiguous()
    assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 0, ptr(gate), ptr(Yb), None, None) == 0
    assert T.lib().tsu_corr_status() == 0
    want = torch.where(gate > 0, ref, torch.zeros_like(ref))
    # one BF16 rounding of a value that is itself good to 1e-4
    assert torch.allclose(Yb.float(), want, rtol=2.0 ** -8 + 1e-4, atol=1e-4 * float(ref.abs().max()))


# 8 x 16 tiles: 1, 6, 148 x 6 + 1, 148 x 12, 148 x 24 + 1, 148 x 50 and 148 x 73 + 7 of them
@pytest.mark.parametrize("n,h,w", [(1, 3, 5), (1, 33, 12), (1, 16 * 7, 8 * 127), (1, 16 * 24, 8 * 74), (1, 16 * 19, 8 * 187), (2, 16 * 50, 8 * 74), (1, 16 * 83, 8 * 130 + 5)])
def test_weight_gradient_work_split(n, h, w, no_tf32):
    X, _, _ = case(n, h, w, 7 * h + w)
    dZ = torch.randn(n, h, w, 32, generator=torch.Generator(device="cuda:0").manual_seed(w), device="cuda:0")
    dZ = dZ.to(torch.bfloat16)
    dW, db = torch.zeros(32, 9, 32, device="cuda:0"), torch.zeros(32, device="cuda:0")
    assert T.lib().tsu_corr_conv3x3_wgrad(ptr(X), ptr(dZ), n, h, w, ptr(dW), ptr(db), None) == 0
    assert T.lib().tsu_corr_status() == 0
    Xp = F.pad(X.double(), (0, 0, 1, 1, 1, 1))
    z = dZ.double().reshape(-1, 32)
    ref = torch.stack([z.T @ Xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, 32) for t in range(9)], dim=1)
    assert float((dW - ref).norm() / ref.norm()) < 1e-4
    assert torch.allclose(dW.double(), ref, rtol=1e-4, atol=1e-4 * float(ref.abs().max()))
    assert torch.allclose(db.double(), z.sum(0), rtol=1e-4, atol=1e-4 * float(z.sum(0).abs().max()))


@pytest.mark.parametrize("off", [0, 8])  # elements of BF16: 0 and 16 bytes past a 32-byte boundary
def test_forward_output_and_gate_alignment(off):
    """The 32-byte and the 16-byte stores and gate loads give the same values."""
    n, h, w = 2, 21, 37
    X, Wt, b = case(n, h, w, 3)
    Wk = Wt.permute(0, 2, 3, 1).reshape(32, 9, 32).contiguous()
    size = n * h * w * 32
    gate0 = torch.roll(X, 3, 3).contiguous()

    def run(o):
        buf = torch.full((size + 64,), 3.0, device="cuda:0", dtype=torch.bfloat16)
        gb = torch.empty(size + 64, device="cuda:0", dtype=torch.bfloat16)
        gb[o:o + size] = gate0.reshape(-1)
        fb = torch.full((size + 64,), 3.0, device="cuda:0")
        Y, g, Yf = buf[o:o + size], gb[o:o + size], fb[o // 2:o // 2 + size]
        assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 1, ptr(g), ptr(Y), None, None) == 0
        assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 0, None, None, ptr(Yf), None) == 0
        assert T.lib().tsu_corr_status() == 0
        assert bool((buf[:o] == 3.0).all()) and bool((buf[o + size:] == 3.0).all())
        assert bool((fb[:o // 2] == 3.0).all()) and bool((fb[o // 2 + size:] == 3.0).all())
        return Y.clone(), Yf.clone()

    for a, c in zip(run(off), run(0)):
        assert torch.equal(a, c)
