"""GPU: the forward convolution of small and narrow images: rows cut into bands
that share a set of column groups (more than 296 rows and at most 8 groups), the
last band not full, bands of several images; and segments of two to six rows,
whose rows all lie at a segment's end, around the accumulator ring."""
import ctypes as C

import pytest

import tsuner_b200 as T

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
F = torch.nn.functional


def ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("n,h,w", [(1, 296, 8), (1, 297, 8), (1, 1000, 8), (1, 1001, 9), (2, 311, 30), (8, 300, 5),
                                   (1, 331, 64), (1, 331, 65), (3, 299, 17), (1, 4001, 24), (1, 1056, 48),
                                   (1, 48, 48), (1, 592, 128), (1, 888, 130), (1, 1480, 128), (1, 1777, 121)])
@pytest.mark.parametrize("gated", [False, True])
def test_small_and_narrow_images(n, h, w, gated):
    was, torch.backends.cudnn.allow_tf32 = torch.backends.cudnn.allow_tf32, False
    try:
        g = torch.Generator(device="cuda:0").manual_seed(1000 * h + w)
        X = torch.randn(n, h, w, 32, generator=g, device="cuda:0").to(torch.bfloat16)
        Wt = (0.1 * torch.randn(32, 32, 3, 3, generator=g, device="cuda:0")).to(torch.bfloat16)
        b = 0.1 * torch.randn(32, generator=g, device="cuda:0")
        gate = torch.randn(X.shape, generator=g, device="cuda:0").to(torch.bfloat16) if gated else None
        Wk = Wt.permute(0, 2, 3, 1).reshape(32, 9, 32).contiguous()
        ref = F.conv2d(X.float().permute(0, 3, 1, 2), Wt.float(), b, padding=1).permute(0, 2, 3, 1)
        if gated:
            ref = ref * (gate > 0)
        buf = torch.full((n * h * w * 32 + 8192,), 7.0, device="cuda:0")  # guard bands on both sides
        Y = buf[4096: 4096 + n * h * w * 32].view(n, h, w, 32)
        assert T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), ptr(b), 0, ptr(gate), None, ptr(Y), None) == 0
        assert T.lib().tsu_corr_status() == 0
        assert (buf[:4096] == 7.0).all() and (buf[4096 + n * h * w * 32:] == 7.0).all()
        # 288 products of 16-bit operands added in FP32: 2^-24 x 288 x the largest partial sum
        assert (Y - ref).abs().max() <= 288 * 2.0 ** -24 * 32 * ref.abs().max().clamp_min(1.0)
    finally:
        torch.backends.cudnn.allow_tf32 = was


def graph_us(n, h, w):
    X = torch.zeros(n, h, w, 32, device="cuda:0", dtype=torch.bfloat16)
    Wk = torch.zeros(32, 9, 32, device="cuda:0", dtype=torch.bfloat16)
    Y = torch.empty_like(X)
    g = torch.cuda.CUDAGraph()
    launch = lambda s: T.lib().tsu_corr_conv3x3(ptr(X), n, h, w, ptr(Wk), None, 0, None, ptr(Y), None, s)  # noqa: E731
    assert launch(None) == 0 and T.lib().tsu_corr_status() == 0
    with torch.cuda.graph(g):
        for _ in range(20):
            assert launch(C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    best = 1e9
    for _ in range(8):
        e[0].record()
        g.replay()
        e[1].record()
        torch.cuda.synchronize()
        best = min(best, e[0].elapsed_time(e[1]) / 20 * 1e3)
    return best


def test_a_narrow_image_takes_no_longer_than_its_pixels_side_by_side():
    """1000 rows of 8 pixels as one image and as eight of 125 rows: the same work
    for the same number of CTAs once the rows are cut into bands (one group of
    columns in sixteen before: 1.6 times)."""
    assert graph_us(1, 1000, 8) < 1.35 * graph_us(8, 125, 8)
