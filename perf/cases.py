"""The work a user has this framework do, as cases that can be timed.

Three families, each through the public Python binding of the C ABI:
  * the time step (`Solver.step`) in the FP64 plain form and the FP32
    precision form, from the golden-fixture grids (a few thousand cells) to
    8192 x 8192, with the boundary kinds, orders and bedload laws the switches
    offer; a whole run through host buffers; and the batched ensemble;
  * the corrector's convolution and weight-gradient kernels on caller-owned
    device buffers;
  * the corrector's training step and prediction.

Inputs are seeded and made on the GPU.  The coast is the repository's own
synthetic one: a 1:50 shelf rising to the east with a fractal (k^-3) bed,
about 20 % dry land, three non-erodible harbour blocks.  "nwave" starts from
still water and is driven by an N-wave through the boundary series; "humps"
starts from Gaussian humps over a smooth current with some suspended load, so
that nearly every wet cell moves; "hump" is the single hump over a noisy slope.
"""
import ctypes as C
import math

import numpy as np
import torch
import torch.nn.functional as F

import tsuner_b200 as T
from tsuner_b200 import corrector as K
from tsuner_b200 import workloads as W
from tsuner_b200.abi import make_params, make_switches

DEV = "cuda:0"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a whole short run on a grid the size of the golden fixtures: upload,
        # reset, 64 steps; latency and launches are all that counts
        dict(name="fp64_run_48x36", kind="step", nx=48, ny=36, dx=40.0, source="humps", precision=0, steps=64,
             restart=True),
        # configuration 1: the 512^2 hump with walls, a chunk of its 2000 steps
        dict(name="fp64_hump_512", kind="step", nx=512, ny=512, dx=10.0, source="hump", precision=0, steps=16),
        # a mid-size coast with odd sides: boundary series, mask, FP64
        dict(name="fp64_nwave_1021x773", kind="step", nx=1021, ny=773, dx=10.0, source="nwave_moving", precision=0,
             steps=4),
        # configuration 2, the headline workload, in the FP64 plain form
        dict(name="fp64_nwave_4096", kind="step", nx=4096, ny=4096, dx=5.0, source="nwave", precision=0, steps=2),
        # the FP32 form on a mid-size coast with odd sides
        dict(name="fp32_nwave_1501x997", kind="step", nx=1501, ny=997, dx=10.0, source="nwave_moving", precision=1,
             steps=8),
        # configuration 3: 8192^2 humps, the largest grid the repository runs
        dict(name="fp32_humps_8192", kind="step", nx=8192, ny=8192, dx=5.0, source="humps", precision=1, steps=2),
        # a user's whole FP32 run through host buffers: upload of state, mask
        # and series, reset, 200 steps, read-back of state and extrema
        dict(name="fp32_host_run_1024", kind="host_run", nx=1024, ny=1024, dx=5.0, source="nwave_moving", precision=1,
             steps=200),
        # configuration 4, fewer members: uneven FP32 grids stepped together
        # with the schedule tsu_ens_create chooses, as the corrector's data
        # generation steps its sources
        dict(name="ensemble_24_128_1024", kind="ensemble", members=24, lo=128, hi=1024, dx=5.0, steps=4),
        # one hidden layer of the corrector over a training batch (8 images of
        # 512^2 padded by 8): convolution, bias, ReLU, BF16 output
        dict(name="conv_relu_8x528", kind="conv", n=8, h=528, w=528, gate=False, fp32_out=False),
        # the same layer's weight and bias gradient
        dict(name="wgrad_8x528", kind="wgrad", n=8, h=528, w=528),
        # two Adam iterations of the corrector at its default size
        dict(name="train_512_b8", kind="train", n=512, factor=4, samples=12, batch=8, iters=2),
        # two fine maps from coarse ones, read back to the host
        dict(name="predict_1024_x2", kind="predict", n=1024, factor=4, samples=2),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step", "ensemble", "conv", "wgrad", "train", "predict",
                       "host_run"])
    if kind == "step":
        prec = rng.choice([0, 1])
        nx, ny = _logint(rng, 40, 4000), _logint(rng, 30, 4000)
        cells = nx * ny
        # both forms from a step or two of a large grid to a chunk of a small one
        steps = 2 * max(1, min(16, int(8e6 // cells)))
        source = rng.choice(["nwave", "nwave_moving", "nwave_moving", "humps", "humps", "hump"])
        c = dict(kind=kind, nx=nx, ny=ny, dx=rng.choice([5.0, 10.0, 20.0, 40.0]), source=source, precision=prec,
                 steps=steps, restart=cells < 20000)
        if not source.startswith("nwave"):
            c["wbc"] = rng.choice([0, 1, 1, 2])
            c["order"] = rng.choice([1, 2, 2, 2, 2])
            c["bedload_law"] = rng.choice([0, 0, 1])
        return c
    if kind == "host_run":
        return dict(kind=kind, nx=_logint(rng, 100, 1400), ny=_logint(rng, 100, 1400), dx=5.0, source="nwave_moving",
                    precision=rng.choice([0, 1]), steps=rng.choice([20, 50, 100]))
    if kind == "ensemble":
        lo = _logint(rng, 40, 200)
        return dict(kind=kind, members=rng.randint(3, 24), lo=lo, hi=_logint(rng, lo + 1, 1024), dx=5.0,
                    steps=rng.choice([4, 8, 16]))
    if kind in ("conv", "wgrad"):
        c = dict(kind=kind, n=rng.randint(1, 8), h=_logint(rng, 48, 1056), w=_logint(rng, 48, 1056))
        c["n"] = max(1, min(c["n"], 4 * 528 * 528 * 8 // (c["h"] * c["w"] * 4)))
        if kind == "conv":
            c["gate"] = rng.choice([False, False, True])
            c["fp32_out"] = rng.choice([False, False, True])
        return c
    f = rng.choice([2, 4])
    n = f * _logint(rng, 32, 512 // f)
    if kind == "train":
        return dict(kind=kind, n=n, factor=f, samples=rng.randint(4, 12), batch=rng.randint(1, 8), iters=2)
    return dict(kind=kind, n=f * _logint(rng, 32, 1024 // f), factor=f, samples=rng.randint(1, 2))


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + salt)


def _field(ny, nx, g, slope=-3.0):
    """Gaussian random field with power spectrum ~ k^slope, unit deviation."""
    kx = torch.fft.rfftfreq(nx, device=DEV, dtype=torch.float64)[None, :]
    ky = torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)[:, None]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** (slope / 2.0)
    amp[0, 0] = 0.0
    spec = torch.randn(ny, nx // 2 + 1, 2, generator=g, device=DEV, dtype=torch.float64)
    f = torch.fft.irfft2(torch.view_as_complex(spec) * amp, s=(ny, nx))
    return f / f.std()


def _coast(case, seed):
    """V[5][ny][nx] float64 (h, qx, qy, H, hc), mask, (CC, tCC) or None, slr."""
    nx, ny, dx, src = case["nx"], case["ny"], case["dx"], case["source"]
    g = _gen(seed)
    r = np.random.default_rng(int(seed))
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5)[None, :] * dx
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5)[:, None] * dx
    V = torch.zeros(5, ny, nx, device=DEV, dtype=torch.float64)
    if src == "hump":
        zb = -50.0 + 0.02 * x + 0.1 * torch.randn(ny, nx, generator=g, device=DEV, dtype=torch.float64)
        s2 = (0.1 * nx * dx) ** 2
        eta = 2.0 * torch.exp(-((x - 0.5 * nx * dx) ** 2 + (y - 0.5 * ny * dx) ** 2) / (2.0 * s2))
        V[0], V[3] = (eta - zb).clamp_min(0.0), -zb
        return V, torch.ones(ny, nx, device=DEV, dtype=torch.int32), None, 0.0
    slr = 0.5
    z = x / 50.0 + 1.5 * _field(ny, nx, g)
    z -= torch.sort(z[:: max(1, ny // 64)].reshape(-1)).values[int(0.8 * z[:: max(1, ny // 64)].numel())].item()
    H = -(z + slr)
    mask = torch.ones(ny, nx, device=DEV, dtype=torch.int32)
    for _ in range(3):
        w, hg = int(r.integers(max(1, nx // 20), max(2, nx // 8))), int(r.integers(max(1, ny // 20), max(2, ny // 8)))
        i0, j0 = int(r.integers(nx // 3, max(nx // 3 + 1, nx - w))), int(r.integers(0, max(1, ny - hg)))
        mask[j0:j0 + hg, i0:i0 + w] = 0
    eta = torch.full((ny, nx), slr, device=DEV, dtype=torch.float64)
    if src != "nwave":
        for _ in range(8):
            a, s = r.uniform(0.5, 4.0), r.uniform(0.02, 0.2) * min(nx, ny) * dx
            xc, yc = r.uniform(0.1, 0.6) * nx * dx, r.uniform(0.1, 0.9) * ny * dx
            eta += a * torch.exp(-((x - xc) ** 2 + (y - yc) ** 2) / (2.0 * s * s))
    V[0] = (eta + H).clamp_min(0.0)
    V[3] = H
    if src != "nwave":
        V[1] = V[0] * (0.3 * _field(ny, nx, g, -4.0))
        V[2] = V[0] * (0.3 * _field(ny, nx, g, -4.0))
        V[4] = V[0] * 1e-4 * (1.0 + torch.tanh(_field(ny, nx, g, -4.0)))
    series = None
    if src.startswith("nwave"):
        series = W.boundary_series(H.cpu().numpy(), slr, 600.0, amp=r.uniform(1.0, 5.0), period=r.uniform(200.0, 600.0))
    return V, mask, series, slr


def _switches(case, series, slr):
    return make_switches(order=case.get("order", 2), wbc=case.get("wbc", 1), read_files=0 if series is None else 1,
                         bedload_law=case.get("bedload_law", 0), precision=case["precision"], eta0=slr)


class _Raw:
    """Device memory the library owns, for torch.as_tensor (no copy); keeps its owner alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, strides=strides, typestr=typestr, version=3)


def _planes(s, owner=None):
    """The solver's current state as a tensor [5][npy][npx] on its own buffer."""
    ptr, pitch, plane, eb = s.device_state()
    raw = _Raw(owner or s, ptr, (5, s.p.npy, s.p.npx), (plane * eb, pitch * eb, eb), "<f%d" % eb)
    return torch.as_tensor(raw, device=DEV)


def _load(s, V, mask, series):
    s.set_state(V)
    s.set_mask(mask)
    if series is not None:
        s.set_boundary_series(*series)


def _member_cases(case):
    """Sides spaced evenly over their logarithm: the quantiles of config 4's draw."""
    m, lo, hi = case["members"], case["lo"], case["hi"]
    return [dict(nx=n, ny=n, dx=case["dx"], source="nwave_moving", precision=1)
            for n in (int(lo * (hi / lo) ** ((k + 0.5) / m)) for k in range(m))]


def _conv_inputs(case, seed):
    g = _gen(seed)
    n, h, w = case["n"], case["h"], case["w"]
    X = torch.relu(torch.randn(n, h, w, 32, generator=g, device=DEV)).to(torch.bfloat16)
    Wk = (torch.randn(32, 9, 32, generator=g, device=DEV) * (2.0 / 288) ** 0.5).to(torch.bfloat16)
    b = 0.1 * torch.randn(32, generator=g, device=DEV)
    gate = torch.relu(torch.randn(n, h, w, 32, generator=g, device=DEV)).to(torch.bfloat16) if case.get("gate") else None
    return X, Wk, b, gate


def _wgrad_inputs(case, seed):
    X, _, _, _ = _conv_inputs(case, seed)
    dZ = (1e-3 * torch.randn(X.shape, generator=_gen(seed, 1), device=DEV)).to(torch.bfloat16)
    return X, dZ


def _corr_inputs(case, seed):
    """Weights of a trained network's size, a site, coarse maps and fine ones."""
    n, f, ns = case["n"], case["factor"], case["samples"]
    g = _gen(seed)
    Wt = torch.randn(6, 32, 9, 32, generator=g, device=DEV) * (2.0 / 288) ** 0.5
    Wt[5] *= 0.3
    B = 0.02 * torch.randn(6, 32, generator=g, device=DEV)
    x = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5)[None, :]
    z = x * (10.0 / 50.0) * (512.0 / n) + 1.5 * _field(n, n, g)
    H = -(z - torch.sort(z.reshape(-1)).values[int(0.8 * z.numel())].item() + 0.5)
    hm = torch.stack([(0.5 + torch.relu(1.5 + _field(n, n, g)) + H).clamp_min(0.0) for _ in range(ns)])
    db = torch.stack([0.05 * _field(n, n, g) * (hm[k] > 0) for k in range(ns)])
    pool = lambda a: F.avg_pool2d(a.reshape(-1, 1, n, n), f).reshape(-1, n // f, n // f)  # noqa: E731
    coarse = torch.stack([pool(hm), pool(db), pool(H[None]).expand(ns, -1, -1)], dim=1)
    return [t.float().cpu().numpy() for t in (Wt, B, H, coarse, torch.stack([hm, db], dim=1))]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "host_run"):
        V, mask, series, slr = _coast(case, seed)
        V, mask = V.cpu().numpy(), mask.cpu().numpy()
        p = make_params(case["nx"], case["ny"], case["dx"], case["dx"])
        s = T.Solver(p, _switches(case, series, slr))
        if kind == "host_run":
            return dict(case=case, s=s, V=V, mask=mask, series=series)
        _load(s, V, mask, series)
        s.reset()
        return dict(case=case, s=s, V=V if case.get("restart") else None, out=_planes(s))
    if kind == "ensemble":
        cs = _member_cases(case)
        ins = [_coast(c, int(seed) * 64 + k) for k, c in enumerate(cs)]
        e = T.Ensemble([make_params(c["nx"], c["ny"], c["dx"], c["dx"]) for c in cs],
                       [_switches(c, i[2], i[3]) for c, i in zip(cs, ins)])
        for m, (V, mask, series, _) in zip(e.members, ins):
            _load(m, V.cpu().numpy(), mask.cpu().numpy(), series)
        e.reset()
        return dict(case=case, e=e, out=[_planes(m, e) for m in e.members])
    if kind == "conv":
        X, Wk, b, gate = _conv_inputs(case, seed)
        Y = torch.empty(X.shape, device=DEV, dtype=torch.float32 if case["fp32_out"] else torch.bfloat16)
        return dict(case=case, X=X, Wk=Wk, b=b, gate=gate, Y=Y)
    if kind == "wgrad":
        X, dZ = _wgrad_inputs(case, seed)
        return dict(case=case, X=X, dZ=dZ)
    Wt, B, H, coarse, fine = _corr_inputs(case, seed)
    c = K.Corrector(case["n"], case["n"], case["factor"], max_batch=case.get("batch", 8))
    c.set_weights(Wt, B)
    c.set_site(H)
    c.add_samples(coarse, fine)
    return dict(case=case, c=c, W=Wt, B=B)


# ------------------------------------------------------------------ one pass
def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "step":
        s = state["s"]
        if state["V"] is not None:  # a short run from its start
            s.set_state(state["V"])
            s.reset()
        s.step(case["steps"])
        return state["out"]
    if kind == "host_run":
        s = state["s"]
        _load(s, state["V"], state["mask"], state["series"])
        s.reset()
        s.step(case["steps"])
        return dict(V=s.state(), extrema=s.extrema(), t=s.time()[0])
    if kind == "ensemble":
        state["e"].step(case["steps"])
        return state["out"]
    if kind == "conv":
        X, Y = state["X"], state["Y"]
        n, h, w, _ = X.shape
        yb, yf = (None, Y) if case["fp32_out"] else (Y, None)
        K._ck(T.lib().tsu_corr_conv3x3(_ptr(X), n, h, w, _ptr(state["Wk"]), _ptr(state["b"]), 0 if case["gate"] else 1,
                                       _ptr(state["gate"]), _ptr(yb), _ptr(yf),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)), "tsu_corr_conv3x3")
        return Y
    if kind == "wgrad":
        X, dZ = state["X"], state["dZ"]
        n, h, w, _ = X.shape
        dW, db = torch.zeros(32, 9, 32, device=DEV), torch.zeros(32, device=DEV)
        K._ck(T.lib().tsu_corr_conv3x3_wgrad(_ptr(X), _ptr(dZ), n, h, w, _ptr(dW), _ptr(db),
                                             C.c_void_p(torch.cuda.current_stream().cuda_stream)),
              "tsu_corr_conv3x3_wgrad")
        return dW, db
    c = state["c"]
    if kind == "train":  # from the same weights each time: set_weights also restarts Adam
        c.set_weights(state["W"], state["B"])
        loss = c.train(case["samples"], case["iters"], case["batch"], lr=1e-3, seed=3)
        return (loss,) + c.weights()
    return c.predict(0, case["samples"])


# ------------------------------------------------------------------ the work
def work(case):
    kind = case["kind"]
    if kind in ("step", "host_run", "ensemble"):
        if kind == "ensemble":
            cells, order = sum(c["nx"] * c["ny"] for c in _member_cases(case)), 2
        else:
            cells, order = case["nx"] * case["ny"], case.get("order", 2)
        fp32 = kind == "ensemble" or case["precision"] == 1
        e = 4 if fp32 else 8
        # the state read and written (order 2: U^n, U*, U^n and U^n again),
        # the mask per stage, the extrema
        per = (5 * e * 5 + 2 if order == 2 else 5 * e * 2 + 1) + 3 * 2 * e
        # rough count of the scheme's arithmetic per cell and stage
        b, f = per * cells * case["steps"], 700.0 * order * cells * case["steps"]
        if kind == "host_run" or case.get("restart"):
            b += cells * 40
        if kind == "host_run":
            b += cells * (40 + 24 + 4)
        return dict(bytes=b, flops=f)
    if kind == "conv":
        px = case["n"] * case["h"] * case["w"]
        return dict(bytes=px * (64 + (128 if case["fp32_out"] else 64) + (64 if case["gate"] else 0)) + 18560,
                    flops=2.0 * px * 288 * 32)
    if kind == "wgrad":
        px = case["n"] * case["h"] * case["w"]
        return dict(bytes=px * 128 + 4 * 9248, flops=2.0 * px * 288 * 32)
    px = (case["n"] + 16) ** 2
    if kind == "train":
        nb = case["iters"] * case["batch"]
        # features, 5 hidden layers written and read twice (forward,
        # backward), 5 input gradients written and read twice
        return dict(bytes=nb * px * 64.0 * (1 + 5 * 3 + 5 * 2), flops=nb * px * 2.0 * 288 * 32 * 17)
    return dict(bytes=case["samples"] * px * (64.0 * (1 + 5 * 2) + 16), flops=case["samples"] * px * 2.0 * 288 * 32 * 6)


# ------------------------------------------------------------------ in 64 bits
EPS = np.finfo(np.float64).eps
G = 9.81


def _velocity(h, qx, qy):
    d, wet = h + EPS, (h >= 1e-6).double()
    u, v = qx / d * wet, qy / d * wet
    m = torch.sqrt(u * u + v * v)
    s = torch.where(m > 10.0, 10.0 / m.clamp_min(1e-300), torch.ones_like(m))
    return u * s, v * s, m.clamp_max(10.0)


def _limit(a, b):
    num, den = a * b.abs() + b * a.abs(), a.abs() + b.abs()
    return torch.where(den > EPS, num / den.clamp_min(1e-300), torch.zeros_like(den))


def _sgn(x):
    return torch.where(x.abs() < EPS, torch.zeros_like(x), torch.sign(x))


def _filter(h, qx, qy, H, hc):
    h = h.clamp_min(0.0)
    c = (hc / (h + EPS)).clamp_min(0.0)
    u, v, _ = _velocity(h, qx, qy)
    return h, h * u, h * v, H, h * c


def _bedload(P, sw, h, u, m):
    if sw.bedload_law == 1:
        return -(sw.grass_ag * u * m * m) / (1.0 - P.porosity)
    O = P.Opar * m * m
    qb = 17.0 * u / (m + EPS) * P.Q * (O - P.OC).clamp_min(0.0) * (O.sqrt() - P.OC ** 0.5).clamp_min(0.0)
    return -(qb * ((h > P.HQB) & (h > 5.0 * P.DS)))


def _flux(P, sw, a, b, fixed):
    """Fluctuations into a and b of an edge, states (h, qn, qt, H, hc) in its frame."""
    ua, va, ma = _velocity(a[0], a[1], a[2])
    ub, vb, mb = _velocity(b[0], b[1], b[2])
    zm = torch.minimum(a[3], b[3])
    ha, hb = (a[0] - a[3] + zm).clamp_min(0.0), (b[0] - b[3] + zm).clamp_min(0.0)
    ca, cb = ha * (a[4] / (a[0] + EPS)), hb * (b[4] / (b[0] + EPS))
    on = fixed.double() * float(sw.bedload)
    Fa = (ha * ua, ha * ua * ua, ha * ua * va, _bedload(P, sw, ha, ua, ma) * on, ca * ua)
    Fb = (hb * ub, hb * ub * ub, hb * ub * vb, _bedload(P, sw, hb, ub, mb) * on, cb * ub)
    sa, sb, hm = ha.sqrt(), hb.sqrt(), 0.5 * (ha + hb)
    um = torch.where(sa + sb > 0, (sa * ua + sb * ub) / (sa + sb).clamp_min(1e-300), torch.full_like(sa, float("nan")))
    cm = torch.sqrt(G * hm)
    SL, SR = torch.fmin(ua - torch.sqrt(G * ha), um - cm), torch.fmax(ub + torch.sqrt(G * hb), um + cm)
    dS = SR - SL
    ok = dS > EPS
    dS = torch.where(ok, dS, torch.ones_like(dS))
    a0 = torch.where(ok, (SR * SL.abs() - SL * SR.abs()) / dS, torch.maximum(SL.abs(), SR.abs()))
    a1 = torch.where(ok, (SR.abs() - SL.abs()) / dS, torch.zeros_like(dS))
    df = [y - x for x, y in zip(Fa, Fb)]
    df[1] = df[1] + G * hm * (hb - ha)
    dU = (hb - ha, ub * hb - ua * ha, vb * hb - va * ha, b[3] - a[3], cb - ca)
    vis = [a0 * u + a1 * f for u, f in zip(dU, df)]
    vis[3] = torch.where(_sgn(a1) == _sgn(df[3]) * _sgn(dU[3]), a1 * df[3], -a1 * df[3])
    return ([0.5 * (f - v) + x for f, v, x in zip(df, vis, Fa)], [0.5 * (f + v) - x for f, v, x in zip(df, vis, Fb)])


def _faces(V, uvc, dim, periodic):
    """Minus- and plus-side faces of every cell along `dim`, and the hydrostatic slope."""
    def shift(q, d):
        if periodic:
            return torch.roll(q, -d, dim)
        n = q.shape[dim]
        edge = q.narrow(dim, n - 1 if d > 0 else 0, 1)
        rest = q.narrow(dim, 1, n - 1) if d > 0 else q.narrow(dim, 0, n - 1)
        return torch.cat([rest, edge] if d > 0 else [edge, rest], dim)

    slope = lambda q: _limit(q - shift(q, -1), shift(q, 1) - q)  # noqa: E731
    h, qx, qy, H, _ = V
    u, v, c = uvc
    dh = slope(h)
    dh = torch.where(0.5 * dh.abs() > h, 2.0 * h * _sgn(dh), dh)
    hl, hr, Hl, Hr = shift(h, -1), shift(h, 1), shift(H, -1), shift(H, 1)
    zl, zr = torch.minimum(Hl, H), torch.minimum(Hr, H)
    deta = _limit((h - H + zl).clamp_min(0) - (hl - Hl + zl).clamp_min(0),
                  (hr - Hr + zr).clamp_min(0) - (h - H + zr).clamp_min(0))
    dz, dqx, dqy, dc = dh - deta, h * slope(u) + u * dh, h * slope(v) + v * dh, slope(c)
    out = []
    for s in (-0.5, 0.5):
        hf = h + s * dh
        out.append(_filter(hf, qx + s * dqx, qy + s * dqy, H + s * dz, (c + s * dc) * hf))
    return out[0], out[1], deta


def _series(CC, tCC, t, sl):
    dt = tCC[1] - tCC[0]
    i = max(int((t - tCC[0]) / dt), 0)
    at = lambda k: CC[i, sl, k] + (CC[i + 1, sl, k] - CC[i, sl, k]) / dt * (t - tCC[i])  # noqa: E731
    H = at(3)
    h = at(0) + H
    return h, at(1) * h, at(2) * h, H, torch.zeros_like(h)


def _sweep(P, sw, lo, hi, mask, dim, t, series):
    """Sum of the fluctuations into each cell from its two edges along `dim`.
    Edge frames: x (qx, qy), y (qy, -qx); the low boundary's normal points out."""
    n = mask.shape[dim]
    rot = (lambda s, g: (s[0], g * s[1], g * s[2], s[3], s[4])) if dim == 1 else \
        (lambda s, g: (s[0], g * s[2], -g * s[1], s[3], s[4]))
    back = (lambda d, g: (d[0], g * d[1], g * d[2], d[3], d[4])) if dim == 1 else \
        (lambda d, g: (d[0], -g * d[2], g * d[1], d[3], d[4]))
    cut = lambda s, a, m: tuple(q.narrow(dim, a, m) for q in s)  # noqa: E731
    out = [torch.zeros(mask.shape, device=mask.device, dtype=torch.float64) for _ in range(5)]

    def add(d, a):
        for q, x in zip(out, d):
            q.narrow(dim, a, x.shape[dim]).add_(x)

    if n > 1:
        Dm, Dp = _flux(P, sw, rot(cut(hi, 0, n - 1), 1), rot(cut(lo, 1, n - 1), 1),
                       mask.narrow(dim, 0, n - 1) * mask.narrow(dim, 1, n - 1))
        add(back(Dm, 1), 0)
        add(back(Dp, 1), 1)
    if sw.wbc == 2:  # the seam: the last cell's far face against the first cell's near one
        Dm, Dp = _flux(P, sw, rot(cut(hi, n - 1, 1), 1), rot(cut(lo, 0, 1), 1), mask.narrow(dim, n - 1, 1))
        add(back(Dm, 1), n - 1)
        add(back(Dp, 1), 0)
        return out
    nx, ny = (mask.shape[1], mask.shape[0])
    for side, g, face in ((0, -1, lo), (n - 1, 1, hi)):
        a = cut(face, side, 1)
        qn = 1 if dim == 1 else 2
        b = list(a)
        if sw.wbc == 1 or sw.read_files:
            b[qn] = -b[qn]
        if series is not None and t < series[1][-2]:
            o = (2 * nx + ny if side == 0 else nx) if dim == 1 else (0 if side == 0 else nx + ny)
            sl = slice(o, o + (ny if dim == 1 else nx))
            b = [q.unsqueeze(dim) for q in _series(series[0], series[1], t, sl)]
        Dm, _ = _flux(P, sw, rot(a, g), rot(tuple(b), g), mask.narrow(dim, side, 1))
        add(back(Dm, g), side)
    return out


def _steps64(p, sw, V, mask, series, steps):
    """`steps` time steps of the scheme in float64; state, extrema, time."""
    if series is not None:
        series = (torch.from_numpy(series[0]).to(DEV), [float(q) for q in series[1]])
    nu, s1 = 1.002e-6, p.R - 1.0
    vs = math.sqrt((13.95 * nu / p.DS) ** 2 + 1.09 * s1 * G * p.DS) - 13.95 * nu / p.DS
    Rp = p.DS * math.sqrt(s1 * G * p.DS) / nu
    Aer = Rp ** 0.6 if Rp > 2.36 else 0.586 * Rp ** 1.23
    Kdep = 1.64 + 0.4 * (p.DS / p.Dsg) ** 1.64
    V = tuple(V)
    ext = [torch.full_like(V[0], -1e30) for _ in range(3)]

    def next_dt(V):
        u, v, _ = _velocity(V[0], V[1], V[2])
        cg = torch.sqrt(G * V[0])
        m = (p.CFL * 0.5 * torch.fmin(p.dx / (u.abs() + cg), p.dy / (v.abs() + cg))).nan_to_num(nan=1e30).min()
        return float(m.float()) if V[0].numel() > 4096 else float(m)

    def stage(V0, Vi, t, dt):
        h, qx, qy, H, hc = Vi
        vel = _velocity(h, qx, qy)
        uvc = (vel[0], vel[1], hc / (h + EPS))
        k = list(Vi)
        div = []
        for dim, q, d in ((1, 1, p.dx), (0, 2, p.dy)):
            if sw.order == 2:
                lo, hi, deta = _faces(Vi, uvc, dim, sw.wbc == 2)
                k[q] = k[q] - dt / d * G * h * deta
            else:
                lo = hi = Vi
            div.append(_sweep(p, sw, lo, hi, mask, dim, t, series))
            del lo, hi
        u, v, m = _velocity(V0[0], V0[1], V0[2])
        f = 1.0 + dt * p.FR * m / (V0[0] + EPS)
        k[1], k[2] = k[1] / f, k[2] / f
        Z5 = (Aer * m * math.sqrt(p.FR) / vs) ** 5
        Fe = (vs * (1 - p.porosity) * (1.3e-7 * Z5 / (1 + 4.3e-7 * Z5))).clamp(0.0, 0.1)
        Fd = (vs * Kdep * (V0[4] / (V0[0] + p.epsilon_h))).clamp(0.0, 0.1)
        phi = (Fe - Fd) * float(sw.suspension)
        k[3], k[4] = k[3] - dt * phi, k[4] + dt * phi
        return [q - (dt / p.dx * a + dt / p.dy * b) for q, a, b in zip(k, *div)]

    t, dt = 0.0, next_dt(V)
    for _ in range(steps):
        if sw.order == 1:
            N = _filter(*stage(V, V, t, dt))
        else:
            S = _filter(*stage(V, V, t, dt))
            N = _filter(*[0.5 * a + 0.5 * b for a, b in zip(V, stage(V, S, t, dt))])
        V = N
        wet = V[0] > p.epsilon_h
        ext[0] = torch.where(wet, torch.maximum(ext[0], V[0]), ext[0])
        ext[1] = torch.maximum(ext[1], V[3])
        ext[2] = torch.where(wet, torch.maximum(ext[2], V[0] - V[3]), ext[2])
        t, dt = t + dt, next_dt(V)
    return V, ext, t


def _as_planes(V, precision, eta0):
    h, qx, qy, H, hc = V
    return torch.stack([h - H - eta0, H, qx, qy, hc] if precision else [h, qx, qy, H, hc])


def _exact_steps(case, seed):
    V, mask, series, slr = _coast(case, seed)
    p = make_params(case["nx"], case["ny"], case["dx"], case["dx"])
    sw = _switches(case, series, slr)
    V, ext, t = _steps64(p, sw, V, mask, series, case["steps"])
    return V, ext, t, slr


def _conv64(X, Wk):
    """Same-padded 3x3 convolution of [n][h][w][32] with [cout][tap][cin], float64."""
    n, h, w, _ = X.shape
    Xp = F.pad(X, (0, 0, 1, 1, 1, 1))
    Y = None
    for tap in range(9):
        y = Xp[:, tap // 3:tap // 3 + h, tap % 3:tap % 3 + w] @ Wk[:, tap].T
        Y = y if Y is None else Y + y
    return Y


def _features64(case, H, coarse, fine):
    """Features, normalised targets and interpolated maps on the padded canvas."""
    n, f, pad = case["n"], case["factor"], 8
    nc = n // f
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    cx = ((i + 0.5) / f - 0.5).clamp(0, nc - 1)
    i0 = cx.long().clamp_max(nc - 1)
    i1, ax = (i0 + 1).clamp_max(nc - 1), cx - cx.floor()
    lerp = lambda q: q[..., i0] * (1 - ax) + q[..., i1] * ax  # noqa: E731
    up = lerp(lerp(coarse.transpose(-1, -2)).transpose(-1, -2))
    wet = (coarse[:, 0] > 0).double().repeat_interleave(f, -1).repeat_interleave(f, -2)
    one = torch.ones_like(up[:, 0])
    feat = torch.stack([up[:, 0] / 2.0, up[:, 1] / 0.05, H / 50.0 * one, (H - up[:, 2]) / 2.0, wet, one,
                        i / max(n - 1, 1) * one, (i / max(n - 1, 1))[:, None] * one], dim=1)
    feat = F.pad(feat, (pad,) * 4, mode="replicate")
    X = F.pad(feat.permute(0, 2, 3, 1), (0, 24))
    return X, torch.stack([(fine[:, 0] - up[:, 0]) / 2.0, (fine[:, 1] - up[:, 1]) / 0.05], dim=-1), up


def _net64(X, Wt, B):
    for k in range(6):
        X = _conv64(X, Wt[k]) + B[k]
        if k < 5:
            X = torch.relu(X)
    return X[:, 8:-8, 8:-8, :2]


def _train64(case, Wt, B, H, coarse, fine):
    Wt, B = [torch.tensor(q, device=DEV, requires_grad=True) for q in (Wt, B)]
    m = [torch.zeros_like(q) for q in (Wt, B, Wt, B)]
    state, M64 = 3, (1 << 64) - 1
    losses = []
    for it in range(1, case["iters"] + 1):
        idx = []
        for _ in range(case["batch"]):  # SplitMix64, as tsu_corr_train draws its batches
            state = (state + 0x9E3779B97F4A7C15) & M64
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
            idx.append((z ^ (z >> 31)) % case["samples"])
        total, gW, gB = 0.0, torch.zeros_like(Wt), torch.zeros_like(B)
        cells = case["batch"] * case["n"] ** 2
        for k in idx:  # one image at a time keeps the graph small
            X, tgt, _ = _features64(case, H, coarse[k:k + 1], fine[k:k + 1])
            loss = ((_net64(X, Wt, B) - tgt) ** 2).sum() / (2 * cells)
            g = torch.autograd.grad(loss, (Wt, B))
            gW, gB, total = gW + g[0], gB + g[1], total + loss.item()
        losses.append(total)
        with torch.no_grad():
            for q, g, a, v in ((Wt, gW, m[0], m[2]), (B, gB, m[1], m[3])):
                a.mul_(0.9).add_(g, alpha=0.1)
                v.mul_(0.999).addcmul_(g, g, value=0.001)
                q -= 1e-3 * (a / (1 - 0.9 ** it)) / ((v / (1 - 0.999 ** it)).sqrt() + 1e-8)
    return torch.tensor(losses), Wt.detach(), B.detach()


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "step":
            V, _, _, slr = _exact_steps(case, seed)
            return _as_planes(V, case["precision"], slr)
        if kind == "host_run":
            if case["nx"] * case["ny"] * case["steps"] > 3e8:
                return None
            V, ext, t, _ = _exact_steps(case, seed)
            return dict(V=torch.stack(V), extrema=tuple(ext), t=t)
        if kind == "ensemble":
            out = []
            for k, c in enumerate(_member_cases(case)):
                V, _, _, slr = _exact_steps(dict(c, steps=case["steps"]), int(seed) * 64 + k)
                out.append(_as_planes(V, 1, slr))
            return out
        if kind == "conv":
            X, Wk, b, gate = _conv_inputs(case, seed)
            Y = _conv64(X.double(), Wk.double()) + b.double()
            return Y * (gate > 0) if gate is not None else torch.relu(Y)
        if kind == "wgrad":
            X, dZ = _wgrad_inputs(case, seed)
            n, h, w, _ = X.shape
            Xp, z = F.pad(X.double(), (0, 0, 1, 1, 1, 1)), dZ.double().reshape(-1, 32)
            dW = torch.stack([z.T @ Xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, 32) for t in range(9)], dim=1)
            return dW, z.sum(0)
        Wt, B, H, coarse, fine = [torch.from_numpy(q).to(DEV).double() for q in _corr_inputs(case, seed)]
        if kind == "predict":
            X, _, up = _features64(case, H, coarse, fine)
            y = torch.cat([_net64(X[k:k + 1], Wt, B) for k in range(len(X))])
            return up[:, 0] + 2.0 * y[..., 0], up[:, 1] + 0.05 * y[..., 1], up[:, 0], up[:, 1]
    return _train64(case, Wt, B, H, coarse, fine)
