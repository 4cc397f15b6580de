"""Timed cases: what a user of this package has it do, through its public calls.

listed() are the cases, draw(rng) gives further ones of the same ranges,
prepare(case, seed) makes what a program holds before the call, run(state) is
one pass, work(case) its necessary bytes and operations and exact(case, seed)
the pass's values in 64 bits by plain torch and numpy.

A case's "kind" is the call, its other fields the call's sizes and options:
nx, thickness, ntilt, span (tilts from -span to span degrees; "uneven" shifts
each by up to 0.4 steps, as measured stage angles are), slices, window and
operator as in IconPlan, before/icon/after the iteration schedule.
"""
import math

import numpy as np
import torch

from feilab_b200 import icon, tools, warmstart

DEV = "cuda"


def _geo(kind, nx, thickness, ntilt, slices, span=60.0, uneven=False, **more):
    return dict(kind=kind, nx=nx, thickness=thickness, ntilt=ntilt, span=span, uneven=uneven, slices=slices, **more)


def listed():
    return [
        # One slice of the small 31-tilt series of the tests: the latency of a single transform.
        dict(_geo("forward", 64, 40, 31, 1, complex=False, window="gauss6"), name="forward_one_small_slice"),
        # Forward transform of a batch at the production size (1024 x 300, 61 tilts), the reference's window.
        dict(_geo("forward", 1024, 300, 61, 32, complex=False, window="gauss6"), name="forward_production"),
        # Adjoint at an odd thickness with measured (uneven) angles and a last group that is not full.
        dict(_geo("adjoint", 512, 257, 55, 21, uneven=True, window="gauss6"), name="adjoint_uneven"),
        # Input stage (row transform, weights, adjoint) of a wide detector with the Kaiser-Bessel window.
        dict(_geo("rhs", 2048, 400, 61, 16, window="kb4"), name="input_stage_wide"),
        # Rows to slices with the plan's default operator, the reference's NUFFT pair, at the small workload's size.
        dict(_geo("solve", 256, 128, 61, 32, operator="nufft", window="gauss6", before=1, icon=8, after=1),
             name="solve_nufft"),
        # The main path: rows to slices at the production size with the Toeplitz operator (10 of its 300 iterations).
        dict(_geo("solve", 1024, 300, 61, 128, operator="toeplitz", window="gauss6", before=1, icon=8, after=1),
             name="solve_toeplitz_production"),
        # A series of an uneven batch: other width and thickness, dropped tilts, few slices.
        dict(_geo("solve", 768, 187, 43, 13, span=52.5, uneven=True, operator="toeplitz", window="gauss6", before=1,
                  icon=12, after=1), name="solve_toeplitz_uneven"),
        # Whole call from a device tilt stack to slices in file layout and their reprojection.
        dict(_geo("reconstruct", 512, 256, 61, 24, operator="toeplitz", window="gauss6", before=2, icon=26, after=2),
             name="reconstruct_stack"),
        # Start of a warm solve: the shipped network on production slices.
        dict(_geo("predict", 1024, 300, 61, 8), name="warm_start_predict"),
        # Training of the network, data parallel: loss and gradients of a batch of 512 x 256 slices.
        dict(_geo("gradients", 512, 256, 61, 16), name="warm_start_gradients"),
        # Volume assembly: the cross-validation mask on square slices, the middle 300 rows kept.
        dict(kind="mask", n=1024, ntilt=61, span=60.0, uneven=False, slices=16, radius=60, ystart=362, thickness=300,
             name="mask_volume"),
        # Pre-processing of a tilt stack: mode subtraction and variance normalisation.
        dict(kind="preprocess", nx=1024, ny=1024, ntilt=61, span=60.0, uneven=False, thickness=300,
             name="preprocess_stack"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "adjoint", "adjoint", "rhs", "solve", "solve", "solve", "solve",
                       "reconstruct", "reconstruct", "predict", "gradients", "mask", "preprocess"])
    ntilt, span, uneven = rng.randint(21, 81), rng.choice([45.0, 52.5, 60.0, 67.5]), rng.random() < 0.5
    if kind == "mask":
        n = rng.choice([128, 256, 512, 1024])
        thickness = rng.randint(n // 8, n // 2)
        return dict(kind=kind, n=n, ntilt=ntilt, span=span, uneven=uneven, slices=rng.randint(1, 16),
                    radius=rng.randint(n // 32, n // 8), ystart=rng.randint(0, n - thickness), thickness=thickness)
    if kind == "preprocess":
        return dict(kind=kind, nx=_log(rng, 100, 1024), ny=_log(rng, 100, 1024), ntilt=ntilt, span=span,
                    uneven=uneven, thickness=rng.randint(50, 400))
    nx, thickness = _log(rng, 64, 2048), _log(rng, 32, 400)
    if rng.random() < 0.4:   # detectors are often a power of two wide
        nx = rng.choice([256, 512, 1024, 2048])
    if kind in ("predict", "gradients"):
        nx = min(nx, 1024)
        slices = max(1, min(rng.randint(1, 16), (16 if kind == "gradients" else 8) * 131072 // (nx * thickness)))
        return _geo(kind, nx, thickness, ntilt, slices, span, uneven)
    # At most the production batch's image points in one call.
    points = {"forward": 32, "adjoint": 32, "rhs": 32, "solve": 64, "reconstruct": 24}[kind] * 307200
    slices = max(1, min(_log(rng, 1, 64), points // (nx * thickness)))
    window = rng.choice(["gauss6", "gauss6", "kb4"])
    if kind == "forward":
        return _geo(kind, nx, thickness, ntilt, slices, span, uneven, complex=rng.random() < 0.4, window=window)
    if kind in ("adjoint", "rhs"):
        return _geo(kind, nx, thickness, ntilt, slices, span, uneven, window=window)
    operator = rng.choice(["toeplitz", "toeplitz", "nufft"])
    if operator == "nufft":
        slices = max(1, slices // 3)
    return _geo(kind, nx, thickness, ntilt, slices, span, uneven, operator=operator, window=window, before=1,
                icon=rng.randint(3, 12), after=rng.randint(0, 2))


# ------------------------------------------------------------------ inputs --
def _tilts(case):
    t = np.linspace(-case["span"], case["span"], case["ntilt"])
    if case["uneven"]:
        t = t + 0.4 * (t[1] - t[0]) * np.sin(2.3 * np.arange(len(t)))
    return t.astype(np.float32)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rows(g, S, nx, thickness, tilts):
    """Projection rows (S, ntilt, nx): Gaussian blobs of every slice plus noise at SNR 0.1, zero mean."""
    blobs = 6
    u = torch.rand((4, S, blobs), generator=g, device=DEV)
    cx, cz = (u[0] - 0.5) * 0.8 * nx, (u[1] - 0.5) * 0.8 * thickness
    sig, amp = 1.0 + u[2] * 0.05 * nx, 0.5 + u[3]
    a = torch.from_numpy(tilts).to(DEV) * (math.pi / 180.0)
    k = torch.arange(nx, device=DEV) + 0.5 - nx / 2.0
    rows = torch.zeros((S, len(tilts), nx), device=DEV)
    for b in range(blobs):
        c = cx[:, b, None] * torch.cos(a) + cz[:, b, None] * torch.sin(a)
        rows += amp[:, b, None, None] * torch.exp(-0.5 * ((k - c[..., None]) / sig[:, b, None, None]) ** 2)
    rows -= rows.mean()
    rows /= rows.std()
    return (rows + math.sqrt(10.0) * torch.randn(rows.shape, generator=g, device=DEV)).contiguous()


def _image(g, S, nx, thickness):
    """Slices (S, nx, thickness): non-negative blobs and noise."""
    m = 0.3 * torch.randn((S, nx, thickness), generator=g, device=DEV)
    u = torch.rand((3, S, 5), generator=g, device=DEV)
    x, y = torch.arange(nx, device=DEV).float(), torch.arange(thickness, device=DEV).float()
    for b in range(5):
        s = 2.0 + 0.1 * thickness * u[2, :, b, None]
        ex = torch.exp(-0.5 * ((x - nx * u[0, :, b, None]) / s) ** 2)
        ey = torch.exp(-0.5 * ((y - thickness * u[1, :, b, None]) / s) ** 2)
        m += ex[:, :, None] * ey[:, None, :]
    return m.contiguous()


def _make(case, seed):
    """The arrays of a case, from its seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind == "mask":
        return _image(g, case["slices"], case["n"], case["n"])
    if kind == "preprocess":
        st = _rows(g, case["ny"], case["nx"], case["thickness"], _tilts(case)).transpose(0, 1).contiguous()
        return st * 40.0 + 1000.0
    S, nx, th = case["slices"], case["nx"], case["thickness"]
    if kind == "forward":
        m = _image(g, S, nx, th)
        return torch.complex(m, 0.1 * torch.randn(m.shape, generator=g, device=DEV)) if case["complex"] else m
    if kind == "adjoint":
        return torch.view_as_complex(torch.randn((S, case["ntilt"] * nx, 2), generator=g, device=DEV))
    if kind in ("predict", "gradients"):
        m = _image(g, S, nx, th)
        A = torch.complex(m + torch.randn(m.shape, generator=g, device=DEV), torch.zeros_like(m)) * float(nx)
        return A, m.clamp_min(0.0)
    rows = _rows(g, S, nx, th, _tilts(case))
    return rows.transpose(0, 1).contiguous() if kind == "reconstruct" else rows


def _weights(case):
    """The shipped network of the nearer of its two training sizes."""
    return warmstart.load_weights(nx=1024, thickness=300) if case["nx"] > 600 else warmstart.load_weights(nx=512, thickness=256)


def prepare(case, seed):
    kind, data = case["kind"], _make(case, seed)
    st = dict(case=case, data=data)
    if kind == "mask":
        t = _tilts(case)
        r05, r03, ex = tools.mask_radius(case["n"], t, radius=case["radius"])
        st["mask"] = tools.Mask(case["n"], t, r05, r03, ex, capacity=case["slices"])
    elif kind == "preprocess":
        st["tilts"] = _tilts(case)
    else:
        st["plan"] = p = icon.IconPlan(case["nx"], case["thickness"], _tilts(case), capacity=case["slices"],
                                       window=case.get("window", "gauss6"))
        if "operator" in case:
            p.set_operator(case["operator"])
        if kind in ("predict", "gradients"):
            params, gain, _ = _weights(case)
            st["net"] = warmstart.Network(p)
            st["net"].set_params(params, gain)
    return st


def run(st):
    case, data = st["case"], st["data"]
    kind = case["kind"]
    if kind == "forward":
        return st["plan"].nufft_forward(data)
    if kind == "adjoint":
        return st["plan"].nufft_adjoint(data)
    if kind == "rhs":
        return st["plan"].prepare_rhs(data)
    if kind == "mask":
        return st["mask"].apply(data, case["ystart"], case["thickness"])
    if kind == "preprocess":
        return tools.preprocess(data, st["tilts"], case["thickness"])
    if kind == "predict":
        return st["net"].predict(data[0])
    if kind == "gradients":
        loss = st["net"].backprop(*data)
        return loss, st["net"].grads()
    iters = (case["before"], case["icon"], case["after"])
    if kind == "solve":
        return st["plan"].solve(st["plan"].prepare_rhs(data), iters, 2, 0.0)
    m, rp = st["plan"].reconstruct_stack(data, 0, case["slices"], iters, 2, 0.0, reproject=True)
    return m, rp


# -------------------------------------------------------------------- work --
LAYERS = [(16, 0, 16, 0), (16, 0, 32, 1), (32, 0, 32, 1), (32, 0, 64, 2), (64, 0, 64, 2), (64, 0, 128, 3),
          (128, 0, 128, 3), (128, 64, 64, 2), (64, 0, 64, 2), (64, 32, 32, 1), (32, 0, 32, 1), (32, 16, 16, 0),
          (16, 0, 16, 0)]     # 3x3 layers of the network: inputs, outputs, level


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    the transforms' FFTs (5 n log2 n) and window sums, the network's products."""
    kind = case["kind"]
    if kind == "mask":
        n, S = case["n"], case["slices"]
        fft = 5 * n * math.log2(n)
        return dict(bytes=4.0 * S * n * (n + case["thickness"]) + 4.0 * n * n,
                    flops=S * fft * (0.5 * n + n + 0.5 * case["thickness"]))
    if kind == "preprocess":
        v = case["nx"] * case["ny"] * case["ntilt"]
        return dict(bytes=8.0 * v, flops=10.0 * v)
    S, N0, N1, nz = case["slices"], case["nx"], case["thickness"], case["ntilt"]
    NN, M = N0 * N1, N0 * nz
    if kind in ("predict", "gradients"):
        px = ((N0 + 7) // 8 * 8) * ((N1 + 7) // 8 * 8)
        f = S * (px * 2 * (9 * 16 + 16) + sum(2 * 9 * (a + b) * c * (px >> (2 * l)) for a, b, c, l in LAYERS))
        if kind == "predict":
            return dict(bytes=12.0 * S * NN, flops=float(f))
        return dict(bytes=12.0 * S * NN, flops=3.0 * f)
    n0, n1 = (2 * 2 ** math.ceil(math.log2(n)) for n in (N0, N1))
    taps = 64 if case.get("window") == "kb4" else 196
    grid = 5.0 * (N1 * n0 * math.log2(n0) + n0 * n1 * math.log2(n1))       # one two-dimensional FFT of a padded slice
    nufft = grid + 4.0 * M * taps
    if kind == "forward":
        c = 2 if case["complex"] else 1
        return dict(bytes=S * (4.0 * c * NN + 8.0 * M), flops=S * (nufft if c == 2 else 0.5 * grid + 4.0 * M * taps))
    if kind == "adjoint":
        return dict(bytes=S * (8.0 * M + 8.0 * NN), flops=S * nufft)
    rhs = S * (5.0 * nz * n0 * math.log2(n0) + nufft)
    if kind == "rhs":
        return dict(bytes=S * (4.0 * M + 8.0 * NN), flops=rhs)
    it = case["before"] + case["icon"] + case["after"]
    per = (2.5 * grid + 8.0 * M * taps) if case["operator"] == "nufft" else 2.5 * grid
    out = 4.0 * NN + (4.0 * N0 if kind == "reconstruct" else 0.0)
    return dict(bytes=S * (4.0 * M + out), flops=rhs + S * it * per)


# ------------------------------------------------------------------- exact --
C = torch.complex128


def _nodes(nx, tilts):
    """Node coordinates (ntilt*nx, 2): detector positions summed up in float
    from -1/2 by 1/nx, times cos and sin of the negated angle, as floats."""
    s = np.empty(nx, np.float32)
    s[0] = -0.5
    s[1:] = np.float32(1.0 / nx)
    s = np.cumsum(s, dtype=np.float32).astype(np.float64)
    a = -tilts.astype(np.float64) * 3.14159265 / 180
    xy = np.stack([np.cos(a)[:, None] * s, np.sin(a)[:, None] * s], -1).astype(np.float32)
    return torch.from_numpy(xy.reshape(-1, 2).astype(np.float64)).to(DEV)


def _density(nx, tilts):
    """Density weights (ntilt*nx): |j - nx/2| times the angle step around a tilt."""
    t, nz = -tilts, len(tilts)
    j = np.abs(np.arange(nx) - nx // 2).astype(np.float32)
    d = np.empty(nz, np.float32)
    d[1:-1] = np.abs(t[:-2] - t[2:])
    d[0], d[-1] = 2 * abs(t[1] - t[0]), 2 * abs(t[-2] - t[-1])
    w = d[:, None] * j[None, :]
    w[:, nx // 2] = 180.0 / (4 * nz)
    return torch.from_numpy(w.reshape(-1).astype(np.float64)).to(DEV)


def _cis(x, k):
    return torch.polar(torch.ones((), dtype=torch.float64, device=DEV), 2 * math.pi * x[:, None] * k[None, :])


def _centred(n):
    return torch.arange(n, device=DEV, dtype=torch.float64) - n // 2


def _ndft(img, xy):
    """sum over the image of img e^(-2 pi i (x0 (X - N0/2) + x1 (Y - N1/2)))."""
    S, N0, N1 = img.shape
    out = []
    for q in xy.split(16384):
        E0, E1 = _cis(-q[:, 0], _centred(N0)), _cis(-q[:, 1], _centred(N1))
        out.append(torch.stack([((E0 @ m) * E1).sum(1) for m in img.to(C)]))
    return torch.cat(out, 1)


def _ndft_adjoint(f, xy, N0, N1):
    img = torch.zeros((f.shape[0], N0, N1), dtype=C, device=DEV)
    for q, v in zip(xy.split(16384), f.to(C).split(16384, 1)):
        E0, E1 = _cis(q[:, 0], _centred(N0)).T.contiguous(), _cis(q[:, 1], _centred(N1))
        for s in range(len(f)):
            img[s] += E0 @ (v[s][:, None] * E1)
    return img


def _line(nx):
    """The 1-D transform of a detector row: e^(-2 pi i p_k (X - nx/2)) [k][X]."""
    p = ((np.arange(nx) - nx / 2.0) / nx).astype(np.float32).astype(np.float64)
    return _cis(-torch.from_numpy(p).to(DEV), _centred(nx))


def _rhs(rows, nx, thickness, tilts):
    b = (rows.to(C) @ _line(nx).T).reshape(len(rows), -1)
    return _ndft_adjoint(b * _density(nx, tilts), _nodes(nx, tilts), nx, thickness)


def _solve(A, nx, thickness, tilts, iters):
    """Steepest descent on the normal equations with A^H W A as the
    convolution it is, values below 0 set to 0 in the middle iterations."""
    xy, w = _nodes(nx, tilts), _density(nx, tilts).to(C)
    P0, P1 = 2 * nx, 2 * thickness
    d0 = torch.arange(1 - nx, nx, device=DEV, dtype=torch.float64)
    d1 = torch.arange(1 - thickness, thickness, device=DEV, dtype=torch.float64)
    t = torch.zeros((P0, P1), dtype=C, device=DEV)
    acc = sum((_cis(q[:, 0], d0) * v[:, None]).T @ _cis(q[:, 1], d1) for q, v in zip(xy.split(16384), w.split(16384)))
    t[d0.long()[:, None] % P0, d1.long()[None, :] % P1] = acc
    F = torch.fft.fft2(t)
    out = []
    for a in A.split(8):
        def op(x):
            return torch.fft.ifft2(torch.fft.fft2(x, s=(P0, P1)) * F)[:, :nx, :thickness]

        m = torch.zeros(a.shape, dtype=torch.float64, device=DEV)
        for it in range(sum(iters)):
            r = op(m.to(C)) - a
            rtr = r.abs().square().sum((1, 2))
            rtar = (r.conj() * op(r)).real.sum((1, 2))
            alpha = torch.where(rtar != 0, rtr / rtar, torch.zeros_like(rtar))
            m = m - alpha[:, None, None] * r.real
            if iters[0] <= it < iters[0] + iters[1]:
                m = m.clamp_min(0.0)
        out.append(m)
    return torch.cat(out)


def _net_loss(p, A, target, gain):
    """Prediction of the network in 64 bits, and with a target its loss."""
    F = torch.nn.functional
    off = 160
    S, N0, N1 = A.shape
    x = A.real.double().transpose(1, 2)
    sc = x.square().mean((1, 2)).sqrt()[:, None, None]
    x = F.pad(x / sc, (0, -N0 % 8, 0, -N1 % 8))[:, None]
    x = torch.relu(F.conv2d(x, p[:144].reshape(3, 3, 16).permute(2, 0, 1)[:, None], p[144:160], padding=1))
    ws = []
    for a, b, n, _ in LAYERS:
        k = 9 * n * (a + b)
        ws.append((p[off:off + k].reshape(3, 3, n, a + b).permute(2, 3, 0, 1), p[off + k:off + k + n]))
        off += k + n

    def conv(i, *v):
        return torch.relu(F.conv2d(torch.cat(v, 1), *ws[i], padding=1))

    def up(v):
        return F.interpolate(v, scale_factor=2, mode="nearest")

    e0 = conv(0, x)
    e1 = conv(2, conv(1, F.avg_pool2d(e0, 2)))
    e2 = conv(4, conv(3, F.avg_pool2d(e1, 2)))
    b = conv(6, conv(5, F.avg_pool2d(e2, 2)))
    d2 = conv(8, conv(7, up(b), e2))
    d1 = conv(10, conv(9, up(d2), e1))
    d0 = conv(12, conv(11, up(d1), e0))
    y = ((d0 * p[off:off + 16][None, :, None, None]).sum(1) + p[off + 16])[:, :N1, :N0]
    if target is None:
        return (sc * gain * y).transpose(1, 2)
    return (y - target.double().transpose(1, 2) / (sc * gain)).square().mean()


def _mask_filter(n, tilts, radius):
    """ICONMask3's filter on the full spectrum: the sampled lines' mask,
    faded in past the radius, times the sampling density's inverse."""
    orig = np.zeros((n, n), np.float32)
    f32 = np.float32
    for t in tilts.astype(np.float64):
        c, s = f32(np.cos((-t - 90) * 0.01745329252)), f32(np.sin((-t - 90) * 0.01745329252))
        j = (np.arange(n) - n // 2).astype(np.float32)
        xf, yf = -j * s + f32(n // 2), j * c + f32(n // 2)
        xi, yi = np.trunc(xf).astype(int), np.trunc(yf).astype(int)
        dx, dy = xf - xi.astype(np.float32), yf - yi.astype(np.float32)
        rot = np.zeros((n, n), np.float32)
        for oy, ox, v in ((0, 0, (1 - dx) * (1 - dy)), (1, 0, (1 - dx) * dy), (0, 1, dx * (1 - dy)), (1, 1, dx * dy)):
            k = (xi + ox >= 0) & (xi + ox < n) & (yi + oy >= 0) & (yi + oy < n)
            np.add.at(rot, (yi[k] + oy, xi[k] + ox), v[k])
        orig += rot
    orig = np.minimum(orig, 1.0)
    mean = float(np.abs(np.diff(tilts)).astype(np.float32).mean(dtype=np.float64))
    full_r = math.ceil(2.0 / (mean / 360.0 * 2 * 3.1415926))
    r05 = int(n / 2.0 * float(f32(radius / (n / 2.0))))
    glen = int(10.0 * (n / 150.0))
    c = glen / 3.0
    e0 = math.exp(-(glen * glen) / (2 * c * c))
    k = np.arange(n)
    d = (k + n // 2) % n - n // 2
    rr = np.trunc(np.sqrt((d[:, None] ** 2 + d[None, :] ** 2).astype(np.float64)))
    o = np.roll(orig.astype(np.float64), (-(n // 2), -(n // 2)), (0, 1))
    x = np.maximum(rr - r05, 0)
    w2 = (np.exp(-(x * x) / (2 * c * c)) - e0) / (1 - e0)
    f = np.where(rr < r05, 1.0, np.where(rr <= r05 + glen, np.maximum(o, w2), o))
    f *= np.where((rr > full_r) & (np.abs(o) > 1e-5), rr / full_r, 1.0)
    for kx in range(n // 2 + 1, n):          # the half spectrum's Hermitian partner
        f[:, kx] = f[(-k) % n, n - kx]
    return torch.from_numpy(f).to(DEV)


def exact(case, seed):
    kind, data = case["kind"], _make(case, seed)
    t = _tilts(case)
    if kind == "mask":
        F = torch.fft.fft2(data.double()) * _mask_filter(case["n"], t, case["radius"])
        return torch.fft.ifft2(F).real[:, case["ystart"]:case["ystart"] + case["thickness"]].contiguous()
    if kind == "preprocess":
        v = data.double()
        xe, ye = int(case["nx"] * 0.1), int(case["ny"] * 0.1)
        core = v[:, ye:case["ny"] - ye, xe:case["nx"] - xe].flatten(1)
        lo, step = core.amin(1), (core.amax(1) - core.amin(1)) / 256.0
        bins = ((core - lo[:, None]) / step[:, None]).floor().long()
        hist = torch.stack([torch.bincount(b, minlength=257)[:256] for b in bins])
        first = (hist == hist.amax(1, keepdim=True)).to(torch.int8).argmax(1)
        v = v - (first * step + lo)[:, None, None]
        var = v.flatten(1).var(1, unbiased=False)
        want = 0.33 * case["thickness"] / np.cos(-t.astype(np.float64) / 180.0 * 3.1415926)
        return v / var.sqrt()[:, None, None] * torch.from_numpy(want).to(DEV).sqrt()[:, None, None]
    nx, th = case["nx"], case["thickness"]
    if kind == "forward":
        return _ndft(data, _nodes(nx, t))
    if kind == "adjoint":
        return _ndft_adjoint(data, _nodes(nx, t), nx, th)
    if kind == "rhs":
        return _rhs(data, nx, th, t)
    if kind in ("predict", "gradients"):
        params, gain, _ = _weights(case)
        p = torch.from_numpy(params.astype(np.float64)).to(DEV)
        if kind == "predict":
            with torch.no_grad():
                return torch.cat([_net_loss(p, a, None, gain) for a in data[0].split(2)])
        loss, grad = 0.0, torch.zeros_like(p)
        for a, m in zip(data[0].split(2), data[1].split(2)):
            q = p.clone().requires_grad_(True)
            part = _net_loss(q, a, m, gain) * (len(a) / case["slices"])
            part.backward()
            loss, grad = loss + float(part.detach()), grad + q.grad
        return loss, grad
    iters = (case["before"], case["icon"], case["after"])
    if kind == "solve":
        return _solve(_rhs(data, nx, th, t), nx, th, t, iters)
    m = _solve(_rhs(data.transpose(0, 1).contiguous(), nx, th, t), nx, th, t, iters)
    f = _ndft(m, _nodes(nx, t[np.abs(t).argmin()][None]))      # reprojected at the smallest angle
    return m.transpose(1, 2).contiguous(), (f @ _line(nx).conj()).real.contiguous()
