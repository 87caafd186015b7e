"""The workloads this engine's speed is judged on.

Each case is one pass through the package's public entry points, as a user's
program makes it, on seeded synthetic stacks of blinking point emitters (uniform
positions, a two-state blink chain, a pixel-integrated Gaussian PSF on a flat
background, Poisson shot noise and Gaussian read noise): the images this path
meets.  ``exact`` gives the same results in float64 from plain torch.
"""
import math

import numpy as np
import torch

import nanopyx_gb300 as nx

_F32 = np.float32


def _esrrf(name, frames, height, width, magnification=5, radius=1.5, sensitivity=1.0,
           per_timepoint=0, correlation="AVG", source="cuda", weighting=True):
    return dict(name=name, kind="esrrf", frames=frames, height=height, width=width,
                magnification=magnification, radius=radius, sensitivity=float(sensitivity),
                per_timepoint=per_timepoint, correlation=correlation, source=source,
                weighting=weighting)


def listed():
    return [
        # a preview of a few frames of a small region: latency and launches count
        _esrrf("esrrf_preview", 10, 32, 32),
        # the default call on a small field of view, resident on the device
        _esrrf("esrrf_default", 100, 100, 100),
        # the benchmark's headline acquisition: two correlations, five timepoints
        _esrrf("esrrf_headline", 500, 512, 512, sensitivity=2, per_timepoint=100,
               correlation="VAR+TAC2"),
        # a cropped camera region of odd size: fractional sensitivity, a short
        # last timepoint, rows that are not a multiple of 16 bytes
        _esrrf("esrrf_ragged", 150, 227, 333, magnification=4, radius=2.0, sensitivity=1.5,
               per_timepoint=60, correlation="TAC2"),
        # a camera file as a TIFF reader returns it: a uint16 NumPy array in,
        # NumPy images out, three timepoints
        _esrrf("esrrf_camera_file", 300, 256, 256, per_timepoint=100, source="uint16"),
        # per-frame maps for a user's own temporal analysis
        dict(name="esrrf_frames", kind="esrrf_st", frames=40, height=400, width=300,
             magnification=2, radius=1.0, sensitivity=1.0, weighting=True),
        # frame blocks folded in as an acquisition delivers them
        dict(name="esrrf_stream", kind="stream", blocks=6, frames=50, height=180, width=180,
             magnification=2, radius=1.5, sensitivity=2.0, correlation="VAR", weighting=True),
        # the Fourier-interpolation option, frames above one 256-pixel tile
        dict(name="esrrf_fourier", kind="fourier", frames=8, height=300, width=260,
             magnification=2, radius=1.5, sensitivity=1.0, correlation="AVG"),
        # the reconstruction grid of a parameter search, 4 radii x 4 sensitivities
        dict(name="sweep_grid", kind="sweep", frames=200, height=256, width=256, magnification=4,
             radii=4, sensitivities=4),
        # the scored parameter search with its default grid and magnification
        dict(name="sweep_scored", kind="scored", frames=100, height=128, width=128,
             magnification=2, radii=2, sensitivities=2),
        # SRRF frames and their temporal image
        dict(name="srrf", kind="srrf", frames=100, height=256, width=256, magnification=5,
             ring=0.5, border=0, order=1),
        # eSRRF-3D of a z-stack time series
        dict(name="esrrf3d", kind="esrrf3d", frames=20, slices=16, height=128, width=128,
             magnification=2, magnification_z=2, radius=1.5, sensitivity=1.0, mode="average"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_MAGS = (2, 3, 4, 5, 5, 6, 8)
_RADII = (1.0, 1.5, 1.5, 2.0, 2.5, 3.0)


def draw(rng):
    kind = rng.choice(["esrrf", "esrrf", "esrrf", "esrrf", "esrrf_st", "stream", "fourier",
                       "sweep", "scored", "srrf", "srrf", "esrrf3d"])
    m = rng.choice(_MAGS)
    radius = rng.choice(_RADII)
    sens = float(rng.choice([1, 1, 2, 3, 1.5]))
    top = work(listed()[2])["flops"]
    while True:
        h, w = _log(rng, 24, 640), _log(rng, 24, 640)
        if kind == "esrrf":
            t = _log(rng, 4, 500)
            c = _esrrf("", t, h, w, m, radius, sens, rng.choice([0, 0, 20, 50, 100]),
                       rng.choice(["AVG", "VAR", "TAC2", "VAR+TAC2"]),
                       rng.choice(["cuda", "cuda", "cuda", "uint16", "float32"]),
                       rng.random() < 0.85)
        elif kind == "esrrf_st":
            c = dict(kind=kind, frames=_log(rng, 1, 60), height=h, width=w, magnification=m,
                     radius=radius, sensitivity=sens, weighting=rng.random() < 0.85)
        elif kind == "stream":
            c = dict(kind=kind, blocks=rng.randint(2, 10), frames=_log(rng, 8, 100), height=h,
                     width=w, magnification=rng.choice((2, 4, 5)), radius=1.5, sensitivity=sens,
                     correlation=rng.choice(["AVG", "VAR", "TAC2"]), weighting=True)
        elif kind == "fourier":
            c = dict(kind=kind, frames=_log(rng, 1, 16), height=_log(rng, 24, 400),
                     width=_log(rng, 24, 400), magnification=rng.choice((2, 2, 3, 4)),
                     radius=radius, sensitivity=sens, correlation=rng.choice(["AVG", "VAR"]))
        elif kind == "sweep":
            c = dict(kind=kind, frames=_log(rng, 10, 200), height=h, width=w,
                     magnification=rng.choice((2, 4, 5)), radii=rng.randint(2, 4),
                     sensitivities=rng.randint(2, 4))
        elif kind == "scored":
            c = dict(kind=kind, frames=_log(rng, 20, 200), height=_log(rng, 64, 256),
                     width=_log(rng, 64, 256), magnification=2, radii=2,
                     sensitivities=rng.randint(2, 3))
        elif kind == "srrf":
            c = dict(kind=kind, frames=_log(rng, 4, 200), height=h, width=w, magnification=m,
                     ring=rng.choice([0.5, 0.5, 1.0, 1.5]), border=rng.choice([0, 0, 2]),
                     order=rng.choice([0, 1, 1, 2]))
        else:
            c = dict(kind=kind, frames=_log(rng, 2, 20), slices=_log(rng, 6, 24),
                     height=_log(rng, 32, 160), width=_log(rng, 32, 160),
                     magnification=rng.choice((1, 2, 2, 3)), magnification_z=rng.choice((1, 2)),
                     radius=rng.choice([1.0, 1.5, 2.0]), sensitivity=rng.choice([1.0, 2.0]),
                     mode=rng.choice(["average", "std"]))
        c.pop("name", None)
        if work(c)["flops"] <= 0.9 * top and _output_values(c) <= 6.0e8 and _cost_ok(c):
            return c


def _output_values(c):
    m2 = c["magnification"] ** 2
    n = c["frames"] if c["kind"] in ("esrrf_st", "srrf") else 1
    return n * c["height"] * c["width"] * m2


def _cost_ok(c):
    if c["kind"] == "fourier":  # keeps the dense operators' work below the largest listed case
        return c["frames"] * c["height"] * c["width"] * c["magnification"] ** 2 <= 1.2e7
    return True


def _sweep_grid(c):
    return ([1.0, 2.0, 3.0, 4.0][:c["sensitivities"]], [1.0, 1.5, 2.0, 2.5][:c["radii"]])


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _blinking(T, H, W, seed):
    """(T, H, W) float32 CUDA stack of blinking emitters."""
    rng = np.random.default_rng(seed)
    E = max(1, round(0.0016 * H * W))
    pos_y, pos_x = rng.uniform(0.0, H, E), rng.uniform(0.0, W, E)
    on, state = np.zeros(E, dtype=bool), np.zeros((T, E), dtype=np.float32)
    for t in range(T):
        u = rng.random(E)
        on = np.where(on, u >= 0.5, u < 0.05)
        state[t] = on
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))

    def profile(pos, n):  # share of the PSF (sigma 1.3 px) in every pixel: (E, n)
        edges = torch.arange(n + 1, dtype=torch.float64, device=dev)
        p = torch.from_numpy(pos).to(dev)
        e = torch.erf((edges[None] - p[:, None]) / (1.3 * math.sqrt(2.0)))
        return (0.5 * (e[:, 1:] - e[:, :-1])).float()

    py, px = profile(pos_y, H), profile(pos_x, W)
    st = torch.from_numpy(state).to(dev)
    out = torch.empty((T, H, W), dtype=torch.float32, device=dev)
    step = max(1, (1 << 24) // (H * (W + E)))
    for a in range(0, T, step):
        lam = torch.matmul((py.t()[None] * st[a:a + step, None, :]), px) * 500.0 + 100.0
        x = torch.poisson(lam, generator=gen)
        out[a:a + step] = x + 2.0 * torch.randn(x.shape, device=dev, generator=gen)
    return out


def _stack(c, seed):
    if c["kind"] == "esrrf3d":
        T, S, H, W = c["frames"], c["slices"], c["height"], c["width"]
        return _blinking(T * S, H, W, seed).reshape(T, S, H, W)
    n = c["frames"] * c.get("blocks", 1)
    return _blinking(n, c["height"], c["width"], seed)


def _host(x, source):
    if source == "uint16":
        return x.round().clamp(0, 65535).to(torch.int32).cpu().numpy().astype(np.uint16)
    return x.cpu().numpy()


def prepare(case, seed):
    c = dict(case)
    x = _stack(c, seed)
    if c["kind"] == "esrrf" and c["source"] != "cuda":
        x = _host(x, c["source"])
    if c["kind"] == "stream":
        x = [b.clone() for b in x.split(c["frames"])]
    return c, x


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _correlation(c):
    names = c["correlation"].split("+")
    return names[0] if len(names) == 1 else tuple(names)


def run(state):
    c, x = state
    kind = c["kind"]
    if kind == "esrrf":
        return nx.eSRRF(x, magnification=c["magnification"], radius=c["radius"],
                        sensitivity=c["sensitivity"], frames_per_timepoint=c["per_timepoint"],
                        temporal_correlation=_correlation(c),
                        doIntensityWeighting=c["weighting"])
    if kind == "esrrf_st":
        return nx.eSRRF_ST().run(x, magnification=c["magnification"], radius=c["radius"],
                                 sensitivity=c["sensitivity"],
                                 doIntensityWeighting=c["weighting"])
    if kind == "stream":
        acc = nx.ESRRFAccumulator(c["height"], c["width"], c["magnification"], c["radius"],
                                  c["sensitivity"], c["weighting"])
        for block in x:
            acc.push(block)
        return acc.finalize_device(_correlation(c))
    if kind == "fourier":
        return nx.eSRRF(x, magnification=c["magnification"], radius=c["radius"],
                        sensitivity=c["sensitivity"], temporal_correlation=_correlation(c),
                        use_fht=True)
    if kind == "sweep":
        sens, radii = _sweep_grid(c)
        return nx.esrrf_parameter_sweep(x, c["magnification"], sens, radii)
    if kind == "scored":
        sens, radii = _sweep_grid(c)
        sweep = nx.ParameterSweep()
        qnr = sweep.run(x, c["magnification"], sens, radii)
        return {"qnr": qnr, "rsp": sweep.RSP_map, "frc": sweep.FRC_map}
    if kind == "srrf":
        frames = nx.SRRF(x, magnification=c["magnification"], ringRadius=c["ring"],
                         border=c["border"])
        return {"frames": frames,
                "image": nx.calculate_SRRF_temporal_correlations(frames, order=c["order"])}
    return nx.eSRRF3D(x, magnification_xy=c["magnification"],
                      magnification_z=c["magnification_z"], radius=c["radius"],
                      sensitivity=c["sensitivity"], mode=c["mode"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _samples(m, radius):
    """Window samples inside the radius per output pixel, averaged over phases."""
    p = _rgc_scalars(radius)
    n = 0
    for py in range(m):
        for j in range(p["start"], p["end"]):
            dy = ((2 * py + 1) // m + j) / 2.0 - (py + 0.5) / m
            for px in range(m):
                for i in range(p["start"], p["end"]):
                    dx = ((2 * px + 1) // m + i) / 2.0 - (px + 0.5) / m
                    n += 0 < math.hypot(dx, dy) <= p["tSO"]
    return n / (m * m)


def work(case):
    c, kind = case, case["kind"]
    m, H, W = c["magnification"], c["height"], c["width"]
    T = c["frames"] * c.get("blocks", 1)
    px, plane = T * H * W, H * W * m * m
    if kind == "esrrf3d":
        p = _window3d(c)
        vox = c["slices"] * c["magnification_z"] * plane
        inputs = px * c["slices"]
        samples = int((p["weight"] > 0).sum())
        return {"bytes": 4.0 * (inputs + vox), "flops": float(T * vox * (25 * samples + 40))}
    if kind == "srrf":
        return {"bytes": 4.0 * (px + T * plane + plane), "flops": float(T * plane * (12 * 32 + 12))}
    if kind in ("sweep", "scored"):
        sens, radii = _sweep_grid(c)
        flops = sum(px * (m * m * (10 * _samples(m, r) + 20 * len(sens)) + 60) for r in radii)
        out = plane * len(sens) * len(radii)
        return {"bytes": 4.0 * (px + (out if kind == "sweep" else 0)), "flops": float(flops)}
    flops = px * (m * m * (10 * _samples(m, c["radius"]) + 20) + 60)
    n_out = T
    size = 4.0
    if kind == "esrrf":
        fpt = c["per_timepoint"] or T
        n_out = -(-T // fpt) * len(c["correlation"].split("+"))
        size = 2.0 if c["source"] == "uint16" else 4.0
    elif kind in ("stream", "fourier"):
        n_out = 1
    if kind == "fourier":  # 2-D transforms of the image (x m) and two gradients (x 2 m)
        for k in (m, 2 * m, 2 * m):
            flops += 5.0 * px * k * k * math.log2(max(4.0, px * k * k / T))
    return {"bytes": size * px + 4.0 * n_out * plane, "flops": float(flops)}


# ---------------------------------------------------------------------------
# the same results in float64 (plain torch)
# ---------------------------------------------------------------------------
def _rgc_scalars(radius):
    sigma = _F32(float(radius) / 2.355)
    fwhm = _F32(radius)
    return dict(tSS=float(_F32(_F32(2) * sigma * sigma)), tSO=float(_F32(_F32(2) * sigma + _F32(1))),
                start=-int(_F32(2) * fwhm), end=int(_F32(2) * fwhm + _F32(1)))


def _cubic(v):
    v = v.abs()
    near = v * v * (1.5 * v - 2.5) + 1.0
    far = ((-0.5 * v + 2.5) * v - 4.0) * v + 2.0
    return torch.where(v < 1, near, torch.where(v < 2, far, torch.zeros_like(v)))


def _resample(x, coords, dim):
    """Catmull-Rom of a float64 tensor along one axis: pixel-centre taps, taps
    outside the image skipped."""
    n = x.shape[dim]
    base = torch.floor(coords - 0.5).long() - 1
    inside = (coords >= 0) & (coords < n)
    shape = [1] * x.dim()
    shape[dim] = coords.numel()
    out = None
    for t in range(4):
        nb = base + t
        w = torch.where(inside & (nb >= 0) & (nb < n), _cubic(coords - (nb + 0.5)),
                        torch.zeros_like(coords))
        part = x.index_select(dim, nb.clamp(0, n - 1)) * w.reshape(shape)
        out = part if out is None else out.add_(part)
    return out


def _coords(n, mag, dev):
    return torch.arange(n * mag, dtype=torch.float64, device=dev) / mag


def _roberts(x):
    up = torch.cat([x[:, :1], x[:, :-1]], 1)
    left = torch.cat([x[:, :, :1], x[:, :, :-1]], 2)
    corner = torch.cat([up[:, :, :1], up[:, :, :-1]], 2)
    return up - left + x - corner, left - up + x - corner


def _half_positions(n, m, J, dev):
    """Positions on the 2m-magnified axis of half-pixel indices -J .. 2n - 1 + J
    (index k sits at k m, clamped to the axis) and which of them count."""
    k = torch.arange(-J, 2 * n + J, device=dev)
    return (k * m).clamp(0, 2 * m * n - 1), (k >= 1) & (k <= 2 * (n * m - 1))


def _rgc(gx, gy, valid_y, valid_x, mag, H, W, m, radius, sensitivity, margin):
    """RGC maps (T, H m, W m) from the gradients at the half-pixel positions
    (T, 2 H + 2 J, 2 W + 2 J); ``mag``: the magnified intensity or None."""
    p = _rgc_scalars(radius)
    J = -p["start"]
    T, dev = gx.shape[0], gx.device
    norm = torch.sqrt(gx * gx + gy * gy)
    norm = torch.where(norm > 0, norm, torch.ones_like(norm))
    ok = (valid_y[:, None] & valid_x[None, :]).double()
    gx, gy = gx / norm * ok, gy / norm * ok
    vy, vx = valid_y.double(), valid_x.double()
    out = torch.zeros((T, H * m, W * m), dtype=torch.float64, device=dev)
    for py in range(m):
        for px in range(m):
            acc = torch.zeros((T, H, W), dtype=torch.float64, device=dev)
            wsum = torch.zeros((H, W), dtype=torch.float64, device=dev)
            for j in range(p["start"], p["end"]):
                cy = (2 * py + 1) // m + j
                dy = cy / 2.0 - (py + 0.5) / m
                ys = slice(cy + J, cy + J + 2 * H - 1, 2)
                for i in range(p["start"], p["end"]):
                    cx = (2 * px + 1) // m + i
                    dx = cx / 2.0 - (px + 0.5) / m
                    d = math.hypot(dx, dy)
                    if not 0 < d <= p["tSO"]:
                        continue
                    w = (d * math.exp(-d * d / p["tSS"])) ** 4
                    xs = slice(cx + J, cx + J + 2 * W - 1, 2)
                    gxs, gys = gx[:, ys, xs], gy[:, ys, xs]
                    toward = torch.add(gxs * (dx / d), gys, alpha=dy / d)
                    across = torch.add(gys * (dx / d), gxs, alpha=-dy / d).abs_()
                    acc += across.mul_(-w).add_(w).mul_(toward < 0)
                    wsum += w * vy[ys][:, None] * vx[xs][None, :]
            r = torch.where(wsum > 0, acc / torch.where(wsum > 0, wsum, torch.ones_like(wsum)),
                            torch.zeros_like(acc)).clamp_(min=0)
            if sensitivity > 1:
                r = r ** float(_F32(sensitivity))
            if mag is not None:
                r = r * mag[:, py::m, px::m]
            out[:, py::m, px::m] = r
    if margin > 0:
        out[:, :margin] = 0
        out[:, max(0, H * m - margin):] = 0
        out[:, :, :margin] = 0
        out[:, :, max(0, W * m - margin):] = 0
    return out


def _margin(radius, m):
    return int(float(_F32(radius)) * m)


def _maps(x, m, radius, sensitivity, weighting):
    """Per-frame eSRRF maps in float64, in blocks of frames."""
    T, H, W = x.shape
    J = -_rgc_scalars(radius)["start"]
    py, vy = _half_positions(H, m, J, x.device)
    px, vx = _half_positions(W, m, J, x.device)
    out = torch.empty((T, H * m, W * m), dtype=torch.float64, device=x.device)
    step = max(1, (1 << 24) // (H * W))
    for a in range(0, T, step):
        b = x[a:a + step].double()
        mag = None
        if weighting:
            mag = _resample(_resample(b, _coords(H, m, x.device), 1), _coords(W, m, x.device), 2)
        g = [_resample(_resample(v, py.double() / (2 * m), 1), px.double() / (2 * m), 2)
             for v in _roberts(b)]
        out[a:a + step] = _rgc(g[0], g[1], vy, vx, mag, H, W, m, radius, sensitivity,
                               _margin(radius, m))
    return out


def _temporal(x, name):
    if name == "AVG":
        return x.mean(0)
    c = x - x.mean(0)
    return (c * c).mean(0) if name == "VAR" else (c[:-1] * c[1:]).sum(0) / (x.shape[0] - 1)


def _macro_pixels(x, m):
    """Divides every image by the mean of its sub-pixel phase."""
    for py in range(m):
        for px in range(m):
            part = x[..., py::m, px::m]
            mean = part.mean(dim=(-2, -1), keepdim=True)
            part /= torch.where(mean != 0, mean, torch.ones_like(mean))
    return x


def _mirror_index(n, size, dev):
    copies = -(-size // n)
    copies += 1 - copies % 2
    up = torch.arange(n, device=dev)
    idx = torch.cat([up if (k - copies // 2) % 2 == 0 else up.flip(0) for k in range(copies)])
    start = (copies * n - size) // 2
    return idx[start:start + size]


def _fourier_piece(x, mag):
    T, h, w = x.shape
    n = 1 << max(0, math.ceil(math.log2(max(h, w))))
    L = n * mag
    sq = x[:, _mirror_index(h, n, x.device)][:, :, _mirror_index(w, n, x.device)]
    spec = torch.fft.rfft2(sq)
    big = torch.zeros((T, L, L // 2 + 1), dtype=torch.complex128, device=x.device)
    keep = (n + 1) // 2
    big[:, :keep, :spec.shape[2]] = spec[:, :keep]
    big[:, L - (n - keep):, :spec.shape[2]] = spec[:, keep:]
    z = torch.fft.irfft2(big, s=(L, L))
    lo, hi = x.amin((1, 2), True), x.amax((1, 2), True)
    zlo, zhi = z.amin((1, 2), True), z.amax((1, 2), True)
    span = zhi - zlo
    z = torch.where(span != 0, (z - zlo) * ((hi - lo) / torch.where(span != 0, span, 1.0)) + lo, z)
    y0, x0 = (L - mag * h) // 2, (L - mag * w) // 2
    return z[:, y0:y0 + mag * h, x0:x0 + mag * w]


def _fourier(x, mag, tile=256, overlap=16):
    T, h, w = x.shape
    if h <= tile and w <= tile:
        return _fourier_piece(x, mag)

    def starts(n):
        s = list(range(0, n, tile - 2 * overlap))
        return s + [n - tile] if s[-1] + tile < n else s

    acc = torch.zeros((T, h * mag, w * mag), dtype=torch.float64, device=x.device)
    wgt = torch.zeros((h * mag, w * mag), dtype=torch.float64, device=x.device)
    for r in starts(h):
        for c in starts(w):
            piece = _fourier_piece(x[:, r:r + tile, c:c + tile], mag)
            hann = [torch.from_numpy(np.hanning(n + 2)[1:-1].astype(_F32).astype(np.float64))
                    .to(x.device) for n in piece.shape[1:]]
            win = hann[0][:, None] * hann[1][None, :]
            ys = slice(r * mag, r * mag + piece.shape[1])
            xs = slice(c * mag, c * mag + piece.shape[2])
            acc[:, ys, xs] += piece * win
            wgt[ys, xs] += win
    return torch.where(wgt > 0, acc / torch.where(wgt > 0, wgt, torch.ones_like(wgt)), acc)


def _fourier_maps(x, m, radius, sensitivity):
    T, H, W = x.shape
    J = -_rgc_scalars(radius)["start"]
    py, vy = _half_positions(H, m, J, x.device)
    px, vx = _half_positions(W, m, J, x.device)
    out = torch.empty((T, H * m, W * m), dtype=torch.float64, device=x.device)
    for t in range(T):
        b = x[t:t + 1].double()
        g = [_fourier(v, 2 * m)[:, py][:, :, px] for v in _roberts(b)]
        out[t] = _rgc(g[0], g[1], vy, vx, _fourier(b, m), H, W, m, radius, sensitivity,
                      _margin(radius, m))[0]
    return out


def _srrf_maps(x, m, ring_radius, border):
    T, H, W = x.shape
    dev = x.device
    radius = float(_F32(ring_radius * m))
    step_angle = float(_F32(2.0 * math.pi / 12.0))
    ring = [(float(_F32(math.cos(float(_F32(step_angle * k))) * radius)),
             float(_F32(math.sin(float(_F32(step_angle * k))) * radius))) for k in range(12)]
    out = torch.empty((T, H * m, W * m), dtype=torch.float64, device=dev)
    rows = torch.arange(H * m, dtype=torch.float64, device=dev) + 0.5
    cols = torch.arange(W * m, dtype=torch.float64, device=dev) + 0.5
    block = max(1, (1 << 24) // (H * W * m * m))
    for a in range(0, T, block):
        b = x[a:a + block].double()
        g = torch.zeros((2,) + tuple(b.shape), dtype=torch.float64, device=dev)
        g[0, :, 1:-1, 1:-1] = b[:, 1:-1, 2:] - b[:, 1:-1, :-2]
        g[1, :, 1:-1, 1:-1] = b[:, 2:, 1:-1] - b[:, :-2, 1:-1]
        acc = torch.zeros((b.shape[0], H * m, W * m), dtype=torch.float64, device=dev)
        for xr, yr in ring:
            v = _resample(_resample(g, (rows + yr) / m, 2), (cols + xr) / m, 3)
            norm = torch.sqrt(v[0] * v[0] + v[1] * v[1])
            dk = 1.0 - (v[0] * yr - v[1] * xr).abs() / torch.where(norm > 0, norm, 1.0) / radius
            dk = torch.where(norm > 0, dk * dk, torch.zeros_like(dk))
            acc += torch.where(v[0] * xr + v[1] * yr > 0, -dk, dk)
        r = (acc / 12.0).clamp_(min=0)
        r *= _resample(_resample(b, _coords(H, m, dev), 1), _coords(W, m, dev), 2)
        edge = (1 + border) * m
        keep = torch.zeros((H * m, W * m), dtype=torch.float64, device=dev)
        keep[edge:max(edge, H * m - edge), edge:max(edge, W * m - edge)] = 1
        out[a:a + block] = r * keep
    return _macro_pixels(out, m)


def _srrf_image(x, order):
    if order == 0:
        return x.amax(0)
    mean = x.mean(0)
    if order == 1:
        return mean
    c = x - mean
    return (c[:-2] * c[1:-1]).sum(0).abs() / x.shape[0]


def _window3d(c):
    radius = c["radius"]
    radius_z = radius * 2.8 / 4.0
    sigma, sigma_z = float(_F32(radius / 2.355)), float(_F32(radius_z / 2.355))
    s = np.arange(-int(radius), int(_F32(radius) + _F32(1)) + 1)
    z = np.arange(-int(radius_z), int(_F32(radius_z) + _F32(1)) + 1)
    j, i, k = np.meshgrid(s, s, z, indexing="ij")
    dxy2 = (i * i + j * j).astype(np.float64)
    d = np.sqrt(dxy2 + k * k)
    w = (d * np.exp(-dxy2 / (2 * sigma * sigma)) * np.exp(-k * k / (2 * sigma_z * sigma_z))) ** 4
    count = (d > 0) & (np.sqrt(dxy2) <= 2 * sigma + 1) & (k <= 2 * sigma_z + 1)
    return dict(s=s, z=z, weight=np.where(count, w, 0.0), margin=int(radius * c["magnification"]),
                margin_z=int(radius_z * c["magnification_z"]))


def _volume(c, x):
    """eSRRF-3D of one timepoint in float64; which samples a voxel reads follows
    from its float32 coordinates, as the reference forms them."""
    T, S, H, W = x.shape
    m, mz, dev = c["magnification"], c["magnification_z"], x.device
    p = _window3d(c)
    mg, mgz = p["margin"], p["margin_z"]
    Sm, Hm, Wm = S * mz, H * m, W * m
    out = torch.zeros((Sm, Hm, Wm), dtype=torch.float64, device=dev)
    if Sm <= 2 * mgz or Hm <= 2 * mg or Wm <= 2 * mg:
        return out

    def axis(n, mag, margin, offsets):  # per offset: sample index, and whether it counts
        centre = torch.arange(margin, n * mag - margin, device=dev).float() / mag
        v = centre[None] + torch.from_numpy(offsets).to(dev).float()[:, None]
        return (v * mag).long().clamp(0, n * mag - 1), (v > 0) & (v <= n - 1)

    iy, oy = axis(H, m, mg, p["s"])
    ix, ox = axis(W, m, mg, p["s"])
    iz, oz = axis(S, mz, mgz, p["z"])
    iz = iz // mz
    maps = []
    for t in range(T):
        v = x[t].double()

        def grad(dim):
            n = v.shape[dim]
            i = torch.arange(n, device=dev)
            hi = v.index_select(dim, (i + (dim > 0)).clamp(0, n - 1))
            return (hi - v.index_select(dim, (i - 1).clamp(0, n - 1))) / 2

        g = torch.stack([grad(2), grad(1), grad(0), v])
        if m > 1:
            g = _resample(_resample(g, _coords(H, m, dev), 2), _coords(W, m, dev), 3)
        acc = torch.zeros((Sm - 2 * mgz, Hm - 2 * mg, Wm - 2 * mg), dtype=torch.float64,
                          device=dev)
        wsum = torch.zeros_like(acc)
        for kz, dz in enumerate(p["z"]):
            slab = g[:3].index_select(1, iz[kz])
            for ky, dy in enumerate(p["s"]):
                rows = slab.index_select(2, iy[ky])
                for kx, dx in enumerate(p["s"]):
                    w = float(p["weight"][ky, kx, kz])
                    if w == 0:
                        continue
                    gx, gy, gz = rows.index_select(3, ix[kx])
                    ok = (oz[kz][:, None, None] & oy[ky][None, :, None]
                          & ox[kx][None, None, :]).double() * w
                    wsum += ok
                    dx, dy, dz = float(dx), float(dy), float(dz)
                    cross = ((gy * dz - gz * dy) ** 2 + (gz * dx - gx * dz) ** 2
                             + (gx * dy - gy * dx) ** 2)
                    norm = gx * gx + gy * gy + gz * gz
                    dk = torch.sqrt(cross / torch.where(norm > 0, norm, 1.0))
                    dk = dk / math.sqrt(dx * dx + dy * dy + dz * dz)
                    toward = gx * dx + gy * dy + gz * dz
                    acc += torch.where((toward < 0) & (norm > 0), 1.0 - dk, 0.0) * ok
        r = (acc / wsum).clamp_(min=0)
        if c["sensitivity"] > 1:
            r = r ** c["sensitivity"]
        z = torch.arange(mgz, Sm - mgz, device=dev) // mz
        maps.append(r * g[3].index_select(0, z)[:, mg:Hm - mg, mg:Wm - mg])
    x = torch.stack(maps)
    res = x.mean(0) if c["mode"] == "average" else torch.sqrt(((x - x.mean(0)) ** 2).mean(0))
    out[mgz:Sm - mgz, mg:Hm - mg, mg:Wm - mg] = res
    return out


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    if kind == "scored":
        return None  # two 1-D searches per image: no plain value in a few seconds
    m = c["magnification"]
    x = _stack(c, seed)
    if kind == "esrrf" and c["source"] == "uint16":
        x = torch.from_numpy(_host(x, "uint16").astype(np.float32)).cuda()
    if kind == "esrrf_st":
        return _maps(x, m, c["radius"], c["sensitivity"], c["weighting"])
    if kind == "srrf":
        frames = _srrf_maps(x, m, c["ring"], c["border"])
        return {"frames": frames, "image": _srrf_image(frames, c["order"])}
    if kind == "esrrf3d":
        return _macro_pixels(_volume(c, x), m)[None]
    if kind == "sweep":
        sens, radii = _sweep_grid(c)
        cols = []
        for r in radii:
            total = [0.0] * len(sens)
            step = max(1, (1 << 28) // (x.shape[1] * x.shape[2] * m * m))
            for a in range(0, x.shape[0], step):
                base = _maps(x[a:a + step], m, r, 1.0, False)
                mag = _maps_intensity(x[a:a + step], m)
                for k, s in enumerate(sens):
                    total[k] = total[k] + ((base ** s) * mag).sum(0)
            cols.append(torch.stack([t / x.shape[0] for t in total]))
        return torch.stack(cols, 1)
    if kind == "fourier":
        maps = _fourier_maps(x, m, c["radius"], c["sensitivity"])
        return _macro_pixels(_temporal(maps, c["correlation"])[None], m)[0]
    names = c["correlation"].split("+")
    fpt = c.get("per_timepoint") or x.shape[0]
    res = {n: [] for n in names}
    for a in range(0, x.shape[0], fpt):
        maps = _maps(x[a:a + fpt], m, c["radius"], c["sensitivity"], c["weighting"])
        for n in names:
            res[n].append(_temporal(maps, n))
        del maps
    res = [_macro_pixels(torch.stack(res[n]), m) for n in names]
    if kind == "stream":
        return res[0]
    res = [r.squeeze() for r in res]
    return res[0] if len(names) == 1 else tuple(res)


def _maps_intensity(x, m):
    b = x.double()
    dev = x.device
    return _resample(_resample(b, _coords(x.shape[1], m, dev), 1),
                     _coords(x.shape[2], m, dev), 2)
