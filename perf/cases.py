"""The work that users of this framework give it, as cases that can be timed.

Each case is one pass through the public Python entry points with the buffers
in device memory, as an imaging program holds them: gridding by W-projection
and W-towers, the learned w-kernel's gridding and its training gradient, the
direct DFT, image formation, the w-kernel generator and W-stacking predict.
Sizes follow the configurations, tests and studies of the repository: 64 to
4096 pixels a side, hundreds to millions of visibilities.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes the inputs from a seed, run() is the pass, exact() the same result in
plain FP64 torch without the framework's code, and work() the bytes and
operations that no implementation can do without.
"""
import importlib
import math

import numpy as np
import torch

rg = importlib.import_module("radio-gridders_b200")

DEV = "cuda:0"
C_LIGHT = 299792458.0
PSWF_C = 7.0 * math.pi  # the generator's taper for 16-cell support, used for every support here


def listed():
    return [
        # The smallest whole job, where latency and launches count: uniform
        # weights, W-projection and the dirty image of a 27-station snapshot
        # (351 baselines x 64 dumps, 512 x 512, w planes 10 lambda apart).
        {"name": "snapshot_512_22k", "kind": "snapshot", "n": 22464, "grid": 512, "wmax": 1750.0, "ksize": 16, "ov": 8},
        # A long W-projection synthesis: 2048 x 2048, w to +-2000 lambda,
        # accumulated into the caller's grid.
        {"name": "wproj_2048_1m", "kind": "wproj", "n": 1000000, "grid": 2048, "wmax": 2000.0, "ksize": 16, "ov": 8,
         "accumulate": True},
        # A small W-towers call: few sub-grids, short kernels.
        {"name": "wtowers_512_22k", "kind": "wtowers", "stations": 27, "dumps": 64, "chans": 1, "grid": 512,
         "sub": 128, "margin": 16, "winc": 10.0, "ksize": 16, "ov": 8, "accumulate": False},
        # The benchmark's W-towers observation: 256 stations, 2.09 M visibilities.
        {"name": "wtowers_2048_2m", "kind": "wtowers", "stations": 256, "dumps": 16, "chans": 4, "grid": 2048,
         "sub": 512, "margin": 16, "winc": 10.0, "ksize": 16, "ov": 32, "accumulate": False},
        # The full-scale observation: 512 stations, 8.37 M visibilities, 4096 x 4096.
        {"name": "wtowers_4096_8m", "kind": "wtowers", "stations": 512, "dumps": 32, "chans": 2, "grid": 4096,
         "sub": 512, "margin": 32, "winc": 20.0, "ksize": 16, "ov": 32, "accumulate": False},
        # W-towers with the learned w-kernel (tensor-core inference of every tap), 128 stations.
        {"name": "learned_2048_520k", "kind": "learned", "stations": 128, "dumps": 16, "chans": 4, "grid": 2048,
         "sub": 512, "margin": 16, "winc": 10.0, "ksize": 16},
        # The backward direction of the learned kernel: one batch's loss and gradient.
        {"name": "gradient_16384", "kind": "gradient", "n": 16384, "ksize": 16},
        # The direct DFT at the precision study's size, in its default mode.
        {"name": "dft_1024_200k", "kind": "dft", "grid": 1024, "n": 200000, "theta": 0.05, "wmax": 2000.0,
         "precision": 1},
        # The all-FP64 DFT that images are judged against, at a ragged size.
        {"name": "dft64_500_20k", "kind": "dft", "grid": 500, "n": 19999, "theta": 0.1, "wmax": 600.0,
         "precision": 2},
        # A dirty image of a grid whose side is not a power of two, grid-corrected.
        {"name": "image_2500", "kind": "image", "grid": 2500, "taper": True},
        # The w-kernel table of a W-projection run: 401 planes, 16 x 16 taps, 8 x oversampled.
        {"name": "wkern_401", "kind": "wkern", "planes": 401, "wmax": 2000.0, "ksize": 16, "ov": 8, "theta": 0.1},
        # Predict (degridding): model visibilities of a point-source sky through the w-stack.
        {"name": "predict_2048_200k", "kind": "predict", "lam": 10240.0, "n": 200000, "points": 50, "dw": 10.0,
         "support_w": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(k):
    return k - k % 2


def draw(rng):
    kind = rng.choice(["snapshot", "wproj", "wproj", "wtowers", "wtowers", "wtowers", "learned", "gradient", "dft",
                       "dft", "image", "image", "wkern", "predict"])
    if kind == "snapshot":
        return {"kind": kind, "n": _log_int(rng, 2000, 200000), "grid": _even(_log_int(rng, 128, 1300)),
                "wmax": float(rng.randint(100, 2000)), "ksize": rng.choice([8, 16]), "ov": rng.choice([4, 8])}
    if kind == "wproj":
        return {"kind": kind, "n": _log_int(rng, 5000, 1500000), "grid": _even(_log_int(rng, 300, 3000)),
                "wmax": float(rng.randint(100, 2000)), "ksize": rng.choice([8, 16, 16, 32]), "ov": rng.choice([4, 8]),
                "accumulate": rng.random() < 0.5}
    if kind == "wtowers":
        sub = rng.choice([128, 256, 512, 512])
        ks = rng.choice([8, 16, 16, 16])
        return {"kind": kind, "stations": rng.randint(20, 256), "dumps": rng.randint(5, 32), "chans": rng.randint(1, 4),
                "grid": _even(_log_int(rng, max(512, 2 * sub), 8 * sub)), "sub": sub, "margin": rng.choice([16, 32]),
                "winc": float(rng.choice([5, 10, 20])), "ksize": ks, "ov": rng.choice([8, 16]),
                "accumulate": rng.random() < 0.5}
    if kind == "learned":
        return {"kind": kind, "stations": rng.randint(20, 128), "dumps": rng.randint(4, 16), "chans": rng.randint(1, 4),
                "grid": _even(_log_int(rng, 512, 2048)), "sub": rng.choice([128, 256, 512]), "margin": 16,
                "winc": float(rng.choice([10, 20])), "ksize": 16}
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 700, 16384), "ksize": rng.choice([8, 16])}
    if kind == "dft":
        precision = rng.choice([1, 1, 2])
        return {"kind": kind, "grid": _log_int(rng, 64, 1024 if precision == 1 else 512),
                "n": _log_int(rng, 1000, 200000 if precision == 1 else 40000), "theta": rng.choice([0.05, 0.1]),
                "wmax": float(rng.randint(100, 2000)), "precision": precision}
    if kind == "image":
        grid = rng.choice([2 ** rng.randint(7, 12), _even(_log_int(rng, 100, 4000)), 10 * _even(_log_int(rng, 20, 400))])
        return {"kind": kind, "grid": grid, "taper": rng.random() < 0.5}
    if kind == "wkern":
        ks, ov = rng.choice([(8, 4), (8, 16), (16, 8), (16, 8), (16, 32)])
        return {"kind": kind, "planes": _log_int(rng, 2, 401 if ks * ov <= 128 else 30),
                "wmax": float(rng.randint(5, 2000)), "ksize": ks, "ov": ov, "theta": rng.choice([0.05, 0.1])}
    return {"kind": kind, "lam": float(10 * rng.randint(128, 1024) * 2), "n": _log_int(rng, 1000, 200000),
            "points": rng.randint(1, 100), "dw": float(rng.choice([10, 20, 50])), "support_w": rng.choice([4, 6])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _pswf(c, x):
    """psi_0(c, x) / psi_0(c, 0): Legendre expansion, coefficients from the
    tridiagonal eigenproblem (Xiao, Rokhlin & Yarvin 2001)."""
    nterms = int(2 * c + 40)
    k = np.arange(0, 2 * nterms, 2).astype(np.float64)
    diag = k * (k + 1) + c * c * (2 * k * (k + 1) - 1) / ((2 * k + 3) * (2 * k - 1))
    j = k[:-1]
    off = c * c * (j + 1) * (j + 2) / ((2 * j + 3) * np.sqrt((2 * j + 1) * (2 * j + 5)))
    vec = np.linalg.eigh(np.diag(diag) + np.diag(off, 1) + np.diag(off, -1))[1][:, 0]
    coef = np.zeros(2 * nterms)
    coef[::2] = vec * np.sqrt(k + 0.5)
    leg = np.polynomial.legendre.legval
    return leg(np.asarray(x, np.float64), coef) / leg(0.0, coef)


def _wkernel(theta, planes, size, ov, c, pixels=128):
    """[planes, ov, ov, size, size] complex128: the non-uniform transform of
    the PSWF-tapered w-screen at the oversampled tap positions."""
    lm = theta * (np.arange(pixels) - pixels // 2) / pixels
    a = _pswf(c, 2.0 * lm / theta)
    f64 = dict(dtype=torch.float64, device=DEV)
    taper = torch.tensor(np.outer(a, a), **f64)
    lt = torch.tensor(lm, **f64)
    omn = 1.0 - torch.sqrt(1.0 - (lt[None, :] ** 2 + lt[:, None] ** 2))
    offs = torch.arange(size, **f64)[None, :] - size // 2 - torch.arange(ov, **f64)[:, None] / ov
    ang = offs.reshape(-1, 1) * (torch.arange(pixels, **f64) - pixels // 2)[None, :] / pixels
    e = torch.exp(-2j * math.pi * ang)
    w = torch.as_tensor(np.asarray(planes, np.float64), device=DEV)
    out = torch.empty((len(w), ov, ov, size, size), dtype=torch.complex128, device=DEV)
    for p0 in range(0, len(w), 64):
        s = taper * torch.exp(2j * math.pi * (w[p0:p0 + 64, None, None] * omn))
        k = (e @ s @ e.T) / (pixels * pixels)
        out[p0:p0 + 64] = k.reshape(-1, ov, size, ov, size).permute(0, 1, 3, 2, 4)
    return out


class _Table:
    """A w-kernel table as the gridders take it."""

    def __init__(self, data, w_min, w_step):
        self.data, self.w_min, self.w_step = data, w_min, w_step


def _tracks(seed, stations, ha_hours, lat, dec, log_radial):
    """uvw in metres, [baseline, time, 3], of a seeded station layout."""
    r = np.random.default_rng(seed)
    q = r.uniform(size=stations)
    rad = 20.0 * 1000.0 ** q if log_radial else 10_000.0 * np.sqrt(q)
    phi = r.uniform(0, 2 * math.pi, stations)
    e, n = rad * np.cos(phi), rad * np.sin(phi)
    la, de = math.radians(lat), math.radians(dec)
    xyz = np.stack([-math.sin(la) * n, e, math.cos(la) * n], 1)
    i, j = np.triu_indices(stations, k=1)
    x, y, z = ((xyz[j] - xyz[i])[:, k:k + 1] for k in range(3))
    h = np.asarray(ha_hours) * math.pi / 12.0
    sh, ch, sd, cd = np.sin(h)[None], np.cos(h)[None], math.sin(de), math.cos(de)
    return np.stack([sh * x + ch * y, -sd * ch * x + sd * sh * y + cd * z, cd * ch * x - cd * sh * y + sd * z], 2)


def _flat(uvw, rel_freq, peak_uv, wmax, n):
    """u, v, w in wavelengths (baseline, time, frequency order) on the device,
    scaled so the longest |u|, |v| is peak_uv and, if wmax is given, |w| wmax."""
    t = torch.as_tensor(uvw, device=DEV)
    f = torch.as_tensor(rel_freq, device=DEV)
    flat = [(t[:, :, k, None] * f).reshape(-1)[:n].contiguous() for k in range(3)]
    scale = peak_uv / max(float(flat[0].abs().max()), float(flat[1].abs().max()))
    flat = [a * scale for a in flat]
    if wmax:
        flat[2] = flat[2] * (wmax / float(flat[2].abs().max()))
    return flat


def _predict(seed, u, v, w, theta, sources, power_law):
    """Visibilities of seeded point sources inside the field of view."""
    r = np.random.default_rng(seed + 77)
    lm = r.uniform(-0.4 * theta, 0.4 * theta, (sources, 2))
    q = r.uniform(size=sources)
    a = (10.0 + q * (1.0 - 10.0)) ** -2.0 if power_law else 0.1 + 0.9 * q
    out = torch.zeros(u.numel(), dtype=torch.complex128, device=DEV)
    for (l, m), amp in zip(lm, a):
        ph = u * l + v * m + w * (math.sqrt(1.0 - l * l - m * m) - 1.0)
        ph = (ph - torch.round(ph)) * (-2.0 * math.pi)
        out += torch.polar(torch.full_like(ph, float(amp)), ph)
    return out


def _synthesis(case, seed, peak_uv, theta):
    """A 27-station synthesis of case['n'] visibilities (351 baselines)."""
    n = case["n"]
    uvw = _tracks(seed, 27, np.linspace(-2.0, 2.0, -(-n // 351)), 10.0, -30.0, False)
    u, v, w = _flat(uvw, np.ones(1), peak_uv, case["wmax"], n)
    return u, v, w, _predict(seed, u, v, w, theta, 10, False)


def _zenith(case, seed, theta):
    """A low-frequency array's zenith observation: uneven tower counts."""
    dumps, ks = case["dumps"], case.get("ksize", 16)
    ha = (np.arange(dumps) - (dumps - 1) / 2) * 120.0 / 3600.0
    uvw = _tracks(seed, case["stations"], ha, -26.8, -26.8, True)
    n = uvw.shape[0] * dumps * case["chans"]
    peak = (case["grid"] / 2 - ks / 2 - 2) / theta
    u, v, w = _flat(uvw, 1.0 + 0.005 * np.arange(case["chans"]), peak, None, n)
    return u, v, w, _predict(seed, u, v, w, theta, 50, True)


THETA = 0.1


def _vis_of(case, seed):
    if case["kind"] in ("snapshot", "wproj"):
        return _synthesis(case, seed, (case["grid"] / 2 - case["ksize"] / 2 - 2) / THETA, THETA)
    if case["kind"] in ("wtowers", "learned"):
        return _zenith(case, seed, THETA)
    return _synthesis(case, seed, case["grid"] / 2 / case["theta"], case["theta"])  # dft


def _planes_of(case):
    """Plane w values of the case's table: the data's w range for
    W-projection (10 lambda apart), half a floor either side for W-towers."""
    if case["kind"] == "wtowers":
        return np.arange(-math.ceil(case["winc"] / 2), math.ceil(case["winc"] / 2) + 1.0)
    hi = math.ceil(case["wmax"] / 10.0) + 1
    return 10.0 * np.arange(-hi, hi + 1.0)


def _table_of(case):
    planes = _planes_of(case)
    data = _wkernel(THETA, planes, case["ksize"], case["ov"], math.pi * (case["ksize"] - 2) / 2.0)
    return _Table(data, float(planes[0]), float(planes[1] - planes[0]))


NET = [("W1", (32, 128)), ("b1", (128,)), ("W2", (128, 128)), ("b2", (128,)), ("W3", (128, 128)), ("b3", (128,)),
       ("W4", (128, 2)), ("b4", (2,))]


def _params(seed):
    r = np.random.default_rng(seed + 5)
    out = []
    for name, shape in NET:
        if name[0] == "b":
            out.append(r.normal(0, 0.05, shape))
        else:
            a = r.normal(0, math.sqrt(2.0 / (21 if name == "W1" else 128)), shape)
            if name == "W1":
                a[21:] = 0.0
            out.append(a)
    return np.concatenate([a.ravel() for a in out]).astype(np.float32)


def _samples(case, seed):
    r = np.random.default_rng(seed)
    n, k = case["n"], case["ksize"]
    s = np.stack([r.uniform(-2000, 2000, n), r.uniform(0, 1, n), r.uniform(0, 1, n), r.integers(0, k, n),
                  r.integers(0, k, n)]).astype(np.float32)
    return s, (0.05 * r.normal(size=(n, 2))).astype(np.float32)


def _sepkern(support, ov=1024, corr=64):
    """A separable PSWF kernel [ov, support] and its grid correction [ov, corr]."""
    c = 0.75 * math.pi * support
    t = np.arange(support)[None, :] - support // 2 + (np.arange(ov)[:, None] + 0.5) / ov
    conv = np.where(np.abs(t) <= support / 2, _pswf(c, np.clip(2.0 * t / support, -1.0, 1.0)), 0.0)
    nu = (np.arange(corr * ov) - corr * ov // 2) / (corr * ov)
    xq, step = np.linspace(0.0, support / 2, 801, retstep=True)
    wq = np.full(xq.size, 2.0)
    wq[1::2] = 4.0
    wq[0] = wq[-1] = 1.0
    f = torch.as_tensor(_pswf(c, 2.0 * xq / support) * wq * step / 3.0, device=DEV)
    cos = torch.cos(2 * math.pi * torch.outer(torch.as_tensor(nu, device=DEV), torch.as_tensor(xq, device=DEV)))
    return np.ascontiguousarray(conv), (2.0 * (cos @ f)).cpu().numpy().reshape(ov, corr)


SUPPORT_UV = 8


def _stack_shape(case):
    n = int(math.floor(THETA * case["lam"]))
    max_w = math.sin(THETA / 2) * math.sqrt(2.0 * n * n)
    return n, 2 * n, int(math.ceil(max_w / case["dw"])) + case["support_w"] + 1


def _sky(case, seed):
    n, _, planes = _stack_shape(case)
    g = torch.Generator(device=DEV).manual_seed(seed)
    du = 1.0 / (2.0 * THETA)
    lim = (n - SUPPORT_UV // 2 - 2) * du
    wlim = (planes // 2 - case["support_w"] // 2 - 1) * case["dw"]
    uvw = torch.rand((3, case["n"]), generator=g, dtype=torch.float64, device=DEV) * 2 - 1
    pts = np.random.default_rng(seed).uniform(-0.45 * THETA, 0.45 * THETA, (case["points"], 2))
    return pts, (uvw[0] * lim).contiguous(), (uvw[1] * lim).contiguous(), (uvw[2] * wlim).contiguous(), du


def _uvgrid(case, seed):
    """A gridded observation's plane: power falling off from the centre."""
    n = case["grid"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    z = torch.view_as_complex(torch.randn((n, n, 2), generator=g, dtype=torch.float64, device=DEV))
    r = (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) / (n / 2)
    return z * torch.exp(-4.0 * (r[None, :] ** 2 + r[:, None] ** 2))


def _taper(case):
    return _pswf(PSWF_C, 2.0 * (np.arange(case["grid"]) - case["grid"] // 2) / case["grid"])


# ---------------------------------------------------------------------------
# the passes
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "ctx": rg.Context(0), "stream": torch.cuda.Stream()}
    ctx = s["ctx"]
    ctx.set_stream(s["stream"].cuda_stream)
    if kind in ("snapshot", "wproj", "wtowers", "learned", "dft"):
        u, v, w, vis = _vis_of(case, seed)
        s["vis"] = rg.Visibilities(u, v, w, vis)
    n = case.get("grid")
    if kind in ("snapshot", "wproj", "wtowers", "learned"):
        s["out"] = torch.zeros((n, n), dtype=torch.complex128, device=DEV)
    if kind in ("snapshot", "wproj", "wtowers"):
        s["table"] = _table_of(case)
    if kind == "snapshot":
        s["weighted"] = torch.empty_like(s["vis"].vis)
        s["image"] = torch.empty((n, n), dtype=torch.float64, device=DEV)
    elif kind in ("learned", "gradient"):
        s["net"] = rg.LearnedKernel(ctx, case["ksize"], case.get("winc", 4000.0) / 2, 0.05)
        s["net"].set_params(_params(seed))
        if kind == "gradient":
            s["samples"], s["targets"] = _samples(case, seed)
    elif kind == "dft":
        s["image"] = torch.empty((n, n), dtype=torch.float64, device=DEV)
    elif kind == "image":
        s["grid"] = _uvgrid(case, seed)
        s["out"] = torch.empty_like(s["grid"])
        s["image"] = torch.empty((n, n), dtype=torch.float64, device=DEV)
        s["taper"] = _taper(case) if case["taper"] else None
    elif kind == "wkern":
        s["planes"] = np.linspace(-case["wmax"], case["wmax"], case["planes"]) * (1 + seed % 997 * 1e-6)
        k = case["ksize"]
        s["out"] = torch.empty((case["planes"], case["ov"], case["ov"], k, k), dtype=torch.complex128, device=DEV)
    elif kind == "predict":
        s["sky"] = _sky(case, seed)
        s["tables"] = _sepkern(SUPPORT_UV), _sepkern(case["support_w"])
        s["out"] = torch.empty(case["n"], dtype=torch.complex128, device=DEV)
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind, n = case["kind"], case.get("grid")
    flags = rg.RG_GRID_OVERWRITE
    if case.get("accumulate"):
        flags = rg.RG_GRID_ACCUMULATE
        with torch.cuda.stream(s["stream"]):
            s["out"].zero_()
    if kind == "snapshot":
        vis = s["vis"]
        ctx.weight(n, THETA, vis, out=s["weighted"])
        ctx.grid_wprojection(s["out"], n, THETA, rg.Visibilities(vis.u, vis.v, vis.w, s["weighted"]), s["table"], flags)
        ctx.image_from_grid(s["out"], image=s["image"])
        return {"weighted": s["weighted"], "image": s["image"]}
    if kind == "wproj":
        return ctx.grid_wprojection(s["out"], n, THETA, s["vis"], s["table"], flags)
    if kind == "wtowers":
        return ctx.grid_wtowers(s["out"], n, THETA, s["vis"], s["table"], case["sub"], case["margin"], case["winc"],
                                flags)
    if kind == "learned":
        return rg.grid_wtowers_learned(ctx, s["net"], s["out"], n, THETA, s["vis"], case["sub"], case["margin"],
                                       case["winc"], flags)
    if kind == "gradient":
        loss, grad = s["net"].gradient(s["samples"], s["targets"])
        return {"loss": loss, "grad": grad}
    if kind == "dft":
        return ctx.dft_image(n, case["theta"], s["vis"], case["precision"], image=s["image"])
    if kind == "image":
        with torch.cuda.stream(s["stream"]):
            s["out"].copy_(s["grid"])  # the image is formed in place: the program keeps its grid
        ctx.image_from_grid(s["out"], image=s["image"], taper_1d=s["taper"])
        return {"grid": s["out"], "image": s["image"]}
    if kind == "wkern":
        return ctx.wkern_generate(case["theta"], s["planes"], case["ksize"], case["ov"], out=s["out"])
    pts, u, v, w, du = s["sky"]
    (conv_uv, corr_lm), (conv_w, corr_n) = s["tables"]
    return ctx.wstack_predict(THETA, case["lam"], pts, u, v, w, du, case["dw"], 0.25, conv_uv, conv_w, corr_lm, corr_n,
                              out=s["out"])


# ---------------------------------------------------------------------------
# the same results in plain FP64
# ---------------------------------------------------------------------------

def _cells(x, ov):
    """Cell and sub-cell index of positions in cells."""
    cell = torch.floor(x + 0.5 / ov)
    return cell.long(), torch.floor((x - cell) * ov + 0.5).long()


def _scatter(acc, offset, side, k, taps_of, vis, linear):
    """acc[offset + footprint] += vis * conj(taps), chunk by chunk. linear:
    the flat index decides what lies inside, else column and row do."""
    ys, xs = torch.meshgrid(torch.arange(k, device=DEV), torch.arange(k, device=DEV), indexing="ij")
    ys, xs = ys.reshape(-1), xs.reshape(-1)
    base, row0, col0 = offset
    step = 1 << 18
    for i in range(0, vis.numel(), step):
        sl = slice(i, i + step)
        val = vis[sl, None] * taps_of(sl).conj()
        row, col = row0[sl, None] + ys, col0[sl, None] + xs
        at = row * side + col
        ok = (at >= 0) & (at < side * side)
        if not linear:
            ok &= (row >= 0) & (row < side) & (col >= 0) & (col < side)
        at = torch.where(ok, at, 0) + base[sl, None]
        val = torch.where(ok, val, 0)
        flat = torch.view_as_real(acc).reshape(-1, 2)
        flat.index_add_(0, at.reshape(-1), torch.view_as_real(val).reshape(-1, 2))


def _table_taps(t, k, plane, fy, fx):
    flat = t.data.reshape(-1, k * k)
    ov = t.data.shape[1]
    row = (plane * ov + fy) * ov + fx
    return lambda sl: flat[row[sl]]


def _plane(w, t):
    return torch.floor((w - t.w_min) / t.w_step + 0.5).long()


def _exact_wproj(case, u, v, w, vis, t):
    n, k, ov = case["grid"], case["ksize"], case["ov"]
    cx, fx = _cells(THETA * u, ov)
    cy, fy = _cells(THETA * v, ov)
    acc = torch.zeros(n * n, dtype=torch.complex128, device=DEV)
    where = (torch.zeros_like(cx), cy + n // 2 - k // 2, cx + n // 2 - k // 2)
    _scatter(acc, where, n, k, _table_taps(t, k, _plane(w, t), fy, fx), vis, False)
    return acc.reshape(n, n)


def _axis_chunk(x, n, chunk, theta):
    count = n // chunk + 1
    origin = chunk * torch.arange(count, dtype=torch.float64, device=DEV) - n // 2
    lo = (origin - 0.5) / theta
    c = torch.searchsorted(lo, x, right=True) - 1
    ok = (c >= 0) & (x < lo[c.clamp(min=0)] + chunk / theta)
    c = c.clamp(min=0)
    return c, ok, ((origin + chunk // 2) / theta)[c]


def _exact_wtowers(case, u, v, w, vis, taps_for):
    """Sub-grid per (tower, w floor), backward transform, the floor's Fresnel
    phase, sum over floors, forward transform, add-back."""
    n, s, m, winc, k = case["grid"], case["sub"], case["margin"], case["winc"], case["ksize"]
    chunk = s - m
    cx, okx, midx = _axis_chunk(u, n, chunk, THETA)
    cy, oky, midy = _axis_chunk(v, n, chunk, THETA)
    wp = torch.floor(w / winc + 0.5)
    keep = (okx & oky).nonzero()[:, 0]
    x, y, wr = (THETA * (u - midx))[keep], (THETA * (v - midy))[keep], (w - wp * winc)[keep]
    tower = (cy * (n // chunk + 1) + cx)[keep]
    wp, vz = wp[keep].long(), vis[keep]
    col, row, taps_of = taps_for(x, y, wr)
    order = torch.argsort(tower)
    grid = torch.zeros((n, n), dtype=torch.complex128, device=DEV)
    lm = THETA * ((torch.arange(s, dtype=torch.float64, device=DEV) + s // 2) % s - s // 2) / s
    ph = winc * (1.0 - torch.sqrt(1.0 - lm[None, :] ** 2 - lm[:, None] ** 2))
    ids, counts = torch.unique_consecutive(tower[order], return_counts=True)
    begin = 0
    for t, cnt in zip(ids.tolist(), counts.tolist()):
        mine = order[begin:begin + cnt]
        begin += cnt
        total = torch.zeros((s, s), dtype=torch.complex128, device=DEV)
        floors = torch.unique(wp[mine])
        for f0 in range(0, len(floors), 64):
            fl = floors[f0:f0 + 64]
            idx = mine[(wp[mine] >= fl[0]) & (wp[mine] <= fl[-1])]
            slot = torch.searchsorted(fl, wp[idx])
            acc = torch.zeros(len(fl) * s * s, dtype=torch.complex128, device=DEV)
            pick = taps_of(idx)
            _scatter(acc, (slot * s * s, row[idx] + s // 2 - k // 2, col[idx] + s // 2 - k // 2), s, k, pick, vz[idx],
                     True)
            sub = torch.fft.ifft2(acc.reshape(-1, s, s))
            for i, f in enumerate(fl.tolist()):
                turns = -f * ph
                turns -= torch.round(turns)
                total += sub[i] * torch.polar(torch.ones_like(turns), 2 * math.pi * turns)
        img = torch.fft.fft2(total)
        ty, tx = divmod(t, n // chunk + 1)
        y0, x0 = chunk * ty - m // 2, chunk * tx - m // 2
        ya, yb, xa, xb = max(0, y0), min(n, y0 + s), max(0, x0), min(n, x0 + s)
        grid[ya:yb, xa:xb] += img[ya - y0:yb - y0, xa - x0:xb - x0]
    return grid


def _exact_image(grid, taper):
    """Hermitian sum, shift, forward transform, shift, real part over the taper."""
    n = grid.shape[0]
    flat = grid.reshape(-1)
    h = flat.clone()
    tail = flat[n + 1:]
    h[n + 1:] += tail.flip(0).conj()
    out = torch.fft.fftshift(torch.fft.fft2(torch.fft.fftshift(h.reshape(n, n))))
    img = out.real.clone()
    if taper is not None:
        t = torch.as_tensor(taper, device=DEV)
        img = img / (t[:, None] * t[None, :])
    return out, img


def _features(w, du, dv, tx, ty, k, wmax):
    half = k / 2.0
    p, q = tx - half - du, ty - half - dv
    f = [w / wmax, 2 * du - 1, 2 * dv - 1, p / half, q / half]
    for z in (p, q):
        for i in range(1, 5):
            f += [torch.cos(math.pi * i * z / (half + 1)), torch.sin(math.pi * i * z / (half + 1))]
    return torch.stack(torch.broadcast_tensors(*f), -1)


def _net(params):
    out, o = [], 0
    for name, shape in NET:
        size = int(np.prod(shape))
        out.append(torch.as_tensor(params[o:o + size].astype(np.float64).reshape(shape), device=DEV))
        o += size
    return out


def _forward(p, f):
    silu = torch.nn.functional.silu
    h = silu(f @ p[0][:21] + p[1])
    h = silu(h @ p[2] + p[3])
    return silu(h @ p[4] + p[5]) @ p[6] + p[7]


def _exact_learned(case, seed, u, v, w, vis):
    k, p, wmax = case["ksize"], _net(_params(seed)), case["winc"] / 2
    ty, tx = torch.meshgrid(*[torch.arange(k, dtype=torch.float64, device=DEV)] * 2, indexing="ij")

    def taps_for(x, y, wr):
        col, row = torch.floor(x), torch.floor(y)
        fx, fy = x - col, y - row

        def taps_of(idx):
            def pick(sl):
                i = idx[sl]
                out = []
                for j in range(0, len(i), 4096):
                    q = i[j:j + 4096]
                    a = _forward(p, _features(wr[q, None], fx[q, None], fy[q, None], tx.reshape(1, -1),
                                              ty.reshape(1, -1), k, wmax)) * 0.05
                    out.append(torch.view_as_complex(a.contiguous()))
                return torch.cat(out)
            return pick
        return col.long(), row.long(), taps_of
    return _exact_wtowers(case, u, v, w, vis, taps_for)


def _exact_gradient(case, seed):
    s, t = _samples(case, seed)
    a = [torch.as_tensor(z.astype(np.float64), device=DEV) for z in s]
    p = [z.requires_grad_() for z in _net(_params(seed))]
    y = _forward(p, _features(*a, case["ksize"], 2000.0))
    loss = ((y - torch.as_tensor(t.astype(np.float64), device=DEV) / 0.05) ** 2).sum() / case["n"]
    loss.backward()
    return {"loss": float(loss), "grad": torch.cat([z.grad.reshape(-1) for z in p])}


def _exact_dft(case, u, v, w, vis):
    n, theta = case["grid"], case["theta"]
    lm = theta * (torch.arange(n, dtype=torch.float64, device=DEV) - n // 2) / n
    uvw, img = torch.stack([u, v, w]), []
    rows = max(1, (1 << 28) // (n * 4096))
    for y in range(0, n, rows):
        m, l = torch.meshgrid(lm[y:y + rows], lm, indexing="ij")
        pix = torch.stack([l.reshape(-1), m.reshape(-1), (1.0 - torch.sqrt(1.0 - l * l - m * m)).reshape(-1)], 1)
        acc = torch.zeros(pix.shape[0], dtype=torch.float64, device=DEV)
        for k in range(0, u.numel(), 4096):
            ph = (pix @ uvw[:, k:k + 4096]).mul_(2 * math.pi)
            z = vis[k:k + 4096]
            acc += torch.cos(ph) @ z.real + torch.sin(ph) @ z.imag
        img.append(acc.reshape(-1, n))
    return 2.0 * torch.cat(img)


def _exact_predict(case, seed):
    n, g, planes = _stack_shape(case)
    pts, u, v, w, du = _sky(case, seed)
    (cuv, klm), (cw, kn) = _sepkern(SUPPORT_UV), _sepkern(case["support_w"])
    lm, nn, lam, dw = klm.ravel(), kn.ravel(), case["lam"], case["dw"]
    sky = {}
    for l, m in pts:
        lc, mc = int(math.floor((l / THETA + 0.5) * n)), int(math.floor((m / THETA + 0.5) * n))
        lq, mq = lc / lam - THETA / 2, mc / lam - THETA / 2
        nq = math.sqrt(1.0 - lq * lq - mq * mq) - 1.0
        a = (lm[int(math.floor(du * lq * len(lm))) + len(lm) // 2] * lm[int(math.floor(du * mq * len(lm))) + len(lm) // 2]
             * nn[int(math.floor(dw * nq * len(nn))) + len(nn) // 2])
        sky[lc, mc] = sky.get((lc, mc), 0.0) + 1.0 / a
    pix = np.array(list(sky)), np.array(list(sky.values()))
    at = ((g - n) // 2 + pix[0] + g // 2) % g
    l, m = (torch.as_tensor(THETA * (pix[0][:, i] - n / 2) / n, device=DEV) for i in (0, 1))
    ph = dw * (1.0 - torch.sqrt(1.0 - l * l - m * m))
    val = torch.as_tensor(pix[1], device=DEV)
    col, row = (torch.as_tensor(at[:, i], device=DEV) for i in (0, 1))
    sw, suv, ow, ouv = cw.shape[1], cuv.shape[1], cw.shape[0], cuv.shape[0]
    cu, cv, cz = torch.ceil(u / du), torch.ceil(v / du), torch.ceil(w / dw)
    ou = torch.floor((u - cu * du).abs() / du * ouv).long()
    ov = torch.floor((v - cv * du).abs() / du * ouv).long()
    oz = torch.floor((w - cz * dw).abs() / dw * ow).long()
    tuv, tw = torch.as_tensor(cuv, device=DEV), torch.as_tensor(cw, device=DEV)
    x0, y0, p0 = cu.long() + n - suv // 2, cv.long() + n - suv // 2, cz.long() + planes // 2 - sw // 2
    out = torch.zeros(u.numel(), dtype=torch.complex128, device=DEV)
    k = torch.arange(suv, device=DEV)
    for p in range(planes):
        turns = (p - planes // 2) * ph
        turns -= torch.round(turns)
        image = torch.zeros((g, g), dtype=torch.complex128, device=DEV)
        image[row, col] = val * torch.polar(torch.ones_like(turns), 2 * math.pi * turns)
        uv = torch.fft.fftshift(torch.fft.fft2(image))
        i = ((p >= p0) & (p < p0 + sw)).nonzero()[:, 0]
        wt = tw[oz[i], p - p0[i]]
        for j, q in zip(i.split(1 << 17), wt.split(1 << 17)):
            z = uv[(y0[j, None] + k)[:, :, None], (x0[j, None] + k)[:, None, :]]
            out[j] += q * (z * tuv[ov[j]][:, :, None] * tuv[ou[j]][:, None, :]).sum((1, 2))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "wkern":
        planes = np.linspace(-case["wmax"], case["wmax"], case["planes"]) * (1 + seed % 997 * 1e-6)
        return _wkernel(case["theta"], planes, case["ksize"], case["ov"], math.pi * (case["ksize"] - 2) / 2.0)
    if kind == "predict":
        return _exact_predict(case, seed)
    if kind == "image":
        grid, image = _exact_image(_uvgrid(case, seed), _taper(case) if case["taper"] else None)
        return {"grid": grid, "image": image}
    u, v, w, vis = _vis_of(case, seed)
    if kind == "dft":
        return _exact_dft(case, u, v, w, vis)
    if kind == "learned":
        return _exact_learned(case, seed, u, v, w, vis)
    t = _table_of(case)
    if kind == "wtowers":
        k, ov = case["ksize"], case["ov"]

        def taps_for(x, y, wr):
            (cx, fx), (cy, fy) = _cells(x, ov), _cells(y, ov)
            plane = _plane(wr, t)
            return cx, cy, lambda idx: _table_taps(t, k, plane[idx], fy[idx], fx[idx])
        return _exact_wtowers(case, u, v, w, vis, taps_for)
    if kind == "snapshot":
        n = case["grid"]
        cell = (torch.floor(THETA * v + 0.5).long() + n // 2) * n + torch.floor(THETA * u + 0.5).long() + n // 2
        vis = vis / torch.bincount(cell, minlength=n * n)[cell]
        return {"weighted": vis, "image": _exact_image(_exact_wproj(case, u, v, w, vis, t), None)[1]}
    return _exact_wproj(case, u, v, w, vis, t)


# ---------------------------------------------------------------------------
# the least that a pass has to move and compute
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    n = case.get("grid", 0)
    cells = float(n) * n
    fft = 5.0 * cells * math.log2(max(2.0, cells))
    if kind in ("wtowers", "learned"):
        nvis = case["stations"] * (case["stations"] - 1) // 2 * case["dumps"] * case["chans"]
    else:
        nvis = case.get("n", 0)
    k2 = float(case.get("ksize", 0)) ** 2
    grid_bytes = 16.0 * cells * (2 if case.get("accumulate") else 1)
    if kind in ("snapshot", "wproj", "wtowers"):
        # inputs and table once, the grid once (twice when accumulated into);
        # eight operations a tap; W-towers also one transform of the plane each way
        table = 16.0 * len(_planes_of(case)) * case["ov"] ** 2 * k2
        used = min(table, 16.0 * nvis * k2)
        out = {"bytes": 40.0 * nvis + used + grid_bytes, "flops": 8.0 * k2 * nvis}
        if kind == "wtowers":
            out["flops"] += 2 * fft
        if kind == "snapshot":  # weights out, the image instead of the grid
            out["bytes"] += 16.0 * nvis - 8.0 * cells
            out["flops"] += fft
        return out
    if kind == "learned":
        return {"bytes": 40.0 * nvis + grid_bytes, "flops": nvis * k2 * 2.0 * (21 * 128 + 2 * 128 * 128 + 256)}
    if kind == "gradient":
        return {"bytes": 28.0 * nvis + 8.0 * 37500, "flops": nvis * 6.0 * (21 * 128 + 2 * 128 * 128 + 256)}
    if kind == "dft":
        return {"bytes": 40.0 * nvis + 8.0 * cells, "flops": 4.0 * cells * nvis}  # two multiply-adds a pair
    if kind == "image":  # grid in, transformed grid and image out
        return {"bytes": 40.0 * cells, "flops": fft}
    if kind == "wkern":  # taps out; both transforms of an even screen, half of it, real phasors
        q, m = case["ksize"] * case["ov"], 128
        return {"bytes": 16.0 * case["planes"] * q * q, "flops": case["planes"] * 4.0 * (m * m / 4 * q + m / 2 * q * q)}
    _, g, planes = _stack_shape(case)
    taps = case["support_w"] * SUPPORT_UV ** 2
    return {"bytes": 40.0 * nvis + 16.0 * planes * g * g,
            "flops": planes * 5.0 * g * g * math.log2(float(g)) + 8.0 * taps * nvis}
