"""Workloads of the correlation-and-fit engine, through its public entry points.

Four kinds of call, as a user's program makes them:
  plan     engine.Plan.execute: one uint16 stack in HBM -> ACF, variance, fits
  batch    engine.Batch.execute: several (binning, offset) jobs over one stack as one graph
  calcacf  GpufitImFCS.calcACF: the plugin's float stack in host memory
  fit      GpufitImFCS.fit: curves in host memory -> parameters

The stacks come from the library's Monte-Carlo simulator (diffusing, bleaching
particles, Poisson photons) with the counts of an EMCCD camera: `GAIN` counts
per photon on an offset of `OFFSET`.  exact() gives the outputs in 64 bits
from plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from imaging_fcs_1_52_gb300 import _lib, engine
from imaging_fcs_1_52_gb300.gpufit_imfcs import FitModel, FitResult, GpufitImFCS, Model

OFFSET, GAIN = 100, 25           # camera counts: offset, counts per photon
FRAMETIME = 1e-3                 # s
PIXEL_UM, PSF_UM = 0.24, 0.4     # pixel size, 1/e^2 radius of the PSF
TIRF_SZ_UM = 1e6 * 0.515 / 1.49  # axial extent of the TIRF model (no axial factor)
BLEACH = {"none": _lib.BLEACH_NONE, "exp": _lib.BLEACH_SINGLE_EXP, "exp2": _lib.BLEACH_DOUBLE_EXP,
          "poly": _lib.BLEACH_POLYNOMIAL}

PLAN = {"kind": "plan", "first": 0, "bin": 1, "step": 1, "dx": 0, "dy": 0, "p": 16, "q": 8, "bleach": "none",
        "order": 4, "gls": False, "bayes": False, "sz_um": TIRF_SZ_UM}


def _plan(name, width, height, frames, **kw):
    return {"name": name, **PLAN, "width": width, "height": height, "frames": frames, **kw}


def listed():
    return [
        # a handful of pixels while looking for settings: latency and launches
        _plan("roi_8x8x4000", 8, 8, 4000),
        # the plugin's ordinary region of interest with its polynomial bleach correction
        _plan("roi_21x21x20000_poly4", 21, 21, 20000, bleach="poly"),
        # a full camera frame of a long recording, exponential bleach: the headline workload
        _plan("frame_128x128x50000_exp", 128, 128, 50000, bleach="exp"),
        # spatial cross-correlation of 2 x 2 binned pixels (the manual's cf 1,1 setting)
        _plan("ccf_128x128x20000_bin2_poly4", 128, 128, 20000, bin=2, step=2, dx=1, dy=1, bleach="poly"),
        # overlapping 5 x 5 windows of a ragged sub-frame, part of the frames, polynomial of order 6
        _plan("odd_101x67x12345_bin5_poly6", 101, 67, 12345, first=345, bin=5, bleach="poly", order=6),
        # two bleaching species: double-exponential correction of a small frame
        _plan("roi_48x48x10000_exp2", 48, 48, 10000, bleach="exp2"),
        # generalised least squares: covariance of the lags, Cholesky, whitened fit
        _plan("gls_64x64x20000", 64, 64, 20000, gls=True),
        # light-sheet model (finite axial extent) with Bayesian model selection
        _plan("bayes_spim_40x40x10000", 40, 40, 10000, bayes=True, sz_um=1.0),
        # the plugin's finer lag-time table, P = 32
        _plan("p32_48x48x20000", 48, 48, 20000, p=32),
        # binnings x offsets over one stack as one graph (diffusion law and cross-correlation, GLS fits)
        {"name": "batch_96x96x10000_gls", "kind": "batch", "width": 96, "height": 96, "frames": 10000, "bins": 2,
         "offsets": 2, "gls": True},
        # the plugin's own call: float stack in host memory, ACF back to host memory
        {"name": "calcacf_64x64x10000", "kind": "calcacf", "width": 64, "height": 64, "frames": 10000, "dx": 0,
         "dy": 0},
        # the plugin's own fit call: one curve per pixel of a full frame
        {"name": "fit_16384", "kind": "fit", "fits": 16384, "points": 72},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["plan"] * 8 + ["batch", "calcacf", "fit"])
    if kind == "fit":
        return {"kind": kind, "fits": log_int(64, 16384), "points": rng.randint(40, 72)}
    width, height = log_int(8, 128), log_int(8, 128)
    if kind == "batch":
        width, height = min(max(width, 16), 96), min(max(height, 16), 96)
        return {"kind": kind, "width": width, "height": height, "frames": log_int(4000, 10000),
                "bins": rng.randint(1, 2), "offsets": rng.randint(1, 2), "gls": rng.random() < 0.5}
    if kind == "calcacf":
        return {"kind": kind, "width": min(width, 64), "height": min(height, 64), "frames": log_int(3000, 10000),
                "dx": rng.randint(0, 1), "dy": rng.randint(0, 1)}
    c = {**PLAN, "width": width, "height": height, "frames": log_int(4500, 50000)}
    c["first"] = rng.choice([0, 0, rng.randint(1, 200)])
    c["bin"] = rng.choice([1, 1, 1, 2, 3, 4, 5])
    c["step"] = rng.choice([1, c["bin"]])
    if rng.random() < 0.3:
        c["dx"], c["dy"] = rng.choice([(1, 0), (0, 1), (1, 1), (2, 0), (0, 2)])
    c["p"] = rng.choice([16, 16, 16, 16, 16, 32])
    c["q"] = rng.choice([8, 8, 8, 7, 6, 5])
    c["bleach"] = rng.choice(["none", "poly", "poly", "exp", "exp", "exp2"])
    c["order"] = rng.randint(2, 8)
    option = rng.choice(["", "", "", "gls", "bayes", "spim"])
    c["gls"] = option == "gls" and c["p"] == 16
    c["bayes"] = option == "bayes"
    if option == "spim":
        c["sz_um"] = round(rng.uniform(0.8, 1.5), 2)
    if c["gls"] or c["p"] == 32 or c["bayes"]:
        c["width"], c["height"] = min(width, 64), min(height, 64)
        c["frames"] = min(c["frames"], 20000)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _stack(width, height, frames, bleach, seed):
    """CUDA uint16 [frames][height][width]: D per 16 x 16 tile from U(0.2, 5) um^2/s, 20 particles per um^2; where
    the case corrects bleaching they bleach over the recording (two pools of unequal rate for the double exponential)."""
    dmap = np.random.default_rng(seed).uniform(0.2, 5.0, ((height + 15) // 16, (width + 15) // 16))
    span = frames * FRAMETIME
    taus = {"none": (0.0,), "exp": (0.4 * span,), "exp2": (0.05 * span, 0.8 * span)}.get(bleach, (span,))
    total = None
    for i, tau in enumerate(taus):
        s = engine.simulate(width, height, frames, frametime=FRAMETIME, steps_per_frame=1, pixel_um=PIXEL_UM,
                            psf_um=PSF_UM, density=20.0 / len(taus), cps=1e4, tau_bleach=tau, offset=0,
                            seed=2 * seed + 1 + i, d_tile_map=dmap)
        if total is None:
            total = s
        else:
            total.view(torch.int16).add_(s.view(torch.int16))
    total.view(torch.int16).mul_(GAIN).add_(OFFSET)
    return total


def _config(c):
    cst = engine.model_constants(pixel_um=PIXEL_UM, binx=c["bin"], biny=c["bin"], psf_um=PSF_UM, sz_um=c["sz_um"],
                                 cfx=c["dx"], cfy=c["dy"])
    return engine.FCSConfig(width=c["width"], height=c["height"], frames=c["first"] + c["frames"], first=c["first"],
                            binx=c["bin"], biny=c["bin"], pixbinx=c["step"], pixbiny=c["step"], cfx=c["dx"],
                            cfy=c["dy"], background=OFFSET, p=c["p"], q=c["q"], frametime=FRAMETIME,
                            bleach=BLEACH[c["bleach"]], poly_order=c["order"], gls=c["gls"], bayes=c["bayes"],
                            cst=cst)


def _batch_jobs(c):
    """The batch as plan cases, one per (binning, offset)."""
    offsets = ((0, 0), (1, 0), (1, 1))[:c["offsets"]]
    return [{**PLAN, "width": c["width"], "height": c["height"], "frames": c["frames"], "bin": b, "step": b,
             "dx": dx, "dy": dy, "gls": c["gls"]} for b in range(1, c["bins"] + 1) for dx, dy in offsets]


def _calcacf_params(c):
    """The plugin's parameters and the output arrays it hands in."""
    w, h = c["width"] - c["dx"], c["height"] - c["dy"]
    ch, num = 73, c["frames"]
    lag, samp = engine.lag_tables(16, 8)
    p = _lib.ACFParameters(width=w, height=h, win_star=c["width"], hin_star=c["height"], w_temp=c["width"],
                           h_temp=c["height"], pixbinX=1, pixbinY=1, binningX=1, binningY=1, firstframe=1,
                           lastframe=num, framediff=num, cfXDistance=c["dx"], cfYDistance=c["dy"], correlatorp=16.0,
                           correlatorq=8.0, frametime=FRAMETIME, background=0, mtab1=float(num - 1),
                           mtabchanumminus1=float((num - int(lag[-1])) // int(samp[-1])),
                           sampchanumminus1=float(samp[-1]), chanum=ch, isNBcalculation=0, bleachcorr_gpu=0,
                           bleachcorr_order=0, nopit=min(num, 1000), ave=num // min(num, 1000))
    out = {"pixels1": np.zeros((ch, h, w)), "blockvararray": np.zeros((ch, h, w)), "NBmean": np.zeros((h, w)),
           "NBcov": np.zeros((h, w)), "blocked1D": np.zeros((2, h, w)), "samp": np.zeros(ch),
           "lag": np.zeros(ch, np.int32)}
    return p, out


def _curves(c, seed):
    """ACF curves of a TIRF recording: N, D, G log-uniform, noise of about 1 % at lag 1, float32."""
    rng = np.random.default_rng(seed)
    n, npts = c["fits"], c["points"]
    lag, _ = engine.lag_tables(16, 8)
    tau = lag[1:1 + npts] * FRAMETIME
    N = np.exp(rng.uniform(math.log(0.5), math.log(20.0), n))
    D = np.exp(rng.uniform(math.log(0.2), math.log(5.0), n))
    G = rng.normal(0.0, 1e-3, n) / N
    cst = _constants(1, 0, 0, TIRF_SZ_UM)
    a, _ = _lateral(torch.tensor(D)[:, None], torch.tensor(tau)[None], cst)
    sd = 0.01 / N[:, None] / np.sqrt(1 + np.arange(npts) / 8.0)[None]
    y = a.numpy() / N[:, None] + G[:, None] + rng.normal(0.0, 1.0, (n, npts)) * sd
    return tau.astype(np.float32), y.astype(np.float32), (1.0 / sd ** 2).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plan":
        cfg = _config(case)
        plan = engine.Plan(cfg)
        return {"kind": kind, "stack": _stack(case["width"], case["height"], cfg.frames, case["bleach"], seed),
                "plan": plan, "out": plan.alloc_device_outputs()}
    if kind == "batch":
        batch = engine.Batch([_config(j) for j in _batch_jobs(case)], lanes=4)
        return {"kind": kind, "stack": _stack(case["width"], case["height"], case["frames"], "none", seed),
                "batch": batch, "out": batch.alloc_device_outputs()}
    if kind == "calcacf":
        s = _stack(case["width"], case["height"], case["frames"], "none", seed)
        pixels = (s.view(torch.int16) - OFFSET).float().cpu().numpy()
        p, out = _calcacf_params(case)
        return {"kind": kind, "pixels": pixels, "params": p, "out": out}
    tau, y, w = _curves(case, seed)
    fm = FitModel(case["fits"], case["points"], True, Model.ACF_1D, tolerance=1e-16, maxNumberIterations=2000,
                  parametersToFit=[i in (0, 1, 4) for i in range(20)], userInfoSize=4 * case["points"])
    fm.data[:] = y.reshape(-1)
    fm.weights[:] = w.reshape(-1)
    fm.userInfo[:] = tau
    init = fm.initialParameters.reshape(case["fits"], 20)
    init[:, 0], init[:, 1] = 1.0, 1e-12
    init[:, 11:] = engine.model_constants(pixel_um=PIXEL_UM, psf_um=PSF_UM)
    return {"kind": kind, "model": fm, "result": FitResult(case["fits"], 20)}


def run(state):
    kind = state["kind"]
    if kind == "plan":
        return state["plan"].execute(state["stack"], state["out"])
    if kind == "batch":
        return state["batch"].execute(state["stack"], state["out"])
    if kind == "calcacf":
        o = state["out"]
        GpufitImFCS.calcACF(state["pixels"], o["pixels1"], o["blockvararray"], o["NBmean"], o["NBcov"],
                            o["blocked1D"], None, o["samp"], o["lag"], state["params"])
        return o
    r = GpufitImFCS.fit(state["model"], state["result"])
    return {"parameters": r.parameters, "states": r.states, "chiSquares": r.chiSquares,
            "numberIterations": r.numberIterations}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _plan_work(c, stack_read=True):
    cfg = _config(c)
    n, ch, num = cfg.npix, cfg.chanum, cfg.num
    n1 = ch - 1
    byt = 2.0 * cfg.width * cfg.height * num * stack_read
    byt += n * (3 * 8.0 * ch + 2 * 4 + 2 * 8 + 11 * 4 + 4 + 4 + 4 + (8 if c["bayes"] else 0))
    # products: p + 1 lags of the frames, p / 2 lags of each binned level
    flops = 2.0 * n * num * (c["p"] + 1 + c["p"] / 2 * (1 - 0.5 ** (c["q"] - 1)))
    if c["gls"]:
        byt += 8.0 * n * n1 * n1
        flops += n * (2.0 * n1 * n1 * (num >> 7) + n1 ** 3 / 3.0 + n1 ** 3 / 3.0)
    return byt, flops


def work(case):
    kind = case["kind"]
    if kind == "plan":
        b, f = _plan_work(case)
    elif kind == "batch":
        jobs = [_plan_work(j, i == 0) for i, j in enumerate(_batch_jobs(case))]
        b, f = sum(x for x, _ in jobs), sum(x for _, x in jobs)
    elif kind == "calcacf":
        px = (case["width"] - case["dx"]) * (case["height"] - case["dy"])
        b = 4.0 * case["width"] * case["height"] * case["frames"] + px * (2 * 8.0 * 73 + 4 * 8)
        f = 2.0 * px * case["frames"] * (17 + 8 * (1 - 0.5 ** 7))
    else:
        b = case["fits"] * (2 * 4.0 * case["points"] + 2 * 4 * 20 + 12)
        f = case["fits"] * case["points"] * 10 * 60.0      # some ten evaluations of the model and its gradient
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _constants(binning, dx, dy, sz_um):
    """Model constants in um: window edge, PSF radius, axial extent, offsets, normalisation."""
    a, s = PIXEL_UM * binning, PSF_UM
    sq = math.sqrt(3.14159265359)
    px = s / sq * (2 * math.exp(-(a / s) ** 2) - 2) + 2 * a * math.erf(a / s)
    vol = 4 * a ** 4 / (px * px)
    return {"a": a, "s": s, "sz": sz_um, "rx": a * dx / binning, "ry": a * dy / binning,
            "norm": vol / (4 * a ** 4)}


def _lateral(D, tau, c):
    """N-free part of the one-component model and its derivative by D."""
    p0 = torch.sqrt(4 * D * tau + c["s"] ** 2)
    isq = 1 / math.sqrt(math.pi)

    def axis(r):
        p1, p2, p3 = c["a"] + r, c["a"] - r, r
        m = torch.expm1(-(p1 / p0) ** 2) + torch.expm1(-(p2 / p0) ** 2) - 2 * torch.expm1(-(p3 / p0) ** 2)
        e = p1 * torch.erf(p1 / p0) + p2 * torch.erf(p2 / p0) - 2 * p3 * torch.erf(p3 / p0)
        return p0 * isq * m + e, m * isq

    lx, dx = axis(c["rx"])
    ly, dy = (lx, dx) if c["ry"] == c["rx"] else axis(c["ry"])
    ax = 1 / torch.sqrt(1 + 4 * D * tau / c["sz"] ** 2)
    lat = lx * ly * c["norm"]
    dlat = (dx * ly + lx * dy) * (2 * tau / p0) * c["norm"]
    return lat * ax, dlat * ax - lat * 2 * tau / c["sz"] ** 2 * ax ** 3


def _least_squares(fun, y, p, iterations, bounded=()):
    """Batched Levenberg-Marquardt: fun(p) -> (values, Jacobian); parameters `bounded` stay >= 0."""
    k = p.shape[1]
    f, J = fun(p)
    r = y - f
    chi = (r * r).sum(1)
    lam = torch.full_like(chi, 1e-3)
    for _ in range(iterations):
        A = J.transpose(1, 2) @ J
        g = (J.transpose(1, 2) @ r[:, :, None])[:, :, 0]
        sc = 1 / torch.sqrt(torch.diagonal(A, dim1=1, dim2=2).clamp_min(1e-300))
        M = A * sc[:, :, None] * sc[:, None, :]
        M = M + lam[:, None, None] * torch.eye(k, dtype=M.dtype, device=M.device)
        M = torch.where(torch.isfinite(M), M, torch.zeros_like(M))
        h = torch.linalg.solve_ex(M, (g * sc)[:, :, None])[0][:, :, 0] * sc
        pn = p + h
        for b in bounded:
            pn[:, b] = pn[:, b].clamp_min(0.0)
        fn, Jn = fun(pn)
        rn = y - fn
        cn = (rn * rn).sum(1)
        ok = cn <= chi
        p = torch.where(ok[:, None], pn, p)
        r = torch.where(ok[:, None], rn, r)
        J = torch.where(ok[:, None, None], Jn, J)
        chi = torch.where(ok, cn, chi)
        lam = torch.where(ok, lam * 0.1, lam * 10).clamp(1e-14, 1e14)
    return p, chi


def _fit(y, w, tau, c, white=None, iterations=80):
    """Least-squares N, D (um^2/s), G from 1, 1, 0; white: L^-1 of each curve's covariance."""
    sw = torch.sqrt(w) if w is not None else torch.ones_like(y)

    def fun(p):
        a, da = _lateral(p[:, 1:2], tau[None], c)
        f = a / p[:, :1] + p[:, 2:3]
        J = torch.stack([-a / p[:, :1] ** 2, da / p[:, :1], torch.ones_like(a)], 2)
        if white is not None:
            return (white @ f[:, :, None])[:, :, 0], white @ J
        return f * sw, J * sw[:, :, None]

    p0 = torch.tensor([1.0, 1.0, 0.0], dtype=y.dtype, device=y.device).repeat(len(y), 1)
    return _least_squares(fun, (white @ y[:, :, None])[:, :, 0] if white is not None else y * sw, p0, iterations)


def _windows(stack, c, x0, y0, ow, oh):
    """Binned window sums less background, [frames][pixels] int64, of windows starting at (x0, y0)."""
    t = stack[c["first"]:].view(torch.int16)[:, y0:y0 + (oh - 1) * c["step"] + c["bin"]].to(torch.int32)
    acc = 0
    for k in range(c["bin"]):
        for i in range(c["bin"]):
            acc = acc + t[:, k:k + (oh - 1) * c["step"] + 1:c["step"],
                          x0 + i:x0 + i + (ow - 1) * c["step"] + 1:c["step"]]
    return acc.reshape(t.shape[0], -1) - OFFSET * c["bin"] ** 2


def _exp_curve(p, t):
    """f0 - sum s (1 - e^{-kt}) / k and its gradient, p = (f0, s1, k1, ...)."""
    f, cols = p[:, :1].expand(-1, t.shape[0]).clone(), [torch.ones((len(p), t.shape[0]), dtype=p.dtype, device=p.device)]
    for m in range((p.shape[1] - 1) // 2):
        s, k = p[:, 1 + 2 * m:2 + 2 * m], p[:, 2 + 2 * m:3 + 2 * m]
        x = k * t[None]
        small = x < 1e-3
        ks = torch.where(k > 0, k, torch.ones_like(k))
        u = torch.where(small, t * (1 - x / 2 + x ** 2 / 6 - x ** 3 / 24 + x ** 4 / 120), -torch.expm1(-x) / ks)
        du = torch.where(small, -t ** 2 * (0.5 - x / 3 + x ** 2 / 8 - x ** 3 / 30 + x ** 4 / 144),
                         (t * torch.exp(-x) - u) / ks)
        f = f - s * u
        cols += [-u, -s * du]
    return f, torch.stack(cols, 2)


def _corrected(v, c):
    """Bleach-corrected values, [frames][pixels] float64, from the averaged traces' fits."""
    num = v.shape[0]
    nopit = min(num, 1000)
    ave = num // nopit
    x = v.to(torch.float64)
    if c["bleach"] == "none":
        return x
    tr = torch.div(v[:nopit * ave].reshape(nopit, ave, -1).sum(1), ave, rounding_mode="trunc").to(torch.float64).T
    t = FRAMETIME * (torch.arange(nopit, dtype=torch.float64, device=v.device) + 0.5) * ave
    tt = FRAMETIME * (torch.arange(1, num + 1, dtype=torch.float64, device=v.device) + 0.5)
    tmax = float(t[-1])
    if c["bleach"] == "poly":
        def basis(z):
            u = z / tmax * 2 - 1
            b = [torch.ones_like(u), u]
            for n in range(1, c["order"]):
                b.append(2 * u * b[-1] - b[-2])
            return torch.stack(b[:c["order"] + 1], 1)
        B = basis(t)
        coef = torch.linalg.solve(B.T @ B, B.T @ tr.T)              # [order + 1][pixels]
        f, f0 = basis(tt) @ coef, (basis(torch.zeros(1, dtype=t.dtype, device=t.device)) @ coef)
        return x / torch.sqrt(f / f0) + f0 * (1 - torch.sqrt(f / f0))
    z, ym = t / tmax, tr.abs().max(1, keepdim=True)[0]
    y = tr / ym
    # start at the best rate of a grid, the amplitudes solved for
    k = torch.cat([torch.zeros(1), 10 ** (-3 + 7 * torch.arange(96) / 95.0)]).to(t)
    E = torch.exp(-k[:, None] * z[None])
    E[0] = z
    E = E - E.mean(1, keepdim=True)
    yc = y - y.mean(1, keepdim=True)
    j = ((yc @ E.T) ** 2 / (E * E).sum(1)[None]).argmax(1)
    c1 = (yc * E[j]).sum(1) / (E[j] ** 2).sum(1)
    c0 = y.mean(1) - c1 * torch.where(j[:, None] == 0, z[None], torch.exp(-k[j][:, None] * z[None])).mean(1)
    zero = j == 0
    p = torch.stack([torch.where(zero, c0, c0 + c1), torch.where(zero, -c1, c1 * k[j]), k[j]], 1)
    p = _least_squares(lambda q: _exp_curve(q, z), y, p, 60, bounded=(2,))[0]
    out = torch.empty_like(x)
    for i in range(0, x.shape[1], 256):
        f = (_exp_curve(p[i:i + 256], tt / tmax)[0] * ym[i:i + 256]).T
        f0 = (p[i:i + 256, 0] * ym[i:i + 256, 0])[None]
        out[:, i:i + 256] = x[:, i:i + 256] / torch.sqrt(f / f0) + f0 * (1 - torch.sqrt(f / f0))
    return out


def _lags(p, q):
    """Lag (frames) and bin width of every channel."""
    lag, samp = list(range(p + 1)), [1] * (p + 1)
    for k in range(1, q):
        lag += [(p // 2 + y) << k for y in range(1, p // 2 + 1)]
        samp += [1 << k] * (p // 2)
    return lag, samp


def _halve(v):
    n = v.shape[0] // 2
    return v[0:2 * n:2] + v[1:2 * n:2]


def _block_index(c0, c1, q):
    """Blocking transform: the block index of each pixel."""
    num, npix = c0.shape
    zero = torch.zeros((1, npix), dtype=c0.dtype, device=c0.device)
    d, e = torch.cat([zero, c0[:num - 2]]), c1[:num - 1]
    dm, Dm = d.mean(0), e.mean(0)
    pr = (d - dm) * (e - Dm)
    blocknum = int(math.floor(math.log2(num - 1))) - 2
    sd, err = [], []
    for _ in range(blocknum):
        n = pr.shape[0]
        v = ((pr * pr).mean(0) - pr.mean(0) ** 2) / (n * (dm * Dm) ** 2)
        sd.append(torch.sqrt(v))
        err.append(sd[-1] / math.sqrt(2 * (n - 1)))
        pr = _halve(pr) / 2
    sd, err = torch.stack(sd).cpu().numpy(), torch.stack(err).cpu().numpy()
    up, lo = sd + err, sd - err
    B = blocknum
    crt = (up[:-1] > lo[1:]) & (up[1:] > lo[:-1])
    cr12 = np.zeros((B, npix), bool)
    cr12[:B - 2] = crt[:-1] & crt[1:]
    pos = sd[1:] > sd[:-1]
    cr3 = np.zeros((B, npix), bool)
    cr3[:B - 2] = pos[:-1] & pos[1:]
    ind = np.zeros(npix, np.int64)
    for i in range(npix):
        last = max([x for x in range(B - 2) if cr3[x, i] and not cr12[x, i]], default=0)
        ok = cr12[:, i].copy()
        ok[:last + 1] = False
        ok[B - 4:B - 2] = False
        found = [x + 1 for x in range(1, B - 4) if ok[x]]
        ind[i] = max(found[0] if found else (B - 3 if B > 3 else B - 1), q - 1)
    return torch.tensor(ind, device=c0.device)


def _covariance(bp):
    """Shrunk covariance of the blocked products [pixels][lags][blocks], with the plugin's accumulation."""
    npx, n1, pn = bp.shape
    m = bp.mean(2)
    e = bp - m[:, :, None]
    cov = e @ e.transpose(1, 2) / (pn - 1)
    var = torch.diagonal(cov, dim1=1, dim2=2)
    med = torch.sort(torch.cat([torch.zeros_like(var[:, :1]), var], 1), 1)[0]
    med = 0.5 * (med[:, n1 // 2] + med[:, (n1 + 1) // 2])
    f = pn / (pn - 1.0) ** 3
    num = (((e * e - var[:, :, None]) ** 2).sum(2) * f).sum(1)
    lv = (num / ((var - med[:, None]) ** 2).sum(1)).clamp(0, 1)
    z = e / torch.sqrt(var)[:, :, None]
    cor = cov / torch.sqrt(var[:, :, None] * var[:, None, :])
    z2 = z * z
    t = z2 @ z2.transpose(1, 2) - 2 * cor * (z @ z.transpose(1, 2)) + pn * cor * cor
    num = torch.zeros(npx, dtype=bp.dtype, device=bp.device)
    for x in range(1, n1):
        T = torch.zeros_like(num)
        for y in range(x):
            T = (T + t[:, x, y]) * f
            num = num + T
    den = (torch.tril(cor, -1) ** 2).sum((1, 2))
    lc = (num / den).clamp(0, 1)
    d = lv[:, None] * med[:, None] + (1 - lv[:, None]) * var
    out = (1 - lc)[:, None, None] * cor * torch.sqrt(d[:, :, None] * d[:, None, :]) / pn
    out.diagonal(dim1=1, dim2=2).copy_(d / pn)
    return out


def _correlate(c0, c1, c, fitted=True):
    """Outputs of a plan for the corrected values c0 (direct) and c1 (displaced), [frames][pixels]."""
    p, q, num = c["p"], c["q"], c0.shape[0]
    lag, samp = _lags(p, q)
    ch, npix = len(lag), c0.shape[1]
    ind = _block_index(c0, c1, q)
    pn_of = {int(i): int(((num - lag[-1]) // samp[-1]) / 2 ** max(int(i) - (q - 1), 0)) for i in torch.unique(ind)}
    acf, var = (torch.empty((npix, ch), dtype=c0.dtype, device=c0.device) for _ in range(2))
    nbm = nbc = None
    blocks = {i: torch.empty((int((ind == i).sum()), ch, pn), dtype=c0.dtype, device=c0.device)
              for i, pn in pn_of.items()} if c["gls"] else {}
    a, b, level = c0, c1, 0
    for x in range(ch):
        while (1 << level) < samp[x]:
            a, b, level = _halve(a), _halve(b), level + 1
        d = lag[x] // samp[x]
        n = a.shape[0] - d
        dm, Dm = a[:n].mean(0), b[d:].mean(0)
        pr = (a[:n] - dm) * (b[d:] - Dm)
        acf[:, x] = pr.mean(0) / (dm * Dm)
        if x == 1:
            nbm, nbc = dm, pr.mean(0)
        for i, pn in pn_of.items():
            at = ind == i
            L = 1 << max(i - level, 0)
            z = pr[:pn * L, at].reshape(pn, L, -1).mean(1)
            nn = dm[at] * Dm[at]
            var[at, x] = ((z * z).mean(0) - z.mean(0) ** 2) / ((pn - 1) * nn * nn)
            if c["gls"]:
                blocks[i][:, x] = (z / nn).T
    out = {"acf": acf, "var": var, "sd": torch.sqrt(var), "nb_mean": nbm, "nb_cov": nbc}
    tau = torch.tensor(lag[1:], dtype=c0.dtype, device=c0.device) * FRAMETIME
    cst = _constants(c["bin"], c["dx"], c["dy"], c["sz_um"])
    if c["gls"]:
        cov = torch.empty((npix, ch - 1, ch - 1), dtype=c0.dtype, device=c0.device)
        for i in pn_of:
            cov[ind == i] = _covariance(blocks[i][:, 1:])
            acf[ind == i] = blocks[i].mean(2)
        acf[:, 0] = 0
        out["covmats"] = cov
        L, info = torch.linalg.cholesky_ex(cov)
        good = (info == 0) & (torch.diagonal(L, dim1=1, dim2=2) ** 2 > 1e-10).all(1)
        L[~good] = torch.eye(ch - 1, dtype=L.dtype, device=L.device)
        white = torch.linalg.solve_triangular(L, torch.eye(ch - 1, dtype=L.dtype, device=L.device).expand_as(L),
                                              upper=False)
        par, chi = _fit(acf[:, 1:], None, tau, cst, white)
        chi = chi / (ch - 3 - 1)
    else:
        par, chi = _fit(acf[:, 1:], 1 / var[:, 1:], tau, cst)
        chi = chi / (ch - 2 - 3 - 1)
        good = torch.isfinite(chi)
    fr = torch.zeros((npix, 11), dtype=c0.dtype, device=c0.device)
    fr[:, 0], fr[:, 1], fr[:, 4] = par[:, 0], par[:, 1] * 1e-12, par[:, 2]
    for i in (0, 1, 4):
        fr[~good, i] = math.nan
    out["fitres"], out["chi2"] = fr, torch.where(good, chi, torch.full_like(chi, math.nan))
    return out


def _plan_exact(c, stack):
    ow = (c["width"] - c["dx"] - c["bin"]) // c["step"] + 1
    oh = (c["height"] - c["dy"] - c["bin"]) // c["step"] + 1
    rows = max(1, min(oh, int(1.2e8 // (ow * c["frames"]))))
    parts = []
    for r in range(0, oh, rows):
        n = min(rows, oh - r)
        v0 = _windows(stack, c, 0, r * c["step"], ow, n)
        c0 = _corrected(v0, c)
        c1 = _corrected(_windows(stack, c, c["dx"], r * c["step"] + c["dy"], ow, n), c) if c["dx"] or c["dy"] else c0
        parts.append(_correlate(c0, c1, c))
    return {k: torch.cat([o[k] for o in parts]) for k in parts[0]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "plan":
        # bayes_prob has no such value: the minimum of a two-component fit to one component is not determined;
        # nor have the outputs behind a double-exponential correction, whose two rates noise leaves undetermined
        if case["bleach"] == "exp2":
            return None
        stack = _stack(case["width"], case["height"], case["first"] + case["frames"], case["bleach"], seed)
        return _plan_exact(case, stack)
    if kind == "batch":
        stack = _stack(case["width"], case["height"], case["frames"], "none", seed)
        return [_plan_exact(j, stack) for j in _batch_jobs(case)]
    if kind == "calcacf":
        c = {**PLAN, **{k: case[k] for k in ("width", "height", "frames", "dx", "dy")}}
        o = _plan_exact(c, _stack(case["width"], case["height"], case["frames"], "none", seed))
        lags = {"pixels1": o["acf"].T.contiguous(), "blockvararray": o["var"].T.contiguous()}
        return {**lags, "NBmean": o["nb_mean"], "NBcov": o["nb_cov"]}
    tau, y, w = (torch.tensor(v, dtype=torch.float64) for v in _curves(case, seed))
    if torch.cuda.is_available():
        tau, y, w = tau.cuda(), y.cuda(), w.cuda()
    par, chi = _fit(y, w, tau, _constants(1, 0, 0, TIRF_SZ_UM))
    full = torch.zeros((len(y), 20), dtype=y.dtype, device=y.device)
    full[:, 0], full[:, 1], full[:, 4] = par[:, 0], par[:, 1] * 1e-12, par[:, 2]
    c = _constants(1, 0, 0, TIRF_SZ_UM)
    full[:, 11:] = torch.tensor([c["a"] * 1e-6, c["a"] * 1e-6, c["s"] * 1e-6, c["sz"] * 1e-6, 0.0, 0.0,
                                 c["norm"] * 4 * c["a"] ** 4 * 1e-12, 1.0, 1.0])
    return {"parameters": full.reshape(-1), "chiSquares": chi}
