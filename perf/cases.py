"""Measured cases: the work a user of this library has it do, through its
public entry points (milne-eddington_b200/me_b200.py).

Whole calls are inversions of Stokes maps already on the GPU; the others are
the blocks an inversion is made of, each through its own entry point: the
forward synthesis with and without its Jacobian, the 9x9 decompositions, the
learned initialiser's inference and its training.  Spectral lines, grids,
parameter distributions and noise are me_maps'.

Maps are synthesised here in FP64 torch from the seed, so that they do not
depend on the library, and the initialiser that a learned start reads is
trained here too, with torch: a fixed network per line and grid, as a program
keeps one.  exact() restates the synthesis, its derivatives and the network in
64 bits.
"""
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir,
                                "milne-eddington_b200"))
import me_b200  # noqa: E402
import me_maps  # noqa: E402

F64 = torch.float64
LIGHT = 299792458.0
# the map of me_maps that a line's distributions and control file come from
MAP = {"fe15648": "fe15648_1024x1024", "fe6302": "fe6302_2048x1024",
       "fe6173": "fe6173_4096x4096"}
NL = {"fe15648": 60, "fe6302": 112, "fe6173": 6}


def listed():
    return [
        # a small region of interest, the reference's own settings: few pixels,
        # so the latency of a round counts
        {"name": "invert_64x64", "kind": "invert", "line": "fe15648", "nl": 60, "px": 4096,
         "precision": "FP32", "start": "guess", "runs": 1, "fit": False},
        # the headline map with the learned start
        {"name": "invert_learned_1m", "kind": "invert", "line": "fe15648", "nl": 60,
         "px": 1048576, "precision": "FP32", "start": "learned", "runs": 5, "fit": False},
        # the reference's restart schedule on a slit-scan sized piece, ragged
        {"name": "invert_restarts_50k", "kind": "invert", "line": "fe15648", "nl": 60,
         "px": 49999, "precision": "FP32", "start": "guess", "runs": 5, "fit": False},
        # everything in FP64, the long grid with weights, fitted profiles wanted
        {"name": "invert_fp64_fit_8k", "kind": "invert", "line": "fe6302", "nl": 112, "px": 8209,
         "precision": "FP64", "start": "guess", "runs": 1, "fit": True},
        # a filtergram: 6 wavelengths through a 21-point instrument filter
        {"name": "invert_filter_262k", "kind": "invert", "line": "fe6173", "nl": 6, "px": 262144,
         "precision": "FP32", "start": "learned", "runs": 5, "fit": False},
        # forward modelling: a synthetic map
        {"name": "synth_262k", "kind": "synth", "line": "fe15648", "nl": 60, "px": 262144,
         "precision": "FP32", "jac": False},
        # response functions of a model atmosphere set, FP64
        {"name": "synth_jac_fp64_10k", "kind": "synth", "line": "fe6302", "nl": 112, "px": 10007,
         "precision": "FP64", "jac": True},
        # response functions of a few pixels: the smallest call
        {"name": "synth_jac_37", "kind": "synth", "line": "fe15648", "nl": 60, "px": 37,
         "precision": "FP32", "jac": True},
        # the trial step's decomposition, one thread per matrix, normal matrices
        {"name": "svd_u_131k", "kind": "svd_u", "n": 9, "count": 131072, "lanes": 1,
         "fast": True, "matrix": "normal"},
        # the full decomposition with V, as svdcmp gives it
        {"name": "svd_20k", "kind": "svd", "n": 9, "count": 20011, "matrix": "normal"},
        # initial guesses for a map from a trained network
        {"name": "predict_300k", "kind": "predict", "line": "fe15648", "nl": 60, "px": 300007},
        # training a network for a line (a shortened schedule)
        {"name": "train_131k", "kind": "train", "line": "fe15648", "nl": 60, "samples": 131072,
         "batch": 4096, "epochs": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["invert"] * 5 + ["synth"] * 4 + ["svd_u"] * 2 + ["svd", "predict", "train"])
    line = rng.choice(["fe15648", "fe15648", "fe6302", "fe6173"])
    nl = {"fe15648": rng.randint(31, 90), "fe6302": rng.randint(64, 128), "fe6173": 6}[line]
    if kind == "invert":
        precision = rng.choice(["FP32", "FP32", "FP64"])
        start = rng.choice(["guess", "learned"])
        # a drawn map is at most what the listed ones of its kind take
        most = {("FP32", "learned"): 262144, ("FP32", "guess"): 49999,
                ("FP64", "learned"): 32768, ("FP64", "guess"): 8209}[precision, start]
        return {"kind": kind, "line": line, "nl": nl, "px": _log(rng, 512, most),
                "precision": precision, "start": start,
                "runs": rng.choice([1, 2, 5]) if precision == "FP32" else 1,
                "fit": rng.random() < 0.3}
    if kind == "synth":
        jac = rng.random() < 0.6
        return {"kind": kind, "line": line, "nl": nl, "px": _log(rng, 1, 20000 if jac else 200000),
                "precision": rng.choice(["FP32", "FP64"]), "jac": jac}
    if kind == "svd_u":
        return {"kind": kind, "n": rng.choice([9, 9, 9, rng.randint(3, 8)]),
                "count": _log(rng, 64, 131072), "lanes": rng.choice([1, 1, 2, 4, 8, 16, 32]),
                "fast": rng.random() < 0.7, "matrix": rng.choice(["normal", "orthogonal"])}
    if kind == "svd":
        return {"kind": kind, "n": rng.choice([9, 9, rng.randint(3, 8)]),
                "count": _log(rng, 64, 40000), "matrix": rng.choice(["normal", "orthogonal"])}
    if kind == "predict":
        return {"kind": kind, "line": line, "nl": nl, "px": _log(rng, 1, 300007)}
    return {"kind": kind, "line": line, "nl": nl, "samples": _log(rng, 8192, 131072),
            "batch": 256 * rng.randint(4, 24), "epochs": rng.randint(1, 2)}


# --------------------------------------------------------------------------
# the model in FP64
# --------------------------------------------------------------------------
def _grid(line, nl):
    if nl == NL[line]:
        return me_maps.wavelengths(MAP[line])
    lam0, step = (15648.5, 0.04) if line == "fe15648" else (6302.5, 0.0215)
    return lam0 + step * (np.arange(nl) - (nl - 1) / 2.0)


@functools.lru_cache(None)
def _weideman(n):
    """Coefficients of Weideman's rational series for w(z) (SIAM J. Numer. Anal. 31, 1497)."""
    m = 2 * n
    el = math.sqrt(n / math.sqrt(2.0))
    t = el * np.tan(np.arange(-m + 1, m) * np.pi / m / 2)
    f = np.concatenate([[0.0], np.exp(-t * t) * (el * el + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (2 * m)
    return el, a[1:n + 1][::-1].copy()


def _faddeeva(nu, a, terms):
    """w(nu + i a) as (Re, Im), in real arithmetic."""
    el, coef = _weideman(terms)
    dr, di = el + a, -nu                       # d = L - i z
    r = 1.0 / (dr * dr + di * di)
    ir, ii = dr * r, -di * r                   # 1 / d
    zr, zi = (el - a) * ir - nu * ii, (el - a) * ii + nu * ir
    pr, pi = torch.zeros_like(zr), torch.zeros_like(zr)
    for c in coef:
        pr, pi = pr * zr - pi * zi + float(c), pr * zi + pi * zr
    sr, si = ir * ir - ii * ii, 2 * ir * ii
    k = 1.0 / math.sqrt(math.pi)
    return 2 * (pr * sr - pi * si) + ir * k, 2 * (pr * si + pi * sr) + ii * k


def _stokes(line, lam, par, terms=48):
    """The Unno-Rachkovsky solution for a Zeeman triplet: [px][4][len(lam)]."""
    w = me_maps.WORKLOADS[MAP[line]]
    lam0, geff = w["lam0"], w["geff"]
    b, th, ph, v, width, a, eta0, s, beta = (par[:, k:k + 1] for k in range(9))
    x0 = (1e3 * (lam - lam0)[None, :] - 1e6 * v * lam0 / LIGHT) / width
    split = b * (4.6686e-10 * geff * lam0 * lam0) / width
    phi, psi = [], []
    for q in (-1, 0, 1):
        h, l = _faddeeva(x0 + q * split, a + 0 * x0, terms)
        phi.append(h / math.sqrt(math.pi))
        psi.append(l / math.sqrt(math.pi))
    st2, ct = torch.sin(th) ** 2, torch.cos(th)
    c2, s2 = torch.cos(2 * ph), torch.sin(2 * ph)
    half = 0.5 * eta0
    ei = 1 + half * (phi[1] * st2 + 0.5 * (phi[0] + phi[2]) * (1 + ct * ct))
    lin, lin_r = (half * st2 * (f[1] - 0.5 * (f[0] + f[2])) for f in (phi, psi))
    eq, eu, ev = lin * c2, lin * s2, half * ct * (phi[0] - phi[2])
    rq, ru, rv = lin_r * c2, lin_r * s2, half * ct * (psi[0] - psi[2])
    er = eq * rq + eu * ru + ev * rv
    r2 = rq * rq + ru * ru + rv * rv
    det = ei * ei * (ei * ei - eq * eq - eu * eu - ev * ev + r2) - er * er
    s1 = s * (1 - beta) / det
    return torch.stack([
        s * beta + s1 * ei * (ei * ei + r2),
        -s1 * (ei * ei * eq + ei * (ev * ru - eu * rv) + rq * er),
        -s1 * (ei * ei * eu + ei * (eq * rv - ev * rq) + ru * er),
        -s1 * (ei * ei * ev + ei * (eu * rq - eq * ru) + rv * er)], dim=1)


def _profiles(line, nl, par, terms=48):
    """Profiles at the observed wavelengths, through the line's filter where it has one."""
    lam = torch.as_tensor(_grid(line, nl), dtype=F64, device=par.device)
    ctl = me_maps.WORKLOADS[MAP[line]]["ctl"]
    if "filter" not in ctl:
        return _stokes(line, lam, par, terms)
    fwhm, points = (float(t) for t in ctl["filter"].split(","))
    off = torch.linspace(-1.5 * fwhm, 1.5 * fwhm, int(points), dtype=F64, device=par.device)
    g = torch.exp(-off * off / (2 * (fwhm / (2 * math.sqrt(2 * math.log(2)))) ** 2))
    sub = (lam[:, None] + 1e-3 * off[None, :]).reshape(-1)
    y = _stokes(line, sub, par, terms)
    return (y.reshape(par.shape[0], 4, nl, int(points)) * (g / g.sum())).sum(-1)


def _chunks(px, points):
    step = max(1, 8_000_000 // points)
    return [(k, min(px, k + step)) for k in range(0, px, step)]


def _points(line, nl):
    return nl * (21 if line == "fe6173" else 1)


def _parameters(line, px, seed):
    """True parameters of a map's pixels, me_maps' distributions: [px][9]."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(px, 9, generator=g, dtype=F64, device="cuda")
    n = torch.randn(px, generator=g, dtype=F64, device="cuda")
    p = torch.empty(px, 9, dtype=F64, device="cuda")
    lo, hi = {"fe15648": (150.0, 350.0), "fe6302": (60.0, 140.0), "fe6173": (20.0, 50.0)}[line]
    weak = (u[:, 7] < 0.6) if line == "fe6302" else torch.zeros_like(u[:, 7], dtype=torch.bool)
    b_lo, b_hi = (500.0, 3500.0) if line == "fe6302" else (0.0, 3000.0)
    p[:, 0] = torch.where(weak, 200.0 * u[:, 0], b_lo + (b_hi - b_lo) * u[:, 0])
    p[:, 1] = torch.arccos(2 * u[:, 1] - 1)
    p[:, 2] = math.pi * u[:, 2]
    p[:, 3] = 1.5 * n
    p[:, 4] = lo + (hi - lo) * u[:, 3]
    p[:, 5] = 0.1 + 0.7 * u[:, 4]
    p[:, 6] = torch.where(weak, 1 + 9 * u[:, 5], 2 + 28 * u[:, 5])
    p[:, 7] = 1.0
    p[:, 8] = 0.1 + 0.5 * u[:, 6]
    return p


def _map(line, nl, px, seed):
    """Noisy profiles [px][4][nl] of a map."""
    par = _parameters(line, px, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 7919)
    out = torch.randn(px, 4, nl, generator=g, dtype=F64, device="cuda")
    out *= me_maps.WORKLOADS[MAP[line]]["noise"]
    for a, b in _chunks(px, _points(line, nl)):
        out[a:b] += _profiles(line, nl, par[a:b], 24)
    return out


# --------------------------------------------------------------------------
# the learned initialiser's network, trained with torch
# --------------------------------------------------------------------------
def _features(prof):
    """I / I_max - 1 and 10 Q, U, V / I_max of [n][4][nl] profiles, and I_max."""
    imax = prof[:, 0, :].amax(1).clamp_min(0)
    x = prof / imax[:, None, None]
    x = torch.cat([x[:, :1] - 1, 10 * x[:, 1:]], dim=1)
    return x.reshape(prof.shape[0], -1), imax


@functools.lru_cache(None)
def _network(line, nl):
    """(standardisation, weights) of a network for this line and grid, on the host: the
    moments fmean, fistd, tmean, tstd and four layers (W [out][in], b)."""
    n, batch, steps = 131072, 4096, 500
    par = _parameters(line, n, 20240607)
    x, imax = _features(_map(line, nl, n, 20240607))
    t = torch.stack([par[:, 0], torch.cos(par[:, 1]), torch.sin(2 * par[:, 2]),
                     torch.cos(2 * par[:, 2]), par[:, 3], par[:, 4], par[:, 5], par[:, 6],
                     par[:, 8], par[:, 7] / imax], dim=1)
    fm, fs, tm, ts = x.mean(0), x.std(0), t.mean(0), t.std(0)
    x, t = ((x - fm) / fs).float(), ((t - tm) / ts).float()
    sizes = [4 * nl, 256, 256, 256, 10]
    g = torch.Generator(device="cuda").manual_seed(1)
    layers = []
    for i, o in zip(sizes[:-1], sizes[1:]):
        scale = math.sqrt((2.0 if o == 256 else 1.0) / i)
        layers += [torch.randn(o, i, generator=g, device="cuda") * scale,
                   torch.zeros(o, device="cuda")]
    layers = [p.requires_grad_() for p in layers]
    opt = torch.optim.Adam(layers, lr=1e-3)
    order = torch.randperm(n, generator=g, device="cuda")
    for k in range(steps):
        for group in opt.param_groups:
            group["lr"] = 2e-3 * 0.5 * (1 + math.cos(math.pi * k / steps))
        at = order[(k * batch) % n:(k * batch) % n + batch]
        loss = (_mlp(x[at], layers) - t[at]).square().mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
    moments = [m.float().cpu() for m in (fm, 1 / fs, tm, ts)]
    return moments, [p.detach().cpu() for p in layers]


def _mlp(x, layers):
    for k in range(0, 8, 2):
        x = torch.nn.functional.linear(x, layers[k], layers[k + 1])
        if k < 6:
            x = torch.nn.functional.gelu(x)
    return x


def _initialiser(line, nl):
    """The network as the library's Initializer, through its file format."""
    (fm, fi, tm, ts), layers = _network(line, nl)
    nip = (4 * nl + 31) // 32 * 32
    pad = torch.nn.functional.pad
    parts = [pad(fm, (0, nip - 4 * nl)), pad(fi, (0, nip - 4 * nl)), tm, ts]
    for k in range(4):
        w, b = layers[2 * k], layers[2 * k + 1]
        if k == 0:
            w = pad(w, (0, nip - 4 * nl))
        if k == 3:
            w, b = pad(w, (0, 0, 0, 22)), pad(b, (0, 22))
        parts += [w.reshape(-1), b]
    fd, path = tempfile.mkstemp(suffix=".bin")
    with os.fdopen(fd, "wb") as f:
        f.write(b"MEMLP001" + np.array([nl, nip], np.int32).tobytes())
        f.write(torch.cat(parts).numpy().astype(np.float32).tobytes())
    try:
        return me_b200.Initializer.load(path)
    finally:
        os.unlink(path)


# --------------------------------------------------------------------------
# prepare, run
# --------------------------------------------------------------------------
def _plan(case, runs=1):
    extra = {"num_run": str(runs)}
    if case["line"] == "fe6302":
        extra["chisq_criteria"] = "1.5"
    text = me_maps.control_text(MAP[case["line"]], precision=case.get("precision", "FP32"),
                                widen_bounds=case["line"] == "fe15648", extra=extra)
    return me_b200.Plan(me_b200.parse_config_text(text), _grid(case["line"], case["nl"]))


def _matrices(case, seed):
    """Normal matrices J^T J of Jacobians with columns of unequal weight, as the first
    trial of an iteration decomposes, or the orthogonal factors later trials do."""
    n, count = case["n"], case["count"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["matrix"] == "orthogonal":
        q = torch.linalg.qr(torch.randn(count, n, n, generator=g, dtype=F64, device="cuda"))[0]
        return q.contiguous()
    scale = torch.logspace(0, 2, n, dtype=F64, device="cuda")
    out = torch.empty(count, n, n, dtype=F64, device="cuda")
    for a, b in _chunks(count, 60 * n):
        j = torch.randn(b - a, 60, n, generator=g, dtype=F64, device="cuda") * scale
        out[a:b] = j.transpose(1, 2) @ j
    return out


def prepare(case, seed):
    kind = case["kind"]
    zeros = functools.partial(torch.zeros, dtype=F64, device="cuda")
    if kind == "invert":
        s = {"kind": kind, "plan": _plan(case, case["runs"]), "px": case["px"],
             "prof": _map(case["line"], case["nl"], case["px"], seed),
             "res": zeros(case["px"], 10),
             "fit": zeros(case["px"], 4, case["nl"]) if case["fit"] else None}
        if case["start"] == "learned":
            s["init"] = _initialiser(case["line"], case["nl"])
            s["plan"].set_initializer(s["init"])
        return s
    if kind == "synth":
        px, nl = case["px"], case["nl"]
        return {"kind": kind, "plan": _plan(case), "px": px, "jac": case["jac"],
                "par": _parameters(case["line"], px, seed), "prof": zeros(px, 4, nl),
                "d": zeros(px, 4, 9, nl) if case["jac"] else None}
    if kind in ("svd_u", "svd"):
        n, count = case["n"], case["count"]
        s = {"kind": kind, "a": _matrices(case, seed), "u": zeros(count, n, n),
             "w": zeros(count, n), "count": count, "n": n}
        if kind == "svd_u":
            return s | {"lanes": case["lanes"], "fast": case["fast"]}
        return s | {"v": zeros(count, n, n)}
    if kind == "predict":
        return {"kind": kind, "init": _initialiser(case["line"], case["nl"]), "px": case["px"],
                "prof": _map(case["line"], case["nl"], case["px"], seed),
                "par": zeros(case["px"], 9)}
    prior = me_maps.train_prior(MAP[case["line"]])
    return {"kind": kind, "plan": _plan(case),
            "params": me_b200.mlp_train_params(samples=case["samples"], batch=case["batch"],
                                               epochs=case["epochs"], seed=seed + 1, **prior)}


@functools.lru_cache(None)
def _stream():
    """The stream that the program's calls are ordered on."""
    return torch.cuda.Stream()


def run(s):
    kind = s["kind"]
    stream = _stream().cuda_stream
    if kind == "invert":
        s["plan"].carry_chisq = 0.0  # a new map
        s["plan"].invert_device(s["prof"].data_ptr(), s["px"], s["res"].data_ptr(),
                                s["fit"].data_ptr() if s["fit"] is not None else 0, stream)
        return [s["res"]] if s["fit"] is None else [s["res"], s["fit"]]
    if kind == "synth":
        if not s["jac"]:
            s["plan"].synthesize_device(s["par"].data_ptr(), s["px"], s["prof"].data_ptr(), stream)
            return [s["prof"]]
        s["plan"].synthesize_jacobian_device(s["par"].data_ptr(), s["px"], 0.1,
                                             s["prof"].data_ptr(), s["d"].data_ptr(), stream)
        return [s["prof"], s["d"]]
    if kind == "svd_u":
        me_b200.svd_u_device(s["a"].data_ptr(), s["count"], s["n"], s["u"].data_ptr(),
                             s["w"].data_ptr(), s["lanes"], s["fast"], stream)
        return [s["u"], s["w"]]
    if kind == "svd":
        me_b200.svd_device(s["a"].data_ptr(), s["count"], s["n"], s["u"].data_ptr(),
                           s["w"].data_ptr(), s["v"].data_ptr(), stream)
        return [s["u"], s["w"], s["v"]]
    if kind == "predict":
        s["init"].predict_device(s["prof"].data_ptr(), s["px"], s["par"].data_ptr(), stream)
        return [s["par"]]
    with me_b200.Initializer.train(s["plan"], s["params"]) as init:
        return [init.get_params(), init.final_loss]


# --------------------------------------------------------------------------
# work, exact
# --------------------------------------------------------------------------
# Operations of the reference's method per event: a synthesis of one
# wavelength 430, with the Jacobian 1735 and the normal equations 684 more, a
# 9x9 solve 14.4 k.
def work(case):
    kind = case["kind"]
    if kind == "invert":
        # iterations a pixel and trials a pixel that these maps take
        it, tr = {("learned", 1): (6, 11), ("guess", 1): (15, 26)}.get(
            (case["start"], min(case["runs"], 2)),
            (7, 14) if case["start"] == "learned" else (40 + 8 * case["runs"], 75 + 15 * case["runs"]))
        m = _points(case["line"], case["nl"])
        flops = it * (m * 1735 + case["nl"] * 684) + tr * (m * 430 + 14400)
        fit = 32 * case["nl"] if case["fit"] else 0
        return {"bytes": case["px"] * (32 * case["nl"] + 80 + fit), "flops": case["px"] * flops}
    if kind == "synth":
        m = _points(case["line"], case["nl"])
        rows = 40 if case["jac"] else 4
        return {"bytes": case["px"] * (72 + 8 * rows * case["nl"]),
                "flops": case["px"] * m * (1735 if case["jac"] else 430)}
    if kind in ("svd_u", "svd"):
        n, c = case["n"], case["count"]
        full = kind == "svd"
        return {"bytes": c * 8 * (n * n * (3 if full else 2) + n),
                "flops": c * (22000 if full else 14400) * (n / 9) ** 3}
    nip = (4 * case["nl"] + 31) // 32 * 32
    macs = nip * 256 + 2 * 256 * 256 + 256 * 32
    if kind == "predict":
        return {"bytes": case["px"] * (32 * case["nl"] + 72), "flops": case["px"] * 2 * macs}
    n = case["samples"]
    return {"bytes": n * (2 * nip + 40) * (1 + case["epochs"]),
            "flops": n * (430 * _points(case["line"], case["nl"]) + case["epochs"] * 6 * macs)}


def _exact_derivatives(case, par):
    """d S / d p_k times the plan's step of p_k: [px][4][9][nl], forward mode."""
    cfg = me_b200.parse_config_text(me_maps.control_text(MAP[case["line"]]))
    step = [cfg.step[k] for k in range(9)]
    step[7] = 0.1
    out = torch.empty(par.shape[0], 4, 9, case["nl"], dtype=F64, device=par.device)
    ad = torch.autograd.forward_ad
    for k in range(9):
        tangent = torch.zeros_like(par)
        tangent[:, k] = step[k]
        with ad.dual_level():
            y = _profiles(case["line"], case["nl"], ad.make_dual(par, tangent))
            out[:, :, k] = ad.unpack_dual(y).tangent
    return out


def _exact_predict(case, seed):
    (fm, fi, tm, ts), layers = _network(case["line"], case["nl"])
    fm, fi, tm, ts = (m.cuda().double() for m in (fm, fi, tm, ts))
    layers = [p.cuda().double() for p in layers]
    x, imax = _features(_map(case["line"], case["nl"], case["px"], seed))
    t = torch.cat([_mlp((y - fm) * fi, layers) for y in x.split(65536)]) * ts + tm
    phi = 0.5 * torch.atan2(t[:, 2], t[:, 3])
    return torch.stack([t[:, 0].clamp_min(0), torch.arccos(t[:, 1].clamp(-1, 1)),
                        torch.where(phi < 0, phi + math.pi, phi), t[:, 4], t[:, 5], t[:, 6],
                        t[:, 7], t[:, 9] * imax, t[:, 8]], dim=1)


def exact(case, seed):
    if case["kind"] == "synth":
        par = _parameters(case["line"], case["px"], seed)
        prof, jac = [], []
        for a, b in _chunks(case["px"], 2 * _points(case["line"], case["nl"])):
            prof.append(_profiles(case["line"], case["nl"], par[a:b]))
            if case["jac"]:
                jac.append(_exact_derivatives(case, par[a:b]))
        return [torch.cat(prof), torch.cat(jac)] if jac else [torch.cat(prof)]
    if case["kind"] == "predict":
        return [_exact_predict(case, seed)]
    # an inversion's and a training's end, and the order and signs of a
    # decomposition's columns, follow the arithmetic of each step
    return None
