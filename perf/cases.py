"""The work that a user of the engine has it do, as cases that can be timed
and compared: model signals, loss gradients, askAdam fits, dictionary starting
points and posterior sampling, from a slice of a few thousand voxels to whole
volumes.  Sizes, protocols and parameter distributions are those of the
package's phantoms, benchmark and tests.

Calls go through the C interface with device arrays, as a pipeline that keeps
its volumes on the GPU makes them, except for the kinds `map` and `sample`,
which are the calls of the model and sampler classes on host arrays.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from gacelle_b200 import Context, _lib, phantoms
from gacelle_b200 import askadam_solver, mcmc_solver
from gacelle_b200.models import _GxModelHandle, gpuR2starMapping

NAMES = {"r2s": ["M0", "R2star"], "r1r2s": ["M0", "R1", "R2star"], "nexi": ["fa", "Da", "De", "ra"],
         "nexi2": ["fa", "Da", "De", "ra", "p2"]}
TINY = 2.220446049250313e-16
BOUNDS = {"r2s": ([0.0, 0.1], [2.0, 200.0]), "r1r2s": ([0.0, 0.1, 0.1], [2.0, 10.0, 200.0]),
          "nexi": ([TINY, TINY, TINY, 1 / 250], [1.0, 3.0, 3.0, 1.0]),
          "nexi2": ([TINY, TINY, TINY, 1 / 250, TINY], [1.0, 3.0, 3.0, 1.0, 1.0])}
START = {"r2s": [1.0, 30.0], "r1r2s": [1.0, 1.0, 30.0], "nexi": [0.4, 2.0, 1.0, 0.05],
         "nexi2": [0.4, 2.0, 1.0, 0.05, 0.3]}
SIGMA = {"r2s": 0.01, "r1r2s": 0.01, "nexi": 0.02, "nexi2": 0.02}
SHELLS = phantoms.nexi_shells()


def listed():
    return [
        # the signal of one slice's maps: the smallest call, launch and wait
        {"name": "signal_slice", "kind": "signal", "model": "r2s", "nvox": 4096, "nx": 0},
        # one loss and gradient, for a caller with an optimiser of its own
        {"name": "gradient_r1r2s", "kind": "gradient", "model": "r1r2s", "nvox": 230_000, "nx": 0, "loss": "mse"},
        # the single-slice R2* fit
        {"name": "fit_r2s_slice", "kind": "fit", "model": "r2s", "nx": 64, "ny": 64, "nz": 1, "loss": "mse",
         "iters": 2000, "tv": 0.0},
        # the whole-volume R2* fit with 3-D total variation
        {"name": "fit_r2s_volume_tv", "kind": "fit", "model": "r2s", "nx": 128, "ny": 128, "nz": 64, "loss": "mse",
         "iters": 4000, "tv": 1e-3},
        # the model class on host images of ragged extents, with the default stopping criteria watching
        {"name": "map_r2s_ragged", "kind": "map", "nx": 61, "ny": 75, "nz": 37, "iters": 1000, "tv": 1e-4},
        # six subjects' masked volumes of uneven size in one call, with B1 maps
        {"name": "fit_r1r2s_batch", "kind": "batch", "nvox": 1_260_000, "volumes": 6, "iters": 400},
        # NEXI on the vertices of both hemispheres
        {"name": "fit_nexi_surface", "kind": "microstructure", "model": "nexi", "nvox": 328_050, "nodes": 14,
         "loss": "mse", "iters": 100},
        # NEXI with the Rician likelihood and the fine powder average
        {"name": "fit_nexi_rician", "kind": "microstructure", "model": "nexi", "nvox": 100_003, "nodes": 100,
         "loss": "rician", "iters": 40},
        # likelihood starting points of a whole brain
        {"name": "match_nexi", "kind": "match", "nvox": 500_000, "entries": 10_000, "model": "nexi"},
        # the ensemble sampler on NEXI, the posterior summarised and not returned
        {"name": "sample_nexi", "kind": "ensemble", "model": "nexi", "nvox": 20_000, "walkers": 64, "steps": 200,
         "thin": 10, "posterior": False},
        # the ensemble sampler on R2*, the posterior returned as well
        {"name": "sample_r2s", "kind": "ensemble", "model": "r2s", "nvox": 12_013, "walkers": 50, "steps": 500,
         "thin": 20, "posterior": True},
        # the sampler class with its default algorithm (Metropolis-Hastings)
        {"name": "sample_r2s_mh", "kind": "sample", "nvox": 4096, "steps": 10_000, "thin": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["signal", "gradient", "fit", "fit", "map", "batch", "microstructure", "microstructure",
                       "match", "ensemble", "ensemble", "sample"])
    if kind == "signal":
        m = rng.choice(["r2s", "r1r2s", "nexi", "nexi2"])
        return {"kind": kind, "model": m, "nvox": _log(rng, 1000, 600_000), "nx": 14 if m.startswith("nexi") else 0}
    if kind == "gradient":
        m = rng.choice(["r2s", "r1r2s", "nexi", "nexi2"])
        return {"kind": kind, "model": m, "nvox": _log(rng, 1000, 400_000), "nx": 14 if m.startswith("nexi") else 0,
                "loss": rng.choice(["mse", "l2"])}
    if kind == "fit":
        if rng.random() < 0.5:
            return {"kind": kind, "model": "r2s", "nx": _log(rng, 32, 200), "ny": _log(rng, 32, 200),
                    "nz": rng.randint(1, 4), "loss": rng.choice(["mse", "mse", "l1"]), "iters": _log(rng, 400, 2000),
                    "tv": 0.0}
        return {"kind": kind, "model": "r2s", "nx": rng.randint(24, 120), "ny": rng.randint(24, 120),
                "nz": rng.randint(8, 60), "loss": "mse", "iters": _log(rng, 400, 4000), "tv": rng.choice([1e-3, 1e-4])}
    if kind == "map":
        return {"kind": kind, "nx": rng.randint(20, 90), "ny": rng.randint(20, 90), "nz": rng.randint(4, 40),
                "iters": _log(rng, 300, 1500), "tv": rng.choice([1e-3, 1e-4, 0.0])}
    if kind == "batch":
        k = rng.randint(1, 6)
        return {"kind": kind, "nvox": k * _log(rng, 2000, 210_000), "volumes": k, "iters": _log(rng, 100, 400)}
    if kind == "microstructure":
        m = rng.choice(["nexi", "nexi", "nexi2"])
        nodes = rng.choice([14, 14, 100])
        top = 300_000 if nodes == 14 else 80_000
        return {"kind": kind, "model": m, "nvox": _log(rng, 1000, top // (1 if m == "nexi" else 2)), "nodes": nodes,
                "loss": rng.choice(["mse", "rician"]) if m == "nexi" else "mse", "iters": _log(rng, 20, 60)}
    if kind == "match":
        return {"kind": kind, "nvox": _log(rng, 1000, 400_000), "entries": rng.choice([2000, 5000, 10_000, 10_000]),
                "model": rng.choice(["nexi", "nexi", "nexi2"])}
    if kind == "ensemble":
        m = rng.choice(["r2s", "r2s", "r1r2s", "nexi"])
        return {"kind": kind, "model": m, "nvox": _log(rng, 500, 12_000), "walkers": rng.choice([16, 32, 50, 64]),
                "steps": _log(rng, 60, 180) if m == "nexi" else _log(rng, 100, 500), "thin": rng.choice([5, 10, 20]),
                "posterior": rng.random() < 0.5}
    return {"kind": kind, "nvox": _log(rng, 1000, 20_000), "steps": _log(rng, 2000, 8000), "thin": 20}


# ---------------------------------------------------------------------------
# Models in the precision of their inputs, by torch alone.  th: [parameter, voxel]; signals [measurement, voxel].
# ---------------------------------------------------------------------------
def _protocol(model):
    if model == "r2s":
        return {"te": phantoms.R2S_TE}
    if model == "r1r2s":
        return {"te": phantoms.R1R2S_TE, "fa": phantoms.R1R2S_FA, "tr": phantoms.R1R2S_TR}
    return {"b": SHELLS[0], "delta": SHELLS[1]}


def _measurements(model):
    return {"r2s": 12, "r1r2s": 24, "nexi": 24, "nexi2": 48}[model]


def _col(a, like):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=like.device).to(like.dtype)


def _signal(model, th, nodes=14, b1=None):
    P = _protocol(model)
    if model == "r2s":
        te = _col(P["te"], th)[:, None]
        return th[0] * torch.exp(-te * th[1])
    if model == "r1r2s":
        te = _col(P["te"], th)[:, None]
        fa = _col(np.deg2rad(P["fa"]), th)[:, None] * (1.0 if b1 is None else b1)
        E1 = torch.exp(-P["tr"] * th[1])
        A = th[0] * torch.sin(fa) * (1 - E1) / (1 - torch.cos(fa) * E1)
        E2 = torch.exp(-te * th[2])
        return (A[:, None, :] * E2[None, :, :]).reshape(-1, th.shape[1])  # echo times fastest
    eps = 1e-8
    f = th[0].clamp(min=eps)
    x2 = torch.linspace(0, 1, nodes, device=th.device, dtype=th.dtype).square()[:, None]
    w = torch.ones(nodes, device=th.device, dtype=th.dtype)[:, None]
    w[0] = w[-1] = 0.5
    w = w / (nodes - 1)
    S0, S2 = [], []
    for b, D in zip(P["b"], P["delta"]):
        d2 = float(b) * th[2]
        r1 = float(D) * th[3]
        r2 = r1 * f / (1 - f)
        d1 = float(b) * th[1] * x2
        l1 = (r1 + r2 + d2 + d1) / 2
        l2 = (torch.sqrt((r1 - r2 - d2 + d1).square() + 4 * r1 * r2) / 2).clamp(min=eps)
        lm = l1 - l2
        p = (f * d1 + (1 - f) * d2 - lm) / (2 * l2)
        M = p * torch.exp(-(l1 + l2)) + (1 - p) * torch.exp(-lm)
        S0.append((w * M).sum(0).clamp(max=1.0))
        if model == "nexi2":
            S2.append((th[4] * (w * M * (1.5 * x2 - 0.5)).sum(0).abs()).clamp(max=1.0))
    return torch.stack(S0 + S2)


def _chunked(fn, n, size):
    return torch.cat([fn(slice(i, min(i + size, n))) for i in range(0, n, size)], dim=-1)


def _maps(model, n, g):
    """Parameters of n voxels in the distributions of the phantoms."""
    def u(lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    if model == "r2s":
        return torch.stack([u(0.5, 1.5), u(10.0, 60.0)])
    if model == "r1r2s":
        return torch.stack([u(0.5, 2.0), u(0.4, 1.5), u(10.0, 60.0)])
    fa, tex = u(0.1, 0.9), u(2.0, 50.0)
    ra = ((1 - fa) / tex).clamp(min=1 / 240)
    th = [fa, u(1.0, 3.0), u(0.5, 1.5), ra]
    return torch.stack(th + ([u(0.05, 0.5)] if model == "nexi2" else []))


def _data(model, th, g, sigma, rician=False, b1=None):
    n = th.shape[1]
    nodes = 100 if model.startswith("nexi") else 0
    S = _chunked(lambda s: _signal(model, th[:, s], nodes, None if b1 is None else b1[s]), n, 65536)
    r = S + sigma * torch.randn(S.shape, generator=g, device="cuda", dtype=torch.float64)
    if rician:
        r = torch.hypot(r, sigma * torch.randn(S.shape, generator=g, device="cuda", dtype=torch.float64))
    return r.float().contiguous()


def _mask(c):
    """A filled slice, or an ellipsoid that touches the volume's faces."""
    d = (c["nx"], c["ny"], c["nz"])
    return np.ones(d, bool) if c["nz"] < 5 else phantoms.ellipsoid_mask(d, 1.05)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _inputs(c, seed):
    """The case's input arrays, on the GPU (host arrays for `map` and `sample`)."""
    g = _gen(seed)
    k = c["kind"]
    if k in ("signal", "gradient"):
        m = c["model"]
        gt = _maps(m, c["nvox"], g)
        if k == "signal":
            return {"theta": gt.float().contiguous()}
        y = _data(m, gt, g, SIGMA[m])
        spread = 0.8 + 0.4 * torch.rand(gt.shape, generator=g, device="cuda", dtype=torch.float64)
        lb, ub = (_col(v, gt)[:, None] for v in BOUNDS[m])
        return {"y": y, "theta": torch.minimum(torch.maximum(gt * spread, lb * 1.01 + 1e-6), ub * 0.99).float()}
    if k in ("fit", "map"):
        mask = _mask(c)
        idx = np.flatnonzero(mask.ravel(order="F") > 0).astype(np.int32)
        gt = _maps("r2s", idx.size, g)
        y = _data("r2s", gt, g, SIGMA["r2s"])
        if k == "fit":
            return {"y": y, "idx": torch.from_numpy(idx).cuda(), "mask": mask}
        img = np.zeros((mask.size, 12), np.float32)
        img[idx] = y.cpu().numpy().T
        return {"img": img.reshape(mask.shape + (12,), order="F"), "mask": mask}
    if k == "batch":
        w = np.arange(1, c["volumes"] + 1) / (c["volumes"] * (c["volumes"] + 1) / 2)
        sizes = [max(1, int(c["nvox"] * x)) for x in w]
        out = []
        for n in sizes:
            gt = _maps("r1r2s", n, g)
            b1 = (0.8 + 0.4 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).float()
            out.append({"y": _data("r1r2s", gt, g, SIGMA["r1r2s"], b1=b1.double()), "b1": b1})
        return {"volumes": out}
    if k == "microstructure":
        gt = _maps(c["model"], c["nvox"], g)
        return {"y": _data(c["model"], gt, g, SIGMA["nexi"], rician=c["loss"] == "rician")}
    if k == "match":
        m, n = c["model"], c["entries"]
        y = _data(m, _maps(m, c["nvox"], g), g, SIGMA["nexi"])
        iv = [(0.01, 0.99), (1.5, 3.0), (0.5, 1.5), (1.0, 100.0), (0.01, 0.99)]
        p = torch.stack([lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
                         for lo, hi in iv])
        p[3] = (1 - p[0]) / p[3]
        D = _signal(m, p[:4] if m == "nexi" else p, 14).float().contiguous()
        # the engine's weights of the even orders: 1 / (2 l + 1)
        w = None if m == "nexi" else torch.tensor([1.0] * 24 + [0.2] * 24, device="cuda")
        return {"y": y, "dict": D, "w": w}
    m = c.get("model", "r2s")
    gt = _maps(m, c["nvox"], g)
    sig = 0.02
    y = _data(m, gt, g, sig)
    x0 = torch.cat([gt, torch.full((1, c["nvox"]), sig, device="cuda", dtype=torch.float64)]).float().contiguous()
    if k == "ensemble":
        return {"y": y, "x0": x0}
    return {"y": y.cpu().numpy(), "x0": x0.cpu().numpy()}


# ---------------------------------------------------------------------------
# The engine's calls
# ---------------------------------------------------------------------------
def _f(t):
    return C.cast(C.c_void_p(t.data_ptr()), _lib._fp)


def _handle(model, nodes):
    if model == "r2s":
        return _GxModelHandle(_lib.MODEL_R2S, te=phantoms.R2S_TE)
    if model == "r1r2s":
        return _GxModelHandle(_lib.MODEL_R1R2S, te=phantoms.R1R2S_TE, fa_deg=phantoms.R1R2S_FA, tr=phantoms.R1R2S_TR)
    return _GxModelHandle(_lib.MODEL_NEXI, bval=SHELLS[0], delta=SHELLS[1], lmax=2 if model == "nexi2" else 0,
                          nx=nodes or 14)


def _context():
    ctx = Context.default()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _opts(model, c):
    """Every iteration is run: no stopping criterion can end the fit."""
    f = {"iteration": c.get("iters", 0), "initialLearnRate": 0.01, "lossFunction": c["loss"], "tol": -math.inf,
         "patienceConvergence": math.inf, "convergenceStepTol": 0.0, "convergenceGradTol": 0.0,
         "voxelSize": [1, 1, 1]}
    if c["loss"] == "rician":
        f["noiseSigma"] = SIGMA[model]
    if c.get("tv", 0.0) > 0:
        f.update({"lambda": [c["tv"]], "regmap": ["R2star"], "TVmode": "3D"})
    return askadam_solver.build_opts(askadam_solver.check_set_default_basic(f), NAMES[model], *BOUNDS[model])


def _start(model, n):
    return torch.tensor(START[model], device="cuda")[:, None].repeat(1, n).contiguous()


def _volume(y, theta0=None, b1=None, idx=None, dims=None):
    v = _lib.GxVolume()
    v.nvox = y.shape[1]
    for i, d in enumerate(dims or (y.shape[1], 1, 1)):
        v.dims[i] = d
    v.data = _f(y)
    if theta0 is not None:
        v.theta0 = _f(theta0)
    if b1 is not None:
        v.b1 = _f(b1)
    if idx is not None:
        v.grid_index = C.cast(C.c_void_p(idx.data_ptr()), _lib._i32p)
    return v


def prepare(case, seed):
    c, k = case, case["kind"]
    s = dict(_inputs(c, seed), kind=k, case=dict(c))
    m = c.get("model", "r2s" if k != "batch" else "r1r2s")
    if k in ("map", "sample"):
        if k == "map":
            s["model"] = gpuR2starMapping(phantoms.R2S_TE)
            s["fitting"] = {"iteration": c["iters"], "initialLearnRate": 0.01, "lossFunction": "mse", "tol": 1e-8,
                            "convergenceValue": 1e-8, "voxelSize": [1, 1, 1]}
            if c["tv"] > 0:
                s["fitting"].update({"lambda": [c["tv"]], "regmap": ["R2star"], "TVmode": "3D"})
        else:
            s["model"] = gpuR2starMapping(phantoms.R2S_TE)
            s["fitting"] = {"algorithm": "MH", "iteration": c["steps"], "thinning": c["thin"],
                            "modelParams": ["M0", "R2star", "noise"], "lb": s["model"].lb, "ub": s["model"].ub,
                            "xStepSize": s["model"].step, "seed": seed, "metric": ["mean", "std", "median", "iqr"],
                            "returnPosterior": False}
            s["pars0"] = {p: s["x0"][i] for i, p in enumerate(s["fitting"]["modelParams"])}
            s["mask"] = np.ones((1, c["nvox"]), bool)
        torch.cuda.synchronize()
        return s
    s["ctx"], s["handle"] = _context(), _handle(m, c.get("nodes", 14))
    new = lambda *shape, dtype=torch.float32: torch.empty(shape, dtype=dtype, device="cuda")  # noqa: E731
    nm, npar = _measurements(m), len(NAMES[m])
    if k == "signal":
        s["out"] = new(nm, c["nvox"])
    elif k == "gradient":
        s["opts"], s["vol"] = _opts(m, c), _volume(s["y"])
        s["theta"] = s["theta"].contiguous()
        s["gtheta"], s["residual"], s["loss"] = new(npar, c["nvox"]), new(nm, c["nvox"]), C.c_double()
    elif k in ("fit", "microstructure"):
        s["opts"] = _opts(m, c)
        s["th0"] = _start(m, s["y"].shape[1])
        s["vol"] = _volume(s["y"], s["th0"], idx=s.get("idx"), dims=s["mask"].shape if "mask" in s else None)
        s["theta"], s["best"], s["res"] = new(*s["th0"].shape), new(*s["th0"].shape), _lib.GxAskadamResult()
        s["res"].final_theta, s["res"].min_theta = _f(s["theta"]), _f(s["best"])
        if k == "microstructure":
            s["residual"] = new(*s["y"].shape)
            s["res"].final_residual = _f(s["residual"])
    elif k == "batch":
        s["opts"] = _opts(m, dict(c, loss="mse"))
        vs, n = s["volumes"], c["volumes"]
        s["vols"], s["results"] = (_lib.GxVolume * n)(), (_lib.GxAskadamResult * n)()
        for i, v in enumerate(vs):
            v["th0"] = _start(m, v["y"].shape[1])
            v["theta"], v["best"] = new(*v["th0"].shape), new(*v["th0"].shape)
            s["vols"][i] = _volume(v["y"], v["th0"], v["b1"])
            s["results"][i].final_theta, s["results"][i].min_theta = _f(v["theta"]), _f(v["best"])
    elif k == "match":
        s["best"], s["sse"] = new(c["nvox"], dtype=torch.int32), new(c["nvox"])
    elif k == "ensemble":
        lb, ub = BOUNDS[m]
        # the noise level is known: pinned for NEXI, sampled otherwise
        lo, hi = (0.02, 0.02) if m == "nexi" else (0.001, 0.1)
        s["lb"], s["ub"] = np.array(lb + [lo]), np.array(ub + [hi])
        o = _lib.GxMcmcOpts()
        o.algorithm, o.iteration, o.thinning, o.burnin, o.repetition = 1, c["steps"], c["thin"], 0.2, 1
        o.nwalker, o.step_size, o.start_range, o.seed = c["walkers"], 2.0, 0.001, seed
        o.lb, o.ub = (v.ctypes.data_as(_lib._dp) for v in (s["lb"], s["ub"]))
        s["mopts"] = o
        s["vol"] = _volume(s["y"], s["x0"])
        nv, n = npar + 1, c["nvox"]
        ns = mcmc_solver.number_of_samples({"iteration": c["steps"], "burnin": 0.2, "thinning": c["thin"]})
        s["out"] = {key: new(nv, n) for key in ("mean", "std", "median", "iqr", "mode")}
        if c["posterior"]:
            s["out"]["posterior"] = new(nv, 1, ns, c["walkers"], n)
        s["mres"] = _lib.GxMcmcResult()
        for key, t in s["out"].items():
            setattr(s["mres"], key, _f(t))
    torch.cuda.synchronize()
    return s


def run(s):
    k, L = s["kind"], _lib.lib()
    if k == "map":
        out = s["model"].fit(s["img"], s["mask"], s["fitting"])
        keys = ("M0", "R2star", "loss", "resloss", "residual", "Niteration")
        return {w: {key: out[w][key] for key in keys} for w in ("final", "min")}
    if k == "sample":
        return mcmc_solver.mcmc().optimisation(s["y"], s["mask"], None, s["pars0"], s["fitting"], s["model"])
    ctx, h, dev = s["ctx"].ptr, C.byref(s["handle"].s), _lib.MEM_DEVICE
    if k == "signal":
        _lib.check(L.gx_forward(ctx, h, dev, s["theta"].data_ptr(), None, s["theta"].shape[1], s["out"].data_ptr()))
        return s["out"]
    if k == "gradient":
        _lib.check(L.gx_model_gradient(ctx, h, dev, C.byref(s["vol"]), C.byref(s["opts"]), s["theta"].data_ptr(),
                                       s["gtheta"].data_ptr(), s["residual"].data_ptr(), C.byref(s["loss"]), None,
                                       None))
        return {"gradient": s["gtheta"], "residual": s["residual"], "loss": s["loss"].value}
    if k in ("fit", "microstructure"):
        _lib.check(L.gx_askadam(ctx, h, dev, C.byref(s["vol"]), 1, C.byref(s["opts"]), C.byref(s["res"])))
        r = {"theta": s["theta"], "best": s["best"], "loss": s["res"].final_loss, "best_loss": s["res"].min_loss}
        if k == "microstructure":
            r["residual"] = s["residual"]
        return r
    if k == "batch":
        n = len(s["volumes"])
        _lib.check(L.gx_askadam(ctx, h, dev, s["vols"], n, C.byref(s["opts"]), s["results"]))
        return [{"theta": v["theta"], "best": v["best"], "loss": r.final_loss}
                for v, r in zip(s["volumes"], s["results"])]
    if k == "match":
        _lib.check(L.gx_dictionary_match(ctx, dev, s["y"].data_ptr(), s["y"].shape[1], s["dict"].data_ptr(),
                                         s["dict"].shape[1], s["y"].shape[0],
                                         None if s["w"] is None else s["w"].data_ptr(), s["best"].data_ptr(),
                                         s["sse"].data_ptr()))
        return {"best": s["best"], "sse": s["sse"]}
    _lib.check(L.gx_mcmc(ctx, h, dev, C.byref(s["vol"]), 1, C.byref(s["mopts"]), C.byref(s["mres"])))
    return s["out"]


# ---------------------------------------------------------------------------
# What a pass cannot do without: inputs read once and outputs written once;
# operations of the models and solvers (a multiply-add is two, any other
# function one).
# ---------------------------------------------------------------------------
def _model_ops(model, nodes, backward):
    """Signal of one voxel [and its adjoint]."""
    if model == "r2s":
        return 12 * (8 if backward else 3)
    if model == "r1r2s":
        return 12 * 2 + 24 * (7 if backward else 1) + 30
    per = {"nexi": (22, 52), "nexi2": (25, 70)}[model]
    return 24 * (nodes or 14) * per[1 if backward else 0]


def work(case):
    c, k = case, case["kind"]
    m = c.get("model", "r1r2s" if k == "batch" else "r2s")
    nm, npar = _measurements(m), len(NAMES[m])
    if k in ("signal", "gradient"):
        n = c["nvox"]
        if k == "signal":
            return {"bytes": 4 * n * (npar + nm), "flops": n * _model_ops(m, c["nx"], False)}
        return {"bytes": 4 * n * (2 * npar + 2 * nm), "flops": n * (_model_ops(m, c["nx"], True) + 3 * nm)}
    if k in ("fit", "map", "batch", "microstructure"):
        n = int(_mask(c).sum()) if "ny" in c else c["nvox"]
        step = _model_ops(m, c.get("nodes", 0), True) + npar * 20 + (24 if c.get("tv", 0) > 0 else 0)
        if c.get("loss") == "rician":
            step += 40 * nm
        io = nm + 3 * npar + (1 if k == "batch" or c.get("tv", 0) > 0 else 0)
        if k == "microstructure":
            io += nm
        if k == "map":
            io += 2 * nm
        return {"bytes": 4 * n * io, "flops": n * c["iters"] * step}
    if k == "match":
        n, e = c["nvox"], c["entries"]
        return {"bytes": 4 * (nm * (n + e) + 2 * n), "flops": n * e * (2 * nm * (1 if m == "nexi" else 2) + 4)}
    nv, n, W = npar + 1, c["nvox"], c.get("walkers", 1)
    ns = mcmc_solver.number_of_samples({"iteration": c["steps"], "burnin": 0.2 if k == "ensemble" else 0.1,
                                        "thinning": c["thin"]})
    by = 4 * n * (nm + nv + (5 if k == "ensemble" else 4) * nv) + (4 * n * W * ns * nv if c.get("posterior") else 0)
    return {"bytes": by, "flops": n * W * c["steps"] * (_model_ops(m, 14, False) + 4 * nm + 60)}


# ---------------------------------------------------------------------------
# The same results in 64 bits, by torch alone
# ---------------------------------------------------------------------------
def _loss(S, y, kind, sigma):
    S = torch.where(torch.isfinite(S), S, torch.zeros((), dtype=S.dtype, device=S.device))
    r = S - y
    if kind == "mse":
        return 0.5 * r * r
    if kind == "l2":
        return r * r
    if kind == "l1":
        return r.abs()
    s2 = sigma * sigma
    return r * r / (2 * s2) - torch.log(torch.special.i0e(y * S / s2)) - torch.log(y / s2)


class _Watch:
    """The default stopping criteria (loss average, step and gradient norms), with the class call's tolerances."""

    def __init__(self):
        self.ema = self.least = None
        self.count = [0, 0, 0]

    def stop(self, e, loss, g, z, last):
        first = self.ema is None
        before = loss if first else self.ema
        self.ema = 0.95 * before + 0.05 * loss
        self.least = loss if first else min(self.least, loss)
        still = abs(self.ema - before) / (abs(before) + 1e-8) <= 1e-8 and e > 20 and self.least - loss <= 1e-8
        step = float((z - last).norm() / (1 + z.norm())) < 1e-6
        flat = float(g.norm()) < 1e-6
        self.count = [n + 1 if on else 0 for n, on in zip(self.count, (still, step, flat))]
        return max(self.count) > 5 or loss < 1e-8


def _fit64(model, y, th0, iters, loss, nodes=14, b1=None, tv=0.0, mask=None, idx=None, nvox=None, sigma=0.02,
           watch=False):
    """askAdam in 64 bits: (losses by epoch, final parameters and residuals);
    `nvox`: the voxels over which the mean is taken (of all chunks)."""
    watch = _Watch() if watch else None
    lb, ub = (_col(v, th0)[:, None] for v in BOUNDS[model])
    eb = 1e-4 * (ub - lb)
    t = ((torch.minimum(torch.maximum(th0, lb + eb), ub - eb)) - lb) / (ub - lb)
    z = torch.log(t / (1 - t))
    m1, m2, last = torch.zeros_like(z), torch.zeros_like(z), z
    n = nvox or y.shape[1]
    losses = []
    mk = None if mask is None else torch.from_numpy(mask.copy()).cuda().permute(2, 1, 0).contiguous().double()
    for e in range(1, iters + 1):
        z.requires_grad_(True)
        th = lb + (ub - lb) * torch.sigmoid(z)
        el = _loss(_signal(model, th, nodes, b1), y, loss, sigma)
        tot = el.sum() / (y.shape[0] * n)
        if tv > 0:
            grid = torch.zeros(mk.numel(), device="cuda", dtype=torch.float64).index_put((idx,), th[-1])
            grid = grid.reshape(mk.shape)
            tot = tot + tv / n * sum(((grid.roll(-1, d) - grid).abs() * mk).sum() for d in range(3))
        g, = torch.autograd.grad(tot, z)
        losses.append(float(tot) if len(losses) % 50 == 49 or e == iters else tot.detach())
        z = z.detach()
        if e == iters or (watch and watch.stop(e, float(losses[-1]), g, z, last)):
            break
        last = z
        m1 = 0.9 * m1 + 0.1 * g
        m2 = 0.999 * m2 + 0.001 * g * g
        z = z - 0.01 * (m1 / (1 - 0.9 ** e)) / (torch.sqrt(m2 / (1 - 0.999 ** e)) + 1e-8)
    return [float(x) for x in losses], th.detach(), el.detach()


def _fits64(model, y, th0, c, chunk, **kw):
    """_fit64 in chunks of voxels: final and least-loss results."""
    n = y.shape[1]

    def go(iters):
        out = []
        for i in range(0, n, chunk):
            s = slice(i, i + chunk)
            a = {k: v[s] if k == "b1" else v for k, v in kw.items()}
            out.append(_fit64(model, y[:, s], th0[:, s], iters, nvox=n, **a))
        return np.sum([o[0] for o in out], axis=0), *(torch.cat([o[j] for o in out], dim=1) for j in (1, 2))
    h, th, el = go(c["iters"])
    kw["watch"] = False
    at = int(np.argmin(h))
    best = (h[at], th, el) if at == len(h) - 1 else (h[at], *go(at + 1)[1:])
    return (h[-1], th, el), best


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("ensemble", "sample"):
        return None  # a random walk has no exact value
    m = c.get("model", "r1r2s" if k == "batch" else "r2s")
    w = work(c)["flops"]
    if w > {"microstructure": 6e11}.get(k, 1e13):
        return None  # over the time that such a run may take
    s = _inputs(c, seed)
    if k == "signal":
        th = s["theta"].double()
        return _chunked(lambda q: _signal(m, th[:, q], 14), c["nvox"], 65536)
    if k == "gradient":
        n, y, th = c["nvox"], s["y"].double(), s["theta"].double()
        g, el = [], []
        for i in range(0, n, 32768):
            t = th[:, i:i + 32768].clone().requires_grad_(True)
            e = _loss(_signal(m, t, 14), y[:, i:i + 32768], c["loss"], SIGMA[m])
            g.append(torch.autograd.grad(e.sum() / y.numel(), t)[0])
            el.append(e.detach())
        el = torch.cat(el, dim=1)
        return {"gradient": torch.cat(g, dim=1), "residual": el, "loss": float(el.sum() / el.numel())}
    if k == "fit":
        y = s["y"].double()
        kw = {"loss": c["loss"], "tv": c["tv"], "mask": s["mask"], "idx": s["idx"].long()}
        a, b = _fits64(m, y, _start(m, y.shape[1]).double(), c, y.shape[1], **kw)
        return {"theta": a[1], "best": b[1], "loss": a[0], "best_loss": b[0]}
    if k == "microstructure":
        y = s["y"].double()
        chunk = max(1, 65536 * 14 // c["nodes"])
        a, b = _fits64(m, y, _start(m, y.shape[1]).double(), c, chunk, loss=c["loss"], nodes=c["nodes"],
                       sigma=SIGMA[m])
        return {"theta": a[1], "best": b[1], "loss": a[0], "best_loss": b[0], "residual": a[2]}
    if k == "batch":
        out = []
        for v in s["volumes"]:
            y = v["y"].double()
            a, b = _fits64(m, y, _start(m, y.shape[1]).double(), c, y.shape[1], loss="mse", b1=v["b1"].double())
            out.append({"theta": a[1], "best": b[1], "loss": a[0]})
        return out
    if k == "match":
        y, D = s["y"].double(), s["dict"].double()
        wt = torch.ones(y.shape[0], 1, device="cuda", dtype=torch.float64) if s["w"] is None else s["w"].double()[:, None]
        E, Cw = (D * D).sum(0), (wt * D * D).sum(0)
        sse = []
        for i in range(0, c["nvox"], 20_000):
            q = y[:, i:i + 20_000]
            sc = (q.T @ D) / E
            sse.append(((wt * q * q).sum(0)[:, None] - 2 * sc * ((wt * q).T @ D) + sc * sc * Cw).amin(1))
        return {"best": None, "sse": torch.cat(sse)}
    # map: the class's start point is the closed-form estimate, clamped to the bounds
    mask = s["mask"]
    idx = np.flatnonzero(mask.ravel(order="F") > 0)
    img = s["img"].reshape(-1, 12, order="F")[idx].astype(np.float64)
    te = phantoms.R2S_TE
    area = sum(0.5 * (abs(img[:, j]) + abs(img[:, j + 1])) * (te[j + 1] - te[j]) for j in range(11))
    with np.errstate(divide="ignore", invalid="ignore"):
        r2 = (abs(img[:, 0]) - abs(img[:, -1])) / area
    r2 = np.where(np.isfinite(r2) & (r2 >= 0.1), np.minimum(r2, 200.0), 0.1)
    th0 = np.stack([np.clip(abs(img[:, 0]).astype(np.float32), 0.0, 2.0), np.clip(r2.astype(np.float32), 0.1, 200.0)])
    y, th0 = torch.from_numpy(img.T.copy()).cuda(), torch.from_numpy(th0.astype(np.float64)).cuda()
    a, b = _fits64("r2s", y, th0, c, y.shape[1], loss="mse", tv=c["tv"], mask=mask,
                   watch=True, idx=torch.from_numpy(idx).cuda())

    def image(v):
        x = np.zeros(mask.size)
        x[idx] = v.cpu().numpy()
        return x.reshape(mask.shape, order="F")
    return {key: {"M0": image(r[1][0]), "R2star": image(r[1][1]), "loss": r[0], "resloss": image(r[2].mean(0)),
                  "residual": r[2].cpu().numpy(), "Niteration": None} for key, r in (("final", a), ("min", b))}
