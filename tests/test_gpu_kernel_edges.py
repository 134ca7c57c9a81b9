"""Edges of the kernels' tiles and dispatch rules, each against the FP64 oracle
or a plain restatement: remainders, the smallest and the largest of a range,
and both sides of each rule."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gacelle_b200 import _lib
from gacelle_b200 import askadam_solver as gx_askadam

from helpers import NAMES, bounds, fitting, models, random_theta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["nexi", "nexi2"])
@pytest.mark.parametrize("nx", [2, 3, 127, 128, 129])
def test_nexi_node_table_and_loop(ctx, kind, nx):
    """Signal and gradient around the largest tabulated node count, with odd
    and even counts.  Bars: of the forward and gradient parity tests, the
    signal's relative to the sum of the magnitudes of its trapezoid's terms:
    that is the signal itself for l = 0, and at most p2 times the l = 0 signal
    for the signed l = 2 integral (its weights are at most 1)."""
    rng = np.random.default_rng(nx)
    n = 65
    gxm, om = models(kind, nx=nx)
    lb, ub = bounds(kind)
    th = random_theta(kind, n, rng).astype(np.float32)
    s = oracle.forward(om, th.astype(np.float64))
    out = np.zeros(s.shape, np.float32)
    _lib.check(_lib.lib().gx_forward(ctx.ptr, C.byref(gxm.s), _lib.MEM_HOST, th.ctypes.data, None, n,
                                     out.ctypes.data))
    scale = np.abs(s)
    if kind == "nexi2":
        scale[24:] = np.maximum(scale[24:], th[4] * scale[:24])
    assert np.max(np.abs(out - s) / np.maximum(scale, 1e-3)) < 2e-5
    y = (s + 0.02 * rng.standard_normal(s.shape)).astype(np.float32)
    f = fitting(lossFunction="mse")
    opts = gx_askadam.build_opts(f, NAMES[kind], lb, ub)
    vol = _lib.GxVolume()
    vol.dims[0], vol.dims[1], vol.dims[2] = n, 1, 1
    vol.nvox = n
    vol.data = y.ctypes.data_as(_lib._fp)
    g, loss = np.zeros_like(th), C.c_double()
    _lib.check(_lib.lib().gx_model_gradient(ctx.ptr, C.byref(gxm.s), _lib.MEM_HOST, C.byref(vol), C.byref(opts),
                                            th.ctypes.data, g.ctypes.data, None, C.byref(loss), None, None))
    Lo, go, _, _, _ = oracle.model_gradient(om, oracle.Volume(y.astype(np.float64)), oracle.adam_opts(lb, ub, f),
                                            th.astype(np.float64))
    assert abs(loss.value - Lo) <= 1e-5 * abs(Lo) + 1e-7
    for k in range(th.shape[0]):
        assert np.max(np.abs(g[k] - go[k])) <= 1e-3 * np.max(np.abs(go[k])) + 1e-12


def _r2s_chain(ctx, te, update, nv, W, steps, weights=None, **over):
    from gacelle_b200 import mcmc_solver
    from gacelle_b200.models import gpuR2starMapping
    rng = np.random.default_rng(len(te))
    m = gpuR2starMapping(te)
    th = np.vstack([rng.uniform(0.5, 1.5, nv), rng.uniform(10, 60, nv)])
    y = (th[0] * np.exp(-te[:, None] * th[1]) + 0.02 * rng.standard_normal((len(te), nv))).astype(np.float32)
    x0 = np.vstack([th, np.full(nv, 0.02)]).astype(np.float32)
    f = mcmc_solver.check_set_default_basic(dict({
        "algorithm": "MH" if update == "mh" else "GW", "iteration": steps, "thinning": 1, "burnin": 0.0,
        "Nwalker": W, "Ensembleupdate": "redblack" if update == "redblack" else "simultaneous", "lb": m.lb,
        "ub": m.ub, "xStepSize": m.step, "seed": 9}, **over))
    eng = mcmc_solver.mcmc(ctx)._run(m, y, weights, x0, None, m.modelParams, f, True)
    ref = oracle.mcmc(oracle.r2s(te), oracle.Volume(y.astype(np.float64)), x0.astype(np.float64), m.lb, m.ub,
                      algorithm="MH" if update == "mh" else "ensemble", iteration=steps, thinning=1, burnin=0.0, nwalker=W,
                      seed=9, x_step=m.step, ensemble_update=f["Ensembleupdate"], want_posterior=True)
    return eng["posterior"], ref["posterior"]


@pytest.mark.parametrize("update", ["simultaneous", "redblack", "mh"])
@pytest.mark.parametrize("n_te", [1, 3, 5, 12, 16, 17])
def test_r2s_chain_decisions(ctx, update, n_te):
    """Chains of the screened acceptance (up to 16 echoes) and of the FP64 one
    (17) take the oracle's moves: same draws, so the samples coincide except
    where the signal's FP32 rounding flips a decision (the bar of the sampler
    parity tests, > 97 % over the first steps)."""
    te = np.linspace(2e-3, 40e-3, n_te) if n_te > 1 else np.array([5e-3])
    pe, po = _r2s_chain(ctx, te, update, 33, 1 if update == "mh" else 50, 12)
    assert pe.shape == po.shape
    assert np.mean(np.abs(pe - po) <= 1e-4 * np.abs(po) + 1e-7) > 0.97


@pytest.mark.parametrize("n_te,nvox,steps", [(1, 1, 15), (8, 31, 16), (9, 33, 17), (12, 32, 33), (13, 64, 1),
                                             (16, 65, 160)])
def test_mh_batched_draws(ctx, n_te, nvox, steps):
    """The kernel whose draws are made ahead by other warps takes the moves of
    the plain one (a chosen block size), bit for bit: same draws and same
    decisions.  Steps around a batch of 16, voxels around a warp, echoes around
    the kernels' bounds."""
    from gacelle_b200 import mcmc_solver
    from gacelle_b200.models import gpuR2starMapping
    rng = np.random.default_rng(n_te + steps)
    te = np.linspace(2e-3, 40e-3, n_te)
    m = gpuR2starMapping(te)
    th = np.vstack([rng.uniform(0.5, 1.5, nvox), rng.uniform(10, 60, nvox)])
    y = (th[0] * np.exp(-te[:, None] * th[1]) + 0.02 * rng.standard_normal((n_te, nvox))).astype(np.float32)
    x0 = np.vstack([th, np.full(nvox, 0.02)]).astype(np.float32)
    out = []
    for block in (0, 64):
        f = mcmc_solver.check_set_default_basic({
            "algorithm": "MH", "iteration": steps, "thinning": 1, "burnin": 0.0, "lb": m.lb, "ub": m.ub,
            "xStepSize": m.step, "seed": 4, "repetition": 2, "blockSize": block})
        out.append(mcmc_solver.mcmc(ctx)._run(m, y, None, x0, None, m.modelParams, f, True))
    for key in ("posterior", "mean", "std"):
        assert np.array_equal(out[0][key], out[1][key], equal_nan=True), key


@pytest.mark.parametrize("n_te", [20, 22, 23, 24])
def test_block_near_the_default_shared_memory_limit(ctx, n_te):
    """A 512-thread block whose measurements and staged protocol lie around
    48 KB together runs, and fits what a 128-thread block fits (each voxel's
    arithmetic does not depend on the block)."""
    from helpers import run_engine
    rng = np.random.default_rng(n_te)
    te = np.linspace(2e-3, 40e-3, n_te)
    th = np.vstack([rng.uniform(0.5, 1.5, 700), rng.uniform(10, 60, 700)])
    y = th[0] * np.exp(-te[:, None] * th[1]) + 0.01 * rng.standard_normal((n_te, 700))
    th0 = np.tile(np.array([[1.0], [30.0]], np.float32), (1, 700))
    a, b = (run_engine("r2s", y, th0, fitting(iteration=20, blockSize=n), NAMES["r2s"], context=ctx, te=te)
            for n in (512, 128))
    assert np.array_equal(a["final_theta"], b["final_theta"])


def _match(ctx, y, D, w=None):
    y, D = np.ascontiguousarray(y, np.float32), np.ascontiguousarray(D, np.float32)
    w = None if w is None else np.ascontiguousarray(w, np.float32)
    best, sse = np.full(y.shape[1], -7, np.int32), np.full(y.shape[1], np.nan, np.float32)
    _lib.check(_lib.lib().gx_dictionary_match(ctx.ptr, _lib.MEM_HOST, y.ctypes.data, y.shape[1], D.ctypes.data,
                                              D.shape[1], y.shape[0], None if w is None else w.ctypes.data,
                                              best.ctypes.data, sse.ctypes.data))
    return best, sse


def _scores(y, D, w=None):
    """sse [voxel, entry] in FP64 by the expanded form; NaN for an entry without a norm."""
    y, D = np.asarray(y, np.float32).astype(np.float64), np.asarray(D, np.float32).astype(np.float64)
    w = np.ones((y.shape[0], 1)) if w is None else np.asarray(w, np.float32).astype(np.float64)[:, None]
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        c = (y.T @ D) / (D * D).sum(0)
        return (w * y * y).sum(0)[:, None] - c * (2 * (w * y).T @ D - c * (w * D * D).sum(0))


@pytest.mark.parametrize("nm", [1, 8, 9, 16, 17, 24, 33, 56, 64, 65])
@pytest.mark.parametrize("nvox,entries", [(1, 127), (127, 128), (129, 129), (260, 1000)])
def test_dictionary_tiles(ctx, nm, nvox, entries):
    """Both kernels around their rule (64 measurements, 128 entries) and around
    the 128-row operand tiles, at scales from 1e-20 to 1e20: the entry of least
    FP64 score, or one whose score equals it to 1e-12 of the voxel's energy."""
    rng = np.random.default_rng(nm * 1000 + nvox)
    y = rng.standard_normal((nm, nvox)) * 10.0 ** rng.uniform(-10, 10, nvox)
    D = rng.standard_normal((nm, entries)) * 10.0 ** rng.uniform(-10, 10, entries)
    best, sse = _match(ctx, y, D)
    s = _scores(y, D)
    A = (np.asarray(y, np.float32).astype(np.float64) ** 2).sum(0)
    got = s[np.arange(nvox), best]
    assert np.all(got - s.min(1) <= 1e-12 * A)
    assert np.all(np.abs(sse - got) <= 1e-6 * np.abs(got) + 1e-12 * A)


def test_dictionary_special_values(ctx):
    """Zero voxels take the first entry with a norm, voxels and entries that are
    not numbers match nothing, of equal entries the first wins, and voxels with
    too many near-identical entries for the kept list are still exact."""
    rng = np.random.default_rng(8)
    D = np.abs(rng.standard_normal((12, 600))) + 0.1
    D[:, 0] = 0.0
    D[3, 1], D[4, 2] = np.nan, np.inf
    D[:, 300:400] = D[:, 200:300]
    y = D[:, rng.integers(200, 600, 150)] * 3.0 + 0.01 * rng.standard_normal((12, 150))
    y[:, 0] = 0.0
    y[5, 1], y[6, 2] = np.nan, np.inf
    best, sse = _match(ctx, y, D)
    assert best[0] == 3 and sse[0] == 0.0
    assert best[1] == best[2] == -1 and np.all(np.isinf(sse[1:3]))
    assert np.array_equal(best[3:], np.nanargmin(_scores(y[:, 3:], D), axis=1))
    assert not np.any((best >= 300) & (best < 400))
    # a fine one-parameter dictionary in random order: many entries within the tensor cores' error
    te = np.linspace(2e-3, 40e-3, 12)[:, None]
    fine = np.exp(-te * rng.permutation(np.linspace(20.0, 20.2, 4000)))
    y = np.exp(-te * rng.uniform(20.0, 20.2, 700)) + 1e-3 * rng.standard_normal((12, 700))
    for n in (5, 700):
        best, _ = _match(ctx, y[:, :n], fine)
        s = _scores(y[:, :n], fine)
        A = (np.asarray(y[:, :n], np.float32).astype(np.float64) ** 2).sum(0)
        assert np.all(s[np.arange(n), best] - s.min(1) <= 1e-12 * A)


def _std_fit(ctx, kind, n, te, block, iters, **over):
    from helpers import run_engine
    rng = np.random.default_rng(n)
    _, om = models(kind, te=te)
    y = oracle.forward(om, random_theta(kind, n, rng)) + 0.01 * rng.standard_normal((len(te) * (1 + (kind != "r2s")), n))
    th0 = np.tile(np.array([[1.0], [30.0]] if kind == "r2s" else [[1.0], [1.0], [30.0]], np.float32), (1, n))
    return run_engine(kind, y, th0, fitting(iteration=iters, blockSize=block, **over), NAMES[kind], context=ctx, te=te)


def _same_fit(a, b, iters):
    for k in ("final_theta", "min_theta", "final_residual", "min_residual"):
        assert np.array_equal(a[k], b[k]), k
    assert a["final_niteration"] == b["final_niteration"] and a["min_niteration"] == b["min_niteration"]
    # the history's per-voxel terms are equal, their FP32 sums over a warp in another order (32 terms: 32 x 2^-24)
    h, g = a["loss_history"][: iters + 1], b["loss_history"][: iters + 1]
    assert np.allclose(h, g, rtol=4e-6, atol=0.0, equal_nan=True)


@pytest.mark.parametrize("n_te", [1, 8, 9, 12, 13, 16, 17])
@pytest.mark.parametrize("kind", ["r2s", "r1r2s"])
def test_fused_kernels_equal_the_general_one(ctx, kind, n_te):
    """The kernels of the standard configuration give the general kernel's
    parameters bit for bit: below, at and above their echo bounds, with volumes
    that end inside a 64-voxel chunk (the general kernel takes 96-thread blocks of R1-R2* and
    1024-thread blocks of R2*)."""
    te = np.linspace(2e-3, 40e-3, n_te) if n_te > 1 else np.array([5e-3])
    general = 1024 if kind == "r2s" else 96
    for n in (1, 33, 450):
        _same_fit(_std_fit(ctx, kind, n, te, 64, 40), _std_fit(ctx, kind, n, te, general, 40), 40)


@pytest.mark.parametrize("iters", [0, 1, 2, 31, 32, 33, 65])
@pytest.mark.parametrize("block", [32, 64, 128, 512])
def test_history_groups(ctx, iters, block):
    """Loss history and stopping statistics of fits that end around a group of
    32 epochs, with one and several warps a block (several volumes' worth of blocks)."""
    te = np.linspace(2e-3, 40e-3, 12)
    over = {"convergenceStepTol": 1e-30, "convergenceGradTol": 1e-30}
    for kind, general in (("r2s", 1024), ("r1r2s", 96)):
        a = _std_fit(ctx, kind, 700, te, block, iters, **over)
        _same_fit(a, _std_fit(ctx, kind, 700, te, general, iters, **over), iters)
        assert np.all(np.isfinite(a["loss_history"]))


@pytest.mark.parametrize("n,iters,over", [
    (99_400, 3, {}), (99_500, 2, {}), (100_003, 59, {"tol": 1e-30}),
    (123_457, 7, {"convergenceStepTol": 1e-30, "convergenceGradTol": 1e-30, "lossFunction": "l2"}),
])
def test_nexi_turns(ctx, n, iters, over):
    """Voxels that fill an SM's warps more than once are fitted in turns of
    (32 voxels, some epochs); with one epoch a launch (chunk) the general kernel
    fits them.  Same parameters bit for bit, around the voxel count of the rule,
    with a last turn of fewer epochs, with weights and statistics; the history's
    FP64 sums of equal terms (about 4000) in another order: 4000 x 2^-53."""
    from helpers import run_engine
    rng = np.random.default_rng(n)
    _, om = models("nexi")
    th = random_theta("nexi", n, rng)
    y = oracle.forward(om, th) + 0.01 * rng.standard_normal((24, n))
    w = rng.uniform(0.3, 1.0, y.shape).astype(np.float32) if "lossFunction" in over else None
    th0 = np.tile(np.array([[0.4], [2.0], [1.0], [0.05]], np.float32), (1, n))
    opts = dict({"tol": 1e-30}, **over)
    a, b = (run_engine("nexi", y, th0, fitting(iteration=iters, chunk=c, **opts), NAMES["nexi"], context=ctx, weights=w)
            for c in (0, 1))
    for k in ("final_theta", "min_theta", "final_residual", "min_residual"):
        assert np.array_equal(a[k], b[k]), k
    assert a["min_niteration"] == b["min_niteration"]
    assert np.allclose(a["loss_history"], b["loss_history"], rtol=1e-12, atol=0.0, equal_nan=True)


@pytest.mark.parametrize("n", [75_700, 75_800])
def test_r2s_pairs_rule(ctx, n):
    """Around the voxel count from which R2* takes two voxels a thread."""
    te = np.linspace(2e-3, 40e-3, 12)
    _same_fit(_std_fit(ctx, "r2s", n, te, 128, 33), _std_fit(ctx, "r2s", n, te, 1024, 33), 33)


@pytest.mark.parametrize("kind", ["r2s", "r1r2s", "nexi", "nexi2"])
@pytest.mark.parametrize("n", [1, 127, 129])
def test_gradient_on_device_arrays(ctx, kind, n):
    """The one-kernel gradient: device and host arrays, weights, a missing
    gradient or residual, against the oracle (the gradient parity test's bars)."""
    import torch
    rng = np.random.default_rng(n)
    gxm, om = models(kind)
    lb, ub = bounds(kind)
    th = random_theta(kind, n, rng).astype(np.float32)
    s = oracle.forward(om, th.astype(np.float64))
    y = (s + 0.02 * rng.standard_normal(s.shape)).astype(np.float32)
    w = rng.uniform(0.2, 1.0, y.shape).astype(np.float32)
    f = fitting(lossFunction="l2")
    opts = gx_askadam.build_opts(f, NAMES[kind], lb, ub)
    Lo, go, ro, _, _ = oracle.model_gradient(om, oracle.Volume(y.astype(np.float64), weights=w.astype(np.float64)),
                                             oracle.adam_opts(lb, ub, f), th.astype(np.float64))
    fp = lambda t: C.cast(C.c_void_p(t.data_ptr()), _lib._fp)  # noqa: E731
    arrays = {}
    for mem in (_lib.MEM_HOST, _lib.MEM_DEVICE):
        dev = "cuda" if mem == _lib.MEM_DEVICE else "cpu"
        ty, tw, tt = (torch.from_numpy(x).to(dev).contiguous() for x in (y, w, th))
        g, r, loss = torch.full_like(tt, -7.0), torch.full_like(ty, -7.0), C.c_double()
        vol = _lib.GxVolume()
        vol.dims[0], vol.dims[1], vol.dims[2], vol.nvox = n, 1, 1, n
        vol.data, vol.weights = fp(ty), fp(tw)
        torch.cuda.synchronize()
        for gp, rp in ((g.data_ptr(), r.data_ptr()), (None, r.data_ptr()), (g.data_ptr(), None)):
            _lib.check(_lib.lib().gx_model_gradient(ctx.ptr, C.byref(gxm.s), mem, C.byref(vol), C.byref(opts),
                                                    tt.data_ptr(), gp, rp, C.byref(loss), None, None))
        arrays[mem] = (g.cpu().numpy(), r.cpu().numpy(), loss.value)
    for a, b in zip(*arrays.values()):
        assert np.allclose(a, b, rtol=1e-12, atol=0.0)
    g, r, loss = arrays[_lib.MEM_HOST]
    assert abs(loss - Lo) <= 1e-5 * abs(Lo) + 1e-7
    assert np.all(np.abs(r - ro) <= 2e-4 * np.abs(ro) + 2e-5)
    for k in range(th.shape[0]):
        assert np.max(np.abs(g[k] - go[k])) <= 1e-3 * np.max(np.abs(go[k])) + 1e-12


@pytest.mark.parametrize("n_te,dims,pairs", [(12, (19, 16, 9), False), (8, (64, 65, 32), True), (12, (64, 65, 32), True),
                                             (16, (64, 65, 32), True)])
@pytest.mark.parametrize("over", [{"convergenceGradTol": 1e-6}, {"convergenceStepTol": 2e-4}, {}])
def test_tv_pairs_with_statistics(ctx, n_te, dims, pairs, over):
    """The TV kernel with stopping statistics over several launches of 200
    epochs, with slices on both sides of the two-voxel variant's rule:
    parameters equal the per-epoch kernel's bit for bit and the fit
    stops at the same epoch; the statistics' FP32 sums differ by their order."""
    import os
    from gacelle_b200 import phantoms, utils
    from helpers import run_engine
    te = np.linspace(2e-3, 40e-3, n_te)
    mask = phantoms.ellipsoid_mask(dims, 1.05)
    data, _ = phantoms.r2s_phantom(mask, 5, te=te)
    idx = utils.mask_index(mask)
    y = utils.reshape_ND2GD(data, idx)
    th0 = np.tile(np.array([[1.0], [30.0]], np.float32), (1, y.shape[1]))
    f = fitting(**dict({"iteration": 410, "lambda": [1e-5], "regmap": ["R2star"], "TVmode": "3D", "patience": 5,
                        "patienceStep": 5, "patienceGrad": 5, "convergenceStepTol": 1e-12, "convergenceGradTol": 1e-12},
                       **over))
    runs = []
    for kernel in ("persistent", "step"):
        os.environ["GACELLE_B200_TV_KERNEL"] = kernel
        try:
            runs.append(run_engine("r2s", y, th0, f, NAMES["r2s"], dims=mask.shape, gidx=idx.astype(np.int32),
                                   context=ctx, te=te))
        finally:
            del os.environ["GACELLE_B200_TV_KERNEL"]
    a, b = runs
    assert bool(a["timing"]["tv_path"] & _lib.TV_PAIRS) == pairs and b["timing"]["tv_path"] == 0
    assert a["final_niteration"] == b["final_niteration"] and a["stop_reason"] == b["stop_reason"]
    for k in ("final_theta", "min_theta", "final_residual"):
        assert np.array_equal(a[k], b[k]), k
    n = a["final_niteration"] + 1
    assert np.allclose(a["loss_history"][:n], b["loss_history"][:n], rtol=4e-6, atol=0.0)


@pytest.mark.parametrize("W,steps", [(2, 1), (16, 16), (51, 5), (43, 6), (64, 8), (57, 9), (64, 16), (41, 25), (32, 64),
                                     (50, 41)])
@pytest.mark.parametrize("nbin", [2, 1001, 9000])
def test_posterior_summaries_by_count(ctx, W, steps, nbin):
    """Median, inter-quartile range and mode of 2 to 2050 samples, around the
    sorting kernel's sizes (256, 512, 1024, 2048) and with a histogram that does
    not fit beside its keys (nbin 9000), against the numpy restatement."""
    from gacelle_b200 import mcmc_solver
    from gacelle_b200.models import gpuR2starMapping
    rng = np.random.default_rng(W)
    te, nv = np.linspace(2e-3, 40e-3, 12), 11
    m = gpuR2starMapping(te)
    th = np.vstack([rng.uniform(0.5, 1.5, nv), rng.uniform(10, 60, nv)])
    y = (th[0] * np.exp(-te[:, None] * th[1]) + 0.02 * rng.standard_normal((12, nv))).astype(np.float32)
    x0 = np.vstack([th, np.full(nv, 0.02)]).astype(np.float32)
    lb, ub = list(m.lb[:2]) + [0.02], list(m.ub[:2]) + [0.02]
    f = mcmc_solver.check_set_default_basic({
        "algorithm": "GW", "iteration": steps, "thinning": 1, "burnin": 0.0, "Nwalker": W, "lb": lb, "ub": ub, "seed": 3,
        "Nbin": nbin, "metric": ["median", "iqr", "mode"]})
    eng = mcmc_solver.mcmc(ctx)._run(m, y, None, x0, None, m.modelParams, f, True, stats=("median", "iqr", "mode"))
    for k in range(3):
        med, iqr, mode = oracle.res2out_summaries(eng["posterior"][k].reshape(-1, nv).T, lb[k], ub[k], nbin=nbin)
        np.testing.assert_array_equal(eng["median"][k], med)
        np.testing.assert_allclose(eng["iqr"][k], iqr, rtol=1e-6, atol=1e-7)
        np.testing.assert_array_equal(eng["mode"][k], mode)
