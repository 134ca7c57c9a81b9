"""Corners of the calls' ranges: values, sizes and options at which a kernel's
shortcut, index or wait could go wrong, each against the oracle, the general
form of the same kernel or a plain restatement."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gacelle_b200 import _lib
from gacelle_b200 import askadam_solver as gx_askadam

from helpers import NAMES, bounds, fitting, models, random_theta

pytestmark = pytest.mark.gpu


def _gradient(ctx, kind, y, th, b1=None, **over):
    """gx_model_gradient on host arrays: fidelity, gradient, residual."""
    n = th.shape[1]
    gxm, _ = models(kind)
    lb, ub = bounds(kind)
    opts = gx_askadam.build_opts(fitting(**over), NAMES[kind], lb, ub)
    vol = _lib.GxVolume()
    vol.dims[0], vol.dims[1], vol.dims[2], vol.nvox = n, 1, 1, n
    g, r, fid = np.zeros_like(th), np.zeros_like(y), C.c_double()
    idx = np.arange(n, dtype=np.int32)
    vol.data, vol.grid_index = y.ctypes.data_as(_lib._fp), idx.ctypes.data_as(_lib._i32p)
    if b1 is not None:
        vol.b1 = b1.ctypes.data_as(_lib._fp)
    _lib.check(_lib.lib().gx_model_gradient(ctx.ptr, C.byref(gxm.s), _lib.MEM_HOST, C.byref(vol), C.byref(opts),
                                            th.ctypes.data, g.ctypes.data, r.ctypes.data, None, C.byref(fid), None))
    return fid.value, g, r


@pytest.mark.parametrize("loss", ["mse", "l2"])
@pytest.mark.parametrize("kind", ["r2s", "r1r2s", "nexi"])
def test_gradient_of_non_finite_predictions(ctx, kind, loss):
    """Voxels whose parameters (or B1) are not numbers, or make the signal
    overflow at every or at some echo times: their non-finite predictions count
    as 0 (utils.set_nan_inf_zero, utils/askadam.m:80), so that the call's loss
    stays a number, as the oracle's does.  With and without a regulariser, whose
    paths are different kernels, the fidelity, the residuals and the gradient of
    an unregularised parameter are the same (bars of the gradient parity tests)."""
    rng = np.random.default_rng(3)
    n = 150
    _, om = models(kind)
    lb, ub = bounds(kind)
    th = random_theta(kind, n, rng).astype(np.float32)
    y = (oracle.forward(om, th.astype(np.float64)) + 0.02 * rng.standard_normal((24 if kind != "r2s" else 12, n))).astype(np.float32)
    b1 = rng.uniform(0.8, 1.2, n).astype(np.float32) if kind == "r1r2s" else None
    odd = [5, 77, 149]
    th[0, 5], th[1, 77] = np.nan, np.nan
    if kind == "nexi":
        th[3, 149] = np.inf
    else:
        th[-1, 149] = -1e6      # overflows at every echo time, in 64 bits as well
        th[-1, 20] = np.inf     # a signal of 0, finite
        odd.append(100)
        th[-1, 100] = -1e5      # in 32 bits at every echo time, in 64 bits at the later ones: not compared below
        y[:, 100] = 0.0
    if b1 is not None:
        b1[64] = np.nan
        odd.append(64)
    fid, g, r = _gradient(ctx, kind, y, th, b1, lossFunction=loss)
    assert np.isfinite(fid)
    # the oracle, over the voxels whose predictions are the same numbers in 32 and 64 bits (its NEXI
    # forward's fmin makes a NaN 1), at the same mean
    keep = np.setdiff1d(np.arange(n), odd if kind == "nexi" else [100])
    f = fitting(lossFunction=loss)
    vol = oracle.Volume(y[:, keep].astype(np.float64), b1=None if b1 is None else b1[keep].astype(np.float64),
                        norm_nvox=float(n))
    Lo, go, ro, _, _ = oracle.model_gradient(om, vol, oracle.adam_opts(lb, ub, f), th[:, keep].astype(np.float64))
    if kind != "nexi":
        assert np.isfinite(Lo) and abs(fid - Lo) <= 1e-5 * abs(Lo) + 1e-7
    assert np.all(np.abs(r[:, keep] - ro) <= 2e-4 * np.abs(ro) + 2e-5)
    fine = np.setdiff1d(np.arange(n), odd)
    at = np.searchsorted(keep, fine)
    for k in range(th.shape[0]):
        assert np.max(np.abs(g[k][fine] - go[k][at])) <= 1e-3 * np.max(np.abs(go[k][at])) + 1e-12
    # the op-by-op kernels, which a regulariser of the last parameter takes
    fid2, g2, r2 = _gradient(ctx, kind, y, th, b1, lossFunction=loss, regmap=[NAMES[kind][-1]], TVmode="2D",
                             **{"lambda": [1e-6]})
    assert abs(fid - fid2) <= 1e-5 * abs(fid2)
    np.testing.assert_allclose(r, r2, rtol=2e-5, atol=2e-6)
    assert np.array_equal(np.isnan(g[:-1]), np.isnan(g2[:-1]))
    for k in range(th.shape[0] - 1):
        assert np.nanmax(np.abs(g[k] - g2[k])) <= 1e-3 * np.nanmax(np.abs(g2[k])) + 1e-12


def _chain(ctx, te, y, x0, update, W, steps, lb, ub, step, weights=None, **over):
    from gacelle_b200 import mcmc_solver
    from gacelle_b200.models import gpuR2starMapping
    m = gpuR2starMapping(te)
    f = mcmc_solver.check_set_default_basic(dict({
        "algorithm": "MH" if update == "mh" else "GW", "iteration": steps, "thinning": 3, "burnin": 0.0, "Nwalker": W,
        "Ensembleupdate": "redblack" if update == "redblack" else "simultaneous", "lb": lb, "ub": ub,
        "xStepSize": step, "seed": 21}, **over))
    solver = mcmc_solver.mcmc(ctx)
    return dict(solver._run(m, y, weights, x0, None, m.modelParams, f, True), n_accepted=solver.last_stats["n_accepted"])


def _same_chains(ctx, n_te, update, noise, scale, nv, steps, blocks):
    """Chains with the FP32 screen and, with unit weights as an array, those
    decided in FP64 throughout, from the same starts."""
    rng = np.random.default_rng(n_te)
    te = np.linspace(2e-3, 40e-3, n_te)
    th = np.vstack([scale * rng.uniform(0.5, 1.5, nv), rng.uniform(10, 60, nv)])
    y = (th[0] * np.exp(-te[:, None] * th[1]) + noise * rng.standard_normal((n_te, nv))).astype(np.float32)
    x0 = np.vstack([th, np.full(nv, noise)]).astype(np.float32)
    lb, ub = [0.0, 0.1, 0.8 * noise], [2.0 * scale, 200.0, 4.0 * noise]
    step = [noise, 50.0 * noise / scale, 0.2 * noise]  # of the posterior's width: about half of the moves are taken
    ones = np.ones_like(y)
    W = 1 if update == "mh" else 17
    a, *rest = [_chain(ctx, te, y, x0, update, W, steps, lb, ub, step, w, blockSize=b)
                for w, b in [(ones, blocks[0])] + [(None, b) for b in blocks]]
    moved = np.mean(np.diff(a["posterior"][0].reshape(-1, nv), axis=0) != 0)
    assert 0.05 < moved
    for b in rest:
        for key in ("posterior", "mean", "std"):
            assert np.array_equal(a[key], b[key], equal_nan=True), key
        assert a["n_accepted"] == b["n_accepted"]


@pytest.mark.parametrize("noise", [0.02, 0.001])
@pytest.mark.parametrize("n_te", [3, 8, 12, 16])
@pytest.mark.parametrize("update,steps", [("simultaneous", 1500), ("redblack", 1500), ("mh", 6000)])
def test_screened_decisions_are_the_fp64_ones(ctx, update, steps, n_te, noise):
    """The screened acceptance takes every decision as the FP64 log-likelihoods
    do, also at small noise, where a residual's last bit is worth most: whole
    chains are equal bit for bit (both Metropolis-Hastings kernels)."""
    _same_chains(ctx, n_te, update, noise, 1.0, 40, steps, (0, 64) if update == "mh" else (0,))


@pytest.mark.parametrize("scale,noise", [(1e-18, 1e-19), (1e-15, 1.5e-16), (1e-15, 1e-16), (1e6, 1e4), (1e19, 1e18)])
@pytest.mark.parametrize("update,steps", [("simultaneous", 300), ("mh", 1200)])
def test_screened_decisions_in_any_unit(ctx, update, steps, scale, noise):
    """The same for data in units whose noise (or its square) leaves FP32's
    normal range, where the screen's bound does not hold."""
    _same_chains(ctx, 12, update, noise, scale, 40, steps, (0, 64) if update == "mh" else (0,))


@pytest.mark.parametrize("weighted", [True, False])
def test_dictionary_match_of_2_30_voxels(ctx, weighted):
    """More than 2^30 voxels of one measurement against one entry, where 32-bit
    steps over the work-list wrap: every voxel is matched, none twice wrongly."""
    import torch
    n = (1 << 30) + 65
    y = torch.full((n,), 2.0, device="cuda")
    y[-1] = 3.0
    D, w = torch.tensor([0.5], device="cuda"), torch.tensor([1.5], device="cuda")
    best = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.lib().gx_dictionary_match(ctx.ptr, _lib.MEM_DEVICE, y.data_ptr(), n, D.data_ptr(), 1, 1,
                                              w.data_ptr() if weighted else None, best.data_ptr(), None))
    assert int(best.min()) == 0 and int(best.max()) == 0
    del y, best
    torch.cuda.empty_cache()


def _match(ctx, y, D):
    y, D = np.ascontiguousarray(y, np.float32), np.ascontiguousarray(D, np.float32)
    best, sse = np.full(y.shape[1], -7, np.int32), np.full(y.shape[1], np.nan, np.float32)
    _lib.check(_lib.lib().gx_dictionary_match(ctx.ptr, _lib.MEM_HOST, y.ctypes.data, y.shape[1], D.ctypes.data,
                                              D.shape[1], y.shape[0], None, best.ctypes.data, sse.ctypes.data))
    return best, sse, ctx.timing()["kernel_launches"]


def _scores(y, D):
    """sse [voxel, entry] in FP64 by the expanded form; NaN for an entry without a norm."""
    y, D = np.asarray(y, np.float32).astype(np.float64), np.asarray(D, np.float32).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        return (y * y).sum(0)[:, None] - (y.T @ D) ** 2 / (D * D).sum(0)


@pytest.mark.parametrize("nm,nvox,entries,tensor", [
    (1, 127, 1535, False), (1, 1, 1536, True), (8, 129, 1537, True), (15, 260, 1663, True), (16, 128, 1023, False),
    (16, 1, 1024, True), (17, 127, 1025, True), (24, 129, 1151, True), (24, 260, 1152, True), (33, 257, 1153, True),
    (48, 3, 1200, True), (56, 130, 1281, True), (64, 383, 1408, True), (65, 129, 1408, False),
    (24, 40000, 599, False), (24, 40001, 600, True), (33, 40000, 1023, False), (8, 39999, 1100, False)])
def test_dictionary_rule_and_tiles(ctx, nm, nvox, entries, tensor):
    """Both kernels on either side of the rule (entries by measurements and
    voxels) and around the 128-row operand tiles, at scales from 1e-20 to 1e20:
    the entry of least FP64 score, or one whose score equals it to 1e-12 of the voxel's
    energy.  The tensor-core path takes four launches, the FP64 kernel two."""
    rng = np.random.default_rng(nm * 1000 + nvox)
    y = rng.standard_normal((nm, nvox)) * 10.0 ** rng.uniform(-10, 10, nvox)
    D = rng.standard_normal((nm, entries)) * 10.0 ** rng.uniform(-10, 10, entries)
    best, sse, launches = _match(ctx, y, D)
    assert launches == (4 if tensor else 2)
    at = np.arange(nvox) if nvox < 1000 else rng.permutation(nvox)[:1000]
    s = _scores(y[:, at], D)
    A = (np.asarray(y[:, at], np.float32).astype(np.float64) ** 2).sum(0)
    got = s[np.arange(at.size), best[at]]
    assert np.all(got - s.min(1) <= 1e-12 * A)
    assert np.all(np.abs(sse[at] - got) <= 1e-6 * np.abs(got) + 1e-12 * A)


def test_dictionary_special_values_on_the_tensor_cores(ctx):
    """Zero voxels take the first entry with a norm, voxels and entries that are
    not numbers match nothing, and of equal entries the first wins, with a
    dictionary that the tensor-core kernel takes."""
    rng = np.random.default_rng(8)
    D = np.abs(rng.standard_normal((20, 1700))) + 0.1
    D[:, 0] = 0.0
    D[3, 1], D[4, 2] = np.nan, np.inf
    D[:, 300:400] = D[:, 200:300]
    y = D[:, rng.integers(200, 1700, 150)] * 3.0 + 0.01 * rng.standard_normal((20, 150))
    y[:, 0] = 0.0
    y[5, 1], y[6, 2] = np.nan, np.inf
    best, sse, launches = _match(ctx, y, D)
    assert launches == 4
    assert best[0] == 3 and sse[0] == 0.0
    assert best[1] == best[2] == -1 and np.all(np.isinf(sse[1:3]))
    assert np.array_equal(best[3:], np.nanargmin(_scores(y[:, 3:], D), axis=1))
    assert not np.any((best >= 300) & (best < 400))


@pytest.mark.parametrize("kind,blocks", [("r2s", (544, 800)), ("r1r2s", (704, 736)), ("nexi", (512,)), ("nexi2", (544, 672))])
@pytest.mark.parametrize("n_te", [12, 17])
def test_mh_large_blocks(ctx, kind, blocks, n_te):
    """Metropolis-Hastings takes a chosen block beyond the threads that its
    registers leave, in blocks as large as they do: chains equal those of
    128-thread blocks bit for bit."""
    from gacelle_b200 import mcmc_solver
    from gacelle_b200.models import gpuJointR1R2starMapping, gpuNEXI, gpuR2starMapping
    te = np.linspace(2e-3, 40e-3, n_te)
    if kind == "r2s":
        m = gpuR2starMapping(te)
    elif kind == "r1r2s":
        m = gpuJointR1R2starMapping(te, 0.03, [5.0, 20.0])
    else:
        m = gpuNEXI(np.tile([1.0, 2.5, 4.0, 6.0, 8.0, 10.0], 4), np.repeat([20.0, 27.0, 35.0, 49.0], 6))
        m._gx_model = lambda: models(kind)[0]
    rng = np.random.default_rng(6)
    nv = 900
    _, om = models(kind, **({"te": te} if kind[0] == "r" else {}))
    th = random_theta(kind, nv, rng)
    s = oracle.forward(om, th)
    y = (s + 0.02 * rng.standard_normal(s.shape)).astype(np.float32)
    x0 = np.vstack([th, np.full(nv, 0.02)]).astype(np.float32)
    lb, ub = bounds(kind)
    out = []
    for block in (128,) + blocks:
        f = mcmc_solver.check_set_default_basic({
            "algorithm": "MH", "iteration": 40, "thinning": 2, "burnin": 0.0, "lb": list(lb) + [0.001],
            "ub": list(ub) + [0.1], "xStepSize": [0.01] * (len(NAMES[kind]) + 1), "seed": 4, "blockSize": block})
        solver = mcmc_solver.mcmc(ctx)
        out.append(solver._run(m, y, None, x0, None, NAMES[kind] + ["noise"], f, True))
        assert solver.last_timing["block_size"] <= block and solver.last_timing["block_size"] >= 128
    for o in out[1:]:
        for key in ("posterior", "mean", "std"):
            assert np.array_equal(out[0][key], o[key], equal_nan=True), key


@pytest.mark.parametrize("kind,loss", [("r2s", "l1"), ("r2s", "l2"), ("r2s", "huber"), ("r2s", "gauss"),
                                       ("r1r2s", "l2")])
def test_fit_blocks_up_to_896(ctx, kind, loss):
    """Fits with stopping statistics in blocks of 800 and 896 threads (72
    registers a thread) equal those in blocks of 128, bit for bit."""
    from helpers import run_engine
    rng = np.random.default_rng(2)
    n = 1000
    _, om = models(kind)
    s = oracle.forward(om, random_theta(kind, n, rng))
    y = s + 0.01 * rng.standard_normal(s.shape)
    th0 = np.tile(np.array([[1.0], [30.0]] if kind == "r2s" else [[1.0], [1.0], [30.0]], np.float32), (1, n))
    a, *rest = (run_engine(kind, y, th0, fitting(iteration=12, blockSize=block, lossFunction=loss, noiseSigma=0.02,
                                                 tol=-np.inf, convergenceStepTol=1e-30, convergenceGradTol=1e-30),
                           NAMES[kind], context=ctx) for block in (128, 800, 896))
    for b in rest:
        for k in ("final_theta", "min_theta", "final_residual"):
            assert np.array_equal(a[k], b[k]), k


@pytest.fixture
def own_ctx():
    from gacelle_b200 import Context
    c = Context(0)
    yield c
    c.close()


def _hooks(ctx, **kw):
    h = _lib.GxTestHooks(0, kw.get("wait_limit_cycles", 0), kw.get("barrier_extra_arrivals", 0))
    _lib.check(_lib.lib().gx_context_set_test_hooks(ctx.ptr, C.byref(h)))


@pytest.mark.parametrize("chunk", [0, 8])
def test_nexi_turns_wait_runs_out(own_ctx, chunk):
    """A wait of the NEXI kernel that takes voxels in turns, for a unit that
    nobody runs, ends at its limit: the call reports GX_ETIMEOUT (in one launch or several)
    and the context stays usable."""
    import time

    from helpers import run_engine
    rng = np.random.default_rng(1)
    n = 100_003
    _, om = models("nexi")
    y = oracle.forward(om, random_theta("nexi", n, rng)) + 0.01 * rng.standard_normal((24, n))
    th0 = np.tile(np.array([[0.4], [2.0], [1.0], [0.05]], np.float32), (1, n))
    f = fitting(iteration=40, chunk=chunk, **({"tol": 1e-30} if chunk else {"tol": -np.inf}))
    good = run_engine("nexi", y, th0, f, NAMES["nexi"], context=own_ctx)
    _hooks(own_ctx, wait_limit_cycles=2_000_000, barrier_extra_arrivals=1000)
    t0 = time.perf_counter()
    with pytest.raises(_lib.GacelleError) as e:
        run_engine("nexi", y, th0, f, NAMES["nexi"], context=own_ctx)
    assert e.value.status == _lib.GX_ETIMEOUT
    assert time.perf_counter() - t0 < 5.0
    _hooks(own_ctx)
    again = run_engine("nexi", y, th0, f, NAMES["nexi"], context=own_ctx)
    np.testing.assert_array_equal(again["final_theta"], good["final_theta"])


@pytest.mark.parametrize("loss,sizes,over", [
    ("rician", [100_003], {}), ("mse", [60_000, 45_003], {"convergenceStepTol": 1e-30, "convergenceGradTol": 1e-30}),
    ("rician", [3, 99_000, 31], {"blockSize": 96}), ("mse", [94_752], {"blockSize": 32})])
def test_nexi_turns_forms(ctx, loss, sizes, over):
    """NEXI fits in turns under the Rician loss, over several volumes and with a
    chosen block equal those of the block kernel (one epoch a launch) bit for bit;
    gx_timing.block_size tells which of the two ran."""
    rng = np.random.default_rng(len(sizes))
    gxm, om = models("nexi")
    lb, ub = bounds("nexi")
    data = []
    for n in sizes:
        s = oracle.forward(om, random_theta("nexi", n, rng))
        data.append(np.abs(s + 0.02 * rng.standard_normal(s.shape)).astype(np.float32))
    runs = []
    for chunk in (0, 1):
        f = fitting(iteration=9, chunk=chunk, lossFunction=loss, noiseSigma=0.02, **dict({"tol": -1e30 if loss == "rician" else 1e-30}, **over))
        opts = gx_askadam.build_opts(f, NAMES["nexi"], lb, ub)
        vols, res, keep = (_lib.GxVolume * len(sizes))(), (_lib.GxAskadamResult * len(sizes))(), []
        for v, r, y in zip(vols, res, data):
            n = y.shape[1]
            th0 = np.tile(np.array([[0.4], [2.0], [1.0], [0.05]], np.float32), (1, n))
            out = [np.zeros((4, n), np.float32), np.zeros((4, n), np.float32), np.zeros_like(y)]
            v.nvox, v.dims[0], v.dims[1], v.dims[2] = n, n, 1, 1
            v.data, v.theta0 = y.ctypes.data_as(_lib._fp), th0.ctypes.data_as(_lib._fp)
            r.final_theta, r.min_theta, r.final_residual = (x.ctypes.data_as(_lib._fp) for x in out)
            keep.append((th0, out))
        _lib.check(_lib.lib().gx_askadam(ctx.ptr, C.byref(gxm.s), _lib.MEM_HOST, vols, len(sizes), C.byref(opts), res))
        runs.append(([k[1] for k in keep], ctx.timing()["block_size"]))
    (a, block_a), (b, block_b) = runs
    assert block_a == 640 and block_b != 640
    for x, y in zip(a, b):
        for p, q in zip(x, y):
            assert np.array_equal(p, q)


def test_autotuner_keeps_kernels_apart(ctx):
    """A block tuned for one kernel is not taken for another: fits of one
    voxel-count class on either side of a rule, and protocols with as many
    measurements but other flip angles, are tuned each; where the kernel has
    no block to choose nothing is tuned."""
    from helpers import run_engine

    def tuned(kind, n, th0, **kw):
        _, om = models(kind, **kw)
        y = np.tile(oracle.forward(om, np.array(th0)[:, None]), (1, n)) + 0.01
        r = run_engine(kind, y, np.tile(np.array(th0, np.float32)[:, None], (1, n)), fitting(iteration=3, tol=-np.inf),
                       NAMES[kind], context=ctx, **kw)
        return r["timing"]["autotuned"]

    nexi = [0.4, 2.0, 1.0, 0.05]
    assert [tuned("nexi", n, nexi, nx=11) for n in (100_003, 80_000, 80_100, 100_003)] == [0, 1, 0, 0]
    te = np.linspace(2e-3, 40e-3, 11)
    assert [tuned("r2s", n, [1.0, 30.0], te=te) for n in (70_000, 80_000, 70_100)] == [1, 1, 0]
    for fa, nte in (([5.0, 20.0], 10), ([5.0, 10.0, 15.0, 20.0], 5)):
        te = np.linspace(2e-3, 40e-3, nte)
        assert tuned("r1r2s", 5000, [1.0, 1.0, 30.0], te=te, fa=fa) == 1
    te = np.linspace(2e-3, 40e-3, 10)
    assert [tuned("r1r2s", n, [1.0, 1.0, 30.0], te=te, fa=[5.0, 20.0]) for n in (8800, 9000, 9600)] == [1, 0, 1]


@pytest.mark.parametrize("loss", ["mse", "rician", "l1"])
@pytest.mark.parametrize("n,nx", [(1, 2), (33, 3), (700, 14), (75_700, 13), (75_800, 14), (300, 129)])
def test_nexi_few_voxels(ctx, n, nx, loss):
    """The NEXI kernel for few voxels (blocks up to 512 threads) gives the
    parameters of the capped one (576 threads) bit for bit: odd and even node
    counts, beyond the node table, around the voxel count of the rule."""
    from helpers import run_engine
    rng = np.random.default_rng(n)
    _, om = models("nexi", nx=nx)
    y = np.abs(oracle.forward(om, random_theta("nexi", n, rng)) + 0.01 * rng.standard_normal((24, n)))
    th0 = np.tile(np.array([[0.4], [2.0], [1.0], [0.05]], np.float32), (1, n))
    a, b, c = (run_engine("nexi", y, th0, fitting(iteration=6, blockSize=block, lossFunction=loss, tol=-1e30,
                                                  noiseSigma=0.02), NAMES["nexi"], context=ctx, nx=nx)
               for block in (128, 512, 576))
    for k in ("final_theta", "min_theta", "final_residual"):
        assert np.array_equal(a[k], c[k]) and np.array_equal(b[k], c[k]), k


def test_dictionary_wait_runs_out(own_ctx):
    """A wait of the tensor-core kernel for products that nobody makes ends at
    its limit: the call reports GX_ETIMEOUT and the next one matches."""
    import time
    rng = np.random.default_rng(5)
    D = np.abs(rng.standard_normal((24, 1500))) + 0.1
    y = D[:, rng.integers(0, 1500, 40_100)] + 0.01 * rng.standard_normal((24, 40_100))
    good, sse, launches = _match(own_ctx, y, D)
    assert launches == 4
    _hooks(own_ctx, wait_limit_cycles=2_000_000, barrier_extra_arrivals=1)
    t0 = time.perf_counter()
    with pytest.raises(_lib.GacelleError) as e:
        _match(own_ctx, y, D)
    assert e.value.status == _lib.GX_ETIMEOUT and "dictionary" in str(e.value)
    assert time.perf_counter() - t0 < 5.0
    _hooks(own_ctx)
    best, sse2, _ = _match(own_ctx, y, D)
    assert np.array_equal(best, good) and np.array_equal(sse, sse2)


def test_arrays_of_more_than_2_31_values(own_ctx):
    """Signals and gradients of arrays [measurement][voxel] with more than 2^31
    values: every row holds what the same voxels give in a small call.  The
    calls whose kernels index such arrays in 32 bits refuse them."""
    import torch
    n, few = (1 << 31) // 24 + 2000, 1000
    gxm, _ = models("r1r2s")
    lb, ub = bounds("r1r2s")
    th = torch.from_numpy(random_theta("r1r2s", few, np.random.default_rng(0)).astype(np.float32)).cuda()
    spread = torch.arange(n, device="cuda") % few
    fp = lambda t: C.cast(C.c_void_p(t.data_ptr()), _lib._fp)  # noqa: E731
    L = _lib.lib()
    opts = gx_askadam.build_opts(fitting(lossFunction="l2", iteration=2), NAMES["r1r2s"], lb, ub)
    out = {}
    for m in (few, n):
        t = th if m == few else th[:, spread].contiguous()
        s = torch.zeros(24, m, device="cuda")
        torch.cuda.synchronize()
        _lib.check(L.gx_forward(own_ctx.ptr, C.byref(gxm.s), _lib.MEM_DEVICE, t.data_ptr(), None, m, s.data_ptr()))
        vol, loss = _lib.GxVolume(), C.c_double()
        vol.dims[0], vol.dims[1], vol.dims[2], vol.nvox, vol.data = m, 1, 1, m, fp(s)
        g, r, t2 = torch.zeros_like(t), torch.zeros_like(s), (t * 1.05).contiguous()
        torch.cuda.synchronize()
        _lib.check(L.gx_model_gradient(own_ctx.ptr, C.byref(gxm.s), _lib.MEM_DEVICE, C.byref(vol), C.byref(opts),
                                       t2.data_ptr(), g.data_ptr(), r.data_ptr(), C.byref(loss), None, None))
        out[m] = [s, g * m, r]  # the gradient is of a mean over m voxels
    for a, b in zip(out[few], out[n]):
        for k in range(a.shape[0]):
            assert torch.allclose(a[k][spread], b[k], rtol=1e-5, atol=1e-12), k
    # refused before anything is read: Metropolis-Hastings, and a fit's residuals
    x0 = torch.cat([t, torch.full((1, n), 0.02, device="cuda")]).contiguous()
    vol.theta0 = fp(x0)
    lo, hi, step = (np.array(v) for v in (list(lb) + [0.001], list(ub) + [0.1], [0.01, 0.01, 1.0, 0.005]))
    o = _lib.GxMcmcOpts()
    o.algorithm, o.iteration, o.thinning, o.burnin, o.repetition, o.nwalker = 0, 2, 1, 0.0, 1, 1
    o.step_size, o.start_range, o.seed = 2.0, 0.001, 3
    o.lb, o.ub, o.x_step = (v.ctypes.data_as(_lib._dp) for v in (lo, hi, step))
    res, fit = _lib.GxMcmcResult(), _lib.GxAskadamResult()
    res.mean, fit.final_residual, fit.final_theta, fit.min_theta = fp(x0), fp(r), fp(g), fp(g)
    with pytest.raises(_lib.GacelleError) as e:
        _lib.check(L.gx_mcmc(own_ctx.ptr, C.byref(gxm.s), _lib.MEM_DEVICE, C.byref(vol), 1, C.byref(o), C.byref(res)))
    assert e.value.status == _lib.GX_EUNSUPPORTED
    with pytest.raises(_lib.GacelleError) as e:
        _lib.check(L.gx_askadam(own_ctx.ptr, C.byref(gxm.s), _lib.MEM_DEVICE, C.byref(vol), 1, C.byref(opts), C.byref(fit)))
    assert e.value.status == _lib.GX_EUNSUPPORTED
    out.clear()
    del s, t, t2, g, r, x0, spread, a, b
    torch.cuda.empty_cache()


@pytest.mark.parametrize("loss", ["mse", "l1"])
@pytest.mark.parametrize("kind", ["r2s", "r1r2s", "nexi"])
@pytest.mark.parametrize("shift", [0, 1, 5, "row"])
def test_gradient_in_place(ctx, kind, loss, shift):
    """Residual written over the data, and gradient over the parameters, whole
    or shifted by some values or a row: the results of separate arrays."""
    import torch
    rng = np.random.default_rng(4)
    n = 3000
    gxm, om = models(kind)
    lb, ub = bounds(kind)
    opts = gx_askadam.build_opts(fitting(lossFunction=loss), NAMES[kind], lb, ub)
    th = random_theta(kind, n, rng).astype(np.float32)
    th[0, 7] = np.nan
    s = oracle.forward(om, random_theta(kind, n, rng))
    y = (s + 0.02 * rng.standard_normal(s.shape)).astype(np.float32)
    fp = lambda a: C.cast(C.c_void_p(a), _lib._fp)  # noqa: E731

    def call(off):
        pad = 0 if off is None else off
        ty, tt = (torch.zeros(x.size + pad, device="cuda") for x in (y, th))
        ty[:y.size], tt[:th.size] = torch.from_numpy(y.ravel()).cuda(), torch.from_numpy(th.ravel()).cuda()
        r, g = (torch.zeros_like(ty), torch.zeros_like(tt)) if off is None else (ty, tt)
        vol, loss_out = _lib.GxVolume(), C.c_double()
        vol.dims[0], vol.dims[1], vol.dims[2], vol.nvox, vol.data = n, 1, 1, n, fp(ty.data_ptr())
        torch.cuda.synchronize()
        _lib.check(_lib.lib().gx_model_gradient(ctx.ptr, C.byref(gxm.s), _lib.MEM_DEVICE, C.byref(vol), C.byref(opts),
                                                tt.data_ptr(), g.data_ptr() + 4 * pad, r.data_ptr() + 4 * pad,
                                                C.byref(loss_out), None, None))
        return r[pad:pad + y.size].cpu().numpy(), g[pad:pad + th.size].cpu().numpy(), loss_out.value

    a, b = call(None), call(n if shift == "row" else shift)
    assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1], equal_nan=True)
    assert np.isclose(a[2], b[2], rtol=1e-12)
