"""Corners of the host side's calls: methods that a user overrides, and the
index forms of the layout helpers."""
import numpy as np
import pytest

from gacelle_b200 import models, utils

TE = np.linspace(2e-3, 40e-3, 6)


def _captured(m, data, mask, **fitting):
    """What fit() hands to the solver: start, weights and masked data."""
    got = {}
    m._solve = lambda data, mask, w, pars0, fitting, extradata=None, masked=None: got.update(
        w=w, pars0=pars0, masked=masked)
    m.fit(data, mask, fitting)
    return got


def _image():
    rng = np.random.default_rng(0)
    mask = rng.uniform(size=(5, 4, 3)) > 0.4
    th = rng.uniform(0.5, 1.5, mask.shape), rng.uniform(10, 60, mask.shape)
    return (th[0][..., None] * np.exp(-TE * th[1][..., None])).astype(np.float32), mask


def test_masked_start_is_the_image_start():
    data, mask = _image()
    m = models.gpuR2starMapping(TE)
    got = _captured(m, data, mask)
    fitting = dict(m.check_set_default({}), lb=m.lb, ub=m.ub)
    x0 = m.determine_x0(data, mask, fitting)
    idx = utils.mask_index(mask)
    assert got["w"] is None and np.array_equal(got["masked"], utils.to_GD(data, mask))
    for p in ("M0", "R2star"):
        assert np.array_equal(utils.param_to_GD(got["pars0"][p], mask, idx, idx.size),
                              utils.param_to_GD(x0[p], mask, idx, idx.size))


@pytest.mark.parametrize("how", ["subclass", "instance", "class"])
@pytest.mark.parametrize("name", ["determine_x0", "estimate_prior", "R2star_trapezoidal"])
def test_overridden_start_is_taken(monkeypatch, how, name):
    """A start of the user's own, in a subclass, on the object or put into the
    class, is the one that fit() takes, with the default start option too."""
    data, mask = _image()
    full = {"M0": np.full(mask.shape, 0.75, np.float32), "R2star": np.full(mask.shape, 17.0, np.float32)}
    own = {"determine_x0": lambda *a: full, "estimate_prior": lambda *a: full,
           "R2star_trapezoidal": lambda *a: full["R2star"].astype(float)}[name]
    cls = models.gpuR2starMapping
    if how == "subclass":
        static = name == "R2star_trapezoidal"
        cls = type("Mine", (cls,), {name: staticmethod(own) if static else own})
    if how == "class":
        monkeypatch.setattr(cls, name, staticmethod(own))
    m = cls(TE)
    if how == "instance":
        setattr(m, name, own)
    got = _captured(m, data, mask)
    idx = utils.mask_index(mask)
    assert np.all(utils.param_to_GD(got["pars0"]["R2star"], mask, idx, idx.size) == 17.0)
    if name != "R2star_trapezoidal":
        assert np.all(utils.param_to_GD(got["pars0"]["M0"], mask, idx, idx.size) == 0.75)


def test_overridden_weights_are_taken():
    """Weights of the user's own are taken whatever isWeighted says."""
    data, mask = _image()

    class Mine(models.gpuR2starMapping):
        @staticmethod
        def compute_optimisation_weights(data, fitting):
            return np.full(data.shape, 0.5)

    assert np.all(_captured(Mine(TE), data, mask)["w"] == 0.5)
    assert _captured(models.gpuR2starMapping(TE), data, mask)["w"] is None
    assert np.any(_captured(models.gpuR2starMapping(TE), data, mask, isWeighted=True)["w"] != 1)


@pytest.mark.parametrize("index", ["indices", "boolean", "slice", "list", "int32", "uint64", "negative"])
def test_reshape_nd2gd_takes_any_row_index(index):
    """Rows of the column-major voxel list by any of numpy's row indices."""
    data, mask = _image()
    flat = mask.ravel(order="F")
    idx = {"indices": np.flatnonzero(flat), "boolean": flat, "slice": slice(3, 20, 2), "list": [5, 1, 7],
           "int32": np.array([5, 1, 7], np.int32), "uint64": np.array([5, 1, 7], np.uint64),
           "negative": np.array([-1, 0])}[index]
    want = data.reshape((mask.size, -1), order="F")[idx].T
    got = utils.reshape_ND2GD(data, idx)
    assert got.flags.c_contiguous and np.array_equal(got, want)
