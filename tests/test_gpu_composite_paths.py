"""The compositor's branches against the oracle, bit for bit: tile lists around
the staging chunk's size, groups of pixels cut by the image border, opacities
above the 0.99 clamp, values that are not finite, and termination thresholds at
and beyond the ends of their range."""
import os

import numpy as np
import pytest

import oracle as O
from lumen_b200.types import RenderOptions, ViewCamera

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NT = max(1, min(16, os.cpu_count() or 1))


def _scene(n, seed, opacity):
    """n splats in front of a small camera, most of them over the whole image."""
    rng = np.random.Generator(np.random.PCG64(seed))
    means = rng.uniform(-1.0, 1.0, size=(n, 3)) * [0.6, 0.4, 1.0] + [0.0, 0.0, 4.0]
    scales = np.exp(rng.uniform(np.log(0.02), np.log(0.6), size=(n, 3)))
    quats = rng.standard_normal(size=(n, 4))
    op = rng.uniform(*opacity, size=n)
    sh = rng.normal(0.0, 0.1, size=(n, 16, 3))
    sh[:, 0] += 0.6
    f = np.float32
    return [a.astype(f) for a in (means, scales, quats, op, sh)]


def _check(scene, cam, opt):
    from lumen_b200 import render as R
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    means, scales, quats, op, sh = scene
    g = R.render(dev(means), dev(scales), dev(quats), dev(op), dev(sh).reshape(-1, 48), cam, opt)
    with np.errstate(all="ignore"):
        o = O.render(means, scales, quats, op, sh, cam, opt, nthreads=NT)
    assert (g.n_visible, g.n_instances) == (o.n_visible, o.n_instances)
    assert np.array_equal(g.n_contrib.cpu().numpy().view(np.uint32), o.n_contrib)
    assert np.array_equal(g.last_idx.cpu().numpy(), o.last_idx)
    for name in ("rgb", "depth", "alpha"):
        a, b = getattr(g, name).cpu().numpy(), getattr(o, name)
        nan = np.isnan(b)
        assert np.array_equal(np.isnan(a), nan), name
        assert np.array_equal(a[~nan].view(np.uint32), b[~nan].view(np.uint32)), name
    return g


def _cam(w, h):
    return ViewCamera((0, 0, 0), (1, 0, 0, 0), 60, 60, w / 2, h / 2, 0.1, 100, w, h)


@pytest.mark.parametrize("size", [(16, 16), (17, 1), (3, 33), (45, 30)])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 255, 256, 257, 515])
def test_tile_lists_around_the_chunk_size(n, size):
    _check(_scene(n, n, (0.01, 0.05)), _cam(*size), RenderOptions())


@pytest.mark.parametrize("n", [40, 700])
def test_opacities_above_the_clamp(n):
    _check(_scene(n, 7 * n, (0.2, 1.0)), _cam(45, 30), RenderOptions(term_mode=0))
    _check(_scene(n, 7 * n, (0.985, 1.0)), _cam(45, 30), RenderOptions(term_mode=1, term_threshold=0.9999))


@pytest.mark.parametrize("what", ["nan colour", "inf colour", "nan conic"])
def test_values_that_are_not_finite(what):
    scene = _scene(600, 3, (0.02, 0.2))
    at = 300   # some chunks before it, some after
    if what == "nan conic":
        scene[1][at] = (1e9, 1e4, 1e9)
        scene[2][at] = (0.8, 0.3, 0.4, 0.2)
    else:
        scene[4][at, 0, 1] = np.nan if what == "nan colour" else np.inf
        scene[1][at] = 0.05
    _check(scene, _cam(45, 30), RenderOptions(white_background=True))


@pytest.mark.parametrize("mode, threshold", [(0, 0.0), (0, 0.5), (0, 2.0), (1, 0.0), (1, 0.3), (1, 0.99), (1, 1.0),
                                             (1, 1.5)])
def test_termination_thresholds(mode, threshold):
    _check(_scene(300, 11, (0.1, 0.98)), _cam(45, 30), RenderOptions(term_mode=mode, term_threshold=threshold))
