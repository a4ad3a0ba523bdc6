"""The depth sort of small frames (one cluster, up to 131072 Gaussians) against
the oracle's order: one CTA and eight, the edges of the keys per thread, the
largest size and the first one beyond it; many distinct depths and few."""
import os

import numpy as np
import pytest

import oracle as O
from lumen_b200.types import RenderOptions, ViewCamera

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NT = max(1, min(16, os.cpu_count() or 1))


@pytest.mark.parametrize("depths", [0, 5])
@pytest.mark.parametrize("n", [2, 1024, 1025, 8192, 8193, 50_001, 131_072, 131_073])
def test_depth_order(n, depths):
    from lumen_b200 import render as R
    rng = np.random.Generator(np.random.PCG64(n + depths))
    f = np.float32
    z = rng.uniform(0.5, 60.0, n) if not depths else rng.integers(1, 1 + depths, n)
    means = (rng.uniform(-0.4, 0.4, (n, 3)) * z[:, None]).astype(f)
    means[:, 2] = z
    scales = np.full((n, 3), 0.002, f)
    quats = np.tile(np.array([1, 0, 0, 0], f), (n, 1))
    op = rng.uniform(0.01, 0.05, n).astype(f)
    sh = np.zeros((n, 16, 3), f)
    cam, opt = ViewCamera((0, 0, 0), (1, 0, 0, 0), 40, 40, 20, 20, 0.1, 100, 40, 40), RenderOptions()
    o = O.render(means, scales, quats, op, sh, cam, opt, nthreads=NT)
    dev = lambda a: torch.from_numpy(a).cuda()
    g = R.render(dev(means), dev(scales), dev(quats), dev(op), dev(sh).reshape(-1, 48), cam, opt)
    assert g.n_visible == o.n_visible and g.n_instances == o.n_instances > 0
    assert np.array_equal(g.sorted_keys.cpu().numpy().view(np.uint64), o.keys_sorted)
    assert np.array_equal(g.sorted_vals.cpu().numpy().view(np.uint32), o.vals_sorted)
