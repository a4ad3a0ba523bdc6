"""Casts through a hierarchy that is not as its build left it for the
Gaussians as they are now: positions or scales changed in place since, links
exchanged, boxes changed. The hits are those of the reference's order over the
nodes and the Gaussians as they are, bit for bit."""
import numpy as np
import pytest

import oracle as O
from test_gpu_raycast_order import _random, _t

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _moved(means, scales, rng):
    means += rng.normal(0, 0.5, means.shape)


def _one_moved(means, scales, rng):
    means[means.shape[0] // 2] += 2.0


def _grown(means, scales, rng):
    scales *= 3.0


@pytest.mark.parametrize("change", [_moved, _one_moved, _grown])
@pytest.mark.parametrize("n,m", [(1, 40), (7, 40), (3000, 400), (70_000, 100)])
def test_gaussians_changed_since_the_build(change, n, m):
    from lumen_b200 import spatial as S
    means, scales, rays = (np.ascontiguousarray(a, np.float32) for a in _random(n, m, n))
    bvh = S.LBVH(_t(means), _t(scales))
    nodes, idx, root, _ = O.bvh_build(means, scales)
    change(means, scales, np.random.default_rng(n))
    bvh.means.copy_(_t(means))
    bvh.scales.copy_(_t(scales))
    _same(bvh, nodes, idx, root, means, scales, rays)


def _same(bvh, nodes, idx, root, means, scales, rays):
    want = np.array([O.raycast(nodes, idx, root, means, scales, r[:3], r[3:], 60.0) for r in rays], O.RAY_HIT_DTYPE)
    got = bvh.raycast(_t(rays), max_dist=60.0).cpu().numpy().view(np.uint32)
    bad = np.nonzero((got != np.ascontiguousarray(want).view(np.uint32).reshape(-1, 6)).any(axis=1))[0]
    assert bad.size == 0, f"{bad.size} rays differ, first {bad[:5]}"


@pytest.mark.parametrize("what", ["links", "box", "leaf"])
def test_nodes_of_the_callers_own(what):
    """Equal distances, so that the order of the leaves shows."""
    from lumen_b200 import spatial as S
    n = 3000
    means, scales, rays = (np.ascontiguousarray(a, np.float32) for a in _random(n, 400, 77))
    means = np.ascontiguousarray(means[np.arange(n) % (n // 3)])
    bvh = S.LBVH(_t(means), _t(scales))
    nodes, idx, root, _ = O.bvh_build(means, scales)
    raw = np.ascontiguousarray(nodes).view(np.int32).reshape(-1, 8)      # a view: the oracle sees the change
    if what == "links":
        rows = np.arange(n, raw.shape[0])[raw[n:, 7] >= 0][::3]
        raw[rows, 3], raw[rows, 7] = raw[rows, 7].copy(), raw[rows, 3].copy()
    elif what == "box":
        raw.view(np.float32)[n + 5 :: 50, 4] -= 1.0
    else:
        raw.view(np.float32)[0:n:20, 0:3] += 0.05
    bvh.nodes.copy_(torch.from_numpy(raw).cuda())
    _same(bvh, raw.reshape(-1).view(nodes.dtype), idx, root, means, scales, rays)


@pytest.mark.parametrize("n", [1, 256, 257, 4096, 4097, 8193])
def test_many_rays_at_once_hit_what_few_do(n):
    """A thread per ray and eight lanes per ray, by the numbers of Gaussians and of rays."""
    from lumen_b200 import spatial as S
    from lumen_b200.types import ViewCamera
    means, scales, rays = _random(n, 33_000, n)
    means[n // 2] = means[0]
    bvh, rays = S.LBVH(_t(means), _t(scales)), _t(rays)
    few = torch.cat([bvh.raycast(rays[k:k + 3000], max_dist=40.0) for k in range(0, rays.shape[0], 3000)])
    assert torch.equal(bvh.raycast(rays, max_dist=40.0), few)
    cam = ViewCamera.from_fov(200, 200, 60.0, position=(0.0, 0.0, -9.0))
    px = torch.rand((140_000, 2), device="cuda", generator=torch.Generator("cuda").manual_seed(n)) * 200.0
    made, made_few = torch.empty((140_000, 6), device="cuda"), torch.empty((140_000, 6), device="cuda")
    few = torch.cat([bvh.pick(cam, px[k:k + 20_000], rays_out=made_few[k:k + 20_000]) for k in range(0, 140_000, 20_000)])
    assert torch.equal(bvh.pick(cam, px, rays_out=made), few) and torch.equal(made, made_few)
