"""Ray casts that take the nearer child first return the hits of the reference's
order, bit for bit, where the order could show: equal distances, rays that
touch a sphere beside a face of its box, NaN positions and scales, distance
limits at and beyond the hits, and directions with vanishing components."""
import numpy as np
import pytest

import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def _check(means, scales, rays, max_dist):
    from lumen_b200 import spatial as S
    means, scales, rays = (np.ascontiguousarray(a, np.float32) for a in (means, scales, rays))
    with np.errstate(all="ignore"):
        nodes, idx, root, _ = O.bvh_build(means, scales)
        want = np.array([O.raycast(nodes, idx, root, means, scales, r[:3], r[3:], max_dist) for r in rays],
                        O.RAY_HIT_DTYPE)
    got = S.LBVH(_t(means), _t(scales)).raycast(_t(rays), max_dist=max_dist).cpu().numpy().view(np.uint32)
    exp = np.ascontiguousarray(want).view(np.uint32).reshape(-1, 6)
    bad = np.nonzero((got != exp).any(axis=1))[0]
    assert bad.size == 0, f"{bad.size} rays differ, first {bad[:5]}"
    return want


def _random(n, m, seed):
    rng = np.random.default_rng(seed)
    means = rng.normal(0, 3, (n, 3))
    scales = rng.uniform(0.01, 0.4, (n, 3))
    origins = rng.uniform(-12, 12, (m, 3))
    dirs = means[rng.integers(0, n, m)] - origins
    return means, scales, np.concatenate([origins, dirs], axis=1)


@pytest.mark.parametrize("n", [1, 2, 3, 1023, 1025, 6000])
def test_equal_distances(n):
    means, scales, rays = _random(n, 300, n)
    means = means[np.arange(n) % max(1, n // 3)]
    want = _check(means, scales, rays, 50.0)
    assert want["hit"].any()


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_rays_touching_spheres_beside_box_faces(axis):
    g = np.stack(np.meshgrid(*[np.arange(-4, 5)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    scales = np.full_like(g, 0.125)                 # spheres of radius 0.375, exact
    u, v = [k for k in range(3) if k != axis]
    rays = []
    for a in (-2.375, -1.625, 0.375, 0.37499997, 0.37500003, 1.0):
        for b in (-0.375, 0.0, 0.5, 3.375):
            for tilt in (0.0, 1e-8, -3e-7, 1e-5):
                o, d = np.zeros(3), np.zeros(3)
                o[u], o[v], o[axis], d[axis], d[u] = a, b, -9.0, 1.0, tilt
                rays.append(np.concatenate([o, d]))
    want = _check(g, scales, np.array(rays), 100.0)
    assert want["hit"].any() and not want["hit"].all()


def test_nan_positions_and_scales():
    means, scales, rays = _random(4000, 400, 5)
    means[7::97, 1] = np.nan
    scales[11::89, 0] = np.nan
    scales[13::311, 2] = np.inf
    _check(means, scales, rays, 60.0)


@pytest.mark.parametrize("max_dist", [0.0, 3.0, float("inf"), float("nan"), -1.0])
def test_distance_limits(max_dist):
    means, scales, rays = _random(3000, 200, 9)
    _check(means, scales, rays, max_dist)


def test_vanishing_directions_and_far_origins():
    means, scales, rays = _random(3000, 240, 21)
    rays[::6, 3:] = 0.0
    rays[1::6, 4] = 0.0
    rays[2::6, 4] = 1e-38 * rays[2::6, 4]
    rays[3::6, 3] *= 1e-7
    rays[4::6, :3] *= 1e4
    rays[4::6, 3:] = -rays[4::6, :3]
    rays[5, 0] = np.inf
    _check(means, scales, rays, 1e6)
