"""The compositing adjoint's sums (splat2d) Gaussian by Gaussian: sums over a
whole screen, the order of the additions within a tile, and large and
needle-like splats against 64 bits."""
import pytest

from lumen_b200.types import RenderOptions, ViewCamera
from test_gpu_backward_sums import _cam, _grads, _scene, _splat2d

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _forward_power(records, px, py):
    """The forward's power [splats, pixels], each operation rounded to 32 bits as there."""
    cx, cy, a, b, c = (records[:, k][:, None] for k in (0, 1, 4, 5, 6))
    dx, dy = px.reshape(1, -1) - cx, py.reshape(1, -1) - cy
    return ((0.5 * a) * dx) * dx + (b * dx) * dy + ((0.5 * c) * dy) * dy


def test_whole_screen_splats_are_summed_tile_by_tile():
    """Splats of nearly constant alpha over 1080p under a constant gradient: a
    colour's gradient is a sum of 2 M nearly equal terms. Added tile by tile
    (8160 additions to a running sum that grows evenly, each rounded by at most
    2^-24 of it) its error is at most 8160 / 2 * 2^-24 = 2.4e-4, and 2e-6 for
    the terms themselves; 16 blocks per tile one by one could be 16 times off."""
    n, cam = 6, ViewCamera((0, 0, 0), (1, 0, 0, 0), 1000, 1000, 960, 540, 0.1, 100, 1920, 1080)
    opt = RenderOptions(term_threshold=0.0)
    k = torch.arange(n, device="cuda")
    means = torch.stack([0.1 * k, -0.1 * k, 4.0 + 0.25 * k], 1).float().contiguous()
    scales = torch.full((n, 3), 1000.0, device="cuda")
    quats = torch.tensor([[1.0, 0.0, 0.0, 0.0]], device="cuda").repeat(n, 1)
    op = 0.05 + 0.017 * k.float()
    sh = torch.zeros((n, 48), device="cuda")
    g_rgb = torch.tensor([0.7, -1.3, 0.37], device="cuda").expand(1080, 1920, 3).contiguous()
    r, got = _splat2d([means, scales, quats, op, sh], cam, opt, g_rgb, None, None)
    rec = r.records.double()
    assert r.n_visible == n and r.n_instances == n * 8160
    ys, xs = torch.arange(1080, device="cuda") + 0.5, torch.arange(1920, device="cuda") + 0.5
    T = torch.ones((1080, 1920), dtype=torch.float64, device="cuda")
    for j in range(n):                                     # in depth order, as the means are
        dx, dy = xs[None, :] - rec[j, 0], ys[:, None] - rec[j, 1]
        power = 0.5 * (rec[j, 4] * dx * dx + rec[j, 6] * dy * dy) + rec[j, 5] * dx * dy
        alpha = rec[j, 3] * torch.exp(-power)
        want = g_rgb[0, 0].double() * (alpha * T).sum()
        assert float(((got[j, 6:9] - want) / want).abs().max()) <= 2.5e-4
        T = T * (1.0 - alpha)


def test_a_tiles_sums_do_not_depend_on_the_order_of_its_warps():
    cam, opt = _cam(16, 16), RenderOptions(term_threshold=0.0)
    scene, up = _scene(300, 11, (0.02, 0.5)), _grads(cam, 11, True, True)
    first = _splat2d(scene, cam, opt, *up)[1]
    assert all(bool((_splat2d(scene, cam, opt, *up)[1] == first).all()) for _ in range(20))


def test_rows_of_large_and_needle_like_splats():
    """Each gradient of each splat, in units of the sum of its terms' sizes:
    every factor of a term is good to 1e-6 (the hardware exponential and its
    argument, the reciprocal), and the transmittance is a product over up to 60
    splats: 6e-5."""
    n, cam, opt = 60, _cam(333, 187), RenderOptions(term_threshold=0.0)
    scene = _scene(n, 3, (0.05, 0.5))
    scene[1][::2, 0] = 2.0
    scene[1][::2, 1:] = 0.01
    scene[1][1::4] = 0.7
    up = _grads(cam, 3, True, True)
    r, got = _splat2d(scene, cam, opt, *up)
    got = got[r.frame.visible_ids[:r.n_visible].long()]
    rec = r.records.double()
    order = torch.sort(torch.floor(r.records[:, 2] * 1000.0), stable=True).indices
    cx, cy, a, b, c, op = (rec[order, k][:, None] for k in (0, 1, 4, 5, 6, 3))
    feat = rec[order][:, [8, 9, 10, 2]]
    py, px = torch.meshgrid(torch.arange(cam.height, device="cuda") + 0.5, torch.arange(cam.width, device="cuda") + 0.5,
                            indexing="ij")
    dx, dy = px.reshape(1, -1) - cx, py.reshape(1, -1) - cy
    power = _forward_power(r.records[order], px, py)
    assert float(power.min()) >= 0.0
    alpha = op * torch.exp(-power.double())
    alpha = torch.where((power <= 4.5) & (alpha >= 0.00392156862), alpha, torch.zeros_like(alpha))
    G = torch.cat([up[0].double().reshape(-1, 3), up[1].double().reshape(-1, 1)], 1)
    before = torch.cat([torch.ones_like(alpha[:1]), torch.cumprod(1.0 - alpha, 0)[:-1]])
    w, T = alpha * before, before[-1] * (1.0 - alpha[-1])

    behind = lambda v: (w * v).flip(0).cumsum(0).flip(0) - w * v       # what is blended behind each splat
    gcol, g_alpha = feat @ G.T, up[2].double().reshape(1, -1)
    s = alpha * (before * gcol + (g_alpha * T - behind(gcol)) / (1.0 - alpha))
    sizes = feat.abs() @ G.T.abs()
    size = alpha * (before * sizes + (g_alpha.abs() * T + behind(sizes)) / (1.0 - alpha))
    geo = [a * dx + b * dy, b * dx + c * dy, -0.5 * dx * dx, -dx * dy, -0.5 * dy * dy, 1.0 / op]
    abs_geo = [(a * dx).abs() + (b * dy).abs(), (b * dx).abs() + (c * dy).abs()] + [v.abs() for v in geo[2:]]
    want = torch.stack([(s * v).sum(1) for v in geo] + [(w * G[:, k]).sum(1) for k in range(4)], 1)
    scale = torch.stack([(size * v).sum(1) for v in abs_geo] + [(w * G[:, k].abs()).sum(1) for k in range(4)], 1)
    err = (got[order] - want).abs() / scale.clamp_min(1e-12)
    assert float(err.max()) <= 6e-5, err.amax(0).tolist()


def test_a_power_clamped_at_zero_moves_neither_centre_nor_conic():
    """Needles without a low pass, whose conics come out indefinite: where the
    power is below 0 the forward takes the constant 0, so a splat that is
    blended at such pixels alone gets a gradient for its opacity and none for
    its centre and conic."""
    n, cam, opt = 40, _cam(37, 26), RenderOptions(term_threshold=0.0, lowpass=0.0)
    scene = _scene(n, 21, (0.05, 0.5))
    scene[1][:, 0] = 2.0
    scene[1][:, 1:] = 1e-5
    r, got = _splat2d(scene, cam, opt, *_grads(cam, 21, False, False))
    got = got[r.frame.visible_ids[:r.n_visible].long()]
    py, px = torch.meshgrid(torch.arange(cam.height, device="cuda") + 0.5, torch.arange(cam.width, device="cuda") + 0.5,
                            indexing="ij")
    power = _forward_power(r.records, px, py)
    only_clamped = (power < 0.0).any(1) & ~((power >= 0.0) & (power <= 4.5)).any(1)
    assert int(only_clamped.sum()) >= 5
    assert bool((got[only_clamped][:, :5] == 0.0).all()) and bool((got[only_clamped][:, 5] != 0.0).all())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_an_upstream_value_that_is_not_finite_stays_with_the_splats_its_pixel_blends(value):
    """A splat that reaches the upper left 4x4 block but not its first pixel
    (2.8 pixels away; a 3-sigma radius of 1.65): that pixel's gradient is none
    of its business."""
    cam, opt = _cam(16, 16), RenderOptions(term_threshold=0.0)
    scene = [t.cuda().contiguous() for t in (
        torch.tensor([[(2.5 - 8) / 60 * 4, (2.5 - 8) / 60 * 4, 4.0]]), torch.full((1, 3), 1e-4),
        torch.tensor([[1.0, 0.0, 0.0, 0.0]]), torch.tensor([0.5]), torch.full((1, 48), 0.1))]
    up = _grads(cam, 4, True, False)
    r, clean = _splat2d(scene, cam, opt, *up)
    assert int(r.n_contrib[0, 0]) == 0 and int(r.n_contrib[2, 2]) == 1
    up[0][0, 0, 1] = value
    up[1][0, 0] = value
    got = _splat2d(scene, cam, opt, *up)[1]
    assert float(((got - clean).abs() / clean.abs().amax().clamp_min(1e-12)).max()) <= 2e-5
