"""The compositing adjoint's sums per splat (splat2d) against dense float64
autograd over the projected records: list lengths around the staging chunk and
the batch, image borders, opacities at the 0.99 clamp, with and without depth
and alpha gradients, and a tile that holds a value that is not finite.

The records, their order and the pixels are the forward's; nothing stops a
pixel (threshold 0). Tolerances: float32 sums with the hardware exponential
and reciprocal, each good to a few 1e-7, over transmittances that multiply up
to a few hundred factors 1 - alpha: 2e-4 of a column's largest entry; near the
clamp a relative error of alpha grows by 1 / (1 - 0.99): 5e-3."""
import ctypes as C

import numpy as np
import pytest

from lumen_b200.types import RenderOptions, ViewCamera

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scene(n, seed, opacity):
    g = torch.Generator().manual_seed(seed)
    u = lambda *s: torch.rand(s, generator=g)
    means = (u(n, 3) * 2 - 1) * torch.tensor([0.5, 0.35, 1.0]) + torch.tensor([0.0, 0.0, 4.0])
    scales = 0.02 * (0.4 / 0.02) ** u(n, 3)
    quats = torch.nn.functional.normalize(torch.randn(n, 4, generator=g), dim=1)
    op = opacity[0] + (opacity[1] - opacity[0]) * u(n)
    sh = 0.05 * torch.randn(n, 48, generator=g)
    sh[:, :3] += 0.5
    return [t.cuda().contiguous() for t in (means, scales, quats, op, sh)]


def _splat2d(scene, cam, opt, g_rgb, g_depth, g_alpha):
    from lumen_b200 import _lib as L
    from lumen_b200 import render as R
    r = R.render(*scene, cam, opt)
    n = scene[0].shape[0]
    grads = [torch.empty_like(t) for t in scene]
    splat2d = torch.empty((n, 12), device="cuda")
    out, img = L.LumenGpuGradients(), L.LumenGpuImage()
    out.means, out.scales, out.quats, out.opacities, out.sh = (t.data_ptr() for t in grads)
    out.splat2d = splat2d.data_ptr()
    img.rgb, img.depth, img.alpha, img.last_idx = (t.data_ptr() for t in (r.rgb, r.depth, r.alpha, r.last_idx))
    fs = r.frame.c_struct()
    ptr = lambda t: None if t is None else t.data_ptr()
    L.check(L.load().lumen_gpu_render_backward(
        C.byref(R.gaussians_struct(*scene)), C.byref(L.view_camera(cam)), C.byref(L.render_options(opt)),
        C.byref(fs), C.byref(img), g_rgb.data_ptr(), ptr(g_depth), ptr(g_alpha), C.byref(out),
        torch.cuda.current_stream().cuda_stream), "backward")
    return r, splat2d[:, :10].double()


def _dense(r, cam, opt, g_rgb, g_depth, g_alpha):
    """[n_visible, 10] gradients of sum(G . outputs) by autograd over the records."""
    rec = r.records.double()
    q = torch.stack([rec[:, k] for k in (0, 1, 4, 5, 6, 3, 8, 9, 10, 2)], 1).requires_grad_(True)
    order = torch.sort(torch.floor(r.records[:, 2] * 1000.0), stable=True).indices
    cx, cy, a, b, c, op, cr, cg, cb, z = q[order].unbind(1)
    py, px = torch.meshgrid(torch.arange(cam.height, device="cuda") + 0.5, torch.arange(cam.width, device="cuda") + 0.5,
                            indexing="ij")
    dx, dy = px.reshape(1, -1) - cx[:, None], py.reshape(1, -1) - cy[:, None]
    power = 0.5 * (a[:, None] * dx * dx + c[:, None] * dy * dy) + b[:, None] * dx * dy
    alpha = (op[:, None] * torch.exp(-power)).clamp_max(0.99)
    alpha = torch.where((power <= 4.5) & (alpha >= 0.00392156862), alpha, torch.zeros_like(alpha))
    logs = torch.log1p(-alpha)
    w = alpha * torch.exp(logs.cumsum(0) - logs)
    T = torch.exp(logs.sum(0))
    bg = T if opt.white_background else 0.0
    rgb = torch.stack([(w * v[:, None]).sum(0) + bg for v in (cr, cg, cb)], 1)
    total = (rgb * g_rgb.double().reshape(-1, 3)).sum()
    if g_depth is not None:
        total = total + ((w * z[:, None]).sum(0) * g_depth.double().reshape(-1)).sum()
    if g_alpha is not None:
        total = total + ((1.0 - T) * g_alpha.double().reshape(-1)).sum()
    return torch.autograd.grad(total, q)[0]


def _cam(w, h):
    return ViewCamera((0, 0, 0), (1, 0, 0, 0), 60, 60, w / 2, h / 2, 0.1, 100, w, h)


def _grads(cam, seed, depth, alpha):
    g = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g).cuda()
    return (rnd(cam.height, cam.width, 3), rnd(cam.height, cam.width) if depth else None,
            rnd(cam.height, cam.width) if alpha else None)


def _check(n, size, opacity, tol, depth, alpha, white):
    cam, opt = _cam(*size), RenderOptions(term_threshold=0.0, white_background=white)
    scene, up = _scene(n, n + size[0], opacity), _grads(cam, n, depth, alpha)
    r, got = _splat2d(scene, cam, opt, *up)
    want = _dense(r, cam, opt, *up)
    got = got[r.frame.visible_ids[:r.n_visible].long()]
    scale = want.abs().amax(0).clamp_min(1e-12)
    err = ((got - want).abs() / scale).amax(0)
    assert float(err.max()) <= tol, err.tolist()


@pytest.mark.parametrize("n", [1, 7, 127, 128, 129, 300])
@pytest.mark.parametrize("size", [(16, 16), (17, 3), (37, 26)])
def test_lists_around_the_chunk_and_the_batch(n, size):
    _check(n, size, (0.02, 0.5), 2e-4, depth=n % 2 == 1, alpha=n > 100, white=n == 128)


@pytest.mark.parametrize("n", [3, 60])
def test_opacities_at_the_clamp(n):
    _check(n, (37, 26), (0.9, 1.0), 5e-3, depth=False, alpha=True, white=False)


@pytest.mark.parametrize("where", ["colour", "upstream"])
def test_values_that_are_not_finite_stay_with_their_pixels(where):
    """One tile; the left half's splats do not reach the pixels of the right half."""
    cam, opt = _cam(16, 16), RenderOptions(term_threshold=0.0)
    scene = _scene(140, 5, (0.05, 0.5))
    scene[0][:, 0] = -0.35 + 0.01 * scene[0][:, 0]
    scene[1].mul_(0.3).clamp_max_(0.03)
    up = _grads(cam, 9, True, False)
    r, clean = _splat2d(scene, cam, opt, *up)
    if where == "colour":
        extra = [t[:1].clone() for t in scene]
        extra[0][0] = torch.tensor([0.4, 0.0, 3.0], device="cuda")
        extra[4][:] = float("nan")
        both = [torch.cat([a, b]).contiguous() for a, b in zip(scene, extra)]
    else:
        up[0][4, 15, 1] = float("inf")
        both = scene
    r2, got = _splat2d(both, cam, opt, *up)
    assert r.n_visible == 140 and bool(torch.isfinite(got[:140]).all())
    scale = clean.abs().amax(0).clamp_min(1e-12)
    assert float(((got[:140] - clean).abs() / scale).max()) <= 2e-5
