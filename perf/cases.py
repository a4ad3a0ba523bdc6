"""What this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` makes what a user's program has
in hand before the call (on the GPU, from a seed), ``run`` is one pass through
the public entry points and ``exact`` the same outputs in 64 bits, in plain
torch. Scene sizes, resolutions and distributions are those of the five
workloads of ``lumen_b200.scenes`` and of the tests' ragged images.

Kinds of case:

* ``frame``: one view through ``render.render`` with its work buffers kept,
  as a viewer or an evaluation loop calls it.
* ``batch``: several views through ``render.render_batch`` (an orbit of one
  scene, or views of two scenes at mixed resolutions).
* ``grad``: the differentiable step of a training loop: ``autograd.render``,
  ``autograd.l1_loss`` and ``backward`` to the five parameter tensors.
* ``pick``: a hierarchy built over a scene and a block of pixels picked
  through it (``spatial.LBVH``), as after an edit of the scene.
* ``serve``: a burst of requests to a render server that keeps the scene
  (``serve.Server``), host images out.
"""
import math

import numpy as np
import torch

from lumen_b200 import autograd, render, scenes, serve, spatial
from lumen_b200.types import RenderOptions, ViewCamera

#: What a case has unless it says otherwise: the parity defaults of RenderOptions.
DEFAULTS = {"layout": "box", "sh_degree": 3, "white": False, "key_mode": 0, "term_mode": 0, "logits": False,
            "orbit": False}


def _case(kind, **kw):
    return {"kind": kind, **DEFAULTS, **kw}


def listed():
    return [
        # the smallest frame: 512 Gaussians, 800x600, the reference's own demo size; launches and latency
        _case("frame", name="frame_512_800x600", n=512, width=800, height=600, layout="grid"),
        # a small scene in a small window, parameters as a trainer stores them
        _case("frame", name="frame_50k_640x480", n=50_000, width=640, height=480, logits=True, term_mode=1),
        # odd sizes, fewer SH coefficients, float depth keys, white background, a camera beside the scene
        _case("frame", name="frame_250k_1279x719", n=250_001, width=1279, height=719, sh_degree=2, key_mode=1,
              white=True, orbit=True),
        # the headline frame: 1M Gaussians at 1080p, stopping at alpha 0.99
        _case("frame", name="frame_1m_1920x1080", n=1_000_000, width=1920, height=1080, term_mode=1),
        # the largest frame: 2M Gaussians at 4K
        _case("frame", name="frame_2m_3840x2160", n=2_000_000, width=3840, height=2160, term_mode=1, orbit=True),
        # 64 orbit views of one scene at 720p, with every output
        _case("batch", name="batch_64x300k_1280x720", n=300_000, views=64, width=1280, height=720, term_mode=1),
        # 9 views of two scenes at mixed resolutions, images only (as a server batches requests)
        _case("batch", name="batch_9_mixed", n=100_000, n2=250_000, views=9, width=0, height=0, term_mode=1),
        # a training step on a subset: few Gaussians, a small image
        _case("grad", name="grad_2k_128x128", n=2_000, width=128, height=128, logits=True),
        # a training step at an odd image size, white background
        _case("grad", name="grad_100k_999x563", n=100_003, width=999, height=563, logits=True, white=True, orbit=True),
        # the training workload: 500k Gaussians at 1080p
        _case("grad", name="grad_500k_1920x1080", n=500_000, width=1920, height=1080, logits=True, term_mode=1),
        # build a hierarchy over 1M Gaussians and pick a 256x256 block of pixels
        _case("pick", name="pick_1m_65536", n=1_000_000, rays=65_536, width=1920, height=1080),
        # a burst of 16 requests for 1080p views of a resident scene of 1M Gaussians
        _case("serve", name="serve_16x1m_1920x1080", n=1_000_000, views=16, width=1920, height=1080, term_mode=1,
              orbit=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """An image about 16:9 to 1:1, odd as often as even."""
    w = _log_int(rng, lo, hi)
    return w, max(1, min(int(w * rng.uniform(0.5, 1.0)), hi * 9 // 16))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "batch", "grad", "grad", "pick", "serve"])
    c = _case(kind, logits=rng.random() < 0.4, term_mode=rng.randint(0, 1), key_mode=rng.choice([0, 0, 1]),
              white=rng.random() < 0.3, sh_degree=rng.choice([0, 1, 2, 3, 3, 3]), orbit=rng.random() < 0.5)
    if kind == "frame":
        w, h = _size(rng, 64, 3840)
        c.update(n=_log_int(rng, 512, 2_000_000), width=w, height=h)
    elif kind == "batch":
        w, h = _size(rng, 96, 1280)
        c.update(n=_log_int(rng, 1_000, 300_000), views=rng.randint(2, 40), width=w, height=h)
        if rng.random() < 0.4:
            c.update(n2=_log_int(rng, 1_000, 250_000), views=rng.randint(2, 12), width=0, height=0)
    elif kind == "grad":
        w, h = _size(rng, 64, 1920)
        c.update(n=_log_int(rng, 1_000, 500_000), width=w, height=h, logits=True)
    elif kind == "pick":
        c.update(n=_log_int(rng, 2_000, 1_000_000), rays=_log_int(rng, 64, 65_536), width=1920, height=1080)
    else:
        w, h = _size(rng, 320, 1920)
        c.update(n=_log_int(rng, 20_000, 1_000_000), views=rng.randint(1, 16), width=w, height=h, orbit=True)
    return c


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _scene(n, layout, logits, gen):
    """[means, scales, quats, opacities, sh] in float32: the distributions of
    scenes.grid_scene and scenes.box_scene, drawn on the GPU."""
    u = lambda *s: torch.rand(s, generator=gen, device="cuda")
    z = lambda *s: torch.randn(s, generator=gen, device="cuda")
    if layout == "grid":
        side = round(n ** (1.0 / 3.0))
        ax = torch.linspace(-1.0, 1.0, side, device="cuda")
        means = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
        means = means + 0.02 * z(n, 3) + torch.tensor([0.0, 0.0, 4.0], device="cuda")
        lo, hi, sigma = 0.02, 0.08, 1.0
    else:
        means = (2.0 * u(n, 3) - 1.0) * torch.tensor([3.0, 2.0, 3.0], device="cuda")
        means = means + torch.tensor([0.0, 0.0, 8.0], device="cuda")
        lo, hi, sigma = 0.003, 0.05, 1.5
    scales = math.log(lo) + u(n, 3) * (math.log(hi) - math.log(lo))
    quats = torch.nn.functional.normalize(z(n, 4), dim=1)
    opac = sigma * z(n)
    sh = 0.05 * z(n, 16, 3)
    sh[:, 0] = 0.5 + 0.15 * z(n, 3)
    if not logits:
        scales, opac = scales.exp(), opac.sigmoid()
    return [t.contiguous() for t in (means, scales, quats, opac, sh.reshape(n, 48))]


def _cameras(case, seed, count):
    """The case's cameras: in front of the scene, or on the orbit around it."""
    sizes = [(case["width"], case["height"])] * count
    if not case["width"]:
        sizes = [scenes.SERVING_RESOLUTIONS[i % 3] for i in range(count)]
    fov = 60.0 if case["layout"] == "grid" else 50.0
    if count == 1 and not case["orbit"]:
        return [ViewCamera.from_fov(*sizes[0], fov)]
    phase = (int(seed) % 997) / 997.0 * 2.0 * math.pi
    orbit = scenes.orbit_cameras(max(count, 4), 64, 64, fov, phase=phase)
    return [ViewCamera.from_fov(w, h, fov, position=c.position, rotation=c.rotation)
            for (w, h), c in zip(sizes, orbit)]


def _options(case):
    return RenderOptions(sh_degree=case["sh_degree"], white_background=case["white"], key_mode=case["key_mode"],
                         term_mode=case["term_mode"], params_are_logits=case["logits"])


def _target(case, gen):
    """A photograph's stand-in: a smooth image and sensor noise, in [0, 1]."""
    coarse = torch.rand((1, 3, 9, 16), generator=gen, device="cuda")
    img = torch.nn.functional.interpolate(coarse, size=(case["height"], case["width"]), mode="bilinear")
    img = img[0].permute(1, 2, 0) + 0.02 * torch.randn((case["height"], case["width"], 3), generator=gen, device="cuda")
    return img.clamp(0.0, 1.0).contiguous()


def _inputs(case, seed):
    gen = _generator(seed)
    groups = [_scene(case["n"], case["layout"], case["logits"], gen)]
    if case.get("n2"):
        groups.append(_scene(case["n2"], case["layout"], case["logits"], gen))
    cams = _cameras(case, seed, case.get("views", 1))
    return groups, cams, gen


def _pixels(case, gen):
    """A square block of pixel centres at a place drawn from the seed."""
    side = max(1, math.isqrt(case["rays"]))
    at = torch.rand(2, generator=gen, device="cuda").cpu()
    x0, y0 = float(at[0]) * (case["width"] - side), float(at[1]) * (case["height"] - side)
    k = torch.arange(case["rays"], device="cuda")
    return torch.stack([math.floor(x0) + (k % side) + 0.5, math.floor(y0) + (k // side) + 0.5], 1).float()


def prepare(case, seed):
    groups, cams, gen = _inputs(case, seed)
    st = {"kind": case["kind"], "options": _options(case), "cameras": cams, "frame": None}
    if case["kind"] == "frame":
        st["params"] = groups[0]
    elif case["kind"] == "grad":
        st["params"] = [t.requires_grad_(True) for t in groups[0]]
        st["target"] = _target(case, gen)
    elif case["kind"] == "pick":
        st["params"], st["pixels"] = groups[0], _pixels(case, gen)
    elif case["kind"] == "batch":
        owned = [render.Scene(*g) for g in groups]
        st["views"] = [(owned[i % len(owned)], c) for i, c in enumerate(cams)]
        st["images"], st["outputs"] = _batch_outputs(case, cams)
    else:
        st["server"] = serve.Server(work_budget_bytes=4 << 30, autotune=False, options=st["options"])
        st["scene"] = st["server"].add_scene(render.Scene(*groups[0]))
        st["out"] = [torch.empty((c.height, c.width, 3), dtype=torch.uint8, pin_memory=True) for c in cams]
    return st


def _batch_outputs(case, cams):
    """The views' images. One resolution: slices of stacked tensors, every
    output. Mixed resolutions: an image, depth and alpha per view."""
    if not case["width"]:
        e = lambda c, *s: torch.empty((c.height, c.width, *s), dtype=torch.float32, device="cuda")
        images = [render.ViewImage(e(c, 3), e(c), e(c), None, None) for c in cams]
        return images, [{"rgb": i.rgb, "depth": i.depth, "alpha": i.alpha} for i in images]
    shape = (len(cams), case["height"], case["width"])
    f = lambda *s: torch.empty(shape + s, dtype=torch.float32, device="cuda")
    i = lambda: torch.empty(shape, dtype=torch.int32, device="cuda")
    out = {"rgb": f(3), "depth": f(), "alpha": f(), "n_contrib": i(), "last_idx": i()}
    return [render.ViewImage(*(out[k][v] for k in ("rgb", "depth", "alpha", "n_contrib", "last_idx")))
            for v in range(len(cams))], out


# ---------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "frame":
        r = render.render(*state["params"], state["cameras"][0], state["options"], frame=state["frame"])
        state["frame"] = r.frame
        return {"rgb": r.rgb, "depth": r.depth, "alpha": r.alpha, "n_contrib": r.n_contrib, "last_idx": r.last_idx,
                "n_visible": r.n_visible, "n_instances": r.n_instances}
    if kind == "batch":
        r = render.render_batch(state["views"], state["options"], frame=state["frame"], images=state["images"])
        state["frame"] = r.frame
        return state["outputs"]
    if kind == "grad":
        rgb, _, _ = autograd.render(*state["params"], state["cameras"][0], state["options"])
        loss = autograd.l1_loss(rgb, state["target"])
        grads = torch.autograd.grad(loss, state["params"])
        return {"loss": loss.detach(), "rgb": rgb.detach(), "means": grads[0], "scales": grads[1], "quats": grads[2],
                "opacities": grads[3], "sh": grads[4]}
    if kind == "pick":
        bvh = spatial.LBVH(state["params"][0], state["params"][1])
        return bvh.pick(state["cameras"][0], state["pixels"])
    requests = [state["server"].submit(state["scene"], c, o) for c, o in zip(state["cameras"], state["out"])]
    return [r.result().image for r in requests]


# ---------------------------------------------------------------- work

def _pixels_of(case):
    return sum(c.width * c.height for c in _cameras(case, 0, case.get("views", 1)))


def _blends(n, width, height):
    """Splats blended per pixel: those whose 4.5-power ellipse covers it
    (screen variance from the mean squared scale at the box's distance), up
    to about 40, where a pixel of these scenes is opaque."""
    var = 0.000443 * (1.072 * height / 8.0) ** 2 + 0.3
    return min(40.0, n * 9.0 * math.pi * var / (width * height))


def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "pick":
        # positions and scales read, one hit per ray written; a box test per level and ray at least
        return {"bytes": 24.0 * n + 32.0 * case["rays"], "flops": 30.0 * case["rays"] * math.log2(n) + 40.0 * n}
    cams = _cameras(case, 0, case.get("views", 1))
    sizes = [case["n"], case.get("n2", case["n"])]
    flops = 0.0
    for i, c in enumerate(cams):
        m = sizes[i % 2]
        # projection and degree-3 colour per Gaussian; about 25 operations per blended splat and pixel
        flops += 500.0 * m + 25.0 * c.width * c.height * _blends(m, c.width, c.height)
    pix = float(sum(c.width * c.height for c in cams))
    read = 236.0 * (n + case.get("n2", 0))
    if kind == "serve":
        return {"bytes": read + 3.0 * pix, "flops": flops}
    if kind == "grad":
        # parameters read, gradients written; the target read, the image written; the adjoint is twice the forward
        return {"bytes": 2.0 * read + 24.0 * pix, "flops": 3.0 * flops}
    return {"bytes": read + (28.0 if case["width"] else 20.0) * pix, "flops": flops}


# ---------------------------------------------------------------- in 64 bits

#: (tile, splat, pixel) triples held at once
TRIPLES = 24_000_000
MIN_ALPHA = 0.00392156862


def _normalized(q):
    return q / q.norm(dim=-1, keepdim=True)


def _rotation(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).reshape(q.shape[:-1] + (3, 3))


def _sh_colour(sh, d, degree):
    x, y, z = d.unbind(-1)
    xx, yy, zz = x * x, y * y, z * z
    one = torch.ones_like(x)
    Y = [0.28209479177387814 * one, -0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x,
         1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
         -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy), -0.5900435899266435 * y * (3 * xx - yy),
         2.890611442640554 * x * y * z, -0.4570457994644658 * y * (4 * zz - xx - yy),
         0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy), -0.4570457994644658 * x * (4 * zz - xx - yy),
         1.445305721320277 * z * (xx - yy), -0.5900435899266435 * x * (xx - 3 * yy)]
    k = (degree + 1) ** 2
    return (0.5 + (sh.reshape(-1, 16, 3)[:, :k] * torch.stack(Y[:k], -1)[..., None]).sum(1)).clamp(0.0, 1.0)


def _project64(p, cam, case):
    """Screen centres, conics, depths, opacities, colours and 3-sigma radii
    of all Gaussians and which of them are visible, in the type of ``p``."""
    means, scales, quats, opac, sh = p
    if case["logits"]:
        scales, opac = scales.exp(), opac.sigmoid()
    f32 = lambda v: torch.tensor(np.float32(v), dtype=torch.float64, device="cuda")
    pos, W = f32(cam.position), _rotation(_normalized(f32(cam.rotation))).T
    fx, fy, cx, cy = (float(np.float32(v)) for v in (cam.fx, cam.fy, cam.cx, cam.cy))
    v = means - pos
    x, y, z = (v @ W.T).unbind(-1)
    seen = (z >= cam.near_plane) & (z <= cam.far_plane) & (opac >= MIN_ALPHA)
    zs = torch.where(seen, z, torch.ones_like(z))
    M = _rotation(_normalized(quats)) * scales.clamp_min(1e-5)[:, None, :]
    zero = torch.zeros_like(zs)
    J = torch.stack([fx / zs, zero, -fx * x / zs ** 2, zero, fy / zs, -fy * y / zs ** 2], -1).reshape(-1, 2, 3)
    T = J @ W @ M
    S = T @ T.transpose(1, 2)
    a, b, c = S[:, 0, 0] + 0.3, S[:, 0, 1], S[:, 1, 1] + 0.3
    det = a * c - b * b
    u, w = fx * x / zs + cx, fy * y / zs + cy
    with torch.no_grad():
        r = torch.ceil(3.0 * torch.sqrt(0.5 * (a + c) + torch.sqrt((0.5 * (a - c)) ** 2 + b * b)))
        seen = seen & (u + r >= 0) & (u - r < cam.width) & (w + r >= 0) & (w - r < cam.height)
    col = _sh_colour(sh, _normalized(v), case["sh_degree"])
    return torch.stack([u, w, z, opac, c / det, -b / det, a / det], -1), col, r, seen


def _instances(geo, r, seen, cam, key_mode):
    """Splat of every (tile, splat) pair in tile order, front to back within
    a tile, with the tiles' starts and counts."""
    idx = torch.nonzero(seen).flatten()
    u, w, z, rr = geo[idx, 0], geo[idx, 1], geo[idx, 2], r[idx]
    key = z if key_mode == 1 else torch.floor(z * 1000.0)
    idx = idx[torch.sort(key, stable=True).indices]
    u, w, rr = geo[idx, 0], geo[idx, 1], r[idx]
    x0, x1 = ((u + s * rr).clamp(0, cam.width - 1).floor().long() // 16 for s in (-1, 1))
    y0, y1 = ((w + s * rr).clamp(0, cam.height - 1).floor().long() // 16 for s in (-1, 1))
    nx = x1 - x0 + 1
    cnt = nx * (y1 - y0 + 1)
    which = torch.repeat_interleave(torch.arange(idx.numel(), device="cuda"), cnt)
    k = torch.arange(which.numel(), device="cuda") - (cnt.cumsum(0) - cnt)[which]
    tile = (y0[which] + k // nx[which]) * cam.tiles_x + x0[which] + k % nx[which]
    order = torch.sort(tile, stable=True).indices
    counts = torch.bincount(tile, minlength=cam.n_tiles)
    return idx[which[order]], counts.cumsum(0) - counts, counts


def _tile_batches(counts, triples=TRIPLES):
    """Tiles grouped by list length, so that the padded lists stay near ``triples``."""
    order = torch.argsort(counts, descending=True)
    lens = counts[order].tolist()
    k = 0
    while k < len(lens) and lens[k] > 0:
        b = max(1, min(len(lens) - k, triples // (256 * lens[k])))
        yield order[k:k + b], lens[k]
        k += b


def _blend(geo, col, splat, starts, counts, tiles, longest, cam, case):
    """(rgb and depth [tiles, 256, 4], alpha [tiles, 256]) and the pixels."""
    j = torch.arange(longest, device="cuda")
    inside = j[None] < counts[tiles][:, None]
    s = splat[(starts[tiles][:, None] + j[None]).clamp_max(splat.numel() - 1)]
    q = torch.arange(256, device="cuda")
    px = (tiles % cam.tiles_x)[:, None] * 16 + (q % 16)[None]
    py = (tiles // cam.tiles_x)[:, None] * 16 + (q // 16)[None]
    g = geo[s][..., None]                                            # [tiles, longest, 7, 1]
    dx, dy = px[:, None] + 0.5 - g[:, :, 0], py[:, None] + 0.5 - g[:, :, 1]
    power = (0.5 * (g[:, :, 4] * dx * dx + g[:, :, 6] * dy * dy) + g[:, :, 5] * dx * dy).clamp_min(0.0)
    alpha = (g[:, :, 3] * torch.exp(-power)).clamp_max(0.99)
    alpha = torch.where((power <= 4.5) & (alpha >= MIN_ALPHA) & inside[..., None], alpha, torch.zeros_like(alpha))
    logs = torch.log1p(-alpha)
    total = logs.cumsum(1)
    before = torch.exp(total - logs)
    with torch.no_grad():
        live = before.detach() > 1e-4 if case["term_mode"] == 0 else 1.0 - before.detach() < 0.99
    wgt = torch.where(live, alpha * before, torch.zeros_like(alpha))
    feat = torch.cat([col, geo[:, 2:3]], 1)[s]                       # r, g, b, depth
    out = torch.einsum("tlp,tlc->tpc", wgt, feat)
    T = torch.exp(torch.where(live, logs, torch.zeros_like(logs)).sum(1))
    return out, T, px, py


def _finish(out, T, case, any_instance):
    rgb = out[..., :3] + (T[..., None] if case["white"] and any_instance else 0.0)
    return rgb, out[..., 3], 1.0 - T


def _render64(p, cam, case):
    geo, col, r, seen = _project64(p, cam, case)
    splat, starts, counts = _instances(geo, r, seen, cam, case["key_mode"])
    h, w = cam.height, cam.width
    some = splat.numel() > 0
    rgb = torch.full((h, w, 3), 1.0 if case["white"] and some else 0.0, dtype=torch.float64, device="cuda")
    depth, alpha = (torch.zeros((h, w), dtype=torch.float64, device="cuda") for _ in range(2))
    for tiles, longest in _tile_batches(counts):
        o, T, px, py = _blend(geo, col, splat, starts, counts, tiles, longest, cam, case)
        c, d, a = _finish(o, T, case, some)
        ok = (px < w) & (py < h)
        rgb[py[ok], px[ok]], depth[py[ok], px[ok]], alpha[py[ok], px[ok]] = c[ok], d[ok], a[ok]
    return rgb, depth, alpha


def _grad64(params, cam, case, target):
    """Loss, image and the gradients of the L1 step: the blended tiles back
    to the projected splats one group of tiles at a time, then through the
    projection."""
    leaf = [t.requires_grad_(True) for t in params]
    geo, col, r, seen = _project64(leaf, cam, case)
    with torch.no_grad():
        rgb = _render64(leaf, cam, case)[0]
        splat, starts, counts = _instances(geo, r, seen, cam, case["key_mode"])
    diff = rgb - target.double()
    up = torch.where(diff >= 0, 1.0, -1.0).double() / diff.numel()
    g2, c2 = geo.detach().requires_grad_(True), col.detach().requires_grad_(True)
    total = [torch.zeros_like(g2), torch.zeros_like(c2)]
    for tiles, longest in _tile_batches(counts, TRIPLES // 4):
        o, T, px, py = _blend(g2, c2, splat, starts, counts, tiles, longest, cam, case)
        ok = (px < cam.width) & (py < cam.height)
        got = torch.autograd.grad((_finish(o, T, case, True)[0][ok] * up[py[ok], px[ok]]).sum(), [g2, c2])
        for t, x in zip(total, got):
            t += x
    grads = torch.autograd.grad([geo, col], leaf, total)
    return diff.abs().mean(), rgb, grads


def exact(case, seed):
    """What ``run`` returns, in 64 bits: images, depths, alphas and gradients.
    Picks and served bytes are whole numbers and have no such value."""
    if case["kind"] in ("pick", "serve"):
        return None
    groups, cams, gen = _inputs(case, seed)
    wide = [[t.double() for t in g] for g in groups]
    if case["kind"] == "grad":
        loss, rgb, g = _grad64(wide[0], cams[0], case, _target(case, gen))
        return {"loss": loss, "rgb": rgb, "means": g[0], "scales": g[1], "quats": g[2], "opacities": g[3], "sh": g[4]}
    views = [_render64(wide[i % len(wide)], c, case) for i, c in enumerate(cams)]
    none = {"n_contrib": None, "last_idx": None}
    if case["kind"] == "frame":
        return {"rgb": views[0][0], "depth": views[0][1], "alpha": views[0][2], "n_visible": None,
                "n_instances": None, **none}
    if not case["width"]:
        return [dict(zip(("rgb", "depth", "alpha"), v)) for v in views]
    return {k: torch.stack([v[i] for v in views]) for i, k in enumerate(("rgb", "depth", "alpha"))} | none
