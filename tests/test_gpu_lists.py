"""The tiles' splat lists, entry by entry: cells cut by the image border, list
lengths around a segment, frames whose scratch is too small for the segments'
notes or the cells' ranges, batches with more cells than a packed key can name,
and emission tickets of one and of several rounds."""
import ctypes as C
import os

import numpy as np
import pytest

import oracle as O
from lumen_b200 import _lib as L
from lumen_b200 import scenes
from lumen_b200.types import RenderOptions, ViewCamera

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

NT = max(1, min(16, os.cpu_count() or 1))


def _scene(n, seed, scale=(0.02, 0.4), spread=(0.9, 0.6)):
    rng = np.random.Generator(np.random.PCG64(seed))
    means = rng.uniform(-1.0, 1.0, size=(n, 3)) * [spread[0], spread[1], 1.0] + [0.0, 0.0, 4.0]
    scales = np.exp(rng.uniform(np.log(scale[0]), np.log(scale[1]), size=(n, 3)))
    quats = rng.standard_normal(size=(n, 4))
    op = rng.uniform(0.02, 0.2, size=n)
    sh = rng.normal(0.0, 0.1, size=(n, 16, 3))
    f = np.float32
    return [a.astype(f) for a in (means, scales, quats, op, sh)]


def _dev(scene):
    means, scales, quats, op, sh = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in scene)
    return means, scales, quats, op, sh.reshape(-1, 48)


def _cam(w, h, f=None):
    f = f or 1.2 * max(w, h)
    return ViewCamera((0, 0, 0), (1, 0, 0, 0), f, f, w / 2, h / 2, 0.1, 100, w, h)


def _check(scene, cam):
    from lumen_b200 import render as R
    g = R.render(*_dev(scene), cam, RenderOptions())
    o = O.render(*scene, cam, RenderOptions(), nthreads=NT)
    assert g.n_instances == o.n_instances > 0
    assert np.array_equal(g.sorted_keys.cpu().numpy().view(np.uint64), o.keys_sorted)
    assert np.array_equal(g.sorted_vals.cpu().numpy().view(np.uint32), o.vals_sorted)
    assert np.array_equal(g.rgb.cpu().numpy().view(np.uint32), o.rgb.view(np.uint32))


@pytest.mark.parametrize("size", [(16, 16), (49, 33), (64, 64), (65, 127), (321, 16), (16, 321), (250, 190)])
def test_cells_at_the_image_border(size):
    _check(_scene(300, size[0]), _cam(*size))


@pytest.mark.parametrize("n", [1, 255, 256, 257, 2047, 2048, 2049, 4100])
def test_lists_around_a_segment(n):
    """One cell of 4x4 tiles, every splat in front of it: one list of n pairs."""
    _check(_scene(n, n, spread=(0.3, 0.3)), _cam(64, 64))


@pytest.mark.parametrize("size", [(1024, 1024), (257 * 64 - 3, 40), (2048, 1024), (1728, 1210)])
@pytest.mark.parametrize("n", [5, 3000])
def test_cell_sort_in_one_pass(n, size):
    """256, 257, 512 and 513 cells: 257 to 512 are sorted in one pass over nine bits."""
    _check(_scene(n, size[0] + n, scale=(0.01, 0.4)), _cam(*size))


@pytest.mark.parametrize("width", [52416, 52432])
def test_cell_digits_of_equal_width(width):
    """4095 cells (12 bits) are sorted as six and six bits, 4100 (13) as eight and five."""
    _check(_scene(2000, width, scale=(0.0005, 0.1), spread=(1.0, 0.004)), _cam(width, 320))


# 2040 cells: the notes of 80 B per cell do not fit the scratch of so few instances, and the cells'
# ranges do not fit the depth keys of 300 splats
@pytest.mark.parametrize("n", [300, 5000])
def test_little_scratch(n):
    from lumen_b200 import render as R
    scene, cam, opt = _scene(n, n, scale=(0.002, 0.004)), _cam(3840, 2160), RenderOptions()
    o = O.render(*scene, cam, opt, nthreads=NT)
    K = o.n_instances
    assert 0 < K < 60_000
    t = _dev(scene)
    g = R.gaussians_struct(*t)
    rgb = torch.empty((cam.height, cam.width, 3), dtype=torch.float32, device="cuda")
    img = L.LumenGpuImage()
    img.rgb = rgb.data_ptr()
    frame = R.Frame.allocate(n, cam.n_tiles, K, torch.device("cuda"))
    fs = frame.c_struct()
    lib, stream = L.load(), torch.cuda.current_stream().cuda_stream
    L.check(lib.lumen_gpu_render_forward(C.byref(g), C.byref(L.view_camera(cam)), C.byref(L.render_options(opt)),
                                         C.byref(fs), C.byref(img), stream), "render_forward")
    counts = L.LumenGpuCounts()
    L.check(lib.lumen_gpu_read_counts(C.byref(fs), C.byref(counts), stream), "read_counts")
    assert counts.error_flags == 0 and int(counts.n_instances) == K
    b = int(counts.sorted_buffer)
    assert np.array_equal(frame.keys[b][:K].cpu().numpy().view(np.uint32), (o.keys_sorted >> np.uint64(32)))
    assert np.array_equal(frame.vals[b][:K].cpu().numpy().view(np.uint32), o.vals_sorted)
    assert np.array_equal(rgb.cpu().numpy().view(np.uint32), o.rgb.view(np.uint32))


def _check_batch(views):
    """The batch's lists against those of its views rendered alone."""
    from lumen_b200 import render as R
    b = R.render_batch(views, RenderOptions())
    keys, vals = b.sorted_keys.cpu().numpy().view(np.uint64), b.sorted_vals.cpu().numpy().view(np.uint32)
    ids = b.frame.frame.visible_ids.cpu().numpy()
    pos = 0
    for v, (scene, cam) in enumerate(views):
        s = R.render(*scene.tensors, cam, RenderOptions())
        k = s.n_instances
        assert k > 0
        assert np.array_equal(keys[pos:pos + k], s.sorted_keys.cpu().numpy().view(np.uint64)
                              + (np.uint64(b.tile_begin[v]) << np.uint64(32)))
        assert np.array_equal(ids[vals[pos:pos + k]],
                              s.frame.visible_ids.cpu().numpy()[s.sorted_vals.cpu().numpy().view(np.uint32)])
        assert torch.equal(b.images[v].rgb, s.rgb)
        pos += k
    assert b.n_instances == pos


@pytest.mark.parametrize("views", [64, 65])
def test_more_cells_than_a_key_packs(views):
    """Views of 4095x1 tiles, 1024 cells each: 65536 cells pack with their masks, more do not."""
    from lumen_b200 import render as R
    scene = R.Scene(*_dev(_scene(150, 3, scale=(0.002, 0.05), spread=(1.8, 0.0005))))
    _check_batch([(scene, _cam(65520, 16, 60000.0))] * views)


@pytest.mark.parametrize("n", [227_000, 227_600])
def test_emission_rounds(n):
    """Two views: one side of 3 tickets of 1024 splats per SM (148) and the other."""
    from lumen_b200 import render as R
    sc = scenes.box_scene(n, seed=5)
    s, op = sc.activated()
    scene = R.Scene(*_dev([a.astype(np.float32) for a in (sc.means, s, sc.quats, op.reshape(-1), sc.sh)]))
    cams = scenes.orbit_cameras(2, 320, 180, fov=50.0, radius=10.0)
    _check_batch([(scene, c) for c in cams])


@pytest.mark.parametrize("size", [(37 * 16, 42 * 16), (5 * 16, 311 * 16), (56 * 16, 185 * 16 - 5), (13 * 16, 797 * 16)])
def test_tiles_in_line(size):
    """1554 to 10360 tiles (1.5 and 10 per resident CTA of 148 SMs) are shaded longest list first."""
    _check(_scene(3000, size[0], scale=(0.001, 0.3)), _cam(*size))


def test_tiles_in_line_backward():
    """The adjoint's sums over 1720 tiles, against 64-bit autograd with its bound at other sizes."""
    from test_gpu_backward_sums import _check as check_gradients
    check_gradients(30, (40 * 16, 43 * 16), (0.02, 0.5), 2e-4, depth=True, alpha=True, white=False)
