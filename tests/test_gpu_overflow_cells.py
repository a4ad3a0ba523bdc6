"""A batch with more cells than a packed key can name, whose instances exceed
its capacity: the lists hold the first `capacity` instances of the depth-ordered
emission, row-major per splat, and the frame reports the capacity alone."""
import ctypes as C

import numpy as np
import pytest

from lumen_b200 import _lib as L
from lumen_b200.types import RenderOptions
from test_gpu_lists import _cam, _dev, _scene

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

VIEWS, WIDTH, HEIGHT = 65, 65520, 48          # 65 x 1024 cells of 4x3 tiles


def _render(scene, capacity):
    from lumen_b200 import render as R
    cam = _cam(WIDTH, HEIGHT, 60000.0)
    views = [(scene, cam)] * VIEWS
    rgb8 = torch.empty((HEIGHT, WIDTH, 3), dtype=torch.uint8, device="cuda")     # one for all: the lists are looked at
    arr = (L.LumenGpuBatchView * VIEWS)()
    for v in arr:
        v.gaussians, v.camera, v.image.rgb8 = scene.struct, L.view_camera(cam), rgb8.data_ptr()
    slots, tiles = C.c_int64(0), C.c_int64(0)
    lib, stream = L.load(), torch.cuda.current_stream().cuda_stream
    L.check(lib.lumen_gpu_batch_sizes(arr, VIEWS, C.byref(slots), C.byref(tiles)), "batch_sizes")
    frame = R.BatchFrame.allocate(slots.value, tiles.value, capacity, VIEWS, torch.device("cuda"))
    fs, counts = frame.frame.c_struct(), L.LumenGpuCounts()
    L.check(lib.lumen_gpu_render_batch(arr, VIEWS, C.byref(L.render_options(RenderOptions())), C.byref(fs), stream),
            "render_batch")
    L.check(lib.lumen_gpu_read_counts(C.byref(fs), C.byref(counts), stream), "read_counts")
    return frame.frame, counts


@pytest.mark.parametrize("part", [0.31, 0.77])
def test_lists_of_the_written_prefix(part):
    from lumen_b200 import render as R
    scene = R.Scene(*_dev(_scene(40, 3, scale=(0.002, 0.05), spread=(1.8, 0.0005))))
    full, counts = _render(scene, 1 << 21)
    K, V = int(counts.n_instances), int(counts.n_visible)
    assert counts.error_flags == 0
    rects = full.rects[:V].cpu().numpy().view(np.uint64)
    depth = full.records[:V, 2].cpu().numpy()
    order = np.argsort((depth * np.float32(1000.0)).astype(np.int64), kind="stable")
    tiles, vals = [], []
    for v in order:
        x0, y0, x1, y1 = (int(rects[v] >> np.uint64(s)) & 0xFFF for s in (0, 12, 24, 36))
        first = (int(rects[v]) >> 48) * 4095 * 3
        t = first + np.arange(y0, y1 + 1)[:, None] * 4095 + np.arange(x0, x1 + 1)[None]
        tiles.append(t.reshape(-1))
        vals.append(np.full(t.size, v))
    tiles, vals = np.concatenate(tiles), np.concatenate(vals)
    assert tiles.size == K
    cap = int(K * part)
    while vals[cap - 1] != vals[cap]:         # inside a splat's tiles
        cap += 1
    frame, counts = _render(scene, cap)
    assert counts.error_flags == L.ERR_CAPACITY and int(counts.n_instances) == K
    b, perm = int(counts.sorted_buffer), np.argsort(tiles[:cap], kind="stable")
    assert np.array_equal(frame.keys[b][:cap].cpu().numpy(), tiles[:cap][perm])
    assert np.array_equal(frame.vals[b][:cap].cpu().numpy(), vals[:cap][perm])
