"""The render server's images where a batch leaves in parts: runs of views of at
least a wave of tiles, small views among large ones, and batches too small to
split. Every image equals its view rendered alone."""
import pytest

from lumen_b200 import scenes
from lumen_b200.types import ViewCamera
from test_gpu_serve import alone_u8, device_scene

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SMALL, MIDDLE, WIDE, TALL = (64, 64), (320, 180), (1280, 720), (70, 2900)


@pytest.mark.parametrize("sizes", [[SMALL] * 40, [MIDDLE] * 9, [WIDE, SMALL, SMALL], [SMALL, WIDE], [SMALL, TALL, MIDDLE] * 6,
                                   [MIDDLE] * 4 + [WIDE] * 3 + [SMALL]])
def test_images_of_a_split_batch(sizes):
    from lumen_b200 import serve
    ds = device_scene(scenes.box_scene(4000, seed=17))
    cams = [ViewCamera.from_fov(w, h, 50.0, position=(0.05 * i, 0.0, -0.1 * i)) for i, (w, h) in enumerate(sizes)]
    outs = [torch.empty((h, w, 3), dtype=torch.uint8, pin_memory=True) for w, h in sizes]
    first, first_out = ViewCamera.from_fov(4200, 4200, 50.0), torch.empty((4200, 4200, 3), dtype=torch.uint8, pin_memory=True)
    with serve.Server(work_budget_bytes=4 << 30, max_views_per_batch=64, max_batches_in_flight=1, autotune=False) as srv:
        sid = srv.add_scene(ds)
        for _ in range(2):
            # the others queue up behind a view of more tiles than a batch holds
            alone = srv.submit(sid, first, first_out)
            res = [h.result(timeout_ms=60_000) for h in [srv.submit(sid, c, o) for c, o in zip(cams, outs)]]
            assert alone.result(timeout_ms=60_000).status == 0 and max(r.batch_views for r in res) > 1
            for r, c in zip(res, cams):
                assert r.status == 0 and torch.equal(r.image, alone_u8(ds, c))


def test_a_server_for_many_views_per_batch():
    """One event per part a batch can have, not per view."""
    from lumen_b200 import serve
    ds = device_scene(scenes.box_scene(500, seed=18))
    cam = ViewCamera.from_fov(65, 33, 50.0)
    with serve.Server(work_budget_bytes=1 << 30, max_views_per_batch=65535, autotune=False) as srv:
        sid = srv.add_scene(ds)
        for h in [srv.submit(sid, cam) for _ in range(300)]:
            r = h.result(timeout_ms=60_000)
            assert r.status == 0 and torch.equal(r.image, alone_u8(ds, cam))
