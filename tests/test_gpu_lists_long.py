"""The tiles' lists where a cell's list is long, and where cells are cut by the
image border while the tiles are ordered by their lists' lengths."""
import pytest

from test_gpu_lists import _cam, _check, _dev, _scene

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1001, 433), (1111, 1111)])
def test_ordered_tiles_with_cells_at_the_border(size):
    """1764 and 4900 tiles; the last column and row of cells hold fewer than 16."""
    _check(_scene(2500, size[0]), _cam(*size))


@pytest.mark.parametrize("n", [8192, 16385, 32768, 32769, 65537, 100_000])
def test_one_long_cell(n):
    """Every splat in front of the one cell: counted whole, and in 2 to 4 parts."""
    _check(_scene(n, n, spread=(0.3, 0.3)), _cam(64, 64))


@pytest.mark.parametrize("size", [(80, 64), (130, 70)])
def test_long_cells_of_unequal_length(size):
    """2 and 6 cells, whose parts begin anywhere in the windows."""
    _check(_scene(90_000, size[0], scale=(0.002, 0.2), spread=(0.4, 0.2)), _cam(*size))


def test_long_cells_of_a_batch():
    from lumen_b200 import render as R
    from lumen_b200.types import RenderOptions
    scene = R.Scene(*_dev(_scene(50_000, 8, spread=(0.3, 0.3))))
    cams = [_cam(64, 64), _cam(100, 40), _cam(64, 64, 90.0), _cam(7, 9)]
    got = R.render_batch([(scene, c) for c in cams], RenderOptions())
    for c, image in zip(cams, got.images):
        alone = R.render(*scene.tensors, c, RenderOptions())
        for a, b in ((image.rgb, alone.rgb), (image.n_contrib, alone.n_contrib), (image.last_idx, alone.last_idx)):
            assert torch.equal(a, b)
