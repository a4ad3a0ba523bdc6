"""The tiles' lists where a cell's list is long, and where cells are cut by the
image border while the tiles are ordered by their lists' lengths."""
import pytest

from test_gpu_lists import _cam, _check, _scene

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1001, 433), (1111, 1111)])
def test_ordered_tiles_with_cells_at_the_border(size):
    """1764 and 4900 tiles; the last column and row of cells hold fewer than 16."""
    _check(_scene(2500, size[0]), _cam(*size))
