"""Frame.allocate: a small frame is one allocation cut into tensors on demand, a
large one a tensor per buffer. Either way the tensors have the buffers' types
and sizes, do not overlap, and are what the C structure points to."""
import pytest

torch = pytest.importorskip("torch")

from lumen_b200 import render as R


def _tensors(f):
    return [f.records, f.visible_ids, f.radii, f.rects, *f.depth_keys, *f.depth_order, *f.keys, *f.vals, f.ranges,
            f.scratch]


def _pointers(s):
    return [s.records, s.visible_ids, s.radii, s.rects, *s.depth_keys, *s.depth_order, *s.keys, *s.vals, s.ranges,
            s.scratch]


@pytest.mark.parametrize("n,tiles,capacity", [(0, 1, 1), (1, 7, 65), (1000, 33, 4097), (100_000, 8160, 800_000),
                                              (400_000, 100, 3_200_000)])
def test_layout(n, tiles, capacity):
    f = R.Frame.allocate(n, tiles, capacity, torch.device("cpu"))
    before = _pointers(f.c_struct())
    n1, i32 = max(n, 1), torch.int32
    assert ("_one" in f.__dict__) == (n < 400_000)
    t = _tensors(f)
    want = [((n1, 12), torch.float32), ((n1,), i32), ((n1,), i32), ((n1,), torch.int64)] + [((n1,), i32)] * 4 \
        + [((capacity,), i32)] * 4 + [((tiles, 2), i32)]
    assert [(tuple(x.shape), x.dtype) for x in t[:-1]] == want and t[-1].dtype == torch.uint8
    s = f.c_struct()
    assert _pointers(s) == before == [x.data_ptr() for x in t]
    assert (s.instance_capacity, s.scratch_bytes) == (capacity, t[-1].numel())
    spans = sorted((x.data_ptr(), x.data_ptr() + x.numel() * x.element_size()) for x in t)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    assert f.fits(n, tiles) and not f.fits(n1 + 1, tiles) and not f.fits(n, tiles + 1)


def test_replaced_tensor_is_used():
    f = R.Frame.allocate(10, 4, 100, torch.device("cpu"))
    f.rects = torch.zeros(10, dtype=torch.int64)
    assert f.c_struct().rects == f.rects.data_ptr()
    with pytest.raises(AttributeError):
        f.no_such_buffer
