"""Root and box queries at the limits of their listing before the count is known: its
capacity, what comes back with the count, and the context's scratch and budget."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _dots(cuda, count, cols=512):
    """`count` one-pixel components, and their roots and boxes (1-based)."""
    per = cols // 2
    rows = 2 * ((count + per - 1) // per) + 1
    k = np.arange(count)
    y, x = 2 * (k // per), 2 * (k % per)
    img = torch.zeros((rows, cols), dtype=torch.bool, device=cuda)
    img[torch.from_numpy(y).to(cuda), torch.from_numpy(x).to(cuda)] = True
    roots = y * cols + x + 1
    return img, roots, np.stack([roots, y + 1, x + 1, y + 1, x + 1], 1)


def _query(ctx, name, labels, capacity):
    per = 5 if name == "ph_ccl_boxes" else 1
    out = np.full((capacity, per) if per > 1 else capacity, -1, dtype=np.int64)
    count = ctypes.c_int64(-1)
    shape = (labels.numel(),) if per == 1 else (1,) + tuple(labels.shape)
    s = torch.cuda.current_stream().cuda_stream
    try:
        ctx.call(name, out.ctypes.data if capacity else None, capacity, ctypes.byref(count), labels.data_ptr(), *shape, s)
    except MemoryError:
        return count.value, None
    return count.value, out


# 2048 come back with the count, 16384 are listed before it is known
@pytest.mark.parametrize("count", [0, 1, 2047, 2048, 2049, 16383, 16384, 16385, 40000, 70000])
def test_every_capacity(ph, cuda, count):
    from ph_gb300 import _lib
    img, roots, boxes = _dots(cuda, count)
    labels = ph.cu_connected_component_labeling(img, reference_grid=False)
    ctx = _lib.Context(0)
    for capacity in (0, 1, 2048, 3000, 16384, 16385, max(count, 1), 100000):   # a small arena first, then a grown one
        for name, want in (("ph_ccl_roots", roots), ("ph_ccl_boxes", boxes)):
            total, got = _query(ctx, name, labels, capacity)
            assert total == count
            m = min(capacity, count)
            assert np.array_equal(got[:m], want[:m]) and (got[m:] == -1).all()
    found, rects = ph.cu_find_valid_labels(labels), ph.cu_bounding_rectangles(labels)
    assert np.array_equal(found, roots) and np.array_equal(rects, boxes)
    assert found.base is None or found.base.size == count       # no larger buffer is kept alive
    assert rects.base is None or rects.base.size == 5 * count


def test_budget_of_the_exact_size(ph, cuda):
    """Room for the components that there are serves the query, without room for 16384."""
    from ph_gb300 import _lib
    img, roots, boxes = _dots(cuda, 40, cols=64)
    labels = ph.cu_connected_component_labeling(img, reference_grid=False)
    ctx = _lib.Context(0, hbm_budget_bytes=4 * labels.numel() + 4096)   # ranks, counts, 40 roots and boxes
    for _ in range(2):
        for name, want in (("ph_ccl_roots", roots), ("ph_ccl_boxes", boxes)):
            total, got = _query(ctx, name, labels, 65536)
            assert total == 40 and got is not None and np.array_equal(got[:40], want)


def test_count_where_the_boxes_do_not_fit(ph, cuda):
    from ph_gb300 import _lib
    img, roots, _ = _dots(cuda, 300)
    labels = ph.cu_connected_component_labeling(img, reference_grid=False)
    ctx = _lib.Context(0, hbm_budget_bytes=4096)
    assert _query(ctx, "ph_ccl_boxes", labels, 1000) == (300, None)
    assert _query(ctx, "ph_ccl_roots", labels, 100)[0] == 300


def test_an_empty_volume_takes_no_ranks(ph, cuda):
    """Without components the arena (and the graphs that hold it) stays as it is."""
    from ph_gb300 import _lib
    labels = ph.cu_connected_component_labeling_batch(torch.zeros((4, 300, 300), dtype=torch.bool, device=cuda))
    ctx = _lib.Context(0)
    out, count = np.zeros((9, 5), np.int64), ctypes.c_int64(-1)
    ctx.call("ph_ccl_boxes", out.ctypes.data, 9, ctypes.byref(count), labels.data_ptr(), 4, 300, 300,
             torch.cuda.current_stream().cuda_stream)
    assert count.value == 0 and ctx.scratch_bytes < 4096


def test_boxes_of_crossing_components(ph, cuda):
    """Components whose boxes grow from many threads at once: rings inside rings, and bars."""
    from oracle import ccl as occl
    from oracle import ref_semantics as ref
    n = 301
    i, j = np.indices((n, n)) - n // 2
    img = (np.maximum(abs(i), abs(j)) % 3 == 0) | (abs(i - j) < 2)
    lab = occl.connected_component_labeling(img.astype(np.float32))
    valid = ref.find_valid_labels(lab)
    want = [(int(v),) + tuple(b) for v, b in zip(valid, ref.bounding_rectangles(lab, valid))]
    labels = ph.cu_connected_component_labeling(torch.from_numpy(img).to(cuda), reference_grid=False)
    assert [tuple(b) for b in ph.cu_bounding_rectangles(labels).tolist()] == want
