"""The warp-per-tile labeling against the C oracle where tiles can go wrong: images
that end inside a tile, slices that start inside one (shorter than a tile too),
runs across words and tiles, unaligned arrays, more components than one query holds."""
import numpy as np
import pytest
import torch

from oracle import ccl as occl
from oracle import ref_semantics as ref
from phtest import to_np

pytestmark = pytest.mark.gpu


def _pattern(kind, shape, rng):
    if kind == "comb":          # teeth joined by a bar at the bottom: long chains of runs
        v = np.zeros(shape, bool)
        v[..., ::2] = True
        v[..., -1, :] = True
        return v
    if kind == "full":
        return np.ones(shape, bool)
    if kind == "diagonal":      # 8-connectivity through tile corners
        i, j = np.indices(shape)[-2:]
        return (i + j) % 7 == 0
    return rng.random(shape) < float(kind)


@pytest.mark.parametrize("kind", ["comb", "full", "diagonal", "0.02", "0.4", "0.6"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 33), (3, 33, 1), (5, 7, 31), (4, 33, 65), (3, 40, 96), (2, 96, 130)])
@pytest.mark.parametrize("dtype", [torch.bool, torch.float32])
def test_batch_labels_and_boxes(ph, cuda, kind, shape, dtype):
    rng = np.random.default_rng(shape[1] * 1000 + shape[2])
    vol = _pattern(kind, shape, rng)
    labels = ph.cu_connected_component_labeling_batch(torch.from_numpy(vol).to(cuda).to(dtype))
    got = to_np(labels.view(torch.int32)).astype(np.uint32)
    per = shape[1] * shape[2]
    want_boxes = []
    for k in range(shape[0]):
        lab = occl.connected_component_labeling(vol[k].astype(np.float32))
        assert np.array_equal(got[k], lab)
        valid = ref.find_valid_labels(lab)
        want_boxes += [(k * per + int(v),) + tuple(b) for v, b in zip(valid, ref.bounding_rectangles(lab, valid))]
    assert [tuple(b) for b in ph.cu_bounding_rectangles(labels).tolist()] == want_boxes


@pytest.mark.parametrize("offset", [1, 3, 16])
def test_unaligned_and_many_components(ph, cuda, offset):
    rows, cols = 300, 257
    buf = torch.zeros(rows * cols + 16, dtype=torch.bool, device=cuda)
    img = buf[offset:offset + rows * cols].view(rows, cols)
    img[::2, ::2] = True                                        # 150 * 129 isolated pixels
    labels = ph.cu_connected_component_labeling(img, reference_grid=False)
    want = occl.connected_component_labeling(to_np(img).astype(np.float32))
    assert np.array_equal(to_np(labels.view(torch.int32)).astype(np.uint32), want)
    assert ph.count_labels(labels) == 150 * 129
    assert np.array_equal(ph.cu_find_valid_labels(labels), ref.find_valid_labels(want))
    assert len(ph.cu_bounding_rectangles(labels)) == 150 * 129


def test_several_values_in_a_tile(ph, cuda):
    rng = np.random.default_rng(3)
    img = rng.integers(0, 4, (70, 95)).astype(np.float32)
    img[20:50, 10:80] = 2.5
    labels = ph.cu_connected_component_labeling(torch.from_numpy(img).to(cuda), reference_grid=False)
    assert np.array_equal(to_np(labels.view(torch.int32)).astype(np.uint32), occl.connected_component_labeling(img))


# more pixels than 16 per thread of the last pass need (2^20), more tiles than get a warp per side (3072)
@pytest.mark.parametrize("kind", ["comb", "diagonal", "0.02", "0.4", "0.6"])
@pytest.mark.parametrize("shape", [(1, 1100, 1003), (1, 2000, 2003), (5, 700, 999)])
@pytest.mark.parametrize("dtype,offset", [(torch.bool, 0), (torch.bool, 4), (torch.float32, 0), (torch.float32, 1)])
def test_large_images(ph, cuda, kind, shape, dtype, offset):
    vol = _pattern(kind, shape, np.random.default_rng(shape[1]))
    buf = torch.zeros(vol.size + 16, dtype=dtype, device=cuda)
    img = buf[offset:offset + vol.size].view(shape)
    img.copy_(torch.from_numpy(vol))
    got = to_np(ph.cu_connected_component_labeling_batch(img).view(torch.int32)).astype(np.uint32)
    for k in range(shape[0]):
        assert np.array_equal(got[k], occl.connected_component_labeling(vol[k].astype(np.float32)))


@pytest.mark.parametrize("cols,rows", [(45, 70), (96, 33), (130, 31)])
def test_runs_of_several_values(ph, cuda, cols, rows):
    """Runs that end at another value, roots that meet in one run from both sides."""
    rng = np.random.default_rng(cols)
    img = rng.integers(1, 3, (rows, cols)).astype(np.float32)
    img[::3, ::2] = 0
    img[5:9] = np.where(np.arange(cols) % 11 < 9, 1.0, 2.0)
    labels = ph.cu_connected_component_labeling(torch.from_numpy(img).to(cuda), reference_grid=False)
    assert np.array_equal(to_np(labels.view(torch.int32)).astype(np.uint32), occl.connected_component_labeling(img))
