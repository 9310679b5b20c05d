"""The radix sort and segmentation behind the grid build, the scan pre-filter
and the clustering (csrc/grid_build.cu), through the filter: one leaf per
segment, means bit-exact with the oracle's in-order FP64 means, which a sort
that is not stable or loses a pair does not give.  Sizes at the edges of the
tiles (4096 and 8192 pairs, 16384 keys) and of the small-tile range (2^19),
with keys of 1 to 4 passes."""
import pathlib
import sys

import numpy as np
import pytest

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parents[1] / "oracle"))
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("span", [0.5, 30.0, 600.0, 2000.0])  # leaves: 1, 2^15, 2^20 (the batch: 2^21), 2^26
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 8193, 16384, 16385, 1 << 19, (1 << 19) + 1])
def test_sorted_segments(pkg, n, span):
    import voxel_filter_ref

    rng = np.random.default_rng(n)
    pts = rng.uniform(0.0, span, (n, 4)).astype(np.float32)
    if span > 100.0:
        pts[:, 2] *= np.float32(0.005)  # a flat scan
    off = np.array([0, n // 3, n], np.int32)
    with pkg.voxel_filter.VoxelFilter(0) as f:
        out, oo = f.filter(pts, off, 1.0)
    ref, ro = voxel_filter_ref.filter_batch(pts, off, 1.0)
    assert np.array_equal(oo, ro)
    assert np.array_equal(out.view(np.uint32), np.ascontiguousarray(ref, np.float32).view(np.uint32))
