"""Calls of the pre-filter that its block-per-scan kernel (csrc/voxel_filter.cu
scan_kernel) must not take, because it writes results while other blocks read:
outputs over the inputs, and offsets that are not a partition of the points
(points outside belong to the first or the last scan, as the general path finds
each point's scan).  Bit for bit against the oracle, at sizes that do go to that
kernel otherwise."""
import numpy as np
import pytest

import voxel_filter_ref as V

pytestmark = pytest.mark.gpu


def _batch(B=300, n=3000):
    rng = np.random.default_rng(11)
    pts = rng.uniform(-20.0, 20.0, (B * n, 4)).astype(np.float32)
    pts[:, 2] *= np.float32(0.02)
    return pts, (np.arange(B + 1) * n).astype(np.int32)


def _run(pkg, torch, pts, off, in_place=(False, False)):
    d_pts, d_off = torch.from_numpy(pts).cuda(), torch.from_numpy(off).cuda()
    d_out = d_pts if in_place[0] else torch.zeros_like(d_pts)
    d_oo = d_off if in_place[1] else torch.zeros_like(d_off)
    torch.cuda.synchronize()
    with pkg.voxel_filter.VoxelFilter(0) as f:
        k = f.filter_device(len(off) - 1, d_pts.data_ptr(), d_off.data_ptr(), len(pts), 1.0, d_out.data_ptr(),
                            d_oo.data_ptr())
    return d_out[:k].cpu().numpy(), d_oo.cpu().numpy()


def _same(got, pts, off):
    ref, ro = V.filter_batch(pts, off, 1.0)
    assert np.array_equal(got[1], ro)
    assert np.array_equal(got[0].view(np.uint32), np.ascontiguousarray(ref, np.float32).view(np.uint32))


@pytest.mark.parametrize("in_place", [(False, False), (True, False), (False, True), (True, True)])
def test_outputs_over_inputs(pkg, in_place):
    torch = pytest.importorskip("torch")
    pts, off = _batch()
    for _ in range(3):
        _same(_run(pkg, torch, pts, off, in_place), pts, off)


@pytest.mark.parametrize("first,last", [(500, 0), (0, -700), (1, -1), (0, 900)])
def test_points_outside_the_offsets(pkg, first, last):
    torch = pytest.importorskip("torch")
    pts, off = _batch()
    cut = off.copy()
    cut[0] += first
    cut[-1] += last
    _same(_run(pkg, torch, pts, cut), pts, off)
