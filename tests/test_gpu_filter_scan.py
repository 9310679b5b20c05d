"""The pre-filter's block-per-scan kernel (csrc/voxel_filter.cu scan_kernel)
bit for bit against the oracle's in-order FP64 means: at the limits that send a
batch to the general path, with empty and single-leaf scans between others, and
with leaves whose FP64 sums are not exact in any order (tiny beside large
magnitudes, infinities, NaN) at each way a leaf is summed (4 lanes, up to 64
points; a warp, up to 2048; the whole scan)."""
import numpy as np
import pytest

import voxel_filter_ref as V

pytestmark = pytest.mark.gpu


def _check(pkg, scans, leaf):
    pts = np.ascontiguousarray(np.concatenate(scans).astype(np.float32))
    off = np.zeros(len(scans) + 1, np.int32)
    off[1:] = np.cumsum([len(s) for s in scans])
    with pkg.voxel_filter.VoxelFilter(0) as f:
        for _ in range(2):  # (a second call on the kept scratch)
            out, oo = f.filter(pts, off, leaf)
    ref, ro = V.filter_batch(pts, off, leaf)
    ref = np.ascontiguousarray(ref, np.float32)
    assert np.array_equal(oo, ro)
    same = out.view(np.uint32) == ref.view(np.uint32)
    assert (same | (np.isnan(out) & np.isnan(ref))).all()


def _cloud(rng, n, span, flat=0.02):
    p = rng.uniform(-span, span, (n, 4))
    p[:, 2] = rng.normal(0.0, flat, n)
    return p


@pytest.mark.parametrize("n", [1, 5, 1023, 65535, 65536, 65537])
@pytest.mark.parametrize("span", [0.4, 12.0, 110.0])  # leaves of 1 m: 1 to 4, ~1250, ~96000 (the general path)
def test_sizes(pkg, n, span):
    rng = np.random.default_rng(n)
    empty = np.zeros((0, 4))
    dropped = np.full((7, 4), np.nan)
    one = np.abs(_cloud(rng, n, 0.4)) + 3.0  # one leaf: at 65536 points beyond the 16-bit counts
    one[:, 2] = 0.5
    # (enough points in all that the batch takes this kernel where its scans fit)
    rest = [_cloud(rng, 9000, span) for _ in range(0 if n < 20000 else 90)]
    _check(pkg, [_cloud(rng, n, span), empty, dropped, one[:n], _cloud(rng, 777, span)] + rest, 1.0)


@pytest.mark.parametrize("m", [2, 17, 64, 65, 300, 2048, 2049, 9000])
@pytest.mark.parametrize("kind", ["tiny", "zero", "inf", "nan", "subnormal"])
def test_leaves_with_inexact_sums(pkg, m, kind):
    rng = np.random.default_rng(m)
    p = _cloud(rng, 12000, 9.0)
    at = rng.choice(len(p), m, replace=False)
    p[at, :3] = rng.uniform(0.0, 1.0, (m, 3)) * [1, 1, 0.9]  # one leaf of at least m points, anywhere in the scan
    if kind == "tiny":
        p[at[::3], 0] *= 10.0 ** rng.uniform(-30, 0, len(at[::3]))
        p[at[1::3], 3] = 3e30
    elif kind == "zero":
        p[at, 3] = 0.0
        p[at[::2], 0] = -0.0
    elif kind == "inf":
        p[at[0], 3] = np.inf
    elif kind == "nan":
        p[at[-1], 3] = np.nan
    else:
        p[at, 3] = rng.uniform(0.0, 1e-38, m)
    _check(pkg, [p, _cloud(rng, 100, 9.0), p[::-1]], 1.0)


@pytest.mark.parametrize("shift", [3.0e9, -5.0e9])
def test_far_scans(pkg, shift):
    rng = np.random.default_rng(1)
    p = _cloud(rng, 5000, 4000.0)
    p[:, 0] += shift  # leaf indices beyond 32 bits, extents within
    _check(pkg, [p, _cloud(rng, 300, 4000.0)], 400.0 if shift > 0 else 0.99e3)
    q = _cloud(rng, 3000, 2000.0)
    q[:, 1] += shift
    _check(pkg, [q], 512.0)
    _check(pkg, [q / 1000.0], 1.0e-3 * 512)
