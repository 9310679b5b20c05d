"""The join passes of the GPU clustering at the edges of their rows and warps:
stretches of a row of exactly a warp's width, clouds of one cell, one cell
thick on an axis, and long chains in either index order on each axis (every
point hangs under the one before it in the sorted order, so a chain is one
tree of that depth), against brute force; labels are whole numbers and equal."""
import numpy as np
import pytest

import ec_ref

pytestmark = pytest.mark.gpu


def _cloud(name, n, rng):
    if name == "cell":  # all in one cell, far from the origin
        return rng.uniform(0, 0.2, (n, 3)) + [1e4, -1e4, 3.0]
    if name.startswith("chain"):  # exact multiples of the tolerance: accepted with equality
        p = np.zeros((n, 3))
        p[:, "xyz".index(name[5])] = np.arange(n)[:: -1 if name.endswith("-") else 1] * 0.5
        return p
    if name == "plane":  # one cell thick, ragged rows
        return np.column_stack([rng.uniform(-9, 9, n), rng.uniform(-9, 9, n), np.full(n, -1.0)])
    return rng.uniform(-3, 3, (n, 3)) * [1.0, 1.0, 0.4]  # "box": many trees of a component meet


@pytest.mark.parametrize("name", ["cell", "chainx", "chainx-", "chainy-", "chainz", "chainz-", "plane", "box"])
@pytest.mark.parametrize("n", [1, 2, 32, 33, 65, 256, 700])
def test_labels_at_the_edges(pkg, name, n):
    rng = np.random.default_rng(n)
    xyz = _cloud(name, n, rng).astype(np.float32)
    with pkg.ec.EuclideanClusters(0) as ec:
        for order in (np.arange(n), rng.permutation(n)):
            assert np.array_equal(ec.labels(xyz[order], 0.5), ec_ref.brute_labels(xyz[order], 0.5))


def _ring(xyz):
    d = np.sqrt(xyz[:, 0] * xyz[:, 0] + xyz[:, 1] * xyz[:, 1])
    return np.digitize(d, np.array([15, 30, 45, 60], np.float32))


@pytest.mark.parametrize("sizes", [(0, 1, 19, 20, 21), (255, 256, 257), (0,) * 9 + (600, 40), (16384, 1, 16385)])
def test_segment_points_equal_extract_of_each_ring(pkg, sizes):
    """Clusters of exactly the least size, empty clouds, more clouds than one
    pass takes, points on the rings' edges and several copies to the device:
    the clustered points of a batch are those of extract() on each ring of each
    cloud, in its order (equal sizes included), with the plain centroid."""
    rng = np.random.default_rng(len(sizes))
    tol = (0.5, 1.1, 1.6, 2.3, float(np.float32(2.6)))
    clouds = []
    for n in sizes:
        at = rng.uniform(-70, 70, (max(n // 20, 1), 2))
        at[: len(at) // 4] = np.array([[15.0, 0.0], [0.0, 30.0], [45.0, 0.0], [-60.0, 0.0]])[np.arange(len(at) // 4) % 4]
        p = np.column_stack([at[np.arange(n) % len(at)] + rng.uniform(-0.2, 0.2, (n, 2)) * (np.arange(n) % 3 > 0)[:, None],
                             rng.uniform(-1, 0, n)])
        clouds.append(p.astype(np.float32))
    with pkg.ec.EuclideanClusters(0) as ec:
        for cloud, (pts, boxes, cen) in zip(clouds, ec.segment_batch(clouds)):
            want, sums = [], []
            for k in range(5):
                ring = cloud[_ring(cloud) == k]
                for idx in ec.extract(ring, tol[k]) if len(ring) else []:
                    want.append(ring[idx])
                    sums.append(np.cumsum(ring[idx].astype(np.float64), 0)[-1] / len(idx))
            want = np.concatenate(want) if want else np.zeros((0, 3), np.float32)
            assert np.array_equal(pts, want)
            kept = [any(np.array_equal(c, s) for s in sums) for c in cen]
            assert all(kept) and len(boxes) == len(cen)
