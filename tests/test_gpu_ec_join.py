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
