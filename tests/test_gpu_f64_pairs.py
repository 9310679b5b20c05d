"""The FP64 derivative pass (csrc/derivatives_f64.cu) leaves out the products
with the zeros of the point Jacobian and Hessian where the inverse covariance
is finite, and evaluates the other voxels as the reference writes it: score,
gradient and Hessian of one evaluation against the FP64 oracle at the edges of
warps and tiles, in both Hessian forms, on a dense map and on one of nearly
empty cells (singular covariances: infinities and NaNs have to come through).

Both sides evaluate every pair with the same FP64 operations and add the pairs
up in different orders: at most ~10^4 terms of 2^-53 each, and two digits for
cancellation between them, is 1e-10 of the largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(got, want, what):
    got, want = np.atleast_1d(got), np.atleast_1d(want)
    assert np.array_equal(np.isnan(got), np.isnan(want)), what
    fin = np.isfinite(want)
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)]), what
    if fin.any():
        assert np.max(np.abs(got[fin] - want[fin])) <= 1e-10 * max(1.0, np.max(np.abs(want[fin]))), what


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("cells", ["dense", "sparse"])
@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 513])
def test_evaluation_vs_oracle(pkg, oracle, binding_mod, compat, cells, n):
    rng = np.random.default_rng(n)
    cloud = np.zeros((4000 if cells == "dense" else 60, 4), np.float32)
    cloud[:, :3] = rng.uniform(-4.0, 4.0, (len(cloud), 3)) * [1.0, 1.0, 0.5]
    cloud[:, 3] = 1.0
    scan = np.ones((n, 4), np.float32)
    scan[:, :3] = rng.uniform(-4.5, 4.5, (n, 3)) * [1.0, 1.0, 0.5]
    p6 = np.array([0.3, -0.2, 0.05, 0.01, -0.02, 0.1])
    trans = scan.copy()
    trans[:, :3] += p6[:3].astype(np.float32)
    names = ("reference_params", "corrected_params")
    prm = getattr(pkg.ndt, names[compat == 0])(1.0, precision=1)
    oprm = getattr(binding_mod, names[compat == 0])()
    with pkg.ndt.Context(prm) as ctx:
        ctx.set_map(cloud)
        got = ctx.derivatives(scan, trans, p6)
    want = oracle.derivatives(oprm, cloud, scan, trans, p6)
    for g, w, what in zip(got, want, ("score", "gradient", "hessian")):
        _same(np.asarray(g).ravel(), np.asarray(w).ravel(), what)
