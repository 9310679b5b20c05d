"""The FP64 derivative pass for scan points that are not finite beside
transformed points that are (ndt_derivatives takes both from the caller): the
products with the zeros of the point Jacobian and Hessian are NaN there and
have to come through, as the reference's expressions give them.  One point and
one voxel at a time, since any other pair's NaN hides the difference, and poses
at which some gradient entries are infinite, not NaN.

Finite entries as test_gpu_f64_pairs.py: the same FP64 terms, 1e-10 of the
largest entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38])
def test_scan_value_vs_oracle(pkg, oracle, binding_mod, compat, value):
    names = ("reference_params", "corrected_params")
    prm = getattr(pkg.ndt, names[compat == 0])(1.0, precision=1)
    oprm = getattr(binding_mod, names[compat == 0])()
    with pkg.ndt.Context(prm) as ctx:
        for k in range(150):
            rng = np.random.default_rng(k)
            # one voxel of 40 points; one far away (compat scales the covariance by the number of cells less one)
            cloud = np.ones((41, 4), np.float32)
            mix = np.eye(3) + 0.8 * rng.uniform(-1, 1, (3, 3))
            cloud[:, :3] = 0.5 + np.clip(rng.normal(0, 0.1, (41, 3)) @ mix, -0.45, 0.45)
            cloud[40, :3] = [0.5, 0.5, 9.5]
            trans = np.ones((1, 4), np.float32)
            trans[0, :3] = 0.5 + rng.uniform(-0.1, 0.1, 3)
            scan = trans.copy()
            scan[0, k % 3] = value
            p6 = np.array([0.0, 0.0, 0.0, *rng.uniform(-1.5, 1.5, 3)])
            ctx.set_map(cloud)
            got = ctx.derivatives(scan, trans, p6)
            want = oracle.derivatives(oprm, cloud, scan, trans, p6)
            for g, w in zip(got, want):
                g, w = np.atleast_1d(g).ravel(), np.atleast_1d(w).ravel()
                assert np.array_equal(np.isnan(g), np.isnan(w)), k
                fin = np.isfinite(w)
                assert np.array_equal(g[~fin & ~np.isnan(w)], w[~fin & ~np.isnan(w)]), k
                if fin.any():
                    assert np.max(np.abs(g[fin] - w[fin])) <= 1e-10 * max(1.0, np.max(np.abs(w[fin]))), k
