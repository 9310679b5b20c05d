"""The probe-window table built by jobs of one and of four window layers
(csrc/grid_build.cu window_kernel: large tables take the latter) against the
dense-index probe: the same probes, occupied probes and pairs, and derivatives
that agree as two FP32 orders of the same pairs do (2e-3 of the largest
entry, as test_gpu_windows.py).  Table sizes at the edges of a job: rows of
32 windows, layers of 4."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (29, 40, 2), (30, 7, 3), (31, 300, 1), (62, 5, 6),
                                  (700, 400, 1), (701, 399, 2), (990, 500, 3), (606, 302, 7)])
def test_window_jobs(pkg, dims):
    rng = np.random.default_rng(sum(dims))
    ext = np.array(dims, np.float32) - 0.5
    m = 60000
    cloud = np.ones((m, 4), np.float32)
    # clusters, so that some cells hold the 6 points a voxel needs and many are empty
    centre = rng.uniform(0.0, 1.0, (m // 20, 3)) * ext
    cloud[:, :3] = np.clip(np.repeat(centre, 20, 0) + rng.normal(0.0, 0.2, (m, 3)), 0.0, ext)
    scan = np.ones((20000, 4), np.float32)
    scan[:, :3] = cloud[rng.integers(0, m, 20000), :3] + rng.normal(0.0, 1.0, (20000, 3))
    got = []
    for dense in (0, 1):
        with pkg.ndt.Context(pkg.ndt.corrected_params(dense_probe=dense)) as ctx:
            ctx.set_map(cloud)
            windows, entries = ctx.window_info()
            _, d, _ = ctx.grid_info()
            assert windows == (0 if dense else int(np.prod(d + 2)))
            score, g, H = ctx.derivatives(scan, scan, np.zeros(6))
            k = ctx.counters()
            got.append((score, g, H, [k[n] for n in ("points", "probes", "occupied_probes", "pairs")]))
    assert got[0][3] == got[1][3]
    assert got[0][3][3] > 0
    for a, b in zip(got[0][:3], got[1][:3]):
        assert np.max(np.abs(a - b)) <= 2e-3 * max(1.0, float(np.max(np.abs(b))))
