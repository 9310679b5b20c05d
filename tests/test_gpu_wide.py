"""The two kernels of the FP32 derivative pass (csrc/derivatives_f32.cu for
many chunks, csrc/derivatives_wide.cu for few) give the same bits: a scan
aligned alone (its few chunks go to the wide kernel) against the same scan in
a batch of copies that has more chunks than the wide kernel takes.  No
tolerance: the lane sums are the same FP32 chains in both.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COPIES = 1500  # more chunks than the wide kernel's limit (5 x 3 x SMs / 4 columns) for any SM count up to 400


def _bits(r):
    out, conv, fit, status = r
    return out.view(np.uint32), conv, fit.view(np.uint64), status


def _same(pkg, prm, cloud, scans, guesses, chunk_tiles, variant, side_pairs=0):
    for scan, guess in zip(scans, guesses):
        with pkg.ndt.Context(prm) as ctx:
            ctx.set_side_queue_capacity(side_pairs)
            ctx.set_chunk_tiles(chunk_tiles)
            ctx.set_kernel_variant(variant)
            ctx.set_map(cloud)
            alone = _bits(ctx.align_batch([scan], [guess]))
            one = ctx.counters()
            many = _bits(ctx.align_batch([scan] * COPIES, [guess] * COPIES))
            all_ = ctx.counters()
        for a, m in zip(alone, many):
            assert (m == a[0]).all()
        for k in ("evaluations", "points", "probes", "occupied_probes", "pairs", "tiles"):
            assert all_[k] == COPIES * one[k], k


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("chunk_tiles,variant", [(8, 6), (1, 6), (9, 6), (64, 6), (8, 4), (20, 4)])
def test_wide_equals_many(pkg, compat, chunk_tiles, variant):
    # 1 m voxels around the walls, sparse rounds far from them; ragged tile and chunk ends
    cfg = pkg.synth.small_config("wide", 12000, 34.0, 12, 700, seed=77, dt=0.4, dyaw_deg=3.0, radius=16.0)
    scene = pkg.synth.make_scene(cfg)
    sizes = (1, 33, 128, 129, 1025, 2600)
    al = [pkg.synth.make_alignment(cfg, scene, i, n_points=n) for i, n in enumerate(sizes)]
    scans, guesses = [a.scan for a in al], [a.guess.copy() for a in al]
    scans.append(scans[-1].copy())
    g = guesses[-1].copy()
    g[3] += 24.0  # partly off the map: tiles with few pairs go through the ring
    guesses.append(g)
    prm = (pkg.ndt.reference_params if compat else pkg.ndt.corrected_params)(1.0)
    prm.max_iterations = 3 if not compat else 0
    _same(pkg, prm, scene.map, scans, guesses, chunk_tiles, variant)


@pytest.mark.parametrize("chunk_tiles", [1, 8])
def test_wide_equals_many_far_coordinates(pkg, chunk_tiles):
    # at 2^25 m a probe step rounds away: 64 probes of one cell, which do not fit one collect call
    rng = np.random.default_rng(3)
    cloud = np.ones((600, 4), np.float32)
    cloud[:, :3] = np.float32(2.0 ** 25) + 4.0 * rng.integers(0, 5, (600, 3))
    scan = np.ascontiguousarray(cloud[rng.integers(0, 600, 130)])
    prm = pkg.ndt.reference_params(1.0)
    guess = np.eye(4, dtype=np.float32).reshape(16)
    with pkg.ndt.Context(prm) as ctx:
        ctx.set_map(cloud)
        ctx.align_batch([scan], [guess])
        assert ctx.counters()["probes"] > 27 * len(scan)  # the generic path, more than one collect call
    # (voxels this far out go through the FP64 side queue: room for every copy's pairs)
    _same(pkg, prm, cloud, [scan], [guess], chunk_tiles, 6, side_pairs=1 << 24)


@pytest.mark.parametrize("compat", [0, 1])
@pytest.mark.parametrize("n,copies", [(1, 1), (130, 1), (2600, 1), (2600, COPIES)])
def test_score_pass_equals_full_evaluation(pkg, compat, n, copies):
    """A score pass sums the score alone; it is the score of the full
    evaluation (score, gradient, Hessian) bit for bit, on both kernels."""
    torch = pytest.importorskip("torch")
    cfg = pkg.synth.small_config("score", 12000, 34.0, 12, 700, seed=78, dt=0.4, dyaw_deg=3.0, radius=16.0)
    scene = pkg.synth.make_scene(cfg)
    a = pkg.synth.make_alignment(cfg, scene, 0, n_points=n)
    T = a.guess.reshape(4, 4)
    x, y, z = a.scan[:, 0], a.scan[:, 1], a.scan[:, 2]
    trans = np.ones_like(a.scan)
    for r in range(3):  # float, left to right, as the derivative pass transforms
        trans[:, r] = ((T[r, 0] * x + T[r, 1] * y) + T[r, 2] * z) + T[r, 3]
    prm = (pkg.ndt.reference_params if compat else pkg.ndt.corrected_params)(1.0)
    with pkg.ndt.Context(prm) as ctx:
        ctx.set_map(scene.map)
        full, _, _ = ctx.derivatives(a.scan, trans, np.zeros(6))
        pts = torch.from_numpy(np.tile(a.scan, (copies, 1))).cuda()
        off = torch.arange(copies + 1, dtype=torch.int32).cuda() * n
        poses = torch.from_numpy(np.tile(a.guess, (copies, 1))).cuda()
        out = torch.zeros(copies, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        ctx.score_batch_device(copies, pts.data_ptr(), off.data_ptr(), copies * n, poses.data_ptr(), out.data_ptr())
        ctx.synchronize()
    assert (out.cpu().numpy().view(np.uint64) == np.float64(full).view(np.uint64)).all()
