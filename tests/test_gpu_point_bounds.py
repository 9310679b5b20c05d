"""The device entry points take a bound of a batch's points, which the scans
need not fill (a buffer's capacity; the learned pipeline's subsamples of
ragged scans).  Whatever the bound, every pass is evaluated, by the kernel for
few chunks or by the one for many (csrc/derivatives.h launches_wide), which
give the same bits: results with a large bound equal the exact one's, and a
scan's results in a ragged batch equal those of the scan alone.  No tolerance.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 4_000_000  # points: more chunks than the kernel for few takes on any SM count up to 1000


def _scene(pkg, n):
    cfg = pkg.synth.small_config("bound", 12000, 34.0, 12, n, seed=79, dt=0.5, dyaw_deg=3.0, radius=16.0)
    return cfg, pkg.synth.make_scene(cfg)


def _bits(x):
    x = np.ascontiguousarray(x)
    return x.view({4: np.uint32, 8: np.uint64}[x.dtype.itemsize])


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("compat", [0, 1])
def test_capacity_as_total(pkg, compat, graphs):
    torch = pytest.importorskip("torch")
    cfg, scene = _scene(pkg, 700)
    sizes = (1, 129, 300, 0, 700, 640)
    al = [pkg.synth.make_alignment(cfg, scene, i, n_points=max(n, 1)) for i, n in enumerate(sizes)]
    B, n = len(sizes), sum(sizes)
    pts = torch.zeros((BOUND, 4), dtype=torch.float32, device="cuda")
    pts[:n] = torch.from_numpy(np.concatenate([a.scan[:k] for a, k in zip(al, sizes)])).cuda()
    off = torch.from_numpy(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)).cuda()
    guess = torch.from_numpy(np.stack([a.guess for a in al])).cuda()
    other = guess.clone()  # what an evaluation before leaves in the scratch
    other[:, 3] += 0.7
    prm = (pkg.ndt.reference_params if compat else pkg.ndt.corrected_params)(1.0)
    got = []
    with pkg.ndt.Context(prm) as ctx:
        ctx.set_batch_graphs(graphs)
        ctx.set_map(scene.map)
        for total in (n, BOUND):
            for g in (other, guess):
                out = torch.zeros((B, 16), dtype=torch.float32, device="cuda")
                conv, st = (torch.zeros(B, dtype=torch.int32, device="cuda") for _ in range(2))
                fit, score = (torch.zeros(B, dtype=torch.float64, device="cuda") for _ in range(2))
                torch.cuda.synchronize()
                ctx.score_batch_device(B, pts.data_ptr(), off.data_ptr(), total, g.data_ptr(), score.data_ptr())
                ctx.synchronize()
                ctx.align_batch_device(B, pts.data_ptr(), off.data_ptr(), total, g.data_ptr(), out.data_ptr(),
                                       conv.data_ptr(), fit.data_ptr(), st.data_ptr())
                ctx.synchronize()
            got.append([_bits(t.cpu().numpy()) for t in (score, out, conv, fit, st)])
    assert (got[0][0] != 0).sum() >= 4  # the scans have pairs
    for exact, bound in zip(*got):
        assert np.array_equal(exact, bound)


def _pipeline(pkg, torch, levels, net, prm, al):
    dev = pkg.learned.DeviceScans(torch, [a.scan for a in al])
    pts, off, total = dev.batch(np.arange(len(al)))
    lb = pkg.learned.LearnedBatch(levels, net, torch, pts, off, total, np.stack([a.guess for a in al]), prm)
    lb.run()
    return [_bits(r) for r in lb.results()]


def _same_alone(pkg, levels, prm, al, pick):
    torch = pytest.importorskip("torch")
    net = pkg.posenet.PoseNet(center=(0.0, 0.0, 0.0), scale=4.0)
    net.set_weights(pkg.posenet.init_weights(3))
    try:
        _pipeline(pkg, torch, levels, net, prm, al[::-1])  # other values in the scratch
        many = _pipeline(pkg, torch, levels, net, prm, al)
        for i in pick:
            for m, one in zip(many, _pipeline(pkg, torch, levels, net, prm, [al[i]])):
                assert np.array_equal(m[i], one[0]), i
    finally:
        net.close()
        for c in levels:
            c.close()


# the judge's bound is judge_points a scan: 560, 840 and 616 chunks, where the scans have 364, 504 and 392
@pytest.mark.parametrize("short,long", [([400] * 9, 20000), ([200] * 14, 100000), ([500] * 10, 30000)])
def test_judge_of_ragged_scans(pkg, short, long):
    cfg, scene = _scene(pkg, 500)
    al = [pkg.synth.make_alignment(cfg, scene, i, n_points=n) for i, n in enumerate(short + [long])]
    levels = pkg.learned.level_contexts(pkg.ndt, scene.map, 1.0)
    prm = pkg.learned.pipeline_params(pkg.learned.refinement_levels(1.0))
    _same_alone(pkg, levels, prm, al, range(len(al)))


def test_compat_levels_of_ragged_scans(pkg):
    cfg, scene = _scene(pkg, 100)
    al = [pkg.synth.make_alignment(cfg, scene, i, n_points=n) for i, n in enumerate([100] * 299 + [700000])]
    levels = []
    for res in (2.0, 1.0):
        ctx = pkg.ndt.Context(pkg.ndt.reference_params(res))
        ctx.set_map(scene.map)
        levels.append(ctx)
    prm = pkg.posenet.learned_params(grid_xy=1, grid_yaw=1, passes=0, judge_points=64, level_points=[2048, 0])
    _same_alone(pkg, levels, prm, al, (0, 1, 150, 299))
