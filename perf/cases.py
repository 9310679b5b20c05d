"""The work that a user of this library has it do, as timed cases.

Eleven kinds of work, each through the entry points that a program calls:

  call      ndt_align_with_map: the DAPHNE align call (scan, guess and map in host memory), as the harness makes it
  scan      ndt_align: one host scan after the other against a map that stays set (corrected NDT, a localiser's loop)
  batch     ndt_align_batch_device: a batch of scans against the map of the call (grid built, then aligned), or
            against a map that stays set; compat or corrected mode, FP32 or FP64 pairs
  rescore   ndt_set_map_device + ndt_score_batch_device: pose hypotheses scored against a fresh map tile
  mapping   ndt_set_map, then align a scan and append it to the map, again and again (the map of ndt_mapping grows)
  learned   ndt_align_batch_learned_device: network proposals, the NDT judge, coarse-to-fine refinement
  train     ndt_mlp_train_step_device: forward, backward and Adam step of the pose network
  filter    ndt_voxel_filter_device: voxel-grid downsampling of raw sweeps
  cluster   ndt_ec_segment_batch: euclidean clustering of host clouds (five distance rings, boxes)

Clouds are the workload of daphne-benchmark_b200/synth.py (a noisy ground
plane and vertical walls, scans within 40 m of a sensor pose, ordered by 2 m
leaf), drawn on the GPU so that large batches are made quickly.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("daphne-benchmark_b200")
ndt, posenet, learned = pkg.ndt, pkg.posenet, pkg.learned

DEV = "cuda"


def listed():
    return [
        # the reference's own call shape on its smallest configuration: latency, copies and launches
        dict(name="call_2k_map60k", kind="call", map=60_000, area=60.0, walls=30, n=2000, res=1.0, compat=1),
        # one scan of a localiser against the map it keeps: up to 30 dependent Newton steps, one launch chain
        dict(name="scan_8k_corrected", kind="scan", map=400_000, area=150.0, walls=120, n=8000, res=1.0, compat=0,
             dt=0.5, dyaw=3.0),
        # the benchmark-scale batch: 256 scans of 8000 points, compat mode, the grid built in the pass
        dict(name="batch_256x8k_compat", kind="batch", map=400_000, area=150.0, walls=120, B=256, lo=8000, hi=8000,
             res=1.0, compat=1, fp64=0, build=1, dt=0.5, dyaw=3.0),
        # ragged scans (1k to 16k points) that converge at different rounds, map kept
        dict(name="batch_1024_ragged", kind="batch", map=400_000, area=150.0, walls=120, B=1024, lo=1000, hi=16000,
             res=1.0, compat=0, fp64=0, build=0, dt=1.0, dyaw=5.0),
        # the largest workload: a 2M-point map at 0.5 m, 4096 scans of 2k to 32k points
        dict(name="batch_4096_fine", kind="batch", map=2_000_000, area=300.0, walls=400, B=4096, lo=2000, hi=32000,
             res=0.5, compat=0, fp64=0, build=1, dt=3.0, dyaw=15.0),
        # the FP64 pair option, used where results are compared with the CPU's
        dict(name="batch_33_fp64", kind="batch", map=250_001, area=120.0, walls=77, B=33, lo=1001, hi=7001, res=1.0,
             compat=0, fp64=1, build=0, dt=0.5, dyaw=3.0),
        # relocalisation: 512 hypotheses on a fresh tile of 2M points at 0.5 m; grid build and one evaluation
        dict(name="rescore_512_map2m", kind="rescore", map=2_000_000, area=300.0, walls=400, B=512, lo=2048, hi=2048,
             res=0.5, dt=1.0, dyaw=5.0),
        # mapping: six odd-sized scans aligned and appended to a growing map
        dict(name="mapping_6x3001", kind="mapping", map=199_999, area=110.0, walls=60, steps=6, n=3001, res=1.0,
             dt=0.3, dyaw=3.0),
        # learned initial pose: 27 starts a scan through the network, judged, refined at 4, 2 and 1 m
        dict(name="learned_256", kind="learned", map=400_000, area=150.0, walls=120, B=256, lo=2000, hi=8000, res=1.0,
             dt=2.0, dyaw=10.0),
        # one training step of the pose network: the batch of the benchmark's schedule
        dict(name="train_256x1024", kind="train", B=256, lo=1500, hi=3000, points=1024),
        # the pre-filter at 256 raw sweeps of 65536 points
        dict(name="filter_256x65536", kind="filter", B=256, lo=65536, hi=65536, leaf=2.0),
        # five clouds of the size of the reference's euclidean_cluster inputs
        dict(name="cluster_5x10k", kind="cluster", clouds=5, n=9600),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "scan", "batch", "batch", "batch", "rescore", "mapping", "learned", "train", "filter",
                       "cluster"])
    m = log(20_000, 2_000_000)
    area = round(math.sqrt(m / 20.0) * rng.uniform(0.8, 1.3), 1)  # about the density of the listed maps
    walls = max(8, int(area * area / 190))
    res = rng.choice([0.5, 1.0, 1.0, 2.0, 0.7])
    scene = dict(map=m, area=area, walls=walls, res=res)
    dt, dyaw = round(rng.uniform(0.2, 3.0), 2), round(rng.uniform(1.0, 15.0), 1)
    if kind == "call":
        return dict(kind=kind, n=log(300, 32000), compat=rng.choice([1, 1, 0]), **scene)
    if kind == "scan":
        return dict(kind=kind, n=log(300, 32000), compat=rng.choice([0, 0, 1]), dt=dt, dyaw=dyaw, **scene)
    if kind == "batch":
        lo = log(500, 8000)
        hi = max(lo, log(lo, 32000))
        fp64 = rng.choice([0, 0, 0, 0, 1])
        cap = 2_000_000 if fp64 else 30_000_000
        return dict(kind=kind, B=max(2, min(log(4, 4096), cap // hi)), lo=lo, hi=hi, compat=rng.choice([0, 1]),
                    fp64=fp64, build=rng.choice([0, 1]), dt=dt, dyaw=dyaw, **scene)
    if kind == "rescore":
        lo = log(500, 4000)
        return dict(kind=kind, B=log(16, 2048), lo=lo, hi=max(lo, log(lo, 4000)), dt=dt, dyaw=dyaw, **scene)
    if kind == "mapping":
        return dict(kind=kind, steps=rng.randint(2, 8), n=log(500, 8000), dt=min(dt, 1.0), dyaw=min(dyaw, 5.0),
                    **scene)
    if kind == "learned":
        lo = log(1000, 4000)
        scene["res"] = rng.choice([0.5, 1.0])
        return dict(kind=kind, B=log(8, 512), lo=lo, hi=max(lo, log(lo, 16000)), dt=dt, dyaw=dyaw, **scene)
    if kind == "train":
        points = log(128, 1024)
        return dict(kind=kind, B=log(16, 1024), lo=log(100, 1500), hi=log(1500, 4000), points=points)
    if kind == "filter":
        lo = log(2000, 65536)
        return dict(kind=kind, B=log(1, 200), lo=lo, hi=max(lo, log(lo, 120_000)), leaf=rng.choice([2.0, 1.0, 0.5, 1.7]))
    return dict(kind="cluster", clouds=rng.randint(1, 12), n=log(500, 20000))


# ---------------------------------------------------------------------------
# Inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _noise(g, n, sigma=0.02):
    return (_rand(g, 4, n).sum(0) - 2.0) * (math.sqrt(3.0) * sigma)


def _scene(g, m, area, walls):
    """Wall table (K x 7: centre, direction, length, height, area) and the map cloud (m x 4 float32)."""
    c = (_rand(g, walls, 2) - 0.5) * area
    ang = _rand(g, walls) * math.pi
    length, height = 2.0 + 8.0 * _rand(g, walls), 1.0 + 3.0 * _rand(g, walls)
    w = torch.stack([c[:, 0], c[:, 1], torch.cos(ang), torch.sin(ang), length, height, length * height], 1)
    n_wall = int(m * float(w[:, 6].sum()) / (area * area + float(w[:, 6].sum())))
    cum = torch.cumsum(w[:, 6], 0)
    pick = torch.searchsorted(cum, _rand(g, n_wall) * cum[-1]).clamp_(max=walls - 1)
    n_ground = m - n_wall
    ground = torch.cat([(_rand(g, n_ground, 2) - 0.5) * area, _noise(g, n_ground)[:, None]], 1)
    pts = torch.cat([ground, _on_walls(g, w, pick)], 0)[torch.randperm(m, generator=g, device=DEV)]
    cloud = torch.ones(m, 4, device=DEV)
    cloud[:, :3] = pts.float()
    return w, cloud


def _on_walls(g, w, pick):
    v = w[pick]
    n = len(pick)
    s, h, e = (_rand(g, n) - 0.5) * v[:, 4], _rand(g, n) * v[:, 5], _noise(g, n)
    return torch.stack([v[:, 0] + s * v[:, 2] - e * v[:, 3], v[:, 1] + s * v[:, 3] + e * v[:, 2], h], 1)


def _sizes(B, lo, hi):
    """B scan sizes, log-uniform in [lo, hi] (the same total for every seed)."""
    if B == 1 or lo == hi:
        return np.full(B, lo, np.int64)
    return np.round(np.exp(np.linspace(math.log(lo), math.log(hi), B))).astype(np.int64)


def _scans(g, walls, area, sizes, dt, dyaw, radius=40.0, order="leaf"):
    """Packed scans in their sensor frames, offsets, and the guesses (truth perturbed by dt, dyaw)."""
    B = len(sizes)
    sizes = sizes[torch.randperm(B, generator=g, device=DEV).cpu().numpy()]
    off = np.zeros(B + 1, np.int64)
    off[1:] = np.cumsum(sizes)
    n = int(off[-1])
    of = torch.repeat_interleave(torch.arange(B, device=DEV), torch.from_numpy(sizes).to(DEV))
    half = area / 2.0
    pose = (_rand(g, B, 2) - 0.5) * half
    yaw = (_rand(g, B) * 2 - 1) * math.pi
    # walls within reach of each sensor, and how much of the visible surface they are
    near = ((walls[None, :, :2] - pose[:, None, :]).square().sum(2) < (radius - 5.0) ** 2) * walls[None, :, 6]
    x0, x1 = (pose - radius).clamp(min=-half), (pose + radius).clamp(max=half)
    ground = (x1 - x0).prod(1) * (math.pi / 4)
    cum = torch.cumsum(near.reshape(-1), 0)
    end = cum[len(walls) - 1::len(walls)]
    tot = torch.diff(end, prepend=end.new_zeros(1))
    is_wall = _rand(g, n) < (tot / (tot + ground))[of]
    xyz = torch.empty(n, 3, device=DEV, dtype=torch.float64)
    wi = torch.nonzero(is_wall)[:, 0]
    ow = of[wi]
    pick = torch.searchsorted(cum, (end - tot)[ow] + tot[ow] * _rand(g, len(wi)).clamp(1e-9, 1 - 1e-9))
    xyz[wi] = _on_walls(g, walls, (pick - ow * len(walls)).clamp(0, len(walls) - 1))
    gi = torch.nonzero(~is_wall)[:, 0]
    og = of[gi]
    p0, lo, ext = pose[og], x0[og], (x1 - x0)[og]
    p = lo + _rand(g, len(gi), 2) * ext
    for _ in range(6):  # inside the circle of view
        out = (p - p0).square().sum(1) > radius * radius
        p = torch.where(out[:, None], lo + _rand(g, len(gi), 2) * ext, p)
    xyz[gi, 0], xyz[gi, 1], xyz[gi, 2] = p[:, 0], p[:, 1], _noise(g, len(gi))
    c, s = torch.cos(yaw)[of], torch.sin(yaw)[of]
    dx, dy = xyz[:, 0] - pose[of, 0], xyz[:, 1] - pose[of, 1]
    scan = torch.ones(n, 4, device=DEV)
    scan[:, 0], scan[:, 1], scan[:, 2] = (c * dx + s * dy).float(), (c * dy - s * dx).float(), xyz[:, 2].float()
    if order == "leaf":  # as a voxel-grid filter leaves them: by 2 m leaf, x fastest
        q = torch.floor(scan[:, :3].double() / 2.0).long() + 1024
        key = ((of * 2048 + q[:, 2]) * 2048 + q[:, 1]) * 2048 + q[:, 0]
    else:  # a raw sweep: by azimuth
        scan[:, 3] = (_rand(g, n) * 255.0).float()
        key = of.double() * 8.0 + torch.atan2(scan[:, 1], scan[:, 0]).double()
    scan = scan[torch.sort(key, stable=True)[1]]
    err = (_rand(g, B, 2) * 2 - 1) * dt
    gy = yaw + (_rand(g, B) * 2 - 1) * math.radians(dyaw)
    guess = torch.zeros(B, 16, device=DEV)
    gc, gs = torch.cos(gy).float(), torch.sin(gy).float()
    guess[:, 0], guess[:, 1], guess[:, 4], guess[:, 5], guess[:, 10], guess[:, 15] = gc, -gs, gs, gc, 1.0, 1.0
    guess[:, 3], guess[:, 7] = (pose[:, 0] + err[:, 0]).float(), (pose[:, 1] + err[:, 1]).float()
    return scan.contiguous(), torch.from_numpy(off.astype(np.int32)).to(DEV), guess


def _clouds(g, clouds, n):
    """Obstacle points around a sensor as euclidean_cluster takes them: most within 15 m, z in [-1.3, 0.5]."""
    out = []
    for _ in range(clouds):
        k = 14 + int(_rand(g, 1) * 30)
        r = torch.where(_rand(g, k) < 0.55, 3.0 + 12.0 * _rand(g, k), 15.0 + 60.0 * _rand(g, k))
        a = _rand(g, k) * 2 * math.pi
        wt = 1.0 / r.square()
        pick = torch.searchsorted(torch.cumsum(wt, 0), _rand(g, n) * wt.sum()).clamp_(max=k - 1)
        b, l, d = _rand(g, k) * math.pi, 0.6 + 7.0 * _rand(g, k), 0.3 + 1.5 * _rand(g, k)
        u, v = (_rand(g, n) - 0.5) * l[pick], (_rand(g, n) - 0.5) * d[pick]
        x = (r * torch.cos(a))[pick] + torch.cos(b)[pick] * u - torch.sin(b)[pick] * v
        y = (r * torch.sin(a))[pick] + torch.sin(b)[pick] * u + torch.cos(b)[pick] * v
        z = -1.3 + 1.8 * _rand(g, n) * (0.3 + 0.7 * _rand(g, k))[pick]
        out.append(torch.stack([x, y, z], 1).float().cpu().numpy())
    return out


def _params(case):
    p = (ndt.reference_params if case.get("compat") else ndt.corrected_params)(case["res"])
    p.precision = int(case.get("fp64", 0))
    return p


def _outputs(B):
    return dict(out=torch.zeros(B, 16, device=DEV), conv=torch.zeros(B, dtype=torch.int32, device=DEV),
                fit=torch.zeros(B, dtype=torch.float64, device=DEV),
                status=torch.zeros(B, dtype=torch.int32, device=DEV))


def _network(seed, center=(0.0, 0.0, 0.0), scale=4.0):
    net = posenet.PoseNet(0, center, scale)
    net.set_weights(posenet.init_weights(seed))
    return net


def _train_inputs(case, seed):
    g = _gen(seed)
    area = 150.0
    walls, _ = _scene(g, 1000, area, 120)
    pts, off, guess = _scans(g, walls, area, _sizes(case["B"], case["lo"], case["hi"]), 2.0, 10.0)
    target = torch.randn(case["B"], 6, generator=g, device=DEV)
    return pts, off, guess, target


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed)
    if kind == "train":
        pts, off, guess, target = _train_inputs(case, seed)
        return dict(case=case, net=_network(seed), pts=pts, off=off, guess=guess, target=target)
    if kind == "filter":
        walls, _ = _scene(g, 1000, 150.0, 120)
        pts, off, _ = _scans(g, walls, 150.0, _sizes(case["B"], case["lo"], case["hi"]), 0.0, 0.0, 60.0, "sweep")
        return dict(case=case, filter=pkg.voxel_filter.VoxelFilter(0), pts=pts, off=off,
                    out=torch.zeros_like(pts), out_off=torch.zeros_like(off))
    if kind == "cluster":
        n = case["clouds"] * case["n"]
        return dict(case=case, ec=pkg.ec.EuclideanClusters(0), clouds=_clouds(g, case["clouds"], case["n"]),
                    got=[np.zeros((n, 3), np.float32), np.zeros((n, 10)), np.zeros((n, 3))])
    walls, cloud = _scene(g, case["map"], case["area"], case["walls"])
    sizes = _sizes(case["B"], case["lo"], case["hi"]) if "B" in case else np.full(case.get("steps", 1), case["n"])
    pts, off, guess = _scans(g, walls, case["area"], sizes, case.get("dt", 0.5), case.get("dyaw", 3.0))
    s = dict(case=case, pts=pts, off=off, guess=guess, cloud=cloud, total=int(sizes.sum()))
    if kind == "learned":
        host = cloud.cpu().numpy()
        s["levels"] = learned.level_contexts(ndt, host, case["res"])
        s["params"] = learned.pipeline_params(learned.refinement_levels(case["res"]))
        s["net"] = _network(seed)
        s.update(_outputs(case["B"]), choice=torch.zeros(case["B"], dtype=torch.int32, device=DEV),
                 start=torch.zeros(case["B"], 16, device=DEV))
        return s
    s["ctx"] = ndt.Context(_params(case))
    if kind in ("call", "scan", "mapping"):  # host buffers, as the harness and a mapping loop hold them
        s["scans"] = list(pts.cpu().numpy().reshape(-1, case["n"], 4))
        s["guesses"] = list(guess.cpu().numpy())
        s["map"] = cloud.cpu().numpy()
        for k in ("pts", "off", "guess", "cloud"):
            del s[k]
        if kind == "scan":
            s["ctx"].set_map(s["map"])
        return s
    if kind == "rescore":
        s["score"] = torch.zeros(case["B"], dtype=torch.float64, device=DEV)
        return s
    s.update(_outputs(case["B"]))
    if not case["build"]:
        torch.cuda.synchronize()  # the context works on its own stream
        s["ctx"].set_map_device(cloud.data_ptr(), case["map"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "call":
        return s["ctx"].align_with_map(s["scans"][0], s["guesses"][0], s["map"])
    if kind == "scan":
        return s["ctx"].align(s["scans"][0], s["guesses"][0])
    if kind == "batch":
        c = s["ctx"]
        if case["build"]:
            c.set_map_device(s["cloud"].data_ptr(), case["map"])
        c.align_batch_device(case["B"], s["pts"].data_ptr(), s["off"].data_ptr(), s["total"], s["guess"].data_ptr(),
                             s["out"].data_ptr(), s["conv"].data_ptr(), s["fit"].data_ptr(), s["status"].data_ptr())
        return [s["out"], s["conv"], s["fit"], s["status"]]
    if kind == "rescore":
        c = s["ctx"]
        c.set_map_device(s["cloud"].data_ptr(), case["map"])
        c.score_batch_device(case["B"], s["pts"].data_ptr(), s["off"].data_ptr(), s["total"], s["guess"].data_ptr(),
                             s["score"].data_ptr())
        return s["score"]
    if kind == "mapping":
        c = s["ctx"]
        c.set_map(s["map"])
        got = []
        for scan, guess in zip(s["scans"], s["guesses"]):
            T, conv, fit = c.align(scan, guess)
            got += [T, conv, fit]
            world = np.ones_like(scan)
            world[:, :3] = scan[:, :3] @ T.reshape(4, 4)[:3, :3].T + T.reshape(4, 4)[:3, 3]
            c.map_append(world)
        return got
    if kind == "learned":
        s["net"].align_learned_device(s["levels"], s["params"], case["B"], s["pts"].data_ptr(), s["off"].data_ptr(),
                                      s["total"], s["guess"].data_ptr(), s["out"].data_ptr(), s["conv"].data_ptr(),
                                      s["fit"].data_ptr(), s["status"].data_ptr(), s["choice"].data_ptr(),
                                      s["start"].data_ptr())
        return [s["out"], s["conv"], s["fit"], s["status"], s["choice"], s["start"]]
    if kind == "train":
        loss, grad = s["net"].train_step(case["B"], s["pts"].data_ptr(), s["off"].data_ptr(), s["guess"].data_ptr(),
                                         s["target"].data_ptr(), lr=2e-3, update=True, max_points=case["points"],
                                         want_grad=True)
        return [loss, grad]
    if kind == "filter":
        k = s["filter"].filter_device(case["B"], s["pts"].data_ptr(), s["off"].data_ptr(), len(s["pts"]),
                                      case["leaf"], s["out"].data_ptr(), s["out_off"].data_ptr())
        return [s["out"], s["out_off"], k]
    clouds = s["ec"].segment_batch(s["clouds"])
    at = [0, 0, 0]
    for c in clouds:  # clustered points, boxes and centroids of all clouds, one after the other
        for i in range(3):
            s["got"][i][at[i]:at[i] + len(c[i])] = c[i]
            at[i] += len(c[i])
    return s["got"] + [np.array([[len(x) for x in c] for c in clouds])]


def work(case):
    """Each input read once and each output written once.  Arithmetic of the
    alignments: a point's transform, its part of the 6-gradient and Hessian
    and one voxel pair (about 300 operations) for the fewest evaluations a run
    makes (compat: 3; corrected: the start, one trial and one closing pass)."""
    kind = case["kind"]
    if kind == "filter":
        n = int(_sizes(case["B"], case["lo"], case["hi"]).sum())
        return dict(bytes=16 * n + 4 * case["B"], flops=10 * n)
    if kind == "cluster":
        n = case["clouds"] * case["n"]
        return dict(bytes=24 * n, flops=100 * n)
    if kind == "train":
        n = int(np.minimum(_sizes(case["B"], case["lo"], case["hi"]), case["points"]).sum())
        w = posenet.num_weights()
        return dict(bytes=16 * n + 28 * w, flops=2 * n * (3 * 64 + 64 * 128) + 6 * case["B"] * (128 * 64 + 64 * 6))
    n = int(_sizes(case["B"], case["lo"], case["hi"]).sum()) if "B" in case else case["n"] * case.get("steps", 1)
    B = case.get("B", case.get("steps", 1))
    m = case["map"] if kind in ("call", "rescore", "mapping") or case.get("build") else 0
    nbytes = 16 * (n + m) + 144 * B
    if kind == "rescore":
        return dict(bytes=nbytes, flops=60 * n + 30 * m)
    flops = 3 * 300 * n + 30 * m
    if kind == "learned":  # 27 starts x 2 passes of the network, 28 scores on 2048 points, three levels
        sizes = _sizes(case["B"], case["lo"], case["hi"])
        net = int(np.minimum(sizes, 1024).sum()) * 54 * 2 * (3 * 64 + 64 * 128)
        flops = net + int(np.minimum(sizes, 2048).sum()) * 28 * 60 + 3 * flops
    return dict(bytes=nbytes, flops=flops)


# ---------------------------------------------------------------------------
# The same in 64 bits, by plain torch
def exact(case, seed):
    kind = case["kind"]
    if kind == "filter":
        s = prepare(case, seed)
        r = 1.0 / np.float32(case["leaf"])
        off = s["off"].long()
        of = torch.repeat_interleave(torch.arange(case["B"], device=DEV), off[1:] - off[:-1])
        q = torch.floor(s["pts"][:, :3] * float(r)).long()
        q = q - q.min(0)[0]
        d = q.max(0)[0] + 1
        key = ((of * d[2] + q[:, 2]) * d[1] + q[:, 1]) * d[0] + q[:, 0]
        u, inv, cnt = torch.unique(key, return_inverse=True, return_counts=True)
        mean = torch.zeros(len(u), 4, dtype=torch.float64, device=DEV).index_add_(0, inv, s["pts"].double())
        out = torch.zeros(len(inv), 4, dtype=torch.float64, device=DEV)
        out[:len(u)] = mean / cnt[:, None]
        return [out, None, None]
    if kind == "train":
        return _train_exact(case, seed)
    if kind == "rescore":
        return _score_exact(case, seed)
    return None  # iterated poses and host clusters: no closed form


def _train_exact(case, seed):
    pts, off, guess, target = _train_inputs(case, seed)
    off = off.cpu().numpy().astype(np.int64)
    w = torch.from_numpy(posenet.init_weights(seed)).to(DEV).double().requires_grad_()
    o = np.cumsum([0, 192, 64, 8192, 128, 8192, 64, 384, 6])
    W1, b1, W2, b2, W3, b3, W4, b4 = (w[o[i]:o[i + 1]] for i in range(8))
    feats = []
    for b in range(case["B"]):
        n = int(off[b + 1] - off[b])
        P = min(n, case["points"])
        at = torch.from_numpy(off[b] + (np.arange(P) * n) // P).to(DEV)
        T = guess[b].double().reshape(4, 4)
        u = (pts[at, :3].double() @ T[:3, :3].T + T[:3, 3]) / 4.0
        h = torch.relu(u @ W1.reshape(64, 3).T + b1)
        feats.append(torch.relu(h @ W2.reshape(128, 64).T + b2).max(0)[0])
    h3 = torch.relu(torch.stack(feats) @ W3.reshape(64, 128).T + b3)
    loss = (h3 @ W4.reshape(6, 64).T + b4 - target.double()).square().mean(1).mean()
    loss.backward()
    return [loss.detach(), w.grad]


def _score_exact(case, seed):
    s = prepare(case, seed)
    res = case["res"]
    cloud, r32 = s["cloud"], torch.tensor(res, dtype=torch.float32, device=DEV)
    lo, hi = cloud[:, :3].min(0)[0] - 0.01, cloud[:, :3].max(0)[0] + 0.01
    dim = ((hi - lo) / r32 + 1).long()

    def cell(v):  # the voxel a float coordinate belongs to
        return ((v - lo) / r32).long()

    def key(c):
        return c[:, 0] + dim[0] * (c[:, 1] + dim[1] * c[:, 2])

    vox, inv, cnt = torch.unique(key(cell(cloud[:, :3])), return_inverse=True, return_counts=True)
    x = cloud[:, :3].double()
    mean = torch.zeros(len(vox), 3, dtype=torch.float64, device=DEV).index_add_(0, inv, x) / cnt[:, None]
    d = x - mean[inv]
    cov = torch.zeros(len(vox), 9, dtype=torch.float64, device=DEV)
    cov.index_add_(0, inv, (d[:, :, None] * d[:, None, :]).reshape(-1, 9))
    use = cnt >= 6
    vox, mean = vox[use], mean[use]
    cov = (cov[use] / (cnt[use] - 1)[:, None]).reshape(-1, 3, 3)
    ev, V = (torch.from_numpy(v).to(DEV) for v in np.linalg.eigh(cov.cpu().numpy()))
    ev = torch.maximum(ev, 0.01 * ev[:, 2:])
    icov = V @ (V.transpose(1, 2) / ev[:, :, None])
    p = s["ctx"].params
    c1, c2 = 10 * (1 - p.outlier_ratio), p.outlier_ratio / float(r32) ** 3
    d3 = -math.log(c2)
    d1 = -math.log(c1 + c2) - d3
    d2 = -2 * math.log((-math.log(c1 * math.exp(-0.5) + c2) - d3) / d1)
    off = s["off"].long()
    of = torch.repeat_interleave(torch.arange(case["B"], device=DEV), off[1:] - off[:-1])
    T = s["guess"].double().reshape(-1, 4, 4)
    score = torch.zeros(case["B"], dtype=torch.float64, device=DEV)
    for at in torch.arange(len(of), device=DEV).split(1 << 20):
        Tb = T[of[at]]
        q = (Tb[:, :3, :3] @ s["pts"][at, :3].double()[:, :, None])[:, :, 0] + Tb[:, :3, 3]
        for k in range(27):
            step = torch.tensor([k % 3 - 1, k // 3 % 3 - 1, k // 9 - 1], dtype=torch.float64, device=DEV)
            v = q + step * res
            inside = ((v >= lo.double()) & (v <= hi.double())).all(1)
            c = key(((v - lo.double()) / float(r32)).long())
            j = torch.searchsorted(vox, c).clamp(max=len(vox) - 1)
            e = q - mean[j]
            ok = inside & (vox[j] == c) & (e.square().sum(1).sqrt() < float(r32))
            ok = torch.nonzero(ok)[:, 0]
            e, j = e[ok], j[ok]
            ex = torch.exp(-d2 * (e * (icov[j] @ e[:, :, None])[:, :, 0]).sum(1) / 2)
            score.index_add_(0, of[at][ok], torch.where(d2 * ex <= 1, -d1 * ex, torch.zeros_like(ex)))
    return score
