"""A map build or append whose sort gave up is reported by the next call that
waits for the context's work, whatever that call is, and nothing is computed
from the map afterwards; the context takes the next map (waits set to give up
before their first poll: ndt_set_sort_wait_limit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(pkg):
    cfg = pkg.synth.small_config("sort", 20000, 40.0, 16, 1500, seed=43, dt=0.4, dyaw_deg=3.0)
    scene = pkg.synth.make_scene(cfg)
    return scene.map, pkg.synth.make_alignment(cfg, scene, 0)


WAITS = {
    "synchronize": lambda c, a, m: c.synchronize(),
    "align": lambda c, a, m: c.align(a.scan, a.guess),
    "derivatives": lambda c, a, m: c.derivatives(a.scan, a.scan, np.zeros(6)),
    "grid_info": lambda c, a, m: c.grid_info(),
    "window_info": lambda c, a, m: c.window_info(),
    "set_map": lambda c, a, m: c.set_map(m),
    "append": lambda c, a, m: c.map_append(m[:5000]),
}


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("step", ["set_map", "append"])
@pytest.mark.parametrize("wait", sorted(WAITS))
def test_reported_by_the_next_wait(pkg, wait, step, graphs):
    cloud, a = _map(pkg)
    with pkg.ndt.Context(pkg.ndt.corrected_params(1.0)) as ctx:
        ctx.set_batch_graphs(graphs)
        ctx.set_map(cloud)
        want = ctx.align(a.scan, a.guess)
        ctx.set_sort_wait_limit(0)
        if step == "set_map":
            ctx.set_map(cloud)
        else:
            ctx.map_append(cloud[:6000])
        ctx.set_sort_wait_limit(-1)
        with pytest.raises(pkg.ndt.NdtError, match="NDT_E_CUDA"):
            WAITS[wait](ctx, a, cloud)
        with pytest.raises(pkg.ndt.NdtError, match="NDT_E_NOMAP"):
            ctx.map_append(cloud[:5000])
        with pytest.raises(pkg.ndt.NdtError, match="NDT_E_NOMAP"):
            ctx.align(a.scan, a.guess)
        ctx.set_map(cloud)
        got = ctx.align(a.scan, a.guess)
        assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]


def test_align_with_map(pkg):
    cloud, a = _map(pkg)
    with pkg.ndt.Context(pkg.ndt.reference_params(1.0)) as ctx:
        want = ctx.align_with_map(a.scan, a.guess, cloud)
        ctx.set_sort_wait_limit(0)
        with pytest.raises(pkg.ndt.NdtError, match="NDT_E_CUDA"):
            ctx.align_with_map(a.scan, a.guess, cloud)
        ctx.set_sort_wait_limit(-1)
        got = ctx.align_with_map(a.scan, a.guess, cloud)
        assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]
