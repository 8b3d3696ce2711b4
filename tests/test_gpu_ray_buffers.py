"""Ray buffers at the counts and of the kinds among which their kernels change:
incoherent rays that refill their lanes, coherent ones by one ray a thread and
by whole warps, buffers that look coherent where they are probed and are not
elsewhere, and the other way round.  The threaded walk's hits bit for bit."""
import numpy as np
import pytest

from artemis_gb300 import kgr
from tests import helpers
from tests.test_gpu_walk_split import edge_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def box():
    return helpers.both("box64", 5)


def same_as_threaded(sc, rays, layout):
    ref = sc.trace_closest_host(rays, kgr.LAYOUT_THREADED)
    assert np.array_equal(sc.trace_closest_host(rays, layout).view(np.uint32), ref.view(np.uint32))
    short = rays.copy()
    finite = ~np.isnan(short[:, 7])
    short[finite, 7] = np.random.default_rng(len(rays)).uniform(0.0, 4.0, finite.sum())
    for r in (rays, short):
        assert np.array_equal(sc.trace_any_host(r, layout), sc.trace_any_host(r, kgr.LAYOUT_THREADED))


@pytest.mark.parametrize("layout", [kgr.LAYOUT_FAST, kgr.LAYOUT_WIDE])
@pytest.mark.parametrize("n", [400003, 777777, 1000001])
def test_incoherent_rays_refill_their_lanes(box, n, layout):
    """Random rays with zero and NaN directions, far origins and every kind of
    tmax among them."""
    g, sc, _ = box
    rays = helpers.random_rays(g, n, n)
    rays[::3] = edge_rays(g, len(rays[::3]))
    same_as_threaded(sc, rays, layout)


def per_thread_rays():
    """Rays that the grid of one ray a thread holds at once."""
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count * 16 * 128


@pytest.mark.parametrize("layout", [kgr.LAYOUT_FAST, kgr.LAYOUT_WIDE])
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("turned", [None, 7, "between"])
def test_coherent_rays_on_both_sides_of_whole_warps(box, turned, over, layout):
    """Camera rays up to and past three rounds of the per-thread grid; with
    every seventh ray turned round (incoherent where the buffer is probed); and
    with random rays everywhere but where it is probed."""
    g, sc, _ = box
    n = 3 * per_thread_rays() + over
    side = int(np.ceil(np.sqrt(n)))
    rays = helpers.camera_rays(kgr.camera(g.eye, g.target, g.fov, 1.0), side, side)[:n].copy()
    if turned == 7:
        rays[::7, 4:7] *= -1.0
    elif turned == "between":
        at = np.arange(n)
        probed = np.zeros(n, bool)
        for k in (1, 3, 5, 7):
            probed |= (at >= k * (n // 8)) & (at < k * (n // 8) + 32)
        rays[~probed] = helpers.random_rays(g, n, 2)[~probed]
    same_as_threaded(sc, rays, layout)
