"""Walks at the counts where their kernels and launch shapes change: ray buffers
of one ray, a partial warp, block and group edges, eight lanes a ray and one
ray a thread (test_gpu_ray_buffers.py has the larger, refilling ones), and
frames on both sides of the cooperative walk's limits and of the register
bound."""
import numpy as np
import pytest

from artemis_gb300 import kgr
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def box():
    return helpers.both("box64", 5)


@pytest.mark.parametrize("layout", [kgr.LAYOUT_FAST, kgr.LAYOUT_WIDE])
@pytest.mark.parametrize("n", [1, 3, 5, 31, 127, 129, 4863, 4865, 9729, 20000, 155649, 200003])
def test_every_ray_is_walked_once(box, n, layout):
    g, sc, osc = box
    rays = helpers.random_rays(g, n, n)
    ref, _ = osc.trace_closest(rays)
    got = sc.trace_closest_host(rays, layout)
    assert np.array_equal(got.view(np.uint32), ref["raw"].view(np.uint32))
    rays[:, 7] = np.random.default_rng(n).uniform(0.0, 4.0, n)
    occ_ref, _ = osc.trace_any(rays)
    assert np.array_equal(sc.trace_any_host(rays, layout), occ_ref)


def edge_rays(g, n):
    """Zero direction components, NaN directions, origins far away and on the
    scene's bounds, tmax 0, negative and NaN, among ordinary rays."""
    rays = helpers.random_rays(g, n, 11)
    rays[0::9, 4] = 0.0
    rays[1::9, 5] = -0.0
    rays[2::9, 4:6] = 0.0
    rays[3::9, 6] = np.nan
    rays[4::9, 0:3] -= 1000.0 * rays[4::9, 4:7]
    rays[5::9, 0] = g.positions[:, 0].min()
    rays[6::27, 7] = 0.0
    rays[15::27, 7] = -1.0
    rays[24::27, 7] = np.nan
    return rays


@pytest.mark.parametrize("n", [4000, 130000])
def test_edge_rays_on_both_sides_of_the_split(box, n):
    g, sc, _ = box
    rays = edge_rays(g, n)
    ref = sc.trace_closest_host(rays, kgr.LAYOUT_THREADED)
    got = sc.trace_closest_host(rays)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(sc.trace_any_host(rays), sc.trace_any_host(rays, kgr.LAYOUT_THREADED))


@pytest.mark.parametrize("scene,max_leaf", [("tiny", 4), ("box64", 1), ("box64", 8), ("terrain_s", 4)])
def test_small_counts_on_every_tree(scene, max_leaf):
    """A root of few children, one triangle a leaf, leaves too large for the
    eight-child tree (the persistent walk takes the rays), a deep tree."""
    g, sc, _ = helpers.both(scene, 2, max_leaf=max_leaf)
    rays = np.concatenate([helpers.random_rays(g, 9001, 3), edge_rays(g, 999)])
    ref = sc.trace_closest_host(rays, kgr.LAYOUT_THREADED)
    assert np.array_equal(sc.trace_closest_host(rays).view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(sc.trace_any_host(rays), sc.trace_any_host(rays, kgr.LAYOUT_THREADED))


@pytest.mark.parametrize("side", [48, 176, 256, 288])
@pytest.mark.parametrize("plugin", ["restir_di", "restir_gi"])
def test_restir_bounces_overlapped_or_not(plugin, side):
    """Bounces whose shadow rays run beside the next closest hits, at path
    counts on each side of the cooperative walk's limits: the same bits as
    one after the other."""
    torch = pytest.importorskip("torch")
    g, sc, _ = helpers.both("box64", 5)
    cam = kgr.camera(g.eye, g.target, g.fov, 1.0)
    images = []
    for overlap in (False, True):
        bufs = helpers.device_buffers(torch, side * side)
        att = kgr.Attachment(plugin)
        att.attach(side, side)
        att.load()
        att.set_option("trace_overlap", overlap)
        for frame in range(2):
            att.render(helpers.launch(cam, side, side, bufs, frame=frame, max_depth=3), sc)
        torch.cuda.synchronize()
        images.append(bufs[0].cpu().numpy())
        att.close()
    assert images[0][:, :3].mean() > 0.0
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))


@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("side", [499, 500, 512])
def test_frames_on_both_sides_of_the_register_bound(block, side):
    """Path counts around the one above which a walk takes more warps an SM:
    the same bits as with the register cap and on the threaded layout."""
    torch = pytest.importorskip("torch")
    g, sc, _ = helpers.both("box64", 5)
    cam = kgr.camera(g.eye, g.target, g.fov, 1.0)
    images = []
    for layout, occupancy in (("fast", 0), ("fast", 1), ("threaded", 0)):
        bufs = helpers.device_buffers(torch, side * side)
        att = kgr.Attachment("path_tracer")
        att.attach(side, side)
        att.load()
        att.set_option("layout", layout)
        att.set_option("trace_block", block)
        att.set_option("trace_occupancy", occupancy)
        att.render(helpers.launch(cam, side, side, bufs, frame=0, max_depth=3), sc)
        torch.cuda.synchronize()
        images.append(bufs[0].cpu().numpy().view(np.uint32))
        att.close()
    assert np.array_equal(images[0], images[1])
    assert np.array_equal(images[0], images[2])


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("layout", [kgr.LAYOUT_FAST, kgr.LAYOUT_WIDE])
@pytest.mark.parametrize("side", [700, 1001])
def test_coherent_ray_buffers(layout, side, mixed):
    """Camera rays, on both sides of the count where their launch changes, and
    the same with every 97th ray turned round: the threaded walk's hits."""
    g, sc, _ = helpers.both("box64", 5)
    rays = helpers.camera_rays(kgr.camera(g.eye, g.target, g.fov, 1.0), side, side)
    if mixed:
        rays[::97, 4:7] *= -1.0
    ref = sc.trace_closest_host(rays, kgr.LAYOUT_THREADED)
    assert np.array_equal(sc.trace_closest_host(rays, layout).view(np.uint32), ref.view(np.uint32))
    assert np.array_equal(sc.trace_any_host(rays, layout), sc.trace_any_host(rays, kgr.LAYOUT_THREADED))
