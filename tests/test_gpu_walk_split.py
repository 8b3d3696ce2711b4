"""The ray-buffer walk at the counts where its split over warps changes: one
ray, a partial warp, block and chunk edges, one ray a warp, a few lanes a
warp, and lanes that refill."""
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
