"""The camera walk of a frame at the path counts where the cooperative walk
gives way, which is earlier on a small tree than on a large one: the threaded
layout's images bit for bit."""
import numpy as np
import pytest

from artemis_gb300 import kgr
from tests import helpers

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["box4k", "terrain_s"])
@pytest.mark.parametrize("w,h", [(304, 192), (305, 192), (304, 256), (305, 256)])
@pytest.mark.parametrize("overlap", [True, False])
def test_camera_walks_on_both_sides_of_the_limits(scene, w, h, overlap):
    """58,368 and 77,824 paths, three and four for each group of lanes that
    152 SMs hold, and a column more."""
    g, sc, _ = helpers.both(scene, 1)
    cam = kgr.camera(g.eye, g.target, g.fov, w / h)
    images = []
    for layout in ("fast", "threaded"):
        bufs = helpers.device_buffers(torch, w * h)
        att = kgr.Attachment("path_tracer")
        att.attach(w, h)
        att.load()
        att.set_option("layout", layout)
        att.set_option("trace_overlap", overlap)
        att.render(helpers.launch(cam, w, h, bufs, frame=1, max_depth=3), sc)
        torch.cuda.synchronize()
        images.append([b.cpu().numpy().view(np.uint32) for b in bufs])
        att.close()
    for a, b in zip(*images):
        assert np.array_equal(a, b)
