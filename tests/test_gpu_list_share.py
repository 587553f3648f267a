"""Ray queues shorter than the list walk's warps can hold are spread over all warps: images equal the walk in
Photon's order for a single ray, the least share, shares between it and a full warp, and just past one (the
grid has a few thousand warps; the queues shrink from bounce to bounce through the sizes below)."""
import numpy as np
import pytest

from photon_b200 import abi, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (203, 97), (257, 251), (401, 399), (640, 331)])
@pytest.mark.parametrize("refills", [(24, 24), (1, 32)])
def test_short_queues_equal_the_walk_in_photons_order(w, h, refills):
    g = native.terrain_scene(65536, 2)
    b = g.build()
    cam, out = g.camera(w / h), []
    for t in (dict(pair_walk=0), dict(trace_refill=refills[0], shadow_refill=refills[1])):
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        r.set_tuning(tail_paths=0, **t)
        r.render(cam, abi.render_settings(w, h, max_depth=8, seed=3), 1)
        out.append(r.download_accumulation())
        r.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
