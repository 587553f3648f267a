"""One renderer that alternates renders on either side of the sizes at which its captured iterations change (class
order from 2^18 paths, ray sorting from 2^21), and renderers of different block sizes side by side: every image
equals a fresh renderer's."""
import numpy as np
import pytest

from photon_b200 import abi, native

pytestmark = pytest.mark.gpu


def test_alternating_renders_equal_fresh_ones():
    g = native.terrain_scene(65536, 2)
    b = g.build()
    w, h, spps = 640, 360, (1, 2, 10)  # 230,400, 460,800 and 2,304,000 paths
    cam, rs = g.camera(w / h), abi.render_settings(w, h, max_depth=5, seed=3)

    def image(r, spp):
        r.reset()
        r.render(cam, rs, spp)
        return r.download_accumulation()

    want = {}
    for spp in spps:
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        want[spp] = image(r, spp)
        r.close()
    r = native.Renderer()
    r.upload(b.desc)
    r.resize(w, h)
    for spp in (10, 1, 10, 2, 1, 2, 1, 10, 10, 2):
        assert np.array_equal(image(r, spp).view(np.uint32), want[spp].view(np.uint32)), spp
    r.set_tuning(graph_bounces=2)
    for spp in (1, 2, 1, 10):
        assert np.array_equal(image(r, spp).view(np.uint32), want[spp].view(np.uint32)), spp
    r.close()


def test_renderers_of_different_block_sizes_side_by_side():
    g = native.terrain_scene(65536, 2)
    b = g.build()
    w, h = 160, 90
    cam, rs, rr = g.camera(w / h), abi.render_settings(w, h, max_depth=5, seed=3), []
    for block in (256, 32, 128, 64):
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        r.set_tuning(trace_block=block)
        rr.append(r)
    images = []
    for t in (dict(pair_walk=5), dict(pair_walk=0), dict(packed=0), dict(wide_shadows=1)):
        for r in rr + rr:
            r.set_tuning(tail_paths=0, **t)
            r.reset()
            r.render(cam, rs, 1)
            images.append(r.download_accumulation())
    for r in rr:
        r.close()
    for img in images[1:]:
        assert np.array_equal(img.view(np.uint32), images[0].view(np.uint32))
