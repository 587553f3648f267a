"""A server and a session lane that hold a scene whose tree may be walked out of order and, later, one whose tree
may not: each request's image and each session's first frame stay those of a renderer that holds the one scene."""
import numpy as np
import pytest

from photon_b200 import abi, native, workloads
from test_deep_stack import _deep_scene
from test_gpu_list_walk import _unnested

pytestmark = pytest.mark.gpu
W, H = 160, 96


def _render(desc, cam, spp):
    r = native.Renderer()
    r.upload(desc)
    walks = r.scene_walks()
    r.resize(W, H)
    r.set_tuning(pair_walk=0, tail_paths=0)
    r.render(cam, abi.render_settings(W, H, max_depth=6, seed=5), spp)
    img = r.download_image()
    r.close()
    return img, walks


def _frame(desc, cam):
    r = native.Renderer()
    r.upload(desc)
    r.resize(W, H)
    r.set_tuning(pair_walk=0, tail_paths=0)
    r.render_denoised(cam, cam, abi.render_settings(W, H, max_depth=6, seed=5), abi.svgf_settings())
    img = r.download_image()
    r.close()
    return img


def test_an_irregular_scene_joins():
    g = native.terrain_scene(65536, 2)
    b = g.build()
    odd, keep = _unnested(b.desc)
    cam = g.camera(W / H)
    want, walks = zip(*(_render(d, cam, 4) for d in (b.desc, odd)))
    assert walks == ((1, 1), (0, 0))
    frames = [_frame(d, cam) for d in (b.desc, odd)]
    s = native.Server(path_capacity=1 << 20, reserve_bytes=-1)
    path = abi.path_options(max_depth=6)

    def image(scene):
        rid = s.submit(scene, cam, W, H, 4, 5, path)
        s.wait(rid)
        return s.fetch(rid, W, H)[0]

    def frame(scene):
        session = s.open_session(scene, W, H)
        rid = s.submit_frame(session, cam, cam, abi.render_settings(W, H, max_depth=6, seed=5))
        s.wait(rid)
        img = s.fetch(rid, W, H)[0]
        s.close_session(session)
        return img

    first = s.add_scene(b.desc)
    assert np.array_equal(image(first), want[0]) and np.array_equal(frame(first), frames[0])
    second = s.add_scene(odd)
    for k in (0, 1, 0):
        assert np.array_equal(image((first, second)[k]), want[k]) and np.array_equal(frame((first, second)[k]), frames[k])
    s.close()


def test_the_walks_an_upload_allows():
    """A built tree is walked out of order, one deeper than the list walk's stack is not, whichever came before."""
    g = native.terrain_scene(65536, 2)
    b = g.build()
    deep, keep = _deep_scene()
    odd, keep2 = _unnested(b.desc)
    r = native.Renderer()
    for desc, walks in ((b.desc, (1, 1)), (deep, (0, 0)), (odd, (0, 0)), (b.desc, (1, 1))):
        r.upload(desc)
        assert r.scene_walks() == walks
    r.close()
