"""Shading in class order over the whole queue (renders of at least 2^18 paths) against shading in queue
order: the same image and G-buffer bit for bit, at the smallest size that takes it, with path counts that
leave partial tiles and warps, with several generations of a small pool, and for batched views."""
import numpy as np
import pytest

from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu


def _scene(kind):
    g = native.box_scene() if kind == "box" else native.terrain_scene(65536, 3)
    return g, g.build()


@pytest.mark.parametrize("kind", ["box", "terrain"])
@pytest.mark.parametrize("w,h,spp,tuning", [
    (512, 512, 1, {}),                               # 2^18 paths exactly
    (509, 519, 2, {}),                               # odd, partial tiles
    (640, 360, 3, dict(path_capacity=(1 << 18) + 77, tail_paths=0)),  # several generations, every bounce queued
    (640, 360, 2, dict(sort_by_material=1, graph_bounces=0)),
])
def test_images_equal_queue_order(kind, w, h, spp, tuning):
    g, b = _scene(kind)
    cam = g.camera(w / h)
    out = []
    for t in (dict(tuning, sort_by_material=0), tuning):
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        r.set_tuning(**t)
        r.render(cam, abi.render_settings(w, h, max_depth=6, seed=2), spp)
        out.append((r.download_accumulation(), *r.download_gbuffer()))
        r.close()
    for x, y in zip(*out):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def test_batched_views_equal_single_renders():
    g, b = _scene("terrain")
    views = workloads.batch_views(b.desc, n=5, seed=4, max_depth=6)
    for v in views:
        v.spp = min(v.spp, 4)
    r = native.Renderer()
    r.upload(b.desc)
    r.render_views(views)
    got = [r.download_view(k, v.width, v.height) for k, v in enumerate(views)]
    r.set_tuning(sort_by_material=0)
    for k, v in enumerate(views):
        r.render_views([v])
        assert np.array_equal(got[k].view(np.uint32), r.download_view(0, v.width, v.height).view(np.uint32))
    r.close()
