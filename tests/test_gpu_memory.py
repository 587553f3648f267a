"""What scenes and path pools hold on the device is what the server counts (its budget bounds it), and buffers
that share memory hold the right thing at the right time."""
import numpy as np
import pytest

from photon_b200 import abi, native

pytestmark = pytest.mark.gpu
SLACK = 12 << 20  # the counted arrays round up to whole device pages; the context's own growth


@pytest.fixture(scope="module")
def cuda():
    return pytest.importorskip("torch").cuda


def _free(cuda):
    cuda.synchronize()
    return cuda.mem_get_info()[0]


def test_a_path_pool_holds_what_is_counted(cuda):
    native.Server(path_capacity=1 << 20, reserve_bytes=-1).close()  # the context and its modules
    before = _free(cuda)
    s = native.Server(path_capacity=1 << 24, reserve_bytes=-1)
    held, counted = before - _free(cuda), s.stats().device_bytes_in_use
    s.close()
    assert counted > 1 << 30
    assert held <= counted + SLACK


def test_a_scene_holds_what_is_counted(cuda):
    box, g = native.box_scene(), native.terrain_scene(1 << 20, 2)
    small, b = box.build(), g.build(gpu=True)
    s = native.Server(path_capacity=1 << 20, reserve_bytes=-1)
    s.add_scene(small.desc)
    before, counted = _free(cuda), s.stats().device_bytes_in_use
    s.add_scene(b.desc)
    held, counted = before - _free(cuda), s.stats().device_bytes_in_use - counted
    s.close()
    assert counted > 150 << 20
    assert held <= counted + SLACK


def test_a_light_rebuild_keeps_little(cuda):
    """Its scratch is 36 bytes per triangle and 12 per texel, 81 MB here; what stays is at most 32 MiB."""
    g = native.terrain_scene(1 << 21, 2)
    b = g.build(gpu=True)
    raw = g.raw
    u = abi.LightUpdate(raw.materials, raw.num_materials, raw.punctual, raw.num_punctual, raw.env_texels, raw.env_width,
                        raw.env_height, raw.env_color, raw.env_intensity, raw.env_rotation)
    r = native.Renderer()
    r.upload(b.desc)
    before = _free(cuda)
    r.rebuild_lights(u)
    held = before - _free(cuda)
    r.close()
    assert held <= (32 << 20) + SLACK


def test_a_pool_that_cannot_grow_leaves_the_renderer_usable(cuda):
    import torch
    g = native.terrain_scene(65536, 2)
    b = g.build()
    cam = g.camera(16 / 9)
    r = native.Renderer()
    r.upload(b.desc)

    def image(w, h, spp):
        r.resize(w, h)
        r.reset()
        r.render(cam, abi.render_settings(w, h, max_depth=4, seed=2), spp)
        return r.download_accumulation()

    want = image(160, 90, 4)
    r.resize(1280, 720)
    held = torch.empty(max(0, _free(cuda) - (700 << 20)), dtype=torch.uint8, device="cuda")  # room for the samples, not for the paths
    try:
        with pytest.raises(native.PhotonError):
            r.render(cam, abi.render_settings(1280, 720, max_depth=4, seed=2), 16)
        again = image(160, 90, 4)
    finally:
        held = None
        torch.cuda.empty_cache()
        r.close()
    assert np.array_equal(again.view(np.uint32), want.view(np.uint32))


def test_an_upload_that_fails_leaves_no_scene(cuda):
    import torch
    small, big = native.terrain_scene(65536, 2), native.terrain_scene(1 << 21, 2)
    b, c = small.build(), big.build(gpu=True)
    cam, rs = small.camera(16 / 9), abi.render_settings(160, 90, max_depth=4, seed=2)
    r = native.Renderer()
    r.resize(160, 90)
    images = []
    for again in (False, True):
        r.upload(b.desc)
        r.reset()
        r.render(cam, rs, 2)
        images.append(r.download_accumulation())
        if again:
            break
        held = torch.empty(max(0, _free(cuda) - (120 << 20)), dtype=torch.uint8, device="cuda")  # the big scene takes 350 MB
        try:
            with pytest.raises(native.PhotonError):
                r.upload(c.desc)
            with pytest.raises(native.PhotonError) as e:
                r.render(cam, rs, 2)
        finally:
            held = None
            torch.cuda.empty_cache()
        assert e.value.code == abi.PT_ERR_NO_SCENE
    r.close()
    assert np.array_equal(images[0].view(np.uint32), images[1].view(np.uint32))


@pytest.mark.parametrize("kind", ["box", "terrain"])
def test_the_class_order_beside_sorted_shadow_rays(kind):
    """The order of the shading and that of the shadow walk share their memory: an iteration that has both."""
    g = native.box_scene() if kind == "box" else native.terrain_scene(65536, 3)
    b = g.build()
    w, h = 2048, 1026  # above the 2^21 paths from which rays are sorted
    cam, out = g.camera(w / h), []
    for t in (dict(sort_by_material=0, sort_rays=0), dict(sort_shadows=4)):
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        r.set_tuning(**t)
        r.render(cam, abi.render_settings(w, h, max_depth=4, seed=2), 1)
        out.append(r.download_accumulation())
        r.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
