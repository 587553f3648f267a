"""Environment tables rebuilt on the device (pt_rebuild_lights) against the host builder's, at the sizes
where the device's tiles and its interval for the mean luminance can go wrong: one texel, rows and columns
past one tile, black and negative texels, and a mean that lies halfway between two floats (which the device
must take in the host's order). Equal tables give renders equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

from photon_b200 import abi, native

pytestmark = pytest.mark.gpu


def _halfway():
    """Two grey texels whose luminances are neighbouring floats: their mean lies halfway between them."""
    lum = lambda v: np.float32(np.float32(np.float32(np.float32(0.2126) * v) + np.float32(np.float32(0.7152) * v)) + np.float32(np.float32(0.0722) * v))  # noqa: E731
    v = np.float32(1.3)
    while True:
        w = np.nextafter(v, np.float32(2))
        if lum(w) == np.nextafter(lum(v), np.float32(2)):
            return np.array([[[v] * 3, [w] * 3]], np.float32)
        v = w


def _env(kind):
    rng = np.random.default_rng(11)
    if kind == "halfway":
        return _halfway()
    w, h = dict(one=(1, 1), wide=(1025, 3), tall=(3, 1025), black=(16, 8), negative=(64, 32), large=(1024, 512))[kind]
    env = rng.exponential(1.0, (h, w, 3)).astype(np.float32)
    if kind == "black":
        env[:] = 0
    if kind == "negative":
        env[::5] -= 0.4
    return env


@pytest.mark.parametrize("kind", ["one", "wide", "tall", "black", "negative", "large", "halfway"])
def test_environment_tables_equal_the_host_builders(kind):
    g = native.terrain_scene(65536, 2)
    before = g.build()
    env = np.ascontiguousarray(_env(kind))
    raw = abi.RawScene.from_buffer_copy(g.raw)
    raw.env_texels, raw.env_height, raw.env_width = env.ctypes.data_as(C.POINTER(abi.Vec3)), env.shape[0], env.shape[1]
    after = native.BuiltScene(raw, keepalive=(g, env))
    d = after.desc
    u = abi.LightUpdate(d.materials, d.num_materials, d.punctual, d.num_punctual, d.env_texels, d.env_width, d.env_height, d.env_color,
                        d.env_intensity, d.env_rotation)
    w, h = 96, 54
    cam, rs = g.camera(w / h), abi.render_settings(w, h, max_depth=4, seed=9)
    out = []
    for rebuild in (True, False):
        r = native.Renderer()
        r.upload(before.desc if rebuild else after.desc)
        r.resize(w, h)
        if rebuild:
            r.rebuild_lights(u)
            r.rebuild_lights(u)  # again, in the scratch that the first call left
        r.render(cam, rs, 4)
        out.append((r.download_accumulation().view(np.uint32), r.light_picks(cam, rs)))
        r.close()
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0])
