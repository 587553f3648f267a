"""The two-steps-at-a-time search of the environment's tables picks the oracle's texel: tables of 1 to 9
entries (where the last steps are taken one by one), around powers of two, and with black texels, whose
entries are equal."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from photon_b200 import abi, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(n, 10 - n) for n in range(1, 10)] + [(15, 17), (31, 33), (64, 3), (257, 65)])
def test_picks_equal_the_oracles(w, h):
    rng = np.random.default_rng(w * 1000 + h)
    env = rng.exponential(1.0, (h, w, 3)).astype(np.float32)
    env[rng.random((h, w)) < 0.3] = 0
    env[0, 0] = 1
    g = native.terrain_scene(65536, 2)
    raw = abi.RawScene.from_buffer_copy(g.raw)
    raw.env_texels, raw.env_height, raw.env_width = env.ctypes.data_as(C.POINTER(abi.Vec3)), h, w
    b = native.BuiltScene(raw, keepalive=(g, env))
    cam, rs = g.camera(160 / 90), abi.render_settings(160, 90, max_depth=4, seed=9)
    r = native.Renderer()
    r.upload(b.desc)
    got = r.light_picks(cam, rs)
    r.close()
    want = O.orc_light_picks(b.desc, cam, rs, 0)
    cells = got.reshape(-1, 4)
    assert len(np.unique(cells[cells[:, 3] == 1][:, 1])) > min(5, w * h // 4)
    assert np.array_equal(got, want)
