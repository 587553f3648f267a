"""The tail by groups of eight lanes (k_tail_group, group_walk) against the queued kernels: the same image
bit for bit for one path up to the most it takes, with groups and warps left over, at full depth, where hits
tie exactly, and where rays fill the group's stack (a pile of parallel triangles, eight siblings entered at
every level)."""
import ctypes as C

import numpy as np
import pytest

from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu


def _raw(g, positions, indices):
    """The generated scene's materials and lights around other triangles (white, material 0)."""
    raw = abi.RawScene.from_buffer_copy(g.raw)
    n = positions.shape[0]
    normals = np.zeros((n, 3), np.float32)
    normals[:, 2] = -1
    uvs, mat = np.zeros((n, 2), np.float32), np.zeros(indices.size // 3, np.int32)
    keep = (g, positions, indices, normals, uvs, mat)
    raw.positions, raw.num_positions = positions.ctypes.data_as(C.POINTER(abi.Vec3)), n
    raw.normals, raw.uvs = normals.ctypes.data_as(C.POINTER(abi.Vec3)), uvs.ctypes.data_as(C.POINTER(abi.Vec2))
    raw.tangents = None
    raw.indices, raw.num_indices = indices.ctypes.data_as(C.POINTER(C.c_int32)), indices.size
    raw.tri_material = mat.ctypes.data_as(C.POINTER(C.c_int32))
    return raw, keep


def _scene(kind):
    if kind == "box":
        g = native.box_scene()
        return g.build(), g.camera
    g = native.terrain_scene(65536, 2)
    if kind == "terrain":
        return g.build(), g.camera
    if kind == "ties":
        raw = abi.RawScene.from_buffer_copy(g.raw)
        n = raw.num_indices
        idx = np.tile(np.ctypeslib.as_array(raw.indices, shape=(n,)), 2).astype(np.int32)
        mat = np.tile(np.ctypeslib.as_array(raw.tri_material, shape=(n // 3,)), 2).astype(np.int32)
        raw.indices, raw.num_indices = idx.ctypes.data_as(C.POINTER(C.c_int32)), 2 * n
        raw.tri_material = mat.ctypes.data_as(C.POINTER(C.c_int32))
        return native.BuiltScene(raw, keepalive=(g, idx, mat)), g.camera
    count = 120000  # pile: triangles that cover the view, one behind the other
    z = np.linspace(1.0, 2.0, count, dtype=np.float32)
    tri = np.array([[-9, -9], [27, -9], [-9, 27]], np.float32)
    pos = np.zeros((count, 3, 3), np.float32)
    pos[:, :, :2], pos[:, :, 2] = tri, z[:, None]
    raw, keep = _raw(g, np.ascontiguousarray(pos.reshape(-1, 3)), np.arange(3 * count, dtype=np.int32))
    return native.BuiltScene(raw, keepalive=keep), lambda aspect: workloads.look_at((0, 0, 0), (0, 0, 1), 40.0, aspect)


@pytest.mark.parametrize("kind", ["box", "terrain", "ties", "pile"])
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (3, 3, 1), (31, 1, 1), (129, 127, 1), (64, 64, 4)])
def test_group_tail_equals_the_queued_kernels(kind, w, h, spp):
    b, camera = _scene(kind)
    cam = camera(w / h)
    out = []
    for tail in (0, 1 << 14):
        r = native.Renderer()
        r.upload(b.desc)
        r.resize(w, h)
        r.set_tuning(tail_paths=tail)
        r.render(cam, abi.render_settings(w, h, max_depth=16, rr_depth=8, seed=3), spp)
        out.append((r.download_accumulation(), *r.download_gbuffer()))
        st = r.stats()
        out[-1] += (np.array([st.rays, st.shadow_rays], np.int64),)
        r.close()
    for x, y in zip(*out):
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint32), np.ascontiguousarray(y).view(np.uint32))
