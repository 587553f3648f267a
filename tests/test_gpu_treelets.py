"""The treelet order of a scene's nodes (order_by_treelets): hits and images by the walks that follow it equal
Photon's, for trees of one node, of a treelet more or less, at the sizes between which one block and a launch per
level order them, and with nodes that the root does not reach."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu


def _patch(n):
    """n triangles around the middle of a height field, a leaf each: n - 1 nodes (one for n = 1)."""
    g = native.terrain_scene(65536, 2)
    raw = abi.RawScene.from_buffer_copy(g.raw)
    idx = np.ctypeslib.as_array(raw.indices, shape=(raw.num_indices,)).reshape(-1, 3)
    mat = np.ctypeslib.as_array(raw.tri_material, shape=(len(idx),))
    pos = np.ctypeslib.as_array(C.cast(raw.positions, C.POINTER(C.c_float)), shape=(raw.num_positions, 3))
    c = pos[idx].mean(1)
    keep = np.sort(np.argsort((((c - c.mean(0))[:, [0, 2]]) ** 2).sum(1), kind="stable")[:n])
    idx, mat = np.ascontiguousarray(idx[keep]).ravel(), np.ascontiguousarray(mat[keep])
    raw.indices, raw.num_indices = idx.ctypes.data_as(C.POINTER(C.c_int32)), idx.size
    raw.tri_material = mat.ctypes.data_as(C.POINTER(C.c_int32))
    return native.BuiltScene(raw, keepalive=(g, idx, mat), max_leaf=1)


def _check(desc, walks):
    w, h = 96, 64
    center, extent = workloads.scene_sphere(desc)
    cam, out = workloads.look_at(np.asarray(center) + 0.8 * extent * np.array([0.3, 1.0, 0.2]), center, 60.0, w / h), []
    for t in (dict(pair_walk=0, tail_paths=0), dict(tail_paths=1 << 14), dict(tail_paths=0)):
        r = native.Renderer()
        r.upload(desc)
        assert r.scene_walks() == walks
        r.resize(w, h)
        r.set_tuning(**t)
        r.render(cam, abi.render_settings(w, h, max_depth=6, seed=3), 1)
        out.append(r.download_accumulation())
        hits = r.trace_primary(cam, w, h, 0, 3)
        r.close()
    want = O.orc_trace_primary(desc, cam, w, h, 0, 3)
    assert (O.hits_tri(want) >= 0).any()
    assert np.array_equal(hits.view(np.uint32), want.view(np.uint32))
    for img in out[1:]:
        assert np.array_equal(img.view(np.uint32), out[0].view(np.uint32))


@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 10, 17, 100, 512, 513, 514, 520, 1500, 5000])
def test_hits_and_images_are_photons(n):
    b = _patch(n)
    assert b.desc.num_nodes == max(1, n - 1)
    _check(b.desc, (1, 1))


@pytest.mark.parametrize("n", [40, 3000])
def test_nodes_that_the_root_does_not_reach(n):
    b = _patch(n)
    nodes = (abi.BvhNode * b.desc.num_nodes)()
    C.memmove(nodes, b.desc.nodes, C.sizeof(nodes))
    nodes[0].left, nodes[0].lcount = -1, 0
    d = abi.SceneDesc.from_buffer_copy(b.desc)
    d.nodes = nodes
    _check(d, (1, 1))


def test_new_lights_keep_the_order():
    b = _patch(3000)
    w, h = 96, 64
    center, extent = workloads.scene_sphere(b.desc)
    cam = workloads.look_at(np.asarray(center) + 0.8 * extent * np.array([0.3, 1.0, 0.2]), center, 60.0, w / h)
    out = []
    for again in (False, True):
        r = native.Renderer()
        r.upload(b.desc)
        if again:
            r.update_lights(b.desc)
        assert r.scene_walks() == (1, 1)
        r.resize(w, h)
        r.render(cam, abi.render_settings(w, h, max_depth=6, seed=3), 2)
        out.append(r.download_accumulation())
        r.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
