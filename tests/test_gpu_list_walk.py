"""The list walk (walk_queue_list: the default walk of order-free trees) against the per-lane walk in
Photon's order and the oracle's restatement: the same hits and images bit for bit, on built scenes, where
hits tie exactly (coincident triangles, which the walk must hand to the exact walk), and on trees that are
not order-free (which keep the walks in Photon's order)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from photon_b200 import abi, native, workloads
from test_deep_stack import _deep_scene

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _render(desc, cam, w, h, spp, depth, **tuning):
    r = native.Renderer()
    r.upload(desc)
    r.resize(w, h)
    r.set_tuning(**tuning)
    r.render(cam, abi.render_settings(w, h, max_depth=depth, seed=3), spp)
    img = r.download_accumulation()
    r.close()
    return img


@pytest.mark.parametrize("triangles", [36, 65536, 262144])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 1), (97, 61), (320, 180)])
def test_images_and_primary_hits_equal_the_walk_in_photons_order(triangles, w, h):
    g = native.box_scene() if triangles == 36 else native.terrain_scene(triangles, 2)
    b = g.build()
    cam = g.camera(w / h)
    ref = _render(b.desc, cam, w, h, 3, 8, pair_walk=0, tail_paths=0)
    for t in (dict(pair_walk=5), dict(pair_walk=1, trace_refill=32, shadow_refill=1), dict(pair_walk=64, trace_block=256)):
        assert np.array_equal(_bits(_render(b.desc, cam, w, h, 3, 8, tail_paths=0, **t)), _bits(ref)), t
    r = native.Renderer()
    r.upload(b.desc)
    assert np.array_equal(_bits(r.trace_primary(cam, w, h, 0, 5)), _bits(O.orc_trace_primary(b.desc, cam, w, h, 0, 5)))
    r.close()


def test_exact_ties_take_photons_triangle():
    """Every triangle of the scene three times over: each hit ties three ways, and Photon's order decides."""
    g = native.terrain_scene(65536, 4)
    raw = abi.RawScene.from_buffer_copy(g.raw)
    n = raw.num_indices
    idx = np.ctypeslib.as_array(raw.indices, shape=(n,))
    mat = np.ctypeslib.as_array(raw.tri_material, shape=(n // 3,))
    idx3, mat3 = np.ascontiguousarray(np.tile(idx, 3), np.int32), np.ascontiguousarray(np.tile(mat, 3), np.int32)
    raw.indices, raw.num_indices = idx3.ctypes.data_as(C.POINTER(C.c_int32)), 3 * n
    raw.tri_material = mat3.ctypes.data_as(C.POINTER(C.c_int32))
    b = native.BuiltScene(raw, keepalive=(g, idx3, mat3))
    w, h = 160, 90
    cam = g.camera(w / h)
    r = native.Renderer()
    r.upload(b.desc)
    got, want = r.trace_primary(cam, w, h, 0, 1), O.orc_trace_primary(b.desc, cam, w, h, 0, 1)
    r.close()
    assert (O.hits_tri(want) >= 0).any()
    assert np.array_equal(_bits(got), _bits(want))


def _unnested(desc):
    """The scene's tree with one inner child's box shrunk to half, so that boxes below stick out of it."""
    nodes = (abi.BvhNode * desc.num_nodes)()
    C.memmove(nodes, desc.nodes, C.sizeof(abi.BvhNode) * desc.num_nodes)
    n = nodes[0]
    n.lmax = abi.Vec3(0.5 * (n.lmin.x + n.lmax.x), n.lmax.y, n.lmax.z)
    d = abi.SceneDesc.from_buffer_copy(desc)
    d.nodes = nodes
    return d, nodes


@pytest.mark.parametrize("kind", ["unnested", "deep"])
def test_trees_that_are_not_order_free_keep_photons_order(kind):
    w, h = 64, 48
    if kind == "deep":
        desc, keep = _deep_scene()
        cam = workloads.look_at((0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 20.0, w / h)
    else:
        g = native.terrain_scene(65536, 2)
        b = g.build()
        desc, keep = _unnested(b.desc)
        cam = g.camera(w / h)
    r = native.Renderer()
    r.upload(desc)
    got = r.trace_primary(cam, w, h, 0, 3)
    r.close()
    assert np.array_equal(_bits(got), _bits(O.orc_trace_primary(desc, cam, w, h, 0, 3)))
    assert np.array_equal(_bits(_render(desc, cam, w, h, 2, 6, pair_walk=5)), _bits(_render(desc, cam, w, h, 2, 6, pair_walk=0)))
