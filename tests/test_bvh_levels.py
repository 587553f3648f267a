"""What an upload makes of a BVH whose nodes are named twice: validation lets such a graph through, so the
depth and the node counts that the list walk and the group tail rely on must not be taken from it."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from photon_b200 import abi, native


def _graph(children):
    """A BVH of inner nodes whose children are the given (left, right) indices; -1: none."""
    nodes = (abi.BvhNode * len(children))()
    for n, (left, right) in zip(nodes, children):
        n.left, n.right, n.lcount, n.rcount = left, right, 0, 0
    return native.lib.pt_bvh_levels(nodes, len(children))


def _spine(n):
    return [(i + 1, -1) for i in range(n - 1)] + [(-1, -1)]


@pytest.mark.parametrize("children,levels", [
    ([(-1, -1)], 1),
    ([(1, 2), (-1, -1), (-1, -1)], 2),
    (_spine(60), 60),
    (_spine(61), 61),
    (_spine(400), 255),
    ([(i + 1, i + 1) for i in range(15)] + [(-1, -1)], 0),               # every node names its successor twice
    ([(1, 2), (3, -1), (3, -1), (-1, -1)], 0),                          # two nodes share a child
    ([(1, 99)] + [(i + 1, -1) for i in range(1, 99)] + [(-1, -1)], 0),  # the last of 99 levels is also the root's child
    ([(-1, -1), (2, -1), (-1, -1)], 2),                                 # nodes that the root does not reach
    ([(1, -1), (1, -1)], -1),
    ([(2, -1), (-1, -1)], -1),
])
def test_levels(children, levels):
    assert _graph(children) == levels


def test_a_built_tree_has_levels():
    b = native.terrain_scene(65536, 2).build()
    assert 10 < native.lib.pt_bvh_levels(b.desc.nodes, b.desc.num_nodes) <= 60


@pytest.mark.gpu
def test_a_shared_subtree_is_walked_in_photons_order():
    """The root names its left child twice: its hits tie with themselves, and the collapse and the depth that
    the other walks need would not hold."""
    g = native.terrain_scene(65536, 2)
    b = g.build()
    nodes = (abi.BvhNode * b.desc.num_nodes)()
    C.memmove(nodes, b.desc.nodes, C.sizeof(nodes))
    n = nodes[0]
    n.rmin, n.rmax, n.right, n.rcount = n.lmin, n.lmax, n.left, n.lcount
    desc = abi.SceneDesc.from_buffer_copy(b.desc)
    desc.nodes = nodes
    w, h = 96, 64
    cam, out = g.camera(w / h), []
    for t in (dict(pair_walk=0, tail_paths=0), dict()):
        r = native.Renderer()
        r.upload(desc)
        assert r.scene_walks() == (0, 0)
        r.resize(w, h)
        r.set_tuning(**t)
        r.render(cam, abi.render_settings(w, h, max_depth=8, seed=3), 2)
        out.append(r.download_accumulation())
        hits = r.trace_primary(cam, w, h, 0, 3)
        r.close()
    assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
    want = O.orc_trace_primary(desc, cam, w, h, 0, 3)
    assert np.array_equal(hits.view(np.uint32), want.view(np.uint32))
    r = native.Renderer()
    r.upload(b.desc)
    assert r.scene_walks() == (1, 1)
    r.close()
