"""Triangles that are hit ahead of their own leaf box: the walks that do not test a leaf the moment Photon does
must still end on Photon's hit, which may be such a triangle only because Photon reached it before another hit
that lies between the two distances.

Two ways to come by them. A fan of planes through the eye, seen edge-on: their computed distance is rounding, and
one of a few thousand rays accepts one. And boxes that start behind their triangles by nearly as much as an
upload's check allows for rounding, 0.8% of the distance: there every ray does."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from photon_b200 import abi, native, workloads

pytestmark = pytest.mark.gpu
FRONT, PLANES = 2.25, 16384  # the fan
EYE = 8192.0                 # the shifted boxes: floats are 2^-10 apart there, and the check allows 0.0082
SHIFT, BEHIND = 8 / 1024, 2 / 1024  # a front triangle's box starts this far behind it, another triangle this far


def _vec(p):
    return abi.Vec3(*(float(x) for x in p))


def _union(p, q):
    return np.minimum(p[0], q[0]), np.maximum(p[1], q[1])


class Tree:
    """A hand-made scene: triangles, and nodes of two sides (box, index, count)."""

    def __init__(self):
        self.tris, self.boxes, self.nodes = [], [], []

    def triangle(self, *points):
        p = np.array(points, np.float32)
        t = abi.TriGeom()
        t.v0, t.e1, t.e2, t.material, t.flags = _vec(p[0]), _vec(p[1] - p[0]), _vec(p[2] - p[0]), 0, 0
        self.tris.append(t)
        self.boxes.append((p.min(0), p.max(0)))
        return len(self.tris) - 1

    def rectangle(self, x0, y0, x1, y1, z):
        """Two triangles; the first one's number."""
        i = self.triangle((x0, y0, z), (x1, y0, z), (x0, y1, z))
        self.triangle((x1, y1, z), (x0, y1, z), (x1, y0, z))
        return i

    def leaf(self, first, count=1, shift=0.0):
        lo, hi = self.boxes[first]
        for k in range(first + 1, first + count):
            lo, hi = _union((lo, hi), self.boxes[k])
        return (lo + np.float32([0, 0, shift]), hi + np.float32([0, 0, shift])), first, count

    def node(self, left, right=None):
        """A node of two sides, which may be calls that build what lies below (a child follows its parent)."""
        me = len(self.nodes)
        self.nodes.append(None)
        sides = [s() if callable(s) else s for s in (left, right) if s]
        self.nodes[me] = sides + [((np.zeros(3), np.zeros(3)), -1, 0)] * (2 - len(sides))
        return (sides[0][0] if len(sides) == 1 else _union(sides[0][0], sides[1][0])), me, 0

    def scene(self):
        g = native.box_scene()
        b = g.build()
        raw = (abi.BvhNode * len(self.nodes))()
        for n, ((lb, li, lc), (rb, ri, rc)) in zip(raw, self.nodes):
            n.lmin, n.lmax, n.left, n.lcount = _vec(lb[0]), _vec(lb[1]), li, lc
            n.rmin, n.rmax, n.right, n.rcount = _vec(rb[0]), _vec(rb[1]), ri, rc
        arr, idx = (abi.TriGeom * len(self.tris))(*self.tris), np.zeros(3 * len(self.tris), np.int32)
        d = abi.SceneDesc.from_buffer_copy(b.desc)
        d.nodes, d.num_nodes, d.tris, d.num_tris = raw, len(raw), arr, len(arr)
        d.indices = idx.ctypes.data_as(C.POINTER(C.c_int32))
        d.emissive, d.num_emissive, d.tri_emissive, d.emissive_alias = None, 0, None, None
        return d, (g, b, raw, arr, idx)


def _apart(t, build, cover, near):
    """The root's first child holds what build() makes, its box entered first for a triangle at `near` beside the
    view; its second, farther one the triangle(s) `cover`, which lie in front of what the first child's boxes say."""
    beside = t.triangle((5, 5, near), (5.1, 5, near), (5, 5.1, near))
    t.node(lambda: t.node(t.leaf(beside), build), lambda: t.node(t.leaf(*cover)))


def _fan(kind, tilt=0.0, ahead=0.006, spread=0.3):
    """kind "pairs": each plane of the fan is the sibling leaf of a strip in front of it."""
    t, a = Tree(), np.linspace(-spread, spread, PLANES + 1)
    z0, z1, zf = FRONT, 1.15 * FRONT, FRONT * (1 - ahead)
    planes, strips = [], []
    for k in range(PLANES):
        y = np.tan(a[k])
        planes.append(t.triangle((-6, z0 * y, z0), (6, z0 * y, z0), (0, z1 * (y + tilt), z1)))
        if kind == "pairs":
            strips.append(t.triangle((-6, zf * y, zf), (6, zf * y, zf), (0, zf * np.tan(a[k + 1]) + 1e-3, zf)))

    def build(lo, hi):
        if hi - lo == 1:
            return t.node(t.leaf(strips[lo]), t.leaf(planes[lo])) if kind == "pairs" else t.leaf(planes[lo])
        mid = (lo + hi) // 2  # (side 0, first on a tie: the strip that starts at the ray, not those that reach it)
        return t.node(lambda: build(mid, hi), lambda: build(lo, mid))

    if kind == "pairs":
        build(0, PLANES)
    else:
        _apart(t, lambda: build(0, PLANES), (t.triangle((-9, -9, zf), (27, -9, zf), (-9, 27, zf)), 1), 0.5)
    return (*t.scene(), lambda aspect: workloads.look_at((0, 0, 0), (0, 0, 1), 30.0, aspect))


def _shifted(kind, tiles=1500):
    """Uneven tiles across the view, each a rectangle at distance 1 whose leaf's box starts SHIFT behind it. kind
    "pairs": its sibling leaf is a rectangle BEHIND it; nodes behind everything keep the walk's stack filled. "apart":
    one rectangle BEHIND it all, under the root's other child."""
    t, rng, z = Tree(), np.random.default_rng(3), EYE + 1
    rects = [(-0.4, -0.4, 0.4, 0.4)]
    while len(rects) < tiles:
        k = int(rng.integers(len(rects)))
        x0, y0, x1, y1 = rects.pop(k)
        f = rng.uniform(0.3, 0.7)
        if x1 - x0 > y1 - y0:
            rects += [(x0, y0, x0 + f * (x1 - x0), y1), (x0 + f * (x1 - x0), y0, x1, y1)]
        else:
            rects += [(x0, y0, x1, y0 + f * (y1 - y0)), (x0, y0 + f * (y1 - y0), x1, y1)]
    front = [t.rectangle(*r, z) for r in rects]
    back = [t.rectangle(*r, z + BEHIND) for r in rects] if kind == "pairs" else []
    far = t.rectangle(-9, -9, -8.9, 9, z + 3)
    far_box = (np.float32([-9, -9, z + 3]), np.float32([9, 9, z + 4]))

    def build(ids):
        if len(ids) == 1:
            x = t.leaf(front[ids[0]], 2, SHIFT)
            return t.node(t.leaf(back[ids[0]], 2), x) if kind == "pairs" else x
        axis = int(np.ptp([rects[k][1] for k in ids]) > np.ptp([rects[k][0] for k in ids]))
        ids = sorted(ids, key=lambda k: rects[k][axis])
        split = lambda: t.node(lambda: build(ids[:len(ids) // 2]), lambda: build(ids[len(ids) // 2:]))  # noqa: E731
        if kind == "apart":
            return split()
        def behind():
            inner = t.node(t.leaf(far, 2))
            return far_box, inner[1], 0
        return t.node(split, behind)

    if kind == "pairs":
        build(list(range(tiles)))
    else:
        _apart(t, lambda: build(list(range(tiles))), (t.rectangle(-0.5, -0.5, 0.5, 0.5, z + BEHIND), 2), EYE + 0.3)
    return (*t.scene(), lambda aspect: workloads.look_at((0, 0, EYE), (0, 0, EYE + 1), 30.0, aspect))


SCENES = {"fan, pairs": lambda: _fan("pairs"), "fan, apart": lambda: _fan("apart"), "fan, tilted": lambda: _fan("apart", 1e-7),
          "shifted, pairs": lambda: _shifted("pairs"), "shifted, apart": lambda: _shifted("apart")}


def _ahead(name, hits):
    """How many rays end on a triangle ahead of its box."""
    tri = O.hits_tri(hits)
    if "shifted" in name:
        return int(((tri >= 0) & (np.abs(hits[..., 0]) < 1.2) & (tri < 3000)).sum())
    return int(((tri >= 0) & (tri % 2 == 0 if "pairs" in name else tri < PLANES)).sum())


@pytest.mark.parametrize("name", SCENES)
def test_list_walk_ends_on_photons_hit(name):
    desc, keep, camera = SCENES[name]()
    r = native.Renderer()
    r.upload(desc)
    assert r.scene_walks()[0] == 1
    cam = camera(1.28)
    r.set_tuning(pair_walk=0)
    want, ahead = r.trace_primary(cam, 96, 75, 0, 1), 0
    assert np.array_equal(want.view(np.uint32), O.orc_trace_primary(desc, cam, 96, 75, 0, 1).view(np.uint32))
    for seed in range(2 if "shifted" in name else 12):
        r.set_tuning(pair_walk=0)
        want = r.trace_primary(cam, 512, 400, 0, seed)
        ahead += _ahead(name, want)
        for visits in (1, 3, 5):
            r.set_tuning(pair_walk=visits)
            got = r.trace_primary(cam, 512, 400, 0, seed)
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), (seed, visits)
    r.close()
    assert ahead > (300000 if "shifted" in name else 20)


@pytest.mark.parametrize("name", SCENES)
def test_group_tail_ends_on_photons_hit(name):
    desc, keep, camera = SCENES[name]()
    w, h, out = 128, 128, []
    for t in (dict(pair_walk=0, tail_paths=0), dict(tail_paths=1 << 14)):
        r = native.Renderer()
        r.upload(desc)
        assert r.scene_walks() == (1, 1)
        r.resize(w, h)
        r.set_tuning(**t)
        out.append([])
        for seed in range(2 if "shifted" in name else 12):
            r.reset()
            r.render(camera(w / h), abi.render_settings(w, h, max_depth=1, seed=seed), 1)
            out[-1] += [r.download_accumulation(), *r.download_gbuffer()]
        r.close()
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
