"""A BVH whose interior child is numbered not above its parent, on small trees of the scene's triangles: the persistent lanes count
it as corruptTree where the plain descent does (the child met first, the one that waits, the one behind a leaf), neither where the
ray does not come to it, and the hits are the same."""
import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer, VtError

pytestmark = pytest.mark.gpu

NODE1, BACK, SELF1 = ("node", 1), ("node", 0), ("node", 1)
# children as (where on the ray, what): triangle a is hit first, b behind it, miss beside the ray
LEAVES = (("a", ("leaf", "a")), ("b", ("leaf", "b")))
TREES = {   # nodes, whether it is counted, the triangle hit
    "sound": ([(("a", NODE1), ("after", ("leaf", "b"))), LEAVES], 0, "a"),
    "met first": ([(("a", BACK), ("b", NODE1)), LEAVES], 1, None),
    "waits for the other": ([(("a", NODE1), ("b", BACK)), LEAVES], 1, None),
    "waits, in the first place": ([(("b", BACK), ("a", NODE1)), LEAVES], 1, None),
    "alone": ([(("beside", NODE1), ("b", BACK)), LEAVES], 1, None),
    "behind a leaf that is missed": ([(("a", ("leaf", "miss")), ("b", BACK)), LEAVES], 1, None),
    "before a leaf": ([(("a", BACK), ("b", ("leaf", "b"))), LEAVES], 1, "b"),
    "hidden by a leaf": ([(("a", ("leaf", "a")), ("b", BACK)), LEAVES], 0, "a"),
    "beside the ray": ([(("a", ("leaf", "a")), ("beside", BACK)), LEAVES], 0, "a"),
    "below the root, hidden": ([(("a", NODE1), ("after", ("leaf", "b"))), (("b", SELF1), ("a", ("leaf", "a")))], 0, "a"),
    "below the root": ([(("a", NODE1), ("after", ("leaf", "b"))), (("a", SELF1), ("b", ("leaf", "b")))], 1, "b"),
}


@pytest.fixture(scope="module")
def renderer():
    r = TwinRenderer.create(dome.make_dome_scene(seed=1, width=8, height=8, level=2), nodes=False)
    yield r
    r.destroy()


@pytest.fixture(scope="module")
def ray(renderer):
    """A ray through the dome from outside, the triangles it meets first and last, one that it misses."""
    o, d = np.array([0.31, -50.0, 1.27]), np.array([0.0, 1.0, 0.0])
    T = np.asarray(renderer.export()["tris"]).view(np.float32).reshape(-1, 4, 4)[: len(renderer.scene["static"]["I"])].astype(np.float64)
    v0, e1, e2 = T[:, 0, :3], T[:, 1, :3], T[:, 2, :3]
    p = np.cross(d, e2)
    det = (e1 * p).sum(1)
    ok = np.abs(det) > 1e-12
    inv = 1.0 / np.where(ok, det, 1.0)
    s = o - v0
    u = (s * p).sum(1) * inv
    q = np.cross(s, e1)
    v, t = (q @ d) * inv, (e2 * q).sum(1) * inv
    inside = np.minimum(np.minimum(u, v), 1 - u - v)
    hits = np.flatnonzero(ok & (inside > 1e-3) & (t > 0))
    a, b = hits[np.argmin(t[hits])], hits[np.argmax(t[hits])]
    assert t[b] - t[a] > 2.0
    return o, d, {"a": int(a), "b": int(b), "miss": int(np.argmin(inside))}, t


def _child(ray, where, what):
    o, _, tris, t = ray
    w = np.zeros(8, np.float32)
    y = o[1] + {"a": t[tris["a"]], "b": t[tris["b"]], "beside": t[tris["a"]], "after": t[tris["b"]] + 5.0}[where]
    x = o[0] + (9.0 if where == "beside" else 0.0)
    w[:3], w[4:7] = (x - 1, y - 0.5, o[2] - 1), (x + 1, y + 0.5, o[2] + 1)
    w.view(np.uint32)[3], w.view(np.uint32)[7] = (what[1], 0) if what[0] == "node" else (tris[what[1]], 1)
    return w


@pytest.mark.parametrize("name", list(TREES))
def test_back_reference(renderer, ray, name):
    nodes, counted, hit = TREES[name]
    o, d, tris, t = ray
    tin = np.stack([np.concatenate([_child(ray, *c) for c in n]) for n in nodes]).reshape(-1, 4)
    out = renderer.unit_test(A.VT_UNIT_TREE, tin, lens=[*o, *d])
    lanes, plain = out[0], out[1]
    assert plain[2] == counted and plain[3] == 0
    assert np.array_equal(lanes.view(np.uint32), plain.view(np.uint32))
    got = int(plain.view(np.uint32)[1])
    if hit:
        assert got == tris[hit] and abs(plain[0] - t[tris[hit]]) <= 1e-4
    else:
        assert got == 0xffffffff


def test_out_of_range_is_refused(renderer, ray):
    o, d, tris, _ = ray
    good = np.concatenate([_child(ray, "a", NODE1), _child(ray, "b", ("leaf", "b"))] * 2)
    for word, value in ((3, 2), (11, 1 << 30), (7, 1 << 31)):
        tin = good.copy()
        tin.view(np.uint32)[word] = value
        if word == 7:
            tin.view(np.uint32)[3] = 0xfffffff0
        with pytest.raises(VtError):
            renderer.unit_test(A.VT_UNIT_TREE, tin, lens=[*o, *d])
    with pytest.raises(VtError):   # one node alone has no room for the two answers
        renderer.unit_test(A.VT_UNIT_TREE, good[:16], lens=[*o, *d])
