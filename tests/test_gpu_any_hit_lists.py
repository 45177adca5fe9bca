"""Any-hit ray lists where their walks change: a stack as deep as the lane-by-lane steps take and one
entry deeper, and the list from which the steps of a large scene are voted."""
from types import SimpleNamespace

import numpy as np
import pytest

from yune_gb300 import scenes, workloads
from yune_gb300.core import Renderer
from yune_gb300.layouts import BVH_NODE, TRIANGLE

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


def _chain(depth):
    """A hierarchy of `depth` levels, each a leaf and the rest: the leaves' triangles face along x, one
    behind the other, so a ray in +x opens the rest first and holds a leaf of every level."""
    n = depth + 1
    x = -0.5 * np.arange(n, dtype=np.float32)
    tris = np.zeros(n, TRIANGLE)
    for v, yz in (("v1", (-1, -1)), ("v2", (1, -1)), ("v3", (0, 1))):
        tris[v][:, 0] = x
        tris[v][:, 1:3] = yz
    tris["v1"][:, 1:3] *= np.linspace(1.0, 0.2, n, dtype=np.float32)[:, None]   # (smaller ones in front)
    for k in ("vn1", "vn2", "vn3"):
        tris[k][:, 0] = 1.0
    nodes = np.zeros(2 * n - 1, BVH_NODE)
    leaf = np.minimum(2 * np.arange(n) + 1, 2 * n - 2)
    nodes["child_idx"] = np.arange(2 * n - 1) + 1
    nodes["vert_len"] = -1
    nodes["child_idx"][leaf] = -1
    nodes["vert_len"][leaf] = 1
    nodes["vert_list"][leaf, 0] = np.arange(n)
    first = np.arange(2 * n - 1) // 2                # the first triangle below a node
    first[leaf] = np.arange(n)
    last = np.full(2 * n - 1, n - 1)
    last[leaf] = np.arange(n)
    nodes["p_min"][:, 0] = x[last] - 0.125
    nodes["p_max"][:, 0] = x[first] + 0.125
    nodes["p_min"][:, 1:3] = -1.0
    nodes["p_max"][:, 1:3] = 1.0
    base = scenes.c0(16, 16)
    return SimpleNamespace(tris=tris, mats=base.mats, lights=base.lights, nodes=nodes)


@pytest.mark.parametrize("depth", [43, 44, 45, 58])   # two entries fewer than the stack's; 44 is the lane steps' last
@pytest.mark.parametrize("n", [33, 5000])
def test_deepest_stacks(r, depth, n):
    s = _chain(depth)
    r.set_tree_mode(0)
    sid = r.upload(s)
    r.set_tree_mode(1)
    assert r.scene_depth(sid) == depth
    rng = np.random.default_rng(depth)
    q = np.zeros((n, 9), np.float32)
    q[:, 0] = -0.5 * (depth + 2)
    q[:, 1:3] = rng.uniform(-1.1, 1.1, (n, 2))
    q[:, 4:7] = np.float32([1.0, 0.0, 0.0]) + rng.normal(0.0, 0.004, (n, 3)).astype(np.float32)
    q[:, 8] = np.where(rng.random(n) < 0.5, np.inf, rng.uniform(0.5, 0.5 * depth, n))
    r.reset_stats()
    hit, _, t = r.trace(sid, q, any_hit=True)
    tri, light, _ = r.trace(sid, q)
    assert r.stats()["stack_overflow"] == 0
    assert np.array_equal(hit == 1, (tri >= 0) | (light >= 0))
    assert (tri >= 0).sum() > n // 10
    r.release(sid)


@pytest.mark.parametrize("n", [(1 << 19) - 1, 1 << 19])
def test_long_lists_of_a_large_scene(r, n):
    s = workloads.mixed_scene(90000, 4, 32, 32, 1)
    sid = r.upload(s)
    q = scenes.box_rays(n, 5)
    q[:, 8] = np.random.default_rng(6).uniform(0.05, 1.5, n).astype(np.float32)
    hit, light, t = r.trace(sid, q, any_hit=True)
    for k in list(range(0, n - 30000, 61001)) + [n - 30000]:
        a, b, c = r.trace(sid, q[k:k + 30000], any_hit=True)
        assert np.array_equal(a, hit[k:k + 30000]) and np.array_equal(b, light[k:k + 30000])
        assert np.array_equal(c.view(np.int32), t[k:k + 30000].view(np.int32))
    r.release(sid)
