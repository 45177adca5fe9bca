"""The upload's and the refit's checks where the device makes them (scenes of 4096 triangles or more)
refuse what the host's refuse, with the same words, and list the same leaves for node arrays whose
order the device leaves to the host."""
import numpy as np
import pytest

from yune_gb300 import _native as N
from yune_gb300 import scenes, workloads
from yune_gb300.core import Renderer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


def _scene(tris):
    return workloads.mixed_scene(tris, 3, 32, 32, 1, scenes.default_cfg())


def _interior(s):
    return np.flatnonzero(s.nodes["child_idx"] > 0)


def _leaf(s):
    return np.flatnonzero((s.nodes["child_idx"] == -1) & (s.nodes["vert_len"] > 0))


BREAK = {
    "material": lambda s: s.tris["matID"].__setitem__(len(s.tris) // 2, len(s.mats)),
    "negative_material": lambda s: s.tris["matID"].__setitem__(7, -1),
    "vert_len": lambda s: s.nodes["vert_len"].__setitem__(_leaf(s)[5], 11),
    "leaf_triangle": lambda s: s.nodes["vert_list"].__setitem__((_leaf(s)[9], 0), len(s.tris)),
    "child_past_the_end": lambda s: s.nodes["child_idx"].__setitem__(_interior(s)[3], len(s.nodes) - 1),
    "material_and_node": lambda s: (s.tris["matID"].__setitem__(11, 99), s.nodes["vert_len"].__setitem__(_leaf(s)[5], 11)),
}


@pytest.mark.parametrize("tris", [1500, 9000])
@pytest.mark.parametrize("what", sorted(BREAK))
def test_refused_alike(r, what, tris):
    words = []
    for repack in (0, 1):
        s = _scene(tris)
        s.tris, s.nodes = s.tris.copy(), s.nodes.copy()
        BREAK[what](s)
        r.set_repack(repack)
        with pytest.raises(N.YuneError) as e:
            r.upload(s)
        words.append((e.value.code, str(e.value)))
    r.set_repack(1)
    assert words[0] == words[1] and words[0][0] == N.YC_E_INVALID


@pytest.mark.parametrize("tris", [1500, 9000])
def test_children_before_their_parent(r, tris):
    # the later half of the node pairs in reverse order: some children lie before their parent, and
    # the reference's pass in index order does not reach them
    s = _scene(tris)
    n = len(s.nodes)
    pairs = (n - 1) // 2
    order = np.concatenate([np.arange(pairs // 2), np.arange(pairs // 2, pairs)[::-1]])
    to = np.concatenate([[0], 1 + np.repeat(order, 2) * 2 + np.tile([0, 1], pairs)])
    nodes = np.empty_like(s.nodes)
    nodes[to] = s.nodes
    up = nodes["child_idx"] > 0
    nodes["child_idx"][up] = to[nodes["child_idx"][up]]
    s.nodes = nodes
    got = []
    for repack in (0, 1):
        r.set_repack(repack)
        sid = r.upload(s)
        got.append((r.scene_digest(sid), r.scene_depth(sid), r.scene_bytes(sid)))
        r.release(sid)
    r.set_repack(1)
    assert got[0] == got[1]


@pytest.mark.parametrize("tris", [1500, 9000])
def test_refit_refused_and_scene_unchanged(r, tris):
    s = _scene(tris)
    sid = r.upload(s)
    before = r.scene_digest(sid)
    moved = s.tris.copy()
    moved["v1"][:, 0] += np.float32(0.01)
    moved["matID"][len(moved) - 1] = len(s.mats)
    with pytest.raises(N.YuneError) as e:
        r.refit(sid, moved)
    assert e.value.code == N.YC_E_INVALID and "triangle %d has matID out of range" % (len(moved) - 1) in str(e.value)
    assert r.scene_digest(sid) == before
    r.release(sid)
