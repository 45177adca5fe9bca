"""A refit of a scene without triangles, or whose leaves the reference never reaches, has no stream
records to rewrite: the stream's array, which is never empty, is left alone."""
import types

import numpy as np
import pytest

import fake_cuda
from yune_gb300 import _native as N
from yune_gb300 import scenes
from yune_gb300.core import Renderer


def _without_triangles():
    s = scenes.c0(32, 24)
    return types.SimpleNamespace(tris=s.tris[:0], mats=s.mats, lights=s.lights, nodes=s.nodes[:0], cam=s.cam, cfg=s.cfg)


def _without_leaves():
    """Two children that the reference does not queue: no triangle and no child of their own."""
    s = scenes.c0(32, 24)
    nodes = s.nodes[:3].copy()
    nodes["child_idx"], nodes["vert_len"] = [1, -1, -1], [-1, 0, 0]
    return types.SimpleNamespace(tris=s.tris, mats=s.mats, lights=s.lights, nodes=nodes, cam=s.cam, cfg=s.cfg)


@pytest.mark.parametrize("make, launches", [(_without_triangles, 0), (_without_leaves, 1)])   # 1: the shading records
def test_launches_of_an_empty_refit(tmp_path, monkeypatch, make, launches):
    fake = fake_cuda.load(tmp_path)
    monkeypatch.setattr(N, "_lib", fake)
    s = make()
    with Renderer(0) as r:
        r.set_repack(0)
        sid = r.upload(s)
        before = fake.fake_launches()
        r.refit(sid, np.ascontiguousarray(s.tris))
        assert fake.fake_launches() - before == launches


@pytest.mark.gpu
@pytest.mark.parametrize("make", [_without_triangles, _without_leaves])
def test_empty_refit_leaves_the_image(make):
    s = make()
    with Renderer(0) as r:
        sid, aid = r.upload(s), r.alloc_accum(32, 24)
        r.set_camera(s.cam)
        got = []
        for _ in range(2):
            r.render_passes(sid, aid, [3, 4], reset_first=1, cfg=s.cfg)
            got.append(r.read_accum(aid))
            r.refit(sid, np.ascontiguousarray(s.tris))
        assert np.array_equal(got[0].view(np.int32), got[1].view(np.int32))
