"""The shading step's shared stages (one copy of the lobe choice, the sampling, the BRDF and
the light loop serves every ray a path sends) against the oracle, bit for bit, where a
path goes through them more than once in a step: lights that close other lights' shadow
rays, MIS rays that miss their light, absorbed lobes, paths cut at their first bounces;
and lights replaced after the upload, whose device copy carries values computed from
them."""
import numpy as np
import pytest

from oracle import oracle_py as O
from yune_gb300 import _native as N
from yune_gb300 import scenes, workloads
from yune_gb300.core import Renderer
from yune_gb300.layouts import ptr

pytestmark = pytest.mark.gpu
W, H = 44, 30


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


def _crossing_lights(lights):
    """Three quads under each other: the lower ones close most shadow rays to the upper ones."""
    out = np.repeat(lights[:1], 3)
    for i in range(3):
        out[i]["pos"][1] -= 0.12 * i
        out[i]["edge_l"] = out[i]["edge_l"] * np.float32(1.0 + 0.7 * i)
        out[i]["ke"][:3] = (3.0 + i, 2.0, 5.0 - i)
    return out


def _same(r, s, sid, passes=2, gi=1):
    seeds = scenes.pass_seeds(77, passes)
    aid = r.alloc_accum(W, H)
    r.set_camera(s.cam)
    r.render_passes(sid, aid, seeds, reset_first=1, gi_check=gi, cfg=s.cfg)
    got = r.read_accum(aid)
    r.free_accum(aid)
    ref = np.zeros((H, W, 4), np.float32)
    for k, sd in enumerate(seeds):
        reset = 1 if k == 0 else 0
        if s.cfg["integrator"] == 0:
            O.render(s, ref, sd, reset, dict(s.cfg, gi_check=gi))
        elif s.cfg["integrator"] == 1:
            O.render_bdpt(s, ref, sd, reset, s.cfg["bdpt_bounces"])
        else:
            O.render_bdpt_mis(s, ref, sd, reset, s.cfg["bdpt_bounces"], s.cfg)
    assert np.array_equal(got.view(np.int32), ref.view(np.int32))


@pytest.mark.parametrize("gi", [0, 1])
@pytest.mark.parametrize("lobe_fix", [0, 1])
@pytest.mark.parametrize("mis", [0, 1])
@pytest.mark.parametrize("max_depth", [0, 1, 16])
def test_shared_stages(r, mis, lobe_fix, max_depth, gi):
    s = workloads.mixed_scene(3000, 11, W, H, 1, scenes.default_cfg(mis=mis, mis_lobe_fix=lobe_fix, max_depth=max_depth))
    s.lights = _crossing_lights(s.lights)
    sid = r.upload(s)
    _same(r, s, sid, gi=gi)
    r.release(sid)


@pytest.mark.parametrize("integrator", [0, 1, 2])
def test_lights_replaced_after_the_upload(r, integrator):
    s = scenes.c0(W, H)
    s.cfg = dict(s.cfg, integrator=integrator, bdpt_bounces=6, mis=1 if integrator == 0 else 0)
    sid = r.upload(s)
    s.lights = _crossing_lights(s.lights)
    N.check(r.L.yc_set_lights(r.h, sid, ptr(s.lights), len(s.lights)), "yc_set_lights")
    _same(r, s, sid)
    r.release(sid)


# An eye vertex's segments go out in rounds of eight at most: light subpaths that need one
# round, two and three; in the shared launch, its sorted form, and the launch of their own, and
# in the tail.
@pytest.mark.parametrize("mixed, sort", [(1, 0), (1, 1), (0, 0)])
@pytest.mark.parametrize("bounces", [3, 9, 20])
@pytest.mark.parametrize("integrator", [1, 2])
@pytest.mark.parametrize("tris", [0, 6000])
@pytest.mark.parametrize("tail", [0, -1])
def test_segments_of_an_eye_vertex(r, tail, tris, integrator, bounces, mixed, sort):
    if sort and not tris:
        pytest.skip("rays are sorted in scenes of at least 4096 triangles")
    s = workloads.mixed_scene(tris, 5, W, H, 1, scenes.default_cfg()) if tris else scenes.c0_bdpt_mis(W, H, lights=4)
    s.cfg = dict(s.cfg, integrator=integrator, bdpt_bounces=bounces, mis=0)
    sid = r.upload(s)
    opts = [(2, tail, -1), (3, mixed, 1), (5, 1 if sort else 65536, 65536), (6, 1 if sort else 65536, 65536)]
    for o, v, _ in opts:
        N.check(r.L.yc_set_option(r.h, o, v), "yc_set_option")
    _same(r, s, sid)
    for o, _, v in opts:
        N.check(r.L.yc_set_option(r.h, o, v), "yc_set_option")
    r.release(sid)


# A shadow ray goes with the path's next ray where the lobe is drawn whatever its result
# (mis_lobe_fix): round by round and in the tail, whose idle lanes walk a path's second ray;
# in the shared launch, its sorted form, and launches of their own.
@pytest.mark.parametrize("tail", [0, -1])
@pytest.mark.parametrize("mixed, sort", [(1, 0), (1, 1), (0, 0)])
@pytest.mark.parametrize("lobe_fix", [0, 1])
@pytest.mark.parametrize("tris, max_depth", [(0, 100000), (6000, 2), (6000, 100000)])
def test_rays_sent_together(r, tris, max_depth, lobe_fix, mixed, sort, tail):
    cfg = scenes.default_cfg(mis=1, mis_lobe_fix=lobe_fix, max_depth=max_depth)
    s = workloads.mixed_scene(tris, 9, W, H, 1, cfg) if tris else scenes.c0(W, H)
    s.cfg = dict(s.cfg, mis_lobe_fix=lobe_fix)
    if tris:
        s.lights = _crossing_lights(s.lights)
    sid = r.upload(s)
    opts = [(2, tail, -1), (3, mixed, 1), (5, 1 if sort else 65536, 65536)]
    for o, v, _ in opts:
        N.check(r.L.yc_set_option(r.h, o, v), "yc_set_option")
    _same(r, s, sid)
    for o, _, v in opts:
        N.check(r.L.yc_set_option(r.h, o, v), "yc_set_option")
    r.release(sid)


@pytest.mark.parametrize("tail", [0, -1])
@pytest.mark.parametrize("lobe_fix, reset", [(0, 1), (1, 1), (1, 0)])
@pytest.mark.parametrize("tris, passes", [(0, 3), (6000, 5)])
def test_passes_of_one_call_equal_a_call_each(r, tris, passes, lobe_fix, reset, tail):
    s = workloads.mixed_scene(tris, 13, W, H, 1, scenes.default_cfg()) if tris else scenes.c0(W, H)
    s.cfg = dict(s.cfg, mis_lobe_fix=lobe_fix)
    sid, seeds = r.upload(s), scenes.pass_seeds(5, passes)
    r.set_camera(s.cam)
    N.check(r.L.yc_set_option(r.h, 2, tail), "yc_set_option")
    got = []
    for step in (passes, 1):
        aid = r.alloc_accum(W, H)
        r.render_passes(sid, aid, seeds[:1], reset_first=1, gi_check=1, cfg=s.cfg)   # something to go on from
        for k in range(0, passes, step):
            r.render_passes(sid, aid, seeds[k:k + step], reset_first=reset if k == 0 else 0, gi_check=1, cfg=s.cfg)
        got.append(r.read_accum(aid))
        r.free_accum(aid)
    N.check(r.L.yc_set_option(r.h, 2, -1), "yc_set_option")
    assert np.array_equal(got[0].view(np.int32), got[1].view(np.int32))
    r.release(sid)
