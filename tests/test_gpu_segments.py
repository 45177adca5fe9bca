"""Bidirectional passes that send fewer segments of an eye vertex a round, as they do where memory is
short (YC_OPT_SEGMENTS): the same bits, through the rounds and through the tail kernel."""
import numpy as np
import pytest

from yune_gb300 import scenes, workloads
from yune_gb300.core import Renderer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


@pytest.mark.parametrize("integrator", [1, 2])
@pytest.mark.parametrize("tris, size", [(0, (65, 33)), (6000, (320, 256))])   # the second: rays and shading sorted
@pytest.mark.parametrize("tail", [0, -1])
@pytest.mark.parametrize("mixed", [1, 0])
def test_images_at_every_number_of_segments(r, integrator, tris, size, tail, mixed):
    s = workloads.mixed_scene(tris, 6, *size, 1) if tris else scenes.c0_bdpt(*size)
    cfg = scenes.default_cfg(integrator=integrator, mis=0, bdpt_bounces=7)
    sid, aid = r.upload(s), r.alloc_accum(*size)
    r.set_camera(s.cam)
    r.set_tail_paths(tail)
    r.set_mixed_trace(mixed)
    got, rays = [], []
    for k in (8, 4, 2, 1):
        r.set_segments(k)
        r.reset_stats()
        r.render_passes(sid, aid, [11, 12], reset_first=1, cfg=cfg)
        got.append(r.read_accum(aid).view(np.int32))
        st = r.stats()
        rays.append((st["rays"], st["samples"], st["stack_overflow"]))
    r.set_segments(8)
    r.set_tail_paths(-1)
    r.set_mixed_trace(1)
    r.free_accum(aid)
    r.release(sid)
    for g, n in zip(got[1:], rays[1:]):
        assert np.array_equal(g, got[0]) and n == rays[0]
