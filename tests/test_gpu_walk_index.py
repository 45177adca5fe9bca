"""The four-child walk index over a scene's two-child nodes (tree mode 1): walks over it give
the hits of the reference node tree (tree mode 0) and of the oracle, at the sizes where its
nodes are partly filled, and the renders that do not use it (a stack limit, a scene without an
index in the batch) give the same bits."""
import numpy as np
import pytest

import leafgen
from oracle import oracle_py as O
from yune_gb300 import scenes, workloads
from yune_gb300.batch import Batch
from yune_gb300.core import Renderer

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(0) as rr:
        yield rr


def _rays(n, lo, hi, seed):
    rng = np.random.default_rng(seed)
    rays = np.zeros((n, 9), np.float32)
    rays[:, :3] = rng.uniform(lo - 1.0, hi + 1.0, (n, 3))
    d = rng.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    axis = rng.integers(0, 3, n // 8)                       # some along an axis: 1/d is infinite
    rays[:n // 8, 4:7] = np.eye(3, dtype=np.float32)[axis]
    rays[:, 3] = 1.0
    rays[:, 8] = np.where(rng.random(n) < 0.5, np.inf, rng.uniform(0.1, 9.0, n))
    return rays


@pytest.mark.parametrize("kind", ["coincident", "grid", "random"])
# leaves; 2049 (2048 nodes): the largest index made in one launch
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 9, 33, 513, 2049, 2050, 3000])
def test_index_walk_equals_reference_tree_walk(r, n, kind):
    s = leafgen.leaf_scene(n, kind, seed=n)
    rays = _rays(4000, s.nodes["p_min"][0, :3].min(), s.nodes["p_max"][0, :3].max(), n)
    got = []
    for tree in (0, 1):
        r.set_tree_mode(tree)
        sid = r.upload(s)
        got.append((r.trace(sid, rays), r.trace(sid, rays, any_hit=True)[0]))
        r.release(sid)
    r.set_tree_mode(1)
    for a, b in zip(got[0][0], got[1][0]):
        assert np.array_equal(a.view(np.int32), b.view(np.int32))
    assert np.array_equal(got[0][1], got[1][1])


def test_any_hit_query_reports_the_first_triangle_of_the_two_child_walk(r):
    """The t of an any-hit query is that of the first accepted triangle in the order of the
    two-child walk (nearer child first), which the host replay walks too."""
    s = workloads.mixed_scene(9000, 5, 16, 16, 1)
    q = _rays(3000, -0.4, 0.4, 3)
    q[:, 8] = 1.5
    sid = r.upload(s)
    hit, _, t = r.trace(sid, q, any_hit=True)
    r.release(sid)
    _, _, tri, tw = scenes.walk_counts(s, q, any_hit=True)
    walked = (tri >= 0) & (O.trace(s, q)[1] < 0)   # (a light in front shortens the segment)
    assert walked.sum() > 100   # (enough of the rays settle by a walk to say something)
    assert np.all(hit[walked] == 1)
    assert np.array_equal(t[walked].view(np.int32), tw[walked].view(np.int32))


@pytest.mark.parametrize("rays", [1, 31, 33, 5000])
def test_ray_queries_equal_oracle(r, rays):
    s = workloads.mixed_scene(9000, 5, 16, 16, 1)
    q = O.seeded_rays(s, rays, seed=rays)
    sid = r.upload(s)
    tri, light, t = r.trace(sid, q)
    r.release(sid)
    ot, ol, ott, over = O.trace(s, q)
    assert over.sum() == 0
    assert np.array_equal(tri, ot) and np.array_equal(light, ol)
    assert np.array_equal(t.view(np.int32), ott.view(np.int32))


def test_render_with_a_stack_limit_walks_the_scenes_own_nodes(r):
    s = workloads.mixed_scene(9000, 6, 48, 32, 1)
    sid = r.upload(s)
    r.set_camera(s.cam)
    out = []
    for limit in (0, r.scene_depth(sid) + 2):
        r.set_stack_limit(limit)
        aid = r.alloc_accum(48, 32)
        r.render_passes(sid, aid, scenes.pass_seeds(4, 3), cfg=s.cfg)
        out.append(r.read_accum(aid))
        r.free_accum(aid)
    r.set_stack_limit(0)
    r.release(sid)
    assert np.array_equal(out[0].view(np.int32), out[1].view(np.int32))


@pytest.mark.parametrize("when", ["before", "running"])
def test_batch_with_a_scene_that_has_no_index(r, when):
    """A job whose scene was uploaded in tree mode 0 joins a batch of indexed scenes, before its
    first launch or between two: every job still gives the bits of its own render."""
    jobs = [workloads.mixed_scene(t, 20 + k, 64, 40, 1) for k, t in enumerate((5000, 2500, 7000))]
    sids = []
    for k, s in enumerate(jobs):
        r.set_tree_mode(0 if k == 1 else 1)
        sids.append(r.upload(s))
    r.set_tree_mode(1)
    seeds = scenes.pass_seeds(8, 6)
    b = Batch(r, pool_paths=1024, rounds_per_launch=2, stack_cap=max(r.scene_depth(sid) for sid in sids) + 2)
    accs = [r.alloc_accum(64, 40) for _ in jobs]
    b.add_job(sids[0], accs[0], jobs[0].cam, seeds, jobs[0].cfg)
    if when == "running":
        b.run(max_launches=3)
    for k in (1, 2):
        b.add_job(sids[k], accs[k], jobs[k].cam, seeds, jobs[k].cfg)
    assert b.run() == 0
    for s, sid, aid in zip(jobs, sids, accs):
        ref = r.alloc_accum(64, 40)
        r.set_camera(s.cam)
        r.render_passes(sid, ref, seeds, cfg=s.cfg)
        assert np.array_equal(r.read_accum(aid).view(np.int32), r.read_accum(ref).view(np.int32))
    b.close()


# Any-hit lists take their steps lane by lane or by vote, spread over half the warps or not, by
# the list's length and the scene's size: the same answers and distances whatever the list.
@pytest.mark.parametrize("tris", [0, 1000, 90000])
@pytest.mark.parametrize("n", [100, 30000, 60000, 262144, 300001])
def test_any_hit_lists_of_every_length(r, tris, n):
    s = workloads.mixed_scene(tris, 4, 32, 32, 1) if tris else scenes.c0(32, 32)
    sid = r.upload(s)
    rays = _rays(n, -1.0, 1.0, seed=n)
    tri, light, t = r.trace(sid, rays, any_hit=True)
    for k in range(0, n, 4096):
        if n > 60000 and (k // 4096) % 9:
            continue
        a, b, c = r.trace(sid, rays[k:k + 4096], any_hit=True)
        assert np.array_equal(a, tri[k:k + 4096]) and np.array_equal(b, light[k:k + 4096])
        assert np.array_equal(c.view(np.int32), t[k:k + 4096].view(np.int32))
    r.release(sid)
