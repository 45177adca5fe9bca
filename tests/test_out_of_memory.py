"""A call that the device's memory does not hold fails with YC_E_NOMEM and leaves the context as
usable as before: the buffers that it gave up are made again by the next call that needs them."""
import numpy as np
import pytest

import fake_cuda
from yune_gb300 import _native as N
from yune_gb300 import scenes, serve, workloads
from yune_gb300.batch import Batch
from yune_gb300.core import Renderer


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_cuda.load(tmp_path_factory.mktemp("fake_cuda"))


@pytest.fixture
def r(fake, monkeypatch):
    monkeypatch.setattr(N, "_lib", fake)
    fake.fake_limit(fake_cuda.NO_LIMIT)
    with Renderer(0) as rr:
        yield rr
    fake.fake_limit(fake_cuda.NO_LIMIT)
    assert fake.fake_bytes() == 0   # everything was given back


@pytest.mark.parametrize("integrator", [0, 1, 2])
@pytest.mark.parametrize("tris", [0, 5000])   # 5000: the rays are sorted
def test_small_frame_after_a_frame_too_large(r, fake, integrator, tris):
    s = workloads.mixed_scene(tris, 5, 16, 16, 1) if tris else scenes.c0(16, 16)
    cfg = scenes.default_cfg(integrator=integrator, bdpt_bounces=4)
    r.set_camera(s.cam)

    def frames(q):
        q.set_repack(0)   # (on the host: kernels do not run here)
        sid, small, large = q.upload(s), q.alloc_accum(320, 256), q.alloc_accum(1024, 1024)
        q.set_camera(s.cam)
        q.render_passes(sid, small, [1, 2], reset_first=1, cfg=cfg)
        return sid, small, large

    sid, small, large = frames(r)
    held = fake.fake_bytes()
    r.render_passes(sid, large, [1, 2], reset_first=1, cfg=cfg)
    need = fake.fake_bytes() - held
    r.close()
    failed = 0
    for share in range(20):   # memory ends at one allocation after another
        with Renderer(0) as q:
            sid, small, large = frames(q)
            buffers = fake.fake_allocations()
            fake.fake_limit(fake.fake_bytes() + need * share // 20)
            try:
                q.render_passes(sid, large, [1, 2], reset_first=1, cfg=cfg)
            except N.YuneError as e:
                assert e.code == N.YC_E_NOMEM
                failed += 1
            fake.fake_limit(fake_cuda.NO_LIMIT)
            q.render_passes(sid, small, [1, 2], reset_first=1, cfg=cfg)
            assert fake.fake_allocations() >= buffers   # whichever of them had to go
    assert failed >= 5


def test_batch_without_memory_for_its_stacks(r, fake):
    """The walks' spill areas are made when a batch runs and when its walks change to the scenes' own
    nodes (a scene without an index joins it): no run goes ahead without them."""
    r.set_repack(0)
    s = workloads.mixed_scene(5000, 5, 16, 16, 1)
    sid, aid = r.upload(s), r.alloc_accum(64, 64)
    r.set_tree_mode(0)
    plain = r.upload(s)
    b = Batch(r, pool_paths=4096, stack_cap=64, stack_smem=2)
    b.add_job(sid, aid, s.cam, [1], s.cfg)
    made = fake.fake_allocations()
    fake.fake_limit(fake.fake_bytes() + 4096)
    with pytest.raises(N.YuneError) as e:
        b.run(max_launches=1)
    assert e.value.code == N.YC_E_NOMEM
    fake.fake_limit(fake_cuda.NO_LIMIT)
    b.run(max_launches=1)
    running = fake.fake_allocations()
    assert running > made
    fake.fake_limit(1)
    with pytest.raises(N.YuneError) as e:
        b.add_job(plain, aid, s.cam, [1], s.cfg)
    fake.fake_limit(fake_cuda.NO_LIMIT)
    b.run(max_launches=1)
    assert e.value.code == N.YC_E_NOMEM and fake.fake_allocations() >= running
    b.add_job(plain, aid, s.cam, [1], s.cfg)
    b.run(max_launches=1)
    assert fake.fake_allocations() > running   # (the job's seeds)


def test_upload_indexes_the_scene_when_its_temporaries_are_gone(r, fake):
    """The least memory that takes an upload takes the scene's walk index too: by then the copies of the
    caller's arrays have been given back."""
    s = workloads.mixed_scene(3000, 5, 16, 16, 1)
    before = fake.fake_bytes()
    sid = r.upload(s)
    whole = fake.fake_bytes()
    assert whole - before > r.scene_bytes(sid)   # (the index is beside the scene's arrays)
    r.release(sid)
    low, high = before, before + 64 * (whole - before)
    while high - low > 256:
        mid = (low + high) // 2
        fake.fake_limit(mid)
        try:
            r.release(r.upload(s))
            high = mid
        except N.YuneError as e:
            assert e.code == N.YC_E_NOMEM
            low = mid
    fake.fake_limit(high)
    r.upload(s)
    assert fake.fake_bytes() == whole


def test_small_upload_makes_few_allocations(r, fake):
    """An allocation and its release are a twentieth of the Cornell box's upload: the scene's six arrays
    and its index, and two blocks of temporaries."""
    n = fake.fake_mallocs()
    r.upload(scenes.c0(16, 16))
    assert fake.fake_mallocs() - n <= 9


SEGMENT = 16 + 4 + 8   # bytes of a segment: its ray, its queue entry and the sort's two lists


def _sorted_bdpt(q, s):
    q.set_repack(0)
    sid, aid = q.upload(s), q.alloc_accum(320, 256)
    q.set_camera(s.cam)
    return lambda: q.render(sid, aid, 1, reset=1, cfg=scenes.default_cfg(integrator=2, bdpt_bounces=4)), aid


def test_bidirectional_pass_with_room_for_one_segment_a_path(r, fake):
    s = workloads.mixed_scene(5000, 5, 16, 16, 1)
    n = 320 * 256
    render, _ = _sorted_bdpt(r, s)
    render()
    room = fake.fake_bytes() - 7 * SEGMENT * n   # eight a path where memory allows
    r.close()
    with Renderer(0) as q:
        render, _ = _sorted_bdpt(q, s)
        fake.fake_limit(room)
        render()
        assert fake.fake_bytes() <= room
        fake.fake_limit(fake_cuda.NO_LIMIT)
        q.free_accum(q.alloc_accum(16, 16))   # memory came back: eight again
        render()
        assert fake.fake_bytes() == room + 7 * SEGMENT * n


def test_segments_option(r, fake):
    render, _ = _sorted_bdpt(r, workloads.mixed_scene(5000, 5, 16, 16, 1))
    for bad in (0, 3, 5, 16, -1):
        with pytest.raises(N.YuneError) as e:
            r.set_segments(bad)
        assert e.value.code == N.YC_E_INVALID
    took = []
    for k in (1, 2, 4, 8):
        r.set_segments(k)
        render()
        took.append(fake.fake_bytes())
    assert np.array_equal(np.diff(took), 320 * 256 * SEGMENT * np.array([1, 2, 4]))


def _indexed(r, fake, need, tris=5000):
    """A scene whose index walks of `need` entries take (the upload reads it from its two control words)."""
    fake.fake_store(8, 0, need)
    return r.upload(workloads.mixed_scene(tris, 5, 16, 16, 1))


def _stack_bytes(fake, run):
    before = fake.fake_bytes()
    run()
    return fake.fake_bytes() - before


def test_batch_stacks_are_as_deep_as_its_scenes_need(r, fake):
    r.set_repack(0)
    s = workloads.mixed_scene(5000, 5, 16, 16, 1)
    sid, aid = _indexed(r, fake, 22), r.alloc_accum(64, 64)
    took = []
    for cap in (0, 64, 200):   # (the scene's own, a server's bound, a generous one)
        b = Batch(r, pool_paths=4096, stack_cap=cap, stack_smem=12)
        b.add_job(sid, aid, s.cam, [1], s.cfg)
        took.append(_stack_bytes(fake, lambda: b.run(max_launches=1)))
        b.close()
    # two launches of a group, an entry beyond the 12 in shared memory 8 bytes for each of 152 * 4 * 128
    # threads, two groups: the bound given, or what the index needs
    assert took == [2 * 2 * (n - 12) * 8 * 152 * 4 * 128 for n in (24, 64, 200)]


@pytest.mark.parametrize("need", [22, 118])
def test_batch_with_its_whole_stacks_in_shared_memory(r, fake, need):
    """Stacks that fit a block's shared memory over the scenes' own nodes are not refused over an index."""
    r.set_repack(0)
    s = workloads.mixed_scene(5000, 5, 16, 16, 1)
    sid, aid = _indexed(r, fake, need), r.alloc_accum(64, 64)
    b = Batch(r, pool_paths=4096, stack_cap=100, stack_smem=120, trace_block=256)
    b.add_job(sid, aid, s.cam, [1], s.cfg)
    b.run(max_launches=1)


def test_batch_joined_by_a_scene_with_a_deeper_index(r, fake):
    r.set_repack(0)
    s = workloads.mixed_scene(5000, 5, 16, 16, 1)
    sid, aid = _indexed(r, fake, 22), r.alloc_accum(64, 64)
    per_entry = 2 * 2 * 8 * 152 * 4 * 128

    def started():
        b = Batch(r, pool_paths=4096, stack_cap=30, stack_smem=12)
        b.add_job(sid, aid, s.cam, [1], s.cfg)
        b.run(max_launches=1)
        return b

    a, b = started(), started()
    deep = _indexed(r, fake, 58)
    b.add_job(deep, aid, s.cam, [1], s.cfg)
    assert _stack_bytes(fake, lambda: b.run(max_launches=1)) == (60 - 30) * per_entry
    a.add_job(deep, aid, s.cam, [1], s.cfg)
    fake.fake_limit(fake.fake_bytes() + 4096)   # no room for its stacks: the scenes' own nodes
    assert _stack_bytes(fake, lambda: a.run(max_launches=1)) == 0


def test_server_keeps_its_scene_budget(r, fake):
    """A scene budget bounds what the resident scenes take on the device, walk indexes included: they get
    none where it holds their arrays alone."""
    r.set_repack(0)
    resident = [scenes.c0(16, 16), workloads.mixed_scene(5000, 5, 16, 16, 1)]
    layouts = [scenes.layout(s) for s in resident]
    need = sum(lay["device_bytes"] for lay in layouts)
    whole = need + sum(scenes.index_bound(lay) for lay in layouts)
    for budget, took in ((need, need), (whole - 1, need), (whole, whole), (None, whole)):
        before = fake.fake_bytes()
        srv = serve.Server(r, resident, hbm_budget=1 << 20, scene_budget=budget, pool_paths=1024)
        srv.close()   # (its batch goes, the scenes stay)
        assert fake.fake_bytes() - before == took
        for sid in srv.sids:
            r.release(sid)
    assert r.walk_index


def test_ray_queries_give_the_buffers_of_long_lists_back(r, fake):
    """Short lists' buffers are kept from call to call, those of a list of millions until the next."""
    sid = r.upload(scenes.c0(16, 16))
    rays = scenes.box_rays(3 << 20, 1)
    r.trace(sid, rays[:1])
    before, per_ray = fake.fake_bytes(), (9 + 2) * 4
    for n, held in ((5000, 5000), (100, 5000), (1 << 20, 1 << 20), (5000, 1 << 20), (3 << 20, 3 << 20),
                    (2 << 20, 2 << 20), (10, 10)):
        r.trace(sid, rays[:n])
        assert fake.fake_bytes() - before == (held - 1) * per_ray
