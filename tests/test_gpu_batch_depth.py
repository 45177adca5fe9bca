"""A scene whose walk index is deeper than those of a running batch, uploaded after its first launch,
joins it: the walks' stacks grow between two runs and every job gives the bits of its own render."""
import numpy as np
import pytest

from yune_gb300 import _native as N
from yune_gb300 import scenes, workloads
from yune_gb300.batch import Batch
from yune_gb300.core import Renderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smem", [4, 64])   # spilled stacks, whole ones in shared memory
def test_deeper_index_joins_a_running_batch(smem):
    jobs = [scenes.c0(64, 40), workloads.mixed_scene(9000, 21, 64, 40, 1)]
    seeds = scenes.pass_seeds(8, 6)
    with Renderer(0) as r:
        sids, accs = [r.upload(jobs[0])], [r.alloc_accum(64, 40) for _ in jobs]
        b = Batch(r, pool_paths=1024, rounds_per_launch=2, stack_cap=20, stack_smem=smem)
        b.add_job(sids[0], accs[0], jobs[0].cam, seeds, jobs[0].cfg)
        assert b.run(max_launches=2) == 1
        sids.append(r.upload(jobs[1]))
        assert r.scene_depth(sids[1]) + 2 <= 20
        b.add_job(sids[1], accs[1], jobs[1].cam, seeds, jobs[1].cfg)
        made = N.device_allocations()
        assert b.run() == 0
        assert N.device_allocations() > made   # (the index is deeper than 20: larger spill areas)
        for s, sid, aid in zip(jobs, sids, accs):
            ref = r.alloc_accum(64, 40)
            r.set_camera(s.cam)
            r.render_passes(sid, ref, seeds, cfg=s.cfg)
            assert np.array_equal(r.read_accum(aid).view(np.int32), r.read_accum(ref).view(np.int32))
