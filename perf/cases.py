"""Performance cases of the rendering core: what a host program has it do, through its public entry points.

A case is a plain dict; `prepare` makes the scene, the device handles and the inputs of one seed, `run` is one call (or
the few calls that belong together) of a user's program, and `work` says what that call cannot do without. One context
is kept for the whole process, as a renderer keeps it; scenes, accumulators and batches belong to a prepared state and
are released with it. Every pass starts its accumulators anew, so a pass on a prepared state always does the same work.

Kinds and the ranges `draw` takes them from:
  frame   the interactive loop: camera, one pass into a cleared accumulator, tonemapped frame to the host
  pass    progressive passes of one frame: unidirectional, naive bidirectional, bidirectional with MIS
  batch   several jobs (scene, frame, passes) in one wavefront of the batch engine
  rays    direct ray queries, from device buffers or host arrays
  load    a new model: BVH build, upload, first pass
  refit   an animation frame: moved triangles, refit, pass
"""
import math
import weakref

import numpy as np
import torch

from yune_gb300 import _native, scenes, workloads
from yune_gb300.batch import Batch
from yune_gb300.core import Renderer
from yune_gb300.layouts import BVH_NODE, ptr

# the options the reference kernels ship with: no MIS, Lambert, roulette after bounce 6
SHIPPED = dict(mis=0, brdf_model=0, rr_threshold=6, mis_lobe_fix=0)
# the options of the mixed workload: next event + MIS, Oren-Nayar, roulette after bounce 3, at most 16 bounces
MIXED = dict(mis=1, brdf_model=1, rr_threshold=3, mis_lobe_fix=0, max_depth=16)
# the mixed workload's kind of jobs, "triangle target:width x height" each
JOBS = "1500:512x512,6000:256x256,20000:1280x720,45000:512x512,90000:1920x1080,150000:1280x720,260000:256x256,400000:1920x1080"


def listed():
    return [
        # a viewer's frame while the camera moves: the smallest frame of the mixed workload, latency counts
        dict(name="frame_box_256", kind="frame", scene="box", tris=0, width=256, height=256, integrator=0, passes=1),
        # the Cornell box configuration at its own size, a few progressive passes between two screen updates
        dict(name="pass_box_512", kind="pass", scene="box", tris=0, width=512, height=512, integrator=0, passes=4),
        # the glass sphere configuration at its own size: long specular paths, one pass
        dict(name="pass_glass_1024", kind="pass", scene="glass", tris=81954, width=1024, height=1024, integrator=0, passes=1),
        # a model of the mixed workload's size in its largest frame
        dict(name="pass_mixed_1080p", kind="pass", scene="mixed", tris=260000, width=1920, height=1080, integrator=0, passes=1),
        # an odd tile of a window with the reference's shipped options (no MIS)
        dict(name="pass_shipped_ragged", kind="pass", scene="mixed", tris=21000, width=1003, height=565, integrator=0, passes=2, shipped=True),
        # the naive bidirectional tracer on a field of spheres with four lights (the stress scene's kind, 1/12 of its size)
        dict(name="bdpt_field_720p", kind="pass", scene="field", tris=820000, width=1280, height=720, integrator=1, passes=1),
        # bidirectional with MIS, Cornell box with four lights at its own size
        dict(name="bdpt_mis_box_512", kind="pass", scene="box4", tris=0, width=512, height=512, integrator=2, passes=2),
        # eight jobs of the mixed workload served in one wavefront
        dict(name="batch_mixed_8", kind="batch", jobs=JOBS, passes=4),
        # visibility rays of a host program (picking, probes): small, host arrays
        dict(name="rays_any_host_4k", kind="rays", scene="box", tris=0, rays=4096, any=1, host=True),
        # incoherent closest-hit queries from device buffers, as a baker or another integrator sends them
        dict(name="rays_closest_1m", kind="rays", scene="glass", tris=81954, rays=1 << 20, any=0, host=False),
        # a new model until its first small frame: BVH build, upload, pass
        dict(name="load_mixed_330k", kind="load", scene="mixed", tris=330000, width=256, height=256, integrator=0, passes=1),
        # an animation frame: new vertex positions, refit, pass
        dict(name="refit_mixed_90k", kind="refit", scene="mixed", tris=90000, width=512, height=512, integrator=0, passes=1),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def frame(lo, hi):
        pixels, aspect = log_int(lo, hi), rng.uniform(0.75, 2.0)
        w = max(16, int(math.sqrt(pixels * aspect)))
        return dict(width=w, height=max(16, pixels // w))

    kind = rng.choice(["frame", "pass", "pass", "pass", "bidir", "bidir", "batch", "rays", "load", "refit"])
    scene = rng.choice(["box", "glass", "mixed", "mixed"])
    tris = {"box": 0, "glass": 34 + 20 * 4 ** rng.randint(3, 6), "mixed": log_int(1000, 500000)}[scene]
    if kind == "frame":
        return dict(kind=kind, scene=scene, tris=tris, integrator=0, passes=1, **frame(64 * 64, 512 * 512))
    if kind == "pass":
        return dict(kind=kind, scene=scene, tris=tris, integrator=0, passes=rng.randint(1, 4), shipped=rng.random() < 0.3,
                    **frame(64 * 64, 1920 * 1080))
    if kind == "bidir":
        scene, tris = rng.choice([("box4", 0), ("field", log_int(20000, 820000))])
        return dict(kind="pass", scene=scene, tris=tris, integrator=rng.choice([1, 2]), passes=1, **frame(96 * 64, 1280 * 720))
    if kind == "batch":
        sizes = ["256x256", "512x512", "1280x720", "611x403", "1920x1080"]
        jobs = ["%d:%s" % (log_int(1000, 400000), rng.choice(sizes)) for _ in range(rng.randint(2, 8))]
        return dict(kind="batch", jobs=",".join(jobs), passes=rng.randint(1, 3))
    if kind == "rays":
        host = rng.random() < 0.4
        return dict(kind=kind, scene=scene, tris=tris, rays=log_int(256, 1 << 16 if host else 1 << 20), any=rng.randint(0, 1), host=host)
    return dict(kind=kind, scene="mixed", tris=log_int(2000, 330000), integrator=0, passes=1, **frame(96 * 64, 512 * 512))


# ---- inputs ----

def _scene(case, seed, width=64, height=64):
    """The scene of a case for one seed: same sizes, other geometry and materials for another seed."""
    kind, tris = case["scene"], case["tris"]
    if kind == "box":
        s = scenes.c0(width, height, seed=seed)
    elif kind == "box4":
        s = scenes.c0_bdpt(width, height, seed=seed)
    elif kind == "glass":
        s = scenes.c1(width, height, seed=seed, level=max(2, int(round(math.log(max(tris - 34, 320) / 20.0, 4)))))
    elif kind == "field":
        grid = max(2, int(round(math.sqrt(tris / 6250.0))))
        s = scenes.c4(width, height, seed=seed, grid=grid, n_level5=grid * grid // 13)
    else:
        s = workloads.mixed_scene(tris, seed, width, height, 1, scenes.default_cfg(**MIXED))
    cfg = dict(s.cfg, integrator=case.get("integrator", 0))
    if cfg["integrator"]:
        cfg.update(mis=0, bdpt_bounces=8)
    if case.get("shipped"):
        cfg.update(SHIPPED)
    s.cfg = cfg
    return s


_CONTEXT = []


def _renderer():
    """The process's one context, kept as a renderer keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(Renderer())
    return _CONTEXT[0]


class _State:
    """What one prepared case holds on the device; released with the last reference (outputs keep their state alive)."""

    def __init__(self, case):
        self.case, self.r = case, _renderer()
        self.scenes, self.accums, self.batch = [], [], None
        weakref.finalize(self, _State._release, self.r, self.scenes, self.accums)

    @staticmethod
    def _release(r, sids, aids):
        if getattr(r, "h", None):
            for sid in sids:
                r.release(sid)
            for aid in aids:
                r.free_accum(aid)

    def upload(self, s):
        self.scenes.append(self.r.upload(s))
        return self.scenes[-1]

    def accum(self, w, h):
        self.accums.append(self.r.alloc_accum(w, h))
        return self.accums[-1]

    def image(self, aid):
        """The accumulator as a tensor on the device, no copy."""
        p = _native.C.c_void_p()
        _native.check(self.r.L.yc_accum_device_ptr(self.r.h, aid, _native.C.byref(p)), "yc_accum_device_ptr")
        return torch.as_tensor(_Image(self, p.value, self.r._accum_shape[aid] + (4,)), device="cuda")


class _Image:
    """The CUDA array interface of an accumulator."""

    def __init__(self, state, address, shape):
        self.state = state
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(address, False), version=3)


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    w, h = case.get("width", 0), case.get("height", 0)
    st.seeds = np.random.default_rng(seed + 7).integers(1, 1 << 32, case.get("passes", 1), dtype=np.uint32)
    if kind == "batch":
        st.batch = Batch(st.r, pool_paths=1 << 20, max_jobs=1 << 16, sort_threshold=65536, groups=4, ray_sort=322, trace_share=50,
                         stack_cap=64)
        st.jobs = []
        for k, text in enumerate(case["jobs"].split(",")):
            tris, size = text.split(":")
            jw, jh = (int(v) for v in size.split("x"))
            s = _scene(dict(scene="mixed", tris=int(tris)), seed * 101 + k, jw, jh)
            st.jobs.append((st.upload(s), st.accum(jw, jh), s.cam, s.cfg))
    elif kind == "rays":
        st.sid = st.upload(_scene(case, seed))
        rays = _rays(case, seed)
        if case["host"]:
            st.rays = rays
        else:
            st.rays = torch.from_numpy(rays).cuda()
            st.tri = torch.empty(case["rays"], dtype=torch.int32, device="cuda")
            st.t = torch.empty(case["rays"], dtype=torch.float32, device="cuda")
    else:
        st.scene = s = _scene(case, seed, w, h)
        st.aid = st.accum(w, h)
        if kind == "frame":
            st.out = _host_frame(w, h)
        if kind == "load":
            st.nodes = np.zeros(2 * len(s.tris) + 1, BVH_NODE)
        else:
            st.sid = st.upload(s)
        if kind == "refit":
            st.moved = _moved(s.tris, seed)
    torch.cuda.synchronize()
    return st


def _host_frame(w, h):
    """A page-locked frame buffer, kept from frame to frame."""
    return torch.empty((h, w, 4), dtype=torch.float32, pin_memory=True).numpy()


def _rays(case, seed):
    """Incoherent rays through the box; visibility rays end within it."""
    rays = scenes.box_rays(case["rays"], seed)
    if case["any"]:
        rays[:, 8] = np.random.default_rng(seed + 1).uniform(0.05, 1.5, case["rays"]).astype(np.float32)
    return rays


def _moved(tris, seed):
    """The triangles under a smooth deformation of at most 2% of the box."""
    out = tris.copy()
    a, b = np.random.default_rng(seed + 3).uniform(3.0, 9.0, 2).astype(np.float32)
    for v in ("v1", "v2", "v3"):
        p = tris[v]
        out[v][:, 0] += 0.01 * np.sin(a * p[:, 1])
        out[v][:, 1] += 0.01 * np.sin(b * p[:, 2])
    return out


# ---- one call ----

def _build(st, s):
    """The model with its BVH built on the device, its nodes in the program's own buffer."""
    n, depth = _native.C.c_int(), _native.C.c_int()
    lib, h = st.r.L, st.r.h
    _native.check(lib.yc_bvh_build(h, ptr(s.tris), len(s.tris), 20, 4, _native.C.byref(n), _native.C.byref(depth)), "yc_bvh_build")
    _native.check(lib.yc_bvh_copy_nodes(h, ptr(st.nodes), len(st.nodes)), "yc_bvh_copy_nodes")
    return scenes.SceneData(s.tris, s.mats, s.lights, st.nodes[:n.value], depth.value, s.cam, s.width, s.height, 1)


def run(st):
    case, r = st.case, st.r
    kind = case["kind"]
    if kind == "batch":
        for sid, aid, cam, cfg in st.jobs:
            st.batch.add_job(sid, aid, cam, st.seeds, cfg)
        st.batch.run()
        return [st.image(aid) for _, aid, _, _ in st.jobs]
    if kind == "rays":
        if case["host"]:
            tri, light, t = r.trace(st.sid, st.rays, any_hit=bool(case["any"]))
            return dict(tri=tri, light=light, t=t)
        r.trace_device(st.sid, st.rays.data_ptr(), case["rays"], bool(case["any"]), st.tri.data_ptr(), st.t.data_ptr())
        return dict(tri=st.tri, t=st.t)
    s = st.scene
    out = {}
    if kind == "load":
        sid = r.upload(_build(st, s))
        out["nodes"] = st.nodes.view(np.uint8)
    else:
        sid = st.sid
        if kind == "refit":
            r.refit(sid, st.moved)
    r.set_camera(s.cam)
    r.render_passes(sid, st.aid, st.seeds, reset_first=1, cfg=s.cfg)
    if kind == "load":
        r.release(sid)
    if kind == "frame":
        out["frame"] = r.tonemap(st.aid, out=st.out)
    out["accum"] = st.image(st.aid)
    return out


# ---- what a call cannot do without ----
# Rays a sample sends on average, child boxes and triangles a ray has to test in a good hierarchy: a slab test is 6
# subtractions, 6 products and 11 minima or maxima, a triangle test up to 52 operations, shading a vertex some 300.
_RAYS = {0: 8.0, 1: 26.0, 2: 22.0}


def _trace_flops(rays, tris):
    boxes = 2.0 * (2.0 + math.log2(max(tris, 34)))
    return rays * (boxes * 23.0 + 0.25 * boxes * 52.0)


def _scene_bytes(tris):
    return 112.0 * max(tris, 34)


def work(case):
    kind = case["kind"]
    if kind == "rays":
        n, tris = case["rays"], max(case["tris"], 34)
        return dict(bytes=44.0 * n + min(_scene_bytes(tris), 400.0 * n), flops=_trace_flops(n, tris))
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for text in case["jobs"].split(","):
            tris, size = text.split(":")
            w, h = size.split("x")
            one = work(dict(kind="pass", tris=int(tris), width=int(w), height=int(h), integrator=0, passes=case["passes"]))
            total = {k: total[k] + one[k] for k in total}
        return total
    n = case["width"] * case["height"]
    rays = _RAYS[case["integrator"]] * n * case["passes"]
    flops = _trace_flops(rays, case["tris"]) + 300.0 * rays
    size = 16.0 * n + _scene_bytes(case["tris"])
    if kind == "frame":
        size += 16.0 * n
    if kind == "load":
        size += 3.0 * _scene_bytes(case["tris"])
    if kind == "refit":
        size += 2.0 * _scene_bytes(case["tris"])
    return dict(bytes=size, flops=flops)


# ---- the same in 64 bits ----

def exact(case, seed):
    if case["kind"] == "rays" and not case["any"] and case["rays"] * max(case["tris"], 34) <= 1e11:
        t = _brute_force(_scene(case, seed), _rays(case, seed))
        return dict(tri=None, light=None, t=t) if case["host"] else dict(tri=None, t=t)
    # an any-hit query answers with whichever triangle it meets first, and the paths of a path-traced image branch on
    # every comparison: neither has a value in 64 bits
    return None


def _brute_force(s, rays):
    """Per ray the distance to its closest surface (the quad lights first, then every triangle), or the ray's length."""
    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a[..., :3], dtype=np.float64)).cuda()

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    def cross(a, b):
        return a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]

    ray = torch.from_numpy(rays.astype(np.float64)).cuda()
    o, d, t = ray[:, 0:3], ray[:, 4:7], ray[:, 8].clone()
    for q in s.lights:
        p, n, el, ew = (dev(q[k]) for k in ("pos", "normal", "edge_l", "edge_w"))
        dn = d @ n
        tl = ((p - o) @ n) / dn
        at = o + d * tl[:, None] - p
        a, b = at @ (el / el.norm()), at @ (ew / ew.norm())
        hit = (dn.abs() > 1e-4) & (tl > 0) & (tl < t) & (a >= 0) & (b >= 0) & (a <= el.norm()) & (b <= ew.norm())
        t = torch.where(hit, tl, t)
    v1, v2, v3 = (dev(s.tris[k]).T for k in ("v1", "v2", "v3"))
    e1, e2 = v2 - v1, v3 - v1
    step = max(1, (1 << 26) // v1.shape[1])
    for k in range(0, len(ray), step):
        ok, dk = o[k:k + step].T[:, :, None], d[k:k + step].T[:, :, None]
        p = cross(dk, e2)
        inv = 1.0 / dot(p, e1)
        sv = ok - v1[:, None, :]
        u = dot(p, sv) * inv
        hit = (u >= 0) & (u <= 1)
        q = cross(sv, e1)
        v, tt = dot(q, dk) * inv, dot(q, e2) * inv
        hit &= (v >= 0) & (u + v <= 1) & (tt > 0)
        t[k:k + step] = torch.minimum(t[k:k + step], torch.where(hit, tt, torch.inf).amin(1))
    return t
