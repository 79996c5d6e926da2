"""What the speed of this framework is measured on: calls of its public entry
points over the sizes, engines and scene kinds that its workloads use.

A case names an entry point (`form`) and its sizes.  Render forms add samples
to fresh accumulation buffers and return all four of them (or, for the context
form, the image read back to the host); the acceleration-structure forms
return the bit patterns of every buffer they write.
"""
import math

import numpy as np
import torch

from mutracer_b200 import abi, batch, blas, scene, serve, trace
from mutracer_b200 import descriptor as D
from mutracer_b200.context import Context, default_settings

# Image sizes of the mixed workload, plus ragged ones (not a multiple of any
# tile): a progressive renderer is called at whatever size its window has.
SIZES = batch.RESOLUTIONS + ((61, 47), (333, 217), (801, 601), (1003, 777))
MAX_PATHS = 8_000_000


def listed():
    return [
        # Picking and autofocus: a handful of rays, the latency of one call.
        dict(name="pick", form="hits", kind="cornell", triangles=36, rays=33),
        # Visibility queries in bulk over the 4M-triangle instanced scene.
        dict(name="hits_1m", form="hits", kind="spheres", triangles=4_000_000, rays=1_000_000),
        # An interactive preview: one progressive pass of a small viewport.
        dict(name="preview", form="plain", kind="cornell", triangles=36, width=256, height=256, spp=1, lights=1,
             zsobol=False, candidates=1),
        # The small plain configuration (Cornell box, 512 x 512), progressive
        # passes through the drop-in call, ZSobol and light candidates on.
        dict(name="plain_cornell", form="plain", kind="cornell", triangles=36, width=512, height=512, spp=8,
             lights=1, zsobol=True, candidates=3),
        # The headline: 1080p, 16 samples, 4M instanced triangles, wavefront.
        dict(name="spheres_1080p", form="stream", kind="spheres", triangles=4_000_000, width=1920, height=1080,
             spp=16, lights=4, jobs=1, zsobol=False, candidates=1),
        # A thumbnail through the same engine: the event loop's launches count.
        dict(name="thumbnail", form="stream", kind="spheres", triangles=50_000, width=333, height=217, spp=2,
             lights=2, jobs=1, zsobol=False, candidates=1),
        # Deep transport: dispersive glass with media, 20 events a path.
        dict(name="glass_720p", form="stream", kind="glass", triangles=32, width=1280, height=720, spp=1, lights=1,
             jobs=2, zsobol=False, candidates=1),
        # Uneven jobs in one persistent launch.
        dict(name="batch_mixed", form="persistent", kind="spheres", triangles=300_000, width=512, height=512, spp=2,
             lights=3, jobs=8, zsobol=False, candidates=1),
        # Requests over resident scenes, batched as they are admitted.
        dict(name="served", form="served", kind="spheres", triangles=1_000_000, width=512, height=512, spp=6,
             lights=3, jobs=12, zsobol=False, candidates=1),
        # The persistent context a host program uses: commit of a descriptor
        # with maps and alpha coverage, render, image read back.
        dict(name="context_room", form="context", kind="room", triangles=2_000, width=801, height=601, spp=8,
             lights=2, zsobol=False, candidates=1),
        # A mesh's acceleration structure built on the device.
        dict(name="blas_build", form="build", triangles=2 * 733 * 811, bins=8),
        # Per-frame update of a deforming mesh (its plan is made once).
        dict(name="blas_refit", form="refit", triangles=2 * 1000 * 1000, bins=8),
    ]


def draw(rng):
    """One more case of the same forms and ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    form = rng.choice(("hits", "plain", "plain", "stream", "stream", "stream", "persistent", "served", "context",
                       "build", "refit"))
    if form in ("build", "refit"):
        side = log(3, 1000)
        return dict(form=form, triangles=2 * side * log(max(3, side // 4), min(1000, side * 4)),
                    bins=rng.choice((8, 8, 16)))
    kind = {"context": "room", "served": "spheres"}.get(form) or rng.choice(("cornell", "spheres", "spheres", "glass"))
    triangles = log(10_000, 4_000_000) if kind == "spheres" else log(200, 20_000) if kind == "room" else 36
    if form == "hits":
        return dict(form=form, kind=kind, triangles=triangles, rays=log(1, 1_000_000))
    width, height = rng.choice(SIZES) if rng.random() < 0.6 else (log(17, 1920), log(13, 1080))
    jobs = rng.randint(2, 8) if form in ("persistent", "served") else rng.choice((1, 1, 3)) if form == "stream" else 1
    limit = MAX_PATHS // {"plain": 4, "persistent": 4, "context": 2}.get(form, 1) // (6 if kind == "glass" else 1)
    while width * height * jobs > limit:
        width, height = max(17, width * 2 // 3), max(13, height * 2 // 3)
    spp = min(log(1, 16), max(1, limit // (width * height * jobs)))
    return dict(form=form, kind=kind, triangles=triangles, width=width, height=height, spp=spp,
                lights=rng.randint(1, 8), jobs=jobs, zsobol=rng.random() < 0.25, candidates=rng.choice((1, 1, 1, 3)))


# ------------------------------------------------------------------- scenes
def uv_sphere(segments, rings):
    v, u = np.meshgrid(np.arange(rings + 1) / rings, np.arange(segments + 1) / segments, indexing="ij")
    th, ph = math.pi * v, 2 * math.pi * u
    pos = np.stack([np.sin(th) * np.cos(ph), np.cos(th), np.sin(th) * np.sin(ph)], -1).reshape(-1, 3)
    a = (np.arange(rings)[:, None] * (segments + 1) + np.arange(segments)[None, :]).reshape(-1)
    b = a + segments + 1
    idx = np.concatenate([np.stack([a, a + 1, b], 1), np.stack([a + 1, b + 1, b], 1)])
    return pos.astype(np.float32), np.stack([u, 1 - v], -1).reshape(-1, 2).astype(np.float32), idx


def room(case, seed):
    """A room descriptor: mapped floor, a cutout panel and a translucent
    sphere among textured and coated ones, a sky and two analytic lights."""
    rng = np.random.default_rng(seed)
    d = D.Descriptor(case["width"], case["height"])
    quad = np.array([[-1, 0, -1], [1, 0, -1], [1, 0, 1], [-1, 0, 1]], np.float32)
    uv = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], np.float32)
    none = D.NO_TEXTURE
    floor = d.add_texture(16, 16, rng.integers(30, 255, (16, 16, 4), dtype=np.uint8) | np.uint8([0, 0, 0, 255]),
                          uv_scale=(3, 3))
    mr = d.add_texture(8, 8, rng.integers(20, 255, (8, 8, 4), dtype=np.uint8), wrap_s=1, wrap_t=2)
    holes = np.full((16, 16, 4), 255, np.uint8)
    holes[..., 3] = np.where(rng.random((16, 16)) < 0.5, 255, 0)
    holes = d.add_texture(16, 16, holes)
    ground = d.add_geometry(quad * np.float32(4), [0, 2, 1, 0, 3, 2], uvs=uv)
    panel = d.add_geometry(np.array([[-.7, 0, 0], [.7, 0, 0], [.7, 1.4, 0], [-.7, 1.4, 0]], np.float32),
                           [0, 1, 2, 0, 2, 3], uvs=uv)
    segments = max(6, int(math.sqrt(case["triangles"] / 4)))
    pos, suv, idx = uv_sphere(2 * segments, segments)
    ball = d.add_geometry(pos, idx.reshape(-1), uvs=suv)
    d.add_mesh(ground, d.add_material(base_color=(1, 1, 1), roughness=0.6, textures=(floor, none, none, none)))
    d.add_mesh(panel, d.add_material(base_color=(1, 1, 1), roughness=0.5, textures=(holes, none, none, none),
                                     extensions=[(54, 1)]), transform=D.translate([0.9, 0, 0.9]))
    for k in range(6):
        kw = (dict(metalness=1.0, textures=(none, none, mr, none)), dict(coat_weight=1.0, coat_roughness=0.1),
              dict(opacity=0.4), dict(transmission=1.0, roughness=0.05), dict(roughness=0.9), dict(roughness=0.2))[k]
        m = d.add_material(**dict(dict(base_color=tuple(rng.uniform(0.2, 0.9, 3)), roughness=0.3), **kw))
        scale = float(rng.uniform(0.3, 0.6))
        d.add_mesh(ball, m, transform=D.translate([1.3 * (k % 3 - 1), scale, 0.2 - 1.2 * (k // 3)], scale))
    d.add_light(D.LIGHT_RECT, intensity=7, size=1.0, height_or_inner=0.8,
                transform=D.look_at([0, 2.9, 0.3], [0, 0, 0]))
    d.add_light(D.LIGHT_SPHERE, color=(1, 0.9, 0.8), intensity=3, size=0.1, transform=D.translate([1.5, 1.5, 1.8]))
    sky = np.full((8, 16, 4), 0.3, np.float32)
    sky[..., 3] = 1
    d.set_environment(d.add_texture_rgba32f(16, 8, sky), intensity=0.5)
    d.set_camera(fov=45, transform=D.look_at([0, 1.5, 4.2], [0, 0.7, 0]))
    return d.to_bytes()


def host_scene(case, seed, width, height):
    if case["kind"] == "cornell":
        host = scene.SceneHost("cornell", width, height, seed)
    elif case["kind"] == "glass":
        host = scene.SceneHost("glass_spheres", width, height, seed, (32,))
    else:
        if case["triangles"] >= 3_000_000:
            params = (256, 16, 28, 2048, case.get("lights", 4))
        else:
            params = batch.JobSpec(0, width, height, 1, case["triangles"], case.get("lights", 4), seed).scene_params()
        host = scene.SceneHost("instanced_spheres", width, height, seed, params)
    u = abi.TraceUniform.from_buffer_copy(host.uniform)
    u.sequence_seed = seed & 0x7FFFFFFF
    flags = host.flags
    if case.get("zsobol"):
        u.zsobol_log_spp = 3
        flags = (flags & ~abi.MTC_SCENE_PATTERN_MASK) | (abi.MT_SAMPLING_ZSOBOL << abi.MTC_SCENE_PATTERN_SHIFT)
    u.direct_light_candidates = case.get("candidates", 1)
    host.set_uniform(u, None, flags)
    return host


def uneven(case):
    """(width, height, spp) of each job: the case's own, then smaller ones."""
    rng = np.random.default_rng(case["width"] + case["height"])
    out = [(case["width"], case["height"], case["spp"])]
    for _ in range(case.get("jobs", 1) - 1):
        k = rng.uniform(0.4, 1.0, 2)
        out.append((max(13, int(case["width"] * k[0])), max(13, int(case["height"] * k[1])),
                    int(rng.integers(1, case["spp"] + 1))))
    return out


def rays_into(host, count, seed):
    """Rays from a shell around the scene to points inside its bounds."""
    rng = np.random.default_rng(seed)
    b = np.array(host.info.world_bounds, np.float64)
    centre, half = 0.5 * (b[:3] + b[3:]), 0.5 * (b[3:] - b[:3])
    v = rng.normal(size=(count, 3))
    v[:, 1] = np.abs(v[:, 1])
    origin = centre + 1.2 * np.linalg.norm(half) * v / np.linalg.norm(v, axis=1, keepdims=True)
    to = centre + half * rng.uniform(-0.8, 0.8, (count, 3)) - origin
    rays = np.zeros((count, 8), np.float32)
    rays[:, :3], rays[:, 4:7] = origin, to / np.linalg.norm(to, axis=1, keepdims=True)
    return torch.from_numpy(rays).cuda()


class OwnedContext(Context):
    """A context given back with the state that holds it."""

    def __del__(self):
        self.destroy()


# -------------------------------------------------------------- the contract
def prepare(case, seed):
    form = case["form"]
    if form in ("build", "refit"):
        side = max(1, int(math.sqrt(case["triangles"] / 2)))
        pos, idx = blas.terrain_mesh(side, max(1, case["triangles"] // (2 * side)), seed=seed)
        pos, idx = torch.from_numpy(pos).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
        builder = blas.BlasBuilder(len(idx), case["bins"])
        out = torch.zeros(max(blas.max_vec4(len(idx)), 1) * 4, dtype=torch.float32, device="cuda")
        if form == "build":
            return dict(form=form, builder=builder, pos=pos, idx=idx, out=out)
        bvh, _ = builder.build(pos, idx, out)
        return dict(form=form, refit=blas.BlasRefit(bvh), out=out,
                    pos=pos * torch.tensor([1.0, 1.0 + 0.01 * (seed % 31), 1.25], device="cuda"))
    if form == "hits":
        host = host_scene(case, seed, 64, 64)
        return dict(form=form, scene=scene.DeviceScene(host), rays=rays_into(host, case["rays"], seed))
    if form == "context":
        settings = default_settings()
        settings.seed = seed & 0x7FFFFFFF
        settings.sampling_pattern = abi.MT_SAMPLING_ZSOBOL if case["zsobol"] else abi.MT_SAMPLING_SOBOL
        settings.direct_light_candidates = case["candidates"]
        return dict(form=form, data=room(case, seed), settings=settings, context=OwnedContext(), spp=case["spp"],
                    out=np.empty((case["height"], case["width"], 4), np.float32))
    if form == "served":
        pool = serve.ScenePool()
        for k in range(3):  # scenes of unequal size, resident
            pool.add(k, host_scene(dict(case, triangles=max(10_000, case["triangles"] >> (2 * k))), seed + k, 256, 256))
        rng = np.random.Generator(np.random.PCG64(seed))
        jobs = [(k % 3, w, h, s, serve.orbit_camera(pool.hosts[k % 3], w, h, rng))
                for k, (w, h, s) in enumerate(uneven(case))]
        server = serve.Server(pool, job_bytes=sum(j[1] * j[2] for j in jobs) * serve.ACCUMULATION_BYTES_PER_PIXEL,
                              quantum=4)
        return dict(form=form, server=server, jobs=jobs)
    jobs = [batch.RenderJob(scene.DeviceScene(host_scene(case, seed + k, w, h)), s, job_id=k)
            for k, (w, h, s) in enumerate(uneven(case))]
    if form == "plain":
        return dict(form=form, jobs=jobs)
    b = batch.StreamBatch(len(jobs)) if form == "stream" else batch.Batch(len(jobs))
    b.set_jobs(jobs)
    return dict(form=form, jobs=jobs, batch=b)


def run(state):
    form = state["form"]
    if form == "hits":
        return trace.query_first_hit(state["scene"], state["rays"])
    if form == "build":
        _, result = state["builder"].build(state["pos"], state["idx"], state["out"])
        return dict(bvh=state["out"].view(torch.int32), vec4=result.vec4_count, depth=result.max_depth)
    if form == "refit":
        area = state["refit"].refit(state["pos"])
        return dict(bvh=state["out"].view(torch.int32), area=area)
    if form == "context":
        state["context"].commit_descriptor(state["data"], state["settings"])
        state["context"].render(state["spp"])
        return state["context"].read_pixels(out=state["out"])
    if form == "served":
        requests = [serve.Request(k, sid, w, h, s, 0.0, cam) for k, (sid, w, h, s, cam) in enumerate(state["jobs"])]
        state["server"].run(requests, keep_outputs=True)
        return [images(r.job) for r in requests]
    for j in state["jobs"]:  # a new frame
        j.acc.zero_()
    if form == "plain":
        for j in state["jobs"]:
            j.render_alone()
    elif form == "stream":
        state["batch"].run()
    else:
        state["batch"].launch()
    return [images(j) for j in state["jobs"]]


def images(job):
    a = job.acc
    return [a.color, a.normal, a.albedo, a.catcher]


# Arithmetic of one path sample: extension and shadow rays times box,
# instance and triangle tests (counted by the CPU checker), plus shading.
PATH_FLOPS = {"cornell": 15e3, "spheres": 11e3, "glass": 60e3, "room": 12e3}
SCENE_BYTES = {"cornell": 4e5, "glass": 2e6, "room": 1e6}


def scene_bytes(case):
    # 16 distinct meshes at most, 256 instances or fewer, their maps and sky
    return SCENE_BYTES.get(case["kind"]) or min(case["triangles"], 260_000) * 70.0 + 8e6


def work(case):
    form, n = case["form"], case["triangles"]
    if form == "build":    # positions and indices in, five vec4 a triangle out; a pass of bins per level
        return dict(bytes=n * (12 + 6 + 80), flops=n * math.log2(n + 1) * 40)
    if form == "refit":    # positions and records in, node boxes rewritten
        return dict(bytes=n * (16 + 6 + 2 * 32), flops=n * 24)
    if form == "hits":
        return dict(bytes=case["rays"] * 64 + min(scene_bytes(case), case["rays"] * 4000.0),
                    flops=case["rays"] * 3500.0)
    jobs = case.get("jobs", 1)
    share = 1.0 if jobs == 1 else (1.0 + (jobs - 1) * 0.49 * 0.5) / jobs   # uneven(): later jobs are smaller
    pixels = case["width"] * case["height"] * jobs * (1.0 if jobs == 1 else (1.0 + (jobs - 1) * 0.49) / jobs)
    paths = case["width"] * case["height"] * case["spp"] * jobs * share
    return dict(bytes=pixels * 96 + scene_bytes(case), flops=paths * PATH_FLOPS[case["kind"]])


def exact(case, seed):
    """None for every case.  Path samples follow discrete decisions (hit, lobe
    and light choices) of 32-bit arithmetic, which 64 bits would take
    otherwise; hits, builds and refits return bit patterns, and a refit's
    area sums boxes of a tree only this framework makes."""
    return None
