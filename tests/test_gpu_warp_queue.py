"""The warp-queue traversal and the megakernels' pixel claims at the sizes where
they could go wrong: ray counts around a warp, a batch and a block, images that
no tile divides, queues with fewer and more rays than lanes, launch shapes that
leave warps idle, and BLAS sizes around the builder's and the refit's runs.
Hits and boxes are bit-exact against the CPU oracle; images are bit-identical
across engines."""
import numpy as np
import pytest

from mutracer_b200 import abi, batch, blas, scene, trace
from tests import oracle_lib
from tests.test_gpu_parity import REL_MSE_BAR, _hits_equal, _image_metrics, _render_pair

pytestmark = pytest.mark.gpu
SMALL = (24, 3, 4, 64, 2)  # instances, meshes, frequency, sky width, lights


@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 127, 128, 129, 4097, 60_001])
def test_first_hits_at_batch_edges(cuda, count, layout):
    import torch
    host = scene.SceneHost("instanced_spheres", 32, 32, 3, SMALL)
    if layout:
        host.set_blas_layout(layout)
    rays = oracle_lib.seeded_rays(host, count, seed=count)
    rays[::7, 4:7] *= -1.0  # some rays leave the scene at once
    got = trace.query_first_hit(scene.DeviceScene(host, cuda), torch.from_numpy(rays).to(cuda)).cpu().numpy()
    same, tie = _hits_equal(got, oracle_lib.first_hits(host, rays))
    assert (same | tie).all()


@pytest.mark.parametrize("layout", [0, 2])
def test_bulk_first_hits_match_smaller_calls(cuda, layout):
    """Ray counts and scenes on either side of the rules that hand rays to lanes
    one by one or for good: the same bits as in calls of a few thousand rays."""
    import torch
    host = scene.SceneHost("instanced_spheres", 32, 32, 3, (24, 6, 6, 64, 2))
    few = scene.SceneHost("cornell", 32, 32, 3)
    if layout:
        host.set_blas_layout(layout)
        few.set_blas_layout(layout)
    for h in (host, few):
        dev = scene.DeviceScene(h, cuda)
        assert (dev.view.bvh_vec4_count > 4096) == (h is host)
        sms = torch.cuda.get_device_properties(cuda).multi_processor_count
        rays = torch.from_numpy(oracle_lib.seeded_rays(h, sms * 60 * 64 + 37, seed=5)).to(cuda)
        part = torch.cat([trace.query_first_hit(dev, r) for r in rays.split(3001)])
        for count in (len(rays), sms * 60 * 64 - 1, sms * 12 * 3 + 1, sms * 12):
            assert torch.equal(trace.query_first_hit(dev, rays[:count].contiguous()), part[:count]), (count, layout)


def _same(a, b):
    import torch
    return all(torch.equal(getattr(a, k), getattr(b, k)) for k in ("color", "normal", "albedo", "catcher"))


@pytest.mark.parametrize("kind,params", [("instanced_spheres", SMALL), ("glass_spheres", (4,))])
@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (9, 5), (257, 3), (33, 131)])
def test_engines_agree_on_ragged_images(cuda, kind, params, size):
    import torch
    host = scene.SceneHost(kind, *size, 5, params)
    dev = scene.DeviceScene(host, cuda)
    plain = batch.RenderJob(dev, 3, device=cuda)
    plain.render_alone()
    torch.cuda.synchronize()
    assert (plain.acc.normal[:, 3] == 3).all()
    for cfg in ((0, 0, 0, 0), (32, 1, 1, 16), (96, 32, 2, 3)):
        job = batch.RenderJob(dev, 3, device=cuda)
        b = batch.Batch(1, abi.BatchConfig.make(*cfg), cuda)
        b.set_jobs([job])
        b.launch()
        torch.cuda.synchronize()
        assert _same(plain.acc, job.acc), cfg
    job = batch.RenderJob(dev, 3, device=cuda)
    sb = batch.StreamBatch(1, stream_config=abi.StreamConfig.make(slots=1024), device=cuda)
    sb.set_jobs([job])
    sb.run()
    torch.cuda.synchronize()
    assert _same(plain.acc, job.acc)


def test_dense_and_sparse_queues_agree(cuda):
    """640,000 pixels: dense rays per warp, the costly classes first, samples
    finished while shading; the same image through 1,024 slots."""
    import torch
    host = scene.SceneHost("instanced_spheres", 1000, 640, 2, SMALL)
    dev = scene.DeviceScene(host, cuda)
    plain = batch.RenderJob(dev, 2, device=cuda)
    plain.render_alone()
    for kw in (dict(), dict(slots=1024, refill_lanes=32, steps_per_check=1), dict(regroup_interval=3, sort_rays=1)):
        job = batch.RenderJob(dev, 2, device=cuda)
        sb = batch.StreamBatch(1, stream_config=abi.StreamConfig.make(**kw), device=cuda)
        sb.set_jobs([job])
        sb.run()
        torch.cuda.synchronize()
        assert _same(plain.acc, job.acc), kw
        assert int(sb.counters[0]) == 2 * 640_000


def test_ragged_image_meets_the_oracle(cuda):
    gpu, ref, _, _ = _render_pair(cuda, scene.SceneHost("cornell", 67, 45, 5), 32)
    rel_mse, luma = _image_metrics(gpu, ref)
    assert rel_mse <= REL_MSE_BAR and luma <= 0.005


def test_persistent_claims_over_uneven_jobs(cuda):
    """Jobs of one pixel, of no samples and of unlike scenes share a launch."""
    import torch
    hosts = [scene.SceneHost("cornell", 1, 1, 1), scene.SceneHost("instanced_spheres", 61, 7, 2, SMALL),
             scene.SceneHost("cornell", 40, 9, 3), scene.SceneHost("glass_spheres", 13, 17, 4, (3,))]
    devs = [scene.DeviceScene(h, cuda) for h in hosts]
    spp = [5, 2, 0, 1]
    for fetch in (1, 16):
        jobs = [batch.RenderJob(d, s, device=cuda) for d, s in zip(devs, spp)]
        b = batch.Batch(len(jobs), abi.BatchConfig.make(items_per_fetch=fetch), cuda)
        b.set_jobs(jobs, spp)
        b.launch()
        torch.cuda.synchronize()
        assert int(b.counters[0]) == 5 + 2 * 61 * 7 + 13 * 17
        for d, s, j in zip(devs, spp, jobs):
            alone = batch.RenderJob(d, s, device=cuda)
            if s:
                alone.render_alone()
            torch.cuda.synchronize()
            assert _same(alone.acc, j.acc)


@pytest.mark.parametrize("side", [(1, 1), (8, 8), (1, 64), (5, 13), (3, 43), (12, 37), (61, 67)])
def test_build_and_refit_at_run_edges(cuda, side):
    """2 to 8,174 triangles: around the 128-primitive warp subtrees, the eleven
    top depths and the 296 runs of the area sum; refitted twice."""
    import torch
    pos, idx = blas.terrain_mesh(*side, seed=side[1])
    want, _ = blas.host_build(pos, idx)
    buf, _ = blas.BlasBuilder(len(idx)).build(torch.from_numpy(pos).to(cuda),
                                              torch.from_numpy(idx.view(np.int32)).to(cuda))
    assert buf.cpu().numpy().tobytes() == want.tobytes()
    buf = buf.clone()
    refit = blas.BlasRefit(buf)
    for k in (0.5, 1.75):
        moved = (pos * np.float32(k)).astype(np.float32)
        area = refit.refit(torch.from_numpy(moved).to(cuda)).item()
        boxes, host_area = blas.host_refit(want, moved)
        assert buf.cpu().numpy().tobytes() == boxes.tobytes()
        # sums of n positive float64 terms in two orders: n rounding steps each
        assert abs(area - host_area) <= 2 * len(want) * np.finfo(np.float64).eps * host_area


def test_refit_area_in_one_launch_and_in_two(cuda):
    """Buffers of up to 591 vec4 hold no more nodes than the area sum has runs: it
    is one launch there, two from 592 on, and the same bits."""
    import torch
    pos, idx = blas.terrain_mesh(2, 20, seed=4)
    want, _ = blas.host_build(pos, idx)
    moved = torch.from_numpy((pos * np.float32(1.5)).astype(np.float32)).to(cuda)
    boxes, host_area = blas.host_refit(want, moved.cpu().numpy())
    areas = []
    for vec4 in (len(want) // 4, 588, 589, 590, 591, 592, 593, 700):
        buf = torch.zeros(vec4 * 4, dtype=torch.float32, device=cuda)
        buf[:len(want)] = torch.from_numpy(want.view(np.float32)).to(cuda)
        areas.append(blas.BlasRefit(buf).refit(moved).item())
        assert buf[:len(want)].cpu().numpy().tobytes() == boxes.tobytes()
    assert len(set(areas)) == 1 and abs(areas[0] - host_area) <= 2 * len(want) * np.finfo(np.float64).eps * host_area


def _records(words, ints, node, rel):
    """The leaf records below `node`, and the first vec4 past the subtree
    (right pointers are relative to `rel`)."""
    ptr = int(ints[node, 3])
    if ptr < 0:
        return [words[node + 2 + k].copy() for k in range(-ptr)], node + 2 - ptr
    left, _ = _records(words, ints, node + 2, rel)
    right, end = _records(words, ints, rel + ptr, rel)
    return left + right, end


def _chain(words, ints, node, rel, records, depth):
    """Overwrites the subtree at `node` with a chain: every right child a leaf
    of one record, every left child the rest, the last leaf holding what is
    left; all boxes those of the root, so that a ray takes all left children
    with every right one on the stack."""
    lo, hi = words[node].copy(), words[node + 1].copy()
    inner = [node + 2 * k for k in range(depth + 1)]
    at = inner[-1]
    for k in range(depth, -1, -1):  # the last left child, then right children from the deepest
        rest = records[depth:] if k == depth else records[k:k + 1]
        words[at], words[at + 1] = lo, hi
        ints[at, 3] = -len(rest)
        words[at + 2:at + 2 + len(rest)] = rest
        if k < depth:
            words[inner[k]], words[inner[k] + 1] = lo, hi
            ints[inner[k], 3] = at - rel
        at += 2 + len(rest)
    return at


@pytest.mark.parametrize("level", ["tlas", "blas"])
@pytest.mark.parametrize("depth", [62, 63, 64, 90])
def test_trees_deeper_than_the_traversal_stack(cuda, level, depth):
    """Chains that fill the 64 entries of a level's stack: the nearer child of a
    node that finds one entry left is dropped, as in the reference, and what is
    below it never hit.  Bit-exact against the oracle in every engine."""
    import torch
    host = scene.SceneHost("instanced_spheres", 40, 24, 3, (400, 1, 6, 64, 2))
    rays = oracle_lib.seeded_rays(host, 3000, seed=depth)
    whole = oracle_lib.first_hits(host, rays)
    words = host.bvh.reshape(-1, 4)
    ints = words.view(np.int32)
    if level == "tlas":
        root, rel = 0, 0
    else:
        base = host.uniform.blas_offset
        roots = {(base + int(e[1]), base + int(host.instances.view(np.int32)[int(e[0]) * 40] & 0x3fffffff))
                 for e in (r.view(np.int32) for r in _records(words, ints, 0, 0)[0])}
        root, rel = max(roots, key=lambda r: len(_records(words, ints, *r)[0]))  # the spheres' mesh
    records, end = _records(words, ints, root, rel)
    assert len(records) > depth + 20
    assert _chain(words, ints, root, rel, records, depth) <= end
    want = oracle_lib.first_hits(host, rays)
    got = trace.query_first_hit(scene.DeviceScene(host, cuda), torch.from_numpy(rays).to(cuda)).cpu().numpy()
    same, tie = _hits_equal(got, want)
    assert (same | tie).all()
    fewer = int(want.view(np.int32).reshape(len(rays), -1)[:, 0].sum()) < int(
        whole.view(np.int32).reshape(len(rays), -1)[:, 0].sum())
    assert fewer == (depth >= 64), "the limit is met at the depth it should be"
    dev = scene.DeviceScene(host, cuda)
    plain, one, job = (batch.RenderJob(dev, 2, device=cuda) for _ in range(3))
    plain.render_alone()
    b = batch.Batch(1, device=cuda)
    b.set_jobs([one])
    b.launch()
    sb = batch.StreamBatch(1, stream_config=abi.StreamConfig.make(slots=1024), device=cuda)
    sb.set_jobs([job])
    sb.run()
    torch.cuda.synchronize()
    assert _same(plain.acc, one.acc) and _same(plain.acc, job.acc)
