"""Lanes of one persistent launch that go from job to job of unlike kinds:
opaque, alpha-covered and dispersive scenes, so that a warp holds lanes with
and without coverage draws and a lane's job changes under way.  Each image is
bit-identical to the job's own, and to the wavefront engine's."""
import ctypes as C

import pytest

from mutracer_b200 import abi, batch, scene
from tests.test_gpu_alpha import alpha_room, decode

pytestmark = pytest.mark.gpu
PARTS = ("color", "normal", "albedo", "catcher")


def _same(a, b):
    import torch
    return all(torch.equal(getattr(a, k), getattr(b, k)) for k in PARTS)


@pytest.fixture(scope="module")
def scenes(cuda):
    hosts = [decode(alpha_room(41, 23)), scene.SceneHost("cornell", 37, 29, 2),
             scene.SceneHost("glass_spheres", 19, 11, 4, (4,)), decode(alpha_room(9, 31))]
    return [scene.DeviceScene(h, cuda) for h in hosts], [3, 4, 1, 2]


@pytest.fixture(scope="module")
def alone(cuda, scenes):
    import torch
    jobs = [batch.RenderJob(d, s, device=cuda) for d, s in zip(*scenes)]
    for j in jobs:
        j.render_alone()
    torch.cuda.synchronize()
    return jobs


# One block of one warp an SM hands every lane several jobs; tiles of one
# pixel's width put unlike jobs side by side in a warp.
@pytest.mark.parametrize("cfg", [(0, 0, 0, 0), (32, 1, 1, 16), (128, 8, 4, 3)])
def test_unlike_jobs_share_a_persistent_launch(cuda, scenes, alone, cfg):
    import torch
    devs, spp = scenes
    order = [0, 1, 2, 3, 1, 0]
    jobs = [batch.RenderJob(devs[k], spp[k], device=cuda) for k in order]
    b = batch.Batch(len(jobs), abi.BatchConfig.make(*cfg), cuda)
    b.set_jobs(jobs)
    b.launch()
    torch.cuda.synchronize()
    for k, j in zip(order, jobs):
        assert _same(alone[k].acc, j.acc), k


def test_unlike_jobs_agree_in_the_other_engines(cuda, scenes, alone):
    import torch
    devs, spp = scenes
    jobs = [batch.RenderJob(d, s, device=cuda) for d, s in zip(devs, spp)]
    sb = batch.StreamBatch(len(jobs), stream_config=abi.StreamConfig.make(slots=1024), device=cuda)
    sb.set_jobs(jobs)
    sb.run()
    fixed = [batch.RenderJob(d, s, device=cuda) for d, s in zip(devs, spp)]
    descs = (abi.JobDesc * len(fixed))(*[j.desc(j.spp) for j in fixed])
    abi.check(abi.lib().mtc_trace_batch_noalloc(descs, len(fixed), None, None, None,
                                                C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    for want, a, b in zip(alone, jobs, fixed):
        assert _same(want.acc, a.acc) and _same(want.acc, b.acc)


@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("threads", [32, 64, 96, 128])
def test_blocks_of_a_given_size_trace_both_layouts(cuda, threads, layout):
    """A host's own block sizes run kernels of their own, in both batched
    entry points: ragged images, with the default and with more blocks an SM
    than fit one."""
    import torch
    host = scene.SceneHost("instanced_spheres", 75, 46, 3, (24, 3, 4, 64, 2))
    if layout:
        host.set_blas_layout(layout)
    dev = scene.DeviceScene(host, cuda)
    want = batch.RenderJob(dev, 2, device=cuda)
    want.render_alone()
    for ctas in (0, 32):
        cfg = abi.BatchConfig.make(threads, 4, ctas, 2)
        job, fixed = batch.RenderJob(dev, 2, device=cuda), batch.RenderJob(dev, 2, device=cuda)
        b = batch.Batch(1, cfg, cuda)
        b.set_jobs([job])
        b.launch()
        descs = (abi.JobDesc * 1)(fixed.desc(2))
        abi.check(abi.lib().mtc_trace_batch_noalloc(descs, 1, C.byref(cfg), None, None,
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        assert _same(want.acc, job.acc) and _same(want.acc, fixed.acc), ctas


@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("size", [(24, 24), (199, 150), (251, 240), (300, 291), (1007, 701), (1403, 901)])
def test_plain_kernels_of_every_block_size(cuda, size, layout):
    """One warp a pixel, then blocks of up to 8, 16 and 32 warps and several a
    multiprocessor: the image of the batched kernel, every pixel once."""
    import torch
    host = scene.SceneHost("instanced_spheres", *size, 3, (24, 3, 4, 64, 2))
    if layout:
        host.set_blas_layout(layout)
    dev = scene.DeviceScene(host, cuda)
    plain, job = batch.RenderJob(dev, 2, device=cuda), batch.RenderJob(dev, 2, device=cuda)
    plain.render_alone()
    b = batch.Batch(1, device=cuda)
    b.set_jobs([job])
    b.launch()
    torch.cuda.synchronize()
    assert (plain.acc.normal[:, 3] == 2).all()
    assert _same(plain.acc, job.acc)


@pytest.mark.parametrize("layout", [0, 2])
@pytest.mark.parametrize("sizes", [[(1, 1)], [(7, 5), (3, 9)], [(24, 24)], [(37, 29)] * 3, [(61, 47)],
                                   [(199, 150), (64, 33)], [(300, 130)]])
def test_tables_of_few_pixels(cuda, sizes, layout):
    """One pixel a block, slices of every size, and the first table that is not
    spread: each image that of its own launch, with any number of items a fetch,
    in a captured launch that then runs another table, and over fixed scratch."""
    import torch
    jobs, want = [], []
    for k, (w, h) in enumerate(sizes):
        host = scene.SceneHost("instanced_spheres", w, h, 3 + k, (24, 3, 4, 64, 2))
        if layout:
            host.set_blas_layout(layout)
        dev = scene.DeviceScene(host, cuda)
        jobs.append(batch.RenderJob(dev, 2 + k, device=cuda))
        want.append(batch.RenderJob(dev, 2 + k, device=cuda))
        want[-1].render_alone()

    def check(run):
        for j in jobs:
            j.acc.zero_()
        torch.cuda.synchronize()
        run()
        torch.cuda.synchronize()
        for a, b in zip(want, jobs):
            assert (a.acc.normal[:, 3] == a.spp).all() and _same(a.acc, b.acc)

    for cfg in ((0, 0, 0, 0), (0, 2, 0, 16), (0, 32, 2, 3)):
        b = batch.Batch(len(jobs), abi.BatchConfig.make(*cfg), cuda)
        b.set_jobs(jobs)
        check(b.launch)
    b = batch.Batch(len(jobs), device=cuda)
    b.set_jobs(jobs[:1])
    b.capture()
    b.set_jobs(jobs)
    check(b.replay)
    descs = (abi.JobDesc * len(jobs))(*[j.desc(j.spp) for j in jobs])
    check(lambda: abi.check(abi.lib().mtc_trace_batch_noalloc(
        descs, len(jobs), None, None, None, C.c_void_p(torch.cuda.current_stream().cuda_stream))))
