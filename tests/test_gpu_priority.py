"""A plain render leaves its multiprocessors block by block: a call on a stream
of higher priority is let in long before a large render ends."""
import pytest

from mutracer_b200 import batch, scene, trace

pytestmark = pytest.mark.gpu


def test_a_pick_gets_in_during_a_large_render(cuda):
    import torch
    big = batch.RenderJob(scene.DeviceScene(scene.SceneHost("cornell", 1920, 1080, 1), cuda), 8, device=cuda)
    picked = scene.DeviceScene(scene.SceneHost("cornell", 32, 32, 1), cuda)
    rays = torch.zeros((4, 8), device=cuda)
    rays[:, 6] = -1.0
    render, pick = torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-5)
    torch.cuda.synchronize()
    trace.query_first_hit(picked, rays, stream=pick)
    big.render_alone(samples=1, stream=render)
    torch.cuda.synchronize()
    start, end, answered = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    start.record(render)
    big.render_alone(stream=render)
    end.record(render)
    trace.query_first_hit(picked, rays, stream=pick)
    answered.record(pick)
    torch.cuda.synchronize()
    # Three blocks a multiprocessor one after another: the first ends after
    # about a third of the render.
    assert start.elapsed_time(answered) < 0.6 * start.elapsed_time(end)
