"""How the library's launches reach the GPU: in a captured graph, and whether any was refused with its attribute. Collected
near the end on purpose: the last test looks back on every launch of the run."""
import numpy as np
import pytest

from b2ctrain_b200 import scenes
from tests.util import Harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [1, 3])
def test_step_in_a_captured_graph(chunks):
    """A training step captured once and replayed twice on other targets equals the steps outside a graph."""
    import torch
    from b2ctrain_b200 import api
    W, H = 200, 120
    scene = scenes.make_splats(5000, 1, 8, log_scale=(-3.0, 0.5))
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 40.0, 10.0), W, H, 120.0)
    scene = scenes.floor_for_cameras(scene, [cam])
    rng = np.random.Generator(np.random.PCG64(6))
    targets = [torch.from_numpy((rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32) | np.uint32(0xFF000000)).view(np.int32)).cuda() for _ in range(2)]
    results = []
    for graphed in (False, True):
        m = api.Model("cuda:0").upload(scene)
        ctx = api.RenderCtx("cuda:0")
        ctx.setup(W, H, m.cap, n_chunks=chunks)
        rp, lp = api.RenderParams(cam, sh_degree=1), api.LossParams()
        grads = torch.zeros((m.n, 11 + 12), device="cuda:0")
        op = api.OptimParams(cam, active_sh_degree=1, t=1, grad_out=grads)
        view = api.ViewGPU(targets[0].clone(), None, W, H)

        def step():
            api.step_begin(ctx)
            api.render_forward(ctx, m, rp, sync=False)
            api.photometric_loss(ctx, view, lp)
            api.accumulate_loss(ctx)
            api.rasterize_backward(ctx, m, rp)
            api.optimizer_step(ctx, m, op)

        step()
        run, graph = step, None
        if graphed:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step()
            run = graph.replay
        out = []
        for t in targets:
            view.rgba.copy_(t)
            grads.zero_()
            run()
            torch.cuda.synchronize()
            out.append((grads.cpu().numpy(), ctx.loss_accum.cpu().numpy(), ctx.out_rgba.cpu().numpy()))
        results.append(out)
    for (ga, la, ia), (gb, lb, ib) in zip(*results):
        assert np.linalg.norm(ga - gb) <= 1e-5 * np.linalg.norm(ga) and abs(la[2] - lb[2]) <= 1e-5 * abs(la[2]) and np.array_equal(ia, ib)


def test_no_launch_was_repeated():
    from b2ctrain_b200 import api
    from tests.test_gpu_kernel_edges import stack_scene
    scene, cam = stack_scene(100, 64, 64)
    Harness(scene, cam).forward()
    assert api.lib().b2k_launches_repeated() == 0
