"""Every gradient lane of every splat against the double oracle, held to what single-precision rounding may move it by. (Relative
norms over whole arrays do not see one bad row among a million, and an optimizer turns the sign of a gradient that nearly
cancels into a whole step.)"""
import numpy as np
import pytest

from b2ctrain_b200 import scenes
from oracle import orc
from tests.test_gpu_kernel_edges import stack_scene
from tests.util import Harness

pytestmark = pytest.mark.gpu

LANES = ("x", "y", "c00", "c01", "c11", "r", "g", "b", "opacity", "refine")


def small_splats(W, H):
    """Splats of less than a pixel: lanes that one or two pixels decide."""
    scene = scenes.make_splats(20000, 1, 5, log_scale=(-7.0, 0.4))
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 30.0, 10.0), W, H, float(H))
    return scenes.floor_for_cameras(scene, [cam]), cam


def needles(W, H):
    """Needles across the image: most of their tiles lie far from their centres, and their conics are nearly singular."""
    scene = scenes.make_splats(400, 1, 6, log_scale=(-5.5, 0.2))
    scene["lscale"][:, 0] = -0.8
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, -60.0, 20.0), W, H, float(H))
    return scenes.floor_for_cameras(scene, [cam]), cam


def wanted(n, W, H, h, v_out, bg, from_totals):
    """Lanes, error bounds and touched splats of the whole-view lists in the harness' context."""
    p0, p1, p2 = (t[:n].cpu().numpy() for t in (h.ctx.proj0, h.ctx.proj1, h.ctx.proj2))
    geo, col = np.concatenate([p0, p1], 1).astype(np.float64), p2[:, :3].astype(np.float64)
    vals, ranges = h.u32(h.ctx.vals_sorted, h.ctx.num_isect), h.u32(h.ctx.tile_ranges)
    rgba, T, last, ranges, _ = orc.raster_fwd(W, H, geo, col, vals, ranges, np.array(bg))
    bound = np.zeros((n, 13))
    want, vis, _ = orc.raster_bwd(n, W, H, geo, col, vals, ranges, np.array(bg), rgba, T, last, v_out, bound=bound, from_totals=from_totals)
    for pix in np.nonzero(last != h.u32(h.ctx.last_idx))[0]:   # another last fragment: on an edge, and with it its tile's list
        tile = (pix // W // 8) * ((W + 7) // 8) + pix % W // 8
        bound[vals[ranges[tile, 0]:ranges[tile, 1]], 10] += 1
    return want, bound, vis


def check(got, want, bound, what):
    sure = bound[:, 10] == 0          # no fragment-pixel on an edge
    assert sure.mean() > 0.5
    for k, lane in enumerate(LANES):
        err = np.abs(got[sure, k] - want[sure, k])
        worst = int(np.argmax(err - bound[sure, k]))
        assert err[worst] <= bound[sure, k][worst], (what, lane, int(np.nonzero(sure)[0][worst]), err[worst], bound[sure, k][worst])


@pytest.mark.parametrize("W,H", [(512, 512), (520, 512)])       # 4,096 and 4,160 tiles: segments of 32 and of 128 fragments
@pytest.mark.parametrize("scene_of", ["small", "needles", 31, 33, 127, 128, 129, 257, 400])
def test_gradient_lanes_per_element(scene_of, W, H):
    scene, cam = small_splats(W, H) if scene_of == "small" else needles(W, H) if scene_of == "needles" else stack_scene(scene_of, W, H)
    n, bg, segments_of_128 = scene["n"], (0.2, 0.1, 0.3), W > 512
    h = Harness(scene, cam, bg=bg)
    h.forward()
    v_out = (np.random.Generator(np.random.PCG64(9)).standard_normal((W * H, 4)) * 1e-3).astype(np.float32)
    v_dev = h.torch.from_numpy(v_out).cuda()
    h.ctx.v_out.copy_(v_dev)
    h.api.rasterize_backward(h.ctx, h.model, h.rp)
    want, bound, _ = wanted(n, W, H, h, v_out, bg, segments_of_128)
    check(h.ctx.v_splat[:n].cpu().numpy().astype(np.float64), want, bound, "whole")
    chunked = h.api.RenderCtx("cuda:0")
    chunked.setup(W, H, h.model.cap, n_chunks=3)
    h.api.render_forward(chunked, h.model, h.rp)
    assert h.torch.equal(chunked.out_rgba, h.ctx.out_rgba)
    chunked.v_out.copy_(v_dev)
    h.api.rasterize_backward(chunked, h.model, h.rp)
    check(chunked.v_splat[:n].cpu().numpy().astype(np.float64), want, bound, "three chunks")


@pytest.mark.parametrize("W,H", [(264, 200), (720, 480)])       # segments of 32 and of 128 fragments
def test_opacity_gradients_of_a_step_of_several_views_per_element(W, H):
    """The accumulator of a step over four views. The opacity row is a fixed multiple of one lane of each view, so its bound is
    that multiple of the lanes' bounds, and a little for the sum over the views."""
    import torch
    from b2ctrain_b200.trainer import Trainer
    scene = scenes.make_splats(30000, 1, 12, log_scale=(-4.0, 0.5))
    cams = [scenes.look_at_camera(scenes.orbit_eye(4.0, a, 10.0), W, H, float(H)) for a in (10.0, 100.0, 190.0, 280.0)]
    scene = scenes.floor_for_cameras(scene, cams)
    n, rng = scene["n"], np.random.Generator(np.random.PCG64(4))
    targets = [torch.from_numpy((rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32) | np.uint32(0xFF000000)).view(np.int32)).cuda() for _ in cams]
    tr = Trainer(scene, W, H, "cuda:0", 0, 1, lr_mean=1e-4, sparse=True)
    total, limit, edge = np.zeros(n), np.zeros(n), np.zeros(n)
    tr.model.adam_t += 1
    for cam, target in zip(cams, targets):
        tr.view_pass(cam, target)
        h = Harness(scene, cam)
        h.forward()
        want, bound, vis = wanted(n, W, H, h, tr.ctx.v_out.cpu().numpy(), (0.0, 0.0, 0.0), W * H > 4096 * 64)
        tiles, ones = np.ones(n, np.uint32), np.zeros((n, 13))
        ones[:, 8] = 1.0
        factor = orc.proj_bwd(scene, cam, ones, vis, tiles)[:, 3]
        total += want[:, 8] * factor
        limit += (bound[:, 8] + 32 * 2.0 ** -24 * np.abs(want[:, 8])) * np.abs(factor)
        edge += bound[:, 10]
    got = tr.grad[:, 3].cpu().numpy().astype(np.float64)
    sure = edge == 0
    assert sure.mean() > 0.5 and np.all(np.abs(got - total)[sure] <= limit[sure])


@pytest.mark.parametrize("chunks", [1, 3])
@pytest.mark.parametrize("W,H", [(512, 512), (520, 512)])       # segments of 32 and of 128 fragments
def test_backward_repeats_on_one_forward(W, H, chunks):
    """Two backwards with different pixel gradients after one forward, the second through the scaled entry: each gives the
    lanes of its own pixel gradients."""
    import ctypes as C
    scene, cam = stack_scene(300, W, H)
    n, bg, rng = scene["n"], (0.2, 0.1, 0.3), np.random.Generator(np.random.PCG64(21))
    h = Harness(scene, cam, bg=bg)
    h.forward()
    ctx = h.api.RenderCtx("cuda:0")
    ctx.setup(W, H, h.model.cap, n_chunks=chunks)
    h.api.render_forward(ctx, h.model, h.rp)
    for scale in (1.0, 8.0, 1.0):
        v_out = (rng.standard_normal((W * H, 4)) * 1e-3).astype(np.float32)
        want, bound, _ = wanted(n, W, H, h, v_out, bg, W > 512)
        ctx.v_out.copy_(h.torch.from_numpy(v_out * np.float32(scale)))
        ctx.v_splat.zero_()
        ctx.vis_flag.zero_()
        cs, ms, opts = ctx.struct(), h.model.struct(), h.rp.struct()
        h.api._check(h.api.lib().b2k_raster_bwd_scaled(C.byref(cs), C.byref(ms), C.byref(opts), C.c_float(scale), h.api._stream(None)), "b2k_raster_bwd_scaled")
        check(ctx.v_splat[:n].cpu().numpy().astype(np.float64), want, bound, scale)


def test_segments_are_long_again_where_short_ones_would_take_too_much_memory():
    """Buffers for more than 2^24 intersections in a small image: checkpoints every 128 fragments, and the same gradients."""
    from b2ctrain_b200 import api
    W = H = 256
    size = lambda cap: api.lib().b2k_bwd_scratch_bytes(W, H, 1, cap)
    assert size(1 << 24) < 600e6 and size((1 << 24) + 1) < 150e6 and size(1 << 25) < 300e6
    scene, cam = stack_scene(300, W, H)
    n, bg = scene["n"], (0.2, 0.1, 0.3)
    v_out = (np.random.Generator(np.random.PCG64(3)).standard_normal((W * H, 4)) * 1e-3).astype(np.float32)
    for cap in (1 << 24, 1 << 25):
        h = Harness(scene, cam, bg=bg, isect_cap=cap)
        h.forward()
        h.ctx.v_out.copy_(h.torch.from_numpy(v_out))
        h.api.rasterize_backward(h.ctx, h.model, h.rp)
        want, bound, _ = wanted(n, W, H, h, v_out, bg, cap > 1 << 24)
        check(h.ctx.v_splat[:n].cpu().numpy().astype(np.float64), want, bound, cap)
