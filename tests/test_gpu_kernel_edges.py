"""GPU kernels at the sizes where a variant begins or ends (edges of batches and tiles, remainders, smallest and largest),
each against the oracle or a reference of the same operation."""
import numpy as np
import pytest

from b2ctrain_b200 import scenes
from oracle import orc
from tests.util import Harness, rel_l2

pytestmark = pytest.mark.gpu


def stack_scene(n, W, H, seed=3):
    """n splats one behind the other over the middle of the image: one list of n fragments in the tiles there. Faint, except
    that the last one is opaque enough for the alpha clamp to act."""
    rng = np.random.Generator(np.random.PCG64(seed))
    scene = scenes.make_splats(n, 1, seed)
    scene["pos_op"][:, :2] = rng.normal(0, 0.003, (n, 2))
    scene["pos_op"][:, 2] = np.linspace(0.5, -0.5, n)          # the camera sits at z = +4: the first is the nearest
    scene["pos_op"][:, 3] = -4.0
    scene["pos_op"][-1, 3] = 9.5
    scene["lscale"][:, :3] = rng.normal(-3.2, 0.1, (n, 3))
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), W, H, float(H))
    return scenes.floor_for_cameras(scene, [cam]), cam


@pytest.mark.parametrize("W,H", [(512, 512), (520, 512)])       # 4,096 and 4,160 tiles: segments of 32 and of 128 fragments
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 129])
def test_backward_segments_and_odd_batches(n, W, H):
    scene, cam = stack_scene(n, W, H)
    rng = np.random.Generator(np.random.PCG64(9))
    bg = (0.2, 0.1, 0.3)
    h = Harness(scene, cam, bg=bg)
    h.forward()
    v_out = (rng.standard_normal((W * H, 4)) * 1e-3).astype(np.float32)
    h.ctx.v_out.copy_(h.torch.from_numpy(v_out))
    h.api.rasterize_backward(h.ctx, h.model, h.rp)
    p0, p1, p2 = (t[:n].cpu().numpy() for t in (h.ctx.proj0, h.ctx.proj1, h.ctx.proj2))
    vals = h.u32(h.ctx.vals_sorted, h.ctx.num_isect)
    want, vis, visw = orc.raster_bwd(n, W, H, np.concatenate([p0, p1], 1).astype(np.float64), p2[:, :3].astype(np.float64), vals,
                                     h.u32(h.ctx.tile_ranges).reshape(-1, 2), np.array(bg), h.ctx.out_rgba.cpu().numpy(), h.ctx.out_feat.cpu().numpy()[:, 3],
                                     h.u32(h.ctx.last_idx), v_out)
    got = h.ctx.v_splat[:n].cpu().numpy()
    assert np.array_equal(h.u32(h.ctx.vis_flag, n) != 0, vis != 0) and vis.all()
    for lane in range(10):
        assert rel_l2(got[:, lane], want[:, lane]) <= 5e-5, lane
    assert np.all(got[:, 10:] == 0)
    assert rel_l2(h.model.vis_weight[:n].cpu().numpy(), visw) <= 1e-5


def bin_scene(n, W, H, wide, seed=5):
    scene = scenes.make_splats(n, 0, seed, log_scale=(-3.5, 0.6))
    scene["lscale"][::max(1, n // max(1, wide)), :3] = -0.7 if wide else -3.5      # splats over most of the image
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 25.0, 10.0), W, H, float(max(W, H)))
    return scenes.floor_for_cameras(scene, [cam]), cam


@pytest.mark.parametrize("W,H,n,wide", [(8, 8, 40, 3),             # one tile
                                        (64, 64, 300, 3),          # one bin of 8x8 tiles
                                        (65, 63, 300, 3),          # a ragged second column of bins
                                        (1040, 72, 5000, 200),     # 17x2 bins: in chunks, splats over more bins than a lane walks alone
                                        (3848, 2312, 600, 40)])    # 61x37 bins: two bands of bin rows
def test_binning_at_the_edges_of_bins_and_bands(W, H, n, wide):
    """Tile sets, list order and ranges are bit-exact functions of the records; a chunked view composites the same image."""
    import torch
    scene, cam = bin_scene(n, W, H, wide)
    h = Harness(scene, cam, isect_cap=1 << 23)
    h.api.project_splats(h.ctx, h.model, h.rp)
    h.api.bin_and_sort(h.ctx, h.model)
    tc_o, vals_o, keys_o, ranges_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)
    tc = h.u32(h.ctx.tile_count, n)
    assert np.array_equal(tc, tc_o)
    assert h.ctx.num_isect == len(vals_o) > n // 2
    assert np.array_equal(h.u32(h.ctx.vals_sorted, len(vals_o)), vals_o)
    assert np.array_equal(h.u32(h.ctx.keys_sorted, len(vals_o)), keys_o)
    assert np.array_equal(h.u32(h.ctx.tile_ranges).reshape(-1, 2), ranges_o)
    assert np.array_equal(h.u32(h.ctx.tile_off, n), np.cumsum(tc[h.u32(h.ctx.order, n)], dtype=np.uint32))
    h.api.rasterize_forward(h.ctx, h.rp)
    chunked = h.api.RenderCtx("cuda:0")
    chunked.setup(W, H, h.model.cap, n_chunks=3, isect_cap=1 << 23)
    h.api.render_forward(chunked, h.model, h.rp)
    assert torch.equal(chunked.out_rgba, h.ctx.out_rgba)


def test_binning_with_more_pairs_than_items_of_256_hold():
    """Two and a half million (bin, splat) pairs: level 2 works on longer items. Every splat appears tile_count times, each
    tile's list is in depth order, and the lists fill the ranges."""
    import torch
    W, H, n = 1024, 1024, 60_000
    scene, cam = bin_scene(n, W, H, 0)
    scene["lscale"][:, :3] = -2.2
    h = Harness(scene, cam, isect_cap=1 << 26)
    h.api.project_splats(h.ctx, h.model, h.rp)
    counts = h.ctx.tile_count[:n].clone()
    h.api.bin_and_sort(h.ctx, h.model)
    total = h.ctx.num_isect
    assert total == int(counts.to(torch.int64).sum()) and total > 20_000_000
    vals, keys = h.ctx.vals_sorted[:total].to(torch.int64), h.ctx.keys_sorted[:total].to(torch.int64)
    assert torch.equal(torch.bincount(vals, minlength=n).to(torch.int32), counts)
    rank = torch.empty(n, dtype=torch.int64, device="cuda:0")
    rank[h.ctx.order[:n].to(torch.int64)] = torch.arange(n, device="cuda:0")
    assert bool((torch.diff(keys * n + rank[vals]) > 0).all())
    r = h.ctx.tile_ranges.view(-1, 2).to(torch.int64)
    assert torch.equal(r[:, 1] - r[:, 0], torch.bincount(keys, minlength=h.ctx.n_tiles))


@pytest.mark.parametrize("kind", ["uniform", "wide", "same", "culled", "all_culled", "any_bits"])
@pytest.mark.parametrize("n", [1, 33, 2048, 2049, 8192, 8193, 100_003, 1_300_001])   # one block, one cluster, then many blocks of middle and large tiles
def test_depth_sort_is_stable_at_every_size(n, kind):
    import ctypes as C
    import torch
    from b2ctrain_b200 import api
    g = torch.Generator(device="cuda:0"); g.manual_seed(n)
    u = torch.rand(n, device="cuda:0", generator=g)
    z = {"wide": torch.exp(u * 27.6 - 4.6).clamp(0.01, 1e10), "same": torch.full_like(u, 2.5)}.get(kind, 3 + 2 * u)
    keys = z.view(torch.int32).clone()
    if kind == "any_bits":   # a caller's own keys
        keys = torch.randint(-2 ** 31, 2 ** 31, (n,), device="cuda:0", generator=g, dtype=torch.int64).to(torch.int32)
    if kind in ("culled", "all_culled"):
        keys[u < (0.5 if kind == "culled" else 2.0)] = -1
    ctx = api.RenderCtx("cuda:0"); ctx.setup(64, 64, n)
    ctx.depth_keys_sorted.copy_(keys); ctx.order.copy_(torch.arange(n, dtype=torch.int32)); ctx.tile_count.zero_(); ctx.hit_info.zero_()
    cs = ctx.struct()
    assert api.lib().b2k_bin_sort(C.byref(cs), n, api._stream(None)) == api.B2K_OK
    wide = keys.to(torch.int64) & 0xFFFFFFFF
    want = torch.argsort(wide, stable=True)
    assert torch.equal(ctx.order.to(torch.int64), want) and torch.equal(ctx.depth_keys_sorted.to(torch.int64) & 0xFFFFFFFF, wide[want])


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("W,H", [(1, 1), (8, 5), (53, 4), (54, 9), (55, 12), (108, 3), (163, 37), (16100, 21)])   # one strip, its edge, many; segments of 8 rows and of the whole image
def test_loss_strips(W, H, masked):
    scene, cam = stack_scene(4, W, H)
    rng = np.random.Generator(np.random.PCG64(W * 64 + H))
    gt = rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32)
    wts = rng.integers(64, 256, W * H).astype(np.uint8) if masked else None
    lp = dict(l1_w=0.8, ssim_w=-0.2, bg=(0.2, 0.1, 0.3), composite=not masked, mask=masked, alpha_lane=masked, match_alpha_weight=0.3, scale=1.7, grad_scale=1.0)
    pred = rng.random((W * H, 4)).astype(np.float32)
    h = Harness(scene, cam, gt, wts, lp)
    h.ctx.out_rgba.copy_(h.torch.from_numpy(pred))
    h.ctx.loss_accum.zero_(); h.ctx.v_out.fill_(1e9)
    h.api.photometric_loss(h.ctx, h.view, h.lp)
    f32 = {k: (np.float32(v) if isinstance(v, float) else v) for k, v in lp.items()}
    f32["bg"] = tuple(np.float32(x) for x in lp["bg"])
    want, v_out = orc.loss(W, H, pred, gt, wts, f32)
    assert abs(float(h.ctx.loss_accum[0].item()) - want) <= 2e-5 * abs(want)
    v = h.ctx.v_out.cpu().numpy()
    assert rel_l2(v, v_out) <= 2e-4 and np.max(np.abs(v - v_out)) <= 2e-3 * np.max(np.abs(v_out))


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 100])
def test_forward_groups_and_colours_that_are_not_finite(n):
    W = H = 64
    scene, cam = stack_scene(n, W, H)
    scene["pos_op"][:, 3] = -1.0
    h = Harness(scene, cam, bg=(0.2, 0.1, 0.3), want_depth=True)
    h.forward()
    p0, p1, p2 = (t[:n].cpu().numpy().astype(np.float64) for t in (h.ctx.proj0, h.ctx.proj1, h.ctx.proj2))
    vals, ranges = h.u32(h.ctx.vals_sorted, h.ctx.num_isect), h.u32(h.ctx.tile_ranges).reshape(-1, 2)
    want = orc.raster_fwd(W, H, np.concatenate([p0, p1], 1), p2[:, :3], vals, ranges, np.array((0.2, 0.1, 0.3)), want_depth=True)
    assert rel_l2(h.ctx.out_rgba.cpu().numpy(), want[0]) <= 1e-6
    # An infinite colour shows in the pixels that see the splat and nowhere else.
    images = []
    for colour in (0.0, 1.0, float("inf")):
        h.ctx.proj2[n // 2, 0] = colour
        h.api.rasterize_forward(h.ctx, h.rp)
        images.append(h.ctx.out_rgba.cpu().numpy())
    sees = images[0][:, 0] != images[1][:, 0]
    assert sees.any() and np.all(np.isposinf(images[2][sees, 0])) and np.array_equal(images[2][~sees], images[0][~sees])
    assert np.array_equal(images[2][:, 1:], images[0][:, 1:])


@pytest.mark.parametrize("chunks", [1, 3])
@pytest.mark.parametrize("n", [1, 3, 4, 31, 32, 33, 65])
def test_evidence_rows_and_odd_batches(n, chunks):
    import torch
    from b2ctrain_b200 import api
    from b2ctrain_b200.evidence import Evidence
    W, H = 61, 40
    scene, cam = stack_scene(n, W, H)
    scene["pos_op"][:, 3] = -1.0
    m = api.Model("cuda:0").upload(scene)
    ctx = api.RenderCtx("cuda:0").setup(W, H, n, n_chunks=chunks)
    rng = np.random.Generator(np.random.PCG64(n))
    gt = rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32)
    wts = rng.integers(0, 256, W * H).astype(np.uint8)
    ev = Evidence(m)
    ev.add_view(ctx, cam, api.ViewGPU(torch.from_numpy(gt.view(np.int32)).cuda(), torch.from_numpy(wts).cuda(), W, H))
    p0, p1 = (t[:n].cpu().numpy().astype(np.float64) for t in (ctx.proj0, ctx.proj1))
    vals, ranges = ctx.vals_sorted.cpu().numpy().view(np.uint32), ctx.tile_ranges.cpu().numpy().view(np.uint32).reshape(chunks, -1, 2)
    last, rgba = ctx.last_idx.cpu().numpy().view(np.uint32) & 0x7FFFFFFF, ctx.out_rgba.cpu().numpy().astype(np.float64)
    want = np.zeros((n, 3))
    for y in range(H):
        for x in range(W):
            i, T, a = y * W + x, 1.0, (gt[y * W + x] >> 24) / 255.0
            w = wts[i] / 255.0
            res = sum(abs(rgba[i, c] - ((gt[i] >> np.uint32(8 * c)) & 255) / 255.0) for c in range(3)) / 3.0
            for ch in range(chunks):
                b, e = ranges[ch, (y // 8) * ctx.tiles_x + x // 8]
                for f in range(b, min(e, last[i])):
                    s = vals[f]
                    dx, dy = x + 0.5 - p0[s, 0], y + 0.5 - p0[s, 1]
                    sigma = 0.5 * (p0[s, 2] * dx * dx + p1[s, 0] * dy * dy) + p0[s, 3] * dx * dy
                    if 0.0 <= sigma <= p1[s, 3]:
                        alpha = min(0.999, p1[s, 1] * np.exp(-sigma))
                        want[s] += T * alpha * w * np.array([a, a * res, 1.0])
                        T *= 1.0 - alpha
    assert rel_l2(ev.view_acc.cpu().numpy(), want) <= 1e-4


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("W,H", [(1, 1), (31, 7), (32, 32), (33, 31), (64, 65), (130, 3)])
def test_metrics_tiles(W, H, masked):
    scene, cam = stack_scene(4, W, H)
    rng = np.random.Generator(np.random.PCG64(W * 64 + H))
    gt = rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32)
    pred = rng.uniform(-0.1, 1.1, (W * H, 4)).astype(np.float32)
    h = Harness(scene, cam, gt)
    h.ctx.out_rgba.copy_(h.torch.from_numpy(pred))
    h.ctx.loss_accum.zero_()
    h.api.eval_metrics(h.ctx, h.view, masked)
    got, want = h.ctx.loss_accum[4:6].cpu().numpy(), orc.eval_metrics(W, H, pred, gt, masked)
    assert np.allclose(got, np.array(want[:2], dtype=np.float64), rtol=2e-5, atol=1e-5)


@pytest.mark.parametrize("degree", range(5))
@pytest.mark.parametrize("first,count", [(0, 1), (0, 63), (0, 64), (3, 65), (64, 130)])
def test_model_rows(degree, first, count):
    import ctypes as C
    import torch
    from b2ctrain_b200 import api
    n, K = 200, (degree + 1) ** 2
    scene = scenes.make_splats(n, degree, 5)
    m = api.Model("cuda:0").upload(scene)
    ms = m.struct()
    want = m.download()
    out = [torch.full((count * w + 4,), 7.0).pin_memory() for w in (4, 4, 4, 3 * K)]
    assert api.lib().b2k_model_rows(C.byref(ms), first, count, *[api._ptr(t) for t in out], api._stream(None)) == api.B2K_OK
    torch.cuda.synchronize()
    for t, k in zip(out, ("pos_op", "quat", "lscale", "sh")):
        assert np.array_equal(t[:-4].numpy(), want[k][first : first + count].reshape(-1)) and bool((t[-4:] == 7.0).all())


def test_more_bin_pairs_than_a_word_counts():
    """Three million splats over a whole 4K image: 4.6 billion pairs of (splat, 8x8-tile bin) in the second chunk. The view
    reports that it does not fit, writes nothing outside its buffers, and the context renders an ordinary view afterwards."""
    import ctypes as C
    import torch
    from b2ctrain_b200 import api
    n, W, H = 3_000_000, 3840, 2160
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), W, H, float(H))
    m = api.Model("cuda:0")
    rng = np.random.Generator(np.random.PCG64(2))
    scene = scenes.make_splats(20000, 0, 3)
    big = {k: np.tile(v, (n // 20000,) + (1,) * (v.ndim - 1)) for k, v in scene.items() if hasattr(v, "ndim")}
    big["pos_op"][:, :3] = rng.uniform(-0.1, 0.1, (n, 3))
    big["pos_op"][:, 3] = -4.0
    big["lscale"][:, :3] = 2.0
    m.upload(dict(scene, n=n, **big))
    ctx = api.RenderCtx("cuda:0")
    ctx.setup(W, H, m.cap, isect_cap=1 << 20, n_chunks=2)
    rp = api.RenderParams(cam, sh_degree=0, bwd_info=False)
    api.render_chunked(ctx, m, rp, sync=False)
    total = C.c_uint32(0)
    cs = ctx.struct()
    assert api.lib().b2k_read_num_isect(C.byref(cs), api._stream(None), C.byref(total)) == api.B2K_ERR_OVERFLOW
    assert total.value > 1 << 20
    small = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    fresh = api.RenderCtx("cuda:0")
    fresh.setup(W, H, small.cap, isect_cap=1 << 22, n_chunks=2)
    ctx._alloc_isect(1 << 22)
    for c in (ctx, fresh):
        api.render_chunked(c, small, rp, sync=True)
    assert torch.equal(ctx.out_rgba, fresh.out_rgba) and ctx.num_isect == fresh.num_isect


@pytest.mark.parametrize("chunks", [1, 2, 3])
@pytest.mark.parametrize("W,H", [(2000, 2000), (3001, 2999)])    # one band of bins, and two
def test_lists_fit_into_buffers_of_exactly_their_size(W, H, chunks):
    """Diagonal needles across the image: their boxes overlap more bins than they hit tiles, so that level 1's pairs do not fit
    where the lists do. Buffers of the lists' size hold the view all the same, and the lists are those of larger buffers."""
    import torch
    from b2ctrain_b200 import api
    n = 40
    scene = scenes.make_splats(n, 0, 3)
    rng = np.random.Generator(np.random.PCG64(8))
    scene["pos_op"][:, :3] = rng.uniform(-0.05, 0.05, (n, 3))
    scene["pos_op"][:, 3] = -1.0
    turn = np.deg2rad(45.0 + rng.uniform(-2, 2, n)) / 2 * np.where(np.arange(n) % 2, 1, -1)
    scene["quat"][:] = np.stack([np.cos(turn), 0 * turn, 0 * turn, np.sin(turn)], 1)
    scene["lscale"][:, :3] = [0.0, -9.0, -9.0]
    scene["pos_op"][-1, :] = [0.0, 0.0, 0.3, 1.0]              # and one splat with a mask, in front of them
    scene["lscale"][-1, :3] = -5.0
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), W, H, float(H))
    scene = scenes.floor_for_cameras(scene, [cam])
    m = api.Model("cuda:0").upload(scene)
    rp = api.RenderParams(cam, sh_degree=0, bwd_info=False)
    wide = api.RenderCtx("cuda:0")
    wide.setup(W, H, m.cap, n_chunks=chunks)
    api.render_forward(wide, m, rp)
    hits = wide.num_isect
    exact = api.RenderCtx("cuda:0")
    exact.setup(W, H, m.cap, isect_cap=hits, n_chunks=chunks)
    api.render_forward(exact, m, rp)
    assert exact.isect_cap == hits and exact.num_isect == hits
    assert torch.equal(exact.out_rgba, wide.out_rgba) and torch.equal(exact.tile_ranges, wide.tile_ranges)
    ranges = wide.tile_ranges.cpu().numpy().reshape(-1, 2)
    a, b = exact.vals_sorted.cpu().numpy(), wide.vals_sorted.cpu().numpy()
    assert all(np.array_equal(a[x:y], b[x:y]) for x, y in ranges if y > x)
    less = api.RenderCtx("cuda:0")                              # one too few is still too few
    less.setup(W, H, m.cap, isect_cap=hits - 1, n_chunks=chunks)
    api.render_forward(less, m, rp)
    assert less.isect_cap > hits - 1 and torch.equal(less.out_rgba, wide.out_rgba)


@pytest.mark.parametrize("n", [1, 5, 511, 512, 5000, 70001])
def test_pairs_sort_at_any_word(n):
    """Keys and values that start one word behind a 16-byte boundary."""
    import torch
    from b2ctrain_b200 import api
    rng = np.random.Generator(np.random.PCG64(n))
    keys = rng.integers(0, 2 ** 32, n, dtype=np.uint64).astype(np.uint32) & np.uint32(0xFFFF00FF)
    order = np.argsort(keys, kind="stable")
    for at in (1, 2, 3):
        arrays = [torch.zeros(n + 4, dtype=torch.int32, device="cuda:0")[at:at + n] for _ in range(4)]
        arrays[0].copy_(torch.from_numpy(keys.view(np.int32)))
        arrays[1].copy_(torch.arange(n, dtype=torch.int32))
        size = api.lib().b2k_sort_pairs_tmp_bytes()
        tmp = torch.zeros(size, dtype=torch.uint8, device="cuda:0")
        assert api.lib().b2k_sort_pairs_u32(*[api._ptr(t) for t in arrays], n, api._ptr(tmp), size, api._stream(None)) == api.B2K_OK
        assert np.array_equal(arrays[0].cpu().numpy().view(np.uint32), keys[order]) and np.array_equal(arrays[1].cpu().numpy(), order)


@pytest.mark.parametrize("chunks", [1, 3])
def test_depth_sort_scratch_at_any_word(chunks):
    """The offsets' array, which the depth sort of many splats borrows, one word behind a 16-byte boundary."""
    import torch
    from b2ctrain_b200 import api
    scene = scenes.make_splats(40001, 0, 4)                      # more than one cluster sorts
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 30.0, 10.0), 320, 200, 200.0)
    m = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    images = []
    for at in (0, 1):
        ctx = api.RenderCtx("cuda:0")
        ctx.setup(320, 200, m.cap, n_chunks=chunks)
        ctx.tile_off = torch.zeros(m.cap + 4, dtype=torch.int32, device="cuda:0")[at:at + m.cap]
        api.render_forward(ctx, m, api.RenderParams(cam, sh_degree=0))
        images.append((ctx.out_rgba.clone(), ctx.order[:m.n].clone()))
    assert all(torch.equal(a, b) for a, b in zip(*images))


def test_chunk_words_at_any_word():
    """The alive words of a chunked view, 64 bits each, in an array of 32-bit words that starts at an odd one."""
    import torch
    from b2ctrain_b200 import api
    W, H = 520, 264
    scene = scenes.make_splats(20000, 0, 4, log_scale=(-2.5, 0.5))
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 30.0, 10.0), W, H, 264.0)
    m = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    images = []
    for at in (0, 1):
        ctx = api.RenderCtx("cuda:0")
        ctx.setup(W, H, m.cap, n_chunks=3)
        words = 32 + ctx.n_tiles + (ctx.tiles_x + 1) * (ctx.tiles_y + 1)
        ctx.chunk_words = torch.zeros(words + 2, dtype=torch.int32, device="cuda:0")[at:at + words]
        api.render_forward(ctx, m, api.RenderParams(cam, sh_degree=0))
        images.append((ctx.out_rgba.clone(), ctx.tile_ranges.clone()))
    assert all(torch.equal(a, b) for a, b in zip(*images))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("W,H", [(54, 9), (1001, 300), (3100, 40)])
def test_loss_gradient_at_any_word(W, H, masked):
    """The pixel gradients' array one float behind a 16-byte boundary."""
    rng = np.random.Generator(np.random.PCG64(W))
    scene, cam = stack_scene(4, W, H)
    gt = rng.integers(0, 2 ** 32, W * H, dtype=np.uint64).astype(np.uint32)
    wts = rng.integers(64, 256, W * H).astype(np.uint8) if masked else None
    lp = dict(l1_w=0.8, ssim_w=-0.2, bg=(0.2, 0.1, 0.3), composite=not masked, mask=masked, alpha_lane=masked, match_alpha_weight=0.3, scale=1.7, grad_scale=1.0)
    h = Harness(scene, cam, gt, wts, lp)
    h.ctx.out_rgba.copy_(h.torch.from_numpy(rng.random((W * H, 4)).astype(np.float32)))
    got = []
    for at in (0, 1):
        buffer = h.torch.full((W * H * 4 + 8,), 7.0, device="cuda:0")
        h.ctx.v_out = buffer[at:at + W * H * 4].view(W * H, 4)
        h.ctx.loss_accum.zero_()
        h.api.photometric_loss(h.ctx, h.view, h.lp)
        assert bool((buffer[:at] == 7.0).all()) and bool((buffer[at + W * H * 4:] == 7.0).all())
        got.append((h.ctx.v_out.cpu().numpy(), float(h.ctx.loss_accum[0].item())))
    (a, la), (b, lb) = got
    assert rel_l2(b, a) <= 1e-6 and abs(la - lb) <= 1e-5 * abs(la)


@pytest.mark.parametrize("W,H,n,wide", [(8, 8, 1, 0), (8, 8, 257, 3), (64, 64, 255, 3), (64, 64, 256, 0), (65, 63, 513, 9), (200, 150, 8193, 40),
                                        (512, 512, 5000, 30), (520, 512, 5000, 30), (1000, 24, 4000, 90)])
@pytest.mark.parametrize("room", [True, False])
def test_small_views_walked(W, H, n, wide, room):
    """Whole views of up to 4,096 tiles are binned by walking the ranks for every bin, given room for the hit words; in buffers of just
    the lists' size some take the general distribution. Runs of 256 ranks, one tile, one bin, ragged bins, large boxes."""
    scene, cam = bin_scene(n, W, H, wide, seed=n)
    h = Harness(scene, cam, isect_cap=1 << 22)
    h.api.project_splats(h.ctx, h.model, h.rp)
    tc_o, vals_o, keys_o, ranges_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)
    if not room:
        h.ctx._alloc_isect(len(vals_o))
    for again in range(2):                                     # the second time from keys and an order that are sorted already
        h.api.bin_and_sort(h.ctx, h.model)
        tc = h.u32(h.ctx.tile_count, n)
        assert h.ctx.num_isect == len(vals_o) > 0 and np.array_equal(tc, tc_o)
        assert np.array_equal(h.u32(h.ctx.vals_sorted, len(vals_o)), vals_o) and np.array_equal(h.u32(h.ctx.keys_sorted, len(vals_o)), keys_o)
        assert np.array_equal(h.u32(h.ctx.tile_ranges).reshape(-1, 2), ranges_o)
        assert np.array_equal(h.u32(h.ctx.tile_off, n), np.cumsum(tc[h.u32(h.ctx.order, n)], dtype=np.uint32))


def walked(W, H, n, cap):
    """Whether a whole view is binned by walking the ranks: few tiles, few tests, room for the hit words."""
    tx, ty = -(-W // 8), -(-H // 8)
    bins = -(-tx // 8) * -(-ty // 8)
    units = bins * -(-n // 256)
    return tx * ty <= 4096 and n * bins <= 1 << 20 and units * 65 <= 2048 * 320 and units * 256 <= cap


def shown_lists(vals, ranges, hidden):
    """The oracle's lists without some splats."""
    keep = ~hidden[vals]
    before = np.concatenate([[0], np.cumsum(keep)])
    out = before[ranges]
    out[out[:, 0] == out[:, 1]] = 0
    return vals[keep], out.astype(np.uint32)


@pytest.mark.parametrize("W,H,n,wide", [(8, 8, 40, 0), (64, 64, 300, 1), (65, 63, 300, 2), (1040, 72, 5000, 10), (333, 217, 3000, 5)])
@pytest.mark.parametrize("walk", [True, False])
def test_both_routes_to_small_views(W, H, n, wide, walk):
    """One tile, one bin, ragged bins by the walk and, in buffers of just the lists' size, by the distribution over bins: the same lists, with all
    splats and with some hidden by a tile count of zero."""
    scene, cam = bin_scene(n, W, H, 0, seed=n)
    scene["lscale"][:, :3] = np.log(1.5 / max(W, H))                # half a pixel
    scene["pos_op"][np.arange(n) % 3 != 0, :3] = 2.0 * np.asarray(cam["pos"], np.float32)     # two of three behind the camera
    if wide:
        scene["lscale"][:: 3 * (n // 3 // wide), :3] = -0.7
    h = Harness(scenes.floor_for_cameras(scene, [cam]), cam, isect_cap=1 << 22)
    h.api.project_splats(h.ctx, h.model, h.rp)
    tc_o, vals_o, keys_o, ranges_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)
    if not walk:
        h.ctx._alloc_isect(len(vals_o))
    assert walked(W, H, n, h.ctx.isect_cap) == walk
    hidden = np.zeros(n, bool)
    for _ in range(2):
        h.api.bin_and_sort(h.ctx, h.model)
        vals, ranges = shown_lists(vals_o, ranges_o, hidden)
        tc = np.where(hidden, 0, tc_o)
        assert h.ctx.num_isect == len(vals) > 0 and np.array_equal(h.u32(h.ctx.vals_sorted, len(vals)), vals)
        assert np.array_equal(h.u32(h.ctx.keys_sorted, len(vals)), keys_o[~hidden[vals_o]])
        assert np.array_equal(h.u32(h.ctx.tile_ranges).reshape(-1, 2), ranges)
        assert np.array_equal(h.u32(h.ctx.tile_off, n), np.cumsum(tc[h.u32(h.ctx.order, n)], dtype=np.uint32))
        hidden[::6] = True
        h.ctx.tile_count[:n:6] = 0


@pytest.mark.parametrize("W,H,n", [(64, 64, 256), (64, 64, 300), (120, 64, 700)])
@pytest.mark.parametrize("short", [0, 1, 5000])
def test_walk_of_dense_runs_into_short_buffers(W, H, n, short):
    """Runs whose splats cover their bin (more hits than fit in shared memory) before and behind sparse ones, in buffers of the lists' size and less:
    the total is reported, the lists end with the buffers and nothing behind them is written; grown, they are whole."""
    import ctypes as C
    import torch
    from b2ctrain_b200 import api
    scene, cam = bin_scene(n, W, H, 0, seed=n)
    scene["lscale"][:, :3] = -5.0
    eye = np.asarray(cam["pos"], np.float32)
    near = np.argsort(np.linalg.norm(scene["pos_op"][:, :3] - eye, axis=1))
    scene["lscale"][near[-256:] if n == 300 else near[:400], :3] = -0.5
    h = Harness(scenes.floor_for_cameras(scene, [cam]), cam, isect_cap=1 << 22)
    h.api.project_splats(h.ctx, h.model, h.rp)
    tc_o, vals_o, keys_o, ranges_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)
    cap = len(vals_o) - short
    h.ctx._alloc_isect(cap)
    backing = {k: torch.full((cap + 512,), 7, dtype=torch.int32, device="cuda:0") for k in ("keys", "vals", "keys_sorted", "vals_sorted")}
    for k, t in backing.items():
        setattr(h.ctx, k, t[:cap])
    assert walked(W, H, n, cap) and len(vals_o) > 12_000
    cs, total = h.ctx.struct(), C.c_uint32(0)
    assert api.lib().b2k_bin_sort(C.byref(cs), n, api._stream(None)) == api.B2K_OK
    assert api.lib().b2k_read_num_isect(C.byref(cs), api._stream(None), C.byref(total)) == (api.B2K_ERR_OVERFLOW if short else api.B2K_OK)
    assert total.value == len(vals_o) and all(bool((t[cap:] == 7).all()) for t in backing.values())
    assert np.array_equal(h.u32(h.ctx.vals_sorted), vals_o[:cap]) and np.array_equal(h.u32(h.ctx.keys_sorted), keys_o[:cap])
    assert np.array_equal(h.u32(h.ctx.tile_ranges).reshape(-1, 2), np.minimum(ranges_o, cap))
    h.api.bin_and_sort(h.ctx, h.model)
    assert h.ctx.num_isect == len(vals_o) and np.array_equal(h.u32(h.ctx.vals_sorted, len(vals_o)), vals_o)
    assert np.array_equal(h.u32(h.ctx.tile_ranges).reshape(-1, 2), ranges_o)


def test_chunks_of_wide_splats():
    """Hundreds of splats over most bins in one round of the distribution: shared out over the block's warps."""
    import torch
    W, H, n = 1040, 264, 6000
    scene, cam = bin_scene(n, W, H, 2000)
    scene["pos_op"][:, 3] = -3.0
    h = Harness(scene, cam, isect_cap=1 << 23)
    h.forward()
    for chunks in (2, 3):
        ctx = h.api.RenderCtx("cuda:0")
        ctx.setup(W, H, h.model.cap, n_chunks=chunks, isect_cap=1 << 23)
        h.api.render_forward(ctx, h.model, h.rp)
        assert torch.equal(ctx.out_rgba, h.ctx.out_rgba) and torch.equal(ctx.out_feat[:, 3], h.ctx.out_feat[:, 3])


@pytest.mark.parametrize("n,log_scale", [(3001, (-4.5, 1.6)), (32771, (-5.5, 1.0)), (49153, (-6.0, 1.0)), (262149, (-7.0, 1.1))])
def test_tile_boxes_of_every_size(n, log_scale):
    """The tile tests are shared out over a warp in units of eight tiles of a row: masks up to 64 tiles, counts of larger boxes there or by a
    warp to each."""
    W, H = 1040, 720
    scene = scenes.make_splats(n, 0, 11, log_scale=log_scale)
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 25.0, 10.0), W, H, float(max(W, H)))
    scene = scenes.floor_for_cameras(scene, [cam])
    h = Harness(scene, cam, isect_cap=1 << 23)
    h.api.project_splats(h.ctx, h.model, h.rp)
    tc_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)[0]
    info = h.u32(h.ctx.hit_info[:n]).reshape(-1, 4)
    large = info[:, 2] == 0xFFFFFFFF
    area = np.where(large, (info[:, 1] & 0xFFFF) * (info[:, 1] >> 16), (info[:, 2] >> 24) * info[:, 3])
    assert (area[~large] == 64).any() and (area == 1).any() and ((area > 64) & (area <= 512)).any() and (area > 512).any()
    masks = np.array([bin(int(a)).count("1") + bin(int(b)).count("1") for a, b in info[:, :2]])
    for project in (False, True):
        assert np.array_equal(h.u32(h.ctx.tile_count, n), tc_o)
        assert np.array_equal(masks[~large], tc_o[~large])
        if not project:
            h.ctx.tile_count.zero_(); h.ctx.hit_info.zero_()
            h.api.count_tiles(h.ctx, h.model)
            assert np.array_equal(h.u32(h.ctx.hit_info[:n]).reshape(-1, 4)[tc_o > 0], info[tc_o > 0])


@pytest.mark.parametrize("W,H", [(8, 8), (32, 32), (40, 24), (64, 64), (61, 43), (128, 33)])
@pytest.mark.parametrize("n", [1, 33, 97])
@pytest.mark.parametrize("log_scale", [(-4.0, 0.05), (0.5, 0.2), (-2.0, 1.0)])
def test_tile_boxes_alike(n, W, H, log_scale):
    """Boxes that are all small, or nearly all as large as the largest of the warp, are tested by their own lane."""
    scene = scenes.make_splats(n, 0, n, log_scale=log_scale)
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 25.0, 10.0), W, H, float(max(W, H)))
    h = Harness(scenes.floor_for_cameras(scene, [cam]), cam)
    h.api.project_splats(h.ctx, h.model, h.rp)
    tc_o = orc.bin_sort(h.ctx.proj0[:n].cpu().numpy(), h.ctx.proj1[:n].cpu().numpy(), W, H)[0]
    info = h.u32(h.ctx.hit_info[:n]).reshape(-1, 4)
    masks = np.array([bin(int(a)).count("1") + bin(int(b)).count("1") for a, b in info[:, :2]])
    large = info[:, 2] == 0xFFFFFFFF
    assert np.array_equal(h.u32(h.ctx.tile_count, n), tc_o) and np.array_equal(masks[~large], tc_o[~large])


@pytest.mark.parametrize("W,H", [(64, 64), (61, 43)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 97, 300])
def test_forward_of_few_tiles_is_that_of_chunks(n, W, H):
    """A team of warps to a tile, two warps, and one warp composite the same image bit for bit, whether pixels close inside a group of
    fragments, at its ends or not at all."""
    import torch
    from b2ctrain_b200 import api
    scene, cam = stack_scene(n, W, H, seed=n)
    scene["pos_op"][:, 3] = np.linspace(-4.0, 3.0, n)
    scene["lscale"][:, :3] = np.random.Generator(np.random.PCG64(n)).normal(-2.5, 0.7, (n, 3))
    m = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    got = []
    for chunks in (1, 2, 3):
        ctx = api.RenderCtx("cuda:0")
        ctx.want_depth = True
        ctx.setup(W, H, m.cap, n_chunks=chunks)
        rp = api.RenderParams(cam, bg=(0.2, 0.1, 0.3), sh_degree=1, bwd_info=False)
        api.render_forward(ctx, m, rp)
        plain = [ctx.out_rgba.clone(), ctx.out_feat[:, 3].clone(), ctx.out_depth.clone()]
        rp.feat = "Normals"
        api.render_forward(ctx, m, rp)
        got.append(plain + [ctx.out_rgba.clone(), ctx.out_feat.clone(), ctx.out_depth.clone()])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 500])
@pytest.mark.parametrize("degree,active", [(0, 0), (1, 1), (2, 1), (3, 3), (4, 2), (4, 4)])
def test_accumulator_rows_are_the_gradients(degree, active, n):
    """A view's rows in an accumulator of zeros are the gradients of the debug lane, float for float."""
    import torch
    from b2ctrain_b200 import api
    W, H = 96, 64
    scene = scenes.floor_for_cameras(scenes.make_splats(n, degree, n + degree), [cam := scenes.look_at_camera(scenes.orbit_eye(3.0, 30.0, 10.0), W, H, 64.0)])
    rng = np.random.Generator(np.random.PCG64(n))
    h = Harness(scene, cam)
    h.rp.sh_degree = active
    got = []
    for split in (False, True):
        h.forward()
        h.ctx.v_out.copy_(torch.from_numpy(np.random.Generator(np.random.PCG64(4)).standard_normal((W * H, 4)).astype(np.float32)))
        h.ctx.v_splat.zero_(); h.ctx.vis_flag.zero_()
        h.api.rasterize_backward(h.ctx, h.model, h.rp)
        if not split:
            lanes, flags = h.ctx.v_splat.clone(), h.ctx.vis_flag.clone()
        else:
            h.ctx.v_splat.copy_(lanes); h.ctx.vis_flag.copy_(flags)      # the order of the replay's reductions is not at issue
        grad = torch.zeros((h.model.n, 11 + 3 * h.model.K()), device="cuda:0")
        op = api.OptimParams(cam, active_sh_degree=active, sparse=True, grad_out=None if split else grad)
        (api.projection_backward(h.ctx, h.model, op, grad) if split else api.optimizer_step(h.ctx, h.model, op))
        assert not bool(h.ctx.vis_flag.any()) and not bool(h.ctx.v_splat[:n].any())
        got.append(grad)
    assert bool(got[0].any()) and torch.equal(got[0], got[1])


@pytest.mark.parametrize("kind", ["uniform", "wide", "same", "culled", "any_bits"])
@pytest.mark.parametrize("n", [8191, 16384, 16385, 24577, 32768, 32769])
def test_depth_sort_in_one_cluster(n, kind):
    """Every number of pairs a thread, full and with one left over, and the first size above."""
    test_depth_sort_is_stable_at_every_size(n, kind)


@pytest.mark.parametrize("W,H", [(64, 64), (528, 520), (1361, 900)])   # segments of 32 and of 128 fragments; tiles listed from the first chunk on
@pytest.mark.parametrize("chunks", [2, 3, 5])
@pytest.mark.parametrize("n", [1, 3, 40])
def test_chunks_without_fragments(n, chunks, W, H):
    """Few splats leave the first chunks without any: nothing but background there, and the backward of every pass starts anew."""
    import torch
    scene, cam = stack_scene(n, W, H)
    scene["pos_op"][:, 3] = 1.0
    h = Harness(scene, cam, bg=(0.2, 0.1, 0.3))
    ctx = h.api.RenderCtx("cuda:0")
    ctx.setup(W, H, h.model.cap, n_chunks=chunks)
    v_out = torch.from_numpy(np.random.Generator(np.random.PCG64(4)).standard_normal((W * H, 4)).astype(np.float32))
    for c in (ctx, h.ctx):
        c.out_rgba.fill_(7.0)
    for _ in range(2):
        for c in (ctx, h.ctx):
            h.api.render_forward(c, h.model, h.rp)
            c.v_out.copy_(v_out)
            c.v_splat.zero_(); c.vis_flag.zero_()
            h.api.rasterize_backward(c, h.model, h.rp)
        assert torch.equal(ctx.out_rgba, h.ctx.out_rgba) and torch.equal(ctx.out_feat[:, 3], h.ctx.out_feat[:, 3])
        assert torch.equal(ctx.vis_flag[:n], h.ctx.vis_flag[:n]) and rel_l2(ctx.v_splat[:n].cpu().numpy(), h.ctx.v_splat[:n].cpu().numpy()) <= 2e-5


@pytest.mark.parametrize("bwd_info", [False, True])
@pytest.mark.parametrize("W,H", [(333, 217), (1361, 900)])
def test_depths_of_chunks(W, H, bwd_info):
    """Depths finished by the compositing, by the blocks that visit tiles without fragments in the last chunk, and in a whole view."""
    import torch
    from b2ctrain_b200 import api
    n = 3000
    scene = scenes.make_splats(n, 1, 8, log_scale=(-3.0, 0.8))
    cam = scenes.look_at_camera(scenes.orbit_eye(3.0, 30.0, 10.0), W, H, float(H))
    m = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    rp = api.RenderParams(cam, bg=(0.2, 0.1, 0.3), sh_degree=1, bwd_info=bwd_info)
    got = []
    for chunks in (1, 2, 3, 5):
        ctx = api.RenderCtx("cuda:0")
        ctx.want_depth = True
        ctx.setup(W, H, m.cap, n_chunks=chunks)
        for _ in range(2):
            ctx.out_rgba.fill_(7.0); ctx.out_depth.fill_(7.0)
            api.render_forward(ctx, m, rp)
        got.append((ctx.out_rgba.clone(), ctx.out_depth.clone(), ctx.out_feat[:, 3].clone()))
    assert bool(torch.isfinite(got[0][1]).any()) and bool(torch.isinf(got[0][1]).any())
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("W,H", [(64, 64), (65, 41)])            # and tiles of which one column, one row is on the image
@pytest.mark.parametrize("front", ["none", "faint", "nearly_closed"])
@pytest.mark.parametrize("n", [15, 16, 17, 31, 32, 33, 48])
def test_stacks_of_opaque_splats(n, front, W, H):
    """Splats at the alpha clamp one behind the other over the whole image: the product of a group's transmittances falls below the
    smallest float, and the pixels close at the second one all the same. Whole views of few tiles, and two and three chunks."""
    import torch
    from b2ctrain_b200 import api
    logits = {"none": [], "faint": [-3.0] * 3, "nearly_closed": [-0.277] * 16}[front]     # the last: 1.2e-4 is left in front of the stack
    scene, cam = stack_scene(len(logits) + n, W, H, seed=n)
    scene["pos_op"][:, :2] = 0.0
    scene["pos_op"][:, 3] = logits + [9.5] * n
    scene["lscale"][:, :3] = 4.5                                  # alpha above the clamp of 0.999 in every pixel
    bg = (0.2, 0.1, 0.3)
    h = Harness(scene, cam, bg=bg, want_depth=True)
    h.api.project_splats(h.ctx, h.model, h.rp)
    h.api.bin_and_sort(h.ctx, h.model)
    ranges = h.u32(h.ctx.tile_ranges).reshape(-1, 2).copy()       # before the forward cuts them behind the last fragment taken
    h.api.rasterize_forward(h.ctx, h.rp)
    N, taken = scene["n"], min(len(logits) + 1, 16)
    p0, p1, p2 = (t[:N].cpu().numpy().astype(np.float64) for t in (h.ctx.proj0, h.ctx.proj1, h.ctx.proj2))
    geo, vals = np.concatenate([p0, p1], 1), h.u32(h.ctx.vals_sorted, h.ctx.num_isect)
    assert len(vals) == N * h.ctx.n_tiles
    rgba, T, last, _, zs = orc.raster_fwd(W, H, geo, p2[:, :3], vals, ranges, np.array(bg), want_depth=True)
    assert np.all(last - ranges[:, 0][(np.arange(H) // 8)[:, None] * h.ctx.tiles_x + np.arange(W) // 8].reshape(-1) == taken)
    # In fp32 the clamp lets 1 - 0.999f through, 4.7e-5 more than 0.001: half of that, 4.7e-8, is seen in an image of order one.
    assert rel_l2(h.ctx.out_rgba.cpu().numpy(), rgba) <= 1e-6 and np.array_equal(h.u32(h.ctx.last_idx), last)
    assert rel_l2(h.ctx.out_feat[:, 3].cpu().numpy(), T) <= 1e-4 and rel_l2(h.ctx.out_depth.cpu().numpy(), zs / (1.0 - T)) <= 1e-6
    v_out = (np.random.Generator(np.random.PCG64(9)).standard_normal((W * H, 4)) * 1e-3).astype(np.float32)
    h.ctx.v_out.copy_(torch.from_numpy(v_out))
    h.api.rasterize_backward(h.ctx, h.model, h.rp)
    want, vis, _ = orc.raster_bwd(N, W, H, geo, p2[:, :3], vals, ranges, np.array(bg), h.ctx.out_rgba.cpu().numpy(), h.ctx.out_feat.cpu().numpy()[:, 3], last, v_out)
    assert np.array_equal(h.u32(h.ctx.vis_flag, N) != 0, vis != 0) and vis.sum() == taken
    assert rel_l2(h.ctx.v_splat[:N, 5:8].cpu().numpy(), want[:, 5:8]) <= 1e-4           # colours: weights alone (again 4.7e-5)
    got = []
    for chunks in (1, 2, 3):
        ctx = api.RenderCtx("cuda:0")
        ctx.want_depth = True
        ctx.setup(W, H, h.model.cap, n_chunks=chunks)
        rp = api.RenderParams(cam, bg=bg, sh_degree=1, bwd_info=False)
        api.render_forward(ctx, h.model, rp)
        plain = [ctx.out_rgba.clone(), ctx.out_feat[:, 3].clone(), ctx.out_depth.clone()]
        rp.feat = "Normals"
        api.render_forward(ctx, h.model, rp)
        got.append(plain + [ctx.out_rgba.clone(), ctx.out_feat.clone(), ctx.out_depth.clone()])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a, b)


# All tiles alive behind the first of two chunks: the team's most, evenly over the blocks, as many as fit at once, in several turns; segments of 128.
@pytest.mark.parametrize("W,H", [(37 * 8, 40 * 8), (37 * 8 - 3, 41 * 8), (42 * 8, 42 * 8 - 5), (48 * 8, 37 * 8), (48 * 8, 38 * 8), (71 * 8 - 1, 65 * 8)])
@pytest.mark.parametrize("logit", [-5.0, -1.0])                  # no pixel closes; most close, at different fragments
def test_second_of_two_chunks(W, H, logit):
    import torch
    n = 400
    scene = scenes.make_splats(n, 1, 12, log_scale=(1.5 if logit < -4.0 else -0.3, 0.3))
    scene["pos_op"][:, 3] = logit
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), W, H, float(max(W, H)))
    h = Harness(scenes.floor_for_cameras(scene, [cam]), cam, bg=(0.2, 0.1, 0.3), isect_cap=1 << 22)
    ctx = h.api.RenderCtx("cuda:0")
    ctx.setup(W, H, h.model.cap, n_chunks=2, isect_cap=1 << 22)
    v_out = torch.from_numpy(np.random.Generator(np.random.PCG64(4)).standard_normal((W * H, 4)).astype(np.float32))
    h.rp.bwd_info = False
    for c in (ctx, h.ctx):
        h.api.render_forward(c, h.model, h.rp)
    assert torch.equal(ctx.out_rgba, h.ctx.out_rgba) and torch.equal(ctx.out_feat[:, 3], h.ctx.out_feat[:, 3])
    words = h.u32(ctx.chunk_words, 32)
    assert logit > -5.0 or words[22 + 1] + words[27 + 1] == ctx.n_tiles          # listed, of the second chunk
    h.rp.bwd_info = True
    for c in (ctx, h.ctx):
        h.api.render_forward(c, h.model, h.rp)
        c.v_out.copy_(v_out)
        c.v_splat.zero_(); c.vis_flag.zero_()
        h.api.rasterize_backward(c, h.model, h.rp)
    assert torch.equal(ctx.out_rgba, h.ctx.out_rgba) and torch.equal(ctx.out_feat[:, 3], h.ctx.out_feat[:, 3])
    assert torch.equal(ctx.vis_flag[:n], h.ctx.vis_flag[:n]) and rel_l2(ctx.v_splat[:n].cpu().numpy(), h.ctx.v_splat[:n].cpu().numpy()) <= 2e-5


@pytest.mark.parametrize("W,H", [(168, 136), (200, 150), (333, 217), (296, 256)])     # 357 to 1,184 tiles: between two and eight to an SM of 148
@pytest.mark.parametrize("n,log_scale,team", [(6000, -4.5, True), (3000, 0.5, False), (300, 0.5, False), (40, -5.0, False)])
def test_forward_of_some_tiles_to_an_sm(W, H, n, log_scale, team):
    """A few long lists go to the team, lists that are all alike or short to two warps a tile: the same image as in chunks, bit for bit, and
    the same gradients. The binning leaves the longest list for the choice, by either route."""
    import torch
    from b2ctrain_b200 import api
    scene = scenes.make_splats(n, 1, 21, log_scale=(log_scale, 0.3))
    scene["pos_op"][:, :3] *= 0.3 if team else 1.0
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), W, H, float(H))
    m = api.Model("cuda:0").upload(scenes.floor_for_cameras(scene, [cam]))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    v_out = torch.from_numpy(np.random.Generator(np.random.PCG64(4)).standard_normal((W * H, 4)).astype(np.float32)).cuda()
    got = []
    for chunks, cap in ((1, 1 << 22), (1, None), (3, 1 << 22)):
        ctx = api.RenderCtx("cuda:0")
        ctx.want_depth = True
        ctx.setup(W, H, m.cap, n_chunks=chunks, isect_cap=got[0][0] if cap is None else cap)    # None: of the lists' size, which may take the general route
        rp = api.RenderParams(cam, bg=(0.2, 0.1, 0.3), sh_degree=1, bwd_info=False)
        api.render_forward(ctx, m, rp)
        if chunks == 1:
            r = ctx.tile_ranges.view(-1, 2).to(torch.int64)
            hits, longest = int(ctx.d_num_isect[0].item()), int(ctx.d_num_isect[3].item())
            assert longest == int((r[:, 1] - r[:, 0]).max()) and (longest >= 128 and 2 * hits <= 3 * sms * longest) == team
        images = [ctx.out_rgba.clone(), ctx.out_feat[:, 3].clone(), ctx.out_depth.clone()]
        rp.feat = "Normals"
        api.render_forward(ctx, m, rp)
        images += [ctx.out_rgba.clone(), ctx.out_feat.clone(), ctx.out_depth.clone()]
        rp.feat, rp.bwd_info = "None", True
        api.render_forward(ctx, m, rp)
        images += [ctx.out_rgba.clone(), ctx.out_depth.clone()]
        ctx.v_out.copy_(v_out)
        ctx.v_splat.zero_(); ctx.vis_flag.zero_()
        api.rasterize_backward(ctx, m, rp)
        got.append((ctx.num_isect, images, ctx.vis_flag[:n].clone(), ctx.v_splat[:n].cpu().numpy()))
    for _, images, flags, lanes in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0][1], images))
        assert torch.equal(got[0][2], flags) and rel_l2(got[0][3], lanes) <= 5e-5
