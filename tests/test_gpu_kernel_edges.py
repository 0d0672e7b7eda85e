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


@pytest.mark.parametrize("W,H", [(512, 512), (520, 512)])       # 4,096 and 4,160 tiles: segments of 32 and of 64 fragments
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
