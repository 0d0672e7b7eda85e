"""The performance cases of this framework: what its users have it do, from a 64x64 preview to 4K cameras of six million
splats, through the public entry points (the operators of b2ctrain_b200.api, trainer.Trainer / Renderer,
host_trainer.HostTrainer / HostRenderer, evidence.Evidence).

Kinds of case
  step      one single-view optimisation step written over the operators, as the reference's training loop has it: render,
            loss, backward, fused projection backward + sparse Adam (rates late in their decay, so that a state stays what
            it is over many passes)
  batch     one optimisation step over many views (trainer.Trainer: several views in flight, one gradient accumulator, one
            Adam update)
  session   a short fit in the C++ host (HostTrainer): some single-view steps, then the loss and the splats back on the host
  frame     one interactive viewer frame (HostRenderer, one camera in flight): RGBA8 (and depth) in pinned host memory
  orbit     a camera path rendered offline (HostRenderer, four cameras in flight): RGBA8 + depth of each in pinned memory
  image     one camera left on the device (trainer.Renderer), with expected depth, or with the normals lane
  eval      one held-out view rendered and scored (squared error and SSIM sums)
  evidence  one view of the multi-view evidence pass (render, replay, fold)

Scenes follow the repository's synthetic benchmark configurations (means uniform in the unit ball, log-normal scales,
cameras on a radius-4 orbit); targets are renders of the same scene before it is perturbed by N(0, 0.01).
"""
import math

import numpy as np
import torch

from b2ctrain_b200 import api, scenes
from b2ctrain_b200.evidence import Evidence
from b2ctrain_b200.host_trainer import HostRenderer, HostTrainer
from b2ctrain_b200.trainer import Renderer, Trainer

DEVICE = "cuda:0"
LATE = 0.01              # learning rates late in their decay, of the defaults
SESSION_STEPS = 16
ORBIT_LANES = 4          # cameras in flight (bench.py's default)
BATCH_LANES = 8          # views in flight (bench.py's default)


def listed():
    return [
        # The smallest configuration of the benchmark: a preview-sized step, where the host path and launches count.
        dict(name="step_2k_64", kind="step", n=2000, degree=1, W=64, H=64, lane="plain"),
        # A masked object capture at an odd size: weights, mask, alpha lane, composite background.
        dict(name="step_20k_masked_333x217", kind="step", n=20011, degree=2, W=333, H=217, lane="weighted"),
        # The one-view-per-step training configuration (500k splats, 1080p).
        dict(name="step_500k_1080p", kind="step", n=500_000, degree=3, W=1920, H=1080, lane="plain"),
        # The stress configuration: heavy-tailed splats that cover hundreds of tiles, masked loss + alpha lane.
        dict(name="step_1m_heavy_1024", kind="step", n=1_000_000, degree=3, W=1024, H=1024, lane="heavy"),
        # Headline training: views of 1080p over three million splats (16 of the benchmark's 64 views a step).
        dict(name="batch16_3m_1080p", kind="batch", n=3_000_000, degree=3, W=1920, H=1080, views=16),
        # A short fit of a small object, driven by the C++ host.
        dict(name="session_8k_200x150", kind="session", n=8000, degree=2, W=200, H=150),
        # An interactive viewer's frame.
        dict(name="frame_100k_720p", kind="frame", n=100_000, degree=3, W=1280, H=720, depth=False),
        # A turntable rendered to host memory.
        dict(name="orbit8_1m_1080p", kind="orbit", n=1_000_000, degree=3, W=1920, H=1080, views=8),
        # The headline render configuration: one 4K camera of six million SH-4 splats, RGB + alpha + depth.
        dict(name="image_6m_4k_depth", kind="image", n=6_000_000, degree=4, W=3840, H=2160, feat="None"),
        # A normals map for meshing, whole-view binning, ragged size.
        dict(name="image_200k_normals_1001x751", kind="image", n=200_003, degree=1, W=1001, H=751, feat="Normals"),
        # Scoring a held-out view.
        dict(name="eval_300k_1237x822", kind="eval", n=300_000, degree=3, W=1237, H=822),
        # Multi-view evidence after training.
        dict(name="evidence_400k_1080p", kind="evidence", n=400_000, degree=0, W=1920, H=1080),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "session", "frame", "orbit", "image", "eval", "evidence"])
    aspect = rng.choice([1.0, 4 / 3, 3 / 2, 16 / 9])
    top = {"session": 300, "image": 2160}.get(kind, 1080)
    H = _log(rng, 48 if kind in ("step", "session") else 240, top)
    W = max(48, int(round(H * aspect)) + rng.randrange(-7, 8))
    c = dict(kind=kind, degree=rng.randrange(5), W=W, H=H)
    if kind == "step":
        c.update(lane=rng.choice(["plain", "plain", "weighted", "heavy"]), n=_log(rng, 1000, 1_000_000))
    elif kind == "batch":
        c.update(n=_log(rng, 50_000, 2_000_000), views=rng.choice([4, 7, 8, 12, 16]), degree=rng.randrange(1, 4))
    elif kind == "session":
        c.update(n=_log(rng, 1000, 40_000))
    elif kind == "frame":
        c.update(n=_log(rng, 10_000, 1_000_000), depth=rng.random() < 0.5)
    elif kind == "orbit":
        c.update(n=_log(rng, 50_000, 1_000_000), views=rng.choice([4, 5, 8]))
    elif kind == "image":
        c.update(n=_log(rng, 50_000, 4_000_000), feat=rng.choice(["None", "None", "Normals"]))
    else:
        c.update(n=_log(rng, 20_000, 1_000_000))
    return c


def _chunks(n):
    """Depth chunks of the front-to-back renderer by scene size: bench.py's rule."""
    return 5 if n >= 4_000_000 else 4 if n >= 1_000_000 else 2 if n >= 250_000 else 1


def _cameras(case, count, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 17))
    az0 = rng.uniform(0.0, 360.0)
    out = []
    for v in range(count):
        eye = scenes.orbit_eye(4.0, az0 + 360.0 * v / count, rng.uniform(-20.0, 40.0))
        out.append(scenes.look_at_camera(eye, case["W"], case["H"], float(case["H"])))
    return out


def _cloud(case, cams, seed):
    """The host-side splat set (the layout of scenes.make_splats), drawn on the device for speed."""
    n, K = case["n"], (case["degree"] + 1) ** 2
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    normal = lambda *s: torch.randn(s, generator=g, device=DEVICE)
    uniform = lambda *s: torch.rand(s, generator=g, device=DEVICE)
    d = normal(n, 3)
    pos = d / d.norm(dim=1, keepdim=True) * uniform(n, 1) ** (1.0 / 3.0)
    if case.get("lane") == "heavy":     # a tenth of the splats cover hundreds of tiles; opacities bimodal
        ls = torch.where(uniform(n, 1) < 0.1, -1.0 + 0.5 * normal(n, 3), -5.0 + 0.5 * normal(n, 3))
        op = torch.where(uniform(n, 1) < 0.5, 4.0 + 0.5 * normal(n, 1), -4.0 + 0.5 * normal(n, 1))
    else:                               # fewer splats are larger ones: the ball stays covered
        ls = (-4.0 + math.log(max(1.0, (500_000 / n) ** 0.25))) + 0.5 * normal(n, 3)
        op = (1.0 if case["kind"] in ("image", "orbit", "frame") else 0.0) + normal(n, 1)
    q = normal(n, 4)
    q = q / q.norm(dim=1, keepdim=True)
    sh = 0.2 * normal(n, K, 3)
    sh[:, 0, :] += 0.5
    near = torch.full((n,), math.inf, device=DEVICE)   # the 3D-filter floor of the nearest camera
    for c in cams:
        eye = torch.from_numpy(np.asarray(c["pos"], np.float32)).to(DEVICE)
        near = torch.minimum(near, (pos - eye).norm(dim=1) / float(c["fx"]))
    ls = torch.cat([ls, (math.sqrt(0.1) * near)[:, None]], 1)
    host = lambda t: t.contiguous().cpu().numpy()
    return dict(n=n, degree=case["degree"], pos_op=host(torch.cat([pos, op], 1)), quat=host(q), lscale=host(ls), sh=host(sh))


def _perturb(m, seed):
    """Moves the device model away from the scene its targets were rendered from."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed + 7777)
    for t, lanes in ((m.pos_op[: m.n], 4), (m.quat[: m.n], 4), (m.lscale[: m.n], 3), (m.sh_dc[:, : m.n], None)):
        t = t if lanes is None else t[:, :lanes]
        t += 0.01 * torch.randn(t.shape, generator=g, device=DEVICE)


def _context(case, m):
    ctx = api.RenderCtx(DEVICE)
    ctx.want_depth = case["kind"] == "image"
    ctx.setup(case["W"], case["H"], m.cap, n_chunks=_chunks(case["n"]))
    return ctx


def _target(ctx, case):
    """The image in the context as a packed RGBA8 target; a centred ellipse in the alpha byte where the loss is masked."""
    out = torch.zeros(case["W"] * case["H"], dtype=torch.int32, device=DEVICE)
    api.pack_rgba8(ctx.out_rgba.clamp(0.0, 1.0), out, alpha_override=255)
    if case.get("lane", "plain") != "plain":
        inside = torch.from_numpy(scenes.ellipse_mask(case["W"], case["H"]).astype(np.int32)).to(DEVICE) > 0
        out = torch.where(inside, out, torch.zeros_like(out))
    return out


def _view(ctx, case, seed):
    weights = None
    if case.get("lane") == "weighted":
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed + 5)
        weights = torch.randint(64, 256, (case["W"] * case["H"],), generator=g, device=DEVICE, dtype=torch.uint8)
    return api.ViewGPU(_target(ctx, case), weights, case["W"], case["H"])


class _State:
    """What a user's program keeps; closes the C++ host's handle with it."""

    def __init__(self, case, **kw):
        self.case = case
        self.handle = None
        self.__dict__.update(kw)

    def __del__(self):
        if self.handle is not None:
            self.handle.close()


def prepare(case, seed):
    kind = case["kind"]
    cams = _cameras(case, case.get("views", 1), seed)
    cloud = _cloud(case, cams, seed)
    W, H, chunks = case["W"], case["H"], _chunks(case["n"])
    cap = 1 << 24 if case["n"] >= 250_000 else 0
    if kind in ("frame", "orbit"):
        depth = case.get("depth", True)
        r = HostRenderer(cloud, W, H, depth=depth, render_chunks=chunks, lanes=ORBIT_LANES if kind == "orbit" else 1, isect_cap=cap)
        pinned = lambda dtype: [torch.zeros((H, W), dtype=dtype, pin_memory=True) for _ in cams]
        return _State(case, handle=r, cams=cams, rgba=pinned(torch.int32), depth=pinned(torch.float32) if depth else [])
    if kind == "image":
        r = Renderer(cloud, W, H, DEVICE, render_chunks=chunks, isect_cap=cap or None)
        rp = api.RenderParams(cams[0], sh_degree=case["degree"], bwd_info=False)
        rp.feat = case["feat"]
        api.render_forward(r.ctx, r.model, rp)          # sizes the intersection buffers
        return _State(case, r=r, cam=cams[0], rp=rp)
    if kind == "batch":
        t = Trainer(cloud, W, H, DEVICE, lr_mean=1e-7, noise_weight=5e-6, noise_clamp=0.02, isect_cap=cap or None, views_in_flight=min(BATCH_LANES, len(cams)),
                    render_chunks=chunks)
        targets = []
        for cam in cams:
            api.render_forward(t.ctx, t.model, api.RenderParams(cam, sh_degree=case["degree"]))
            targets.append(_target(t.ctx, case))
        _perturb(t.model, seed)
        return _State(case, t=t, cams=cams, targets=targets)
    if kind == "session":
        m = api.Model(DEVICE).upload(cloud)
        ctx = _context(case, m)
        api.render_forward(ctx, m, api.RenderParams(cams[0], sh_degree=case["degree"]))
        target = _target(ctx, case).cpu().numpy()
        _perturb(m, seed)
        rates = {k: LATE * v for k, v in dict(lr_mean=1.6e-4, lr_rot=2e-3, lr_scale=5e-3, lr_opac=0.012, lr_dc=2e-3, lr_sh_rest=2e-4).items()}
        h = HostTrainer(m.download(), W, H, views_in_flight=1, render_chunks=chunks, **rates)
        h.add_view(cams[0], target)
        return _State(case, handle=h)
    # step, eval, evidence: the operators on a model and a context
    m = api.Model(DEVICE).upload(cloud)
    ctx = _context(case, m)
    rp = api.RenderParams(cams[0], sh_degree=case["degree"], bwd_info=kind != "eval")
    api.render_forward(ctx, m, rp)                      # sizes the intersection buffers
    view = _view(ctx, case, seed)
    _perturb(m, seed)
    if kind == "evidence":
        return _State(case, m=m, ctx=ctx, cam=cams[0], view=view, ev=Evidence(m, DEVICE))
    lane = case.get("lane", "plain")
    lp = api.LossParams()
    if lane != "plain":
        lp = api.LossParams(mask=True, alpha_lane=True, composite=lane == "weighted", bg=(0.2, 0.1, 0.3) if lane == "weighted" else (0.0, 0.0, 0.0), scale=2.5)
        rp.bg = lp.bg
    op = api.OptimParams(cams[0], active_sh_degree=case["degree"], t=0, lr_mean=LATE * 1.6e-4, lr_rot=LATE * 2e-3, lr_scale=LATE * 5e-3, lr_opac=LATE * 0.012,
                         lr_dc=LATE * 2e-3, lr_sh_rest=LATE * 2e-4, noise_weight=5e-6, noise_clamp=0.02, sparse=True)
    return _State(case, m=m, ctx=ctx, rp=rp, view=view, lp=lp, op=op)


def _model_state(m):
    """Parameters, moments and statistics of the device model: what a step leaves behind."""
    return {k: getattr(m, k) for k in ("pos_op", "quat", "lscale", "sh_dc", "sh_hi", "m_pos_op", "v_pos_op", "m_quat", "v_quat", "m_lscale", "v_lscale", "m_sh_dc",
                                       "m_sh_hi", "v_sh", "refine_norm", "max_screen", "vis_count", "vis_weight", "last_step")}


def run(s):
    kind = s.case["kind"]
    if kind == "step":
        s.op.t += 1
        s.op.step += 1
        api.step_begin(s.ctx)
        api.render_forward(s.ctx, s.m, s.rp, sync=False)
        api.photometric_loss(s.ctx, s.view, s.lp)
        api.accumulate_loss(s.ctx)
        api.rasterize_backward(s.ctx, s.m, s.rp)
        api.optimizer_step(s.ctx, s.m, s.op)
        return dict(_model_state(s.m), image=s.ctx.out_rgba, loss=s.ctx.loss_accum)
    if kind == "batch":
        loss = s.t.step(s.cams, s.targets)
        return dict(_model_state(s.t.model), loss=loss)
    if kind == "session":
        stream = torch.cuda.current_stream().cuda_stream
        for _ in range(SESSION_STEPS):
            s.handle.step([0], stream)
        loss = s.handle.read_loss(stream)
        splats = s.handle.download()
        return dict(loss=loss, **{k: splats[k] for k in ("pos_op", "quat", "lscale", "sh")})
    if kind in ("frame", "orbit"):
        stream = torch.cuda.current_stream().cuda_stream
        for i, cam in enumerate(s.cams):
            s.handle.render(cam, stream, host_rgba8=s.rgba[i].data_ptr(), host_depth=s.depth[i].data_ptr() if s.depth else None)
        s.handle.finish()
        return s.rgba + s.depth
    if kind == "image":
        if s.case["feat"] != "None":
            api.render_forward(s.r.ctx, s.r.model, s.rp, sync=False)
            return s.r.ctx.out_rgba, s.r.ctx.out_depth, s.r.ctx.out_feat
        return s.r.render(s.cam)
    if kind == "eval":
        api.step_begin(s.ctx)
        api.render_forward(s.ctx, s.m, s.rp, sync=False)
        api.eval_metrics(s.ctx, s.view)
        return s.ctx.out_rgba, s.ctx.loss_accum
    s.ev.add_view(s.ctx, s.cam, s.view)
    return s.ev.acc, s.ev.view_acc


def work(case):
    """What a pass cannot do without. Every splat's geometry is read once (pos_op, quat, lscale), and every splat's colour
    coefficients once where it can be seen; images, targets and updated splats move once. A view leaves about one touched
    splat for sixteen pixels and evaluates about forty fragments a pixel in the benchmark scenes (measured there)."""
    n, P, K, kind = case["n"], case["W"] * case["H"], (case["degree"] + 1) ** 2, case["kind"]
    views = case.get("views", 1)
    lanes = 11 + 3 * K
    touched = min(n, P // 16)
    splats, project = n * (48 + 12 * K), n * (250 + 6 * K)
    forward = P * 40 * 24
    train = P * (40 * 90 + 3 * 400)
    update = touched * (lanes * 12 + 100)   # parameters, first moments written; moments read; second moments
    if kind == "step":
        return dict(bytes=splats + update + P * 20, flops=project + forward + train + touched * 20 * lanes)
    if kind == "batch":
        seen = min(n, views * touched)
        return dict(bytes=splats + seen * (lanes * 12 + 100) + views * P * 4, flops=views * (project + forward + train) + seen * 20 * lanes)
    if kind == "session":
        return dict(bytes=SESSION_STEPS * (splats + update + P * 4) + n * (48 + 12 * K), flops=SESSION_STEPS * (project + forward + train + touched * 20 * lanes))
    if kind in ("frame", "orbit"):
        return dict(bytes=views * (splats + P * (8 if case.get("depth", True) else 4)), flops=views * (project + forward))
    if kind == "image":
        return dict(bytes=splats + P * (20 if case["feat"] == "None" else 36), flops=project + forward)
    if kind == "eval":
        return dict(bytes=splats + P * 20, flops=project + forward + P * 3 * 130)
    return dict(bytes=splats + n * (32 + 32 + 12 + 12) + P * 4, flops=project + 2 * forward)


def tolerance(case):
    """Images are sums of fp32 products in a fixed order, quantised images and counts derive from them. Gradients are fp32
    sums over hundreds of pixels in no fixed order, of terms with both signs; Adam turns them into steps whose sign is
    that of the gradient, so a parameter may differ by one step where a gradient cancels to nothing. A fragment on the
    edge of the 1/255 opacity cut, or a pixel on the edge of the transmittance stop, may fall either way."""
    if case["kind"] in ("step", "batch", "session"):
        return {"rel": 5e-5, "max": 2e-2, "differ": 1e-5}
    if case["kind"] in ("frame", "orbit", "image"):
        return {"rel": 1e-5, "max": 5e-3, "differ": 1e-5}
    return {"rel": 1e-5, "max": 5e-3}
