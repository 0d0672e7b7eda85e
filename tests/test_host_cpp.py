"""The C++ host mirror of the reference API (b2ctrain_b200/host): it builds with the host compiler, and its Harness
(the mould of the reference's own test harness, tests/tests.cpp:61-102) reproduces the oracle's loss and gradients."""
import os
import subprocess

import numpy as np
import pytest

from oracle import orc
from tests.util import TOL_GRAD_REL_L2, TOL_IMAGE_ABS, TOL_LOSS_REL, check_against_fd, load_gradcheck, rel_l2

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "b2ctrain_b200", "host")


def build_harness():
    from b2ctrain_b200 import build
    build.build()
    subprocess.run(["make", "-C", HOST], check=True, capture_output=True)
    return os.path.join(HOST, "harness")


def test_host_mirror_builds():
    exe = build_harness()
    assert os.path.exists(exe)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 2 and "usage" in r.stderr


def write_scene(path, scene, cam, gt, wts, lp):
    n, deg = scene["n"], scene["degree"]
    with open(path, "wb") as f:
        np.array([n, deg, cam["W"], cam["H"], int(lp.get("composite", 0)), int(lp.get("mask", 0)), int(lp.get("alpha_lane", 0)),
                  int(wts is not None)], np.int32).tofile(f)
        fl = [cam["fx"], cam["fy"], cam["cx"], cam["cy"], *cam["R"], *cam["t"], *lp.get("bg", (0, 0, 0)), lp.get("l1_w", 0.8),
              lp.get("ssim_w", -0.2), lp.get("match_alpha_weight", 0.1), lp.get("scale", 1.0)]
        np.array(fl, np.float32).tofile(f)
        for a in (scene["pos_op"][:, :3], scene["lscale"][:, :3], scene["quat"], scene["pos_op"][:, 3], scene["lscale"][:, 3], scene["sh"]):
            np.ascontiguousarray(a, np.float32).tofile(f)
        np.ascontiguousarray(gt, np.uint32).tofile(f)
        if wts is not None:
            np.ascontiguousarray(wts, np.uint8).tofile(f)


@pytest.mark.gpu
@pytest.mark.parametrize("mode,chunks", [(0, 1), (1, 1), (1, 3)])
def test_host_harness_matches_oracle_and_reference_golden(mode, chunks, tmp_path):
    exe = build_harness()
    scene, cam, gt, wts, lp, z = load_gradcheck(mode)
    write_scene(tmp_path / "scene.bin", scene, cam, gt, wts, lp)
    r = subprocess.run([exe, str(tmp_path / "scene.bin"), str(tmp_path / "out.bin")] + ([str(chunks)] if chunks > 1 else []), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    raw = open(tmp_path / "out.bin", "rb").read()
    loss = np.frombuffer(raw, np.float64, 1, 0)[0]
    isect, threw = np.frombuffer(raw, np.uint32, 2, 8)
    P, per = cam["W"] * cam["H"], 11 + 3 * (scene["degree"] + 1) ** 2
    img = np.frombuffer(raw, np.float32, P * 4, 16).reshape(P, 4)
    grad = np.frombuffer(raw, np.float32, scene["n"] * per, 16 + P * 16).reshape(scene["n"], per)
    assert threw == 1 and isect > 0
    assert abs(loss - float(z["ref_loss"])) <= TOL_LOSS_REL * abs(float(z["ref_loss"]))
    want = orc.step(scene, cam, np.array(lp["bg"], np.float64), gt, wts, lp, backward=True, want_image=True)
    assert np.max(np.abs(img - want["rgba"])) <= TOL_IMAGE_ABS
    assert rel_l2(grad, want["grad"]) <= TOL_GRAD_REL_L2
    fails, total, _ = check_against_fd(grad, z)
    assert fails == 0 and total > 150


def test_reference_test_harness_compiles_against_the_mirror_headers(tmp_path):
    """The reference's own gradient-test scaffolding (Scene, make_scene and Harness, tests/tests.cpp:22-102), taken from the
    reference checkout at test time and compiled UNCHANGED against the mirror's header set (gpu/render.h, gpu/loss.h,
    gpu/optim.h, model.h, ply.h on the include path), then linked with the host library. Skipped where no reference tree
    is present (nothing of the reference is stored in this repository)."""
    ref = orc.reference_tree()
    if ref is None:
        pytest.skip("no reference checkout here")
    build_harness()
    lines = open(os.path.join(ref, "tests", "tests.cpp")).read().splitlines()
    start = next(i for i, l in enumerate(lines) if l.startswith("struct Scene {"))
    end = next(i for i, l in enumerate(lines) if l.startswith("static float g_eps"))
    body = "\n".join(lines[start:end])
    assert "struct Harness {" in body and "optimizer_step(ctx, model, op, 0);" in body
    src = tmp_path / "ref_harness.cpp"
    src.write_text('#include "gpu/render.h"\n#include "gpu/loss.h"\n#include "gpu/optim.h"\n#include "model.h"\n#include "ply.h"\n#include "gpu/refine.h"\n'
                   '#include "train/evidence.h"\n#include <random>\n#include <cstdio>\n#include <cmath>\n#include <cstdlib>\nusing namespace b2c;\n' + body +
                   "\nint main() { Scene s = make_scene(1, 8); Harness h; h.tc = true; return (int)s.cloud.n - 8; }\n")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    pkg = os.path.join(ROOT, "b2ctrain_b200")
    r = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{HOST}", f"-I{cuda}/include", str(src), "-o", str(tmp_path / "ref_harness"), f"-L{pkg}", "-lb2chost", "-lb2k",
                        f"-L{cuda}/lib64", "-lcudart", f"-Wl,-rpath,{pkg}", f"-Wl,-rpath,{cuda}/lib64"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]


STEP_PROGRAM = r"""
#include "trainer.h"
#include <cstdio>
#include <random>
using namespace b2c;
int main() {
  std::mt19937 rng(7);
  std::uniform_real_distribution<float> u(-1.f, 1.f);
  SplatCloud c; c.resize(100000, 1);
  for (float& p : c.pos) p = u(rng);
  for (float& s : c.log_scale) s = -4.f;
  for (float& s : c.sh) s = 0.5f * u(rng);
  Camera cam; cam.width = 1280; cam.height = 720; cam.fx = cam.fy = 720.f; cam.cx = 640.f; cam.cy = 360.f; cam.t[2] = 4.f; cam.update_pos();
  std::vector<uint32_t> target(1280 * 720, 0xFF808080u);
  StepConfig cfg; cfg.views_in_flight = 1; cfg.isect_cap = 1 << 24; cfg.lr_mean = 1e-4f;
  StepTrainer tr(c, 1280, 720, cfg);
  tr.add_view(cam, target.data());
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return 2;
  int running = 0;
  for (int k = 0; k < 4; k++) { tr.step({0}, s); running += cudaStreamQuery(s) != cudaSuccess; }
  printf("running after step: %d\n", running);
  tr.step_ahead({0}, s);
  tr.settle();
  printf("running after settle: %d\n", (int)(cudaStreamQuery(s) != cudaSuccess));
  return 0;
}
"""


@pytest.mark.gpu
def test_one_view_step_is_complete_when_it_returns(tmp_path):
    """StepTrainer::step of one view leaves nothing on the stream, so that a caller may read the public model at once, in any way."""
    build_harness()
    src, exe = tmp_path / "step.cpp", tmp_path / "step"
    src.write_text(STEP_PROGRAM)
    cuda, pkg = os.environ.get("CUDA_HOME", "/usr/local/cuda"), os.path.join(ROOT, "b2ctrain_b200")
    r = subprocess.run(["g++", "-std=c++17", "-O1", f"-I{HOST}", f"-I{cuda}/include", str(src), "-o", str(exe), f"-L{pkg}", "-lb2chost", "-lb2k", f"-L{cuda}/lib64", "-lcudart",
                        f"-Wl,-rpath,{pkg}", f"-Wl,-rpath,{cuda}/lib64"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split("\n")[:2] == ["running after step: 0", "running after settle: 0"], r.stdout + r.stderr
