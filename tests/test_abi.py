"""CPU tests of the drop-in boundary: the C-ABI library loads and exports every symbol include/b2k.h declares, and
argument validation answers with a status instead of touching a device."""
import ctypes as C
import os
import re

import pytest

from b2ctrain_b200 import api, build, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    build.build()
    return api.lib()


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "b2k.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b2k_[a-z0-9_]+)\s*\(", text)))


def test_header_and_binding_table_agree():
    assert declared_symbols() == sorted(api.SIGNATURES)


def test_every_declared_symbol_is_exported(lib):
    for name in declared_symbols():
        assert hasattr(lib, name), name


def test_status_strings(lib):
    assert lib.b2k_error_string(api.B2K_OK) == b"ok"
    assert b"overflow" in lib.b2k_error_string(api.B2K_ERR_OVERFLOW)
    assert lib.b2k_version().startswith(b"b2k")


def test_null_arguments_are_rejected_without_a_device(lib):
    assert lib.b2k_project(None, None, None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_bin_sort(None, 0, None) == api.B2K_ERR_ARG
    assert lib.b2k_raster_fwd(None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_loss_photometric(None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_raster_bwd(None, None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_optim_fused(None, None, None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_adam(None, None, None, None) == api.B2K_ERR_ARG
    assert lib.b2k_adam_range(None, None, None, 0, 0, None) == api.B2K_ERR_ARG
    assert lib.b2k_render_chunked(None, None, None, None, None) == api.B2K_ERR_ARG
    one_chunk = api.B2kCtx(); one_chunk.n_chunks = 1   # the chunked renderer wants 2 to 5 chunks
    assert lib.b2k_render_chunked(C.byref(api.B2kModel()), C.byref(api.B2kCamera()), C.byref(api.B2kRenderOpts()), C.byref(one_chunk), None) == api.B2K_ERR_ARG
    m = api.B2kModel(); m.n, m.cap, m.degree = 4, 2, 1   # cap < n
    assert lib.b2k_project(C.byref(m), C.byref(api.B2kCamera()), C.byref(api.B2kRenderOpts()), C.byref(api.B2kCtx()), None) == api.B2K_ERR_ARG
    assert lib.b2k_sort_tmp_bytes(1000, 1 << 22) > 0


def test_unsupported_lanes_raise():
    rp = api.RenderParams(dict(), sh_degree=1)
    rp.hollow_z = object()
    with pytest.raises(RuntimeError, match="unsupported lane"):
        rp.struct()
    with pytest.raises(RuntimeError, match="unsupported lane"):
        api.OptimParams(dict(), frozen=True).struct()
    with pytest.raises(RuntimeError, match="unsupported lane"):
        api.LossParams(normal_scale=0.5).struct(api.ViewGPU(None))


def test_records_follow_tensors_whose_storage_changes_in_place():
    """A tensor of a model or context may get other memory without being set anew (Tensor.data, set_, resize_, the instance's
    dictionary): the record of the next call has its present address."""
    import torch
    m, ctx = api.Model("cpu"), api.RenderCtx("cpu")
    m.upload(scenes.make_splats(100, 1, 1))
    ctx.setup(64, 48, m.cap)
    for owner, name, field in ((m, "pos_op", "pos_op"), (m, "sh_hi", "sh_hi"), (ctx, "v_out", "v_out"), (ctx, "d_num_isect", "num_isect"), (ctx, "sort_tmp", "sort_tmp")):
        t = getattr(owner, name)
        assert getattr(owner.struct(), field) == t.data_ptr()
        t.data = torch.zeros_like(t)
        assert getattr(owner.struct(), field) == t.data_ptr()
        t.set_(torch.zeros_like(t))
        assert getattr(owner.struct(), field) == t.data_ptr()
        t.resize_(t.numel() * 64)
        assert getattr(owner.struct(), field) == t.data_ptr()
        vars(owner)[name] = torch.zeros_like(t)
        assert getattr(owner.struct(), field) == vars(owner)[name].data_ptr()
    assert ctx.struct().sort_tmp_bytes == ctx.sort_tmp.numel()


def test_records_take_what_an_assignment_takes():
    """Values that a native-layout pack refuses: floats beyond single precision, integers beyond 32 bits, numbers as text."""
    import math
    import numpy as np
    cam = scenes.look_at_camera((0.0, 0.0, 4.0), 64, 48, 60.0)
    plain = api.camera_from(cam)
    odd = api.camera_from(dict(cam, fx="60.0", lim_pos_x=1e39, lim_neg_y=-1e300, W="64", R=[np.float64(x) for x in np.asarray(cam["R"]).reshape(-1)]))
    assert odd.fx == plain.fx and odd.lim_pos_x == math.inf and odd.lim_neg_y == -math.inf and odd.W == 64 and list(odd.R) == list(plain.R) and list(odd.pos) == list(plain.pos)
    op = api.OptimParams(cam, t=2 ** 31 + 5, seed=-3, step=2 ** 32 + 7, lr_mean=1e40, active_sh_degree=2).struct()
    assert op.t == 5 - 2 ** 31 and op.seed == 2 ** 32 - 3 and op.step == 7 and op.lr_mean == math.inf and op.active_sh_degree == 2 and op.sparse in (0, 1)
    rp = api.RenderParams(cam, bg=(1e39, "0.5", np.float32(0.25)), sh_degree=3).struct()
    assert list(rp.bg) == [math.inf, 0.5, 0.25] and rp.sh_degree == 3 and not rp.pos_override
    lp = api.LossParams(scale=1e39, bg=(0.25, 0.5, 1.0), mask=True)

    class View:
        rgba = weights = None

    ls = lp.struct(View)
    assert ls.scale == math.inf and list(ls.bg) == [0.25, 0.5, 1.0] and ls.mask == 1 and not ls.rgba
    with pytest.raises(TypeError):
        api.LossParams(scale="1").struct(View)


def test_rows_of_the_model_need_aligned_outputs(lib):
    """b2k_model_rows writes 16 bytes at a time: an output at another address is an argument error, not a fault."""
    import torch
    m = api.Model("cpu").upload(scenes.make_splats(8, 1, 1))
    ms = m.struct()
    out = [torch.zeros(8 * w + 4) for w in (4, 4, 4, 12)]
    assert all(t.data_ptr() % 16 == 0 for t in out)
    for k in range(4):
        ptrs = [C.c_void_p(t.data_ptr() + (4 if j == k else 0)) for j, t in enumerate(out)]
        assert lib.b2k_model_rows(C.byref(ms), 0, 0, *ptrs, None) == api.B2K_ERR_ARG
    assert lib.b2k_model_rows(C.byref(ms), 0, 0, *[C.c_void_p(t.data_ptr()) for t in out], None) == api.B2K_OK
